"""The joins this library is timed on, through its public entry points.

A case names a scheme, the two sides' rows and payload types, the key
distribution and the radix bits (empty: phj_autotune_radix chooses).  The
inputs are made on the device by the library's seeded generator (the
host-buffer case: then copied to pinned host memory), as the benchmark and
the request loop make them; the context outlives the cases, as in a program
that joins more than once.

A join's output is a set of rows: their order differs from run to run.
run() returns the whole output as it stands on the device; JoinRows puts the
rows in an order of their own only when somebody reads them, so that two
outputs can be compared value by value and a pass pays for the join alone.
How many rows match depends on the seed, so the ordered columns are filled
up with zeros to one length and the number of rows stands beside them.
All outputs are moved keys and payloads, no computed numbers: there is
nothing for a 64-bit computation to add, so there is no exact().
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phj-bench_gb300"))

import phj_gpu as P  # noqa: E402

K, M = 1 << 10, 1 << 20
WIDTH = {"u8": 1, "u16": 2, "u32": 4, "u64": 8, "u128": 16}
SIGNED = {"u8": torch.uint8, "u16": torch.int16, "u32": torch.int32, "u64": torch.int64, "u128": torch.int64}
TYPESTR = {"u8": "|u1", "u16": "<i2", "u32": "<i4", "u64": "<i8", "u128": "<i8"}
# mean rows of a repeated build key: 1 + successes of p = 3/4, at most 16 in all
MULTIPLICITY = sum(0.75 ** j for j in range(16))


def listed():
    return [
        # one small request, alone: the smallest size of the request stream; latency and launches are all of it
        dict(name="pure_4k_x_32k", scheme="pure", keys="unique", build=4 * K, probe=32 * K, left="u64", right="u32", match=700, bits=""),
        # a dimension join whose tables stay in L2 (permutation keys, every row matches), one radix pass
        dict(name="pure_1m_x_8m", scheme="pure", keys="dense", build=M, probe=8 * M, left="u64", right="u32", match=1000, bits="8"),
        # an ordinary join of odd sizes: narrow build payloads, two probe payloads, half of the rows match
        dict(name="pure_3m_x_37m", scheme="pure", keys="unique", build=3_000_017, probe=37_000_003, left="u32,u16,u8", right="u32,u64",
             match=500, bits=""),
        # the benchmark's default workload: both sides far beyond L2
        dict(name="pure_16m_x_256m", scheme="pure", keys="unique", build=16 * M, probe=256 * M, left="u64,u32", right="u64", match=900,
             bits="8,8"),
        # many-to-many: build keys repeat (about 4 rows a key, at most 16), 16-byte payload
        dict(name="multi_32m_x_128m", scheme="pure", keys="multi", build=32 * M, probe=128 * M, left="u8,u16,u128", right="u32", match=500,
             bits=""),
        # the unpartitioned scheme at a size where its table is four times the L2's reach
        dict(name="chj_4m_x_64m", scheme="chj", keys="unique", build=4 * M, probe=64 * M, left="u64,u32", right="u64", match=900, bits=""),
        # best-effort partitioning under Zipf skew within a byte budget, at an ordinary size ...
        dict(name="bep_8m_x_64m", scheme="bep", keys="zipf", build=8 * M, probe=64 * M, left="u64", right="u32", match=1000, bits="6,6,6",
             budget_mib=608),
        # ... and at the benchmark's (32 MiB for each of 152 SMs)
        dict(name="bep_64m_x_512m", scheme="bep", keys="zipf", build=64 * M, probe=512 * M, left="u64", right="u32", match=1000,
             bits="6,6,6", budget_mib=4864),
        # a serving batch: 64 small requests (build rows spread over 4K..256K) in one call
        dict(name="batch_64", scheme="batch", keys="unique", joins=64, build=4 * K, build_most=256 * K, fan=18, left="u64,u32", right="u64",
             match=600),
        # host buffers in, host buffers out (pinned): the form a host caller uses
        dict(name="host_2m_x_24m", scheme="host", keys="unique", build=2 * M, probe=24 * M, left="u64,u32", right="u64", match=900,
             bits="6,6"),
        # the partition operator by itself
        dict(name="shuffle_32m", scheme="shuffle", keys="unique", build=32 * M, left="u64,u32", bits="8,8"),
        # a small join into the caller's own columns, without allocating
        dict(name="noalloc_16k_x_256k", scheme="noalloc", keys="unique", build=16 * K, probe=256 * K, left="u64", right="u32", match=800),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    scheme = rng.choice(["pure", "pure", "pure", "multi", "chj", "bep", "batch", "host", "shuffle", "noalloc"])
    types = ["u32", "u64"]
    left = ",".join(rng.choice(types) for _ in range(rng.randint(1, 3)))
    right = ",".join(rng.choice(types) for _ in range(rng.randint(1, 2)))
    match = rng.randint(100, 1000)
    if scheme == "batch":
        lo = _log(rng, 4 * K, 32 * K)
        return dict(scheme="batch", keys="unique", joins=rng.randint(2, 64), build=lo, build_most=_log(rng, lo, 256 * K), fan=rng.randint(4, 32),
                    left=left, right=right, match=match)
    if scheme == "shuffle":
        n = _log(rng, 64 * K, 32 * M)
        return dict(scheme="shuffle", keys="unique", build=n, left=left, bits=rng.choice(["8", "6,6", "8,8", "6,6,6"]))
    if scheme == "noalloc":
        b = _log(rng, 256, 64 * K)
        return dict(scheme="noalloc", keys=rng.choice(["unique", "dense"]), build=b, probe=_log(rng, 4 * b, 32 * b), left=left, right=right,
                    match=match)
    if scheme == "multi":
        b = _log(rng, 4 * K, 16 * M)
        return dict(scheme=rng.choice(["pure", "pure", "chj"]), keys="multi", build=b, probe=_log(rng, 2 * b, 6 * b),
                    left=rng.choice([left, "u8,u16,u128"]), right=right, match=match, bits="")
    if scheme == "bep":
        b = _log(rng, 16 * K, 16 * M)
        p = _log(rng, 4 * b, 16 * b)
        return dict(scheme="bep", keys=rng.choice(["zipf", "unique"]), build=b, probe=p, left=left.split(",")[0], right=right, match=match,
                    bits=rng.choice(["6,6", "8,8", "6,6,6"]), budget_mib=max(8, (p * 12 >> 20) * rng.choice([1, 2, 8]) // 8))
    b = _log(rng, 4 * K, 8 * M if scheme == "pure" else 4 * M)
    p = _log(rng, 4 * b, 32 * b if scheme == "pure" else 16 * b)
    if scheme == "host":
        b, p = _log(rng, 64 * K, 2 * M), 0
        p = _log(rng, 4 * b, 12 * b)
        return dict(scheme="host", keys="unique", build=b, probe=p, left=left, right=right, match=match, bits=rng.choice(["8", "6,6"]))
    return dict(scheme=scheme, keys=rng.choice(["unique", "unique", "dense"]), build=b, probe=p, left=left, right=right, match=match, bits="")


def _types(text):
    return [P.TYPE_NAMES[t] for t in text.split(",")]


def _bits(case):
    return [int(b) for b in case["bits"].split(",")] if case["bits"] else P.autotune_radix(case["build"], case["probe"])


def _sides(ctx, case, build, probe, seed):
    """A build and a probe table of the case's key distribution."""
    left = _types(case["left"])
    key_seed = seed * 1_000_003 + 17
    if case["keys"] == "dense":
        b = ctx.generate(1, build, key_seed + 1, 0, left)
        return b, ctx.generate(3, probe, key_seed + 2, 0, _types(case["right"]), domain=max(build, build * 1000 // case["match"]))
    if case["keys"] == "multi":
        b = ctx.generate(2, build, key_seed + 1, key_seed, left)
        return b, ctx.generate(4, probe, key_seed + 2, key_seed, _types(case["right"]), domain=b.gen_distinct, match_permille=case["match"])
    b = ctx.generate(0, build, key_seed + 1, key_seed, left)
    if case["keys"] == "zipf":
        return b, ctx.generate(5, probe, key_seed + 2, key_seed, _types(case["right"]), domain=build, theta=1.0)
    return b, ctx.generate(4, probe, key_seed + 2, key_seed, _types(case["right"]), domain=build, match_permille=case["match"])


def _batch_rows(case):
    """Build and probe rows of a batch's joins: build rows evenly spread over the logarithm."""
    n, lo, hi = case["joins"], case["build"], case["build_most"]
    rows = [int(round(lo * (hi / lo) ** (j / max(1, n - 1)))) for j in range(n)]
    return [(b, b * case["fan"] - j) for j, b in enumerate(rows)]


def _pinned(n, t):
    w = WIDTH[t]
    a = torch.empty(n * w, dtype=torch.uint8, pin_memory=True).numpy()
    return a.view(np.uint64).reshape(n, 2) if t == "u128" else a.view(P.TYPE_DTYPE[P.TYPE_NAMES[t]])


def prepare(case, seed):
    ctx = P.default_context()
    s = dict(case=case, ctx=ctx, scheme=case["scheme"])
    if case["scheme"] == "batch":
        pairs = [_sides(ctx, case, b, p, seed * 131 + j) for j, (b, p) in enumerate(_batch_rows(case))]
        s.update(builds=[b for b, _ in pairs], probes=[p for _, p in pairs])
    elif case["scheme"] == "shuffle":
        s.update(build=ctx.generate(0, case["build"], seed * 7 + 1, seed * 1_000_003 + 17, _types(case["left"])), bits=_bits(case))
    else:
        s["build"], s["probe"] = _sides(ctx, case, case["build"], case["probe"], seed)
        if case["scheme"] in ("pure", "bep", "host"):
            s["bits"] = _bits(case)
    if case["scheme"] == "noalloc":
        n = case["probe"]  # build keys are unique: at most one row for each probe row
        cols = {"keys": torch.empty(n, dtype=torch.int64, device="cuda")}
        for side in ("left", "right"):
            for i, t in enumerate(case[side].split(",")):
                cols[f"{side}{i}"] = torch.empty(n, dtype=SIGNED[t], device="cuda")
        s["out"] = cols
        s["at"] = (cols["keys"].data_ptr(), [cols[k].data_ptr() for k in cols if k.startswith("left")],
                   [cols[k].data_ptr() for k in cols if k.startswith("right")])
    if case["scheme"] == "host":
        streams = []
        for table, types in ((s.pop("build"), case["left"].split(",")), (s.pop("probe"), case["right"].split(","))):
            t = table.download()
            keys, cols = _pinned(t.total_rows, "u64"), [_pinned(t.total_rows, x) for x in types]
            for to, a in zip([keys] + cols, [t.keys] + t.payloads):
                to[...] = a
            streams.append(P.BlockStream(t.types, keys, cols))
        s["build"], s["probe"] = streams
        n = case["probe"]
        s["out"] = (_pinned(n, "u64"), [_pinned(n, t) for t in case["left"].split(",")], [_pinned(n, t) for t in case["right"].split(",")])
    return s


def run(s):
    ctx, scheme, case = s["ctx"], s["scheme"], s["case"]
    if scheme == "pure":
        return JoinRows(_device_columns, [ctx.run_phj_pure(s["build"], s["probe"], s["bits"])[0]], case)
    if scheme == "chj":
        return JoinRows(_device_columns, [ctx.run_chj(s["build"], s["probe"])[0]], case)
    if scheme == "bep":
        return JoinRows(_device_columns, [ctx.run_phj_bep(s["build"], s["probe"], s["bits"], case["budget_mib"])[0]], case)
    if scheme == "batch":
        return JoinRows(_device_columns, ctx.run_batch(s["builds"], s["probes"])[0], case)
    if scheme == "host":
        keys, left, right = s["out"]
        rows, _ = ctx.run_phj_pure_host(s["build"], s["probe"], s["bits"], keys, left, right)
        return JoinRows(_host_columns, (rows, s["out"]), case)
    if scheme == "noalloc":
        rows = ctx.run_chj_noalloc(s["build"], s["probe"], case["probe"], *s["at"])
        return JoinRows(_own_columns, (rows, s["out"]), case)
    return JoinRows(_shuffled_columns, ctx.radix_shuffle(s["build"], s["bits"]), case)


class JoinRows(dict):
    """A join's output columns by name, whole; put into a fixed row order when they are first read."""

    def __init__(self, read, held, case):
        super().__init__()
        self.read, self.held, self.case = read, held, case

    def _filled(self):
        if not len(self):
            self.update(self.read(self.held, self.case))
            self.held = None
        return self

    def __iter__(self):
        return dict.__iter__(self._filled())

    def __getitem__(self, k):
        return dict.__getitem__(self._filled(), k)

    def keys(self):
        return dict.keys(self._filled())

    def items(self):
        return dict.items(self._filled())


class _Column:
    """n rows of a device column, for torch."""

    def __init__(self, at, rows, t):
        self.__cuda_array_interface__ = dict(shape=(rows, 2) if t == "u128" else (rows,), typestr=TYPESTR[t], data=(int(at), False), version=3)


def _mixed(cols):
    """A 64-bit mix of each row's values (rows that are equal in all columns get the same)."""
    h = None
    for c in cols.values():
        for v in (c.unbind(1) if c.dim() == 2 else (c,)):
            h = v.to(torch.int64) if h is None else h.mul(-7046029254386353131).add_(v)
            h = h ^ ((h >> 29) & 0x7FFFFFFFF)
            h.mul_(-4658895280553007687)
            h ^= (h >> 32) & 0xFFFFFFFF
    return h


def _most_rows(case):
    """More output rows than a seed of this case comes to."""
    n = _expected_rows(case)
    return int(n * (1.25 if case["keys"] == "multi" else 1.02)) + 4096


def _ordered(cols, case):
    order = torch.sort(_mixed(cols)).indices
    n = len(order)
    out = {"rows": n}
    for k, c in cols.items():
        full = torch.zeros((max(n, _most_rows(case)),) + tuple(c.shape[1:]), dtype=c.dtype, device=c.device)
        torch.index_select(c, 0, order, out=full[:n])
        out[k] = full
    return out


def _device_columns(outputs, case):
    import ctypes as C
    parts = []
    for j, out in enumerate(outputs):
        n, keys, left, right = out.rows, C.c_void_p(), (C.c_void_p * P.MAX_PAYLOADS)(), (C.c_void_p * P.MAX_PAYLOADS)()
        out.ctx._check(out.ctx.lib.phj_output_device_columns(out.handle, C.byref(keys), left, right))
        at = {"keys": (keys.value, "u64")}
        at.update({f"left{i}": (left[i], t) for i, t in enumerate(case["left"].split(","))})
        at.update({f"right{i}": (right[i], t) for i, t in enumerate(case["right"].split(","))})
        cols = {k: torch.as_tensor(_Column(p, n, t), device="cuda") if n else
                torch.empty((0, 2) if t == "u128" else 0, dtype=SIGNED[t], device="cuda") for k, (p, t) in at.items()}
        if len(outputs) > 1:
            cols["join"] = torch.full((n,), j, dtype=torch.int32, device="cuda")
        parts.append(cols)
    whole = parts[0] if len(parts) == 1 else {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    whole = _ordered(whole, case)
    torch.cuda.synchronize()  # the columns go back to the library's pool with `outputs`
    return whole


def _signed(a, t):
    return torch.from_numpy(a.view(np.uint8 if t == "u8" else "i%d" % min(8, WIDTH[t])))


def _host_columns(held, case):
    rows, (keys, left, right) = held
    cols = {"keys": _signed(keys[:rows], "u64")}
    cols.update({f"left{i}": _signed(c[:rows], t) for i, (c, t) in enumerate(zip(left, case["left"].split(",")))})
    cols.update({f"right{i}": _signed(c[:rows], t) for i, (c, t) in enumerate(zip(right, case["right"].split(",")))})
    return _ordered({k: c.cuda() for k, c in cols.items()}, case)


def _own_columns(held, case):
    rows, cols = held
    return _ordered({k: c[:rows] for k, c in cols.items()}, case)


def _shuffled_columns(held, case):
    """Partitions in their order; a partition's rows have none of their own."""
    table, counts = held
    t = table.download()
    cols = {"keys": _signed(t.keys, "u64").cuda()}
    cols.update({f"left{i}": _signed(c, x).cuda() for i, (c, x) in enumerate(zip(t.payloads, case["left"].split(",")))})
    counts = torch.from_numpy(counts.astype(np.int64)).cuda()
    part = torch.repeat_interleave(torch.arange(len(counts), device="cuda", dtype=torch.int32), counts)
    order = torch.sort(_mixed(cols)).indices
    order = order[torch.sort(part[order], stable=True).indices]
    return dict({k: c[order] for k, c in cols.items()}, partition_rows=counts)


def _pairs(case):
    return _batch_rows(case) if case["scheme"] == "batch" else [(case["build"], case["probe"])]


def _expected_rows(case):
    rate = 1.0 if case["keys"] == "zipf" else case["match"] / 1000
    if case["keys"] == "multi":
        rate *= MULTIPLICITY
    return rate * sum(p for _, p in _pairs(case))


def work(case):
    """Each input row read once, each output row written once."""
    lw = sum(WIDTH[t] for t in case["left"].split(","))
    if case["scheme"] == "shuffle":
        return {"bytes": 2 * case["build"] * (8 + lw), "flops": 0}
    rw = sum(WIDTH[t] for t in case["right"].split(","))
    return {"bytes": sum(b * (8 + lw) + p * (8 + rw) for b, p in _pairs(case)) + _expected_rows(case) * (8 + lw + rw), "flops": 0}
