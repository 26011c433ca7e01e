"""The measuring autotuner (phj-bench_gb300/autotune.py): candidate
generation and cache keys on the CPU; on the GPU, a tuned configuration
joins bit-exactly and a second call is served from the cache."""
import pytest

import autotune as A
import oracle as O
import phj_gpu as P
from golden import cases


def test_split_bits_follows_the_cli():
    assert A.split_bits(16, 2) == [8, 8]
    assert A.split_bits(17, 2) == [9, 8]
    assert A.split_bits(10, 3) == [4, 3, 3]


def test_radix_candidates_surround_the_heuristic():
    cands = A.radix_candidates(16 << 20)
    assert [8, 8] in cands and [16] in cands and [6, 6, 6] in cands
    assert all(1 <= sum(c) <= 24 and max(c) <= 16 for c in cands)
    assert all(abs(sum(c) - 16) <= 2 for c in cands)


def test_shape_key_buckets_sizes_and_widths():
    k1 = A.shape_key("phj-pure", 1 << 20, 1 << 24, [P.U64], [P.U32])
    k2 = A.shape_key("phj-pure", (1 << 20) + 5, (1 << 24) + 9, [P.U64], [P.U32])
    k3 = A.shape_key("phj-pure", 1 << 20, 1 << 24, [P.U64, P.U32], [P.U32])
    assert k1 == k2 != k3


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", ["phj-pure", "phj"])
def test_tuned_join_is_bit_exact_and_cached(ctx, tmp_path, scheme):
    b, p = cases.make("c3_mini")
    tb, tp = ctx.upload(b), ctx.upload(p)
    cache = str(tmp_path / "tune.json")
    try:
        cfg = A.tune(ctx, tb, tp, scheme=scheme, reps=1, budget_mib=1, cache_path=cache)
        assert cfg["trials"] > 5 and cfg["ms"] > 0
        if scheme == "phj":
            out, _ = ctx.run_phj_bep(tb, tp, cfg["pass_bits"], 1)
        else:
            out, _ = ctx.run_phj_pure(tb, tp, cfg["pass_bits"])
        assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(out.download())) == ""
        out.free()
        again = A.tune(ctx, tb, tp, scheme=scheme, cache_path=cache)
        assert again["cached"] and again["pass_bits"] == cfg["pass_bits"]
    finally:
        A.reset(ctx)
        tb.free(), tp.free()


class OneLaunchContext:
    """A context whose PHJ-PURE joins run in one launch at default options."""

    def __init__(self):
        self.options, self.runs = {}, []

    def set_int(self, name, value):
        self.options[name] = value

    def flush_l2(self):
        pass

    def run_phj_pure(self, b, p, bits):
        class Out:
            def fingerprint(self):
                return (1, 2, 3)

            def free(self):
                pass

        class Res:
            e2e_wall_ms = 1.0 - 0.001 * len(self.runs)  # each a little faster than the last, as noise may have it
        general = any(self.options.get(k, d) != d for k, d in (("table_cap_pct", 200), ("p1_tile_rows", 0), ("p1_stages", 0),
                                                                ("probe_materialize", -1), ("probe_pass_bits", 0)))
        self.last = "probe_fused" if general else "small_join"
        self.runs.append((tuple(bits), self.last))
        return Out(), Res()

    def kernel_times(self):
        return [{"name": self.last, "form": self.last}]


def test_radix_bits_are_not_tuned_where_one_launch_joins():
    class Table:
        rows, types = 5000, [P.U64]

    ctx = OneLaunchContext()
    cfg = A.tune(ctx, Table(), Table(), cache_path=None)
    assert cfg["pass_bits"] == P.autotune_radix(5000)
    assert {bits for bits, _ in ctx.runs} == {tuple(cfg["pass_bits"])}
    assert any(form == "probe_fused" for _, form in ctx.runs)
