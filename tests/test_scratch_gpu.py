"""The scratch memory a context keeps between calls ("scratch_bytes"): it is
sized by what a call holds at a time, so the scratch of one step is the next
one's again, and a call that runs out of memory beside it goes on without."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def sides(ctx, build, probe, repeat=1, types=(P.U64,)):
    distinct = build // repeat
    bk = np.resize(G.gen_keys(0, distinct, 901, 902), build)
    b = P.BlockStream(list(types), bk, G.payload_columns(903, list(types), build))
    p = P.BlockStream([P.U32], G.gen_keys(4, probe, 904, 902, domain=distinct, match_permille=500), G.payload_columns(905, [P.U32], probe))
    return b, p, ctx.upload(b), ctx.upload(p)


def kept(options, build, probe, call, repeat=1):
    """The block a new context keeps once a first call has said how much it
    needs: it is there for the second, and the third finds it large enough."""
    with P.Context(0) as c:
        for k, v in options.items():
            c.set_int(k, v)
        b, p, t, u = sides(c, build, probe, repeat)
        fp = O.join_fingerprint(b, p)
        sizes = []
        for _ in range(3):
            out, _ = call(c, t, u)
            sizes.append(c.get_int("scratch_bytes"))
            assert tuple(out.fingerprint()) == tuple(fp)
            out.free()
        t.free(), u.free()
        assert sizes[0] == 0 and sizes[1] == sizes[2] > 0
        return sizes[2]


def test_batches_use_the_same_scratch():
    # 24 batches of 1 MiB keep no more than 3 do
    call = lambda c, t, u: c.run_phj_bep(t, u, [6, 6], 1)  # noqa: E731
    few, many = (kept({"bep_engine": 1}, 100_000, n, call) for n in (262_144, 2_097_152))
    assert many == few


def test_tables_that_cannot_be_used_go_back():
    # repeated keys: the tables tried first (one 8-byte payload in the cells)
    # are not held beside the ones that are used
    call = lambda c, t, u: c.run_phj_pure(t, u, [12])  # noqa: E731
    tried, plain = (kept({"probe_materialize": 0, "pack_build": pack}, 1 << 20, 1 << 20, call, repeat=4) for pack in (1, 0))
    assert tried <= plain * 1.01


def test_a_call_out_of_memory_beside_the_block_is_run_again_once():
    # a large join's block, then a join whose output does not fit beside it
    # but does without it: the first call is run again, the later ones are not
    with P.Context(0) as c:
        c.set_int("probe_materialize", 0)
        _, _, t, u = sides(c, 1 << 21, 1 << 12)
        for _ in range(3):
            c.run_phj_pure(t, u, [12])[0].free()
        block = c.get_int("scratch_bytes")
        assert block > (64 << 20)
        t.free(), u.free()
        b, p, t, u = sides(c, 1 << 18, 1 << 20)
        fp = tuple(O.join_fingerprint(b, p))
        inputs = (1 << 18) * 16 + (1 << 20) * 12
        out = (1 << 20) * 20
        c.set_int("test_memory_limit_mib", (inputs + out + block - (8 << 20)) >> 20)
        launches = []
        for _ in range(6):
            n0 = c.launch_count()
            o, _ = c.run_phj_pure(t, u, [10])
            launches.append(c.launch_count() - n0)
            assert tuple(o.fingerprint()) == fp
            o.free()
        c.set_int("test_memory_limit_mib", 0)
        assert launches[0] > launches[1] and launches[1:] == [launches[1]] * 5, launches
        t.free(), u.free()


def test_growing_the_block_waits_for_no_other_stream():
    torch = pytest.importorskip("torch")
    with P.Context(0) as c:
        small, large = (sides(c, n, 4 * n) for n in (1 << 17, 1 << 20))
        for s in (small, large):  # every kernel once, and the first block's size
            c.run_phj_pure(s[2], s[3], [10])[0].free()
        c.run_phj_pure(small[2], small[3], [10])[0].free()
        before = c.get_int("scratch_bytes")
        huge = sides(c, 1 << 21, 1 << 22)
        c.run_phj_pure(huge[2], huge[3], [10])[0].free()
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(1_000_000_000)  # about half a second
            done = torch.cuda.Event()
            done.record()
        c.run_phj_pure(huge[2], huge[3], [10])[0].free()
        assert not done.query()
        assert c.get_int("scratch_bytes") > before
        torch.cuda.synchronize()
        for s in (small, large, huge):
            s[2].free(), s[3].free()


def test_trim_gives_the_kept_memory_back():
    torch = pytest.importorskip("torch")
    with P.Context(0) as c:
        b, p, t, u = sides(c, 1 << 21, 1 << 23)
        fp = tuple(O.join_fingerprint(b, p))
        for _ in range(3):
            c.run_phj_pure(t, u, [12])[0].free()
        out, _ = c.run_phj_pure(t, u, [12])
        block = c.get_int("scratch_bytes")
        assert block > (64 << 20)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        c.trim()
        assert c.get_int("scratch_bytes") == 0
        assert torch.cuda.mem_get_info()[0] >= free + block - (4 << 20)
        assert tuple(out.fingerprint()) == fp
        out.free()
        out, _ = c.run_phj_pure(t, u, [12])
        assert tuple(out.fingerprint()) == fp
        for o in (out, t, u):
            o.free()


@pytest.mark.parametrize("scheme,limit", [("pure", 64), ("chj", 52)])
def test_tables_of_counted_sizes_where_the_estimated_ones_do_not_fit(scheme, limit):
    # 400K rows of 12 payload bytes on 400K: 12.8 MB of inputs, 8 partitioned
    # (PHJ-PURE), 3.2 of chains, 6.4 packed, 9.6 of output, and 33.6 MB of
    # tables by estimate (25.6 planned in CHJ) against 16.8 counted
    with P.Context(0) as c:
        c.set_int("probe_materialize", 0)
        b, p, t, u = sides(c, 400_000, 400_000, types=(P.U64, P.U32))
        fp = tuple(O.join_fingerprint(b, p))
        c.set_int("test_memory_limit_mib", limit)
        launches = []
        for _ in range(4):
            n0 = c.launch_count()
            o, _ = c.run_phj_pure(t, u, [10]) if scheme == "pure" else c.run_chj(t, u)
            launches.append(c.launch_count() - n0)
            assert tuple(o.fingerprint()) == fp
            o.free()
        assert launches[0] > launches[1] == launches[2] == launches[3], launches
        c.set_int("test_memory_limit_mib", 0)
        t.free(), u.free()
