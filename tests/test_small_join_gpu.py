"""Joins of a small build side in one launch against the oracle, and against
the general path that a pinned option keeps: one row a side, around a warp's
chunk (32 and 128 probe rows), a CTA's threads (1024) and a piece (8192
rows), several pieces, keys that repeat inside and across pieces, more
output rows than probe rows (two launches), a long probe side of a build
side that repeats (the general path takes over), every payload
width and no payload, twice in a row (the counter starts cleared)."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def sides(build, probe, tb, tp, repeat, match):
    distinct = max(build // repeat, 1)
    bk = np.resize(G.gen_keys(0, distinct, 601, 602), build)
    pk = G.gen_keys(4, probe, 603, 602, domain=distinct, match_permille=match)
    return P.BlockStream(tb, bk, G.payload_columns(604, tb, build)), P.BlockStream(tp, pk, G.payload_columns(605, tp, probe))


@pytest.mark.parametrize("build,probe,tb,tp,repeat,match", [
    (1, 1, [P.U64], [P.U32], 1, 1000),
    (3, 33, [], [], 1, 500),
    (1023, 127, [P.U32, P.U16, P.U8], [P.U64], 1, 900),
    (1025, 152 * 1024 + 1, [P.U64, P.U32], [P.U64, P.U8], 1, 600),   # 128 rows a warp instead of 32
    (8192, 5000, [P.U128, P.U8], [P.U16, P.U128], 1, 700),
    (8193, 30_001, [P.U64], [P.U64], 1, 800),                        # two pieces
    (60_000, 20_000, [P.U32] * 8, [P.U8] * 8, 1, 800),               # eight pieces, eight columns a side
    (20_000, 40_000, [P.U64], [P.U32], 5, 150),                      # repeats, fewer output than probe rows
    (20_000, 9000, [P.U64, P.U128], [P.U32], 20_000, 1000),          # one key: 20,000 rows a match
    (3000, 20_000, [P.U16, P.U64], [P.U32], 4, 900),                 # more output rows than probe rows
    (3000, 400_001, [P.U64], [P.U32], 2, 300),                       # repeats and a long probe side: the general path
    (65_536, 4000, [P.U64], [P.U32], 1, 900),                        # the most build rows
])
def test_rows_equal_the_oracle(ctx, build, probe, tb, tp, repeat, match):
    b, p = sides(build, probe, tb, tp, repeat, match)
    if build == 20_000 and repeat == 20_000:
        p = P.BlockStream(tp, p.keys[:40], [c[:40] for c in p.payloads])
    expected = O.join_rows(b, p)
    t, u = ctx.upload(b), ctx.upload(p)
    general = repeat > 1 and p.total_rows > 400_000
    for pinned in (False, False, True):
        for scheme in ("pure", "chj"):
            if pinned:
                ctx.set_int("probe_materialize", 0)
            try:
                out, _ = ctx.run_phj_pure(t, u, [6]) if scheme == "pure" else ctx.run_chj(t, u)
            finally:
                ctx.set_int("probe_materialize", -1)
            if scheme == "pure":
                assert ("small_join" in {k["name"] for k in ctx.kernel_times()}) == (not pinned and not general)
            assert O.compare_outputs(expected, O.serialize_output(out.download())) == ""
            out.free()
    t.free(), u.free()


def test_an_output_of_the_probe_rows_does_not_fit():
    # few of the rows match, and memory holds the join's rows but not one for
    # each probe row: the general path counts them first
    with P.Context(0) as c:
        tb, tp = [P.U128, P.U128], [P.U32]
        b, p = sides(1000, 4_000_000, tb, tp, 1, 20)
        expected = O.join_rows(b, p)
        t, u = c.upload(b), c.upload(p)
        inputs = 1000 * 40 + 4_000_000 * 12
        c.set_int("test_memory_limit_mib", (inputs >> 20) + 100)  # (one row each: 168 MiB)
        for _ in range(2):
            out, _ = c.run_phj_pure(t, u, [6])
            assert "small_join" not in {k["name"] for k in c.kernel_times()}
            assert O.compare_outputs(expected, O.serialize_output(out.download())) == ""
            out.free()
        t.free(), u.free()


@pytest.mark.parametrize("scheme", ["pure", "chj"])
def test_a_join_of_2_32_rows_is_refused(ctx, scheme):
    # one key on both sides: 65,536 x 70,000 output rows
    t = ctx.upload(P.BlockStream([P.U32], np.full(65_536, 9, np.uint64), [np.arange(65_536, dtype=np.uint32)]))
    u = ctx.upload(P.BlockStream([], np.full(70_000, 9, np.uint64), []))
    with pytest.raises(P.PhjError) as e:
        ctx.run_phj_pure(t, u, [6]) if scheme == "pure" else ctx.run_chj(t, u)
    assert e.value.status == P.ERR_CAPACITY and str(65_536 * 70_000) in str(e.value)
    t.free(), u.free()


@pytest.mark.parametrize("build,probe,distinct,tb,tp,match", [
    (1000, 3000, 200, [P.U64], [P.U32], 900),                  # five rows a key: one more than a lane writes alone
    (1000, 3001, 15, [P.U64, P.U32], [P.U16], 700),            # 66 or 67 rows: chains start at any row
    (1003, 500, 1, [P.U128, P.U8], [P.U128], 800),             # one key, 16-byte columns on both sides
    (8192, 200_001, 125, [P.U16], [P.U8, P.U64], 30),          # long probe side, few chunks of 128 a warp
    (60_000, 300_000, 3000, [P.U32], [], 100),                 # ... and many, eight pieces
    (60_000, 300_000, 30_000, [P.U32], [P.U32], 300),          # two rows a key, in pieces of their own
])
def test_long_chains(ctx, build, probe, distinct, tb, tp, match):
    bk = np.resize(G.gen_keys(0, distinct, 611, 612), build)
    bk[build // 2:build // 2 + 40] = bk[3]                     # and one key more often than the others
    b = P.BlockStream(tb, bk, G.payload_columns(613, tb, build))
    p = P.BlockStream(tp, G.gen_keys(4, probe, 614, 612, domain=distinct, match_permille=match), G.payload_columns(615, tp, probe))
    expected = O.join_fingerprint(b, p)
    t, u = ctx.upload(b), ctx.upload(p)
    for _ in range(2):
        out, _ = ctx.run_phj_pure(t, u, [6])
        assert "small_join" in {k["name"] for k in ctx.kernel_times()}
        assert out.fingerprint() == expected
        out.free()
    t.free(), u.free()


@pytest.mark.parametrize("cap", [1, 4097, 33_002])
def test_chains_past_the_capacity(ctx, cap):
    # the no-allocation join: rows past the caller's columns are counted, and
    # nothing is written behind them
    torch = pytest.importorskip("torch")
    b, p = sides(1000, 2000, [P.U64], [P.U32], 67, 900)
    rows = O.join_fingerprint(b, p)[0]
    t, u = ctx.upload(b), ctx.upload(p)
    keys, left = (torch.full((rows,), -7, dtype=torch.int64, device="cuda") for _ in range(2))
    right = torch.full((rows,), -7, dtype=torch.int32, device="cuda")
    with pytest.raises(P.PhjError) as e:
        ctx.run_chj_noalloc(t, u, cap, keys.data_ptr(), [left.data_ptr()], [right.data_ptr()])
    assert e.value.status == P.ERR_CAPACITY and e.value.rows == rows > cap
    assert all((c[cap:] == -7).all() for c in (keys, left, right))
    of = {}
    for k, v in zip(b.keys.tolist(), b.payloads[0].tolist()):
        of.setdefault(k, set()).add(v)
    assert all(v % 2**64 in of[k % 2**64] for k, v in zip(keys[:cap].tolist(), left[:cap].tolist()))
    t.free(), u.free()


@pytest.mark.parametrize("option,value,default", [("p1_tile_rows", 2048, 0), ("p1_stages", 2, 0), ("probe_pass_bits", 5, 0), ("table_cap_pct", 150, 200),
                                                  ("pack_build", 0, 1), ("probe_fused", 0, 1), ("probe_materialize", 1, -1)])
def test_an_option_of_the_general_path_keeps_it(ctx, option, value, default):
    b, p = sides(3000, 9000, [P.U64], [P.U32], 1, 700)
    for v, small in ((default, True), (value, False)):
        ctx.set_int(option, v)
        try:
            r = P.runPHJ(b, p, [6], ctx=ctx)
        finally:
            ctx.set_int(option, default)
        assert ("small_join" in {k["form"] for k in ctx.kernel_times()}) == small
        assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""


def test_one_launch_counts_as_the_probe(ctx):
    b, p = sides(3000, 9000, [P.U64], [P.U32], 1, 700)
    t, u = ctx.upload(b), ctx.upload(p)
    with pytest.raises(P.PhjError):
        ctx.run_phj_pure(t, u, [16, 9])  # the bits are checked all the same
    out, r = ctx.run_phj_pure(t, u, [6])
    assert r.build_shuffle.wall_ms == r.build.wall_ms == r.probe_shuffle.wall_ms == 0
    assert r.probe.wall_ms == pytest.approx(r.e2e_wall_ms) and r.e2e_wall_ms > 0
    out.free()
    out, r = ctx.run_chj(t, u)
    assert r.build.wall_ms == 0 and r.probe.wall_ms == pytest.approx(r.e2e_wall_ms)
    for o in (out, t, u):
        o.free()
