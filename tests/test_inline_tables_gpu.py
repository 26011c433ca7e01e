"""PHJ-PURE's inline leaf tables (unique keys, at most 8 build payload bytes,
sized by estimate) against the oracle: every payload width that packs into 8
bytes and no payload, one radix bit, leaves of about 32 rows (the fewest they
take) and of thousands, chunk edges of the probe, keys that mark empty cells
(small integers) on both sides, a leaf past its estimate and repeated keys
(the general tables take over), with and without the probe side's pass.  The
same joins with 12 payload bytes go through the estimated general tables."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def join(ctx, bk, pk, bt, pt, bits, mat):
    b = P.BlockStream(bt, bk, G.payload_columns(701, bt, len(bk)))
    p = P.BlockStream(pt, pk, G.payload_columns(702, pt, len(pk)))
    expected = O.join_rows(b, p)
    ctx.set_int("probe_materialize", mat)
    try:
        r = P.runPHJ(b, p, bits, ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    names = {k["name"] for k in ctx.kernel_times()}
    assert O.compare_outputs(expected, O.serialize_output(r.output)) == ""
    return names


@pytest.mark.parametrize("bt", [[], [P.U8], [P.U16, P.U8], [P.U32], [P.U8, P.U32, P.U16], [P.U64], [P.U8] * 8, [P.U64, P.U32]])
@pytest.mark.parametrize("mat", [0, 1])
def test_payload_widths(ctx, bt, mat):
    bk = G.gen_keys(0, 70_001, 703, 704)
    pk = G.gen_keys(4, 256 * 41 + 3, 705, 704, domain=70_001, match_permille=700)
    names = join(ctx, bk, pk, bt, [P.U32, P.U8], [6, 4], mat)
    assert ("build_inline" in names) == (bt != [P.U64, P.U32])


@pytest.mark.parametrize("build,probe,bits", [(33_000, 1, [10]), (4096, 255, [7]), (4096, 257, [1]), (70_000, 5000, [11]), (70_000, 5000, [4, 3]), (9000, 3000, [1]),
                                              (70_000, 5000, [4])])
def test_leaf_sizes_and_chunk_edges(ctx, build, probe, bits):
    bk = G.gen_keys(0, build, 706, 707)
    names = join(ctx, bk, G.gen_keys(4, probe, 708, 707, domain=build, match_permille=800), [P.U64], [P.U64], bits, 0)
    assert "build_inline" in names


def test_keys_that_mark_empty_cells(ctx):
    # unique small integers and the extremes: the markers are among them
    bk = np.concatenate([np.arange(0, 9000, 3, dtype=np.uint64), np.array([2**64 - 1], dtype=np.uint64)])
    pk = np.concatenate([np.arange(0, 20_000, dtype=np.uint64), np.array([2**64 - 1, 2**63], dtype=np.uint64)])
    assert "build_inline" in join(ctx, bk, pk, [P.U32], [P.U16], [4], 0)


@pytest.mark.parametrize("bt", [[P.U32], [P.U64, P.U32]])
@pytest.mark.parametrize("mat", [0, 1])
@pytest.mark.parametrize("how", ["skew", "repeats", "both"])
def test_builds_the_estimate_does_not_hold_for(ctx, bt, mat, how):
    keys = G.gen_keys(0, 400_000, 709, 710)
    leaf = O.leaf_ids(keys, 5)
    skewed = np.concatenate([keys[leaf == 3][:9000], keys[leaf != 3][:8000]])
    bk = {"skew": skewed, "repeats": np.resize(keys[:9000], 20_000), "both": np.resize(skewed, 25_000)}[how]
    join(ctx, bk, np.concatenate([keys[:9000], skewed[::2]]), bt, [P.U32], [5], mat)


@pytest.mark.parametrize("bt", [[P.U32], [P.U64, P.U32]])
@pytest.mark.parametrize("rows,kept", [(400, True), (600, False)])
def test_a_crowded_leaf_is_not_kept_past_the_load(ctx, bt, rows, kept):
    # 32 leaves of about 300 rows, the estimate 411 (cells for 412 rows at the
    # default load in an inline table, for 512 in a general one): a leaf of
    # 600 rows fits neither at that load, though it has fewer rows than cells
    keys = G.gen_keys(0, 400_000, 721, 722)
    leaf = O.leaf_ids(keys, 5)
    bk = np.concatenate([keys[leaf == 3][:rows], keys[leaf != 3][: 9600 - rows]])
    b = P.BlockStream(bt, bk, G.payload_columns(723, bt, len(bk)))
    p = P.BlockStream([P.U32], bk[::3], G.payload_columns(724, [P.U32], len(bk[::3])))
    ctx.set_int("probe_materialize", 0)
    try:
        r = P.runPHJ(b, p, [5], ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    names = [k["name"] for k in ctx.kernel_times()]
    general = names.count("build_leaf_tables")
    assert general == (0 if kept else 1) + (bt == [P.U64, P.U32]), names
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""


@pytest.mark.parametrize("bt", [[P.U32], [P.U64, P.U32]])
@pytest.mark.parametrize("crowded", [0, 1, 2047, 4095])
def test_one_crowded_leaf_of_many(ctx, bt, crowded):
    # found wherever it is among 4,096 leaves of 40 rows; repeated keys make it
    keys = G.gen_keys(0, 400_000, 731, 732)
    leaf = O.leaf_ids(keys, 12)
    bk = np.concatenate([keys[:160_000], np.repeat(keys[leaf == crowded][:1], 700)])
    b = P.BlockStream(bt, bk, G.payload_columns(733, bt, len(bk)))
    pk = np.concatenate([keys[::40], keys[leaf == crowded][:3]])
    p = P.BlockStream([P.U32], pk, G.payload_columns(734, [P.U32], len(pk)))
    r = P.runPHJ(b, p, [6, 6], ctx=ctx)
    assert "build_leaf_tables" in {k["name"] for k in ctx.kernel_times()}
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""


@pytest.mark.parametrize("mat,builds", [(0, 1), (1, 1)])
def test_large_tables_in_input_order_are_counted(ctx, mat, builds):
    # 3M rows of 12 payload bytes in 16,384 leaves: 268 MB of tables by
    # estimate, past L2; probed in input order their sizes are counted
    b = ctx.generate(0, 3_000_000, 761, 762, [P.U64, P.U32])
    p = ctx.generate(4, 3_000_000, 763, 762, [P.U32], domain=3_000_000, match_permille=700)
    ctx.set_int("probe_materialize", mat)
    try:
        out, r = ctx.run_phj_pure(b, p, [7, 7])
    finally:
        ctx.set_int("probe_materialize", -1)
    assert [k["name"] for k in ctx.kernel_times()].count("build_leaf_tables") == builds
    tables = (268 if mat else 134) * 10**6
    inputs, copies, out_bytes = 3_000_000 * 32, 3_000_000 * (2 * 20 + 8 + 16 + 12 * mat), 3_000_000 * 24
    assert abs(r.peak_mem_bytes - (inputs + copies + out_bytes + tables)) < 30 * 10**6, r.peak_mem_bytes
    for o in (out, b, p):
        o.free()
