"""Host-buffer PHJ-PURE in the chunks the default option gives (96 MiB of
probe rows, here 136 bytes a row: several chunks and a short last one) and in
pinned ones, against the oracle."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,chunk", [(1_600_003, None), (740_171, None), (1_600_003, 300_000)])
def test_host_chunks_equal_the_oracle(ctx, rows, chunk):
    bt, pt = [P.U64], [P.U128] * 8
    b = P.BlockStream(bt, G.gen_keys(0, 50_000, 901, 902), G.payload_columns(903, bt, 50_000))
    p = P.BlockStream(pt, G.gen_keys(4, rows, 904, 902, domain=50_000, match_permille=60), G.payload_columns(905, pt, rows))
    expected = O.join_rows(b, p)
    n = len(expected)
    keys, left = np.empty(n, np.uint64), [np.empty(n, np.uint64)]
    right = [np.empty((n, 2), np.uint64) for _ in pt]
    if chunk:
        ctx.set_int("host_chunk_rows", chunk)
    try:
        got, _ = ctx.run_phj_pure_host(b, p, [4, 4], keys, left, right)
    finally:
        ctx.set_int("host_chunk_rows", 16 << 20)
    assert got == n
    assert O.compare_outputs(expected, O.serialize_output(P.JoinOutput(bt, pt, keys, left, right))) == ""


@pytest.mark.parametrize("pinned,chunks", [((True, True, True, True), 4), ((True, True, False, True), 2), ((True, True, True, False), 2),
                                           ((True, False, True, True), 2), ((False, True, True, True), 2)])
def test_pageable_columns_take_large_chunks(pinned, chunks):
    # 5.9M rows of 40 bytes (225 MiB): a quarter of a chunk, then chunks of
    # 2.5M between pinned columns; a quarter and the rest where a probe or an
    # output column is pageable
    bt, pt = [P.U64], [P.U64] * 4
    rows = 5_900_000
    b = P.BlockStream(bt, G.gen_keys(0, 50_000, 911, 912), G.payload_columns(913, bt, 50_000))
    pk, cols = G.gen_keys(4, rows, 914, 912, domain=50_000, match_permille=60), G.payload_columns(915, pt, rows)
    fp = O.join_fingerprint(b, P.BlockStream(pt, pk, cols))
    with P.Context(0) as c:
        new = [c.pinned if x else (lambda shape, dtype: np.zeros(shape, dtype)) for x in pinned]
        hk, hc = new[0]((rows,), np.uint64), [new[1]((rows,), np.uint64) for _ in pt]
        for to, a in zip([hk] + hc, [pk] + cols):
            to[...] = a
        keys, left, right = c.pinned((fp[0],), np.uint64), [new[2]((fp[0],), np.uint64)], [new[3]((fp[0],), np.uint64) for _ in pt]
        got, _ = c.run_phj_pure_host(b, P.BlockStream(pt, hk, hc), [4, 4], keys, left, right)
        assert got == fp[0]
        assert [k["name"] for k in c.kernel_times()].count("probe_lookup") == chunks
        out = P.JoinOutput(bt, pt, keys, left, right)
        assert O.rows_fingerprint(O.serialize_output(out), bt, pt) == tuple(fp)
