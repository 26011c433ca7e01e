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
