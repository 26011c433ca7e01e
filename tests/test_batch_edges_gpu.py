"""The batched join's kernels at the sizes where they can go wrong: one row a
side, around a tile's rows (2048, 4096) and a table piece's (2048), around a
warp's chunk of 128 probe rows, keys that repeat across pieces, a batch whose
rows are wider than the last one's (the workspace's tile changes), every
payload width and no payload.  Rows equal the oracle's."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def pair(i, build, probe, tb, tp, repeat=1):
    bk = G.gen_keys(0, max(build // repeat, 1), 100 + i, 200 + i)
    bk = np.resize(bk, build) if build else bk[:0]
    pk = G.gen_keys(4, probe, 300 + i, 200 + i, domain=max(build // repeat, 1), match_permille=700) if probe else np.zeros(0, dtype=np.uint64)
    return P.BlockStream(tb, bk, G.payload_columns(400 + i, tb, build)), P.BlockStream(tp, pk, G.payload_columns(500 + i, tp, probe))


NARROW = [pair(0, 1, 1, [P.U64], [P.U32]), pair(1, 1024, 127, [P.U64, P.U32], [P.U64]), pair(2, 1025, 129, [], [P.U8]),
          pair(3, 2047, 4095, [P.U32], []), pair(4, 2049, 4097, [P.U16, P.U8], [P.U64]), pair(5, 4096, 8192, [P.U64], [P.U64]),
          pair(6, 33_333, 100_001, [P.U64, P.U32], [P.U64])]
WIDE = [pair(10, 5000, 20_001, [P.U128] * 4, [P.U128] * 8), pair(11, 700, 3000, [P.U8] * 8, [P.U16, P.U128]),
        pair(12, 3000, 500, [P.U64], [P.U32], repeat=3000),      # one key, two pieces
        pair(13, 6000, 900, [P.U128, P.U8], [P.U64], repeat=7)]


@pytest.mark.parametrize("graph", [0, 1])
def test_rows_equal_the_oracle(ctx, graph):
    ctx.set_int("batch_graph", graph)
    try:
        for sides in (NARROW, WIDE, NARROW):
            bs, ps = [ctx.upload(b) for b, _ in sides], [ctx.upload(p) for _, p in sides]
            outs, _ = ctx.run_batch(bs, ps)
            for (b, p), o in zip(sides, outs):
                expected = O.join_rows(b, p)
                assert o.rows == len(expected)
                assert O.compare_outputs(expected, O.serialize_output(o.download())) == ""
                o.free()
            for t in bs + ps:
                t.free()
    finally:
        ctx.set_int("batch_graph", 1)
