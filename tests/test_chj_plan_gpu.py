"""CHJ's table planned on the device, against the oracle: one build row, rows
around a CTA's first step and past one step of all CTAs, every row in one
sub-table (the most cells a row), and two sub-tables of which one is full of
one key."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def build_keys(how):
    if isinstance(how, int):
        return G.gen_keys(0, how, 921, 922)
    keys = G.gen_keys(0, 900_000, 921, 922)
    slot = O.leaf_ids(keys, 8)
    one = keys[slot == 17]
    return one if how == "one" else np.concatenate([one, np.repeat(keys[slot == 200][:1], 1500)])


@pytest.mark.parametrize("how", [1, 1023, 4097, 152 * 4096 + 1, "one", "key"])
def test_planned_tables_equal_the_oracle(ctx, how):
    bk = build_keys(how)
    pk = np.concatenate([bk[::5][:50_000], G.gen_keys(0, 777, 923, 924)])
    b = P.BlockStream([P.U32, P.U64], bk, G.payload_columns(925, [P.U32, P.U64], len(bk)))
    p = P.BlockStream([P.U16], pk, G.payload_columns(926, [P.U16], len(pk)))
    ctx.set_int("probe_materialize", 0)  # (past the small joins' form)
    try:
        r = P.runCHJ(b, p, ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""
