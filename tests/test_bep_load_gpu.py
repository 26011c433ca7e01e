"""PHJ (BEP) against the oracle when "table_cap_pct" makes the leaf tables
larger than two cells a row and one crowded leaf keeps them from a common
size: the largest table is then more than twice its rows, and the builds take
their shared memory from the tables as they are laid out.  Tables of 64 to
512 cells (a warp's and a CTA's build), all three forms of the scheme."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def crowded(most, few, seed):
    """Build keys of 256 leaves with about `few` rows, one of them with `most`."""
    keys = G.gen_keys(0, 400_000, seed, seed + 1)
    leaf = O.leaf_ids(keys, 8)
    return np.concatenate([keys[leaf == 77][:most], keys[leaf != 77][: 256 * few]])


@pytest.mark.parametrize("pct,most,few", [(300, 45, 8), (300, 20, 4), (800, 20, 4), (800, 45, 8), (800, 64, 9), (110, 100, 10)])
@pytest.mark.parametrize("form", ["engine", "batches", "host"])
def test_largest_table_past_two_cells_a_row(ctx, pct, most, few, form):
    bk = crowded(most, few, 811)
    tb, tp = [P.U64, P.U32], [P.U32]
    b = P.BlockStream(tb, bk, G.payload_columns(812, tb, len(bk)))
    pk = np.concatenate([bk, G.gen_keys(0, 3000, 813, 814), bk[:most]])
    p = P.BlockStream(tp, pk, G.payload_columns(815, tp, len(pk)))
    expected = O.join_rows(b, p)
    ctx.set_int("table_cap_pct", pct)
    ctx.set_int("bep_engine", 0 if form == "engine" else 1)
    try:
        if form == "host":
            keys = np.zeros(len(expected), np.uint64)
            left = [np.zeros(len(expected), P.TYPE_DTYPE[t]) for t in tb]
            right = [np.zeros(len(expected), P.TYPE_DTYPE[t]) for t in tp]
            rows, _ = ctx.run_phj_bep_host(b, p, [4, 4], 1, keys, left, right)
            assert rows == len(expected)
            got = P.JoinOutput(tb, tp, keys, left, right)
        else:
            got = P.runPhjBep(b, p, [4, 4], bep_budget_mib=1, ctx=ctx).output
    finally:
        ctx.set_int("table_cap_pct", 200)
        ctx.set_int("bep_engine", 0)
    assert O.compare_outputs(expected, O.serialize_output(got)) == ""
