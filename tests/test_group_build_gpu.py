"""PHJ-PURE on repeated build keys where the build itself groups a leaf's rows
(more than 11 radix bits, leaf tables in shared memory), against the oracle:
every key repeated, three keys among unique leaves, one key of thousands of
rows, leaves of about 60 and 1500 rows (256 and 1024 threads, tables at the
estimated and at the counted size), leaves too large for shared memory, and
payload columns of every width."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def build_keys(how, spread):
    keys = G.gen_keys(0, 250_000 if spread == "even" else 400_000, 811, 812)
    if spread != "even":  # 16 of 4096 leaves: about 1560 rows each, or 5 of about 6000
        leaf = O.leaf_ids(keys, 12)
        keys = keys[leaf < 16] if spread == "few_leaves" else np.concatenate([keys[O.leaf_ids(keys, 6) == 3]])
    if how == "all":
        return np.repeat(keys[: len(keys) // 4], np.arange(len(keys) // 4) % 7 + 1)
    if how == "three":
        return np.concatenate([keys, np.repeat(keys[:3], 5)])
    return np.concatenate([np.repeat(keys[5], 1800), keys])


@pytest.mark.parametrize("spread", ["even", "few_leaves", "dense_bucket"])
@pytest.mark.parametrize("how", ["all", "three", "one"])
@pytest.mark.parametrize("bt,mat", [([], 0), ([P.U8, P.U16, P.U128], 1), ([P.U32, P.U64], 0)])
def test_grouped_builds_equal_the_oracle(ctx, how, spread, bt, mat):
    bk = build_keys(how, spread)
    rng = np.random.default_rng(813)
    bk = bk[rng.permutation(len(bk))]
    pk = np.concatenate([bk[::9], G.gen_keys(0, 3001, 814, 815)])
    if how == "one":  # the repeated key is probed a few times only
        pk = pk[~((pk == build_keys(how, spread)[0]) & (np.arange(len(pk)) > 40))]
    b = P.BlockStream(bt, bk, G.payload_columns(816, bt, len(bk)))
    p = P.BlockStream([P.U32], pk, G.payload_columns(817, [P.U32], len(pk)))
    ctx.set_int("probe_materialize", mat)
    try:
        r = P.runPHJ(b, p, [6, 6], ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""
