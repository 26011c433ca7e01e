"""PHJ (BEP) with the device budget against the oracle at the edges of its
steps: one probe row, rows around a scatter step and a slice, first passes of
1 to 11 bits, several and single steps a wave (budgets of 1, 16 and 256 MiB),
leaf tables on both sides of 256 cells, repeated build keys, and every
payload width (a 16-byte probe column takes the chain-following probe)."""
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def inputs(n_build, n_probe, types_b, types_p, repeats, seed):
    if repeats:
        bk, domain = G.gen_multi_match_keys(n_build, seed, seed + 1)
    else:
        bk, domain = G.gen_keys(0, n_build, seed, seed + 1), n_build
    pk = G.gen_keys(4, n_probe, seed + 2, seed + 1, domain=domain, match_permille=700)
    return (P.BlockStream(list(types_b), bk, G.payload_columns(seed + 3, list(types_b), n_build)),
            P.BlockStream(list(types_p), pk, G.payload_columns(seed + 4, list(types_p), n_probe)))


@pytest.mark.parametrize("bits,n_build,n_probe,budget", [
    ([1], 1, 1, 1), ([1], 220, 127, 1), ([1], 300, 128 * 152 + 1, 1), ([1, 12], 9000, 70_001, 1), ([11], 200_000, 300_017, 1),
    ([11, 2], 50_001, 2047, 16), ([6, 7], 400_000, 900_001, 16), ([3], 600, 1_300_003, 256), ([10], 100_003, 2_000_001, 256),
])
@pytest.mark.parametrize("types_b,types_p,repeats", [
    ((P.U64, P.U64), (P.U32,), False), ((P.U32,), (P.U8, P.U16, P.U64), False), ((), (), False), ((P.U8, P.U16), (P.U32, P.U64), True),
    ((P.U128, P.U8), (P.U16, P.U128), False),
])
def test_bep_rows_equal_the_oracle(ctx, bits, n_build, n_probe, budget, types_b, types_p, repeats):
    b, p = inputs(n_build, n_probe, types_b, types_p, repeats, 611)
    r = P.runPhjBep(b, p, bits, bep_budget_mib=budget, ctx=ctx)
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""
