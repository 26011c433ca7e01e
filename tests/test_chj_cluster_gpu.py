"""CHJ with the probe side first put in sub-table order (probe_materialize 1)
against the oracle and against the probe in input order: unique, repeated
and edge keys, every payload width, irregular blocks, one probe row and row
counts around a tile."""
import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P
from golden import cases

pytestmark = pytest.mark.gpu


def odd(probe):
    b, p = P.BlockStream([P.U32, P.U8], G.gen_keys(0, 5001, 81, 82), G.payload_columns(83, [P.U32, P.U8], 5001),
                         block_rows=np.array([4000, 1, 1000], dtype=np.uint32)), None
    p = P.BlockStream([P.U64, P.U16], G.gen_keys(4, probe, 84, 82, domain=5001, match_permille=600), G.payload_columns(85, [P.U64, P.U16], probe))
    return b, p


@pytest.mark.parametrize("name", cases.NAMES + [1, 1023, 4097, 60_001])
def test_clustered_rows_equal_the_oracle(ctx, name):
    b, p = cases.make(name) if isinstance(name, str) else odd(name)
    expected = O.join_rows(b, p)
    for how in (1, 0):
        ctx.set_int("probe_materialize", how)
        try:
            r = P.runCHJ(b, p, ctx=ctx)
        finally:
            ctx.set_int("probe_materialize", -1)
        assert O.compare_outputs(expected, O.serialize_output(r.output)) == ""


@pytest.mark.parametrize("build,types,pack,clustered", [
    (3_000_000, [P.U64, P.U32], 1, True),     # one kernel looks up and projects: the line is 1.2 x L2
    (3_000_000, [P.U64, P.U32], 0, False),    # two kernels: twice L2
    (3_000_000, [P.U64] * 3, 1, False),
    (6_000_000, [P.U64] * 3, 1, True),
])
def test_when_the_probe_side_is_put_in_order(ctx, build, types, pack, clustered):
    b = ctx.generate(0, build, 751, 752, types)
    p = ctx.generate(4, 4_000_000, 753, 752, [P.U64], domain=build, match_permille=700)
    fps = []
    for m in (-1, 0):
        ctx.set_int("pack_build", pack)
        ctx.set_int("probe_materialize", m)
        try:
            out, _ = ctx.run_chj(b, p)
        finally:
            ctx.set_int("pack_build", 1)
            ctx.set_int("probe_materialize", -1)
        assert ("probe_scatter" in {k["name"] for k in ctx.kernel_times()}) == (clustered and m < 0)
        fps.append(out.fingerprint())
        out.free()
    assert fps[0] == fps[1]
    b.free(), p.free()
