"""The kernel behind each timing record: a step's name is the same whichever
kernel did it, its form is the kernel's.  And the general one-pass probe of
CHJ at its chunk edges (256 probe rows), which a join this small takes only
when an option pins it."""
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P

pytestmark = pytest.mark.gpu


def sides(build, probe, tb, tp, match=700):
    b = P.BlockStream(tb, G.gen_keys(0, build, 741, 742), G.payload_columns(743, tb, build))
    return b, P.BlockStream(tp, G.gen_keys(4, probe, 744, 742, domain=build, match_permille=match), G.payload_columns(745, tp, probe))


def forms(ctx, name):
    return [k["form"] for k in ctx.kernel_times() if k["name"] == name]


@pytest.mark.parametrize("build,probe,tb,pinned,scheme,name,form", [
    (3000, 9000, [P.U64], False, "pure", "small_join", "small_join"),
    (3000, 9000, [P.U64], False, "chj", "probe_fused", "small_join"),
    (3000, 9000, [P.U64], True, "chj", "probe_fused", "probe_fused"),
    (3000, 9000, [P.U64], True, "pure", "probe_fused", "probe_inline"),
    (3000, 9000, [P.U8], True, "pure", "probe_inline", "probe_inline"),
    (3000, 9000, [P.U64, P.U32], True, "pure", "probe_fused", "probe_fused"),
    (100_000, 400_000, [P.U64], False, "pure", "probe_fused", "probe_inline"),
    (100_000, 400_000, [P.U64, P.U32], False, "pure", "probe_fused", "probe_fused"),
])
def test_record_forms(ctx, build, probe, tb, pinned, scheme, name, form):
    b, p = sides(build, probe, tb, [P.U32])
    ctx.set_int("probe_materialize", 0 if pinned else -1)
    try:
        P.runCHJ(b, p, ctx=ctx) if scheme == "chj" else P.runPHJ(b, p, [6], ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    assert forms(ctx, name) == [form]
    assert all(k["form"] for k in ctx.kernel_times())


@pytest.mark.parametrize("probe,form", [(4000, "small_join"), (2_000_000, "noalloc_probe")])
def test_noalloc_form(ctx, probe, form):
    b, p = sides(50_000, probe, [], [])
    t, u = ctx.upload(b), ctx.upload(p)
    with pytest.raises(P.PhjError) as e:
        ctx.run_chj_noalloc(t, u, 0, 0, [], [])
    assert e.value.status == P.ERR_CAPACITY
    assert forms(ctx, "noalloc_probe") == [form]
    t.free(), u.free()


@pytest.mark.parametrize("rows,match", [(1, 1000), (255, 1000), (256, 0), (257, 500), (512 * 3 + 1, 1000)])
@pytest.mark.parametrize("tb", [[P.U64, P.U32], [P.U64], [P.U32], []])
def test_chj_one_pass_probe_at_chunk_edges(ctx, rows, match, tb):
    b, p = sides(3000, rows, tb, [P.U64], match)
    ctx.set_int("probe_materialize", 0)
    try:
        r = P.runCHJ(b, p, ctx=ctx)
    finally:
        ctx.set_int("probe_materialize", -1)
    assert forms(ctx, "probe_fused") == ["probe_fused"]
    assert O.compare_outputs(O.join_rows(b, p), O.serialize_output(r.output)) == ""
