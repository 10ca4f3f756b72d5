"""A launch shape that memory is short for: the batch goes on with the shape that it had, and
with the same fields (TM_PROBE_LIST_GROW refuses the allocation on the host)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(tmg, ctx, model, inst, init, shapes, probe):
    ctx.set_test_probe(probe)
    try:
        b = tmg.Batch(ctx, model, inst, tmg.TM_FP32)
    finally:
        ctx.set_test_probe(0)
    b.upload(init)
    b.advance(33)                                   # step graphs exist, with the list's addresses in them
    seen = []
    for rows, ctas in shapes:
        try:
            b.set_launch(rows, ctas)
            seen.append((b.get_launch(), None))
        except tmg.TMError as e:
            seen.append((b.get_launch(), e.code))
        b.advance(33, [b.step, b.step + 33])
    fin = b.download()
    b.close()
    return seen, fin


@pytest.mark.parametrize("kind", ["dp", "rietkerk"])
def test_list_that_cannot_grow_leaves_the_batch_as_it_was(kind):
    import trophic_maelstorm_gb300 as tmg
    from trophic_maelstorm_gb300 import _lib
    ctx = tmg.Context(0)
    rng = np.random.default_rng(3)
    # 8-row tasks: more than four CTAs per SM of 8 warps have tasks only above 4,864 tasks
    Ls = [700, 33, 1100]
    if kind == "dp":
        model, inst = tmg.dp_model(dt=0.1), tmg.instances(Ls, [1, 2, 3], 0.53)
        init = [rng.uniform(0.0, 2.0, (L, L)).astype(np.float32) for L in Ls]
    else:
        model, inst = tmg.rietkerk_model(), tmg.instances(Ls, [1, 2, 3], 0.9)
        init = [np.stack([rng.uniform(0, 4, (L, L)), rng.uniform(0.1, 6, (L, L)), rng.uniform(0.5, 9, (L, L))])
                .astype(np.float32) for L in Ls]
    # (0, 64): more segments than there are; (16, 64): more entries too; (1, 1): fewer of both
    shapes = [(0, 64), (16, 64), (1, 1), (0, 0), (16, 2)]
    plain, want = _run(tmg, ctx, model, inst, init, [(0, 0)] * len(shapes), 0)
    grown, free = _run(tmg, ctx, model, inst, init, shapes, 0)
    assert [code for _, code in grown] == [None] * len(shapes) and grown[0][0] == (8, 64) and grown[1][0] == (16, 64)
    held, got = _run(tmg, ctx, model, inst, init, shapes, _lib.TM_PROBE_LIST_GROW)
    for k in range(len(Ls)):
        assert np.array_equal(free[k], want[k]) and np.array_equal(got[k], want[k])
    assert held[0] == ((8, 64), None)               # accepted, with the blocks the list has room for
    before = (8, 64)
    for (rows, ctas), (shape, code) in zip(shapes, held):
        asked = (rows or before[0], ctas or before[1])
        assert (shape, code) in ((asked, None), (before, _lib.TM_ERR_NOMEM)), (rows, ctas, shape, code)
        before = shape
    # 33 sites wide lattices in 32-site strips: 16-row tasks need more entries than were made for 8
    assert held[1] == ((8, 64), _lib.TM_ERR_NOMEM)
    ctx.close()
