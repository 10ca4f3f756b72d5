"""FP32 draw: Poisson means through every length of the unrolled search and past its end,
and boosted shapes down to where 1/k and U^(1/k) leave the normal range.  Bit for bit
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampler", [0, 1])
@pytest.mark.parametrize("dt,lo,hi", [(0.1, -3, 0.6), (0.06, -0.5, 0.2), (0.1, -30, -1)],
                         ids=["m-to-60", "around-32", "tiny-shapes"])
def test_fp32_draw_matches_oracle(oracle, dt, lo, hi, sampler):
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(17)
    ctx = tmg.Context(0)
    Ls = [33, 96, 257]
    model = tmg.dp_model(dt=dt, sampler=sampler)
    init = []
    for L in Ls:
        f = (10.0 ** rng.uniform(lo, hi, (L, L))).astype(np.float32)
        f[rng.random((L, L)) < 0.3] = 0.0
        init.append(f)
    b = tmg.Batch(ctx, model, tmg.instances(Ls, [2 + k for k in range(len(Ls))], 0.53), tmg.TM_FP32)
    b.upload(init)
    _, st = b.advance(4, [])
    fin = b.download()
    b.close()
    ctx.close()
    for k, L in enumerate(Ls):
        p = oracle.DPParams(0.53, 0.0, model.b, model.c, model.D, model.sigma, model.dt, model.dx, model.clamp_lo,
                            model.clamp_eps, model.remainder, model.sampler)
        _, _, want, ost = oracle.dp_run(p, init[k], 2 + k, 4, [4])
        assert np.array_equal(fin[k], want), (k, L)
        assert st[k] == ost


@pytest.mark.parametrize("n", [1, 30])
def test_fp32_default_rows_do_not_change_the_fields(n):
    """A batch large enough for 16-row tasks, and one below: the same bits as 8-row and 5-row tasks."""
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(23)
    ctx = tmg.Context(0)
    Ls = [513] * n + [40]
    init = [(rng.uniform(0.0, 2.0, (L, L)) * (rng.random((L, L)) < 0.5)).astype(np.float32) for L in Ls]
    got = []
    for rows in (0, 8, 5):
        b = tmg.Batch(ctx, tmg.dp_model(dt=0.1), tmg.instances(Ls, list(range(len(Ls))), 0.53), tmg.TM_FP32)
        if rows:
            b.set_launch(rows, 0)
        elif n == 30:
            assert b.get_launch()[0] == 16
        b.upload(init)
        b.advance(3, [])
        got.append(b.download())
        b.close()
    ctx.close()
    for k in range(len(Ls)):
        assert np.array_equal(got[0][k], got[1][k]) and np.array_equal(got[0][k], got[2][k])


def test_fp32_list_grows_with_the_grid():
    """More blocks per SM than a batch was created for: its list of deferred sites is laid out again."""
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(29)
    ctx = tmg.Context(0)
    f = rng.uniform(0.0, 2.0, (700, 700)).astype(np.float32)
    got = []
    for launches in ([], [(1, 0), (0, 64), (0, 2)], [(1, 64)]):
        b = tmg.Batch(ctx, tmg.dp_model(dt=0.1), tmg.instances([700], [3], 0.53), tmg.TM_FP32)
        b.upload([f])
        b.advance(1, [])
        for rows, ctas in launches:
            b.set_launch(rows, ctas)
            b.advance(1, [])
        b.advance(4 - 1 - len(launches), [])
        got.append(b.download()[0])
        b.close()
    ctx.close()
    assert np.array_equal(got[0], got[2]) and np.array_equal(got[0], got[1])
