"""The launch shape that a batch reports is the one it runs with, in both precisions; the
fields and the measurements do not depend on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,resident", [(0, 2), (1, 4)], ids=["fp64", "fp32"])
def test_ctas_per_sm(precision, resident):
    import trophic_maelstorm_gb300 as tmg
    dtype = np.float64 if precision == 0 else np.float32
    rng = np.random.default_rng(5)
    ctx = tmg.Context(0)
    Ls = [300, 33, 257]
    init = [(rng.uniform(0.0, 2.0, (L, L)) * (rng.random((L, L)) < 0.6)).astype(dtype) for L in Ls]
    got = []
    for shape in (None, (1, 1), (1, 2), (2, 3), (1, 64), "auto"):
        b = tmg.Batch(ctx, tmg.dp_model(dt=0.1), tmg.instances(Ls, [4, 5, 6], 0.53), precision)
        assert b.get_launch()[1] == resident                  # a new batch: the resident blocks
        b.upload(init)
        if shape == "auto":
            assert b.autotune(2)[1] in (1, 2, 3, 4)
        elif shape:
            b.set_launch(*shape)
            assert b.get_launch() == shape
        obs, _ = b.advance(4, [0, 2, 4])
        got.append((obs[:, :, 1], b.download()))
        b.close()
    ctx.close()
    for active, fields in got[1:]:
        assert np.array_equal(active, got[0][0])
        assert all(np.array_equal(f, w) for f, w in zip(fields, got[0][1]))
