"""The Rietkerk RK4 tiles at the sizes where their paths change: bulk row copies (whole
16-byte rows at least a 72-site region wide, one or two segments per row) against
per-thread loads, ragged right and bottom edges, FP64 tile heights, and arguments the
Newton reciprocals hand to the general one.  Bit for bit against the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(oracle, m, R):
    return oracle.rk_params(R=R, sampler=m.sampler)


def _off_step(oracle, m, R, f):
    """The oracle's noise-off step followed by the model's clamp (the oracle's step has none)."""
    want = oracle.rk_det_step(_params(oracle, m, R), f)
    want[(want < want.dtype.type(m.clamp_eps)) & (want >= want.dtype.type(m.clamp_lo))] = 0.0
    return want


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("det", [0, 1], ids=["noise", "off"])
@pytest.mark.parametrize("L", [7, 70, 71, 72, 73, 74, 76, 128, 130, 133, 200])
def test_tile_edges_match_oracle(oracle, precision, det, L):
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    m = tmg.rietkerk_model(deterministic=det)
    dtype = np.float64 if precision == 0 else np.float32
    rng = np.random.default_rng(L)
    f0 = [np.stack([rng.uniform(0, 4, (L, L)), rng.uniform(0.1, 6, (L, L)), rng.uniform(0.5, 9, (L, L))]).astype(dtype)
          for _ in range(2)]
    f0[1][0][: L // 2] = 0.0                               # bare ground: zero products
    Rs = [0.9, 1.2]
    b = tmg.Batch(ctx, m, tmg.instances([L, L], [3, 4], Rs), precision)
    b.upload(f0)
    _, st = b.advance(3, [])
    fin = b.download()
    b.close()
    ctx.close()
    assert not st.any()
    for k in range(2):
        want = f0[k]
        if det:
            for _ in range(3):
                want = _off_step(oracle, m, Rs[k], want)
        else:
            _, _, want, _ = oracle.rk_run(_params(oracle, m, Rs[k]), f0[k], 3 + k, 3, [])
        assert np.array_equal(fin[k], want), (k, L)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("planted", [-5.0, 1e30, 3e-39, np.inf, np.nan])
def test_reciprocal_range_matches_oracle(oracle, precision, planted):
    """W = -k1 (a division by zero), W beyond and below the range of the FP32 method, Inf, NaN."""
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    m = tmg.rietkerk_model(deterministic=1)
    dtype = np.float64 if precision == 0 else np.float32
    L = 96
    rng = np.random.default_rng(1)
    f0 = np.stack([rng.uniform(0, 4, (L, L)), rng.uniform(0.1, 6, (L, L)), rng.uniform(0.5, 9, (L, L))]).astype(dtype)
    f0[1, 5, 6] = planted
    f0[1, 64, 65] = planted * 1e8
    b = tmg.Batch(ctx, m, tmg.instances([L], [3], 0.9), precision)
    b.upload([f0])
    b.advance(1, [])
    fin = b.download()[0]
    b.close()
    ctx.close()
    with np.errstate(all="ignore"):
        want = _off_step(oracle, m, 0.9, f0)
    assert np.array_equal(fin, want, equal_nan=True)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("L", [31, 64, 129])
def test_tile_status_bits(L, precision):
    """A step size far above the stability bound: O goes negative, then overflows; the
    status bits are those of the fields that the tiles stored, each step."""
    import trophic_maelstorm_gb300 as tmg
    dtype = np.float64 if precision == 0 else np.float32
    ctx = tmg.Context(0)
    rng = np.random.default_rng(3)
    b = tmg.Batch(ctx, tmg.rietkerk_model(dt=0.05, deterministic=1), tmg.instances([L, L], [4, 5], 0.9), precision)
    calm = np.stack([np.zeros((L, L)), np.ones((L, L)), np.ones((L, L))]).astype(dtype)
    wild = np.stack([rng.uniform(0, 1, (L, L)), np.full((L, L), 0.5), 1.0 + rng.uniform(-0.1, 0.1, (L, L))]).astype(dtype)
    b.upload([calm, wild])
    want = [0, 0]
    seen = 0
    with np.errstate(all="ignore"):
        for _ in range(100):
            _, st = b.advance(1, [])
            for k, f in enumerate(b.download()):
                want[k] |= (0 if np.all(np.isfinite(f)) else 0x1) | (0x2 if np.any(f < 0) else 0)
                assert int(st[k]) == want[k]
            seen |= want[1]
    b.close()
    ctx.close()
    assert seen == 0x3
