"""The consumer's movement with shifts of any size: beyond half the lattice, beyond what an
int can double, and from infinite velocities (which land where the largest int does).
Both stencil paths (narrower and wider than the lattice), both precisions, against a
scatter written out here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

I_MIN, I_MAX = -(1 << 31), (1 << 31) - 1


def _landing(v, pref, axis):
    """Rows (axis 0) or columns the shifted centres fall on: i + v pref in the array's
    precision, rounded half away from 0, clipped to an int, wrapped."""
    L = v.shape[0]
    i = np.arange(L, dtype=v.dtype)
    t = (i[:, None] if axis == 0 else i[None, :]) + v * v.dtype.type(pref)
    r = np.trunc(t) + np.where(np.abs(t - np.trunc(t)) >= 0.5, np.sign(t), 0)
    return np.clip(r.astype(np.float64), I_MIN, I_MAX).astype(np.int64) % L


def _wrapped(g, L):
    w = np.zeros(L)
    for d in range(-len(g) + 1, len(g)):
        w[d % L] += g[abs(d)]
    return w


def _scatter(rho, gam, vx, vy, pref, gD, gV, eps=1e-10):
    L = rho.shape[0]
    with np.errstate(all="ignore"):
        mx, my = _landing(vx, pref, 0), _landing(vy, pref, 1)
    d, v = _wrapped(gD, L), _wrapped(gV, L)
    out = np.zeros((L, L))
    for i in range(L):
        for j in range(L):
            m, g = float(rho[i, j]), float(gam[i, j])
            if m < eps:
                continue
            dr, dc = g * np.roll(d, i), g * np.roll(d, j)
            vr, vc = (1 - g) * np.roll(v, mx[i, j]), (1 - g) * np.roll(v, my[i, j])
            out += m * np.outer(dr + vr, dc + vc)
    return out


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("L,D", [(10, 1.0), (24, 1.0), (40, 0.3)], ids=["wide", "narrow", "narrow-small"])
@pytest.mark.parametrize("far", [[30.0, -47.0], [2.0 ** 30, -2.0 ** 30], [2.0 ** 31, -2.0 ** 31, 1e300], [np.inf, -np.inf]],
                         ids=["laps", "doubling", "beyond-int", "inf"])
def test_far_shifts_match_scatter(far, L, D, precision):
    torch = pytest.importorskip("torch")
    import trophic_maelstorm_gb300 as tmg
    dtype = np.float64 if precision == tmg.TM_FP64 else np.float32
    rng = np.random.default_rng(L)
    rho = rng.uniform(0.5, 3, (L, L))
    rho[rng.random((L, L)) < 0.3] = 0.0
    gam = rng.uniform(0, 1, (L, L))
    vx, vy = rng.uniform(-1, 1, (2, L, L))
    for k, f in enumerate(far):                     # a few sources that carry mass
        for v, (i, j) in ((vx, (k, 3)), (vy, (L - 1 - k, 5))):
            rho[i, j] = 2.0 + k
            v[i, j] = f
    with np.errstate(over="ignore"):
        a = [x.astype(dtype) for x in (rho, gam, vx, vy)]
    p = tmg.fke_parameters(D, 1.0, 1.0, 1.2)
    want = _scatter(*a, p.pref, p.gD, p.gV)
    ts = [torch.as_tensor(x, device="cuda") for x in a]
    tol, floor = (1e-12, 1e-14) if precision == tmg.TM_FP64 else (2e-5, 1e-6 * want.max())
    for ws in (None, tmg.api.fke_workspace(L, precision)):
        got = tmg.fke_advdiff(*ts, p, precision=precision, workspace=ws).cpu().numpy()
        np.testing.assert_allclose(got, want, rtol=tol, atol=floor)
