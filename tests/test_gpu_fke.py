"""The consumer's movement at the sizes where its kernels change path: lattices as wide as
a stencil or one narrower, ragged column segments of 256, shifts listed by bits (up to 3)
or scanned, and shifts beyond the lattice.  Against the oracle's scatter; sums of at most a
few hundred non-negative terms, so FP64 agrees to 1e-12 and FP32 to 2e-5 as in the fixture
test.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workspace", [False, True], ids=["alloc", "ws"])
@pytest.mark.parametrize("L,D,vmax", [(10, 1.0, 1.0), (11, 1.0, 1.0), (12, 1.0, 9.0), (33, 0.3, 0.2), (255, 1.0, 4.0),
                                      (256, 2.0, 4.4), (257, 1.0, 6.0), (300, 0.3, 1.0), (40, 1.0, 100.0)])
def test_fke_paths_match_oracle(oracle, L, D, vmax, workspace):
    pytest.importorskip("torch")
    import torch
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(L)
    rho = rng.uniform(0, 3, (L, L))
    rho[rng.random((L, L)) < 0.3] = 0.0
    rho[0, 1] = 5e-11                                          # below eps
    gam = rng.uniform(0, 1, (L, L))
    vx, vy = rng.uniform(-vmax, vmax, (2, L, L))
    p = tmg.fke_parameters(D, 1.0, 1.0, 1.2)
    want = oracle.fke_advdiff(rho, gam, vx, vy, p.pref, p.gD, p.gV).reshape(L, L)
    gam[rho < 1e-10] = np.nan                                  # a source without mass must not matter
    for precision, dtype, tol in ((tmg.TM_FP64, np.float64, 1e-12), (tmg.TM_FP32, np.float32, 2e-5)):
        ts = [torch.as_tensor(a.astype(dtype), device="cuda") for a in (rho, gam, vx, vy)]
        if precision == tmg.TM_FP32:
            # the shift is the rounding of the precision's own product: compare where both agree
            f = [t.double().cpu().numpy() for t in ts]
            want = oracle.fke_advdiff(f[0], np.nan_to_num(f[1]), _shifts(f[2], p.pref, 0), _shifts(f[3], p.pref, 1), 1.0, p.gD,
                                      p.gV).reshape(L, L)
        ws = tmg.api.fke_workspace(L, precision) if workspace else None
        got = tmg.fke_advdiff(*ts, p, precision=precision, workspace=ws).cpu().numpy()
        np.testing.assert_allclose(got, want, rtol=tol, atol=1e-14 if precision == tmg.TM_FP64 else 1e-6 * want.max())


def _shifts(v, pref, axis):
    """Whole-site shifts as FP32 rounds them: round(i + v pref) - i, halves away from 0."""
    L = v.shape[0]
    i = np.arange(L, dtype=np.float32)
    i = i[:, None] if axis == 0 else i[None, :]
    t = i + v.astype(np.float32) * np.float32(pref)
    return (np.trunc(t + np.copysign(np.float32(0.5), t)).astype(np.float64) - i).astype(np.float64)
