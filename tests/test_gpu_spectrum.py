"""Annuli of the power spectrum summed straight from the transform, at sides and bin widths
where their limits fall on lattice modes, and the plan a batch keeps between calls.
Against numpy's FFT and histogram; the sums agree to rounding (1e-9 of the peak power, as
the fixture test).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy(f, bw):
    L = f.shape[0]
    m = f.max()
    p = np.abs(np.fft.fft2(f / (m if m != 0 else 1.0))) ** 2
    fr = np.fft.fftfreq(L) * L
    k = np.sqrt(fr[:, None] ** 2 + fr[None, :] ** 2).reshape(-1)
    start = 1 - bw / 2                                          # edges e_b = 1 - w/2 + b w (np.arange rounds them otherwise)
    e = start + bw * np.arange(int(np.ceil((L // 2 + 1 - start) / bw)))
    s, _ = np.histogram(k, e, weights=p.reshape(-1))
    n, _ = np.histogram(k, e)
    return 0.5 * (e[1:] + e[:-1]), np.where(n > 0, s / np.maximum(n, 1), 0.0) * np.pi * (e[1:] ** 2 - e[:-1] ** 2)


@pytest.mark.parametrize("bw", [0.3, 0.5, 1.0, 2.0])
def test_annuli_match_numpy(bw):
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    Ls = [4, 5, 8, 33, 64, 101, 130]
    rng = np.random.default_rng(3)
    fields = [rng.uniform(0, 2, (L, L)) for L in Ls]
    b = tmg.Batch(ctx, tmg.dp_model(), tmg.instances(Ls, list(range(len(Ls))), 0.5), tmg.TM_FP64)
    b.upload(fields)
    first = {}
    for k in list(range(len(Ls))) + [2, 2, 5]:                  # kept plan reused, replaced, reused
        kv, pw = b.power_spectrum(k, 0, bw)
        want_k, want = _numpy(fields[k], bw)
        assert np.array_equal(kv, want_k)
        np.testing.assert_allclose(pw, want, rtol=1e-9, atol=1e-9 * want.max())
        assert np.array_equal(first.setdefault(k, pw), pw)       # the same bits on every call
    b.close()
    ctx.close()
