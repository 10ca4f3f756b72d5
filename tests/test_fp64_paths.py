"""The FP64 arithmetic and draw paths that GB300's slow FP64 pipe made worth writing.

Host: the integer multiply, divide and square root (tm_f64.cuh, which compiles
for the host too) against the host's IEEE operations, bit for bit, and the bound
under which the FP32 Poisson search decides for the FP64 one.  GPU: FP64 fields
against the oracle, bit for bit, at states that reach every carried list of the
step (dilute fronts, shapes below 1, Poisson means around 32 and 100).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WRAP = r"""
#include "%s"
#define EACH(NAME, EXPR) extern "C" void NAME(const double* a, const double* b, double* o, long n) \
    { for (long i = 0; i < n; ++i) o[i] = EXPR; }
EACH(w_mul, tmf::mul(a[i], b[i]))
EACH(w_div, tmf::div(a[i], b[i]))
EACH(w_sqrt, tmf::sqrt(a[i]))
EACH(w_trunc, (double)tmf::trunc_f32(a[i]))
extern "C" void w_unit(const unsigned long long* x, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = tmf::open_unit(x[i]); }
extern "C" void w_int(const unsigned* x, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = tmf::from_u31(x[i]); }
"""


@pytest.fixture(scope="module")
def f64(tmp_path_factory):
    d = tmp_path_factory.mktemp("f64")
    hdr = os.path.join(REPO, "trophic_maelstorm_gb300", "csrc", "tm_f64.cuh")
    (d / "w.cpp").write_text(WRAP % hdr)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", str(d / "w.so"),
                    str(d / "w.cpp")], check=True)
    return ctypes.CDLL(str(d / "w.so"))


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _bits(a):
    return np.where(np.isnan(a), np.uint64(0x7ff8000000000000), a.view(np.uint64))


def _operands(n, spread, seed):
    """Random signs, exponents of the given spread (None: the whole range) and mantissas with long runs of ones and zeros."""
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = rng.integers(0, 52, n).astype(np.uint64)
    run = (np.uint64(1) << k) - np.uint64(1)
    kind = rng.integers(0, 5, n)
    full = np.uint64((1 << 52) - 1)
    m = np.select([kind == 0, kind == 1, kind == 2], [m | run, m & ~run, full - (m & np.uint64(3))], m)
    e = rng.integers(0, 2048, n) if spread is None else 1023 + rng.integers(-spread, spread + 1, n)
    u = (rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)) | (e.astype(np.uint64) << np.uint64(52)) | m
    return u.view(np.float64)


@pytest.mark.parametrize("spread", [0, 3, 60, 520, None])
def test_integer_arithmetic_is_ieee(f64, spread):
    n = 400_000
    a, b = _operands(n, spread, 1), _operands(n, spread, 2)
    edge = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072014e-308,
                     1.7976931348623157e308, 1.0 - 2.0 ** -53, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52])
    a = np.concatenate([np.repeat(edge, len(edge)), a])
    b = np.concatenate([np.tile(edge, len(edge)), b])
    o = np.empty_like(a)
    with np.errstate(all="ignore"):
        f64.w_mul(_p(a), _p(b), _p(o), ctypes.c_long(a.size))
        assert np.array_equal(_bits(o), _bits(a * b))
        f64.w_div(_p(a), _p(b), _p(o), ctypes.c_long(a.size))
        assert np.array_equal(_bits(o), _bits(a / b))
        f64.w_sqrt(_p(a), _p(b), _p(o), ctypes.c_long(a.size))
        assert np.array_equal(_bits(o), _bits(np.sqrt(a)))


def test_conversions(f64):
    rng = np.random.default_rng(3)
    x = rng.integers(0, 1 << 53, 200_000, dtype=np.uint64) >> rng.integers(0, 53, 200_000).astype(np.uint64)
    x = np.concatenate([np.arange(64, dtype=np.uint64), np.uint64((1 << 53) - 1) - np.arange(64, dtype=np.uint64),
                        np.uint64(1 << 52) + np.arange(64, dtype=np.uint64), x])
    o = np.empty(x.size)
    f64.w_unit(_p(x), _p(o), ctypes.c_long(x.size))
    assert np.array_equal(o, (x.astype(np.float64) + 0.5) * 2.0 ** -53)
    n = (x & np.uint64(0x7fffffff)).astype(np.uint32)
    f64.w_int(_p(n), _p(o), ctypes.c_long(n.size))
    assert np.array_equal(o, n.astype(np.float64))
    v = np.abs(_operands(100_000, 100, 4))
    o = np.empty_like(v)
    f64.w_trunc(_p(v), _p(v), _p(o), ctypes.c_long(v.size))
    assert np.all(o <= v) and np.all(o >= v * (1 - 2.0 ** -23))


def test_poisson_search_bound():
    """FP32 tails of the search stay within (m + 4) 2^-22 of the FP64 tails (the derivation allows (m + 2) 2^-22)."""
    rng = np.random.default_rng(5)
    m = np.concatenate([rng.uniform(0, 32, 40_000), 32 * 10.0 ** -rng.uniform(0, 9, 20_000), rng.uniform(28, 32, 20_000)])
    m = m[m < 32]
    mf = (m.view(np.uint64) & ~np.uint64((1 << 29) - 1)).view(np.float64).astype(np.float32)   # truncated, as the kernel does
    bound = (mf + np.float32(4)) * np.float32(2.0 ** -22)
    p, q = np.exp(-m), -np.expm1(-m)
    pf = np.exp(-mf.astype(np.float64)).astype(np.float32)
    # the kernel's e^-m and 1 - e^-m carry a few roundings more than the nearest value
    qf = (-np.expm1(-mf.astype(np.float64))).astype(np.float32)
    for i in range(1, 97):
        p = p * m / i
        q = q - p
        pf = (pf * mf) * np.float32(1.0 / i)
        qf = qf - pf
        assert np.all(np.abs(q - qf) < bound * (1 - 0.1))


@pytest.mark.gpu
@pytest.mark.parametrize("sampler,remainder", [(0, 0), (1, 1)])
@pytest.mark.parametrize("dt,scale", [(0.1, 1.0), (0.1, 0.02), (0.05, 1.0), (0.012, 1.0)],
                         ids=["m17", "dilute", "m37", "m165"])
def test_fp64_draw_paths_match_oracle(oracle, dt, scale, sampler, remainder):
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    rng = np.random.default_rng(7)
    Ls = [1, 2, 31, 33, 65, 130]
    model = tmg.dp_model(dt=dt, sampler=sampler, remainder=remainder, clamp_lo=-1e-80 if remainder else 0.0,
                         clamp_eps=1e-12 if remainder else 0.0)
    inst = tmg.instances(Ls, [5 + k for k in range(len(Ls))], 0.53)
    init = []
    for L in Ls:
        f = scale * rng.uniform(0.0, 2.0, (L, L))
        f[rng.random((L, L)) < (0.0 if scale == 1.0 else 0.7)] = 0.0      # dilute: fronts, empty rows
        f[L // 2:, :] *= rng.random() < 0.5 or L < 30
        init.append(f)
    b = tmg.Batch(ctx, model, inst, tmg.TM_FP64)
    b.upload(init)
    _, st = b.advance(7, [])
    fin = b.download()
    b.close()
    ctx.close()
    for k, L in enumerate(Ls):
        p = oracle.DPParams(0.53, 0.0, model.b, model.c, model.D, model.sigma, model.dt, model.dx, model.clamp_lo,
                            model.clamp_eps, model.remainder, model.sampler)
        _, _, want, ost = oracle.dp_run(p, init[k], 5 + k, 7, [7])
        assert np.array_equal(fin[k], want), (k, L)
        assert st[k] == ost


@pytest.mark.gpu
@pytest.mark.parametrize("sampler", [0, 1])
@pytest.mark.parametrize("dt", [0.02, 0.004, 0.0007], ids=["m100", "m500", "m2900"])
def test_fp64_transformed_rejection_matches_oracle(oracle, dt, sampler):
    """Poisson means through 32, 100 and 4096 (where the FP32 decisions end), bit for bit."""
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    rng = np.random.default_rng(11)
    Ls = [33, 130]
    model = tmg.dp_model(dt=dt, sampler=sampler)
    b = tmg.Batch(ctx, model, tmg.instances(Ls, [3, 4], 0.53), tmg.TM_FP64)
    init = [rng.uniform(0.0, 3.0, (L, L)) ** 2 for L in Ls]
    b.upload(init)
    _, st = b.advance(5, [])
    fin = b.download()
    b.close()
    ctx.close()
    for k, L in enumerate(Ls):
        p = oracle.DPParams(0.53, 0.0, model.b, model.c, model.D, model.sigma, model.dt, model.dx, model.clamp_lo,
                            model.clamp_eps, model.remainder, model.sampler)
        _, _, want, ost = oracle.dp_run(p, init[k], 3 + k, 5, [5])
        assert np.array_equal(fin[k], want), (k, L)
        assert st[k] == ost
