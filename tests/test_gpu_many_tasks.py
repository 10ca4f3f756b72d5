"""Batches with several times more tiles or tasks than the GPU runs at once, so that every
block goes round its loop: tile copies started ahead and rotating buffers, tiles that come
by copies next to tiles that load by thread, both FP64 tile heights, and lists of carried
sites and prefetched tasks that pass from lattice to lattice.  Bit for bit against the
oracle.
"""
import numpy as np
import pytest

SMS = 152
FP32_BLOCKS, FP64_BLOCKS = 2 * SMS, SMS               # resident tile blocks


def _tiles(Ls, rows):
    return sum(-(-L // 64) * -(-L // rows) for L in Ls)


def _fp64_rows(Ls):
    """Tile rows an FP64 batch takes: the busiest SM's warps of cells over the four stages."""
    def cost(ty):
        warps = 0
        for s in range(4):
            ring = (72 - 2 * (s + 1)) * (ty + 8 - 2 * (s + 1)) - 64 * ty
            warps += 64 * ty // 32 + (ring + 31) // 32
        return -(-_tiles(Ls, ty) // SMS) * warps
    return 24 if cost(24) <= cost(12) else 12


def _order(Ls, seed):
    return [Ls[i] for i in np.random.default_rng(seed).permutation(len(Ls))]


# 76, 72, 128 and 200 come by copies in FP32 (whole 16-byte rows, a region wide), 70 and 133 by thread;
# FP64 copies interior tiles of even sides
RAGGED = _order([76, 70, 133, 128, 72, 200] * 11, 1)
TALL = [96] * 80                                        # 8 tiles of 24 rows
LOW = _order([84, 133, 60] * 18, 2)                      # wasted rows and a last wave that favour 12


def test_the_batches_are_what_they_are_meant_to_be():
    assert _tiles(RAGGED, 32) > 2 * FP32_BLOCKS
    for Ls, rows in ((TALL, 24), (LOW, 12)):
        assert _fp64_rows(Ls) == rows and _tiles(Ls, rows) > 2 * FP64_BLOCKS


def _frames(Ls, dtype, seed):
    rng = np.random.default_rng(seed)
    f = []
    for k, L in enumerate(Ls):
        x = np.stack([rng.uniform(0, 4, (L, L)), rng.uniform(0.1, 6, (L, L)), rng.uniform(0.5, 9, (L, L))]).astype(dtype)
        if k % 3 == 1:
            x[0][: L // 2] = 0.0                         # bare ground
        f.append(x)
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("det", [0, 1], ids=["noise", "off"])
@pytest.mark.parametrize("precision,Ls", [(1, RAGGED), (0, TALL), (0, LOW)], ids=["fp32", "fp64-24rows", "fp64-12rows"])
def test_tiles_beyond_one_wave_match_oracle(oracle, precision, Ls, det):
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    m = tmg.rietkerk_model(deterministic=det)
    init = _frames(Ls, np.float64 if precision == 0 else np.float32, 7)
    Rs = [0.8 + 0.01 * (k % 40) for k in range(len(Ls))]
    b = tmg.Batch(ctx, m, tmg.instances(Ls, [100 + k for k in range(len(Ls))], Rs), precision)
    b.upload(init)
    _, st = b.advance(2, [])
    fin = b.download()
    b.close()
    ctx.close()
    assert not st.any()
    for k, L in enumerate(Ls):
        p = oracle.rk_params(R=Rs[k], sampler=m.sampler)
        if det:
            want = init[k]
            for _ in range(2):
                want = oracle.rk_det_step(p, want)
                want[(want < want.dtype.type(m.clamp_eps)) & (want >= want.dtype.type(m.clamp_lo))] = 0.0
        else:
            _, _, want, _ = oracle.rk_run(p, init[k], 100 + k, 2, [])
        assert np.array_equal(fin[k], want), (k, L)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("sampler,dt", [(0, 0.1), (0, 0.05), (1, 0.012)], ids=["m17", "m37", "m165"])
def test_tasks_beyond_one_wave_match_oracle(oracle, precision, sampler, dt):
    """One-row tasks, seven for each warp in FP64 and half as many in FP32; dense, dilute,
    single-site and empty lattices in turn, so that a warp's lists mix them all."""
    import trophic_maelstorm_gb300 as tmg
    ctx = tmg.Context(0)
    dtype = np.float64 if precision == 0 else np.float32
    Ls = _order([130] * 16 + [65] * 30 + [33] * 20, 3)
    assert sum(L * -(-L // 32) for L in Ls) > 7 * 2 * 8 * SMS
    rng = np.random.default_rng(11)
    init = []
    for k, L in enumerate(Ls):
        f = rng.uniform(0.0, 2.0, (L, L)) ** (1 + k % 2)
        if k % 4 == 1:
            f *= 0.02 * (rng.random((L, L)) < 0.3)        # fronts, shapes below 1
        elif k % 4 == 2:
            f *= 0.0
            f[rng.integers(L), rng.integers(L)] = 1.0
        elif k % 8 == 7:
            f *= 0.0
        init.append(f.astype(dtype))
    model = tmg.dp_model(dt=dt, sampler=sampler)
    seeds = [40 + k for k in range(len(Ls))]
    b = tmg.Batch(ctx, model, tmg.instances(Ls, seeds, 0.53), precision)
    b.set_launch(1, 0)
    b.upload(init)
    _, st = b.advance(3, [])
    fin = b.download()
    b.close()
    ctx.close()
    for k, L in enumerate(Ls):
        p = oracle.DPParams(0.53, 0.0, model.b, model.c, model.D, model.sigma, model.dt, model.dx, model.clamp_lo,
                            model.clamp_eps, model.remainder, model.sampler)
        _, _, want, ost = oracle.dp_run(p, init[k], seeds[k], 3, [3])
        assert np.array_equal(fin[k], want), (k, L)
        assert st[k] == ost
