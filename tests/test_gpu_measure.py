"""Sums of a measurement: tasks reported in stretches, groups of them summed by the warps
that finish last, and one kernel for both (tm_measure.cu).

Bound: the values are non-negative and every sum is a tree of at most 2^-53 a level over
less than 64 levels and 2^-48 for the FP32 pairs, so a mean lies within 1e-12 of the
exact one; counts and squared distances are whole and exact.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("Ls", [[1], [128], [129, 1, 300, 31, 700], [2300, 64]],
                         ids=["one-task", "512-tasks", "mixed", "groups-of-512"])
def test_measurement_sums(Ls, precision, rows):
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(3)
    ctx = tmg.Context(0)
    prec, dtype = (tmg.TM_FP32, np.float32) if precision == "fp32" else (tmg.TM_FP64, np.float64)
    fields = []
    for L in Ls:
        f = rng.uniform(0.0, 3.0, (L, L)) * (rng.random((L, L)) < 0.6)
        f[L // 3:L // 2] = 0.0                                # whole rows of zeros
        fields.append(f.astype(dtype))
    model = tmg.dp_model(dt=0.1)
    b = tmg.Batch(ctx, model, tmg.instances(Ls, [1 + k for k in range(len(Ls))], 0.5), prec)
    b.set_launch(rows, 0)
    b.upload(fields)
    for step in (1, 2):                                       # the counters are left as they were found
        obs, _ = b.advance(1, [step])
        out = b.download()
        for k, L in enumerate(Ls):
            v = np.asarray(out[k], np.float64).reshape(L, L)
            want = math.fsum(v.ravel()) / (L * L)
            assert abs(obs[0, k, 0] - want) <= 1e-12 * max(abs(want), 1e-300), (k, L)
            assert obs[0, k, 1] == np.count_nonzero(v > 0)
    b.close()
    rk = tmg.rietkerk_model()
    fields3 = [rng.uniform(0.0, 3.0, (3, L, L)).astype(dtype) for L in Ls]
    b = tmg.Batch(ctx, rk, tmg.instances(Ls, [1 + k for k in range(len(Ls))], 1.0), prec)
    b.set_launch(rows, 0)
    b.upload(fields3)
    for step in (1, 2):
        obs, _ = b.advance(1, [step])
        out = b.download()
        for k, L in enumerate(Ls):
            v = np.asarray(out[k], np.float64).reshape(3, L * L)
            for f in range(3):
                want = math.fsum(v[f]) / (L * L)
                assert abs(obs[0, k, f] - want) <= 1e-12 * max(abs(want), 1e-300), (k, L, f)
            assert obs[0, k, 3] == np.count_nonzero(v[0] > 0)
    b.close()
    ctx.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("rows", [1, 8])
def test_spreading_sums(precision, rows):
    """Squared distances of a cluster away from the edge, from a lattice of many groups."""
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(4)
    ctx = tmg.Context(0)
    prec, dtype = (tmg.TM_FP32, np.float32) if precision == "fp32" else (tmg.TM_FP64, np.float64)
    Ls = [40, 600]
    fields = []
    for L in Ls:
        f = np.zeros((L, L), dtype)
        f[10:L - 10, 12:L - 9] = (rng.uniform(0.5, 3.0, (L - 20, L - 21)) * (rng.random((L - 20, L - 21)) < 0.5)).astype(dtype)
        fields.append(f)
    b = tmg.Batch(ctx, tmg.dp_model(dt=0.1), tmg.instances(Ls, [3, 4], 0.5), prec)
    b.set_launch(rows, 0)
    b.set_spreading(True, 5, 7)
    b.upload(fields)
    for step in (1, 2):
        obs, _ = b.advance(1, [step])
        out = b.download()
        for k, L in enumerate(Ls):
            v = np.asarray(out[k], np.float64).reshape(L, L)
            want = math.fsum(v.ravel()) / (L * L)
            y, x = np.nonzero(v > 0)
            assert abs(obs[0, k, 0] - want) <= 1e-12 * want
            assert obs[0, k, 1] == y.size
            # centre (cx, cy) as the batch takes it, row against cy and column against cx
            assert obs[0, k, 2] == int(((y - 7) ** 2 + (x - 5) ** 2).sum())
    b.close()
    ctx.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_ramp_across_measurements_matches_oracle(oracle, precision):
    """A ramp's constants are queued for runs of steps that measurements, graphs and calls cut differently."""
    import trophic_maelstorm_gb300 as tmg
    rng = np.random.default_rng(9)
    ctx = tmg.Context(0)
    prec, dtype = (tmg.TM_FP32, np.float32) if precision == "fp32" else (tmg.TM_FP64, np.float64)
    L, a, a_step, n = 33, 0.72, -3e-4, 150
    model = tmg.dp_model(dt=0.1)
    init = rng.uniform(0.5, 1.5, (L, L)).astype(dtype)
    p = oracle.DPParams(a, a_step, model.b, model.c, model.D, model.sigma, model.dt, model.dx, model.clamp_lo, model.clamp_eps,
                        model.remainder, model.sampler)
    meas = [1, 2, 3, 20, 31, 32, 33, 66, 100, 101, 140, 150]
    mean, active, want, _ = oracle.dp_run(p, init, 5, n, meas)
    for calls in ([n], [1, 40, 5, 104]):
        b = tmg.Batch(ctx, model, tmg.instances([L, L], [4, 5], a, a_step), prec)
        b.upload([init, init])
        got, at = [], 0
        for steps in calls:
            now = [m for m in meas if at < m <= at + steps]
            obs, _ = b.advance(steps, now)
            got += [obs[j, 1] for j in range(len(now))]
            at += steps
        assert np.array_equal(b.download()[1], want)
        b.close()
        for j in range(len(meas)):
            assert abs(got[j][0] - mean[j]) <= 1e-12 * mean[j] and got[j][1] == active[j]
    ctx.close()
