"""The plan and buffers that a batch keeps for its next power spectrum can be given back."""
import numpy as np
import pytest


def test_release_rejects_null():
    from trophic_maelstorm_gb300 import _lib
    assert _lib.lib().tm_batch_release_work(None) == _lib.TM_ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_release_gives_the_memory_back(precision):
    torch = pytest.importorskip("torch")
    import trophic_maelstorm_gb300 as tmg
    L = 2048
    rng = np.random.default_rng(1)
    ctx = tmg.Context(0)
    b = tmg.Batch(ctx, tmg.dp_model(), tmg.instances([L, 32], [1, 2], 0.5), precision)
    b.upload([rng.uniform(0.0, 2.0, (n, n)) for n in (L, 32)])
    b.release_work()                                   # nothing kept yet
    first = b.power_spectrum(0)
    b.release_work()                                   # the transform's code stays loaded
    free = torch.cuda.mem_get_info(0)[0]
    again = b.power_spectrum(0)
    held = free - torch.cuda.mem_get_info(0)[0]
    assert held >= 16 * L * L                          # image and half spectrum, 8 bytes a site each
    b.release_work()
    assert free - torch.cuda.mem_get_info(0)[0] <= held // 16
    b.release_work()
    small = b.power_spectrum(1)
    third = b.power_spectrum(0)
    assert len(small[0]) < len(third[0])
    for k, p in (again, third):
        assert np.array_equal(k, first[0]) and np.array_equal(p, first[1])
    b.close()
    ctx.close()
