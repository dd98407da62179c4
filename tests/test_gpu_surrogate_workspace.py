"""The training buffers that a handle keeps between calls: the same gradients, to the bit, as on a
fresh handle when the batch size and the sample set change from call to call; no more than 64 MiB kept;
given back where an allocation of the handle finds no memory."""
import numpy as np
import pytest

import lbmgpu
from test_gpu_surrogate import lattice, pack, seeded_params

pytestmark = pytest.mark.gpu

KEPT = 64 << 20


def samples(n):
    rng = np.random.default_rng(n)
    return rng.standard_normal((n, 12), dtype=np.float32), rng.standard_normal((n, 10), dtype=np.float32)


def gradients(lat, n, batch):
    lat.surrogate_params(pack(seeded_params(3)))
    lat.surrogate_load_samples(*samples(n))
    loss = lat.surrogate_train(epochs=1, batch=batch, lr=1e-4, seed=1)
    return loss, lat.surrogate_grads(), lat.surrogate_params()


def test_same_bits_over_changing_batches():
    calls = [(700, 128), (700, 320), (700, 128), (1500, 128), (900, 64), (900, 32768), (700, 128)]
    lat, *_ = lattice()
    with lat:
        kept = [gradients(lat, *c) for c in calls]
    for c, (loss, g, p) in zip(calls, kept):
        fresh, *_ = lattice()
        with fresh:
            loss2, g2, p2 = gradients(fresh, *c)
        assert loss == loss2, c
        assert np.array_equal(g, g2) and np.array_equal(p, p2), c


@pytest.mark.parametrize("batch,kept", [(256, True), (4096, True), (32768, False)])
def test_large_buffers_are_given_back(batch, kept):
    lat, *_ = lattice()
    with lat:
        lat.surrogate_load_samples(*samples(600))
        before = lat.device_bytes()
        for _ in range(2):
            lat.surrogate_train(epochs=1, batch=batch, lr=1e-4, seed=1)
            held = lat.device_bytes() - before
            assert 0 < held <= KEPT if kept else held == 0


def test_given_back_where_memory_is_short():
    lat, *_ = lattice()
    with lat:
        lat.surrogate_load_samples(*samples(600))
        before = lat.device_bytes()
        want = gradients(lat, 600, 256)
        assert lat.device_bytes() > before
        with pytest.raises(lbmgpu.LbmGpuError):
            lat.surrogate_collect(True, capacity=1 << 42)  # more than any device: the allocation is refused
        assert lat.device_bytes() == before
        got = gradients(lat, 600, 256)
    assert want[0] == got[0] and np.array_equal(want[1], got[1]) and np.array_equal(want[2], got[2])
