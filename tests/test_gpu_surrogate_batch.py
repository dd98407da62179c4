"""The surrogate's bias gradients (column sums in slices of the batch, the last block adding them) at batch
sizes below, at and across a slice's 256 staged rows, against torch autograd of the same network, its operands
rounded to BF16 like the device's.  The device also rounds the backward operands (relative 2^-9 each, a
few per layer): 2e-2 in the relative 2-norm, the bound of the 512-row gradients."""
import numpy as np
import pytest
import torch

from test_gpu_surrogate import bf16, lattice, pack, seeded_params, unpack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 576, 2112, 4160])
def test_bias_gradients(n):
    d = seeded_params(3)
    rng = np.random.default_rng(n)
    x = (rng.normal(size=(n, 12)) * d["x_std"] + d["x_mean"]).astype(np.float32)
    y = (rng.normal(size=(n, 10)) * d["y_std"] + d["y_mean"]).astype(np.float32)
    lat, *_ = lattice()
    with lat:
        lat.surrogate_params(pack(d))
        lat.surrogate_load_samples(x, y)
        lat.surrogate_train(epochs=1, batch=n, lr=1e-6, seed=1, refit=False)
        got = unpack(lat.surrogate_grads())
    P = {k: torch.tensor(d[k], requires_grad=k[0] in "Wb") for k in d}
    h = (torch.tensor(x) - P["x_mean"]) / P["x_std"]
    h = bf16(h) + bf16(h - bf16(h))
    for L in (1, 2, 3):
        h = bf16(torch.nn.functional.gelu(h @ bf16(P[f"W{L}"]).T + P[f"b{L}"], approximate="tanh"))
    out = h @ bf16(P["W4"]).T + P["b4"]
    ((out - (torch.tensor(y) - P["y_mean"]) / P["y_std"]) ** 2).mean().backward()
    for k in ("b1", "b2", "b3", "b4"):
        g = P[k].grad.numpy()
        assert np.linalg.norm(got[k] - g) < 2e-2 * np.linalg.norm(g), k
