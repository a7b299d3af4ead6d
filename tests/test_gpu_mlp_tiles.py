"""The network's kernels at the edges of their tiles, against the numpy oracle
of the same BF16 rounding points: forward passes of part-filled warps and of
arrays that are not aligned for wide accesses, gradients of batches that are
not a multiple of a block's 64 samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(kgpu, n, offset=0):
    import torch
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 16)).astype(np.float32)
    buf = torch.zeros(n * 16 + 4, dtype=torch.float32, device="cuda")
    x = buf[offset:offset + n * 16].view(n, 16)
    x.copy_(torch.from_numpy(X))
    return kgpu.Mlp(seed=3), X, x


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 15, 17, 255, 40003])
def test_forward_tiles(kgpu, n, offset):
    from oracle import mlp_oracle
    mlp, X, x = make(kgpu, n, offset)
    y = mlp.forward(x).cpu().numpy()
    e = mlp_oracle.predict(mlp.get(), X)
    # a last-place difference of a sum can move an activation by one BF16 ulp
    # (2^-8); 128 of them average out in the outputs
    assert np.abs(y - e).max() <= 2e-2 * np.abs(e).max() and np.abs(y - e).mean() <= 1e-3 * np.abs(e).max()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 63, 65, 1000])
def test_gradient_tiles(kgpu, n, offset):
    import torch
    from oracle import mlp_oracle
    mlp, X, x = make(kgpu, n, offset)
    T = np.random.default_rng(n + 1).normal(size=(n, kgpu.MLP_OUT)).astype(np.float32)
    g, loss = mlp.gradient(x, torch.from_numpy(T).cuda())
    el, eg = mlp_oracle.gradient(mlp.get(), X, T)
    # as the existing gradient test: BF16 roundings of activations and errors
    assert abs(loss - el) <= 1e-3 * el
    assert np.linalg.norm(g - eg) <= 2e-2 * np.linalg.norm(eg)
