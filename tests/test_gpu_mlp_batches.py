"""Gradients of the training step at the edges of its launches - the smallest batch,
one with a CTA per tile, one past the SM count (a CTA's second tile and two tiles in
flight in the forward pass) - and after an update (the transposed weight copy),
against the oracle with the tolerances of test_gpu_mlp.py."""
import numpy as np
import pytest

from test_gpu_mlp import ctx, make_mlp  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [256, 2048, 256 * 81])
def test_mlp_gradients_by_batch(ctx, M):  # noqa: F811
    import torch
    import mlp_oracle as mo
    net = make_mlp(ctx, max_batch=M, seed=5)
    rng = np.random.default_rng(M)
    X = rng.standard_normal((M, 12)).astype(np.float32)
    T = rng.standard_normal((M, 10)).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    net.train_step(Xd, Td, lr=1e-3)  # non-zero biases
    W, b = net.get_params()
    loss, gW, gb = net.train_step(Xd, Td, lr=0.0, update=False, grads=True)
    wl, wW, wb = mo.train_grads(W, b, X, T)
    assert loss == pytest.approx(wl, rel=1e-4)
    for l in range(5):
        sl = slice(mo.WOFF[l], mo.WOFF[l] + mo.LN[l] * mo.LK[l])
        assert np.linalg.norm(gW[sl] - wW[sl]) < 5e-3 * np.linalg.norm(wW[sl]), l
        sb = slice(mo.BOFF[l], mo.BOFF[l] + mo.LN[l])
        assert np.linalg.norm(gb[sb] - wb[sb]) < 5e-3 * np.linalg.norm(wb[sb]), l


def test_training_memory_per_row(ctx):  # noqa: F811
    """Inputs 32, outputs and their gradients 64 each, pre-activations 2048 (their
    gradients in place), activations 1024, weight and bias partials 1681 bytes a row."""
    import torch
    M = 1 << 17
    make_mlp(ctx, max_batch=256, seed=1).close()  # the kernels' code
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    net = make_mlp(ctx, max_batch=M, seed=1)
    used = free - torch.cuda.mem_get_info()[0]
    net.close()
    assert used <= 4913 * M + (48 << 20)  # allocations in 2 MB pages, the parameters
