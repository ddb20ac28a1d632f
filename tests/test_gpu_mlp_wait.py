"""A completion wait that runs out for one thread of each CTA only: every kernel of the
network still ends, with the timeout status, and the next call works - at batches with
one tile per CTA and with two in flight, the thread in either tile's group."""
import numpy as np
import pytest

from test_gpu_mlp import ctx, make_mlp  # noqa: F401

pytestmark = pytest.mark.gpu
TIMEOUT = 3


def times_out(net, thread, call):
    import ocfd
    ocfd.check(net.lib.ocfd_check_mlp_late_thread(net.h, thread))
    with pytest.raises(ocfd.OcfdError) as e:
        call()
    assert e.value.status == TIMEOUT
    ocfd.check(net.lib.ocfd_check_mlp_late_thread(net.h, -1))


@pytest.mark.parametrize("thread", [0, 37, 300, 511])
@pytest.mark.parametrize("M", [256, 256 * 160])
def test_one_thread_runs_out(ctx, M, thread):  # noqa: F811
    import torch
    net = make_mlp(ctx, max_batch=M, seed=3)
    rng = np.random.default_rng(M)
    X = torch.from_numpy(rng.standard_normal((M, 12)).astype(np.float32)).cuda()
    T = torch.from_numpy(rng.standard_normal((M, 10)).astype(np.float32)).cuda()
    Y = net.forward(X)
    grads = net.train_step(X, T, update=False, grads=True)
    times_out(net, thread, lambda: net.forward(X))
    times_out(net, thread, lambda: net.train_step(X, T, update=False, grads=True))
    assert torch.equal(net.forward(X), Y)
    for a, b in zip(net.train_step(X, T, update=False, grads=True), grads):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,thread", [(100, 5), (128 * 400, 290)])
def test_surrogate_substep_runs_out(ctx, n, thread):  # noqa: F811
    import torch
    from ocfd import surrogate
    from ocfd.react import state_tpx
    net = make_mlp(ctx)
    guard = surrogate.Guard(200.0, 5000.0, 1.0, 1e9, 0.0, 1.0, 1.0, 1e-3, 0.0, 0.0)
    U = torch.as_tensor(state_tpx(ctx, *surrogate.mixtures(np.random.default_rng(1), n)), device="cuda").contiguous()
    want, got = U.clone(), U.clone()
    fb = surrogate.cells_surrogate(ctx, net, guard, want, 1e-8)
    times_out(net, thread, lambda: surrogate.cells_surrogate(ctx, net, guard, U.clone(), 1e-8))
    assert surrogate.cells_surrogate(ctx, net, guard, got, 1e-8) == fb
    assert torch.equal(got, want)
