"""A captured box call keeps its scratch while the 0D cells' calls of the same context
grow theirs: the replay on new inputs gives what a call on them gives."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu


def test_captured_box_call_beside_cell_calls(oracle):
    import torch
    import ocfd
    from ocfd import mlp, surrogate
    from ocfd.react import state_tpx
    ctx, other = ocfd.Context(), ocfd.Context()
    n, dxinv = (9, 8, 7), [1.0e4, 1.1e4, 0.9e4]
    S, sp, S2, sp2 = [torch.from_numpy(x).cuda() for seed in (4, 5)
                      for x in inputs.chem_state(*n, seed=seed, oracle=oracle)]

    def rhs(c, out):
        c.rhs_chem_box(S, sp, out[0], out[1], (0, 0, 0), tuple(m - 1 for m in n), dxinv, 1)

    def outputs():
        return [torch.full((k,) + n[::-1], float("nan"), dtype=torch.float64, device="cuda") for k in (5, 9)]
    got, want = outputs(), outputs()
    rhs(ctx, got)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        rhs(ctx, got)
    net = mlp.Mlp(ctx, 256, 1)
    guard = surrogate.Guard(200.0, 5000.0, 1.0, 1e9, 0.0, 1.0, 1.0, 1e-3, 0.0, 0.0)
    cells = 1 << 20
    U = torch.as_tensor(state_tpx(ctx, *surrogate.mixtures(np.random.default_rng(1), cells)), device="cuda").contiguous()
    surrogate.cells_surrogate(ctx, net, guard, U, 1e-8)
    S.copy_(S2)
    sp.copy_(sp2)
    keep = [torch.zeros(1 << 20, dtype=torch.float64, device="cuda") for _ in range(8)]  # takes what was freed
    g.replay()
    torch.cuda.synchronize()
    assert all(not k.any() for k in keep)
    rhs(other, want)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
