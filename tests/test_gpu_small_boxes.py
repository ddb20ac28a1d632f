"""Per-box right-hand sides of boxes that take the small tile shapes (8x4x4, 4x4x4,
4x4x2, 8x2x2), with remainders in every direction: bit for bit the values of the same
cells and faces in a call on the whole box, which takes 8^3 tiles."""
import pytest

import inputs

pytestmark = pytest.mark.gpu
N = (48, 40, 40)


@pytest.fixture(scope="module")
def whole():
    import torch
    import ocfd
    return ocfd.Context(), torch.from_numpy(inputs.ideal_state(*N, seed=12)).cuda()


def rhs(ctx, S, lo, hi, flags):
    import torch
    n = [h - l + 1 for l, h in zip(lo, hi)]
    dS = torch.full((5, n[2], n[1], n[0]), float("nan"), dtype=torch.float64, device="cuda")
    fl = [torch.full((5, n[2] + (d == 2), n[1] + (d == 1), n[0] + (d == 0)), float("nan"), dtype=torch.float64,
                     device="cuda") for d in range(3)]
    ctx.rhs_regular_box(S, dS, lo, hi, [48.0, 40.0, 44.0], flags, flux=fl, S_begin=(-4, -4, -4))
    torch.cuda.synchronize()
    return [dS] + fl


@pytest.mark.parametrize("n", [(1, 1, 1), (4, 4, 2), (5, 3, 7), (9, 17, 2), (20, 12, 8), (31, 5, 18), (30, 31, 5)])
@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("fp32", [0, 4])
def test_small_box_equals_whole(whole, n, visc, fp32):
    import torch
    ctx, S = whole
    full = rhs(ctx, S, (0, 0, 0), tuple(m - 1 for m in N), visc | fp32)
    lo = (3, 6, 9)
    got = rhs(ctx, S, lo, tuple(l + m - 1 for l, m in zip(lo, n)), visc | fp32)
    for k, (a, b) in enumerate(zip(got, full)):
        idx = tuple(slice(lo[d], lo[d] + n[d] + (k == d + 1)) for d in (2, 1, 0))
        assert torch.equal(a, b[(slice(None),) + idx]), k
