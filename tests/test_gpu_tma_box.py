"""TMA-staged tiles of one box on arrays that allow the staging and on arrays that do not
- an odd x offset, odd strides, a base off the 16-byte boundary: refused there, and the
same divergence and face fluxes, bit for bit, as the per-box call's own tile."""
import ctypes

import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [1, 6, 7, 8])
@pytest.mark.parametrize("nx,grow,skew,allowed", [(24, 4, 0, True), (22, 4, 0, True), (24, 3, 0, False), (23, 4, 0, False),
                                                  (24, 4, 1, False)])
def test_staged_box(tile, nx, grow, skew, allowed):
    import torch
    import ocfd
    from ocfd._abi import Array4, Box, array4, box, declare
    from ocfd.context import _stream_ptr
    AP = ctypes.POINTER(Array4)
    declare("ocfd_check_rhs_f32_tile", ctypes.c_int,
            [ctypes.c_void_p, AP, AP, AP, Box, ctypes.POINTER(ctypes.c_double), ctypes.c_int32,
             ctypes.POINTER(ctypes.c_int32), ctypes.c_void_p])
    ctx, n, cut = ocfd.Context(), (nx, 16, 12), 4 - grow
    S = inputs.ideal_state(*n, seed=5, jump=True, mach=0.8)
    S = np.ascontiguousarray(S[(slice(None),) + 3 * (slice(cut, -cut or None),)])
    buf = torch.zeros(S.size + 1, dtype=torch.float64, device="cuda")
    St = buf[skew:skew + S.size].view(S.shape)
    St.copy_(torch.from_numpy(S))
    hi, dxinv, begin = tuple(m - 1 for m in n), [24.0, 24.0, 24.0], (-grow,) * 3

    def outputs():
        return [torch.full((5,) + tuple(n[d] + (d == k) for d in (2, 1, 0)), float("nan"), dtype=torch.float64,
                           device="cuda") for k in (-1, 0, 1, 2)]
    want, got = outputs(), outputs()
    ctx.rhs_regular_box(St, want[0], (0, 0, 0), hi, dxinv, ocfd.FLUX_FP32, flux=want[1:], S_begin=begin)
    staged = ctypes.c_int32(-1)
    a = [array4(St, begin)] + [array4(t) for t in got]
    ocfd.check(ocfd.load().ocfd_check_rhs_f32_tile(ctx.h, a[0], a[1], (Array4 * 3)(*a[2:]), box((0, 0, 0), hi),
                                                   (ctypes.c_double * 3)(*dxinv), tile, ctypes.byref(staged),
                                                   _stream_ptr(None)))
    torch.cuda.synchronize()
    assert staged.value == int(allowed and tile >= 6)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
