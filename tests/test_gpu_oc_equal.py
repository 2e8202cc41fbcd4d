"""stg_oc_update_noalloc returns stg_oc_update's design and multiplier bit for bit, as the header
promises, in every form of the update: one cluster (8^3 to 24^3), cells in registers (32^3,
64^3) and cells read for each probe (96^3), with the smallest and the largest filter. One
volume that differs in its last bit can turn a bisection step round, and the designs then differ by
1e-9, so nothing less than equal sums will do.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [8, 16, 24, 32, 64, 96])
@pytest.mark.parametrize("rmin", [1.0, 1.5, 4.0])
def test_both_updates_are_the_same_bits(stg, n, rmin):
    rng = np.random.default_rng(n)
    s = stg.Solver(n)
    for frac, scale in ((0.2, 1.0), (0.4, 1e14), (0.7, 1e-6)):
        x = 0.05 + 0.9 * rng.random((n, n, n))
        dc = -scale * rng.random((n, n, n))
        dc[rng.random(dc.shape) < 0.1] *= -1.0
        ref, lam_ref = s.oc_update(rmin, x, dc, frac)
        dx, ddc = torch.from_numpy(x).cuda(), torch.from_numpy(dc).cuda()
        out, lam = torch.full_like(dx, -1.0), ctypes.c_double()
        stg.check(stg.lib().stg_oc_update_noalloc(n, rmin, dx.data_ptr(), ddc.data_ptr(), frac, 0.2, 0.0, 1.0, out.data_ptr(),
                                                  ctypes.byref(lam), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert lam.value == lam_ref
        assert np.array_equal(out.cpu().numpy(), ref)
    s.close()
