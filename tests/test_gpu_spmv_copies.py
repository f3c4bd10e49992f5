"""cfd_spmv takes the stored copy of the present system: a copy of the asked
precision if the system has one, else the FP64 copy, else the low-precision copy
that is the only one; never what an earlier system left behind.

Tolerance: the product and the value it is compared with each add at most 15 * 5
entries in FP64, 2 * 75 * 1.1e-16 of the sum of their magnitudes, 2e-14; another
copy differs by 2^-25 and more of its entries."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params, perturbed_freestream

pytestmark = pytest.mark.gpu

FP64, FP32, BF16, LOW = capi.PREC_FP64, capi.PREC_FP32, capi.PREC_BF16, capi.PREC_LOW_ONLY


def _rounded(a, precision):
    if precision == FP32:
        return a.astype(np.float32).astype(np.float64)
    if precision == BF16:
        m, e = np.frexp(a)
        return np.ldexp(np.rint(256.0 * m), e - 8)
    return a


# (storage of the systems one after the other; None: one set by the caller)
@pytest.mark.parametrize("systems", [(FP32 | LOW,), (BF16 | LOW,), (FP32, FP64), (BF16, None), (FP32 | LOW, BF16),
                                     (FP64, FP32 | LOW), (FP32, BF16 | LOW), (BF16 | LOW, None, FP32 | LOW)])
@pytest.mark.parametrize("asked", [FP64, FP32, BF16])
def test_the_product_takes_a_copy_of_this_system(gpu_available, systems, asked):
    import torch

    m = box_mesh((5, 4, 6), jitter=0.15, seed=5, rcm=2)
    n = m.nnode
    rng = np.random.default_rng(3)
    x = rng.uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params(mach=0.3, mach_min=0.3, cfl_min=10.0, cfl_max=10.0)) as s:
        IA, JA, _ = s.get_block_pattern()
        for k, storage in enumerate(systems):
            if storage is None:
                s.set_system(rng.uniform(-1.0, 1.0, (len(JA), 25)), np.zeros((n, 5)))
            else:
                s.set_state(perturbed_freestream(m, 1.4, 0.3, 1.25, noise=0.01, seed=k))
                s.residual_step(0)
                s.Compute_Jacobian(1, 0, precision=storage)
        A = s.get_system()[0].reshape(-1, 5, 5)
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), asked)
        s.synchronize()
        y = yd.cpu().numpy()
    # get_system gives the FP64 copy, or the only one widened
    last = FP64 if systems[-1] is None else systems[-1]
    copy = asked if asked == last else FP64
    terms = _rounded(A, copy) * x[JA][:, None, :]
    want = np.add.reduceat(terms.sum(axis=2), IA[:-1], axis=0)
    scale = np.add.reduceat(np.abs(terms).sum(axis=2), IA[:-1], axis=0)
    assert np.all(np.abs(y - want) <= 2e-14 * scale)
