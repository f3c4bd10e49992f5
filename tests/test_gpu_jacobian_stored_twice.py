"""The Jacobian stored twice, in FP64 and in FP32 or BF16, with four lanes per
row (up to 16,000 rows) and with two: every block of the low-precision matrix is
the rounded FP64 one, as a product with it shows, and the FP64 matrix is that of
the assembly that stores it alone.

Tolerances: the diagonal blocks are sums of at most 30 blocks in another order,
30 * 1.1e-16 of their largest term, 1e-13.  The product and the value it is
compared with each add at most 15 * 5 rounded entries in FP64: 2 * 75 * 1.1e-16
of the sum of their magnitudes, 2e-14."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params, perturbed_freestream, to_rup
from tests._util import relerr

pytestmark = pytest.mark.gpu


def _bf16(a):
    """a rounded once, to eight significant bits (ties to even)."""
    m, e = np.frexp(a)
    return np.ldexp(np.rint(256.0 * m), e - 8)


# 4,913 and 15,625 rows: four lanes; 16,250 and 20,944 (ragged): two
@pytest.mark.parametrize("size", [16, 24, (25, 24, 24), (33, 21, 27)])
@pytest.mark.parametrize("low", ["FP32", "BF16"])
@pytest.mark.parametrize("rup", [0, 1])
@pytest.mark.parametrize("kw", [dict(), dict(flux_scheme=capi.FLUX_ROE_THORNBER),
                                dict(flux_scheme=capi.FLUX_ROE_PRECOND, precond_method=capi.PRECOND_TURKEL, precond_mach=0.3)])
def test_both_matrices(gpu_available, kw, rup, low, size):
    import torch

    m = box_mesh(size, jitter=0.15, seed=5, rcm=2)
    n = m.nnode
    Q = perturbed_freestream(m, 1.4, 0.3, 1.25, noise=0.01, seed=1)
    if rup:
        Q = to_rup(Q, 1.4, 0.0)
    prec = capi.PREC_FP32 if low == "FP32" else capi.PREC_BF16
    x = np.random.default_rng(2).uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params(mach=0.3, mach_min=0.3, cfl_min=10.0, cfl_max=10.0, variables=rup, **kw)) as s:
        s.set_state(Q)
        s.residual_step(0)
        s.Compute_Jacobian(1, 0, include_diss=1, precision=capi.PREC_FP64)
        A1, B1, _ = s.get_system()
        s.Compute_Jacobian(1, 0, include_diss=1, precision=prec)
        A, B, _ = s.get_system()
        IA, JA, _ = s.get_block_pattern()
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), prec)
        s.synchronize()
        y = yd.cpu().numpy()
    A, A1 = A.reshape(-1, 5, 5), A1.reshape(-1, 5, 5)
    assert np.array_equal(B, B1)
    assert relerr(A, A1) <= 1e-13
    R = A.astype(np.float32).astype(np.float64) if low == "FP32" else _bf16(A)
    terms = R * x[JA][:, None, :]
    want = np.add.reduceat(terms.sum(axis=2), IA[:-1], axis=0)
    scale = np.add.reduceat(np.abs(terms).sum(axis=2), IA[:-1], axis=0)
    assert np.all(np.abs(y - want) <= 2e-14 * scale)
