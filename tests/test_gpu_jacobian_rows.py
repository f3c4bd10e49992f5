"""The row-wise Jacobian assembly and the block SpMV at their edges: meshes of
one partly filled warp, of exactly one, with a ragged last one; rows of one
block and of many, row counts that do not fill a CTA.

Tolerances: FP64 Jacobian 1e-12 normwise (sums of up to 30 terms of a few
rounding errors each); low-precision-only systems round every off-diagonal
block once and sum the diagonal from up to 27 rounded ones, 28 units in the last
place: 28 * 2^-24 in FP32, 28 * 2^-8 in BF16.  SpMV: sums of up to 65 blocks
of five products, 325 * 1.1e-16."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params
from oracle import restatement
from tests._util import make_case, params_from, relerr
from tests.test_gpu_ilu_solves import _graph_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(capi.PREC_FP64, 1e-12), (capi.PREC_FP32 | capi.PREC_LOW_ONLY, 28 * 2.0 ** -24),
                                           (capi.PREC_BF16 | capi.PREC_LOW_ONLY, 28 * 2.0 ** -8)])
@pytest.mark.parametrize("size", [(1, 1, 1), (3, 3, 1), (6, 4, 3), (11, 9, 8)])
def test_jacobian_rows_match_the_oracle(gpu_available, size, precision, tol):
    m, cfg, Q = make_case(mesh=box_mesh(size, jitter=0.15, seed=5, rcm=2), seed=7)
    o = restatement.first_order_step(m, cfg, Q, gs_sweeps=1)
    with Euler3DGPU(m, params_from(cfg)) as s:
        s.set_state(Q)
        s.begin_iteration(0)
        s.Apply_Boundary_Condition(0)
        s.Compute_Residual(1)
        s.Compute_DeltaT(0)
        s.Compute_Jacobian(1, 0, precision=precision)
        A, B, _ = s.get_system()
    assert relerr(A, o["A"]) <= tol
    assert relerr(B, o["B"]) <= 1e-12


@pytest.mark.parametrize("n,degree", [(1, 0), (5, 2), (24, 4), (25, 9), (700, 14), (301, 60)])
def test_spmv_rows_of_any_length(gpu_available, n, degree):
    import torch

    m = _graph_mesh(n, degree, 8)
    rng = np.random.default_rng(9)
    rs = restatement.Session(m, {})
    A, x = rng.uniform(-1.0, 1.0, (len(rs.JA), 5, 5)), rng.uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params()) as s:
        s.set_system(A.reshape(-1, 25), np.zeros((n, 5)))
        xd = torch.from_numpy(x).cuda()
        yd = torch.full_like(xd, float("nan"))
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), capi.PREC_FP64)
        s.synchronize()
        y = yd.cpu().numpy()
    assert relerr(y, rs.spmv(A, x)) <= 325 * 1.2e-16
