"""The block-multicolour ILU(0) on rows that no block couples, more patches of
one colour than are prefetched ahead: the forward solve's regions are empty and
an application is the inverse of the diagonal blocks.

Tolerances: the diagonal blocks are 5 I plus entries below 0.2, of condition
below 2; FP64 100 * 1.1e-16 over a 5x5 inverse and product, FP32 factors stored
to 6e-8 each."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, capi, default_params
from tests._util import relerr
from tests.test_gpu_ilu_solves import _graph_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(capi.PREC_FP64, 1e-14), (capi.PREC_FP32, 1e-6)])
@pytest.mark.parametrize("edges", [0, 3])  # 3: a second colour, whose patches have lower blocks
def test_uncoupled_rows(gpu_available, edges, precision, tol):
    import torch

    n = 32 * 700 + 1
    m = _graph_mesh(n, 0, 3)
    if edges:
        pairs = np.array([[0, 40], [31, 64], [n - 33, n - 1]], np.int32)
        rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
        ia = np.zeros(n + 1, np.int32)
        np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
        m.edge_nodes, m.edge_areav = pairs, np.ones((3, 3))
        m.n2n_ia, m.n2n_ja = ia, cols[np.argsort(rows, kind="stable")].astype(np.int32)
    rng = np.random.default_rng(6)
    x = rng.uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params()) as s:
        IA, JA, IAU = s.get_block_pattern()
        A = np.zeros((len(JA), 5, 5))
        A[IAU] = 5.0 * np.eye(5) + rng.uniform(-0.2, 0.2, (n, 5, 5))  # the off-diagonal blocks are zero
        s.set_system(A.reshape(-1, 25), rng.uniform(-1.0, 1.0, (n, 5)))
        s.solve_gmres(restart=5, max_iters=1, rtol=1e-6, precond=capi.PC_ILU0_MC, precision=precision,
                      allow_not_converged=True)
        xd = torch.from_numpy(x).cuda()
        zd = torch.full_like(xd, float("nan"))
        s.precond_apply_device(xd.data_ptr(), zd.data_ptr())
        s.synchronize()
        z = zd.cpu().numpy()
    assert relerr(z, np.linalg.solve(A[IAU], x[:, :, None])[:, :, 0]) <= tol
