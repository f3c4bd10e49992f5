"""The block SpMV on rows that end at every place of a batch of blocks in flight
(1 to 12 blocks per row, in one matrix and alone), in every storage precision.

Tolerance: sums of at most 12 blocks of five products in FP64, 60 * 1.1e-16 of
the sum of magnitudes, against the stored (rounded) matrix."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, box_mesh, capi, default_params
from oracle import restatement
from tests._util import make_case, params_from, relerr

pytestmark = pytest.mark.gpu


def _rows(lengths):
    """Stars: for every length L a hub with L - 1 leaves, so rows of L and of 2 blocks."""
    pairs, n = [], 0
    for L in lengths:
        pairs += [(n, n + k) for k in range(1, L)]
        n += L
    pairs = np.array(pairs, np.int32).reshape(-1, 2)
    rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return Mesh(nnode=n, nghost=0, edge_nodes=pairs, edge_areav=np.ones((len(pairs), 3)),
                bedge_nodes=np.zeros((0, 2), np.int32), bedge_areav=np.zeros((0, 3)),
                bedge_type=np.zeros(0, np.int32), cvol=np.ones(n), coords=np.zeros((n, 3)), n2n_ia=ia,
                n2n_ja=cols[order].astype(np.int32))


@pytest.mark.parametrize("lengths", [[k] for k in range(1, 13)] + [list(range(1, 13)) * 7])
def test_rows_of_every_length(gpu_available, lengths):
    import torch

    m = _rows(lengths)
    rng = np.random.default_rng(9)
    rs = restatement.Session(m, {})
    A, x = rng.uniform(-1.0, 1.0, (len(rs.JA), 5, 5)), rng.uniform(-1.0, 1.0, (m.nnode, 5))
    with Euler3DGPU(m, default_params()) as s:
        s.set_system(A.reshape(-1, 25), np.zeros((m.nnode, 5)))
        xd = torch.from_numpy(x).cuda()
        yd = torch.full_like(xd, float("nan"))
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), capi.PREC_FP64)
        s.synchronize()
        y = yd.cpu().numpy()
    bound = rs.spmv(np.abs(A), np.abs(x))
    assert np.all(np.abs(y - rs.spmv(A, x)) <= 60 * 1.2e-16 * bound)


@pytest.mark.parametrize("precision", [capi.PREC_FP32, capi.PREC_BF16])
def test_low_precision_matrices(gpu_available, precision):
    import torch

    m, cfg, Q = make_case(mesh=box_mesh((6, 5, 4), jitter=0.15, seed=5, rcm=2), seed=7)
    rng = np.random.default_rng(9)
    x = rng.uniform(-1.0, 1.0, (m.nnode, 5))
    with Euler3DGPU(m, params_from(cfg)) as s:
        s.set_state(Q)
        s.residual_step(0)
        s.Compute_Jacobian(1, 0, precision=precision | capi.PREC_LOW_ONLY)
        A = s.get_system()[0]
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), precision)
        s.synchronize()
        y = yd.cpu().numpy()
    rs = restatement.Session(m, {})
    assert relerr(y, rs.spmv(A, x)) <= 15 * 5 * 1.2e-16 * 10
