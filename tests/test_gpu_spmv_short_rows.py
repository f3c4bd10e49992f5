"""The block SpMV on both sides of the rule that gives short rows a lane per
output: planes and lines of nodes (3 to 5 blocks per row), hexahedra (7, BF16 by
the size of the matrix) and tets, ragged ends included, in every precision.

Tolerance: the product and the value it is compared with each add at most 15 * 5
entries in FP64, 2 * 75 * 1.1e-16 of the sum of their magnitudes, 2e-14."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, box_mesh, capi, default_params, perturbed_freestream

pytestmark = pytest.mark.gpu

LOW = capi.PREC_LOW_ONLY


def _grid(nx, ny, nz):
    """Nodes of a grid joined along its lines."""
    I = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    pairs = np.concatenate([np.stack([a.ravel(), b.ravel()], 1) for a, b in
                            ((I[:, :, :-1], I[:, :, 1:]), (I[:, :-1], I[:, 1:]), (I[:-1], I[1:]))])
    n = I.size
    rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return Mesh(nnode=n, nghost=0, edge_nodes=pairs.astype(np.int32), edge_areav=np.ones((len(pairs), 3)),
                bedge_nodes=np.zeros((0, 2), np.int32), bedge_areav=np.zeros((0, 3)),
                bedge_type=np.zeros(0, np.int32), cvol=np.ones(n), coords=np.zeros((n, 3)), n2n_ia=ia,
                n2n_ja=cols[order].astype(np.int32))


MESHES = {
    "one row": lambda: _grid(1, 1, 1),
    "line": lambda: _grid(1001, 1, 1),
    "plane": lambda: _grid(37, 53, 1),
    "slab": lambda: _grid(40, 31, 3),       # 6.2 blocks per row
    "hexahedra": lambda: _grid(19, 22, 17),
    "hexahedra past L2": lambda: _grid(75, 74, 72),  # 2.77 M blocks, 139 MB in BF16
    "tets": lambda: box_mesh((9, 8, 7), jitter=0.15, seed=5, rcm=2),
}


@pytest.mark.parametrize("storage", [capi.PREC_FP64, capi.PREC_FP32 | LOW, capi.PREC_BF16 | LOW])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_products(gpu_available, mesh, storage):
    import torch

    m = MESHES[mesh]()
    n = m.nnode
    x = np.random.default_rng(3).uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params(mach=0.3, mach_min=0.3, cfl_min=10.0, cfl_max=10.0)) as s:
        s.set_state(perturbed_freestream(m, 1.4, 0.3, 1.25, noise=0.01, seed=1))
        s.begin_iteration(0)
        s.Compute_Jacobian(0, 0, precision=storage)
        A = s.get_system()[0].reshape(-1, 5, 5)
        IA, JA, _ = s.get_block_pattern()
        xd = torch.from_numpy(x).cuda()
        yd = torch.full_like(xd, float("nan"))
        s.spmv_device(xd.data_ptr(), yd.data_ptr(), storage & ~LOW)
        s.synchronize()
        y = yd.cpu().numpy()
    terms = A * x[JA][:, None, :]
    want = np.add.reduceat(terms.sum(axis=2), IA[:-1], axis=0)
    scale = np.add.reduceat(np.abs(terms).sum(axis=2), IA[:-1], axis=0)
    assert np.all(np.abs(y - want) <= 2e-14 * scale)

