"""Block Gauss-Seidel on both sides of the rule that gives wide levels a launch
each: layered graphs whose mean rows per level lie just below and above it, one
wide level alone, wide and narrow levels mixed.  Every direction, and a solve
that stops early; bit for bit against the oracle's sequential sweeps (the RMS
sums its rows in another order: n terms of relative rounding 1.1e-16)."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, default_params
from oracle import restatement

pytestmark = pytest.mark.gpu


def _layered(widths, links, seed=3):
    """Layers of the given widths; every node joined to `links` random ones of the layer before."""
    rng = np.random.default_rng(seed)
    starts = np.concatenate([[0], np.cumsum(widths)])
    pairs = [np.zeros((0, 2), np.int64)]
    for k in range(1, len(widths)):
        b = np.repeat(np.arange(starts[k], starts[k + 1]), links)
        pairs.append(np.stack([rng.integers(starts[k - 1], starts[k], len(b)), b], 1))
    pairs = np.unique(np.concatenate(pairs), axis=0)
    n, e = int(starts[-1]), len(pairs)
    rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return Mesh(nnode=n, nghost=0, edge_nodes=pairs.astype(np.int32), edge_areav=np.ones((e, 3)),
                bedge_nodes=np.zeros((0, 2), np.int32), bedge_areav=np.zeros((0, 3)),
                bedge_type=np.zeros(0, np.int32), cvol=np.ones(n), coords=rng.random((n, 3)), n2n_ia=ia,
                n2n_ja=cols[order].astype(np.int32))


# limits: 1 block per row 1035 rows, 4 blocks 1139, 6 blocks 1209, 22 blocks and more 1750
MESHES = {
    "one level, cluster": lambda: _layered([1035], 0),
    "one level, launches": lambda: _layered([1036], 0),
    "two levels, launches": lambda: _layered([3000, 3000], 3),
    "layers, cluster": lambda: _layered([1150] * 5, 3),
    "layers, launches": lambda: _layered([1300] * 5, 3),
    "long rows, cluster": lambda: _layered([1700] * 3, 20),
    "long rows, launches": lambda: _layered([1800] * 3, 20),
    "uneven, cluster": lambda: _layered([3000, 5, 200, 7], 3),
    "uneven, launches": lambda: _layered([9000, 5, 1], 3),
}


@pytest.mark.parametrize("direction", [0, 1, 2])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_wide_and_narrow_levels(gpu_available, mesh, direction):
    m = MESHES[mesh]()
    n = m.nnode
    rng = np.random.default_rng(4)
    rs = restatement.Session(m, {})
    A = rng.uniform(-1.0, 1.0, (len(rs.JA), 5, 5)) / (5.0 * np.repeat(np.diff(rs.IA), np.diff(rs.IA)))[:, None, None]
    A[rs.IAU] += 3.0 * np.eye(5)
    B = rng.uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params()) as s:
        s.set_system(A.reshape(-1, 25), B)
        for sweeps in (1, 4, 60):  # 60: the residual reaches the stopping level first
            rms = s.MC_Iterative_Block_LU_Jacobi_CRS(sweeps, direction)
            Xo, rmso = rs.block_gs(A, B, sweeps, direction)
            assert np.array_equal(s.get_system()[2], Xo)
            assert abs(rms - rmso) <= n * 1.2e-16 * abs(rmso)
