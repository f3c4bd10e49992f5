"""Block Gauss-Seidel with a sweep per launch against the oracle's sequential
sweeps, bit for bit: one row, levels narrower and wider than the cluster's
chunk, rows longer than the staged part, every direction, and a solve that
stops early.  The RMS sums its rows in another order than the oracle: n terms of
relative rounding 1.1e-16 each."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, default_params
from oracle import restatement
from tests.test_gpu_ilu_solves import _graph_mesh

pytestmark = pytest.mark.gpu

MESHES = {
    "one row": lambda: _graph_mesh(1, 0, 3),
    "wide levels": lambda: _graph_mesh(1500, 3, 3),
    "long rows": lambda: _graph_mesh(230, 40, 3),
    "box": lambda: box_mesh((9, 8, 7), seed=3, rcm=2),
}


@pytest.mark.parametrize("direction", [0, 1, 2])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_sweeps_match_the_oracle_bit_for_bit(gpu_available, mesh, direction):
    m = MESHES[mesh]()
    n = m.nnode
    rng = np.random.default_rng(4)
    rs = restatement.Session(m, {})
    A = rng.uniform(-1.0, 1.0, (len(rs.JA), 5, 5)) / (5.0 * np.repeat(np.diff(rs.IA), np.diff(rs.IA)))[:, None, None]
    A[rs.IAU] += 3.0 * np.eye(5)
    B = rng.uniform(-1.0, 1.0, (n, 5))
    with Euler3DGPU(m, default_params()) as s:
        s.set_system(A.reshape(-1, 25), B)
        for sweeps in (1, 5, 60):  # 60: the residual reaches the stopping level first
            rms = s.MC_Iterative_Block_LU_Jacobi_CRS(sweeps, direction)
            _, _, X = s.get_system()
            Xo, rmso = rs.block_gs(A, B, sweeps, direction)
            assert np.array_equal(X, Xo)
            assert abs(rms - rmso) <= n * 1.2e-16 * abs(rmso)
