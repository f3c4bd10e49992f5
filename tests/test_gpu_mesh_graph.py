"""Meshes whose node graph is not that of their edges: the Jacobians, which
place an edge's blocks by the graph's rows, refuse them; a residual step, which
needs the edges alone, runs as on the mesh with the right graph."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi
from tests._util import make_case, params_from

pytestmark = pytest.mark.gpu


def _moved(m):
    """One neighbour less in row 0, one more in the last row."""
    ia, ja = m.n2n_ia.copy(), m.n2n_ja.tolist()
    ja.pop(0)
    ja.append(0)
    ia[1:-1] -= 1
    return ia, np.array(ja, np.int32)


def _twice(m):
    """Row 3 names its first neighbour twice and its last one not at all."""
    ia, ja = m.n2n_ia.copy(), m.n2n_ja.copy()
    ja[ia[4] - 1] = ja[ia[3]]
    return ia, ja


def _other(m):
    """Row 3 names a node that is no neighbour of it."""
    ia, ja = m.n2n_ia.copy(), m.n2n_ja.copy()
    ja[ia[3]] = m.nnode - 1
    return ia, ja


def _shuffled(m):
    """The right graph with every row reversed."""
    ia, ja = m.n2n_ia.copy(), m.n2n_ja.copy()
    for i in range(m.nnode):
        ja[ia[i]:ia[i + 1]] = ja[ia[i]:ia[i + 1]][::-1]
    return ia, ja


@pytest.mark.parametrize("graph,right", [(_moved, False), (_twice, False), (_other, False), (_shuffled, True)])
def test_jacobian_needs_the_graph_of_the_edges(gpu_available, graph, right):
    m, cfg, Q = make_case(mesh=box_mesh((5, 4, 3), seed=5), seed=7)
    out = []
    for ia, ja in ((m.n2n_ia, m.n2n_ja), graph(m)):
        m.n2n_ia, m.n2n_ja = ia, ja
        with Euler3DGPU(m, params_from(cfg)) as s:
            s.set_state(Q)
            s.residual_step(0)
            res = s.get_residual()
            if out and not right:
                for call in (lambda: s.Compute_Jacobian(1, 0),
                             lambda: s.Compute_Jacobian(1, 0, precision=capi.PREC_FP32 | capi.PREC_LOW_ONLY),
                             lambda: s.Compute_Jacobian_FiniteDifference(1, 0)):
                    with pytest.raises(capi.CfdError) as e:
                        call()
                    assert e.value.code == -2  # CFD_ERR_MESH
                out.append(res)
                continue
            s.Compute_Jacobian(1, 0)
            out.append((*res, s.get_system()[0]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
