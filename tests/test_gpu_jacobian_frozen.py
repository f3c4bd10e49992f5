"""The Jacobian of a state with a time step of zero (CFL 0: nothing may move):
V/dt is infinite on the diagonal of the diagonal blocks and touches no other
entry."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi
from tests._util import make_case, params_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(5, 4, 3), (26, 25, 24)])  # four lanes per row, and one
def test_a_time_step_of_zero_stays_on_the_diagonal(gpu_available, size):
    m, cfg, Q = make_case(mesh=box_mesh(size, jitter=0.15, seed=5, rcm=2), seed=7)
    with Euler3DGPU(m, params_from(dict(cfg, cfl_min=0.0, cfl_max=0.0))) as s:
        s.set_state(Q)
        s.residual_step(0)
        assert not np.any(s.get_deltat())
        IA, JA, IAU = s.get_block_pattern()
        s.Compute_Jacobian(0, 0)
        A0 = s.get_system()[0]
        s.Compute_Jacobian(1, 0)
        A = s.get_system()[0]
    eye = np.zeros((len(JA), 5, 5), bool)
    eye[IAU] = np.eye(5, dtype=bool)
    assert np.all(np.isposinf(A[eye]))
    assert np.array_equal(A[~eye], A0[~eye])
