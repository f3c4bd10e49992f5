"""GMRES on a system with a block that is not finite: an error and no solution,
also with a tolerance that the zero start already meets (its defect B - A 0 is
not finite), and with a right-hand side that is not finite."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("rtol", [1e-6, 1.0, 2.0])
def test_a_block_that_is_not_finite_is_reported(gpu_available, rtol, bad):
    m = box_mesh((4, 3, 2), seed=3)
    with Euler3DGPU(m, default_params()) as s:
        IA, JA, IAU = s.get_block_pattern()
        A = np.zeros((len(JA), 5, 5))
        A[IAU] = 5.0 * np.eye(5)
        A[IAU[7] + 1, 2, 1] = bad
        s.set_system(A.reshape(-1, 25), np.ones((m.nnode, 5)))
        with pytest.raises(capi.CfdError) as e:
            s.solve_gmres(restart=5, max_iters=5, rtol=rtol, precond=capi.PC_NONE)
        assert e.value.code == -6  # CFD_ERR_NUMERIC
        assert not np.any(s.get_system()[2])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_right_hand_side_that_is_not_finite_is_reported(gpu_available, bad):
    m = box_mesh((4, 3, 2), seed=3)
    with Euler3DGPU(m, default_params()) as s:
        IA, JA, IAU = s.get_block_pattern()
        A, B = np.zeros((len(JA), 5, 5)), np.ones((m.nnode, 5))
        A[IAU] = 5.0 * np.eye(5)
        B[11, 3] = bad
        s.set_system(A.reshape(-1, 25), B)
        for precond in (capi.PC_NONE, capi.PC_BLOCK_JACOBI, capi.PC_ILU0_MC):
            with pytest.raises(capi.CfdError) as e:
                s.solve_gmres(restart=5, max_iters=5, rtol=1e-6, precond=precond)
            assert e.value.code == -6
            assert not np.any(s.get_system()[2])


def test_a_tolerance_met_at_the_start(gpu_available):
    m = box_mesh((4, 3, 2), seed=3)
    with Euler3DGPU(m, default_params()) as s:
        IA, JA, IAU = s.get_block_pattern()
        A = np.zeros((len(JA), 5, 5))
        A[IAU] = 5.0 * np.eye(5)
        s.set_system(A.reshape(-1, 25), np.ones((m.nnode, 5)))
        st = s.solve_gmres(restart=5, max_iters=5, rtol=1.0, precond=capi.PC_NONE)
        assert (st.iterations, st.rel_residual) == (0, 1.0)
        assert not np.any(s.get_system()[2])
