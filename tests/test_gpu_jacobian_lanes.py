"""The Jacobian with four lanes per row and with one: meshes just below and
above the limit of 16,000 rows, with rows of 7 to 15 blocks and a ragged end,
every flux mode, both sets of variables, and all forms of storage.  The blocks
of an edge come out of the same operations on either side, so the two forms are
compared through the oracle (Roe, conservative) and through each other: a row's
off-diagonal blocks are those of the same edge on a mesh of the other size.

Tolerances: FP64 1e-12 normwise against the oracle; the sums of at most 30
blocks in another order differ by 30 * 1.1e-16 of their largest term, 1e-13."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, box_mesh, capi, default_params, perturbed_freestream, to_rup
from oracle import restatement
from tests._util import make_case, params_from, relerr

pytestmark = pytest.mark.gpu

LOW32, LOW16 = capi.PREC_FP32 | capi.PREC_LOW_ONLY, capi.PREC_BF16 | capi.PREC_LOW_ONLY


# 24 x 24 x 24 hexes: 15,625 rows, four lanes; 25 x 24 x 24: 16,250 rows, one
@pytest.mark.parametrize("size", [(24, 24, 24), (25, 24, 24)])
@pytest.mark.parametrize("precision,tol", [(capi.PREC_FP64, 1e-12), (capi.PREC_FP32, 1e-12), (LOW32, 28 * 2.0 ** -24),
                                           (LOW16, 28 * 2.0 ** -8)])
def test_both_sides_of_the_limit_match_the_oracle(gpu_available, size, precision, tol):
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


def _padded(m, k):
    """m with k more nodes that nothing couples (past the limit, the same rows go to one lane each)."""
    n = m.nnode
    bn = m.bedge_nodes.copy()
    bn[:, 1] += k
    return Mesh(nnode=n + k, nghost=m.nghost, edge_nodes=m.edge_nodes, edge_areav=m.edge_areav, bedge_nodes=bn,
                bedge_areav=m.bedge_areav, bedge_type=m.bedge_type, cvol=np.r_[m.cvol, np.ones(k)],
                coords=np.r_[m.coords, np.zeros((k, 3))], n2n_ia=np.r_[m.n2n_ia, np.full(k, m.n2n_ia[-1])].astype(np.int32),
                n2n_ja=m.n2n_ja)


@pytest.mark.parametrize("precision", [capi.PREC_FP64, LOW32, LOW16])
@pytest.mark.parametrize("rup", [0, 1])
@pytest.mark.parametrize("kw", [dict(), dict(entropy_fix=1), dict(flux_scheme=capi.FLUX_ROE_THORNBER),
                                dict(flux_scheme=capi.FLUX_ROE_PRECOND, precond_method=capi.PRECOND_TURKEL, precond_mach=0.3)])
def test_one_and_four_lanes_agree(gpu_available, kw, rup, precision):
    m = box_mesh((9, 7, 6), jitter=0.15, seed=5, rcm=2)
    n, nb = m.nnode, len(m.n2n_ja) + m.nnode
    Q = perturbed_freestream(m, 1.4, 0.3, 1.25, noise=0.01, seed=1)
    if rup:
        Q = to_rup(Q, 1.4, 0.0)
    out = []
    for mesh in (m, _padded(m, 16001 - n)):
        k = mesh.nnode - n
        q = np.concatenate([Q[:, :n], np.repeat(Q[:, :1], k, axis=1), Q[:, n:]], axis=1)
        with Euler3DGPU(mesh, default_params(mach=0.3, mach_min=0.3, cfl_min=10.0, cfl_max=10.0, variables=rup, **kw)) as s:
            s.set_state(q)
            s.residual_step(0)
            s.Compute_Jacobian(1, 0, include_diss=1, precision=precision)
            A, B, _ = s.get_system()
        out.append((A[:nb], B[:n]))
    (A4, B4), (A1, B1) = out
    assert np.array_equal(B4, B1)
    IAU = np.array([np.searchsorted(np.sort(np.r_[m.n2n_ja[m.n2n_ia[i]:m.n2n_ia[i + 1]], i]), i) + m.n2n_ia[i] + i
                    for i in range(n)])
    off = np.ones(nb, bool)
    off[IAU] = False
    assert np.array_equal(A4[off], A1[off])
    # the stored diagonal blocks: rounded once more in the low-precision forms
    assert relerr(A4, A1) <= {capi.PREC_FP64: 1e-13, LOW32: 2.0 ** -23, LOW16: 2.0 ** -7}[precision]
