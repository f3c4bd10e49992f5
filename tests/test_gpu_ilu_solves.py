"""The block-multicolour ILU(0) solves against the oracle's ILU(0) of the
permuted system, at the sizes where the patch layout can go wrong: one partly
filled patch, ragged last patches, patches whose off-patch blocks exceed the
staged part, and rows of a hundred blocks, whose lists do not fit beside the
staged blocks.

Tolerances: the systems are block diagonally dominant (diagonal 5, the other
entries of a row sum to about 1 in magnitude), so a solve amplifies an error by
less than 2.  FP64: sums of up to 500 products, 500 * 1.1e-16 * 2 < 1e-12.
FP32 factors: each stored to 6e-8, two solves and the factors' own history,
below 1e-6."""
import ctypes as C

import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, box_mesh, capi, default_params
from oracle import restatement
from tests._util import relerr
from tests.test_gpu_linsolve import _permuted_system

pytestmark = pytest.mark.gpu


def _graph_mesh(n, degree, seed):
    """n nodes joined to about `degree` others each, at random (no geometry: the systems are set by the caller)."""
    rng = np.random.default_rng(seed)
    pairs = rng.integers(0, n, (n * degree // 2, 2))
    pairs = np.unique(np.sort(pairs[pairs[:, 0] != pairs[:, 1]], axis=1), axis=0)
    e = len(pairs)
    rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return Mesh(nnode=n, nghost=0, edge_nodes=pairs.astype(np.int32), edge_areav=np.ones((e, 3)),
                bedge_nodes=np.zeros((0, 2), np.int32), bedge_areav=np.zeros((0, 3)),
                bedge_type=np.zeros(0, np.int32), cvol=np.ones(n), coords=rng.random((n, 3)), n2n_ia=ia,
                n2n_ja=cols[order].astype(np.int32))


CASES = {
    "one partly filled patch": lambda: box_mesh((1, 2, 1), seed=3),
    "one full patch": lambda: box_mesh((3, 3, 1), seed=3),
    "ragged": lambda: box_mesh((11, 3, 6), seed=3, rcm=2),
    "many patches": lambda: box_mesh((31, 26, 19), seed=3, rcm=2),
    "off-patch blocks past the staged part": lambda: _graph_mesh(610, 60, 4),
    "lists past the staged part": lambda: _graph_mesh(1900, 100, 5),
}


@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_FP32])
@pytest.mark.parametrize("case", list(CASES))
def test_multicolour_solves_match_the_oracle(gpu_available, case, precision):
    import torch

    m = CASES[case]()
    n = m.nnode
    rng = np.random.default_rng(6)
    with Euler3DGPU(m, default_params()) as s:
        IA, JA, IAU = s.get_block_pattern()
        A = rng.uniform(-1.0, 1.0, (len(JA), 5, 5)) / (5.0 * np.repeat(np.diff(IA), np.diff(IA)))[:, None, None]
        A[IAU] += 5.0 * np.eye(5)
        B = rng.uniform(-1.0, 1.0, (n, 5))
        x = rng.uniform(-1.0, 1.0, (n, 5))
        order = np.empty(n, np.int32)
        ncol = C.c_int()
        capi.check(capi.lib.cfd_ilu_mc_order(s.handle, capi.ptr(order), C.byref(ncol)), "cfd_ilu_mc_order")
        s.set_system(A.reshape(-1, 25), B)
        s.solve_gmres(restart=5, max_iters=1, rtol=1e-14, precond=capi.PC_ILU0_MC, precision=precision,
                      allow_not_converged=True)
        xd = torch.from_numpy(x).cuda()
        zd = torch.empty_like(xd)
        for _ in range(2):  # the second apply reads the vectors the first one left
            s.precond_apply_device(xd.data_ptr(), zd.data_ptr())
        s.synchronize()
        z = zd.cpu().numpy()
    IAp, JAp, IAUp, Ap, _, pos = _permuted_system(IA, JA, IAU, A, B, order)
    p = restatement._p
    F, zp, xp = np.zeros_like(Ap), np.zeros((n, 5)), np.ascontiguousarray(x[order])
    assert restatement.lib.orc_ilu0(n, p(IAp), p(JAp), p(IAUp), p(Ap), p(F)) == 0
    restatement.lib.orc_ilu0_apply(n, p(IAp), p(JAp), p(IAUp), p(F), p(xp), p(zp))
    assert relerr(z, zp[pos]) <= (1e-12 if precision == capi.PREC_FP64 else 1e-6)
