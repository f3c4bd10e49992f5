"""The block-multicolour ILU(0) where a patch's rows hang on one another in one
chain of 32 levels (rows coupled to the next one, as a mesh numbered along its
lines), on both sides of the rule that gives a colour's patches a warp or a CTA
each, with and without blocks between the patches beside the chain's ends;
against the oracle's ILU(0) of the permuted system.

Tolerances as for the other systems of this dominance (diagonal 5, a row's other
entries sum to about 1): FP64 sums of at most 25 products per entry and solves
that amplify by less than 2, 1e-12; FP32 factors stored to 6e-8 each, 1e-6."""
import ctypes as C

import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, Mesh, capi, default_params
from oracle import restatement
from tests._util import relerr
from tests.test_gpu_linsolve import _permuted_system

pytestmark = pytest.mark.gpu


def _banded(n, offsets):
    """Rows i and i + k coupled for every k of offsets."""
    pairs = np.concatenate([np.stack([np.arange(n - k), np.arange(k, n)], 1) for k in offsets])
    rows, cols = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return Mesh(nnode=n, nghost=0, edge_nodes=pairs.astype(np.int32), edge_areav=np.ones((len(pairs), 3)),
                bedge_nodes=np.zeros((0, 2), np.int32), bedge_areav=np.zeros((0, 3)),
                bedge_type=np.zeros(0, np.int32), cvol=np.ones(n), coords=np.zeros((n, 3)), n2n_ia=ia,
                n2n_ja=cols[order].astype(np.int32))


@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_FP32])
# two colours of 220 patches (a CTA each) and of 250 (a warp each); 5 blocks per row: 300 and 450 patches a colour
@pytest.mark.parametrize("n,offsets", [(32 * 440, (1,)), (32 * 500, (1,)), (32 * 500 - 7, (1,)), (32 * 600, (1, 40)),
                                       (32 * 900 + 5, (1, 40)), (32 * 1400, (1, 2, 40))])
def test_chains_match_the_oracle(gpu_available, n, offsets, precision):
    import torch

    m = _banded(n, offsets)
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
        s.precond_apply_device(xd.data_ptr(), zd.data_ptr())
        s.synchronize()
        z = zd.cpu().numpy()
    IAp, JAp, IAUp, Ap, _, pos = _permuted_system(IA, JA, IAU, A, B, order)
    p = restatement._p
    F, zp, xp = np.zeros_like(Ap), np.zeros((n, 5)), np.ascontiguousarray(x[order])
    assert restatement.lib.orc_ilu0(n, p(IAp), p(JAp), p(IAUp), p(Ap), p(F)) == 0
    restatement.lib.orc_ilu0_apply(n, p(IAp), p(JAp), p(IAUp), p(F), p(xp), p(zp))
    assert relerr(z, zp[pos]) <= (1e-12 if precision == capi.PREC_FP64 else 1e-6)
