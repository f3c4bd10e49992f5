"""One context that goes from one preconditioner to another: every application
of the block-multicolour ILU(0) equals a fresh context's, bit for bit, although
the factor buffers in between were given back and taken again in another size
and storage type (on the caller's own stream, where applies are captured)."""
import numpy as np
import pytest

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params

pytestmark = pytest.mark.gpu

MC64, MC32 = (capi.PC_ILU0_MC, capi.PREC_FP64), (capi.PC_ILU0_MC, capi.PREC_FP32)
BJ64, ILU64 = (capi.PC_BLOCK_JACOBI, capi.PREC_FP64), (capi.PC_ILU0, capi.PREC_FP64)


@pytest.mark.parametrize("sequence", [(MC64, BJ64, MC32, MC64), (MC64, MC32, ILU64, MC32, BJ64, MC64, BJ64, MC32)])
def test_applies_equal_a_fresh_contexts(gpu_available, sequence):
    import torch

    m = box_mesh((14, 11, 9), seed=3, rcm=2)
    rng = np.random.default_rng(2)
    st = torch.cuda.Stream()
    x = torch.from_numpy(rng.uniform(-1.0, 1.0, (m.nnode, 5))).cuda()
    z = torch.empty_like(x)
    torch.cuda.synchronize()

    def context():
        s = Euler3DGPU(m, default_params(), stream=st.cuda_stream)
        IA, JA, IAU = s.get_block_pattern()
        g = np.random.default_rng(6)
        A = g.uniform(-1.0, 1.0, (len(JA), 5, 5)) / (5.0 * np.repeat(np.diff(IA), np.diff(IA)))[:, None, None]
        A[IAU] += 5.0 * np.eye(5)
        s.set_system(A.reshape(-1, 25), g.uniform(-1.0, 1.0, (m.nnode, 5)))
        return s

    def apply(s, kind, precision):
        s.solve_gmres(restart=4, max_iters=1, rtol=1e-14, precond=kind, precision=precision, allow_not_converged=True)
        s.precond_apply_device(x.data_ptr(), z.data_ptr())
        s.synchronize()
        return z.cpu().numpy()

    want = {}
    for key in set(sequence):
        with context() as s:
            want[key] = apply(s, *key)
    with context() as s:
        for key in sequence:
            assert np.array_equal(apply(s, *key), want[key])
