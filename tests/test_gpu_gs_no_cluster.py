"""Block Gauss-Seidel where the sweep's cluster cannot be resident (a
partitioned GPU): the sweeps take a launch per level and equal the oracle's bit
for bit.  The runtime's answers are faked in a child process: no cluster fits,
and a launch that asks for one fails."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from cfdsolutions_b200 import box_mesh
from oracle import restatement

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <cuda_runtime_api.h>
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c) {
    (void)f; (void)c;
    *n = 0;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    for (unsigned k = 0; k < c->numAttrs; k++)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) return cudaErrorLaunchOutOfResources;
    cudaError_t (*real)(const cudaLaunchConfig_t *, const void *, void **) = dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    return real(c, f, args);
}
"""

CHILD = """
import sys
import numpy as np
from cfdsolutions_b200 import Euler3DGPU, box_mesh, default_params
z = np.load(sys.argv[1])
with Euler3DGPU(box_mesh((9, 8, 7), seed=3, rcm=2), default_params()) as s:
    s.set_system(z["A"].reshape(-1, 25), z["B"])
    out = {}
    for d in (0, 1, 2):
        out["rms%d" % d] = s.MC_Iterative_Block_LU_Jacobi_CRS(7, d)
        out["X%d" % d] = s.get_system()[2]
np.savez(sys.argv[2], **out)
"""


def test_sweeps_without_a_resident_cluster(gpu_available, tmp_path):
    m = box_mesh((9, 8, 7), seed=3, rcm=2)
    n = m.nnode
    rs = restatement.Session(m, {})
    rng = np.random.default_rng(4)
    A = rng.uniform(-1.0, 1.0, (len(rs.JA), 5, 5)) / (5.0 * np.repeat(np.diff(rs.IA), np.diff(rs.IA)))[:, None, None]
    A[rs.IAU] += 3.0 * np.eye(5)
    B = rng.uniform(-1.0, 1.0, (n, 5))
    (tmp_path / "fake.c").write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", str(tmp_path / "fake.so"),
                    str(tmp_path / "fake.c"), "-ldl"], check=True)
    np.savez(tmp_path / "in.npz", A=A, B=B)
    env = dict(os.environ, LD_PRELOAD=str(tmp_path / "fake.so"), PYTHONPATH=str(ROOT))
    subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "in.npz"), str(tmp_path / "out.npz")], check=True,
                   env=env, cwd=ROOT, timeout=300)
    z = np.load(tmp_path / "out.npz")
    for d in (0, 1, 2):
        X, rms = rs.block_gs(A, B, 7, d)
        assert np.array_equal(z[f"X{d}"], X)
        assert abs(float(z[f"rms{d}"]) - rms) <= n * 1.2e-16 * abs(rms)
