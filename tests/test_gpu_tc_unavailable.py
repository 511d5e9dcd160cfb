"""A build whose grouped GEMM did not get the registers that its warps share out: the library works without that kernel. A
preloaded shim reports another number for every kernel it is asked about."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *attr, const void *func) {
    void *rt = dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD);
    cudaError_t (*real)(struct cudaFuncAttributes *, const void *) = rt ? dlsym(rt, "cudaFuncGetAttributes") : 0;
    cudaError_t e = real ? real(attr, func) : cudaErrorUnknown;
    if (e == cudaSuccess) attr->numRegs = 136;
    return e;
}
"""

SCRIPT = r"""
import sys
import numpy as np
from colibri_b200 import workloads as W
from colibri_b200.backend import Backend, MoeLayer
from tests.util import upload_qt

be = Backend()
assert be.init_devices((0,)) == 1
D, I, E, K, M = 256, 128, 8, 2, 64
lg, x = W.router_logits(M, E, 2), W.activations(M, D, 1)
for fmt, gs in ((4, 32), (2, 0), (7, 0)):
    ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, fmt, gs, 5 + e)] for e in range(E)]
    side = [[e[k] for e in ex] for k in range(3)]
    lay = MoeLayer(be, D, I, E, K, *side, 0, 0, max_rows=M)
    layers, groups = [], []
    for mode in (0, 1, 2):
        be.set_tensor_core(mode)
        layers.append(lay(x, lg)[0].copy())
        ok, y = be.run_expert_group(side[0][:2], side[1][:2], side[2][:2], [40, 24], x, D)
        assert ok
        groups.append(y.copy())
    same = all(np.array_equal(o[0], a) for o in (layers, groups) for a in o)
    assert np.isfinite(layers[0]).all() and np.any(layers[0]) and same == (sys.argv[1] == "without"), (fmt, gs)
    assert be.kernel_status(0) == 0
    lay.free()
be.shutdown()
print("ok")
"""


def run(what, **env):
    r = subprocess.run([sys.executable, "-c", SCRIPT, what], cwd=ROOT, env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
    return r.stderr


def test_the_kernel_is_used_where_it_can_be():
    assert "grouped GEMM" not in run("with")


def test_the_library_works_without_it(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("no host C compiler")
    src, lib = tmp_path / "regs.c", tmp_path / "regs.so"
    src.write_text(SHIM)
    subprocess.check_call(["gcc", "-D_GNU_SOURCE", "-I/usr/local/cuda/include", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"])
    assert "not used" in run("without", LD_PRELOAD=str(lib))
