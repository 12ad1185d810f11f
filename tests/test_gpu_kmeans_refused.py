"""A cooperative launch that is refused as too large (a context with only a part of the SMs) is made with fewer CTAs, and
its results stay those of the full launch bit for bit.  The refusal is made on the host: a child process runs with a
``cudaLaunchKernelExC`` in front of the runtime's that refuses cooperative grids above a limit and passes on all else."""

import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

FAKE = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
static unsigned limit = 0, refused = 0;
extern "C" void fake_limit(unsigned n) { limit = n, refused = 0; }
extern "C" unsigned fake_refused(void) { return refused; }
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* func, void** args) {
    typedef cudaError_t (*Launch)(const cudaLaunchConfig_t*, const void*, void**);
    static Launch real = reinterpret_cast<Launch>(dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaLaunchKernelExC"));
    for (unsigned i = 0; i < cfg->numAttrs; ++i)
        if (cfg->attrs[i].id == cudaLaunchAttributeCooperative && cfg->attrs[i].val.cooperative && limit && cfg->gridDim.x > limit) {
            ++refused;
            return cudaErrorCooperativeLaunchTooLarge;
        }
    return real(cfg, func, args);
}
"""

CHILD = r"""
import ctypes, os, sys
import torch
from reskv_b200._extension import load_extension
from reskv_b200.synthetic import mixture

fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
ops = load_extension("compression")
# several CTAs per unit, a unit per CTA, several units per CTA, two segments of a unit in a CTA, long segments
for b, h, t in ((1, 8, 8128), (8, 8, 2000), (40, 8, 130), (16, 8, 3000), (1, 1, 20000)):
    k, v = (mixture(b, h, t, seed=i, device="cuda") for i in range(2))
    calls = (lambda: [x for side in ops.kmeans_pair(k, v, 32, 4) for x in side], lambda: ops.kmeans(k, 32, 4, False))
    for call in calls:
        fake.fake_limit(0)
        want = call()
        for limit in (147, 100, 37, 5, 1):
            fake.fake_limit(limit)
            got = call()
            assert all(torch.equal(x, y) for x, y in zip(got, want)), (b, h, t, limit)
        assert fake.fake_refused() > 0  # the last limit is below every grid
print("agree")
"""


def test_refused_launch_gives_the_same_results(tmp_path):
    cuda = Path(os.environ.get("CUDA_HOME") or "/usr/local/cuda")
    if not shutil.which("g++") or not (cuda / "include" / "cuda_runtime_api.h").exists():
        pytest.skip("no compiler or CUDA headers for the fake launch")
    source, fake = tmp_path / "fake.cpp", tmp_path / "fake.so"
    source.write_text(FAKE)
    subprocess.run(["g++", "-shared", "-fPIC", f"-I{cuda / 'include'}", str(source), "-o", str(fake), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(fake), PYTHONPATH=str(ROOT))
    run = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "agree" in run.stdout, run.stdout + run.stderr
