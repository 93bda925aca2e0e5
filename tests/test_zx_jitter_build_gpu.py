"""The tensor-core kernels once more in a build that disturbs their timing.

Compiled with ``-DTFF_JITTER=<ns>`` every arrival at an mbarrier and every return from a wait is held back, one
time in three, by a pseudo-random pause (csrc/tcgen05.cuh), and so is every warp behind a barrier of the few-row tile
attention.  Warps that usually keep step then fall out of it by more than a pipeline stage, and a kernel that relied
on the usual timing fails at once: the prompt attention
whose four softmax warps shared one counted barrier for "probabilities written" passed these tests in the normal
build nearly always and fails ten of thirteen of them in this one.  The library is built into a temporary folder
(half a minute) and the kernel tests run against it in a process of their own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SELECT = ("prompt_attention or flash_attention or gemm_tc or qkv_projection or norm_gate_up or gate_up_product "
          "or gemm_swiglu or attention_at_long_context or far_key or window_edge or attention_of_few_rows or gemm_f32 "
          "or portions_and_decoded_tokens or attention_over_plain_rows")
FILES = ("test_kernels_gpu.py", "test_dominex_gpu.py", "test_kadodra_gpu.py")


def test_kernel_tests_pass_with_disturbed_timing(tmp_path):
    env = dict(os.environ, TFFINFER_NVCC_FLAGS="-DTFF_JITTER=3000", TFFINFER_BUILD_DIR=str(tmp_path / "build"))
    build = subprocess.run([sys.executable, "-c", "from tffinfer_b200.csrc import build; build.library_path(verbose=False)"],
                           cwd=ROOT, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900)
    if build.returncode != 0:
        pytest.skip("the jitter build could not be compiled here: " + build.stdout[-400:])
    run = subprocess.run([sys.executable, "-m", "pytest", *(os.path.join(ROOT, "tests", f) for f in FILES), "-m", "gpu",
                          "-q", "-x", "-p", "no:cacheprovider", "-k", SELECT],
                         cwd=ROOT, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900)
    tail = run.stdout[-3000:]
    assert run.returncode == 0, "kernel tests failed in the build with disturbed timing:\n" + tail
    assert " passed" in tail and "no tests ran" not in tail, tail
