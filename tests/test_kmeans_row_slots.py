"""CPU (nvcc alone): the k-means producers start a slot's next copy on a vote whose operand the compiler must not be able to decide, or the
wait for the reads of the slot's rows goes with it.  A branch that the compiler has decided calls nothing, so a call of a function that is
not defined tells whether the operand was left open: the device linker then has something to complain about."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")

SOURCE = """
#include "kmeans_tc.cuh"
__device__ void called_if_open(float* x);
__global__ void probe(float* x, uint32_t never) {
  float any = 0.0f;
  for (int i = 0; i < 2; ++i) any = fmaxf(any, fabsf(x[32 * i + threadIdx.x]));
  if (!(%s)) called_if_open(x);
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no CUDA compiler")
@pytest.mark.parametrize("operand,left_open", [("f2c::tc::arrived(any, never)", True), ("any < 1.0f", True), ("!(any < 0.0f)", False)])
def test_the_vote_on_a_slots_reads_is_not_decided_by_the_compiler(tmp_path, operand, left_open):
    """The kernel's operand; one that depends on the data, as a control; and one that is always true, which must be found out."""
    (tmp_path / "probe.cu").write_text(SOURCE % operand)
    arch = ["-gencode", "arch=compute_100a,code=sm_100a"]
    cmd = [NVCC, "-std=c++17", "-O3", "--expt-relaxed-constexpr", *arch, "-rdc=true", "-I", os.path.join(ROOT, "f2cgt_b200", "csrc"), "-c", "probe.cu", "-o", "probe.o"]
    subprocess.run(cmd, cwd=tmp_path, check=True, capture_output=True, text=True)
    link = subprocess.run([NVCC, *arch, "-dlink", "probe.o", "-o", "linked.o"], cwd=tmp_path, capture_output=True, text=True)
    assert ("called_if_open" in link.stderr + link.stdout) == left_open, link.stderr
    assert (link.returncode != 0) == left_open


def test_the_kernel_votes_with_that_operand():
    text = open(os.path.join(ROOT, "f2cgt_b200", "csrc", "kmeans_tc.cuh")).read()
    assert "if (__all_sync(0xffffffffu, arrived(any, p.never))) fetch(" in text
