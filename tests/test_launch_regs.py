"""The exact kernels' check of their registers before a launch keeps a good answer only:
where the runtime cannot be asked, for once, the next launch asks again.  The
function is compiled by itself, against stand-ins for the two runtime calls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = """
#include <atomic>
#include <cstdio>
constexpr int EX_LAUNCH_REGS = 96, cudaSuccess = 0;
struct cudaFuncAttributes { int numRegs; };
int answers[] = {2, 0, 0}, asked = 0, regs = 96;
int cudaFuncGetAttributes(cudaFuncAttributes *a, void (*)()) {
    a->numRegs = regs;
    return answers[asked++];
}
int cudaGetLastError() { return 0; }
template <int N> void kernel() {}
%s
int main() {
    const bool failed = launch_regs_ok<kernel<1>>(), again = launch_regs_ok<kernel<1>>();
    const bool kept = launch_regs_ok<kernel<1>>();
    const int times = asked;
    regs = 80;
    std::printf("%%d %%d %%d %%d %%d\\n", failed, again, kept, times, launch_regs_ok<kernel<2>>());
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_a_failed_question_is_asked_again(tmp_path):
    with open(os.path.join(ROOT, "knn-cuda_b200", "csrc", "knn_exact_core.cuh")) as f:
        src = f.read()
    start = src.index("template <auto kern>\nbool launch_regs_ok()")
    (tmp_path / "regs.cpp").write_text(MAIN % src[start:src.index("\n}\n", start) + 3])
    exe = str(tmp_path / "regs")
    subprocess.run(["g++", "-std=c++17", "-o", exe, str(tmp_path / "regs.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.split()
    # (asked twice for the first kernel: the failure, then the answer that is kept)
    assert out == ["0", "1", "1", "2", "0"]
