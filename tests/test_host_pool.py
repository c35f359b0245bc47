"""The host threads that gather pageable input: where the system has no room for them
the pool works with fewer, or with the calling thread alone.  The class is compiled
by itself and run with too little address space for its threads' stacks."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = """
#include <condition_variable>
#include <cstdio>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>
%s
int main() {
    HostPool pool(15);
    int sum = 0;
    std::mutex mu;
    for (int round = 0; round < 3; ++round)
        pool.run(100, [&](int i) {
            std::lock_guard<std::mutex> g(mu);
            sum += i;
        });
    std::printf("%%d\\n", sum);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
@pytest.mark.parametrize("room_kb", [0, 120000, 60000])
def test_pool_without_room_for_its_threads(tmp_path, room_kb):
    with open(os.path.join(ROOT, "knn-cuda_b200", "csrc", "knn_api.cu")) as f:
        src = f.read()
    start = src.index("class HostPool {")
    cls = src[start:src.index("\n};\n", start) + 4]
    (tmp_path / "pool.cpp").write_text(MAIN % cls)
    exe = str(tmp_path / "pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-o", exe, str(tmp_path / "pool.cpp")],
                   check=True)
    limit = f"ulimit -s 8192 && ulimit -v {room_kb} && " if room_kb else ""
    run = subprocess.run(["bash", "-c", limit + exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == str(3 * 4950), run.stdout + run.stderr
