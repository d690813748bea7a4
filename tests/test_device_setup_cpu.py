"""Launch set-up on a process with several devices, without a GPU: the launchers of the line transforms and of the two-pass
passes, compiled against a CUDA runtime that only records, run on device 0, on device 1 and on both again. The opt-in to
shared memory above 48 KB belongs to the device it was asked for on, so each device needs its own, once."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = """
#include "linefft_kernels.cuh"
#include "twopass_kernels.cuh"

namespace simk {
void* device_alloc(size_t, size_t*, int*) { return nullptr; }
void device_free(void*, size_t, int) {}
const float2* twopass_table(Context&, int, long long) { return nullptr; }
CUtensorMap encode_tensor_map_2d(const void*, unsigned long long, unsigned long long, unsigned, unsigned) { return {}; }
CUtensorMap encode_tensor_map_2d(void*, unsigned long long, unsigned long long, unsigned, unsigned) { return {}; }
}
extern "C" {
int fake_launches();
int fake_refused();
int fake_most_opt_ins();
}
using namespace simk;

void launches_on(int device) {
    cudaSetDevice(device);
    alignas(Context) static unsigned char memory[sizeof(Context)];  // no member that the launchers read needs its constructor
    Context& c = reinterpret_cast<Context&>(memory);
    c.sm_count = 148;
    try {
        LineArgs<float2> line{};
        line.lines = 1024;
        line.n = line.ny = 1024;
        line.scale = 1.0f;
        launch_line<1024, false, float2>(line, true, nullptr);
        launch_line<1024, false, float2>(line, false, nullptr);
    } catch (...) {
    }
    try {
        launch_two_rows<512>(c, nullptr, nullptr, nullptr, 512, 512, 1, 1, 1.0f);
    } catch (...) {
    }
    try {
        TwoPassCols a;
        a.ny = 512;
        a.count = 64;
        launch_two_cols_m<512, 0>(c, nullptr, a, nullptr);
    } catch (...) {
    }
}
int main() {
    for (int device : {0, 1, 0, 1, 3}) {
        launches_on(device);
        printf("%d %d\\n", fake_refused(), fake_launches());
    }
    printf("%d\\n", fake_most_opt_ins());
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="needs nvcc")
def test_every_device_gets_its_own_set_up(tmp_path):
    src, obj, exe = (str(tmp_path / name) for name in ("setup.cu", "setup.o", "setup"))
    with open(src, "w") as f:
        f.write(SOURCE)
    for args in ([NVCC, "-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++17", "-c",
                  "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "simulatokit_b200", "csrc"), "-I",
                  os.path.join(ROOT, "include"), src, "-o", obj],
                 [NVCC, "-cudart", "none", "-std=c++17", obj, os.path.join(ROOT, "tests", "fake_cudart.cpp"),
                  "-o", exe], [exe]):
        r = subprocess.run(args, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == "0 4 0 8 0 12 0 16 0 20 1".split()
