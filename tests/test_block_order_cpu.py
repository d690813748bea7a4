"""The order in which freed device blocks go back to their pool, without a GPU: hostio.cu compiled against a CUDA runtime
whose events and waits only record what comes before what, and in which no call waits for the device by itself. A block may
have been used on any context's stream, so every stream's work has to come before it goes back: work of the call that gives
it back, of calls that have returned, of other contexts, on the stream a context had before; a stream that a user's capture
has is left alone."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = r"""
#include <cstdio>
#include <new>

#include "context.cuh"

extern "C" {
void fake_work(cudaStream_t);
void fake_capture(cudaStream_t, int);
int fake_unordered_frees();
int fake_recorded_in_capture();
int fake_blocks();
void fake_reserve(unsigned long long);
}
using namespace simk;

struct Made {  // a context with a stream and a fence: nothing else of it is used
    alignas(Context) unsigned char memory[sizeof(Context)] = {};
    Context& c = reinterpret_cast<Context&>(memory);
    Made() {
        new (&c.fence) std::unique_ptr<StreamFence>();
        cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking);
        device_context_made(c);
    }
};

int main() {
    Made a, b;
    auto say = [&](const char* what) {
        printf("%s %d %d %d\n", what, fake_unordered_frees(), fake_recorded_in_capture(), fake_blocks());
    };
    {
        const ActiveContext active(a.c);
        DeviceBuffer x(1000);
        fake_work(a.c.stream);
    }
    say("in-call");
    DeviceBuffer kept(5000), shared(70000);
    {
        const ActiveContext active(a.c);
        fake_work(a.c.stream);
    }
    kept.release();
    say("after-call");
    {
        const ActiveContext active(b.c);
        fake_work(b.c.stream);
    }
    {
        const ActiveContext active(a.c);
        fake_work(a.c.stream);
        shared.release();
    }
    say("other-context");
    DeviceBuffer moved(300);
    {
        const ActiveContext active(b.c);
        fake_work(b.c.stream);
    }
    device_stream_leaves(b.c);
    cudaStreamCreateWithFlags(&b.c.stream, cudaStreamNonBlocking);
    {
        const ActiveContext active(b.c);
        fake_work(b.c.stream);
    }
    moved.release();
    say("stream-changed");
    fake_capture(a.c.stream, 1);
    {
        const ActiveContext active(a.c);
        DeviceBuffer x(1000);
        fake_work(a.c.stream);
    }
    fake_capture(a.c.stream, 0);
    say("captured");
    {
        const ActiveContext active(a.c);
        fake_work(a.c.stream);
        const ActiveContext inner(b.c);
        fake_work(b.c.stream);
        DeviceBuffer x(1 << 20);
    }
    say("nested");
    device_context_gone(0, std::move(a.c.fence));
    {
        const ActiveContext active(b.c);
        fake_work(b.c.stream);
    }
    DeviceBuffer last(8);
    last.release();
    say("one-gone");
    DeviceBuffer some(1 << 20);
    fake_reserve(3 << 20);
    printf("held %zu\n", device_held_free(0));
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="needs nvcc")
def test_blocks_go_back_behind_every_stream(tmp_path):
    src, exe = str(tmp_path / "order.cu"), str(tmp_path / "order")
    with open(src, "w") as f:
        f.write(SOURCE)
    csrc = os.path.join(ROOT, "simulatokit_b200", "csrc")
    objects = []
    for name in (src, os.path.join(csrc, "hostio.cu")):
        objects.append(str(tmp_path / (os.path.basename(name) + ".o")))
        r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++17", "-c",
                            "--expt-relaxed-constexpr", "-I", csrc, "-I", os.path.join(ROOT, "include"), name, "-o",
                            objects[-1]], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    for args in ([NVCC, "-cudart", "none", "-std=c++17", *objects, os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o",
                  exe], [exe]):
        r = subprocess.run(args, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    *lines, held = [line.split() for line in r.stdout.splitlines()]
    assert held == ["held", str(2 << 20)]  # of what the pool holds, the block in use is not free
    assert [line[0] for line in lines] == ["in-call", "after-call", "other-context", "stream-changed", "captured", "nested",
                                           "one-gone"]
    for what, unordered, recorded_in_capture, blocks in lines:
        assert (unordered, recorded_in_capture) == ("0", "0"), what
    assert [int(line[3]) for line in lines] == [0, 1, 0, 0, 0, 0, 0]
