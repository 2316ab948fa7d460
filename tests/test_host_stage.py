"""When the host entry points page-lock memory (csrc/host_stage.cuh): not when a handle is made, not at its first call,
once at the second; and where it is refused, calls go on with ordinary memory.  The header is host code, compiled here
against a stand-in for the CUDA runtime that counts."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cufcm_fil_b200" / "csrc"

MAIN = r"""
#include "host_stage.cuh"
#include <cstdio>
#include <cstdlib>
static cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
static int locks = 0, frees = 0, refuse = 0, errors_cleared = 0, copies = 0;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    ++locks;
    if (mode != cudaStreamCaptureModeRelaxed) std::exit(5);  // would break a capture in another thread
    if (refuse) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { ++frees; std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    ++copies;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
    const cudaStreamCaptureMode was = mode;
    mode = *m;
    *m = was;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { ++errors_cleared; return cudaSuccess; }
}
int main(int argc, char **argv) {
    refuse = std::atoi(argv[1]);
    const int n = std::atoi(argv[2]);  // floats each way
    const size_t b = sizeof(float) * n;
    cufil::HostStage s;
    if (s.alloc(2 * b) != cudaSuccess) return 1;
    std::printf("%d", locks);
    float *in = static_cast<float *>(std::malloc(b + 1)), *out = static_cast<float *>(std::malloc(b + 1));
    for (int call = 0; call < 4; ++call) {
        for (int i = 0; i < n; ++i) in[i] = call * 1000.0f + i;
        s.open();
        if (s.put(0, in, b / 2, nullptr) || s.put(b / 2, in + n / 2, b - b / 2, nullptr) || s.up(b, nullptr)) return 2;
        for (int i = 0; i < n; ++i) s.at<float>(b)[i] = 2.0f * s.at<float>(0)[i];  // the work
        if (s.down(b, b, nullptr) || s.take(out, b, b, nullptr)) return 3;
        for (int i = 0; i < n; ++i)
            if (out[i] != 2.0f * in[i]) return 4;
        std::printf(" %d", locks);
    }
    s.release();
    if (mode != cudaStreamCaptureModeGlobal) return 6;
    std::printf(" freed %d cleared %d copies %d", frees, errors_cleared, copies);
}
"""


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    d = tmp_path_factory.mktemp("stage")
    (d / "main.cpp").write_text(MAIN)
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1]
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-I", str(CSRC), "-I", str(cuda / "include"), "-x", "c++",
                    str(d / "main.cpp"), "-o", str(d / "stage")], check=True)
    return lambda refuse, n: subprocess.run([str(d / "stage"), str(refuse), str(n)], check=True, capture_output=True,
                                            text=True).stdout


@pytest.mark.parametrize("refuse,n,want", [
    (0, 1000, "0 0 1 1 1 freed 1 cleared 0 copies 8"),       # one copy each way
    (1, 1000, "0 0 1 1 1 freed 0 cleared 1 copies 8"),       # refused once, not asked again
    (0, 1 << 20, "0 0 0 0 0 freed 0 cleared 0 copies 12"),   # above the limit: the arrays as they are
    (0, 0, "0 0 1 1 1 freed 1 cleared 0 copies 0")])         # nothing to copy
def test_page_locking(stage, refuse, n, want):
    assert stage(refuse, n) == want
