"""An allocation that is refused leaves the array empty (DevArray, dg_internal.h): handles keep
such arrays and grow them by their size, so one that claimed a size without memory would
be used as a null pointer by the next call.  Against a fake cudaMalloc, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
#include "dg_internal.h"
#include <cstdlib>
static size_t limit = 1000;
static int frees = 0;
extern "C" cudaError_t cudaMalloc(void **p, size_t bytes) {
    if (bytes > limit) return cudaErrorMemoryAllocation;   // *p as it was
    *p = malloc(bytes);
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p) {
    frees++;
    free(p);
    return cudaSuccess;
}
#define WANT(c) do { if (!(c)) { printf("line %d: %s\\n", __LINE__, #c); return 1; } } while (0)
int main() {
    dg::DevArray<double> a;
    WANT(a.alloc(1000) == cudaErrorMemoryAllocation && a.p == nullptr && a.n == 0);
    WANT(a.alloc(100) == cudaSuccess && a.p && a.n == 100 && a.bytes() == 800);
    WANT(a.alloc(1000) == cudaErrorMemoryAllocation && a.p == nullptr && a.n == 0 && a.bytes() == 0 && frees == 1);
    limit = 1 << 20;
    WANT(a.alloc(1000) == cudaSuccess && a.p && a.n == 1000);
    WANT(a.alloc(0) == cudaSuccess && a.p == nullptr && a.n == 0 && frees == 2);
    puts("ok");
}
"""


def test_a_refused_array_is_empty(tmp_path):
    (tmp_path / "refused.cpp").write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "gdistger-re_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-isystem", os.path.join(cuda, "include"), str(tmp_path / "refused.cpp"), "-o", str(tmp_path / "refused")],
                   check=True)
    r = subprocess.run([str(tmp_path / "refused")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
