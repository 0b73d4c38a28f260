"""Which memory the gradient kernel is given: copies of the caller's rows and targets, never the caller's arrays, even
where the device could read them in place (a mapped file cut short would then fault the GPU).  The entry point is
compiled against a stand-in for the CUDA runtime that hands out host memory, and a kernel launch that looks at its
pointers; no GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

from colo import _build

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "colo_host.h"
#include "colo_mlp.h"
static const float *g_x, *g_t;
static uint64_t g_n;
static int g_bad = 1;
extern "C" {
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
namespace colo {
colo_status set_err(colo_ctx*, colo_status st, const std::string&) { return st; }
colo_status run_guarded(colo_ctx*, const std::function<colo_status()>& fn) { return fn(); }
void mlp_forward(const float*, const float*, uint64_t, float*, cudaStream_t) {}
void mlp_adam(float*, float*, float*, float*, int, float, cudaStream_t) {}
void mlp_grad(const float*, const float* x, const float* t, const uint32_t*, uint64_t n, float* g, float* l, cudaStream_t) {
    const bool own_x = x + n * kMlpIn <= g_x || x >= g_x + n * kMlpIn, own_t = t + n <= g_t || t >= g_t + n;
    g_bad = !own_x || !own_t || n != g_n || std::memcmp(x, g_x, n * kMlpIn * 4) || std::memcmp(t, g_t, n * 4);
    *l = g[0] = 1.f;
}
}
int main() {
    colo_ctx ctx;
    ctx.host_reads = HOST_READS;
    g_n = 37;
    std::vector<float> x(g_n * colo::kMlpIn), t(g_n), p(colo::kMlpParams), g(colo::kMlpParams);
    for (size_t i = 0; i < x.size(); ++i) x[i] = (float)i;
    for (size_t i = 0; i < t.size(); ++i) t[i] = -(float)i;
    g_x = x.data();
    g_t = t.data();
    float loss = 0;
    const colo_status st = colo_model_grad(&ctx, p.data(), g_x, g_t, g_n, g.data(), &loss);
    return st == COLO_OK && loss == 1.f && g[0] == 1.f && !g_bad ? 0 : 1;
}
"""


@pytest.mark.parametrize("host_reads", ["true", "false"])
def test_gradient_works_on_copies(tmp_path, host_reads):
    inc = Path(_build.nvcc()).resolve().parent.parent / "include"
    src = tmp_path / "rows.cpp"
    src.write_text("#include <cstring>\n" + HARNESS)
    exe = tmp_path / "rows"
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", f"-DHOST_READS={host_reads}", f"-I{_build.CSRC}", f"-I{_build.INCLUDE}",
                    f"-I{inc}", str(src), str(_build.CSRC / "colo_model.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
