"""Kernels that need more shared memory than a launch has by default, in a process with several contexts
(as with environments on two devices): the raised limit is a property of a function on one device, so
every environment has to raise it where it lives before its first launch. A program steps one environment
in the device's primary context and one in a context of its own; its linker hands it every call that
raises a limit and every launch, and each launch above 48 KB must follow a raise in the same context. The
two steps must succeed and give the same bits. The heights of the two-sweep kernels that need as much, each
in a process of its own."""
import glob
import os
import subprocess

import pytest

from skewtcloudsim_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "skewt.h"

// ---- the raised limits and the launches, by context
#include <map>
#include <utility>
static std::map<std::pair<CUcontext, const void*>, int> raised;
static int big = 0, bare = 0;
static CUcontext here() { CUcontext c = nullptr; cuCtxGetCurrent(&c); return c; }
static void launched(const void* f, size_t smem) {
    if (smem <= 48 * 1024) return;
    ++big;
    const auto it = raised.find({here(), f});
    if (it == raised.end() || size_t(it->second) < smem) ++bare;
}
extern "C" {
cudaError_t __real_cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v);
cudaError_t __wrap_cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    const cudaError_t r = __real_cudaFuncSetAttribute(f, a, v);
    if (r == cudaSuccess && a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        cudaKernel_t k = nullptr;  // what <<<>>> passes to the runtime
        cudaGetKernel(&k, f);
        raised[{here(), f}] = raised[{here(), (const void*)k}] = v;
    }
    return r;
}
cudaError_t __real___cudaLaunchKernel(cudaKernel_t f, dim3 g, dim3 b, void** p, size_t m, cudaStream_t s);
cudaError_t __wrap___cudaLaunchKernel(cudaKernel_t f, dim3 g, dim3 b, void** p, size_t m, cudaStream_t s) {
    launched((const void*)f, m);
    return __real___cudaLaunchKernel(f, g, b, p, m, s);
}
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** p);
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** p) {
    launched(f, c->dynamicSmemBytes);
    return __real_cudaLaunchKernelExC(c, f, p);
}
cudaError_t __real_cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** p, size_t m, cudaStream_t s);
cudaError_t __wrap_cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** p, size_t m, cudaStream_t s) {
    launched(f, m);
    return __real_cudaLaunchCooperativeKernel(f, g, b, p, m, s);
}
}

static int run(int rows, std::vector<float>& th) {
    const int X = 64, Y = 32, Z = 32, N = X * Y * Z;
    skt_grid_desc g{};
    g.nx = X; g.ny = Y; g.nz = Z; g.voxel = 100.0f;
    skt_env* env = nullptr;
    if (skt_create(&g, nullptr, &env) != SKT_OK) { std::printf("create: %s\n", skt_last_error(nullptr)); return 1; }
    std::vector<float> t(N), vel(3 * N, 0.0f), qv(N, 0.001f), gT(X * Z, 300.0f), gp(X * Z, 1000.0f), p(N);
    std::vector<int32_t> gh(X * Z, 0);
    for (int z = 0; z < Z; ++z)
        for (int y = 0; y < Y; ++y)
            for (int x = 0; x < X; ++x) {
                const int c = x + X * (y + Y * z);
                t[c] = 300.0f + 0.3f * y + 0.01f * ((x * 7 + z * 3) % 11);
                p[c] = 1000.0f - 9.0f * y;
            }
    skt_status st = skt_init(env, t.data(), vel.data(), qv.data(), gT.data(), gp.data(), p.data(), nullptr, gh.data(), 0, 0);
    if (st != SKT_OK) { std::printf("init: %s\n", skt_last_error(env)); return 1; }
    skt_tuning tn{};
    skt_get_tuning(env, &tn);
    tn.diffuse_depth = 2;
    tn.diffuse_rows = rows;
    if (skt_set_tuning(env, &tn) != SKT_OK) { std::printf("tuning: %s\n", skt_last_error(env)); return 1; }
    st = skt_step(env, 0.5f, 1.0f, 1);
    if (st != SKT_OK && st != SKT_NOT_CONVERGED) { std::printf("step: %s\n", skt_last_error(env)); return 1; }
    th.resize(N);
    if (skt_read_field(env, SKT_POTTEMP, 0, th.data(), N) != SKT_OK) { std::printf("read: %s\n", skt_last_error(env)); return 1; }
    skt_destroy(env);
    return 0;
}

int main(int, char** argv) {
    const int rows = std::atoi(argv[1]);
    std::vector<float> a, b;
    if (run(rows, a)) return 1;
    CUcontext ctx = nullptr;
    if (cuCtxCreate(&ctx, nullptr, 0, 0) != CUDA_SUCCESS) return 2;  // and current
    if (run(rows, b)) return 3;
    std::printf("%d launches above 48 KB, %d without a raised limit\n", big, bare);
    if (big == 0 || bare > 0) return 5;
    return std::memcmp(a.data(), b.data(), a.size() * 4) ? 4 : 0;
}
"""


@pytest.fixture(scope="module")
def program(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("context")
    src, exe = d / "context.cu", d / "context"
    src.write_text(SOURCE)
    objs = sorted(glob.glob(os.path.join(build.BUILD, "skt_*.o")))
    assert len(objs) == len(build.SOURCES), objs
    wrap = [a for f in ("cudaFuncSetAttribute", "__cudaLaunchKernel", "cudaLaunchKernelExC", "cudaLaunchCooperativeKernel")
            for a in ("-Xlinker", "--wrap=" + f)]
    subprocess.run([build.nvcc(), *wrap, *build.ARCH, "-std=c++17", "-I", os.path.join(build.ROOT, "include"), str(src), *objs, "-lcuda", "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("rows", [6, 8, 14])
def test_step_in_a_second_context(program, rows):
    r = subprocess.run([program, str(rows)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
