"""A call that ran out of device memory leaves no buffer behind that counts as allocated: the
same call again fails the same way, or works once there is memory.

The surrogate's host code is linked against a stand-in for the CUDA runtime that takes
device memory from the heap and can refuse any one allocation, and against launchers that
check the pointers they are given.
"""
import os
import subprocess
import sys

import pytest

import cgppd_gb300.build  # noqa: F401  (the package also exports a function of that name)

build = sys.modules["cgppd_gb300.build"]

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
#include <cuda_runtime.h>

int allocations = 0, refuse = 0;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = nullptr;
    if (++allocations == refuse)
        return cudaErrorMemoryAllocation;
    *p = calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}
"""

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include "cgppd_surrogate.h"
#include "surrogate_internal.h"

extern int allocations, refuse;  // refuse: which allocation from now on (0: none)
static int bad = 0;

namespace cgppd {
cudaError_t net_set_limits() { return cudaSuccess; }
cudaError_t launch_net_rows(const NetRowsArgs &a, bool backward, int, cudaStream_t)
{
    if (!a.X || !a.P || !a.wtiles || !a.err || (backward ? !a.act || !a.y : !a.o))
        ++bad;
    return cudaSuccess;
}
cudaError_t launch_net_wgrad(const NetWgradArgs &a, cudaStream_t) { bad += !a.act || !a.part; return cudaSuccess; }
cudaError_t launch_net_update(const NetUpdateArgs &a, NetUpdateMode, cudaStream_t)
{
    bad += !a.loss_sum || !a.G;
    return cudaSuccess;
}
cudaError_t launch_net_copies(const float *P, __nv_bfloat16 *, __nv_bfloat16 *, cudaStream_t)
{
    bad += !P;
    return cudaSuccess;
}
cudaError_t launch_permutation(int n, uint64_t, int *perm, int *partner, unsigned long long *place, unsigned *left,
                               int, cudaStream_t)
{
    if (!perm || !partner || !place || !left)
        ++bad;
    else
        memset(perm, 0, n * sizeof(int));
    return cudaSuccess;
}
}

int main()
{
    const int rows = 128, n = 300;
    std::vector<float> X(n * 8, 0.5f), y(n, 1.f), out(n);
    for (int call = 0; call < 2; ++call)         // predict, train
        for (int which = 1; which <= 12; ++which) {
            refuse = 0;
            cgppd_surrogate *s = cgppd_surrogate_create(rows, 1);
            cgppd_surrogate_add_samples(s, X.data(), y.data(), n);
            auto run = [&] {
                return call == 0 ? cgppd_surrogate_predict(s, X.data(), n, out.data())
                                 : cgppd_surrogate_train(s, 1, 1e-3f, 25.f, 0.25f, y.data());
            };
            int rc[3];
            for (int k = 0; k < 2; ++k) {        // the same allocation refused twice
                allocations = 0, refuse = which;
                rc[k] = run();
                if (allocations < which)         // (the call makes fewer)
                    rc[k] = 0;
            }
            allocations = 0, refuse = 0;
            rc[2] = run();
            printf("%d %d: %d %d %d\n", call, which, rc[0], rc[1], rc[2]);
            if (rc[2] != 0)
                ++bad;
            cgppd_surrogate_destroy(s);
        }
    printf("bad %d\n", bad);
    return bad != 0;
}
"""


def test_after_a_refused_allocation(tmp_path):
    try:
        home = build.cuda_home()
    except RuntimeError:
        pytest.skip("no nvcc")
    (tmp_path / "harness.cu").write_text(HARNESS)
    (tmp_path / "runtime.cpp").write_text(RUNTIME)
    exe = str(tmp_path / "harness")
    inc = ["-I" + build.CSRC, "-I" + os.path.join(build.ROOT, "include")]
    subprocess.run([os.path.join(home, "bin", "nvcc"), build.GENCODE, "-std=c++17", "--expt-relaxed-constexpr",
                    "-cudart", "shared"] + inc +
                   ["-o", exe, str(tmp_path / "harness.cu"), str(tmp_path / "runtime.cpp"), os.path.join(build.CSRC, "surrogate_host.cu"),
                    os.path.join(build.CSRC, "status.cpp")], check=True)
    env = dict(os.environ, LD_LIBRARY_PATH=os.path.join(home, "lib64"))
    r = subprocess.run([exe], env=env, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "0 1: -1" in r.stdout and "1 1: -1" in r.stdout  # the stand-in did refuse
