"""A call that ran out of device memory leaves no buffer behind that counts as allocated: the
same call again fails the same way, or works once there is memory.

The host code is linked against a stand-in for the CUDA runtime that takes device memory
from the heap and can refuse any one allocation; the surrogate's also against launchers
that check the pointers they are given, the energy calls against a launch that does.
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
#include <set>
#include <cuda_runtime.h>

int allocations = 0, refuse = 0, copies = 0;
std::set<void *> freed;

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
cudaError_t cudaFree(void *p) { freed.insert(p); return cudaSuccess; }  // (kept, so that no address comes twice)
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    ++copies;
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


ENERGY = r"""
#include <cstdio>
#include <set>
#include <cuda_runtime.h>
#include "cgppd_cuda_functions.h"

extern int allocations, refuse;
extern std::set<void *> freed;
static int bad = 0, launches = 0;

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **args)
{
    for (int k : {5, 6, 7, 8, 9, 10}) {  // the scratch pointers (partials .. group tickets)
        void *p = *static_cast<void **>(args[k]);
        for (void *f : freed)
            if (p == nullptr || (p >= f && p < static_cast<char *>(f) + 512))
                ++bad;
    }
    ++launches;
    return cudaSuccess;
}

int main()
{
    float4 *p = reinterpret_cast<float4 *>(16);
    float out[1], table[1];
    cudaStream_t st = reinterpret_cast<cudaStream_t>(32);
    auto call = [&](int n) { CUDA_EonDevice_async(p, p, 0, 0, 0, 0, out, 1, 32, n, 0, st); };
    bindLJTexture(table);
    call(1000);
    allocations = 0, refuse = 1;
    call(8000);  // needs more room and is refused it
    refuse = 0;
    call(1000);
    call(8000);
    printf("launches %d bad %d\n", launches, bad);
    return bad != 0 || launches != 3;
}
"""


def compile_and_run(tmp_path, harness, sources):
    try:
        home = build.cuda_home()
    except RuntimeError:
        pytest.skip("no nvcc")
    (tmp_path / "harness.cu").write_text(harness)
    (tmp_path / "runtime.cpp").write_text(RUNTIME)
    exe = str(tmp_path / "harness")
    inc = ["-I" + build.CSRC, "-I" + os.path.join(build.ROOT, "include")]
    subprocess.run([os.path.join(home, "bin", "nvcc"), build.GENCODE, "-std=c++17", "--expt-relaxed-constexpr",
                    "-cudart", "shared"] + inc + ["-o", exe, str(tmp_path / "harness.cu"),
                                                  str(tmp_path / "runtime.cpp")] + sources, check=True)
    env = dict(os.environ, LD_LIBRARY_PATH=os.path.join(home, "lib64"))
    r = subprocess.run([exe], env=env, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_surrogate_after_a_refused_allocation(tmp_path):
    out = compile_and_run(tmp_path, HARNESS, [os.path.join(build.CSRC, f) for f in ("surrogate_host.cu", "status.cpp")])
    assert "0 1: -1" in out and "1 1: -1" in out  # the stand-in did refuse


def test_energy_call_after_a_refused_allocation(tmp_path):
    build.build()
    compile_and_run(tmp_path, ENERGY, [os.path.join(build.BUILD, f) for f in
                                       ("cuda_functions.cu.o", "host_amino_acids.cpp.o", "status.cpp.o")])
