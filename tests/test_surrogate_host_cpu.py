"""What the surrogate's host code launches, against launchers that record it."""
import os

from test_failed_allocation_cpu import build, compile_and_run

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include "cgppd_surrogate.h"
#include "surrogate_internal.h"


extern int copies;
static int rows_fwd = 0, rows_bwd = 0, wgrad = 0, update[3] = {0, 0, 0};

namespace cgppd {
cudaError_t net_set_limits() { return cudaSuccess; }
cudaError_t launch_net_rows(const NetRowsArgs &a, bool backward, int, cudaStream_t)
{
    ++(backward ? rows_bwd : rows_fwd);
    for (int i = 0; a.y && i < a.rows; ++i)
        a.r2[i] = 1.f;
    return cudaSuccess;
}
cudaError_t launch_net_wgrad(const NetWgradArgs &, cudaStream_t) { ++wgrad; return cudaSuccess; }
cudaError_t launch_net_update(const NetUpdateArgs &a, NetUpdateMode mode, cudaStream_t)
{
    ++update[mode];
    *a.loss_sum = 0.f;
    for (int i = 0; i < a.rows; ++i)
        *a.loss_sum += a.r2[i];
    return cudaSuccess;
}
cudaError_t launch_net_copies(const float *, __nv_bfloat16 *, __nv_bfloat16 *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_permutation(int, uint64_t, int *, int *, unsigned long long *, unsigned *, int, cudaStream_t)
{
    return cudaSuccess;
}
}

int main()
{
    cgppd_surrogate *s = cgppd_surrogate_create(1152, 1);
    std::vector<float> X(1152 * 8, 0.5f), y(1152, 1.f), g(cgppd_surrogate_num_params());
    float loss = 0.f;
    auto show = [&](const char *what, int rc) {
        printf("%s: rc %d loss %g rows %d %d wgrad %d update %d %d %d\n", what, rc, loss, rows_fwd, rows_bwd, wgrad,
               update[0], update[1], update[2]);
        rows_fwd = rows_bwd = wgrad = update[0] = update[1] = update[2] = 0;
        loss = 0.f;
    };
    int rc = cgppd_surrogate_loss_grad(s, X.data(), y.data(), 1024, &loss, nullptr);
    show("loss", rc);
    rc = cgppd_surrogate_loss_grad(s, X.data(), y.data(), 1152, &loss, nullptr);
    show("loss of an uneven batch", rc);
    rc = cgppd_surrogate_loss_grad(s, X.data(), y.data(), 1024, &loss, g.data());
    show("gradient", rc);
    copies = 0;
    rc = cgppd_surrogate_loss_grad(s, X.data(), y.data(), 1152, &loss, g.data());
    show("gradient of an uneven batch", rc);
    printf("copies %d\n", copies);
    cgppd_surrogate_destroy(s);
}
"""


def test_launches_of_loss_and_gradient(tmp_path):
    out = compile_and_run(tmp_path, HARNESS, [os.path.join(build.CSRC, f) for f in ("surrogate_host.cu", "status.cpp")])
    assert out.splitlines() == [
        "loss: rc 0 loss 1 rows 1 0 wgrad 0 update 1 0 0",
        "loss of an uneven batch: rc 0 loss 1 rows 1 0 wgrad 0 update 1 0 0",
        "gradient: rc 0 loss 1 rows 0 1 wgrad 1 update 0 1 0",
        "gradient of an uneven batch: rc -1 loss 0 rows 0 0 wgrad 0 update 0 0 0",
        "copies 0",
    ]
