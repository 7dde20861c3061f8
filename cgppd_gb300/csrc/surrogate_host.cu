// surrogate_host.cu -- the pair-energy surrogate object: parameters, dataset, training.
//
// Training is plain mini-batch Adam on the mean squared error against targets clipped
// to +-clip kcal/mol (clashes only need to read as "large").  A step is three launches of
// the project's own kernels (mlp_kernels.cu), enqueued without waiting; an epoch's
// losses and the error flag are read once, at its end.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "cgppd_surrogate.h"
#include "devbuf.h"
#include "status.h"
#include "surrogate.cuh"
#include "surrogate_internal.h"


using namespace cgppd;

namespace {

uint64_t splitmix64(uint64_t &s)
{
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

float uniform_pm(uint64_t &s, float a)
{
    const double u = (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0);
    return (float)((2.0 * u - 1.0) * a);
}

// Rows of features staged on the device by one inference launch (2 MB of features).
constexpr int kStageRows = 65536;

}  // namespace

struct cgppd_surrogate {
    int batch = 0;
    int k_split = 0;
    int max_ctas = 1;
    uint64_t seed = 0;
    int adam_t = 0;
    cudaStream_t stream = nullptr;
    // page-locked words the end of a call is read through: error flag, loss sum
    struct Ends {
        unsigned err;
        float loss_sum;
    } *ends = nullptr;

    DevBuf<float> P, G, am, av;
    DevBuf<__nv_bfloat16> Wf, wtiles;
    // one batch: inputs, tile images and partial gradient sums (k_net_rows, k_net_wgrad)
    DevBuf<float> X, y, xb, dO, r2, wpart, losses;
    DevBuf<__nv_bfloat16> act;
    DevBuf<unsigned> err;
    // inference: staged features and predictions of up to kStageRows rows
    DevBuf<float> stageX, stageO;
    // dataset
    DevBuf<float> dsX, dsY;
    DevBuf<int> perm, partner;
    DevBuf<unsigned long long> place;
    DevBuf<unsigned> left;
    std::vector<float> hX, hY;   // host mirror of the dataset (appended by collect/set)
    bool ds_dirty = true;

    ~cgppd_surrogate()
    {
        if (stream)
            cudaStreamDestroy(stream);
        if (ends)
            cudaFreeHost(ends);
    }

    int init(int b, uint64_t sd)
    {
        batch = b;
        seed = sd;
        k_split = std::min(batch, 1024);
        int dev = 0;
        if (cgppd_check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "surrogate stream") != 0 ||
            cgppd_check(cudaMallocHost(&ends, sizeof(Ends)), "surrogate result words") != 0 ||
            cgppd_check(cudaGetDevice(&dev), "surrogate device") != 0 ||
            cgppd_check(cudaDeviceGetAttribute(&max_ctas, cudaDevAttrMultiProcessorCount, dev), "surrogate device") != 0 ||
            cgppd_check(net_set_limits(), "surrogate shared-memory limits") != 0)
            return -1;
        const size_t tiles = (size_t)batch / kNetRows;
        if (P.zero(kSurParamsPad) || G.zero(kSurParamsPad) || am.zero(kSurParamsPad) || av.zero(kSurParamsPad) ||
            Wf.alloc(3 * kSurH * kSurH) || wtiles.alloc(6 * kSurH * kSurH) || X.zero((size_t)batch * kSurIn) ||
            y.zero(batch) || act.alloc(kActKinds * tiles * kNetTileElems) || xb.alloc((size_t)batch * kSurIn) ||
            dO.alloc(batch) || r2.alloc(batch) || wpart.alloc((size_t)3 * (batch / k_split) * kSurH * kSurH) || losses.zero(1) || err.zero(1))
            return -1;
        // PyTorch-Linear-style initialisation: U(-1/sqrt(fan_in), 1/sqrt(fan_in))
        std::vector<float> p(kSurParamsPad, 0.f);
        uint64_t s = seed ^ 0x5EED5EEDull;
        auto fill = [&](int off, int count, int fan_in) {
            const float a = 1.0f / std::sqrt((float)fan_in);
            for (int i = 0; i < count; ++i)
                p[off + i] = uniform_pm(s, a);
        };
        fill(kOffW1, kSurH * kSurIn, kSurIn);
        fill(kOffB1, kSurH, kSurIn);
        for (int l = 2; l <= 4; ++l) {
            fill(sur_w_off(l), kSurH * kSurH, kSurH);
            fill(sur_b_off(l), kSurH, kSurH);
        }
        fill(kOffW5, kSurH, kSurH);
        fill(kOffB5, 1, kSurH);
        return set_params(p.data());
    }

    int set_params(const float *host)
    {
        if (cgppd_check(cudaMemcpyAsync(P.ptr, host, kSurParams * sizeof(float), cudaMemcpyHostToDevice, stream),
                        "surrogate params") ||
            cgppd_check(launch_net_copies(P.ptr, Wf.ptr, wtiles.ptr, stream), "surrogate bf16 copies"))
            return -1;
        return cgppd_check(cudaStreamSynchronize(stream), "surrogate bf16 copies");
    }

    // Enqueue predictions of n rows of device features.
    int enqueue_forward(const float *dX, int n, float *dO)
    {
        NetRowsArgs r{};
        r.X = dX;
        r.rows = n;
        r.P = P.ptr;
        r.wtiles = wtiles.ptr;
        r.o = dO;
        r.err = err.ptr;
        return cgppd_check(launch_net_rows(r, false, max_ctas, stream), "surrogate forward pass");
    }

    // The weight gradients of n rows are summed over whole splits of them.
    int check_splits(int n) const
    {
        const int ks = std::min(n, k_split);
        if (n % ks != 0 || ks % 64 != 0)
            return cgppd_fail("surrogate: batch must be a multiple of 64 (and of the split size)");
        return 0;
    }

    // Enqueue the loss sum over n rows (n % 128 == 0, n <= batch) into *loss and, with
    // `grad`, their gradient: into G, or straight into an Adam step of rate `lr` (lr > 0).
    // `rows_of` (with `grad`): the batch's rows of dX / dY (targets clipped), or null for rows
    // 0 .. n - 1.
    int enqueue_step(const float *dX, const float *dY, const int *rows_of, float clip, int n, bool grad, float lr,
                     float *loss)
    {
        const int ks = std::min(n, k_split);
        if (grad && check_splits(n))
            return -1;
        const int tiles = (n + kNetRows - 1) / kNetRows;
        NetRowsArgs r{};
        r.X = dX;
        r.y = dY;
        r.perm = rows_of;
        r.clip = clip;
        r.rows = n;
        r.P = P.ptr;
        r.wtiles = wtiles.ptr;
        r.act = act.ptr;
        r.xb = xb.ptr, r.dO = dO.ptr, r.r2 = r2.ptr;
        r.err = err.ptr;
        if (cgppd_check(launch_net_rows(r, grad, max_ctas, stream), "surrogate forward and backward pass"))
            return -1;
        NetUpdateArgs u{};
        u.wpart = wpart.ptr;
        u.splits = n / ks;
        u.act = act.ptr;
        u.xb = xb.ptr, u.dO = dO.ptr, u.r2 = r2.ptr;
        u.rows = n;
        u.G = G.ptr;
        u.loss_sum = loss;
        if (!grad)
            return cgppd_check(launch_net_update(u, kNetLossOnly, stream), "surrogate loss");
        NetWgradArgs w{};
        w.act = act.ptr;
        w.tiles = tiles;
        w.splits = u.splits;
        w.split_tiles = ks / kNetRows;
        w.part = wpart.ptr;
        w.err = err.ptr;
        if (cgppd_check(launch_net_wgrad(w, stream), "surrogate weight gradients"))
            return -1;
        if (lr > 0.f) {
            ++adam_t;
            u.P = P.ptr, u.m = am.ptr, u.v = av.ptr;
            u.lr = lr, u.b1 = 0.9f, u.b2 = 0.999f, u.eps = 1e-8f;
            u.c1 = 1.f - std::pow(u.b1, (float)adam_t), u.c2 = 1.f - std::pow(u.b2, (float)adam_t);
            u.Wf = Wf.ptr, u.wtiles = wtiles.ptr;
        }
        return cgppd_check(launch_net_update(u, lr > 0.f ? kNetAdam : kNetGradient, stream), "surrogate update");
    }

    // Wait for the stream and report a GEMM that gave up; the loss sum at `loss` (if any)
    // is in ends->loss_sum afterwards.
    int finish(const float *loss = nullptr)
    {
        if (cgppd_check(cudaMemcpyAsync(&ends->err, err.ptr, sizeof(unsigned), cudaMemcpyDeviceToHost, stream), "err") ||
            (loss && cgppd_check(cudaMemcpyAsync(&ends->loss_sum, loss, sizeof(float), cudaMemcpyDeviceToHost, stream),
                                 "loss")) ||
            cgppd_check(cudaStreamSynchronize(stream), "surrogate sync"))
            return -1;
        if (ends->err)
            return cgppd_fail("surrogate: a tensor-core GEMM timed out waiting for its MMAs");
        return 0;
    }

    int upload_dataset()
    {
        if (!ds_dirty)
            return 0;
        if (dsX.upload(hX) || dsY.upload(hY))
            return -1;
        ds_dirty = false;
        return 0;
    }

    // predictions for n rows of features (host or device memory), kStageRows at a time
    int predict(const float *Xsrc, int n, float *out_host)
    {
        const int chunk = std::min(n, kStageRows);
        if (n > 0 && (stageX.reserve((size_t)chunk * kSurIn) || stageO.reserve(chunk)))
            return -1;
        for (int s0 = 0; s0 < n; s0 += chunk) {
            const int cnt = std::min(chunk, n - s0);
            if (cgppd_check(cudaMemcpyAsync(stageX.ptr, Xsrc + (size_t)s0 * kSurIn,
                                            (size_t)cnt * kSurIn * sizeof(float), cudaMemcpyDefault, stream),
                            "features") ||
                enqueue_forward(stageX.ptr, cnt, stageO.ptr) ||
                cgppd_check(cudaMemcpyAsync(out_host + s0, stageO.ptr, cnt * sizeof(float), cudaMemcpyDeviceToHost,
                                            stream),
                            "predictions") ||
                finish())
                return -1;
        }
        return 0;
    }
};

// ------------------------------------------------------------------ C ABI

extern "C" {

cgppd_surrogate *cgppd_surrogate_create(int batch, unsigned long long seed)
{
    if (batch <= 0 || batch % 128 != 0) {
        cgppd_fail("cgppd_surrogate_create: batch must be a positive multiple of 128");
        return nullptr;
    }
    auto *s = new cgppd_surrogate();
    if (s->init(batch, seed) != 0) {
        delete s;
        return nullptr;
    }
    return s;
}

void cgppd_surrogate_destroy(cgppd_surrogate *s) { delete s; }

int cgppd_surrogate_num_params(void) { return kSurParams; }

int cgppd_surrogate_get_params(cgppd_surrogate *s, float *out)
{
    if (!s || !out)
        return cgppd_fail("cgppd_surrogate_get_params: null argument");
    return cgppd_check(cudaMemcpy(out, s->P.ptr, kSurParams * sizeof(float), cudaMemcpyDeviceToHost), "get params");
}

int cgppd_surrogate_set_params(cgppd_surrogate *s, const float *in)
{
    if (!s || !in)
        return cgppd_fail("cgppd_surrogate_set_params: null argument");
    return s->set_params(in);
}

int cgppd_surrogate_loss_grad(cgppd_surrogate *s, const float *X, const float *y, int n, float *loss, float *grad)
{
    if (!s || !X || !y)
        return cgppd_fail("cgppd_surrogate_loss_grad: null argument");
    if (n <= 0 || n > s->batch || n % 128 != 0)
        return cgppd_fail("cgppd_surrogate_loss_grad: n must be a multiple of 128 no larger than the batch");
    if (grad && s->check_splits(n))  // (before copies from the caller's memory are under way)
        return -1;
    if (cgppd_check(cudaMemcpyAsync(s->X.ptr, X, (size_t)n * kSurIn * sizeof(float), cudaMemcpyHostToDevice, s->stream),
                    "X") ||
        cgppd_check(cudaMemcpyAsync(s->y.ptr, y, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, s->stream), "y") ||
        s->enqueue_step(s->X.ptr, s->y.ptr, nullptr, 0.f, n, grad != nullptr, 0.f, s->losses.ptr))
        return -1;
    if (grad && cgppd_check(cudaMemcpyAsync(grad, s->G.ptr, kSurParams * sizeof(float), cudaMemcpyDeviceToHost,
                                            s->stream),
                            "grad"))
        return -1;
    if (s->finish(s->losses.ptr))
        return -1;
    if (loss)
        *loss = s->ends->loss_sum / (float)n;
    return 0;
}

int cgppd_surrogate_predict(cgppd_surrogate *s, const float *X, int n, float *out)
{
    if (!s || (!X && n > 0) || (!out && n > 0))
        return cgppd_fail("cgppd_surrogate_predict: null argument");
    return s->predict(X, n, out);
}

int cgppd_surrogate_add_samples(cgppd_surrogate *s, const float *X, const float *y, int n)
{
    if (!s || n < 0 || (n > 0 && (!X || !y)))
        return cgppd_fail("cgppd_surrogate_add_samples: bad argument");
    s->hX.insert(s->hX.end(), X, X + (size_t)n * kSurIn);
    s->hY.insert(s->hY.end(), y, y + n);
    s->ds_dirty = true;
    return 0;
}

int cgppd_surrogate_clear_samples(cgppd_surrogate *s)
{
    if (!s)
        return cgppd_fail("cgppd_surrogate_clear_samples: null surrogate");
    s->hX.clear();
    s->hY.clear();
    s->ds_dirty = true;
    return 0;
}

long long cgppd_surrogate_num_samples(cgppd_surrogate *s) { return s ? (long long)s->hY.size() : -1; }

int cgppd_surrogate_get_samples(cgppd_surrogate *s, float *X, float *y, long long n)
{
    if (!s || n > (long long)s->hY.size())
        return cgppd_fail("cgppd_surrogate_get_samples: bad argument");
    std::memcpy(X, s->hX.data(), (size_t)n * kSurIn * sizeof(float));
    std::memcpy(y, s->hY.data(), (size_t)n * sizeof(float));
    return 0;
}

// Train on the first (1 - val_fraction) of the samples (in their stored order, which
// the collector already randomises), `epochs` passes in a seeded shuffled order.
// history[2 * e] = training RMSE of epoch e (clipped targets, running over its
// batches), history[2 * e + 1] = RMSE on the held-out samples with |y| <= clip.
int cgppd_surrogate_train(cgppd_surrogate *s, int epochs, float lr, float clip, float val_fraction, float *history)
{
    if (!s || epochs < 0 || !(lr > 0.f) || !(clip > 0.f) || val_fraction < 0.f || val_fraction >= 1.f)
        return cgppd_fail("cgppd_surrogate_train: bad argument");
    const long long total = (long long)s->hY.size();
    const long long nval = (long long)(val_fraction * (double)total);
    const long long ntrain = total - nval;
    const int B = s->batch;
    if (ntrain < B)
        return cgppd_fail("cgppd_surrogate_train: fewer training samples than one batch");
    if (s->upload_dataset())
        return -1;
    if (ntrain > INT32_MAX)
        return cgppd_fail("cgppd_surrogate_train: too many samples");
    if (s->perm.reserve(ntrain) || s->partner.reserve(ntrain) || s->place.reserve(ntrain) || s->left.reserve(3))
        return -1;
    uint64_t rs = s->seed ^ 0x7A11ull;
    const long long nb = ntrain / B;
    if (s->losses.reserve(nb))
        return -1;
    for (int e = 0; e < epochs; ++e) {
        // the order of a sequential shuffle with splitmix64(rs), drawn on the device
        if (cgppd_check(launch_permutation((int)ntrain, rs, s->perm.ptr, s->partner.ptr, s->place.ptr, s->left.ptr,
                                           s->max_ctas, s->stream),
                        "permutation"))
            return -1;
        rs += (uint64_t)(ntrain - 1) * 0x9E3779B97F4A7C15ull;
        for (long long b = 0; b < nb; ++b)
            if (s->enqueue_step(s->dsX.ptr, s->dsY.ptr, s->perm.ptr + b * B, clip, B, true, lr, s->losses.ptr + b))
                return -1;
        std::vector<float> sums(nb);
        if (cgppd_check(cudaMemcpyAsync(sums.data(), s->losses.ptr, nb * sizeof(float), cudaMemcpyDeviceToHost,
                                        s->stream),
                        "training losses") ||
            s->finish())
            return -1;
        double sse = 0.0;  // every 16th batch and the last
        long long nlog = 0;
        for (long long b = 0; b < nb; ++b)
            if (b == nb - 1 || b % 16 == 0) {
                sse += (double)(sums[b] / (float)B);
                ++nlog;
            }
        if (history) {
            history[2 * e] = (float)std::sqrt(sse / (double)std::max(1ll, nlog));
            history[2 * e + 1] = -1.f;
        }
        if (history && nval > 0) {
            std::vector<float> pred(nval);
            if (s->predict(s->dsX.ptr + ntrain * kSurIn, (int)nval, pred.data()))
                return -1;
            double se = 0.0;
            long long cnt = 0;
            for (long long i = 0; i < nval; ++i) {
                const float yt = s->hY[ntrain + i];
                if (std::fabs(yt) <= clip) {
                    se += (double)(pred[i] - yt) * (double)(pred[i] - yt);
                    ++cnt;
                }
            }
            history[2 * e + 1] = cnt ? (float)std::sqrt(se / (double)cnt) : -1.f;
        }
    }
    return 0;
}

}  // extern "C"

namespace cgppd {
const float *surrogate_device_params(const cgppd_surrogate *s) { return s ? s->P.ptr : nullptr; }
const __nv_bfloat16 *surrogate_device_wf(const cgppd_surrogate *s) { return s ? s->Wf.ptr : nullptr; }
int surrogate_append_device_samples(cgppd_surrogate *s, const float *dX, const float *dY, int n)
{
    std::vector<float> x((size_t)n * kSurIn), y(n);
    if (cgppd_check(cudaMemcpy(x.data(), dX, x.size() * sizeof(float), cudaMemcpyDeviceToHost), "samples") ||
        cgppd_check(cudaMemcpy(y.data(), dY, y.size() * sizeof(float), cudaMemcpyDeviceToHost), "samples"))
        return -1;
    return cgppd_surrogate_add_samples(s, x.data(), y.data(), n);
}
}  // namespace cgppd
