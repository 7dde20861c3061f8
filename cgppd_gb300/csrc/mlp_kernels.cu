// mlp_kernels.cu -- training and batched inference of the pair-energy surrogate.
//
// A training step is three launches: k_net_rows<true> (forward and backward over the
// rows of the mini-batch), k_net_wgrad (the 256 x 256 weight gradients, split over the
// rows) and k_net_update (the partial sums, then Adam and the BF16 copies, or the
// gradient itself).  Inference is k_net_rows<false>.
//
// Every GEMM runs on the tcgen05 tensor cores in BF16 with FP32 accumulation in tensor
// memory.  The hidden width (256 units) is the M side of every product, the rows of the
// batch the N side: one thread then owns one unit (a tensor-memory lane) and walks over
// rows (columns), biases are registers, and a thread's eight consecutive rows are one
// 16-byte piece of an operand.  Activations and activation
// gradients live in one tile image, 256 units x 64 rows (tc05.cuh): as written by the
// epilogue it is the MN-major B operand of the next layer, and, copied to global memory
// in one bulk copy, the K-major A and B operands of the weight gradient (K = rows).  No
// transposed copy is made anywhere.  Layer 1 (K = 8) and the output dot product stay in
// FP32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "surrogate.cuh"
#include "surrogate_internal.h"
#include "tc05.cuh"

namespace cgppd {

namespace {

constexpr int kTileBytes = kNetTileElems * 2;  // 256 x 64 bf16
constexpr int kRowWarps = 16;                  // epilogue warps: one thread per unit and half of the rows
constexpr int kNetThreads = (kRowWarps + 1) * 32;  // and one warp that loads weights and issues MMAs
constexpr int kRing = 4;                       // staged weight chunks: one 256 x 256 layer
constexpr int kNetSmem = (kRing + 2) * kTileBytes + kNetRows * (kSurIn + 2) * 4;
constexpr int kTmemBlock = 2 * kNetRows;       // columns of one product: 2 halves of 128 units x 64 rows
static_assert(kNetSmem <= 227 * 1024, "k_net_rows shared memory");

// Wait limit of the kernels' barriers (polls; a poll suspends the thread for a while).
constexpr long long kPolls = 1ll << 22;

__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// One thread's 16 rows of its unit into a tile image (pieces c, c + 1).
__device__ __forceinline__ void store16(unsigned char *tile, int unit, int c, const uint32_t *w)
{
    *reinterpret_cast<uint4 *>(tile + tc05::tile_offset(unit, c)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4 *>(tile + tc05::tile_offset(unit, c + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
}

// 1 / x on the SFU: relative error at most 2^-23, results below the normal range flushed.
__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// bf16(silu(z)) of 16 values, the same bits as rounding the quotient z / (1 + exp(-z)).
// z times the SFU reciprocal is within 2^-22 of that quotient (2^-23 of the reciprocal, half
// a unit of the product and of the quotient each): four units in the last place.  The two
// therefore round to different BF16 values only where the low 16 bits lie that close to a
// half (0x8000); a pair with such a value (one in 2000; also any for z < -80, where the
// reciprocal nears the end of the normal range) takes the divisions.  A third of the
// division's instructions: the epilogues are bound by issue slots.
__device__ __forceinline__ void silu16(const float *z, uint32_t *w)
{
    // low halves + 0x8008: 0 .. 16 within eight units of the half (the carry into the
    // upper half widens its window by one)
    uint32_t near_half[8], lows = 0xffffffffu;
    float zmin = z[0];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float z0 = z[2 * i], z1 = z[2 * i + 1];
        const float h0 = z0 * rcp_approx(1.0f + __expf(-z0)), h1 = z1 * rcp_approx(1.0f + __expf(-z1));
        w[i] = pack_bf16(h0, h1);
        near_half[i] = __byte_perm(__float_as_uint(h0), __float_as_uint(h1), 0x5410) + 0x80088008u;
        lows = __vminu2(lows, near_half[i]);
        zmin = fminf(zmin, fminf(z0, z1));
    }
    const bool low = zmin < -80.0f;
    if ((lows & 0xffffu) < 18u || lows < (18u << 16) || low) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((near_half[i] & 0xffffu) < 18u || near_half[i] < (18u << 16) || low)
                w[i] = pack_bf16(silu(z[2 * i]), silu(z[2 * i + 1]));
    }
}

// Layer 1 of one row in FP32.
__device__ __forceinline__ float layer1(const float *w1, float b1, const float *x)
{
    const float4 a = *reinterpret_cast<const float4 *>(x), b = *reinterpret_cast<const float4 *>(x + 4);
    float z = b1;
    z = fmaf(w1[0], a.x, z), z = fmaf(w1[1], a.y, z), z = fmaf(w1[2], a.z, z), z = fmaf(w1[3], a.w, z);
    z = fmaf(w1[4], b.x, z), z = fmaf(w1[5], b.y, z), z = fmaf(w1[6], b.z, z), z = fmaf(w1[7], b.w, z);
    return z;
}

// Forward pass of 64-row tiles (BWD: and the whole backward pass down to layer 1, the
// loss being a sum over rows).  One CTA per tile at a time, one CTA per SM: 16 warps run
// the epilogues, the last warp's first thread streams the weights (six 128 KB layers
// from L2 through a ring of four 64-wide K chunks, the next layer's loads under the
// epilogue) and issues the MMAs.  The three forward accumulators stay in tensor memory
// for the backward pass, which needs SiLU' of them: no pre-activation goes to memory.
// 64 rows: a batch of 8192 is 128 CTAs.  The MMAs (N = 64) then read shared memory more
// than they compute (32 a layer, about 0.85 us); 128-row tiles would halve that share but
// leave 88 SMs idle and double the epilogues (exp and division of 32 values a thread,
// about 2 us), whose chain bounds the kernel.
template <bool BWD>
__global__ void __launch_bounds__(kNetThreads, 1) k_net_rows(NetRowsArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[kRing], empty[kRing], done[2];
    __shared__ uint32_t tmem_base;
    unsigned char *s_h[2] = {smem + kRing * kTileBytes, smem + (kRing + 1) * kTileBytes};
    float *s_x = reinterpret_cast<float *>(smem + (kRing + 2) * kTileBytes);
    float *s_y = s_x + kNetRows * kSurIn, *s_do = s_y + kNetRows;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const bool mma_warp = warp == kRowWarps;
    // epilogue thread -> unit (tensor-memory lane of one 128-unit half) and row half
    const int quad = warp & 3, uh = (warp >> 2) & 1, rh = (warp >> 3) & 1;
    const int unit = uh * 128 + quad * 32 + lane, row0 = rh * (kNetRows / 2);
    constexpr int kGemms = BWD ? 6 : 3;
    const int ntiles = (a.rows + kNetRows - 1) / kNetRows;
    const int mine = ((int)blockIdx.x < ntiles) ? (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int total = mine * kGemms;

    if (mma_warp) {
        tc05::tmem_alloc(&tmem_base, 512);
        if (lane == 0) {
            for (int c = 0; c < kRing; ++c) {
                tc05::mbar_init(&full[c], 1);
                tc05::mbar_init(&empty[c], 1);
            }
            tc05::mbar_init(&done[0], 1);
            tc05::mbar_init(&done[1], 1);
        }
    }
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(uh * kNetRows + row0);
    int ok = 1;
    int loaded = 0, used = 0, issued = 0;  // the MMA thread's progress, in GEMMs

    auto load_weights = [&](int g) {  // the MMA thread: the four K chunks of GEMM g
        const __nv_bfloat16 *w = a.wtiles + (size_t)(g % kGemms) * kRing * kNetTileElems;
        for (int c = 0; c < kRing; ++c) {
            tc05::mbar_expect(&full[c], kTileBytes);
            tc05::bulk_load(tc05::smem_u32(smem + c * kTileBytes), w + (size_t)c * kNetTileElems, kTileBytes, &full[c]);
        }
        loaded = g + 1;
    };
    // The MMA thread: D[256 units x 64 rows] of GEMM g = weights x the operand tile `h`
    // into tensor-memory block `blk`, one 128-unit half after the other (the first half's
    // epilogue starts under the second half's MMAs), then the next GEMM's weight loads as
    // the chunks come free.  The descriptors are one base plus constants: built per MMA,
    // the issuing thread took 115 cycles an MMA instead of the 50 that reading the
    // operands (6 KB at 128 bytes a cycle) takes.
    const uint64_t wdesc = tc05::desc_k_major(tc05::smem_u32(smem));
    auto gemm = [&](int g, const unsigned char *h, int blk) {
        constexpr uint32_t idesc = tc05::idesc_bf16_f32(128, kNetRows, true);
        const uint64_t hdesc = tc05::desc_mn_major(tc05::smem_u32(h));
        const uint32_t d = tmem + (uint32_t)(blk * kTmemBlock);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
#pragma unroll
            for (int c = 0; c < kRing; ++c) {
                if (half == 0) {
                    ok = (ok && tc05::mbar_wait(&full[c], (uint32_t)(g & 1), kPolls)) ? 1 : 0;
                    tc05::fence_after_sync();
                }
                if (ok)
#pragma unroll
                    for (int kk = 0; kk < tc05::kChunkK / 16; ++kk)
                        tc05::mma_f16(d + (uint32_t)(half * kNetRows),
                                      wdesc + (uint32_t)((c * kTileBytes + half * (kTileBytes / 2) + 256 * kk) >> 4),
                                      hdesc + (uint32_t)((2048 * (c * 4 + kk)) >> 4), idesc, c > 0 || kk > 0);
                if (half == 1 && ok)
                    tc05::mma_commit(&empty[c]);
            }
            if (ok)
                tc05::mma_commit(&done[half]);
        }
        if (!ok) {  // the MMAs issued so far, for the wait at the end
            tc05::mma_commit(&done[1]);
            issued = g + 1;
            return;
        }
        used = issued = g + 1;
        if (g + 1 < total) {
            for (int c = 0; c < kRing && ok; ++c)
                ok = tc05::mbar_wait(&empty[c], (uint32_t)(g & 1), kPolls) ? 1 : 0;
            if (ok)
                load_weights(g + 1);
        }
    };
    // After an epilogue: its operand tile is visible to the tensor cores and bulk copies,
    // every thread knows whether all waits so far ended.
    auto publish = [&]() -> bool {
        tc05::fence_proxy_async();
        tc05::fence_before_sync();
        ok = __syncthreads_and(ok);
        tc05::fence_after_sync();
        return ok != 0;
    };
    auto wait_gemm = [&](int g) {
        if (!mma_warp) {
            ok = tc05::mbar_wait(&done[uh], (uint32_t)(g & 1), kPolls) ? ok : 0;
            tc05::fence_after_sync();
            __syncwarp();
        }
    };
    const bool mma_thread = mma_warp && lane == 0;
    // the tile just published: GEMM g over it, and (BWD) its copy to global memory as
    // tile image `kind` of batch tile `tile`
    auto advance = [&](int g, int buf, int blk, int tile, int kind) {
        if (mma_thread) {
            gemm(g, s_h[buf], blk);
            if (BWD) {
                tc05::bulk_store(a.act + ((size_t)kind * ntiles + tile) * kNetTileElems, tc05::smem_u32(s_h[buf]),
                                 kTileBytes);
                tc05::bulk_store_wait_read();
            }
        }
    };
    // forward epilogue of the accumulator block `blk`: h = silu(acc + bias) into `buf`
    auto forward_epilogue = [&](int blk, float bias, unsigned char *buf) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float v[16];
            tc05::tmem_ld16(lane_base + (uint32_t)(blk * kTmemBlock + q * 16), v);
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 16; ++i)
                v[i] += bias;
            silu16(v, w);
            store16(buf, unit, (row0 >> 3) + 2 * q, w);
        }
    };

    float w1[kSurIn], b1 = 0.f, b2 = 0.f, b3 = 0.f, b4 = 0.f, w5 = 0.f;
    if (!mma_warp) {
#pragma unroll
        for (int i = 0; i < kSurIn; ++i)
            w1[i] = a.P[kOffW1 + unit * kSurIn + i];
        b1 = a.P[kOffB1 + unit], b2 = a.P[kOffB2 + unit], b3 = a.P[kOffB3 + unit], b4 = a.P[kOffB4 + unit];
        w5 = a.P[kOffW5 + unit];
    }
    if (mma_thread && total > 0)
        load_weights(0);

    int g = 0;  // GEMMs so far
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        __syncthreads();  // the previous tile's readers of s_x are done
        if (!mma_warp) {
            const int r = t >> 3, i = t & 7, row = tile * kNetRows + r;
            float x = 0.f;
            if (row < a.rows) {
                const int src = a.perm ? a.perm[row] : row;
                x = a.X[(size_t)src * kSurIn + i];
                if (BWD && i == 0) {
                    const float y = a.y[src];
                    s_y[r] = a.perm ? fminf(a.clip, fmaxf(-a.clip, y)) : y;
                }
            }
            s_x[r * kSurIn + i] = x;
            if (BWD && row < a.rows)
                a.xb[(size_t)i * a.rows + row] = x;
        }
        __syncthreads();
        // ---- layer 1 and the three hidden GEMMs
        if (!mma_warp) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float z[16];
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    z[i] = layer1(w1, b1, s_x + (row0 + q * 16 + i) * kSurIn);
                silu16(z, w);
                store16(s_h[0], unit, (row0 >> 3) + 2 * q, w);
            }
        }
        if (!publish())
            break;
        advance(g, 0, 0, tile, kActH1);
        wait_gemm(g);
        if (!mma_warp)
            forward_epilogue(0, b2, s_h[1]);
        if (!publish())
            break;
        advance(g + 1, 1, 1, tile, kActH1 + 1);
        wait_gemm(g + 1);
        if (!mma_warp)
            forward_epilogue(1, b3, s_h[0]);
        if (!publish())
            break;
        advance(g + 2, 0, 2, tile, kActH1 + 2);
        wait_gemm(g + 2);
        if (!mma_warp)
            forward_epilogue(2, b4, s_h[1]);
        if (!publish())
            break;
        if (BWD && mma_thread)  // (its read of the tile is waited for before the next publish)
            tc05::bulk_store(a.act + ((size_t)(kActH1 + 3) * ntiles + tile) * kNetTileElems, tc05::smem_u32(s_h[1]),
                             kTileBytes);
        // ---- output: warp w takes rows 8 w .. 8 w + 7, lane l the units l, l + 32, ...
        if (warp < kNetRows / 8) {
            float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < kSurH / 32; ++j) {
                const int u = lane + 32 * j;
                const float wu = a.P[kOffW5 + u];
                const uint4 h = *reinterpret_cast<const uint4 *>(s_h[1] + tc05::tile_offset(u, warp));
                s[0] = fmaf(bf16_lo(h.x), wu, s[0]), s[1] = fmaf(bf16_hi(h.x), wu, s[1]);
                s[2] = fmaf(bf16_lo(h.y), wu, s[2]), s[3] = fmaf(bf16_hi(h.y), wu, s[3]);
                s[4] = fmaf(bf16_lo(h.z), wu, s[4]), s[5] = fmaf(bf16_hi(h.z), wu, s[5]);
                s[6] = fmaf(bf16_lo(h.w), wu, s[6]), s[7] = fmaf(bf16_hi(h.w), wu, s[7]);
            }
            float mine_s = 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
                if (lane == q)
                    mine_s = s[q];
            }
            if (lane < 8) {
                const int r = warp * 8 + lane, row = tile * kNetRows + r;
                const float out = mine_s + a.P[kOffB5];
                if (row < a.rows && a.o)
                    a.o[row] = out;
                if (BWD) {
                    const float res = (row < a.rows) ? out - s_y[r] : 0.f;
                    const float d = 2.0f * res / (float)a.rows;
                    s_do[r] = d;
                    if (row < a.rows) {
                        a.dO[row] = d;
                        a.r2[row] = res * res;
                    }
                } else if (a.y && row < a.rows) {
                    const float res = out - a.y[row];
                    a.dO[row] = 2.0f * res / (float)a.rows;
                    a.r2[row] = res * res;
                }
            }
        }
        if (!BWD) {
            g += kGemms;
            continue;
        }
        __syncthreads();
        // ---- backward: dZ4 = (dO w5) silu'(z4), then dZ_l = (W_{l+1}^T dZ_{l+1}) silu'(z_l)
        if (!mma_warp) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float v[16];
                tc05::tmem_ld16(lane_base + (uint32_t)(2 * kTmemBlock + q * 16), v);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    v[i] += b4;
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const float d0 = s_do[row0 + q * 16 + i], d1 = s_do[row0 + q * 16 + i + 1];
                    w[i >> 1] = pack_bf16(d0 * w5 * silu_grad(v[i]), d1 * w5 * silu_grad(v[i + 1]));
                }
                store16(s_h[0], unit, (row0 >> 3) + 2 * q, w);
            }
        }
        if (mma_thread)  // the copy of H4 has read its tile before any warp may pass to writing dZ3 there
            tc05::bulk_store_wait_read();
        if (!publish())
            break;
        auto weighted_slopes = [](const float *v, const float *z, uint32_t *w) {
#pragma unroll
            for (int i = 0; i < 16; i += 2)
                w[i >> 1] = pack_bf16(v[i] * silu_grad(z[i]), v[i + 1] * silu_grad(z[i + 1]));
        };
        auto backward_epilogue = [&](int blk, int zblk, float bias, unsigned char *buf) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float v[16], z[16];
                tc05::tmem_ld16(lane_base + (uint32_t)(blk * kTmemBlock + q * 16), v);
                tc05::tmem_ld16(lane_base + (uint32_t)(zblk * kTmemBlock + q * 16), z);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    z[i] += bias;
                uint32_t w[8];
                weighted_slopes(v, z, w);
                store16(buf, unit, (row0 >> 3) + 2 * q, w);
            }
        };
        advance(g + 3, 0, 3, tile, kActZ1 + 3);
        wait_gemm(g + 3);
        if (!mma_warp)
            backward_epilogue(3, 1, b3, s_h[1]);
        if (!publish())
            break;
        advance(g + 4, 1, 2, tile, kActZ1 + 2);
        wait_gemm(g + 4);
        if (!mma_warp)
            backward_epilogue(2, 0, b2, s_h[0]);
        if (!publish())
            break;
        advance(g + 5, 0, 3, tile, kActZ1 + 1);
        wait_gemm(g + 5);
        if (!mma_warp) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float v[16], z[16];
                tc05::tmem_ld16(lane_base + (uint32_t)(3 * kTmemBlock + q * 16), v);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    z[i] = layer1(w1, b1, s_x + (row0 + q * 16 + i) * kSurIn);
                uint32_t w[8];
                weighted_slopes(v, z, w);
                store16(s_h[1], unit, (row0 >> 3) + 2 * q, w);
            }
        }
        if (!publish())
            break;
        if (mma_thread) {
            tc05::bulk_store(a.act + ((size_t)kActZ1 * ntiles + tile) * kNetTileElems, tc05::smem_u32(s_h[1]),
                             kTileBytes);
            tc05::bulk_store_wait_read();
        }
        g += kGemms;
    }

    ok = __syncthreads_and(ok);
    if (mma_thread) {
        if (!ok) {
            // a wait ran out: report it, and give the copies and MMAs still in flight a
            // second bounded wait before the memory they use is given back
            atomicOr(a.err, 1u);
            if (loaded > used)
                for (int c = 0; c < kRing; ++c)
                    tc05::mbar_wait(&full[c], (uint32_t)((loaded - 1) & 1), kPolls);
            if (issued > 0)
                tc05::mbar_wait(&done[1], (uint32_t)((issued - 1) & 1), kPolls);
        }
        if (BWD)
            tc05::bulk_store_wait_done();
    }
    tc05::fence_before_sync();
    __syncthreads();
    if (mma_warp) {
        tc05::fence_after_sync();
        tc05::tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------ weight gradients

// dW_l[o][i] = sum over rows of dZ_l[o] H_{l-1}[i] for one 128 x 128 quarter of one
// layer and one split of the rows (both operands K-major tiles, K = rows): partial sums
// in FP32.  Splits of 1024 rows: 96 CTAs for a batch of 8192, each 16 chunks of 32 KB
// through a four-stage ring; finer splits read the operands no faster and write more
// partial sums.  Bound by the loads from L2.
constexpr int kWgStages = 4;
constexpr int kWgSmem = kWgStages * kTileBytes;
constexpr int kWgThreads = 160;  // four epilogue warps and the loading / MMA warp

__global__ void __launch_bounds__(kWgThreads) k_net_wgrad(NetWgradArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[kWgStages], empty[kWgStages], done;
    __shared__ uint32_t tmem_base;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int mh = blockIdx.x >> 1, nh = blockIdx.x & 1, layer = blockIdx.y, split = blockIdx.z;
    const int nk = a.split_tiles, k0 = split * nk;
    if (warp == 4) {
        tc05::tmem_alloc(&tmem_base, 128);
        if (lane == 0) {
            for (int c = 0; c < kWgStages; ++c) {
                tc05::mbar_init(&full[c], 1);
                tc05::mbar_init(&empty[c], 1);
            }
            tc05::mbar_init(&done, 1);
        }
    }
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    const uint32_t tmem = tmem_base;
    int ok = 1;
    if (t == 128) {
        constexpr uint32_t idesc = tc05::idesc_bf16_f32(128, 128, false);
        constexpr int kHalf = kNetTileElems / 2;
        const __nv_bfloat16 *A = a.act + ((size_t)(kActZ1 + 1 + layer) * a.tiles + k0) * kNetTileElems + mh * kHalf;
        const __nv_bfloat16 *B = a.act + ((size_t)(kActH1 + layer) * a.tiles + k0) * kNetTileElems + nh * kHalf;
        const uint32_t base = tc05::smem_u32(smem);
        const uint64_t desc0 = tc05::desc_k_major(base);
        auto load = [&](int k) {
            const int s = k % kWgStages;
            tc05::mbar_expect(&full[s], kTileBytes);
            tc05::bulk_load(base + s * kTileBytes, A + (size_t)k * kNetTileElems, kTileBytes / 2, &full[s]);
            tc05::bulk_load(base + s * kTileBytes + kTileBytes / 2, B + (size_t)k * kNetTileElems, kTileBytes / 2,
                            &full[s]);
        };
        int loaded = 0, k = 0;
        for (; loaded < nk && loaded < kWgStages - 1; ++loaded)
            load(loaded);
        for (; k < nk; ++k) {
            const int s = k % kWgStages;
            ok = tc05::mbar_wait(&full[s], (uint32_t)((k / kWgStages) & 1), kPolls) ? 1 : 0;
            if (!ok)
                break;
            tc05::fence_after_sync();
            const uint64_t da = desc0 + (uint32_t)((s * kTileBytes) >> 4), db = da + (uint32_t)(kTileBytes >> 5);
#pragma unroll
            for (int kk = 0; kk < tc05::kChunkK / 16; ++kk)
                tc05::mma_f16(tmem, da + (uint32_t)(16 * kk), db + (uint32_t)(16 * kk), idesc, (k > 0) || (kk > 0));
            tc05::mma_commit(&empty[s]);
            if (loaded < nk) {  // into the stage of chunk k - 1, once its MMAs are done
                if (k > 0)
                    ok = tc05::mbar_wait(&empty[(k - 1) % kWgStages], (uint32_t)(((k - 1) / kWgStages) & 1), kPolls)
                             ? 1
                             : 0;
                if (!ok)
                    break;
                load(loaded++);
            }
        }
        tc05::mma_commit(&done);
        if (!ok)  // copies in flight before the shared memory is given back
            for (int q = k; q < loaded; ++q)
                tc05::mbar_wait(&full[q % kWgStages], (uint32_t)((q / kWgStages) & 1), kPolls);
    }
    __syncwarp();
    ok = tc05::mbar_wait(&done, 0, kPolls) ? ok : 0;
    tc05::fence_after_sync();
    ok = __syncthreads_and(ok);
    if (!ok) {
        if (t == 0)
            atomicOr(a.err, 1u);
    } else if (warp < 4) {
        const int o = mh * 128 + warp * 32 + lane;
        float *c = a.part + (((size_t)layer * a.splits + split) * kSurH + o) * kSurH + nh * 128;
#pragma unroll
        for (int n0 = 0; n0 < 128; n0 += 16) {
            float v[16];
            tc05::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)n0, v);
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4 *>(c + n0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
    }
    tc05::fence_before_sync();
    __syncthreads();
    if (warp == 4) {
        tc05::fence_after_sync();
        tc05::tmem_dealloc(tmem, 128);
    }
}

// ------------------------------------------------------------------ parameter update

// BF16 copies of the weights w[0..3] = W_l[4 o4 + q][i], l = layer + 2: row-major (the
// engine's screening kernel) and the K-chunk tile images of the forward GEMM (units x
// inputs) and of the backward GEMM (inputs x units).
__device__ __forceinline__ void store_copies(const float *w, int layer, int o4, int i, __nv_bfloat16 *Wf,
                                             __nv_bfloat16 *wtiles)
{
    unsigned char *fw = reinterpret_cast<unsigned char *>(wtiles + ((size_t)layer * kRing + (i >> 6)) * kNetTileElems);
    unsigned char *bw =
        reinterpret_cast<unsigned char *>(wtiles + ((size_t)(5 - layer) * kRing + (o4 >> 4)) * kNetTileElems);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int o = o4 * 4 + q;
        const __nv_bfloat16 h = __float2bfloat16_rn(w[q]);
        Wf[((size_t)layer * kSurH + o) * kSurH + i] = h;
        *reinterpret_cast<__nv_bfloat16 *>(fw + tc05::tile_offset(o, (i & 63) >> 3) + (i & 7) * 2) = h;
    }
    *reinterpret_cast<uint2 *>(bw + tc05::tile_offset(i, (o4 >> 1) & 7) + (o4 & 1) * 8) =
        make_uint2(pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]));
}

// Adam on one FP32 master parameter (bias-corrected); returns the new value.  The
// contractions are spelled out: an optimiser's path amplifies a last-bit difference, and
// every inlined copy has to round alike.
__device__ __forceinline__ float adam(const NetUpdateArgs &a, int k, float gi)
{
    const float mi = fmaf(1.f - a.b1, gi, __fmul_rn(a.b1, a.m[k]));
    const float vi = fmaf(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, a.v[k]));
    a.m[k] = mi;
    a.v[k] = vi;
    const float p = a.P[k] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
    a.P[k] = p;
    return p;
}

constexpr int kUpdW = 3 * kSurH * kSurH / 4 / 256;  // blocks on the 256 x 256 weights
constexpr int kUpdW1 = 4 * kSurH / 8;               // blocks on layer 1, eight units and two inputs each
constexpr int kUpdV = 4 * kSurH / 8 + kUpdW1;       // blocks on the per-unit vectors and layer 1

// Fixed-order sum of one value per thread over 256 threads, complete in thread 0.
__device__ float block_sum256(float v, float *red)
{
#pragma unroll
    for (int w = 16; w > 0; w >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, w);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w)
            s += red[w];
    __syncthreads();
    return s;
}

// The sum of acc[0..7] of the four lanes u, u + 8, u + 16, u + 24 (a unit's 32 rows), in
// the tree order of a warp with one lane per row.
__device__ __forceinline__ float rows_sum(float *acc)
{
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e)
            acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    return ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
}

// acc[e] += h_e, and += h_e u_e, for a thread's eight rows.
__device__ __forceinline__ void add_rows(uint4 h, float *acc)
{
    acc[0] += bf16_lo(h.x), acc[1] += bf16_hi(h.x), acc[2] += bf16_lo(h.y), acc[3] += bf16_hi(h.y);
    acc[4] += bf16_lo(h.z), acc[5] += bf16_hi(h.z), acc[6] += bf16_lo(h.w), acc[7] += bf16_hi(h.w);
}

__device__ __forceinline__ void fma_rows(uint4 h, float4 u0, float4 u1, float *acc)
{
    acc[0] = fmaf(bf16_lo(h.x), u0.x, acc[0]), acc[1] = fmaf(bf16_hi(h.x), u0.y, acc[1]);
    acc[2] = fmaf(bf16_lo(h.y), u0.z, acc[2]), acc[3] = fmaf(bf16_hi(h.y), u0.w, acc[3]);
    acc[4] = fmaf(bf16_lo(h.z), u1.x, acc[4]), acc[5] = fmaf(bf16_hi(h.z), u1.y, acc[5]);
    acc[6] = fmaf(bf16_lo(h.w), u1.z, acc[6]), acc[7] = fmaf(bf16_hi(h.w), u1.w, acc[7]);
}

// The rest of the gradient and what is done with it.  ADAM: the optimiser step and the
// BF16 copies at once (the gradient is not stored).  The first blocks sum eight units of
// one tile image over all rows (biases: dZ; output weights: H4 dO; layer 1: dZ1 and
// dZ1 X): warp (q, half) takes rows 64 q + 32 half + 0..31 of every 256, its lane (u, c)
// the piece of eight rows of unit u, so that a load of a warp is four whole lines.  One
// block sums dO (output bias) and the squared residuals (loss).  A thread of the other
// kUpdW blocks sums the split partials of four output units of one input, so that splits
// are read coalesced.  Bound by the latency of a handful of dependent L2 reads.
template <bool ADAM>
__global__ void __launch_bounds__(256) k_net_update(NetUpdateArgs a)
{
    const int t = threadIdx.x, v = (int)blockIdx.x + a.first;
    if (v > kUpdV) {
        const int b = v - kUpdV - 1, layer = b >> 6, o4 = b & 63, i = t;
        const float *p = a.wpart + (size_t)layer * a.splits * kSurH * kSurH + (size_t)o4 * 4 * kSurH + i;
        float gsum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int s = 0; s < a.splits; ++s) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                gsum[q] += p[(size_t)s * kSurH * kSurH + q * kSurH];
        }
        const int k0 = sur_w_off(layer + 2) + o4 * 4 * kSurH + i;
        if (ADAM) {
            float w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                w[q] = adam(a, k0 + q * kSurH, gsum[q]);
            store_copies(w, layer, o4, i, a.Wf, a.wtiles);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                a.G[k0 + q * kSurH] = gsum[q];
        }
        return;
    }
    const int warp = t >> 5, lane = t & 31;
    if (v == kUpdV) {
        __shared__ float red[8];
        float d = 0.f, r = 0.f;
        for (int i = t; i < a.rows; i += 256) {
            d += a.dO[i];
            r += a.r2[i];
        }
        d = block_sum256(d, red);
        r = block_sum256(r, red);
        if (t == 0) {
            *a.loss_sum = r;
            if (ADAM)
                adam(a, kOffB5, d);
            else
                a.G[kOffB5] = d;
        }
        return;
    }
    const int tiles = a.rows / kNetRows, q = warp >> 1, u = lane & 7, c = (warp & 1) * 4 + (lane >> 3);
    __shared__ float sums[3][8][8];
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const bool first_layer = v >= kUpdV - kUpdW1;
    // vector 0..2: b2..b4, 3: w5; then layer 1, two inputs a block, the first with the bias
    const int vec = v >> 5, w1 = v - (kUpdV - kUpdW1), i0 = (w1 & 3) * 2;
    const int unit = (first_layer ? w1 >> 2 : v & 31) * 8 + u;
    const int kind = first_layer ? kActZ1 : vec < 3 ? kActZ1 + 1 + vec : kActH1 + 3;
    const unsigned char *img = reinterpret_cast<const unsigned char *>(a.act + (size_t)kind * tiles * kNetTileElems) +
                               tc05::tile_offset(unit, c);
    if (!first_layer) {
        if (vec < 3) {
#pragma unroll 8
            for (int tile = q; tile < tiles; tile += 4)
                add_rows(*reinterpret_cast<const uint4 *>(img + (size_t)tile * kTileBytes), acc);
        } else {
#pragma unroll 4
            for (int tile = q; tile < tiles; tile += 4) {
                const float4 *d = reinterpret_cast<const float4 *>(a.dO + tile * kNetRows + c * 8);
                fma_rows(*reinterpret_cast<const uint4 *>(img + (size_t)tile * kTileBytes), d[0], d[1], acc);
            }
        }
        const float s = rows_sum(acc);
        if (lane < 8)
            sums[0][warp][u] = s;
    } else {
        float d[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e)
                d[i][e] = 0.f;
#pragma unroll 4
        for (int tile = q; tile < tiles; tile += 4) {
            const uint4 h = *reinterpret_cast<const uint4 *>(img + (size_t)tile * kTileBytes);
            add_rows(h, acc);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 *x =
                    reinterpret_cast<const float4 *>(a.xb + (size_t)(i0 + i) * a.rows + tile * kNetRows + c * 8);
                fma_rows(h, x[0], x[1], d[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float s = rows_sum(d[i]);
            if (lane < 8)
                sums[i][warp][u] = s;
        }
        const float s = rows_sum(acc);
        if (lane < 8)
            sums[2][warp][u] = s;
    }
    __syncthreads();
    const int j = t >> 3;  // which sum of unit u
    if (j >= (!first_layer ? 1 : i0 == 0 ? 3 : 2))
        return;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w)
        s += sums[j][w][u];
    const int k = !first_layer ? (vec < 3 ? sur_b_off(2 + vec) : kOffW5) + unit
                  : j < 2      ? kOffW1 + unit * kSurIn + i0 + j
                               : kOffB1 + unit;
    if (ADAM)
        adam(a, k, s);
    else
        a.G[k] = s;
}

// The BF16 copies of parameters set by the host.
__global__ void __launch_bounds__(256) k_net_copies(const float *P, __nv_bfloat16 *Wf, __nv_bfloat16 *wtiles)
{
    const int layer = blockIdx.x >> 6, o4 = blockIdx.x & 63, i = threadIdx.x;
    float w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        w[q] = P[sur_w_off(layer + 2) + (o4 * 4 + q) * kSurH + i];
    store_copies(w, layer, o4, i, Wf, wtiles);
}

}  // namespace

// ------------------------------------------------------------------ launchers

cudaError_t net_set_limits()
{
    cudaError_t e = cudaFuncSetAttribute(k_net_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNetSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_net_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNetSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_net_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem);
    return e;
}

cudaError_t launch_net_rows(const NetRowsArgs &a, bool backward, int max_ctas, cudaStream_t st)
{
    const int tiles = (a.rows + kNetRows - 1) / kNetRows;
    const int grid = tiles < max_ctas ? tiles : max_ctas;
    if (backward)
        k_net_rows<true><<<grid, kNetThreads, kNetSmem, st>>>(a);
    else
        k_net_rows<false><<<grid, kNetThreads, kNetSmem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_net_wgrad(const NetWgradArgs &a, cudaStream_t st)
{
    k_net_wgrad<<<dim3(4, 3, a.splits), kWgThreads, kWgSmem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_net_update(const NetUpdateArgs &args, NetUpdateMode mode, cudaStream_t st)
{
    NetUpdateArgs a = args;
    constexpr int kBlocks = kUpdW + kUpdV + 1;
    a.first = mode == kNetLossOnly ? kUpdV : 0;
    const int blocks = mode == kNetLossOnly ? 1 : kBlocks;
    if (mode == kNetAdam)
        k_net_update<true><<<blocks, 256, 0, st>>>(a);
    else
        k_net_update<false><<<blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_net_copies(const float *P, __nv_bfloat16 *Wf, __nv_bfloat16 *wtiles, cudaStream_t st)
{
    k_net_copies<<<kUpdW, 256, 0, st>>>(P, Wf, wtiles);
    return cudaGetLastError();
}

}  // namespace cgppd
