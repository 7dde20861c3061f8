// cuda_functions.cu -- the drop-in C ABI of the reference's CUDA energy module
// (src/cudaExterns.h:14-90, src/CudaFunctions.cu:20-277, :724-961), rebuilt for sm_103a.
//
// Callers keep the reference's packed layout: float4 pos[P] = (x, y, z, w) with
// w = rigid_domain_uid + bond_fraction (-2 for padding), float4 meta[P] =
// (type, charge, vdW radius, w) with w = molecule_id + chain_fraction (-1 for a
// crowder).  The pair rules are those of the reference's flexible-linker build.
//
// Kernel: a CTA takes 128 residues y (four warps of 32) against one, two or four blocks
// of 32 residues x on or after them.  Per block the 32 x are copied charged first, two to a
// record (one packed operation serves two pairs); each warp then decides once per block:
// nothing to do (all pairs excluded), no pair excluded (the packed loop, Debye-Hueckel for
// the charged records only, the minimum image only on the axes where the block's bounding
// box and the warp's residues leave more than one image), or a mixture (a scalar loop with
// the exclusion tests per pair).  Pair terms are FP32, at most eight to a partial sum,
// folded into float-float accumulators, reduced per CTA in float-float.  The last CTA to finish (ticket counters) reduces all CTA partials
// in a fixed order, so the total is deterministic.  Scratch (partials + tickets +
// result) is per (device, stream), allocated on first use and reused.
#include <cstdio>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "cgppd_common.cuh"
#include "host/amino_acids.h"
#include "pair_terms.cuh"
#include "status.h"
#include "cgppd_cuda_functions.h"

using namespace cgppd;

namespace {

constexpr int kTile = 128;                 // residues y of a CTA, one per thread
constexpr int kThreads = kTile;
constexpr int kWarps = kThreads / 32;
constexpr int kBlock = 32;                 // residues of an x block and of a warp's y block
constexpr int kTypes = 20;
// Tiles of a call from which a CTA takes four (two) x blocks, see x_blocks.
constexpr int kFourBlocks = 40, kTwoBlocks = 34;
// Slack (A) on the box test that drops the minimum image: covers the rounding of the
// relative positions.
constexpr float kImageSlack = 0.05f;

__constant__ float c_boxdim;  // CUDA_setBoxDimension, module state per device
// cgppd_set_repulsive_crowding: the reference's compile-time REPULSIVE_CROWDING
// (src/definitions.h:18) as process-wide module state, read at each launch
std::atomic<int> g_repulsive_crowding{0};

// CTAs are reduced in groups of kGroup: the last CTA of a group to finish sums the
// group's partials, the last group to finish sums the group sums.
constexpr int kGroup = 32;

struct Scratch {
    unsigned *ticket = nullptr;   // group completion counter, self-resetting
    unsigned *flags = nullptr;    // bit 0: residue type index out of range
    double *result = nullptr;     // {LJ raw, DH raw, total kcal/mol, flags of the call}
    double *host = nullptr;       // page-locked copy of result (synchronous entry points), written by the kernel
    double *partials = nullptr;   // 16 bytes per CTA: its LJ and DH sums as float-float
    float4 *gsums = nullptr;      // 16 bytes per group: its LJ and DH sums as float-float
    unsigned *gtickets = nullptr; // CTA completion counter per group, self-resetting
    size_t capacity = 0;          // CTAs the partials can hold
};

// Scratch layout for `cap` CTAs: [ticket, flags | pad to 256] [result: 4 doubles | pad]
// [partials: 16 bytes per CTA] [group sums: 16 bytes per group] [group tickets: 4 bytes
// per group]; the counters (the first 8 bytes and the group tickets) start at zero.
constexpr size_t scratch_groups(size_t cap) { return (cap + kGroup - 1) / kGroup; }
constexpr size_t scratch_gsums_at(size_t cap) { return 512 + 16 * cap; }
constexpr size_t scratch_gtickets_at(size_t cap) { return scratch_gsums_at(cap) + 16 * scratch_groups(cap); }
constexpr size_t scratch_bytes(size_t cap) { return scratch_gtickets_at(cap) + 4 * scratch_groups(cap); }

void scratch_view(unsigned char *base, size_t cap, Scratch &s)
{
    s.ticket = reinterpret_cast<unsigned *>(base);
    s.flags = reinterpret_cast<unsigned *>(base + 4);
    s.result = reinterpret_cast<double *>(base + 256);
    s.partials = reinterpret_cast<double *>(base + 512);
    s.gsums = reinterpret_cast<float4 *>(base + scratch_gsums_at(cap));
    s.gtickets = reinterpret_cast<unsigned *>(base + scratch_gtickets_at(cap));
    s.capacity = cap;
}

std::mutex g_mu;
std::map<std::pair<int, cudaStream_t>, Scratch> g_scratch;
std::map<int, const float *> g_bound_table;  // bindLJTexture, per device

__device__ __forceinline__ float frac_int(float w, float &ip)
{
    ip = truncf(w);
    return w - ip;
}

// The Lennard-Jones part of lj_term with the table value m4e = -4 Eij (RT units) and the
// mixed radius sigma_ij: u = m4e s6 (s6 - 1), and 2 Eij - u on the repulsive branch
// (Eij > 0, s6 > 1/2); one multiplication less than lj_term.
__device__ __forceinline__ float lj_m4(float m4e, float sigma_ij, float inv_r2)
{
    const float s2 = sigma_ij * sigma_ij * inv_r2;
    const float s6 = s2 * s2 * s2;
    float u = m4e * fmaf(s6, s6, -s6);
    if (m4e < 0.0f && s6 > 0.5f)
        u = fmaf(-0.5f, m4e, -u);
    return u;
}

// The keys of the exclusion rules over 32 residues, as ranges of their bit patterns (two
// sets of floats whose bit-pattern ranges are disjoint share no value): nonzero rigid
// domain, nonzero bond fraction, chain fraction, molecule id (>= 0); an empty range has
// lo > hi.  flags: bit 0 padding, 1 crowder, 2 a residue without a rigid domain.
struct Keys {
    int dlo, dhi, blo, bhi, clo, chi, mlo, mhi, flags;
};

__device__ __forceinline__ Keys warp_keys(bool real, bool crowd, float dom, float bond, float chain, float mol)
{
    const int none_lo = 0x7fffffff, none_hi = (int)0x80000000;
    // + 0.0f turns -0 into +0: the exclusion tests compare keys as floats, where -0 == +0
    const int d = __float_as_int(dom + 0.0f), b = __float_as_int(bond + 0.0f), c = __float_as_int(chain + 0.0f),
              m = __float_as_int(mol + 0.0f);
    const bool hd = real && dom != 0.0f, hb = real && bond != 0.0f, hm = real && mol >= 0.0f;
    Keys k;
    k.dlo = __reduce_min_sync(0xffffffffu, hd ? d : none_lo), k.dhi = __reduce_max_sync(0xffffffffu, hd ? d : none_hi);
    k.blo = __reduce_min_sync(0xffffffffu, hb ? b : none_lo), k.bhi = __reduce_max_sync(0xffffffffu, hb ? b : none_hi);
    k.clo = __reduce_min_sync(0xffffffffu, real ? c : none_lo);
    k.chi = __reduce_max_sync(0xffffffffu, real ? c : none_hi);
    k.mlo = __reduce_min_sync(0xffffffffu, hm ? m : none_lo), k.mhi = __reduce_max_sync(0xffffffffu, hm ? m : none_hi);
    k.flags = (int)__reduce_or_sync(0xffffffffu, (real ? 0u : 1u) | (crowd ? 2u : 0u) |
                                                     (real && dom == 0.0f ? 4u : 0u));
    return k;
}

__device__ __forceinline__ bool disjoint(int alo, int ahi, int blo, int bhi) { return ahi < blo || bhi < alo; }

// One block of 32 residues x.
struct XBlock {
    float4 xy[16], zw[16], qt[16];  // records of two: (x0, x1, y0, y1), (z0, z1, s0/2, s1/2), (q0, q1, row0, row1)
    float4 pos[32];                 // as given: position, half radius
    float4 key[32];                 // domain, bond, chain, molecule
    float4 meta[32];                // charge, table row (bytes), flags (1 padding, 2 crowder)
    Keys keys;
    int k1, k2;                     // residues in charged and uncharged records (multiples of 4)
    float3 mid, half;               // of the bounding box
};

// Orders floats as signed integers.
__device__ __forceinline__ int ordered(float f)
{
    const int i = __float_as_int(f);
    return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unordered(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

__device__ __forceinline__ void box_axis(float v, bool use, float &mid, float &half)
{
    const float lo = unordered(__reduce_min_sync(0xffffffffu, use ? ordered(v) : 0x7f7fffff));
    const float hi = unordered(__reduce_max_sync(0xffffffffu, use ? ordered(v) : (int)0x80800000));
    mid = 0.5f * (lo + hi);
    half = 0.5f * (hi - lo);
}

// Warp: the block's copies from the residue (p, m) of each lane.  `copied`: the residue
// takes part in the packed loop.
__device__ __forceinline__ void build_block(XBlock &X, float4 p, float4 m, int type, bool copied, bool pad, bool crowd)
{
    const int lane = threadIdx.x & 31;
    float dom, mol;
    const float bond = frac_int(p.w, dom), chain = frac_int(m.w, mol);
    const Keys k = warp_keys(!pad, crowd, dom, bond, chain, mol);
    float3 mid, half;
    box_axis(p.x, copied, mid.x, half.x);
    box_axis(p.y, copied, mid.y, half.y);
    box_axis(p.z, copied, mid.z, half.z);
    const int row = type * kTypes * 4;
    X.pos[lane] = make_float4(p.x, p.y, p.z, 0.5f * m.z);
    X.key[lane] = make_float4(dom, bond, chain, mol);
    X.meta[lane] = make_float4(m.y, __int_as_float(row), __int_as_float((pad ? 1 : 0) | (crowd ? 2 : 0)), 0.f);
    // charged residues first, then the others, filled up to a multiple of four with the last
    // one's place and radius, no charge and the table's row of zeros
    const unsigned all = __ballot_sync(0xffffffffu, copied), chg = __ballot_sync(0xffffffffu, copied && m.y != 0.0f);
    const unsigned below = (1u << lane) - 1u;
    const int n = __popc(all), nq = __popc(chg);
    const int at = (chg >> lane & 1u) ? __popc(chg & below) : nq + __popc(all & ~chg & below);
    const int n4 = (n + 3) & ~3, k1 = min((nq + 3) & ~3, n4);
    auto put = [&](int k, float q, int r) {
        const int h = k & 1;
        float *a = reinterpret_cast<float *>(&X.xy[k >> 1]), *b = reinterpret_cast<float *>(&X.zw[k >> 1]),
              *c = reinterpret_cast<float *>(&X.qt[k >> 1]);
        a[h] = p.x, a[2 + h] = p.y;
        b[h] = p.z, b[2 + h] = 0.5f * m.z;
        c[h] = q, c[2 + h] = __int_as_float(r);
    };
    if (copied) {
        put(at, m.y, row);
        if (at == n - 1)
            for (int e = n; e < n4; ++e)
                put(e, 0.0f, kTypes * kTypes * 4);
    }
    if (lane == 0) {
        X.keys = k;
        X.k1 = k1;
        X.k2 = n4 - k1;
        X.mid = mid;
        X.half = half;
    }
}

// A thread's residue y: negated position, shift -L k to its image nearest the block's
// middle, half radius, charge, its column of the table.
struct YLane {
    f2 nx, ny, nz, sx, sy, sz, w, q;
    const char *col;
};

// Which differences x - y need what.  The difference of the positions as given is exact for
// close residues and the shift is exact, so all forms give min_image's bits (positions
// relative to the block's middle save the shift's addition, but round: ten times the
// error of a contact's energy).
constexpr int kPlain = 0, kShift = 8;  // bits 0, 1, 2: the minimum image per pair on that axis

template <int MODE, int AXIS>
__device__ __forceinline__ f2 difference(f2 x, f2 ny, f2 shift, f2 nL, f2 invL)
{
    const f2 d = f2_add(x, ny);
    if (MODE & AXIS)
        return min_image2(d, nL, invL);
    return (MODE & kShift) ? f2_add(d, shift) : d;
}

// R records of a block with y, terms added in order to four partial sums each of the
// Lennard-Jones and (DH) Debye-Hueckel part.
template <bool DH, int MODE, int R>
__device__ __forceinline__ void block_records(const XBlock &X, int r, const YLane &y, f2 nL, f2 invL, f2 *lj, f2 *dh)
{
    Pair2 e[R];
    float closest = 0.0f;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const ulonglong2 xy = reinterpret_cast<const ulonglong2 *>(X.xy)[r + k],
                         zw = reinterpret_cast<const ulonglong2 *>(X.zw)[r + k];
        const int2 row = reinterpret_cast<const int2 *>(&X.qt[r + k])[1];
        e[k] = lj2_sq<DH>(difference<MODE, 1>(xy.x, y.nx, y.sx, nL, invL),
                          difference<MODE, 2>(xy.y, y.ny, y.sy, nL, invL),
                          difference<MODE, 4>(zw.x, y.nz, y.sz, nL, invL), f2_add(zw.y, y.w),
                          f2_pack(*reinterpret_cast<const float *>(y.col + row.x),
                                  *reinterpret_cast<const float *>(y.col + row.y)));
        closest = fmaxf(closest, closest2(e[k]));
    }
    if (closest > 0.5f) {
#pragma unroll
        for (int k = 0; k < R; ++k)
            repulsive2(e[k]);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        lj[k & 1] = f2_add(lj[k & 1], e[k].u);
        if (DH)
            dh[k & 1] = f2_add(dh[k & 1], dh2(e[k], f2_mul(reinterpret_cast<const f2 *>(&X.qt[r + k])[0], y.q)));
    }
}

__device__ __forceinline__ float sum4(const f2 *v)
{
    float a, b, c, d;
    f2_unpack(v[0], a, b);
    f2_unpack(v[1], c, d);
    return (a + b) + (c + d);
}

// A whole block (no pair of it excluded) with y: the charged records in full, the others
// the Lennard-Jones part alone.  Two records at a time and rolled loops: with four, and
// one more copy of each loop for the odd pair, the warps of an SM were spread over more
// code than its instruction caches hold (69 M pairs: 100 us, 6 of 13 stall cycles an
// instruction waiting for instructions; 71 us like this, issue slots 74 % busy while the
// SMs are, FMA pipes 57 %).
template <int MODE>
__device__ __forceinline__ void clean_block(const XBlock &X, const YLane &y, float L, float invL, FF &lj, FF &dh)
{
    const f2 nL = f2_dup(-L), invL2 = f2_dup(invL);
    f2 u[2] = {0ull, 0ull}, d[2] = {0ull, 0ull};
    const int r1 = X.k1 >> 1, r2 = r1 + (X.k2 >> 1);
    int r = 0;
#pragma unroll 1
    for (; r < r1; r += 2)
        block_records<true, MODE, 2>(X, r, y, nL, invL2, u, d);
#pragma unroll 1
    for (; r < r2; r += 2)
        block_records<false, MODE, 2>(X, r, y, nL, invL2, u, d);
    ff_add(lj, sum4(u));
    ff_add(dh, sum4(d));
}

// ------------------------------------------------------------------ work of a call

// x blocks of a CTA for nt tiles: the blocks of a CTA are a serial chain, so one while that
// leaves SMs short of warps, more once the copies and keys of a CTA cost more than the
// chain.  us a call with 1 / 2 / 4 blocks:
//   tiles                    28               34               39               44
//   async, three streams      8.4/ 8.7/10.2   12.4/11.0/12.0   15.9/14.4/13.3   20.3/18.7/15.4
//   async, one stream        16.9/19.0/24.5   20.8/21.4/27.5   25.0/25.1/29.7   29.6/29.5/31.9
//   synchronous              28.3/30.9/35.0   32.9/32.9/37.9   37.0/36.8/40.0   40.7/41.1/42.5
//   synchronous, NC          25.5/25.7/26.2   29.9/28.4/28.7   34.4/32.3/32.7   38.0/35.4/34.6
//   tiles                    48               56               64              100
//   async, three streams     23.9/21.9/18.0   32.0/29.4/24.3   41.3/37.8/31.4   99.1/90.7/75.5
//   async, one stream        32.5/33.0/35.7   41.5/40.9/41.5   50.0/49.1/48.9  109.4/102.3/93.1
//   synchronous              44.1/43.4/47.0   52.4/51.5/52.5   61.7/59.7/59.7  120.7/113.2/104.1
//   synchronous, NC          40.7/38.7/37.3   49.3/46.1/43.2   57.7/54.0/50.2  114.0/104.4/93.0
// The size is all that a call knows of what runs beside it, so the lines lie between the
// two: two blocks from 34 tiles, where they take 11 % off calls on several streams and add 3 %
// to others (at 30: 5 against 11); four from 40, where they take 12 to 18 % off calls on
// several streams and add up to 15 % to others (at 38 and 39 they would take 4 to 8 and add
// 18 to 19); from 60 tiles on they are the best, or level, for all.
__host__ __device__ constexpr int x_blocks(int nt) { return nt >= kFourBlocks ? 4 : nt >= kTwoBlocks ? 2 : 1; }

// CTAs of a call: for each tile ty the chunks of x blocks on or after it, rows of
// decreasing length.
__host__ __device__ constexpr int chunks(int nt, int nx) { return 4 * nt / nx; }
__host__ __device__ constexpr int energy_ctas(int nt)
{
    const int nx = x_blocks(nt), nc = chunks(nt, nx), step = 4 / nx;
    return nt * nc - step * (nt * (nt - 1) / 2);
}
// CTA b -> tile ty and chunk: row ty starts at f(ty) = ty nc - step ty (ty - 1) / 2.
__device__ __forceinline__ void cta_work(int b, int nt, int nx, int &ty, int &chunk)
{
    const int nc = chunks(nt, nx), step = 4 / nx;
    auto first = [&](int r) { return r * nc - step * (r * (r - 1) / 2); };
    const float h = (float)nc / (float)step + 0.5f;
    int r = (int)(h - sqrtf(fmaxf(0.0f, h * h - 2.0f * (float)b / (float)step)));
    r = max(0, min(nt - 1, r));
    while (r > 0 && first(r) > b)
        --r;
    while (r < nt - 1 && first(r + 1) <= b)
        ++r;
    ty = r;
    chunk = step * r + (b - first(r));
}

// kNC: non-crowder pairs of different molecules only (E_TiledKernelNC).  kRC: the
// REPULSIVE_CROWDING form of the crowder pairs.
template <bool kNC, bool kRC, int NX>
__global__ void __launch_bounds__(kThreads) k_tile_energy(const float4 *__restrict__ pos, const float4 *__restrict__ meta,
                                                          int P, int nt, const float *__restrict__ lj_raw,
                                                          double *__restrict__ partials, unsigned *__restrict__ ticket,
                                                          unsigned *__restrict__ flags, double *__restrict__ result,
                                                          float4 *__restrict__ gsums, unsigned *__restrict__ gtickets,
                                                          float *__restrict__ async_out, int async_count,
                                                          double *__restrict__ host)
{
    __shared__ XBlock s_x[NX];
    __shared__ float s_m4[(kTypes + 1) * kTypes];  // -4 Eij in RT units, [x type][y type]; a row of zeros
    __shared__ FF s_red[2][kWarps];
    __shared__ bool s_last;

    // a dependent launch (see launch_energy): nothing global is touched before the
    // stream's previous kernel has completed
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int ty, chunk;
    cta_work(blockIdx.x, nt, NX, ty, chunk);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // the x and y records first, so that their loads overlap the table's
    const int x = (chunk * NX + warp) * kBlock + lane, y = ty * kTile + t;
    float4 px = make_float4(0.f, 0.f, 0.f, kPadder), mx = make_float4(0.f, 0.f, 0.f, 0.f), py = px, my = mx;
    if (warp < NX && x < P) {
        px = pos[x];
        mx = meta[x];
    }
    if (y < P) {
        py = pos[y];
        my = meta[y];
    }
    for (int k = t; k < kTypes * kTypes; k += kThreads)
        s_m4[k % kTypes * kTypes + k / kTypes] = -4.0f * (kLambda * (lj_raw[k] - kE0));
    if (t < kTypes)
        s_m4[kTypes * kTypes + t] = 0.0f;
    // the async form's output other than the total: zeroed by every CTA, a slice each
    if (async_out != nullptr && async_count > 1) {
        const int per = (async_count - 1 + (int)gridDim.x - 1) / (int)gridDim.x;
        const int k0 = 1 + (int)blockIdx.x * per, k1 = min(async_count, k0 + per);
        for (int k = k0 + t; k < k1; k += kThreads)
            async_out[k] = 0.0f;
    }
    // residue types are checked once per residue (0..19; padding is excluded anyway): the
    // pair loops then index the table without a bounds test
    unsigned bad = 0;
    if (warp < NX) {
        const bool pad = px.w == kPadder, crowd = mx.w == kCrowder;
        int xt = __float2int_rn(mx.x);
        if ((unsigned)xt >= (unsigned)kTypes) {
            // crowders read no table entry where they are excluded (kNC) or repulsive
            // only (kRC; the reference then gives them the type -1)
            bad |= (pad || (crowd && (kNC || kRC))) ? 0u : 1u;
            xt = 0;
        }
        build_block(s_x[warp], px, mx, xt, !pad && !(kNC && crowd), pad, crowd);
    }
    // this thread's y residue and its warp's keys
    const bool ypad = py.w == kPadder, ycrowd = my.w == kCrowder;
    const bool active = (py.w > kPadder) && (!kNC || !ycrowd);
    float ydom, ymol;
    const float ybond = frac_int(py.w, ydom), ychain = frac_int(my.w, ymol);
    const Keys yk = warp_keys(!ypad, ycrowd, ydom, ybond, ychain, ymol);
    int yt = __float2int_rn(my.x);
    if ((unsigned)yt >= (unsigned)kTypes) {
        bad |= (!active || (kRC && ycrowd)) ? 0u : 1u;
        yt = 0;
    }
    const float L = c_boxdim, invL = (L != 0.0f) ? 1.0f / L : 0.0f;
    const char *col = reinterpret_cast<const char *>(s_m4 + yt);
    const bool any_active = __any_sync(0xffffffffu, active);
    FF lj{0.f, 0.f}, dh{0.f, 0.f};
    __syncthreads();

    const int ys = ty * (kTile / kBlock) + warp;
    for (int b = 0; any_active && b < NX; ++b) {
        const int xs = chunk * NX + b;
        const XBlock &X = s_x[b];
        const Keys &xk = X.keys;
        if (xs < ys || X.k1 + X.k2 == 0)
            continue;
        bool none, clean;  // every pair excluded; no pair excluded
        if (kNC) {
            none = xk.mlo == xk.mhi && yk.mlo == yk.mhi && xk.mlo == yk.mlo;
            clean = xs != ys && disjoint(xk.mlo, xk.mhi, yk.mlo, yk.mhi);
        } else {
            none = xk.dlo == xk.dhi && yk.dlo == yk.dhi && xk.dlo == yk.dlo && ((xk.flags | yk.flags) & 4) == 0;
            clean = xs != ys && disjoint(xk.dlo, xk.dhi, yk.dlo, yk.dhi) && disjoint(xk.blo, xk.bhi, yk.blo, yk.bhi) &&
                    (xs - ys > 1 || disjoint(xk.clo, xk.chi, yk.clo, yk.chi));
            if (kRC)
                clean = clean && ((xk.flags | yk.flags) & 2) == 0;
        }
        if (none)
            continue;
        if (clean) {
            // y's image nearest the block's middle; on the axes where that lies inside the half
            // box less the block's half extent for the whole warp, it is the image of every pair
            auto image = [&](float d) { return __fadd_rn(__fmaf_rn(d, invL, 12582912.0f), -12582912.0f); };
            const float3 d = make_float3(X.mid.x - py.x, X.mid.y - py.y, X.mid.z - py.z);
            const float3 k = make_float3(image(d.x), image(d.y), image(d.z));
            const float lim = 0.5f * L - kImageSlack;
            auto outside = [&](float dd, float kk, float half) {
                return !(fabsf(fmaf(-L, kk, dd)) + half < lim && fabsf(kk) <= 2.0f);  // (-L k is exact)
            };
            const unsigned mode = (outside(d.x, k.x, X.half.x) ? 1u : 0u) | (outside(d.y, k.y, X.half.y) ? 2u : 0u) |
                                  (outside(d.z, k.z, X.half.z) ? 4u : 0u) |
                                  (k.x != 0.0f || k.y != 0.0f || k.z != 0.0f ? 8u : 0u);
            const unsigned any = __reduce_or_sync(0xffffffffu, active && L != 0.0f ? mode : 0u);
            const YLane yl{f2_dup(-py.x), f2_dup(-py.y), f2_dup(-py.z), f2_dup(-L * k.x), f2_dup(-L * k.y),
                           f2_dup(-L * k.z), f2_dup(0.5f * my.z), f2_dup(my.y), col};
            if (any == 0u)
                clean_block<kPlain>(X, yl, L, invL, lj, dh);
            else if (any == 8u)
                clean_block<kShift>(X, yl, L, invL, lj, dh);
            else if ((any & 7u) == 1u)
                clean_block<kShift | 1>(X, yl, L, invL, lj, dh);
            else if ((any & 7u) == 2u)
                clean_block<kShift | 2>(X, yl, L, invL, lj, dh);
            else if ((any & 7u) == 4u)
                clean_block<kShift | 4>(X, yl, L, invL, lj, dh);
            else
                clean_block<7>(X, yl, L, invL, lj, dh);
            continue;
        }
        // branch-free: every pair is evaluated and the excluded ones (padding, the pair
        // itself on the diagonal: possibly inf / NaN) are selected away
        const bool ydom_nz = ydom != 0.f, ybond_nz = ybond != 0.f, near = xs - ys <= 1, diag = xs == ys;
        float l0 = 0.f, l1 = 0.f, d0 = 0.f, d1 = 0.f;
#pragma unroll 2
        for (int j = 0; j < kBlock; ++j) {
            const float4 xkey = X.key[j], xm = X.meta[j], xp = X.pos[j];
            const int xflags = __float_as_int(xm.z);
            bool excl = (xflags & 1) || (diag && j <= lane);
            if (kNC)
                excl = excl || (xflags & 2) || xkey.w == ymol;
            else
                excl = excl || (ydom_nz && xkey.x == ydom) || (ybond_nz && xkey.y == ybond) ||
                       (near && xkey.z == ychain && abs(xs * kBlock + j - y) < 4);
            const float dx = min_image(py.x - xp.x, L, invL);
            const float dy = min_image(py.y - xp.y, L, invL);
            const float dz = min_image(py.z - xp.z, L, invL);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const float inv_r = rsqrt_sfu(r2);
            const float m4 = *reinterpret_cast<const float *>(col + __float_as_int(xm.y));
            float lt = lj_m4(m4, 0.5f * my.z + xp.w, rcp_sfu(r2));
            float dt = dh_term(my.y * xm.x, r2 * inv_r, inv_r);
            if (kRC && (ycrowd || (xflags & 2))) {
                // REPULSIVE_CROWDING (src/CudaFunctions.cu:335-338, :492-498): (6/r)^12 in RT
                // units below 15 A, no Debye-Hueckel term
                const float sc = 6.0f * inv_r, s2 = sc * sc, s6 = s2 * s2 * s2;
                lt = (r2 * inv_r < kRepulsiveCutoff) ? s6 * s6 : 0.f;
                dt = 0.f;
            }
            lt = excl ? 0.f : lt;
            dt = excl ? 0.f : dt;
            if (j & 1) {
                l1 += lt;
                d1 += dt;
            } else {
                l0 += lt;
                d0 += dt;
            }
        }
        ff_add(lj, l0 + l1);
        ff_add(dh, d0 + d1);
    }
    if (!active)
        lj = dh = FF{0.f, 0.f};

    // the stream's next call may be scheduled once every CTA is past its pair work: its
    // CTAs then spread over SMs that are mostly idle, and wait for this kernel to end
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // CTA reduction in float-float on the FP32 pipe (the FP64 unit is slow on this part).
    // Each CTA leaves (LJ hi, LJ lo, DH hi, DH lo) in its 16-byte partials slot.
    float4 *part4 = reinterpret_cast<float4 *>(partials);
    lj = ff_warp_sum(lj);
    dh = ff_warp_sum(dh);
    bad = __any_sync(0xffffffffu, bad) ? 1u : 0u;
    if (lane == 0) {
        s_red[0][warp] = lj;
        s_red[1][warp] = dh;
        if (bad)
            atomicOr(flags, 1u);
    }
    __syncthreads();
    const int ngroups = ((int)gridDim.x + kGroup - 1) / kGroup;
    const int g = blockIdx.x / kGroup, gsize = min(kGroup, (int)gridDim.x - g * kGroup);
    if (t == 0) {
        FF a = s_red[0][0], b = s_red[1][0];
        for (int w = 1; w < kWarps; ++w) {
            ff_add_ff(a, s_red[0][w]);
            ff_add_ff(b, s_red[1][w]);
        }
        part4[blockIdx.x] = make_float4(a.hi, a.lo, b.hi, b.lo);
        __threadfence();
        s_last = atomicAdd(&gtickets[g], 1u) == (unsigned)gsize - 1u;
    }
    __syncthreads();
    if (!s_last || warp != 0)
        return;

    // Last CTA of its group: the group's partials in a fixed order (float-float, one warp);
    // a call of one group ends here.
    __threadfence();
    FF a{0.f, 0.f}, b{0.f, 0.f};
    if (lane < gsize) {
        const float4 p = __ldcg(&part4[g * kGroup + lane]);
        a = FF{p.x, p.y};
        b = FF{p.z, p.w};
    }
    a = ff_warp_sum(a);
    b = ff_warp_sum(b);
    if (lane == 0)
        gtickets[g] = 0u;
    if (ngroups > 1) {
        unsigned last = 0;
        if (lane == 0) {
            gsums[g] = make_float4(a.hi, a.lo, b.hi, b.lo);
            __threadfence();
            last = atomicAdd(ticket, 1u) == (unsigned)ngroups - 1u;
        }
        if (!__shfl_sync(0xffffffffu, last, 0))
            return;
        // Last group: every group's sum in a fixed order, float-float, then FP64 once.
        __threadfence();
        a = b = FF{0.f, 0.f};
        for (int k = lane; k < ngroups; k += 32) {
            const float4 p = __ldcg(&gsums[k]);
            ff_add_ff(a, FF{p.x, p.y});
            ff_add_ff(b, FF{p.z, p.w});
        }
        a = ff_warp_sum(a);
        b = ff_warp_sum(b);
    }
    if (lane == 0) {
        const double lj_raw_sum = ff_value(a), dh_raw_sum = ff_value(b);
        const double total = lj_raw_sum * (double)kRTtoKcal + dh_raw_sum * (double)kDHFactor;
        const double f = (double)atomicExch(flags, 0u);
        result[0] = lj_raw_sum;
        result[1] = dh_raw_sum;
        result[2] = total;
        result[3] = f;
        if (host != nullptr) {
            host[2] = total;
            host[3] = f;
        }
        if (async_out != nullptr && async_count > 0)
            async_out[0] = (float)total;
        if (ngroups > 1)
            *ticket = 0u;
    }
}

int current_device()
{
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

// Scratch for `blocks` CTAs on (current device, stream); g_mu must be held.
Scratch *scratch_for(cudaStream_t stream, size_t blocks)
{
    Scratch &s = g_scratch[std::make_pair(current_device(), stream)];
    if (s.capacity < blocks) {
        const size_t cap = blocks < 256 ? 256 : blocks;
        unsigned char *base = nullptr;
        if (cgppd_check(cudaMalloc(&base, scratch_bytes(cap)), "scratch allocation") != 0)
            return nullptr;  // (what there is stays: smaller calls still fit)
        // (the clear runs on the legacy stream, which the caller's stream need not wait for)
        if (cgppd_check(cudaMemset(base, 0, scratch_bytes(cap)), "scratch clear") != 0 ||
            cgppd_check(cudaStreamSynchronize(cudaStreamLegacy), "scratch clear") != 0) {
            cudaFree(base);
            return nullptr;
        }
        if (s.ticket != nullptr)
            cudaFree(s.ticket);
        scratch_view(base, cap, s);
    }
    return &s;
}

const float *bound_table()
{
    auto it = g_bound_table.find(current_device());
    return it == g_bound_table.end() ? nullptr : it->second;
}

// Launch the tile kernel on `stream`.  Returns 0 on success.  On a stream of the caller
// (the asynchronous entry point) the launch is a programmatic dependent one: the grid
// may be scheduled once every CTA of the stream's previous kernel has finished its pair
// work (for a previous call of this kernel), and each CTA waits for that kernel's
// completion (griddepcontrol.wait) before it reads or writes global memory, so the
// ordering the caller sees is that of a plain launch.
int launch_energy(bool nc, const float4 *pos, const float4 *meta, int P, const float *table, Scratch *s,
                  float *async_out, int async_count, cudaStream_t stream)
{
    const int nt = (P + kTile - 1) / kTile;
    // crowders take no part in the non-crowder sum, so its form has no crowder variant
    const bool rc = g_repulsive_crowding.load() != 0;
    const int nx = x_blocks(nt);
    auto kern = nc   ? (nx == 4 ? k_tile_energy<true, false, 4> : nx == 2 ? k_tile_energy<true, false, 2>
                                                                          : k_tile_energy<true, false, 1>)
                : rc ? (nx == 4 ? k_tile_energy<false, true, 4> : nx == 2 ? k_tile_energy<false, true, 2>
                                                                          : k_tile_energy<false, true, 1>)
                     : (nx == 4 ? k_tile_energy<false, false, 4> : nx == 2 ? k_tile_energy<false, false, 2>
                                                                           : k_tile_energy<false, false, 1>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)energy_ctas(nt));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    const bool dependent = stream != cudaStreamLegacy && stream != nullptr;
    cfg.attrs = dependent ? attr : nullptr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cgppd_check(cudaLaunchKernelEx(&cfg, kern, pos, meta, P, nt, table, s->partials, s->ticket, s->flags,
                                          s->result, s->gsums, s->gtickets, async_out, async_count, s->host),
                       "energy kernel launch");
}

// Synchronous total on the legacy default stream (the reference's stream 0).
void eon_device_sync(bool nc, float4 *pos, float4 *meta, double *result, int datasetSize)
{
    *result = 0.0;
    if (datasetSize <= 0)
        return;
    std::lock_guard<std::mutex> lock(g_mu);
    const float *table = bound_table();
    if (table == nullptr) {
        cgppd_fail("CUDA_EonDevice: no contact table bound (call bindLJTexture first)");
        return;
    }
    const int nt = (datasetSize + kTile - 1) / kTile;
    Scratch *s = scratch_for(cudaStreamLegacy, (size_t)energy_ctas(nt));
    if (s == nullptr)
        return;
    // the result comes back through page-locked memory that the kernel writes: waiting for
    // the stream is then all that is left to do (two blocking copies of 24 and 4 bytes took
    // 15 us of a call)
    if (s->host == nullptr &&
        cgppd_check(cudaHostAlloc(&s->host, 4 * sizeof(double), cudaHostAllocMapped | cudaHostAllocPortable),
                    "result words") != 0)
        return;
    if (launch_energy(nc, pos, meta, datasetSize, table, s, nullptr, 0, cudaStreamLegacy) != 0 ||
        cgppd_check(cudaStreamSynchronize(cudaStreamLegacy), "energy result") != 0)
        return;
    const volatile double *host = s->host;
    if (host[3] != 0.0)
        cgppd_fail("CUDA_EonDevice: residue type index outside the 20x20 table");
    *result = host[2];
}

}  // namespace

extern "C" {

// Reference src/CudaFunctions.cu:20-32: report the last CUDA error and throw.
void __throwLastCudaError(const char *errorMessage, const char *file, const int line)
{
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        std::fprintf(stderr, "%s(%i) : getLastCudaError() CUDA error : %s : (%d) %s.\n", file, line, errorMessage,
                     (int)err, cudaGetErrorString(err));
        throw errorMessage;
    }
}

// Reference src/CudaFunctions.cu:75-104: a device copy of the contact table.
float *LJPotentialDataToDevice(AminoAcids *a)
{
    float *dev = nullptr;
    if (cgppd_check(cudaMalloc(&dev, sizeof(float) * 400), "LJPotentialDataToDevice") != 0)
        return nullptr;
    cgppd_check(cudaMemcpy(dev, &a->LJpotentials[0][0], sizeof(float) * 400, cudaMemcpyHostToDevice),
                "LJPotentialDataToDevice copy");
    return dev;
}

// Reference src/CudaFunctions.cu:106-125: copy the table into a caller-allocated buffer.
void copyLJPotentialDataToDevice(float *dev_LJPotentialData, AminoAcids *a)
{
    cgppd_check(cudaMemcpy(dev_LJPotentialData, &a->LJpotentials[0][0], sizeof(float) * 400, cudaMemcpyHostToDevice),
                "Failed to copy contact potentials");
}

// Reference src/CudaFunctions.cu:36-47: make `ljp` the table the energy kernels read on
// the current device.  The kernels read it through the read-only path after staging it
// in shared memory; there is no texture object to bind.
void bindLJTexture(float *ljp)
{
    std::lock_guard<std::mutex> lock(g_mu);
    g_bound_table[current_device()] = ljp;
}

void unbindLJTexture()
{
    std::lock_guard<std::mutex> lock(g_mu);
    g_bound_table.erase(current_device());
}

// Reference src/CudaFunctions.cu:157-167: periodic box edge, module state per device.
void CUDA_setBoxDimension(float value)
{
    cgppd_check(cudaMemcpyToSymbol(c_boxdim, &value, sizeof(value)), "Set boxdim");
}

void CUDA_freeBoxDimension()
{
    float zero = 0.0f;
    cudaMemcpyToSymbol(c_boxdim, &zero, sizeof(zero));
}

// Reference src/CudaFunctions.cu:198-277.  `LJPotentials` is never dereferenced (the
// reference callers pass an uninitialised pointer); the bound table is used.  The
// residue/molecule count arguments are accepted and unused, as in the reference.
void CUDA_EonDevice(float4 *residuePositions, float4 *residueMeta, int *residueCount, int *moleculePositions,
                    int *moleculeCount, float *LJPotentials, double *result, int blockSize, int datasetSize,
                    int sharedMemSize)
{
    (void)residueCount, (void)moleculePositions, (void)moleculeCount, (void)LJPotentials, (void)blockSize,
        (void)sharedMemSize;
    eon_device_sync(false, residuePositions, residueMeta, result, datasetSize);
}

// Reference src/CudaFunctions.cu:724-754: non-crowder, different-molecule pairs only.
void CUDA_EonDeviceNC(float4 *residuePositions, float4 *residueMeta, int *residueCount, int *moleculePositions,
                      int *moleculeCount, float *LJPotentials, double *result, int blockSize, int datasetSize,
                      int sharedMemSize)
{
    (void)residueCount, (void)moleculePositions, (void)moleculeCount, (void)LJPotentials, (void)blockSize,
        (void)sharedMemSize;
    eon_device_sync(true, residuePositions, residueMeta, result, datasetSize);
}

// Reference src/CudaFunctions.cu:176-190.  The caller owns `device_result`
// (resultSize*resultSize floats) and sums it after syncing `stream`; this writes the
// total to element 0 and zero everywhere else, which sums to the same value.
void CUDA_EonDevice_async(float4 *residuePositions, float4 *residueMeta, int *residueCount, int *moleculePositions,
                          int *moleculeCount, float *LJPotentials, float *device_result, int resultSize,
                          int blockSize, int datasetSize, int sharedMemSize, cudaStream_t stream)
{
    (void)residueCount, (void)moleculePositions, (void)moleculeCount, (void)LJPotentials, (void)blockSize,
        (void)sharedMemSize;
    if (datasetSize <= 0 || resultSize <= 0)
        return;
    std::lock_guard<std::mutex> lock(g_mu);
    const float *table = bound_table();
    if (table == nullptr) {
        cgppd_fail("CUDA_EonDevice_async: no contact table bound (call bindLJTexture first)");
        return;
    }
    const int nt = (datasetSize + kTile - 1) / kTile;
    Scratch *s = scratch_for(stream, (size_t)energy_ctas(nt));
    if (s == nullptr)
        return;
    launch_energy(false, residuePositions, residueMeta, datasetSize, table, s, device_result,
                  resultSize * resultSize, stream);
}

// The reference selects the crowder potential at compile time (REPULSIVE_CROWDING,
// src/definitions.h:18; off in its default build); this library selects it at run
// time for every later energy call of the process: 0 (default) the full potential for
// crowder pairs, 1 the repulsive (6/r)^12 term below 15 A without Debye-Hueckel.
// Returns the previous setting.
int cgppd_set_repulsive_crowding(int on)
{
    return g_repulsive_crowding.exchange(on ? 1 : 0);
}

// Components of the last synchronous call on the current device (LJ raw, DH raw,
// total): a library extension used by the tests.
int cgppd_last_energy_components(double *out3)
{
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_scratch.find(std::make_pair(current_device(), cudaStreamLegacy));
    if (it == g_scratch.end())
        return -1;
    return cgppd_check(cudaMemcpy(out3, it->second.result, 3 * sizeof(double), cudaMemcpyDeviceToHost),
                       "component copy");
}

}  // extern "C"

// ------------------------------------------------------------------ allocation-free variant
//
// Some hosts of this library cannot allocate device memory while they evaluate
// energies: code that runs inside another framework's memory pool or under a fixed
// device-memory budget, and callers that must not introduce allocation calls into a
// timed or real-time loop.  CUDA_EonDevice_noalloc gives them the CUDA_EonDevice
// result without any allocation: its scratch (CTA partials, completion ticket, error
// flags, result slot) is a file-scope __device__ array, which every GPU that loads the
// library holds until the process exits.
namespace {

constexpr int kNoAllocMaxResidues = 16384;                       // datasetSize limit
constexpr int kNoAllocMaxTiles = kNoAllocMaxResidues / kTile;    // 128-residue tiles
constexpr int kNoAllocMaxCtas = 8384;                            // CTAs the array has room for
constexpr size_t kNoAllocBytes = scratch_bytes(kNoAllocMaxCtas);  // 139,896 bytes (layout: scratch_view)
static_assert(kNoAllocBytes == 139896, "the documented size of the static scratch");
constexpr bool no_alloc_fits()
{
    for (int nt = 1; nt <= kNoAllocMaxTiles; ++nt)
        if (energy_ctas(nt) > kNoAllocMaxCtas)
            return false;
    return true;
}
static_assert(no_alloc_fits(), "every accepted size fits the static scratch");

__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
// Calls on one device share that device's array and are serialised; each device has
// its own copy of the array, so calls on different devices do not wait for each other.
std::mutex g_noalloc_mu[kMaxDevices];

// In host code g_noalloc_scratch names a host-side stand-in, not device memory; the
// kernel needs the device address, looked up with the device current.  The lookup
// allocates nothing and is repeated on every call, so the address stays valid after a
// cudaDeviceReset (which reloads the module, possibly elsewhere); the first lookup on a
// device also loads the library's device code there.
unsigned char *noalloc_scratch()
{
    void *p = nullptr;
    if (cgppd_check(cudaGetSymbolAddress(&p, g_noalloc_scratch), "CUDA_EonDevice_noalloc set-up") != 0)
        return nullptr;
    return static_cast<unsigned char *>(p);
}

}  // namespace

extern "C" {

// Same arguments and result as CUDA_EonDevice.  The first call on a device loads the
// library's device code there if nothing else has, and should come before any stream
// capture.  datasetSize above 16384 residues is rejected with an error (result 0).
// Every call on a device shares that device's array and leaves the last call's data in
// it; the ticket and error flags are cleared before each launch.  Two calls whose
// kernels overlap on the GPU would race on the array: this function holds a per-device
// lock and returns only after its kernel and result copy have finished, so calls made
// through it on one device do not overlap.
void CUDA_EonDevice_noalloc(float4 *residuePositions, float4 *residueMeta, int *residueCount,
                            int *moleculePositions, int *moleculeCount, float *LJPotentials, double *result,
                            int blockSize, int datasetSize, int sharedMemSize)
{
    (void)residueCount, (void)moleculePositions, (void)moleculeCount, (void)LJPotentials, (void)blockSize,
        (void)sharedMemSize;
    *result = 0.0;
    if (datasetSize <= 0)
        return;
    if (datasetSize > kNoAllocMaxResidues) {
        cgppd_fail("CUDA_EonDevice_noalloc: datasetSize exceeds the 16384-residue limit of its static scratch");
        return;
    }
    const int dev = current_device();
    if (dev < 0 || dev >= kMaxDevices) {
        cgppd_fail("CUDA_EonDevice_noalloc: device ordinal above 63");
        return;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu[dev]);
    const float *table = nullptr;
    {
        std::lock_guard<std::mutex> tlock(g_mu);
        table = bound_table();
    }
    if (table == nullptr) {
        cgppd_fail("CUDA_EonDevice_noalloc: no contact table bound (call bindLJTexture first)");
        return;
    }
    unsigned char *base = noalloc_scratch();
    if (base == nullptr)
        return;
    Scratch s;
    scratch_view(base, kNoAllocMaxCtas, s);
    if (cgppd_check(cudaMemsetAsync(base, 0, 8, cudaStreamLegacy), "CUDA_EonDevice_noalloc clear") != 0 ||
        cgppd_check(cudaMemsetAsync(s.gtickets, 0, 4 * scratch_groups(kNoAllocMaxCtas), cudaStreamLegacy),
                    "CUDA_EonDevice_noalloc clear") != 0)
        return;
    if (launch_energy(false, residuePositions, residueMeta, datasetSize, table, &s, nullptr, 0, cudaStreamLegacy) != 0)
        return;
    double host[4];
    if (cgppd_check(cudaMemcpy(host, s.result, sizeof(host), cudaMemcpyDeviceToHost), "CUDA_EonDevice_noalloc copy") != 0)
        return;
    if (host[3] != 0.0) {
        cgppd_fail("CUDA_EonDevice_noalloc: residue type index outside the 20x20 table");
        return;
    }
    *result = host[2];
}

}  // extern "C"
