// pair_terms.cuh -- Kim-Hummer pair terms two at a time in packed FP32 arithmetic, shared by
// the Monte Carlo engine and the drop-in energy kernel.
#pragma once

#include "cgppd_common.cuh"

namespace cgppd {

// ------------------------------------------------------------------ packed pairs
// Two FP32 values in one 64-bit register pair.  The packed add, multiply and fma round
// each half as the scalar instruction does; an FMA pipe takes two cycles for one, so the
// FP32 peak is the scalar one, but a loop that is bound by issue slots (28 of them per
// Lennard-Jones pair, 14 on the FMA pipes) gets half of its arithmetic slots back.
typedef unsigned long long f2;

__device__ __forceinline__ f2 f2_pack(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ f2 f2_dup(float v) { return f2_pack(v, v); }

__device__ __forceinline__ void f2_unpack(f2 v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// ------------------------------------------------------------------ pair terms

// Two Lennard-Jones terms (m4 (s6^2 - s6), the repulsive branch left to repulsive2) and what the Debye-Hueckel terms need.
struct Pair2 {
    f2 u, r2, inv, m4, s6;
};

// min_image of two differences; nL holds -L.
__device__ __forceinline__ f2 min_image2(f2 d, f2 nL, f2 invL)
{
    return f2_fma(nL, f2_add(f2_fma(d, invL, f2_dup(12582912.0f)), f2_dup(-12582912.0f)), d);
}

__device__ __forceinline__ Pair2 lj2(f2 dx, f2 dy, f2 dz, f2 sigma, f2 m4)
{
    Pair2 p;
    p.r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
    float ra, rb;
    f2_unpack(p.r2, ra, rb);
    p.inv = f2_pack(rsqrt_sfu(ra), rsqrt_sfu(rb));
    p.m4 = m4;
    const f2 so = f2_mul(sigma, p.inv), s2 = f2_mul(so, so);
    p.s6 = f2_mul(f2_mul(s2, s2), s2);
    float sa, sb;
    f2_unpack(p.s6, sa, sb);
    p.u = f2_mul(m4, f2_fma(p.s6, p.s6, f2_pack(-sa, -sb)));
    return p;
}

// 1/x on the SFU (PTX rcp.approx.ftz.f32, max relative error about 2^-23).
__device__ __forceinline__ float rcp_sfu(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two Lennard-Jones terms from sigma^2 / r^2.  DH: 1 / r^2 as the square of the rsqrt that
// the Debye-Hueckel term needs anyway; otherwise the SFU reciprocal of r^2, whose error
// enters s6 three times where the rsqrt's enters six times.
template <bool DH>
__device__ __forceinline__ Pair2 lj2_sq(f2 dx, f2 dy, f2 dz, f2 sigma, f2 m4)
{
    Pair2 p;
    p.r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
    float ra, rb;
    f2_unpack(p.r2, ra, rb);
    p.inv = DH ? f2_pack(rsqrt_sfu(ra), rsqrt_sfu(rb)) : f2_pack(rcp_sfu(ra), rcp_sfu(rb));
    p.m4 = m4;
    const f2 s2 = f2_mul(f2_mul(sigma, sigma), DH ? f2_mul(p.inv, p.inv) : p.inv);
    p.s6 = f2_mul(f2_mul(s2, s2), s2);
    float sa, sb;
    f2_unpack(p.s6, sa, sb);
    p.u = f2_mul(m4, f2_fma(p.s6, p.s6, f2_pack(-sa, -sb)));
    return p;
}

// The larger s6 of the two pairs: above 1/2 (closer than 2^(1/6) sigma) one may lie in the
// repulsive branch's range; rare, so the branch is taken out of the straight path.
__device__ __forceinline__ float closest2(const Pair2 &p)
{
    float a, b;
    f2_unpack(p.s6, a, b);
    return fmaxf(a, b);
}

__device__ __forceinline__ void repulsive2(Pair2 &p)
{
    float a, b, ma, mb, ua, ub;
    f2_unpack(p.s6, a, b);
    f2_unpack(p.m4, ma, mb);
    f2_unpack(p.u, ua, ub);
    if (ma < 0.0f && a > 0.5f)
        ua = fmaf(-0.5f, ma, -ua);
    if (mb < 0.0f && b > 0.5f)
        ub = fmaf(-0.5f, mb, -ub);
    p.u = f2_pack(ua, ub);
}

// The Debye-Hueckel terms, qq = q_i q_j of each pair.
__device__ __forceinline__ f2 dh2(const Pair2 &p, f2 qq)
{
    const f2 arg = f2_mul(f2_mul(p.r2, p.inv), f2_dup(-kLog2e / kXi));
    float ea, eb;
    f2_unpack(arg, ea, eb);
    return f2_mul(f2_mul(qq, f2_pack(ex2_sfu(ea), ex2_sfu(eb))), p.inv);
}

// The terms with the Debye-Hueckel part.
__device__ __forceinline__ f2 with_dh2(const Pair2 &p, f2 qq)
{
    const f2 arg = f2_mul(f2_mul(p.r2, p.inv), f2_dup(-kLog2e / kXi));
    float ea, eb;
    f2_unpack(arg, ea, eb);
    return f2_fma(f2_mul(qq, f2_pack(ex2_sfu(ea), ex2_sfu(eb))), p.inv, p.u);
}

}  // namespace cgppd
