// Device-side pair arithmetic shared by the cluster-list force kernels and
// the reference-layout kernels: the packed FP32x2 LJ + screened-Coulomb pair
// function, the exact 22-bit cluster-centre difference, warp reductions and
// the PME excluded-pair kernel h(x).
#pragma once

#include "common.cuh"
#include "ewald_fit.h"

namespace spgnb
{
namespace
{

constexpr float kTwoPow32 = 4294967296.0f;

__device__ __forceinline__ float3 pair_offset(float ex, float ey, float ez, float4 pi, float4 pj, bool image,
                                              const SysDesc& D)
{
    float dx = (ex - pi.x) + pj.x;
    float dy = (ey - pi.y) + pj.y;
    float dz = (ez - pi.z) + pj.z;
    if (image)
    {
        const float sx = rintf(dx * D.rcell.a11 + dy * D.rcell.a21 + dz * D.rcell.a31);
        const float sy = rintf(dy * D.rcell.a22 + dz * D.rcell.a32);
        const float sz = rintf(dz * D.rcell.a33);
        dx -= sx * D.cell.a11 + sy * D.cell.a21 + sz * D.cell.a31;
        dy -= sy * D.cell.a22 + sz * D.cell.a32;
        dz -= sz * D.cell.a33;
    }
    return make_float3(dx, dy, dz);
}

// ------------------------------------------------ packed FP32x2 pair math
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// Fixed (c, c) constants of the packed arithmetic in constant memory, so the
// FP32x2 instructions read them as constant-bank operands instead of
// building register pairs each time.
static __constant__ float2 kPk[1] = {{-1.0f, -1.0f}};
enum PackedConst
{
    kPkMinusOne = 0
};
// pair_scalar2's LJ energy is -12 times the energy (A/(12 r^12) - B/(6 r^6))
// and its Coulomb energy -1 times the energy: the kernels scale the sums once
constexpr float kLjEnergyScale = -1.0f / 12.0f;
constexpr float kCoulombEnergyScale = -1.0f;

// Degree-5 polynomials by Horner's rule.  The packed instruction takes one
// constant operand, so the numerator's leading coefficient comes in a
// register (lead) and the denominator is monic.
__device__ __forceinline__ float2 polyx2(float2 x, float2 lead, const float2 (&c)[6])
{
    float2 p = __ffma2_rn(lead, x, c[4]);
    p = __ffma2_rn(p, x, c[3]);
    p = __ffma2_rn(p, x, c[2]);
    p = __ffma2_rn(p, x, c[1]);
    return __ffma2_rn(p, x, c[0]);
}

__device__ __forceinline__ float2 polyx2_monic(float2 x, const float2 (&c)[6])
{
    float2 p = __fadd2_rn(x, c[4]);
    p = __ffma2_rn(p, x, c[3]);
    p = __ffma2_rn(p, x, c[2]);
    p = __ffma2_rn(p, x, c[1]);
    return __ffma2_rn(p, x, c[0]);
}

// v where the list word pairs the atom (w & bit) and r2 is inside the cutoff,
// else 0: the bit test, the comparison and their conjunction in two
// instructions (a logic operation with a predicate result).
__device__ __forceinline__ float inside_or_zero(float v, float r2, float rc2, unsigned w, unsigned bit)
{
    float o;
    asm("{\n\t.reg .pred p, q;\n\t.reg .b32 d;\n\t"
        "setp.lt.f32 q, %2, %3;\n\t"
        "lop3.and.b32 d|p, %4, %5, 0, 0xC0, q;\n\t"
        "selp.f32 %0, %1, 0f00000000, p;\n\t}"
        : "=f"(o)
        : "f"(v), "f"(r2), "f"(rc2), "r"(w), "r"(bit));
    return o;
}

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The hardware approximations with subnormals flushed (PTX rsqrt.approx.ftz,
// rcp.approx.ftz), without the range handling of rsqrtf and __fdividef: r^2
// of a listed pair is far from the subnormal range.  So are the fits' monic
// denominators and their reciprocals: in w they lie between 0.028 and 7.3, in
// r^2 they are divided by the fifth power of the scale of w, which the choice
// between the two forms keeps at 1e-6 or more (launch_pair_ft): 7.3e30 at
// most, its reciprocal 1.4e-31.
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A fit's numerator and (monic) denominator as polynomials in r^2, (c, c) pairs.
struct EwaldPoly
{
    float2 p[6], q[6];
};

// One system's pair-function parameters as (v, v) pairs, made once per atom
// pair and kept in registers over its list.
struct PairParams2
{
    float2 w_scale, nbeta3, nbeta, beta_2_sqrtpi, nb2_log2e;
    float rc2, beta;
};

__device__ __forceinline__ PairParams2 pack_params(const ForceParams& pc)
{
    PairParams2 q;
    q.w_scale = f2(pc.w_scale);
    q.nbeta3 = f2(-pc.beta3);
    q.nbeta = f2(-pc.beta);
    q.beta_2_sqrtpi = f2(pc.beta * 1.1283791670955126f);
    q.nb2_log2e = f2(-pc.beta * pc.beta * 1.4426950408889634f);  // -w log2(e) = -beta^2 r^2 log2(e)
    q.rc2 = pc.rc2;
    q.beta = pc.beta;
    return q;
}

// pair_scalar for two pairs at once; nA = -A, nqq = -q_i q_j (the kernels keep
// a cluster's charges negated), so that the Coulomb term joins the LJ term in
// one fused multiply-add.  Without energies the screened Coulomb force uses
// the K fit; with energies it uses the M fit and exp(-w):
// beta^3 K(w) = beta (M(w) - 2/sqrt(pi) exp(-w)) / r^2, so
//   F_c/qq = (t + beta 2/sqrt(pi) exp(-w)) / r^2,  E_c/qq = t,  t = 1/r - beta M(w).
// e_lj comes out as -12 E_lj and e_c as -E_c; the kernels scale the sums once.
// FIT 1: the fits in w / W_MAX; FIT 2: the same fits as polynomials in r^2
// with -beta^3 (K) or -beta (M) in the numerator, ep, made for the one system
// of a call: two packed instructions fewer a pair.  FIT 0: erfc.
// lead: the numerator's leading coefficient (fit_lead).
template <bool ENERGY, int FIT>
__device__ __forceinline__ float2 fit_lead(const EwaldPoly& ep)
{
    float2 l = FIT == 2 ? ep.p[5] : (ENERGY ? kEwaldMP2[5] : kEwaldKP2[5]);
    // opaque, so that it stays in registers over the list instead of being
    // moved there for every pair
    asm volatile("" : "+f"(l.x), "+f"(l.y));
    return l;
}

template <bool ENERGY, int FIT>
__device__ __forceinline__ float2 pair_scalar2(float2 r2, float2 nqq, float2 nA, float2 B, const PairParams2& pc,
                                               const EwaldPoly& ep, float2 lead, float2& e_lj, float2& e_c)
{
    // the hardware reciprocal square root alone: a Newton step on top of it
    // moves the forces' error against FP64 by 1e-8 relative RMS and costs
    // four packed instructions a word
    const float2 rinv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 r2inv = __fmul2_rn(rinv, rinv);
    const float2 r3inv = __fmul2_rn(rinv, r2inv);
    const float2 r6inv = __fmul2_rn(r3inv, r3inv);
    // u = (-A/r^6 + B)/r^6 serves the force and, plus B/r^6, the energy
    const float2 u = __fmul2_rn(__ffma2_rn(nA, r6inv, B), r6inv);
    if (ENERGY) e_lj = __ffma2_rn(B, r6inv, u);  // -A/r^12 + 2B/r^6 = -12 E_lj
    if (FIT != 0)
    {
        float2 s;  // K: 1/r^3 - beta^3 K;  M: t
        if (FIT == 2)
        {
            const float2 q = polyx2_monic(r2, ep.q);
            s = __ffma2_rn(polyx2(r2, lead, ep.p), make_float2(rcp_approx(q.x), rcp_approx(q.y)), ENERGY ? rinv : r3inv);
        }
        else
        {
            const float2 x = __fmul2_rn(r2, pc.w_scale);
            const float2 p = ENERGY ? polyx2(x, lead, kEwaldMP2) : polyx2(x, lead, kEwaldKP2);
            const float2 q = ENERGY ? polyx2_monic(x, kEwaldMQ2) : polyx2_monic(x, kEwaldKQ2);
            const float2 k = __fmul2_rn(p, make_float2(rcp_approx(q.x), rcp_approx(q.y)));
            s = ENERGY ? __ffma2_rn(pc.nbeta, k, rinv) : __ffma2_rn(pc.nbeta3, k, r3inv);
        }
        if (!ENERGY) return __ffma2_rn(nqq, s, __fmul2_rn(u, r2inv));
        const float2 wl = __fmul2_rn(r2, pc.nb2_log2e);
        const float2 E = make_float2(ex2_approx(wl.x), ex2_approx(wl.y));
        e_c = __fmul2_rn(nqq, s);
        return __fmul2_rn(r2inv, __ffma2_rn(nqq, __ffma2_rn(pc.beta_2_sqrtpi, E, s), u));
    }
    float c[2], e[2];
    const float rr[2] = {r2.x, r2.y}, ri[2] = {rinv.x, rinv.y}, q[2] = {nqq.x, nqq.y};
    for (int h2 = 0; h2 < 2; h2++)
    {
        const float r = rr[h2] * ri[h2];
        const float br = pc.beta * r;
        const float erfcv = erfcf(br);
        c[h2] = q[h2] * ri[h2] * ri[h2] * ri[h2] * __fmaf_rn(br * 1.1283791670955126f, __expf(-br * br), erfcv);
        e[h2] = q[h2] * erfcv * ri[h2];
    }
    if (ENERGY) e_c = make_float2(e[0], e[1]);
    return __fadd2_rn(__fmul2_rn(u, r2inv), make_float2(c[0], c[1]));
}

// A difference of two 22-bit cluster-centre coordinates, wrapped to
// [-2^21, 2^21) (minimum image of the centres) and converted exactly: the
// wrapped value plus 2^23 + 2^21 is an integer below 2^23 + 2^22, whose float
// bit pattern is 0x4B000000 | value.
__device__ __forceinline__ float centre_step(int qj, int qi)
{
    return __int_as_float(((qj - qi + 0x200000) & 0x3fffff) | 0x4b000000) - 10485760.0f;
}


__device__ __forceinline__ void load_rec(const SlotRec* r, float4& pos, int4& aux)
{
    pos = r->pos;
    aux = r->aux;
}

// Adds to a 64-bit sum in global memory without reading it back (the compiler
// makes a returning ATOMG of an unused atomicAdd here).
__device__ __forceinline__ void red_add(long long* p, long long v)
{
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sums eight per-lane FP32 values over the warp in FP64: lanes 4r..4r+3
// return the total of v[r].  The values are transposed through shared memory
// (rows padded to 36 floats, so that the lanes' 16-byte reads fall on
// different banks): lane 4r + k adds eight lanes' share of row r, and two
// exchanges join the four parts.  33 instructions, where the same sum as
// int64 values by shuffles takes about 110.  buf: 8 * kSumRow floats.
constexpr int kSumRow = 36;
__device__ __forceinline__ double lane_totals8(float* buf, const float (&v)[8], int lane)
{
    __syncwarp();  // the buffer's last use
#pragma unroll
    for (int r = 0; r < 8; r++) buf[r * kSumRow + lane] = v[r];
    __syncwarp();
    const float4* row = reinterpret_cast<const float4*>(buf + (lane >> 2) * kSumRow + (lane & 3) * 8);
    const float4 x = row[0], y = row[1];
    double s = (((double)x.x + (double)x.y) + ((double)x.z + (double)x.w)) +
               (((double)y.x + (double)y.y) + ((double)y.z + (double)y.w));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s;
}

// PME excluded-pair correction (Particle_Mesh::PME_Excluded_Force_With_Atom_Energy,
// PM_force.cpp:918-997): reciprocal space includes every pair, excluded ones
// too, so their smooth part erf(beta r)/r is taken back out.  One thread per
// atom walks its (upper-triangular) exclusion list, as the reference does:
//   dr = min image(r_j - r_i),  x = beta r,
//   F_i += q_i q_j beta^3 h(x) dr,  F_j -= the same,  E_i -= q_i q_j erf(x)/r,
//   W_i -= F (x) dr (the reference's symmetric virial form),
// with h(x) = (erf(x) - 2/sqrt(pi) x exp(-x^2)) / x^3.  Below x = 0.7, h is
// summed from its Taylor series (the series of erf and of x exp(-x^2)
// combined: h = 2/sqrt(pi) sum_{n>=1} (-1)^(n+1) 2n x^(2n-2) / ((2n+1) n!))
// instead of the difference of two nearly equal numbers, so the correction
// keeps FP32 precision at bonded distances.  Forces accumulate in int64 fixed
// point (the partner's share by atomics), the energy total likewise, so the
// result does not depend on the order.
__device__ __forceinline__ float excl_h(float x)
{
    const float x2 = x * x;
    if (x < 0.7f)
    {
        // 2/sqrt(pi) * (2/3 - 2/5 x^2 + 1/7 x^4 - 1/27 x^6 + 1/132 x^8 - 1/780 x^10 + 1/5400 x^12
        //               - 1/42840 x^14)
        float p = -1.0f / 42840.0f;
        p = __fmaf_rn(p, x2, 1.0f / 5400.0f);
        p = __fmaf_rn(p, x2, -1.0f / 780.0f);
        p = __fmaf_rn(p, x2, 1.0f / 132.0f);
        p = __fmaf_rn(p, x2, -1.0f / 27.0f);
        p = __fmaf_rn(p, x2, 1.0f / 7.0f);
        p = __fmaf_rn(p, x2, -0.4f);
        p = __fmaf_rn(p, x2, 2.0f / 3.0f);
        return 1.1283791670955126f * p;
    }
    return (erff(x) - 1.1283791670955126f * x * expf(-x2)) / (x2 * x);
}

}  // namespace
}  // namespace spgnb
