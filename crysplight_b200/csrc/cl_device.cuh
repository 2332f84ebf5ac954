// cl_device.cuh — device-side building blocks of the transport engine:
// Philox4x32-10 streams, Float32 elementary functions, and the per-photon
// physics primitives the transport kernel's state machine composes.
//
// Arithmetic contract (what makes results identical to the reference's CPU
// transport, src/transport.jl):
//   * compiled with --fmad=false: no multiply-add contraction, every float
//     operation rounds once as in Julia;
//   * IEEE division and square root (no fast-math);
//   * log/sin/cos of Float32 arguments are evaluated in Float64 and rounded
//     once to Float32 (see cl_logf / cl_sincosf);
//   * expressions keep the reference's association and draw order.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "cl_tables.h"

namespace cl {

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11), as keyed in src/philox.jl:5-28.
// ---------------------------------------------------------------------------
constexpr uint32_t PHILOX_M0 = 0xD2511F53u;
constexpr uint32_t PHILOX_M1 = 0xCD9E8D57u;
constexpr uint32_t PHILOX_W0 = 0x9E3779B9u;
constexpr uint32_t PHILOX_W1 = 0xBB67AE85u;

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)PHILOX_M0 * c.x;   // IMAD.WIDE.U32
        const uint64_t p1 = (uint64_t)PHILOX_M1 * c.z;
        const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += PHILOX_W0;
        k1 += PHILOX_W1;
    }
    return c;
}

// The same rounds with the key schedule (k0 + r*W0, k1 + r*W1, r = 0..9)
// precomputed: rk[2r], rk[2r+1].  With rk in the constant bank the XORs take
// their key operand straight from it.
__device__ __forceinline__ uint4 philox4x32_10_rk(uint4 c, const uint32_t* __restrict__ rk)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)PHILOX_M0 * c.x;
        const uint64_t p1 = (uint64_t)PHILOX_M1 * c.z;
        const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
        c = make_uint4(hi1 ^ c.y ^ rk[2 * r], lo1, hi0 ^ c.w ^ rk[2 * r + 1], lo0);
    }
    return c;
}

// randu, src/philox.jl:62: ((x >>> 8) + 1.0f0) * 2^-24, exact, in (0, 1].
// (x >> 8) < 2^24 converts exactly, and (f + 1) * 2^-24 = f * 2^-24 + 2^-24 is
// representable, so one fused multiply-add gives the same bits as the
// reference's add then multiply (neither rounds).
__device__ __forceinline__ float u32_to_randu(uint32_t x)
{
    return __fmaf_rn((float)(x >> 8), 0x1p-24f, 0x1p-24f);
}

// A photon's uniform stream (PhiloxStream, src/philox.jl:34-62): key = seed,
// counter = (pid lo, pid hi, block, 0).  The uniforms are buffered, already
// converted by randu, in a per-lane ring of 32 floats in shared memory (rings
// of 28, 36, 40 and 48 words measured 3-15% slower on the BGO+ESR scan): word i
// of the lane at column tid sits in row i % 32, every access free of bank
// conflicts.  Blocks are generated ahead of use, two at a time, at one
// convergent point of the warp loop, and consumed in order, so the sequence of
// uniforms is exactly the reference's.
//
// An iteration consumes at most 7 uniforms and reads them at fixed byte
// offsets 0 .. 6 RING_ROW from its first one: rows 0..5 are stored a second
// time in rows 32..37, so that no read wraps and an offset is an immediate of
// the load instead of an add, a compare and a select per uniform.
constexpr uint32_t RING_ROW = 1024;           // bytes: 256 columns, the largest block the kernels launch
constexpr int RING_ROWS = 38;
constexpr uint32_t RING_BYTES = RING_ROWS * RING_ROW;
constexpr uint32_t RING_MASK = 32 * RING_ROW - 1;
constexpr int DRAWS_PER_ITER = 7;

struct Rng {
    uint32_t pid_lo, pid_hi;
    uint32_t block;          // blocks generated (4 uniforms each)
    uint32_t pos;            // uniforms consumed x RING_ROW + 4 tid: the next uniform is at pos & RING_MASK
};

__device__ __forceinline__ void rng_init(Rng& r, uint64_t pid)
{
    r.pid_lo = (uint32_t)pid;
    r.pid_hi = (uint32_t)(pid >> 32);
    r.block = 0;
    r.pos = 4u * threadIdx.x;
}

// Buffered uniforms x RING_ROW - 4 tid (0 <= 4 tid < RING_ROW); both counts
// wrap, their difference does not.
__device__ __forceinline__ int32_t rng_level(const Rng& r)
{
    return (int32_t)(r.block * (4u * RING_ROW) - r.pos);
}
// A lane without a photon: neither short of uniforms nor with room for more.
__device__ __forceinline__ void rng_park(Rng& r) { r.pos = (r.block * 4u - 28u) * RING_ROW; }
__device__ __forceinline__ bool rng_short(const Rng& r) { return rng_level(r) <= (DRAWS_PER_ITER - 1) * (int32_t)RING_ROW; }
__device__ __forceinline__ bool rng_room(const Rng& r) { return rng_level(r) <= 24 * (int32_t)RING_ROW; }
__device__ __forceinline__ bool rng_under(const Rng& r) { return rng_level(r) <= -(int32_t)RING_ROW; }

// Ring accesses by 32-bit shared address (volatile: a read stays behind the
// fill that stored it).
__device__ __forceinline__ float ring_word(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void ring_store(uint32_t a, float v)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v));
}

// Two consecutive blocks at once (independent Philox chains interleave); needs
// rng_room.  The write row is a multiple of 8: the stores never wrap.
__device__ __forceinline__ void rng_fill(Rng& r, uint32_t ring, const uint32_t* rk)
{
    const uint4 o = philox4x32_10_rk(make_uint4(r.pid_lo, r.pid_hi, r.block, 0u), rk);
    const uint4 q = philox4x32_10_rk(make_uint4(r.pid_lo, r.pid_hi, r.block + 1u, 0u), rk);
    const uint32_t row = (r.block * (4u * RING_ROW)) & RING_MASK;
    const uint32_t a = ring + row + 4u * threadIdx.x;
    const float f[8] = {u32_to_randu(o.x), u32_to_randu(o.y), u32_to_randu(o.z), u32_to_randu(o.w),
                        u32_to_randu(q.x), u32_to_randu(q.y), u32_to_randu(q.z), u32_to_randu(q.w)};
#pragma unroll
    for (int i = 0; i < 8; ++i) ring_store(a + i * RING_ROW, f[i]);
    if (row == 0u) {
#pragma unroll
        for (int i = 0; i < RING_ROWS - 32; ++i) ring_store(a + (32 + i) * RING_ROW, f[i]);
    }
    r.block += 2u;
}

// A register-only stream for the diagnostics kernel (same sequence).
struct SimpleStream {
    uint32_t pid_lo, pid_hi, block, b0, b1, b2, b3;
    int n;
};

__device__ __forceinline__ float simple_randu(SimpleStream& s, uint32_t k0, uint32_t k1)
{
    if (s.n == 0) {
        const uint4 o = philox4x32_10(make_uint4(s.pid_lo, s.pid_hi, s.block, 0u), k0, k1);
        s.block += 1u;
        s.b0 = o.x; s.b1 = o.y; s.b2 = o.z; s.b3 = o.w;
        s.n = 4;
    }
    const uint32_t x = s.b0;
    s.b0 = s.b1; s.b1 = s.b2; s.b2 = s.b3;
    s.n -= 1;
    return u32_to_randu(x);
}

// ---------------------------------------------------------------------------
// Float32 elementary functions.  Each is evaluated in Float64 to about 2^-51
// relative error and rounded once, so it returns the correctly rounded
// Float32 except when the exact value lies within ~2^-51 of a rounding
// boundary.  Arguments outside the transport's domain take a slow path
// through the CUDA double-precision library functions.
// ---------------------------------------------------------------------------

// Out-of-domain arguments (never reached by the transport): CUDA's Float64
// functions, kept out of line so the hot loop stays small.
static __device__ __noinline__ float slow_logf(float x) { return __double2float_rn(log((double)x)); }
static __device__ __noinline__ float2 slow_sincosf(float x)
{
    const double xd = (double)x;
    return make_float2(__double2float_rn(sin(xd)), __double2float_rn(cos(xd)));
}

// Natural log.  Table-driven (Tang 1990): x = 2^e * m, m in [sqrt(1/2), sqrt(2)),
// m = F_j (1 + r) with F_j = 1 + j/64, ln x = e ln2 + ln F_j + log1p(r),
// |r| < 1/90, log1p by its Taylor series to r^8.
__device__ __forceinline__ float cl_logf(float x, const double2* __restrict__ tab)
{
    const uint32_t b = __float_as_uint(x);
    if (b - 0x00800000u >= 0x7f000000u)       // not a positive normal finite float
        return slow_logf(x);
    int e = (int)(b >> 23) - 127;
    uint32_t mb = b & 0x007fffffu;
    const int hi = mb >= 0x3504f3u;          // m >= sqrt(2): use m/2, e+1
    e += hi;
    mb |= hi ? 0x3f000000u : 0x3f800000u;
    const double m = (double)__uint_as_float(mb);
    const int j = __double2int_rn((m - 1.0) * 64.0);
    const double F = 1.0 + (double)j * 0.015625;
    const double2 t = tab[j - CLM_LOG_JMIN];
    const double r = (m - F) * t.x;            // m - F is exact
    double p = CLM_L8;
    p = fma(p, r, CLM_L7);
    p = fma(p, r, CLM_L6);
    p = fma(p, r, CLM_L5);
    p = fma(p, r, CLM_L4);
    p = fma(p, r, CLM_L3);
    p = fma(p, r, CLM_L2);
    const double lp = fma(p * r, r, r);        // log1p(r)
    const double res = fma((double)e, CLM_LN2, t.y) + lp;
    return __double2float_rn(res);
}

// log of a uniform ((x>>8)+1)*2^-24: always a positive normal float, so the
// domain check of cl_logf is not needed.
__device__ __forceinline__ float cl_logf_u(float x, const double2* __restrict__ tab)
{
    const uint32_t b = __float_as_uint(x);
    int e = (int)(b >> 23) - 127;
    uint32_t mb = b & 0x007fffffu;
    const int hi = mb >= 0x3504f3u;
    e += hi;
    mb |= hi ? 0x3f000000u : 0x3f800000u;
    const double m = (double)__uint_as_float(mb);
    const int j = __double2int_rn((m - 1.0) * 64.0);
    const double F = 1.0 + (double)j * 0.015625;
    const double2 t = tab[j - CLM_LOG_JMIN];
    const double r = (m - F) * t.x;
    double p = CLM_L8;
    p = fma(p, r, CLM_L7);
    p = fma(p, r, CLM_L6);
    p = fma(p, r, CLM_L5);
    p = fma(p, r, CLM_L4);
    p = fma(p, r, CLM_L3);
    p = fma(p, r, CLM_L2);
    const double lp = fma(p * r, r, r);
    const double res = fma((double)e, CLM_LN2, t.y) + lp;
    return __double2float_rn(res);
}

// sin and cos together, table-driven, for the azimuths 2*pi*u in (0, 2*pi] and
// the facet tilts in [0, 1.2): x = j/64 + r with |r| <= 1/128.  j/64 and r are
// exact in Float32 (j/64 is a multiple of x's last place and r is smaller than
// x), so the reduction is three Float32 operations and only r is widened; a
// grid of multiples of 2*pi/256, which is not exact, took five Float64
// operations and two longer polynomials (20 Float64 operations in all, now
// 10; Float64 issues at half the Float32 rate).  (sin, cos)(j/64) come from a
// 404-entry table in shared memory, sin r and cos r - 1 from two-term
// polynomials (the last cosine term economised: 2^-56 of the result).  All
// 2^24 azimuths and every Float32 in [0, 1.2) round to the correctly rounded
// sine and cosine.  BGO + ESR scan (51.2M photons) 149.5 -> 143.9 ms, 3,001 CsI(Tl) events 33.4 -> 32.6 ms.
// The Float64 coefficients sit in the constant bank, so every Float64
// instruction takes its coefficient as an operand (a 64-bit immediate cannot
// be encoded and would first be moved into registers).
static __constant__ double c_sc_coef[4] = {CLM_TS5, CLM_TS3, CLM_TC4, CLM_TC2};

// 32-bit shared-memory addresses: through pointers the compiler derives the
// window's base again at every use in the transport loop.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cl_sincosf_core(float x, uint32_t sctab, float* sp, float* cp)
{
    // j = rint(64 x) by the 1.5*2^23 shift: the sum's bits are 0x4B400000 + j,
    // and 16 times them (mod 2^32) the table offset plus a constant
    const float sh = __fmaf_rn(x, 64.0f, 12582912.0f);
    const float rf = __fmaf_rn(sh - 12582912.0f, -0.015625f, x);
    double S, C;
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(S), "=d"(C) : "r"(__float_as_uint(sh) * 16u + (sctab - 0xB4000000u)));
    const double r = (double)rf;
    const double r2 = r * r;
    const double sr = fma(r * r2, fma(c_sc_coef[0], r2, c_sc_coef[1]), r);    // sin r
    const double cm1 = r2 * fma(c_sc_coef[2], r2, c_sc_coef[3]);              // cos r - 1
    *sp = __double2float_rn(fma(C, sr, fma(S, cm1, S)));
    *cp = __double2float_rn(fma(-S, sr, fma(C, cm1, C)));
}

// The same for any argument (diagnostics): outside the core's range, CUDA's
// Float64 functions.
__device__ __forceinline__ void cl_sincosf(float x, uint32_t sctab, float* sp, float* cp)
{
    if (!(x >= 0.0f && x <= 6.2831855f)) {
        const float2 sc = slow_sincosf(x);
        *sp = sc.x;
        *cp = sc.y;
        return;
    }
    if (x == 0.0f) {                           // sin(+-0) = +-0, cos(+-0) = 1
        *sp = x;
        *cp = 1.0f;
        return;
    }
    cl_sincosf_core(x, sctab, sp, cp);
}

// ---------------------------------------------------------------------------
// Transport parameters (flattened OpticalParams / Readout / TimeBinning / Box).
// ---------------------------------------------------------------------------
struct Physics {
    float L0, L1, L2;
    float n_crystal, n_coupling, abs_len, ray_len, wrap_R, sigma_alpha, pde;
    float inv_v;                 // n_crystal / c, ns per mm
    float cx, cy, r2, sur_R, pitch, bin_ns, tau;
    int32_t nx, ny, nbins, max_bounces;
    uint32_t key0, key1;
    uint32_t rk[20];             // Philox round keys
    float qc2, qa2;              // (n_crystal/n_coupling)^2, (n_crystal/1)^2
    float abs_rate, ray_rate;    // -log2(e) / length, NaN: no quick test (survive_below)
    float fresnel_margin;        // error bound of the quick Fresnel test, +Inf: no quick test
    uint8_t abs_finite, ray_finite, wrap_specular, air_gap;
    uint8_t disc, sur_specular, two_sided, pad_;
};

enum : int32_t { FACE_XP = 1, FACE_XM = 2, FACE_YP = 3, FACE_YM = 4, FACE_BACK = 5, FACE_FRONT = 6 };
enum : int32_t {
    ST_FLYING = 0, ST_DETECTED = 1, ST_ABS_BULK = 2, ST_ABS_WALL = 3,
    ST_ABS_SIPM = 4, ST_CAP = 5, ST_ABS_SUR = 6
};

constexpr float TWO_PI_F = 6.2831854820251465f;   // 2f0*Float32(pi), exact doubling
constexpr float C_MM_NS = 299.792458f;

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float ex2_approx(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Correctly rounded square root and reciprocal of arguments well inside the
// normal range (2^-40 .. 2^40; sqrt_mid also of 0), without the range tests and
// slow paths of the general functions: an approximation refined by residuals
// that are exact in a fused multiply-add (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1990)).  Both equal the IEEE operations for every Float32 mantissa
// (tested over all of them).
__device__ __forceinline__ float sqrt_mid(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(x, 0x1p-60f)));
    const float g = x * y, h = 0.5f * y;
    const float e = __fmaf_rn(-h, g, 0.5f);
    const float g1 = __fmaf_rn(g, e, g), h1 = __fmaf_rn(h, e, h);
    return __fmaf_rn(__fmaf_rn(-g1, g1, x), h1, g1);
}
__device__ __forceinline__ float rcp_mid(float x)
{
    const float r = rcp_approx(x);
    const float r1 = __fmaf_rn(r, __fmaf_rn(-x, r, 1.0f), r);
    return __fmaf_rn(r1, __fmaf_rn(-x, r1, 1.0f), r1);
}

// fresnel, src/optics.jl:10-19, where sin2t = (n1/n2)^2 (1 - cosi^2) < 1.
static __device__ __noinline__ float fresnel_R(float n1, float n2, float sin2t, float cosi)
{
    const float cost = sqrtf(1.0f - sin2t);
    const float a = (n1 * cosi - n2 * cost) / (n1 * cosi + n2 * cost);
    const float b = (n1 * cost - n2 * cosi) / (n1 * cost + n2 * cosi);
    return 0.5f * (a * a + b * b);
}

// Reflection at an interface: total, or u < R.  R is estimated with approximate
// reciprocals and root: the estimate and the reference's rounded R each lie
// within 2^-20 of the Fresnel formula in the same operands (a handful of
// relative errors of 2^-22 at most in quotients of magnitude <= 1), so outside
// fresnel_margin = 2^-17 the estimate decides; inside it (1.5e-5 of the
// draws) the exact expression does.  Two IEEE divisions and a root less, each
// with a branch of its own.
// The bound holds for indices in [1e-3, 1e3]; others always take the exact one.
__host__ __device__ inline float fresnel_margin(float n1, float n2)
{
    const bool plain = n1 >= 1e-3f && n1 <= 1e3f && n2 >= 1e-3f && n2 <= 1e3f;
    return plain ? 0x1p-17f : __builtin_inff();
}
__device__ __forceinline__ bool fresnel_reflects(const Physics& P, float n2, float sin2t, float cosi, float u)
{
    const bool tir = sin2t >= 1.0f;
    const float ct = sqrt_approx(1.0f - sin2t);        // NaN beyond the critical angle
    const float p = P.n_crystal * cosi, s = n2 * cosi;
    const float a = __fmaf_rn(-n2, ct, p) * rcp_approx(__fmaf_rn(n2, ct, p));
    const float b = __fmaf_rn(P.n_crystal, ct, -s) * rcp_approx(__fmaf_rn(P.n_crystal, ct, s));
    const float over = __fmaf_rn(0.5f, __fmaf_rn(a, a, b * b), -u);      // R - u
    bool refl = tir || over > 0.0f;
    if (!tir && !(fabsf(over) > P.fresnel_margin)) refl = u < fresnel_R(P.n_crystal, n2, sin2t, cosi);
    return refl;
}

// A bound below exp(-d / length) (rate = -log2(e) / length): a uniform u below
// it has -length log u > d in the reference's rounding too.  The exponent's
// and ex2's errors and that of the Float32 product length * log u stay below
// 2^-17 in log2 u wherever a uniform (>= 2^-24) can be below the bound; 2^-15
// is taken off.
// A length that is not positive gives NaN, for which no uniform is below the
// bound.
__host__ __device__ inline float survive_rate(float len)
{
    return len > 0.0f ? (float)(-1.4426950408889634 / (double)len) : __builtin_nanf("");
}
__device__ __forceinline__ float survive_below(float d, float rate)
{
    return ex2_approx(__fmaf_rn(d, rate, -0x1p-15f));
}

// v > L ? L : (v < 0 ? 0 : v), NaN kept, in two instructions.
__device__ __forceinline__ float clamp_to(float v, float L)
{
    float r;
    asm("{\n\t.reg .f32 m;\n\tmin.NaN.f32 m, %1, %2;\n\tmax.NaN.f32 %0, m, 0f00000000;\n\t}" : "=f"(r) : "f"(v), "f"(L));
    return r;
}

// Distance along one axis to the face the direction points at:
// u > 0 ? (L - p) / u : (u < 0 ? -p / u : Inf).  The numerator is selected
// first, so a warp whose lanes point both ways runs one division, not two.
__device__ __forceinline__ float axis_distance(float L, float p, float u)
{
    const float q = (u > 0.0f ? L - p : -p) / u;
    return (u > 0.0f || u < 0.0f) ? q : __int_as_float(0x7f800000);
}

// wall_hit, src/geometry.jl:19-32.
static __device__ __noinline__ int32_t wall_hit(const Physics& P, float x, float y, float z,
                                            float ux, float uy, float uz, float& d)
{
    const float dx = axis_distance(P.L0, x, ux);
    const float dy = axis_distance(P.L1, y, uy);
    const float dz = axis_distance(P.L2, z, uz);
    if (dx <= dy && dx <= dz) { d = dx; return ux > 0.0f ? FACE_XP : FACE_XM; }
    if (dy <= dz)             { d = dy; return uy > 0.0f ? FACE_YP : FACE_YM; }
    d = dz;
    return uz > 0.0f ? FACE_BACK : FACE_FRONT;
}

// wall_hit without its three IEEE divisions: the axis comes from approximate
// quotients, and only the winner's is made exact.  Returns false where the
// approximation does not decide (two axes within 2^-19 of each other, a
// distance or direction component near zero, positions outside the crystal,
// NaN): the caller then takes wall_hit.
//
// The quotient d = n/u: r = rcp(u) refined by one Newton step, q = n r, then
// q + r (n - q u) with the residual exact in a fused multiply-add, which is the
// correctly rounded quotient (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34
// (1990)) when r is the correctly rounded reciprocal: so it is for every
// Float32 mantissa but all-ones, which the theorem excludes and for which the
// exact expression is taken.  With m > 2^-30 and |u| > 2^-40 nothing
// under- or overflows.
__device__ __forceinline__ bool wall_hit_fast(const Physics& P, float x, float y, float z, float ux, float uy,
                                              float uz, float& d, int32_t& face, float& cosw)
{
    const float nx = (ux > 0.0f ? P.L0 : 0.0f) - x;
    const float ny = (uy > 0.0f ? P.L1 : 0.0f) - y;
    const float nz = (uz > 0.0f ? P.L2 : 0.0f) - z;
    const float qx = nx * rcp_approx(ux), qy = ny * rcp_approx(uy), qz = nz * rcp_approx(uz);
    const float lo = fminf(qx, qy), hi = fmaxf(qx, qy);
    const float m = fminf(lo, qz), second = fminf(hi, fmaxf(lo, qz));
    const bool on_x = qx == m, on_y = !on_x && qy == m;
    const float u = on_x ? ux : (on_y ? uy : uz);
    const float n = on_x ? nx : (on_y ? ny : nz);
    const float au = fabsf(u);
    float r = rcp_approx(u);
    r = __fmaf_rn(r, __fmaf_rn(-u, r, 1.0f), r);
    const float q = n * r;
    d = __fmaf_rn(r, __fmaf_rn(-q, u, n), q);
    face = (on_x ? 2 : (on_y ? 4 : 6)) - (u > 0.0f ? 1 : 0);
    cosw = au;
    return second > m * 1.000002f && m > 0x1p-30f && au > 0x1p-40f &&
           (__float_as_uint(u) & 0x7fffffu) != 0x7fffffu;
}

// Direction about the inward normal of a face from cos(theta) = ct and the
// other two components (a, b): the tail of lambertian_dir, src/optics.jl:119-137.
__device__ __forceinline__ void lambertian_from(int32_t face, float ct, float a, float b,
                                                float& ux, float& uy, float& uz)
{
    // the inward normal component on the face's axis, (a, b) on the other two
    // in axis order (XP: (-ct, a, b), YM: (a, ct, b), BACK: (a, b, -ct), ...),
    // by selects
    const float n = (face & 1) ? -ct : ct;
    ux = face <= 2 ? n : a;
    uy = face <= 2 ? a : (face <= 4 ? n : b);
    uz = face > 4 ? n : b;
}

// The tail of rayleigh_dir, src/optics.jl:93-111: rotate u by the polar
// cosine mu about itself; (cb, sb) = sin(theta) (cos, sin) of the azimuth.
__device__ __forceinline__ void rayleigh_rotate(float mu, float cb, float sb,
                                                float& ux, float& uy, float& uz)
{
    // t1 = (-uy, ux, 0)/|(ux, uy)| if |uz| < 0.9, else (0, -uz, uy)/|(uy, uz)|:
    // the same operations on selected operands (one square root and division
    // for a warp whose lanes take both cases)
    const bool zlow = fabsf(uz) < 0.9f;
    const float pa = zlow ? ux : uy, pb = zlow ? uy : uz;
    // both sums of squares are those of a unit vector's components, >= 0.19
    float inv = rcp_mid(sqrt_mid(pa * pa + pb * pb));
    const float t1x = zlow ? -pb * inv : 0.0f;
    const float t1y = zlow ? pa * inv : -pb * inv;
    const float t1z = zlow ? 0.0f : pa * inv;
    const float t2x = uy * t1z - uz * t1y;
    const float t2y = uz * t1x - ux * t1z;
    const float t2z = ux * t1y - uy * t1x;
    const float vx = mu * ux + cb * t1x + sb * t2x;
    const float vy = mu * uy + cb * t1y + sb * t2y;
    const float vz = mu * uz + cb * t1z + sb * t2z;
    inv = rcp_mid(sqrt_mid(vx * vx + vy * vy + vz * vz));
    ux = vx * inv; uy = vy * inv; uz = vz * inv;
}

// Order-preserving map of a float onto uint32 (for atomicMin on times).
__device__ __forceinline__ uint32_t float_key(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
constexpr uint32_t INF_KEY = 0xFF800000u;   // float_key(+Inf)

}  // namespace cl
