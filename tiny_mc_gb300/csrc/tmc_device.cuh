// tmc_device.cuh — device building blocks of the photon walk (sm_103a).
//
// Reference: computacionparalela/tiny_mc photon.c:6-51 (one photon per call,
// global libc rand()).  Here one thread carries one photon at a time; the
// random numbers come from a Philox-4x32-10 stream keyed by the photon id, so
// the walk of photon p is the same whichever thread, warp or launch runs it.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "tmc.h"

namespace tmc {

constexpr unsigned FULL_MASK = 0xffffffffu;

// ----------------------------------------------------------------- Philox
// Philox-4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11).  The ten round keys
// depend only on the seed, so they are precomputed on the host and passed in
// the kernel parameter block: every XOR with a key then reads the constant
// bank instead of spending an add per round.
constexpr uint32_t PHILOX_M0 = 0xD2511F53u;
constexpr uint32_t PHILOX_M1 = 0xCD9E8D57u;
constexpr uint32_t PHILOX_W0 = 0x9E3779B9u;
constexpr uint32_t PHILOX_W1 = 0xBB67AE85u;

struct PhiloxKeys {
    uint32_t k0[10];
    uint32_t k1[10];
};

inline PhiloxKeys make_philox_keys(uint64_t seed)
{
    PhiloxKeys k;
    uint32_t a = (uint32_t)seed, b = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; ++r) {
        k.k0[r] = a;
        k.k1[r] = b;
        a += PHILOX_W0;
        b += PHILOX_W1;
    }
    return k;
}

// Counter {c0, c1, c2, c3} -> four 32-bit words.
__device__ __forceinline__ uint4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                               const PhiloxKeys &K)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned long long p0 = (unsigned long long)PHILOX_M0 * c0;
        const unsigned long long p1 = (unsigned long long)PHILOX_M1 * c2;
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ K.k0[r];
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ K.k1[r];
        c1 = (uint32_t)p1;
        c3 = (uint32_t)p0;
        c0 = n0;
        c2 = n2;
    }
    return make_uint4(c0, c1, c2, c3);
}

// The parts of a photon's Philox blocks that do not depend on the block
// number: the counter is {block, 0, id low, id high}, so half of the first
// round and half of the second are the same for every block of a photon.
struct PhotonKey {
    uint32_t a, b, c, d;
};

__device__ __forceinline__ PhotonKey photon_key(unsigned long long pid, const PhiloxKeys &K)
{
    const unsigned long long p1 = (unsigned long long)PHILOX_M1 * (uint32_t)pid;
    const unsigned long long q0 = (unsigned long long)PHILOX_M0 * ((uint32_t)(p1 >> 32) ^ K.k0[0]);
    PhotonKey k;
    k.a = (uint32_t)p1 ^ K.k0[1];
    k.b = (uint32_t)(pid >> 32) ^ K.k1[0];
    k.c = (uint32_t)(q0 >> 32) ^ K.k1[1];
    k.d = (uint32_t)q0;
    return k;
}

// philox4x32_10(blk, 0, id low, id high) with the photon's key parts.
__device__ __forceinline__ uint4 philox_block(uint32_t blk, const PhotonKey &k, const PhiloxKeys &K)
{
    const unsigned long long p0 = (unsigned long long)PHILOX_M0 * blk;
    const unsigned long long p1 = (unsigned long long)PHILOX_M1 * ((uint32_t)(p0 >> 32) ^ k.b);
    uint32_t c0 = (uint32_t)(p1 >> 32) ^ k.a, c1 = (uint32_t)p1, c2 = (uint32_t)p0 ^ k.c, c3 = k.d;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        const unsigned long long q0 = (unsigned long long)PHILOX_M0 * c0;
        const unsigned long long q1 = (unsigned long long)PHILOX_M1 * c2;
        const uint32_t n0 = (uint32_t)(q1 >> 32) ^ c1 ^ K.k0[r];
        const uint32_t n2 = (uint32_t)(q0 >> 32) ^ c3 ^ K.k1[r];
        c1 = (uint32_t)q1;
        c3 = (uint32_t)q0;
        c0 = n0;
        c2 = n2;
    }
    return make_uint4(c0, c1, c2, c3);
}

// rand() of photon.c: 31 bits of a Philox word; 0 becomes 1 so that
// -log(rand()/RAND_MAX) is always finite (the reference's logf(0) case).
__device__ __forceinline__ uint32_t rand31(uint32_t word)
{
    return max(word >> 1, 1u);
}

// The 31 bits as a float, rounded once; 0 stays 0.
__device__ __forceinline__ float rand_float(uint32_t word)
{
    return __uint2float_rn(word >> 1);
}

// rand()/(float)RAND_MAX: (float)RAND_MAX is exactly 2^31, so the quotient is
// the correctly rounded int->float conversion scaled by 2^-31 (exact).  The
// 0 -> 1 mapping commutes with the conversion.
__device__ __forceinline__ float uniform01(float r)
{
    return fmaxf(r, 1.0f) * 0x1p-31f;
}

// 2.0f*rand()/(float)RAND_MAX - 1.0f: 2*fl(r)/2^31 is exact, so one fused
// multiply-add rounds exactly once where photon.c rounds once (the "- 1").
// rand31's 0 -> 1 mapping is left out here because it cannot change the
// result: -1 + 2^-30 rounds to -1.0f (the float spacing next to -1 is 2^-24),
// the same value r = 0 gives.
__device__ __forceinline__ float uniform_pm1(float r)
{
    return fmaf(r, 0x1p-30f, -1.0f);
}

// ------------------------------------------------------------ arithmetic
// The library's logarithm for TMC_MATH_EXACT, division-free: x = 2^k m with
// m in [sqrt(1/2), sqrt(2)), f = m - 1 (exact), log(m) = f + f^2 R(f) with R
// a degree-8 polynomial (the Chebyshev interpolant of log1p(f)/f at 10 nodes
// on [sqrt(1/2)-1, sqrt(2)-1], coefficients rounded to float; oracle/logfit.py
// derives them), evaluated by Horner with fused multiply-adds, and log x =
// k ln2_hi + (k ln2_lo + log m) with ln2 split so k ln2_hi is exact.  Every
// step is one IEEE-rounded operation (fma rounds once), so the CPU
// restatement reproduces it bit for bit.  Max error 0.86 ulp over every float
// in [2^-31, 1] (98.3% correctly rounded).
__device__ __forceinline__ float log_exact(float x)
{
    const uint32_t ix = __float_as_uint(x);
    const int k = (int)((ix + 0x004afb0du) >> 23) - 127;
    const float m = __uint_as_float(ix - ((uint32_t)k << 23));
    const float f = __fsub_rn(m, 1.0f);
    const float f2 = __fmul_rn(f, f);
    float r = -0x1.31335ap-4f;
    r = __fmaf_rn(r, f, 0x1.064786p-3f);
    r = __fmaf_rn(r, f, -0x1.0fb036p-3f);
    r = __fmaf_rn(r, f, 0x1.22cf10p-3f);
    r = __fmaf_rn(r, f, -0x1.5423b0p-3f);
    r = __fmaf_rn(r, f, 0x1.999e86p-3f);
    r = __fmaf_rn(r, f, -0x1.000424p-2f);
    r = __fmaf_rn(r, f, 0x1.55555ep-2f);
    r = __fmaf_rn(r, f, -0x1.fffff8p-2f);
    const float lm = __fmaf_rn(f2, r, f);
    const float kf = __int2float_rn(k);
    return __fmaf_rn(kf, 0.693145751953125f, __fmaf_rn(kf, 1.42860682e-6f, lm));
}

// The forms that flush denormals: the same values as the plain ones without
// their range checks (eight instructions less per photon step over the
// logarithm and the two square roots).  U >= 2^-31 and 1 - t >= 2^-24 or 0; a
// radius below 2^-63 mean free paths is taken as 0.
__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// photon.c's float expressions, IEEE-rounded one operation at a time.
struct ExactMath {
    static constexpr uint32_t id = TMC_MATH_EXACT;
    // -logf(U), photon.c:21
    __device__ static __forceinline__ float step_length(float U) { return -log_exact(U); }
    // x += t * u, photon.c:22-24
    __device__ static __forceinline__ float move(float x, float t, float u)
    {
        return __fadd_rn(x, __fmul_rn(t, u));
    }
    // sqrtf(x*x + y*y + z*z) * shells_per_mfp, photon.c:26
    __device__ static __forceinline__ float radius_shells(float x, float y, float z, float spm)
    {
        const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
        return __fmul_rn(__fsqrt_rn(r2), spm);
    }
    // xi1*xi1 + xi2*xi2, photon.c:39
    __device__ static __forceinline__ float norm2(float a, float b)
    {
        return __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
    }
    static constexpr float ONE = 1.0f;   // the launch direction's w
    static constexpr bool CHEAP_DIRECTION = false;
    // photon.c:41-43 from an accepted try
    __device__ static __forceinline__ void direction(float t, float xi1, float xi2, float &u, float &v, float &w)
    {
        u = fmaf(2.0f, t, -1.0f);
        const float sc = __fsqrt_rn(__fdiv_rn(__fsub_rn(1.0f, __fmul_rn(u, u)), t));
        v = __fmul_rn(xi1, sc);
        w = __fmul_rn(xi2, sc);
    }
    __device__ static __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
};

// Hardware approximations (MUFU lg2 / sqrt), contraction allowed.
struct FastMath {
    static constexpr uint32_t id = TMC_MATH_FAST;
    // twice the step; directions are kept halved (both scalings are exact)
    __device__ static __forceinline__ float step_length(float U)
    {
        float l;
        asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(U));
        return l * (-2.0f * 0.693147182464599609375f);
    }
    __device__ static __forceinline__ float move(float x, float t, float u) { return fmaf(t, u, x); }
    __device__ static __forceinline__ float radius_shells(float x, float y, float z, float spm)
    {
        return sqrt_approx(fmaf(x, x, fmaf(y, y, z * z))) * spm;
    }
    __device__ static __forceinline__ float norm2(float a, float b) { return fmaf(a, a, b * b); }
    static constexpr float ONE = 0.5f;   // the launch direction's w, halved
    static constexpr bool CHEAP_DIRECTION = true;
    // (1-u^2)/t with u = 2t-1 is 4(1-t): sqrt of it is 2 sqrt(1-t)
    __device__ static __forceinline__ void direction(float t, float xi1, float xi2, float &u, float &v, float &w)
    {
        u = t - 0.5f;
        const float sc = sqrt_approx(1.0f - t);
        v = xi1 * sc;
        w = xi2 * sc;
    }
    __device__ static __forceinline__ float mul(float a, float b) { return a * b; }
};

// ---------------------------------------------------------------- tallies
// A photon's weight is kept times 2^20, so that w and w^2 in tally units of
// 2^-40 are one multiplication away: w 2^40 = W 2^20 and fl(w w) 2^40 =
// fl(W W) with W = w 2^20 (both scalings are exact; weights whose unscaled
// product would be denormal deposit zero units either way).
constexpr float WEIGHT_ONE = 0x1p20f;
__device__ __forceinline__ float weight_units(float W) { return W * 0x1p20f; }
__device__ __forceinline__ float weight2_units(float W) { return __fmul_rn(W, W); }

// A deposit of q units (0 <= q <= 2^40, not necessarily whole) as 32-bit
// halves of rint(q), round to nearest even.  Adding 2^55, whose float spacing
// is 2^32, with rounding towards zero leaves floor(q / 2^32) in the low
// mantissa bits: hi_bits = UNITS_HI_BIAS + that.  The rest is exact in float
// (it is the low part of q's own significand) and below 2^32; its correctly
// rounded conversion is the low word.  Five instructions, against six for a
// truncating conversion and back.
constexpr uint32_t UNITS_HI_BIAS = 0x5B000000u;   // the bits of 2^55f
__device__ __forceinline__ void units_split(float q, uint32_t &lo, uint32_t &hi_bits)
{
    const float a = __fadd_rz(q, 0x1p55f);
    hi_bits = __float_as_uint(a);
    lo = __float2uint_rn(__fsub_rn(q, __fsub_rn(a, 0x1p55f)));
}

// Shared-memory atomics by 32-bit shared address.
__device__ __forceinline__ uint32_t atom_shared_add(uint32_t addr, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v));
    return old;
}
__device__ __forceinline__ void red_shared_add(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v));
}

// Add a deposit (units_split's halves) to a 64-bit shared-memory tally kept as
// two 32-bit words, with native 32-bit shared atomics: the carry out of the
// low word goes into the high word.  The caller bounds the sum below 2^64.
__device__ __forceinline__ void tally_add_nowrap(uint32_t lo_addr, uint32_t hi_addr, uint32_t lo, uint32_t hi_bits)
{
    const uint32_t old = atom_shared_add(lo_addr, lo);
    uint32_t hi;   // hi_bits - UNITS_HI_BIAS + (old + lo carries)
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %2;\n\taddc.u32 %0, %3, %4;\n\t}"
        : "=r"(hi)
        : "r"(old), "r"(lo), "r"(hi_bits), "n"(0u - UNITS_HI_BIAS));
    red_shared_add(hi_addr, hi);
}

// The same where the sum may wrap: a wrap of the high word carries 2^64 units
// into the 128-bit global tally, which receives only such carries until the
// final flush.  wraps (may be null) additionally counts this tally's wraps.
__device__ __forceinline__ void tally_add(uint32_t *sh_lo, uint32_t *sh_hi, unsigned long long *g_hi,
                                          uint32_t lo, uint32_t hi_bits, uint32_t *wraps = nullptr)
{
    uint32_t hi = hi_bits - UNITS_HI_BIAS;
    const uint32_t old = atomicAdd(sh_lo, lo);
    hi += (old + lo < old) ? 1u : 0u;
    const uint32_t oh = atomicAdd(sh_hi, hi);
    if (oh + hi < oh) {
        atomicAdd(g_hi, 1ull);
        if (wraps)
            atomicAdd(wraps, 1u);
    }
}

// Flush a 64-bit partial sum into a 128-bit global tally.
__device__ __forceinline__ void flush128(unsigned long long *g_lo, unsigned long long *g_hi,
                                         unsigned long long v)
{
    if (v) {
        const unsigned long long old = atomicAdd(g_lo, v);
        if (old + v < old)
            atomicAdd(g_hi, 1ull);
    }
}

// A deposit straight into a shell's 128-bit global tally (four words).  Both
// sums' low words are added before either carry is looked at, so that one
// atomic's way to the L2 and back hides the other's.
__device__ __forceinline__ void deposit_global(unsigned long long *gs, float weight)
{
    uint32_t l, h;
    units_split(weight_units(weight), l, h);
    const unsigned long long v = ((unsigned long long)(h - UNITS_HI_BIAS) << 32) | l;
    units_split(weight2_units(weight), l, h);
    const unsigned long long v2 = ((unsigned long long)(h - UNITS_HI_BIAS) << 32) | l;
    const unsigned long long old = atomicAdd(&gs[0], v), old2 = atomicAdd(&gs[2], v2);
    if (old + v < old)
        atomicAdd(&gs[1], 1ull);
    if (old2 + v2 < old2)
        atomicAdd(&gs[3], 1ull);
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

}  // namespace tmc
