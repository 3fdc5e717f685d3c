// cbl_arith.cuh - integer arithmetic of one Bellard term on sm_103a.
//
// A term of series f at index k < d is x = frac(2^(10(d-k)) / m), m = den0*k + den1
// (Bellard.cl:739-749, Bellard_div2by1.cl:327-350). The reference computes
// r = 2^(10e) mod m by Montgomery exponentiation (Bellard.cl:380-461) and then
// forms the fraction r/m in double-double or by an exact 4-limb division
// (Bellard_div2by1.cl:339-341).
//
// Here one Montgomery ladder produces r6 = 2^(10e + 192) mod m, and the six
// 32-bit quotient digits of r/m fall out of six Montgomery reduction steps run
// downwards: with r_j = 2^(10e + 32j) mod m,
//     q_j = floor(r_{j-1} * 2^32 / m) = -r_j * m^-1 mod 2^32 = r_j * mp mod 2^32
//     r_{j-1} = (r_j + q_j * m) / 2^32
// (exact division by the odd m), so q_j is the Montgomery multiplier of the
// step and no division is ever executed. The chain ends at r_0 = 2^(10e) mod m.
//
// Eight residue kinds:
//   width 1 (m < 2^17; the formulas hold below 2^28): R = 2^32, residues kept lazily in [0, 4m).
//   lazy width 1 (2^17 <= m < 2^29): R = 2^32, residues in [0, 2m).
//   middle width 1 (2^29 <= m < 2^31; holds from 2^25): R = 2^32, residues in [0, m).
//   strict width 1 (2^31 <= m < 2^32): R = 2^32, residues in [0, m) up to sign.
//   float-quotient width 2 (2^32 <= m < 94 * 2^32): R = 2^24, residues below 8m,
//     the top of each square taken off by a float quotient.
//   short width 2 (94 * 2^32 <= m < 39 * 2^40): R = 2^50, residues in [0, 4m).
//   width 2 (39 * 2^40 <= m < 2^60): R = 2^64 by two word steps, residues in [0, 4m).
//   wide width 2 (2^60 <= m < 2^62): the same steps with residues in [0, 2m).
// The ladder step is y <- REDC(y^2) << b with b the next exponent bit; in the
// lazy kinds 16m < R keeps the result below 4m with no conditional subtraction.
#pragma once
#include <stdint.h>
#include <type_traits>
#include "cbl_internal.h"

namespace cbl {

// -m^-1 mod 2^32 for odd m: (3m) xor 2 is an inverse to 5 bits; three Newton
// steps x <- x(2 - mx) take it to 40 bits.
__device__ __forceinline__ uint32_t neg_inv32(uint32_t m)
{
    uint32_t x = (m * 3u) ^ 2u;
    x *= 2u - m * x;
    x *= 2u - m * x;
    x *= 2u - m * x;
    return 0u - x;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ------------------------------------------------------------ start values --
// The ladder starts from a value congruent to 2^(Rb+1) (the exponent's leading
// one already consumed). Two float-reciprocal quotient estimates with 32-bit
// conversions only: q1 = trunc(2^E0 / m) is off by at most 2^(E0-21)/m + 1, so
// r1 = 2^E0 - q1 m is small; q2 = rint(r1 / m) is then off by less than 1 and
// r1 - q2 m lies in (-m, m).

// trunc(x) for a positive float x < 2^63, as a 64-bit integer, from its bits.
__device__ __forceinline__ uint64_t float_to_u64_trunc(float x)
{
    const uint32_t bits = __float_as_uint(x);
    const int e = (int)((bits >> 23) & 0xffu) - 127;
    const uint64_t mant = (uint64_t)((bits & 0x7fffffu) | 0x800000u);
    return e >= 23 ? (mant << (e - 23)) : (mant >> (23 - e));
}

// Width 1 (3 <= m < 2^28): a value in (0, 2m) congruent to 2^33.
__device__ __forceinline__ uint32_t w1_start(uint32_t m)
{
    const float inv = rcp_approx(__uint2float_rn(m));
    const uint32_t q1 = __float2uint_rz(8589934592.0f * inv);          // < 2^32 for m >= 3
    const int32_t r1 = (int32_t)(0u - q1 * m);                          // 2^33 - q1 m, |r1| < 2^29
    const int32_t q2 = __float2int_rn(__int2float_rn(r1) * inv);
    return (uint32_t)(r1 + (1 - q2) * (int32_t)m);
}

// Width 2: a value in (0, 2m) congruent to 2^(R + p), 1 <= p <= 15, for R = 50 (2^32 <= m
// < 2^46) or R = 64 (2^44 <= m < 2^62). The first quotient leaves |r1| <= 2^(R+p-22) + m,
// so r1 / m is below 2^13 and its rounded estimate off by a few thousandths.
// (R = 50 checked in float32 emulation over 4e5 moduli, every p, with reciprocals off by up
// to 2 ulps.)
template <int R>
__device__ __forceinline__ uint64_t w2_start(uint64_t m, uint32_t p)
{
    const uint32_t m0 = (uint32_t)m, m1 = (uint32_t)(m >> 32);
    const float fm = __fmaf_rn(__uint2float_rn(m1), 4294967296.0f, __uint2float_rn(m0));
    const float inv = rcp_approx(fm);
    const float scale = __int_as_float((int)((127u + R + p) << 23));            // 2^(R+p)
    const uint64_t q1 = float_to_u64_trunc(scale * inv);
    const uint64_t top = R + p < 64 ? 1ull << ((R + p) & 63) : 0ull;           // mod 2^64
    const int64_t r1 = (int64_t)(top - q1 * m);
    const float fr1 = __fmaf_rn(__int2float_rn((int32_t)(r1 >> 32)), 4294967296.0f,
                                __uint2float_rn((uint32_t)r1));
    const int32_t q2 = __float2int_rn(fr1 * inv);
    return (uint64_t)(r1 + (int64_t)(1 - q2) * (int64_t)m);
}

// ------------------------------------------------------------ exponent walk --
// The step of a ladder's last exponent bit: a plain step, but for the strict kind.
struct W1SState;
template <typename State>
__device__ __forceinline__ void last_step(State &st, uint32_t b)
{
    if constexpr (std::is_same<State, W1SState>::value) st.last_step(b);
    else st.step(b);
}

// Calls st.step(b) for every bit of Ep after its leading one, most significant
// first. When Ep >= 2^32 the 32 bits of the low word run fully unrolled.
template <typename State>
__device__ __forceinline__ void walk_bits(uint64_t Ep, State &st)
{
    const uint32_t hi = (uint32_t)(Ep >> 32), lo = (uint32_t)Ep;
    if (hi != 0) {
        const int nb = 32 - __clz(hi);
        uint32_t h = (hi << (32 - nb)) << 1;
        for (int i = 1; i < nb; ++i) {
            st.step(h >> 31);
            h <<= 1;
        }
#pragma unroll
        for (int i = 31; i >= 0; --i) st.step((lo >> i) & 1u);
    } else {
        const int nb = 32 - __clz(lo);
        uint32_t l = (lo << (32 - nb)) << 1;
        for (int i = 1; i < nb; ++i) {
            st.step(l >> 31);
            l <<= 1;
        }
    }
}

// Start from the leading up-to-NB bits of Ep at once (value p), then walk the
// rest, the last bit by last_step (a kind may finish its residue there); st.y is
// set by start(p). Ep has more than NB bits.
template <int NB, typename State, typename Start>
__device__ __forceinline__ void walk_bits_start(uint64_t Ep, State &st, Start start)
{
    const uint32_t hi = (uint32_t)(Ep >> 32), lo = (uint32_t)Ep;
    if (hi != 0) {
        const int nb = 32 - __clz(hi);
        const int t = nb < NB ? nb : NB;
        start(st, hi >> (nb - t));
        uint32_t h = (nb - t) > 0 ? hi << (32 - (nb - t)) : 0u;
        for (int i = t; i < nb; ++i) {
            st.step(h >> 31);
            h <<= 1;
        }
#pragma unroll
        for (int i = 31; i >= 1; --i) st.step((lo >> i) & 1u);
    } else {
        const int nb = 32 - __clz(lo);
        start(st, lo >> (nb - NB));
        uint32_t l = lo << (32 - (nb - NB));
        for (int i = NB + 1; i < nb; ++i) {
            st.step(l >> 31);
            l <<= 1;
        }
    }
    last_step(st, lo & 1u);
}

// ------------------------------------------------- multiply-add chains --
// Every REDC word step below is written as a PTX carry chain of mad.lo.cc /
// madc.hi over 32-bit words. A 64-bit multiply-add (mad.wide with a 64-bit
// addend) issues more slowly on sm_103a than the two chained halves, and the
// carry out of the chain comes for free.

// hi(u m + (t0, t1)) mod 2^32, where u m + t0 = 0 mod 2^32 (a REDC word step).
__device__ __forceinline__ uint32_t redc_word(uint32_t u, uint32_t m, uint32_t t0, uint32_t t1)
{
    uint32_t r;
    asm("{\n\t.reg .u32 x;\n\t"
        "mad.lo.cc.u32 x, %1, %2, %3;\n\t"
        "madc.hi.u32 %0, %1, %2, %4;\n\t}"
        : "=r"(r)
        : "r"(u), "r"(m), "r"(t0), "r"(t1));
    return r;
}

// As redc_word, also returning the carry out of the high word in c (0 or 1).
__device__ __forceinline__ uint32_t redc_word_c(uint32_t u, uint32_t m, uint32_t t0, uint32_t t1, uint32_t &c)
{
    uint32_t r;
    asm("{\n\t.reg .u32 x;\n\t"
        "mad.lo.cc.u32 x, %2, %3, %4;\n\t"
        "madc.hi.cc.u32 %0, %2, %3, %5;\n\t"
        "addc.u32 %1, 0, 0;\n\t}"
        : "=r"(r), "=r"(c)
        : "r"(u), "r"(m), "r"(t0), "r"(t1));
    return r;
}

// ---------------------------------------------------------------- width 1 --
// y in [0,4m), m < 2^28: REDC_2^32(y^2) << b, again in [0,4m).
__device__ __forceinline__ uint32_t w1_sqr(uint32_t y, uint32_t m, uint32_t mp, uint32_t b)
{
    const uint64_t t = (uint64_t)y * y;                 // < 16 m^2 < 2^60
    const uint32_t u = (uint32_t)t * mp;
    return redc_word(u, m, (uint32_t)t, (uint32_t)(t >> 32)) << b;   // (t + u m) / 2^32 < 2m
}

struct W1State {
    uint32_t y, m, mp;
    __device__ __forceinline__ void step(uint32_t b) { y = w1_sqr(y, m, mp, b); }
};

// r6 = 2^E mod m in [0, m) for E >= 33 (m < 2^28, odd, >= 3).
__device__ __forceinline__ uint32_t w1_pow2(uint64_t E, uint32_t m, uint32_t mp)
{
    W1State st{w1_start(m), m, mp};                     // invariant y = 2^(32 + prefix of E - 32)
    walk_bits(E - 32, st);
    uint32_t y = st.y;
    y = min(y, y - 2u * m);                            // [0,4m) -> [0,2m)
    y = min(y, y - m);                                 //        -> [0,m)
    return y;
}

// N quotient digits of r_0 / m from r_N (digit 0 least significant), and r_0.
// Valid for any odd m < 2^32, m > 1.
template <int N>
__device__ __forceinline__ uint32_t w1_digits(uint32_t r, uint32_t m, uint32_t mp, uint32_t q[N])
{
#pragma unroll
    for (int j = 0; j < N; ++j) {
        q[j] = r * mp;
        r = __umulhi(q[j], m) + 1u;                     // (r + q m) / 2^32 < m: r > 0, so its low word carries
    }
    return r;
}

// --------------------------------------------------------- strict width 1 --
// 2^31 <= m < 2^32: R = 2^32, residues up to sign, y in [0, m) standing for y or -y:
// squaring forgets the sign, so REDC by subtraction needs no correction at all. With
// u = t0 m^-1 the low words of t = y^2 and u m are equal; t1 = hi(t) and h = hi(u m) are
// below m, so y = |t1 - h| = max - min is too, and the doubling takes the smaller of y
// and m - y first. Minimum, maximum and addition issue at twice the rate of compare,
// select and shift. The ladder's last step tells y from -y again.
// (Signed residues with one compare and select a step: 58.6e9 terms/s, 66.5e9 so; position
// 1e9 31.9 -> 30.4 ms.)
struct W1SState {
    uint32_t y, m, ip;                                  // ip = m^-1 mod 2^32
    __device__ __forceinline__ void square(uint32_t &t1, uint32_t &h) const
    {
        const uint64_t t = (uint64_t)y * y;
        t1 = (uint32_t)(t >> 32);
        h = __umulhi((uint32_t)t * ip, m);
    }
    __device__ __forceinline__ void step(uint32_t b)
    {
        uint32_t t1, h;
        square(t1, h);
        const uint32_t d = max(t1, h) - min(t1, h);
        y = min(d, m - d) << b;
    }
    // the step that leaves the residue itself
    __device__ __forceinline__ void last_step(uint32_t b)
    {
        uint32_t t1, h;
        square(t1, h);
        const uint32_t z = t1 < h ? t1 - h + m : t1 - h, w = m - z;
        y = b == 0 ? z : z >= w ? z - w : z + z;
    }
};

// ------------------------------------------------------ middle width 1 --
// 2^25 <= m < 2^31: R = 2^32, residues in [0, m). The doubling comes first:
// t = y (2^b y) < 2m^2 < 2^63 and u m < 2^63, so the word step has no carry
// out and REDC(t) = REDC(y^2) 2^b mod m is below 2m; one min(z, z - m)
// brings it below m. (Two ALU operations fewer than reducing, then doubling
// and reducing again.)
__device__ __forceinline__ uint32_t w1m_sqr(uint32_t y, uint32_t m, uint32_t mp, uint32_t b)
{
    const uint64_t t = (uint64_t)y * (y << b);
    const uint32_t u = (uint32_t)t * mp;
    const uint32_t z = redc_word(u, m, (uint32_t)t, (uint32_t)(t >> 32));   // < 2m
    return min(z, z - m);
}

struct W1MState {
    uint32_t y, m, mp;
    __device__ __forceinline__ void step(uint32_t b) { y = w1m_sqr(y, m, mp, b); }
};

// 2^(32 + p) mod m in [0, m), 1 <= p <= 15, 2^28 <= m < 2^32: q1 <= 2^19 is
// off by at most one, so one correction either way suffices.
__device__ __forceinline__ uint32_t w1s_start(uint32_t m, uint32_t p)
{
    const float inv = rcp_approx(__uint2float_rn(m));
    const float scale = __int_as_float((int)((127u + 32u + p) << 23));
    const uint32_t q1 = __float2uint_rz(scale * inv);
    int64_t r = (int64_t)(1ull << (32 + p)) - (int64_t)q1 * (int64_t)m;   // in [-m, 2m)
    r += (r < 0) ? (int64_t)m : 0;
    r -= (r >= (int64_t)m) ? (int64_t)m : 0;
    return (uint32_t)r;
}

// A value congruent to 2^(32 + p) for m < 2^31 with 2^(32 + p) / m < 2^22: below m from
// m = 2^28 on (p <= 15), below 1.8m otherwise. The float quotient (three roundings of
// 2^-24: within 0.75, and 0.1 from 2^28 on) less 0.8 is rounded down, so -q m mod 2^32
// is the positive rest, below 2m from 2^28 on and below 2.8m otherwise.
__device__ __forceinline__ uint32_t w1m_start(uint32_t m, uint32_t p)
{
    const float inv = rcp_approx(__uint2float_rn(m));
    const float scale = __int_as_float((int)((127u + 32u + p) << 23));
    const uint32_t r = 0u - __float2uint_rz(__fmaf_rn(scale, inv, -0.8f)) * m;
    return min(r, r - m);
}

struct W1MStart {
    __device__ __forceinline__ void operator()(W1MState &st, uint32_t p) const { st.y = w1m_start(st.m, p); }
};

// ------------------------------------------------------- lazy width 1 --
// 2^17 <= m < 2^29: the middle kind's step without its correction. With y < 2m,
// y (2^b y) < 8m^2 and REDC gives less than 8m^2 / 2^32 + m < 2m again. (Shifting
// one multiplicand, not the result, keeps the bound to 2^29.)
struct W1LState {
    uint32_t y, m, mp;
    __device__ __forceinline__ void step(uint32_t b)
    {
        const uint64_t t = (uint64_t)y * (y << b);
        const uint32_t u = (uint32_t)t * mp;
        y = redc_word(u, m, (uint32_t)t, (uint32_t)(t >> 32));
    }
    __device__ __forceinline__ uint32_t residue() const { return min(y, y - m); }
};

struct W1LStart {
    __device__ __forceinline__ void operator()(W1LState &st, uint32_t p) const { st.y = w1m_start(st.m, p); }
};

// r6 = 2^E mod m in [0, m) from the leading NB bits of E - 32 at once: NB = 3 for
// 2^17 <= m, 4 for 2^25 <= m (the start's bound on 2^(32 + p) / m).
template <int NB>
__device__ __forceinline__ uint32_t w1l_pow2(uint64_t E, uint32_t m, uint32_t mp)
{
    W1LState st{0, m, mp};
    walk_bits_start<NB>(E - 32, st, W1LStart{});
    return st.residue();
}

// r6 = 2^E mod m in [0, m) for E >= 42, 2^25 <= m < 2^31. The start value
// takes the leading up-to-four bits of E - 32 at once.
__device__ __forceinline__ uint32_t w1m_pow2(uint64_t E, uint32_t m, uint32_t mp)
{
    W1MState st{0, m, mp};
    walk_bits_start<4>(E - 32, st, W1MStart{});
    return st.y;
}

struct W1SStart {
    __device__ __forceinline__ void operator()(W1SState &st, uint32_t p) const
    {
        st.y = w1s_start(st.m, p);
    }
};

// r6 = 2^E mod m in [0, m) for E >= 33 (2^31 <= m < 2^32), from the same
// 4-bit start value.
__device__ __forceinline__ uint32_t w1s_pow2(uint64_t E, uint32_t m, uint32_t mp)
{
    W1SState st{0, m, 0u - mp};
    walk_bits_start<4>(E - 32, st, W1SStart{});
    return st.y;
}

// ---------------------------------------------------------------- width 2 --
// y = (y0,y1) in [0,4m), m = (m0,m1) with 2^28 <= m < 2^60 (so y1 < 2^30,
// m1 < 2^28, T + U m < 2^125): REDC_2^64(y^2) << b by two 32-bit word steps,
// again in [0,4m) because 16m < 2^64.
__device__ __forceinline__ void w2_sqr(uint32_t &y0, uint32_t &y1, uint32_t m0, uint32_t m1,
                                       uint32_t mp, uint32_t b)
{
    // T = y^2 = t0 + t1 2^32 + t2 2^64 + t3 2^96  (< 16 m^2 < 2^124)
    const uint64_t a = (uint64_t)y0 * y0;
    const uint64_t p = (uint64_t)y0 * (y1 << 1);        // y1 < 2^30
    const uint64_t s = (uint64_t)y1 * y1;
    const uint32_t t0 = (uint32_t)a;
    uint32_t t1, t2, t3;
    asm("add.cc.u32 %0, %3, %4;\n\t"
        "addc.cc.u32 %1, %5, %6;\n\t"
        "addc.u32 %2, %7, 0;"
        : "=r"(t1), "=r"(t2), "=r"(t3)
        : "r"((uint32_t)(a >> 32)), "r"((uint32_t)p), "r"((uint32_t)(p >> 32)), "r"((uint32_t)s),
          "r"((uint32_t)(s >> 32)));
    // word step 1: s = (T + u0 m) / 2^32 = (t1, t2, t3) + hi(u0 m0) + c + u0 m1,
    // c the carry out of u0 m0 + t0 (whose low word is 0)
    const uint32_t u0 = t0 * mp;
    uint32_t s0, s1, s2;
    asm("{\n\t.reg .u32 x, h, e2, e3;\n\t"
        "mad.lo.cc.u32 x, %3, %4, %5;\n\t"
        "madc.hi.cc.u32 h, %3, %4, %6;\n\t"
        "addc.cc.u32 e2, %7, 0;\n\t"
        "addc.u32 e3, %8, 0;\n\t"
        "mad.lo.cc.u32 %0, %3, %9, h;\n\t"
        "madc.hi.cc.u32 %1, %3, %9, e2;\n\t"
        "addc.u32 %2, e3, 0;\n\t}"
        : "=r"(s0), "=r"(s1), "=r"(s2)
        : "r"(u0), "r"(m0), "r"(t0), "r"(t1), "r"(t2), "r"(t3), "r"(m1));
    // word step 2: z = (s + u1 m) / 2^32 < 2m
    const uint32_t u1 = s0 * mp;
    uint32_t z0, z1;
    asm("{\n\t.reg .u32 x, h, e2;\n\t"
        "mad.lo.cc.u32 x, %2, %3, %4;\n\t"
        "madc.hi.cc.u32 h, %2, %3, %5;\n\t"
        "addc.u32 e2, %6, 0;\n\t"
        "mad.lo.cc.u32 %0, %2, %7, h;\n\t"
        "madc.hi.u32 %1, %2, %7, e2;\n\t}"
        : "=r"(z0), "=r"(z1)
        : "r"(u1), "r"(m0), "r"(s0), "r"(s1), "r"(s2), "r"(m1));
    y1 = __funnelshift_l(z0, z1, b);
    y0 = z0 << b;
}

struct W2State {
    uint32_t y0, y1, m0, m1, mp;
    __device__ __forceinline__ void step(uint32_t b) { w2_sqr(y0, y1, m0, m1, mp, b); }
};

__device__ __forceinline__ uint64_t two_words(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

// Start of a two-word ladder from the leading bits of its exponent.
template <int R>
struct W2Start {
    template <typename State>
    __device__ __forceinline__ void operator()(State &st, uint32_t p) const
    {
        const uint64_t y = w2_start<R>(two_words(st.m0, st.m1), p);
        st.y0 = (uint32_t)y;
        st.y1 = (uint32_t)(y >> 32);
    }
};

// Residue in [0, m) of a lazy state in [0, 4m).
template <typename State>
__device__ __forceinline__ uint64_t lazy_residue(const State &st)
{
    const uint64_t m = two_words(st.m0, st.m1);
    uint64_t r = two_words(st.y0, st.y1);
    r = min(r, r - 2 * m);
    return min(r, r - m);
}

// r6 = 2^E mod m in [0, m) for E >= 65 (2^44 <= m < 2^60), the leading up-to-four
// bits of E - 64 at once.
__device__ __forceinline__ uint64_t w2_pow2(uint64_t E, uint64_t m, uint32_t mp)
{
    W2State st{0, 0, (uint32_t)m, (uint32_t)(m >> 32), mp};
    walk_bits_start<4>(E - 64, st, W2Start<64>{});
    return lazy_residue(st);
}

// -------------------------------------------- width 2, m < 39 * 2^40 --
// 2^32 <= m < 39 * 2^40 (m1 < 2^13.3), y in [0,4m) (y1 < 2^15.3), R = 2^50: one 32-bit
// REDC word step and one 18-bit step. y^2 = y0^2 + y0 (2 y1) 2^32 + y1^2 2^64 with
// y1^2 < 2^31, so word step 1 is
//   s = (y0^2 + u0 m0) / 2^32 + y1^2 2^32 + y0 (2 y1) + u0 m1 < 2^62.6,
// one carry chain whose carry out of the first multiply-add lands on y1^2
// (no carry leaves the chain). The 18-bit step takes u1 = s0 mp mod 2^18, so
// u1 m1 < 2^32 is a single low multiply (a 32-bit step needs two words there):
// X = s + u1 m0 + u1 m1 2^32 < 16 m^2 / 2^32 + 2^18 m < 2^64 for m < 39 * 2^40, its low 18
// bits zero, and X / 2^18 < 16 m^2 / 2^50 + m < 1.7m. The doubling joins that
// shift: y = X >> (18 - b). 14 multiply halves per step instead of 16. (With a 16-bit
// step the same code reached 2^44; moduli from there on took the general step.)
__device__ __forceinline__ void w2s_sqr(uint32_t &y0, uint32_t &y1, uint32_t m0, uint32_t m1, uint32_t mp,
                                        uint32_t b)
{
    const uint64_t A = (uint64_t)y0 * y0;
    const uint32_t a0 = (uint32_t)A, a1 = (uint32_t)(A >> 32);
    const uint32_t u0 = a0 * mp;
    const uint32_t ysq = y1 * y1;
    const uint32_t y2 = y1 << 1;
    uint32_t s0, s1;
    asm("{\n\t.reg .u32 x0, x1, w, t0, t1;\n\t"
        "mad.lo.cc.u32 x0, %2, %3, %4;\n\t"     // u0 m0 + y0^2: low word 0
        "madc.hi.cc.u32 x1, %2, %3, %5;\n\t"
        "addc.u32 w, %6, 0;\n\t"                // y1^2 + carry
        "mad.lo.cc.u32 t0, %7, %8, x1;\n\t"     // + y0 (2 y1)
        "madc.hi.u32 t1, %7, %8, w;\n\t"
        "mad.lo.cc.u32 %0, %2, %9, t0;\n\t"     // + u0 m1
        "madc.hi.u32 %1, %2, %9, t1;\n\t}"
        : "=r"(s0), "=r"(s1)
        : "r"(u0), "r"(m0), "r"(a0), "r"(a1), "r"(ysq), "r"(y0), "r"(y2), "r"(m1));
    const uint32_t u1 = (s0 * mp) & 0x3ffffu;
    uint32_t x0, x1;
    asm("mad.lo.cc.u32 %0, %2, %3, %4;\n\t"     // u1 m0 + s: low 18 bits 0
        "madc.hi.u32 %1, %2, %3, %5;\n\t"
        "mad.lo.u32 %1, %2, %6, %1;"              // + u1 m1 2^32
        : "=&r"(x0), "=&r"(x1)
        : "r"(u1), "r"(m0), "r"(s0), "r"(s1), "r"(m1));
    const uint32_t sh = 18u - b;
    y0 = __funnelshift_r(x0, x1, sh);
    y1 = x1 >> sh;
}

struct W2SState {
    uint32_t y0, y1, m0, m1, mp;
    __device__ __forceinline__ void step(uint32_t b) { w2s_sqr(y0, y1, m0, m1, mp, b); }
};

// r6 = 2^E mod m in [0, m) for E >= 65, 2^32 <= m < 39 * 2^40: the ladder runs in
// Montgomery form with R = 2^50 on the bits of E - 50, the leading up-to-four at once.
__device__ __forceinline__ uint64_t w2s_pow2(uint64_t E, uint64_t m, uint32_t mp)
{
    W2SState st{0, 0, (uint32_t)m, (uint32_t)(m >> 32), mp};
    walk_bits_start<4>(E - 50, st, W2Start<50>{});
    return lazy_residue(st);
}

// ------------------------------------------------ width 2, m < 94 * 2^32 --
// 2^32 <= m < 94 * 2^32 (positions up to 1e11): the square is reduced from both
// ends at once. Its top comes off by a float quotient, its bottom by a 24-bit
// Montgomery step, with one multiplier v = u + (q - o) 2^24 for both:
//   u = y^2 m^-1 mod 2^24          (exact, from the low word of y^2)
//   q ~ floor(y^2 / (2^24 m))      (float, from the top 23 bits of y)
//   X = y^2 - v m = 2^24 z, z = y^2 2^-24 mod m up to a multiple of m.
// The float work is done before the high words of y^2 would be needed, so y^2
// and v m are formed mod 2^64 only: 8 multiply halves a step (y0^2, u, y0 y1,
// v0 n0, v0 n1, v1 n0 with n = 2^64 - m) against 14 in w2s_sqr, which pays
// for the full square and two exact word steps.
// Floats: the 23 bits y >> 18 are used as they are, as a denormal (2^-149 each);
// s carries 2^119 of that, so t = s (y >> 18) is y / sqrt(2^24 m) times 2^-30,
// and t^2 + 2^-60 (2^23 - o) has q - o in its low mantissa bits.
// Bounds: s <= 2^125 / sqrt(m) and t are rounded down, so q never exceeds
// y^2 / (2^24 m). It falls short by the floor (1), the truncation of y (2^-5 y/m)
// and the roundings (12 2^-24 q), so with y < B m
//   X / (2^24 m) lies in (o - 1, o + 1 + B / 32 + 12 2^-48 B^2 m), B twice that.
// o = 2 (m < 15 * 2^34): z in (m, 3.95m), q >= 2 always. o = 1 (CK): z in (0, 2.65m),
// X < 2^64 up to m = 94 * 2^32; there q - 1 may be -1, so it is offset by 2^22 and
// ck takes the offset's 2^46 m out of X again (a register more). In both y < 2^41.
template <bool CK>
struct W2FState {
    uint32_t y0, y1, n0, n1, ip;                        // y, 2^64 - m, m^-1 mod 2^32
    uint32_t top;                                       // y >> 18
    float s;
    // X = y^2 - v m
    __device__ __forceinline__ void square(uint32_t &x0, uint32_t &x1) const
    {
        const float t = __fmul_rd(__uint_as_float(top), s);
        const uint32_t q = __float_as_uint(__fmaf_rd(t, t, (CK ? 12582911.0f : 8388606.0f) * 8.67361737988403547e-19f));
        const uint64_t a = (uint64_t)y0 * y0;
        const uint32_t u = (uint32_t)a * ip;
        const uint32_t v0 = __byte_perm(u, q, 0x4210), v1 = __byte_perm(q, 0u, 0x4421);
        const uint32_t p = y0 * y1 + (CK ? (0u - n0) << 13 : 0u);
        uint32_t h;
        asm("{\n\t.reg .u32 g;\n\t"
            "mad.lo.cc.u32 %0, %2, %3, %4;\n\t"         // y0^2 + v0 n0
            "madc.hi.u32 g, %2, %3, %5;\n\t"
            "mad.lo.u32 g, %2, %6, g;\n\t"              // + v0 n1 2^32
            "mad.lo.u32 %1, %7, %3, g;\n\t}"            // + v1 n0 2^32
            : "=&r"(x0), "=r"(h)
            : "r"(v0), "r"(n0), "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"(n1), "r"(v1));
        x1 = h + (p << 1);                              // + y0 (2 y1) 2^32
    }
    // y = X >> (24 - b)
    __device__ __forceinline__ void step(uint32_t b)
    {
        uint32_t x0, x1;
        square(x0, x1);
        const uint32_t sh = 8u | b;
        y0 = __funnelshift_l(x0, x1, sh);
        y1 = __funnelshift_l(x1, 0u, sh);
        top = __funnelshift_r(y0, y1, 18);
    }
    // Constants of the ladder and its start y = 2^(24 + p) up to a multiple of m,
    // 1 <= p <= 31: the float quotient (below 2^23) is within 2.5 of 2^(24+p) / m,
    // so y lies in (m/2, 4.5m) with two m added back. s: m rounded up, one Newton
    // step on the approximate root with the residual formed exactly, less one ulp.
    __device__ __forceinline__ void start(uint64_t m, uint32_t mp, uint32_t p)
    {
        const uint64_t n = 0ull - m;
        n0 = (uint32_t)n;
        n1 = (uint32_t)(n >> 32);
        ip = 0u - mp;
        const float fm = __fmaf_ru(__uint2float_rn((uint32_t)(m >> 32)), 4294967296.0f, __uint2float_ru((uint32_t)m));
        const float r0 = rsqrt_approx(fm);
        const float h = fm * r0;
        const float e = __fmaf_rn(-__fmaf_rn(fm, r0, -h), r0, __fmaf_rn(-h, r0, 1.0f));
        const float r = __fmaf_rn(0.5f * e, r0, r0);
        s = __uint_as_float(__float_as_uint(4.25352958651173080e37f * r) - 1u);     // 2^125 r
        const float i0 = r * r;
        const float inv = __fmaf_rn(i0, __fmaf_rn(-fm, i0, 1.0f), i0);
        const float scale = __int_as_float((int)((127u + 24u + p) << 23));          // 2^(24+p)
        const uint32_t q = __float2uint_rz(scale * inv);
        const uint64_t y = (1ull << (24 + p)) + 2 * m - (uint64_t)q * m;
        y0 = (uint32_t)y;
        y1 = (uint32_t)(y >> 32);
        top = __funnelshift_r(y0, y1, 18);
    }
    // y -> [0, m): a float quotient that is low by at most one.
    __device__ __forceinline__ uint64_t finish(uint64_t m) const
    {
        const float t = __fmul_rd(__uint_as_float(top), s);
        const uint32_t k = __float2uint_rz(__fmaf_rn(t * s, 1.03397576569128459e-25f, -0.001f));    // 2^-83
        const uint64_t y = (((uint64_t)y1 << 32) | y0) - (uint64_t)k * m;
        return min(y, y - m);
    }
};

// The ladder runs in Montgomery form with R = 2^24 on Ep = E - 24, Ep >= 2^5:
// the five leading bits at once, then one step a bit.
template <bool CK>
__device__ __forceinline__ uint64_t w2f_pow2(uint64_t E, uint64_t m, uint32_t mp)
{
    const uint64_t Ep = E - 24;
    W2FState<CK> st;
    int i = 64 - __clzll((long long)Ep) - 5;
    st.start(m, mp, (uint32_t)(Ep >> i));
    for (--i; i >= 0; --i) st.step((uint32_t)(Ep >> i) & 1u);
    return st.finish(m);
}

// Two ladders in turn, of terms whose exponents agree above bit S in the whole
// warp (e_max the largest, 630 above the smallest): those bits are taken from one
// value P, so that both ladders share the shift counts; the low S bits come from
// each exponent. A group across a multiple of 2^S (1 % at S = 16) runs its ladders
// one after the other. S = 13 measured 566.1 ms at 1e10, S = 16 561.6 ms. Exponents
// below 2^48 (kW2FExp) keep P in one word.
template <bool CK>
__device__ __forceinline__ void w2f_pow2_pair(uint64_t EA, uint64_t ma, uint32_t mpa, uint64_t EB, uint64_t mb,
                                              uint32_t mpb, uint64_t e_max, uint64_t &ra, uint64_t &rb)
{
    constexpr int S = 16;
    const uint32_t P = (uint32_t)((e_max - 24) >> S);
    if (e_max >= (1ull << (S + 6)) && (uint32_t)((e_max - 630 - 24) >> S) == P) {
        W2FState<CK> A, B;
        int j = 27 - __clz(P);
        A.start(ma, mpa, P >> j);
        B.start(mb, mpb, P >> j);
#pragma unroll 8
        for (--j; j >= 0; --j) {
            const uint32_t bit = (P >> j) & 1u;
            A.step(bit);
            B.step(bit);
        }
        const uint32_t la = (uint32_t)(EA - 24), lb = (uint32_t)(EB - 24);
#pragma unroll
        for (int l = S - 1; l >= 0; --l) {
            A.step(la >> l & 1u);
            B.step((l < 6 ? la : lb) >> l & 1u);        // EA - EB = 320 = 5 * 2^6
        }
        ra = A.finish(ma);
        rb = B.finish(mb);
        return;
    }
    ra = w2f_pow2<CK>(EA, ma, mpa);
    rb = w2f_pow2<CK>(EB, mb, mpb);
}

// ------------------------------------------------------- width 2, m >= 2^60 --
// 2^60 <= m < 2^62 (positions up to 999999999999999999): residues in [0, 2m).
// REDC(y^2) < 4m^2/2^64 + m < 2m still holds and T + U m < 2^127, so the
// two-word step of w2_sqr applies; only the doubling needs min(y, y - 2m).
struct W2XState {
    uint32_t y0, y1, m0, m1, mp;
    uint64_t m2;                                        // 2m
    __device__ __forceinline__ void step(uint32_t b)
    {
        w2_sqr(y0, y1, m0, m1, mp, b);                  // < 4m < 2^64
        uint64_t y = ((uint64_t)y1 << 32) | y0;
        y = min(y, y - m2);                             // < 2m
        y0 = (uint32_t)y;
        y1 = (uint32_t)(y >> 32);
    }
};

__device__ __forceinline__ W2XState w2x_state(uint64_t m, uint32_t mp)
{
    return W2XState{0, 0, (uint32_t)m, (uint32_t)(m >> 32), mp, 2 * m};
}

// r6 = 2^E mod m in [0, m) for E >= 65, 2^44 <= m < 2^62.
__device__ __forceinline__ uint64_t w2x_pow2(uint64_t E, uint64_t m, uint32_t mp)
{
    W2XState st = w2x_state(m, mp);
    walk_bits_start<4>(E - 64, st, W2Start<64>{});
    const uint64_t r = two_words(st.y0, st.y1);         // below 2m
    return min(r, r - m);
}

// N REDC steps down from r < m (two-word m): q[j] are the quotient digits and
// the result is r 2^(-32 N) mod m.
template <int N>
__device__ __forceinline__ uint64_t w2_redc_down(uint64_t r, uint64_t m, uint32_t mp, uint32_t q[N])
{
    const uint32_t m0 = (uint32_t)m, m1 = (uint32_t)(m >> 32);
    uint32_t r0 = (uint32_t)r, r1 = (uint32_t)(r >> 32);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        q[j] = r0 * mp;
        // (r + q m) / 2^32 = hi(q m0 + r) + c 2^32 + q m1 < m, c the carry out
        asm("{\n\t.reg .u32 x, h, c;\n\t"
            "mad.lo.cc.u32 x, %2, %3, %4;\n\t"
            "madc.hi.cc.u32 h, %2, %3, %5;\n\t"
            "addc.u32 c, 0, 0;\n\t"
            "mad.lo.cc.u32 %0, %2, %6, h;\n\t"
            "madc.hi.u32 %1, %2, %6, c;\n\t}"
            : "=r"(r0), "=r"(r1)
            : "r"(q[j]), "r"(m0), "r"(r0), "r"(r1), "r"(m1));
    }
    return ((uint64_t)r1 << 32) | r0;
}

// Two ladders at once (terms k and k+32 of one lane): when both exponents have
// the same bit length (in the same word) the steps interleave, giving the
// scheduler two independent chains; otherwise they run one after the other.
template <int NB, typename State, typename Start>
__device__ __forceinline__ void walk_bits_start_pair(uint64_t EpA, uint64_t EpB, State &A, State &B, Start start)
{
    const uint32_t ha = (uint32_t)(EpA >> 32), la = (uint32_t)EpA, hb = (uint32_t)(EpB >> 32), lb = (uint32_t)EpB;
    const uint32_t wa = ha ? ha : la, wb = hb ? hb : lb;         // word holding the leading bits
    const int nba = 32 - __clz(wa), nbb = 32 - __clz(wb);
    if ((ha == 0) != (hb == 0) || nba != nbb || nba < NB) {
        walk_bits_start<NB>(EpA, A, start);
        walk_bits_start<NB>(EpB, B, start);
        return;
    }
    start(A, wa >> (nba - NB));
    start(B, wb >> (nbb - NB));
    uint32_t ga = (nba - NB) > 0 ? wa << (32 - (nba - NB)) : 0u, gb = (nbb - NB) > 0 ? wb << (32 - (nbb - NB)) : 0u;
    const int n = ha != 0 ? nba : nba - 1;                       // the last bit is not among these
    for (int i = NB; i < n; ++i) {
        A.step(ga >> 31);
        B.step(gb >> 31);
        ga <<= 1;
        gb <<= 1;
    }
    if (ha != 0) {
#pragma unroll
        for (int i = 31; i >= 1; --i) {
            A.step((la >> i) & 1u);
            B.step((lb >> i) & 1u);
        }
    }
    last_step(A, la & 1u);
    last_step(B, lb & 1u);
}

// Two ladders of a warp's group of 64 terms (k and k+32 of every lane; ep_max the
// group's largest exponent, 630 above its smallest). When the group's exponents
// agree above bit S, those bits come from one word P and both ladders share the
// shift counts, and so they do in the last six bits (EpA - EpB = 320 = 5 * 2^6).
// Other groups, and exponents outside [2^(S+4) + 630, 2^(S+32)), walk their own bits.
// LONG (the short two-word kind): exponents from 2^(S+32) on too, whose bits above S are
// walked in two words (2^28 terms at 1e14, m from 2e12 on: 11.51 ms; 11.78 ms when such
// groups walked their own bits). The general kinds do without: with it there too the
// short kind ran 0.5 % slower at 1e13 (10.82 against 10.76 ms), one kernel holding all.
// S = 12 / 13 / 14 / 15 / 16 measured 113.9 / 110.4 / 108.9 / 108.2 / 107.6 ms on 512 positions
// below 1e8.
constexpr int kGroupBits = 16;
template <int NB, bool LONG = false, typename State, typename Start>
__device__ __forceinline__ void walk_bits_group(uint64_t EpA, uint64_t EpB, uint64_t ep_max, State &A, State &B,
                                                Start start)
{
    constexpr int S = kGroupBits;
    const uint32_t P = (uint32_t)(ep_max >> S);
    if (ep_max >= (1ull << (S + 4)) + 630 && (LONG || ep_max >> (S + 32) == 0) &&
        (LONG ? (ep_max - 630) >> S == ep_max >> S : (uint32_t)((ep_max - 630) >> S) == P)) {
        const uint32_t over = LONG ? (uint32_t)(ep_max >> (S + 32)) : 0u;
        int more = 32 - __clz(over);                         // common bits below the first word's
        uint32_t W = LONG ? __funnelshift_r(P, over, more) : P;
        int j = 32 - NB - __clz(W);
        start(A, W >> j);
        start(B, W >> j);
        for (;;) {
#pragma unroll 4
            for (--j; j >= 0; --j) {
                const uint32_t b = (W >> j) & 1u;
                A.step(b);
                B.step(b);
            }
            if (!LONG || more == 0) break;
            W = P;
            j = more;
            more = 0;
        }
        const uint32_t la = (uint32_t)EpA, lb = (uint32_t)EpB;
#pragma unroll
        for (int l = S - 1; l >= 1; --l) {
            A.step((la >> l) & 1u);
            B.step(((l < 6 ? la : lb) >> l) & 1u);
        }
        last_step(A, la & 1u);
        last_step(B, la & 1u);
        return;
    }
    walk_bits_start_pair<NB>(EpA, EpB, A, B, start);
}

struct W1Start1 {                                        // the single-bit start of the width-1 kind
    __device__ __forceinline__ void operator()(W1State &st, uint32_t) const { st.y = w1_start(st.m); }
};

// ------------------------------------------------------------ fixed point --
// Accumulator of N 32-bit digits, digit 0 least significant: 192 bits for the
// integer mode, 128 for the double-double mode's terms.
template <int N>
struct Acc {
    uint32_t w[N];
};
typedef Acc<6> Acc192;

template <int N>
__device__ __forceinline__ void acc_zero(Acc<N> &a)
{
#pragma unroll
    for (int j = 0; j < N; ++j) a.w[j] = 0;
}

__device__ __forceinline__ void acc_add(Acc<6> &a, const uint32_t q[6])
{
    asm("add.cc.u32  %0, %0, %6;\n\t"
        "addc.cc.u32 %1, %1, %7;\n\t"
        "addc.cc.u32 %2, %2, %8;\n\t"
        "addc.cc.u32 %3, %3, %9;\n\t"
        "addc.cc.u32 %4, %4, %10;\n\t"
        "addc.u32    %5, %5, %11;"
        : "+r"(a.w[0]), "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3]), "+r"(a.w[4]), "+r"(a.w[5])
        : "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]));
}

__device__ __forceinline__ void acc_add(Acc<4> &a, const uint32_t q[4])
{
    asm("add.cc.u32  %0, %0, %4;\n\t"
        "addc.cc.u32 %1, %1, %5;\n\t"
        "addc.cc.u32 %2, %2, %6;\n\t"
        "addc.u32    %3, %3, %7;"
        : "+r"(a.w[0]), "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3])
        : "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]));
}

// a <- -a (mod 2^128).
__device__ __forceinline__ void acc_negate(Acc<4> &a)
{
    asm("sub.cc.u32  %0, 0, %0;\n\t"
        "subc.cc.u32 %1, 0, %1;\n\t"
        "subc.cc.u32 %2, 0, %2;\n\t"
        "subc.u32    %3, 0, %3;"
        : "+r"(a.w[0]), "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3]));
}

// a <- -a - c (mod 2^192): the sum of c negative terms NOT(q_i) = -q_i - 1.
__device__ __forceinline__ void acc_negate_minus(Acc192 &a, uint32_t c)
{
    // -a - c = ~a + (1 - c), with (1 - c) sign-extended to 192 bits.
#pragma unroll
    for (int j = 0; j < 6; ++j) a.w[j] = ~a.w[j];
    const uint32_t add = 1u - c;
    const uint32_t ext = (c > 1) ? 0xffffffffu : 0u;
    asm("add.cc.u32  %0, %0, %6;\n\t"
        "addc.cc.u32 %1, %1, %7;\n\t"
        "addc.cc.u32 %2, %2, %7;\n\t"
        "addc.cc.u32 %3, %3, %7;\n\t"
        "addc.cc.u32 %4, %4, %7;\n\t"
        "addc.u32    %5, %5, %7;"
        : "+r"(a.w[0]), "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3]), "+r"(a.w[4]), "+r"(a.w[5])
        : "r"(add), "r"(ext));
}

}  // namespace cbl
