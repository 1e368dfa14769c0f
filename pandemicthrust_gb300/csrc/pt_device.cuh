// pt_device.cuh - device-side building blocks of the daily simulation step:
// Threefry counters, the float "fishing" lookups and the model tables.
//
// Every float operation that decides a result uses an explicit round-to-nearest
// intrinsic (__fmul_rn, __fdiv_rn, __fsub_rn, __uint2float_rn), so the arithmetic
// matches the reference's IEEE single-precision code whatever the compiler flags
// (no contraction, no approximate division).
#pragma once
#include <cstdint>
#include "pt_kernels.h"

namespace ptk {

// ---------------------------------------------------------------- tables
// PandemicSim.cu:328-481 (model constants; identical in every simulation).
static __constant__ float c_child_age_cdf[5] = {0.24f, 0.47f, 0.72f, 0.85f, 1.0f};
static __constant__ float c_workplace_pdf[kTypes] = {
    0.06586f, 0.05802f, 0.30227f, 0.0048f, 0.00997f, 0.203f, 0.09736f,
    0.10598f, 0.00681f, 0.02599f, 0.f, 0.08749f, 0.03181f, 0.00064f};
static __constant__ int c_type_max_contacts[kTypes] = {3, 3, 3, 2, 2, 3, 3, 2, 2, 2, 0, 2, 2, 2};
static __constant__ float c_weekday_errand_pdf[kTypes] = {0, 0, 0, 0, 0, 0, 0, 0, 0,
                                                   0.61919f, 0, 0.27812f, 0.06601f, 0.03668f};
static __constant__ float c_weekend_errand_pdf[kTypes] = {0, 0, 0, 0, 0, 0, 0, 0, 0,
                                                   0.51493f, 0, 0.25586f, 0.1162f, 0.113f};
// The reciprocals of the errand probabilities, rounded to nearest (each quotient
// folded by the compiler in IEEE single precision; 0 where the probability is 0,
// a row the search below never ends on).
static __constant__ float c_weekday_errand_rcp[kTypes] = {0, 0, 0, 0, 0, 0, 0, 0, 0,
                                                   1.0f / 0.61919f, 0, 1.0f / 0.27812f, 1.0f / 0.06601f,
                                                   1.0f / 0.03668f};
static __constant__ float c_weekend_errand_rcp[kTypes] = {0, 0, 0, 0, 0, 0, 0, 0, 0,
                                                   1.0f / 0.51493f, 0, 1.0f / 0.25586f, 1.0f / 0.1162f,
                                                   1.0f / 0.113f};
static __constant__ int c_hh_adults[9] = {1, 1, 2, 1, 2, 1, 2, 1, 2};
static __constant__ int c_hh_children[9] = {0, 1, 0, 2, 1, 3, 2, 4, 3};
static __constant__ float c_hh_cdf[9] = {0.279f, 0.319f, 0.628f, 0.671f, 0.8f, 0.812f, 0.939f, 0.944f, 1.0f};
// Contacts per errand hour for weekday profiles 0..3 (3 = afterschool) and the
// errand slot of each of the two weekend errand contacts (PandemicSim.cu:445-481).
static __constant__ int c_weekday_assign[4][2] = {{2, 0}, {0, 2}, {1, 1}, {2, 0}};
static __constant__ int c_weekend_assign[6][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {0, 2}, {1, 2}};

// ---------------------------------------------------------------- Threefry
// Threefry-2x64-20 and 2x32-20 (Salmon et al., SC'11; the Random123 rotation
// tables).  The integer (ALU) pipe bounds every kernel that draws many blocks: a
// 64-bit rotation is two funnel shifts and an XOR two logic operations, 76 ALU
// instructions a block, and each 64-bit add takes two more.  So the adds are kept off
// that pipe where it can be done: the high word is a multiply-add with carry by a 1 the
// compiler cannot see (FMA pipe), the first round's sum of the two key-added counter
// words is 2 ctr + (k0 + k1), and each key injection of x0 is folded into the next
// round's add (three operands).  Measured alone on a GB300: 110 ALU and 135
// instructions a block, 239 cycles a warp, against 126 / 147 / 275 with plain
// add / add-with-carry pairs, 257 with every add as a multiply-add, 300 and more with
// rotations or low words as wide multiplies.
struct u64h { uint32_t lo, hi; };

__device__ __forceinline__ u64h mk(uint64_t v) { return {(uint32_t)v, (uint32_t)(v >> 32)}; }
__device__ __forceinline__ uint64_t pack64(u64h v) { return ((uint64_t)v.hi << 32) | v.lo; }

static __constant__ uint32_t c_one = 1u;   // (not const: the compiler may not fold it)

__device__ __forceinline__ uint64_t add64(uint64_t a, uint64_t b)
{
    const u64h x = mk(a), y = mk(b);
    u64h r;
    asm("add.cc.u32 %0, %2, %4;\n\tmadc.lo.u32 %1, %3, %6, %5;"
        : "=r"(r.lo), "=r"(r.hi) : "r"(x.lo), "r"(x.hi), "r"(y.lo), "r"(y.hi), "r"(c_one));
    return pack64(r);
}

template <int R>
__device__ __forceinline__ uint64_t rotl64(uint64_t v)
{
    const u64h x = mk(v);
    if constexpr (R == 32) {
        return pack64({x.hi, x.lo});
    } else if constexpr (R < 32) {
        return pack64({__funnelshift_l(x.hi, x.lo, R), __funnelshift_l(x.lo, x.hi, R)});
    } else {
        return pack64({__funnelshift_l(x.lo, x.hi, R - 32), __funnelshift_l(x.hi, x.lo, R - 32)});
    }
}

struct TfKey {
    uint64_t k0, k1, k2;   // key schedule: k2 = parity ^ k0 ^ k1
    uint32_t k32_0, k32_1, k32_2;
};

__device__ __forceinline__ TfKey make_key(const SimConst &c)
{
    TfKey k;
    k.k0 = c.key0;
    k.k1 = c.key1;
    k.k2 = 0x1BD11BDAA9FC1A22ULL ^ c.key0 ^ c.key1;
    k.k32_0 = (uint32_t)c.key0;
    k.k32_1 = (uint32_t)c.key1;
    k.k32_2 = 0x1BD11BDAu ^ k.k32_0 ^ k.k32_1;
    return k;
}

// Counter {ctr, ctr}; returns the block as the reference's union reads it:
// w[0] = lo(x0), w[1] = hi(x0), w[2] = lo(x1), w[3] = hi(x1).
__device__ __forceinline__ void tf2x64(const TfKey &k, uint64_t ctr, uint32_t w[4])
{
    // x0 holds the sum of a round; x1 its rotated and XORed word
    uint64_t x0 = 2 * ctr + (k.k0 + k.k1), x1 = ctr + k.k1;
    const uint64_t ks[3] = {k.k0, k.k1, k.k2};
#pragma unroll
    for (int blk = 0; blk < 5; blk++) {
        x1 = rotl64<16>(x1) ^ x0;
        x0 = add64(x1, x0);
        x1 = ((blk & 1) == 0 ? rotl64<42>(x1) : rotl64<32>(x1)) ^ x0;
        x0 = add64(x1, x0);
        x1 = ((blk & 1) == 0 ? rotl64<12>(x1) : rotl64<24>(x1)) ^ x0;
        x0 = add64(x1, x0);
        x1 = ((blk & 1) == 0 ? rotl64<31>(x1) : rotl64<21>(x1)) ^ x0;
        const int s = blk + 1;
        x1 += ks[(s + 1) % 3] + (uint64_t)s;
        x0 += s < 5 ? ks[s % 3] + x1 : ks[s % 3];   // with the next round's add
    }
    w[0] = (uint32_t)x0; w[1] = (uint32_t)(x0 >> 32); w[2] = (uint32_t)x1; w[3] = (uint32_t)(x1 >> 32);
}

template <int R>
__device__ __forceinline__ void mix32(uint32_t &x0, uint32_t &x1)
{
    x0 += x1;
    x1 = __funnelshift_l(x1, x1, R);
    x1 ^= x0;
}

__device__ __forceinline__ void tf2x32(const TfKey &k, uint32_t ctr, uint32_t w[2])
{
    uint32_t x0 = ctr + k.k32_0, x1 = ctr + k.k32_1;
    const uint32_t ks[3] = {k.k32_0, k.k32_1, k.k32_2};
#pragma unroll
    for (int blk = 0; blk < 5; blk++) {
        if ((blk & 1) == 0) {
            mix32<13>(x0, x1); mix32<15>(x0, x1); mix32<26>(x0, x1); mix32<6>(x0, x1);
        } else {
            mix32<17>(x0, x1); mix32<29>(x0, x1); mix32<16>(x0, x1); mix32<24>(x0, x1);
        }
        const uint32_t s = blk + 1;
        x0 += ks[s % 3];
        x1 += ks[(s + 1) % 3] + s;
    }
    w[0] = x0; w[1] = x1;
}

// ---------------------------------------------------------------- fishing
// (float)r / UNSIGNED_MAX: the divisor converts to 2^32, so this is exact scaling.
__device__ __forceinline__ float to_unit(uint32_t r) { return __fmul_rn(__uint2float_rn(r), 0x1p-32f); }

// device_setup_fishHouseholdType, PandemicSim.cu:2360-2371
__device__ __forceinline__ int fish_household_type(uint32_t r)
{
    float y = to_unit(r);
    int row = 0;
    while (y > c_hh_cdf[row] && row < 8) row++;
    return row;
}

__device__ __forceinline__ int business_in_type(const SimConst &c, float frac, int type)
{
    int count = c.type_count[type];
    int b = __float2int_rz(__fmul_rn(frac, __int2float_rn(count)));
    if (b >= count) b = count - 1;
    return b + c.type_offset[type];
}

// device_setup_fishWorkplace, PandemicSim.cu:2374-2399
__device__ __forceinline__ int fish_workplace(const SimConst &c, uint32_t r)
{
    float y = to_unit(r);
    int row = 0;
    while (c_workplace_pdf[row] < y && row < kTypes - 1) {
        y = __fsub_rn(y, c_workplace_pdf[row]);
        row++;
    }
    return business_in_type(c, __fdiv_rn(y, c_workplace_pdf[row]), row);
}

// device_setup_fishSchoolAndAge, PandemicSim.cu:2402-2442
__device__ __forceinline__ int fish_school_and_age(const SimConst &c, uint32_t r, int *age)
{
    float y = to_unit(r);
    int row = 0;
    while (row < 4 && y > c_child_age_cdf[row]) row++;
    float frac;
    if (row == 0) {
        frac = __fdiv_rn(y, c_child_age_cdf[0]);
    } else {
        float pdf_here = __fsub_rn(c_child_age_cdf[row], c_child_age_cdf[row - 1]);
        float y_here = __fsub_rn(y, c_child_age_cdf[row - 1]);
        frac = __fdiv_rn(y_here, pdf_here);
    }
    *age = row;
    return business_in_type(c, frac, row + 3);
}

// x / d rounded to nearest, for the errand probabilities d with r = RN(1/d): one
// multiply and Markstein's correction (P. Markstein, IBM J. Res. Dev. 34(1), 1990):
// q = RN(x r), e = x - q d exactly (a fused multiply-add), RN(q + e r).  It equals
// __fdiv_rn(x, d) for x = 0 and every float x in [2^-32, 1] (the values the errand
// search divides) and every row the search can end on; pt_selftest_errand_lookup
// checks all of them, and the whole search on every 32-bit draw.
__device__ __forceinline__ float div_rn_recip(float x, float d, float r)
{
    const float q = __fmul_rn(x, r);
    const float e = __fmaf_rn(-q, d, x);
    return __fmaf_rn(e, r, q);
}

// The errand-type search of device_fishAfterschoolOrErrandDestination_weekday (its
// adult branch, PandemicSim.cu:2909-2947) and device_fishWeekendErrandDestination
// (PandemicSim.cu:1017-1044):
//     row = 9; while (y > pdf[row] && row < 13) { y = y - pdf[row]; row++; }
//     frac = y / pdf[row];
// without branches.  The chain of subtractions runs to the end and the stop is
// selected: once y <= pdf[t], every later remainder is <= 0 (the probabilities are
// >= 0), so every later test fails too, as the loop would have stopped.  Returns the
// row; frac receives the quotient.
template <bool WEEKEND>
__device__ __forceinline__ int errand_row(float y, float &frac)
{
    const float *pdf = WEEKEND ? c_weekend_errand_pdf : c_weekday_errand_pdf;
    const float *rcp = WEEKEND ? c_weekend_errand_rcp : c_weekday_errand_rcp;
    float x = y, d = pdf[9], rd = rcp[9], f = y;
    int row = 9;
#pragma unroll
    for (int t = 9; t < kTypes - 1; t++) {
        const bool go = f > pdf[t];
        f = __fsub_rn(f, pdf[t]);
        row = go ? t + 1 : row;
        x = go ? f : x;
        d = go ? pdf[t + 1] : d;
        rd = go ? rcp[t + 1] : rd;
    }
    frac = div_rn_recip(x, d, rd);
    return row;
}

// The same search as the reference writes it: the loop and the IEEE division.  Kept
// as the self-test's reference for errand_row.
template <bool WEEKEND>
__device__ __forceinline__ int errand_row_loop(float y, float &frac)
{
    const float *pdf = WEEKEND ? c_weekend_errand_pdf : c_weekday_errand_pdf;
    int row = 9;
    while (y > pdf[row] && row < kTypes - 1) {
        y = __fsub_rn(y, pdf[row]);
        row++;
    }
    frac = __fdiv_rn(y, pdf[row]);
    return row;
}

// The schedule kernel's form of the same draw.  A destination is row i of an errand
// table in shared memory (ErrandRow, built per instance and hour): rows 0-3 are the
// errand types 9, 11, 12 and 13, row 4 the afterschool type 8 of weekday children.
// Everything runs on the draw itself, w = (float)r, with every probability scaled by
// 2^32: scaling by a power of two commutes with each rounding below, so row, quotient
// and business number are those of errand_row.  Type 10 has probability 0 and a
// remainder past type 9 is above 0, so the search never ends there and its
// subtraction of 0 is left out.
constexpr float kTwo32 = 4294967296.f;
template <bool WEEKEND>
struct ErrandPdf {
    static constexpr float p9 = (WEEKEND ? 0.51493f : 0.61919f), p11 = (WEEKEND ? 0.25586f : 0.27812f),
                           p12 = (WEEKEND ? 0.1162f : 0.06601f), p13 = (WEEKEND ? 0.113f : 0.03668f);
};
constexpr int kErrandRows = 5;

struct __align__(32) ErrandRow {
    float d, r;     // 2^32 x the type's probability and 2^-32 x its reciprocal rounded to nearest
    float count;    // locations of the type
    int first;      // bucket of the type's first location in this hour
    int last;       // and of its last one
};

// Row i of the table of one hour.
template <bool WEEKEND>
__device__ __forceinline__ ErrandRow errand_table_row(const SimConst &c, int i, int hour_base, int lo)
{
    typedef ErrandPdf<WEEKEND> P;
    const int type = i == 4 ? 8 : (i == 0 ? 9 : 10 + i);
    ErrandRow e;
    // children: the quotient is the draw itself, y = w 2^-32
    e.d = i == 4 ? kTwo32 : kTwo32 * (i == 0 ? P::p9 : (i == 1 ? P::p11 : (i == 2 ? P::p12 : P::p13)));
    e.r = (i == 4 ? 1.f : (i == 0 ? 1.0f / P::p9 : (i == 1 ? 1.0f / P::p11 : (i == 2 ? 1.0f / P::p12 : 1.0f / P::p13)))) /
          kTwo32;
    e.count = __int2float_rn(c.type_count[type]);
    e.first = hour_base + c.type_offset[type] - lo;
    e.last = e.first + c.type_count[type] - 1;
    return e;
}

// 1 when x > 0, else 0, for |x| = 0 or >= 2^-60
__device__ __forceinline__ float unit_step(float x)
{
    float t;
    asm("mul.rn.sat.f32 %0, %1, 0f6F800000;" : "=f"(t) : "f"(x));   // x 2^96, clamped to [0, 1]
    return t;
}

// The byte offset of draw w's row in a table (`base`: the offset of row 0, or of row 4
// with `p9` above every draw, for a child) and the remainder x the quotient divides.
// All on the floating-point pipe, which the Threefry blocks leave idle: the steps
// t1 >= t2 >= t3 are 0 or 1 (differences of floats are 0 or far above 2^-60 here), x
// takes the subtractions in the loop's order and rounding, and the offset is summed
// in the bits of denormal floats, where adding is integer adding.
constexpr float kNoRow = 0x1p100f;   // p9 of a child: no draw exceeds it
template <bool WEEKEND>
__device__ __forceinline__ int errand_step(float w, float p9, int base, float &x)
{
    typedef ErrandPdf<WEEKEND> P;
    constexpr float p11 = kTwo32 * P::p11, p12 = kTwo32 * P::p12;
    const float f1 = __fsub_rn(w, p9), f2 = __fsub_rn(f1, p11), f3 = __fsub_rn(f2, p12);
    const float t1 = unit_step(f1), t2 = unit_step(f2), t3 = unit_step(f3);
    x = __fmaf_rn(-t3, p12, __fmaf_rn(-t2, p11, __fmaf_rn(-t1, p9, w)));
    constexpr int row = (int)sizeof(ErrandRow);
    const float step = __int_as_float(row);
    return __float_as_int(__fmaf_rn(t3, step, __fmaf_rn(t2, step, __fmaf_rn(t1, step, __int_as_float(base)))));
}

template <bool WEEKEND>
__device__ __forceinline__ float errand_p9(bool adult) { return adult ? kTwo32 * ErrandPdf<WEEKEND>::p9 : kNoRow; }

// The bucket draw r falls into: business_in_type's rounding and clamp on the table.
template <bool WEEKEND>
__device__ __forceinline__ int errand_bucket(const ErrandRow *rows, uint32_t r, float p9, int base)
{
    float x;
    const int at = errand_step<WEEKEND>(__uint2float_rn(r), p9, base, x);
    const ErrandRow &e = *reinterpret_cast<const ErrandRow *>(reinterpret_cast<const char *>(rows) + at);
    const float4 q = *reinterpret_cast<const float4 *>(&e.d);   // d, r, count, first
    const int b = __float2int_rz(__fmul_rn(div_rn_recip(x, q.x, q.y), q.z));
    return min(__float_as_int(q.w) + b, e.last);
}

// device_fishAfterschoolOrErrandDestination_weekday, PandemicSim.cu:2909-2947
// (unsigned business number, as the reference).  Children go to an afterschool
// location (type 8); adults to an errand type drawn by errand_row.  Both are computed
// and one is selected, so a warp of adults and children does not diverge.
__device__ __forceinline__ int fish_weekday_dest(const SimConst &c, uint32_t r, bool adult)
{
    const float y = to_unit(r);
    float fa;
    const int ta = errand_row<false>(y, fa);
    const int type = adult ? ta : 8;   // 8: BUSINESS_TYPE_AFTERSCHOOL
    const float frac = adult ? fa : y;
    int count = c.type_count[type];
    unsigned int b = __float2uint_rz(__fmul_rn(frac, __int2float_rn(count)));
    if (b >= (unsigned int)count) b = (unsigned int)(count - 1);
    b += (unsigned int)c.type_offset[type];
    return (int)b;
}

// device_fishWeekendErrandDestination, PandemicSim.cu:1017-1044
__device__ __forceinline__ int fish_weekend_dest(const SimConst &c, uint32_t r)
{
    float frac;
    const int row = errand_row<true>(to_unit(r), frac);
    return business_in_type(c, frac, row);
}

// device_generateWeekendErrands, PandemicSim.cu:980-1014: three distinct hours of
// ten, each with a destination.  The reference's key is destination + hour * L;
// weekend destinations all lie in [lo, L) (lo = first location of type 9), so the
// bucket index used here is the order-preserving compact form hour * R + dest - lo,
// R = L - lo.
__device__ __forceinline__ void weekend_hours(const uint32_t w[3], int &h1, int &h2, int &h3)
{
    h1 = (int)(w[0] % 10u);
    h2 = (int)(w[1] % 10u);
    h3 = (int)(w[2] % 10u);
    if (h2 == h1) h2 = h2 == 9 ? 0 : h2 + 1;
    // h1 and h2 differ, so two steps pass both whichever comes first
    if (h3 == h1 || h3 == h2) h3 = h3 == 9 ? 0 : h3 + 1;
    if (h3 == h1 || h3 == h2) h3 = h3 == 9 ? 0 : h3 + 1;
}

__device__ __forceinline__ void weekend_errands(const SimConst &c, const TfKey &k, uint64_t ctr, int lo, int R,
                                                int out[3])
{
    uint32_t w[8];
    tf2x64(k, ctr, w);
    tf2x64(k, ctr + 1, w + 4);
    int h1, h2, h3;
    weekend_hours(w, h1, h2, h3);
    out[0] = fish_weekend_dest(c, w[3]) - lo + h1 * R;
    out[1] = fish_weekend_dest(c, w[4]) - lo + h2 * R;
    out[2] = fish_weekend_dest(c, w[5]) - lo + h3 * R;
}

// ---------------------------------------------------------------- interventions
// The interventions have no counterpart in the reference.  Their random choices come
// from this hash, not from the reference's Threefry counter stream, so a run whose
// interventions are all zero draws exactly the reference's numbers.  The mix is the
// splitmix64 finaliser (Steele, Lea and Flood, OOPSLA 2014); the high 32 bits of
// mix(mix(key0 ^ (key1 << 1) ^ tag) ^ (day << 32 | person)) decide.
__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__host__ __device__ __forceinline__ uint64_t intervention_hash(uint64_t key0, uint64_t key1, uint64_t tag, int day,
                                                               int person)
{
    const uint64_t k = splitmix64(key0 ^ (key1 << 1) ^ tag);
    return splitmix64(k ^ (((uint64_t)(uint32_t)day << 32) | (uint32_t)person)) >> 32;
}

// School-type locations: types 3-7 (the children's schools by age band,
// PandemicSim.cu:2402-2442), contiguous in location order.
__device__ __forceinline__ bool is_school(const SimConst &c, int loc)
{
    return loc >= c.type_offset[3] && loc < c.type_offset[7] + c.type_count[7];
}

// device_getWorkplaceMaxContacts, PandemicSim.cu:3492-3511
__device__ __forceinline__ int workplace_max_contacts(const SimConst &c, int loc)
{
    int lid = loc % c.L;
    int t = 0, off, cnt, mx;
    do {
        off = c.type_offset[t];
        cnt = c.type_count[t];
        mx = c_type_max_contacts[t];
        t++;
    } while (lid >= off + cnt);
    return mx;
}

// device_getInfectionProfile, PandemicSim.cu:3974-3988
__device__ __forceinline__ int infection_profile(const SimConst &c, uint32_t r)
{
    int p = (int)(r % 3u) + 2;
    if (to_unit(r) > c.pct_sympt) p += 3;
    return p;
}

// device_calculateInfectionProbability, PandemicSim.cu:2307-2326
__device__ __forceinline__ float infection_probability(const SimConst &c, int profile, int pday, int strain, int ksum)
{
    if (ksum == 0) ksum = 1;
    float avg = __fmul_rn(c.shedding[profile][pday], c.infectiousness[strain]);
    return __fdiv_rn(avg, __int2float_rn(ksum));
}

}  // namespace ptk
