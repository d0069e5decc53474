/*
 * IEEE-754 binary64 addition, subtraction and multiplication, rounded to nearest with ties to even,
 * computed with 32-bit integer instructions.
 *
 * Why: the step kernels are bound by the fp64 pipe, which takes an addition or multiplication of a warp
 * every 19 cycles per SM, while the 32-bit pipes mostly idle.  Issuing a share of a kernel's fp64
 * operations through these functions runs the pipes side by side.  The results are bit-identical to the
 * hardware instruction for every input, so the arithmetic of the step (and its parity with the
 * reference) does not change.  Cost per warp and SM, measured in streams of independent operations: an
 * addition 25 cycles (57 instructions, 45 of them on the ALU pipe, which takes one every half cycle), a
 * multiplication by a prepared factor 12 cycles (31 instructions, 14 ALU and 14 multiply-add).
 *
 * Method (the definition of the format, nothing more): unpack sign, exponent and significand; for a
 * sum, align the smaller significand, add or subtract, normalise; for a product, form the product of
 * the significands from 32 x 32-bit partial products; round to nearest even.  The fast path covers
 * normal operands with a normal result; everything else is handed to the hardware instruction in a
 * branch that is not taken in practice.  Bits that only decide rare ties are not formed at all: where
 * they could matter, the hardware decides too.  The host build of the same source (tests) checks the
 * fast path against the host's IEEE arithmetic.
 */
#ifndef FQSB_FQ_SOFT64_H
#define FQSB_FQ_SOFT64_H

#include "fq_math.h"

#if defined(__CUDA_ARCH__)
/* Slow paths: not inlined, so the compiler branches around them instead of predicating an fp64
 * instruction into every call site (a predicated one takes its pipe cycles even when no lane needs it:
 * the step at N = 2^22 takes 225 us with inlined ones, 159 us with calls). */
static __device__ __noinline__ double fq_s_hw_add(double a, double b)
{
    return __dadd_rn(a, b);
}
static __device__ __noinline__ double fq_s_hw_mul(double a, double b)
{
    return __dmul_rn(a, b);
}
FQ_HD uint32_t fq_s_lo(double x)
{
    return (uint32_t)__double2loint(x);
}
FQ_HD uint32_t fq_s_hi(double x)
{
    return (uint32_t)__double2hiint(x);
}
FQ_HD double fq_s_make(uint32_t hi, uint32_t lo)
{
    return __hiloint2double((int)hi, (int)lo);
}
/* (hi:lo) >> n, low word, n in [0, 32] */
FQ_HD uint32_t fq_s_shr64lo(uint32_t lo, uint32_t hi, uint32_t n)
{
    return __funnelshift_rc(lo, hi, n);
}
/* (hi:lo) << n, high word, n in [0, 32] */
FQ_HD uint32_t fq_s_shl64hi(uint32_t lo, uint32_t hi, uint32_t n)
{
    return __funnelshift_lc(lo, hi, n);
}
FQ_HD uint32_t fq_s_max(uint32_t a, uint32_t b)
{
    return umax(a, b);
}
FQ_HD uint32_t fq_s_min(uint32_t a, uint32_t b)
{
    return umin(a, b);
}
FQ_HD uint32_t fq_s_clz(uint32_t x)
{
    return (uint32_t)__clz((int)x);
}
/* subtract: (mh:ml:g) = (xh:xl:0) - (h:l:g), else (xh:xl:0) + (h:l:g); one predicated chain each */
FQ_HD void fq_s_addsub96(uint32_t diff, uint32_t xh, uint32_t xl, uint32_t h, uint32_t l, uint32_t& g, uint32_t& mh,
                         uint32_t& ml)
{
    asm("{\n\t"
        ".reg .pred p;\n\t"
        "setp.lt.s32 p, %7, 0;\n\t"
        "@p sub.cc.u32  %0, 0, %0;\n\t"
        "@p subc.cc.u32 %1, %4, %6;\n\t"
        "@p subc.u32    %2, %3, %5;\n\t"
        "@!p add.cc.u32 %1, %4, %6;\n\t"
        "@!p addc.u32   %2, %3, %5;\n\t"
        "}"
        : "+r"(g), "=&r"(ml), "=&r"(mh)
        : "r"(xh), "r"(xl), "r"(h), "r"(l), "r"(diff));
}
/* (rh:rl) = (ah:al) + (c != 0) */
FQ_HD void fq_s_add64c(uint32_t ah, uint32_t al, uint32_t c, uint32_t& rh, uint32_t& rl)
{
    asm("{\n\t"
        ".reg .u32 t;\n\t"
        "add.cc.u32  t, %4, 0xffffffff;\n\t"
        "addc.cc.u32 %0, %2, 0;\n\t"
        "addc.u32    %1, %3, 0;\n\t"
        "}"
        : "=&r"(rl), "=r"(rh)
        : "r"(al), "r"(ah), "r"(c));
}
/* (rh:rl) = (ah:al) + (t:0) + (g >= 2^31) */
FQ_HD void fq_s_round64(uint32_t ah, uint32_t al, uint32_t g, uint32_t t, uint32_t& rh, uint32_t& rl)
{
    asm("{\n\t"
        ".reg .u32 z;\n\t"
        "add.cc.u32  z, %4, 0x80000000;\n\t"
        "addc.cc.u32 %0, %2, 0;\n\t"
        "addc.u32    %1, %3, %5;\n\t"
        "}"
        : "=&r"(rl), "=r"(rh)
        : "r"(al), "r"(ah), "r"(g), "r"(t));
}
/* words 3, 2, 1 of the product of (ah:al) < 2^53 and (bh:bl) */
FQ_HD void fq_s_mul53(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, uint32_t& p3, uint32_t& p2, uint32_t& p1)
{
    const uint64_t t1 = (uint64_t)ah * bl + __umulhi(al, bl); /* < 2^54 */
    const uint64_t t2 = (uint64_t)al * bh + (uint32_t)t1;
    const uint64_t t3 = (uint64_t)ah * bh + (t1 >> 32) + (t2 >> 32);
    p1 = (uint32_t)t2;
    p2 = (uint32_t)t3;
    p3 = (uint32_t)(t3 >> 32);
}
#define FQ_S_UNLIKELY(x) __builtin_expect(!!(x), 0)
#else
#if defined(FQ_S_COUNT_SLOW)
/* host checks count how often the hardware path was taken, to show the fast path is exercised */
extern long long fq_s_slow_count;
#define FQ_S_NOTE_SLOW() (++fq_s_slow_count)
#else
#define FQ_S_NOTE_SLOW() ((void)0)
#endif
static inline double fq_s_hw_add(double a, double b)
{
    FQ_S_NOTE_SLOW();
    return a + b;
}
static inline double fq_s_hw_mul(double a, double b)
{
    FQ_S_NOTE_SLOW();
    return a * b;
}
static inline uint32_t fq_s_lo(double x)
{
    return (uint32_t)fq_bits(x);
}
static inline uint32_t fq_s_hi(double x)
{
    return (uint32_t)(fq_bits(x) >> 32);
}
static inline double fq_s_make(uint32_t hi, uint32_t lo)
{
    return fq_from_bits(((uint64_t)hi << 32) | lo);
}
static inline uint32_t fq_s_shr64lo(uint32_t lo, uint32_t hi, uint32_t n)
{
    n = n > 32 ? 32 : n;
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> n);
}
static inline uint32_t fq_s_shl64hi(uint32_t lo, uint32_t hi, uint32_t n)
{
    n = n > 32 ? 32 : n;
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << n) >> 32);
}
static inline uint32_t fq_s_max(uint32_t a, uint32_t b)
{
    return a > b ? a : b;
}
static inline uint32_t fq_s_min(uint32_t a, uint32_t b)
{
    return a < b ? a : b;
}
static inline uint32_t fq_s_clz(uint32_t x)
{
    return x ? (uint32_t)__builtin_clz(x) : 32u;
}
static inline void fq_s_addsub96(uint32_t diff, uint32_t xh, uint32_t xl, uint32_t h, uint32_t l, uint32_t& g,
                                 uint32_t& mh, uint32_t& ml)
{
    const unsigned __int128 x = (unsigned __int128)(((uint64_t)xh << 32) | xl) << 32;
    const unsigned __int128 y = ((unsigned __int128)(((uint64_t)h << 32) | l) << 32) | g;
    const unsigned __int128 r = (int32_t)diff < 0 ? x - y : x + y;
    g = (uint32_t)r;
    ml = (uint32_t)(r >> 32);
    mh = (uint32_t)(r >> 64);
}
static inline void fq_s_add64c(uint32_t ah, uint32_t al, uint32_t c, uint32_t& rh, uint32_t& rl)
{
    const uint64_t r = (((uint64_t)ah << 32) | al) + (c != 0u ? 1u : 0u);
    rh = (uint32_t)(r >> 32);
    rl = (uint32_t)r;
}
static inline void fq_s_round64(uint32_t ah, uint32_t al, uint32_t g, uint32_t t, uint32_t& rh, uint32_t& rl)
{
    const uint64_t r = (((uint64_t)ah << 32) | al) + ((uint64_t)t << 32) + (g >> 31);
    rh = (uint32_t)(r >> 32);
    rl = (uint32_t)r;
}
static inline void fq_s_mul53(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, uint32_t& p3, uint32_t& p2,
                              uint32_t& p1)
{
    const uint64_t t1 = (uint64_t)ah * bl + (((uint64_t)al * bl) >> 32);
    const uint64_t t2 = (uint64_t)al * bh + (uint32_t)t1;
    const uint64_t t3 = (uint64_t)ah * bh + (t1 >> 32) + (t2 >> 32);
    p1 = (uint32_t)t2;
    p2 = (uint32_t)t3;
    p3 = (uint32_t)(t3 >> 32);
}
#define FQ_S_UNLIKELY(x) __builtin_expect(!!(x), 0)
#endif

/* What fq_s_add_words leaves over.  Sums that cancel (opposite signs, exponents at most one apart, both well
 * above the subnormals) are exact and formed here as well; the rest is the hardware's. */
#if defined(__CUDA_ARCH__)
static __device__ __noinline__ double fq_s_add_rest(double a, double b)
#else
static inline double fq_s_add_rest(double a, double b)
#endif
{
    const uint64_t x = fq_bits(a), y = fq_bits(b);
    const int ex = (int)((x >> 52) & 0x7ff), ey = (int)((y >> 52) & 0x7ff);
    const int e = ex < ey ? ex : ey;
    if (e < 56 || ex > 0x7fe || ey > 0x7fe || ex - e > 1 || ey - e > 1 || (int64_t)(x ^ y) >= 0) {
        return fq_s_hw_add(a, b);
    }
    const uint64_t one = 1ULL << 52;
    const uint64_t mx = ((x & (one - 1)) | one) << (ex - e), my = ((y & (one - 1)) | one) << (ey - e);
    const bool less = mx < my;
    uint64_t m = less ? my - mx : mx - my;
    const uint32_t hi = (uint32_t)(m >> 32);
    const int z = (int)(hi != 0u ? fq_s_clz(hi) : 32u + fq_s_clz((uint32_t)m)) - 11;
    if (m == 0 || z < 0) {
        return fq_s_hw_add(a, b);
    }
    m <<= z;
    return fq_from_bits(((less ? y : x) & (1ULL << 63)) | ((uint64_t)(e - z - 1) << 52) + m);
}

/*
 * x + y of two doubles given as words (b's sign already flipped for a subtraction); a and b are the
 * same values, for the hardware path.  Bound by the ALU pipe.
 *
 * The operands are ordered by their high words alone; y's significand is aligned into 96 bits
 * (h:l:g, g below the last place of x), added to or subtracted from x's, and normalised so that the
 * leading bit sits at bit 53 of (mh:ml) and the bit below the last place at bit 0.  No sticky bit is
 * kept: bits of y below g can change the rounding only where the bits kept below the rounding bit are
 * all zero, and that case is left to fq_s_add_rest, as are a result below 2^-20 of x (or negative, when
 * the high words were equal) and operands or results near the ends of the exponent range.  A y that is
 * zero or subnormal needs no test: whatever its significand, it is far below half a place of x.
 */
FQ_HD double fq_s_add_words(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, double a, double b)
{
    const uint32_t A = ah & 0x7fffffffu, B = bh & 0x7fffffffu;
    const bool swap = A < B;
    const uint32_t X = fq_s_max(A, B), Y = fq_s_min(A, B);
    const uint32_t xl = swap ? bl : al, yl = swap ? al : bl;
    const uint32_t sx = swap ? bh : ah; /* sign and exponent of the result before normalisation */
    const uint32_t mxh = (X & 0xfffffu) | 0x100000u, myh = (Y & 0xfffffu) | 0x100000u;
    uint32_t d = (X >> 20) - (Y >> 20);
    d = fq_s_min(d, 63u);
    const bool far = d > 31u;
    const uint32_t w2 = far ? 0u : myh, w1 = far ? myh : yl, w0 = far ? yl : 0u;
    const uint32_t n = d & 31u;
    uint32_t g = fq_s_shr64lo(w0, w1, n);
    const uint32_t l = fq_s_shr64lo(w1, w2, n), h = w2 >> n;
    uint32_t mh, ml;
    fq_s_addsub96(ah ^ bh, mxh, xl, h, l, g, mh, ml);
    /* leading bit to 53: by 0 after a carry, 1 normally, more after a cancellation */
    const uint32_t z = fq_s_clz(mh) - 10u;
    mh = fq_s_shl64hi(ml, mh, z);
    ml = fq_s_shl64hi(g, ml, z);
    g <<= (z & 31u);
    if (FQ_S_UNLIKELY(X - 0x03800000u >= 0x7fe00000u - 0x03800000u || z > 21u || (g == 0u && w0 != 0u))) {
        return fq_s_add_rest(a, b);
    }
    /* nearest even: bit 0 of ml is the rounding bit, bit 1 the last place, g what is left below */
    uint32_t qh, ql;
    fq_s_add64c(mh, ml, g | (ml & 2u), qh, ql);
    /* the implicit bit (and a carry out of the significand) adds into the exponent field */
    return fq_s_make((qh >> 1) + ((sx & 0xfff00000u) - (z << 20)), fq_s_shr64lo(ql, qh, 1));
}

FQ_HD double fq_sadd(double a, double b)
{
    return fq_s_add_words(fq_s_hi(a), fq_s_lo(a), fq_s_hi(b), fq_s_lo(b), a, b);
}

FQ_HD double fq_ssub(double a, double b)
{
    const uint32_t bh = fq_s_hi(b) ^ 0x80000000u;
    return fq_s_add_words(fq_s_hi(a), fq_s_lo(a), bh, fq_s_lo(b), a, fq_s_make(bh, fq_s_lo(b)));
}

/*
 * A factor prepared for fq_smulc: its significand with the leading bit at 63 (ch:cl), the range of
 * exponent fields of the other operand for which operand and product are normal (first one, and how
 * many, both << 21), and what is added to the other operand's sign and exponent (e).  A factor that
 * is not normal has an empty range: the hardware multiplies.
 */
typedef struct {
    uint32_t ch, cl, lo, span, e;
    double c;
} fq_sfactor;

#if defined(__CUDACC__)
__host__ __device__
#endif
static inline fq_sfactor fq_s_factor(double c)
{
    fq_sfactor f;
    const uint64_t b = fq_bits(c);
    const int ec = (int)((b >> 52) & 0x7ff);
    const uint64_t m = ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 11;
    /* product's exponent field ex + ec - 1023, one more when the significands' product reaches 2 and
     * one more when it rounds up to the next power of two */
    const int lo = 1024 - ec < 1 ? 1 : 1024 - ec, hi = 0x7fd + 1022 - ec > 0x7fe ? 0x7fe : 0x7fd + 1022 - ec;
    f.c = c;
    f.ch = (uint32_t)(m >> 32);
    f.cl = (uint32_t)m;
    f.lo = (uint32_t)lo << 21;
    f.span = ec == 0 || ec == 0x7ff || hi < lo ? 0u : (uint32_t)(hi - lo + 1) << 21;
    f.e = ((uint32_t)(ec - 1023) << 20) + (uint32_t)((b >> 63) << 31);
    return f;
}

/*
 * x * f: the 53 x 64-bit product of the significands as 32-bit multiply-adds (without the low word of
 * its lowest partial product), its top 53 bits in (p3:p2) and the bits below in p1.  A p1 of exactly
 * half a place goes to the hardware (a tie, or bits below that were not formed).
 */
FQ_HD double fq_smulc(double x, const fq_sfactor f)
{
    const uint32_t xh = fq_s_hi(x), xl = fq_s_lo(x);
    uint32_t p3, p2, p1;
    fq_s_mul53((xh & 0xfffffu) | 0x100000u, xl, f.ch, f.cl, p3, p2, p1);
    uint32_t t = (xh & 0xfff00000u) + f.e;
    if (!(p3 & 0x100000u)) {
        p3 = fq_s_shl64hi(p2, p3, 1);
        p2 = fq_s_shl64hi(p1, p2, 1);
        p1 <<= 1;
        t -= 0x100000u;
    }
    if (FQ_S_UNLIKELY((xh << 1) - f.lo >= f.span || p1 == 0x80000000u)) {
        return fq_s_hw_mul(x, f.c);
    }
    uint32_t rh, rl;
    fq_s_round64(p3, p2, p1, t, rh, rl);
    return fq_s_make(rh, rl);
}

FQ_HD double fq_smul(double a, double b)
{
    const uint32_t ah = fq_s_hi(a), al = fq_s_lo(a), bh = fq_s_hi(b), bl = fq_s_lo(b);
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    uint32_t p3, p2, p1;
    /* b's significand with its leading bit at 63 */
    fq_s_mul53((ah & 0xfffffu) | 0x100000u, al, fq_s_shl64hi(bl, bh & 0xfffffu, 11) | 0x80000000u, bl << 11, p3, p2,
               p1);
    uint32_t e = ea + eb - 1023u;
    if (!(p3 & 0x100000u)) {
        p3 = fq_s_shl64hi(p2, p3, 1);
        p2 = fq_s_shl64hi(p1, p2, 1);
        p1 <<= 1;
        e -= 1u;
    }
    if (FQ_S_UNLIKELY(ea - 1u >= 0x7feu || eb - 1u >= 0x7feu || e >= 0x7fdu || p1 == 0x80000000u)) {
        return fq_s_hw_mul(a, b);
    }
    uint32_t rh, rl;
    fq_s_round64(p3, p2, p1, ((ah ^ bh) & 0x80000000u) + (e << 20), rh, rl);
    return fq_s_make(rh, rl);
}

#endif
