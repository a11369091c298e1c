// ov_fxlaw.cuh - the segment law of an accepted cell on 64-bit integer
// mantissas, for the FP64 path.
//
// GB300 runs FP64 at 1/64 of its FP32 rate: one warp instruction holds an
// SM's FP64 pipe for 16 cycles, while 32x32+64-bit integer multiply-adds run
// at half the FP32 rate and integer adds at the full rate (measured: 58, 116
// and 1.8 lanes a cycle and SM for IMAD.WIDE, IADD and DFMA).  The law
// (octree.c:321-342)
//     w = (R x S) (|R| + |R+S|) / (|R||R+S| (|R||R+S| + R.(R+S)))
// therefore runs on fixed-point coordinates (FxFrame: counted from the box, every
// separation below 2^61 units u, so offsets of FP64 magnitude down to 2^-9 of
// the largest convert exactly), left-normalised per interaction, with 2 to 9
// IMAD.WIDE per product.  Each of the two square roots and the quotient
// starts from the FP32 hardware approximation and takes two exact integer
// residuals (24 -> 46 -> 60 bits).  Every step keeps at least 55 bits (the law
// against long double: 2.5e-17 of |R||S| w / |R x S| beyond the last digit of the
// sums, whatever the seeds' errors), so a term is closer to the real-number value than the FP64 law's, whose R x Rp1
// cancels by |R| / |S|; the terms add up exactly, in 96 bits.
//
// What this cannot decide or would lose bits on is left to the FP64 law:
// interactions nearer than 2^47 units (a 2,000th to a 5,500th of a cubic box's side,
// wherever the box lies; 2^51 where coordinates had to be rounded), ends at
// distances that differ fourfold, or seen almost 90 degrees or more apart (where the reference's
// ndot filter drops them).
//
// Host and device: the arithmetic is integer apart from the FP32 seeds, whose
// last bits do not show in the result.
#ifndef OV_FXLAW_CUH
#define OV_FXLAW_CUH

#include <math.h>
#include <stdint.h>
#include <string.h>

// FP64 cell view of the integer law (64 bytes).  c: centre of mass in units
// u; s: circulation in units u, shifted left by e so that its largest
// component is in [2^60, 2^61), as sh 2^32 + sl; n: |s|^2 / 2^64.
// e = kFxNone: not representable (FP64 law); e = kFxZero: zero circulation
// (no velocity).  shift: separations below 2^(60 - shift) units are left to the
// FP64 law.
struct alignas(16) CellFX {
    int64_t c[3];
    int sh[3], sl[3];
    int64_t n;
    int e, shift;
};
constexpr int kFxNone = -1, kFxZero = -2;
// Largest shift: kFxMaxShift keeps a coordinate's rounding to a unit below 2^-52 of
// the separation; where both sides are whole numbers of units without rounding
// (most of a box: all but its 512th next to the planes from which it is counted) the
// separation is exact, and kFxWholeShift is where terms pass 2^58 units of the sums;
// kFxRoundShift does for coordinates that lose bits when they are counted from
// the box's corner (2^7 units at most: points far outside the box toward 0)
// (65,536 nodes in a 200th of their open box: traversal 10.9 ms with 9 throughout, late
// cells evaluated one by one where their list was full; 6.8 with 9 and the list flushed,
// 4.8 with 13).
constexpr int kFxMaxShift = 9, kFxWholeShift = 13, kFxRoundShift = 2;
// Terms add up in units 2^kFxUnit / u.  A term's error is about 2^-8 units (the
// aligned quotient's last bit), and terms with a quotient above 2^63 units, the
// nearest, are left to the FP64 law: the unit of a tree's sums (2,000 terms)
// sends it a handful, that of direct sums (10^6 terms) a few hundred.
constexpr int kFxUnit = -105, kFxUnitDirect = -110;
constexpr int kFxTerms = 31;       // terms a sum holds: each is at most 2^58 units
constexpr double kFxLimit = 2305843009213693952.0;   // 2^61: coordinates are below

// Fixed-point coordinates: x in units u is x inv + at, u = 1 / inv.
struct FxFrame {
    double inv, u, at[3];
    int e;       // inv = 2^e
    int whole;   // largest shift of whole coordinates
};
static inline FxFrame fx_unit(int e)   // unit 2^e, counted from 0
{
    // Not below 2^-75, and the shift so that what the law takes is at least 2^-24 =
    // 6e-8 away at one end and a quarter of that at the other, where the reference's
    // filters (|R|, |R+S| < 1e-8) drop nothing: closer cells, of boxes smaller than
    // 3e-4, are left to the FP64 law, which has the filters.
    if (e < -75) e = -75;
    const int s = 60 + 24 + e;
    return FxFrame{ldexp(1.0, -e), ldexp(1.0, e), {0, 0, 0}, -e, s < kFxWholeShift ? s : kFxWholeShift};
}

// The frame of a box: counted from 0 where the box is within its length of it,
// else from the corner nearest to 0 rounded to 2^-22 of the box (coordinates of the
// box then lose nothing), so that the unit depends on the box's lengths; it leaves
// a period on either side (image query points, stage positions) below 2^61 units.
// (A unit taken from the largest coordinate leaves most interactions of a box far
// from 0 to the FP64 law: 65,536 nodes in a box of side 0.1, traversal 3.6 ms at 0,
// 9.6 at 10 and 17.2 at 50; 3.7 wherever it lies so.)
static inline FxFrame fx_frame(const double lo[3], const double hi[3])
{
    FxFrame f;
    double o[3], L = 0, m = 0;
    for (int a = 0; a < 3; ++a) L = fmax(L, fabs(hi[a] - lo[a]));
    const double step = ldexp(1.0, (int)ceil(log2(L > 0 ? L : 1.0)) - 22);
    for (int a = 0; a < 3; ++a) {
        o[a] = lo[a] > L ? floor(lo[a] / step) * step : (hi[a] < -L ? ceil(hi[a] / step) * step : 0.0);
        m = fmax(m, fmax(fabs(lo[a] - o[a]), fabs(hi[a] - o[a])) + 2 * fabs(hi[a] - lo[a]));
    }
    f = fx_unit((int)ceil(log2(m > 0 ? m : 1.0)) - 61);
    for (int a = 0; a < 3; ++a) f.at[a] = -o[a] * f.inv;
    return f;
}

#if defined(__CUDA_ARCH__)
#define FX_INLINE __device__ __forceinline__
FX_INLINE int fx_clz(unsigned x) { return __clz((int)x); }
FX_INLINE float fx_rsqrt(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
FX_INLINE float fx_rcp(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
FX_INLINE int fx_int(float x) { return __float2int_rn(x); }
// x >> n for any n >= 0 (the PTX shift clamps)
FX_INLINE int64_t fx_shr(int64_t x, int n) { int64_t y; asm("shr.s64 %0, %1, %2;" : "=l"(y) : "l"(x), "r"(n)); return y; }
// c + a b as one IMAD.WIDE (written out: the compiler keeps the sum apart)
FX_INLINE int64_t fx_mad(int a, int b, int64_t c)
{
    int64_t d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
FX_INLINE uint64_t fx_madu(unsigned a, unsigned b, uint64_t c)
{
    uint64_t d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
#else
#define FX_INLINE static inline
FX_INLINE int fx_clz(unsigned x) { return x ? __builtin_clz(x) : 32; }
FX_INLINE float fx_rsqrt(float x) { return 1.0f / sqrtf(x); }
FX_INLINE float fx_rcp(float x) { return 1.0f / x; }
FX_INLINE int fx_int(float x) { return (int)rintf(x); }
FX_INLINE int64_t fx_shr(int64_t x, int n) { return x >> (n < 63 ? n : 63); }
FX_INLINE int64_t fx_mad(int a, int b, int64_t c) { return c + (int64_t)a * b; }
FX_INLINE uint64_t fx_madu(unsigned a, unsigned b, uint64_t c) { return c + (uint64_t)a * b; }
#endif

FX_INLINE uint64_t fx_bits(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}

// x is a whole number: no bits of its fraction below 1
FX_INLINE bool fx_whole(double x)
{
    const uint64_t b = fx_bits(x);
#if defined(__CUDA_ARCH__)
    const int low = __ffsll((long long)(b | (1ull << 52))) - 1;
#else
    const int low = __builtin_ctzll(b | (1ull << 52));
#endif
    return (int)((b >> 52) & 0x7ff) - 1023 + low >= 52 || b << 1 == 0;
}

// Largest shift that a coordinate r = x inv + at allows, -1: 2^61 or more, or no
// number.  r is a multiple of x's last bit, so it was rounded only if it is of a
// larger magnitude than x inv.
FX_INLINE int fx_shift(double r, double x, const FxFrame &f)
{
    const int er = (int)((fx_bits(r) >> 52) & 0x7ff), ex = (int)((fx_bits(x) >> 52) & 0x7ff);
    if (er >= 1023 + 61) return -1;
    if (er != 0 && er - ex > f.e) return kFxRoundShift;
    return fx_whole(r) ? f.whole : kFxMaxShift;
}

FX_INLINE int fx_hi(int64_t x) { return (int)(x >> 32); }
FX_INLINE int64_t fx_mul(int a, int b) { return (int64_t)a * b; }

// x = h 2^32 + l with l signed
struct fx_split {
    int h, l;
};
FX_INLINE fx_split fx_parts(int64_t x)
{
    const unsigned lo = (unsigned)x;
    return fx_split{(int)((unsigned)fx_hi(x) + (lo >> 31)), (int)lo};
}

// A sum of terms: h + l / 2^32 units.
struct fx_sum {
    int64_t h;
    unsigned l;
};
FX_INLINE double fx_value(const fx_sum &s) { return (double)s.h + (double)s.l * 2.3283064365386963e-10; }

// s += h + l / 2^32
FX_INLINE void fx_add(fx_sum &s, int64_t h, unsigned l)
{
#if defined(__CUDA_ARCH__)
    unsigned a = (unsigned)s.h, b = (unsigned)(s.h >> 32);
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(s.l), "+r"(a), "+r"(b) : "r"(l), "r"((unsigned)h), "r"((unsigned)(h >> 32)));
    s.h = (int64_t)(((uint64_t)b << 32) | a);
#else
    const uint64_t t = (uint64_t)s.l + l;
    s.l = (unsigned)t;
    s.h += h + (int64_t)(t >> 32);
#endif
}

// sqrt(a) 2^32 for 2^50 <= a < 2^62, to a few units whatever the seed's last bits
FX_INLINE int64_t fx_sqrt(int64_t a)
{
    const float f = fmaf((float)(unsigned)fx_hi(a), 4294967296.0f, (float)(unsigned)a);
    const float y = fx_rsqrt(f);
    const int m = fx_int(f * y);
    // a = (m + w / 2^16 + v / 2^32)^2: w from an exact residual, v from what that leaves
    // less w^2, whose FP32 value does.  (A factor m + w / 2^17 rounded to 32 bits costs
    // the second residual w / 2, 2^-49 of the root at the lower end; w^2 in integers
    // 0.5 to 1 % of an evaluation.)
    const int64_t r = fx_mad(-m, m, a);
    const float wf = (float)(int)(r >> 10) * (y * 33554432.0f);
    const int w = fx_int(wf);
    const int64_t r2 = fx_mad(-w, m, r << 15);
    const int v = fx_int(fmaf(wf * -4.76837158203125e-7f, wf, (float)(int)(r2 >> 4)) * (y * 1048576.0f));
    return fx_mad(w, 65536, v) + ((int64_t)m << 32);
}

// hi 64 bits of a b for 0 <= a, b < 2^63 (less the carry of the low parts)
FX_INLINE int64_t fx_mulhi(int64_t a, int64_t b)
{
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
    const uint64_t mid = fx_madu(al, bh, (uint64_t)ah * bl);
    return (int64_t)fx_madu(ah, bh, mid >> 32);
}

// The view of a cell or segment from its coordinates in units u; fits: they
// are below 2^61.
FX_INLINE CellFX fx_cell(const int64_t c[3], const int64_t s[3], bool fits, int shift = kFxMaxShift)
{
    CellFX o;
    uint64_t m = 0;
    for (int i = 0; i < 3; ++i) m |= (uint64_t)(s[i] < 0 ? -s[i] : s[i]);
    const int hi = fx_clz((unsigned)(m >> 32)), lo = fx_clz((unsigned)m);
    o.e = !fits ? kFxNone : (m ? (m >> 32 ? hi : 32 + lo) - 3 : kFxZero);
    o.n = 0;
    int64_t low = 0;
    for (int i = 0; i < 3; ++i) {
        o.c[i] = c[i];
        const fx_split p = fx_parts(o.e > 0 ? (int64_t)((uint64_t)s[i] << o.e) : s[i]);
        o.sh[i] = p.h;
        o.sl[i] = p.l;
        o.n = fx_mad(p.h, p.h, o.n);
        low = fx_mad(p.h, p.l, low);
    }
    o.n += low >> 31;
    o.shift = shift;
    return o;
}

// Adds the law's term for cell c seen from q (units u) to sum where `take` is
// set and the law can decide; returns that (no branches: what is left to the
// FP64 law is rare).  shift: the largest that q allows.  mag, when given, gains a bound on the term's
// magnitude (over the components, in the sum's units, to FP32 precision).
template <int Unit = kFxUnit>
FX_INLINE bool fx_law(const CellFX &c, const int64_t q[3], bool take, fx_sum sum[3], int shift = kFxMaxShift,
                      float *mag = nullptr)
{
    int64_t R[3];
    unsigned top = 0;
    for (int i = 0; i < 3; ++i) {
        R[i] = c.c[i] - q[i];
        const int h = fx_hi(R[i]);
        top |= (unsigned)(h ^ (h >> 31));
    }
    const int sr = fx_clz(top) - 3;
    bool ok = take && (unsigned)sr <= (unsigned)(shift < c.shift ? shift : c.shift) && c.e >= 0;
    const int s = (sr < c.e ? sr : c.e) & 63, ds = (c.e - s) & 63;
    // a = |R|^2, m = R.S, both / 2^64
    fx_split r[3];
    int64_t a = 0, ax = 0, m = 0, mx = 0;
    for (int i = 0; i < 3; ++i) {
        r[i] = fx_parts((int64_t)((uint64_t)R[i] << s));
        a = fx_mad(r[i].h, r[i].h, a);
        ax = fx_mad(r[i].h, r[i].l, ax);
        m = fx_mad(r[i].h, c.sh[i], m);
        mx = fx_mad(r[i].h, c.sl[i], mx);
        mx = fx_mad(r[i].l, c.sh[i], mx);
    }
    a += ax >> 31;
    m = (m + fx_hi(mx)) >> ds;
    const int64_t dot = a + m;                                     // R.(R+S)
    const int64_t b = dot + m + fx_shr(c.n, 2 * ds);               // |R+S|^2
    const int at = fx_hi(a), bt = fx_hi(b);
    ok = ok && (at >> 4) <= bt && (bt >> 4) <= at && fx_hi(dot) > (at + bt) >> 10;
    const int64_t A = fx_sqrt(a), B = fx_sqrt(b);
    const int64_t g = fx_mulhi(A, B), h = g + dot;
    const uint64_t len = (uint64_t)A + (uint64_t)B;
    const int lg = (fx_clz((unsigned)fx_hi(g)) - 1) & 63, lh = lg - 1;   // g <= h <= 2 g
    const int ls = fx_clz((unsigned)(len >> 32));
    const uint64_t num = len << ls;                                                                  // [2^63, 2^64)
    const int64_t D = fx_mulhi((int64_t)((uint64_t)g << lg), (int64_t)((uint64_t)h << (lh & 63)));   // [2^59, 2^62)
    // Q = num 2^58 / D: the first 24 bits, then two residuals
    const fx_split d = fx_parts(D);
    const float y = fx_rcp((float)d.h);
    const int q0 = fx_int((float)(unsigned)(num >> 32) * (y * 67108864.0f));
    const int64_t e1 = fx_mad(-q0, d.h, (int64_t)(num >> 6)) + fx_hi(fx_mul(-q0, d.l));
    const int q1 = fx_int((float)(int)(e1 >> 6) * (y * 4194304.0f));
    const int64_t e2 = fx_mad(-q1, d.h, e1 << 16) + fx_hi(fx_mul(-q1, d.l));
    const int q2 = fx_int((float)(int)(e2 >> 4) * (y * 1048576.0f));
    const int64_t Q = fx_mad(q1, 65536, q2) + ((int64_t)q0 << 32);
    // the term is (R x S) / 2^64 Q / 2^64 2^ex, ex = lg + lh - ls + 2 s - e - 122
    const int down = Unit + 122 + ls + c.e - lg - lh - 2 * s;
    ok = ok && down >= 0;
    const fx_split k = fx_parts(ok ? fx_shr(Q, down) : 0);
    // (p.h + 1) 2^32 |k| / 2^64 bounds a component's term
    const float size = mag ? fmaf((float)k.h, 1.0f, (float)k.l * 2.3283064e-10f) : 0.0f;
    for (int i = 0; i < 3; ++i) {
        const int u = i == 2 ? 0 : i + 1, v = i == 0 ? 2 : i - 1;
        int64_t x = fx_mul(r[u].h, c.sl[v]);
        x = fx_mad(r[u].l, c.sh[v], x);
        x = fx_mad(-r[v].h, c.sl[u], x);
        x = fx_mad(r[v].l, -c.sh[u], x);   // (-r.l overflows for r.l = -2^31)
        x = fx_mad(r[u].h, c.sh[v], fx_hi(x));
        x = fx_mad(-r[v].h, c.sh[u], x);
        const fx_split p = fx_parts(x);
        int64_t low = fx_mad(p.h, k.l, fx_hi(fx_mul(p.l, k.l)));
        low = fx_mad(p.l, k.h, low);
        if (mag) *mag = fmaf(fabsf((float)p.h) + 1.0f, size, *mag);
        fx_add(sum[i], fx_mad(p.h, k.h, fx_hi(low)), (unsigned)low);
    }
    return ok;
}

#endif
