// se2p_fft_ff.cu -- batched 1D complex FFTs of contiguous rows in
// float-float arithmetic (the FP64 form's k-space transforms).
//
// cuFFT's double-precision C2C of the grid lengths the spectral Ewald method
// uses (2688 = 2^7 3 7 at tolerance 1e-10 and a million points) runs on the
// FP64 pipe, which GB300 provides at 1/73 of its FP32 rate: the four 1D
// passes of one evaluation took 7 ms, more than any other stage.  Here each
// row is transformed in shared memory with float-float arithmetic (about 48
// significant bits) on the FP32 pipe.  The FFT's rounding errors are spread
// over all modes, and the k-space sums average them: errors of 2^-46 relative
// to the spectra's mean magnitude, injected into the oracle's transforms,
// change its SLP and DLP k-space results by 1e-15 to 7e-15, far inside the
// 1e-12 parity bound (the systematic errors of float-float Gaussian weights
// do not average out, which is why the spread and gather stay exact).
//
// One CTA per row: the row is read once as doubles (staged in shared memory
// for the exponent scan), scaled by a power of two that
// puts its largest entry near 2^64 (exact; the FFT of a row of L <= 2^13
// values grows it by at most L), split into float-float pairs with integer
// operations, transformed by mixed-radix Stockham stages (radices 12, 8, 7,
// 6, 5, 4, 3, 2, ping-pong between two shared buffers), and written back as doubles
// rebuilt with integer operations (float <-> double conversions run at the
// FP64 rate on GB300).  Twiddles exp(-2 pi i m / L) come from a per-length
// table built in long double on the host; the odd radices take their
// constants cos, sin(2 pi m / R) from the same table (entry m L / R).
//
// The transform is unnormalised with cuFFT's sign convention (forward
// exp(-2 pi i j k / L)), so it replaces cufftExecZ2Z on the same layout.
#include "se2p_internal.cuh"
#include <algorithm>
#include <climits>
#include <math_constants.h>

namespace se2p {

namespace {

// Two FP32 numbers in one register pair: an instruction on pairs takes the FP32
// pipe two cycles (65 per clock and SM measured, against 127 scalar ones) but one
// issue slot, and the kernel is bound by issue.  A complex number is a pair (re,
// im) of heads and one of tails, so its sums, products with a real, and shared
// memory accesses are half as many instructions.
typedef unsigned long long f2;

__device__ __forceinline__ f2 pk(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 upk(f2 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f2 swap2(f2 a)
{
    const float2 v = upk(a);
    return pk(v.y, v.x);
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
constexpr f2 kM1 = 0xbf800000bf800000ull;            // (-1, -1)
// a - b, rounded once (the product with -1 is exact)
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, kM1, a); }
__device__ __forceinline__ f2 neg2(f2 a) { return mul2(a, kM1); }

// TwoSum, Fast2Sum and TwoProduct of both numbers (se2p_ff.cuh has the scalar ones).
__device__ __forceinline__ void two_sum2(f2 a, f2 b, f2 &s, f2 &e)
{
    s = add2(a, b);
    const f2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ void two_diff2(f2 a, f2 b, f2 &s, f2 &e)
{
    s = sub2(a, b);
    const f2 bb = sub2(s, a);
    e = sub2(sub2(a, sub2(s, bb)), add2(b, bb));
}
__device__ __forceinline__ void fast_two_sum2(f2 a, f2 b, f2 &s, f2 &e)
{
    s = add2(a, b);
    e = sub2(b, sub2(s, a));
}

struct fc {
    f2 h, l;       // (re, im) heads and tails
};

__device__ __forceinline__ fc fc_add(const fc &a, const fc &b)
{
    f2 s, e;
    two_sum2(a.h, b.h, s, e);
    e = add2(e, add2(a.l, b.l));
    fc r;
    fast_two_sum2(s, e, r.h, r.l);
    return r;
}
__device__ __forceinline__ fc fc_sub(const fc &a, const fc &b)
{
    f2 s, e;
    two_diff2(a.h, b.h, s, e);
    e = add2(e, sub2(a.l, b.l));
    fc r;
    fast_two_sum2(s, e, r.h, r.l);
    return r;
}
// a * (s i), s = +-1: (-s im, s re); sg = (-s, s)
__device__ __forceinline__ fc fc_mul_si(const fc &a, f2 sg) { return {mul2(swap2(a.h), sg), mul2(swap2(a.l), sg)}; }
// a times the real c, cl (in both halves)
__device__ __forceinline__ fc fc_mulr(const fc &a, f2 c, f2 cl)
{
    const f2 p = mul2(a.h, c);
    f2 e = fma2(a.h, c, neg2(p));
    e = fma2(a.h, cl, e);
    e = fma2(a.l, c, e);
    fc r;
    fast_two_sum2(p, e, r.h, r.l);
    return r;
}

// A twiddle (c, sn) = exp(+-2 pi i m / L) as the product takes it: c and its
// tail in both halves, (-sn, sn) and its tails.
struct tw2 {
    f2 c, cl, s, sl;
};

// a * w: a c + (im, re)(-sn, sn), the two products' heads summed by TwoSum.
__device__ __forceinline__ fc fc_mul(const fc &a, const tw2 &w)
{
    const f2 p1 = mul2(a.h, w.c);
    f2 e1 = fma2(a.h, w.c, neg2(p1));
    e1 = fma2(a.h, w.cl, e1);
    e1 = fma2(a.l, w.c, e1);
    const f2 bh = swap2(a.h), bl = swap2(a.l);
    const f2 p2 = mul2(bh, w.s);
    f2 e2 = fma2(bh, w.s, neg2(p2));
    e2 = fma2(bh, w.sl, e2);
    e2 = fma2(bl, w.s, e2);
    f2 s, t;
    two_sum2(p1, p2, s, t);
    t = add2(t, add2(e1, e2));
    fc r;
    fast_two_sum2(s, t, r.h, r.l);
    return r;
}

// Entry m of the table: two 16-byte words (c, c, cl, cl), (-sn, sn, -snl, snl).
__device__ __forceinline__ tw2 tw_load(const ulonglong2 *tw, int m)
{
    const ulonglong2 a = __ldg(tw + 2 * m), b = __ldg(tw + 2 * m + 1);
    return {a.x, a.y, b.x, b.y};
}

// Shared buffer: heads, then tails, of Lp = sh_len(L) pairs each, element k at k +
// k/16: the padding pair per 16 keeps the stride-R stores of the early stages
// (R = 2, 4, 8) free of bank conflicts.
__host__ __device__ __forceinline__ int sh_len(int L) { return L + (L >> 4) + 1; }
__device__ __forceinline__ fc sh_get(const f2 *b, int Lp, int k)
{
    k += k >> 4;
    return {b[k], b[Lp + k]};
}
__device__ __forceinline__ void sh_put(f2 *b, int Lp, int k, const fc &v)
{
    k += k >> 4;
    b[k] = v.h;
    b[Lp + k] = v.l;
}
__device__ __forceinline__ fc fc_make(float2 re, float2 im) { return {pk(re.x, im.x), pk(re.y, im.y)}; }

// Radix-R butterflies of one Stockham stage.  Input element r of butterfly j
// is A[j + r L/R]; it is multiplied by w^(k r L/(Ns R)), k = j mod Ns, the
// R-point DFT is taken, and output r goes to B[(j / Ns) Ns R + k + r Ns].
template <int R>
__device__ __forceinline__ void dft(fc *v, f2 sg, const tw2 *cst);

template <>
__device__ __forceinline__ void dft<2>(fc *v, f2, const tw2 *)
{
    const fc a = v[0], b = v[1];
    v[0] = fc_add(a, b);
    v[1] = fc_sub(a, b);
}

template <>
__device__ __forceinline__ void dft<4>(fc *v, f2 sg, const tw2 *)
{
    const fc t0 = fc_add(v[0], v[2]), t1 = fc_sub(v[0], v[2]);
    const fc t2 = fc_add(v[1], v[3]), t3 = fc_mul_si(fc_sub(v[1], v[3]), sg);   // W4 = s i
    v[0] = fc_add(t0, t2);
    v[2] = fc_sub(t0, t2);
    v[1] = fc_add(t1, t3);
    v[3] = fc_sub(t1, t3);
}

// cst[0].c = sqrt(1/2)
template <>
__device__ __forceinline__ void dft<8>(fc *v, f2 sg, const tw2 *cst)
{
    fc e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<4>(e, sg, nullptr);
    dft<4>(o, sg, nullptr);
    // W8 = (1 + s i) sqrt(1/2), W8^2 = s i, W8^3 = (-1 + s i) sqrt(1/2)
    const fc o1 = fc_mulr(fc_add(o[1], fc_mul_si(o[1], sg)), cst[0].c, cst[0].cl);
    const fc o2 = fc_mul_si(o[2], sg);
    const fc o3 = fc_mulr(fc_sub(fc_mul_si(o[3], sg), o[3]), cst[0].c, cst[0].cl);
    v[0] = fc_add(e[0], o[0]);
    v[4] = fc_sub(e[0], o[0]);
    v[1] = fc_add(e[1], o1);
    v[5] = fc_sub(e[1], o1);
    v[2] = fc_add(e[2], o2);
    v[6] = fc_sub(e[2], o2);
    v[3] = fc_add(e[3], o3);
    v[7] = fc_sub(e[3], o3);
}

// Float-float dot-product accumulator: the heads are summed by TwoSum, and
// each product's FMA-formed error, its cross terms and the TwoSum errors go
// into an unnormalised tail; one normalisation at the end.  A term costs 12
// FP32 operations against 18 for a product and an add normalised separately.
struct ffacc {
    f2 s, t;
};
__device__ __forceinline__ ffacc acc_prod(f2 c, f2 cl, const fc &x)
{
    const f2 p = mul2(c, x.h);
    f2 e = fma2(c, x.h, neg2(p));
    e = fma2(c, x.l, e);
    e = fma2(cl, x.h, e);
    return {p, e};
}
__device__ __forceinline__ void acc_add(ffacc &a, f2 h, f2 l)
{
    f2 s, q;
    two_sum2(a.s, h, s, q);
    a.s = s;
    a.t = add2(a.t, add2(q, l));
}
__device__ __forceinline__ fc acc_get(const ffacc &a)
{
    fc r;
    two_sum2(a.s, a.t, r.h, r.l);
    return r;
}

// Odd R: with s_n = a_n + a_(R-n), d_n = a_n - a_(R-n),
// A_k = a_0 + sum_n cos(2 pi n k / R) s_n, B_k = sum_n sin(2 pi n k / R) d_n,
// X_k = A_k + s i B_k, X_(R-k) = A_k - s i B_k.  cst[m] = (cos, sin)(2 pi m / R),
// m = 1 .. (R-1)/2, each in both halves of .c and .s.  The sums X_0, A_k and B_k
// are float-float dot products (ffacc).
template <int R>
__device__ __forceinline__ void dft_odd(fc *v, f2 sg, const tw2 *cst)
{
    constexpr int h = (R - 1) / 2;
    fc sm[h], df[h];
#pragma unroll
    for (int n = 1; n <= h; n++) {
        sm[n - 1] = fc_add(v[n], v[R - n]);
        df[n - 1] = fc_sub(v[n], v[R - n]);
    }
    const fc a0 = v[0];
    ffacc x0 = {a0.h, a0.l};
#pragma unroll
    for (int n = 0; n < h; n++) acc_add(x0, sm[n].h, sm[n].l);
#pragma unroll
    for (int k = 1; k <= h; k++) {
        ffacc A = {a0.h, a0.l}, B = {0, 0};
#pragma unroll
        for (int n = 1; n <= h; n++) {
            int m = (n * k) % R;
            const bool neg = m > h;                  // sin(2 pi (R-m)/R) = -sin(2 pi m/R)
            if (neg) m = R - m;
            const tw2 &w = cst[m - 1];
            const ffacc pa = acc_prod(w.c, w.cl, sm[n - 1]);
            acc_add(A, pa.s, pa.t);
            ffacc pb = acc_prod(w.s, w.sl, df[n - 1]);
            if (neg) pb = {neg2(pb.s), neg2(pb.t)};
            if (n == 1) B = pb;
            else acc_add(B, pb.s, pb.t);
        }
        const fc a = acc_get(A), b = fc_mul_si(acc_get(B), sg);
        v[k] = fc_add(a, b);
        v[R - k] = fc_sub(a, b);
    }
    v[0] = acc_get(x0);
}

template <>
__device__ __forceinline__ void dft<3>(fc *v, f2 sg, const tw2 *cst) { dft_odd<3>(v, sg, cst); }
template <>
__device__ __forceinline__ void dft<5>(fc *v, f2 sg, const tw2 *cst) { dft_odd<5>(v, sg, cst); }
template <>
__device__ __forceinline__ void dft<7>(fc *v, f2 sg, const tw2 *cst) { dft_odd<7>(v, sg, cst); }

// R = 6 = 2 x 3 by the prime-factor (Good-Thomas) split, with no inner
// twiddles: 3-point DFTs of inputs (0, 2, 4) and (3, 5, 1), then 2-point
// DFTs of their outputs, which land at (3 k1 + 4 k2) mod 6.  cst as for R = 3.
template <>
__device__ __forceinline__ void dft<6>(fc *v, f2 sg, const tw2 *cst)
{
    fc a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
    dft_odd<3>(a, sg, cst);
    dft_odd<3>(b, sg, cst);
    v[0] = fc_add(a[0], b[0]);
    v[3] = fc_sub(a[0], b[0]);
    v[4] = fc_add(a[1], b[1]);
    v[1] = fc_sub(a[1], b[1]);
    v[2] = fc_add(a[2], b[2]);
    v[5] = fc_sub(a[2], b[2]);
}

// R = 12 = 4 x 3: inputs (3 n1 + 4 n2) mod 12, outputs (9 k1 + 4 k2) mod 12.
template <>
__device__ __forceinline__ void dft<12>(fc *v, f2 sg, const tw2 *cst)
{
    fc t[4][3];
#pragma unroll
    for (int n = 0; n < 4; n++) {
#pragma unroll
        for (int m = 0; m < 3; m++) t[n][m] = v[(3 * n + 4 * m) % 12];
        dft_odd<3>(t[n], sg, cst);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) {
        fc u[4] = {t[0][m], t[1][m], t[2][m], t[3][m]};
        dft<4>(u, sg, nullptr);
#pragma unroll
        for (int n = 0; n < 4; n++) v[(9 * n + 4 * m) % 12] = u[n];
    }
}

// tw: the table of the transform's sign; tw0: the forward one, whose entries m L / R
// give the butterflies' constants.
template <int R>
__device__ void stage(const f2 *A, f2 *B, int L, int Ns, unsigned magic, f2 sg,
                      const ulonglong2 *tw, const ulonglong2 *tw0)
{
    // the constants of the R-point DFT from the twiddle table
    constexpr f2 kPM = 0xbf8000003f800000ull;        // (1, -1)
    constexpr int O = R % 3 == 0 ? 3 : R;
    constexpr int NC = O & 1 ? O / 2 : 1;
    tw2 cst[NC];
    if (R == 8) {
        cst[0] = tw_load(tw0, L / 8);                // exp(-i pi/4): re = sqrt(1/2)
    } else if (O & 1) {
#pragma unroll
        for (int m = 1; m <= O / 2; m++) {
            const tw2 w = tw_load(tw0, m * (L / O));   // sn = -sin: (-sn, sn) = (sin, -sin)
            cst[m - 1] = {w.c, w.cl, mul2(w.s, kPM), mul2(w.sl, kPM)};
        }
    }
    const int nb = L / R, stride = L / (Ns * R), Lp = sh_len(L);
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        const int k = Ns == 1 ? 0 : j - (int)__umulhi((unsigned)j, magic) * Ns;   // j mod Ns
        fc v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = sh_get(A, Lp, j + r * nb);
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; r++) v[r] = fc_mul(v[r], tw_load(tw, k * r * stride));
        }
        dft<R>(v, sg, cst);
        const int o = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) sh_put(B, Lp, o + r * Ns, v[r]);
    }
}

// exact: hi + lo rebuilt as a double with integer operations (truncated to
// 53 bits), times 2^e.  hi, lo normalised float-float (|lo| <= ulp(hi)/2),
// finite, and the result in the normal range.
__device__ __forceinline__ double ff_to_double_scaled(float hi, float lo, int e)
{
    const unsigned hb = __float_as_uint(hi), lb = __float_as_uint(lo);
    const int eh = (int)((hb >> 23) & 0xff);
    if (eh == 0) return 0.0;
    if (eh == 0xff)                                  // inf, NaN (no conversion: it would be hoisted)
        return __longlong_as_double((long long)((unsigned long long)(hb >> 31) << 63 | 0x7ffull << 52 |
                                                (unsigned long long)(hb & 0x7fffffu) << 29));
    long long m = (long long)((hb & 0x7fffffu) | 0x800000u) << 29;   // units 2^(eh-179)
    const int el = (int)((lb >> 23) & 0xff);
    if (el != 0) {
        const long long ml = (long long)((lb & 0x7fffffu) | 0x800000u);
        const int sh = el - eh + 29;
        long long d = sh >= 0 ? (ml << sh) : (sh > -40 ? (ml >> (-sh)) : 0);
        m += ((lb ^ hb) >> 31) ? -d : d;
    }
    int be = eh + 896 + e;                           // biased double exponent of 2^52 m ... units
    if (m >= (1ll << 53)) {
        m >>= 1;
        be++;
    } else if (m < (1ll << 52)) {
        m <<= 1;
        be--;
    }
    if (be <= 0) return 0.0;
    if (be >= 0x7ff) return hi > 0.f ? CUDART_INF : -CUDART_INF;
    const unsigned long long bits = ((unsigned long long)(hb >> 31) << 63) |
                                    ((unsigned long long)be << 52) |
                                    ((unsigned long long)m & ((1ull << 52) - 1));
    return __longlong_as_double((long long)bits);
}

// a > 0 rounded to 24 bits (to nearest, ties up): the float's bit pattern,
// and in *rem the remainder a - rounded (|rem| <= 2^(bits-25)).  a < 2^62.
__device__ __forceinline__ unsigned u64_round_float(unsigned long long a, long long *rem)
{
    const int nb = 64 - __clzll(a);
    const int sh = nb - 24;
    unsigned long long mh;
    if (sh <= 0) {
        mh = a << (-sh);
        if (rem) *rem = 0;
    } else {
        mh = (a + (1ull << (sh - 1))) >> sh;
        if (rem) *rem = (long long)a - (long long)(mh << sh);
    }
    int ex = nb - 1;
    if (mh >> 24) {                                  // rounding carried into bit 24
        mh >>= 1;
        ex++;
    }
    return ((unsigned)(ex + 127) << 23) | ((unsigned)mh & 0x7fffffu);
}

// An int64 (|v| < 2^62) as float-float with integer operations.
__device__ __forceinline__ float2 ll_to_ff(long long v)
{
    if (v == 0) return make_float2(0.f, 0.f);
    const unsigned sv = v < 0 ? 0x80000000u : 0u;
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    long long r;
    const float hi = __uint_as_float(sv | u64_round_float(a, &r));
    if (r == 0) return make_float2(hi, 0.f);
    const unsigned sr = ((r < 0) != (v < 0)) ? 0x80000000u : 0u;
    const unsigned long long ar = r < 0 ? 0ull - (unsigned long long)r : (unsigned long long)r;
    return make_float2(hi, __uint_as_float(sr | u64_round_float(ar, nullptr)));
}

// d 2^-e as float-float (ff_split of the scaled value, the scaling done on
// the exponent field)
__device__ __forceinline__ float2 ff_split_scaled(double d, int e)
{
    const int ex = (__double2hiint(d) >> 20) & 0x7ff;
    if (ex == 0) return make_float2(0.f, 0.f);
    if (ex == 0x7ff) return ff_split(d);             // inf, NaN stay so
    const int ne = ex - e;
    if (ne <= 0) return make_float2(0.f, 0.f);
    const long long b = __double_as_longlong(d);
    const long long nb = (b & ~(0x7ffll << 52)) | ((long long)ne << 52);
    return ff_split(__longlong_as_double(nb));
}

constexpr int kFftThreads = 384;   // at most, 24 warps on an SM (80 registers)

__global__ void __launch_bounds__(kFftThreads, 2) k_fft_rows_ff(double2 *__restrict__ data, int64_t rows,
                                                        FftRowsFF p, const float4 *__restrict__ tab)
{
    chain_enter();
    extern __shared__ __align__(16) f2 fsh[];
    __shared__ int emax_w[kFftThreads / 32];
    const int L = p.L, Lp = sh_len(L);
    const float sf = (float)p.sign;
    const f2 s = pk(-sf, sf);
    const ulonglong2 *tw0 = reinterpret_cast<const ulonglong2 *>(tab);
    const ulonglong2 *tw = p.sign < 0 ? tw0 : tw0 + 2 * L;
    const int half = 2 * Lp + (2 * Lp & 1);
    f2 *A = fsh, *B = fsh + half;
    // fused pack from int64 planes: the values need no row scaling (|v| <
    // 2^60 stays far inside the float range after the transform's growth by
    // at most L); the 2^-S of the fixed-point grid is applied on the way out
    const unsigned long long bnd = p.bound ? *p.bound : kFixedOff;
    const bool fixed_in = p.pack_in && bnd != kFixedOff;
    const int S = fixed_in ? fix_shift(bnd) : 0;
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        double2 *d = data + row * L;
        const int64_t q = p.Mx ? row / p.Mx : 0, xr = row - q * p.Mx;
        int64_t off_re = (2 * q) * p.G + xr * L, off_im = (2 * q + 1) * p.G + xr * L;
        bool has_im = 2 * q + 1 < p.npl_in;
        if (p.fold && 2 * q + 1 == p.npl_in) {        // the folded plane: rows xr, xr + Mx/2
            off_im = (2 * q) * p.G + (xr + p.Mx / 2) * L;
            has_im = true;
        }
        int e;
        if (fixed_in) {
            const long long *g = static_cast<const long long *>(p.pack_in);
            for (int k = threadIdx.x; k < L; k += blockDim.x) {
                const long long vr = g[off_re + k], vi = has_im ? g[off_im + k] : 0;
                sh_put(A, Lp, k, fc_make(ll_to_ff(vr), ll_to_ff(vi)));
            }
            e = -S;
        } else {
            // the row as doubles into B (2 Lp pairs >= L double2), and its
            // largest exponent
            double2 *raw = reinterpret_cast<double2 *>(B);
            int em = 0;
            for (int k = threadIdx.x; k < L; k += blockDim.x) {
                double2 v;
                if (p.pack_in) {
                    const double *g = static_cast<const double *>(p.pack_in);
                    v = make_double2(g[off_re + k], has_im ? g[off_im + k] : 0.0);
                } else {
                    v = d[k];
                }
                raw[k] = v;
                em = max(em, max((__double2hiint(v.x) >> 20) & 0x7ff, (__double2hiint(v.y) >> 20) & 0x7ff));
            }
            for (int o = 16; o > 0; o >>= 1) em = max(em, __shfl_xor_sync(~0u, em, o));
            if ((threadIdx.x & 31) == 0) emax_w[threadIdx.x >> 5] = em;
            __syncthreads();
            em = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) em = max(em, emax_w[w]);
            // scale 2^-e brings the largest finite entry to [2^63, 2^64) (no
            // scaling of a zero row or of one with an inf or NaN, which then
            // spreads through the row as in an FP64 transform)
            e = (em == 0 || em == 0x7ff) ? 0 : em - 1023 - 63;
            for (int k = threadIdx.x; k < L; k += blockDim.x) {
                const double2 v = raw[k];
                sh_put(A, Lp, k, fc_make(ff_split_scaled(v.x, e), ff_split_scaled(v.y, e)));
            }
        }
        __syncthreads();
        int Ns = 1;
        for (int st = 0; st < p.nst; st++) {
            const int R = p.radix[st];
            const unsigned mg = p.magic[st];
            switch (R) {
            case 12: stage<12>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 8: stage<8>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 4: stage<4>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 6: stage<6>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 2: stage<2>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 7: stage<7>(A, B, L, Ns, mg, s, tw, tw0); break;
            case 5: stage<5>(A, B, L, Ns, mg, s, tw, tw0); break;
            default: stage<3>(A, B, L, Ns, mg, s, tw, tw0); break;
            }
            Ns *= R;
            f2 *t = A;
            A = B;
            B = t;
            __syncthreads();
        }
        if (p.unpack_out) {
            // fused unpack: real and imaginary parts to their planes, with the
            // largest |value| for the fixed-point gather
            const bool has_im = 2 * q + 1 < p.npl_out;
            unsigned long long m = 0;
            for (int k = threadIdx.x; k < L; k += blockDim.x) {
                const fc v = sh_get(A, Lp, k);
                const float2 vh = upk(v.h), vl = upk(v.l);
                const double re = ff_to_double_scaled(vh.x, vl.x, e);
                p.unpack_out[off_re + k] = re;
                m = max(m, (unsigned long long)__double_as_longlong(fabs(re)));
                if (has_im) {
                    const double im = ff_to_double_scaled(vh.y, vl.y, e);
                    p.unpack_out[off_im + k] = im;
                    m = max(m, (unsigned long long)__double_as_longlong(fabs(im)));
                }
            }
            if (p.gmax) {
                for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(~0u, m, o));
                if ((threadIdx.x & 31) == 0 && m) atomicMax(p.gmax + q, m);
            }
        } else {
            for (int k = threadIdx.x; k < L; k += blockDim.x) {
                const fc v = sh_get(A, Lp, k);
                const float2 vh = upk(v.h), vl = upk(v.l);
                d[k] = make_double2(ff_to_double_scaled(vh.x, vl.x, e),
                                    ff_to_double_scaled(vh.y, vl.y, e));
            }
        }
        // the next row reuses both buffers and emax_w
        A = fsh;
        B = fsh + half;
        __syncthreads();
    }
}

}  // namespace

bool fft_rows_ff_plan(int L, FftRowsFF &p)
{
    p.L = L;
    p.nst = 0;
    if (L < 2 || L > kFftFFMaxLen) return false;
    // The factorisation into the butterflies at hand that costs least: per point and
    // stage the butterfly's instructions (counted from the code) and 55 for the
    // twiddle, shared memory and the barrier.  2688 = 8 4 12 7: 2^20 points 11.21 ms
    // against 11.33 as 8 8 6 7 (14, 16, 10 as butterflies spill registers: 11.24 to 11.72).
    static const int kR[] = {12, 8, 7, 6, 5, 4, 3, 2};
    static const int kC[] = {55, 38, 55, 44, 43, 22, 33, 11};
    constexpr int NR = sizeof kR / sizeof *kR;
    int n = L;
    int best = INT_MAX, pick[kFftFFMaxStages], at = 0, depth = 0, cost = 0;
    // (depth first, each factor no larger than the one before; at: the next to try)
    for (;;) {
        if (n == 1 && cost < best) {
            best = cost;
            p.nst = depth;
            for (int i = 0; i < depth; i++) p.radix[i] = kR[pick[i]];
        }
        while (at < NR && !(n % kR[at] == 0 && n > 1 && depth < kFftFFMaxStages &&
                            cost + kC[at] + 55 < best))
            at++;
        if (at < NR) {
            pick[depth++] = at;
            n /= kR[at];
            cost += kC[at] + 55;
        } else if (depth > 0) {
            at = pick[--depth];
            n *= kR[at];
            cost -= kC[at] + 55;
            at++;
        } else {
            break;
        }
    }
    if (best == INT_MAX) return false;
    // powers of two first: the early stages' strided stores are free of bank conflicts
    // for them
    std::stable_partition(p.radix, p.radix + p.nst, [](int r) { return (r & (r - 1)) == 0; });
    unsigned long long Ns = 1;
    for (int st = 0; st < p.nst; st++) {
        // (the first stage, Ns = 1, takes k = 0 without it)
        p.magic[st] = Ns == 1 ? 0u : (unsigned)(((1ull << 32) + Ns - 1) / Ns);
        Ns *= (unsigned long long)p.radix[st];
    }
    return true;
}

void fft_rows_ff_twiddles(int L, float4 *host)
{
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int m = 0; m < L; m++) {
        const long double a = -2.0L * pi * (long double)m / (long double)L;
        const long double c = cosl(a), sn = sinl(a);
        const float ch = (float)c, sh = (float)sn;
        const float cl = (float)(c - (long double)ch), sl = (float)(sn - (long double)sh);
        host[2 * m] = host[2 * (L + m)] = make_float4(ch, ch, cl, cl);
        host[2 * m + 1] = make_float4(-sh, sh, -sl, sl);
        host[2 * (L + m) + 1] = make_float4(sh, -sh, sl, -sl);
    }
}

cudaError_t launch_fft_rows_ff(double2 *data, int64_t rows, const FftRowsFF &p, const float4 *tw,
                               cudaStream_t st, int64_t &launches)
{
    if (rows <= 0) return cudaSuccess;
    auto bytes = [](int L) { return sizeof(f2) * 2 * ((size_t)(2 * sh_len(L) + 1) & ~(size_t)1); };
    const size_t smem = bytes(p.L);
    // (the limit is the process's, not the launch's: that of the longest row, so that
    // another thread's call cannot lower it in between)
    cudaError_t e = cudaFuncSetAttribute(k_fft_rows_ff, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bytes(kFftFFMaxLen));
    if (e != cudaSuccess) return e;
    const int per_sm = (int)std::max<size_t>(1, (size_t)(200 * 1024) / (smem + 1024));
    const int64_t cap = (int64_t)sm_count() * per_sm;
    const unsigned g = (unsigned)(rows < cap ? rows : cap);
    // 768 threads on an SM over the rows its shared memory holds, at least 128 a row, so
    // that one row's barriers are another's work.  L = 1344 (four rows): a gradient of
    // 2^18 points 7.43 ms with 256 threads at 16 warps per SM, 7.14 with 128, and at 24
    // warps 6.89 with 128, 6.78 with 192, 7.20 with 256 (later code); L = 640: 50,000
    // points 733, 694, then 650 us at 16 warps and 634 at 24; L = 2688 (two rows): 2^20
    // points 10.97 ms with 256 threads at 16 warps, 10.92 with 384 at 24.
    const int threads = std::max(128, std::min(kFftThreads, 768 / per_sm / 32 * 32));
    launch_chained(k_fft_rows_ff, g, threads, smem, st, data, rows, p, tw);
    launches++;
    return cudaGetLastError();
}

}  // namespace se2p
