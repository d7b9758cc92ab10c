// Per-sample tropical Monte Carlo kernel body, compiled at run time for one graph
// topology (the host prepends the constants below and compiles with NVRTC for
// sm_103a, so every edge endpoint is a compile-time constant and all matrices live
// in registers).
//
// Required definitions:
//   FT_E, FT_V        edges, vertices            FT_K        eps orders
//   FT_LOOPS          loop number                FT_RANK     rank of the reduced P
//   FT_PREC           0: plain FP64, 1: mixed FP32 with FP64 sampling decisions
//   FT_MODE           0: undeformed integrand (srcs/feynman_integral.hpp:218-276)
//                     1: deformed integrand  (srcs/feynman_integral.hpp:278-362)
//   FT_ONLY_PSI       1 when W = 0 and one eps order (only psi is needed)
//   FT_RECORD         1: write per-sample records
//   FT_BLOCK          threads per block
//   FT_EK[], FT_EL[]  edge endpoints (FT_EK[e] > FT_EL[e])
//
// One thread owns one sample at a time and walks a contiguous block of samples of
// the seed's single xoshiro256+ stream, so the samples are exactly those of the
// reference run with one OpenMP thread (srcs/feynman_integral.hpp:144-164).
//
// Numerical design (the reference's algebra, restated for a GPU thread):
//  * Sector draw (srcs/tropical_sampling.hpp:468-564): the cut scan compares running
//    sums of Jr/r against u*Jr in FP64 in the reference's order, so the removal order
//    is bit-identical.  Where the table fits in shared memory (E <= 12) both forms compare
//    the draw with 28-bit thresholds and repeat the step in FP64 when that does not
//    decide; beyond, the mixed form scans in FP32 with a rigorous margin.  The mixed
//    form keeps log X in a two-float sum; the FP64 form takes its powers in fixed point.
//  * The deleted vertex of the reduced Laplacian is always the last one of the
//    kernel's labels (the host numbers the vertices without external momentum first,
//    so it is an external one).  Any choice gives the same psi, phi/psi and
//    derivatives (matrix-tree theorem and momentum conservation); the reference's
//    choice only affects rounding.
//  * The real reduced Laplacian is eliminated in conductance form: pivots are sums
//    of positive conductances and updates add positive products, so psi = det L *
//    prod X has full relative accuracy whatever the spread of X.
//  * phi/psi = -tr(L^-1 P~) with P~ = sum_r sigma_r q_r q_r^T (host eigen-split):
//    each term is a forward substitution with the elimination multipliers.  The
//    mixed form's complex block instead contracts P~'s external block with L(y)^-1
//    directly, one quadratic form of P~ per row of the substitution's triangular map.
//  * Deformed branch: L^-1 from the positive factors, x-derivatives of phi/psi
//    (srcs/laplacian.hpp:102-215), the complex Laplacian eliminated in the same
//    conductance form with a pivot-growth check (the FP64 form's failing samples take
//    a complete-pivoting LU, srcs/feynman_integral.hpp:305; the mixed form runs this
//    elimination and V in two-float and hands the rare failing samples to FP64), and
//    the Jacobian determinant det(I + i*lambda' H X) (srcs/feynman_integral.hpp:312) as
//    that of D^2/X + i*lambda' D H D, D ~ X^1/2 powers of two: its real part is diagonal
//    and at least 1, so symmetric elimination without pivoting is stable.
//  * Updates on structural zeros of the eliminations (from each topology's fill
//    pattern, generated by the host) and additions to zero are left out.

#ifndef FT_E
#error "topology constants missing"
#endif
#ifndef FT_MINB
#define FT_MINB 1
#endif
// 1: the module holds the batch kernels (many integrals of this topology per launch)
#ifndef FT_BATCH
#define FT_BATCH 0
#endif
// The sampling kernel (0) and the FP64 pass over hand-offs (1, FP64 form) are modules of their
// own: each holds the straight-line code of a sample.  In one module an FP64 class took 1.3 s
// (triangle), 6.9 (double box) and 10.8 (3-loop ladder) to compile on 8 host cores; the sampling
// kernel alone 0.8, 4.3 and 7.3.  Mixed classes compile theirs and the two FP64 modules side by
// side: double box 6.2 -> 4.2 s, ladder 12.4 -> 6.8.
#ifndef FT_PART
#define FT_PART 0
#endif

typedef unsigned long long u64;
typedef unsigned int u32;

// Code size: the per-topology kernel is straight-line code (every loop unrolled so
// that the small matrices stay in registers), and the FP32 library functions carry
// large slow paths.  FT_VARIANT bit 0 keeps one out-of-line copy of each FP32
// transcendental, so the code the SM streams per sample fits the instruction caches
// better; bit 2 starts every sample with a block-wide barrier, so that the block's
// warps walk the code together and share its instruction fetches;
// bit 3 keeps one out-of-line copy of each larger
// two-float routine (logarithm, exponential, e^(ix), complex inverse, argument), bit 4
// of the complex two-float product and multiply-add.
#ifndef FT_VARIANT
#define FT_VARIANT 0
#endif
#if (FT_VARIANT & 1)
#define FT_MATHFN __noinline__
#else
#define FT_MATHFN __forceinline__
#endif
#if (FT_VARIANT & 8)
#define FT_BIGFN __noinline__
#else
#define FT_BIGFN __forceinline__
#endif
#if (FT_VARIANT & 16)
#define FT_CXFN __noinline__
#else
#define FT_CXFN __forceinline__
#endif
static __device__ FT_MATHFN float m_exp(float x) { return expf(x); }
static __device__ FT_MATHFN float m_exp2(float x) { return exp2f(x); }
static __device__ FT_MATHFN float m_log2(float x) { return log2f(x); }
static __device__ FT_MATHFN void m_sincos(float x, float* s, float* c) { sincosf(x, s, c); }

#define FT_N (FT_V - 1)
// reduced vertices [0, FT_Q0) carry no external momentum: the vectors q_r of P~ vanish
// there (the host labels the internal vertices first), so the forward substitutions
// of the quadratic forms start at row FT_Q0
#ifndef FT_Q0
#define FT_Q0 0
#endif
// Structural pattern of the eliminations, generated per topology: NZC(i, j) (i < j) a
// conductance between i and j that can be non-zero when i is eliminated (an edge or
// fill), NZG(i) a conductance to ground, NZM(i, j) an entry of M^-1 that can be
// non-zero.  Updates on structural zeros are left out.
#define NZC(i, j) (FT_NZC[i][j] != 0)
#define NZG(i) (FT_NZG[i] != 0)
#define NZM(i, j) (FT_NZM[i][j] != 0)
// Contributions to a conductance come from edges, then from eliminated vertices: FT_CF[i][j]
// (FT_GF[i] for the ground) is the first of those vertices, -1 with an edge before; the
// first contribution is assigned, not added to zero.  FT_CS, FT_GS: more than one
// contribution (a sum, which the two-float forms renormalise before it is used).
#define ADDS_C(k, i, j) (FT_CF[i][j] < (k))
#define ADDS_G(k, i) (FT_GF[i] < (k))
#define SUMS_C(i, j) (FT_CS[i][j] != 0)
#define SUMS_G(i) (FT_GS[i] != 0)
// edge e is the first to contribute to its conductance slot (the pair of endpoints, or
// the ground slot of its lower endpoint): its conductance is assigned, not added to zero
static __device__ constexpr bool first_in_slot(int e)
{
    for (int f = 0; f < e; f++)
        if (FT_EK[f] == FT_EK[e] && FT_EL[f] == FT_EL[e]) return false;
    return true;
}
#define FT_FULL ((1u << FT_E) - 1u)

// ------------------------------------------------------------------ parameter block
// doubles: 0 D, 1 W, 2 IGtr, 3 def_ref, 4 norm = 1/(D/2*L+W), 5 Jr(full), 6 -norm D/2, 7 -norm W,
// then m2[E], nu[E], sigma[RANK], q[RANK][N], then P~ on the external rows [Q0, N)
// (its upper triangle row by row, off-diagonal entries doubled)
#define P_D 0
#define P_W 1
#define P_IGTR 2
#define P_DEF 3
#define P_NORM 4
#define P_JRFULL 5
#define P_NORM_F 6
#define P_NORM_G 7
#define LN2_D 0.693147180559945309417
#define P_M2 8
#define P_NU (8 + FT_E)
#define P_SIG (8 + 2 * FT_E)
#define P_Q (8 + 2 * FT_E + FT_RANK)
#define FT_NE (FT_N - FT_Q0)
#define P_PT (8 + 2 * FT_E + FT_RANK + FT_RANK * FT_N)
#define P_SIZE (P_PT + FT_NE * (FT_NE + 1) / 2)
// entry (j, k), j <= k, of the external block of P~ (indices from Q0)
#define PT_AT(j, k) (P_PT + (j) * FT_NE - (j) * ((j) - 1) / 2 + ((k) - (j)))
// the same block as floats follows at prm + P_SIZE, then in two-float as (hi, hi, lo, lo)
// float4s at prm + P_PAIR (the mixed form reads only those two)
#define P_PAIR ((P_SIZE + (P_SIZE + 1) / 2 + 1) & ~1)

// ------------------------------------------------------------------ table layout
// [w64 | Jr64 | rinv64 : 8 bytes each][pad to 16][rinv32 hi | rinv32 lo | meta : 4 bytes each]
// then the cut thresholds (FT_CUT: one u32 per edge of every subgraph, see find_cut) or,
// for tables read from global memory, [w32 | Jr32 : 4 bytes each] for the running-sum
// scan.  meta: offset of the subgraph's thresholds << 16 | mass-momentum spanning << 7 |
// loop number.
#define T_ENTRIES (1u << FT_E)
#define T_W64 0
#define T_JR64 (8u * T_ENTRIES)
#define T_RI64 (16u * T_ENTRIES)
#define T_F32 ((24u * T_ENTRIES + 15u) & ~15u)
#define T_RH32 (T_F32)                    // 1/r in two-float: high parts, low parts
#define T_RL32 (T_F32 + 4u * T_ENTRIES)
#define T_META (T_F32 + 8u * T_ENTRIES)
#define T_Q (T_F32 + 12u * T_ENTRIES)
#define T_W32 (T_F32 + 12u * T_ENTRIES)
#define T_JR32 (T_F32 + 16u * T_ENTRIES)
#define FT_CUT (!FT_TABLE_GLOBAL)
#if FT_CUT
#define T_QBYTES (2u * FT_E * T_ENTRIES)  // E 2^(E-1) thresholds
#else
#define T_QBYTES 0u
#endif
#define META_OFF(m) ((m) >> 16)
#define META_MM(m) (((m) >> 7) & 1u)
#define META_L(m) ((m) & 127u)

// ------------------------------------------------------------------ accumulator slots
// per eps order j: [8j + 0..7] = re S1 (hi, lo), re S2 (hi, lo), im S1 (hi, lo), im S2 (hi, lo)
// then [8K] kept, [8K+1] dropped, [8K+2] queued, [8K+3] exact sampling steps,
// [8K+4] robust factorisations
#define ACC_KEPT (8 * FT_K)
#define ACC_DROPPED (8 * FT_K + 1)
#define ACC_QUEUED (8 * FT_K + 2)
#define ACC_EXACT (8 * FT_K + 3)
#define ACC_ROBUST (8 * FT_K + 4)
#define ACC_SLOTS (8 * FT_K + 8)

// record flags
#define REC_DROPPED 1
#define REC_QUEUED 2
#define REC_EXACT 4
#define REC_ROBUST 8

// ------------------------------------------------------------------ small helpers
static __device__ __forceinline__ u64 rotl64(u64 x, int k) { return (x << k) | (x >> (64 - k)); }

struct xo {
    u64 a, b, c, d;
    __device__ __forceinline__ u64 next()
    {
        const u64 out = a + d;
        const u64 t = b << 17;
        c ^= a;
        d ^= b;
        b ^= c;
        a ^= d;
        c ^= t;
        d = rotl64(d, 45);
        return out;
    }
};

static __device__ __forceinline__ void rewind(xo& g, int n)
{
    // n steps back: b = y ^ (b << 17) with y = b' ^ c' solved by substitution
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        const u64 d1 = rotl64(g.d, 19);
        const u64 y = g.b ^ g.c;
        const u64 b = y ^ (y << 17) ^ (y << 34) ^ (y << 51);
        const u64 c1 = g.c ^ (b << 17);
        g.a ^= d1;
        g.b = b;
        g.c = c1 ^ g.a;
        g.d = d1 ^ b;
    }
}

static __device__ __forceinline__ double u01(u64 x) { return (double)(x >> 11) * 0x1.0p-53; }

template <class T>
struct cx {
    T re, im;
};
template <class T>
static __device__ __forceinline__ cx<T> cmk(T r, T i)
{
    cx<T> z;
    z.re = r;
    z.im = i;
    return z;
}
template <class T>
static __device__ __forceinline__ cx<T> operator+(cx<T> a, cx<T> b) { return cmk(a.re + b.re, a.im + b.im); }
template <class T>
static __device__ __forceinline__ cx<T> operator-(cx<T> a, cx<T> b) { return cmk(a.re - b.re, a.im - b.im); }
template <class T>
static __device__ __forceinline__ cx<T> operator*(cx<T> a, cx<T> b)
{
    return cmk(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
template <class T>
static __device__ __forceinline__ cx<T> operator*(T s, cx<T> a) { return cmk(s * a.re, s * a.im); }
// reciprocals: IEEE division in FP64; the correctly rounded reciprocal instruction
// sequence in FP32 (a division there expands to a long inline sequence)
static __device__ __forceinline__ double rcp_(double x) { return 1.0 / x; }
static __device__ __forceinline__ float rcp_(float x) { return __frcp_rn(x); }
template <class T>
static __device__ __forceinline__ cx<T> crecip(cx<T> z)
{
    // scaled so that |z|^2 cannot overflow in single precision
    const T s = fmax(fabs(z.re), fabs(z.im));
    const T is = rcp_(s);
    const T r = z.re * is, i = z.im * is;
    const T id = rcp_(s * (r * r + i * i));
    return cmk(r * id, -i * id);
}
static __device__ __forceinline__ double cabs_(cx<double> z) { return hypot(z.re, z.im); }
// principal logarithm and real power (the reference's std::log / std::pow on
// complex<double>, srcs/feynman_integral.hpp:310,327,354)
static __device__ __forceinline__ cx<double> clog_(cx<double> z) { return cmk(log(hypot(z.re, z.im)), atan2(z.im, z.re)); }
static __device__ __forceinline__ cx<double> cpow_(cx<double> z, double y)
{
    double lr = log(hypot(z.re, z.im)), th = atan2(z.im, z.re);
    double s, c, m = exp(y * lr);
    sincos(y * th, &s, &c);
    return cmk(m * c, m * s);
}

#if FT_PREC == 0
// ------------------------------------------------------------------ FP64 functions
// The FP64 pipe takes 16 cycles of the whole SM per warp instruction (64x fewer lanes than
// FP32) and bounds the FP64 form, with nine tenths of the issue slots idle.  Its powers,
// exponentials, logarithms, sines and cosines are therefore evaluated in 64-bit fixed point
// on the integer pipes (about 200 instructions each, where table-driven FP64 versions
// issued 12 to 31 FP64 ones, several times their cost), table-driven after Tang (ACM TOMS
// 15 (1989), 16 (1990), 17 (1991)) with Taylor polynomials, and assembled into doubles by
// their bits.  A logarithm's error is below 2^-61 and is multiplied by the exponent, so the
// fixed-point powers take exponents below 32 only (their error before the final rounding is
// then below 2^-55: 0.75 ulp); sines and cosines are within 2^-58 absolute, the sine of a
// small angle within 0.75 ulp.  Reciprocals and arguments stay on the FP64 pipe (3 and 17
// instructions).  Arguments outside the stated ranges take the CUDA library's function (out of
// line).  Qn: a fixed-point number in units of 2^-n.
static __device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
static __device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
static __device__ __forceinline__ bool finite_(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
static __device__ __forceinline__ double pow2_of(int e) { return __hiloint2double((1023 + e) << 20, 0); }
static __device__ __forceinline__ bool normal_positive(double x) { return (u32)(hi_word(x) - 0x00100000) < 0x7fe00000u; }
// the significand of a normal x, Q63 in [1, 2)
static __device__ __forceinline__ u64 mantissa_of(double x) { return ((u64)__double_as_longlong(x) << 11) | (1ull << 63); }
// w 2^e, w in Q63 with its top bit set, rounded to a double (e in the normal range)
static __device__ __forceinline__ double round_q63(u64 w, int e)
{
    return __longlong_as_double((long long)(((u64)(1022 + e) << 52) + (w >> 11) + ((w >> 10) & 1ull)));
}
// v in Qq as a double
static __device__ __forceinline__ double double_of(u64 v, int q)
{
    if (v == 0ull) return 0.0;
    const int lz = __clzll((long long)v);
    return round_q63(v << lz, 63 - lz - q);
}
// log2 of m 2^-52 in [1, 2): Q62 in [0, 1].  With i its top 8 fraction bits, r_i is 10 bits at
// least 1024 / M, so that z = M r / 1024 - 1 is exact and in [0, 0.005)
static __device__ __forceinline__ u64 log2_q62(u64 m)
{
    const ulonglong2 t = FT_LOG64[(m >> 44) & 255ull];   // r, -log2(r / 1024) in Q62
    const u64 z = (m * t.x - (1ull << 62)) << 8;        // Q70
    u64 h = (1ull << 63) / 7ull;                         // Q63
    h = (1ull << 63) / 6ull - (__umul64hi(z, h) >> 6);
    h = (1ull << 63) / 5ull - (__umul64hi(z, h) >> 6);
    h = (1ull << 63) / 4ull - (__umul64hi(z, h) >> 6);
    h = (1ull << 63) / 3ull - (__umul64hi(z, h) >> 6);
    h = (1ull << 63) / 2ull - (__umul64hi(z, h) >> 6);
    const u64 l = z - (__umul64hi(__umul64hi(z, z), h) >> 5);   // log1p z, Q70
    const u64 f = t.y + (__umul64hi(l, FT_LOG2E_Q63) >> 7);
    return f < (1ull << 62) ? f : (1ull << 62);
}
// 2^(f - n), f in Q64
static __device__ __forceinline__ double exp2_q64(u64 f, int n)
{
    const u64 T = FT_EXP64[f >> 56];                     // 2^(j/256), Q63
    const u64 w = __umul64hi(f << 8, FT_LN2_Q64);       // Q72, below ln2/256
    u64 h = (1ull << 63) / 120ull;
    h = (1ull << 63) / 24ull + (__umul64hi(w, h) >> 8);
    h = (1ull << 63) / 6ull + (__umul64hi(w, h) >> 8);
    h = (1ull << 63) / 2ull + (__umul64hi(w, h) >> 8);
    h = (1ull << 63) + (__umul64hi(w, h) >> 8);
    const u64 R = T + (__umul64hi(T, __umul64hi(w, h)) >> 7);
    return round_q63(R, -n);
}
static __device__ __noinline__ double pow_slow(double x, double y) { return pow(x, y); }
// v 2^-64 of the signed 128-bit v, shifted by s in [-58, 6]: integer part i, fraction f in Q64
static __device__ __forceinline__ void shift_fixed(long long hi, u64 lo, int s, int& i, u64& f)
{
    if (s >= 0) {
        i = (int)(((u64)hi << s) | ((lo >> 1) >> (63 - s)));
        f = lo << s;
    } else {
        i = (int)(hi >> -s);
        f = (lo >> -s) | ((u64)hi << (64 + s));
    }
}
// (1 - u)^y, u = (x >> 11) 2^-53, y in [2^-60, 32)
static __device__ __forceinline__ double pow_1mu(u64 x, double y)
{
    const u64 q = (~x & ~0x7ffull) + 0x800ull;   // (1 - u) 2^64, 0 for u = 0
    if (q == 0ull) return 1.0;
    const int ey = (hi_word(y) >> 20) - 1023;   // negative y: far below
    if ((u32)(ey + 60) > 64u) return pow_slow(1.0 - u01(x), y);
    const int lz = __clzll((long long)q);
    // y (K - F), -log2(1 - u) = K - F: the product with K is exact, with F a Q62 one
    const u64 F = log2_q62((q << lz) >> 11), m = mantissa_of(y);
    const u64 k = (m >> 11) * (u64)(1 + lz), p = __umul64hi(m, F << 1), lo = (k << 10) - p;
    int n;
    u64 f;
    shift_fixed((long long)((k >> 54) - ((k << 10) < p)), lo, ey + 2, n, f);
    if (n > 1000) return pow_slow(1.0 - u01(x), y);
    return exp2_q64(0ull - f, n + (f != 0ull));
}
// log2 x = k + f of a positive normal x, f in Q62 in [0, 1], k an integer
struct log2_parts {
    int k;
    u64 f;
};
static __device__ __forceinline__ log2_parts log2_64(double x)
{
    log2_parts r;
    r.k = (hi_word(x) >> 20) - 1023;
    r.f = log2_q62((u64)__double_as_longlong(x) & 0xfffffffffffffull | (1ull << 52));
    return r;
}
// The logarithms (|log2| + 1) that the power of exponent a takes in fixed point: |a log2| is
// at most 500, so that a product of two powers stays in range and none of its factors is
// infinite or zero by itself, and |a| is in [2^-60, 32) or 0.
static __device__ __forceinline__ int log2_limit(double a)
{
    const int e = exponent_of(a) - 1022;   // |a| < 2^e
    if (e == -1022) return 500;
    return (u32)(e + 59) > 64u ? 0 : 500 >> max(e, 0);
}
static __device__ __forceinline__ bool in_reach(log2_parts l, int limit) { return abs(l.k) < limit; }
// i + f 2^-64 += a (l.k + l.f): the product with k is exact, with f a Q62 one
static __device__ __forceinline__ void add_product(double a, log2_parts l, int& i, u64& f)
{
    const int ea = exponent_of(a) - 1023;
    if (ea < -60) return;   // 0
    const u64 m = mantissa_of(a), k = (m >> 11) * (u64)abs(l.k), p = __umul64hi(m, l.f << 1);
    u64 lo = k << 10, hi = k >> 54;
    if (l.k < 0) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0ull);
    }
    lo += p;
    hi += lo < p;
    if (hi_word(a) < 0) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0ull);
    }
    int I;
    u64 F;
    shift_fixed((long long)hi, lo, ea + 2, I, F);
    f += F;
    i += I + (f < F);
}
// 2^(a (la.k + la.f) + b (lb.k + lb.f)), both in reach
static __device__ __forceinline__ double power_product(double a, log2_parts la, double b, log2_parts lb)
{
    int i = 0;
    u64 f = 0ull;
    add_product(a, la, i, f);
    add_product(b, lb, i, f);
    return exp2_q64(f, -i);
}
// log2 x - L log2 y as a double, its error below 2^-61 (L + 1) before the rounding
static __device__ __forceinline__ double log2_difference(log2_parts x, log2_parts y, int L)
{
    const int k = x.k - L * y.k;
    const u64 p = y.f * (u64)L, d = x.f - p, add = (u64)(long long)k << 62;
    u64 lo = d + add, hi = (u64)((long long)k >> 2) - __umul64hi(y.f, (u64)L) - (x.f < p) + (lo < add);
    const bool neg = (long long)hi < 0;
    if (neg) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0ull);
    }
    if ((hi | lo) == 0ull) return 0.0;
    const int lz = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
    const u64 w = lz >= 64 ? lo << (lz - 64) : (lz ? (hi << lz) | (lo >> (64 - lz)) : hi);
    const double v = round_q63(w, 127 - lz - 62);
    return neg ? -v : v;
}
static __device__ __noinline__ void sincos_slow(double x, double* s, double* c) { sincos(x, s, c); }
// 256 steps per turn, 64 of them in the table
static __device__ __forceinline__ void sincos_64(double x, double& sn, double& cs)
{
    if ((u32)(hi_word(x) & 0x7fffffff) > 0x40f86a00u) {   // |x| > 1e5
        sincos_slow(x, &sn, &cs);
        return;
    }
    const int ex = exponent_of(x) - 1023;
    if (ex < -30) {   // x^2/6 below 2^-62
        sn = x;
        cs = 1.0;
        return;
    }
    // |x| 128/pi = m C 2^e, C in Q58 and 64 more bits
    const int S = 57 - ex;
    const u64 m = mantissa_of(x), c0 = m * FT_STEPS_Q58;
    const u64 lo = c0 + __umul64hi(m, FT_STEPS_LO);
    const u64 hi = __umul64hi(m, FT_STEPS_Q58) + (lo < c0);
    const u32 k = S < 64 ? (u32)(hi >> (S & 63)) : 0u;
    const u64 f = S < 64 ? (hi << ((64 - S) & 63)) | (lo >> (S & 63)) : (S < 128 ? hi >> (S - 64) : 0ull);   // Q64
    const u64 w = __umul64hi(f, FT_STEP_Q69), w2 = __umul64hi(w, w);   // Q69, Q74
    u64 h = (1ull << 63) / 120ull - (__umul64hi(w2, (1ull << 63) / 5040ull) >> 10);
    h = (1ull << 63) / 6ull - (__umul64hi(w2, h) >> 10);
    const u64 ratio = (1ull << 63) - (__umul64hi(w2, h) >> 10);   // sin w / w, Q63
    const u64 s = __umul64hi(w, ratio);                            // sin w, Q68
    h = (1ull << 63) / 720ull - (__umul64hi(w2, (1ull << 63) / 40320ull) >> 10);
    h = (1ull << 63) / 24ull - (__umul64hi(w2, h) >> 10);
    h = (1ull << 63) / 2ull - (__umul64hi(w2, h) >> 10);
    const u64 v = __umul64hi(w2, h);   // 1 - cos w, Q73
    const ulonglong2 T = FT_SC64[k & 63u];   // sin, cos of k pi/128, Q63
    const u64 A = (T.x >> 1) + (__umul64hi(T.y, s) >> 5) - (__umul64hi(T.x, v) >> 10);
    const u64 B0 = (T.y >> 1) - (__umul64hi(T.y, v) >> 10), B1 = __umul64hi(T.x, s) >> 5;
    // in the first step |x| itself times sin w / w, which keeps the relative accuracy
    const double a = double_of(k ? A : __umul64hi(m, ratio), k ? 62 : 62 - ex);
    const double b = double_of(B0 > B1 ? B0 - B1 : 0ull, 62);
    const bool odd = (k >> 6) & 1u, up = (k >> 7) & 1u;   // quadrant
    sn = odd ? b : a;
    cs = odd ? a : b;
    if (up != (hi_word(x) < 0)) sn = -sn;
    if (odd != up) cs = -cs;
}

static __device__ __noinline__ double rcp_slow(double x) { return 1.0 / x; }
static __device__ __forceinline__ double rcp64(double x)
{
    if ((u32)(exponent_of(x) - 23) > 2000u) return rcp_slow(x);
    // seed r with e = 1 - x r below 2^-19; r (1 + e + e^2) leaves e^3
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
static __device__ __noinline__ double arg_slow(double y, double x) { return atan2(y, x); }
// principal argument of re + i im: with x, y the larger and smaller modulus, c = i/128 the
// rounded ratio, atan(y/x) = atan c + atan((y - c x) / (x + c y)), the last below 1/256
static __device__ __forceinline__ double arg_64(double re, double im)
{
    const double ar = fabs(re), ai = fabs(im);
    const bool sw = hi_word(ai) > hi_word(ar);
    const double x = sw ? ai : ar, y = sw ? ar : ai;
    const int hx = hi_word(x), hy = hi_word(y);
    if ((u32)((hx >> 20) - 23) > 2000u) return arg_slow(im, re);
    const int d = (hy >> 20) - (hx >> 20);   // <= 0
    const float fx = __int_as_float(0x3f800000 | ((hx & 0xfffff) << 3));
    const float fy = d < -30 ? 0.0f : __int_as_float((0x3f800000 | ((hy & 0xfffff) << 3)) + d * 0x800000);
    const int i = (int)(fy * __frcp_rn(fx) * 128.0f + 0.5f);
    const double2 a = FT_ATAN64[2 * i], b = FT_ATAN64[2 * i + 1];   // c, hi; lo, -
    const double num = fma(-a.x, x, y), den = fma(a.x, y, x);
    const double r = rcp64(den);
    double z = num * r;
    z = fma(fma(-z, den, num), r, z);
    const double z2 = z * z;
    const double v = fma(z2 * z, fma(z2, fma(z2, -1.0 / 7.0, 1.0 / 5.0), -1.0 / 3.0), z) + b.x;
    // the octant: K +- (hi + v), K = 0, pi/2 or pi
    const bool left = hi_word(re) < 0;
    const bool minus = sw != left;   // the angle from the axis counts backwards
    const double K = sw ? 1.57079632679489655800 : (left ? 3.14159265358979311600 : 0.0);
    const double Kl = sw ? 6.12323399573676603587e-17 : (left ? 1.22464679914735317720e-16 : 0.0);
    const double A = (minus ? K - a.y : K + a.y) + (minus ? Kl - v : Kl + v);
    return hi_word(im) < 0 ? -A : A;
}
// 1/z: |z|^2 within range (else the scaled form)
static __device__ __noinline__ cx<double> cinv_slow(cx<double> z) { return crecip(z); }
static __device__ __forceinline__ cx<double> cinv_64(cx<double> z)
{
    const int e = max(exponent_of(z.re), exponent_of(z.im)) - 1023;
    if (e > 480 || e < -480) return cinv_slow(z);
    const double m = rcp64(fma(z.re, z.re, z.im * z.im));
    return cmk(z.re * m, -z.im * m);
}

// The FP64 pass over hand-offs runs a handful of samples through code that no instruction cache
// holds: its time is that of fetching it (150 us for one sample).  There the functions are
// called (COLD), where the sampling kernels, whose warps share the code, inline them: 14
// hand-offs of the 3-loop ladder (E = 10) took 0.6 ms more of its 7.9 ms inlined; with 7 and 8
// edges no difference.
static __device__ __noinline__ double pow_1mu_call(u64 x, double y) { return pow_1mu(x, y); }
static __device__ __noinline__ log2_parts log2_call(double x) { return log2_64(x); }
static __device__ __noinline__ double power_call(double a, log2_parts la, double b, log2_parts lb)
{
    return power_product(a, la, b, lb);
}
static __device__ __noinline__ double2 sincos_call(double x)
{
    double2 r;
    sincos_64(x, r.x, r.y);
    return r;
}
static __device__ __noinline__ double arg_call(double re, double im) { return arg_64(re, im); }
static __device__ __noinline__ cx<double> cinv_call(cx<double> z) { return cinv_64(z); }
template <bool COLD>
struct fn64 {
    static __device__ __forceinline__ double pow1mu(u64 x, double y) { return COLD ? pow_1mu_call(x, y) : pow_1mu(x, y); }
    static __device__ __forceinline__ log2_parts log2(double x) { return COLD ? log2_call(x) : log2_64(x); }
    static __device__ __forceinline__ double power(double a, log2_parts la, double b, log2_parts lb)
    {
        return COLD ? power_call(a, la, b, lb) : power_product(a, la, b, lb);
    }
    static __device__ __forceinline__ void sincos(double x, double& sn, double& cs)
    {
        if (COLD) {
            const double2 r = sincos_call(x);
            sn = r.x;
            cs = r.y;
        } else {
            sincos_64(x, sn, cs);
        }
    }
    static __device__ __forceinline__ double arg(double re, double im) { return COLD ? arg_call(re, im) : arg_64(re, im); }
    static __device__ __forceinline__ cx<double> cinv(cx<double> z) { return COLD ? cinv_call(z) : cinv_64(z); }
};
// ------------------------------------------------------------------ robust complex LU
// Complete-pivoting LU of the complex reduced Laplacian (largest modulus, first in
// column-major order), used when the static elimination reports pivot growth.
// Returns det and -tr(L^-1 P~).
static __device__ void robust_complex(const cx<double>* y, const double* prm, cx<double>& det, cx<double>& pphi)
{
    cx<double> A[FT_N * FT_N];
    int rp[FT_N], cp[FT_N];
    for (int i = 0; i < FT_N * FT_N; i++) A[i] = cmk(0.0, 0.0);
    for (int e = 0; e < FT_E; e++) {
        const int k = FT_EK[e], l = FT_EL[e];
        A[l * FT_N + l] = A[l * FT_N + l] + y[e];
        if (k == FT_V - 1) continue;
        A[k * FT_N + k] = A[k * FT_N + k] + y[e];
        A[k * FT_N + l] = A[k * FT_N + l] - y[e];
        A[l * FT_N + k] = A[l * FT_N + k] - y[e];
    }
    int nt = 0;
    for (int k = 0; k < FT_N; k++) {
        int br = k, bc = k;
        double best = -1.0;
        for (int c = k; c < FT_N; c++)
            for (int r = k; r < FT_N; r++) {
                double s = cabs_(A[r * FT_N + c]);
                if (s > best) {
                    best = s;
                    br = r;
                    bc = c;
                }
            }
        rp[k] = br;
        cp[k] = bc;
        if (br != k) {
            for (int c = 0; c < FT_N; c++) {
                cx<double> t = A[k * FT_N + c];
                A[k * FT_N + c] = A[br * FT_N + c];
                A[br * FT_N + c] = t;
            }
            nt++;
        }
        if (bc != k) {
            for (int r = 0; r < FT_N; r++) {
                cx<double> t = A[r * FT_N + k];
                A[r * FT_N + k] = A[r * FT_N + bc];
                A[r * FT_N + bc] = t;
            }
            nt++;
        }
        cx<double> inv = crecip(A[k * FT_N + k]);
        for (int r = k + 1; r < FT_N; r++) A[r * FT_N + k] = A[r * FT_N + k] * inv;
        for (int r = k + 1; r < FT_N; r++)
            for (int c = k + 1; c < FT_N; c++) A[r * FT_N + c] = A[r * FT_N + c] - A[r * FT_N + k] * A[k * FT_N + c];
    }
    det = cmk(1.0, 0.0);
    for (int i = 0; i < FT_N; i++) det = det * A[i * FT_N + i];
    if (nt & 1) det = cmk(-det.re, -det.im);
    // -tr(L^-1 P~), P~ = sum_r sigma_r q_r q_r^T: sum_r sigma_r q_r^T L^-1 q_r
    cx<double> tr = cmk(0.0, 0.0);
    for (int r = 0; r < FT_RANK; r++) {
        cx<double> b[FT_N];
        for (int i = 0; i < FT_N; i++) b[i] = cmk(prm[P_Q + r * FT_N + i], 0.0);
        for (int k = 0; k < FT_N; k++) {
            cx<double> t = b[k];
            b[k] = b[rp[k]];
            b[rp[k]] = t;
        }
        for (int i = 0; i < FT_N; i++)
            for (int j = 0; j < i; j++) b[i] = b[i] - A[i * FT_N + j] * b[j];
        for (int i = FT_N - 1; i >= 0; i--) {
            for (int j = i + 1; j < FT_N; j++) b[i] = b[i] - A[i * FT_N + j] * b[j];
            b[i] = b[i] * crecip(A[i * FT_N + i]);
        }
        for (int k = FT_N - 1; k >= 0; k--) {
            cx<double> t = b[k];
            b[k] = b[cp[k]];
            b[cp[k]] = t;
        }
        cx<double> s = cmk(0.0, 0.0);
        for (int i = 0; i < FT_N; i++) s = s + prm[P_Q + r * FT_N + i] * b[i];
        tr = tr + prm[P_SIG + r] * s;
    }
    pphi = cmk(-tr.re, -tr.im);
}

// ------------------------------------------------------------------ robust derivatives
// x-derivatives of phi/psi by the reference's route (srcs/feynman_integral.hpp:166-194,
// 283-287; srcs/laplacian.hpp:14-99, 102-215), for samples where an edge's conductance
// 1/x_e dwarfs the rest of the network between its ends: the fixed ground of the
// unrolled path then leaves both ends floating together, and the potential and
// resistance differences across the edge cancel.  Grounding the vertex with the
// smallest sum of incident x (the reference's choice) ties such an edge to the ground.
// Reduced Laplacian with that ground, LDL^T with diagonal pivoting, L^-1, L^-1 P L^-T,
// then the derivatives as differences of their entries.  Runtime indices, out of line:
// it runs for a few samples in 1e4 (edge weights below 1 make tiny x more frequent).
static __device__ __noinline__ void robust_derivatives(const double* X, const double* Xi, const double* prm,
                                                       double* dphi, double (*H)[FT_E])
{
    double XV[FT_V];
#pragma unroll 1
    for (int v = 0; v < FT_V; v++) XV[v] = 0.0;
#pragma unroll 1
    for (int e = 0; e < FT_E; e++) {
        XV[FT_EK[e]] += X[e];
        XV[FT_EL[e]] += X[e];
    }
    int gnd = 0;
#pragma unroll 1
    for (int v = 1; v < FT_V; v++)
        if (XV[gnd] > XV[v]) gnd = v;
    int map[FT_V];
#pragma unroll 1
    for (int v = 0; v < FT_V; v++) map[v] = v < gnd ? v : (v > gnd ? v - 1 : FT_N);
    // reduced Laplacian A and contracted scalar products B (P from its rank split; the
    // ground-V-1 row and column follow from momentum conservation)
    double A[FT_N][FT_N], B[FT_N][FT_N];
#pragma unroll 1
    for (int i = 0; i < FT_N; i++)
#pragma unroll 1
        for (int j = 0; j < FT_N; j++) A[i][j] = 0.0;
#pragma unroll 1
    for (int e = 0; e < FT_E; e++) {
        const int k = map[FT_EK[e]], l = map[FT_EL[e]];
        if (k < FT_N) A[k][k] += Xi[e];
        if (l < FT_N) A[l][l] += Xi[e];
        if (k < FT_N && l < FT_N) {
            A[k][l] -= Xi[e];
            A[l][k] -= Xi[e];
        }
    }
    auto Pfull = [&](int i, int j) -> double {
        // P[i][j] of the V x V matrix with zero row and column sums
        double s = 0.0;
#pragma unroll 1
        for (int r = 0; r < FT_RANK; r++) {
            double qi = 0.0, qj = 0.0;
            if (i < FT_N) {
                qi = prm[P_Q + r * FT_N + i];
            } else {
#pragma unroll 1
                for (int m = 0; m < FT_N; m++) qi -= prm[P_Q + r * FT_N + m];
            }
            if (j < FT_N) {
                qj = prm[P_Q + r * FT_N + j];
            } else {
#pragma unroll 1
                for (int m = 0; m < FT_N; m++) qj -= prm[P_Q + r * FT_N + m];
            }
            s += prm[P_SIG + r] * qi * qj;
        }
        return s;
    };
#pragma unroll 1
    for (int v = 0; v < FT_V; v++) {
        if (v == gnd) continue;
#pragma unroll 1
        for (int w = 0; w < FT_V; w++) {
            if (w == gnd) continue;
            B[map[v]][map[w]] = Pfull(v, w);
        }
    }
    // A = P^T L D L^T P (diagonal pivoting); then A^-1 column by column into C
    int perm[FT_N];
#pragma unroll 1
    for (int i = 0; i < FT_N; i++) perm[i] = i;
#pragma unroll 1
    for (int k = 0; k < FT_N; k++) {
        int pk = k;
#pragma unroll 1
        for (int i = k + 1; i < FT_N; i++)
            if (fabs(A[i][i]) > fabs(A[pk][pk])) pk = i;
        if (pk != k) {
#pragma unroll 1
            for (int j = 0; j < FT_N; j++) {
                const double t = A[k][j];
                A[k][j] = A[pk][j];
                A[pk][j] = t;
            }
#pragma unroll 1
            for (int j = 0; j < FT_N; j++) {
                const double t = A[j][k];
                A[j][k] = A[j][pk];
                A[j][pk] = t;
            }
            const int t = perm[k];
            perm[k] = perm[pk];
            perm[pk] = t;
        }
        const double dk = A[k][k];
        // Schur update of the whole (symmetric) trailing block, so that later pivot
        // swaps see current values in both triangles; row k keeps the unscaled column
#pragma unroll 1
        for (int i = k + 1; i < FT_N; i++) {
            const double f = A[i][k] / dk;
#pragma unroll 1
            for (int j = k + 1; j < FT_N; j++) A[i][j] -= f * A[k][j];
        }
#pragma unroll 1
        for (int i = k + 1; i < FT_N; i++) A[i][k] /= dk;
    }
    // columns of the inverse: solve L D L^T y = P e_c; C[perm[i]][c] = y_i
    double C[FT_N][FT_N];
#pragma unroll 1
    for (int c = 0; c < FT_N; c++) {
        double y[FT_N];
#pragma unroll 1
        for (int i = 0; i < FT_N; i++) {
            double t = perm[i] == c ? 1.0 : 0.0;
#pragma unroll 1
            for (int j = 0; j < i; j++) t -= A[i][j] * y[j];
            y[i] = t;
        }
#pragma unroll 1
        for (int i = 0; i < FT_N; i++) y[i] /= A[i][i];
#pragma unroll 1
        for (int i = FT_N - 1; i >= 0; i--)
#pragma unroll 1
            for (int j = i + 1; j < FT_N; j++) y[i] -= A[j][i] * y[j];
#pragma unroll 1
        for (int i = 0; i < FT_N; i++) C[perm[i]][c] = y[i];
    }
    // S = C B C^T (into A, reusing it)
#pragma unroll 1
    for (int i = 0; i < FT_N; i++)
#pragma unroll 1
        for (int j = 0; j < FT_N; j++) {
            double t = 0.0;
#pragma unroll 1
            for (int k = 0; k < FT_N; k++) t += C[i][k] * B[k][j];
            A[i][j] = t;
        }
#pragma unroll 1
    for (int i = 0; i < FT_N; i++)
#pragma unroll 1
        for (int j = 0; j < FT_N; j++) {
            double t = 0.0;
#pragma unroll 1
            for (int k = 0; k < FT_N; k++) t += A[i][k] * C[j][k];
            B[i][j] = t;
        }
    // derivatives (srcs/laplacian.hpp:127-213): differences of S = B and of C
    auto S = [&](int i, int j) -> double { return (i == FT_N || j == FT_N) ? 0.0 : B[i][j]; };
    auto T = [&](int i, int j) -> double { return (i == FT_N || j == FT_N) ? 0.0 : C[i][j]; };
#pragma unroll 1
    for (int a = 0; a < FT_E; a++) {
        const int ka = map[FT_EK[a]], la = map[FT_EL[a]];
        const double s = S(ka, ka) + S(la, la) - 2.0 * S(ka, la);
        const double t = T(ka, ka) + T(la, la) - 2.0 * T(ka, la);
        const double xa = Xi[a] * Xi[a];
        const double xas = xa * s;
        dphi[a] = -xas;
        H[a][a] = 2.0 * xas * (Xi[a] - xa * t);
#pragma unroll 1
        for (int b = a + 1; b < FT_E; b++) {
            const int kb = map[FT_EK[b]], lb = map[FT_EL[b]];
            const double s2 = S(ka, kb) + S(la, lb) - S(ka, lb) - S(la, kb);
            const double t2 = T(ka, kb) + T(la, lb) - T(ka, lb) - T(la, kb);
            H[a][b] = -2.0 * xa * (Xi[b] * Xi[b]) * s2 * t2;
        }
    }
}

#endif

// ------------------------------------------------------------------ sector draw
struct table_ref {
    const void* q;              // cut thresholds (w in the working precision where FT_CUT is 0)
    const void* Jr;             // Jr in the working precision (FT_CUT 0 only)
    const void* ri;             // 1/r in FP64, or its two-float high parts
    const float* rl;            // two-float low parts of 1/r (mixed)
    const u32* meta;
    const unsigned char* gm;    // global copy (FP64 sections for exact re-checks)
};

#if FT_BATCH
// The batch kernels' current work item and its instance's table (global copy), written
// by the block's first thread between items and read where they are used, so that
// neither is held in registers across the per-sample code.
__shared__ unsigned long long s_batch_item;
__shared__ const unsigned char* s_batch_tab;
#define TABLE_GM(t) s_batch_tab
#define FT_EXACT_TABLE(t) ((t).gm ? (t).gm : s_batch_tab)
// first word of an FP64-pass queue entry: item << 28 | lane << 18 | offset of the
// sample in the lane's chunk (the other four hold the sample's stream state)
#define BQ_ITEM_SHIFT 28
#define BQ_LANE_SHIFT 18
#else
#define TABLE_GM(t) ((t).gm)
#define FT_EXACT_TABLE(t) ((t).gm)
#endif

// The reference's comparison, exactly (srcs/tropical_sampling.hpp:468-501: FP64 running
// sums of Jr/r in ascending edge order, the first above u * Jr(gamma), else the last
// edge): used when a threshold comparison cannot decide.  Out of line: it runs for a
// few steps per 1e4 samples at most.
static __device__ __noinline__ int exact_cut(u64 x, u32 sub, const unsigned char* __restrict__ gm)
{
    const double* w64 = (const double*)(gm + T_W64);
    const double* Jr64 = (const double*)(gm + T_JR64);
    const double R = u01(x) * Jr64[sub];
    double TT = 0.0;
    int cut = 0;
    for (int c = 0; c < FT_E; c++) {
        if ((sub >> c) & 1u) {
            TT += w64[sub ^ (1u << c)];
            cut = c;
            if (TT > R) break;
        }
    }
    return cut;
}

#if FT_CUT
// The cut of a subgraph of n edges for the draw x, h = x >> 32: the first edge whose running
// sum T_k = sum_{k' <= k} Jr/r (its edges in ascending order) exceeds u Jr.  The host
// stores per edge floor(2^28 T_k / Jr) << 4 | edge number, so the answer is the first
// entry above h, found by a binary search of ceil(log2 n) dependent shared-memory reads,
// the same for every lane (all lanes have subgraphs of n edges), instead of a scan whose
// trips are those of the warp's slowest lane (up to n of them).  Thresholds and h are
// exact to one unit of 2^-28: a probe within 18 of h does not decide, `unsure` is set and
// the caller repeats the step in FP64 (exact_cut).  The two thresholds that bound the
// answer are always among the probes.
static __device__ __forceinline__ int find_cut(u32 h, u32 sub, u32 meta, const table_ref& t, int n, bool& unsure)
{
    if (n == 1) return __ffs(sub) - 1;
    const u32* q = (const u32*)t.q + META_OFF(meta);
    int lo = 0;
#pragma unroll
    for (int m = n; m > 1;) {   // the answer is among entries lo .. lo + m - 1
        const int half = m / 2;
        const u32 e = q[lo + half - 1];
        unsure |= h - e + 18u <= 36u;
        lo += h >= e ? half : 0;
        m -= half;
    }
    return (int)(q[lo] & 15u);
}
#elif FT_PREC == 1
// Tables in global memory: the running sums in FP32 with a rigorous margin (|T32 - T64| <=
// (2E) 2^-24 Jr, |R32 - R64| <= 4 2^-24 Jr), up to the first sure decision.
static __device__ __forceinline__ int scan_cut(u64 x, u32 sub, const table_ref& t, bool& unsure)
{
    const float* w = (const float*)t.q;
    const float JJr = ((const float*)t.Jr)[sub];
    const float Rf = (float)(u32)(x >> 40) * 0x1.0p-24f * JJr;
    const float margin = (float)(2 * FT_E + 8) * 0x1.0p-24f * JJr;
    float T = 0.0f;
    int cut = 0;
    for (u32 left = sub; left != 0u; left &= left - 1u) {
        cut = __ffs(left) - 1;
        T += w[sub ^ (1u << cut)];
        const float d = T - Rf;
        if (d > margin) break;
        if (d >= -margin) unsure = true;
    }
    return cut;
}
#endif

#if FT_PREC == 0
#if FT_CUT
static __device__ __noinline__ int find_cut_call(u32 h, u32 sub, u32 meta, const table_ref& t, int n, bool& unsure)
{
    return find_cut(h, sub, meta, t, n, unsure);
}
#endif
template <bool COLD>
static __device__ __forceinline__ void draw_sector64(xo& g, const table_ref& t, const unsigned char* gm,
                                                     double Jr_full, double* X, double& F, double& Gv,
                                                     unsigned char* ord)
{
    const double* ri = (const double*)t.ri;
    u32 sub = FT_FULL, meta = t.meta[FT_FULL];
    double XX = 1.0;
    F = 1.0;
    Gv = 0.0;
#if !FT_CUT
    const double* w = (const double*)t.q;
    const double* Jr = (const double*)t.Jr;
    double JJr = Jr_full;
#endif
#pragma unroll
    for (int j = 0; j < FT_E; j++) {
        const u64 x = g.next();
#if FT_CUT
        bool unsure = false;
        int e = COLD ? find_cut_call((u32)(x >> 32), sub, meta, t, FT_E - j, unsure)
                     : find_cut((u32)(x >> 32), sub, meta, t, FT_E - j, unsure);
        if (unsure) e = exact_cut(x, sub, gm);
        sub ^= 1u << e;
#else
        const double R = u01(x) * JJr;
        double T = 0.0;
        int e = 0;
        // the subgraph's edges in ascending order (its set bits) until the running sum
        // passes R, else the last one
        for (u32 left = sub; left != 0u; left &= left - 1u) {
            e = __ffs(left) - 1;
            T += w[sub ^ (1u << e)];
            if (T > R) break;
        }
        sub ^= 1u << e;
        JJr = Jr[sub];
#endif
        const double rinv = ri[sub];
        const u32 m = t.meta[sub];
        if (META_MM(meta) && !META_MM(m)) Gv = XX;
#pragma unroll
        for (int k = 0; k < FT_E; k++)
            if (k == e) X[k] = XX;
        if (META_L(m) < META_L(meta)) F *= XX;
        meta = m;
        if (FT_RECORD) ord[j] = (unsigned char)e;
        if (j < FT_E - 1) XX *= fn64<COLD>::pow1mu(g.next(), rinv);
    }
}

// ------------------------------------------------------------------ integrand, FP64
// powers of the undeformed integrand out of the fixed-point ones' reach, as the reference takes them
// (srcs/feynman_integral.hpp:246-262): out = R per eps order, false when dropped
static __device__ __noinline__ bool undeformed_slow(double psi, double pxi, double D, double W, double IGtr, double* out)
{
    double R = IGtr * pow(psi, -D / 2.);
    if (!isfinite(R)) return false;
#if !FT_ONLY_PSI
    R *= pow(pxi, -W);
    if (!isfinite(R)) return false;
#endif
    out[0] = R;
    if (FT_K > 1) {
        const double ef = log(psi) - FT_LOOPS * log(pxi);
        for (int j = 1; j < FT_K; j++) {
            R *= ef / (double)j;
            out[j] = R;
        }
    }
    return true;
}
static __device__ __noinline__ double scale_slow(double psi_tr, double Gv, double D, double W, double norm)
{
    return pow(pow(psi_tr, -D / 2.) * pow(1.0 / Gv, W), norm);
}
#if FT_MODE == 1
static __device__ __noinline__ cx<double> powers_slow(cx<double> psi, cx<double> v, double D, double W, cx<double>& lp,
                                                      cx<double>& lv)
{
    lp = clog_(psi);
    lv = clog_(v);
    return cpow_(psi, -D / 2.) * cpow_(v, -W);
}
// The derivatives by the reference's route of the sample drawn just before g, for an edge
// whose ends float together.  Differences of the potentials' products cancel there to
// eps / x_e^2: below x_e = 1e-8 the phases are rounding noise, and the last bit of X decides
// them.  So the sample is drawn again with the general functions, which keeps the values
// that the plain FP64 form gives: with X from pow_1mu a single sample of 3e6 moved double
// box integrals by up to 5e-7 (6 of 40 kinematics by more than 1e-9), with this by 1e-12.
static __device__ __noinline__ bool derivatives_slow(xo g, const unsigned char* gm, const double* prm,
                                                     const double (*G)[FT_N], double* dphi, double (*H)[FT_E])
{
    bool cancel = false;
    for (int e = 0; e < FT_E; e++) {
        const int k = FT_EK[e], l = FT_EL[e];
        if (k == FT_V - 1) continue;
        const double big = G[k][k] + G[l][l], t = big - 2.0 * G[k][l];
        cancel |= !(t > 1e-7 * big);
    }
    if (!cancel) return false;
    const double* ri = (const double*)(gm + T_RI64);
    const u32* meta = (const u32*)(gm + T_META);
    double X[FT_E], Xi[FT_E];
    double XX = 1.0, F = 1.0, Gv = 0.0;
    u32 sub = FT_FULL;
    rewind(g, 2 * FT_E - 1);
#pragma unroll 1
    for (int j = 0; j < FT_E; j++) {
        const int e = exact_cut(g.next(), sub, gm);
        const u32 m0 = meta[sub];
        sub ^= 1u << e;
        const u32 m = meta[sub];
        if (META_MM(m0) && !META_MM(m)) Gv = XX;
        X[e] = XX;
        if (META_L(m) < META_L(m0)) F *= XX;
        if (j < FT_E - 1) XX *= pow(1.0 - u01(g.next()), ri[sub]);
    }
    const double tgt = pow(F, -prm[P_D] / 2.) * pow(F / (Gv * F), prm[P_W]);
    const double scale = pow(tgt, prm[P_NORM]);
    for (int e = 0; e < FT_E; e++) {
        X[e] *= scale;
        Xi[e] = 1.0 / X[e];
    }
    robust_derivatives(X, Xi, prm, dphi, H);
    return true;
}
#endif

// X: unnormalised sector point, psi_tr and Gv = xi_tr / psi_tr there; returns R per eps
// order, false when dropped.  `robust` reports that the complete-pivoting LU or the
// reference's route to the derivatives was needed.  g: the stream behind the sample's draws.
template <bool COLD>
static __device__ __forceinline__ bool integrand64(const double* prm, double* X, double psi_tr, double Gv,
                                                   const xo& g, const unsigned char* gm, cx<double>* out,
                                                   bool& robust)
{
    const double D = prm[P_D], W = prm[P_W], IGtr = prm[P_IGTR];
    // normalise so that psi_tr^(-D/2) (psi_tr/xi_tr)^W = 1 (srcs/feynman_integral.hpp:201-204)
    double scale;
    {
        const log2_parts lf = fn64<COLD>::log2(psi_tr), lg = fn64<COLD>::log2(Gv);
        if (normal_positive(psi_tr) && normal_positive(Gv) &&
            in_reach(lf, min(log2_limit(0.5 * D), log2_limit(prm[P_NORM_F]))) &&
            in_reach(lg, min(log2_limit(W), log2_limit(prm[P_NORM_G])))) {
            scale = fn64<COLD>::power(prm[P_NORM_F], lf, prm[P_NORM_G], lg);
        } else {
            scale = scale_slow(psi_tr, Gv, D, W, prm[P_NORM]);
        }
    }
    double Xi[FT_E];
    double Xprod = 1.0;
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        X[e] *= scale;
        Xi[e] = rcp64(X[e]);
        Xprod = e == 0 ? X[e] : Xprod * X[e];
    }
    // the real reduced Laplacian in conductance form (every value positive)
    double a[FT_N][FT_N], d[FT_N], id[FT_N];
    {
        double c[FT_N][FT_N], g[FT_N];
#pragma unroll
        for (int e = 0; e < FT_E; e++) {
            const int k = FT_EK[e], l = FT_EL[e];
            double& slot = (k == FT_V - 1) ? g[l] : c[l][k];
            slot = first_in_slot(e) ? Xi[e] : slot + Xi[e];
        }
#pragma unroll
        for (int k = 0; k < FT_N; k++) {
            double dk = 0.0;
            bool any = NZG(k);
            if (any) dk = g[k];
#pragma unroll
            for (int j = k + 1; j < FT_N; j++)
                if (NZC(k, j)) {
                    dk = any ? dk + c[k][j] : c[k][j];
                    any = true;
                }
            d[k] = dk;
            id[k] = rcp64(dk);
#pragma unroll
            for (int i = k + 1; i < FT_N; i++)
                if (NZC(k, i)) a[k][i] = c[k][i] * id[k];
#pragma unroll
            for (int i = k + 1; i < FT_N; i++) {
                if (!NZC(k, i)) continue;
                if (NZG(k)) g[i] = ADDS_G(k, i) ? fma(a[k][i], g[k], g[i]) : a[k][i] * g[k];
#pragma unroll
                for (int j = i + 1; j < FT_N; j++)
                    if (NZC(k, j)) c[i][j] = ADDS_C(k, i, j) ? fma(a[k][i], c[k][j], c[i][j]) : a[k][i] * c[k][j];
            }
        }
    }
    robust = false;
#if FT_MODE == 0
    double det = d[0];
#pragma unroll
    for (int k = 1; k < FT_N; k++) det *= d[k];
    const double psi = det * Xprod;
    double pxi = 1.0;
#if !FT_ONLY_PSI
    // V = -sum_r sigma_r q_r^T L^-1 q_r + sum_e m2_e X_e
    pxi = 0.0;
#pragma unroll
    for (int r = 0; r < FT_RANK; r++) {
        double y[FT_N], s = 0.0;
#pragma unroll
        for (int i = FT_Q0; i < FT_N; i++) {
            double yi = prm[P_Q + r * FT_N + i];
#pragma unroll
            for (int k = FT_Q0; k < i; k++)
                if (NZC(k, i)) yi = fma(a[k][i], y[k], yi);
            y[i] = yi;
            s = i == FT_Q0 ? yi * yi * id[i] : fma(yi * yi, id[i], s);
        }
        pxi = r == 0 ? -(prm[P_SIG + r] * s) : fma(-prm[P_SIG + r], s, pxi);
    }
#pragma unroll
    for (int e = 0; e < FT_E; e++) pxi = fma(prm[P_M2 + e], X[e], pxi);
#endif
    const log2_parts lp = fn64<COLD>::log2(psi), lv = fn64<COLD>::log2(pxi);
    if (!normal_positive(psi) || !normal_positive(pxi) || !in_reach(lp, log2_limit(0.5 * D)) ||
        !in_reach(lv, log2_limit(W))) {
        double R[FT_K];
        const bool ok = undeformed_slow(psi, pxi, D, W, IGtr, R);
#pragma unroll
        for (int j = 0; j < FT_K; j++) out[j] = cmk(R[j], 0.0);
        return ok;
    }
#if FT_ONLY_PSI
    const double v = IGtr * fn64<COLD>::power(-0.5 * D, lp, 0.0, lv);
    if (!finite_(v)) return false;
    out[0] = cmk(v, 0.0);
#else
    double v = IGtr * fn64<COLD>::power(-0.5 * D, lp, -W, lv);
    if (!finite_(v)) return false;
    out[0] = cmk(v, 0.0);
    if (FT_K > 1) {
        const double ef = LN2_D * log2_difference(lp, lv, FT_LOOPS);
#pragma unroll
        for (int j = 1; j < FT_K; j++) {
            v *= ef * (1.0 / (double)j);
            out[j] = cmk(v, 0.0);
        }
    }
#endif
    return true;
#else
    const double kappa = prm[P_DEF];
    // N = M^-1 (entrywise non-negative), G = L^-1 = N diag(1/d) N^T
    double Nm[FT_N][FT_N], Nd[FT_N][FT_N];
#pragma unroll
    for (int i = FT_N - 1; i >= 0; i--) {
#pragma unroll
        for (int j = i + 1; j < FT_N; j++) {
            if (!NZM(i, j)) continue;
            double s = 0.0;
            bool any = false;
            if (NZC(i, j)) {
                s = a[i][j];
                any = true;
            }
#pragma unroll
            for (int k = i + 1; k < j; k++)
                if (NZC(i, k) && NZM(k, j)) {
                    s = any ? fma(a[i][k], Nm[k][j], s) : a[i][k] * Nm[k][j];
                    any = true;
                }
            Nm[i][j] = s;
            Nd[i][j] = s * id[j];
        }
    }
    double G[FT_N][FT_N];
#pragma unroll
    for (int i = 0; i < FT_N; i++)
#pragma unroll
        for (int j = i; j < FT_N; j++) {
            double s = 0.0;
            bool any = false;
            if (i == j || NZM(i, j)) {
                s = i == j ? id[j] : Nd[i][j];
                any = true;
            }
#pragma unroll
            for (int k = j + 1; k < FT_N; k++)
                if (NZM(i, k) && NZM(j, k)) {
                    s = any ? fma(Nm[i][k], Nd[j][k], s) : Nm[i][k] * Nd[j][k];
                    any = true;
                }
            G[i][j] = s;
            G[j][i] = s;
        }
    // Per edge its power of two D ~ X^1/2 and w = D / X^2; hb = w h_r . b_e with h_r = L^-1 q_r,
    // b_e = e_k - e_l (ground row zero), so that
    //   s_ab = -2 kappa sum_r sigma_r hb_a hb_b,  t_ab = b_a^T G b_b
    // give kappa D_a D_b H_ab = s_ab t_ab (the diagonal s_aa (t_aa - X_a)) and
    // theta_a = kappa m2_a + s_aa X_a^2 / (2 D_a^2) (srcs/laplacian.hpp:102-215)
    int ex[FT_E];   // D = 2^ex
    double hb[FT_RANK][FT_E];
    {
        double w[FT_E];
#pragma unroll
        for (int e = 0; e < FT_E; e++) {
            ex[e] = max(-500, min(500, (exponent_of(X[e]) - 1023) >> 1));
            w[e] = Xi[e] * Xi[e] * pow2_of(ex[e]);
        }
#pragma unroll
        for (int r = 0; r < FT_RANK; r++) {
            double h[FT_N];
#pragma unroll
            for (int i = 0; i < FT_N; i++) {
                double s = 0.0;
#pragma unroll
                for (int j = FT_Q0; j < FT_N; j++) {
                    const double q = prm[P_Q + r * FT_N + j];
                    s = j == FT_Q0 ? G[i][j] * q : fma(G[i][j], q, s);
                }
                h[i] = s;
            }
#pragma unroll
            for (int e = 0; e < FT_E; e++) {
                const int k = FT_EK[e], l = FT_EL[e];
                hb[r][e] = ((k == FT_V - 1) ? -h[l] : h[k] - h[l]) * w[e];
            }
        }
    }
    double A[FT_E][FT_E];   // kappa D H D, upper triangle
    double theta[FT_E];
    bool cancel = false;
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const int ke = FT_EK[e], le = FT_EL[e];
        double w[FT_N];   // row e of (edge incidence) L^-1
#pragma unroll
        for (int v = 0; v < FT_N; v++)
            w[v] = ke == FT_V - 1 ? -G[le][v] : (le == FT_V - 1 ? G[ke][v] : G[ke][v] - G[le][v]);
        auto wd = [&](int k, int l) -> double { return k == FT_V - 1 ? -w[l] : (l == FT_V - 1 ? w[k] : w[k] - w[l]); };
        double sg[FT_RANK];
        double s = 0.0;
#pragma unroll
        for (int r = 0; r < FT_RANK; r++) {
            sg[r] = (-2.0 * kappa * prm[P_SIG + r]) * hb[r][e];
            s = r == 0 ? sg[r] * hb[r][e] : fma(sg[r], hb[r][e], s);
        }
        const double t = wd(ke, le);
        // an edge whose ends may float together: its resistance difference cancels (t below
        // 2^-21 of the entries it comes from, by their exponents; derivatives_slow tests for 1e-7)
        if (ke != FT_V - 1) {
            const int big = max(exponent_of(G[ke][ke]), exponent_of(G[le][le]));
            cancel |= hi_word(t) < 0 || exponent_of(t) < big - 20;
        }
        A[e][e] = s * (t - X[e]);
        theta[e] = fma(s * (X[e] * X[e]), pow2_of(-2 * ex[e] - 1), kappa * prm[P_M2 + e]);
#pragma unroll
        for (int f = e + 1; f < FT_E; f++) {
            double s2 = 0.0;
#pragma unroll
            for (int r = 0; r < FT_RANK; r++) s2 = r == 0 ? sg[r] * hb[r][f] : fma(sg[r], hb[r][f], s2);
            A[e][f] = s2 * wd(FT_EK[f], FT_EL[f]);
        }
    }
    if (cancel) {
        double dphi[FT_E], H[FT_E][FT_E], Gm[FT_N][FT_N];   // Gm: so that G stays in registers
#pragma unroll
        for (int k = 0; k < FT_N; k++)
#pragma unroll
            for (int l = 0; l < FT_N; l++) Gm[k][l] = G[k][l];
        if (derivatives_slow(g, gm, prm, Gm, dphi, H)) {
            robust = true;
#pragma unroll
            for (int e = 0; e < FT_E; e++) {
                theta[e] = (dphi[e] + prm[P_M2 + e]) * kappa;
#pragma unroll
                for (int f = e; f < FT_E; f++) A[e][f] = kappa * H[e][f] * pow2_of(ex[e]) * pow2_of(ex[f]);
            }
        }
    }
    // deformation x -> x exp(i theta), theta = -lambda (d(phi/psi)/dx + m^2)
    // (srcs/feynman_integral.hpp:290-310)
    cx<double> cy[FT_E];
    double xnu = 0.0;
    cx<double> cXprod = cmk(1.0, 0.0), cV = cmk(0.0, 0.0);
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        double sn, cs;
        fn64<COLD>::sincos(theta[e], sn, cs);
        const cx<double> cX = cmk(X[e] * cs, X[e] * sn);
        cy[e] = cmk(Xi[e] * cs, -Xi[e] * sn);   // 1 / cX
        const double m2 = prm[P_M2 + e];
        xnu = e == 0 ? prm[P_NU] * theta[0] : fma(prm[P_NU + e], theta[e], xnu);
        cXprod = e == 0 ? cX : cXprod * cX;
        cV = e == 0 ? m2 * cX : cmk(fma(m2, cX.re, cV.re), fma(m2, cX.im, cV.im));
    }
    // the deformed Laplacian, its determinant and -tr(L^-1 P~): U the unit lower triangular
    // map of the forward substitution on the external rows, sum_i (u_i^T P~ u_i) / d_i
    cx<double> cdet = cmk(1.0, 0.0), cphi = cmk(0.0, 0.0);
    bool growth = true;
    {
        cx<double> c[FT_N][FT_N], g[FT_N], ca[FT_N][FT_N], ci[FT_N];
#pragma unroll
        for (int e = 0; e < FT_E; e++) {
            const int k = FT_EK[e], l = FT_EL[e];
            cx<double>& slot = (k == FT_V - 1) ? g[l] : c[l][k];
            slot = first_in_slot(e) ? cy[e] : slot + cy[e];
        }
        auto expo = [](cx<double> z) -> int { return max(exponent_of(z.re), exponent_of(z.im)); };
        auto cfma = [](cx<double> x, cx<double> y, cx<double> z) -> cx<double> {
            return cmk(fma(x.re, y.re, fma(-x.im, y.im, z.re)), fma(x.re, y.im, fma(x.im, y.re, z.im)));
        };
#pragma unroll
        for (int k = 0; k < FT_N; k++) {
            cx<double> dk = cmk(0.0, 0.0);
            int big = 0;
            bool any = NZG(k);
            if (any) {
                dk = g[k];
                big = expo(g[k]);
            }
#pragma unroll
            for (int j = k + 1; j < FT_N; j++) {
                if (!NZC(k, j)) continue;
                dk = any ? dk + c[k][j] : c[k][j];
                big = max(big, expo(c[k][j]));
                any = true;
            }
            growth &= expo(dk) > big - 26;   // a pivot above about 1e-8 of its row, by the exponents
            cdet = k == 0 ? dk : cdet * dk;
            ci[k] = fn64<COLD>::cinv(dk);
#pragma unroll
            for (int i = k + 1; i < FT_N; i++)
                if (NZC(k, i)) ca[k][i] = c[k][i] * ci[k];
#pragma unroll
            for (int i = k + 1; i < FT_N; i++) {
                if (!NZC(k, i)) continue;
                if (NZG(k)) g[i] = ADDS_G(k, i) ? cfma(ca[k][i], g[k], g[i]) : ca[k][i] * g[k];
#pragma unroll
                for (int j = i + 1; j < FT_N; j++)
                    if (NZC(k, j)) c[i][j] = ADDS_C(k, i, j) ? cfma(ca[k][i], c[k][j], c[i][j]) : ca[k][i] * c[k][j];
            }
        }
#if FT_NE > 0
        cx<double> U[FT_NE][FT_NE];
#pragma unroll
        for (int ii = 0; ii < FT_NE; ii++) {
            const int i = FT_Q0 + ii;
#pragma unroll
            for (int jj = 0; jj < ii; jj++) {
                const int j = FT_Q0 + jj;
                if (!NZM(j, i)) continue;
                cx<double> u = cmk(0.0, 0.0);
                bool any = false;
                if (NZC(j, i)) {
                    u = ca[j][i];
                    any = true;
                }
#pragma unroll
                for (int kk = jj + 1; kk < ii; kk++) {
                    const int k = FT_Q0 + kk;
                    if (!NZC(k, i) || !NZM(j, k)) continue;
                    u = any ? cfma(ca[k][i], U[kk][jj], u) : ca[k][i] * U[kk][jj];
                    any = true;
                }
                U[ii][jj] = u;
            }
            cx<double> Q = cmk(prm[PT_AT(ii, ii)], 0.0);
            bool real = true;
#pragma unroll
            for (int jj = 0; jj < ii; jj++) {
                if (!NZM(FT_Q0 + jj, i)) continue;
                cx<double> w = prm[PT_AT(jj, jj)] * U[ii][jj];
#pragma unroll
                for (int kk = jj + 1; kk < ii; kk++) {
                    if (!NZM(FT_Q0 + kk, i)) continue;
                    const double p = prm[PT_AT(jj, kk)];
                    w = cmk(fma(p, U[ii][kk].re, w.re), fma(p, U[ii][kk].im, w.im));
                }
                w.re += prm[PT_AT(jj, ii)];
                Q = cfma(U[ii][jj], w, Q);
                real = false;
            }
            cphi = real ? cmk(fma(-Q.re, ci[i].re, cphi.re), fma(-Q.re, ci[i].im, cphi.im))
                        : cfma(cmk(-Q.re, -Q.im), ci[i], cphi);
        }
#endif
    }
    if (!growth) {
        robust = true;
        robust_complex(cy, prm, cdet, cphi);
    }
    const cx<double> cPsi = cXprod * cdet;
    cV = cV + cphi;
    // det(I + i kappa H X) = det(D^2/X + i kappa D H D) prod X/D^2: the real part is positive
    // and diagonal, so the symmetric elimination needs no pivoting (srcs/feynman_integral.hpp:312-320)
    cx<double> detJ = cmk(1.0, 0.0);
    {
        cx<double> J[FT_E][FT_E];
#pragma unroll
        for (int e = 0; e < FT_E; e++)
#pragma unroll
            for (int f = e; f < FT_E; f++) J[e][f] = cmk(e == f ? pow2_of(2 * ex[e]) * Xi[e] : 0.0, A[e][f]);
#pragma unroll
        for (int k = 0; k < FT_E; k++) {
            const cx<double> piv = J[k][k];
            detJ = k == 0 ? piv : detJ * piv;
            if (k == FT_E - 1) continue;
            const cx<double> inv = fn64<COLD>::cinv(piv);
#pragma unroll
            for (int i = k + 1; i < FT_E; i++) {
                // the first row's entries have no real part
                const cx<double> f = k == 0 ? cmk(-J[0][i].im * inv.im, J[0][i].im * inv.re) : J[k][i] * inv;
#pragma unroll
                for (int j = i; j < FT_E; j++) {
                    const cx<double> q = J[k][j];
                    if (k == 0)
                        J[i][j] = cmk(fma(f.im, q.im, J[i][j].re), fma(-f.re, q.im, J[i][j].im));
                    else
                        J[i][j] = cmk(fma(-f.re, q.re, fma(f.im, q.im, J[i][j].re)),
                                      fma(-f.re, q.im, fma(-f.im, q.re, J[i][j].im)));
                }
            }
        }
    }
    {
        int sum = 0;
#pragma unroll
        for (int e = 0; e < FT_E; e++) sum += ex[e];
        sum = max(-1000, min(1000, sum));
        detJ = (Xprod * pow2_of(-sum) * pow2_of(-sum)) * detJ;   // prod X / D^2
    }
    // cR = IGtr cPsi^(-D/2) cV^(-W) det J e^(i nu . theta)
    cx<double> ef, pw;   // log cPsi - L log cV, the powers
    const double np = fma(cPsi.re, cPsi.re, cPsi.im * cPsi.im), nv = fma(cV.re, cV.re, cV.im * cV.im);
    const log2_parts a2 = fn64<COLD>::log2(np), b2 = fn64<COLD>::log2(nv);
    if (normal_positive(np) && normal_positive(nv) && in_reach(a2, log2_limit(0.25 * D)) &&
        in_reach(b2, log2_limit(0.5 * W))) {
        const double ap = fn64<COLD>::arg(cPsi.re, cPsi.im), av = fn64<COLD>::arg(cV.re, cV.im);
        ef = cmk(0.5 * LN2_D * log2_difference(a2, b2, FT_LOOPS), fma(-(double)FT_LOOPS, av, ap));
        const double m = fn64<COLD>::power(-0.25 * D, a2, -0.5 * W, b2);
        double sn, cs;
        fn64<COLD>::sincos(fma(-0.5 * D, ap, -W * av), sn, cs);
        pw = cmk(m * cs, m * sn);
    } else {
        cx<double> lp, lv;
        pw = powers_slow(cPsi, cV, D, W, lp, lv);
        ef = cmk(lp.re - FT_LOOPS * lv.re, lp.im - FT_LOOPS * lv.im);
    }
    double sn, cs;
    fn64<COLD>::sincos(xnu, sn, cs);
    cx<double> cR = (IGtr * pw) * (detJ * cmk(cs, sn));
    if (!finite_(cR.re) || !finite_(cR.im)) return false;
    out[0] = cR;
    if (FT_K > 1) {
#pragma unroll
        for (int j = 1; j < FT_K; j++) {
            cR = cR * ((1.0 / (double)j) * ef);
            out[j] = cR;
        }
    }
    return true;
#endif
}

#else
// ------------------------------------------------------------------ mixed form: FP32 values and pairs
// Pairs of FP32 values use the paired instructions (add, mul, fma .f32x2, each component
// rounded as the scalar operation): the same rate per result, half the issue slots and
// half the instruction fetches, which bound the mixed kernels.  The undeformed form
// evaluates two consecutive samples of a thread's range side by side (one component per
// sample); the deformed form, whose live state would not fit the registers twice, one
// sample, with its exponentials, logarithms and phases for two edges at a time.
typedef float2 fv;

static __device__ __forceinline__ fv fv_of(float a) { return make_float2(a, a); }
static __device__ __forceinline__ fv operator+(fv a, fv b) { return __fadd2_rn(a, b); }
static __device__ __forceinline__ fv operator*(fv a, fv b) { return __fmul2_rn(a, b); }
static __device__ __forceinline__ fv fma_(fv a, fv b, fv c) { return __ffma2_rn(a, b, c); }
static __device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
static __device__ __forceinline__ fv operator-(fv a, fv b) { return __ffma2_rn(b, fv_of(-1.0f), a); }
static __device__ __forceinline__ fv operator-(fv a) { return __fmul2_rn(a, fv_of(-1.0f)); }
static __device__ __forceinline__ fv mul_(fv a, fv b) { return a * b; }
static __device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }   // never contracted
static __device__ __forceinline__ fv abs_(fv a) { return make_float2(fabsf(a.x), fabsf(a.y)); }
static __device__ __forceinline__ float abs_(float a) { return fabsf(a); }
static __device__ __forceinline__ void set_all(fv& r, float a) { r = fv_of(a); }
static __device__ __forceinline__ void set_all(float& r, float a) { r = a; }
template <class V>
static __device__ __forceinline__ V all_of(float a)
{
    V r;
    set_all(r, a);
    return r;
}
// reciprocal to an ulp (the approximate instruction), for values that a Newton step or the
// two-float reciprocal refines
static __device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
static __device__ __forceinline__ fv rcp_fast(fv x) { return make_float2(rcp_fast(x.x), rcp_fast(x.y)); }
template <class V>
static __device__ __forceinline__ V rcp_newton(V x)
{
    const V r = rcp_fast(x);
    return fma_(r, fma_(x, -r, all_of<V>(1.0f)), r);
}

// Two-float numbers hi + lo (about 48 significant bits) from error-free transformations
// (Knuth's two-sum, Dekker's fast two-sum, the FMA two-product).  They run on the FP32
// pipe, which is 64x wider than the FP64 pipe on this GPU.
template <class V>
struct tf {
    V hi, lo;
};
typedef tf<float> sf;
typedef tf<fv> df;
template <class V>
static __device__ __forceinline__ tf<V> tf_mk(V h, V l)
{
    tf<V> r;
    r.hi = h;
    r.lo = l;
    return r;
}
template <class V>
static __device__ __forceinline__ tf<V> tf_zero()
{
    return tf_mk(all_of<V>(0.0f), all_of<V>(0.0f));
}
template <class V>
static __device__ __forceinline__ tf<V> two_sum(V a, V b)
{
    const V s = a + b, bb = s - a;
    return tf_mk(s, (a - (s - bb)) + (b - bb));
}
// |a| >= |b| or a = 0
template <class V>
static __device__ __forceinline__ tf<V> fast_two_sum(V a, V b)
{
    const V s = a + b;
    return tf_mk(s, b - (s - a));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_norm(tf<V> x)
{
    return fast_two_sum(x.hi, x.lo);
}
// Sums whose low part is not renormalised (`_n`): it stays within a few ulps of the
// terms' high parts, so further sums lose nothing; chains renormalise once, at their
// end, before the value is multiplied or inverted.
template <class V>
static __device__ __forceinline__ tf<V> tf_add_n(tf<V> x, tf<V> y)
{
    const tf<V> s = two_sum(x.hi, y.hi);
    return tf_mk(s.hi, s.lo + (x.lo + y.lo));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_sub_n(tf<V> x, tf<V> y)
{
    const V s = x.hi - y.hi, bb = s - x.hi;
    const V e = (x.hi - (s - bb)) - (y.hi + bb);
    return tf_mk(s, e + (x.lo - y.lo));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_add(tf<V> x, tf<V> y)
{
    return tf_norm(tf_add_n(x, y));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_sub(tf<V> x, tf<V> y)
{
    return tf_norm(tf_sub_n(x, y));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_neg(tf<V> x)
{
    return tf_mk(-x.hi, -x.lo);
}
// A product cannot cancel: its low part stays within ~1.5 ulp of the high one, which
// every consumer handles, so it is returned without renormalisation.
template <class V>
static __device__ __forceinline__ tf<V> tf_mul(tf<V> x, tf<V> y)
{
    const V p = mul_(x.hi, y.hi);
    V e = fma_(x.hi, y.hi, -p);
    e = fma_(x.hi, y.lo, e);
    return tf_mk(p, fma_(x.lo, y.hi, e));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_fma_n(tf<V> x, tf<V> y, tf<V> z)
{
    const tf<V> p = tf_mul(x, y);
    const tf<V> s = two_sum(p.hi, z.hi);
    return tf_mk(s.hi, s.lo + (p.lo + z.lo));
}
// x s, s a float
template <class V>
static __device__ __forceinline__ tf<V> tf_mulf(tf<V> x, V s)
{
    const V p = mul_(x.hi, s);
    return tf_mk(p, fma_(x.lo, s, fma_(x.hi, s, -p)));
}
template <class V>
static __device__ __forceinline__ tf<V> tf_addf_n(tf<V> x, V y)
{
    const tf<V> s = two_sum(x.hi, y);
    return tf_mk(s.hi, s.lo + x.lo);
}
template <class V>
static __device__ __forceinline__ tf<V> tf_inv(tf<V> x)
{
    // one Newton step from the FP32 reciprocal r: 1/x = r (1 + e), e = 1 - x r exact to
    // 2^-47 by the FMA; |r e| stays within an ulp or two of r
    const V r = rcp_fast(x.hi), nr = -r;
    const V e = fma_(x.lo, nr, fma_(x.hi, nr, all_of<V>(1.0f)));
    return tf_mk(r, r * e);
}
template <class V>
static __device__ __forceinline__ V tf_f(tf<V> x)
{
    return x.hi + x.lo;
}
static __device__ __forceinline__ df pair_of(sf a, sf b) { return tf_mk(make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)); }
static __device__ __forceinline__ sf first_of(df a) { return tf_mk(a.hi.x, a.lo.x); }
static __device__ __forceinline__ sf second_of(df a) { return tf_mk(a.hi.y, a.lo.y); }
// parameter i, stored as (hi, hi, lo, lo)
static __device__ __forceinline__ sf prm_sf(const float4* pp, int i)
{
    const float4 v = pp[i];
    return tf_mk(v.x, v.z);
}
static __device__ __forceinline__ fv prm_fv(const float4* pp, int i) { return *(const float2*)(pp + i); }

// log(1 - u), u = (x >> 11) 2^-53, of two draws, to about 1e-12 absolute, with integer and FP32
// instructions only (64-bit conversions and FP64 would run on the FP64 pipe).
// Table-driven reduction after Tang (ACM TOMS 16, 1990): 1 - u = 2^kk M with M in [1, 2)
// held as two floats (46 fraction bits); c_i = 1 + (i + 1/2)/64 for the top 6 fraction
// bits i, r_i = fl(1/c_i) and -log r_i (two-float) from FT_LOGTAB; z = M r_i - 1 (|z| <
// 1/100) from exact products, log M = -log r_i + log1p(z) with log1p(z) = z - z^2/2 +
// z^3/3 - z^4/4 + z^5/5, the terms past z in FP32.
struct log_arg {
    float m, l, r, nh, nl, k;
};
static __device__ __forceinline__ log_arg log_split(u64 x)
{
    const u64 q = (~x & ~0x7ffull) + 0x800ull;   // (1 - u) 2^64, 0 for u = 0
    const int lz = __clzll((long long)q);
    const u64 mb = q << (lz & 63);
    const u32 hi = (u32)(mb >> 32) | 0x80000000u;
    log_arg a;
    a.m = __int_as_float((int)((hi >> 8) + 0x3f000000u));
    a.l = __int_as_float((int)((__funnelshift_r((u32)mb, hi, 17) & 0x7fffffu) | 0x4b000000u));
    const float4 t = FT_LOGTAB[(hi >> 25) & 63u];
    a.r = t.x;
    a.nh = t.y;
    a.nl = t.z;
    a.k = lz == 64 ? 0.0f : 8388608.0f - __int_as_float(0x4b000001 + lz);   // -1 - lz
    return a;
}
static __device__ FT_BIGFN df log1m_pair(u64 xa, u64 xb)
{
    const log_arg a = log_split(xa), b = log_split(xb);
    const fv m = make_float2(a.m, b.m), r = make_float2(a.r, b.r), kk = make_float2(a.k, b.k);
    const fv ml = (make_float2(a.l, b.l) - fv_of(8388608.0f)) * fv_of(0x1.0p-46f);
    // z = M r - 1: m r = p + e exactly, p - 1 exact (p within 1 % of 1)
    const fv p = m * r;
    const df z = fast_two_sum(p - fv_of(1.0f), fma_(ml, r, fma_(m, r, -p)));
    const fv zh = z.hi;
    const fv tail = zh * zh *
                    fma_(zh, fma_(zh, fma_(zh, fv_of(0.2f), fv_of(-0.25f)), fv_of(0.333333343f)), fv_of(-0.5f));
    // kk ln2 with ln2 in three parts (the first has 16 bits: the product is exact)
    const df s = fast_two_sum(kk * fv_of(0.693145751953125f), make_float2(a.nh, b.nh));
    const df t = two_sum(s.hi, zh);
    const fv lo = fma_(kk, fv_of(1.428606765330187e-06f), make_float2(a.nl, b.nl)) +
                  fma_(kk, fv_of(5.497923e-14f), z.lo + tail);
    return fast_two_sum(t.hi, (t.lo + s.lo) + lo);
}

// the draw of the step undecided by the thresholds, in FP64; g stands `back` draws behind it
static __device__ __noinline__ int exact_step(xo g, int back, u32 sub, const unsigned char* gm)
{
    rewind(g, back);
    return exact_cut(g.next(), sub, gm);
}

// The thread's scratch in shared memory, [slot][thread]: log X of edge e (part 0 hi, 1 lo),
// later overwritten by 1/X; with FT_SCRATCH 1 also the deformation angles, with 2 the
// upper triangle of kappa D H D: values that live across the long blocks of the
// deformed integrand and would otherwise be spilled to local memory, whose frames (256
// threads of 2 KB on every SM) are read back from L2.
#if FT_MODE == 0
typedef fv scr;
#else
typedef float scr;
#endif
#define SCR(slot) (((scr*)lxs)[(slot) * FT_BLOCK + threadIdx.x])
#define LX(e, p) SCR((e) * 2 + (p))
#define SCR_TH(e, p) SCR(2 * FT_E + (e) * 2 + (p))
#define SCR_H(a, b) SCR(4 * FT_E + (a) * FT_E - (a) * ((a) - 1) / 2 + ((b) - (a)))

#if FT_MODE == 0
// Sectors of two consecutive samples: log X per edge into the scratch (X in the order of
// removal, srcs/tropical_sampling.hpp:503-564), log psi_tr and log(xi_tr / psi_tr).  The
// first sample's draws are taken ahead, so that both walk their steps together.
static __device__ __forceinline__ void draw_pair(xo& g, const table_ref& t, unsigned char* lxs, df& lF, df& lG,
                                                 u32& exA, u32& exB, unsigned char* ordA, unsigned char* ordB)
{
    const float* ri = (const float*)t.ri;
    u32 hA[FT_E];
    u64 yA[FT_E];
#if !FT_CUT
    u32 lA[FT_E];
#endif
#pragma unroll
    for (int j = 0; j < FT_E; j++) {
        const u64 x = g.next();
        hA[j] = (u32)(x >> 32);
#if !FT_CUT
        lA[j] = (u32)x;
#endif
        yA[j] = j < FT_E - 1 ? g.next() : 0ull;
    }
    u32 sA = FT_FULL, sB = FT_FULL, mA = t.meta[FT_FULL], mB = mA;
    df lxx = tf_zero<fv>();
    lF = lG = lxx;
    exA = exB = 0;
#pragma unroll
    for (int j = 0; j < FT_E; j++) {
        const u64 xB = g.next();
        bool uA = false, uB = false;
#if FT_CUT
        int cA = find_cut(hA[j], sA, mA, t, FT_E - j, uA), cB = find_cut((u32)(xB >> 32), sB, mB, t, FT_E - j, uB);
#else
        int cA = scan_cut(((u64)hA[j] << 32) | lA[j], sA, t, uA), cB = scan_cut(xB, sB, t, uB);
#endif
        if (uA) {
            cA = exact_step(g, 2 * FT_E, sA, TABLE_GM(t));
            exA++;
        }
        if (uB) {
            cB = exact_step(g, 1, sB, TABLE_GM(t));
            exB++;
        }
        sA ^= 1u << cA;
        sB ^= 1u << cB;
        const u32 nA = t.meta[sA], nB = t.meta[sB];
        // the subgraph stops being mass-momentum spanning: xi_tr / psi_tr
        if (META_MM(mA) && !META_MM(nA)) {
            lG.hi.x = lxx.hi.x;
            lG.lo.x = lxx.lo.x;
        }
        if (META_MM(mB) && !META_MM(nB)) {
            lG.hi.y = lxx.hi.y;
            lG.lo.y = lxx.lo.y;
        }
        LX(cA, 0).x = lxx.hi.x;
        LX(cA, 1).x = lxx.lo.x;
        LX(cB, 0).y = lxx.hi.y;
        LX(cB, 1).y = lxx.lo.y;
        // it loses a loop: psi_tr
        if (j > 0) {
            const bool dA = META_L(nA) < META_L(mA), dB = META_L(nB) < META_L(mB);
            lF = tf_add_n(lF, tf_mk(make_float2(dA ? lxx.hi.x : 0.0f, dB ? lxx.hi.y : 0.0f),
                                    make_float2(dA ? lxx.lo.x : 0.0f, dB ? lxx.lo.y : 0.0f)));
        }
        mA = nA;
        mB = nB;
        if (FT_RECORD) {
            ordA[j] = (unsigned char)cA;
            ordB[j] = (unsigned char)cB;
        }
        if (j < FT_E - 1) {
            const df r = tf_mk(make_float2(ri[sA], ri[sB]), make_float2(t.rl[sA], t.rl[sB]));
            const df inc = tf_mul(log1m_pair(yA[j], g.next()), r);
            lxx = j == 0 ? inc : tf_norm(tf_add_n(lxx, inc));
        }
    }
    lF = tf_norm(lF);
}

#else
// Sector of one sample: log X per edge into the scratch (X in the order of removal,
// srcs/tropical_sampling.hpp:503-564), log psi_tr and log(xi_tr / psi_tr) in two-float.
// The phase of a deformed integrand moves by |theta| per unit of log X, so log X is
// carried to ~1e-12.  The logarithms are taken two draws at a time.
static __device__ __forceinline__ void draw_one(xo& g, const table_ref& t, unsigned char* lxs, sf& lF, sf& lG, u32& ex,
                                                unsigned char* ord)
{
    const float* ri = (const float*)t.ri;
    u32 sub = FT_FULL, meta = t.meta[FT_FULL];
    sf lxx = tf_zero<float>();
    lF = lG = lxx;
    ex = 0;
    u64 x = g.next();   // the draw of the next cut
    df l;
#pragma unroll
    for (int j = 0; j < FT_E; j++) {
        u64 x1 = 0;
        if (j < FT_E - 1 && !(j & 1)) {
            const u64 y0 = g.next();
            x1 = g.next();
            const u64 y1 = j < FT_E - 2 ? g.next() : y0;
            l = log1m_pair(y0, y1);
        }
        // draws taken from this cut's one on: x y0 x1 y1 at an even step (x y0 x1 and x at the
        // last two), x y1 at an odd one (x at the last)
        const int back = j & 1 ? (j < FT_E - 1 ? 2 : 1) : (j < FT_E - 2 ? 4 : (j < FT_E - 1 ? 3 : 1));
        bool unsure = false;
#if FT_CUT
        int c = find_cut((u32)(x >> 32), sub, meta, t, FT_E - j, unsure);
#else
        int c = scan_cut(x, sub, t, unsure);
#endif
        if (unsure) {
            c = exact_step(g, back, sub, TABLE_GM(t));
            ex++;
        }
        sub ^= 1u << c;
        const u32 m = t.meta[sub];
        if (META_MM(meta) && !META_MM(m)) lG = lxx;   // it stops being mass-momentum spanning: xi_tr / psi_tr
        LX(c, 0) = lxx.hi;
        LX(c, 1) = lxx.lo;
        if (j > 0 && META_L(m) < META_L(meta)) lF = tf_add_n(lF, lxx);   // it loses a loop: psi_tr
        meta = m;
        if (FT_RECORD) ord[j] = (unsigned char)c;
        if (j < FT_E - 1) {
            const sf inc = tf_mul(j & 1 ? second_of(l) : first_of(l), tf_mk(ri[sub], t.rl[sub]));
            lxx = j == 0 ? inc : tf_norm(tf_add_n(lxx, inc));
            x = j & 1 ? g.next() : x1;
        }
    }
    lF = tf_norm(lF);
}

#endif

// positive value m * 2^e with m in [1, 2) per sample: products without overflow
struct mexp {
    fv m;
    int ea, eb;
    bool ba, bb;
};
static __device__ __forceinline__ void mx_lane(float& m, int& e, bool& bad)
{
    const int b = __float_as_int(m);
    const int be = (b >> 23) & 0xff;
    bad |= (be == 0) | (be == 255) | (b < 0);
    e += be - 127;
    m = __int_as_float((b & 0x007fffff) | 0x3f800000);
}
static __device__ __forceinline__ void mx_mul(mexp& a, fv x)
{
    a.m = a.m * x;
    mx_lane(a.m.x, a.ea, a.ba);
    mx_lane(a.m.y, a.eb, a.bb);
}
static __device__ __forceinline__ mexp mx_one()
{
    mexp r;
    r.m = fv_of(1.0f);
    r.ea = r.eb = 0;
    r.ba = r.bb = false;
    return r;
}
static __device__ __forceinline__ fv fv_log2(fv x) { return make_float2(m_log2(x.x), m_log2(x.y)); }
static __device__ __forceinline__ fv fv_ints(int a, int b) { return make_float2((float)a, (float)b); }
#define RLN2_HI 1.44269502162933349609375f
#define RLN2_LO 1.925963033500011e-8f
#define LN2_F 0.69314718055994531f
// a natural logarithm in base 2
template <class V>
static __device__ __forceinline__ tf<V> tf_log2e(tf<V> x)
{
    return tf_mul(x, tf_mk(all_of<V>(RLN2_HI), all_of<V>(RLN2_LO)));
}
static __device__ __forceinline__ bool finite_(float x) { return isfinite(x); }

// undeformed integrand: relative size of V below which the FP32 evaluation hands the
// sample to FP64
#ifndef V_CANCEL
#define V_CANCEL 0.05f
#endif
// smallest pivot-to-row ratio accepted in the FP32 elimination of the Jacobian
#ifndef PIVOT_GROWTH
#define PIVOT_GROWTH 0.02f
#endif

#if FT_MODE == 0
// Undeformed integrand (srcs/feynman_integral.hpp:218-276) of two samples in FP32, in the
// frame X_e = exp(lx_e - sh).  Components of `bad`: the FP32 evaluation cannot be trusted
// (the sample then goes to the FP64 pass).
static __device__ __forceinline__ void integrand_pair(const float4* pp, const float* pf, unsigned char* lxs, df lF,
                                                      df lG, fv* out, bool& badA, bool& badB)
{
    const float D2 = 0.5f * pf[P_D], W = pf[P_W], IGtr = pf[P_IGTR];
    fv lmin = fv_of(0.0f);
#pragma unroll
    for (int e = 0; e < FT_E; e++) lmin = make_float2(fminf(lmin.x, LX(e, 0).x), fminf(lmin.y, LX(e, 0).y));
    // sh an integer near the middle of the range; R and the eps factor are ratios to the
    // tropical approximants and do not depend on it
    const fv sh = make_float2(rintf(0.5f * lmin.x), rintf(0.5f * lmin.y));
    fv X[FT_E], Xi[FT_E];
    mexp det = mx_one();
    df sumlx = tf_zero<fv>();   // log prod X
    badA = badB = false;
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const df a = tf_norm(tf_addf_n(tf_mk(LX(e, 0), LX(e, 1)), -sh));
        sumlx = e == 0 ? a : tf_add_n(sumlx, a);
        const fv ep = make_float2(m_exp(a.hi.x), m_exp(a.hi.y));
        X[e] = fma_(ep, a.lo, ep);
        Xi[e] = rcp_newton(X[e]);
        badA |= !(fabsf(a.hi.x) < 80.0f);   // beyond FP32's exponential
        badB |= !(fabsf(a.hi.y) < 80.0f);
    }
    sumlx = tf_norm(sumlx);
    const df lFs = tf_norm(tf_addf_n(lF, fv_of(-(float)FT_LOOPS) * sh));   // log psi_tr in the frame
    const df lGs = tf_norm(tf_addf_n(lG, -sh));                            // log V_tr = log(xi_tr / psi_tr)
    // conductance-form elimination (all values positive)
    fv c[FT_N][FT_N], g[FT_N], d[FT_N], id[FT_N], a[FT_N][FT_N];
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const int k = FT_EK[e], l = FT_EL[e];
        fv& slot = (k == FT_V - 1) ? g[l] : c[l][k];
        slot = first_in_slot(e) ? Xi[e] : slot + Xi[e];
    }
#pragma unroll
    for (int k = 0; k < FT_N; k++) {
        fv dk = g[k];
        bool any = NZG(k);
#pragma unroll
        for (int j = k + 1; j < FT_N; j++)
            if (NZC(k, j)) {
                dk = any ? dk + c[k][j] : c[k][j];
                any = true;
            }
        d[k] = dk;
        id[k] = rcp_newton(dk);
        mx_mul(det, dk);
#pragma unroll
        for (int i = k + 1; i < FT_N; i++)
            if (NZC(k, i)) a[k][i] = c[k][i] * id[k];
#pragma unroll
        for (int i = k + 1; i < FT_N; i++) {
            if (!NZC(k, i)) continue;
            if (NZG(k)) g[i] = ADDS_G(k, i) ? fma_(a[k][i], g[k], g[i]) : a[k][i] * g[k];
#pragma unroll
            for (int j = i + 1; j < FT_N; j++)
                if (NZC(k, j)) c[i][j] = ADDS_C(k, i, j) ? fma_(a[k][i], c[k][j], c[i][j]) : a[k][i] * c[k][j];
        }
    }
    badA |= det.ba;
    badB |= det.bb;
    // log2 psi (exponents and prod X exact, the rest in FP32), log2(psi / psi_tr)
    const df l2psi = tf_norm(tf_addf_n(tf_addf_n(tf_log2e(sumlx), fv_ints(det.ea, det.eb)), fv_log2(det.m)));
    const df lpsi = tf_sub(l2psi, tf_log2e(lFs));
#if FT_ONLY_PSI
    const df t = tf_norm(tf_mulf(lpsi, fv_of(-D2)));
    const fv R = make_float2(m_exp2(t.hi.x) * (1.0f + t.lo.x * LN2_F), m_exp2(t.hi.y) * (1.0f + t.lo.y * LN2_F));
    out[0] = fv_of(IGtr) * R;
#else
    // V = -sum_r sigma_r q_r^T L^-1 q_r + sum_e m2_e X_e
    fv v = fv_of(0.0f), mag = fv_of(0.0f);
#pragma unroll
    for (int r = 0; r < FT_RANK; r++) {
        fv y[FT_N], s = fv_of(0.0f);
#pragma unroll
        for (int i = FT_Q0; i < FT_N; i++) {
            fv yi = prm_fv(pp, P_Q + r * FT_N + i);
#pragma unroll
            for (int k = FT_Q0; k < i; k++)
                if (NZC(k, i)) yi = fma_(a[k][i], y[k], yi);
            y[i] = yi;
            s = i == FT_Q0 ? yi * yi * id[i] : fma_(yi * yi, id[i], s);
        }
        const fv w = prm_fv(pp, P_SIG + r) * s;
        v = v - w;
        mag = mag + abs_(w);
    }
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const fv w = prm_fv(pp, P_M2 + e) * X[e];
        v = v + w;
        mag = mag + abs_(w);
    }
    // cancellation, or a sign the FP64 pass must decide
    badA |= !(v.x > V_CANCEL * mag.x);
    badB |= !(v.y > V_CANCEL * mag.y);
    mexp V = mx_one();
    mx_mul(V, v);
    const df l2v = fast_two_sum(fv_ints(V.ea, V.eb), fv_log2(V.m));
    const df lv = tf_sub(l2v, tf_log2e(lGs));   // log2(V / V_tr)
    const df t = tf_norm(tf_add_n(tf_mulf(lpsi, fv_of(-D2)), tf_mulf(lv, fv_of(-W))));
    fv R = make_float2(m_exp2(t.hi.x) * (1.0f + t.lo.x * LN2_F), m_exp2(t.hi.y) * (1.0f + t.lo.y * LN2_F));
    badA |= !finite_(R.x) || V.ba;
    badB |= !finite_(R.y) || V.bb;
    R = fv_of(IGtr) * R;
    out[0] = R;
    if (FT_K > 1) {
        const fv ef = fv_of(LN2_F) * tf_f(tf_add(l2psi, tf_mulf(l2v, fv_of(-(float)FT_LOOPS))));
#pragma unroll
        for (int j = 1; j < FT_K; j++) {
            R = R * (ef * fv_of(1.0f / (float)j));
            out[j] = R;
        }
    }
#endif
}
#else
// ------------------------------------------------------------------ deformed integrand
struct cdf {
    sf re, im;
};
static __device__ __forceinline__ cdf cdf_mk(sf r, sf i)
{
    cdf z;
    z.re = r;
    z.im = i;
    return z;
}
static __device__ __forceinline__ cdf cdf_add_n(cdf a, cdf b) { return cdf_mk(tf_add_n(a.re, b.re), tf_add_n(a.im, b.im)); }
static __device__ __forceinline__ cdf cdf_norm(cdf a) { return cdf_mk(tf_norm(a.re), tf_norm(a.im)); }
static __device__ __forceinline__ cdf cdf_scale(sf s, cdf a) { return cdf_mk(tf_mul(s, a.re), tf_mul(s, a.im)); }
// x1 y1 - x2 y2 and x1 y1 + x2 y2, the low parts not renormalised
template <class V>
static __device__ __forceinline__ tf<V> dot_sub_n(tf<V> x1, tf<V> y1, tf<V> x2, tf<V> y2)
{
    const tf<V> p = tf_mul(x1, y1);
    const V n = mul_(-x2.hi, y2.hi);
    V l = fma_(x2.hi, y2.hi, n);   // x2 y2 + n, exactly
    l = fma_(x2.hi, y2.lo, l);
    l = fma_(x2.lo, y2.hi, l);
    const tf<V> s = two_sum(p.hi, n);
    return tf_mk(s.hi, s.lo + (p.lo - l));
}
template <class V>
static __device__ __forceinline__ tf<V> dot_add_n(tf<V> x1, tf<V> y1, tf<V> x2, tf<V> y2)
{
    const tf<V> p = tf_mul(x1, y1), q = tf_mul(x2, y2);
    const tf<V> s = two_sum(p.hi, q.hi);
    return tf_mk(s.hi, s.lo + (p.lo + q.lo));
}
static __device__ FT_CXFN cdf operator*(cdf a, cdf b)
{
    return cdf_norm(cdf_mk(dot_sub_n(a.re, b.re, a.im, b.im), dot_add_n(a.re, b.im, a.im, b.re)));
}
// a b + c, the sums' low parts left as they are (renormalised where the value is used)
static __device__ FT_CXFN cdf cdf_fma_n(cdf a, cdf b, cdf c)
{
    return cdf_add_n(cdf_mk(dot_sub_n(a.re, b.re, a.im, b.im), dot_add_n(a.re, b.im, a.im, b.re)), c);
}
static __device__ FT_BIGFN cdf cdf_inv(cdf a)
{
    const sf m = tf_inv(tf_norm(dot_add_n(a.re, a.re, a.im, a.im)));
    return cdf_mk(tf_mul(a.re, m), tf_mul(tf_neg(a.im), m));
}
// z 2^-k for the exponent k of z's larger part (exact), the exponent added to k;
// ok false where z is zero or not finite
static __device__ __forceinline__ float exp_scale(float re, float im, int& k, bool& ok)
{
    const float mx = fmaxf(fabsf(re), fabsf(im));
    const int be = (__float_as_int(mx) >> 23) & 0xff;
    const bool fine = be > 0 && be < 254;
    ok &= fine;
    k += fine ? be - 127 : 0;
    return __int_as_float((fine ? 254 - be : 127) << 23);
}
static __device__ __forceinline__ void cdf_renorm(cdf& z, int& k, bool& ok)
{
    const float sc = exp_scale(z.re.hi, z.im.hi, k, ok);
    z.re.hi *= sc;
    z.re.lo *= sc;
    z.im.hi *= sc;
    z.im.lo *= sc;
}

// e^a for two two-floats a (|a| < 80) in two-float, about 1e-12 relative; table-driven
// after Tang (ACM TOMS 15, 1989): a = (32 m + j) ln2/32 + s with |s| <= ln2/64,
// e^a = 2^m 2^(j/32) e^s, 2^(j/32) as two floats from FT_EXPTAB, e^s = 1 + s + s^2/2 +
// s^3/6 + s^4/24 with the terms past s in FP32.  ln2/32 = C1 + C2 + C3, C1 with 11
// significant bits so that k C1 is exact for |k| < 2^13.
static __device__ FT_BIGFN df exp_pair(df a)
{
    const float C1 = 0x1.62cp-6f, C2 = 0x1.217f7ep-17f, C3 = -0x1.c610cap-42f, MAGIC = 12582912.0f;
    // k = rint(32 a / ln2) by the rounding of the addition; its integer in the low bits
    const fv kb = fma_(a.hi, fv_of(46.1662407f), fv_of(MAGIC));
    const fv kf = kb - fv_of(MAGIC);
    const int kx = __float_as_int(kb.x) - 0x4b400000, ky = __float_as_int(kb.y) - 0x4b400000;
    // a - k C1 is exact; k C2 = p2 + e2 exactly
    const fv p2 = kf * fv_of(-C2);
    const fv e2 = fma_(kf, fv_of(C2), p2);
    df s = two_sum(fma_(kf, fv_of(-C1), a.hi), p2);
    s = fast_two_sum(s.hi, s.lo + fma_(kf, fv_of(-C3), a.lo - e2));
    const fv sh = s.hi;
    const fv tail = sh * sh * fma_(sh, fma_(sh, fv_of(0.0416666679f), fv_of(0.166666672f)), fv_of(0.5f));
    // e^s = 1 + es
    const df es = fast_two_sum(sh, s.lo + tail);
    df E = fast_two_sum(fv_of(1.0f), es.hi);
    E.lo = E.lo + es.lo;
    const float2 tx = FT_EXPTAB[kx & 31], ty = FT_EXPTAB[ky & 31];
    const df pr = tf_norm(tf_mul(tf_mk(make_float2(tx.x, ty.x), make_float2(tx.y, ty.y)), E));
    const fv sc = make_float2(__int_as_float((127 + (kx >> 5)) << 23), __int_as_float((127 + (ky >> 5)) << 23));
    return tf_mk(pr.hi * sc, pr.lo * sc);
}

// e^(ix) = cos x + i sin x of two angles to ~1e-13 (|x| < 1e5), table-driven after Tang: x = k pi/64 + r with
// |r| <= pi/128, pi/64 in three FP32 parts (x.hi - k P1 is exact: both are multiples of
// the same power of two and the difference is small); sin(k pi/64), cos(k pi/64) as float
// pairs from FT_SCTAB (k mod 128); sin r = r - r^3/6 + r^5/120 and cos r = 1 - r^2/2 +
// r^4/24 - r^6/720 with r and r^2 in two-float and the terms below 3e-6 in FP32; then
// the product of the two.
static __device__ __forceinline__ void expi_pair(df x, cdf* out)
{
    const float P1 = 0x1.921fb6p-5f, P2 = -0x1.777a5cp-30f, P3 = -0x1.ee59dap-55f, MAGIC = 12582912.0f;
    const fv kb = fma_(x.hi, fv_of(0x1.45f306p+4f), fv_of(MAGIC));
    const fv k = kb - fv_of(MAGIC);
    const df r = fast_two_sum(fma_(k, fv_of(-P1), x.hi), fma_(k, fv_of(-P3), fma_(k, fv_of(-P2), x.lo)));
    const fv rh = r.hi, r2 = rh * rh;
    // sin r = r + rh^3 (-1/6 + rh^2/120)
    const df sr = fast_two_sum(rh, fma_(rh * r2, fma_(r2, fv_of(0x1.111112p-7f), fv_of(-0x1.555556p-3f)), r.lo));
    // cos r = 1 - (rh^2 + 2 rh r.lo)/2 + rh^4/24 - rh^6/720, with rh^2 = r2 + qe exactly
    const fv qe = fma_(rh, rh, -r2);
    df cr = fast_two_sum(fv_of(1.0f), fv_of(-0.5f) * r2);
    cr.lo = cr.lo + fma_(r2 * r2, fma_(r2, fv_of(-0x1.6c16c2p-10f), fv_of(0x1.555556p-5f)),
                           fma_(-rh, r.lo, fv_of(-0.5f) * qe));
    const float4 tx = FT_SCTAB[__float_as_int(kb.x) & 127], ty = FT_SCTAB[__float_as_int(kb.y) & 127];
    const df sa = tf_mk(make_float2(tx.x, ty.x), make_float2(tx.y, ty.y));
    const df ca = tf_mk(make_float2(tx.z, ty.z), make_float2(tx.w, ty.w));
        const df re = tf_norm(dot_sub_n(ca, cr, sa, sr)), im = tf_norm(dot_add_n(ca, sr, sa, cr));
    out[0] = cdf_mk(first_of(re), first_of(im));
    out[1] = cdf_mk(second_of(re), second_of(im));
}

// |theta| beyond which expi_pair's reduction is not used (the FP64 pass takes the sample)
#define THETA_MAX 1e5f

// Principal argument of (x + xl) + i (y + yl) to about 1e-9: with a, b the larger and smaller
// modulus and c = i/64 their rounded ratio, atan(b/a) = atan c + atan z, z = (b - c a) /
// (a + c b) below 1/128, the first from FT_ATANTAB as two floats; then the octant.  (atanf of
// the rounded ratio kept 1.5e-7, which D/2 and W multiply.)  Zero gives 0.
static __device__ FT_BIGFN sf arg_f2(float x, float y, float xl, float yl)
{
    const float ax = fabsf(x), ay = fabsf(y);
    const float bxl = x < 0.0f ? -xl : xl, byl = y < 0.0f ? -yl : yl;
    const bool sw = ay > ax, left = x < 0.0f;
    const float a = sw ? ay : ax, b = sw ? ax : ay, al = sw ? byl : bxl, bl = sw ? bxl : byl;
    const float ib = fmaf(b * rcp_fast(a), 64.0f, 12582912.0f);   // i in the low bits
    const float c = (ib - 12582912.0f) * 0.015625f;
    const float num = fmaf(-c, a, b) + fmaf(-c, al, bl);
    const float z = num * rcp_newton(fmaf(c, b, a));
    const float2 T = FT_ATANTAB[__float_as_int(ib) & 127];
    sf v = fast_two_sum(T.x, z);
    v.lo += fmaf(z * z * z, -0.333333343f, T.y);
    // K +- v, K = 0, pi/2 or pi
    if (sw != left) v = tf_neg(v);
    const float K = sw ? 1.57079637f : (left ? 3.14159274f : 0.0f);
    const float Kl = sw ? -4.37113883e-8f : (left ? -8.74227766e-8f : 0.0f);
    v = tf_add(tf_mk(K, Kl), v);
    if (!(a > 0.0f)) v = tf_zero<float>();
    return y < 0.0f ? tf_neg(v) : v;
}
// log of a positive two-float x in two-float, to about 1e-9 (tables and steps of log1m_pair)
static __device__ FT_BIGFN sf log_tf(sf x)
{
    const int bits = __float_as_int(x.hi);
    const int e = (bits >> 23) - 127;
    const float sc = __int_as_float((127 - e) << 23);   // 2^-e
    const float4 T = FT_LOGTAB[(bits >> 17) & 63];
    const float z = fmaf(x.hi * sc, T.x, -1.0f) + x.lo * sc * T.x;
    const float kk = (float)e;
    const sf s = two_sum(kk * 0.693145751953125f, T.y);
    const sf t = two_sum(s.hi, z);
    const float tail = z * z * fmaf(z, fmaf(z, fmaf(z, 0.2f, -0.25f), 0.333333343f), -0.5f);
    return fast_two_sum(t.hi, (t.lo + s.lo) + (fmaf(kk, 1.428606765330187e-06f, T.z) + tail));
}
static __device__ __forceinline__ sf times_ln2(int k)
{
    const float f = (float)k;
    return fast_two_sum(f * 0.693145751953125f, f * 1.428606765330187e-06f);
}
// |z|^2 in two-float
static __device__ __forceinline__ sf norm2(cdf z) { return tf_norm(dot_add_n(z.re, z.re, z.im, z.im)); }
static __device__ __forceinline__ sf arg_of(cdf z) { return arg_f2(z.re.hi, z.im.hi, z.re.lo, z.im.lo); }
// principal argument reduced to (-pi, pi] in two-float
static __device__ __forceinline__ sf wrap_pi(sf x)
{
    const float TWO_PI_HI = 6.28318548202514648f, TWO_PI_LO = -1.7484555e-7f;
    const float f = tf_f(x);
    const float k = rintf(f * 0.159154943091895336f);
    // k 2 pi as an exact two-float product
    const float p = mul_(k, -TWO_PI_HI);
    const float e = fma_(k, (TWO_PI_HI), p);
    return tf_norm(tf_addf_n(tf_norm(tf_addf_n(x, p)), -fma_(k, (TWO_PI_LO), e)));
}

// deformed integrand, the two-float complex block (det L(y) and V): smallest accepted
// pivot-to-row ratio, smallest |V| relative to the sum of its terms' magnitudes, and
// largest W qmag / |V| (qmag: the magnitudes of every term summed into V, through the
// row quadratic forms).  Two-float arithmetic keeps ~1e-14 of these magnitudes and
// the sector point and contour it starts from ~1e-12, so the bounds only catch samples
// whose cancellation would amplify that to ~1e-7.
#ifndef ACC_GROWTH
#define ACC_GROWTH 1e-5f
#endif
#ifndef ACC_V_CANCEL
#define ACC_V_CANCEL 1e-6f
#endif
#ifndef ACC_V_AMPLIFY
#define ACC_V_AMPLIFY 1e5f
#endif
struct cblock {
    cdf V;
    cdf det;
    int e;       // det L(y) = det 2^e
    bool ok;     // pivots above ACC_GROWTH of their rows, the determinant finite and non-zero
    float mag;   // sum of the magnitudes of V's terms: masses, and one term per external row
    float qmag;  // the same through the row quadratic forms: sum_i |1/d_i| sum_jk |P~_jk| |U_ij| |U_ik| + mag
};
static __device__ __forceinline__ float cmag_hi(const cdf& z) { return abs_(z.re.hi) + abs_(z.im.hi); }

// the deformation angles and the upper triangle of kappa D H D, in the scratch or not
struct angles {
#if FT_SCRATCH >= 1
    __device__ __forceinline__ void set(unsigned char* lxs, int e, sf v)
    {
        SCR_TH(e, 0) = v.hi;
        SCR_TH(e, 1) = v.lo;
    }
    __device__ __forceinline__ sf get(unsigned char* lxs, int e) const { return tf_mk(SCR_TH(e, 0), SCR_TH(e, 1)); }
#else
    sf v[FT_E];
    __device__ __forceinline__ void set(unsigned char*, int e, sf x) { v[e] = x; }
    __device__ __forceinline__ sf get(unsigned char*, int e) const { return v[e]; }
#endif
};
struct hessian {
#if FT_SCRATCH >= 2
    __device__ __forceinline__ void set(unsigned char* lxs, int a, int b, float v) { SCR_H(a, b) = v; }
    __device__ __forceinline__ float get(unsigned char* lxs, int a, int b) const { return SCR_H(a, b); }
#else
    float v[FT_E][FT_E];
    __device__ __forceinline__ void set(unsigned char*, int a, int b, float x) { v[a][b] = x; }
    __device__ __forceinline__ float get(unsigned char*, int a, int b) const { return v[a][b]; }
#endif
};
#define XI(e) tf_mk(LX(e, 0), LX(e, 1))
// D, a power of two with D^2 / X in [1, 4), from 1/X
static __device__ __forceinline__ int edge_exp(float xi) { return -((((__float_as_int(xi) >> 23) & 255) - 127) >> 1); }
static __device__ __forceinline__ float edge_scale(float xi) { return __int_as_float((edge_exp(xi) + 127) << 23); }

// The deformed Laplacian at the sample (srcs/feynman_integral.hpp:293-310) and V there
// (:322-336) in two-float complex arithmetic, for every deformed sample: in FP32 both
// suffer cancellation (the spanning-tree sum with phases, the quadratic forms against
// the mass terms), and their errors enter the integrand as D/2 arg psi and W arg V.
// Conductances y_e = e^(-i theta_e) / X_e from the two-float contour and sector point,
// the conductance-form elimination of `elim`, the product of its pivots (rescaled by
// powers of two as it goes: det L(y) = det 2^e) and
// V = -sum_jk P~_jk (L(y)^-1)_jk + sum_e m2_e X_e e^(i theta_e) (the reference's
// -sum_r sigma_r q_r^T L^-1 q_r, contracted with P~ itself here).
static __device__ __forceinline__ void complex_block(unsigned char* lxs, const angles& th, const float4* pp, cblock& o)
{
    cdf c[FT_N][FT_N], g[FT_N];
    cdf v, ei[2];
    float mag = 0.0f;
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        if (!(e & 1)) expi_pair(pair_of(th.get(lxs, e), th.get(lxs, e + 1 < FT_E ? e + 1 : e)), ei);
        const cdf eix = ei[e & 1];
        const sf xi = XI(e);
        const cdf y = cdf_mk(tf_mul(xi, eix.re), tf_mul(tf_neg(xi), eix.im));
        const int k = FT_EK[e], l = FT_EL[e];
        cdf& slot = (k == FT_V - 1) ? g[l] : c[l][k];
        slot = first_in_slot(e) ? y : cdf_add_n(slot, y);
        const sf m2x = tf_mul(prm_sf(pp, P_M2 + e), tf_inv(xi));
        const cdf mt = cdf_scale(m2x, eix);
        v = e == 0 ? mt : cdf_add_n(v, mt);
        mag = mag + abs_(m2x.hi);
    }
    cdf a[FT_N][FT_N], dinv[FT_N], det;
    o.e = 0;
    o.ok = true;
#pragma unroll
    for (int k = 0; k < FT_N; k++) {
        if (NZG(k) && SUMS_G(k)) g[k] = cdf_norm(g[k]);
        cdf dk;
        float row;
        bool any = NZG(k);
        if (any) {
            dk = g[k];
            row = cmag_hi(g[k]);
        }
#pragma unroll
        for (int j = k + 1; j < FT_N; j++) {
            if (!NZC(k, j)) continue;
            if (SUMS_C(k, j)) c[k][j] = cdf_norm(c[k][j]);
            dk = any ? cdf_add_n(dk, c[k][j]) : c[k][j];
            row = any ? row + cmag_hi(c[k][j]) : cmag_hi(c[k][j]);
            any = true;
        }
        dk = cdf_norm(dk);
        o.ok &= cmag_hi(dk) > ACC_GROWTH * row;
        det = k == 0 ? dk : det * dk;
        cdf_renorm(det, o.e, o.ok);
        dinv[k] = cdf_inv(dk);
#pragma unroll
        for (int i = k + 1; i < FT_N; i++)
            if (NZC(k, i)) a[k][i] = c[k][i] * dinv[k];
#pragma unroll
        for (int i = k + 1; i < FT_N; i++) {
            if (!NZC(k, i)) continue;
            if (NZG(k)) g[i] = ADDS_G(k, i) ? cdf_fma_n(a[k][i], g[k], g[i]) : a[k][i] * g[k];
#pragma unroll
            for (int j = i + 1; j < FT_N; j++)
                if (NZC(k, j)) c[i][j] = ADDS_C(k, i, j) ? cdf_fma_n(a[k][i], c[k][j], c[i][j]) : a[k][i] * c[k][j];
        }
    }
    // The momentum part, sum_jk P~_jk (L(y)^-1)_jk over the external rows [Q0, N) (P~
    // vanishes elsewhere).  The forward substitution is y = U q with U unit lower
    // triangular, U_ij = sum_{j <= k < i} a_ki U_kj, so L^-1 = U^T diag(1/d) U there and
    // the part is sum_i (u_i^T P~ u_i) / d_i, u_i the i-th row of U: one quadratic form of
    // P~ per row instead of one forward substitution per term of its low-rank split.
    float qmag = 0.0f;
#if FT_NE > 0
    {
        auto ptd = [&](int j, int k) -> sf { return prm_sf(pp, PT_AT(j, k)); };
        cdf U[FT_NE][FT_NE];   // U[i][j], j < i (indices from Q0)
        cdf vq;
#pragma unroll
        for (int ii = 0; ii < FT_NE; ii++) {
            const int i = FT_Q0 + ii;
#pragma unroll
            for (int jj = 0; jj < ii; jj++) {
                const int j = FT_Q0 + jj;
                cdf u;
                int terms = 0;
                if (NZC(j, i)) {
                    u = a[j][i];
                    terms = 1;
                }
#pragma unroll
                for (int kk = jj + 1; kk < ii; kk++) {
                    const int k = FT_Q0 + kk;
                    if (!NZC(k, i) || !NZM(j, k)) continue;
                    u = terms ? cdf_fma_n(a[k][i], U[kk][jj], u) : a[k][i] * U[kk][jj];
                    terms++;
                }
                if (terms) U[ii][jj] = terms > 1 ? cdf_norm(u) : u;
            }
            // Q = u^T P~ u with u = (U_i0 .. U_i,i-1, 1): Q = P_ii + sum_j u_j w_j,
            // w_j = sum_{j <= k < i} P_jk u_k + P_ji (off-diagonal P doubled)
            const sf pii = ptd(ii, ii);
            cdf Q = cdf_mk(pii, tf_zero<float>());
            float qm = abs_(pii.hi);
            bool one = true;
#pragma unroll
            for (int jj = 0; jj < ii; jj++) {
                if (!NZM(FT_Q0 + jj, i)) continue;
                const sf pj = ptd(jj, ii);
                cdf w = cdf_scale(ptd(jj, jj), U[ii][jj]);
                float wm = abs_(ptd(jj, jj).hi) * cmag_hi(U[ii][jj]);
#pragma unroll
                for (int kk = jj + 1; kk < ii; kk++) {
                    if (!NZM(FT_Q0 + kk, i)) continue;
                    w = cdf_add_n(w, cdf_scale(ptd(jj, kk), U[ii][kk]));
                    wm = fma_(abs_(ptd(jj, kk).hi), cmag_hi(U[ii][kk]), wm);
                }
                w.re = tf_add_n(w.re, pj);
                w = cdf_norm(w);
                wm = wm + abs_(pj.hi);
                Q = cdf_fma_n(U[ii][jj], w, Q);
                qm = fma_(cmag_hi(U[ii][jj]), wm, qm);
                one = false;
            }
            const cdf t = one ? cdf_scale(pii, dinv[i]) : cdf_norm(Q) * dinv[i];
            vq = ii == 0 ? t : cdf_add_n(vq, t);
            mag = mag + cmag_hi(t);
            qmag = fma_(qm, cmag_hi(dinv[i]), qmag);
        }
        v = cdf_mk(tf_sub_n(v.re, vq.re), tf_sub_n(v.im, vq.im));
    }
#endif
    o.V = cdf_norm(v);
    o.det = det;
    o.mag = mag;
    o.qmag = qmag + mag;
}

// x-derivatives of phi/psi at the sample point (srcs/laplacian.hpp:102-215) and the
// deformation angle theta = -lambda (d(phi/psi)/dx + m^2) (srcs/feynman_integral.hpp:290-291).
// Everything here is a difference of entries of L^-1, which cancels in FP32 for a
// sizeable fraction of sectors, so the block runs in two-float arithmetic: the
// conductance-form elimination (all operations on positive values), G = L^-1, the
// potentials h_r = G q_r and their drops across the edges, the effective-resistance
// combinations t, and the Minkowski products s.  Reads 1/X from the scratch; outputs theta
// and the upper triangle of kappa D H D in FP32, D ~ X^1/2 a power of two per edge: with
// hb = D / X^2 h . b_e and s_ab = -2 kappa sum_r sigma_r hb_a hb_b its entries are s_ab t_ab
// (the diagonal s_aa (t_aa - X_a)), two roundings each, and theta_a = kappa m2_a + s_aa X_a^2 /
// (2 D_a^2).
static __device__ __forceinline__ void derivatives(unsigned char* lxs, const float4* pp, angles& th, hessian& H,
                                                        bool& cancel)
{
    sf c[FT_N][FT_N], g[FT_N];
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const int k = FT_EK[e], l = FT_EL[e];
        sf& slot = (k == FT_V - 1) ? g[l] : c[l][k];
        slot = first_in_slot(e) ? XI(e) : tf_add_n(slot, XI(e));
    }
    sf a[FT_N][FT_N], id[FT_N];
#pragma unroll
    for (int k = 0; k < FT_N; k++) {
        if (NZG(k) && SUMS_G(k)) g[k] = tf_norm(g[k]);
        sf dk;
        bool any = NZG(k);
        if (any) dk = g[k];
#pragma unroll
        for (int j = k + 1; j < FT_N; j++)
            if (NZC(k, j)) {
                if (SUMS_C(k, j)) c[k][j] = tf_norm(c[k][j]);
                dk = any ? tf_add_n(dk, c[k][j]) : c[k][j];
                any = true;
            }
        id[k] = tf_inv(tf_norm(dk));
#pragma unroll
        for (int i = k + 1; i < FT_N; i++)
            if (NZC(k, i)) a[k][i] = tf_mul(c[k][i], id[k]);
#pragma unroll
        for (int i = k + 1; i < FT_N; i++) {
            if (!NZC(k, i)) continue;
            if (NZG(k)) g[i] = ADDS_G(k, i) ? tf_fma_n(a[k][i], g[k], g[i]) : tf_mul(a[k][i], g[k]);
#pragma unroll
            for (int j = i + 1; j < FT_N; j++)
                if (NZC(k, j)) c[i][j] = ADDS_C(k, i, j) ? tf_fma_n(a[k][i], c[k][j], c[i][j]) : tf_mul(a[k][i], c[k][j]);
        }
    }
    // N = M^-1 (unit upper triangular, non-negative), G = N diag(1/d) N^T
    sf Nm[FT_N][FT_N];
#pragma unroll
    for (int i = FT_N - 1; i >= 0; i--) {
#pragma unroll
        for (int j = i + 1; j < FT_N; j++) {
            if (!NZM(i, j)) continue;
            sf s;
            int terms = 0;
            if (NZC(i, j)) {
                s = a[i][j];
                terms = 1;
            }
#pragma unroll
            for (int k = i + 1; k < j; k++)
                if (NZC(i, k) && NZM(k, j)) {
                    s = terms ? tf_fma_n(a[i][k], Nm[k][j], s) : tf_mul(a[i][k], Nm[k][j]);
                    terms++;
                }
            Nm[i][j] = terms > 1 ? tf_norm(s) : s;
        }
    }
    // Nd[j][k] = N[j][k] / d_k, so that each term of G is one two-float multiply-add
    sf Nd[FT_N][FT_N];
#pragma unroll
    for (int j = 0; j < FT_N; j++)
#pragma unroll
        for (int k = j + 1; k < FT_N; k++)
            if (NZM(j, k)) Nd[j][k] = tf_mul(Nm[j][k], id[k]);
    sf G[FT_N][FT_N];
#pragma unroll
    for (int i = 0; i < FT_N; i++)
#pragma unroll
        for (int j = i; j < FT_N; j++) {
            // k = j term has N[j][j] = 1
            sf s = tf_zero<float>();
            int terms = 0;
            if (i == j || NZM(i, j)) {
                s = (i == j) ? id[j] : Nd[i][j];
                terms = 1;
            }
#pragma unroll
            for (int k = j + 1; k < FT_N; k++)
                if (NZM(i, k) && NZM(j, k)) {
                    s = terms ? tf_fma_n(Nm[i][k], Nd[j][k], s) : tf_mul(Nm[i][k], Nd[j][k]);
                    terms++;
                }
            G[i][j] = G[j][i] = terms > 1 ? tf_norm(s) : s;
        }
    sf hb[FT_RANK][FT_E];
#pragma unroll
    for (int r = 0; r < FT_RANK; r++) {
        sf h[FT_N];
#pragma unroll
        for (int i = 0; i < FT_N; i++) {
            sf s = tf_zero<float>();
#pragma unroll
            for (int j = FT_Q0; j < FT_N; j++) {
                const sf q = prm_sf(pp, P_Q + r * FT_N + j);
                s = j == FT_Q0 ? tf_mul(G[i][j], q) : tf_fma_n(G[i][j], q, s);
            }
            h[i] = s;
        }
#pragma unroll
        for (int e = 0; e < FT_E; e++) {
            const int k = FT_EK[e], l = FT_EL[e];
            const sf xi = XI(e), xa = tf_mul(xi, xi);
            const float D = edge_scale(xi.hi);
            hb[r][e] = tf_mul((k == FT_V - 1) ? tf_norm(tf_neg(h[l])) : tf_sub(h[k], h[l]), tf_mk(xa.hi * D, xa.lo * D));
        }
    }
    const sf kappa = prm_sf(pp, P_DEF);
    sf ks[FT_RANK];   // -2 kappa sigma
#pragma unroll
    for (int r = 0; r < FT_RANK; r++) {
        ks[r] = tf_mul(prm_sf(pp, P_SIG + r), kappa);
        ks[r] = tf_mk(-2.0f * ks[r].hi, -2.0f * ks[r].lo);
    }
#pragma unroll
    for (int a2 = 0; a2 < FT_E; a2++) {
        const int ka = FT_EK[a2], la = FT_EL[a2];
        // w = row a2 of (edge incidence) L^-1, w_v = G_{ka v} - G_{la v} (the ground's row of
        // L^-1 is zero): edge a2's resistance combination with any edge (k, l),
        // G_ka,k + G_la,l - G_ka,l - G_la,k, is then w_k - w_l.  The entries no edge
        // pair reads are dropped at compile time.
        sf w[FT_N];
#pragma unroll
        for (int v = 0; v < FT_N; v++)
            w[v] = ka == FT_V - 1 ? tf_neg(G[la][v]) : (la == FT_V - 1 ? G[ka][v] : tf_sub_n(G[ka][v], G[la][v]));
        auto wd = [&](int k, int l) -> sf {
            return k == FT_V - 1 ? tf_neg(w[l]) : (l == FT_V - 1 ? w[k] : tf_sub_n(w[k], w[l]));
        };
        sf sig_hb[FT_RANK];
        sf s = tf_zero<float>();
#pragma unroll
        for (int r = 0; r < FT_RANK; r++) {
            sig_hb[r] = tf_mul(ks[r], hb[r][a2]);
            s = r == 0 ? tf_mul(sig_hb[r], hb[r][a2]) : tf_fma_n(sig_hb[r], hb[r][a2], s);
        }
        if (FT_RANK > 1) s = tf_norm(s);
        const sf t = tf_norm(wd(ka, la));
        // an edge whose ends float together: the FP64 pass takes the sample
        if (ka != FT_V - 1) {
            cancel |= !(t.hi > 1e-7f * (G[ka][ka].hi + G[la][la].hi));
        }
        const sf xi = XI(a2), x = tf_inv(xi);
        const float D = edge_scale(xi.hi), iD2 = 0.5f / (D * D);   // powers of two
        const sf q = tf_mul(s, tf_mul(x, x));
        th.set(lxs, a2, tf_add(tf_mul(kappa, prm_sf(pp, P_M2 + a2)), tf_mk(q.hi * iD2, q.lo * iD2)));
        H.set(lxs, a2, a2, tf_f(tf_mul(s, tf_sub(t, x))));
#pragma unroll
        for (int b = a2 + 1; b < FT_E; b++) {
            const int kb = FT_EK[b], lb = FT_EL[b];
            sf s2 = tf_zero<float>();
#pragma unroll
            for (int r = 0; r < FT_RANK; r++)
                s2 = r == 0 ? tf_mul(sig_hb[r], hb[r][b]) : tf_fma_n(sig_hb[r], hb[r][b], s2);
            H.set(lxs, a2, b, tf_f(s2) * tf_f(wd(kb, lb)));
        }
    }
}

// Deformed integrand (srcs/feynman_integral.hpp:278-362) of a sample, in the frame X_e =
// exp(lx_e - sh).  False: the evaluation cannot be trusted (the sample then goes to the
// FP64 pass).
static __device__ __forceinline__ bool integrand_one(const float4* pp, const float* pf, unsigned char* lxs, sf lF,
                                                     sf lG, cx<float>* out)
{
    const float D2 = 0.5f * pf[P_D], W = pf[P_W], IGtr = pf[P_IGTR];
    float lmin = 0.0f;
#pragma unroll
    for (int e = 0; e < FT_E; e++) lmin = fminf(lmin, LX(e, 0));
    // sh an integer near the middle of the range; R and the eps factor are ratios to the
    // tropical approximants and do not depend on it
    const float sh = rintf(0.5f * lmin);
    // 1/X in two-float for the derivative block and the complex Laplacian (theta is a
    // function of X whose phase effect grows with |theta|), over log X in the scratch;
    // log prod X in the frame
    bool bad = false;
    df sums = tf_zero<fv>();
#pragma unroll
    for (int e = 0; e < FT_E; e += 2) {
        const int f = e + 1 < FT_E ? e + 1 : e;
        const df na = tf_norm(tf_sub_n(tf_mk(fv_of(sh), fv_of(0.0f)), pair_of(XI(e), XI(f))));
        const df xi = exp_pair(na);
        const sf na1 = f == e ? tf_zero<float>() : second_of(na);
        sums = e == 0 ? na : tf_add_n(sums, f == e ? pair_of(first_of(na), na1) : na);
        LX(e, 0) = xi.hi.x;
        LX(e, 1) = xi.lo.x;
        LX(f, 0) = xi.hi.y;
        LX(f, 1) = xi.lo.y;
        // outside the two-float exponential's range: the FP64 pass takes it
        bad |= !(fabsf(na.hi.x) < 69.0f) || !(fabsf(na.hi.y) < 69.0f);
    }
    const sf sumlx = tf_neg(FT_E > 1 ? tf_add(first_of(sums), second_of(sums)) : first_of(sums));
    const sf lFs = tf_norm(tf_addf_n(lF, -(float)FT_LOOPS * sh));   // log psi_tr in the frame
    const sf lGs = tf_norm(tf_addf_n(lG, -sh));                     // log V_tr = log(xi_tr / psi_tr)
    angles th;
    cx<float> pj;
    int pe = 0;
    {
        hessian H;
        derivatives(lxs, pp, th, H, bad);
        // det(I + i kappa H X) = det(D^2/X + i kappa D H D) prod X/D^2 (srcs/feynman_integral.hpp:312-320):
        // the real part is diagonal and at least 1, so the symmetric elimination needs no
        // pivoting (no pivot's real part falls below); FP32, the pivots' product rescaled by powers
        // of two (pj 2^pe).  Before the complex block, so that H is no longer live there.
        cx<float> J[FT_E][FT_E];
#pragma unroll
        for (int a = 0; a < FT_E; a++)
#pragma unroll
            for (int b = a; b < FT_E; b++) J[a][b] = cmk(0.0f, H.get(lxs, a, b));
        bool ok = true;
#pragma unroll
        for (int e = 0; e < FT_E; e++) {
            const sf xi = XI(e);
            const int ex = edge_exp(xi.hi);
            J[e][e].re = tf_f(xi) * __int_as_float((2 * ex + 127) << 23);
            pe -= 2 * ex;   // prod X is taken with its logarithm
        }
#pragma unroll
        for (int k = 0; k < FT_E; k++) {
            const cx<float> piv = J[k][k];
            const float m = fabsf(piv.re) + fabsf(piv.im);
            float row = m;
#pragma unroll
            for (int j = k + 1; j < FT_E; j++) row += fabsf(J[k][j].re) + fabsf(J[k][j].im);
            const float n2 = fmaf(piv.re, piv.re, piv.im * piv.im);
            ok &= m > PIVOT_GROWTH * row && n2 < 1e36f;
            pj = k == 0 ? piv : pj * piv;
            if ((k & 1) || k == FT_E - 1) {   // |piv| < 1e18: two of them stay in range
                const float sc = exp_scale(pj.re, pj.im, pe, ok);
                pj = cmk(pj.re * sc, pj.im * sc);
            }
            const float id = rcp_newton(n2);
            const cx<float> inv = cmk(piv.re * id, -piv.im * id);
#pragma unroll
            for (int i = k + 1; i < FT_E; i++) {
                const cx<float> f = J[k][i] * inv;
#pragma unroll
                for (int j = i; j < FT_E; j++) J[i][j] = J[i][j] - f * J[k][j];
            }
        }
        bad |= !ok;
    }
    // phase sums in two-float: sum theta and nu . theta
    sf xnu = tf_zero<float>(), thsum = xnu;
#pragma unroll
    for (int e = 0; e < FT_E; e++) {
        const sf t = th.get(lxs, e), tn = tf_mulf(t, pp[P_NU + e].x);
        thsum = e == 0 ? t : tf_add_n(thsum, t);
        xnu = e == 0 ? tn : tf_add_n(xnu, tn);
        bad |= !(fabsf(t.hi) < THETA_MAX);
    }
    thsum = tf_norm(thsum);
    xnu = tf_norm(xnu);
    if (bad) return false;
    cblock cb;
    complex_block(lxs, th, pp, cb);
    // two-float pivots lose ~1e-14 / growth
    if (!cb.ok) return false;
    // V = Vn 2^ve, |Vn| in [1, 2 sqrt 2)
    cdf Vn = cb.V;
    int ve = 0;
    bool ok = true;
    cdf_renorm(Vn, ve, ok);
    if (!ok || ve > 126) return false;
    const float vsc = __int_as_float((127 - ve) << 23);   // 2^-ve
    const sf vn2 = norm2(Vn);
    const float vm = sqrtf(vn2.hi);
    // V in two-float keeps ~1e-14 of its terms' magnitudes (and ~1e-12 from the sector
    // point and contour it is built from): samples where V cancels to below 1e-6 of its
    // terms, or where W qmag / |V| exceeds 1e5, go to the FP64 pass
    if (!(vm > ACC_V_CANCEL * (cb.mag * vsc)) || !(W * (cb.qmag * vsc) < ACC_V_AMPLIFY * vm)) return false;
    // an argument within 1e-5 of the branch cut: the FP64 pass decides the branch
    const sf av2 = arg_of(Vn);
    const float av = tf_f(av2);
    // arg cPsi = sum theta + arg det L(y), reduced to the principal branch in two-float
    const sf apsi2 = wrap_pi(tf_add(thsum, arg_of(cb.det)));
    const float apsi = tf_f(apsi2);
    if (fabsf(av) > 3.14158265f || fabsf(apsi) > 3.14158265f) return false;
    // log |cPsi| and log |V|, then
    // log |cR / IGtr| = -D/2 log(|cPsi| / psi_tr) - W log(|V| / V_tr) + log |det J|
    auto half = [](sf a) -> sf { return tf_mk(0.5f * a.hi, 0.5f * a.lo); };
    const sf lpsi = tf_add(tf_add_n(sumlx, times_ln2(cb.e)), half(log_tf(norm2(cb.det))));
    const sf lv = tf_add(times_ln2(ve), half(log_tf(vn2)));
    const float pn = pj.re * pj.re;
    const sf pn2 = tf_mk(fmaf(pj.im, pj.im, pn), fmaf(pj.re, pj.re, -pn));
    sf t = tf_add_n(tf_mulf(tf_sub(lpsi, lFs), -D2), tf_mulf(tf_sub(lv, lGs), -W));
    t = tf_add_n(t, tf_add_n(tf_add_n(sumlx, times_ln2(pe)), half(log_tf(tf_norm(pn2)))));
    t = tf_norm(t);
    // arg cR = -D/2 arg cPsi + arg det J + nu . theta - W arg V (two-float sum)
    const sf aj = arg_f2(pj.re, pj.im, 0.0f, 0.0f);
    const sf ang = tf_norm(tf_add_n(tf_add_n(tf_mulf(apsi2, -D2), xnu), tf_add_n(aj, tf_mulf(av2, -W))));
    float sn, cs;
    m_sincos(ang.hi, &sn, &cs);
    const float c2 = fmaf(-ang.lo, sn, cs), s2 = fmaf(ang.lo, cs, sn);
    const float mod = m_exp(t.hi) * (1.0f + t.lo);
    if (!isfinite(mod)) return false;
    const sf ig = prm_sf(pp, P_IGTR);
    const float im = fmaf(mod, ig.hi, mod * ig.lo);
    const cx<float> c = cmk(im * c2, im * s2);
    out[0] = c;
    if (FT_K > 1) {
        // orders j: c ef^j / j!, ef = log cPsi - L log V (srcs/feynman_integral.hpp:336-341)
        const float nl = -(float)FT_LOOPS;
        const cdf ef = cdf_mk(tf_add(lpsi, tf_mulf(lv, nl)), tf_add(apsi2, tf_mulf(av2, nl)));
        cdf z = cdf_mk(tf_mk(c.re, 0.0f), tf_mk(c.im, 0.0f));
        float fact = 1.0f;
#pragma unroll
        for (int j = 1; j < FT_K; j++) {
            z = z * ef;
            fact *= 1.0f / (float)j;
            out[j] = cmk(z.re.hi * fact, z.im.hi * fact);
        }
    }
    return true;
}
#endif
#endif

// ------------------------------------------------------------------ accumulation
// stream state from 4 words (16-byte aligned)
static __device__ __forceinline__ xo load_state(const u64* __restrict__ s)
{
    const ulonglong2 a = *(const ulonglong2*)s, b = *(const ulonglong2*)(s + 2);
    xo g;
    g.a = a.x;
    g.b = a.y;
    g.c = b.x;
    g.d = b.y;
    return g;
}

// ------------------------------------------------------------------ start states
// The state of a stream after t strides, from the stride's matrices A^n over GF(2) (T the
// generator's step, A = T^S; written by ft_stride_matrices): first, for every nibble n of
// the state and value v of it, its image under A^l, l < 32, as [16 n + v][l] (4 words
// each), then A^(32 8^d v), v = 1 .. 7, for the octal digits d of t / 32 (1024 words each).
#define MAT_LANES 131072u
// g <- M g by the whole warp: lane l owns input bits 8l .. 8l+7 (column c of M is the four
// words M[4c .. 4c+3]); the partial results are XOR-reduced across the warp
static __device__ __forceinline__ u64 warp_xor(u64 x)
{
    return ((u64)__reduce_xor_sync(0xffffffffu, (u32)(x >> 32)) << 32) | __reduce_xor_sync(0xffffffffu, (u32)x);
}
static __device__ __noinline__ xo warp_apply(const u64* __restrict__ M, xo g)
{
    const u32 lane = threadIdx.x & 31u;
    const u64 word = lane < 8u ? g.a : lane < 16u ? g.b : lane < 24u ? g.c : g.d;
    const u32 bits = (u32)(word >> ((lane & 7u) * 8u)) & 255u;
    u64 r0 = 0, r1 = 0, r2 = 0, r3 = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const u64 mask = 0ull - (u64)((bits >> k) & 1u);
        const ulonglong2* col = (const ulonglong2*)(M + 4u * (lane * 8u + k));
        const ulonglong2 lo = __ldg(col), hi = __ldg(col + 1);
        r0 ^= lo.x & mask;
        r1 ^= lo.y & mask;
        r2 ^= hi.x & mask;
        r3 ^= hi.y & mask;
    }
    g.a = warp_xor(r0);
    g.b = warp_xor(r1);
    g.c = warp_xor(r2);
    g.d = warp_xor(r3);
    return g;
}
// g, the same in all lanes, to t strides on in the lane of thread t (t / 32 the same in all
// lanes): one product per octal digit by the warp together, then every lane its own A^lane
// g, whose nibbles are the same in all lanes: 64 reads of a kilobyte, eight in flight (a
// thread's five products of 256 masked columns, one after the other, took 300 us of a call
// with 1e5 one-loop samples and a third of its batch; the columns of the set bits, twice the
// bytes, 20 us).
static __device__ __noinline__ xo start_state(xo g, const u64* __restrict__ mats, u32 t, int digits)
{
    u32 w = t >> 5;
#pragma unroll 1
    for (int d = 0; d < digits; d++, w >>= 3)
        if (w & 7u) g = warp_apply(mats + MAT_LANES + (size_t)(d * 7u + (w & 7u) - 1u) * 1024u, g);
    u64 r0 = 0, r1 = 0, r2 = 0, r3 = 0;
    const ulonglong2* p = (const ulonglong2*)mats + (t & 31u) * 2u;
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
        const u64 word = k < 2 ? g.a : k < 4 ? g.b : k < 6 ? g.c : g.d;
        const u32 half = (u32)(k & 1 ? word >> 32 : word);
        ulonglong2 lo[8], hi[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const ulonglong2* e = p + ((k * 8 + i) * 16 + ((half >> (4 * i)) & 15u)) * 64u;
            lo[i] = __ldg(e);
            hi[i] = __ldg(e + 1);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            r0 ^= lo[i].x;
            r1 ^= lo[i].y;
            r2 ^= hi[i].x;
            r3 ^= hi[i].y;
        }
    }
    g.a = r0;
    g.b = r1;
    g.c = r2;
    g.d = r3;
    return g;
}

// ------------------------------------------------------------------ table staging
// FP64 form: shared = [1/r64 | meta | thresholds].  Mixed form: shared = [1/r32 hi |
// 1/r32 lo | meta | thresholds].
#if FT_TABLE_GLOBAL
#define SM_USED 0u
#else
#define SM_USED (12u * T_ENTRIES + T_QBYTES)
#endif
static __device__ __forceinline__ void copy_bytes(unsigned char* dst, const unsigned char* __restrict__ src, u32 bytes)
{
    const u32 n16 = bytes / 16u;
    for (u32 i = threadIdx.x; i < n16; i += blockDim.x) ((uint4*)dst)[i] = ((const uint4*)src)[i];
    for (u32 i = n16 * 16u + threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

// the table's sections: in global memory (large tables, L2 / L1 cached)
static __device__ __forceinline__ table_ref global_table(const unsigned char* __restrict__ tab)
{
    table_ref t;
    t.gm = tab;
#if FT_CUT
    t.q = tab + T_Q;
    t.Jr = nullptr;
#elif FT_PREC == 0
    t.q = tab + T_W64;
    t.Jr = tab + T_JR64;
#else
    t.q = tab + T_W32;
    t.Jr = tab + T_JR32;
#endif
    t.ri = tab + (FT_PREC == 0 ? T_RI64 : T_RH32);
    t.rl = (const float*)(tab + T_RL32);
    t.meta = (const u32*)(tab + T_META);
    return t;
}

// the same in global memory or the staged copy in shared memory
static __device__ __forceinline__ table_ref table_at(unsigned char* sm, const unsigned char* __restrict__ tab)
{
#if FT_TABLE_GLOBAL
    (void)sm;
    return global_table(tab);
#else
    table_ref t;
    t.gm = tab;
    t.Jr = nullptr;
    t.ri = sm;
    t.rl = (const float*)(sm + 4u * T_ENTRIES);
    t.meta = (const u32*)(sm + 8u * T_ENTRIES);
    t.q = sm + 12u * T_ENTRIES;
    return t;
#endif
}

// the block's copy of a staged table (no barrier)
static __device__ __forceinline__ void copy_table(unsigned char* sm, const unsigned char* __restrict__ tab)
{
#if FT_TABLE_GLOBAL
    (void)sm;
    (void)tab;
#else
#if FT_PREC == 0
    copy_bytes(sm, tab + T_RI64, 8u * T_ENTRIES);
    copy_bytes(sm + 8u * T_ENTRIES, tab + T_META, 4u * T_ENTRIES + T_QBYTES);   // adjacent
#else
    copy_bytes(sm, tab + T_RH32, 12u * T_ENTRIES + T_QBYTES);
#endif
#endif
}

static __device__ __forceinline__ table_ref stage_table(unsigned char* sm, const unsigned char* __restrict__ tab)
{
    copy_table(sm, tab);
#if !FT_TABLE_GLOBAL
    __syncthreads();
#endif
    return table_at(sm, tab);
}

// ------------------------------------------------------------------ accumulators
// Per-thread sums live in shared memory (slot-major, so a warp touches consecutive
// words), which keeps them out of the register budget of the sampling code:
//   FP64 form: Neumaier-compensated FP64 sums per sample.
//   mixed form: Kahan-compensated FP32 sums per sample, folded every FT_FOLD samples
//   (and at the end) into one double-double sum per warp.  A Kahan sum's error does not
//   grow with the number of terms, so the fold only has to be rare enough to cost
//   nothing; one FP64 sum per warp instead of two FP64 words per thread leaves the
//   shared memory to the cut thresholds (the cube's block: 40 KB of sums instead of 123).
// Slots: 4 per eps order (re f, re f^2, im f, im f^2).
// Dropped, queued, exact and robust samples are rare and counted per block; kept is what
// remains of the samples the block owns.
#if FT_MODE == 0
#define ACC_PARTS 2   // undeformed integrand: real parts only
#else
#define ACC_PARTS 4
#endif
#define ACC_NS (ACC_PARTS * FT_K)
#define ACC_SMEM_OFFSET ((SM_USED + 15u) & ~15u)
#define FT_WARPS (FT_BLOCK / 32)
#define FT_FOLD 1024
#if FT_PREC == 1
// after the sums: the threads' log X (draw_pair), two floats per edge and sample
#define LX_SMEM_OFFSET ((ACC_SMEM_OFFSET + 16u * ACC_NS * FT_WARPS + 8u * ACC_NS * FT_BLOCK + 15u) & ~15u)
#else
#define LX_SMEM_OFFSET 0u
#endif

enum { CNT_OWNED, CNT_DROPPED, CNT_QUEUED, CNT_EXACT, CNT_ROBUST, CNT_N };
__shared__ u64 s_count[CNT_N];

// slot s = (order j, part q) -> output pair 4 j + q
static __device__ __forceinline__ int out_pair(int s) { return 4 * (s / ACC_PARTS) + (s % ACC_PARTS); }

// the block's counters and the output slots no sum is kept for (the first threads)
static __device__ __forceinline__ void write_counts(double* dst)
{
    for (int s = threadIdx.x; s < ACC_SLOTS; s += FT_BLOCK) {
        if (s < 8 * FT_K) {
            if (ACC_PARTS == 2 && (s & 4)) dst[s] = 0.0;
            continue;
        }
        double v = 0.0;
        if (s == ACC_KEPT) v = (double)(s_count[CNT_OWNED] - s_count[CNT_DROPPED] - s_count[CNT_QUEUED]);
        if (s == ACC_DROPPED) v = (double)s_count[CNT_DROPPED];
        if (s == ACC_QUEUED) v = (double)s_count[CNT_QUEUED];
        if (s == ACC_EXACT) v = (double)s_count[CNT_EXACT];
        if (s == ACC_ROBUST) v = (double)s_count[CNT_ROBUST];
        dst[s] = v;
    }
}

// (h, l) += (bh, bl): h the rounded sum, the errors collected in l and not renormalised, so
// that a chain of additions waits for one FP64 addition per term (the FP64 pipe takes 16
// cycles per warp instruction)
static __device__ __forceinline__ void dd_acc(double& h, double& l, double bh, double bl)
{
    const double s = h + bh, bb = s - h;
    l += ((h - (s - bb)) + (bh - bb)) + bl;
    h = s;
}
static __device__ __forceinline__ void dd_norm(double& h, double& l)
{
    const double s = h + l;
    l = l - (s - h);
    h = s;
}
static __device__ __forceinline__ void warp_dd_sum(double& h, double& l)
{
#pragma unroll 1
    for (int off = 16; off; off >>= 1) {
        const double oh = __shfl_down_sync(0xffffffffu, h, off), ol = __shfl_down_sync(0xffffffffu, l, off);
        dd_acc(h, l, oh, ol);
    }
    dd_norm(h, l);
}

// Sum of n pairs x[k step] + x[k step + second] by a warp, in every lane: integers of 128 bits
// relative to the largest exponent (114 bits below it), so that the order does not matter and
// the FP64 pipe is left alone, on which each of a double-double tree's additions takes 7 times
// 16 cycles of the SM.  False where that does not hold: infinite or NaN terms, more than 2048
// pairs.  GLOBAL: x was written by other blocks.
template <bool GLOBAL>
static __device__ __noinline__ bool fixed_sum(const double* x, u32 step, u32 second, u32 n, double& h, double& l)
{
    const u32 lane = threadIdx.x & 31u;
    auto word = [&](u32 i) -> u64 {
        return (u64)(GLOBAL ? __ldcg((const long long*)x + i) : ((const long long*)x)[i]);
    };
    u32 top = 0;
    for (u32 k = lane; k < n; k += 32u)
        top = max(top, max((u32)(word(k * step) >> 52) & 2047u, (u32)(word(k * step + second) >> 52) & 2047u));
    const int emax = max(1, (int)__reduce_max_sync(0xffffffffu, top));
    if (emax == 2047 || n > 2048u) return false;
    u64 lo = 0, hi = 0;
    for (u32 k = lane; k < n; k += 32u)
#pragma unroll
        for (u32 i = 0; i < 2; i++) {
            const u64 b = word(k * step + (i ? second : 0u));
            const int e = (int)(b >> 52) & 2047, sh = 61 - emax + (e ? e : 1);
            const u64 m = (b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
            u64 ml = sh >= 0 ? m << sh : sh > -64 ? m >> -sh : 0ull, mh = sh > 0 ? m >> (64 - sh) : 0ull;
            if ((long long)b < 0) {
                ml = 0ull - ml;
                mh = ~mh + (ml == 0ull);
            }
            lo += ml;
            hi += mh + (lo < ml);
        }
#pragma unroll 1
    for (int off = 16; off; off >>= 1) {
        const u64 ol = __shfl_xor_sync(0xffffffffu, lo, off), oh = __shfl_xor_sync(0xffffffffu, hi, off);
        lo += ol;
        hi += oh + (lo < ol);
    }
    // hi 2^64 + lo to double-double; |hi| < 2^62
    const long long sh = (long long)hi;
    h = (double)sh;
    l = (double)(sh - (long long)h) + (double)lo * 0x1p-64;
    const int q = emax - 1075 - 61 + 64;   // of the value's 2^64
    h = ldexp(h, q);
    l = ldexp(l, q);
    dd_norm(h, l);
    return true;
}

struct accum {
    unsigned char* base;

    __device__ __forceinline__ void count(int c, u32 n)
    {
        if (n) atomicAdd(&s_count[c], (u64)n);
    }
    // A warp's threads first: a 64-bit addition in shared memory is a compare-and-swap loop,
    // and the block's 256 to 512 threads took 10 us of every launch and batch item in it.
    __device__ __forceinline__ void add_owned(u64 owned)
    {
        const u32 lo = __reduce_add_sync(0xffffffffu, (u32)owned & 0xffffffu);
        const u32 mid = __reduce_add_sync(0xffffffffu, (u32)(owned >> 24) & 0xffffffu);
        const u32 hi = __reduce_add_sync(0xffffffffu, (u32)(owned >> 48));
        if ((threadIdx.x & 31u) == 0) atomicAdd(&s_count[CNT_OWNED], (u64)lo + ((u64)mid << 24) + ((u64)hi << 48));
    }

#if FT_PREC == 0
    __device__ __forceinline__ double& S(int s) { return ((double*)base)[s * FT_BLOCK + threadIdx.x]; }
    __device__ __forceinline__ double& C(int s) { return ((double*)base)[(ACC_NS + s) * FT_BLOCK + threadIdx.x]; }

    // block-wide (ends with a barrier)
    __device__ __forceinline__ void init(unsigned char* smem_acc)
    {
        base = smem_acc;
#pragma unroll
        for (int s = 0; s < ACC_NS; s++) {
            S(s) = 0.0;
            C(s) = 0.0;
        }
        if (threadIdx.x < CNT_N) s_count[threadIdx.x] = 0;
        __syncthreads();
    }

    __device__ __forceinline__ void nadd(int slot, double v)
    {
        const double s = S(slot);
        const double t = s + v;
        // the larger term first, by the exponents
        const bool big = exponent_of(s) >= exponent_of(v);
        C(slot) += ((big ? s : v) - t) + (big ? v : s);
        S(slot) = t;
    }

    __device__ __forceinline__ void add64(const cx<double>* R)
    {
#pragma unroll
        for (int j = 0; j < FT_K; j++) {
            if (FT_ONLY_PSI && j > 0) break;
            nadd(ACC_PARTS * j + 0, R[j].re);
            nadd(ACC_PARTS * j + 1, R[j].re * R[j].re);
            if (ACC_PARTS == 4) {
                nadd(ACC_PARTS * j + 2, R[j].im);
                nadd(ACC_PARTS * j + 3, R[j].im * R[j].im);
            }
        }
    }

    // block-wide: every thread of the block calls it with the samples it owned; the
    // block's sums go to dst[0 .. ACC_SLOTS).  A warp takes whole slots.
    __device__ __forceinline__ void finish(double* dst, u64 owned)
    {
        add_owned(owned);
        __syncthreads();
        const int lane = threadIdx.x & 31;
#pragma unroll 1
        for (int s = threadIdx.x >> 5; s < ACC_NS; s += FT_WARPS) {
            double h = 0.0, l = 0.0;
            if (!fixed_sum<false>((const double*)base + s * FT_BLOCK, 1, ACC_NS * FT_BLOCK, FT_BLOCK, h, l)) {
                h = l = 0.0;
#pragma unroll 1
                for (int t = lane; t < FT_BLOCK; t += 32) {
                    const double sv = ((const double*)base)[s * FT_BLOCK + t];
                    const double cv = ((const double*)base)[(ACC_NS + s) * FT_BLOCK + t];
                    dd_acc(h, l, sv, cv);
                }
                warp_dd_sum(h, l);
            }
            if (lane == 0) {
                dst[2 * out_pair(s)] = h;
                dst[2 * out_pair(s) + 1] = l;
            }
        }
        write_counts(dst);
    }
#else
    // from base: the warps' double-double sums [slot][warp] (hi, lo), then Sf, Cf
    // [slot][thread]
    __device__ __forceinline__ double2& W(int s, int w) { return ((double2*)base)[s * FT_WARPS + w]; }
    __device__ __forceinline__ float& Sf(int s)
    {
        return ((float*)(base + 16 * ACC_NS * FT_WARPS))[s * FT_BLOCK + threadIdx.x];
    }
    __device__ __forceinline__ float& Cf(int s)
    {
        return ((float*)(base + 16 * ACC_NS * FT_WARPS))[(ACC_NS + s) * FT_BLOCK + threadIdx.x];
    }

    // block-wide (ends with a barrier)
    __device__ __forceinline__ void init(unsigned char* smem_acc)
    {
        base = smem_acc;
#pragma unroll
        for (int s = 0; s < ACC_NS; s++) {
            Sf(s) = 0.0f;
            Cf(s) = 0.0f;
            if ((threadIdx.x & 31) == 0) W(s, threadIdx.x >> 5) = make_double2(0.0, 0.0);
        }
        if (threadIdx.x < CNT_N) s_count[threadIdx.x] = 0;
        __syncthreads();
    }

    __device__ __forceinline__ void add32(const cx<float>* R)
    {
#pragma unroll
        for (int j = 0; j < FT_K; j++) {
            if (FT_ONLY_PSI && j > 0) break;
            const float re = R[j].re, im = R[j].im;
            const float v[4] = {re, re * re, im, im * im};
#pragma unroll
            for (int q = 0; q < ACC_PARTS; q++) {
                const int o = ACC_PARTS * j + q;
                const float sf = Sf(o);
                const float y = v[q] - Cf(o);
                const float tt = sf + y;
                Cf(o) = (tt - sf) - y;
                Sf(o) = tt;
            }
        }
    }

    // the FP32 value x in units of 2^(emax - 184) (24 bits of significand, 34 below the largest)
    static __device__ __forceinline__ long long fixed_of(float x, int emax)
    {
        const int b = __float_as_int(x), e = (b >> 23) & 255;
        const long long m = (b & 0x7fffff) | (e ? 0x800000 : 0);
        const int sh = 34 - emax + (e ? e : 1);
        const long long v = sh >= 0 ? m << sh : (sh > -32 ? m >> -sh : 0);
        return b < 0 ? -v : v;
    }
    // warp-wide: the warp's FP32 sums into its double-double ones.  The lanes' values are added
    // as integers, 58 bits below the largest: the FP64 pipe takes 16 cycles of the whole SM
    // per warp instruction, and a double-double tree over the lanes kept a small launch's
    // 16 warps at its end for 130 us (11 now).
    __device__ __noinline__ void fold()
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
        for (int s0 = 0; s0 < ACC_NS; s0 += 32) {
            long long mine = 0;
            int emine = 0;
            bool slow = false;
#pragma unroll 1
            for (int i = 0; i < 32 && s0 + i < ACC_NS; i++) {
                const float a = Sf(s0 + i), c = Cf(s0 + i);
                const u32 ea = ((u32)__float_as_int(a) >> 23) & 255u, ec = ((u32)__float_as_int(c) >> 23) & 255u;
                const int emax = (int)__reduce_max_sync(0xffffffffu, ea > ec ? ea : ec);
                if (emax == 255) {
                    slow = true;   // infinite or NaN sums: below
                    continue;
                }
                long long v = fixed_of(a, emax) - fixed_of(c, emax);
#pragma unroll
                for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == i) {
                    mine = v;
                    emine = emax;
                }
            }
            if (s0 + lane < ACC_NS) {
                const double unit = __longlong_as_double((long long)(emine - 184 + 1023) << 52);
                const double h = (double)mine, l = (double)(mine - (long long)h);
                double2 w = W(s0 + lane, warp);
                dd_acc(w.x, w.y, h * unit, l * unit);
                W(s0 + lane, warp) = w;
            }
            __syncwarp();
#pragma unroll 1
            for (int i = 0; slow && i < 32 && s0 + i < ACC_NS; i++) {
                const float a = Sf(s0 + i), c = Cf(s0 + i);
                if (__any_sync(0xffffffffu, !isfinite(a) || !isfinite(c))) {
                    double h = (double)a - (double)c, l = 0.0;
                    warp_dd_sum(h, l);
                    if (lane == 0) {
                        double2 w = W(s0 + i, warp);
                        dd_acc(w.x, w.y, h, l);
                        W(s0 + i, warp) = w;
                    }
                }
            }
        }
#pragma unroll 1
        for (int s = 0; s < ACC_NS; s++) {
            Sf(s) = 0.0f;
            Cf(s) = 0.0f;
        }
    }

    // block-wide: every thread of the block calls it with the samples it owned; the
    // block's sums go to dst[0 .. ACC_SLOTS)
    __device__ __forceinline__ void finish(double* dst, u64 owned)
    {
        add_owned(owned);
        fold();
        __syncthreads();
        for (int s = threadIdx.x; s < ACC_NS; s += FT_BLOCK) {
            double2 w = W(s, 0);
#pragma unroll 1
            for (int k = 1; k < FT_WARPS; k++) {
                const double2 v = W(s, k);
                dd_acc(w.x, w.y, v.x, v.y);
            }
            dd_norm(w.x, w.y);
            dst[2 * out_pair(s)] = w.x;
            dst[2 * out_pair(s) + 1] = w.y;
        }
        write_counts(dst);
    }
#endif
};

#if !FT_BATCH
// The launch's sums, by the block that finishes last: parts [p0, p1) added into out, a warp
// per slot (the moments in double-double).  `ticket` counts the finished blocks and wraps
// to zero for the next launch.
static __device__ __forceinline__ bool last_block(unsigned int* ticket)
{
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(ticket, gridDim.x - 1u) == gridDim.x - 1u;
    __syncthreads();
    __threadfence();
    return last;
}
// unit u of the sums (a moment's pair, or a counter) over n parts, by a warp; in lane 0
#define FT_UNITS (4 * FT_K + 5)
static __device__ __noinline__ void sum_unit(int u, const double* parts, unsigned int n, double& h, double& l)
{
    const unsigned int lane = threadIdx.x & 31u;
    const bool pair = u < 4 * FT_K;
    const double* v = parts + (pair ? 2 * u : 4 * FT_K + u);
    h = l = 0.0;
    if (ACC_PARTS == 2 && pair && (u & 2)) return;   // no imaginary parts
    if (pair) {
        if (fixed_sum<true>(v, ACC_SLOTS, 1, n, h, l)) return;
        h = l = 0.0;
#pragma unroll 4
        for (unsigned int k = lane; k < n; k += 32u)
            dd_acc(h, l, __ldcg(v + (size_t)k * ACC_SLOTS), __ldcg(v + (size_t)k * ACC_SLOTS + 1));
        warp_dd_sum(h, l);
    } else {   // whole numbers below 2^52: their integers from the bits
        u64 c = 0;
        for (unsigned int k = lane; k < n; k += 32u)
            c += (u64)__double_as_longlong(__ldcg(v + (size_t)k * ACC_SLOTS) + 0x1p52) & 0xfffffffffffffull;
#pragma unroll
        for (int off = 16; off; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
        h = (double)c;
    }
}
static __device__ __forceinline__ void write_unit(int u, double h, double l, double* out)
{
    if (u < 4 * FT_K) {
        out[2 * u] = h;
        out[2 * u + 1] = l;
    } else {
        out[4 * FT_K + u] = h;
    }
}
static __device__ __forceinline__ void sum_parts(const double* parts, unsigned int n, double* out)
{
#pragma unroll 1
    for (int u = threadIdx.x >> 5; u < FT_UNITS; u += FT_WARPS) {
        double h, l;
        sum_unit(u, parts, n, h, l);
        if ((threadIdx.x & 31u) == 0) write_unit(u, h, l, out);
    }
    if (threadIdx.x < 3) out[8 * FT_K + 5 + threadIdx.x] = 0.0;
}
#endif

template <class T>
static __device__ __forceinline__ void write_record(u64 i, const unsigned char* ord, const cx<T>* R, bool ok,
                                                    unsigned char flags, unsigned char* rec_order, double* rec_R,
                                                    unsigned char* rec_flags)
{
    for (int e = 0; e < FT_E; e++) rec_order[i * FT_E + e] = ord[e];
    for (int j = 0; j < FT_K; j++) {
        rec_R[(i * FT_K + j) * 2] = ok ? (double)R[j].re : 0.0;
        rec_R[(i * FT_K + j) * 2 + 1] = ok ? (double)R[j].im : 0.0;
    }
    rec_flags[i] = flags;
}

#if FT_PREC == 0
// one sample in FP64 from stream state g (advanced past the sample's 2E-1 draws)
template <bool COLD>
static __device__ __forceinline__ void sample64(xo& g, const table_ref& tr, const double* prm, u64 i, accum& A,
                                                unsigned char flags, unsigned char* rec_order, double* rec_X,
                                                double* rec_R, unsigned char* rec_flags)
{
    unsigned char ord[FT_E];
    cx<double> R[FT_K];
#pragma unroll
    for (int j = 0; j < FT_K; j++) R[j] = cmk(0.0, 0.0);
    double X[FT_E];
    double F, Gv;
    draw_sector64<COLD>(g, tr, FT_EXACT_TABLE(tr), prm[P_JRFULL], X, F, Gv, ord);
    if (FT_RECORD)
        for (int e = 0; e < FT_E; e++) rec_X[i * FT_E + e] = X[e];
    bool rob = false;
    const bool ok = integrand64<COLD>(prm, X, F, Gv, g, FT_EXACT_TABLE(tr), R, rob);
    if (rob) {
        A.count(CNT_ROBUST, 1);
        flags |= REC_ROBUST;
    }
    if (!ok) {
        A.count(CNT_DROPPED, 1);
        flags |= REC_DROPPED;
    } else {
        A.add64(R);
    }
    if (FT_RECORD) write_record(i, ord, R, ok, flags, rec_order, rec_R, rec_flags);
}
#endif

// ------------------------------------------------------------------ one thread's samples
// Samples [first, last) of the stream, g holding the state of sample `first`.  In the
// mixed form, samples whose FP32 evaluation is not trustworthy are queued for the FP64
// pass and left out of the sums here: 5 words, the sample (its index in the
// single-integral kernels; item << BQ_ITEM_SHIFT | lane << BQ_LANE_SHIFT | (i - first)
// naming the block's work item in the batch kernels) and its stream state.
// Every thread of the block makes `chunk` trips (two samples a trip in the
// undeformed mixed form).  With the barrier (FT_VARIANT bit 2) the block starts each trip together: the
// warps then run the same stretch of the (long, straight-line) per-sample code at the
// same time and share its instruction fetches.
#if FT_PREC == 1
static __device__ __noinline__ void queue_sample(xo g, u64 i, u64 offset, u64* __restrict__ queue,
                                                 unsigned int* __restrict__ qcount, unsigned int qcap, int back)
{
    const unsigned int slot = atomicAdd(qcount, 1u);
    if (slot >= qcap) return;
    rewind(g, back);   // to the sample's first draw
    u64* q = queue + (size_t)slot * 5;
#if FT_BATCH
    q[0] = (s_batch_item << BQ_ITEM_SHIFT) | ((u64)threadIdx.x << BQ_LANE_SHIFT) | offset;
#else
    q[0] = i;
#endif
    q[1] = g.a;
    q[2] = g.b;
    q[3] = g.c;
    q[4] = g.d;
}
#endif

static __device__ __forceinline__ void sample_range(xo& g, const table_ref& tr, const double* __restrict__ prm,
                                                    u64 first, u64 last, u64 chunk, accum& A, unsigned char* lxs,
                                                    u64* __restrict__ queue, unsigned int* __restrict__ qcount,
                                                    unsigned int qcap, unsigned char* __restrict__ rec_order,
                                                    double* __restrict__ rec_X, double* __restrict__ rec_R,
                                                    unsigned char* __restrict__ rec_flags)
{
#if FT_PREC == 0
    (void)lxs;
    for (u64 k = 0; k < chunk; k++) {
#if FT_VARIANT & 4
        __syncthreads();
#endif
        const u64 i = first + k;
        if (i >= last) continue;
        sample64<false>(g, tr, prm, i, A, 0, rec_order, rec_X, rec_R, rec_flags);
    }
#else
    const float* pf = (const float*)(prm + P_SIZE);
    const float4* pp = (const float4*)(prm + P_PAIR);
    const int per = FT_MODE == 0 ? 2 : 1;   // samples of a trip
    for (u64 k = 0; k < chunk; k += per) {
#if FT_VARIANT & 4
        __syncthreads();
#endif
        if ((k & (FT_FOLD - 1)) == FT_FOLD - per) A.fold();
        const u64 i = first + k;
        if (i >= last) continue;
        unsigned char ord[2][FT_E];
        cx<float> r[2][FT_K];
        u32 ex[2] = {0, 0};
        bool bad[2] = {true, true};
#pragma unroll
        for (int j = 0; j < FT_K; j++) r[0][j] = r[1][j] = cmk(0.0f, 0.0f);
#if FT_MODE == 0
        const int n = i + 1 < last ? 2 : 1;   // the second half of an odd last sample's pair is left out
        df lF, lG;
        fv R[FT_K];
#pragma unroll
        for (int j = 0; j < FT_K; j++) R[j] = fv_of(0.0f);
        draw_pair(g, tr, lxs, lF, lG, ex[0], ex[1], ord[0], ord[1]);
#else
        const int n = 1;
        sf lF, lG;
        draw_one(g, tr, lxs, lF, lG, ex[0], ord[0]);
#endif
        if (FT_RECORD)
            for (int e = 0; e < FT_E; e++) {
#if FT_MODE == 0
                rec_X[i * FT_E + e] = exp((double)LX(e, 0).x + (double)LX(e, 1).x);
                if (n > 1) rec_X[(i + 1) * FT_E + e] = exp((double)LX(e, 0).y + (double)LX(e, 1).y);
#else
                rec_X[i * FT_E + e] = exp((double)LX(e, 0) + (double)LX(e, 1));
#endif
            }
#if FT_MODE == 0
        integrand_pair(pp, pf, lxs, lF, lG, R, bad[0], bad[1]);
#pragma unroll
        for (int j = 0; j < FT_K; j++) {
            r[0][j].re = R[j].x;
            r[1][j].re = R[j].y;
        }
#else
        bad[0] = !integrand_one(pp, pf, lxs, lF, lG, r[0]);
#endif
#pragma unroll
        for (int h = 0; h < per; h++) {
            if (h >= n) break;
            A.count(CNT_EXACT, ex[h]);
            if (bad[h]) {
                A.count(CNT_QUEUED, 1);
                queue_sample(g, i + h, k + h, queue, qcount, qcap, (per - h) * (2 * FT_E - 1));
            } else {
                A.add32(r[h]);
            }
            if (FT_RECORD)
                write_record(i + h, ord[h], r[h], !bad[h],
                             (unsigned char)((bad[h] ? REC_QUEUED : 0) | (ex[h] ? REC_EXACT : 0)), rec_order, rec_R,
                             rec_flags);
        }
    }
#endif
}

#if !FT_BATCH
#if !FT_PART
// ------------------------------------------------------------------ single-integral kernels
// Thread t of the launch owns samples [t*chunk, min(nsamples, (t+1)*chunk)) counted
// from the launch's first sample, whose stream state is (s0 .. s3).  Block b writes its
// partial sums to acc_out[b * ACC_SLOTS ...]; the last one to finish adds them into
// final_out (NULL in the mixed form, whose FP64 pass does it).
extern "C" __global__ void __launch_bounds__(FT_BLOCK, FT_MINB) ft_sample(
    const double* __restrict__ prm, const unsigned char* __restrict__ tab, const u64* __restrict__ mats, int digits,
    u64 s0, u64 s1, u64 s2, u64 s3, u64 nsamples, u64 chunk, double* acc_out, u64* __restrict__ queue,
    unsigned int* __restrict__ qcount, unsigned int qcap, unsigned int* __restrict__ ticket, double* final_out,
    unsigned char* __restrict__ rec_order, double* __restrict__ rec_X, double* __restrict__ rec_R,
    unsigned char* __restrict__ rec_flags)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const table_ref tr = stage_table(smem, tab);

    const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    xo g;
    g.a = s0;
    g.b = s1;
    g.c = s2;
    g.d = s3;
    g = start_state(g, mats, t, digits);

    u64 first = (u64)t * chunk;
    u64 last = first + chunk;
    if (last > nsamples) last = nsamples;

    accum A;
    A.init(smem + ACC_SMEM_OFFSET);
    sample_range(g, tr, prm, first, last, chunk, A, smem + LX_SMEM_OFFSET, queue, qcount, qcap, rec_order, rec_X,
                 rec_R, rec_flags);
    A.finish(acc_out + (size_t)blockIdx.x * ACC_SLOTS, first < last ? last - first : 0);
    if (final_out && last_block(ticket)) sum_parts(acc_out, gridDim.x, final_out);
}

#elif FT_PREC == 0
// FP64 pass over the samples a mixed launch queued (grid-stride over the entries).  The
// blocks with entries add their sums after the nparts of the sampling launch in acc_out.
// Meanwhile the last blocks add those parts (a unit of the sums each, one warp: the FP64
// pipe is the bound) into the part after all of them, so that the block that finishes last
// has only this one and the few with entries to add into final_out; it clears the count.
extern "C" __global__ void __launch_bounds__(FT_BLOCK) ft_sample_queue(
    const double* __restrict__ prm, const unsigned char* __restrict__ tab, const u64* __restrict__ queue,
    unsigned int* __restrict__ qcount, unsigned int qcap, double* acc_out, unsigned int nparts,
    unsigned int* __restrict__ ticket, double* final_out, unsigned char* __restrict__ rec_order,
    double* __restrict__ rec_X, double* __restrict__ rec_R, unsigned char* __restrict__ rec_flags)
{
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned int n = *qcount;
    if (n > qcap) n = qcap;
    const unsigned int busy = min((n + FT_BLOCK - 1u) / FT_BLOCK, gridDim.x);   // blocks with entries
    if (blockIdx.x < busy) {
        const table_ref tr = stage_table(smem, tab);
        accum A;
        A.init(smem + ACC_SMEM_OFFSET);
        u64 owned = 0;
        for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
            const u64* q = queue + (size_t)k * 5;
            owned++;
            xo g;
            g.a = q[1];
            g.b = q[2];
            g.c = q[3];
            g.d = q[4];
            sample64<true>(g, tr, prm, q[0], A, REC_QUEUED, rec_order, rec_X, rec_R, rec_flags);
        }
        A.finish(acc_out + (size_t)(nparts + 1u + blockIdx.x) * ACC_SLOTS, owned);
    }
    // acc_out: [sampling launch's parts][their sum][the busy blocks' parts]
    if (threadIdx.x < 32) {
#pragma unroll 1
        for (int u = gridDim.x - 1u - blockIdx.x; u < FT_UNITS; u += gridDim.x) {
            double h, l;
            sum_unit(u, acc_out, nparts, h, l);
            if (threadIdx.x == 0) write_unit(u, h, l, acc_out + (size_t)nparts * ACC_SLOTS);
        }
    }
    if (last_block(ticket)) {
        const double* rest = acc_out + (size_t)nparts * ACC_SLOTS;
        if (busy == 0) {
            for (int s = threadIdx.x; s < ACC_SLOTS; s += FT_BLOCK)
                final_out[s] = s < 8 * FT_K + 5 ? __ldcg(rest + s) : 0.0;
        } else {
            sum_parts(rest, busy + 1u, final_out);
        }
        if (threadIdx.x == 0) *qcount = 0u;
    }
}
#endif

#else
// ------------------------------------------------------------------ batch kernels
// Many integrals of this topology (each with its own kinematics, table, seed and N)
// in one persistent launch.  The samples of instance i are cut into work items of
// FT_BLOCK * chunk consecutive samples; items are numbered instance after instance
// (instance i owns items [first_item, first_item + nitems)).  A block takes the next
// item from a device counter, thread t of the block owns samples
// [item_base + t*chunk, item_base + (t+1)*chunk) of the instance, and the block writes
// the item's sums to acc_out[item * ACC_SLOTS ...].  inst_state[4 i ..] is the stream state
// of instance i's first sample (computed by a preparation kernel); a warp reaches its item
// with the powers B^(8^d v) of the item stride B = T^(FT_BLOCK chunk (2E-1)) (1024 words
// each, v = 1 .. 7 per octal digit d), then its threads with the chunk's matrices
// (start_state).
struct batch_inst {
    const double* prm;          // parameter block of the instance (P_SIZE doubles, floats, two-floats)
    const unsigned char* tab;   // J(gamma) table of the instance (global layout)
    u64 nsamples;
    u64 first_item;
    u64 nitems;
    u64 pad[3];
};

// the instance owning `item`: the last instance whose first_item <= item
static __device__ __forceinline__ int find_instance(const batch_inst* __restrict__ inst, int ninst, u64 item)
{
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (inst[mid].first_item <= item)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// parameter block of the current instance, staged beside its table (P_SIZE doubles,
// the same as floats, then the two-float quadruples)
#define PRM_WORDS (P_PAIR + 2 * P_SIZE)

#if !FT_PART
extern "C" __global__ void __launch_bounds__(FT_BLOCK, FT_MINB) ft_sample_batch(
    const batch_inst* __restrict__ inst, int ninst, const u64* __restrict__ total_items,
    const u64* __restrict__ inst_state, const u64* __restrict__ item_mats, const u64* __restrict__ mats, u64 chunk,
    unsigned long long* __restrict__ counter, double* __restrict__ acc_out, u64* __restrict__ queue,
    unsigned int* __restrict__ qcount, unsigned int qcap)
{
    extern __shared__ __align__(16) unsigned char smem[];
    // the instance's table and parameters sit at fixed shared-memory addresses, so the
    // per-sample code holds no pointer to them in registers
    __shared__ __align__(16) double s_prm[PRM_WORDS];
    __shared__ int s_inst;
    int cur = -1;
#if FT_PREC == 0
    chunk = total_items[3];   // the run's, from the class's header: the launch's own is of the capture
#endif
    for (;;) {
        if (threadIdx.x == 0) {
            const u64 it = atomicAdd(counter, 1ull);
            s_batch_item = it;
            s_inst = it < *total_items ? find_instance(inst, ninst, it) : -1;
        }
        // also orders this item's staging after every thread's previous item
        __syncthreads();
        const int id = s_inst;
        if (id < 0) break;
        if (id != cur) {
            copy_table(smem, inst[id].tab);
            const double* __restrict__ src = inst[id].prm;
            for (int k = threadIdx.x; k < PRM_WORDS; k += FT_BLOCK) s_prm[k] = src[k];
            if (threadIdx.x == 0) s_batch_tab = inst[id].tab;
            __syncthreads();
            cur = id;
        }
#if FT_TABLE_GLOBAL
        const table_ref tr = table_at(smem, s_batch_tab);
#else
        const table_ref tr = table_at(smem, nullptr);
#endif
        const u64 it = s_batch_item;
        const u64 n = inst[id].nsamples;
        const u64 first = (it - inst[id].first_item) * (u64)FT_BLOCK * chunk + (u64)threadIdx.x * chunk;
        u64 last = first + chunk;
        if (last > n) last = n;
        xo g = load_state(inst_state + (size_t)id * 4);
        {
            const u64* M = item_mats;
#pragma unroll 1
            for (u64 k = it - inst[id].first_item; k; k >>= 3, M += 7u * 1024u)
                if (k & 7u) g = warp_apply(M + (size_t)((k & 7u) - 1u) * 1024u, g);
        }
        g = start_state(g, mats, threadIdx.x, 2);
        accum A;
        A.init(smem + ACC_SMEM_OFFSET);
        sample_range(g, tr, s_prm, first, last, chunk, A, smem + LX_SMEM_OFFSET, queue, qcount, qcap, nullptr, nullptr,
                     nullptr, nullptr);
        // read before the reduction's barriers, after which the first thread may take
        // the next item
        double* dst = acc_out + s_batch_item * ACC_SLOTS;
        A.finish(dst, first < last ? last - first : 0);
    }
}

#elif FT_PREC == 0
// Exact, order-independent sum of doubles: digit j of an accumulator (a signed 64-bit
// counter) weighs 2^(32 j - 1074); v = m 2^(p - 1074) with its integer significand m
// (53 bits) enters as the three 32-bit digits of m 2^(p mod 32) at digit p / 32, so
// every add is exact and integer addition makes the result independent of the order
// in which the threads' atomics land.  Non-finite values are not added (the FP64 pass
// keeps only finite samples).
static __device__ __forceinline__ void exact_add(u64* __restrict__ dig, double v)
{
    const u64 b = (u64)__double_as_longlong(v);
    const int be = (int)((b >> 52) & 0x7ffull);
    if (be == 0x7ff) return;
    u64 m = b & 0xfffffffffffffull;
    int p = 0;
    if (be) {
        m |= 1ull << 52;
        p = be - 1;
    }
    if (m == 0) return;
    const int j = p >> 5, sh = p & 31;
    const u64 lo = m << sh, hi = sh ? (m >> (64 - sh)) : 0ull;
    const bool neg = (b >> 63) != 0;
    const u64 c0 = lo & 0xffffffffull, c1 = lo >> 32;
    atomicAdd(dig + j, neg ? 0ull - c0 : c0);
    if (c1) atomicAdd(dig + j + 1, neg ? 0ull - c1 : c1);
    if (hi) atomicAdd(dig + j + 2, neg ? 0ull - hi : hi);
}

// FP64 pass over the samples a mixed batch launch queued: each entry names its work
// item (hence the instance) and carries the sample's stream state.  Each kept sample's
// values go exactly into the instance's accumulators in qacc (FT_XA_DIGITS words each):
// per eps order j accumulators 4j + 0..3 = re f, re f^2, im f, im f^2; then the
// counters kept, dropped, robust (integer atomics).
extern "C" __global__ void __launch_bounds__(FT_BLOCK) ft_sample_queue_batch(
    const batch_inst* __restrict__ inst, int ninst, const u64* __restrict__ queue,
    const unsigned int* __restrict__ qcount, unsigned int qcap, u64* __restrict__ qacc)
{
    unsigned int n = *qcount;
    if (n > qcap) n = qcap;
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const u64* q = queue + (size_t)k * 5;
        const u64 item = q[0] >> BQ_ITEM_SHIFT;
        xo g;
        g.a = q[1];
        g.b = q[2];
        g.c = q[3];
        g.d = q[4];
        const int id = find_instance(inst, ninst, item);
        const double* prm = inst[id].prm;
        const unsigned char* tab = inst[id].tab;
        const table_ref tr = global_table(tab);
        cx<double> R[FT_K];
#pragma unroll
        for (int j = 0; j < FT_K; j++) R[j] = cmk(0.0, 0.0);
        double X[FT_E];
        double F, Gv;
        unsigned char ord[FT_E];
        draw_sector64<true>(g, tr, FT_EXACT_TABLE(tr), prm[P_JRFULL], X, F, Gv, ord);
        bool rob = false;
        const bool ok = integrand64<true>(prm, X, F, Gv, g, FT_EXACT_TABLE(tr), R, rob);
        u64* qa = qacc + (size_t)id * (4 * FT_K * FT_XA_DIGITS + 4);
        u64* cnt = qa + 4 * FT_K * FT_XA_DIGITS;
        if (rob) atomicAdd(cnt + 2, 1ull);
        if (!ok) {
            atomicAdd(cnt + 1, 1ull);
            continue;
        }
        atomicAdd(cnt, 1ull);
#pragma unroll
        for (int j = 0; j < FT_K; j++) {
            if (FT_ONLY_PSI && j > 0) break;
            exact_add(qa + (4 * j + 0) * FT_XA_DIGITS, R[j].re);
            exact_add(qa + (4 * j + 1) * FT_XA_DIGITS, R[j].re * R[j].re);
            if (ACC_PARTS == 4) {
                exact_add(qa + (4 * j + 2) * FT_XA_DIGITS, R[j].im);
                exact_add(qa + (4 * j + 3) * FT_XA_DIGITS, R[j].im * R[j].im);
            }
        }
    }
}
#endif
#endif  // FT_BATCH

