// Line operators of the FP64 method in block fixed point.
//
// GB300 retires 2 FP64 lane operations per SM and clock, 64 of mad.wide.s32
// and 64 to 128 of the simple integer operations (all measured; the pipes run
// at the same time), so a line sum done in FP64 costs 27 x 64 issue cycles per
// field of a K = 5 line and the FP64 pipe is the method's bound.  The sums are
// linear maps with constant coefficients, which integer arithmetic evaluates
// as well: the values of one line (its nodes, the neighbour values at its two
// ends) are brought to one exponent, that of the largest, as 56-bit integers,
// multiplied by coefficients held as 59-bit integers, summed exactly and
// rounded once to double.
//
// Both factors are pairs of 28-bit halves held in 32 bits (h 2^28 + l), so
// that the 3 bits that sums of a line's values grow by need no carry, and a
// product is three mad.wide.s32 (the fourth, low x low, is dropped).
//
// Error: the largest of a line's values is 2^55 to 2^56 units, truncating a value
// loses less than a unit, a product drops its low x low part, a sum is floored
// once at an eighth of a unit.  In all at most 131 eighths, scaled by the row sum
// (test_fixed_line.py), that is 66 x 2^-55 of (largest value x row sum); a chain
// of K + 4 FP64 operations rounds to 2^-53 of its partial sums each time.
// Measured on lines of resolved sound waves, see fix_equation: 4 to 40 times
// below FP64 sums.
//
// The bound is one of the line, not of the row: a value more than 8 times below
// the largest keeps fewer than 53 bits, and a row that gives the largest little
// weight is the less precise for it.  Random values, each 1/8 of its neighbour
// on the line, rms error at K = 4 / 5 / 8 (FP64 sums in brackets): of the line's
// largest result 2.5e-16 / 2.5e-16 / 2.6e-16 (2.7e-16 / 2.0e-16 / 3.8e-16), of
// each row's own absolute sum 2.4e-16 / 5.0e-16 / 7.4e-16 (1.5e-16 / 1.9e-16 /
// 1.7e-16), and with lumped mass, whose inner rows do not see the neighbours,
// 5.9e-15 / 8.3e-15 / 1.9e-14 (1.1e-16 / 4.8e-15 / 1.1e-16).
//
// What fixed point cannot hold (an infinity or NaN on the line, a largest
// value outside 2^-823 .. 2^877) is left to an FP64 evaluation of that line by
// the caller; so is a line of denormals.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace dg {

// h 2^28 + l
struct FixVal {
    int h, l;
};
__host__ __device__ __forceinline__ FixVal operator+(const FixVal& a, const FixVal& b)
{
    return {a.h + b.h, a.l + b.l};
}
__host__ __device__ __forceinline__ FixVal operator-(const FixVal& a, const FixVal& b)
{
    return {a.h - b.h, a.l - b.l};
}

__host__ __device__ __forceinline__ long long fix_bits(double v)
{
#ifdef __CUDA_ARCH__
    return __double_as_longlong(v);
#else
    long long b;
    std::memcpy(&b, &v, 8);
    return b;
#endif
}

__host__ __device__ __forceinline__ double fix_double(long long b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double v;
    std::memcpy(&v, &b, 8);
    return v;
#endif
}

// High word of |v|: ordered like |v|, its exponent field in bits 20..30.
__host__ __device__ __forceinline__ int fix_abs_hi(double v) { return (int)(fix_bits(v) >> 32) & 0x7fffffff; }

// v in units of 2^(E - 1078), truncated towards zero: halves below 2^28 of
// v's sign.  E is at least v's exponent field.
__host__ __device__ __forceinline__ FixVal fix_from(double v, int E)
{
    const long long b = fix_bits(v);
    const int hi = (int)(b >> 32);
    const int sh = (int)((unsigned)((E << 20) - (hi & 0x7ff00000)) >> 20);
    unsigned long long m = (((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)b) << 3;
#ifdef __CUDA_ARCH__
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));  // amounts above 63 give 0
#else
    m = sh > 63 ? 0 : m >> sh;
#endif
    const int sign = (hi >> 31) | 1;
    FixVal x;
    x.h = (int)(m >> 28) * sign;
    x.l = (int)((unsigned)m & 0xfffffffu) * sign;
    return x;
}

// Position of the leading one, -1 for 0.
__host__ __device__ __forceinline__ int fix_top(unsigned x)
{
#ifdef __CUDA_ARCH__
    int b;
    asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(x));
    return b;
#else
    return x ? 31 - __builtin_clz(x) : -1;
#endif
}

// R 2^(e - 1085) rounded to nearest (e: the unit's exponent plus 1085), |R| <
// 2^63; the result is a normal number or zero for the exponents the callers
// admit.  Integer work alone (21 instructions; a branch for small R or
// __clzll cost 25 to 28), for kernels that need the FP64 pipe; a negative R
// counts one unit less.
__host__ __device__ __forceinline__ double fix_to(long long R, int e)
{
    const int s = (int)(R >> 63);
    const unsigned h = (unsigned)(R >> 32) ^ (unsigned)s, l = (unsigned)R ^ (unsigned)s;
    const int b = h ? fix_top(h) : fix_top(l) - 32;
    // leading bit to 62, round at bit 10, then 53 bits whose leading one adds
    // to the exponent field
    unsigned long long a = (((unsigned long long)h << 32) | l) << ((30 - b) & 63);
    a = (a + 512u) >> 10;
    unsigned hi = (unsigned)(a >> 32) + ((unsigned)(b + e - 31) << 20);
    hi = ((h | l) ? hi : 0u) | ((unsigned)s & 0x80000000u);
    return fix_double((long long)(((unsigned long long)hi << 32) | (unsigned)a));
}

// The same by one conversion on the FP64 pipe (7 instructions), for kernels
// that leave that pipe idle.
__host__ __device__ __forceinline__ double fix_to_fp64(long long R, int e)
{
    const long long d = fix_bits((double)R);
    return fix_double(d + (R ? (long long)(e - 1085) << 52 : 0));
}

// sum_i c_i x_i in eighths of x's unit (c in 2^-59): the cross products first,
// then the high products on top of their carry.
template <int N>
__host__ __device__ __forceinline__ long long fix_dot(const FixVal (&x)[N], const FixVal (&c)[N])
{
    long long t = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        t += (long long)x[i].h * c[i].l;
        t += (long long)x[i].l * c[i].h;
    }
    t >>= 28;
#pragma unroll
    for (int i = 0; i < N; i++) t += (long long)x[i].h * c[i].h;
    return t;
}

// The even-odd line operator, for one or two equations.  D is
// centro-antisymmetric, D[K-1-i][K-1-j] = -D[i][j], and the lift columns are
// mirrored, so with e_j = v_j + v_{K-1-j}, o_j = v_j - v_{K-1-j} (j < H = K/2)
// and the face quantities X, Y at the two ends (s: sum, d: difference) both
// outputs i and K-1-i come from the same two half-length sums:
//   P_i = sum_j E_ij e_j + Dc_i v_H + BX_i sX + BY_i dY
//   Q_i = sum_j O_ij o_j            + AX_i dX + AY_i sY
//   out_i = P_i + Q_i, out_{K-1-i} = Q_i - P_i,
//   out_H = sum_j Dm_j o_j + MX dX + MY sY   (K odd).
// The numerical flux at the left end is x X + y Y and at the right end
// -x X + y Y, with the lift columns folded in.
//
// An operator is antisymmetric to some rounding only.  What row K-1-i has beyond
// the mirror image of row i is added with the high halves alone (RP, RQ:
// integers below 2^27 of the coefficients' 2^59), so that the operator is the
// given one to its last bit, up to an asymmetry of 1e-12.  At K = 2, 3 and 5
// that work (3 to 5 % of a stage kernel) is left out where the asymmetry is no
// more than the rounding of an FP64 solve for D (fix_noise): rows i < H then
// stand for their mirror images, which at K = 3 and 5 is the closer operator
// (relative distance of the library's D from the exact one, mirrored / as
// solved: 2.7e-16 / 5.0e-16 and 7.8e-16 / 1.6e-15; K = 2: 5.2e-16 / 4.9e-16).
// At K = 4, 7, 8 the solved one is (5.3e-16 / 4.9e-16, 1.1e-15 / 9.9e-16,
// 2.7e-15 / 2.5e-15).
__host__ __device__ constexpr bool fix_rest(int K) { return K == 4 || K > 5; }
// The library's operators, exact and lumped, are off by up to 1.5e-16 (K = 2),
// 1.1e-15 (K = 3) and 1.7e-15 (K = 5) of the largest entry.
constexpr double fix_noise(int K) { return K == 2 ? 0x1p-51 : 0x1p-48; }

template <int K, int NEQ>
struct FixLine {
    static constexpr int H = K / 2, ODD = K & 1, NP = H + ODD + NEQ, NQ = H + NEQ;
    // rows (E_i, Dc_i, BX_i, BY_i), (O_i, AX_i, AY_i), (Dm, MX, MY); no Y with one equation
    FixVal P[NEQ][H][NP], Q[NEQ][H][NQ], M[NEQ][NQ];
    int RP[NEQ][H + ODD][NP], RQ[NEQ][H][NQ];
    int rest;        // RP and RQ apply (always with fix_rest)
    int e_out[NEQ];  // output unit's exponent, plus 1085, relative to the line's exponent
};

// A kernel's operator: the line of axis 0 (a kernel parameter, so that its
// coefficients are constant-bank operands), which serves the other axes too:
// theirs differ by the factor 1/w_a alone, applied to the results where the
// element is not a cube.
template <int K, int NEQ>
struct FixOps {
    FixLine<K, NEQ> line;
    double ws[3];  // w_0 / w_a
    int pm;        // jumps enter the other equation scaled by 2^pm (make_stage_fix)
    int cube;      // ws is 1
};

// Outputs emit(i, out_i), i = 0..K-1, from node values v (sums of at most two
// fix_from values) and face quantities (X at most four, Y at most two).  An
// output is handed over as soon as it is known, so that no register holds it.
// REST: whether RP and RQ apply, 2 where L.rest says so: as a branch that costs
// a stage launch 1 % at most and a gradient launch 8 to 11 % (K = 3, 5).
template <int K, int NEQ, int REST = 2, typename Emit>
__host__ __device__ __forceinline__ void fix_line(const FixLine<K, NEQ>& L, int eq, const FixVal (&v)[K],
                                                  const FixVal& X0, const FixVal& XN, const FixVal& Y0,
                                                  const FixVal& YN, Emit emit)
{
    using F = FixLine<K, NEQ>;
    constexpr int H = F::H, ODD = F::ODD, NP = F::NP, NQ = F::NQ;
    const bool rest = fix_rest(K) || (REST == 2 ? L.rest != 0 : REST != 0);
    FixVal p[NP], q[NQ];
#pragma unroll
    for (int j = 0; j < H; j++) {
        p[j] = v[j] + v[K - 1 - j];
        q[j] = v[j] - v[K - 1 - j];
    }
    if (ODD) p[H] = v[H];
    p[H + ODD] = X0 + XN;
    q[H] = X0 - XN;
    if (NEQ > 1) {
        p[NP - 1] = Y0 - YN;
        q[NQ - 1] = Y0 + YN;
    }
#pragma unroll
    for (int i = 0; i < H; i++) {
        const long long P = fix_dot(p, L.P[eq][i]), Q = fix_dot(q, L.Q[eq][i]);
        emit(i, P + Q);
        long long t = 0;
        if (rest) {
#pragma unroll
            for (int j = 0; j < NP; j++) t += (long long)p[j].h * L.RP[eq][i][j];
#pragma unroll
            for (int j = 0; j < NQ; j++) t += (long long)q[j].h * L.RQ[eq][i][j];
        }
        emit(K - 1 - i, Q - P + (t >> 28));
    }
    if (ODD) {
        long long t = 0;
        if (rest) {
#pragma unroll
            for (int j = 0; j < NP; j++) t += (long long)p[j].h * L.RP[eq][H][j];
        }
        emit(H, fix_dot(q, L.M[eq]) + (t >> 28));
    }
}

// Exponent fields of a line's largest value that fixed point takes.
constexpr int kFixMinExp = 200, kFixMaxExp = 1900;

__host__ __device__ __forceinline__ int fix_max(int a, int b) { return a > b ? a : b; }

// fix_abs_hi of a value in memory, of which it reads the high word alone, so
// that no value is held while a line's others are read.
__host__ __device__ __forceinline__ int fix_abs_hi_at(const double* p)
{
#ifdef __CUDA_ARCH__
    return reinterpret_cast<const int*>(p)[1] & 0x7fffffff;
#else
    return fix_abs_hi(*p);
#endif
}

// One equation of a line: outputs out[i st] from the node values v[j st]
// (+ w[j st] with TWO), their counterparts vo (+ wo) across the two ends and
// the jumps y across them that enter with the factor 2^py (FixFlux).  v, w and
// out may be the same memory.  The exponent is that of the largest of these
// values alone: an equation's sums keep their bits however large the other
// equation's fluxes are, of which it sees no more than the jumps, formed in
// FP64.  One exponent for both equations needs no FP64 subtractions and fewer
// conversions (us per stage launch on 8 M nodes, K = 2 .. 8: 359 / 361 / 300 / 337 /
// 352 / 389 / 384, this form 439 / 389 / 330 / 362 / 380 / 410 / 419; at rest 363 /
// 346 / 269 / 297 / 281 / 301 / 287 and 375 / 372 / 313 / 323 / 310 / 310 / 320), but
// loses the smaller flux: 5e-8 of the momentum sums at 1e-8 of a sound wave's
// density.  Lines of resolved sound waves (3 to 12 elements long), rms error of
// a sum in units of its own absolute sum, K = 2 .. 8: one exponent 3.7e-16 /
// 3.4e-16 / 5.6e-16 / 8.1e-16 / 6.0e-16 / 1.3e-15 / 2.8e-15, this form 1.2e-17 /
// 7.5e-17 / 1.9e-17 / 2.4e-17 / 2.1e-17 / 4.2e-17 / 4.1e-17, FP64 sums 5.2e-16 /
// 4.8e-16 / 3.0e-16 / 2.6e-16 / 2.6e-16 / 2.3e-16 / 4.0e-16.
// False, and nothing written, when fixed point cannot hold the values (zeros it
// can).
template <int K, bool TWO>
__host__ __device__ __forceinline__ bool fix_equation(const FixLine<K, 2>& L, int eq, int py, const double* v,
                                                      const double* w, int st, const double (&vo)[2],
                                                      const double (&wo)[2], double y0, double yN, double* out)
{
    int t = fix_max(fix_abs_hi(vo[0]), fix_abs_hi(vo[1]));
    if (TWO) t = fix_max(t, fix_max(fix_abs_hi(wo[0]), fix_abs_hi(wo[1])));
#pragma unroll
    for (int j = 0; j < K; j++) {
        t = fix_max(t, fix_abs_hi_at(v + j * st));
        if (TWO) t = fix_max(t, fix_abs_hi_at(w + j * st));
    }
    const int ty = fix_max(fix_abs_hi(y0), fix_abs_hi(yN)), E = fix_max(t >> 20, (ty >> 20) - py);
    if (E < kFixMinExp || E > kFixMaxExp) {
        // zeros are all there is ahead of a wave: no arithmetic for them
        if ((t | ty) != 0) return false;
        int low = (int)(fix_bits(vo[0]) | fix_bits(vo[1]) | fix_bits(y0) | fix_bits(yN));
        if (TWO) low |= (int)(fix_bits(wo[0]) | fix_bits(wo[1]));
#pragma unroll
        for (int j = 0; j < K; j++) low |= (int)(fix_bits(v[j * st]) | (TWO ? fix_bits(w[j * st]) : 0));
        if (low) return false;
#pragma unroll
        for (int j = 0; j < K; j++) out[j * st] = 0.0;
        return true;
    }
    FixVal x[K], X0 = fix_from(vo[0], E), XN = fix_from(vo[1], E);
#pragma unroll
    for (int j = 0; j < K; j++) x[j] = fix_from(v[j * st], E);
    if (TWO) {
        X0 = X0 + fix_from(wo[0], E);
        XN = XN + fix_from(wo[1], E);
#pragma unroll
        for (int j = 0; j < K; j++) x[j] = x[j] + fix_from(w[j * st], E);
    }
    const int eo = E + L.e_out[eq];
    fix_line<K, 2>(L, eq, x, X0 + x[0], XN + x[K - 1], fix_from(y0, E + py), fix_from(yN, E + py),
                   [&](int i, long long o) { out[i * st] = fix_to(o, eo); });
    return true;
}

// ------------------------------------------------------------------ host
// The operator from rows (D_i0..D_i,K-1, L0_i, LN_i) and, per equation, the
// flux factors x, y (value x X + y Y at the left end, -x X + y Y at the right;
// with sig < 0 the right value is x X and Y is not used) and the power of two
// by which Y's scale differs: coefficients of D and X enter times 2^-r, of Y
// times 2^(py - r).  False when the rows are not mirror symmetric
// (D_{K-1-i,K-1-j} = -D_ij, L0_{K-1-i} = sig LN_i, to 1e-12 of the largest) or
// the scale is out of range: the caller then keeps the FP64 kernels.
struct FixFlux {
    double x, y;
    int py;
};

// Coefficients as unevaluated sums of two doubles: halves of sums of rows and
// their products with the flux factors keep the bits that 2^-59 can hold.
struct FixSum {
    double hi, lo;
    FixSum() = default;
    FixSum(double a) : hi(a), lo(0.0) {}
    FixSum(double a, double b) : hi(a), lo(b) {}
};
inline FixSum fix_half_sum(double a, double b)
{
    const double s = a + b, t = s - a;
    return {0.5 * s, 0.5 * ((a - (s - t)) + (b - t))};
}
inline FixSum operator*(const FixSum& a, double b)
{
    const double p = a.hi * b;
    return {p, std::fma(a.hi, b, -p) + a.lo * b};
}
inline long long fix_coef(const FixSum& c, double scale)  // scale: a power of two
{
    return (long long)std::llrint(c.hi * scale) + (long long)std::llrint(c.lo * scale);
}
inline FixVal fix_split(long long c)
{
    FixVal v;
    v.h = (int)((c + (1 << 27)) >> 28);  // balanced: -2^27 <= l < 2^27
    v.l = (int)(c - (long long)v.h * (1 << 28));
    return v;
}

template <int K, int NEQ, typename Row>
inline bool fix_axis(const Row* rows, int sig, const FixFlux (&f)[NEQ], FixLine<K, NEQ>& L)
{
    using F = FixLine<K, NEQ>;
    constexpr int H = F::H, ODD = F::ODD, NP = F::NP, NQ = F::NQ;
    double dmax = 0.0, lmax = 0.0;
    for (int i = 0; i < K; i++) {
        for (int j = 0; j < K; j++) dmax = std::fmax(dmax, std::fabs(rows[i][j]));
        lmax = std::fmax(lmax, std::fmax(std::fabs(rows[i][K]), std::fabs(rows[i][K + 1])));
    }
    if (!std::isfinite(dmax) || !std::isfinite(lmax)) return false;
    auto symmetric = [&](double tol) {
        for (int i = 0; i < K; i++) {
            for (int j = 0; j < K; j++)
                if (!(std::fabs(rows[i][j] + rows[K - 1 - i][K - 1 - j]) <= tol * dmax)) return false;  // NaN too
            if (!(std::fabs(rows[K - 1 - i][K] - sig * rows[i][K + 1]) <= tol * lmax)) return false;
        }
        return true;
    };
    if (!symmetric(1e-12)) return false;
    L.rest = fix_rest(K) || !symmetric(fix_noise(K));
    // Row i as coefficients of the even part (e, v_H, sX, dY) and of the odd
    // part (o, dX, sY) of equation q.
    double y[NEQ];
    for (int q = 0; q < NEQ; q++) y[q] = std::ldexp(f[q].y, f[q].py);
    auto parts = [&](int q, int i, FixSum p[], FixSum o[]) {
        for (int j = 0; j < H; j++) {
            p[j] = fix_half_sum(rows[i][j], rows[i][K - 1 - j]);
            o[j] = fix_half_sum(rows[i][j], -rows[i][K - 1 - j]);
        }
        if (ODD) p[H] = rows[i][H];
        const FixSum A = fix_half_sum(rows[i][K], sig * rows[i][K + 1]), B = fix_half_sum(rows[i][K], -sig * rows[i][K + 1]);
        p[H + ODD] = B * f[q].x;
        o[H] = A * f[q].x;
        if (NEQ > 1) {
            p[NP - 1] = B * y[q];
            o[NQ - 1] = A * y[q];
        }
    };
    FixSum p[NP], o[NQ];
    double top = 0.0;  // largest row sum
    for (int q = 0; q < NEQ; q++)
        for (int i = 0; i < K; i++) {
            double sp = 0.0, so = 0.0;
            parts(q, i, p, o);
            for (int j = 0; j < NP; j++) sp += std::fabs(p[j].hi);
            for (int j = 0; j < NQ; j++) so += std::fabs(o[j].hi);
            top = std::fmax(top, std::fmax(sp, so));
        }
    if (!std::isfinite(top)) return false;
    int r = 0;
    if (top > 0.0) {
        std::frexp(2.02 * top, &r);  // row sums below 2^r / 2.02
        if (r < -80 || r > 80) return false;
    }
    const double scale = std::ldexp(1.0, 59 - r);
    for (int q = 0; q < NEQ; q++) {
        long long cp[K][NP], co[K][NQ];
        for (int i = 0; i < K; i++) {
            parts(q, i, p, o);
            for (int j = 0; j < NP; j++) cp[i][j] = fix_coef(p[j], scale);
            for (int j = 0; j < NQ; j++) co[i][j] = fix_coef(o[j], scale);
        }
        for (int i = 0; i < H; i++) {
            for (int j = 0; j < NP; j++) {
                L.P[q][i][j] = fix_split(cp[i][j]);
                L.RP[q][i][j] = (int)(cp[K - 1 - i][j] + cp[i][j]);
            }
            for (int j = 0; j < NQ; j++) {
                L.Q[q][i][j] = fix_split(co[i][j]);
                L.RQ[q][i][j] = (int)(co[K - 1 - i][j] - co[i][j]);
            }
        }
        for (int j = 0; j < NQ; j++) L.M[q][j] = fix_split(co[H][j]);
        if (ODD)
            for (int j = 0; j < NP; j++) L.RP[q][H][j] = (int)cp[H][j];
        L.e_out[q] = r + 4;
    }
    return true;
}

}  // namespace dg
