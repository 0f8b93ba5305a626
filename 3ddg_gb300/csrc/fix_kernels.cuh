// FP64 kernels of one RK stage with the line operators in block fixed point
// (fixed_line.cuh): the LDG gradient and the stage update.  Fields, fluxes and
// the RK combination are FP64 (16 FP64 operations per node and stage), as are the
// jumps across the faces (4 per line); what is linear with constant coefficients
// (line sums, face terms, lifts) is integer work of the line owners, which runs
// beside the FP64 pipe.
//
// Mapping: a CTA takes fix_epb(K) whole elements.  In the node phases thread t
// has node t of the CTA's nodes, in the line phase line t of its lines (3 K^2
// per element), both packed densely over elements, so that small elements
// (K = 2: 8 nodes, 12 lines) fill warps too.
#pragma once

#include "dg_kernels.cuh"
#include "fixed_line.cuh"
#include "pdl.cuh"

namespace dg {

__host__ __device__ constexpr int fix_epb(int K) { return K == 2 ? 16 : K == 3 ? 9 : K <= 5 ? 2 : 1; }
__host__ __device__ constexpr int fix_threads(int K) { return (fix_epb(K) * K * K * K + 31) / 32 * 32; }
__host__ __device__ constexpr int fix_rounds(int K)
{
    return (fix_epb(K) * 3 * K * K + fix_threads(K) - 1) / fix_threads(K);
}
// Nodes in shared memory: z-lines padded to an odd length, so that the lanes
// of a warp that walk neighbouring z-lines hit different banks.
__host__ __device__ constexpr int fix_pitch(int K) { return K | 1; }
__host__ __device__ constexpr int fix_slots(int K) { return K * K * fix_pitch(K); }
template <int K>
__device__ __forceinline__ int fix_slot(int n)
{
    return (K & 1) ? n : n + n / K;
}

__device__ __forceinline__ void copy_async8(void* smem, const void* global)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Line task t of a CTA: element slot le, axis a, first node b0 (node index),
// the position fi of its ends among the K^2 nodes of their faces (the order of
// the boundary tables), and the stride st along it, sb0 and sst the same in
// shared memory.
template <int K>
struct FixTask {
    int le, a, b0, fi, st, sb0, sst;
    __device__ __forceinline__ explicit FixTask(int task)
    {
        constexpr int K2 = K * K, P = fix_pitch(K);
        le = task / (3 * K2);
        const int r = task - le * 3 * K2, t = r % K2, hi = t / K, lo = t % K;
        a = r / K2;
        // x-lines over (y, z), y-lines over (x, z), z-lines over (x, y): neighbouring
        // lanes at neighbouring z where the line allows it
        b0 = a == 0 ? t : (a == 1 ? hi * K2 + lo : t * K);
        sb0 = a == 0 ? hi * P + lo : (a == 1 ? hi * K * P + lo : t * P);
        fi = a == 1 ? lo * K + hi : t;
        st = a == 0 ? K2 : (a == 1 ? K : 1);
        sst = a == 0 ? K * P : (a == 1 ? P : 1);
    }
};

// Face-table entries of the two ends of this thread's lines.
template <int K>
__device__ __forceinline__ void fix_codes(const MeshDev<double>& m, int e0, int (&code)[fix_rounds(K)][2])
{
#pragma unroll
    for (int r = 0; r < fix_rounds(K); r++) {
        const int task = threadIdx.x + r * fix_threads(K);
        const FixTask<K> L(task);
        const bool live = task < fix_epb(K) * 3 * K * K && e0 + L.le < m.n_elem;
#pragma unroll
        for (int s = 0; s < 2; s++) code[r][s] = live ? __ldg(m.nbr + (size_t)(e0 + L.le) * 6 + 2 * L.a + s) : 0;
    }
}

// Neighbour (or exterior) values at the two ends of a line: drho
// alone, or (FLUXES) the momentum and mass fluxes f0, f1 and with WITH_Q the
// gradient qo, read from flux_in in flux mode 2 and else evaluated.
template <bool FLUXES, bool WITH_Q, int K, int FLUX = 0>
__device__ __forceinline__ void fix_end_values(const StageIO<double>& io, const MeshDev<double>& m,
                                               const OpConst<double, K>& C, const int (&code)[2],
                                               const FixTask<K>& L, double (&f0)[2], double (&f1)[2], double (&qo)[2])
{
#pragma unroll
    for (int side = 0; side < 2; side++) {
        f1[side] = qo[side] = 0.0;
        double ro, uo = 0.0;
        if (code[side] >= 0) {
            const size_t o2 = (size_t)code[side] * io.np + L.b0 + (side ? 0 : (K - 1) * L.st);
            if (WITH_Q) qo[side] = io.q[(size_t)L.a * io.fs + o2];
            if (FLUXES && FLUX == 2) {
                f0[side] = io.flux_in[o2];
                f1[side] = io.flux_in[(size_t)(1 + L.a) * io.fs + o2];
                continue;
            }
            ro = io.src[o2];
            if (FLUXES) uo = io.src[(size_t)(1 + L.a) * io.fs + o2];
        } else if (m.bnd_src) {
            exterior<double, K>(m, C, -1 - code[side], side, L.fi, ro, uo);
        } else {
            ro = 0.0;  // no boundary tables: zero outside
        }
        f0[side] = FLUXES ? momentum_flux(ro, C.k1, C.k2) : ro;
        if (FLUXES) f1[side] = mass_flux(uo, ro, C.r0, C.linear_mass);
    }
}

// ------------------------------------------------------------ LDG gradient
template <int K>
struct FixGradSmem {
    double r[fix_slots(K)];
    double g[3][fix_slots(K)];
};

// The line in FP64, for values fixed point cannot hold (and lines of zeros),
// with axis 0's operator like the fixed-point form.
template <int K>
__device__ __noinline__ void grad_line_fp64(const OpConst<double, K>& C, FixGradSmem<K>& S, int a, int sb0, int sst,
                                            double ro0, double roN)
{
    double v[K];
    long long any = fix_bits(ro0) | fix_bits(roN);
#pragma unroll
    for (int j = 0; j < K; j++) {
        v[j] = S.r[sb0 + j * sst];
        any |= fix_bits(v[j]);
    }
    if (any << 1 == 0) {  // +-0 everywhere
#pragma unroll 1
        for (int j = 0; j < K; j++) S.g[a][sb0 + j * sst] = 0.0;
        return;
    }
    const double f0 = ro0 + v[0], fN = roN + v[K - 1];
#pragma unroll 1
    for (int i = 0; i < K; i++) {
        const double* row = C.rows[0][i];
        double s = row[K] * f0;
        s += row[K + 1] * fN;
#pragma unroll
        for (int j = 0; j < K; j++) s += row[j] * v[j];
        S.g[a][sb0 + i * sst] = s;
    }
}

// REST: the operator's RP and RQ apply (K = 2, 3, 5; always at the other orders).
template <int K, bool REST>
__global__ void __launch_bounds__(fix_threads(K))
ldg_gradient_fix_kernel(StageIO<double> io, MeshDev<double> m, const __grid_constant__ OpConst<double, K> C,
                        const __grid_constant__ FixOps<K, 1> F)
{
    constexpr int K2 = K * K, K3 = K2 * K, EPB = fix_epb(K), T = fix_threads(K), RL = fix_rounds(K);
    __shared__ FixGradSmem<K> sm[EPB];
    const int tid = threadIdx.x, e0 = blockIdx.x * EPB;
    const int el = tid / K3, n = tid - el * K3;
    const bool act = el < EPB && e0 + el < m.n_elem;
    const size_t off = (size_t)(e0 + el) * io.np + n;
    int code[RL][2];
    fix_codes<K>(m, e0, code);
    pdl_wait();
    pdl_next();
    if (act) copy_async8(&sm[el].r[fix_slot<K>(n)], io.src + off);
    copy_async_commit();
    double ro[RL][2];
#pragma unroll
    for (int r = 0; r < RL; r++) {
        const int task = tid + r * T;
        ro[r][0] = ro[r][1] = 0.0;
        const FixTask<K> L(task);
        if (task >= EPB * 3 * K2 || e0 + L.le >= m.n_elem) continue;
        double unused_u[2], unused_q[2];
        fix_end_values<false, false, K>(io, m, C, code[r], L, ro[r], unused_u, unused_q);
    }
    copy_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RL; r++) {
        const int task = tid + r * T;
        const FixTask<K> L(task);
        if (task >= EPB * 3 * K2 || e0 + L.le >= m.n_elem) continue;
        FixGradSmem<K>& S = sm[L.le];
        double v[K];
        int top = max(fix_abs_hi(ro[r][0]), fix_abs_hi(ro[r][1]));
#pragma unroll
        for (int j = 0; j < K; j++) {
            v[j] = S.r[L.sb0 + j * L.sst];
            top = max(top, fix_abs_hi(v[j]));
        }
        const int E = top >> 20;
        if (E < kFixMinExp || E > kFixMaxExp) {
            grad_line_fp64<K>(C, S, L.a, L.sb0, L.sst, ro[r][0], ro[r][1]);
            continue;
        }
        FixVal x[K];
#pragma unroll
        for (int j = 0; j < K; j++) x[j] = fix_from(v[j], E);
        const int eo = E + F.line.e_out[0];
        double* out = &S.g[L.a][L.sb0];
        const FixVal X0 = fix_from(ro[r][0], E) + x[0], XN = fix_from(ro[r][1], E) + x[K - 1];
        fix_line<K, 1, REST>(F.line, 0, x, X0, XN, X0, XN,
                             [&](int i, long long o) { out[i * L.sst] = fix_to_fp64(o, eo); });
    }
    __syncthreads();
    if (!act) return;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double g = sm[el].g[a][fix_slot<K>(n)];
        io.q_out[(size_t)a * io.fs + off] = F.cube || a == 0 ? g : g * F.ws[a];
    }
}

// ------------------------------------------------------------ stage
// Per element: the volume fluxes f_mom, f_mass (x, y, z) and the gradient of
// every node; a line owner replaces its line's f_mass and gradient along its
// axis by the mass and momentum results.
template <int K>
struct FixSmem {
    double fm[fix_slots(K)];
    double fa[3][fix_slots(K)];
    double q[3][fix_slots(K)];
};

// One equation of a line in FP64, for values fixed point cannot hold, with axis
// 0's operator like the fixed-point form: v (+ w) at the line's nodes, g its
// lift-scaled face fluxes.
template <int K>
__device__ __noinline__ void stage_line_fp64(const OpConst<double, K>& C, const double* pv, const double* pw, int sst,
                                             double g0, double gN, double* out)
{
    double v[K];
#pragma unroll
    for (int j = 0; j < K; j++) v[j] = pw ? pv[j * sst] + pw[j * sst] : pv[j * sst];
#pragma unroll 1
    for (int i = 0; i < K; i++) {
        const double* row = C.rows[0][i];
        double s = row[K] * g0;
        s += row[K + 1] * gN;
#pragma unroll
        for (int j = 0; j < K; j++) s += row[j] * v[j];
        out[i * sst] = s;
    }
}

// One line of the stage: the mass equation's sums (of f_mass + G and its face
// terms) into S.fa[a], the momentum equation's into S.q[a].  With the face
// coefficients of a uniform medium the numerical fluxes are x X + y Y at the
// left and -x X + y Y at the right end (FixLine), with
//   momentum  X = f_mom' + f_mom,              Y = f_mass' - f_mass
//   mass      X = f_mass' + f_mass + G' + G,   Y = f_mom' - f_mom
// (' across the face): the sums are exact in fixed point, the differences FP64.
template <int K, bool DIFF>
__device__ __forceinline__ void stage_fix_line(const OpConst<double, K>& C, const FixLine<K, 2>& L, int pm,
                                               FixSmem<K>& S, int a, int sb0, int sst, const double (&fmo)[2],
                                               const double (&fao)[2], const double (&qo)[2], int do_adv)
{
    const int sN = sb0 + (K - 1) * sst;
    double* fm = &S.fm[sb0];
    double* fa = &S.fa[a][sb0];
    double* q = &S.q[a][sb0];
    const double ya0 = fmo[0] - S.fm[sb0], yaN = fmo[1] - S.fm[sN];
    // before the mass results replace f_mass
    const double ym0 = fao[0] - S.fa[a][sb0], ymN = fao[1] - S.fa[a][sN];
    if (!fix_equation<K, DIFF>(L, 1, -pm, fa, q, sst, fao, qo, ya0, yaN, fa)) {
        double g[2];
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const double* c = C.cA[0][s];
            const int o = s ? sN : sb0;
            g[s] = (s ? yaN : ya0) * c[0] + fao[s] * c[2] + S.fa[a][o] * c[3];
            if (DIFF) g[s] += C.cQ[0][s] * (qo[s] + S.q[a][o]);
        }
        stage_line_fp64<K>(C, fa, DIFF ? q : nullptr, sst, g[0], g[1], fa);
    }
    if (do_adv && !fix_equation<K, false>(L, 0, pm, fm, nullptr, sst, fmo, fmo, ym0, ymN, q)) {
        double g[2];
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const double* c = C.cM[0][s];
            g[s] = fmo[s] * c[0] + S.fm[s ? sN : sb0] * c[1] + (s ? ymN : ym0) * c[2];
        }
        stage_line_fp64<K>(C, fm, nullptr, sst, g[0], g[1], q);
    }
}

// What bounds these kernels and what they measured (ms per launch at 32.8 M
// nodes, even-odd or per-node FP64 line sums -> fixed point):
//   K          2           3           4           5           6           7           8
//   stage      8.99->1.74  4.49->1.54  3.85->1.31  3.85->1.44  4.28->1.54  4.69->1.77  5.67->1.66
//   gradient   1.54->0.55  1.10->0.41  1.11->0.41  1.11->0.38  1.40->0.49  1.60->0.51  1.69->0.52
// At K = 5 a stage launch keeps the FP64 pipe 73 % busy, the integer pipe 54 %,
// the issue slots 61 % and HBM at 66 % of a copy: no unit is the bound by itself,
// the barriers between the node and line phases are (a quarter of the warps'
// time), so resident warps count most.  Registers per thread of the stage kernel
// and elements per CTA were chosen by that.  us per launch on 8 M nodes at 32 / 40 /
// 48 / 56 / 64 registers:
//   K = 2  686 / 527 / 448 / 432 / 459    K = 6  536 / 537 / 389 / 377 / 411
//   K = 3  572 / 384 / 387 / 417 / 417    K = 7  572 / 422 / 410 / 410 / 535
//   K = 4  414 / 373 / 329 / 334 / 334    K = 8  408 / 439 / 512 / 512 / 512
//   K = 5  497 / 366 / 355 / 390 / 389
// and, before an exponent per equation, K = 4 at 1 / 2 / 4 / 6 elements 383 / 296 /
// 311 / 349.  At the registers chosen the kernels that read fluxes spill 0 to 28
// bytes per thread up to K = 7 and 210 to 300 at K = 8, where more registers cost
// more in resident warps.  Converting results on the FP64 pipe (fix_to_fp64)
// instead saves integer work where that pipe is the scarcer one: 346 for 329 us.
__host__ __device__ constexpr int fix_regs(int K) { return K == 8 ? 32 : K == 6 || K == 2 ? 56 : 48; }
__host__ __device__ constexpr int fix_min_blocks(int K) { return 65536 / (fix_regs(K) * fix_threads(K)); }
// The stage input and the old state are fetched into shared memory at the
// start where they fit beside the line data.
__host__ __device__ constexpr bool fix_staged(int K) { return K < 8; }

// Flux modes and PACK as in stage_kernel.
template <int K, bool DIFF, int FLUX, bool PACK>
__global__ void __launch_bounds__(fix_threads(K), fix_min_blocks(K))
stage_fix_kernel(StageIO<double> io, MeshDev<double> m, const __grid_constant__ OpConst<double, K> C,
                 const __grid_constant__ FixOps<K, 2> F, int do_adv, int do_sponge)
{
    constexpr int K2 = K * K, K3 = K2 * K, EPB = fix_epb(K), T = fix_threads(K), RL = fix_rounds(K);
    constexpr bool STAGED = fix_staged(K);
    __shared__ FixSmem<K> sm[EPB];
    __shared__ double st[STAGED ? 8 : 1][STAGED ? T : 1];
    const int tid = threadIdx.x, e0 = blockIdx.x * EPB;
    const int el = tid / K3, n = tid - el * K3, sn = fix_slot<K>(n);
    const int e = e0 + el;
    const bool act = el < EPB && e < m.n_elem;
    const size_t off = (size_t)e * io.np + n;
    int code[RL][2];
    fix_codes<K>(m, e0, code);
    pdl_wait();
    pdl_next();

    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    if (act) {
        FixSmem<K>& S = sm[el];
        if (DIFF)
#pragma unroll
            for (int a = 0; a < 3; a++) copy_async8(&S.q[a][sn], io.q + (size_t)a * io.fs + off);
        if (FLUX == 2) {
            copy_async8(&S.fm[sn], io.flux_in + off);
#pragma unroll
            for (int a = 0; a < 3; a++) copy_async8(&S.fa[a][sn], io.flux_in + (size_t)(1 + a) * io.fs + off);
        }
        copy_async_commit();
        if (STAGED) {
            if (FLUX == 2)
#pragma unroll
                for (int f = 0; f < 4; f++) copy_async8(&st[f][tid], io.src + (size_t)f * io.fs + off);
            if (io.old)
#pragma unroll
                for (int f = 0; f < 4; f++) copy_async8(&st[4 + f][tid], io.old + (size_t)f * io.fs + off);
        }
        copy_async_commit();
        if (FLUX != 2) {
#pragma unroll
            for (int f = 0; f < 4; f++) s4[f] = io.src[(size_t)f * io.fs + off];
            S.fm[sn] = do_adv ? momentum_flux(s4[0], C.k1, C.k2) : 0.0;
#pragma unroll
            for (int a = 0; a < 3; a++)
                S.fa[a][sn] = do_adv ? mass_flux(s4[1 + a], s4[0], C.r0, C.linear_mass) : 0.0;
        }
    }

    // neighbour (or exterior) fluxes and gradients at the ends of this
    // thread's lines
    double fmo[RL][2], fao[RL][2], qo[RL][2];
#pragma unroll
    for (int r = 0; r < RL; r++) {
        const int task = tid + r * T;
        const FixTask<K> L(task);
        if (task >= EPB * 3 * K2 || e0 + L.le >= m.n_elem) continue;
        fix_end_values<true, DIFF, K, FLUX>(io, m, C, code[r], L, fmo[r], fao[r], qo[r]);
        if (FLUX != 2 && !do_adv) fmo[r][0] = fmo[r][1] = fao[r][0] = fao[r][1] = 0.0;
    }
    copy_async_wait<1>();
    __syncthreads();

#pragma unroll
    for (int r = 0; r < RL; r++) {
        const int task = tid + r * T;
        const FixTask<K> L(task);
        if (task >= EPB * 3 * K2 || e0 + L.le >= m.n_elem) continue;
        stage_fix_line<K, DIFF>(C, F.line, F.pm, sm[L.le], L.a, L.sb0, L.sst, fmo[r], fao[r], qo[r], do_adv);
    }
    copy_async_wait<0>();
    __syncthreads();
    if (!act) return;

    const FixSmem<K>& S = sm[el];
    double rr[4];
#pragma unroll
    for (int a = 0; a < 3; a++) rr[1 + a] = do_adv ? S.q[a][sn] : 0.0;
    if (F.cube) {
        rr[0] = S.fa[0][sn] + S.fa[1][sn];
        rr[0] += S.fa[2][sn];
    } else {
        rr[0] = S.fa[0][sn] + S.fa[1][sn] * F.ws[1];
        rr[0] += S.fa[2][sn] * F.ws[2];
        rr[2] *= F.ws[1];
        rr[3] *= F.ws[2];
    }
    // cb - ca sigma of this element: tabulated per stage by the host, computed
    // here when absent
    const double cbe = io.elem_b ? __ldg(io.elem_b + e) : io.cb - (do_sponge ? io.ca * __ldg(m.sigma + e) : 0.0);
    double vo[4];
#pragma unroll
    for (int f = 0; f < 4; f++) {
        const size_t o = (size_t)f * io.fs + off;
        if (FLUX == 2) s4[f] = STAGED ? st[f][tid] : io.src[o];
        double v = rr[f] + s4[f] * cbe;
        if (io.old) v += (STAGED ? st[4 + f][tid] : io.old[o]) * io.cc;
        io.dst[o] = v;
        vo[f] = v;
    }
    if (FLUX >= 1) {
        // the next stage's fluxes, evaluated as that stage would from dst
        io.flux_out[off] = momentum_flux(vo[0], C.k1, C.k2);
#pragma unroll
        for (int a = 0; a < 3; a++)
            io.flux_out[(size_t)(1 + a) * io.fs + off] = mass_flux(vo[1 + a], vo[0], C.r0, C.linear_mass);
    }
    if constexpr (PACK) {
        const size_t gi = grid_index(io.pack_map, e, n);
#pragma unroll
        for (int f = 0; f < 4; f++) io.pack[(size_t)f * io.pack_gsize + gi] = vo[f];
    }
}

// ------------------------------------------------------------ host
// w_0 / w_a of an operator; false when axis a's D and face coefficients are
// not axis 0's times that.
template <int K>
inline bool fix_axes(const OpConst<double, K>& C, bool stage, double ws[3], int& cube)
{
    cube = 1;
    ws[0] = 1.0;
    int big = 0;  // the largest entry of D's first row, for the ratio
    for (int j = 1; j < K; j++)
        if (std::fabs(C.rows[0][0][j]) > std::fabs(C.rows[0][0][big])) big = j;
    const double d0 = C.rows[0][0][big];
    for (int a = 1; a < 3; a++) {
        const double w = d0 != 0.0 ? C.rows[a][0][big] / d0 : 1.0;
        if (!(w > 0x1p-40 && w < 0x1p40)) return false;
        ws[a] = w;
        if (w != 1.0) cube = 0;
        auto same = [&](double x, double x0, double top) {
            return std::fabs(x - x0 * w) <= 1e-14 * std::fabs(top * w) || x == x0 * w;
        };
        for (int i = 0; i < K; i++) {
            for (int j = 0; j < K; j++)
                if (!same(C.rows[a][i][j], C.rows[0][i][j], d0)) return false;
            for (int j = K; j < K + 2; j++)  // the gradient's flux factors are in its lift columns
                if (!(stage ? C.rows[a][i][j] == C.rows[0][i][j] : same(C.rows[a][i][j], C.rows[0][i][j], C.rows[0][i][j])))
                    return false;
        }
        for (int s = 0; stage && s < 2; s++) {
            for (int i = 0; i < 4; i++)
                if (!same(C.cM[a][s][i], C.cM[0][s][i], C.cM[0][s][i]) || !same(C.cA[a][s][i], C.cA[0][s][i], C.cA[0][s][i]))
                    return false;
            if (!same(C.cQ[a][s], C.cQ[0][s], C.cQ[0][s])) return false;
        }
    }
    return true;
}

// Fixed-point operator of the stage operator C; false when its face
// coefficients are not those of a uniform medium, its rows not mirror
// symmetric, or its scales out of range.
template <int K>
inline bool make_stage_fix(const OpConst<double, K>& C, FixOps<K, 2>& F)
{
    std::memset(&F, 0, sizeof F);
    if (!fix_axes<K>(C, true, F.ws, F.cube)) return false;
    const double x = C.cM[0][0][0], y = C.cM[0][0][2], g = C.cA[0][0][0], h = C.cA[0][0][2];
    const double m[2][4] = {{x, x, y, -y}, {-x, -x, y, -y}}, r[2][4] = {{g, -g, h, h}, {g, -g, -h, -h}};
    const double tm = 1e-14 * std::fmax(std::fabs(x), std::fabs(y)), tr = 1e-14 * std::fmax(std::fabs(g), std::fabs(h));
    for (int s = 0; s < 2; s++) {
        for (int i = 0; i < 4; i++)
            if (!(std::fabs(C.cM[0][s][i] - m[s][i]) <= tm) || !(std::fabs(C.cA[0][s][i] - r[s][i]) <= tr)) return false;
        if (!(std::fabs(C.cQ[0][s] - (s ? -h : h)) <= 1e-14 * std::fabs(h))) return false;
    }
    // jumps of the momentum flux enter the mass equation times 2^pm ~ rho0 / c (of
    // the mass flux the momentum equation times 2^-pm), so that their coefficients
    // are of the size of the others
    const double k = h != 0.0 ? g / h : 1.0;
    if (!(k > 0x1p-40 && k < 0x1p40)) return false;
    F.pm = (int)std::lround(std::log2(k));
    const FixFlux f[2] = {{x, y, F.pm}, {h, g, -F.pm}};
    return fix_axis<K, 2>(C.rows[0], 1, f, F.line);
}

// The same of the gradient operator (its flux factors are in the lift
// columns, so the right end's lift has the opposite sign).
template <int K>
inline bool make_grad_fix(const OpConst<double, K>& C, FixOps<K, 1>& F)
{
    std::memset(&F, 0, sizeof F);
    const FixFlux f[1] = {{1.0, 0.0, 0}};
    return fix_axes<K>(C, false, F.ws, F.cube) && fix_axis<K, 1>(C.rows[0], -1, f, F.line);
}

// The gradient kernel of operator F.
template <int K>
inline auto fix_gradient(const FixOps<K, 1>& F)
{
    return fix_rest(K) || F.line.rest ? ldg_gradient_fix_kernel<K, true> : ldg_gradient_fix_kernel<K, fix_rest(K)>;
}

}  // namespace dg
