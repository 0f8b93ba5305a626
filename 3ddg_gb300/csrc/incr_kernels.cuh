// FP32 kernels of one RK stage (increment form): the LDG gradient and the
// stage update.  Bound by issue, the L1 data pipe and the latency of the global
// loads, not by arithmetic (64^3 elements at N = 4, stage kernel: issue
// slots 68 % busy, L1 wavefronts 58 %, HBM 55 %).
//
// Mapping: a CTA takes incr_epb(K) whole elements.  Thread t has node t of
// their nodes, packed densely; the lines of one axis, packed over the elements,
// belong to whole warps, a lane per line, so that the line code is
// instantiated per axis and its operator rows and face coefficients are
// immediate constant-bank operands.  A line's two ends are exactly the two face
// nodes whose numerical fluxes it needs, so its owner loads their neighbour
// values, evaluates both face terms and all K outputs; per node and axis that
// is (K + 2) / K shared-memory operands instead of the 2 (K + 2) of a thread
// per node summing its own lines.  Small elements share a CTA: a warp slice per
// element left 24 of 32 lanes idle at K = 2 and 5 at K = 3.
//
// us per launch on ~8 M nodes (stage / gradient), per-node sums in a warp
// slice per element (K <= 4) or line owners over unpadded z-lines (K > 4) ->
// this form:
//   K = 2  497 / 191 -> 184 / 81    K = 5 (32.8 M nodes)  532 / 230 -> 542 / 217
//   K = 3  236 / 100 -> 165 / 69    K = 7                 161 / 69  -> 161 / 62
//   K = 4  177 /  81 -> 134 / 59    K = 8                 192 / 70  -> 172 / 59
// and with 32-bit field offsets (incr_at), ~32.8 M nodes, K = 2 .. 8:
//   714 / 305, 646 / 259, 511 / 220, 506 / 213, 625 / 227, 631 / 253, 690 / 220
#pragma once

#include "dg_kernels.cuh"

namespace dg {

__host__ __device__ constexpr int incr_epb(int K) { return K == 2 ? 16 : K == 3 ? 7 : K == 4 ? 4 : 1; }
// warps per axis
__host__ __device__ constexpr int incr_wpa(int K) { return (incr_epb(K) * K * K + 31) / 32; }
__host__ __device__ constexpr int incr_threads(int K)
{
    const int nodes = (incr_epb(K) * K * K * K + 31) / 32 * 32, lines = 3 * 32 * incr_wpa(K);
    return nodes > lines ? nodes : lines;
}

// Line t of axis A (t = the two other coordinates, z varying fastest where it
// is one of them): its first node and stride, the position of its ends among
// the K^2 nodes of their faces (the order of the boundary tables), and its
// place in shared memory, where z-lines are padded to an odd length (K = 6 loses
// more by the index arithmetic than by its two-way bank conflicts).
template <int K>
struct IncrLine {
    static constexpr int P = K == 6 ? 6 : K | 1, LAST = incr_threads(K) - 1;
    // one element per CTA: every thread has a slot, so that no store is predicated
    static constexpr int SLOTS = incr_epb(K) > 1 ? K * K * P : P == K ? LAST + 1 : LAST + LAST / K + 1;
    __device__ __forceinline__ static int node(int a, int t) { return a == 0 ? t : (a == 1 ? t / K * K * K + t % K : t * K); }
    __device__ __forceinline__ static int face(int a, int t) { return a == 1 ? t % K * K + t / K : t; }
    __device__ __forceinline__ static int slot(int n) { return P == K ? n : n + n / K; }
    template <int A>
    __device__ __forceinline__ static int first_slot(int t)
    {
        return A == 0 ? t / K * P + t % K : (A == 1 ? t / K * K * P + t % K : t * P);
    }
    template <int A>
    __device__ __forceinline__ static constexpr int slot_stride()
    {
        return A == 0 ? K * P : (A == 1 ? P : 1);
    }
};

// This thread's node and line.
template <int K>
struct IncrTask {
    static constexpr int K2 = K * K, K3 = K2 * K, EPB = incr_epb(K), WPA = incr_wpa(K);
    int el, n, e;      // element slot, node, element
    int le, la, lt;    // line: element slot, axis, number
    bool act, owner;
    __device__ __forceinline__ explicit IncrTask(int n_elem)
    {
        const int tid = threadIdx.x, e0 = blockIdx.x * EPB, w = tid / 32;
        el = EPB == 1 ? 0 : tid / K3;
        n = tid - el * K3;
        e = e0 + el;
        act = n < K3 && el < EPB && e < n_elem;
        la = w / WPA;
        const int l = (w % WPA) * 32 + tid % 32;
        le = EPB == 1 ? 0 : l / K2;
        lt = l - le * K2;
        owner = la < 3 && le < EPB && lt < K2 && e0 + le < n_elem;
    }
};

// Value ``off`` of field f of a buffer.  The field's address is the same for all
// threads; with Off = unsigned, for fields below 4 GiB, a thread's 32-bit byte
// offset is added to it by the load itself: a tenth fewer instructions and no
// spills at K = 5 (541 -> 509 us per stage launch at 64^3 elements; K = 7 161 ->
// 143).  Larger fields take Off = size_t.
template <typename Off, typename T>
__device__ __forceinline__ T* incr_at(T* base, size_t fs, int f, Off off)
{
    return (T*)((char*)(base + (size_t)f * fs) + off * (Off)sizeof(T));
}
// Whether the fields of a problem are below 4 GiB.
inline bool incr_narrow(size_t fs) { return fs * sizeof(float) < ((size_t)1 << 32); }

template <bool PDL, typename Off>
__device__ __forceinline__ float incr_in(const StageIO<float>& io, int f, Off off)
{
    float v = pdl_load<PDL>(incr_at(io.src, io.fs, f, off));
    if (io.inc) v += pdl_load<PDL>(incr_at(io.inc, io.fs, f, off));
    return v;
}

// Neighbour (or exterior) values at the two ends of a line: drho always, the
// normal velocity with WITH_U, the gradient with WITH_Q.
template <bool WITH_U, bool WITH_Q, bool PDL, typename Off, int K>
__device__ __forceinline__ void incr_end_values(const StageIO<float>& io, const MeshDev<float>& m,
                                                const OpConst<float, K>& C, const int code[2], int a, int t,
                                                float ro[2], float uo[2], float qo[2])
{
    const int st = axis_stride<K>(a), b0 = IncrLine<K>::node(a, t);
#pragma unroll
    for (int side = 0; side < 2; side++) {
        ro[side] = uo[side] = qo[side] = 0.f;
        if (code[side] >= 0) {
            const Off o2 = (Off)code[side] * io.np + b0 + (side ? 0 : (K - 1) * st);
            ro[side] = incr_in<PDL>(io, 0, o2);
            if (WITH_U) uo[side] = incr_in<PDL>(io, 1 + a, o2);
            if (WITH_Q) qo[side] = pdl_load<PDL>(incr_at(io.q, io.fs, a, o2));
        } else {
            float u2;
            exterior<float, K>(m, C, -1 - code[side], side, IncrLine<K>::face(a, t), ro[side], u2);
            if (WITH_U) uo[side] = u2;
        }
    }
}

template <typename M>
__device__ __forceinline__ void incr_end_codes(const M& m, int e, int a, int code[2])
{
#pragma unroll
    for (int side = 0; side < 2; side++) code[side] = __ldg(m.nbr + (size_t)e * 6 + 2 * a + side);
}

// ------------------------------------------------------------ LDG gradient
// One line: the central flux of drho at both ends (its factors are in the lift
// columns); the owner stores its line's K values of G_A itself.
template <int A, int K>
__device__ __forceinline__ void incr_grad_line(const OpConst<float, K>& C, const float* r, int t, const float ro[2],
                                               float* __restrict__ q_elem)
{
    constexpr int st = axis_stride<K>(A), sst = IncrLine<K>::template slot_stride<A>();
    const int b0 = IncrLine<K>::node(A, t), s0 = IncrLine<K>::template first_slot<A>(t);
    float v[K];
#pragma unroll
    for (int j = 0; j < K; j++) v[j] = r[s0 + j * sst];
    const float f0 = ro[0] + v[0], fN = ro[1] + v[K - 1];
#pragma unroll
    for (int i = 0; i < K; i++) {
        const float* row = C.rows[A][i];
        float s2 = row[K] * f0;
        s2 += row[K + 1] * fN;
#pragma unroll
        for (int j = 0; j < K; j++) s2 += row[j] * v[j];
        q_elem[b0 + i * st] = s2;
    }
}

// Resident CTAs per SM asked of the compiler for the gradient kernel: it waits
// on memory latency and fits 40 registers (32 up to K = 4).
__host__ __device__ constexpr int incr_grad_blocks(int K)
{
    return 65536 / ((K <= 4 ? 32 : 40) * incr_threads(K));
}

template <int K, bool PDL, typename Off>
__global__ void __launch_bounds__(incr_threads(K), incr_grad_blocks(K))
incr_gradient_kernel(StageIO<float> io, MeshDev<float> m, const OpConst<float, K> C)
{
    __shared__ float r[incr_epb(K)][IncrLine<K>::SLOTS];
    const IncrTask<K> T(m.n_elem);
    const int el = blockIdx.x * incr_epb(K) + T.le;
    int code[2] = {0, 0};
    if (T.owner) incr_end_codes(m, el, T.la, code);
    if constexpr (PDL) {
        pdl_wait();
        pdl_next();
    }
    float ro[2] = {0.f, 0.f}, unused_u[2], unused_q[2];
    float rho = 0.f;
    if (T.act) rho = incr_in<PDL>(io, 0, (Off)T.e * io.np + T.n);
    if (T.owner) incr_end_values<false, false, PDL, Off, K>(io, m, C, code, T.la, T.lt, ro, unused_u, unused_q);
    if (incr_epb(K) == 1 || T.act) r[T.el][IncrLine<K>::slot(T.n)] = rho;
    __syncthreads();
    if (T.owner) {
        float* q = io.q_out + (size_t)T.la * io.fs + (size_t)el * io.np;
        if (T.la == 0) incr_grad_line<0, K>(C, r[T.le], T.lt, ro, q);
        else if (T.la == 1) incr_grad_line<1, K>(C, r[T.le], T.lt, ro, q);
        else incr_grad_line<2, K>(C, r[T.le], T.lt, ro, q);
    }
}

// ------------------------------------------------------------ stage
// Per element, for each axis: the pair (f_mom, f_mass + G) of every node (one
// 8-byte load feeds two FMAs of a line sum), and its own mass flux and
// gradient, which the line owners replace by their (density, momentum) results.
template <int K>
struct IncrSmem {
    float2 f[3][IncrLine<K>::SLOTS];
    float m[3][IncrLine<K>::SLOTS];
    float q[3][IncrLine<K>::SLOTS];
};

// One line: the face terms at its two ends from the prefetched neighbour
// values, then the sums.
template <int A, bool DIFF, int K>
__device__ __forceinline__ void incr_stage_line(const OpConst<float, K>& C, IncrSmem<K>& S, int t, const float ro[2],
                                                const float uo[2], const float qo[2], int do_adv)
{
    constexpr int st = IncrLine<K>::template slot_stride<A>();
    const int b0 = IncrLine<K>::template first_slot<A>(t);
    float2 g[2];
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const int nf = b0 + (side ? (K - 1) * st : 0);
        const float fm_s = S.f[A][nf].x, fa_s = S.m[A][nf];
        float gm = 0.f, gr = 0.f;
        if (do_adv) {
            const float fmo = momentum_flux(ro[side], C.k1, C.k2);
            const float fao = mass_flux(uo[side], ro[side], C.r0, C.linear_mass);
            const float* cm = C.cM[A][side];
            const float* cr = C.cA[A][side];
            gm = fmo * cm[0] + fm_s * cm[1] + fao * cm[2] + fa_s * cm[3];
            gr = fmo * cr[0] + fm_s * cr[1] + fao * cr[2] + fa_s * cr[3];
        }
        if (DIFF) gr += C.cQ[A][side] * (qo[side] + S.q[A][nf]);
        g[side].x = gm;
        g[side].y = gr;
    }
    float2 v[K];
#pragma unroll
    for (int j = 0; j < K; j++) v[j] = S.f[A][b0 + j * st];
#pragma unroll
    for (int i = 0; i < K; i++) {
        const float* row = C.rows[A][i];
        float sm = row[K] * g[0].x, sr = row[K] * g[0].y;
        sm += row[K + 1] * g[1].x;
        sr += row[K + 1] * g[1].y;
#pragma unroll
        for (int j = 0; j < K; j++) {
            sm += row[j] * v[j].x;
            sr += row[j] * v[j].y;
        }
        S.m[A][b0 + i * st] = sr;
        S.q[A][b0 + i * st] = sm;
    }
}

// Resident CTAs per SM asked of the compiler: 40 registers up to K = 5.
__host__ __device__ constexpr int incr_min_blocks(int K) { return K <= 5 ? 65536 / (40 * incr_threads(K)) : 0; }

// A node's own values.
template <bool DIFF, bool PDL, typename Off>
__device__ __forceinline__ void incr_own_values(const StageIO<float>& io, Off off, float ub[4], float dv[4],
                                                float cmp[4], float q[3])
{
#pragma unroll
    for (int f = 0; f < 4; f++) {
        ub[f] = pdl_load<PDL>(incr_at(io.src, io.fs, f, off));
        if (io.inc) dv[f] = pdl_load<PDL>(incr_at(io.inc, io.fs, f, off));
        if (io.final_stage) cmp[f] = *incr_at(io.comp, io.fs, f, off);
    }
    if (DIFF)
#pragma unroll
        for (int a = 0; a < 3; a++) q[a] = pdl_load<PDL>(incr_at(io.q, io.fs, a, off));
}

// Its volume fluxes (and gradient) into shared memory.
template <bool DIFF, int K>
__device__ __forceinline__ void incr_node_fluxes(const OpConst<float, K>& C, IncrSmem<K>& S, int sn, const float ub[4],
                                                 const float dv[4], const float q[3], int do_adv)
{
    const float rho = ub[0] + dv[0];
    const float u[3] = {ub[1] + dv[1], ub[2] + dv[2], ub[3] + dv[3]};
    float fmom = 0.f, fmass[3] = {0.f, 0.f, 0.f};
    if (do_adv) {
        fmom = momentum_flux(rho, C.k1, C.k2);
#pragma unroll
        for (int a = 0; a < 3; a++) fmass[a] = mass_flux(u[a], rho, C.r0, C.linear_mass);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        S.f[a][sn].x = fmom;
        S.f[a][sn].y = DIFF ? fmass[a] + q[a] : fmass[a];
        S.m[a][sn] = fmass[a];
        if (DIFF) S.q[a][sn] = q[a];
    }
}

// Its stage combination, from the three lines through it.
template <int K, typename Off>
__device__ __forceinline__ void incr_update(const StageIO<float>& io, const IncrSmem<K>& S, int sn, Off off,
                                            float sig, const float ub[4], const float dv[4], const float cmp[4],
                                            int do_adv)
{
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        r[0] += S.m[a][sn];
        r[1 + a] = do_adv ? S.q[a][sn] : 0.f;
    }
    const float ks = io.ca * sig;
    const float cbe = io.cb - ks, ce = io.eps - ks;
#pragma unroll
    for (int f = 0; f < 4; f++) {
        float d = r[f] + ub[f] * ce;
        if (io.inc) d += dv[f] * cbe;
        if (io.final_stage) {
            // Kahan-compensated u <- u + d
            const float y = d - cmp[f];
            const float t = ub[f] + y;
            *incr_at(io.comp, io.fs, f, off) = (t - ub[f]) - y;
            *incr_at(io.dst, io.fs, f, off) = t;
        } else {
            *incr_at(io.dst, io.fs, f, off) = d;
        }
    }
}

// Stage input s = u + d (u = ``src``, d = ``inc``, absent in stage 1):
//   d_out = R' + d (cb - ca sigma) + u (eps - ca sigma)   (= ca R + cb d + eps u)
// and in the final stage u <- u + d_out by a Kahan-compensated sum into
// ``dst`` (the other u buffer) and ``comp``.  Every global load a thread makes
// is issued before the first value is used.
//
// One element per CTA (K >= 5).  The packed form below at one element per CTA
// does the same but measured 3 to 5 % slower at K = 5 (558 to 570 us per launch
// at 64^3 elements), so this keeps a kernel of its own.
template <int K, bool DIFF, bool PDL, typename Off>
__global__ void __launch_bounds__(incr_threads(K), incr_min_blocks(K))
incr_stage_kernel(StageIO<float> io, MeshDev<float> m, const OpConst<float, K> C, int do_adv, int do_sponge)
{
    constexpr int K2 = K * K, K3 = K2 * K, WPA = incr_wpa(K);
    __shared__ IncrSmem<K> S;
    const int n = threadIdx.x, e = blockIdx.x;
    const bool act = n < K3;
    const Off off = (Off)e * io.np + n;
    const int sn = IncrLine<K>::slot(n);
    // line owner: warp group la, line lt of that axis
    const int la = n / 32 / WPA, lt = (n / 32 % WPA) * 32 + n % 32;
    const bool owner = la < 3 && lt < K2;
    int code[2] = {0, 0};
    if (owner) incr_end_codes(m, e, la, code);
    const float sig = (act && do_sponge) ? __ldg(m.sigma + e) : 0.f;
    if constexpr (PDL) {
        pdl_wait();
        pdl_next();
    }
    float ub[4] = {0.f, 0.f, 0.f, 0.f}, dv[4] = {0.f, 0.f, 0.f, 0.f};
    float cmp[4] = {0.f, 0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
    if (act) incr_own_values<DIFF, PDL>(io, off, ub, dv, cmp, q);
    float ro[2], uo[2], qo[2];
    if (owner) incr_end_values<true, DIFF, PDL, Off, K>(io, m, C, code, la, lt, ro, uo, qo);
    incr_node_fluxes<DIFF, K>(C, S, sn, ub, dv, q, do_adv);
    __syncthreads();
    if (owner) {
        if (la == 0) incr_stage_line<0, DIFF, K>(C, S, lt, ro, uo, qo, do_adv);
        else if (la == 1) incr_stage_line<1, DIFF, K>(C, S, lt, ro, uo, qo, do_adv);
        else incr_stage_line<2, DIFF, K>(C, S, lt, ro, uo, qo, do_adv);
    }
    __syncthreads();
    if (act) incr_update<K>(io, S, sn, off, sig, ub, dv, cmp, do_adv);
}

// Several elements per CTA (K <= 4).
template <int K, bool DIFF, bool PDL, typename Off>
__global__ void __launch_bounds__(incr_threads(K), incr_min_blocks(K))
incr_packed_stage_kernel(StageIO<float> io, MeshDev<float> m, const OpConst<float, K> C, int do_adv, int do_sponge)
{
    __shared__ IncrSmem<K> sm[incr_epb(K)];
    const IncrTask<K> T(m.n_elem);
    const Off off = (Off)T.e * io.np + T.n;
    const int sn = IncrLine<K>::slot(T.n);
    int code[2] = {0, 0};
    if (T.owner) incr_end_codes(m, blockIdx.x * incr_epb(K) + T.le, T.la, code);
    const float sig = (T.act && do_sponge) ? __ldg(m.sigma + T.e) : 0.f;
    if constexpr (PDL) {
        pdl_wait();
        pdl_next();
    }
    float ub[4] = {0.f, 0.f, 0.f, 0.f}, dv[4] = {0.f, 0.f, 0.f, 0.f};
    float cmp[4] = {0.f, 0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
    if (T.act) incr_own_values<DIFF, PDL>(io, off, ub, dv, cmp, q);
    float ro[2], uo[2], qo[2];
    if (T.owner) incr_end_values<true, DIFF, PDL, Off, K>(io, m, C, code, T.la, T.lt, ro, uo, qo);
    if (T.act) incr_node_fluxes<DIFF, K>(C, sm[T.el], sn, ub, dv, q, do_adv);
    __syncthreads();
    if (T.owner) {
        IncrSmem<K>& S = sm[T.le];
        if (T.la == 0) incr_stage_line<0, DIFF, K>(C, S, T.lt, ro, uo, qo, do_adv);
        else if (T.la == 1) incr_stage_line<1, DIFF, K>(C, S, T.lt, ro, uo, qo, do_adv);
        else incr_stage_line<2, DIFF, K>(C, S, T.lt, ro, uo, qo, do_adv);
    }
    __syncthreads();
    if (T.act) incr_update<K>(io, sm[T.el], sn, off, sig, ub, dv, cmp, do_adv);
}

}  // namespace dg
