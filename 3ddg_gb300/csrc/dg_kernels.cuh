// sm_103a kernels for one stage of the DG right-hand side and its RK update.
//
// Two launches per RK stage (one without diffusion):
//   ldg_gradient_fix_kernel (FP64, fix_kernels.cuh), incr_gradient_kernel
//   (FP32, incr_kernels.cuh)
//                        G_a = -D_c d(drho)/dx_a by LDG with the central flux
//                        (Element::OperateQFromDRho, cppsrc/Element.cpp:623-690;
//                        stored pre-multiplied by -D_c, the diffusive flux)
//   stage_fix_kernel (FP64), incr_stage_kernel (FP32 increment form)
//                        volume + face terms of the advection operator
//                        (Element::OperateUFromV, cppsrc/Element.cpp:475-620),
//                        LDG divergence (Element::OperateDRhoFromQ, :691-758),
//                        sponge (Element::OperateSponge, :760-781) and the RK
//                        stage combination (Element::selfWeightedAdd, :288-307)
//                        fused into one pass over the state.
// This file: what they share, and the FP64 kernels for operators without a
// fixed-point form (ldg_gradient_kernel, stage_kernel).
//
// Mapping: one thread per node, one warp-aligned slice of NPT threads per
// element, EPB elements per CTA.  Each thread loads its node (and the
// neighbour values its face work needs) before the first use; the element
// stages its volume fluxes in shared memory; face fluxes and line sums follow
// after barriers.  The reference's per-line QR solve of
// (M q w) x = S q f - F becomes
//     x = (1/w) D f - (1/(q w)) (M^-1 e_0 F_0 + M^-1 e_N F_N),  D = M^-1 S,
// with D and the lift columns computed once on the host in FP64.
//
// FP64: every constant factor is folded on the host into the per-launch
// operator (OpConst): the RK stage weight ca, 1/w_a and the equations' lift
// scales go into per-axis copies of D and into the face-flux coefficients, the
// gradient carries -D_c so that the LDG divergence and the mass-flux
// divergence share one line sum, and the sponge folds into the RK combination
// (its per-element weight tabulated by the host).  The kernels of
// fix_kernels.cuh evaluate the folded line operators in block fixed point;
// ldg_gradient_kernel and stage_kernel below sum every node's three lines in
// FP64, for operators that have no such form (matrix files whose D is not
// centro-antisymmetric).  Each stage writes the volume fluxes of its output
// for the next stage to read (flux modes), so no face neighbour's flux is
// evaluated twice.
//
// Neighbour face values are read straight from the neighbour element (same
// block or another block of the same HBM pool) through the face table, which
// replaces the halo ring and Grid::communicate.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

#include "pdl.cuh"

namespace dg {

__host__ __device__ constexpr int npt_of(int K) { return (K * K * K + 31) / 32 * 32; }
__host__ __device__ constexpr int epb_of(int K) { return K <= 3 ? 4 : (K == 4 ? 2 : 1); }

// A 16-byte vector of T (the widest per-thread global load).
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
};
template <>
struct Vec16<double> {
    using type = double2;
};

// Length of one operator row: K entries of D, the two lift entries, padded to
// whole 16-byte vectors.
template <typename T, int K>
__host__ __device__ constexpr int oprow_len()
{
    return (K + 2 + (int)(16 / sizeof(T)) - 1) / (int)(16 / sizeof(T)) * (int)(16 / sizeof(T));
}

// Per-launch operator constants, in device memory.
//   stage kernel:    D[a] = ca D / w_a;   cM, cA: face coefficients of the
//                    momentum / mass equations times ca * (lift scale);
//                    cQ[a] = (+0.5, -0.5) ca / w_a (central flux of G).
//   gradient kernel: D[a] = D_c D / w_a;  lift columns times the central-flux
//                    factors (+0.5, -0.5) D_c / w_a (cQ unused).
// rows[a][i] = (D[a][i][0..K-1], L0[i], LN[i], 0...) with the lift columns
// L0 = M^-1 e_0, LN = M^-1 e_N, so that a thread loads its row of each axis
// with one or two 16-byte loads.
// Face coefficients act on (f_mom other, f_mom self, f_mass other, f_mass self).
template <typename T, int K>
struct OpConst {
    alignas(16) T rows[3][K][oprow_len<T, K>()];
    T cM[3][2][4];
    T cA[3][2][4];
    T cQ[3][2];
    T k1, k2;              // f_mom(rho) = rho (k1 + k2 rho) = c^2/rho0 (rho + B/A rho^2 / (2 rho0))
    T r0;                  // f_mass(u, rho) = u (rho + rho0), or u rho0 when B/A = 0
    T inv_c2, inv_z;       // source exterior state: drho = p / c^2, u = p / (rho0 c)
    int linear_mass;
};

// Mesh arrays on the device (see mesh.h).
template <typename T>
struct MeshDev {
    const int* nbr;        // n_elem * 6, faces -X +X -Y +Y -Z +Z
    const T* sigma;        // n_elem
    const T* bnd_ic;       // n_bnd * 2 * K^2
    const T* bnd_ap;       // n_bnd * K^2
    const int* bnd_src;    // n_bnd: 1 on the source face
    int n_elem;
    int ic_live;           // exterior = IC halo values (first stage after creation)
    T src_p;               // source pressure at this stage's time
};

// Element-major state  <->  node-duplicated [X][Y][Z] grid layout (the
// reference's HDF5 dataset order, cppsrc/HDF5Functions.cpp:173-208).
struct GridMap {
    int K, nb[3], ne[3], E[3], elem_per_block;
};

__device__ __forceinline__ size_t grid_index(const GridMap& g, int e, int n)
{
    const int blk = e / g.elem_per_block, le = e % g.elem_per_block;
    const int b0 = blk / (g.nb[1] * g.nb[2]), b1 = (blk / g.nb[2]) % g.nb[1], b2 = blk % g.nb[2];
    const int l0 = le / (g.ne[1] * g.ne[2]), l1 = (le / g.ne[2]) % g.ne[1], l2 = le % g.ne[2];
    const int K = g.K;
    const size_t ii = (size_t)(b0 * g.ne[0] + l0) * K + n / (K * K);
    const size_t jj = (size_t)(b1 * g.ne[1] + l1) * K + (n / K) % K;
    const size_t kk = (size_t)(b2 * g.ne[2] + l2) * K + n % K;
    return (ii * ((size_t)g.E[1] * K) + jj) * ((size_t)g.E[2] * K) + kk;
}

// Stage input/output.  R' = ca R_ops is what the folded operator produces
// (R_ops: advection + diffusion, without the sponge).
//   PLAIN (FP64 method), stage input s = ``src``:
//       dst = R' + s (cb - ca sigma) + cc old         (= ca R + cb s + cc old)
//   INCR (FP32 form), stage input s = u + d (u = ``src``, d = ``inc``, absent
//   in stage 1):
//       d_out = R' + d (cb - ca sigma) + u (eps - ca sigma)
//                                                     (= ca R + cb d + eps u)
//       and in the final stage u <- u + d_out with a Kahan-compensated sum
//       into ``dst`` (the other u buffer) and ``comp``.
template <typename T>
struct StageIO {
    const T* src;
    const T* inc;
    const T* old;
    T* dst;
    T* comp;
    const T* q;            // LDG gradient (times -D_c), 3 fields
    T* q_out;              // gradient kernel output
    const T* elem_b;       // PLAIN: cb - ca sigma per element for this stage (null: from sigma)
    const T* flux_in;      // PLAIN, flux mode 2: volume fluxes of src (f_mom, f_mass x, y, z)
    T* flux_out;           // PLAIN, flux modes 1, 2: the same of dst
    size_t fs;             // field stride (n_elem * NP)
    int np;                // nodes per element in memory
    T ca, cb, cc, eps;
    int final_stage;
    // PLAIN, PACK: the output also written in host order ([X][Y][Z] per
    // field, fields gsize apart) for a download
    double* pack;
    GridMap pack_map;
    size_t pack_gsize;
};

template <typename T>
__device__ __forceinline__ T momentum_flux(T d, const T k1, const T k2)
{
    return d * (k1 + k2 * d);
}

template <typename T>
__device__ __forceinline__ T mass_flux(T u, T d, const T r0, int linear)
{
    // cppsrc/kernelFuncs.cpp:23-29
    return linear ? u * r0 : u * (d + r0);
}

template <typename T>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};

// Volume-flux output of the FP64 unpack kernels (f null: none): the fluxes
// of the state they write, so that the first stage after an upload reads
// them like any later stage.
template <typename T>
struct FluxOut {
    T* f;
    T k1, k2, r0;
    int linear;
};

// The flux constants of the stage operators and of FluxOut, from one place
// so that both evaluate bit-identical fluxes.
template <typename T>
inline FluxOut<T> flux_consts(T* f, double rho0, double c0, double b_over_a)
{
    FluxOut<T> o;
    o.f = f;
    o.k1 = (T)(c0 * c0 / rho0);
    o.k2 = (T)(b_over_a * 0.5 * c0 * c0 / (rho0 * rho0));
    o.r0 = (T)rho0;
    o.linear = b_over_a == 0.0 ? 1 : 0;
    return o;
}

template <typename T>
__device__ __forceinline__ void write_fluxes(const FluxOut<T>& fo, size_t fs, size_t o, T d, const T u[3])
{
    fo.f[o] = momentum_flux(d, fo.k1, fo.k2);
#pragma unroll
    for (int a = 0; a < 3; a++) fo.f[(size_t)(1 + a) * fs + o] = mass_flux(u[a], d, fo.r0, fo.linear);
}

template <typename T, int K>
struct GradSmem {
    T r[npt_of(K)];
    T fl[3][2][K * K];
};

template <typename T>
__device__ __forceinline__ T load_in(const StageIO<T>& io, int f, size_t off)
{
    return __ldg(io.src + (size_t)f * io.fs + off);
}

// Exterior value at a domain-boundary face node: the tone burst on the source
// face, else the IC halo values during the first stage, else zero.
template <typename T, int K>
__device__ __forceinline__ void exterior(const MeshDev<T>& m, const OpConst<T, K>& C, int slot,
                                         int side, int fi, T& ro, T& uo)
{
    if (m.bnd_src[slot]) {
        T p = m.src_p * m.bnd_ap[(size_t)slot * K * K + fi];
        ro = p * C.inv_c2;
        uo = (side == 0 ? p : -p) * C.inv_z;
    } else if (m.ic_live) {
        ro = m.bnd_ic[((size_t)slot * 2 + 0) * K * K + fi];
        uo = m.bnd_ic[((size_t)slot * 2 + 1) * K * K + fi];
    } else {
        ro = T(0);
        uo = T(0);
    }
}

template <int K>
__host__ __device__ constexpr int axis_stride(int a)
{
    return a == 0 ? K * K : (a == 1 ? K : 1);
}

// Face nodes of an element, numbered t = (2 a + side) K^2 + fi for the faces
// -X +X -Y +Y -Z +Z, fi = c[(a+1)%3] K + c[(a+2)%3]: the element's node on
// the face (nf) and the neighbour's node across it (nn, in the neighbour).
// The decoding is tabulated per order at compile time (one packed word per
// face node: a 2 bits, side 1, fi 7, nf 10, nn 10), so that a thread loads its
// face nodes' entries (coalesced) instead of redoing the integer arithmetic.
template <int K>
struct FaceTable {
    int v[6 * K * K];
    constexpr FaceTable() : v{}
    {
        constexpr int K2 = K * K;
        for (int t = 0; t < 6 * K2; t++) {
            const int a = t / (2 * K2), side = (t / K2) & 1, fi = t % K2, p = side ? K - 1 : 0;
            const int nf = a == 0 ? p * K2 + fi : (a == 1 ? (fi % K) * K2 + p * K + fi / K : fi * K + p);
            const int nn = nf + (side ? -(K - 1) : (K - 1)) * (a == 0 ? K2 : (a == 1 ? K : 1));
            v[t] = a | (side << 2) | (fi << 3) | (nf << 10) | (nn << 20);
        }
    }
};
template <int K>
__device__ const FaceTable<K> kFaceTable{};

// The same decoding by integer arithmetic (no memory access).
template <int K>
struct FaceNodeArith {
    int a, side, fi, nf, nn;
    __device__ __forceinline__ explicit FaceNodeArith(int t)
    {
        constexpr int K2 = K * K;
        a = t / (2 * K2);
        side = (t / K2) & 1;
        fi = t % K2;
        const int p = side ? K - 1 : 0;
        nf = a == 0 ? p * K2 + fi : (a == 1 ? (fi % K) * K2 + p * K + fi / K : fi * K + p);
        nn = nf + (side ? -(K - 1) : (K - 1)) * axis_stride<K>(a);
    }
};

template <int K>
struct FaceNode {
    int a, side, fi, nf, nn;
    __device__ __forceinline__ explicit FaceNode(int t)
    {
        const int w = __ldg(&kFaceTable<K>.v[t]);
        a = w & 3;
        side = (w >> 2) & 1;
        fi = (w >> 3) & 127;
        nf = (w >> 10) & 1023;
        nn = (w >> 20) & 1023;
    }
};

// ---------------------------------------------------------------------------
// LDG gradient, stored as G_a = -D_c Q_a = (D_c / w_a)(D drho + M^-1 e_0 F_0 +
// M^-1 e_N F_N) with the central flux F_0 = (drho_o[N] + drho_s[0]) / 2,
// F_N = -(drho_s[N] + drho_o[0]) / 2.
// ---------------------------------------------------------------------------
// Each thread's rows of the per-launch operator (its index along each axis),
// loaded once through L1 into registers.  The operator lives in global memory:
// indexing kernel-parameter space with a per-thread index would serialise on
// the address-divergence unit.
template <typename T, int K>
struct OpRows {
    T d[3][K], l0[3], ln[3];
    __device__ __forceinline__ void load(const OpConst<T, K>& C, const int c[3], bool act)
    {
        using V = typename Vec16<T>::type;
        constexpr int RL = oprow_len<T, K>(), NV = RL * (int)sizeof(T) / 16;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int ia = act ? c[a] : 0;
            T row[RL];
            const V* src = reinterpret_cast<const V*>(C.rows[a][ia]);
#pragma unroll
            for (int v = 0; v < NV; v++) reinterpret_cast<V*>(row)[v] = __ldg(src + v);
#pragma unroll
            for (int j = 0; j < K; j++) d[a][j] = row[j];
            l0[a] = row[K];
            ln[a] = row[K + 1];
        }
    }
};

template <typename T, int K>
__global__ void __launch_bounds__(npt_of(K) * epb_of(K))
ldg_gradient_kernel(StageIO<T> io, MeshDev<T> m, const OpConst<T, K>* __restrict__ Cp)
{
    constexpr int K2 = K * K, K3 = K * K * K, NPT = npt_of(K), NF = 6 * K2, R = (NF + NPT - 1) / NPT;
    __shared__ GradSmem<T, K> sm_all[epb_of(K)];
    GradSmem<T, K>& S = sm_all[threadIdx.y];
    const OpConst<T, K>& C = *Cp;
    const int n = threadIdx.x;
    const int e = blockIdx.x * epb_of(K) + threadIdx.y;
    const bool live = e < m.n_elem;
    const bool act = n < K3 && live;
    const int c[3] = {n / K2, (n / K) % K, n % K};
    // Face nodes assigned densely (see stage_kernel): their neighbour (or
    // exterior) values are loaded with the thread's own node.
    int code[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int t = n + r * NPT;
        code[r] = 0;
        if (live && t < NF) {
            const FaceNode<K> F(t);
            code[r] = __ldg(m.nbr + (size_t)e * 6 + 2 * F.a + F.side);
        }
    }
    T rho = T(0);
    if (act) rho = load_in(io, 0, (size_t)e * io.np + n);
    T ro[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        ro[r] = T(0);
        const int t = n + r * NPT;
        if (!live || t >= NF) continue;
        const FaceNode<K> F(t);
        if (code[r] >= 0) {
            ro[r] = load_in(io, 0, (size_t)code[r] * io.np + F.nn);
        } else {
            T uo;
            exterior<T, K>(m, C, -1 - code[r], F.side, F.fi, ro[r], uo);
        }
    }
    OpRows<T, K> R_;
    R_.load(C, c, act);
    S.r[n] = rho;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int t = n + r * NPT;
        if (!live || t >= NF) continue;
        const FaceNode<K> F(t);
        S.fl[F.a][F.side][F.fi] = ro[r] + S.r[F.nf];  // flux factors are in the lift columns
    }
    __syncthreads();
    if (!act) return;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int st = axis_stride<K>(a);
        const int base = n - c[a] * st;
        const int fi = c[(a + 1) % 3] * K + c[(a + 2) % 3];
        T s = R_.l0[a] * S.fl[a][0][fi];
        s += R_.ln[a] * S.fl[a][1][fi];
#pragma unroll
        for (int j = 0; j < K; j++) s += R_.d[a][j] * S.r[base + j * st];
        io.q_out[(size_t)a * io.fs + (size_t)e * io.np + n] = s;
    }
}

// Shared memory of a stage kernel, per element: for each axis a, the pair
// (f_mom, f_mass along a + G_a) of every node (one 8- or 16-byte load feeds
// two FMAs of a line sum), the pair (momentum, density) of every face term
// [axis][side][face node], and each node's own mass flux and gradient, which
// the face phase reads (and the batch's line owners reuse for their results).
template <typename T, int K>
struct PlainSmem {
    typename Pair<T>::type f[3][npt_of(K)];
    typename Pair<T>::type g[3][2][K * K];
    T m[3][npt_of(K)];
    T q[3][npt_of(K)];
};

// ---------------------------------------------------------------------------
// One RK stage of the plain (FP64) form: R = L(stage input), then the stage
// combination dst = R' + s (cb - ca sigma) + cc old.
//
// Per-node FP64 sums, for operators without a fixed-point form (see
// fix_kernels.cuh).  The face fluxes are assigned densely: thread n of an
// element evaluates face nodes n, n + NPT, ... of its 6 K^2, reading the
// element's own values from shared memory (a thread per node evaluating its
// own faces would issue every axis's face arithmetic in nearly every warp).
// The neighbour values of those face nodes are loaded with the thread's own
// node.
// ---------------------------------------------------------------------------
// Face term (x momentum, y density) of face node nf of an element on axis a,
// side ``side``: the numerical flux (impedance upwind for advection, central
// for LDG) times its lift scale, from the element's own values in shared
// memory and the neighbour (or exterior) values ro, uo (drho and the normal
// velocity, or in flux mode 2 their momentum and mass fluxes) and qo.
template <typename T, int K, bool DIFF, int FLUX>
__device__ __forceinline__ typename Pair<T>::type face_term(const OpConst<T, K>& C, const PlainSmem<T, K>& S,
                                                            int a, int side, int nf, T ro, T uo, T qo, int do_adv)
{
    const T fm_s = S.f[a][nf].x, fa_s = S.m[a][nf];
    T gm = T(0), gr = T(0);
    if (do_adv) {
        const T fmo = FLUX == 2 ? ro : momentum_flux(ro, C.k1, C.k2);
        const T fao = FLUX == 2 ? uo : mass_flux(uo, ro, C.r0, C.linear_mass);
        const T* cm = C.cM[a][side];
        const T* cr = C.cA[a][side];
        gm = fmo * cm[0] + fm_s * cm[1] + fao * cm[2] + fa_s * cm[3];
        gr = fmo * cr[0] + fm_s * cr[1] + fao * cr[2] + fa_s * cr[3];
    }
    if (DIFF) gr += C.cQ[a][side] * (qo + S.q[a][nf]);
    typename Pair<T>::type g;
    g.x = gm;
    g.y = gr;
    return g;
}

//
// Flux modes (FLUX; 1 and 2 only with advection on):
//   0: the volume fluxes of the element's nodes and of its face neighbours'
//      nodes are evaluated from the state;
//   1: as 0, and the fluxes of the output state are written to flux_out;
//   2: both are read from flux_in (the fluxes of src, written by the stage
//      that produced it) and those of the output are written to flux_out.
// Mode 2 trades 64 bytes of HBM traffic per node for the FP64 instructions
// of evaluating every interior face node's neighbour flux a second time
// (its own element evaluates it for its line sums).
//
// PACK: the stage's output is also written in host order to io.pack (the
// last stage of a step whose result is downloaded: a launch of its own for
// that took 20 to 30 us on 2.1 M nodes).
template <typename T, int K, bool DIFF, int FLUX, bool PACK = false>
__global__ void __launch_bounds__(npt_of(K) * epb_of(K))
stage_kernel(StageIO<T> io, MeshDev<T> m, const OpConst<T, K>* __restrict__ Cp, int do_adv, int do_sponge)
{
    constexpr int K2 = K * K, K3 = K * K * K, NPT = npt_of(K), NF = 6 * K2, R = (NF + NPT - 1) / NPT;
    constexpr int EPB = epb_of(K);
    __shared__ PlainSmem<T, K> sm_all[EPB];
    PlainSmem<T, K>& S = sm_all[threadIdx.y];
    const OpConst<T, K>& C = *Cp;
    const int n = threadIdx.x;
    const int e = blockIdx.x * EPB + threadIdx.y;
    const bool live = e < m.n_elem;
    const bool act = n < K3 && live;
    const int c[3] = {n / K2, (n / K) % K, n % K};
    const size_t off = (size_t)e * io.np + n;
    OpRows<T, K> R_;
    R_.load(C, c, act);

    T rho = T(0), u[3] = {T(0), T(0), T(0)}, q[3] = {T(0), T(0), T(0)};
    T fl[4] = {T(0), T(0), T(0), T(0)};
    if (act) {
        if (FLUX != 2) {  // mode 2 needs the state only for the stage combination
            rho = load_in(io, 0, off);
#pragma unroll
            for (int a = 0; a < 3; a++) u[a] = load_in(io, 1 + a, off);
        }
        if (DIFF)
#pragma unroll
            for (int a = 0; a < 3; a++) q[a] = __ldg(io.q + (size_t)a * io.fs + off);
        if (FLUX == 2)
#pragma unroll
            for (int f = 0; f < 4; f++) fl[f] = __ldg(io.flux_in + (size_t)f * io.fs + off);
    }
    // Neighbour (or exterior) values of this thread's face nodes: drho and
    // the normal velocity, or in flux mode 2 their momentum and mass fluxes.
    // The element's 6 K^2 face nodes are dealt out densely (slots n, n + NPT, ...).
    T ro[R], uo[R], qo[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        ro[r] = uo[r] = qo[r] = T(0);
        const int t = n + r * NPT;
        if (!live || t >= NF) continue;
        const FaceNode<K> F(t);
        const int code = __ldg(m.nbr + (size_t)e * 6 + 2 * F.a + F.side);
        if (code >= 0) {
            const size_t o2 = (size_t)code * io.np + F.nn;
            if (FLUX == 2) {
                ro[r] = __ldg(io.flux_in + o2);
                uo[r] = __ldg(io.flux_in + (size_t)(1 + F.a) * io.fs + o2);
            } else {
                ro[r] = load_in(io, 0, o2);
                uo[r] = load_in(io, 1 + F.a, o2);
            }
            if (DIFF) qo[r] = __ldg(io.q + (size_t)F.a * io.fs + o2);
        } else {
            exterior<T, K>(m, C, -1 - code, F.side, F.fi, ro[r], uo[r]);
            if (FLUX == 2) {
                const T fm = momentum_flux(ro[r], C.k1, C.k2);
                uo[r] = mass_flux(uo[r], ro[r], C.r0, C.linear_mass);
                ro[r] = fm;
            }
        }
    }

    T fmom = T(0), fmass[3] = {T(0), T(0), T(0)};
    if (FLUX == 2) {
        fmom = fl[0];
#pragma unroll
        for (int a = 0; a < 3; a++) fmass[a] = fl[1 + a];
    } else if (do_adv) {
        fmom = momentum_flux(rho, C.k1, C.k2);
#pragma unroll
        for (int a = 0; a < 3; a++) fmass[a] = mass_flux(u[a], rho, C.r0, C.linear_mass);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        S.f[a][n].x = fmom;
        S.f[a][n].y = DIFF ? fmass[a] + q[a] : fmass[a];
        S.m[a][n] = fmass[a];
        if (DIFF) S.q[a][n] = q[a];
    }
    __syncthreads();

    // Face terms: the numerical flux times its lift scale.
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int t = n + r * NPT;
        if (!live || t >= NF) continue;
        const FaceNode<K> F(t);
        S.g[F.a][F.side][F.fi] = face_term<T, K, DIFF, FLUX>(C, S, F.a, F.side, F.nf, ro[r], uo[r], qo[r], do_adv);
    }
    __syncthreads();
    if (!act) return;

    // The density equation is one FMA chain through the three axes (no
    // per-axis partial sums to add): the kernel is bound by FP64 issue, so
    // every FP64 instruction saved per node counts.
    T r_rho = T(0), r_u[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int st = axis_stride<K>(a), base = n - c[a] * st;
        const int fi = c[(a + 1) % 3] * K + c[(a + 2) % 3];
        const typename Pair<T>::type g0 = S.g[a][0][fi], gN = S.g[a][1][fi];
        T sm = R_.l0[a] * g0.x;
        sm += R_.ln[a] * gN.x;
        r_rho += R_.l0[a] * g0.y;
        r_rho += R_.ln[a] * gN.y;
#pragma unroll
        for (int j = 0; j < K; j++) {
            const typename Pair<T>::type v = S.f[a][base + j * st];
            sm += R_.d[a][j] * v.x;
            r_rho += R_.d[a][j] * v.y;
        }
        r_u[a] = do_adv ? sm : T(0);
    }
    // cb - ca sigma of this element: tabulated per stage by the host, so that
    // no thread spends FP64 instructions on it; computed here when absent.
    const T cbe = io.elem_b ? __ldg(io.elem_b + e) : io.cb - (do_sponge ? io.ca * __ldg(m.sigma + e) : T(0));
    if (FLUX == 2) {
        rho = load_in(io, 0, off);
#pragma unroll
        for (int a = 0; a < 3; a++) u[a] = load_in(io, 1 + a, off);
    }

    const T r[4] = {r_rho, r_u[0], r_u[1], r_u[2]};
    const T s4[4] = {rho, u[0], u[1], u[2]};
    T vo[4];
#pragma unroll
    for (int f = 0; f < 4; f++) {
        const size_t o = (size_t)f * io.fs + off;
        T v = r[f] + s4[f] * cbe;
        if (io.old) v += io.old[o] * io.cc;
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
        for (int f = 0; f < 4; f++) io.pack[(size_t)f * io.pack_gsize + gi] = (double)vo[f];
    }
}

// Host-side construction of the per-launch operators from the FP64 line
// operators (M^-1 S, lift columns) and the problem constants.
// ``rk_ca`` is the stage weight of R (1 for a bare right-hand side).
template <typename T, int K>
inline OpConst<T, K> make_stage_const(double rk_ca, const double* deriv, const double* lift0, const double* liftN,
                                      const double w[3], double rho0, double c0, double b_over_a,
                                      double diff_const)
{
    OpConst<T, K> C{};
    for (int a = 0; a < 3; a++)
        for (int i = 0; i < K; i++) {
            C.rows[a][i][K] = (T)lift0[i];
            C.rows[a][i][K + 1] = (T)liftN[i];
        }
    // Face-flux coefficients as the reference forms them (cppsrc/Element.cpp:542-556
    // left, :581-595 right); z = rho0 c0 and r = rho0 on both sides.
    const double r0 = rho0, z1 = r0 * c0, z2 = r0 * c0, r1 = r0, r2 = r0;
    const double cL0[4] = {z1 * r2 / (z1 + z2), z2 * r1 / (z1 + z2), z1 * z2 / r2 / (z1 + z2),
                           -1.0 * z1 * z2 / r1 / (z1 + z2)};
    const double cL1[4] = {z2 / r2 / (z1 + z2), z1 / r1 / (z1 + z2), r2 / (z1 + z2), -1.0 * r1 / (z1 + z2)};
    const double cR0[4] = {z2 * r1 / (z1 + z2), z1 * r2 / (z1 + z2), z1 * z2 / r1 / (z1 + z2),
                           -1.0 * z1 * z2 / r2 / (z1 + z2)};
    const double cR1[4] = {z1 / r1 / (z1 + z2), z2 / r2 / (z1 + z2), r1 / (z1 + z2), -1.0 * r2 / (z1 + z2)};
    for (int a = 0; a < 3; a++) {
        for (int i = 0; i < K; i++)
            for (int j = 0; j < K; j++) C.rows[a][i][j] = (T)(rk_ca * deriv[i * K + j] / w[a]);
        // momentum: lift scale -1/(rho0 w); left flux F_0 = -(fmo cL0[0] + fms cL0[1]
        // + fao cL0[2] + fas cL0[3]), right F_N = fms cR0[0] + fmo cR0[1] + fas cR0[2] + fao cR0[3]
        const double km = rk_ca * (-1.0 / (r0 * w[a]));
        const double lm[4] = {-cL0[0], -cL0[1], -cL0[2], -cL0[3]};
        const double rm[4] = {cR0[1], cR0[0], cR0[3], cR0[2]};
        // mass: lift scale -rho0/w; left F_0 = -(fao cL1[0] + fas cL1[1] + fmo cL1[2] + fms cL1[3]),
        // right F_N = fas cR1[0] + fao cR1[1] + fms cR1[2] + fmo cR1[3]
        const double ka = rk_ca * (-r0 / w[a]);
        const double la[4] = {-cL1[2], -cL1[3], -cL1[0], -cL1[1]};
        const double ra[4] = {cR1[3], cR1[2], cR1[1], cR1[0]};
        for (int i = 0; i < 4; i++) {
            C.cM[a][0][i] = (T)(km * lm[i]);
            C.cM[a][1][i] = (T)(km * rm[i]);
            C.cA[a][0][i] = (T)(ka * la[i]);
            C.cA[a][1][i] = (T)(ka * ra[i]);
        }
        // LDG divergence of G = -D_c Q: (1/w)(D G + lift(central flux of G))
        C.cQ[a][0] = (T)(0.5 * rk_ca / w[a]);
        C.cQ[a][1] = (T)(-0.5 * rk_ca / w[a]);
    }
    const FluxOut<T> fc = flux_consts<T>(nullptr, r0, c0, b_over_a);
    C.k1 = fc.k1;
    C.k2 = fc.k2;
    C.r0 = fc.r0;
    C.inv_c2 = (T)(1.0 / (c0 * c0));
    C.inv_z = (T)(1.0 / (r0 * c0));
    C.linear_mass = fc.linear;
    (void)diff_const;
    return C;
}

template <typename T, int K>
inline OpConst<T, K> make_grad_const(const double* deriv, const double* lift0, const double* liftN,
                                     const double w[3], double rho0, double c0, double diff_const)
{
    OpConst<T, K> C{};
    for (int a = 0; a < 3; a++) {
        // central flux of drho, (+0.5, -0.5) D_c / w_a, folded into the lift
        // columns: the kernels lift the plain face sum (own + other)
        const double q0 = 0.5 * diff_const / w[a], qN = -0.5 * diff_const / w[a];
        for (int i = 0; i < K; i++) {
            for (int j = 0; j < K; j++) C.rows[a][i][j] = (T)(diff_const * deriv[i * K + j] / w[a]);
            C.rows[a][i][K] = (T)(lift0[i] * q0);
            C.rows[a][i][K + 1] = (T)(liftN[i] * qN);
        }
        C.cQ[a][0] = C.cQ[a][1] = T(1);
    }
    C.inv_c2 = (T)(1.0 / (c0 * c0));
    C.inv_z = (T)(1.0 / (rho0 * c0));
    return C;
}

// State <-> host-order arrays rho [X][Y][Z], vel [3][X][Y][Z], walked in host
// order so that rho/vel may be pinned host memory read or written directly by
// the kernel (streaming, coalesced on the host side), or device staging.  A
// CTA takes one (x, y) row at a time and its threads walk z, so the element
// arithmetic is 32-bit and mostly per row.
struct RowMap {
    int elem_xy;  // element-index part of the row's element coordinates
    int node_xy;  // (a K + b) K: node-index part of the row
};

__device__ __forceinline__ RowMap row_map(const GridMap& g, int ii, int jj)
{
    const int K = g.K;
    const int gx = ii / K, gy = jj / K;
    const int bx = gx / g.ne[0], by = gy / g.ne[1], lx = gx % g.ne[0], ly = gy % g.ne[1];
    return {(bx * g.nb[1] + by) * g.nb[2] * g.elem_per_block + (lx * g.ne[1] + ly) * g.ne[2],
            ((ii % K) * K + jj % K) * K};
}

__device__ __forceinline__ size_t row_offset(const GridMap& g, int np, const RowMap& r, int kk)
{
    const int gz = kk / g.K;
    const int e = r.elem_xy + (gz / g.ne[2]) * g.elem_per_block + gz % g.ne[2];
    return (size_t)e * np + r.node_xy + kk % g.K;
}

template <typename T>
__global__ void pack_host_order_kernel(const T* __restrict__ state, size_t fs, int np, GridMap g,
                                       double* __restrict__ rho, double* __restrict__ vel, size_t gsize)
{
    const int Y = g.E[1] * g.K, Z = g.E[2] * g.K, rows = g.E[0] * g.K * Y;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const RowMap r = row_map(g, row / Y, row % Y);
        for (int kk = threadIdx.x; kk < Z; kk += blockDim.x) {
            const size_t o = row_offset(g, np, r, kk), i = (size_t)row * Z + kk;
            if (rho) rho[i] = (double)state[o];
            if (vel)
#pragma unroll
                for (int a = 0; a < 3; a++) vel[a * gsize + i] = (double)state[(size_t)(1 + a) * fs + o];
        }
    }
}

template <typename T>
__global__ void unpack_host_order_kernel(T* __restrict__ state, size_t fs, int np, GridMap g,
                                         const double* __restrict__ rho, const double* __restrict__ vel, size_t gsize,
                                         FluxOut<T> fo)
{
    const int Y = g.E[1] * g.K, Z = g.E[2] * g.K, rows = g.E[0] * g.K * Y;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const RowMap r = row_map(g, row / Y, row % Y);
        for (int kk = threadIdx.x; kk < Z; kk += blockDim.x) {
            const size_t o = row_offset(g, np, r, kk), i = (size_t)row * Z + kk;
            const T d = (T)rho[i];
            T u[3];
            state[o] = d;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                u[a] = (T)vel[a * gsize + i];
                state[(size_t)(1 + a) * fs + o] = u[a];
            }
            if (fo.f) write_fluxes(fo, fs, o, d, u);
        }
    }
}

// Host-order device staging -> state, walked in element order: the state
// writes are contiguous per element and the scattered side is the read
// (K-value runs along z), which costs less than partial-sector writes.  For
// device memory only; pinned host memory is read by unpack_host_order_kernel.
template <typename T>
__global__ void unpack_elem_order_kernel(T* __restrict__ state, size_t fs, int np, GridMap g, int n_elem,
                                         const double* __restrict__ rho, const double* __restrict__ vel, size_t gsize,
                                         FluxOut<T> fo)
{
    const int K3 = g.K * g.K * g.K;
    const size_t total = (size_t)n_elem * np;
    for (size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x; s < total; s += (size_t)gridDim.x * blockDim.x) {
        const int e = (int)(s / np), n = (int)(s % np);
        if (n >= K3) continue;
        const size_t i = grid_index(g, e, n);
        const T d = (T)rho[i];
        T u[3];
        state[s] = d;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            u[a] = (T)vel[a * gsize + i];
            state[(size_t)(1 + a) * fs + s] = u[a];
        }
        if (fo.f) write_fluxes(fo, fs, s, d, u);
    }
}

template <typename T>
__global__ void pack_grid_kernel(const T* __restrict__ state, size_t fs, int np, int nfields,
                                 GridMap g, int n_elem, double* __restrict__ out, size_t gsize)
{
    const int K3 = g.K * g.K * g.K;
    const long long total = (long long)n_elem * K3;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int e = (int)(i / K3), n = (int)(i % K3);
        const size_t gi = grid_index(g, e, n);
        for (int f = 0; f < nfields; f++)
            out[(size_t)f * gsize + gi] = (double)state[(size_t)f * fs + (size_t)e * np + n];
    }
}


}  // namespace dg
