// K4: two-phase colour-gradient step (2phase/lbm_solver_3d_2phase_sparse.py, "TP").
//
// The reference's step (TP:626-632) is colission (MRT + colour gradient + CapA
// surface tension + recolouring + colour push, :302-373), streaming1,
// Boundary_condition, streaming3 (macros, colour sums, psi, :587-606) and
// Boundary_condition_psi (:445-487).  Collision at a node needs psi at its
// neighbours *after* the previous step, so one step is two launches:
//
//   A  tp_colour_kernel: pull the colour distributions.  rho_r(y) = sum over s
//      of g_r(y - e_s)[s] (or g_r(y)[LR[s]] when y - e_s is solid), g recomputed
//      at the source from its stored (rho_r, rho_b, v) and its 9 recolouring
//      amounts; then psi = rho_r - rho_b/(rho_r + rho_b) (TP:606, kept as the
//      reference writes it) and constant-psi faces.
//   B  tp_flow_kernel: gather F, face BCs, macros; colour gradient C from psi of
//      the neighbours (clamped on constant-psi faces, TP:390-429); psi-dependent
//      relaxation (TP:278-300); CapA terms in meq (TP:316-322); MRT + script Guo;
//      store f, v, rho and the node's 9 recolouring amounts (TP:352-364) for the
//      next step's launch A.
//
// The colour sums are taken in direction order 0..18, one of the orders the
// reference's atomic += can produce; the CPU oracle uses the same order, so
// the two agree bit for bit.
//
// What a node's neighbours pull of it, (rho_r, rho_b, v_x, v_y) as one 16-byte
// record, v_z and its 9 amounts, launch B leaves behind, so a direction costs three
// loads.  Sources, and the psi neighbours of launch B away from the lattice
// faces, come from the neighbour links (lbm_links.cuh).  v and rho are stored
// only when the caller reads them next (MACROS) or, for v, where a pressure
// face needs the previous step's.
//
// 131^3 drainage, FP32, 898k nodes: 81.0 us a step against 98.4 with six scalar
// loads a direction and map lookups.  Launch A is bound by L1 wavefronts (every
// direction reads its own 24 unaligned bytes: 71% of the data pipe, 65% of the
// issue slots), launch B by issue slots (66%) and latency at 72 registers; its psi
// loads wait together with the populations' (after the faces 83.0 us).  Storing the 38 recoloured
// populations instead (two values a direction in launch A) took a third of the
// wavefronts but 140 MB more DRAM traffic a step: 94 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "lbm_kernels.cuh"
#include "lbm_linkgather.cuh"

// Resident 128-thread CTAs per SM of the two launches (FP32 and 16-bit), us a step
// on the same lattice / on a 50 x 44 x 37 sample, before records were looked up with
// the links (81.0 / 13.1 since): 10 and 7 81.8 / 13.3; 10 and 8
// 81.7 / 14.6; 10 and 9 86.6 / 16.4; 10 and 6 87.5 / 15.6; 9 and 7 88.1, 12 and 7 84.2.
#ifndef LBM_TP_MINBLOCKS_A
#define LBM_TP_MINBLOCKS_A 10
#endif
#ifndef LBM_TP_MINBLOCKS_B
#define LBM_TP_MINBLOCKS_B 7
#endif

namespace {
using namespace lbmk;

constexpr int TP_THREADS = 128;

template <typename R>
struct TpConsts {
    SpConsts<R> sp;
    R wl, wg, lg0, l1, l2, g1, g2;  // TP:102-110, folded to R
    R psi_solid, capa, hcapa;       // hcapa = 0.5 * capa
    int32_t psi_bc[6];
    int32_t any_psi_bc;
    R psi_val[6], psi_rr[6], psi_rb[6];
};

// What launch A pulls of a node, beside v_z and the amounts.
template <typename R>
struct __align__(4 * sizeof(R)) ColourRec {
    R rr, rb, vx, vy;
};

// Compute_S_local (TP:278-300): s_v and s_other from psi.
template <typename R>
__device__ __forceinline__ void s_local(const TpConsts<R>& T, R psi, R& sv, R& so) {
    if (psi > (R)0) {
        if (psi > (R)0.1) sv = T.wl;
        else sv = (T.lg0 + T.l1 * psi) + (T.l2 * psi) * psi;
    } else {
        if (psi < (R)-0.1) sv = T.wg;
        else sv = (T.lg0 + T.g1 * psi) + (T.g2 * psi) * psi;
    }
    so = ((R)8.0 * ((R)2.0 - sv)) / ((R)8.0 - sv);
}

// periodic_index_for_psi (TP:390-429) for one coordinate.
__device__ __forceinline__ int psi_wrap(int x, int n, int bc_lo, int bc_hi) {
    if (x < 0) return bc_lo == 0 ? n - 1 : 0;
    if (x > n - 1) return bc_hi == 0 ? 0 : n - 1;
    return x;
}

// Compute_C (TP:259-276): C = sum_s 3 w_s e_s psi(x + e_s), psi_solid at solid
// neighbours; zero when |rho_r - rho_b| > 0.9 next to a solid.
template <typename R>
__device__ __forceinline__ void colour_gradient(const TpConsts<R>& T, const int32_t* __restrict__ map,
                                                const R* __restrict__ psi, int i, int j, int k, R rr, R rb, R& Cx,
                                                R& Cy, R& Cz) {
    const int nx = T.sp.nx, ny = T.sp.ny, nz = T.sp.nz;
    const int xm = psi_wrap(i - 1, nx, T.psi_bc[0], T.psi_bc[1]), xp = psi_wrap(i + 1, nx, T.psi_bc[0], T.psi_bc[1]);
    const int ym = psi_wrap(j - 1, ny, T.psi_bc[2], T.psi_bc[3]), yp = psi_wrap(j + 1, ny, T.psi_bc[2], T.psi_bc[3]);
    const int zm = psi_wrap(k - 1, nz, T.psi_bc[4], T.psi_bc[5]), zp = psi_wrap(k + 1, nz, T.psi_bc[4], T.psi_bc[5]);
    Cx = (R)0;
    Cy = (R)0;
    Cz = (R)0;
    bool touch = false;
#pragma unroll
    for (int s = 1; s < 19; ++s) {
        const int ex = lbm_ex(s), ey = lbm_ey(s), ez = lbm_ez(s);
        const int x = ex > 0 ? xp : (ex < 0 ? xm : i);
        const int y = ey > 0 ? yp : (ey < 0 ? ym : j);
        const int z = ez > 0 ? zp : (ez < 0 ? zm : k);
        const int nb = __ldg(map + x + nx * (y + ny * z));
        R ps;
        if (nb >= 0) {
            ps = psi[nb];
        } else {
            ps = T.psi_solid;
            touch = true;
        }
        const R t = ((R)3.0 * (R)lbm_w(s)) * ps;
        if (ex != 0) Cx = ex > 0 ? Cx + t : Cx - t;
        if (ey != 0) Cy = ey > 0 ? Cy + t : Cy - t;
        if (ez != 0) Cz = ez > 0 ? Cz + t : Cz - t;
    }
    R dr = rr - rb;
    if (dr < (R)0) dr = -dr;
    if (dr > (R)0.9 && touch) {
        Cx = (R)0;
        Cy = (R)0;
        Cz = (R)0;
    }
}

// Colour gradient of a node away from the lattice faces: the neighbour at
// x + e_s is the pull source of the opposite direction.  Same order of terms.
template <typename R>
__device__ __forceinline__ void colour_gradient_links(const TpConsts<R>& T, const NodeLinks& K, int n, const R* psi,
                                                      R rr, R rb, R& Cx, R& Cy, R& Cz) {
    Cx = (R)0;
    Cy = (R)0;
    Cz = (R)0;
#define LBM_CG(S)                                                          \
    {                                                                      \
        constexpr int q = lbm_lr(S);                                       \
        constexpr int ex = lbm_ex(S), ey = lbm_ey(S), ez = lbm_ez(S);      \
        R ps = T.psi_solid;                                                \
        if (!(K.bits >> q & 1u)) ps = psi[K.template source<q>(n)];        \
        const R t = ((R)3.0 * (R)lbm_w(S)) * ps;                           \
        if constexpr (ex != 0) Cx = ex > 0 ? Cx + t : Cx - t;              \
        if constexpr (ey != 0) Cy = ey > 0 ? Cy + t : Cy - t;              \
        if constexpr (ez != 0) Cz = ez > 0 ? Cz + t : Cz - t;              \
    }
    LBM_ALL_DIRS(LBM_CG)
#undef LBM_CG
    R dr = rr - rb;
    if (dr < (R)0) dr = -dr;
    if (dr > (R)0.9 && (K.bits & 0x7fffeu)) {
        Cx = (R)0;
        Cy = (R)0;
        Cz = (R)0;
    }
}

// Normal C / |C| and recolouring amounts of the 9 opposite pairs (TP:346-364):
// cospsi_p for kk = 2p+1; all zero when |C| = 0 (no recolouring).
template <typename R>
__device__ __forceinline__ void recolour_amounts(R rr, R rb, R vx, R vy, R vz, R Cx, R Cy, R Cz, R cc, R u15, R* nrm,
                                                 R* cs) {
    R q[12];
#pragma unroll
    for (int p = 0; p < 12; ++p) q[p] = (R)0;
    if (cc > (R)0) {
        q[9] = Cx;
        q[10] = Cy;
        q[11] = Cz;
#define LBM_RC(P) q[P] = lbm_edot<2 * P + 1, R>(Cx, Cy, Cz);
        LBM_RC(0) LBM_RC(1) LBM_RC(2) LBM_RC(3) LBM_RC(4) LBM_RC(5) LBM_RC(6) LBM_RC(7) LBM_RC(8)
#undef LBM_RC
        quotients(q, cc);
#define LBM_RC(P)                                                                                       \
    {                                                                                                   \
        constexpr int kk = 2 * P + 1;                                                                   \
        /* feq of kk and kk + 1 (e.u and -e.u) for both colours (lbm_feq, term by term) */              \
        const R eu = lbm_edot<kk, R>(vx, vy, vz);                                                       \
        const R e3 = (R)3.0 * eu, e45 = ((R)4.5 * eu) * eu;                                             \
        const R tp = (((R)1.0 + e3) + e45) - u15, tm = (((R)1.0 - e3) + e45) - u15;                     \
        const R wr = (R)lbm_w(kk) * rr, wb = (R)lbm_w(kk) * rb;                                         \
        const R ga = wr * tp, gb = wr * tm, ba = wb * tp, bb = wb * tm;                                 \
        R cp = ga < gb ? ga : gb;                                                                       \
        cp = cp < ba ? cp : ba;                                                                         \
        cp = cp < bb ? cp : bb;                                                                         \
        q[P] = cp * q[P];                                                                               \
    }
        LBM_RC(0) LBM_RC(1) LBM_RC(2) LBM_RC(3) LBM_RC(4) LBM_RC(5) LBM_RC(6) LBM_RC(7) LBM_RC(8)
#undef LBM_RC
    }
#pragma unroll
    for (int p = 0; p < 9; ++p) cs[p] = q[p];
#pragma unroll
    for (int d = 0; d < 3; ++d) nrm[d] = q[9 + d];
}

// Two-phase MRT collision (TP:302-344) of F in place.
template <typename R, int FORCE, bool FAST>
__device__ __forceinline__ void collide_tp(R* F, R r, R vx, R vy, R vz, R cc, R n0, R n1, R n2, R sv, R so,
                                           const TpConsts<R>& T) {
    R m[19];
    if constexpr (FAST) mrt_moments_fast<R>(F, m);
    else mrt_moments<R>(F, m);
    R meq[19];
#pragma unroll
    for (int s = 0; s < 19; ++s) meq[s] = (R)0;
    meq[0] = r; meq[3] = vx; meq[5] = vy; meq[7] = vz;
    meq[1] = lbm_usq(vx, vy, vz);
    meq[9] = (((R)2 * vx) * vx - vy * vy) - vz * vz;
    meq[11] = vy * vy - vz * vz;
    meq[13] = vx * vy; meq[14] = vy * vz; meq[15] = vx * vz;
    const R hc = T.hcapa * cc;
    meq[1] = meq[1] + T.capa * cc;
    meq[9] = meq[9] + hc * ((((R)2 * n0) * n0 - n1 * n1) - n2 * n2);
    meq[11] = meq[11] + hc * (n1 * n1 - n2 * n2);
    meq[13] = meq[13] + hc * (n0 * n1);
    meq[14] = meq[14] + hc * (n1 * n2);
    meq[15] = meq[15] + hc * (n0 * n2);
#pragma unroll
    for (int s = 0; s < 19; ++s) {
        const int kd = lbm_skind(s);
        if (kd == 0) continue;
        const R S = kd == 1 ? sv : so;
        if constexpr (FAST) m[s] = lbm_fma<R>(S, meq[s] - m[s], m[s]);
        else m[s] = m[s] - S * (m[s] - meq[s]);
    }
    if constexpr (FORCE) {
        R G[19];
        guo_dense<R, FORCE>(G, vx, vy, vz, T.sp.fext, 1);   // GuoF, TP:242-248
        R fg[19];
        if constexpr (FAST) mrt_moments_fast<R>(G, fg);
        else mrt_moments<R>(G, fg);
#pragma unroll
        for (int s = 0; s < 19; ++s) {
            const int kd = lbm_skind(s);
            const R S = kd == 0 ? (R)0 : (kd == 1 ? sv : so);
            if constexpr (FAST) m[s] = lbm_fma<R>((R)1 - (R)0.5 * S, fg[s], m[s]);
            else m[s] = m[s] + ((R)1 - (R)0.5 * S) * fg[s];
        }
    }
    if constexpr (FAST) mrt_back_fast<R>(m, F);
    else mrt_back<R>(m, F);
}

// Everything B does after the macros: recolouring amounts, collision, and what
// the next launch A pulls.
template <int STORE, int FORCE>
__device__ __forceinline__ void tp_collide_and_store(typename Codec<STORE>::R* F, typename Codec<STORE>::R r,
                                                     typename Codec<STORE>::R vx, typename Codec<STORE>::R vy,
                                                     typename Codec<STORE>::R vz, int n,
                                                     typename Codec<STORE>::R ref_own,
                                                     const TpConsts<typename Codec<STORE>::R>& T,
                                                     typename Codec<STORE>::R Cx, typename Codec<STORE>::R Cy,
                                                     typename Codec<STORE>::R Cz, typename Codec<STORE>::R psi,
                                                     typename Codec<STORE>::R rr, typename Codec<STORE>::R rb,
                                                     typename Codec<STORE>::T* __restrict__ fout,
                                                     ColourRec<typename Codec<STORE>::R>* __restrict__ crec,
                                                     typename Codec<STORE>::R* __restrict__ pull_vz,
                                                     typename Codec<STORE>::R* __restrict__ cs_out) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    const int64_t np = T.sp.np;
    const R cc = sqrt(lbm_usq(Cx, Cy, Cz));
    const R u15 = (R)1.5 * lbm_usq(vx, vy, vz);
    R nrm[3], cs[9];
    recolour_amounts<R>(rr, rb, vx, vy, vz, Cx, Cy, Cz, cc, u15, nrm, cs);
#pragma unroll
    for (int p = 0; p < 9; ++p) cs_out[p * np + n] = cs[p];
    crec[n] = {rr, rb, vx, vy};
    pull_vz[n] = vz;
    R sv, so;
    s_local<R>(T, psi, sv, so);
    collide_tp<R, FORCE, Cd::DEV>(F, r, vx, vy, vz, cc, nrm[0], nrm[1], nrm[2], sv, so, T);
    store_node<STORE>(F, fout, n, ref_own, T.sp.seed);
}

// Programmatic dependent launch between the step's launches (A, B, next A):
// a launch's CTAs may become resident while the previous launch drains; they
// load their coordinates, then wait for it to complete before touching any
// state (the wait returns at once for a launch without the attribute).
__device__ __forceinline__ void tp_pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename K, typename... Args>
cudaError_t tp_launch_pdl(K kernel, int grid, int block, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// ---------------------------------------------------------------- launch A
// Direction Q: what the node at x - e_Q (or, bounced, the node itself in the
// opposite direction) sends.  EXC: some node of the warp has a record.
template <int Q, bool EXC, typename R>
__device__ __forceinline__ void colour_pull_one(const NodeLinks& K, const int32_t* rec, int64_t np, int n,
                                                const ColourRec<R>* crec, const R* pull_vz, const R* cs,
                                                R& acc_r, R& acc_b) {
    bool bounce = false;
    int m = n;
    if constexpr (Q != 0) {
        bounce = K.bits >> Q & 1u;
        if (!bounce) m = K.template source<Q>(n);
        if constexpr (EXC)
            if (bounce && (K.bits & LBM_LINK_EXC)) {
                const int to = __ldg(rec + Q);
                if (to >= 0) {
                    m = to;
                    bounce = false;
                }
            }
    }
    const ColourRec<R> a = crec[m];
    const R vz = pull_vz[m];
    R eu = lbm_edot<Q, R>(a.vx, a.vy, vz);
    if (bounce) eu = -eu;  // direction LR[Q] at the node itself: e_LR = -e_Q
    R t = (R)1.0 + (R)3.0 * eu;
    t = t + ((R)4.5 * eu) * eu;
    t = t - (R)1.5 * lbm_usq(a.vx, a.vy, vz);
    R gr = ((R)lbm_w(Q) * a.rr) * t;
    R gb = ((R)lbm_w(Q) * a.rb) * t;
    if constexpr (Q != 0) {
        // pair kk = 2p+1 gets +cospsi for red (kk) and -cospsi (kk+1); blue opposite
        R c = cs[((Q - 1) >> 1) * np + m];
        if (((Q & 1) != 0) == bounce) c = -c;
        gr = gr + c;
        gb = gb - c;
    }
    acc_r = acc_r + gr;
    acc_b = acc_b + gb;
}

template <typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 4 : LBM_TP_MINBLOCKS_A) tp_colour_kernel(
    const __grid_constant__ TpConsts<R> T, const ColourRec<R>* crec_prev, const R* vz_prev, const R* cs_prev,
    R* __restrict__ rr_out, R* __restrict__ rb_out, R* __restrict__ psi_out, const __grid_constant__ LbmLinks L,
    const uint32_t* __restrict__ coord) {
    tp_pdl_launch_dependents();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= T.sp.n_fluid) return;
    NodeLinks K;
    K.load(L, n);
    const bool exc = K.any_record();
    const int32_t* rec = K.record(L);
    // records and amounts of the previous flow launch; psi is rewritten below
    const ColourRec<R>* crec = wait_previous(crec_prev);
    const R* vz = launder(vz_prev);
    const R* cs = launder(cs_prev);
    R ar = (R)0, ab = (R)0;
    if (exc) {
#define LBM_CP(Q) colour_pull_one<Q, true, R>(K, rec, T.sp.np, n, crec, vz, cs, ar, ab);
        LBM_CP(0) LBM_ALL_DIRS(LBM_CP)
#undef LBM_CP
    } else {
#define LBM_CP(Q) colour_pull_one<Q, false, R>(K, rec, T.sp.np, n, crec, vz, cs, ar, ab);
        LBM_CP(0) LBM_ALL_DIRS(LBM_CP)
#undef LBM_CP
    }
    R psi = ar - ab / (ar + ab);  // TP:606 as written
    if (T.any_psi_bc && (K.bits & LBM_LINK_EDGE)) {
        const uint32_t pc = __ldg(coord + n);
        const int i = lbm_pi(pc), j = lbm_pj(pc), k = lbm_pk(pc);
#pragma unroll 1
        for (int f = 0; f < 6; ++f) {
            if (!T.psi_bc[f]) continue;
            const int hi = f & 1;
            const int c = f < 2 ? i : (f < 4 ? j : k);
            const int nmax = f < 2 ? T.sp.nx : (f < 4 ? T.sp.ny : T.sp.nz);
            if (c != (hi ? nmax - 1 : 0)) continue;
            psi = T.psi_val[f];
            ar = T.psi_rr[f];
            ab = T.psi_rb[f];
        }
    }
    rr_out[n] = ar;
    rb_out[n] = ab;
    psi_out[n] = psi;
}

// ---------------------------------------------------------------- launch B
template <int STORE, int FORCE, bool MACROS>
__global__ void __launch_bounds__(128, STORE == LBM_STORE_F64 ? 2 : LBM_TP_MINBLOCKS_B) tp_flow_kernel(
    const __grid_constant__ TpConsts<typename Codec<STORE>::R> T, const typename Codec<STORE>::T* f_prev,
    typename Codec<STORE>::T* __restrict__ fout, const int32_t* __restrict__ map, const uint32_t* __restrict__ coord,
    const __grid_constant__ LbmLinks L, typename Codec<STORE>::R* v, typename Codec<STORE>::R* __restrict__ rho_out,
    const typename Codec<STORE>::R* rr_new, const typename Codec<STORE>::R* rb_new,
    const typename Codec<STORE>::R* psi_new, ColourRec<typename Codec<STORE>::R>* __restrict__ crec,
    typename Codec<STORE>::R* __restrict__ pull_vz, typename Codec<STORE>::R* __restrict__ cs_out) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    const SpConsts<R>& C = T.sp;
    tp_pdl_launch_dependents();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= C.n_fluid) return;
    NodeLinks K;
    K.load(L, n);
    int i = 0, j = 0, k = 0;
    if (Cd::RHOREF || (K.bits & (LBM_LINK_EDGE | LBM_LINK_EXC))) {
        const uint32_t pc = __ldg(coord + n);
        i = lbm_pi(pc);
        j = lbm_pj(pc);
        k = lbm_pk(pc);
    }
    LinkRef<R> rx;
    if constexpr (Cd::RHOREF) rx = LinkRef<R>(sp_ref(C), i, C.nx, K);
    const int64_t np = C.np;
    // rho_r, rho_b, psi of the colour launch; f, v of the previous step
    const auto* fin = wait_previous(f_prev);
    const R* psi = launder(psi_new);
    const R rr = launder(rr_new)[n], rb = launder(rb_new)[n];
    R F[19];
    LinkGather<STORE, Cd::RHOREF>::all(F, fin, L, K, n, rx);
    // (before the faces: its loads then wait together with those of F)
    R Cx, Cy, Cz;
    if (K.bits & (LBM_LINK_EDGE | LBM_LINK_EXC)) colour_gradient<R>(T, map, psi, i, j, k, rr, rb, Cx, Cy, Cz);
    else colour_gradient_links<R>(T, K, n, psi, rr, rb, Cx, Cy, Cz);
    const R psi_own = psi[n];
    if (K.bits & LBM_LINK_FACE) apply_faces<R, Cd::DEV>(F, i, j, k, n, C, map, v);  // v: previous step
    R r = F[0];
#pragma unroll
    for (int s = 1; s < 19; ++s) r = r + F[s];
    const R rho = Cd::DEV ? (R)1 + r : r;
    R vx = vsum<0>(F), vy = vsum<1>(F), vz = vsum<2>(F);
    velocity<R, FORCE>(vx, vy, vz, rho, C.fhalf);
    if (MACROS) rho_out[n] = rho;
    if (MACROS || (K.bits & LBM_LINK_PRESSURE)) {
        v[n] = vx;
        v[np + n] = vy;
        v[2 * np + n] = vz;
    }
    tp_collide_and_store<STORE, FORCE>(F, r, vx, vy, vz, n, rx.at, T, Cx, Cy, Cz, psi_own, rr, rb, fout, crec,
                                       pull_vz, cs_out);
}

// Initial state (TP:174-187) and the first collision: rho = 1, v = 0, F = feq(1, 0),
// rho_r = (psi + 1)/2, rho_b = 1 - rho_r, psi = the input psi (dense, psi0).
template <int STORE>
__global__ void tp_psi_kernel(const __grid_constant__ TpConsts<typename Codec<STORE>::R> T,
                              const uint32_t* __restrict__ coord, const float* __restrict__ psi0,
                              typename Codec<STORE>::R* __restrict__ psi) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= T.sp.n_fluid) return;
    const uint32_t pc = __ldg(coord + n);
    psi[n] = (typename Codec<STORE>::R)psi0[lbm_pi(pc) + (int64_t)T.sp.nx * (lbm_pj(pc) + (int64_t)T.sp.ny * lbm_pk(pc))];
}

template <int STORE, int FORCE>
__global__ void tp_init_kernel(const __grid_constant__ TpConsts<typename Codec<STORE>::R> T,
                               typename Codec<STORE>::T* __restrict__ fout, const int32_t* __restrict__ map,
                               const uint32_t* __restrict__ coord, typename Codec<STORE>::R* __restrict__ v,
                               typename Codec<STORE>::R* __restrict__ rho_out, typename Codec<STORE>::R* __restrict__ rr,
                               typename Codec<STORE>::R* __restrict__ rb, const typename Codec<STORE>::R* __restrict__ psi,
                               ColourRec<typename Codec<STORE>::R>* __restrict__ crec,
                               typename Codec<STORE>::R* __restrict__ pull_vz,
                               typename Codec<STORE>::R* __restrict__ cs_out) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= T.sp.n_fluid) return;
    const uint32_t pc = __ldg(coord + n);
    const int i = lbm_pi(pc), j = lbm_pj(pc), k = lbm_pk(pc);
    const int64_t np = T.sp.np;
    const R p = psi[n];
    const R r0 = (p + (R)1.0) / (R)2.0;
    const R b0 = (R)1.0 - r0;
    rr[n] = r0;
    rb[n] = b0;
    v[n] = (R)0;
    v[np + n] = (R)0;
    v[2 * np + n] = (R)0;
    rho_out[n] = (R)1.0;
    R F[19];
    if constexpr (Cd::DEV) lbm_feq_dev_all<R>((R)0, (R)0, (R)0, (R)0, F);
    else lbm_feq_all<R>((R)1.0, (R)0, (R)0, (R)0, F);
    R Cx, Cy, Cz;
    colour_gradient<R>(T, map, psi, i, j, k, r0, b0, Cx, Cy, Cz);
    tp_collide_and_store<STORE, FORCE>(F, Cd::DEV ? (R)0 : (R)1.0, (R)0, (R)0, (R)0, n, lbm_ref_at(sp_ref(T.sp), i), T,
                                       Cx, Cy, Cz, p, r0, b0, fout, crec, pull_vz, cs_out);
}

template <typename R>
TpConsts<R> make_tp(const LbmHandle* h) {
    const LbmParams& p = h->p;
    TpConsts<R> T{};
    T.sp = sp_make_consts<R>(h);
    const double wl = 1.0 / (p.niu_l / (1.0 / 3.0) + 0.5);
    const double wg = 1.0 / (p.niu_g / (1.0 / 3.0) + 0.5);
    const double lg0 = 2 * wl * wg / (wl + wg);
    const double l1 = 2 * (wl - lg0) * 10, l2 = -l1 / 0.2;
    const double g1 = 2 * (lg0 - wg) * 10, g2 = g1 / 0.2;
    T.wl = (R)wl; T.wg = (R)wg; T.lg0 = (R)lg0; T.l1 = (R)l1; T.l2 = (R)l2; T.g1 = (R)g1; T.g2 = (R)g2;
    T.psi_solid = (R)p.psi_solid;
    T.capa = (R)p.cap_a;
    T.hcapa = (R)0.5 * T.capa;
    T.any_psi_bc = 0;
    for (int f = 0; f < 6; ++f) {
        T.psi_bc[f] = p.psi_bc[f];
        T.any_psi_bc |= p.psi_bc[f] != 0;
        T.psi_val[f] = (R)p.psi_val[f];
        T.psi_rr[f] = (T.psi_val[f] + (R)1.0) / (R)2.0;
        T.psi_rb[f] = (R)1.0 - T.psi_rr[f];
    }
    return T;
}

template <int STORE>
int tp_init_t(LbmHandle* h) {
    using R = typename Codec<STORE>::R;
    using Tt = typename Codec<STORE>::T;
    const TpConsts<R> T = make_tp<R>(h);
    h->cur = 0;
    const int grid = (int)((h->n_fluid + h->block - 1) / h->block);
    tp_psi_kernel<STORE><<<grid, h->block, 0, h->stream>>>(T, h->d_coord, h->d_psi0, (R*)h->d_psi);
    auto k = h->force ? tp_init_kernel<STORE, FORCE_ANY> : tp_init_kernel<STORE, FORCE_NONE>;
    k<<<grid, h->block, 0, h->stream>>>(T, (Tt*)h->d_f[0], h->d_map, h->d_coord, (R*)h->d_v, (R*)h->d_rho,
                                        (R*)h->d_rr, (R*)h->d_rb, (const R*)h->d_psi, (ColourRec<R>*)h->d_crec,
                                        (R*)h->d_pull_vz, (R*)h->d_cs);
    int rc = lbm_cuda_check(h, cudaGetLastError(), "tp_init_kernel launch");
    if (!rc) rc = lbm_cuda_check(h, cudaStreamSynchronize(h->stream), "tp_init");
    return rc;
}

template <int STORE, int FORCE>
int tp_steps_t(LbmHandle* h, int32_t nsteps, bool macros_last) {
    using R = typename Codec<STORE>::R;
    using Tt = typename Codec<STORE>::T;
    TpConsts<R> T = make_tp<R>(h);
    const int block = std::min<int>(h->block, TP_THREADS);
    const int grid = (int)((h->n_fluid + block - 1) / block);
    for (int32_t it = 0; it < nsteps; ++it) {
        T.sp.seed = (uint32_t)(h->steps_done + it);   // global step index: rounding bits of this step
        cudaError_t e = tp_launch_pdl(tp_colour_kernel<R>, grid, block, h->stream, T, (const ColourRec<R>*)h->d_crec,
                                      (const R*)h->d_pull_vz, (const R*)h->d_cs, (R*)h->d_rr, (R*)h->d_rb,
                                      (R*)h->d_psi, h->links, (const uint32_t*)h->d_coord);
        int rc = lbm_cuda_check(h, e != cudaSuccess ? e : cudaGetLastError(), "tp_colour_kernel launch");
        if (rc) return rc;
        auto kb = macros_last && it == nsteps - 1 ? tp_flow_kernel<STORE, FORCE, true> : tp_flow_kernel<STORE, FORCE, false>;
        e = tp_launch_pdl(kb, grid, block, h->stream, T, (const Tt*)h->d_f[h->cur], (Tt*)h->d_f[h->cur ^ 1],
                          (const int32_t*)h->d_map, (const uint32_t*)h->d_coord, h->links, (R*)h->d_v, (R*)h->d_rho,
                          (const R*)h->d_rr, (const R*)h->d_rb, (const R*)h->d_psi, (ColourRec<R>*)h->d_crec,
                          (R*)h->d_pull_vz, (R*)h->d_cs);
        rc = lbm_cuda_check(h, e != cudaSuccess ? e : cudaGetLastError(), "tp_flow_kernel launch");
        if (rc) return rc;
        h->cur ^= 1;
    }
    return LBM_OK;
}

template <int STORE>
int tp_steps(LbmHandle* h, int32_t n, bool macros_last) {
    switch (force_kind(h)) {
    case FORCE_NONE: return tp_steps_t<STORE, FORCE_NONE>(h, n, macros_last);
    case FORCE_X: return tp_steps_t<STORE, FORCE_X>(h, n, macros_last);
    }
    return tp_steps_t<STORE, FORCE_ANY>(h, n, macros_last);
}

}  // namespace

int tp_launch_init(LbmHandle* h) {
    if (h->n_fluid == 0) {   // all solid: nothing to initialise (an empty grid is not launchable)
        h->cur = 0;
        return LBM_OK;
    }
    switch (h->p.storage) {
    case LBM_STORE_F32: return tp_init_t<LBM_STORE_F32>(h);
    case LBM_STORE_F16_DEV: return tp_init_t<LBM_STORE_F16_DEV>(h);
    case LBM_STORE_BF16_DEV: return tp_init_t<LBM_STORE_BF16_DEV>(h);
    case LBM_STORE_F32_DEV: return tp_init_t<LBM_STORE_F32_DEV>(h);
    case LBM_STORE_F64: return tp_init_t<LBM_STORE_F64>(h);
    }
    return lbm_set_err(h, LBM_EINVAL, "unknown storage");
}

int tp_launch_steps(LbmHandle* h, int32_t n, bool macros_last) {
    if (h->n_fluid == 0) return LBM_OK;
    switch (h->p.storage) {
    case LBM_STORE_F32: return tp_steps<LBM_STORE_F32>(h, n, macros_last);
    case LBM_STORE_F16_DEV: return tp_steps<LBM_STORE_F16_DEV>(h, n, macros_last);
    case LBM_STORE_BF16_DEV: return tp_steps<LBM_STORE_BF16_DEV>(h, n, macros_last);
    case LBM_STORE_F32_DEV: return tp_steps<LBM_STORE_F32_DEV>(h, n, macros_last);
    case LBM_STORE_F64: return tp_steps<LBM_STORE_F64>(h, n, macros_last);
    }
    return lbm_set_err(h, LBM_EINVAL, "unknown storage");
}
