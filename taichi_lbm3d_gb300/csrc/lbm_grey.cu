// Grey-scale (partial bounce-back) single-phase step over the compacted
// fluid-node list.  GS = Grey_Scale/lbm_solver_3d_Macro_Sukop.py (taichi_LBM3D tree).
//
// The reference's sweeps per step (GS:330-336) are colission (GS:203-218),
// streaming0 (GS:234-240), streaming1 (GS:243-252), Boundary_condition on the
// x faces (GS:263-293) and streaming3 (GS:296-312).  In pull form, with the
// post-collision populations f as the state between launches, a fluid node x
// receives for each direction s from y = x - e_s (periodic wrap):
//   y fluid:  F[s] = f(y)[s] + ns(y) (f(x)[LR s] - f(y)[s])
//             (streaming0 at y mixes with the opposite population of the
//             cell the population moves to, which is x itself)
//   y solid:  F[s] keeps its previous value: streaming1 only pushes from
//             fluid cells, so that slot still holds init's feq(s, 1, 0) = w_s,
//             or, on a fixed-velocity x face, what the face rule wrote last step
// then the x faces, rho/v (+ F/2 rho), and the single-phase MRT collision with
// the script's Guo term (same arithmetic as the single-phase step).
//
// Extra per-node data: ns (grey value) [np].  Fixed-velocity x faces keep
// their post-face F in a side array [2][ny*nz][19] (the in-place face rule
// reads the stale slots), initialised to w_s by lbm_init.
#include <cuda_runtime.h>

#include <algorithm>

#include "lbm_common.cuh"
#include "lbm_internal.h"
#include "lbm_kernels.cuh"
#include "lbm_linkgather.cuh"

namespace {
using namespace lbmk;

// Value of a slot that no fluid cell pushes into: feq(s, 1, 0) = w_s (GS:120-127);
// 0 in deviation form.
template <int S, typename R, bool DEV>
__device__ __forceinline__ R grey_rest() {
    return DEV ? (R)0 : (R)lbm_w(S);
}

// F of a node through the neighbour links (solid upstream: the rest value).
// Fo: the node's own post-collision populations, the partners of the mixing.
template <int STORE, bool EXC>
__device__ __forceinline__ void grey_gather(typename Codec<STORE>::R* F, const typename Codec<STORE>::R* Fo,
                                            const typename Codec<STORE>::T* fin,
                                            const typename Codec<STORE>::R* __restrict__ ns, const NodeLinks& K,
                                            const int32_t* rec, int n, const LinkRef<typename Codec<STORE>::R>& rx) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    F[0] = Fo[0];   // streaming0 mixes it with itself
#define LBM_G(S)                                                                                   \
    {                                                                                              \
        bool solid = K.bits >> S & 1u;                                                             \
        int src = solid ? n : K.template source<S>(n);   /* loads from n are discarded */          \
        if constexpr (EXC) {                                                                       \
            const int to = solid && (K.bits & LBM_LINK_EXC) ? __ldg(rec + S) : -1;                 \
            src = to >= 0 ? to : src;                                                              \
            solid = solid && to < 0;                                                               \
        }                                                                                          \
        R a = Cd::template dec<S>(fin[lbm_eoff32(src) + 32 * S]);                                  \
        if constexpr (Cd::RHOREF) a = lbm_fma<R>((R)lbm_w(S), rx.template of<S>(), a);             \
        const R mixed = a + __ldg(ns + src) * (Fo[lbm_lr(S)] - a);                                 \
        F[S] = solid ? grey_rest<S, R, Cd::DEV>() : mixed;                                         \
    }
    LBM_ALL_DIRS(LBM_G)
#undef LBM_G
}

// Fixed-velocity x face: slots whose upstream cell is solid hold what the face
// rule wrote at the previous step (side array), not w_s.
template <typename R>
__device__ __forceinline__ void grey_face_restore(R* F, int i, int j, int k, const SpConsts<R>& C,
                                                  const int32_t* __restrict__ map, const R* st) {
    const int xm = i == 0 ? C.nx - 1 : i - 1, xp = i == C.nx - 1 ? 0 : i + 1;
    const int ym = j == 0 ? C.ny - 1 : j - 1, yp = j == C.ny - 1 ? 0 : j + 1;
    const int zm = k == 0 ? C.nz - 1 : k - 1, zp = k == C.nz - 1 ? 0 : k + 1;
    const Rows rows = make_rows(C.nx, C.ny, i, j, k, ym, yp, zm, zp);
#define LBM_R(S) \
    if (pull_source<S, true>(map, rows, i, xm, xp) < 0) F[S] = st[S];
    LBM_ALL_DIRS(LBM_R)
#undef LBM_R
}

// Sources from the neighbour links, every load unconditional (a solid source reads
// the node itself and discards it: loads behind a branch ran one after another, 22.2k
// FP32 and 22.7k FP16), 8 CTAs of 128 per SM (64 registers; 24.5k FP32 at 9,
// 28.7k FP32 deviation form at 7).  192^3 grey field, MLUPS against the map
// kernel with IEEE divisions and the dense Guo term: FP32 forced along x 25.1k /
// 18.3k, FP32 with pressure faces 26.4k / 23.5k, FP32 deviation form 30.3k / 26.9k,
// FP16 29.9k / 25.7k.  Bound by issue (74% of the slots, 1118 instructions a node) and
// the latency of 55 loads a node.
constexpr int GREY_THREADS = 128;

template <int STORE, int FORCE, bool MACROS>
__global__ void __launch_bounds__(GREY_THREADS, STORE == LBM_STORE_F64 ? 2 : 8) grey_step_kernel(
    const __grid_constant__ SpConsts<typename Codec<STORE>::R> C, const typename Codec<STORE>::T* f_prev,
    typename Codec<STORE>::T* __restrict__ fout, const __grid_constant__ LbmLinks L, const int32_t* __restrict__ map,
    const uint32_t* __restrict__ coord, const typename Codec<STORE>::R* __restrict__ ns,
    typename Codec<STORE>::R* face_stale, typename Codec<STORE>::R* vprev, typename Codec<STORE>::R* __restrict__ rho_out,
    typename Codec<STORE>::R* __restrict__ v_out) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    // programmatic dependent launch, as in the single-phase step: the next
    // step's CTAs may start once all of these run; they wait below before
    // reading populations or the face side array
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= C.n_fluid) return;
    NodeLinks K;
    K.load(L, n);
    const bool exc = K.any_record();
    const int32_t* rec = K.record(L);
    const bool on = K.bits & LBM_LINK_FACE;
    int i = 0, j = 0, k = 0;
    if (Cd::RHOREF || on) {
        const uint32_t pc = __ldg(coord + n);
        i = lbm_pi(pc);
        j = lbm_pj(pc);
        k = lbm_pk(pc);
    }
    LinkRef<R> rx;
    if constexpr (Cd::RHOREF) rx = LinkRef<R>(sp_ref(C), i, C.nx, K);
    const int64_t np = C.np;
    const auto* fin = wait_previous(f_prev);

    R F[19];
    {
        R Fo[19];
        const typename Cd::T* own = fin + lbm_eoff32(n);
#define LBM_OWN(S)                                                                        \
    Fo[S] = Cd::template dec<S>(own[32 * S]);                                             \
    if constexpr (Cd::RHOREF) Fo[S] = lbm_fma<R>((R)lbm_w(S), rx.at, Fo[S]);
        LBM_OWN(0) LBM_ALL_DIRS(LBM_OWN)
#undef LBM_OWN
        if (exc) grey_gather<STORE, true>(F, Fo, fin, ns, K, rec, n, rx);
        else grey_gather<STORE, false>(F, Fo, fin, ns, K, rec, n, rx);
    }

    if (on) {
        // x faces only (GS:263-293); velocity faces read and keep their stale slots
        R* st = nullptr;
        if (face_stale && i == 0 && C.bc[0] == LBM_BC_VELOCITY) st = face_stale + (int64_t)19 * (j + C.ny * k);
        if (face_stale && i == C.nx - 1 && C.bc[1] == LBM_BC_VELOCITY)
            st = face_stale + (int64_t)19 * ((int64_t)C.ny * C.nz + j + C.ny * k);
        if (st) grey_face_restore<R>(F, i, j, k, C, map, st);
        apply_faces<R, Cd::DEV>(F, i, j, k, n, C, map, vprev);
        if (st) {
#pragma unroll
            for (int s = 0; s < 19; ++s) st[s] = F[s];
        }
    }

    // streaming3 (GS:296-312)
    R r = F[0];
#pragma unroll
    for (int s = 1; s < 19; ++s) r = r + F[s];
    const R rho = Cd::DEV ? (R)1 + r : r;
    R vx = vsum<0>(F), vy = vsum<1>(F), vz = vsum<2>(F);
    velocity<R, FORCE>(vx, vy, vz, rho, C.fhalf);
    if (K.bits & LBM_LINK_PRESSURE) {
        vprev[n] = vx;
        vprev[np + n] = vy;
        vprev[2 * np + n] = vz;
    }
    if constexpr (MACROS) {
        rho_out[n] = rho;
        v_out[n] = vx;
        v_out[np + n] = vy;
        v_out[2 * np + n] = vz;
    }
    // colission (GS:203-218): the single-phase MRT collision with the script's Guo term
    collide_sp<R, FORCE, Cd::DEV>(F, r, vx, vy, vz, C);
    store_node<STORE>(F, fout, n, rx.at, C.seed);
}

template <int STORE, int FORCE, bool MACROS>
int launch_grey(LbmHandle* h, const SpConsts<typename Codec<STORE>::R>& C) {
    using T = typename Codec<STORE>::T;
    using R = typename Codec<STORE>::R;
    const T* fin = (const T*)h->d_f[h->cur];
    T* fout = (T*)h->d_f[h->cur ^ 1];
    cudaLaunchConfig_t cfg = {};
    const int block = std::min<int>(h->block, GREY_THREADS);
    cfg.gridDim = dim3((unsigned)((h->n_fluid + block - 1) / block));
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, grey_step_kernel<STORE, FORCE, MACROS>, C, fin, fout, h->links,
                                             (const int32_t*)h->d_map, (const uint32_t*)h->d_coord,
                                             (const R*)h->d_ns, (R*)h->d_gstale, (R*)h->d_vprev, (R*)h->d_rho,
                                             (R*)h->d_v);
    h->cur ^= 1;
    return lbm_cuda_check(h, e != cudaSuccess ? e : cudaGetLastError(), "grey_step_kernel launch");
}

template <int STORE, int FORCE>
int run_grey_t(LbmHandle* h, int32_t n, bool macros_last) {
    SpConsts<typename Codec<STORE>::R> C = sp_make_consts<typename Codec<STORE>::R>(h);
    for (int32_t it = 0; it < n; ++it) {
        C.seed = (uint32_t)(h->steps_done + it);
        const int rc = macros_last && it == n - 1 ? launch_grey<STORE, FORCE, true>(h, C) : launch_grey<STORE, FORCE, false>(h, C);
        if (rc) return rc;
    }
    return LBM_OK;
}

template <int STORE>
int run_grey(LbmHandle* h, int32_t n, bool macros_last) {
    if constexpr (!Codec<STORE>::DEV)
        if (force_kind(h) == FORCE_X) return run_grey_t<STORE, FORCE_X>(h, n, macros_last);
    return h->force ? run_grey_t<STORE, FORCE_ANY>(h, n, macros_last) : run_grey_t<STORE, FORCE_NONE>(h, n, macros_last);
}

}  // namespace

int grey_launch_steps(LbmHandle* h, int32_t n, bool macros_last) {
    switch (h->p.storage) {
    case LBM_STORE_F32: return run_grey<LBM_STORE_F32>(h, n, macros_last);
    case LBM_STORE_F16_DEV: return run_grey<LBM_STORE_F16_DEV>(h, n, macros_last);
    case LBM_STORE_BF16_DEV: return run_grey<LBM_STORE_BF16_DEV>(h, n, macros_last);
    case LBM_STORE_F32_DEV: return run_grey<LBM_STORE_F32_DEV>(h, n, macros_last);
    case LBM_STORE_F64: return run_grey<LBM_STORE_F64>(h, n, macros_last);
    }
    return lbm_set_err(h, LBM_EINVAL, "unknown storage");
}
