// Pull gather through the neighbour links (lbm_links.cuh), shared by the step
// kernels that use them.
#pragma once
#include "lbm_common.cuh"
#include "lbm_internal.h"
#include "lbm_links.cuh"

namespace lbmk {

// Wait for the previous step (programmatic dependent launch), and hand back the
// pointer to what it wrote.  The populations must not be read through a const
// __restrict__ pointer here: such loads count as invariant for the kernel's whole
// life and may be moved above the wait.
template <typename T>
__device__ __forceinline__ const T* wait_previous(const T* p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("" : "+l"(p)::"memory");
    return p;
}

// The same for a second pointer, after the wait.
template <typename T>
__device__ __forceinline__ const T* launder(const T* p) {
    asm volatile("" : "+l"(p)::"memory");
    return p;
}

// A node's links: loaded before the wait (they never change between steps).
struct NodeLinks {
    int4 a, b;          // the group's row starts
    uint32_t w, bits;
    int lane;           // place in the group
    int slot;           // the node's record, for nodes that have one (LBM_LINK_EXC)
    __device__ __forceinline__ void load(const LbmLinks& L, int n) {
        const int4* head = reinterpret_cast<const int4*>(L.head + n / LBM_LINK_GROUP);
        a = __ldg(head);
        b = __ldg(head + 1);
        const uint2 x = __ldg(L.node + n);
        w = x.x;
        bits = x.y;
        lane = n & (LBM_LINK_GROUP - 1);
        slot = bits & LBM_LINK_EXC ? find(L, n) : 0;
    }
    // Found without a vote, since which lanes are together at a vote is not fixed;
    // with the links, since after the gather its latency adds to a step (24 x 192 x
    // 192 all fluid, f32dev: 30.2 us, 27.7 so).
    __device__ __forceinline__ int find(const LbmLinks& L, int n) const {
        const int2 r = __ldg(reinterpret_cast<const int2*>(L.recs + n / LBM_LINK_GROUP));
        return r.x + __popc((uint32_t)r.y & ((1u << lane) - 1u));
    }
    // Node across in row r.
    template <int RW>
    __device__ __forceinline__ int rank() const {
        const int4& h = RW < 4 ? a : b;
        const int start = (RW & 3) == 0 ? h.x : (RW & 3) == 1 ? h.y : (RW & 3) == 2 ? h.z : h.w;
        const uint32_t q = RW < 6 ? w >> (5 * RW) & 31u : bits >> (22 + 5 * (RW - 6)) & 31u;
        return start + lane + (int)q;
    }
    // Pull source of direction S of node n (where its bit is clear).
    template <int S>
    __device__ __forceinline__ int source(int n) const {
        constexpr int ex = lbm_ex(S), ey = lbm_ey(S), ez = lbm_ez(S);
        if constexpr (ey == 0 && ez == 0) {
            return n - ex;
        } else {
            constexpr int rw = lbm_link_row(ey, ez);
            if constexpr (ex > 0) return rank<rw>() - 1;
            // x + 1 ranks after x only where x itself is fluid
            if constexpr (ex < 0) return rank<rw>() + (int)(~bits >> lbm_link_dir(rw, 0) & 1u);
            return rank<rw>();
        }
    }
    __device__ __forceinline__ const int32_t* record(const LbmLinks& L) const { return record(L, slot); }
    static __device__ __forceinline__ const int32_t* record(const LbmLinks& L, int slot) {
        return L.rec + (int64_t)LBM_LINK_REC * slot;
    }
    // Whether to take the code that looks for records: it serves every node, the
    // code without only those that have none.
    __device__ __forceinline__ bool any_record() const { return __any_sync(__activemask(), bits & LBM_LINK_EXC); }
};

// Reference density of the 16-bit codecs at a node and its sources at x - 1 and
// x + 1: stepped from the node's own value in a group without an x face, from
// the wrapped x in the others (the rounding of gather_node).
template <typename R>
struct LinkRef {
    R at = (R)0, xm = (R)0, xp = (R)0;
    LinkRef() = default;
    __device__ __forceinline__ LinkRef(const LbmRef<R>& ref, int i, int nx, const NodeLinks& K) {
        at = lbm_ref_at(ref, i);
        xm = at - ref.b;
        xp = at + ref.b;
        if (K.w & LBM_LINK_XFACE) {
            xm = lbm_fma<R>(ref.b, (R)(i == 0 ? nx - 1 : i - 1), ref.a);
            xp = lbm_fma<R>(ref.b, (R)(i == nx - 1 ? 0 : i + 1), ref.a);
        }
    }
    __device__ __forceinline__ void scale(R k) {
        at = at * k;
        xm = xm * k;
        xp = xp * k;
    }
    template <int S>
    __device__ __forceinline__ R of() const {
        return lbm_ex(S) > 0 ? xm : (lbm_ex(S) < 0 ? xp : at);
    }
};

// All of a node's pulled populations.  Direction s and its opposite are
// neighbours in the slot order, so the own opposite slot is the own slot s moved
// by one: both candidates of the load share the immediate offset of slot s.
// RAW: in the codec's own scale (Codec::SCALE), rx scaled alike.
template <int STORE, bool REF, bool RAW = false>
struct LinkGather {
    using Cd = Codec<STORE>;
    using T = typename Cd::T;
    using R = typename Cd::R;
    template <int S>
    static __device__ __forceinline__ R get(T x) {
        if constexpr (RAW) return Cd::template raw<S>(x);
        else return Cd::template dec<S>(x);
    }
    // The source as decoded; debug builds take the node itself for one outside the
    // nodes and record the failure (3).
    static __device__ __forceinline__ int checked(int src, int n) {
#ifdef LBM_DEBUG
        if (g_lbm_debug_nlimit > 0 && (unsigned)src >= (unsigned)g_lbm_debug_nlimit) {
            lbm_debug_fail(3);
            return n;
        }
#endif
        (void)n;
        return src;
    }
    template <int S>
    static __device__ __forceinline__ void one(R* F, const T* fin, int own, const NodeLinks& K, int n, const LinkRef<R>& rx) {
        const bool bounce = K.bits >> S & 1u;
        const int a = bounce ? own + 32 * (lbm_lr(S) - S) : lbm_eoff32(checked(K.template source<S>(n), n));
        F[S] = get<S>(fin[a + 32 * S]);
        if constexpr (REF) F[S] = lbm_fma<R>((R)lbm_w(S), bounce ? rx.at : rx.template of<S>(), F[S]);
    }
    // Explicit sources of the links that the node word cannot express.
    static __device__ __forceinline__ void recorded(R* F, const T* fin, const LbmLinks& L, const NodeLinks& K, int n,
                                                    const LinkRef<R>& rx) {
        if (!(K.bits & LBM_LINK_EXC)) return;
        // (with a reference density there is no register for the slot: 256^3 pack BF16
        // 146.2 us, 8 bytes spilled, against 141.5)
        const int4* rec = reinterpret_cast<const int4*>(K.record(L, REF ? K.find(L, n) : K.slot));
        int4 to;
#define LBM_X(S, SRC)                                                                         \
    if (SRC >= 0) {                                                                           \
        F[S] = get<S>(fin[lbm_eoff32(checked(SRC, n)) + 32 * S]);                             \
        if constexpr (REF) F[S] = lbm_fma<R>((R)lbm_w(S), rx.template of<S>(), F[S]);         \
    }
        to = __ldg(rec);
        LBM_X(1, to.y) LBM_X(2, to.z) LBM_X(3, to.w)
        to = __ldg(rec + 1);
        LBM_X(4, to.x) LBM_X(5, to.y) LBM_X(6, to.z) LBM_X(7, to.w)
        to = __ldg(rec + 2);
        LBM_X(8, to.x) LBM_X(9, to.y) LBM_X(10, to.z) LBM_X(11, to.w)
        to = __ldg(rec + 3);
        LBM_X(12, to.x) LBM_X(13, to.y) LBM_X(14, to.z) LBM_X(15, to.w)
        to = __ldg(rec + 4);
        LBM_X(16, to.x) LBM_X(17, to.y) LBM_X(18, to.z)
#undef LBM_X
    }
    static __device__ __forceinline__ void all(R* F, const T* fin, const LbmLinks& L, const NodeLinks& K, int n,
                                               const LinkRef<R>& rx) {
        const int own = lbm_eoff32(n);
        F[0] = get<0>(fin[own]);
        if constexpr (REF) F[0] = lbm_fma<R>((R)lbm_w(0), rx.at, F[0]);
#define LBM_G(S) one<S>(F, fin, own, K, n, rx);
        LBM_ALL_DIRS(LBM_G)
#undef LBM_G
        recorded(F, fin, L, K, n, rx);
    }
};

}  // namespace lbmk
