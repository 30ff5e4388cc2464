// Builds the neighbour links (lbm_links.cuh) of a lattice from its dense map
// and packed coordinates: one warp per group of 32 nodes, two passes (tables
// and record counts, then the records of the groups that have some).
#include <cuda_runtime.h>

#include <algorithm>

#include "lbm_common.cuh"
#include "lbm_internal.h"
#include "lbm_links.cuh"

namespace {

struct LinkBuild {
    const int32_t* map;
    const uint32_t* coord;
    int32_t nx, ny, nz, n_fluid;
    int32_t bc[6];
    int32_t bc_form;
    int32_t every;        // records on replaced nodes too (two phases: the colours are pulled there)
    uint2* node;
    LbmLinkHead* head;
    LbmLinkRecs* recs;
    int32_t* rec;
    int32_t cap;          // records allocated
    int32_t* total;       // records needed
};

struct Row {
    int src[3];           // sources at x - 1, x, x + 1 (wrapped), -1 solid
    bool cross[3];        // the link crosses a periodic x face
    int rank;             // rank of the cell across, -1 when no link of the row needs it
};

// Links of the row (e_y, e_z) of a node; WIDE: the row's three cells, else the one across.
// A row across a periodic y or z face is a row like any other; of a whole node, whose
// pulls are replaced, it counts as crossed, so that it does not bend the group's line.
template <bool WIDE>
__device__ __forceinline__ Row link_row(const LinkBuild& B, int ey, int ez, int i, int j, int k, bool whole) {
    const int y = j - ey, z = k - ez;
    const int yw = y < 0 ? B.ny - 1 : (y >= B.ny ? 0 : y), zw = z < 0 ? B.nz - 1 : (z >= B.nz ? 0 : z);
    const int64_t row = (int64_t)B.nx * (yw + (int64_t)B.ny * zw);
    Row o;
    o.rank = -1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        o.src[d] = -1;
        o.cross[d] = false;
        if (!WIDE && d != 1) continue;
        const int x = i + d - 1;
        const int xw = x < 0 ? B.nx - 1 : (x >= B.nx ? 0 : x);
        o.cross[d] = x != xw || (whole && (y != yw || z != zw));
        o.src[d] = __ldg(B.map + row + xw);
    }
    if (o.src[1] >= 0 && !o.cross[1]) o.rank = o.src[1];
    else if (o.src[0] >= 0 && !o.cross[0]) o.rank = o.src[0] + 1;
    else if (o.src[2] >= 0 && !o.cross[2]) o.rank = o.src[2];
    return o;
}

template <bool FILL>
__global__ void __launch_bounds__(128) link_build_kernel(const LinkBuild B, int ngroup) {
    const int group = (blockIdx.x * 128 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (group >= ngroup) return;
    if constexpr (FILL)
        if (B.recs[group].lanes == 0) return;
    const int n = group * LBM_LINK_GROUP + lane;
    const bool live = n < B.n_fluid;
    const uint32_t pc = live ? B.coord[n] : 0u;
    const int i = lbm_pi(pc), j = lbm_pj(pc), k = lbm_pk(pc);
    uint32_t bits = live ? 0u : 0x7fffeu;   // padding: every direction from the own slots
    bool whole = false;                     // a face condition replaces all that the node pulls
    Row own{};
    if (live) {
        const bool at[6] = {i == 0, i == B.nx - 1, j == 0, j == B.ny - 1, k == 0, k == B.nz - 1};
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            if (!at[f] || B.bc[f] == LBM_BC_PERIODIC) continue;
            bits |= LBM_LINK_FACE;
            if (B.bc[f] == LBM_BC_PRESSURE) bits |= LBM_LINK_PRESSURE;
            // (the in-place velocity form reads what was pulled)
            whole |= !B.every && (B.bc[f] == LBM_BC_PRESSURE || B.bc_form == 0);
        }
        if (at[0] || at[1] || at[2] || at[3] || at[4] || at[5]) bits |= LBM_LINK_EDGE;
        own = link_row<true>(B, 0, 0, i, j, k, whole);
#pragma unroll
        for (int d = 0; d < 3; d += 2) {
            if (own.src[d] < 0 || own.cross[d]) bits |= d ? 4u : 2u;
            if (own.src[d] >= 0 && own.cross[d] && !whole) bits |= LBM_LINK_EXC;
        }
    }
    int start[8];
    uint32_t w0 = __any_sync(0xffffffffu, live && (i == 0 || i == B.nx - 1)) ? LBM_LINK_XFACE : 0u, w1 = 0, far = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        int rank = -1;
        if (live) {
            const Row o = r < 4 ? link_row<true>(B, lbm_link_ey(r), lbm_link_ez(r), i, j, k, whole)
                                : link_row<false>(B, lbm_link_ey(r), lbm_link_ez(r), i, j, k, whole);
            rank = o.rank;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (r >= 4 && d != 1) continue;
                const int s = lbm_link_dir(r, 1 - d);   // source x + d - 1 belongs to e_x = 1 - d
                if (o.src[d] < 0 || o.cross[d]) bits |= 1u << s;
                if (o.src[d] >= 0 && o.cross[d] && !whole) bits |= LBM_LINK_EXC;
            }
        }
        start[r] = __reduce_min_sync(0xffffffffu, rank >= 0 ? rank - lane : 0x7fffffff);
        if (start[r] == 0x7fffffff) start[r] = 0;
        uint32_t q = rank >= 0 ? (uint32_t)(rank - lane - start[r]) : 0u;
        if (q > 31u) {
            q = 0;
            far |= 1u << r;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if (r < 4 || d == 1) bits |= 1u << lbm_link_dir(r, 1 - d);
            if (!whole) bits |= LBM_LINK_EXC;
        }
        if (r < 6) w0 |= q << (5 * r);
        else w1 |= q << (22 + 5 * (r - 6));
    }
    const uint32_t exc = __ballot_sync(0xffffffffu, bits & LBM_LINK_EXC);
    if constexpr (!FILL) {
        int v = start[0];
#pragma unroll
        for (int r = 1; r < 8; ++r)
            if (lane == r) v = start[r];
        if (lane < 8) B.head[group].start[lane] = v;
        if (lane == 0) B.recs[group] = {exc ? atomicAdd(B.total, __popc(exc)) : 0, exc};
        B.node[n] = make_uint2(w0, w1 | bits);
    } else if (bits & LBM_LINK_EXC) {
        const int slot = B.recs[group].first + __popc(exc & ((1u << lane) - 1u));
        if (slot >= B.cap) return;               // the host allocates more and builds again
        int32_t* out = B.rec + (int64_t)LBM_LINK_REC * slot;
        out[0] = out[19] = -1;
        out[1] = own.cross[0] ? own.src[0] : -1;
        out[2] = own.cross[2] ? own.src[2] : -1;
#pragma unroll 1
        for (int r = 0; r < 8; ++r) {
            const Row o = link_row<true>(B, lbm_link_ey(r), lbm_link_ez(r), i, j, k, whole);
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if (r < 4 || d == 1) out[lbm_link_dir(r, 1 - d)] = o.cross[d] || (far >> r & 1u) ? o.src[d] : -1;
        }
    }
}

}  // namespace

// Links of `count` lattices whose maps and coordinates lie in h->d_map and
// h->d_coord (node numbers local to each lattice); one allocation
// (h->d_links).  Records: room for every node of the periodic x faces and for the
// groups where a row starts anew across a y or z face; geometries that need more
// (rows far from a line) get a second one.
int links_build(LbmHandle* h, const LbmLinkLattice* lat, int count) {
    const LbmParams& p = h->p;
    const int64_t ngroup = h->np / LBM_LINK_GROUP;
    int64_t cap = 32;
    for (int q = 0; q < count; ++q) {
        const LbmLinkLattice& l = lat[q];
        const int64_t area[3] = {(int64_t)l.ny * l.nz, LBM_LINK_GROUP * (int64_t)l.nz, LBM_LINK_GROUP};
        int64_t seam = 0;
        for (int f = 0; f < 6; ++f)
            if (p.two_phase || p.bc[f] == LBM_BC_PERIODIC || (p.bc[f] == LBM_BC_VELOCITY && p.bc_form != 0)) seam += area[f / 2];
        cap += std::min<int64_t>(seam, l.n_fluid) + l.n_fluid / 512;
    }
    size_t bytes = 0;
    auto drop = [&](int code) {
        cudaFree(h->d_links);
        h->d_links = nullptr;
        h->links = LbmLinks{};
        h->device_bytes -= (int64_t)bytes;
        return code;
    };
    for (;;) {
        const size_t node = sizeof(uint2) * h->np, head = sizeof(LbmLinkHead) * ngroup;
        const size_t recs = (sizeof(LbmLinkRecs) * (ngroup + 1) + 15) / 16 * 16;   // + the count
        bytes = node + head + recs + sizeof(int32_t) * LBM_LINK_REC * cap;
        int rc = lbm_cuda_check(h, cudaMalloc(&h->d_links, bytes), "neighbour links");
        if (rc) {
            h->d_links = nullptr;
            return rc;
        }
        h->device_bytes += (int64_t)bytes;
        char* at = (char*)h->d_links;
        const LbmLinks L{(uint2*)at, (LbmLinkHead*)(at + node), (LbmLinkRecs*)(at + node + head), (int32_t*)(at + node + head + recs)};
        h->links = L;
        int32_t* d_total = (int32_t*)(L.recs + ngroup);
        rc = lbm_cuda_check(h, cudaMemsetAsync(d_total, 0, sizeof(int32_t), h->stream), "link records");
        if (rc) return drop(rc);
        for (int pass = 0; pass < 2; ++pass)
            for (int q = 0; q < count; ++q) {
                const LbmLinkLattice& l = lat[q];
                LinkBuild B{};
                B.map = h->d_map + l.map_off;
                B.coord = h->d_coord + l.node_begin;
                B.nx = l.nx; B.ny = l.ny; B.nz = l.nz;
                B.n_fluid = l.n_fluid;
                for (int f = 0; f < 6; ++f) B.bc[f] = p.bc[f];
                B.bc_form = p.bc_form;
                B.every = p.two_phase;
                B.node = (uint2*)L.node + l.node_begin;
                B.head = (LbmLinkHead*)L.head + l.node_begin / LBM_LINK_GROUP;
                B.recs = (LbmLinkRecs*)L.recs + l.node_begin / LBM_LINK_GROUP;
                B.rec = (int32_t*)L.rec;
                B.cap = (int32_t)cap;
                B.total = d_total;
                // a lone lattice fills the padding of its arrays too (at most 64 nodes)
                const int groups = count == 1 ? (int)ngroup : (l.n_fluid + LBM_LINK_GROUP - 1) / LBM_LINK_GROUP;
                if (!groups) continue;
                if (pass == 0) link_build_kernel<false><<<(groups + 3) / 4, 128, 0, h->stream>>>(B, groups);
                else link_build_kernel<true><<<(groups + 3) / 4, 128, 0, h->stream>>>(B, groups);
            }
        rc = lbm_cuda_check(h, cudaGetLastError(), "link_build_kernel launch");
        int32_t total = 0;
        if (!rc) rc = lbm_cuda_check(h, cudaMemcpyAsync(&total, d_total, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream), "link records");
        if (!rc) rc = lbm_cuda_check(h, cudaStreamSynchronize(h->stream), "neighbour links");
        if (rc) return drop(rc);
        if (total <= cap) return LBM_OK;
        drop(LBM_OK);
        cap = total;
    }
}
