// Neighbour links of the compacted node list, built once per geometry
// (lbm_links.cu) and read by the step kernels (lbm_linkgather.cuh).
//
// The 18 pull sources of a node lie in 9 lattice rows (one per (e_y, e_z)).
// Nodes are numbered in cell order, so the fluid cells of a row are consecutive
// and one number per row, the rank of the cell straight across, gives all three
// sources x - 1, x, x + 1 of that row: rank - 1, rank, rank + (x is fluid).
// The own row needs none.  Along 32 consecutive nodes the rank of each of the 8
// other rows keeps close to a straight line: LbmLinkHead holds its start, a node
// word the 5-bit distance of its rank from start + lane and one bit per direction
// "take the own opposite slot" (solid source: halfway bounce-back).  That is 9
// bytes a node (8 + 32 per 32 nodes; LbmLinkRecs is read by nodes with a record), read in order, in the place of 18 lookups
// in the dense map (4 bytes a cell in three z planes, behind a load of the
// coordinates).  On sphere packs of porosity 0.25 to 0.5 the 5 bits fall short
// in 0.1% to 0.3% of the groups of 32 nodes (8 bits cost 3.5 bytes a node more).
//
// A link that this cannot express, i.e. one that crosses a periodic x face or is
// more than 31 from the row's line (as where 32 nodes lie on both sides of a periodic
// y or z face's first row), has its bit set too, the node's LBM_LINK_EXC
// bit is set, and an explicit record of 20 int32 holds the source of each such
// direction (-1 in the others).  Records of 32 nodes are consecutive in node
// order; LbmLinkRecs has the first one and the lanes that have one, so that a node
// finds its own without asking the other lanes.  Single-phase nodes whose populations a face condition
// replaces whole need none for what they pull.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define LBM_LINK_GROUP 32
#define LBM_LINK_REC 20
// LbmLinkNode.y: bit 0 as here, bits 1..18 the directions, 22..31 rows 6 and 7;
// .x: rows 0..5 at 5 bits each, bit 30 as here.
#define LBM_LINK_EXC 1u              // the node has a record
#define LBM_LINK_FACE (1u << 19)     // on a face with a boundary condition
#define LBM_LINK_PRESSURE (1u << 20) // on a fixed-pressure face
#define LBM_LINK_EDGE (1u << 21)     // on a face of the lattice
#define LBM_LINK_XFACE (1u << 30)    // (.x) some node of the group is on an x face

struct __align__(16) LbmLinkHead {
    int32_t start[8];  // rows ordered as lbm_link_ey / lbm_link_ez
};

struct __align__(8) LbmLinkRecs {
    int32_t first;     // first record of the group
    uint32_t lanes;    // its nodes that have one
};

struct LbmLinks {
    const uint2* node;            // [np]
    const LbmLinkHead* head;      // [np / 32]
    const LbmLinkRecs* recs;      // [np / 32]
    const int32_t* rec;           // LBM_LINK_REC per record
};

// A lattice among those whose links are built together.
struct LbmLinkLattice {
    int32_t nx, ny, nz, n_fluid;
    int64_t map_off;      // first cell of its map
    int64_t node_begin;   // first node (a multiple of 32)
};

// (e_y, e_z) of row r: rows 0..3 hold three directions each, 4..7 one.
__host__ __device__ constexpr int lbm_link_ey(int r) {
    return (r == 0 || r == 4 || r == 6) ? 1 : (r == 1 || r == 5 || r == 7) ? -1 : 0;
}
__host__ __device__ constexpr int lbm_link_ez(int r) {
    return (r == 2 || r == 4 || r == 7) ? 1 : (r == 3 || r == 5 || r == 6) ? -1 : 0;
}
__host__ __device__ constexpr int lbm_link_row(int ey, int ez) {
    for (int r = 0; r < 8; ++r)
        if (lbm_link_ey(r) == ey && lbm_link_ez(r) == ez) return r;
    return -1;
}
// Direction of row r with e_x = ex (rows 4..7: ex = 0 only).
__host__ __device__ constexpr int lbm_link_dir(int r, int ex) {
    return r == 0 ? (ex == 0 ? 3 : ex > 0 ? 7 : 10)
         : r == 1 ? (ex == 0 ? 4 : ex > 0 ? 9 : 8)
         : r == 2 ? (ex == 0 ? 5 : ex > 0 ? 11 : 14)
         : r == 3 ? (ex == 0 ? 6 : ex > 0 ? 13 : 12)
                  : 11 + r;
}
