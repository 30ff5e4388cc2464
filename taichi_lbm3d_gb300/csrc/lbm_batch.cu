// K5: many independent porous subvolumes advanced together, one launch per time
// step, `check_every` steps captured into one CUDA graph.
//
// Layout: the compacted fluid nodes of all subvolumes are concatenated (each
// subvolume starts on a multiple of 32 so no population chunk straddles two);
// each subvolume has its own dense node map and neighbour links holding node
// indices local to the subvolume.  A CTA offsets the population and link arrays
// to its subvolume's first node once (64-bit), and the 32-bit offset
// arithmetic of the gather stays local, so the batch as a whole may exceed
// 2^31 population elements.  Work is cut into tiles (subvolume, local node
// range), one CTA each, one thread a node.  Converged subvolumes leave the tile list, which is
// rewritten in device memory and the graph captured again.  The node update is
// the single-phase step of K1 (all faces periodic, optional body force) in any
// storage mode.
//
// Convergence: the last step of each graph writes, per tile, the FP64 sum of
// v along x; the host sums tiles in order per subvolume (deterministic) and
// compares the Darcy velocity with the previous check.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "lbm_kernels.cuh"
#include "lbm_linkgather.cuh"

using BatchSub = LbmLinkLattice;

struct BatchTile {
    int32_t first32;        // first node of the subvolume / 32
    int32_t begin, end;     // local node range (begin a multiple of 32)
    int32_t sub;
};

// Per-subvolume views of the concatenated arrays (node indices become local).
template <typename T>
__device__ __forceinline__ T* sub_pop(T* f, int64_t node_begin) {
    return f + lbm_eoff(node_begin);
}
template <typename T>
__device__ __forceinline__ T* sub_node(T* a, int64_t node_begin) {
    return a ? a + node_begin : a;
}

struct LbmBatch {
    LbmHandle h;                        // shared params, stream, populations, coords, map
    std::vector<BatchSub> subs;
    std::vector<int32_t> tile_len;      // per subvolume
    std::vector<uint8_t> active;
    std::vector<BatchTile> tiles;       // current (active) tile list
    BatchSub* d_subs = nullptr;
    BatchTile* d_tiles = nullptr;
    uint32_t* d_seed = nullptr;         // first step of the launch group (16-bit rounding seed)
    double* d_partial = nullptr;        // per tile
    int64_t max_tiles = 0;
    int32_t block = 128;
    cudaGraphExec_t graph = nullptr;
    int32_t graph_steps = 0;
    std::vector<int64_t> steps;         // per subvolume
    uint32_t seed_step = 0;             // steps taken since init (16-bit rounding seed)
    bool initialized = false;
};

namespace {
using namespace lbmk;

// One CTA per tile, steps in programmatic dependent launch: tile and links are
// loaded while the step before drains.  Eight subvolumes of edges 48 to 160 (4.07 M
// fluid nodes, body force), MLUPS, against a persistent grid whose CTAs claimed
// 1024-node tiles from a counter and looked sources up in the dense maps: FP16
// 42.0k / 32.0k, FP32 deviation form 37.9k / 30.9k, FP32 31.0k / 20.2k.  Bound by
// issue (75% of the slots) and latency as the single-lattice kernel.  Tiles of 64 and 128 threads run
// alike, of 256 5% slower.
template <int STORE, int FORCE, bool CHECK>
__global__ void __launch_bounds__(256, STORE == LBM_STORE_F64 ? 1 : FORCE && !Codec<STORE>::DEV ? 4 : 5)
    batch_step_kernel(const __grid_constant__ SpConsts<typename Codec<STORE>::R> C, const BatchTile* __restrict__ tiles,
                      const typename Codec<STORE>::T* f_prev, typename Codec<STORE>::T* __restrict__ fout,
                      const __grid_constant__ LbmLinks links, const uint32_t* __restrict__ seed_base,
                      double* __restrict__ partial) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    constexpr bool RAW = Cd::SCALE != 1;
    constexpr int SC = RAW ? Cd::SCALE : 1;
    __shared__ double s_red[32];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int4 t4 = __ldg(reinterpret_cast<const int4*>(tiles + blockIdx.x));
    const int64_t first = (int64_t)t4.x * 32;
    const LbmLinks L{links.node + first, links.head + t4.x, links.recs + t4.x, links.rec};
    const int n = t4.y + threadIdx.x;
    const bool live = n < t4.z;
    NodeLinks K;
    K.load(L, live ? n : t4.y);
    // 16-bit codecs: all faces periodic, so the reference density is 0; the
    // rounding bits are those of a single lattice at the same step (step
    // index = the launch group's first step, set before the group, + k)
    const uint32_t seed = *seed_base + C.seed;
    const LinkRef<R> none{};
    const typename Cd::T* fin = sub_pop(wait_previous(f_prev), first);
    typename Cd::T* out = sub_pop(fout, first);
    double acc = 0.0;
    if (live) {
        R F[19];
        LinkGather<STORE, false, RAW>::all(F, fin, L, K, n, none);
        R r = F[0];
#pragma unroll
        for (int s = 1; s < 19; ++s) r = r + F[s];
        const R rho = Cd::DEV ? (R)SC + r : r;   // times SC, as the sums over F
        R vx = vsum<0>(F), vy = vsum<1>(F), vz = vsum<2>(F);
        const R fhalf[3] = {C.fhalf[0] * (R)SC, C.fhalf[1] * (R)SC, C.fhalf[2] * (R)SC};
        velocity<R, FORCE>(vx, vy, vz, rho, fhalf);
        if constexpr (CHECK) acc += (double)vx;
        collide_sp<R, FORCE, Cd::DEV, SC>(F, r, vx, vy, vz, C);
        if constexpr (RAW) store_node_raw<STORE>(F, out, n, (R)0, seed);
        else store_node<STORE>(F, out, n, (R)0, seed);
    }
    if constexpr (CHECK) {
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += s_red[w];
            partial[blockIdx.x] = s;
        }
    }
}

// rho [cell] and v [cell][3] of one subvolume from its current populations (the
// macroscopic step of the next update, without collision or store); solid 1 and 0.
template <int STORE, bool FORCE>
__global__ void batch_macros_kernel(const __grid_constant__ SpConsts<typename Codec<STORE>::R> C, BatchSub sd,
                                    const typename Codec<STORE>::T* __restrict__ fin, const int32_t* __restrict__ map,
                                    float* __restrict__ rho_out, float* __restrict__ v_out) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (int64_t)sd.nx * sd.ny * sd.nz) return;
    const int32_t* smap = map + sd.map_off;
    const int n = smap[c];
    float o[4] = {1.0f, 0.0f, 0.0f, 0.0f};
    if (n >= 0) {
        const int i = (int)(c % sd.nx), j = (int)(c / sd.nx % sd.ny), k = (int)(c / ((int64_t)sd.nx * sd.ny));
        R F[19];
        gather_node<STORE>(F, sub_pop(fin, sd.node_begin), smap, n, sd.nx, sd.ny, sd.nz, i, j, k);
        R r = F[0];
#pragma unroll
        for (int s = 1; s < 19; ++s) r = r + F[s];
        const R rho = Cd::DEV ? (R)1 + r : r;
        R vx = vsum<0>(F) / rho, vy = vsum<1>(F) / rho, vz = vsum<2>(F) / rho;
        if constexpr (FORCE) {
            vx = vx + C.fhalf[0] / rho;
            vy = vy + C.fhalf[1] / rho;
            vz = vz + C.fhalf[2] / rho;
        }
        o[0] = (float)rho;
        o[1] = (float)vx;
        o[2] = (float)vy;
        o[3] = (float)vz;
    }
    rho_out[c] = o[0];
#pragma unroll
    for (int d = 0; d < 3; ++d) v_out[3 * c + d] = o[1 + d];
}

template <int STORE, bool FORCE>
__global__ void batch_init_kernel(const __grid_constant__ SpConsts<typename Codec<STORE>::R> C,
                                  typename Codec<STORE>::T* __restrict__ fout, const BatchSub* __restrict__ subs,
                                  int n_sub) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    if (blockIdx.y >= (unsigned)n_sub) return;
    const BatchSub sd = subs[blockIdx.y];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= sd.n_fluid) return;
    R F[19];
    if constexpr (Cd::DEV) lbm_feq_dev_all<R>((R)0, (R)0, (R)0, (R)0, F);
    else lbm_feq_all<R>((R)1, (R)0, (R)0, (R)0, F);
    const R r = Cd::DEV ? (R)0 : (R)1;
    collide_sp<R, FORCE, Cd::DEV>(F, r, (R)0, (R)0, (R)0, C);
    store_node<STORE>(F, sub_pop(fout, sd.node_begin), n, (R)0, ~0u);   // as the single-lattice init
}

int batch_err(LbmBatch* b, int code, const std::string& m) { return lbm_set_err(&b->h, code, m); }

template <int STORE>
int launch_one(LbmBatch* b, int k, bool check, cudaStream_t s) {
    using Cd = Codec<STORE>;
    using T = typename Cd::T;
    using R = typename Cd::R;
    LbmHandle* h = &b->h;
    SpConsts<R> C = sp_make_consts<R>(h);
    C.seed = (uint32_t)k;   // step within the launch group; the group's first step is read on the device
    const int cur = k & 1;
    const T* fin = (const T*)h->d_f[cur];
    T* fout = (T*)h->d_f[cur ^ 1];
    if (b->tiles.empty()) return LBM_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)b->tiles.size());
    cfg.blockDim = dim3((unsigned)b->block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = k > 0 ? 1 : 0;   // the first step of a group waits for the seed in stream order
    cudaError_t e = cudaSuccess;
    auto args = [&](auto kern) {
        e = cudaLaunchKernelEx(&cfg, kern, C, (const BatchTile*)b->d_tiles, fin, fout, h->links,
                               (const uint32_t*)b->d_seed, b->d_partial);
    };
    constexpr int X = Cd::DEV ? FORCE_ANY : FORCE_X;   // (the deviation form has one kernel for every force)
    switch (force_kind(h)) {
    case FORCE_NONE:
        if (check) args(batch_step_kernel<STORE, FORCE_NONE, true>);
        else args(batch_step_kernel<STORE, FORCE_NONE, false>);
        break;
    case FORCE_X:
        if (check) args(batch_step_kernel<STORE, X, true>);
        else args(batch_step_kernel<STORE, X, false>);
        break;
    default:
        if (check) args(batch_step_kernel<STORE, FORCE_ANY, true>);
        else args(batch_step_kernel<STORE, FORCE_ANY, false>);
    }
    return lbm_cuda_check(h, e != cudaSuccess ? e : cudaGetLastError(), "batch_step_kernel launch");
}

int launch_dispatch(LbmBatch* b, int k, bool check, cudaStream_t s) {
    switch (b->h.p.storage) {
    case LBM_STORE_F32: return launch_one<LBM_STORE_F32>(b, k, check, s);
    case LBM_STORE_F16_DEV: return launch_one<LBM_STORE_F16_DEV>(b, k, check, s);
    case LBM_STORE_BF16_DEV: return launch_one<LBM_STORE_BF16_DEV>(b, k, check, s);
    case LBM_STORE_F32_DEV: return launch_one<LBM_STORE_F32_DEV>(b, k, check, s);
    case LBM_STORE_F64: return launch_one<LBM_STORE_F64>(b, k, check, s);
    }
    return batch_err(b, LBM_EINVAL, "unknown storage");
}

template <int STORE>
int init_t(LbmBatch* b) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    LbmHandle* h = &b->h;
    const SpConsts<R> C = sp_make_consts<R>(h);
    int maxn = 1;
    for (auto& s : b->subs) maxn = std::max(maxn, s.n_fluid);
    dim3 grid((maxn + 255) / 256, (unsigned)b->subs.size());
    auto k = h->force ? batch_init_kernel<STORE, true> : batch_init_kernel<STORE, false>;
    k<<<grid, 256, 0, h->stream>>>(C, (typename Cd::T*)h->d_f[0], b->d_subs, (int)b->subs.size());
    return lbm_cuda_check(h, cudaGetLastError(), "batch_init_kernel launch");
}

template <int STORE>
int macros_t(LbmBatch* b, int q, float* rho, float* v) {
    using Cd = Codec<STORE>;
    using R = typename Cd::R;
    LbmHandle* h = &b->h;
    const SpConsts<R> C = sp_make_consts<R>(h);
    const BatchSub sd = b->subs[q];
    const int grid = (int)(((int64_t)sd.nx * sd.ny * sd.nz + 127) / 128);
    auto k = h->force ? batch_macros_kernel<STORE, true> : batch_macros_kernel<STORE, false>;
    k<<<grid, 128, 0, h->stream>>>(C, sd, (const typename Cd::T*)h->d_f[0], h->d_map, rho, v);
    return lbm_cuda_check(h, cudaGetLastError(), "batch_macros_kernel launch");
}

void destroy_graph(LbmBatch* b) {
    if (b->graph) cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
    b->graph_steps = 0;
}

int rebuild_tiles(LbmBatch* b) {
    b->tiles.clear();
    for (size_t q = 0; q < b->subs.size(); ++q) {
        if (!b->active[q]) continue;
        const BatchSub& s = b->subs[q];
        const int len = std::min((std::max(32, b->tile_len[q]) + 31) / 32 * 32, b->block);   // whole link groups
        for (int a = 0; a < s.n_fluid; a += len)
            b->tiles.push_back({(int32_t)(s.node_begin / 32), a, std::min(s.n_fluid, a + len), (int32_t)q});
    }
    LbmHandle* h = &b->h;
    destroy_graph(b);   // its grids are the tile count
    if ((int64_t)b->tiles.size() > b->max_tiles) return batch_err(b, LBM_EINVAL, "tile list exceeds its allocation");
    const int32_t nt = (int32_t)b->tiles.size();
    int rc = 0;
    if (nt) rc = lbm_cuda_check(h, cudaMemcpyAsync(b->d_tiles, b->tiles.data(), sizeof(BatchTile) * nt, cudaMemcpyHostToDevice, h->stream), "copy tiles");
    if (!rc) rc = lbm_cuda_check(h, cudaStreamSynchronize(h->stream), "rebuild tiles");
    return rc;
}

// Capture `nsteps` steps (the last one writes the per-tile partials) into a graph.
int capture(LbmBatch* b, int32_t nsteps) {
    LbmHandle* h = &b->h;
    destroy_graph(b);
    cudaGraph_t g;
    int rc = lbm_cuda_check(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
    if (rc) return rc;
    for (int k = 0; k < nsteps && !rc; ++k) rc = launch_dispatch(b, k, k == nsteps - 1, h->stream);
    cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc) return rc;
    rc = lbm_cuda_check(h, e, "end capture");
    if (rc) return rc;
    rc = lbm_cuda_check(h, cudaGraphInstantiate(&b->graph, g, 0), "graph instantiate");
    cudaGraphDestroy(g);
    if (!rc) b->graph_steps = nsteps;
    return rc;
}

}  // namespace

extern "C" {

int lbm_batch_destroy(LbmBatch* b);

int lbm_batch_create(const LbmParams* params, int32_t n_sub, const int32_t* dims, const int8_t* solids,
                     LbmBatch** out) {
    if (!params || !dims || !solids || !out || n_sub < 1) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: bad argument");
    *out = nullptr;
    for (int f = 0; f < 6; ++f)
        if (params->bc[f] != 0) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: batched subvolumes are periodic on all faces");
    if (params->two_phase) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: single phase only");
    LbmParams p = *params;
    p.nx = p.ny = p.nz = 1;
    LbmHandle* tmp = nullptr;
    int rc = lbm_create(&p, &tmp);   // device checks, stream
    if (rc) return rc;
    LbmBatch* b = new LbmBatch();
    b->h = std::move(*tmp);
    tmp->stream = nullptr;
    lbm_destroy(tmp);
    LbmHandle* h = &b->h;
    // concatenate the subvolumes
    int64_t cells = 0, nodes = 0;
    std::vector<int32_t> map;
    std::vector<uint32_t> coord;
    for (int q = 0; q < n_sub; ++q) {
        const int nx = dims[3 * q], ny = dims[3 * q + 1], nz = dims[3 * q + 2];
        if (nx < 1 || ny < 1 || nz < 1 || nx > 2047 || ny > 2047 || nz > 1023) {
            lbm_batch_destroy(b);
            return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: bad subvolume size");
        }
        const int64_t nc = (int64_t)nx * ny * nz;
        BatchSub s{nx, ny, nz, 0, (int64_t)map.size(), nodes};
        const int8_t* sol = solids + cells;
        int64_t nf = 0;
        map.resize(map.size() + nc);
        for (int64_t c = 0; c < nc; ++c) {
            if (sol[c] > 0) { map[s.map_off + c] = -1; continue; }
            map[s.map_off + c] = (int32_t)nf;   // checked against the local limit below
            const int i = (int)(c % nx), j = (int)((c / nx) % ny), k = (int)(c / ((int64_t)nx * ny));
            coord.push_back(lbm_pack(i, j, k));
            ++nf;
        }
        if (nf >= ((int64_t)1 << 31) / 19) {
            lbm_batch_destroy(b);
            return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: subvolume has too many fluid nodes");
        }
        s.n_fluid = (int32_t)nf;
        const int64_t padded = (nf + 31) / 32 * 32;
        coord.resize(coord.size() + (padded - nf), 0);
        nodes += padded;
        cells += nc;
        b->subs.push_back(s);
    }
    if (nodes >= ((int64_t)1 << 31) - 64) { lbm_batch_destroy(b); return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_create: too many nodes"); }
    h->n_fluid = (int32_t)nodes;
    h->np = (nodes + 63) / 64 * 64;
    coord.resize(h->np, 0);
    h->ncell = cells;
    b->active.assign(n_sub, 1);
    b->tile_len.assign(n_sub, 128);
    b->steps.assign(n_sub, 0);
    b->max_tiles = 0;
    for (auto& s : b->subs) b->max_tiles += (s.n_fluid + 31) / 32;   // tiles of >= 32 nodes
    auto alloc = [&](void** ptr, size_t bytes) {
        if (rc) return;
        if (cudaMalloc(ptr, bytes ? bytes : 16) != cudaSuccess) rc = lbm_set_err(nullptr, LBM_ENOMEM, "lbm_batch_create: out of device memory");
        else h->device_bytes += (int64_t)bytes;
    };
    alloc((void**)&h->d_map, sizeof(int32_t) * map.size());
    alloc((void**)&h->d_coord, sizeof(uint32_t) * h->np);
    alloc(&h->d_f[0], h->elem * 19 * h->np);
    alloc(&h->d_f[1], h->elem * 19 * h->np);
    alloc((void**)&b->d_subs, sizeof(BatchSub) * n_sub);
    alloc((void**)&b->d_tiles, sizeof(BatchTile) * b->max_tiles);
    alloc((void**)&b->d_partial, sizeof(double) * b->max_tiles);
    alloc((void**)&b->d_seed, sizeof(uint32_t));
    if (!rc) rc = lbm_cuda_check(h, cudaMemcpy(h->d_map, map.data(), sizeof(int32_t) * map.size(), cudaMemcpyHostToDevice), "copy map");
    if (!rc) rc = lbm_cuda_check(h, cudaMemcpy(h->d_coord, coord.data(), sizeof(uint32_t) * h->np, cudaMemcpyHostToDevice), "copy coord");
    if (!rc) rc = lbm_cuda_check(h, cudaMemcpy(b->d_subs, b->subs.data(), sizeof(BatchSub) * n_sub, cudaMemcpyHostToDevice), "copy subs");
    if (!rc) rc = links_build(h, b->subs.data(), n_sub);
    if (rc) { lbm_batch_destroy(b); return rc; }
    h->have_geometry = true;
    *out = b;
    return LBM_OK;
}

int lbm_batch_destroy(LbmBatch* b) {
    if (!b) return LBM_OK;
    LbmHandle* h = &b->h;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    destroy_graph(b);
    cudaFree(b->d_subs);
    cudaFree(b->d_tiles);
    cudaFree(b->d_partial);
    cudaFree(b->d_seed);
    cudaFree(h->d_links);
    cudaFree(h->d_map);
    cudaFree(h->d_coord);
    cudaFree(h->d_f[0]);
    cudaFree(h->d_f[1]);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete b;
    return LBM_OK;
}

// Threads per CTA, and the nodes of a CTA's tile per subvolume: whole link groups of 32, at most its threads.
int lbm_batch_configure(LbmBatch* b, const int32_t* tile_len, int32_t block) {
    if (!b || !tile_len) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_configure: NULL argument");
    if (block < 64 || block > 256 || block % 32) return batch_err(b, LBM_EINVAL, "lbm_batch_configure: block must be 64..256, multiple of 32");
    for (size_t q = 0; q < b->subs.size(); ++q) {
        if (tile_len[q] < 32) return batch_err(b, LBM_EINVAL, "lbm_batch_configure: tile length < 32");
        b->tile_len[q] = tile_len[q];
    }
    b->block = block;
    if (!b->initialized) return LBM_OK;
    // the kernel has a thread for every node of a tile: tiles in use are cut again
    cudaSetDevice(b->h.device);
    return rebuild_tiles(b);
}

int lbm_batch_init(LbmBatch* b) {
    if (!b) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_init: NULL");
    LbmHandle* h = &b->h;
    cudaSetDevice(h->device);
    int rc = LBM_OK;
    std::fill(b->active.begin(), b->active.end(), (uint8_t)1);
    std::fill(b->steps.begin(), b->steps.end(), (int64_t)0);
    switch (h->p.storage) {
    case LBM_STORE_F32: rc = init_t<LBM_STORE_F32>(b); break;
    case LBM_STORE_F16_DEV: rc = init_t<LBM_STORE_F16_DEV>(b); break;
    case LBM_STORE_BF16_DEV: rc = init_t<LBM_STORE_BF16_DEV>(b); break;
    case LBM_STORE_F32_DEV: rc = init_t<LBM_STORE_F32_DEV>(b); break;
    case LBM_STORE_F64: rc = init_t<LBM_STORE_F64>(b); break;
    default: rc = batch_err(b, LBM_EINVAL, "unknown storage");
    }
    if (!rc) rc = rebuild_tiles(b);
    b->seed_step = 0;
    destroy_graph(b);
    b->initialized = rc == LBM_OK;
    return rc;
}

// Step index of the next launch group's first step (rounding seed), written to
// the device before the group; advanced by the group's steps.
static int set_seed_base(LbmBatch* b, int32_t chunk) {
    const uint32_t v = b->seed_step;
    b->seed_step += (uint32_t)chunk;
    return lbm_cuda_check(&b->h, cudaMemcpyAsync(b->d_seed, &v, sizeof(v), cudaMemcpyHostToDevice, b->h.stream),
                          "seed base");
}

// Run `nsteps` (even) steps of all active subvolumes: graph launches of
// `chunk` steps when use_graph, else plain launches.  Leaves per-tile partials
// of the last step in device memory.
static int batch_run(LbmBatch* b, int32_t nsteps, int32_t chunk, int32_t use_graph) {
    LbmHandle* h = &b->h;
    if (use_graph) {
        if (b->graph_steps != chunk) {
            int rc = capture(b, chunk);
            if (rc) return rc;
        }
        for (int32_t done = 0; done < nsteps; done += chunk) {
            int rc = set_seed_base(b, chunk);
            if (!rc) rc = lbm_cuda_check(h, cudaGraphLaunch(b->graph, h->stream), "graph launch");
            if (rc) return rc;
        }
        return LBM_OK;
    }
    for (int32_t done = 0; done < nsteps; done += chunk) {
        int rc = set_seed_base(b, chunk);
        for (int k = 0; k < chunk && !rc; ++k) rc = launch_dispatch(b, k, k == chunk - 1, h->stream);
        if (rc) return rc;
    }
    return LBM_OK;
}

int lbm_batch_step(LbmBatch* b, int32_t nsteps, int32_t chunk, int32_t use_graph) {
    if (!b) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_step: NULL");
    if (!b->initialized) return batch_err(b, LBM_ESTATE, "lbm_batch_step: call lbm_batch_init first");
    if (chunk < 2 || chunk > 4096 || chunk % 2 || nsteps % chunk)
        return batch_err(b, LBM_EINVAL, "lbm_batch_step: chunk must be even, <= 4096, and divide nsteps");
    cudaSetDevice(b->h.device);
    int rc = batch_run(b, nsteps, chunk, use_graph);
    if (!rc) rc = lbm_cuda_check(&b->h, cudaStreamSynchronize(b->h.stream), "batch step");
    if (!rc)
        for (size_t q = 0; q < b->subs.size(); ++q)
            if (b->active[q]) b->steps[q] += nsteps;
    return rc;
}

// Darcy velocity along x of every active subvolume after the last step (the
// sum of v_x over its fluid nodes / its cells); inactive ones keep their value.
static int batch_darcy(LbmBatch* b, double* darcy) {
    LbmHandle* h = &b->h;
    std::vector<double> part(b->tiles.size());
    int rc = 0;
    if (!part.empty())
        rc = lbm_cuda_check(h, cudaMemcpy(part.data(), b->d_partial, sizeof(double) * part.size(), cudaMemcpyDeviceToHost), "copy partials");
    if (rc) return rc;
    std::vector<double> sum(b->subs.size(), 0.0);
    for (size_t t = 0; t < b->tiles.size(); ++t) sum[b->tiles[t].sub] += part[t];
    for (size_t q = 0; q < b->subs.size(); ++q)
        if (b->active[q]) {
            const BatchSub& s = b->subs[q];
            darcy[q] = sum[q] / ((double)s.nx * s.ny * s.nz);
        }
    return LBM_OK;
}

int lbm_batch_run_to_convergence(LbmBatch* b, double tol, int32_t check_every, int64_t max_steps, int32_t use_graph,
                                 double* darcy, int64_t* steps, int32_t* converged) {
    if (!b || !darcy || !steps || !converged) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_run_to_convergence: NULL");
    if (check_every < 2 || check_every > 4096 || check_every % 2)
        return batch_err(b, LBM_EINVAL, "lbm_batch_run_to_convergence: check_every must be even and <= 4096");
    if (!b->initialized) return batch_err(b, LBM_ESTATE, "lbm_batch_run_to_convergence: call lbm_batch_init first");
    LbmHandle* h = &b->h;
    cudaSetDevice(h->device);
    const size_t ns = b->subs.size();
    std::vector<double> prev(ns, 0.0), cur(ns, 0.0);
    std::vector<uint8_t> have(ns, 0);
    for (size_t q = 0; q < ns; ++q) converged[q] = 0;
    int64_t done = 0;
    while (done < max_steps) {
        bool any = false;
        for (size_t q = 0; q < ns; ++q) any |= b->active[q] != 0;
        if (!any) break;
        int rc = batch_run(b, check_every, check_every, use_graph);
        if (!rc) rc = lbm_cuda_check(h, cudaStreamSynchronize(h->stream), "batch run");
        if (rc) return rc;
        done += check_every;
        for (size_t q = 0; q < ns; ++q)
            if (b->active[q]) b->steps[q] += check_every;
        rc = batch_darcy(b, cur.data());
        if (rc) return rc;
        bool changed = false;
        for (size_t q = 0; q < ns; ++q) {
            if (!b->active[q]) continue;
            if (!std::isfinite(cur[q])) return batch_err(b, LBM_EDIVERGED, "subvolume diverged");
            if (have[q] && std::fabs(cur[q] - prev[q]) <= tol * std::fabs(cur[q])) {
                b->active[q] = 0;
                converged[q] = 1;
                changed = true;
            }
            prev[q] = cur[q];
            have[q] = 1;
        }
        if (changed) {
            rc = rebuild_tiles(b);
            if (rc) return rc;
        }
    }
    for (size_t q = 0; q < ns; ++q) {
        darcy[q] = cur[q];
        steps[q] = b->steps[q];
    }
    return LBM_OK;
}

int lbm_batch_get_macros(LbmBatch* b, int32_t sub, float* rho, float* v) {
    if (!b || !rho || !v) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_get_macros: NULL");
    if (sub < 0 || sub >= (int32_t)b->subs.size()) return batch_err(b, LBM_EINVAL, "lbm_batch_get_macros: bad subvolume");
    LbmHandle* h = &b->h;
    cudaSetDevice(h->device);
    const BatchSub sd = b->subs[sub];
    const int64_t nc = (int64_t)sd.nx * sd.ny * sd.nz;
    // the second population buffer holds nothing between runs of an even number of steps
    const size_t bytes[2] = {sizeof(float) * (size_t)nc, sizeof(float) * 3 * (size_t)nc};
    float* own = nullptr;
    float* d_out = (float*)h->d_f[1];
    if (bytes[0] + bytes[1] > h->elem * 19 * (size_t)h->np) {
        if (cudaMalloc((void**)&own, bytes[0] + bytes[1]) != cudaSuccess)
            return batch_err(b, LBM_ENOMEM, "lbm_batch_get_macros: out of device memory");
        d_out = own;
    }
    int rc = 0;
    switch (h->p.storage) {
    case LBM_STORE_F32: rc = macros_t<LBM_STORE_F32>(b, sub, d_out, d_out + nc); break;
    case LBM_STORE_F16_DEV: rc = macros_t<LBM_STORE_F16_DEV>(b, sub, d_out, d_out + nc); break;
    case LBM_STORE_BF16_DEV: rc = macros_t<LBM_STORE_BF16_DEV>(b, sub, d_out, d_out + nc); break;
    case LBM_STORE_F32_DEV: rc = macros_t<LBM_STORE_F32_DEV>(b, sub, d_out, d_out + nc); break;
    case LBM_STORE_F64: rc = macros_t<LBM_STORE_F64>(b, sub, d_out, d_out + nc); break;
    }
    void* const host[2] = {rho, v};
    if (!rc) host_touch(host, bytes, 2);
    for (int q = 0; q < 2 && !rc; ++q)
        rc = lbm_cuda_check(h, cudaMemcpyAsync(host[q], d_out + (q ? nc : 0), bytes[q], cudaMemcpyDeviceToHost, h->stream), "copy macros");
    const int rs = lbm_cuda_check(h, cudaStreamSynchronize(h->stream), "batch macros");
    cudaFree(own);
    return rc ? rc : rs;
}

int lbm_batch_get_stream(LbmBatch* b, void** stream) {
    if (!b || !stream) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_get_stream: NULL");
    *stream = (void*)b->h.stream;
    return LBM_OK;
}

int lbm_batch_info(LbmBatch* b, int64_t* n_nodes, int64_t* n_fluid, int32_t* grid, int32_t* n_tiles) {
    if (!b) return lbm_set_err(nullptr, LBM_EINVAL, "lbm_batch_info: NULL");
    int64_t nf = 0;
    for (auto& s : b->subs) nf += s.n_fluid;
    if (n_nodes) *n_nodes = b->h.n_fluid;
    if (n_fluid) *n_fluid = nf;
    if (grid) *grid = (int32_t)b->tiles.size();
    if (n_tiles) *n_tiles = (int32_t)b->tiles.size();
    return LBM_OK;
}

}  // extern "C"
