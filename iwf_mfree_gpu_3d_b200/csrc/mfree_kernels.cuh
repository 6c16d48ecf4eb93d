// mfree_kernels.cuh -- kernel declarations and helpers shared by the step's
// translation units.
#pragma once

#include <string>

#include "mfree_device.cuh"

namespace mfree {

constexpr int HASH_BLOCK = 256;
constexpr int BLANK_GROUP = 128;  // hash blocks per group of blanked counts
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
// Tiles of a scan up to which each of its blocks adds up the tiles before its
// own; beyond, kb_scan_top scans the tile sums first: the additions grow with
// the square of the cells, a launch does not.  Scan in us, additions / kb_scan_top
// (eager event times, some 5 us a kernel are the events'): 8,193 tiles 37 / 42,
// 16,001 68 / 66, 31,251 151 / 116, 128,001 1,427 / 433.
constexpr int SCAN_FLAT = 8192;
__host__ __device__ constexpr int scan_tiles_of(int num_cell) { return (num_cell + 1 + SCAN_TILE - 1) / SCAN_TILE; }
// blocks of a scene's kb_finalize: one per 256 particles, for many particles
// eight per SM (of 148), each of which looks over more of the contact bitmap (4.1M
// particles: 16,100 blocks took 54 us to find the few in contact)
constexpr int FIN_BLOCK = 256, FIN_BLOCKS_MAX = 8 * 148;
__host__ __device__ constexpr int finalize_blocks(int n) {
    return (n + FIN_BLOCK - 1) / FIN_BLOCK < FIN_BLOCKS_MAX ? (n + FIN_BLOCK - 1) / FIN_BLOCK : FIN_BLOCKS_MAX;
}
constexpr int NRES = 20;           // reduced accumulators per particle

// half-step state x + dt/2 * xdot of the predictor (leap_frog.cu:42-70); the
// pair kernel's epilogue recomputes it with the same expressions
struct HalfStep {
    float x, y, z, vx, vy, vz, rho, T;
    float S[6];  // xx yy zz xy xz yz
};

template <bool PREC>
__device__ __forceinline__ HalfStep half_step(float h2, float4 pos, float4 vel, float4 sa, float4 sb, float4 da,
                                              float4 dv, float4 dsa, float4 dsb, float4 lo, float4 lob) {
    HalfStep o;
    if (PREC) {
        o.x = pos.x + fmaf(h2, da.x, lo.x);
        o.y = pos.y + fmaf(h2, da.y, lo.y);
        o.z = pos.z + fmaf(h2, da.z, lo.z);
        o.vx = vel.x + fmaf(h2, dv.x, lo.w);
        o.vy = vel.y + fmaf(h2, dv.y, lob.x);
        o.vz = vel.z + fmaf(h2, dv.z, lob.y);
    } else {
        o.x = fmaf(h2, da.x, pos.x);
        o.y = fmaf(h2, da.y, pos.y);
        o.z = fmaf(h2, da.z, pos.z);
        o.vx = fmaf(h2, dv.x, vel.x);
        o.vy = fmaf(h2, dv.y, vel.y);
        o.vz = fmaf(h2, dv.z, vel.z);
    }
    o.rho = fmaf(h2, da.w, vel.w);
    o.T = fmaf(h2, dv.w, sb.z);
    o.S[0] = fmaf(h2, dsa.x, sa.x);
    o.S[1] = fmaf(h2, dsa.y, sa.y);
    o.S[2] = fmaf(h2, dsa.z, sa.z);
    o.S[3] = fmaf(h2, dsa.w, sa.w);
    o.S[4] = fmaf(h2, dsb.x, sb.x);
    o.S[5] = fmaf(h2, dsb.y, sb.y);
    return o;
}

// particle inside the box of tool k at this step (the contact kernels' early
// reject, tool_3d_gpu.cu:607-614), for a tool that is set up and alive
__device__ __forceinline__ bool in_tool_box(const StepArgs &a, int k, float x, float y, float z) {
    const ToolDev &T = a.tools[k];
    if (T.num_tris == 0) return false;
    const DevClock *c = a.clk;
    if (c->t < T.birth || c->t > T.death) return false;
    const ToolClock &b = c->tool[k];
    return x > b.bbmin[0] && x < b.bbmax[0] && y > b.bbmin[1] && y < b.bbmax[1] && z > b.bbmin[2] && z < b.bbmax[2];
}
__device__ __forceinline__ bool contact_candidate(const StepArgs &a, float x, float y, float z) {
    bool in = false;
    for (int k = 0; k < a.p.num_tools; k++) in |= in_tool_box(a, k, x, y, z);
    return in;
}

// ------------------------------------------------------ batched launches --
// The step's kernels run over a table of scenes: one scene (a context's own
// one-entry table) or many independent scenes of a batch, one launch per
// kernel either way, so a scene's arithmetic is the same compiled code alone
// and in a batch.  Every scene keeps
// its own state, cell list (a segment of its own) and clock; the table lists
// each scene's arguments once per state parity and, per kernel family, the
// first block (or tile) of every scene: block b of a launch belongs to the
// scene s with prefix[s] <= b < prefix[s + 1].
struct BatchTable {
    const StepArgs *args;  // [2 s + parity]
    const int *pblk;       // particle blocks of 256 threads (hash, scatter, gather, finalize)
    const int *stile;      // scan tiles of SCAN_TILE cells
    const int *irun;       // runs of pair-kernel tiles
    int nscenes;
    int *tile_next;        // work queue of the pair kernel: next entry of tile_list (reset by kb_clock)
    int *tile_count;       // entries of tile_list (reset by kb_clock)
    int2 *tile_list;       // non-empty pair-kernel tiles of every scene: (tile of the scene, scene * 16 + depth)
    int tile_max;          // entries it has room for
};

// Pair-kernel tiles.  A bundle is TX x TY columns of a scene's cell grid
// (numbered y fastest); the tile list cuts its levels along z into tiles of up
// to Params::tile_z levels and tile_cap targets, skipping empty levels.  So
// tiles come out about equally full, at the surfaces of a block and in dense
// or thin regions too (tiles of a fixed depth held 156 targets of the 211 of a
// full one on the 1M-particle block).
// A tile is named by bundle * gnz + its first level, and its depth.
// The cutting is one chain of some 0.4 us a tile, so a bundle is cut in runs of
// TILE_RUN levels, each by a warp of its own (4 x 4 x 2000 particles, a step:
// 244 us as one run, 106 us as thirteen).
constexpr int TX = 4, TY = 4, TILE_RUN = 128;
constexpr int TILE_HALO_MAX = 1640;  // records the halo of a tile should hold at most (estimated from its bundle)
struct TileGeo {
    int X0, Y0, Z0, zl, nzr, depth;
};
__host__ __device__ __forceinline__ TileGeo tile_geo(const Params &P, int t, int depth) {
    const int nby = (P.gny + TY - 1) / TY;
    const int b = t / P.gnz;
    TileGeo g;
    g.X0 = b / nby * TX;
    g.Y0 = b % nby * TY;
    g.Z0 = t - b * P.gnz;
    g.depth = depth;
    g.zl = g.Z0 - 2 > 0 ? g.Z0 - 2 : 0;
    const int zh = g.Z0 + depth + 1 < P.gnz - 1 ? g.Z0 + depth + 1 : P.gnz - 1;
    g.nzr = zh - g.zl + 2;  // cell starts per halo column of the tile (inclusive end)
    return g;
}
__host__ __device__ __forceinline__ int num_bundles(const Params &P) {
    return ((P.gnx + TX - 1) / TX) * ((P.gny + TY - 1) / TY);
}
__host__ __device__ __forceinline__ int bundle_runs(const Params &P) { return (P.gnz + TILE_RUN - 1) / TILE_RUN; }
// Particles of a bundle below level z, up to a constant: the sum of its columns'
// cell starts, modulo 2^32 (sixteen of them pass 2^31 from 134M particles on).
// The difference of two is the number of particles between the levels.
__host__ __device__ __forceinline__ unsigned bundle_below(int nx, int ny, int nz, const int *__restrict__ first,
                                                          const TileGeo &G, int z) {
    unsigned n = 0;
#pragma unroll
    for (int c = 0; c < TX * TY; c++) {
        const int cx = G.X0 + c / TY, cy = G.Y0 + c % TY;
        if (cx < nx && cy < ny) n += unsigned(first[(cx * ny + cy) * nz + z]);
    }
    return n;
}
// Whether a tile of depth > 1 that begins on level z0 is too deep: beyond the
// depth limit or the end of its run, with more than tile_cap targets, or with a
// halo (estimated as four times the bundle's own particles in the halo's
// levels) beyond TILE_HALO_MAX.  Depth 1 is always taken.
__host__ __device__ __forceinline__ bool tile_too_deep(const Params &P, int z0, int z_end, int depth,
                                                       int targets, int halo) {
    return depth > P.tile_z || z0 + depth > z_end || targets > P.tile_cap || 4 * halo > TILE_HALO_MAX;
}
// An upper bound of a scene's tiles, whatever cuts them: each begins on a level
// of a bundle where no other tile of the bundle begins, and holds a particle.
// (One counted from the limits alone is not safe: at 70 to 100 particles a
// level of a bundle the halo cuts every tile to one level, long before tile_cap.)
inline long long max_tiles(const Params &P) {
    const long long levels = (long long)num_bundles(P) * P.gnz;
    return levels < P.n_init ? levels : P.n_init;
}

// Programmatic dependent launch: a step's kernels are launched while the one
// before still runs (launch_after), so that launch latency and block start-up
// are hidden; each begins with begin_after, which waits until the kernel before
// has completed and its writes are visible, and only then lets the next one
// start.  So a kernel never overlaps the work of another, only its launch.
// Inside a stream capture the launches are plain: in a graph the programmatic
// edges cost more than they hide (8,000 particles, a step: eager 142 -> 129 us,
// graph 74.6 -> 76.3 us).
__device__ __forceinline__ void begin_after() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... K, class... A>
inline cudaError_t launch_after(void (*kern)(K...), int grid, int block, size_t smem, cudaStream_t s, A &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(unsigned(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaError_t e = cudaStreamIsCapturing(s, &cap)) return e;
    cfg.attrs = &at;
    cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, K(args)...);
}

// scene of block x: the last s with prefix[s] <= x (prefix has nscenes + 1 entries)
__device__ __forceinline__ int find_scene(const int *__restrict__ prefix, int nscenes, int x) {
    int lo = 0, hi = nscenes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// scene s's arguments for the parity of its current step, read in place
// (read-only through the kernel, so the loads stay in L1 after the first warp)
__device__ __forceinline__ const StepArgs &scene_args(const BatchTable &T, int s) {
    const StepArgs *a0 = T.args + 2 * s;
    return a0[a0->clk->parity & 1];
}

// copies scene s's arguments for the parity of its current step into shared
// memory; every thread of the block calls it, a barrier must follow
__device__ __forceinline__ void load_scene_args(StepArgs &dst, const BatchTable &T, int s) {
    const StepArgs *a0 = T.args + 2 * s;
    const int4 *src = reinterpret_cast<const int4 *>(a0 + (a0->clk->parity & 1));
    int4 *d = reinterpret_cast<int4 *>(&dst);
    for (int k = threadIdx.x; k < int(sizeof(StepArgs) / 16); k += blockDim.x) d[k] = src[k];
}

// Adds a block's particles to the counts of their cells (counted: a thread's
// cell, all ones for none) and to the sums of the scan's tiles.  Particles come
// in last step's sorted order, so a warp's cells run in stretches: the first
// lane of each adds its length (about 14 atomics a warp instead of 32).  A
// block's particles lie in one or two tiles: it adds them up in shared memory
// for the tiles around its middle thread's, and once to memory (an atomic a
// warp on the few tile sums took 13 us on 1M particles).
__device__ __forceinline__ void count_cells(const StepArgs &a, unsigned counted) {
    constexpr unsigned NEAR = 32;
    __shared__ int near_sum[NEAR];
    __shared__ unsigned near0;
    const int lane = threadIdx.x & 31;
    const unsigned none = 0xffffffffu, tile = counted == none ? none : counted / SCAN_TILE;
    if (threadIdx.x < NEAR) near_sum[threadIdx.x] = 0;
    if (threadIdx.x == HASH_BLOCK / 2) near0 = tile == none ? none : max(tile, NEAR / 2) - NEAR / 2;
    __syncthreads();
    const unsigned n0 = near0;
    auto stretches = [&](unsigned v, auto &&add) {
        const unsigned prev = __shfl_up_sync(0xffffffffu, v, 1);
        const bool start = lane == 0 || prev != v;
        const unsigned starts = __ballot_sync(0xffffffffu, start);
        if (start && v != none) {
            const unsigned after = starts & ~((2u << lane) - 1u);
            add(v, (after ? __ffs(after) - 1 : 32) - lane);
        }
    };
    stretches(counted, [&](unsigned v, int n) { atomicAdd(a.s.count + v, n); });
    stretches(tile, [&](unsigned v, int n) {
        if (n0 != none && v - n0 < NEAR) atomicAdd(&near_sum[v - n0], n);
        else atomicAdd(a.s.tile_sum + v, n);
    });
    __syncthreads();
    if (threadIdx.x < NEAR && near_sum[threadIdx.x]) atomicAdd(a.s.tile_sum + n0 + threadIdx.x, near_sum[threadIdx.x]);
}
// the blanked particles of a hash block, and of its group of blocks
__device__ __forceinline__ void note_blanked(const StepArgs &a, int bid, int nb) {
    a.s.blank_block[bid] = nb;
    if (nb) atomicAdd(a.s.blank_group + bid / BLANK_GROUP, nb);
}

__global__ void kb_clock(BatchTable T, int record_mode);
__global__ void kb_hash(BatchTable T);
// top: a scene has more than SCAN_FLAT tiles (launch_scan_top_batch comes first then)
cudaError_t launch_scan_top_batch(const BatchTable &T, cudaStream_t s);
cudaError_t launch_scan_batch(const BatchTable &T, bool top, int blocks, cudaStream_t s);
__global__ void kb_scatter(BatchTable T);
cudaError_t launch_gather_predict_batch(const BatchTable &T, bool precision, int blocks, cudaStream_t s);
__global__ void kb_finalize(BatchTable T);
__global__ void kb_force_final(BatchTable T);
// one pair-kernel launch over the tiles of every scene (all scenes share the
// variant); grid <= 0 only prepares the variant
cudaError_t launch_interact_batch(const BatchTable &T, bool cspm, int conduction, bool precision, int grid,
                                  cudaStream_t s);

// the sort kernels on arguments passed by value, for the allocation-free
// cell-list build (mfree_static.cu)
__global__ void k_scan(StepArgs a);
__global__ void k_scatter(StepArgs a);
__global__ void k_cell_fixup(StepArgs a);

// initial particle state from the constructor's device arrays (mfree_create)
cudaError_t launch_init_state(int n, const float4 *pos, const float4 *vel, const float *rho, const float *T,
                              const float *h, const float *fixed, const float *tool_p, const State &S, int *perm,
                              cudaStream_t s);

// message returned by mfree_last_error() (mfree_host.cu)
void set_last_error(const std::string &msg);

// sustained FP32 FMA throughput of the current device in TFLOP/s (mfree_probe.cu)
double fp32_peak_probe(int num_sms);

}  // namespace mfree
