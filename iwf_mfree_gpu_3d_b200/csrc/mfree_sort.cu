// mfree_sort.cu -- start of the step: clock, blanking + cell hash, stable
// counting sort by cell, and the gather that fuses the reorder with the
// predictor, the equation of state and the artificial stress.
//
// Reference path replaced (src/leap_frog.cu:133-151):
//   blanking::update + do_blanking          actions_gpu.cu:489-531, blanking.cpp:43-51
//   grid_base::update_geometry (locked)     grid_gpu_base.cu:166-183
//   compute_hashes                          grid_gpu_base.cu:41-63
//   adapt_particle_number (thrust::count)   grid_gpu_base.cu:141-164
//   do_sort: sequence + stable sort_by_key, cell range build, reorder_data
//                                           grid_gpu_green.cu:24-125,265-297
//   init, predict                           leap_frog.cu:30-70
//   do_material_eos, do_corrector_artificial_stress  actions_gpu.cu:40-132
//
// The sort is a stable counting sort: an atomic histogram of cell ids (and of
// the scan's tiles), an exclusive scan (which is also the cell-range table the
// pair loop reads), an atomic scatter, and a gather that takes each entry to
// its rank by previous index within its cell.  Four kernels (and a scan of the
// tile sums on grids of many cells): for small scenes the launches are what the
// sort costs (~3.5 us each; separate reduction, scan of the tile sums and
// per-cell fix-up made it seven).  The result equals thrust's stable
// sort_by_key of (cell id, 0..n-1): cells ascending, previous order inside a
// cell, blanked particles (cell id INT_MAX in the reference) last in previous
// order.
// N stays on the device: no host round trip per step.
#include "mfree_kernels.cuh"

namespace mfree {

// ----------------------------------------------------------------- clock --
// batched kernels: block b of the launch is block b - prefix[s] of scene s,
// whose arguments the block reads in place (a copy into shared memory, one
// barrier per block, cost these short blocks more than it saved)
template <class F> __device__ __forceinline__ void run_batched(const BatchTable &T, const int *prefix, F &&body) {
    const int s = find_scene(prefix, T.nscenes, blockIdx.x);
    body(scene_args(T, s), int(blockIdx.x) - prefix[s]);
}

// record_mode: 0 no, 1 yes, 2 every Params::record_every steps
__device__ __forceinline__ void clock_body(const StepArgs &a, int record_mode) {
    DevClock *c = a.clk;
    const Params &P = a.p;
    if (c->pending) {
        c->t = c->t + P.dt;  // main(): global_time_current += dt after each iteration
        c->parity ^= 1;      // the last step's output is this step's input
    }
    c->pending = 1;
    c->max_disp = 0u;
    const float t = c->t;
    c->record = record_mode == 1 ? 1
                : record_mode == 2 ? (P.record_every > 0 && (c->step_index % P.record_every) == 0)
                                   : 0;
    c->step_index++;
    if (P.blank_on)
        for (int d = 0; d < 3; d++) {
            c->blank_min[d] = P.blank_min0[d] + t * P.blank_vel[d];
            c->blank_max[d] = P.blank_max0[d] + t * P.blank_vel[d];
        }
    if (P.grid_moving)
        for (int d = 0; d < 3; d++) c->grid_min[d] = P.grid_min0[d] + t * P.grid_vel[d];
    for (int k = 0; k < P.num_tools; k++) {
        if (a.tools[k].num_tris == 0) continue;  // update_tool returns early without boxed triangles
        for (int d = 0; d < 3; d++) {
            c->tool[k].bbmin[d] += P.dt * a.tools[k].vel[d];
            c->tool[k].bbmax[d] += P.dt * a.tools[k].vel[d];
        }
    }
}

// one thread per scene; thread 0 also resets the batch's pair-kernel queue
__global__ void kb_clock(BatchTable T, int record_mode) {
    begin_after();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {
        *T.tile_next = 0;
        *T.tile_count = 0;
    }
    if (s < T.nscenes) clock_body(T.args[2 * s], record_mode);
}

// ------------------------------------------------- blanking + cell hash --
__device__ __forceinline__ void hash_body(const StepArgs &a, int bid) {
    const Params &P = a.p;
    const int i = bid * HASH_BLOCK + threadIdx.x;
    int blank = 0;
    unsigned counted = 0xffffffffu;  // the cell this particle is counted in (none: all ones)
    if (i < P.n_init) {
        float4 p = a.a.pos4[i];
        float4 ft = a.a.ft4[i];
        float blanked = ft.w;
        if (P.blank_on) {
            float4 v = a.a.vel4[i];
            const DevClock *c = a.clk;
            bool fast = __fadd_rn(__fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y)), __fmul_rn(v.z, v.z)) >= P.vmax2;
            bool in = p.x >= c->blank_min[0] && p.x <= c->blank_max[0] && p.y >= c->blank_min[1] &&
                      p.y <= c->blank_max[1] && p.z >= c->blank_min[2] && p.z <= c->blank_max[2];
            if (fast || !in) {
                blanked = 1.f;
            } else if (blanked != 0.f) {
                // inside and slow: the reference unblanks unless a rate is NaN/Inf
                // (actions_gpu.cu:504-529), and a particle that is not blanked
                // stays so either way -- the rates are read only to unblank
                float4 da = a.a.da4[i], dv = a.a.dv4[i], dsa = a.a.dsa4[i], dsb = a.a.dsb4[i];
                bool bad = nan_or_inf(da.x) || nan_or_inf(da.y) || nan_or_inf(da.z) || nan_or_inf(dv.x) ||
                           nan_or_inf(dv.y) || nan_or_inf(dv.z) || nan_or_inf(dsa.x) || nan_or_inf(dsa.y) ||
                           nan_or_inf(dsa.z) || nan_or_inf(dsa.w) || nan_or_inf(dsb.y) || nan_or_inf(dsb.x) ||
                           nan_or_inf(da.w) || nan_or_inf(dv.w);
                if (!bad) blanked = 0.f;
            }
            if (blanked == 1.f) {  // count blanked particles carrying a NaN/Inf position or rate
                float4 da = a.a.da4[i], dv = a.a.dv4[i], dsa = a.a.dsa4[i], dsb = a.a.dsb4[i];
                bool bad = nan_or_inf(p.x) || nan_or_inf(p.y) || nan_or_inf(p.z) || nan_or_inf(da.x) ||
                           nan_or_inf(da.y) || nan_or_inf(da.z) || nan_or_inf(dv.x) || nan_or_inf(dv.y) ||
                           nan_or_inf(dv.z) || nan_or_inf(dsa.x) || nan_or_inf(dsa.y) || nan_or_inf(dsa.z) ||
                           nan_or_inf(dsa.w) || nan_or_inf(dsb.x) || nan_or_inf(dsb.y) || nan_or_inf(da.w) ||
                           nan_or_inf(dv.w);
                if (bad) atomicAdd(&a.clk->nan_blanked, 1ull);
            }
        }
        unsigned key = unsigned(P.num_cell);
        if (blanked != 1.f) {
            const float *gmin = P.grid_moving ? a.clk->grid_min : P.grid_min0;
            int ix = int(__fdiv_rn(__fsub_rn(p.x, gmin[0]), P.gdx));
            int iy = int(__fdiv_rn(__fsub_rn(p.y, gmin[1]), P.gdx));
            int iz = int(__fdiv_rn(__fsub_rn(p.z, gmin[2]), P.gdx));
            if (ix >= 0 && ix < P.gnx && iy >= 0 && iy < P.gny && iz >= 0 && iz < P.gnz) {
                key = unsigned((ix * P.gny + iy) * P.gnz + iz);
            } else {
                blanked = 1.f;  // outside the cell grid but not blanked: taken out (counted)
                atomicAdd(&a.clk->out_of_grid, 1ull);
            }
        }
        if (blanked != ft.w) {
            ft.w = blanked;
            a.a.ft4[i] = ft;
        }
        a.s.key[i] = key;
        if (key < unsigned(P.num_cell)) counted = key;
        else blank = 1;
    }
    count_cells(a, counted);
    int nb = __syncthreads_count(blank);
    if (threadIdx.x == 0) note_blanked(a, bid, nb);
}
__global__ void __launch_bounds__(HASH_BLOCK) kb_hash(BatchTable T) {
    begin_after();
    run_batched(T, T.pblk, [](const StepArgs &a, int b) { hash_body(a, b); });
}

// ------------------------------------------------------------- the scan --
// exclusive scan of count[0..num_cell) into first[0..num_cell]; first[num_cell] = N
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_sums[lane] = w;  // inclusive
    }
    __syncthreads();
    int pre = warp > 0 ? warp_sums[warp - 1] : 0;
    total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return pre + x - v;
}

// exclusive scan of the tile sums in place, for grids of many tiles
__device__ __forceinline__ void scan_top_body(const StepArgs &a) {
    __shared__ int ws[32];
    constexpr int PER = 8;
    const int tiles = scan_tiles_of(a.p.num_cell);
    if (tiles <= SCAN_FLAT) return;
    int carry = 0;
    for (int b = 0; b < tiles; b += 1024 * PER) {
        const int t = b + int(threadIdx.x) * PER;
        int v[PER], s = 0, total;
#pragma unroll
        for (int k = 0; k < PER; k++) s += v[k] = t + k < tiles ? a.s.tile_sum[t + k] : 0;
        int ex = carry + block_exclusive_scan(s, ws, total);
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (t + k < tiles) a.s.tile_sum[t + k] = ex;
            ex += v[k];
        }
        carry += total;
    }
}
// one block per scene
__global__ void __launch_bounds__(1024) kb_scan_top(BatchTable T) {
    begin_after();
    scan_top_body(scene_args(T, blockIdx.x));
}

// Up to SCAN_FLAT tiles each block sums the tiles before its own (1,734 on the
// 4.1M-particle scene: seven loads a thread), so the tile sums need no scan.
// TOP: kb_scan_top has run and scanned those of scenes of more tiles.
template <bool TOP> __device__ __forceinline__ void scan_body(const StepArgs &a, int bid) {
    __shared__ int ws[32];
    const int nc = a.p.num_cell;
    int total, before = 0;
    const bool scanned = TOP && scan_tiles_of(nc) > SCAN_FLAT;
    if (!scanned)
        for (int t = threadIdx.x; t < bid; t += SCAN_THREADS) before += a.s.tile_sum[t];
    else if (threadIdx.x == 0)
        before = a.s.tile_sum[bid];
    block_exclusive_scan(before, ws, total);
    const int start = total;
    const int base = bid * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
    // (the counters and the first table start on 16 bytes, or are read and written one by one)
    const bool vec = base + SCAN_ITEMS <= nc && ((size_t(a.s.count) | size_t(a.s.first)) & 15) == 0;
    static_assert(SCAN_ITEMS == 8, "two vectors a thread");
    if (vec) {
        const int4 x = reinterpret_cast<const int4 *>(a.s.count + base)[0],
                   y = reinterpret_cast<const int4 *>(a.s.count + base)[1];
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) v[k] = base + k < nc ? a.s.count[base + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) s += v[k];
    int ex = block_exclusive_scan(s, ws, total) + start;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {  // v becomes the exclusive scan
        const int n = v[k];
        v[k] = ex;
        ex += n;
    }
    if (vec) {
        int4 *f = reinterpret_cast<int4 *>(a.s.first + base);
        f[0] = make_int4(v[0], v[1], v[2], v[3]);
        f[1] = make_int4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            if (base + k > nc) break;
            a.s.first[base + k] = v[k];
            if (base + k == nc) a.clk->n_active = v[k];  // first[nc] = N
        }
    }
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(StepArgs a) {
    begin_after();
    scan_body<false>(a, blockIdx.x);
}
template <bool TOP> __global__ void __launch_bounds__(SCAN_THREADS) kb_scan(BatchTable T) {
    begin_after();
    run_batched(T, T.stile, [](const StepArgs &a, int b) { scan_body<TOP>(a, b); });
}

// ---------------------------------------------------------- the scatter --
// out: sorted position -> previous position, a cell's entries in no order yet
__device__ __forceinline__ void scatter_body(const StepArgs &a, int bid, int *out) {
    __shared__ int ws[32];
    const Params &P = a.p;
    {   // the tile sums are done with: zero for the next step
        const int tiles = scan_tiles_of(P.num_cell), nb = (P.n_init + HASH_BLOCK - 1) / HASH_BLOCK;
        for (int t = bid * HASH_BLOCK + threadIdx.x; t < tiles; t += nb * HASH_BLOCK) a.s.tile_sum[t] = 0;
    }
    const int i = bid * HASH_BLOCK + threadIdx.x;
    const int N = a.clk->n_active;
    unsigned key = i < P.n_init ? a.s.key[i] : 0u;
    int blank = (i < P.n_init && key >= unsigned(P.num_cell)) ? 1 : 0;
    int total, rank = 0;
    if (N < P.n_init) {  // blanked particles: those of the groups and blocks before this one come first
        const int g = bid / BLANK_GROUP;
        int before = 0;
        for (int t = threadIdx.x; t < g; t += HASH_BLOCK) before += a.s.blank_group[t];
        for (int t = g * BLANK_GROUP + threadIdx.x; t < bid; t += HASH_BLOCK) before += a.s.blank_block[t];
        block_exclusive_scan(before, ws, total);
        const int start = total;
        rank = start + block_exclusive_scan(blank, ws, total);
    }
    // one atomic per stretch of equal keys in the warp (the hash kernel's
    // stretches): its first lane takes the stretch's length off the cell's
    // count (which leaves count[] zero for the next step) and the stretch
    // fills its slots in lane order
    const int lane = threadIdx.x & 31;
    const unsigned counted = (i < P.n_init && !blank) ? key : 0xffffffffu;
    const unsigned prev = __shfl_up_sync(0xffffffffu, counted, 1);
    const bool start = lane == 0 || prev != counted;
    const unsigned starts = __ballot_sync(0xffffffffu, start);
    const unsigned upto = starts & ((2u << lane) - 1u);  // starts at or below this lane
    const int head = 31 - __clz(upto);
    const unsigned after = starts & ~((2u << lane) - 1u);
    const int end = after ? __ffs(after) - 1 : 32;
    int old = 0;
    if (start && counted != 0xffffffffu) old = atomicSub(&a.s.count[counted], end - lane);
    old = __shfl_sync(0xffffffffu, old, head);
    if (i >= P.n_init) return;
    if (!blank) {
        const int d = a.s.first[key] + old - (end - head) + (lane - head);
        if (bounds_ok(a.clk, d, P.n_init)) out[d] = i;
    } else {
        const int d = N + rank;
        if (bounds_ok(a.clk, d, P.n_init)) out[d] = i;
    }
}
__global__ void __launch_bounds__(HASH_BLOCK) k_scatter(StepArgs a) {
    begin_after();
    scatter_body(a, blockIdx.x, a.s.perm);
}

// order each cell's entries by previous index (stable within the cell), in
// place; the step's gather ranks them instead
__device__ __forceinline__ void cell_fixup_body(const StepArgs &a, int bid) {
    const int c = bid * 256 + threadIdx.x;
    if (c >= a.p.num_cell) return;
    const int s = a.s.first[c], e = a.s.first[c + 1];
    if (e - s < 2) return;
    if (!bounds_ok(a.clk, s, a.p.n_init) || !bounds_ok(a.clk, e - 1, a.p.n_init)) return;
    int *p = a.s.perm;
    for (int k = s + 1; k < e; k++) {
        int v = p[k];
        int m = k - 1;
        while (m >= s && p[m] > v) {
            p[m + 1] = p[m];
            m--;
        }
        p[m + 1] = v;
    }
}
__global__ void __launch_bounds__(256) k_cell_fixup(StepArgs a) {
    begin_after();
    cell_fixup_body(a, blockIdx.x);
}

// The pair kernel's list of non-empty tiles: one warp per run of a bundle of
// every scene.  Lane k holds bundle_below of level base + k, so a tile's depth
// is one ballot over the lanes behind its first level; the run's tiles are
// appended with one atomic per 32 of them.  The order of the list changes which
// block runs a tile, never a result.
__device__ __forceinline__ void tile_list_body(const BatchTable &T, int g, int lane) {
    if (g >= T.irun[T.nscenes]) return;
    const int s = find_scene(T.irun, T.nscenes, g);
    const StepArgs &a = scene_args(T, s);
    const Params &P = a.p;
    const int nx = P.gnx, ny = P.gny, nz = P.gnz, nb = num_bundles(P);
    int bun = g - T.irun[s], z_begin = 0;  // the bundles' first runs come first, then their second ones
    for (; bun >= nb; bun -= nb) z_begin += TILE_RUN;
    const int z_end = min(z_begin + TILE_RUN, nz);
    const TileGeo G = tile_geo(P, bun * nz, 1);
    const int *__restrict__ first = a.s.first;
    int base = 0;
    unsigned F = 0;
    auto load = [&](int z) {
        base = z;
        F = bundle_below(nx, ny, nz, first, G, min(z + lane, nz));
    };
    auto at = [&](int z) { return __shfl_sync(0xffffffffu, F, min(z, nz) - base); };
    load(max(z_begin - 2, 0));
    int2 mine = make_int2(0, 0);
    int n = 0;
    auto flush = [&] {
        int k = 0;
        if (lane == 0) k = atomicAdd(T.tile_count, n);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (lane < n && bounds_ok(a.clk, k + lane, T.tile_max)) T.tile_list[k + lane] = mine;
        n = 0;
    };
    for (int z0 = z_begin; z0 < z_end;) {
        if (min(z0 + TILE_Z_MAX + 2, nz) > base + 31) load(max(z0 - 2, 0));
        // the first level with a target (a level past the window: look again there)
        const unsigned below = at(z0);
        const unsigned some = __ballot_sync(0xffffffffu, base + lane > z0 && base + lane <= nz && int(F - below) > 0);
        if (some == 0) {
            z0 = base + 31;
            continue;
        }
        const int zf = base + __ffs(some) - 2;
        if (zf > z0) {
            z0 = zf;
            continue;  // (the window may have to move)
        }
        // lane d: would a tile of depth d fit?
        const int d = lane;
        const int in = int(__shfl_sync(0xffffffffu, F, min(max(min(z0 + d, nz) - base, 0), 31)) - below);
        const int halo = int(__shfl_sync(0xffffffffu, F, min(max(min(z0 + d + 2, nz) - base, 0), 31)) - at(max(z0 - 2, 0)));
        const unsigned bad = __ballot_sync(0xffffffffu, d > 1 && tile_too_deep(P, z0, z_end, d, in, halo));
        const int depth = bad ? __ffs(bad) - 2 : 1;
        if (lane == n) mine = make_int2(bun * nz + z0, s * 16 + depth);
        if (++n == 32) flush();
        z0 += depth;
    }
    if (n > 0) flush();
}

// the first blocks build the tile list (the cell starts are final once the scan
// has run), the others scatter
__global__ void __launch_bounds__(HASH_BLOCK) kb_scatter(BatchTable T) {
    begin_after();
    const int tb = (T.irun[T.nscenes] + 7) / 8, b = int(blockIdx.x) - tb;
    if (b < 0) {
        tile_list_body(T, int(blockIdx.x) * 8 + int(threadIdx.x >> 5), int(threadIdx.x & 31));
        return;
    }
    const int s = find_scene(T.pblk, T.nscenes, b);
    const StepArgs &a = scene_args(T, s);
    scatter_body(a, b - T.pblk[s], a.s.perm_raw);
}

// --------------------------------------------- gather + predictor + EOS --
template <bool PREC> __device__ __forceinline__ void gather_predict_body(const StepArgs &a, int bid) {
    const Params &P = a.p;
    int i = bid * 256 + threadIdx.x;
    {   // the groups' blanked counts are done with: zero for the next step
        const int groups = (P.n_init + HASH_BLOCK * BLANK_GROUP - 1) / (HASH_BLOCK * BLANK_GROUP);
        if (i < groups) a.s.blank_group[i] = 0;
    }
    if (i >= P.n_init) return;
    const int N = a.clk->n_active;
    int src = a.s.perm_raw[i];
    if (src < 0 || src >= P.n_init) {  // cannot happen for a consistent sort; never read out of bounds
        atomicAdd(&a.clk->out_of_grid, 1ull << 32);
        src = i;
    }
    const unsigned key = a.s.key[src];
    if (i < N && key < unsigned(P.num_cell)) {
        // the entry's place in its cell: its rank by previous index (a cell
        // holds about two; the scatter leaves them in no order)
        const int c0 = a.s.first[key], c1 = a.s.first[key + 1];
        if (c1 - c0 > 1 && bounds_ok(a.clk, c0, P.n_init) && bounds_ok(a.clk, c1 - 1, P.n_init)) {
            i = c0;
            for (int k = c0; k < c1; k++) i += a.s.perm_raw[k] < src ? 1 : 0;
        }
    }
    a.s.perm[i] = src;
    const State &A = a.a, &B = a.b;
    float4 pos = A.pos4[src], vel = A.vel4[src], sa = A.sa4[src], sb = A.sb4[src];
    float4 da = A.da4[src], dv = A.dv4[src], dsa = A.dsa4[src], dsb = A.dsb4[src];
    float4 fc = A.fc4[src], ft = A.ft4[src], bc = A.bc4[src];
    B.pos4[i] = pos; B.vel4[i] = vel; B.sa4[i] = sa; B.sb4[i] = sb;
    B.da4[i] = da; B.dv4[i] = dv; B.dsa4[i] = dsa; B.dsb4[i] = dsb;
    B.fc4[i] = fc; B.ft4[i] = ft; B.bc4[i] = bc;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), lob = lo;
    if (PREC) {
        lo = A.lo4[src];
        lob = A.lo4b[src];
        B.lo4[i] = lo;
        B.lo4b[i] = lob;
    }
    a.s.key_sorted[i] = key;
    if (i >= N) return;  // blanked: frozen
    const float h2 = 0.5f * P.dt;
    HalfStep hs = half_step<PREC>(h2, pos, vel, sa, sb, da, dv, dsa, dsb, lo, lob);
    {   // the step's largest predictor move in cells (the pair kernel's pruning margin): a
        // warp maximum, raised in the clock only when it is larger than the value there
        float d = fmaxf(fabsf(hs.x - pos.x), fmaxf(fabsf(hs.y - pos.y), fabsf(hs.z - pos.z))) / P.gdx;
        if (!(d <= PRUNE_DISP_MAX)) d = 2.0f * PRUNE_DISP_MAX;  // NaN, Inf or beyond the cap
        const unsigned act = __activemask();
        const unsigned m = __reduce_max_sync(act, __float_as_uint(d));  // d >= 0: bits order as values
        if ((threadIdx.x & 31) == __ffs(act) - 1 && m > *(volatile unsigned *)&a.clk->max_disp) {
            const unsigned cap = __float_as_uint(PRUNE_DISP_MAX);
            const unsigned old = atomicMax(&a.clk->max_disp, m);
            if (m > cap && old <= cap) atomicAdd(&a.clk->full_stencil_steps, 1ull);  // once per step
        }
    }
    const bool tool = fc.w == 1.f;
    float prs = 0.f;
    float Rr[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (!tool) {
        prs = P.c0sq * (hs.rho - P.rho0);
        if (P.stresseps != 0.f)
            artificial_stress(hs.S[0], hs.S[1], hs.S[2], hs.S[3], hs.S[4], hs.S[5], prs, hs.rho, P.stresseps, Rr);
    }
    const float ir2 = 1.0f / (hs.rho * hs.rho);
    const Records &r = a.r;
    r.f[REC_P][i] = make_float4(hs.x, hs.y, hs.z, fc.w);  // raw tool_particle value
    float4 *x = r.f[REC_V] + size_t(i) * REC_X;  // V, A, B, R, C interleaved
    x[REC_V - 1] = make_float4(hs.vx, hs.vy, hs.vz, hs.rho);
    x[REC_A - 1] = make_float4((hs.S[0] - prs) * ir2, hs.S[3] * ir2, hs.S[4] * ir2, hs.S[5] * ir2);
    x[REC_B - 1] = make_float4((hs.S[1] - prs) * ir2, (hs.S[2] - prs) * ir2, sqrtf(P.K / hs.rho), pos.w);
    x[REC_R - 1] = make_float4(Rr[0], Rr[3], Rr[4], Rr[5]);
    x[REC_C - 1] = make_float4(Rr[1], Rr[2], hs.T, P.mass / hs.rho);
    if (P.diagnostics) a.s.pos_half[i] = make_float4(hs.x, hs.y, hs.z, 0.f);
}
template <bool PREC> __global__ void __launch_bounds__(256) kb_gather_predict(BatchTable T) {
    begin_after();
    run_batched(T, T.pblk, [](const StepArgs &a, int b) { gather_predict_body<PREC>(a, b); });
}

// the initial state of a context from the constructor's arrays (particle_gpu,
// particle_gpu.cu:20-117: zeros except the given fields); the optional arrays
// may be NULL
__global__ void __launch_bounds__(256) k_init_state(int n, const float4 *pos, const float4 *vel, const float *rho,
                                                    const float *T, const float *h, const float *fixed,
                                                    const float *tool_p, State S, int *perm) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 p = pos[i], v = vel[i];
    S.pos4[i] = make_float4(p.x, p.y, p.z, h[i]);
    S.vel4[i] = make_float4(v.x, v.y, v.z, rho[i]);
    S.sa4[i] = z;
    S.sb4[i] = make_float4(0.f, 0.f, T ? T[i] : 0.f, 0.f);
    S.da4[i] = z;
    S.dv4[i] = z;
    S.dsa4[i] = z;
    S.dsb4[i] = make_float4(0.f, 0.f, 0.f, fixed ? fixed[i] : 0.f);
    S.fc4[i] = make_float4(0.f, 0.f, 0.f, tool_p ? tool_p[i] : 0.f);
    S.ft4[i] = z;
    S.bc4[i] = make_float4(0.f, 0.f, 0.f, __int_as_float(i));  // creation index
    S.lo4[i] = z;
    S.lo4b[i] = z;
    perm[i] = i;
}

cudaError_t launch_init_state(int n, const float4 *pos, const float4 *vel, const float *rho, const float *T,
                              const float *h, const float *fixed, const float *tool_p, const State &S, int *perm,
                              cudaStream_t s) {
    k_init_state<<<(n + 255) / 256, 256, 0, s>>>(n, pos, vel, rho, T, h, fixed, tool_p, S, perm);
    return cudaGetLastError();
}

cudaError_t launch_scan_top_batch(const BatchTable &T, cudaStream_t s) {
    return launch_after(kb_scan_top, T.nscenes, 1024, 0, s, T);
}
cudaError_t launch_scan_batch(const BatchTable &T, bool top, int blocks, cudaStream_t s) {
    return launch_after(top ? kb_scan<true> : kb_scan<false>, blocks, SCAN_THREADS, 0, s, T);
}
cudaError_t launch_gather_predict_batch(const BatchTable &T, bool precision, int blocks, cudaStream_t s) {
    return launch_after(precision ? kb_gather_predict<true> : kb_gather_predict<false>, blocks, 256, 0, s, T);
}

}  // namespace mfree
