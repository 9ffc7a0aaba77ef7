// kernels_grid.cuh -- neighbour grid on sm_103a: cell hash, counting sort
// with one atomic per particle, segmented exclusive scan, scatter and a
// deterministic per-cell order (ascending particle index), plus the gathers
// that build the cell-sorted float4 copies the pair kernels stream.
//
// Replaces find_particle_bins, zero_gridcount, count_particles_in_bins,
// prefix_sum, copy_celloffset_to_backup and insert_particles_in_bin_array
// (kernels/common.cl:372-529).  Output fields gridcell, gridcount,
// celloffset and cellparticles have the reference's meaning and layout; the
// order inside a cell is ascending particle index (the reference's is the
// atomic race order).
#pragma once

#include <cooperative_groups.h>

#include "kernels_common.cuh"

// The scatter is a chain of dependent loads (work entry -> scene -> gridcell
// -> celloffset), so each of its blocks takes SPH_WIDE consecutive work
// entries per pass and runs their chains side by side: the loads of all
// entries are issued before any result is used, and a launch needs a quarter
// of the blocks.
#define SPH_WIDE 4

struct WideItem {
    const SceneDesc *S;  // null: no entry, or the scene idles
    unsigned item;
    bool valid;          // item < the scene's active count
};

__device__ __forceinline__ void wide_items(const SceneDesc *__restrict__ scenes, const BlockMap &map, unsigned v0,
                                           WideItem (&w)[SPH_WIDE]) {
#pragma unroll
    for (int j = 0; j < SPH_WIDE; ++j) {
        w[j].S = nullptr;
        w[j].item = 0u;
        w[j].valid = false;
        const unsigned v = v0 + j;
        if (v < map.num) {
            const BlockWork bw = map.work[v];
            const SceneDesc *S = scenes + bw.scene;
            if (!scene_idle(*S)) {
                w[j].S = S;
                w[j].item = bw.first + threadIdx.x;
                w[j].valid = w[j].item < active_count(*S);
            }
        }
    }
}

#define SPH_FOR_WIDE(map)                                                                       \
    follow_previous();                                                                          \
    for (unsigned v0_ = blockIdx.x * SPH_WIDE; v0_ < (map).num; v0_ += gridDim.x * SPH_WIDE) { \
        WideItem W[SPH_WIDE];                                                                   \
        wide_items(scenes, map, v0_, W);
#define SPH_END_WIDE }

// Blocks for a wide launch over `map`, at most `cap`.
__host__ __device__ inline unsigned wide_grid(unsigned num, unsigned cap) {
    const unsigned g = (num + SPH_WIDE - 1) / SPH_WIDE;
    const unsigned c = g < cap ? g : cap;
    return c ? c : 1u;
}

// find_particle_bins' cell coordinate (common.cl:372-391): clamp((uint)((p
// - b0)/(b1 - b0)*R), 0, R-1) with each float operation individually
// rounded and a saturating conversion; *outside is set for a particle
// outside gridbounds.
__device__ __forceinline__ unsigned cell_of(const SceneDesc &S, float3 p, bool *outside) {
    const float *gb = S.gridbounds;
    const float q[3] = {p.x, p.y, p.z};
    unsigned c[3];
    bool out = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = gb[2 * a], hi = gb[2 * a + 1];
        const float r = (float)S.gridres[a];
        const float v = __fmul_rn(__fdiv_rn(__fsub_rn(q[a], lo), __fsub_rn(hi, lo)), r);
        unsigned u = __float2uint_rz(v);  // saturating: negative and NaN -> 0
        if (u > S.gridres[a] - 1) u = S.gridres[a] - 1;
        out |= !(v >= 0.f && v < r);
        c[a] = u;
    }
    *outside = out;
    return c[2] * S.gridres[0] * S.gridres[1] + c[1] * S.gridres[0] + c[0];
}

// find_particle_bins (common.cl:372-391) fused with count_particles_in_bins
// (:401-408).  Each particle keeps its arrival slot within the cell, from
// one atomic per particle: a chain of dependent accesses bounds the pass,
// not the counts' atomics in L2, and combining a warp's lanes by cell first
// with a match instruction took longer than the atomics it saved.  The scan
// tiles' totals are counted in shared memory first: a few dozen tiles hold
// a scene of 100,000 particles, and once these are no longer in cell order
// every lane's atomic went to one of those few words (with the zeroing 29 ->
// 16 us, and 30 -> 23 us for 1M particles in order).  Looking the totals up
// in the scan instead, tile by tile, took its time from 8 to 14 us.  A grid
// of more than SPH_BIN_TILES tiles spreads them enough to add directly.
// (One work entry per block: the wide form measured slower here.)
#define SPH_BIN_TILES 512
__global__ void k_bin_count(const SceneDesc *__restrict__ scenes, BlockMap map, int do_count) {
    __shared__ unsigned tiles[SPH_BIN_TILES];
    SPH_FOR_WORK(map)
    const unsigned n = active_count(S);
    if (item - threadIdx.x >= n) continue;
    const unsigned few = do_count && S.num_scan_blocks <= SPH_BIN_TILES ? S.num_scan_blocks : 0u;
    if (few) {
        for (unsigned t = threadIdx.x; t < few; t += blockDim.x) tiles[t] = 0u;
        __syncthreads();
    }
    if (item < n) {
        bool outside;
        const unsigned cell = cell_of(S, ld3(S.position, item), &outside);
        if (do_count) {
            if (few) atomicAdd(tiles + cell / SPH_SCAN_TILE, 1u);
            else atomicAdd(S.scan_sums + cell / SPH_SCAN_TILE, 1u);
            S.slot[item] = atomicAdd(S.gridcount + cell, 1u);
        }
        S.gridcell[item] = cell;
        if (outside) atomicOr(S.status, (unsigned)STATUS_OUTSIDE_GRID);
    }
    if (few) {
        __syncthreads();
        for (unsigned t = threadIdx.x; t < few; t += blockDim.x)
            if (tiles[t]) atomicAdd(S.scan_sums + t, tiles[t]);
        __syncthreads();  // the next entry clears them
    }
    SPH_END_WORK
}

// zero_gridcount (common.cl:392-400) for every scene of the launch, one
// block per scan tile of SPH_SCAN_TILE cells: the counts, the tile's total
// (which k_bin_count accumulates) and, once per scene, the length of the
// solid-phase list (which the gather makes).
__global__ void __launch_bounds__(SPH_SCAN_THREADS) k_zero_cells(const SceneDesc *__restrict__ scenes, BlockMap map) {
    follow_previous();
    for (unsigned vb = blockIdx.x; vb < map.num; vb += gridDim.x) {
        const BlockWork bw = map.work[vb];
        const SceneDesc &S = scenes[bw.scene];
        if (scene_idle(S)) continue;
        const unsigned end = min(bw.first + SPH_SCAN_TILE, S.num_cells);
        for (unsigned c = bw.first + threadIdx.x; c < end; c += blockDim.x) S.gridcount[c] = 0u;
        if (threadIdx.x == 0) {
            S.scan_sums[bw.first / SPH_SCAN_TILE] = 0u;
            if (bw.first == 0 && S.solid_list) S.solid_list[0] = 0u;
        }
    }
}

// count_particles_in_bins alone, for a driver that calls the reference's
// kernels one by one (gridcell already computed).
__global__ void k_count_only(const SceneDesc *__restrict__ scenes, BlockMap map) {
    SPH_FOR_WORK(map)
    if (item < active_count(S)) {
        unsigned cell = S.gridcell[item];
        if (cell >= S.num_cells) cell = S.num_cells - 1;  // host-written garbage
        S.slot[item] = atomicAdd(S.gridcount + cell, 1u);
    }
    SPH_END_WORK
}

// ---- segmented exclusive scan of gridcount -> celloffset (prefix_sum,
// common.cl:409-515, restated as a correct two-phase scan) -------------------

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned *total) {
    __shared__ unsigned warp_sums[32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned x = v;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(SPH_FULL_MASK, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    const unsigned nw = blockDim.x >> 5;
    if (warp == 0) {
        unsigned w = lane < nw ? warp_sums[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            unsigned y = __shfl_up_sync(SPH_FULL_MASK, w, o);
            if (lane >= (unsigned)o) w += y;
        }
        if (lane < nw) warp_sums[lane] = w;
    }
    __syncthreads();
    unsigned before = warp ? warp_sums[warp - 1] : 0u;
    *total = warp_sums[nw - 1];
    __syncthreads();
    return before + x - v;
}

// Phase 1: each tile's total, from coalesced loads.
__global__ void __launch_bounds__(SPH_SCAN_THREADS) k_scan_reduce(const SceneDesc *__restrict__ scenes,
                                                                  BlockMap map) {
    follow_previous();
    for (unsigned vb = blockIdx.x; vb < map.num; vb += gridDim.x) {
        const BlockWork bw = map.work[vb];
        const SceneDesc &S = scenes[bw.scene];
        if (scene_idle(S)) continue;
        const unsigned end = min(bw.first + SPH_SCAN_TILE, S.num_cells);
        unsigned sum = 0;
        for (unsigned c = bw.first + threadIdx.x; c < end; c += blockDim.x) sum += S.gridcount[c];
        unsigned total;
        block_exclusive_scan(sum, &total);
        if (threadIdx.x == 0) S.scan_sums[bw.first / SPH_SCAN_TILE] = total;
    }
}

// Phase 2: each tile adds up the totals of its scene's earlier tiles, then
// scans its cells through shared memory (coalesced loads and stores).
__global__ void __launch_bounds__(SPH_SCAN_THREADS) k_scan_down(const SceneDesc *__restrict__ scenes, BlockMap map) {
    follow_previous();
    __shared__ unsigned tile[SPH_SCAN_TILE];
    constexpr unsigned per = SPH_SCAN_TILE / SPH_SCAN_THREADS;
    for (unsigned vb = blockIdx.x; vb < map.num; vb += gridDim.x) {
        const BlockWork bw = map.work[vb];
        const SceneDesc &S = scenes[bw.scene];
        if (scene_idle(S)) continue;
        const unsigned t = bw.first / SPH_SCAN_TILE;
        unsigned part = 0;
        for (unsigned j = threadIdx.x; j < t; j += blockDim.x) part += S.scan_sums[j];
        unsigned base;
        block_exclusive_scan(part, &base);
        const unsigned end = min(bw.first + SPH_SCAN_TILE, S.num_cells);
        for (unsigned k = threadIdx.x; k < SPH_SCAN_TILE; k += blockDim.x) {
            const unsigned c = bw.first + k;
            tile[k] = c < end ? S.gridcount[c] : 0u;
        }
        __syncthreads();
        unsigned v[per], sum = 0;
#pragma unroll
        for (unsigned j = 0; j < per; ++j) {
            v[j] = tile[threadIdx.x * per + j];
            sum += v[j];
        }
        unsigned total;
        unsigned run = base + block_exclusive_scan(sum, &total);
#pragma unroll
        for (unsigned j = 0; j < per; ++j) {
            tile[threadIdx.x * per + j] = run;
            run += v[j];
        }
        __syncthreads();
        for (unsigned k = threadIdx.x; bw.first + k < end; k += blockDim.x) S.celloffset[bw.first + k] = tile[k];
        __syncthreads();  // the next tile reuses `tile`
    }
}

// insert_particles_in_bin_array (common.cl:523-529) without atomics: each
// particle and its cell go to place celloffset[cell] + its arrival slot, in
// arrival order, of the scene's unsorted list.
__global__ void k_scatter(const SceneDesc *__restrict__ scenes, BlockMap map) {
    SPH_FOR_WIDE(map)
    unsigned cell[SPH_WIDE], slot[SPH_WIDE];
#pragma unroll
    for (int j = 0; j < SPH_WIDE; ++j)
        if (W[j].valid) {
            cell[j] = W[j].S->gridcell[W[j].item];
            slot[j] = W[j].S->slot[W[j].item];
        }
    unsigned off[SPH_WIDE];
#pragma unroll
    for (int j = 0; j < SPH_WIDE; ++j) {
        off[j] = 0xffffffffu;
        if (W[j].valid && cell[j] < W[j].S->num_cells) off[j] = W[j].S->celloffset[cell[j]];
    }
#pragma unroll
    for (int j = 0; j < SPH_WIDE; ++j)
        if (off[j] != 0xffffffffu) {
            const SceneDesc &S = *W[j].S;
            const unsigned dst = off[j] + slot[j];
            if (dst < S.pnum) {
                S.unsorted[dst] = W[j].item;
                S.unsorted[S.pnum + dst] = cell[j];
            }
        }
    SPH_END_WIDE
}

// Cell-sorted copies of particle i at place k: spos = position (and velocity,
// density when asked; for solids also the rest position with the body
// number -- and in a mixed scene SPH_SOLID_PHASE_BIT for a solid-phase
// particle -- and mass/density0 in the velocity copy's w), so that the pair
// loops stream float4s.  Also what every pair pass would otherwise work out
// again in each thread, while this memory-bound work leaves issue slots to
// spare: the particle's stencil rows (srow) and the scene's constants
// (write_scene_pair).
__device__ __forceinline__ void gather_one(const SceneDesc &S, unsigned k, unsigned i, unsigned cell, int with_vel,
                                           int with_dens, int with_solid) {
    const float3 p = ld3(S.position, i);
    const bool solid = with_solid && S.spos0;
    float3 v = make_float3(0.f, 0.f, 0.f);
    if (with_vel || solid) v = ld3(S.velocity, i);
    S.spos[k] = make_float4(p.x, p.y, p.z, 0.f);
    S.srow[k] = make_uint2(cell, StencilRows(S, cell).bits);
    if (k == 0) write_scene_pair(S);
    if (with_vel || solid) S.svel[k] = make_float4(v.x, v.y, v.z, solid ? __fdiv_rn(*S.mass, S.density0[i]) : 0.f);
    if (with_dens) S.sdens[k] = S.density[i];
    if (solid) {
        // rest position, and the body number's bits in w
        const float3 p0 = ld3(S.originalpos, i);
        unsigned w = S.body_number[i];
        if (S.phase && S.phase[i]) {
            w |= SPH_SOLID_PHASE_BIT;
            // the lanes here together append their places to the list
            namespace cg = cooperative_groups;
            const cg::coalesced_group g = cg::coalesced_threads();
            unsigned at = 0;
            if (g.thread_rank() == 0) at = atomicAdd(S.solid_list, g.size());
            at = g.shfl(at, 0) + g.thread_rank();
            if (at < S.pnum) S.solid_list[1 + at] = k;
        }
        S.spos0[k] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(w));
    }
}

// A cell of m of the scene's n particles is crowded when one walk over all n
// particles' cells (0.5 ns each by a block) orders it faster than comparing
// its particles with each other (26 ns a step, m steps a thread).  So there
// are few such cells: one may start in each 257 entries, 48 in a scene.
__device__ __forceinline__ bool crowded_cell(unsigned m, unsigned n) { return m > 256u + n / 48u; }

// A crowded cell in canonical order (and, GATHER, its sorted copies), by the
// whole block: the particles' cells in index order, a run of 32 x
// SPH_CROWD_ITEMS a warp.
#define SPH_CROWD_ITEMS 16
template <bool GATHER>
__device__ __noinline__ void order_crowded_cell(const SceneDesc &S, unsigned cell, unsigned n, int with_vel,
                                                int with_solid) {
    __shared__ unsigned found[32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const unsigned off = S.celloffset[cell], cnt = S.gridcount[cell];
    const unsigned *cells = S.gridcell;
    unsigned r = off;
    for (unsigned i0 = 0; i0 < n; i0 += blockDim.x * SPH_CROWD_ITEMS) {
        const unsigned i = i0 + warp * 32u * SPH_CROWD_ITEMS + lane;
        unsigned at[SPH_CROWD_ITEMS], hit = 0;
#pragma unroll
        for (unsigned j = 0; j < SPH_CROWD_ITEMS; ++j) at[j] = cells[min(i + 32u * j, n - 1u)];
#pragma unroll
        for (unsigned j = 0; j < SPH_CROWD_ITEMS; ++j)
            hit |= (unsigned)(i + 32u * j < n && at[j] == cell) << j;
        const unsigned mine = __reduce_add_sync(SPH_FULL_MASK, __popc(hit));
        __syncthreads();
        if (lane == 0) found[warp] = mine;
        __syncthreads();
        const unsigned f = lane < warps ? found[lane] : 0u;
        unsigned to = r + __reduce_add_sync(SPH_FULL_MASK, lane < warp ? f : 0u);
        r += __reduce_add_sync(SPH_FULL_MASK, f);
        if (!mine) continue;
#pragma unroll 1
        for (unsigned j = 0; j < SPH_CROWD_ITEMS; ++j) {
            const bool in = hit >> j & 1u;
            const unsigned here = __ballot_sync(SPH_FULL_MASK, in);
            const unsigned k = to + __popc(here & ((1u << lane) - 1u));
            to += __popc(here);
            // (past the cell's end only with inconsistent host-written tables)
            if (in && k - off < cnt) {
                S.cellparticles[k] = i + 32u * j;
                if (GATHER) gather_one(S, k, i + 32u * j, cell, with_vel, 0, with_solid);
            }
        }
    }
}

// Canonical order inside each cell: ascending particle index.  One thread
// per entry of the unsorted list: its particle's place in the cell is the
// number of the cell's particles with a smaller index.  A crowded cell is
// ordered by the block that holds its first entry (a pile of 500,000 of 1M
// particles 40.5 -> 0.94 ms, of 10,000 of 100,000 300 -> 92 us, and 91 -> 92
// us without a pile, against comparisons in every cell).  GATHER: a substep,
// where nothing changes between the order and the pair passes; the
// particle's sorted copies are written here too, and a crowded cell is
// compared like any other: the pair passes test each of its particles
// against all others at ten times that cost (20,000 of 1M particles 0.6 of
// 8.4 ms), and the walk's registers cost every 1M-particle substep 7 us.  Bound: latency of the chain entry -> table ->
// the cell's entries and fields -> stores.  With the scatter 47 -> 33 us at
// 1M particles, against an order, a sort of crowded cells and a gather in
// launches of their own (four launches; a 1,000-particle substep 59 -> 55
// us).
#define SPH_CROWDED_STARTS 4  // cells above 256 that can start in 1,024 entries
template <bool GATHER>
__global__ void k_rank_cells(const SceneDesc *__restrict__ scenes, BlockMap map, int with_vel, int with_solid) {
    __shared__ unsigned starts[1 + SPH_CROWDED_STARTS];
    SPH_FOR_WORK(map)
    const unsigned n = active_count(S);
    unsigned crowded = 0xffffffffu;  // the crowded cell that starts at this entry
    if (item < n) {
        const unsigned x = S.unsorted[item], cell = S.unsorted[S.pnum + item];
        // inconsistent tables come only from host-written garbage: skip
        if (x < S.pnum && cell < S.num_cells) {
            const unsigned off = S.celloffset[cell], cnt = S.gridcount[cell];
            if (off <= item && item - off < cnt && cnt <= S.pnum - off) {
                if (!GATHER && crowded_cell(cnt, n)) {
                    if (item == off) crowded = cell;
                } else {
                    const unsigned *U = S.unsorted + off;
                    unsigned r = off;
#pragma unroll 4
                    for (unsigned a = 0; a < cnt; ++a) r += U[a] < x;
                    S.cellparticles[r] = x;
                    if (GATHER) gather_one(S, r, x, cell, with_vel, 0, with_solid);
                }
            }
        }
    }
    if (!GATHER && __syncthreads_or(crowded != 0xffffffffu)) {
        if (threadIdx.x == 0) starts[0] = 0u;
        __syncthreads();
        if (crowded != 0xffffffffu) {
            const unsigned q = atomicAdd(starts, 1u);
            if (q < SPH_CROWDED_STARTS) starts[1 + q] = crowded;
        }
        __syncthreads();
        const unsigned num = min(starts[0], (unsigned)SPH_CROWDED_STARTS);
        for (unsigned q = 0; q < num; ++q) order_crowded_cell<false>(S, starts[1 + q], n, 0, 0);
        __syncthreads();  // the next entry clears them
    }
    SPH_END_WORK
}

// The sorted copies from the fields, for pair kernels called by name.
__global__ void k_gather(const SceneDesc *__restrict__ scenes, BlockMap map, int with_vel, int with_dens,
                         int with_solid) {
    SPH_FOR_WORK(map)
    if (item < active_count(S)) {
        unsigned i = S.cellparticles[item];
        if (i >= S.pnum) i = 0;  // host-written garbage
        gather_one(S, item, i, S.gridcell[i], with_vel, with_dens, with_solid);
    }
    SPH_END_WORK
}

// ---- a small scene's grid in one launch -----------------------------------------
//
// compute_particle_bins, and with GATHER the sorted copies, of one scene by
// one thread-block cluster: the phases that are launches of their own for a
// large scene, with a cluster barrier (hardware, no spinning) between them.
// A small scene's launches are bound by latency: each starts blocks, reads
// its work entry and scene and waits for a chain or two of dependent
// accesses, and the next starts only then.
// A thread keeps its particles' cells and slots in registers, up to
// SPH_SMALL_ITEMS of them.
#define SPH_SMALL_BLOCKS 8
#define SPH_SMALL_THREADS 512
#define SPH_SMALL_ITEMS 4
#define SPH_SMALL_PARTICLES (SPH_SMALL_BLOCKS * SPH_SMALL_THREADS * SPH_SMALL_ITEMS)
#define SPH_SMALL_CELLS 65536
// Crowded cells here, where a walk takes 6.5 us at most, a thread's
// comparisons run for up to four particles one after another (17 ns a step),
// and the cluster's blocks share the cells: 4,096 of 16,384 particles in one
// cell 300 -> 27 us, all of them 1,133 -> 31 us, 20.0 -> 21.1 us without a
// pile.
__device__ __forceinline__ bool crowded_small(unsigned m, unsigned n) { return m > 256u + n / 256u; }
#define SPH_SMALL_CROWDED (SPH_SMALL_PARTICLES / 257)

template <bool GATHER>
__global__ void __launch_bounds__(SPH_SMALL_THREADS) k_grid_small(const SceneDesc *__restrict__ scenes, int with_vel,
                                                                  int with_solid) {
    follow_previous();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ unsigned totals[SPH_SMALL_BLOCKS];
    // crowded cells: their number and themselves, in block 0
    __shared__ unsigned crowded[1 + SPH_SMALL_CROWDED];
    const SceneDesc &S = scenes[0];
    if (scene_idle(S)) return;
    constexpr unsigned threads = SPH_SMALL_BLOCKS * SPH_SMALL_THREADS;
    const unsigned rank = cluster.block_rank(), me = rank * SPH_SMALL_THREADS + threadIdx.x;
    const unsigned n = active_count(S), cells = S.num_cells;
    for (unsigned c = me; c < cells; c += threads) S.gridcount[c] = 0u;
    if (me == 0 && S.solid_list) S.solid_list[0] = 0u;
    if (threadIdx.x == 0) crowded[0] = 0u;
    unsigned *const all_crowded = cluster.map_shared_rank(crowded, 0);
    unsigned cell[SPH_SMALL_ITEMS], slot[SPH_SMALL_ITEMS];
#pragma unroll
    for (int j = 0; j < SPH_SMALL_ITEMS; ++j) {
        const unsigned i = me + j * threads;
        if (i < n) {
            bool outside;
            cell[j] = cell_of(S, ld3(S.position, i), &outside);
            S.gridcell[i] = cell[j];
            if (outside) atomicOr(S.status, (unsigned)STATUS_OUTSIDE_GRID);
        }
    }
    cluster.sync();  // the counts are zero
#pragma unroll
    for (int j = 0; j < SPH_SMALL_ITEMS; ++j)
        if (me + j * threads < n) slot[j] = atomicAdd(S.gridcount + cell[j], 1u);
    cluster.sync();  // the counts are final
    // the scan: a block takes a range of cells, a thread a run of it
    const unsigned share = (cells + SPH_SMALL_BLOCKS - 1) / SPH_SMALL_BLOCKS;
    const unsigned run = (share + SPH_SMALL_THREADS - 1) / SPH_SMALL_THREADS;
    const unsigned end = min(cells, (rank + 1) * share);
    const unsigned c0 = min(end, rank * share + threadIdx.x * run), c1 = min(end, c0 + run);
    unsigned sum = 0, total;
    for (unsigned c = c0; c < c1; ++c) {
        const unsigned m = S.gridcount[c];
        sum += m;
        if (crowded_small(m, n)) {
            const unsigned q = atomicAdd(all_crowded, 1u);
            if (q < SPH_SMALL_CROWDED) all_crowded[1 + q] = c;
        }
    }
    unsigned off = block_exclusive_scan(sum, &total);
    if (threadIdx.x < SPH_SMALL_BLOCKS) cluster.map_shared_rank(totals, threadIdx.x)[rank] = total;
    cluster.sync();  // every block's total is in every block
    for (unsigned b = 0; b < rank; ++b) off += totals[b];
    for (unsigned c = c0; c < c1; ++c) {
        S.celloffset[c] = off;
        off += S.gridcount[c];
    }
    cluster.sync();  // the offsets are written
    unsigned first[SPH_SMALL_ITEMS];
#pragma unroll
    for (int j = 0; j < SPH_SMALL_ITEMS; ++j)
        if (me + j * threads < n) first[j] = S.celloffset[cell[j]];
#pragma unroll
    for (int j = 0; j < SPH_SMALL_ITEMS; ++j)
        if (me + j * threads < n) S.unsorted[first[j] + slot[j]] = me + j * threads;
    // the list's end before the last barrier: block 0 may end after it
    const unsigned num_crowded = min(all_crowded[0], (unsigned)SPH_SMALL_CROWDED);
    if (rank && threadIdx.x < num_crowded) crowded[1 + threadIdx.x] = all_crowded[1 + threadIdx.x];
    cluster.sync();  // the cells' lists are complete
#pragma unroll 1
    for (int j = 0; j < SPH_SMALL_ITEMS; ++j) {
        const unsigned i = me + j * threads;
        if (i >= n) break;
        const unsigned cnt = S.gridcount[cell[0]];
        if (!crowded_small(cnt, n)) {
            const unsigned *U = S.unsorted + first[0];
            unsigned k = first[0];
#pragma unroll 4
            for (unsigned a = 0; a < cnt; ++a) k += U[a] < i;
            S.cellparticles[k] = i;
            if (GATHER) gather_one(S, k, i, cell[0], with_vel, 0, with_solid);
        }
#pragma unroll
        for (int q = 0; q + 1 < SPH_SMALL_ITEMS; ++q) cell[q] = cell[q + 1], first[q] = first[q + 1];
    }
    // (the loop of a thread ends with its particles: together again)
    __syncthreads();
    for (unsigned q = rank; q < num_crowded; q += SPH_SMALL_BLOCKS)
        order_crowded_cell<GATHER>(S, crowded[1 + q], n, with_vel, with_solid);
}
