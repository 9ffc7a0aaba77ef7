// kernels.cu -- the sm_103a kernels of the per-substep particle pipeline
// and the host functions that enqueue them (see launch.h).
#include <stdio.h>

#include <algorithm>
#include <atomic>

#include "kernels_fluid.cuh"
#include "kernels_grid.cuh"
#include "kernels_mixed.cuh"
#include "kernels_rigid.cuh"
#include "kernels_solid.cuh"
#include "launch.h"

#define SPH_SPLIT_PARTICLES 40000ull

// Launches a kernel that begins with follow_previous() (kernels_common.cuh).
// With L.overlap its blocks may start as the kernel ahead runs out of work,
// which hides the launch and the blocks' start: a small scene's kernels called
// by name (three scenes' substeps overlapping / one alone) 20.5 / 56 -> 17.5 /
// 46.5 us at 8,000 fluid particles, 28.2 / 77.8 -> 21.3 / 57.2 us at 1,539 SVK
// particles.  Large launches lose by it (65,536 corotational particles 68 ->
// 96 us): blocks that wait hold the SMs' slots, and start on the split of
// their memory that the kernel ahead runs with, so only scenes whose grid is
// one launch overlap (sph_small_grid; 32,768 SVK particles 33 -> 37 us).
template <class... P, class... A>
static void sph_launch(const Launch &L, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = L.stream;
    cudaLaunchAttribute at[2];
    cfg.attrs = at;
    if (L.overlap) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (L.carveout) {
        at[cfg.numAttrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        at[cfg.numAttrs++].val.sharedMemCarveout = L.carveout;
    }
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

static inline unsigned grid_for(const BlockMap &m, unsigned cap) {
    unsigned g = m.num < cap ? m.num : cap;
    return g ? g : 1;
}

static void small_grid_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at, cudaStream_t stream) {
    cfg->gridDim = dim3(SPH_SMALL_BLOCKS);
    cfg->blockDim = dim3(SPH_SMALL_THREADS);
    cfg->stream = stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = SPH_SMALL_BLOCKS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}

template <bool GATHER>
static void launch_grid_small(const Launch &L, bool vel, bool solid) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2];
    small_grid_config(&cfg, at, L.stream);
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = L.overlap ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_grid_small<GATHER>, L.scenes, vel ? 1 : 0, solid ? 1 : 0);
}

// what a kernel may have without asking for more
static_assert(sizeof(DensityStage<false>) <= 48 * 1024 && sizeof(DensityStage<true>) <= 48 * 1024 &&
                  solid_smem_bytes(false, SPH_STAGED_BLOCK / 32) <= 48 * 1024 && solid_smem_bytes(true, 3) <= 48 * 1024,
              "staging buffers");

// Split against whole passes of a fluid, us a substep with three scenes' substeps
// overlapping / one scene's alone: 1,000 particles 14.2 / 40.4 -> 10.3 /
// 28.8, 8,000 15.8 / 43.1 -> 12.2 / 32.7, 25,000 20.2 / 51.3 -> 17.6 / 41.1,
// 39,304 22.1 / 53.3 -> 20.2 / 43.1, 64,000 27.2 / 55.7 -> 31.1 / 57.5: from
// there on the schedulers are full and a block's repeated set-up costs more
// than its shorter chain saves.  (Solids: corotational 4,000 31.5 / 88 ->
// 19.0 / 47, 40,960 60.9 / 127 -> 63.0 / 108; SVK 32,768 44.5 / 101 -> 38.3 /
// 80, 64,000 63.1 / 118 -> 66.7 / 105.)
bool sph_split_rows(unsigned long long particles) { return particles <= SPH_SPLIT_PARTICLES; }

// One cluster against five launches, us a substep with three scenes' substeps
// overlapping / one scene's alone: 1,000 particles 19.2 / 53.6 -> 16.5 /
// 47.6, a 4,000-particle corotational beam 38.2 / 102.4 -> 35.3 / 94.2, 8,000
// particles by name 27.2 / 80.9 -> 22.0 / 65.8.  At 32,768 it is no gain (4
// blocks: 38.0, 8: 40.5, 16: 36.7 against 37.9, and more alone), so the line
// is at the 16,384 that four particles a thread hold.  Blocks of 1024
// threads, or 16 of 512, measured within 4% of 8 of 512, which is the
// largest cluster every configuration runs.
bool sph_small_grid(unsigned pnum, unsigned num_cells) {
    if (pnum > SPH_SMALL_PARTICLES || num_cells > SPH_SMALL_CELLS) return false;
    // what the device can run, asked once per device (0: not yet, 1: no, 2: yes)
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int v = known[dev].load();
    if (!v) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[1];
        small_grid_config(&cfg, at, nullptr);
        int clusters = 0;
        v = cudaOccupancyMaxActiveClusters(&clusters, k_grid_small<true>, &cfg) == cudaSuccess && clusters > 0 ? 2 : 1;
        if (v == 1) cudaGetLastError();
        known[dev].store(v);
    }
    return v == 2;
}

cudaError_t sph_check_launch(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) sph_set_error("%s: %s", what, cudaGetErrorString(e));
    return e;
}

void sph_launch_find_bins(const Launch &L) {
    sph_launch(L, k_bin_count, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles, 0);
}

void sph_launch_zero_cells(const Launch &L) {
    sph_launch(L, k_zero_cells, grid_for(L.scan, L.grid_cap), SPH_SCAN_THREADS, 0, L.scenes, L.scan);
}

void sph_launch_count(const Launch &L) {
    sph_launch(L, k_count_only, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles);
}

void sph_launch_scan(const Launch &L, bool sums_ready) {
    if (!sums_ready)
        sph_launch(L, k_scan_reduce, grid_for(L.scan, L.grid_cap), SPH_SCAN_THREADS, 0, L.scenes, L.scan);
    sph_launch(L, k_scan_down, grid_for(L.scan, L.grid_cap), SPH_SCAN_THREADS, 0, L.scenes, L.scan);
}

void sph_launch_insert(const Launch &L, bool gather, bool vel, bool solid) {
    sph_launch(L, k_scatter, wide_grid(L.particles.num, L.grid_cap), L.block, 0, L.scenes, L.particles);
    const unsigned g = grid_for(L.particles, L.grid_cap);
    if (gather)
        sph_launch(L, k_rank_cells<true>, g, L.block, 0, L.scenes, L.particles, vel ? 1 : 0, solid ? 1 : 0);
    else
        sph_launch(L, k_rank_cells<false>, g, L.block, 0, L.scenes, L.particles, 0, 0);
}

void sph_launch_bin_count(const Launch &L) {
    sph_launch_zero_cells(L);
    sph_launch(L, k_bin_count, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles, 1);
}

void sph_launch_bins(const Launch &L) {
    if (L.small_grid) return launch_grid_small<false>(L, false, false);
    sph_launch_bin_count(L);
    sph_launch_scan(L, true);
    sph_launch_insert(L);
}

void sph_launch_bins_gather(const Launch &L, bool vel, bool solid) {
    if (L.small_grid) return launch_grid_small<true>(L, vel, solid);
    sph_launch_bin_count(L);
    sph_launch_scan(L, true);
    sph_launch_insert(L, true, vel, solid);
}

void sph_launch_gather(const Launch &L, bool vel, bool dens, bool solid) {
    sph_launch(L, k_gather, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles, vel ? 1 : 0,
                                                                          dens ? 1 : 0, solid ? 1 : 0);
}

// Blocks of a SPLIT launch: each map entry in groups of 32 particles, `per`
// of them.
static unsigned split_grid(const Launch &L, const BlockMap &m, unsigned per) {
    const unsigned long long g = (unsigned long long)m.num * per;
    return g < L.grid_cap ? (g ? (unsigned)g : 1u) : L.grid_cap;
}

#define SPH_STAGED_WARPS (SPH_STAGED_BLOCK / 32u)

template <bool PLANES>
static void launch_density(const Launch &L, const BlockMap &m, int original, int mask, int skip_solids) {
    if (L.split_rows)
        sph_launch(L, k_density<PLANES, true>, split_grid(L, m, SPH_STAGED_WARPS), dim3(32, 3),
                   sizeof(DensityStage<true>), L.scenes, m, original, mask, skip_solids, SPH_STAGED_WARPS);
    else
        sph_launch(L, k_density<PLANES, false>, grid_for(m, L.grid_cap), SPH_STAGED_BLOCK, sizeof(DensityStage<false>),
                   L.scenes, m, original, mask, skip_solids, 1u);
}

void sph_launch_density(const Launch &L, bool original, bool mask, bool skip_solids) {
    const int o = original ? 1 : 0, m = mask ? 1 : 0, sk = skip_solids ? 1 : 0;
    launch_density<false>(L, L.staged, o, m, sk);
    if (!L.no_symmetry_planes) launch_density<true>(L, L.staged, o, m, 0);
}

void sph_launch_density_fused(const Launch &L, const Launch *fluids) {
    if (fluids && fluids->staged.num) launch_density<false>(L, fluids->staged, 0, 1, 1);
    if (!L.no_symmetry_planes) launch_density<true>(L, L.staged, 0, 1, 0);
}

template <bool MIXED>
static void launch_forces_masked(const Launch &L, int step) {
    const BlockMap &m = L.pair_particles;
    const unsigned per = L.pair_block / 32u;
    if (L.split_rows)
        sph_launch(L, k_forces_fluids_masked<MIXED, true>, split_grid(L, m, per), dim3(32, 3), 0, L.scenes, m, step, per);
    else
        sph_launch(L, k_forces_fluids_masked<MIXED>, grid_for(m, L.grid_cap), L.pair_block, 0, L.scenes, m, step, 1u);
}

void sph_launch_forces_fluids(const Launch &L, bool fuse_step, bool masked) {
    const unsigned g = grid_for(L.pair_particles, L.grid_cap);
    const int step = fuse_step ? 1 : 0;
    if (masked) {
        if (!L.all_mixed) launch_forces_masked<false>(L, step);
        if (L.has_mixed) launch_forces_masked<true>(L, step);
    } else {
        if (!L.all_mixed) sph_launch(L, k_forces_fluids<false>, g, L.pair_block, 0, L.scenes, L.pair_particles, step);
        if (L.has_mixed) sph_launch(L, k_forces_fluids<true>, g, L.pair_block, 0, L.scenes, L.pair_particles, step);
    }
}

void sph_launch_original_density_mixed(const Launch &L) {
    sph_launch(L, k_original_density_mixed, grid_for(L.pair_particles, L.grid_cap), L.pair_block, 0, L.scenes, L.pair_particles);
}

// Blocks over the solid-phase list, whose length only the device knows: a
// fixed number at most, which loop over what is left of it.
#define SPH_LIST_BLOCK 128u
static unsigned solid_grid(const Launch &L) {
    const unsigned most = (L.particles.num * L.block + SPH_LIST_BLOCK - 1u) / SPH_LIST_BLOCK;
    const unsigned cap = std::min(L.grid_cap, 152u * 16u);
    return most < cap ? (most ? most : 1u) : cap;
}

void sph_launch_deformations_mixed(const Launch &L, bool masked, bool with_stress) {
    sph_launch(L, k_deformations_mixed, solid_grid(L), SPH_LIST_BLOCK, 0, L.scenes, masked ? 1 : 0,
               with_stress ? 1 : 0);
}

void sph_launch_forces_solids_mixed(const Launch &L, bool sorted) {
    if (sorted) sph_launch(L, k_forces_solids_mixed<true>, solid_grid(L), SPH_LIST_BLOCK, 0, L.scenes);
    else sph_launch(L, k_forces_solids_mixed<false>, solid_grid(L), SPH_LIST_BLOCK, 0, L.scenes);
}

void sph_launch_step_forward(const Launch &L, bool planes_only) {
    sph_launch(L, k_step_forward, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles,
                                                                                planes_only ? 1 : 0);
}

void sph_launch_plane_constraints(const Launch &L) {
    sph_launch(L, k_plane_constraints, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles);
}

void sph_launch_init_original_position(const Launch &L) {
    sph_launch(L, k_init_original_position, grid_for(L.particles, L.grid_cap), L.block, 0, L.scenes, L.particles);
}

void sph_launch_rotations_and_strains(const Launch &L, bool with_density, bool with_stress) {
    const BlockMap &m = L.staged;
    const unsigned w = SPH_STAGED_WARPS;
    const int d = with_density ? 1 : 0, st = with_density && with_stress ? 1 : 0;
    if (L.split_rows)
        sph_launch(L, k_rotations_and_strains<true>, split_grid(L, m, w), dim3(32, 3), solid_smem_bytes(true, 3),
                   L.scenes, m, d, st, w);
    else
        sph_launch(L, k_rotations_and_strains<false>, grid_for(m, L.grid_cap), dim3(32, w), solid_smem_bytes(false, w),
                   L.scenes, m, d, st, 1u);
    if (!L.no_symmetry_planes)
        sph_launch(L, k_rotations_and_strains_planes, grid_for(L.pair_particles, L.grid_cap), L.pair_block, 0, L.scenes,
                   L.pair_particles);
}

void sph_launch_stresses(const Launch &L, bool corot, bool sorted, bool planes_only) {
    const unsigned g = grid_for(L.particles, L.grid_cap);
    if (sorted) {
        if (corot) sph_launch(L, k_stresses_sorted<true>, g, L.block, 0, L.scenes, L.particles, planes_only ? 1 : 0);
        else sph_launch(L, k_stresses_sorted<false>, g, L.block, 0, L.scenes, L.particles, planes_only ? 1 : 0);
    } else {
        if (corot) sph_launch(L, k_stresses_corot, g, L.block, 0, L.scenes, L.particles);
        else sph_launch(L, k_stresses_svk, g, L.block, 0, L.scenes, L.particles);
    }
}

void sph_launch_deformations(const Launch &L, bool with_density, bool with_stress) {
    const BlockMap &m = L.staged;
    const unsigned w = SPH_STAGED_WARPS;
    const int d = with_density ? 1 : 0, st = with_density && with_stress ? 1 : 0;
    if (L.split_rows)
        sph_launch(L, k_deformations<true>, split_grid(L, m, w), dim3(32, 3), solid_smem_bytes(true, 3), L.scenes, m, d,
                   st, w);
    else
        sph_launch(L, k_deformations<false>, grid_for(m, L.grid_cap), dim3(32, w), solid_smem_bytes(false, w), L.scenes,
                   m, d, st, 1u);
    if (!L.no_symmetry_planes)
        sph_launch(L, k_deformations_planes, grid_for(L.pair_particles, L.grid_cap), L.pair_block, 0, L.scenes,
                   L.pair_particles);
}

template <bool COROT>
static void launch_forces_solids(const Launch &L, bool masked, int step) {
    const BlockMap &m = L.staged;
    const unsigned w = SPH_STAGED_WARPS, gp = split_grid(L, m, w), g = grid_for(m, L.grid_cap);
    const dim3 part(32, 3), whole(32, w);
    const size_t sp = solid_force_smem_bytes(3), sw = solid_force_smem_bytes(w);
    if (L.split_rows) {
        if (masked) sph_launch(L, k_forces_solids<COROT, true, true>, gp, part, sp, L.scenes, m, step, w);
        else sph_launch(L, k_forces_solids<COROT, false, true>, gp, part, sp, L.scenes, m, 0, w);
    } else {
        if (masked) sph_launch(L, k_forces_solids<COROT, true, false>, g, whole, sw, L.scenes, m, step, 1u);
        else sph_launch(L, k_forces_solids<COROT, false, false>, g, whole, sw, L.scenes, m, 0, 1u);
    }
    if (!L.no_symmetry_planes)
        sph_launch(L, k_forces_solids_planes<COROT>, grid_for(L.pair_particles, L.grid_cap), L.pair_block, 0, L.scenes,
                   L.pair_particles);
}

void sph_launch_forces_solids(const Launch &L, bool corot, bool masked, bool fuse_step) {
    const int step = masked && fuse_step ? 1 : 0;
    if (corot) launch_forces_solids<true>(L, masked, step);
    else launch_forces_solids<false>(L, masked, step);
}

void sph_launch_solid_passes(const Launch &L, bool corot, PhaseMark mark, void *ctx) {
    auto phase = [&](const char *name) {
        if (mark) mark(ctx, name);
    };
    const bool planes = !L.no_symmetry_planes;
    phase(corot ? "rotations_and_strains" : "deformations");
    if (corot) sph_launch_rotations_and_strains(L, true, true);
    else sph_launch_deformations(L, true, true);
    if (planes) {
        phase("stresses");
        sph_launch_stresses(L, corot, true, true);
    }
    phase("forces_solids+step");
    sph_launch_forces_solids(L, corot, true, true);
    if (planes) {
        phase("step_forward");
        sph_launch_step_forward(L, true);
    }
}

void sph_launch_set_body_position(const Launch &L, unsigned body, const float pos[3]) {
    float3 p = make_float3(pos[0], pos[1], pos[2]);
    k_set_body_position<<<grid_for(L.particles, L.grid_cap), L.block, 0, L.stream>>>(L.scenes, L.particles, body, p);
    k_store_body_vec<<<1, 32, 0, L.stream>>>(L.scenes, 0, body, p);
}

void sph_launch_set_body_rotation(const Launch &L, unsigned body, const float euler[3]) {
    float3 e = make_float3(euler[0], euler[1], euler[2]);
    k_set_body_rotation<<<grid_for(L.particles, L.grid_cap), L.block, 0, L.stream>>>(L.scenes, L.particles, body);
    k_store_body_vec<<<1, 32, 0, L.stream>>>(L.scenes, 1, body, e);
}

void sph_launch_populate_cuboid(const Launch &L, const float c1[3], const float c2[3], const unsigned size[3]) {
    dim3 block(8, 8, 4);
    dim3 grid((size[0] + 7) / 8, (size[1] + 7) / 8, (size[2] + 3) / 4);
    k_populate_cuboid<<<grid, block, 0, L.stream>>>(L.scenes, make_float3(c1[0], c1[1], c1[2]),
                                                    make_float3(c2[0], c2[1], c2[2]), make_uint3(size[0], size[1], size[2]));
}

void sph_launch_rotate_particles(const Launch &L, float ax, float ay, float az) {
    k_rotate_particles<<<grid_for(L.particles, L.grid_cap), L.block, 0, L.stream>>>(L.scenes, L.particles, ax, ay, az);
}

// The substep recipes a reference driver issues by name:
//   fluids: compute_particle_bins, compute_density, compute_forces_fluids,
//           step_forward (src/mex/simstep_fluid.c:18-23)
//   corotational solid: bins, compute_density,
//           compute_rotations_and_strains, compute_stresses,
//           compute_forces_solids, step_forward (scripts/sph/systems.py:194-204)
//   SVK solid: the same with compute_deformations (systems.py:225-235)
// Positions do not move between the bins and the integrator, so the sorted
// copies are gathered once, the force pass walks the candidate masks the
// density pass recorded, and for fluids the integrator is fused into the
// force pass.
void sph_launch_substep(const Launch &L, SphMaterial mat, PhaseMark mark, void *ctx) {
    auto phase = [&](const char *name) {
        if (mark) mark(ctx, name);
    };
    const bool vel = mat == MAT_FLUID || mat == MAT_MIXED, solid = mat != MAT_FLUID;
    if (L.small_grid) {
        phase("grid");
        sph_launch_bins_gather(L, vel, solid);
    } else {
        phase("bin_count");
        sph_launch_bin_count(L);
        phase("scan");
        sph_launch_scan(L, true);
        phase("insert+gather");
        sph_launch_insert(L, true, vel, solid);
    }
    if (mat == MAT_MIXED) {
        // fluid and solid particles in one scene (extension): the fluid
        // recipe, with the solids' elastic passes before the force pass,
        // which adds the fluid-solid pair terms and steps every particle
        phase("density");
        sph_launch_density(L, false, true, false);
        phase("deformations (solid phase)");
        sph_launch_deformations_mixed(L, true, true);
        phase("forces_solids (solid phase)");
        sph_launch_forces_solids_mixed(L, true);
        phase("forces_fluids+step");
        sph_launch_forces_fluids(L, true, true);
        if (L.num_rigid) {
            phase("rigid_bodies");
            sph_launch_rigid(L);
        }
        phase(nullptr);
        return;
    }
    if (mat == MAT_FLUID || !L.no_symmetry_planes) {
        // a plane-free solid's density is summed by its first solid pass
        phase("density");
        sph_launch_density(L, false, mat == MAT_FLUID, mat != MAT_FLUID);
    }
    if (mat == MAT_FLUID) {
        phase("forces_fluids+step");
        sph_launch_forces_fluids(L, true, true);
        if (L.num_rigid) {
            phase("rigid_bodies");
            sph_launch_rigid(L);
        }
        phase(nullptr);
        return;
    }
    sph_launch_solid_passes(L, mat == MAT_COROT, mark, ctx);
    if (L.num_rigid) {
        phase("rigid_bodies");
        sph_launch_rigid(L);
    }
    phase(nullptr);
}

void sph_launch_rigid(const Launch &L) {
    if (!L.num_rigid || !L.rigid) return;
    const dim3 grid(SPH_RIGID_BLOCKS, L.num_rigid);
    k_rigid_reduce<<<grid, SPH_RIGID_THREADS, 0, L.stream>>>(L.scenes, L.rigid);
    k_rigid_integrate<<<L.num_rigid, 32, 0, L.stream>>>(L.scenes, L.rigid, L.num_rigid);
    k_rigid_scatter<<<grid, SPH_RIGID_THREADS, 0, L.stream>>>(L.scenes, L.rigid);
}

void sph_launch_rigid_reset(const Launch &L) {
    const unsigned g = L.num_scenes < 1024 ? L.num_scenes : 1024;
    k_rigid_reset<<<g ? g : 1, 64, 0, L.stream>>>(L.scenes, L.num_scenes);
}

// End of a batched substep: each scene with a finite quota left uses one.
__global__ void k_count_down(const SceneDesc *__restrict__ scenes, unsigned num_scenes) {
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < num_scenes; s += gridDim.x * blockDim.x) {
        unsigned *q = scenes[s].steps_left;
        if (!q) continue;
        const unsigned v = *q;
        if (v != 0u && v != SPH_STEPS_UNLIMITED) *q = v - 1u;
    }
}

__global__ void k_set_steps(unsigned *steps_left, unsigned steps) { *steps_left = steps; }

void sph_launch_count_down(const Launch &L) {
    unsigned g = (L.num_scenes + 255) / 256;
    k_count_down<<<g ? g : 1, 256, 0, L.stream>>>(L.scenes, L.num_scenes);
}

void sph_launch_set_steps(unsigned *steps_left, unsigned steps, cudaStream_t stream) {
    k_set_steps<<<1, 1, 0, stream>>>(steps_left, steps);
}

// Recording: the copy reads the counters, the tick (one thread, after the
// copy in stream order) advances them.
__global__ void k_record_copy(RecordPlan p) {
    const unsigned long long step = p.counters[0];
    if ((step + 1) % p.every) return;
    unsigned *dst = p.ring + (size_t)(p.counters[1] % p.frames) * p.frame_words;
    size_t base = 0;
    for (unsigned r = 0; r < p.num_ranges; ++r) {
        const uint2 rg = p.ranges[r];
        for (size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x; w < rg.y; w += (size_t)gridDim.x * blockDim.x)
            dst[base + w] = p.blob[rg.x + w];
        base += rg.y;
    }
}

__global__ void k_record_tick(RecordPlan p) {
    const unsigned long long step = p.counters[0] + 1;
    p.counters[0] = step;
    if (step % p.every == 0) p.counters[1] += 1;
}

void sph_launch_record(const RecordPlan &p, cudaStream_t stream) {
    unsigned g = (p.frame_words + 255) / 256;
    if (g > 1024) g = 1024;
    k_record_copy<<<g ? g : 1, 256, 0, stream>>>(p);
    k_record_tick<<<1, 1, 0, stream>>>(p);
}

// Segment copy by `stride` threads, of which this is thread t0: in 16-byte
// words where both ends allow, else 4-byte words, else bytes.
__device__ __forceinline__ void copy_segment(const CopySeg &g, size_t t0, size_t stride) {
    const uintptr_t align = (uintptr_t)g.src | (uintptr_t)g.dst;
    size_t done = 0;
    if ((((uintptr_t)g.src ^ (uintptr_t)g.dst) & 15u) == 0) {
        // source and destination at the same offset within 16 bytes: the
        // bytes up to the first 16-byte boundary, 16-byte words, the tail
        size_t head = (16u - ((uintptr_t)g.src & 15u)) & 15u;
        if (head > g.bytes) head = g.bytes;
        for (size_t c = t0; c < head; c += stride) g.dst[c] = g.src[c];
        const size_t n = (g.bytes - head) / 16;
        const uint4 *s = reinterpret_cast<const uint4 *>(g.src + head);
        uint4 *d = reinterpret_cast<uint4 *>(g.dst + head);
#pragma unroll 4
        for (size_t w = t0; w < n; w += stride) d[w] = s[w];
        done = head + n * 16;
    } else if (align % 4 == 0) {
        const size_t n = g.bytes / 4;
        const unsigned *s = reinterpret_cast<const unsigned *>(g.src);
        unsigned *d = reinterpret_cast<unsigned *>(g.dst);
        for (size_t w = t0; w < n; w += stride) d[w] = s[w];
        done = n * 4;
    }
    for (size_t c = done + t0; c < g.bytes; c += stride) g.dst[c] = g.src[c];
}

// Block row y copies segment y.
__global__ void k_copy_segments(const CopySeg *__restrict__ segs, unsigned first) {
    copy_segment(segs[first + blockIdx.y], (size_t)blockIdx.x * blockDim.x + threadIdx.x,
                 (size_t)gridDim.x * blockDim.x);
}
__global__ void k_copy_inline(InlineSegs segs) {
    if (blockIdx.y < SPH_INLINE_SEGS)
        copy_segment(segs.seg[blockIdx.y], (size_t)blockIdx.x * blockDim.x + threadIdx.x,
                     (size_t)gridDim.x * blockDim.x);
}

void sph_launch_copy_inline(const InlineSegs &segs, cudaStream_t stream) {
    // a block per 16 KB: four 16-byte words a thread
    unsigned long long top = 1;
    for (unsigned q = 0; q < segs.count; ++q) top = segs.seg[q].bytes > top ? segs.seg[q].bytes : top;
    k_copy_inline<<<dim3((unsigned)((top + 16383) / 16384), segs.count), 256, 0, stream>>>(segs);
}

void sph_launch_copy_segments(const CopySeg *segs, unsigned count, unsigned long long max_bytes,
                              cudaStream_t stream) {
    // 64 KB per block (sixteen 16-byte words per thread, four in flight):
    // a segment's blocks share gridDim.x, so the large segments' count
    // sets it and the small segments' extra blocks exit at once
    const unsigned long long per_block = 256ull * 16 * 16;
    unsigned gx = (unsigned)((max_bytes + per_block - 1) / per_block);
    gx = gx < 1 ? 1 : gx > 256 ? 256 : gx;
    for (unsigned first = 0; first < count; first += 65535u) {
        const unsigned gy = count - first < 65535u ? count - first : 65535u;
        k_copy_segments<<<dim3(gx, gy), 256, 0, stream>>>(segs, first);
    }
}

// splitmix64 (Steele, Lea and Flood, 2014; the finaliser of Vigna's
// xorshift generators): a 64-bit counter-based mix.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    unsigned long long z = x + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_lattice(SceneDesc S, LatticeGen g, unsigned count) {
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < count; p += gridDim.x * blockDim.x) {
        const unsigned q[3] = {p % g.nx, p / g.nx % g.ny, p / (g.nx * g.ny)};
        for (int a = 0; a < 3; ++a) {
            const unsigned long long z = splitmix64(g.seed * 0x100000000ull + 3ull * p + (unsigned long long)a);
            const double u = (double)(z >> 11) * 0x1.0p-53;
            const double off = __dmul_rn(g.jitter, __dsub_rn(__dmul_rn(2.0, u), 1.0));
            const double x = __dadd_rn(__dadd_rn(__dmul_rn((double)q[a], g.spacing), g.origin[a]), off);
            S.position[3 * (size_t)p + a] = __double2float_rn(x);
        }
        if (S.body_number)
            const_cast<unsigned *>(S.body_number)[p] = p < g.clamp_layers * g.nx * g.ny ? 1u : 0u;
        if (g.identity_rotation && S.rotation)
            for (int c = 0; c < 9; ++c) S.rotation[9 * (size_t)p + c] = (c % 4 == 0) ? 1.f : 0.f;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *const_cast<unsigned *>(S.n) = count;
}

void sph_launch_lattice(const SceneDesc &d, const LatticeGen &g, cudaStream_t stream) {
    const unsigned count = g.nx * g.ny * g.nz;
    unsigned grid = (count + 255) / 256;
    grid = grid < 1 ? 1 : grid > 4096 ? 4096 : grid;
    k_lattice<<<grid, 256, 0, stream>>>(d, g, count);
}
