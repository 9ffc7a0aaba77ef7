// kernels_fluid.cuh -- per-particle pair passes for density and WCSPH
// forces, the symplectic-Euler integrator and plane constraints (sm_103a).
//
// Pair passes run one thread per cell-sorted particle k (i =
// cellparticles[k]) so a warp covers a few neighbouring cells and shares
// their neighbour rows in L1; neighbours are streamed from the float4
// copies built by gather_one.  Sums are FP32, blocked per stencil row: a
// row's terms added in order, the nine row sums with Kahan compensation.
#pragma once

#include "kernels_common.cuh"
#include "kernels_rigid.cuh"


// compute_density (common.cl:610-690) and compute_original_density
// (solids.cl:99-170): rho_i = m * sum_j W_poly6(|x_j - x_i|), j = i
// included, plus mirror images across the symmetry planes.  With
// `original` the result goes to density0 and no neighbour count is kept.
//
// The stencil is walked as 9 rows (dz outer, dy inner, as the reference's
// z, y, x loops): cells x-1..x+1 of one (z, y) row are one contiguous range
// of the cell-sorted order.  A block stages the three rows of a z plane in
// shared memory at a time: per row, the range its particles' rows lie in
// (from its first and last particle's cell; the block's particles are
// consecutive in the sort) goes into one array per coordinate, by
// asynchronous copies that run while the plane before is worked on.
// A lane then tests four consecutive candidates from three 16-byte loads
// (lanes of one cell read the same address, a broadcast; the cells' ranges
// start 8 floats apart, in different banks).
// A row is taken in two steps:
//   - near_bits tests 32 candidates without a branch, two per packed
//     FP32x2 instruction, and collects the signs of r^2 - bound with one
//     funnel shift per candidate.  Its bound lies 2^-20 above the exact one
//     (and the smallest normal float, for radii whose squares underflow),
//     more than the fused sum can differ from the rounded one, so no
//     neighbour is missed;
//   - the set bits (about 34 of 216 candidates) are walked in candidate
//     order with the exact arithmetic of a direct walk: each adds its
//     density term, and the few that are not within h lose their bit.
// Values, order and arithmetic of the sums are those of a direct walk,
// which a row takes whose range does not lie in the staged one (inconsistent
// host-written tables), or whose particle lies within h of a symmetry plane.
// A plane whose ranges are wider than the buffer is staged row by row, and a
// row that is wider in pieces, whose candidates are tested as they come.
// Against a direct walk of every row of such a plane (a few blocks, which
// end last): 27 particles a cell, 8,000 particles 50 -> 24 us and 97,336
// 117 -> 64 us, 216 a cell 281 -> 76 and 1,001 -> 457 us, 10,000 of 100,000
// particles in one cell 1,437 -> 389 us.
// The sum is blocked: each stencil row's terms are added in candidate
// order, and the nine row sums with Kahan compensation (one compensated
// add per row instead of per neighbour).
//
// With `want_mask` (fused fluid substeps, where positions cannot change
// before the force pass) each fluid particle also records, per row, which
// candidates lie within h (kernels_common.cuh, candidate masks).  The stores
// of one row are one coalesced store per warp.  num_neighbours is the number
// of set bits, less the few candidates at exactly h.
// A plane's buffer of 896 candidates holds the ranges of 128 particles:
// about 440 in a lattice of 8 per cell, 600 in one of 27.
//
// SPLIT (small launches): a block is three warps over the same 32 particles,
// one per z plane, each with a buffer of its own; the nine row sums meet in
// shared memory and are added in the same order, so the bits are the same.
// Where there are fewer warps than the schedulers can hold, a warp's own
// chain of nine rows is the time of the pass.
//
// Bound: issue slots, 4,310 warp instructions per 32 particles at 1M (a third
// each for the walk, near_bits, and row bounds, staging and masks) against
// 5,001 for testing each candidate exactly as it comes, from rows staged per
// warp: 160 -> 144 us at 1M particles when it was taken (ncu; 148 with what
// takes denser planes), 1M-particle substep 384 -> 373 us.
//
// The buffers (two in turn, or one per plane), and each row's staged range
// (first index, padded length).
template <bool SPLIT>
struct DensityStage {
    static constexpr unsigned size = SPLIT ? 256 : 896;
    float xyz[SPLIT ? 3 : 2][3 * size];
    uint2 range[9];
    float rows[SPLIT ? 9 : 1][32];      // row sums
    unsigned counts[SPLIT ? 3 : 1][32];
    unsigned cands[SPLIT ? 3 : 1][32];  // candidates, or SPH_NCAND_SCAN
};

// Asynchronous 4-byte copy from global to shared memory.
__device__ __forceinline__ void copy_word_async(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// p = (rho - rho0) stiffness (fluids.cl:33-36), rounded as written.
__device__ __forceinline__ float fluid_pressure(float rho, float rho0, float stiff) {
    return __fmul_rn(__fsub_rn(rho, rho0), stiff);
}

template <bool PLANES, bool MASK, bool SPLIT>
__device__ __forceinline__ void density_block(const SceneDesc &S, unsigned n, unsigned first,
                                              DensityStage<SPLIT> &stage, int original) {
    constexpr unsigned STAGE = DensityStage<SPLIT>::size;
    const unsigned flat = SPLIT ? threadIdx.y * 32u + threadIdx.x : threadIdx.x;
    const unsigned k = first + threadIdx.x;
    const bool active = k < n;
    const ScenePair B = scene_pair(S);
    const float h = B.h, h2 = B.h2;
    const float4 *spos = S.spos;
    const unsigned pnum = S.pnum;
    const StencilRows rows(S, active ? S.srow[k] : make_uint2(0u, 0u));
    if (flat < 9u) {
        // row r's ranges of the block's particles lie between its first
        // particle's cell x-1 and its last one's x+1 (by cell index, so past
        // an end of the grid's row they take in neighbouring rows too)
        const int r = flat;
        const long long d = (long long)(r / 3 - 1) * rows.layer + (r % 3 - 1) * (long long)rows.R0;
        const long long c0 = (long long)S.srow[first].x + d - 1,
                        c1 = (long long)S.srow[min(first + blockDim.x, n) - 1u].x + d + 1;
        const long long top = (long long)S.num_cells - 1;
        unsigned b = 0, e = 0;
        if (c1 >= 0 && c0 <= top) {
            const unsigned x0 = (unsigned)(c0 < 0 ? 0 : c0), x1 = (unsigned)(c1 > top ? top : c1);
            b = S.celloffset[x0];
            e = min(S.celloffset[x1] + S.gridcount[x1], pnum);
        }
        const unsigned a = b & ~3u;
        stage.range[r] = make_uint2(a, b < e ? (e - a + 3u) & ~3u : 0u);
    }
    const float3 ipos = active ? xyz(spos[k]) : make_float3(0.f, 0.f, 0.f);
    const NegPoint nip = neg_point(ipos);
    const float2 nx = make_float2(-ipos.x, -ipos.x), ny = make_float2(-ipos.y, -ipos.y),
                 nz = make_float2(-ipos.z, -ipos.z);
    const float wide = __fmaf_rn(B.le, 1.f + 0x1p-20f, 0x1p-126f);
    const float2 nb = make_float2(-wide, -wide);
    Planes P;
    if (PLANES) {
        load_planes(S, ipos, h, P);
        if (!active) P.imask = 0;
    }
    Kahan rho;
    unsigned count = 0, total = 0;
    bool overflow = false;
    __syncthreads();
    // where plane dz's rows start in its buffer; past STAGE: not staged
    auto plane_at = [&](int dz, unsigned (&at)[4], unsigned (&ua)[3]) {
        at[0] = 0;
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const uint2 g = stage.range[3 * dz + dy];
            ua[dy] = g.x;
            at[dy + 1] = at[dy] + min(g.y, STAGE + 4u);  // (no sum overflows)
        }
    };
    auto stage_one = [&](float *to, unsigned kk) {
        // up to three past the range: any value (capacity bounds it)
        const float *p = reinterpret_cast<const float *>(spos + min(kk, pnum - 1u));
        copy_word_async(to, p);
        copy_word_async(to + STAGE, p + 1);
        copy_word_async(to + 2 * STAGE, p + 2);
    };
    auto stage_plane = [&](int dz) {
        unsigned at[4], ua[3];
        plane_at(dz, at, ua);
        if (at[3] > STAGE) return;
        float *to = stage.xyz[SPLIT ? dz : dz & 1];
#pragma unroll 1
        for (unsigned t = threadIdx.x; t < at[3]; t += blockDim.x)
            stage_one(to + t, t + (t < at[1] ? ua[0] : t < at[2] ? ua[1] - at[1] : ua[2] - at[2]));
    };
    // the threads that share a buffer together: a split launch's warps have
    // one each, and may differ in whether their planes fit
    auto sync = [] {
        if (SPLIT) __syncwarp();
        else __syncthreads();
    };
    auto stage_row = [&](float *to, unsigned from, unsigned num) {
        sync();  // what the buffer held is done with
#pragma unroll 1
        for (unsigned t = threadIdx.x; t < num; t += blockDim.x) stage_one(to + t, from + t);
        copies_wait();
        sync();
    };
    // every candidate of [from, from + len) from the copies
    auto direct = [&](unsigned from, unsigned len, unsigned &lo, unsigned &hi, float &rowsum) {
#pragma unroll 1
        for (unsigned t = 0; t < len; ++t) {
            const float4 j4 = spos[from + t];
            const float r2 = dist2(j4, nip);
            if (r2 <= B.le) {
                const float d = fmaxf(h2 - r2, 0.f);
                rowsum = __fadd_rn(rowsum, d * d * d);
                count += r2 <= B.lt;
                if (MASK && t < 32u) lo |= 0x80000000u >> t;
                if (MASK && t >= 32u && t < 64u) hi |= 0x80000000u >> (t - 32u);
            }
            if (PLANES && P.imask) {
                const float3 jpos = xyz(j4);
                const unsigned jm = plane_jmask(P, jpos, h);
                // subsets of jm in increasing order: the reference's
                // plane_bits order restricted to the subsets it keeps
                for (unsigned sb = (0u - jm) & jm; sb; sb = (sb - jm) & jm) {
                    float3 ref = jpos;
                    for (unsigned s2 = 0; s2 < P.count; ++s2)
                        if (sb & (1u << s2)) ref = reflect3(ref, P.p[s2], P.n[s2]);
                    const float m2 = norm2(sub3(ref, ipos));
                    if (m2 <= B.lt) {
                        const float d = fmaxf(h2 - m2, 0.f);
                        rowsum = __fadd_rn(rowsum, d * d * d);
                        ++count;
                    }
                }
            }
        }
    };
    // a row whose range is wider than the buffer, in pieces, every candidate
    // as it comes: without a branch, since a term beyond h is zero
    auto wide_row = [&](int r, unsigned b, unsigned e, float *buf, unsigned &lo, unsigned &hi, float &rowsum) {
        const uint2 g = stage.range[r];
        const bool staged = b - g.x < g.y && e - g.x <= g.y && !(PLANES && P.imask);
#pragma unroll 1
        for (unsigned p = g.x; p - g.x < g.y; p += STAGE) {
            stage_row(buf, p, min(g.x + g.y - p, STAGE));
            const unsigned le = staged ? max(p, min(e, p + STAGE)) : p, lb = min(le, max(b, p));
            auto visit = [&](unsigned t) {
                const float r2 = dist2(make_float4(buf[t], buf[STAGE + t], buf[2 * STAGE + t], 0.f), nip);
                const float d = fmaxf(h2 - r2, 0.f);
                rowsum = __fadd_rn(rowsum, d * d * d);
                count += r2 <= B.lt;
                return r2 <= B.le;
            };
            // (a row longer than 64, which the later passes scan, has no bits
            // past 64)
            const unsigned lm = MASK ? min(le, max(lb, b + 64u)) : lb;
#pragma unroll 1
            for (unsigned kk = lb; kk < lm; ++kk) {
                const unsigned at = kk - b;
                if (!visit(kk - p)) continue;
                if (at < 32u) lo |= 0x80000000u >> at;
                else hi |= 0x80000000u >> (at - 32u);
            }
#pragma unroll 4
            for (unsigned t = lm - p; t < le - p; ++t) visit(t);
        }
        if (!staged) direct(b, e - b, lo, hi, rowsum);
    };
    // the exact walk over the staged candidates of a chunk's bits (candidate
    // src + t at bit 31 - t), in order; returns the bits that are within h
    auto walk = [&](unsigned m, const float *__restrict__ src, float &rowsum) {
        unsigned hit = m;
#pragma unroll 1
        while (m) {
            const unsigned t = take_first(m);
            const float r2 = dist2(make_float4(src[t], src[STAGE + t], src[2 * STAGE + t], 0.f), nip);
            // beyond h by a rounding: h2 - r2 <= 0 adds nothing
            const float d = fmaxf(h2 - r2, 0.f);
            rowsum = __fadd_rn(rowsum, d * d * d);
            if (!(r2 <= B.lt)) {
                // at h, or beyond by a rounding: not counted
                --count;
                if (!(r2 <= B.le)) {
                    hit ^= 0x80000000u >> t;
                    ++count;
                }
            }
        }
        count += __popc(hit);
        return hit;
    };
    const int dz0 = SPLIT ? (int)threadIdx.y : 0, dz1 = SPLIT ? dz0 + 1 : 3;
    stage_plane(dz0);
#pragma unroll 1
    for (int dz = dz0; dz < dz1; ++dz) {
        unsigned b[3], e[3], at[4], ua[3];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            b[dy] = e[dy] = 0;
            if (active) rows.row(S, 3 * dz + dy, &b[dy], &e[dy]);
        }
        plane_at(dz, at, ua);
        const bool fits = at[3] <= STAGE;
        float *buf = stage.xyz[SPLIT ? dz : dz & 1];
        copies_wait();
        __syncthreads();  // this plane is staged, and the other buffer is free
        if (dz + 1 < dz1) stage_plane(dz + 1);
        // the plane's rows in turn: [0] of each array, which then moves up
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            const unsigned len = e[0] - b[0];
            // the row's mask in two words
            unsigned lo = 0, hi = 0;
            // the row's density terms in candidate order; the row sums are
            // added with Kahan compensation (blocked summation)
            float rowsum = 0.f;
            const unsigned range = at[1] - at[0];
            if (!fits) {
                // a plane that does not fit is staged row by row
                if (range > STAGE) wide_row(3 * dz + dy, b[0], e[0], buf, lo, hi, rowsum);
                else stage_row(buf, ua[0], range);
            }
            // (an empty row takes the direct walk, of no candidate)
            if (range > STAGE) {
                // done
            } else if (b[0] - ua[0] < range && e[0] - ua[0] <= range && !(PLANES && P.imask)) {
                // chunks of 32 candidates, from the row's start rounded down
                // to a multiple of four: candidate c0 + t of the rounded row
                // is bit 31 - t, and the first `o` belong to the cells before
                const unsigned o = b[0] & 3u, tot = len ? o + len : 0u;
                const float *src = buf + (fits ? at[0] : 0u) + (b[0] - o - ua[0]);
                if (tot) {
                    unsigned m = near_bits<STAGE>(src, min((tot + 3u) >> 2, 8u), nx, ny, nz, nb) & (0xffffffffu >> o);
                    if (tot < 32u) m &= ~(0xffffffffu >> tot);
                    m = walk(m, src, rowsum);
                    lo = m << o;
                }
#pragma unroll 1
                for (unsigned c0 = 32; c0 < tot; c0 += 32) {
                    const unsigned rem = tot - c0;
                    unsigned m = near_bits<STAGE>(src + c0, min((rem + 3u) >> 2, 8u), nx, ny, nz, nb);
                    if (rem < 32u) m &= ~(0xffffffffu >> rem);
                    m = walk(m, src + c0, rowsum);
                    // candidate b + t at bit 31 - t of the row's mask
                    if (c0 == 32u) {
                        lo |= __funnelshift_l(m, 0u, o);
                        hi = m << o;
                    } else if (c0 == 64u) {
                        hi |= __funnelshift_l(m, 0u, o);
                    }
                }
            } else {
                direct(b[0], len, lo, hi, rowsum);
            }
            if (SPLIT) stage.rows[3 * dz + dy][threadIdx.x] = rowsum;
            else rho.add(rowsum);
            if (MASK && active) {
                store_row_mask(S, k, 3 * dz + dy, len, lo, hi);
                overflow |= len > 64;
                total += len;
            }
            b[0] = b[1], e[0] = e[1], ua[0] = ua[1], at[0] = at[1], at[1] = at[2];
            b[1] = b[2], e[1] = e[2], ua[1] = ua[2], at[2] = at[3];
        }
    }
    if (SPLIT) {
        stage.counts[dz0][threadIdx.x] = count;
        stage.cands[dz0][threadIdx.x] = overflow ? SPH_NCAND_SCAN : total;
        __syncthreads();
        if (dz0) return;
#pragma unroll
        for (int r = 0; r < 9; ++r) rho.add(stage.rows[r][threadIdx.x]);
        count = total = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const unsigned c = stage.cands[q][threadIdx.x];
            count += stage.counts[q][threadIdx.x];
            overflow |= c == SPH_NCAND_SCAN;
            total += c;
        }
    }
    const unsigned i = active ? min(S.cellparticles[k], pnum - 1) : 0u;
    if (active) {
        const float value = rho.s * B.coef * *S.mass;
        if (original) {
            S.density0[i] = value;
        } else {
            S.density[i] = value;
            S.num_neighbours[i] = count;
            S.sdens[k] = value;
        }
        if (MASK) {
            S.ncand[k] = overflow ? SPH_NCAND_SCAN : total;
            // the force pass reads a neighbour's pressure with its position
            // and its reciprocal density with its velocity (spare w lanes);
            // a mixed scene's solid particle stores its pressure clamped at
            // 0 and its reciprocal density negated, which marks it solid
            float pv = fluid_pressure(value, *S.restdens, *S.stiffness);
            float rv = rcp_approx(value);
            if (S.phase && S.phase[i]) {
                pv = fmaxf(pv, 0.f);
                rv = -rv;
            }
            S.spos[k].w = pv;
            S.svel[k].w = rv;
        }
    }
}

// Two instantiations, each skipping the other's scenes: the plane variant
// (launched only when some scene has symmetry planes) keeps the common
// plane-free loop free of its registers.
// SPLIT: blocks of (32, 3) threads, each map entry `per` of them.
template <bool PLANES, bool SPLIT = false>
__global__ void __launch_bounds__(SPLIT ? 96 : 512, SPLIT ? 10 : 2)
    k_density(const SceneDesc *__restrict__ scenes, BlockMap map, int original, int want_mask, int skip_solids,
              unsigned per) {
    extern __shared__ __align__(16) unsigned char sm_stage[];
    DensityStage<SPLIT> &stage = *reinterpret_cast<DensityStage<SPLIT> *>(sm_stage);
    SPH_FOR_GROUPS(map, SPLIT ? per : 1u, 32u)
    if (has_planes(S) != PLANES) continue;
    // in a fused substep a plane-free solid's first solid pass sums its density
    if (skip_solids && !PLANES && (S.programs & (PROG_COROT | PROG_SVK))) continue;
    const unsigned n = active_count(S);
    if (first >= n) continue;
    __syncthreads();  // the block's last entry is done with the buffers
    if (want_mask && S.nbmask && (S.programs & PROG_FLUIDS) && !original)
        density_block<PLANES, true, SPLIT>(S, n, first, stage, original);
    else
        density_block<PLANES, false, SPLIT>(S, n, first, stage, original);
    SPH_END_WORK
}

// APPLY_CUBE_BOUNDS(ipos, f, -2.0, 2.0) (common.cl:37-43): a repulsive
// band 0.2 wide inside [-2, 2]^3; the bounds are double literals, so the
// tests and the update are evaluated in double as in the source.  The tests
// (double)p < -2 + (double)0.2f and (double)p > 2 - (double)0.2f run in FP32
// without changing a result: p converts to double exactly, and the bounds
// (-+1.7999999970197678) lie strictly between two floats, so they hold iff
// p <= -0x1.cccccep+0 or p >= 0x1.cccccep+0, the floats just outside them.
// Only a particle inside the band takes the double update; FP64 warp
// instructions are slow on this part, and the test runs for every particle.
#define SPH_CUBE_BAND_LO (-0x1.cccccep+0f)
#define SPH_CUBE_BAND_HI (0x1.cccccep+0f)
__device__ __forceinline__ float cube_bound(float p, float f) {
    const double mn = -2.0, mx = 2.0;
    if (p <= SPH_CUBE_BAND_LO) return (float)((double)f + (1.0 / (-(mn) + (double)p) - 5.0));
    if (p >= SPH_CUBE_BAND_HI) return (float)((double)f - (1.0 / (mx - (double)p) - 5.0));
    return f;
}

// compute_forces_fluids (kernels/fluids.cl:1-63): pressure
// p = (rho - rho0) * stiffness, spiky-gradient pressure and Laplacian
// viscosity pair terms divided by rho_i rho_j, times the mass, plus the
// cube band.  A pair at exactly zero distance contributes nothing (the
// reference produces NaN there).  `fuse_step` also integrates particle i (step_forward) from
// the sorted copies, which no other thread reads afterwards.
__device__ __forceinline__ void integrate(const SceneDesc &S, unsigned i, float3 f, float3 v, float3 p);

// Particle i's side of the fluid pair term.
struct FluidI {
    float3 ipos, ivel;
    float2 nxy, nvxy;  // -ipos and -ivel's x, y lanes (the packed differences)
    float inv_rhoi, pi, h, rho0, stiff;
    float vk, pk;  // visc kv and -kv / 2, the pair term's constant factors
    float le;
};

__device__ __forceinline__ FluidI fluid_i(const SceneDesc &S, float3 ipos, float3 ivel, float rhoi) {
    FluidI I;
    I.ipos = ipos;
    I.ivel = ivel;
    I.nxy = make_float2(-ipos.x, -ipos.y);
    I.nvxy = make_float2(-ivel.x, -ivel.y);
    I.inv_rhoi = rcp_approx(rhoi);
    const ScenePair B = scene_pair(S);
    I.h = B.h;
    I.le = B.le;
    I.rho0 = *S.restdens;
    I.stiff = *S.stiffness;
    I.pi = fluid_pressure(rhoi, I.rho0, I.stiff);
    I.vk = __fmul_rn(*S.viscosity, B.kv);
    I.pk = __fmul_rn(-0.5f, B.kv);
    return I;
}

// 1/sqrt(x) of a normal x from the special-function unit (rsqrtf without
// its scaling of denormals).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One neighbour's pressure + viscosity term (fluids.cl:37-56), added to f,
// from the neighbour's pressure pj and reciprocal density inv_rhoj.  Every
// rounding is pinned, so the scan and the mask walk produce the same sum,
// and a pair's two terms are opposite to the last bit.  (Taking the factors
// common to all terms out of them and adding with fused multiply-adds saves
// a tenth of the instructions, but the terms are then rounded with their
// sums: the momentum of a free mixed scene drifted 4.6 times as far.)
// Distinct particles at exactly zero distance (and i itself) contribute
// nothing.  IN_RANGE: the caller walks the density pass's masks, whose
// candidates passed r^2 <= le with the same positions and arithmetic, so
// that test is not repeated.
template <bool IN_RANGE = false>
__device__ __forceinline__ void fluid_pair_p(const FluidI &I, float pi, float3 jpos, float3 jvel, float pj,
                                             float inv_rhoj, BlockSum3 &f) {
    // d = x_j - x_i and r^2 as sub3 and norm2 compute them, the x and y
    // lanes in packed FP32x2 instructions (each lane rounded alike)
    const float2 dxy = __fadd2_rn(make_float2(jpos.x, jpos.y), I.nxy);
    const float dz = __fsub_rn(jpos.z, I.ipos.z);
    const float2 sq = __fmul2_rn(dxy, dxy);
    const float r2 = __fadd_rn(__fadd_rn(sq.x, sq.y), __fmul_rn(dz, dz));
    if (!IN_RANGE && !(r2 <= I.le)) return;
    float rinv = rsqrt_normal(r2);
    if (r2 < 0x1p-126f) {  // zero or denormal
        if (r2 == 0.f) return;
        rinv = rsqrtf(r2);
    }
    const float din = __fsub_rn(I.h, __fmul_rn(r2, rinv));
    const float inv_didj = __fmul_rn(I.inv_rhoi, inv_rhoj);
    const float vterm = __fmul_rn(din, I.vk);
    const float pterm = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fadd_rn(pi, pj), I.pk), rinv), din), din);
    // (d pterm + (v_j - v_i) vterm) / (rho_i rho_j), per lane as
    // __fmul_rn(__fmaf_rn(d, pterm, __fmul_rn(rv, vterm)), inv_didj)
    const float2 rvxy = __fadd2_rn(make_float2(jvel.x, jvel.y), I.nvxy);
    const float rvz = __fsub_rn(jvel.z, I.ivel.z);
    const float2 fxy = __fmul2_rn(__ffma2_rn(dxy, make_float2(pterm, pterm), __fmul2_rn(rvxy, make_float2(vterm, vterm))),
                                  make_float2(inv_didj, inv_didj));
    f.rxy = __fadd2_rn(f.rxy, fxy);
    f.rz = __fadd_rn(f.rz, __fmul_rn(__fmaf_rn(dz, pterm, __fmul_rn(rvz, vterm)), inv_didj));
}

// The end of a fluid particle's force pass: mass, cube band, store, step.
// `extra`: force already on the particle (a mixed scene's solid particle
// carries its elastic force, which the fluid pair terms add to).
__device__ __forceinline__ void fluid_finish(const SceneDesc &S, unsigned i, const FluidI &I, const BlockSum3 &f,
                                             int fuse_step, float3 extra = make_float3(0.f, 0.f, 0.f)) {
    const float m = *S.mass;
    float3 fi = f.get() * m;
    fi = make_float3(fi.x + extra.x, fi.y + extra.y, fi.z + extra.z);
    fi.x = cube_bound(I.ipos.x, fi.x);
    fi.y = cube_bound(I.ipos.y, fi.y);
    fi.z = cube_bound(I.ipos.z, fi.z);
    st3(S.force, i, fi);
    if (fuse_step) integrate(S, i, fi, I.ivel, I.ipos);
}

// Mixed fluid-solid scenes (extension; `phase` field): a solid particle's
// fluid pair terms cover its fluid neighbours only (its solid neighbours
// act through the elastic force), a fluid particle's cover every neighbour;
// a pair with a solid particle takes both pressures clamped at 0 (it
// pushes, never pulls).
template <bool MIXED>
__device__ __forceinline__ bool mixed_solid(const SceneDesc &S, unsigned i) {
    return MIXED && S.phase && S.phase[i] != 0u;
}
template <bool MIXED>
__device__ __forceinline__ float3 mixed_extra(const SceneDesc &S, unsigned i, bool solid_i) {
    return (MIXED && solid_i) ? ld3(S.force, i) : make_float3(0.f, 0.f, 0.f);
}
// One neighbour of the masked force walk, from its position (pressure in
// w) and velocity (reciprocal density in w, negated for a mixed scene's
// solid particle).
template <bool MIXED>
__device__ __forceinline__ void walk_pair(const FluidI &I, bool solid_i, float4 p, float4 v, BlockSum3 &f) {
    if (MIXED) {
        const bool solid_j = v.w < 0.f;
        if (solid_i && solid_j) return;
        if (solid_i || solid_j)
            return fluid_pair_p<true>(I, fmaxf(I.pi, 0.f), xyz(p), xyz(v), fmaxf(p.w, 0.f), fabsf(v.w), f);
    }
    fluid_pair_p<true>(I, I.pi, xyz(p), xyz(v), p.w, v.w, f);
}

// The stencil scan: every candidate of the rows [r0, r1), in the reference's
// order; row_end(r) closes each.
template <bool MIXED, class RowEnd>
__device__ __forceinline__ void fluid_scan(const SceneDesc &S, const StencilRows &rows, int r0, int r1, const FluidI &I,
                                           BlockSum3 &f, bool solid_i, RowEnd &&row_end) {
    const float4 *spos = S.spos;
    const float4 *svel = S.svel;
    const float *sdens = S.sdens;
#pragma unroll 1
    for (int r = r0; r < r1; ++r) {
        unsigned b, e;
        rows.row(S, r, &b, &e);
        for (unsigned kk = b; kk < e; ++kk) {
            const bool solid_j = MIXED && S.phase[min(S.cellparticles[kk], S.pnum - 1)] != 0u;
            if (solid_i && solid_j) continue;
            const float rho = sdens[kk];
            float pi = I.pi, pj = fluid_pressure(rho, I.rho0, I.stiff);
            if (MIXED && (solid_i || solid_j)) {
                pi = fmaxf(pi, 0.f);
                pj = fmaxf(pj, 0.f);
            }
            fluid_pair_p(I, pi, xyz(spos[kk]), xyz(svel[kk]), pj, rcp_approx(rho), f);
        }
        row_end(r);
    }
}

template <bool MIXED>
__global__ void k_forces_fluids(const SceneDesc *__restrict__ scenes, BlockMap map, int fuse_step) {
    SPH_FOR_WORK(map)
    if (MIXED && !S.phase) continue;  // the plain instantiation covers those
    if (!MIXED && S.phase) continue;
    if (item < active_count(S)) {
        const unsigned k = item;
        const unsigned i = min(S.cellparticles[k], S.pnum - 1);
        const FluidI I = fluid_i(S, xyz(S.spos[k]), xyz(S.svel[k]), S.sdens[k]);
        const bool solid_i = mixed_solid<MIXED>(S, i);
        BlockSum3 f;
        fluid_scan<MIXED>(S, StencilRows(S, S.srow[k]), 0, 9, I, f, solid_i, [&](int) { f.end_row(); });
        fluid_finish(S, i, I, f, fuse_step, mixed_extra<MIXED>(S, i, solid_i));
    }
    SPH_END_WORK
}

// The fused-substep force pass: walks the candidate masks the density pass
// recorded, row by row and two neighbours at a time, reading each
// neighbour's position with its pressure in w and its velocity with its
// reciprocal density in w (two float4 loads).  Lanes whose masks overflowed
// scan the stencil (SPLIT: each warp its plane's rows; 8,000 particles of 27
// a cell 162 -> 67 us, against all nine by one of the three).
// Bound: latency of the gathers (issue slots 64% used; 2 neighbours in
// flight a thread, 32 warps an SM).  Masks whose first candidate is the top
// bit (one leading-zero count finds the next), no count of neighbours here
// and a reciprocal root without denormals' scaling: 132.9M -> 117.1M warp
// instructions, 162 -> 153 us at 1M particles; 150 us with one form of the
// scan, which took the spills with it.
// At most 64 registers (56: 175 against 168 us with the step at 1M, 72: 174).
// SPLIT as in the density pass: blocks of (32, 3) threads, a warp per z
// plane, the row sums added in the same order by the first; 72 registers.
template <bool MIXED, bool SPLIT = false>
__global__ void __maxnreg__(SPLIT ? 72 : 64)
    k_forces_fluids_masked(const SceneDesc *__restrict__ scenes, BlockMap map, int fuse_step, unsigned per) {
    __shared__ float rows_sum[SPLIT ? 9 : 1][3][32];
    SPH_FOR_GROUPS(map, SPLIT ? per : 1u, 32u)
    if (MIXED && !S.phase) continue;  // the plain instantiation covers those
    if (!MIXED && S.phase) continue;
    const unsigned n = active_count(S);
    if (SPLIT) {
        if (first >= n) continue;
        __syncthreads();  // the block's last entry is done with the sums
    }
    const int r0 = SPLIT ? 3 * (int)threadIdx.y : 0, r1 = SPLIT ? r0 + 3 : 9;
    const unsigned k = first + threadIdx.x;
    // a block's warps stay together to its end, where their sums meet
    const bool active = k < n;
    if (SPLIT || active) {
        const unsigned kc = SPLIT ? min(k, n - 1u) : k;  // an idle lane repeats the last particle
        const unsigned i = min(S.cellparticles[kc], S.pnum - 1);
        const FluidI I = fluid_i(S, xyz(S.spos[kc]), xyz(S.svel[kc]), S.sdens[kc]);
        const StencilRows rows(S, S.srow[kc]);
        const bool solid_i = mixed_solid<MIXED>(S, i);
        BlockSum3 f;
        auto end_row = [&](int r) {
            if (SPLIT) {
                rows_sum[r][0][threadIdx.x] = f.rxy.x;
                rows_sum[r][1][threadIdx.x] = f.rxy.y;
                rows_sum[r][2][threadIdx.x] = f.rz;
                f = BlockSum3();
            } else {
                f.end_row();
            }
        };
        if (active && S.ncand[kc] != SPH_NCAND_SCAN) {
            const float4 *spos = S.spos;
            const float4 *svel = S.svel;
            // two neighbours per iteration: both loads are in flight
            // before the first pair's arithmetic (same order)
            // the next row's bounds and low mask word are loaded while this
            // row is walked
            unsigned nb, ne;
            rows.row(S, r0, &nb, &ne);
            unsigned nlo = S.nbmask[(size_t)(2 * r0) * S.pnum + k];
#pragma unroll 1
            for (int r = r0; r < r1; ++r) {
                unsigned b = nb;
                const unsigned len = ne - nb;
                unsigned lo = nlo & first_bits(len);
                if (r + 1 < r1) {
                    rows.row(S, r + 1, &nb, &ne);
                    nlo = S.nbmask[(size_t)(2 * (r + 1)) * S.pnum + k];
                }
                unsigned hi = len > 32u ? S.nbmask[(size_t)(2 * r + 1) * S.pnum + k] & first_bits(len - 32u) : 0u;
                // k itself (row 4, its own cell's) adds no force
                if (r == 4) {
                    const unsigned self = k - b;
                    if (self < 32u) lo &= ~(0x80000000u >> self);
                    else if (self < 64u) hi &= ~(0x80000000u >> (self - 32u));
                }
                // the row's two mask words in turn
#pragma unroll 1
                for (unsigned w = 0, m = lo; w < 2; ++w, m = hi, b += 32) {
                    while (m) {
                        const unsigned t1 = take_first(m);
                        const float4 p1 = spos[b + t1], v1 = svel[b + t1];
                        if (m) {
                            const unsigned t2 = take_first(m);
                            const float4 p2 = spos[b + t2], v2 = svel[b + t2];
                            walk_pair<MIXED>(I, solid_i, p1, v1, f);
                            walk_pair<MIXED>(I, solid_i, p2, v2, f);
                        } else {
                            walk_pair<MIXED>(I, solid_i, p1, v1, f);
                        }
                    }
                }
                end_row(r);
            }
        } else if (active) {
            fluid_scan<MIXED>(S, rows, r0, r1, I, f, solid_i, end_row);
        }
        if (SPLIT) {
            __syncthreads();
            if (r0 || !active) continue;
#pragma unroll
            for (int r = 0; r < 9; ++r)
                f.total.add(make_float3(rows_sum[r][0][threadIdx.x], rows_sum[r][1][threadIdx.x],
                                        rows_sum[r][2][threadIdx.x]));
        }
        fluid_finish(S, i, I, f, fuse_step, mixed_extra<MIXED>(S, i, solid_i));
    }
    SPH_END_WORK
}

// step_forward (common.cl:691-722): a = f/m + g, v += dt a, x += dt v;
// particles of a fixed (non-dynamic) body are skipped, and so are those of
// a rigid body (extension), which its own step moves.  An optional
// `wallbounds` field (extension) mirrors particles that leave the box back
// inside and reverses their normal velocity.
__device__ __forceinline__ void integrate(const SceneDesc &S, unsigned i, float3 f, float3 v, float3 p) {
    // fixed bodies stay put; rigid bodies are moved by k_rigid_scatter
    if (body_skips_step(S, i)) return;
    const float m = *S.mass, dt = *S.timestep;
    const float3 g = make_float3(S.gravity[0], S.gravity[1], S.gravity[2]);
    const float3 a = make_float3(f.x / m + g.x, f.y / m + g.y, f.z / m + g.z);
    st3(S.acceleration, i, a);
    float3 vn = make_float3(v.x + dt * a.x, v.y + dt * a.y, v.z + dt * a.z);
    float3 pn = make_float3(p.x + dt * vn.x, p.y + dt * vn.y, p.z + dt * vn.z);
    if (S.wallbounds) {
        float *pc = &pn.x, *vc = &vn.x;
        for (int a2 = 0; a2 < 3; ++a2) {
            float lo = S.wallbounds[2 * a2], hi = S.wallbounds[2 * a2 + 1];
            if (pc[a2] < lo) {
                pc[a2] = lo + (lo - pc[a2]);
                vc[a2] = -vc[a2];
            } else if (pc[a2] > hi) {
                pc[a2] = hi - (pc[a2] - hi);
                vc[a2] = -vc[a2];
            }
        }
    }
    if (!(isfinite(pn.x) && isfinite(pn.y) && isfinite(pn.z))) atomicOr(S.status, (unsigned)STATUS_NONFINITE);
    st3(S.position, i, pn);
    st3(S.velocity, i, vn);
}

__global__ void k_step_forward(const SceneDesc *__restrict__ scenes, BlockMap map, int planes_only) {
    SPH_FOR_WORK(map)
    // a fused substep's plane-free solids were stepped by their force pass
    if (planes_only && !has_planes(S)) continue;
    if (item < active_count(S)) {
        const unsigned i = item;
        integrate(S, i, ld3(S.force, i), ld3(S.velocity, i), ld3(S.position, i));
    }
    SPH_END_WORK
}

// apply_plane_constraints (kernels/constraints.cl:1-30): project masked
// particles onto each of their planes and remove the normal velocity.
__global__ void k_plane_constraints(const SceneDesc *__restrict__ scenes, BlockMap map) {
    SPH_FOR_WORK(map)
    if (item < active_count(S)) {
        const unsigned i = item;
        const unsigned mask = S.plane_constraints_particles[i];
        if (mask) {
            float3 p = ld3(S.position, i), v = ld3(S.velocity, i);
            for (unsigned c = 0; c < S.num_plane_constraints && c < 32; ++c) {
                if (!(mask & (1u << c))) continue;
                const float *pl = S.plane_constraints + 6 * c;
                float3 pt = make_float3(pl[0], pl[1], pl[2]), nm = make_float3(pl[3], pl[4], pl[5]);
                float dp = dot3(nm, sub3(p, pt));
                p = make_float3(p.x - dp * nm.x, p.y - dp * nm.y, p.z - dp * nm.z);
                float dv = dot3(nm, v);
                v = make_float3(v.x - dv * nm.x, v.y - dv * nm.y, v.z - dv * nm.z);
            }
            st3(S.position, i, p);
            st3(S.velocity, i, v);
        }
    }
    SPH_END_WORK
}

// init_original_position (solids.cl:84-95)
__global__ void k_init_original_position(const SceneDesc *__restrict__ scenes, BlockMap map) {
    SPH_FOR_WORK(map)
    if (item < active_count(S)) st3(S.originalpos, item, ld3(S.position, item));
    SPH_END_WORK
}
