// kernels_common.cuh -- device helpers shared by every sm_103a kernel of the
// pipeline: scene/block-map iteration, IEEE-exact distance tests, Kahan
// sums, the 27-cell neighbour walk and the symmetry-plane images.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sph_internal.h"

#define SPH_FULL_MASK 0xffffffffu
#define SPH_PI_F 3.1415926535f

// A batched scene whose substep quota is used up: every kernel leaves it
// (fields, grid tables and scratch) untouched.
__device__ __forceinline__ bool scene_idle(const SceneDesc &S) { return S.steps_left && *S.steps_left == 0u; }

// The start of every kernel that sph_launch (kernels.cu) may start before the
// kernel ahead of it in the stream has ended: it waits for that end (and for
// its memory), and only then lets the kernel behind it start in turn, so no
// more than one launch waits on the SMs.  A launch without that attribute
// passes straight through.  A waiting kernel is on the SMs while the one
// ahead still writes, so such kernels read with ordinary loads: the
// non-coherent ones (__ldg, const __restrict__ parameters) are only for
// memory that nothing writes while the kernel lives, which here is the scene
// table and the block maps.
__device__ __forceinline__ void follow_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Iterate the virtual blocks of a segment-aware launch.  Inside the body,
// `S` is the block's scene and `item` this thread's item index in it.
// Blocks of idle scenes are skipped (uniformly for the whole block).
#define SPH_FOR_WORK(map)                                                      \
    follow_previous();                                                         \
    for (unsigned vb_ = blockIdx.x; vb_ < (map).num; vb_ += gridDim.x) {       \
        const BlockWork bw_ = (map).work[vb_];                                 \
        const SceneDesc &S = scenes[bw_.scene];                                \
        if (scene_idle(S)) continue;                                           \
        const unsigned item = bw_.first + threadIdx.x;
#define SPH_END_WORK }
// The same with each map entry in `per` groups of `size` items, one group
// per pass: `first` is the group's first item.
#define SPH_FOR_GROUPS(map, per, size)                                         \
    follow_previous();                                                         \
    for (unsigned vb_ = blockIdx.x; vb_ < (map).num * (per); vb_ += gridDim.x) { \
        const BlockWork bw_ = (map).work[vb_ / (per)];                         \
        const SceneDesc &S = scenes[bw_.scene];                                \
        if (scene_idle(S)) continue;                                           \
        const unsigned first = bw_.first + (size) * (vb_ % (per));

// Active particle count, clamped to the store's capacity so that a bad `n`
// written from the host can never index past the fields.
__device__ __forceinline__ unsigned active_count(const SceneDesc &S) {
    unsigned n = *S.n;
    return n < S.pnum ? n : S.pnum;
}

// ---- IEEE-exact helpers (no FMA contraction) --------------------------------
// These reproduce the oracle's individually rounded float operations so that
// cell indices and neighbour decisions are bit-identical.

__device__ __forceinline__ float3 sub3(float3 a, float3 b) {
    return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
// (x*x + y*y) + z*z, the order OpenCL's length()/dot() are restated in
__device__ __forceinline__ float norm2(float3 d) {
    return __fadd_rn(__fadd_rn(__fmul_rn(d.x, d.x), __fmul_rn(d.y, d.y)), __fmul_rn(d.z, d.z));
}
// norm2(sub3(a, b)) with the x and y lanes in packed FP32x2 instructions
// (sm_100 and later; each lane rounds as the scalar instruction does, and
// a + (-b) is a - b exactly): the same value in 6 instructions instead of
// 8.  `b` is passed as its negated x, y pair and its z.
struct NegPoint {
    float2 nxy;
    float z;
};
__device__ __forceinline__ NegPoint neg_point(float3 b) {
    NegPoint o;
    o.nxy = make_float2(-b.x, -b.y);
    o.z = b.z;
    return o;
}
__device__ __forceinline__ float dist2(float4 a, const NegPoint &b) {
    const float2 dxy = __fadd2_rn(make_float2(a.x, a.y), b.nxy);
    const float dz = __fsub_rn(a.z, b.z);
    const float2 sq = __fmul2_rn(dxy, dxy);
    return __fadd_rn(__fadd_rn(sq.x, sq.y), __fmul_rn(dz, dz));
}
__device__ __forceinline__ float dot3(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
// v - (2n) * dot(n, v - p): a mirror image across a symmetry plane
__device__ __forceinline__ float3 reflect3(float3 v, float3 p, float3 n) {
    float d = dot3(n, sub3(v, p));
    float3 tn = make_float3(2.f * n.x, 2.f * n.y, 2.f * n.z);
    return make_float3(__fsub_rn(v.x, __fmul_rn(tn.x, d)), __fsub_rn(v.y, __fmul_rn(tn.y, d)),
                       __fsub_rn(v.z, __fmul_rn(tn.z, d)));
}

// Squared-distance bounds equivalent to the reference's tests on
// dist = sqrt(r2) (correctly rounded):
//   r2 <= lt  <=>  dist <  h        r2 <= le  <=>  dist <= h
struct DistBounds {
    float lt, le;
};
__device__ __forceinline__ float next_up(float x) { return __uint_as_float(__float_as_uint(x) + 1u); }
__device__ __forceinline__ float next_down(float x) { return __uint_as_float(__float_as_uint(x) - 1u); }
__device__ __forceinline__ DistBounds dist_bounds(float h) {
    DistBounds b;
    float x = __fmul_rn(h, h);
    // largest x with sqrt_rn(x) < h
    float lt = x;
    for (int k = 0; k < 6 && lt > 0.f && __fsqrt_rn(lt) >= h; ++k) lt = next_down(lt);
    for (int k = 0; k < 6 && __fsqrt_rn(next_up(lt)) < h; ++k) lt = next_up(lt);
    // largest x with sqrt_rn(x) <= h
    float le = x;
    for (int k = 0; k < 6 && le > 0.f && __fsqrt_rn(le) > h; ++k) le = next_down(le);
    for (int k = 0; k < 6 && __fsqrt_rn(next_up(le)) <= h; ++k) le = next_up(le);
    b.lt = lt;
    b.le = le;
    return b;
}

#define SPH_MAX_PLANES 8

// What the pair passes need of a scene's smoothing radius: h, h^2 (rounded
// on its own), the distance bounds, 45 / (pi h^6) and the poly6
// normalisation 315 / (64 pi h^9) (common.cl:78-90).  The bounds take some
// ten square roots and the factors two divisions, so they are evaluated once
// per scene with the sorted copies, which every pair pass follows, and not in
// every thread.
// With the stencil rows' divisions moved the same way: 1M-particle substep
// 396 -> 384 us, a 4,000-particle corotational beam 40.1 -> 38.0 us.
struct ScenePair {
    float h, h2, lt, le, kv, coef;
};
__device__ __forceinline__ void write_scene_pair(const SceneDesc &S) {
    const float h = *S.h, h2 = __fmul_rn(h, h);
    const DistBounds b = dist_bounds(h);
    const float h3 = h2 * h;
    // a plane with a zero normal (an unset slot of the store's field) is
    // never live (load_planes)
    unsigned live = 0;
    for (unsigned c = 0; c < 6u * min(S.num_symmetry_planes, (unsigned)SPH_MAX_PLANES); ++c)
        live |= c % 6u >= 3u && S.symmetry_planes[c] != 0.f;
    S.pair_consts[0] = make_float4(h, h2, b.lt, b.le);
    S.pair_consts[1] = make_float4(45.0f / (SPH_PI_F * h3 * h3), 315.0f / (64.0f * SPH_PI_F * h3 * h3 * h3),
                                   __uint_as_float(live), 0.f);
}
__device__ __forceinline__ ScenePair scene_pair(const SceneDesc &S) {
    const float4 a = S.pair_consts[0], b = S.pair_consts[1];
    return ScenePair{a.x, a.y, a.z, a.w, b.x, b.y};
}
// Whether a scene takes the symmetry-plane variants of the pair passes: some
// plane is set.  A store built from a conf has slots for planes whether or
// not the program sets them, and with none set the plane-free variants do
// the same work in a fraction of the time (a 1,701-particle strain bar
// through the named recipe 317 -> 210 us a substep).
__device__ __forceinline__ bool has_planes(const SceneDesc &S) {
    return S.num_symmetry_planes != 0u && __float_as_uint(S.pair_consts[1].z) != 0u;
}

// 1/x from the special-function unit (rcp.approx.ftz.f32: at most 1 ulp
// from the rounded reciprocal, denormals flushed).  One instruction in place
// of the IEEE-rounded reciprocal's sequence; deterministic, so every walk of
// a pair sum that uses it rounds alike.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Kahan-compensated float accumulator.
struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) { add_rounded(__fsub_rn(x, c)); }
    // a b, rounded with its addition
    __device__ __forceinline__ void add_product(float a, float b) { add_rounded(__fmaf_rn(a, b, -c)); }
    __device__ __forceinline__ void add_rounded(float y) {
        float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
};
struct Kahan3 {
    Kahan x, y, z;
    __device__ __forceinline__ void add(float3 v) { x.add(v.x); y.add(v.y); z.add(v.z); }
    __device__ __forceinline__ void add_product(float3 v, float w) {
        x.add_product(v.x, w);
        y.add_product(v.y, w);
        z.add_product(v.z, w);
    }
    __device__ __forceinline__ float3 get() const { return make_float3(x.s, y.s, z.s); }
};
// Parts of a sum, each with what its own compensation holds back: the parts
// are added with the exact rounding error of each addition (the two-sum of
// Knuth, TAOCP vol. 2, 4.2.2), so the total is rounded once, with its factor,
// whatever cancels between them.
struct CompensatedSum {
    float s, lo;
    __device__ __forceinline__ CompensatedSum(float s_, float lo_) : s(s_), lo(lo_) {}
    __device__ __forceinline__ explicit CompensatedSum(const Kahan &k) : s(k.s), lo(-k.c) {}
    __device__ __forceinline__ void add(const CompensatedSum &o) {
        const float t = __fadd_rn(s, o.s);
        const float b = __fsub_rn(t, s);
        const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(o.s, b));
        lo = __fadd_rn(__fadd_rn(lo, o.lo), err);
        s = t;
    }
    // the sum times a factor
    __device__ __forceinline__ float times(float w) const { return __fmaf_rn(s, w, __fmul_rn(lo, w)); }
};
// Blocked compensated sum of float3 terms: the terms of one stencil row are
// added in order onto a row sum (one rounding each, no compensation; the x
// and y lanes packed), and each row's sum into the total with Kahan
// compensation.  end_row() closes a row; every walk over a particle's
// stencil calls it once for each of the nine rows, empty or outside the
// grid, so that two walks over the same neighbours in the same order give
// the same bits.
struct BlockSum3 {
    float2 rxy = make_float2(0.f, 0.f);
    float rz = 0.f;
    Kahan3 total;
    __device__ __forceinline__ void end_row() {
        total.add(make_float3(rxy.x, rxy.y, rz));
        rxy = make_float2(0.f, 0.f);
        rz = 0.f;
    }
    __device__ __forceinline__ float3 get() const { return total.get(); }
};

__device__ __forceinline__ float3 ld3(const float *p, size_t i) {
    return make_float3(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}
__device__ __forceinline__ void st3(float *p, size_t i, float3 v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
__device__ __forceinline__ float3 xyz(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator-(float3 a) { return make_float3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return make_float3(a.x * s, a.y * s, a.z * s); }

// ---- cell walk ----------------------------------------------------------------

// FOR_PARTICLES_IN_RANGE (common.cl:49-68) on the cell-sorted order: the 27
// cells are visited z, y, x as in the reference, and because cells x-1..x+1
// of one (z, y) row are consecutive in the sort, each row is one contiguous
// range [celloffset[first], celloffset[last] + gridcount[last]).  `f(kk)` is
// called for every sorted neighbour index kk in the reference's order.
// `row_end()` is called after each of the nine rows (dz outer, dy inner),
// including rows outside the grid.
template <class F, class G>
__device__ __forceinline__ void for_each_neighbour(const SceneDesc &S, unsigned cell, F &&f, G &&row_end) {
    const unsigned R0 = S.gridres[0], R1 = S.gridres[1], R2 = S.gridres[2];
    const unsigned layer = R0 * R1;
    const unsigned cz = cell / layer;
    const unsigned rem = cell - cz * layer;
    const unsigned cy = rem / R0;
    const unsigned cx = rem - cy * R0;
    const unsigned x0 = cx > 0 ? cx - 1 : 0;
    const unsigned x1 = cx + 1 < R0 ? cx + 1 : R0 - 1;
    const unsigned *off = S.celloffset;
    const unsigned *cnt = S.gridcount;
    for (int dz = -1; dz <= 1; ++dz) {
        int z = (int)cz + dz;
        for (int dy = -1; dy <= 1; ++dy) {
            int y = (int)cy + dy;
            if (z >= 0 && z < (int)R2 && y >= 0 && y < (int)R1) {
                unsigned row = (unsigned)z * layer + (unsigned)y * R0;
                unsigned b = off[row + x0];
                unsigned e = off[row + x1] + cnt[row + x1];
                if (e > S.pnum) e = S.pnum;  // only reachable with inconsistent host-written tables
                for (unsigned kk = b; kk < e; ++kk) f(kk);
            }
            row_end();
        }
    }
}
template <class F>
__device__ __forceinline__ void for_each_neighbour(const SceneDesc &S, unsigned cell, F &&f) {
    for_each_neighbour(S, cell, f, [] {});
}

// Row r of particle k's stencil (dz outer, dy inner, as the reference's
// z, y, x loops): cells x-1..x+1 of one (z, y) row are consecutive in the
// cell-sorted order, so a row is one range [b, e); empty when the row lies
// outside the grid.  The rows' presence and x extent are packed into one
// word when the stencil is set up.
struct StencilRows {
    unsigned cell, layer, R0;
    // bit r: row r lies in the grid; bit 9 + r: its cell x-1 exists;
    // bit 18 + r: its cell x+1 exists
    unsigned bits;
    // of a cell: three integer divisions, done once per particle (gather_one)
    __device__ __forceinline__ StencilRows(const SceneDesc &S, unsigned cell_) {
        cell = cell_;
        R0 = S.gridres[0];
        const unsigned R1 = S.gridres[1], R2 = S.gridres[2];
        layer = R0 * R1;
        const unsigned cz = cell / layer;
        const unsigned rem = cell - cz * layer;
        const unsigned cy = rem / R0;
        const unsigned cx = rem - cy * R0;
        const unsigned xm = cx > 0, xp = cx + 1 < R0;
        bits = 0;
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const int z = (int)cz + r / 3 - 1, y = (int)cy + r % 3 - 1;
            if (z < 0 || z >= (int)R2 || y < 0 || y >= (int)R1) continue;
            bits |= (1u << r) | (xm << (9 + r)) | (xp << (18 + r));
        }
    }
    // as gather_one stored it
    __device__ __forceinline__ StencilRows(const SceneDesc &S, uint2 stored) {
        cell = stored.x;
        bits = stored.y;
        R0 = S.gridres[0];
        layer = R0 * S.gridres[1];
    }
    __device__ __forceinline__ void row(const SceneDesc &S, int r, unsigned *b, unsigned *e) const {
        *b = *e = 0;
        if (!((bits >> r) & 1u)) return;
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        const unsigned c = (unsigned)((int)cell + dz * (int)layer + dy * (int)R0);
        const unsigned x0 = c - ((bits >> (9 + r)) & 1u), x1 = c + ((bits >> (18 + r)) & 1u);
        unsigned bb = S.celloffset[x0];
        unsigned ee = S.celloffset[x1] + S.gridcount[x1];
        if (ee > S.pnum) ee = S.pnum;  // only with inconsistent host-written tables
        if (bb > ee) bb = ee;
        *b = bb;
        *e = ee;
    }
};

// ---- staged candidates ----------------------------------------------------------

// Which of the staged candidates p .. p + 4 ng - 1 (16-byte aligned, ng
// 1..8) may lie within the bound: candidate p + t at bit 31 - t.  nx, ny,
// nz: the particle's negated coordinates; nb: the negated bound, each twice.
// The differences are the exact test's; r^2 - bound is a chain of fused
// multiply-adds (3 packed operations fewer).  A NaN has its sign clear.
template <unsigned STRIDE>
__device__ __forceinline__ unsigned near_bits(const float *__restrict__ p, unsigned ng, float2 nx, float2 ny, float2 nz,
                                              float2 nb) {
    unsigned acc = 0;
#pragma unroll 1
    for (unsigned g = 0; g < ng; ++g, p += 4) {
        const float4 X = *reinterpret_cast<const float4 *>(p);
        const float4 Y = *reinterpret_cast<const float4 *>(p + STRIDE);
        const float4 Z = *reinterpret_cast<const float4 *>(p + 2 * STRIDE);
        auto two = [&](float2 x, float2 y, float2 z) {
            const float2 dx = __fadd2_rn(x, nx), dy = __fadd2_rn(y, ny), dz = __fadd2_rn(z, nz);
            const float2 s = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nb)));
            acc = __funnelshift_l(__float_as_uint(s.x), acc, 1);
            acc = __funnelshift_l(__float_as_uint(s.y), acc, 1);
        };
        two(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y));
        two(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w));
    }
    return acc << (32u - 4u * ng);
}

// ---- candidate masks -----------------------------------------------------------
// The first pair pass of a fused substep records, per stencil row r of
// sorted particle k, which candidates the later passes need: candidate b_r
// + t is bit 31 - t of the row's low word for t < 32, and bit 63 - t of its
// high word up to t = 63 (first candidate in the top bit, the order the
// passes take them in: a leading-zero count finds the next).  The low word
// is at nbmask[(2r) * pnum + k], the high word at nbmask[(2r+1) * pnum + k]
// (only for rows of more than 32 candidates); ncand[k] = SPH_NCAND_SCAN when
// a row exceeds 64 and the later passes must scan.

// Records row r's mask: low word always, high word for rows over 32.
__device__ __forceinline__ void store_row_mask(const SceneDesc &S, unsigned k, int r, unsigned len, unsigned lo,
                                               unsigned hi) {
    S.nbmask[(size_t)(2 * r) * S.pnum + k] = lo;
    if (len > 32u) S.nbmask[(size_t)(2 * r + 1) * S.pnum + k] = hi;
}

// Bits of the candidates [0, len) of a mask word.
__device__ __forceinline__ unsigned first_bits(unsigned len) {
    return len >= 32u ? 0xffffffffu : ~(0xffffffffu >> len);
}

// A row's mask words as recorded, with bits past the row's end cleared
// (every visited index stays inside [b, e)).
struct RowMask {
    unsigned lo, hi;
};
__device__ __forceinline__ RowMask load_row_mask(const SceneDesc &S, unsigned k, int r, unsigned len) {
    RowMask m;
    m.lo = S.nbmask[(size_t)(2 * r) * S.pnum + k] & first_bits(len);
    m.hi = len > 32u ? S.nbmask[(size_t)(2 * r + 1) * S.pnum + k] & first_bits(len - 32u) : 0u;
    return m;
}

// The next candidate of a mask word, taken out of it.
__device__ __forceinline__ unsigned take_first(unsigned &m) {
    const unsigned t = (unsigned)__clz((int)m);
    m ^= 0x80000000u >> t;
    return t;
}

// Calls f(kk) for the candidates of particle k's recorded masks in rows
// [r0, r1), in order.
// PREFETCH: the next row's bounds and low mask word are loaded while a row
// is walked (it pays in the corotational pass 2; the solid force passes,
// at their register cap, run slower with it).
template <bool PREFETCH = false, class F>
__device__ __forceinline__ void for_each_masked(const SceneDesc &S, unsigned k, const StencilRows &rows, F &&f,
                                                int r0 = 0, int r1 = 9) {
    unsigned nb = 0, ne = 0, nlo = 0;
    if (PREFETCH) {
        rows.row(S, r0, &nb, &ne);
        nlo = S.nbmask[(size_t)(2 * r0) * S.pnum + k];
    }
#pragma unroll 1
    for (int r = r0; r < r1; ++r) {
        unsigned b, e;
        RowMask mask;
        if (PREFETCH) {
            b = nb;
            e = ne;
            const unsigned len = e - b;
            mask.lo = nlo & first_bits(len);
            if (r + 1 < r1) {
                rows.row(S, r + 1, &nb, &ne);
                nlo = S.nbmask[(size_t)(2 * (r + 1)) * S.pnum + k];
            }
            mask.hi = len > 32u ? S.nbmask[(size_t)(2 * r + 1) * S.pnum + k] & first_bits(len - 32u) : 0u;
        } else {
            rows.row(S, r, &b, &e);
            mask = load_row_mask(S, k, r, e - b);
        }
        // the row's two mask words in turn
#pragma unroll 1
        for (unsigned w = 0, m = mask.lo; w < 2; ++w, m = mask.hi, b += 32)
            while (m) f(b + take_first(m));
    }
}

// ---- symmetry planes (the SYMMETRY blocks, e.g. common.cl:647-686) ----------

struct Planes {
    float3 p[SPH_MAX_PLANES], n[SPH_MAX_PLANES];
    unsigned count;
    unsigned imask;  // planes that i itself passes (|n.(x_i - p)| <= h)
};

__device__ __forceinline__ void load_planes(const SceneDesc &S, float3 ipos, float h, Planes &P) {
    P.count = S.num_symmetry_planes < SPH_MAX_PLANES ? S.num_symmetry_planes : SPH_MAX_PLANES;
    P.imask = 0;
    for (unsigned k = 0; k < P.count; ++k) {
        const float *pl = S.symmetry_planes + 6 * k;
        P.p[k] = make_float3(pl[0], pl[1], pl[2]);
        P.n[k] = make_float3(pl[3], pl[4], pl[5]);
        // a zero normal makes jplane_dist 0 < 1e-5 for every j: never live
        bool live = !(P.n[k].x == 0.f && P.n[k].y == 0.f && P.n[k].z == 0.f);
        if (live && !(fabsf(dot3(P.n[k], sub3(ipos, P.p[k]))) > h)) P.imask |= 1u << k;
    }
}

// Planes of the i-live set that j also passes (|n.(x_j - p)| in [1e-5, h]).
// The reference tests (double)jd < 1.0e-5; jd converts to double exactly
// and 1e-5 lies strictly between two floats, so the test holds iff jd <=
// 0x1.4f8b58p-17f, the float just below it (FP32, no FP64 instruction per
// candidate).
#define SPH_PLANE_EPS_BELOW 0x1.4f8b58p-17f
__device__ __forceinline__ unsigned plane_jmask(const Planes &P, float3 jpos, float h) {
    unsigned m = 0;
    for (unsigned k = 0; k < P.count; ++k) {
        if (!(P.imask & (1u << k))) continue;
        float jd = fabsf(dot3(P.n[k], sub3(jpos, P.p[k])));
        if (!(jd > h) && !(jd <= SPH_PLANE_EPS_BELOW)) m |= 1u << k;
    }
    return m;
}
