// kernels_mixed.cuh -- fluid and elastic solid particles in one scene
// (extension; sm_103a).
//
// The reference runs one program per store (src/opencl/particle_system_host.c:
// 184-313), so a scene is either a fluid (kernels/fluids.cl) or a solid
// (kernels/solid_svk.cl).  A mixed scene lists both programs and carries a
// per-particle `phase` field: 0 = fluid, 1 = St. Venant-Kirchhoff solid.
//   - Density (common.cl:610-690) covers every neighbour, whatever its
//     phase; a solid particle's rest density (solids.cl:99-170) covers its
//     solid neighbours only.
//   - A solid particle's deformation gradient and elastic pair forces
//     (solid_svk.cl:82-367) cover its solid neighbours only, with the
//     store's `solid_viscosity` in place of `viscosity` when present.
//   - Every pair with at least one fluid particle takes the fluid pair term
//     of fluids.cl:1-63 -- pressure from each particle's own density
//     through the fluid's equation of state, plus viscosity -- which is
//     antisymmetric, so the momentum one particle gains the other loses.
//     A fluid particle sums it over all its neighbours; a solid particle
//     over its fluid neighbours, added to its elastic force
//     (k_forces_fluids_masked<true>, kernels_fluid.cuh).
// Rigid bodies (body_dynamic 2) are fluid-phase particles and move as
// bodies, as in a fluid scene.
#pragma once

#include "kernels_solid.cuh"

// Rest density of a mixed scene's particles: the poly6 sum over neighbours
// of the particle's own phase (j = i included), from the cell-sorted
// positions, in the stencil's order.
__global__ void k_original_density_mixed(const SceneDesc *__restrict__ scenes, BlockMap map) {
    SPH_FOR_WORK(map)
    if (!S.phase) continue;
    if (item < active_count(S)) {
        const unsigned k = item;
        const unsigned i = min(S.cellparticles[k], S.pnum - 1);
        const SolidConsts C = solid_consts(S);
        const float3 ipos = xyz(S.spos[k]);
        const unsigned ph = S.phase[i];
        Kahan rho;
        for_each_neighbour(S, S.srow[k].x, [&](unsigned kk) {
            const unsigned j = min(S.cellparticles[kk], S.pnum - 1);
            if (S.phase[j] != ph) return;
            const float r2 = norm2(sub3(xyz(S.spos[kk]), ipos));
            if (r2 <= C.le) {
                const float d = fmaxf(C.h2 - r2, 0.f);
                rho.add(d * d * d);
            }
        });
        S.density0[i] = rho.s * C.coef * C.mass;
    }
    SPH_END_WORK
}

// A candidate kk of a mixed scene's solid particle k is a solid partner
// when it is another particle (kk != k) of the solid phase: both read from
// the sorted rest-position copy (spos0, gathered with the phase bit), so
// the test needs no dependent load through cellparticles.
__device__ __forceinline__ bool solid_partner(float4 q4, unsigned kk, unsigned k) {
    return kk != k && (__float_as_uint(q4.w) & SPH_SOLID_PHASE_BIT) != 0u;
}

// f(kk) for particle k's solid partners kk != k that are within h now, or (REST) at rest, in the reference's order, from the sorted
// copies: 32 candidates at a time are tested first, exactly and without the
// work of f, which every lane would otherwise issue whenever any lane of its
// warp met a partner.
template <bool REST, class F>
__device__ __forceinline__ void for_each_partner(const SceneDesc &S, unsigned k, const StencilRows &rows, float3 ipos,
                                                 float3 ipos0, float le, F &&f) {
    const float4 *spos = S.spos;
    const float4 *spos0 = S.spos0;
    const NegPoint nip = neg_point(ipos), nip0 = neg_point(ipos0);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
        unsigned b, e;
        rows.row(S, r, &b, &e);
#pragma unroll 1
        for (; b < e; b += 32u) {
            const unsigned cn = min(e - b, 32u);
            unsigned m = 0;
#pragma unroll 4
            for (unsigned t = 0; t < cn; ++t) {
                const float4 p = spos[b + t], q = spos0[b + t];
                const bool in = dist2(p, nip) <= le || (REST && dist2(q, nip0) <= le);
                if (in && solid_partner(q, b + t, k)) m |= 0x80000000u >> t;
            }
#pragma unroll 1
            while (m) f(b + take_first(m));
        }
    }
}

// The solid passes of a mixed scene run over the list of its solid-phase
// particles (a few percent of a large scene), a thread each, not over every
// particle.  Mixed scenes run as stores of their own: one scene.
// Against a thread per particle of the whole scene: deformations with the
// stresses 38 + 12 -> 29 us, forces 97 -> 82 us for 32,768 solid particles
// among 1,085,513; the substep 577 -> 542 us, three scenes overlapping 464 -> 431.
// (Three warps per 32 of them, one per z plane, halve both times, but their
// sums are then added in another order, and the stresses of an undeformed
// solid are nothing but the rounding of such sums.)
#define SPH_FOR_SOLIDS(S, k)                                                                     \
    follow_previous();                                                                           \
    const SceneDesc &S = scenes[0];                                                              \
    if (!S.phase || !S.spos0) return;                                                            \
    const unsigned solids_ = min(S.solid_list[0], S.pnum);                                       \
    for (unsigned g_ = blockIdx.x * blockDim.x + threadIdx.x; g_ < solids_;                      \
         g_ += gridDim.x * blockDim.x) {                                                         \
        const unsigned k = min(S.solid_list[1 + g_], S.pnum - 1u);
#define SPH_END_SOLIDS }

// compute_deformations (solid_svk.cl:82-175) of a mixed scene's solid
// particles over their solid neighbours: F = Apq Aqq^-1 with
// Apq = sum W(|p|) p q^T and Aqq = sum W(|p|) q q^T over j != i, |p| <= h.
// Needs the sorted copies gathered with the rest positions.  `masked` (a
// fused substep, after the density pass of the same positions): walks the
// density pass's candidate masks, which hold exactly the candidates with
// |p| <= h, in candidate order, so the sums are those of the scan (which a
// named call runs).  `with_stress`: also compute_stresses for the particle,
// as k_stresses_svk would, and the sorted copy of the stress with density0
// beside it.
__global__ void k_deformations_mixed(const SceneDesc *__restrict__ scenes, int masked, int with_stress) {
    SPH_FOR_SOLIDS(S, k)
    const unsigned i = min(S.cellparticles[k], S.pnum - 1);
    const SolidConsts C = solid_consts(S);
    const float3 ipos = xyz(S.spos[k]);
    const float3 ipos0 = xyz(S.spos0[k]);
    float a[15] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // Apq, then Aqq
    // a candidate that is no partner adds zeros (its rest position may be
    // anything): as a branch the test held back the loads after it
    auto add = [&](float4 p4, float4 q4, bool partner) {
        const float3 p = sub3(xyz(p4), ipos);
        const float d = fmaxf(C.h2 - norm2(p), 0.f);
        const float w = partner ? d * d * d : 0.f;
        const float3 qj = sub3(xyz(q4), ipos0);
        const float3 q = make_float3(partner ? qj.x : 0.f, partner ? qj.y : 0.f, partner ? qj.z : 0.f);
        add_outer(p * w, q, a);
        const float3 wq = q * w;
        a[9] = __fmaf_rn(wq.x, q.x, a[9]);
        a[10] = __fmaf_rn(wq.y, q.y, a[10]);
        a[11] = __fmaf_rn(wq.z, q.z, a[11]);
        a[12] = __fmaf_rn(wq.x, q.y, a[12]);
        a[13] = __fmaf_rn(wq.x, q.z, a[13]);
        a[14] = __fmaf_rn(wq.y, q.z, a[14]);
    };
    const StencilRows rows(S, S.srow[k]);
    if (masked && S.ncand[k] != SPH_NCAND_SCAN)
        for_each_masked(S, k, rows, [&](unsigned kk) {
            const float4 q4 = S.spos0[kk], p4 = S.spos[kk];
            add(p4, q4, solid_partner(q4, kk, k));
        });
    else
        for_each_partner<false>(S, k, rows, ipos, ipos0, C.le, [&](unsigned kk) { add(S.spos[kk], S.spos0[kk], true); });
    float inv[6], F[9];
    sym_inverse(a + 9, inv);
    mul_as(a, inv, F);
    for (int c = 0; c < 9; ++c) S.deformation[9 * (size_t)i + c] = F[c];
    if (with_stress) {
        float o[6];
        svk_stress(S, F, o);
        for (int c = 0; c < 6; ++c) S.stress[6 * (size_t)i + c] = o[c];
        S.sstress[2 * (size_t)k] = make_float4(o[0], o[1], o[2], o[3]);
        S.sstress[2 * (size_t)k + 1] = make_float4(o[4], o[5], S.density0[i], 0.f);
    }
    SPH_END_SOLIDS
}

// compute_forces_solids (solid_svk.cl:182-367) of a mixed scene's solid
// particles over their solid neighbours j != i with rest or current
// distance <= h: the elastic pair term from both stresses and the
// Laplacian viscosity (solid_viscosity when the store has it).  Writes
// force, force_elastic, force_viscous and cutoff_force (no symmetry
// planes: the cut-off force is the whole force); the fluid force pass then
// adds the particle's fluid pair terms and steps it.  The candidate tests
// read the sorted copies (gathered with the rest positions); a neighbour's
// velocity, densities and stress come from its sorted copies too in a fused
// substep (SORTED: those of the density pass and of k_deformations_mixed),
// from the fields in a named call, the same values.
template <bool SORTED>
__global__ void k_forces_solids_mixed(const SceneDesc *__restrict__ scenes) {
    SPH_FOR_SOLIDS(S, k)
    const unsigned i = min(S.cellparticles[k], S.pnum - 1);
    const SolidConsts C = solid_consts(S);
    const float3 ipos = xyz(S.spos[k]);
    const float3 ivel = ld3(S.velocity, i);
    const float3 ipos0 = xyz(S.spos0[k]);
    float si[6];
    for (int c = 0; c < 6; ++c) si[c] = S.stress[6 * (size_t)i + c];
    const float rho0i = S.density0[i];
    Kahan3 fe_s, fv_s;
    auto visit = [&](unsigned kk) {
        const float4 q4 = S.spos0[kk];
        const float3 jpos = xyz(S.spos[kk]);
        const float3 x = sub3(ipos0, xyz(q4));
        const float r2 = norm2(sub3(jpos, ipos));
        float3 jvel;
        float sj[6], rho0j, rhoj;
        if (SORTED) {
            const float4 s0 = S.sstress[2 * (size_t)kk], s1 = S.sstress[2 * (size_t)kk + 1];
            jvel = xyz(S.svel[kk]);
            rhoj = S.sdens[kk];
            sj[0] = s0.x, sj[1] = s0.y, sj[2] = s0.z, sj[3] = s0.w, sj[4] = s1.x, sj[5] = s1.y;
            rho0j = s1.z;
        } else {
            const unsigned j = min(S.cellparticles[kk], S.pnum - 1);
            jvel = ld3(S.velocity, j);
            rho0j = S.density0[j];
            rhoj = S.density[j];
            for (int c = 0; c < 6; ++c) sj[c] = S.stress[6 * (size_t)j + c];
        }
        const float vivj = C.mass * C.mass / rho0i / rho0j;
        const float mrj = C.mass / rhoj;
        const float3 gx = spiky_grad(x, C.h, C.kv, C.le);
        const float3 f_ji = sym_vec(si, gx) * (-vivj);
        const bool jbody = (__float_as_uint(q4.w) & ~SPH_SOLID_PHASE_BIT) != 0u;
        const float3 f_ij = jbody ? -f_ji : sym_vec(sj, -gx) * (-vivj);
        const float3 fe = f_ij - f_ji;
        const float lap = r2 <= C.le ? C.kv * (C.h - sqrtf(r2)) : 0.f;
        const float3 fv = (jvel - ivel) * (mrj * lap);
        fe_s.add(fe);
        fv_s.add(fv);
    };
    for_each_partner<true>(S, k, StencilRows(S, S.srow[k]), ipos, ipos0, C.le, visit);
    const float visc = S.solid_viscosity ? *S.solid_viscosity : *S.viscosity;
    const float3 fe = fe_s.get() * 0.5f, fv = fv_s.get() * visc;
    st3(S.force, i, fe + fv);
    st3(S.force_elastic, i, fe);
    st3(S.force_viscous, i, fv);
    st3(S.cutoff_force, i, fe + fv);
    SPH_END_SOLIDS
}
