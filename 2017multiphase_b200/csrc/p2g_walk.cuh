// p2g_walk.cuh — the pair loop of the warp-staged face gathers, shared by the
// transfers (k_p2g.cu) and the adjoint's replay of them (k_adjoint.cu).
#pragma once
#include "mp_dev.cuh"

namespace mpk {

// padded slot of the t-th staged particle: one spare float4 per 8, so lanes
// whose ranges start about a cell (8 particles) apart hit different banks
MPD uint32_t p2g_slot(uint32_t t) { return t + (t >> 3); }
__host__ __device__ constexpr int p2g_slots(int cap) { return cap + cap / 8; }

// The three faces of a node (i, j, k): sums of weights and of weighted velocities
struct FaceSums {
    float wx = 0, sx = 0, wy = 0, sy = 0, wz = 0, sz = 0;
};
// Adds the staged particles [lo, hi) to a node's faces in ascending order, the
// z-face those below hz. A face takes a pair with r2 <= its cut (negative: the
// face does not take this column); beyond 1.4^2 the weight is exactly zero and
// the pair adds nothing. Weights are formed for all three faces without a branch
// (a branch per face around a division cost 86 instructions a particle where
// this takes about 60), the sums are predicated. Particles of another type are
// staged far away, so no cut takes them.
MPD void p2g_walk(const float4* __restrict__ sp, const float4* __restrict__ sv, uint32_t lo, uint32_t hi, uint32_t hz,
                  float3 gpx, float3 gpy, float3 gpz, float cutx, float cuty, float cutz, FaceSums& F) {
    #pragma unroll 2
    for (uint32_t p = lo; p < hi; ++p) {
        const float4 q = sp[p2g_slot(p)], v = sv[p2g_slot(p)];
        const float3 ps = mk3(q.x, q.y, q.z);
        const float3 dx = ps - gpx, dy = ps - gpy, dz = ps - gpz;
        const float r2x = dot(dx, dx), r2y = dot(dy, dy), r2z = dot(dz, dz);
        auto weight = [&](float r2) {
            return v.w * fmaxf(quot_in_range(1.4f * 1.4f, fmaxf(r2, 0.0001f)) - 1.0f, 0.0f);
        };
        const float ax = weight(r2x), ay = weight(r2y), az = weight(r2z);
        if (r2x <= cutx) { F.wx += ax; F.sx += ax * v.x; }
        if (r2y <= cuty) { F.wy += ay; F.sy += ay * v.y; }
        if (r2z <= cutz && p < hz) { F.wz += az; F.sz += az * v.z; }
    }
}
constexpr float P2G_FAR = 1e15f;   // scaled position of a staged particle that no face takes

}  // namespace mpk
