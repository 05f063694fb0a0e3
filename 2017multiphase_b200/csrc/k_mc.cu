// k_mc.cu — marching-cubes surface extraction on the 2x grid.
//
// Reference: runMC_smooth (Multiphase/Multiphase/spray.cu:804-979) with the
// density kernels genWaterDensfield_GY / _liquidAndGas / _Gas
// (spray_k.cu:1528-1772), classifyVoxel (1853), compactVoxels (1891),
// markActiveEdge_MC (2172), generateTriangles_indices (2074), the Taubin
// smoothing kernels (2408-2440) and calnormal_k / normalizeTriangleNor_k
// (2223-2260). Differences that make the output deterministic:
//   * each shared vertex is interpolated once, from its edge's lower node
//     (the reference lets every voxel touching the edge write it);
//   * smoothing displacements and normals are per-vertex gathers over the
//     incident triangles in ascending triangle order (the reference uses
//     float atomics);
//   * output buffers are device memory owned by the context (the reference
//     wrote into OpenGL vertex buffers).
// The reference's smoothMesh applies lambda = 0.5 and then mu = -0.53 with the
// weights already cleared, so only the lambda half-step has an effect; that is
// what is computed here.
#include "ctx.cuh"
#include <type_traits>

using namespace mpk;

namespace {

struct McGrid {
    int NXMC, NYMC, NZMC;   // voxels
    int W, H, D;            // nodes
    float hm;               // node spacing
};

// The solid field: one thread per node, its 4 x 4 x 4 cells in the reference's
// (di, dj, dk, particle) order with per-cell partial sums.
__global__ void __launch_bounds__(256, 6) k_mc_density_solid(McGrid m, Tiles T, Cells cl, const float4* __restrict__ pos,
                                                             float* __restrict__ dens) {
    const float hm = m.hm, R = hm;
    const float cut = hm * hm * 1.001f;
    MP_GRID_LOOP(t, T.threads()) {
        int i, j, k; if (!tile_ijk(T, t, i, j, k)) continue;
        const float3 p = mk3((float)i * hm, (float)j * hm, (float)k * hm);
        float3 center = mk3(0.0f);
        float wsum = 0.0f;
        #pragma unroll 1
        for (int a = max(i - 2, 0); a <= min(i + 1, m.NXMC - 1); ++a) {
            #pragma unroll 1
            for (int b = max(j - 2, 0); b <= min(j + 1, m.NYMC - 1); ++b) {
                const int cb = a * m.NYMC * m.NZMC + b * m.NZMC;
                #pragma unroll 1
                for (int cc = max(k - 2, 0); cc <= min(k + 1, m.NZMC - 1); ++cc) {
                    if (!(__ldg(cl.tmask + cb + cc) & (1u << MP_TYPESOLID))) continue;
                    float3 res = mk3(0.0f);
                    const uint32_t q1 = __ldg(cl.off + cb + cc + 1);
                    #pragma unroll 1
                    for (uint32_t q = __ldg(cl.off + cb + cc); q < q1; ++q) {
                        const float4 o = __ldg(pos + q);
                        if (pflag(o) != MP_TYPESOLID) continue;
                        const float3 d = xyz(o) - p;
                        const float d2 = dot(d, d);
                        // beyond the kernel radius the pair adds nothing: skip it
                        // before the sqrt (exact test with margin)
                        if (d2 > cut) continue;
                        const float dis = sqrtf(d2);
                        if (!(dis < R)) continue;
                        float w = dis / (4 * hm);
                        w = 1 - w * w;
                        w = (float)fmax((double)(w * w * w), 0.0);
                        res.x += o.x * w; res.y += o.y * w; res.z += o.z * w; wsum += w;
                    }
                    center += res;
                }
            }
        }
        const bool border = (i * j * k == 0 || i == m.NXMC || j == m.NYMC || k == m.NZMC);
        const float r = 0.75f * hm, thigh = 0.51f, tlow = 0.49f;
        float phi = -r;
        if (wsum > 0) {
            center /= wsum;
            float Ev = fmaxf(center.x, fmaxf(center.y, center.z)) / (4 * hm);
            float gamma = (thigh - Ev) / (thigh - tlow);
            float f = (Ev < tlow) ? 1 : gamma * gamma * gamma - 3 * gamma * gamma + 3 * gamma;
            phi = (length(p - center) - r * f);
        }
        if (border) phi = fminf(phi, -10.0f);
        dens[(i * m.H + j) * m.D + k] = phi;
    }
}

// The fluid and gas fields (weight (R^2 - dis^2)^3 within R = 2 node spacings).
// A thread computes the nodes (i, j0, k) and (i, j0 + 1, k). For each of the 4 x
// 5 cell columns of their union window it walks the particles of the column's
// cells k-2 .. k+1 in one loop: they are consecutive in the sorted order, and
// with about one particle per 2x cell a loop per cell spends more on its header
// than on its particle. Each node keeps the reference's order and sums: the
// per-cell partial sums (res) are added to the centre when the first particle
// of another cell comes, every node sees its cells and their particles in the
// (di, dj, dk, particle) order, and a column outside a node's window gives it
// weight 0. A weight is max(R^2 - dis^2, 0)^3: the rounded R^2 and dis^2 are
// monotone in R and dis, so it is zero exactly where dis >= R, and a zero
// weight adds +0 (the sums never hold -0). Issue-bound: about 45 instructions
// a node and particle where the loop per cell with sqrtf took 90; warps whose
// window touches no brick with an air particle do not carry the gas sums.
// 256^3 fluid + gas: 37.6 -> 19 ms.
template <int SURF, bool GAS2, bool INRANGE>
__global__ void __launch_bounds__(256, 4) k_mc_pairs(McGrid m, Tiles T, Cells cl, const float4* __restrict__ pos,
                                                     float* __restrict__ dens, int scene, float* __restrict__ dens2,
                                                     const uint8_t* __restrict__ air_brick) {
    const float hm = m.hm, R = hm * 2, RR = R * R;
    const float tiny = RR * 8.7e-19f;   // below it dis^2 does not change R^2 - dis^2
    const uint32_t gas_types = (1u << MP_TYPEAIR) | (scene != MP_SCENE_INTERACTION ? (1u << MP_TYPEAIRSOLO) : 0u);
    const uint32_t types = SURF == MP_MC_FLUID ? ((1u << MP_TYPEAIR) | (1u << MP_TYPEAIRSOLO) | (1u << MP_TYPEFLUID)) : gas_types;
    // T.threads() and the stride are multiples of the warp, and a warp's lanes
    // share i and j: all lanes take part in the votes
    MP_GRID_LOOP(t, T.threads()) {
        int i, jt, k;
        const bool live = tile_ijk(T, t, i, jt, k);
        if (!__any_sync(0xffffffffu, live)) continue;
        const int j0 = 1 + 2 * jt;
        i += 1; k += 1;   // the nodes inside the border
        const bool air = live && brick_marked(air_brick, (m.NYMC + 7) / 8, (m.NZMC + 7) / 8, max(i - 2, 0) >> 3,
                                              min(i + 1, m.NXMC - 1) >> 3, max(j0 - 2, 0) >> 3, min(j0 + 2, m.NYMC - 1) >> 3,
                                              max(k - 2, 0) >> 3, min(k + 1, m.NZMC - 1) >> 3);
        const bool warp_air = __any_sync(0xffffffffu, air);
        const float px = (float)i * hm, py0 = (float)j0 * hm, py1 = (float)(j0 + 1) * hm, pz = (float)k * hm;
        // the cells k-2 .. k+1 inside the grid, as bounds of the off entries
        const int kb0 = live ? max(k - 2, 0) : 0, kb1 = live ? k - 1 : 0, kb2 = live ? k : 0, kb3 = live ? k + 1 : 0,
                  kb4 = live ? min(k + 2, m.NZMC) : 0;
        // [0..2] centre, [3..5] partial sums of the current cell; ws: weights
        float c0[6] = {0, 0, 0, 0, 0, 0}, c1[6] = {0, 0, 0, 0, 0, 0}, ws0 = 0, ws1 = 0;
        float g0[6] = {0, 0, 0, 0, 0, 0}, g1[6] = {0, 0, 0, 0, 0, 0}, gw0 = 0, gw1 = 0;
        auto add = [](float (&c)[6], float& ws, float keep, float flush, float ox, float oy, float oz, float w) {
            // centre += res when another cell starts (x * 1 + y and x * 0 + y
            // are exact, one rounding each as the plain sums)
            c[0] = __fmaf_rn(c[3], flush, c[0]); c[1] = __fmaf_rn(c[4], flush, c[1]); c[2] = __fmaf_rn(c[5], flush, c[2]);
            c[3] = __fmaf_rn(c[3], keep, ox * w); c[4] = __fmaf_rn(c[4], keep, oy * w); c[5] = __fmaf_rn(c[5], keep, oz * w);
            ws += w;
        };
        auto close = [](float (&c)[6]) {
            #pragma unroll
            for (int e = 0; e < 3; e++) { c[e] += c[e + 3]; c[e + 3] = 0.0f; }
        };
        auto walk = [&](auto u0, auto u1, auto with_gas, int cb) {
            constexpr bool U0 = decltype(u0)::value, U1 = decltype(u1)::value, GAS = decltype(with_gas)::value;
            const uint32_t* o = cl.off + cb;
            const uint32_t B0 = __ldg(o + kb0), B1 = __ldg(o + kb1), B2 = __ldg(o + kb2), B3 = __ldg(o + kb3), B4 = __ldg(o + kb4);
            #pragma unroll 1
            for (uint32_t q = B0; q < B4; ++q) {
                const float4 s = __ldg(pos + q);
                const uint32_t f = (uint32_t)pflag(s);
                const float dx = s.x - px, dz = s.z - pz;
                const float xx = dx * dx, zz = dz * dz;
                const float dy0 = s.y - py0, dy1 = s.y - py1;
                const float e0 = (xx + dy0 * dy0) + zz, e1 = (xx + dy1 * dy1) + zz;
                const bool first = q == B0 || q == B1 || q == B2 || q == B3;
                // other types, and positions that are not finite, add nothing
                if (!(((types >> (f & 31u)) & 1u) && (U0 ? e0 : e1) < 1e30f)) {
                    if (first) {
                        if (U0) { close(c0); if (GAS) close(g0); }
                        if (U1) { close(c1); if (GAS) close(g1); }
                    }
                    continue;
                }
                const float flush = first ? 1.0f : 0.0f, keep = 1.0f - flush;
                auto weight = [&](float d2) {
                    const float dc = fmaxf(d2, tiny);
                    const float dis = INRANGE ? sqrt_in_range(dc) : sqrtf(dc);
                    const float w = fmaxf(RR - dis * dis, 0.0f);
                    return w * w * w;
                };
                const bool gas = GAS && ((gas_types >> (f & 31u)) & 1u);
                if (U0) {
                    const float w = weight(e0);
                    add(c0, ws0, keep, flush, s.x, s.y, s.z, w);
                    if (GAS) add(g0, gw0, keep, flush, s.x, s.y, s.z, gas ? w : 0.0f);
                }
                if (U1) {
                    const float w = weight(e1);
                    add(c1, ws1, keep, flush, s.x, s.y, s.z, w);
                    if (GAS) add(g1, gw1, keep, flush, s.x, s.y, s.z, gas ? w : 0.0f);
                }
            }
        };
        // a column with its gas sums only where a lane's cells in it hold an air
        // particle: most warps near a bubble meet it in a few columns
        auto column = [&](auto u0, auto u1, int cb) {
            if (GAS2 && warp_air) {
                bool here = false;
                const uint8_t* tm = cl.tmask + cb;
                for (int c = kb0; c < kb4; c++) here |= (__ldg(tm + c) & ((1u << MP_TYPEAIR) | (1u << MP_TYPEAIRSOLO))) != 0;
                if (__any_sync(0xffffffffu, here)) { walk(u0, u1, std::true_type{}, cb); return; }
            }
            walk(u0, u1, std::false_type{}, cb);
        };
        if (SURF == MP_MC_FLUID || warp_air) {
            using T1 = std::true_type; using F1 = std::false_type;
            #pragma unroll 1
            for (int a = max(i - 2, 0); a <= min(i + 1, m.NXMC - 1); ++a) {
                const int col = a * m.NYMC * m.NZMC + (j0 - 2) * m.NZMC;
                if (j0 - 2 >= 0) column(T1{}, F1{}, col);
                #pragma unroll 1
                for (int b = j0 - 1; b <= min(j0 + 1, m.NYMC - 1); ++b) column(T1{}, T1{}, col + (b - j0 + 2) * m.NZMC);
                if (j0 + 2 < m.NYMC) column(F1{}, T1{}, col + 4 * m.NZMC);
            }
        }
        if (!live) continue;
        #pragma unroll
        for (int u = 0; u < 2; u++) {
            const int j = j0 + u;
            if (j > m.H - 2) continue;
            const float3 p = mk3(px, u ? py1 : py0, pz);
            auto field = [&](const float (&c)[6], float ws, float r) {
                if (!(ws > 0)) return -r;
                return r - length(p - mk3(c[0] + c[3], c[1] + c[4], c[2] + c[5]) / ws);
            };
            const int idx = (i * m.H + j) * m.D + k;
            dens[idx] = field(u ? c1 : c0, u ? ws1 : ws0, SURF == MP_MC_FLUID ? 0.5f * hm : 0.8f * hm);
            if (GAS2) dens2[idx] = field(u ? g1 : g0, u ? gw1 : gw0, 0.8f * hm);
        }
    }
}
// the border nodes of one or two fields
__global__ void k_mc_border(McGrid m, float* __restrict__ dens, float* __restrict__ dens2) {
    const int fi = m.H * m.D, fj = m.W * m.D, fk = m.W * m.H;
    MP_GRID_LOOP(t, 2 * (fi + fj + fk)) {
        int r = t, i, j, k;
        if (r < 2 * fi) { i = r < fi ? 0 : m.W - 1; r %= fi; j = r / m.D; k = r % m.D; }
        else if ((r -= 2 * fi) < 2 * fj) { j = r < fj ? 0 : m.H - 1; r %= fj; i = r / m.D; k = r % m.D; }
        else { r -= 2 * fj; k = r < fk ? 0 : m.D - 1; r %= fk; i = r / m.H; j = r % m.H; }
        const int idx = (i * m.H + j) * m.D + k;
        dens[idx] = -1000.0f;
        if (dens2) dens2[idx] = -1000.0f;
    }
}

// raises *flag when some cell's type mask has `bits`
__global__ void k_mc_any_type(long long n, const uint8_t* __restrict__ tmask, uint32_t bits, uint32_t* flag) {
    MP_GRID_LOOP(c, n) {
        bool hit = (tmask[c] & bits) != 0;
        if (__any_sync(__activemask(), hit) && (threadIdx.x & 31) == (unsigned)(__ffs(__activemask()) - 1))
            atomicOr(flag, 1u);
    }
}
// the solid field when no cell holds a SOLID particle: every node has wsum = 0,
// so the density pass writes -r, and -10 on the border (its min with -r)
__global__ void k_mc_solid_empty(McGrid m, float* __restrict__ dens) {
    const long long tot = (long long)m.W * m.H * m.D;
    const float r = 0.75f * m.hm;
    MP_GRID_LOOP(t, tot) {
        int i, j, k; getijk3((int)t, m.H, m.D, i, j, k);
        bool border = (i * j * k == 0 || i == m.NXMC || j == m.NYMC || k == m.NZMC);
        dens[t] = border ? fminf(-r, -10.0f) : -r;
    }
}

__device__ __forceinline__ float node(const McGrid& m, const float* d, int i, int j, int k) {
    return d[(size_t)i * m.H * m.D + (size_t)j * m.D + k];
}
// corner v of the cube at (i, j, k) is bit v of its case: (0,0,0), (1,0,0),
// (1,1,0), (0,1,0), then the same at k + 1
__device__ __forceinline__ uint32_t cube_index(const McGrid& m, const float* d, int i, int j, int k) {
    float f[8] = {node(m, d, i, j, k), node(m, d, i + 1, j, k), node(m, d, i + 1, j + 1, k), node(m, d, i, j + 1, k),
                  node(m, d, i, j, k + 1), node(m, d, i + 1, j, k + 1), node(m, d, i + 1, j + 1, k + 1), node(m, d, i, j + 1, k + 1)};
    uint32_t ci = 0;
    #pragma unroll
    for (int v = 0; v < 8; v++) ci += (uint32_t)(f[v] < 0.0f) << v;
    return ci;
}
// edge id = 3 * node + (x: 1, y: 0, z: 2) at the edge's lower node (GetEdgeID, spray_k.cu:1926-1959)
__device__ __forceinline__ uint32_t edge_gid(const McGrid& m, int i, int j, int k, int e) {
    // bit e of each mask: the lower node of cube edge e is one further along i, j, k;
    // edges 0, 2, 4, 6 run along i, 1, 3, 5, 7 along j, 8 to 11 along k
    const uint32_t nd = (uint32_t)((i + (int)(0x622u >> e & 1u)) * m.H * m.D + (j + (int)(0xc44u >> e & 1u)) * m.D + (k + (int)(0x0f0u >> e & 1u)));
    return 3u * nd + (e >= 8 ? 2u : ((uint32_t)e & 1u) ^ 1u);
}

// ---- extraction in two row passes --------------------------------------------------
// A warp owns a row of nodes (i, j, *). Voxels and edges are numbered by their
// node, row by row, so one scan over rows gives every row its first active
// voxel, first index and first vertex; the count pass reads the field once and
// the emit pass only the rows that hold something. (Flags and scans over all
// voxels and all three edges of every node moved about 10 GB a surface of a 256^3
// simulation grid; measured, both surfaces of the 128 x 96 x 144 grid took 5.43 ms
// with them and 4.33 ms with the row passes, count 65 us and emit 57 us a surface.)
struct McTables {
    const int32_t* nv;        // vertices of a case
    const int32_t* tri;       // its edges, 16 a case
    const uint32_t* edges;    // its edges as a mask
    int complete;             // every case uses every edge that it crosses
};
struct McNode {
    uint32_t ci;        // case of the voxel whose lowest corner this node is
    bool voxel;         // there is one
    uint32_t edges;     // vertices on this node's edges: bit 0 along y, 1 along x, 2 along z
};
// whether some voxel at the edge of axis ax (0 x, 1 y, 2 z) at node (i, j, k) uses
// it (tables whose cases leave crossed edges out)
__device__ __noinline__ bool mc_edge_used(const McGrid& m, const float* d, const uint32_t* masks, int ax, int i, int j, int k) {
    // the edge's number in the voxel that lies p back along the next axis and q
    // back along the one after
    const int num[3][2][2] = {{{0, 4}, {2, 6}}, {{3, 1}, {7, 5}}, {{8, 11}, {9, 10}}};
    for (int p = 0; p < 2; p++)
        for (int q = 0; q < 2; q++) {
            const int a = i - (ax == 1 ? q : (ax == 2 ? p : 0)), b = j - (ax == 0 ? p : (ax == 2 ? q : 0)),
                      c = k - (ax == 0 ? q : (ax == 1 ? p : 0));
            if (a < 0 || b < 0 || c < 0 || a >= m.NXMC || b >= m.NYMC || c >= m.NZMC) continue;
            if (__ldg(masks + cube_index(m, d, a, b, c)) >> num[ax][p][q] & 1u) return true;
        }
    return false;
}
// Signs along a row of nodes (i, j, *), 32 nodes of it at a time, lane by lane
// (all lanes of the warp): the four nodes (i, j), (i+1, j), (i+1, j+1), (i, j+1) at
// a lane's k as bits 0 .. 3. Two steps of loads are in flight ahead of use.
struct McRow {
    const float *r0, *r1;
    int dj, D;
    float4 ahead;
    uint32_t cur, next;
    __device__ __forceinline__ float4 load(int k) const {
        const int q = min(k, D - 1);
        return make_float4(r0[q], r1[q], r1[q + dj], r0[q + dj]);
    }
    static __device__ __forceinline__ uint32_t nib(float4 f) {
        return (uint32_t)(f.x < 0.0f) | (uint32_t)(f.y < 0.0f) << 1 | (uint32_t)(f.z < 0.0f) << 2 | (uint32_t)(f.w < 0.0f) << 3;
    }
    // out of the grid, the nodes beside repeat the row's own
    __device__ __forceinline__ McRow(const McGrid& m, const float* __restrict__ d, int i, int j) {
        const int lane = threadIdx.x & 31;
        r0 = d + ((size_t)i * m.H + j) * m.D;
        r1 = r0 + (i + 1 < m.W ? (size_t)m.H * m.D : 0);
        dj = j + 1 < m.H ? m.D : 0;
        D = m.D;
        const float4 a = load(lane), b = load(lane + 32);
        ahead = load(lane + 64);
        cur = nib(a); next = nib(b);
    }
    // the cases (node signs at k, and at k + 1 above them) of this step, then on
    __device__ __forceinline__ uint32_t step(int k) {
        uint32_t up = __shfl_down_sync(0xffffffffu, cur, 1);
        const uint32_t n0 = __shfl_sync(0xffffffffu, next, 0);
        if ((threadIdx.x & 31) == 31) up = n0;
        const uint32_t ci = cur | up << 4;
        cur = next; next = nib(ahead); ahead = load(k + 96);
        return ci;
    }
};
// the node (i, j, k) whose case is ci
__device__ __forceinline__ McNode mc_node(const McGrid& m, const float* __restrict__ d, const McTables& T, int i, int j, int k,
                                          uint32_t ci) {
    McNode o;
    o.ci = ci;
    o.voxel = i + 1 < m.W && j + 1 < m.H && k + 1 < m.D;
    o.edges = 0;
    if (k < m.D) {
        const uint32_t s = ci & 1u;
        if ((ci >> 3 & 1u) != s) o.edges |= 1u;
        if ((ci >> 1 & 1u) != s) o.edges |= 2u;
        if (k + 1 < m.D && (ci >> 4 & 1u) != s) o.edges |= 4u;
        if (o.edges && !T.complete) {
            if ((o.edges & 1u) && !mc_edge_used(m, d, T.edges, 1, i, j, k)) o.edges &= ~1u;
            if ((o.edges & 2u) && !mc_edge_used(m, d, T.edges, 0, i, j, k)) o.edges &= ~2u;
            if ((o.edges & 4u) && !mc_edge_used(m, d, T.edges, 2, i, j, k)) o.edges &= ~4u;
        }
    }
    return o;
}
// per row: active voxels, indices, vertices; and every voxel's case
__global__ void __launch_bounds__(256) k_mc_count(McGrid m, const float* __restrict__ dens, McTables T,
                                                  uint8_t* __restrict__ cube, uint4* __restrict__ rows) {
    const int lane = threadIdx.x & 31, nrow = m.W * m.H;
    for (int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); row < nrow; row += (int)(gridDim.x * blockDim.x >> 5)) {
        const int i = row / m.H, j = row - i * m.H;
        uint32_t act = 0, idx = 0, vert = 0;
        uint8_t* cr = cube + ((size_t)i * m.NYMC + j) * m.NZMC;
        McRow R(m, dens, i, j);
        for (int k = lane; k - lane < m.D; k += 32) {
            const uint32_t ci = R.step(k);
            const bool plain = ci == 0u || ci == 255u;
            if (i + 1 < m.W && j + 1 < m.H && k + 1 < m.D) cr[k] = (uint8_t)ci;
            if (!__any_sync(0xffffffffu, !plain)) continue;
            const McNode o = mc_node(m, dens, T, i, j, k, ci);
            if (o.voxel) {
                const uint32_t nv = (uint32_t)__ldg(T.nv + o.ci);
                idx += nv;
                act += nv > 0 ? 1u : 0u;
            }
            vert += __popc(o.edges);
        }
        act = __reduce_add_sync(0xffffffffu, act);
        idx = __reduce_add_sync(0xffffffffu, idx);
        vert = __reduce_add_sync(0xffffffffu, vert);
        if (lane == 0) rows[row] = make_uint4(act, idx, vert, 0u);
    }
}
// exclusive scan of three counts: inside blocks of 1024 rows, then over the
// blocks' totals (one block)
__device__ __forceinline__ uint4 add3(uint4 a, uint4 b) { return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, 0u); }
__device__ __forceinline__ uint4 scan3_block(uint4 v, uint4* ws, uint4* total) {   // 1024 threads
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4 s = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint4 t = make_uint4(__shfl_up_sync(0xffffffffu, s.x, o), __shfl_up_sync(0xffffffffu, s.y, o),
                                   __shfl_up_sync(0xffffffffu, s.z, o), 0u);
        if (lane >= o) s = add3(s, t);
    }
    if (lane == 31) ws[warp] = s;
    __syncthreads();
    uint4 pre = make_uint4(0, 0, 0, 0), tot = pre;
    for (int w = 0; w < 32; w++) {
        if (w == warp) pre = tot;
        tot = add3(tot, ws[w]);
    }
    __syncthreads();
    *total = tot;
    return make_uint4(pre.x + s.x - v.x, pre.y + s.y - v.y, pre.z + s.z - v.z, 0u);
}
__global__ void __launch_bounds__(1024) k_mc_scan_rows(int n, const uint4* __restrict__ rows, uint4* __restrict__ first,
                                                       uint4* __restrict__ blocks) {
    __shared__ uint4 ws[32];
    const int r = blockIdx.x * 1024 + threadIdx.x;
    uint4 tot;
    const uint4 p = scan3_block(r < n ? rows[r] : make_uint4(0, 0, 0, 0), ws, &tot);
    if (r < n) first[r] = p;
    if (threadIdx.x == 0) blocks[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(1024) k_mc_scan_blocks(int n, uint4* __restrict__ blocks, uint32_t* __restrict__ totals) {
    __shared__ uint4 ws[32];
    uint4 run = make_uint4(0, 0, 0, 0);
    for (int b0 = 0; b0 < n; b0 += 1024) {
        const int b = b0 + threadIdx.x;
        uint4 tot;
        const uint4 p = scan3_block(b < n ? blocks[b] : make_uint4(0, 0, 0, 0), ws, &tot);
        if (b < n) blocks[b] = add3(p, run);
        run = add3(run, tot);
    }
    if (threadIdx.x == 0) { totals[0] = run.x; totals[1] = run.y; totals[2] = run.z; }
}
// the active voxels in order with their first index, the vertices, and each
// crossed edge's vertex number
__global__ void __launch_bounds__(256) k_mc_emit(McGrid m, const float* __restrict__ dens, McTables T,
                                                 const uint4* __restrict__ rows, const uint4* __restrict__ first,
                                                 const uint4* __restrict__ blocks, uint32_t* __restrict__ act,
                                                 uint32_t* __restrict__ act_idx, uint32_t* __restrict__ es,
                                                 float3* __restrict__ verts) {
    const int lane = threadIdx.x & 31, nrow = m.W * m.H;
    const unsigned below = (1u << lane) - 1u;
    for (int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); row < nrow; row += (int)(gridDim.x * blockDim.x >> 5)) {
        const uint4 cnt = rows[row];
        if (!(cnt.x | cnt.z)) continue;
        const uint4 at = add3(first[row], blocks[row >> 10]);
        uint32_t a0 = at.x, x0 = at.y, v0 = at.z;
        const int i = row / m.H, j = row - i * m.H;
        McRow R(m, dens, i, j);
        for (int k = lane; k - lane < m.D; k += 32) {
            const uint32_t ci = R.step(k);
            if (!__any_sync(0xffffffffu, ci != 0u && ci != 255u)) continue;
            const McNode o = mc_node(m, dens, T, i, j, k, ci);
            const uint32_t nv = o.voxel ? (uint32_t)__ldg(T.nv + o.ci) : 0u;
            const unsigned on = __ballot_sync(0xffffffffu, nv > 0);
            if (on) {
                uint32_t s = nv;   // inclusive sum along the warp
                #pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xffffffffu, s, d);
                    if (lane >= d) s += t;
                }
                if (nv) {
                    const uint32_t q = a0 + __popc(on & below);
                    act[q] = (uint32_t)((i * m.NYMC + j) * m.NZMC + k);
                    act_idx[q] = x0 + s - nv;
                }
                a0 += __popc(on);
                x0 += __shfl_sync(0xffffffffu, s, 31);
            }
            const unsigned b0 = __ballot_sync(0xffffffffu, o.edges & 1u), b1 = __ballot_sync(0xffffffffu, o.edges & 2u),
                           b2 = __ballot_sync(0xffffffffu, o.edges & 4u);
            if (o.edges) {
                uint32_t v = v0 + __popc(b0 & below) + __popc(b1 & below) + __popc(b2 & below);
                const uint32_t nd = (uint32_t)((i * m.H + j) * m.D + k);
                const float vs = m.hm;
                const float3 p0 = mk3((float)i * vs, (float)j * vs, (float)k * vs);
                const float f0 = node(m, dens, i, j, k);
                #pragma unroll
                for (int off = 0; off < 3; off++) {   // y, x, z
                    if (!(o.edges >> off & 1u)) continue;
                    const float3 p1 = p0 + (off == 1 ? mk3(vs, 0, 0) : (off == 0 ? mk3(0, vs, 0) : mk3(0, 0, vs)));
                    const float f1 = off == 1 ? node(m, dens, i + 1, j, k) : (off == 0 ? node(m, dens, i, j + 1, k) : node(m, dens, i, j, k + 1));
                    const float t = (0.0f - f0) / (f1 - f0);
                    verts[v] = p0 + t * (p1 - p0);
                    es[3 * (size_t)nd + off] = v;
                    v++;
                }
            }
            v0 += __popc(b0) + __popc(b1) + __popc(b2);
        }
    }
}
__global__ void k_mc_indices(McGrid m, uint32_t nact, const uint32_t* __restrict__ act, const uint8_t* __restrict__ cube,
                             const uint32_t* __restrict__ act_idx, const int32_t* __restrict__ nvt,
                             const int32_t* __restrict__ tri, const uint32_t* __restrict__ es, uint32_t* __restrict__ idx) {
    MP_GRID_LOOP(a, nact) {
        uint32_t v = act[a];
        int i, j, k; getijk3((int)v, m.NYMC, m.NZMC, i, j, k);
        int ci = cube[v];
        int nv = __ldg(nvt + ci);
        uint32_t base = act_idx[a];
        for (int t = 0; t < nv; t++) idx[base + t] = es[edge_gid(m, i, j, k, __ldg(tri + ci * 16 + t))];
    }
}
// vertex -> incident (triangle corner) slots, ascending
__global__ void k_mc_inc_count(uint32_t nidx, const uint32_t* __restrict__ idx, uint32_t* __restrict__ cnt) {
    MP_GRID_LOOP(s, nidx) atomicAdd(cnt + idx[s], 1u);
}
__global__ void k_mc_inc_fill(uint32_t nidx, const uint32_t* __restrict__ idx, const uint32_t* __restrict__ start,
                              uint32_t* __restrict__ cnt, uint32_t* __restrict__ inc) {
    MP_GRID_LOOP(s, nidx) {
        uint32_t v = idx[s];
        uint32_t r = atomicSub(cnt + v, 1u) - 1u;
        inc[start[v] + r] = (uint32_t)s;
    }
}
__global__ void k_mc_inc_sort(uint32_t nv, const uint32_t* __restrict__ start, uint32_t* __restrict__ inc) {
    MP_GRID_LOOP(v, nv) {
        uint32_t s0 = start[v];
        sort_distinct_run(inc, s0, start[v + 1] - s0, [](uint32_t) {});
    }
}
__global__ void k_mc_smooth(uint32_t nv, const uint32_t* __restrict__ start, const uint32_t* __restrict__ inc,
                            const uint32_t* __restrict__ idx, const float3* __restrict__ vin, float3* __restrict__ vout) {
    MP_GRID_LOOP(v, nv) {
        float3 pq = vin[v];
        float3 disp = mk3(0.0f);
        int w = 0;
        for (uint32_t s = start[v]; s < start[v + 1]; s++) {
            uint32_t slot = inc[s];
            uint32_t t = slot / 3, c = slot % 3;
            uint32_t o1 = idx[3 * t + (c == 0 ? 1 : 0)];
            uint32_t o2 = idx[3 * t + (c == 2 ? 1 : 2)];
            disp += vin[o1] - pq;
            disp += vin[o2] - pq;
            w += 2;
        }
        vout[v] = (w > 0) ? pq + 0.5f * disp / (float)w : pq;
    }
}
__global__ void k_mc_normals(uint32_t nv, const uint32_t* __restrict__ start, const uint32_t* __restrict__ inc,
                             const uint32_t* __restrict__ idx, const float3* __restrict__ verts, float3* __restrict__ nrm) {
    MP_GRID_LOOP(v, nv) {
        float3 n = mk3(0.0f);
        for (uint32_t s = start[v]; s < start[v + 1]; s++) {
            uint32_t t = inc[s] / 3;
            float3 p1 = verts[idx[3 * t]], p2 = verts[idx[3 * t + 1]], p3 = verts[idx[3 * t + 2]];
            n += cross(p2 - p1, p3 - p1);
        }
        if (length(n) > 0) n = normalize(n);
        nrm[v] = n;
    }
}

}  // namespace

static int readback(MpCtx* c, const uint32_t* dptr, uint32_t* h) {
    MP_CUDA(c, cudaMemcpyAsync(h, dptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
    MP_CUDA(c, cudaStreamSynchronize(c->stream));
    return MP_OK;
}

static McGrid mc_grid(const MpCtx* c) {
    McGrid m;
    m.NXMC = 2 * c->G.NX; m.NYMC = 2 * c->G.NY; m.NZMC = 2 * c->G.NZ;
    m.W = m.NXMC + 1; m.H = m.NYMC + 1; m.D = m.NZMC + 1;
    m.hm = c->G.h / (float)(m.NXMC / c->G.NX);
    return m;
}

// the density gather of one surface, or of fluid and gas together (dens2)
template <int SURF, bool GAS2>
static void launch_density(MpCtx* c, const McGrid& m, float* dens, float* dens2) {
    const Cells cl{c->cell_off, c->tmask};
    if constexpr (SURF == MP_MC_SOLID) {
        const Tiles T = make_tiles(m.W, m.H, m.D);
        k_mc_density_solid<<<mp_blocks(T.threads(), 256), 256, 0, c->stream>>>(m, T, cl, c->pos, dens);
    } else {
        const Tiles T = make_tiles(m.W - 2, (m.H - 1) / 2, m.D - 2);   // two interior nodes along j per thread
        // node spacings whose squares, and those times 2^-60, are well inside
        // the range of sqrt_in_range; other scales take sqrtf
        const bool in_range = m.hm > 1e-5f && m.hm < 1e10f;
        auto k = in_range ? k_mc_pairs<SURF, GAS2, true> : k_mc_pairs<SURF, GAS2, false>;
        k<<<mp_blocks(T.threads(), 256), 256, 0, c->stream>>>(m, T, cl, c->pos, dens, c->P.scene, dens2, c->air_brick);
        const long long edge = 2LL * (m.H * m.D + m.W * m.D + m.W * m.H);
        k_mc_border<<<mp_blocks(edge, 256), 256, 0, c->stream>>>(m, dens, dens2);
        c->launches++;
    }
}
static int mc_extract(MpCtx* c, const McGrid& m, int surface, const float* dens);

// one runMC_smooth surface (spray.cu:804-979)
int k_mc(MpCtx* c, int surface, bool keep_field) {
    if (!c->mc_sorted) { c->err = "mc: particles are not sorted on the 2x grid (call mp_mc_presort)"; return MP_ERR_STATE; }
    const McGrid m = mc_grid(c);
    cudaStream_t s = c->stream;
    bool solid_empty = false;
    if (surface == MP_MC_SOLID) {
        const long long nvox = (long long)m.NXMC * m.NYMC * m.NZMC;
        MP_CUDA(c, cudaMemsetAsync(c->u32_scratch + 4, 0, sizeof(uint32_t), s));
        k_mc_any_type<<<mp_blocks(nvox, 256), 256, 0, s>>>(nvox, c->tmask, 1u << MP_TYPESOLID, c->u32_scratch + 4);
        c->launches++;
        MP_CHECK_LAUNCH(c);
        uint32_t any = 1;
        MP_TRY(readback(c, c->u32_scratch + 4, &any));
        solid_empty = any == 0;
    }
    if (solid_empty) {
        // every node negative: no voxel is active, every case 255; the field and
        // the cases are written unless the caller's next surface replaces them
        McSurface& out = c->mc[surface];
        out.nverts = out.nindices = out.active = 0;
        c->S.mc_active_voxels[surface] = c->S.mc_verts[surface] = c->S.mc_indices[surface] = 0;
        c->mc_last_dens = c->mc_dens;
        if (keep_field) {
            k_mc_solid_empty<<<mp_blocks((long long)m.W * m.H * m.D, 256), 256, 0, s>>>(m, c->mc_dens);
            c->launches++;
            MP_CHECK_LAUNCH(c);
            MP_CUDA(c, cudaMemsetAsync(c->mc_cube, 0xff, (size_t)m.NXMC * m.NYMC * m.NZMC, s));
        }
        return MP_OK;
    } else {
        KtScope kt(c, MP_KT_MC_DENS);
        if (surface == MP_MC_SOLID) launch_density<MP_MC_SOLID, false>(c, m, c->mc_dens, nullptr);
        else if (surface == MP_MC_FLUID) launch_density<MP_MC_FLUID, false>(c, m, c->mc_dens, nullptr);
        else launch_density<MP_MC_GAS, false>(c, m, c->mc_dens, nullptr);
    }
    c->launches++;
    return mc_extract(c, m, surface, c->mc_dens);
}

// the fluid and gas surfaces of one step from a single density pass (the
// same fields and meshes as k_mc(FLUID) followed by k_mc(GAS))
int k_mc_fluid_gas(MpCtx* c) {
    if (!c->mc_sorted) { c->err = "mc: particles are not sorted on the 2x grid (call mp_mc_presort)"; return MP_ERR_STATE; }
    const McGrid m = mc_grid(c);
    {
        KtScope kt(c, MP_KT_MC_DENS);
        launch_density<MP_MC_FLUID, true>(c, m, c->mc_dens, c->mc_dens2);
    }
    c->launches++;
    MP_TRY(mc_extract(c, m, MP_MC_FLUID, c->mc_dens));
    return mc_extract(c, m, MP_MC_GAS, c->mc_dens2);
}

// incidence lists of a surface's vertices (vstart: nv+1, inc: nidx), each
// list ascending
static int mc_incidence(MpCtx* c, const McSurface& out, uint32_t nv, uint32_t nidx) {
    cudaStream_t s = c->stream;
    MP_CUDA(c, cudaMemsetAsync(c->mc_fill, 0, sizeof(uint32_t) * (nv + 1), s));
    k_mc_inc_count<<<mp_blocks(nidx, 256), 256, 0, s>>>(nidx, out.indices, c->mc_fill);
    c->launches++;
    MP_TRY(mp_scan_u32(c, c->mc_fill, c->mc_vstart, nv));
    k_mc_inc_fill<<<mp_blocks(nidx, 256), 256, 0, s>>>(nidx, out.indices, c->mc_vstart, c->mc_fill, c->mc_inc);
    k_mc_inc_sort<<<mp_blocks(nv, 256), 256, 0, s>>>(nv, c->mc_vstart, c->mc_inc);
    c->launches += 2;
    MP_CHECK_LAUNCH(c);
    return MP_OK;
}

// runMC_interaction's stored-surface branch (spray.cu:788-794): calNormals
// on the surface as it stands (moved by the solid motion), no re-extraction
int k_mc_renormal(MpCtx* c, int surface) {
    McSurface& out = c->mc[surface];
    const uint32_t nv = (uint32_t)out.nverts, nidx = (uint32_t)out.nindices;
    if (nv == 0) return MP_OK;
    MP_TRY(mc_incidence(c, out, nv, nidx));
    k_mc_normals<<<mp_blocks(nv, 256), 256, 0, c->stream>>>(nv, c->mc_vstart, c->mc_inc, out.indices, out.verts,
                                                              out.normals);
    c->launches++;
    MP_CHECK_LAUNCH(c);
    return MP_OK;
}

// classification, compaction, vertices, indices, smoothing and normals of one
// surface from its nodal field
static int mc_extract(MpCtx* c, const McGrid& m, int surface, const float* dens) {
    cudaStream_t s = c->stream;
    McSurface& out = c->mc[surface];
    out.nverts = out.nindices = out.active = 0;
    c->mc_last_dens = dens;
    const McTables T{c->mc_numverts, c->mc_tri, c->mc_edge_mask, c->mc_complete};
    const int nrow = m.W * m.H, nblk = (nrow + 1023) / 1024, warps = mp_blocks(32LL * nrow, 256);
    uint32_t* totals = c->u32_scratch + 8;
    k_mc_count<<<warps, 256, 0, s>>>(m, dens, T, c->mc_cube, c->mc_rows);
    k_mc_scan_rows<<<nblk, 1024, 0, s>>>(nrow, c->mc_rows, c->mc_first, c->mc_blocks);
    k_mc_scan_blocks<<<1, 1024, 0, s>>>(nblk, c->mc_blocks, totals);
    c->launches += 3;
    MP_CHECK_LAUNCH(c);
    uint32_t tot[3] = {0, 0, 0};
    MP_CUDA(c, cudaMemcpyAsync(tot, totals, sizeof(tot), cudaMemcpyDeviceToHost, s));
    MP_CUDA(c, cudaStreamSynchronize(s));
    const uint32_t nact = tot[0], nidx = tot[1], nv = tot[2];
    out.active = (int)nact;
    c->S.mc_active_voxels[surface] = (int)nact;
    c->S.mc_verts[surface] = 0; c->S.mc_indices[surface] = 0;
    if (nact == 0) return MP_OK;
    if ((long long)nidx > 3LL * c->P.mc_max_tris) { c->err = "mc: triangle cap exceeded"; return MP_ERR_CAPACITY; }
    if ((long long)nv > c->P.mc_max_verts) { c->err = "mc: vertex cap exceeded"; return MP_ERR_CAPACITY; }
    k_mc_emit<<<warps, 256, 0, s>>>(m, dens, T, c->mc_rows, c->mc_first, c->mc_blocks, c->mc_compact, c->mc_cbase,
                                    c->mc_escan, out.verts);
    k_mc_indices<<<mp_blocks(nact, 256), 256, 0, s>>>(m, nact, c->mc_compact, c->mc_cube, c->mc_cbase, c->mc_numverts,
                                                      c->mc_tri, c->mc_escan, out.indices);
    c->launches += 2;
    MP_CHECK_LAUNCH(c);
    MP_TRY(mc_incidence(c, out, nv, nidx));
    if (c->P.b_smooth_mc) {
        for (int it = 0; it < c->P.smooth_iters; it++) {
            k_mc_smooth<<<mp_blocks(nv, 256), 256, 0, s>>>(nv, c->mc_vstart, c->mc_inc, out.indices, out.verts, c->mc_tmpv);
            c->launches++;
            std::swap(out.verts, c->mc_tmpv);   // both hold mc_max_verts
        }
    }
    k_mc_normals<<<mp_blocks(nv, 256), 256, 0, s>>>(nv, c->mc_vstart, c->mc_inc, out.indices, out.verts, out.normals);
    c->launches++;
    MP_CHECK_LAUNCH(c);
    out.nverts = (int)nv; out.nindices = (int)nidx;
    c->S.mc_verts[surface] = (int)nv;
    c->S.mc_indices[surface] = (int)nidx;
    return MP_OK;
}
