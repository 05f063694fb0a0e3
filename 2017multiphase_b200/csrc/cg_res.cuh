// cg_res.cuh — the whole CG solve in one cooperative kernel whose vectors stay
// on chip, for grids that fit (up to about 2.3M cells in FP32); included by
// k_cg.cu (uses its Red, the operators and the flag and scalar slots).
//
// What bounds it: a CG iteration has two dot products that everything after
// them depends on. With one launch per pass an iteration cost 20 us at 32^3
// and 64^3 and 27 us at 96^3, however small the grid: launch, a ring of tiles
// through shared memory, partial sums through the last block. Here a CTA per
// SM keeps its tile of k-rows for the whole solve (p with a one-row halo and x
// in shared memory, r and A p in registers), so an iteration costs one or two
// all-to-all exchanges through L2 and the stencil out of shared memory.
//
// One exchange (ONE; FP32 vectors, up to RES_ONE_Q groups a thread): the new
// r . r is also r.r - 2 alpha r.z + alpha^2 z.z (z = A p), so r.z and z.z travel
// with p.z, and beta is known without a second exchange, but for the rounding of
// the new r (about 1e-7 / sqrt(cells) of r . r). The true r . r comes with the next
// exchange. Where its beta rounds to another float, in a few of a hundred iterations,
// p and z are formed again from the last p, which is kept beside the new one;
// alpha, the stop rule and the count use the true r . r too. So nothing is
// approximated: the operations on the vectors are those of two exchanges, and
// only the FP64 sums add their terms in another order. (Left alone, one float of
// beta off changes where the iteration stops: 2.5e-4 in a velocity at a tolerance
// of 1e-6.)
// The halo carries z instead of r, from which the readers form r as its owner does.
// us an iteration with two exchanges -> one: 4.3 -> 3.6 (32^3), 5.0 -> 3.9 (64^3),
// 6.5 -> 5.9 (96^3), 7.6 -> 7.3 (104^3). With six groups a thread the two more dot
// products and the halo's z cost what the exchange takes (112^3: 8.5 and 8.4;
// 120^3: 9.1 and 9.3), so there it stays at two. FP64 vectors use beta unrounded
// and always take two.
//
// Exchanges carry no fence and no atomics: every 64-bit word that a CTA
// publishes holds 32 bits of payload and a 32-bit tag that no earlier exchange
// used, so a reader that finds the tag has the payload (a 64-bit access is a
// single access), and polling overlaps the latency of partial sums and halo
// rows. A CTA's FP64 partial sum is two such words; every CTA reads all of
// them and adds them in the same order, so all take the same decision. A slot
// is written again only after its readers have published something that
// follows their read in program order: the partial sums of the other dot
// product, or, with one exchange, those of the next iteration, for which there
// are two buffers in turn. Each CTA's slot has 256 bytes of its
// own: 148 CTAs that polled slots packed 16 bytes apart took 8000 cycles an
// exchange, at 256 bytes 2300 (writes to a line that others poll queue up).
//
// Arithmetic: operands, operations and their order are those of the passes
// (k_cg_tma, k_cg_v4, k_cg_pm) for given alpha and beta; the FP64 dot products
// add their terms in another order, so that once in a while an alpha or beta
// rounds to the float beside it.
//
// The launch is cooperative (its CTAs wait on one another) and every wait is
// bounded: after RES_WAIT_NS the CTA raises DONE_TIMEOUT and returns, and the
// solve is done again by the passes.
#pragma once

namespace {

constexpr int RES_T = 512, RES_W = RES_T / 32;
constexpr int RES_MAX_BLK = 160;      // five polling warps of 32 slots
constexpr int RES_ONE_Q = 4;          // one exchange an iteration up to as many groups a thread
constexpr int RES_SLOT = 32;          // words from one CTA's slot to the next
constexpr size_t RES_SLOT_WORDS = 2 * (size_t)RES_MAX_BLK * RES_SLOT;
constexpr unsigned long long RES_WAIT_NS = 1000000000ull;

// Tiles of ti x tj k-rows (ResGeom). A row is padded to whole groups of V
// cells (16 bytes), KG groups a row; group G of a tile is row G / KG, and thread
// t owns groups t, t + RES_T, ...; Q (ResPlan) is their number per thread,
// rounded up to a built kernel. A published group is four words, at its
// owner's place in p, so publishing needs no address of its own.
__device__ __forceinline__ uint64_t res_word(uint32_t tag, uint32_t bits) { return ((uint64_t)tag << 32) | bits; }
__device__ __forceinline__ void res_st2(uint64_t* w, uint64_t a, uint64_t b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void res_ld2(const uint64_t* w, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
}
__device__ __forceinline__ bool res_tag(uint64_t v, uint32_t tag) { return (uint32_t)(v >> 32) == tag; }
__device__ __forceinline__ void res_put(uint64_t* w, double v, uint32_t tag) {
    res_st2(w, res_word(tag, (uint32_t)__double2loint(v)), res_word(tag, (uint32_t)__double2hiint(v)));
}
template <class R> struct alignas(16) ResGroup {
    static constexpr int V = 16 / sizeof(R);
    R v[V];
};
__device__ __forceinline__ void res_put_group(uint64_t* w, const ResGroup<float>& g, uint32_t tag) {
    res_st2(w, res_word(tag, __float_as_uint(g.v[0])), res_word(tag, __float_as_uint(g.v[1])));
    res_st2(w + 2, res_word(tag, __float_as_uint(g.v[2])), res_word(tag, __float_as_uint(g.v[3])));
}
__device__ __forceinline__ void res_put_group(uint64_t* w, const ResGroup<double>& g, uint32_t tag) {
    res_put(w, g.v[0], tag);
    res_put(w + 2, g.v[1], tag);
}
__device__ __forceinline__ void res_words_to(const uint64_t (&w)[4], ResGroup<float>& g) {
    #pragma unroll
    for (int e = 0; e < 4; e++) g.v[e] = __uint_as_float((uint32_t)w[e]);
}
__device__ __forceinline__ void res_words_to(const uint64_t (&w)[4], ResGroup<double>& g) {
    g.v[0] = __hiloint2double((int)(uint32_t)w[1], (int)(uint32_t)w[0]);
    g.v[1] = __hiloint2double((int)(uint32_t)w[3], (int)(uint32_t)w[2]);
}
// counts polls; true once RES_WAIT_NS have passed since its first clock reading
__device__ __forceinline__ bool res_late(uint32_t n, unsigned long long& t0) {
    if ((n & 255u) != 0) return false;
    const unsigned long long t = tt_clock_ns();
    if (t0 == 0) t0 = t;
    return t - t0 > RES_WAIT_NS;
}
__device__ __forceinline__ double res_warp_sum(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// acc + a b as the passes form it: the product of two floats is exact in
// FP64, so one fused operation rounds as the two do
__device__ __forceinline__ double res_mad(float a, float b, double acc) { return __fma_rn((double)a, (double)b, acc); }
__device__ __forceinline__ double res_mad(double a, double b, double acc) { return acc + a * b; }

template <class R, class Op, int Q, bool ONE>
__global__ void __launch_bounds__(RES_T, 1)
    k_cg_res(Op op, ResGeom G, const R* __restrict__ b, R* __restrict__ x, uint64_t* __restrict__ exch,
             uint64_t* __restrict__ slots, Red Rd, int tolmode, float tol, int maxiter, uint32_t epoch) {
    extern __shared__ __align__(16) unsigned char res_raw[];
    constexpr int NS = ONE ? 4 : 1;      // sums of the exchange after A p
    __shared__ double ws[NS][RES_W];
    __shared__ __align__(16) double ws2[NS][RES_MAX_BLK / 32 + 1];
    __shared__ R coef[8];
    __shared__ int failed_;
    volatile int& failed = failed_;
    using Grp = ResGroup<R>;
    constexpr int V = Grp::V;
    const Grid& g = op.g;
    const int NZ = g.NZ, KG = G.KG, nblk = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bi = blockIdx.x / G.nbj, bj = blockIdx.x - bi * G.nbj;
    const int i0 = bi * G.ti, j0 = bj * G.tj;
    const int til = min(G.ti, g.NX - i0), tjl = min(G.tj, g.NY - j0);
    const int ng = til * tjl * KG;                                // own groups
    const int hrows = 2 * (G.ti + G.tj), nhg = hrows * KG;        // halo rows and groups
    const int rows_p = (G.ti + 2) * (G.tj + 2);                   // rows of p, as of the exchange buffer's part per CTA
    const int sI = (tjl + 2) * KG;                                // groups from one plane to the next
    Grp* const p = reinterpret_cast<Grp*>(res_raw);               // (til + 2) x (tjl + 2) rows
    const size_t np_ = (size_t)(G.ti + 2) * (G.tj + 2) * KG;      // ONE: p twice, the last one and the next
    Grp* const xs = p + (ONE ? 2 : 1) * np_;                      // own groups
    Grp* const hr = xs + (size_t)G.ti * G.tj * KG;                // r of the halo rows
    Grp* const hz = hr + nhg;                                     // ONE: A p of the halo rows
    int2* const thalo = reinterpret_cast<int2*>(hz + (ONE ? nhg : 0));   // halo row -> (its owner's row or -1, row of p)

    // ---- set-up --------------------------------------------------------------
    if (tid == 0) failed = 0;
    if (tid < 8) coef[tid] = op.template diag<R>(tid);
    Grp zero;
    #pragma unroll
    for (int e = 0; e < V; e++) zero.v[e] = (R)0;
    for (int s = tid; s < (til + 2) * sI; s += RES_T) {
        p[s] = zero;
        if (ONE) p[np_ + s] = zero;
    }
    for (int h = tid; h < hrows; h += RES_T) {
        // the rows beside the tile: low i, high i (tj rows each), low j, high j
        // (ti rows each); tiles beside it along i have its tjl, along j its til
        int src = -1, dst = 0;
        if (h < 2 * G.tj) {
            const bool hi = h >= G.tj;
            const int lj = hi ? h - G.tj : h;
            if (lj < tjl && (hi ? bi + 1 < G.nbi : bi > 0)) {
                src = ((int)blockIdx.x + (hi ? G.nbj : -G.nbj)) * rows_p + (hi ? 1 : G.ti) * (tjl + 2) + lj + 1;
                dst = (hi ? til + 1 : 0) * (tjl + 2) + lj + 1;
            }
        } else {
            const bool hi = h >= 2 * G.tj + G.ti;
            const int li = h - 2 * G.tj - (hi ? G.ti : 0);
            if (li < til && (hi ? bj + 1 < G.nbj : bj > 0)) {
                const int tjn = hi ? min(G.tj, g.NY - j0 - G.tj) : G.tj;
                src = ((int)blockIdx.x + (hi ? 1 : -1)) * rows_p + (li + 1) * (tjn + 2) + (hi ? 1 : tjn);
                dst = (li + 1) * (tjl + 2) + (hi ? tjl + 1 : 0);
            }
        }
        thalo[h] = make_int2(src, dst);
    }
    // per own group: r, A p, the cells' neighbour bytes (k_nb8's; 0x40: the cell
    // exists), their types, and the place in p with two flags
    constexpr uint32_t AT_PUB = 1u << 31;      // a row that the CTA beside reads
    constexpr uint32_t AT_WALLS = 1u << 30;    // a cell of the warp's groups has a wall beside it along i or j
    constexpr uint32_t AT = AT_WALLS - 1;
    Grp r[Q], z[Q];
    uint32_t nb[Q], ty[Op::kTypedDiag ? Q : 1], at[Q];
    double acc = 0;
    #pragma unroll
    for (int q = 0; q < Q; q++) {
        r[q] = zero; nb[q] = 0; at[q] = 0;
        if (ONE) z[q] = zero;   // published whether it holds an unknown or not
        if (Op::kTypedDiag) ty[q] = 0;
        const int gq = tid + RES_T * q;
        if (gq >= ng) continue;
        const int row = gq / KG, kg = gq - row * KG, li = row / tjl, lj = row - li * tjl;
        at[q] = (uint32_t)((li + 1) * sI + (lj + 1) * KG + kg);
        if ((li == 0 && bi > 0) || (li == til - 1 && bi + 1 < G.nbi) || (lj == 0 && bj > 0) ||
            (lj == tjl - 1 && bj + 1 < G.nbj))
            at[q] |= AT_PUB;
        const int i = i0 + li, j = j0 + lj;
        #pragma unroll
        for (int e = 0; e < V; e++) {
            const int k = V * kg + e;
            if (k >= NZ) continue;
            const int gI = g.NY * NZ, gJ = NZ, idx = i * gI + j * gJ + k;
            uint32_t m = 0x40;
            if (op.mask(idx, i, j, k)) {
                m |= 0x80;
                if (op.fixed(idx + gI)) m |= 1;
                if (op.fixed(idx + gJ)) m |= 2;
                if (op.fixed(idx + 1)) m |= 4;
                if (op.fixed(idx - gI)) m |= 8;
                if (op.fixed(idx - gJ)) m |= 16;
                if (op.fixed(idx - 1)) m |= 32;
                r[q].v[e] = (R)(b[idx] + (R)(-1.0f) * (R)0);
                acc = res_mad(r[q].v[e], r[q].v[e], acc);
                if (Op::kTypedDiag) ty[q] |= (uint32_t)(op.type(idx) & 7) << (8 * e);
            }
            nb[q] |= m << (8 * e);
        }
        xs[gq] = zero;
    }
    #pragma unroll
    for (int q = 0; q < Q; q++)
        if (__any_sync(0xffffffffu, (nb[q] & 0x1b1b1b1bu) != 0)) at[q] |= AT_WALLS;
    __syncthreads();
    constexpr uint32_t UNK = V == 4 ? 0x80808080u : 0x8080u;      // any cell an unknown

    uint64_t* const slot1 = slots;                            // p . A p
    uint64_t* const slot2 = slots + RES_MAX_BLK * RES_SLOT;   // r . r
    // a CTA's partial sum into its slot: warp sums, then warp 0 adds them
    auto publish_sum = [&](uint64_t* slot, double v, uint32_t tag) {
        v = res_warp_sum(v);
        if (lane == 0) ws[0][warp] = v;
        __syncthreads();
        if (warp == 0) {
            double s = lane < RES_W ? ws[0][lane] : 0.0;
            #pragma unroll
            for (int o = RES_W / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) res_put(slot + RES_SLOT * blockIdx.x, s, tag);
        }
    };
    // four of them: the first steps of a warp's sums halve the number of values too
    auto publish_sums4 = [&](uint64_t* slot, const double (&v)[NS], uint32_t tag) {
        const bool h16 = lane & 16, h8 = lane & 8;
        const double x0 = (h16 ? v[1 & (NS - 1)] : v[0]) + __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[1 & (NS - 1)], 16);
        const double x1 = (h16 ? v[3 & (NS - 1)] : v[2 & (NS - 1)]) +
                          __shfl_xor_sync(0xffffffffu, h16 ? v[2 & (NS - 1)] : v[3 & (NS - 1)], 16);
        double y = (h8 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, h8 ? x0 : x1, 8);
        #pragma unroll
        for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if ((lane & 7) == 0) ws[((h16 ? 1 : 0) + (h8 ? 2 : 0)) & (NS - 1)][warp] = y;
        __syncthreads();
        if (warp == 0) {
            const int e = lane & (NS - 1);
            static_assert(RES_W == 16, "two warps' sums a lane");
            double s = ws[e][lane >> 2] + ws[e][(lane >> 2) + 8];
            #pragma unroll
            for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane < NS) res_put(slot + RES_SLOT * blockIdx.x + 2 * lane, s, tag);
        }
    };
    // the first warps after warp 0 collect all partial sums
    auto poll_sums = [&](const uint64_t* slot, uint32_t tag) {
        const int s = (warp - 1) * 32 + lane;
        if (warp >= 1 && warp <= RES_MAX_BLK / 32) {
            double v = 0;
            if (s < nblk) {
                uint64_t lo, hi;
                unsigned long long t0 = 0;
                for (uint32_t n = 1;; ++n) {
                    res_ld2(slot + RES_SLOT * s, lo, hi);
                    if (res_tag(lo, tag) && res_tag(hi, tag)) break;
                    if (res_late(n, t0)) { failed = 1; break; }
                }
                v = __hiloint2double((int)(uint32_t)hi, (int)(uint32_t)lo);
            }
            v = res_warp_sum(v);
            if (lane == 0) ws2[0][warp - 1] = v;
        }
    };
    // the same for four sums a CTA: four lanes read a slot's 64 bytes, 16 each, so
    // an exchange is as many line requests as with one sum (a lane a slot with four
    // loads each: 9 us an iteration at 64^3 instead of 5)
    auto poll_sums4 = [&](const uint64_t* slot, uint32_t tag) {
        if (warp < 1 || warp > RES_MAX_BLK / 32) return;
        constexpr int U = 4;
        const int e = lane & (NS - 1), s0 = (warp - 1) * 32 + (lane >> 2);
        uint64_t lo[U], hi[U];
        unsigned want = 0;
        #pragma unroll
        for (int u = 0; u < U; u++) {
            lo[u] = hi[u] = 0;
            if (s0 + 8 * u < nblk) want |= 1u << u;
        }
        const unsigned have = want;
        unsigned long long t0 = 0;
        for (uint32_t n = 1; want; ++n) {
            #pragma unroll
            for (int u = 0; u < U; u++)
                if (want >> u & 1u) res_ld2(slot + RES_SLOT * (s0 + 8 * u) + 2 * e, lo[u], hi[u]);
            #pragma unroll
            for (int u = 0; u < U; u++)
                if (res_tag(lo[u], tag) && res_tag(hi[u], tag)) want &= ~(1u << u);
            if (res_late(n, t0)) { failed = 1; break; }
        }
        double v = 0;
        #pragma unroll
        for (int u = 0; u < U; u++)
            if (have >> u & 1u) v += __hiloint2double((int)(uint32_t)hi[u], (int)(uint32_t)lo[u]);
        __syncwarp();
        #pragma unroll
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane < NS) ws2[lane][warp - 1] = v;
    };
    auto sums = [&](int e = 0) {
        double t = 0;
        #pragma unroll
        for (int w = 0; w < RES_MAX_BLK / 32; w++) t += ws2[e][w];
        return t;
    };
    // two halo buffers in turn where an iteration has one exchange
    const size_t half = ONE ? (size_t)nblk * rows_p * KG * 4 : 0;
    uint64_t* const mine = exch + (size_t)blockIdx.x * rows_p * KG * 4;
    auto publish_rows = [&](int q, const Grp& v, int buf, uint32_t tag) {
        if (at[q] & AT_PUB) res_put_group(mine + buf * half + (size_t)(at[q] & AT) * 4, v, tag);
    };
    // the halo rows, HB groups in flight per thread
    auto poll_halo = [&](Grp* to, int buf, uint32_t tag) {
        constexpr int HB = 3;
        for (int h0 = tid; h0 < nhg; h0 += HB * RES_T) {
            const uint64_t* src[HB];
            uint32_t pending = 0;
            #pragma unroll
            for (int e = 0; e < HB; e++) {
                const int hg = h0 + e * RES_T;
                src[e] = exch;
                if (hg < nhg) {
                    const int h = hg / KG, row = thalo[h].x;
                    if (row >= 0) { src[e] = exch + buf * half + ((size_t)row * KG + (hg - h * KG)) * 4; pending |= 1u << e; }
                }
            }
            unsigned long long t0 = 0;
            for (uint32_t n = 1; pending; ++n) {
                uint64_t w[HB][4];
                #pragma unroll
                for (int e = 0; e < HB; e++)
                    if (pending >> e & 1u) { res_ld2(src[e], w[e][0], w[e][1]); res_ld2(src[e] + 2, w[e][2], w[e][3]); }
                #pragma unroll
                for (int e = 0; e < HB; e++)
                    if ((pending >> e & 1u) && res_tag(w[e][0], tag) && res_tag(w[e][1], tag) && res_tag(w[e][2], tag) &&
                        res_tag(w[e][3], tag)) {
                        Grp v;
                        res_words_to(w[e], v);
                        to[h0 + e * RES_T] = v;
                        pending &= ~(1u << e);
                    }
                if (res_late(n, t0)) { failed = 1; break; }
            }
        }
    };

    #pragma unroll
    for (int q = 0; q < Q; q++) publish_rows(q, r[q], 1, epoch);
    publish_sum(slot2, acc, epoch);
    poll_sums(slot2, epoch);
    poll_halo(hr, 1, epoch);
    __syncthreads();
    double rr = sums(), a = rr;
    const double eps = tolmode == MP_TOL_REF_ABS ? (double)(tol * (float)g.n) : (double)tol * (double)tol * rr;
    unsigned done = (rr < eps || (tolmode == MP_TOL_REL && eps == 0.0)) ? DONE_CONV : DONE_RUN;
    if (failed) done = DONE_TIMEOUT;
    int it = 0;
    double beta = 0;
    double rr_part = acc;   // ONE: this thread's part of r . r
    bool again = false;     // ONE: beta was not the estimated one
    uint32_t tag = epoch, turn = 0;
    while (done == DONE_RUN && it < maxiter) {
        Grp* const pn = p + (ONE && (it & 1) ? np_ : 0);
        const Grp* const po = p + (ONE && !(it & 1) ? np_ : 0);
        // ---- p = r + beta p on the own cells and the halo -----------------------
        // (cells that are not unknowns hold r = p = 0 throughout)
        const R bf = (R)beta;
        #pragma unroll
        for (int q = 0; q < Q; q++)
            if (nb[q] & UNK) {
                Grp* c = pn + (at[q] & AT);
                if (it == 0) *c = r[q];
                else {
                    Grp v = po[at[q] & AT];
                    #pragma unroll
                    for (int e = 0; e < V; e++) v.v[e] = (R)(r[q].v[e] + bf * v.v[e]);
                    *c = v;
                }
            }
        for (int hg = tid; hg < nhg; hg += RES_T) {
            const int h = hg / KG;
            const int2 t = thalo[h];
            if (t.x >= 0) {
                const size_t c = (size_t)t.y * KG + (hg - h * KG);
                Grp w = hr[hg];
                if (it > 0) {
                    const Grp v = po[c];
                    #pragma unroll
                    for (int e = 0; e < V; e++) w.v[e] = (R)(w.v[e] + bf * v.v[e]);
                }
                pn[c] = w;
            }
        }
        __syncthreads();
        // ---- z = A p, p . z ----------------------------------------------------
        double az[NS] = {};   // p . z; ONE: r . z, z . z, r . r too
        #pragma unroll
        for (int q = 0; q < Q; q++) {
            if (!(nb[q] & UNK)) continue;
            const Grp* c = pn + (at[q] & AT);
            const Grp cur = *c, xp = c[sI], xm = c[-sI], yp = c[KG], ym = c[-KG];
            const R* cs = reinterpret_cast<const R*>(c);
            R line[V + 2];
            line[0] = cs[-1]; line[V + 1] = cs[V];
            #pragma unroll
            for (int e = 0; e < V; e++) line[e + 1] = cur.v[e];
            // a wall beside a cell along k (the first and last cells of every
            // row) is a select in every warp; along i and j whole warps have
            // none, so those four selects are a branch all lanes take alike
            auto row = [&](auto with_walls) {
                constexpr bool walls = decltype(with_walls)::value;
                #pragma unroll
                for (int e = 0; e < V; e++) {
                    const uint32_t m = nb[q] >> (8 * e);
                    const R c0 = cur.v[e];
                    R s = (Op::kTypedDiag ? coef[(ty[q] >> (8 * e)) & 7u] : op.template diag<R>(0)) * c0;
                    s = op.template comb<R>(s, walls && (m & 1u) ? c0 : xp.v[e]);
                    s = op.template comb<R>(s, walls && (m & 2u) ? c0 : yp.v[e]);
                    s = op.template comb<R>(s, (m & 4u) ? c0 : line[e + 2]);
                    s = op.template comb<R>(s, walls && (m & 8u) ? c0 : xm.v[e]);
                    s = op.template comb<R>(s, walls && (m & 16u) ? c0 : ym.v[e]);
                    s = op.template comb<R>(s, (m & 32u) ? c0 : line[e]);
                    s = op.template finish_rec<R>(s);
                    z[q].v[e] = (m & 0x80u) ? s : (R)0;
                    az[0] = res_mad(z[q].v[e], c0, az[0]);   // + 0 off the unknowns, where p = 0
                    if constexpr (ONE) {
                        az[1] = res_mad(z[q].v[e], r[q].v[e], az[1]);
                        az[2] = res_mad(z[q].v[e], z[q].v[e], az[2]);
                    }
                }
            };
            if (at[q] & AT_WALLS) row(std::true_type{});
            else row(std::false_type{});
        }
        ++tag;
        if constexpr (ONE) {
            uint64_t* const slot = slot1 + turn * (RES_SLOT / 2);
            az[3] = rr_part;
            #pragma unroll
            for (int q = 0; q < Q; q++) publish_rows(q, z[q], turn, tag);
            publish_sums4(slot, az, tag);
            poll_sums4(slot, tag);
            poll_halo(hz, turn, tag);
            turn ^= 1u;
        } else {
            publish_sum(slot1, az[0], tag);
            poll_sums(slot1, tag);
        }
        __syncthreads();
        const double zp = sums();
        if (failed) { done = DONE_TIMEOUT; break; }
        if constexpr (ONE) {
            if (it > 0) {
                rr = sums(3);
                if (rr < eps) { done = DONE_CONV; break; }
                const float bt = (float)(rr / a);
                if (!again && __float_as_uint(bt) != __float_as_uint((float)beta)) {
                    // p and z are formed again (from the last p) with the true beta
                    beta = bt;
                    again = true;
                    continue;
                }
                again = false;
                a = rr;
            }
        }
        if (zp == 0) { done = DONE_ZP0; break; }
        const R af = (R)(a / zp);
        // ---- x += alpha p, r -= alpha z, r . r -----------------------------------
        acc = 0;
        #pragma unroll
        for (int q = 0; q < Q; q++) {
            if (nb[q] & UNK) {
                const Grp pv = pn[at[q] & AT];
                Grp xv = xs[tid + RES_T * q];
                #pragma unroll
                for (int e = 0; e < V; e++)
                    if (nb[q] & (0x80u << (8 * e))) {
                        xv.v[e] = xv.v[e] + af * pv.v[e];
                        r[q].v[e] = r[q].v[e] + (-af) * z[q].v[e];
                        acc = res_mad(r[q].v[e], r[q].v[e], acc);
                    }
                xs[tid + RES_T * q] = xv;
            }
            if (!ONE) publish_rows(q, r[q], 0, tag + 1);
        }
        it++;
        if constexpr (ONE) {
            // the halo rows' r as their owners form it (both are 0 off the unknowns)
            for (int hg = tid; hg < nhg; hg += RES_T)
                if (thalo[hg / KG].x >= 0) {
                    Grp v = hr[hg];
                    const Grp w = hz[hg];
                    #pragma unroll
                    for (int e = 0; e < V; e++) v.v[e] = v.v[e] + (-af) * w.v[e];
                    hr[hg] = v;
                }
            rr_part = acc;
            if (it < maxiter) {
                const double ad = (double)af;
                beta = (float)(((a - 2.0 * ad * sums(1)) + ad * ad * sums(2)) / a);
                continue;
            }
        }
        ++tag;
        publish_sum(slot2, acc, tag);
        poll_sums(slot2, tag);
        if (!ONE) poll_halo(hr, 0, tag);
        __syncthreads();
        rr = sums();
        if (failed) { done = DONE_TIMEOUT; break; }
        if (rr < eps) done = DONE_CONV;
        else if (it >= maxiter) done = DONE_CAP;
        else { beta = rr / a; a = rr; }
    }
    // ---- results ---------------------------------------------------------------
    #pragma unroll
    for (int q = 0; q < Q; q++) {
        const int gq = tid + RES_T * q;
        if (gq >= ng) continue;
        const int row = gq / KG, kg = gq - row * KG, li = row / tjl, lj = row - li * tjl;
        const Grp xv = xs[gq];
        #pragma unroll
        for (int e = 0; e < V; e++)
            if (V * kg + e < NZ) x[((i0 + li) * g.NY + j0 + lj) * NZ + V * kg + e] = xv.v[e];
    }
    if (done == DONE_TIMEOUT) {
        if (tid == 0) atomicExch(&Rd.flag[F_DONE], (unsigned)DONE_TIMEOUT);
    } else if (blockIdx.x == 0 && tid == 0) {
        Rd.scal[S_RR] = rr;
        Rd.flag[F_ITERS] = (unsigned)it;
        atomicCAS(&Rd.flag[F_DONE], 0xffffffffu, done);   // the host's "not written" value; a timeout stays
    }
}

// groups per thread that kernels are built for: r and A p take eight registers
// a group, of 128 a thread
inline int res_round_q(int q) {
    for (int v : {1, 2, 3, 4, 6, 8})
        if (q <= v) return v;
    return 0;
}
inline size_t res_smem(const ResGeom& t, bool one) {
    const size_t hrows = 2 * (size_t)(t.ti + t.tj);
    return 16 * (size_t)t.KG * ((one ? 2 : 1) * ((size_t)(t.ti + 2) * (t.tj + 2) + hrows) + (size_t)t.ti * t.tj) + 8 * hrows;
}
// The tiling with the least work for the busiest thread: about 100 issue slots
// for an own group (three passes over it), 50 for a halo group, and 2 for
// each CTA that all the others poll (its slot's line apart, that is nearly free). nblk = 0 when no tiling fits the SMs'
// registers and shared memory.
template <class R> inline ResPlan res_plan(const Grid& g, int sms, size_t smem_max, bool one) {
    ResPlan best;
    best.one = one;
    double best_cost = 1e300;
    const int maxblk = std::min(sms, RES_MAX_BLK), V = ResGroup<R>::V, KG = (g.NZ + V - 1) / V;
    for (int ti = 1; ti <= g.NX; ti++) {
        const int nbi = (g.NX + ti - 1) / ti;
        if (nbi > maxblk) continue;
        for (int tj = 1; tj <= g.NY; tj++) {
            const int nbj = (g.NY + tj - 1) / tj;
            if ((long long)nbi * nbj > maxblk) continue;
            const long long ng = (long long)ti * tj * KG, nhg = 2LL * (ti + tj) * KG;
            const int q = (int)((ng + RES_T - 1) / RES_T), Q = q > 8 ? 0 : res_round_q(q);
            if (!Q) break;
            const ResGeom t{ti, tj, nbi, nbj, KG};
            const size_t sm = res_smem(t, one);
            if (sm > smem_max) continue;
            const double cost = (100.0 * ng + 50.0 * nhg) / 128.0 + 2.0 * nbi * nbj;
            if (cost < best_cost) {
                best_cost = cost;
                best.g = t; best.nblk = nbi * nbj; best.Q = Q; best.smem = sm;
            }
        }
    }
    return best;
}
// words of a plan's halo exchange (slots excluded)
inline size_t res_exch_words(const ResPlan& P) { return (size_t)(P.one ? 2 : 1) * P.nblk * (P.g.ti + 2) * (P.g.tj + 2) * P.g.KG * 4; }

}  // namespace
