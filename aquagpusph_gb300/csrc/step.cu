// The step kernels compiled with the reference's arithmetic (-fmad=false,
// IEEE division and square root): aqua::exact.  Also the mode-independent
// kernels of the step: the chunk list of the sweep, the end-of-step scalar
// update and the ihoc export.
#include "aqua_internal.cuh"
#include "kernels.cuh"

namespace aqua {

namespace exact {
#define AQUA_FAST_ARITH 0
#include "step_kernels.cuh"
#undef AQUA_FAST_ARITH
}  // namespace exact

namespace {

// Cell-aligned chunks of <= 32 sorted particles: s starts a chunk when it is
// 0, 32, 64, ... particles past the first particle of its cell.  One
// atomicAdd per block of 1024 reserves the block's chunks (in sorted order
// within the block), so the shared counter sees few atomics.
constexpr int kChunkThreads = 1024;
__global__ void __launch_bounds__(kChunkThreads)
k_chunks(const uint32_t* skeys, const uint2* cells, uint32_t N, uint2* chunks,
         DevScalars* sc)
{
    __shared__ uint32_t s_count[kChunkThreads / 32];
    if (sc->err)
        return;
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool start = false;
    uint2 w = make_uint2(0, 0);
    if (s < N) {
        const uint2 se = cells[skeys[s]];
        start = ((s - se.x) & 31u) == 0u;
        w = make_uint2(s, min(32u, se.y - s));
    }
    const unsigned b = __ballot_sync(0xffffffffu, start);
    if (lane == 0)
        s_count[warp] = __popc(b);
    __syncthreads();
    if (warp == 0) {
        // exclusive scan of the warps' counts, one reservation for the block
        const uint32_t v = lane < kChunkThreads / 32 ? s_count[lane] : 0u;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t base = 0;
        if (lane == 0 && total)
            base = atomicAdd(&sc->n_chunks, total);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < kChunkThreads / 32)
            s_count[lane] = base + incl - v;
    }
    __syncthreads();
    if (start)
        chunks[s_count[warp] + __popc(b & ((1u << lane) - 1u))] = w;
}

// Place of the 64 sub-cells of a cell (4 x 4 x 4, x fastest; 8 x 8 in 2-D)
// along a Hilbert curve: consecutive places are neighbouring sub-cells
__constant__ uint8_t kHilbert3[64] = {
    0, 3, 60, 63, 1, 2, 61, 62, 30, 31, 32, 33, 29, 28, 35, 34,
    7, 4, 59, 56, 6, 5, 58, 57, 25, 24, 39, 38, 26, 27, 36, 37,
    8, 11, 52, 55, 15, 12, 51, 48, 16, 23, 40, 47, 19, 20, 43, 44,
    9, 10, 53, 54, 14, 13, 50, 49, 17, 22, 41, 46, 18, 21, 42, 45
};
__constant__ uint8_t kHilbert2[64] = {
    0, 3, 4, 5, 58, 59, 60, 63, 1, 2, 7, 6, 57, 56, 61, 62,
    14, 13, 8, 9, 54, 55, 50, 49, 15, 12, 11, 10, 53, 52, 51, 48,
    16, 17, 30, 31, 32, 33, 46, 47, 19, 18, 29, 28, 35, 34, 45, 44,
    20, 23, 24, 27, 36, 39, 40, 43, 21, 22, 25, 26, 37, 38, 41, 42
};

// Clusters of every cell: its particles, ordered along a Hilbert curve
// through its sub-cells (ties in sorted order), cut every 8 (or 4) into
// cperm[first .. end) and clu.  Full clusters wherever the particles lie:
// groups by octant, which fill clusters of 8 on a lattice, hold 5 to 10
// particles in a flow that has left it.  A block takes 256 sorted positions,
// reserves list entries for the cells that start there with one atomicAdd
// (the order of the lists does not matter) and its warps take those cells.
//
// CELLS = false (quad sweep): clu is the work list, in any order.
// CELLS = true (clustered sweep, 3-D): the work list holds cells (work, wcl);
// a cell's clusters take the slots of clu from its first sorted index on, the
// boundary elements and then the probes come last, in clusters of their own
// (mixed with the elements the fluid's clusters lose their compact boxes: a
// 5.88M step on a lattice took 6.73 ms, then 6.52, and a 5.9M call off it 8.57,
// then 8.45), and crow holds the cell's neighbourhood as 9 rows of 3 cells.
// Where the step is swept by octant (sweep_by_octant()), a cell's clusters are
// octants (8 consecutive places), joined while they fit into 8, if all of them do.
constexpr int kClusterThreads = 256;
// A cell of more particles (parked ones, no fluid cell: 512 with h = 4 spacings in
// 3-D) would keep its warp for long: 20,000 parked particles in 2-D, 336 us a step.
constexpr uint32_t kLargeCell = 1024;
template<int D, bool CELLS>
__global__ void __launch_bounds__(kClusterThreads)
k_cell_clusters(Consts c, StepArgs a, const float4* pos)
{
    constexpr int NWARP = kClusterThreads / 32;
    // places of the boundary elements and the probes, and of no particle
    constexpr uint32_t kWalls = 64, kProbes = 65, kNone = 66;
    __shared__ uint4 s_cell[kClusterThreads];  // (first, count, clusters before, -)
    __shared__ uint32_t s_cnt[NWARP][kNone];
    __shared__ uint4 s_warp[NWARP];
    __shared__ uint2 s_large[2];
    __shared__ uint32_t s_base;
    // the curve (constant memory serves one address at a time: 212 us for 5.88M
    // particles, now 166)
    __shared__ uint8_t s_place[64];
    if (__syncthreads_or(threadIdx.x == 0 && a.sc->err))
        return;  // one read for the whole block
    const bool octants = CELLS && sweep_by_octant(a.sc);
    if (threadIdx.x < 64)
        s_place[threadIdx.x] = D == 3 ? kHilbert3[threadIdx.x] : kHilbert2[threadIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t s0 = blockIdx.x * kClusterThreads + threadIdx.x;
    uint32_t n = 0;
    if (s0 < a.N) {
        const uint32_t key = a.skeys[s0];
        if (s0 == 0 || a.skeys[s0 - 1] != key)
            n = a.b.cells[key].y - s0;
    }
    const uint32_t P = a.cluster;  // 4 or 8
    // CELLS = false: the block's part of a cell of more than kLargeCell
    // particles, cut in sorted order
    uint32_t large = 0;  // the particles from this position on, if a cluster starts here
    if constexpr (!CELLS) {
        if (threadIdx.x == 0) {
            s_large[0] = s_large[1] = make_uint2(0u, 0u);
            if (n == 0 && s0 < a.N) {
                const uint2 se = a.b.cells[a.skeys[s0]];
                if (se.y - se.x > kLargeCell)
                    s_large[0] = se;
            }
        }
        __syncthreads();
        if (n > kLargeCell) {  // one at most
            s_large[1] = make_uint2(s0, s0 + n);
            n = 0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint2 se = s_large[k];
            if (s0 >= se.x && s0 < se.y) {
                a.b.cperm[s0] = s0;
                large = (s0 - se.x) % P == 0 ? se.y - s0 : 0u;
            }
        }
    }
    const unsigned lb = __ballot_sync(0xffffffffu, large > 0);
    const uint32_t ncl = (n + P - 1u) / P;
    // exclusive scan over the block: cells and clusters
    uint32_t xc = ncl;
    const unsigned starts = __ballot_sync(0xffffffffu, n > 0);
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, xc, o);
        if (lane >= o)
            xc += y;
    }
    if (lane == 31)
        s_warp[warp] = make_uint4((uint32_t)__popc(starts), xc, (uint32_t)__popc(lb), 0u);
    __syncthreads();
    uint32_t cells = 0, clusters = 0, n_cells = 0, n_clusters = 0;
    uint32_t larges = 0, n_large = 0;
    for (int w = 0; w < NWARP; w++) {
        const uint4 v = s_warp[w];
        if (w < warp) {
            cells += v.x;
            clusters += v.y;
            larges += v.z;
        }
        n_cells += v.x;
        n_clusters += v.y;
        n_large += v.z;
    }
    if (n > 0)
        s_cell[cells + __popc(starts & lt)] = make_uint4(s0, n, clusters + xc - ncl, 0u);
    if (threadIdx.x == 0)
        s_base = n_cells + n_large
                     ? atomicAdd(&a.sc->n_chunks, CELLS ? n_cells : n_clusters + n_large)
                     : 0u;
    __syncthreads();
    const uint32_t base = s_base;
    if (large)
        a.b.clu[base + n_clusters + larges + __popc(lb & lt)] = make_uint2(s0, min(P, large));
    for (uint32_t w = warp; w < n_cells; w += NWARP) {
        const uint4 cell = s_cell[w];
        const uint32_t first = cell.x, cnt = cell.y;
        const uint32_t kc = a.dst.cid[first];
        const CaseScalars& cs = a.cs[kc];
        // row (dy, dz) = (lane % 3 - 1, lane / 3 - 1) of the neighbourhood:
        // cells x-1 .. x+1, as one run of sorted indices (lanes 0-8; the cell
        // table is read here and the row written after the clusters, so the
        // loads overlap the work below)
        uint2 rc3[3] = { make_uint2(1u, 0u), make_uint2(1u, 0u), make_uint2(1u, 0u) };
        uint32_t key = 0;
        if (CELLS) {
            key = a.skeys[first];
            if (lane < 9) {
                const uint32_t nx = cs.n_cells[0];
                const uint32_t nxy = cs.n_cells[0] * cs.n_cells[1];
                const uint32_t k0 = key + (uint32_t)(lane % 3 - 1) * nx +
                                    (uint32_t)(lane / 3 - 1) * nxy - 1u;
                for (int d = 0; d < 3; d++)
                    rc3[d] = a.b.cells[k0 + d];
            }
        }
        uint32_t walls = 0, probes = 0;
        // clusters by octant: their number (0: none) and, lane k, the first
        // place and the particles of cluster k
        uint32_t nko = 0, oat = 0, on = 0;
        if (cnt > P || CELLS) {
            const float scale = (D == 3 ? 4.f : 8.f) * c.idist;
            auto place = [&](uint32_t s) -> uint32_t {
                const int im = a.dst.imove[s];
                if (im <= 0)
                    return im == 0 ? kProbes : kWalls;
                const float4 p = pos[s];
                const uint32_t x = (uint32_t)((p.x - cs.r_min[0]) * scale);
                const uint32_t y = (uint32_t)((p.y - cs.r_min[1]) * scale);
                if (D == 2)
                    return s_place[(x & 7u) | ((y & 7u) << 3)];
                const uint32_t z = (uint32_t)((p.z - cs.r_min[2]) * scale);
                return s_place[(x & 3u) | ((y & 3u) << 2) | ((z & 3u) << 4)];
            };
            __syncwarp();
            s_cnt[warp][lane] = 0;
            s_cnt[warp][32 + lane] = 0;
            if (lane < 2)
                s_cnt[warp][kWalls + lane] = 0;
            __syncwarp();
            for (uint32_t b = 0; b < cnt; b += 32) {
                const bool v = b + lane < cnt;
                const uint32_t g = v ? place(first + b + lane) : kNone;
                const unsigned m = __match_any_sync(0xffffffffu, g);
                if (v && lane == __ffs(m) - 1)
                    s_cnt[warp][g] += (uint32_t)__popc(m);
                __syncwarp();
            }
            // counts -> first positions (lane holds places 2 lane, 2 lane + 1)
            const uint32_t c0 = s_cnt[warp][2 * lane], c1 = s_cnt[warp][2 * lane + 1];
            walls = s_cnt[warp][kWalls];
            probes = s_cnt[warp][kProbes];
            uint32_t x = c0 + c1;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o)
                    x += y;
            }
            if (octants) {
                uint32_t prev = 0, start = 0, open = 0;
                bool fit = true;
                for (int o = 0; o < 8; o++) {
                    const uint32_t end = __shfl_sync(0xffffffffu, x, 4 * o + 3);
                    const uint32_t co = end - prev;
                    fit = fit && co <= 8u;
                    if (open + co > 8u) {
                        nko++;
                        start = prev;
                        open = 0;
                    }
                    open += co;
                    prev = end;
                    if (lane == (int)nko) {
                        oat = start;
                        on = open;
                    }
                }
                nko++;
                if (!fit || prev == 0)
                    nko = 0;
            }
            __syncwarp();
            s_cnt[warp][2 * lane] = x - c0 - c1;
            s_cnt[warp][2 * lane + 1] = x - c1;
            if (lane == 0) {
                s_cnt[warp][kWalls] = cnt - probes - walls;
                s_cnt[warp][kProbes] = cnt - probes;
            }
            __syncwarp();
            for (uint32_t b = 0; b < cnt; b += 32) {
                const bool v = b + lane < cnt;
                const uint32_t s = first + b + lane;
                const uint32_t g = v ? place(s) : kNone;
                const unsigned m = __match_any_sync(0xffffffffu, g);
                if (v)
                    a.b.cperm[first + s_cnt[warp][g] + (uint32_t)__popc(m & lt)] = s;
                __syncwarp();
                if (v && lane == __ffs(m) - 1)
                    s_cnt[warp][g] += (uint32_t)__popc(m);
                __syncwarp();
            }
        } else if ((uint32_t)lane < cnt) {
            a.b.cperm[first + lane] = first + lane;
        }
        // clusters of the others, of the boundary elements and of the probes;
        // at most as many as particles
        // (CELLS = false: only the order, the list has ceil(cnt / P) places)
        const uint32_t n0 = CELLS ? cnt - probes - walls : cnt, n1 = CELLS ? cnt - probes : cnt;
        const uint32_t k0 = nko ? nko : (n0 + P - 1u) / P;
        const uint32_t k1 = k0 + (n1 - n0 + P - 1u) / P;
        const uint32_t nk = k1 + (cnt - n1 + P - 1u) / P;
        const uint32_t slot0 = CELLS ? first : base + cell.z;
        for (uint32_t k = lane; k < nk; k += 32) {
            const uint32_t at = k < k0   ? P * k
                                : k < k1 ? n0 + P * (k - k0)
                                         : n1 + P * (k - k1);
            const uint32_t end = k < k0 ? n0 : k < k1 ? n1 : cnt;
            a.b.clu[slot0 + k] = k < nko ? make_uint2(first + oat, on)
                                         : make_uint2(first + at, min(P, end - at));
        }
        if (CELLS) {
            if (lane == 0) {
                a.b.work[base + w] = make_uint2(key, first);
                a.b.wcl[base + w] = make_uint4(first, first + cnt, kc, nk);
            }
            if (lane < 9) {
                uint32_t lo = 0xffffffffu, hi = 0;
                for (int d = 0; d < 3; d++) {
                    if (rc3[d].x < rc3[d].y) {
                        lo = min(lo, rc3[d].x);
                        hi = max(hi, rc3[d].y);
                    }
                }
                a.b.crow[(size_t)(base + w) * 9 + lane] =
                    hi > lo ? make_uint2(lo, hi - lo) : make_uint2(0u, 0u);
            }
        }
    }
}

// Looks whether the particles lie on a lattice: the cells of kOctantCells of them,
// the clusters that the fluid makes by whole octants (joined while they fit into
// 8; an octant of more counts as many as its particles) and as cuts of 8.
constexpr uint32_t kOctantCells = 2048;
__global__ void __launch_bounds__(256)
k_octants(Consts c, StepArgs a)
{
    __shared__ uint32_t s_sum[2];
    if (threadIdx.x < 2)
        s_sum[threadIdx.x] = 0;
    if (__syncthreads_or(threadIdx.x == 0 && a.sc->err))
        return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w = blockIdx.x * 8u + (threadIdx.x >> 5);
    const uint32_t s0 = (uint32_t)((uint64_t)w * a.N / kOctantCells);
    const uint2 se = a.b.cells[a.skeys[s0]];
    const CaseScalars& cs = a.cs[a.dst.cid[s0]];
    const float scale = 4.f * c.idist;
    uint32_t n = 0;  // lane o < 8: particles of octant o along the curve
    for (uint32_t b = se.y - se.x > kLargeCell ? se.y : se.x; b < se.y; b += 32) {
        uint32_t o = 8;
        if (b + lane < se.y && a.dst.imove[b + lane] > 0) {
            const float4 p = a.b.rec0[b + lane];
            const uint32_t x = (uint32_t)((p.x - cs.r_min[0]) * scale) & 3u;
            const uint32_t y = (uint32_t)((p.y - cs.r_min[1]) * scale) & 3u;
            const uint32_t z = (uint32_t)((p.z - cs.r_min[2]) * scale) & 3u;
            o = kHilbert3[x | (y << 2) | (z << 4)] / 8u;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const unsigned m = __ballot_sync(0xffffffffu, o == k);
            if (lane == k)
                n += (uint32_t)__popc(m);
        }
    }
    uint32_t total = 0, clusters = 0, open = 0;
    for (int o = 0; o < 8; o++) {
        const uint32_t co = __shfl_sync(0xffffffffu, n, o);
        total += co;
        if (co > 8u) {
            clusters += co;
            continue;
        }
        if (open + co > 8u) {
            clusters++;
            open = 0;
        }
        open += co;
    }
    clusters += open > 0;
    if (lane == 0 && total > 8u) {
        atomicAdd(&s_sum[0], clusters);
        atomicAdd(&s_sum[1], (total + 7u) / 8u);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_sum[1]) {
        atomicAdd(&a.sc->by_octant, s_sum[0]);
        atomicAdd(&a.sc->by_cut, s_sum[1]);
    }
}

// End of step of every case: dt = min(dt_var) (Reduction tool), assert
// dt > 0, t += dt, iter += 1 (set_scalar tools); for a rolling case, the new
// roll angle and rate at the new time (the reference's motion tools run
// after the time step, cfd/motion.xml:59-71).
__global__ void
k_finalize(DevScalars* sc, CaseScalars* cs, const CaseMotion* cm,
           uint32_t n_cases)
{
    if (sc->err)
        return;
    for (uint32_t k = threadIdx.x; k < n_cases; k += blockDim.x) {
        CaseScalars& c = cs[k];
        const float dt = __uint_as_float(c.dt_next);
        if (!(dt > 0.f) || isinf(dt)) {
            atomicOr(&sc->err, kErrDt);
            continue;
        }
        c.dt = dt;
        c.t = (float)((double)c.t + (double)dt);
        c.iter = c.iter + 1;
        if (cm[k].enabled) {
            const double w = (double)cm[k].angular_freq;
            const double A = (double)cm[k].amplitude;
            const double psi = A * sin(w * (double)c.t);
            c.psi_in = c.psi;
            c.cos_psi_in = c.cos_psi;
            c.sin_psi_in = c.sin_psi;
            c.psi = (float)psi;
            c.omega = (float)(A * w * cos(w * (double)c.t));
            c.cos_psi = (float)cos((double)c.psi);
            c.sin_psi = (float)sin((double)c.psi);
        }
    }
}

// Prescribed roll of the boundary elements and probes of a moving case
// about `center` (z axis): un-transform with the previous angle, velocity
// from the new rate, transform with the new angle
// (cfd/Motions/UnTransform.cl, Velocity.cl, Transform.cl).
template<int D>
__global__ void __launch_bounds__(256)
k_motion(StepArgs a)
{
    constexpr int VS = Vec<D>::VS;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.N || a.sc->err)
        return;
    const VarSet& T = a.dst;
    const uint32_t k = T.cid[i];
    const CaseMotion& m = a.cm[k];
    if (!m.enabled || T.iset[i] != m.iset || T.imove[i] == 1)
        return;
    const CaseScalars& c = a.cs[k];
    float r[4], n[4], t[4];
    Vec<D>::load(T.r, i, r);
    Vec<D>::load(T.normal, i, n);
    Vec<D>::load(T.tangent, i, t);
    // un-transform (rotation by -psi_in about z, around the centre)
    for (int d = 0; d < VS; d++)
        r[d] = r[d] - m.center[d];
    const float ci = c.cos_psi_in, si = -c.sin_psi_in;
    float rl[4], nl[4], tl[4];
    for (int d = 0; d < 4; d++) {
        rl[d] = r[d];
        nl[d] = n[d];
        tl[d] = t[d];
    }
    rl[0] = ci * r[0] - si * r[1];
    rl[1] = si * r[0] + ci * r[1];
    nl[0] = ci * n[0] - si * n[1];
    nl[1] = si * n[0] + ci * n[1];
    tl[0] = ci * t[0] - si * t[1];
    tl[1] = si * t[0] + ci * t[1];
    // velocity of the rotation in the local frame, then rotated
    const float cp = c.cos_psi, sp = c.sin_psi;
    float ul[4] = { 0.f, 0.f, 0.f, 0.f }, u[4] = { 0.f, 0.f, 0.f, 0.f };
    ul[0] = -c.omega * rl[1];
    ul[1] = c.omega * rl[0];
    u[0] = cp * ul[0] - sp * ul[1];
    u[1] = sp * ul[0] + cp * ul[1];
    // transform with the new angle
    float ro[4], no[4], to[4];
    for (int d = 0; d < 4; d++) {
        ro[d] = rl[d];
        no[d] = nl[d];
        to[d] = tl[d];
    }
    ro[0] = cp * rl[0] - sp * rl[1];
    ro[1] = sp * rl[0] + cp * rl[1];
    no[0] = cp * nl[0] - sp * nl[1];
    no[1] = sp * nl[0] + cp * nl[1];
    to[0] = cp * tl[0] - sp * tl[1];
    to[1] = sp * tl[0] + cp * tl[1];
    for (int d = 0; d < VS; d++)
        ro[d] = ro[d] + m.center[d];
    float nn = 0.f, tt = 0.f;
    for (int d = 0; d < VS; d++) {
        nn = nn + no[d] * no[d];
        tt = tt + to[d] * to[d];
    }
    nn = sqrtf(nn);
    tt = sqrtf(tt);
    for (int d = 0; d < VS; d++) {
        no[d] = no[d] / nn;
        to[d] = to[d] / tt;
    }
    Vec<D>::store(T.r, i, ro);
    Vec<D>::store(T.normal, i, no);
    Vec<D>::store(T.tangent, i, to);
    Vec<D>::store(T.u, i, u);
}

// One launch for the copies of a state (and its records): a copy call each
// costs 2 us and more a field on the GPU, 27 fields a state in and out (5
// tanks, 46,545 particles: 296 us a pass, then 209; 406,402 in 3-D: 1,029,
// then 866).  Sixteen-byte words where both ends are aligned to them; the rows
// of the grid's y dimension are the spans.
constexpr int kSpanThreads = 256;
__global__ void __launch_bounds__(kSpanThreads)
k_copy_spans(CopySpans sp, StateRecords rec)
{
    const uint32_t y = blockIdx.y;
    const uint64_t t0 = blockIdx.x * (uint64_t)kSpanThreads + threadIdx.x;
    const uint64_t step = (uint64_t)gridDim.x * kSpanThreads;
    if ((int)y < sp.n) {
        uint32_t* d = sp.dst[y];
        const uint32_t* s = sp.src[y];
        const uint64_t n = sp.words[y];
        uint64_t done = 0;
        if (((reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(s)) & 15) == 0) {
            const uint64_t q = n / 4;
            uint4* d4 = reinterpret_cast<uint4*>(d);
            const uint4* s4 = reinterpret_cast<const uint4*>(s);
            for (uint64_t k = t0; k < q; k += 4 * step) {
                uint4 v[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (k + u * step < q)
                        v[u] = s4[k + u * step];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (k + u * step < q)
                        d4[k + u * step] = v[u];
            }
            done = q * 4;
        }
        for (uint64_t k = done + t0; k < n; k += step)
            d[k] = s[k];
        return;
    }
    // the last row: case ids and records
    if (!rec.cid)
        return;
    for (uint64_t k = t0; k < rec.N; k += step)
        rec.cid[k] = 0;
    if (t0 == 0) {
        *rec.sc = rec.sc0;
        rec.cs[0] = rec.cs0;
        rec.cm[0] = rec.cm0;
        rec.offsets[0] = 0;
        rec.offsets[1] = rec.N;
    }
}

// case id of every particle from the case offsets
__global__ void
k_set_case_ids(uint32_t* cid, const uint32_t* offsets, uint32_t n_cases,
               uint32_t N)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N)
        return;
    uint32_t lo = 0, hi = n_cases;  // offsets[lo] <= i < offsets[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (offsets[mid] <= i)
            lo = mid;
        else
            hi = mid;
    }
    cid[i] = lo;
}

__global__ void
k_export_ihoc(const uint2* cells, uint32_t* ihoc, uint32_t ncap,
              const DevScalars* sc)
{
    const uint32_t nw = sc->total_cells;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncap && c < nw;
         c += gridDim.x * blockDim.x)
        ihoc[c] = cells[c].x;
}

}  // namespace

template<int D>
cudaError_t
launch_gather(bool fast, const Consts& c, const StepArgs& a, cudaStream_t s)
{
    return fast ? fast::launch_gather_impl<D>(c, a, s)
                : exact::launch_gather_impl<D>(c, a, s);
}

template<int D>
cudaError_t
launch_sweep(bool fast, const Consts& c, const StepArgs& a, unsigned grid,
             int variant, cudaStream_t s)
{
    if (a.N) {
        k_chunks<<<(a.N + kChunkThreads - 1) / kChunkThreads, kChunkThreads, 0,
                   s>>>(a.skeys, a.b.cells, a.N, a.b.chunks, a.sc);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return e;
    }
    return fast ? fast::launch_sweep_impl<D>(c, a, grid, variant, s)
                : exact::launch_sweep_impl<D>(c, a, grid, variant, s);
}

template<int D>
cudaError_t
launch_clusters(const Consts& c, const StepArgs& a, cudaStream_t s)
{
    if (a.N == 0)
        return cudaSuccess;
    const unsigned grid = (a.N + kClusterThreads - 1) / kClusterThreads;
    if (D == 3 && a.clustered && a.N > kOctantMin)
        k_octants<<<kOctantCells / 8, 256, 0, s>>>(c, a);
    if (D == 3 && a.clustered)
        k_cell_clusters<3, true><<<grid, kClusterThreads, 0, s>>>(c, a, a.b.rec0);
    else
        k_cell_clusters<D, false><<<grid, kClusterThreads, 0, s>>>(c, a, a.b.posq);
    return cudaGetLastError();
}

template<int D>
cudaError_t
launch_sweep_quad(bool fast, const Consts& c, const StepArgs& a, unsigned sms,
                  cudaStream_t s)
{
    return fast ? fast::launch_sweep_quad_impl<D>(c, a, sms, s)
                : exact::launch_sweep_quad_impl<D>(c, a, sms, s);
}

template<int D>
cudaError_t
launch_bi_walls(bool fast, const Consts& c, const StepArgs& a, unsigned sms,
                cudaStream_t s)
{
    return fast ? fast::launch_bi_walls_impl<D>(c, a, sms, s)
                : exact::launch_bi_walls_impl<D>(c, a, sms, s);
}

cudaError_t
launch_finalize(DevScalars* sc, CaseScalars* cs, const CaseMotion* cm,
                uint32_t n_cases, cudaStream_t s)
{
    k_finalize<<<1, 256, 0, s>>>(sc, cs, cm, n_cases);
    return cudaGetLastError();
}

template<int D>
cudaError_t
launch_motion(const StepArgs& a, cudaStream_t s)
{
    if (a.N == 0)
        return cudaSuccess;
    k_motion<D><<<(a.N + 255) / 256, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t
launch_copy_spans(const CopySpans& sp, const StateRecords& rec, cudaStream_t s)
{
    uint64_t most = rec.cid ? rec.N : 0;
    for (int k = 0; k < sp.n; k++)
        most = sp.words[k] > most ? sp.words[k] : most;
    if (most == 0)
        return cudaSuccess;
    // four 16-byte words a thread, at most 16 blocks a row and SM
    const uint64_t blocks = (most + kSpanThreads * 16ull - 1) / (kSpanThreads * 16ull);
    const unsigned gx = (unsigned)(blocks < 152ull * 16 ? blocks : 152ull * 16);
    k_copy_spans<<<dim3(gx, (unsigned)sp.n + (rec.cid ? 1u : 0u)), kSpanThreads, 0, s>>>(sp, rec);
    return cudaGetLastError();
}

cudaError_t
launch_set_case_ids(uint32_t* cid, const uint32_t* offsets, uint32_t n_cases,
                    uint32_t N, cudaStream_t s)
{
    if (N == 0)
        return cudaSuccess;
    k_set_case_ids<<<(N + 255) / 256, 256, 0, s>>>(cid, offsets, n_cases, N);
    return cudaGetLastError();
}

cudaError_t
launch_export_ihoc(const uint2* cells, uint32_t* ihoc, uint32_t ncap,
                   const DevScalars* sc, cudaStream_t s)
{
    const unsigned g = min((ncap + 255u) / 256u, 152u * 8u);
    k_export_ihoc<<<g > 0 ? g : 1u, 256, 0, s>>>(cells, ihoc, ncap, sc);
    return cudaGetLastError();
}

template cudaError_t launch_bi_walls<2>(bool, const Consts&, const StepArgs&,
                                        unsigned, cudaStream_t);
template cudaError_t launch_bi_walls<3>(bool, const Consts&, const StepArgs&,
                                        unsigned, cudaStream_t);
template cudaError_t launch_clusters<2>(const Consts&, const StepArgs&, cudaStream_t);
template cudaError_t launch_clusters<3>(const Consts&, const StepArgs&, cudaStream_t);
template cudaError_t launch_sweep_quad<2>(bool, const Consts&, const StepArgs&,
                                          unsigned, cudaStream_t);
template cudaError_t launch_sweep_quad<3>(bool, const Consts&, const StepArgs&,
                                          unsigned, cudaStream_t);
template cudaError_t launch_motion<2>(const StepArgs&, cudaStream_t);
template cudaError_t launch_motion<3>(const StepArgs&, cudaStream_t);
template cudaError_t launch_gather<2>(bool, const Consts&, const StepArgs&, cudaStream_t);
template cudaError_t launch_gather<3>(bool, const Consts&, const StepArgs&, cudaStream_t);
template cudaError_t launch_sweep<2>(bool, const Consts&, const StepArgs&, unsigned,
                                     int, cudaStream_t);
template cudaError_t launch_sweep<3>(bool, const Consts&, const StepArgs&, unsigned,
                                     int, cudaStream_t);

}  // namespace aqua
