// colo_bucket.cu -- grid bucketing: a stable radix sort of points by cell key
// into a cell CSR with (cell, feature) runs, per-cell feature masks and the
// geometric 3x3 occupied-neighbour table; then the per-cell neighbourhood
// lists that the join walks.
//
// Replaces CountCellFeatures (Codes/DeviceProcess.cu:312-369) and
// kernel_CountCellFeatures (Codes/DeviceProcess_Kernel.h:629-647): instead of
// dense totalCells x F count/start arrays, only occupied cells and runs are
// stored, so grids of 10^10 cells cost nothing.
#include <algorithm>

#include "colo_batch.h"
#include "colo_device.cuh"

namespace colo {
namespace {

// Cell keys, packed coordinates, cleared neighbour counts and (vals non-null)
// point ids, and the digit starts of every radix pass over the keys
// (block-private counts added to hist once per block; the last block to finish
// scans them in place), so the sort does not read the keys again to count
// them.  When the sort runs a pass its first pass makes the ids itself.
template <class KT>
__global__ void __launch_bounds__(256, 4) k_cell_keys(
    uint64_t n, uint32_t F, const uint32_t* __restrict__ fstart, const uint32_t* __restrict__ fjob,
    const JobGrid* __restrict__ grids, KT* __restrict__ keys, uint32_t* __restrict__ vals, float2* __restrict__ xy, uint32_t* __restrict__ nb_cnt,
    BatchCtrl* __restrict__ ctrl, RadixPlan plan, unsigned long long* __restrict__ hist) {
    static_assert(kRadixDigits == 512, "two digits a thread in the scan");
    __shared__ uint32_t h[kRadixMaxPasses * kRadixDigits];
    __shared__ bool s_last;
    for (int i = threadIdx.x; i < plan.n * kRadixDigits; i += blockDim.x) h[i] = 0;
    __syncthreads();
    // each block takes one contiguous range of points (coalesced, and a
    // thread's successive points are blockDim apart, so the feature found for
    // one point usually covers the next)
    const uint64_t per = ((n + gridDim.x - 1) / gridDim.x + blockDim.x - 1) / blockDim.x * blockDim.x;
    const uint64_t i0 = (uint64_t)blockIdx.x * per, i1 = i0 + per < n ? i0 + per : n;
    uint32_t f = 0, flo = 1, fhi = 0;   // cached feature, its point range [flo, fhi) and its job
    JobGrid g{};
    auto seek = [&](uint64_t i) {
        if (i >= flo && i < fhi) return;
        f = feature_of((uint32_t)i, F, fstart);
        flo = fstart[f];
        fhi = f + 1 < F ? fstart[f + 1] : (uint32_t)n;
        g = grids[fjob[f]];
    };
    auto put = [&](uint64_t i, float xi, float yi) {
        xy[i] = make_float2(xi, yi);
        nb_cnt[i] = 0;
        uint64_t c = ref_cell(g, xi, yi);
        if (c >= g.total) {
            atomicAdd(&ctrl->flags.out_of_grid, 1u);
            c = g.total - 1;
        }
        const KT key = (KT)(g.key_base + c);
        keys[i] = key;
        if (vals) vals[i] = (uint32_t)i;
        for (int p = 0; p < plan.n; ++p)
            atomicAdd(&h[p * kRadixDigits + ((uint32_t)(key >> plan.shift[p]) & ((1u << plan.width[p]) - 1u))], 1u);
    };
    // several points' coordinates in flight (the loads come from memory or over the host link)
    constexpr int kUnroll = 4;
    for (uint64_t i = i0 + threadIdx.x; i < i1; i += (uint64_t)kUnroll * blockDim.x) {
        seek(i);
        const uint64_t last = i + (uint64_t)(kUnroll - 1) * blockDim.x;
        if (last < i1 && last < fhi) {   // one feature
            float xs[kUnroll], ys[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const uint64_t q = i - g.p0 + (uint64_t)u * blockDim.x;
                xs[u] = __ldg(g.x + q);
                ys[u] = __ldg(g.y + q);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) put(i + (uint64_t)u * blockDim.x, xs[u], ys[u]);
        } else {
            for (uint64_t q = i; q <= last && q < i1; q += blockDim.x) {
                seek(q);
                put(q, __ldg(g.x + (q - g.p0)), __ldg(g.y + (q - g.p0)));
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < plan.n * kRadixDigits; i += blockDim.x) {
        const uint32_t v = h[i];
        if (v) atomicAdd(&hist[i], (unsigned long long)v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&ctrl->keys_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int p = 0; p < plan.n; ++p) {
        unsigned long long* hp = hist + p * kRadixDigits + 2 * threadIdx.x;
        unsigned long long tot;
        const unsigned long long v = __ldcg(hp), v1 = __ldcg(hp + 1);
        const unsigned long long at = block_excl_scan<unsigned long long>(v + v1, &tot);
        hp[0] = at;
        hp[1] = at + v;
    }
}

// Cells and runs in one pass over the sorted keys.  A block takes a 2048-point
// tile (eight warp segments of 256 points, 32 consecutive points at a time): per
// point its feature (from the feature start table, points being grouped by
// feature; it stays in L1); a cell starts where the key changes, a run where the
// key or the feature does (a point's predecessor comes from the lane before it,
// lane 0's from the last lane of the round before).  The features of four rounds
// are searched side by side, which hides most of the chain of dependent loads
// (20M points, nothing gathered: 297 -> 200 us; one search at a time without lane
// 0's second search 273, eight at a time 198, the starts in shared memory 207).
// The tile's head counts go through a decoupled look-back (warp 0 for cells, warp
// 1 for runs), and the heads are written at the offsets found, as far as the
// arrays reach (capM, capR: a launch with no room counts them).
// The last tile records the totals and the end entries.
//
// GATHER also writes the points' coordinates in cell order (and, for several jobs,
// their features), which makes the lists' and the join's reads of them nearly
// sequential.  The 8-byte reads by id move a DRAM sector each once the
// coordinates outgrow L2, for every point, and the join looks at a tenth of them:
// from kGatherPoints on they stay in id order and the lists hold ids (20M points:
// this kernel 495 -> 298 us, a mine 3.99 -> 3.83 ms; 1M to 4M: within 1% either
// way; 128 jobs of 30,000: 2% slower ungathered, so several jobs always gather).
//
// Bound by the gather, else by instruction issue and the wait for the look-back.
//
// After a sort that timed out the keys are not a sorted permutation: nothing
// is written, the totals stay zero and every later kernel finds no cells.  A
// look-back that waits too long counts the heads before its tile itself.
constexpr uint64_t kGatherPoints = 1ull << 23;   // 64 MiB of coordinates, half of L2
constexpr int kHeadThreads = 256, kHeadRounds = 8, kHeadTile = kHeadThreads * kHeadRounds;
constexpr int kHeadWarps = kHeadThreads / 32;

template <class KT, bool GATHER>
__global__ void __launch_bounds__(kHeadThreads, 6) k_heads(
    uint64_t n, uint32_t F, const KT* __restrict__ keys, const uint32_t* __restrict__ sid,
    const float2* __restrict__ xy, const uint32_t* __restrict__ fstart, const uint32_t* __restrict__ fjob,
    float2* __restrict__ sxy, uint32_t* __restrict__ sfeat, uint64_t* __restrict__ ckey,
    uint32_t* __restrict__ crun, uint32_t* __restrict__ cjob, uint32_t* __restrict__ rfeat,
    uint32_t* __restrict__ rstart, uint32_t* __restrict__ rcell, uint32_t* __restrict__ scell, uint64_t capM,
    uint64_t capR, unsigned long long* __restrict__ status, uint32_t* __restrict__ ticket,
    BatchCtrl* __restrict__ ctrl) {
    __shared__ uint32_t s_tile, s_heads[2][kHeadWarps];
    __shared__ unsigned long long s_prefix[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = ctrl->flags.timeout ? 0xffffffffu : atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile == 0xffffffffu) return;
    const uint64_t seg = (uint64_t)tile * kHeadTile + (uint64_t)w * (32 * kHeadRounds);
    KT key[kHeadRounds];
    uint32_t f[kHeadRounds], chm = 0, rhm = 0;   // the lane's own head bits, one a round
    uint32_t cc = 0, rc = 0;
    uint32_t top = 1;
    while (top < F && top < 1u << 31) top <<= 1;
#pragma unroll
    for (int r0 = 0; r0 < kHeadRounds; r0 += 4) {   // four searches at a time
        uint32_t id[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t p = seg + (uint64_t)(r0 + i) * 32 + lane;
            id[i] = p < n ? sid[p] : 0u;
            key[r0 + i] = p < n ? keys[p] : KT(0);
            f[r0 + i] = 0;
        }
        if (GATHER) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint64_t p = seg + (uint64_t)(r0 + i) * 32 + lane;
                if (p < n) sxy[p] = xy[id[i]];
            }
        }
        for (uint32_t step = top >> 1; step > 0; step >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t mid = f[r0 + i] + step;
                if (mid < F && fstart[mid] <= id[i]) f[r0 + i] = mid;
            }
        if (GATHER && sfeat) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint64_t p = seg + (uint64_t)(r0 + i) * 32 + lane;
                if (p < n) sfeat[p] = f[r0 + i];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kHeadRounds; ++r) {
        const uint64_t p = seg + (uint64_t)r * 32 + lane;
        const bool in = p < n;
        KT pkey = __shfl_up_sync(0xffffffffu, key[r], 1);
        uint32_t pf = __shfl_up_sync(0xffffffffu, f[r], 1);
        if (r > 0) {   // lane 0's predecessor: the last lane's point of the round before
            const KT k31 = __shfl_sync(0xffffffffu, key[r > 0 ? r - 1 : 0], 31);
            const uint32_t f31 = __shfl_sync(0xffffffffu, f[r > 0 ? r - 1 : 0], 31);
            if (lane == 0) {
                pkey = k31;
                pf = f31;
            }
        } else if (lane == 0 && in && p > 0) {
            pkey = keys[p - 1];
            pf = feature_of(sid[p - 1], F, fstart);
        }
        const bool ch = in && (p == 0 || pkey != key[r]);
        const bool rh = ch || (in && pf != f[r]);
        chm |= (ch ? 1u : 0u) << r;
        rhm |= (rh ? 1u : 0u) << r;
        cc += __popc(__ballot_sync(0xffffffffu, ch));
        rc += __popc(__ballot_sync(0xffffffffu, rh));
    }
    if (lane == 0) {
        s_heads[0][w] = cc;
        s_heads[1][w] = rc;
    }
    __syncthreads();
    if (w < 2) {
        uint32_t agg = 0;
        for (int i = 0; i < kHeadWarps; ++i) agg += s_heads[w][i];
        unsigned long long* st = status + (w == 0 ? 0 : gridDim.x);
        unsigned long long prefix;
        if (!warp_lookback(st, tile, agg, prefix)) {   // the heads before this tile, counted here
            unsigned long long add = 0;
            for (uint64_t p = lane; p < (uint64_t)tile * kHeadTile; p += 32) {
                const bool ch = p == 0 || keys[p - 1] != keys[p];
                add += ch || (w == 1 && feature_of(sid[p - 1], F, fstart) != feature_of(sid[p], F, fstart));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
            prefix = add;
            lookback_publish(st, tile, prefix + agg);
        }
        if (lane == 0) s_prefix[w] = prefix;
    }
    __syncthreads();
    uint32_t cb = (uint32_t)s_prefix[0], rb = (uint32_t)s_prefix[1];   // heads before this round
    for (int i = 0; i < w; ++i) {
        cb += s_heads[0][i];
        rb += s_heads[1][i];
    }
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < kHeadRounds; ++r) {
        const uint64_t p = seg + (uint64_t)r * 32 + lane;
        const bool ch = chm >> r & 1u, rh = rhm >> r & 1u;
        const uint32_t chb = __ballot_sync(0xffffffffu, ch), rhb = __ballot_sync(0xffffffffu, rh);
        const uint32_t c = cb + __popc(chb & lt) + (ch ? 1u : 0u) - 1u;   // the cell of p
        const uint32_t ri = rb + __popc(rhb & lt);
        if (scell && p < n) scell[p] = c;
        if (ch && c < capM) {
            ckey[c] = key[r];
            crun[c] = ri;
            cjob[c] = fjob[f[r]];
        }
        if (rh && ri < capR) {
            rfeat[ri] = f[r];
            rstart[ri] = (uint32_t)p;
            rcell[ri] = c;
        }
        cb += __popc(chb);
        rb += __popc(rhb);
    }
    // the warp of the last point ends with every head counted
    if (lane == 0 && seg < n && n - seg <= 32 * kHeadRounds) {
        ctrl->M = cb;
        ctrl->Rn = rb;
        if (cb <= capM && rb <= capR) {
            crun[cb] = rb;
            rstart[rb] = (uint32_t)n;
        }
    }
}

// Per cell its feature mask (bit lf of word lf / 32 for each of its runs' local
// features): a thread walks the cell's runs, which ascend by feature, and writes
// every word of the row (no clearing pass, no atomics).  The row table comes
// with it (rows > 0): rowstart[Y] = first occupied cell whose key is at or after
// the first key of grid row Y (rows of all jobs, job j's row y at Y = row_base_j
// + y), rowstart[rows] = M.  The runs per feature (frun) are counted in the same walk, in a
// block histogram when the features fit (a kernel of its own over the runs, with its copies and
// its wait, took 72 us on the 20M workload).
constexpr uint32_t kRunHist = 8192;

__global__ void k_cell_masks(const BatchCtrl* __restrict__ ctrl, const uint64_t* __restrict__ ckey,
                             const uint32_t* __restrict__ crun, const uint32_t* __restrict__ rfeat,
                             const uint32_t* __restrict__ cjob, const JobGrid* __restrict__ grids, uint32_t W,
                             uint32_t* __restrict__ cmask, uint64_t rows, uint32_t J, uint32_t* __restrict__ rowstart,
                             uint32_t F, uint32_t* __restrict__ frun) {
    extern __shared__ uint32_t s_run[];   // F counters (F <= kRunHist)
    const bool local = F <= kRunHist;
    const uint64_t M = ctrl->M;
    if (local)
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x) s_run[i] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t c = t0; c < M; c += step) {
        const uint32_t f0 = grids[cjob[c]].f0;
        uint32_t r = crun[c];
        const uint32_t r1 = crun[c + 1];
        uint32_t* row = cmask + c * W;
        for (uint32_t w = 0; w < W; ++w) {
            uint32_t bits = 0;
            for (; r < r1; ++r) {
                const uint32_t f = rfeat[r], lf = f - f0;
                if ((lf >> 5) != w) break;
                bits |= 1u << (lf & 31);
                atomicAdd(local ? &s_run[f] : &frun[f], 1u);
            }
            row[w] = bits;
        }
    }
    __syncthreads();
    if (local)
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x)
            if (s_run[i]) atomicAdd(&frun[i], s_run[i]);
    if (!rows) return;
    for (uint64_t Y = t0; Y <= rows; Y += step) {
        if (Y == rows) {
            rowstart[Y] = (uint32_t)M;
            break;
        }
        uint32_t lo = 0, hi = J;   // last job whose first row is <= Y
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (grids[mid].row_base <= Y) lo = mid;
            else hi = mid;
        }
        const JobGrid g = grids[lo];
        const uint64_t key = g.key_base + (Y - g.row_base) * g.gx;
        rowstart[Y] = (uint32_t)lower_bound_dev(ckey, (uint64_t)0, M, key);
    }
}

// A cell's occupied neighbours (nbrs[c]).  Keys ascend along a grid row, so the up
// to three neighbours of a row are consecutive cells: x and y are the positions of
// the first one in the row below (dy = -1) and above, the cell's own row surrounds c.
//   z bits 0-8    occupied, bit (dy+1)*3 + (dx+1)
//     bits 9-11   the reference's stencil takes column dx (bit 9 + dx+1)
//     bits 12-15  c is the first occupied cell of its quad q in (ey, ex) order (the
//                 level filter counts each full quad once, at that cell)
//     bits 16-19  quad q lies in the grid
//   w             the job's first feature
// Quad q has lower-left cell (cx+qx, cy+qy), qx = (q & 1) - 1, qy = (q >> 1) - 1, and
// holds c at corner (ex, ey) = (-qx, -qy); quads outside 0 <= bx <= gx-2,
// 0 <= by <= gy-2 are never full and are first nowhere.
//
// rowstart (optional, rows + 1 entries) bounds the search of a row to the
// cells of that row.  Bound by the searches' dependent loads (most of the
// instructions).  Nine positions and a byte a cell, 37 bytes in strided stores, made
// this 185 us, the quad masks 201 and the neighbourhood lists 192 at 20M points (8.3M
// cells); with these 16 bytes they take 167, 162 and 170.
__global__ void __launch_bounds__(128, 16) k_neighbours(const BatchCtrl* __restrict__ ctrl,
                                                        const uint64_t* __restrict__ ckey,
                                                        const uint32_t* __restrict__ cjob,
                                                        const JobGrid* __restrict__ grids,
                                                        const uint32_t* __restrict__ rowstart,
                                                        uint4* __restrict__ nbrs) {
    const uint64_t M = ctrl->M;
    for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < M; c += (uint64_t)gridDim.x * blockDim.x) {
        const JobGrid g = grids[cjob[c]];
        const uint64_t key = ckey[c];
        uint64_t ucx, ucy;
        cell_col_row(key - g.key_base, g.gx, ucx, ucy);
        const int64_t cx = (int64_t)ucx, cy = (int64_t)ucy;
        const int64_t x0 = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < (int64_t)g.gx ? cx + 1 : cx;
        uint32_t first[2] = {0, 0}, occ = 1u << 4;
        if (cx > 0 && c > 0 && ckey[c - 1] == key - 1) occ |= 1u << 3;
        if (cx + 1 < (int64_t)g.gx && c + 1 < M && ckey[c + 1] == key + 1) occ |= 1u << 5;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t ny = cy + 2 * r - 1;
            if (ny < 0 || ny >= (int64_t)g.gy) continue;
            const uint64_t row = g.key_base + (uint64_t)ny * g.gx, k0 = row + (uint64_t)x0, k1 = row + (uint64_t)x1;
            // 32-bit positions (M < 2^32): the search is most of this kernel's instructions
            uint32_t lo = r == 0 ? 0u : (uint32_t)c + 1u, hi = r == 0 ? (uint32_t)c : (uint32_t)M;
            if (rowstart) {
                const uint64_t Y = g.row_base + (uint64_t)ny;
                lo = rowstart[Y];
                hi = rowstart[Y + 1];
            }
            while (lo < hi) {
                const uint32_t mid = lo + ((hi - lo) >> 1);
                if (ckey[mid] < k0) lo = mid + 1;
                else hi = mid;
            }
            first[r] = lo;
            for (uint32_t pos = lo; pos < (uint32_t)M; ++pos) {
                const uint64_t k = ckey[pos];
                if (k > k1) break;
                occ |= 1u << (r * 6 + 1 + (int)((int64_t)(k - row) - cx));
            }
        }
        uint32_t bits = occ;
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
            if (ref_adjacent_col((uint32_t)cx, (uint32_t)(cx + dx), g.gx)) bits |= 1u << (10 + dx);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int qx = (q & 1) - 1, qy = (q >> 1) - 1;
            const int64_t bx = cx + qx, by = cy + qy;
            if (!(bx >= 0 && by >= 0 && bx + 2 <= (int64_t)g.gx && by + 2 <= (int64_t)g.gy)) continue;
            bits |= 1u << (16 + q);
            const int ex = -qx, ey = -qy;
            bool is_first = true;
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                if (e >= ey * 2 + ex) break;
                const int ox = (e & 1) - ex, oy = (e >> 1) - ey;
                if (occ >> ((oy + 1) * 3 + (ox + 1)) & 1u) is_first = false;
            }
            if (is_first) bits |= 1u << (12 + q);
        }
        nbrs[c] = make_uint4(first[0], first[1], bits, g.f0);
    }
}

// Neighbour q = (dy+1)*3 + (dx+1) of cell c, or -1 (there are fewer than 2^31 cells).
__device__ __forceinline__ int32_t neighbour(const uint4& v, uint32_t c, int q) {
    if (!(v.z >> q & 1u)) return -1;
    const uint32_t before = __popc(v.z & (((1u << (q % 3)) - 1u) << (q / 3 * 3)));
    const uint32_t at = q < 3 ? v.x : q < 6 ? c - (v.z >> 3 & 1u) : v.y;
    return (int32_t)(at + before);
}

// Per cell: the feature masks of the four quads (2x2 cell blocks) containing
// the cell, qmask[(c*4 + q)*W + w] with q = (qy+1)*2 + (qx+1) for the quad
// whose lower-left cell is (cx+qx, cy+qy), qx, qy in {-1, 0} -- q ascends in
// the quads' (by, bx) order.  A quad outside 0 <= bx <= gx-2,
// 0 <= by <= gy-2 gets an empty mask, so it is never full.
// nbmask[c*W + w] = union of the masks of the occupied cells of c's 3x3 block.
// One thread per cell and WT mask words (WT = W); rows are read and written
// as 16-byte vectors when W is a multiple of 4.
template <int WT>
__device__ __forceinline__ void ld_row(const uint32_t* __restrict__ p, uint32_t (&o)[WT]) {
    if constexpr (WT % 4 == 0) {
#pragma unroll
        for (int i = 0; i < WT / 4; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + i);
            o[4 * i] = v.x;
            o[4 * i + 1] = v.y;
            o[4 * i + 2] = v.z;
            o[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < WT; ++i) o[i] = __ldg(p + i);
    }
}

template <int WT>
__device__ __forceinline__ void st_row(uint32_t* __restrict__ p, const uint32_t (&v)[WT]) {
    if constexpr (WT % 4 == 0) {
#pragma unroll
        for (int i = 0; i < WT / 4; ++i)
            reinterpret_cast<uint4*>(p)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < WT; ++i) p[i] = v[i];
    }
}

constexpr int kQuadThreads = 128;

// Features a block of cells counts in shared memory for the driver-list sizes
// (larger batches count with global atomics).
constexpr uint32_t kQuadHist = 1024;

// Per cell: the 3x3 mask (nbmask), the queue of cells that need a neighbourhood
// list, the queue of cells with a quad of quad_min features or more, their four
// quad masks, and the driver-list sizes: dcnt[f] = cells of that queue whose 3x3
// mask holds f.  Most cells have no such quad (94% at 1M and at 20M points), and
// no pattern of three is bounded by them: without their 64 bytes of quad masks and
// their entries in the driver lists this kernel took 201 us instead of 262 at 20M
// points, the lists 27 instead of 157 and the level filters 334 instead of 430.  A block walks spans of consecutive cells (so that
// queued cells stay near each other: the list kernel reads their neighbourhoods)
// and keeps one histogram for all of them (one global atomic per
// feature per block at the end); a warp's 32 cells are counted by a bit
// transpose (lane b holds feature b's column of the warp's cell x feature
// matrix and adds its popcount).  Cells for the list queue collect in a small
// buffer of their warp, which is written out 32 at a time (one global atomic per
// 32 queued cells and no block barrier; an atomic and three barriers per 128
// cells made every warp wait for the atomic's round trip: 0.29 ms became 0.26 ms,
// 20M points).
template <int WT>
__global__ void __launch_bounds__(kQuadThreads) k_quad_masks(
    BatchCtrl* __restrict__ ctrl, const uint4* __restrict__ nbrs, const uint32_t* __restrict__ cmask,
    uint32_t* __restrict__ qmask, uint32_t* __restrict__ nbmask, uint32_t* __restrict__ listq,
    uint32_t* __restrict__ quadq, uint32_t* __restrict__ pairq, uint32_t quad_min, bool several, uint32_t F, uint32_t* __restrict__ dcnt) {
    const uint64_t M = ctrl->M;
    __shared__ uint32_t s_hist[kQuadHist];
    __shared__ uint32_t s_queue[kQuadThreads / 32][3][64];
    const bool local_hist = F <= kQuadHist;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (local_hist)
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    uint32_t listed = 0, quads = 0, pairs = 0;   // cells in the warp's buffers (below 32 between rounds)
    auto put = [&](uint32_t* queue, uint32_t& queued, bool mine, uint32_t c, LineCounter& total, uint32_t* out) {
        const uint32_t has = __ballot_sync(0xffffffffu, mine);
        if (mine) queue[queued + __popc(has & ((1u << lane) - 1u))] = c;
        queued += __popc(has);
        if (queued >= 32) {
            __syncwarp();
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&total.v, 32ull);
            out[__shfl_sync(0xffffffffu, at, 0) + lane] = queue[lane];
            queued -= 32;
            const uint32_t rest = (uint32_t)lane < queued ? queue[32 + lane] : 0u;
            __syncwarp();
            if ((uint32_t)lane < queued) queue[lane] = rest;
        }
    };
    auto flush = [&](const uint32_t* queue, uint32_t queued, LineCounter& total, uint32_t* out) {
        unsigned long long at = 0;
        if (lane == 0 && queued) at = atomicAdd(&total.v, (unsigned long long)queued);
        at = __shfl_sync(0xffffffffu, at, 0);
        if ((uint32_t)lane < queued) out[at + lane] = queue[lane];
    };
    // A warp takes 128 consecutive cells, 32 at a time, next to the block's other warps (32 when
    // there are too few for every block): its queued cells stay together, and blocks that run at
    // the same time read neighbouring rows (one far-apart range per block: 297 us, 20M points).
    const uint32_t rounds = M >= (uint64_t)gridDim.x * (4 * kQuadThreads) ? 4u : 1u;
    const uint64_t span = (uint64_t)rounds * kQuadThreads;
    for (uint64_t q0 = (uint64_t)blockIdx.x * span; q0 < M; q0 += (uint64_t)gridDim.x * span)
    for (uint32_t round = 0; round < rounds; ++round) {
        const uint64_t c = q0 + ((uint64_t)wid * rounds + round) * 32 + lane;
        bool above = false, useful = false, paired = false;
        uint32_t all[WT];
#pragma unroll
        for (int w = 0; w < WT; ++w) all[w] = 0;
        uint32_t f0 = 0;
        if (c < M) {
            const uint4 around = nbrs[c];
            f0 = around.w;
            int32_t nb[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) nb[q] = neighbour(around, (uint32_t)c, q);
            uint32_t m[9][WT];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                if (nb[q] >= 0) {
                    ld_row<WT>(cmask + (uint64_t)nb[q] * WT, m[q]);
                } else {
#pragma unroll
                    for (int w = 0; w < WT; ++w) m[q][w] = 0;
                }
#pragma unroll
                for (int w = 0; w < WT; ++w) all[w] |= m[q][w];
            }
            uint32_t feats = 0;
#pragma unroll
            for (int w = 0; w < WT; ++w) feats += __popc(all[w]);
            paired = feats >= 2;
            // the cell needs a neighbourhood list when its 3x3 block holds a
            // feature above its own lowest one (m[4] is the cell's own mask; the block
            // is the union over all nine slots, a superset of the adjacent cells):
            // such cells are queued for the list kernels
            bool seen = false;
#pragma unroll
            for (int w = 0; w < WT; ++w) {
                const uint32_t own = m[4][w];
                if (seen) {
                    above |= all[w] != 0;
                } else if (own) {
                    seen = true;
                    const uint32_t low = own & (0u - own);
                    above |= (all[w] & ~((low << 1) - 1u)) != 0;
                }
            }
            // the masks of quad q (empty where the quad leaves the grid)
            auto quad = [&](int q, uint32_t (&qm)[WT]) {
                const int qx = (q & 1) - 1, qy = (q >> 1) - 1;
                const bool valid = around.z >> (16 + q) & 1u;
                uint32_t n = 0;
#pragma unroll
                for (int w = 0; w < WT; ++w) {
                    qm[w] = valid ? (m[(qy + 1) * 3 + qx + 1][w] | m[(qy + 1) * 3 + qx + 2][w] |
                                     m[(qy + 2) * 3 + qx + 1][w] | m[(qy + 2) * 3 + qx + 2][w])
                                  : 0u;
                    n += __popc(qm[w]);
                }
                return n;
            };
            uint32_t qm[WT];
#pragma unroll
            for (int q = 0; q < 4; ++q) useful |= quad(q, qm) >= quad_min;
            // the readers: the driver lists (queued quads) and the pairs (queued pairs, or every run)
            if (!pairq || paired || useful) st_row<WT>(nbmask + c * WT, all);
            if (useful) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    quad(q, qm);
                    st_row<WT>(qmask + (c * 4 + q) * WT, qm);
                }
            } else {
#pragma unroll
                for (int w = 0; w < WT; ++w) all[w] = 0;   // in no driver list
            }
        }
        // driver-list sizes (lanes of another job than lane 0's, at job boundaries of a
        // batch, count one bit at a time)
        {
            const uint32_t fl = __shfl_sync(0xffffffffu, f0, 0);
            if (__all_sync(0xffffffffu, c >= M || f0 == fl)) {
#pragma unroll
                for (int w = 0; w < WT; ++w) {
                    if (!__any_sync(0xffffffffu, all[w])) continue;
                    const uint32_t f = fl + (uint32_t)w * 32 + (uint32_t)lane;
                    const uint32_t n = __popc(warp_transpose32(all[w]));
                    if (n) {
                        if (local_hist) atomicAdd(&s_hist[f], n);
                        else atomicAdd(&dcnt[f], n);
                    }
                }
            } else {
#pragma unroll
                for (int w = 0; w < WT; ++w)
                    for (uint32_t bits = all[w]; bits; bits &= bits - 1)
                        atomicAdd(&dcnt[f0 + (uint32_t)w * 32 + (uint32_t)(__ffs(bits) - 1)], 1u);
            }
        }
        put(s_queue[wid][0], listed, above, (uint32_t)c, ctrl->nlistq, listq);
        put(s_queue[wid][1], quads, useful, (uint32_t)c, ctrl->nquadq, quadq);
        if (pairq) put(s_queue[wid][2], pairs, paired, (uint32_t)c, ctrl->npairq, pairq);
        if (several && round + 1 == rounds) {   // the warp's next cells may be another job's
            __syncwarp();
            flush(s_queue[wid][1], quads, ctrl->nquadq, quadq);
            quads = 0;
        }
        __syncwarp();
    }
    flush(s_queue[wid][0], listed, ctrl->nlistq, listq);
    flush(s_queue[wid][1], quads, ctrl->nquadq, quadq);
    if (pairq) flush(s_queue[wid][2], pairs, ctrl->npairq, pairq);
    if (local_hist) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x)
            if (s_hist[i]) atomicAdd(&dcnt[i], s_hist[i]);
    }
}

// ---------------------------------------------------------------------------
// Neighbourhood lists.  For cell c the adjacent cells A(c) (the
// reference's stencil, ascending cell ids) contribute their runs; NRL(c)
// orders them by (feature, cell), which is the order the reference's kernels
// visit candidates of one feature.  For each run of c the list suffix with
// higher features holds exactly the join targets of the run's points.
// ---------------------------------------------------------------------------

__device__ __forceinline__ int adjacent_cells(uint32_t c, const uint4* __restrict__ nbrs, int32_t* out) {
    const uint4 around = nbrs[c];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int32_t v = neighbour(around, c, q);
        if (v >= 0 && (around.z >> (9 + q % 3) & 1u)) out[cnt++] = v;
    }
    return cnt;
}

// A cell's list keeps only the points of adjacent runs with a feature above the
// cell's lowest own feature: an anchor reads the list from its own run's suffix
// on, and the lowest own run's suffix starts past every entry of feature <= its
// own.  Most lists are then empty; the cells whose 3x3 mask allows one were
// queued by k_quad_masks.

// The bounds lie where the kernel's time is flat on 14 workloads (within 5%) with half and twice of each, but
// for these: 64 runs 117 -> 147 us and 16 anchors 117 -> 143 (400,000 clustered points; 64 anchors 100 there,
// the same elsewhere), 256 points 411 -> 556 (a batch of 128 jobs).
constexpr uint32_t kBigRuns = 128, kBigPoints = 512;   // cells with longer lists are merged by their whole warp
constexpr uint32_t kHeavyAnchors = 32;   // cells with more anchors are listed by their whole warp

// The point at sorted position p as lists and anchors name it: by that position
// where the coordinates were gathered (ids is null), else by its id.
__device__ __forceinline__ uint32_t list_point(const uint32_t* __restrict__ ids, uint32_t p) { return ids ? ids[p] : p; }

// The points at sorted positions st .. st + rc - 1 for every lane; runs of more
// than 32 points by the whole warp.
__device__ __forceinline__ void put_run(uint32_t* __restrict__ targets, uint64_t at, const uint32_t* __restrict__ ids,
                                        uint32_t st, uint32_t rc, int lane) {
    if (rc <= 32)
        for (uint32_t q = 0; q < rc; ++q) targets[at + q] = list_point(ids, st + q);
    for (uint32_t m = __ballot_sync(0xffffffffu, rc > 32); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const uint64_t aj = __shfl_sync(0xffffffffu, at, j);
        const uint32_t sj = __shfl_sync(0xffffffffu, st, j), nj = __shfl_sync(0xffffffffu, rc, j);
        for (uint32_t q = lane; q < nj; q += 32) targets[aj + q] = list_point(ids, sj + q);
    }
}

// The list of cell c by a whole warp, from `first` on.  In the full (feature,
// slot) order the points of a run of feature f in adjacent slot s start at the
// sum over slots of the points with a feature below f plus those of earlier
// slots' runs of f; the kept list drops the points of feature <= the cell's
// lowest own feature.  A slot's points are one range of sorted positions, so the
// points before a run are a difference of run starts, and a slot's runs below a feature
// are the bits below it in the cell's mask (ListRanks, in shared memory).  Per own run
// of the cell: the first target with a higher feature and the targets from there on.
// Binary searches for those ranks, a chain of loads each, took 147 us instead of 75 on
// 200,000 dense points.
struct ListRanks {
    uint32_t* first;   // [9] a slot's first run
    uint32_t* kept;    // [9] its first kept run
    uint32_t* start;   // [9] that run's first sorted position
    uint32_t* pre;     // [10] kept runs before the slot
    uint32_t* mask;    // [9][W]
    uint16_t* below;   // [9][W + 1]: bits in the words before; the last: all
    static __host__ __device__ size_t words(uint32_t W) { return 37 + 9 * W + (9 * (W + 1) + 1) / 2; }
    __device__ __forceinline__ ListRanks(uint32_t* at, uint32_t W)
        : first(at), kept(at + 9), start(at + 18), pre(at + 27), mask(at + 37),
          below(reinterpret_cast<uint16_t*>(at + 37 + 9 * W)) {}
    // runs of slot t with a local feature below lf
    __device__ __forceinline__ uint32_t rank(int t, uint32_t lf, uint32_t W) const {
        const uint32_t w = lf >> 5;
        return below[t * (W + 1) + w] + (w < W ? __popc(mask[t * W + w] & ((1u << (lf & 31)) - 1u)) : 0u);
    }
    __device__ __forceinline__ bool has(int t, uint32_t lf, uint32_t W) const { return mask[t * W + (lf >> 5)] >> (lf & 31) & 1u; }
};

__device__ __forceinline__ void list_cell_warp(uint32_t c, int lane, uint64_t first, uint32_t* room,
                                               const uint4* __restrict__ nbrs, const uint32_t* __restrict__ cmask,
                                               uint32_t W, const uint32_t* __restrict__ crun,
                                               const uint32_t* __restrict__ rfeat, const uint32_t* __restrict__ rstart,
                                               const uint32_t* __restrict__ ids, uint32_t* __restrict__ targets,
                                               uint64_t* run_sfx, uint32_t* run_L) {
    const ListRanks ranks(room, W);
    const uint4 around = nbrs[c];
    const uint32_t f0 = around.w, fmin = rfeat[crun[c]] - f0;
    __syncwarp();   // the ranks of the cell before may still be read
    int na = 0;
    uint32_t kept = 0;   // runs kept so far
    uint64_t total = 0;
    for (int q = 0; q < 9; ++q) {
        const int32_t v = neighbour(around, c, q);
        if (v < 0 || !(around.z >> (9 + q % 3) & 1u)) continue;
        const uint32_t word = (uint32_t)lane < W ? cmask[(uint64_t)v * W + lane] : 0u;
        const uint32_t n = __popc(word), incl = warp_incl_scan(n);
        if ((uint32_t)lane < W) {
            ranks.mask[na * W + lane] = word;
            ranks.below[na * (W + 1) + lane] = (uint16_t)(incl - n);
        }
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        if (lane == 31) ranks.below[na * (W + 1) + W] = (uint16_t)all;
        __syncwarp();
        const uint32_t r0 = crun[v], q0 = r0 + ranks.rank(na, fmin + 1, W), s0 = rstart[q0];
        if (lane == 0) {
            ranks.first[na] = r0;
            ranks.kept[na] = q0;
            ranks.start[na] = s0;
            ranks.pre[na] = kept;
        }
        kept += r0 + all - q0;
        total += rstart[r0 + all] - s0;
        ++na;
    }
    __syncwarp();
    for (uint32_t e0 = 0; e0 < kept; e0 += 32) {
        const uint32_t e = e0 + lane;
        uint64_t at = first;
        uint32_t st = 0, rc = 0;
        if (e < kept) {
            int sl = 0;
            while (sl + 1 < na && ranks.pre[sl + 1] <= e) ++sl;
            const uint32_t r = ranks.kept[sl] + (e - ranks.pre[sl]);
            const uint32_t lf = rfeat[r] - f0;
#pragma unroll 3
            for (int t = 0; t < na; ++t) {
                uint32_t lb = ranks.first[t] + ranks.rank(t, lf, W);
                if (t < sl && ranks.has(t, lf, W)) lb += 1;   // earlier slots' runs of f come first
                at += rstart[lb] - ranks.start[t];
            }
            st = rstart[r];
            rc = rstart[r + 1] - st;
        }
        put_run(targets, at, ids, st, rc, lane);
    }
    for (uint32_t r = crun[c] + lane; r < crun[c + 1]; r += 32) {
        const uint32_t lf = rfeat[r] - f0;
        uint64_t before = 0;
#pragma unroll 3
        for (int t = 0; t < na; ++t) before += rstart[ranks.first[t] + ranks.rank(t, lf + 1, W)] - ranks.start[t];
        run_sfx[r] = first + before;
        run_L[r] = (uint32_t)(total - before);
    }
}

// Neighbourhood lists and the join's anchors in one pass over the queued cells.
// A thread takes a cell: its list is the 9-way merge, by (feature, slot), of the
// adjacent cells' runs above the lowest own feature (each slot ascending by
// feature), written as the runs' points.  The running point count P gives the
// suffixes: the cell's own run of feature f reads the list from P targets on,
// P taken after every entry of feature <= f.  Then every point of an own run with
// targets is listed as an anchor, those with long lists from the array's back.
//
// Bound by the merge's chain of dependent loads.  The lists and anchors are not
// in cell order: a warp reserves its 32 cells' room with one atomic per total,
// so nothing is counted or scanned over the cells and runs beforehand (the order
// within a list is all that a result depends on).  With the two scans, the count
// and the clears that this replaces, 413 us of kernels became 147 us on the 20M
// workload when the lists still held runs (175 us now that they hold points, which
// takes the join from 325 to 78); the 200,000-point dense one, whose few long lists
// share a neighbourhood, 327 became 147, and 75 with ranks from the masks.
// Eight blocks an SM (64 registers) hide more of the chain than the six that the
// compiler's choice of registers left (154 against 172 us at 20M points, lists of runs).
// Lists past `cap` targets are not written; the host sees it in the total and runs
// the kernel again with room for all.
__global__ void __launch_bounds__(128, 8) k_neighbour_lists(
    uint64_t npoints, const uint32_t* __restrict__ listq, BatchCtrl* __restrict__ ctrl,
    const uint4* __restrict__ nbrs, const uint32_t* __restrict__ cmask, uint32_t W,
    const uint32_t* __restrict__ crun, const uint32_t* __restrict__ rfeat,
    const uint32_t* __restrict__ rstart, const uint32_t* __restrict__ ids, uint64_t cap,
    uint32_t* __restrict__ targets, uint64_t* run_sfx, uint32_t* run_L, uint4* __restrict__ act) {
    extern __shared__ uint32_t s_ranks[];   // a ListRanks a warp
    const uint32_t n = (uint32_t)ctrl->nlistq.v;
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5), w = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    // Consecutive cells share their neighbours, so a warp takes 32 consecutive ones.  A queue of
    // fewer than four cells a warp is dealt out one by one to as many warps as take 16 each: long
    // lists sit next to each other in it, and their merges then run side by side
    // (dense 200,000 points: 135 us against 353 us; lists elsewhere cost the same either way).
    const bool deal = n < 4 * nw;
    const uint64_t dealt = deal ? (n + 15) / 16 : 0;
    for (uint64_t i0 = deal ? w : w * 32; i0 < (deal ? dealt : n); i0 += nw * 32) {
        const uint64_t i = deal ? i0 + (uint64_t)lane * dealt : i0 + lane;
        const bool in = i < n && (!deal || lane < 16);
        uint32_t c = 0, r0 = 0, r1 = 0, kept = 0, points = 0;
        // each slot's cursor starts at its first run above the lowest own feature
        uint32_t h[9], e[9], f[9];
        int own = 0;
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            h[t] = e[t] = 0;
            f[t] = 0xffffffffu;
        }
        if (in) {
            c = listq[i];
            r0 = crun[c];
            r1 = crun[c + 1];
            const uint32_t fmin = rfeat[r0];
            int32_t adj[9];
            const int na = adjacent_cells(c, nbrs, adj);
#pragma unroll
            for (int t = 0; t < 9; ++t)
                if (t < na) {
                    e[t] = crun[adj[t] + 1];
                    h[t] = (uint32_t)lower_bound_dev(rfeat, (uint64_t)crun[adj[t]], (uint64_t)e[t], fmin + 1);
                    if (h[t] < e[t]) {
                        f[t] = rfeat[h[t]];
                        points += rstart[e[t]] - rstart[h[t]];
                    }
                    kept += e[t] - h[t];
                    if ((uint32_t)adj[t] == c) own = t;
                }
        }
        const uint64_t pincl = warp_incl_scan((uint64_t)points);
        const uint64_t ptot = __shfl_sync(0xffffffffu, pincl, 31);
        if (ptot == 0) continue;
        const uint32_t runs = __reduce_add_sync(0xffffffffu, kept);
        unsigned long long pb = 0;
        if (lane == 0) {
            pb = atomicAdd(&ctrl->targets.v, (unsigned long long)ptot);
            atomicAdd(&ctrl->list_runs.v, (unsigned long long)runs);
        }
        pb = __shfl_sync(0xffffffffu, pb, 0);
        if (pb + ptot > cap) continue;   // no room: the host runs the kernel again
        const uint64_t first = pb + (pincl - points);
        const bool big = kept > kBigRuns || points > kBigPoints;
        if (kept && !big) {
            // the lowest own run's suffix is the whole list
            run_sfx[r0] = first;
            run_L[r0] = points;
            for (uint32_t r = r0 + 1; r < r1; ++r) run_L[r] = 0;
            uint32_t P = 0, pend_r = 0, pend_f = 0;
            bool pend = false;
            for (;;) {
                int ts = 0;
                uint32_t fm = f[0];
#pragma unroll
                for (int t = 1; t < 9; ++t)
                    if (f[t] < fm) {
                        fm = f[t];
                        ts = t;
                    }
                if (fm == 0xffffffffu) break;
                if (pend && pend_f < fm) {
                    run_sfx[pend_r] = first + P;
                    run_L[pend_r] = points - P;
                    pend = false;
                }
                uint32_t r = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t)
                    if (t == ts) {
                        r = h[t]++;
                        f[t] = h[t] < e[t] ? rfeat[h[t]] : 0xffffffffu;
                    }
                const uint32_t st = rstart[r], rc = rstart[r + 1] - st;
                for (uint32_t q = 0; q < rc; ++q) targets[first + P + q] = list_point(ids, st + q);
                P += rc;
                if (ts == own) {
                    pend = true;
                    pend_r = r;
                    pend_f = fm;
                }
            }
        }
        for (uint32_t m = __ballot_sync(0xffffffffu, big); m; m &= m - 1) {   // the merge above is serial in the list
            const int j = __ffs(m) - 1;
            const uint32_t cj = __shfl_sync(0xffffffffu, c, j);
            const uint64_t fj = __shfl_sync(0xffffffffu, first, j);
            list_cell_warp(cj, lane, fj, s_ranks + (threadIdx.x >> 5) * ListRanks::words(W), nbrs, cmask, W, crun, rfeat, rstart, ids, targets, run_sfx, run_L);
        }
        __syncwarp();
        // anchors: the points of own runs with targets, short lists and long ones
        uint32_t ns = 0, nl = 0;
        uint64_t np = 0;
        if (kept)
            for (uint32_t r = r0; r < r1; ++r) {
                const uint32_t L = run_L[r];
                if (!L) continue;
                const uint32_t rc = rstart[r + 1] - rstart[r];
                if (L <= kLongList) ns += rc;
                else nl += rc;
                np += (uint64_t)rc * L;
            }
        const uint32_t sincl = warp_incl_scan(ns), lincl = warp_incl_scan(nl);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
        unsigned long long sb = 0, lb = 0;
        if (lane == 31) {
            if (sincl) sb = atomicAdd(&ctrl->anchors.v, (unsigned long long)sincl);
            if (lincl) lb = atomicAdd(&ctrl->long_anchors.v, (unsigned long long)lincl);
            if (np) atomicAdd(&ctrl->pairs.v, (unsigned long long)np);
        }
        uint64_t so = __shfl_sync(0xffffffffu, sb, 31) + (sincl - ns);
        uint64_t lo = npoints - 1 - (__shfl_sync(0xffffffffu, lb, 31) + (lincl - nl));   // downwards
        const bool heavy = ns + nl > kHeavyAnchors;
        if (ns + nl && !heavy)
            for (uint32_t r = r0; r < r1; ++r) {
                const uint32_t L = run_L[r];
                if (!L) continue;
                const uint32_t st = rstart[r], rc = rstart[r + 1] - st;
                const uint64_t sfx = run_sfx[r];
                for (uint32_t q = 0; q < rc; ++q)
                    act[L <= kLongList ? so++ : lo--] = make_uint4(list_point(ids, st + q), L, (uint32_t)sfx, (uint32_t)(sfx >> 32));
            }
        for (uint32_t m = __ballot_sync(0xffffffffu, heavy); m; m &= m - 1) {   // the loop above is serial in the points
            const int j = __ffs(m) - 1;
            const uint32_t s0 = __shfl_sync(0xffffffffu, r0, j), s1 = __shfl_sync(0xffffffffu, r1, j);
            uint64_t sj = __shfl_sync(0xffffffffu, so, j), lj = __shfl_sync(0xffffffffu, lo, j);
            for (uint32_t r = s0; r < s1; ++r) {   // the whole warp reads the run
                const uint32_t L = run_L[r];
                if (!L) continue;
                const uint32_t st = rstart[r], rc = rstart[r + 1] - st;
                const uint64_t sfx = run_sfx[r];
                const bool is_long = L > kLongList;
                for (uint32_t q = lane; q < rc; q += 32)
                    act[is_long ? lj - q : sj + q] = make_uint4(list_point(ids, st + q), L, (uint32_t)sfx, (uint32_t)(sfx >> 32));
                if (is_long) lj -= rc;
                else sj += rc;
            }
        }
    }
}

inline unsigned grid_for(uint64_t n, int threads) {
    uint64_t g = (n + threads - 1) / threads;
    return (unsigned)(g == 0 ? 1 : g);
}

}  // namespace

// A queue of cells for the pairs' bounds costs the quad masks up to 4 us and pays from here on: 2M
// points 41 -> 35 us for the two kernels, 4M 84 -> 65, 20M 319 -> 232; 1M 29 -> 33.
constexpr uint64_t kPairQueuePoints = 1ull << 21;

// Bounded batches reserve at most this much for arrays laid out by bounds (and no more than
// a sixteenth of the device, and blocks of 256 MiB and more no more than half of what is
// free); the 20M-point workload takes 5 GB.  Larger ones wait for the number of cells and
// runs before their per-cell arrays are laid out.
constexpr uint64_t kBoundBytes = 8ull << 30, kSmallBounds = 256ull << 20;
// Look-back words of all digit passes in one clear, up to this much and a 1024th of the device; above (67
// million points with eight passes, 89 with three of nine bits, 134 with four of eight) one pass's words
// are cleared before each pass.
constexpr uint64_t kSortStatusBytes = 256ull << 20;
// Room for the lists' targets and for neighbours before their numbers are known: four targets
// per point (nine at most: a point is adjacent to nine cells) and eight neighbours per point (0.14 on the 20M workload, 16 on that batch,
// 30 in dense clusters).  What does not fit is built again with the counted room.
inline uint64_t list_room(uint64_t n) { return std::min<uint64_t>(9 * n, 4 * n + 65536); }
inline uint64_t neighbour_room(const Batch& b) { return std::min<uint64_t>(b.single_cap(), 8 * b.N + 65536); }

namespace {

void lay_points(Batch& b, Carver& c) {
    c.add(b.xy, b.N);
    // written by every launch of the heads, one that only counts them too
    if (b.gathered) c.add(b.sxy, b.N);
    if (b.gathered && b.J > 1) c.add(b.sfeat, b.N);
    c.add(b.sid, b.N);
    c.add(b.nb_beg, b.N);
    c.add(b.nb_cnt, b.N);
}
void lay_heads(Batch& b, Carver& c, uint64_t M, uint64_t R) {
    c.add(b.ckey, M);
    c.add(b.crun, M + 1);
    c.add(b.cjob, M);
    c.add(b.rfeat, R);
    c.add(b.rstart, R + 1);
    c.add(b.rcell, R);
    if (b.keep_scell) c.add(b.scell, b.N);
}
void lay_cells(Batch& b, Carver& c, uint64_t M, uint64_t R) {
    c.add(b.cmask, M * b.W);
    c.add(b.nbmask, M * b.W);
    c.add(b.qmask, M * 4 * b.W);
    c.add(b.nbrs, M);
    c.add(b.listq, M);
    c.add(b.quadq, M);
    if (b.pair_queue) c.add(b.pairq, M);
    c.add(b.run_sfx, R);
    c.add(b.run_L, R);
    if (b.row_table) c.add(b.rowstart, b.rows + 1);
}
void lay_lists(Batch& b, Carver& c) { c.add(b.targets, b.targets_cap); }
void lay_act(Batch& b, Carver& c) { c.add(b.act, b.N); }

// The row table when it is not much larger than the cell list.
bool wants_row_table(const Batch& b, uint64_t cells) {
    return b.rows < (1ull << 31) && b.rows <= 4 * cells + (1u << 20);
}

template <class KT>
void launch_heads(Batch& b, const KT* keys, uint64_t capM, uint64_t capR) {
    const uint64_t tiles = (b.N + kHeadTile - 1) / kHeadTile;
    KScope ks("cell_heads");
    auto* const kernel = b.gathered ? k_heads<KT, true> : k_heads<KT, false>;
    kernel<<<(unsigned)tiles, kHeadThreads, 0, b.s>>>(
        b.N, b.F, keys, b.sid.get(), b.xy.get(), b.fstart.get(), b.fjob.get(), b.sxy.get(), b.sfeat.get(),
        b.ckey.get(), b.crun.get(), b.cjob.get(), b.rfeat.get(), b.rstart.get(), b.rcell.get(),
        capM ? b.scell.get() : nullptr, capM, capR, b.head_status.get(), b.tickets.get() + b.plan.n, b.ctrl.get());
    COLO_LAUNCH_CHECK();
    count_launch();
}

// Waits for the totals of the sort and the heads.
void read_sizes(Batch& b) {
    BatchCtrl h;
    COLO_CUDA(cudaMemcpyAsync(&h, b.ctrl.get(), sizeof(h), cudaMemcpyDeviceToHost, b.s));
    stream_wait(b.s);
    if (h.flags.timeout) throw StatusError{COLO_ERR_TIMEOUT, "radix sort: a tile waited too long for its predecessors"};
    b.M = h.M;
    b.Rn = h.Rn;
}

// Cell keys, the stable sort by key, and the sorted point copies with the cells and runs,
// with KT = 32-bit keys when every key fits (less traffic per radix pass), else 64-bit.
template <class KT>
void sort_and_compact(Batch& b) {
    cudaStream_t s = b.s;
    const uint64_t n = b.N;
    const bool sorts = n > 1 && b.plan.n > 0;
    // the sort's buffers: the ids end in b.sid, whichever of the two the last pass writes
    DevBuf<unsigned char> mem;
    Span<KT> ka, kb;
    Span<uint32_t> other;
    Carver::place(mem, s, [&](Carver& c) {
        c.add(ka, n);
        c.add(kb, n);
        c.add(other, n);
        if (b.sort_shared) c.add(b.sort_status, radix_status_words(n, b.plan));
    });
    {
        KScope ks("cell_keys");
        const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, (uint64_t)b.sms * 8);
        // the ids are written here only when the sort runs no pass (its first pass makes them)
        k_cell_keys<KT><<<(unsigned)(blocks ? blocks : 1), 256, 0, s>>>(
            n, b.F, b.fstart.get(), b.fjob.get(), b.grids.get(), ka.get(), sorts ? nullptr : b.sid.get(),
            b.xy.get(), b.nb_cnt.get(), b.ctrl.get(), b.plan, b.hist.get());
        COLO_LAUNCH_CHECK();
        count_launch();
    }
    const KT* keys = ka.get();
    if (sorts) {
        const bool odd = (b.plan.n & 1) != 0;
        RadixBufs<KT> bufs{ka.get(), kb.get(), odd ? other.get() : b.sid.get(), odd ? b.sid.get() : other.get()};
        radix_sort(bufs, n, b.plan, s, b.hist.get(), b.sort_status.get(), b.sort_shared, b.tickets.get(),
                   &b.flags()->timeout, b.test_spin);
        keys = bufs.ka;
    }
    if (b.bounded) {
        launch_heads<KT>(b, keys, b.capM, b.capR);
        return;
    }
    // heads laid out for every point when that is small against the device, else counted first
    const size_t all = Carver::bytes([&](Carver& c) { lay_heads(b, c, n, n); });
    if (!b.exact && all <= b.device_bytes / 16) {
        Carver::place(b.mem_heads, s, [&](Carver& c) { lay_heads(b, c, n, n); });
        b.reserved_bytes = all;
        launch_heads<KT>(b, keys, n, n);
        read_sizes(b);
    } else {
        launch_heads<KT>(b, keys, 0, 0);
        read_sizes(b);
        Carver::place(b.mem_heads, s, [&](Carver& c) { lay_heads(b, c, b.M, b.Rn); });
        const uint64_t tiles = (n + kHeadTile - 1) / kHeadTile;
        COLO_CUDA(cudaMemsetAsync(b.head_status.get(), 0, 2 * tiles * 8, s));
        COLO_CUDA(cudaMemsetAsync(b.tickets.get() + b.plan.n, 0, 4, s));
        launch_heads<KT>(b, keys, b.M, b.Rn);
    }
    b.capM = b.M;
    b.capR = b.Rn;
}

}  // namespace

void bucket_layout(Batch& b, Carver& c) {
    const uint64_t tiles = (b.N + kHeadTile - 1) / kHeadTile, sw = b.N ? radix_status_words(b.N, b.plan) : 0;
    b.sort_shared = sw * 8 * (uint64_t)b.plan.n > std::min<uint64_t>(kSortStatusBytes, b.device_bytes / 1024);
    c.add(b.hist, (uint64_t)std::max(b.plan.n, 1) * kRadixDigits);
    c.add(b.tickets, (uint64_t)b.plan.n + 1);
    c.add(b.head_status, 2 * tiles);
    if (!b.sort_shared) c.add(b.sort_status, sw * (uint64_t)b.plan.n);
}

void bucket_points(Batch& b) {
    cudaStream_t s = b.s;
    const uint64_t n = b.N;
    // everything up to the pairs' bounds in one block laid out by bounds, when that is small
    // enough to reserve; a device that has no such block left takes the other way
    b.capM = b.capR = n;
    b.targets_cap = list_room(n);
    b.nb_cap = neighbour_room(b);
    b.row_table = wants_row_table(b, n);
    b.gathered = b.J > 1 || n <= kGatherPoints;
    b.pair_queue = b.J == 1 && n >= kPairQueuePoints;
    auto bounds = [&](Carver& c) {
        lay_points(b, c);
        lay_heads(b, c, n, n);
        lay_cells(b, c, n, n);
        lay_lists(b, c);
        lay_act(b, c);
        c.add(b.nb, b.nb_cap);
    };
    const uint64_t need = Carver::bytes(bounds);
    b.bounded = !b.exact && need <= std::min<uint64_t>(kBoundBytes, b.device_bytes / 16) &&
                (need <= kSmallBounds || leaves_half(b.ctx, need));
    if (b.bounded) {
        try {
            Carver::place(b.mem_points, s, bounds);
            b.reserved_bytes = need;
            note_block(b.ctx, need);
        } catch (const StatusError& e) {
            if (e.st != COLO_ERR_NOMEM) throw;
            b.bounded = false;
        }
    }
    if (!b.bounded) {
        b.nb_cap = 0;
        b.nb = Span<uint32_t>();
        Carver::place(b.mem_points, s, [&](Carver& c) { lay_points(b, c); });
    }
    if (b.key_bits <= 32) sort_and_compact<uint32_t>(b);
    else sort_and_compact<uint64_t>(b);
    if (!b.bounded) {
        b.row_table = wants_row_table(b, b.M);
        Carver::place(b.mem_cells, s, [&](Carver& c) { lay_cells(b, c, b.M, b.Rn); });
    }
    const uint64_t capM = b.capM;
    {
        KScope ks("cell_masks");
        const uint64_t items = std::max<uint64_t>(capM, b.row_table ? b.rows + 1 : 0);
        const unsigned grid = (unsigned)std::min<uint64_t>(grid_for(items, 256), (uint64_t)b.sms * 8);
        k_cell_masks<<<grid, 256, b.F <= kRunHist ? b.F * 4 : 0, s>>>(
            b.ctrl.get(), b.ckey.get(), b.crun.get(), b.rfeat.get(), b.cjob.get(), b.grids.get(), b.W, b.cmask.get(),
            b.row_table ? b.rows : 0, b.J, b.rowstart.get(), b.F, b.frun());
        COLO_LAUNCH_CHECK();
        count_launch();
    }
    {
        KScope ks("cell_neighbours");
        const unsigned grid = (unsigned)std::min<uint64_t>(grid_for(capM, 128), (uint64_t)b.sms * 64);
        k_neighbours<<<grid, 128, 0, s>>>(b.ctrl.get(), b.ckey.get(), b.cjob.get(), b.grids.get(),
                                          b.row_table ? b.rowstart.get() : nullptr, b.nbrs.get());
        COLO_LAUNCH_CHECK();
        count_launch();
    }
    {
        KScope ks("quad_masks");
        // one wave of resident blocks (each keeps one histogram for all its cells)
#define COLO_QM(WW)                                                                                          \
    do {                                                                                                     \
        int per_sm = 1;                                                                                      \
        COLO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_quad_masks<WW>, kQuadThreads, 0)); \
        const unsigned qblocks = (unsigned)std::max<uint64_t>(                                               \
            1, std::min<uint64_t>(grid_for(capM, kQuadThreads), (uint64_t)b.sms * (uint64_t)std::max(per_sm, 1))); \
        k_quad_masks<WW><<<qblocks, kQuadThreads, 0, s>>>(                                                   \
            b.ctrl.get(), b.nbrs.get(), b.cmask.get(), b.qmask.get(), b.nbmask.get(), b.listq.get(),         \
            b.quadq.get(), b.pair_queue ? b.pairq.get() : nullptr, b.quad_min, b.J > 1, b.F, b.dcnt());                               \
    } while (0)
        switch (b.W) {
            case 1: COLO_QM(1); break;
            case 2: COLO_QM(2); break;
            case 3: COLO_QM(3); break;
            case 4: COLO_QM(4); break;
            case 5: COLO_QM(5); break;
            case 6: COLO_QM(6); break;
            case 7: COLO_QM(7); break;
            case 8: COLO_QM(8); break;
            case 12: COLO_QM(12); break;
            case 16: COLO_QM(16); break;
            case 24: COLO_QM(24); break;
            case 32: COLO_QM(32); break;
            default: throw StatusError{COLO_ERR_CAPACITY, "the quad filter handles at most 1024 features per job"};
        }
#undef COLO_QM
        COLO_LAUNCH_CHECK();
        count_launch();
    }
}

void build_neighborhoods(Batch& b) {
    cudaStream_t s = b.s;
    if (!b.bounded && !b.act.get()) {
        Carver::place(b.mem_act, s, [&](Carver& c) { lay_act(b, c); });
        b.targets_cap = std::min<uint64_t>(9 * b.N, b.N / 2 + 65536);   // (large batches: less in reserve)
        Carver::place(b.mem_lists, s, [&](Carver& c) { lay_lists(b, c); });
    }
    if (b.lists_built) {   // the lists did not fit: room for all of them (targets_cap), and the totals from zero
        Carver::place(b.mem_lists, s, [&](Carver& c) { lay_lists(b, c); });
        COLO_CUDA(cudaMemsetAsync(&b.ctrl.get()->targets, 0, 5 * sizeof(LineCounter), s));
    }
    b.lists_built = true;
    const unsigned qgrid = (unsigned)std::min<uint64_t>(grid_for(b.capM, 128), (uint64_t)b.sms * 16);
    KScope ks("neighbour_lists");
    k_neighbour_lists<<<qgrid, 128, 4 * ListRanks::words(b.W) * 4, s>>>(b.N, b.listq.get(), b.ctrl.get(), b.nbrs.get(), b.cmask.get(), b.W, b.crun.get(),
                                            b.rfeat.get(), b.rstart.get(),
                                            b.gathered ? nullptr : b.sid.get(), b.targets_cap, b.targets.get(), b.run_sfx.get(), b.run_L.get(),
                                            b.act.get());
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace colo
