// colo_filter.cu -- cell-aggregate upper-bound filter.
//
// Semantics (filter2_Kernel + threshold_Kernel, Codes/DeviceProcess_Kernel.h:
// 469-509 and 545-573): a quad is a 2x2 block of reference cells with lower
// corner (bx, by), 0 <= bx <= gx-2, 0 <= by <= gy-2.  It is full for
// candidate c when every member j < min(k, 8) has a point in one of its four
// cells.  U_c is the union of the cells of full quads; the bound of member j
// is the sum over U_c of that member's cell counts (members j >= 8 keep 0).
// The reference's degree-2 kernel (filter2_2_Kernel, 512-543) reads an
// uninitialised index, so pairs use the same rule.
//
// Pairs: if cell C holds feature f, C lies in U_{f,g} exactly when g occurs
// in the union of the valid quads around C, which is C's clipped 3x3 block.
// So every pair bound is one pass over the runs: for each run (C, f) and
// each feature g of the 3x3 block, add count(C, f) to bound(f side of {f,g}).
// The accumulator is an F x F matrix in shared memory.
//
// Level k >= 3: a cell is in U_c when one of its four quads is full; the
// cells tested for c are those with c's driver member (the one with the
// fewest cells) in their 3x3 block, which holds every cell of U_c, and a quad of
// three features.  Those cells are listed once per mine, per feature (driver
// lists), so a level touches only the lists of its drivers.
#include <algorithm>
#include <cstring>

#include "colo_batch.h"
#include "colo_device.cuh"

namespace colo {
namespace {

constexpr int kFilterThreads = 256, kPairThreads = 1024;   // a pair block: 256 to 1024 threads
constexpr int kMaxW = 32;  // mask words per cell (1024 features per job); rows of 9+ words are padded
                           // to 12, 16, 24 or 32 words when the batch is set up
constexpr uint64_t kAccMax = 16384;   // block-private level sums (64 KB of shared memory)

// One thread per run (C, f); a block owns a contiguous range of runs, so the
// job changes rarely and the F x F accumulator lives in shared memory.  cjob is
// null for a one-job batch (job 0 everywhere): the mask load then waits on one
// dependent load (the run's cell) instead of three.
__global__ void __launch_bounds__(kPairThreads) k_filter_pairs(
    const BatchCtrl* __restrict__ ctrl, const uint32_t* __restrict__ rcell, const uint32_t* __restrict__ cjob,
    const JobGrid* __restrict__ grids, const uint32_t* __restrict__ nbmask,
    uint32_t W, const uint32_t* __restrict__ rfeat, const uint32_t* __restrict__ rstart,
    const uint64_t* __restrict__ job_off, uint32_t* __restrict__ ub2, uint32_t acc_dim) {
    extern __shared__ uint32_t acc[];   // acc_dim x acc_dim (acc_dim = 0: no privatisation)
    __shared__ int32_t cur_job;
    const uint64_t Rn = ctrl->Rn;
    const uint64_t per = ((Rn + gridDim.x - 1) / gridDim.x + blockDim.x - 1) / blockDim.x * blockDim.x;
    const uint64_t r0 = (uint64_t)blockIdx.x * per;
    const uint64_t r1 = r0 + per < Rn ? r0 + per : Rn;
    if (r0 >= r1) return;
    const uint32_t accn = acc_dim * acc_dim;
    for (uint32_t i = threadIdx.x; i < accn; i += blockDim.x) acc[i] = 0;
    if (threadIdx.x == 0) cur_job = cjob ? (int32_t)cjob[rcell[r0]] : 0;
    __syncthreads();
    for (uint64_t base = r0; base < r1; base += blockDim.x) {
        const int32_t jb = cjob ? (int32_t)cjob[rcell[base]] : 0;
        if (jb != cur_job) {   // flush the accumulator on a job change (uniform branch)
            __syncthreads();
            uint32_t nf = grids[cur_job].nf;
            for (uint32_t i = threadIdx.x; acc_dim && i < nf * nf; i += blockDim.x) {
                uint32_t v = acc[(i / nf) * acc_dim + (i % nf)];
                if (v) atomicAdd(&ub2[job_off[cur_job] + i], v);
            }
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < accn; i += blockDim.x) acc[i] = 0;
            if (threadIdx.x == 0) cur_job = jb;
            __syncthreads();
        }
        const uint64_t r = base + threadIdx.x;
        if (r < r1) {
            const uint32_t c = rcell[r];
            const uint32_t job = cjob ? cjob[c] : 0u;
            const JobGrid g = grids[job];
            if (g.gx >= 2 && g.gy >= 2) {
                const bool priv = acc_dim && (int32_t)job == cur_job && g.nf <= acc_dim;
                const uint32_t lf = rfeat[r] - g.f0, cnt = rstart[r + 1] - rstart[r];
                for (uint32_t w = 0; w < W; ++w) {
                    uint32_t bits = nbmask[(uint64_t)c * W + w];
                    while (bits) {
                        int bpos = __ffs(bits) - 1;
                        bits &= bits - 1;
                        uint32_t lg = w * 32 + bpos;
                        if (lg == lf) continue;
                        if (priv) atomicAdd(&acc[lf * acc_dim + lg], cnt);
                        else atomicAdd(&ub2[job_off[job] + (uint64_t)lf * g.nf + lg], cnt);
                    }
                }
            }
        }
    }
    __syncthreads();
    if (acc_dim) {
        uint32_t nf = grids[cur_job].nf;
        for (uint32_t i = threadIdx.x; i < nf * nf; i += blockDim.x) {
            uint32_t v = acc[(i / nf) * acc_dim + (i % nf)];
            if (v) atomicAdd(&ub2[job_off[cur_job] + i], v);
        }
    }
}

// The same for one job of many points: over the runs of the queued cells (two features or more in
// their 3x3 block; the others are in no pair's bound).  A warp takes 32 cells of
// the queue and their runs one after another, a run a lane, so a cell of many runs costs as
// much a run as one of few.  Bound by the masks' loads and the shared atomics; a thread for
// each of all runs took 157 us at 20M points (8.9M runs, one cell in nine queued), this 67.
__global__ void __launch_bounds__(kPairThreads) k_filter_pairs_queue(
    const BatchCtrl* __restrict__ ctrl, const uint32_t* __restrict__ pairq, const uint32_t* __restrict__ crun,
    const JobGrid* __restrict__ grids, const uint32_t* __restrict__ nbmask, uint32_t W,
    const uint32_t* __restrict__ rfeat, const uint32_t* __restrict__ rstart, uint32_t* __restrict__ ub2,
    uint32_t acc_dim) {
    extern __shared__ uint32_t acc[];   // acc_dim x acc_dim, acc_dim the job's features or 0 (no privatisation)
    const JobGrid& g = grids[0];
    if (g.gx < 2 || g.gy < 2) return;
    const uint32_t nf = g.nf, accn = acc_dim * acc_dim;
    for (uint32_t i = threadIdx.x; i < accn; i += blockDim.x) acc[i] = 0;
    __syncthreads();
    const uint64_t n = ctrl->npairq.v;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t i0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; i0 < n; i0 += warps * 32) {
        uint32_t c = 0, r0 = 0, runs = 0;
        if (i0 + lane < n) {
            c = pairq[i0 + lane];
            r0 = crun[c];
            runs = crun[c + 1] - r0;
        }
        const uint32_t incl = warp_incl_scan(runs), excl = incl - runs;
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        for (uint32_t t0 = 0; t0 < tot; t0 += 32) {
            const uint32_t t = t0 + lane;
            int j = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t ev = __shfl_sync(0xffffffffu, excl, j + step);
                if (ev <= t) j += step;
            }
            const uint32_t cj = __shfl_sync(0xffffffffu, c, j);
            const uint32_t r = __shfl_sync(0xffffffffu, r0 - excl, j) + t;
            if (t >= tot) continue;
            const uint32_t lf = rfeat[r], cnt = rstart[r + 1] - rstart[r];
            for (uint32_t w = 0; w < W; ++w)
                for (uint32_t bits = nbmask[(uint64_t)cj * W + w]; bits; bits &= bits - 1) {
                    const uint32_t lg = w * 32 + (uint32_t)(__ffs(bits) - 1);
                    if (lg == lf) continue;
                    if (acc_dim) atomicAdd(&acc[lf * acc_dim + lg], cnt);
                    else atomicAdd(&ub2[(uint64_t)lf * nf + lg], cnt);
                }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < accn; i += blockDim.x)
        if (acc[i]) atomicAdd(&ub2[i], acc[i]);
}

template <int WT>
__device__ __forceinline__ bool covers(const uint32_t* __restrict__ qm, const uint32_t (&need)[WT]) {
    bool ok = true;
#pragma unroll
    for (int w = 0; w < WT; ++w) ok &= (qm[w] & need[w]) == need[w];
    return ok;
}

template <int WT>
__device__ __forceinline__ bool covers(const uint32_t (&qm)[WT], const uint32_t (&need)[WT]) {
    bool ok = true;
#pragma unroll
    for (int w = 0; w < WT; ++w) ok &= (qm[w] & need[w]) == need[w];
    return ok;
}

// One mask row of WT words; rows start on a multiple of WT words from a
// 256-byte-aligned base, so 4-word rows load as one 16-byte vector.
template <int WT>
__device__ __forceinline__ void load_row(const uint32_t* __restrict__ p, uint32_t (&out)[WT]) {
    if constexpr (WT % 4 == 0) {
#pragma unroll
        for (int i = 0; i < WT / 4; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + i);
            out[4 * i] = v.x;
            out[4 * i + 1] = v.y;
            out[4 * i + 2] = v.z;
            out[4 * i + 3] = v.w;
        }
    } else if constexpr (WT % 2 == 0) {
#pragma unroll
        for (int i = 0; i < WT / 2; ++i) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(p) + i);
            out[2 * i] = v.x;
            out[2 * i + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < WT; ++i) out[i] = __ldg(p + i);
    }
}

// ---- driver lists -----------------------------------------------------------
// The list of feature f holds the queued cells (quadq) whose 3x3 block holds f (bit
// f of nbmask); the lists of the wanted features (the level drivers) are filled
// here, their sizes come from the quad masks' kernel.  A block owns a range of
// the queue and walks it twice, 256 cells (one per thread) at a time.
// A warp's 32 cells are a bit matrix (cell x feature) per mask word;
// transposed, lane b holds feature b's column.  Pass 0 adds the columns'
// popcounts to a block histogram; one global atomic per (block, feature) then
// reserves the block's range of each list; pass 1 adds them again, the
// atomic's old value placing the warp's cells in that range, and lane b
// writes its column's cells.  Order within a list is not fixed (the level
// filter sums over it).  Batches with more than kDilHist features skip the
// histogram: one global atomic per (warp, feature).
constexpr uint32_t kDilHist = 2048;
constexpr int kDilThreads = 256;

// Bits of cell z's mask word w that are wanted: the want bitset (global
// features) taken from bit f0 + 32 w on.  The bitset holds one spare word.
__device__ __forceinline__ uint32_t dil_wanted(const uint32_t* __restrict__ want, uint32_t f0, int w, uint32_t row) {
    const uint32_t p = f0 + (uint32_t)w * 32;
    const uint32_t lo = __ldg(want + (p >> 5)), hi = __ldg(want + (p >> 5) + 1);
    return row & __funnelshift_r(lo, hi, p & 31);
}

template <int WT>
__global__ void __launch_bounds__(kDilThreads) k_dil_fill(uint64_t n, uint64_t per,
                                                          const uint32_t* __restrict__ quadq,
                                                          const uint32_t* __restrict__ cjob,
                                                          const JobGrid* __restrict__ grids,
                                                          const uint32_t* __restrict__ nbmask, uint32_t F,
                                                          const uint64_t* __restrict__ doff,
                                                          uint32_t* __restrict__ cursor, uint32_t* __restrict__ dlist,
                                                          const uint32_t* __restrict__ want) {
    // F bases, then F counters and F touched features (F <= kDilHist; sized by the launch)
    extern __shared__ unsigned long long s_base[];
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_base + (F <= kDilHist ? F : 0));
    uint32_t* s_touch = s_cnt + (F <= kDilHist ? F : 0);
    __shared__ uint32_t s_nt, s_cell[kDilThreads];
    const bool local = F <= kDilHist;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t z0 = (uint64_t)blockIdx.x * per, z1 = z0 + per < n ? z0 + per : n;
    if (local)
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x) s_cnt[i] = 0;
    if (threadIdx.x == 0) s_nt = 0;
    __syncthreads();
    for (int pass = local ? 0 : 1; pass < 2; ++pass) {
        for (uint64_t t0 = z0; t0 < z1; t0 += kDilThreads) {
            const bool in = t0 + threadIdx.x < z1;
            const uint32_t z = in ? quadq[t0 + threadIdx.x] : 0u;
            const uint32_t* zw = s_cell + (threadIdx.x & ~31u);   // the warp's cells
            __syncwarp();
            s_cell[threadIdx.x] = z;
            __syncwarp();
            uint32_t row[WT];
            uint32_t f0 = 0;
            if (in) {
                f0 = grids[cjob ? cjob[z] : 0u].f0;
                load_row<WT>(nbmask + (uint64_t)z * WT, row);
#pragma unroll
                for (int w = 0; w < WT; ++w)   // a nonzero word lies below F, so its bitset words exist
                    if (row[w]) row[w] = dil_wanted(want, f0, w, row[w]);
            } else {
#pragma unroll
                for (int w = 0; w < WT; ++w) row[w] = 0;
            }
            // one job's cells at a time (a warp holds cells of several only at the jobs' borders in
            // the queue)
            for (uint32_t todo = __ballot_sync(0xffffffffu, in); todo;) {
                const uint32_t fl = __shfl_sync(0xffffffffu, f0, __ffs(todo) - 1);
                const bool mine = in && f0 == fl;
                todo &= ~__ballot_sync(0xffffffffu, mine);
#pragma unroll
                for (int w = 0; w < WT; ++w) {
                    const uint32_t bits_w = mine ? row[w] : 0u;
                    if (!__any_sync(0xffffffffu, bits_w)) continue;
                    const uint32_t col = warp_transpose32(bits_w);
                    const uint32_t cells = __popc(col);
                    if (!cells) continue;
                    const uint32_t f = fl + (uint32_t)w * 32 + lane;
                    uint64_t o;
                    if (local) {
                        const uint32_t old = atomicAdd(&s_cnt[f], cells);
                        if (pass == 0) {
                            if (old == 0) s_touch[atomicAdd(&s_nt, 1u)] = f;
                            continue;
                        }
                        o = s_base[f] + old;
                    } else {
                        o = doff[f] + atomicAdd(&cursor[f], cells);
                    }
                    uint32_t* dst = dlist + o;
                    for (uint32_t bits = col; bits; bits &= bits - 1) *dst++ = zw[__ffs(bits) - 1];
                }
            }
        }
        if (pass == 0) {   // reserve the block's ranges; pass 1 counts again from zero
            __syncthreads();
            const uint32_t nt = s_nt;
            for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
                const uint32_t f = s_touch[i];
                s_base[f] = doff[f] + atomicAdd(&cursor[f], s_cnt[f]);
                s_cnt[f] = 0;
            }
            __syncthreads();
        }
    }
}

// Level k >= 3 over the driver lists.  Candidates are grouped by driver
// (group g: driver feature gfeat[g], candidates order[gstart[g] ..
// gstart[g] + gcount[g])); a unit is 32 cells of the driver's list times up
// to cu (8, 16 or 32, autotuned) of its candidates, units of one cell chunk
// adjacent (they read the same quad masks).  A warp takes a unit: lane = cell, loop over the
// candidates; a (cell Z, candidate c) pair is tested exactly as in a scan
// of every cell with the driver in its 3x3 block: Z is in U_c when one of
// its four quads covers c's members, each cell of U_c is met once, and a
// full quad is counted at its first occupied cell (nbrs).  Lane t loads the
// unit's candidate t up front (a candidate then comes by shuffles, not by
// dependent loads), and a candidate's counts are summed over the warp's cells
// before one atomic per sum, into a block-private accumulator when the level's
// counters fit (acc_n).  One atomic per cell and sum cost a batch of 128 jobs,
// whose counters do not fit, 1.25 ms against 0.65 ms; single mines take the same
// time either way.
template <int WT>
__global__ void __launch_bounds__(256, (WT <= 4 ? 5 : (WT <= 6 ? 4 : (WT <= 8 ? 2 : 1)))) k_filter_drv(
    uint64_t nunits, uint32_t ngroups, const uint64_t* __restrict__ uoff, const uint32_t* __restrict__ gfeat,
    const uint32_t* __restrict__ gstart, const uint32_t* __restrict__ gcount, const uint64_t* __restrict__ doff,
    const uint32_t* __restrict__ dlist, const uint32_t* __restrict__ order, const uint32_t* __restrict__ need_all,
    const uint32_t* __restrict__ lmem, uint32_t k, const uint32_t* __restrict__ qmask,
    const uint32_t* __restrict__ cmask, const uint32_t* __restrict__ crun, const uint4* __restrict__ nbrs,
    const uint32_t* __restrict__ rstart, uint32_t* __restrict__ ub, unsigned long long* __restrict__ stats,
    uint32_t acc_n, uint32_t cu) {
    constexpr uint32_t W = WT;
    constexpr bool kCacheQuads = WT <= 8;
    // need masks by shuffle (else loaded per candidate: at 2 to 4 words the shuffles' registers
    // spill, 0.45 against 0.43 ms on the 20M workload; at 1 and 7 words shuffles are faster)
    constexpr bool kShuffleNeed = WT == 1 || (WT > 4 && WT <= 8);
    extern __shared__ uint32_t acc[];
    const uint32_t m = k < kMaxMembersFiltered ? k : kMaxMembersFiltered;
    const uint32_t stride = m + 2;
    const int lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < acc_n; i += blockDim.x) acc[i] = 0;
    __syncthreads();
    const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t u = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < nunits; u += nwarps) {
        uint32_t lo = 0, hi = ngroups;   // the group of unit u: last g with uoff[g] <= u
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(uoff + mid) <= u) lo = mid;
            else hi = mid;
        }
        const uint32_t f = __ldg(gfeat + lo), G = __ldg(gcount + lo), gs = __ldg(gstart + lo);
        const uint32_t gch = (G + cu - 1) / cu;
        const uint64_t local = u - __ldg(uoff + lo);
        const uint64_t cc = local / gch;
        const uint32_t gc = (uint32_t)(local - cc * gch);
        const uint64_t l0 = __ldg(doff + f), L = __ldg(doff + f + 1) - l0;
        const uint64_t zi = cc * 32 + (uint64_t)lane;
        const bool valid = zi < L;
        const uint64_t Z = valid ? __ldg(dlist + l0 + zi) : 0u;
        const uint32_t* q4 = qmask + Z * 4 * W;
        uint32_t qr[kCacheQuads ? 4 : 1][kCacheQuads ? WT : 1];
        // the cell's own mask, first run and first quads, issued with its quads (most list cells
        // are in U_c of some candidate, and these loads would otherwise wait for the first)
        uint32_t cm[WT];
        uint32_t q0 = 0, qf = 0;
#pragma unroll
        for (int w = 0; w < WT; ++w) cm[w] = 0;
        if constexpr (kCacheQuads) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int w = 0; w < WT; ++w) qr[q][w] = 0;
        }
        if (valid) {
            if constexpr (kCacheQuads) {
#pragma unroll
                for (int q = 0; q < 4; ++q) load_row<WT>(q4 + q * W, qr[q]);
            }
            load_row<WT>(cmask + Z * W, cm);
            q0 = crun[Z];
            qf = nbrs[Z].z >> 12 & 15u;
        }
        // lane t: the unit's candidate t
        const uint32_t t0 = gc * cu, cnt = t0 + cu < G ? cu : G - t0;
        uint32_t c_l = 0, lm_l[4] = {0, 0, 0, 0}, need_l[kShuffleNeed ? WT : 1];
        if ((uint32_t)lane < cnt) {
            c_l = __ldg(order + gs + t0 + lane);
            load_row<4>(lmem + (uint64_t)c_l * 4, lm_l);
            if constexpr (kShuffleNeed) load_row<WT>(need_all + (uint64_t)c_l * W, need_l);
        }
        for (uint32_t t = 0; t < cnt; ++t) {
            const uint32_t c = __shfl_sync(0xffffffffu, c_l, t);
            uint32_t need[WT];
            if constexpr (kShuffleNeed) {
#pragma unroll
                for (int w = 0; w < WT; ++w) need[w] = __shfl_sync(0xffffffffu, need_l[w], t);
            } else {
                load_row<WT>(need_all + (uint64_t)c * W, need);
            }
            uint32_t full = 0;
            if (valid) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    bool ok;
                    if constexpr (kCacheQuads) {
                        ok = covers<WT>(qr[q], need);
                    } else {
                        uint32_t qm[WT];
                        load_row<WT>(q4 + q * W, qm);
                        ok = covers<WT>(qm, need);
                    }
                    if (ok) full |= 1u << q;
                }
            }
            const uint32_t cells = __ballot_sync(0xffffffffu, full != 0);
            if (!cells) continue;
            // the warp's sums, lane r holding sum r: members' counts, full quads, cells
            uint32_t sum = (uint32_t)lane == m + 1 ? (uint32_t)__popc(cells) : 0u;
#pragma unroll
            for (int jp = 0; jp < kMaxMembersFiltered / 2; ++jp) {
                if ((uint32_t)jp * 2 >= m) break;
                const uint32_t lm = __shfl_sync(0xffffffffu, lm_l[jp], t);   // members 2 jp and 2 jp + 1
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t jj = jp * 2 + h;
                    if (jj >= m) break;
                    const uint32_t lf = (lm >> (h * 16)) & 0xFFFFu, wq = lf >> 5;
                    uint32_t v = 0;
                    if (full) {
                        uint32_t rk = 0, word = 0;
#pragma unroll
                        for (int w = 0; w < WT; ++w) {
                            if ((uint32_t)w < wq) rk += __popc(cm[w]);
                            if ((uint32_t)w == wq) word = cm[w];
                        }
                        if (word >> (lf & 31) & 1u) {
                            const uint32_t ri = q0 + rk + __popc(word & ((1u << (lf & 31)) - 1u));
                            v = rstart[ri + 1] - rstart[ri];
                        }
                    }
                    v = __reduce_add_sync(0xffffffffu, v);
                    if ((uint32_t)lane == jj) sum = v;
                }
            }
            const uint32_t nq = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(full & qf));
            if ((uint32_t)lane == m) sum = nq;
            if ((uint32_t)lane < stride && sum) {
                if (acc_n) atomicAdd(&acc[c * stride + lane], sum);
                else if ((uint32_t)lane < m) atomicAdd(&ub[(uint64_t)c * k + lane], sum);
                else if (stats) atomicAdd(&stats[(uint64_t)c * 2 + (lane - m)], (unsigned long long)sum);
            }
        }
    }
    if (acc_n) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < acc_n; i += blockDim.x) {
            const uint32_t v = acc[i];
            if (!v) continue;
            const uint32_t c = i / stride, r = i - c * stride;
            if (r < m) atomicAdd(&ub[(uint64_t)c * k + r], v);
            else if (stats) atomicAdd(&stats[(uint64_t)c * 2 + (r - m)], (unsigned long long)v);
        }
    }
}

}  // namespace

#define COLO_W_SWITCH(W, MACRO)                                                                   \
    switch (W) {                                                                                  \
        case 1: MACRO(1); break;                                                                  \
        case 2: MACRO(2); break;                                                                  \
        case 3: MACRO(3); break;                                                                  \
        case 4: MACRO(4); break;                                                                  \
        case 5: MACRO(5); break;                                                                  \
        case 6: MACRO(6); break;                                                                  \
        case 7: MACRO(7); break;                                                                  \
        case 8: MACRO(8); break;                                                                  \
        case 12: MACRO(12); break;                                                                \
        case 16: MACRO(16); break;                                                                \
        case 24: MACRO(24); break;                                                                \
        case 32: MACRO(32); break;                                                                \
        default: throw StatusError{COLO_ERR_INTERNAL, "mask words not padded to a supported width"}; \
    }

namespace {

// The lists of every feature in `need` (and of those already filled): the lists are filled
// again for the union when a feature is missing.
void driver_lists_fill(Batch& b, const std::vector<uint8_t>& need) {
    bool missing = false;
    for (uint32_t f = 0; f < b.F; ++f) missing |= need[f] && !b.dlist_have[f];
    if (!missing) return;
    cudaStream_t s = b.s;
    std::vector<uint32_t> want((b.F + 31) / 32 + 1, 0);   // one spare word for the kernel's funnel shift
    b.h_doff.assign(b.F + 1, 0);
    for (uint32_t f = 0; f < b.F; ++f) {
        b.dlist_have[f] |= need[f];
        if (b.dlist_have[f]) want[f >> 5] |= 1u << (f & 31);
        b.h_doff[f + 1] = b.h_doff[f] + (b.dlist_have[f] ? b.h_dcnt[f] : 0);
    }
    const uint64_t total = b.h_doff[b.F];
    b.dlist.alloc(total ? total : 1, s);
    // offsets, the want bitset and the cleared cursors: one upload
    std::vector<uint64_t> in(b.F + 1 + (want.size() + b.F + 1) / 2, 0);
    std::copy(b.h_doff.begin(), b.h_doff.end(), in.begin());
    std::memcpy(in.data() + b.F + 1, want.data(), want.size() * 4);
    b.doff.alloc(in.size(), s);
    uint32_t* d_want = reinterpret_cast<uint32_t*>(b.doff.get() + b.F + 1);
    uint32_t* d_cursor = d_want + want.size();
    staged_upload(b.ctx, s, b.doff.get(), in.data(), in.size() * 8);
    if (total == 0) return;
    // one range of consecutive cells per block (a multiple of 256 cells), one wave of resident blocks;
    // shared memory for the block histogram of the batch's features (none past kDilHist)
    const size_t dsmem = b.F <= kDilHist ? (size_t)b.F * 16 : 0;
    KScope ks("driver_lists");
#define COLO_DF(WW)                                                                                              \
    do {                                                                                                         \
        int per_sm = 1;                                                                                          \
        COLO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dil_fill<WW>, kDilThreads, dsmem));   \
        uint64_t blocks = std::min<uint64_t>((b.quad_cells + kDilThreads - 1) / kDilThreads,                              \
                                             (uint64_t)b.sms * (uint64_t)std::max(per_sm, 1));                   \
        const uint64_t per = ((b.quad_cells + blocks - 1) / blocks + kDilThreads - 1) / kDilThreads * kDilThreads;        \
        blocks = (b.quad_cells + per - 1) / per;                                                                          \
        k_dil_fill<WW><<<(unsigned)blocks, kDilThreads, dsmem, s>>>(b.quad_cells, per, b.quadq.get(),            \
                                                               b.J > 1 ? b.cjob.get() : nullptr,                 \
                                                               b.grids.get(), b.nbmask.get(), b.F, b.doff.get(), \
                                                               d_cursor, b.dlist.get(), d_want);             \
    } while (0)
    COLO_W_SWITCH(b.W, COLO_DF)
#undef COLO_DF
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace

void filter_pairs(Batch& b) {
    cudaStream_t s = b.s;
    if (b.W > kMaxW) throw StatusError{COLO_ERR_CAPACITY, "the filter handles at most 1024 features per job"};
    uint32_t acc_dim = b.Fmax_local;
    size_t smem = (size_t)acc_dim * acc_dim * 4;
    if (smem > 200 * 1024) {
        acc_dim = 0;
        smem = 0;
    }
    if (smem > 48 * 1024)
        COLO_CUDA(cudaFuncSetAttribute(b.pair_queue ? (const void*)k_filter_pairs_queue : (const void*)k_filter_pairs,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // as many resident threads per SM as the accumulators leave: blocks of 256 threads where eight
    // fit (each with its share of the runs), larger ones where the accumulator is large
    // (200 features, 160 KB, one block an SM: 72 -> 31 us; 100 features, 40 KB, 20M points: 66 -> 48)
    const uint64_t fit = smem ? std::max<uint64_t>(1, (200 * 1024) / smem) : 8;
    unsigned threads = kFilterThreads;
    auto resident = [&](unsigned t) { return std::min<uint64_t>(fit, 2048 / t) * t; };
    for (unsigned t = 2 * kFilterThreads; t <= (unsigned)kPairThreads; t *= 2)
        if (resident(t) > resident(threads)) threads = t;
    const uint64_t per_sm = std::min<uint64_t>(fit, 2048 / threads);
    const uint64_t blocks = std::min<uint64_t>((uint64_t)b.sms * per_sm, (b.capR + threads - 1) / threads);
    if (!blocks) return;
    KScope ks("filter_pairs");
    if (b.pair_queue) {
        k_filter_pairs_queue<<<(unsigned)blocks, threads, smem, s>>>(
            b.ctrl.get(), b.pairq.get(), b.crun.get(), b.grids.get(), b.nbmask.get(), b.W, b.rfeat.get(),
            b.rstart.get(), b.ub2(), acc_dim);
        COLO_LAUNCH_CHECK();
        count_launch();
        return;
    }
    k_filter_pairs<<<(unsigned)blocks, threads, smem, s>>>(
        b.ctrl.get(), b.rcell.get(), b.J > 1 ? b.cjob.get() : nullptr, b.grids.get(), b.nbmask.get(), b.W,
        b.rfeat.get(), b.rstart.get(), b.job_off.get(), b.ub2(), acc_dim);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void filter_level(Batch& b, const uint32_t* h_cand, const uint32_t* h_job, uint64_t ncand, uint32_t k,
                  uint32_t* d_ub, unsigned long long* d_stats) {
    if (ncand == 0) return;
    if (b.W > kMaxW) throw StatusError{COLO_ERR_CAPACITY, "the filter handles at most 1024 features per job"};
    cudaStream_t s = b.s;
    const uint32_t m = k < kMaxMembersFiltered ? k : (uint32_t)kMaxMembersFiltered;
    // driver = member with the shortest driver list (the fewest cells with it in
    // their 3x3 block: the cells its candidates are tested on); candidates
    // grouped by driver; per candidate its need mask and local member ids
    // (16 bits each)
    std::vector<uint32_t> drv(ncand), need((size_t)ncand * b.W, 0), lmem((size_t)ncand * 4, 0);
    for (uint64_t c = 0; c < ncand; ++c) {
        const uint32_t* mem = h_cand + c * k;
        const uint32_t f0 = b.jobs[h_job[c]].grid.f0;
        uint32_t best = mem[0];
        uint64_t bn = UINT64_MAX;
        for (uint32_t j = 0; j < m; ++j) {
            const uint64_t nr = b.h_dcnt[mem[j]];
            if (nr < bn) {
                bn = nr;
                best = mem[j];
            }
            uint32_t lf = mem[j] - f0;
            need[(size_t)c * b.W + (lf >> 5)] |= 1u << (lf & 31);
            lmem[(size_t)c * 4 + (j >> 1)] |= lf << ((j & 1) * 16);
        }
        drv[c] = best;
    }
    std::vector<uint32_t> order(ncand);
    for (uint64_t c = 0; c < ncand; ++c) order[c] = (uint32_t)c;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t c) { return drv[a] < drv[c]; });
    std::vector<uint32_t> dcount(b.F, 0), dstart(b.F, 0);
    for (uint64_t i = 0; i < ncand; ++i) {
        const uint32_t fd = drv[order[i]];
        if (dcount[fd]++ == 0) dstart[fd] = (uint32_t)i;
    }
    uint64_t nitems = 0;   // (driver cell, candidate) pairs: the work the driver choice bounds
    for (uint32_t f = 0; f < b.F; ++f) nitems += (uint64_t)dcount[f] * (b.h_frun_off[f + 1] - b.h_frun_off[f]);
    b.filter_items += nitems;
    if (nitems == 0) return;
    {
        std::vector<uint8_t> need(b.F, 0);   // the drivers' lists (a later level's new driver refills)
        for (uint64_t c = 0; c < ncand; ++c) need[drv[c]] = 1;
        driver_lists_fill(b, need);
    }
    // groups (one per driver) and their units: 32 list cells x up to cu candidates
    const uint32_t cu = (b.filter_unit == 8 || b.filter_unit == 16) ? (uint32_t)b.filter_unit : 32u;
    std::vector<uint32_t> gfeat, gstart, gcount;
    std::vector<uint64_t> uoff(1, 0);
    for (uint32_t f = 0; f < b.F; ++f) {
        if (!dcount[f]) continue;
        const uint64_t L = b.h_doff[f + 1] - b.h_doff[f];
        gfeat.push_back(f);
        gstart.push_back(dstart[f]);
        gcount.push_back(dcount[f]);
        uoff.push_back(uoff.back() + (L + 31) / 32 * ((dcount[f] + cu - 1) / cu));
    }
    const uint32_t ngroups = (uint32_t)gfeat.size();
    const uint64_t nunits = uoff.back();
    if (nunits == 0) return;
    // one upload: need | lmem | order | gfeat | gstart | gcount | uoff (u64), mask rows and the
    // u64 part on 16-byte boundaries
    auto up4 = [](size_t v) { return (v + 3) & ~(size_t)3; };
    const size_t n_need = up4(need.size()), n_lmem = up4(lmem.size()), n_ord = up4(order.size());
    const size_t n_g = up4(ngroups);
    std::vector<uint32_t> pack(n_need + n_lmem + n_ord + 3 * n_g + 2 * uoff.size(), 0);
    size_t o = 0;
    std::copy(need.begin(), need.end(), pack.begin() + o);
    o += n_need;
    std::copy(lmem.begin(), lmem.end(), pack.begin() + o);
    o += n_lmem;
    std::copy(order.begin(), order.end(), pack.begin() + o);
    o += n_ord;
    std::copy(gfeat.begin(), gfeat.end(), pack.begin() + o);
    std::copy(gstart.begin(), gstart.end(), pack.begin() + o + n_g);
    std::copy(gcount.begin(), gcount.end(), pack.begin() + o + 2 * n_g);
    o += 3 * n_g;
    std::memcpy(pack.data() + o, uoff.data(), uoff.size() * 8);
    DevBuf<uint32_t> dpack;
    dpack.alloc(pack.size(), s);
    staged_upload(b.ctx, s, dpack.get(), pack.data(), pack.size() * 4);
    const uint32_t* d_need = dpack.get();
    const uint32_t* d_lmem = d_need + n_need;
    const uint32_t* d_order = d_lmem + n_lmem;
    const uint32_t* d_gfeat = d_order + n_ord;
    const uint32_t* d_gstart = d_gfeat + n_g;
    const uint32_t* d_gcount = d_gstart + n_g;
    const uint64_t* d_uoff = reinterpret_cast<const uint64_t*>(d_gcount + n_g);
    // block-private sums when the level's counters fit in 64 KB of shared memory
    const uint64_t acc64 = ncand * (uint64_t)(m + 2);
    const uint32_t acc_n = acc64 <= kAccMax ? (uint32_t)acc64 : 0u;
    const size_t smem = (size_t)acc_n * 4;
    // a grid-stride loop over units (one warp each): as many blocks as fit at once
    auto grid = [&](const void* fn) {
        if (smem > 48 * 1024)
            COLO_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        COLO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, smem));
        const uint64_t cap = (uint64_t)b.sms * (uint64_t)(per_sm > 0 ? per_sm : 1);
        const uint64_t want = (nunits + 7) / 8;
        return (unsigned)(want < cap ? want : cap);
    };
    KScope ks("filter_level");
#define COLO_FL(WW)                                                                                             \
    k_filter_drv<WW><<<grid((const void*)k_filter_drv<WW>), 256, smem, s>>>(                                    \
        nunits, ngroups, d_uoff, d_gfeat, d_gstart, d_gcount, b.doff.get(), b.dlist.get(), d_order, d_need,       \
        d_lmem, k, b.qmask.get(), b.cmask.get(), b.crun.get(), b.nbrs.get(), b.rstart.get(), d_ub, d_stats, acc_n, cu)
    COLO_W_SWITCH(b.W, COLO_FL)
#undef COLO_FL
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace colo
