// colo_level.cu -- level-wise instance tables and participation bitmaps.
//
// Reference semantics (generalInstanceTableSlotCounter_Kernel and
// generateInstanceTableGeneral_Kernel, Codes/DeviceProcess_Kernel.h:255-385;
// degree 2: 12-100): for a candidate (c_0..c_{k-1}) with parent table
// T(c_0..c_{k-2}), row r extends by b when b is an instance of c_{k-1} in a
// cell adjacent to r[0]'s cell with sq(r[i], b) <= R^2 for every i.  The
// candidates b of r are exactly N+_{c_{k-1}}(r[0]), a contiguous slice of the
// neighbour CSR (features ascend along each list), so the cell test and the
// r[0] distance test are already done; rows check the other k-2 members.
//
// Work decomposition: a warp owns a chunk of 32 parent rows.  Their slices are
// flattened with a warp prefix sum and the warp walks the flattened items 32
// at a time, so a row with 10^4 candidates and a row with none cost the same
// per item (load-balanced expand).  Output rows are ordered by parent row and
// then by candidate, which is the order of the flattened items: a hit's row is
// the rows of the candidate's earlier chunks plus the hits before it in its own
// chunk, one ballot per step.  So the count pass leaves one number per chunk,
// and the fill needs the scan of those (a count and an offset per parent row
// took 12 bytes a row and scans of 0.93 ms a mine on a batch of 128 jobs; the
// chunks' scans take 0.12 ms).  Output rows are written column-major (one
// coalesced stream per column).  Participation bits are set with atomicOr on
// 32-bit words.
//
// The count pass takes the candidates that share a parent table together
// (k_level_count): they read the same rows and the same lists.
//
// The single pass (presized tables, COLO_MODE_LEARNED) writes rows in the
// same order as count + fill: a warp takes its chunk by ticket (chunks of
// warps already running come first), counts its hits, publishes the count,
// and looks back over the candidate's earlier chunks (decoupled look-back,
// every wait bounded) for the rows before it; it then writes its rows at
// their exact offsets, replaying the ballots it kept (steps beyond the kept
// ones are evaluated again).
#include <algorithm>

#include "colo_batch.h"
#include "colo_device.cuh"

namespace colo {
namespace {

enum { MODE_FILL = 1, MODE_SINGLE = 2 };

// Participation bits: a word is read (from L2) before the atomic, so a bit
// already set costs a load, not another atomic on the same address -- in
// dense data thousands of rows hit the same few words.  A stale read only
// costs an extra (idempotent) atomic.
__device__ __forceinline__ void set_bit(uint32_t* words, uint32_t bit) {
    uint32_t* w = &words[bit >> 5];
    const uint32_t m = 1u << (bit & 31);
    if (!(__ldcg(w) & m)) atomicOr(w, m);
}

constexpr unsigned long long kChunkA = 1ull << 62;   // chunk count published
constexpr unsigned long long kChunkP = 2ull << 62;   // inclusive prefix published
constexpr unsigned long long kChunkVal = (1ull << 62) - 1;
constexpr uint32_t kChunkSpin = 1u << 22;

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The last group (or candidate) whose first chunk is at or before ch, by a 32-way search: the
// lanes probe 32 evenly spaced prefixes per round, so a few dependent loads instead of one per
// halving.
__device__ __forceinline__ uint64_t chunk_owner(const uint64_t* __restrict__ first_chunk, uint64_t n, uint64_t ch) {
    const int lane = threadIdx.x & 31;
    uint64_t lo = 0, hi = n;   // answer in [lo, hi)
    while (hi - lo > 1) {
        const uint64_t span = hi - lo;
        const uint64_t step = span <= 32 ? 1 : (span + 31) / 32;
        const uint64_t probe = lo + (uint64_t)lane * step;
        const bool le = probe < hi && first_chunk[probe] <= ch;
        const uint32_t bal = __ballot_sync(0xffffffffu, le);   // lane 0 (probe lo) is always set
        const int last = 31 - __clz(bal);
        const uint64_t nlo = lo + (uint64_t)last * step;
        hi = nlo + step < hi ? nlo + step : hi;
        lo = nlo;
    }
    return lo;
}

// ---- count pass -------------------------------------------------------------
// Candidates that share a parent table (their first k-1 members) are counted
// together, up to 32 at a time: group g holds candidates gstart[g] ..
// gstart[g+1], whose last members, its extensions, ascend.  A warp reads the
// chunk's rows and walks, per row, the slice of its list from the first
// extension's feature to the last one's; lane e knows extension e's id range,
// and an item finds its extension by a search over the lanes (none for groups of
// one).  Per (row, extension) one lane, the first of its hits in the step, marks
// the row and adds the step's hits in shared memory.
//
// Bound by the chain of dependent loads a chunk starts with (rows, list starts,
// two searches in the list): sharing it among the extensions is what this kernel
// is for: the counts of a batch of 128 jobs (levels 2 to 6, 29,514 candidates)
// went 7.73 -> 3.14 ms, of the 20M workload 0.46 -> 0.38 ms, of 200,000 dense
// points 1.22 -> 1.02 ms; a level of a few thousand rows takes 2 us longer.  Held
// to 40 registers (32 for pairs) for more resident warps: with the compiler's own
// choice from size 5 on the same counts took 3.79, 0.38 and 1.32 ms; list entries
// fetched two steps ahead and coordinates one (more registers) gained nothing.
//
// K = pattern size (2..8), or 0 for a runtime size read from the descriptor
// (members kept in global memory, slower; only reached for k > 8).
constexpr int kCountWarps = 8;

// VERDICT: the candidates' filter bounds are tested here (ub, need; not for pairs).
// SPLIT: 1 << split_log warps share a chunk: each reads its rows and takes every so many-th step of
// their items (chunk_rows zeroed beforehand).
template <int K, bool VERDICT, bool SPLIT>
__global__ void __launch_bounds__(32 * kCountWarps, K == 2 ? 8 : 6) k_level_count(
    const CandDesc* __restrict__ cands, const uint32_t* __restrict__ gstart, const uint64_t* __restrict__ gchunk,
    uint64_t ngroups, uint64_t chunk0, uint64_t nchunks, const uint64_t* __restrict__ nb_beg,
    const uint32_t* __restrict__ nb_cnt, const uint32_t* __restrict__ nb, const float2* __restrict__ xy,
    unsigned long long* __restrict__ items, unsigned long long* __restrict__ ticket, int persistent,
    const uint32_t* __restrict__ ub, const uint32_t* __restrict__ need, uint32_t split_log) {
    constexpr int KR = (K == 0) ? 1 : K;   // register members kept for K > 0
    __shared__ uint32_t s_cnt[kCountWarps][32], s_row[kCountWarps][32];   // hits per extension, extensions hit per row
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    s_cnt[wid][lane] = 0;
    s_row[wid][lane] = 0;
    __syncwarp();
    for (bool once = true;; once = false) {
        uint64_t ch = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (persistent) {
            unsigned long long tk = 0;
            if (lane == 0) tk = atomicAdd(ticket, 1ull);
            ch = __shfl_sync(0xffffffffu, tk, 0);
        } else if (!once) {
            break;
        }
        if (ch >= (SPLIT ? nchunks << split_log : nchunks)) break;
        const uint32_t part = SPLIT ? (uint32_t)ch & ((1u << split_log) - 1u) : 0u;
        ch = chunk0 + (SPLIT ? ch >> split_log : ch);
        const uint64_t g = chunk_owner(gchunk, ngroups, ch);
        const uint32_t q0 = gstart[g], n = gstart[g + 1] - q0;
        const CandDesc& d = cands[q0];
        const uint32_t k = (K == 0) ? d.k : (uint32_t)K;
        const uint64_t row = (ch - gchunk[g]) * 32 + lane;
        const bool valid = row < d.prow;
        // lane e: extension e's ids (a lane without one gets none) and its candidate's bitmaps
        uint32_t est = 0xffffffffu, eend = 0;
        uint64_t ebm = 0;
        if ((uint32_t)lane < n) {
            const CandDesc& c = cands[q0 + lane];
            est = c.last_start;
            eend = c.last_end;
            ebm = c.bm_base + c.last_off;
        }
        if (VERDICT) {
            // the filter's verdict was not waited for: a candidate passes when every member's bound
            // reaches the least one that its ratio test accepts; the others extend no row
            bool pass = (uint32_t)lane < n;
            if (pass)
                for (uint32_t i = 0; i < k; ++i) pass &= ub[(uint64_t)(q0 + lane) * k + i] >= need[(uint64_t)(q0 + lane) * k + i];
            if (!pass) eend = 0;
            if (!__any_sync(0xffffffffu, pass)) {
                if (!SPLIT && (uint32_t)lane < n) cands[q0 + lane].chunk_rows[row >> 5] = 0;
                continue;
            }
        }
        const float R2 = d.R2, hu = d.R2hu;

        // row members (ids) and coordinates of members 1..k-2
        uint32_t rid[KR];
        float rx[KR], ry[KR];
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            rid[i] = 0;
            rx[i] = 0.f;
            ry[i] = 0.f;
        }
        uint32_t a0 = 0, len = 0;
        uint64_t from = 0;
        if (valid) {
            a0 = d.parent ? d.parent[row] : d.mem[0].start + (uint32_t)row;
            if (K > 0) {
                rid[0] = a0;
#pragma unroll
                for (int i = 1; i < KR - 1; ++i) {
                    rid[i] = d.parent[(uint64_t)i * d.pstride + row];
                    const float2 pi = xy[rid[i]];
                    rx[i] = pi.x;
                    ry[i] = pi.y;
                }
            }
            const uint32_t cnt = nb_cnt[a0];
            const uint64_t o0 = nb_beg[a0];   // (unset where cnt is 0; loaded beside it)
            const uint32_t b0 = lower_bound_u32(nb + o0, 0u, cnt, d.last_start);   // 32-bit positions within the list
            len = lower_bound_u32(nb + o0, b0, cnt, cands[q0 + n - 1].last_end) - b0;
            from = o0 + b0;
        }
        // flatten the 32 slices: item t of the chunk is entry from_j + t of the lists, j its row's lane
        const uint32_t incl = warp_incl_scan(len);
        const uint32_t excl = incl - len;
        from -= excl;
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t mine = 0;   // items of the chunk's extensions (this lane's)
        for (uint32_t t0 = SPLIT ? part * 32 : 0u; t0 < total; t0 += SPLIT ? 32u << split_log : 32u) {
            const uint32_t item = t0 + lane;
            int j = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t ev = __shfl_sync(0xffffffffu, excl, j + step);
                if (ev <= item) j += step;
            }
            const uint64_t from_j = __shfl_sync(0xffffffffu, from, j);
            bool ok = item < total;
            const uint32_t b = ok ? nb[from_j + item] : 0u;
            float2 pb = make_float2(0.f, 0.f);
            if (K != 2 && ok) pb = xy[b];
            // the item's extension: the last one that starts at or before b, if b is one of its ids
            int e = 0;
            if (n > 1) {
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    if ((uint32_t)step >= n) continue;
                    const uint32_t v = __shfl_sync(0xffffffffu, est, e + step);   // lanes past n hold no start
                    if (v <= b) e += step;
                }
                const uint32_t eend_e = __shfl_sync(0xffffffffu, eend, e);   // (by every lane)
                ok = ok && b < eend_e;
            }
            const uint32_t est_e = __shfl_sync(0xffffffffu, est, e);
            const uint64_t bm_e = __shfl_sync(0xffffffffu, ebm, e);
            mine += ok ? 1u : 0u;
            if (K == 0) {
                if (ok && k > 2) {
                    const uint64_t prow_j = row - lane + (uint64_t)j;
                    for (uint32_t i = 1; i + 1 < k && ok; ++i) {
                        const float2 pr = xy[d.parent[(uint64_t)i * d.pstride + prow_j]];
                        ok = ref_within(pr.x, pr.y, pb.x, pb.y, R2, hu);
                    }
                }
            } else if (K > 2) {
#pragma unroll
                for (int i = 1; i < KR - 1; ++i) {
                    const float xi = __shfl_sync(0xffffffffu, rx[i], j);
                    const float yi = __shfl_sync(0xffffffffu, ry[i], j);
                    ok = ok && ref_within(xi, yi, pb.x, pb.y, R2, hu);
                }
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, ok);
            if (!bal) continue;
            // hits of one row and extension are next to each other: the first one acts for them
            const uint32_t before = bal & lt;
            const int prev = before ? 31 - __clz(before) : lane;
            const uint32_t key = (uint32_t)j << 5 | (uint32_t)e;
            const uint32_t pkey = __shfl_sync(0xffffffffu, key, prev);
            const bool lead = ok && (!before || pkey != key);
            const uint32_t leads = __ballot_sync(0xffffffffu, lead);
            if (ok) set_bit(d.bitmap + bm_e, b - est_e);
            if (lead) {
                const uint32_t later = leads & ~lt & ~(1u << lane);   // the next leader ends this one's hits
                const uint32_t upto = later ? (1u << (__ffs(later) - 1)) - 1u : 0xffffffffu;
                atomicAdd(&s_cnt[wid][e], (uint32_t)__popc(bal & ~lt & upto));
                atomicOr(&s_row[wid][j], 1u << e);
            }
        }
        __syncwarp();
        const uint32_t hits = s_cnt[wid][lane];
        uint32_t marks = s_row[wid][lane];
        __syncwarp();
        s_cnt[wid][lane] = 0;
        s_row[wid][lane] = 0;
        if ((uint32_t)lane < n) {
            const CandDesc& c = cands[q0 + lane];
            if (!SPLIT) c.chunk_rows[row >> 5] = hits;
            else if (hits) atomicAdd(&c.chunk_rows[row >> 5], hits);
            if (hits) atomicAdd(c.rows, (unsigned long long)hits);
        }
        if (items && total) {
            mine = __reduce_add_sync(0xffffffffu, mine);
            if (lane == 0 && mine) atomicAdd(items, (unsigned long long)mine);
        }
        for (; marks; marks &= marks - 1) {
            const uint64_t bm = cands[q0 + __ffs(marks) - 1].bm_base;
            set_bit(d.bitmap + bm, a0 - d.mem[0].start);   // (members 0..k-2 are every extension's)
            if (K > 0) {
#pragma unroll
                for (int q = 1; q < KR - 1; ++q) set_bit(d.bitmap + bm + d.mem[q].off, rid[q] - d.mem[q].start);
            } else {
                for (uint32_t i = 1; i + 1 < k; ++i)
                    set_bit(d.bitmap + bm + d.mem[i].off, d.parent[(uint64_t)i * d.pstride + row] - d.mem[i].start);
            }
        }
        __syncwarp();
    }
}

// ---- fill and single pass ---------------------------------------------------
// K as in the count pass.  The kernel is latency-bound (a chain of dependent
// loads per warp), so the fill form is held to fewer registers for more resident
// warps: pairs at six 256-thread blocks per SM, size 3 at five, size 4 at four (a
// few registers spill; larger sizes would spill more).  On the 20M workload the
// fills went 0.173 -> 0.158 ms per step.
template <int K, int MODE>
__global__ void __launch_bounds__(256, (MODE == MODE_FILL && K == 2) ? 6 : (MODE != MODE_SINGLE && K == 3) ? 5 : (MODE != MODE_SINGLE && K == 4) ? 4 : 1) k_level(
    const CandDesc* __restrict__ cands, const uint64_t* __restrict__ chunk_off, uint64_t ncand,
    uint64_t nchunks, const uint64_t* __restrict__ nb_beg, const uint32_t* __restrict__ nb_cnt,
    const uint32_t* __restrict__ nb,
    const float2* __restrict__ xy, uint32_t* __restrict__ overflow, unsigned long long* __restrict__ items,
    unsigned long long* __restrict__ chunk_status, unsigned long long* __restrict__ ticket,
    uint32_t* __restrict__ timeout, int persistent) {
    constexpr int KR = (K == 0) ? 1 : K;   // register members kept for K > 0
    const int lane = threadIdx.x & 31;
    // one chunk per warp, or (persistent) warps that take chunk tickets until none is left; the
    // single pass always takes tickets, so its chunks run in the order warps start them
    const bool by_ticket = MODE == MODE_SINGLE || persistent;
    for (bool first = true;; first = false) {
    uint64_t ch = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (by_ticket) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(ticket, 1ull);
        ch = __shfl_sync(0xffffffffu, tk, 0);
    } else if (!first) {
        break;
    }
    if (ch >= nchunks) break;
    const uint64_t lo = chunk_owner(chunk_off, ncand, ch);
    const CandDesc& d = cands[lo];
    const uint32_t k = (K == 0) ? d.k : (uint32_t)K;
    const uint64_t row = (ch - chunk_off[lo]) * 32 + lane;
    const bool valid = row < d.prow;
    const uint64_t bm_last = d.bm_base + d.last_off;
    const uint32_t last_start = d.last_start, last_end = d.last_end;
    const float R2 = d.R2, hu = d.R2hu;

    // row members (ids) and coordinates of members 1..k-2
    uint32_t rid[KR];
    float rx[KR], ry[KR];
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        rid[i] = 0;
        rx[i] = 0.f;
        ry[i] = 0.f;
    }
    uint32_t a0 = 0;
    uint64_t slo = 0, shi = 0;
    if (valid) {
        a0 = d.parent ? d.parent[row] : d.mem[0].start + (uint32_t)row;
        if (K > 0) {
            rid[0] = a0;
#pragma unroll
            for (int i = 1; i < KR - 1; ++i) {
                rid[i] = d.parent[(uint64_t)i * d.pstride + row];
                const float2 pi = xy[rid[i]];
                rx[i] = pi.x;
                ry[i] = pi.y;
            }
        }
        const uint32_t cnt = nb_cnt[a0];
        const uint64_t o0 = nb_beg[a0];   // (unset where cnt is 0; loaded beside it)
        const uint32_t* list = nb + o0;
        const uint32_t b0 = lower_bound_u32(list, 0u, cnt, last_start);   // 32-bit positions within the list
        slo = o0 + b0;
        shi = o0 + lower_bound_u32(list, b0, cnt, last_end);
    }
    // flatten the 32 slices
    uint32_t len = (uint32_t)(shi - slo);
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const uint32_t excl = incl - len;
    const uint64_t from = slo - excl;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (MODE == MODE_SINGLE && items && lane == 0 && total) atomicAdd(items, (unsigned long long)total);
    uint32_t hits = 0;               // hits of the chunk so far
    bool mine = false;               // this lane's row has a hit
    uint64_t out0 = 0;               // output row of the chunk's first hit
    if (MODE == MODE_FILL) out0 = d.offs[row >> 5] - d.offs[0];   // offsets are a slice of the level's scan
    const uint32_t lt = (1u << lane) - 1u;
    bool ovf = false;
    const uint64_t chunk_row0 = row - lane;

    // item t0 + lane: its owner row (lane j), and whether b extends the row (the other k-2
    // members within R)
    struct Item {
        int j;
        uint32_t b;
        bool active;
    };
    auto locate = [&](uint32_t t0) {
        Item it;
        const uint32_t item = t0 + lane;
        it.active = item < total;
        int j = 0;
#pragma unroll
        for (int bstep = 16; bstep > 0; bstep >>= 1) {
            uint32_t ev = __shfl_sync(0xffffffffu, excl, j + bstep);
            if (ev <= item) j += bstep;
        }
        it.j = j;
        // slo - excl, so that item t of the warp is entry from_j + t of the lists
        const uint64_t from_j = __shfl_sync(0xffffffffu, from, j);
        it.b = it.active ? nb[from_j + item] : 0u;
        return it;
    };
    auto extends = [&](const Item& it) {
        bool ok = it.active;
        if (K == 0) {
            if (it.active && k > 2) {
                const float2 pb = xy[it.b];
                const uint64_t prow_j = chunk_row0 + (uint64_t)it.j;
                for (uint32_t i = 1; i + 1 < k && ok; ++i) {
                    uint32_t ri = d.parent[(uint64_t)i * d.pstride + prow_j];
                    const float2 pr = xy[ri];
                    ok = ref_within(pr.x, pr.y, pb.x, pb.y, R2, hu);
                }
            }
        } else if (K > 2) {
            float xb = 0.f, yb = 0.f;
            if (it.active) {
                const float2 pb = xy[it.b];
                xb = pb.x;
                yb = pb.y;
            }
#pragma unroll
            for (int i = 1; i < KR - 1; ++i) {
                float xi = __shfl_sync(0xffffffffu, rx[i], it.j);
                float yi = __shfl_sync(0xffffffffu, ry[i], it.j);
                ok = ok && ref_within(xi, yi, xb, yb, R2, hu);
            }
        }
        return ok;
    };
    // lanes of step t0 that belong to my own row
    auto own_mask = [&](uint32_t t0) {
        int r0 = (int)excl - (int)t0, r1 = (int)incl - (int)t0;
        r0 = r0 < 0 ? 0 : r0;
        r1 = r1 > 32 ? 32 : r1;
        return (r1 > r0) ? ((r1 - r0 == 32) ? 0xffffffffu : (((1u << (r1 - r0)) - 1u) << r0)) : 0u;
    };
    // writes the hits of one step
    auto write_step = [&](const Item& it, bool ok, uint32_t bal, uint64_t col_stride, bool capped) {
        const uint64_t pos = out0 + hits + __popc(bal & lt);
        const bool room = !capped || pos < d.out_cap;
        if (ok && !room) ovf = true;
        const bool wr = ok && room;
        if (K > 0) {
#pragma unroll
            for (int i = 0; i < KR - 1; ++i) {
                uint32_t v = __shfl_sync(0xffffffffu, rid[i], it.j);
                if (wr) d.out[(uint64_t)i * col_stride + pos] = v;
            }
        } else if (wr) {
            const uint64_t prow_j = chunk_row0 + (uint64_t)it.j;
            d.out[pos] = d.parent ? d.parent[prow_j] : d.mem[0].start + (uint32_t)prow_j;
            for (uint32_t i = 1; i + 1 < k; ++i)
                d.out[(uint64_t)i * col_stride + pos] = d.parent[(uint64_t)i * d.pstride + prow_j];
        }
        if (wr) d.out[(uint64_t)(k - 1) * col_stride + pos] = it.b;
    };

    uint32_t bal_lo = 0, bal_hi = 0;   // single pass: ballot of step s kept in lane s % 32 (s < 64)
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const Item it = locate(t0);
        const bool ok = extends(it);
        const uint32_t bal = __ballot_sync(0xffffffffu, ok);
        if (MODE == MODE_SINGLE) {
            mine |= (bal & own_mask(t0)) != 0;
            if (ok) set_bit(d.bitmap + bm_last, it.b - last_start);
            const uint32_t step = t0 >> 5;
            if (step < 32 && lane == (int)step) bal_lo = bal;
            else if (step >= 32 && step < 64 && lane == (int)(step - 32)) bal_hi = bal;
        }
        if (MODE == MODE_FILL) write_step(it, ok, bal, d.out_rows, false);
        hits += __popc(bal);
    }
    if (MODE == MODE_SINGLE) {
        // the chunk's rows, then the rows of the candidate's earlier chunks: the warp reads 32
        // predecessors' words at once, back to the nearest published prefix
        const uint32_t wsum = hits;
        const uint64_t first = chunk_off[lo];
        unsigned long long prefix = 0;
        if (lane == 0) *(volatile unsigned long long*)(chunk_status + ch) = (first == ch ? kChunkP : kChunkA) | wsum;
        if (first != ch) {
            uint32_t spins = 0;
            int64_t base = (int64_t)ch - 1;
            while (true) {
                const int64_t t = base - lane;
                // words before the candidate's first chunk read as an empty published prefix
                const unsigned long long v =
                    t >= (int64_t)first ? *(volatile const unsigned long long*)(chunk_status + t) : kChunkP;
                const unsigned long long flag = v & ~kChunkVal;
                const uint32_t pm = __ballot_sync(0xffffffffu, flag == kChunkP);
                const uint32_t zm = __ballot_sync(0xffffffffu, flag == 0);
                const int fp = pm ? __ffs(pm) - 1 : 32;                 // nearest published prefix
                const uint32_t upto = fp == 32 ? 0xffffffffu : ((2u << fp) - 1u);
                if (zm & upto) {                                         // a chunk before it not counted yet
                    if (++spins > kChunkSpin) {                          // give up: report it, write with what we have
                        if (lane == 0) atomicOr(timeout, 1u);
                        break;
                    }
                    __nanosleep(64);
                    continue;
                }
                prefix += warp_sum_u64(((upto >> lane) & 1u) ? (v & kChunkVal) : 0ull);
                if (fp < 32) break;
                base -= 32;
            }
            if (lane == 0) *(volatile unsigned long long*)(chunk_status + ch) = kChunkP | (prefix + wsum);
        }
        out0 = prefix;
        hits = 0;
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
            const Item it = locate(t0);
            const uint32_t step = t0 >> 5;
            bool ok;
            if (step < 64) {
                const uint32_t kept = __shfl_sync(0xffffffffu, step < 32 ? bal_lo : bal_hi, (int)(step & 31));
                ok = it.active && ((kept >> lane) & 1u);
            } else {
                ok = extends(it);
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, ok);
            write_step(it, ok, bal, d.out_cap, true);
            hits += __popc(bal);
        }
    }
    if (MODE == MODE_SINGLE) {
        if (__any_sync(0xffffffffu, ovf) && lane == 0) atomicOr(&overflow[lo], 1u);
    }
    if (MODE == MODE_SINGLE && lane == 0) {
        d.chunk_rows[row >> 5] = hits;
        if (hits) atomicAdd(d.rows, (unsigned long long)hits);
    }
    if (MODE == MODE_SINGLE && valid) {
        if (mine) {
            uint32_t* bm = d.bitmap + d.bm_base;
            set_bit(bm, a0 - d.mem[0].start);
            if (K > 0) {
#pragma unroll
                for (int q = 1; q < KR - 1; ++q) set_bit(bm + d.mem[q].off, rid[q] - d.mem[q].start);
            } else {
                for (uint32_t i = 1; i + 1 < k; ++i)
                    set_bit(bm + d.mem[i].off, d.parent[(uint64_t)i * d.pstride + row] - d.mem[i].start);
            }
        }
    }
    }   // chunks of this warp
}

// Kept tables, row-major: one y block row per piece.  Bound by the copy that follows over the host
// link; turning the columns into rows on the host, table by table, took 20 us a table.
__global__ void __launch_bounds__(256) k_table_rows(const TablePiece* __restrict__ pieces, uint32_t k,
                                                    uint32_t* __restrict__ out) {
    const TablePiece p = pieces[blockIdx.y];
    const uint64_t words = p.rows * k;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i / k;
        out[p.at + i] = p.cols[(i - row * k) * p.stride + p.row0 + row];
    }
}

// Participation statistics: per (candidate, member) [A, last, first, full]
// where A counts set bits in [0, n-2] (the window getParticipationIndex sums,
// Codes/DeviceProcess.cu:108-132).  A block takes one (candidate, member)
// pair (blockIdx.x) and one span of kPiSpan bitmap words (blockIdx.y; spans
// past the member's bitmap leave at once) and adds its counts to the zeroed
// statistics; the spans holding bit 0 and bit n-1 also record first and last.
constexpr uint32_t kPiSpan = 16384;

__global__ void __launch_bounds__(256) k_level_pi(const CandDesc* __restrict__ cands, uint32_t k,
                                                  uint64_t* __restrict__ stats) {
    const uint64_t c = blockIdx.x / k;
    const uint32_t j = blockIdx.x - (uint32_t)(c * k);
    const CandDesc& d = cands[c];
    const MemberInfo mi = d.mem[j];
    const uint32_t n = mi.n;
    const uint32_t nw = (n + 31) / 32;
    const uint32_t w0 = blockIdx.y * kPiSpan;
    if (w0 >= nw) return;
    const uint32_t w1 = w0 + kPiSpan < nw ? w0 + kPiSpan : nw;
    const uint32_t* w = d.bitmap + d.bm_base + mi.off;
    const uint32_t lim = n - 1;   // bits in the window [0, n-2]
    unsigned long long cntA = 0, cntFull = 0;
    for (uint32_t i = w0 + threadIdx.x; i < w1; i += blockDim.x) {
        const uint32_t v = w[i];
        cntFull += __popc(v);
        const uint32_t wb = i * 32;
        const uint32_t mask = wb + 32 <= lim ? 0xffffffffu : (wb >= lim ? 0u : (1u << (lim - wb)) - 1u);
        cntA += __popc(v & mask);
    }
    __shared__ unsigned long long red[8];
    for (int o = 16; o > 0; o >>= 1) {
        cntA += __shfl_down_sync(0xffffffffu, cntA, o);
        cntFull += __shfl_down_sync(0xffffffffu, cntFull, o);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) red[wid] = cntA | (cntFull << 32);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long A = 0, Fu = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
            A += red[q] & 0xffffffffull;
            Fu += red[q] >> 32;
        }
        uint64_t* o = stats + (c * k + j) * 4;
        if (A) atomicAdd(reinterpret_cast<unsigned long long*>(o + 0), A);
        if (Fu) atomicAdd(reinterpret_cast<unsigned long long*>(o + 3), Fu);
        if (w0 == 0) o[2] = w[0] & 1u;
        if ((lim >> 5) >= w0 && (lim >> 5) < w1) o[1] = (w[lim >> 5] >> (lim & 31)) & 1u;
    }
}

template <int MODE>
void launch_level(Batch& b, const LevelWork& w, uint32_t k, uint32_t* ovf) {
    if (w.nchunks == 0) return;
    KScope ks(MODE == MODE_FILL ? "level_fill" : "level_single");
    const unsigned block = (b.level_block == 64 || b.level_block == 128) ? (unsigned)b.level_block : 256u;
    uint64_t threads = w.nchunks * 32;
    unsigned grid = (unsigned)((threads + block - 1) / block);
    // persistent queue: as many blocks as are resident at once (64 registers a thread: 32 warps
    // an SM), their warps taking chunk tickets (the ticket word follows the chunk words)
    const int persistent = (b.level_queue && MODE != MODE_SINGLE && w.ticket) ? 1 : 0;
    if (persistent) {
        const uint64_t cap = (uint64_t)b.sms * (32u * 32u / block);
        if (grid > cap) grid = (unsigned)cap;
    }
#define COLO_LVL(KK)                                                                              \
    k_level<KK, MODE><<<grid, block, 0, b.s>>>(w.cands, w.chunk_off, w.ncand, w.nchunks, b.nb_beg.get(), b.nb_cnt.get(), \
                                            b.nb.get(), b.xy.get(), ovf, w.items, w.chunk_status, w.ticket,    \
                                            &b.flags()->timeout, persistent)
    switch (k) {
        case 2: COLO_LVL(2); break;
        case 3: COLO_LVL(3); break;
        case 4: COLO_LVL(4); break;
        case 5: COLO_LVL(5); break;
        case 6: COLO_LVL(6); break;
        case 7: COLO_LVL(7); break;
        case 8: COLO_LVL(8); break;
        default: COLO_LVL(0); break;
    }
#undef COLO_LVL
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace

uint32_t count_split(const Batch& b, uint64_t nchunks) {
    // Where lists are long (four or more pairs tested a point) and the chunks do not fill the GPU,
    // up to 32 warps share a chunk: a chunk of long lists is hundreds of steps for one warp, and the
    // first levels of dense data are a thousand such chunks.  Counts with 14 to 30 pairs a point: 198 -> 158 us
    // (100,000 points), 970 -> 878 (200,000), 280 -> 134 (one hotspot of 4,000 points), and within 1% where
    // the chunks are many.  Short lists have no steps to share: at 3.2 pairs a point 42 -> 49.  512 warps an
    // SM are slower (1,094 on the 200,000 points); 64 are on the hotspot (184), but not on the 100,000 (130).
    const uint64_t warps = (uint64_t)b.sms * 192;
    uint32_t log = 0;
    while (b.join_pairs >= 4 * b.N && log < 5 && (nchunks << (log + 1)) <= warps) ++log;
    return log;
}

void level_count(Batch& b, const CountWork& w, uint32_t k) {
    if (w.nchunks == 0) return;
    KScope ks("level_count");
    const unsigned block = (b.level_block == 64 || b.level_block == 128) ? (unsigned)b.level_block : 256u;
    const uint32_t split_log = w.split_log;
    unsigned grid = (unsigned)(((w.nchunks << split_log) * 32 + block - 1) / block);
    const int persistent = (b.level_queue && w.ticket) ? 1 : 0;   // as launch_level's
    if (persistent) grid = (unsigned)std::min<uint64_t>(grid, (uint64_t)b.sms * (32u * 32u / block));
#define COLO_CNT(KK, V, S)                                                                                        \
    k_level_count<KK, V, S><<<grid, block, 0, b.s>>>(w.cands, w.gstart, w.gchunk, w.ngroups, w.chunk0, w.nchunks, \
                                               b.nb_beg.get(), b.nb_cnt.get(), b.nb.get(), b.xy.get(), w.items,   \
                                               w.ticket, persistent, w.ub, w.need, split_log)
#define COLO_CNT_K(KK)                                   \
    do {                                                 \
        if (w.ub && split_log) COLO_CNT(KK, true, true); \
        else if (w.ub) COLO_CNT(KK, true, false);        \
        else if (split_log) COLO_CNT(KK, false, true);   \
        else COLO_CNT(KK, false, false);                 \
    } while (0)
    switch (k) {
        case 2:
            if (split_log) COLO_CNT(2, false, true);
            else COLO_CNT(2, false, false);
            break;
        case 3: COLO_CNT_K(3); break;
        case 4: COLO_CNT_K(4); break;
        case 5: COLO_CNT_K(5); break;
        case 6: COLO_CNT_K(6); break;
        case 7: COLO_CNT_K(7); break;
        case 8: COLO_CNT_K(8); break;
        default: COLO_CNT_K(0); break;
    }
#undef COLO_CNT_K
#undef COLO_CNT
    COLO_LAUNCH_CHECK();
    count_launch();
}
void level_fill(Batch& b, const LevelWork& w, uint32_t k) { launch_level<MODE_FILL>(b, w, k, nullptr); }
void level_single(Batch& b, const LevelWork& w, uint32_t k, uint32_t* d_overflow) {
    launch_level<MODE_SINGLE>(b, w, k, d_overflow);
}

void table_rows(cudaStream_t s, const TablePiece* d_pieces, uint32_t n, uint32_t k, uint64_t most_words, uint32_t* out) {
    if (n == 0 || most_words == 0) return;
    KScope ks("table_rows");
    const unsigned gx = (unsigned)std::min<uint64_t>((most_words + 255) / 256, 1024);
    k_table_rows<<<dim3(gx, n), 256, 0, s>>>(d_pieces, k, out);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void level_pi(Batch& b, const CandDesc* d_cands, uint64_t ncand, uint32_t k, uint64_t* d_stats) {
    if (ncand == 0) return;
    if (ncand * k >= (1ull << 31)) throw StatusError{COLO_ERR_CAPACITY, "too many candidates in one level"};
    KScope ks("level_pi");
    // spans per member: enough for the largest feature of the batch
    uint32_t fmax = 0;
    for (uint32_t f = 0; f < b.F; ++f) fmax = std::max(fmax, b.h_fcount[f]);
    const uint32_t spans = std::max<uint32_t>(1, ((fmax + 31) / 32 + kPiSpan - 1) / kPiSpan);
    k_level_pi<<<dim3((unsigned)(ncand * k), spans), 256, 0, b.s>>>(d_cands, k, d_stats);
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace colo
