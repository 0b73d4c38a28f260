// colo_join.cu -- cell-pair spatial join producing the neighbour lists
//   N+(a) = {b : feat(b) > feat(a), cell(b) adjacent to cell(a), sq(a,b) <= R^2}
// each ordered by (feature, neighbour cell, b): exactly the order in which
// degree2TableSlotCounter_Kernel / generalInstanceTableSlotCounter_Kernel
// visit candidates (Codes/DeviceProcess_Kernel.h:12-55, 255-316).
//
// An anchor's targets are one slice of its cell's neighbourhood list (the
// suffix with higher features), so points without targets cost nothing and the
// anchors of a cell read the same list.  A warp takes a tile of 32 anchors,
// flattens their slices with a prefix sum and tests 32 (anchor, target) pairs a
// step whatever the slices' lengths; an anchor with a long slice gets a warp to
// itself.
//
// Single pass: a tile reserves room for all its pairs with one atomic and
// writes its hits there end to end, in the order of the flattened pairs, which
// is the order of each anchor's list; no counting pass is needed.  When that
// room would be too large, a count pass + scan + fill pass produces a compact
// layout instead.
#include <algorithm>
#include <cmath>
#include <vector>

#include "colo_batch.h"
#include "colo_device.cuh"

namespace colo {
namespace {

enum { J_SINGLE = 0, J_COUNT = 1, J_FILL = 2 };

constexpr int kLongSteps = 4;        // steps of 32 targets an iteration for an anchor with a long slice
constexpr uint64_t kJoinWaves = 8;   // waves of resident blocks at most (warps take tiles grid-stride)

// Bound by instruction issue and the dependent loads target -> coordinates.  Groups of eight lanes
// per anchor walking the lists run by run left most lanes idle, since runs average two points:
// 0.33 ms became 0.095 ms on 20 million points (1.2 M anchors, 2.7 M pairs; 0.11 ms on the 1.5 M and 3.7 M of
// another seed), 2.2 became 0.83 ms on a
// batch of 128 jobs (134 M pairs), 0.36 became 0.042 ms on 200,000 dense points (6 M pairs), where
// the longest slices alone, eight lanes each, took most of it.  Six blocks an SM (40 registers, some
// spilled) suit many short slices best (batch: 0.93 ms against 1.08 ms at four).
// `per` anchors a tile (32 / lanes per anchor).  The anchors are counted on the device; tiles are
// taken grid-stride.  Lists or neighbours that did not fit their room are left to a later launch.
template <int MODE>
__global__ void __launch_bounds__(256, 6) k_join(
    BatchCtrl* __restrict__ ctrl, uint64_t npoints, uint64_t targets_cap, uint64_t nb_cap, int per,
    const uint4* __restrict__ act, const uint32_t* __restrict__ ids, const uint32_t* __restrict__ sfeat,
    const float2* __restrict__ coords, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ fjob,
    const JobGrid* __restrict__ grids, uint64_t* __restrict__ nb_beg, uint32_t* __restrict__ nb_cnt,
    uint32_t* __restrict__ nb, unsigned long long* __restrict__ total) {
    if (ctrl->targets.v > targets_cap || (MODE == J_SINGLE && ctrl->pairs.v > nb_cap)) return;
    const uint64_t A = ctrl->anchors.v, AL = ctrl->long_anchors.v;
    const uint64_t tiles = (A + per - 1) / per;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long found = 0;
    // long slices first: they take longest
    for (uint64_t i = warp; i < AL + tiles; i += warps) {
        if (i < AL) {
            const uint4 an = act[npoints - 1 - i];
            const uint32_t a = ids ? ids[an.x] : an.x, L = an.y;
            const float2 pa = coords[an.x];
            const JobGrid& g = grids[fjob ? fjob[sfeat[an.x]] : 0u];   // fjob is null for one-job batches
            const float R2 = g.R2, hu = g.R2hu;
            const uint32_t* list = targets + ((uint64_t)an.w << 32 | an.z);
            unsigned long long base = 0;
            if (MODE == J_SINGLE && lane == 0) base = atomicAdd(&ctrl->nb_used.v, (unsigned long long)L);
            if (MODE == J_SINGLE) base = __shfl_sync(0xffffffffu, base, 0);
            if (MODE == J_FILL) base = nb_beg[a];
            uint32_t k = 0;
            for (uint32_t t0 = 0; t0 < L; t0 += 32 * kLongSteps) {   // several steps' loads in flight
                uint32_t p[kLongSteps];
                float2 pb[kLongSteps];
#pragma unroll
                for (int i = 0; i < kLongSteps; ++i) p[i] = t0 + i * 32 + lane < L ? list[t0 + i * 32 + lane] : 0xffffffffu;
#pragma unroll
                for (int i = 0; i < kLongSteps; ++i) pb[i] = p[i] != 0xffffffffu ? coords[p[i]] : make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < kLongSteps; ++i) {
                    const bool ok = p[i] != 0xffffffffu && ref_within(pa.x, pa.y, pb[i].x, pb[i].y, R2, hu);
                    const uint32_t bal = __ballot_sync(0xffffffffu, ok);
                    if (MODE != J_COUNT && ok) nb[base + k + __popc(bal & lt)] = ids ? ids[p[i]] : p[i];
                    k += __popc(bal);
                }
            }
            if (lane == 0) {
                nb_cnt[a] = k;
                if (MODE == J_SINGLE) nb_beg[a] = base;
            }
            found += k;
            continue;
        }
        const uint64_t at = (i - AL) * per + lane;
        const bool in = lane < per && at < A;
        uint32_t a = 0, L = 0;
        float xa = 0.f, ya = 0.f, R2 = 0.f, hu = 0.f;
        uint64_t from = 0, beg = 0;
        if (in) {
            const uint4 an = act[at];
            L = an.y;
            from = (uint64_t)an.w << 32 | an.z;
            a = ids ? ids[an.x] : an.x;
            const float2 pa = coords[an.x];
            xa = pa.x;
            ya = pa.y;
            const JobGrid& g = grids[fjob ? fjob[sfeat[an.x]] : 0u];
            R2 = g.R2;
            hu = g.R2hu;
            if (MODE == J_FILL) beg = nb_beg[a];
        }
        const uint32_t incl = warp_incl_scan(L), excl = incl - L;
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        from -= excl;   // pair t of the tile is target from_j + t, j its anchor's lane
        unsigned long long base = 0;
        if (MODE == J_SINGLE && lane == 0 && tot) base = atomicAdd(&ctrl->nb_used.v, (unsigned long long)tot);
        if (MODE == J_SINGLE) base = __shfl_sync(0xffffffffu, base, 0);
        uint32_t hits = 0, before = 0, mine = 0;   // the tile's so far; those before this lane's anchor; this anchor's
        for (uint32_t t0 = 0; t0 < tot; t0 += 32) {
            const uint32_t t = t0 + lane;
            int j = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t ev = __shfl_sync(0xffffffffu, excl, j + step);
                if (ev <= t) j += step;
            }
            const uint64_t from_j = __shfl_sync(0xffffffffu, from, j);
            const float xj = __shfl_sync(0xffffffffu, xa, j), yj = __shfl_sync(0xffffffffu, ya, j);
            // one job: one threshold; several: the anchor's own
            const float R2j = fjob ? __shfl_sync(0xffffffffu, R2, j) : __shfl_sync(0xffffffffu, R2, 0);
            const float huj = fjob ? __shfl_sync(0xffffffffu, hu, j) : __shfl_sync(0xffffffffu, hu, 0);
            bool ok = false;
            uint32_t p = 0;
            if (t < tot) {
                p = targets[from_j + t];
                const float2 pb = coords[p];
                ok = ref_within(xj, yj, pb.x, pb.y, R2j, huj);
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, ok);
            // lanes of this step before and in this lane's own slice
            const uint32_t r0 = excl <= t0 ? 0u : excl - t0 < 32 ? excl - t0 : 32u;
            const uint32_t r1 = incl <= t0 ? 0u : incl - t0 < 32 ? incl - t0 : 32u;
            const uint32_t m0 = r0 == 32 ? 0xffffffffu : (1u << r0) - 1u, m1 = r1 == 32 ? 0xffffffffu : (1u << r1) - 1u;
            if (MODE == J_FILL) {
                // compact layout: the pair's place in its own anchor's list
                const uint64_t beg_j = __shfl_sync(0xffffffffu, beg, j);
                const uint32_t mine_j = __shfl_sync(0xffffffffu, mine, j);
                const uint32_t own_j = __shfl_sync(0xffffffffu, m1 & ~m0, j);
                if (ok) nb[beg_j + mine_j + __popc(bal & own_j & lt)] = ids ? ids[p] : p;
            }
            if (MODE == J_SINGLE && ok) nb[base + hits + __popc(bal & lt)] = ids ? ids[p] : p;
            before += __popc(bal & m0);
            mine += __popc(bal & m1 & ~m0);
            hits += __popc(bal);
        }
        if (in) {
            nb_cnt[a] = mine;
            if (MODE == J_SINGLE) nb_beg[a] = base + before;
        }
        found += hits;
    }
    // the list total, added to one of kEntrySlots counters on separate lines by each warp
    if (MODE == J_SINGLE && lane == 0 && found) atomicAdd(total + (warp % kEntrySlots) * kEntryStride, found);
}

// `anchors`: as many as there are (and `longs` of them with long lists), or bounds.
void run_join(Batch& b, int mode, uint64_t anchors, uint64_t longs) {
    const int per = 32 / (b.join_group > 0 ? b.join_group : 1);
    const uint64_t warps = longs + (anchors - longs + per - 1) / per;
    const unsigned grid = (unsigned)std::min<uint64_t>((warps + 7) / 8, (uint64_t)b.sms * 6 * kJoinWaves);
    if (grid == 0) return;
    KScope ks(mode == J_SINGLE ? "join" : mode == J_COUNT ? "join_count" : "join_fill");
#define COLO_JOIN(MD)                                                                                            \
    k_join<MD><<<grid, 256, 0, b.s>>>(b.ctrl.get(), b.N, b.targets_cap, b.nb_cap, per, b.act.get(),              \
                                      b.gathered ? b.sid.get() : nullptr, b.sfeat.get(),                        \
                                      b.gathered ? b.sxy.get() : b.xy.get(), b.targets.get(),                   \
                                      b.J > 1 ? b.fjob.get() : nullptr, b.grids.get(), b.nb_beg.get(),          \
                                      b.nb_cnt.get(), b.nb.get(), b.dE.get())
    if (mode == J_SINGLE) COLO_JOIN(J_SINGLE);
    else if (mode == J_COUNT) COLO_JOIN(J_COUNT);
    else COLO_JOIN(J_FILL);
#undef COLO_JOIN
    COLO_LAUNCH_CHECK();
    count_launch();
}

__global__ void k_sqdist(const float* __restrict__ x1, const float* __restrict__ y1,
                         const float* __restrict__ x2, const float* __restrict__ y2, uint64_t n,
                         float* __restrict__ out, float R2, float hu, uint8_t* __restrict__ within) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = ref_sqdist(x1[i], y1[i], x2[i], y2[i]);
    if (within) within[i] = ref_within(x1[i], y1[i], x2[i], y2[i], R2, hu) ? 1 : 0;
}

}  // namespace

void join_queue(Batch& b) {
    b.join_queued = true;
    run_join(b, J_SINGLE, b.N, 0);
    b.E = UINT64_MAX;
}

// A point without targets keeps the zero count that the cell-key pass gave it; its list
// start is never read (every reader takes nb_cnt first).
void join_neighbors(Batch& b) {
    cudaStream_t s = b.s;
    const uint64_t A = b.active_anchors, AL = b.long_anchors, U = b.join_pairs;
    b.join_queued = false;
    // larger layouts are counted first and then compact
    const bool single = U <= b.single_cap();
    auto room = [&](uint64_t n) {
        b.nb_cap = n;
        Carver::place(b.mem_nb, s, [&](Carver& c) { c.add(b.nb, std::max<uint64_t>(n, 1)); });
    };
    if (single) {
        // total entries: summed by the join's warps and read at the mine's next wait
        if (U > b.nb_cap || !b.nb.get()) room(U);
        COLO_CUDA(cudaMemsetAsync(b.dE.get(), 0, kEntrySlots * kEntryStride * 8, s));
        COLO_CUDA(cudaMemsetAsync(&b.ctrl.get()->nb_used, 0, sizeof(LineCounter), s));
        run_join(b, J_SINGLE, A, AL);
        b.E = UINT64_MAX;
    } else {
        run_join(b, J_COUNT, A, AL);
        uint64_t E = 0;
        scan_u32_to_u64(b.nb_cnt.get(), b.nb_beg.get(), b.N, s, &E);
        room(E);
        run_join(b, J_FILL, A, AL);
        b.E = E;
    }
}

uint64_t sum_entries(const unsigned long long* dE) {
    uint64_t t = 0;
    for (int i = 0; i < kEntrySlots; ++i) t += dE[(size_t)i * kEntryStride];
    return t;
}

uint64_t neighbor_entries(Batch& b) {
    if (b.E == UINT64_MAX) {
        std::vector<unsigned long long> e(kEntrySlots * kEntryStride);
        COLO_CUDA(cudaMemcpyAsync(e.data(), b.dE.get(), e.size() * 8, cudaMemcpyDeviceToHost, b.s));
        stream_wait(b.s);
        b.E = sum_entries(e.data());
    }
    return b.E;
}

void eval_sqdist(const float* x1, const float* y1, const float* x2, const float* y2, uint64_t n,
                 float* out, cudaStream_t s, float R2, uint8_t* within) {
    if (n == 0) return;
    float hu = (std::nextafter(R2, INFINITY) - R2) * 0.5f;
    k_sqdist<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x1, y1, x2, y2, n, out, R2, hu, within);
    COLO_LAUNCH_CHECK();
    count_launch();
}

}  // namespace colo
