// colo_prims.cu -- device-wide scan and a stable LSD radix sort (hand-written,
// no library).  The reference uses thrust::exclusive_scan / sort_by_key
// (Codes/DeviceProcess.cu:342-344); these are their replacements.
#include "colo_device.cuh"
#include "colo_internal.h"

namespace colo {

thread_local uint64_t g_launches = 0;
thread_local KTimer* g_ktimer = nullptr;

namespace {

constexpr int kScanThreads = 256;
// Single-pass scan (decoupled look-back): a block takes the next tile number
// from a counter, sums its 4096 items, publishes the sum, and warp 0 reads its
// predecessors' published words 32 at a time, back to the nearest inclusive
// prefix; the tile then publishes its own inclusive prefix and writes its
// items.  Tiles are numbered in the order blocks start, so a tile only waits
// on tiles whose blocks are already running.  The wait is bounded: past the
// limit the tile sums its predecessors' items itself (slow, but exact), so a
// scan never yields a wrong offset.  A warp reads its segment 32 consecutive
// items per round (coalesced loads and stores).
constexpr int kScan1Items = 16;
constexpr int kScan1Tile = kScanThreads * kScan1Items;
template <class Tin, class Tout>
__global__ void __launch_bounds__(kScanThreads, 5) k_scan_1p(const Tin* __restrict__ in, Tout* __restrict__ out,
                                                          uint64_t n, unsigned long long* __restrict__ status,
                                                          uint32_t* __restrict__ ticket, Tout* __restrict__ total) {
    __shared__ uint32_t s_tile;
    __shared__ unsigned long long s_prefix;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t seg = (uint64_t)tile * kScan1Tile + (uint64_t)w * (32 * kScan1Items);
    Tin v[kScan1Items];   // kept in the input type (half the registers for 32-bit counts)
    Tout sum = 0;
#pragma unroll
    for (int i = 0; i < kScan1Items; ++i) {
        const uint64_t p = seg + (uint64_t)i * 32 + lane;
        v[i] = p < n ? in[p] : Tin(0);
        sum += (Tout)v[i];
    }
    Tout tot;
    const Tout ex_thread = block_excl_scan<Tout>(sum, &tot);
    if (w == 0) {
        unsigned long long prefix;
        if (!warp_lookback(status, tile, (unsigned long long)tot, prefix)) {   // the predecessors' items, summed here
            unsigned long long add = 0;
            for (uint64_t p = lane; p < (uint64_t)tile * kScan1Tile; p += 32) add += (unsigned long long)(Tout)in[p];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
            prefix = add;
            lookback_publish(status, tile, prefix + (unsigned long long)tot);
        }
        if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    Tout carry = __shfl_sync(0xffffffffu, ex_thread, 0) + (Tout)s_prefix;
#pragma unroll
    for (int i = 0; i < kScan1Items; ++i) {
        const Tout x = (Tout)v[i];
        const Tout inc = warp_incl_scan(x);
        const uint64_t p = seg + (uint64_t)i * 32 + lane;
        if (p < n) out[p] = carry + inc - x;
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (total && threadIdx.x == 0 && (uint64_t)(tile + 1) * kScan1Tile >= n) *total = (Tout)s_prefix + tot;
}

template <class Tin, class Tout>
void scan_impl(const Tin* in, Tout* out, uint64_t n, cudaStream_t s, Tout* total_host, Tout* total_dev) {
    KScope ks("scan");
    const uint64_t tiles = n ? (n + kScan1Tile - 1) / kScan1Tile : 0;
    if (tiles >= (1ull << 32)) throw StatusError{COLO_ERR_CAPACITY, "scan supports < 2^32 tiles"};
    // status words, then the tile counter and the total: one clear
    DevBuf<unsigned long long> st;
    st.alloc(tiles + 2, s);
    st.zero(s);
    uint32_t* ticket = reinterpret_cast<uint32_t*>(st.get() + tiles);
    Tout* tot = reinterpret_cast<Tout*>(st.get() + tiles + 1);
    if (tiles) {
        k_scan_1p<Tin, Tout><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, st.get(), ticket, tot);
        COLO_LAUNCH_CHECK();
        count_launch();
    }
    if (total_dev) COLO_CUDA(cudaMemcpyAsync(total_dev, tot, sizeof(Tout), cudaMemcpyDeviceToDevice, s));
    if (total_host) {
        COLO_CUDA(cudaMemcpyAsync(total_host, tot, sizeof(Tout), cudaMemcpyDeviceToHost, s));
        stream_wait(s);
    }
}

// ---------------------------------------------------------------------------
// Radix sort
// ---------------------------------------------------------------------------

// Tile shape: 512 threads of 8 items (4096-key tiles) and four resident blocks
// per SM (32-bit keys: 32 registers, a few spilled; 4 x 43 KB of shared memory, of
// which 64-bit keys, 59 KB a block, leave three), three with
// digits of nine bits (55 KB; four measured the same and spill).  Ranking takes most
// of a pass: without any look-back a sort of random keys is a quarter faster, no more.
// 2048-key tiles of 256 threads (eight blocks an SM) and 8192-key tiles of 1024
// (two) take 8% longer, 256 threads of 16 items more than either.
constexpr int kSortThreads = 512, kSortRounds = 8, kSortTile = kSortThreads * kSortRounds;
constexpr int sort_blocks(int RB) { return RB == 8 ? 4 : 3; }

// Shared memory of one sort block (dynamic): the tile's keys and ids (bulk-copy
// targets, 16-byte aligned), each digit's global base, the per-warp digit
// counts and each digit's tile-local start.
template <class KT, int RB>
struct SortSmem {
    static constexpr int W = kSortThreads / 32, R = 1 << RB, tile = kSortTile;
    static constexpr size_t key_at = 0;
    static constexpr size_t val_at = key_at + (size_t)tile * sizeof(KT);
    static constexpr size_t base_at = val_at + (size_t)tile * sizeof(uint32_t);
    static constexpr size_t wh_at = base_at + (size_t)R * sizeof(unsigned long long);
    static constexpr size_t off_at = wh_at + (size_t)W * R * sizeof(uint16_t);
    static constexpr size_t bytes = off_at + (size_t)R * sizeof(uint32_t);
    static_assert(val_at % 16 == 0 && base_at % 8 == 0, "alignment");
};


// ---------------------------------------------------------------------------
// One-sweep LSD radix sort: the digit histograms of every pass come with the
// keys (k_cell_keys), then one kernel per pass.  A block takes the next tile number
// from a counter, ranks its keys stably, publishes its per-digit counts, and
// looks back over the preceding tiles' published counts (a tile that has
// finished its own look-back publishes its inclusive prefix, which ends the
// walk) to place its keys.  Tiles are numbered in the order blocks start, so
// a block only waits on tiles of blocks already running.  Every wait is
// bounded: past the limit the block sets *err, uses what it has and finishes
// (the host reports COLO_ERR_TIMEOUT).  The key's bits are split evenly over
// the fewest passes of at most 8 bits (narrower digits leave more keys per digit in
// a tile, so the scatter writes longer runs), or of at most 9 where that saves a
// pass: 25 to 27 bits take 80 us in 4 passes for 1M points, 68 in 3; 33 to 36 bits of 2M
// points 155 us in 5, 139 in 4; where both take as many (20M points, 32 bits) wide digits
// gain nothing.
//
// A key's peers in its warp (the lanes with its digit) come from one ballot per bit:
// match_any over the digit took 8% longer (20M points: 688 -> 636 us a sort).
// ---------------------------------------------------------------------------

constexpr unsigned long long kFlagA = 1ull << 62;   // tile count published
constexpr unsigned long long kFlagP = 2ull << 62;   // inclusive prefix published
constexpr unsigned long long kValMask = (1ull << 62) - 1;
constexpr uint32_t kSpinLimit = 1u << 22;

// Bulk (TMA engine) copy of a full tile from global to shared memory,
// completing on an mbarrier: one thread issues it, every thread waits.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// dst and src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Waits for phase `parity` of the barrier at most `limit` polls; false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
    for (uint32_t it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// A full tile's keys and ids come into shared memory by one bulk copy each
// (bulk != 0: the host checked that both arrays are 16-byte aligned); the
// ranking reads them from there, and the same buffers then stage the tile
// in digit order.  vin == nullptr: the ids are the input positions (the first
// pass over keys in id order), generated rather than read.
template <class KT, int RB>
__global__ void __launch_bounds__(kSortThreads, sort_blocks(RB)) k_onesweep(
    const KT* __restrict__ kin, const uint32_t* __restrict__ vin, KT* __restrict__ kout, uint32_t* __restrict__ vout,
    uint64_t n, int shift, uint32_t dmask, const unsigned long long* __restrict__ gofs,
    unsigned long long* __restrict__ status, uint32_t* __restrict__ ticket, uint32_t* __restrict__ err, int bulk,
    uint32_t spin_limit, int withhold, int pass) {
    constexpr int R = 1 << RB;
    constexpr int kSortWarps = kSortThreads / 32;
    // digits per thread in the look-back (1 or 2); with more threads than digits the
    // first R threads take one each
    constexpr int D = R >= kSortThreads ? R / kSortThreads : 1;
    static_assert(R < kSortThreads || D * kSortThreads == R, "digit count");
    using SM = SortSmem<KT, RB>;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    KT* s_key = reinterpret_cast<KT*>(s_dyn + SM::key_at);
    uint32_t* s_val = reinterpret_cast<uint32_t*>(s_dyn + SM::val_at);
    unsigned long long* s_base = reinterpret_cast<unsigned long long*>(s_dyn + SM::base_at);  // digit's global base
    uint16_t (*wh)[R] = reinterpret_cast<uint16_t (*)[R]>(s_dyn + SM::wh_at);                 // per-warp digit counts
    uint32_t* s_off = reinterpret_cast<uint32_t*>(s_dyn + SM::off_at);                       // digit's tile-local start
    const bool owner = (int)threadIdx.x * D < R;   // this thread owns digits in the look-back
    __shared__ alignas(8) uint64_t s_bar;
    __shared__ uint32_t s_tile, s_skip;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        // an earlier pass that timed out left keys whose digit counts no longer match the
        // histograms, so its positions could leave the array: every later pass writes nothing
        // (the word holds the failed pass + 1; the previous launch has finished, so every
        // block of this pass reads the same value)
        const uint32_t e = *(volatile const uint32_t*)err;
        s_skip = e != 0u && e < (uint32_t)pass + 1u;
        s_tile = atomicAdd(ticket, 1u);
        if (bulk && !s_skip) mbar_init(&s_bar, 1);
    }
    for (int i = threadIdx.x; i < kSortWarps * R / 2; i += blockDim.x) reinterpret_cast<uint32_t*>(wh)[i] = 0;
    __syncthreads();
    if (s_skip) return;
    const uint32_t tile = s_tile;
    const uint64_t tile0 = (uint64_t)tile * kSortTile;
    const uint64_t base = tile0 + (uint64_t)w * (32 * kSortRounds);
    const bool staged = bulk && n - tile0 >= (uint64_t)kSortTile;   // full tiles only (uniform in the block)
    if (staged) {
        if (threadIdx.x == 0) {
            mbar_expect_tx(&s_bar, kSortTile * (uint32_t)(sizeof(KT) + (vin ? sizeof(uint32_t) : 0)));
            bulk_g2s(s_key, kin + tile0, kSortTile * (uint32_t)sizeof(KT), &s_bar);
            if (vin) bulk_g2s(s_val, vin + tile0, kSortTile * (uint32_t)sizeof(uint32_t), &s_bar);
        }
        const bool done = mbar_wait(&s_bar, 0, kSpinLimit);
        if (!__syncthreads_and(done ? 1 : 0)) {
            // the copy did not complete for every thread in time: report it, give it one
            // more bounded wait (it writes into this block's shared memory) and leave, the
            // whole block together; the host turns err into a timeout
            if (threadIdx.x == 0) atomicCAS(err, 0u, (uint32_t)pass + 1u);
            mbar_wait(&s_bar, 0, kSpinLimit);
            return;
        }
    }
    KT key[kSortRounds];
    uint32_t val[kSortRounds];
    uint32_t rank[kSortRounds];
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const uint64_t i = base + (uint64_t)r * 32 + lane;
        const bool ok = i < n;
        const uint32_t li = (uint32_t)(i - tile0);
        key[r] = ok ? (staged ? s_key[li] : kin[i]) : 0;
        val[r] = !ok ? 0u : !vin ? (uint32_t)i : staged ? s_val[li] : vin[i];
        const uint32_t d = ok ? ((uint32_t)(key[r] >> shift) & dmask) : 0xFFFFu;
        uint32_t peers = __ballot_sync(0xffffffffu, ok);
        if (!ok) peers = ~peers;
        for (uint32_t bit = 1; bit <= dmask; bit <<= 1) {
            const uint32_t v = __ballot_sync(0xffffffffu, d & bit);
            peers &= d & bit ? v : ~v;
        }
        const int leader = __ffs(peers) - 1;
        uint32_t old = 0;
        if (ok && lane == leader) {
            old = wh[w][d];
            wh[w][d] = (uint16_t)(old + __popc(peers));
        }
        old = __shfl_sync(0xffffffffu, old, leader);
        rank[r] = ok ? old + __popc(peers & lt) : 0xFFFFFFFFu;
        __syncwarp();
    }
    __syncthreads();
    {
        // thread t owns digits t*D .. t*D + D-1
        uint32_t cnt[D], sum = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const int d = threadIdx.x * D + i;
            uint32_t c = 0;
            if (owner)
                for (int ww = 0; ww < kSortWarps; ++ww) {
                    const uint32_t t = wh[ww][d];
                    wh[ww][d] = (uint16_t)c;
                    c += t;
                }
            cnt[i] = c;
            sum += c;
        }
        uint32_t tot;
        uint32_t ex = block_excl_scan<uint32_t>(sum, &tot);
        // status words and look-back for the dmask + 1 digits in use only (a tile's words
        // are R apart: packing them closer measured slower)
        const uint32_t nd = dmask + 1;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const int d = threadIdx.x * D + i;
            if (!owner) break;
            s_off[d] = ex;
            ex += cnt[i];
            if ((uint32_t)d >= nd) continue;
            volatile unsigned long long* st = status + (uint64_t)tile * R + d;
            unsigned long long prefix = 0;
            if (tile == 0) {
                if (!withhold) *st = kFlagP | cnt[i];   // withhold: a test of the bounded wait below
            } else {
                *st = kFlagA | cnt[i];
                uint32_t spins = 0;
                for (int64_t t = (int64_t)tile - 1; t >= 0;) {
                    const unsigned long long v = *(volatile const unsigned long long*)(status + (uint64_t)t * R + d);
                    const unsigned long long flag = v & ~kValMask;
                    if (flag == 0) {
                        if (++spins > spin_limit) {   // give up: positions from a partial prefix
                            atomicCAS(err, 0u, (uint32_t)pass + 1u);   // stay below the true ones
                            break;
                        }
                        __nanosleep(64);
                        continue;
                    }
                    prefix += v & kValMask;
                    if (flag == kFlagP) break;
                    --t;
                }
                *st = kFlagP | (prefix + cnt[i]);
            }
            s_base[d] = gofs[d] + prefix;
        }
    }
    __syncthreads();
    // stage the tile in digit order, then write it out: consecutive threads
    // write consecutive positions of one digit's range
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        if (rank[r] == 0xFFFFFFFFu) continue;
        const uint32_t d = (uint32_t)(key[r] >> shift) & dmask;
        const uint32_t lp = s_off[d] + wh[w][d] + rank[r];
        s_key[lp] = key[r];
        s_val[lp] = val[r];
    }
    __syncthreads();
    const uint32_t valid = (uint32_t)(n - tile0 < (uint64_t)kSortTile ? n - tile0 : (uint64_t)kSortTile);
    for (uint32_t i = threadIdx.x; i < valid; i += kSortThreads) {
        const KT k = s_key[i];
        const uint32_t d = (uint32_t)(k >> shift) & dmask;
        const uint64_t pos = s_base[d] + (i - s_off[d]);
        kout[pos] = k;
        vout[pos] = s_val[i];
    }
}

}  // namespace

uint64_t scan_words(uint64_t n) { return (n + kScan1Tile - 1) / kScan1Tile + 1; }

void scan_u32_to_u64(const uint32_t* in, uint64_t* out, uint64_t n, unsigned long long* words, cudaStream_t s) {
    const uint64_t tiles = (n + kScan1Tile - 1) / kScan1Tile;
    if (tiles >= (1ull << 31)) throw StatusError{COLO_ERR_CAPACITY, "scan supports < 2^31 tiles"};
    if (!tiles) return;
    KScope ks("scan");
    k_scan_1p<uint32_t, uint64_t><<<(unsigned)tiles, kScanThreads, 0, s>>>(
        in, out, n, words, reinterpret_cast<uint32_t*>(words + tiles), nullptr);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void scan_u32_to_u64(const uint32_t* in, uint64_t* out, uint64_t n, cudaStream_t s,
                     uint64_t* total_host, uint64_t* total_dev) {
    scan_impl<uint32_t, uint64_t>(in, out, n, s, total_host, total_dev);
}

void scan_u64_to_u64(const uint64_t* in, uint64_t* out, uint64_t n, cudaStream_t s,
                     uint64_t* total_host, uint64_t* total_dev) {
    scan_impl<uint64_t, uint64_t>(in, out, n, s, total_host, total_dev);
}

namespace {

// Digit width the passes are compiled for (the first pass is the widest).
int plan_bits(const RadixPlan& plan) { return plan.n && plan.width[0] > 8 ? 9 : 8; }

template <class KT, int RB>
void radix_sort_impl(RadixBufs<KT>& bufs, uint64_t n, const RadixPlan& plan, cudaStream_t s,
                     const unsigned long long* hist, unsigned long long* status, bool shared, uint32_t* tickets,
                     uint32_t* err, uint32_t test_spin) {
    if (n >= (1ull << 32)) throw StatusError{COLO_ERR_CAPACITY, "radix sort supports < 2^32 items"};
    using SM = SortSmem<KT, RB>;
    constexpr int R = 1 << RB;
    const uint32_t ntiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
    // several blocks per SM: ask for the largest shared-memory carveout
    COLO_CUDA(cudaFuncSetAttribute((const void*)k_onesweep<KT, RB>,
                                   cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    COLO_CUDA(cudaFuncSetAttribute((const void*)k_onesweep<KT, RB>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM::bytes));
    for (int p = 0; p < plan.n; ++p) {
        KScope ks("radix_sort");   // one timed launch per digit pass
        const uint32_t dm = (1u << plan.width[p]) - 1u;
        // shared words: those of the digits in use are cleared for every pass (a pitched clear:
        // a tile's words stay R apart, which spreads the polled lines over L2)
        unsigned long long* st = status + (shared ? 0 : (uint64_t)p * ntiles * R);
        if (shared)
            COLO_CUDA(cudaMemset2DAsync(st, R * 8, 0, ((size_t)1 << plan.width[p]) * 8, ntiles, s));
        const int bulk = ((uintptr_t)bufs.ka % 16 == 0 && (uintptr_t)bufs.va % 16 == 0) ? 1 : 0;
        const uint32_t* vin = p == 0 ? nullptr : bufs.va;   // the first pass makes the ids (no read)
        k_onesweep<KT, RB><<<ntiles, kSortThreads, SM::bytes, s>>>(
            bufs.ka, vin, bufs.kb, bufs.vb, n, plan.shift[p], dm, hist + p * kRadixDigits, st, tickets + p, err, bulk,
            test_spin ? test_spin : kSpinLimit, test_spin && p == 0 ? 1 : 0, p);
        COLO_LAUNCH_CHECK();
        count_launch();
        std::swap(bufs.ka, bufs.kb);
        std::swap(bufs.va, bufs.vb);
    }
}

}  // namespace

uint64_t radix_status_words(uint64_t n, const RadixPlan& plan) {
    return (n + kSortTile - 1) / kSortTile << plan_bits(plan);
}

RadixPlan radix_plan(int bits) {
    // fewest passes of at most 9 bits, widths as even as possible (25 bits: 9 + 8 + 8)
    RadixPlan plan{};
    if (bits <= 0) return plan;
    plan.n = (bits + kRadixBits - 1) / kRadixBits;
    for (int p = 0, sh = 0; p < plan.n; ++p) {
        plan.width[p] = bits / plan.n + (p < bits % plan.n ? 1 : 0);
        plan.shift[p] = sh;
        sh += plan.width[p];
    }
    return plan;
}

void radix_sort(RadixBufs<uint32_t>& bufs, uint64_t n, const RadixPlan& plan, cudaStream_t s,
                const unsigned long long* hist, unsigned long long* status, bool shared, uint32_t* tickets,
                uint32_t* err, uint32_t test_spin) {
    (plan_bits(plan) == 9 ? radix_sort_impl<uint32_t, 9> : radix_sort_impl<uint32_t, 8>)(
        bufs, n, plan, s, hist, status, shared, tickets, err, test_spin);
}

void radix_sort(RadixBufs<uint64_t>& bufs, uint64_t n, const RadixPlan& plan, cudaStream_t s,
                const unsigned long long* hist, unsigned long long* status, bool shared, uint32_t* tickets,
                uint32_t* err, uint32_t test_spin) {
    (plan_bits(plan) == 9 ? radix_sort_impl<uint64_t, 9> : radix_sort_impl<uint64_t, 8>)(
        bufs, n, plan, s, hist, status, shared, tickets, err, test_spin);
}

}  // namespace colo
