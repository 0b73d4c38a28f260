// colo_batch.h -- device state of one mining batch and the stage launchers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "colo_internal.h"

namespace colo {

// Queues a copy of host bytes through the context's page-locked staging (no wait; colo_mine.cpp).
void staged_upload(colo_ctx* ctx, cudaStream_t s, void* dst, const void* src, size_t bytes);
// Device memory that buffers may take now: free, or idle in the pool (colo_mine.cpp).
uint64_t device_room(const colo_ctx* ctx);
// A buffer of this size takes no more than half of that, or none that the pool does not hold already.
bool leaves_half(const colo_ctx* ctx, uint64_t bytes);
// Notes a block that the mine holds from start to end (the pool's headroom leaves it out).
void note_block(colo_ctx* ctx, uint64_t bytes);

// Host description of one job inside a batch.
struct JobHost {
    JobGrid grid;
    uint64_t p0 = 0, np = 0;     // point range
};

// A counter that many warps add to at once, on a 128-byte line of its own: atomics on one
// address are taken one after another, those on different lines side by side.
struct alignas(128) LineCounter {
    unsigned long long v;
};

// Totals of a batch on the device: cleared before bucketing, filled by its
// kernels, and read back once (settle).  dcnt, frun and ub2 follow it directly.
struct alignas(128) BatchCtrl {
    DevFlags flags;
    uint32_t M, Rn;              // occupied cells, runs
    uint32_t keys_done;          // blocks of the cell-key pass that have added their histograms
    LineCounter nlistq;          // cells queued for a neighbourhood list
    LineCounter nquadq;          // cells with a quad of quad_min features or more
    LineCounter npairq;          // with pairq: cells with two features or more in their 3x3 block
    // neighbourhood lists: target points, runs, anchors with short and with long lists, and the
    // pair evaluations (= room that the single-pass join may need)
    LineCounter targets, list_runs, anchors, long_anchors, pairs;
    LineCounter nb_used;         // room taken by the single-pass join's tiles
};

// Largest single-pass neighbour layout (entries): 4 GiB, and a 64th of the device.
constexpr uint64_t kSinglePassCap = 1ull << 30;

struct Batch {
    colo_ctx* ctx = nullptr;
    cudaStream_t s = 0;
    int sms = 148;
    // sizes
    uint64_t N = 0;              // points
    uint32_t F = 0;              // features (global)
    uint32_t J = 0;              // jobs
    uint32_t W = 1;              // mask words per cell (max local feature count / 32)
    uint32_t Fmax_local = 0;
    uint64_t M = 0;              // occupied cells (known after settle, or earlier when not bounded)
    uint64_t Rn = 0;             // (cell, feature) runs (the same)
    uint64_t key_bits = 1;
    // Sizes that bucketing finds are kept on the device, and arrays over cells, runs, list
    // entries and neighbours are laid out for an upper bound (capM, capR, targets_cap, nb_cap), so
    // that everything up to the pairs' bounds is queued without a host wait.  Batches whose
    // bounds are too large a reservation wait for the sizes instead (bounded = false).  `exact`
    // asks for that, and for heads that are counted first: the second attempt of a call whose
    // arrays did not all fit the device (fit_device).
    bool bounded = true, exact = false;
    uint64_t reserved_bytes = 0;   // of the arrays laid out for more than the batch turns out to need
    uint64_t capM = 0, capR = 0;
    uint64_t device_bytes = 0;   // the device's memory, as the layouts' rules see it
    // the largest single-pass neighbour layout (entries)
    uint64_t single_cap() const { return device_bytes / 256 < kSinglePassCap ? device_bytes / 256 : kSinglePassCap; }
    // host copies of small arrays
    std::vector<JobHost> jobs;
    std::vector<uint32_t> h_fstart, h_fcount, h_fjob;
    std::vector<uint64_t> h_job_off;    // pairs' bounds of job j start at h_job_off[j] (J + 1 entries)
    std::vector<uint32_t> h_frun_off;   // prefix of the number of runs (occupied cells) per feature
    // one allocation: feature and job tables (uploaded with one copy), then the cleared words:
    // the totals with the per-feature counts and the pairs' bounds, and the kernels' counters
    DevBuf<unsigned char> mem0;
    Span<uint32_t> fstart, fcount, fjob;
    Span<JobGrid> grids;
    Span<uint64_t> job_off;
    Span<BatchCtrl> ctrl;        // followed by dcnt[F], frun[F], ub2[job_off[J]]
    uint64_t ctrl_bytes = 0;     // of all four
    Span<unsigned long long> dE; // neighbour entries, spread over counters
    Span<unsigned long long> hist, head_status, sort_status;
    Span<uint32_t> tickets;      // one per digit pass, then the head kernel's
    RadixPlan plan{};
    bool sort_shared = false;    // one pass's look-back words, cleared per pass
    uint32_t* dcnt() const { return reinterpret_cast<uint32_t*>(ctrl.get() + 1); }
    uint32_t* frun() const { return dcnt() + F; }
    uint32_t* ub2() const { return frun() + F; }
    DevFlags* flags() const { return &ctrl.get()->flags; }
    // points (by id; the jobs' own coordinates are in their grids)
    DevBuf<unsigned char> mem_points, mem_heads, mem_cells, mem_lists, mem_act, mem_nb;
    Span<float2> xy;             // coordinates by id, packed (built by the cell-key pass)
    // bucketed (sorted by cell key, then id)
    Span<uint32_t> sid, sfeat, scell;     // sfeat for several jobs, scell (cell of each sorted point) only when keep_scell
    Span<float2> sxy;                     // coordinates in cell-sorted order, where gathered
    bool gathered = false;                // lists and anchors name points by sorted position, else by id
    bool keep_scell = false;              // colo_stage_cells reports each point's cell
    // cells
    Span<uint64_t> ckey;
    Span<uint32_t> crun, cjob;            // crun with an end entry
    uint64_t h2d_points = 0;     // bytes of point data copied to the device for this batch
    uint64_t rows = 0;           // grid rows of all jobs (row table size - 1)
    bool row_table = false;
    Span<uint32_t> rowstart;     // per grid row: first occupied cell at or after the row (unless too large)
    Span<uint4> nbrs;            // per cell: its occupied neighbours, stencil columns and quads (k_neighbours)
    Span<uint32_t> cmask;
    // feature mask of a cell's geometric 3x3 block (with pairq: of its cells and of quadq's only)
    Span<uint32_t> nbmask;
    // the cells with two features or more there: one job of kPairQueuePoints points or more
    bool pair_queue = false;
    Span<uint32_t> pairq;
    Span<uint32_t> listq;        // cells whose 3x3 block has a feature above their lowest own one
    // per cell of quadq: masks of the 4 quads containing it ([M][4][W], other cells' rows unwritten)
    Span<uint32_t> qmask;
    // the cells with a quad of at least quad_min features: no other cell is in a candidate's U_c
    // (a candidate of three or more members needs a quad that covers three)
    Span<uint32_t> quadq;
    uint32_t quad_min = 3;
    uint64_t quad_cells = 0;     // their number (known after settle)
    // driver lists: for global feature f, the cells of quadq whose 3x3 block holds f
    // (nbmask bit), dlist[doff[f] .. doff[f+1]), in no particular order; the
    // level filters test exactly these cells for the candidates f drives
    DevBuf<uint32_t> dlist;
    DevBuf<uint64_t> doff;
    std::vector<uint64_t> h_dcnt;    // cells per feature's list (every feature)
    std::vector<uint64_t> h_doff;    // offsets of the lists filled (features in dlist_have; others empty)
    std::vector<uint8_t> dlist_have; // features whose lists are filled (by the level filters, on demand)
    // runs: run r's points are sorted positions rstart[r] .. rstart[r+1] (rstart has an end entry)
    Span<uint32_t> rfeat, rstart, rcell;
    // neighbourhood lists: for each cell with targets, the points of its adjacent
    // cells' runs above the cell's lowest own feature, ordered by (feature, cell, id);
    // the lists are in no particular order
    Span<uint32_t> targets;
    uint64_t targets_cap = 0, nrl_total = 0;   // nrl_total: runs in the lists
    // scratch of the list kernel, per own run of those cells: first target with a higher
    // feature (absolute index), and the targets from there to the list's end
    Span<uint64_t> run_sfx;
    Span<uint32_t> run_L;
    // the join's anchors (points of runs with targets), in no particular order: point, number
    // of targets, first target (low, high word); anchors of at most
    // kLongList targets from the front, the others from the back
    Span<uint4> act;
    // neighbour lists N+(a) = nb[nb_beg[a] .. nb_beg[a] + nb_cnt[a]), each in
    // (feature, neighbour cell, id) order; nb_beg[a] is set only where nb_cnt[a] > 0
    Span<uint64_t> nb_beg;
    Span<uint32_t> nb_cnt, nb;
    uint64_t E = 0;              // neighbour entries (UINT64_MAX: still on the device in dE)
    uint64_t nb_cap = 0;         // allocated entries (upper bound in single-pass mode)
    uint64_t join_pairs = 0;     // pair distance evaluations
    uint64_t active_anchors = 0; // anchors whose cell has higher-feature neighbours
    uint64_t long_anchors = 0;   // of them, with long lists
    bool lists_built = false, join_queued = false;
    int join_group = 1;          // lanes per anchor in the join (autotuned): a warp takes 32 / join_group anchors
    int filter_unit = 32;        // candidates per warp unit in the level filter (autotuned: 8, 16, 32)
    int level_block = 256;       // threads per block of the level kernels (autotuned: 64, 128, 256)
    int level_queue = 0;         // 1: level count/fill kernels as a persistent work queue (autotuned)
    uint32_t test_spin = 0;      // tests only: the sort's look-back gives up after this many polls
    uint64_t filter_items = 0;   // (driver cell, candidate) items of the level filters
};

// colo_bucket.cu
void bucket_layout(Batch& b, Carver& c); // the cleared words of mem0 that bucketing uses, after the upload
void bucket_points(Batch& b);            // cells, runs, masks, neighbours, runs per feature (launches; see bounded)
void build_neighborhoods(Batch& b);      // neighbourhood lists and anchors (launches)
// colo_join.cu
constexpr int kEntrySlots = 64, kEntryStride = 16;   // dE: counters on separate 128-byte lines
constexpr uint32_t kLongList = 64;                   // targets above which an anchor gets a warp to itself
void join_queue(Batch& b);               // single-pass join into nb_cap entries, skipped on the device when they
                                         // or the lists did not fit (bounded batches, before settle)
void join_neighbors(Batch& b);           // neighbour CSR (after settle)
uint64_t neighbor_entries(Batch& b);     // E (waits for the device sum once)
uint64_t sum_entries(const unsigned long long* dE);   // of a copy of dE
// Level-k candidates of every job from its prevalent (k-1)-patterns (km1
// features each, lexicographic), with each candidate's prefix pattern index;
// a null entry is a job with no next level.  colo_apriori.cu.
void apriori_device(cudaStream_t s, const std::vector<const std::vector<uint32_t>*>& prev, uint32_t km1,
                    std::vector<std::vector<uint32_t>>& out, std::vector<std::vector<uint32_t>>& parent);
// colo_filter.cu
// Driver lists: their sizes are counted by the quad masks' kernel; the lists
// themselves are filled by the level filters for the drivers of their
// candidates (a level whose drivers are not all filled yet fills the union of
// the old and new ones).
// Level-2 upper bounds of every pair of every job into the batch's ub2:
// ub2[job_off[j] + lf*Fj + lg] is the bound of feature lf's side of pair {lf, lg}
// (launch only).
void filter_pairs(Batch& b);
// Level-k upper bounds for host candidates cand[c*k + j] (global features) of
// jobs job[c]: d_ub[c*k + j] (zeroed by the caller).  d_stats (optional,
// zeroed, 2 per candidate): full quads and cells of U_c.
void filter_level(Batch& b, const uint32_t* h_cand, const uint32_t* h_job, uint64_t ncand, uint32_t k,
                  uint32_t* d_ub, unsigned long long* d_stats);

// colo_level.cu --------------------------------------------------------------
// One member of a candidate: its feature's first point id and instances, and where its
// participation bitmap starts (words from the candidate's bm_base).
struct alignas(16) MemberInfo {
    uint32_t start, n, off, feature;
};

// One candidate's view for the level kernels.  What a kernel needs first (the last member's
// id range, the threshold) is written out, so that it waits on one load.
struct CandDesc {
    const uint32_t* parent;      // column-major parent table (k-1 columns); nullptr: implicit (k=2)
    uint64_t prow;               // parent rows (k=2: anchors of member 0)
    uint64_t pstride;            // parent column stride (>= prow)
    const MemberInfo* mem;       // its k members
    uint32_t* chunk_rows;        // rows per chunk of 32 parent rows (count pass output)
    const uint64_t* offs;        // the level's scan of them from this candidate's first chunk on (fill pass input)
    uint32_t* out;               // column-major output table (k columns, rows = total)
    uint64_t out_rows;           // rows of the output table (column stride)
    uint64_t out_cap;            // capacity (single-pass mode; also its column stride)
    unsigned long long* rows;    // count pass: rows of this candidate (atomic sum)
    uint32_t* bitmap;            // the level's bitmap words; this candidate's members' start at
    uint64_t bm_base;            // bm_base + their off
    uint32_t last_start, last_end, last_off;   // the last member's point ids and bitmap offset
    float R2, R2hu;              // the job's threshold (JobGrid)
    uint32_t job;
    uint32_t k;
};

struct LevelWork {
    const CandDesc* cands;       // device array
    const uint64_t* chunk_off;   // device: prefix of 32-row chunks per candidate (ncand+1)
    uint64_t ncand;
    uint64_t nchunks;
    unsigned long long* items;   // optional: sum of candidate-slice lengths examined
    unsigned long long* chunk_status = nullptr;   // single pass: nchunks words, zeroed
    unsigned long long* ticket = nullptr;         // single pass: chunk ticket counter, zeroed
};

// The count pass's candidates in groups that share a parent table: group g is candidates
// gstart[g] .. gstart[g+1] (at most kGroupMax), neighbours in the candidate order, and its chunks
// of parent rows start at gchunk[g].
constexpr uint32_t kGroupMax = 32;
struct CountWork {
    const CandDesc* cands;       // device arrays
    const uint32_t* gstart;
    const uint64_t* gchunk;
    uint64_t ngroups;
    uint64_t nchunks;            // of all groups
    unsigned long long* items;   // optional: sum of candidate-slice lengths examined
    unsigned long long* ticket;  // chunk tickets of the persistent queue, zeroed
    uint64_t chunk0 = 0;         // gchunk[0]
    // non-null: candidates c whose bounds ub[c*k + j] do not all reach need[c*k + j] are passed over
    const uint32_t* ub = nullptr;
    const uint32_t* need = nullptr;
    // 1 << split_log warps share a chunk (count_split of nchunks; the chunk_rows are then cleared first)
    uint32_t split_log = 0;
};
uint32_t count_split(const Batch& b, uint64_t nchunks);

// count pass: rows per chunk + bitmaps; fill pass: rows; single pass: rows per
// chunk + bitmaps + rows at their count-and-fill positions (overflow recorded per
// candidate; a look-back that waits too long sets the batch's timeout flag).
void level_count(Batch& b, const CountWork& w, uint32_t k);
void level_fill(Batch& b, const LevelWork& w, uint32_t k);
void level_single(Batch& b, const LevelWork& w, uint32_t k, uint32_t* d_overflow);
// Participation statistics per candidate and member: [A, last, first, full]
// (A = set bits in [0, n-2]), added into d_stats, which must be zero.
void level_pi(Batch& b, const CandDesc* d_cands, uint64_t ncand, uint32_t k, uint64_t* d_stats);

// Rows row0 .. row0 + rows of a column-major table, row-major at word `at` of `out`.
struct TablePiece {
    const uint32_t* cols;
    uint64_t stride, row0, rows, at;
};
void table_rows(cudaStream_t s, const TablePiece* d_pieces, uint32_t n, uint32_t k, uint64_t most_words, uint32_t* out);

// Squared-distance evaluation of the reference expression for n pairs; with
// `within`, also the kernels' decision ref_within(...) for threshold R2.
void eval_sqdist(const float* x1, const float* y1, const float* x2, const float* y2, uint64_t n,
                 float* out, cudaStream_t s, float R2 = 0.0f, uint8_t* within = nullptr);

}  // namespace colo
