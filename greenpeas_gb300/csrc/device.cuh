// device.cuh -- structures shared by the host driver and the sm_103a kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gpc {

// Device error bits (one word per pipeline run).
enum : uint32_t {
  DEV_ERR_TIMEOUT = 1u,    // a bounded wait (mbarrier or look-back) gave up
  DEV_ERR_COLLISION = 2u,  // equal 128-bit keys, different symptoms
  DEV_FLAG_MIXED = 4u,     // equal sort keys, different 128-bit keys: re-sort on 64 bits, then on all 128
  DEV_FLAG_TG_OVF = 8u,    // target buffer too small: grow and re-run the merge
  DEV_FLAG_BIG_BUCKET = 16u,  // a bucket exceeds the in-CTA capacity: use the global sort
  DEV_FLAG_LONG = 32u,        // a symptom has more targets than the target-list stride: widen it
  DEV_ERR_NOISE = 128u,       // a noise-tensor entry is outside its channel's range
};

// One circuit as the kernels see it.  All arrays are device pointers.
struct CircuitDev {
  const uint64_t *ops;        // tape, epoch-major, [slot][qubit] inside an epoch
  const uint32_t *ep_opoff;   // [n_epochs]
  const uint32_t *ep_k;       // [n_epochs]
  const uint32_t *ep_ptoff;   // [n_epochs + 1]
  const uint32_t *ep_chunk;   // [n_epochs] copy chunk of each epoch
  const uint32_t *ch_off;     // [n_chunks] first op of each chunk
  const uint32_t *ch_bytes;   // [n_chunks]
  const uint32_t *inj_lo;     // [w] first epoch injecting into word j (0xFFFFFFFF: none)
  const uint32_t *inj_hi;     // [w] last epoch injecting into word j
  ulonglong2 *snap;           // [w][npoints] (X row, Z row) at each point; stored where either is non-zero (nzm)
  uint2 *band;                // [w] point range covered by the walk of word j
  unsigned long long *nzm;    // [npoints][mw] (zeroed) bit j: word j's rows at the point are non-zero
  const uint64_t *rec;        // [R] noise records
  const double *rec_p;        // [R]
  const uint32_t *rec_moff;   // [R + 1]
  uint64_t *mdesc;            // [M] mechanism descriptors (global path)
  double *mp;                 // [M] mechanism probabilities (global path)
  uint32_t nq, qpad, n_epochs, w;
  uint32_t npoints, M, R;
  uint32_t tcap;              // most targets of a listed symptom (0: no target lists, merge from snapshots)
  uint32_t n_chunks, chunk_cap;
  uint32_t mbase;             // first mechanism of this circuit in the batch-wide arrays
  uint32_t bbase, bbits;      // first bucket of this circuit, log2 of its bucket count
  uint32_t mw;                // 64-bit mask words per point: ceil(w / 64)
};

// *p += v as a reduction that returns nothing (the thread does not wait for
// the L2 round trip of an atomic whose old value it would not use).
__device__ __forceinline__ void red_add(uint32_t *p, uint32_t v) {
  asm volatile("red.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Index of the circuit holding item x: the last c with base[c] <= x (base[0 .. n - 1]).
__device__ __forceinline__ uint32_t find_circuit(const uint32_t *base, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (base[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

constexpr int SORT_THREADS = 256;
constexpr int SORT_IPT = 8;
constexpr int SORT_TILE = SORT_THREADS * SORT_IPT;
constexpr int RADIX_BITS = 8;
constexpr int RADIX = 1 << RADIX_BITS;
constexpr int MERGE_THREADS = 256;
constexpr uint32_t SLOT_CAP = 256;  // slots of one bucket in the compile pipeline
constexpr uint32_t WARP_CAP = 128;  // bucket items of a warp's own shared memory
constexpr uint32_t SCAN_TILE = 1024;    // bucket aggregates one scan block covers
constexpr uint32_t SCAN_THREADS = 256;  // threads of a scan block (4 aggregates each)

inline uint32_t sort_tiles(uint32_t n) { return (n + SORT_TILE - 1) / SORT_TILE; }
inline uint32_t merge_tiles(uint32_t n) { return (n + MERGE_THREADS - 1) / MERGE_THREADS; }

// ---- launch wrappers (defined in the .cu files) ----------------------------
struct WalkLaunch {
  const CircuitDev *circs;  // device array
  const uint2 *items;       // device array of (circuit, first word of the CTA)
  uint32_t n_items;
  uint32_t threads, qpt, qpad;
  uint32_t chunk_cap;       // bytes of each of the two chunk buffers
  uint32_t max_epochs, max_chunks;  // largest tables of the launch (staged in shared memory if they fit)
  uint32_t words;           // detector words per CTA (1, or 2 with 1 or 2 qubits per thread)
  uint32_t *err;
  // Persistent launch (null: one CTA per item): a zeroed counter from which
  // resident CTAs take items until none are left.  Circuits of any slot count
  // up to qpad share the launch; the items should come longest first.
  uint32_t *queue;
};
cudaError_t launch_walk(const WalkLaunch &L, cudaStream_t s);
cudaError_t walk_set_smem_limit();  // call once per device before launching walks

// ---- segmented walk (one circuit) -------------------------------------------
// The epochs are cut into time segments s = [b_s, b_{s+1}) at clean cuts
// (walk_segment_bounds, lower.hpp).  A word whose walk spans segments s0..K
// (K: the last segment for words holding observables, else the one holding
// the word's last measurement) runs as
//   launch A: SEG_FIRST  -- [e0, b_{s0+1}) from zero rows, with snapshots; exit rows -> a state;
//             SEG_AFF    -- each segment s in (s0, K) holding measurements of the word,
//                           from zero rows, no snapshots; exit rows -> a state (c_s);
//             SEG_XFER   -- per segment s and 64-row column c, the walk of unit rows
//                           without measurement bits: column c of the transfer matrix A_s;
//   launch B: SEG_REST   -- segment s in (s0, K]: entry rows composed from the
//                           first part's exit through A and c of segments
//                           (s0, s), then the segment walked with snapshots
//                           (the last one on to the end, or until the rows vanish).
// A word that spans one segment is a single SEG_FIRST item walking to the end.
// States are [2 qpad] u64 rows: X of slots 0..qpad-1, then Z of the same slots.
enum : uint32_t { SEG_FIRST = 0, SEG_AFF = 1, SEG_XFER = 2, SEG_REST = 3 };
// Entries of a transfer row kept as a sparse list (rows with more are read
// from the dense transfer columns): measured on code circuits, rows hold 1-3
// entries on average and up to 12 where a cut falls inside a round.
constexpr uint32_t kSegRowCap = 16;
// Entries of a row that the compose prefetches (one 16-byte load; entries
// kSegNear .. kSegRowCap - 1, rare, are loaded when they are needed).
constexpr uint32_t kSegNear = 8;
struct SegItem {
  uint32_t kind;
  uint32_t idx;             // word (SEG_XFER: first transfer column of the item's SegLaunch::cols)
  uint32_t e_begin, e_end;  // epochs walked
  uint32_t state;           // FIRST/AFF/XFER: state written at exit (0xFFFFFFFF: none); REST: entry state
  uint32_t s_from, s_to;    // REST: compose through segments [s_from, s_to) before walking; XFER: s_from
                            // is the segment
  uint32_t pad;
};
static_assert(sizeof(SegItem) == 32, "segment item is 32 bytes");
struct SegLaunch {
  const CircuitDev *circ;   // the circuit
  const SegItem *items;
  uint32_t n_items;
  uint32_t threads, qpt, qpad;
  uint32_t max_epochs;
  uint32_t cols;            // transfer columns a SEG_XFER item walks (ncol is a multiple of it)
  uint64_t *state;          // [states][2 qpad]
  uint32_t xfer0;           // state of segment s's transfer column c: xfer0 + s * ncol + c
  uint32_t ncol;            // 64-row columns of a transfer matrix: ceil(2 qpad / 64), rounded up to cols
  const uint32_t *aff;      // [w][S] state of word j's SEG_AFF walk of segment s (0xFFFFFFFF: no measurements)
  uint32_t S;
  uint32_t *xcnt;           // [S][2 qpad] (zeroed) entries of each transfer row
  uint16_t *xlst;           // entries 0..7 [S][2 qpad][kSegNear], then entries 8..15 [S][2 qpad][8]
};
// Dynamic shared memory of a segment launch (0: it does not fit a CTA).
size_t walk_seg_smem_bytes(const SegLaunch &L);
cudaError_t launch_walk_seg(const SegLaunch &L, bool rest, cudaStream_t s);  // launch A, or (rest) launch B
bool walk_seg_supported(uint32_t qpad, uint32_t qpt);
uint32_t walk_seg_cols(uint32_t qpad, uint32_t qpt);  // transfer columns per SEG_XFER item
// Staged epoch/chunk table bytes for a launch (0: the tables are read from global memory).
uint32_t walk_table_bytes(uint32_t max_epochs, uint32_t max_chunks);
size_t walk_smem_bytes(uint32_t qpad, uint32_t chunk_cap, uint32_t table_bytes, uint32_t words);
uint32_t walk_max_threads(uint32_t qpt);  // 0: no walk instance for this many qubits per thread
bool walk_queue_supported(uint32_t qpt, uint32_t words);  // a persistent walk instance exists

// One bucket slot (64 bytes): an item is one symptom of one noise record, with
// the record's mechanisms that have it merged.  Its 128-bit key, then (first
// mechanism, targets | mechanisms merged << 24, probability), then its first
// targets: 16 16-bit ones when every circuit of the run has at most 65,536
// detectors and observables (narrow), else 8 32-bit ones; unused ones are zero.
// Later targets sit in the first mechanism's row of the target lists.  With
// the targets in a row of their own, the grouping and the emission read one
// scattered sector per item for them (32 mixed surface codes: emission 42 -> 37
// us with them here).
// The group stage overwrites the tail of a bucket's first slots with one record
// per group: (head mechanism, targets before the group inside the bucket << 8 |
// the head's slot, probability).  For gradients it also overwrites the keys with
// 32-bit words: of slot s, [0] the first mechanism and [3] the mechanisms merged
// of the item at sorted position s; for s < groups, [1] the first sorted
// position of group s.
struct SlotTail {
  uint32_t m, t;
  double p;
};
static_assert(sizeof(SlotTail) == 16, "slot tail is 16 bytes");
constexpr uint32_t kSlotCount = 0xFFFFFFu;  // target count in SlotTail::t (saturated)
struct alignas(64) Slot {
  ulonglong2 key;
  SlotTail tail;
  uint32_t list[8];
};
static_assert(sizeof(Slot) == 64, "a slot is two 32-byte sectors");
__host__ __device__ __forceinline__ uint32_t *slot_perm(Slot *bucket, uint32_t s) {
  return reinterpret_cast<uint32_t *>(&bucket[s].key);
}
__host__ __device__ __forceinline__ const uint32_t *slot_perm(const Slot *bucket, uint32_t s) {
  return reinterpret_cast<const uint32_t *>(&bucket[s].key);
}
// Items of a bucket counter (its high half counts mechanisms; past 2^16 of
// either the counter wraps, but the run was flagged long before).
__device__ __forceinline__ uint32_t bucket_items(uint32_t count) { return count & 0xFFFFu; }

struct KeyLaunch {
  const CircuitDev *circs;  // [n_circ]
  const uint32_t *kbase;    // [n_circ] first key warp of each circuit
  uint32_t n_circ, M;       // circuits, mechanisms of the whole batch
  uint32_t n_warps, chunk;  // key warps, of `chunk` mechanisms each: ceil(mechanisms / chunk) of each circuit
  uint32_t *first;          // [n_warps] first record of each warp (launch_key_prep); of a circuit's first warp 0
  uint32_t *bucket_count;   // [buckets of the batch] (zeroed) items | mechanisms << 16
  Slot *slot;               // [buckets * SLOT_CAP] bucket slots
  uint32_t *tl;             // [M][tstride] targets past a slot's
  uint32_t tstride, narrow;
  uint32_t keep;            // gradients (one circuit): an item's m is its record << 4 | its first component
  uint32_t *list_total;     // += targets written to the lists (for traffic accounting)
  uint32_t *err;
  ulonglong2 *key;          // [M] global path (one circuit)
};
constexpr uint32_t KEY_THREADS = 256;
uint32_t key_chunk(uint64_t mechanisms);  // mechanisms per key warp for a run of this many
// Finds each key warp's first record (one thread per warp).
cudaError_t launch_key_prep(const KeyLaunch &L, cudaStream_t s);
// Bucket path: the records' symptoms keyed, listed and filed in their buckets.
cudaError_t launch_keys(const KeyLaunch &L, cudaStream_t s);
// Global path: every mechanism's key, descriptor and probability.
cudaError_t launch_keys_all(const KeyLaunch &L, cudaStream_t s);

// Merge of the compile pipeline (no inter-CTA waits).  The key kernel has put
// every item into a slot of its bucket (SLOT_CAP slots per bucket; more than
// SLOT_CAP mechanisms raise DEV_FLAG_BIG_BUCKET).
//  group: one warp per bucket
//         orders its items (by the top 6 bits of the key's second half, then by
//         key, then by mechanism), checks collisions, folds each group's
//         probability and overwrites the bucket's first slots with one record
//         per group (SlotTail); bucket aggregates (groups, targets) and their
//         per-tile sums;
//  scan:  exclusive scan of the bucket aggregates, one block per SCAN_TILE
//         buckets (tile sums give each block its prefix); small runs fold it
//         into the emission;
//  emit:  one warp per bucket writes its groups' probabilities, offsets and
//         target lists to the DEM arrays.
struct GroupLaunch {
  const uint32_t *tl;       // [M][tstride] targets past a slot's
  uint32_t tcap, tstride, narrow;
  Slot *slot;               // [nb * SLOT_CAP] items; afterwards one group record per group in the tails and
                            // (keep) the saved permutation in the keys (slot_perm)
  uint32_t keep;            // gradients: keep the permutation; an item's m is its record << 4 | its first component
  const uint32_t *rec_moff; // (keep) first mechanism of each record
  const uint32_t *count;    // [nb] (bucket_items)
  uint32_t nb;
  uint2 *bagg;              // [nb] (groups, targets) of each bucket
  uint2 *bout;              // [nb] exclusive prefix of bagg
  uint2 *tsum;              // [ceil(nb / SCAN_TILE)] (zeroed) per-tile sums of bagg
  double *out_prob;
  uint32_t *out_off;
  uint32_t *out_tg;
  uint32_t tg_cap;
  uint32_t *totals;         // [0] groups, [1] targets, [3] += bucketed items
  const uint32_t *cbbase;   // [n_circ] first bucket of each circuit
  uint32_t n_circ;
  uint2 *cout;              // [n_circ] (first slot, first target) of each circuit's output
  uint32_t *err;
  uint32_t *host_res;       // one circuit: [flags, groups, targets] in page-locked host memory, written by the
                            // emission where emit_folds() (else the host copies them)
};
constexpr uint32_t kFoldBuckets = 32768;  // most buckets whose places the emission finds itself
inline bool emit_folds(uint32_t nb) { return nb <= kFoldBuckets; }
cudaError_t launch_group(const GroupLaunch &L, cudaStream_t s);

// ---- noise-rate gradients (single circuit) ----------------------------------
// Record probabilities from a [n_ticks][4] FP64 noise tensor: record r takes
// its source's rate through its channel's split, looked up in qtab[src][kind]
// (kind 0: X/Y/Z error or measurement flip, 1: DEPOLARIZE1, 2: DEPOLARIZE2),
// which the host fills with the same split formulas as the text path.
// Records without a source keep their probability.
struct ParamLaunch {
  const uint64_t *rec;
  const uint32_t *rec_src;
  double *rec_p;
  uint32_t R, n_src;
  const double *qtab;  // [n_src][3]
};
cudaError_t launch_param_rec(const ParamLaunch &L, cudaStream_t s);

// Adjoint of the merge and of the channel splits:
//  group:  one warp per bucket, a lane per sorted position: dL/dq_m = dL/dp_g *
//          prod_{j in g, j != m} (1 - 2 q_j) from prefix and suffix product
//          scans along the group's run in the saved permutation;
//  source: dL/dnoise[e] = sum over the records of source e of (the sum of the
//          record's mechanisms' dL/dq) * dq/dp, the split's slope at the
//          source's rate (stab[src][kind], filled by the host).
struct AdjointLaunch {
  const Slot *slot;        // saved permutation (see GroupLaunch)
  const uint32_t *count;
  const uint2 *bagg, *bout;
  uint32_t nb;
  const double *rec_p;     // [R] each record's component probability of the forward (from the noise tensor)
  const double *grad_out;  // [groups] dL/dp of each merged mechanism
  double *gq;              // [M] (zeroed) dL/dq summed over each item's mechanisms, at its first mechanism
  const uint64_t *rec;
  const uint32_t *rec_moff;
  const double *stab;      // [n_src][3] dq/dp of each source and channel kind
  const uint32_t *src_off, *src_rec;  // records of each source (CSR, record order)
  uint32_t n_src;
  double *grad_noise;      // [n_src]
};
cudaError_t launch_adjoint(const AdjointLaunch &L, cudaStream_t s);
cudaError_t launch_scan_emit(const GroupLaunch &L, cudaStream_t s);

// ---- global path (used when a bucket is too large for one CTA) -------------
// Onesweep radix sort of (u64 key, u32 value) pairs on the `bits` bits from bit `shift0` on.
struct SortScratch {
  uint32_t *hist;      // [passes][RADIX]
  uint32_t *status;    // [passes][tiles][RADIX]
  uint32_t *tile_ctr;  // [passes]
  uint32_t *err;
  unsigned long long spin_ns;  // a look-back wait gives up (DEV_ERR_TIMEOUT) after this long
  // Test of the bounded look-back: tile 0 of the first pass keeps its digit
  // counts to itself, so the waits of the tiles after it run out.
  uint32_t hold_first;
};
size_t sort_scratch_words(uint32_t n, uint32_t bits);
// The first pass reads its keys from `first`, every `stride`-th u64, and its values from `vals` or (index_vals)
// takes the keys' indices; the passes then alternate between (keys_alt, vals_alt) and (keys, vals).
cudaError_t launch_sort(const uint64_t *first, uint32_t stride, bool index_vals, uint64_t *keys, uint64_t *keys_alt,
                        uint32_t *vals, uint32_t *vals_alt, uint32_t n, uint32_t shift0, uint32_t bits,
                        const SortScratch &scr, cudaStream_t s, bool *result_in_alt);

// Gathers key128[perm[i]].y into out[i] (second pass of a 128-bit sort).
cudaError_t launch_gather_hi(const ulonglong2 *key, const uint32_t *perm, uint64_t *out, uint32_t n, cudaStream_t s);

struct MergeLaunch {
  const CircuitDev *c_dev;  // single circuit
  const uint32_t *perm;     // sorted mechanism ids
  const uint64_t *sortkey;  // sorted keys (for the mixed-run check)
  uint64_t sort_mask;       // key bits the sort compared (0: skip the mixed-run check)
  const ulonglong2 *key;    // 128-bit key per mechanism
  uint32_t n;
  double *out_prob;
  uint32_t *out_off;
  uint32_t *out_tg;
  uint32_t tg_cap;
  unsigned long long *status;  // [tiles]
  uint32_t *tile_ctr;
  uint32_t *totals;  // [0] groups, [1] targets
  uint32_t *err;
  unsigned long long spin_ns;  // a look-back wait gives up (DEV_ERR_TIMEOUT) after this long
};
cudaError_t launch_merge(const MergeLaunch &L, cudaStream_t s);

}  // namespace gpc
