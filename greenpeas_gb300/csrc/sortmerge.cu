// sortmerge.cu -- symptom keys, radix bucketing / onesweep sort, merge (sm_103a).
//
// Replaces the reference's K3-K7 (Policies/Compute/CUDA.hpp:184-189,276-343,
// 422-497; CUDAHandlers.hpp:67-139): set-bit extraction truncated at 32 bits
// + a 64-bit FNV hash with no collision check, CUB radix sort, a gather of
// probabilities, CUB reduce-by-key and a gather of the full class matrix.
//
//  * key_items_kernel: a warp takes a run of noise records.  Each record's
//    mechanisms (the Pauli components of its channel) are the XORs of the
//    snapshot rows of its one or two points; the components of one symptom
//    become one item, with a 128-bit key K = XOR_j H(j, word_j) over the
//    symptom's words (H(j, 0) = 0, so the empty symptom has key 0) and its
//    target list, filed in a slot of its bucket (the top bits of K).
//  * group_kernel: orders a bucket's items by key, checks
//    every item's full target list against its run's (collision check) and
//    folds the run's probabilities with p <- p(1-q) + q(1-p)
//    (CUDAHandlers.hpp:124-139) in FP64; group_scan_kernel and emit_kernel
//    write the groups to the DEM arrays.  The empty symptom is dropped
//    (Driver.hpp:185).
//  * global path, used when a bucket overflows (more than SLOT_CAP mechanisms):
//    key_all_kernel keys every mechanism on its own; LSD onesweep radix sort of all keys (one
//    kernel per 8-bit digit, tile ranks by warp match/popc, decoupled
//    look-back for digit offsets) and a merge kernel over the sorted run.
#include <algorithm>
#include <cstdint>

#include "device.cuh"
#include "group.cuh"
#include "lower.hpp"

namespace gpc {
namespace {

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint64_t pauli_sel(ulonglong2 s, uint32_t P) {
  return (s.x & (0ull - (uint64_t)(P & 1u))) ^ (s.y & (0ull - (uint64_t)((P >> 1) & 1u)));
}

__device__ __forceinline__ uint64_t mk_desc(uint32_t pa, uint32_t Pa, uint32_t pb, uint32_t Pb) {
  return (uint64_t)(pa & 0x3FFFFFFFu) | ((uint64_t)(Pa & 3u) << 30) | ((uint64_t)(pb & 0x3FFFFFFFu) << 32) |
         ((uint64_t)(Pb & 3u) << 62);
}

// Components of each record type as (Pauli a | Pauli b << 2); Pauli: 1 X, 2 Z, 3 Y.
// Two-qubit lists follow stim's order IX IY IZ XI XX XY XZ YI YX YY YZ ZI ZX ZY ZZ,
// restricted to the correlation level's set (Mixer.hpp:13-20).
#define PP(a, b) ((a) | ((b) << 2))
__constant__ uint8_t kComp[6][15] = {
    {0},
    {PP(1, 0), PP(2, 0)},
    {PP(1, 0), PP(3, 0), PP(2, 0)},
    {PP(0, 1), PP(0, 2), PP(1, 0), PP(1, 1), PP(2, 0), PP(2, 2)},
    {PP(0, 1), PP(0, 3), PP(0, 2), PP(1, 0), PP(1, 1), PP(1, 2), PP(3, 0), PP(2, 0), PP(2, 1), PP(2, 2)},
    {PP(0, 1), PP(0, 3), PP(0, 2), PP(1, 0), PP(1, 1), PP(1, 3), PP(1, 2), PP(3, 0), PP(3, 1), PP(3, 3), PP(3, 2),
     PP(2, 0), PP(2, 1), PP(2, 3), PP(2, 2)},
};
#undef PP

// find_circuit by a warp: 32 places per round of loads.
__device__ __forceinline__ uint32_t find_circuit_warp(const uint32_t *base, uint32_t n, uint32_t x) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lo = 0, len = n;
  while (len > 1) {
    const uint32_t step = (len + 31u) / 32u, at = lane * step;
    const uint32_t le = __ballot_sync(0xFFFFFFFFu, at < len && __ldg(base + lo + at) <= x);
    const uint32_t k = (31u - __clz(le)) * step;
    lo += k;
    len = min(step, len - k);
  }
  return lo;
}

// ---- keys of the bucket path ---------------------------------------------------
//
// Bound by instructions (863 a warp of 32 mechanisms when a thread followed
// one mechanism: its words, two 64-bit mixes per word, its targets), so the
// work is done once per distinct thing instead of once per mechanism.  A
// record's mechanisms are the XORs of the (X, Z) rows of its one or two points,
// selected by s = Pauli a | Pauli b << 2, so over the words a record touches
// (entries) each entry holds the span of four rows: 1 or 3 distinct non-zero
// values for 97% of the entries of the code circuits, 3, 7 or 15 distinct
// symptoms for a two-qubit channel's 15 components.  A warp takes the records
// that start among L.chunk mechanisms:
//   records  (a lane each)  masks of the non-zero words, one entry per set word;
//   entries  (a lane each)  rows, their coordinates in a basis of their span
//                           (lut: nibble s is the coordinate of value s; equal
//                           coordinates, equal values), the distinct values, the
//                           targets of the union and each row as a bit mask of them;
//   values   (a lane each)  the 128-bit hash of (word, value);
//   records                 the selections whose symptom vanishes (a subgroup: the
//                           nibbles that are zero in every entry), one item per
//                           coset, with as many of the channel's components
//                           as lie in it (a coset's components share the symptom
//                           and the probability, so they are merged here);
//   items    (a lane each)  key = XOR of the values' hashes, targets, a slot.
// Warps never wait for one another.  Measured on 32 mixed surface codes (4.0M
// mechanisms): 863 -> ~590 instructions per 32 mechanisms, 212 -> 126 us, and
// a third fewer items for the grouping (203 -> 153 us, 10 -> 2 for the buckets
// of more than a warp's items); surface d = 25 60 -> 46 us, [[144,12,12]] (one
// wave of warps, bound by a warp's latency) 15.8 -> 17.5 and its grouping 18.7
// -> 13.2.  Kept out: 48 registers for a fifth block an SM (spills: 152 us), and
// a copy of the launch's parameters on the stack (151 us).
constexpr uint32_t kKeyWarps = 8;
constexpr uint32_t kKeyEntries = 64;   // entries a warp holds at once
constexpr uint32_t kKeyValues = 128;   // distinct values
constexpr uint32_t kKeyTargets = 160;  // targets of the records' unions (up to 32 a record)
constexpr uint32_t kKeyItems = 256;
constexpr uint32_t kKeyRecords = 128;  // records of a warp (one mechanism each at least: key_chunk)

// Components present (bit s) and their place in the component list, by record type (kComp).
__constant__ uint16_t kPresent[6] = {0, 0x0006, 0x000E, 0x0536, 0x177E, 0xFFFE};
// (nibble s is the place of component s)
__constant__ uint64_t kPlace[6] = {0, 0x100, 0x1200, 0x50100300420, 0x1095208406730, 0x9D51AE628C407B30};

struct KeyWarp {
  ulonglong2 h[kKeyValues];  // (value, word), then its hash
  uint64_t lut[kKeyEntries];
  uint4 rows[32];            // Xa, Za, Xb, Zb of each record over its targets
  double p[32];
  uint32_t ent[kKeyEntries]; // word | record << 18 | point a set << 26 | point b set << 27
  uint32_t targets[kKeyTargets];
  uint32_t pa[32], pb[32], moff[32];
  uint16_t hb[kKeyEntries];  // first value of each entry
  uint16_t tstart[32], vstart[32];  // first target and first value of each record
  uint16_t join[32];         // selections that join components of one symptom (bit s)
  uint16_t item[kKeyItems];  // record << 4 | s
  uint64_t place[32];        // kPlace of the record's type
  uint16_t present[32];      // the record's components (bit s)
  uint8_t e0[32], e1[32];
  uint32_t late[kKeyRecords / 32];  // records left for key_late_records
};

// Probability that an odd number of `c` independent events of probability q happens.
__device__ __forceinline__ double repeat_merge(double q, uint32_t c) {
  double p = q;
  uint32_t k = 1;
  for (; 2 * k <= c; k *= 2) p = xor_merge(p, p);
  for (; k < c; ++k) p = xor_merge(p, q);
  return p;
}

// m with its bits permuted by s -> s ^ k.
__device__ __forceinline__ uint32_t xor_bits16(uint32_t m, uint32_t k) {
  if (k & 1u) m = ((m >> 1) & 0x5555u) | ((m & 0x5555u) << 1);
  if (k & 2u) m = ((m >> 2) & 0x3333u) | ((m & 0x3333u) << 2);
  if (k & 4u) m = ((m >> 4) & 0x0F0Fu) | ((m & 0x0F0Fu) << 4);
  if (k & 8u) m = ((m >> 8) & 0x00FFu) | ((m & 0x00FFu) << 8);
  return m;
}

// A record's subgroup of selections without a symptom, as far as it can join two of its components.
__device__ __forceinline__ uint32_t joining(uint32_t type, uint32_t zero) {
  return type >= REC_DEP2_L0 ? zero : type == REC_PAULI ? 0x1u : zero & 0xFu;
}

// One component of every coset with a symptom: the one with the smallest s.
__device__ __forceinline__ uint32_t coset_heads(uint32_t present, uint32_t zero, uint32_t join) {
  uint32_t heads = present & ~zero;
  for (uint32_t ks = join & ~1u; ks; ks &= ks - 1) {
    const uint32_t k = __ffs(ks) - 1u;
    const uint32_t top = 31u - __clz(k);  // s ^ k < s where s has k's top bit
    const uint32_t larger = top == 0 ? 0xAAAAu : top == 1 ? 0xCCCCu : top == 2 ? 0xF0F0u : 0xFF00u;
    heads &= ~(xor_bits16(present, k) & larger);
  }
  return heads;
}

// Files an item in its bucket: one 64-byte slot as two 32-byte stores.  The
// bucket's counter counts items in its low half and mechanisms in its high
// half: a bucket overflows by its mechanisms, whatever is merged beforehand.
__device__ __forceinline__ void file_item(const KeyLaunch &L, uint32_t bbase, uint32_t bbits, uint32_t tcap, uint64_t hx,
                                          uint64_t hy, uint32_t m, uint32_t cnt, uint32_t mult, double p,
                                          const uint32_t (&l)[8]) {
  if ((hx | hy) == 0) {  // a non-empty symptom hashed to 0
    atomicOr(L.err, DEV_ERR_COLLISION);
    return;
  }
  if (cnt > tcap) atomicOr(L.err, DEV_FLAG_LONG);
  const uint32_t b = bbase + (uint32_t)(hx >> (64u - bbits));
  const uint32_t old = atomicAdd(L.bucket_count + b, 1u | (mult << 16));
  const uint32_t slot = old & 0xFFFFu;
  if ((old >> 16) + mult > SLOT_CAP) atomicOr(L.err, DEV_FLAG_BIG_BUCKET);
  if (slot >= SLOT_CAP) return;
  Slot *s = L.slot + (size_t)b * SLOT_CAP + slot;
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(s), "l"(hx), "l"(hy),
               "l"((uint64_t)m | (uint64_t)(min(cnt, kSlotCount) | (mult << 24)) << 32), "l"(__double_as_longlong(p)));
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(&s->list[0]), "r"(l[0]), "r"(l[1]),
               "r"(l[2]), "r"(l[3]), "r"(l[4]), "r"(l[5]), "r"(l[6]), "r"(l[7]));
}

// ---- records of long symptoms
//
// Where a record holds more words, values or targets than the warp's arrays, or
// so few records fit them that most lanes would idle, the warp leaves the
// records for its end (the calls below in the loop itself would cost every
// record their registers) and then follows their components through the words,
// as many records of a type at a time as have components for the 32 lanes.
// Bound by the instructions of the words' hashes and lists, and for few
// mechanisms by the chain of the words' loads.  A memory of 400 qubits measured
// 100 times without resets, every measurement a detector (460k mechanisms,
// symptoms of up to 100 targets): one record at a time 6,390 us, side by side
// 350; a thread per mechanism, which is slower for short symptoms, 222.

// Components of a record, the lanes it takes in key_records_direct.
__device__ __forceinline__ uint32_t components(uint32_t type) {
  return type == REC_PAULI ? 1u : (uint32_t)__popc((uint32_t)kPresent[type]);
}
// Selections that are no component of the type (nibble l: lane l's; 0: none), a second one for some lanes.
__constant__ uint64_t kSpare[6][2] = {{0, 0}, {0x3, 0}, {0, 0}, {0xCB9763, 0xFED}, {0xFEDB7, 0}, {0, 0}};

// `n` records of one type side by side.  The components of one symptom are
// merged as in key_items_kernel, which wants the selections without a symptom:
// SPARE, the type's components are not all of them (correlation levels 0 and
// 1), and each lane looks out for up to two more.
template <bool SPARE>
__device__ __forceinline__ uint32_t key_records_direct(const KeyLaunch &L, const CircuitDev &C, uint32_t r0, uint32_t n,
                                                       uint32_t type, uint32_t *stage) {
  const uint32_t lane = threadIdx.x & 31u, width = components(type);
  const uint32_t k = lane / width, l0 = k * width, place = lane - l0;
  const bool in = k < n;
  const uint32_t r = r0 + (in ? k : 0u);
  const uint64_t d = __ldg(C.rec + r);
  const uint32_t s = type == REC_PAULI ? (uint32_t)(d >> 60) & 15u : kComp[type][place];
  const uint32_t s1 = SPARE ? (uint32_t)(kSpare[type][0] >> (4u * place)) & 15u : 0u;
  const uint32_t s2 = SPARE ? (uint32_t)(kSpare[type][1] >> (4u * place)) & 15u : 0u;
  const bool has_a = in && ((s | s1 | s2) & 3u), has_b = in && ((s | s1 | s2) >> 2);
  const uint32_t np = C.npoints, mw = C.mw, tcap = C.tcap;
  const bool narrow = L.narrow;
  const uint32_t m = C.mbase + __ldg(C.rec_moff + r) + place;
  uint32_t *const far = L.tl + (size_t)m * L.tstride - (narrow ? 16u : 8u);  // (the row holds the targets past the slot's)
  // the item's first targets, [word][lane]
  __syncwarp();
  for (uint32_t i = 0; i < 8; ++i) stage[i * 32u + lane] = 0;
  uint64_t hx = 0, hy = 0, any1 = 0, any2 = 0;
  uint32_t cnt = 0;
  auto word = [&](uint32_t j, uint64_t v) {
    const ulonglong2 h = word_hash(j, v);
    hx ^= h.x;
    hy ^= h.y;
    for (; v; v &= v - 1, ++cnt) {
      const uint32_t t = j * 64u + (uint32_t)(__ffsll((long long)v) - 1);
      if (cnt >= (narrow ? 16u : 8u)) {
        if (cnt < tcap) far[cnt] = t;
      } else if (narrow) {
        reinterpret_cast<uint16_t *>(stage)[((cnt >> 1) * 32u + lane) * 2u + (cnt & 1u)] = (uint16_t)t;
      } else {
        stage[cnt * 32u + lane] = t;
      }
    }
  };
  const uint32_t pa = (uint32_t)(d & 0x0FFFFFFFu), pb = (uint32_t)((d >> 28) & 0x0FFFFFFFu);
  const unsigned long long *ma = C.nzm + (size_t)pa * mw, *mb = C.nzm + (size_t)pb * mw;
  const ulonglong2 *const snap_a = C.snap + pa, *const snap_b = C.snap + pb;
  for (uint32_t i = 0; i < mw; ++i) {
    const uint64_t ba = has_a ? __ldg(ma + i) : 0ull, bb = has_b ? __ldg(mb + i) : 0ull;
    for (uint64_t bits = ba | bb; bits;) {  // (two words' rows on the way at once; four targets a store: no gain)
      const uint32_t b0 = (uint32_t)(__ffsll((long long)bits) - 1);
      bits &= bits - 1;
      const uint32_t b1 = bits ? (uint32_t)(__ffsll((long long)bits) - 1) : 64u;
      bits &= bits - 1;
      const size_t j0 = (size_t)(i * 64u + b0) * np, j1 = (size_t)(i * 64u + b1) * np;
      ulonglong2 xa = make_ulonglong2(0, 0), xb = xa, ya = xa, yb = xa;
      if ((ba >> b0) & 1ull) xa = snap_a[j0];
      if ((bb >> b0) & 1ull) xb = snap_b[j0];
      if (b1 < 64u && ((ba >> b1) & 1ull)) ya = snap_a[j1];
      if (b1 < 64u && ((bb >> b1) & 1ull)) yb = snap_b[j1];
      if constexpr (SPARE) {
        any1 |= pauli_sel(xa, s1) ^ pauli_sel(xb, s1 >> 2) | pauli_sel(ya, s1) ^ pauli_sel(yb, s1 >> 2);
        any2 |= pauli_sel(xa, s2) ^ pauli_sel(xb, s2 >> 2) | pauli_sel(ya, s2) ^ pauli_sel(yb, s2 >> 2);
      }
      const uint64_t v0 = pauli_sel(xa, s) ^ pauli_sel(xb, s >> 2), v1 = pauli_sel(ya, s) ^ pauli_sel(yb, s >> 2);
      if (v0) word(i * 64u + b0, v0);
      if (v1) word(i * 64u + b1, v1);
    }
  }
  const uint32_t group = (uint32_t)(((1ull << width) - 1ull) << l0);  // the record's lanes (those past the last record's: one too)
  __syncwarp();
  const uint32_t zero = 1u | __reduce_or_sync(group, (cnt ? 0u : 1u << s) | (any1 ? 0u : 1u << s1) | (any2 ? 0u : 1u << s2));
  const uint32_t present = type == REC_PAULI ? 1u << s : kPresent[type], join = joining(type, zero);
  if (!in || !((coset_heads(present, zero, join) >> s) & 1u)) return 0;
  uint32_t l[8];
#pragma unroll
  for (uint32_t i = 0; i < 8; ++i) l[i] = stage[i * 32u + lane];
  const uint32_t mult = (uint32_t)__popc(xor_bits16(join, s) & present);
  file_item(L, C.bbase, C.bbits, tcap, hx, hy, L.keep ? r << 4 | place : m, cnt, mult, repeat_merge(__ldg(C.rec_p + r), mult), l);
  return cnt;
}

// The records that a warp postponed: bits of `late`, from its first record on.
__device__ __noinline__ uint32_t key_late_records(const KeyLaunch &L, const CircuitDev &C, uint32_t first, KeyWarp &S) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t listed = 0;
  for (uint32_t p = 0; p < kKeyRecords;) {
    // bits p .. p + 31
    const uint32_t hi = p / 32u + 1u < kKeyRecords / 32u ? S.late[p / 32u + 1u] : 0u;
    const uint32_t bits = __funnelshift_r(S.late[p / 32u], hi, p & 31u);
    if (bits == 0) {
      p += 32;
      continue;
    }
    p += (uint32_t)__ffs((int)bits) - 1u;
    const uint32_t run = bits >> (__ffs((int)bits) - 1);  // from its first record on
    const uint32_t type = (run >> lane) & 1u ? (uint32_t)(__ldg(C.rec + first + p + lane) >> 56) & 15u : 16u;
    const uint32_t type0 = __shfl_sync(0xFFFFFFFFu, type, 0);
    const uint32_t other = __ballot_sync(0xFFFFFFFFu, type != type0);
    const uint32_t n = min(other ? (uint32_t)__ffs((int)other) - 1u : 32u, 32u / components(type0));
    uint32_t *const stage = reinterpret_cast<uint32_t *>(S.h);
    listed += kSpare[type0][0] ? key_records_direct<true>(L, C, first + p, n, type0, stage)
                               : key_records_direct<false>(L, C, first + p, n, type0, stage);
    p += n;
  }
  return listed;
}

__global__ void __launch_bounds__(kKeyWarps * 32, 4) key_items_kernel(const __grid_constant__ KeyLaunch L) {
  __shared__ KeyWarp s_warp[kKeyWarps];
  const uint32_t lane = threadIdx.x & 31u;
  KeyWarp &S = s_warp[threadIdx.x >> 5];
  const uint32_t w = blockIdx.x * kKeyWarps + (threadIdx.x >> 5);
  if (w >= L.n_warps) return;
  const uint32_t c = L.n_circ == 1 ? 0u : find_circuit_warp(L.kbase, L.n_circ, w);
  const CircuitDev &C = L.circs[c];
  const uint32_t r_end = w + 1 < L.n_warps ? L.first[w + 1] : 0u;  // (0: the last warp of its circuit)
  const uint32_t mw = C.mw, np = C.npoints, bbase = C.bbase, bbits = C.bbits, tcap = C.tcap;
  const ulonglong2 *const snap = C.snap;
  constexpr uint32_t ALL = 0xFFFFFFFFu;
  uint32_t listed = 0;  // targets written by this lane's items
  if (lane < kKeyRecords / 32) S.late[lane] = 0;
  // How many of the next records key_records_direct would take at a time: those of the first one's type.
  auto side_by_side = [&](uint64_t d, uint32_t nrec) -> uint32_t {
    const uint32_t type = (uint32_t)(d >> 56) & 15u, type0 = __shfl_sync(ALL, type, 0);
    const uint32_t other = __ballot_sync(ALL, lane >= nrec || type != type0);
    return min(other ? (uint32_t)__ffs((int)other) - 1u : 32u, 32u / components(type0));
  };
  // Leaves n records (32 at most) to key_late_records, from the warp's record r on.
  auto postpone = [&](uint32_t r, uint32_t n) {
    const uint64_t bits = (uint64_t)(0xFFFFFFFFu >> (32u - n)) << (r & 31u);
    if (lane == 0) {
      S.late[r / 32u] |= (uint32_t)bits;
      if (bits >> 32) S.late[r / 32u + 1u] |= (uint32_t)(bits >> 32);
    }
  };
  // the records from r0 on, as many at a time as fit the warp's arrays
  const uint32_t first = L.first[w];
  for (uint32_t r0 = first, r1 = r_end ? r_end : C.R; r0 < r1;) {
    const uint32_t nrec = min(r1 - r0, 32u);
    uint64_t d = 0;
    uint32_t words = 0, present = 0;
    bool has_a = false, has_b = false;
    const unsigned long long *ma = C.nzm, *mb = C.nzm;
    __syncwarp();
    if (lane < nrec) {
      d = __ldg(C.rec + r0 + lane);
      const uint32_t pa = (uint32_t)(d & 0x0FFFFFFFu), pb = (uint32_t)((d >> 28) & 0x0FFFFFFFu);
      const uint32_t type = (uint32_t)((d >> 56) & 15u);
      S.p[lane] = __ldg(C.rec_p + r0 + lane);
      S.moff[lane] = C.mbase + __ldg(C.rec_moff + r0 + lane);
      S.pa[lane] = pa;
      S.pb[lane] = pb;
      S.place[lane] = kPlace[type];
      S.rows[lane] = make_uint4(0, 0, 0, 0);
      present = type == REC_PAULI ? 1u << ((uint32_t)(d >> 60) & 15u) : kPresent[type];
      S.present[lane] = (uint16_t)present;
      has_a = (present & 0xEEEEu) != 0;
      has_b = (present & 0xFFF0u) != 0;
      ma += (size_t)pa * mw;
      mb += (size_t)pb * mw;
      for (uint32_t i = 0; i < mw; ++i)
        words += (uint32_t)__popcll((has_a ? __ldg(ma + i) : 0ull) | (has_b ? __ldg(mb + i) : 0ull));
    }
    // the next records whose words fit the entries
    uint32_t inc = words;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(ALL, inc, o);
      if (lane >= (uint32_t)o) inc += x;
    }
    uint32_t take = (uint32_t)__popc(__ballot_sync(ALL, lane < nrec && inc <= kKeyEntries));
    // (twice as many: records of a few words, as the bicycle codes', are better off here; side_by_side is
    // asked only where its bound, 32 / components, allows it: [[288,12,18]] 117.35 -> 117.05 us a run)
    if (take < nrec && take * components((uint32_t)(__shfl_sync(ALL, d, 0) >> 56) & 15u) < 16u) {
      const uint32_t beside = side_by_side(d, nrec);
      if (2u * take < beside) {
        postpone(r0 - first, beside);
        r0 += beside;
        continue;
      }
    }
    uint32_t over = take;  // first record that does not fit the arrays below
    const uint32_t E = take ? __shfl_sync(ALL, inc, take - 1u) : 0u;
    if (lane < take) {
      uint32_t at = inc - words;
      S.e0[lane] = (uint8_t)at;
      S.e1[lane] = (uint8_t)inc;
      for (uint32_t i = 0; i < mw; ++i) {
        const uint64_t ba = has_a ? __ldg(ma + i) : 0ull, bb = has_b ? __ldg(mb + i) : 0ull;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint32_t wa = (uint32_t)(ba >> (32 * half)), wb = (uint32_t)(bb >> (32 * half));
          for (uint32_t bits = wa | wb; bits; bits &= bits - 1) {
            const uint32_t low = bits & (0u - bits);
            S.ent[at++] = (i * 64u + 32u * half + (uint32_t)(31 - __clz(low))) | (lane << 18) |
                          (wa & low ? 1u << 26 : 0u) | (wb & low ? 1u << 27 : 0u);
          }
        }
      }
    }
    __syncwarp();
    uint32_t H = 0, TG = 0;  // values and targets of the entries so far
    for (uint32_t x0 = 0; x0 < E; x0 += 32) {
      const uint32_t x = x0 + lane;
      const bool in = x < E;
      const uint32_t en = in ? S.ent[x] : 0u, j = en & 0x3FFFFu, k = (en >> 18) & 255u;
      const ulonglong2 *sj = snap + (size_t)j * np;
      ulonglong2 ra = make_ulonglong2(0, 0), rb = ra;
      if ((en >> 26) & 1u) ra = sj[S.pa[k]];  // (a point's snapshot of word j exists only where its bit is set)
      if ((en >> 27) & 1u) rb = sj[S.pb[k]];
      // coordinates c0..c3 of the rows in a basis b0..b3 of their span (n of them, in order of appearance)
      const uint64_t v0 = ra.x, v1 = ra.y, v2 = rb.x, v3 = rb.y;
      uint32_t span = 1, c0 = 0, c1 = 0, c2 = 0, c3 = 0;  // span: 2^n
      auto fresh = [&]() -> uint32_t {
        span *= 2;
        return span / 2;
      };
      if (v0) c0 = fresh();
      if (v1) c1 = v1 == v0 ? c0 : fresh();
      if (v2) c2 = v2 == v0 ? c0 : v2 == v1 ? c1 : v2 == (v0 ^ v1) ? c0 ^ c1 : fresh();
      if (v3) {
        const uint64_t y = v3 ^ v2;
        c3 = v3 == v0 ? c0 : v3 == v1 ? c1 : v3 == (v0 ^ v1) ? c0 ^ c1 : y == 0 ? c2 : y == v0 ? c2 ^ c0
             : y == v1 ? c2 ^ c1 : y == (v0 ^ v1) ? c2 ^ c0 ^ c1 : fresh();
      }
      const uint32_t nv = span - 1u;
      const uint64_t u = v0 | v1 | v2 | v3;
      const uint32_t nt = (uint32_t)__popcll(u);
      uint32_t both = nv << 16 | nt;  // inclusive scan of (values, targets)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(ALL, both, o);
        if (lane >= (uint32_t)o) both += y;
      }
      const uint32_t iv = both >> 16, it = both & 0xFFFFu;
      const uint32_t hb = H + iv - nv, tb = TG + it - nt;
      if (in && x == S.e0[k]) {
        S.tstart[k] = (uint16_t)min(tb, 0xFFFFu);
        S.vstart[k] = (uint16_t)min(hb, 0xFFFFu);
      }
      __syncwarp();
      if (in) {
        const uint32_t off = tb - S.tstart[k];
        if (hb + nv > kKeyValues || off + nt > 32u || tb + nt > kKeyTargets) {
          over = min(over, k);
        } else {
          uint64_t lut = (uint64_t)c0 << 4;
          lut |= (lut ^ (c1 * 0x11u)) << 8;
          lut |= (lut ^ (c2 * 0x1111u)) << 16;
          lut |= (lut ^ (c3 * 0x11111111ull)) << 32;
          S.lut[x] = lut;
          S.hb[x] = (uint16_t)hb;
          if (nv) {
            const uint64_t b0 = v0 ? v0 : v1 ? v1 : v2 ? v2 : v3;
            S.h[hb] = make_ulonglong2(b0, j);
            if (nv > 1) {
              const uint64_t b1 = c1 == 2u ? v1 : c2 == 2u ? v2 : v3;
              S.h[hb + 1] = make_ulonglong2(b1, j);
              S.h[hb + 2] = make_ulonglong2(b0 ^ b1, j);
              if (nv > 3) {
                const uint64_t b2 = c2 == 4u ? v2 : v3;
                for (uint32_t y = 4; y <= nv; ++y) {
                  const uint64_t v = (y & 1u ? b0 : 0ull) ^ (y & 2u ? b1 : 0ull) ^ (y & 4u ? b2 : 0ull) ^ (y & 8u ? v3 : 0ull);
                  S.h[hb + y - 1u] = make_ulonglong2(v, j);
                }
              }
            }
          }
          uint32_t m0 = 0, m1 = 0, m2 = 0, m3 = 0;
          uint32_t at = 1u << off;
          uint32_t *tg = S.targets + tb;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint32_t w0 = (uint32_t)(v0 >> (32 * half)), w1 = (uint32_t)(v1 >> (32 * half)),
                           w2 = (uint32_t)(v2 >> (32 * half)), w3 = (uint32_t)(v3 >> (32 * half));
            for (uint32_t bits = (uint32_t)(u >> (32 * half)); bits; bits &= bits - 1, at <<= 1) {
              const uint32_t low = bits & (0u - bits);
              *tg++ = j * 64u + (uint32_t)(31 - __clz(low)) + 32u * half;
              if (w0 & low) m0 |= at;
              if (w1 & low) m1 |= at;
              if (w2 & low) m2 |= at;
              if (w3 & low) m3 |= at;
            }
          }
          if (m0) atomicOr(&S.rows[k].x, m0);
          if (m1) atomicOr(&S.rows[k].y, m1);
          if (m2) atomicOr(&S.rows[k].z, m2);
          if (m3) atomicOr(&S.rows[k].w, m3);
        }
      }
      H += __shfl_sync(ALL, iv, 31);
      TG += __shfl_sync(ALL, it, 31);
    }
    over = __reduce_min_sync(ALL, over);
    if (over < take) {  // only the records before it (theirs is all in place)
      const uint32_t beside = side_by_side(d, nrec);
      if (2u * over < beside) {
        postpone(r0 - first, beside);
        r0 += beside;
        continue;
      }
      take = over;
      H = S.vstart[over];
    }
    __syncwarp();
    for (uint32_t y = lane; y < H; y += 32) {
      const ulonglong2 v = S.h[y];
      S.h[y] = word_hash((uint32_t)v.y, v.x);
    }
    // the items of each record
    uint32_t heads = 0;
    if (lane < take) {
      uint64_t z = 0;
      for (uint32_t x = S.e0[lane]; x < S.e1[lane]; ++x) z |= S.lut[x];
      z |= z >> 1;  // zero nibbles, gathered into 16 bits
      z |= z >> 2;
      z = ~z & 0x1111111111111111ull;
      z = (z | z >> 3) & 0x0303030303030303ull;
      z = (z | z >> 6) & 0x000F000F000F000Full;
      z = (z | z >> 12) & 0x000000FF000000FFull;
      const uint32_t zero = (uint32_t)(z | z >> 24) & 0xFFFFu;
      const uint32_t join = joining((uint32_t)(d >> 56) & 15u, zero);
      heads = coset_heads(present, zero, join);
      S.join[lane] = (uint16_t)join;
    }
    uint32_t at = (uint32_t)__popc(heads);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(ALL, at, o);
      if (lane >= (uint32_t)o) at += x;
    }
    take = (uint32_t)__popc(__ballot_sync(ALL, lane < take && at <= kKeyItems));
    const uint32_t items = __shfl_sync(ALL, at, take - 1u);
    at -= (uint32_t)__popc(heads);
    if (lane >= take) heads = 0;
    for (; heads; heads &= heads - 1) S.item[at++] = (uint16_t)(lane << 4 | (__ffs(heads) - 1u));
    __syncwarp();
    for (uint32_t q0 = 0; q0 < items; q0 += 32) {
      const uint32_t q = q0 + lane;
      const bool in = q < items;
      const uint32_t it = in ? S.item[q] : 0u, k = it >> 4, s = it & 15u;
      uint64_t hx = 0, hy = 0;
      if (in) {
        // (s's half of the 16 nibbles)
        const uint32_t *lut = reinterpret_cast<const uint32_t *>(S.lut) + (s >> 3), sh = 4u * (s & 7u);
        for (uint32_t x = S.e0[k], x1 = S.e1[k]; x < x1; ++x) {
          const uint32_t id = (lut[2 * x] >> sh) & 15u;
          if (id) {
            const ulonglong2 h = S.h[S.hb[x] + id - 1u];
            hx ^= h.x;
            hy ^= h.y;
          }
        }
      }
      const uint4 rows = S.rows[k];
      uint32_t t = in ? (s & 1u ? rows.x : 0u) ^ (s & 2u ? rows.y : 0u) ^ (s & 4u ? rows.z : 0u) ^ (s & 8u ? rows.w : 0u) : 0u;
      const uint32_t cnt = (uint32_t)__popc(t);
      const uint32_t *tg = S.targets + S.tstart[k];
      uint32_t l[8] = {};
      if (L.narrow) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (i % 4 == 0 && !__any_sync(ALL, t != 0)) break;
          if (t) {
            l[i / 2] |= tg[__ffs(t) - 1] << (i % 2 * 16);
            t &= t - 1;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i % 4 == 0 && !__any_sync(ALL, t != 0)) break;
          if (t) {
            l[i] = tg[__ffs(t) - 1];
            t &= t - 1;
          }
        }
      }
      if (!in) continue;
      const uint32_t place = (uint32_t)(S.place[k] >> (4u * s)) & 15u, m = S.moff[k] + place;
      if (t) {  // the rest of a long list
        uint32_t *far = L.tl + (size_t)m * L.tstride;
        for (uint32_t i = 0; t; t &= t - 1, ++i)
          if (i < L.tstride) far[i] = tg[__ffs(t) - 1];
      }
      const uint32_t mult = (uint32_t)__popc(xor_bits16(S.join[k], s) & S.present[k]);
      listed += cnt;
      file_item(L, bbase, bbits, tcap, hx, hy, L.keep ? (r0 + k) << 4 | place : m, cnt, mult, repeat_merge(S.p[k], mult), l);
    }
    r0 += take;
  }
  __syncwarp();
  if (__any_sync(ALL, lane < kKeyRecords / 32 && S.late[lane])) listed += key_late_records(L, C, L.first[w], S);
  const uint32_t tot = __reduce_add_sync(ALL, listed);
  if (lane == 0 && tot) red_add(L.list_total, tot);
}

// ---- records of mechanisms (global path, gradients; one circuit) --------------

// Thread per key warp: its first record, the first that starts at or after the warp's first mechanism.
__global__ void key_prep_kernel(KeyLaunch L) {
  const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= L.n_warps) return;
  const uint32_t c = find_circuit(L.kbase, L.n_circ, w);
  const CircuitDev &C = L.circs[c];
  const uint32_t m = (w - L.kbase[c]) * L.chunk;
  uint32_t lo = 0, hi = C.R;  // rec_moff[lo - 1] < m <= rec_moff[hi]
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(C.rec_moff + mid) < m) lo = mid + 1;
    else hi = mid;
  }
  L.first[w] = lo;
}

// Record of mechanism m (one circuit): a search of rec_moff from the record
// before the first of m's key warp on (each record holds a mechanism at least,
// so m's record lies within the warp's mechanisms of it).
__device__ __forceinline__ uint32_t record_of(const uint32_t *first, uint32_t chunk, const uint32_t *rec_moff, uint32_t R,
                                              uint32_t m) {
  const uint32_t f = first[m / chunk];
  uint32_t lo = f ? f - 1u : 0u;
  uint32_t hi = min(R, lo + chunk + 2u);
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(rec_moff + mid) <= m) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Global path: every mechanism's descriptor, probability and 128-bit key, a thread each.
__global__ void __launch_bounds__(KEY_THREADS) key_all_kernel(KeyLaunch L) {
  const uint32_t m = blockIdx.x * KEY_THREADS + threadIdx.x;
  if (m >= L.M) return;
  const CircuitDev &C = L.circs[0];
  const uint32_t r = record_of(L.first, L.chunk, C.rec_moff, C.R, m);
  const uint64_t d = __ldg(C.rec + r);
  const uint32_t type = (uint32_t)((d >> 56) & 15u);
  const uint32_t comp = type == 0 ? (uint32_t)(d >> 60) & 15u : kComp[type][m - __ldg(C.rec_moff + r)];
  uint32_t pa = (uint32_t)(d & 0x0FFFFFFFu), pb = (uint32_t)((d >> 28) & 0x0FFFFFFFu);
  uint32_t Pa = comp & 3u, Pb = comp >> 2;
  if (Pa == 0) {  // a component on point b only is stored with b as its first point
    pa = pb;
    Pa = Pb;
    Pb = 0;
  }
  if (Pb == 0) pb = 0;
  C.mdesc[m] = mk_desc(pa, Pa, pb, Pb);
  C.mp[m] = __ldg(C.rec_p + r);
  uint64_t hx = 0, hy = 0;
  bool nonzero = false;
  const uint32_t np = C.npoints, mw = C.mw;
  const unsigned long long *ma = C.nzm + (size_t)pa * mw, *mb = C.nzm + (size_t)pb * mw;
  for (uint32_t i = 0; i < mw; ++i) {
    // a point's snapshot of word j exists only where its own bit is set
    const uint64_t ba = __ldg(ma + i), bb = Pb ? __ldg(mb + i) : 0ull;
    for (uint64_t bits = ba | bb; bits; bits &= bits - 1) {
      const uint32_t bit = (uint32_t)(__ffsll((long long)bits) - 1);
      const uint32_t j = i * 64u + bit;
      const ulonglong2 *sj = C.snap + (size_t)j * np;
      uint64_t v = 0;
      if ((ba >> bit) & 1ull) v = pauli_sel(sj[pa], Pa);
      if ((bb >> bit) & 1ull) v ^= pauli_sel(sj[pb], Pb);
      if (!v) continue;
      nonzero = true;
      const ulonglong2 h = word_hash(j, v);
      hx ^= h.x;
      hy ^= h.y;
    }
  }
  L.key[m] = make_ulonglong2(hx, hy);
  if (nonzero && (hx | hy) == 0) atomicOr(L.err, DEV_ERR_COLLISION);  // a non-empty symptom hashed to 0
}

// ---- onesweep radix sort ----------------------------------------------------

// Key i of a sort: every `stride`-th u64 (2: the first halves of 128-bit keys).
__global__ void sort_hist_kernel(const uint64_t *__restrict__ keys, uint32_t stride, uint32_t n, uint32_t shift0,
                                 uint32_t passes, uint32_t *__restrict__ hist) {
  __shared__ uint32_t h[8][RADIX];
  for (uint32_t i = threadIdx.x; i < 8 * RADIX; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint64_t k = keys[(size_t)i * stride] >> shift0;
    for (uint32_t p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (p * RADIX_BITS)) & (RADIX - 1)], 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < passes * RADIX; i += blockDim.x) {
    const uint32_t v = (&h[0][0])[i];
    if (v) atomicAdd(hist + i, v);
  }
}

constexpr uint32_t ST_AGG = 1u << 30;     // tile aggregate published
constexpr uint32_t ST_PREFIX = 2u << 30;  // inclusive prefix published
constexpr uint32_t ST_MASK = (1u << 30) - 1;

// One digit of a sort.  vin null: the values are the keys' indices (a sort's first pass), and the
// keys are every `stride`-th u64.
// Bound by the look-back's latency (118k items are 58 tiles, all resident at once, and a pass moves
// 2.8 MB): a thread loads the status of kLook predecessors before it uses any, so a chain of tiles
// whose counts are published costs one round trip per kLook tiles (10.1 -> 6.8 us a pass; 32 at a time
// and tiles of 512 or 1,024 items: 10-11 us; of 4,096: 8.0).  Each block scans the pass's histogram
// itself, while its keys are on the way (a launch of its own for that: 2.5 us).
constexpr int kLook = 8;
__global__ void __launch_bounds__(SORT_THREADS) sort_pass_kernel(
    const uint64_t *__restrict__ kin, uint32_t stride, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
    uint32_t *__restrict__ vout, uint32_t n, uint32_t shift, const uint32_t *__restrict__ hist,
    uint32_t *__restrict__ status, uint32_t *__restrict__ tile_ctr, uint32_t *__restrict__ err,
    unsigned long long spin_ns, uint32_t hold_tile0) {
  constexpr int WARPS = SORT_THREADS / 32;
  __shared__ uint32_t wcount[WARPS][RADIX];
  __shared__ uint32_t dbase[RADIX];
  __shared__ uint32_t s_wtot[RADIX / 32];  // each digit warp's share of the histogram
  __shared__ uint32_t s_tile;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < WARPS * RADIX; i += SORT_THREADS) (&wcount[0][0])[i] = 0;
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1u);
  uint32_t gofs = 0;  // the digit's first position: a scan of the pass's histogram, each block its own
  if (threadIdx.x < RADIX) {
    const uint32_t own = hist[threadIdx.x];
    gofs = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, gofs, o);
      if (lane >= (uint32_t)o) gofs += v;
    }
    if (lane == 31) s_wtot[warp] = gofs;
    gofs -= own;
  }
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t base = tile * SORT_TILE + warp * (32 * SORT_IPT) + lane;

  uint64_t key[SORT_IPT];
  uint32_t val[SORT_IPT];
  uint32_t dig[SORT_IPT];
  uint32_t rank[SORT_IPT];
#pragma unroll
  for (int k = 0; k < SORT_IPT; ++k) {
    const uint32_t idx = base + k * 32;
    if (idx < n) {
      key[k] = kin[(size_t)idx * stride];
      val[k] = vin ? vin[idx] : idx;
      dig[k] = (uint32_t)(key[k] >> shift) & (RADIX - 1);
    } else {
      key[k] = 0;
      val[k] = 0;
      dig[k] = RADIX;  // not counted
    }
  }
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < SORT_IPT; ++k) {
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, dig[k]);
    const uint32_t leader = __ffs(peers) - 1u;
    uint32_t b = 0;
    if (dig[k] < RADIX) b = wcount[warp][dig[k]];
    rank[k] = b + __popc(peers & lt);
    __syncwarp();
    if (lane == leader && dig[k] < RADIX) wcount[warp][dig[k]] = b + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive scan over warps, tile count, look-back
  if (threadIdx.x < RADIX) {
    const uint32_t d = threadIdx.x;
    for (uint32_t v = 0; v < warp; ++v) gofs += s_wtot[v];
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t c = wcount[w][d];
      wcount[w][d] = sum;
      sum += c;
    }
    volatile uint32_t *st = status;
    if (tile == 0) {
      if (!hold_tile0) st[d] = ST_PREFIX | sum;  // (held: a test of the waits below)
      dbase[d] = gofs;
    } else {
      st[(size_t)tile * RADIX + d] = ST_AGG | sum;
      uint32_t excl = 0;
      int32_t t = (int32_t)tile - 1;
      unsigned long long t0 = 0;
      bool found = false;
      while (t >= 0 && !found) {
        uint32_t s[kLook];
#pragma unroll
        for (int k = 0; k < kLook; ++k) s[k] = t >= k ? st[(size_t)(t - k) * RADIX + d] : 0u;
        int used = 0;
#pragma unroll
        for (int k = 0; k < kLook; ++k) {
          if (used == k && !found && (s[k] & ~ST_MASK) != 0) {
            excl += s[k] & ST_MASK;
            found = (s[k] & ST_PREFIX) != 0;
            used = k + 1;
          }
        }
        t -= used;
        if (used) {
          t0 = 0;
        } else if (t0 == 0) {
          t0 = globaltimer();
        } else if (globaltimer() - t0 > spin_ns) {
          atomicOr(err, DEV_ERR_TIMEOUT);
          break;
        }
      }
      // (no fence: the status word is all that is passed on)
      st[(size_t)tile * RADIX + d] = ST_PREFIX | (excl + sum);
      dbase[d] = gofs + excl;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < SORT_IPT; ++k) {
    if (dig[k] < RADIX) {
      const uint32_t pos = dbase[dig[k]] + wcount[warp][dig[k]] + rank[k];
      if (pos < n) {  // always true unless a look-back wait timed out
        kout[pos] = key[k];
        vout[pos] = val[k];
      }
    }
  }
}

__global__ void gather_hi_kernel(const ulonglong2 *__restrict__ key, const uint32_t *__restrict__ perm,
                                 uint64_t *__restrict__ out, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = perm[i] < n ? key[perm[i]].y : 0ull;  // (an index past n: a sort pass timed out)
}

// ---- merge ------------------------------------------------------------------

constexpr unsigned long long MS_AGG = 1ull << 62;
constexpr unsigned long long MS_PREFIX = 2ull << 62;

__device__ __forceinline__ unsigned long long ms_pack(uint32_t cnt, uint32_t tg) {
  return ((unsigned long long)(cnt & 0x3FFFFFFFu) << 32) | tg;
}

// Warp 0 resolves the exclusive prefix of tile `tile` over tiles [0, tile)
// by decoupled look-back, kWide predecessors a lane and step, after the tile
// published its (count, targets) aggregate with publish_aggregate.  Returns
// the prefix in every lane.
constexpr int kWide = 4;

__device__ __forceinline__ void publish_aggregate(unsigned long long *status, uint32_t tile, uint32_t agg_c,
                                                  uint32_t agg_t) {
  *(volatile unsigned long long *)(status + tile) = (tile == 0 ? MS_PREFIX : MS_AGG) | ms_pack(agg_c, agg_t);
}

__device__ __forceinline__ void warp_lookback(unsigned long long *status, uint32_t tile, uint32_t agg_c,
                                              uint32_t agg_t, uint32_t *err, unsigned long long spin_ns,
                                              uint32_t *pre_c, uint32_t *pre_t) {
  const uint32_t lane = threadIdx.x & 31u;
  volatile unsigned long long *st = status;
  uint32_t ec = 0, et = 0;
  int32_t base = (int32_t)tile - 1;
  unsigned long long t0 = 0;
  bool done = base < 0;
  while (!done) {
    unsigned long long s[kWide];
#pragma unroll
    for (int k = 0; k < kWide; ++k) {
      const int32_t idx = base - k * 32 - (int32_t)lane;
      s[k] = idx >= 0 ? st[idx] : (MS_PREFIX | 0ull);
    }
    uint32_t c = 0, t = 0;
    int used = 0;
#pragma unroll
    for (int k = 0; k < kWide; ++k) {
      const uint32_t flag = (uint32_t)(s[k] >> 62);
      const uint32_t ready = __ballot_sync(0xFFFFFFFFu, flag != 0);
      const uint32_t pref = __ballot_sync(0xFFFFFFFFu, flag == 2u);
      // lanes up to (and including) the nearest prefix must all be ready
      const uint32_t need = pref ? ((pref & (0u - pref)) << 1) - 1u : 0xFFFFFFFFu;
      if (used == k && !done && (ready & need) == need) {
        used = k + 1;
        done = pref != 0;
        if ((need >> lane) & 1u) {
          c += (uint32_t)((s[k] >> 32) & 0x3FFFFFFFu);
          t += (uint32_t)s[k];
        }
      }
    }
    if (used == 0) {
      if (t0 == 0) t0 = globaltimer();
      else if (globaltimer() - t0 > spin_ns) {
        if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
        break;
      }
      continue;
    }
    t0 = 0;
    ec += c;
    et += t;
    base -= used * 32;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ec += __shfl_xor_sync(0xFFFFFFFFu, ec, o);
    et += __shfl_xor_sync(0xFFFFFFFFu, et, o);
  }
  // (no fence: the word is all that is passed on)
  if (lane == 0 && tile != 0) st[tile] = MS_PREFIX | ms_pack(ec + agg_c, et + agg_t);
  *pre_c = ec;
  *pre_t = et;
}

// A mechanism's points, and mask word i of the words where each of them has a snapshot (a word whose bit is
// clear has none stored: its rows were zero there).
struct SymptomMask {
  uint64_t a = 0, b = 0;  // of the first and the second point
};
__device__ __forceinline__ SymptomMask symptom_mask(const CircuitDev &C, uint64_t d, uint32_t i) {
  const uint32_t pa = (uint32_t)(d & 0x3FFFFFFFu), Pa = (uint32_t)((d >> 30) & 3u);
  const uint32_t pb = (uint32_t)((d >> 32) & 0x3FFFFFFFu), Pb = (uint32_t)(d >> 62);
  SymptomMask m;
  if (Pa) m.a = __ldg(C.nzm + (size_t)pa * C.mw + i);
  if (Pb) m.b = __ldg(C.nzm + (size_t)pb * C.mw + i);
  return m;
}

// Word j of mechanism descriptor d (bit j % 64 of the mask words m).
__device__ __forceinline__ uint64_t symptom_word(const CircuitDev &C, uint64_t d, uint32_t j, const SymptomMask &m) {
  const ulonglong2 *sj = C.snap + (size_t)j * C.npoints;
  uint64_t v = 0;
  if ((m.a >> (j & 63u)) & 1ull) v = pauli_sel(sj[d & 0x3FFFFFFFu], (uint32_t)((d >> 30) & 3u));
  if ((m.b >> (j & 63u)) & 1ull) v ^= pauli_sel(sj[(d >> 32) & 0x3FFFFFFFu], (uint32_t)(d >> 62));
  return v;
}

// One thread per sorted position; one warp folds the tile's runs.  FP64 runs at 2 lanes a cycle and SM,
// so lanes that fold nothing new are what a fold must avoid: with 8 positions a lane and then a segmented
// scan over the lanes, a tile of 256 costs 13 warp-wide merges (every warp scanning its 32 positions: 40,
// and the carries as many again).  A run still open at its tile's end is read on by the block,
// MERGE_THREADS positions at a time, and folded by the same warp; the tile's counts are published before
// that and its predecessors' read after, 128 a step.  118k mechanisms in runs of 300: 26 -> 15.6 us
// (one thread following its run alone: 503).  What is left is a chain of ~10 dependent loads (4.5k
// cycles to the keys and symptoms, 4k in the open run, 3k in the look-back).  The tree is deterministic
// and differs from a left-to-right fold by a few ulps.
__global__ void __launch_bounds__(MERGE_THREADS) merge_kernel(MergeLaunch L) {
  constexpr uint32_t NW = MERGE_THREADS / 32;
  const CircuitDev C = *L.c_dev;
  __shared__ uint32_t s_tile;
  __shared__ uint32_t wsum_c[MERGE_THREADS / 32], wsum_t[MERGE_THREADS / 32];
  __shared__ uint32_t s_pre_c, s_pre_t;
  constexpr uint32_t FP = MERGE_THREADS / 32;   // positions a lane of the folding warp takes
  __shared__ double s_q[32 * (FP + 1)];         // the positions' probabilities, a padded row per folding lane
  __shared__ double s_p[MERGE_THREADS];         // folded probability of the run that starts at a position
  __shared__ uint32_t s_head[NW];               // where runs start, a bit per position
  __shared__ ulonglong2 s_key;                  // the key of the run open at the tile's end
  __shared__ uint32_t s_open;                   // its first position in the tile (MERGE_THREADS: none follows)
  if (threadIdx.x == 0) s_tile = atomicAdd(L.tile_ctr, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t i = tile * MERGE_THREADS + threadIdx.x;
  const uint32_t n = L.n;
  const uint32_t ntiles = (n + MERGE_THREADS - 1) / MERGE_THREADS;

  bool head = false, newgroup = true;
  uint32_t ntg = 0, m = 0;
  double q = 0.0;  // (0 leaves a run as it is)
  ulonglong2 k = make_ulonglong2(0, 0);
  // After a sort pass timed out (DEV_ERR_TIMEOUT, the compile fails) the
  // permutation may hold stale entries: an index past n is never followed.
  m = i < n ? L.perm[i] : 0u;
  if (i < n && m >= n) {
    atomicOr(L.err, DEV_ERR_TIMEOUT);
    m = 0;
  } else if (i < n) {
    k = L.key[m];
    q = __ldg(C.mp + m);
    const uint64_t d = __ldg(C.mdesc + m);
    const uint32_t mp = i > 0 ? L.perm[i - 1] : n;
    uint64_t dp = 0;
    if (mp < n) {
      const ulonglong2 kp = L.key[mp];
      dp = __ldg(C.mdesc + mp);
      newgroup = kp.x != k.x || kp.y != k.y;
      if (newgroup && ((L.sortkey[i] ^ L.sortkey[i - 1]) & L.sort_mask) == 0 && L.sort_mask) atomicOr(L.err, DEV_FLAG_MIXED);
    }
    // One loop for both kinds of position, two words at a time: a head counts its targets, another one's
    // full symptom is compared with its predecessor's on the words either can be non-zero in.
    bool diff = false;
    for (uint32_t mi = 0; mi < C.mw; ++mi) {
      const SymptomMask ma = symptom_mask(C, d, mi), mb = newgroup ? SymptomMask{} : symptom_mask(C, dp, mi);
      for (uint64_t bits = ma.a | ma.b | mb.a | mb.b; bits;) {
        const uint32_t j0 = mi * 64u + (uint32_t)(__ffsll((long long)bits) - 1);
        bits &= bits - 1;
        const bool two = bits != 0;
        const uint32_t j1 = two ? mi * 64u + (uint32_t)(__ffsll((long long)bits) - 1) : j0;
        bits &= bits - 1;
        const uint64_t a0 = symptom_word(C, d, j0, ma), a1 = two ? symptom_word(C, d, j1, ma) : 0ull;
        if (newgroup) {
          ntg += __popcll(a0) + __popcll(a1);
        } else {
          const uint64_t b0 = symptom_word(C, dp, j0, mb), b1 = two ? symptom_word(C, dp, j1, mb) : 0ull;
          diff |= a0 != b0 || a1 != b1;
        }
      }
    }
    const bool empty = (k.x | k.y) == 0;
    // (a non-empty symptom hashed to zero is a collision too)
    if (diff || (newgroup && empty && ntg)) atomicOr(L.err, DEV_ERR_COLLISION);
    head = newgroup && !empty;
    if (!head) ntg = 0;
  }
  // block-wide exclusive scan of (head, ntg)
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t c_in = head ? 1u : 0u, t_in = ntg;
  uint32_t c_inc = c_in, t_inc = t_in;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, c_inc, off), b = __shfl_up_sync(0xFFFFFFFFu, t_inc, off);
    if (lane >= (uint32_t)off) {
      c_inc += a;
      t_inc += b;
    }
  }
  if (lane == 31) {
    wsum_c[warp] = c_inc;
    wsum_t[warp] = t_inc;
  }
  const uint32_t qi = threadIdx.x / FP * (FP + 1) + threadIdx.x % FP;
  s_q[qi] = q;
  const uint32_t hb = __ballot_sync(0xFFFFFFFFu, newgroup);
  if (lane == 0) s_head[warp] = hb;
  if (threadIdx.x == MERGE_THREADS - 1) s_key = k;
  __syncthreads();
  uint32_t agg_c = 0, agg_t = 0;  // the tile's, in warp 0
  if (threadIdx.x < 32) {
    const uint32_t wc = lane < NW ? wsum_c[lane] : 0u, wt = lane < NW ? wsum_t[lane] : 0u;
    uint32_t ec = wc, et = wt;
#pragma unroll
    for (uint32_t o = 1; o < NW; o <<= 1) {
      const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, ec, o), b = __shfl_up_sync(0xFFFFFFFFu, et, o);
      if (lane >= o) {
        ec += a;
        et += b;
      }
    }
    const uint32_t ac = __shfl_sync(0xFFFFFFFFu, ec, NW - 1), at = __shfl_sync(0xFFFFFFFFu, et, NW - 1);
    if (lane < NW) {
      wsum_c[lane] = ec - wc;
      wsum_t[lane] = et - wt;
    }
    if (lane == 0) publish_aggregate(L.status, tile, ac, at);
    agg_c = ac;
    agg_t = at;
  } else if (warp == 1) {
    // lane l folds positions [FP l, FP l + FP); a run that starts there goes on over the lanes after
    const uint32_t h = (s_head[lane * FP / 32] >> (lane * FP % 32)) & ((1u << FP) - 1u);
    double acc = 0.0, lead = 0.0;  // the run open after the lane's positions; what precedes its first start
    uint32_t cur = MERGE_THREADS;
#pragma unroll
    for (uint32_t e = 0; e < FP; ++e) {
      const double v = s_q[lane * (FP + 1) + e];
      if ((h >> e) & 1u) {
        if (cur < MERGE_THREADS) s_p[cur] = acc;
        else lead = acc;
        cur = lane * FP + e;
        acc = v;
      } else {
        acc = xor_merge(acc, v);
      }
    }
    const uint32_t starts = __ballot_sync(0xFFFFFFFFu, h != 0);
    // x: the fold from the lane's first position to the next start
    const uint32_t stop = starts >> lane ? lane + (uint32_t)__ffs((int)(starts >> lane)) - 1u : 31u;
    double x = h ? lead : acc;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const double y = __shfl_down_sync(0xFFFFFFFFu, x, o);
      if (lane + o <= stop) x = xor_merge(x, y);
    }
    const double y = __shfl_down_sync(0xFFFFFFFFu, x, 1);
    if (h) s_p[cur] = lane == 31 ? acc : xor_merge(acc, y);
    const uint32_t last = starts ? 31u - (uint32_t)__clz((int)starts) : 0u;  // the lane of the tile's last start
    if (lane == last) {
      const bool full = (uint64_t)(tile + 1) * MERGE_THREADS <= n;
      s_open = h && full && (s_key.x | s_key.y) != 0 ? cur : MERGE_THREADS;
    }
  }
  __syncthreads();
  // A run still open at the tile's end: the block reads its positions in the tiles after, warp 1 folds them.
  if (s_open < MERGE_THREADS) {
    const ulonglong2 ko = s_key;
    double acc = 0.0;
    uint32_t i2 = (tile + 1) * MERGE_THREADS + threadIdx.x;
    for (uint32_t m2 = i2 < n ? L.perm[i2] : n;;) {
      double q2 = 0.0;
      bool same = false;
      i2 += MERGE_THREADS;
      const uint32_t next = i2 < n ? L.perm[i2] : n;
      if (m2 < n) {  // (past n: the end, or a stale entry after a timed-out sort pass)
        const ulonglong2 k2 = L.key[m2];
        const double p2 = __ldg(C.mp + m2);
        same = k2.x == ko.x && k2.y == ko.y;
        if (same) q2 = p2;
      }
      m2 = next;
      s_q[qi] = q2;
      const int all = __syncthreads_and(same ? 1 : 0);
      if (warp == 1) {
#pragma unroll
        for (uint32_t e = 0; e < FP; ++e) acc = xor_merge(acc, s_q[lane * (FP + 1) + e]);
      }
      if (!all) break;
      __syncthreads();
    }
    if (warp == 1) {
#pragma unroll
      for (uint32_t o = 16; o > 0; o >>= 1) acc = xor_merge(acc, __shfl_down_sync(0xFFFFFFFFu, acc, o));
      if (lane == 0) s_p[s_open] = xor_merge(s_p[s_open], acc);
    }
  }
  // (the predecessors' aggregates are published by now)
  if (threadIdx.x < 32) {
    uint32_t pc = 0, pt = 0;
    warp_lookback(L.status, tile, agg_c, agg_t, L.err, L.spin_ns, &pc, &pt);
    if (lane == 0) {
      s_pre_c = pc;
      s_pre_t = pt;
      if (tile == ntiles - 1) {
        L.totals[0] = pc + agg_c;
        L.totals[1] = pt + agg_t;
        if (pc + agg_c <= n) L.out_off[pc + agg_c] = pt + agg_t;  // the closing offset (past n only after a timed-out look-back)
        if (pt + agg_t > L.tg_cap) atomicOr(L.err, DEV_FLAG_TG_OVF);
      }
    }
  }
  __syncthreads();
  if (!head) return;
  const uint32_t slot = s_pre_c + wsum_c[warp] + c_inc - c_in;
  if (slot >= n) return;  // only after a timed-out look-back
  const uint32_t toff = s_pre_t + wsum_t[warp] + t_inc - t_in;
  const double p = s_p[threadIdx.x];
  L.out_prob[slot] = p;
  L.out_off[slot] = toff;
  if ((uint64_t)toff + ntg <= L.tg_cap) {
    const uint64_t d = __ldg(C.mdesc + m);
    uint32_t o = toff;
    for (uint32_t mi = 0; mi < C.mw; ++mi) {  // the masked words, ascending: the targets stay ascending
      const SymptomMask mk = symptom_mask(C, d, mi);
      for (uint64_t bits = mk.a | mk.b; bits; bits &= bits - 1) {
        const uint32_t j = mi * 64u + (uint32_t)(__ffsll((long long)bits) - 1);
        uint64_t v = symptom_word(C, d, j, mk);
        while (v) {
          L.out_tg[o++] = j * 64u + (uint32_t)(__ffsll((long long)v) - 1);
          v &= v - 1;
        }
      }
    }
  }
}

// ---- merge of the compile pipeline ---------------------------------------

// Buckets per block (one warp each) of grouping, emission and their adjoint: a block holds its shared memory
// until its slowest warp is done, so small blocks keep more warps running (8 -> 4, grouping: 32 mixed surface
// codes 145 -> 138 us, d = 25 39 -> 36; adjoint of [[144,12,12]] 17 -> 14.6; 2: the same).
constexpr uint32_t GW_WARPS = 4;

// Row of an item's later targets: its first mechanism.
__device__ __forceinline__ const uint32_t *far_targets(const GroupLaunch &L, uint32_t m) {
  if (L.keep) m = __ldg(L.rec_moff + (m >> 4)) + (m & 15u);
  return L.tl + (size_t)m * L.tstride;
}

// The targets of two items: the slots' first ones as two 16-byte words (unused
// entries are zero), the rest of longer lists from their rows.
__device__ __forceinline__ bool slot_lists_equal(const GroupLaunch &L, const Slot *a, uint32_t ma, const Slot *b,
                                                 uint32_t mb, uint32_t n) {
  const uint4 *va = reinterpret_cast<const uint4 *>(a->list), *vb = reinterpret_cast<const uint4 *>(b->list);
  const uint4 x0 = va[0], y0 = vb[0], x1 = va[1], y1 = vb[1];
  if ((x0.x ^ y0.x) | (x0.y ^ y0.y) | (x0.z ^ y0.z) | (x0.w ^ y0.w) | (x1.x ^ y1.x) | (x1.y ^ y1.y) | (x1.z ^ y1.z) |
      (x1.w ^ y1.w))
    return false;
  const uint32_t inl = L.narrow ? 16u : 8u;
  return n <= inl || lists_equal(far_targets(L, ma), far_targets(L, mb), n - inl);
}

// A bucket's groups in its slots.  A group's record: (head mechanism, targets
// before it in the bucket << 8 | the head's slot) in the tail of slot g, its
// probability beside it (every slot of the bucket has been read into shared
// memory, and no list is written over).
struct SlotRuns {
  const GroupLaunch &L;
  Slot *bslot;
  const uint32_t *m;
  __device__ __forceinline__ uint32_t count(uint32_t t) const { return t & kSlotCount; }
  __device__ __forceinline__ bool equal(uint32_t a, uint32_t b, uint32_t n) const {
    return slot_lists_equal(L, bslot + a, m[a], bslot + b, m[b], n);
  }
  __device__ __forceinline__ void group(uint32_t g, uint32_t head, uint32_t before, uint32_t s) const {
    *reinterpret_cast<uint2 *>(&bslot[g].tail) = make_uint2(m[head], before << 8 | head);
    if (L.keep) slot_perm(bslot, g)[1] = s;
  }
  __device__ __forceinline__ void prob(uint32_t g, double p) const { bslot[g].tail.p = p; }
};

// One warp's bucket of n <= CAP items.  Returns (groups, targets).
template <uint32_t CAP>
__device__ __forceinline__ uint2 group_warp(const GroupLaunch &L, GroupItems<CAP> &G, uint32_t b, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  Slot *const bslot = L.slot + (size_t)b * SLOT_CAP;
  for (uint32_t i = lane; i < n; i += 32) {
    const ulonglong2 k = bslot[i].key;
    const SlotTail t = bslot[i].tail;
    G.key[i] = k;
    G.m[i] = t.m;
    G.t[i] = t.t;
    G.p[i] = t.p;
  }
  __syncwarp();
  if constexpr (CAP > 128) {
    order_items<CAP / 32, true>(G, n);
  } else {
    if (n <= 32) order_items<1, true>(G, n);
    else if (n <= 64) order_items<2, true>(G, n);
    else order_items<4, true>(G, n);
  }
  if (L.keep) {  // the saved permutation for the adjoint
    for (uint32_t s = lane; s < n; s += 32) {
      slot_perm(bslot, s)[0] = G.m[G.ord[s]];
      slot_perm(bslot, s)[3] = G.t[G.ord[s]] >> 24;  // the mechanisms merged into the item
    }
  }
  return fold_runs(G, n, L.tcap, L.err, SlotRuns{L, bslot, G.m});
}

// One warp per bucket.  A bucket of more than WARP_CAP items (repeated symptoms)
// is left to the block's last warp to finish, which then has the block's
// shared memory to itself; no warp waits for another.
// Bound by latency and instructions (a warp's chain is two DRAM round trips,
// the sort and the scan; the FP64 pipe is a third busy).  Ordering by a sort of
// 32-bit words took the place of a counting sort into 64 sub-bins with a rank
// inside each: 32 mixed surface codes (94k buckets of ~30 items) 153 -> 145 us,
// and the launch for large buckets is gone ([[144,12,12]]: grouping, scan and
// emission 23.9 -> 19.2 us).  A block barrier before the large buckets cost
// 13 us of 158.
__global__ void __launch_bounds__(GW_WARPS * 32) group_kernel(const __grid_constant__ GroupLaunch L) {
  __shared__ union Shared {
    GroupItems<WARP_CAP> w[GW_WARPS];
    GroupItems<SLOT_CAP> all;
    __device__ Shared() {}
  } S;
  __shared__ uint32_t s_done;
  if (threadIdx.x == 0) s_done = 0;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u, wi = threadIdx.x >> 5;
  const uint32_t b0 = blockIdx.x * GW_WARPS, b = b0 + wi;
  const uint32_t n = b < L.nb ? bucket_items(L.count[b]) : 0u;
  auto put = [&](uint32_t bucket, uint2 a, uint32_t items) {
    if (lane != 0) return;
    L.bagg[bucket] = a;
    if (a.x == 0) return;
    red_add(&L.tsum[bucket / SCAN_TILE].x, a.x);
    red_add(&L.tsum[bucket / SCAN_TILE].y, a.y);
    red_add(L.totals + 3, items);
  };
  // (a bucket past SLOT_CAP items overflowed: flagged by the key pass, the run is redone another way)
  const bool big = n > WARP_CAP && n <= SLOT_CAP;
  if (b < L.nb && !big) {
    uint2 agg = make_uint2(0, 0);
    if (n && n <= WARP_CAP) agg = group_warp(L, S.w[wi], b, n);
    put(b, agg, n);
  }
  __syncwarp();
  uint32_t done = 0;
  if (lane == 0) {
    __threadfence_block();
    done = atomicAdd(&s_done, big ? 0x101u : 1u) + (big ? 0x101u : 1u);
  }
  done = __shfl_sync(0xFFFFFFFFu, done, 0);
  if ((done & 255u) < GW_WARPS || (done >> 8) == 0) return;
  __threadfence_block();
  for (uint32_t k = 0; k < GW_WARPS && b0 + k < L.nb; ++k) {
    const uint32_t nk = bucket_items(L.count[b0 + k]);
    if (nk <= WARP_CAP || nk > SLOT_CAP) continue;
    const uint2 a = group_warp(L, S.all, b0 + k, nk);
    put(b0 + k, a, nk);
    __syncwarp();
  }
}

// Exclusive scan of the bucket aggregates: block t covers buckets
// [t * SCAN_TILE, (t + 1) * SCAN_TILE) and starts from the sum of the tile
// sums before it.  The aggregates go through shared memory both ways, so the
// block's global loads and stores are coalesced while each thread scans
// SCAN_TILE / SCAN_THREADS consecutive ones.  The last block writes the totals.
__global__ void __launch_bounds__(SCAN_THREADS) group_scan_kernel(GroupLaunch L) {
  constexpr uint32_t PER = SCAN_TILE / SCAN_THREADS, NW = SCAN_THREADS / 32;
  __shared__ uint2 stage[SCAN_TILE];
  __shared__ uint2 red[NW], wsum[NW];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint32_t tile = blockIdx.x;
  const size_t b0 = (size_t)tile * SCAN_TILE;
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    const size_t i = b0 + (size_t)k * SCAN_THREADS + t;
    stage[k * SCAN_THREADS + t] = i < L.nb ? L.bagg[i] : make_uint2(0, 0);
  }
  uint2 pre = make_uint2(0, 0);
  for (uint32_t k = t; k < tile; k += SCAN_THREADS) {
    const uint2 a = L.tsum[k];
    pre.x += a.x;
    pre.y += a.y;
  }
  pre.x = __reduce_add_sync(0xFFFFFFFFu, pre.x);
  pre.y = __reduce_add_sync(0xFFFFFFFFu, pre.y);
  if (lane == 0) red[warp] = pre;
  __syncthreads();  // (also: the staged aggregates are visible)
  pre = make_uint2(0, 0);
#pragma unroll
  for (uint32_t w = 0; w < NW; ++w) {
    pre.x += red[w].x;
    pre.y += red[w].y;
  }
  uint2 v[PER];
  uint2 loc = make_uint2(0, 0);
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    v[k] = stage[t * PER + k];
    loc.x += v[k].x;
    loc.y += v[k].y;
  }
  // exclusive scan of loc over the block
  uint2 inc = loc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t ax = __shfl_up_sync(0xFFFFFFFFu, inc.x, o), ay = __shfl_up_sync(0xFFFFFFFFu, inc.y, o);
    if (lane >= (uint32_t)o) {
      inc.x += ax;
      inc.y += ay;
    }
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint2 run = make_uint2(pre.x + inc.x - loc.x, pre.y + inc.y - loc.y);
  for (uint32_t w = 0; w < warp; ++w) {
    run.x += wsum[w].x;
    run.y += wsum[w].y;
  }
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    stage[t * PER + k] = run;  // (each thread rewrites only the entries it read)
    run.x += v[k].x;
    run.y += v[k].y;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    const size_t i = b0 + (size_t)k * SCAN_THREADS + t;
    if (i < L.nb) L.bout[i] = stage[k * SCAN_THREADS + t];
  }
  if (tile == gridDim.x - 1 && t == SCAN_THREADS - 1) {
    L.totals[0] = run.x;
    L.totals[1] = run.y;
    L.out_off[run.x] = run.y;  // the closing offset
    if (run.y > L.tg_cap) atomicOr(L.err, DEV_FLAG_TG_OVF);
  }
}

// One warp's bucket: its groups to the DEM arrays from slot `out.x` and target `out.y` on.
__device__ __forceinline__ void emit_bucket(const GroupLaunch &L, uint32_t b, uint2 agg, uint2 out, SlotTail t, SlotTail tn1) {
  const uint32_t lane = threadIdx.x & 31u, tcap = L.tcap;
  const Slot *const bslot = L.slot + (size_t)b * SLOT_CAP;
  for (uint32_t g = lane; g < agg.x; g += 32) {
    if (g != lane) {
      t = bslot[g].tail;
      if (g + 1 < agg.x) tn1 = bslot[g + 1].tail;  // (slot g + 1 <= SLOT_CAP - 1)
    }
    const uint32_t slot = out.x + g, toff = out.y + (t.t >> 8);
    L.out_prob[slot] = t.p;
    L.out_off[slot] = toff;
    // the group's targets run to the next group's (the bucket's total after
    // the last); a list longer than the rows was flagged by the key pass and
    // the run is redone with wider rows, so only the rows' targets are copied
    const uint32_t ntg = min((g + 1 < agg.x ? tn1.t >> 8 : agg.y) - (t.t >> 8), tcap);
    if ((uint64_t)toff + ntg <= L.tg_cap) {
      const uint4 *src = reinterpret_cast<const uint4 *>(bslot[t.t & 255u].list);
      const uint4 x0 = src[0], x1 = src[1];
      const uint32_t l[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
      uint32_t *o = L.out_tg + toff;
      if (L.narrow) {
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k)
          if (k < ntg) o[k] = (l[k / 2] >> (k % 2 * 16)) & 0xFFFFu;
      } else {
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
          if (k < ntg) o[k] = l[k];
      }
      const uint32_t inl = L.narrow ? 16u : 8u;
      if (ntg > inl) {
        const uint32_t *far = far_targets(L, t.m);
        for (uint32_t k = inl; k < ntg; ++k) o[k] = __ldg(far + k - inl);
      }
    }
  }
}

// One warp per bucket: the bucket's groups to the DEM arrays.  FOLD: the blocks
// find their buckets' places themselves (the tile sums before the block's tile
// and the aggregates before it in the tile: a few loads a thread for up to
// kFoldBuckets buckets), which saves a small run the scan kernel; the block of
// a circuit's first bucket writes the circuit's place, the last block the
// totals (a single circuit's to page-locked host memory as well: the copy of
// those 12 bytes that the host waited for cost 5 us of an 85-us run).
template <bool FOLD>
__global__ void __launch_bounds__(GW_WARPS * 32) emit_kernel(const __grid_constant__ GroupLaunch L) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wi = tid >> 5;
  const uint32_t b0 = blockIdx.x * GW_WARPS, b = b0 + wi;
  // the first records load beside the bucket's aggregate and offset (a slot
  // past the groups holds whatever it held: only the ones below agg.x are used)
  SlotTail t{}, tn1{};
  uint2 agg = make_uint2(0, 0), out;
  if (b < L.nb) {
    t = L.slot[(size_t)b * SLOT_CAP + lane].tail;
    tn1 = L.slot[(size_t)b * SLOT_CAP + lane + 1].tail;
    agg = L.bagg[b];
  }
  if constexpr (FOLD) {
    __shared__ uint2 s_sum[GW_WARPS], s_agg[GW_WARPS];
    const uint32_t tile = b0 / SCAN_TILE;
    uint2 pre = make_uint2(0, 0);
    for (uint32_t k = tid; k < tile; k += GW_WARPS * 32) {
      const uint2 a = L.tsum[k];
      pre.x += a.x;
      pre.y += a.y;
    }
    for (uint32_t k = tile * SCAN_TILE + tid; k < b0; k += GW_WARPS * 32) {
      const uint2 a = L.bagg[k];
      pre.x += a.x;
      pre.y += a.y;
    }
    pre.x = __reduce_add_sync(0xFFFFFFFFu, pre.x);
    pre.y = __reduce_add_sync(0xFFFFFFFFu, pre.y);
    if (lane == 0) {
      s_sum[wi] = pre;
      s_agg[wi] = agg;
    }
    __syncthreads();
    out = make_uint2(0, 0);
#pragma unroll
    for (uint32_t k = 0; k < GW_WARPS; ++k) {
      out.x += s_sum[k].x + (k < wi ? s_agg[k].x : 0u);
      out.y += s_sum[k].y + (k < wi ? s_agg[k].y : 0u);
    }
    if (b < L.nb && lane == 0) L.bout[b] = out;
    if (b == L.nb - 1 && lane == 0) {
      const uint2 end = make_uint2(out.x + agg.x, out.y + agg.y);
      L.totals[0] = end.x;
      L.totals[1] = end.y;
      L.out_off[end.x] = end.y;  // the closing offset
      const uint32_t flag = end.y > L.tg_cap ? DEV_FLAG_TG_OVF : 0u;
      if (flag) atomicOr(L.err, flag);
      if (L.host_res) {  // (no kernel after this one sets a flag)
        L.host_res[0] = *(volatile uint32_t *)L.err | flag;
        L.host_res[1] = end.x;
        L.host_res[2] = end.y;
      }
    }
    for (uint32_t c = lane; c < L.n_circ; c += 32)
      if (L.cbbase[c] == b) L.cout[c] = out;
  } else {
    if (blockIdx.x == 0)
      for (uint32_t c = tid; c < L.n_circ; c += GW_WARPS * 32) L.cout[c] = L.bout[L.cbbase[c]];
    out = b < L.nb ? L.bout[b] : make_uint2(0, 0);
  }
  if (b < L.nb) emit_bucket(L, b, agg, out, t, tn1);
}

// ---- noise-rate gradients ---------------------------------------------------

// Channel kind of a record type: 0 X/Y/Z error or measurement flip, 1 DEPOLARIZE1, 2 DEPOLARIZE2.
__device__ __forceinline__ uint32_t channel_kind(uint32_t type) {
  return (type == REC_DEP1_L0 || type == REC_DEP1_L12) ? 1u : type >= REC_DEP2_L0 ? 2u : 0u;
}

__global__ void param_rec_kernel(ParamLaunch L) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L.R) return;
  const uint32_t src = L.rec_src[r];
  if (src >= L.n_src) return;
  L.rec_p[r] = L.qtab[(size_t)src * 3 + channel_kind((uint32_t)((L.rec[r] >> 56) & 15u))];
}

// One warp per bucket, a lane per sorted position.  An item of c mechanisms of
// probability q counts as f^c, f = 1 - 2q, in its run's product; its entry
// (first mechanism) takes the derivative by all c of them, dL/dp_g * c f^(c-1)
// * the run's other items'.  The products before and after an item are
// segmented scans, forward over the chunks of 32 positions and then backward.
// Bound by latency and the FP64 pipe (two multiplications a cycle and SM): with
// a lane per run that walked it, every step of the longest run of 32 took the
// pipe for 16 cycles (43 us on [[144,12,12]] walking in global memory with a
// search of each item's record, 24 in shared memory; now 16).
constexpr uint32_t ADJ_THREADS = 128;
__global__ void __launch_bounds__(GW_WARPS * 32) adjoint_group_kernel(const __grid_constant__ AdjointLaunch A) {
  __shared__ double s_pre[GW_WARPS][SLOT_CAP];
  __shared__ uint32_t s_start[GW_WARPS][SLOT_CAP / 32];  // bit per sorted position: a run starts there
  constexpr uint32_t ALL = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u, wi = threadIdx.x >> 5;
  const uint32_t b = blockIdx.x * GW_WARPS + wi;
  if (b >= A.nb) return;
  const uint32_t n = bucket_items(A.count[b]);
  const uint32_t groups = A.bagg[b].x, out0 = A.bout[b].x;
  if (n == 0 || n > SLOT_CAP) return;
  const Slot *const bslot = A.slot + (size_t)b * SLOT_CAP;
  double *pre = s_pre[wi];
  uint32_t *start = s_start[wi];
  if (lane < SLOT_CAP / 32) start[lane] = 0;
  __syncwarp();
  for (uint32_t k = lane; k < groups; k += 32) {
    const uint32_t s = slot_perm(bslot, k)[1];
    atomicOr(start + s / 32, 1u << (s & 31u));
  }
  __syncwarp();
  // an item's f and count; its power f^c
  auto item = [&](uint32_t s, uint32_t &id, uint32_t &c, double &f) {
    const uint4 w = *reinterpret_cast<const uint4 *>(slot_perm(bslot, s));
    id = w.x;
    c = w.w;
    f = 1.0 - 2.0 * __ldg(A.rec_p + (w.x >> 4));  // (the forward's, from the noise tensor)
  };
  auto power = [&](double f, uint32_t c) {
    double x = c & 1u ? f : 1.0;
    for (uint32_t k = c >> 1; k; k >>= 1) {
      f *= f;
      if (k & 1u) x *= f;
    }
    return x;
  };
  const uint32_t chunks = (n + 31u) / 32u;
  uint32_t id = 0, c = 1, g1 = 0;  // the last chunk's items stay in registers for the way back; g1: runs before the chunk
  double f = 1.0, carry = 1.0;
  for (uint32_t k = 0; k < chunks; ++k) {
    const uint32_t s = k * 32 + lane, hb = start[k];
    const uint32_t le = hb & (ALL >> (31u - lane));
    const uint32_t first = le ? 31u - __clz(le) : 0u;
    id = 0;
    c = 1;
    f = 1.0;
    if (s < n) item(s, id, c, f);
    double x = power(f, c);
    const uint32_t longest = __reduce_max_sync(ALL, lane - first + 1u);
    for (uint32_t o = 1; o < longest; o <<= 1) {
      const double y = __shfl_up_sync(ALL, x, o);
      if (lane >= first + o) x *= y;
    }
    if (le == 0) x *= carry;
    double before = __shfl_up_sync(ALL, x, 1);  // inclusive -> exclusive
    if (lane == 0) before = carry;
    if ((hb >> lane) & 1u) before = 1.0;
    if (s < n) pre[s] = before;
    carry = __shfl_sync(ALL, x, 31);
    if (k + 1 < chunks) g1 += (uint32_t)__popc(hb);
  }
  carry = 1.0;         // product of the items of the chunk after that go on with the open run
  bool open = false;   // the chunk after starts inside a run
  for (uint32_t k = chunks; k-- > 0;) {
    const uint32_t s = k * 32 + lane, hb = start[k];
    if (k + 1 < chunks) {
      id = 0;
      c = 1;
      f = 1.0;
      if (s < n) item(s, id, c, f);
      g1 -= (uint32_t)__popc(hb);
    }
    const uint32_t after = lane == 31u ? 0u : hb >> (lane + 1u);
    const uint32_t end = after ? lane + (uint32_t)__ffs(after) : 32u;  // the run is lanes .. end - 1 of the chunk
    double x = power(f, c);
    const uint32_t longest = __reduce_max_sync(ALL, end - lane);
    for (uint32_t o = 1; o < longest; o <<= 1) {
      const double y = __shfl_down_sync(ALL, x, o);
      if (lane + o < end) x *= y;
    }
    const bool goes_on = end == 32u && open;
    if (goes_on) x *= carry;
    double behind = __shfl_down_sync(ALL, x, 1);
    if (lane == 31) behind = open ? carry : 1.0;
    if (lane + 1u == end && end < 32u) behind = 1.0;
    if (s < n) {
      const uint32_t g = g1 + (uint32_t)__popc(hb & (ALL >> (31u - lane))) - 1u;  // (a run open at the chunk's start: the one before)
      double v = A.grad_out[out0 + g] * pre[s] * behind;
      if (c > 1) v *= (double)c * power(f, c - 1);
      A.gq[__ldg(A.rec_moff + (id >> 4)) + (id & 15u)] = v;
    }
    carry = __shfl_sync(ALL, x, 0);
    open = (hb & 1u) == 0;
  }
}

// One block per source: dL/dnoise[e] = the sum over the source's records of
// (the sum of the record's entries) * the split's slope.  A thread takes every
// ADJ_THREADS-th record, then shuffle trees and the warps in order: a fixed
// order (one thread per source, one record after another: 26 us on
// [[144,12,12]]; a warp per source 10, now 6).
__global__ void __launch_bounds__(ADJ_THREADS) adjoint_source_kernel(const __grid_constant__ AdjointLaunch A) {
  __shared__ double s_sum[ADJ_THREADS / 32];
  const uint32_t lane = threadIdx.x & 31u, e = blockIdx.x;
  double sum = 0.0;
  for (uint32_t k = A.src_off[e] + threadIdx.x, end = A.src_off[e + 1]; k < end; k += ADJ_THREADS) {
    const uint32_t r = A.src_rec[k];
    double q = 0.0;
    for (uint32_t m = A.rec_moff[r], m1 = A.rec_moff[r + 1]; m < m1; ++m) q += A.gq[m];
    sum += q * A.stab[(size_t)e * 3 + channel_kind((uint32_t)((A.rec[r] >> 56) & 15u))];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
  if (lane == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t k = 1; k < ADJ_THREADS / 32; ++k) sum += s_sum[k];
    A.grad_noise[e] = sum;
  }
}

}  // namespace

cudaError_t launch_param_rec(const ParamLaunch &L, cudaStream_t s) {
  if (L.R == 0) return cudaSuccess;
  param_rec_kernel<<<(L.R + 255) / 256, 256, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_adjoint(const AdjointLaunch &A, cudaStream_t s) {
  if (A.nb) adjoint_group_kernel<<<(A.nb + GW_WARPS - 1) / GW_WARPS, GW_WARPS * 32, 0, s>>>(A);
  if (A.n_src) adjoint_source_kernel<<<A.n_src, ADJ_THREADS, 0, s>>>(A);
  return cudaGetLastError();
}

cudaError_t launch_key_prep(const KeyLaunch &L, cudaStream_t s) {
  if (L.M == 0) return cudaSuccess;
  key_prep_kernel<<<(L.n_warps + 127) / 128, 128, 0, s>>>(L);
  return cudaGetLastError();
}

// A warp's steps cost about as much for two two-qubit records as for eight, but
// a small run wants them side by side: as many mechanisms a warp as make one
// wave of warps, 16 to 128.  Measured (16 / 36 / 64 / 128 mechanisms a warp,
// us): [[72,12,6]] at L1 (28k mechanisms) 9.7 / 12 / 17 / 29, [[144,12,12]]
// (164k) 22 / 17.5 / 20 / 29, surface d = 25 (979k) 98 / 59 / 46 / 46, 32 mixed
// surface codes (4.0M) 382 / 212 / 153 / 126.
uint32_t key_chunk(uint64_t mechanisms) {
  const uint64_t wave = 152u * 4u * kKeyWarps;
  return (uint32_t)std::min<uint64_t>(128, std::max<uint64_t>(16, (mechanisms + wave - 1) / wave));
}

cudaError_t launch_keys(const KeyLaunch &L, cudaStream_t s) {
  if (L.M == 0) return cudaSuccess;
  key_items_kernel<<<(L.n_warps + kKeyWarps - 1) / kKeyWarps, kKeyWarps * 32, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_keys_all(const KeyLaunch &L, cudaStream_t s) {
  if (L.M == 0) return cudaSuccess;
  if (L.n_circ != 1) return cudaErrorInvalidValue;
  key_all_kernel<<<(L.M + KEY_THREADS - 1) / KEY_THREADS, KEY_THREADS, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_group(const GroupLaunch &L, cudaStream_t s) {
  if (L.nb == 0) return cudaSuccess;
  group_kernel<<<(L.nb + GW_WARPS - 1) / GW_WARPS, GW_WARPS * 32, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_scan_emit(const GroupLaunch &L, cudaStream_t s) {
  if (L.nb == 0) return cudaSuccess;
  const uint32_t blocks = (L.nb + GW_WARPS - 1) / GW_WARPS;
  if (emit_folds(L.nb)) {
    emit_kernel<true><<<blocks, GW_WARPS * 32, 0, s>>>(L);
  } else {
    group_scan_kernel<<<(L.nb + SCAN_TILE - 1) / SCAN_TILE, SCAN_THREADS, 0, s>>>(L);
    emit_kernel<false><<<blocks, GW_WARPS * 32, 0, s>>>(L);
  }
  return cudaGetLastError();
}

size_t sort_scratch_words(uint32_t n, uint32_t bits) {
  const uint32_t passes = (bits + RADIX_BITS - 1) / RADIX_BITS;
  // hist + status + tile counters, for a 128-bit fallback as well (2 sorts)
  return 2 * ((size_t)passes * RADIX + (size_t)passes * sort_tiles(n) * RADIX + passes);
}

cudaError_t launch_sort(const uint64_t *first, uint32_t stride, bool index_vals, uint64_t *keys, uint64_t *keys_alt,
                        uint32_t *vals, uint32_t *vals_alt, uint32_t n, uint32_t shift0, uint32_t bits,
                        const SortScratch &scr, cudaStream_t s, bool *result_in_alt) {
  *result_in_alt = false;
  if (n == 0) return cudaSuccess;
  const uint32_t passes = (bits + RADIX_BITS - 1) / RADIX_BITS;
  if (passes == 0 || passes > 8) return cudaErrorInvalidValue;
  const uint32_t tiles = sort_tiles(n);
  uint32_t hb = (n + 1023) / 1024;
  if (hb > 152u * 4u) hb = 152u * 4u;
  sort_hist_kernel<<<hb, 1024, 0, s>>>(first, stride, n, shift0, passes, scr.hist);
  uint64_t *ki = keys, *ko = keys_alt;
  uint32_t *vi = vals, *vo = vals_alt;
  for (uint32_t p = 0; p < passes; ++p) {
    sort_pass_kernel<<<tiles, SORT_THREADS, 0, s>>>(p == 0 ? first : ki, p == 0 ? stride : 1u,
                                                    p == 0 && index_vals ? nullptr : vi, ko, vo, n,
                                                    shift0 + p * RADIX_BITS, scr.hist + p * RADIX,
                                                    scr.status + (size_t)p * tiles * RADIX, scr.tile_ctr + p,
                                                    scr.err, scr.spin_ns, p == 0 ? scr.hold_first : 0u);
    uint64_t *tk = ki;
    ki = ko;
    ko = tk;
    uint32_t *tv = vi;
    vi = vo;
    vo = tv;
  }
  *result_in_alt = (passes & 1u) != 0;
  return cudaGetLastError();
}

cudaError_t launch_gather_hi(const ulonglong2 *key, const uint32_t *perm, uint64_t *out, uint32_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  uint32_t blocks = (n + 255) / 256;
  if (blocks > 152u * 16u) blocks = 152u * 16u;
  gather_hi_kernel<<<blocks, 256, 0, s>>>(key, perm, out, n);
  return cudaGetLastError();
}

cudaError_t launch_merge(const MergeLaunch &L, cudaStream_t s) {
  if (L.n == 0) return cudaSuccess;
  const uint32_t tiles = merge_tiles(L.n);
  merge_kernel<<<tiles, MERGE_THREADS, 0, s>>>(L);
  return cudaGetLastError();
}

}  // namespace gpc
