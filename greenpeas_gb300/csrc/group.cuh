// group.cuh -- symptom keys and the grouping of one bucket's items, shared by
// the compile pipeline (sortmerge.cu) and the allocation-free merge
// (static_merge.cu).
#pragma once

#include <cstdint>
#include <type_traits>

#include "device.cuh"

namespace gpc {
namespace {

// murmur3 64-bit finaliser (a published bijective mixer).
__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

// Two independent mixes of (word index, non-zero word value).
__device__ __forceinline__ ulonglong2 word_hash(uint32_t j, uint64_t v) {
  const uint64_t jj = (uint64_t)j + 1;
  return make_ulonglong2(fmix64(v * 0x9E3779B97F4A7C15ull + jj * 0xC2B2AE3D27D4EB4Full),
                         fmix64(v * 0xD6E8FEB86659FD93ull + jj * 0xA0761D6478BD642Full + 0x8EBC6AF09C88C6E3ull));
}

// a(1-b) + b(1-a), written as a + b(1-2a): two fused multiply-adds.
__device__ __forceinline__ double xor_merge(double a, double b) { return fma(b, fma(-2.0, a, 1.0), a); }

// (key, m) order: key.x, then key.y, then mechanism id.
__device__ __forceinline__ bool item_less(ulonglong2 a, uint32_t ma, ulonglong2 b, uint32_t mb) {
  if (a.x != b.x) return a.x < b.x;
  if (a.y != b.y) return a.y < b.y;
  return ma < mb;
}

__device__ __forceinline__ bool key_eq(ulonglong2 a, ulonglong2 b) { return a.x == b.x && a.y == b.y; }

// Loads a target list as 16-byte vectors (rows are 16-byte aligned).
__device__ __forceinline__ bool lists_equal(const uint32_t *a, const uint32_t *b, uint32_t n) {
  const uint4 *va = reinterpret_cast<const uint4 *>(a), *vb = reinterpret_cast<const uint4 *>(b);
  for (uint32_t k = 0; k * 4 < n; ++k) {
    const uint4 x = __ldg(va + k), y = __ldg(vb + k);
    const uint32_t rem = n - k * 4;
    if (x.x != y.x || (rem > 1 && x.y != y.y) || (rem > 2 && x.z != y.z) || (rem > 3 && x.w != y.w)) return false;
  }
  return true;
}

// What a bucket's grouping holds in shared memory: its items as they were
// filed, and the sorted order.
template <uint32_t CAP>
struct GroupItems {
  ulonglong2 key[CAP];
  double p[CAP];
  uint32_t m[CAP], t[CAP];
  uint32_t sv[CAP];  // position in the words' order -> mechanism
  std::conditional_t<CAP <= 256, uint8_t, uint16_t> ord[CAP];  // sorted position -> item
};

// Bitonic sort of 32 R words, R per lane: word r * 32 + lane is v[r].
template <int R>
__device__ __forceinline__ void sort_words(uint32_t (&v)[R]) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int k = 2; k <= 32 * R; k *= 2) {
#pragma unroll
    for (int j = k / 2; j > 0; j /= 2) {
      if (j >= 32) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int q = r ^ (j / 32);
          if (q > r) {
            const bool up = (r * 32 & k) == 0;
            const uint32_t lo = min(v[r], v[q]), hi = max(v[r], v[q]);
            v[r] = up ? lo : hi;
            v[q] = up ? hi : lo;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, v[r], j);
          const bool up = k < 32 ? (lane & k) == 0 : (r * 32 & k) == 0;
          v[r] = ((lane & j) == 0) == up ? min(v[r], o) : max(v[r], o);
        }
      }
    }
  }
}

// The DEM's order inside a bucket: top 6 bits of the key's second half, then the key, then the mechanism.
// (BIN; without it, the key alone).
template <bool BIN, typename G_t>
__device__ __forceinline__ bool item_before(const G_t &G, uint32_t a, uint32_t b) {
  const uint32_t ba = (uint32_t)(G.key[a].y >> 58), bb = (uint32_t)(G.key[b].y >> 58);
  return BIN && ba != bb ? ba < bb : item_less(G.key[a], G.m[a], G.key[b], G.m[b]);
}

// Orders the n <= 32 R items of G: G.ord.  The words sorted are 24 bits of the
// order's key (BIN: 6 of the second half, 18 of the first after the bits that
// all items share; else 24 of the first) above the item's index: one shuffle and one min/max a step.
// Items of equal words are then put in mechanism order: the runs' bounds come
// from ballots, so that an item only counts the smaller mechanisms of its run
// (with a search for the bounds through the items, 40 symptoms of 250 copies
// took 307 us here, now 64; a run of 30 mixed surface codes: 703 -> 695).  When
// two different keys share a word (a few in 10^6 buckets) every item's place is
// counted from the full keys instead.
template <int R, bool BIN, typename G_t>
__device__ __forceinline__ void order_items(G_t &G, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t ALL = 0xFFFFFFFFu;
  uint64_t hx[R];
  uint32_t differ = 0;
  const uint64_t x0 = G.key[0].x;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = r * 32 + lane;
    hx[r] = i < n ? G.key[i].x : x0;
    differ |= (uint32_t)((hx[r] ^ x0) >> 32);
  }
  differ = __reduce_or_sync(ALL, differ);
  const uint32_t same = differ ? (uint32_t)__clz(differ) : 32u;  // leading bits all share
  uint32_t v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = r * 32 + lane;
    v[r] = ALL;
    const uint32_t top = (uint32_t)((hx[r] << same) >> 32);
    if (i < n) v[r] = (BIN ? (uint32_t)(G.key[i].y >> 58) << 26 | (top >> 14) << 8 : top & 0xFFFFFF00u) | i;
  }
  sort_words<R>(v);
  bool mixed = false;
  if constexpr (R == 1) {
    const uint32_t i = v[0] & 255u;
    uint32_t m = 0;
    ulonglong2 k = make_ulonglong2(0, 0);
    if (lane < n) {
      m = G.m[i];
      k = G.key[i];
    }
    const uint32_t word = v[0] >> 8, left = __shfl_up_sync(ALL, word, 1);
    const uint64_t lx = __shfl_up_sync(ALL, k.x, 1), ly = __shfl_up_sync(ALL, k.y, 1);
    const bool start = lane == 0 || left != word || lane >= n;
    mixed = !start && (lx != k.x || ly != k.y);
    const uint32_t starts = __ballot_sync(ALL, start);
    const uint32_t first = 31u - __clz(starts & (ALL >> (31u - lane)));
    const uint32_t after = lane == 31u ? 0u : starts >> (lane + 1u);
    const uint32_t end = after ? lane + (uint32_t)__ffs(after) : 32u;  // the run is lanes [first, end)
    const uint32_t longest = __reduce_max_sync(ALL, end - first);
    uint32_t place = first;
    for (uint32_t o = 1; o < longest; ++o) {
      const uint32_t a = __shfl_up_sync(ALL, m, o), b = __shfl_down_sync(ALL, m, o);
      place += (lane >= first + o && a < m ? 1u : 0u) + (lane + o < end && b < m ? 1u : 0u);
    }
    if (lane < n) G.ord[place] = i;
  } else {
    uint32_t starts[R];  // positions whose word differs from the one before
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t s = r * 32 + lane;
      uint32_t left = __shfl_up_sync(ALL, v[r], 1);
      if (r > 0) {
        const uint32_t x = __shfl_sync(ALL, v[r > 0 ? r - 1 : 0], 31);
        if (lane == 0) left = x;
      }
      const bool tie = s > 0 && s < n && ((left ^ v[r]) >> 8) == 0;
      if (tie) mixed |= !key_eq(G.key[left & 255u], G.key[v[r] & 255u]);
      starts[r] = __ballot_sync(ALL, !tie);
      if (s < n) G.sv[s] = G.m[v[r] & 255u];  // the mechanisms in the words' order
    }
    __syncwarp();
    uint32_t open = 0;  // start of the run that is open at the chunk's first position
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t s = r * 32 + lane;
      const uint32_t le = starts[r] & (ALL >> (31u - lane)), gt = lane == 31u ? 0u : starts[r] >> (lane + 1u);
      const uint32_t first = le ? r * 32 + 31u - (uint32_t)__clz((int)le) : open;
      uint32_t end = 32u * R;
#pragma unroll
      for (int q = R - 1; q > r; --q)
        if (starts[q]) end = q * 32 + (uint32_t)__ffs((int)starts[q]) - 1u;
      if (gt) end = s + (uint32_t)__ffs((int)gt);
      end = min(end, n);
      if (s < n) {
        const uint32_t mi = G.sv[s];
        uint32_t place = first;
        for (uint32_t q = first; q < end; ++q) place += G.sv[q] < mi ? 1u : 0u;
        G.ord[place] = v[r] & 255u;
      }
      if (starts[r]) open = r * 32 + 31u - (uint32_t)__clz((int)starts[r]);
    }
  }
  if (__any_sync(ALL, mixed)) {
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32) {
      uint32_t place = 0;
      for (uint32_t q = 0; q < n; ++q) place += item_before<BIN>(G, q, i) ? 1u : 0u;
      G.ord[place] = i;
    }
  }
  __syncwarp();
}

// Groups of the n ordered items of G, 32 sorted positions at a time, and their
// number and targets.  Each group's probability is a segmented inclusive scan
// of the XOR-merge over its run: log2(longest run in the chunk) shuffle steps
// with every lane busy (FP64 throughput is scarce on this part), plus the
// value carried in from the previous chunk.  The scan is a tree, so its
// rounding differs from a left-to-right fold by a few ulps; it is
// deterministic.  `io`: targets of an item (count of its t), whether two items'
// lists are equal, and where a group's head (with the targets before it) and
// probability go.
template <uint32_t CAP, typename IO>
__device__ __forceinline__ uint2 fold_runs(const GroupItems<CAP> &G, uint32_t n, uint32_t tcap, uint32_t *err, const IO &io) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t gcount = 0, tcount = 0;
  uint32_t carry_head = 0;  // item of the run open at the end of the previous chunk
  double carry = 0.0;
  for (uint32_t s0 = 0; s0 < n; s0 += 32) {
    const uint32_t s = s0 + lane;
    const bool in = s < n;
    bool head = false, last = false;  // of its run
    uint32_t i = 0, nt = 0;
    double x = 0.0;
    if (in) {
      i = G.ord[s];
      nt = io.count(G.t[i]);
      x = G.p[i];
      const ulonglong2 k = G.key[i];
      head = s == 0 || !key_eq(G.key[G.ord[s - 1]], k);
      last = s + 1 >= n || !key_eq(G.key[G.ord[s + 1]], k);
    }
    const uint32_t hb = __ballot_sync(0xFFFFFFFFu, head);
    // the run of each position: it starts at lane `seg` of this chunk, or
    // (seg < 0) continues the run open at the end of the previous chunk
    const uint32_t le = hb & (0xFFFFFFFFu >> (31u - lane));
    const int seg = le ? 31 - __clz(le) : -1;
    const uint32_t seg0 = seg < 0 ? 0u : (uint32_t)seg;
    {
      // collision check: every item of a run against the run's head (full target lists)
      const uint32_t ih = seg < 0 ? carry_head : (uint32_t)G.ord[s0 + seg0];
      // (a list longer than the rows was flagged by the key pass and the run is redone with wider rows)
      if (in && !head && nt <= tcap && (io.count(G.t[ih]) != nt || !io.equal(i, ih, nt))) atomicOr(err, DEV_ERR_COLLISION);
      carry_head = __shfl_sync(0xFFFFFFFFu, ih, 31);
    }
    const uint32_t tv = head ? nt : 0u;
    uint32_t inc = tv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= (uint32_t)o) inc += a;
    }
    const uint32_t maxlen = __reduce_max_sync(0xFFFFFFFFu, in ? lane - seg0 + 1 : 0u);
    for (uint32_t d = 1; d < maxlen; d <<= 1) {
      const double y = __shfl_up_sync(0xFFFFFFFFu, x, d);
      if (lane >= d && lane - d >= seg0) x = xor_merge(y, x);
    }
    if (seg < 0) x = xor_merge(carry, x);
    if (head) io.group(gcount + __popc(hb & ((1u << lane) - 1u)), i, tcount + inc - tv, s);
    if (last)  // the run's last item holds its value
      io.prob(seg < 0 ? gcount - 1u : gcount + __popc(hb & ((1u << seg0) - 1u)), x);
    carry = __shfl_sync(0xFFFFFFFFu, x, 31);
    gcount += __popc(hb);
    tcount += __shfl_sync(0xFFFFFFFFu, inc, 31);
  }
  return make_uint2(gcount, tcount);
}

}  // namespace
}  // namespace gpc
