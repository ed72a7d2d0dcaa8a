// static_merge.cu -- merge raw error mechanisms into a DEM without allocating memory.
//
// Some callers cannot call cudaMalloc: code that runs while another runtime
// owns the device memory pool (a decoder or control loop that reserved its
// memory up front and must not grow it or synchronise the device in an
// allocation), or code whose memory budget is fixed at start-up.  For them,
// gpc_merge_mechanisms_static() runs the merge stage of the compile -- key
// hashing, radix bucketing, in-CTA sort and the FP64 XOR-merge -- on
// buffers the caller passes, with every piece of scratch memory taken from
// one file-scope static device array instead of an allocation.
//
// The scratch array is kStaticScratchBytes (about 2.3 MiB) and stays
// resident on every GPU that loads this library until the process exits.
// It bounds one call to kStaticMaxMechanisms (65,536) mechanisms.  All calls
// on a device share it: calls that overlap on the GPU (different streams,
// or different host threads) race and corrupt each other's results, so
// callers must serialise them.  Each call clears the counters it needs.
//
// Host code cannot use the array's name as a device address; the first call
// on each device looks the address up with cudaGetSymbolAddress (so make
// that first call outside any stream capture) and caches it per device.
//
// Four launches, each bound by its latency (65,536 mechanisms are a fraction of
// a wave): keys and bucket counts; the scatter into buckets, whose blocks scan
// the 1,024 counts themselves; a warp per bucket that orders and folds it as the
// compile does (group.cuh); the emission, whose blocks sum the aggregates
// before their buckets.  50,001 mechanisms of 20,000 symptoms: 37 us a call, against
// 65 with a setup, a scan, a one-thread finish and a CTA per bucket that ranked
// its items against one another and waited for the buckets before it.
#include <cstdint>
#include <mutex>

#include "../../include/gpc.h"
#include "device.cuh"
#include "group.cuh"

namespace gpc {
namespace {

constexpr uint32_t kStaticMaxMechanisms = 1u << 16;
constexpr uint32_t kStaticBucketBits = 10;
constexpr uint32_t kStaticBuckets = 1u << kStaticBucketBits;
constexpr uint32_t kMaxDevices = 64;

// Byte layout of the scratch array.
constexpr size_t A256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffKey = 0;                                                    // ulonglong2[max], then GroupRec[max]
constexpr size_t kOffBKey = A256(kOffKey + 16ull * kStaticMaxMechanisms);        // ulonglong2[max]
constexpr size_t kOffBM = A256(kOffBKey + 16ull * kStaticMaxMechanisms);         // uint32[max]
constexpr size_t kOffOffset = A256(kOffBM + 4ull * kStaticMaxMechanisms);        // uint32[nb]
constexpr size_t kOffAgg = A256(kOffOffset + 4ull * kStaticBuckets);             // uint2[nb]
constexpr size_t kOffZero = A256(kOffAgg + 8ull * kStaticBuckets);               // start of per-call zeroed part
constexpr size_t kOffCount = kOffZero;                                           // uint32[nb]
constexpr size_t kOffCursor = A256(kOffCount + 4ull * kStaticBuckets);           // uint32[nb]
constexpr size_t kOffErr = A256(kOffCursor + 4ull * kStaticBuckets);             // uint32
constexpr size_t kStaticScratchBytes = A256(kOffErr + 4);
constexpr size_t kZeroBytes = kStaticScratchBytes - kOffZero;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

std::mutex g_setup_mu;
void *g_scratch_addr[kMaxDevices] = {};

enum : uint32_t { STATIC_ERR_BAD_LIST = 64u };

struct StaticMerge {
  const uint32_t *tn, *tl;  // the caller's mechanisms
  const double *p;
  uint32_t n, stride;
  double *out_prob;
  uint32_t *out_off, *out_tg;
  uint32_t tg_cap;
  uint32_t *result;
  ulonglong2 *key, *bkey;   // keys by mechanism, then by bucket
  uint32_t *bm;             // mechanisms by bucket
  uint32_t *count, *cursor, *offset;
  uint2 *agg;               // (groups, targets) of each bucket
  uint32_t *err;
};

// One group of a bucket: its head mechanism, the targets before it in the bucket, its probability.
struct GroupRec {
  uint32_t m, before;
  double p;
};
static_assert(sizeof(GroupRec) == sizeof(ulonglong2), "group records take the keys' place");

constexpr uint32_t kThreads = 256;
constexpr uint32_t kGroupWarps = 4;        // buckets per block of the grouping
constexpr uint32_t kWarpItems = 256;       // items one warp orders; up to kBucketItems take the block
constexpr uint32_t kBucketItems = 1024;    // more are reported (DEV_FLAG_BIG_BUCKET)

// Bucket of a key: its top bits.
__device__ __forceinline__ uint32_t bucket_of(uint64_t x) { return (uint32_t)(x >> (64u - kStaticBucketBits)); }

// One thread per mechanism: 128-bit key of its target list, bucket histogram.
__global__ void __launch_bounds__(kThreads) static_key_kernel(const __grid_constant__ StaticMerge S) {
  const uint32_t m = blockIdx.x * kThreads + threadIdx.x;
  if (m >= S.n) return;
  uint32_t nt = S.tn[m];
  if (nt > S.stride) {
    atomicOr(S.err, STATIC_ERR_BAD_LIST);
    nt = S.stride;
  }
  const uint4 *t = reinterpret_cast<const uint4 *>(S.tl + (size_t)m * S.stride);  // (rows are 16-byte aligned)
  uint64_t hx = 0, hy = 0, v = 0;
  uint32_t cur = 0xFFFFFFFFu, prev = 0;
  bool bad = false;
  auto close = [&]() {
    if (v) {
      const ulonglong2 h = word_hash(cur, v);
      hx ^= h.x;
      hy ^= h.y;
    }
  };
  for (uint32_t k = 0; k < nt; k += 4) {
    const uint4 x = __ldg(t + k / 4);
    const uint32_t b4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      if (k + q >= nt) break;
      const uint32_t b = b4[q];
      bad |= k + q > 0 && b <= prev;  // targets must ascend
      prev = b;
      const uint32_t j = b >> 6;
      if (j != cur) {
        close();
        cur = j;
        v = 0;
      }
      v |= 1ull << (b & 63u);
    }
  }
  close();
  if (bad) atomicOr(S.err, STATIC_ERR_BAD_LIST);
  S.key[m] = make_ulonglong2(hx, hy);
  if ((hx | hy) == 0) {
    if (nt) atomicOr(S.err, DEV_ERR_COLLISION);
  } else {
    red_add(S.count + bucket_of(hx), 1u);
  }
}

// Moves every non-empty mechanism to its bucket.  Each block scans the counts;
// block 0 also writes the offsets.
__global__ void __launch_bounds__(kThreads) static_scatter_kernel(const __grid_constant__ StaticMerge S) {
  static_assert(kStaticBuckets == 4 * kThreads, "four buckets a thread");
  __shared__ uint32_t s_off[kStaticBuckets];
  __shared__ uint32_t s_warp[kThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t m = blockIdx.x * kThreads + tid;
  const ulonglong2 key = m < S.n ? S.key[m] : make_ulonglong2(0, 0);
  const bool item = (key.x | key.y) != 0;
  const uint32_t place = item ? atomicAdd(S.cursor + bucket_of(key.x), 1u) : 0u;
  const uint4 c = reinterpret_cast<const uint4 *>(S.count)[tid];
  const uint32_t sum = c.x + c.y + c.z + c.w;
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (uint32_t)o) inc += x;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t run = inc - sum;
  for (uint32_t w = 0; w < warp; ++w) run += s_warp[w];
  const uint4 off = make_uint4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
  reinterpret_cast<uint4 *>(s_off)[tid] = off;
  if (blockIdx.x == 0) reinterpret_cast<uint4 *>(S.offset)[tid] = off;
  __syncthreads();
  if (!item) return;
  const uint32_t at = s_off[bucket_of(key.x)] + place;
  S.bkey[at] = key;
  S.bm[at] = m;
}

// A bucket's groups as records in its range of the keys' array.
struct StaticRuns {
  const StaticMerge &S;
  GroupRec *rec;
  const uint32_t *m;
  __device__ __forceinline__ uint32_t count(uint32_t t) const { return t; }
  __device__ __forceinline__ bool equal(uint32_t a, uint32_t b, uint32_t n) const {
    return lists_equal(S.tl + (size_t)m[a] * S.stride, S.tl + (size_t)m[b] * S.stride, n);
  }
  __device__ __forceinline__ void group(uint32_t g, uint32_t head, uint32_t before, uint32_t) const {
    rec[g].m = m[head];
    rec[g].before = before;
  }
  __device__ __forceinline__ void prob(uint32_t g, double p) const { rec[g].p = p; }
};

// Items [first, first + n) of a bucket that starts at `base`, a thread each.
template <uint32_t CAP>
__device__ __forceinline__ void load_items(const StaticMerge &S, GroupItems<CAP> &G, uint32_t base, uint32_t n,
                                           uint32_t first, uint32_t step) {
  for (uint32_t i = first; i < n; i += step) {
    const uint32_t m = S.bm[base + i];
    G.key[i] = S.bkey[base + i];
    G.m[i] = m;
    // a list longer than the stride was reported (and cut to the stride) by the key pass; every read of a
    // count is cut the same way, so no list is read past its row
    G.t[i] = min(__ldg(S.tn + m), S.stride);
    G.p[i] = __ldg(S.p + m);
  }
}

// Places of a block's n <= kBucketItems items: a thread holds the keys of all its
// items and passes over the bucket once (20,000 mechanisms in runs of 900: the
// whole merge 826 -> 294 us; with a pass per item each step waits for its key
// in shared memory).
__device__ __forceinline__ void place_items(GroupItems<kBucketItems> &G, uint32_t n) {
  constexpr uint32_t T = kGroupWarps * 32u, PER = kBucketItems / T;
  ulonglong2 k[PER];
  uint32_t m[PER], place[PER];
#pragma unroll
  for (uint32_t r = 0; r < PER; ++r) {
    const uint32_t i = threadIdx.x + r * T;
    k[r] = i < n ? G.key[i] : make_ulonglong2(0, 0);
    m[r] = i < n ? G.m[i] : 0u;
    place[r] = 0;
  }
  for (uint32_t q = 0; q < n; ++q) {
    const ulonglong2 kq = G.key[q];
    const uint32_t mq = G.m[q];
#pragma unroll
    for (uint32_t r = 0; r < PER; ++r)
      place[r] += (kq.x < k[r].x) | ((kq.x == k[r].x) & ((kq.y < k[r].y) | ((kq.y == k[r].y) & (mq < m[r])))) ? 1u : 0u;
  }
#pragma unroll
  for (uint32_t r = 0; r < PER; ++r) {
    const uint32_t i = threadIdx.x + r * T;
    if (i < n) G.ord[place[r]] = (uint16_t)i;
  }
}

// One warp per bucket; a bucket of more than kWarpItems items is ordered by its
// block (each thread counts its items' places) and folded by one warp.
__global__ void __launch_bounds__(kGroupWarps * 32) static_group_kernel(const __grid_constant__ StaticMerge S) {
  __shared__ union Shared {
    GroupItems<kWarpItems> w[kGroupWarps];
    GroupItems<kBucketItems> all;
    __device__ Shared() {}
  } M;
  const uint32_t lane = threadIdx.x & 31u, wi = threadIdx.x >> 5;
  const uint32_t b0 = blockIdx.x * kGroupWarps, b = b0 + wi;
  const uint32_t n = S.count[b], base = S.offset[b];
  if (n <= kWarpItems || n > kBucketItems) {
    uint2 agg = make_uint2(0, 0);
    if (n > kBucketItems) {
      if (lane == 0) atomicOr(S.err, DEV_FLAG_BIG_BUCKET);
    } else if (n) {
      GroupItems<kWarpItems> &G = M.w[wi];
      load_items(S, G, base, n, lane, 32u);
      __syncwarp();
      if (n <= 32) order_items<1, false>(G, n);
      else if (n <= 64) order_items<2, false>(G, n);
      else if (n <= 128) order_items<4, false>(G, n);
      else order_items<8, false>(G, n);
      agg = fold_runs(G, n, S.stride, S.err, StaticRuns{S, reinterpret_cast<GroupRec *>(S.key) + base, G.m});
    }
    if (lane == 0) S.agg[b] = agg;
  }
  if (!__syncthreads_or(n > kWarpItems && n <= kBucketItems ? 1 : 0)) return;
  for (uint32_t k = 0; k < kGroupWarps; ++k) {
    const uint32_t nk = S.count[b0 + k], bk = S.offset[b0 + k];
    if (nk <= kWarpItems || nk > kBucketItems) continue;
    load_items(S, M.all, bk, nk, threadIdx.x, kGroupWarps * 32u);
    __syncthreads();
    place_items(M.all, nk);
    __syncthreads();
    if (wi == 0) {
      const uint2 a = fold_runs(M.all, nk, S.stride, S.err, StaticRuns{S, reinterpret_cast<GroupRec *>(S.key) + bk, M.all.m});
      if (lane == 0) S.agg[b0 + k] = a;
    }
    __syncthreads();
  }
}

// One warp per bucket: its groups to the caller's arrays.  The last bucket's
// warp closes the offsets and reports the totals and flags.
__global__ void __launch_bounds__(kThreads) static_emit_kernel(const __grid_constant__ StaticMerge S) {
  constexpr uint32_t NW = kThreads / 32;
  __shared__ uint2 s_sum[NW], s_agg[NW];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wi = tid >> 5;
  const uint32_t b0 = blockIdx.x * NW, b = b0 + wi;
  const uint2 agg = S.agg[b];
  const GroupRec *rec = reinterpret_cast<const GroupRec *>(S.key) + S.offset[b];
  uint2 pre = make_uint2(0, 0);
  for (uint32_t k = tid; k < b0; k += kThreads) {
    const uint2 a = S.agg[k];
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
  uint2 out = make_uint2(0, 0);
#pragma unroll
  for (uint32_t k = 0; k < NW; ++k) {
    out.x += s_sum[k].x + (k < wi ? s_agg[k].x : 0u);
    out.y += s_sum[k].y + (k < wi ? s_agg[k].y : 0u);
  }
  if (b == kStaticBuckets - 1 && lane == 0) {
    const uint2 end = make_uint2(out.x + agg.x, out.y + agg.y);
    S.result[0] = end.x;
    S.result[1] = end.y;
    S.result[2] = *S.err | (end.y > S.tg_cap ? DEV_FLAG_TG_OVF : 0u);
    S.result[3] = 0;
    S.out_off[end.x] = end.y;
  }
  for (uint32_t g = lane; g < agg.x; g += 32) {
    const GroupRec r = rec[g];
    const uint32_t slot = out.x + g, toff = out.y + r.before;
    const uint32_t ntg = (g + 1 < agg.x ? rec[g + 1].before : agg.y) - r.before;
    S.out_prob[slot] = r.p;
    S.out_off[slot] = toff;
    if ((uint64_t)toff + ntg > S.tg_cap) continue;
    const uint4 *src = reinterpret_cast<const uint4 *>(S.tl + (size_t)r.m * S.stride);
    for (uint32_t k = 0; k < ntg; k += 4) {
      const uint4 x = __ldg(src + k / 4);
      S.out_tg[toff + k] = x.x;
      if (k + 1 < ntg) S.out_tg[toff + k + 1] = x.y;
      if (k + 2 < ntg) S.out_tg[toff + k + 2] = x.z;
      if (k + 3 < ntg) S.out_tg[toff + k + 3] = x.w;
    }
  }
}

}  // namespace
}  // namespace gpc

extern "C" gpc_status gpc_merge_mechanisms_static(const uint32_t *num_targets, const uint32_t *targets,
                                                  uint32_t stride, const double *probs, uint32_t n,
                                                  double *out_probs, uint32_t *out_offsets, uint32_t *out_targets,
                                                  uint32_t out_target_cap, uint32_t *result, void *stream) {
  using namespace gpc;
  if (n > kStaticMaxMechanisms) return GPC_ERR_CAPACITY;  // more mechanisms than the static scratch holds
  if (!num_targets || !targets || !probs || !out_probs || !out_offsets || !out_targets || !result || stride == 0)
    return GPC_ERR_INVALID;
  // target lists are read as 16-byte vectors
  if (stride % 4 != 0 || (reinterpret_cast<uintptr_t>(targets) & 15u) != 0) return GPC_ERR_INVALID;
  // list lengths are cut to the stride, so n * stride bounds every target
  // count and offset the kernels form in 32 bits
  if ((uint64_t)n * stride > 0xFFFFFFFFull) return GPC_ERR_CAPACITY;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || (uint32_t)dev >= kMaxDevices) return GPC_ERR_CUDA;
  char *base;
  {
    std::lock_guard<std::mutex> lk(g_setup_mu);
    if (!g_scratch_addr[dev]) {
      void *p = nullptr;
      if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p) {
        (void)cudaGetLastError();
        return GPC_ERR_CUDA;
      }
      g_scratch_addr[dev] = p;
    }
    base = static_cast<char *>(g_scratch_addr[dev]);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  StaticMerge S{};
  S.tn = num_targets;
  S.tl = targets;
  S.p = probs;
  S.n = n;
  S.stride = stride;
  S.out_prob = out_probs;
  S.out_off = out_offsets;
  S.out_tg = out_targets;
  S.tg_cap = out_target_cap;
  S.result = result;
  S.key = reinterpret_cast<ulonglong2 *>(base + kOffKey);
  S.bkey = reinterpret_cast<ulonglong2 *>(base + kOffBKey);
  S.bm = reinterpret_cast<uint32_t *>(base + kOffBM);
  S.offset = reinterpret_cast<uint32_t *>(base + kOffOffset);
  S.agg = reinterpret_cast<uint2 *>(base + kOffAgg);
  S.count = reinterpret_cast<uint32_t *>(base + kOffCount);
  S.cursor = reinterpret_cast<uint32_t *>(base + kOffCursor);
  S.err = reinterpret_cast<uint32_t *>(base + kOffErr);

  if (cudaMemsetAsync(base + kOffZero, 0, kZeroBytes, s) != cudaSuccess) return GPC_ERR_CUDA;
  const uint32_t blocks = (n + kThreads - 1) / kThreads;
  if (n) static_key_kernel<<<blocks, kThreads, 0, s>>>(S);
  static_scatter_kernel<<<blocks ? blocks : 1, kThreads, 0, s>>>(S);
  static_group_kernel<<<kStaticBuckets / kGroupWarps, kGroupWarps * 32, 0, s>>>(S);
  static_emit_kernel<<<kStaticBuckets / (kThreads / 32), kThreads, 0, s>>>(S);
  return cudaGetLastError() == cudaSuccess ? GPC_OK : GPC_ERR_CUDA;
}
