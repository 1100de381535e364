// rk_prims.cu -- device-wide primitives used by the neighbour-list rebuild:
// exclusive prefix sum of int64 counts and a stable LSD radix sort of 64-bit
// keys (8 bits per pass, one kernel per pass).
#include <cstdint>

#include "rk_engine.cuh"

namespace rk {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int64_t kScanTile = (int64_t)kScanThreads * kScanItems;

static inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

__device__ __forceinline__ int64_t warp_incl_scan(int64_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

__global__ void k_tile_sums(const int64_t* __restrict__ in, int64_t n, int64_t* __restrict__ sums) {
  __shared__ int64_t ws[32];
  const int64_t base = blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t t = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    int64_t idx = base + k;
    if (idx < n) t += in[idx];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x < 32) {
    int64_t v = ws[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
  }
}

__global__ void k_tile_scan(const int64_t* in, int64_t* out, int64_t n, const int64_t* __restrict__ block_ofs) {
  __shared__ int64_t ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t t = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    int64_t idx = base + k;
    v[k] = idx < n ? in[idx] : 0;
    t += v[k];
  }
  int64_t x = warp_incl_scan(t);
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int64_t w = ws[lane];
    w = warp_incl_scan(w);
    ws[lane] = w;
  }
  __syncthreads();
  int64_t excl = x - t + (warp > 0 ? ws[warp - 1] : 0) + (block_ofs ? block_ofs[blockIdx.x] : 0);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    int64_t idx = base + k;
    if (idx < n) out[idx] = excl;
    excl += v[k];
  }
}

size_t scan_temp_bytes(int64_t n) {
  size_t total = 0;
  while (n > kScanTile) {
    int64_t nb = cdiv(n, kScanTile);
    total += (size_t)nb * sizeof(int64_t);
    n = nb;
  }
  return total + 256;
}

// out[k] = sum_{m<k} in[m]; in and out may alias.
void exclusive_scan_i64(const int64_t* in, int64_t* out, int64_t n, void* temp, cudaStream_t st) {
  if (n <= 0) return;
  if (n <= kScanTile) {
    k_tile_scan<<<1, kScanThreads, 0, st>>>(in, out, n, nullptr);
    return;
  }
  int64_t nb = cdiv(n, kScanTile);
  int64_t* sums = (int64_t*)temp;
  void* rest = (void*)(sums + nb);
  k_tile_sums<<<(unsigned)nb, kScanThreads, 0, st>>>(in, n, sums);
  exclusive_scan_i64(sums, sums, nb, rest, st);
  k_tile_scan<<<(unsigned)nb, kScanThreads, 0, st>>>(in, out, n, sums);
}

// ------------------------------------------------------------ radix sort ----
// Stable LSD sort, 8 bits per pass, one read and one write of the keys per
// pass: the digit counts of all passes come from one sweep over the keys (a
// pass only permutes them), and a pass's blocks learn where their keys go
// from the running totals that the blocks before them publish (a block waits
// only for blocks that took their tickets earlier, hence are running, and
// counts their keys itself when the wait lasts too long).  A
// histogram, a scan of blocks x 256 counts and a scatter per pass took 39 us
// at 165 000 keys and 41 us at 1.6 M, most of it launches and the scatter's
// 64 barriers per block.
constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int64_t kSortTile = (int64_t)kSortThreads * kSortItems;
constexpr int kMaxPasses = 8;

// Scratch: digit counts of every pass, a ticket counter per pass, then one
// status word per block and digit: pass << 56 | state << 54 | count, state 1
// the block's own count, 2 the total including all blocks before it (the pass
// tag makes the words of earlier passes stale).
struct SortTemp {
  unsigned int* hist;           // kMaxPasses * 256
  unsigned int* ticket;         // kMaxPasses
  unsigned long long* status;   // blocks * 256
};
constexpr size_t kSortHead = (size_t)kMaxPasses * 256 * sizeof(unsigned int) + 256;
__host__ __device__ __forceinline__ SortTemp sort_temp(void* temp) {
  SortTemp t;
  t.hist = (unsigned int*)temp;
  t.ticket = t.hist + kMaxPasses * 256;
  t.status = (unsigned long long*)((char*)temp + kSortHead);
  return t;
}

// Digits of pass p: bits [lo + 8 p, lo + 8 p + 8), fewer in the last pass when
// the range is not a multiple of 8 (the bits at and above hi must not take
// part in the order).
__global__ void __launch_bounds__(kSortThreads) k_radix_counts(const uint64_t* __restrict__ keys, int64_t n, int lo,
                                                               int hi, void* temp) {
  __shared__ unsigned h[kMaxPasses][256];
  const int passes = (hi - lo + 7) >> 3;
  for (int p = 0; p < passes; p++) h[p][threadIdx.x] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * kSortThreads;
  for (int64_t k = blockIdx.x * (int64_t)kSortThreads + threadIdx.x; k < n; k += stride) {
    const uint64_t x = keys[k];
    for (int p = 0, sh = lo; p < passes; p++, sh += 8) {
      const unsigned mask = hi - sh < 8 ? (1u << (hi - sh)) - 1u : 255u;
      atomicAdd(&h[p][(unsigned)(x >> sh) & mask], 1u);
    }
  }
  __syncthreads();
  const SortTemp t = sort_temp(temp);
  for (int p = 0; p < passes; p++)
    if (h[p][threadIdx.x]) atomicAdd(&t.hist[p * 256 + threadIdx.x], h[p][threadIdx.x]);
}

// exclusive scan of one value per thread over the block (ws: a word per warp)
__device__ __forceinline__ unsigned block_excl_scan(unsigned v, unsigned* ws) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  unsigned before = x - v;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++)
    if (w < warp) before += ws[w];
  return before;
}

// One pass.  Each warp ranks 16 x 32 consecutive keys with warp matches, the
// block's keys are put in digit order in shared memory and written out as
// runs.  A thread waits for the blocks before through at most RK_SORT_SPINS
// reads (far more than a running predecessor needs); then the block counts the
// digits of all keys in front of its tile itself, from the pass's input, which
// is complete: the sort ends, and its result is right, whatever the blocks
// before do.
#ifndef RK_SORT_SPINS
#define RK_SORT_SPINS (1 << 24)
#endif
constexpr int kSortSpins = RK_SORT_SPINS;
__global__ void __launch_bounds__(kSortThreads, 3) k_radix_pass(const uint64_t* __restrict__ in, uint64_t* __restrict__ out,
                                                             int64_t n, int sh, unsigned mask, int pass, void* temp) {
  __shared__ uint64_t skey[kSortTile];
  __shared__ unsigned whist[kSortWarps][256];
  __shared__ unsigned lbase[256], ws[kSortWarps];
  __shared__ long long gofs[256];
  __shared__ unsigned s_block;
  __shared__ int s_late;
  const SortTemp T = sort_temp(temp);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) {
    s_block = atomicAdd(&T.ticket[pass], 1u);
    s_late = 0;
  }
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) whist[w][t] = 0;
  __syncthreads();
  const int64_t blk = s_block;
  const int64_t tile = blk * kSortTile;
  const int count = (int)(n - tile < kSortTile ? n - tile : kSortTile);
  uint64_t key[kSortItems];
  unsigned short rank[kSortItems];
  const int first = warp * kSortItems * 32 + lane;
#pragma unroll
  for (int u = 0; u < kSortItems; u++) key[u] = first + 32 * u < count ? in[tile + first + 32 * u] : ~0ull;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int u = 0; u < kSortItems; u++) {
    const bool valid = first + 32 * u < count;
    const unsigned d = (unsigned)(key[u] >> sh) & mask;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u + mask);
    unsigned base = 0;
    if (valid) base = whist[warp][d];
    __syncwarp();
    if (valid && (peers & lt) == 0u) whist[warp][d] = base + __popc(peers);
    __syncwarp();
    rank[u] = (unsigned short)(base + __popc(peers & lt));
  }
  __syncthreads();
  // digit t: its count per warp becomes the offset of each warp's keys
  unsigned tot = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    const unsigned c = whist[w][t];
    whist[w][t] = tot;
    tot += c;
  }
  volatile unsigned long long* st = T.status;
  const unsigned long long tag = ((unsigned long long)(pass + 1)) << 56, val = (1ull << 54) - 1ull;
  __threadfence();
  st[blk * 256 + t] = tag | ((blk == 0 ? 2ull : 1ull) << 54) | (unsigned long long)tot;
  const unsigned lb = block_excl_scan(tot, ws);
  lbase[t] = lb;
  const unsigned gb = block_excl_scan(T.hist[pass * 256 + t], ws);  // first position of digit t
  unsigned long long before = 0;
  int spins = 0;
  bool late = false;
  for (int64_t p = blk - 1; p >= 0;) {
    const unsigned long long v = st[p * 256 + t];
    if ((v >> 56) != (tag >> 56)) {
      if (spins++ >= kSortSpins) {
        late = true;
        s_late = 1;
        break;
      }
      continue;
    }
    before += v & val;
    if (((v >> 54) & 3ull) == 2ull) break;
    p--;
  }
  auto publish = [&]() {
    __threadfence();
    st[blk * 256 + t] = tag | (2ull << 54) | (before + tot);
  };
  if (blk > 0 && !late) publish();
  __syncthreads();
  if (s_late) {  // (skey is not in use yet)
    unsigned* front = reinterpret_cast<unsigned*>(skey);
    front[t] = 0;
    __syncthreads();
    for (int64_t k = t; k < tile; k += kSortThreads) atomicAdd(&front[(unsigned)(in[k] >> sh) & mask], 1u);
    __syncthreads();
    before = front[t];
    if (late) publish();
  }
  gofs[t] = (long long)gb + (long long)before - (long long)lb;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kSortItems; u++)
    if (first + 32 * u < count) {
      const unsigned d = (unsigned)(key[u] >> sh) & mask;
      skey[lbase[d] + whist[warp][d] + rank[u]] = key[u];
    }
  __syncthreads();
  for (int k = t; k < count; k += kSortThreads) {
    const uint64_t x = skey[k];
    out[gofs[(unsigned)(x >> sh) & mask] + k] = x;
  }
}

size_t sort_temp_bytes(int64_t n) { return kSortHead + (size_t)cdiv(n > 0 ? n : 1, kSortTile) * 256 * sizeof(uint64_t); }

// Stable sort of keys on bits [lo_bit, hi_bit); tmp has n slots.  The
// result ends in keys.  Returns the number of kernels launched.
int radix_sort_u64(uint64_t* keys, uint64_t* tmp, int64_t n, int lo_bit, int hi_bit, void* temp,
                   cudaStream_t st) {
  if (n <= 1) return 0;
  const int64_t nb = cdiv(n, kSortTile);
  cudaMemsetAsync(temp, 0, sort_temp_bytes(n), st);
  const int64_t hb = cdiv(n, 4 * kSortThreads);
  k_radix_counts<<<(unsigned)(hb < 152 * 4 ? hb : 152 * 4), kSortThreads, 0, st>>>(keys, n, lo_bit, hi_bit, temp);
  uint64_t* src = keys;
  uint64_t* dst = tmp;
  int pass = 0;
  for (int sh = lo_bit; sh < hi_bit; sh += 8, pass++) {
    const unsigned mask = hi_bit - sh < 8 ? (1u << (hi_bit - sh)) - 1u : 255u;
    k_radix_pass<<<(unsigned)nb, kSortThreads, 0, st>>>(src, dst, n, sh, mask, pass, temp);
    uint64_t* x = src;
    src = dst;
    dst = x;
  }
  if (pass & 1) cudaMemcpyAsync(keys, src, (size_t)n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st);
  return 1 + pass;
}

}  // namespace rk
