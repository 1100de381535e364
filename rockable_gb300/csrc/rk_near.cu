// rk_near.cu -- the near set: the few entries of the neighbour list that can
// be active in the next steps.
//
// The list holds every sub-contact within dVerlet (about a tenth of a grain);
// of its entries only a few percent touch, and between two list updates the
// bodies move a small part of dVerlet.  An entry is left out of the near set
// when its two sub-elements are farther apart than the two bodies' allowances
// together and nothing remembers a contact: it has no bond, its history is
// zero and its last overlap was not negative.  As long as no point of any body
// has moved by more than its allowance since, such an entry cannot be active:
// every law needs the contact point on both sub-elements and their distance
// below the radii, and it would neither read nor change any history (a
// separated or lost sub-contact of zero history keeps a zero history; an
// earlier dn counts only when negative).  The steps that another step of the
// same call follows therefore compute the near set alone, with the same
// results bit for bit; the last step of a call computes the whole list, so
// that every entry's dn is the last state's.
//
// The set is checked against the positions after every drift (near_track) and
// made anew in the same step when a body has used up its allowance or the
// list has changed; nothing is assumed about how the bodies got there, so
// controls and positions set by the host between calls are covered.
//
// The distances are float with the positions' differences taken in FP64, less
// a margin above their rounding errors; the allowance of a body grows with
// its speed: it balances the cost of making the set (about the cost of 0.15
// full passes) against the entries that a larger allowance keeps,
// sqrt(0.15 dVerlet rate dt), at least dVerlet / 128.
#include <algorithm>

#include "rk_guard.cuh"
#include "rk_near.cuh"

namespace rk {

// the body's allowance for its present speed bound
__device__ __forceinline__ float allowance(const Scene& s, int64_t b) {
  const float dv = (float)s.dVerlet;
  return fmaxf(dv * (1.f / 128.f), sqrtf(0.15f * dv * s.rate[b] * (float)s.dt));
}

// Whether the narrow phase has to compute entry e of the near set in this
// step (far: its sub-elements are proven apart, inside: with the projection
// inside).  It need not where it would leave the entry inactive and its
// history as it is: apart with a history of zero, or apart with the
// projection inside (a separated sub-contact keeps its history).  Then the
// act flag is cleared, and an old negative overlap, which the Avalanche law
// would read, becomes zero.
__device__ __forceinline__ bool zero_history(const Scene& s, int64_t e) {
  bool zero = s.fn[e] == 0.0;
#pragma unroll
  for (int d = 0; d < 3; d++) zero = zero && s.ft[3 * e + d] == 0.0 && s.mom[3 * e + d] == 0.0;
  return zero;
}
__device__ __forceinline__ bool compute_needed(const Scene& s, int64_t e, bool apart, bool inside) {
  if (!apart || !(inside || zero_history(s, e))) return true;
  s.act[e] = 0;
  if (s.dn[e] < 0.0) s.dn[e] = 0.0;
  return false;
}

// First kernel: lists what the step's narrow phase has to compute (srec).
// While the set is up to date it looks at the set's records (nrec); when it is
// not, at every entry, and makes the set (near flags and records) as well.
// The FP32 test runs here, at the occupancy of a light kernel, so that the
// FP64 path is issued for dense warps of the entries that need it: about half
// of the near set of a flowing pile.
__global__ void __launch_bounds__(128) k_near_entries(Scene s) {
  const bool stale = s.flags[FLAG_NEAR_STALE] != 0ull;
  if (step_halted(s)) return;
  int* slow = s.fast_body ? s.slow : nullptr;  // (the mixed form's kernel takes entries)
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane;
  if (!stale) {
    int64_t cnt[4];
#pragma unroll
    for (int t = 0; t < 4; t++) cnt[t] = (int64_t)s.flags[FLAG_NNEAR + t];
    const int64_t total = padded_total(cnt);
    for (int64_t k0 = first; k0 < total; k0 += stride) {
      int type;
      int64_t r;
      padded_place(cnt, k0, lane, &type, &r);
      bool need = false;
      int4 R = make_int4(0, 0, 0, 0), G = R;
      const int64_t len = type == 0 ? cnt[0] : type == 1 ? cnt[1] : type == 2 ? cnt[2] : cnt[3];
      if (r < len) {
        const int64_t at = (int64_t)s.flags[FLAG_TOFS + type] + r;
        R = s.nrec[2 * at];
        G = s.nrec[2 * at + 1];
        need = s.bonds && s.bond[R.x] >= 0;
        if (!need) {
          bool inside;
          const float D = near_distance(s, R.y, R.z, (uint32_t)R.w, G, &inside);
          need = compute_needed(s, R.x, D - (float)(s.rad[R.y] + s.rad[R.z]) * (1.f + 1e-6f) > 0.f, inside);
        }
      }
      append_record(s, need, type, R, G, FLAG_NSLOW, s.srec, slow, lane);
    }
    return;
  }
  for (int64_t k0 = first; k0 < s.ne; k0 += stride) {
    const int64_t k = k0 + lane;
    bool near = false, need = false;
    int type = 0;
    int4 R = make_int4(0, 0, 0, 0), G = R;
    if (k < s.ne) {
      const int e = s.nperm[k];
      const uint32_t ts = s.etsub[e];
      const int i = s.ei[e], j = s.ej[e];
      type = tsub_type(ts);
      R = make_int4(e, i, j, (int)ts);
      G = s.egv[e];
      near = need = s.bond[e] >= 0;
      if (!near) {
        bool inside;
        const float D = near_distance(s, i, j, ts, G, &inside);
        const float rsum = (float)(s.rad[i] + s.rad[j]) * (1.f + 1e-6f);
        // out of reach: in the set only while it remembers a contact
        near = !(D - rsum > allowance(s, i) + allowance(s, j)) || s.dn[e] < 0.0 || !zero_history(s, e);
        if (near) need = compute_needed(s, e, D - rsum > 0.f, inside);
        else s.act[e] = 0;
      }
      s.nflag[e] = near ? 1 : 0;
    }
    append_record(s, near, type, R, G, FLAG_NNEW, s.nrec, nullptr, lane);
    append_record(s, need, type, R, G, FLAG_NSLOW, s.srec, slow, lane);
  }
}

// Position p of body b's resultant in the serial order (j-side entries before
// its own block, its block, the rest of the j side), as a glist word.
__device__ __forceinline__ int serial_entry(const Scene& s, int64_t p, int64_t nA, int64_t nAB, int64_t i0, int64_t j0,
                                            int64_t js) {
  if (p >= nA && p < nAB) return (int)(i0 + (p - nA)) | (int)(((p - nA) % kGatherLanes) << kGlistLane);
  const int64_t q = p < nA ? p : js - j0 + (p - nAB);  // position in the j-side list
  return s.jlist[j0 + q] | (int)((unsigned)(q % kGatherLanes) << kGlistLane) | (int)0x80000000;
}

// Second kernel: each body's near entries in the serial order of its
// resultant (mixed form: its own block, then the j side), one warp per body, a
// block for the big ones (bodies whose resultant the step does not use have
// none), and the snapshot the set is checked against.  The last block puts the
// set into use.  At least 6 blocks per SM, the launch's resident wave: with the
// 48 registers it takes otherwise 50 000 bodies lost 0.4 % of the step.
constexpr int kNearThreads = 256;
__global__ void __launch_bounds__(kNearThreads, 6) k_near_bodies(Scene s) {
  const bool stale = s.flags[FLAG_NEAR_STALE] != 0ull;
  if (step_halted(s)) return;
  if (s.sk_ctl) skin_batch_step_end(s);
  if (!stale) return;
  __shared__ int wsum[kNearThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int g = blockIdx.x; g < s.nbig; g += gridDim.x) {
    const int64_t b = s.big[g];
    const int64_t i0 = s.iofs[b], i1 = s.iofs[b + 1], j0 = s.jofs[b], j1 = s.jofs[b + 1], js = s.fast_body ? j0 : s.jsplit[b];
    const int64_t nA = js - j0, nAB = nA + (i1 - i0), L = nAB + (j1 - js);
    int* out = s.glist + i0 + j0;
    int cnt = 0;
    for (int64_t c0 = 0; c0 < L; c0 += 4 * kNearThreads) {  // four consecutive positions a thread
      int x[4];
      int m = 0;
      const int64_t p0 = c0 + 4 * threadIdx.x;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        x[u] = p0 + u < L ? serial_entry(s, p0 + u, nA, nAB, i0, j0, js) : 0;
        if (p0 + u < L && s.nflag[x[u] & kGlistEntry]) m |= 1 << u;
      }
      int inc = __popc(m);
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) wsum[warp] = inc;
      __syncthreads();
      int before = cnt + inc - __popc(m), all = cnt;
      for (int w = 0; w < kNearThreads / 32; w++) {
        if (w < warp) before += wsum[w];
        all += wsum[w];
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if ((m >> u) & 1) out[before++] = x[u];
      cnt = all;
      __syncthreads();
    }
    if (threadIdx.x == 0) s.gcnt[b] = cnt;
  }
  const int64_t nw = (int64_t)gridDim.x * (kNearThreads / 32);
  for (int64_t b = blockIdx.x * (int64_t)(kNearThreads / 32) + warp; b < s.n; b += nw) {
    const int64_t i0 = s.iofs[b], i1 = s.iofs[b + 1], j0 = s.jofs[b], j1 = s.jofs[b + 1], js = s.fast_body ? j0 : s.jsplit[b];
    const int64_t nA = js - j0, nAB = nA + (i1 - i0), L = nAB + (j1 - js);
    const bool used = s.needres[b] != 0;
    if (!(used && L > kNearBig)) {
      int* out = s.glist + i0 + j0;
      int cnt = 0;
      for (int64_t c0 = 0; used && c0 < L; c0 += 32) {
        const int64_t p = c0 + lane;
        int x = 0;
        bool near = false;
        if (p < L) {
          x = serial_entry(s, p, nA, nAB, i0, j0, js);
          near = s.nflag[x & kGlistEntry] != 0;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, near);
        if (near) out[cnt + __popc(bal & lt)] = x;
        cnt += __popc(bal);
      }
      if (lane == 0) s.gcnt[b] = cnt;
    }
    if (lane < 3) s.npos[3 * b + lane] = s.pos[3 * b + lane];
    else if (lane < 7) s.nq[4 * b + lane - 3] = s.Q[4 * b + lane - 3];
    else if (lane == 7) s.nallow[b] = allowance(s, b) * (1.f - 1e-5f);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&s.flags[FLAG_NEAR_TICKET], 1ull) == gridDim.x - 1ull) {
      for (int t = 0; t < 4; t++) {
        s.flags[FLAG_NNEAR + t] = s.flags[FLAG_NNEW + t];
        s.flags[FLAG_NNEW + t] = 0ull;
      }
      s.flags[FLAG_NEAR_TICKET] = 0ull;
      s.flags[FLAG_NEAR_MADE]++;
      s.flags[FLAG_NEAR_STALE] = 0ull;
    }
  }
}

int launch_near_update(const Scene& s, cudaStream_t st) {
  // (an update of a small scene's set is a warp per SM: blocks of one warp)
  const int ct = s.ne < kSmallLaunch * 32 * 32 ? 32 : 128;
  const int64_t cb = std::min<int64_t>((s.ne + ct - 1) / ct, 152 * 1536 / ct);
  const int64_t bb = std::min<int64_t>((s.n + 7) / 8, 152 * 6);
  k_near_entries<<<(unsigned)std::max<int64_t>(cb, 1), ct, 0, st>>>(s);
  k_near_bodies<<<(unsigned)std::max<int64_t>(bb, 1), kNearThreads, 0, st>>>(s);
  return 2;
}

}  // namespace rk
