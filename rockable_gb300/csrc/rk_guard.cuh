// rk_guard.cuh -- per-body evaluation of the learned skin's exact guard
// (see rk_skin.cu for the bounds), shared by the kernels that run it once per
// step of the skin mode.
#pragma once
#include "rk_bits.cuh"
#include "rk_engine.cuh"
#include "rk_near.cuh"

namespace rk {

// Upper bound of the rotation angle between two unit quaternions: with c
// the shorter of the chords |q - q0| and |q + q0|, the angle is
// 4 asin(c / 2) <= 2 c (1 + c).
__device__ __forceinline__ double quat_chord(const double* q, const double* q0) {
  double m2 = 0.0, p2 = 0.0;
  for (int d = 0; d < 4; d++) {
    const double m = q[d] - q0[d], p = q[d] + q0[d];
    m2 += m * m;
    p2 += p * p;
  }
  return sqrt(fmin(m2, p2));
}
__device__ __forceinline__ double rot_bound(const double* q, const double* q0) {
  const double c = quat_chord(q, q0);
  return 2.0 * c * (1.0 + c);
}

// The snapshot body b's guard compares with, its swing radius and its largest
// delta so far.
struct SkinRef {
  double x[3], q[4];
  float sw, maxd;
};
__device__ __forceinline__ SkinRef skin_ref(const Scene& s, int64_t b) {
  SkinRef r;
#pragma unroll
  for (int d = 0; d < 3; d++) r.x[d] = s.sk_ref_pos[3 * b + d];
#pragma unroll
  for (int d = 0; d < 4; d++) r.q[d] = s.sk_ref_q[4 * b + d];
  r.sw = s.sk_rsw[b];
  r.maxd = s.sk_maxd[b];
  return r;
}
// Largest value of the warp's lanes; values that are not numbers count as zero
// (the others are not negative, so that their bits compare as they do).
__device__ __forceinline__ float warp_max(float x) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(x, 0.f))));
}

// Guard of body b (position x, orientation q) for the state a step leaves;
// every thread of the block must call it (block reduction, blocks of at most
// 512 threads; b == n: no body).  sk_out (zeroed before the step): [0] max
// delta, [1] max |v| of the free bodies, [2] max g (float bits, atomicMax),
// [3] number of flagged bodies (g >= flag_at), [4..5] unused,
// [6] max delta and [7] max g bounded for the state after the NEXT step:
// the next drift's motion is bounded from the velocities and accelerations
// this step leaves (free bodies); driven bodies do not move between steps
// when no control drives them, which is the only case the host uses the
// bound for.
// r: the body's snapshot; path: its path bound (driven bodies: none, infinity).
// k: the body's velocity, acceleration, angular velocity and angular
// acceleration as floats; only the velocity without `predict`.
__device__ __forceinline__ void skin_guard_core(const Scene& s, int64_t b, const double* x, const double* q,
                                                const SkinRef& r, float path, const float* k, bool predict) {
  unsigned int* out = s.sk_out;
  float dmax = 0.f, vmax = 0.f, gmax = 0.f, pdmax = 0.f, pgmax = 0.f;
  unsigned nflag = 0;
  if (b < s.n) {
    const bool free_body = b >= s.n_driven;
    // differences in FP64, the rest in float rounded up (relative 1e-5 covers
    // the float rounding of the norms, 1e-12 m the conversions)
    const float dx = d2f(x[0] - r.x[0]), dy = d2f(x[1] - r.x[1]), dz = d2f(x[2] - r.x[2]);
    float m2 = 0.f, p2 = 0.f;
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const float m = d2f(q[d] - r.q[d]), p = d2f(q[d] + r.q[d]);
      m2 += m * m;
      p2 += p * p;
    }
    const float chord = sqrtf(fminf(m2, p2)) * (1.f + 1e-5f);
    dmax = (sqrtf(dx * dx + dy * dy + dz * dz) + 2.f * chord * (1.f + chord) * r.sw) * (1.f + 1e-5f) + 1e-12f;
    const float md = fmaxf(r.maxd, dmax);
    s.sk_maxd[b] = md;
    gmax = fminf(path, 2.f * md);
    const bool f = gmax >= s.sk_flag_at;
    s.sk_flag[b] = f ? 1 : 0;
    nflag = f ? 1u : 0u;
    if (free_body) {
      const float vx = k[0], vy = k[1], vz = k[2];
      vmax = sqrtf(vx * vx + vy * vy + vz * vz);
    }
    if (predict && free_body) {
      // bound of the next drift: |dt v + dt^2/2 a| and a rotation of at most
      // |w| dt + |alpha| dt^2/2 (the normalised quaternion update, 1 % margin
      // for its second-order terms); a step of angle t moves the chord c by at
      // most t/2, so 2c(1 + c) grows by at most t (1 + 2c + t/2).  Only decides
      // when the exact values must be read, so a bound is enough.
      const float ax = k[3], ay = k[4], az = k[5];
      const float wx = k[6], wy = k[7], wz = k[8];
      const float lx = k[9], ly = k[10], lz = k[11];
      const float dt = (float)s.dt, dt2 = (float)s.dt2_2;
      const float dxb = dt * vmax + dt2 * sqrtf(ax * ax + ay * ay + az * az);
      const float thb = dt * sqrtf(wx * wx + wy * wy + wz * wz) + dt2 * sqrtf(lx * lx + ly * ly + lz * lz);
      const float inc = 1.01f * (dxb + thb * r.sw * (1.f + 2.f * chord + thb)) + 1e-12f;
      pdmax = dmax + inc;
      pgmax = fminf(path + inc, 2.f * fmaxf(md, pdmax));
    } else {
      pdmax = dmax;
      pgmax = gmax;
    }
  }
  // warp, then block reduction through shared memory: one atomic per block
  // and quantity (the block size is at most 512 threads)
  dmax = warp_max(dmax);
  vmax = warp_max(vmax);
  gmax = warp_max(gmax);
  if (predict) {
    pdmax = warp_max(pdmax);
    pgmax = warp_max(pgmax);
  }
  nflag = __reduce_add_sync(0xffffffffu, nflag);
  __shared__ float red[16][5];
  __shared__ unsigned redn[16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) {
    red[warp][0] = dmax;
    red[warp][1] = vmax;
    red[warp][2] = gmax;
    red[warp][3] = pdmax;
    red[warp][4] = pgmax;
    redn[warp] = nflag;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nw; w++) {
      dmax = fmaxf(dmax, red[w][0]);
      vmax = fmaxf(vmax, red[w][1]);
      gmax = fmaxf(gmax, red[w][2]);
      pdmax = fmaxf(pdmax, red[w][3]);
      pgmax = fmaxf(pgmax, red[w][4]);
      nflag += redn[w];
    }
    atomicMax(&out[0], __float_as_uint(dmax));
    atomicMax(&out[1], __float_as_uint(vmax));
    atomicMax(&out[2], __float_as_uint(gmax));
    if (nflag) atomicAdd(&out[3], nflag);
    if (predict) {
      atomicMax(&out[6], __float_as_uint(pdmax));
      atomicMax(&out[7], __float_as_uint(pgmax));
    }
  }
}

// In a batch the guard is evaluated by the kernel that makes the drift (the
// positions it leaves are the step's), so that its reduction is complete when
// the next kernel starts.
__device__ __forceinline__ void skin_guard_drift(const Scene& s, int64_t b, const BodyState& k, const SkinRef& r) {
  const float v[3] = {d2f(k.v[0]), d2f(k.v[1]), d2f(k.v[2])};
  skin_guard_core(s, b, k.x, k.q, r, k.path, v, false);
}

// Without a batch, by the resultant kernel, with the prediction; have: kin
// holds the 12 values, otherwise they are read back.
__device__ __forceinline__ void skin_guard_body(const Scene& s, int64_t b, bool have = false, const float* kin = nullptr) {
  double x[3] = {}, q[4] = {};
  float k[12] = {}, path = INFINITY;
  SkinRef r = {};
  if (b < s.n) {
    r = skin_ref(s, b);
    if (b >= s.n_driven) path = s.sk_path[b];
#pragma unroll
    for (int d = 0; d < 3; d++) x[d] = s.pos[3 * b + d];
#pragma unroll
    for (int d = 0; d < 4; d++) q[d] = s.Q[4 * b + d];
    if (have) {
#pragma unroll
      for (int d = 0; d < 12; d++) k[d] = kin[d];
    } else if (b >= s.n_driven) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        k[d] = d2f(s.vel[3 * b + d]);
        k[3 + d] = d2f(s.acc[3 * b + d]);
        k[6 + d] = d2f(s.vrot[3 * b + d]);
        k[9 + d] = d2f(s.arot[3 * b + d]);
      }
    }
  }
  skin_guard_core(s, b, x, q, r, path, k, true);
}

// First kernel of a batched skin step (the drift): whether the step before it
// asked the batch to halt; the kernels behind it then return at once
// (step_halted).
__device__ __forceinline__ bool batch_halted(const Scene& s) {
  if (s.sk_ctl == nullptr) return false;
  if ((s.sk_ctl[0] | s.sk_ctl[16]) == 0u) return false;
  if (blockIdx.x == 0 && threadIdx.x == 0) s.sk_ctl[0] = 1u;
  return true;
}

// End of a batched skin step (control block sk_ctl, see rk_skin.cu), called by
// a kernel behind the drift (on the near set by k_near_bodies, most of whose
// launches have nothing else to do): one warp reads the step's guard words, a lane
// per word, counts the step and asks for a halt when the host has to act -- a
// refresh is due or the batch's step budget is spent -- and otherwise zeroes
// the guard words for the next step.
__device__ __forceinline__ void skin_batch_step_end(const Scene& s) {
  if (blockIdx.x != gridDim.x - 1 || threadIdx.x >= 32) return;
  volatile unsigned int* ctl = s.sk_ctl;
  volatile unsigned int* out = s.sk_out;
  const int l = threadIdx.x;
  const unsigned full = 0xffffffffu;
  const unsigned v = l < 8 ? ctl[l] : l < 16 ? out[l - 8] : 0u;
  const unsigned ex = __shfl_sync(full, v, 1) + 1u, since = __shfl_sync(full, v, 2) + 1u;
  const unsigned budget = __shfl_sync(full, v, 3), interval = __shfl_sync(full, v, 4);
  const float trig = __uint_as_float(__shfl_sync(full, v, 5));
  const unsigned path = __shfl_sync(full, v, 6);
  const unsigned g0 = __shfl_sync(full, v, 8), g2 = __shfl_sync(full, v, 10);
  const float crit = __uint_as_float(path ? g2 : g0);
  const bool halt = crit >= trig || since >= interval || ex >= budget;
  if (l == 1) ctl[1] = ex;
  else if (l == 2) ctl[2] = since;
  else if (l >= 8 && l < 16) {
    ctl[l] = v;
    if (!halt) out[l - 8] = 0u;
  } else if (l == 16 && halt) {
    ctl[16] = 1u;
  }
}

}  // namespace rk
