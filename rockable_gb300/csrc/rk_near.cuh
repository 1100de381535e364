// rk_near.cuh -- the near set (see rk_near.cu): its check, run for every body
// by the kernel that makes the step's drift, the FP32 distance of an entry's
// sub-elements, and the loop of the narrow phase over what a step has to compute.
#pragma once
#include "rk_bits.cuh"
#include "rk_engine.cuh"

namespace rk {

// A body's state after the step's drift, in the registers of its thread
// (path: the skin's path-length bound, when that is kept).
struct BodyState {
  double x[3], v[3], q[4], w[3];
  float path;
};
__device__ __forceinline__ BodyState body_state(const Scene& s, int64_t b) {
  BodyState k;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    k.x[d] = s.pos[3 * b + d];
    k.v[d] = s.vel[3 * b + d];
    k.w[d] = s.vrot[3 * b + d];
  }
#pragma unroll
  for (int d = 0; d < 4; d++) k.q[d] = s.Q[4 * b + d];
  k.path = INFINITY;  // driven bodies are moved by their controls, not by the drift: no path
  return k;
}
// What near_track compares with.  Loaded before the drift's first store it
// shares the round of loads that the drift waits for anyway.
struct NearRef {
  double x[3], q[4];
  float sw, allow;
  bool stale;
};
__device__ __forceinline__ NearRef near_ref(const Scene& s, int64_t b) {
  NearRef r;
#pragma unroll
  for (int d = 0; d < 3; d++) r.x[d] = s.npos[3 * b + d];
#pragma unroll
  for (int d = 0; d < 4; d++) r.q[d] = s.nq[4 * b + d];
  r.sw = s.swing[b];
  r.allow = s.nallow[b];
  r.stale = s.flags[FLAG_NEAR_STALE] != 0ull;
  return r;
}
// The step's counters, emptied by the thread of body 0.
__device__ __forceinline__ void step_counters(const Scene& s, int64_t b) {
  if (b != 0) return;
  s.flags[FLAG_NACTIVE] = 0ull;
  if (s.sk_out && !s.sk_ctl)
    for (int d = 0; d < 8; d++) s.sk_out[d] = 0u;
}
// Check of the present near set for body b at the step's positions (k): the
// largest motion of a point of the body since the set was made, |x - x0| plus
// the swing radius times the rotation bound 2 c (1 + c) of the quaternion
// chord c (differences in FP64, the rest in float rounded up, as in the skin's
// guard), against the body's allowance.  A motion that is not a number fails
// the check.
__device__ __forceinline__ void near_check(const Scene& s, const BodyState& k, const NearRef& r) {
  const double* q = k.q;
  float d2 = 0.f, m2 = 0.f, p2 = 0.f;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float x = d2f(k.x[d] - r.x[d]);
    d2 += x * x;
  }
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const double q0 = r.q[d];
    const float m = d2f(q[d] - q0), p = d2f(q[d] + q0);
    m2 += m * m;
    p2 += p * p;
  }
  const float c = sqrtf(fminf(m2, p2)) * (1.f + 1e-5f);
  const float moved = (sqrtf(d2) + 2.f * c * (1.f + c) * r.sw) * (1.f + 1e-5f) + 1e-12f;
  if (!(moved < r.allow)) s.flags[FLAG_NEAR_STALE] = 1ull;
}
// Both, and the body's speed bound and FP32 orientation for the next near set.
__device__ __forceinline__ void near_track(const Scene& s, int64_t b, const BodyState& k, const NearRef& r) {
  step_counters(s, b);
  float v2 = 0.f, w2 = 0.f;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float v = d2f(k.v[d]), w = d2f(k.w[d]);
    v2 += v * v;
    w2 += w * w;
  }
  s.rate[b] = sqrtf(v2) + sqrtf(w2) * r.sw;
  s.qf[b] = make_float4(d2f(k.q[0]), d2f(k.q[1]), d2f(k.q[2]), d2f(k.q[3]));
  if (!r.stale) near_check(s, k, r);
}

struct N3 {
  float x, y, z;
};
__device__ __forceinline__ N3 n3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ N3 operator+(N3 a, N3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ N3 operator-(N3 a, N3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ N3 operator*(float k, N3 a) { return {k * a.x, k * a.y, k * a.z}; }
__device__ __forceinline__ float ndot(N3 a, N3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ N3 ncross(N3 a, N3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float namax(N3 a) { return fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))); }
__device__ __forceinline__ float sat01(float t) { return fminf(fmaxf(t, 0.f), 1.f); }

__device__ __forceinline__ N3 nrot(float4 q, N3 u) {  // q = (w, x, y, z)
  const N3 v = {q.y, q.z, q.w};
  const N3 t = 2.f * ncross(v, u);
  return u + q.x * t + ncross(v, t);
}

__device__ __forceinline__ float seg_d2(N3 p, N3 a, N3 b) {
  const N3 ab = b - a, ap = p - a;
  const float l2 = ndot(ab, ab);
  const float t = l2 > 0.f ? sat01(ndot(ap, ab) / l2) : 0.f;
  const N3 d = ap - t * ab;
  return ndot(d, d);
}

// A lower bound of the distance between the two sub-elements of entry e (not
// counting the rounding radii), from its FP32 vertices in coordinates relative
// to body j's centre.  A vertex of body i is the sum of its offset and the
// centres' difference, which cancel where the bodies touch: mag, which the
// margins scale with, covers half that difference besides the vertices (the
// sum errs by up to 6e-7 of it; the margins are 2e-6 of it and more).  With
// inside, also whether the projection or the closest points lie inside their ranges by more than the rounding errors, so that
// the narrow phase finds the same.
__device__ __forceinline__ float near_distance(const Scene& s, int i, int j, uint32_t ts, int4 G, bool* inside) {
  const int type = tsub_type(ts);
  const float4 qi = s.qf[i], qj = s.qf[j];
  const N3 dx = n3((float)(s.pos[3 * (int64_t)i] - s.pos[3 * (int64_t)j]),
                   (float)(s.pos[3 * (int64_t)i + 1] - s.pos[3 * (int64_t)j + 1]),
                   (float)(s.pos[3 * (int64_t)i + 2] - s.pos[3 * (int64_t)j + 2]));
  auto I = [&](int k) {
    const float4 u = s.uvf[k];
    return dx + nrot(qi, n3(u.x, u.y, u.z));
  };
  auto J = [&](int k) {
    const float4 u = s.uvf[k];
    return nrot(qj, n3(u.x, u.y, u.z));
  };
  float D, mag = 0.5f * namax(dx);
  if (type == 0) {
    const N3 a = I(G.x), b = J(G.y), d = a - b;
    mag = fmaxf(mag, fmaxf(namax(a), namax(b)));
    D = sqrtf(ndot(d, d));
    if (inside) *inside = true;
  } else if (type == 1) {
    const N3 a = I(G.x), p = J(G.y), q = J(G.z);
    mag = fmaxf(mag, fmaxf(namax(a), fmaxf(namax(p), namax(q))));
    D = sqrtf(seg_d2(a, p, q));
    if (inside) {
      const N3 E = q - p;
      const float E2 = ndot(E, E), r = ndot(a - p, E) / E2;
      const float tol = 1e-5f + 4e-6f * mag * rsqrtf(E2) * (1.f + fabsf(r));
      *inside = r > tol && r < 1.f - tol;
    }
  } else if (type == 2) {
    // point to polygon: to the plane when its projection is inside, else to
    // the nearest side; `off` is how far the polygon's vertices lie off the
    // plane of the narrow phase (that of its first, second and last vertex)
    const bool tri = G.w >= 0;
    int nv = 3, o = 0;
    const int* fv = nullptr;
    if (!tri) {
      const int fo = s.face_ofs[s.shape[j]] + tsub_jsub(ts);
      fv = s.face_verts + s.face_vofs[fo];
      nv = s.face_vofs[fo + 1] - s.face_vofs[fo];
      o = (int)s.gv_ofs[j];
    }
    const N3 a = I(G.x);
    const N3 A = J(tri ? G.y : o + fv[0]), B = J(tri ? G.z : o + fv[1]), C = J(tri ? G.w : o + fv[nv - 1]);
    const N3 bA = B - A, cA = C - A, w = a - A;
    N3 n = ncross(bA, cA);
    const float nn = ndot(n, n);
    mag = fmaxf(fmaxf(mag, namax(a)), fmaxf(namax(A), fmaxf(namax(B), namax(C))));
    float best = 3.0e38f, off = 0.f;
    // (a needle's float normal is not usable: its entries stay in the set)
    if (!(nn > 1e-5f * fmaxf(ndot(bA, bA), ndot(cA, cA)) * fminf(ndot(bA, bA), ndot(cA, cA)))) {
      if (inside) *inside = false;
      return -1.f;
    }
    n = rsqrtf(nn) * n;
    const float dist = ndot(w, n);
    const N3 e1 = rsqrtf(ndot(bA, bA)) * bA, e2 = ncross(n, e1);
    const float o1 = ndot(w, e1), o2 = ndot(w, e2);
    int odd = 0;
    float lo = 3.0e38f, hi = -3.0e38f;  // the projection's signed distances from the sides
    N3 pa = n3(0.f, 0.f, 0.f);
    for (int k = 0; k < nv; k++) {
      const N3 pb = k + 1 == nv ? n3(0.f, 0.f, 0.f) : tri ? (k == 0 ? bA : cA) : J(o + fv[k + 1]) - A;
      const float a1 = ndot(pa, e1), b1 = ndot(pb, e1), a2 = ndot(pa, e2), b2 = ndot(pb, e2);
      if ((a2 < o2 && b2 >= o2) || (b2 < o2 && a2 >= o2))
        if (a1 + (o2 - a2) / (b2 - a2) * (b1 - a1) < o1) odd = 1 - odd;
      best = fminf(best, seg_d2(w, pa, pb));
      if (inside) {
        const float l = rsqrtf((b1 - a1) * (b1 - a1) + (b2 - a2) * (b2 - a2));
        const float side = ((b1 - a1) * (o2 - a2) - (b2 - a2) * (o1 - a1)) * l;
        lo = fminf(lo, side);
        hi = fmaxf(hi, side);
      }
      off = fmaxf(off, fabsf(ndot(pb, n)));
      mag = fmaxf(mag, namax(pb + A));
      pa = pb;
    }
    if (odd) best = fminf(best, dist * dist);
    D = sqrtf(best) - 4.f * off;
    if (inside) {
      const float tol = 1e-8f + 4e-6f * mag + 4.f * off;
      *inside = lo > tol || hi < -tol;
    }
  } else {
    const N3 p1 = I(G.x), q1 = I(G.y), p2 = J(G.z), q2 = J(G.w);
    mag = fmaxf(mag, fmaxf(fmaxf(namax(p1), namax(q1)), fmaxf(namax(p2), namax(q2))));
    const N3 d1 = q1 - p1, d2 = q2 - p2, r = p1 - p2;
    const float a = ndot(d1, d1), e = ndot(d2, d2), b = ndot(d1, d2), c = ndot(d1, r), f = ndot(d2, r);
    const float den = a * e - b * b;
    if (den > 1e-3f * a * e) {
      float u = sat01((b * f - c * e) / den), t = (b * u + f) / e;
      if (t < 0.f) {
        t = 0.f;
        u = sat01(-c / a);
      } else if (t > 1.f) {
        t = 1.f;
        u = sat01((b - c) / a);
      }
      const N3 w = r + u * d1 - t * d2;
      D = sqrtf(ndot(w, w));
      // (well conditioned, and clear of the narrow phase's parallel threshold)
      const float tol = 1e-5f + 4e-5f * mag * rsqrtf(fminf(a, e)) * 3.f;
      if (inside)
        *inside = den > 2e-12f + 0.01f * a * e && u > tol && u < 1.f - tol && t > tol && t < 1.f - tol;
    } else {
      if (inside) *inside = false;
      // nearly parallel (sine of the angle below 0.032): the smallest
      // distance lies at an end up to that sine (its square rounded up)
      // times the shorter edge
      const float m = fminf(fminf(seg_d2(p1, p2, q2), seg_d2(q1, p2, q2)), fminf(seg_d2(p2, p1, q1), seg_d2(q2, p1, q1)));
      D = sqrtf(m) - sqrtf((fmaxf(den, 0.f) / fmaxf(a * e, 1e-37f) + 1e-6f) * fminf(a, e));
    }
  }
  // float errors: a few units of the coordinates' last place, and of D's
  return D - (1e-7f + 4e-6f * mag + 1e-4f * fabsf(D));
}

// Appends the record (entry, bodies, types; global vertex indices) of the
// lanes with ok to the list of its type (two int4 per position), or with
// `only_entry` its entry alone.
__device__ __forceinline__ void append_record(const Scene& s, bool ok, int type, int4 a, int4 b, int counter, int4* out,
                                              int* only_entry, int lane) {
  for (int t = 0; t < 4; t++) {
    const unsigned bal = __ballot_sync(0xffffffffu, ok && type == t);
    if (!bal) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&s.flags[counter + t], (unsigned long long)__popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (ok && type == t) {
      const int64_t at = (int64_t)(s.flags[FLAG_TOFS + t] + base) + __popc(bal & ((1u << lane) - 1u));
      if (only_entry) {
        only_entry[at] = a.x;
      } else {
        out[2 * at] = a;
        out[2 * at + 1] = b;
      }
    }
  }
}

// Lane-wise position in four type lists laid one after the other, each padded
// to whole warps: warp w of the launch gets the list *t and the place *r in it
// (r >= cnt[t]: none), so that no warp mixes types -- a warp issues every
// type's FP64 instructions one after the other, and in a small scene its time
// is the step's.
__device__ __forceinline__ int64_t padded_total(const int64_t* cnt) {
  int64_t n = 0;
#pragma unroll
  for (int t = 0; t < 4; t++) n += (cnt[t] + 31) & ~(int64_t)31;
  return n;
}
__device__ __forceinline__ void padded_place(const int64_t* cnt, int64_t base, int lane, int* t, int64_t* r) {
  int64_t b = base;
  int u = 0;
#pragma unroll
  for (int q = 0; q < 3; q++)
    if (u == q) {
      const int64_t len = (cnt[q] + 31) & ~(int64_t)31;
      if (b >= len) {
        b -= len;
        u = q + 1;
      }
    }
  *t = u;
  *r = b + lane;
}

// The records of the entries that the step's narrow phase has to compute
// (k_near_entries lists them by type): its threads call full on dense warps,
// and the last block to finish empties the lists for the next step.
template <class Full>
__device__ __forceinline__ void near_narrow(const Scene& s, Full full) {
  int64_t cnt[4];
#pragma unroll
  for (int t = 0; t < 4; t++) cnt[t] = (int64_t)s.flags[FLAG_NSLOW + t];
  const int64_t total = padded_total(cnt);
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < total; base += stride) {
    int t;
    int64_t r;
    padded_place(cnt, base, lane, &t, &r);
    bool active = false;
    const int64_t len = t == 0 ? cnt[0] : t == 1 ? cnt[1] : t == 2 ? cnt[2] : cnt[3];
    if (r < len) {
      const int64_t at = (int64_t)s.flags[FLAG_TOFS + t] + r;
      active = full(s.srec[2 * at], s.srec[2 * at + 1]);
    }
    const unsigned m = __ballot_sync(0xffffffffu, active);
    if (lane == 0 && m) atomicAdd(&s.flags[FLAG_NACTIVE], (unsigned long long)__popc(m));
  }
  __syncthreads();  // every thread of the block has read the counts
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&s.flags[FLAG_SLOW_TICKET], 1ull) == gridDim.x - 1ull) {
      for (int t = 0; t < 4; t++) s.flags[FLAG_NSLOW + t] = 0ull;
      s.flags[FLAG_SLOW_TICKET] = 0ull;
    }
  }
}

}  // namespace rk
