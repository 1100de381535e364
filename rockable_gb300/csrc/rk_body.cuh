// rk_body.cuh -- per-body kernels of the step (drift, world vertices of the
// listed bodies, resultants + Newton-Euler + second half-kick with the fused
// learned-skin guard), included twice: by rk_step.cu, compiled without
// contraction into fused multiply-adds (kernels in rk::exact, the FP64 form
// that reproduces the reference arithmetic bit for bit), and by rk_fast.cu,
// compiled with it (rk::fused: only the world-vertex kernel, with
// RK_BODY_GLOB_ONLY defined; the mixed form has its own drift and resultant
// kernels there).  Define RK_BODY_NS before including.
#ifndef RK_BODY_HELPERS
#define RK_BODY_HELPERS
#include "rk_engine.cuh"
#include "rk_guard.cuh"
#include "rk_near.cuh"

namespace rk {

__device__ __forceinline__ V3 ld3(const double* a, int64_t k) { return v3(a[3 * k], a[3 * k + 1], a[3 * k + 2]); }
__device__ __forceinline__ void st3(double* a, int64_t k, V3 v) {
  a[3 * k] = v.x;
  a[3 * k + 1] = v.y;
  a[3 * k + 2] = v.z;
}
__device__ __forceinline__ Q4 ldq(const double* a, int64_t k) {
  return q4(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
}
__device__ __forceinline__ void stq(double* a, int64_t k, Q4 q) {
  a[4 * k] = q.s;
  a[4 * k + 1] = q.v.x;
  a[4 * k + 2] = q.v.y;
  a[4 * k + 3] = q.v.z;
}

__device__ __forceinline__ V3 euler_domega(V3 I, V3 w, V3 M) {
  return v3((M.x - (I.z - I.y) * w.y * w.z) / I.x, (M.y - (I.x - I.z) * w.z * w.x) / I.y,
            (M.z - (I.y - I.x) * w.x * w.y) / I.z);
}

// The body force plugin's force and moment on free body b, each starting at
// zero (the plugins' getForceAndMoment).
__device__ __forceinline__ void body_force(const Scene& s, int64_t b, V3& f, V3& m) {
  f = v3(0, 0, 0);
  m = v3(0, 0, 0);
  const double* p = s.bf;
  if (s.bf_kind == RK_BF_ATTRACTING_POINT) {  // BodyForce_AttractingPoint.cpp:51-59
    V3 d = v3(p[0], p[1], p[2]) - ld3(s.pos, b);
    const double l2 = norm2(d);
    if (l2 > 0.0) {
      d = d * (1.0 / sqrt(l2));
      f = (s.mass[b] * p[3]) * d;
    }
  } else if (s.bf_kind == RK_BF_PREFERRED_DIRECTION) {  // BodyForce_PreferredDirection.cpp:58-80
    V3 axisB = qrot(ldq(s.Q, b), v3(p[0], p[1], p[2]));
    normalize(axisB);
    const V3 axis = v3(p[3], p[4], p[5]);
    V3 u = cross(axis, axisB);
    normalize(u);
    const double cosa = dot(axisB, axis);
    double angle = acos(cosa);
    double sgn = -1.0;
    if (cosa < 0.0) {
      sgn = 1.0;
      angle = p[7] - angle;
    }
    m = ((p[6] * sgn) * u) * angle;
  } else if (s.bf_kind == RK_BF_VISCOUS_FLUID) {  // BodyForce_ViscousFluid.cpp:47-58
    const V3 v = ld3(s.vel, b);
    f = ((p[0] * p[1]) * s.bf_surf[b]) * v3(v.x * v.x, v.y * v.y, v.z * v.z);
  }
}

// Imposed force / moment components of a driven body (Rockable.cpp:2904-2928);
// a free body starts from the body force (Rockable.cpp:2887-2901: zero plus
// the plugin's force and moment).
__device__ __forceinline__ void init_resultant(const Scene& s, int64_t b, V3& F, V3& M) {
  F = v3(0, 0, 0);
  M = v3(0, 0, 0);
  if (b >= s.n_driven) {
    if (s.bf_kind != RK_BF_NONE) {
      V3 f, m;
      body_force(s, b, f, m);
      F = F + f;
      M = M + m;
    }
    return;
  }
  for (int k = 0; k < s.ncontrols; k++) {
    const Control c = s.controls[k];
    if (c.body != b) continue;
    switch (c.type) {
      case RK_X_FOR: F.x = c.value; break;
      case RK_Y_FOR: F.y = c.value; break;
      case RK_Z_FOR: F.z = c.value; break;
      case RK_XROT_MOM: M.x = c.value; break;
      case RK_YROT_MOM: M.y = c.value; break;
      case RK_ZROT_MOM: M.z = c.value; break;
      case RK_XYZROT_MOM: M = v3(c.vec[0], c.vec[1], c.vec[2]); break;
      default: break;
    }
  }
}

// Resultant force and moment of body b (is_heavy 0 or 1) in the serial order.
__device__ __forceinline__ void body_resultant(const Scene& s, int64_t b, V3& F, V3& M) {
  if (s.is_heavy[b]) {  // summed by k_gather_heavy, in the same order
    F = ld3(s.force, b);
    M = ld3(s.moment, b);
  } else {
    init_resultant(s, b, F, M);
    // Resultants in the serial order of the active entries (key order): the
    // j-side entries before b's own block, b's block, the remaining j-side.
    // Four positions of that sequence are loaded together, then added in
    // order (same sums, a quarter of the dependent load chains).
    const int64_t i0 = s.iofs[b], i1 = s.iofs[b + 1];
    const int64_t j0 = s.jofs[b], j1 = s.jofs[b + 1], js = s.jsplit[b];
    const int64_t nA = js - j0, nAB = nA + (i1 - i0), L = nAB + (j1 - js);
    for (int64_t p0 = 0; p0 < L; p0 += 4) {
      int64_t e[4];
      bool jside[4], on[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int64_t p = p0 + u;
        on[u] = p < L;
        jside[u] = p < nA || p >= nAB;
        e[u] = !on[u] ? 0 : (p < nA ? (int64_t)s.jlist[j0 + p] : (p < nAB ? i0 + (p - nA) : (int64_t)s.jlist[js + (p - nAB)]));
      }
      bool a[4];
#pragma unroll
      for (int u = 0; u < 4; u++) a[u] = on[u] && s.act[e[u]];
      V3 f[4], m[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (a[u]) {
          f[u] = ld3(s.cf, e[u]);
          m[u] = jside[u] ? ld3(s.cmj, e[u]) : ld3(s.cmi, e[u]);
        } else {
          f[u] = v3(0, 0, 0);
          m[u] = v3(0, 0, 0);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (!a[u]) continue;
        F = jside[u] ? F - f[u] : F + f[u];
        M = M + m[u];
      }
    }
  }
}

__device__ __forceinline__ void finish_body(const Scene& s, int64_t b, V3 F, V3 M, int apply_kick,
                                            float* kin = nullptr);
__device__ __forceinline__ void gather_body(const Scene& s, int64_t b, int apply_kick) {
  if (s.is_heavy[b] == 2) {
    // a driven body whose resultant feeds no state (no force / moment
    // control): summed on demand by k_gather_heavy when downloaded
    st3(s.acc, b, v3(0, 0, 0));
    st3(s.arot, b, v3(0, 0, 0));
    return;
  }
  V3 F, M;
  body_resultant(s, b, F, M);
  finish_body(s, b, F, M, apply_kick);
}

// Newton-Euler and the second half-kick of body b from its resultant; kin
// (may be null): a free body's velocity, acceleration, angular velocity and
// angular acceleration after the step, as floats, for the skin's guard.
__device__ __forceinline__ void finish_body(const Scene& s, int64_t b, V3 F, V3 M, int apply_kick, float* kin) {
  const bool driven = b < s.n_driven;
  const double fm = 1.0 - s.num_damp, fp = 1.0 + s.num_damp;
  const V3 vel = ld3(s.vel, b), vrot = ld3(s.vrot, b);
  const double mass = s.mass[b];
  const V3 inertia = ld3(s.inertia, b);
  const Q4 q = ldq(s.Q, b);
  if (driven) {
    V3 acc = v3(0, 0, 0), arot = v3(0, 0, 0);
    if (s.num_damp > 0.0) {  // Rockable.cpp:3814-3835
      for (int k = 0; k < s.ncontrols; k++) {
        const Control c = s.controls[k];
        if (c.body != b) continue;
        if (c.type == RK_X_FOR) F.x *= (F.x * vel.x > 0.0) ? fm : fp;
        else if (c.type == RK_Y_FOR) F.y *= (F.y * vel.y > 0.0) ? fm : fp;
        else if (c.type == RK_Z_FOR) F.z *= (F.z * vel.z > 0.0) ? fm : fp;
      }
    }
    for (int k = 0; k < s.ncontrols; k++) {  // Rockable.cpp:3448-3507
      const Control c = s.controls[k];
      if (c.body != b) continue;
      switch (c.type) {
        case RK_X_FOR: acc.x = F.x / mass; break;
        case RK_Y_FOR: acc.y = F.y / mass; break;
        case RK_Z_FOR: acc.z = F.z / mass; break;
        case RK_XROT_MOM: case RK_YROT_MOM: case RK_ZROT_MOM: case RK_XYZROT_MOM: {
          Q4 qi = qconj(q);
          V3 w;
          if (c.type == RK_XROT_MOM) w = v3(vrot.x, 0.0, 0.0);
          else if (c.type == RK_YROT_MOM) w = v3(0.0, vrot.y, 0.0);
          else if (c.type == RK_ZROT_MOM) w = v3(0.0, 0.0, vrot.z);
          else w = vrot;
          V3 om = qrot(qi, w);
          V3 Mb = qrot(qi, M);
          V3 dw = qrot(q, euler_domega(inertia, om, Mb));
          if (c.type == RK_XROT_MOM) arot.x = dw.x;
          else if (c.type == RK_YROT_MOM) arot.y = dw.y;
          else if (c.type == RK_ZROT_MOM) arot.z = dw.z;
          else arot = dw;
        } break;
        default: break;
      }
    }
    V3 v = vel, wr = vrot;
    if (apply_kick) {  // Rockable.cpp:2084-2117
      for (int k = 0; k < s.ncontrols; k++) {
        const Control c = s.controls[k];
        if (c.body != b) continue;
        switch (c.type) {
          case RK_X_FOR: v.x += s.dt_2 * acc.x; break;
          case RK_Y_FOR: v.y += s.dt_2 * acc.y; break;
          case RK_Z_FOR: v.z += s.dt_2 * acc.z; break;
          case RK_XROT_MOM: wr.x += s.dt_2 * arot.x; break;
          case RK_YROT_MOM: wr.y += s.dt_2 * arot.y; break;
          case RK_ZROT_MOM: wr.z += s.dt_2 * arot.z; break;
          case RK_XYZROT_MOM: wr = wr + s.dt_2 * arot; break;
          default: break;
        }
      }
    }
    st3(s.acc, b, acc);
    st3(s.arot, b, arot);
    st3(s.vel, b, v);
    st3(s.vrot, b, wr);
  } else {
    if (s.num_damp > 0.0) {  // Rockable.cpp:3837-3866
      double factor = (dot(F, vel) > 0.0) ? fm : fp;
      F = F * factor;
      factor = (dot(M, vrot) > 0.0) ? fm : fp;
      M = M * factor;
    }
    V3 acc = vdiv(F, mass) + v3(s.gravity[0], s.gravity[1], s.gravity[2]);
    Q4 qi = qconj(q);
    V3 om = qrot(qi, vrot);
    V3 Mb = qrot(qi, M);
    V3 arot = qrot(q, euler_domega(inertia, om, Mb));
    st3(s.acc, b, acc);
    st3(s.arot, b, arot);
    V3 v = vel, wr = vrot;
    if (apply_kick) {
      v = vel + s.dt_2 * acc;
      wr = vrot + s.dt_2 * arot;
      st3(s.vel, b, v);
      st3(s.vrot, b, wr);
    }
    if (kin) {
      const V3 k[4] = {v, acc, wr, arot};
#pragma unroll
      for (int d = 0; d < 4; d++) {
        kin[3 * d] = d2f(k[d].x);
        kin[3 * d + 1] = d2f(k[d].y);
        kin[3 * d + 2] = d2f(k[d].z);
      }
    }
  }
  st3(s.force, b, F);
  st3(s.moment, b, M);
}

}  // namespace rk
#endif  // RK_BODY_HELPERS

namespace rk {
namespace RK_BODY_NS {

#ifndef RK_BODY_GLOB_ONLY
// ----------------------------------------------------------------- K1 ----
__device__ __forceinline__ BodyState drift_body(const Scene& s, int64_t i) {
  V3 p = ld3(s.pos, i), v = ld3(s.vel, i), a = ld3(s.acc, i);
  V3 w = ld3(s.vrot, i), al = ld3(s.arot, i);
  Q4 q = ldq(s.Q, i);
  const Q4 q0 = q;
  float path = s.sk_path ? s.sk_path[i] : 0.f;
  const V3 dx = s.dt * v + s.dt2_2 * a;
  p = p + dx;
  v = v + s.dt_2 * a;
  qaddscaled(q, qdot(q, w), s.dt);
  qaddscaled(q, qddot(q, w, al), s.dt2_2);
  qnormalize(q);
  w = w + s.dt_2 * al;
  if (s.sk_path) {
    // learned-skin path bound: |dx| plus the rotation angle of the step
    // (at most 2c(1 + c) for the chord c = |q - q0| of unit quaternions)
    // times the swing radius, rounded up
    const float cx = d2f(q.s - q0.s), cy = d2f(q.v.x - q0.v.x), cz = d2f(q.v.y - q0.v.y), cw = d2f(q.v.z - q0.v.z);
    const float c = sqrtf(cx * cx + cy * cy + cz * cz + cw * cw);
    const float ex = d2f(dx.x), ey = d2f(dx.y), ez = d2f(dx.z);
    const float inc = sqrtf(ex * ex + ey * ey + ez * ez) + 2.f * c * (1.f + c) * s.sk_rsw[i];
    path += inc * (1.f + 1e-5f) + 1e-12f;
    s.sk_path[i] = path;
  }
  st3(s.pos, i, p);
  st3(s.vel, i, v);
  stq(s.Q, i, q);
  st3(s.vrot, i, w);
  return {{p.x, p.y, p.z}, {v.x, v.y, v.z}, {q.s, q.v.x, q.v.y, q.v.z}, {w.x, w.y, w.z}, path};
}
// the free bodies' drift; every body's part of the near set's check and of a
// batched skin step's guard (GUARD).  What these compare with is loaded before
// the drift's stores, so that it shares the drift's round of loads (loaded
// after them, scenes of 3000 to 200 000 bodies take the same time within 1 %,
// 22 000 to 30 000 up to 1 % more).
template <bool GUARD>
__global__ void k_drift(Scene s) {
  if (GUARD && batch_halted(s)) return;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  BodyState k = {};
  SkinRef ref = {};
  if (i < s.n) {
    const NearRef near = near_ref(s, i);
    if (GUARD) ref = skin_ref(s, i);
    k = i >= s.n_driven ? drift_body(s, i) : body_state(s, i);
    near_track(s, i, k, near);
  }
  if (GUARD) skin_guard_drift(s, i < s.n ? i : s.n, k, ref);
}

#endif  // RK_BODY_GLOB_ONLY

// global vertex k of body b: pos + Q (h v)
// With only_listed, the vertices of s.lv (the bodies with neighbour-list
// entries): within a step only the narrow phase reads these positions, and
// only for bodies in the list; a list update recomputes every body first
// (a partial refresh, the bodies of its pairs: `mark`).
__global__ void k_glob_vertices(Scene s, int only_listed, const uint8_t* mark) {
  if (step_halted(s)) return;
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= (only_listed ? s.nlv : s.nvert)) return;
  if (only_listed) k = s.lv[k];
  int b = s.gv_body[k];
  if (mark && !mark[b]) return;
  const V3 u = v3(s.uv64[3 * k], s.uv64[3 * k + 1], s.uv64[3 * k + 2]);  // h v, computed at upload
  V3 r = qrot(ldq(s.Q, b), u);
  V3 g = ld3(s.pos, b) + r;
  st3(s.gv, k, g);
  if (s.gvr) {
    s.gvr[3 * k] = (float)r.x;
    s.gvr[3 * k + 1] = (float)r.y;
    s.gvr[3 * k + 2] = (float)r.z;
  }
}

#ifndef RK_BODY_GLOB_ONLY
__global__ void k_gather_accel(Scene s, int apply_kick) {
  if (step_halted(s)) return;
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b < s.n) gather_body(s, b, apply_kick);
  // the learned skin's guard on the state this step leaves (all lanes)
  if (s.sk_out && apply_kick && !s.sk_ctl) skin_guard_body(s, b < s.n ? b : s.n);
  if (s.sk_ctl) skin_batch_step_end(s);
}

// The same on the near set: a body's few near entries (glist, in the serial
// order) instead of its whole list.
//   Sums: 8 lanes per body look at 32 positions together (whole lists: 64),
// queue the active ones, a few of them, in order, load 8 of these at a time,
// and lanes 0-5 add one component each in the serial order: one FP64
// instruction per contact instead of six, and a single chain of loads (word,
// flag, force) for the lists that most bodies have; one per 8 positions
// measured 13.2 instead of 12.2 us at 6000 blocks and 1.7 % more a step at
// 1700 grains.
// (A warp-wide FP64 instruction holds its scheduler for 64 cycles
// on GB300 however many lanes it has and however independent it is.)
//   Update: then one thread per body.
// That is kBodies = 16 per block, for scenes that 8 such blocks per SM hold.
// Larger scenes (kBodies = 128) have warps enough for one thread per body
// throughout, whose updates fill their warps (50 000 grains: 34 us, against
// 43 us in blocks of 32 bodies).
// The first nbig blocks take a big body each (walls under force control:
// thousands of entries): the whole block loads 128 positions at a time and
// packs the active ones in shared memory, and six lanes add them in the
// serial order while the next positions are on their way.
// Bodies whose resultant the step does not use (driven, no force or moment
// control) have no state to update.
// 3000 grains 42 us (GEOM list, thread per body) before; the box of 200 000
// grains 1.19 ms on whole lists with shuffles instead of shared memory.
// WHOLE: the same on the whole list, for small scenes (kBodies = 16): every
// body that is not deferred (is_heavy 2), its positions found through the
// serial order.
constexpr int kGatherNear = 128;
template <int kBodies, bool WHOLE>
__global__ void __launch_bounds__(kGatherNear) k_gather_near(Scene s, int apply_kick) {
  if (step_halted(s)) return;
  __shared__ double sh[2][kGatherNear][6];
  __shared__ double res[kBodies == kGatherNear ? 1 : kBodies][6];
  __shared__ int wcnt[2][kGatherNear / 32];
  constexpr int kAhead = WHOLE ? 8 : 4;  // positions a lane looks at together
  __shared__ int queue[kBodies == kGatherNear ? 1 : kGatherNear / 8][8 * kAhead];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t guard = s.n;
  float kin[12] = {};  // the guard's velocities and accelerations of a free body
  bool have = false;
  double sum[6] = {0, 0, 0, 0, 0, 0};  // the resultant of body `guard`
  double c[6];
  bool on = false;
  // position p of a list (WHOLE: of the body whose offsets are in `own`), and
  // what its entry adds
  int64_t own[5] = {0, 0, 0, 0, 0};  // j-side positions before the own block, end of the block, iofs, jofs, jsplit
  auto word = [&](const int* list, int p) {
    if (!WHOLE) return list[p];
    if (p < own[0]) return (int)(s.jlist[own[3] + p] | 0x80000000);
    if (p < own[1]) return (int)(own[2] + (p - own[0]));
    return (int)(s.jlist[own[4] + (p - own[1])] | 0x80000000);
  };
  auto contribution = [&](int x) {
    const int64_t e = x & kGlistEntry;
    const bool jside = x < 0;
    const V3 f = ld3(s.cf, e), m = ld3(jside ? s.cmj : s.cmi, e);
    c[0] = jside ? -f.x : f.x; c[1] = jside ? -f.y : f.y; c[2] = jside ? -f.z : f.z;
    c[3] = m.x; c[4] = m.y; c[5] = m.z;
  };
  auto fetch = [&](const int* list, int p, int L) {
    on = false;
    if (p >= L) return;
    const int x = word(list, p);
    on = s.act[x & kGlistEntry] != 0;
    if (on) contribution(x);
  };
  // whether the step uses body b's resultant, and the length of its list
  auto used = [&](int64_t b) { return WHOLE ? s.is_heavy[b] != 2 : s.needres[b] != 0; };
  auto list_of = [&](int64_t b, int& L) -> const int* {
    if (!WHOLE) {
      L = s.gcnt[b];
      return s.glist + s.iofs[b] + s.jofs[b];
    }
    own[2] = s.iofs[b];
    own[3] = s.jofs[b];
    own[4] = s.jsplit[b];
    own[0] = own[4] - own[3];
    own[1] = own[0] + (s.iofs[b + 1] - own[2]);
    L = (int)(own[1] + (s.jofs[b + 1] - own[4]));
    return nullptr;
  };
  auto component = [&](V3 F, V3 M, int d) {
    return d == 0 ? F.x : d == 1 ? F.y : d == 2 ? F.z : d == 3 ? M.x : d == 4 ? M.y : M.z;
  };
  if ((int)blockIdx.x < s.nbig) {
    const int64_t b = s.big[blockIdx.x];
    int L;
    const int* list = list_of(b, L);
    V3 F, M;
    init_resultant(s, b, F, M);
    double acc = component(F, M, lane);
    fetch(list, threadIdx.x, L);
    int buf = 0;
    for (int p0 = 0; p0 < L; p0 += kGatherNear, buf ^= 1) {
      const unsigned bal = __ballot_sync(0xffffffffu, on);
      if (lane == 0) wcnt[buf][warp] = __popc(bal);
      __syncthreads();
      int at = __popc(bal & ((1u << lane) - 1u)), all = 0;
      for (int w = 0; w < kGatherNear / 32; w++) {
        if (w < warp) at += wcnt[buf][w];
        all += wcnt[buf][w];
      }
      if (on)
#pragma unroll
        for (int d = 0; d < 6; d++) sh[buf][at][d] = c[d];
      __syncthreads();
      fetch(list, p0 + kGatherNear + threadIdx.x, L);
      if (warp == 0 && lane < 6) {
        int k = 0;
        for (; k + 8 <= all; k += 8) {
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; u++) v[u] = sh[buf][k + u][lane];
#pragma unroll
          for (int u = 0; u < 8; u++) acc = acc + v[u];
        }
        for (; k < all; k++) acc = acc + sh[buf][k][lane];
      }
    }
    if (warp == 0 && lane < 6) res[0][lane] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      guard = b;
#pragma unroll
      for (int d = 0; d < 6; d++) sum[d] = res[0][d];
    }
  } else {
    const int64_t b0 = ((int64_t)blockIdx.x - s.nbig) * kBodies;
    if constexpr (kBodies == kGatherNear) {  // (near set only)
      const int64_t b = b0 + threadIdx.x;
      if (b < s.n) {
        const int64_t base = s.iofs[b] + s.jofs[b];
        const bool take = s.needres[b] != 0;
        if (!(take && s.iofs[b + 1] + s.jofs[b + 1] - base > kNearBig)) guard = b;
        if (take && guard == b) {
          const int L = s.gcnt[b];
          const int* list = s.glist + base;
          V3 F, M;
          init_resultant(s, b, F, M);
          for (int p0 = 0; p0 < L; p0 += 4) {  // four positions loaded together, added in order
            int x[4];
            bool a[4];
            V3 f[4], m[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = p0 + u < L ? list[p0 + u] : 0;
#pragma unroll
            for (int u = 0; u < 4; u++) a[u] = p0 + u < L && s.act[x[u] & kGlistEntry];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int64_t e = x[u] & kGlistEntry;
              f[u] = a[u] ? ld3(s.cf, e) : v3(0, 0, 0);
              m[u] = a[u] ? ld3(x[u] < 0 ? s.cmj : s.cmi, e) : v3(0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
              if (!a[u]) continue;
              F = x[u] < 0 ? F - f[u] : F + f[u];
              M = M + m[u];
            }
          }
          const double r[6] = {F.x, F.y, F.z, M.x, M.y, M.z};
#pragma unroll
          for (int d = 0; d < 6; d++) sum[d] = r[d];
        }
      }
    } else {
      const int g = threadIdx.x >> 3, l = threadIdx.x & 7, shift = lane & 24;
      double(*stage)[6] = &sh[0][8 * g];  // this group's 8 contributions
      for (int r = 0; r < kBodies; r += kGatherNear / 8) {
        const int64_t b = b0 + r + g;
        const int* list = nullptr;
        int L = 0;
        double acc = 0.0;
        if (b < s.n && used(b)) {
          if (!(s.needres[b] && s.iofs[b + 1] + s.jofs[b + 1] - s.iofs[b] - s.jofs[b] > kNearBig)) {
            list = list_of(b, L);
            if (b < s.n_driven || s.bf_kind != RK_BF_NONE) {
              V3 F, M;
              init_resultant(s, b, F, M);
              acc = component(F, M, l);
            }
          }
        }
        int Lw = L;  // positions of the warp's longest list
        Lw = max(Lw, __shfl_xor_sync(0xffffffffu, Lw, 8));
        Lw = max(Lw, __shfl_xor_sync(0xffffffffu, Lw, 16));
        for (int p0 = 0; p0 < Lw; p0 += 8 * kAhead) {
          int x[kAhead];
          bool a[kAhead];
#pragma unroll
          for (int u = 0; u < kAhead; u++) x[u] = p0 + 8 * u + l < L ? word(list, p0 + 8 * u + l) : 0;
#pragma unroll
          for (int u = 0; u < kAhead; u++) a[u] = p0 + 8 * u + l < L && s.act[x[u] & kGlistEntry];
          int cnt = 0;
#pragma unroll
          for (int u = 0; u < kAhead; u++) {
            const unsigned bal = (__ballot_sync(0xffffffffu, a[u]) >> shift) & 0xffu;
            if (a[u]) queue[g][cnt + __popc(bal & ((1u << l) - 1u))] = x[u];
            cnt += __popc(bal);
          }
          __syncwarp();
          int most = cnt;
          most = max(most, __shfl_xor_sync(0xffffffffu, most, 8));
          most = max(most, __shfl_xor_sync(0xffffffffu, most, 16));
          for (int m = 0; m < most; m += 8) {
            if (m + l < cnt) {
              contribution(queue[g][m + l]);
#pragma unroll
              for (int d = 0; d < 6; d++) stage[l][d] = c[d];
            }
            __syncwarp();
            if (l < 6)
              for (int k = 0; k < min(cnt - m, 8); k++) acc = acc + stage[k][l];
            __syncwarp();
          }
        }
        if (l < 6) res[r + g][l] = acc;
      }
      __syncthreads();
      if (threadIdx.x < kBodies) {
        const int64_t b = b0 + threadIdx.x;
        if (b < s.n && !(s.needres[b] && s.iofs[b + 1] + s.jofs[b + 1] - s.iofs[b] - s.jofs[b] > kNearBig)) {
          guard = b;
#pragma unroll
          for (int d = 0; d < 6; d++) sum[d] = res[threadIdx.x][d];
        }
      }
    }
  }
  if (guard < s.n && used(guard)) {
    finish_body(s, guard, v3(sum[0], sum[1], sum[2]), v3(sum[3], sum[4], sum[5]), apply_kick, kin);
    have = guard >= s.n_driven;
  } else if (WHOLE && guard < s.n) {
    // a driven body whose resultant feeds no state: summed on demand
    st3(s.acc, guard, v3(0, 0, 0));
    st3(s.arot, guard, v3(0, 0, 0));
  }
  if (s.sk_out && apply_kick && !s.sk_ctl) skin_guard_body(s, guard, have, kin);
  if (WHOLE && s.sk_ctl) skin_batch_step_end(s);
}

#endif  // RK_BODY_GLOB_ONLY

}  // namespace RK_BODY_NS
}  // namespace rk
