// rk_cand.cuh -- candidate sub-contacts of the neighbour-list rebuild: float
// NEAR tests and classification, and the kernel that lists the candidates.
//
// Included twice: by rk_cand.cu, with fused multiply-adds, for Rockable's NEAR
// predicates (there the float arithmetic only classifies, with margins; what
// it leaves undecided is decided in FP64 by rk_nl.cu), and by rk_nl.cu,
// without them, for the learned skin's distance-only tests (whose float
// result is the list).
#pragma once
#include "rk_bits.cuh"
#include "rk_engine.cuh"

namespace rk {

// ------------------------------------------ geometric NEAR (skin mode) ----
// Distance-only tests on float coordinates (the vertex spheres' centres are
// the vertices): vertex-vertex, vertex-segment, vertex-polygon and
// segment-segment distances against R_b + R_p + dVerlet plus a rounding
// margin.  Rockable's NEAR predicates also require the projection of a
// vertex inside the face, or the closest points inside both edges, so a
// sub-contact can start to touch after an arbitrarily small sliding motion;
// with distances only, every sub-contact that touches now was within
// dVerlet of touching at its last test whenever the motion since is below
// dVerlet -- what makes the learned-skin guard exact.  Used only with the
// learned skin; the plain and mixed forms keep the reference predicates.
struct G3 {
  float x, y, z;
};
__device__ __forceinline__ G3 gsub(G3 a, G3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ G3 gmad(G3 a, float t, G3 d) { return {a.x + t * d.x, a.y + t * d.y, a.z + t * d.z}; }
__device__ __forceinline__ float gdot(G3 a, G3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ G3 gcross(G3 a, G3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ G3 gpt(float4 a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ float clamp01(float t) { return fminf(fmaxf(t, 0.f), 1.f); }

__device__ __forceinline__ float pt_seg_d2(G3 p, G3 a, G3 b) {
  const G3 ab = gsub(b, a), ap = gsub(p, a);
  const float l2 = gdot(ab, ab);
  const float t = l2 > 0.f ? clamp01(gdot(ap, ab) / l2) : 0.f;
  const G3 d = gmad(ap, -t, ab);
  return gdot(d, d);
}

// squared distance of a point to the line through a and b
__device__ __forceinline__ float pt_line_d2(G3 p, G3 a, G3 b) {
  const G3 ab = gsub(b, a), ap = gsub(p, a);
  const float l2 = gdot(ab, ab);
  const float t = l2 > 0.f ? gdot(ap, ab) / l2 : 0.f;
  const G3 d = gmad(ap, -t, ab);
  return gdot(d, d);
}

// true when the lines through two segments are farther apart than sqrt(lim2)
// (the line distance bounds the segment distance from below); never for
// nearly parallel lines, where that distance is ill-conditioned
__device__ __forceinline__ bool lines_far(G3 p1, G3 q1, G3 p2, G3 q2, float lim2) {
  const G3 d1 = gsub(q1, p1), d2 = gsub(q2, p2), r = gsub(p1, p2);
  const G3 n = gcross(d1, d2);
  const float nn = gdot(n, n);
  if (!(nn > 1e-6f * gdot(d1, d1) * gdot(d2, d2))) return false;
  const float rn = gdot(r, n);
  return rn * rn > lim2 * nn;
}

// Float classification in front of the FP64 NEAR predicates (Rockable's,
// above): from the float world coordinates of the sub-elements (the vertex
// spheres' centres, rounded to nearest from the FP64 world vertices: errors
// of a few 1e-8 of the coordinates' magnitude `mag`), each returns 1 only
// when the FP64 predicate is true for sure -- its distance within `alim` (the
// NEAR distance shrunk by the rejection's rounding margin) and its projection
// parameters or point inside their ranges by more than their rounding error
// -- and -1 only when it is false for sure: a projection parameter or point
// outside its range by more than that error.  On 0 the FP64 predicate
// decides.  (The distance rejections sit at the call sites.)
__device__ __forceinline__ bool accept_vv(G3 a, G3 b, float alim) {
  const G3 d = gsub(a, b);
  return alim > 0.f && gdot(d, d) <= alim * alim;
}
__device__ __forceinline__ int classify_ve(G3 p, G3 a, G3 b, float alim, float dmax, float mag) {
  const G3 E = gsub(b, a), w = gsub(p, a);
  const float E2 = gdot(E, E);
  if (!(E2 > 0.f)) return 0;
  const float r = gdot(w, E) / E2;
  const float tol = 1e-5f + 4e-6f * mag * rsqrtf(E2) * (1.f + fabsf(r));
  if (r < -dmax - tol || r > 1.f + dmax + tol) return -1;  // the FP64 projection test fails too
  if (!(alim > 0.f) || !(r >= -dmax + tol && r <= 1.f + dmax - tol)) return 0;
  const G3 d = gmad(w, -r, E);
  return gdot(d, d) <= alim * alim ? 1 : 0;
}
__device__ __forceinline__ int classify_vf_tri(G3 p, G3 A, G3 B, G3 C, float alim, float mag) {
  const G3 bA = gsub(B, A), cA = gsub(C, A), w = gsub(p, A);
  G3 n = gcross(bA, cA);
  const float nn = gdot(n, n);
  // a well-shaped triangle (the sine of its angle at A above 1e-3), so that
  // the float normal and in-plane distances carry only rounding errors
  if (!(nn > 1e-6f * gdot(bA, bA) * gdot(cA, cA))) return 0;
  const float inv = rsqrtf(nn);
  n = {n.x * inv, n.y * inv, n.z * inv};
  const float dist = gdot(w, n);
  const G3 P = gmad(w, -dist, n);
  const float tol = 1e-9f + 2e-6f * mag;
  const G3 ed[3] = {bA, gsub(cA, bA), {-cA.x, -cA.y, -cA.z}};
  const G3 st[3] = {{0.f, 0.f, 0.f}, bA, cA};
  bool inside = true;
  for (int q = 0; q < 3; q++) {  // counter-clockwise about n: inside is to the left of every edge
    const float side = gdot(gcross(ed[q], gsub(P, st[q])), n) * rsqrtf(gdot(ed[q], ed[q]));
    if (side < -tol) return -1;  // projection outside the triangle: even crossing number in FP64 too
    inside = inside && side > tol;
  }
  return inside && alim > 0.f && fabsf(dist) <= alim ? 1 : 0;
}
__device__ __forceinline__ int classify_ee(G3 pi0, G3 pi1, G3 pj0, G3 pj1, float alim, float mag) {
  const G3 Ei = gsub(pi1, pi0), Ej = gsub(pj1, pj0), w = gsub(pi0, pj0);
  const float c = gdot(Ei, Ei), d = gdot(Ej, Ej), e = gdot(Ei, Ej);
  const float f = c * d - e * e;
  // well away from the FP64 test's parallel threshold (1e-12) and from
  // parallel edges (the sine of their angle above 0.1)
  if (!(f > 2e-12f + 0.01f * c * d)) return 0;
  const float a = gdot(Ei, w), b = gdot(Ej, w);
  const float fi = 1.f / f;
  const float ss = (e * b - a * d) * fi, tt = (c * b - e * a) * fi;
  const float tol = 1e-5f + 4e-5f * mag * rsqrtf(fminf(c, d)) * (1.f + fabsf(ss) + fabsf(tt));
  if (ss < -tol || ss > 1.f + tol || tt < -tol || tt > 1.f + tol) return -1;  // closest points off an edge
  if (!(alim > 0.f) || !(ss >= tol && ss <= 1.f - tol && tt >= tol && tt <= 1.f - tol)) return 0;
  const G3 n = gsub(gmad(pi0, ss, Ei), gmad(pj0, tt, Ej));
  return gdot(n, n) <= alim * alim ? 1 : 0;
}

// squared distance of two segments: the closest-point parameters minimise
// |p1 + s d1 - p2 - t d2| over [0,1]^2 (interior stationary point, else the
// best clamped edge of the square)
__device__ __forceinline__ float seg_seg_d2(G3 p1, G3 q1, G3 p2, G3 q2) {
  const G3 d1 = gsub(q1, p1), d2 = gsub(q2, p2), r = gsub(p1, p2);
  const float a = gdot(d1, d1), e = gdot(d2, d2), f = gdot(d2, r), c = gdot(d1, r), b = gdot(d1, d2);
  float s = 0.f, t = 0.f;
  if (a <= 1e-30f && e <= 1e-30f) {
    s = t = 0.f;
  } else if (a <= 1e-30f) {
    t = clamp01(f / e);
  } else if (e <= 1e-30f) {
    s = clamp01(-c / a);
  } else {
    const float den = a * e - b * b;
    s = den > 0.f ? clamp01((b * f - c * e) / den) : 0.f;
    t = (b * s + f) / e;
    if (t < 0.f) {
      t = 0.f;
      s = clamp01(-c / a);
    } else if (t > 1.f) {
      t = 1.f;
      s = clamp01((b - c) / a);
    }
  }
  const G3 w = gsub(gmad(p1, s, d1), gmad(p2, t, d2));
  return gdot(w, w);
}

// squared distance of a point to a planar polygon (vertices in order)
__device__ __forceinline__ float pt_poly_d2(const Scene& s, const float4* sp, int sh, int f, G3 p) {
  const int fo = s.face_ofs[sh] + f;
  const int v0 = s.face_vofs[fo], nbv = s.face_vofs[fo + 1] - v0;
  const int* fv = s.face_verts + v0;
  const G3 A = gpt(sp[fv[0]]), B = gpt(sp[fv[1]]), C = gpt(sp[fv[nbv - 1]]);
  G3 n = gcross(gsub(B, A), gsub(C, A));
  const float nn = gdot(n, n);
  float best = 3.0e38f;
  if (nn > 0.f) {
    const float inv = rsqrtf(nn);
    n = {n.x * inv, n.y * inv, n.z * inv};
    const float dist = gdot(gsub(p, A), n);
    // crossing number of the projection, in the plane
    const G3 u = gsub(B, A);
    const float iu = rsqrtf(fmaxf(gdot(u, u), 1e-30f));
    const G3 e1 = {u.x * iu, u.y * iu, u.z * iu};
    const G3 e2 = gcross(n, e1);
    const G3 q = gsub(p, A);
    const float o1 = gdot(q, e1), o2 = gdot(q, e2);
    int odd = 0;
    for (int k = 0; k < nbv; k++) {
      const G3 pa = gsub(gpt(sp[fv[k]]), A), pb = gsub(gpt(sp[fv[k + 1 == nbv ? 0 : k + 1]]), A);
      const float a1 = gdot(pa, e1), b1 = gdot(pb, e1), a2 = gdot(pa, e2), b2 = gdot(pb, e2);
      if ((a2 < o2 && b2 >= o2) || (b2 < o2 && a2 >= o2))
        if (a1 + (o2 - a2) / (b2 - a2) * (b1 - a1) < o1) odd = 1 - odd;
    }
    if (odd) best = dist * dist;
  }
  for (int k = 0; k < nbv; k++)
    best = fminf(best, pt_seg_d2(p, gpt(sp[fv[k]]), gpt(sp[fv[k + 1 == nbv ? 0 : k + 1]])));
  return best;
}

// classify_vf_tri on a face of the partner's shape (triangles only: other
// polygons go to the FP64 predicate)
__device__ __forceinline__ int classify_vf(const Scene& s, const float4* sp, int sh, int f, G3 p, float alim,
                                           float mag) {
  const int fo = s.face_ofs[sh] + f;
  const int v0 = s.face_vofs[fo], nbv = s.face_vofs[fo + 1] - v0;
  if (nbv != 3) return 0;
  const int* fv = s.face_verts + v0;
  return classify_vf_tri(p, gpt(sp[fv[0]]), gpt(sp[fv[1]]), gpt(sp[fv[2]]), alim, mag);
}

constexpr int kCandWarps = 4;  // warps per block
// counters of a candidate pass, after the number of keys: undecided candidates, those the FP64 predicate rejected
constexpr int kCandUnsure = 2, kCandRejected = 3;

// Root-versus-leaf test of the two-level pruning: true when a sub-element
// sphere (centre, radius in .w) lies farther than `reach` from the other
// body's vertex box bx (float: centre, 3 axes, half extents).  The box holds
// that body's core, so such an element is farther than `reach` from every
// sub-element of it; the margin covers the float rounding of the box, the
// centre and the projections.
__device__ __forceinline__ bool box_far(const float* bx, float4 c, float reach, float slack) {
  const float dx = c.x - bx[0], dy = c.y - bx[1], dz = c.z - bx[2];
  float d2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float t = fabsf(dx * bx[3 + 3 * k] + dy * bx[4 + 3 * k] + dz * bx[5 + 3 * k]) - bx[12 + k];
    if (t > 0.f) d2 += t * t;
  }
  float lim = c.w + reach;
  lim = lim + 1e-4f * lim + slack + 1e-6f * (fabsf(dx) + fabsf(dy) + fabsf(dz) + bx[12] + bx[13] + bx[14]);
  return d2 > lim * lim;
}

// One warp's lists in dynamic shared memory, sized by the shapes' largest
// vertex, edge and face counts (fixed 1024-entry lists held the kernel to 4
// blocks per SM), per side: the vertices' coordinates along the pair's
// separating direction (negated for side 0), owner vertices, edges, faces;
// and side 1's vertices as partners.
struct CandLists {
  float* q[2];
  uint16_t *own[2], *other, *e[2], *f[2];
};
__host__ __device__ inline size_t cand_list_bytes(int mv, int me, int mf) {
  return (size_t)((2 * mv * 4 + 2 * (3 * mv + 2 * me + 2 * mf) + 15) / 16 * 16);
}
__device__ __forceinline__ CandLists cand_lists(char* p, int mv, int me, int mf) {
  CandLists L;
  L.q[0] = reinterpret_cast<float*>(p);
  L.q[1] = L.q[0] + mv;
  L.own[0] = reinterpret_cast<uint16_t*>(L.q[1] + mv);
  L.own[1] = L.own[0] + mv;
  L.other = L.own[1] + mv;
  L.e[0] = L.other + mv;
  L.e[1] = L.e[0] + me;
  L.f[0] = L.e[1] + me;
  L.f[1] = L.f[0] + mf;
  return L;
}

// Slab between two bodies' cores along one direction: the owner's vertices
// all lie below bmax, the partner's above pmin (coordinates along the unit
// direction, relative to the partner's centre; also left per vertex in L.q,
// negated for the owner).
struct Slab {
  float bmax, pmin;
};

__device__ __forceinline__ unsigned int slab_ord(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// A direction that separates the vertices of b and p about as far as their
// hulls are apart, by Gilbert's algorithm on the hulls' difference, the whole
// warp on one pair: each step takes the two hulls' extreme vertices along the
// current difference v (a lane per vertex, warp-wide integer min / max
// reductions of ordered float bits) and moves v to the point of the segment
// towards their difference that is nearest the origin.  Any direction gives
// a valid slab; a few steps make it tight enough for the pruning, and the
// search stops once the gap exceeds `enough` (no sub-element can be near).
__device__ __forceinline__ Slab pair_slab(const float4* sb, int nvb, const float4* sp, int nvp, G3 cb, G3 cp,
                                          float enough, float tol, int lane, const CandLists& L) {
  const unsigned full = 0xffffffffu;
  const int b0 = min(lane, nvb - 1), b1 = min(lane + 32, nvb - 1), p0 = min(lane, nvp - 1), p1 = min(lane + 32, nvp - 1);
  const G3 xb0 = gsub(gpt(sb[b0]), cp), xp0 = gsub(gpt(sp[p0]), cp);
  G3 xb1 = xb0, xp1 = xp0;
  if (nvb > 32) xb1 = gsub(gpt(sb[b1]), cp);
  if (nvp > 32) xp1 = gsub(gpt(sp[p1]), cp);
  G3 v = gsub(cp, cb), dir = {0.f, 0.f, 0.f};
  float best = -3.0e38f;
  Slab S = {3.0e38f, -3.0e38f};
  for (int it = 0; it < 12; it++) {
    const float v2 = gdot(v, v);
    if (!(v2 > 1e-20f)) break;
    const float inv = rsqrtf(v2);
    const G3 d = {v.x * inv, v.y * inv, v.z * inv};
    const float tb0 = gdot(xb0, d), tb1 = gdot(xb1, d), tp0 = gdot(xp0, d), tp1 = gdot(xp1, d);
    const bool ub = tb1 > tb0, up = tp1 < tp0;
    const unsigned ob = slab_ord(ub ? tb1 : tb0), op = slab_ord(up ? tp1 : tp0);
    const unsigned mb = __reduce_max_sync(full, ob), mp = __reduce_min_sync(full, op);
    const int lb = __ffs(__ballot_sync(full, ob == mb)) - 1, lp = __ffs(__ballot_sync(full, op == mp)) - 1;
    const float bmax = __shfl_sync(full, ub ? tb1 : tb0, lb), pmin = __shfl_sync(full, up ? tp1 : tp0, lp);
    if (pmin - bmax > best) {
      best = pmin - bmax;
      S.bmax = bmax;
      S.pmin = pmin;
      dir = d;
    }
    const float len = v2 * inv;
    if (best > enough || len - best < tol) break;
    const G3 eb = ub ? xb1 : xb0, ep = up ? xp1 : xp0;
    const G3 w = {__shfl_sync(full, ep.x, lp) - __shfl_sync(full, eb.x, lb),
                  __shfl_sync(full, ep.y, lp) - __shfl_sync(full, eb.y, lb),
                  __shfl_sync(full, ep.z, lp) - __shfl_sync(full, eb.z, lb)};
    const G3 vw = gsub(v, w);
    const float l2 = gdot(vw, vw);
    if (!(l2 > 1e-20f)) break;
    v = gmad(v, -clamp01(gdot(v, vw) / l2), vw);
  }
  if (lane < nvb) L.q[0][lane] = -gdot(xb0, dir);
  if (lane + 32 < nvb) L.q[0][lane + 32] = -gdot(xb1, dir);
  if (lane < nvp) L.q[1][lane] = gdot(xp0, dir);
  if (lane + 32 < nvp) L.q[1][lane + 32] = gdot(xp1, dir);
  __syncwarp();
  return S;
}

// Indices k < n with pred(k), in increasing order, written by the warp.
template <class Pred>
__device__ __forceinline__ int warp_list(uint16_t* list, int n, int lane, Pred pred) {
  int cnt = 0;
  for (int base = 0; base < n; base += 32) {
    const int k = base + lane;
    const bool ok = k < n && pred(k);
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (ok) list[cnt + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)k;
    cnt += __popc(bal);
  }
  __syncwarp();
  return cnt;
}

// Appends the keys of the lanes with ok; those the float classification left
// undecided (unsure) are also listed by their position.
__device__ __forceinline__ void warp_emit(bool ok, bool unsure, uint64_t key, int lane, uint64_t* out, uint32_t* unc,
                                          int64_t cap, unsigned long long* counter) {
  const unsigned bal = __ballot_sync(0xffffffffu, ok);
  if (!bal) return;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(counter, (unsigned long long)__popc(bal));
  base = __shfl_sync(0xffffffffu, base, 0);
  const unsigned lt = (1u << lane) - 1u;
  const unsigned long long at = base + __popc(bal & lt);
  if (ok && (int64_t)at < cap) out[at] = key;
  const unsigned un = __ballot_sync(0xffffffffu, ok && unsure);
  if (!un) return;
  if (lane == 0) base = atomicAdd(counter + kCandUnsure, (unsigned long long)__popc(un));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (ok && unsure) {
    const unsigned long long u = base + __popc(un & lt);
    if ((int64_t)u < cap) unc[u] = (uint32_t)at;
  }
}

// Whether owner vertex v of body b can pass the OBB cull of Rockable.cpp:
// 1385-1391 (the vertex cube against p's OBB enlarged by dVerlet), from the
// box's three axes alone: 0 no, 1 yes for sure, 2 undecided (rk_nl.cu's
// cull_hit decides).  With the distance-only tests: whether the vertex can
// reach the partner's bounding sphere.
template <bool GEOM>
__device__ __forceinline__ int cull_class(const Scene& s, float4 pv, int p, float fr, float reach, float4 cp) {
  if (GEOM) {
    const float dx = pv.x - cp.x, dy = pv.y - cp.y, dz = pv.z - cp.z;
    const float mg = fmaxf(fmaxf(fmaxf(fabsf(cp.x), fabsf(cp.y)), fabsf(cp.z)) + cp.w,
                           fmaxf(fmaxf(fabsf(pv.x), fabsf(pv.y)), fabsf(pv.z)));
    float lim = reach + cp.w;
    lim = lim + 1e-4f * lim + 1e-6f * mg + 2e-6f;
    return dx * dx + dy * dy + dz * dz <= lim * lim ? 1 : 0;
  }
  const float* o = s.bobbf + 15 * (int64_t)p;
  const float dmax = (float)s.dVerlet;
  const float dx = pv.x - o[0], dy = pv.y - o[1], dz = pv.z - o[2];
  const float mag = fmaxf(fmaxf(fabsf(o[0]), fabsf(o[1])), fabsf(o[2])) + o[12] + o[13] + o[14] + 3.f * dmax + fr;
  bool in = true;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float* e = o + 3 + 3 * i;
    const float t = fabsf(dx * e[0] + dy * e[1] + dz * e[2]), ext = o[12 + i] + dmax;
    const float m = 1e-6f * (mag + t) + 1e-9f;
    if (t > ext + fr * (fabsf(e[0]) + fabsf(e[1]) + fabsf(e[2])) + m) return 0;
    in = in && t < ext - m;
  }
  return in ? 1 : 2;
}

// Candidate sub-contacts of the pairs: one warp per pair of bodies (side 0 the
// lower index), which lists the candidates of both directions (owner 0 ->
// partner 1: vertex-vertex, vertex-edge, vertex-face, edge-edge; owner 1 ->
// partner 0: vertex-edge, vertex-face; Rockable.cpp:1385-1432).  The lanes
// first narrow both bodies down to the sub-elements that can be near the
// other one -- a separating slab between the two cores, then the other body's
// bounding sphere (vertices: its box; the role of Rockable's per-shape OBB
// trees, Rockable.cpp:1440-1541, Shape.cpp:628-670); index lists in shared
// memory --
// and then sweep the products of the lists 32 candidates at a time: float
// sphere prefilter, float classification of the NEAR predicate, and what that
// accepts or leaves undecided is appended with one atomic per warp and ballot.
// Within a half-pair the keys come out in ascending order (the key sort
// relies on it).  The float tests only skip candidates that cannot be NEAR,
// so the NEAR set is exactly the one of testing every candidate.
// Measured on the packed column of 50 000 grains (1.6 M entries): 7.92 ms
// with the vertex cull and the FP64 predicates inlined, one warp per
// half-pair and no slab; 3.14 ms (plus 0.60 ms for the vertex cull) with the
// slab and the FP64 work apart; 2.1 ms with both directions of a pair in one
// warp, fused multiply-adds, 6 blocks per SM (80 registers) and no box test
// for edges and faces.  Bound by the instruction stream.
template <bool GEOM>
__global__ void __launch_bounds__(32 * kCandWarps, 6)
k_candidates(Scene s, const uint64_t* pairs, int64_t np, int mv, int me, int mf, uint64_t* out, uint32_t* unc,
             int64_t cap, unsigned long long* counter) {
  extern __shared__ __align__(16) char list_mem[];
  const int lane = threadIdx.x & 31;
  const CandLists L = cand_lists(list_mem + (threadIdx.x >> 5) * cand_list_bytes(mv, me, mf), mv, me, mf);
  const int64_t stride = (int64_t)gridDim.x * kCandWarps;
  for (int64_t h = (int64_t)blockIdx.x * kCandWarps + (threadIdx.x >> 5); h < np; h += stride) {
    __syncwarp();  // the previous pair's lists have been read
    const uint64_t key = pairs[h];
    const int b = (int)(key >> 21), p = (int)(key & ((1u << 21) - 1));
    const int shb = s.shape[b], shp = s.shape[p];
    const double Rb = s.rad[b], Rp = s.rad[p], dmax = s.dVerlet;
    const int nvb = s.vert_ofs[shb + 1] - s.vert_ofs[shb];
    const int nvp = s.vert_ofs[shp + 1] - s.vert_ofs[shp];
    const float4* sb = s.sph + s.sph_ofs[b];
    const float4* sp = s.sph + s.sph_ofs[p];
    // conservative float filter: a candidate whose bounding spheres are
    // farther apart than the NEAR distance allows cannot be NEAR
    const float sum = d2f(Rb + Rp + dmax);
    const float4 cb = make_float4(d2f(s.pos[3 * (int64_t)b]), d2f(s.pos[3 * (int64_t)b + 1]),
                                  d2f(s.pos[3 * (int64_t)b + 2]), s.bnd[b]);
    const float4 cp = make_float4(d2f(s.pos[3 * (int64_t)p]), d2f(s.pos[3 * (int64_t)p + 1]),
                                  d2f(s.pos[3 * (int64_t)p + 2]), s.bnd[p]);
    // margin for the float rounding of coordinates of magnitude up to `mag`
    // (about 16 ulps of it) on top of a relative 1e-4
    const float mag = fmaxf(fmaxf(fmaxf(fabsf(cb.x), fabsf(cb.y)), fabsf(cb.z)) + cb.w,
                            fmaxf(fmaxf(fabsf(cp.x), fabsf(cp.y)), fabsf(cp.z)) + cp.w);
    const float slack = 1e-6f * mag + 2e-6f;
    auto far = [&](float4 a, float4 c, float extent) {
      float dx = a.x - c.x, dy = a.y - c.y, dz = a.z - c.z;
      float lim = sum + extent;
      lim = lim + 1e-4f * lim + slack;
      return dx * dx + dy * dy + dz * dz > lim * lim;
    };
    const float ve_ext = d2f(1.0 + 2.0 * dmax);
    const float glim = sum + 1e-4f * sum + slack;
    const float glim2 = glim * glim;
    const float alim = sum - (1e-4f * sum + slack);  // float acceptance: the NEAR distance shrunk by the margin
    const float dmaxf = d2f(dmax);
    // an owner vertex meets the partner's edges up to dmax x their length
    // beyond their ends (the vertex-edge projection test), so its reach
    // grows by that much (an edge is at most the body's diameter long)
    const float vreach = sum + 2.f * dmaxf * fmaxf(cb.w, cp.w);
    // the slab between the two cores along a separating direction: an element
    // beyond the NEAR distance from the other core's side of it is farther
    // than that from all of the other body's elements; a pair whose gap
    // exceeds the NEAR distance keeps none
    const float slim = vreach + 1e-4f * vreach + slack;
    const Slab S = pair_slab(sb, nvb, sp, nvp, gpt(cb), gpt(cp), slim, 0.05f * sum, lane, L);
    if (S.pmin - S.bmax > slim) continue;
    // an element of a side stays when its least L.q is at most the side's limit
    const float lim0 = -(S.pmin - slim), lim1 = S.bmax + slim;
    int nown0 = 0, nown1 = 0, nother = 0, ne0 = 0, ne1 = 0, nf0 = 0, nf1 = 0;
#pragma unroll 1
    for (int side = 0; side < 2; side++) {
      const int sh = side ? shp : shb, nv = side ? nvp : nvb, body = side ? b : p;  // body: the other one
      const float4* sx = side ? sp : sb;
      const float4 co = side ? cb : cp;
      const float* bx = s.bbox + 15 * (int64_t)body;
      const float* q = side ? L.q[1] : L.q[0];
      const float lim = side ? lim1 : lim0;
      const int eofs = s.edge_ofs[sh], ne = s.edge_ofs[sh + 1] - eofs;
      const int fofs = s.face_ofs[sh], nf = s.face_ofs[sh + 1] - fofs;
      const float fr = d2f((side ? Rp : Rb) + dmax);
      uint16_t* own = side ? L.own[1] : L.own[0];
      // owner vertices: those that can pass the cull, bit 15 when undecided
      int cnt = 0, all = 0;
      for (int base = 0; base < nv; base += 32) {
        const int v = base + lane;
        bool near = v < nv && q[v] <= lim;
        if (near) near = !box_far(bx, sx[v], vreach, slack);
        if (side) {  // (as partners of the other side's vertices: without the cull)
          const unsigned bal = __ballot_sync(0xffffffffu, near);
          if (near) L.other[all + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)v;
          all += __popc(bal);
        }
        const int cc = near ? cull_class<GEOM>(s, sx[v], body, fr, sum, co) : 0;
        const unsigned bal = __ballot_sync(0xffffffffu, cc != 0);
        if (cc) own[cnt + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)(v | (cc == 2 ? 0x8000 : 0));
        cnt += __popc(bal);
      }
      const int ke = warp_list(side ? L.e[1] : L.e[0], ne, lane, [&](int e) {
        const int* ev = s.edges + 2 * (eofs + e);
        if (fminf(q[ev[0]], q[ev[1]]) > lim) return false;
        float4 se = sx[nv + e];
        se.w *= ve_ext;  // the vertex-edge test's extended edge
        return !far(se, co, co.w + se.w);
      });
      const int kf = warp_list(side ? L.f[1] : L.f[0], nf, lane, [&](int f) {
        float low = 3.0e38f;
        for (int k = s.face_vofs[fofs + f]; k < s.face_vofs[fofs + f + 1]; k++) low = fminf(low, q[s.face_verts[k]]);
        if (low > lim) return false;
        const float4 sf = sx[nv + ne + f];
        return !far(sf, co, co.w + sf.w);
      });
      if (side) {
        nown1 = cnt; nother = all; ne1 = ke; nf1 = kf;
      } else {
        nown0 = cnt; ne0 = ke; nf0 = kf;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int dir = 0; dir < 2; dir++) {  // owner side dir
      const uint32_t kb = (uint32_t)(dir ? p : b), kp = (uint32_t)(dir ? b : p);
      const int shp_ = dir ? shb : shp, nvq = dir ? nvb : nvp;  // the partner's
      const int eofs = s.edge_ofs[shp_], nep = s.edge_ofs[shp_ + 1] - eofs;
      const float4* so = dir ? sp : sb;
      const float4* sq = dir ? sb : sp;
      const uint16_t* own = dir ? L.own[1] : L.own[0];
      const uint16_t* pe = dir ? L.e[0] : L.e[1];
      const uint16_t* pf = dir ? L.f[0] : L.f[1];
      const int nown = dir ? nown1 : nown0, npe = dir ? ne0 : ne1, npf = dir ? nf0 : nf1;
      // vertex-vertex (in the direction 0 -> 1 only)
      for (int base = 0, tot = dir ? 0 : nown * nother; base < tot; base += 32) {
        const int c = base + lane;
        bool ok = false, unsure = false;
        int v = 0, w = 0;
        if (c < tot) {
          v = own[c / nother];
          w = L.other[c % nother];
          unsure = (v & 0x8000) != 0;
          v &= 0x7fff;
          if (GEOM) {
            const G3 d = gsub(gpt(so[v]), gpt(sq[w]));
            ok = gdot(d, d) <= glim2;
          } else {
            ok = !far(so[v], sq[w], 0.f);
            unsure = unsure || !accept_vv(gpt(so[v]), gpt(sq[w]), alim);
          }
        }
        warp_emit(ok, unsure, entry_key(kb, kp, 0u, (uint32_t)v, (uint32_t)w), lane, out, unc, cap, counter);
      }
      // vertex-edge
      for (int base = 0, tot = nown * npe; base < tot; base += 32) {
        const int c = base + lane;
        bool ok = false, unsure = false;
        int v = 0, e = 0;
        if (c < tot) {
          v = own[c / npe];
          e = pe[c % npe];
          unsure = (v & 0x8000) != 0;
          v &= 0x7fff;
          const float4 se = sq[nvq + e];
          const int* ev = s.edges + 2 * (eofs + e);
          const G3 pv = gpt(so[v]), e0 = gpt(sq[ev[0]]), e1 = gpt(sq[ev[1]]);
          if (GEOM) {
            ok = !far(so[v], se, se.w) && pt_seg_d2(pv, e0, e1) <= glim2;
          } else if (!far(so[v], se, ve_ext * se.w) && pt_line_d2(pv, e0, e1) <= glim2) {
            // (exact rejection first: Rockable's vertex-edge test accepts a
            // projection slightly off the edge, never a line distance above it)
            const int c_ = classify_ve(pv, e0, e1, alim, dmaxf, mag);
            ok = c_ >= 0;
            unsure = unsure || c_ == 0;
          }
        }
        warp_emit(ok, unsure, entry_key(kb, kp, 1u, (uint32_t)v, (uint32_t)e), lane, out, unc, cap, counter);
      }
      // vertex-face
      for (int base = 0, tot = nown * npf; base < tot; base += 32) {
        const int c = base + lane;
        bool ok = false, unsure = false;
        int v = 0, f = 0;
        if (c < tot) {
          v = own[c / npf];
          f = pf[c % npf];
          unsure = (v & 0x8000) != 0;
          v &= 0x7fff;
          const float4 sf = sq[nvq + nep + f];
          if (!far(so[v], sf, sf.w) && pt_poly_d2(s, sq, shp_, f, gpt(so[v])) <= glim2) {
            if (GEOM) {
              ok = true;
            } else {  // (exact rejection first: NEAR needs the polygon within reach)
              const int c_ = classify_vf(s, sq, shp_, f, gpt(so[v]), alim, mag);
              ok = c_ >= 0;
              unsure = unsure || c_ == 0;
            }
          }
        }
        warp_emit(ok, unsure, entry_key(kb, kp, 2u, (uint32_t)v, (uint32_t)f), lane, out, unc, cap, counter);
      }
      // edge-edge (in the direction 0 -> 1 only)
      for (int base = 0, tot = dir ? 0 : ne0 * npe; base < tot; base += 32) {
        const int c = base + lane;
        bool ok = false, unsure = false;
        int e1 = 0, e2 = 0;
        if (c < tot) {
          e1 = L.e[0][c / npe];
          e2 = pe[c % npe];
          const float4 s1 = so[nvb + e1], s2 = sq[nvq + e2];
          if (!far(s1, s2, s1.w + s2.w)) {
            const int* ea = s.edges + 2 * (s.edge_ofs[shb] + e1);
            const int* eb = s.edges + 2 * (eofs + e2);
            const G3 a0 = gpt(so[ea[0]]), a1 = gpt(so[ea[1]]), b0 = gpt(sq[eb[0]]), b1 = gpt(sq[eb[1]]);
            if (GEOM) {
              // nearly parallel edges (ill-conditioned closest points) within
              // sphere reach are kept: an extra entry is harmless, a missing one not
              const G3 d1 = gsub(a1, a0), d2 = gsub(b1, b0), nx = gcross(d1, d2);
              const bool parallel = !(gdot(nx, nx) > 1e-6f * gdot(d1, d1) * gdot(d2, d2));
              ok = parallel || seg_seg_d2(a0, a1, b0, b1) <= glim2;
            } else if (!lines_far(a0, a1, b0, b1, glim2)) {
              // (exact rejection first: NEAR needs the edges' lines within reach)
              const int c_ = classify_ee(a0, a1, b0, b1, alim, mag);
              ok = c_ >= 0;
              unsure = c_ == 0;
            }
          }
        }
        warp_emit(ok, unsure, entry_key(kb, kp, 3u, (uint32_t)e1, (uint32_t)e2), lane, out, unc, cap, counter);
      }
    }
  }
}

}  // namespace rk
