// Kernels of the batched rigid-body step, templated on the bulk type R and the
// island type W (plain form: double/double; precision form: float/double).
//
//   k_integrate    one thread per body (four in small float64 batches):
//                  RigidBody.Integrate + CalculateDerivedData
//                  (rigidbody.go:213-299)
//   k_narrowphase  one CTA per world, worlds pulled from a device queue; body
//                  rows staged in shared memory with bulk async copies; the
//                  plane test and all ordered pairs in the reference's loop
//                  order (examples/cubedrop.go:41-67), compacted with warp
//                  prefix sums so the contact list order is the reference's
//   k_resolve      (cz_resolve.cuh) G lanes per world, 32/G worlds per warp,
//                  worlds pulled from a device queue: prepareContacts,
//                  adjustPositions, adjustVelocities (contact.go:204-445)
#pragma once
#include <cuda_runtime.h>

#include "cz_layout.cuh"
#include "cz_math.cuh"

namespace cz {

constexpr unsigned FULL = 0xffffffffu;

// ============================================================== integrate

// RigidBody.Integrate + CalculateDerivedData of body row i
// (rigidbody.go:213-299), in place in the batch rows.
template <class R, class W>
__device__ __forceinline__ void integrate_body(const BatchView<R>& v, long long i, R dt, R sleep_bias) {
  if (!v.awake[i]) return;  // rigidbody.go:214-216
  const long long S = v.nb_pad;
  R* b = v.body + i;
#define F(r) b[(long long)(r) * S]
  const R zero = (R)0;
  const R invm = F(B_INVM);
  // lastFrameAccelleration = Acceleration + forceAccum * inverseMass (forceAccum is 0)
  v3<R> lfa = V<R>(F(B_AX), F(B_AY), F(B_AZ));
  add_scaled(lfa, V<R>(zero, zero, zero), invm);
  m3<R> iw;
#pragma unroll
  for (int k = 0; k < 9; ++k) iw.m[k] = F(B_IW0 + k);
  // angularAcceleration = iitWorld * torqueAccum (torqueAccum is 0)
  v3<R> ang = mulv(iw, V<R>(zero, zero, zero));
  v3<R> vel = V<R>(F(B_VX), F(B_VY), F(B_VZ));
  v3<R> rot = V<R>(F(B_RX), F(B_RY), F(B_RZ));
  add_scaled(vel, lfa, dt);
  add_scaled(rot, ang, dt);
  mul_with(vel, F(B_LINPOW));
  mul_with(rot, F(B_ANGPOW));
  v3<R> pos = V<R>(F(B_PX), F(B_PY), F(B_PZ));
  add_scaled(pos, vel, dt);
  q4<R> q{F(B_QW), F(B_QX), F(B_QY), F(B_QZ)};
  add_scaled_vector(q, rot, dt);
  // CalculateDerivedData: renormalise (island type), transform, world inertia
  q4<W> qw = cvtq<W>(q);
  qnormalize_island<R, W>(qw);
  q = cvtq<R>(qw);
  R rm[9];
  rotation_of(q, rm);
  m3<R> ib;
#pragma unroll
  for (int k = 0; k < 9; ++k) ib.m[k] = F(B_IB0 + k);
  iw = world_inertia(rm, ib);
  // sleep bookkeeping, rigidbody.go:248-258
  if (v.can_sleep[i]) {
    R cm = dot(vel, vel) + dot(rot, rot);
    R motion = sleep_bias * F(B_MOTION) + ((R)1 - sleep_bias) * cm;
    if (motion < (R)0.3) {
      v.awake[i] = 0;
      vel = V<R>(zero, zero, zero);
      rot = V<R>(zero, zero, zero);
    } else if (motion > (R)3.0) {
      motion = (R)3.0;
    }
    F(B_MOTION) = motion;
  }
  F(B_PX) = pos.x; F(B_PY) = pos.y; F(B_PZ) = pos.z;
  F(B_QW) = q.w; F(B_QX) = q.x; F(B_QY) = q.y; F(B_QZ) = q.z;
  F(B_VX) = vel.x; F(B_VY) = vel.y; F(B_VZ) = vel.z;
  F(B_RX) = rot.x; F(B_RY) = rot.y; F(B_RZ) = rot.z;
  F(B_LX) = lfa.x; F(B_LY) = lfa.y; F(B_LZ) = lfa.z;
#pragma unroll
  for (int k = 0; k < 9; ++k) F(B_IW0 + k) = iw.m[k];
#undef F
}

template <class R, class W>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 2) k_integrate(BatchView<R> v, R dt, R sleep_bias) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // the work queues of the frame's launches that follow on the stream
  if (i < 4) v.queue[i] = 0;
  if (i >= v.nb_run) return;
  integrate_body<R, W>(v, v.first_body + i, dt, sleep_bias);
}

// integrate_body by four lanes, for small float64 batches: lane c (c < 3) has
// component c of the vectors and row c of the world inertia, lane c (c < 4)
// component c of the quaternion; what a sum needs whole meets by shuffles.
// Each component is the one-lane formula's.  A float64 warp instruction costs
// its scheduler the same for any mask, and a body on one lane takes about 300
// of them, on four 110.  Every lane of the warp calls it; `valid` where i is a
// body.
template <class R>
__device__ __forceinline__ void integrate_body_spread(const BatchView<R>& v, long long i, bool valid, R dt,
                                                      R sleep_bias) {
  const int c4 = threadIdx.x & 3, c = c4 != 3 ? c4 : 0;
  const bool on = valid && v.awake[i];  // rigidbody.go:214-216
  const bool sleeps = on && v.can_sleep[i];
  const long long S = v.nb_pad;
  R* b = v.body + i;
#define F(r) b[(long long)(r) * S]
  const R zero = (R)0;
  R lfa = zero, vel = zero, rot = zero, pos = zero, acc = zero, motion = zero;
  R i0 = zero, i1 = zero, i2 = zero, i3 = zero, i4 = zero, i5 = zero, i6 = zero, i7 = zero, i8 = zero;
  if (on) {
    lfa = F(B_AX + c) + zero * F(B_INVM);
    const R ang = F(B_IW0 + c) * zero + F(B_IW0 + 3 + c) * zero + F(B_IW0 + 6 + c) * zero;
    vel = (F(B_VX + c) + lfa * dt) * F(B_LINPOW);
    rot = (F(B_RX + c) + ang * dt) * F(B_ANGPOW);
    pos = F(B_PX + c) + vel * dt;
    acc = F(B_QW + c4);
    i0 = F(B_IB0); i1 = F(B_IB0 + 1); i2 = F(B_IB0 + 2);
    i3 = F(B_IB0 + 3); i4 = F(B_IB0 + 4); i5 = F(B_IB0 + 5);
    i6 = F(B_IB0 + 6); i7 = F(B_IB0 + 7); i8 = F(B_IB0 + 8);
    if (sleeps) motion = F(B_MOTION);
  }
  auto get = [&](R a, int from) { return __shfl_sync(FULL, a, from, 4); };
  // Quaternion.AddScaledVector (quaternion.go:18-33): component c4 of (0, rot dt) * q
  {
    const R turn = rot * dt;
    const R q1 = get(acc, c4 == 0 ? 1 : 0), q2 = get(acc, c4 == 1 ? 3 : (c4 == 2 ? 1 : 2));
    const R q3 = get(acc, c4 == 1 ? 2 : (c4 == 3 ? 1 : 3));
    const R u1 = get(turn, c4 < 2 ? 0 : c4 - 1), u2 = get(turn, c4 < 2 ? 1 : (c4 == 2 ? 2 : 0));
    const R u3 = get(turn, c4 < 2 ? 2 : c4 - 2);
    const R a1 = u1 * q1, a2 = u2 * q2, a3 = u3 * q3;
    R t = zero * acc;
    t = c4 == 0 ? t - a1 : t + a1;
    t = c4 == 0 ? t - a2 : t + a2;
    t = t - a3;
    acc += t * (R)0.5;
  }
  // CalculateDerivedData: renormalise, transform, world inertia (row c)
  {
    const R sq = acc * acc;
    const R s0 = get(sq, 0), s1 = get(sq, 1), s2 = get(sq, 2), s3 = get(sq, 3);
    if (on) acc = normalize_component<R>(s0 + s1 + s2 + s3, acc, c4);
  }
  const q4<R> q{get(acc, 0), get(acc, 1), get(acc, 2), get(acc, 3)};
  R r[9];
  rotation_of(q, r);
  const R ra = c == 0 ? r[0] : (c == 1 ? r[1] : r[2]), rb = c == 0 ? r[3] : (c == 1 ? r[4] : r[5]);
  const R rc = c == 0 ? r[6] : (c == 1 ? r[7] : r[8]);
  const R ta = ra * i0 + rb * i1 + rc * i2, tb = ra * i3 + rb * i4 + rc * i5, tc = ra * i6 + rb * i7 + rc * i8;
  const R w0 = ta * r[0] + tb * r[3] + tc * r[6], w3 = ta * r[1] + tb * r[4] + tc * r[7];
  const R w6 = ta * r[2] + tb * r[5] + tc * r[8];
  // sleep bookkeeping, rigidbody.go:248-258
  bool falls = false;
  if (__any_sync(FULL, sleeps)) {
    const R vv = vel * vel, rr = rot * rot;
    const R cm = (get(vv, 0) + get(vv, 1) + get(vv, 2)) + (get(rr, 0) + get(rr, 1) + get(rr, 2));
    if (sleeps) {
      motion = sleep_bias * motion + ((R)1 - sleep_bias) * cm;
      falls = motion < (R)0.3;
      if (falls) vel = rot = zero;
      else if (motion > (R)3.0) motion = (R)3.0;
    }
  }
  __syncwarp();
  if (!on) return;
  F(B_QW + c4) = acc;
  if (c4 == 3) {
    if (sleeps) F(B_MOTION) = motion;
    if (falls) v.awake[i] = 0;
    return;
  }
  F(B_PX + c) = pos;
  F(B_VX + c) = vel;
  F(B_RX + c) = rot;
  F(B_LX + c) = lfa;
  F(B_IW0 + c) = w0;
  F(B_IW0 + 3 + c) = w3;
  F(B_IW0 + 6 + c) = w6;
#undef F
}

// Four lanes per body in float64 for launches of up to kSpreadBodies rows,
// where a scheduler has one or two such warps: one world of 20 cubes 14 -> 10 us
// a frame, 60 falling worlds of 30 bodies x 10 frames 1469 -> 1332 us (with CTAs
// of 256 threads 12 us and 1372); one launch over 10000 rows takes 24.5 us
// either way, over 15600 24.5 with a lane per body and 36.4 so.  With more
// bodies the float64 pipes are full and the lanes' idle quarter counts (4 x 110
// instructions per 32 bodies for 300).  A rollout's parts share the GPU, but
// not in step: up to twice as many rows in the batch.  20 frames from the fall,
// a lane per body and four: 200 worlds of 30 bodies 2.67 and 2.61 ms, 500 of 30
// 2.84 and 2.83, 600 of 30 2.91 both, 1000 of 32 3.31 and 3.39, 4096 of 8 to 64
// 10.5 and 11.3.
constexpr long long kSpreadBodies = 8192;
template <class R>
__global__ void __launch_bounds__(256) k_integrate_spread(BatchView<R> v, R dt, R sleep_bias) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 4) v.queue[t] = 0;
  const long long i = t >> 2;
  integrate_body_spread<R>(v, v.first_body + (i < v.nb_run ? i : 0), i < v.nb_run, dt, sleep_bias);
}

// ============================================================== narrowphase

template <class R> struct NPContact {
  R px, py, pz, nx, ny, nz, pen;
  int b0, b1;
};

// Shared-memory tile of one world for the narrowphase.
template <class R> struct NPTile {
  R* stage;      // [11][nbs]: PX PY PZ QW QX QY QZ HX HY HZ RAD (bulk-copied)
  R* T;          // [12][nbs]: collider transforms
  int* shape;    // [nbs] (bulk-copied)
  float* cull;   // [5][nbs]: centre xyz, bounding radius |h|_2 (or r), |h|_1 (or r)
  int nbs;
  __device__ __forceinline__ R s(int r, int i) const { return stage[r * nbs + i]; }
  __device__ __forceinline__ xf<R> xform(int i) const {
    xf<R> t;
#pragma unroll
    for (int r = 0; r < 12; ++r) t.m[r] = T[r * nbs + i];
    return t;
  }
  // column c of body i's transform (an axis, or with c = 3 the centre), for any c
  __device__ __forceinline__ v3<R> axis(int i, int c) const {
    const R* t = T + (size_t)(3 * c) * nbs + i;
    return V<R>(t[0], t[nbs], t[2 * nbs]);
  }
  __device__ __forceinline__ v3<R> half(int i) const { return V<R>(s(7, i), s(8, i), s(9, i)); }
  __device__ __forceinline__ R radius(int i) const { return s(10, i); }
};

// Integer keys in the order of non-negative values (both zeros alike).
__device__ __forceinline__ unsigned sort_key(float v) { return v == 0.f ? 0u : __float_as_uint(v); }
__device__ __forceinline__ unsigned long long sort_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b << 1) == 0ull ? 0ull : b;
}

template <class R>
__device__ __forceinline__ R transform_to_axis(const xf<R>& t, const v3<R>& h, const v3<R>& axis) {
  // colliders.go:762-770
  return h.x * fabs_<R>(dot(axis, t.axis(0))) + h.y * fabs_<R>(dot(axis, t.axis(1))) +
         h.z * fabs_<R>(dot(axis, t.axis(2)));
}

// The outcome of CollisionCube.CheckAgainstCube's axes for a pair of boxes
// (colliders.go:575-627), in both orders of the pair: the axis of smallest
// penetration (0-2 and 3-5 the boxes' own, 6 + 3i + j the edge pairs; 255:
// none) and the smallest of the first six alone.
template <class R> struct SatResult {
  R pen;
  int code;  // best | best_single << 8 of (one, two), and << 16, << 24 of (two, one); kSatApart: a separating axis
};
constexpr int kSatApart = -1;

// penetrationOnAxis, colliders.go:445-456, of two boxes whose centres are tc apart
template <class R>
__device__ __forceinline__ R axis_penetration(const xf<R>& t1, const v3<R>& h1, const xf<R>& t2, const v3<R>& h2,
                                              const v3<R>& tc, v3<R> axis) {
  normalize(axis);
  const R one = transform_to_axis(t1, h1, axis);
  const R two = transform_to_axis(t2, h2, axis);
  const R dist = fabs_<R>(dot(tc, axis));
  return one + two - dist;
}

// Whether one of box i1's own axes separates the boxes: the first three of
// their axes, by one lane.
template <class R> __device__ __forceinline__ bool sat_apart_first(const NPTile<R>& tl, int i1, int i2) {
  const xf<R> t1 = tl.xform(i1), t2 = tl.xform(i2);
  const v3<R> h1 = tl.half(i1), h2 = tl.half(i2);
  v3<R> tc = t2.axis(3);
  sub(tc, t1.axis(3));
  bool apart = false;
#pragma unroll 1
  for (int q = 0; q < 3 && !apart; ++q) {
    const v3<R> axis = tl.axis(i1, q);
    apart = !(sqmag(axis) < Lim<R>::eps()) && axis_penetration(t1, h1, t2, h2, tc, axis) < (R)0;
  }
  return apart;
}

// tryAxis (colliders.go:458-477) for the fifteen axes of a pair of boxes, an
// axis per lane of a group of 16 (l = 0..15), the smallest penetration (the
// first of equal ones, as the reference's loop keeps) by shuffles.  Every lane
// of the warp calls it.  The axes of (two, one) are the same vectors or their
// negatives, and every term of a penetration is the same or its magnitude is,
// so one set of fifteen serves both orders; only the order in which equal
// penetrations are met differs.
// On one lane the fifteen axes are one chain (about 60 us of float64 latency),
// and a warp runs it for the twenty or so box pairs of a small world, most of
// them in both orders: 15 axes' instructions for 20 lanes, against half of 10.
template <class R>
__device__ __forceinline__ SatResult<R> sat_axes(const NPTile<R>& tl, int i1, int i2, int l) {
  using Key = decltype(sort_key((R)0));
  const unsigned gmask = 0xFFFFu << (threadIdx.x & 16);
  const int ei = (l - 6) / 3, ej = (l - 6) % 3;  // edge axes
  v3<R> axis = tl.axis(l < 3 || l > 5 ? i1 : i2, l < 3 ? l : (l < 6 ? l - 3 : (l < 15 ? ei : 0)));
  if (l > 5) axis = cross(axis, tl.axis(i2, l < 15 ? ej : 0));
  const xf<R> t1 = tl.xform(i1), t2 = tl.xform(i2);
  const v3<R> h1 = tl.half(i1), h2 = tl.half(i2);
  v3<R> tc = t2.axis(3);
  sub(tc, t1.axis(3));
  R p = (R)0;
  bool tried = l < 15 && !(sqmag(axis) < Lim<R>::eps());
  if (tried) p = axis_penetration(t1, h1, t2, h2, tc, axis);
  SatResult<R> r;
  r.pen = (R)0;
  r.code = kSatApart;
  const bool apart = (__ballot_sync(FULL, tried && p < (R)0) & gmask) != 0;
  tried = tried && p < Lim<R>::max_value();  // a candidate (NaN never is)
  // integer keys of the (here non-negative) penetrations
  const Key none = ~(Key)0;
  const Key key = tried && !(p < (R)0) ? sort_key(p) : none;
  Key all = key, own = l < 6 ? key : none;
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) {
    const Key a = __shfl_xor_sync(FULL, all, d, 16), o = __shfl_xor_sync(FULL, own, d, 16);
    all = a < all ? a : all;
    own = o < own ? o : own;
  }
  // the first axis with the smallest value, in the pair's order and in the other's
  const int back = l < 3 ? l + 3 : (l < 6 ? l - 3 : 6 + 3 * ej + ei);
  const unsigned at_all = __ballot_sync(FULL, key == all && all != none) & gmask;
  const unsigned at_own = __ballot_sync(FULL, l < 6 && key == own && own != none) & gmask;
  int b_all = key == all && all != none ? back : 255, b_own = l < 6 && key == own && own != none ? back : 255;
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) {
    b_all = min(b_all, __shfl_xor_sync(FULL, b_all, d, 16));
    b_own = min(b_own, __shfl_xor_sync(FULL, b_own, d, 16));
  }
  const int best = at_all ? (__ffs(at_all) - 1) & 15 : 255, single = at_own ? (__ffs(at_own) - 1) & 15 : 255;
  r.pen = __shfl_sync(FULL, p, best & 15, 16);
  if (!apart) r.code = best | single << 8 | b_all << 16 | (b_own & 0x7F) << 24;
  return r;
}

// The same axes on one lane, in the reference's loop (an axis apart ends it),
// for the order (i1, i2) alone.
template <class R> __device__ __forceinline__ SatResult<R> sat_serial(const NPTile<R>& tl, int i1, int i2) {
  const xf<R> t1 = tl.xform(i1), t2 = tl.xform(i2);
  const v3<R> h1 = tl.half(i1), h2 = tl.half(i2);
  v3<R> tc = t2.axis(3);
  sub(tc, t1.axis(3));
  SatResult<R> r;
  r.pen = Lim<R>::max_value();
  r.code = kSatApart;
  int best = 255, single = 255;
#pragma unroll 1
  for (int l = 0; l < 15; ++l) {
    v3<R> axis = tl.axis(l < 3 || l > 5 ? i1 : i2, l < 3 ? l : (l < 6 ? l - 3 : (l - 6) / 3));
    if (l > 5) axis = cross(axis, tl.axis(i2, (l - 6) % 3));
    if (!(sqmag(axis) < Lim<R>::eps())) {
      const R p = axis_penetration(t1, h1, t2, h2, tc, axis);
      if (p < (R)0) return r;
      if (p < r.pen) {
        r.pen = p;
        best = l;
      }
    }
    if (l == 5) single = best;
  }
  r.code = best | single << 8;
  return r;
}

// fillPointFaceBoxBox, colliders.go:479-517, of boxes one and two
template <class R>
__device__ __forceinline__ void fill_point_face(const NPTile<R>& tl, int one, int two, const v3<R>& tc, int best, R pen,
                                                NPContact<R>& c) {
  v3<R> nrm = tl.axis(one, best);
  if (dot(nrm, tc) > (R)0) mul_with(nrm, (R)-1);
  const xf<R> t = tl.xform(two);
  v3<R> vv = tl.half(two);
  if (dot(t.axis(0), nrm) < (R)0) vv.x = -vv.x;
  if (dot(t.axis(1), nrm) < (R)0) vv.y = -vv.y;
  if (dot(t.axis(2), nrm) < (R)0) vv.z = -vv.z;
  v3<R> p = xf_mul(t, vv);
  c.px = p.x; c.py = p.y; c.pz = p.z;
  c.nx = nrm.x; c.ny = nrm.y; c.nz = nrm.z;
  c.pen = pen;
  c.b0 = one;
  c.b1 = two;
}

// contactPoint, colliders.go:519-573
template <class R>
__device__ __forceinline__ v3<R> edge_contact_point(const v3<R>& p1, const v3<R>& d1, R s1, const v3<R>& p2,
                                                    const v3<R>& d2, R s2, bool use_one) {
  R sm1 = sqmag(d1);
  R sm2 = sqmag(d2);
  R d12 = dot(d2, d1);
  v3<R> to = p1;
  sub(to, p2);
  R ds1 = dot(d1, to);
  R ds2 = dot(d2, to);
  R denom = sm1 * sm2 - d12 * d12;
  if (fabs_<R>(denom) < Lim<R>::eps()) return use_one ? p1 : p2;
  R mua = (d12 * ds2 - sm2 * ds1) / denom;
  R mub = (sm1 * ds2 - d12 * ds1) / denom;
  if (mua > s1 || mua < -s1 || mub > s2 || mub < -s2) return use_one ? p1 : p2;
  v3<R> c1 = d1;
  mul_with(c1, mua);
  add(c1, p1);
  v3<R> c2 = d2;
  mul_with(c2, mub);
  add(c2, p2);
  mul_with(c1, (R)0.5);
  mul_with(c2, (R)0.5);
  add(c1, c2);
  return c1;
}

// CollisionCube.CheckAgainstCube past its axes (colliders.go:628-710): the
// contact for the axis `best` of penetration `pen` (sat_axes).
template <class R>
__device__ int cube_contact(const NPTile<R>& tl, int i1, int i2, int best, int best_single, R pen, NPContact<R>& c,
                            uint32_t& err) {
  if (best > 14) {  // only with non-finite transforms; the reference panics here
    err |= ST_NONFINITE;
    return 0;
  }
  v3<R> tc = tl.axis(i2, 3);
  sub(tc, tl.axis(i1, 3));
  if (best < 6) {
    const bool second = best > 2;
    if (second) mul_with(tc, (R)-1);
    fill_point_face(tl, second ? i2 : i1, second ? i1 : i2, tc, second ? best - 3 : best, pen, c);
    return 1;
  }
  best -= 6;
  const int ai = best / 3, bi = best % 3;
  v3<R> oa = tl.axis(i1, ai);
  v3<R> ob = tl.axis(i2, bi);
  v3<R> axis = cross(oa, ob);
  normalize(axis);
  if (dot(axis, tc) > (R)0) mul_with(axis, (R)-1);
  const xf<R> t1 = tl.xform(i1), t2 = tl.xform(i2);
  const v3<R> h1 = tl.half(i1), h2 = tl.half(i2);
  R e1[3] = {h1.x, h1.y, h1.z};
  R e2[3] = {h2.x, h2.y, h2.z};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (i == ai) e1[i] = (R)0;
    else if (dot(t1.axis(i), axis) > (R)0) e1[i] = -e1[i];
    if (i == bi) e2[i] = (R)0;
    else if (dot(t2.axis(i), axis) < (R)0) e2[i] = -e2[i];
  }
  v3<R> p1 = xf_mul(t1, V<R>(e1[0], e1[1], e1[2]));
  v3<R> p2 = xf_mul(t2, V<R>(e2[0], e2[1], e2[2]));
  const R s1 = ai == 0 ? h1.x : (ai == 1 ? h1.y : h1.z);
  const R s2 = bi == 0 ? h2.x : (bi == 1 ? h2.y : h2.z);
  v3<R> vtx = edge_contact_point(p1, oa, s1, p2, ob, s2, best_single > 2);
  c.px = vtx.x; c.py = vtx.y; c.pz = vtx.z;
  c.nx = axis.x; c.ny = axis.y; c.nz = axis.z;
  c.pen = pen;
  c.b0 = i1;
  c.b1 = i2;
  return 1;
}

// CollisionCube.CheckAgainstSphere, colliders.go:368-441.  `svel` is the
// sphere body's velocity, read only for the zero-normal fallback.
template <class R>
__device__ int cube_sphere(const xf<R>& tc, const v3<R>& h, int ic, const xf<R>& ts, R r, int is,
                           const R* svel_rows, long long svel_stride, NPContact<R>& c) {
  v3<R> pos = ts.axis(3);
  v3<R> rel = xf_inv(tc, pos);
  if (fabs_<R>(rel.x) - r > h.x || fabs_<R>(rel.y) - r > h.y || fabs_<R>(rel.z) - r > h.z) return 0;
  R hh[3] = {h.x, h.y, h.z};
  R rc[3] = {rel.x, rel.y, rel.z};
  R cl[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    R d = rc[i];
    if (d > hh[i]) d = hh[i];
    else if (d < -hh[i]) d = -hh[i];
    cl[i] = d;
  }
  v3<R> dc = V<R>(cl[0], cl[1], cl[2]);
  sub(dc, rel);
  R dist = sqmag(dc);
  if (dist > r * r) return 0;
  v3<R> cw = xf_mul(tc, V<R>(cl[0], cl[1], cl[2]));
  v3<R> nrm = cw;
  sub(nrm, pos);
  // colliders.go:417-421; the precision form also takes the fallback when the
  // centre needed no clamping (float32 rounding of the round trip exceeds the
  // reference's absolute 1e-14)
  if (real_equal<R>(mag(nrm), (R)0) || (sizeof(R) < sizeof(double) && dist == (R)0)) {
    nrm = V<R>(svel_rows[0], svel_rows[svel_stride], svel_rows[2 * svel_stride]);
  }
  normalize(nrm);
  R pen = r;
  if (!real_equal<R>(dist, (R)0)) pen -= sqrt_<R>(dist);
  else pen = (R)0;
  c.px = cw.x; c.py = cw.y; c.pz = cw.z;
  c.nx = nrm.x; c.ny = nrm.y; c.nz = nrm.z;
  c.pen = pen;
  c.b0 = ic;
  c.b1 = is;
  return 1;
}

// CollisionSphere.CheckAgainstSphere, colliders.go:215-254
template <class R>
__device__ __forceinline__ int sphere_sphere(const v3<R>& p1, R r1, int i1, const v3<R>& p2, R r2, int i2,
                                             NPContact<R>& c) {
  v3<R> mid = p1;
  sub(mid, p2);
  R size = mag(mid);
  if (size <= (R)0 || size >= r1 + r2) return 0;
  v3<R> pt = mid;
  mul_with(pt, (R)0.5);
  add(pt, p1);
  v3<R> nrm = mid;
  mul_with(nrm, (R)1 / size);
  c.px = pt.x; c.py = pt.y; c.pz = pt.z;
  c.nx = nrm.x; c.ny = nrm.y; c.nz = nrm.z;
  c.pen = r1 + r2 - size;
  c.b0 = i1;
  c.b1 = i2;
  return 1;
}

// CollisionSphere.CheckAgainstHalfSpace (colliders.go:178-207)
template <class R>
__device__ __forceinline__ int plane_sphere(const NPTile<R>& tl, int i, const BatchView<R>& v, NPContact<R>& c) {
  const v3<R> pn = V<R>(v.plane_nx, v.plane_ny, v.plane_nz);
  const v3<R> pos = V<R>(tl.T[9 * tl.nbs + i], tl.T[10 * tl.nbs + i], tl.T[11 * tl.nbs + i]);
  const R r = tl.radius(i);
  const R d = dot(pn, pos) - r;
  if (!(d <= v.plane_offset)) return 0;
  v3<R> p = pn;
  mul_with(p, d + r * (R)-1);
  add(p, pos);
  c.px = p.x; c.py = p.y; c.pz = p.z;
  c.nx = pn.x; c.ny = pn.y; c.nz = pn.z;
  c.pen = -d;
  c.b0 = i;
  c.b1 = -1;
  return 1;
}

// Vertex k of CollisionCube.CheckAgainstHalfSpace (colliders.go:306-366,
// 750-760; bit b of k set: component b negative): whether it gives a contact,
// and the contact.
template <class R>
__device__ __forceinline__ bool plane_vertex(const NPTile<R>& tl, int i, int k, const BatchView<R>& v,
                                             NPContact<R>& c) {
  const v3<R> pn = V<R>(v.plane_nx, v.plane_ny, v.plane_nz);
  const R off = v.plane_offset;
  const xf<R> t = tl.xform(i);
  const v3<R> h = tl.half(i);
  const R proj = transform_to_axis(t, h, pn);
  const R cd = dot(pn, t.axis(3)) - proj;
  if (!(cd <= off)) return false;
  const v3<R> vp = xf_mul(t, V<R>((k & 1) ? -h.x : h.x, (k & 2) ? -h.y : h.y, (k & 4) ? -h.z : h.z));
  const R vd = dot(vp, pn);
  if (!(vd <= off)) return false;
  v3<R> p = pn;
  mul_with(p, vd - off);
  add(p, vp);
  c.px = p.x; c.py = p.y; c.pz = p.z;
  c.nx = pn.x; c.ny = pn.y; c.nz = pn.z;
  c.pen = off - vd;
  c.b0 = i;
  c.b1 = -1;
  return true;
}

// Conservative float32 rejection tests.  Each returns true only when the
// reference's own test is certain to report no contact, so skipping the full
// test changes no result:
//   box-box      bounding spheres apart by 10% of the radii + 1 mm: the boxes
//                are disjoint by more than the separating-axis test's rounding
//                and more than its skipping of near-parallel edge axes
//                (|a x b|^2 < 1e-7, colliders.go:461) can hide;
//   sphere-sphere  centres farther than r1 + r2 + 1 mm (colliders.go:227);
//   box-sphere   centre distance above |h|_1 + 3r + 1 mm, so some axis has
//                |rel_i| - r > h_i (the early exit of colliders.go:374-378).
// The margins dwarf the float32 rounding of positions (1e-5 relative is
// added); non-finite centres never reject.
struct Cull {
  const float* c;
  int nbs;
  __device__ __forceinline__ float d2_scale(int i, int j, float& scale) const {
    float dx = c[j] - c[i];
    float dy = c[nbs + j] - c[nbs + i];
    float dz = c[2 * nbs + j] - c[2 * nbs + i];
    scale = 1.f + fabsf(c[i]) + fabsf(c[nbs + i]) + fabsf(c[2 * nbs + i]) + fabsf(c[j]) + fabsf(c[nbs + j]) +
            fabsf(c[2 * nbs + j]);
    return dx * dx + dy * dy + dz * dz;
  }
  __device__ __forceinline__ float rb(int i) const { return c[3 * nbs + i]; }  // |h|_2 or r
  __device__ __forceinline__ float rl(int i) const { return c[4 * nbs + i]; }  // |h|_1 or r
  __device__ __forceinline__ bool boxes(int i, int j) const {
    float sc, d2 = d2_scale(i, j, sc);
    float t = (rb(i) + rb(j)) * 1.1f + 1e-3f + 1e-5f * sc;
    return d2 > t * t;
  }
  __device__ __forceinline__ bool spheres(int i, int j) const {
    float sc, d2 = d2_scale(i, j, sc);
    float t = rb(i) + rb(j) + 1e-3f + 1e-5f * sc;
    return d2 > t * t;
  }
  __device__ __forceinline__ bool box_sphere(int box, int sph) const {
    float sc, d2 = d2_scale(box, sph, sc);
    float t = rl(box) + 3.f * rb(sph) + 1e-3f + 1e-5f * sc;
    return d2 > t * t;
  }
};

// Whether the float32 culls rule out any contact of the ordered pair (i, j).
template <class R> __device__ __forceinline__ bool pair_culled(const NPTile<R>& tl, int i, int j) {
  const int si = tl.shape[i], sj = tl.shape[j];
  const Cull cl{tl.cull, tl.nbs};
  if (sj == 0) return si == 0 ? cl.spheres(i, j) : cl.box_sphere(i, j);
  return si == 0 ? cl.box_sphere(j, i) : cl.boxes(i, j);
}

// One ordered pair (i, j) past the culls with a sphere in it:
// CheckForCollisions(collider i, collider j) (colliders.go:718-747 with the
// forwarding of colliders.go:209-213).
template <class R>
__device__ int sphere_pair(const NPTile<R>& tl, int i, int j, const BatchView<R>& v, int bstart, NPContact<R>& c) {
  const int si = tl.shape[i], sj = tl.shape[j];
  if (si == 0 && sj == 0)
    return sphere_sphere(V<R>(tl.T[9 * tl.nbs + i], tl.T[10 * tl.nbs + i], tl.T[11 * tl.nbs + i]), tl.radius(i), i,
                         V<R>(tl.T[9 * tl.nbs + j], tl.T[10 * tl.nbs + j], tl.T[11 * tl.nbs + j]), tl.radius(j), j, c);
  // a cube and a sphere, in either order: one call site
  const int bx = si != 0 ? i : j, sp = si != 0 ? j : i;
  return cube_sphere(tl.xform(bx), tl.half(bx), bx, tl.xform(sp), tl.radius(sp), sp,
                     v.body + (long long)B_VX * v.nb_pad + bstart + sp, v.nb_pad, c);
}

// Whether a float32 cull rules out any contact of body i with the half-space
// n.x <= offset: a sphere's d = n.c - r (colliders.go:190-192), a cube's
// n.c - (projected half-size) with the projection at most |n| |h|_2
// (colliders.go:750-770); the margin is the pair culls' (1 mm + 1e-5 of the
// magnitudes).  A cube with a non-rigid Offset has an infinite radius.
template <class R> __device__ __forceinline__ bool plane_culled(const NPTile<R>& tl, int i, const BatchView<R>& v) {
  const float nx = (float)v.plane_nx, ny = (float)v.plane_ny, nz = (float)v.plane_nz, off = (float)v.plane_offset;
  const float cx = tl.cull[i], cy = tl.cull[tl.nbs + i], cz = tl.cull[2 * tl.nbs + i];
  const float d = nx * cx + ny * cy + nz * cz;
  const float nlen = sqrtf(nx * nx + ny * ny + nz * nz) * 1.0001f;
  const float r = tl.shape[i] == 0 ? tl.cull[3 * tl.nbs + i] : tl.cull[3 * tl.nbs + i] * nlen;
  const float scale = 1.f + (fabsf(cx) + fabsf(cy) + fabsf(cz)) * nlen + fabsf(off);
  return d - r > off + 1e-3f + 1e-5f * scale;  // false for NaN and infinite radii
}

// ---- bulk async copy (TMA engine) helpers
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
// Bounded wait on an mbarrier phase; false if it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit) {
  unsigned a = smem_addr(bar);
  for (int it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Units past the culls held for their full tests: room for a round of culls
// (up to 1024 units) on top of a partly filled list, and at least one body's
// units (the grid path lists a body's units together).
constexpr int kSurvivors = 1280;
// np_flush's scratch for a CTA of bd threads: the box pairs' penetrations,
// outcomes and the unit that holds them, the chunk's order by kind of test, its
// counts, and per-kind counts of each warp (7 kinds x 8 warps)
template <class R> __host__ __device__ constexpr int np_sort_ints(int bd) {
  return (int)(sizeof(R) / 4) * bd + 4 * bd + 64;
}
__host__ __device__ inline int np_surv_cap(int nbs) { return nbs + 1 > kSurvivors ? ((nbs + 32) & ~31) : kSurvivors; }

template <class R> __host__ __device__ inline size_t np_smem_bytes(int nbs) {
  size_t b = 16;                                  // mbarrier + pad
  b += (size_t)(11 + 12) * nbs * sizeof(R);       // staged rows + transforms
  b += (size_t)nbs * sizeof(int);                 // shape
  b += (size_t)5 * nbs * sizeof(float);           // cull data
  b += 2 * 33 * sizeof(int);                      // scan scratch (double-buffered) + world id + wait outcome
  b += (size_t)np_surv_cap(nbs) * sizeof(int);    // units past the culls, awaiting their full tests
  b += (size_t)np_sort_ints<R>(256) * sizeof(int) + 8;  // np_flush's scratch (aligned)
  return b;
}

// Whether a collider Offset's rotation part is orthonormal to within 1e-5
// (a reflection included): then the collider transform is an isometry up to
// rounding and the cube's bounding radii hold.  NaN fails.
template <class R> __device__ __forceinline__ bool offset_is_rigid(const R (&o)[12]) {
  bool ok = true;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const float d = (float)o[3 * a] * (float)o[3 * b] + (float)o[3 * a + 1] * (float)o[3 * b + 1] +
                      (float)o[3 * a + 2] * (float)o[3 * b + 2];
      ok = ok && fabsf(d - (a == b ? 1.f : 0.f)) <= 1e-5f;
    }
  return ok;
}

// Collider transforms (SetAsTransform x Offset) and the float32 cull data of
// the staged bodies of one world, by the whole CTA.  `off` is the world's
// first body in the Offset rows (row stride `so`), or null for the identity.
// A cube whose Offset is not rigid gets infinite bounding radii: its pairs are
// never culled.
template <class R>
__device__ __forceinline__ void np_build_tile(const NPTile<R>& tl, int n, const R* __restrict__ off, long long so) {
  const int nbs = tl.nbs;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    v3<R> p = V<R>(tl.s(0, i), tl.s(1, i), tl.s(2, i));
    q4<R> q{tl.s(3, i), tl.s(4, i), tl.s(5, i), tl.s(6, i)};
    xf<R> t;
    bool rigid = true;
    if (off) {
      R o[12];
#pragma unroll
      for (int r = 0; r < 12; ++r) o[r] = off[r * so + i];
      t = collider_transform(p, q, o);
      rigid = offset_is_rigid(o);
    } else {
      t = collider_transform(p, q);
    }
#pragma unroll
    for (int r = 0; r < 12; ++r) tl.T[r * nbs + i] = t.m[r];
    float rb, rl;
    if (tl.shape[i] == 0) {
      rb = rl = (float)tl.s(10, i);
    } else if (!rigid) {
      rb = rl = __int_as_float(0x7f800000);
    } else {
      float hx = (float)tl.s(7, i), hy = (float)tl.s(8, i), hz = (float)tl.s(9, i);
      rb = sqrtf(hx * hx + hy * hy + hz * hz) * 1.0001f;
      rl = (hx + hy + hz) * 1.0001f;
    }
    tl.cull[i] = (float)t.m[9];
    tl.cull[nbs + i] = (float)t.m[10];
    tl.cull[2 * nbs + i] = (float)t.m[11];
    tl.cull[3 * nbs + i] = rb;
    tl.cull[4 * nbs + i] = rl;
  }
}

// Block-wide scan of one chunk's per-unit contact counts in unit order: the
// thread's exclusive offset and the chunk total.  The warp totals are
// double-buffered (scan[32 * parity]), so a chunk needs two barriers.
__device__ __forceinline__ void np_chunk_scan(int cnt, int* scan, int parity, int* excl, int* total) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarps = (blockDim.x + 31) >> 5;
  int x = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int y = __shfl_up_sync(FULL, x, d);
    if (lane >= d) x += y;
  }
  int* wt = scan + 32 * parity;
  if (lane == 31) wt[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int t = lane < nwarps ? wt[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int y = __shfl_up_sync(FULL, t, d);
      if (lane >= d) t += y;
    }
    if (lane < nwarps) wt[lane] = t;
  }
  __syncthreads();
  *excl = (wid > 0 ? wt[wid - 1] : 0) + x - cnt;
  *total = wt[nwarps - 1];
}

// Write a contact at slot `off` of the world's contact slab, within its
// capacity.
template <class R>
__device__ __forceinline__ void np_emit(const BatchView<R>& v, long long cs, int cap, int off, const NPContact<R>& c) {
  if (off >= cap) return;
  R* o = v.contact + cs + off;
  const long long S = v.nc_total;
  o[C_PX * S] = c.px; o[C_PY * S] = c.py; o[C_PZ * S] = c.pz;
  o[C_NX * S] = c.nx; o[C_NY * S] = c.ny; o[C_NZ * S] = c.nz;
  o[C_PEN * S] = c.pen;
  o[C_FRIC * S] = (R)0.9;
  o[C_REST * S] = (R)0.1;
  v.contact_bodies[cs + off] = pack_bodies(c.b0, c.b1);
}

// The full tests of the listed units (unit u = i * n + k: k = 0 the
// half-space, else the pair with j = k - 1, skipping i), in chunks of the
// CTA's size, emitting their contacts in list order at out onwards.  Within a
// chunk the units are taken in order of their kind of test (half-space with a
// sphere, with a cube; sphere-sphere, sphere-cube, cube-cube, in float64 with
// i < j ahead of i > j, which mostly take the other order's axes), stably, so the
// lanes of a warp mostly run one test's code; the counts are then scanned in
// list order, so every contact lands where the list order puts it (the
// reference's contact order).  The two tests with many parts are spread over
// lanes: a cube's half-space test takes a lane per vertex (eight), which keeps
// its vertex's contact until the scan says where it goes, and a cube pair's
// axes take sixteen (sat_axes).  On a thread each, a warp ran the eight
// vertices twice (count, write) and the fifteen axes one after the other for
// whatever few lanes had them.  Narrowphase of 8192 worlds x 32 bodies, float64
// 1.50 -> 0.69 ms a frame (0.73 with the two orders of the pairs mixed); of one
// world of 20 cubes in float64 84 -> 39 us.  sortw: np_sort_ints(blockDim.x) ints.
template <class R, bool LARGE>
__device__ void np_flush(const NPTile<R>& tl, const BatchView<R>& v, int bstart, int n, long long cs, int cap,
                         const int* surv, int nsurv, int* scan, int& parity, int& out, uint32_t& err, int* sortw) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, bd = blockDim.x, nwarps = (bd + 31) >> 5;
  R* satp = reinterpret_cast<R*>(((size_t)sortw + 7) & ~(size_t)7);
  int* satc = reinterpret_cast<int*>(satp + bd);  // outcome of the pair held here
  int* satr = satc + bd;                          // the unit holding this unit's outcome; a cube's vertices (bits)
  int* perm = satr + bd;
  int* cntb = perm + bd;
  int* wcnt = cntb + bd;  // [kind * 8 + warp]
  for (int sb = 0; sb < nsurv; sb += bd) {
    const int m = nsurv - sb < bd ? nsurv - sb : bd;
    constexpr bool kOrders = sizeof(R) == 8;  // (in float32 the kind costs what it saves)
    int key = kOrders ? 6 : 5;  // no unit
    if (tid < m) {
      const int uu = surv[sb + tid];
      const int i = uu / n, k = uu - i * n;
      if (k == 0) {
        key = tl.shape[i] != 0 ? 1 : 0;
      } else {
        int j = k - 1;
        if (j >= i) ++j;
        key = 2 + (tl.shape[i] != 0 ? 1 : 0) + (tl.shape[j] != 0 ? 1 : 0);
        if (kOrders && key == 4 && i > j) key = 5;
      }
    }
    int rank = 0;
#pragma unroll
    for (int q = 0; q < (kOrders ? 7 : 6); ++q) {
      const unsigned bal = __ballot_sync(FULL, key == q);
      if (key == q) rank = __popc(bal & ((1u << lane) - 1u));
      if (lane == 0) wcnt[q * 8 + wid] = __popc(bal);
    }
    __syncthreads();
    int dst = rank, n0 = 0, n1 = 0, n23 = 0, n4 = 0;
    for (int w2 = 0; w2 < nwarps; ++w2) {
      const int a = wcnt[w2], b = wcnt[8 + w2], c2 = wcnt[16 + w2], c3 = wcnt[24 + w2], d = wcnt[32 + w2];
      const int e = kOrders ? wcnt[40 + w2] : 0;
      n0 += a;
      n1 += b;
      n23 += c2 + c3;
      n4 += d + e;
      dst += (key > 0 ? a : 0) + (key > 1 ? b : 0) + (key > 2 ? c2 : 0) + (key > 3 ? c3 : 0) + (key > 4 ? d : 0) +
             (kOrders && key > 5 ? e : 0);
      if (w2 < wid) dst += wcnt[key * 8 + w2];
    }
    perm[dst] = tid;
    __syncthreads();
    // Cube pairs: an axis per lane.  With Offsets, cubes whose Offset is not
    // rigid are never culled and most of their pairs are apart: where there are
    // more than two passes, a lane per pair tries three axes first (1000 worlds
    // of 31 bodies, float32: 54 -> 41 us; without Offsets the culls leave near
    // pairs, and 8192 x 32 settled bodies took 187 us with it, 175 without).
    // In a world of more than kPairedBodies the chunks are full of pairs whose
    // other order is in another chunk.  float32 then takes a lane per pair for
    // all its axes, float64 the three axes first (LARGE: the code is left out where
    // no world needs it).  64 piles of 1024 cubes, falling and settled: float32
    // 1.24 -> 0.91 and 2.19 -> 1.73 ms a frame, float64 3.90 -> 1.69 and 7.43 ->
    // 6.05; 600 of 72, float64, 0.82 -> 0.27 and 1.53 -> 1.33.
    const bool large = LARGE && n > kPairedBodies;
    const bool serial = sizeof(R) == 4 && large;
    if (serial) {
      if (tid < n4) {
        const int at = perm[n0 + n1 + n23 + tid];
        const int uu = surv[sb + at];
        const int i = uu / n, k = uu - i * n;
        const SatResult<R> r = sat_serial(tl, i, k - 1 >= i ? k : k - 1);
        satp[at] = r.pen;
        satc[at] = r.code;
        satr[at] = at;
      }
      n4 = 0;
    }
    const bool pre = (v.offset != nullptr || large) && n4 > bd >> 3;
    if (pre) {
      if (tid < n4) {
        const int at = perm[n0 + n1 + n23 + tid];
        const int uu = surv[sb + at];
        const int i = uu / n, k = uu - i * n;
        satc[at] = sat_apart_first(tl, i, k - 1 >= i ? k : k - 1) ? kSatApart : 0;
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int g = tid >> 4; g < ((n4 + 1) & ~1); g += bd >> 4) {  // both groups of a warp together
      const bool on = g < n4;
      const int at = perm[n0 + n1 + n23 + (on ? g : 0)], l = tid & 15;
      const int uu = surv[sb + at];
      const int i = uu / n, k = uu - i * n;
      const int j = k - 1 >= i ? k : k - 1;
      // (i, j) with i > j takes the outcome of (j, i) where the chunk has it
      int other = -1;
      const bool apart = pre && satc[at] == kSatApart;
      if (on && i > j && !apart)
        for (int q = l; q < m; q += 16)
          if (surv[sb + q] == j * n + i) other = q;  // j's k is i: i > j
      const unsigned have = __ballot_sync(FULL, other >= 0) & (0xFFFFu << (lane & 16));
      other = __shfl_sync(FULL, other, have ? __ffs(have) - 1 : lane);
      const bool need = on && !have && !apart;
      if (__any_sync(FULL, need)) {
        const SatResult<R> r = sat_axes(tl, i, j, l);
        if (need && l == 0) {
          satp[at] = r.pen;
          satc[at] = r.code;
        }
      }
      if (on && l == 0) satr[at] = have ? other : at;
    }
    // half-space with a cube: a vertex per lane; in float64 the last pass keeps
    // its contacts (in float32 they are computed again: held, they cost a CTA per SM)
    constexpr bool kKeep = sizeof(R) == 8;
    NPContact<R> vc;
    bool vhit = false;
    const int passes = (8 * n1 + bd - 1) / bd;
#pragma unroll 1
    for (int q = 0; q < passes; ++q) {
      const int g = (q * bd + tid) >> 3;
      const int at = perm[n0 + (g < n1 ? g : 0)];
      vhit = g < n1 && plane_vertex(tl, surv[sb + at] / n, tid & 7, v, vc);
      const unsigned bits = (__ballot_sync(FULL, vhit) >> (lane & 24)) & 0xFFu;
      if (g < n1 && (tid & 7) == 0) satr[at] = (int)bits;
    }
    __syncthreads();
    const int src = perm[tid];  // this thread tests the chunk's unit src
    int cnt = 0;
    bool cube_plane = false;
    NPContact<R> c;
    if (src < m) {
      const int uu = surv[sb + src];
      const int i = uu / n, k = uu - i * n;
      const int j = k - 1 >= i ? k : k - 1;
      cube_plane = k == 0 && tl.shape[i] != 0;
      if (cube_plane) {
        cnt = __popc((unsigned)satr[src]);
      } else if (k == 0) {
        cnt = plane_sphere(tl, i, v, c);
      } else if (tl.shape[i] != 0 && tl.shape[j] != 0) {
        const int at = satr[src];
        int code = satc[at];
        if (code != kSatApart) {
          if (at != src) code = (int)((unsigned)code >> 16);  // the pair's other order
          cnt = cube_contact(tl, i, j, code & 0xFF, (code >> 8) & 0x7F, satp[at], c, err);
        }
      } else {
        cnt = sphere_pair(tl, i, j, v, bstart, c);
      }
    }
    cntb[src] = cnt;
    __syncthreads();
    int excl, total;
    np_chunk_scan(cntb[tid], scan, parity, &excl, &total);  // list order
    parity ^= 1;
    cntb[tid] = excl;
    __syncthreads();
    if (cnt > 0 && !cube_plane) np_emit<R>(v, cs, cap, out + cntb[src], c);
#pragma unroll 1
    for (int q = passes - 1; q >= 0; --q) {
      const int g = (q * bd + tid) >> 3;
      if (g < n1) {
        const int at = perm[n0 + g];
        if (!kKeep || q < passes - 1) vhit = plane_vertex(tl, surv[sb + at] / n, tid & 7, v, vc);
        if (vhit) np_emit<R>(v, cs, cap, out + cntb[at] + __popc((unsigned)satr[at] & ((1u << (tid & 7)) - 1u)), vc);
      }
    }
    out += total;
    __syncthreads();  // perm and cntb are reused by the next chunk
  }
}

// ---- broadphase: a uniform grid over a large world's bodies
//
// A pair (i, j) passes the float32 culls only if its centres are within
// reach_i + reach_j + 1 mm + 1e-5 (1 + |c_i|_1 + |c_j|_1), with reach = the
// larger of 1.1 |h|_2 and |h|_1 for a box, 3 r for a sphere (the thresholds
// of Cull).  With cells at least that wide for every pair of the world, the
// pairs the culls keep are all between neighbouring cells: the grid drops
// only pairs the culls reject.  Each body's kept units are listed in
// ascending unit order and bodies in index order, so the contact list is the
// all-pairs path's, bit for bit.

// Grid scratch inside the staged position / orientation rows, which are
// dead once the collider transforms are built.
struct NPGrid {
  float* red;   // [8 warps][8] block reductions
  int* info;    // [8]: ok, gx, gy, gz, ncells, last list length
  float* finfo; // [4]: origin xyz, cell size
  int* cell;    // [cells_cap + 1] counts, then cursor / end of each cell
  int* sorted;  // [n] bodies ordered by cell
  int* cellof;  // [n] linear cell of each body
  int cells_cap;
};

template <class R> __device__ __forceinline__ NPGrid np_grid_scratch(const NPTile<R>& tl) {
  NPGrid g;
  unsigned char* base = reinterpret_cast<unsigned char*>(tl.stage);
  const int words = (int)((size_t)7 * tl.nbs * sizeof(R) / 4);
  g.red = reinterpret_cast<float*>(base);
  g.info = reinterpret_cast<int*>(base) + 64;
  g.finfo = reinterpret_cast<float*>(g.info + 8);
  g.sorted = g.info + 12;
  g.cellof = g.sorted + tl.nbs;
  g.cell = g.cellof + tl.nbs;
  g.cells_cap = words - 76 - 2 * tl.nbs - 1;
  return g;
}

// Block-wide max of 8 floats (NaN in any input gives NaN through the
// comparison trick below: a value that is not >= itself is kept).
__device__ __forceinline__ void np_block_max8(float (&x)[8], float* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float y = __shfl_xor_sync(FULL, x[q], d);
      x[q] = (y > x[q] || y != y) ? y : x[q];
    }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < 8; ++q) red[wid * 8 + q] = x[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    float m = red[q];
    for (int k = 1; k < nw; ++k) {
      const float y = red[k * 8 + q];
      m = (y > m || y != y) ? y : m;
    }
    x[q] = m;
  }
  __syncthreads();
}

// Builds the grid of one world; false (uniform over the CTA) when it would
// not help or cannot be sized: non-finite centres or radii (a non-rigid
// Offset's infinite radius included), or more cells than the scratch holds.
template <class R> __device__ bool np_grid_build(const NPTile<R>& tl, int n, const NPGrid& g, int* scan, int& parity) {
  const int nbs = tl.nbs;
  float x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = -__int_as_float(0x7f800000);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float cx = tl.cull[i], cy = tl.cull[nbs + i], cz = tl.cull[2 * nbs + i];
    const float rb = tl.cull[3 * nbs + i], rl = tl.cull[4 * nbs + i];
    const float reach = tl.shape[i] == 0 ? 3.f * rb : fmaxf(1.1f * rb, rl);
    const float fin = (isfinite(cx) && isfinite(cy) && isfinite(cz) && isfinite(reach)) ? 0.f : 1.f;
    // max of: the centres (the box's upper corner), their negations (the
    // lower corner), the reach, non-finite flag
    const float v8[8] = {cx, cy, cz, -cx, -cy, -cz, reach, fin};
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = (v8[q] > x[q] || v8[q] != v8[q]) ? v8[q] : x[q];
  }
  np_block_max8(x, g.red);
  if (threadIdx.x == 0) {
    int ok = x[7] == 0.f && x[6] == x[6];
    // |c|_1 of every centre is at most the larger corner's per axis
    const float m1 = fmaxf(fabsf(x[0]), fabsf(x[3])) + fmaxf(fabsf(x[1]), fabsf(x[4])) +
                     fmaxf(fabsf(x[2]), fabsf(x[5]));
    // cell size: every kept pair is within 2 * max reach + the culls' margin
    const float L = (2.f * x[6] + 1e-3f + 1e-5f * (1.f + 2.f * m1)) * 1.001f + 1e-6f;
    const float ox = -x[3], oy = -x[4], oz = -x[5];
    int gx = 0, gy = 0, gz = 0;
    if (ok && L > 0.f) {
      const float ex = (x[0] - ox) / L, ey = (x[1] - oy) / L, ez = (x[2] - oz) / L;
      ok = ex < 1e6f && ey < 1e6f && ez < 1e6f;
      if (ok) {
        gx = (int)ex + 1;
        gy = (int)ey + 1;
        gz = (int)ez + 1;
        ok = (long long)gx * gy * gz <= g.cells_cap;
      }
    } else {
      ok = 0;
    }
    g.info[0] = ok;
    g.info[1] = gx;
    g.info[2] = gy;
    g.info[3] = gz;
    g.info[4] = gx * gy * gz;
    g.finfo[0] = ox;
    g.finfo[1] = oy;
    g.finfo[2] = oz;
    g.finfo[3] = L;
  }
  __syncthreads();
  if (!g.info[0]) return false;
  const int gx = g.info[1], gy = g.info[2], gz = g.info[3], nc = g.info[4];
  const float ox = g.finfo[0], oy = g.finfo[1], oz = g.finfo[2], L = g.finfo[3];
  for (int c = threadIdx.x; c <= nc; c += blockDim.x) g.cell[c] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int cx = min((int)((tl.cull[i] - ox) / L), gx - 1);
    const int cy = min((int)((tl.cull[nbs + i] - oy) / L), gy - 1);
    const int cz = min((int)((tl.cull[2 * nbs + i] - oz) / L), gz - 1);
    const int c = (cz * gy + cy) * gx + cx;
    g.cellof[i] = c;
    atomicAdd(&g.cell[c], 1);
  }
  __syncthreads();
  // exclusive scan of the counts: cell[c] = first slot of cell c
  int run = 0;
  for (int b0 = 0; b0 < nc; b0 += blockDim.x) {
    const int c = b0 + threadIdx.x;
    const int cnt = c < nc ? g.cell[c] : 0;
    int excl, total;
    np_chunk_scan(cnt, scan, parity, &excl, &total);
    parity ^= 1;
    if (c < nc) g.cell[c] = run + excl;
    run += total;
  }
  __syncthreads();
  // scatter; afterwards cell[c] is the end of cell c (the start of c + 1)
  for (int i = threadIdx.x; i < n; i += blockDim.x) g.sorted[atomicAdd(&g.cell[g.cellof[i]], 1)] = i;
  __syncthreads();
  return true;
}

// Body i's units past the culls from its 27 neighbouring cells: counted, or
// written at dst (plane unit, then the pairs, unsorted).
template <class R>
__device__ int np_grid_units(const NPTile<R>& tl, const BatchView<R>& v, const NPGrid& g, int n, int i, int* dst) {
  int cnt = 0;
  if (!plane_culled(tl, i, v)) {
    if (dst) dst[cnt] = i * n;
    ++cnt;
  }
  const int gx = g.info[1], gy = g.info[2], gz = g.info[3];
  const int c = g.cellof[i];
  const int cx = c % gx, cy = (c / gx) % gy, cz = c / (gx * gy);
  for (int dz = -1; dz <= 1; ++dz) {
    if (cz + dz < 0 || cz + dz >= gz) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      if (cy + dy < 0 || cy + dy >= gy) continue;
      for (int dx = -1; dx <= 1; ++dx) {
        if (cx + dx < 0 || cx + dx >= gx) continue;
        const int nc = ((cz + dz) * gy + cy + dy) * gx + cx + dx;
        const int s0 = nc == 0 ? 0 : g.cell[nc - 1], s1 = g.cell[nc];
        for (int s = s0; s < s1; ++s) {
          const int j = g.sorted[s];
          if (j == i || pair_culled(tl, i, j)) continue;
          if (dst) dst[cnt] = i * n + (j < i ? j + 1 : j);
          ++cnt;
        }
      }
    }
  }
  return cnt;
}

// The narrowphase of world w, its bodies' tile built: the ordered units
// culled, the kept ones listed (scap of them at a time) and tested, the
// contacts emitted in the reference's order; sets the world's contact count.
// Every thread of the CTA calls it.
template <class R, NPMode MODE>
__device__ void np_world(const NPTile<R>& tl, const BatchView<R>& v, int w, int n, int bstart, int* scan,
                         int& chunk_parity, int* surv, int scap) {
  const int tid = threadIdx.x;
  const long long cs = v.contact_start[w];
  const int cap = v.contact_cap[w];
  const int U = n * n;  // ordered units: for body i, the half-space (k = 0), then k - 1 = j skipping i
  int out = 0, nsurv = 0;
  uint32_t err = 0;
  const NPGrid g = np_grid_scratch(tl);
  if (MODE == NP_GRID && v.grid_min_bodies > 0 && n >= v.grid_min_bodies && np_grid_build(tl, n, g, scan, chunk_parity)) {
    // Grid: each body's kept units (counted, then listed and sorted), as
    // many bodies at a time as the list holds, then their full tests.
    for (int ib = 0; ib < n;) {
      const int i = ib + tid;
      const int cnt = i < n ? np_grid_units(tl, v, g, n, i, nullptr) : 0;
      int excl, total;
      np_chunk_scan(cnt, scan, chunk_parity, &excl, &total);
      chunk_parity ^= 1;
      const bool fits = i < n && excl + cnt <= scap;  // a prefix of the bodies: at least body ib
      const int m = __syncthreads_count(fits);
      if (fits) {
        int* d = surv + excl;
        np_grid_units(tl, v, g, n, i, d);
        for (int a = 1; a < cnt; ++a) {  // ascending unit order (the plane unit, k = 0, first)
          const int key = d[a];
          int b = a - 1;
          while (b >= 0 && d[b] > key) {
            d[b + 1] = d[b];
            --b;
          }
          d[b + 1] = key;
        }
        if (tid == m - 1) g.info[5] = excl + cnt;
      }
      __syncthreads();
      nsurv = g.info[5];
      np_flush<R, MODE != NP_SMALL>(tl, v, bstart, n, cs, cap, surv, nsurv, scan, chunk_parity, out, err, surv + scap);
      __syncthreads();
      ib += m;
    }
  } else {
    // All pairs: the culls run over every unit, upt consecutive units per
    // thread and one scan per round; the units they keep are listed in unit
    // order and get their full tests in chunks of the CTA's size, so the
    // lanes of a warp run the costly tests together.  Counting, scanning and
    // emitting in list order keeps the reference's contact order.
    const int bd = blockDim.x;
    int upt = (scap - bd) / bd;
    upt = upt < 1 ? 1 : (upt > 8 ? 8 : upt);
    const int round = bd * upt;  // at most scap - bd: the list never overflows
    for (int base = 0; base < U; base += round) {
      const int u0 = base + tid * upt;
      unsigned keep = 0;
      if (u0 < U) {
        int i = u0 / n, k = u0 - i * n;
        for (int q = 0; q < upt && u0 + q < U; ++q) {
          int j = k - 1;
          if (j >= i) ++j;
          if (k == 0 ? !plane_culled(tl, i, v) : !pair_culled(tl, i, j)) keep |= 1u << q;
          if (++k == n) {
            k = 0;
            ++i;
          }
        }
      }
      int excl, total;
      np_chunk_scan(__popc(keep), scan, chunk_parity, &excl, &total);
      chunk_parity ^= 1;
      for (int o = nsurv + excl; keep; keep &= keep - 1) surv[o++] = u0 + __ffs(keep) - 1;
      nsurv += total;
      if (nsurv <= scap - round && base + round < U) continue;
      __syncthreads();
      np_flush<R, MODE != NP_SMALL>(tl, v, bstart, n, cs, cap, surv, nsurv, scan, chunk_parity, out, err, surv + scap);
      nsurv = 0;
      __syncthreads();
    }
  }
  if (err) {
    atomicOr(&v.world_status[w], err);
    atomicOr(v.status, err);
  }
  if (tid == 0) {
    v.contact_count[w] = out;
    atomicAdd(&v.counters[0], (unsigned long long)out);
    if (out > cap) {
      atomicOr(&v.world_status[w], ST_CAPACITY);
      atomicOr(v.status, ST_CAPACITY);
    }
  }
}

// NP_SMALL and NP_LARGE compile the all-pairs path alone (worlds too small for
// the grid), so its registers and occupancy stay those of that path; in float32
// it is bounded to 64 registers (8 CTAs of 128 threads per SM; 240 bytes
// spilled): with few contacts a world is a chain of staging and barriers, and
// 16384 worlds of 14 bodies took 155 us against 178 with 80 registers (6 CTAs);
// 8192 worlds of 32 settled bodies 175 against 170, and 200 unbounded.
template <class R, NPMode MODE>
__global__ void __launch_bounds__(256, sizeof(R) == 4 && MODE != NP_GRID ? 4 : 0) k_narrowphase(BatchView<R> v, int nbs) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem);
  NPTile<R> tl;
  tl.nbs = nbs;
  tl.stage = reinterpret_cast<R*>(smem + 16);
  tl.T = tl.stage + 11 * nbs;
  tl.shape = reinterpret_cast<int*>(tl.T + 12 * nbs);
  tl.cull = reinterpret_cast<float*>(tl.shape + nbs);
  int* scan = reinterpret_cast<int*>(tl.cull + 5 * nbs);  // [2][32] + [64] world id + [65] wait outcome
  int* surv = scan + 66;                                   // [kSurvivors] units past the culls
  const int tid = threadIdx.x;
  if (tid == 0) mbar_init(bar, 1);
  __syncthreads();
  unsigned phase = 0;
  int chunk_parity = 0;
  for (;;) {
    if (tid == 0) {
      unsigned q = atomicAdd(&v.queue[0], 1u);
      scan[64] = q < (unsigned)v.num_worlds ? v.order[q] : -1;
    }
    __syncthreads();
    const int w = scan[64];
    if (w < 0) break;
    const int n = v.body_count[w];
    const int bstart = v.body_start[w];
    if (n > nbs) {
      if (tid == 0) {
        v.world_status[w] |= ST_BODY_LIMIT;
        atomicOr(v.status, ST_BODY_LIMIT);
        v.contact_count[w] = 0;
      }
      __syncthreads();
      continue;
    }
    const int n4 = (n + 3) & ~3;
    if (tid == 0 && n4 > 0) {
      // order smem accesses of the previous world before the async-proxy writes
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      const unsigned rb = (unsigned)(n4 * sizeof(R));
      mbar_expect_tx(bar, rb * 11u + (unsigned)(n4 * sizeof(int)) + (unsigned)v.wait_extra_tx);
#pragma unroll 1
      for (int r = 0; r < 11; ++r) bulk_g2s(tl.stage + r * nbs, v.body + (long long)r * v.nb_pad + bstart, rb, bar);
      bulk_g2s(tl.shape, v.shape + bstart, (unsigned)(n4 * sizeof(int)), bar);
    }
    if (n4 > 0) {
      // Thread 0 waits, bounded, and decides for the CTA; the others then
      // observe the completed phase themselves (their acquire of the copies).
      if (tid == 0) scan[65] = mbar_wait(bar, phase, v.wait_limit) ? 1 : 0;
      __syncthreads();
      const bool ok = scan[65] != 0;
      if (!ok) {
        // Give up on this CTA's worlds (the copies are a few KB, so this
        // signals a fault) and report it.  The copies issued may still be
        // landing in this CTA's shared memory: one more bounded wait for
        // them before the CTA ends.
        if (tid == 0) {
          v.world_status[w] |= ST_TIMEOUT;
          atomicOr(v.status, ST_TIMEOUT);
          mbar_wait(bar, phase, v.wait_limit);
        }
        __syncthreads();
        return;
      }
      if (tid != 0) mbar_wait(bar, phase, v.wait_limit);
      phase ^= 1u;
    }
    np_build_tile(tl, n, v.offset ? v.offset + bstart : nullptr, v.nb_pad);
    __syncthreads();
    np_world<R, MODE>(tl, v, w, n, bstart, scan, chunk_parity, surv, np_surv_cap(nbs));
    __syncthreads();
  }
}

// The narrowphase for a caller's list of units of one world (colliders.go:
// CheckAgainstHalfSpace when j < 0, else CheckForCollisions(i, j)), in the
// list's order, replacing the world's contact list: one CTA, bodies staged by
// plain loads, the same tests, scan and emission as k_narrowphase.  Indices
// are validated by the host.
template <class R>
__global__ void __launch_bounds__(256) k_collide(BatchView<R> v, int w, const int2* __restrict__ units, int nunits,
                                                 int nbs) {
  extern __shared__ __align__(128) unsigned char smem[];
  NPTile<R> tl;
  tl.nbs = nbs;
  tl.stage = reinterpret_cast<R*>(smem + 16);
  tl.T = tl.stage + 11 * nbs;
  tl.shape = reinterpret_cast<int*>(tl.T + 12 * nbs);
  tl.cull = reinterpret_cast<float*>(tl.shape + nbs);
  int* scan = reinterpret_cast<int*>(tl.cull + 5 * nbs);
  const int tid = threadIdx.x;
  const int n = v.body_count[w];
  const int bstart = v.body_start[w];
  for (int i = tid; i < n; i += blockDim.x) {
#pragma unroll
    for (int r = 0; r < 11; ++r) tl.stage[r * nbs + i] = v.body[(long long)r * v.nb_pad + bstart + i];
    tl.shape[i] = v.shape[bstart + i];
  }
  __syncthreads();
  np_build_tile(tl, n, v.offset ? v.offset + bstart : nullptr, v.nb_pad);
  __syncthreads();
  const long long cs = v.contact_start[w];
  const int cap = v.contact_cap[w];
  int* surv = scan + 66;
  const int scap = np_surv_cap(nbs);
  int out = 0, parity = 0, nsurv = 0;
  uint32_t err = 0;
  for (int base = 0; base < nunits; base += blockDim.x) {
    const int u = base + tid;
    bool keep = false;
    int2 un = make_int2(0, 0);
    if (u < nunits) {
      un = units[u];
      keep = un.y < 0 ? !plane_culled(tl, un.x, v) : !pair_culled(tl, un.x, un.y);
    }
    int excl, total;
    np_chunk_scan(keep ? 1 : 0, scan, parity, &excl, &total);
    parity ^= 1;
    if (keep) surv[nsurv + excl] = un.x * n + (un.y < 0 ? 0 : (un.y < un.x ? un.y + 1 : un.y));
    nsurv += total;
    if (nsurv + (int)blockDim.x <= scap && base + (int)blockDim.x < nunits) continue;
    __syncthreads();
    np_flush<R, true>(tl, v, bstart, n, cs, cap, surv, nsurv, scan, parity, out, err, surv + scap);
    nsurv = 0;
    __syncthreads();
  }
  if (err) {
    atomicOr(&v.world_status[w], err);
    atomicOr(v.status, err);
  }
  if (tid == 0) {
    v.contact_count[w] = out;
    atomicAdd(&v.counters[0], (unsigned long long)out);
    if (out > cap) {
      atomicOr(&v.world_status[w], ST_CAPACITY);
      atomicOr(v.status, ST_CAPACITY);
    }
  }
}

}  // namespace cz

#include "cz_resolve.cuh"
#include "cz_resolve_big.cuh"
