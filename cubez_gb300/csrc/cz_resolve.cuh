// ResolveContacts (contact.go:204-445) for batches of worlds.
//
// One warp holds 32 / G worlds; the G lanes of a world solve its islands (the
// connected components of its contacts, build_islands) side by side, eight
// lanes to an island.  Within a group of lanes the contacts are lane-strided:
// the argmax is a butterfly whose tie-break is the reference's first-maximum
// rule, and the per-iteration update of every contact touching the two
// resolved bodies is lane-parallel.  The change of the resolved contact's two
// bodies is spread over the group: lane 4i + c forms component c of body i
// (velocity_change, position_change), and the changes reach the updated
// contacts by shuffles.  On GB300 a float64 warp instruction costs the same
// pipe time whatever its active mask, and a float32 iteration is bound by the
// instructions it issues, so both forms gain from lanes that work side by
// side: several islands (or worlds) in one instruction, and one component per
// lane instead of all of them on one.
//
// A contact's working values are one record (CREC reals), a body's another
// (BREC): an update reads four or five 16-byte pieces of one record where the
// rows of a structure of arrays took seventeen loads, each with its own
// address.  The friction solve's matrices do not change during
// adjustVelocities and are computed once per contact, off the chain
// (friction_prepare).
//
// Also here: k_resolve_wide (small batches: four warps to a world),
// k_warm_features (the learned warm start's features, tensor-core inference and
// plan, launched before k_resolve) and the shared pieces of k_resolve_big
// (cz_resolve_big.cuh).
#pragma once
#include <type_traits>

#include "cz_layout.cuh"
#include "cz_math.cuh"
#include "cz_mlp.cuh"

namespace cz {

// calculateContactBasis's second column, contact.go:114-156: a function of
// the normal alone.
template <class R> __device__ __forceinline__ v3<R> contact_tangent(const v3<R>& n) {
  if (fabs_<R>(n.x) > fabs_<R>(n.y)) {
    const R s = (R)1 / sqrt_<R>(n.z * n.z + n.x * n.x);
    return V<R>(n.z * s, (R)0, n.x * -s);
  }
  const R s = (R)1 / sqrt_<R>(n.z * n.z + n.y * n.y);
  return V<R>((R)0, -n.z * s, n.y * s);
}
// its third column (contact.go:136-138, 149-151), from the first two
template <class R> __device__ __forceinline__ v3<R> contact_bitangent(const v3<R>& n, const v3<R>& ty) {
  if (fabs_<R>(n.x) > fabs_<R>(n.y)) return V<R>(n.y * ty.x, n.z * ty.x - n.x * ty.z, -n.y * ty.x);
  return V<R>(n.y * ty.z - n.z * ty.y, -n.x * ty.z, n.x * ty.y);
}

// four consecutive reals of a record (16- or 32-byte aligned)
template <class R> struct quad {
  R a, b, c, d;
};
__device__ __forceinline__ quad<float> ld4(const float* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  return {t.x, t.y, t.z, t.w};
}
__device__ __forceinline__ quad<double> ld4(const double* p) {
  const double2 s = reinterpret_cast<const double2*>(p)[0], t = reinterpret_cast<const double2*>(p)[1];
  return {s.x, s.y, t.x, t.y};
}
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void st4(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

// The resolver's view of one world.
template <class R, class W, bool SM> struct RCtx {
  W* bw;        // [n][7]: position xyz, orientation wxyz (island type)
  R* br;        // [n][BREC]: body records
  uint8_t* aw;  // [n] awake
  int nbs;
  R* cr;        // [C][CREC]: contact records
  // packed bodies of this world's contacts.  SM (worlds of at most 64 bodies):
  // bits 0-7 and 8-15 the bodies (0xFF: none), bits 16-31 the contact's index
  // in the narrowphase's list (the records are in island order); else the
  // narrowphase's packing (pack_bodies), and the records in its order
  int* cb;
  R* delta;  // warm start: [6] rows of the velocity and rotation change per body (row stride wst)
  int* wi;   // [WS_NINT] integer rows (WsInt)
  long long wst;
  R* jw;     // impulse rows J0..J2 of the learned paths, by the contact's list index (row stride jst)
  long long jst;
  R* kw;     // per contact, K_ROW reals: K of the friction solve (inverted in W, kept in R), 9,
             // then the response matrix's first row, 3
  const R* gmat;  // friction / restitution rows of the contact list (null: 0.9 / 0.1)
  long long gst;
  R dt;
  bool all_awake;  // every body of the warp's worlds was awake when loaded
  static __device__ __forceinline__ int B0(int p) { return SM ? p & 0xFF : body0_of(p); }
  static __device__ __forceinline__ int B1(int p) {
    if (!SM) return body1_of(p);
    const int b = (p >> 8) & 0xFF;
    return b == 0xFF ? -1 : b;
  }
  __device__ __forceinline__ void set_pair(int k, int b0, int b1, int list_index) const {
    cb[k] = SM ? (int)((b0 & 0xFFu) | ((b1 & 0xFFu) << 8) | ((unsigned)list_index << 16)) : pack_bodies(b0, b1);
  }
  __device__ __forceinline__ int pair(int k) const { return cb[k]; }
  // the contact's index in the narrowphase's list
  __device__ __forceinline__ int list_index(int k) const { return SM ? (int)((unsigned)cb[k] >> 16) : k; }
  __device__ __forceinline__ W& P(int c, int i) const { return bw[i * 7 + c]; }
  __device__ __forceinline__ R* body(int i) const { return br + i * BREC; }
  __device__ __forceinline__ R* rec(int k) const { return cr + (long long)k * CREC; }
  __device__ __forceinline__ R& J(int c, int o) const { return jw[(long long)c * jst + o]; }
  __device__ __forceinline__ const R* krow(int k) const { return kw + (long long)k * K_ROW; }
  __device__ __forceinline__ int& WI(int r, int i) const { return wi[(long long)r * wst + i]; }
  __device__ __forceinline__ R& Delta(int r, int i) const { return delta[(long long)r * wst + i]; }
  __device__ __forceinline__ v3<R> Bv(int r, int i) const {
    const R* b = body(i) + r;
    return V<R>(b[0], b[1], b[2]);
  }
  __device__ __forceinline__ m3<R> iit(int i) const {
    m3<R> m;
    const R* b = body(i) + BR_IIT;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.m[k] = b[k];
    return m;
  }
  // materials, by list index
  __device__ __forceinline__ R friction(int o) const { return gmat ? gmat[o] : (R)0.9; }
  __device__ __forceinline__ R restitution(int o) const { return gmat ? gmat[gst + o] : (R)0.1; }
  // contactToWorld: columns normal, tangent y, tangent z
  __device__ __forceinline__ m3<R> basis(int k) const {
    const R* r = rec(k);
    const quad<R> a = ld4(r), b = ld4(r + 4);
    m3<R> m;
    m.m[0] = a.a; m.m[1] = a.b; m.m[2] = a.c; m.m[3] = a.d;
    m.m[4] = b.a; m.m[5] = b.b; m.m[6] = b.c; m.m[7] = b.d;
    m.m[8] = r[8];
    return m;
  }
  __device__ __forceinline__ v3<R> rel(int side, int k) const {
    const R* r = rec(k) + (side == 0 ? CR_R0 : CR_R1);
    return V<R>(r[0], r[1], r[2]);
  }
};

// ---------------------------------------------------------------- argmax keys
// Order-preserving keys: key(v) > 0 exactly when v > eps and v is not NaN;
// for such values key order is value order (IEEE bit patterns of positive
// numbers sort like the numbers).
__device__ __forceinline__ unsigned long long key_of(double v, double eps) {
  long long b = __double_as_longlong(v);
  long long e = __double_as_longlong(eps);
  return (b > e && b <= 0x7FF0000000000000LL) ? (unsigned long long)b : 0ull;
}
__device__ __forceinline__ unsigned key_of(float v, float eps) {
  int b = __float_as_int(v);
  int e = __float_as_int(eps);
  return (b > e && b <= 0x7F800000) ? (unsigned)b : 0u;
}

// The first maximum over a whole warp by warp reductions (redux.sync): the
// largest key, then the smallest index among the lanes holding it; a 64-bit
// key is reduced by its high half, then its low half.
__device__ __forceinline__ void warp_first_max(unsigned& key, int& idx) {
  const unsigned m = __reduce_max_sync(0xffffffffu, key);
  idx = (int)__reduce_min_sync(0xffffffffu, key == m ? (unsigned)idx : 0xffffffffu);
  key = m;
}
__device__ __forceinline__ void warp_first_max(unsigned long long& key, int& idx) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  idx = (int)__reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? (unsigned)idx : 0xffffffffu);
  key = ((unsigned long long)mh << 32) | ml;
}

// Largest key over the L lanes of a group, smallest index among equal keys
// (the first maximum of the reference's scan, contact.go:238-245, 394-402).
template <int L, class K> __device__ __forceinline__ void group_first_max(K& key, int& idx) {
  if constexpr (L == 32) {
    warp_first_max(key, idx);
  } else {
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1) {
      const K ok = __shfl_xor_sync(0xffffffffu, key, off);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
      if (ok > key || (ok == key && oi < idx)) {
        key = ok;
        idx = oi;
      }
    }
  }
}

// The last frame's acceleration along contact k's normal over the frame, of
// its awake bodies (contact.go:88-101).  It changes only with the awake flags
// of its bodies, so adjustVelocities keeps it in the record (CR_VFA) and
// forms it again where a body woke.
template <class R, class W, bool SM>
__device__ __forceinline__ R frame_velocity(const RCtx<R, W, SM>& x, int b0, int b1, const v3<R>& n) {
  R vfa = (R)0;
  // LastFrameAcceleration * duration, formed when the body is loaded (the
  // reference's product, once instead of at every use)
  if (x.aw[b0]) vfa += dot(x.Bv(BR_LFA, b0), n);
  if (b1 >= 0 && x.aw[b1]) vfa -= dot(x.Bv(BR_LFA, b1), n);
  return vfa;
}
// calculateDesiredDeltaVelocity, contact.go:87-112
template <class R> __device__ __forceinline__ R desired_dv(R cvx, R vfa, R restitution) {
  const R rest = fabs_<R>(cvx) < (R)0.25 ? (R)0 : restitution;
  return -cvx - rest * (cvx - vfa);
}

// calculateLocalVelocity, contact.go:158-182
template <class R, class W, bool SM>
__device__ __forceinline__ v3<R> local_velocity(const RCtx<R, W, SM>& x, int body, const v3<R>& rp, const m3<R>& C) {
  v3<R> vel = cross(x.Bv(BR_ROT, body), rp);
  add(vel, x.Bv(BR_VEL, body));
  v3<R> cv = mulv_t(C, vel);
  v3<R> acc = x.Bv(BR_LFA, body);  // LastFrameAcceleration * duration
  acc = mulv_t(C, acc);
  acc.x = (R)0;
  add(cv, acc);
  return cv;
}

// calculateInternals, contact.go:59-85, of the contact at list index o (row
// src of the narrowphase's rows), into record k.
template <class R, class W, bool SM>
__device__ void prepare_contact(const RCtx<R, W, SM>& x, const BatchView<R>& v, long long src, int k, int o) {
  const long long S = v.nc_total;
  const R* g = v.contact + src;
  v3<R> n = V<R>(g[C_NX * S], g[C_NY * S], g[C_NZ * S]);
  const v3<R> p = V<R>(g[C_PX * S], g[C_PY * S], g[C_PZ * S]);
  const int raw = v.contact_bodies[src];
  int b0 = body0_of(raw), b1 = body1_of(raw);
  if (b0 < 0) {
    mul_with(n, (R)-1);
    b0 = b1;
    b1 = -1;
  }
  x.set_pair(k, b0, b1, o);
  const v3<R> ty = contact_tangent(n);  // calculateContactBasis
  const v3<R> tz = contact_bitangent(n, ty);
  m3<R> C;
  C.m[0] = n.x; C.m[1] = n.y; C.m[2] = n.z;
  C.m[3] = ty.x; C.m[4] = ty.y; C.m[5] = ty.z;
  C.m[6] = tz.x; C.m[7] = tz.y; C.m[8] = tz.z;
  v3<R> rp0 = p;
  sub(rp0, V<R>((R)(x.P(0, b0)), (R)(x.P(1, b0)), (R)(x.P(2, b0))));
  v3<R> cv = local_velocity(x, b0, rp0, C);
  v3<R> rp1 = V<R>((R)0, (R)0, (R)0);
  if (b1 >= 0) {
    rp1 = p;
    sub(rp1, V<R>((R)(x.P(0, b1)), (R)(x.P(1, b1)), (R)(x.P(2, b1))));
    v3<R> cv1 = local_velocity(x, b1, rp1, C);
    sub(cv, cv1);
  }
  R* r = x.rec(k);
  st4(r, n.x, n.y, n.z, ty.x);
  st4(r + 4, ty.y, ty.z, tz.x, tz.y);
  st4(r + 8, tz.z, rp0.x, rp0.y, rp0.z);
  st4(r + 12, rp1.x, rp1.y, rp1.z, g[C_PEN * S]);
  st4(r + 16, cv.x, cv.y, cv.z, desired_dv(cv.x, frame_velocity(x, b0, b1, n), x.restitution(o)));
}

// SetAwake(true) (rigidbody.go:182-187) through matchAwakeState
// (contact.go:184-202), for the contact with pair bb, by the lanes of a group
// with `on`; `first` marks the one that writes.  Every lane of the warp calls
// it; true (for the whole warp) when a body woke.
template <class R, class W, bool SM>
__device__ __forceinline__ bool match_awake(const RCtx<R, W, SM>& x, int bb, bool on, bool first) {
  if (x.all_awake) return false;  // no body falls asleep in the resolver
  bool woke = false;
  int t = 0;
  if (on) {
    const int b0 = x.B0(bb), b1 = x.B1(bb);
    if (b1 >= 0) {
      const bool a0 = x.aw[b0] != 0, a1 = x.aw[b1] != 0;
      woke = a0 != a1;
      t = a0 ? b1 : b0;
    }
  }
  if (!__any_sync(0xffffffffu, woke)) return false;
  __syncwarp();
  if (woke && first) {
    x.aw[t] = 1;
    x.body(t)[BR_MOTION] = (R)(0.3 * 2.0);
  }
  __syncwarp();
  return true;
}

// CalculateDerivedData for a body that is asleep during adjustPositions
// (contact.go:380-382): renormalise, refresh the world inverse inertia.
template <class R, class W, bool SM>
__device__ __noinline__ void derive_asleep(RCtx<R, W, SM> x, const BatchView<R>& v, int bstart, int body) {
  q4<R> q{(R)x.P(3, body), (R)x.P(4, body), (R)x.P(5, body), (R)x.P(6, body)};
  q4<W> qw = cvtq<W>(q);
  qnormalize_island<R, W>(qw);
  q = cvtq<R>(qw);
  R rm[9];
  rotation_of(q, rm);
  m3<R> ib;
#pragma unroll
  for (int k = 0; k < 9; ++k) ib.m[k] = v.body[(long long)(B_IB0 + k) * v.nb_pad + bstart + body];
  m3<R> iw = world_inertia(rm, ib);
  R* b = x.body(body) + BR_IIT;
#pragma unroll
  for (int k = 0; k < 9; ++k) b[k] = iw.m[k];
  x.P(3, body) = (W)q.w; x.P(4, body) = (W)q.x; x.P(5, body) = (W)q.y; x.P(6, body) = (W)q.z;
}

// applyPositionChange, contact.go:285-386, of contact k by the first eight
// lanes (sl = 0..7) of a group with `on`; every lane of the warp calls both
// parts.  The four lanes 4i..4i+3 move body i: lane 4i + c (c < 3) forms
// component c of its inertia's vectors, of its moves and of its position, and
// (c < 4) its own component of the quaternion; the vectors meet by shuffles
// where a dot product or a matrix row needs them whole, the two bodies where
// the total does (summed in the reference's order), and every lane of a body
// decides the clamps and the renormalisation alike (the precision form's
// island, or Normalize in the float64 form).  A float64 warp instruction takes
// its scheduler's float64 unit 64 cycles whatever its active mask, so the
// number of them is what counts: about 110 where one lane per body's formulas
// took 160.  The operations on every value are the one-lane formula's, so the
// bits are the same.  Lane 4i + c returns component c of body i's linear and
// angular change.  position_load reads what it needs, as velocity_load does.
template <class R, class W> struct PositionIn {
  v3<R> n, rp;         // normal, the body's relative position
  R nc, np, nq;        // components c and the cross product's other two
  R rc, rp1, rq1;
  R i0, i1, i2, im;    // the body's inertia row c, inverse mass
  R penetration;
  W acc, at;           // quaternion component c, position component c
  int b;
};
template <class R, class W, bool SM>
__device__ __forceinline__ void position_load(const RCtx<R, W, SM>& x, PositionIn<R, W>& in, int k, int bb, bool on,
                                              int sl) {
  const R z = (R)0;
  const int i = (sl >> 2) & 1, c4 = sl & 3, c = c4 != 3 ? c4 : 0;
  const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;
  in.n = in.rp = V<R>(z, z, z);
  in.nc = in.np = in.nq = in.rc = in.rp1 = in.rq1 = in.i0 = in.i1 = in.i2 = in.im = in.penetration = z;
  in.b = -1;
  in.acc = in.at = (W)0;
  if (!on) return;
  const R* r = x.rec(k);
  const R* rel = r + (i == 0 ? CR_R0 : CR_R1);
  in.n = V<R>(r[0], r[1], r[2]);
  in.rp = V<R>(rel[0], rel[1], rel[2]);
  in.nc = r[CR_N + c]; in.np = r[CR_N + p]; in.nq = r[CR_N + q];
  in.rc = rel[c]; in.rp1 = rel[p]; in.rq1 = rel[q];
  in.penetration = r[CR_PEN];
  in.b = i == 0 ? x.B0(bb) : x.B1(bb);
  if (in.b >= 0) {
    const R* bd = x.body(in.b);
    in.i0 = bd[BR_IIT + c]; in.i1 = bd[BR_IIT + 3 + c]; in.i2 = bd[BR_IIT + 6 + c];
    in.im = bd[BR_INVM];
    in.acc = x.P(3 + c4, in.b);
    in.at = x.P(c, in.b);
  }
}
template <class R, class W, bool SM>
__device__ __forceinline__ void position_change(const RCtx<R, W, SM>& x, const BatchView<R>& v,
                                                const PositionIn<R, W>& in, int bstart, bool on, int sl, R& linc,
                                                R& angc) {
  const int i = (sl >> 2) & 1, c4 = sl & 3, c = c4 != 3 ? c4 : 0, src = sl & 4;
  const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;
  const R z = (R)0;
  auto all = [&](R a) {
    return V<R>(__shfl_sync(0xffffffffu, a, 0, 4), __shfl_sync(0xffffffffu, a, 1, 4),
                __shfl_sync(0xffffffffu, a, 2, 4));
  };
  const int b = in.b;
  const bool act = on && b >= 0;
  // angular inertia: dot(cross(iitWorld * cross(rp, n), rp), n)
  const v3<R> a = all(in.rp1 * in.nq - in.rq1 * in.np);
  const R wc = in.i0 * a.x + in.i1 * a.y + in.i2 * a.z;
  const R wp = __shfl_sync(0xffffffffu, wc, p, 4), wq = __shfl_sync(0xffffffffu, wc, q, 4);
  const v3<R> d = all(wp * in.rq1 - wq * in.rp1);
  const R angI = act ? dot(d, in.n) : z;
  const R linI = act ? in.im : z;
  const R angO = __shfl_xor_sync(0xffffffffu, angI, 4);
  const R linO = __shfl_xor_sync(0xffffffffu, linI, 4);
  const int bO = __shfl_xor_sync(0xffffffffu, b, 4);
  R share = z;
  if (act) {
    const int b0 = i == 0 ? b : bO, b1 = i == 0 ? bO : b;
    R total = z;
    if (b0 >= 0) total += (i == 0 ? linI : linO) + (i == 0 ? angI : angO);
    if (b1 >= 0) total += (i == 0 ? linO : linI) + (i == 0 ? angO : angI);
    // angI / total on the even lanes, linI / total on the odd ones
    share = ((c4 & 1) == 0 ? angI : linI) / total;
  }
  const R share_o = __shfl_xor_sync(0xffffffffu, share, 1);
  const R pc = in.rc + in.nc * -dot(in.rp, in.n);  // the projection's component c
  const v3<R> pp = all(pc * pc);
  linc = angc = z;
  W acc = in.acc;
  R qr = z;
  if (act) {
    const R sign = i != 0 ? (R)-1 : (R)1;
    R am = sign * in.penetration * ((c4 & 1) == 0 ? share : share_o);
    R lm = sign * in.penetration * ((c4 & 1) == 0 ? share_o : share);
    const R maxm = (R)0.2 * sqrt_<R>(pp.x + pp.y + pp.z);
    if (am < -maxm) {
      R tm = am + lm;
      am = -maxm;
      lm = tm - am;
    } else if (am > maxm) {
      R tm = am + lm;
      am = maxm;
      lm = tm - am;
    }
    if (am != (R)0) angc = wc * (am / angI);
    linc = in.nc * lm;
    // the quaternion, narrowed by its component lanes for the increment
    // (add_scaled_vector_island's first step)
    qr = cvt_fast<R>(acc);
  }
  // component c4 of (0, ang) * q (quaternion.go:45-53), each lane its own:
  //   w: 0 qw - ax qx - ay qy - az qz     x: 0 qx + ax qw + ay qz - az qy
  //   y: 0 qy + ay qw + az qx - ax qz     z: 0 qz + az qw + ax qy - ay qx
  const R q1 = __shfl_sync(0xffffffffu, qr, src + (c4 == 0 ? 1 : 0), 8);
  const R q2 = __shfl_sync(0xffffffffu, qr, src + (c4 == 1 ? 3 : (c4 == 2 ? 1 : 2)), 8);
  const R q3 = __shfl_sync(0xffffffffu, qr, src + (c4 == 1 ? 2 : (c4 == 3 ? 1 : 3)), 8);
  const R u1 = __shfl_sync(0xffffffffu, angc, c4 < 2 ? 0 : c4 - 1, 4);
  const R u2 = __shfl_sync(0xffffffffu, angc, c4 < 2 ? 1 : (c4 == 2 ? 2 : 0), 4);
  const R u3 = __shfl_sync(0xffffffffu, angc, c4 < 2 ? 2 : c4 - 2, 4);
  if (act) {
    // Position.AddScaled(normal, linearMove), and the quaternion increment
    if (c4 < 3) x.P(c, b) = in.at + cvt_fast<W>(linc);
    const R a1 = u1 * q1, a2 = u2 * q2, a3 = u3 * q3;
    R t = (R)0 * qr;
    t = c4 == 0 ? t - a1 : t + a1;
    t = c4 == 0 ? t - a2 : t + a2;
    t = t - a3;
    acc += cvt_fast<W>(t * (R)0.5);
  }
  // qnormalize_island on the four components
  const W sq = act ? acc * acc : (W)0;
  const W s0 = __shfl_sync(0xffffffffu, sq, src, 8), s1 = __shfl_sync(0xffffffffu, sq, src + 1, 8);
  const W s2 = __shfl_sync(0xffffffffu, sq, src + 2, 8), s3 = __shfl_sync(0xffffffffu, sq, src + 3, 8);
  bool asleep = false;
  if (act) {
    const W s = s0 + s1 + s2 + s3;
    const W e = s - (W)1;
    const W ae = fabs(e);
    if (sizeof(R) != sizeof(W) && ae < (W)4e-7) {
    } else if (sizeof(R) != sizeof(W) && ae < (W)0x1p-11) {
      acc *= (W)1 + e * ((W)-0.5 + e * ((W)0.375 + e * ((W)-0.3125 + e * (W)0.2734375)));
    } else {  // on the same sum
      acc = normalize_component<W>(s, acc, c4);
    }
    asleep = !x.all_awake && !x.aw[b];
    // an asleep body's CalculateDerivedData reads the stored (R-rounded) orientation
    x.P(3 + c4, b) = asleep ? (W)(R)acc : acc;
  }
  if (!x.all_awake && __any_sync(0xffffffffu, asleep)) {
    __syncwarp();
    if (asleep && c4 == 0) derive_asleep(x, v, bstart, b);
    __syncwarp();
  }
}

template <class R> __device__ __forceinline__ m3<R> skew(const v3<R>& v) {  // contact.go:612-616
  m3<R> m;
  m.m[0] = (R)0; m.m[3] = -v.z; m.m[6] = v.y;
  m.m[1] = v.z; m.m[4] = (R)0; m.m[7] = -v.x;
  m.m[2] = -v.y; m.m[5] = v.x; m.m[8] = (R)0;
  return m;
}

// The response matrix of calculateFrictionImpulse (contact.go:540-575): the
// contact-frame velocity change per unit impulse of both bodies, in R.
template <class R, class W, bool SM>
__device__ __forceinline__ m3<R> friction_response(const RCtx<R, W, SM>& x, int k, int b0, int b1, const m3<R>& C) {
  R inv_mass = x.body(b0)[BR_INVM];
  m3<R> itt = skew(x.rel(0, k));
  m3<R> dvw = mulm(itt, x.iit(b0));
  dvw = mulm(dvw, itt);
  mulm_with(dvw, (R)-1);
  if (b1 >= 0) {
    itt = skew(x.rel(1, k));
    m3<R> d2 = mulm(itt, x.iit(b1));
    d2 = mulm(d2, itt);
    mulm_with(d2, (R)-1);
#pragma unroll
    for (int q = 0; q < 9; ++q) dvw.m[q] += d2.m[q];
    inv_mass += x.body(b1)[BR_INVM];
  }
  m3<R> dv = transpose(C);
  dv = mulm(dv, dvw);
  dv = mulm(dv, C);
  dv.m[0] += inv_mass;
  dv.m[4] += inv_mass;
  dv.m[8] += inv_mass;
  return dv;
}

// What adjustVelocities needs of contact k and does not change: the matrices
// of its friction solve, K = Invert(response) in W (contact.go:577-580,
// matrix.go:125-153), kept in R for the solve, and the response's first row
// (R); and its frame velocity (CR_VFA, in the place of the penetration, which
// only adjustPositions uses).  They depend on the relative positions, the
// basis, the inverse masses, the bodies' world inverse inertia and awake
// flags, of which adjustVelocities changes only the last, so computing them
// once, lane-parallel, at the start of the phase gives exactly the values the
// reference recomputes at every iteration; the sequential chain then only
// forms K * (desired delta velocity, -vy, -vz).
template <class R, class W, bool SM> __device__ __forceinline__ void friction_prepare(const RCtx<R, W, SM>& x, int k) {
  const int bb = x.pair(k);
  const int b0 = x.B0(bb), b1 = x.B1(bb);
  const m3<R> C = x.basis(k);
  x.rec(k)[CR_VFA] = frame_velocity(x, b0, b1, V<R>(C.m[0], C.m[1], C.m[2]));
  if (x.friction(x.list_index(k)) == (R)0) return;  // calculateFrictionlessImpulse needs neither
  const m3<R> dv = friction_response(x, k, b0, b1, C);
  m3<W> dv_w;
#pragma unroll
  for (int q = 0; q < 9; ++q) dv_w.m[q] = (W)(dv.m[q]);
  const m3<W> K = invert(dv_w);
  R* o = x.kw + (long long)k * K_ROW;
  st4(o, (R)K.m[0], (R)K.m[1], (R)K.m[2], (R)K.m[3]);
  st4(o + 4, (R)K.m[4], (R)K.m[5], (R)K.m[6], (R)K.m[7]);
  st4(o + 8, (R)K.m[8], dv.m[0], dv.m[3], dv.m[6]);
}

// applyVelocityChange, contact.go:447-494, of contact k by the first eight
// lanes (sl = 0..7) of a group with `on`; every lane of the warp calls both
// parts.  Lane 4i + c (c < 3) forms component c of the friction solve's product
// (calculateFrictionImpulse, contact.go:533-606, from friction_prepare's
// matrices), of the impulse, and of body i's velocity and rotation changes,
// which it adds to the body and returns; the vectors in between meet by
// shuffles, and the friction cone is decided on every lane alike.  Every
// component is the one-lane formula's (mulv's row, cross's component,
// add_scaled), so the bits are the same; one lane forming all of them issued
// about twice the instructions.  velocity_load reads all of it, so that the
// caller's other loads and one latency cover it.
template <class R> struct VelocityIn {
  R k0, k1, k2, k9, k10, k11;  // K's row c, the response's first row
  R n, ty, tz;                 // the basis, row c
  R rp, rq;                    // the relative position's other components
  R i0, i1, i2, im, vel, rot;  // the body's inertia row, inverse mass, velocity and rotation c
  R cvy, cvz, ddv;
  int b, bb;
};
template <class R, class W, bool SM>
__device__ __forceinline__ void velocity_load(const RCtx<R, W, SM>& x, VelocityIn<R>& in, int k, int bb, bool on,
                                              int sl) {
  const R z = (R)0;
  const int i = (sl >> 2) & 1, c = (sl & 3) != 3 ? sl & 3 : 0;
  const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;
  in = VelocityIn<R>{z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, -1, bb};
  if (!on) return;
  const R* kr = x.krow(k);
  in.k0 = kr[c]; in.k1 = kr[3 + c]; in.k2 = kr[6 + c];
  in.k9 = kr[9]; in.k10 = kr[10]; in.k11 = kr[11];
  const R* r = x.rec(k);
  const quad<R> m = ld4(r + CR_CV);
  in.cvy = m.b; in.cvz = m.c; in.ddv = m.d;
  in.n = r[CR_N + c]; in.ty = r[CR_TY + c]; in.tz = r[CR_TZ + c];
  const R* rel = r + (i == 0 ? CR_R0 : CR_R1);
  in.rp = rel[p];
  in.rq = rel[q];
  in.b = i == 0 ? x.B0(bb) : x.B1(bb);
  if (in.b >= 0) {
    const R* bd = x.body(in.b);
    in.vel = bd[BR_VEL + c];
    in.rot = bd[BR_ROT + c];
    in.i0 = bd[BR_IIT + c]; in.i1 = bd[BR_IIT + 3 + c]; in.i2 = bd[BR_IIT + 6 + c];
    in.im = bd[BR_INVM];
  }
}
// err collects status bits.
template <class R, class W, bool LEARN, bool SM>
__device__ __forceinline__ void velocity_change(const RCtx<R, W, SM>& x, const BatchView<R>& v,
                                                const VelocityIn<R>& in, int k, bool on, int sl, R& vc, R& rc,
                                                uint32_t& err) {
  const int i = (sl >> 2) & 1;
  const bool comp = (sl & 3) != 3;
  const int c = comp ? sl & 3 : 0;
  const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;  // cross component c = a_p b_q - a_q b_p
  const R z = (R)0;
  const int o = SM ? (int)((unsigned)in.bb >> 16) : k;  // the list index
  R icc = z, fr = (R)0.9;
  bool frictionless = false;
  v3<R> ic = V<R>(z, z, z);
  if (on) {
    fr = x.friction(o);
    frictionless = fr == z;
    if (frictionless) {
      // calculateFrictionlessImpulse, contact.go:496-531 (rare: every lane)
      const int b0 = x.B0(in.bb);
      const R* r = x.rec(k);
      const v3<R> r0 = x.rel(0, k), n = V<R>(r[0], r[1], r[2]);
      v3<R> d = cross(r0, n);
      d = mulv(x.iit(b0), d);
      d = cross(d, r0);
      R dvel = dot(d, n);
      dvel += x.body(b0)[BR_INVM];
      if (x.B1(in.bb) < 0 && sl == 0) err |= ST_FRICTIONLESS_NIL;
      ic = V<R>(in.ddv / dvel, z, z);
    } else {
      // component c of K * (desired delta velocity, -vy, -vz) (mulv's row c)
      icc = in.k0 * in.ddv + in.k1 * -in.cvy + in.k2 * -in.cvz;
    }
  }
  {
    const R i0 = __shfl_sync(0xffffffffu, icc, 0, 4), i1 = __shfl_sync(0xffffffffu, icc, 1, 4);
    const R i2 = __shfl_sync(0xffffffffu, icc, 2, 4);
    // the dynamic friction of contact.go:586-604, its two quotients by the
    // planar length on two lanes
    R planar = z;
    bool slides = false;
    if (on && !frictionless) {
      ic = V<R>(i0, i1, i2);
      planar = sqrt_<R>(ic.y * ic.y + ic.z * ic.z);
      slides = planar > ic.x * fr;
    }
    if (__any_sync(0xffffffffu, slides)) {
      R part = z;
      if (slides) part = (c == 2 ? ic.z : ic.y) / planar;
      const R py = __shfl_sync(0xffffffffu, part, 1, 4), pz = __shfl_sync(0xffffffffu, part, 2, 4);
      if (slides) {
        ic.y = py;
        ic.z = pz;
        ic.x = in.k9 + in.k10 * fr * ic.y + in.k11 * fr * ic.z;
        ic.x = in.ddv / ic.x;
        ic.y *= fr * ic.x;
        ic.z *= fr * ic.x;
      }
    }
  }
  if (LEARN && on && v.mode == 1 && sl == 0) {  // harvest: total impulse applied at this contact
    x.J(0, o) += ic.x;
    x.J(1, o) += ic.y;
    x.J(2, o) += ic.z;
  }
  // component c of the impulse contactToWorld * ic (mulv's row c)
  R impc = z;
  if (on) impc = in.n * ic.x + in.ty * ic.y + in.tz * ic.z;
  const R ip = __shfl_sync(0xffffffffu, impc, p, 4), iq = __shfl_sync(0xffffffffu, impc, q, 4);
  const bool act = on && in.b >= 0;
  // component c of cross(r0, imp) (body 0) or cross(imp, r1) (body 1)
  R crc = z;
  if (act) {
    const R m1 = in.rp * iq, m2 = in.rq * ip;
    crc = i == 0 ? m1 - m2 : m2 - m1;
  }
  const R cx = __shfl_sync(0xffffffffu, crc, 0, 4), cy = __shfl_sync(0xffffffffu, crc, 1, 4);
  const R cz = __shfl_sync(0xffffffffu, crc, 2, 4);
  vc = rc = z;
  if (act) {
    // rc = iitWorld * cross (mulv's row c); vc = 0 + imp * (+-inverse mass)
    rc = in.i0 * cx + in.i1 * cy + in.i2 * cz;
    vc += impc * (i == 0 ? in.im : -in.im);
    if (comp && sl < 8) {
      R* bd = x.body(in.b);
      bd[BR_VEL + c] = in.vel + vc;
      bd[BR_ROT + c] = in.rot + rc;
    }
  }
}

// Whether contact bodies (kb0, kb1) are the resolved bodies d0, d1 (d1 < 0:
// none): x, y the resolved body that contact body 0, 1 is, else -1.  A contact
// body is at most one of the two, so a contact takes at most two changes:
// body 0's first, then body 1's, which is the order of the reference's (b, d)
// loops (contact.go:254-280, 412-440).
__device__ __forceinline__ int2 touching(int kb0, int kb1, int d0, int d1) {
  int2 e;
  e.x = kb0 == d0 ? 0 : (d1 >= 0 && kb0 == d1 ? 1 : -1);
  e.y = kb1 < 0 ? -1 : (kb1 == d0 ? 0 : (d1 >= 0 && kb1 == d1 ? 1 : -1));
  return e;
}

// The update of a contact after resolving a contact between bodies d0, d1:
// its penetration (VEL false, contact.go:254-280) or contact velocity and
// desired delta velocity (VEL true, contact.go:412-440).  update_load reads
// what it needs of contact k with pair bb (where `valid`), which the change of the resolved
// contact does not touch, so the caller loads ahead of computing that change;
// update_apply takes the change, of which lanes 4d + c of the group of L lanes
// hold component c of resolved body d's, and returns the value the argmax
// reads (penetration or desired delta velocity).  A contact touching neither
// body is left alone.  Every lane of the warp calls both.
// Most contacts touch one of the two bodies: one pass over the formula with
// the side selected; the contacts between the two take a second.
template <class R> struct Touched {
  int k, bb;
  int2 e;
  bool valid;
  quad<R> q0, q1, q2, q3, m;  // the record: basis, relative positions, penetration or frame velocity; cv, ddv
};
template <bool VEL, class R, class W, bool SM>
__device__ __forceinline__ void update_load(const RCtx<R, W, SM>& x, Touched<R>& t, int k, int bb, bool valid, int d0,
                                            int d1) {
  t.k = k;
  t.valid = valid;
  t.e = make_int2(-1, -1);
  t.bb = bb;
  t.m = t.q3 = quad<R>{(R)0, (R)0, (R)0, (R)0};
  if (!valid) return;
  t.e = touching(x.B0(t.bb), x.B1(t.bb), d0, d1);
  const R* r = x.rec(k);
  if (VEL) t.m = ld4(r + CR_CV);
  t.q3 = ld4(r + 12);
  if (t.e.x < 0 && t.e.y < 0) return;
  t.q0 = ld4(r);
  t.q2 = ld4(r + 8);
  if (VEL) t.q1 = ld4(r + 4);
}
template <bool VEL, class R, class W, bool SM>
__device__ __forceinline__ R update_apply(const RCtx<R, W, SM>& x, Touched<R>& t, R lin, R ang, int L, bool woke) {
  const bool hit = t.e.x >= 0 || t.e.y >= 0, both = t.e.x >= 0 && t.e.y >= 0;
  R value = VEL ? t.m.d : t.q3.d;
  if (!__any_sync(0xffffffffu, hit)) return value;
  const m3<R> C{{t.q0.a, t.q0.b, t.q0.c, t.q0.d, t.q1.a, t.q1.b, t.q1.c, t.q1.d, t.q2.a}};
  const v3<R> n = V<R>(t.q0.a, t.q0.b, t.q0.c);
  const bool first0 = t.e.x >= 0;  // the first change is contact body 0's
  // the change of resolved body d at relative position r, in the contact's terms
  auto from = [&](int d) { return V<R>(__shfl_sync(0xffffffffu, lin, d, L), __shfl_sync(0xffffffffu, lin, d + 1, L),
                                       __shfl_sync(0xffffffffu, lin, d + 2, L)); };
  auto turn = [&](int d) { return V<R>(__shfl_sync(0xffffffffu, ang, d, L), __shfl_sync(0xffffffffu, ang, d + 1, L),
                                       __shfl_sync(0xffffffffu, ang, d + 2, L)); };
  auto moved = [&](const v3<R>& dl, const v3<R>& da, const v3<R>& r) {
    v3<R> dv = cross(da, r);
    add(dv, dl);
    if constexpr (VEL) return mulv_t(C, dv);
    else return V<R>(dot(dv, n), (R)0, (R)0);
  };
  const int s1 = 4 * ((t.e.x >= 0 ? t.e.x : t.e.y) > 0);
  const v3<R> dl = from(s1), da = turn(s1);
  const v3<R> r1 = V<R>(t.q3.a, t.q3.b, t.q3.c);
  const v3<R> rf = first0 ? V<R>(t.q2.b, t.q2.c, t.q2.d) : r1;
  auto apply = [&](const v3<R>& a, bool plus) {
    if constexpr (VEL) {
      t.m.a = plus ? t.m.a + a.x : t.m.a - a.x;
      t.m.b = plus ? t.m.b + a.y : t.m.b - a.y;
      t.m.c = plus ? t.m.c + a.z : t.m.c - a.z;
    } else {
      value = plus ? value - a.x : value + a.x;
    }
  };
  if (__any_sync(0xffffffffu, both)) {
    // both terms at once (independent until they are added, in order)
    const int s2 = 4 * (t.e.y > 0);
    const v3<R> dl2 = from(s2), da2 = turn(s2);
    if (hit) {
      const v3<R> a = moved(dl, da, rf), a2 = moved(dl2, da2, r1);
      apply(a, first0);
      if (both) apply(a2, false);
    }
  } else if (hit) {
    apply(moved(dl, da, rf), first0);
  }
  if (hit) {
    R* r = x.rec(t.k);
    if constexpr (VEL) {
      R vfa = t.q3.d;
      if (woke) r[CR_VFA] = vfa = frame_velocity(x, x.B0(t.bb), x.B1(t.bb), n);
      value = desired_dv(t.m.a, vfa, x.restitution(x.list_index(t.k)));
      st4(r + CR_CV, t.m.a, t.m.b, t.m.c, value);
    } else {
      r[CR_PEN] = value;
    }
  }
  return value;
}

// The same update (update_load and update_apply) of contact k with pair bb by
// four lanes, lane c (of 4) the component c of the change and of the contact
// velocity: for the float64 form, whose update is bound by the number of
// float64 instructions, where a group has lanes to spare (14 or, with both
// bodies touched, 24 of them for L / 4 contacts, against 34 or 64 for L).
template <bool VEL, class R, class W, bool SM>
__device__ __forceinline__ R update_spread(const RCtx<R, W, SM>& x, int k, int bb, bool valid, int d0, int d1, R lin,
                                           R ang, int L, bool woke) {
  const R z = (R)0;
  const int c4 = threadIdx.x & 3, c = c4 != 3 ? c4 : 0;
  const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;
  const int2 e = valid ? touching(x.B0(bb), x.B1(bb), d0, d1) : make_int2(-1, -1);
  const bool both = e.x >= 0 && e.y >= 0, first0 = e.x >= 0;
  R r0p = z, r0q = z, r1p = z, r1q = z, col0 = z, col1 = z, col2 = z, m = z, vfa = z;
  if (valid) {
    const R* r = x.rec(k);
    r0p = r[CR_R0 + p]; r0q = r[CR_R0 + q];
    r1p = r[CR_R1 + p]; r1q = r[CR_R1 + q];
    const R* col = r + CR_N + (VEL ? 3 * c : 0);
    col0 = col[0]; col1 = col[1]; col2 = col[2];
    m = VEL ? r[CR_CV + c] : r[CR_PEN];
    if (VEL) vfa = r[CR_VFA];
  }
  auto term = [&](int d, R rp, R rq) {
    const R ap = __shfl_sync(0xffffffffu, ang, d + p, L), aq = __shfl_sync(0xffffffffu, ang, d + q, L);
    const R dv = ap * rq - aq * rp + __shfl_sync(0xffffffffu, lin, d + c, L);
    const R x0 = __shfl_sync(0xffffffffu, dv, 0, 4), x1 = __shfl_sync(0xffffffffu, dv, 1, 4);
    const R x2 = __shfl_sync(0xffffffffu, dv, 2, 4);
    return x0 * col0 + x1 * col1 + x2 * col2;
  };
  const R t = term(4 * ((e.x >= 0 ? e.x : e.y) > 0), first0 ? r0p : r1p, first0 ? r0q : r1q);
  // a velocity takes body 0's term and gives body 1's back, a penetration the other way round
  m = first0 == VEL ? m + t : m - t;
  if (__any_sync(0xffffffffu, both)) {
    const R t2 = term(4 * (e.y > 0), r1p, r1q);
    if (both) m = VEL ? m - t2 : m + t2;
  }
  R value = m;
  if (valid) {
    R* r = x.rec(k);
    if (VEL) {
      if (woke) vfa = frame_velocity(x, x.B0(bb), x.B1(bb), V<R>(r[0], r[1], r[2]));
      if (c4 < 3) r[CR_CV + c] = m;
      value = desired_dv(m, vfa, x.restitution(SM ? (int)((unsigned)bb >> 16) : k));
      if (c4 == 0) {
        if (woke) r[CR_VFA] = vfa;
        r[CR_DDV] = value;
      }
    } else if (c4 == 0) {
      r[CR_PEN] = m;
    }
  }
  return value;
}

// A world's bodies from the batch rows into the records of x, by the `step`
// lanes of a group (lane index `first`).
// Returns whether this lane's bodies are all awake.  With `lab`, all but the
// bodies of label `keep`.
template <class R, class W, bool SM>
__device__ __forceinline__ bool load_bodies(const RCtx<R, W, SM>& x, const BatchView<R>& v, long long bstart, int n,
                                            int first, int step, const uint8_t* lab = nullptr, int keep = -1) {
  const long long S = v.nb_pad;
  bool awake = true;
#pragma unroll 1
  for (int i = first; i < n; i += step) {
    if (lab && lab[i] == keep) continue;
    const R* g = v.body + bstart + i;
    auto F = [&](int r) { return g[(long long)r * S]; };
    x.P(0, i) = (W)F(B_PX); x.P(1, i) = (W)F(B_PY); x.P(2, i) = (W)F(B_PZ);
    x.P(3, i) = (W)F(B_QW); x.P(4, i) = (W)F(B_QX); x.P(5, i) = (W)F(B_QY); x.P(6, i) = (W)F(B_QZ);
    R* b = x.body(i);
    st4(b, F(B_VX), F(B_VY), F(B_VZ), F(B_RX));
    st4(b + 4, F(B_RY), F(B_RZ), F(B_IW0), F(B_IW1));
    st4(b + 8, F(B_IW2), F(B_IW3), F(B_IW4), F(B_IW5));
    st4(b + 12, F(B_IW6), F(B_IW7), F(B_IW8), F(B_INVM));
    st4(b + 16, F(B_LX) * x.dt, F(B_LY) * x.dt, F(B_LZ) * x.dt, F(B_MOTION));
    x.aw[i] = v.awake[bstart + i];
    awake = awake && x.aw[i] != 0;
  }
  return awake;
}
// ... and back
template <class R, class W, bool SM>
__device__ __forceinline__ void store_bodies(const RCtx<R, W, SM>& x, const BatchView<R>& v, long long bstart, int n,
                                             int first, int step) {
  const long long S = v.nb_pad;
#pragma unroll 1
  for (int i = first; i < n; i += step) {
    R* g = v.body + bstart + i;
#pragma unroll
    for (int r = 0; r < 7; ++r) g[(long long)(B_PX + r) * S] = (R)x.P(r, i);
    const R* b = x.body(i);
    const quad<R> q0 = ld4(b), q1 = ld4(b + 4), q2 = ld4(b + 8), q3 = ld4(b + 12);
    g[B_VX * S] = q0.a; g[B_VY * S] = q0.b; g[B_VZ * S] = q0.c;
    g[B_RX * S] = q0.d; g[B_RY * S] = q1.a; g[B_RZ * S] = q1.b;
    g[B_IW0 * S] = q1.c; g[B_IW1 * S] = q1.d; g[B_IW2 * S] = q2.a; g[B_IW3 * S] = q2.b; g[B_IW4 * S] = q2.c;
    g[B_IW5 * S] = q2.d; g[B_IW6 * S] = q3.a; g[B_IW7 * S] = q3.b; g[B_IW8 * S] = q3.c;
    g[B_MOTION * S] = b[BR_MOTION];
    v.awake[bstart + i] = x.aw[i];
  }
}
// ResolveContacts' effect on the caller's Contact values that the phases do
// not produce: the swapped bodies and normal of calculateInternals.
template <class R, class W, bool SM>
__device__ __forceinline__ void write_back_contact(const RCtx<R, W, SM>& x, const BatchView<R>& v, long long cst,
                                                   int k) {
  const long long S = v.nc_total;
  const R* r = x.rec(k);
  const long long o = cst + x.list_index(k);
  v.contact[C_NX * S + o] = r[0];
  v.contact[C_NY * S + o] = r[1];
  v.contact[C_NZ * S + o] = r[2];
  v.contact_bodies[o] = pack_bodies(x.B0(x.pair(k)), x.B1(x.pair(k)));
}

// ---------------------------------------------------------------- world slots
// Shared memory of one world: body and contact records, packed bodies, awake
// flags, the island table.  The learned paths keep their per-body scratch and
// the impulse rows in global memory, so they use the same slot (and reach the
// same occupancy) as the plain resolver.
// The float64 form gathers the contacts touching the two resolved bodies
// before updating them (resolve_phase); room for one gather.
constexpr int kTouchList = 64;
template <class R> __host__ __device__ constexpr bool gathers_updates() { return sizeof(R) == 8; }

template <class R, class W> __host__ __device__ inline size_t rs_slot_bytes(int nbs, int cs) {
  size_t b = (size_t)7 * nbs * sizeof(W);
  b += (size_t)BREC * nbs * sizeof(R);
  b += (size_t)CREC * cs * sizeof(R);
  b += (size_t)cs * sizeof(int);
  b += (size_t)((nbs + 15) & ~15);
  if (gathers_updates<R>()) b += (size_t)kTouchList * sizeof(int);
  b += (size_t)(nbs + 4) * sizeof(uint16_t);      // first record of each island
  b += (size_t)nbs * (sizeof(uint16_t) + 1);      // build_islands: cursors, labels
  return (b + 15) & ~(size_t)15;
}

template <class R, class W> struct Slot {
  RCtx<R, W, true> x;
  int* ml;          // [kTouchList] contacts touching the two bodies just resolved (float64 form)
  R* cr_s;
  int* cb_s;
  uint16_t* ist;    // [nbs + 1] first record of each island
  uint16_t* cur;    // [nbs] next free record of the island with smallest body i
  uint8_t* lab;     // [nbs] smallest body of the body's island
};

template <class R, class W>
__device__ __forceinline__ Slot<R, W> make_slot(unsigned char* base, int nbs, int cs, R dt) {
  Slot<R, W> s;
  RCtx<R, W, true>& x = s.x;
  x.nbs = nbs;
  x.dt = dt;
  x.bw = reinterpret_cast<W*>(base);
  x.br = reinterpret_cast<R*>(x.bw + 7 * nbs);
  s.cr_s = x.br + BREC * nbs;
  s.cb_s = reinterpret_cast<int*>(s.cr_s + (size_t)CREC * cs);
  x.aw = reinterpret_cast<uint8_t*>(s.cb_s + cs);
  s.ml = reinterpret_cast<int*>(x.aw + ((nbs + 15) & ~15));
  s.ist = reinterpret_cast<uint16_t*>(s.ml + (gathers_updates<R>() ? kTouchList : 0));
  s.cur = s.ist + nbs + 4;
  s.lab = reinterpret_cast<uint8_t*>(s.cur + nbs);
  x.delta = x.jw = nullptr;
  x.wi = nullptr;
  x.wst = x.jst = 0;
  return s;
}

template <class R, class W>
__device__ __forceinline__ void bind_contacts(Slot<R, W>& s, const BatchView<R>& v, int C, int cs, long long cst) {
  RCtx<R, W, true>& x = s.x;
  if (C <= cs) {
    x.cr = s.cr_s;
    x.cb = s.cb_s;
  } else {
    x.cr = v.work + cst * CREC;
    x.cb = v.work_bodies + cst;
  }
  x.gmat = v.uniform_material ? nullptr : v.contact + (long long)C_FRIC * v.nc_total + cst;
  x.gst = (long long)(C_REST - C_FRIC) * v.nc_total;
  x.kw = v.kmat + cst * K_ROW;
}

// the learned paths' global scratch of the world whose bodies start at bstart
template <class R, class W>
__device__ __forceinline__ void bind_ws(RCtx<R, W, true>& x, const BatchView<R>& v, long long bstart, long long cst) {
  x.wst = v.nb_pad;
  x.delta = v.ws_rows + bstart;
  x.wi = v.ws_int + bstart;
  x.jw = v.ws_imp + cst;
  x.jst = v.nc_total;
}

// The 18 features of a contact at the start of adjustVelocities, all in the
// contact basis where they are vectors: the number of contacts between body 0
// and other bodies, a half-space flag, the contact velocity (3), penetration, desired delta
// velocity, the response matrix (6: nn, tt, ss, nt, ns, ts), the impulse that
// would resolve the contact alone along its normal (desired delta velocity /
// response nn), and per body the contacts touching it and their summed
// positive desired delta velocities (2 + 2).
template <class R, class W, bool SM> __device__ void contact_features(const RCtx<R, W, SM>& x, int k, float* f) {
  const int bb = x.pair(k);
  const int b0 = x.B0(bb), b1 = x.B1(bb);
  const R* r = x.rec(k);
  const v3<R> cv = V<R>(r[CR_CV], r[CR_CV + 1], r[CR_CV + 2]);
  const R ddv = r[CR_DDV];
  f[0] = (float)x.WI(WS_NBB, b0);
  f[1] = b1 < 0 ? 1.f : 0.f;
  f[2] = (float)cv.x; f[3] = (float)cv.y; f[4] = (float)cv.z;
  f[5] = (float)r[CR_PEN];
  f[6] = (float)ddv;
  const m3<R> K = friction_response(x, k, b0, b1, x.basis(k));
  f[7] = (float)K.m[0]; f[8] = (float)K.m[4]; f[9] = (float)K.m[8];
  f[10] = (float)K.m[3]; f[11] = (float)K.m[6]; f[12] = (float)K.m[7];
  f[13] = K.m[0] > (R)0 ? (float)(ddv / K.m[0]) : 0.f;
  f[14] = (float)x.WI(WS_DEG, b0);
  f[15] = b1 >= 0 ? (float)x.WI(WS_DEG, b1) : 0.f;
  f[16] = (float)(unsigned)x.WI(WS_LOAD, b0) * (1.f / kLoadScale);
  f[17] = b1 >= 0 ? (float)(unsigned)x.WI(WS_LOAD, b1) * (1.f / kLoadScale) : 0.f;
}

template <int G> __device__ __forceinline__ int group_sum(int v) {
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// The warm start of one world, planned by k_warm_features for its bodies
// whose contacts are all with the half-space ("grounded" bodies), at the state
// adjustVelocities starts from (adjustPositions changes no velocity).  A
// grounded body's contacts depend on that body's velocity alone, so each one
// is warm-started independently:
//  1. Predictions of its contacts are projected: normal impulse >= 0,
//     friction inside the cone |J_t| <= friction * J_n.  Contacts of other
//     bodies get none.
//  2. The body's velocity and rotation change of all those impulses,
//     accumulated in contact order (deterministic); the half-space contacts
//     of a body are one run of the contact list when the narrowphase made
//     them, else the whole list is scanned.
//  3. A line search picks the body's scale s in [0, 1]: none of its contacts
//     may be pushed past what resolving it would do (normal velocity at most
//     velocity + max(desired delta, 0) + the velocity epsilon), and no
//     tangential speed may grow beyond max(current, epsilon).  The resolver
//     only removes approaching velocity, so it could not undo an overshoot.
//  4. The plan: the body's change times s in the delta rows, each contact's
//     velocity change times its body's s in the impulse rows (zeros where the
//     warm start does nothing); warm_start_apply adds them.
// The 32 lanes of a warp plan one world.  Adds this lane's warm-started bodies
// and the sum of their scales to *nw and *ssum.
template <class R, class W, bool SM>
__device__ void warm_start_plan(const RCtx<R, W, SM>& x, int n, int C, int lane, int* nw, float* ssum) {
  const R z = (R)0, eps = (R)0.01;
  for (int k = lane; k < C; k += 32) {
    const int bb = x.pair(k);
    v3<R> J = V<R>(x.J(0, k), x.J(1, k), x.J(2, k));
    if (x.B1(bb) >= 0 || x.WI(WS_NBB, x.B0(bb)) != 0 || !(J.x > z)) J = V<R>(z, z, z);  // also NaN
    const R lim = x.friction(k) * J.x;
    const R planar = sqrt_<R>(J.y * J.y + J.z * J.z);
    if (planar > lim) {
      const R f = planar > z ? lim / planar : z;
      J.y *= f;
      J.z *= f;
    }
    if (!(planar == planar)) J = V<R>(z, z, z);
    x.J(0, k) = J.x;
    x.J(1, k) = J.y;
    x.J(2, k) = J.z;
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    v3<R> dvel = V<R>(z, z, z), drot = V<R>(z, z, z);
    const int deg = x.WI(WS_DEG, i);
    if (x.WI(WS_NBB, i) == 0 && deg > 0) {
      const m3<R> I = x.iit(i);
      const R invm = x.body(i)[BR_INVM];
      const int first = x.WI(WS_FIRST, i), last = x.WI(WS_LAST, i);
      const bool run = last - first + 1 == deg;
      for (int k = run ? first : 0; k <= (run ? last : C - 1); ++k) {
        if (!run && x.B0(x.pair(k)) != i) continue;
        const v3<R> J = V<R>(x.J(0, k), x.J(1, k), x.J(2, k));
        if (J.x == z) continue;
        const v3<R> imp = mulv(x.basis(k), J);
        add(drot, mulv(I, cross(x.rel(0, k), imp)));
        add_scaled(dvel, imp, invm);
      }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      x.Delta(r, i) = (&dvel.x)[r];
      x.Delta(3 + r, i) = (&drot.x)[r];
    }
    x.WI(WS_SCALE, i) = __float_as_int(1.f);
  }
  __syncwarp();
  // contact velocity change at s = 1 (into the impulse rows) and the largest
  // scale each contact allows; a body's scale is the smallest of its contacts'
  for (int k = lane; k < C; k += 32) {
    const int bb = x.pair(k);
    const int b0 = x.B0(bb);
    if (x.B1(bb) >= 0 || x.WI(WS_NBB, b0) != 0) {
      x.J(0, k) = z;
      x.J(1, k) = z;
      x.J(2, k) = z;
      continue;
    }
    const m3<R> Ck = x.basis(k);
    const v3<R> dr = V<R>(x.Delta(3, b0), x.Delta(4, b0), x.Delta(5, b0));
    const v3<R> dl = V<R>(x.Delta(0, b0), x.Delta(1, b0), x.Delta(2, b0));
    v3<R> dv = cross(dr, x.rel(0, k));
    add(dv, dl);
    const v3<R> dcv = mulv_t(Ck, dv);
    x.J(0, k) = dcv.x;
    x.J(1, k) = dcv.y;
    x.J(2, k) = dcv.z;
    R sk = (R)1;
    const R ddv = x.rec(k)[CR_DDV];
    if (dcv.x > z) {
      const R q = ((ddv > z ? ddv : z) + eps) / dcv.x;
      if (q < sk) sk = q;
    }
    const R ty = x.rec(k)[CR_CV + 1], tz = x.rec(k)[CR_CV + 2];
    const R a = dcv.y * dcv.y + dcv.z * dcv.z;
    if (a > z) {
      const R t2 = ty * ty + tz * tz;
      const R bound2 = t2 > eps * eps ? t2 : eps * eps;
      const R hb = ty * dcv.y + tz * dcv.z;
      // largest s with |t + s dt|^2 <= bound^2: root of a s^2 + 2 hb s + (t2 - bound2)
      const R disc = hb * hb - a * (t2 - bound2);
      const R q = (-hb + sqrt_<R>(disc > z ? disc : z)) / a;
      if (q < sk) sk = q;
    }
    float sf = (float)sk;
    if (!(sf >= 0.f)) sf = 0.f;  // NaN or negative: no warm start
    if (sf < 1.f) atomicMin(&x.WI(WS_SCALE, b0), __float_as_int(sf));  // non-negative floats order as ints
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    bool moved = false;
#pragma unroll
    for (int r = 0; r < 6; ++r) moved |= x.Delta(r, i) != z;
    const R sb = (R)__int_as_float(x.WI(WS_SCALE, i));
    if (moved) {
      ++*nw;
      *ssum += (float)sb;
    }
#pragma unroll
    for (int r = 0; r < 6; ++r) x.Delta(r, i) = moved && sb != z ? sb * x.Delta(r, i) : z;
  }
  __syncwarp();
  for (int k = lane; k < C; k += 32) {
    const int bb = x.pair(k);
    const int b0 = x.B0(bb);
    if (x.B1(bb) >= 0 || x.WI(WS_NBB, b0) != 0) continue;
    const R sb = (R)__int_as_float(x.WI(WS_SCALE, b0));
#pragma unroll
    for (int c = 0; c < 3; ++c) x.J(c, k) = x.J(c, k) != z ? sb * x.J(c, k) : z;
  }
}

// The planned warm start, applied at the start of adjustVelocities: each body
// takes its scaled change, each contact its scaled velocity change and a
// recomputed desired delta velocity, as adjustVelocities does after an
// impulse (contact.go:416-445).  A body or contact with nothing planned keeps
// its values bit for bit.  Every lane of the warp calls it (it synchronises
// the warp); `on` selects the groups warm-starting.  Returns the bodies this
// lane moved.
template <class R, class W, int G, bool SM>
__device__ int warm_start_apply(const RCtx<R, W, SM>& x, int n, int C, int gl, bool on) {
  const R z = (R)0;
  int moved = 0;
  for (int i = gl; on && i < n; i += G) {
    bool any = false;
#pragma unroll
    for (int r = 0; r < 6; ++r) any |= x.Delta(r, i) != z;
    if (!any) continue;
    ++moved;
#pragma unroll
    for (int r = 0; r < 6; ++r) x.body(i)[BR_VEL + r] += x.Delta(r, i);
  }
  __syncwarp();
  for (int k = gl; on && k < C; k += G) {
    const int o = x.list_index(k);
    const v3<R> dcv = V<R>(x.J(0, o), x.J(1, o), x.J(2, o));
    if (dcv.x == z && dcv.y == z && dcv.z == z) continue;
    R* r = x.rec(k);
    v3<R> cv = V<R>(r[CR_CV], r[CR_CV + 1], r[CR_CV + 2]);
    add(cv, dcv);
    st4(r + CR_CV, cv.x, cv.y, cv.z, desired_dv(cv.x, r[CR_VFA], x.restitution(o)));
  }
  return moved;
}

// ---------------------------------------------------------------- islands
// The connected components of a world's contacts over its bodies ("islands";
// the half-space is no body).  Resolving a contact reads and changes its two
// bodies and the contacts touching them, so the reference's sequence of
// resolved contacts, restricted to one island, depends on that island alone:
// it is the island's own first-maximum sequence.  As long as the world's
// iterations stay within its budget, the islands can therefore be solved side
// by side, each by its own group of lanes, and every body, contact and count
// comes out the same bit for bit.  Only when the budget runs out does the
// order between the islands matter (which of them got the last iterations);
// such a world is put back and solved as one list (resolve_phase, LIST false).
//
// Why: a settled world of 32 bodies has about 28 islands (spheres and cubes
// resting alone, a few small heaps) and 130 iterations a frame, of which the
// longest island has 25, and an iteration keeps 9 of 32 lanes busy.  Solved
// one after the other, the iterations were 85 % of a frame.

// Lanes per island.  8: a resting cube has at most 8 contacts, and the eight
// lanes are what the spread changes above use; worlds with fewer lanes are one
// list.
constexpr int kIslandLanes = 8;

// Finds the islands of a world's C contacts (contact_bodies at list positions
// cst..) and their places: island i's records are [ist[i], ist[i + 1]), the
// ones with many contacts first; lab[b] is the smallest body of b's island,
// cur[lab] the first record of that island (the caller advances it).  Returns
// the number of islands.  sc: scratch of 3 * 64 ints.  The G lanes of a group
// (gl) list one world of n <= 64 bodies; every lane of the warp calls it.
template <int G, class R>
__device__ __forceinline__ int build_islands(const BatchView<R>& v, long long cst, int n, int nbs, int C, int gl,
                                             int* sc, uint16_t* ist, uint16_t* cur, uint8_t* lab8) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const unsigned gmask = G == 32 ? FULL : (((1u << G) - 1u) << (lane - gl));
  int* lab = sc;        // smallest body of the island
  int* cnt = sc + 64;   // at that body: the island's contacts
  int* ord = sc + 128;  // islands (their smallest bodies) in order
  const int* pairs = v.contact_bodies + cst;
#pragma unroll 1
  for (int i = gl; i < n; i += G) {
    lab[i] = i;
    cnt[i] = 0;
  }
  __syncwarp();
  // Labels only fall, to a body of the same island; done when every contact
  // joins equal labels.  Each round also follows the labels' labels, so a
  // chain of bodies takes few rounds.
  for (bool more = true; __any_sync(FULL, more);) {
    more = false;
#pragma unroll 1
    for (int k = gl; k < C; k += G) {
      const int bb = pairs[k];
      const int b0 = body0_of(bb), b1 = body1_of(bb);
      if (b0 < 0 || b1 < 0) continue;
      const int l0 = lab[b0], l1 = lab[b1];
      if (l0 == l1) continue;
      const int lo = min(l0, l1);
      atomicMin(&lab[max(l0, l1)], lo);
      atomicMin(&lab[b0], lo);
      atomicMin(&lab[b1], lo);
      more = true;
    }
    __syncwarp();
#pragma unroll 1
    for (int i = gl; i < n; i += G) atomicMin(&lab[i], lab[lab[i]]);
    __syncwarp();
  }
#pragma unroll 1
  for (int k = gl; k < C; k += G) {
    const int bb = pairs[k];
    const int b0 = body0_of(bb);
    atomicAdd(&cnt[lab[b0 < 0 ? body1_of(bb) : b0]], 1);
  }
#pragma unroll 1
  for (int i = gl; i < n; i += G) lab8[i] = (uint8_t)lab[i];
  __syncwarp();
  int ni = 0;
#pragma unroll 1
  for (int c = 0; c < 5; ++c)
#pragma unroll 1
    for (int base = 0; base < nbs; base += G) {
      const int i = base + gl;
      const int m = i < n ? cnt[i] : 0;
      const bool hit = m > 0 && c == (m >= 24 ? 0 : m >= 12 ? 1 : m >= 6 ? 2 : m >= 3 ? 3 : 4);
      const unsigned bal = __ballot_sync(FULL, hit) & gmask;
      if (hit) ord[ni + __popc(bal & below)] = i;
      ni += __popc(bal);
    }
  __syncwarp();
  int carry = 0;
#pragma unroll 1
  for (int base = 0; base < nbs; base += G) {
    const int p = base + gl;
    const int r = p < ni ? ord[p] : 0;
    const int len = p < ni ? cnt[r] : 0;
    int sum = len;
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
      const int y = __shfl_up_sync(FULL, sum, d, G);
      if (gl >= d) sum += y;
    }
    if (p < ni) {
      ist[p] = (uint16_t)(carry + sum - len);
      cur[r] = (uint16_t)(carry + sum - len);
    }
    carry += __shfl_sync(FULL, sum, G - 1, G);
  }
  if (gl == 0) ist[ni] = (uint16_t)C;
  __syncwarp();
  return ni;
}

// The record of contact k of a world in island order: its island's next free
// one.  Called with k ascending over the lanes of a world, G at a time (`on`
// where there is one), so an island's records keep the list's order.  Every
// lane of the warp calls it.
template <int G, class R>
__device__ __forceinline__ int next_record(const BatchView<R>& v, long long cst, int k, bool on, int gl, uint16_t* cur,
                                           const uint8_t* lab) {
  const int lane = threadIdx.x & 31;
  int r = 0;
  if (on) {
    const int bb = v.contact_bodies[cst + k];
    const int b0 = body0_of(bb);
    r = lab[b0 < 0 ? body1_of(bb) : b0];
  }
  const unsigned same = __match_any_sync(FULL, on ? (lane - gl) * 64 + r : -1 - lane);
  const int p = on ? cur[r] + __popc(same & ((1u << lane) - 1u)) : 0;
  __syncwarp();
  if (on && (same >> lane) == 1u) cur[r] = (uint16_t)(p + 1);
  __syncwarp();
  return p;
}

// adjustPositions (VEL false, contact.go:231-283) or adjustVelocities (VEL
// true, contact.go:388-445) of the worlds with `run` set, G lanes per world.
// Every lane of the warp calls it.
//
// The groups of L = 8 lanes each take the next island when their own is done;
// when no world of the warp has more than one island left, all its G lanes
// take that one (L = G): the islands left last are the long ones, and a round
// of theirs is then one update pass instead of one per eight contacts.  With
// `whole`, the world is one list for all G lanes from the start, the
// reference's own order of work.  WARPS > 1: the world is shared by as many
// warps; a group of lanes starts on island `seat` and takes further ones from
// shared[0], and shared[1] counts the world's iterations.  Equal values go to the contact that comes
// first in the narrowphase's list.  `over` is set when the iterations wanted
// exceed max_it.
//
// One body of code serves every width: with an instance each for the islands,
// the last island and the whole list, the warps of an SM ran from so much code
// that 8 of 15 stall cycles per instruction were instruction fetches.
//
// A lane's best key covers its contacts of the range in order (strict >, so
// its own first maximum).  In float32 the update pass, which visits them all,
// also finds the next one.  The float64 form first gathers the contacts
// touching the resolved bodies (a ballot per L contacts) and updates those,
// one per lane: walking all of them costs a whole warp instruction on the
// float64 pipe for every position with a match anywhere in the warp; the next
// argmax is then a separate scan.  The reference's loop visits every contact
// but changes only these, and each update touches only its own contact
// (contact.go:254-280, 412-440), so the result is the same bit for bit.
struct Progress {
  int used;    // iterations
  int rounds;  // rounds this world took part in
  bool over;   // the world wants more than max_it iterations
};
template <class R> using KeyOf = decltype(key_of((R)0, (R)0));
// What a phase runs: the records [s, e) as one list for all lanes (`list`), or
// the islands, leaving out the one that starts at record s; each until its
// first value's key is below `stop`.
template <class Key> struct Span {
  bool list;
  int s, e;
  Key stop;
};
// Of the islands under way when the budget ended, the one to go on from: its
// records, its iterations, and the smallest key among theirs and its next, the
// largest of the islands'.  tie: some list met a first value of key Span::stop.
template <class Key> struct Resume {
  Key stop;
  int s, e, its;
  bool tie;
};
template <class R, class W, int G, bool VEL, bool LEARN, int WARPS = 1>
__device__ __forceinline__ Progress resolve_phase(const RCtx<R, W, true>& x, const BatchView<R>& v, int bstart, int gl,
                                                  int max_it, bool run, Span<KeyOf<R>> sp, int ni, const uint16_t* ist,
                                                  int* ml_world, uint32_t& err, Resume<KeyOf<R>>& rs, int seat = 0,
                                                  int* shared = nullptr) {
  using Key = KeyOf<R>;
  constexpr bool kResume = G == 32;
  constexpr bool kGather = gathers_updates<R>();
  constexpr int kValue = VEL ? CR_DDV : CR_PEN;
  const int lane = threadIdx.x & 31;
  const unsigned wmask = G == 32 ? FULL : (((1u << G) - 1u) << (lane - gl));
  Progress pr{0, 0, false};
  int L = G, sl = gl, s = sp.s, e = sp.e, next = 0, len = 0, cap = kTouchList, its = 0;
  Key low = ~(Key)0;  // smallest key of the island's iterations
  unsigned lmask = wmask;
  int* ml = ml_world;
  if (G > kIslandLanes && !sp.list) {
    L = kIslandLanes;
    sl = gl % L;
    lmask = 0xFFu << (lane - sl);
    cap = kTouchList / (G / L);
    ml = ml_world + gl / L * cap;
    s = e = 0;  // no island yet: the first round's maxima are zero
  } else {
    ni = 0;
  }
  bool have = run, scan = true;
  Key best = 0;
  int bidx = 0x7fffffff;
  auto consider = [&](int k, int bb, R value) {
    const Key key = key_of(value, (R)0.01);
    const int id = (int)((unsigned)bb & 0xFFFF0000u) | k;  // by list index
    if (key > best || (key == best && id < bidx)) {
      best = key;
      bidx = id;
    }
  };
#pragma unroll 1
  for (;;) {
    if (__any_sync(FULL, scan)) {
      if (scan) {
        best = 0;
        bidx = 0x7fffffff;
#pragma unroll 1
        for (int k = s + sl; have && k < e; k += L) consider(k, x.pair(k), x.rec(k)[kValue]);
      }
      scan = false;
      len = (int)__reduce_max_sync(FULL, (unsigned)(have ? e - s : 0));  // the longest of the warp's groups'
    }
    if (G > kIslandLanes && L == kIslandLanes)
      group_first_max<kIslandLanes>(best, bidx);
    else
      group_first_max<G>(best, bidx);
    const unsigned leaders = __ballot_sync(FULL, sl == 0) & wmask;
    const bool fin = have && best < sp.stop;
    const unsigned done = __ballot_sync(FULL, fin);
    if (done) {
      const unsigned m = done & leaders;
      if (fin) {  // the next island, in the order of the groups
        int isl;
        if constexpr (WARPS > 1) {
          isl = seat;
          if (seat < 0) {
            if (sl == 0) isl = atomicAdd(&shared[0], 1);
            isl = __shfl_sync(lmask, isl, lane - sl);
          }
          seat = -1;
          next = isl;
        } else {
          isl = next + __popc(m & ((1u << (lane - sl)) - 1u));
        }
        have = isl < ni;
        if (have) {
          if (kResume && ist[isl] >= sp.s) ++isl;
          s = ist[isl];
          e = ist[isl + 1];
        }
        its = 0;
        low = ~(Key)0;
        scan = true;
      }
      if (WARPS == 1) next += __popc(m);
      continue;
    }
    const unsigned live = __ballot_sync(FULL, have);
    if (!live) break;
    const int act = __popc(live & leaders);
    if (G > kIslandLanes && L == kIslandLanes &&
        (WARPS == 1 ? __all_sync(FULL, act <= 1 && next >= ni) : act <= 1 && __any_sync(FULL, next >= ni))) {
      // all lanes of the world on its last island
      const unsigned held = live & wmask;
      const int from = held ? __ffs(held) - 1 : lane;
      s = __shfl_sync(FULL, s, from);
      e = __shfl_sync(FULL, e, from);
      if (kResume) {
        its = __shfl_sync(FULL, its, from);
        low = __shfl_sync(FULL, low, from);
      }
      have = held != 0;
      L = G;
      sl = gl;
      lmask = wmask;
      cap = kTouchList;
      ml = ml_world;
      scan = true;
      continue;
    }
    if (kResume) {
      rs.tie = rs.tie || (have && best == sp.stop);
      low = best < low ? best : low;
    }
    int before = pr.used;
    if (WARPS > 1) {
      if (lane == 0) before = atomicAdd(&shared[1], act);
      before = __shfl_sync(FULL, before, 0);
    }
    if (act && before + act > max_it) {
      pr.over = true;
      if (kResume) {
        Key c = have ? low : 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          const Key y = __shfl_xor_sync(FULL, c, d);
          c = y > c ? y : c;
        }
        const int from = __ffs(__ballot_sync(FULL, have && low == c)) - 1;
        rs.stop = c;
        rs.s = __shfl_sync(FULL, s, from);
        rs.e = __shfl_sync(FULL, e, from);
        rs.its = __shfl_sync(FULL, its, from);
      }
    }
    ++its;
    pr.used += act;
    pr.rounds += act > 0;
    if (pr.over) have = false;
    const int k = bidx & 0xFFFF;
    const int bb = have ? x.pair(k) : 0;
    const int d0 = have ? x.B0(bb) : -2, d1 = have ? x.B1(bb) : -2;
    R lin, ang;
    bool woke = false;
    const bool mine = have && sl < 8;
    auto change = [&]() {
      // (loaded here: held across the first update_load they would spill)
      std::conditional_t<VEL, VelocityIn<R>, PositionIn<R, W>> in;
      if constexpr (VEL)
        velocity_load(x, in, k, bb, mine, sl);
      else
        position_load(x, in, k, bb, mine, sl);
      woke = match_awake(x, bb, have, sl == 0);
      if constexpr (VEL)
        velocity_change<R, W, LEARN>(x, v, in, k, mine, sl, lin, ang, err);
      else
        position_change(x, v, in, bstart, mine, sl, lin, ang);
    };
    if constexpr (kGather) {
      change();
      int m = 0;
#pragma unroll 1
      for (int base = 0; base < len; base += L) {
        const int j = s + base + sl;
        bool hit = false;
        if (have && j < e) {
          const int kb = x.pair(j);
          const int2 h = touching(x.B0(kb), x.B1(kb), d0, d1);
          hit = h.x >= 0 || h.y >= 0;
        }
        const unsigned bal = __ballot_sync(FULL, hit) & lmask;
        if (hit) ml[m + __popc(bal & ((1u << lane) - 1u))] = j;
        m += __popc(bal);
        if (__any_sync(FULL, m > cap - L) || base + L >= len) {
          __syncwarp();
          const int mm = (int)__reduce_max_sync(FULL, (unsigned)m);
          if (L > kIslandLanes && mm <= L / 2) {
#pragma unroll 1
            for (int q = sl >> 2; q - (sl >> 2) < mm; q += L / 4) {
              const int j = q < m ? ml[q] : 0;
              update_spread<VEL>(x, j, q < m ? x.pair(j) : 0, q < m, d0, d1, lin, ang, L, woke);
            }
          } else {
#pragma unroll 1
            for (int q = sl; q - sl < mm; q += L) {
              Touched<R> t;
              const int j = q < m ? ml[q] : 0;
              update_load<VEL>(x, t, j, q < m ? x.pair(j) : 0, q < m, d0, d1);
              update_apply<VEL>(x, t, lin, ang, L, woke);
            }
          }
          __syncwarp();
          m = 0;
        }
      }
      scan = have;
    } else {
      best = 0;
      bidx = 0x7fffffff;
#pragma unroll 1
      for (int base = 0; base < len; base += L) {
        // the first contacts' records load while the change is computed
        Touched<R> t;
        const int j = s + base + sl;
        const bool valid = have && j < e;
        update_load<VEL>(x, t, j, valid ? x.pair(j) : 0, valid, d0, d1);
        if (base == 0) change();
        const R value = update_apply<VEL>(x, t, lin, ang, L, woke);
        if (t.valid) consider(t.k, t.bb, value);
      }
    }
    __syncwarp();
  }
  return pr;
}

// A phase of the worlds with `run` set: their islands side by side (unless
// they are all `hard`: their last solve ran out of iterations); then, as
// one list, the worlds whose islands want more iterations than the budget,
// after restart(over, ...) has put them back (not with `once`: such a world
// only reports the whole budget used; nor a world of one island, whose list
// it is).
//
// With a world per warp less is put back.  The reference
// resolves the contact with the first value, over all islands: island j's
// t-th iteration comes in the order of m_j(t), the smallest of the island's
// first values so far (what follows a smaller value but is larger is resolved
// before any other island's value that the smaller one was ahead of).  When
// the budget ends, let U be the island under way whose smallest value so far,
// its next included, is the largest, c.  Every iteration U has had is ahead of
// every other island's from its first value below c on; so U has had none too
// many, and of the others only those with m_j > c come before U's next.  The
// others are put back and run to their first value below c; U goes on from
// where it is until its first value is below c; and if the budget has not
// ended by then, the world stands as the one list would have it, and goes on
// as that.  The whole world is put back where a value equals c (its place is
// then a matter of list order), where the others do not reach c within the
// budget (islands not begun), and where an error flag was set.  Half of the
// worlds out of budget were not in the frame before, and one of them is the
// chain that its launch waits for: 8192 worlds of 32 bodies took 1.20 ms at
// frame 120 and 1.19 at 300 with the whole world put back, 0.97 and 0.88 so
// (float64: 4.52 and 4.80, 3.99 and 4.16).
template <class R, class W, int G, bool VEL, bool LEARN, class F>
__device__ __forceinline__ Progress resolve_worlds(const RCtx<R, W, true>& x, const BatchView<R>& v, int bstart, int C,
                                                   int gl, int max_it, bool run, int ni, const uint16_t* ist, int* ml,
                                                   bool hard, bool once, uint32_t& err, F&& restart) {
  using Key = KeyOf<R>;
  constexpr int kNone = 0x7fffffff;
  Progress pr{0, 0, false};
  uint32_t er = 0;
  if constexpr (G == 32) {
    Span<Key> sp{false, kNone, C, 1};
    int part = 0, others = ni, ls = 0, le = 0;
    bool over = false;
#pragma unroll 1
    for (;;) {
      Resume<Key> rs{0, 0, 0, 0, false};
      const Progress p = resolve_phase<R, W, G, VEL, LEARN>(x, v, bstart, gl, max_it - pr.used, run, sp, others, ist,
                                                            ml, er, rs);
      pr.rounds += p.rounds;
      over = over || p.over;
      const bool bad = __any_sync(FULL, er != 0 || (part == 1 && rs.tie));
      if (part == 0 && p.over && !once && ni > 1 && !bad) {
        ls = rs.s;
        le = rs.e;
        pr.used = rs.its;
        sp = Span<Key>{false, ls, C, rs.stop};
        others = ni - 1;
        restart(true, ls, le);
        part = 1;
      } else if ((part == 0 && p.over && !once && ni > 1) || (part == 1 && (p.over || bad))) {
        restart(true, 0, 0);
        er = 0;
        pr.used = 0;
        sp = Span<Key>{true, 0, C, 1};
        part = 3;
      } else {
        pr.used += p.used;
        if (part == 0 || part == 3 || p.over) break;
        sp = part == 1 ? Span<Key>{true, ls, le, sp.stop} : Span<Key>{true, 0, C, 1};
        ++part;
      }
    }
    pr.over = over;
    if (over) pr.used = max_it;
  } else {
    bool on = run;
#pragma unroll 1
    for (bool whole = G == kIslandLanes || __all_sync(FULL, !run || hard);; whole = true) {
      Resume<Key> rs{0, 0, 0, 0, false};
      const Progress p = resolve_phase<R, W, G, VEL, LEARN>(
          x, v, bstart, gl, max_it, on, Span<Key>{whole, whole ? 0 : kNone, C, 1}, ni, ist, ml, er, rs);
      if (on) {
        pr.rounds += p.rounds;
        pr.used = p.over ? max_it : p.used;
      }
      // as one list, the budget's end is the reference's
      pr.over = pr.over || (on && p.over);
      on = on && p.over && !whole && !once && ni > 1;
      if (!__any_sync(FULL, on)) break;
      restart(on, 0, 0);
      if (on) er = 0;
    }
  }
  err |= er;
  return pr;
}

// label of the island of records [ks, ke), -1 for none
template <class R, class W>
__device__ __forceinline__ int island_label(const RCtx<R, W, true>& x, int ks, int ke, const uint8_t* lab) {
  if (ks >= ke) return -1;
  const int bb = x.pair(ks);
  return lab[x.B0(bb) < 0 ? x.B1(bb) : x.B0(bb)];
}
// Puts the worlds with `on` back to the state adjustPositions starts from, all
// but the island of the records [ks, ke), if any.  (Out of the kernel's code,
// as restart_velocities.)
template <class R, class W, int G>
__device__ __noinline__ void restart_positions(RCtx<R, W, true> x, const BatchView<R>& v, long long bstart,
                                               long long cst, int n, int C, int gl, bool on, int ks, int ke,
                                               const uint8_t* lab) {
  __syncwarp();
  if (on) load_bodies(x, v, bstart, n, gl, G, lab, island_label(x, ks, ke, lab));
#pragma unroll 1
  for (int k = gl; on && k < C; k += G)
    if (k < ks || k >= ke) x.rec(k)[CR_PEN] = v.contact[C_PEN * v.nc_total + cst + x.list_index(k)];
  __syncwarp();
}

// Puts the worlds with `on` back to the state adjustVelocities starts from:
// velocities, rotations, motion and awake flags (the batch rows still hold the
// values before the solve; awake_bits are the flags after adjustPositions,
// whose matchAwakeState may have woken bodies), and the contact velocities and
// desired delta velocities prepareContacts left (same velocities, relative
// positions, basis and awake flags); all but the island of the records
// [ks, ke), if any.  Harvested impulse totals start again at
// zero.  Every lane of the warp calls it.
// (Rare, so its code stays out of the kernel's: __noinline__, by value.)
template <class R, class W, int G>
__device__ __noinline__ void restart_velocities(RCtx<R, W, true> x, const R* body, const uint8_t* awake, long long S,
                                                long long bstart, int n, int C, int gl, bool on, unsigned awake_bits,
                                                bool harvest, int ks, int ke, const uint8_t* lab) {
  const R* g = body + bstart;
  const int keep = island_label(x, ks, ke, lab);
  __syncwarp();
  for (int i = gl; on && i < n; i += G) {
    if (lab[i] == keep) continue;
    R* b = x.body(i);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      b[BR_VEL + r] = g[(B_VX + r) * S + i];
      b[BR_ROT + r] = g[(B_RX + r) * S + i];
    }
    x.aw[i] = awake[bstart + i];
  }
  __syncwarp();
  for (int k = gl; on && k < C; k += G) {
    if (k >= ks && k < ke) continue;
    const int bb = x.pair(k), o = x.list_index(k);
    const int b0 = x.B0(bb), b1 = x.B1(bb);
    const m3<R> Ck = x.basis(k);
    v3<R> cv = local_velocity(x, b0, x.rel(0, k), Ck);
    if (b1 >= 0) sub(cv, local_velocity(x, b1, x.rel(1, k), Ck));
    const R vfa = frame_velocity(x, b0, b1, V<R>(Ck.m[0], Ck.m[1], Ck.m[2]));
    st4(x.rec(k) + CR_CV, cv.x, cv.y, cv.z, desired_dv(cv.x, vfa, x.restitution(o)));
    if (harvest) {
      x.J(0, o) = (R)0;
      x.J(1, o) = (R)0;
      x.J(2, o) = (R)0;
    }
  }
  __syncwarp();
  for (int i = gl, j = 0; on && i < n; i += G, ++j) {
    if (lab[i] == keep) continue;
    const bool was = x.aw[i] != 0, now = (awake_bits >> j) & 1u;
    x.body(i)[BR_MOTION] = now && !was ? (R)(0.3 * 2.0) : g[B_MOTION * S + i];
    if (now && !was) x.aw[i] = 1;
  }
  __syncwarp();
  for (int k = gl; on && k < C; k += G) {
    if (k >= ks && k < ke) continue;
    const int bb = x.pair(k);
    const R* r = x.rec(k);
    x.rec(k)[CR_VFA] = frame_velocity(x, x.B0(bb), x.B1(bb), V<R>(r[0], r[1], r[2]));
  }
  __syncwarp();
}

// v.mode: 0 plain, 1 harvest (plain, copying k_warm_features' features and
// writing the applied impulses), 2 learned warm start (applying
// k_warm_features' plan) with fallback to the plain solve.  LEARN = false
// compiles the plain resolver alone (v.mode is ignored), so the learned paths
// cost the plain kernel no registers.
// ---------------------------------------------------------------- one frame per world
// Survivor list of the narrowphase inside the fused frame (one warp per CTA).
constexpr int kFrameSurvivors = 128;

// Bytes of the narrowphase tile of one world in the fused frame: staged rows
// and collider transforms, shapes, cull data, scan scratch, survivor list.
template <class R> __host__ __device__ inline size_t frame_tile_bytes(int nbs) {
  size_t b = (size_t)(11 + 12) * nbs * sizeof(R) + (size_t)nbs * sizeof(int) + (size_t)5 * nbs * sizeof(float);
  b += (66 + kFrameSurvivors + np_sort_ints<R>(32)) * sizeof(int) + 8;
  return (b + 15) & ~(size_t)15;
}
// The fused frame's slot: the resolver's, large enough for the narrowphase
// tile too (the narrowphase runs first, in the same bytes).
template <class R, class W> __host__ __device__ inline size_t frame_slot_bytes(int nbs, int cs) {
  const size_t a = rs_slot_bytes<R, W>(nbs, cs), b = frame_tile_bytes<R>(nbs);
  return a > b ? a : b;
}

// Integrate + the colliders' derived data of world w's bodies, then its
// narrowphase, by the calling warp, the tile in the shared memory at base:
// the first two steps of the frame of examples/cubedrop.go:69-75, as
// k_integrate and k_narrowphase run them.
template <class R, class W>
__device__ void frame_front(const BatchView<R>& v, int w, int n, int bstart, int nbs, R dt, R sleep_bias,
                            unsigned char* base) {
  const int lane = threadIdx.x;
  for (int i = lane; i < n; i += 32) integrate_body<R, W>(v, (long long)bstart + i, dt, sleep_bias);
  __syncwarp();
  NPTile<R> tl;
  tl.nbs = nbs;
  tl.stage = reinterpret_cast<R*>(base);
  tl.T = tl.stage + 11 * nbs;
  tl.shape = reinterpret_cast<int*>(tl.T + 12 * nbs);
  tl.cull = reinterpret_cast<float*>(tl.shape + nbs);
  int* scan = reinterpret_cast<int*>(tl.cull + 5 * nbs);
  int* surv = scan + 66;
  for (int i = lane; i < n; i += 32) {
#pragma unroll
    for (int r = 0; r < 11; ++r) tl.stage[r * nbs + i] = v.body[(long long)r * v.nb_pad + bstart + i];
    tl.shape[i] = v.shape[bstart + i];
  }
  __syncwarp();
  np_build_tile(tl, n, v.offset ? v.offset + bstart : nullptr, v.nb_pad);
  __syncwarp();
  int parity = 0;
  np_world<R, NP_SMALL>(tl, v, w, n, bstart, scan, parity, surv, kFrameSurvivors);
  __syncwarp();
}

// The resolver: G lanes per world, worlds from the device queue.  FRAME (the
// fused frame): each world's integrate and narrowphase first
// (frame_front), so one launch runs a whole frame (one world per warp, plain
// resolver).
// Most warps per CTA (each its own slot and its own worlds from the queue; the
// host picks the count).  Registers: float32 with one world per warp has 128,
// 16 warps per SM: at 96 (18 warps, what shared memory allows) the loops'
// spills missed the little L1 that the slots leave.
template <class R, int G, bool FRAME> __host__ __device__ constexpr int rs_wpc() {
  return sizeof(R) == 4 && G == 32 && !FRAME ? 8 : 1;
}
template <class R, class W, int G, bool LEARN, bool FRAME = false>
__global__ void __launch_bounds__(32 * rs_wpc<R, G, FRAME>(),
                                  FRAME ? (sizeof(R) == 4 ? 16 : 8)
                                        : (G == 32 && sizeof(R) == 4 ? 2 : 8))
    k_resolve(BatchView<R> v, int nbs, int cs, R dt, R sleep_bias = (R)0) {
  static_assert(!FRAME || (G == 32 && !LEARN), "the fused frame runs one world per warp, plain");
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int NG = 32 / G;
  const int lane = threadIdx.x & 31;
  const int grp = lane / G, gl = lane % G;
  const int mode = LEARN ? v.mode : 0;
  const size_t slot_bytes = FRAME ? frame_slot_bytes<R, W>(nbs, cs) : rs_slot_bytes<R, W>(nbs, cs);
  Slot<R, W> sl = make_slot<R, W>(smem + (size_t)((threadIdx.x >> 5) * NG + grp) * slot_bytes, nbs, cs, dt);
  RCtx<R, W, true>& x = sl.x;
  for (;;) {
    unsigned q0 = 0;
    if (lane == 0) q0 = atomicAdd(&v.queue[1], (unsigned)NG);
    q0 = __shfl_sync(FULL, q0, 0);
    if (q0 >= (unsigned)v.num_worlds) break;
    const unsigned qi = q0 + grp;
    bool has = qi < (unsigned)v.num_worlds;
    const int w = has ? v.order_rs[qi] : 0;
    if (has && v.big_count > 0 && v.body_count[w] > nbs) has = false;  // a world of k_resolve_big
    const int n = has ? v.body_count[w] : 0;
    const int bstart = has ? v.body_start[w] : 0;
    if constexpr (FRAME) {
      if (has && n <= nbs) frame_front<R, W>(v, w, n, bstart, nbs, dt, sleep_bias, smem);
      __syncwarp();
    }
    int C = has ? v.contact_count[w] : 0;
    // about half of the worlds whose adjustVelocities ran out of its budget do
    // so again in the next frame: they are solved as one list at once
    const bool hard = G < 32 && has && (v.cost[w] & kExhausted) != 0;
    if (has) {
      const int cap = v.contact_cap[w];
      if (C > cap) C = cap;  // the world is already flagged ST_CAPACITY
      if (gl == 0) {
        v.pos_iters[w] = 0;
        v.vel_iters[w] = 0;
        v.cost[w] = 0;
      }
    }
    bool active = has && C > 0 && dt > (R)0;  // ResolveContacts guards, contact.go:210-212
    if (active && n > nbs) {
      if (gl == 0) {
        atomicOr(&v.world_status[w], ST_BODY_LIMIT);
        atomicOr(v.status, ST_BODY_LIMIT);
      }
      active = false;
    }
    const long long cst = has ? v.contact_start[w] : 0;
    bind_contacts(sl, v, C, cs, cst);
    if (LEARN && mode) bind_ws(x, v, bstart, cst);
    constexpr int L = kIslandLanes;
    constexpr bool kIslands = G > L;
    const int Ca = active ? C : 0;
    x.all_awake = __all_sync(FULL, !active || load_bodies(x, v, bstart, n, gl, G));
    int ni = 0;
    // (its scratch is the contact tile, which prepare_contact fills next)
    if constexpr (kIslands)
      ni = build_islands<G>(v, cst, active ? n : 0, nbs, Ca, gl, reinterpret_cast<int*>(sl.cr_s), sl.ist, sl.cur,
                            sl.lab);
    __syncwarp();
    int Cmax = Ca;  // next_record needs every lane of the warp
    if (G < 32) Cmax = (int)__reduce_max_sync(FULL, (unsigned)Cmax);
#pragma unroll 1
    for (int base = 0; base < Cmax; base += G) {
      const int k = base + gl;
      int p = k;
      if constexpr (kIslands) p = next_record<G>(v, cst, k, k < Ca, gl, sl.cur, sl.lab);
      if (k < Ca) prepare_contact(x, v, cst + k, p, k);
    }
    __syncwarp();
    const int max_it = v.max_iterations >= 0 ? v.max_iterations : C * v.iter_mult;
    const bool solve = active && max_it > 0;
    uint32_t err = 0;
    // ---------------- adjustPositions, contact.go:231-283
    const Progress pos = resolve_worlds<R, W, G, false, LEARN>(
        x, v, bstart, C, gl, max_it, solve, ni, sl.ist, sl.ml, false, false, err, [&](bool over, int ks, int ke) {
          restart_positions<R, W, G>(x, v, bstart, cst, n, C, gl, over, ks, ke, sl.lab);
        });
    const int pos_used = pos.used;
    if (active && v.contact_writeback)  // the caller's Contact.Penetration after ResolveContacts
      for (int k = gl; k < C; k += G) v.contact[C_PEN * v.nc_total + cst + x.list_index(k)] = x.rec(k)[CR_PEN];
    if (solve)
#pragma unroll 1
      for (int k = gl; k < C; k += G) friction_prepare(x, k);
    __syncwarp();
    // awake flags after adjustPositions, of this lane's bodies (restart_velocities)
    unsigned awake_bits = 0;
    for (int i = gl, j = 0; solve && i < n; i += G, ++j) awake_bits |= (x.aw[i] ? 1u : 0u) << j;
    // ---------------- learned warm start / harvest set-up
    long long hv_base = -1;
    // the per-body aggregates and the predicted impulses come from k_warm_features
    if (LEARN && mode == 1)  // harvest: the impulse totals start at zero
      for (int k = gl; solve && k < C; k += G) {
        x.J(0, k) = (R)0;
        x.J(1, k) = (R)0;
        x.J(2, k) = (R)0;
      }
    __syncwarp();
    if (LEARN && mode == 1) {
      // every lane takes part in the shuffle; only solving groups reserve rows
      unsigned long long b0 = 0;
      if (solve && gl == 0) b0 = atomicAdd(v.hv_count, (unsigned long long)C);
      b0 = __shfl_sync(FULL, b0, grp * G);
      if (solve && (long long)(b0 + C) <= v.hv_cap) {
        hv_base = (long long)b0;
        for (int k = gl; k < C; k += G) {
          const float* f = v.ws_feat + (cst + k) * MLP_IN;  // written by k_warm_features
          float* o = v.hv_features + (hv_base + k) * MLP_IN;
#pragma unroll
          for (int c = 0; c < MLP_IN; ++c) o[c] = f[c];
        }
      }
    }
    bool warmed = false;  // this world had a warm-started body
    // a world whose last solve used more than max_it >> warm_shift iterations
    // (a quarter by default) is solved plainly: hard worlds are the ones that
    // exhaust the budget and are then re-solved (a re-solve costs a whole
    // solve in lockstep)
    const bool warm_ok = LEARN && mode == 2 && solve && !v.ws_world[w];
    if (LEARN && mode == 2) {
      const int nw = warm_start_apply<R, W, G>(x, n, C, gl, warm_ok);
      __syncwarp();
      warmed = group_sum<G>(nw) > 0;
    }
    // ---------------- adjustVelocities, contact.go:388-445
    auto restart = [&](bool over, int ks, int ke) {
      if (__any_sync(FULL, over))
        restart_velocities<R, W, G>(x, v.body, v.awake, v.nb_pad, bstart, n, C, gl, over, awake_bits,
                                    LEARN && mode == 1, ks, ke, sl.lab);
    };
    int vel_used = 0, rounds = 2 * pos.rounds;
    bool exhausted = false;
    bool todo = solve;
    for (bool first = true; __any_sync(FULL, todo); first = false) {
      const Progress vel = resolve_worlds<R, W, G, true, LEARN>(x, v, bstart, C, gl, max_it, todo, ni, sl.ist, sl.ml,
                                                                hard, first && warmed, err, restart);
      bool again = false;
      if (todo) {
        vel_used += vel.used;
        rounds += vel.rounds;
        exhausted = vel.over;
        if (LEARN && mode == 2 && first) {
          // the plain resolver has the last word: a warm-started world that
          // used all its iterations is solved again by the plain path (a
          // world without a warm-started body was solved plainly)
          if (gl == 0) v.ws_world[w] = ((long long)vel.used << v.warm_shift) > max_it;
          again = warmed && vel.used >= max_it;
          if (again && gl == 0) atomicAdd(&v.counters[4], 1ull);
        }
      }
      if (LEARN) restart(again, 0, 0);
      todo = again;
    }
    if (LEARN && mode == 2 && warm_ok && gl == 0) atomicAdd(&v.counters[5], 1ull);
    if (err) {
      atomicOr(&v.world_status[w], err);
      atomicOr(v.status, err);
    }
    if (LEARN && mode == 1 && hv_base >= 0) {
      for (int k = gl; k < C; k += G) {
        float* lab = v.hv_labels + (hv_base + k) * MLP_OUT;
        lab[0] = (float)x.J(0, k);
        lab[1] = (float)x.J(1, k);
        lab[2] = (float)x.J(2, k);
      }
    }
    if (has && gl == 0) {
      v.pos_iters[w] = pos_used;
      v.cost[w] = rounds | (exhausted ? kExhausted : 0);
      v.vel_iters[w] = vel_used;
      atomicAdd(&v.counters[1], (unsigned long long)pos_used);
      atomicAdd(&v.counters[2], (unsigned long long)vel_used);
      atomicAdd(&v.counters[3], (unsigned long long)C);
    }
    if (active && v.contact_writeback)
      for (int k = gl; k < C; k += G) write_back_contact(x, v, cst, k);
    if (active) store_bodies(x, v, bstart, n, gl, G);
    __syncwarp();
  }
}


// ---------------------------------------------------------------- k_resolve_wide
// The resolver for small batches, up to seven worlds per SM (wide_rule in
// cz_api.cu): four warps to a world, one CTA each.  With one warp a small batch leaves three of an SM's four
// schedulers idle, and in float64 each scheduler has its own quarter of the
// SM's float64 rate, so a warp on its own is bound by its scheduler's unit.
// The preparation is split over the warps, and so are the world's islands
// (side by side within a warp where there are more than warps); bodies,
// records, friction matrices and lists are in shared memory, which such a batch
// has to spare.  A world whose islands want more iterations than its budget
// goes on as in resolve_worlds, the one island and the one list by the first
// warp.
constexpr int kWideWarps = 4;
// What the warps share: the next island, the iterations (resolve_phase), then
// per call the sum of the iterations, the most rounds, whether a warp met the
// budget, a tie or an error flag, and each warp's island to go on from.
template <class Key> struct WideShared {
  int island, count, used, rounds, over, tie, err, world, islands;
  Resume<Key> rs[kWideWarps];
};
// shared memory of one world, with tiles of cs contacts
template <class R, class W> __host__ __device__ inline size_t wide_smem_bytes(int nbs, int cs) {
  size_t b = rs_slot_bytes<R, W>(nbs, cs);
  b += (size_t)K_ROW * cs * sizeof(R);
  b += (size_t)kWideWarps * kTouchList * sizeof(int);
  b += (size_t)kWideWarps * nbs * sizeof(uint16_t);
  b = (b + 15) & ~(size_t)15;
  return b + sizeof(WideShared<KeyOf<R>>);
}

// resolve_worlds for one world by the CTA's warps
template <class R, class W, bool VEL, class F>
__device__ __forceinline__ Progress wide_phase(const RCtx<R, W, true>& x, const BatchView<R>& v, int bstart, int C,
                                               int max_it, int ni, const uint16_t* ist, int* ml,
                                               WideShared<KeyOf<R>>* sh, uint32_t& err, F&& restart) {
  using Key = KeyOf<R>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  Span<Key> sp{false, 0x7fffffff, C, 1};
  int part = 0, others = ni, ls = 0, le = 0;
  Progress pr{0, 0, false};
  bool over = false;
  uint32_t er = 0;
#pragma unroll 1
  for (;;) {
    if (threadIdx.x == 0) {
      sh->island = kWideWarps * (32 / kIslandLanes);
      sh->count = sh->used = sh->rounds = sh->over = sh->tie = sh->err = 0;
    }
    if (lane == 0) sh->rs[wid].stop = 0;
    __syncthreads();
    Resume<Key> rs{0, 0, 0, 0, false};
    const Progress p = resolve_phase<R, W, 32, VEL, false, kWideWarps>(
        x, v, bstart, lane, max_it - pr.used, !sp.list || wid == 0, sp, others, ist, ml, er, rs,
        wid + kWideWarps * (lane / kIslandLanes), &sh->island);
    if (rs.tie) sh->tie = 1;
    if (er) sh->err = 1;
    if (lane == 0) {
      atomicAdd(&sh->used, p.used);
      atomicMax(&sh->rounds, p.rounds);
      if (p.over) {
        sh->over = 1;
        sh->rs[wid] = rs;
      }
    }
    __syncthreads();
    const int used = sh->used;
    const bool out = sh->over != 0, bad = sh->err != 0 || (part == 1 && sh->tie != 0);
    pr.rounds += sh->rounds;
    over = over || out;
    rs = sh->rs[0];
#pragma unroll
    for (int q = 1; q < kWideWarps; ++q)
      if (sh->rs[q].stop > rs.stop) rs = sh->rs[q];
    __syncthreads();
    if (part == 0 && out && ni > 1 && !bad) {
      ls = rs.s;
      le = rs.e;
      pr.used = rs.its;
      sp = Span<Key>{false, ls, C, rs.stop};
      others = ni - 1;
      restart(ls, le);
      part = 1;
    } else if ((part == 0 && out && ni > 1) || (part == 1 && (out || bad))) {
      restart(0, 0);
      er = 0;
      pr.used = 0;
      sp = Span<Key>{true, 0, C, 1};
      part = 3;
    } else {
      pr.used += used;
      if (part == 0 || part == 3 || out) break;
      sp = part == 1 ? Span<Key>{true, ls, le, sp.stop} : Span<Key>{true, 0, C, 1};
      ++part;
    }
    __syncthreads();
  }
  pr.over = over;
  if (over) pr.used = max_it;
  err |= er;
  return pr;
}

// PER_SM worlds fit an SM's registers: one of its own keeps 1.5 % with the
// registers it wants (float64 180, float32 179; three leave 168).
template <class R, class W, int PER_SM>
__global__ void __launch_bounds__(32 * kWideWarps, PER_SM) k_resolve_wide(BatchView<R> v, int nbs, int cs, R dt) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int T = 32 * kWideWarps;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  Slot<R, W> sl = make_slot<R, W>(smem, nbs, cs, dt);
  RCtx<R, W, true>& x = sl.x;
  R* k_tile = reinterpret_cast<R*>(smem + rs_slot_bytes<R, W>(nbs, cs));
  int* ml = reinterpret_cast<int*>(k_tile + (size_t)K_ROW * cs) + wid * kTouchList;
  uint16_t* curs = reinterpret_cast<uint16_t*>(reinterpret_cast<int*>(k_tile + (size_t)K_ROW * cs) +
                                               kWideWarps * kTouchList);
  uint16_t* cur = curs + wid * nbs;
  WideShared<KeyOf<R>>* sh = reinterpret_cast<WideShared<KeyOf<R>>*>(
      smem + (((size_t)(reinterpret_cast<unsigned char*>(curs + kWideWarps * nbs) - smem) + 15) & ~(size_t)15));
  for (;;) {
    if (tid == 0) sh->world = (int)atomicAdd(&v.queue[1], 1u);
    __syncthreads();
    const int qi = sh->world;
    if (qi >= v.num_worlds) break;
    const int w = v.order_rs[qi];
    const int n = v.body_count[w];
    if (n > nbs) {  // a world of k_resolve_big
      __syncthreads();
      continue;
    }
    const int bstart = v.body_start[w];
    int C = v.contact_count[w];
    if (C > v.contact_cap[w]) C = v.contact_cap[w];  // the world is already flagged ST_CAPACITY
    const bool active = C > 0 && dt > (R)0;  // ResolveContacts guards, contact.go:210-212
    int pos_used = 0, vel_used = 0, cost = 0;
    uint32_t err = 0;
    if (active) {
      const long long cst = v.contact_start[w];
      bind_contacts(sl, v, C, cs, cst);
      if (C <= cs) x.kw = k_tile;
      x.all_awake = __syncthreads_and(load_bodies(x, v, bstart, n, tid, T));
      if (wid == 0) {
        const int ni = build_islands<32>(v, cst, n, nbs, C, lane, reinterpret_cast<int*>(sl.cr_s), sl.ist, sl.cur,
                                         sl.lab);
        if (lane == 0) sh->islands = ni;
      }
      __syncthreads();
      const int ni = sh->islands;
      // every warp counts the places of all contacts, and prepares its share
      for (int i = lane; i < n; i += 32) cur[i] = sl.cur[i];
      __syncwarp();
#pragma unroll 1
      for (int base = 0; base < C; base += 32) {
        const int k = base + lane;
        const int p = next_record<32>(v, cst, k, k < C, lane, cur, sl.lab);
        if ((base >> 5) % kWideWarps == wid && k < C) prepare_contact(x, v, cst + k, p, k);
      }
      __syncthreads();
      const int max_it = v.max_iterations >= 0 ? v.max_iterations : C * v.iter_mult;
      if (max_it > 0) {
        const Progress pos = wide_phase<R, W, false>(
            x, v, bstart, C, max_it, ni, sl.ist, ml, sh, err, [&](int ks, int ke) {
              load_bodies(x, v, bstart, n, tid, T, sl.lab, island_label(x, ks, ke, sl.lab));
              for (int k = tid; k < C; k += T)
                if (k < ks || k >= ke) x.rec(k)[CR_PEN] = v.contact[C_PEN * v.nc_total + cst + x.list_index(k)];
            });
        pos_used = pos.used;
        cost = 2 * pos.rounds;
      }
      if (v.contact_writeback)  // the caller's Contact.Penetration after ResolveContacts
        for (int k = tid; k < C; k += T) v.contact[C_PEN * v.nc_total + cst + x.list_index(k)] = x.rec(k)[CR_PEN];
      __syncthreads();
      if (max_it > 0) {
#pragma unroll 1
        for (int k = tid; k < C; k += T) friction_prepare(x, k);
        // awake flags after adjustPositions, of the first warp's lanes' bodies
        unsigned awake_bits = 0;
        for (int i = lane, j = 0; i < n; i += 32, ++j) awake_bits |= (x.aw[i] ? 1u : 0u) << j;
        __syncthreads();
        const Progress vel = wide_phase<R, W, true>(
            x, v, bstart, C, max_it, ni, sl.ist, ml, sh, err, [&](int ks, int ke) {
              if (wid == 0)
                restart_velocities<R, W, 32>(x, v.body, v.awake, v.nb_pad, bstart, n, C, lane, true, awake_bits, false,
                                             ks, ke, sl.lab);
            });
        vel_used = vel.used;
        cost += vel.rounds;
      }
      if (err) {
        atomicOr(&v.world_status[w], err);
        atomicOr(v.status, err);
      }
      if (v.contact_writeback)
        for (int k = tid; k < C; k += T) write_back_contact(x, v, cst, k);
      store_bodies(x, v, bstart, n, tid, T);
    }
    if (tid == 0) {
      v.pos_iters[w] = pos_used;
      v.vel_iters[w] = vel_used;
      v.cost[w] = cost;
      atomicAdd(&v.counters[1], (unsigned long long)pos_used);
      atomicAdd(&v.counters[2], (unsigned long long)vel_used);
      atomicAdd(&v.counters[3], (unsigned long long)C);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- k_warm_features
// Shared-memory copy of the inference weights (fragment layouts of MlpDev).
constexpr size_t WF_W1 = 0;                       // [64][32] bf16
constexpr size_t WF_W2 = WF_W1 + 64 * 32 * 2;     // [64][64]
constexpr size_t WF_W3 = WF_W2 + 64 * 64 * 2;     // [64][64]
constexpr size_t WF_W4 = WF_W3 + 64 * 64 * 2;     // [8][64]
constexpr size_t WF_B1 = WF_W4 + 8 * 64 * 2;      // f32 [64]
constexpr size_t WF_B2 = WF_B1 + 64 * 4;
constexpr size_t WF_B3 = WF_B2 + 64 * 4;
constexpr size_t WF_B4 = WF_B3 + 64 * 4;          // [8]
constexpr size_t WF_MU = WF_B4 + 8 * 4;           // [32]
constexpr size_t WF_IS = WF_MU + 32 * 4;          // [32]
constexpr size_t WF_OS = WF_IS + 32 * 4;          // [4]
constexpr size_t WF_BYTES = WF_OS + 16;
constexpr int kWfWarps = 4;                       // worlds in flight per CTA

// bytes of one warp's body rows, and of a CTA
template <class R, class W> __host__ __device__ inline size_t wf_slot_bytes(int nbs) {
  return ((size_t)7 * nbs * sizeof(W) + (size_t)BREC * nbs * sizeof(R) + (size_t)((nbs + 15) & ~15) + 15) & ~(size_t)15;
}
template <class R, class W> __host__ __device__ inline size_t wf_smem_bytes(int nbs) {
  return WF_BYTES + kWfWarps * wf_slot_bytes<R, W>(nbs);
}

// The learned warm start's features and predictions, ahead of k_resolve and
// off its sequential path: one warp per world, kWfWarps worlds per CTA, the
// network's weights staged once per CTA in shared memory.  A warp takes the
// worlds k_resolve will warm-start (in harvest mode, v.mode == 1: every world
// it solves), stages the bodies, runs calculateInternals (prepare_contact) into
// the world's global working rows, accumulates the per-body aggregates
// (integer atomics: order-free, deterministic) and computes each contact's
// features; mode 2 predicts the impulses in 16-contact BF16 tensor-core tiles
// into the impulse rows, mode 1 writes the features to ws_feat for the harvest.
// Same bodies, contacts and arithmetic as k_resolve's own prepareContacts, so
// the features describe the state adjustVelocities starts from.
template <class R, class W>
__global__ void __launch_bounds__(32 * kWfWarps) k_warm_features(BatchView<R> v, int nbs, R dt) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // weights: global (v.mlp) -> shared
  {
    auto copy = [&](size_t off, const void* src, size_t bytes) {
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
      uint4* d4 = reinterpret_cast<uint4*>(smem + off);
      for (size_t i = tid; i < bytes / 16; i += blockDim.x) d4[i] = s4[i];
    };
    if (v.mode == 2) {
      copy(WF_W1, v.mlp.W1, 64 * 32 * 2);
      copy(WF_W2, v.mlp.W2, 64 * 64 * 2);
      copy(WF_W3, v.mlp.W3, 64 * 64 * 2);
      copy(WF_W4, v.mlp.W4, 8 * 64 * 2);
      copy(WF_B1, v.mlp.b1, 64 * 4);
      copy(WF_B2, v.mlp.b2, 64 * 4);
      copy(WF_B3, v.mlp.b3, 64 * 4);
      copy(WF_B4, v.mlp.b4, 8 * 4);
      float* mu = reinterpret_cast<float*>(smem + WF_MU);
      float* is = reinterpret_cast<float*>(smem + WF_IS);
      float* os = reinterpret_cast<float*>(smem + WF_OS);
      for (int c = tid; c < 32; c += blockDim.x) {
        mu[c] = c < MLP_IN ? v.mlp.mu[c] : 0.f;
        is[c] = c < MLP_IN ? v.mlp.inv_sigma[c] : 0.f;
      }
      for (int c = tid; c < 4; c += blockDim.x) os[c] = c < MLP_OUT ? v.mlp.out_scale[c] : 0.f;
    }
  }
  __syncthreads();
  MlpDev m;
  m.W1 = reinterpret_cast<const __nv_bfloat16*>(smem + WF_W1);
  m.W2 = reinterpret_cast<const __nv_bfloat16*>(smem + WF_W2);
  m.W3 = reinterpret_cast<const __nv_bfloat16*>(smem + WF_W3);
  m.W4 = reinterpret_cast<const __nv_bfloat16*>(smem + WF_W4);
  m.b1 = reinterpret_cast<const float*>(smem + WF_B1);
  m.b2 = reinterpret_cast<const float*>(smem + WF_B2);
  m.b3 = reinterpret_cast<const float*>(smem + WF_B3);
  m.b4 = reinterpret_cast<const float*>(smem + WF_B4);
  const float* mu = reinterpret_cast<const float*>(smem + WF_MU);
  const float* isg = reinterpret_cast<const float*>(smem + WF_IS);
  const float* osc = reinterpret_cast<const float*>(smem + WF_OS);
  unsigned char* slot = smem + WF_BYTES + (size_t)wid * wf_slot_bytes<R, W>(nbs);
  RCtx<R, W, true> x;
  x.nbs = nbs;
  x.dt = dt;
  x.bw = reinterpret_cast<W*>(slot);
  x.br = reinterpret_cast<R*>(x.bw + 7 * nbs);
  x.aw = reinterpret_cast<uint8_t*>(x.br + BREC * nbs);
  x.delta = nullptr;
  x.kw = nullptr;
  x.all_awake = false;
  const bool harvest = v.mode == 1;
  for (;;) {
    unsigned q = 0;
    if (lane == 0) q = atomicAdd(&v.queue[2], 1u);
    q = __shfl_sync(FULL, q, 0);
    if (q >= (unsigned)v.num_worlds) break;
    const int w = v.first_world + (int)q;
    const int n = v.body_count[w];
    int C = v.contact_count[w];
    const int cap = v.contact_cap[w];
    if (C > cap) C = cap;
    const int max_it = v.max_iterations >= 0 ? v.max_iterations : C * v.iter_mult;
    // the worlds k_resolve solves, and warm-starts unless solving plainly
    if (C <= 0 || dt <= (R)0 || n > nbs || max_it <= 0 || (!harvest && v.ws_world[w])) continue;
    const long long bstart = v.body_start[w];
    const long long cst = v.contact_start[w];
    x.cr = v.work + cst * CREC;
    x.cb = v.work_bodies + cst;
    x.gmat = v.uniform_material ? nullptr : v.contact + (long long)C_FRIC * v.nc_total + cst;
    x.gst = (long long)(C_REST - C_FRIC) * v.nc_total;
    bind_ws(x, v, bstart, cst);
    load_bodies(x, v, bstart, n, lane, 32);
    for (int i = lane; i < n; i += 32) {
      x.WI(WS_DEG, i) = 0;
      x.WI(WS_NBB, i) = 0;
      x.WI(WS_LOAD, i) = 0;
      x.WI(WS_FIRST, i) = 0x7fffffff;
      x.WI(WS_LAST, i) = -1;
    }
    __syncwarp();
    for (int k = lane; k < C; k += 32) {
      prepare_contact(x, v, cst + k, k, k);
      const int bb = x.pair(k);
      const int b0 = x.B0(bb), b1 = x.B1(bb);
      const float dd = (float)x.rec(k)[CR_DDV];
      const int fx = dd > 0.f ? (int)(fminf(dd, 100.f) * kLoadScale + 0.5f) : 0;
      atomicAdd(&x.WI(WS_DEG, b0), 1);
      atomicAdd(&x.WI(WS_LOAD, b0), fx);
      if (b1 >= 0) {
        atomicAdd(&x.WI(WS_DEG, b1), 1);
        atomicAdd(&x.WI(WS_LOAD, b1), fx);
        atomicAdd(&x.WI(WS_NBB, b0), 1);
        atomicAdd(&x.WI(WS_NBB, b1), 1);
      } else {
        atomicMin(&x.WI(WS_FIRST, b0), k);
        atomicMax(&x.WI(WS_LAST, b0), k);
      }
    }
    __syncwarp();
    if (harvest) {
      for (int k = lane; k < C; k += 32) contact_features(x, k, v.ws_feat + (cst + k) * MLP_IN);
      __syncwarp();
      continue;
    }
    for (int t0 = 0; t0 < C; t0 += 16) {
      // lanes 0..15 compute one contact's normalised features each; the tile
      // reaches the MMA fragments and back by shuffles alone
      unsigned row[16];
      const int k = t0 + lane;
      const bool mine = lane < 16 && k < C;
      float f[MLP_IN];
      if (mine) contact_features(x, k, f);
#pragma unroll
      for (int c = 0; c < MLP_K1; c += 2) {
        float lo = 0.f, hi = 0.f;
        if (mine && c < MLP_IN) lo = (f[c] - mu[c]) * isg[c];
        if (mine && c + 1 < MLP_IN) hi = (f[c + 1] - mu[c + 1]) * isg[c + 1];
        row[c / 2] = pack_bf16(lo, hi);
      }
      unsigned a[2][4];
      rows_to_a(row, a);
      float o[4], y[3];
      mlp_forward_tile(m, a, o);
      out_to_rows(o, y);
      if (mine) {
#pragma unroll
        for (int c = 0; c < 3; ++c) x.J(c, k) = (R)(y[c] * osc[c]);
      }
    }
    __syncwarp();
    int nw = 0;
    float ssum = 0.f;
    warm_start_plan(x, n, C, lane, &nw, &ssum);
    if (nw) {
      atomicAdd(&v.counters[6], (unsigned long long)((double)ssum * 1e6 + 0.5));
      atomicAdd(&v.counters[7], (unsigned long long)nw);
    }
    __syncwarp();
  }
}

}  // namespace cz

