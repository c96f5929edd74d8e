// ResolveContacts (contact.go:204-445) for worlds whose bodies do not fit the
// shared-memory slot of k_resolve (hundreds to thousands of bodies).
//
// One warp per world (four in float64, sharing each iteration): such a world is
// mostly one island, so its iterations are one chain, and what counts is the
// latency of an iteration.
//   * Body and contact records are in global memory (L1/L2); a record is two
//     cache lines at most, where rows took a line per value.
//   * The argmax is over two levels of chunk maxima in shared memory, kept by
//     refreshing the chunks of the contacts an iteration changed, instead of a
//     scan over every contact's value.
//   * After prepareContacts every body gets the list of its contacts (counting
//     sort by body), so the update after each resolved contact visits only the
//     contacts of the two resolved bodies: the reference's loop over every
//     contact skips the others, so the visited set and each contact's
//     arithmetic are the same (contact_update), and the bits too.  The order
//     of the visits does not matter: each contact's update reads only its own
//     record and the resolved contact's changes.
//   * The packed bodies, the keys and the lists are in shared memory where the
//     world's contacts fit it, so the records an update will need are known,
//     and loaded, while the resolved contact's change is computed.
#pragma once
#include "cz_resolve.cuh"

namespace cz {

constexpr int kBigChunks = 512;  // chunks of a world's contacts (16 each up to 8192 contacts)
constexpr int kBigTops = kBigChunks / 16;  // groups of 16 chunks: one per lane

// the change shared between the warps (16-byte multiple)
template <class R> __host__ __device__ constexpr size_t big_change_bytes() { return 16 * sizeof(R) + 16; }
// shared memory ahead of the per-contact arrays: maxima and their contacts of
// the chunks and of the groups of chunks, list starts and ends of n bodies
template <class R> __host__ __device__ inline size_t big_fixed_bytes(int n) {
  return (size_t)(kBigChunks + kBigTops) * (sizeof(R) + sizeof(int)) + (size_t)2 * ((n + 3) & ~3) * sizeof(int) +
         big_change_bytes<R>();
}
// per contact: key, packed bodies, two list entries
template <class R> __host__ __device__ constexpr size_t big_contact_bytes() { return sizeof(R) + 3 * sizeof(int); }

__device__ __forceinline__ void prefetch_line(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// The first maximum of 16 consecutive keys (16-byte aligned): adjacent pairs,
// so that the left one of equals is the earlier.
template <class Key> __device__ __forceinline__ void first_max16(const Key* p, Key& best, int& at) {
  constexpr int V = 16 / (int)sizeof(Key);
  union {
    uint4 v[16 / V];
    Key k[16];
  } u;
#pragma unroll
  for (int i = 0; i < 16 / V; ++i) u.v[i] = reinterpret_cast<const uint4*>(p)[i];
  int ix[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) ix[i] = i;
#pragma unroll
  for (int w = 8; w > 0; w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const bool right = u.k[2 * i + 1] > u.k[2 * i];
      u.k[i] = right ? u.k[2 * i + 1] : u.k[2 * i];
      ix[i] = right ? ix[2 * i + 1] : ix[2 * i];
    }
  best = u.k[0];
  at = ix[0];
}

// The maxima of a world's keys by chunk and by group of 16 chunks, with the
// first contact holding each: the world's argmax is one load per lane and the
// warp reductions.
template <class Key> struct BigKeys {
  Key* key;      // [C], zeros up to a whole chunk where `padded`
  Key* cmax;     // [kBigChunks] (zeros beyond the last chunk)
  int* cfirst;   // [kBigChunks]
  Key* tmax;     // [kBigTops]
  int* tfirst;   // [kBigTops]
  int C, shift;  // chunk of contact k: k >> shift
  bool padded;   // chunks of 16, whole
  // a chunk's first maximum again, by one lane
  __device__ __forceinline__ void refresh_chunk(int ch) const {
    Key best = 0;
    int at = 0;
    const int k0 = ch << shift;
    if (padded) {
      first_max16(key + k0, best, at);
      at += k0;
    } else {
      const int k1 = min(C, k0 + (1 << shift));
#pragma unroll 1
      for (int k = k0; k < k1; ++k) {
        const Key q = key[k];
        if (q > best) {
          best = q;
          at = k;
        }
      }
    }
    cmax[ch] = best;
    cfirst[ch] = at;
  }
  __device__ __forceinline__ void refresh_top(int t) const {
    Key best;
    int at;
    first_max16(cmax + 16 * t, best, at);
    tmax[t] = best;
    tfirst[t] = cfirst[16 * t + at];
  }
};

// Warps per world.  In float64 each of an SM's four schedulers has its own
// quarter of the float64 rate, and a warp alone is bound by its own: four
// warps share an iteration's updates, four lanes to a contact (update_spread),
// while its argmax and the resolved contact's change stay with one chain:
// 64 piles of 1024 cubes x 3 frames 128.8 -> 113.7 ms, 600 of 72 cubes (two
// worlds to a scheduler) 14.4 -> 13.7.  In float32 the updates are a sixth of
// an iteration, about what the barriers cost.
template <class R> __host__ __device__ constexpr int big_warps() { return sizeof(R) == 8 ? 4 : 1; }
// A CTA is four warps in both forms: the preparation takes them all, and with
// one-warp CTAs the worlds of an SM met on the same schedulers.  float32, x 3
// frames: 64 piles of 1024 cubes 42.1 -> 40.7 ms, 600 of 72 cubes 4.17 -> 3.61
// (with two warps 41.0 and 3.78).
constexpr int kBigThreads = 128;
// the resolved contact's change, for the other warps
template <class R> struct BigChange {
  R lin[8], ang[8];
  int woke;
};
template <int NW> __device__ __forceinline__ void big_sync() {
  if (NW > 1) __syncthreads();
  else __syncwarp();
}

// adjustPositions (VEL false) or adjustVelocities (VEL true) of one world by
// its warps; returns the iterations used.
template <class R, class W, bool VEL, class Key>
__device__ __forceinline__ int big_phase(const RCtx<R, W, false>& x, const BatchView<R>& v, int bstart,
                                         const BigKeys<Key>& bk, const int2* span, const int* adj,
                                         int max_it, BigChange<R>* chg, uint32_t& err) {
  constexpr int NW = big_warps<R>(), T = 32 * NW;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int C = bk.C;
  for (int k = tid; k < C; k += T) bk.key[k] = key_of(x.rec(k)[VEL ? CR_DDV : CR_PEN], (R)0.01);
  if (bk.padded && C + tid < ((C + 15) & ~15)) bk.key[C + tid] = 0;
  big_sync<NW>();
  const int nch = (C + (1 << bk.shift) - 1) >> bk.shift;
  for (int ch = tid; ch < kBigChunks; ch += T) {
    if (ch < nch) {
      bk.refresh_chunk(ch);
    } else {
      bk.cmax[ch] = 0;
      bk.cfirst[ch] = 0;
    }
  }
  big_sync<NW>();
  if (wid == 0) bk.refresh_top(lane);
  big_sync<NW>();
  int used = 0;
  while (used < max_it) {
    Key best = bk.tmax[lane];
    int k = bk.tfirst[lane];
    warp_first_max(best, k);
    if (best == 0) break;
    const int bb = x.pair(k);
    const int d0 = x.B0(bb), d1 = x.B1(bb);
    // the two bodies' lists
    int o0, l0, o1, l1;
    auto spans = [&]() {
      const int2 a = span[d0], b = d1 >= 0 ? span[d1] : make_int2(0, 0);
      o0 = a.x;
      l0 = a.y - a.x;
      o1 = b.x;
      l1 = b.y - b.x;
    };
    // this lane's contact of the two bodies' lists (32 at a time); one that
    // touches both bodies is visited in d0's list
    int q, qb;
    auto entry = [&](int e) {
      q = -1;
      qb = 0;
      if (e >= l0 + l1) return;
      q = e < l0 ? adj[o0 + e] : adj[o1 + e - l0];
      qb = x.pair(q);
      if (e >= l0 && (x.B0(qb) == d0 || x.B1(qb) == d0)) q = -1;
    };
    R lin, ang;
    if constexpr (NW > 1) {
      // every warp's contacts, eight at a time; the first warp's change
      const int first = 8 * wid + (lane >> 2);
      const bool lead = (lane & 3) == 0;
      std::conditional_t<VEL, VelocityIn<R>, PositionIn<R, W>> in;
      if (wid == 0) {
        if constexpr (VEL)
          velocity_load(x, in, k, bb, lane < 8, lane);
        else
          position_load(x, in, k, bb, lane < 8, lane);
      }
      spans();
      entry(first);
      if (q >= 0) prefetch_line(x.rec(q) + 16 * (lane & 1));
      if (wid == 0) {
        const bool woke = match_awake(x, bb, true, lane == 0);
        if constexpr (VEL)
          velocity_change<R, W, false>(x, v, in, k, lane < 8, lane, lin, ang, err);
        else
          position_change(x, v, in, bstart, lane < 8, lane, lin, ang);
        if (lane < 8) {
          chg->lin[lane] = lin;
          chg->ang[lane] = ang;
        }
        if (lane == 0) chg->woke = woke;
      }
      __syncthreads();
      lin = chg->lin[lane & 7];
      ang = chg->ang[lane & 7];
      const bool woke = chg->woke != 0;
      for (int base = 0; base < l0 + l1; base += 8 * NW) {
        if (base > 0) entry(base + first);
        if (base + 8 * wid < l0 + l1) {
          const R value = update_spread<VEL>(x, q < 0 ? 0 : q, qb, q >= 0, d0, d1, lin, ang, 32, woke);
          if (q >= 0 && lead) {
            bk.key[q] = key_of(value, (R)0.01);
            if (VEL) prefetch_line(x.krow(q));
          }
        }
      }
      const bool again = l0 + l1 > 8 * NW;
      __syncthreads();
      for (int base = 0; base < l0 + l1; base += 8 * NW) {
        if (again) entry(base + first);
        if (q >= 0 && lead) bk.refresh_chunk(q >> bk.shift);  // lanes of one chunk find the same
      }
      __syncthreads();
      for (int base = 0; base < l0 + l1; base += 8 * NW) {
        if (again) entry(base + first);
        if (q >= 0 && lead) bk.refresh_top(q >> bk.shift >> 4);
      }
      __syncthreads();
    } else {
      // what the change needs, then the touched records: they load while the
      // change is computed
      std::conditional_t<VEL, VelocityIn<R>, PositionIn<R, W>> in;
      if constexpr (VEL)
        velocity_load(x, in, k, bb, lane < 8, lane);
      else
        position_load(x, in, k, bb, lane < 8, lane);
      spans();
      entry(lane);
      Touched<R> t;
      update_load<VEL>(x, t, q, qb, q >= 0, d0, d1);
      const bool woke = match_awake(x, bb, true, lane == 0);
      if constexpr (VEL)
        velocity_change<R, W, false>(x, v, in, k, lane < 8, lane, lin, ang, err);
      else
        position_change(x, v, in, bstart, lane < 8, lane, lin, ang);
      for (int base = 0; base < l0 + l1; base += 32) {
        if (base > 0) {
          entry(base + lane);
          update_load<VEL>(x, t, q, qb, q >= 0, d0, d1);
        }
        const R value = update_apply<VEL>(x, t, lin, ang, 32, woke);
        if (t.valid) {
          bk.key[t.k] = key_of(value, (R)0.01);
          // the next contact to resolve is mostly one of these
          if (VEL) prefetch_line(x.krow(t.k));
        }
        __syncwarp();
        if (t.valid) bk.refresh_chunk(t.k >> bk.shift);  // lanes of one chunk find the same
        __syncwarp();
        if (t.valid) bk.refresh_top(t.k >> bk.shift >> 4);
        __syncwarp();
      }
    }
    ++used;
  }
  return used;
}

// One world of C contacts by its warps.  TILE: its per-contact arrays are in
// shared memory, which the compiler then knows (csm: their capacity).
template <class R, class W, bool TILE>
__device__ __forceinline__ void big_world(const BatchView<R>& v, R dt, int csm, int w, int C, unsigned char* smem) {
  using Key = decltype(key_of((R)0, (R)0));
  constexpr int T = kBigThreads;
  const int tid = threadIdx.x, lane = tid & 31;
  const int n = v.body_count[w];
  const int bstart = v.body_start[w];
  const long long cst = v.contact_start[w];
  BigKeys<Key> bk;
  bk.C = C;
  bk.shift = 4;
  while (((C - 1) >> bk.shift) >= kBigChunks) ++bk.shift;
  bk.cmax = reinterpret_cast<Key*>(smem);
  bk.tmax = bk.cmax + kBigChunks;
  bk.cfirst = reinterpret_cast<int*>(bk.tmax + kBigTops);
  bk.tfirst = bk.cfirst + kBigChunks;
  // list starts and ends (first the counts, then the fill cursors)
  int2* span = reinterpret_cast<int2*>(bk.tfirst + kBigTops);
  BigChange<R>* chg = reinterpret_cast<BigChange<R>*>(span + ((n + 3) & ~3));
  unsigned char* tile = reinterpret_cast<unsigned char*>(chg) + big_change_bytes<R>();
  RCtx<R, W, false> x;
  x.nbs = n;
  x.dt = dt;
  x.bw = reinterpret_cast<W*>(v.big_bw) + (long long)bstart * 7;
  x.br = v.big_br + (long long)bstart * BREC;
  x.aw = v.big_aw + bstart;
  x.cr = v.work + cst * CREC;
  x.gmat = v.uniform_material ? nullptr : v.contact + (long long)C_FRIC * v.nc_total + cst;
  x.gst = (long long)(C_REST - C_FRIC) * v.nc_total;
  x.delta = x.jw = nullptr;
  x.wi = nullptr;
  x.wst = x.jst = 0;
  x.kw = v.kmat + cst * K_ROW;
  int* adj;
  bk.padded = TILE;
  if (TILE) {
    bk.key = reinterpret_cast<Key*>(tile);
    x.cb = reinterpret_cast<int*>(bk.key + csm);
    adj = x.cb + csm;
  } else {
    bk.key = static_cast<Key*>(v.big_key) + cst;
    x.cb = v.work_bodies + cst;
    adj = v.big_adj + 2 * cst;
  }
  const bool awake = load_bodies(x, v, bstart, n, tid, T);
  x.all_awake = __syncthreads_and(awake) != 0;
  for (int k = tid; k < C; k += T) prepare_contact(x, v, cst + k, k, k);
  for (int i = tid; i < n; i += T) span[i].y = 0;
  __syncthreads();
  // contact lists per body: count, exclusive scan, fill
  for (int k = tid; k < C; k += T) {
    const int bb = x.pair(k);
    atomicAdd(&span[x.B0(bb)].y, 1);
    if (x.B1(bb) >= 0) atomicAdd(&span[x.B1(bb)].y, 1);
  }
  __syncthreads();
  int carry = 0;
  for (int base = 0; tid < 32 && base < n; base += 32) {
    const int i = base + lane;
    const int c = i < n ? span[i].y : 0;
    int s = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(FULL, s, d);
      if (lane >= d) s += y;
    }
    if (i < n) {
      span[i] = make_int2(carry + s - c, carry + s - c);
    }
    carry += __shfl_sync(FULL, s, 31);
  }
  __syncthreads();
  for (int k = tid; k < C; k += T) {
    const int bb = x.pair(k);
    adj[atomicAdd(&span[x.B0(bb)].y, 1)] = k;
    if (x.B1(bb) >= 0) adj[atomicAdd(&span[x.B1(bb)].y, 1)] = k;
  }
  __syncthreads();
  const int max_it = v.max_iterations >= 0 ? v.max_iterations : C * v.iter_mult;
  uint32_t err = 0;
  const bool solves = tid < 32 * big_warps<R>();
  const int pos_used = !solves ? 0 : big_phase<R, W, false>(x, v, bstart, bk, span, adj, max_it, chg, err);
  __syncthreads();
  if (v.contact_writeback)
    for (int k = tid; k < C; k += T) v.contact[C_PEN * v.nc_total + cst + k] = x.rec(k)[CR_PEN];
  for (int k = tid; k < C; k += T) friction_prepare(x, k);
  __syncthreads();
  const int vel_used = !solves ? 0 : big_phase<R, W, true>(x, v, bstart, bk, span, adj, max_it, chg, err);
  __syncthreads();
  if (err) {
    atomicOr(&v.world_status[w], err);
    atomicOr(v.status, err);
  }
  if (tid == 0) {
    v.pos_iters[w] = pos_used;
    v.vel_iters[w] = vel_used;
    atomicAdd(&v.counters[1], (unsigned long long)pos_used);
    atomicAdd(&v.counters[2], (unsigned long long)vel_used);
    atomicAdd(&v.counters[3], (unsigned long long)C);
  }
  if (v.contact_writeback)
    for (int k = tid; k < C; k += T) write_back_contact(x, v, cst, k);
  store_bodies(x, v, bstart, n, tid, T);
}

template <class R, class W>
__global__ void __launch_bounds__(kBigThreads, sizeof(R) == 8 ? 3 : 4) k_resolve_big(BatchView<R> v, R dt, int csm) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int w = v.big_list[blockIdx.x];
  int C = v.contact_count[w];
  if (C > v.contact_cap[w]) C = v.contact_cap[w];  // the world is already flagged ST_CAPACITY
  if (C <= 0 || dt <= (R)0) {                      // ResolveContacts guards, contact.go:210-212
    if (threadIdx.x == 0) {
      v.pos_iters[w] = 0;
      v.vel_iters[w] = 0;
      atomicAdd(&v.counters[3], (unsigned long long)C);
    }
  } else if (C <= csm && C <= 16 * kBigChunks) {
    big_world<R, W, true>(v, dt, csm, w, C, smem);
  } else {
    big_world<R, W, false>(v, dt, csm, w, C, smem);
  }
}

}  // namespace cz
