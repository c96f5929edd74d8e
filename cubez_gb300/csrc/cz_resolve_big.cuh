// ResolveContacts (contact.go:204-445) for worlds whose bodies do not fit the
// shared-memory slot of k_resolve (hundreds to thousands of bodies).
//
// One warp per world: such a world is mostly one island, so its iterations are
// one chain, and what counts is the latency of an iteration.
//   * Body and contact records are in global memory (L1/L2); a record is two
//     cache lines at most, where rows took a line per value.
//   * The argmax is over chunk maxima in shared memory (at most kBigChunks),
//     kept by refreshing the chunks of the contacts an iteration changed,
//     instead of a scan over every contact's value.
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

// shared memory ahead of the per-contact arrays: chunk maxima and their first
// contacts, list starts and ends of n bodies
template <class R> __host__ __device__ inline size_t big_fixed_bytes(int n) {
  return (size_t)kBigChunks * (sizeof(R) + sizeof(int)) + (size_t)2 * ((n + 3) & ~3) * sizeof(int);
}
// per contact: key, packed bodies, two list entries
template <class R> __host__ __device__ constexpr size_t big_contact_bytes() { return sizeof(R) + 3 * sizeof(int); }

// The chunk maxima of a world's keys and the first contact holding each.
template <class Key> struct BigKeys {
  Key* key;     // [C]
  Key* cmax;    // [kBigChunks]
  int* cfirst;  // [kBigChunks]
  int C, shift;  // chunk of contact k: k >> shift
  // the chunk's first maximum again, by one lane
  __device__ __forceinline__ void refresh(int ch) const {
    const int k0 = ch << shift, k1 = min(C, k0 + (1 << shift));
    Key best = 0;
    int at = k0;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      const Key q = key[k];
      if (q > best) {
        best = q;
        at = k;
      }
    }
    cmax[ch] = best;
    cfirst[ch] = at;
  }
};

// adjustPositions (VEL false) or adjustVelocities (VEL true) of one world by
// its warp; returns the iterations used.
template <class R, class W, bool VEL, class Key>
__device__ __forceinline__ int big_phase(const RCtx<R, W, false>& x, const BatchView<R>& v, int bstart,
                                         const BigKeys<Key>& bk, const int* off, const int* end, const int* adj,
                                         int max_it, uint32_t& err) {
  const int lane = threadIdx.x;
  const int C = bk.C;
  const int nch = (C + (1 << bk.shift) - 1) >> bk.shift;
  for (int k = lane; k < C; k += 32) bk.key[k] = key_of(x.rec(k)[VEL ? CR_DDV : CR_PEN], (R)0.01);
  __syncwarp();
  for (int ch = lane; ch < nch; ch += 32) bk.refresh(ch);
  __syncwarp();
  int used = 0;
  while (used < max_it) {
    Key best = 0;
    int ch = 0x7fffffff;
    for (int c = lane; c < nch; c += 32) {
      const Key q = bk.cmax[c];
      if (q > best) {
        best = q;
        ch = c;
      }
    }
    warp_first_max(best, ch);
    if (best == 0) break;
    const int k = bk.cfirst[ch];
    const int bb = x.pair(k);
    const int d0 = x.B0(bb), d1 = x.B1(bb);
    const int o0 = off[d0], l0 = end[d0] - o0;
    const int o1 = d1 >= 0 ? off[d1] : 0, l1 = d1 >= 0 ? end[d1] - o1 : 0;
    // this lane's contact of the two bodies' lists (32 at a time); one that
    // touches both bodies is visited in d0's list
    auto entry = [&](int e) {
      if (e >= l0 + l1) return -1;
      const int q = e < l0 ? adj[o0 + e] : adj[o1 + e - l0];
      if (e >= l0) {
        const int qb = x.pair(q);
        if (x.B0(qb) == d0 || x.B1(qb) == d0) return -1;
      }
      return q;
    };
    // its record loads while the resolved contact's change is computed
    Touched<R> t;
    const int q = entry(lane);
    update_load<VEL>(x, t, q, q >= 0, d0, d1);
    const bool woke = match_awake(x, bb, true, lane == 0);
    R lin, ang;
    if constexpr (VEL)
      velocity_change<R, W, false>(x, v, k, lane < 8, lane, lin, ang, err);
    else
      position_change(x, v, bstart, k, lane < 8, lane, lin, ang);
    for (int base = 0; base < l0 + l1; base += 32) {
      if (base > 0) {
        const int r = entry(base + lane);
        update_load<VEL>(x, t, r, r >= 0, d0, d1);
      }
      const R value = update_apply<VEL>(x, t, lin, ang, 32, woke);
      if (t.valid) bk.key[t.k] = key_of(value, (R)0.01);
      __syncwarp();
      if (t.valid) bk.refresh(t.k >> bk.shift);  // lanes of one chunk find the same
      __syncwarp();
    }
    ++used;
  }
  return used;
}

template <class R, class W>
__global__ void __launch_bounds__(32, 4) k_resolve_big(BatchView<R> v, R dt, int csm) {
  using Key = decltype(key_of((R)0, (R)0));
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x;
  const int w = v.big_list[blockIdx.x];
  const int n = v.body_count[w];
  const int bstart = v.body_start[w];
  const long long cst = v.contact_start[w];
  int C = v.contact_count[w];
  if (C > v.contact_cap[w]) C = v.contact_cap[w];  // the world is already flagged ST_CAPACITY
  if (C <= 0 || dt <= (R)0) {                      // ResolveContacts guards, contact.go:210-212
    if (lane == 0) {
      v.pos_iters[w] = 0;
      v.vel_iters[w] = 0;
      atomicAdd(&v.counters[3], (unsigned long long)C);
    }
    return;
  }
  BigKeys<Key> bk;
  bk.C = C;
  bk.shift = 4;
  while (((C - 1) >> bk.shift) >= kBigChunks) ++bk.shift;
  bk.cmax = reinterpret_cast<Key*>(smem);
  bk.cfirst = reinterpret_cast<int*>(bk.cmax + kBigChunks);
  // list starts and ends (first the counts, then the fill cursors)
  int* off = bk.cfirst + kBigChunks;
  int* end = off + ((n + 3) & ~3);
  unsigned char* tile = reinterpret_cast<unsigned char*>(end + ((n + 3) & ~3));
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
  if (C <= csm) {
    bk.key = reinterpret_cast<Key*>(tile);
    x.cb = reinterpret_cast<int*>(bk.key + csm);
    adj = x.cb + csm;
  } else {
    bk.key = static_cast<Key*>(v.big_key) + cst;
    x.cb = v.work_bodies + cst;
    adj = v.big_adj + 2 * cst;
  }
  x.all_awake = __all_sync(FULL, load_bodies(x, v, bstart, n, lane, 32));
  __syncwarp();
  for (int k = lane; k < C; k += 32) prepare_contact(x, v, cst + k, k, k);
  for (int i = lane; i < n; i += 32) end[i] = 0;
  __syncwarp();
  // contact lists per body: count, exclusive scan, fill
  for (int k = lane; k < C; k += 32) {
    const int bb = x.pair(k);
    atomicAdd(&end[x.B0(bb)], 1);
    if (x.B1(bb) >= 0) atomicAdd(&end[x.B1(bb)], 1);
  }
  __syncwarp();
  int carry = 0;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const int c = i < n ? end[i] : 0;
    int s = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(FULL, s, d);
      if (lane >= d) s += y;
    }
    if (i < n) {
      off[i] = carry + s - c;
      end[i] = carry + s - c;
    }
    carry += __shfl_sync(FULL, s, 31);
  }
  __syncwarp();
  for (int k = lane; k < C; k += 32) {
    const int bb = x.pair(k);
    adj[atomicAdd(&end[x.B0(bb)], 1)] = k;
    if (x.B1(bb) >= 0) adj[atomicAdd(&end[x.B1(bb)], 1)] = k;
  }
  __syncwarp();
  const int max_it = v.max_iterations >= 0 ? v.max_iterations : C * v.iter_mult;
  uint32_t err = 0;
  const int pos_used = big_phase<R, W, false>(x, v, bstart, bk, off, end, adj, max_it, err);
  __syncwarp();
  if (v.contact_writeback)
    for (int k = lane; k < C; k += 32) v.contact[C_PEN * v.nc_total + cst + k] = x.rec(k)[CR_PEN];
  for (int k = lane; k < C; k += 32) friction_prepare(x, k);
  __syncwarp();
  const int vel_used = big_phase<R, W, true>(x, v, bstart, bk, off, end, adj, max_it, err);
  __syncwarp();
  if (err) {
    atomicOr(&v.world_status[w], err);
    atomicOr(v.status, err);
  }
  if (lane == 0) {
    v.pos_iters[w] = pos_used;
    v.vel_iters[w] = vel_used;
    atomicAdd(&v.counters[1], (unsigned long long)pos_used);
    atomicAdd(&v.counters[2], (unsigned long long)vel_used);
    atomicAdd(&v.counters[3], (unsigned long long)C);
  }
  if (v.contact_writeback)
    for (int k = lane; k < C; k += 32) write_back_contact(x, v, cst, k);
  store_bodies(x, v, bstart, n, lane, 32);
}

}  // namespace cz
