// noise.cuh — amplitude damping (crates/ppvm-pauli-sum/src/sum/noise.rs:132-163).
//
// The Heisenberg adjoint of amplitude damping on qubit q maps
//   I -> I,   X -> sqrt(1-g) X,   Y -> sqrt(1-g) Y,   Z -> (1-g) Z + g I,
// through map_insert (data.rs:204-226): a Z term (parent) is scaled in place and its child,
// the same word with I on q and coefficient v * g, is merged with `+=` into an existing term
// or appended after all terms, in parent order.  Unlike a rotation's child, this child can
// only land on a term with I on q, which is not a parent itself, so every key still receives
// at most two contributions and the result is bit-identical to the reference's.
//
//   k_damp_pair   every term with I or Z on q meets its counterpart (the other of the two) in the
//                 epoch-tagged table, and the second to arrive hands each the other's
//                 coefficient, as k_rot_pair does for a rotation
//   k_damp_apply  parents scaled by (1-g), I terms add their parent's child, X and Y scaled by
//                 sqrt(1-g); the children without a term appended, in parent order; its last
//                 block publishes the live count
//
// (A scan into records, an index of the children, a probe of every I term, an apply pass and a
// commit took five launches: 45 us on a sum of 75,000 terms, against 20 for the two.)  The
// capacity check runs in k_damp_apply before any coefficient changes, so a replay after growth
// starts from unmodified terms.
#pragma once

#include "kernels.cuh"

namespace ppvm {

// qw, bit: the plane word and bit of the damped qubit.
template <int W>
__global__ void __launch_bounds__(256)
k_damp_pair(Planes P, Ctrl* ctrl, unsigned qw, uint64_t bit, unsigned long long* link, unsigned long long* table,
            unsigned long long table_cap, unsigned tepoch, int op) {
  pdl_wait();
  __shared__ unsigned s_cnt[2];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  if ((unsigned long long)blockIdx.x * blockDim.x >= N) return;
  if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long tsize = next_pow2_ull(N + N / 2 < 1024 ? 1024 : N + N / 2);
  if (tsize > table_cap) tsize = table_cap;
  const unsigned long long mask = tsize - 1;
  unsigned parents = 0, pairs = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    if (P.x[(unsigned long long)qw * P.cap + i] & bit) continue;  // X or Y
    uint64_t x[W], z[W], kz[W];
    load_key<W>(P, i, x, z);
    bool parent = false;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const uint64_t m = w == (int)qw ? bit : 0ull;
      parent |= (z[w] & m) != 0;
      kz[w] = z[w] & ~m;  // they meet at the key with I
    }
    parents += parent;
    const uint64_t h = table_hash<W>(x, kz);
    const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
    const unsigned long long mine = make_slot(tepoch, tag, (unsigned)i);
    unsigned long long slot = h & mask, probes = 0, cur = ld_volatile(&table[slot]);
    while (true) {
      if (slot_epoch(cur) != (tepoch & 0xFFFFu)) {
        const unsigned long long prev = atomicCAS(&table[slot], cur, mine);
        if (prev == cur) break;
        cur = prev;  // taken meanwhile: examine what is there now
        continue;
      }
      if (slot_tag(cur) == tag) {
        const unsigned j = slot_idx(cur);
        uint64_t jx[W], jz[W];
        load_key<W>(P, j, jx, jz);
        bool eq = true;
#pragma unroll
        for (int w = 0; w < W; ++w) eq &= (jx[w] == x[w]) & (jz[w] == (z[w] ^ (w == (int)qw ? bit : 0ull)));
        if (eq) {
          link[i] = link_bits(P.c[j]);
          link[j] = link_bits(P.c[i]);
          ++pairs;
          break;
        }
      }
      slot = (slot + 1) & mask;
      if (++probes > tsize) {
        set_err(ctrl, kErrProbe, op);
        break;
      }
      cur = ld_volatile(&table[slot]);
    }
  }
  parents = __reduce_add_sync(kFull, parents);
  pairs = __reduce_add_sync(kFull, pairs);
  if ((threadIdx.x & 31) == 0) {
    if (parents) atomicAdd(&s_cnt[0], parents);
    if (pairs) atomicAdd(&s_cnt[1], pairs);
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_cnt[threadIdx.x])
    atomicAdd(threadIdx.x == 0 ? &ctrl->rot_s : &ctrl->rot_pairs, (unsigned long long)s_cnt[threadIdx.x]);
}

// om = 1 - g, gm = g, sxy = sqrt(1 - g).
template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_damp_apply(Planes P, Ctrl* ctrl, unsigned qw, uint64_t bit, double om, double gm, double sxy,
             unsigned long long* link, unsigned long long* ts, unsigned epoch, int op, OpLog* log) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  const unsigned long long ns = ld_volatile(&ctrl->rot_s);
  const unsigned long long nchild = ns - ld_volatile(&ctrl->rot_pairs);
  if (N + nchild > P.cap) {  // nothing has been written: the host grows the storage and replays this op
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctrl->cap_needed = N + nchild;
      set_err(ctrl, kErrCapacity, op);
    }
    return;
  }
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned long long ntiles = (N + TILE - 1) / TILE;
  const unsigned blocks = (unsigned)(ntiles < 1 ? 1 : ntiles < gridDim.x ? ntiles : gridDim.x);
  if (blockIdx.x >= blocks) return;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  while (ntiles) {
    const unsigned tile = next_tile(&ctrl->tickets[1], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    unsigned ballots[ITEMS];
    double kc[ITEMS];
    unsigned long long kl[ITEMS];
    bool xy[ITEMS], zz[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      if (i < N) {
        xy[k] = (P.x[(unsigned long long)qw * P.cap + i] & bit) != 0;
        zz[k] = (P.z[(unsigned long long)qw * P.cap + i] & bit) != 0;
        kl[k] = link[i];
        kc[k] = P.c[i];
      }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      bool child = false;
      if (i < N) {
        const bool linked = kl[k] != kNoLink;
        if (xy[k]) {
          P.c[i] = __dmul_rn(kc[k], sxy);
        } else if (zz[k]) {
          P.c[i] = __dmul_rn(kc[k], om);
          child = !linked;
        } else if (linked) {
          P.c[i] = __dadd_rn(kc[k], __dmul_rn(__longlong_as_double((long long)kl[k]), gm));
        }
        if (linked) link[i] = kNoLink;
      }
      ballots[k] = __ballot_sync(kFull, child);
    }
    if (nchild) {
      const unsigned agg = tile_ranks<BLOCK, ITEMS>(ballots, s_base);
      const unsigned long long excl = lookback(ts, tile, agg, epoch, ctrl, op, &s_slot);
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        if ((ballots[k] >> lane) & 1u) {
          const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
          const unsigned long long r =
              N + excl + s_base[k * NW + warp] + __popc(ballots[k] & ((1u << lane) - 1u));
          uint64_t x[W], z[W];
          load_key<W>(P, i, x, z);
#pragma unroll
          for (int w = 0; w < W; ++w)
            if (w == (int)qw) z[w] &= ~bit;
          store_key<W>(P, r, x, z);
          P.c[r] = __dmul_rn(kc[k], gm);
        }
      }
    }
  }
  if (last_of_blocks(&ctrl->done, blocks) && threadIdx.x == 0) {
    for (int t = 0; t < 4; ++t) ctrl->tickets[t] = 0;
    ctrl->rot_s = ctrl->rot_pairs = 0;
    if (ld_volatile_int(&ctrl->err)) return;
    log[op].n_in = N;
    log[op].n_s = ns;
    log[op].n_new = nchild;
    log[op].n_out = N + nchild;
    ctrl->n = N + nchild;
  }
}

}  // namespace ppvm
