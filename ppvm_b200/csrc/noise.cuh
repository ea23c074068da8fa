// noise.cuh — the channels with one child per parent: amplitude damping and the loss channel
// (crates/ppvm-pauli-sum/src/sum/noise.rs:132-163, 165-181).
//
// The Heisenberg adjoint of amplitude damping on qubit q maps
//   I -> I,   X -> sqrt(1-g) X,   Y -> sqrt(1-g) Y,   Z -> (1-g) Z + g I,
// through map_insert (data.rs:204-226): a Z term (parent) is scaled in place and its child,
// the same word with I on q and coefficient v * g, is merged with `+=` into an existing term
// or appended after all terms, in parent order.  Unlike a rotation's child, this child can
// only land on a term with I on q, which is not a parent itself, so every key still receives
// at most two contributions and the result is bit-identical to the reference's.  The loss
// channel of a lossy sum has the same shape, with L in the place of Z:
//   L -> L + p I,   I, X, Y, Z -> (1-p) themselves.
//
//   k_branch_pair   every term with I or the parent letter on q meets its counterpart (the other of
//                   the two) in the epoch-tagged table, and the second to arrive hands each the
//                   other's coefficient, as k_rot_pair does for a rotation
//   k_branch_apply  every term scaled by its letter's factor; I terms add their parent's child; the
//                   children without a term appended, in parent order; its last block
//                   publishes the live count
//
// (A scan into records, an index of the children, a probe of every I term, an apply pass and a
// commit took five launches for damping, index, count and emit into the other planes three for the
// loss channel.  These are launches between dependent small passes: five layers of a noisy 7x7
// lattice take 11.8 ms instead of 12.1, four lossy layers on 40 qubits 6.1 instead of 7.4.)
// The capacity check runs in k_branch_apply before any coefficient changes, so a replay after
// growth starts from unmodified terms.
#pragma once

#include "kernels.cuh"

namespace ppvm {

// A channel on one qubit: word qw and bit of the qubit, word pw of the plane that tells the
// parent letter from I (damping: the Z plane's qw; loss: the X plane's loss word), and the factors.
struct Branch {
  uint64_t bit;
  uint32_t qw, pw;
  uint32_t loss;  // 1: loss channel (parents L), 0: amplitude damping (parents Z)
  // factors: the parent's own, its child's, an I term's, any other term's
  double parent, child, ident, other;
};

// Whether term i is touched (I or the parent letter on the qubit) and whether it is a parent.
__device__ __forceinline__ bool branch_touched(const Planes& P, const Branch& b, unsigned long long i, bool& parent) {
  const uint64_t x = P.x[(unsigned long long)b.qw * P.cap + i], z = P.z[(unsigned long long)b.qw * P.cap + i];
  parent = ((b.loss ? P.x[(unsigned long long)b.pw * P.cap + i] : z) & b.bit) != 0;
  return !((b.loss ? x | z : x) & b.bit);
}

template <int W>
__global__ void __launch_bounds__(256)
k_branch_pair(Planes P, Ctrl* ctrl, Branch b, unsigned long long* link, unsigned long long* table,
              unsigned long long table_cap, unsigned tepoch, int op) {
  pdl_wait();
  __shared__ unsigned s_cnt[2];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->rot_n = N;  // for the apply kernel
  if ((unsigned long long)blockIdx.x * blockDim.x >= N) return;
  if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long tsize = next_pow2_ull(N + N / 2 < 1024 ? 1024 : N + N / 2);
  if (tsize > table_cap) tsize = table_cap;
  const unsigned long long mask = tsize - 1;
  unsigned parents = 0, pairs = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    bool parent;
    if (!branch_touched(P, b, i, parent)) continue;
    uint64_t x[W], z[W], kx[W], kz[W];
    load_key<W>(P, i, x, z);
#pragma unroll
    for (int w = 0; w < W; ++w) {  // they meet at the key with I
      const uint64_t m = w == (int)b.pw ? b.bit : 0ull;
      kx[w] = x[w] & ~(b.loss ? m : 0ull);
      kz[w] = z[w] & ~(b.loss ? 0ull : m);
    }
    parents += parent;
    const uint64_t h = table_hash<W>(kx, kz);
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
        for (int w = 0; w < W; ++w) {
          const uint64_t m = w == (int)b.pw ? b.bit : 0ull;
          eq &= (jx[w] == (x[w] ^ (b.loss ? m : 0ull))) & (jz[w] == (z[w] ^ (b.loss ? 0ull : m)));
        }
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

template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_branch_apply(Planes P, Ctrl* ctrl, Branch b, unsigned long long* link, unsigned long long* ts, unsigned epoch,
               int op, OpLog* log) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  if (ld_volatile_int(&ctrl->err)) return;
  // as in k_rot_apply: the blocks that take part follow from a count that the commit below leaves alone
  const unsigned long long N = ld_volatile(&ctrl->rot_n);
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
    bool touched[ITEMS], parent[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      if (i < N) {
        touched[k] = branch_touched(P, b, i, parent[k]);
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
        // a factor of 1 leaves every value as it is
        double nc = __dmul_rn(kc[k], !touched[k] ? b.other : parent[k] ? b.parent : b.ident);
        if (touched[k] && parent[k]) child = !linked;
        else if (linked) nc = __dadd_rn(nc, __dmul_rn(__longlong_as_double((long long)kl[k]), b.child));
        P.c[i] = nc;
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
            if (w == (int)b.pw) (b.loss ? x : z)[w] &= ~b.bit;
          store_key<W>(P, r, x, z);
          P.c[r] = __dmul_rn(kc[k], b.child);
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
