// kernels.cuh — the hot-path kernels of the Pauli-propagation engine (sm_100a).
//
// Rotation exp(-i theta/2 G) on a sum held in SoA planes, reference semantics of
// PauliSum::map_insert (crates/ppvm-pauli-sum/src/sum/data.rs:204-226):
//   k_rot_pair   partner search: each anticommuting term inserts one of K, K^G into an
//                epoch-tagged table; the second of a pair to arrive links both (a child K^G can
//                only collide with its partner term, so every key receives at most two
//                contributions)
//   k_rot_apply  parent <- c*cos (+ partner's c*(eps*sin)); partnerless parents append their
//                child in parent order, so the term order stays the reference's IndexMap order;
//                its last block publishes the new live count
// Clifford runs (sum/clifford.rs) and diagonal noise (sum/noise.rs) are one in-place pass
// (k_clifford); truncation (data.rs:275-311, strategy.rs) is an in-place stable compaction.
#pragma once

#include "common.cuh"

namespace ppvm {

constexpr unsigned kNone = 0xFFFFFFFFu;

template <int W>
__device__ __forceinline__ void load_key(const Planes& P, unsigned long long i, uint64_t (&x)[W],
                                         uint64_t (&z)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    x[w] = P.x[(unsigned long long)w * P.cap + i];
    z[w] = P.z[(unsigned long long)w * P.cap + i];
  }
}
template <int W>
__device__ __forceinline__ void store_key(const Planes& P, unsigned long long i,
                                          const uint64_t (&x)[W], const uint64_t (&z)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    P.x[(unsigned long long)w * P.cap + i] = x[w];
    P.z[(unsigned long long)w * P.cap + i] = z[w];
  }
}
// Dense record of an anticommuting term: [x0..x(W-1), z0..z(W-1), coeff bits].
template <int W>
__device__ __forceinline__ void load_rec(const uint64_t* rec, unsigned long long s, uint64_t (&x)[W],
                                         uint64_t (&z)[W], double& c) {
  const uint64_t* r = rec + s * (2 * W + 1);
#pragma unroll
  for (int w = 0; w < W; ++w) x[w] = r[w];
#pragma unroll
  for (int w = 0; w < W; ++w) z[w] = r[W + w];
  c = __longlong_as_double((long long)r[2 * W]);
}

// The generator as it acts on the term with X words x: on a lossy sum (g.lw != 0) it skips
// the term's lost qubits, which is the reference's loss fallback of rotate_2
// (crates/ppvm-pauli-sum/src/sum/rot2.rs:26-33) extended to any support: a lost qubit has
// x = z = 0, so the anticommutation test and the sign are those of the full generator and only
// the child's bits differ.
template <int W>
__device__ __forceinline__ void gen_on(const Gen& g, const uint64_t (&x)[W], uint64_t (&gx)[W],
                                       uint64_t (&gz)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint64_t lost = 0;
#pragma unroll
    for (int v = 0; v < W; ++v)
      if (g.lw && v == w + (int)g.lw) lost = x[v];
    gx[w] = g.gx[w] & ~lost;
    gz[w] = g.gz[w] & ~lost;
  }
}

template <int W>
struct ItemsFor {
  // terms per thread of a look-back tile: small enough that a sum of 10^5..10^6 terms
  // spreads over a few tiles per SM (a 256-thread tile holds 256 * ITEMS terms)
  static constexpr int value = W <= 2 ? 4 : (W <= 4 ? 2 : 1);
};

// ---------------------------------------------------------------------------------------
// Rotations.  Both kernels read the terms in place: a term's anticommutation test needs only the
// generator's words, so a term that commutes costs those words and nothing is copied aside.
// (Copying the anticommuting terms into dense records first, as an ordered compaction of its
// own, and committing in a fourth kernel made a gate four launches and moved about 3 (16W + 8)
// bytes more per anticommuting term.)
// ---------------------------------------------------------------------------------------

// The words of term i that a rotation by g needs (word masks: xm of the X plane, zm of the Z
// plane); the others are zero.
template <int W>
__device__ __forceinline__ void load_words(const Planes& P, unsigned long long i, unsigned xm, unsigned zm,
                                           uint64_t (&x)[W], uint64_t (&z)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    x[w] = (xm >> w) & 1u ? P.x[(unsigned long long)w * P.cap + i] : 0ull;
    z[w] = (zm >> w) & 1u ? P.z[(unsigned long long)w * P.cap + i] : 0ull;
  }
}

// link[i]: the bits of the coefficient of term i's partner, or kNoLink.  kNoLink is a NaN that no
// arithmetic makes; a coefficient that is that very NaN is linked as another NaN.
constexpr unsigned long long kNoLink = ~0ull;
__device__ __forceinline__ unsigned long long link_bits(double c) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(c);
  return b == kNoLink ? kNoLink - 1 : b;
}

// k_rot_pair: finds, for each anticommuting term, whether its partner K^G is also present.  The
// term inserts its index at the one of K and K^G without the generator's first bit (on a lossy
// sum, whose terms each see their own part of the generator: the smaller) in an epoch-tagged
// table; the second of a pair to arrive hands each the other's coefficient in link[] (all kNoLink between rotations: k_rot_apply
// clears the links it reads), so that the apply pass reads and writes nothing at random.
// xmask/zmask: the words of the X/Z plane that the test reads.
// Bound by the random 8-byte table accesses: one thread per term at full occupancy keeps as many
// in flight as the SMs can hold.
template <int W>
__global__ void __launch_bounds__(256)
k_rot_pair(Planes P, Ctrl* ctrl, Gen g, unsigned xmask, unsigned zmask, unsigned long long* link,
           unsigned long long* table, unsigned long long table_cap, unsigned tepoch, int op) {
  pdl_wait();
  __shared__ unsigned s_cnt[2];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->rot_n = N;  // for the apply kernel
  if ((unsigned long long)blockIdx.x * blockDim.x >= N) return;
  if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  // at most N entries: full to 2/3 when every term anticommutes and none has a partner
  unsigned long long tsize = next_pow2_ull(N + N / 2 < 1024 ? 1024 : N + N / 2);
  if (tsize > table_cap) tsize = table_cap;
  const unsigned long long mask = tsize - 1;
  // the generator's first bit: word cw of the X plane (cx) or of the Z plane, mask cm
  int cw = 0;
  bool cx = false;
  uint64_t cm = 0;
#pragma unroll
  for (int w = W - 1; w >= 0; --w)
    if (g.gx[w] | g.gz[w]) {
      cw = w;
      cx = g.gx[w] != 0;
      cm = cx ? g.gx[w] : g.gz[w];
    }
  cm &= ~cm + 1;
  unsigned mine_s = 0, mine_p = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    uint64_t x[W], z[W], px[W], pz[W];
    load_words<W>(P, i, xmask, zmask, x, z);
    if (!anticommutes<W>(g, x, z)) continue;
    ++mine_s;
    load_key<W>(P, i, x, z);
    gen_on<W>(g, x, px, pz);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      px[w] ^= x[w];
      pz[w] ^= z[w];
    }
    bool use_p;
    if (g.lw) {
      use_p = key_less<W>(px, pz, x, z);
    } else {  // of the two keys, the one without the generator's first bit
      uint64_t b = 0;
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (w == cw) b = cx ? x[w] : z[w];
      use_p = b & cm;
    }
    uint64_t rx[W], rz[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      rx[w] = use_p ? px[w] : x[w];
      rz[w] = use_p ? pz[w] : z[w];
    }
    const uint64_t h = table_hash<W>(rx, rz);
    const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
    const unsigned long long mine = make_slot(tepoch, tag, (unsigned)i);
    unsigned long long slot = h & mask;
    unsigned long long probes = 0;
    while (true) {
      unsigned long long cur = ld_volatile(&table[slot]);
      if (slot_epoch(cur) != (tepoch & 0xFFFFu)) {
        const unsigned long long prev = atomicCAS(&table[slot], cur, mine);
        if (prev == cur) break;  // inserted; the partner (if any) will find us
        continue;                // slot was taken meanwhile: examine it again
      }
      if (slot_tag(cur) == tag) {
        const unsigned j = slot_idx(cur);
        uint64_t jx[W], jz[W];
        load_key<W>(P, j, jx, jz);
        // j is our partner iff its key is exactly K ^ G
        bool eq = true;
#pragma unroll
        for (int w = 0; w < W; ++w) eq &= (jx[w] == px[w]) & (jz[w] == pz[w]);
        if (eq) {
          link[i] = link_bits(P.c[j]);
          link[j] = link_bits(P.c[i]);
          ++mine_p;
          break;
        }
      }
      slot = (slot + 1) & mask;
      if (++probes > tsize) {
        set_err(ctrl, kErrProbe, op);
        break;
      }
    }
  }
  mine_s = __reduce_add_sync(kFull, mine_s);
  mine_p = __reduce_add_sync(kFull, mine_p);
  if ((threadIdx.x & 31) == 0) {
    if (mine_s) atomicAdd(&s_cnt[0], mine_s);
    if (mine_p) atomicAdd(&s_cnt[1], mine_p);
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_cnt[threadIdx.x])
    atomicAdd(threadIdx.x == 0 ? &ctrl->rot_s : &ctrl->rot_pairs, (unsigned long long)s_cnt[threadIdx.x]);
}

// k_rot_apply: new coefficients in place, children appended in parent order (one decoupled
// look-back per tile of terms).  xmask/zmask: the test's words, gm: the words of the generator (of
// both planes; the sign needs them).  The last of the blocks that have tiles publishes the
// live count.  Which blocks have tiles follows from the count the pair kernel saw (rot_n), not from
// the live one: a block that starts after the commit (the grid can be larger than what is resident
// at once) would take the new count's tiles for its own.  A late block may also read rot_s after its
// reset: then there are no tiles, and block 0 alone, which is never late, takes part.
// A streaming pass: every access but the appended children is at the term itself.
template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_rot_apply(Planes P, Ctrl* ctrl, Gen g, unsigned xmask, unsigned zmask, unsigned gm, double sn, double cs,
            unsigned long long* link, unsigned long long* ts, unsigned epoch, int op, OpLog* log) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->rot_n);
  const unsigned long long ns = ld_volatile(&ctrl->rot_s);
  const unsigned long long nchild = ns - 2 * ld_volatile(&ctrl->rot_pairs);
  if (N + nchild > P.cap) {  // nothing has been written: the host grows the storage and replays this op
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctrl->cap_needed = N + nchild;
      set_err(ctrl, kErrCapacity, op);
    }
    return;
  }
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned long long ntiles = ns == 0 ? 0 : (N + TILE - 1) / TILE;
  const unsigned blocks = (unsigned)(ntiles < 1 ? 1 : ntiles < gridDim.x ? ntiles : gridDim.x);
  if (blockIdx.x >= blocks) return;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  while (ntiles) {
    const unsigned tile = next_tile(&ctrl->tickets[1], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    // loads of all the thread's terms first, stores after them
    unsigned ballots[ITEMS], bits[ITEMS];  // 1: anticommutes, 2: eps of its child is +1, 4: eps of its partner's
    double kc[ITEMS];
    unsigned long long kl[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      bits[k] = 0;
      if (i < N) {
        uint64_t x[W], z[W];
        load_words<W>(P, i, xmask, zmask, x, z);
        bits[k] = anticommutes<W>(g, x, z);
      }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      if (bits[k]) {
        uint64_t x[W], z[W], ex[W], ez[W];
        load_words<W>(P, i, gm, gm, x, z);
        kl[k] = link[i];
        kc[k] = P.c[i];
        if (rot_sign<W>(g, x, z) > 0.0) bits[k] |= 2u;
        gen_on<W>(g, x, ex, ez);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          x[w] ^= ex[w];
          z[w] ^= ez[w];
        }
        if (rot_sign<W>(g, x, z) > 0.0) bits[k] |= 4u;
      }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      const bool child = bits[k] && kl[k] == kNoLink;
      if (bits[k]) {
        double nc = __dmul_rn(kc[k], cs);
        if (!child) {
          const double eps_j = bits[k] & 4u ? 1.0 : -1.0;
          nc = __dadd_rn(nc, __dmul_rn(__longlong_as_double((long long)kl[k]), eps_j * sn));
          link[i] = kNoLink;
        }
        P.c[i] = nc;
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
          uint64_t x[W], z[W], ex[W], ez[W];
          load_key<W>(P, i, x, z);
          gen_on<W>(g, x, ex, ez);
#pragma unroll
          for (int w = 0; w < W; ++w) {
            x[w] ^= ex[w];
            z[w] ^= ez[w];
          }
          store_key<W>(P, r, x, z);
          P.c[r] = __dmul_rn(kc[k], (bits[k] & 2u ? 1.0 : -1.0) * sn);
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

// ---------------------------------------------------------------------------------------
// Truncation: keep iff !(|c| < thr) and weight <= maxw (CombinedStrategy order does not
// matter for the kept set).  Dropped terms whose key is preserved are collected in order
// and re-appended after the kept ones (data.rs:283-310).  In place: a tile publishes its
// aggregate only after loading all of its terms, and writes go to positions <= its reads.
// ---------------------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ bool preserved(const uint64_t (&x)[W], const uint64_t (&z)[W],
                                          const uint64_t* pres_keys, const int* pres_table,
                                          unsigned pres_mask) {
  unsigned long long slot = hash_key<W>(x, z) & pres_mask;
  for (unsigned probe = 0; probe <= pres_mask; ++probe) {
    const int j = pres_table[slot];
    if (j < 0) return false;
    const uint64_t* k = pres_keys + (unsigned long long)j * 2 * W;
    bool eq = true;
#pragma unroll
    for (int w = 0; w < W; ++w) eq &= (k[w] == x[w]) & (k[W + w] == z[w]);
    if (eq) return true;
    slot = (slot + 1) & pres_mask;
  }
  return false;
}

template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_truncate(Planes P, Ctrl* ctrl, double thr, unsigned long long maxw, const uint64_t* pres_keys,
           const int* pres_table, unsigned pres_mask, int npres, uint64_t* side,
           unsigned long long* ts, unsigned epoch, int op, OpLog* log, unsigned long long maxlw, unsigned lw) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  __shared__ unsigned s_base2[ITEMS * (BLOCK / 32) + 1];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned long long ntiles = (N + TILE - 1) / TILE;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    log[op].n_in = N;
    if (N == 0) {
      ctrl->n_s = 0;
      ctrl->n_side = 0;
    }
  }
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  const bool wcap = maxw != ~0ull;
  for (;;) {
    const unsigned tile = next_tile(&ctrl->tickets[2], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    uint64_t kx[ITEMS][W], kz[ITEMS][W];
    double kc[ITEMS];
    unsigned keep_b[ITEMS], side_b[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      bool keep = false, sd = false;
      if (i < N) {
        load_key<W>(P, i, kx[k], kz[k]);
        kc[k] = P.c[i];
        keep = !(fabs(kc[k]) < thr);
        if (wcap) keep = keep && (weight<W>(kx[k], kz[k]) <= maxw);
        if (lw && maxlw != ~0ull) {  // MaxLossWeight: lost qubits, the X plane's upper words
          unsigned lost = 0;
#pragma unroll
          for (int w = 0; w < W; ++w)
            if (w >= (int)lw) lost += __popcll(kx[k][w]);
          keep = keep && lost <= maxlw;
        }
        if (!keep && npres > 0) sd = preserved<W>(kx[k], kz[k], pres_keys, pres_table, pres_mask);
      }
      keep_b[k] = __ballot_sync(kFull, keep);
      side_b[k] = __ballot_sync(kFull, sd);
    }
    const unsigned agg = tile_ranks<BLOCK, ITEMS>(keep_b, s_base);
    const unsigned agg2 = npres > 0 ? tile_ranks<BLOCK, ITEMS>(side_b, s_base2) : 0u;
    const unsigned long long packed = (unsigned long long)agg | ((unsigned long long)agg2 << 32);
    const unsigned long long excl = lookback(ts, tile, packed, epoch, ctrl, op, &s_slot);
    const unsigned long long kexcl = excl & 0xFFFFFFFFull, sexcl = excl >> 32;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned lt = (1u << lane) - 1u;
      if ((keep_b[k] >> lane) & 1u) {
        const unsigned long long r = kexcl + s_base[k * NW + warp] + __popc(keep_b[k] & lt);
        store_key<W>(P, r, kx[k], kz[k]);
        P.c[r] = kc[k];
      }
      if ((side_b[k] >> lane) & 1u) {
        const unsigned long long r = sexcl + s_base2[k * NW + warp] + __popc(side_b[k] & lt);
        uint64_t* rec = side + r * (2 * W + 1);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          rec[w] = kx[k][w];
          rec[W + w] = kz[k][w];
        }
        rec[2 * W] = (uint64_t)__double_as_longlong(kc[k]);
      }
    }
    if (tile == ntiles - 1 && threadIdx.x == 0) {
      ctrl->n_s = kexcl + agg;
      ctrl->n_side = sexcl + agg2;
    }
  }
}

// Appends the preserved-but-dropped terms after the kept ones and publishes the count.
template <int W>
__global__ void k_commit_truncate(Planes P, Ctrl* ctrl, const uint64_t* side, int op, OpLog* log) {
  pdl_wait();
  if (threadIdx.x == 0 && blockIdx.x == 0)
    for (int t = 0; t < 4; ++t) ctrl->tickets[t] = 0;
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long kept = ctrl->n_s, nside = ctrl->n_side;
  for (unsigned long long j = threadIdx.x; j < nside; j += blockDim.x) {
    uint64_t x[W], z[W];
    double c;
    load_rec<W>(side, j, x, z, c);
    store_key<W>(P, kept + j, x, z);
    P.c[kept + j] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->n = kept + nside;
    log[op].n_out = kept + nside;
    log[op].n_s = ctrl->n_s;
  }
}

// ---------------------------------------------------------------------------------------
// Clifford runs and diagonal channels: one in-place pass applying a list of local ops.
// ---------------------------------------------------------------------------------------
enum CliffCode : uint32_t {
  C_X = 0, C_Y, C_Z, C_H, C_S, C_SDAG, C_SQX, C_SQXDAG, C_SQY, C_SQYDAG,
  C_CNOT, C_CZ, C_CY,
  C_PAULI_ERROR, C_DEP1, C_DEP2,
  C_ROTC,  // Clifford-angle rotation on 1-2 qubits: axis bits in ax/az, sign of sin in f0
  C_PERR2  // two-qubit Pauli error: factor table f0 (16 doubles each) of the launch's tables
};

struct DevOp {
  uint32_t code;
  uint16_t w0, b0, w1, b1;
  uint16_t ax, az;  // bit0: qubit0, bit1: qubit1 (axis of C_ROTC)
  uint16_t two;
  uint16_t lw;      // lossy sums: first loss word of the X plane (two-qubit ops skip lost qubits)
  double f0, f1, f2;
};

constexpr int kMaxOpsPerLaunch = 256;
constexpr int kCliffBlock = 128;

template <int W, int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_clifford(Planes P, Ctrl* ctrl, const DevOp* ops, int nops, int op0, OpLog* log,
           const double* __restrict__ perr2) {
  pdl_wait();
  __shared__ DevOp s_ops[kMaxOpsPerLaunch];
  __shared__ uint64_t s_x[W][BLOCK];
  __shared__ uint64_t s_z[W][BLOCK];
  if (ld_volatile_int(&ctrl->err)) return;
  for (int o = threadIdx.x; o < nops; o += BLOCK) s_ops[o] = ops[o];
  __syncthreads();
  const unsigned long long N = ld_volatile(&ctrl->n);
  if (blockIdx.x == 0 && threadIdx.x == 0 && log) {
    for (int o = 0; o < nops; ++o) {
      log[op0 + o].n_in = N;
      log[op0 + o].n_s = N;
      log[op0 + o].n_new = 0;
      log[op0 + o].n_out = N;
    }
  }
  const unsigned t = threadIdx.x;
  for (unsigned long long i = (unsigned long long)blockIdx.x * BLOCK + t; i < N;
       i += (unsigned long long)gridDim.x * BLOCK) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      s_x[w][t] = P.x[(unsigned long long)w * P.cap + i];
      s_z[w][t] = P.z[(unsigned long long)w * P.cap + i];
    }
    double c = P.c[i];
    bool neg = false;
    for (int o = 0; o < nops; ++o) {
      const DevOp& d = s_ops[o];
      const uint64_t m0 = 1ull << d.b0, m1 = 1ull << d.b1;
      uint64_t x0w = s_x[d.w0][t], z0w = s_z[d.w0][t];
      const bool x0 = x0w & m0, z0 = z0w & m0;
      // lossy sums: which of the op's qubits are lost.  One-qubit ops need no test (a lost
      // qubit has x = z = 0, which every one-qubit rule leaves alone); two-qubit Cliffords,
      // depolarize2 and the two-qubit Pauli error skip the term (phase/clifford.rs:77,92,168;
      // noise.rs:98-102,122); a Clifford-angle rotation acts on the qubits that are not lost.
      bool l0 = false, l1 = false;
      if (d.lw) {
        const bool skip2 = d.code == C_CNOT || d.code == C_CZ || d.code == C_CY || d.code == C_DEP2 ||
                           d.code == C_PERR2;
        l0 = s_x[d.lw + d.w0][t] & m0;
        l1 = (skip2 || (d.code == C_ROTC && d.two)) ? (bool)(s_x[d.lw + d.w1][t] & m1) : false;
        if ((l0 || l1) && skip2) continue;
      }
      switch (d.code) {
        case C_X: neg ^= z0; break;
        case C_Y: neg ^= x0 ^ z0; break;
        case C_Z: neg ^= x0; break;
        case C_H:
          neg ^= x0 & z0;
          s_x[d.w0][t] = (x0w & ~m0) | (z0 ? m0 : 0);
          s_z[d.w0][t] = (z0w & ~m0) | (x0 ? m0 : 0);
          break;
        case C_S: neg ^= x0 & !z0; s_z[d.w0][t] = z0w ^ (x0 ? m0 : 0); break;
        case C_SDAG: neg ^= x0 & z0; s_z[d.w0][t] = z0w ^ (x0 ? m0 : 0); break;
        case C_SQX: neg ^= x0 & z0; s_x[d.w0][t] = x0w ^ (z0 ? m0 : 0); break;
        case C_SQXDAG: neg ^= !x0 & z0; s_x[d.w0][t] = x0w ^ (z0 ? m0 : 0); break;
        case C_SQY:
          neg ^= !x0 & z0;
          s_x[d.w0][t] = (x0w & ~m0) | (z0 ? m0 : 0);
          s_z[d.w0][t] = (z0w & ~m0) | (x0 ? m0 : 0);
          break;
        case C_SQYDAG:
          neg ^= x0 & !z0;
          s_x[d.w0][t] = (x0w & ~m0) | (z0 ? m0 : 0);
          s_z[d.w0][t] = (z0w & ~m0) | (x0 ? m0 : 0);
          break;
        case C_CNOT: case C_CZ: case C_CY: {
          const bool xc = x0, zc = z0;
          const bool xt = s_x[d.w1][t] & m1, zt = s_z[d.w1][t] & m1;
          bool nzc = zc, nxt = xt, nzt = zt;
          if (d.code == C_CNOT) {
            neg ^= xc & zt & (xt == zc);
            nzc = zc ^ zt;
            nxt = xt ^ xc;
          } else if (d.code == C_CZ) {
            neg ^= xc & xt & (zc ^ zt);
            nzc = zc ^ xt;
            nzt = zt ^ xc;
          } else {
            neg ^= xc & (xt ^ zt) & !(zc ^ zt);
            nzc = zc ^ xt ^ zt;
            nxt = xt ^ xc;
            nzt = zt ^ xc;
          }
          s_z[d.w0][t] = (s_z[d.w0][t] & ~m0) | (nzc ? m0 : 0);
          s_x[d.w1][t] = (s_x[d.w1][t] & ~m1) | (nxt ? m1 : 0);
          s_z[d.w1][t] = (s_z[d.w1][t] & ~m1) | (nzt ? m1 : 0);
          break;
        }
        case C_PAULI_ERROR: {
          const int code = (int)x0 | ((int)z0 << 1);
          if (code == 1) c = __dmul_rn(c, d.f0);
          else if (code == 2) c = __dmul_rn(c, d.f1);
          else if (code == 3) c = __dmul_rn(c, d.f2);
          break;
        }
        case C_DEP1: if (x0 | z0) c = __dmul_rn(c, d.f0); break;
        case C_PERR2: {  // factor of (P_q0, P_q1), code x | z << 1 on each qubit
          const bool x1 = s_x[d.w1][t] & m1, z1 = s_z[d.w1][t] & m1;
          const int code = ((int)x0 | ((int)z0 << 1)) << 2 | (int)x1 | ((int)z1 << 1);
          if (code) c = __dmul_rn(c, perr2[16 * (int)d.f0 + code]);
          break;
        }
        case C_DEP2: {
          const bool x1 = s_x[d.w1][t] & m1, z1 = s_z[d.w1][t] & m1;
          if (x0 | z0 | x1 | z1) c = __dmul_rn(c, d.f0);
          break;
        }
        case C_ROTC: {
          const bool ax0 = (d.ax & 1) && !l0, az0 = (d.az & 1) && !l0;
          bool x1 = false, z1 = false, ax1 = false, az1 = false;
          if (d.two) {
            x1 = s_x[d.w1][t] & m1;
            z1 = s_z[d.w1][t] & m1;
            ax1 = ((d.ax >> 1) & 1) && !l1;
            az1 = ((d.az >> 1) & 1) && !l1;
          }
          const bool anti = ((x0 & az0) ^ (z0 & ax0)) ^ ((x1 & az1) ^ (z1 & ax1));
          if (!anti) break;
          // phase of G*P per qubit (see rot_sign)
          auto g1 = [](bool gx, bool gz, bool px, bool pz) -> int {
            if (gx & !gz) return (px & pz) ? 1 : ((!px & pz) ? -1 : 0);
            if (gx & gz) return (!px & pz) ? 1 : ((px & !pz) ? -1 : 0);
            if (!gx & gz) return (px & !pz) ? 1 : ((px & pz) ? -1 : 0);
            return 0;
          };
          const int e = g1(ax0, az0, x0, z0) + g1(ax1, az1, x1, z1);
          const double eps = (((e + 1) & 3) == 0) ? 1.0 : -1.0;
          neg ^= (eps * d.f0) < 0.0;
          if (ax0) s_x[d.w0][t] ^= m0;
          if (az0) s_z[d.w0][t] ^= m0;
          if (d.two) {
            if (ax1) s_x[d.w1][t] ^= m1;
            if (az1) s_z[d.w1][t] ^= m1;
          }
          break;
        }
        default: break;
      }
    }
#pragma unroll
    for (int w = 0; w < W; ++w) {
      P.x[(unsigned long long)w * P.cap + i] = s_x[w][t];
      P.z[(unsigned long long)w * P.cap + i] = s_z[w][t];
    }
    P.c[i] = neg ? -c : c;
  }
}

// ---------------------------------------------------------------------------------------
// Reductions (deterministic: fixed element->thread map and fixed trees).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ double block_sum(double v, double* s_red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(kFull, v, o));
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (unsigned w = 0; w < blockDim.x / 32; ++w) r = __dadd_rn(r, s_red[w]);
  }
  __syncthreads();
  return r;
}

// Sum of coefficients of words without X bits: trace("Z?*") = overlap_with_zero.
template <int W>
__global__ void __launch_bounds__(256) k_owz(Planes P, const Ctrl* ctrl, double* partials) {
  pdl_wait();
  __shared__ double s_red[8];
  const unsigned long long N = ld_volatile(&ctrl->n);
  double acc = 0.0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    uint64_t any = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) any |= P.x[(unsigned long long)w * P.cap + i];
    if (any == 0) acc = __dadd_rn(acc, P.c[i]);
  }
  const double b = block_sum(acc, s_red);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
}

static __global__ void k_sum_partials(const double* partials, int n, Ctrl* ctrl) {
  pdl_wait();
  __shared__ double s_red[8];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc = __dadd_rn(acc, partials[i]);
  const double b = block_sum(acc, s_red);
  if (threadIdx.x == 0) ctrl->sum = b;
}

// PauliPattern matcher (crates/ppvm-pauli-word/src/pattern/contains.rs:120-151).
struct PatItem {
  uint32_t kind;    // 0 = Position, 1 = Star, 2 = Repeat
  uint32_t accept;  // bit c set if Pauli code c (0=I 1=X 2=Z 3=Y) is accepted
  uint64_t arg;
};

// First qubit at or after pos whose bit in m is clear; n if there is none below n.
template <int W>
__device__ __forceinline__ unsigned first_clear(const uint64_t (&m)[W], unsigned pos, unsigned n) {
  unsigned r = n;
#pragma unroll
  for (int w = W - 1; w >= 0; --w) {
    uint64_t c = ~m[w];
    if ((int)(pos >> 6) == w) c &= ~0ull << (pos & 63);
    if (w >= (int)(pos >> 6) && c) r = w * 64 + (unsigned)__ffsll((long long)c) - 1;
  }
  return r < n ? r : n;
}

// Whether the word matches the pattern (items in order, then only I).  The qubits an item accepts
// are one mask per word, and a step over a stretch of them is one search for a clear bit: the
// cost is per item, not per qubit.  x, z: the qubits' words (wr of them on a lossy sum, whose
// lost qubits, lost[], match no item; crates/ppvm-pauli-word/src/pattern/contains.rs:25-41).
template <int W>
__device__ bool pattern_match(const PatItem* items, int nitems, unsigned n, const uint64_t (&x)[W],
                              const uint64_t (&z)[W], const uint64_t (&lost)[W]) {
  unsigned pos = 0;
  uint64_t id[W];  // qubits that hold I
#pragma unroll
  for (int w = 0; w < W; ++w) id[w] = ~(x[w] | z[w] | lost[w]);
  for (int it = 0; it < nitems; ++it) {
    const PatItem p = items[it];
    uint64_t acc[W];
#pragma unroll
    for (int w = 0; w < W; ++w)
      acc[w] = ((p.accept & 1u ? id[w] : 0ull) | (p.accept & 2u ? x[w] & ~z[w] : 0ull) |
                (p.accept & 4u ? ~x[w] & z[w] : 0ull) | (p.accept & 8u ? x[w] & z[w] : 0ull)) & ~lost[w];
    if (p.kind == 0) {  // I up to qubit arg, which is accepted
      if (p.arg < pos || p.arg >= n || first_clear<W>(id, pos, n) < p.arg) return false;
      const unsigned q = (unsigned)p.arg;
      if (first_clear<W>(acc, q, n) == q) return false;
      pos = q + 1;
    } else {
      const unsigned to = first_clear<W>(acc, pos, n);
      if (p.kind == 1) {
        pos = to;
      } else if (p.arg == 0) {  // takes the accepted stretch; fails if that reaches the end
        if (to == n && to != pos) return false;
        pos = to;
      } else {
        if (to - pos < p.arg) return false;
        pos += (unsigned)p.arg;
      }
    }
  }
  return first_clear<W>(id, pos, n) == n;
}

template <int W>
__global__ void __launch_bounds__(256)
k_trace(Planes P, const Ctrl* ctrl, const PatItem* items, int nitems, unsigned nq, double* partials,
        unsigned lw) {
  __shared__ double s_red[8];
  const unsigned long long N = ld_volatile(&ctrl->n);
  double acc = 0.0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    uint64_t x[W], z[W];
    load_key<W>(P, i, x, z);
    uint64_t lost[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      lost[w] = 0ull;
#pragma unroll
      for (int v = 0; v < W; ++v)
        if (lw && v == w + (int)lw) lost[w] = x[v];
    }
    if (pattern_match<W>(items, nitems, nq, x, z, lost)) acc = __dadd_rn(acc, P.c[i]);
  }
  const double b = block_sum(acc, s_red);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
}

template <int W>
__global__ void __launch_bounds__(256) k_weights(Planes P, const Ctrl* ctrl, uint32_t* out) {
  const unsigned long long N = ld_volatile(&ctrl->n);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    uint64_t x[W], z[W];
    load_key<W>(P, i, x, z);
    out[i] = weight<W>(x, z);
  }
}

// The largest weight into *out (0 before the launch).
template <int W>
__global__ void __launch_bounds__(256) k_max_weight(Planes P, const Ctrl* ctrl, unsigned long long* out) {
  const unsigned long long N = ld_volatile(&ctrl->n);
  unsigned m = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    uint64_t x[W], z[W];
    load_key<W>(P, i, x, z);
    m = max(m, weight<W>(x, z));
  }
  m = __reduce_max_sync(kFull, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, (unsigned long long)m);
}

// ---------------------------------------------------------------------------------------
// Key index (cold paths: construction `+=`, overlap, equality).  table slot -> term index.
// ---------------------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ void index_insert(const Planes& P, unsigned long long i,
                                             unsigned long long* table, unsigned long long mask,
                                             unsigned tepoch, Ctrl* ctrl) {
  uint64_t x[W], z[W];
  load_key<W>(P, i, x, z);
  const uint64_t h = table_hash<W>(x, z);
  const unsigned long long mine = make_slot(tepoch, (unsigned)(h >> 48), (unsigned)i);
  unsigned long long slot = h & mask;
  for (unsigned long long probe = 0; probe <= mask; ++probe) {
    const unsigned long long cur = ld_volatile(&table[slot]);
    if (slot_epoch(cur) != (tepoch & 0xFFFFu)) {
      const unsigned long long prev = atomicCAS(&table[slot], cur, mine);
      if (prev == cur) return;
      continue;
    }
    slot = (slot + 1) & mask;
  }
  set_err(ctrl, kErrProbe, -1);
}

template <int W>
__device__ __forceinline__ long long index_find(const Planes& P, const uint64_t (&x)[W],
                                                const uint64_t (&z)[W], const unsigned long long* table,
                                                unsigned long long mask, unsigned tepoch) {
  const uint64_t h = table_hash<W>(x, z);
  const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
  unsigned long long slot = h & mask;
  for (unsigned long long probe = 0; probe <= mask; ++probe) {
    const unsigned long long cur = table[slot];
    if (slot_epoch(cur) != (tepoch & 0xFFFFu)) return -1;
    if (slot_tag(cur) == tag) {
      uint64_t jx[W], jz[W];
      load_key<W>(P, slot_idx(cur), jx, jz);
      bool eq = true;
#pragma unroll
      for (int w = 0; w < W; ++w) eq &= (jx[w] == x[w]) & (jz[w] == z[w]);
      if (eq) return slot_idx(cur);
    }
    slot = (slot + 1) & mask;
  }
  return -1;
}

template <int W>
__global__ void __launch_bounds__(256)
k_build_index(Planes P, Ctrl* ctrl, unsigned long long* table, unsigned long long mask, unsigned tepoch) {
  const unsigned long long N = ld_volatile(&ctrl->n);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x)
    index_insert<W>(P, i, table, mask, tepoch, ctrl);
}

// `ps += (word, c)` for k new terms, strictly in order (one thread): existing key -> c += v,
// new key -> append (crates/ppvm-traits/src/map/hashmap.rs:40-44).
template <int W>
__global__ void k_add_terms_seq(Planes P, Ctrl* ctrl, const uint64_t* nx, const uint64_t* nz,
                                const double* nc, unsigned long long k, unsigned long long* table,
                                unsigned long long mask, unsigned tepoch) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  unsigned long long N = ctrl->n;
  for (unsigned long long t = 0; t < k; ++t) {
    uint64_t x[W], z[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      x[w] = nx[t * W + w];
      z[w] = nz[t * W + w];
    }
    const long long j = index_find<W>(P, x, z, table, mask, tepoch);
    if (j >= 0) {
      P.c[j] = __dadd_rn(P.c[j], nc[t]);
    } else {
      if (N >= P.cap) {
        set_err(ctrl, kErrCapacity, -1);
        return;
      }
      store_key<W>(P, N, x, z);
      P.c[N] = nc[t];
      index_insert<W>(P, N, table, mask, tepoch, ctrl);
      ++N;
    }
  }
  ctrl->n = N;
}

// sum over b's terms of b[k] * a[k] (a indexed by `table`), per-block partials.
template <int W>
__global__ void __launch_bounds__(256)
k_overlap(Planes A, Planes B, const Ctrl* bctrl, const unsigned long long* table,
          unsigned long long mask, unsigned tepoch, double* partials, unsigned long long* mismatch) {
  __shared__ double s_red[8];
  const unsigned long long NB = ld_volatile(&bctrl->n);
  double acc = 0.0;
  unsigned miss = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < NB;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    uint64_t x[W], z[W];
    load_key<W>(B, i, x, z);
    const long long j = index_find<W>(A, x, z, table, mask, tepoch);
    const double bv = B.c[i];
    if (j >= 0) {
      acc = __dadd_rn(acc, __dmul_rn(bv, A.c[j]));
      if (!(A.c[j] == bv)) ++miss;
    } else {
      acc = __dadd_rn(acc, __dmul_rn(bv, 0.0));
      ++miss;
    }
  }
  const double b = block_sum(acc, s_red);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  // one count per warp: an atomic per thread on the one word cost more than the lookups
  miss = __reduce_add_sync(kFull, miss);
  if ((threadIdx.x & 31) == 0 && miss) atomicAdd(mismatch, (unsigned long long)miss);
}

}  // namespace ppvm
