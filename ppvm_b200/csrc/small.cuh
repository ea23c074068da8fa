// small.cuh — op lists on small sums: one CTA, one launch, the sum in shared memory.
//
// A sum of a few hundred terms leaves the GPU idle, and every kernel of the per-op pipelines is then
// a few microseconds of launch and memory latency: a 20-qubit Trotter chain of 410 ops took
// 2.2 ms for at most 900 terms, a single-gate call 40 us.  k_small interprets the list in one CTA
// (cta.cuh), at block-barrier cost per op, as long as the terms fit into shared memory.  An op
// that would outgrow it, or one it does not know, ends the launch before anything of that op
// is written; the host goes on from there with the pipelines, which are the faster from about
// that size on (they spread over all SMs).
//
// Every op gives the pipelines' terms, coefficients and order: rotations, damping, Cliffords,
// diagonal noise and TRUNCATE keep the reference's IndexMap order; a fused run (rotations on
// distinct qubits, RX or RZ, in a sum without exact order) is applied gate by gate and its
// terms are then sorted as the fused run writes them: untouched terms in order, then the
// groups by their first member, members by coordinate (runs.cuh).
#pragma once

#include "cta.cuh"
#include "runs.cuh"

namespace ppvm {

constexpr int kSmallBlock = 512;
constexpr int kSmallItems = 4;
constexpr int kSmallOps = 2048;                  // ops per launch
// Sums of more terms take the pipelines at once.  200 rotations on a closed sum, interpreter / pipelines:
// 450 terms 525 / 1704 us on 20 qubits, 880 / 2408 on 400.  Above 512 it would still be the faster on a sum
// that stays as it is (900 terms, 20 qubits: 1178 / 2708), but not where the region holds 1024
// terms (900 terms, 400 qubits: 3018 / 2814, as it is left and entered in vain), and a sum that grows
// leaves it after a few ops.
constexpr unsigned long long kSmallStart = 512;
// A head of fewer ops before one that the interpreter does not take (a long stretch of local ops, a
// two-qubit Pauli error) is left to the pipelines.  Interpreting it would pay from about 4 ops on (16
// rotations before 100 Cliffords, 20 qubits, 20 terms: 88 / 147 us); the line is a safe one.
constexpr size_t kSmallHead = 64;
// Longer stretches of local ops go to the composed Clifford pass, whose cost hardly depends on their
// length.  Six stretches of k ops between rotations, 300 terms, interpreter / pipelines: 150 qubits, k = 48
// 208 / 248 us, k = 64 248 / 264; 400 qubits, k = 48 297 / 294, k = 64 408 / 301.
constexpr int small_local(int W) { return W <= 4 ? 64 : 48; }

// Terms the region holds: as many as fit into shared memory with the pair table and the sort keys.
template <int W>
struct SmallFor {
  static constexpr unsigned cap = W <= 3 ? 2048 : 1024;
  static constexpr size_t smem = 8 * ((size_t)(2 * W + 2) * cap + cap / 2 + 2 * cap) + 8 * (size_t)cap;
};

enum SKind : uint32_t { S_ROT = 0, S_LOCAL, S_TRUNC, S_DAMP };

struct alignas(8) SmallOp {
  DevOp d;       // qubits, axes; local ops: code and factors
  uint32_t kind;
  uint32_t run;  // gates of the fused run that starts here (0: none starts)
  double a, b, c;  // rotation: sin, cos; damping: gamma, 1 - gamma, sqrt(1 - gamma)
};

// Up to this many ops travel as a kernel argument instead of an upload (a single-gate call).
constexpr int kSmallInline = 4;
struct SmallInline {
  SmallOp op[kSmallInline];
};

// A rotation (DAMP: amplitude damping) with the reference's semantics on N <= BLOCK * ITEMS terms:
// thread t owns terms t, t + BLOCK, ... throughout, so nothing is listed, and three barriers
// separate linking the pairs, ranking the children and using the results.  Returns the new size, or
// more than the region holds, with no term changed.
template <int W, bool DAMP>
__device__ __forceinline__ unsigned small_rotate(const Region<W>& R, const SmallOp& op, unsigned N, unsigned epoch,
                                                 unsigned* s_base, int& perr) {
  constexpr int BLOCK = kSmallBlock, ITEMS = kSmallItems, NW = BLOCK / 32;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const DevOp d = op.d;
  const unsigned long long mask = R.tsize - 1;
  unsigned bits = 0;  // per item, 4 bits: touched, eps of the child is +1, eps of the partner's is +1; DAMP: touched, Z
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const unsigned i = k * BLOCK + threadIdx.x;
    if (i >= N) continue;
    bool x0, z0, x1, z1;
    term_bits<W>(R, d, i, x0, z0, x1, z1);
    if constexpr (DAMP) {
      if (x0) continue;
      bits |= (1u | (unsigned)z0 << 1) << (4 * k);
    } else {
      const RotBits rb = rot_bits(d, x0, z0, x1, z1);
      if (!rb.anti) continue;
      const RotBits pb = rot_bits(d, x0 ^ (bool)(d.ax & 1), z0 ^ (bool)(d.az & 1), x1 ^ (d.two && (d.ax & 2)),
                                  z1 ^ (d.two && (d.az & 2)));
      bits |= (1u | (unsigned)rb.eps_plus << 1 | (unsigned)pb.eps_plus << 2) << (4 * k);
    }
    uint64_t x[W], z[W], px[W], pz[W], kx[W], kz[W];
    rload<W>(R, i, x, z);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      px[w] = x[w];
      pz[w] = z[w];
    }
    if constexpr (DAMP) wflip<W>(pz, d.w0, 1ull << d.b0);
    else flip_gen<W>(d, px, pz);
    const bool use_p = (!DAMP && (d.ax & 1)) ? x0 : z0;  // meet at the key without the flipped bit on q0
#pragma unroll
    for (int w = 0; w < W; ++w) {
      kx[w] = use_p ? px[w] : x[w];
      kz[w] = use_p ? pz[w] : z[w];
    }
    const uint64_t h = table_hash<W>(kx, kz);
    const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
    const unsigned long long me = make_slot(epoch, tag, i);
    unsigned long long slot = h & mask, probes = 0, cur = ld_volatile(&R.table[slot]);
    while (true) {
      if (slot_epoch(cur) != (epoch & 0xFFFFu)) {
        const unsigned long long prev = atomicCAS(&R.table[slot], cur, me);
        if (prev == cur) break;
        cur = prev;
        continue;
      }
      if (slot_tag(cur) == tag) {
        const unsigned j = slot_idx(cur);
        uint64_t jx[W], jz[W];
        rload<W>(R, j, jx, jz);
        bool eq = true;
#pragma unroll
        for (int w = 0; w < W; ++w) eq &= (jx[w] == px[w]) & (jz[w] == pz[w]);
        if (eq) {
          R.link[i] = link_word(R.c[j]);
          R.link[j] = link_word(R.c[i]);
          break;
        }
      }
      slot = (slot + 1) & mask;
      if (++probes > mask) {
        perr = 1;  // cannot happen: twice as many slots as terms
        break;
      }
      cur = ld_volatile(&R.table[slot]);
    }
  }
  if (!__syncthreads_or(bits != 0)) {
    if constexpr (!DAMP) return N;
  }
  unsigned bal[ITEMS];
  unsigned long long lw[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const unsigned b = bits >> (4 * k);
    lw[k] = b & 1u ? R.link[k * BLOCK + threadIdx.x] : 0ull;
    bal[k] = __ballot_sync(kFull, (b & 1u) && lw[k] == 0ull && (!DAMP || (b & 2u)));
  }
  const unsigned made = tile_ranks<BLOCK, ITEMS>(bal, s_base);
  if (N + made > (unsigned)R.cap || perr) return (unsigned)R.cap + 1;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const unsigned i = k * BLOCK + threadIdx.x, b = bits >> (4 * k);
    if (b & 1u) {
      const double c = R.c[i], lc = __longlong_as_double((long long)~lw[k]);
      double nc, cc;
      if constexpr (DAMP) {
        cc = __dmul_rn(c, op.a);
        nc = b & 2u ? __dmul_rn(c, op.b) : lw[k] ? __dadd_rn(c, __dmul_rn(lc, op.a)) : c;
      } else {
        cc = __dmul_rn(c, (b & 2u ? 1.0 : -1.0) * op.a);
        nc = __dmul_rn(c, op.b);
        if (lw[k]) nc = __dadd_rn(nc, __dmul_rn(lc, (b & 4u ? 1.0 : -1.0) * op.a));
      }
      if (lw[k]) R.link[i] = 0ull;
      R.c[i] = nc;
      if ((bal[k] >> lane) & 1u) {
        const unsigned pos = N + s_base[k * NW + warp] + __popc(bal[k] & lt);
        uint64_t x[W], z[W];
        rload<W>(R, i, x, z);
        if constexpr (DAMP) wflip<W>(z, d.w0, 1ull << d.b0);
        else flip_gen<W>(d, x, z);
        rstore<W>(R, pos, x, z);
        R.c[pos] = cc;
      }
    } else if (DAMP && i < N) {  // X or Y
      R.c[i] = __dmul_rn(R.c[i], op.c);
    }
  }
  __syncthreads();
  return N + made;
}

// The run's qubits, and whether every group fits the fused run (at most kRunMaxK coordinates).
template <int W>
__device__ __forceinline__ bool small_run_begin(const Region<W>& R, unsigned N, const SmallOp* ops, unsigned len,
                                                bool rx, unsigned long long* s_q, uint64_t (&Q)[W]) {
  __syncthreads();
  if (threadIdx.x < W) s_q[threadIdx.x] = 0ull;
  __syncthreads();
  for (unsigned j = threadIdx.x; j < len; j += kSmallBlock) atomicOr(&s_q[ops[j].d.w0], 1ull << ops[j].d.b0);
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) Q[w] = s_q[w];
  bool wide = false;
  for (unsigned i = threadIdx.x; i < N; i += kSmallBlock) {
    unsigned k = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) k += __popcll((rx ? R.z : R.x)[(size_t)w * R.cap + i] & Q[w]);
    wide |= k > (unsigned)kRunMaxK;
  }
  return !__syncthreads_or(wide);
}

// The sum's terms after the gates of a run that began with N0 terms, sorted as the fused run writes
// them.  The original terms still hold indices below N0 (gates only append), so a group's
// first member is the smallest of them with the group's key.
template <int W>
__device__ __forceinline__ void small_run_sort(const Region<W>& R, unsigned N0, unsigned N, bool rx,
                                               const uint64_t (&Q)[W], unsigned epoch, unsigned long long* key) {
  const unsigned long long mask = R.tsize - 1;
  const uint64_t* V = rx ? R.z : R.x;
  const uint64_t* F = rx ? R.x : R.z;
  auto group = [&](unsigned i, uint64_t (&v)[W], uint64_t (&f)[W]) {
    unsigned k = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      v[w] = V[(size_t)w * R.cap + i];
      f[w] = F[(size_t)w * R.cap + i] & ~(v[w] & Q[w]);
      k += __popcll(v[w] & Q[w]);
    }
    return k;
  };
  // the slot of a group holds the smallest index seen of it
  for (unsigned i = threadIdx.x; i < N0; i += kSmallBlock) {
    uint64_t v[W], f[W];
    if (group(i, v, f) == 0) continue;
    const uint64_t h = table_hash<W>(v, f);
    const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
    const unsigned long long me = make_slot(epoch, tag, i);
    unsigned long long slot = h & mask, cur = ld_volatile(&R.table[slot]);
    for (unsigned long long probes = 0; probes <= mask;) {
      if (slot_epoch(cur) != (epoch & 0xFFFFu)) {
        const unsigned long long prev = atomicCAS(&R.table[slot], cur, me);
        if (prev == cur) break;
        cur = prev;
        continue;
      }
      if (slot_tag(cur) == tag) {
        uint64_t jv[W], jf[W];
        group(slot_idx(cur), jv, jf);
        bool eq = true;
#pragma unroll
        for (int w = 0; w < W; ++w) eq &= (jv[w] == v[w]) & (jf[w] == f[w]);
        if (eq) {
          atomicMin(&R.table[slot], me);  // same epoch and tag: the smaller index
          break;
        }
      }
      slot = (slot + 1) & mask;
      ++probes;
      cur = ld_volatile(&R.table[slot]);
    }
  }
  __syncthreads();
  unsigned n2 = 1;
  while (n2 < N) n2 <<= 1;
  // sort keys: untouched by index; touched after them by (first member, coordinate); the term's
  // index below
  for (unsigned i = threadIdx.x; i < n2; i += kSmallBlock) {
    unsigned long long k = ~0ull;
    if (i < N) {
      uint64_t v[W], f[W];
      unsigned hi = i;
      if (group(i, v, f)) {
        const uint64_t h = table_hash<W>(v, f);
        const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
        unsigned long long slot = h & mask;
        unsigned first = 0;
        for (unsigned long long probes = 0; probes <= mask; ++probes) {  // found: the group has an original member
          const unsigned long long cur = R.table[slot];
          if (slot_epoch(cur) != (epoch & 0xFFFFu)) break;
          if (slot_tag(cur) == tag) {
            uint64_t jv[W], jf[W];
            group(slot_idx(cur), jv, jf);
            bool eq = true;
#pragma unroll
            for (int w = 0; w < W; ++w) eq &= (jv[w] == v[w]) & (jf[w] == f[w]);
            if (eq) {
              first = slot_idx(cur);
              break;
            }
          }
          slot = (slot + 1) & mask;
        }
        unsigned c = 0, t = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const uint64_t fw = F[(size_t)w * R.cap + i];
          uint64_t m = v[w] & Q[w];
          while (m) {
            const int b = __ffsll((long long)m) - 1;
            c |= (unsigned)((fw >> b) & 1ull) << t;
            ++t;
            m &= m - 1;
          }
        }
        hi = 1u << 30 | first << kRunMaxK | c;
      }
      k = (unsigned long long)hi << 32 | i;
    }
    key[i] = k;
  }
  __syncthreads();
  for (unsigned size = 2; size <= n2; size <<= 1)
    for (unsigned d = size >> 1; d; d >>= 1) {
      for (unsigned e = threadIdx.x; e < n2 / 2; e += kSmallBlock) {
        const unsigned a = ((e & ~(d - 1)) << 1) | (e & (d - 1)), b = a | d;
        const unsigned long long ka = key[a], kb = key[b];
        if ((ka > kb) == ((a & size) == 0)) {
          key[a] = kb;
          key[b] = ka;
        }
      }
      __syncthreads();
    }
  // every term to its place (all reads before all writes)
  constexpr int PER = (int)(SmallFor<W>::cap / kSmallBlock);
  uint64_t x[PER][W], z[PER][W];
  double c[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const unsigned i = u * kSmallBlock + threadIdx.x;
    if (i < N) {
      const unsigned from = (unsigned)key[i];
      rload<W>(R, from, x[u], z[u]);
      c[u] = R.c[from];
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const unsigned i = u * kSmallBlock + threadIdx.x;
    if (i < N) {
      rstore<W>(R, i, x[u], z[u]);
      R.c[i] = c[u];
    }
  }
  __syncthreads();
}

// ops: the list in device memory, or null for the ops in `few`.  log and host: the op log and the
// control block in the host's own (pinned) memory, written directly, so that a call needs no copy
// back.
template <int W>
__global__ void __launch_bounds__(kSmallBlock)
k_small(Planes P, Ctrl* ctrl, const SmallOp* __restrict__ ops, const SmallInline few, unsigned nops, int op0,
        double thr, unsigned long long maxw, OpLog* log, Ctrl* host) {
  pdl_wait();
  constexpr int BLOCK = kSmallBlock, ITEMS = kSmallItems, NW = BLOCK / 32;
  __shared__ unsigned s_base[ITEMS * NW + 1];
  __shared__ unsigned long long s_or[2 * W];
  __shared__ int s_perr;
  __shared__ unsigned long long s_q[W];
  // the ops from index s0 on: an op read from global memory would cost its latency each time
  constexpr unsigned OPS = 64;
  __shared__ SmallOp s_ops[OPS];
  static_assert(kSmallInline <= OPS, "the ops in few fit the buffer");
  if (!ops && threadIdx.x == 0)
    for (unsigned o = 0; o < nops; ++o) s_ops[o] = few.op[o];
  unsigned s0 = 0;
  auto fetch = [&](unsigned at) {
    __syncthreads();
    if (!ops) return;
    s0 = at;
    const unsigned n = min(OPS, nops - at) * (unsigned)(sizeof(SmallOp) / 8);
    for (unsigned t = threadIdx.x; t < n; t += BLOCK)
      reinterpret_cast<unsigned long long*>(s_ops)[t] = reinterpret_cast<const unsigned long long*>(ops + at)[t];
    __syncthreads();
  };
  extern __shared__ __align__(16) uint64_t s_small[];
  constexpr unsigned CAP = SmallFor<W>::cap;
  const Region<W> R = region_at<W>(s_small, CAP, 2 * CAP);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(R.table + 2 * CAP);
  unsigned N = (unsigned)ld_volatile(&ctrl->n);  // at most kSmallStart: the host knows the count
  uint64_t sx[W], sz[W];
#pragma unroll
  for (int w = 0; w < W; ++w) sx[w] = sz[w] = 0ull;
  for (unsigned i = threadIdx.x; i < N; i += BLOCK) {
    uint64_t x[W], z[W];
    load_key<W>(P, i, x, z);
    rstore<W>(R, i, x, z);
    R.c[i] = P.c[i];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      sx[w] |= x[w];
      sz[w] |= z[w];
    }
  }
  for (unsigned t = threadIdx.x; t < 2 * CAP; t += BLOCK) R.table[t] = 0ull;
  for (unsigned t = threadIdx.x; t < CAP; t += BLOCK) R.link[t] = 0ull;
  if (threadIdx.x == 0) s_perr = 0;
  block_or<W>(sx, sz, s_or);
  unsigned epoch = 0, pc = 0;
  unsigned run_end = 0, run_at = 0, run_n = 0;  // the fused run being applied: [run_at, run_end), its first size
  bool run_rx = false;
  uint64_t Q[W];
  // an op's live count; n_s and n_new of these ops are not recorded per kernel
  auto logop = [&](unsigned o, unsigned n_in, unsigned n_out) {
    if (threadIdx.x == 0) {
      OpLog& l = log[op0 + o];
      l.n_in = n_in;
      l.n_s = 0;
      l.n_new = n_out > n_in ? n_out - n_in : 0;
      l.n_out = n_out;
    }
  };
  fetch(0);
  while (pc < nops) {
    if (pc - s0 >= OPS) fetch(pc);
    const SmallOp& op = s_ops[pc - s0];
    const uint32_t kind = op.kind;
    if (epoch >= 0xFFF0u) {  // pair-table epochs about to wrap
      __syncthreads();
      for (unsigned t = threadIdx.x; t < 2 * CAP; t += BLOCK) R.table[t] = 0ull;
      __syncthreads();
      epoch = 0;
    }
    if (kind == S_TRUNC) {
      const unsigned kept = (unsigned)cta_truncate<W, BLOCK, ITEMS>(R, N, thr, maxw, s_base, s_or, sx, sz);
      logop(pc, N, kept);
      N = kept;
      ++pc;
      continue;
    }
    if (kind == S_LOCAL) {
      unsigned j = pc;
      while (j < nops && j - s0 < OPS && s_ops[j - s0].kind == S_LOCAL) ++j;
#pragma unroll
      for (int w = 0; w < W; ++w) sx[w] = sz[w] = 0ull;
      for (unsigned i = threadIdx.x; i < N; i += BLOCK) {
        uint64_t x[W], z[W];
        rload<W>(R, i, x, z);
        double c = R.c[i];
        bool neg = false;
        for (unsigned o = pc; o < j; ++o) local_op<W>(s_ops[o - s0].d, x, z, c, neg);
        rstore<W>(R, i, x, z);
        R.c[i] = neg ? -c : c;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          sx[w] |= x[w];
          sz[w] |= z[w];
        }
      }
      block_or<W>(sx, sz, s_or);
      for (unsigned o = pc; o < j; ++o) logop(o, N, N);
      pc = j;
      continue;
    }
    if (kind == S_DAMP) {
      const unsigned n_out = small_rotate<W, true>(R, op, N, ++epoch, s_base, s_perr);
      if (n_out > CAP) break;
      logop(pc, N, n_out);
      N = n_out;
      ++pc;
      continue;
    }
    const DevOp d = op.d;
    if (op.run) {  // a fused run starts: its terms as they are, in case it outgrows the region
      run_rx = (d.ax & 1) != 0;
      if (!small_run_begin<W>(R, N, ops ? ops + pc : s_ops + pc, op.run, run_rx, s_q, Q)) break;  // too wide: the pipeline cuts it
      run_at = pc;
      run_end = pc + op.run;
      run_n = N;
      for (unsigned i = threadIdx.x; i < N; i += BLOCK) {
        uint64_t x[W], z[W];
        rload<W>(R, i, x, z);
        store_key<W>(P, i, x, z);
        P.c[i] = R.c[i];
      }
    }
    const unsigned n_in = N;
    if (rot_may_touch<W>(d, sx, sz)) {
      const unsigned n_out = small_rotate<W, false>(R, op, N, ++epoch, s_base, s_perr);
      if (n_out > CAP) break;
      N = n_out;
      join_gen<W>(d, sx, sz);
    }
    logop(pc, n_in, N);
    ++pc;
    if (pc == run_end) {
      small_run_sort<W>(R, run_n, N, run_rx, Q, ++epoch, keys);
      run_end = 0;
    }
  }
  __syncthreads();
  if (run_end > pc) {  // stopped inside a run: the terms before it are in P
    N = run_n;
    pc = run_at;
  } else {
    for (unsigned i = threadIdx.x; i < N; i += BLOCK) {
      uint64_t x[W], z[W];
      rload<W>(R, i, x, z);
      store_key<W>(P, i, x, z);
      P.c[i] = R.c[i];
    }
  }
  if (threadIdx.x == 0) {
    ctrl->n = N;
    host->n = N;
    host->small_pc = pc;
    host->err = 0;
  }
}

}  // namespace ppvm
