// cta.cuh — a sum held and advanced by one CTA.
//
// The terms of the sum, a pair table and a list of indices lie in one region of words, in global
// or in shared memory (the arrays are generic pointers); the CTA applies ops to it in order, with
// the reference's semantics (crates/ppvm-pauli-sum/src/sum/data.rs:204-311) and term order, and
// its only synchronisation is the block barrier.  Used by the batched sums (batch.cu: one CTA
// per instance) and by the list interpreter of small single sums (small.cuh).
#pragma once

#include "tableau.cuh"

namespace ppvm {

__host__ __device__ inline unsigned long long region_words(int W, unsigned long long cap, unsigned long long tsize) {
  return (unsigned long long)(2 * W + 2) * cap + (cap + 1) / 2 + tsize;
}

template <int W>
struct Region {
  uint64_t* x;
  uint64_t* z;
  double* c;
  unsigned long long* link;  // per term: its partner's coefficient, complemented (0 = none; all 0 between ops)
  uint32_t* sidx;            // anticommuting terms: each warp's list at the start of its chunk of terms
  unsigned long long* table;
  unsigned long long cap, tsize;
};

// The region layout from its first word b (in the pool, or in shared memory).
template <int W>
__device__ __forceinline__ Region<W> region_at(uint64_t* b, unsigned long long cap, unsigned long long tsize) {
  Region<W> r;
  r.cap = cap;
  r.tsize = tsize;
  r.x = b;
  r.z = b + (size_t)W * cap;
  r.c = reinterpret_cast<double*>(b + (size_t)2 * W * cap);
  r.link = reinterpret_cast<unsigned long long*>(b + (size_t)(2 * W + 1) * cap);
  r.sidx = reinterpret_cast<uint32_t*>(b + (size_t)(2 * W + 2) * cap);
  r.table = reinterpret_cast<unsigned long long*>(b + (size_t)(2 * W + 2) * cap + (cap + 1) / 2);
  return r;
}
template <int W>
__device__ __forceinline__ void rload(const Region<W>& R, unsigned long long i, uint64_t (&x)[W], uint64_t (&z)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    x[w] = R.x[(size_t)w * R.cap + i];
    z[w] = R.z[(size_t)w * R.cap + i];
  }
}
template <int W>
__device__ __forceinline__ void rstore(const Region<W>& R, unsigned long long i, const uint64_t (&x)[W],
                                       const uint64_t (&z)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    R.x[(size_t)w * R.cap + i] = x[w];
    R.z[(size_t)w * R.cap + i] = z[w];
  }
}
// word w of a W-word array without dynamic register indexing
template <int W>
__device__ __forceinline__ uint64_t wsel(const uint64_t (&a)[W], unsigned w) {
  uint64_t v = 0;
#pragma unroll
  for (int k = 0; k < W; ++k) v = (k == (int)w) ? a[k] : v;
  return v;
}
template <int W>
__device__ __forceinline__ void wflip(uint64_t (&a)[W], unsigned w, uint64_t m) {
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (k == (int)w) a[k] ^= m;
}
template <int W>
__device__ __forceinline__ void wset_bits(uint64_t (&a)[W], unsigned w, uint64_t m) {
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (k == (int)w) a[k] |= m;
}
template <int W>
__device__ __forceinline__ void wset(uint64_t (&a)[W], unsigned w, unsigned b, bool v) {
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (k == (int)w) a[k] = (a[k] & ~(1ull << b)) | ((uint64_t)v << b);
}

// Rotation on at most two qubits with axes (ax, az) (bit 0: q0, bit 1: q1).  For a word with
// bits (x0, z0) at q0 and (x1, z1) at q1: whether it anticommutes, and eps of its child
// (+1 exactly when the anticommuting qubit's single-qubit phase in G*P is -1, as rot_sign).
struct RotBits {
  bool anti;
  bool eps_plus;
};
__device__ __forceinline__ RotBits rot_bits(const DevOp& d, bool x0, bool z0, bool x1, bool z1) {
  const bool ax0 = d.ax & 1, az0 = d.az & 1, ax1 = d.two && (d.ax & 2), az1 = d.two && (d.az & 2);
  RotBits r;
  r.anti = ((x0 & az0) ^ (z0 & ax0)) ^ ((x1 & az1) ^ (z1 & ax1));
  const bool m0 = (ax0 & !az0 & !x0 & z0) | (ax0 & az0 & x0 & !z0) | (!ax0 & az0 & x0 & z0);
  const bool m1 = (ax1 & !az1 & !x1 & z1) | (ax1 & az1 & x1 & !z1) | (!ax1 & az1 & x1 & z1);
  r.eps_plus = m0 | m1;
  return r;
}

template <int W>
__device__ __forceinline__ void op_bits(const DevOp& d, const uint64_t (&x)[W], const uint64_t (&z)[W], bool& x0,
                                        bool& z0, bool& x1, bool& z1) {
  x0 = (wsel<W>(x, d.w0) >> d.b0) & 1ull;
  z0 = (wsel<W>(z, d.w0) >> d.b0) & 1ull;
  x1 = (wsel<W>(x, d.w1) >> d.b1) & 1ull;
  z1 = (wsel<W>(z, d.w1) >> d.b1) & 1ull;
}

template <int W>
__device__ __forceinline__ void flip_gen(const DevOp& d, uint64_t (&x)[W], uint64_t (&z)[W]) {
  if (d.ax & 1) wflip<W>(x, d.w0, 1ull << d.b0);
  if (d.az & 1) wflip<W>(z, d.w0, 1ull << d.b0);
  if (d.two) {
    if (d.ax & 2) wflip<W>(x, d.w1, 1ull << d.b1);
    if (d.az & 2) wflip<W>(z, d.w1, 1ull << d.b1);
  }
}

// Bits of term i at the op's qubits, read from the planes (two words at most).
template <int W>
__device__ __forceinline__ void term_bits(const Region<W>& R, const DevOp& d, unsigned long long i, bool& x0,
                                          bool& z0, bool& x1, bool& z1) {
  x0 = (R.x[(size_t)d.w0 * R.cap + i] >> d.b0) & 1ull;
  z0 = (R.z[(size_t)d.w0 * R.cap + i] >> d.b0) & 1ull;
  x1 = z1 = false;
  if (d.two) {
    x1 = (R.x[(size_t)d.w1 * R.cap + i] >> d.b1) & 1ull;
    z1 = (R.z[(size_t)d.w1 * R.cap + i] >> d.b1) & 1ull;
  }
}

// One local op (Clifford, Clifford-angle rotation or diagonal noise) on a word, the rules of
// the per-op pass (crates/ppvm-pauli-sum/src/sum/clifford.rs:37-221, sum/noise.rs:17-129).
template <int W>
__device__ __forceinline__ void local_op(const DevOp& d, uint64_t (&x)[W], uint64_t (&z)[W], double& c, bool& neg) {
  bool x0, z0, x1, z1;
  op_bits<W>(d, x, z, x0, z0, x1, z1);
  switch (d.code) {
    case C_PAULI_ERROR: {
      const int k = (int)x0 | ((int)z0 << 1);
      if (k == 1) c = __dmul_rn(c, d.f0);
      else if (k == 2) c = __dmul_rn(c, d.f1);
      else if (k == 3) c = __dmul_rn(c, d.f2);
      return;
    }
    case C_DEP1:
      if (x0 | z0) c = __dmul_rn(c, d.f0);
      return;
    case C_DEP2:
      if (x0 | z0 | x1 | z1) c = __dmul_rn(c, d.f0);
      return;
    default: break;
  }
  const bool two = d.code == C_CNOT || d.code == C_CZ || d.code == C_CY || (d.code == C_ROTC && d.two);
  if (!two) x1 = z1 = false;
  cliff_rule<bool>(d, x0, z0, x1, z1, neg);
  wset<W>(x, d.w0, d.b0, x0);
  wset<W>(z, d.w0, d.b0, z0);
  if (two) {
    wset<W>(x, d.w1, d.b1, x1);
    wset<W>(z, d.w1, d.b1, z1);
  }
}

// ORs the block's masks into s_or (2W words) and returns them to every thread.
template <int W>
__device__ __forceinline__ void block_or(uint64_t (&ox)[W], uint64_t (&oz)[W], unsigned long long* s_or) {
  __syncthreads();
  if (threadIdx.x < 2 * W) s_or[threadIdx.x] = 0ull;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const unsigned xl = __reduce_or_sync(kFull, (unsigned)ox[w]), xh = __reduce_or_sync(kFull, (unsigned)(ox[w] >> 32));
    const unsigned zl = __reduce_or_sync(kFull, (unsigned)oz[w]), zh = __reduce_or_sync(kFull, (unsigned)(oz[w] >> 32));
    if ((threadIdx.x & 31) == 0) {
      atomicOr(&s_or[w], (unsigned long long)xh << 32 | xl);
      atomicOr(&s_or[W + w], (unsigned long long)zh << 32 | zl);
    }
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    ox[w] = s_or[w];
    oz[w] = s_or[W + w];
  }
}

// The coefficient in a link word (its complement), and back: 0 means no link, so the one NaN
// whose complement is 0 is linked as another NaN.
__device__ __forceinline__ unsigned long long link_word(double c) {
  const unsigned long long v = ~(unsigned long long)__double_as_longlong(c);
  return v ? v : 1ull;
}

// Shared-memory scratch of the CTA's pair step.
template <int W, int NW>
struct CtaShared {
  unsigned cnt[NW], child[NW];  // per warp: its list's length, its children
  unsigned long long orw[2 * W];
  int perr;                     // a probe ran round the table
};

// What cta_pair found: S touched terms in the warps' lists, C children to append, and this
// warp's share [rlo, rhi) of their ranks, whose children go to N + at, N + at + 1, ...
template <int NW>
struct CtaPlan {
  unsigned S, C, at, rlo, rhi, chunk;
  unsigned pre[NW];
};

// Index of the touched term of rank r.
template <int W, int NW>
__device__ __forceinline__ unsigned cta_nth(const Region<W>& R, const CtaPlan<NW>& p, unsigned r) {
  unsigned at = r;  // warp w's list starts at w * chunk
#pragma unroll
  for (int w = 1; w < NW; ++w)
    if (r >= p.pre[w]) at = w * p.chunk + (r - p.pre[w]);
  return R.sidx[at];
}

// First half of a rotation exp(-i theta/2 G), G on d's one or two qubits: lists the terms that
// anticommute with G, links the pairs and counts the children.  Nothing but links, lists and table
// entries is written, so a caller without room for the children can stop here.  Returns false
// when nothing is touched.  Each warp lists its own chunk of the terms, in order and without a
// barrier; the pair K, K^G meets in the table at one of the two keys, and the second to arrive
// hands each the other's coefficient.
template <int W, int BLOCK, int ITEMS>
__device__ __forceinline__ bool cta_pair(const Region<W>& R, const DevOp& d, unsigned N, unsigned epoch,
                                         CtaShared<W, BLOCK / 32>& sh, CtaPlan<BLOCK / 32>& p) {
  constexpr int NW = BLOCK / 32;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  p.chunk = ((N + NW - 1) / NW + 31u) & ~31u;
  const unsigned lo = min(N, warp * p.chunk), hi = min(N, lo + p.chunk);
  unsigned cnt = 0;
  for (unsigned b0 = lo; b0 < hi; b0 += 32 * ITEMS) {
    bool a[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned i = b0 + k * 32 + lane;
      a[k] = false;
      if (i < hi) {
        bool x0, z0, x1, z1;
        term_bits<W>(R, d, i, x0, z0, x1, z1);
        a[k] = rot_bits(d, x0, z0, x1, z1).anti;
      }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned m = __ballot_sync(kFull, a[k]);
      if (a[k]) R.sidx[lo + cnt + __popc(m & lt)] = b0 + k * 32 + lane;
      cnt += __popc(m);
    }
  }
  if (lane == 0) sh.cnt[warp] = cnt;
  if (!__syncthreads_or(cnt != 0)) return false;
  p.S = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    p.pre[w] = p.S;
    p.S += sh.cnt[w];
  }
  const unsigned long long mask = R.tsize - 1;
  for (unsigned r = threadIdx.x; r < p.S; r += BLOCK) {
    const unsigned i = cta_nth<W, NW>(R, p, r);
    uint64_t x[W], z[W], px[W], pz[W], kx[W], kz[W];
    rload<W>(R, i, x, z);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      px[w] = x[w];
      pz[w] = z[w];
    }
    flip_gen<W>(d, px, pz);
    // of the two keys, the one without the flipped bit on q0
    const bool use_p = ((d.ax & 1 ? wsel<W>(x, d.w0) : wsel<W>(z, d.w0)) >> d.b0) & 1ull;
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
        cur = prev;  // taken meanwhile: examine what is there now
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
        sh.perr = 1;  // cannot happen with tsize >= 2 * cap; reported, not trapped
        break;
      }
      cur = ld_volatile(&R.table[slot]);
    }
  }
  __syncthreads();
  // each warp counts the children of its share of the ranks; their places follow from the counts
  const unsigned share = ((p.S + NW - 1) / NW + 31u) & ~31u;
  p.rlo = min(p.S, warp * share);
  p.rhi = min(p.S, p.rlo + share);
  unsigned kids = 0;
  for (unsigned r = p.rlo + lane; r < p.rhi; r += 32) {
    kids += R.link[cta_nth<W, NW>(R, p, r)] == 0ull;
  }
  kids = __reduce_add_sync(kFull, kids);
  if (lane == 0) sh.child[warp] = kids;
  __syncthreads();
  p.C = p.at = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    if (w < (int)warp) p.at += sh.child[w];
    p.C += sh.child[w];
  }
  return true;
}

// Second half: new coefficients in place (parent c*cs, + partner's c*(eps*sn)), children c*(eps*sn)
// appended in parent order (there is room).
template <int W, int BLOCK>
__device__ __forceinline__ void cta_apply(const Region<W>& R, const DevOp& d, double sn, double cs,
                                          unsigned long long N, const CtaPlan<BLOCK / 32>& p) {
  constexpr int NW = BLOCK / 32;
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  unsigned at = p.at;
  for (unsigned r0 = p.rlo; r0 < p.rhi; r0 += 32) {
    const unsigned r = r0 + lane;
    unsigned i = 0;
    double made = 0.0;
    bool child = false;
    if (r < p.rhi) {
      i = cta_nth<W, NW>(R, p, r);
      const double c = R.c[i];
      const unsigned long long lw = R.link[i];
      bool x0, z0, x1, z1;
      term_bits<W>(R, d, i, x0, z0, x1, z1);
      child = lw == 0ull;
      made = __dmul_rn(c, (rot_bits(d, x0, z0, x1, z1).eps_plus ? 1.0 : -1.0) * sn);
      double nc = __dmul_rn(c, cs);
      if (lw) {
        // the partner's key is K^G: its eps from this term's bits with G's bits flipped
        x0 ^= (bool)(d.ax & 1);
        z0 ^= (bool)(d.az & 1);
        if (d.two) {
          x1 ^= (bool)(d.ax & 2);
          z1 ^= (bool)(d.az & 2);
        }
        nc = __dadd_rn(nc, __dmul_rn(__longlong_as_double((long long)~lw),
                                     (rot_bits(d, x0, z0, x1, z1).eps_plus ? 1.0 : -1.0) * sn));
        R.link[i] = 0ull;
      }
      R.c[i] = nc;
    }
    const unsigned m = __ballot_sync(kFull, child);
    if (child) {
      const unsigned long long pos = N + at + __popc(m & lt);
      uint64_t x[W], z[W];
      rload<W>(R, i, x, z);
      flip_gen<W>(d, x, z);
      rstore<W>(R, pos, x, z);
      R.c[pos] = made;
    }
    at += __popc(m);
  }
}

// Whether the rotation (one or two qubits) can touch a term of a sum whose X and Z bits lie in sx, sz.
template <int W>
__device__ __forceinline__ bool rot_may_touch(const DevOp& d, const uint64_t (&sx)[W], const uint64_t (&sz)[W]) {
  bool x0, z0, x1, z1;
  op_bits<W>(d, sx, sz, x0, z0, x1, z1);
  return ((d.az & 1) && x0) || ((d.ax & 1) && z0) || (d.two && (((d.az & 2) && x1) || ((d.ax & 2) && z1)));
}

// The generator's bits joined to the sum's (its children may hold them).
template <int W>
__device__ __forceinline__ void join_gen(const DevOp& d, uint64_t (&sx)[W], uint64_t (&sz)[W]) {
  if (d.ax & 1) wset_bits<W>(sx, d.w0, 1ull << d.b0);
  if (d.az & 1) wset_bits<W>(sz, d.w0, 1ull << d.b0);
  if (d.two) {
    if (d.ax & 2) wset_bits<W>(sx, d.w1, 1ull << d.b1);
    if (d.az & 2) wset_bits<W>(sz, d.w1, 1ull << d.b1);
  }
}

// Stable in-place compaction with the truncation rule; returns the kept count and recomputes the
// sum's bits.  A tile's reads finish (inside tile_ranks) before its writes, and every write
// goes to a position at or below the word it came from.
template <int W, int BLOCK, int ITEMS>
__device__ __forceinline__ unsigned long long cta_truncate(const Region<W>& R, unsigned long long N, double thr,
                                                           unsigned long long maxw, unsigned* s_base,
                                                           unsigned long long* s_or, uint64_t (&sx)[W],
                                                           uint64_t (&sz)[W]) {
  constexpr int NW = BLOCK / 32;
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const bool wcap = maxw != ~0ull;
  unsigned long long kept = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) sx[w] = sz[w] = 0ull;
  for (unsigned long long base = 0; base < N; base += TILE) {
    uint64_t kx[ITEMS][W], kz[ITEMS][W];
    double kc[ITEMS];
    unsigned bal[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      bool keep = false;
      if (i < N) {
        rload<W>(R, i, kx[k], kz[k]);
        kc[k] = R.c[i];
        keep = !(fabs(kc[k]) < thr);
        if (wcap) keep = keep && (weight<W>(kx[k], kz[k]) <= maxw);
      }
      bal[k] = __ballot_sync(kFull, keep);
    }
    const unsigned agg = tile_ranks<BLOCK, ITEMS>(bal, s_base);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
      if ((bal[k] >> lane) & 1u) {
        const unsigned long long r = kept + s_base[k * NW + warp] + __popc(bal[k] & lt);
        rstore<W>(R, r, kx[k], kz[k]);
        R.c[r] = kc[k];
#pragma unroll
        for (int w = 0; w < W; ++w) {
          sx[w] |= kx[k][w];
          sz[w] |= kz[k][w];
        }
      }
    kept += agg;
    __syncthreads();
  }
  block_or<W>(sx, sz, s_or);
  return kept;
}

}  // namespace ppvm
