// runs.cuh — fused runs of single-qubit X-type or Z-type rotations.
//
// A run is a sequence of RX rotations on distinct qubits (or of RZ rotations on distinct
// qubits) with no other op in between, optionally ending in TRUNCATE.  During such a run a
// term's Z plane (RX) or X plane (RZ) never changes: it is the invariant plane v.  Gate j on
// qubit q acts on a term iff v has bit q, and then only flips bit q of the other plane f.
// So the terms sharing (v, f with the bits M = v & Q cleared) — Q the run's qubits — form a
// group that evolves on its own: its members are the 2^|M| words f0 | pdep(c, M), c in
// [0, 2^|M|).  The reference processes the run gate by gate over the whole map
// (PauliSum::map_insert per gate, crates/ppvm-pauli-sum/src/sum/data.rs:204-226); here each
// group is loaded once, the gates of the run are applied in the same order with the same
// arithmetic as a butterfly over coordinates c in registers (existence tracked
// separately from the coefficient, as a map entry exists even with coefficient 0), and the
// truncation that ends the run is applied before anything is written back.  The term set
// and every coefficient are identical to the reference's; only the output order differs
// (untouched terms in order, then groups by their first member, members by coordinate).
//
// Kernels, in order: k_run_classify (group keys into a hash table, members counted; terms
// outside every group compacted to the output with the truncation), k_run_order
// (deterministic group numbering by first member, member offsets), k_run_scatter (member
// lists), then k_run_tiles or, for many small groups, k_run_lanes (butterfly + truncation + ordered
// write; the last block publishes the counts and the op log), and k_run_place when the
// tiles left their order to it.
#pragma once

#include "kernels.cuh"

namespace ppvm {

constexpr int kRunMaxK = 10;       // groups of up to 10 coordinates (2^10 slots) are fused
constexpr int kRunMaxGates = 256;  // gates per fused run
constexpr int kRunLaneK = 3;       // groups of up to 3 coordinates (8 slots) run on one lane
constexpr int kRunWarps = 4;       // warps of a k_run_lanes block
constexpr unsigned long long kRunTileMinGroups = 8192;  // fewer groups: never one per lane
constexpr unsigned long long kRunLogScratchBit = 1ull << 63;  // in the op log of a run's first gate
constexpr int kErrFallback = 4;    // device error: a group exceeds kRunMaxK; rerun per gate

struct RunDesc {
  uint32_t cls;   // 0: RX run (v = z plane, f = x plane); 1: RZ run (v = x, f = z)
  uint32_t L;     // gates
  uint64_t Q[kMaxW];
  uint32_t q[kRunMaxGates];
  double sn[kRunMaxGates];
  double cs[kRunMaxGates];
};

struct RunScratch {
  uint32_t* gslot;     // per term: group slot (kNone = untouched)
  uint32_t* grp_min;   // per table slot: smallest member index
  uint32_t* grp_cnt;   // per table slot: member count
  uint32_t* grp_ord;   // per table slot: group ordinal
  uint32_t* g_start;   // per group
  uint32_t* g_cnt;
  uint32_t* g_rep;
  uint32_t* g_fill;
  uint32_t* mcoord;    // per member, in group order: its coordinate index (bits of f at M)
  double* mcoef;       // per member, in group order: its coefficient
  uint64_t* gkey;      // per group: v[W] then f outside the coordinates, f0[W]
  unsigned long long* created;  // per gate of the run: children created
};

template <int W>
__device__ __forceinline__ void split_planes(uint32_t cls, const uint64_t (&x)[W], const uint64_t (&z)[W],
                                             uint64_t (&v)[W], uint64_t (&f)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    v[w] = cls == 0 ? z[w] : x[w];
    f[w] = cls == 0 ? x[w] : z[w];
  }
}

// ---------------------------------------------------------------------------------------
// Classifies every term and, in the same pass, writes the terms the run does not touch
// (no qubit of the run in the invariant plane) to the front of the output planes, in index
// order, with the run's TRUNCATE applied to them (tile ranks + decoupled look-back).  Touched
// terms join their group in the hash table.
template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_run_classify(Planes P, Planes O, Ctrl* ctrl, const RunDesc* rd, RunScratch R, unsigned long long* table,
               unsigned long long tmask, unsigned tepoch, int trunc, double thr, unsigned long long maxw,
               unsigned long long* ts, unsigned epoch, int op, unsigned turn) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  __shared__ int s_err;
  __shared__ unsigned long long s_large, s_slots;
  __shared__ uint16_t s_gidx[64 * W];  // qubit -> its gate's index in the run
  if (threadIdx.x == 0) s_large = s_slots = 0;
  if (threadIdx.x == 0) s_err = ld_volatile_int(&ctrl->err);
  for (unsigned j = threadIdx.x; j < rd->L; j += BLOCK) s_gidx[rd->q[j]] = (uint16_t)j;
  __syncthreads();
  if (s_err) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned long long ntiles = (N + TILE - 1) / TILE;
  if (blockIdx.x == 0 && threadIdx.x == 0 && N == 0) ctrl->n_s = 0;
  const uint32_t cls = rd->cls;
  uint64_t Q[W];
#pragma unroll
  for (int w = 0; w < W; ++w) Q[w] = rd->Q[w];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  const bool wcap = maxw != ~0ull;
  // groups opened by this thread that are too large for a lane, and the slots of all it opened
  unsigned large = 0;
  unsigned long long slots = 0;
  for (;;) {
    const unsigned tile = next_tile(&ctrl->tickets[1], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    uint64_t kx[ITEMS][W], kz[ITEMS][W];
    double kc[ITEMS];
    unsigned bal[ITEMS];
    unsigned fb = 0;  // fallback: the largest gate cut among this thread's wide terms
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const unsigned long long i = base + (unsigned long long)it * BLOCK + threadIdx.x;
      bool keep = false;
      if (i < N) {
        uint64_t v[W], f[W], M[W];
        load_key<W>(P, i, kx[it], kz[it]);
        split_planes<W>(cls, kx[it], kz[it], v, f);
        unsigned k = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          M[w] = v[w] & Q[w];
          k += __popcll(M[w]);
          f[w] &= ~M[w];
        }
        if (k == 0) {  // untouched by the run
          R.gslot[i] = kNone;
          kc[it] = P.c[i];
          keep = true;
          if (trunc) {
            keep = !(fabs(kc[it]) < thr);
            if (wcap) keep = keep && (weight<W>(kx[it], kz[it]) <= maxw);
          }
        } else if (k > (unsigned)kRunMaxK) {
          // v is invariant through the run, so this term and all its descendants keep these
          // k coordinates: the run from gate p on, p = 1 + the gate index of the term's
          // (k - kRunMaxK)-th coordinate in gate order, holds at most kRunMaxK of them.  The
          // host runs the gates before the largest such p one at a time and fuses the rest.
          unsigned hi[kRunMaxK + 1];  // the kRunMaxK+1 largest gate indices, descending
          unsigned nhi = 0;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            uint64_t m = M[w];
            while (m) {
              unsigned gi = s_gidx[w * 64 + (__ffsll((long long)m) - 1)];
              m &= m - 1;
              if (nhi == kRunMaxK + 1 && gi <= hi[kRunMaxK]) continue;
              unsigned r = nhi < kRunMaxK + 1 ? nhi++ : kRunMaxK;
              while (r > 0 && hi[r - 1] < gi) {
                hi[r] = hi[r - 1];
                --r;
              }
              hi[r] = gi;
            }
          }
          fb = max(fb, hi[kRunMaxK] + 1u);  // reported once per warp below
          R.gslot[i] = kNone;
        } else {
          const uint64_t h = table_hash<W>(v, f);
          const unsigned tag = (unsigned)(h >> 48) & 0xFFFFu;
          const unsigned long long mine = make_slot(tepoch, tag, (unsigned)i);
          unsigned long long slot = h & tmask;
          unsigned long long probes = 0;
          while (true) {
            const unsigned long long cur = ld_volatile(&table[slot]);
            if (slot_epoch(cur) != (tepoch & 0xFFFFu)) {
              const unsigned long long prev = atomicCAS(&table[slot], cur, mine);
              if (prev != cur) continue;
              large += k > (unsigned)kRunLaneK;
              slots += 1u << k;
              break;  // new group
            }
            if (slot_tag(cur) == tag) {
              uint64_t jx[W], jz[W], jv[W], jf[W];
              load_key<W>(P, slot_idx(cur), jx, jz);
              split_planes<W>(cls, jx, jz, jv, jf);
              bool eq = true;
#pragma unroll
              for (int w = 0; w < W; ++w) eq &= (jv[w] == v[w]) & ((jf[w] & ~M[w]) == f[w]);
              if (eq) break;  // same group
            }
            slot = (slot + 1) & tmask;
            if (++probes > tmask) {
              set_err(ctrl, kErrProbe, op);
              break;
            }
          }
          R.gslot[i] = (uint32_t)slot;
          atomicMin(&R.grp_min[slot], (uint32_t)i);
          atomicAdd(&R.grp_cnt[slot], 1u);
        }
      }
      bal[it] = __ballot_sync(kFull, keep);
    }
    // terms with more than kRunMaxK coordinates: one report per warp instead of one atomic on
    // the same two words per term (a wide run has millions of such terms)
    fb = __reduce_max_sync(kFull, fb);
    if (fb && lane == 0) {
      if (ld_volatile(&ctrl->fb_cut) < fb) atomicMax(&ctrl->fb_cut, (unsigned long long)fb);
      if (!ld_volatile_int(&ctrl->err)) set_err(ctrl, kErrFallback, op);
    }
    const unsigned agg = tile_ranks<BLOCK, ITEMS>(bal, s_base);
    const unsigned long long excl = lookback(ts, tile, agg, epoch, ctrl, op, &s_slot);
#pragma unroll
    for (int it = 0; it < ITEMS; ++it)
      if ((bal[it] >> lane) & 1u) {
        const unsigned long long r = excl + s_base[it * NW + warp] + __popc(bal[it] & ((1u << lane) - 1u));
        store_key<W>(O, r, kx[it], kz[it]);
        O.c[r] = kc[it];
      }
    if (tile == ntiles - 1 && threadIdx.x == 0) ctrl->n_s = excl + agg;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) slots += __shfl_down_sync(kFull, slots, o);
  large = __reduce_add_sync(kFull, large);
  if (lane == 0 && slots) {
    atomicAdd(&s_slots, slots);
    if (large) atomicAdd(&s_large, (unsigned long long)large);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_slots) {
    atomicAdd(&ctrl->run_slots[turn], s_slots);
    if (s_large) atomicAdd(&ctrl->run_large[turn], s_large);
  }
}

// Numbers the groups by their smallest member (index order) and lays out member lists.
// While the sum holds fewer than 2^21 terms (every block reads the same N), both running
// counts travel in one look-back value, groups in the low 21 bits and members in the next 21:
// one chain per tile instead of two.
constexpr int kOrderPackBits = 21;
template <int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_run_order(Ctrl* ctrl, RunScratch R, unsigned long long* ts_a, unsigned long long* ts_b, unsigned ep_a,
            unsigned ep_b, int op) {
  pdl_wait();
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_base[ITEMS * (BLOCK / 32) + 1];
  __shared__ unsigned long long s_cnt[BLOCK];
  if (ld_volatile_int(&ctrl->err)) return;
  const unsigned long long N = ld_volatile(&ctrl->n);
  constexpr unsigned long long TILE = (unsigned long long)BLOCK * ITEMS;
  const unsigned long long ntiles = (N + TILE - 1) / TILE;
  if (blockIdx.x == 0 && threadIdx.x == 0 && N == 0) {
    ctrl->n_pairs = 0;   // groups
    ctrl->n_side = 0;    // members
  }
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  for (;;) {
    const unsigned tile = next_tile(&ctrl->tickets[0], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    unsigned ballots[ITEMS];
    unsigned cnts[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
      bool rep = false;
      cnts[k] = 0;
      if (i < N) {
        const uint32_t s = R.gslot[i];
        if (s != kNone) {
          const uint32_t first = R.grp_min[s], cnt = R.grp_cnt[s];  // both loads in flight at once
          if (first == (uint32_t)i) {
            rep = true;
            cnts[k] = cnt;
          }
        }
      }
      ballots[k] = __ballot_sync(kFull, rep);
    }
    const unsigned agg = tile_ranks<BLOCK, ITEMS>(ballots, s_base);
    // member-count prefix in index order: per item k, warp-level scan, then across (k, warp)
    // The per-(k,warp) sums are small; a second rank table over counts is built in s_cnt.
    unsigned long long item_pre[ITEMS];
    unsigned long long warp_tot[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      unsigned long long v = cnts[k];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, v, o);
        if (lane >= (unsigned)o) v += t;
      }
      item_pre[k] = v - cnts[k];
      warp_tot[k] = __shfl_sync(kFull, v, 31);
    }
    // s_cnt[k*NW + warp] = warp totals; exclusive scan by thread 0 (ITEMS*NW <= 64 entries)
    __syncthreads();
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) s_cnt[k * NW + warp] = warp_tot[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long run = 0;
      for (int e = 0; e < ITEMS * NW; ++e) {
        const unsigned long long t = s_cnt[e];
        s_cnt[e] = run;
        run += t;
      }
      s_cnt[ITEMS * NW] = run;
    }
    __syncthreads();
    const unsigned long long agg_cnt = s_cnt[ITEMS * NW];
    unsigned long long excl, excl_cnt;
    if (N < (1ull << kOrderPackBits)) {
      const unsigned long long both =
          lookback(ts_a, tile, (unsigned long long)agg | (agg_cnt << kOrderPackBits), ep_a, ctrl, op, &s_slot);
      excl = both & ((1ull << kOrderPackBits) - 1);
      excl_cnt = both >> kOrderPackBits;
    } else {
      excl = lookback(ts_a, tile, agg, ep_a, ctrl, op, &s_slot);
      excl_cnt = lookback(ts_b, tile, agg_cnt, ep_b, ctrl, op, &s_slot);
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      if ((ballots[k] >> lane) & 1u) {
        const unsigned long long i = base + (unsigned long long)k * BLOCK + threadIdx.x;
        const unsigned long long ord = excl + s_base[k * NW + warp] + __popc(ballots[k] & ((1u << lane) - 1u));
        const unsigned long long start = excl_cnt + s_cnt[k * NW + warp] + item_pre[k];
        const uint32_t s = R.gslot[i];
        R.grp_ord[s] = (uint32_t)ord;
        R.g_start[ord] = (uint32_t)start;
        R.g_cnt[ord] = cnts[k];
        R.g_rep[ord] = (uint32_t)i;
        R.g_fill[ord] = 0;
      }
    }
    if (tile == ntiles - 1 && threadIdx.x == 0) {
      ctrl->n_pairs = excl + agg;        // groups
      ctrl->n_side = excl_cnt + agg_cnt; // members (touched terms)
    }
  }
}

// Lays out each group's members contiguously, as (coordinate index, coefficient) records,
// and the group's key (from its representative), so that the group kernels read one span per group
// instead of gathering members by index.  A member's coordinate index has bit t set when f
// has a 1 at the t-th lowest qubit of M = v & Q (the order the group kernels use).  Also hands
// the group table back clean: grp_min and grp_cnt were last read by k_run_order, so every
// member resets its slot (same values from every member), and the next run needs no
// clearing pass.  After a device error the host clears both arrays instead.
template <int W>
__global__ void __launch_bounds__(256) k_run_scatter(Planes P, Ctrl* ctrl, const RunDesc* rd, RunScratch R, unsigned turn) {
  pdl_wait();
  if (ld_volatile_int(&ctrl->err)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->run_large[turn ^ 1u] = ctrl->run_slots[turn ^ 1u] = 0;  // for the next run
  const unsigned long long N = ld_volatile(&ctrl->n);
  const uint32_t cls = rd->cls;
  uint64_t Q[W];
#pragma unroll
  for (int w = 0; w < W; ++w) Q[w] = rd->Q[w];
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t s = R.gslot[i];
    if (s == kNone) continue;
    uint64_t x[W], z[W], v[W], f[W];
    load_key<W>(P, i, x, z);  // the term's own data: in flight with the group lookups below
    const double coef = P.c[i];
    const uint32_t o = R.grp_ord[s];
    const uint32_t pos = R.g_start[o] + atomicAdd(&R.g_fill[o], 1u);
    split_planes<W>(cls, x, z, v, f);
    unsigned c = 0, t = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t m = v[w] & Q[w];
      while (m) {
        const int b = __ffsll((long long)m) - 1;
        c |= (unsigned)((f[w] >> b) & 1ull) << t;
        ++t;
        m &= m - 1;
      }
    }
    R.mcoord[pos] = c;
    R.mcoef[pos] = coef;
    if (R.g_rep[o] == (uint32_t)i) {
      uint64_t* gk = R.gkey + (unsigned long long)o * 2 * W;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        gk[w] = v[w];
        gk[W + w] = f[w] & ~(v[w] & Q[w]);
      }
    }
    R.grp_min[s] = kNone;
    R.grp_cnt[s] = 0u;
  }
}

// Publishes the count after the run and fills the op log of its gates (and its TRUNCATE):
// one warp of the last block of k_run_tiles or k_run_lanes.  Gate j's live count is n0 plus the children
// the gates before it created (an exclusive scan of the created counts, 8 gates per lane).
__device__ __forceinline__ void run_commit(Ctrl* ctrl, RunScratch R, int op0, int L, int trunc_op, OpLog* log,
                                           bool scratch, unsigned long long cap) {
  const unsigned lane = threadIdx.x & 31;
  if (ld_volatile_int(&ctrl->err)) {
    if (lane < 4) ctrl->tickets[lane] = 0;
    return;
  }
  constexpr int PER = kRunMaxGates / 32;
  unsigned long long made[PER], tot = 0;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int j = (int)lane * PER + e;
    made[e] = j < L ? ld_volatile(&R.created[j]) : 0ull;
    tot += made[e];
  }
  unsigned long long incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(kFull, incl, o);
    if (lane >= (unsigned)o) incl += t;
  }
  const unsigned long long total = __shfl_sync(kFull, incl, 31);
  const unsigned long long n0 = ld_volatile(&ctrl->n);
  unsigned long long run = n0 + incl - tot;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int j = (int)lane * PER + e;
    if (j < L) {
      log[op0 + j].n_in = run;
      run += made[e];
      log[op0 + j].n_new = made[e];
      log[op0 + j].n_out = run;
      log[op0 + j].n_s = 0;
      R.created[j] = 0;  // clean for the next run
    }
  }
  __syncwarp();
  if (lane == 0) {
    const unsigned long long ngroups = ld_volatile(&ctrl->n_pairs);
    const unsigned long long nun = ld_volatile(&ctrl->n_s);
    for (int t = 0; t < 4; ++t) ctrl->tickets[t] = 0;
    // scratch mode: the counter holds every group output; they reach O in k_run_place
    const unsigned long long cap_needed = scratch ? nun + ld_volatile(&ctrl->scr_top) : ld_volatile(&ctrl->cap_needed);
    if (scratch) {
      ctrl->scr_top = 0;
      if (cap_needed > cap) {
        ctrl->cap_needed = cap_needed;
        set_err(ctrl, kErrCapacity, op0);
        return;
      }
    }
    // touched terms (profiling bytes); bit 63 says the run took scratch mode
    log[op0].n_s = ld_volatile(&ctrl->n_side) | (scratch ? kRunLogScratchBit : 0ull);
    if (L > 1) log[op0 + L - 1].n_s = (ngroups == 0) ? 0 : cap_needed - nun;  // group outputs
    const unsigned long long out = (ngroups == 0) ? nun : cap_needed;
    if (trunc_op >= 0) {
      log[trunc_op].n_in = n0 + total;
      log[trunc_op].n_out = out;
    }
    ctrl->n = out;
  }
}

// ---- a group on a warp ------------------------------------------------------------------------
constexpr int kTileWarps = 8;             // warps of a k_run_tiles block
constexpr int kTileSlots = 1 << kRunMaxK;  // slots of shared memory per warp: the largest group's
constexpr size_t kTileSmem = sizeof(unsigned long long) * kTileWarps * kTileSlots;
constexpr unsigned long long kNoSlot = ~0ull;  // a slot without a term (see link_bits for that NaN)

// The gates of a group's coordinates in run order.
struct TileGates {
  double cs[kRunMaxK], sn[kRunMaxK];
  uint16_t gate[kRunMaxK];  // r-th gate: its index in the run
  uint8_t bit[kRunMaxK];    // r-th gate: its coordinate bit
  unsigned k;
};

// A group of at most 32 * NR slots on one warp, slot c = 32 r + lane in lane's register r: members loaded
// through the warp's shared slots, then the gates in run order.  A gate on one of the five low
// coordinate bits pairs lanes (shuffles), on a higher one registers; either way a slot's new value
// is the reference's map_insert on the pair (crates/ppvm-pauli-sum/src/sum/rot1.rs:73,124: eps of a member
// with bit b is +1 for b = 0 under RX, for b = 1 under RZ), with existence tracked apart from the value.
// The survivors of the run's TRUNCATE are counted and written back to the shared slots (the others empty).  Children
// made per gate are added to created (null: not).  In shared memory, a pair per lane and step, the
// same butterflies took 4 times the instructions and a round of shared-memory latency per pair.
template <int NR>
__device__ __noinline__ unsigned tile_survivors(const TileGates& g, unsigned long long* slots,
                                                const uint32_t* __restrict__ mcoord, const double* __restrict__ mcoef,
                                                unsigned cnt, double eps_a, bool trunc, bool wok, double thr,
                                                unsigned* created) {
  const unsigned lane = threadIdx.x & 31;
  double c[NR];
  unsigned ex = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) slots[32 * r + lane] = kNoSlot;
  __syncwarp();
  for (unsigned m = lane; m < cnt; m += 32) slots[mcoord[m]] = link_bits(mcoef[m]);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const unsigned long long u = slots[32 * r + lane];
    c[r] = __longlong_as_double((long long)u);
    ex |= (unsigned)(u != kNoSlot) << r;
  }
  for (unsigned i = 0; i < g.k; ++i) {
    const unsigned t = g.bit[i];
    const double cs = g.cs[i], sn = g.sn[i];
    unsigned made;
    if (t < 5) {
      const bool hi = (lane >> t) & 1u;
      const double in = (hi ? eps_a : -eps_a) * sn;  // what the partner's value is worth here
      const unsigned other = __shfl_xor_sync(kFull, ex, 1u << t);
      made = hi ? 0u : (unsigned)__popc(ex ^ other);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const double o = __shfl_xor_sync(kFull, c[r], 1u << t);
        const double own = __dmul_rn(c[r], cs), got = __dmul_rn(o, in), sum = __dadd_rn(own, got);
        c[r] = (ex >> r) & 1u ? ((other >> r) & 1u ? sum : own) : got;
      }
      ex |= other;
    } else {
      made = 0;
      const double ia = -eps_a * sn, ib = eps_a * sn;
#pragma unroll
      for (int u = 0; (1 << u) < NR; ++u) {
        if ((int)t - 5 != u) continue;
        unsigned low = 0;  // registers with bit u clear
#pragma unroll
        for (int r = 0; r < NR; ++r)
          if (!((r >> u) & 1)) {
            low |= 1u << r;
            const int q = r | 1 << u;
            const bool ea = (ex >> r) & 1u, eb = (ex >> q) & 1u;
            const double ca = c[r], cb = c[q];
            const double oa = __dmul_rn(ca, cs), ga = __dmul_rn(cb, ia), ob = __dmul_rn(cb, cs), gb = __dmul_rn(ca, ib);
            c[r] = ea ? (eb ? __dadd_rn(oa, ga) : oa) : ga;
            c[q] = eb ? (ea ? __dadd_rn(ob, gb) : ob) : gb;
          }
        const unsigned a = ex & low, b = (ex >> (1 << u)) & low;
        made = (unsigned)__popc(a ^ b);
        ex = (a | b) | (a | b) << (1 << u);
      }
    }
    if (created) {
      made = __reduce_add_sync(kFull, made);
      if (lane == 0 && made) atomicAdd(&created[g.gate[i]], made);
    }
  }
  unsigned keep = trunc && !wok ? 0u : ex;
  if (trunc) {
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (fabs(c[r]) < thr) keep &= ~(1u << r);
  }
  const unsigned n = __reduce_add_sync(kFull, __popc(keep));
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) slots[32 * r + lane] = (keep >> r) & 1u ? link_bits(c[r]) : kNoSlot;
  __syncwarp();
  return n;
}

// A group as its warp holds it: key, coordinates (lane t's q: the t-th coordinate qubit).
template <int W>
struct WarpGroup {
  uint64_t v[W], f0[W];
  unsigned k, q;
  bool wok;  // every member's weight (that of v | f0: the coordinates lie inside v) passes the cap

  __device__ __forceinline__ void coordinates(const uint64_t (&Q)[W], unsigned long long maxw) {
    const unsigned lane = threadIdx.x & 31;
    unsigned wt = 0;
    k = q = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t m = v[w] & Q[w];
      const unsigned c = __popcll(m);
      if (lane >= k && lane < k + c) {
        for (unsigned u = k; u < lane; ++u) m &= m - 1;
        q = w * 64 + (unsigned)__ffsll((long long)m) - 1;
      }
      k += c;
      wt += __popcll(v[w] | f0[w]);
    }
    wok = maxw == ~0ull || wt <= maxw;
  }

  // The coordinates' gates, in run order.
  __device__ __forceinline__ void gates(TileGates& G, const RunDesc* rd, const uint16_t* s_gidx) const {
    const unsigned lane = threadIdx.x & 31;
    const unsigned key = lane < k ? s_gidx[q] : 0xFFFFu;
    unsigned rank = 0;
    for (unsigned t = 0; t < k; ++t) rank += __shfl_sync(kFull, key, t) < key;
    __syncwarp();
    if (lane < k) {
      G.bit[rank] = (uint8_t)lane;
      G.gate[rank] = (uint16_t)key;
      G.cs[rank] = rd->cs[key];
      G.sn[rank] = rd->sn[key];
    }
    if (lane == 0) G.k = k;
    __syncwarp();
  }

  // Slots of the warp's shared memory that the group's survivors take.
  __device__ __forceinline__ unsigned slots() const { return k <= 5 ? 32u : 1u << k; }

  __device__ __forceinline__ unsigned survivors(const TileGates& G, unsigned long long* sl, const RunScratch& R,
                                                unsigned start, unsigned cnt, double eps_a, bool trunc, double thr,
                                                unsigned* created) const {
    const uint32_t* mc = R.mcoord + start;
    const double* mv = R.mcoef + start;
    if (k <= 5) return tile_survivors<1>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
    switch (k) {
      case 6: return tile_survivors<2>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
      case 7: return tile_survivors<4>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
      case 8: return tile_survivors<8>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
      case 9: return tile_survivors<16>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
      default: return tile_survivors<32>(G, sl, mc, mv, cnt, eps_a, trunc, wok, thr, created);
    }
  }

  // Writes the survivors to O from index `out` on, in coordinate order: from sl where tile_survivors
  // left them, or (again) after running the group once more through sl.
  __device__ __forceinline__ void emit(const Planes& O, unsigned long long out, uint32_t cls, TileGates& G,
                                       unsigned long long* sl, bool again, const RunDesc* rd, const uint16_t* s_gidx,
                                       const RunScratch& R, unsigned start, unsigned cnt, double eps_a, bool trunc,
                                       double thr) const {
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    if (again) {
      gates(G, rd, s_gidx);
      survivors(G, sl, R, start, cnt, eps_a, trunc, thr, nullptr);
    }
    uint64_t fl[W];  // f with this lane's low coordinate bits; a chunk of 32 slots adds its high ones
#pragma unroll
    for (int w = 0; w < W; ++w) {
      fl[w] = f0[w];
#pragma unroll
      for (unsigned t = 0; t < 5; ++t) {
        const unsigned qt = __shfl_sync(kFull, q, t);
        if (t < k && (int)(qt >> 6) == w && ((lane >> t) & 1u)) fl[w] |= 1ull << (qt & 63);
      }
    }
    const unsigned nchunk = k > 5 ? 1u << (k - 5) : 1u;
    for (unsigned ch = 0; ch < nchunk; ++ch) {
      const unsigned long long u = sl[32 * ch + lane];
      const unsigned bal = __ballot_sync(kFull, u != kNoSlot);
      uint64_t f[W];
#pragma unroll
      for (int w = 0; w < W; ++w) f[w] = fl[w];
      for (unsigned hb = ch; hb; hb &= hb - 1) {
        const unsigned qt = __shfl_sync(kFull, q, 4u + (unsigned)__ffs((int)hb));
#pragma unroll
        for (int w = 0; w < W; ++w)
          if ((int)(qt >> 6) == w) f[w] |= 1ull << (qt & 63);
      }
      const unsigned long long r = out + __popc(bal & lt);
      if (u != kNoSlot && r < O.cap) {
        if (cls == 0) store_key<W>(O, r, f, v);
        else store_key<W>(O, r, v, f);
        O.c[r] = __longlong_as_double((long long)u);
      }
      out += __popc(bal);
    }
    __syncwarp();
  }
};

// ---- lane mode: one group per lane ------------------------------------------------------

// A small group on one lane: its slots in registers (slot c at coef[c], existence bit c of
// ex), its key and coordinate qubits, the gates of its coordinates in run order.
template <int W>
struct LaneGroup {
  uint64_t v[W], f0[W];
  uint16_t pos[kRunLaneK];  // qubit of coordinate bit t (ascending)
  uint8_t ord[kRunLaneK];   // coordinate bits in gate order
  unsigned k;
  bool wok;
  double coef[1 << kRunLaneK];
  unsigned ex;
};

// Loads group g's key on this lane: v, f0, its coordinates; false when it has more than
// kRunLaneK coordinates (the warp runs it instead).
template <int W>
__device__ __forceinline__ bool lane_key(LaneGroup<W>& G, unsigned long long g, const RunDesc* rd,
                                         const RunScratch& R, const uint16_t* s_gidx, bool wcap,
                                         unsigned long long maxw) {
  const uint64_t* gk = R.gkey + g * 2 * W;
  unsigned k = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    G.v[w] = gk[w];
    G.f0[w] = gk[W + w];
    k += __popcll(G.v[w] & rd->Q[w]);
  }
  G.k = k;
  if (k > (unsigned)kRunLaneK) return false;
  unsigned t = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint64_t m = G.v[w] & rd->Q[w];
    while (m) {
      const int b = __ffsll((long long)m) - 1;
      m &= m - 1;
      if (t < (unsigned)kRunLaneK) G.pos[t] = (uint16_t)(w * 64 + b);
      ++t;
    }
  }
  // coordinate bits by gate position (insertion sort of at most 3)
  for (unsigned a = 0; a < k; ++a) G.ord[a] = (uint8_t)a;
  for (unsigned a = 1; a < k; ++a)
    for (unsigned b = a; b > 0 && s_gidx[G.pos[G.ord[b - 1]]] > s_gidx[G.pos[G.ord[b]]]; --b) {
      const uint8_t tmp = G.ord[b - 1];
      G.ord[b - 1] = G.ord[b];
      G.ord[b] = tmp;
    }
  G.wok = true;
  if (wcap) {
    unsigned wt = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) wt += __popcll(G.v[w] | G.f0[w]);
    G.wok = wt <= maxw;
  }
  return true;
}

// The members and the butterfly of a small group on its lane, the same arithmetic in the same
// gate order as tile_survivors; children made per gate go to s_created.
template <int W>
__device__ __forceinline__ void lane_run(LaneGroup<W>& G, unsigned start, unsigned cnt, uint32_t cls,
                                         const RunScratch& R, const uint16_t* s_gidx, const double* s_cs,
                                         const double* s_sn, unsigned* s_created) {
  constexpr int SZ = 1 << kRunLaneK;
  G.ex = 0;
#pragma unroll
  for (int c = 0; c < SZ; ++c) G.coef[c] = 0.0;
  for (uint32_t m = 0; m < cnt; ++m) {
    const unsigned c = R.mcoord[start + m];
    const double v = R.mcoef[start + m];
#pragma unroll
    for (int e = 0; e < SZ; ++e)
      if (e == (int)c) G.coef[e] = v;
    G.ex |= 1u << c;
  }
  const double eps_a = cls == 0 ? 1.0 : -1.0, eps_b = -eps_a;
  for (unsigned r = 0; r < G.k; ++r) {
    const unsigned t = G.ord[r];
    const unsigned j = s_gidx[G.pos[t]];
    const unsigned bit = 1u << t;
    const double cs = s_cs[j], sn = s_sn[j];
    unsigned made = 0;
#pragma unroll
    for (int a = 0; a < SZ; ++a) {
      if ((a & (int)bit) || a >= (1 << G.k)) continue;
      const int b = a | (int)bit;
      double ca = 0.0, cb = 0.0;
#pragma unroll
      for (int e = 0; e < SZ; ++e) {  // registers only: slots picked by compile-time index
        if (e == a) ca = G.coef[e];
        if (e == b) cb = G.coef[e];
      }
      const bool ea = (G.ex >> a) & 1u, eb = (G.ex >> b) & 1u;
      double na = ca, nb = cb;
      if (ea && eb) {
        na = __dadd_rn(__dmul_rn(ca, cs), __dmul_rn(cb, eps_b * sn));
        nb = __dadd_rn(__dmul_rn(cb, cs), __dmul_rn(ca, eps_a * sn));
      } else if (ea) {
        na = __dmul_rn(ca, cs);
        nb = __dmul_rn(ca, eps_a * sn);
        G.ex |= 1u << b;
        ++made;
      } else if (eb) {
        nb = __dmul_rn(cb, cs);
        na = __dmul_rn(cb, eps_b * sn);
        G.ex |= 1u << a;
        ++made;
      }
#pragma unroll
      for (int e = 0; e < SZ; ++e) {
        if (e == a) G.coef[e] = na;
        if (e == b) G.coef[e] = nb;
      }
    }
    if (made) atomicAdd(&s_created[j], made);
  }
}

// Whether slot c of a small group is written (it exists and passes the run's TRUNCATE).
template <int W>
__device__ __forceinline__ bool lane_keep(const LaneGroup<W>& G, int c, int trunc, double thr) {
  if (!((G.ex >> c) & 1u)) return false;
  if (!trunc) return true;
  double v = 0.0;
#pragma unroll
  for (int e = 0; e < (1 << kRunLaneK); ++e)
    if (e == c) v = G.coef[e];
  return G.wok && !(fabs(v) < thr);
}

// Writes a small group's survivors, in coordinate order, to D from index out on.
template <int W>
__device__ __forceinline__ void lane_write(const LaneGroup<W>& G, Planes D, unsigned long long out, uint32_t cls,
                                           int trunc, double thr) {
#pragma unroll
  for (int c = 0; c < (1 << kRunLaneK); ++c) {
    if (c >= (1 << G.k) || !lane_keep<W>(G, c, trunc, thr)) continue;
    if (out < D.cap) {
      uint64_t f[W], x[W], z[W];
#pragma unroll
      for (int w = 0; w < W; ++w) f[w] = G.f0[w];
      for (unsigned t = 0; t < G.k; ++t)
        if ((c >> t) & 1) {
          const unsigned q = G.pos[t];
#pragma unroll
          for (int w = 0; w < W; ++w)
            if (w == (int)(q >> 6)) f[w] |= 1ull << (q & 63);
        }
#pragma unroll
      for (int w = 0; w < W; ++w) {
        x[w] = cls == 0 ? f[w] : G.v[w];
        z[w] = cls == 0 ? G.v[w] : f[w];
      }
      store_key<W>(D, out, x, z);
      D.c[out] = G.coef[c];
    }
    ++out;
  }
}

// Whether a run's groups go one per lane: forced (mode 3), or chosen from kRunTileMinGroups groups on, by
// how many of them are too large for a lane.  The warp runs those one after the other, and the order
// puts alike groups side by side, so that one warp may get 32 of them: 0.16 ms of tail at 4 to 6
// coordinates, 0.5 at 8, 2.3 at 10, while the other lanes' groups cost nearly nothing.  RX runs of 10
// gates on groups of one coordinate and a share of K, group kernel and placement in us, tiles / lanes:
//   none large: always lanes (3 gates, 3.0M terms in full groups on 200 qubits: 1920 / 260);
//   300,000 groups, scattered: 1 % of K = 5 598 / 101 (144 qubits), of K = 10 1834 / 687, 20 % of K = 6
//   531 / 339 (40 qubits), all of K = 5 602 / 813; side by side, the worst: 0.2 % of K = 10 2365 / 2385;
//   40,000 groups, scattered: 5 % of K = 4 94 / 44, 20 % of K = 7 139 / 181; side by side: 5 % of K = 4
//   92 / 187, of K = 8 149 / 646.
// So lanes are taken when no group is large; in runs of mostly single members up to one in 8 may be (all
// large: 1.3M groups of 90 slots 23.7 ms, 12.4 in tiles); from kRunLaneMany groups on, where tiles leave their
// order to k_run_place, one in 16 whatever the members (at one in 6 a kicked-Ising layer of 4M terms takes 12.6
// ms in tiles and 14.8 in lanes).
constexpr unsigned long long kRunLaneMany = 1ull << 18;
struct RunCounts {
  unsigned long long groups, members, large, slots, untouched;
};
__device__ __forceinline__ RunCounts run_counts(const Ctrl* ctrl, unsigned turn) {
  return {ld_volatile(&ctrl->n_pairs), ld_volatile(&ctrl->n_side), ld_volatile(&ctrl->run_large[turn]),
          ld_volatile(&ctrl->run_slots[turn]), ld_volatile(&ctrl->n_s)};
}
// The group kernels and k_run_place read the same counts and decide alike; those not needed return.
__device__ __forceinline__ bool run_lanes(const RunCounts& c, unsigned mode) {
  if (mode != 0) return mode == 3;
  if (c.groups < kRunTileMinGroups) return false;
  return c.large == 0 || (2 * c.members < 3 * c.groups && 8 * c.large <= c.groups) ||
         (c.groups >= kRunLaneMany && 16 * c.large <= c.groups);
}

// Whether tiles leave their order to k_run_place (scratch mode): from scratch_min groups on, unless the
// groups are large.  Placing moves every term once more: 1.3M groups of 90 slots (1.1e8 terms) 13.1 + 5.9 ms,
// 12.4 in order; 2.6M groups of a kicked-Ising layer 4.3 + 1.6, 6.9 in order.  A threshold set below the
// default asks for scratch mode whatever the groups.
constexpr unsigned long long kScratchSlots = 32;
__device__ __forceinline__ bool run_scratch(const RunCounts& c, unsigned long long scratch_min) {
  return c.groups >= scratch_min && (scratch_min < kRunLaneMany || c.slots <= kScratchSlots * c.groups);
}

// One group per lane, for runs of many small groups (run_lanes).  A warp takes 32 consecutive groups
// by one ticket.  A group of at most kRunLaneK coordinates runs on its lane alone; the larger ones are
// run by the whole warp, one after the other, and keep their survivors in the warp's slots as long
// as these hold them (the rest is run again to be written).  One warp scan and one look-back place
// the 32 groups.
template <int W>
__global__ void __launch_bounds__(kRunWarps * 32, 5)
k_run_lanes(Planes O, Ctrl* ctrl, const RunDesc* rd, RunScratch R, int trunc, double thr, unsigned long long maxw,
            unsigned long long* ts, unsigned epoch, int op, int trunc_op, OpLog* log, unsigned mode, unsigned turn) {
  pdl_wait();
  __shared__ unsigned long long s_slot[kRunWarps][kTileSlots];
  __shared__ TileGates s_g[kRunWarps];
  __shared__ unsigned s_created[kRunMaxGates];
  __shared__ double s_cs[kRunMaxGates], s_sn[kRunMaxGates];
  __shared__ uint16_t s_gidx[64 * W];  // qubit -> its gate's index in the run
  const RunCounts rc = run_counts(ctrl, turn);
  if (ld_volatile_int(&ctrl->err) || !run_lanes(rc, mode)) return;
  const unsigned long long ngroups = rc.groups, ubase = rc.untouched;  // untouched survivors go first
  const unsigned long long ntiles = (ngroups + 31) / 32;
  const unsigned long long want = (ntiles + kRunWarps - 1) / kRunWarps;
  const unsigned blocks = (unsigned)(want < 1 ? 1 : want < gridDim.x ? want : gridDim.x);
  if (blockIdx.x >= blocks) return;
  const uint32_t L = rd->L, cls = rd->cls;
  for (unsigned j = threadIdx.x; j < L; j += blockDim.x) {
    s_created[j] = 0;
    s_cs[j] = rd->cs[j];
    s_sn[j] = rd->sn[j];
    s_gidx[rd->q[j]] = (uint16_t)j;  // the qubits of a run are distinct
  }
  __syncthreads();
  uint64_t Q[W];
#pragma unroll
  for (int w = 0; w < W; ++w) Q[w] = rd->Q[w];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool wcap = maxw != ~0ull;
  const double eps_a = cls == 0 ? 1.0 : -1.0;
  TileGates& G = s_g[warp];
  unsigned long long* slots = s_slot[warp];
  for (;;) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(&ctrl->tickets[2], 1ull);
    t = __shfl_sync(kFull, t, 0);
    if (t >= ntiles) break;
    const unsigned long long g = t * 32 + lane;
    const bool valid = g < ngroups;
    LaneGroup<W> LG;
    bool small = false;
    unsigned mine = 0, gs = 0, gc = 0;
    if (valid) {
      gs = R.g_start[g];
      gc = R.g_cnt[g];
      small = lane_key<W>(LG, g, rd, R, s_gidx, wcap, maxw);
      if (small) {
        lane_run<W>(LG, gs, gc, cls, R, s_gidx, s_cs, s_sn, s_created);
#pragma unroll
        for (int c = 0; c < (1 << kRunLaneK); ++c)
          if (c < (1 << LG.k)) mine += lane_keep<W>(LG, c, trunc, thr);
      }
    }
    const unsigned big = __ballot_sync(kFull, valid && !small);
    unsigned off = kTileSlots, used = 0;  // a large group's slots (kTileSlots: none kept)
    auto large = [&](WarpGroup<W>& B, unsigned l) {  // lane l's group on the warp
#pragma unroll
      for (int w = 0; w < W; ++w) {
        B.v[w] = __shfl_sync(kFull, LG.v[w], l);
        B.f0[w] = __shfl_sync(kFull, LG.f0[w], l);
      }
      B.coordinates(Q, maxw);
    };
    for (unsigned bb = big; bb; bb &= bb - 1) {
      const unsigned l = (unsigned)(__ffs(bb) - 1);
      WarpGroup<W> B;
      large(B, l);
      B.gates(G, rd, s_gidx);
      const unsigned size = B.slots();
      const bool fits = used + size <= (unsigned)kTileSlots;
      if (!fits) {  // it goes through the slots from the first on: what was kept there is run again too
        off = kTileSlots;
        used = kTileSlots;
      }
      const unsigned at = fits ? used : 0u;
      const unsigned n = B.survivors(G, slots + at, R, __shfl_sync(kFull, gs, l), __shfl_sync(kFull, gc, l), eps_a,
                                     trunc, thr, s_created);
      if (fits) used += size;
      if (lane == l) {
        mine = n;
        off = fits ? at : (unsigned)kTileSlots;
      }
    }
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(kFull, incl, o);
      if (lane >= (unsigned)o) incl += v;
    }
    const unsigned total = __shfl_sync(kFull, incl, 31);
    const unsigned pre = incl - mine;
    const unsigned long long base = ubase + warp_lookback(ts, t, total, epoch, ctrl, op);
    if (valid && small) lane_write<W>(LG, O, base + pre, cls, trunc, thr);
    for (unsigned bb = __ballot_sync(kFull, valid && !small && mine); bb; bb &= bb - 1) {
      const unsigned l = (unsigned)(__ffs(bb) - 1);
      const unsigned long long at = base + __shfl_sync(kFull, pre, l);
      const unsigned o = __shfl_sync(kFull, off, l);
      WarpGroup<W> B;
      large(B, l);
      const bool again = o >= (unsigned)kTileSlots;
      B.emit(O, at, cls, G, slots + (again ? 0u : o), again, rd, s_gidx, R, __shfl_sync(kFull, gs, l),
             __shfl_sync(kFull, gc, l), eps_a, trunc, thr);
    }
    if (t == ntiles - 1 && lane == 0) {
      ctrl->cap_needed = base + total;
      if (base + total > O.cap) set_err(ctrl, kErrCapacity, op);
    }
    __syncwarp();
  }
  __syncthreads();
  for (unsigned j = threadIdx.x; j < L; j += blockDim.x)
    if (s_created[j]) atomicAdd(&R.created[j], (unsigned long long)s_created[j]);
  if (last_of_blocks(&ctrl->done, blocks) && warp == 0) run_commit(ctrl, R, op, (int)L, trunc_op, log, false, O.cap);
}

constexpr unsigned long long kTileManyGroups = 1ull << 15;  // from here on a warp takes several groups of a tile

// The groups of a run in tiles of consecutive groups, a tile per block and ticket, PER groups per warp:
// keys and coordinates, the butterflies in registers (tile_survivors), one look-back per tile for
// the output offset, and the survivors written chunk by chunk of 32 slots, in coordinate order.
// PER is 1 below kTileManyGroups groups, where a tile's latency is what counts (ticket, dependent
// loads, look-back, about a microsecond each), and up to 4 (2 above 256 qubits) from there on, where the
// look-backs and barriers per group do, as far as the groups fit a warp's slots on average (60,000
// groups of 256 slots: 325 us with 4, 416 with 1): the warp's keys, starts and members then come in one
// load each.  A warp whose groups do not fit its slots together runs those that are left out again to
// write them.  On the 12 x 12 headline (5,400 groups of 120 slots, 640,000 terms out) a run takes 50 us;
// one warp per group in shared memory, placed group by group, took 72.
// 1024 slots a warp and two blocks an SM: with 512 slots a group of 10 coordinates went through them
// twice and was run three times (5,400 of them 357 us instead of 121; 1.1e8 terms of an unbudgeted 10 x 10
// circuit 28.9 ms instead of 12.4); three blocks leave 80 registers, whose spills and less L1 make the
// headline 2.75 ms instead of 2.68 and a kicked-Ising layer of 4M terms 12.9 instead of 12.0.
template <int W>
__global__ void __launch_bounds__(kTileWarps * 32, 2)
k_run_tiles(Planes O, Planes S, Ctrl* ctrl, const RunDesc* rd, RunScratch R, int trunc, double thr,
            unsigned long long maxw, unsigned long long* ts, unsigned epoch, int op, int trunc_op, OpLog* log,
            unsigned long long scratch_min, unsigned mode, unsigned turn) {
  pdl_wait();
  constexpr int BLOCK = kTileWarps * 32;
  constexpr unsigned MANY = W <= 4 ? 4 : 2;  // a warp's keys: MANY * 2W <= 32 words, one per lane
  extern __shared__ unsigned long long s_tiles[];  // kTileWarps * kTileSlots
  __shared__ TileGates s_g[kTileWarps];
  __shared__ unsigned s_created[kRunMaxGates];
  __shared__ uint16_t s_gidx[64 * W];  // qubit -> its gate's index in the run
  __shared__ unsigned s_cnt[kTileWarps], s_tile;
  __shared__ unsigned long long s_base;
  const RunCounts rc = run_counts(ctrl, turn);
  if (ld_volatile_int(&ctrl->err) || run_lanes(rc, mode)) return;
  const unsigned long long ngroups = rc.groups, ubase = rc.untouched;  // untouched survivors go first
  const bool scratch = run_scratch(rc, scratch_min);  // the same in every block
  unsigned per = scratch || ngroups >= kTileManyGroups ? MANY : 1u;
  while (per > 1 && per * rc.slots > (unsigned long long)kTileSlots * ngroups) per >>= 1;  // so many fit on average
  const unsigned long long ntiles = (ngroups + kTileWarps * per - 1) / (kTileWarps * per);
  const unsigned blocks = (unsigned)(ntiles < 1 ? 1 : ntiles < gridDim.x ? ntiles : gridDim.x);
  if (blockIdx.x >= blocks) return;
  const uint32_t L = rd->L, cls = rd->cls;
  for (unsigned j = threadIdx.x; j < L; j += BLOCK) {
    s_created[j] = 0;
    s_gidx[rd->q[j]] = (uint16_t)j;  // the qubits of a run are distinct
  }
  uint64_t Q[W];
#pragma unroll
  for (int w = 0; w < W; ++w) Q[w] = rd->Q[w];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double eps_a = cls == 0 ? 1.0 : -1.0;
  TileGates& G = s_g[warp];
  unsigned long long* slots = s_tiles + warp * kTileSlots;
  // The warp's groups of a tile; per lane b: group b's start, members, survivors and slots (kTileSlots:
  // none kept), beside one word of the warp's keys.
  struct Held {
    uint64_t kw;
    unsigned gs, gc, n, off, ng;
  } H;
  auto load = [&](WarpGroup<W>& B, unsigned b) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      B.v[w] = __shfl_sync(kFull, H.kw, b * 2 * W + w);
      B.f0[w] = __shfl_sync(kFull, H.kw, b * 2 * W + W + w);
    }
    B.coordinates(Q, maxw);
  };
  // Groups g0, g0 + 1, ... (at most per): run and counted; returns their survivors.
  auto count = [&](unsigned long long g0) -> unsigned {
    H.ng = g0 >= ngroups ? 0u : (unsigned)(ngroups - g0 < per ? ngroups - g0 : per);
    H.kw = lane < H.ng * 2 * W ? R.gkey[g0 * 2 * W + lane] : 0ull;
    H.gs = lane < H.ng ? R.g_start[g0 + lane] : 0u;
    H.gc = lane < H.ng ? R.g_cnt[g0 + lane] : 0u;
    H.n = 0;
    H.off = kTileSlots;
    if (H.ng > 1) {  // the members of all the warp's groups lie together: on their way while the keys are read
      const unsigned m0 = __shfl_sync(kFull, H.gs, 0);
      const unsigned m1 = __shfl_sync(kFull, H.gs, H.ng - 1) + __shfl_sync(kFull, H.gc, H.ng - 1);
      if (m0 + lane * 4 < m1) {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(R.mcoef + m0 + lane * 4));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(R.mcoord + m0 + lane * 4));
      }
    }
    unsigned used = 0, mine = 0;
    for (unsigned b = 0; b < H.ng; ++b) {
      WarpGroup<W> B;
      load(B, b);
      B.gates(G, rd, s_gidx);
      const unsigned size = B.slots();
      const bool fits = used + size <= (unsigned)kTileSlots;
      if (!fits) {  // it goes through the slots from the first on: what was kept there is run again too
        if (lane < b) H.off = kTileSlots;
        used = kTileSlots;
      }
      const unsigned off = fits ? used : 0u;
      const unsigned n = B.survivors(G, slots + off, R, __shfl_sync(kFull, H.gs, b), __shfl_sync(kFull, H.gc, b), eps_a,
                                     trunc, thr, s_created);
      if (fits) used += size;
      if (lane == b) {
        H.n = n;
        H.off = fits ? off : (unsigned)kTileSlots;
      }
      mine += n;
    }
    return mine;
  };
  // Their survivors to D, from index `out` on.
  auto emit = [&](const Planes& D, unsigned long long out) {
    for (unsigned b = 0; b < H.ng; ++b) {
      const unsigned n = __shfl_sync(kFull, H.n, b);
      if (n == 0) continue;
      const unsigned off = __shfl_sync(kFull, H.off, b);
      const bool again = off >= (unsigned)kTileSlots;
      WarpGroup<W> B;
      load(B, b);
      B.emit(D, out, cls, G, slots + (again ? 0u : off), again, rd, s_gidx, R, __shfl_sync(kFull, H.gs, b),
             __shfl_sync(kFull, H.gc, b), eps_a, trunc, thr);
      out += n;
    }
  };
  __syncthreads();
  if (scratch) {
    // many groups: the warps work on their own, each one's survivors to the scratch planes wherever a
    // counter puts them; k_run_place moves every group's block to its place
    for (;;) {
      unsigned long long t = 0;
      if (lane == 0) t = atomicAdd(&ctrl->tickets[2], 1ull);
      const unsigned long long g0 = __shfl_sync(kFull, t, 0) * per;
      if (g0 >= ngroups) break;
      const unsigned mine = count(g0);
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(&ctrl->scr_top, (unsigned long long)mine);
      at = __shfl_sync(kFull, at, 0);
      unsigned pre = H.n;  // lane b: survivors of the groups up to b
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        const unsigned u = __shfl_up_sync(kFull, pre, o);
        if (lane >= (unsigned)o) pre += u;
      }
      if (lane < H.ng) {
        const unsigned long long b = at + pre - H.n;
        R.g_rep[g0 + lane] = (uint32_t)(b < 0xFFFFFFFFull ? b : 0xFFFFFFFFull);  // (< capacity < 2^32)
        R.g_fill[g0 + lane] = H.n;
      }
      emit(S, at);
      __syncwarp();
    }
  } else {
    while (ntiles) {
      const unsigned tile = next_tile(&ctrl->tickets[2], &s_tile);
      if (tile >= ntiles) break;
      const unsigned mine = count(((unsigned long long)tile * kTileWarps + warp) * per);
      if (lane == 0) s_cnt[warp] = mine;
      __syncthreads();
      unsigned total = 0, before = 0;
#pragma unroll
      for (int w = 0; w < kTileWarps; ++w) {
        const unsigned n = s_cnt[w];
        if (w < (int)warp) before += n;
        total += n;
      }
      const unsigned long long base = ubase + lookback(ts, tile, total, epoch, ctrl, op, &s_base);
      if (tile == ntiles - 1 && threadIdx.x == 0) {
        ctrl->cap_needed = base + total;
        if (base + total > O.cap) set_err(ctrl, kErrCapacity, op);
      }
      emit(O, base + before);
    }
  }
  __syncthreads();
  for (unsigned j = threadIdx.x; j < L; j += BLOCK)
    if (s_created[j]) atomicAdd(&R.created[j], (unsigned long long)s_created[j]);
  if (last_of_blocks(&ctrl->done, blocks) && warp == 0)
    run_commit(ctrl, R, op, (int)L, trunc_op, log, scratch, O.cap);
}

// Scratch mode of a fused run (many groups): k_run_tiles left each group's survivors in a
// contiguous block of the scratch planes S, at R.g_rep[g] (R.g_fill[g] of them).  Groups are
// taken in tiles of BLOCK * ITEMS, in group order: one decoupled look-back per tile gives the
// tile's output offset, a block scan the offsets of its groups, and the block's warps then
// copy whole blocks (one term per lane) to O.  The result is the look-back mode's, term for
// term, at one look-back per tile instead of one per group.
template <int W, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK)
k_run_place(Planes S, Planes O, Ctrl* ctrl, RunScratch R, unsigned long long scratch_min, unsigned long long* ts,
            unsigned epoch, int op, unsigned mode, unsigned turn) {
  pdl_wait();
  constexpr int NW = BLOCK / 32;
  constexpr int TILE = BLOCK * ITEMS;
  __shared__ unsigned s_tile;
  __shared__ unsigned long long s_slot;
  __shared__ unsigned s_wsum[ITEMS * NW + 1];
  __shared__ uint32_t s_src[TILE], s_cnt[TILE];
  __shared__ unsigned long long s_dst[TILE];
  __shared__ int s_skip;
  if (threadIdx.x == 0) {
    const RunCounts rc = run_counts(ctrl, turn);
    s_skip = ld_volatile_int(&ctrl->err) || rc.groups == 0 || !run_scratch(rc, scratch_min) || run_lanes(rc, mode);
  }
  __syncthreads();
  if (s_skip) return;  // the same in every block (look-back mode, or an earlier error)
  const unsigned long long ngroups = ld_volatile(&ctrl->n_pairs), ubase = ld_volatile(&ctrl->n_s);
  const unsigned long long ntiles = (ngroups + TILE - 1) / TILE;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (;;) {
    const unsigned tile = next_tile(&ctrl->tickets[0], &s_tile);
    if (tile >= ntiles) break;
    const unsigned long long base = (unsigned long long)tile * TILE;
    unsigned cnt[ITEMS], pre[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long gi = base + (unsigned long long)k * BLOCK + threadIdx.x;
      cnt[k] = gi < ngroups ? R.g_fill[gi] : 0u;
      unsigned v = cnt[k];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, v, o);
        if (lane >= (unsigned)o) v += t;
      }
      pre[k] = v - cnt[k];
      if (lane == 31) s_wsum[k * NW + warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // group order inside the tile: item k, then warp, then lane
      unsigned run = 0;
      for (int e = 0; e < ITEMS * NW; ++e) {
        const unsigned t = s_wsum[e];
        s_wsum[e] = run;
        run += t;
      }
      s_wsum[ITEMS * NW] = run;
    }
    __syncthreads();
    const unsigned long long excl = lookback(ts, tile, s_wsum[ITEMS * NW], epoch, ctrl, op, &s_slot);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const unsigned long long gi = base + (unsigned long long)k * BLOCK + threadIdx.x;
      const int q = k * BLOCK + threadIdx.x;
      s_cnt[q] = cnt[k];
      s_src[q] = gi < ngroups ? R.g_rep[gi] : 0u;
      s_dst[q] = ubase + excl + s_wsum[k * NW + warp] + pre[k];
    }
    __syncthreads();
    for (int q = warp; q < TILE; q += NW) {  // one group per warp, one term per lane
      const unsigned n = s_cnt[q];
      const unsigned long long src = s_src[q], dst = s_dst[q];
      for (unsigned e = lane; e < n; e += 32) {
        const unsigned long long a = src + e, b = dst + e;
        if (a < S.cap && b < O.cap) {  // the commit checked that everything fits
#pragma unroll
          for (int w = 0; w < W; ++w) {
            O.x[(unsigned long long)w * O.cap + b] = S.x[(unsigned long long)w * S.cap + a];
            O.z[(unsigned long long)w * O.cap + b] = S.z[(unsigned long long)w * S.cap + a];
          }
          O.c[b] = S.c[a];
        }
      }
    }
    __syncthreads();  // the tile arrays are rewritten by the block's next tile
  }
  if (last_block_done(&ctrl->done) && threadIdx.x == 0) ctrl->tickets[0] = 0;
}

}  // namespace ppvm
