// learned.cu — the term-priority network of learned truncation: parameters, training
// (forward, backward and Adam as hand-written kernels, BF16 tensor cores with FP32
// accumulation) and batch prediction.  The network scores a term by the predicted
// log10 |contribution| of the term to <O> at the end of the circuit; ppvm_truncate_budget
// (engine.cu) uses the score as the priority of a term-budget truncation.
//
// No counterpart in the reference: ppvm truncates by |coefficient| and Pauli weight only
// (crates/ppvm-pauli-sum/src/strategy.rs:12-170).

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ppvm_cuda.h"
#include "mlp.cuh"

namespace ppvm {
void set_last_error(const std::string& msg);
}

using namespace ppvm;

struct ppvm_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  float* params = nullptr;  // FP32 master copy (flat)
  float* m = nullptr;       // Adam moments
  float* v = nullptr;
  float* grads = nullptr;
  float* loss = nullptr;    // [0] = sum of squared errors of the last pass
  float* slabs = nullptr;   // [kMaxTrainBlocks][kSlab]: per-block gradient partials + loss
  MlpWeights* w = nullptr;  // packed device weights
  int step = 0;
  float* d_feats = nullptr;  // training / prediction inputs (grown on demand)
  float* d_tgt = nullptr;
  uint32_t* d_order = nullptr;  // sample orders and learning rates of two epochs, and their pinned twin
  uint32_t* h_order = nullptr;
  size_t order_cap = 0, pinned_words = 0;
  cudaEvent_t half_free[2] = {nullptr, nullptr};  // each half's last upload
  float* d_out = nullptr;
  size_t data_cap = 0;
};

namespace ppvm {
const MlpWeights* mlp_device_weights(const ppvm_mlp* m) { return m ? m->w : nullptr; }
int mlp_device(const ppvm_mlp* m) { return m ? m->device : -1; }
}  // namespace ppvm

namespace {

constexpr int kTrainWarps = 4;
constexpr int kMaxTrainBlocks = 296;
constexpr int kSlab = (kMlpParams + 1 + 3) & ~3;  // the parameters' gradients, then the block's loss

ppvm_status mfail(ppvm_status s, const std::string& msg) {
  ppvm::set_last_error(msg);
  return s;
}

#define MCUDA(expr)                                                                          \
  do {                                                                                       \
    cudaError_t e_ = (expr);                                                                 \
    if (e_ != cudaSuccess)                                                                   \
      return mfail(e_ == cudaErrorMemoryAllocation ? PPVM_ECAPACITY : PPVM_ECUDA,            \
                   std::string(#expr) + ": " + cudaGetErrorString(e_));                      \
  } while (0)

#define MTRY(expr)                \
  do {                            \
    ppvm_status s_ = (expr);      \
    if (s_ != PPVM_OK) return s_; \
  } while (0)

// FP32 master parameters -> packed BF16/FP32 device weights.
__global__ void k_mlp_pack(const float* p, MlpWeights* w) {
  for (int i = threadIdx.x; i < kMlpH * kLdW1; i += blockDim.x) {
    const int n = i / kLdW1, k = i % kLdW1;
    w->w1[i] = __float2bfloat16_rn(k < kMlpIn ? p[kOffW1 + n * kMlpIn + k] : 0.0f);
  }
  for (int i = threadIdx.x; i < kMlpH * kMlpH; i += blockDim.x) {
    const int n = i / kMlpH, k = i % kMlpH;
    const __nv_bfloat16 b = __float2bfloat16_rn(p[kOffW2 + i]);
    w->w2[n * kLdW2 + k] = b;
    w->w2t[k * kLdW2 + n] = b;
  }
  for (int i = threadIdx.x; i < kMlpH; i += blockDim.x) {
    w->b1[i] = p[kOffB1 + i];
    w->b2[i] = p[kOffB2 + i];
    w->w3[i] = p[kOffW3 + i];
  }
  if (threadIdx.x == 0) w->b3 = p[kOffB3];
}

// One Adam update: the moments in place, the new parameter returned.
__device__ __forceinline__ float adam_step(float p, float& m, float& v, float g, float lr_t, float b1, float b2,
                                           float eps) {
  m = b1 * m + (1.0f - b1) * g;
  v = b2 * v + (1.0f - b2) * g * g;
  return p - lr_t * m / (sqrtf(v) + eps);
}

// Parameter i's packed copies (W1's zero padding is set once by k_mlp_pack).
__device__ __forceinline__ void pack_param(MlpWeights* w, int i, float pi) {
  if (i < kOffB1) {
    const int n = (i - kOffW1) / kMlpIn, k = (i - kOffW1) % kMlpIn;
    w->w1[n * kLdW1 + k] = __float2bfloat16_rn(pi);
  } else if (i < kOffW2) {
    w->b1[i - kOffB1] = pi;
  } else if (i < kOffB2) {
    const int n = (i - kOffW2) / kMlpH, k = (i - kOffW2) % kMlpH;
    const __nv_bfloat16 b = __float2bfloat16_rn(pi);
    w->w2[n * kLdW2 + k] = b;
    w->w2t[k * kLdW2 + n] = b;
  } else if (i < kOffW3) {
    w->b2[i - kOffB2] = pi;
  } else if (i < kOffB3) {
    w->w3[i - kOffW3] = pi;
  } else {
    w->b3 = pi;
  }
}

// Adam on the flat parameter vector, one thread per parameter: the minibatch gradient (the
// training blocks' slabs summed in block order), the update, and the parameter's own packed
// copies written, so no thread waits for another.
__global__ void __launch_bounds__(256) k_mlp_adam(float* p, float* m, float* v, const float* slabs, int nslabs,
                                                  float* loss, MlpWeights* w, float lr_t, float b1, float b2,
                                                  float eps) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kMlpParams) return;
  float gi = 0.0f;  // the minibatch gradient: slabs summed in block order
  for (int b = 0; b < nslabs; ++b) gi += slabs[(size_t)b * kSlab + i];
  if (i == kMlpParams) {  // the loss slot
    *loss += gi;
    return;
  }
  float mi = m[i], vi = v[i];
  const float pi = adam_step(p[i], mi, vi, gi, lr_t, b1, b2, eps);
  m[i] = mi;
  v[i] = vi;
  p[i] = pi;
  pack_param(w, i, pi);
}

// A lane's share of a 16-row sample tile: half of row r0 + lane/2's features, and the targets of
// rows r0 + g and r0 + g + 8 (0 past the end).  Loaded apart from its use, so that the loads of
// the next minibatch's tile are in flight across the update of this one.
struct SampleTile {
  float4 f;
  float tg[2];
};
__device__ __forceinline__ void load_samples(SampleTile& S, const float* feats, const float* targets,
                                             const uint32_t* order, unsigned long long r0, unsigned long long rend) {
  const int lane = threadIdx.x & 31;
  const unsigned long long row = r0 + (lane >> 1);
  S.f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (row < rend) {
    const unsigned long long s = order ? order[row] : row;
    S.f = *reinterpret_cast<const float4*>(feats + s * kMlpIn + 4 * (lane & 1));
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned long long r = r0 + (lane >> 2) + 8 * h;
    S.tg[h] = targets && r < rend ? targets[order ? order[r] : r] : 0.0f;
  }
}

// The tile's features as a BF16 [16][16] tile (upper 8 columns 0).
__device__ __forceinline__ void stage_features(__nv_bfloat16* sX, const SampleTile& S) {
  const int lane = threadIdx.x & 31;
  uint2* row = reinterpret_cast<uint2*>(sX + (lane >> 1) * kMlpK1);
  row[lane & 1] = make_uint2(pack_bf16(S.f.x, S.f.y), pack_bf16(S.f.z, S.f.w));
  row[2 + (lane & 1)] = make_uint2(0u, 0u);
  __syncwarp();
}

// Row stride of the warps' [16][64] staging tiles: 144 bytes, so that the 8 rows of an ldmatrix land
// in different banks.
constexpr int kStageLd = kMlpH + 8;
constexpr int kTileHalves = 16 * kMlpK1 + 2 * 16 * kStageLd;  // sX, sD, sH of a warp

// Four transposed 8 x 8 blocks; lane i gives the address of row i % 8 of block i / 8.
__device__ __forceinline__ void ldmatrix4_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

// sG[i] += v, or sG[i] = v for a warp's first tile (FIRST: nothing has been added yet).
template <bool FIRST>
__device__ __forceinline__ void acc_to(float* sG, int i, float v) {
  sG[i] = FIRST ? v : sG[i] + v;
}
// The same for entries i (even), i + 1.
template <bool FIRST>
__device__ __forceinline__ void acc_to2(float* sG, int i, float lo, float hi) {
  float2* d = reinterpret_cast<float2*>(sG + i);
  const float2 o = FIRST ? make_float2(0.0f, 0.0f) : *d;
  *d = FIRST ? make_float2(lo, hi) : make_float2(o.x + lo, o.y + hi);
}

// Sums a per-thread column partial over the 8 row groups of the warp (lanes with equal t)
// and adds it to the CTA gradient: cols 8j + 2t, 8j + 2t + 1 of vector `off`.
template <bool FIRST>
__device__ __forceinline__ void add_cols(float* sG, int off, int j, float lo, float hi) {
  lo += __shfl_xor_sync(0xffffffffu, lo, 4);
  lo += __shfl_xor_sync(0xffffffffu, lo, 8);
  lo += __shfl_xor_sync(0xffffffffu, lo, 16);
  hi += __shfl_xor_sync(0xffffffffu, hi, 4);
  hi += __shfl_xor_sync(0xffffffffu, hi, 8);
  hi += __shfl_xor_sync(0xffffffffu, hi, 16);
  const int lane = threadIdx.x & 31;
  if (lane < 4) {  // the warp's own gradient copy: each entry always written by the same lane
    acc_to<FIRST>(sG, off + 8 * j + 2 * lane, lo);
    acc_to<FIRST>(sG, off + 8 * j + 2 * lane + 1, hi);
  }
}

// Forward + backward of one warp over a 16-sample tile at row r0 (rows below `end`): gradients of the
// squared error scaled by inv_n into the warp's copy sG, the squared errors into lsum.
template <bool FIRST>
__device__ __forceinline__ void train_tile(const MlpWeights& W, const SampleTile& S, unsigned long long r0,
                                           unsigned long long end, float inv_n, __nv_bfloat16* sX, float* sG,
                                           float& lsum) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  __nv_bfloat16* sD = sX + 16 * kMlpK1;   // [16][64]: dZ2, later dZ1
  __nv_bfloat16* sH = sD + 16 * kStageLd;  // [16][64]: H1
  stage_features(sX, S);
  MlpTile T;
  mlp_forward<true>(sX, W, T);
  // output error of rows g and g+8
  float dy[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float d = 0.0f;
    if (r0 + g + 8 * h < end) {
      const float e = T.y[h] - S.tg[h];
      if (t == 0) lsum += e * e;
      d = 2.0f * e * inv_n;
    }
    dy[h] = d;
  }
  // layer 3: dW3 = sum dy h2, db3 = sum dy; layer-2 pre-activation gradient dZ2
  float dz2[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    add_cols<FIRST>(sG, kOffW3, j, dy[0] * T.h2[j][0] + dy[1] * T.h2[j][2], dy[0] * T.h2[j][1] + dy[1] * T.h2[j][3]);
    const float wl = W.w3[8 * j + 2 * t], wh = W.w3[8 * j + 2 * t + 1];
    dz2[j][0] = dy[0] * wl * T.g2[j][0];
    dz2[j][1] = dy[0] * wh * T.g2[j][1];
    dz2[j][2] = dy[1] * wl * T.g2[j][2];
    dz2[j][3] = dy[1] * wh * T.g2[j][3];
    add_cols<FIRST>(sG, kOffB2, j, dz2[j][0] + dz2[j][2], dz2[j][1] + dz2[j][3]);
  }
  {
    float s = (t == 0) ? dy[0] + dy[1] : 0.0f;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) acc_to<FIRST>(sG, kOffB3, s);
  }
  // stage dZ2 and H1 (BF16, row-major [16][64]) for the weight gradient of layer 2
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 8 * j + 2 * t;
    *reinterpret_cast<uint32_t*>(sD + g * kStageLd + c) = pack_bf16(dz2[j][0], dz2[j][1]);
    *reinterpret_cast<uint32_t*>(sD + (g + 8) * kStageLd + c) = pack_bf16(dz2[j][2], dz2[j][3]);
    *reinterpret_cast<uint32_t*>(sH + g * kStageLd + c) = T.h1[j / 2][2 * (j % 2)];
    *reinterpret_cast<uint32_t*>(sH + (g + 8) * kStageLd + c) = T.h1[j / 2][2 * (j % 2) + 1];
  }
  __syncwarp();
  // rows of the 8 x 8 blocks that this lane addresses: A blocks (k half, column half) in the order
  // (0,0) (0,1) (1,0) (1,1); B blocks (k half, n-tile) in the order (0,0) (1,0) (0,1) (1,1)
  const int lr = lane & 7, lb = lane >> 3;
  const __nv_bfloat16* aD = sD + (lr + 8 * (lb >> 1)) * kStageLd + 8 * (lb & 1);
  const __nv_bfloat16* bH = sH + (lr + 8 * (lb & 1)) * kStageLd + 8 * (lb >> 1);
  // dW2[n][k] += sum_r dZ2[r][n] H1[r][k]: A = dZ2^T (64 x 16), B = H1 (16 x 64)
#pragma unroll
  for (int jj = 0; jj < 4; ++jj) {
    uint32_t b[4];
    ldmatrix4_t(b, bH + 16 * jj);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      uint32_t a[4];
      ldmatrix4_t(a, aD + 16 * mt);
      const int n0 = 16 * mt + g;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(acc, a, b[2 * e], b[2 * e + 1]);
        const int col = 16 * jj + 8 * e + 2 * t;
        acc_to2<FIRST>(sG, kOffW2 + n0 * kMlpH + col, acc[0], acc[1]);
        acc_to2<FIRST>(sG, kOffW2 + (n0 + 8) * kMlpH + col, acc[2], acc[3]);
      }
    }
  }
  // dH1 = dZ2 W2 (A from the dZ2 fragments, B = W2T), dZ1 = dH1 * gelu'(Z1)
  float dz1[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) dz1[j][e] = 0.0f;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    uint32_t a[4];
    a[0] = pack_bf16(dz2[2 * kk][0], dz2[2 * kk][1]);
    a[1] = pack_bf16(dz2[2 * kk][2], dz2[2 * kk][3]);
    a[2] = pack_bf16(dz2[2 * kk + 1][0], dz2[2 * kk + 1][1]);
    a[3] = pack_bf16(dz2[2 * kk + 1][2], dz2[2 * kk + 1][3]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat16* wr = W.w2t + (8 * j + g) * kLdW2 + 16 * kk;
      mma_bf16(dz1[j], a, *reinterpret_cast<const uint32_t*>(wr + 2 * t),
               *reinterpret_cast<const uint32_t*>(wr + 2 * t + 8));
    }
  }
  __syncwarp();  // every lane has read sD before it is overwritten with dZ1
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e) dz1[j][e] *= T.g1[j][e];
    add_cols<FIRST>(sG, kOffB1, j, dz1[j][0] + dz1[j][2], dz1[j][1] + dz1[j][3]);
    const int c = 8 * j + 2 * t;
    *reinterpret_cast<uint32_t*>(sD + g * kStageLd + c) = pack_bf16(dz1[j][0], dz1[j][1]);
    *reinterpret_cast<uint32_t*>(sD + (g + 8) * kStageLd + c) = pack_bf16(dz1[j][2], dz1[j][3]);
  }
  __syncwarp();
  // dW1[n][k] += sum_r dZ1[r][n] X[r][k]: A = dZ1^T (64 x 16), B = X (16 x 8 real columns)
  uint32_t bx[4];
  ldmatrix4_t(bx, sX + (lr + 8 * (lb & 1)) * kMlpK1 + 8 * (lb >> 1));  // blocks 2 and 3: the zero columns
#pragma unroll
  for (int mt = 0; mt < 4; ++mt) {
    uint32_t a[4];
    ldmatrix4_t(a, aD + 16 * mt);
    const int n0 = 16 * mt + g;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16(acc, a, bx[0], bx[1]);
    acc_to2<FIRST>(sG, kOffW1 + n0 * kMlpIn + 2 * t, acc[0], acc[1]);
    acc_to2<FIRST>(sG, kOffW1 + (n0 + 8) * kMlpIn + 2 * t, acc[2], acc[3]);
  }
  __syncwarp();  // sX, sD and sH are rewritten by the next tile
}

// One virtual block (kTrainWarps warps) of a minibatch of `count` samples spread over `blocks` of
// them: block `block`'s warps take tiles block * kTrainWarps + warp, then every
// blocks * kTrainWarps-th.  Deterministic: every warp accumulates into its own gradient copy
// (each entry always updated by the same lane), block_slab sums the copies in a fixed order
// into the block's slab (gradients, then the loss), and the consumer sums the slabs in block
// order.  `first` holds the samples of the warp's first tile.  Called by warps 0 .. kTrainWarps - 1.
__device__ __forceinline__ void train_tiles(const MlpWeights& W, const float* feats, const float* targets,
                                            const uint32_t* order, unsigned long long start, unsigned long long count,
                                            float inv_n, unsigned block, unsigned blocks, const SampleTile& first,
                                            __nv_bfloat16* sX, float* sG, float* s_loss) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float lsum = 0.0f;
  const unsigned long long end = start + count, ntiles = (count + 15) / 16;
  unsigned long long tile = (unsigned long long)block * kTrainWarps + warp;
  if (tile < ntiles) {
    train_tile<true>(W, first, start + tile * 16, end, inv_n, sX, sG, lsum);
  } else {
    for (int i = lane; i < kMlpParams; i += 32) sG[i] = 0.0f;
  }
  for (tile += (unsigned long long)blocks * kTrainWarps; tile < ntiles; tile += (unsigned long long)blocks * kTrainWarps) {
    SampleTile S;
    load_samples(S, feats, targets, order, start + tile * 16, end);
    train_tile<false>(W, S, start + tile * 16, end, inv_n, sX, sG, lsum);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if (lane == 0) s_loss[warp] = lsum;
}

// The warps' gradient copies and losses summed in warp order into the block's slab (all threads,
// after a block barrier).
__device__ __forceinline__ void block_slab(const float* sG0, const float* s_loss, float* slab) {
  for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) {
    float v = sG0[i];
#pragma unroll
    for (int w = 1; w < kTrainWarps; ++w) v += sG0[w * kSlab + i];
    slab[i] = v;
  }
  if (threadIdx.x == 0) {
    float l = s_loss[0];
    for (int w = 1; w < kTrainWarps; ++w) l += s_loss[w];
    slab[kMlpParams] = l;
  }
}

// Forward + backward over samples order[start .. start+count) of (feats, targets), one minibatch.
__global__ void __launch_bounds__(kTrainWarps * 32)
k_mlp_train(const MlpWeights* Wg, const float* feats, const float* targets, const uint32_t* order,
            unsigned long long start, unsigned long long count, float inv_n, float* slabs) {
  extern __shared__ __align__(16) unsigned char smem[];
  MlpWeights& W = *reinterpret_cast<MlpWeights*>(smem);
  float* sG0 = reinterpret_cast<float*>(smem + sizeof(MlpWeights));  // kTrainWarps copies of kSlab
  __nv_bfloat16* sX0 = reinterpret_cast<__nv_bfloat16*>(sG0 + kTrainWarps * kSlab);
  __shared__ float s_loss[kTrainWarps];
  const int warp = threadIdx.x >> 5;
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(Wg);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&W);
    for (int i = threadIdx.x; i < (int)(sizeof(MlpWeights) / 4); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  SampleTile S;
  load_samples(S, feats, targets, order, start + ((unsigned long long)blockIdx.x * kTrainWarps + warp) * 16,
               start + count);
  train_tiles(W, feats, targets, order, start, count, inv_n, blockIdx.x, gridDim.x, S, sX0 + warp * kTileHalves,
              sG0 + warp * kSlab, s_loss);
  __syncthreads();
  block_slab(sG0, s_loss, slabs + (size_t)blockIdx.x * kSlab);
}

// A whole epoch of minibatch steps in one launch: one cluster of at most kMaxCluster CTAs, CTA b
// standing for block b of each step's k_mlp_train launch.  Every CTA keeps the parameters,
// the Adam moments and the packed weights in its shared memory and applies the same update to all
// of them from all slabs (summed in block order), so a step needs one cluster barrier and no
// weight ever crosses the CTAs.  The slabs alternate between two buffers: a CTA writes a
// buffer again only after a barrier that every reader of its last contents has reached.  The
// results are those of the launches, bit for bit.  Warps kTrainWarps and up only help to sum
// and update.  A step was two dependent launches (29 us at 512 samples); what bounds it now is
// the chain of one tile's products and the cluster's reads of the slabs (L2).
constexpr int kMaxCluster = 16;
constexpr int kEpochThreads = 256;

__global__ void __launch_bounds__(kEpochThreads)
k_mlp_epoch(float* p_g, float* m_g, float* v_g, MlpWeights* Wg, const float* feats, const float* targets,
            const uint32_t* order, unsigned long long n, unsigned long long batch, const float* lr_t, float b1,
            float b2, float eps, float* slabs, float* loss) {
  extern __shared__ __align__(16) unsigned char smem[];
  MlpWeights& W = *reinterpret_cast<MlpWeights*>(smem);
  float* sG0 = reinterpret_cast<float*>(smem + sizeof(MlpWeights));
  __nv_bfloat16* sX0 = reinterpret_cast<__nv_bfloat16*>(sG0 + kTrainWarps * kSlab);
  float* sp = reinterpret_cast<float*>(sX0 + kTrainWarps * kTileHalves);  // parameters, moments
  float* sm = sp + kSlab;
  float* sv = sm + kSlab;
  __shared__ float s_loss[kTrainWarps];
  const int warp = threadIdx.x >> 5;
  const unsigned cta = blockIdx.x;  // one cluster: the rank in it
  for (int i = threadIdx.x; i < (int)(sizeof(MlpWeights) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t*>(&W)[i] = reinterpret_cast<const uint32_t*>(Wg)[i];
  for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) {
    sp[i] = p_g[i];
    sm[i] = m_g[i];
    sv[i] = v_g[i];
  }
  float lsum = threadIdx.x == 0 ? *loss : 0.0f;
  SampleTile S;  // the warp's first tile of the coming step
  const unsigned long long mine = ((unsigned long long)cta * kTrainWarps + warp) * 16;
  if (warp < kTrainWarps) load_samples(S, feats, targets, order, mine, n < batch ? n : batch);
  __syncthreads();
  unsigned step = 0;
  for (unsigned long long st = 0; st < n; st += batch, ++step) {
    const unsigned long long cnt = n - st < batch ? n - st : batch;
    const unsigned tiles = (unsigned)((cnt + 15) / 16);
    const unsigned blocks = (tiles + kTrainWarps - 1) / kTrainWarps;  // as launch_train: at most the cluster
    float* buf = slabs + (size_t)(step & 1) * kMaxCluster * kSlab;
    if (cta < blocks) {
      if (warp < kTrainWarps)
        train_tiles(W, feats, targets, order, st, cnt, 1.0f / (float)cnt, cta, blocks, S, sX0 + warp * kTileHalves,
                    sG0 + warp * kSlab, s_loss);
      __syncthreads();
      block_slab(sG0, s_loss, buf + (size_t)cta * kSlab);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (warp < kTrainWarps && st + batch < n)
      load_samples(S, feats, targets, order, st + batch + mine, n - st - batch < batch ? n : st + 2 * batch);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const float lr = lr_t[step];
    // four parameters at a time, four slabs' loads in flight; each parameter's slabs still added in
    // block order (entries past kMlpParams, the loss's and the padding's, are updated by nobody)
    for (int q = threadIdx.x; q < kSlab / 4; q += blockDim.x) {
      float gq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      const float4* src = reinterpret_cast<const float4*>(buf) + q;
      for (unsigned b = 0; b < blocks; b += 4) {
        float4 v[4];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
          if (b + u < blocks) v[u] = __ldcg(src + (size_t)(b + u) * (kSlab / 4));
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
          if (b + u < blocks) {
            gq[0] += v[u].x;
            gq[1] += v[u].y;
            gq[2] += v[u].z;
            gq[3] += v[u].w;
          }
      }
      float4 p4 = reinterpret_cast<float4*>(sp)[q], m4 = reinterpret_cast<float4*>(sm)[q],
             v4 = reinterpret_cast<float4*>(sv)[q];
      float pe[4] = {p4.x, p4.y, p4.z, p4.w}, me[4] = {m4.x, m4.y, m4.z, m4.w}, ve[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * q + e;
        if (i == kMlpParams) s_loss[0] = gq[e];
        if (i >= kMlpParams) continue;
        pe[e] = adam_step(pe[e], me[e], ve[e], gq[e], lr, b1, b2, eps);
        pack_param(&W, i, pe[e]);
      }
      reinterpret_cast<float4*>(sp)[q] = make_float4(pe[0], pe[1], pe[2], pe[3]);
      reinterpret_cast<float4*>(sm)[q] = make_float4(me[0], me[1], me[2], me[3]);
      reinterpret_cast<float4*>(sv)[q] = make_float4(ve[0], ve[1], ve[2], ve[3]);
    }
    __syncthreads();
    if (threadIdx.x == 0) lsum += s_loss[0];
    __syncthreads();  // before the next step's losses
  }
  if (cta == 0) {
    for (int i = threadIdx.x; i < (int)(sizeof(MlpWeights) / 4); i += blockDim.x)
      reinterpret_cast<uint32_t*>(Wg)[i] = reinterpret_cast<const uint32_t*>(&W)[i];
    for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) {
      p_g[i] = sp[i];
      m_g[i] = sm[i];
      v_g[i] = sv[i];
    }
    if (threadIdx.x == 0) *loss = lsum;
  }
}

// Sums the slabs of k_mlp_train's blocks in block order: the gradient (one thread per
// parameter), and the loss into *loss (thread kMlpParams).
__global__ void __launch_bounds__(256) k_mlp_reduce(const float* slabs, int nslabs, float* grads, float* loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kMlpParams) return;
  float v = 0.0f;
  for (int b = 0; b < nslabs; ++b) v += slabs[(size_t)b * kSlab + i];
  if (i < kMlpParams) grads[i] = v;
  else *loss += v;
}

// Scores of n feature rows (one warp per 16 rows).
__global__ void __launch_bounds__(128) k_mlp_predict(const MlpWeights* Wg, const float* feats, unsigned long long n,
                                                     float* out) {
  __shared__ MlpWeights W;
  __shared__ __align__(16) __nv_bfloat16 sX[4][16 * kMlpK1];
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(Wg);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&W);
    for (int i = threadIdx.x; i < (int)(sizeof(MlpWeights) / 4); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const unsigned long long ntiles = (n + 15) / 16;
  for (unsigned long long tile = (unsigned long long)blockIdx.x * 4 + warp; tile < ntiles;
       tile += (unsigned long long)gridDim.x * 4) {
    SampleTile S;
    load_samples(S, feats, nullptr, nullptr, tile * 16, n);
    stage_features(sX[warp], S);
    MlpTile T;
    mlp_forward<false>(sX[warp], W, T);
    if (t == 0) {
      if (tile * 16 + g < n) out[tile * 16 + g] = T.y[0];
      if (tile * 16 + g + 8 < n) out[tile * 16 + g + 8] = T.y[1];
    }
    __syncwarp();
  }
}

size_t train_smem() {
  return sizeof(MlpWeights) + sizeof(float) * kTrainWarps * kSlab + sizeof(__nv_bfloat16) * kTrainWarps * kTileHalves;
}
size_t epoch_smem() { return train_smem() + sizeof(float) * 3 * kSlab; }

// One epoch of minibatches of at most kMaxCluster blocks as a single cluster; *done says whether it
// was launched (false: the device cannot place such a cluster).
ppvm_status launch_epoch(ppvm_mlp* m, unsigned blocks, unsigned long long n, unsigned long long batch,
                         const uint32_t* d_order, const float* d_lr, float b1, float b2, float eps, bool* done) {
  *done = false;
  static const bool never = [] {  // PPVM_MLP_EPOCH=never: two launches per step (for the tests)
    const char* e = std::getenv("PPVM_MLP_EPOCH");
    return e && std::strcmp(e, "never") == 0;
  }();
  if (never) return PPVM_OK;
  MCUDA(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)epoch_smem()));
  MCUDA(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kEpochThreads);
  cfg.dynamicSmemBytes = epoch_smem();
  cfg.stream = m->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = blocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, k_mlp_epoch, &cfg) != cudaSuccess || fit < 1) {
    cudaGetLastError();
    return PPVM_OK;
  }
  MCUDA(cudaLaunchKernelEx(&cfg, k_mlp_epoch, m->params, m->m, m->v, m->w, (const float*)m->d_feats,
                           (const float*)m->d_tgt, d_order, n, batch, d_lr, b1, b2, eps, m->slabs, m->loss));
  *done = true;
  return PPVM_OK;
}

ppvm_status ensure_data(ppvm_mlp* m, size_t n) {
  if (n <= m->data_cap) return PPVM_OK;
  cudaFree(m->d_feats);
  cudaFree(m->d_tgt);
  cudaFree(m->d_out);
  m->d_feats = nullptr;
  m->d_tgt = nullptr;
  m->d_out = nullptr;
  m->data_cap = 0;
  MCUDA(cudaMalloc(&m->d_feats, sizeof(float) * kMlpIn * n));
  MCUDA(cudaMalloc(&m->d_tgt, sizeof(float) * n));
  MCUDA(cudaMalloc(&m->d_out, sizeof(float) * n));
  m->data_cap = n;
  return PPVM_OK;
}

// One pinned buffer of a destroyed network is kept for the next one (page-locking and unlocking take
// milliseconds); ppvm_release_cached_memory gives it back.
constexpr size_t kKeepPinnedWords = (size_t)4 << 20;
std::mutex g_pinned_mu;
uint32_t* g_pinned = nullptr;
size_t g_pinned_words = 0;

uint32_t* take_pinned(size_t words, size_t* got) {
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  if (!g_pinned || g_pinned_words < words) return nullptr;
  uint32_t* p = g_pinned;
  *got = g_pinned_words;
  g_pinned = nullptr;
  return p;
}

void give_pinned(uint32_t* p, size_t words) {  // no copy from it is in flight
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  if (!g_pinned && words <= kKeepPinnedWords) {
    g_pinned = p;
    g_pinned_words = words;
  } else {
    cudaFreeHost(p);
  }
}

// Room for `words` 4-byte words of orders and learning rates (the stream is idle).
ppvm_status ensure_order(ppvm_mlp* m, size_t words) {
  for (cudaEvent_t& e : m->half_free)
    if (!e) MCUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  if (words <= m->order_cap) return PPVM_OK;
  cudaFree(m->d_order);
  give_pinned(m->h_order, m->pinned_words);
  m->d_order = nullptr;
  m->h_order = nullptr;
  m->order_cap = 0;
  MCUDA(cudaMalloc(&m->d_order, sizeof(uint32_t) * words));
  m->h_order = take_pinned(words, &m->pinned_words);
  if (!m->h_order) {
    MCUDA(cudaMallocHost(&m->h_order, sizeof(uint32_t) * words));
    m->pinned_words = words;
  }
  m->order_cap = words;
  return PPVM_OK;
}

// Forward + backward of one minibatch into the slabs; *nslabs = the number of slabs written.
ppvm_status launch_train(ppvm_mlp* m, const uint32_t* d_order, unsigned long long start, unsigned long long count, float inv_n,
                         int* nslabs) {
  static std::atomic<unsigned long long> attr{0};  // one bit per device
  const unsigned long long bit = 1ull << (m->device & 63);
  if (!(attr.load(std::memory_order_acquire) & bit)) {
    MCUDA(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem()));
    attr.fetch_or(bit, std::memory_order_release);
  }
  const unsigned long long tiles = (count + 15) / 16;
  const unsigned grid = (unsigned)std::max<unsigned long long>(
      1, std::min<unsigned long long>((tiles + kTrainWarps - 1) / kTrainWarps, kMaxTrainBlocks));
  k_mlp_train<<<grid, kTrainWarps * 32, train_smem(), m->stream>>>(m->w, m->d_feats, m->d_tgt,
                                                                   d_order, start, count, inv_n, m->slabs);
  MCUDA(cudaGetLastError());
  *nslabs = (int)grid;
  return PPVM_OK;
}

uint64_t splitmix(uint64_t& s) {
  s += 0x9E3779B97F4A7C15ull;
  uint64_t z = s;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

namespace ppvm {
void release_mlp_staging() {
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  if (g_pinned) cudaFreeHost(g_pinned);
  g_pinned = nullptr;
}
}  // namespace ppvm

extern "C" {

ppvm_status ppvm_mlp_destroy(ppvm_mlp* m) {
  if (!m) return PPVM_OK;
  cudaSetDevice(m->device);
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaFree(m->params);
  cudaFree(m->m);
  cudaFree(m->v);
  cudaFree(m->grads);
  cudaFree(m->loss);
  cudaFree(m->slabs);
  cudaFree(m->w);
  cudaFree(m->d_feats);
  cudaFree(m->d_tgt);
  cudaFree(m->d_order);
  give_pinned(m->h_order, m->pinned_words);
  for (cudaEvent_t e : m->half_free)
    if (e) cudaEventDestroy(e);
  cudaFree(m->d_out);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
  return PPVM_OK;
}

ppvm_status ppvm_mlp_set_params(ppvm_mlp* m, const float* params, size_t n) {
  if (!m || !params || n != (size_t)kMlpParams) return mfail(PPVM_EINVAL, "need the 4801 network parameters");
  MCUDA(cudaSetDevice(m->device));
  MCUDA(cudaMemcpyAsync(m->params, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, m->stream));
  MCUDA(cudaMemsetAsync(m->m, 0, sizeof(float) * kMlpParams, m->stream));
  MCUDA(cudaMemsetAsync(m->v, 0, sizeof(float) * kMlpParams, m->stream));
  k_mlp_pack<<<1, 256, 0, m->stream>>>(m->params, m->w);
  MCUDA(cudaGetLastError());
  MCUDA(cudaStreamSynchronize(m->stream));
  m->step = 0;
  return PPVM_OK;
}

ppvm_status ppvm_mlp_get_params(const ppvm_mlp* m, float* params, size_t n) {
  if (!m || !params || n != (size_t)kMlpParams) return mfail(PPVM_EINVAL, "need room for 4801 parameters");
  MCUDA(cudaSetDevice(m->device));
  MCUDA(cudaMemcpyAsync(params, m->params, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, m->stream));
  MCUDA(cudaStreamSynchronize(m->stream));
  return PPVM_OK;
}

ppvm_status ppvm_mlp_create(ppvm_mlp** out, uint64_t seed, int device) {
  if (!out) return mfail(PPVM_EINVAL, "null out pointer");
  *out = nullptr;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) return mfail(PPVM_ENODEV, std::string("no CUDA device: ") + cudaGetErrorString(e));
  if (device < 0 || device >= count) return mfail(PPVM_EINVAL, "device ordinal out of range");
  MCUDA(cudaSetDevice(device));
  ppvm_mlp* m = new ppvm_mlp();
  m->device = device;
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&m->params, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->m, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->v, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->grads, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->loss, sizeof(float)) != cudaSuccess || cudaMalloc(&m->w, sizeof(MlpWeights)) != cudaSuccess ||
      cudaMalloc(&m->slabs, sizeof(float) * kSlab * kMaxTrainBlocks) != cudaSuccess) {
    ppvm_mlp_destroy(m);
    return mfail(PPVM_ECAPACITY, "device allocation failed");
  }
  // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases (seeded splitmix64)
  std::vector<float> p(kMlpParams, 0.0f);
  uint64_t s = seed;
  auto u = [&](float a) { return (float)(((splitmix(s) >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0) * a; };
  for (int i = 0; i < kMlpH * kMlpIn; ++i) p[kOffW1 + i] = u(1.0f / std::sqrt((float)kMlpIn));
  for (int i = 0; i < kMlpH * kMlpH; ++i) p[kOffW2 + i] = u(1.0f / std::sqrt((float)kMlpH));
  for (int i = 0; i < kMlpH; ++i) p[kOffW3 + i] = u(1.0f / std::sqrt((float)kMlpH));
  ppvm_status st = ppvm_mlp_set_params(m, p.data(), p.size());
  if (st != PPVM_OK) {
    ppvm_mlp_destroy(m);
    return st;
  }
  *out = m;
  return PPVM_OK;
}

ppvm_status ppvm_mlp_grad(ppvm_mlp* m, const float* feats, const float* targets, size_t n, float* grads, float* loss) {
  if (!m || !feats || !targets || !grads || n == 0) return mfail(PPVM_EINVAL, "bad argument");
  MCUDA(cudaSetDevice(m->device));
  MTRY(ensure_data(m, n));
  MCUDA(cudaMemcpyAsync(m->d_feats, feats, sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, m->stream));
  MCUDA(cudaMemcpyAsync(m->d_tgt, targets, sizeof(float) * n, cudaMemcpyHostToDevice, m->stream));
  MCUDA(cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
  int nslabs = 0;
  MTRY(launch_train(m, nullptr, 0, n, 1.0f / (float)n, &nslabs));
  k_mlp_reduce<<<(kMlpParams + 1 + 255) / 256, 256, 0, m->stream>>>(m->slabs, nslabs, m->grads, m->loss);
  MCUDA(cudaGetLastError());
  MCUDA(cudaMemcpyAsync(grads, m->grads, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, m->stream));
  float ls = 0.f;
  MCUDA(cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCUDA(cudaStreamSynchronize(m->stream));
  if (loss) *loss = ls / (float)n;
  return PPVM_OK;
}

ppvm_status ppvm_mlp_train(ppvm_mlp* m, const float* feats, const float* targets, size_t n, int epochs, int batch,
                           float lr, uint64_t seed, float* last_epoch_loss) {
  if (!m || !feats || !targets || n == 0 || epochs <= 0 || batch <= 0 || !(lr > 0.0f))
    return mfail(PPVM_EINVAL, "bad argument");
  if (n >= 0xFFFFFFFFull) return mfail(PPVM_EINVAL, "too many samples");
  MCUDA(cudaSetDevice(m->device));
  MTRY(ensure_data(m, n));
  MCUDA(cudaMemcpyAsync(m->d_feats, feats, sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, m->stream));
  MCUDA(cudaMemcpyAsync(m->d_tgt, targets, sizeof(float) * n, cudaMemcpyHostToDevice, m->stream));
  // Each epoch's sample order and learning rates are written into one half of a pinned buffer while
  // the GPU trains on the other half's.
  const size_t nsteps = (n + (size_t)batch - 1) / (size_t)batch, half = n + nsteps;  // 4-byte words
  MTRY(ensure_order(m, 2 * half));
  uint64_t s = seed;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const unsigned long long first_tiles = (std::min<size_t>((size_t)batch, n) + 15) / 16;
  const unsigned long long blocks = (first_tiles + kTrainWarps - 1) / kTrainWarps;
  float ls = 0.f;
  for (int ep = 0; ep < epochs; ++ep) {
    uint32_t* order = m->h_order + (ep & 1) * half;
    float* lr_t = reinterpret_cast<float*>(order + n);
    const uint32_t* d_order = m->d_order + (ep & 1) * half;
    const float* d_lr = reinterpret_cast<const float*>(d_order + n);
    if (ep >= 2) MCUDA(cudaEventSynchronize(m->half_free[ep & 1]));  // its copy of two epochs ago is done
    for (size_t i = 0; i < n; ++i) order[i] = (uint32_t)i;
    for (size_t i = n - 1; i > 0; --i) std::swap(order[i], order[splitmix(s) % (i + 1)]);  // Fisher-Yates
    for (size_t k = 0; k < nsteps; ++k) {
      const float step = (float)(m->step + (int)k + 1);
      lr_t[k] = lr * std::sqrt(1.0f - std::pow(b2, step)) / (1.0f - std::pow(b1, step));
    }
    MCUDA(cudaMemcpyAsync(m->d_order + (ep & 1) * half, order, sizeof(uint32_t) * half, cudaMemcpyHostToDevice,
                          m->stream));
    MCUDA(cudaEventRecord(m->half_free[ep & 1], m->stream));
    MCUDA(cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
    bool done = false;
    if (blocks <= (unsigned long long)kMaxCluster)
      MTRY(launch_epoch(m, (unsigned)blocks, n, (unsigned long long)batch, d_order, d_lr, b1, b2, eps, &done));
    for (size_t st = 0, k = 0; !done && st < n; st += (size_t)batch, ++k) {
      const size_t cnt = std::min<size_t>((size_t)batch, n - st);
      int nslabs = 0;
      MTRY(launch_train(m, d_order, st, cnt, 1.0f / (float)cnt, &nslabs));
      k_mlp_adam<<<(kMlpParams + 1 + 255) / 256, 256, 0, m->stream>>>(m->params, m->m, m->v, m->slabs, nslabs,
                                                                       m->loss, m->w, lr_t[k], b1, b2, eps);
      MCUDA(cudaGetLastError());
    }
    m->step += (int)nsteps;
  }
  MCUDA(cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCUDA(cudaStreamSynchronize(m->stream));
  if (last_epoch_loss) *last_epoch_loss = ls / (float)n;
  return PPVM_OK;
}

ppvm_status ppvm_mlp_predict(ppvm_mlp* m, const float* feats, size_t n, float* out) {
  if (!m || !feats || !out) return mfail(PPVM_EINVAL, "null argument");
  if (n == 0) return PPVM_OK;
  MCUDA(cudaSetDevice(m->device));
  MTRY(ensure_data(m, n));
  MCUDA(cudaMemcpyAsync(m->d_feats, feats, sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, m->stream));
  const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>((n + 63) / 64, 1184));
  k_mlp_predict<<<grid, 128, 0, m->stream>>>(m->w, m->d_feats, n, m->d_out);
  MCUDA(cudaGetLastError());
  MCUDA(cudaMemcpyAsync(out, m->d_out, sizeof(float) * n, cudaMemcpyDeviceToHost, m->stream));
  MCUDA(cudaStreamSynchronize(m->stream));
  return PPVM_OK;
}

}  // extern "C"
