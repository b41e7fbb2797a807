// Training of the warm-start network, one launch per step for everything but
// Adam: forward, mean-squared error, backward and weight gradients of 128 batch
// rows per CTA, on the 5th-generation tensor cores.
//
// A step of batch 8,192 is 1.7 GFLOP, a microsecond of tensor work; as eleven
// GEMM launches and five others it took 105 us, each launch waiting for the last
// and passing activations and gradients through global memory (graph replay; the
// GEMMs of gemm_tc.cu remain for other batch sizes). Here a CTA keeps its 128
// rows on chip from input to weight gradients:
//   * weights and the activations of all layers in shared memory (209 KB), each
//     once: the K-major core-matrix layout of a row-major tile is, with the two
//     strides exchanged and the MMA's transpose bit set, also the MN-major layout
//     of its transpose, so the same bytes serve the forward product, the
//     gradient of the activations and the gradient of the weights;
//   * the three layers' pre-activations in tensor memory (3 x 128 columns), which
//     the backward epilogues read for GELU'; the last 128 columns and those of
//     layers already done take the other products;
//   * eight stages of MMAs, one thread issuing, one commit and one bounded wait
//     each; 512 threads run the epilogues (thread = row, warpgroup = a quarter of
//     the columns) and sum the bias gradients while the MMAs run;
//   * the weight gradients of the 128 rows go to global memory with 16-byte
//     vector reductions.
// What bounds it is the latency of that chain: 29 us for any batch up to 19,456
// (issue 26 %, barriers a third of the stalls; two warpgroups instead of four
// 33 us). With Adam a step of 8,192 rows takes 31.3 us (105 before; 37.0 with
// ordinary launches in place of the dependent ones, see wait_for_previous).
// Roundings (bf16 activations and gradients, fp32 sums) are those of the GEMM
// path; only the order of the fp32 sums over rows differs.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "mlp_math.cuh"
#include "pcgb.h"
#include "tc_common.cuh"

namespace pcgb_mlp_train {

using pcgb_mlp::bf16;
using namespace pcgb_tc;

constexpr int NIN = 16, HID = 128, NOUT = 8;
constexpr int LDX = NIN + 8, LDH = HID + 8;
constexpr int ROWS = 128;     // batch rows of a CTA
constexpr int THREADS = 512;  // four warpgroups
constexpr int TMEM_COLS = 512;
constexpr unsigned kWaitLimit = 1u << 22;

struct __align__(1024) TrainSmem {
  bf16 w1[HID * NIN];
  bf16 w2[HID * HID];
  bf16 w3[HID * HID];
  bf16 w4[16 * HID];  // rows >= NOUT are zero
  bf16 x[ROWS * NIN];
  bf16 dy[ROWS * 16];  // columns >= NOUT are zero
  bf16 act[3][ROWS * HID];
  bf16 dz[ROWS * HID];  // one layer after the other
  float bias[3][HID];
  float bias4[NOUT];
  unsigned long long mbar;
  uint32_t tmem_base;
};

struct TrainArgs {
  const bf16* x;         // (batch, LDX) rows of this step
  const float* t;        // (batch, NOUT) targets
  const bf16* w[4];      // bf16 weights, rows x (in + 8)
  const float* mw[4];    // fp32 masters; column `in` holds the bias
  float* grad[4];        // (rows, in + 8), added to
  int nout;
  float count;           // batch * nout, what the mean runs over
  float* loss_sum;       // added to
  int* status;
  unsigned wait_limit;
  long long skip_block;  // failure-path test: this CTA never issues its first stage (-1 = none)
};

// rows x kdim bf16 (global leading dimension ldg) -> K-major core matrices, rows >= live zero
__device__ __forceinline__ void stage_rows(bf16* dst, const bf16* src, int rows, int live, int kdim, int ldg) {
  unsigned char* base = reinterpret_cast<unsigned char*>(dst);
  for (int c = threadIdx.x; c < rows * (kdim / 8); c += THREADS) {
    const int r = c / (kdim / 8), k = (c % (kdim / 8)) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < live) v = *reinterpret_cast<const uint4*>(src + (long long)r * ldg + k);
    *reinterpret_cast<uint4*>(base + core_off(r, k, kdim)) = v;
  }
}

// Descriptors of the K = 16 slice kk of a staged tile whose rows hold `kdim`
// elements: as a K-major operand (rows = M or N), and as an MN-major one (its
// rows are the MMA's K, its columns M or N).
__device__ __forceinline__ uint64_t k_major(uint32_t tile, int kdim, int kk) {
  return smem_desc(tile + uint32_t(kk) * 256u, 128u, uint32_t(kdim / 8) * 128u);
}
__device__ __forceinline__ uint64_t mn_major(uint32_t tile, int kdim, int kk) {
  const uint32_t group = uint32_t(kdim / 8) * 128u;  // next 8 rows
  return smem_desc(tile + uint32_t(2 * kk) * group, group, 128u);
}
constexpr uint32_t kTransA = 1u << 15, kTransB = 1u << 16;

// Column sums of the bf16 (ROWS x HID) tile dz into column `col` of grad: a warp
// reads whole core matrices (lane = row of 8 and pair of columns, no bank
// conflicts), eight columns each.
__device__ __forceinline__ void bias_grad(const bf16* dz, float* grad, int ld, int col) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(dz);
  static_assert(THREADS / 32 == HID / 8, "one warp per group of eight columns");
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int r = 0; r < ROWS / 8; ++r) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(
        base + r * (HID / 8) * 128 + warp * 128 + (lane >> 2) * 16 + (lane & 3) * 4));
    s0 += f.x;
    s1 += f.y;
  }
#pragma unroll
  for (int o = 16; o >= 4; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (lane < 4) {
    const int n = warp * 8 + lane * 2;
    atomicAdd(&grad[(long long)n * ld + col], s0);
    atomicAdd(&grad[(long long)(n + 1) * ld + col], s1);
  }
}

// `cols` accumulator columns of this thread's TMEM lane into row `row` of grad
__device__ __forceinline__ void add_row(uint32_t taddr, float* row, int cols) {
  for (int c = 0; c < cols; c += 16) {
    float v[16];
    tmem_ld16(taddr + uint32_t(c), v);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      atomicAdd(reinterpret_cast<float4*>(row + c + 4 * q), make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
  }
}

// 16 bf16 columns [c, c + 16) of row r of a (ROWS x HID) tile
__device__ __forceinline__ void put16(bf16* tile, int r, int c, const uint32_t (&w)[8]) {
  unsigned char* p = reinterpret_cast<unsigned char*>(tile) + core_off(r, c, HID);
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(p + 128) = make_uint4(w[4], w[5], w[6], w[7]);
}

// The launches of a run follow each other with programmatic dependent launch:
// a kernel starts while the one before it still runs, does what needs nothing of
// it, and waits here until that one has completed and its writes are visible.
// The first launch of a call is an ordinary one, so whatever ran before it
// (the batches' preparation) is complete for all of them; every kernel lets the
// next one start only after its own wait, so two launches back is complete too.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__global__ void __launch_bounds__(THREADS, 1) mlp_train_step_kernel(const TrainArgs p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp >> 2;            // columns [32 quarter, 32 quarter + 32)
  const int r = (warp & 3) * 32 + lane;     // row of the tile = TMEM lane
  const long long row0 = (long long)blockIdx.x * ROWS;

  stage_rows(S.x, p.x + row0 * LDX, ROWS, ROWS, NIN, LDX);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  wait_for_previous();
  let_next_start();
  stage_rows(S.w1, p.w[0], HID, HID, NIN, LDX);
  stage_rows(S.w2, p.w[1], HID, HID, HID, LDH);
  stage_rows(S.w3, p.w[2], HID, HID, HID, LDH);
  stage_rows(S.w4, p.w[3], 16, NOUT, HID, LDH);
  for (int c = threadIdx.x; c < 3 * HID; c += THREADS) {
    const int l = c / HID, n = c % HID;
    S.bias[l][n] = l == 0 ? p.mw[0][n * LDX + NIN] : p.mw[l][n * LDH + HID];
  }
  if (threadIdx.x < NOUT) S.bias4[threadIdx.x] = p.mw[3][threadIdx.x * LDH + HID];
  fence_async_smem();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();

  const uint32_t tb = S.tmem_base;
  const uint32_t trow = tb + (uint32_t((warp & 3) * 32) << 16);  // this warp's lanes
  const uint32_t mbar = smem_u32(&S.mbar);
  const uint32_t xs = smem_u32(S.x), w1 = smem_u32(S.w1), w2 = smem_u32(S.w2), w3 = smem_u32(S.w3),
                 w4 = smem_u32(S.w4), dy = smem_u32(S.dy), dz = smem_u32(S.dz);
  const uint32_t a1 = smem_u32(S.act[0]), a2 = smem_u32(S.act[1]), a3 = smem_u32(S.act[2]);
  constexpr uint32_t Z3 = 256, WORK = 384;  // TMEM columns: z1 0, z2 128, z3 256, work 384
  constexpr uint32_t ID = idesc_bf16(128, HID), ID16 = idesc_bf16(128, 16);
  bool lost = false, skipped = false;
  uint32_t phase = 0;

  // MMAs of a stage: what the threads wrote to shared memory before the barrier
  // is visible to them, and every earlier TMEM read is done
  for (int stage = 0; stage < 8 && !lost; ++stage) {
    if (threadIdx.x == 0) {
      fence_after_sync();
      skipped = stage == 0 && (long long)blockIdx.x == p.skip_block;
      if (!skipped) {
        switch (stage) {
          case 0: mma_bf16(tb, k_major(xs, NIN, 0), k_major(w1, NIN, 0), ID, 0u); break;
          case 1:
          case 2:
#pragma unroll
            for (int kk = 0; kk < HID / 16; ++kk)
              mma_bf16(tb + uint32_t(stage) * 128u, k_major(stage == 1 ? a1 : a2, HID, kk),
                       k_major(stage == 1 ? w2 : w3, HID, kk), ID, kk > 0);
            break;
          case 3:
#pragma unroll
            for (int kk = 0; kk < HID / 16; ++kk)
              mma_bf16(tb + WORK, k_major(a3, HID, kk), k_major(w4, HID, kk), ID16, kk > 0);
            break;
          case 4:  // dA3 = dy W4
            mma_bf16(tb + WORK, k_major(dy, 16, 0), mn_major(w4, HID, 0), ID | kTransB, 0u);
            break;
          case 5:  // dA2 = dz3 W3, dW3 = dz3^T a2
          case 6:  // dA1 = dz2 W2, dW2 = dz2^T a1, dW4^T = a3^T dy
#pragma unroll
            for (int kk = 0; kk < HID / 16; ++kk)
              mma_bf16(tb + WORK, k_major(dz, HID, kk), mn_major(stage == 5 ? w3 : w2, HID, kk), ID | kTransB, kk > 0);
#pragma unroll
            for (int kk = 0; kk < ROWS / 16; ++kk)
              mma_bf16(tb + Z3, mn_major(dz, HID, kk), mn_major(stage == 5 ? a2 : a1, HID, kk),
                       ID | kTransA | kTransB, kk > 0);
            if (stage == 6) {
#pragma unroll
              for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tb + 128u, mn_major(a3, HID, kk), mn_major(dy, 16, kk), ID16 | kTransA | kTransB, kk > 0);
            }
            break;
          default:  // dW1 = dz1^T x
#pragma unroll
            for (int kk = 0; kk < ROWS / 16; ++kk)
              mma_bf16(tb + Z3, mn_major(dz, HID, kk), mn_major(xs, NIN, kk), ID16 | kTransA | kTransB, kk > 0);
            break;
        }
        mma_commit(mbar);
      }
    }
    // bias gradients of the layer whose dz the MMAs are reading
    if (stage == 5) bias_grad(S.dz, p.grad[2], LDH, HID);
    if (stage == 6) bias_grad(S.dz, p.grad[1], LDH, HID);
    if (stage == 7) bias_grad(S.dz, p.grad[0], LDX, NIN);
    const bool ok = threadIdx.x != 0 || mbar_wait(mbar, phase, p.wait_limit);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
      lost = true;
      break;
    }
    fence_after_sync();
    if (stage < 3) {  // a = gelu(z + b)
      const uint32_t z = trow + uint32_t(stage) * 128u;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = quarter * 32 + q * 16;
        float v[16];
        tmem_ld16(z + uint32_t(c), v);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float2 g = __bfloat1622float2(pcgb_mlp::bits_bf162(
              pcgb_mlp::gelu2x_col_pack_bf16(v[i] + S.bias[stage][c + i], v[i + 1] + S.bias[stage][c + i + 1], i)));
          w[i / 2] = pcgb_mlp::pack_bf16(0.5f * g.x, 0.5f * g.y);  // exact
        }
        put16(S.act[stage], r, c, w);
      }
    } else if (stage == 3) {  // loss and its gradient
      float l = 0.f, d[NOUT];
      if (quarter == 0) {
        float y[16];
        tmem_ld16(trow + WORK, y);
#pragma unroll
        for (int k = 0; k < NOUT; ++k) {
          d[k] = 0.f;
          if (k < p.nout) {
            const float e = y[k] + S.bias4[k] - p.t[(row0 + r) * NOUT + k];
            d[k] = 2.f * e / p.count;
            l += e * e / p.count;
          }
        }
        uint4 o;
        o.x = pcgb_mlp::pack_bf16(d[0], d[1]);
        o.y = pcgb_mlp::pack_bf16(d[2], d[3]);
        o.z = pcgb_mlp::pack_bf16(d[4], d[5]);
        o.w = pcgb_mlp::pack_bf16(d[6], d[7]);
        unsigned char* q = reinterpret_cast<unsigned char*>(S.dy) + core_off(r, 0, 16);
        *reinterpret_cast<uint4*>(q) = o;
        *reinterpret_cast<uint4*>(q + 128) = make_uint4(0, 0, 0, 0);
        // bias gradient of the last layer, from the rounded values
#pragma unroll
        for (int k = 0; k < NOUT; ++k) {
          float s = __bfloat162float(__float2bfloat16_rn(d[k]));
#pragma unroll
          for (int m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
          if (lane == 0 && k < p.nout) atomicAdd(&p.grad[3][k * LDH + HID], s);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) l += __shfl_xor_sync(0xffffffffu, l, m);
        if (lane == 0 && p.loss_sum) atomicAdd(p.loss_sum, l);
      }
    } else if (stage < 7) {  // dz = dA gelu'(z + b) of layer 3, 2, 1
      const int layer = 6 - stage;
      const uint32_t z = trow + uint32_t(layer) * 128u;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = quarter * 32 + q * 16;
        float v[16], zz[16];
        tmem_ld16(trow + WORK + uint32_t(c), v);
        tmem_ld16(z + uint32_t(c), zz);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2)
          w[i / 2] = pcgb_mlp::pack_bf16(v[i] * pcgb_mlp::gelu_grad_col(zz[i] + S.bias[layer][c + i], i),
                                         v[i + 1] * pcgb_mlp::gelu_grad_col(zz[i + 1] + S.bias[layer][c + i + 1], i + 1));
        put16(S.dz, r, c, w);
      }
      // weight gradients of the layer above (thread r = output unit r)
      if (stage == 5) add_row(trow + Z3 + uint32_t(quarter * 32), p.grad[2] + (long long)r * LDH + quarter * 32, 32);
      if (stage == 6) {
        add_row(trow + Z3 + uint32_t(quarter * 32), p.grad[1] + (long long)r * LDH + quarter * 32, 32);
        if (quarter == 0) {  // dW4^T: thread r = input unit r
          float v[16];
          tmem_ld16(trow + 128u, v);
#pragma unroll
          for (int k = 0; k < NOUT; ++k)
            if (k < p.nout) atomicAdd(&p.grad[3][k * LDH + r], v[k]);
        }
      }
    } else if (quarter == 0) {
      add_row(trow + Z3, p.grad[0] + (long long)r * LDX, NIN);
    }
    fence_async_smem();   // shared-memory writes -> visible to the tensor cores
    fence_before_sync();  // this thread's TMEM reads are done
    __syncthreads();
  }
  if (lost && threadIdx.x == 0) {
    // the lost stage may still complete: one more bounded wait before its TMEM goes back
    if (!skipped) (void)mbar_wait(mbar, phase ^ 1u, p.wait_limit);
    if (p.status) atomicExch(p.status, 1);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(TMEM_COLS) : "memory");
  }
}

// Adam on all four layers in one launch (arithmetic of adam_kernel in mlp.cu).
struct AdamArgs {
  float *master[4], *m[4], *v[4], *grad[4];
  bf16* wbf[4];
  int size[4], live[4];  // elements, and how many of them belong to live rows
  float lr, b1, b2, eps;
  const float* corr;     // bias corrections and learning-rate scale of this step
  const int* status;     // set once a step's gradients are incomplete (see mlp_train_step_kernel), or null
};
__global__ void __launch_bounds__(256) adam_all_kernel(const AdamArgs a) {
  wait_for_previous();
  let_next_start();
  int i = int(blockIdx.x) * 256 + int(threadIdx.x), l = 0;
  while (l < 4 && i >= a.size[l]) i -= a.size[l++];
  if (l == 4) return;
  const float c1 = a.corr[0], c2 = a.corr[1];
  const float lr = a.lr * a.corr[2];
  const float gi = a.grad[l][i];
  a.grad[l][i] = 0.f;
  if (i >= a.live[l] || (a.status && *a.status)) return;  // nothing is learned from an incomplete gradient
  const float mi = a.b1 * a.m[l][i] + (1.f - a.b1) * gi;
  const float vi = a.b2 * a.v[l][i] + (1.f - a.b2) * gi * gi;
  a.m[l][i] = mi;
  a.v[l][i] = vi;
  const float w = a.master[l][i] - lr * (mi / c1) / (sqrtf(vi / c2) + a.eps);
  a.master[l][i] = w;
  a.wbf[l][i] = __float2bfloat16_rn(w);
}

// Sums and sums of squares of the transformed targets about their value at voxel
// 0, in double, per block: partial[(block * nout + k) * 2], and that value in
// origin[k]. Kinds as prepare_targets_kernel: p / max signal, p, log p.
__device__ __forceinline__ double target_of(const float* params, double smax, long long n, long long v, int k, int kind) {
  const double p = double(params[(long long)k * n + v]);
  return kind == 0 ? p / smax : (kind == 2 ? log(p < 1e-30 ? 1e-30 : p) : p);
}
__global__ void __launch_bounds__(256) target_stats_kernel(const float* signals, int nin, const float* params, int nout,
                                                           int4 kinds_lo, int4 kinds_hi, long long n, double* partial,
                                                           double* origin) {
  const int kinds[8] = {kinds_lo.x, kinds_lo.y, kinds_lo.z, kinds_lo.w, kinds_hi.x, kinds_hi.y, kinds_hi.z, kinds_hi.w};
  __shared__ double base[NOUT], part[8][NOUT][2];
  const auto signal_max = [&](long long v) {
    float m = signals[v];
    for (int i = 1; i < nin && !isnan(m); ++i) {  // a NaN stays, as in torch.max
      const float x = signals[(long long)i * n + v];
      if (!(x <= m)) m = x;
    }
    return double(m < 1e-20f ? 1e-20f : m);
  };
  if (int(threadIdx.x) < nout) {
    base[threadIdx.x] = target_of(params, signal_max(0), n, 0, threadIdx.x, kinds[threadIdx.x]);
    if (blockIdx.x == 0) origin[threadIdx.x] = base[threadIdx.x];
  }
  __syncthreads();
  double s[NOUT] = {}, q[NOUT] = {};
  for (long long v = (long long)blockIdx.x * 256 + threadIdx.x; v < n; v += (long long)gridDim.x * 256) {
    const double smax = signal_max(v);
#pragma unroll
    for (int k = 0; k < NOUT; ++k) {
      if (k >= nout) break;
      const double d = target_of(params, smax, n, v, k, kinds[k]) - base[k];
      s[k] += d;
      q[k] += d * d;
    }
  }
#pragma unroll
  for (int k = 0; k < NOUT; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      q[k] += __shfl_xor_sync(0xffffffffu, q[k], o);
    }
    if ((threadIdx.x & 31) == 0) {
      part[threadIdx.x >> 5][k][0] = s[k];
      part[threadIdx.x >> 5][k][1] = q[k];
    }
  }
  __syncthreads();
  if (int(threadIdx.x) < 2 * nout) {
    const int k = threadIdx.x >> 1, j = threadIdx.x & 1;
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += part[w][k][j];
    partial[((long long)blockIdx.x * nout + k) * 2 + j] = t;
  }
}
constexpr int kStatBlocks = 304;

thread_local std::string g_err;
int fail(int code, const char* msg) {
  g_err = msg;
  return code;
}

}  // namespace pcgb_mlp_train

using namespace pcgb_mlp_train;

extern "C" {

const char* pcgb_mlp_train_last_error(void) { return g_err.c_str(); }

int pcgb_mlp_train_target_stats(const float* signals, int nin, const float* params, int nout, const int* kinds,
                                int64_t n, double* scratch, double* mean, double* stdv, void* stream) {
  g_err.clear();
  if (n < 1 || nin < 1 || nout < 1 || nout > NOUT || !signals || !params || !kinds || !scratch || !mean || !stdv)
    return fail(PCGB_EINVAL, "bad target_stats arguments");
  static_assert(PCGB_TARGET_STATS_DOUBLES == NOUT + kStatBlocks * NOUT * 2, "scratch size");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t need = (n + 255) / 256;
  const int blocks = int(need < kStatBlocks ? need : kStatBlocks);
  int kd[8] = {};
  for (int k = 0; k < nout; ++k) kd[k] = kinds[k];
  target_stats_kernel<<<blocks, 256, 0, st>>>(signals, nin, params, nout, make_int4(kd[0], kd[1], kd[2], kd[3]),
                                              make_int4(kd[4], kd[5], kd[6], kd[7]), n, scratch + NOUT, scratch);
  cudaError_t e = cudaGetLastError();
  std::vector<double> host(size_t(NOUT) + size_t(blocks) * nout * 2);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(host.data(), scratch, host.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(PCGB_ECUDA, cudaGetErrorString(e));
  for (int k = 0; k < nout; ++k) {
    double s = 0.0, q = 0.0;
    for (int b = 0; b < blocks; ++b) {
      s += host[NOUT + (size_t(b) * nout + k) * 2];
      q += host[NOUT + (size_t(b) * nout + k) * 2 + 1];
    }
    mean[k] = host[k] + s / double(n);
    const double var = (q - s * s / double(n)) / double(n);
    stdv[k] = std::sqrt(var < 0.0 ? 0.0 : var);
  }
  return PCGB_OK;
}

int pcgb_mlp_train_steps(const pcgb_mlp_train_net* net, const void* x_rows, const float* targets, int64_t n_batches,
                         int64_t batch, int64_t first_step, int64_t steps, double lr, double b1, double b2, double eps,
                         const float* corr, float* loss_sum, int* status, unsigned wait_limit, int64_t skip_block,
                         int update, void* stream) {
  g_err.clear();
  if (!net || net->nout < 1 || net->nout > NOUT) return fail(PCGB_EINVAL, "nout must be 1..8");
  if (batch < ROWS || batch % ROWS || batch > (int64_t(1) << 30) || n_batches < 1 || first_step < 0 || steps < 0)
    return fail(PCGB_EINVAL, "batch must be a multiple of 128, with at least one batch");
  if (!x_rows || !targets || !corr) return fail(PCGB_EINVAL, "inputs, targets and Adam constants are required");
  // rows are read and gradients written in 16-byte pieces
  bool aligned = reinterpret_cast<uintptr_t>(x_rows) % 16 == 0;
  for (int l = 0; l < 4; ++l) {
    if (!net->w_bf16[l] || !net->master[l] || !net->m[l] || !net->v[l] || !net->grad[l])
      return fail(PCGB_EINVAL, "weights, moments and gradients are required");
    aligned = aligned && reinterpret_cast<uintptr_t>(net->w_bf16[l]) % 16 == 0 &&
              reinterpret_cast<uintptr_t>(net->grad[l]) % 16 == 0;
  }
  if (!aligned) return fail(PCGB_EINVAL, "inputs, weights and gradients must be 16-byte aligned");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int smem = int(sizeof(TrainSmem));
  cudaError_t e = cudaFuncSetAttribute(mlp_train_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return fail(PCGB_ECUDA, cudaGetErrorString(e));
  const int rows[4] = {HID, HID, HID, NOUT}, live[4] = {HID, HID, HID, net->nout}, ld[4] = {LDX, LDH, LDH, LDH};
  TrainArgs p{};
  AdamArgs a{};
  int total = 0;
  for (int l = 0; l < 4; ++l) {
    p.w[l] = static_cast<const bf16*>(net->w_bf16[l]);
    p.mw[l] = net->master[l];
    p.grad[l] = net->grad[l];
    a.master[l] = net->master[l];
    a.m[l] = net->m[l];
    a.v[l] = net->v[l];
    a.grad[l] = net->grad[l];
    a.wbf[l] = static_cast<bf16*>(net->w_bf16[l]);
    a.size[l] = rows[l] * ld[l];
    a.live[l] = live[l] * ld[l];
    total += a.size[l];
  }
  p.nout = net->nout;
  p.count = float(batch * net->nout);
  p.loss_sum = loss_sum;
  p.status = status;
  p.wait_limit = wait_limit ? wait_limit : kWaitLimit;
  p.skip_block = skip_block;
  a.lr = float(lr);
  a.b1 = float(b1);
  a.b2 = float(b2);
  a.eps = float(eps);
  a.status = status;
  cudaLaunchAttribute pdl{};
  pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.stream = st;
  cfg.attrs = &pdl;
  for (int64_t s = 0; s < steps; ++s) {
    const int64_t b = (first_step + s) % n_batches;
    p.x = static_cast<const bf16*>(x_rows) + b * batch * LDX;
    p.t = targets + b * batch * NOUT;
    cfg.gridDim = dim3(unsigned(batch / ROWS));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = size_t(smem);
    cfg.numAttrs = s > 0 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, mlp_train_step_kernel, p);
    if (e == cudaSuccess && update) {
      a.corr = corr + 3 * (first_step + s);
      cfg.gridDim = dim3(unsigned((total + 255) / 256));
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = 0;
      cfg.numAttrs = 1;
      e = cudaLaunchKernelEx(&cfg, adam_all_kernel, a);
    }
    if (e != cudaSuccess) return fail(PCGB_ECUDA, cudaGetErrorString(e));
  }
  return PCGB_OK;
}

}  // extern "C"
