// Warm-start network of the inversion: an MLP from the observed Stokes vector
// to the node values of the model, trained and run with hand-written BF16
// kernels (sm_100a): tcgen05 tensor-core GEMMs (bf16 operands, FP32
// accumulation in tensor memory) with fused bias / GELU / GELU' epilogues,
// an MSE loss kernel and Adam on FP32 master weights.  It has no counterpart in the reference,
// whose initial guess is the model in the control file (or the Stokes-moment
// assists of SET_TAU, src/invert3d.f90:492-727).
//
// Layouts: activations row-major [batch][features] in bf16; weights W[out][in]
// row-major (bf16 copy for the GEMMs, FP32 master for Adam); biases FP32.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/fz_b200.h"
#include "fz_tc.cuh"

namespace {

constexpr int MLP_MAXL = 8;

enum GemmMode { NT = 0, NN = 1, TN = 2 };
enum Epi { EPI_FWD_GELU = 0, EPI_FWD_LIN = 1, EPI_BWD_GELU = 2, EPI_F32 = 3 };

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

// C (M x N) = A B^T with the logical operands of each mode:
//   NT: A[m][k] = a[m*lda + k],  B[n][k] = b[n*ldb + k]   (Y = X W^T)
//   NN: A[m][k] = a[m*lda + k],  B[n][k] = b[k*ldb + n]   (dX = dZ W)
//   TN: A[m][k] = a[k*lda + m],  B[n][k] = b[k*ldb + n]   (dW = dZ^T X)
// and the epilogues
//   EPI_FWD_GELU: z = C + bias[n] -> zout (fp32, pre-activation), out = bf16(gelu(z))
//   EPI_FWD_LIN : z = C + bias[n] -> fout (fp32)
//   EPI_BWD_GELU: out = bf16(C * gelu'(zin[m][n]))
//   EPI_F32     : fout = C (fp32)
// on the fifth-generation tensor cores (tcgen05), fed by the tensor memory
// accelerator.  An operand is K-major (AMN / BMN false: K contiguous, the
// forward's X and W) or MN-major (true: MN contiguous, the backward's dZ^T,
// X^T and W^T), the tensor core reading either layout; what a box holds
// beyond the operand's edge the copy fills with zeros, so any M, N and K run
// here as long as the row strides are multiples of 16 bytes (the widths are
// multiples of 8; dL/dz of the last layer is kept at a padded stride).
//
// Persistent CTAs of 320 threads, two per SM, walk the 128 x BN output tiles
// (n fastest: neighbours share the rows of A in L2).  K runs in blocks of 64
// through ST shared-memory stages of one ring that goes on from tile to
// tile.  Warp 8's lane 0 issues the bulk tensor copies of a stage, 128-byte
// swizzled, and arms the stage's "full" mbarrier with their byte count; warp
// 9's lane 0 waits for it, issues the block's four tcgen05.mma into one of
// two accumulators in tensor memory and commits them to the stage's "empty"
// mbarrier, the tile's last block also to the accumulator's "tfull"; warps
// 0-7 read that accumulator back (tcgen05.ld; warp w: TMEM lanes 32 (w % 4),
// half of the columns), hand it back through "tempty" and apply the epilogue
// while the other accumulator fills.  The epilogue is what bounds the wide
// layers (erff on every output costs about as much issue time as the MMAs
// take), hence the second accumulator.  Every sum runs over K in the same order at each
// BN, so the tile width does not change a result.
// BN: 16 where N <= 16 (the output layer: an eighth of the columns of a 128
// tile would be in use), 64 where 128-wide tiles would leave CTAs of the
// chip without one (a training batch), else 128.  Against one tile per CTA with
// the epilogue after its MMAs, and threads staging the operands of the 13
// outputs (896-1024-1024-512-13): 16,384 rows forward 59 / 62 / 35 / 31 us
// per layer -> 42 / 45 / 30 / 9; of a batch of 1,024, the output layer 30 -> 8,
// its dW 102 -> 10 and dX 39 -> 8, the others 12-18 -> 9-13.  At 16,384 rows
// the tensor pipe is then busy 40 %, the issue slots 53 %: neither full, the
// rest is the L2's latency against 192 KB of tiles in flight per SM.
// Every wait is bounded (2 s): one that runs out sets the error flag and the
// CTA frees its tensor memory.
constexpr int TM_BM = 128, TM_BK = 64;
constexpr int TM_TILE_A = TM_BM * TM_BK * 2;
constexpr int TM_EPI_WARPS = 8, TM_THREADS = (TM_EPI_WARPS + 2) * 32;
constexpr unsigned long long TC_WAIT_NS = 2000000000ull;
__host__ __device__ constexpr int tm_tile_b(int bn) { return bn * TM_BK * 2; }
__host__ __device__ constexpr int tm_stages(int bn) { return bn == 128 ? 3 : bn == 64 ? 4 : 5; }
__host__ __device__ constexpr int tm_smem(int bn) {   // + the 1 KB alignment
  return tm_stages(bn) * (TM_TILE_A + tm_tile_b(bn)) + 1024;
}

// 16 columns nb.. of row m of the accumulator through the epilogue; vec: the
// row stride and the bases allow 16-byte accesses.
template <int EPI>
__device__ __forceinline__ void epi_cols(float v[16], size_t o, int nb, int N, bool vec,
                                         const float* __restrict__ bias, const float* __restrict__ zin,
                                         float* __restrict__ zout, float* __restrict__ fout,
                                         __nv_bfloat16* __restrict__ out) {
  if (vec && nb + 16 <= N) {
    if (EPI == EPI_FWD_GELU || EPI == EPI_FWD_LIN)
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(bias + nb + i));
        v[i] += b.x;
        v[i + 1] += b.y;
        v[i + 2] += b.z;
        v[i + 3] += b.w;
      }
    if (EPI == EPI_BWD_GELU || EPI == EPI_FWD_GELU) {
      if (EPI == EPI_FWD_GELU && zout)
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<float4*>(zout + o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      if (EPI == EPI_BWD_GELU)
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 z = __ldg(reinterpret_cast<const float4*>(zin + o + i));
          v[i] *= gelu_d(z.x);
          v[i + 1] *= gelu_d(z.y);
          v[i + 2] *= gelu_d(z.z);
          v[i + 3] *= gelu_d(z.w);
        }
      uint32_t h[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 t = EPI == EPI_FWD_GELU ? __floats2bfloat162_rn(gelu(v[2 * i]), gelu(v[2 * i + 1]))
                                                     : __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t*>(&t);
      }
      *reinterpret_cast<uint4*>(out + o) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(out + o + 8) = make_uint4(h[4], h[5], h[6], h[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        *reinterpret_cast<float4*>(fout + o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int n = nb + i;
    if (n >= N) continue;
    if (EPI == EPI_BWD_GELU) {
      out[o + i] = __float2bfloat16_rn(v[i] * gelu_d(zin[o + i]));
    } else if (EPI == EPI_F32) {
      fout[o + i] = v[i];
    } else {
      const float z = v[i] + bias[n];
      if (EPI == EPI_FWD_GELU) {
        if (zout) zout[o + i] = z;
        out[o + i] = __float2bfloat16_rn(gelu(z));
      } else {
        fout[o + i] = z;
      }
    }
  }
}

template <int EPI, bool AMN, bool BMN, int BN>
__global__ void __launch_bounds__(TM_THREADS, 2)
    k_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, int M, int N, int K,
           const float* __restrict__ bias, const float* __restrict__ zin, float* __restrict__ zout,
           float* __restrict__ fout, __nv_bfloat16* __restrict__ out, int ldc, int* __restrict__ err) {
  static_assert(!BMN || BN >= 64, "an MN-major box is 64 wide");
  constexpr int ST = tm_stages(BN), TILE_B = tm_tile_b(BN), STAGE = TM_TILE_A + TILE_B;
  constexpr uint32_t TCOLS = 2 * BN;   // two accumulators: 256, 128 or 32 columns
  extern __shared__ unsigned char tm_raw[];
  __shared__ __align__(8) uint64_t full[ST], empty[ST], tfull[2], tempty[2];
  __shared__ uint32_t tbase;
  __shared__ int bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the swizzled tiles start on a 1 KB boundary
  const uint32_t raw = fztc::smem_addr(tm_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* tiles = tm_raw + (base - raw);
  if (warp == 0) {
    fztc::tmem_alloc(&tbase, TCOLS);
    fztc::tmem_relinquish();
  }
  if (tid == TM_EPI_WARPS * 32) {
    fztc::tma_prefetch(&ta);
    fztc::tma_prefetch(&tb);
    for (int i = 0; i < ST; ++i) {
      fztc::mbar_init(&full[i], 1);
      fztc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      fztc::mbar_init(&tfull[i], 1);
      fztc::mbar_init(&tempty[i], TM_EPI_WARPS);
    }
    bad = 0;
    fztc::fence_mbar_init();
  }
  fztc::fence_before_sync();
  __syncthreads();
  fztc::fence_after_sync();
  const uint32_t tmem = tbase;
  const int nkb = (K + TM_BK - 1) / TM_BK;
  const int ntn = (N + BN - 1) / BN, tiles_mn = ntn * ((M + TM_BM - 1) / TM_BM);
  if (warp == TM_EPI_WARPS) {
    if (lane == 0) {
      int st = 0;
      uint32_t round = 0;   // of the ring; a stage's use of round r frees on its "empty" phase r
      bool ok = true;
      for (int t = blockIdx.x; t < tiles_mn && ok; t += gridDim.x) {
        const int m0 = (t / ntn) * TM_BM, n0 = (t % ntn) * BN;
        for (int kb = 0; kb < nkb; ++kb) {
          if (round > 0 && !fztc::mbar_wait(&empty[st], (round - 1) & 1, TC_WAIT_NS)) {
            ok = false;
            break;
          }
          unsigned char* sa = tiles + (size_t)st * STAGE;
          unsigned char* sb = sa + TM_TILE_A;
          fztc::mbar_arrive_expect_tx(&full[st], STAGE);
          // K-major: one 64 (K) x rows box; MN-major: 64 (MN) x 64 (K)
          // boxes, the next 64 MN elements 8 KB on
          if (AMN) {
            fztc::tma_load_2d(sa, &ta, m0, kb * TM_BK, &full[st]);
            fztc::tma_load_2d(sa + TM_TILE_A / 2, &ta, m0 + 64, kb * TM_BK, &full[st]);
          } else {
            fztc::tma_load_2d(sa, &ta, kb * TM_BK, m0, &full[st]);
          }
          if (BMN) {
            fztc::tma_load_2d(sb, &tb, n0, kb * TM_BK, &full[st]);
            if (BN == 128) fztc::tma_load_2d(sb + TILE_B / 2, &tb, n0 + 64, kb * TM_BK, &full[st]);
          } else {
            fztc::tma_load_2d(sb, &tb, kb * TM_BK, n0, &full[st]);
          }
          if (++st == ST) {
            st = 0;
            ++round;
          }
        }
      }
      if (!ok) {   // the copies in flight: the ST uses before this one
        atomicExch(&bad, 1);
        for (int i = 0; i < ST; ++i) fztc::mbar_wait(&full[i], (i < st ? round : round - 1) & 1, TC_WAIT_NS);
      }
    }
    __syncwarp();
  } else if (warp == TM_EPI_WARPS + 1) {
    if (lane == 0) {
      const uint32_t idesc = fztc::idesc_bf16_major(TM_BM, BN, AMN, BMN);
      int st = 0, i = 0;
      uint32_t round = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles_mn && ok; t += gridDim.x, ++i) {
        const uint32_t acc = tmem + (uint32_t)((i & 1) * BN);
        if (i >= 2) {   // the accumulator's tile i - 2 has been read
          ok = fztc::mbar_wait(&tempty[i & 1], ((i >> 1) - 1) & 1, TC_WAIT_NS);
          if (!ok) break;
          fztc::fence_after_sync();
        }
        for (int kb = 0; kb < nkb; ++kb) {
          if (!fztc::mbar_wait(&full[st], round & 1, TC_WAIT_NS)) {
            ok = false;
            break;
          }
          fztc::fence_after_sync();
          const uint32_t sa = base + (uint32_t)st * STAGE, sb = sa + TM_TILE_A;
#pragma unroll
          for (int ks = 0; ks < TM_BK / 16; ++ks) {
            const uint64_t da =
                AMN ? fztc::desc_sw128_mn(sa + 2048 * ks, TM_TILE_A / 2) : fztc::desc_sw128(sa + 32 * ks);
            const uint64_t db = BMN ? fztc::desc_sw128_mn(sb + 2048 * ks, TILE_B / 2) : fztc::desc_sw128(sb + 32 * ks);
            fztc::mma_bf16(acc, da, db, idesc, (kb > 0 || ks > 0) ? 1u : 0u);
          }
          fztc::commit(&empty[st]);
          if (++st == ST) {
            st = 0;
            ++round;
          }
        }
        if (ok) fztc::commit(&tfull[i & 1]);
      }
      if (!ok) atomicExch(&bad, 1);
    }
    __syncwarp();
  } else {
    constexpr int COLS = BN >= 32 ? BN / 2 : BN;   // per warp; at BN = 16 warps 4-7 only hand back
    const int q = warp & 3, half = warp >> 2;
    const bool mine = half * COLS < BN;
    const bool vec = (ldc & 7) == 0 && (((uintptr_t)fout | (uintptr_t)zout | (uintptr_t)out | (uintptr_t)zin) & 15) == 0;
    int i = 0;
    for (int t = blockIdx.x; t < tiles_mn; t += gridDim.x, ++i) {
      const int m = (t / ntn) * TM_BM + 32 * q + lane, n0 = (t % ntn) * BN + half * COLS;
      if (!fztc::mbar_wait(&tfull[i & 1], (i >> 1) & 1, TC_WAIT_NS)) {
        atomicExch(&bad, 1);
        break;
      }
      fztc::fence_after_sync();
      const uint32_t acc = tmem + (uint32_t)((i & 1) * BN) + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * COLS);
#pragma unroll 1
      for (int cc = 0; cc < COLS && mine; cc += 16) {
        float v[16];
        __syncwarp();
        fztc::tmem_ld16(acc + (uint32_t)cc, v);
        if (m < M && n0 + cc < N)
          epi_cols<EPI>(v, (size_t)m * ldc + n0 + cc, n0 + cc, N, vec, bias, zin, zout, fout, out);
      }
      __syncwarp();
      fztc::fence_before_sync();
      if (lane == 0) fztc::mbar_arrive(&tempty[i & 1]);
    }
  }
  fztc::fence_before_sync();
  __syncthreads();
  if (tid == 0 && *(volatile int*)&bad) atomicExch(err, 1);
  if (warp == 0) fztc::tmem_dealloc(tmem, TCOLS);
}

// Training-step state on the device, so that one captured step replays for
// every batch: the position in the epoch's batch order and the Adam step.
struct TrainState {
  int bi;
  int step;
};

// Row offset of the current batch (order: the epoch's batch permutation).
__device__ __forceinline__ size_t batch_row(const int* order, const TrainState* st, int n) {
  return order ? (size_t)order[st->bi] * n : 0;
}

// MSE loss 1/(n*nout) sum lw_j (y - t)^2 (lw: per-output weights, null =
// all 1) and dL/dy in bf16, rows at stride ldd
__global__ void k_mse(int n, int nout, const float* __restrict__ y, const float* __restrict__ t,
                      __nv_bfloat16* __restrict__ dy, int ldd, float* __restrict__ loss, const int* __restrict__ order,
                      const TrainState* __restrict__ st, const float* __restrict__ lw = nullptr) {
  __shared__ float red[8];
  t += batch_row(order, st, n) * nout;
  const size_t total = (size_t)n * nout;
  float s = 0.0f;
  const float sc = 2.0f / (float)total;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const float d = y[i] - t[i];
    const float wd = lw ? lw[i % nout] * d : d;
    s += wd * d;
    dy[i / nout * ldd + i % nout] = __float2bfloat16_rn(sc * wd);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) b += red[i];
    atomicAdd(loss, b / (float)total);
  }
}

// bias gradient: column sums of dZ (bf16, n x m at row stride ld, a multiple
// of 8), each in row order.  A block of 128 threads takes 32 columns: tiles
// of CS_ROWS rows stream into two shared-memory buffers (16-byte async
// copies) while the first warp adds the previous tile, a lane per column.
// The sum is one chain of FP32 additions (n x 4 cycles: 2.2 us at 1024
// rows), which the copies keep fed; reading the rows straight from memory
// the chain waited for every load (67 us at 1024 x 1024, now 8).  With `st` (the
// last layer's sums of a training step) it also advances the step state:
// after the loss has read the batch's position and before any Adam update.
constexpr int CS_COLS = 32, CS_ROWS = 256;
__global__ void __launch_bounds__(128) k_colsum(int n, int m, const __nv_bfloat16* __restrict__ dz, int ld,
                                                float* __restrict__ db, TrainState* __restrict__ st) {
  __shared__ __align__(16) __nv_bfloat16 buf[2][CS_ROWS][CS_COLS];
  const int tid = threadIdx.x, c0 = blockIdx.x * CS_COLS;
  if (st && blockIdx.x == 0 && tid == 0) {
    st->bi += 1;
    st->step += 1;
  }
  auto fetch = [&](int r0, int b) {
    for (int i = tid; i < CS_ROWS * (CS_COLS / 8); i += 128) {
      const int r = i / (CS_COLS / 8), c = 8 * (i % (CS_COLS / 8));
      if (r0 + r < n && c0 + c < ld)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(fztc::smem_addr(&buf[b][r][c])),
                     "l"(dz + (size_t)(r0 + r) * ld + c0 + c)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float s = 0.0f;
  fetch(0, 0);
  for (int r0 = 0, b = 0; r0 < n; r0 += CS_ROWS, b ^= 1) {
    fetch(r0 + CS_ROWS, b ^ 1);   // empty past the last row
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (tid < 32) {
      const int nr = min(CS_ROWS, n - r0);
#pragma unroll 16
      for (int r = 0; r < nr; ++r) s += __bfloat162float(buf[b][r][tid]);
    }
    __syncthreads();
  }
  if (tid < 32 && c0 + tid < m) db[c0 + tid] = s;
}

// Eight FP32 values at x (vec: 16-byte aligned) as bf16 in one 16-byte word.
__device__ __forceinline__ uint4 pack8(const float* __restrict__ x, bool vec) {
  float v[8];
  if (vec) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(x)), b = __ldg(reinterpret_cast<const float4*>(x) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = x[i];
  }
  uint32_t h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    h[i] = *reinterpret_cast<const uint32_t*>(&t);
  }
  return make_uint4(h[0], h[1], h[2], h[3]);
}

// x (n8 groups of eight FP32 values) as bf16; y is 16-byte aligned.  Bound by
// its 6 bytes per value: a thread moves 32 bytes in, 16 out (14.7 M values:
// 28 -> 14 us against one value at a time).
__global__ void k_to_bf16(size_t n8, const float* __restrict__ x, __nv_bfloat16* __restrict__ y) {
  const bool vec = ((uintptr_t)x & 15) == 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x)
    reinterpret_cast<uint4*>(y)[i] = pack8(x + 8 * i, vec);
}

// Observed Stokes rows (n x d, FP64, GAIN-normalised) standardised with the
// training set's mean and spread, (x - mu) / sd in FP32, as bf16 inputs.
__global__ void k_obs_bf16(size_t n, int d, const double* __restrict__ x, const float* __restrict__ mu,
                           const float* __restrict__ sd, __nv_bfloat16* __restrict__ y) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(i % d);
    y[i] = __float2bfloat16_rn(((float)x[i] - mu[f]) / sd[f]);
  }
}

// the current batch's rows (n x d, d a multiple of 8) of x as bf16
__global__ void k_batch_bf16(int n, int d, const float* __restrict__ x, const int* __restrict__ order,
                             const TrainState* __restrict__ st, __nv_bfloat16* __restrict__ y) {
  x += batch_row(order, st, n) * d;
  const bool vec = ((uintptr_t)x & 15) == 0;
  const size_t total = (size_t)n * d / 8;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
    reinterpret_cast<uint4*>(y)[i] = pack8(x + 8 * i, vec);
}

// Adam (Kingma & Ba 2015) of one value: FP32 master w, moments m1, m2
struct AdamK {
  float lr, b1, b2, eps;
};
__device__ __forceinline__ void adam1(const AdamK& k, float c1, float c2, float gi, float& w, float& m1, float& m2) {
  const float a = k.b1 * m1 + (1.0f - k.b1) * gi;
  const float b = k.b2 * m2 + (1.0f - k.b2) * gi * gi;
  m1 = a;
  m2 = b;
  w = w - k.lr * (a * c1) / (sqrtf(b * c2) + k.eps);
}

// Adam of one layer's weights (n4 groups of four) and biases (nb), the bf16
// copy of the weights refreshed; the bias corrections 1/(1 - b^t) of step
// t = st->step (already advanced).  Bound by its 30 bytes per weight; the
// two powers per thread are paid once for four weights and the biases need
// no launch of their own (eight launches, 49 us -> four, 26 us, for 2.5 M
// parameters).
struct AdamP {
  size_t n4;
  int nb;
  float *w, *m, *v, *b, *mb, *vb;
  const float *g, *gb;
  __nv_bfloat16* wb;
};
__global__ void __launch_bounds__(256) k_adam(AdamP p, AdamK k, const TrainState* __restrict__ st) {
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float t = (float)st->step;
  const float c1 = 1.0f / (1.0f - powf(k.b1, t)), c2 = 1.0f / (1.0f - powf(k.b2, t));
  for (size_t i = i0; i < p.n4; i += (size_t)gridDim.x * blockDim.x) {
    const float4 g = __ldg(reinterpret_cast<const float4*>(p.g) + i);
    float4 w = reinterpret_cast<float4*>(p.w)[i], m = reinterpret_cast<float4*>(p.m)[i],
           v = reinterpret_cast<float4*>(p.v)[i];
    adam1(k, c1, c2, g.x, w.x, m.x, v.x);
    adam1(k, c1, c2, g.y, w.y, m.y, v.y);
    adam1(k, c1, c2, g.z, w.z, m.z, v.z);
    adam1(k, c1, c2, g.w, w.w, m.w, v.w);
    reinterpret_cast<float4*>(p.w)[i] = w;
    reinterpret_cast<float4*>(p.m)[i] = m;
    reinterpret_cast<float4*>(p.v)[i] = v;
    const __nv_bfloat162 lo = __floats2bfloat162_rn(w.x, w.y), hi = __floats2bfloat162_rn(w.z, w.w);
    reinterpret_cast<uint2*>(p.wb)[i] =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
  for (size_t i = i0; i < (size_t)p.nb; i += (size_t)gridDim.x * blockDim.x)
    adam1(k, c1, c2, p.gb[i], p.b[i], p.mb[i], p.vb[i]);
}

// deterministic initial weights: uniform(-1,1)*sqrt(6/(fan_in+fan_out)) from a
// counter-based hash (splitmix64)
__global__ void k_init(size_t n, float* __restrict__ w, unsigned long long seed, float scale) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const float u = (float)((z >> 40) * (1.0 / 16777216.0)) * 2.0f - 1.0f;
    w[i] = u * scale;
  }
}

}  // namespace

struct fz_mlp {
  int device = 0;
  int nl = 0;                 // layers
  int dim[MLP_MAXL + 1] = {};
  // per layer: FP32 master W (out x in) and b, bf16 W, grads, Adam moments
  float *W[MLP_MAXL] = {}, *b[MLP_MAXL] = {}, *gW[MLP_MAXL] = {}, *gb[MLP_MAXL] = {};
  float *mW[MLP_MAXL] = {}, *vW[MLP_MAXL] = {}, *mb[MLP_MAXL] = {}, *vb[MLP_MAXL] = {};
  __nv_bfloat16* Wb[MLP_MAXL] = {};
  // activations for a batch capacity
  int cap = 0;
  __nv_bfloat16* act[MLP_MAXL + 1] = {};   // act[0] = input (bf16), act[l] = gelu(z_l)
  float* z[MLP_MAXL] = {};                 // pre-activations
  float* yout = nullptr;                    // last layer output (fp32), for the loss
  __nv_bfloat16* dz[MLP_MAXL] = {};        // dL/dz per layer, rows at stride ldz
  float* loss = nullptr;
  long long step = 0;
  cudaStream_t stream = nullptr;
  // the backward pass's branches: weight gradients and bias sums beside the
  // chain of dL/dz
  cudaStream_t sw = nullptr, sb = nullptr;
  cudaEvent_t ez[MLP_MAXL] = {}, eb[MLP_MAXL] = {}, ew = nullptr;
  TrainState* tstate = nullptr;   // device
  int* order = nullptr;           // device batch order of one epoch
  int order_cap = 0;
  int* d_err = nullptr;           // set by a tensor-core GEMM that gave up waiting for its MMAs
  int nsm = 148;
  float* d_lw = nullptr;          // per-output loss weights (null: all 1)
};

namespace {

int mlp_fail(cudaError_t e) {
  if (e != cudaSuccess) {
    std::fprintf(stderr, "fz_b200 mlp: CUDA error %s\n", cudaGetErrorString(e));
    return FZ_ERR_CUDA;
  }
  return 0;
}
#define MLP_CK(x)                 \
  do {                            \
    int _rc = mlp_fail(x);        \
    if (_rc) return _rc;          \
  } while (0)

// Row stride of dL/dz: 16-byte rows for the tensor maps (the hidden widths
// are multiples of 8 already).
int ldz(const fz_mlp* p, int l) { return (p->dim[l + 1] + 7) & ~7; }

int grid1(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 16); }

int mlp_reserve(fz_mlp* p, int n) {
  if (n <= p->cap) return 0;
  for (int l = 0; l <= p->nl; ++l) cudaFree(p->act[l]), p->act[l] = nullptr;
  for (int l = 0; l < p->nl; ++l) {
    cudaFree(p->z[l]), p->z[l] = nullptr;
    cudaFree(p->dz[l]), p->dz[l] = nullptr;
  }
  cudaFree(p->yout);
  p->yout = nullptr;
  p->cap = 0;
  for (int l = 0; l <= p->nl; ++l) MLP_CK(cudaMalloc(&p->act[l], (size_t)n * p->dim[l] * sizeof(__nv_bfloat16)));
  for (int l = 0; l < p->nl; ++l) {
    MLP_CK(cudaMalloc(&p->z[l], (size_t)n * p->dim[l + 1] * sizeof(float)));
    MLP_CK(cudaMalloc(&p->dz[l], (size_t)n * ldz(p, l) * sizeof(__nv_bfloat16)));
  }
  MLP_CK(cudaMalloc(&p->yout, (size_t)n * p->dim[p->nl] * sizeof(float)));
  p->cap = n;
  return 0;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// to the driver library); null when the driver does not provide it.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return EncodeTiledFn(nullptr);
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// A bf16 operand as a 2-D tensor map with 128-byte swizzling: `inner`
// contiguous elements by `outer` rows at stride ld, in boxes of 64 x box
// (a box may reach over the operand's edges: zeros).  K-contiguous operands
// are inner K, outer rows; MN-contiguous ones inner MN, outer K.
bool tmap(CUtensorMap* m, const __nv_bfloat16* p, int inner, int outer, int ld, int box) {
  const EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t boxes[2] = {64, (cuuint32_t)box};
  const cuuint32_t es[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(p), dims, strides, boxes, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE, int EPI, int BN>
int gemm_bn(const fz_mlp* p, cudaStream_t s, int M, int N, int K, const __nv_bfloat16* A, int lda,
            const __nv_bfloat16* B, int ldb, const float* bias, const float* zin, float* zout, float* fout,
            __nv_bfloat16* out, int ldc) {
  constexpr bool AMN = MODE == TN, BMN = MODE != NT;
  CUtensorMap ma, mb;
  if (!(AMN ? tmap(&ma, A, M, K, lda, TM_BK) : tmap(&ma, A, K, M, lda, TM_BM)) ||
      !(BMN ? tmap(&mb, B, N, K, ldb, TM_BK) : tmap(&mb, B, K, N, ldb, BN))) {
    std::fprintf(stderr, "fz_b200 mlp: no tensor map for a GEMM operand\n");
    return FZ_ERR_CUDA;
  }
  const long long tiles = (long long)((N + BN - 1) / BN) * ((M + TM_BM - 1) / TM_BM);
  const int grid = (int)std::min<long long>(tiles, 2 * p->nsm);
  k_gemm<EPI, AMN, BMN, BN><<<grid, TM_THREADS, tm_smem(BN), s>>>(ma, mb, M, N, K, bias, zin, zout, fout, out, ldc,
                                                                  p->d_err);
  return 0;
}

template <int MODE, int EPI>
int gemm(const fz_mlp* p, cudaStream_t s, int M, int N, int K, const __nv_bfloat16* A, int lda,
         const __nv_bfloat16* B, int ldb, const float* bias, const float* zin, float* zout, float* fout,
         __nv_bfloat16* out, int ldc) {
  if constexpr (MODE == NT) {
    if (N <= 16) return gemm_bn<MODE, EPI, 16>(p, s, M, N, K, A, lda, B, ldb, bias, zin, zout, fout, out, ldc);
  }
  const long long wide = (long long)((N + 127) / 128) * ((M + TM_BM - 1) / TM_BM);
  if (wide < 2 * p->nsm) return gemm_bn<MODE, EPI, 64>(p, s, M, N, K, A, lda, B, ldb, bias, zin, zout, fout, out, ldc);
  return gemm_bn<MODE, EPI, 128>(p, s, M, N, K, A, lda, B, ldb, bias, zin, zout, fout, out, ldc);
}

template <int EPI, bool AMN, bool BMN, int BN>
cudaError_t gemm_attr() {
  auto* k = &k_gemm<EPI, AMN, BMN, BN>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, tm_smem(BN));
  return e == cudaSuccess ? cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100) : e;
}

// The GEMMs' shared memory above the default 48 KB (set once, before any
// stream capture).
int gemm_attrs() {
  const cudaError_t es[] = {gemm_attr<EPI_FWD_GELU, false, false, 16>(), gemm_attr<EPI_FWD_GELU, false, false, 64>(),
                            gemm_attr<EPI_FWD_GELU, false, false, 128>(), gemm_attr<EPI_FWD_LIN, false, false, 16>(),
                            gemm_attr<EPI_FWD_LIN, false, false, 64>(), gemm_attr<EPI_FWD_LIN, false, false, 128>(),
                            gemm_attr<EPI_BWD_GELU, false, true, 64>(), gemm_attr<EPI_BWD_GELU, false, true, 128>(),
                            gemm_attr<EPI_F32, true, true, 64>(), gemm_attr<EPI_F32, true, true, 128>()};
  for (cudaError_t e : es)
    if (e != cudaSuccess) {
      std::fprintf(stderr, "fz_b200 mlp: CUDA error %s\n", cudaGetErrorString(e));
      return FZ_ERR_CUDA;
    }
  return 0;
}

// forward of n rows already in act[0] into y; the pre-activations are kept
// for a backward pass only when keep_z
int mlp_fwd(fz_mlp* p, int n, float* y, bool keep_z = true) {
  for (int l = 0; l < p->nl; ++l) {
    const int in = p->dim[l], out = p->dim[l + 1];
    const int rc = l + 1 < p->nl
                       ? gemm<NT, EPI_FWD_GELU>(p, p->stream, n, out, in, p->act[l], in, p->Wb[l], in, p->b[l], nullptr,
                                                keep_z ? p->z[l] : nullptr, nullptr, p->act[l + 1], out)
                       : gemm<NT, EPI_FWD_LIN>(p, p->stream, n, out, in, p->act[l], in, p->Wb[l], in, p->b[l], nullptr,
                                               nullptr, y, nullptr, out);
    if (rc) return rc;
  }
  return 0;
}

// backward from dz[nl-1]; fills gW, gb and, with `k`, updates the parameters
// (Adam).  dL/dz runs down the layers on the caller's stream; beside it, as
// soon as a layer's dL/dz is there, its weight gradient on sw and its bias
// sums on sb (a training batch fills less than the chip with any one of
// them; a step of 1,024 rows took 460 us in one chain of the former kernels, 104
// now).  A layer's update follows its gradients and the product that still
// reads its weights: on sw, the first layer's on the stream itself.
int mlp_bwd(fz_mlp* p, int n, const AdamK* k) {
  cudaStream_t s = p->stream;
  auto adam = [&](int l, cudaStream_t t) {
    const size_t n4 = (size_t)p->dim[l] * p->dim[l + 1] / 4;
    const AdamP a{n4,       p->dim[l + 1], p->W[l],  p->mW[l], p->vW[l], p->b[l],
                  p->mb[l], p->vb[l],      p->gW[l], p->gb[l], p->Wb[l]};
    k_adam<<<grid1(n4), 256, 0, t>>>(a, *k, p->tstate);
  };
  for (int l = p->nl - 1; l >= 0; --l) {
    const int in = p->dim[l], out = p->dim[l + 1], ld = ldz(p, l);
    int rc = 0;
    MLP_CK(cudaEventRecord(p->ez[l], s));   // dL/dz of layer l (and the last reader of W of layer l + 1)
    MLP_CK(cudaStreamWaitEvent(p->sw, p->ez[l], 0));
    MLP_CK(cudaStreamWaitEvent(p->sb, p->ez[l], 0));
    k_colsum<<<(out + CS_COLS - 1) / CS_COLS, 128, 0, p->sb>>>(n, out, p->dz[l], ld, p->gb[l],
                                                               k && l == p->nl - 1 ? p->tstate : nullptr);
    MLP_CK(cudaEventRecord(p->eb[l], p->sb));
    if (l > 0)   // dZ_{l-1} = (dZ_l W_l) * gelu'(z_{l-1})
      rc = gemm<NN, EPI_BWD_GELU>(p, s, n, in, out, p->dz[l], ld, p->Wb[l], in, nullptr, p->z[l - 1], nullptr, nullptr,
                                  p->dz[l - 1], in);
    // dW (out x in) = dZ^T (out x n) X (n x in)
    if (!rc)
      rc = gemm<TN, EPI_F32>(p, l > 0 ? p->sw : s, out, in, n, p->dz[l], ld, p->act[l], in, nullptr, nullptr, nullptr,
                             p->gW[l], nullptr, in);
    if (rc) return rc;
    if (k && l + 1 < p->nl) {
      MLP_CK(cudaStreamWaitEvent(p->sw, p->eb[l + 1], 0));
      adam(l + 1, p->sw);
    }
  }
  MLP_CK(cudaStreamWaitEvent(s, p->eb[0], 0));
  if (k) adam(0, s);
  MLP_CK(cudaEventRecord(p->ew, p->sw));
  MLP_CK(cudaStreamWaitEvent(s, p->ew, 0));
  return 0;
}

}  // namespace

extern "C" {

int fz_mlp_create(fz_mlp** out, int nlayers, const int* dims, unsigned long long seed, int device) {
  if (!out || nlayers < 1 || nlayers > MLP_MAXL || !dims) return FZ_ERR_ARG;
  for (int l = 0; l <= nlayers; ++l)
    if (dims[l] <= 0 || (l < nlayers && dims[l] % 8)) return FZ_ERR_ARG;   // input widths: 16-byte rows
  fz_mlp* p = new (std::nothrow) fz_mlp;
  if (!p) return FZ_ERR_NOMEM;
  p->device = device;
  p->nl = nlayers;
  for (int l = 0; l <= nlayers; ++l) p->dim[l] = dims[l];
  int rc = 0;
  auto fail = [&](int code) {
    fz_mlp_destroy(p);
    return code;
  };
  if ((rc = mlp_fail(cudaSetDevice(device)))) return fail(rc);
  if ((rc = mlp_fail(cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, device)))) return fail(rc);
  for (cudaStream_t* q : {&p->stream, &p->sw, &p->sb})
    if ((rc = mlp_fail(cudaStreamCreateWithFlags(q, cudaStreamNonBlocking)))) return fail(rc);
  if ((rc = mlp_fail(cudaEventCreateWithFlags(&p->ew, cudaEventDisableTiming)))) return fail(rc);
  for (int l = 0; l < nlayers; ++l)
    for (cudaEvent_t* q : {&p->ez[l], &p->eb[l]})
      if ((rc = mlp_fail(cudaEventCreateWithFlags(q, cudaEventDisableTiming)))) return fail(rc);
  for (int l = 0; l < nlayers; ++l) {
    const size_t nw = (size_t)dims[l] * dims[l + 1];
    float** f32[] = {&p->W[l], &p->gW[l], &p->mW[l], &p->vW[l]};
    for (float** q : f32)
      if ((rc = mlp_fail(cudaMalloc(q, nw * sizeof(float))))) return fail(rc);
    float** f32b[] = {&p->b[l], &p->gb[l], &p->mb[l], &p->vb[l]};
    for (float** q : f32b)
      if ((rc = mlp_fail(cudaMalloc(q, dims[l + 1] * sizeof(float))))) return fail(rc);
    if ((rc = mlp_fail(cudaMalloc(&p->Wb[l], nw * sizeof(__nv_bfloat16))))) return fail(rc);
    const float sc = std::sqrt(6.0f / (float)(dims[l] + dims[l + 1]));
    k_init<<<grid1(nw), 256, 0, p->stream>>>(nw, p->W[l], seed + 1000003ull * l, sc);
    k_to_bf16<<<grid1(nw / 8), 256, 0, p->stream>>>(nw / 8, p->W[l], p->Wb[l]);
    cudaMemsetAsync(p->b[l], 0, dims[l + 1] * sizeof(float), p->stream);
    cudaMemsetAsync(p->mW[l], 0, nw * sizeof(float), p->stream);
    cudaMemsetAsync(p->vW[l], 0, nw * sizeof(float), p->stream);
    cudaMemsetAsync(p->mb[l], 0, dims[l + 1] * sizeof(float), p->stream);
    cudaMemsetAsync(p->vb[l], 0, dims[l + 1] * sizeof(float), p->stream);
  }
  if ((rc = mlp_fail(cudaMalloc(&p->loss, sizeof(float))))) return fail(rc);
  if ((rc = mlp_fail(cudaMalloc(&p->d_err, sizeof(int))))) return fail(rc);
  if ((rc = mlp_fail(cudaMemsetAsync(p->d_err, 0, sizeof(int), p->stream)))) return fail(rc);
  if ((rc = gemm_attrs())) return fail(rc);
  if ((rc = mlp_fail(cudaStreamSynchronize(p->stream)))) return fail(rc);
  *out = p;
  return 0;
}

namespace {
// FZ_ERR_CUDA when a tensor-core GEMM of p gave up waiting (after the stream
// has completed); the flag is cleared.
int mlp_tc_status(fz_mlp* p) {
  int e = 0;
  if (mlp_fail(cudaMemcpy(&e, p->d_err, sizeof(int), cudaMemcpyDeviceToHost))) return FZ_ERR_CUDA;
  if (!e) return 0;
  cudaMemset(p->d_err, 0, sizeof(int));
  std::fprintf(stderr, "fz_b200 mlp: a tensor-core GEMM gave up waiting for its MMAs\n");
  return FZ_ERR_CUDA;
}
}  // namespace

int fz_mlp_destroy(fz_mlp* p) {
  if (!p) return 0;
  cudaSetDevice(p->device);
  if (p->stream) cudaStreamSynchronize(p->stream);
  for (int l = 0; l < MLP_MAXL; ++l) {
    cudaFree(p->W[l]);
    cudaFree(p->b[l]);
    cudaFree(p->gW[l]);
    cudaFree(p->gb[l]);
    cudaFree(p->mW[l]);
    cudaFree(p->vW[l]);
    cudaFree(p->mb[l]);
    cudaFree(p->vb[l]);
    cudaFree(p->Wb[l]);
    cudaFree(p->z[l]);
    cudaFree(p->dz[l]);
  }
  for (int l = 0; l <= MLP_MAXL; ++l) cudaFree(p->act[l]);
  cudaFree(p->yout);
  cudaFree(p->loss);
  cudaFree(p->d_err);
  cudaFree(p->d_lw);
  cudaFree(p->tstate);
  cudaFree(p->order);
  for (cudaStream_t q : {p->stream, p->sw, p->sb})
    if (q) cudaStreamDestroy(q);
  for (int l = 0; l < MLP_MAXL; ++l) {
    if (p->ez[l]) cudaEventDestroy(p->ez[l]);
    if (p->eb[l]) cudaEventDestroy(p->eb[l]);
  }
  if (p->ew) cudaEventDestroy(p->ew);
  delete p;
  return 0;
}

// Parameters as FP32 in layer order: W0 (out x in), b0, W1, b1, ...
long long fz_mlp_nparams(const fz_mlp* p) {
  if (!p) return FZ_ERR_ARG;
  long long n = 0;
  for (int l = 0; l < p->nl; ++l) n += (long long)p->dim[l] * p->dim[l + 1] + p->dim[l + 1];
  return n;
}

int fz_mlp_get_params(fz_mlp* p, float* host, int grads) {
  if (!p || !host) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  MLP_CK(cudaStreamSynchronize(p->stream));
  size_t o = 0;
  for (int l = 0; l < p->nl; ++l) {
    const size_t nw = (size_t)p->dim[l] * p->dim[l + 1];
    MLP_CK(cudaMemcpy(host + o, grads ? p->gW[l] : p->W[l], nw * sizeof(float), cudaMemcpyDeviceToHost));
    o += nw;
    MLP_CK(cudaMemcpy(host + o, grads ? p->gb[l] : p->b[l], p->dim[l + 1] * sizeof(float), cudaMemcpyDeviceToHost));
    o += p->dim[l + 1];
  }
  return 0;
}

int fz_mlp_set_params(fz_mlp* p, const float* host) {
  if (!p || !host) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  size_t o = 0;
  for (int l = 0; l < p->nl; ++l) {
    const size_t nw = (size_t)p->dim[l] * p->dim[l + 1];
    MLP_CK(cudaMemcpyAsync(p->W[l], host + o, nw * sizeof(float), cudaMemcpyHostToDevice, p->stream));
    o += nw;
    MLP_CK(cudaMemcpyAsync(p->b[l], host + o, p->dim[l + 1] * sizeof(float), cudaMemcpyHostToDevice, p->stream));
    o += p->dim[l + 1];
    k_to_bf16<<<grid1(nw / 8), 256, 0, p->stream>>>(nw / 8, p->W[l], p->Wb[l]);
  }
  MLP_CK(cudaGetLastError());
  MLP_CK(cudaStreamSynchronize(p->stream));
  return 0;
}

// Forward on device rows x (n x dim0, fp32) -> y (n x dimL, fp32), in chunks.
int fz_mlp_forward_device(fz_mlp* p, int n, const float* d_x, float* d_y, void* stream) {
  if (!p || n <= 0 || !d_x || !d_y) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  const int chunk = 16384;
  int rc = mlp_reserve(p, std::min(n, chunk));
  if (rc) return rc;
  cudaStream_t s = p->stream;
  cudaEvent_t ev;
  MLP_CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  if (stream) {   // order after the caller's stream
    cudaEventRecord(ev, (cudaStream_t)stream);
    cudaStreamWaitEvent(s, ev, 0);
  }
  const int d0 = p->dim[0], dl = p->dim[p->nl];
  for (int i = 0; i < n && !rc; i += chunk) {
    const int m = std::min(chunk, n - i);
    const size_t n8 = (size_t)m * d0 / 8;
    k_to_bf16<<<grid1(n8), 256, 0, s>>>(n8, d_x + (size_t)i * d0, p->act[0]);
    rc = mlp_fwd(p, m, d_y + (size_t)i * dl, false);
  }
  cudaEventRecord(ev, s);
  if (stream) cudaStreamWaitEvent((cudaStream_t)stream, ev, 0);
  int r2 = mlp_fail(cudaGetLastError());
  if (rc) r2 = rc;
  if (!stream) {
    cudaStreamSynchronize(s);
    if (!r2) r2 = mlp_tc_status(p);
  }
  cudaEventDestroy(ev);
  return r2;
}

// Forward of observed Stokes rows: d_obs (n x dim0, FP64) standardised by
// d_mu, d_sd (dim0, FP32) on the way to bf16, then the network; y (n x
// dimL, FP32).  Enqueued after the work on `stream`, which waits for it.
int fz_mlp_forward_obs_device(fz_mlp* p, int n, const double* d_obs, const float* d_mu, const float* d_sd, float* d_y,
                              void* stream) {
  if (!p || n <= 0 || !d_obs || !d_mu || !d_sd || !d_y) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  const int chunk = 16384;
  int rc = mlp_reserve(p, std::min(n, chunk));
  if (rc) return rc;
  cudaStream_t s = p->stream;
  cudaEvent_t ev;
  MLP_CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  cudaEventRecord(ev, (cudaStream_t)stream);
  cudaStreamWaitEvent(s, ev, 0);
  const int d0 = p->dim[0], dl = p->dim[p->nl];
  for (int i = 0; i < n && !rc; i += chunk) {
    const int m = std::min(chunk, n - i);
    k_obs_bf16<<<grid1((size_t)m * d0), 256, 0, s>>>((size_t)m * d0, d0, d_obs + (size_t)i * d0, d_mu, d_sd,
                                                      p->act[0]);
    rc = mlp_fwd(p, m, d_y + (size_t)i * dl, false);
  }
  cudaEventRecord(ev, s);
  cudaStreamWaitEvent((cudaStream_t)stream, ev, 0);
  const int r2 = mlp_fail(cudaGetLastError());
  cudaEventDestroy(ev);
  return rc ? rc : r2;
}

// Per-output weights of the training loss (host, nout values), or none
// (w null: every output weighs 1).
int fz_mlp_set_loss_weights(fz_mlp* p, const float* w, int n) {
  if (!p) return FZ_ERR_ARG;
  if (w && n != p->dim[p->nl]) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  if (p->stream) MLP_CK(cudaStreamSynchronize(p->stream));
  if (!w) {
    cudaFree(p->d_lw);
    p->d_lw = nullptr;
    return 0;
  }
  for (int j = 0; j < n; ++j)
    if (!(w[j] >= 0.0f) || !std::isfinite(w[j])) return FZ_ERR_ARG;
  if (!p->d_lw) MLP_CK(cudaMalloc(&p->d_lw, (size_t)n * sizeof(float)));
  MLP_CK(cudaMemcpyAsync(p->d_lw, w, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, p->stream));
  MLP_CK(cudaStreamSynchronize(p->stream));
  return 0;
}

int fz_mlp_io(const fz_mlp* p, int* nin, int* nout) {
  if (!p) return FZ_ERR_ARG;
  if (nin) *nin = p->dim[0];
  if (nout) *nout = p->dim[p->nl];
  return 0;
}

// Loss and gradients of one batch (no update); loss to *loss (host).
int fz_mlp_grad_device(fz_mlp* p, int n, const float* d_x, const float* d_t, float* loss) {
  if (!p || n <= 0 || !d_x || !d_t) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  int rc = mlp_reserve(p, n);
  if (rc) return rc;
  cudaStream_t s = p->stream;
  const int d0 = p->dim[0], dl = p->dim[p->nl];
  const size_t n8 = (size_t)n * d0 / 8;
  k_to_bf16<<<grid1(n8), 256, 0, s>>>(n8, d_x, p->act[0]);
  rc = mlp_fwd(p, n, p->yout);
  if (!rc) rc = mlp_fail(cudaMemsetAsync(p->loss, 0, sizeof(float), s));
  if (!rc) {
    k_mse<<<grid1((size_t)n * dl), 256, 0, s>>>(n, dl, p->yout, d_t, p->dz[p->nl - 1], ldz(p, p->nl - 1), p->loss,
                                                nullptr, nullptr, p->d_lw);
    rc = mlp_bwd(p, n, nullptr);
  }
  if (!rc) rc = mlp_fail(cudaGetLastError());
  if (!rc && loss) rc = mlp_fail(cudaMemcpyAsync(loss, p->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
  const int r2 = mlp_fail(cudaStreamSynchronize(s));
  return rc ? rc : r2 ? r2 : mlp_tc_status(p);
}

// Mini-batch Adam training over n device rows for `epochs` passes (rows
// visited in a fixed permutation per epoch from `seed`); mean loss of the
// last epoch to *loss.
int fz_mlp_train_device(fz_mlp* p, int n, const float* d_x, const float* d_t, int batch, int epochs, float lr,
                        unsigned long long seed, float* loss) {
  if (!p || n <= 0 || !d_x || !d_t || batch <= 0 || epochs <= 0) return FZ_ERR_ARG;
  MLP_CK(cudaSetDevice(p->device));
  int rc = mlp_reserve(p, batch);
  if (rc) return rc;
  cudaStream_t s = p->stream;
  const int d0 = p->dim[0], dl = p->dim[p->nl];
  const int nb = n / batch;
  if (nb <= 0) return FZ_ERR_ARG;
  if (!p->tstate && (rc = mlp_fail(cudaMalloc(&p->tstate, sizeof(TrainState))))) return rc;
  if (nb > p->order_cap) {
    cudaFree(p->order);
    p->order = nullptr;
    p->order_cap = 0;
    if ((rc = mlp_fail(cudaMalloc(&p->order, nb * sizeof(int))))) return rc;
    p->order_cap = nb;
  }
  // One training step (batch gather, forward, loss, backward, Adam, state
  // advance) captured once as a CUDA graph and replayed for every batch: the
  // batch offset and the Adam step come from the device state.
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  if ((rc = mlp_fail(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)))) return rc;
  {
    const AdamK k{lr, 0.9f, 0.999f, 1e-8f};
    k_batch_bf16<<<grid1((size_t)batch * d0 / 8), 256, 0, s>>>(batch, d0, d_x, p->order, p->tstate, p->act[0]);
    rc = mlp_fwd(p, batch, p->yout);
    if (!rc) {
      k_mse<<<grid1((size_t)batch * dl), 256, 0, s>>>(batch, dl, p->yout, d_t, p->dz[p->nl - 1], ldz(p, p->nl - 1),
                                                      p->loss, p->order, p->tstate, p->d_lw);
      rc = mlp_bwd(p, batch, &k);
    }
  }
  const int r2 = mlp_fail(cudaStreamEndCapture(s, &graph));
  if (!rc) rc = r2;
  if (!rc) rc = mlp_fail(cudaGraphInstantiate(&exec, graph, 0));
  // batch order: a fixed random permutation of the batch indices per epoch
  std::vector<int> order(nb);
  unsigned long long st = seed | 1ull;
  float last = 0.0f;
  for (int e = 0; e < epochs && !rc; ++e) {
    for (int i = 0; i < nb; ++i) order[i] = i;
    for (int i = nb - 1; i > 0; --i) {
      st ^= st << 13;
      st ^= st >> 7;
      st ^= st << 17;
      const int j = (int)(st % (unsigned long long)(i + 1));
      std::swap(order[i], order[j]);
    }
    const TrainState ts{0, (int)p->step};
    rc = mlp_fail(cudaMemcpyAsync(p->order, order.data(), nb * sizeof(int), cudaMemcpyHostToDevice, s));
    if (!rc) rc = mlp_fail(cudaMemcpyAsync(p->tstate, &ts, sizeof(ts), cudaMemcpyHostToDevice, s));
    if (!rc) rc = mlp_fail(cudaMemsetAsync(p->loss, 0, sizeof(float), s));
    for (int bi = 0; bi < nb && !rc; ++bi) rc = mlp_fail(cudaGraphLaunch(exec, s));
    p->step += nb;
    float h = 0.0f;
    if (!rc) rc = mlp_fail(cudaMemcpyAsync(&h, p->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    if (!rc) rc = mlp_fail(cudaStreamSynchronize(s));
    last = h / (float)nb;
  }
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  if (!rc) rc = mlp_fail(cudaGetLastError());
  if (!rc) rc = mlp_tc_status(p);
  if (loss) *loss = last;
  return rc;
}

}  // extern "C"
