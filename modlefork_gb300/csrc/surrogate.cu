// surrogate.cu - the learned surrogate's kernels on sm_103a: BF16 tensor-core convolutions
// (tcgen05.mma with FP32 accumulators in tensor memory, operands staged by TMA) for the
// forward pass, the data gradient and the weight gradient of a 1D convolution over
// channels-last activations, and the memory-bound steps around them (pooling, upsampling with
// skip concatenation, bias gradients, loss, Adam, input assembly, the training targets of a
// simulated band and per-map scores).  C ABI in include/mgpu_surrogate.h.
//
// A 1D convolution with `taps` taps (centre tap at offset `pad`) over X[B][L][Cin] is an
// implicit GEMM:
//   Y[b, l, n] = sum_t sum_c X[b, l + t - pad, c] * W[n][t][c]      (M = positions, N = Cout,
//                                                                    K = taps x Cin)
// TMA loads the A tile of tap t directly from X at row offset t - pad, or one tile with the rows of all taps,
// into which tap t's operand starts t rows: rows outside [0, L) come back as zeros, which is the
// convolution's zero padding.  The data gradient is the same
// product with the taps reversed and W transposed; the weight gradient contracts over the
// positions (K = B x L) with both operands M/N-major.
//
// The forward kernels come in four forms (one CTA per tile or persistent; per-thread output
// rows or a staged epilogue that writes 32-row boxes to shared memory and stores them with
// TMA).  The staged epilogue can store the same box to several places at once, which lets a
// U-Net's convolutions fill their skip concatenations, upsampled halves and pooled inputs
// directly (msur_conv_forward_fused).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "../../include/mgpu_surrogate.h"
#include "umma.cuh"

namespace sg {

using bf16 = __nv_bfloat16;
constexpr int BM = 128;  // positions (or output channels in the weight gradient) per tile
constexpr int BK = 64;   // K elements per pipeline stage: one 128-byte swizzle row of BF16
constexpr int THREADS = 192;  // warp 0 TMA, warp 1 MMA (and TMEM), warps 2-5 epilogue

// Error bits of the kernels' bounded waits (msur_take_error).
enum : unsigned { ERR_PRODUCER = 1u, ERR_MMA = 2u, ERR_EPILOGUE = 4u };

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}
// The logistic function 1 / (1 + 2^(-z log2 e)) as two hardware approximations (relative error about 2^-22), SiLU
// and its derivative: the epilogues evaluate one per output element.  Flushing subnormals loses nothing here:
// added to 1 a subnormal exponential vanishes, and the reciprocal of a sum above 2^126 is 0, the limit.  SiLU
// compared over all 2^32 arguments with z times the fast division 1 / (1 + __expf(-z)): the same outputs.
__device__ __forceinline__ float logistic(float z) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.44269504088896340736f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
__device__ __forceinline__ float silu(float z) { return z * logistic(z); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = logistic(z);
  return s * (1.0f + z * (1.0f - s));
}

// ---------------------------------------------------------------------------------------
// Forward / data-gradient convolution: K-major A (activations) and B (weights)
// ---------------------------------------------------------------------------------------
struct ConvArgs {
  CUtensorMap tm_a;  // activations [B][L][Cin]: dims {Cin, L, B}, box {64, 128, 1}
  CUtensorMap tm_b;  // weights [N][taps * Cin]: dims {taps * Cin, N}, box {64, BN}
  int B, L, Cin, taps, pad;
  int n_valid;     // output channels written (columns >= n_valid are dropped)
  int out_stride;  // elements per output row
  int act;         // MSUR_ACT_*
  const float* bias;   // [n_valid] or null
  const bf16* gate;    // multiply by silu'(gate[row, col]) (row stride out_stride) or null
  bf16* out_pre;       // value before the activation, or null
  bf16* out_post;      // value after the activation, or null
  float* out_f32;      // FP32 value before the activation, or null
  unsigned* err;
  // staged epilogue: each epilogue warp writes its 32 rows of a 64-column unit to
  // shared memory and stores them with TMA.  Maps over [B][L][n_valid] with row stride
  // out_stride and 128-byte swizzled boxes of 32 rows: FP32 boxes of 32 columns, BF16 of 64.
  CUtensorMap tm_f32, tm_pre, tm_post;
  // fused copies of the post-activation output (staged epilogue only): a second copy into
  // another row-strided buffer (the skip half of a concatenation), and an upsampled copy, each
  // output row l stored at rows 2l and 2l + 1 of its buffer (two maps over the even and the odd
  // rows); out_post may then be null
  CUtensorMap tm_skip, tm_dup0, tm_dup1;
  // and an average-pooled copy: rows 2m and 2m + 1 of a staged box into row m, as msur_pool2 computes it
  // from the BF16 values (16-row boxes)
  CUtensorMap tm_pool;
  int has_skip, has_dup, has_pool;
};

constexpr int STAGE_OUT_BYTES = 4 * 2 * 4096;  // four epilogue warps x two 4 KB buffers

template <int BN>
__host__ __device__ constexpr uint32_t tmem_cols() {
  return BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : (BN <= 256 ? 256 : 512)));
}

// Epilogue of one 32-column chunk of one output row: bias, the gated SiLU derivative, and
// the FP32 / pre-activation / post-activation stores (columns >= n_valid dropped).
__device__ __forceinline__ void conv_epilogue_chunk(const ConvArgs& a, float (&v)[32], size_t row, int col0) {
  const int nv = min(32, a.n_valid - col0);
  const size_t off = row * a.out_stride + col0;
  if (a.bias) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] += (j < nv) ? __ldg(a.bias + col0 + j) : 0.0f;
  }
  if (a.gate) {
    if (nv == 32) {
      const uint4* g4 = reinterpret_cast<const uint4*>(a.gate + off);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 u = __ldg(g4 + k);
        const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const __nv_bfloat162 g2 = *reinterpret_cast<const __nv_bfloat162*>(&w4[h]);
          v[8 * k + 2 * h] *= dsilu(__low2float(g2));
          v[8 * k + 2 * h + 1] *= dsilu(__high2float(g2));
        }
      }
    } else {
      for (int j = 0; j < nv; ++j) v[j] *= dsilu(__bfloat162float(a.gate[off + j]));
    }
  }
  if (a.out_f32) {
    if (nv == 32) {
      float4* o4 = reinterpret_cast<float4*>(a.out_f32 + off);
#pragma unroll
      for (int k = 0; k < 8; ++k) o4[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    } else {
      for (int j = 0; j < nv; ++j) a.out_f32[off + j] = v[j];
    }
  }
  if (a.out_pre) {
    if (nv == 32) {
      uint4* o4 = reinterpret_cast<uint4*>(a.out_pre + off);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t w4[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const __nv_bfloat162 p = __floats2bfloat162_rn(v[8 * k + 2 * h], v[8 * k + 2 * h + 1]);
          w4[h] = *reinterpret_cast<const uint32_t*>(&p);
        }
        o4[k] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
      }
    } else {
      for (int j = 0; j < nv; ++j) a.out_pre[off + j] = __float2bfloat16(v[j]);
    }
  }
  if (a.out_post) {
    if (a.act == MSUR_ACT_SILU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
    }
    if (nv == 32) {
      uint4* o4 = reinterpret_cast<uint4*>(a.out_post + off);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t w4[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const __nv_bfloat162 p = __floats2bfloat162_rn(v[8 * k + 2 * h], v[8 * k + 2 * h + 1]);
          w4[h] = *reinterpret_cast<const uint32_t*>(&p);
        }
        o4[k] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
      }
    } else {
      for (int j = 0; j < nv; ++j) a.out_post[off + j] = __float2bfloat16(v[j]);
    }
  }
}

// One 32-row x 128-byte box goes through this warp's staging buffer (one or two 4 KB buffers used in
// turn; nb counts the warp's stores).  stage_begin waits until the buffer's previous store has
// read it; the lanes then write their rows with the 128-byte swizzle (16-byte unit k of row r at
// unit k ^ (r % 8), which also keeps the eight lanes of each vector store on distinct banks);
// stage_end makes the writes visible to the bulk-copy proxy and lane 0 issues the TMA store.
__device__ __forceinline__ uint8_t* stage_begin(uint8_t* stg, int nb, int bufs) {
  if (nb >= bufs && umma::elect()) {
    if (bufs == 2) umma::bulk_wait_read<1>();
    else umma::bulk_wait_read<0>();
  }
  __syncwarp();
  return stg + (bufs == 2 ? (nb & 1) * 4096 : 0);
}
__device__ __forceinline__ void stage_put(uint8_t* buf, int k, uint4 w) {
  const int lane = threadIdx.x & 31;
  *reinterpret_cast<uint4*>(buf + lane * 128 + ((k ^ (lane & 7)) << 4)) = w;
}
__device__ __forceinline__ void stage_end(const CUtensorMap* map, uint8_t* buf, int& nb, int x, int y, int z) {
  umma::fence_async_smem();
  __syncwarp();
  if (umma::elect()) {
    umma::tma_store_3d(map, buf, x, y, z);
    umma::bulk_commit();
  }
  __syncwarp();  // a tcgen05.ld may follow, which wants the warp converged
  ++nb;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// 32 columns (col0 ..) of this thread's row as the epilogue's value: accumulator, bias, gated SiLU derivative.
__device__ __forceinline__ void conv_value32(const ConvArgs& a, uint32_t tmem_cols32, const bf16* gate, int col0,
                                             float (&v)[32]) {
  umma::tmem_ld32(tmem_cols32, v);
  const int nv = a.n_valid - col0;
  if (a.bias) {
    if (nv >= 32 && (reinterpret_cast<uintptr_t>(a.bias) & 15u) == 0) {
      const float4* b4 = reinterpret_cast<const float4*>(a.bias + col0);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float4 bb = __ldg(b4 + k);
        v[4 * k] += bb.x;
        v[4 * k + 1] += bb.y;
        v[4 * k + 2] += bb.z;
        v[4 * k + 3] += bb.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] += (j < nv) ? __ldg(a.bias + col0 + j) : 0.0f;
    }
  }
  if (gate) {
    if (nv >= 32) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(gate) + k);
        const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const __nv_bfloat162 g2 = *reinterpret_cast<const __nv_bfloat162*>(&w4[h]);
          v[8 * k + 2 * h] *= dsilu(__low2float(g2));
          v[8 * k + 2 * h + 1] *= dsilu(__high2float(g2));
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < nv) v[j] *= dsilu(__bfloat162float(gate[j]));
    }
  }
}

// Staged epilogue of one unit: 32 rows (y .. y+31 of sequence z) x 64 columns from col0: the FP32 (two boxes),
// pre-activation and post-activation (one box each) outputs through shared memory and TMA.  Rows >= L and
// columns >= n_valid are dropped by the stores.  Collective over the warp; the caller waits for the
// stores (staged_drain) before the block exits.
//
// One pass over the accumulator per output, 32 columns at a time: a warp comes through here once per tile, so what
// it runs has to be short loops.  As straight code over 64 columns and all outputs at once the fetches bound
// it: 8100 cycles for 128 columns, of which 5300 with every memory operation and all arithmetic left out.
__device__ __forceinline__ void conv_epilogue_unit(const ConvArgs& a, uint32_t tmem_unit, uint8_t* stg, int bufs,
                                                   int& nb, int col0, int y, int z) {
  if (y >= a.L || col0 >= a.n_valid) return;
  const int lane = threadIdx.x & 31;
  // rows past the end read the last row's gate; their values are dropped
  const bf16* gate = a.gate ? a.gate + (static_cast<size_t>(z) * a.L + min(y + lane, a.L - 1)) * a.out_stride + col0
                            : nullptr;
  if (a.out_f32) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      if (col0 + 32 * h >= a.n_valid) break;
      float v[32];
      conv_value32(a, tmem_unit + 32 * h, gate ? gate + 32 * h : nullptr, col0 + 32 * h, v);
      uint8_t* buf = stage_begin(stg, nb, bufs);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        stage_put(buf, k, make_uint4(__float_as_uint(v[4 * k]), __float_as_uint(v[4 * k + 1]),
                                     __float_as_uint(v[4 * k + 2]), __float_as_uint(v[4 * k + 3])));
      stage_end(&a.tm_f32, buf, nb, col0 + 32 * h, y, z);
    }
  }
  const bool post = a.out_post || a.has_skip || a.has_dup || a.has_pool;
#pragma unroll 1
  for (int out = a.out_pre ? 0 : 1; out < (post ? 2 : 1); ++out) {
    uint8_t* buf = stage_begin(stg, nb, bufs);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      float v[32];
      conv_value32(a, tmem_unit + 32 * h, gate ? gate + 32 * h : nullptr, col0 + 32 * h, v);
      if (out == 1 && a.act == MSUR_ACT_SILU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        stage_put(buf, 4 * h + k,
                  make_uint4(pack_bf16x2(v[8 * k], v[8 * k + 1]), pack_bf16x2(v[8 * k + 2], v[8 * k + 3]),
                             pack_bf16x2(v[8 * k + 4], v[8 * k + 5]), pack_bf16x2(v[8 * k + 6], v[8 * k + 7])));
    }
    // one staged box, stored to every destination of its value
    umma::fence_async_smem();
    __syncwarp();
    if (umma::elect()) {
      if (out == 0) {
        umma::tma_store_3d(&a.tm_pre, buf, col0, y, z);
      } else {
        if (a.out_post) umma::tma_store_3d(&a.tm_post, buf, col0, y, z);
        if (a.has_skip) umma::tma_store_3d(&a.tm_skip, buf, col0, y, z);
        if (a.has_dup) {
          umma::tma_store_3d(&a.tm_dup0, buf, col0, y, z);
          umma::tma_store_3d(&a.tm_dup1, buf, col0, y, z);
        }
      }
      umma::bulk_commit();
    }
    __syncwarp();
    ++nb;
    if (out == 1 && a.has_pool) {
      // rows 2m and 2m + 1 of the staged box are averaged into row m of a 16-row box (y is a multiple of 32):
      // 16 rows x 8 units of 16 bytes, four to a lane
      uint4 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (lane >> 3) + 4 * i, k = lane & 7;
        const uint4 p0 = *reinterpret_cast<const uint4*>(buf + 2 * m * 128 + ((k ^ ((2 * m) & 7)) << 4));
        const uint4 p1 = *reinterpret_cast<const uint4*>(buf + (2 * m + 1) * 128 + ((k ^ ((2 * m + 1) & 7)) << 4));
        const uint32_t x0[4] = {p0.x, p0.y, p0.z, p0.w}, x1[4] = {p1.x, p1.y, p1.z, p1.w};
        uint32_t q[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x0[h]));
          const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x1[h]));
          q[h] = pack_bf16x2(0.5f * (fa.x + fb.x), 0.5f * (fa.y + fb.y));
        }
        w[i] = make_uint4(q[0], q[1], q[2], q[3]);
      }
      uint8_t* pbuf = stage_begin(stg, nb, bufs);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (lane >> 3) + 4 * i, k = lane & 7;
        *reinterpret_cast<uint4*>(pbuf + m * 128 + ((k ^ (m & 7)) << 4)) = w[i];
      }
      stage_end(&a.tm_pool, pbuf, nb, col0, y >> 1, z);
    }
  }
}

// Every TMA store of this warp has completed (before the block and its shared memory exit).
__device__ __forceinline__ void staged_drain() {
  if (umma::elect()) umma::bulk_wait_all();
  __syncwarp();
}

template <int BN, int STAGES, bool STAGED>
__global__ void __launch_bounds__(THREADS, 1) conv_fwd_kernel(const __grid_constant__ ConvArgs a) {
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TCOLS = tmem_cols<BN>();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = umma::warp_index(), lane = threadIdx.x % 32;
  const int n0 = blockIdx.x * BN, l0 = blockIdx.y * BM, b = blockIdx.z;
  const int kc = a.Cin / BK;
  const int nk = a.taps * kc;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    umma::mbar_init(done, 1);
    umma::fence_barrier_init();
    umma::tma_prefetch(&a.tm_a);
    umma::tma_prefetch(&a.tm_b);
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, TCOLS);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  umma::pdl_wait();
  umma::pdl_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    int issued = 0;
    for (int s = 0; s < nk; ++s) {
      const int st = s % STAGES;
      if (!umma::mbar_wait_warp(&empty[st], ((s / STAGES) & 1) ^ 1, a.err, ERR_PRODUCER)) break;
      uint8_t* sa = smem + st * STAGE_BYTES;
      const int t = s / kc, c0 = (s % kc) * BK;
      if (umma::elect()) {
        umma::mbar_arrive_expect_tx(&full[st], STAGE_BYTES);
        umma::tma_load_3d(sa, &a.tm_a, &full[st], c0, l0 + t - a.pad, b);
        umma::tma_load_2d(sa + A_BYTES, &a.tm_b, &full[st], t * a.Cin + c0, n0);
      }
      issued = s + 1;
    }
    // drain: every issued copy has landed before the block can exit
    for (int s = issued > STAGES ? issued - STAGES : 0; s < issued; ++s)
      umma::mbar_wait_warp(&full[s % STAGES], (s / STAGES) & 1, a.err, ERR_PRODUCER);
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma::idesc_bf16_f32(BM, BN, false, false);
    for (int s = 0; s < nk; ++s) {
      const int st = s % STAGES;
      if (!umma::mbar_wait_warp(&full[st], (s / STAGES) & 1, a.err, ERR_MMA)) break;
      const uint32_t sa = umma::smem_u32(smem + st * STAGE_BYTES);
      if (umma::elect()) {
        umma::mma_bf16_x4<2>(tmem, umma::sdesc_sw128_lo(sa), umma::sdesc_sw128_lo(sa + A_BYTES), idesc, s);
        umma::mma_commit(&empty[st]);
      }
    }
    if (umma::elect()) umma::mma_commit(done);
    __syncwarp();
  } else {
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, one output row per thread
    const int q = warp & 3;
    const int l = l0 + 32 * q + lane;
    const bool row_ok = l < a.L;
    const size_t row = static_cast<size_t>(b) * a.L + (row_ok ? l : 0);
    const bool ok = umma::mbar_wait_warp(done, 0, a.err, ERR_EPILOGUE);
    umma::fence_after_sync();
    if constexpr (STAGED) {
      if (ok) {
        int nb = 0;
#pragma unroll 1
        for (int u = 0; u < BN / 64; ++u)
          conv_epilogue_unit(a, tmem + (static_cast<uint32_t>(32 * q) << 16) + u * 64,
                             smem + STAGES * STAGE_BYTES + 1024 + q * 8192, 2, nb, n0 + u * 64, l0 + 32 * q, b);
        staged_drain();
      }
    } else if (ok) {
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        float v[32];
        umma::tmem_ld32(tmem + (static_cast<uint32_t>(32 * q) << 16) + c * 32, v);
        const int col0 = n0 + c * 32;
        if (row_ok && col0 < a.n_valid) conv_epilogue_chunk(a, v, row, col0);
        __syncwarp();  // tcgen05.ld is .sync.aligned: the rows past the end rejoin before the next one
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, TCOLS);
  }
}

// ---------------------------------------------------------------------------------------
// The same convolution as a persistent kernel: each CTA walks tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ... (N tile fastest, then position tile, then sequence) with two to eight
// TMEM accumulators, so the epilogue of one tile overlaps the MMAs of the next and a CTA's
// set-up (barriers, TMEM allocation, tensor-map prefetch) is paid once.
//
// What bounds it: with few input channels memory and the epilogue (two transcendental operations per element),
// with many the operands' way from L2 to shared memory (about 70 bytes per clock and SM), between them the
// MMA warp's own steps.  So
//  - up to four groups of four epilogue warps take the 64-column units of the tiles in turn;
//  - a tile's activations are loaded once for all taps (ConvPlan::aslots): the chunk of 64 input channels is
//    kept as 128 + taps - 1 rows, and tap t's operand starts t rows into it;
//  - weights whose K steps all fit stay for the CTA's life (ConvPlan::wres).
// The order of the products (tap, then channel) is that of the plain form, so are the results.
// 256 maps, with four epilogue warps, both operands by stage and single-thread loops / now: 192 to 64 channels
// at 4000 positions 174 / 87 us, 128 to 128 at 2000 82 / 48, 384 to 128 at 2000 171 / 117, 896 to 384 at
// 500 271 / 173 (with tiles of 192 columns instead of 128), 1024 to 512 at 250 129 / 117.
//
// Warps: 0 weights (and activations per K step without slots), 1 MMA and TMEM, 2 activation
// slots, from 4 on the epilogue (warp w reads TMEM lanes 32 (w % 4) .. +31).
// Barriers: full / empty per stage and afull / aempty per slot (TMA <-> MMA), tfull / tempty per
// accumulator (MMA <-> epilogue warps), done (the MMA issuer's last commit).
// ---------------------------------------------------------------------------------------
constexpr int PTHREADS = 640;  // at most: four warps and up to four groups of four epilogue warps
constexpr int SLOT_BYTES = (BM + 8) * BK * 2;  // a chunk of up to 8 more rows than the tile, 1 KB aligned
constexpr int MAX_STAGES = 16, MAX_SLOTS = 12;

struct ConvPlan {
  int ntn, ntl, ntiles;
  int stages;  // operand stages
  int aslots;  // activation slots (0: activations travel with the weights, stage by stage)
  int wres;    // stages == K steps: every CTA keeps one N tile and loads its weights once
  int groups;  // groups of four epilogue warps
  int bufs;    // 4 KB staging buffers per epilogue warp (0: epilogue without staging)
};

// Shared-memory addresses of the persistent kernel's barriers (arrays of 8 bytes) and buffers.
struct ConvSmem {
  uint32_t full, empty, afull, aempty, tfull, tempty, done, ring, slots;
};

// The MMA warp's loop.  What it issues runs behind it, so a step of the loop must not take longer than its
// products (64 to 512 cycles per K step): addresses are stepped, the next stage's barrier is tested before the
// step's products go out, and the first and last tap, which acquire and release slots, have loops of their own.
template <int BN, int ACCS, bool ASLOTS, bool WRES>
__device__ __forceinline__ void conv_mma_loop(const ConvArgs& a, const ConvPlan& p, const ConvSmem& m, uint32_t tmem,
                                              int kc) {
  constexpr uint32_t idesc = umma::idesc_bf16_f32(BM, BN, false, false);
  constexpr uint32_t W_BYTES = BN * BK * 2, STAGE = W_BYTES + (ASLOTS ? 0 : BM * BK * 2);
  const uint32_t full_end = m.full + 8 * p.stages;
  const int taps = a.taps;
  int acc = 0, base = 0;              // accumulator, slot of the tile's first chunk
  uint32_t tph = 1, ph = 0, aph = 0;  // parities of the phases waited for
  uint32_t fb = m.full, sb = m.ring;  // the stage's barrier and operands
  uint32_t d = tmem, accumulate = 0;
  bool first = true;
  bool ready = !WRES && umma::mbar_test(fb, 0);
  auto tap_loop = [&](auto acquire, auto release, int tap) {
    uint32_t sa = m.slots + base * SLOT_BYTES + tap * (BK * 2), sl = 8 * base;
    if (WRES && !first && !decltype(acquire)::value) {  // nothing to wait for
      if (umma::elect()) {
        uint32_t a_lo = umma::sdesc_sw128_lo(sa), b_lo = umma::sdesc_sw128_lo(sb);
        for (int c = 0; c < kc; ++c) {
          umma::mma_bf16_x4<2>(d, a_lo, b_lo, idesc, 1);
          if (decltype(release)::value) umma::mma_commit(m.aempty + sl + 8 * c);
          a_lo += SLOT_BYTES / 16;
          b_lo += W_BYTES / 16;
        }
      }
      sb += kc * W_BYTES;
      if (decltype(release)::value) fb = m.full, sb = m.ring;
      return true;
    }
    for (int c = 0; c < kc; ++c) {
      if (ASLOTS && decltype(acquire)::value)
        if (!umma::mbar_wait_warp(m.afull + sl, aph, a.err, ERR_MMA)) return false;
      if (WRES ? first : !__all_sync(0xFFFFFFFFu, ready))
        if (!umma::mbar_wait_warp(fb, ph, a.err, ERR_MMA)) return false;
      const uint32_t eb = fb + (m.empty - m.full);
      const uint32_t b_lo = umma::sdesc_sw128_lo(sb), a_lo = umma::sdesc_sw128_lo(ASLOTS ? sa : sb + W_BYTES);
      fb += 8;
      sb += STAGE;
      if (fb == full_end) fb = m.full, sb = m.ring, ph ^= 1;
      if (!WRES) ready = umma::mbar_test(fb, ph);
      if (umma::elect()) {
        umma::mma_bf16_x4<2>(d, a_lo, b_lo, idesc, accumulate);
        if (!WRES) umma::mma_commit(eb);
        if (ASLOTS && decltype(release)::value) umma::mma_commit(m.aempty + sl);
      }
      accumulate = 1;
      sa += SLOT_BYTES;
      sl += 8;
    }
    if (WRES && decltype(release)::value) fb = m.full, sb = m.ring;
    return true;
  };
  const std::true_type yes;
  const std::false_type no;
  for (int t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
    if (!umma::mbar_wait_warp(m.tempty + 8 * acc, tph, a.err, ERR_MMA)) break;
    umma::fence_after_sync();
    d = tmem + acc * BN;
    accumulate = 0;
    bool ok = true;
    if (!ASLOTS) {
      for (int tap = 0; tap < taps && ok; ++tap) ok = tap_loop(no, no, tap);
    } else if (taps == 1) {
      ok = tap_loop(yes, yes, 0);
    } else {
      ok = tap_loop(yes, no, 0);
      for (int tap = 1; tap < taps - 1 && ok; ++tap) ok = tap_loop(no, no, tap);
      if (ok) ok = tap_loop(no, yes, taps - 1);
    }
    if (!ok) break;
    if (umma::elect()) umma::mma_commit(m.tfull + 8 * acc);
    if (++acc == ACCS) acc = 0, tph ^= 1;
    if (ASLOTS && (base += kc) == p.aslots) base = 0, aph ^= 1;
    first = false;
  }
  // every MMA this warp issued has completed before TMEM is released
  if (umma::elect()) umma::mma_commit(m.done);
  umma::mbar_wait_warp(m.done, 0, a.err, ERR_MMA);
}

// The tiles of a CTA one after the other, without dividing for each (four dependent divisions were a third of
// a short tile's time).
struct TileWalk {
  int t, n, l, b, dn, dl, db;
  __device__ explicit TileWalk(const ConvPlan& p)
      : t(blockIdx.x), n(blockIdx.x % p.ntn), l((blockIdx.x / p.ntn) % p.ntl), b(blockIdx.x / (p.ntn * p.ntl)),
        dn(gridDim.x % p.ntn), dl((gridDim.x / p.ntn) % p.ntl), db(gridDim.x / (p.ntn * p.ntl)) {}
  __device__ void next(const ConvPlan& p) {
    t += gridDim.x;
    n += dn;
    l += dl;
    b += db;
    if (n >= p.ntn) n -= p.ntn, ++l;
    if (l >= p.ntl) l -= p.ntl, ++b;
  }
};

template <int BN, bool STAGED>
__global__ void __launch_bounds__(PTHREADS, 1)
    conv_fwd_persistent_kernel(const __grid_constant__ ConvArgs a, const __grid_constant__ ConvPlan p) {
  constexpr int W_BYTES = BN * BK * 2;
  constexpr int ACCS = BN == 64 ? 8 : (BN == 128 ? 4 : 2);
  constexpr uint32_t TCOLS = tmem_cols<ACCS * BN>();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const slots = align1024(smem_raw);
  uint8_t* const ring = slots + p.aslots * SLOT_BYTES;
  const int stage_bytes = W_BYTES + (p.aslots ? 0 : BM * BK * 2);
  uint8_t* const bars = ring + p.stages * stage_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(bars);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* afull = empty + MAX_STAGES;
  uint64_t* aempty = afull + MAX_SLOTS;
  uint64_t* tfull = aempty + MAX_SLOTS;
  uint64_t* tempty = tfull + 8;
  uint64_t* done = tempty + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = umma::warp_index(), lane = threadIdx.x % 32;
  const int kc = a.Cin / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < p.aslots; ++s) {
      umma::mbar_init(&afull[s], 1);
      umma::mbar_init(&aempty[s], 1);
    }
    for (int k = 0; k < ACCS; ++k) {
      umma::mbar_init(&tfull[k], 1);
      umma::mbar_init(&tempty[k], 4 * (BN / 64));
    }
    umma::mbar_init(done, 1);
    umma::fence_barrier_init();
    umma::tma_prefetch(&a.tm_a);
    umma::tma_prefetch(&a.tm_b);
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, TCOLS);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  umma::pdl_wait();
  umma::pdl_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    int st = 0, issued = 0;
    uint32_t ph = 1;  // parity of the empty barrier's phase before the first
    bool ok = true;
    for (TileWalk w(p); w.t < p.ntiles && ok; w.next(p)) {
      const int n0 = w.n * BN, l0 = w.l * BM;
      for (int tap = 0; tap < a.taps && ok; ++tap) {
        for (int c = 0; c < kc; ++c) {
          ok = umma::mbar_wait_warp(&empty[st], ph, a.err, ERR_PRODUCER);
          if (!ok) break;
          uint8_t* dst = ring + st * stage_bytes;
          if (umma::elect()) {
            umma::mbar_arrive_expect_tx(&full[st], stage_bytes);
            if (!p.aslots) umma::tma_load_3d(dst + W_BYTES, &a.tm_a, &full[st], c * BK, l0 + tap - a.pad, w.b);
            umma::tma_load_2d(dst, &a.tm_b, &full[st], tap * a.Cin + c * BK, n0);
          }
          ++issued;
          if (++st == p.stages) st = 0, ph ^= 1;
        }
      }
      if (p.wres) break;
    }
    // drain: every issued copy has landed before the block can exit
    for (int q = max(0, issued - p.stages); q < issued; ++q)
      umma::mbar_wait_warp(&full[q % p.stages], (q / p.stages) & 1, a.err, ERR_PRODUCER);
  } else if (warp == 2) {
    const uint32_t bytes = (BM + a.taps - 1) * BK * 2;
    int sl = 0, issued = 0;
    uint32_t ph = 1;
    bool ok = p.aslots > 0;
    for (TileWalk w(p); w.t < p.ntiles && ok; w.next(p)) {
      for (int c = 0; c < kc; ++c) {
        ok = umma::mbar_wait_warp(&aempty[sl], ph, a.err, ERR_PRODUCER);
        if (!ok) break;
        if (umma::elect()) {
          umma::mbar_arrive_expect_tx(&afull[sl], bytes);
          umma::tma_load_3d(slots + sl * SLOT_BYTES, &a.tm_a, &afull[sl], c * BK, w.l * BM - a.pad, w.b);
        }
        ++issued;
        if (++sl == p.aslots) sl = 0, ph ^= 1;
      }
    }
    for (int q = max(0, issued - p.aslots); q < issued; ++q)
      umma::mbar_wait_warp(&afull[q % p.aslots], (q / p.aslots) & 1, a.err, ERR_PRODUCER);
  } else if (warp == 1) {
    const ConvSmem m{umma::smem_u32(full),  umma::smem_u32(empty),  umma::smem_u32(afull),
                     umma::smem_u32(aempty), umma::smem_u32(tfull), umma::smem_u32(tempty),
                     umma::smem_u32(done),  umma::smem_u32(ring),   umma::smem_u32(slots)};
    if (p.wres) {
      conv_mma_loop<BN, ACCS, true, true>(a, p, m, tmem, kc);
    } else if (p.aslots) {
      conv_mma_loop<BN, ACCS, true, false>(a, p, m, tmem, kc);
    } else {
      conv_mma_loop<BN, ACCS, false, false>(a, p, m, tmem, kc);
    }
  } else if (warp >= 4) {
    // the CTA's 64-column units, tile after tile, go round the groups
    constexpr int UNITS = BN / 64;
    const int q = warp & 3;
    uint8_t* const stg = bars + 1024 + (warp - 4) * p.bufs * 4096;
    int acc = 0, nb = 0, u = (warp - 4) >> 2;
    uint32_t ph = 0;
    for (TileWalk w(p);; u += p.groups) {
      while (u >= UNITS) {
        u -= UNITS;
        w.next(p);
        if (++acc == ACCS) acc = 0, ph ^= 1;
      }
      if (w.t >= p.ntiles) break;
      const bool ok = umma::mbar_wait_warp(&tfull[acc], ph, a.err, ERR_EPILOGUE);
      umma::fence_after_sync();
      if (!ok) break;
      const int col0 = w.n * BN + u * 64;
      const int y = w.l * BM + 32 * q;
      const uint32_t unit = tmem + (static_cast<uint32_t>(32 * q) << 16) + acc * BN + u * 64;
      if constexpr (STAGED) {
        conv_epilogue_unit(a, unit, stg, p.bufs, nb, col0, y, w.b);
      } else {
        const int l = y + lane;
        const bool row_ok = l < a.L;
        const size_t row = static_cast<size_t>(w.b) * a.L + (row_ok ? l : 0);
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          float v[32];
          umma::tmem_ld32(unit + c * 32, v);
          if (row_ok && col0 + c * 32 < a.n_valid) conv_epilogue_chunk(a, v, row, col0 + c * 32);
          __syncwarp();
        }
      }
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&tempty[acc]);
    }
    if constexpr (STAGED) staged_drain();
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, TCOLS);
  }
}

// ---------------------------------------------------------------------------------------
// Weight gradient: dW[n][t][c] += sum_{b,l} dZ[b, l, n] X[b, l + t - pad, c], split over the
// (b, 64-position block) range; M = output channels (128 per tile), N = input channels (BN per
// tile), one TMEM accumulator of BN columns per tap; both operands M/N-major.
//
// A block's 64 (+ taps - 1) positions of X are loaded once: tap t's operand starts t rows into them.  Where
// the bias gradient is wanted too, the epilogue warps of the first input-channel tile add up the dZ blocks as they
// pass through shared memory (25 launches of 4 to 17 us in a network's pass).  Together with warp-uniform issue
// loops: the backward pass of 16 maps lost 100 us of 1255 for both passes.
//
// The splits' partial sums meet in dw.  A thread holds one output channel's row of the accumulators;
// adding it word by word (32 rows per warp and instruction) took longer than the products: 113 of
// 133 us for 16 x 999 positions, 256 to 256 channels.  So eight warps put half a tap's row per thread into shared
// memory (rows padded by 16 bytes: conflict-free 16-byte stores), and each thread adds its row with one bulk
// reduction (cp.reduce.async.bulk, up to 256 contiguous bytes) that runs while the next tap is read, or
// the next accumulation's products.  16 x 2000 positions, 128 to 128 channels: 15.6 us with four warps and all
// reductions at the end, of which 4.5 and 6.3 were these two.
// ---------------------------------------------------------------------------------------
constexpr int WTHREADS = 320;  // warp 0 TMA, warp 1 MMA and TMEM, warps 2-9 epilogue

struct WgradArgs {
  CUtensorMap tm_dz;  // [B][L][Cout]: dims {Cout, L, B}, box {64, 64, 1}
  CUtensorMap tm_x;   // [B][L][Cin]: dims {Cin, L, B}, box {64, 64 + taps - 1, 1}
  int B, L, Cin, Cout, taps, pad;
  int lblocks;        // 64-position blocks per sequence
  int total;          // B * lblocks
  int per_split;      // blocks per split
  int per_phase;      // blocks per accumulation: a split's accumulators are added to dw this often
  int bulk;           // dw is 16-byte aligned: bulk reductions
  float* dw;          // [Cout][taps][Cin], accumulated into
  float* db;          // [Cout], accumulated into, or null
  unsigned* err;
};

template <int NT>
__host__ __device__ constexpr int wgrad_box_bytes() {  // 64 + NT - 1 rows, 1 KB aligned
  return (64 + (NT > 1 ? 8 : 0)) * 128;
}
template <int BN, int NT>
__host__ __device__ constexpr int wgrad_stage_bytes() {
  return 2 * 8192 + (BN / 64) * wgrad_box_bytes<NT>();
}
// A thread's staging row: half a tap's columns, padded by 16 bytes.
template <int BN>
__host__ __device__ constexpr int wgrad_row_bytes() {
  return BN / 2 * 4 + 16;
}

template <int BN, int NT, int STAGES>
__global__ void __launch_bounds__(WTHREADS, 1) wgrad_kernel(const __grid_constant__ WgradArgs a) {
  constexpr int BOX = 64 * 64 * 2;  // one 64 x 64 BF16 box
  constexpr int A_BYTES = 2 * BOX;  // 128 output channels
  constexpr int XBOX = wgrad_box_bytes<NT>();
  constexpr int STAGE_BYTES = wgrad_stage_bytes<BN, NT>();
  constexpr uint32_t STAGE_LOAD = A_BYTES + (BN / 64) * (64 + NT - 1) * 128;
  constexpr uint32_t TCOLS = NT * BN <= 128 ? 128 : (NT * BN <= 256 ? 256 : 512);
  static_assert(NT * BN <= 512, "accumulators exceed tensor memory");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* const staging = smem + STAGES * STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + 256 * wgrad_row_bytes<BN>());
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint64_t* drained = done + 1;  // the accumulators have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  float* bias_part = reinterpret_cast<float*>(full + 32);  // [4 warps][128 channels]

  const int warp = umma::warp_index(), lane = threadIdx.x % 32;
  const int c0 = blockIdx.x * BN, n0 = blockIdx.y * BM;
  const int kb0 = blockIdx.z * a.per_split;
  const int kb1 = min(a.total, kb0 + a.per_split);
  const int nk = kb1 > kb0 ? kb1 - kb0 : 0;
  const bool bias = a.db != nullptr && blockIdx.x == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], bias ? 5 : 1);  // the products, and the warps that add up dZ
    }
    umma::mbar_init(done, 1);
    umma::mbar_init(drained, 8);
    umma::fence_barrier_init();
    umma::tma_prefetch(&a.tm_dz);
    umma::tma_prefetch(&a.tm_x);
  }
  if (warp == 1) umma::tmem_alloc(tmem_slot, TCOLS);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  umma::pdl_wait();
  umma::pdl_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    int issued = 0, st = 0;
    uint32_t ph = 1;
    int bb = kb0 / a.lblocks, l0 = (kb0 % a.lblocks) * 64;
    for (int s = 0; s < nk; ++s) {
      if (!umma::mbar_wait_warp(&empty[st], ph, a.err, ERR_PRODUCER)) break;
      uint8_t* sa = smem + st * STAGE_BYTES;
      if (umma::elect()) {
        umma::mbar_arrive_expect_tx(&full[st], STAGE_LOAD);
        umma::tma_load_3d(sa, &a.tm_dz, &full[st], n0, l0, bb);
        umma::tma_load_3d(sa + BOX, &a.tm_dz, &full[st], n0 + 64, l0, bb);
#pragma unroll
        for (int j = 0; j < BN / 64; ++j)
          umma::tma_load_3d(sa + A_BYTES + j * XBOX, &a.tm_x, &full[st], c0 + 64 * j, l0 - a.pad, bb);
      }
      issued = s + 1;
      if (++st == STAGES) st = 0, ph ^= 1;
      if ((l0 += 64) >= a.lblocks * 64) l0 = 0, ++bb;
    }
    for (int s = issued > STAGES ? issued - STAGES : 0; s < issued; ++s)
      umma::mbar_wait_warp(&full[s % STAGES], (s / STAGES) & 1, a.err, ERR_PRODUCER);
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma::idesc_bf16_f32(BM, BN, true, true);
    int st = 0, in = 0;  // stage, blocks in this accumulation
    uint32_t ph = 0, dph = 0;
    for (int s = 0; s < nk; ++s) {
      if (in == a.per_phase) {
        if (umma::elect()) umma::mma_commit(done);
        if (!umma::mbar_wait_warp(drained, dph, a.err, ERR_MMA)) break;
        umma::fence_after_sync();
        dph ^= 1;
        in = 0;
      }
      if (!umma::mbar_wait_warp(&full[st], ph, a.err, ERR_MMA)) break;
      const uint32_t sa = umma::smem_u32(smem) + st * STAGE_BYTES;
      const uint32_t a_lo = umma::sdesc_sw128_lo(sa, BOX), b_lo = umma::sdesc_sw128_lo(sa + A_BYTES, XBOX);
      if (umma::elect()) {
#pragma unroll
        for (int t = 0; t < NT; ++t) umma::mma_bf16_x4<128>(tmem + t * BN, a_lo, b_lo + 8 * t, idesc, in);
        umma::mma_commit(&empty[st]);
      }
      ++in;
      if (++st == STAGES) st = 0, ph ^= 1;
    }
    if (umma::elect()) umma::mma_commit(done);
    __syncwarp();
  } else if (nk > 0) {
    constexpr int HALF = BN / 2;
    const int q = warp & 3, half = warp >= 6;
    const int n = n0 + 32 * q + lane, cc = c0 + half * HALF;
    const bool inside = n < a.Cout && cc < a.Cin;
    const uint32_t cols = tmem + (static_cast<uint32_t>(32 * q) << 16) + half * HALF;
    uint8_t* const row = staging + (threadIdx.x - 64) * wgrad_row_bytes<BN>();
    // bias: thread e: 8 channels (16-byte unit e % 16 of the two boxes), rows 8 (e / 16) .. + 7 of each block
    const int e = threadIdx.x - 64, unit = e & 15;
    float sum[8] = {};
    int st = 0;
    uint32_t ph = 0, dph = 0;
    bool ok = true;
    for (int s0 = 0; s0 < nk && ok; s0 += a.per_phase, dph ^= 1) {
      if (bias && !half) {
        const int s1 = min(nk, s0 + a.per_phase);
        for (int s = s0; s < s1; ++s) {
          ok = umma::mbar_wait_warp(&full[st], ph, a.err, ERR_EPILOGUE);
          if (!ok) break;
          const uint32_t rows = umma::smem_u32(smem) + st * STAGE_BYTES + (unit >> 3) * BOX + (e >> 4) * 1024;
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            uint32_t x[4];
            umma::ld_shared_v4(x, rows + r * 128 + (((unit & 7) ^ r) << 4));
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[h]));
              sum[2 * h] += f.x;
              sum[2 * h + 1] += f.y;
            }
          }
          // Reads through the generic proxy before a write through the async one: an arrival alone does not
          // order them, and rows were seen to be lost to the copy that fills this stage next.  Every lane
          // fences its own loads, then one arrives for the warp.
          umma::fence_async_smem();
          __syncwarp();
          if (lane == 0) umma::mbar_arrive(&empty[st]);
          if (++st == STAGES) st = 0, ph ^= 1;
        }
        if (!ok) break;
      }
      ok = umma::mbar_wait_warp(done, dph, a.err, ERR_EPILOGUE);
      if (!ok) break;
      umma::fence_after_sync();
      // tap by tap: this half's columns of the thread's row to shared memory, and on to dw while the next tap's
      // are read
#pragma unroll 1
      for (int t = 0; t < NT; ++t) {
        float v[HALF];
        if constexpr (HALF == 64) {
          umma::tmem_ld64(cols + t * BN, v);
        } else {
          umma::tmem_ld32(cols + t * BN, v);
        }
        if (t == NT - 1) {
          umma::fence_before_sync();
          __syncwarp();
          if (lane == 0) umma::mbar_arrive(drained);
        }
        if (inside) {
          float* dst = a.dw + (static_cast<size_t>(n) * a.taps + t) * a.Cin + cc;
          if (a.bulk) {
            umma::bulk_wait_read<0>();  // the row's previous reduction has read it
            float4* to = reinterpret_cast<float4*>(row);
#pragma unroll
            for (int k = 0; k < HALF / 4; ++k) to[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            umma::fence_async_smem();  // this thread's values, read by its own reduction
            umma::bulk_reduce_add_f32(dst, to, 4 * min(HALF, a.Cin - cc));
            umma::bulk_commit();
          } else {
            const int nv = min(HALF, a.Cin - cc);
#pragma unroll
            for (int j = 0; j < HALF; ++j)
              if (j < nv) atomicAdd(dst + j, v[j]);
          }
        }
        __syncwarp();  // channels past Cout rejoin: the next tcgen05.ld is .sync.aligned
      }
    }
    if (bias && !half) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        sum[k] += __shfl_xor_sync(0xFFFFFFFFu, sum[k], 16);
        if (lane < 16) bias_part[(e >> 5) * 128 + 8 * unit + k] = sum[k];
      }
      __syncwarp();
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the four warps that add up
      if (ok && n0 + e < a.Cout)
        atomicAdd(a.db + n0 + e, (bias_part[e] + bias_part[128 + e]) + (bias_part[256 + e] + bias_part[384 + e]));
    }
    umma::bulk_wait_all();
    __syncwarp();
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, TCOLS);
  }
}

// ---------------------------------------------------------------------------------------
// Memory-bound steps (channels-last BF16 unless noted)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float ldbf(const bf16* p) { return __bfloat162float(*p); }

// y[b, l, c] = (x[b, 2l, c] + x[b, 2l + 1, c]) / 2, l < Lout
__global__ void pool2_kernel(const bf16* x, int B, int Lout, int C, bf16* y) {
  const size_t n = static_cast<size_t>(B) * Lout * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    const size_t bl = i / C;
    const int l = bl % Lout;
    const int b = bl / Lout;
    const size_t src = (static_cast<size_t>(b) * 2 * Lout + 2 * l) * C + c;
    y[i] = __float2bfloat16(0.5f * (ldbf(x + src) + ldbf(x + src + C)));
  }
}

// dz[b, l, c] = (dpool[b, l/2, c] / 2 + dcat[b, l, cat_off + c]) * silu'(z[b, l, c]) over l < L
// (dpool may be null when L is odd at its end, dcat may be null)
__global__ void skip_grad_kernel(const bf16* dpool, int Lp, const bf16* dcat, int cat_stride, int cat_off,
                                 const bf16* z, int B, int L, int C, bf16* dz) {
  const size_t n = static_cast<size_t>(B) * L * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    const size_t bl = i / C;
    const int l = bl % L;
    const int b = bl / L;
    float g = 0.0f;
    if (dpool && l / 2 < Lp) g += 0.5f * ldbf(dpool + (static_cast<size_t>(b) * Lp + l / 2) * C + c);
    if (dcat) g += ldbf(dcat + bl * cat_stride + cat_off + c);
    dz[i] = __float2bfloat16(g * dsilu(ldbf(z + i)));
  }
}

// out[b, l, :] = [x[b, l/2, 0:C1], skip[b, l, 0:C2]]
__global__ void upcat_kernel(const bf16* x, const bf16* skip, int B, int L, int C1, int C2, bf16* out) {
  const int C = C1 + C2;
  const size_t n = static_cast<size_t>(B) * L * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    const size_t bl = i / C;
    const int l = bl % L;
    const int b = bl / L;
    out[i] = c < C1 ? x[(static_cast<size_t>(b) * (L / 2) + l / 2) * C1 + c] : skip[bl * C2 + (c - C1)];
  }
}

// dz[b, l', c] = (dcat[b, 2l', c] + dcat[b, 2l' + 1, c]) * silu'(z[b, l', c]), c < C1
__global__ void upcat_bwd_kernel(const bf16* dcat, const bf16* z, int B, int Lh, int C1, int C, bf16* dz) {
  const size_t n = static_cast<size_t>(B) * Lh * C1;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C1;
    const size_t bl = i / C1;
    const int l = bl % Lh;
    const int b = bl / Lh;
    const size_t r = static_cast<size_t>(b) * 2 * Lh + 2 * l;
    const float g = ldbf(dcat + r * C + c) + ldbf(dcat + (r + 1) * C + c);
    dz[i] = __float2bfloat16(g * dsilu(ldbf(z + i)));
  }
}

// ---- the same steps eight channels (16 bytes) per thread, for channel counts, strides and
// offsets that are multiples of 8 and 16-byte aligned buffers (every shape of the network)
__device__ __forceinline__ void ld8(const bf16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[k]);
    f[2 * k] = __low2float(h);
    f[2 * k + 1] = __high2float(h);
  }
}
__device__ __forceinline__ void st8(bf16* p, const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    w[k] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void pool2_v8_kernel(const bf16* x, int B, int Lout, int C, bf16* y) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const int C8 = C / 8;
  const size_t n = static_cast<size_t>(B) * Lout * C8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % C8) * 8;
    const size_t bl = i / C8;  // b * Lout + l
    const size_t src = 2 * bl * C + c;  // row 2l of sequence b: (b * 2 Lout + 2 l) * C
    float a[8], b[8];
    ld8(x + src, a);
    ld8(x + src + C, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = 0.5f * (a[k] + b[k]);
    st8(y + bl * C + c, a);
  }
}

__global__ void skip_grad_v8_kernel(const bf16* dpool, int Lp, const bf16* dcat, int cat_stride, int cat_off,
                                    const bf16* z, int B, int L, int C, bf16* dz) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const int C8 = C / 8;
  const size_t n = static_cast<size_t>(B) * L * C8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % C8) * 8;
    const size_t bl = i / C8;
    const int l = bl % L;
    const int b = bl / L;
    float g[8] = {0, 0, 0, 0, 0, 0, 0, 0}, t[8];
    if (dpool && l / 2 < Lp) {
      ld8(dpool + (static_cast<size_t>(b) * Lp + l / 2) * C + c, t);
#pragma unroll
      for (int k = 0; k < 8; ++k) g[k] += 0.5f * t[k];
    }
    if (dcat) {
      ld8(dcat + bl * cat_stride + cat_off + c, t);
#pragma unroll
      for (int k = 0; k < 8; ++k) g[k] += t[k];
    }
    ld8(z + bl * C + c, t);
#pragma unroll
    for (int k = 0; k < 8; ++k) g[k] *= dsilu(t[k]);
    st8(dz + bl * C + c, g);
  }
}

__global__ void upcat_v8_kernel(const bf16* x, const bf16* skip, int B, int L, int C1, int C2, bf16* out) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const int C = C1 + C2, C8 = C / 8;
  const size_t n = static_cast<size_t>(B) * L * C8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % C8) * 8;
    const size_t bl = i / C8;
    const int l = bl % L;
    const int b = bl / L;
    const bf16* src = c < C1 ? x + (static_cast<size_t>(b) * (L / 2) + l / 2) * C1 + c : skip + bl * C2 + (c - C1);
    *reinterpret_cast<uint4*>(out + bl * C + c) = *reinterpret_cast<const uint4*>(src);
  }
}

__global__ void upcat_bwd_v8_kernel(const bf16* dcat, const bf16* z, int B, int Lh, int C1, int C, bf16* dz) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const int C8 = C1 / 8;
  const size_t n = static_cast<size_t>(B) * Lh * C8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % C8) * 8;
    const size_t bl = i / C8;  // b * Lh + l
    const size_t r = 2 * bl;   // row 2l of sequence b in dcat
    float a[8], b[8], t[8];
    ld8(dcat + r * C + c, a);
    ld8(dcat + (r + 1) * C + c, b);
    ld8(z + bl * C1 + c, t);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = (a[k] + b[k]) * dsilu(t[k]);
    st8(dz + bl * C1 + c, a);
  }
}

// db[c] += sum over rows of dz[r * stride + c], c < C; one block column of 32 channels per block
__global__ void bias_grad_kernel(const bf16* dz, size_t rows, int C, int stride, float* db) {
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.0f;
  if (c < C) {
    for (size_t r = blockIdx.y * (size_t)blockDim.y + threadIdx.y; r < rows; r += (size_t)gridDim.y * blockDim.y)
      s += ldbf(dz + r * stride + c);
  }
  __shared__ float red[8][33];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    for (int k = 1; k < blockDim.y; ++k) s += red[k][threadIdx.x];
    atomicAdd(db + c, s);
  }
}

// Two floats in a register pair and the packed operations on them: each half rounds as the scalar operation does,
// at half the instructions.
struct F2 {
  unsigned long long v = 0;
};
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_get(F2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v));
  return a;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  asm("sub.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v));
  return a;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v));
  return a;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c.v) : "l"(a.v), "l"(b.v));
  return c;
}
__device__ __forceinline__ F2 operator-(F2 a) {
  a.v ^= 0x8000000080000000ull;
  return a;
}
// Two running sums side by side, each as a sum h, the rounding errors l of its additions and the products' low parts,
// and l's own rounding errors m: without m the sums of squares of a map of 2.4 M values were 1e-15 to
// 2e-15 off, FP64 sums 1e-16 to 1e-15.
struct PairSum2 {
  F2 h, l, m;
  __device__ __forceinline__ F2 high(F2 x) {
    const F2 t = h + x, z = t - h, e = (h - (t - z)) + (x - z);
    h = t;
    return e;
  }
  __device__ __forceinline__ void low(F2 x) {
    const F2 t = l + x, z = t - l;
    m = m + ((l - (t - z)) + (x - z));
    l = t;
  }
  __device__ __forceinline__ void add(F2 x) { l = l + high(x); }
  __device__ __forceinline__ void add(F2 x, F2 rest) {
    l = l + high(x);
    m = m + rest;
  }
  __device__ __forceinline__ void add_product(F2 a, F2 b) {
    const F2 p = a * b;
    low(high(p));
    low(f2_fma(a, b, -p));
  }
  // (a + al)^2 and (a + al) (b + bl).  The products of the low parts are below half a unit of everything in l and
  // would round away there, al^2 always downwards: they go to m.
  __device__ __forceinline__ void add_square(F2 a, F2 al) {
    const F2 p = a * a;
    low(high(p));
    low(f2_fma(a + a, al, f2_fma(a, a, -p)));
    m = f2_fma(al, al, m);
  }
  __device__ __forceinline__ void add_product(F2 a, F2 al, F2 b, F2 bl) {
    const F2 p = a * b;
    low(high(p));
    low(f2_fma(al, b, f2_fma(a, bl, f2_fma(a, b, -p))));
    m = f2_fma(al, bl, m);
  }
  __device__ __forceinline__ double value() const {
    float x, y, u, w, c, d;
    f2_get(h, x, y);
    f2_get(l, u, w);
    f2_get(m, c, d);
    const float t = __fadd_rn(x, y), z = __fsub_rn(t, x);
    const float r = __fadd_rn(__fsub_rn(x, __fsub_rn(t, z)), __fsub_rn(y, z));
    return static_cast<double>(t) + ((static_cast<double>(u) + static_cast<double>(w)) +
                                     (static_cast<double>(r) + static_cast<double>(__fadd_rn(c, d))));
  }
};
__device__ __forceinline__ void exact_difference(F2 a, F2 b, F2& h, F2& l) {
  h = a - b;
  const F2 z = h - a;
  l = (a - (h - z)) - (b + z);
}

// The same eight channels (16 bytes) per thread: a block covers 64 channels and 32 rows at a time.  Reads at
// the memory's rate (the scalar form above took 1.0 of a batch-16 gradient's 4.9 ms of kernel time).
__global__ void __launch_bounds__(256) bias_grad_v8_kernel(const bf16* __restrict__ dz, size_t rows, int C,
                                                           int stride, float* db) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const int g = threadIdx.x & 7, y = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + g * 8;
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < C) {
    const size_t step = static_cast<size_t>(gridDim.y) * 32;
    size_t r = static_cast<size_t>(blockIdx.y) * 32 + y;
    for (; r + 3 * step < rows; r += 4 * step) {
      float t[4][8];
#pragma unroll
      for (int k = 0; k < 4; ++k) ld8(dz + (r + k * step) * stride + c, t[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += t[k][e];
    }
    for (; r < rows; r += step) {
      float t[8];
      ld8(dz + r * stride + c, t);
#pragma unroll
      for (int e = 0; e < 8; ++e) s[e] += t[e];
    }
  }
  __shared__ float red[32][65];
#pragma unroll
  for (int e = 0; e < 8; ++e) red[y][g * 8 + e] = s[e];
  __syncthreads();
  if (threadIdx.x < 64 && static_cast<int>(blockIdx.x * 64 + threadIdx.x) < C) {
    float sum = 0.0f;
    for (int k = 0; k < 32; ++k) sum += red[k][threadIdx.x];
    atomicAdd(db + blockIdx.x * 64 + threadIdx.x, sum);
  }
}

// Mean-squared error over n_valid channels of each row: loss += sum (p - t)^2 (FP64 per block),
// dp[r, c] = scale * (p - t) for c < n_valid and 0 for the padded channels up to dstride.
__global__ void mse_kernel(const float* pred, int pstride, const float* target, int tstride, size_t rows, int n_valid,
                           bf16* dp, int dstride, float scale, double* loss) {
  double acc = 0.0;
  const size_t n = rows * static_cast<size_t>(dstride);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % dstride;
    const size_t r = i / dstride;
    float g = 0.0f;
    if (c < n_valid) {
      const float d = pred[r * pstride + c] - target[r * tstride + c];
      acc += static_cast<double>(d) * d;
      g = scale * d;
    }
    if (dp) dp[i] = __float2bfloat16(g);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double red[32];
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) s += red[w];
    atomicAdd(loss, s);
  }
}

// Four channels per thread (counts and strides multiples of 4, aligned buffers), the squares summed as floats with
// their errors (PairSum2) per 64 values and then in FP64.  Sums of 64 squares are 5e-17 off (a loop in FP64
// 3e-16); a single low part, without the errors of its own sums, left 1.4e-14, of which 1.2e-15 had one
// sign and stayed in the total.  32 registers, so that the eight blocks per SM of the grid are there at once: 65 us for
// 16 maps (81 with the 40 that the compiler takes, 60 with the single low part; the memory needs 60).  I:
// 32-bit indexes where they reach.
template <typename I>
__global__ void __launch_bounds__(256, 8) mse_v4_kernel(const float* __restrict__ pred, int pstride,
                                                     const float* __restrict__ target, int tstride, size_t rows,
                                                     int n_valid, bf16* dp, int dstride, float scale, double* loss) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const I q = dstride / 4;  // groups of four channels per row
  const I n = static_cast<I>(rows) * q, step = static_cast<I>(gridDim.x) * blockDim.x;
  double acc = 0.0;
  I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x;
  while (i < n) {
    PairSum2 t;
    uint32_t mx = 0;
    const I first = i;
    for (int k = 0; k < 16 && i < n; ++k, i += step) {
      const I row = i / q;
      const int c = static_cast<int>(i - row * q) * 4;
      const size_t r = row;
      float d[4] = {0, 0, 0, 0};
      if (c < n_valid) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(pred + r * pstride + c));
        const float4 b = __ldg(reinterpret_cast<const float4*>(target + r * tstride + c));
        d[0] = a.x - b.x, d[1] = a.y - b.y, d[2] = a.z - b.z, d[3] = a.w - b.w;
#pragma unroll
        for (int e = 0; e < 4; ++e) mx = max(mx, __float_as_uint(fabsf(d[e])));
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const F2 d2 = f2(d[e], d[e + 1]);
          t.add_product(d2, d2);
        }
      }
      if (dp)
        *reinterpret_cast<uint2*>(dp + r * dstride + c) =
            make_uint2(pack_bf16x2(scale * d[0], scale * d[1]), pack_bf16x2(scale * d[2], scale * d[3]));
    }
    if (mx < 0x58800000u && (mx >= 0x30800000u || mx == 0)) {
      acc += t.value();
    } else {  // out of the pairs' range (see map_sums_pair_kernel): FP64
      I j = first;
      for (int k = 0; k < 16 && j < n; ++k, j += step) {
        const I row = j / q;
        const int c = static_cast<int>(j - row * q) * 4;
        const size_t r = row;
        for (int e = 0; e < 4 && c < n_valid; ++e) {
          const float x = pred[r * pstride + c + e] - target[r * tstride + c + e];
          acc += static_cast<double>(x) * x;
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double red[8];
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[w];
    atomicAdd(loss, s);
  }
}

// Adam with decoupled weight decay on FP32 masters; also writes the BF16 copy the MMAs read.
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, size_t n, float lr, float b1, float b2,
                            float eps, float wd, float bc1, float bc2, float gscale, bf16* p_bf16) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i] * gscale;
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float pi = p[i] * (1.0f - lr * wd);
    pi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p[i] = pi;
    if (p_bf16) p_bf16[i] = __float2bfloat16(pi);
  }
}

// Four parameters per thread and access (n a multiple of 4, 16-byte aligned buffers).
__global__ void __launch_bounds__(256) adam_v4_kernel(float4* p, const float4* g, float4* m, float4* v, size_t n4,
                                                      float lr, float b1, float b2, float eps, float wd, float bc1,
                                                      float bc2, float gscale, uint2* p_bf16) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    float4 p4 = p[i], m4 = m[i], v4 = v[i];
    const float4 g4 = g[i];
    const float* ge = &g4.x;
    float *pe = &p4.x, *me = &m4.x, *ve = &v4.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gi = ge[k] * gscale;
      const float mi = b1 * me[k] + (1.0f - b1) * gi;
      const float vi = b2 * ve[k] + (1.0f - b2) * gi * gi;
      me[k] = mi;
      ve[k] = vi;
      float pi = pe[k] * (1.0f - lr * wd);
      pi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
      pe[k] = pi;
    }
    m[i] = m4;
    v[i] = v4;
    p[i] = p4;
    if (p_bf16) p_bf16[i] = make_uint2(pack_bf16x2(p4.x, p4.y), pack_bf16x2(p4.z, p4.w));
  }
}

// wt[c][t'][n] = w[n][taps - 1 - t'][c]: the data gradient's weights (transposed, taps reversed)
__global__ void weight_transpose_kernel(const bf16* w, int N, int taps, int C, bf16* wt) {
  const size_t n = static_cast<size_t>(N) * taps * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int o = i % N;
    const size_t ct = i / N;
    const int t = ct % taps;
    const int c = ct / taps;
    wt[i] = w[(static_cast<size_t>(o) * taps + (taps - 1 - t)) * C + c];
  }
}

// The same for a list of convolutions in one launch (the data gradients' weights of a whole network after an
// optimiser step): 64 x 64 (output channel, input channel) blocks of one tap through shared memory, so that
// both sides move 128-byte rows.  Channel counts must be multiples of 8 and buffers 16-byte aligned.
struct TransposeList {
  int count;
  int first[MSUR_MAX_TRANSPOSES + 1];  // first block of each convolution
  const bf16* w[MSUR_MAX_TRANSPOSES];
  bf16* wt[MSUR_MAX_TRANSPOSES];
  int N[MSUR_MAX_TRANSPOSES], taps[MSUR_MAX_TRANSPOSES], C[MSUR_MAX_TRANSPOSES];
};
__global__ void __launch_bounds__(256) weight_transpose_list_kernel(const __grid_constant__ TransposeList a) {
  int k = 0;
  while (k + 1 < a.count && static_cast<int>(blockIdx.x) >= a.first[k + 1]) ++k;
  const int N = a.N[k], T = a.taps[k], C = a.C[k];
  const int nn = (N + 63) / 64, nc = (C + 63) / 64;
  int blk = blockIdx.x - a.first[k];
  const int c0 = (blk % nc) * 64;
  blk /= nc;
  const int n0 = (blk % nn) * 64, t = blk / nn;
  __shared__ bf16 tile[64][66];
  const int g = threadIdx.x & 7, y = threadIdx.x >> 3;  // 8 channels of one row, 32 rows at a time
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int n = n0 + y + 32 * h, c = c0 + 8 * g;
    if (n < N && c < C) {
      const uint4 u = *reinterpret_cast<const uint4*>(a.w[k] + (static_cast<size_t>(n) * T + (T - 1 - t)) * C + c);
      const bf16* e = reinterpret_cast<const bf16*>(&u);
#pragma unroll
      for (int q = 0; q < 8; ++q) tile[8 * g + q][y + 32 * h] = e[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = c0 + y + 32 * h, n = n0 + 8 * g;
    if (c < C && n < N) {
      uint4 u;
      bf16* e = reinterpret_cast<bf16*>(&u);
#pragma unroll
      for (int q = 0; q < 8; ++q) e[q] = tile[y + 32 * h][8 * g + q];
      *reinterpret_cast<uint4*>(a.wt[k] + (static_cast<size_t>(c) * T + t) * N + n) = u;
    }
  }
}

// x[b, l, 0:4] = track[b][0:4][l], x[b, l, 4:8] = params[b][0:4], x[b, l, 8:C] = 0
__global__ void assemble_input_kernel(const float* track, const float* params, int B, int L, int C, bf16* x) {
  const size_t n = static_cast<size_t>(B) * L * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    const size_t bl = i / C;
    const int l = bl % L;
    const int b = bl / L;
    float v = 0.0f;
    if (c < 4) v = track[(static_cast<size_t>(b) * 4 + c) * L + l];
    else if (c < 8) v = params[b * 4 + (c - 4)];
    x[i] = __float2bfloat16(v);
  }
}

// Eight channels (16 bytes) per thread: only the first group of a row reads anything.  I: 32-bit indexes where
// they reach (a 64-bit division per 16 bytes costs more than the store).
template <typename I>
__global__ void __launch_bounds__(256) assemble_input_v8_kernel(const float* track, const float* params, int B, int L,
                                                                int C, uint4* x) {
  umma::pdl_wait();
  umma::pdl_trigger();
  const I C8 = C / 8, n = static_cast<I>(B) * L * C8;
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < n; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const I bl = i / C8;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (i - bl * C8 == 0) {
      const I b = bl / L, l = bl - b * L;
      const size_t S = L;  // a channel's stride: three of them may be past 2^31
      const float* t = track + static_cast<size_t>(b) * 4 * S + l;
      const float4 q = make_float4(params[b * 4], params[b * 4 + 1], params[b * 4 + 2], params[b * 4 + 3]);
      u = make_uint4(pack_bf16x2(t[0], t[S]), pack_bf16x2(t[2 * S], t[3 * S]), pack_bf16x2(q.x, q.y), pack_bf16x2(q.z, q.w));
    }
    x[i] = u;
  }
}

// Training target of a summed band (column-major u32, ncols x nrows): per bin j (a column of
// the band, its nrows diagonals) T[j, d] = log1p(band[j, d] * nrows / sum_d band[j, d]), 0 for
// an empty bin.  One warp per bin.
__global__ void band_target_kernel(const uint32_t* band, size_t ncols, int nrows, float* out) {
  const size_t warps = (static_cast<size_t>(gridDim.x) * blockDim.x) / 32;
  for (size_t j = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32; j < ncols; j += warps) {
    const uint32_t* col = band + j * nrows;
    unsigned long long s = 0;
    for (int d = threadIdx.x % 32; d < nrows; d += 32) s += col[d];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double scale = s ? static_cast<double>(nrows) / static_cast<double>(s) : 0.0;
    for (int d = threadIdx.x % 32; d < nrows; d += 32)
      out[j * nrows + d] = static_cast<float>(log1p(static_cast<double>(col[d]) * scale));
  }
}

// Per map m (n values each): sums for Pearson r and relative L2 of pred against ref, in FP64:
// out[m] = {sum p', sum r', sum p'^2, sum r'^2, sum p' r', sum (p - r)^2} with p' = p - mean_p,
// r' = r - mean_r when means (2 per map) are given, the raw values otherwise: the two passes of
// the reference's Pearson (mean, then covariances of the deviations).
//
// FP64's accuracy at the FP32 pipes' rate (FP64 runs at 1/64 of it on sm_103a: 11 FP64 operations per
// element took 1.7 ms for 32 maps of 2.4 M values, of which the memory needs 0.1).  Each thread sums chunks of 128
// elements in two pairs of floats: differences, products and sums with their exact rounding errors (Knuth's
// two-sum, two-product by FMA), and adds each chunk's pair to FP64 totals.  The means are split into a float
// m and a remainder d: the deviations from m are exact pairs, and d enters the FP64 totals,
// sum (a - d)^2 = sum a^2 - 2 d sum a + n d^2.  Low parts are summed with their own rounding errors and the
// products of two low parts apart from the rest, so that nothing an element loses adds up: emulated against exact
// sums for maps of 2.4 M values, the threads' sums are 1e-17 to 3e-17 off (FP64 sums 5e-17 to 7e-17), r 3e-16 (5e-16)
// and the relative L2 3e-16 (7e-16); most of both is the blocks' FP64 additions.
// A chunk with values outside [2^-30, 2^50) in size throughout, infinities or NaN is summed in FP64.
// WHICH: the sums wanted (bit k: sum k); MEANS: deviations from the means, raw values otherwise.
// The sums come two to a packed operation (PairSum2), and two loads of each side run ahead (more, or three blocks
// per SM, spill): 0.62 ms for the scores of those maps, 3.4 in FP64.  With single low parts it took 0.47, but was
// up to 9e-15 off.
constexpr int SUM_VECS = 32;  // float4 per thread and chunk
template <bool VEC, bool MEANS, unsigned WHICH>
__global__ void __launch_bounds__(256, 2) map_sums_pair_kernel(const float* pred, size_t pstride_map, const float* ref,
                                                            size_t rstride_map, size_t n, const double* means,
                                                            double* out) {
  const int m = blockIdx.y;
  const float* __restrict__ p = pred + m * pstride_map;
  const float* __restrict__ r = ref + m * rstride_map;
  const double mp = MEANS ? means[2 * m] : 0.0, mr = MEANS ? means[2 * m + 1] : 0.0;
  const float fp = static_cast<float>(mp), fr = static_cast<float>(mr);
  const double dp = mp - fp, dr = mr - fr;
  double s[6] = {0, 0, 0, 0, 0, 0};
  const size_t span = static_cast<size_t>(SUM_VECS) * 256 * 4;  // elements of a block's step
  const uint32_t LO = 0x30800000u, HI = 0x58800000u;           // 2^-30, 2^50
  auto load2 = [&](float4& x, float4& y, size_t i) {
    if (i < n) {
      x = __ldg(reinterpret_cast<const float4*>(p + i));
      y = __ldg(reinterpret_cast<const float4*>(r + i));
    }
  };
  const bool means_ok = __float_as_uint(fabsf(fp)) < HI && __float_as_uint(fabsf(fr)) < HI;
  for (size_t base = blockIdx.x * span; base < n; base += gridDim.x * span) {
    PairSum2 t[6];
    uint32_t mxp = 0, mxr = 0;
    int k = 0;
    const F2 fp2 = f2(fp, fp), fr2 = f2(fr, fr);
    // two loads of each side in flight while the ones before them are summed
    float4 qp[2], qr[2];
    const size_t first = base + threadIdx.x * 4;
    if constexpr (VEC) {
#pragma unroll
      for (int u = 0; u < 2; ++u) load2(qp[u], qr[u], first + u * 1024);
    }
#pragma unroll 2
    for (int v = 0; v < SUM_VECS; ++v) {
      const size_t i = first + static_cast<size_t>(v) * 1024;
      if (i >= n) break;
      float a[4], b[4];
      int valid = 4;
      if constexpr (VEC) {
        const float4 pa = qp[v & 1], rb = qr[v & 1];
        a[0] = pa.x, a[1] = pa.y, a[2] = pa.z, a[3] = pa.w;
        b[0] = rb.x, b[1] = rb.y, b[2] = rb.z, b[3] = rb.w;
        if (v + 2 < SUM_VECS) load2(qp[v & 1], qr[v & 1], i + 2048);
      } else {
        valid = static_cast<int>(n - i < 4 ? n - i : 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          a[e] = e < valid ? p[i + e] : fp;  // no deviation
          b[e] = e < valid ? r[i + e] : fr;
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        mxp = max(mxp, __float_as_uint(fabsf(a[e])));
        mxr = max(mxr, __float_as_uint(fabsf(b[e])));
      }
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const F2 a2 = f2(a[e], a[e + 1]), b2 = f2(b[e], b[e + 1]);
        if constexpr (MEANS) {
          F2 ah, al, bh, bl;
          exact_difference(a2, fp2, ah, al);
          exact_difference(b2, fr2, bh, bl);
          if constexpr (WHICH & 1) t[0].add(ah, al);
          if constexpr (WHICH & 2) t[1].add(bh, bl);
          if constexpr (WHICH & 4) t[2].add_square(ah, al);
          if constexpr (WHICH & 8) t[3].add_square(bh, bl);
          if constexpr (WHICH & 16) t[4].add_product(ah, al, bh, bl);
        } else {
          if constexpr (WHICH & 1) t[0].add(a2);
          if constexpr (WHICH & 2) t[1].add(b2);
          if constexpr (WHICH & 4) t[2].add_product(a2, a2);
          if constexpr (WHICH & 8) t[3].add_product(b2, b2);
          if constexpr (WHICH & 16) t[4].add_product(a2, b2);
        }
        if constexpr (WHICH & 32) {
          F2 h, l;
          if (VEC || e + 1 < valid) {
            exact_difference(a2, b2, h, l);
          } else {
            exact_difference(f2(e < valid ? a[e] : 0.0f, 0.0f), f2(e < valid ? b[e] : 0.0f, 0.0f), h, l);
          }
          t[5].add_square(h, l);
        }
      }
      k += valid;
    }
    const bool plain = means_ok && mxp < HI && mxr < HI && (mxp >= LO || (mxp == 0 && fp == 0.0f)) &&
                       (mxr >= LO || (mxr == 0 && fr == 0.0f));
    if (plain) {
      const double sa = t[0].value(), sb = t[1].value(), c = k;
      s[0] += sa - c * dp;
      s[1] += sb - c * dr;
      s[2] += t[2].value() - 2.0 * dp * sa + c * dp * dp;
      s[3] += t[3].value() - 2.0 * dr * sb + c * dr * dr;
      s[4] += t[4].value() - dr * sa - dp * sb + c * dp * dr;
      s[5] += t[5].value();
    } else if (k > 0) {  // nothing of fp, fr, dp, dr, which are infinite or NaN for means outside float's range
      for (int v = 0; v < SUM_VECS; ++v) {
        for (int e = 0; e < 4; ++e) {
          const size_t i = base + (static_cast<size_t>(v) * 256 + threadIdx.x) * 4 + e;
          if (i >= n) break;
          const double a = p[i] - mp, b = r[i] - mr, d = static_cast<double>(p[i]) - r[i];
          s[0] += a;
          s[1] += b;
          s[2] += a * a;
          s[3] += b * b;
          s[4] += a * b;
          s[5] += d * d;
        }
      }
    }
  }
  __shared__ double red[6][8];
  for (int k = 0; k < 6; ++k) {
    double x = s[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (threadIdx.x % 32 == 0) red[k][threadIdx.x / 32] = x;
  }
  __syncthreads();
  if (threadIdx.x < 6 && ((WHICH >> threadIdx.x) & 1u)) {
    double x = 0;
    for (int w = 0; w < 8; ++w) x += red[threadIdx.x][w];
    atomicAdd(out + 6 * m + threadIdx.x, x);
  }
}

// Gather the first n_valid channels of rows with stride `stride` into a dense [rows][n_valid] FP32
// array (the head's padded output to the band layout), optionally in place-compatible.
__global__ void compact_rows_kernel(const float* in, int stride, size_t rows, int n_valid, float* out) {
  const size_t n = rows * static_cast<size_t>(n_valid);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = in[(i / n_valid) * stride + i % n_valid];
}

}  // namespace sg

// =========================================================================================
// Host side
// =========================================================================================
using namespace sg;

namespace {

thread_local char g_err[512];
std::mutex g_mu;
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
unsigned* g_dev_err[64] = {};
// pipeline depth of the forward/data-gradient convolution per N tile width (64, 128, 256): with one CTA
// per tile its stages (fewer let more CTAs share an SM, so one tile's epilogue overlaps another's main loop), in
// the persistent form where conv_plan starts
int g_conv_stages[3] = {4, 3, 4};
// kernel form per N tile width: bit 0 the persistent kernel (two to eight TMEM accumulators),
// bit 1 the staged epilogue (outputs through shared memory and TMA stores)
int g_conv_form[3] = {2, 2, 2};

int conv_slot(int bn) { return bn == 256 ? 2 : (bn == 128 ? 1 : 0); }

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_ok(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return MSUR_OK;
  return fail(MSUR_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int setup(unsigned** err) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_encode) {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
      return fail(MSUR_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  int dev = 0;
  int rc = cuda_ok(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return fail(MSUR_ERR_UNSUPPORTED, "device %d out of range", dev);
  if (!g_dev_err[dev]) {
    rc = cuda_ok(cudaMalloc(&g_dev_err[dev], sizeof(unsigned)), "cudaMalloc(error flag)");
    if (rc) return rc;
    rc = cuda_ok(cudaMemset(g_dev_err[dev], 0, sizeof(unsigned)), "cudaMemset(error flag)");
    if (rc) return rc;
  }
  *err = g_dev_err[dev];
  return MSUR_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// BF16 tensor map with 128-byte swizzling: dims[0] innermost.
int make_map(CUtensorMap* m, const void* base, int rank, const uint64_t* dims, const uint32_t* box) {
  cuuint64_t gd[3], gs[2];
  cuuint32_t bx[3], es[3] = {1, 1, 1};
  uint64_t stride = 2;
  for (int i = 0; i < rank; ++i) {
    gd[i] = dims[i];
    bx[i] = box[i];
    if (i > 0) gs[i - 1] = stride;
    stride *= dims[i];
  }
  const CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), gd, gs, bx, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MSUR_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
  return MSUR_OK;
}

// Output map of the staged epilogue: [B][L][n_valid] elements of elem_bytes with row stride
// out_stride, boxes of box_x columns x 32 rows, 128-byte swizzle.
int make_out_map(CUtensorMap* m, void* base, CUtensorMapDataType type, int elem_bytes, int n_valid, int out_stride,
                 int L, int B, int box_x, int box_rows = 32) {
  const cuuint64_t gd[3] = {static_cast<cuuint64_t>(n_valid), static_cast<cuuint64_t>(L), static_cast<cuuint64_t>(B)};
  const cuuint64_t gs[2] = {static_cast<cuuint64_t>(out_stride) * elem_bytes,
                            static_cast<cuuint64_t>(out_stride) * elem_bytes * L};
  const cuuint32_t bx[3] = {static_cast<cuuint32_t>(box_x), static_cast<cuuint32_t>(box_rows), 1}, es[3] = {1, 1, 1};
  const CUresult r = g_encode(m, type, 3, base, gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MSUR_ERR_CUDA, "cuTensorMapEncodeTiled (output) failed (%d)", static_cast<int>(r));
  return MSUR_OK;
}

// Map of the upsampled copy: output row l of sequence b at element ((b * 2L + 2l + parity) *
// row_stride) of base, n_valid columns, boxes of 64 BF16 columns x 32 rows.
int make_dup_map(CUtensorMap* m, void* base, int parity, int n_valid, int row_stride, int L, int B) {
  const cuuint64_t gd[3] = {static_cast<cuuint64_t>(n_valid), static_cast<cuuint64_t>(L), static_cast<cuuint64_t>(B)};
  const cuuint64_t gs[2] = {static_cast<cuuint64_t>(row_stride) * 2 * 2,
                            static_cast<cuuint64_t>(row_stride) * 2 * 2 * L};
  const cuuint32_t bx[3] = {64, 32, 1}, es[3] = {1, 1, 1};
  void* b0 = static_cast<char*>(base) + static_cast<size_t>(parity) * row_stride * 2;
  const CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, b0, gd, gs, bx, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MSUR_ERR_CUDA, "cuTensorMapEncodeTiled (upsampled) failed (%d)", static_cast<int>(r));
  return MSUR_OK;
}

// Dynamic shared memory of a forward kernel: operand stages, alignment slack, the barriers (a
// 1 KB block when the staged epilogue's buffers follow it).
template <int BN, int STAGES, bool STAGED>
constexpr int conv_smem() {
  return STAGES * (BM * BK * 2 + BN * BK * 2) + 1024 + (STAGED ? 1024 + STAGE_OUT_BYTES : 256);
}

// Launch as a programmatic dependent of the stream's previous kernel: set-up and launch latency overlap
// its tail (the 23 convolutions of one map: 277 to 227 us; gradients of 16 maps:
// 1.66 to 1.47 ms; a single convolution called again and again: 35.6 to 34.1 us).  Only kernels that begin with pdl_wait.
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, int threads, int smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// Once per kernel and device: the shared-memory permission (asking the runtime on every launch took
// longer than the launch).
struct KernelLimits {
  std::atomic<bool> set[64] = {};
  int get(const void* kern, int smem) {
    int dev = 0;
    int rc = cuda_ok(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return fail(MSUR_ERR_UNSUPPORTED, "device %d out of range", dev);
    if (set[dev].load(std::memory_order_acquire)) return MSUR_OK;
    rc = cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "smem attribute");
    if (!rc) set[dev].store(true, std::memory_order_release);
    return rc;
  }
};

template <int BN, int STAGES, bool STAGED>
int launch_conv(const ConvArgs& a, int ntiles_n, cudaStream_t st) {
  constexpr int smem = conv_smem<BN, STAGES, STAGED>();
  auto kern = conv_fwd_kernel<BN, STAGES, STAGED>;
  static KernelLimits limits;
  const int rc = limits.get(reinterpret_cast<const void*>(kern), smem);
  if (rc) return rc;
  dim3 grid(ntiles_n, (a.L + BM - 1) / BM, a.B);
  return cuda_ok(launch_pdl(kern, grid, THREADS, smem, st, a),
                 "conv_fwd_kernel launch");
}

int sm_count(int* out) {
  static std::atomic<int> count[64] = {};
  int dev = 0;
  int rc = cuda_ok(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return fail(MSUR_ERR_UNSUPPORTED, "device %d out of range", dev);
  int n = count[dev].load(std::memory_order_relaxed);
  if (!n) {
    rc = cuda_ok(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "SM count");
    if (rc) return rc;
    count[dev].store(n, std::memory_order_relaxed);
  }
  *out = n;
  return MSUR_OK;
}

// How the persistent kernel uses its shared memory (ConvPlan), in this order of preference:
//  1. more than one tap, and all weights of an N tile fit beside the slots of one or two tiles: weights stay;
//  2. more than one tap, and the slots fit beside at least three weight stages;
//  3. both operands stage by stage (a single tap reads its activations once anyway: the head's convolution of
//     256 maps took 508 us with slots, 465 without).
// A single tile's slots do when its chunks, freed one by one in its last tap, leave the next tile's first loads
// four K steps or more ahead (192 to 64 channels at 4000 positions, 256 maps: 128 us with one
// tile's three slots, 92 with six).  Epilogue groups: as many as fit up to four, two without an activation.
ConvPlan conv_plan(int bn, int cin, int taps, int cout, int L, int B, int stages, bool staged, bool heavy, int sms,
                   int* grid, int* smem) {
  constexpr int ROOM = 227 * 1024 - 2048;  // alignment slack and the barriers
  const int kc = cin / BK, nk = taps * kc, w = bn * BK * 2;
  const int group = staged ? 4 * 4096 : 0, most = heavy ? 4 : 2;
  ConvPlan p{};
  p.ntn = (cout + bn - 1) / bn;
  p.ntl = (L + BM - 1) / BM;
  p.ntiles = p.ntn * p.ntl * B;
  *grid = std::min(p.ntiles, sms);
  const int fixed = sms / p.ntn * p.ntn;  // a grid whose stride keeps a CTA's N tile
  const int least = kc >= 4 ? kc : 2 * kc;
  const bool slots = taps > 1 && taps - 1 <= 8 && least <= MAX_SLOTS;
  int used = 0;
  if (slots && nk <= MAX_STAGES && fixed > 0) {
    for (int g = most; g >= 2 && !p.groups; --g) {
      if (nk * w + least * SLOT_BYTES + g * group > ROOM) continue;
      p.groups = g;
      p.wres = 1;
      p.stages = nk;
      p.aslots = least;
      *grid = std::min(p.ntiles, fixed);
    }
  }
  for (int st = stages; slots && st >= std::min(3, stages) && !p.groups; --st) {
    for (int g = most; g >= 2 && !p.groups; --g) {
      if (st * w + least * SLOT_BYTES + g * group > ROOM) continue;
      p.groups = g;
      p.stages = st;
      p.aslots = least;
    }
  }
  for (int st = stages; st >= 2 && !p.groups; --st) {
    for (int g = most; g >= 2 && !p.groups; --g) {
      if (st * (w + BM * BK * 2) + g * group > ROOM) continue;
      p.groups = g;
      p.stages = st;
    }
  }
  used = p.stages * (w + (p.aslots ? 0 : BM * BK * 2)) + p.aslots * SLOT_BYTES + p.groups * group;
  if (p.aslots && p.aslots + kc <= MAX_SLOTS && used + kc * SLOT_BYTES <= ROOM) {
    p.aslots += kc;
    used += kc * SLOT_BYTES;
  }
  // with a tile or two per CTA the ring's depth is what hides a load (one map: 200 us with four stages, 186)
  const int stage = w + (p.aslots ? 0 : BM * BK * 2);
  while (!p.wres && p.stages < 8 && p.stages < nk && used + stage <= ROOM) ++p.stages, used += stage;
  p.bufs = staged ? 1 : 0;
  if (staged && used + p.groups * group <= ROOM) {
    p.bufs = 2;
    used += p.groups * group;
  }
  *smem = 2048 + used;
  return p;
}

template <int BN, bool STAGED>
int launch_conv_persistent(const ConvArgs& a, const ConvPlan& p, int grid, int smem, cudaStream_t st) {
  auto kern = conv_fwd_persistent_kernel<BN, STAGED>;
  static KernelLimits limits;
  const int rc = limits.get(reinterpret_cast<const void*>(kern), 227 * 1024);
  if (rc) return rc;
  return cuda_ok(launch_pdl(kern, dim3(grid), 128 + 128 * p.groups, smem, st, a, p), "conv_fwd_persistent_kernel launch");
}

int dispatch_conv_persistent(int bn, const ConvArgs& a, const ConvPlan& p, int grid, int smem, cudaStream_t st) {
  const bool staged = p.bufs > 0;
  switch (bn) {
    case 64:
      return staged ? launch_conv_persistent<64, true>(a, p, grid, smem, st)
                    : launch_conv_persistent<64, false>(a, p, grid, smem, st);
    case 128:
      return staged ? launch_conv_persistent<128, true>(a, p, grid, smem, st)
                    : launch_conv_persistent<128, false>(a, p, grid, smem, st);
    case 192:
      return staged ? launch_conv_persistent<192, true>(a, p, grid, smem, st)
                    : launch_conv_persistent<192, false>(a, p, grid, smem, st);
    default:
      return staged ? launch_conv_persistent<256, true>(a, p, grid, smem, st)
                    : launch_conv_persistent<256, false>(a, p, grid, smem, st);
  }
}

template <int BN>
int dispatch_conv(const ConvArgs& a, int ntn, bool staged, int stages, cudaStream_t st) {
  if (stages == 2) return staged ? launch_conv<BN, 2, true>(a, ntn, st) : launch_conv<BN, 2, false>(a, ntn, st);
  if (stages == 3) return staged ? launch_conv<BN, 3, true>(a, ntn, st) : launch_conv<BN, 3, false>(a, ntn, st);
  return staged ? launch_conv<BN, 4, true>(a, ntn, st) : launch_conv<BN, 4, false>(a, ntn, st);
}

template <int BN, int NT, int STAGES>
int launch_wgrad(const WgradArgs& a, int splits, cudaStream_t st) {
  constexpr int smem = STAGES * wgrad_stage_bytes<BN, NT>() + 256 * wgrad_row_bytes<BN>() + 1024 + 256 + 2048;  // alignment, barriers, bias sums
  auto kern = wgrad_kernel<BN, NT, STAGES>;
  static KernelLimits limits;
  const int rc = limits.get(reinterpret_cast<const void*>(kern), smem);
  if (rc) return rc;
  dim3 grid((a.Cin + BN - 1) / BN, (a.Cout + BM - 1) / BM, splits);
  return cuda_ok(launch_pdl(kern, grid, WTHREADS, smem, st, a), "wgrad_kernel launch");
}

// The current device's SMs, for grids that any number suits (a GB300's where the query fails: the launch then
// reports what is wrong).
unsigned sms() {
  int n = 0;
  return sm_count(&n) == MSUR_OK && n > 0 ? static_cast<unsigned>(n) : 152u;
}

unsigned grid_for(size_t n, unsigned block = 256) {
  const size_t g = (n + block - 1) / block, most = 32 * sms();
  return static_cast<unsigned>(g < most ? (g ? g : 1) : most);
}

}  // namespace

extern "C" {

const char* msur_last_error_string(void) { return g_err; }

int msur_take_error(unsigned* code) {
  unsigned* err = nullptr;
  int rc = setup(&err);
  if (rc) return rc;
  unsigned h = 0;
  rc = cuda_ok(cudaMemcpy(&h, err, sizeof(h), cudaMemcpyDeviceToHost), "read error flag");
  if (rc) return rc;
  if (h) rc = cuda_ok(cudaMemset(err, 0, sizeof(unsigned)), "clear error flag");
  if (code) *code = h;
  return rc;
}

static int conv_forward_impl(const void* x, int B, int L, int Cin, const void* w, int Cout, int taps,
                             const float* bias, int act, void* out_pre, void* out_post, float* out_f32,
                             int out_stride, int n_valid, const void* gate, void* out_skip, int skip_stride,
                             void* out_dup, int dup_stride, void* out_pool, int pool_stride, int form, int stages,
                             void* stream) {
  if (!x || !w || B <= 0 || L <= 0 || Cin <= 0 || Cout <= 0 || taps <= 0 || n_valid <= 0 || n_valid > Cout)
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: bad shape or null pointer");
  if (Cin % BK) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: Cin (%d) must be a multiple of 64", Cin);
  if (taps % 2 == 0) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: taps must be odd");
  if (!out_pre && !out_post && !out_f32 && !out_skip && !out_dup && !out_pool)
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: no output");
  if (out_pool && (L % 2)) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward_fused: pooling needs an even L");
  if ((out_skip && (skip_stride < n_valid || (skip_stride % 8) || !aligned16(out_skip))) ||
      (out_dup && (dup_stride < n_valid || (dup_stride % 8) || !aligned16(out_dup))) ||
      (out_pool && (pool_stride < n_valid || (pool_stride % 8) || !aligned16(out_pool))))
    return fail(MSUR_ERR_INVALID_ARG,
                "msur_conv_forward_fused: copies must be 16-byte aligned, their strides multiples of 8 and >= n_valid");
  const bool primary = out_pre || out_post || out_f32;
  if ((primary && (out_stride < n_valid || (out_stride % 8))) ||
      !aligned16(x) || !aligned16(w) || (out_pre && !aligned16(out_pre)) || (out_post && !aligned16(out_post)) ||
      (out_f32 && !aligned16(out_f32)) || (gate && !aligned16(gate)))
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: buffers must be 16-byte aligned, out_stride a multiple of 8");
  if (act != MSUR_ACT_NONE && act != MSUR_ACT_SILU) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_forward: bad act");
  unsigned* err = nullptr;
  int rc = setup(&err);
  if (rc) return rc;
  const int slot = conv_slot(Cout <= 64 ? 64 : (Cout % 256 == 0 ? 256 : 128));
  if (form < 0) form = g_conv_form[slot];
  if (stages < 0) stages = g_conv_stages[slot];
  // A tile is one CTA's chain of K steps, and a step's time is its operands' transfer, so while the tiles
  // leave SMs idle a narrower one halves the chain's time on twice the SMs (the products and their order
  // are the same).  One map: the deep levels have 2 to 16 tiles at 256 columns, 8 to 64 at 64.
  const bool persistent = (form & 1) != 0, staged = (form & 2) != 0;
  int nsm = 0;
  rc = sm_count(&nsm);
  if (rc) return rc;
  int BN = slot == 2 ? 256 : (slot == 1 ? 128 : 64);
  if (persistent && slot == 1 && Cout % 192 == 0) BN = 192;
  while (BN > 64 && static_cast<long long>((Cout + BN - 1) / BN) * ((L + BM - 1) / BM) * B < nsm)
    BN = BN == 192 ? 64 : BN / 2;
  ConvArgs a;
  std::memset(&a, 0, sizeof(a));
  const uint64_t dims_a[3] = {static_cast<uint64_t>(Cin), static_cast<uint64_t>(L), static_cast<uint64_t>(B)};
  ConvPlan plan{};
  int grid = 0, smem = 0;
  if (persistent)
    plan = conv_plan(BN, Cin, taps, Cout, L, B, stages, staged, act == MSUR_ACT_SILU || gate, nsm, &grid, &smem);
  const uint32_t box_a[3] = {64, static_cast<uint32_t>(plan.aslots ? BM + taps - 1 : BM), 1};
  rc = make_map(&a.tm_a, x, 3, dims_a, box_a);
  if (rc) return rc;
  const uint64_t dims_b[2] = {static_cast<uint64_t>(taps) * Cin, static_cast<uint64_t>(Cout)};
  const uint32_t box_b[2] = {64, static_cast<uint32_t>(BN)};
  rc = make_map(&a.tm_b, w, 2, dims_b, box_b);
  if (rc) return rc;
  a.B = B;
  a.L = L;
  a.Cin = Cin;
  a.taps = taps;
  a.pad = (taps - 1) / 2;
  a.n_valid = n_valid;
  a.out_stride = out_stride;
  a.act = act;
  a.bias = bias;
  a.gate = static_cast<const bf16*>(gate);
  a.out_pre = static_cast<bf16*>(out_pre);
  a.out_post = static_cast<bf16*>(out_post);
  a.out_f32 = out_f32;
  a.err = err;
  const int ntn = (Cout + BN - 1) / BN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // kernel form: bit 0 the persistent kernel, bit 1 the staged epilogue (outputs through shared
  // memory and TMA)
  if ((out_skip || out_dup || out_pool) && (!staged || gate))
    return fail(MSUR_ERR_UNSUPPORTED, "msur_conv_forward_fused: the fused copies need the staged form (bit 1) "
                                      "for N tile %d and no gate", BN);
  if (staged) {
    if (out_f32) rc = make_out_map(&a.tm_f32, out_f32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, n_valid, out_stride, L, B, 32);
    if (!rc && out_pre)
      rc = make_out_map(&a.tm_pre, out_pre, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, n_valid, out_stride, L, B, 64);
    if (!rc && out_post)
      rc = make_out_map(&a.tm_post, out_post, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, n_valid, out_stride, L, B, 64);
    if (!rc && out_skip)
      rc = make_out_map(&a.tm_skip, out_skip, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, n_valid, skip_stride, L, B, 64);
    if (!rc && out_dup) rc = make_dup_map(&a.tm_dup0, out_dup, 0, n_valid, dup_stride, L, B);
    if (!rc && out_dup) rc = make_dup_map(&a.tm_dup1, out_dup, 1, n_valid, dup_stride, L, B);
    if (!rc && out_pool)
      rc = make_out_map(&a.tm_pool, out_pool, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, n_valid, pool_stride, L / 2, B, 64,
                        16);
    if (rc) return rc;
    a.has_skip = out_skip ? 1 : 0;
    a.has_dup = out_dup ? 1 : 0;
    a.has_pool = out_pool ? 1 : 0;
  }
  if (persistent) return dispatch_conv_persistent(BN, a, plan, grid, smem, st);
  if (BN == 256) return dispatch_conv<256>(a, ntn, staged, stages, st);
  if (BN == 128) return dispatch_conv<128>(a, ntn, staged, stages, st);
  return dispatch_conv<64>(a, ntn, staged, stages, st);
}

int msur_conv_forward(const void* x, int B, int L, int Cin, const void* w, int Cout, int taps, const float* bias,
                      int act, void* out_pre, void* out_post, float* out_f32, int out_stride, int n_valid,
                      const void* gate, void* stream) {
  return conv_forward_impl(x, B, L, Cin, w, Cout, taps, bias, act, out_pre, out_post, out_f32, out_stride, n_valid,
                           gate, nullptr, 0, nullptr, 0, nullptr, 0, -1, -1, stream);
}

int msur_conv_forward_fused(const void* x, int B, int L, int Cin, const void* w, int Cout, int taps,
                            const float* bias, int act, void* out_post, int out_stride, void* out_skip,
                            int skip_stride, void* out_dup, int dup_stride, void* out_pool, int pool_stride,
                            int n_valid, void* stream) {
  return conv_forward_impl(x, B, L, Cin, w, Cout, taps, bias, act, nullptr, out_post, nullptr, out_stride, n_valid,
                           nullptr, out_skip, skip_stride, out_dup, dup_stride, out_pool, pool_stride, -1, -1, stream);
}

int msur_conv_set_stages(int bn, int stages) {
  if ((bn != 64 && bn != 128 && bn != 256) || stages < 2 || stages > 4)
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_set_stages: N tile 64, 128 or 256 and 2 to 4 stages");
  std::lock_guard<std::mutex> lk(g_mu);
  g_conv_stages[bn == 256 ? 2 : (bn == 128 ? 1 : 0)] = stages;
  return MSUR_OK;
}

int msur_conv_set_form(int bn, int form) {
  if ((bn != 64 && bn != 128 && bn != 256) || form < 0 || form > 3)
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_set_form: N tile 64, 128 or 256 and form 0 to 3");
  std::lock_guard<std::mutex> lk(g_mu);
  g_conv_form[conv_slot(bn)] = form;
  return MSUR_OK;
}

int msur_conv_get_form(int bn) {
  if (bn != 64 && bn != 128 && bn != 256) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_get_form: bad N tile");
  return g_conv_form[conv_slot(bn)];
}

int msur_conv_set_persistent(int bn, int on) {
  if (bn != 64 && bn != 128 && bn != 256) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_set_persistent: bad N tile");
  std::lock_guard<std::mutex> lk(g_mu);
  int& f = g_conv_form[conv_slot(bn)];
  f = (f & 2) | (on ? 1 : 0);
  return MSUR_OK;
}

int msur_conv_get_persistent(int bn) {
  if (bn != 64 && bn != 128 && bn != 256) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_get_persistent: bad N tile");
  return g_conv_form[conv_slot(bn)] & 1;
}

int msur_conv_get_stages(int bn) {
  if (bn != 64 && bn != 128 && bn != 256) return fail(MSUR_ERR_INVALID_ARG, "msur_conv_get_stages: bad N tile");
  return g_conv_stages[bn == 256 ? 2 : (bn == 128 ? 1 : 0)];
}

static int conv_wgrad_impl(const void* x, const void* dz, int B, int L, int Cin, int Cout, int taps, float* dw, float* db,
                           int splits, void* stream) {
  if (!x || !dz || !dw || B <= 0 || L <= 0 || Cin <= 0 || Cout <= 0 || (taps != 1 && taps != 3))
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_wgrad: bad shape or null pointer (taps must be 1 or 3)");
  if ((Cin % 8) || (Cout % 8) || !aligned16(x) || !aligned16(dz))
    return fail(MSUR_ERR_INVALID_ARG, "msur_conv_wgrad: channels must be multiples of 8, buffers 16-byte aligned");
  unsigned* err = nullptr;
  int rc = setup(&err);
  if (rc) return rc;
  WgradArgs a;
  std::memset(&a, 0, sizeof(a));
  const uint64_t dz_dims[3] = {static_cast<uint64_t>(Cout), static_cast<uint64_t>(L), static_cast<uint64_t>(B)};
  const uint64_t x_dims[3] = {static_cast<uint64_t>(Cin), static_cast<uint64_t>(L), static_cast<uint64_t>(B)};
  const uint32_t box[3] = {64, 64, 1};
  rc = make_map(&a.tm_dz, dz, 3, dz_dims, box);
  const uint32_t xbox[3] = {64, static_cast<uint32_t>(64 + taps - 1), 1};
  if (!rc) rc = make_map(&a.tm_x, x, 3, x_dims, xbox);
  if (rc) return rc;
  a.B = B;
  a.L = L;
  a.Cin = Cin;
  a.Cout = Cout;
  a.taps = taps;
  a.pad = (taps - 1) / 2;
  a.lblocks = (L + 63) / 64;
  a.total = B * a.lblocks;
  const bool automatic = splits <= 0;
  if (automatic) {
    // one CTA per SM and one wave
    const int bn = taps == 3 && Cin <= 64 ? 64 : 128;
    const int tiles = ((Cin + bn - 1) / bn) * ((Cout + BM - 1) / BM);
    splits = std::max(1, static_cast<int>(sms()) / tiles);
  }
  if (splits > a.total) splits = a.total;
  a.per_split = (a.total + splits - 1) / splits;
  splits = (a.total + a.per_split - 1) / a.per_split;
  a.per_phase = a.per_split;
  if (automatic) {
    // The tensor core's sums lose accuracy with their length, so an accumulation takes no more blocks than with
    // two waves of 128-wide tiles on 152 SMs (the accuracy does not follow the device's): 64 x 1000 positions, 256 to 256 channels, 9e-7 of the gradient's norm,
    // 1.8e-6 with a split's blocks in one.
    const int tiles = ((Cin + 127) / 128) * ((Cout + BM - 1) / BM);
    const int chains = std::min(a.total, (2 * 152 + tiles - 1) / tiles);
    a.per_phase = std::min(a.per_split, (a.total + chains - 1) / chains);
  }
  a.dw = dw;
  a.db = db;
  a.bulk = aligned16(dw) ? 1 : 0;
  a.err = err;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (taps == 3) {
    if (Cin <= 64) return launch_wgrad<64, 3, 6>(a, splits, st);
    return launch_wgrad<128, 3, 4>(a, splits, st);
  }
  return launch_wgrad<128, 1, 4>(a, splits, st);
}

int msur_conv_wgrad(const void* x, const void* dz, int B, int L, int Cin, int Cout, int taps, float* dw, int splits,
                    void* stream) {
  return conv_wgrad_impl(x, dz, B, L, Cin, Cout, taps, dw, nullptr, splits, stream);
}

int msur_pool2(const void* x, int B, int Lout, int C, void* y, void* stream) {
  if (!x || !y || B <= 0 || Lout <= 0 || C <= 0) return fail(MSUR_ERR_INVALID_ARG, "msur_pool2: bad argument");
  const size_t n = static_cast<size_t>(B) * Lout * C;
  if (C % 8 == 0 && aligned16(x) && aligned16(y)) {
    return cuda_ok(launch_pdl(pool2_v8_kernel, dim3(grid_for(n / 8)), 256, 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(x), B, Lout, C,
                              static_cast<bf16*>(y)),
                   "pool2_v8_kernel launch");
  }
  pool2_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(x), B, Lout, C,
                                                                           static_cast<bf16*>(y));
  return cuda_ok(cudaGetLastError(), "pool2_kernel launch");
}

int msur_skip_grad(const void* dpool, int Lp, const void* dcat, int cat_stride, int cat_off, const void* z, int B,
                   int L, int C, void* dz, void* stream) {
  if (!z || !dz || B <= 0 || L <= 0 || C <= 0) return fail(MSUR_ERR_INVALID_ARG, "msur_skip_grad: bad argument");
  const size_t n = static_cast<size_t>(B) * L * C;
  if (C % 8 == 0 && cat_stride % 8 == 0 && cat_off % 8 == 0 && aligned16(z) && aligned16(dz) &&
      (!dpool || aligned16(dpool)) && (!dcat || aligned16(dcat))) {
    return cuda_ok(launch_pdl(skip_grad_v8_kernel, dim3(grid_for(n / 8)), 256, 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(dpool), Lp,
                              static_cast<const bf16*>(dcat), cat_stride, cat_off,
                              static_cast<const bf16*>(z), B, L, C, static_cast<bf16*>(dz)),
                   "skip_grad_v8_kernel launch");
  }
  skip_grad_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const bf16*>(dpool), Lp, static_cast<const bf16*>(dcat), cat_stride, cat_off,
      static_cast<const bf16*>(z), B, L, C, static_cast<bf16*>(dz));
  return cuda_ok(cudaGetLastError(), "skip_grad_kernel launch");
}

int msur_upcat(const void* x, const void* skip, int B, int L, int C1, int C2, void* out, void* stream) {
  if (!x || !skip || !out || B <= 0 || L <= 0 || (L % 2)) return fail(MSUR_ERR_INVALID_ARG, "msur_upcat: bad argument");
  const size_t n = static_cast<size_t>(B) * L * (C1 + C2);
  if (C1 % 8 == 0 && C2 % 8 == 0 && aligned16(x) && aligned16(skip) && aligned16(out)) {
    return cuda_ok(launch_pdl(upcat_v8_kernel, dim3(grid_for(n / 8)), 256, 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(x),
                              static_cast<const bf16*>(skip), B, L, C1, C2, static_cast<bf16*>(out)),
                   "upcat_v8_kernel launch");
  }
  upcat_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const bf16*>(x), static_cast<const bf16*>(skip), B, L, C1, C2, static_cast<bf16*>(out));
  return cuda_ok(cudaGetLastError(), "upcat_kernel launch");
}

int msur_upcat_bwd(const void* dcat, const void* z, int B, int Lh, int C1, int C, void* dz, void* stream) {
  if (!dcat || !z || !dz || B <= 0 || Lh <= 0 || C1 > C) return fail(MSUR_ERR_INVALID_ARG, "msur_upcat_bwd: bad argument");
  const size_t n = static_cast<size_t>(B) * Lh * C1;
  if (C1 % 8 == 0 && C % 8 == 0 && aligned16(dcat) && aligned16(z) && aligned16(dz)) {
    return cuda_ok(launch_pdl(upcat_bwd_v8_kernel, dim3(grid_for(n / 8)), 256, 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(dcat),
                              static_cast<const bf16*>(z), B, Lh, C1, C, static_cast<bf16*>(dz)),
                   "upcat_bwd_v8_kernel launch");
  }
  upcat_bwd_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const bf16*>(dcat), static_cast<const bf16*>(z), B, Lh, C1, C, static_cast<bf16*>(dz));
  return cuda_ok(cudaGetLastError(), "upcat_bwd_kernel launch");
}

int msur_bias_grad(const void* dz, uint64_t rows, int C, int stride, float* db, void* stream) {
  if (!dz || !db || C <= 0 || stride < C) return fail(MSUR_ERR_INVALID_ARG, "msur_bias_grad: bad argument");
  if (C % 8 == 0 && stride % 8 == 0 && aligned16(dz)) {
    // four blocks per SM, but at least four rows per thread
    const unsigned gx = (C + 63) / 64;
    const uint64_t most = (rows + 127) / 128;
    const unsigned gy = static_cast<unsigned>(std::min<uint64_t>(std::max(1u, 4 * sms() / gx), most ? most : 1));
    return cuda_ok(launch_pdl(bias_grad_v8_kernel, dim3(gx, gy), 256, 0, static_cast<cudaStream_t>(stream),
                              static_cast<const bf16*>(dz), rows, C, stride, db),
                   "bias_grad_v8_kernel launch");
  }
  dim3 block(32, 8);
  const uint64_t gy = (rows + 8 * 64 - 1) / (8 * 64);
  dim3 grid((C + 31) / 32, static_cast<unsigned>(gy < 512 ? (gy ? gy : 1) : 512));
  bias_grad_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(dz), rows, C,
                                                                          stride, db);
  return cuda_ok(cudaGetLastError(), "bias_grad_kernel launch");
}

int msur_mse(const float* pred, int pstride, const float* target, int tstride, uint64_t rows, int n_valid, void* dp,
             int dstride, float scale, double* loss, void* stream) {
  if (!pred || !target || !loss || n_valid <= 0 || pstride < n_valid || tstride < n_valid || dstride < n_valid)
    return fail(MSUR_ERR_INVALID_ARG, "msur_mse: bad argument");
  const size_t n = rows * static_cast<size_t>(dstride);
  if (n_valid % 4 == 0 && pstride % 4 == 0 && tstride % 4 == 0 && dstride % 4 == 0 && aligned16(pred) &&
      aligned16(target) && (!dp || (reinterpret_cast<uintptr_t>(dp) & 7u) == 0)) {
    const unsigned blocks = std::min(grid_for(n / 4), 8 * sms());
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n / 4 < (1ull << 31)) {
      return cuda_ok(launch_pdl(mse_v4_kernel<unsigned>, dim3(blocks), 256, 0, st, pred, pstride, target,
                                tstride, rows, n_valid, static_cast<bf16*>(dp), dstride, scale, loss),
                     "mse_v4_kernel launch");
    } else {
      return cuda_ok(launch_pdl(mse_v4_kernel<size_t>, dim3(blocks), 256, 0, st, pred, pstride, target,
                                tstride, rows, n_valid, static_cast<bf16*>(dp), dstride, scale, loss),
                     "mse_v4_kernel launch");
    }
  }
  mse_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(pred, pstride, target, tstride, rows, n_valid,
                                                                         static_cast<bf16*>(dp), dstride, scale, loss);
  return cuda_ok(cudaGetLastError(), "mse_kernel launch");
}

int msur_adam(float* p, const float* g, float* m, float* v, uint64_t n, float lr, float b1, float b2, float eps,
              float wd, int step, float gscale, void* p_bf16, void* stream) {
  if (!p || !g || !m || !v || step <= 0) return fail(MSUR_ERR_INVALID_ARG, "msur_adam: bad argument");
  const float bc1 = 1.0f - std::pow(b1, static_cast<float>(step));
  const float bc2 = 1.0f - std::pow(b2, static_cast<float>(step));
  if (n % 4 == 0 && aligned16(p) && aligned16(g) && aligned16(m) && aligned16(v) &&
      (!p_bf16 || (reinterpret_cast<uintptr_t>(p_bf16) & 7u) == 0)) {
    adam_v4_kernel<<<grid_for(n / 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<float4*>(p), reinterpret_cast<const float4*>(g), reinterpret_cast<float4*>(m),
        reinterpret_cast<float4*>(v), n / 4, lr, b1, b2, eps, wd, bc1, bc2, gscale, static_cast<uint2*>(p_bf16));
    return cuda_ok(cudaGetLastError(), "adam_v4_kernel launch");
  }
  adam_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(p, g, m, v, n, lr, b1, b2, eps, wd, bc1,
                                                                          bc2, gscale, static_cast<bf16*>(p_bf16));
  return cuda_ok(cudaGetLastError(), "adam_kernel launch");
}

int msur_weight_transpose(const void* w, int N, int taps, int C, void* wt, void* stream) {
  if (!w || !wt || N <= 0 || taps <= 0 || C <= 0) return fail(MSUR_ERR_INVALID_ARG, "msur_weight_transpose: bad argument");
  const size_t n = static_cast<size_t>(N) * taps * C;
  weight_transpose_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(w), N,
                                                                                      taps, C, static_cast<bf16*>(wt));
  return cuda_ok(cudaGetLastError(), "weight_transpose_kernel launch");
}

int msur_run(const msur_op* ops, int n, void* stream) {
  if (n < 0 || (n && !ops)) return fail(MSUR_ERR_INVALID_ARG, "msur_run: bad argument");
  for (int k = 0; k < n; ++k) {
    const msur_op& o = ops[k];
    const int* i = o.i;
    void* const* p = o.p;
    int rc = MSUR_OK;
    switch (o.kind) {
      case MSUR_OP_CONV:
        rc = conv_forward_impl(p[0], i[0], i[1], i[2], p[1], i[3], i[4], static_cast<const float*>(p[2]), i[5], p[3],
                               p[4], static_cast<float*>(p[5]), i[6], i[7], p[6], p[7], i[8], p[8], i[9], p[9], i[10],
                               o.form, o.stages, stream);
        break;
      case MSUR_OP_WGRAD:
        rc = conv_wgrad_impl(p[0], p[1], i[0], i[1], i[2], i[3], i[4], static_cast<float*>(p[2]),
                             static_cast<float*>(p[3]), i[5], stream);
        break;
      case MSUR_OP_POOL2:
        rc = msur_pool2(p[0], i[0], i[1], i[2], p[1], stream);
        break;
      case MSUR_OP_SKIP_GRAD:
        rc = msur_skip_grad(p[0], i[0], p[1], i[1], i[2], p[2], i[3], i[4], i[5], p[3], stream);
        break;
      case MSUR_OP_UPCAT:
        rc = msur_upcat(p[0], p[1], i[0], i[1], i[2], i[3], p[2], stream);
        break;
      case MSUR_OP_UPCAT_BWD:
        rc = msur_upcat_bwd(p[0], p[1], i[0], i[1], i[2], i[3], p[2], stream);
        break;
      default:
        rc = fail(MSUR_ERR_INVALID_ARG, "msur_run: operation %d has an unknown kind %d", k, o.kind);
    }
    if (rc) return rc;
  }
  return MSUR_OK;
}

int msur_weight_transpose_list(int count, const void* const* w, const int* N, const int* taps, const int* C,
                               void* const* wt, void* stream) {
  if (count <= 0 || count > MSUR_MAX_TRANSPOSES || !w || !N || !taps || !C || !wt)
    return fail(MSUR_ERR_INVALID_ARG, "msur_weight_transpose_list: bad argument");
  TransposeList a;
  std::memset(&a, 0, sizeof(a));
  a.count = count;
  int blocks = 0;
  for (int k = 0; k < count; ++k) {
    if (!w[k] || !wt[k] || N[k] <= 0 || taps[k] <= 0 || C[k] <= 0)
      return fail(MSUR_ERR_INVALID_ARG, "msur_weight_transpose_list: bad entry %d", k);
    if ((N[k] % 8) || (C[k] % 8) || !aligned16(w[k]) || !aligned16(wt[k]))
      return fail(MSUR_ERR_INVALID_ARG, "msur_weight_transpose_list: entry %d: channels must be multiples of 8, "
                                        "buffers 16-byte aligned", k);
    a.first[k] = blocks;
    a.w[k] = static_cast<const bf16*>(w[k]);
    a.wt[k] = static_cast<bf16*>(wt[k]);
    a.N[k] = N[k];
    a.taps[k] = taps[k];
    a.C[k] = C[k];
    blocks += ((N[k] + 63) / 64) * ((C[k] + 63) / 64) * taps[k];
  }
  a.first[count] = blocks;
  weight_transpose_list_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return cuda_ok(cudaGetLastError(), "weight_transpose_list_kernel launch");
}

int msur_assemble_input(const float* track, const float* params, int B, int L, int C, void* x, void* stream) {
  if (!track || !params || !x || C < 8 || (C % 8)) return fail(MSUR_ERR_INVALID_ARG, "msur_assemble_input: bad argument");
  const size_t n = static_cast<size_t>(B) * L * C;
  if (aligned16(x)) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n / 8 < (1ull << 31)) {
      return cuda_ok(launch_pdl(assemble_input_v8_kernel<unsigned>, dim3(grid_for(n / 8)), 256, 0, st,
                                track, params, B, L, C, static_cast<uint4*>(x)),
                     "assemble_input_v8_kernel launch");
    } else {
      return cuda_ok(launch_pdl(assemble_input_v8_kernel<size_t>, dim3(grid_for(n / 8)), 256, 0, st, track,
                                params, B, L, C, static_cast<uint4*>(x)),
                     "assemble_input_v8_kernel launch");
    }
  }
  assemble_input_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(track, params, B, L, C,
                                                                                   static_cast<bf16*>(x));
  return cuda_ok(cudaGetLastError(), "assemble_input_kernel launch");
}

int msur_band_target(const uint32_t* band, uint64_t ncols, int nrows, float* out, void* stream) {
  if (!band || !out || nrows <= 0) return fail(MSUR_ERR_INVALID_ARG, "msur_band_target: bad argument");
  band_target_kernel<<<grid_for(ncols * 32), 256, 0, static_cast<cudaStream_t>(stream)>>>(band, ncols, nrows, out);
  return cuda_ok(cudaGetLastError(), "band_target_kernel launch");
}

}  // extern "C"

namespace {
template <unsigned WHICH>
void launch_map_sums(const float* pred, uint64_t ps, const float* ref, uint64_t rs, uint64_t n, dim3 grid,
                     const double* means, double* out, bool vec, cudaStream_t st) {
  if (vec && means) map_sums_pair_kernel<true, true, WHICH><<<grid, 256, 0, st>>>(pred, ps, ref, rs, n, means, out);
  else if (vec) map_sums_pair_kernel<true, false, WHICH><<<grid, 256, 0, st>>>(pred, ps, ref, rs, n, means, out);
  else if (means) map_sums_pair_kernel<false, true, WHICH><<<grid, 256, 0, st>>>(pred, ps, ref, rs, n, means, out);
  else map_sums_pair_kernel<false, false, WHICH><<<grid, 256, 0, st>>>(pred, ps, ref, rs, n, means, out);
}
}  // namespace

extern "C" {

int msur_map_sums_of(unsigned which, const float* pred, uint64_t pstride_map, const float* ref, uint64_t rstride_map,
                     uint64_t n, int nmaps, const double* means, double* out, void* stream) {
  if (!pred || !ref || !out || nmaps <= 0 || nmaps > 65535) return fail(MSUR_ERR_INVALID_ARG, "msur_map_sums: bad argument");
  // blocks of 32768 elements, about eight per SM over all maps
  const uint64_t steps = (n + 32767) / 32768, most = std::max(1, 8 * static_cast<int>(sms()) / nmaps);
  const dim3 grid(static_cast<unsigned>(std::min(steps, most)), nmaps);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = n % 4 == 0 && pstride_map % 4 == 0 && rstride_map % 4 == 0 && aligned16(pred) && aligned16(ref);
  if (which == MSUR_SUMS_RAW) launch_map_sums<MSUR_SUMS_RAW>(pred, pstride_map, ref, rstride_map, n, grid, means, out, vec, st);
  else if (which == MSUR_SUMS_CENTRED)
    launch_map_sums<MSUR_SUMS_CENTRED>(pred, pstride_map, ref, rstride_map, n, grid, means, out, vec, st);
  else if (which == MSUR_SUMS_ALL) launch_map_sums<MSUR_SUMS_ALL>(pred, pstride_map, ref, rstride_map, n, grid, means, out, vec, st);
  else return fail(MSUR_ERR_INVALID_ARG, "msur_map_sums_of: unknown selection %u", which);
  return cuda_ok(cudaGetLastError(), "map_sums_pair_kernel launch");
}

int msur_map_sums(const float* pred, uint64_t pstride_map, const float* ref, uint64_t rstride_map, uint64_t n,
                  int nmaps, const double* means, double* out, void* stream) {
  return msur_map_sums_of(MSUR_SUMS_ALL, pred, pstride_map, ref, rstride_map, n, nmaps, means, out, stream);
}

int msur_compact_rows(const float* in, int stride, uint64_t rows, int n_valid, float* out, void* stream) {
  if (!in || !out || n_valid <= 0 || stride < n_valid) return fail(MSUR_ERR_INVALID_ARG, "msur_compact_rows: bad argument");
  const size_t n = rows * static_cast<size_t>(n_valid);
  compact_rows_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(in, stride, rows, n_valid, out);
  return cuda_ok(cudaGetLastError(), "compact_rows_kernel launch");
}

}  // extern "C"
