// Block-of-tokens INT8 quantiser of the INT8 x FP8 attention path: x[b, h, n, :] bf16 (any strides) ->
// y[b, h, n, align16(D)] int8 and one fp32 scale per block of `block` consecutive tokens (all D features):
//   scale = max|x| / 127 over the block,  y = trunc(x / scale)  (0 when the block is all zero), padding columns 0.
// Optionally x is first reduced by a bf16 vector per head, x - sub rounded to bf16 (the reference takes the mean over
// the tokens off K with a tensor subtraction of its own, attention.py:157: one pass over K less).
// Stands in for the Triton kernel and its wrapper in ac4k_kernel's python/ac4k_kernel/ops/attention.py:18-48 and
// :51-99 (`tl.cast(fp32 -> int8)` truncates toward zero; the division is a true fp32 division).
//
// One CTA per (token block, head, batch entry): the block (at most 128 x 256 bf16) is read once,
// reduced to its maximum through shared memory, and written back as bytes.  HBM traffic 2 + 1 bytes per element.
// `beside` (q in ac4k_attention_quantize_int8, and V's quantiser): the kernel runs beside the quantiser in front of it in the stream
// instead of behind it.  That one let it start after its own wait, so what both read is complete; neither reads what the other
// writes, and the outputs of both were allocated before the first was launched.  The wait comes at the end instead, so that whoever
// waits for this kernel has waited for that one too.
// Three kernels: the block staged in shared memory by a TMA load (features a multiple of 8 and at most 256, aligned
// strides: the usual case), 16-byte vectors held in registers, single elements for anything else.
#include <algorithm>

#include "gemm_common.cuh"

namespace ac4k {

static constexpr int kQ8Threads = 256;
static constexpr int kQ8MaxElemsPerThread = 128;     // 128 tokens x 256 features / 256 threads

// Any strides and alignment (odd head dimensions above all): a warp takes whole rows, a lane four neighbouring features of
// each, so that no index is divided and the codes leave as words.  The first 128 features of the block stay in registers
// between the maximum and the codes (packed bf16: eight rows a warp), further ones are read again from L1 / L2.  The quotient
// as in quantize8_by_reciprocal below.  [11, 100, 12, 65]: 23 us (k) and 13 us (q) with one element per thread and step, an index
// division and an fp32 division each; 15 and 15 without the index division and the registers; 8.5 each like this.
static constexpr int kQ8AnyRows = 8;       // rows of the block that a warp takes at most

// trunc(RN(f / s)), |f / s| <= 127, as a byte; rs = RN(1 / s)
__device__ __forceinline__ uint32_t quantize_code(float f, float s, float rs) {
  const float t = __fmul_rn(f, rs);
  const float fl = __fsub_rn(__fadd_rd(fabsf(t), 8388608.0f), 8388608.0f);
  if (fabsf(__fsub_rn(__fsub_rn(fabsf(t), fl), 0.5f)) < 0.4999f)
    return __float_as_uint(__fadd_rn(copysignf(fl, t), 12582912.0f)) & 0xffu;
  if (f == 0.0f) return 0u;
  return (uint32_t)__float2int_rz(__fdiv_rn(f, s)) & 0xffu;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) quantize_int8_block_kernel(
    int8_t *__restrict__ y, float *__restrict__ scale, const uint16_t *__restrict__ x, int N, int D, int Dp, int block, int nblk,
    int64_t sb, int64_t sh, int64_t sn, int64_t sd, int H, const uint16_t *__restrict__ sub, int64_t ub, int64_t uh, bool beside) {
  constexpr int kWarps = THREADS / 32;
  __shared__ float red[kWarps];
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int n0 = blk * block;
  const int rows = min(block, N - n0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint16_t *src = x + b * sb + h * sh + (int64_t)(n0 + warp) * sn;      // this warp's first row
  const uint16_t *subp = sub != nullptr ? sub + b * ub + h * uh : nullptr;
  const int64_t row_step = kWarps * sn;
  // four features of one row as packed bf16 pairs; u: the packed vector to take off
  auto load_sub = [&](int c0, uint32_t (&u)[2]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t e = subp != nullptr && c0 + i < D ? (uint32_t)__ldg(subp + c0 + i) : 0u;
      u[i >> 1] = (i & 1) ? (u[i >> 1] | (e << 16)) : e;
    }
  };
  auto load4 = [&](const uint16_t *row, int c0, const uint32_t (&u)[2], uint32_t (&v)[2]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t e = c0 + i < D ? (uint32_t)__ldg(row + (c0 + i) * sd) : 0u;
      v[i >> 1] = (i & 1) ? (v[i >> 1] | (e << 16)) : e;
    }
    if (subp != nullptr) {      // x - sub rounded to bf16, as a bf16 tensor subtraction gives it
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&v[i]), *reinterpret_cast<const __nv_bfloat162 *>(&u[i]));
        v[i] = *reinterpret_cast<const uint32_t *>(&d);
      }
    }
  };
  uint32_t am2 = 0, keep[kQ8AnyRows][2];
  if (!beside) grid_dependency_wait();
  grid_launch_dependents();
  for (int c0 = 4 * lane; c0 < Dp; c0 += 128) {
    uint32_t u[2];
    load_sub(c0, u);
    const uint16_t *row = src;
#pragma unroll
    for (int i = 0; i < kQ8AnyRows; ++i, row += row_step) {
      uint32_t v[2] = {0u, 0u};
      if (warp + i * kWarps < rows) load4(row, c0, u, v);
      am2 = max_bf16x2(am2, max_bf16x2(abs_bf16x2(v[0]), abs_bf16x2(v[1])));
      if (c0 < 128) { keep[i][0] = v[0]; keep[i][1] = v[1]; }
    }
  }
  float amax = hmax_bf16x2_to_f32(am2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) amax = fmaxf(amax, red[w]);
  const float s = __fdiv_rn(amax, 127.0f);
  const float rs = __frcp_rn(s);
  if (threadIdx.x == 0) scale[((int64_t)b * H + h) * nblk + blk] = s;
  int8_t *dst = y + (((int64_t)b * H + h) * N + n0 + warp) * Dp;
  const bool words = (reinterpret_cast<uintptr_t>(y) & 3) == 0;       // (Dp is a multiple of 16)
  for (int c0 = 4 * lane; c0 < Dp; c0 += 128) {
    uint32_t u[2];
    if (c0 >= 128) load_sub(c0, u);
    const uint16_t *row = src;
#pragma unroll
    for (int i = 0; i < kQ8AnyRows; ++i, row += row_step) {
      if (warp + i * kWarps >= rows) break;
      uint32_t v[2] = {keep[i][0], keep[i][1]};
      if (c0 >= 128) load4(row, c0, u, v);
      uint32_t o = 0;
      if (s != 0.0f) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          o |= quantize_code(__uint_as_float((k & 1) ? (v[k >> 1] & 0xffff0000u) : (v[k >> 1] << 16)), s, rs) << (8 * k);
      }
      int8_t *at = dst + (int64_t)(i * kWarps) * Dp + c0;
      if (words) *reinterpret_cast<uint32_t *>(at) = o;
      else
        for (int k = 0; k < 4; ++k) at[k] = (int8_t)(o >> (8 * k));
    }
  }
  if (beside) grid_dependency_wait();
}

// The usual case: features contiguous, D a multiple of 8, rows 16-byte aligned.  A thread takes 16-byte vectors of eight
// features (consecutive threads = consecutive vectors of a row, then the next row), keeps them packed in registers,
// and writes eight bytes per vector.  VPT: vectors per thread, >= block * D / 8 / 256.
template <int VPT>
__global__ void __launch_bounds__(kQ8Threads) quantize_int8_block_vec_kernel(
    int8_t *__restrict__ y, float *__restrict__ scale, const uint16_t *__restrict__ x, int N, int D, int Dp, int block, int nblk,
    int64_t sb, int64_t sh, int64_t sn, int H, const uint16_t *__restrict__ sub, int64_t ub, int64_t uh, bool beside) {
  __shared__ float red[kQ8Threads / 32];
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int n0 = blk * block;
  const int rows = min(block, N - n0);
  const uint16_t *src = x + b * sb + h * sh + (int64_t)n0 * sn;
  const int vpr = D / 8, vpr_out = Dp / 8;            // vectors per input row / per output row (padding included)
  const int nvec = rows * vpr_out;
  uint4 v[VPT];
  __nv_bfloat162 am2 = __floats2bfloat162_rn(0.0f, 0.0f);
  if (!beside) grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = i * kQ8Threads + threadIdx.x;
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (e < nvec) {
      const int r = e / vpr_out, c = e - r * vpr_out;
      if (c < vpr) {
        v[i] = __ldcs(reinterpret_cast<const uint4 *>(src + (int64_t)r * sn) + c);
        __nv_bfloat162 *h2 = reinterpret_cast<__nv_bfloat162 *>(&v[i]);
        if (sub != nullptr) {      // x - sub rounded to bf16, as a bf16 tensor subtraction gives it
          const uint4 u = __ldg(reinterpret_cast<const uint4 *>(sub + b * ub + h * uh) + c);
          const __nv_bfloat162 *u2 = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
          for (int k = 0; k < 4; ++k) h2[k] = __hsub2(h2[k], u2[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) am2 = __hmax2(am2, __habs2(h2[k]));
      }
    }
  }
  float amax = fmaxf(__low2float(am2), __high2float(am2));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kQ8Threads / 32; ++w) amax = fmaxf(amax, red[w]);
  const float s = __fdiv_rn(amax, 127.0f);
  if (threadIdx.x == 0) scale[((int64_t)b * H + h) * nblk + blk] = s;
  uint2 *dst = reinterpret_cast<uint2 *>(y + (((int64_t)b * H + h) * N + n0) * Dp);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = i * kQ8Threads + threadIdx.x;
    if (e < nvec) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      uint32_t o[2] = {0u, 0u};
      if (s != 0.0f) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float f = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
          o[k >> 2] |= ((uint32_t)__float2int_rz(__fdiv_rn(f, s)) & 0xffu) << (8 * (k & 3));
        }
      }
      __stcs(dst + e, make_uint2(o[0], o[1]));
    }
  }
  if (beside) grid_dependency_wait();
}

// Eight elements of a 16-byte vector -> eight int8 codes trunc(RN(f / s)), |f / s| <= 127, without a division or a
// float -> int conversion per element (both run on the 16-per-clock pipe, which bounds the kernel otherwise).  With
// rs = RN(1 / s), t = f * rs is within 1.5 * 2^-23 * |f / s| < 2.3e-5 of the correctly rounded quotient, so the two
// truncate alike unless t lies that close to an integer.  floor(|t|) comes from adding 2^23 with round-down, its
// fraction is exact, and the code is the low byte of sign(t) * floor(|t|) + 1.5 * 2^23 (two's complement for free).
// Returns false - and the caller takes the true division for the whole vector - if any fraction is within 1e-4 of an
// integer (zero, infinities and NaNs included).
__device__ __forceinline__ bool quantize8_by_reciprocal(const uint4 &v, float rs, uint32_t (&o)[2]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t m[8];
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float f = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
    const float t = __fmul_rn(f, rs);
    const float fl = __fsub_rn(__fadd_rd(fabsf(t), 8388608.0f), 8388608.0f);
    const float frac = __fsub_rn(fabsf(t), fl);
    ok = ok && (fabsf(__fsub_rn(frac, 0.5f)) < 0.4999f);
    m[k] = __float_as_uint(__fadd_rn(copysignf(fl, t), 12582912.0f));
  }
  o[0] = __byte_perm(__byte_perm(m[0], m[1], 0x0040), __byte_perm(m[2], m[3], 0x0040), 0x5410);
  o[1] = __byte_perm(__byte_perm(m[4], m[5], 0x0040), __byte_perm(m[6], m[7], 0x0040), 0x5410);
  return ok;
}

// The same quantiser with the block staged in shared memory by one TMA load (a box of D features x `block` tokens of the
// [B, H, N, D] tensor, whatever its strides; tokens past N arrive as zeros): no thread holds the block in registers
// while it is in flight, so seven CTAs fit on an SM instead of four and the loads of all of them are outstanding at
// once.  D a multiple of 8 and at most 256, strides multiples of 8 elements, base 16-byte aligned.
__global__ void __launch_bounds__(kQ8Threads) quantize_int8_block_tma_kernel(
    const __grid_constant__ CUtensorMap tmap, int8_t *__restrict__ y, float *__restrict__ scale, int N, int D, int Dp, int block,
    int nblk, int H, const uint16_t *__restrict__ sub, int64_t ub, int64_t uh, bool beside, unsigned int *status,
    unsigned long long wait_ns) {
  extern __shared__ __align__(128) uint8_t q8_tile[];
  __shared__ __align__(8) uint64_t bar_mem;
  __shared__ float red[kQ8Threads / 32];
  using namespace ptx;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int n0 = blk * block;
  const int rows = min(block, N - n0);
  const uint32_t bar = smem_u32(&bar_mem), tile = smem_u32(q8_tile);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (!beside) grid_dependency_wait();
  grid_launch_dependents();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, (uint32_t)(block * D * 2));     // the whole box, rows past N included (zeros)
    tma_load_4d(tile, &tmap, 0, n0, h, b, bar);
  }
  if (!mbar_wait(bar, 0, wait_ns)) {
    if (threadIdx.x == 0) atomicExch(status, kStatusTimeoutProducer);
    return;
  }
  const int vpr = D / 8, vpr_out = Dp / 8;            // vectors per input row / per output row (padding included)
  const int nvec = rows * vpr_out;
  const int shift = (vpr_out & (vpr_out - 1)) == 0 ? __ffs(vpr_out) - 1 : -1;     // rows of a power of two of vectors
  auto row_col = [&](int e, int &r, int &c) {
    if (shift >= 0) { r = e >> shift; c = e & (vpr_out - 1); }
    else { r = e / vpr_out; c = e - r * vpr_out; }
  };
  const uint16_t *subp = sub != nullptr ? sub + b * ub + h * uh : nullptr;
  auto load_vec = [&](int r, int c) {
    uint4 v;
    asm volatile("ld.shared::cta.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(tile + (uint32_t)(r * D + c * 8) * 2u));
    if (subp != nullptr) {      // x - sub rounded to bf16, as a bf16 tensor subtraction gives it
      __nv_bfloat162 *h2 = reinterpret_cast<__nv_bfloat162 *>(&v);
      const uint4 u = __ldg(reinterpret_cast<const uint4 *>(subp) + c);
      const __nv_bfloat162 *u2 = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
      for (int k = 0; k < 4; ++k) h2[k] = __hsub2(h2[k], u2[k]);
    }
    return v;
  };
  __nv_bfloat162 am2 = __floats2bfloat162_rn(0.0f, 0.0f);
  for (int e = threadIdx.x; e < nvec; e += kQ8Threads) {
    int r, c;
    row_col(e, r, c);
    if (c < vpr) {
      const uint4 v = load_vec(r, c);
      const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
      for (int k = 0; k < 4; ++k) am2 = __hmax2(am2, __habs2(h2[k]));
    }
  }
  float amax = fmaxf(__low2float(am2), __high2float(am2));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kQ8Threads / 32; ++w) amax = fmaxf(amax, red[w]);
  const float s = __fdiv_rn(amax, 127.0f);
  const float rs = __frcp_rn(s);
  if (threadIdx.x == 0) scale[((int64_t)b * H + h) * nblk + blk] = s;
  uint2 *dst = reinterpret_cast<uint2 *>(y + (((int64_t)b * H + h) * N + n0) * Dp);
  for (int e = threadIdx.x; e < nvec; e += kQ8Threads) {
    int r, c;
    row_col(e, r, c);
    uint32_t o[2] = {0u, 0u};
    if (c < vpr && s != 0.0f) {
      const uint4 v = load_vec(r, c);
      if (!quantize8_by_reciprocal(v, rs, o)) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        o[0] = o[1] = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float f = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
          o[k >> 2] |= ((uint32_t)__float2int_rz(__fdiv_rn(f, s)) & 0xffu) << (8 * (k & 3));
        }
      }
    }
    __stcs(dst + e, make_uint2(o[0], o[1]));
  }
  if (beside) grid_dependency_wait();
}

// K of the attention operator, less its mean over the tokens, for up to 1024 tokens: a cluster of one CTA per 128 tokens holds the
// head's keys in registers, adds up the columns (fp32; through shared memory and, from CTA to CTA, distributed shared memory, in the
// same order in each), rounds the mean to bf16, and quantises what is left as above.  One read of K and one launch, where the mean by
// itself is a launch of 5 us in front.  Lanes and rows as in quantize_int8_block_kernel; D <= 128, features contiguous or not.
static constexpr int kMeanThreads = 512, kMeanMaxCtas = 8;
static_assert(AC4K_ATTENTION_MEAN_TOKENS == 128 * kMeanMaxCtas, "one CTA per 128 keys");

template <bool VEC4>
__global__ void __launch_bounds__(kMeanThreads) quantize_int8_block_mean_kernel(
    int8_t *__restrict__ y, float *__restrict__ scale, const uint16_t *__restrict__ x, int N, int D, int Dp, int64_t sb, int64_t sh,
    int64_t sn, int64_t sd, int H) {
  constexpr int kWarps = kMeanThreads / 32, kRows = 128 / kWarps;
  __shared__ float red[kWarps];
  __shared__ __align__(16) float sums[kWarps][128];
  __shared__ float peer[kMeanMaxCtas][128];
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z, nblk = gridDim.x;
  if (nblk > 1) ptx::cluster_arrive_relaxed();
  const int n0 = blk * 128;
  const int rows = min(128, N - n0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = 4 * lane;
  const uint16_t *src = x + b * sb + h * sh + (int64_t)(n0 + warp) * sn;
  uint32_t keep[kRows][2];
  float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const uint16_t *row = src + (int64_t)(i * kWarps) * sn;
    uint32_t v[2] = {0u, 0u};
    if (warp + i * kWarps < rows) {
      if (VEC4) {
        if (c0 < D) {
          const uint2 w = __ldg(reinterpret_cast<const uint2 *>(row + c0));
          v[0] = w.x;
          v[1] = w.y;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (c0 + k < D) v[k >> 1] |= (uint32_t)__ldg(row + (c0 + k) * sd) << (16 * (k & 1));
      }
    }
    keep[i][0] = v[0];
    keep[i][1] = v[1];
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) sum[k] += __uint_as_float((k & 1) ? (keep[i][k >> 1] & 0xffff0000u) : (keep[i][k >> 1] << 16));
  *reinterpret_cast<float4 *>(&sums[warp][c0]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
  __syncthreads();
  if (nblk > 1) ptx::cluster_wait();                            // every CTA of the cluster runs
  if (threadIdx.x < 128) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += sums[w][threadIdx.x];
    peer[blk][threadIdx.x] = t;
    for (int c = 0; c < nblk; ++c)
      if (c != blk) ptx::st_shared_cluster_u32(ptx::map_to_cta(ptx::smem_u32(&peer[blk][threadIdx.x]), c), __float_as_uint(t));
  }
  if (nblk > 1) ptx::cluster_sync();
  else __syncthreads();
  uint32_t u[2];
  {
    float m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m[k] = 0.0f;
      for (int c = 0; c < nblk; ++c) m[k] += peer[c][c0 + k];
      m[k] = __fdiv_rn(m[k], (float)N);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const __nv_bfloat162 h2 = __floats2bfloat162_rn(m[2 * k], m[2 * k + 1]);
      u[k] = *reinterpret_cast<const uint32_t *>(&h2);
    }
  }
  uint32_t am2 = 0;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    if (warp + i * kWarps >= rows) break;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&keep[i][k]), *reinterpret_cast<const __nv_bfloat162 *>(&u[k]));
      keep[i][k] = *reinterpret_cast<const uint32_t *>(&d);       // (features past D: 0 - 0)
    }
    am2 = max_bf16x2(am2, max_bf16x2(abs_bf16x2(keep[i][0]), abs_bf16x2(keep[i][1])));
  }
  float amax = hmax_bf16x2_to_f32(am2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) amax = fmaxf(amax, red[w]);
  const float s = __fdiv_rn(amax, 127.0f);
  const float rs = __frcp_rn(s);
  if (threadIdx.x == 0) scale[((int64_t)b * H + h) * nblk + blk] = s;
  if (c0 < Dp) {
    int8_t *dst = y + (((int64_t)b * H + h) * N + n0 + warp) * Dp + c0;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      if (warp + i * kWarps >= rows) break;
      uint32_t o = 0;
      if (s != 0.0f) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          o |= quantize_code(__uint_as_float((k & 1) ? (keep[i][k >> 1] & 0xffff0000u) : (keep[i][k >> 1] << 16)), s, rs) << (8 * k);
      }
      *reinterpret_cast<uint32_t *>(dst + (int64_t)(i * kWarps) * Dp) = o;
    }
  }
}

static int quantize_int8_block_mean(void *out, float *scale, const void *in, const int64_t shape[4], const int64_t stride[4], cudaStream_t stream) {
  const int64_t B = shape[0], H = shape[1], N = shape[2], D = shape[3], nblk = ceil_div(N, 128);
  const bool vec4 = stride[3] == 1 && D % 4 == 0 && stride[0] % 4 == 0 && stride[1] % 4 == 0 && stride[2] % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 7) == 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nblk, (unsigned)H, (unsigned)B);
  cfg.blockDim = dim3(kMeanThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)nblk;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  AC4K_CUDA_TRY(cudaLaunchKernelEx(&cfg, vec4 ? quantize_int8_block_mean_kernel<true> : quantize_int8_block_mean_kernel<false>, static_cast<int8_t *>(out),
                                   scale, static_cast<const uint16_t *>(in), (int)N, (int)D, (int)align_up(D, 16), stride[0], stride[1], stride[2],
                                   stride[3], (int)H));
  return 0;
}

}  // namespace ac4k

using namespace ac4k;

static int quantize_int8_block(void *out, float *scale, const void *in, const int64_t shape[4], const int64_t stride[4], int64_t block,
                               const void *sub, const int64_t sub_stride[2], bool beside, cudaStream_t stream) {
  if (!shape || !stride) return fail(AC4K_ERR_NULL, "shape/stride is NULL");
  const int64_t B = shape[0], H = shape[1], N = shape[2], D = shape[3];
  if (B < 0 || H < 0 || N < 0 || D < 0) return fail(AC4K_ERR_SHAPE, "negative dimension");
  if (block < 16 || block > 128 || (block & (block - 1))) return fail(AC4K_ERR_SHAPE, "the token block must be a power of two in [16, 128], got %lld", (long long)block);
  if (B == 0 || H == 0 || N == 0 || D == 0) return 0;
  if (!out || !scale || !in) return fail(AC4K_ERR_NULL, "out/scale/in is NULL");
  const int64_t Dp = align_up(D, 16);
  if (block * Dp > (int64_t)kQ8MaxElemsPerThread * kQ8Threads)
    return fail(AC4K_ERR_UNSUPPORTED, "block x align16(D) up to %d elements is built, got %lld x %lld", kQ8MaxElemsPerThread * kQ8Threads,
                (long long)block, (long long)Dp);
  if (H > 65535 || B > 65535 || N > INT32_MAX) return fail(AC4K_ERR_SHAPE, "dimension too large");
  if ((reinterpret_cast<uintptr_t>(in) & 1) || (reinterpret_cast<uintptr_t>(scale) & 3)) return fail(AC4K_ERR_ALIGN, "in must be 2-byte and scale 4-byte aligned");
  if (sub && !sub_stride) return fail(AC4K_ERR_NULL, "sub_stride is NULL");
  const uint16_t *subp = static_cast<const uint16_t *>(sub);
  const int64_t ub = sub ? sub_stride[0] : 0, uh = sub ? sub_stride[1] : 0;
  const int64_t nblk = ceil_div(N, block);
  dim3 grid((unsigned)nblk, (unsigned)H, (unsigned)B);
  const bool vec = stride[3] == 1 && D % 8 == 0 && stride[0] % 8 == 0 && stride[1] % 8 == 0 && stride[2] % 8 == 0 &&
                   (reinterpret_cast<uintptr_t>(in) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0 &&
                   (!sub || ((reinterpret_cast<uintptr_t>(sub) & 15) == 0 && ub % 8 == 0 && uh % 8 == 0));
  // the TMA-staged kernel: additionally D <= 256 (one box row), and a device of compute capability 10
  if (vec && D <= 256 && stride[2] > 0) {
    DeviceInfo di;
    if (int e = get_device_info(&di)) return e;
    CUtensorMap tm;
    if (di.cc_major == 10 && get_tmap_bf16_4d(in, shape, stride, (int)block, &tm) == 0) {
      unsigned int *status = device_status_ptr();
      if (!status) return fail(AC4K_ERR_DEVICE, "cannot resolve the device status word");
      const size_t smem = (size_t)block * D * 2;
      static PerDevice<int> attr_set;
      int dummy = 0;
      if (int e = attr_set.get(&dummy, [&](int &v) {
            AC4K_CUDA_TRY(cudaFuncSetAttribute(quantize_int8_block_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 256 * 2));
            v = 1;
            return 0;
          }))
        return e;
      return launch_kernel<true>(quantize_int8_block_tma_kernel, grid, kQ8Threads, smem, stream, tm, static_cast<int8_t *>(out), scale, (int)N,
                                 (int)D, (int)Dp, (int)block, (int)nblk, (int)H, subp, ub, uh, beside, status, ptx::kWaitTimeoutNs);
    }
  }
  if (vec) {
    const int64_t vpt = ceil_div(block * (Dp / 8), kQ8Threads);
#define AC4K_Q8V_LAUNCH(V)                                                                                                            \
  return launch_kernel<true>(quantize_int8_block_vec_kernel<V>, grid, kQ8Threads, 0, stream, static_cast<int8_t *>(out), scale,           \
                             static_cast<const uint16_t *>(in), (int)N, (int)D, (int)Dp, (int)block, (int)nblk, stride[0], stride[1],  \
                             stride[2], (int)H, subp, ub, uh, beside)
    if (vpt <= 2) AC4K_Q8V_LAUNCH(2);
    if (vpt <= 4) AC4K_Q8V_LAUNCH(4);
    if (vpt <= 8) AC4K_Q8V_LAUNCH(8);
    AC4K_Q8V_LAUNCH(16);
#undef AC4K_Q8V_LAUNCH
  }
#define AC4K_Q8_LAUNCH(T)                                                                                                                  \
  return launch_kernel<true>(quantize_int8_block_kernel<T>, grid, T, 0, stream, static_cast<int8_t *>(out), scale,                           \
                             static_cast<const uint16_t *>(in), (int)N, (int)D, (int)Dp, (int)block, (int)nblk, stride[0], stride[1], stride[2], \
                             stride[3], (int)H, subp, ub, uh, beside)
  static_assert(kQ8AnyRows * (512 / 32) >= 128 && kQ8AnyRows * (128 / 32) >= 32, "rows of a block");
  // 16 warps; four where the blocks are short and there are enough of them for the chip, since every warp walks the features,
  // however few rows it has: [1, 4096, 16, 66] in blocks of 16 took 34.8 us with 16 warps and takes 19.3 with four, in blocks of 32
  // 23.3 and 17.2; [1, 64, 1, 65] in blocks of 16 2.3 and 3.6.  Blocks of 64 and 128: 16 warps are as fast as eight or faster.
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  if (block <= 32 && nblk * H * B >= 2 * (int64_t)di.sms) AC4K_Q8_LAUNCH(128);
  AC4K_Q8_LAUNCH(512);
#undef AC4K_Q8_LAUNCH
}

extern "C" int ac4k_quantize_int8_block(void *out, float *scale, const void *in, const int64_t shape[4], const int64_t stride[4],
                                        int64_t block, const void *sub, const int64_t sub_stride[2], ac4k_stream_t stream) {
  return quantize_int8_block(out, scale, in, shape, stride, block, sub, sub_stride, false, static_cast<cudaStream_t>(stream));
}

extern "C" int ac4k_attention_quantize_int8(void *q8, float *q_sf, void *k8, float *k_sf, void *v8, float *v_sf, const void *q,
                                            const int64_t q_stride[4], const void *k, const int64_t k_stride[4], const void *v,
                                            const int64_t v_stride[4], const void *k_mean, const int64_t mean_stride[2], int64_t B, int64_t H,
                                            int64_t Nq, int64_t Nkv, int64_t D, int64_t Dv, ac4k_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!q_stride || !k_stride || !v_stride) return fail(AC4K_ERR_NULL, "a stride is NULL");
  if (B <= 0 || H <= 0 || Nq <= 0 || Nkv <= 0 || D <= 0 || D > 128 || Dv <= 0) return fail(AC4K_ERR_SHAPE, "dimensions must be positive and D at most 128");
  const int64_t q_shape[4] = {B, H, Nq, D}, k_shape[4] = {B, H, Nkv, D};
  if (k_mean) {
    if (int e = quantize_int8_block(k8, k_sf, k, k_shape, k_stride, 128, k_mean, mean_stride, false, stream)) return e;
  } else {
    if (Nkv > AC4K_ATTENTION_MEAN_TOKENS) return fail(AC4K_ERR_SHAPE, "the mean of more than %d keys has to be given", AC4K_ATTENTION_MEAN_TOKENS);
    if (!k8 || !k_sf || !k) return fail(AC4K_ERR_NULL, "k8/k_sf/k is NULL");
    if (H > 65535 || B > 65535) return fail(AC4K_ERR_SHAPE, "dimension too large");
    if ((reinterpret_cast<uintptr_t>(k) & 1) || ((reinterpret_cast<uintptr_t>(k_sf) | reinterpret_cast<uintptr_t>(k8)) & 3))
      return fail(AC4K_ERR_ALIGN, "k must be 2-byte, k8 and k_sf 4-byte aligned");
    if (int e = quantize_int8_block_mean(k8, k_sf, k, k_shape, k_stride, stream)) return e;
  }
  if (int e = quantize_int8_block(q8, q_sf, q, q_shape, q_stride, 64, nullptr, nullptr, true, stream)) return e;
  const int64_t v_shape[4] = {B, H, Dv, Nkv}, v_order[4] = {v_stride[0], v_stride[1], v_stride[3], v_stride[2]};
  return launch_fp8_beside(v8, v_sf, v, 2.25f, v_shape, v_order, stream);
}
