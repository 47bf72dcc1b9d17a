// BF16 -> NVFP4 quantiser and the global-scale (amax) reduction for sm_100a.
//
// Semantics follow ac4k_kernel's lib/cuda/sm120/quantize_nvfp4.cu:49-157 (block of 16,
// pair of scales packed four to a word, K padded to 64, scale rows padded to 16) with its
// approximate reciprocals replaced by correctly rounded fp32 operations:
//     alpha = 1 / g ;  sf = e4m3(alpha * (amax16 * fp32(1/6))) ;
//     r = sf ? alpha * (1 / float(sf)) : 0 ;  code = e2m1(float(x) * r)
// Four kernels: a tiled one for rows that are contiguous along K (the linear path) and a flat one for those tensors that are too
// small for its tiles, a transposing one for rows that are contiguous along the cross dimension (attention's V), and a strided one
// (any cross/reduce strides, optional K permutation) for everything else.
#include <algorithm>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace ac4k {

__device__ __forceinline__ uint32_t quantize8(const uint4 &v, float r) {
  float f[8];
  f[0] = __fmul_rn(__uint_as_float(v.x << 16), r);
  f[1] = __fmul_rn(__uint_as_float(v.x & 0xFFFF0000u), r);
  f[2] = __fmul_rn(__uint_as_float(v.y << 16), r);
  f[3] = __fmul_rn(__uint_as_float(v.y & 0xFFFF0000u), r);
  f[4] = __fmul_rn(__uint_as_float(v.z << 16), r);
  f[5] = __fmul_rn(__uint_as_float(v.z & 0xFFFF0000u), r);
  f[6] = __fmul_rn(__uint_as_float(v.w << 16), r);
  f[7] = __fmul_rn(__uint_as_float(v.w & 0xFFFF0000u), r);
  return f32x8_to_e2m1x8(f);
}

// Where a quantiser kernel takes the tensor's global scale from: a scalar on the device, or the per-CTA maxima (bf16 bits)
// that amax_partial_kernel left, which every CTA reduces for itself (the first one stores the scale for the caller).  The
// second form needs no zeroed accumulator, i.e. no memset in front of the reduction.
struct ScaleSource {
  const float *g;
  const uint32_t *partial;
  int n_partial;
  float max_scale;
  float *g_out;
  bool last_first;      // tiled kernel: take the row tiles from the last to the first
};

// maximum of one value per thread over the CTA, in every thread (s_m: one word per warp; ends with all threads past a barrier)
__device__ __forceinline__ uint32_t cta_max(uint32_t m, uint32_t *s_m) {
  m = __reduce_max_sync(0xFFFFFFFFu, m);
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  m = (int)(threadIdx.x & 31) < nw ? s_m[threadIdx.x & 31] : 0u;
  return __reduce_max_sync(0xFFFFFFFFu, m);
}

// 1 / global scale, in every thread.  PARTIAL: called by all threads of the CTA, behind the dependency wait.
template <bool PARTIAL>
__device__ __forceinline__ float resolve_alpha(const ScaleSource &src, uint32_t *s_m) {
  if (!PARTIAL) return load_alpha(src.g);
  uint32_t m = 0;
  for (int i = threadIdx.x; i < src.n_partial; i += blockDim.x) m = max(m, __ldcg(src.partial + i));
  const float g = global_scale_of(cta_max(m, s_m), src.max_scale);
  if ((blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) *src.g_out = g;
  return alpha_of(g);
}

// ----------------------------------------------------------------------------------------
// Tiled kernel: one CTA = 128 rows x 256 K-elements, one thread = one 16-element block per
// pass (16 rows x 16 blocks per pass, 8 passes).  A thread loads its block with one 32-byte
// load (half a warp reads 512 contiguous bytes of a row), needs no shuffle for the block amax,
// multiplies with packed fp32x2 instructions, stores 8 bytes of codes (a warp writes two runs
// of 128 bytes) and drops its scale byte into a shared-memory image of the scale tile that is
// written out with full-width stores at the end.  The reciprocal of the e4m3 scale comes from
// a 128-entry table built once per CTA (the scale has only 127 non-negative values).
// The kernel is instruction-issue bound, not bandwidth bound, if written naively: the first
// version (one thread = 8 elements, pair shuffle, IEEE reciprocal per thread) issued ~113
// instructions per 8 elements and reached 4.7 TB/s.
// ----------------------------------------------------------------------------------------
static constexpr int kTileRows = 128;
static constexpr int kThreads = 256;
static constexpr int kBatch = 4;      // passes whose loads are issued together

struct Block16 { uint32_t w[8]; };

template <bool WIDE>
__device__ __forceinline__ Block16 load_block16(const uint16_t *p) {
  Block16 b;
  if (WIDE) {
    uint64_t a0, a1, a2, a3;
    asm volatile("ld.global.nc.L1::no_allocate.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(a0), "=l"(a1), "=l"(a2), "=l"(a3) : "l"(p));
    b.w[0] = (uint32_t)a0; b.w[1] = (uint32_t)(a0 >> 32); b.w[2] = (uint32_t)a1; b.w[3] = (uint32_t)(a1 >> 32);
    b.w[4] = (uint32_t)a2; b.w[5] = (uint32_t)(a2 >> 32); b.w[6] = (uint32_t)a3; b.w[7] = (uint32_t)(a3 >> 32);
  } else {
    const uint4 lo = __ldcs(reinterpret_cast<const uint4 *>(p)), hi = __ldcs(reinterpret_cast<const uint4 *>(p) + 1);
    b.w[0] = lo.x; b.w[1] = lo.y; b.w[2] = lo.z; b.w[3] = lo.w;
    b.w[4] = hi.x; b.w[5] = hi.y; b.w[6] = hi.z; b.w[7] = hi.w;
  }
  return b;
}

// TK: K elements of a CTA's tile, 256 or - for rows of at most 128 elements (attention's q and k: one head's
// features), where half of a 256-wide tile's threads would have nothing to load - 128.
template <int SF_LAYOUT, bool WIDE, int TK, bool PARTIAL>
__device__ __forceinline__ void
nvfp4_quantize_tile(uint8_t *__restrict__ out, uint32_t *__restrict__ sf, const uint16_t *__restrict__ in, const ScaleSource &src,
                    int64_t M, int64_t K, int64_t d1, int64_t stride0, int64_t stride1, int64_t row_stride) {
  constexpr int kTileK = TK, kTileKch = TK / 64;
  constexpr int kRowThreads = TK / 16;                  // threads (16-element blocks) per row of the tile
  constexpr int kPassRows = kThreads / kRowThreads;     // rows the CTA covers per pass
  __shared__ uint32_t s_sf[kTileKch * kTileRows];
  __shared__ float s_rcp[128];
  __shared__ uint32_t s_m[kThreads / 32];

  const int64_t Kp = align_up(K, 64);
  const int64_t KT = Kp / 64;
  const int64_t M16 = align_up(M, 16);
  const int64_t MT = ceil_div(M, 128);
  const int64_t batch = blockIdx.z;
  const int64_t by = src.last_first ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
  const int64_t r0 = by * kTileRows;
  const int64_t k0 = (int64_t)blockIdx.x * kTileK;
  const int blk = threadIdx.x % kRowThreads, prow = threadIdx.x / kRowThreads;

  if (threadIdx.x < 128) {
    // 1 / float(e4m3 byte), correctly rounded; entry 0 is 0 so that a zero scale zeroes the block
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)threadIdx.x, __NV_E4M3);
    const float v = __half2float(__half(h));
    s_rcp[threadIdx.x] = threadIdx.x ? __frcp_rn(v) : 0.0f;
  }
  __syncthreads();
  const int64_t k = k0 + blk * 16;
  const bool k_live = k < Kp;   // block belongs to the (padded) output
  const bool k_data = k < K;    // block has input data (K % 16 == 0 on this path)
  const uint16_t *in_p = in + (batch / d1) * stride0 + (batch % d1) * stride1 + (r0 + prow) * row_stride + k;
  uint8_t *out_p = out + (batch * M + r0 + prow) * (Kp / 2) + k / 2;
  uint8_t *s_bytes = reinterpret_cast<uint8_t *>(s_sf);
  const int kch = blk >> 2, sub = blk & 3;

  if (PARTIAL) grid_dependency_wait();
  grid_launch_dependents();
  const float alpha = resolve_alpha<PARTIAL>(src, s_m);

#pragma unroll 1
  for (int p0 = 0; p0 < kTileRows / kPassRows; p0 += kBatch) {
    Block16 v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int64_t row = r0 + (p0 + u) * kPassRows + prow;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[u].w[i] = 0;
      if (row < M && k_data) v[u] = load_block16<WIDE>(in_p + (int64_t)(p0 + u) * kPassRows * row_stride);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int row_l = (p0 + u) * kPassRows + prow;
      const bool row_ok = r0 + row_l < M;
      const Block16 &b = v[u];
      uint32_t m = max_bf16x2(max_bf16x2(max_bf16x2(abs_bf16x2(b.w[0]), abs_bf16x2(b.w[1])),
                                         max_bf16x2(abs_bf16x2(b.w[2]), abs_bf16x2(b.w[3]))),
                              max_bf16x2(max_bf16x2(abs_bf16x2(b.w[4]), abs_bf16x2(b.w[5])),
                                         max_bf16x2(abs_bf16x2(b.w[6]), abs_bf16x2(b.w[7]))));
      const float amax = hmax_bf16x2_to_f32(m);
      const float s = __fmul_rn(alpha, __fmul_rn(amax, kOneSixth));
      uint16_t pk;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pk) : "f"(0.0f), "f"(s));
      const uint32_t sb = pk & 0x7Fu;
      const float r = __fmul_rn(alpha, s_rcp[sb]);
      if (row_ok && k_live) {
        uint2 codes;
        codes.x = quantize8_x2(b.w[0], b.w[1], b.w[2], b.w[3], r);
        codes.y = quantize8_x2(b.w[4], b.w[5], b.w[6], b.w[7], r);
        __stcs(reinterpret_cast<uint2 *>(out_p + (int64_t)(p0 + u) * kPassRows * (Kp / 2)), codes);
      }
      int off;
      if (SF_LAYOUT == AC4K_SF_AC4K)
        off = (kch * kTileRows + row_l) * 4 + sub;
      else
        off = kch * 512 + (row_l & 31) * 16 + (row_l >> 5) * 4 + sub;
      s_bytes[off] = row_ok ? (uint8_t)sb : (uint8_t)0;
    }
  }
  __syncthreads();

  // write the scale image: kTileKch groups of 128 words
  for (int t = threadIdx.x; t < kTileKch * kTileRows; t += kThreads) {
    const int c = t >> 7, w = t & 127;
    const int64_t k64 = k0 / 64 + c;
    if (k64 >= KT) continue;
    if (SF_LAYOUT == AC4K_SF_AC4K) {
      const int64_t row = r0 + w;
      if (row < M16) sf[(batch * KT + k64) * M16 + row] = s_sf[t];
    } else {
      sf[((batch * MT + by) * KT + k64) * 128 + w] = s_sf[t];
    }
  }
}

template <int SF_LAYOUT, bool WIDE, bool PARTIAL>
__global__ void __launch_bounds__(kThreads)
nvfp4_quantize_tiled_kernel(uint8_t *__restrict__ out, uint32_t *__restrict__ sf, const uint16_t *__restrict__ in, const ScaleSource src,
                            int64_t M, int64_t K, int64_t d1, int64_t stride0, int64_t stride1, int64_t row_stride) {
  nvfp4_quantize_tile<SF_LAYOUT, WIDE, 256, PARTIAL>(out, sf, in, src, M, K, d1, stride0, stride1, row_stride);
}
// Narrow tiles, and five CTAs per SM: 48 registers, where the compiler's own choice is 58 (which is the faster one for the wide tiles).
// [1, 75600, 40, 128]: 166 us with four, 153 with five.
template <int SF_LAYOUT, bool WIDE, bool PARTIAL>
__global__ void __launch_bounds__(kThreads, 5)
nvfp4_quantize_tiled128_kernel(uint8_t *__restrict__ out, uint32_t *__restrict__ sf, const uint16_t *__restrict__ in, const ScaleSource src,
                               int64_t M, int64_t K, int64_t d1, int64_t stride0, int64_t stride1, int64_t row_stride) {
  nvfp4_quantize_tile<SF_LAYOUT, WIDE, 128, PARTIAL>(out, sf, in, src, M, K, d1, stride0, stride1, row_stride);
}

// ----------------------------------------------------------------------------------------
// Strided kernel: one thread = one 16-element block, scalar loads with arbitrary element
// strides; `PERMUTE` applies the K permutation of quantize_nvfp4.cu:86-100 (each group of
// 32 viewed as [4][4][2] and transposed in its first two modes).  Threads are laid out so
// that neighbouring lanes walk the dimension with the smaller stride.
// ----------------------------------------------------------------------------------------
template <int SF_LAYOUT, bool PERMUTE, bool ROW_FASTEST, bool PARTIAL>
__global__ void __launch_bounds__(256)
nvfp4_quantize_strided_kernel(uint8_t *__restrict__ out, uint8_t *__restrict__ sf,
                              const uint16_t *__restrict__ in, const ScaleSource src,
                              int64_t M, int64_t K, int64_t d1, int64_t stride0, int64_t stride1,
                              int64_t stride_m, int64_t stride_k) {
  const int64_t Kp = align_up(K, 64);
  const int64_t KT = Kp / 64;
  const int64_t nblk = Kp / 16;
  const int64_t M16 = align_up(M, 16);
  const int64_t MT = ceil_div(M, 128);
  const int64_t rows_sf = (SF_LAYOUT == AC4K_SF_AC4K) ? M16 : MT * 128;
  const int64_t batch = blockIdx.z;

  int64_t row, blk;
  if (ROW_FASTEST) {   // 32 rows x 8 blocks per CTA
    row = (int64_t)blockIdx.y * 32 + (threadIdx.x & 31);
    blk = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  } else {             // 8 rows x 32 blocks per CTA
    row = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5);
    blk = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
  }
  __shared__ uint32_t s_m[8];
  if (PARTIAL) grid_dependency_wait();
  grid_launch_dependents();
  const float alpha = resolve_alpha<PARTIAL>(src, s_m);
  if (row >= rows_sf || blk >= nblk) return;

  const uint16_t *in_b = in + (batch / d1) * stride0 + (batch % d1) * stride1;

  uint32_t w[8];
  uint32_t amax = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t pair = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t p = blk * 16 + j * 2 + h;   // position in the (permuted) output row
      int64_t k = p;
      if (PERMUTE) {
        const int64_t q = p & 31;
        k = (p - q) + 8 * ((q & 7) >> 1) + 2 * (q >> 3) + (q & 1);
      }
      uint32_t e = 0;
      if (row < M && k < K) e = __ldg(in_b + row * stride_m + k * stride_k);
      pair |= e << (16 * h);
      const uint32_t a = e & 0x7FFFu;
      amax = a > amax ? a : amax;
    }
    w[j] = pair;
  }
  const BlockScale bs = block_scale(bf16_bits_to_f32(amax), alpha);

  if (row < M) {
    uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
    uint2 codes = make_uint2(quantize8(lo, bs.r), quantize8(hi, bs.r));
    *reinterpret_cast<uint2 *>(out + (batch * M + row) * (Kp / 2) + blk * 8) = codes;
  }
  const uint8_t b = (row < M) ? bs.byte : (uint8_t)0;
  const int64_t k64 = blk >> 2;
  if (SF_LAYOUT == AC4K_SF_AC4K) {
    sf[((batch * KT + k64) * M16 + row) * 4 + (blk & 3)] = b;
  } else {
    const int64_t mt = row >> 7, rl = row & 127;
    sf[((batch * MT + mt) * KT + k64) * 512 + (rl & 31) * 16 + (rl >> 5) * 4 + (blk & 3)] = b;
  }
}

// ----------------------------------------------------------------------------------------
// Transposing kernel: rows contiguous in memory along the CROSS dimension (stride_m == 1) and strided
// along K -- attention's V, quantised along the keys with the head dimension as output rows.  The
// strided kernel above reads 64 bytes per warp load there and writes 8-byte pieces 'Kp / 2' apart.
// Here one CTA takes 128 K-elements x 128 rows: a thread loads 32 words (two neighbouring rows x 32
// consecutive K-elements; a warp reads 128 contiguous bytes per load), quantises its four blocks of
// 16 in registers, and codes and scale bytes go through shared memory so that each output row leaves
// as 64 contiguous bytes and the scales as whole words.
// ----------------------------------------------------------------------------------------
template <int SF_LAYOUT, bool PERMUTE, bool PARTIAL>
__global__ void __launch_bounds__(256)
nvfp4_quantize_transposed_kernel(uint8_t *__restrict__ out, uint8_t *__restrict__ sf, const uint16_t *__restrict__ in,
                                 const ScaleSource src, int64_t M, int64_t K, int64_t d1, int64_t stride0,
                                 int64_t stride1, int64_t stride_k) {
  __shared__ uint4 s_codes[128][4 + 1];          // [row][32-element group of the tile], padded
  __shared__ uint32_t s_sf[2][128];              // [K = 64 step of the tile][row]: four scale bytes
  const int64_t Kp = align_up(K, 64), KT = Kp / 64, M16 = align_up(M, 16), MT = ceil_div(M, 128);
  const int64_t batch = blockIdx.z;
  const int64_t k0 = (int64_t)blockIdx.x * 128, m0 = (int64_t)blockIdx.y * 128;
  const int cx = threadIdx.x & 63, kg = threadIdx.x >> 6;
  const int64_t m = m0 + 2 * cx, kb = k0 + 32 * kg;           // this thread: rows m, m + 1; K-elements kb .. kb + 31
  const uint16_t *base = in + (batch / d1) * stride0 + (batch % d1) * stride1;
  __shared__ uint32_t s_m[8];
  if (PARTIAL) grid_dependency_wait();
  grid_launch_dependents();
  const float alpha = resolve_alpha<PARTIAL>(src, s_m);

  uint32_t w[32];                                // w[j]: element kb + j of row m (low half) and of row m + 1 (high half)
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    w[j] = 0u;
    if (m < M && kb + j < K) w[j] = __ldg(reinterpret_cast<const uint32_t *>(base + (kb + j) * stride_k + m));
  }
  uint32_t bytes[2] = {0u, 0u};                  // the two block scales of this group, for row m and row m + 1
  uint4 codes[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    // pairs of consecutive K-elements of row m + r, in output order: position pair j holds elements src(2 j), src(2 j) + 1
    uint32_t pr[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      int e = 2 * j;
      if (PERMUTE) e = 8 * (((2 * j) & 7) >> 1) + 2 * ((2 * j) >> 3);
      pr[j] = __byte_perm(w[e], w[e + 1], r == 0 ? 0x5410 : 0x7632);
    }
    uint32_t cw[4];
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
      uint32_t amax = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = pr[8 * blk + j] & 0x7FFF7FFFu;
        amax = max(amax, max(a & 0xFFFFu, a >> 16));
      }
      const BlockScale bs = block_scale(bf16_bits_to_f32(amax), alpha);
      cw[2 * blk] = quantize8(make_uint4(pr[8 * blk], pr[8 * blk + 1], pr[8 * blk + 2], pr[8 * blk + 3]), bs.r);
      cw[2 * blk + 1] = quantize8(make_uint4(pr[8 * blk + 4], pr[8 * blk + 5], pr[8 * blk + 6], pr[8 * blk + 7]), bs.r);
      bytes[r] |= (uint32_t)((m + r < M) ? bs.byte : (uint8_t)0) << (8 * blk);
    }
    codes[r] = make_uint4(cw[0], cw[1], cw[2], cw[3]);
  }
  s_codes[2 * cx][kg] = codes[0];
  s_codes[2 * cx + 1][kg] = codes[1];
  // scale bytes: group kg covers blocks 2 (kg & 1), 2 (kg & 1) + 1 of K = 64 step kg >> 1
  reinterpret_cast<uint16_t *>(&s_sf[kg >> 1][2 * cx])[kg & 1] = (uint16_t)bytes[0];
  reinterpret_cast<uint16_t *>(&s_sf[kg >> 1][2 * cx + 1])[kg & 1] = (uint16_t)bytes[1];
  __syncthreads();
  // codes: 128 rows x 64 bytes, four threads per row
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int row = v >> 2, g = v & 3;
    if (m0 + row < M && k0 + 32 * g < Kp)
      *reinterpret_cast<uint4 *>(out + (batch * M + m0 + row) * (Kp / 2) + (k0 + 32 * g) / 2) = s_codes[row][g];
  }
  // scales: one word per row and K = 64 step
  {
    const int row = threadIdx.x & 127, ks = threadIdx.x >> 7;
    const int64_t k64 = k0 / 64 + ks, rg = m0 + row;
    const int64_t rows_sf = (SF_LAYOUT == AC4K_SF_AC4K) ? M16 : MT * 128;
    if (k64 < KT && rg < rows_sf) {
      uint32_t *sfw = reinterpret_cast<uint32_t *>(sf);
      if (SF_LAYOUT == AC4K_SF_AC4K)
        sfw[(batch * KT + k64) * M16 + rg] = s_sf[ks][row];
      else
        sfw[((batch * MT + blockIdx.y) * KT + k64) * 128 + (row & 31) * 4 + (row >> 5)] = s_sf[ks][row];
    }
  }
}

// ----------------------------------------------------------------------------------------
// Flat kernel, for tensors whose 128-row tiles would leave most of the chip idle (decode and short prompts): the 16-element
// blocks of the tensor, in memory order, one per thread, which keeps it in registers from the maximum to the codes.
//   CLUSTER  one cluster of up to eight CTAs holds the whole tensor and combines its maxima through distributed shared
//            memory: global scale, codes and block scales in one launch.
//   else     the maxima come from amax_partial_kernel; the data are loaded in front of the dependency wait (they were
//            complete before that kernel began).
// Four neighbouring lanes hold the blocks of one K = 64 step and write its scale word together.
// ----------------------------------------------------------------------------------------
template <int SF_LAYOUT, bool CLUSTER, int THREADS>
__global__ void __launch_bounds__(THREADS)
nvfp4_quantize_flat_kernel(uint8_t *__restrict__ out, uint32_t *__restrict__ sf, const uint16_t *__restrict__ in,
                           const ScaleSource src, int M, int K, int nbatch, int d1, int64_t stride0, int64_t stride1,
                           int64_t row_stride) {
  __shared__ uint32_t s_m[THREADS / 32];
  __shared__ uint32_t s_peer[8];
  const int Kp = (K + 63) / 64 * 64, KT = Kp / 64, nblk = Kp / 16;
  const int rows_sf = SF_LAYOUT == AC4K_SF_AC4K ? (M + 15) / 16 * 16 : (M + 127) / 128 * 128;
  const int items = nbatch * M * nblk;
  const int stride = gridDim.x * blockDim.x;
  const int it = blockIdx.x * blockDim.x + threadIdx.x;         // this thread's block
  if (CLUSTER && gridDim.x > 1) ptx::cluster_arrive_relaxed();  // (waited for where the first store to a peer is)
  auto sf_word = [&](int b, int row, int k64) -> int64_t {
    if (SF_LAYOUT == AC4K_SF_AC4K) return ((int64_t)b * KT + k64) * rows_sf + row;
    return (((int64_t)b * (rows_sf >> 7) + (row >> 7)) * KT + k64) * 128 + (row & 31) * 4 + ((row & 127) >> 5);
  };
  // (the other order, which lets a GEMM begin its weight prefetch under the GEMM before, measures the same: 12.1 us for
  // quantise + GEMM at 1 x 8192 x 8192)
  if (CLUSTER) grid_dependency_wait();
  grid_launch_dependents();

  Block16 v;
#pragma unroll
  for (int i = 0; i < 8; ++i) v.w[i] = 0;
  const int row_all = it / nblk, blk = it - row_all * nblk;
  const int b = row_all / M, row = row_all - b * M;
  if (it < items && blk * 16 < K)
    v = load_block16<false>(in + (int64_t)(b / d1) * stride0 + (int64_t)(b % d1) * stride1 + row * row_stride + blk * 16);
  // scale words of the padding rows
  if (!CLUSTER) grid_dependency_wait();
  {
    const int pad = rows_sf - M, words = nbatch * KT * pad;
    for (int w = it; w < words; w += stride) {
      const int bk = w / pad, r = w - bk * pad, bw = bk / KT;
      sf[sf_word(bw, M + r, bk - bw * KT)] = 0u;
    }
  }
  float alpha;
  if (CLUSTER) {
    const uint32_t *w = v.w;
    // (the 0 takes NaNs out, as in thread_amax)
    const uint32_t m2 = max_bf16x2(0u, max_bf16x2(max_bf16x2(max_bf16x2(abs_bf16x2(w[0]), abs_bf16x2(w[1])), max_bf16x2(abs_bf16x2(w[2]), abs_bf16x2(w[3]))),
                                                  max_bf16x2(max_bf16x2(abs_bf16x2(w[4]), abs_bf16x2(w[5])), max_bf16x2(abs_bf16x2(w[6]), abs_bf16x2(w[7])))));
    uint32_t m = cta_max(max(m2 & 0xFFFFu, m2 >> 16), s_m);
    if (gridDim.x > 1) {
      const uint32_t rank = ptx::cluster_ctarank();
      ptx::cluster_wait();                                        // every CTA of the cluster runs
      if (threadIdx.x < gridDim.x) ptx::st_shared_cluster_u32(ptx::map_to_cta(ptx::smem_u32(s_peer + rank), threadIdx.x), m);
      ptx::cluster_sync();
      m = 0;
      for (int i = 0; i < (int)gridDim.x; ++i) m = max(m, s_peer[i]);
    }
    const float g = global_scale_of(m, src.max_scale);
    if (it == 0) *src.g_out = g;
    alpha = alpha_of(g);
  } else {
    alpha = resolve_alpha<true>(src, s_m);
  }
  {
    const uint32_t *w = v.w;
    const float s = __fmul_rn(alpha, __fmul_rn(amax16_bf16(w), kOneSixth));
    uint16_t pk;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pk) : "f"(0.0f), "f"(s));
    const uint32_t sb = pk & 0x7Fu;
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)sb, __NV_E4M3);
    const float r = __fmul_rn(alpha, sb ? __frcp_rn(__half2float(__half(h))) : 0.0f);
    uint32_t word = sb << (8 * (threadIdx.x & 3));
    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
    if (it < items) {
      uint2 codes;
      codes.x = quantize8_x2(w[0], w[1], w[2], w[3], r);
      codes.y = quantize8_x2(w[4], w[5], w[6], w[7], r);
      *reinterpret_cast<uint2 *>(out + (int64_t)it * 8) = codes;
      if ((blk & 3) == 0) sf[sf_word(b, row, blk >> 2)] = word;
    }
  }
}

// ----------------------------------------------------------------------------------------
// Global scale: max|x| / max_scale.  Division is monotonic, so each CTA divides its own
// maximum and combines with an integer atomicMax on the (non-negative) float bits, the
// same scheme as the reference's Triton kernel (python/ac4k_kernel/ops/quant.py:21-46).
// ----------------------------------------------------------------------------------------
// this thread's share of max|x| (bf16 bits) of `n` contiguous values
__device__ __forceinline__ uint32_t thread_amax(const uint16_t *__restrict__ x, int64_t n) {
  uint32_t m2 = 0;   // packed pair of running maxima (bf16 bits, sign cleared)
  uint32_t m1 = 0;   // scalar head/tail
  // head: elements before the first 16-byte boundary
  const uintptr_t addr = reinterpret_cast<uintptr_t>(x);
  int64_t head = ((16 - (addr & 15)) & 15) / 2;
  if (head > n) head = n;
  const int64_t nvec = (n - head) / 8;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthr = (int64_t)gridDim.x * blockDim.x;
  const uint4 *xv = reinterpret_cast<const uint4 *>(x + head);
  int64_t i = tid;
  for (; i + 3 * nthr < nvec; i += 4 * nthr) {
    uint4 a = __ldcs(xv + i), b = __ldcs(xv + i + nthr), c = __ldcs(xv + i + 2 * nthr),
          d = __ldcs(xv + i + 3 * nthr);
    uint32_t ma = max_bf16x2(max_bf16x2(abs_bf16x2(a.x), abs_bf16x2(a.y)),
                             max_bf16x2(abs_bf16x2(a.z), abs_bf16x2(a.w)));
    uint32_t mb = max_bf16x2(max_bf16x2(abs_bf16x2(b.x), abs_bf16x2(b.y)),
                             max_bf16x2(abs_bf16x2(b.z), abs_bf16x2(b.w)));
    uint32_t mc = max_bf16x2(max_bf16x2(abs_bf16x2(c.x), abs_bf16x2(c.y)),
                             max_bf16x2(abs_bf16x2(c.z), abs_bf16x2(c.w)));
    uint32_t md = max_bf16x2(max_bf16x2(abs_bf16x2(d.x), abs_bf16x2(d.y)),
                             max_bf16x2(abs_bf16x2(d.z), abs_bf16x2(d.w)));
    m2 = max_bf16x2(m2, max_bf16x2(max_bf16x2(ma, mb), max_bf16x2(mc, md)));
  }
  for (; i < nvec; i += nthr) {
    uint4 a = __ldcs(xv + i);
    m2 = max_bf16x2(m2, max_bf16x2(max_bf16x2(abs_bf16x2(a.x), abs_bf16x2(a.y)),
                                   max_bf16x2(abs_bf16x2(a.z), abs_bf16x2(a.w))));
  }
  if (tid < head) m1 = x[tid] & 0x7FFFu;
  const int64_t tail0 = head + nvec * 8;
  if (tail0 + tid < n) {
    uint32_t e = x[tail0 + tid] & 0x7FFFu;
    m1 = e > m1 ? e : m1;
  }
  return max(max(m2 & 0xFFFFu, m2 >> 16), m1);
}

__global__ void __launch_bounds__(512)
global_scale_kernel(const uint16_t *__restrict__ x, int64_t n, float max_scale, float *g_out) {
  __shared__ uint32_t s_m[16];
  const uint32_t m = cta_max(thread_amax(x, n), s_m);
  if (threadIdx.x == 0 && m != 0) atomicMax(reinterpret_cast<int *>(g_out), __float_as_int(global_scale_of(m, max_scale)));
}

// The same reduction up to one value per CTA; the quantiser that follows finishes it (ScaleSource).
__global__ void __launch_bounds__(512)
amax_partial_kernel(const uint16_t *__restrict__ x, int64_t n, uint32_t *__restrict__ partial) {
  __shared__ uint32_t s_m[16];
  // in this order: a quantiser that is running has every CTA of this grid past its wait, so `x` is complete for it too
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t m = cta_max(thread_amax(x, n), s_m);
  if (threadIdx.x == 0) partial[blockIdx.x] = m;
}

}  // namespace ac4k

using namespace ac4k;

static int check_view(const int64_t shape[4], const int64_t stride[4]) {
  if (!shape || !stride) return fail(AC4K_ERR_NULL, "shape/stride is NULL");
  for (int i = 0; i < 4; ++i)
    if (shape[i] < 0) return fail(AC4K_ERR_SHAPE, "shape[%d] = %lld is negative", i, (long long)shape[i]);
  return 0;
}

extern "C" int ac4k_global_scale_bf16(const void *x, int64_t numel, float max_scale, float *g_out,
                                      ac4k_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!g_out) return fail(AC4K_ERR_NULL, "g_out is NULL");
  if (numel < 0) return fail(AC4K_ERR_SHAPE, "numel is negative");
  if (numel > 0 && !x) return fail(AC4K_ERR_NULL, "x is NULL");
  if (reinterpret_cast<uintptr_t>(x) & 1) return fail(AC4K_ERR_ALIGN, "x must be 2-byte aligned");
  if (!(max_scale > 0.0f)) return fail(AC4K_ERR_SHAPE, "max_scale must be positive");
  AC4K_CUDA_TRY(cudaMemsetAsync(g_out, 0, sizeof(float), stream));
  if (numel == 0) return 0;
  const int threads = 512;
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  int64_t blocks = ceil_div(ceil_div(numel, 8), (int64_t)threads * 4);
  if (blocks > (int64_t)di.sms * 4) blocks = (int64_t)di.sms * 4;     // four resident CTAs of 512 threads per SM
  if (blocks < 1) blocks = 1;
  global_scale_kernel<<<(unsigned)blocks, threads, 0, stream>>>(static_cast<const uint16_t *>(x), numel,
                                                               max_scale, g_out);
  AC4K_LAUNCH_CHECK("global_scale_kernel");
  return 0;
}

static int check_quantize(const void *out, const void *sf, const void *in, const int64_t shape[4], const int64_t stride[4], int sf_layout) {
  if (int e = check_view(shape, stride)) return e;
  if (!out || !sf) return fail(AC4K_ERR_NULL, "out/sf is NULL");
  if (sf_layout != AC4K_SF_AC4K && sf_layout != AC4K_SF_TILE128X4)
    return fail(AC4K_ERR_ENUM, "unknown sf_layout %d", sf_layout);
  const int64_t nbatch = shape[0] * shape[1];
  if (nbatch == 0 || shape[2] == 0 || shape[3] == 0) return 0;   // nothing to write (padding needs K > 0 rows)
  if (!in) return fail(AC4K_ERR_NULL, "in is NULL");
  if (nbatch > 65535) return fail(AC4K_ERR_SHAPE, "outer dims product %lld exceeds 65535", (long long)nbatch);
  if ((reinterpret_cast<uintptr_t>(out) & 7) || (reinterpret_cast<uintptr_t>(sf) & 3))
    return fail(AC4K_ERR_ALIGN, "out must be 8-byte and sf 4-byte aligned");
  return 0;
}

// rows contiguous along K in whole 16-byte pieces, no permutation: the tiled and flat kernels
static bool rows_vectorised(const void *in, const int64_t shape[4], const int64_t stride[4], int swizzle) {
  return !swizzle && stride[3] == 1 && (shape[3] % 16 == 0) && (stride[2] % 8 == 0) && (stride[0] % 8 == 0) && (stride[1] % 8 == 0) &&
         ((reinterpret_cast<uintptr_t>(in) & 15) == 0);
}

template <bool PARTIAL>
static int quantize_impl(void *out, void *sf, const void *in, const ScaleSource &src, const int64_t shape[4], const int64_t stride[4],
                         int swizzle, int sf_layout, cudaStream_t stream) {
  const int64_t d0 = shape[0], d1 = shape[1], M = shape[2], K = shape[3];
  const int64_t nbatch = d0 * d1;
  const int64_t Kp = align_up(K, 64);
  const uint16_t *inp = static_cast<const uint16_t *>(in);

  const bool vec_ok = rows_vectorised(in, shape, stride, swizzle);
  int rc = 0;
  if (vec_ok) {
    const bool wide = (stride[2] % 16 == 0) && (stride[0] % 16 == 0) && (stride[1] % 16 == 0) &&
                      ((reinterpret_cast<uintptr_t>(in) & 31) == 0);
    const int tile_k = Kp <= 128 ? 128 : 256;
    dim3 grid((unsigned)ceil_div(Kp, (int64_t)tile_k), (unsigned)ceil_div(M, kTileRows), (unsigned)nbatch);
    if (ceil_div(M, kTileRows) > 65535) return fail(AC4K_ERR_SHAPE, "M too large");
#define AC4K_LAUNCH_TILED(KERNEL, L, W)                                                           \
  rc = launch_kernel<PARTIAL>(KERNEL<L, W, PARTIAL>, grid, kThreads, 0, stream,                    \
                                 static_cast<uint8_t *>(out), static_cast<uint32_t *>(sf), inp, src, M, K, d1, \
                                 stride[0], stride[1], stride[2])
#define AC4K_LAUNCH_TILED_K(L, W)                                                                 \
  do { if (tile_k == 128) AC4K_LAUNCH_TILED(nvfp4_quantize_tiled128_kernel, L, W); else AC4K_LAUNCH_TILED(nvfp4_quantize_tiled_kernel, L, W); } while (0)
    if (sf_layout == AC4K_SF_AC4K) {
      if (wide) AC4K_LAUNCH_TILED_K(AC4K_SF_AC4K, true); else AC4K_LAUNCH_TILED_K(AC4K_SF_AC4K, false);
    } else {
      if (wide) AC4K_LAUNCH_TILED_K(AC4K_SF_TILE128X4, true); else AC4K_LAUNCH_TILED_K(AC4K_SF_TILE128X4, false);
    }
#undef AC4K_LAUNCH_TILED_K
#undef AC4K_LAUNCH_TILED
    return rc;
  }

  const int64_t rows_sf = (sf_layout == AC4K_SF_AC4K) ? align_up(M, 16) : align_up(M, 128);
  const bool row_fastest = stride[2] < stride[3];
  // rows contiguous along the cross dimension, K strided: the transposing kernel
  const bool tr_ok = stride[2] == 1 && M % 2 == 0 && stride[3] % 2 == 0 && stride[0] % 2 == 0 && stride[1] % 2 == 0 &&
                     ((reinterpret_cast<uintptr_t>(in) & 3) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) &&
                     ceil_div(M, 128) <= 65535;
  if (tr_ok) {
    dim3 g((unsigned)ceil_div(Kp, 128), (unsigned)ceil_div(M, 128), (unsigned)nbatch);
#define AC4K_LAUNCH_TR(L, P)                                                                                        \
  rc = launch_kernel<PARTIAL>(nvfp4_quantize_transposed_kernel<L, P, PARTIAL>, g, 256, 0, stream, static_cast<uint8_t *>(out), \
                                 static_cast<uint8_t *>(sf), inp, src, M, K, d1, stride[0], stride[1], stride[3])
    if (sf_layout == AC4K_SF_AC4K) {
      if (swizzle) AC4K_LAUNCH_TR(AC4K_SF_AC4K, true); else AC4K_LAUNCH_TR(AC4K_SF_AC4K, false);
    } else {
      if (swizzle) AC4K_LAUNCH_TR(AC4K_SF_TILE128X4, true); else AC4K_LAUNCH_TR(AC4K_SF_TILE128X4, false);
    }
#undef AC4K_LAUNCH_TR
    return rc;
  }
  dim3 grid;
  if (row_fastest)
    grid = dim3((unsigned)ceil_div(Kp / 16, 8), (unsigned)ceil_div(rows_sf, 32), (unsigned)nbatch);
  else
    grid = dim3((unsigned)ceil_div(Kp / 16, 32), (unsigned)ceil_div(rows_sf, 8), (unsigned)nbatch);
  if (grid.y > 65535) return fail(AC4K_ERR_SHAPE, "M too large for the strided path");
#define AC4K_LAUNCH_STRIDED(L, P, R)                                                             \
  rc = launch_kernel<PARTIAL>(nvfp4_quantize_strided_kernel<L, P, R, PARTIAL>, grid, 256, 0, stream, \
                                 static_cast<uint8_t *>(out), static_cast<uint8_t *>(sf), inp, src, M, K, d1, \
                                 stride[0], stride[1], stride[2], stride[3])
  const int sel = (sf_layout == AC4K_SF_TILE128X4 ? 4 : 0) | (swizzle ? 2 : 0) | (row_fastest ? 1 : 0);
  switch (sel) {
    case 0: AC4K_LAUNCH_STRIDED(AC4K_SF_AC4K, false, false); break;
    case 1: AC4K_LAUNCH_STRIDED(AC4K_SF_AC4K, false, true); break;
    case 2: AC4K_LAUNCH_STRIDED(AC4K_SF_AC4K, true, false); break;
    case 3: AC4K_LAUNCH_STRIDED(AC4K_SF_AC4K, true, true); break;
    case 4: AC4K_LAUNCH_STRIDED(AC4K_SF_TILE128X4, false, false); break;
    case 5: AC4K_LAUNCH_STRIDED(AC4K_SF_TILE128X4, false, true); break;
    case 6: AC4K_LAUNCH_STRIDED(AC4K_SF_TILE128X4, true, false); break;
    default: AC4K_LAUNCH_STRIDED(AC4K_SF_TILE128X4, true, true); break;
  }
#undef AC4K_LAUNCH_STRIDED
  return rc;
}

extern "C" int ac4k_quantize_nvfp4(void *out, void *sf, const void *in, const float *global_scale,
                                   const int64_t shape[4], const int64_t stride[4], int swizzle,
                                   int sf_layout, ac4k_stream_t stream) {
  if (!global_scale) return fail(AC4K_ERR_NULL, "global_scale is NULL");
  if (int e = check_quantize(out, sf, in, shape, stride, sf_layout)) return e;
  if (shape[0] * shape[1] == 0 || shape[2] == 0 || shape[3] == 0) return 0;
  const ScaleSource src{global_scale, nullptr, 0, 0.0f, nullptr, false};
  return quantize_impl<false>(out, sf, in, src, shape, stride, swizzle, sf_layout, static_cast<cudaStream_t>(stream));
}

// The flat kernel over one cluster: at most 8 CTAs of a block per thread (four blocks per thread were slower than two
// launches over the whole chip: 9.6 against 7.1 us for 50 x 8192)
static constexpr int kFlatThreads = 1024;
static_assert(AC4K_QUANTIZE_ONE_LAUNCH_BLOCKS == 8 * kFlatThreads, "one block per thread of the largest cluster");

template <int L>
static int launch_flat(void *out, void *sf, const void *in, const ScaleSource &src, const int64_t shape[4], const int64_t stride[4],
                       int64_t items, bool cluster, cudaStream_t stream) {
  const int64_t nbatch = shape[0] * shape[1];
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  uint8_t *o = static_cast<uint8_t *>(out);
  uint32_t *f = static_cast<uint32_t *>(sf);
  const uint16_t *x = static_cast<const uint16_t *>(in);
  if (cluster) {
    // as many CTAs as give a thread one block (or four padding words), up to eight
    const int64_t rows_sf = align_up(shape[2], L == AC4K_SF_AC4K ? 16 : 128);
    const int64_t work = items + nbatch * (rows_sf - shape[2]) * ceil_div(shape[3], 64) / 4;
    int ctas = 1;
    while (ctas < 8 && (int64_t)ctas * kFlatThreads < work) ctas *= 2;
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3((unsigned)(ctas == 1 ? align_up(work, 128) : kFlatThreads));
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ctas;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    AC4K_CUDA_TRY(cudaLaunchKernelEx(&cfg, nvfp4_quantize_flat_kernel<L, true, kFlatThreads>, o, f, x, src, (int)shape[2],
                                     (int)shape[3], (int)nbatch, (int)shape[1], stride[0], stride[1], stride[2]));
    return 0;
  }
  cfg.gridDim = dim3((unsigned)ceil_div(items, 256));
  cfg.blockDim = dim3(256);
  AC4K_CUDA_TRY(cudaLaunchKernelEx(&cfg, nvfp4_quantize_flat_kernel<L, false, 256>, o, f, x, src, (int)shape[2], (int)shape[3],
                                   (int)nbatch, (int)shape[1], stride[0], stride[1], stride[2]));
  return 0;
}

template <bool OVERLAP>
static int launch_reduction(unsigned blocks, const uint16_t *x, int64_t n, uint32_t *partial, cudaStream_t stream) {
  return launch_kernel<OVERLAP>(amax_partial_kernel, dim3(blocks), 512, 0, stream, x, n, partial);
}

// Whether the one-launch kernel of quantize_nvfp4_resident.cu is asked (it may still decline).  One launch / two, us, calls in a graph:
//   columns contiguous (attention's V): always.  V of [1, 16384, 16, 128] 26.7 / 50.6, [1, 75600, 40, 128] 297 / 450, [1, 1000, 16, 128]
//     5.1 / 12.7, [1, 104, 8, 128] 4.1 / 6.2; 16 keys, an eighth of a tile, [1, 16, 400, 128] 7.7 / 8.7; eight channels, [1, 1000, 16, 8] 4.9 / 6.9
//   rows, four to seven of its tiles an SM, or 2^24 to 2^25 elements.  1000 x 5120 7.2 / 9.4, 2048 x 4096 8.6 / 11.0, 4100 x 4096
//     15.9 / 22.6, 8192 x 4096 28.2 / 32.7.  Below, 666 x 4096 has the flat kernel (5.2; 800 x 4096 6.6 / 5.3).  Between and
//     above, one launch is the faster one too since its CTAs meet without a grid barrier (3000 x 4096 12.6 / 13.3, 4096 x 4096 15.1 / 16.2, 12000 x
//     4096 42.1 / 45.1): the lines are where they were drawn before that
//   and of these not where most of a tile would be padding: a tile has 128 rows of one matrix.  With a third of them used they are even
//     (64 matrices of 1024 columns, 48 rows 8.0 / 8.3, 32 rows 8.1 / 7.5, 16 rows 7.8 / 6.8; four rows of 4096 x 2048 553 / 215; one row of 2^25
//     2200 / 791), and from 36 tiles an SM on with three quarters (2048 columns, 65 rows: 28 tiles an SM 23.6 / 25.9, 43 33.3 / 32.9, 54 41.5 /
//     38.4; 1024 columns, 100 rows, 32 tiles 29.4 / 31.8).  Rows that the vectorised kernels do not take go through the strided one, which is
//     so much slower that only the first of the two lines counts (64 rows of 1032 columns, 29 tiles 23.5 / 41; 32 rows of 2056 39.3 / 37.3)
static bool takes_one_launch(const int64_t shape[4], const int64_t stride[4], int swizzle, bool vec, int sms) {
  if (swizzle || stride[3] != 1) return true;
  const int64_t M = shape[2], rows = align_up(M, 128), nbatch = shape[0] * shape[1], numel = nbatch * M * shape[3];
  const int64_t tiles = nbatch * (rows / 128) * ceil_div(shape[3], 64);
  if (rows > 3 * M) return false;
  if (tiles >= 4 * (int64_t)sms && tiles <= 7 * (int64_t)sms) return true;
  return numel > (1 << 24) && numel <= (1 << 25) && (!vec || 3 * rows <= 4 * M || tiles <= 36 * (int64_t)sms);
}
#ifdef AC4K_DEBUG_HOOKS
// the same for a 16-byte aligned tensor
extern "C" __attribute__((visibility("default"))) int ac4k_debug_takes_one_launch(const int64_t shape[4], const int64_t stride[4], int swizzle, int sms) {
  return takes_one_launch(shape, stride, swizzle, rows_vectorised(nullptr, shape, stride, swizzle), sms);
}
#endif

extern "C" int ac4k_quantize_nvfp4_dynamic(void *out, void *sf, float *g_out, void *scratch, const void *in, float max_scale,
                                           const int64_t shape[4], const int64_t stride[4], int swizzle, int sf_layout,
                                           ac4k_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!g_out) return fail(AC4K_ERR_NULL, "g_out is NULL");
  if (!(max_scale > 0.0f)) return fail(AC4K_ERR_SHAPE, "max_scale must be positive");
  if (int e = check_quantize(out, sf, in, shape, stride, sf_layout)) return e;
  const int64_t nbatch = shape[0] * shape[1], M = shape[2], K = shape[3];
  const int64_t numel = nbatch * M * K;
  if (numel == 0) return ac4k_global_scale_bf16(in, 0, max_scale, g_out, stream_);
  if (reinterpret_cast<uintptr_t>(in) & 1) return fail(AC4K_ERR_ALIGN, "in must be 2-byte aligned");
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  // Routes by size (measured on a B200; microseconds of the whole call on resident inputs stand beside the kernels):
  //   whole tensor in the registers of one cluster            one launch
  //   takes_one_launch(), which see                            the one-launch kernel of quantize_nvfp4_resident.cu
  //   up to 2^24 elements                                      maxima per CTA, then a quantiser that reduces them: two launches,
  //                                                            the second one set up under the first
  //   larger                                                   zeroed accumulator + atomic maximum + quantiser: a few hundred
  //                                                            words read by each of thousands of CTAs would cost more
  const bool vec = rows_vectorised(in, shape, stride, swizzle);
  const int64_t Kp = align_up(K, 64), items = nbatch * M * (Kp / 16);
  ScaleSource src{nullptr, nullptr, 0, max_scale, g_out, false};
  if (vec && items <= AC4K_QUANTIZE_ONE_LAUNCH_BLOCKS)
    return sf_layout == AC4K_SF_AC4K ? launch_flat<AC4K_SF_AC4K>(out, sf, in, src, shape, stride, items, true, stream)
                                     : launch_flat<AC4K_SF_TILE128X4>(out, sf, in, src, shape, stride, items, true, stream);
  if (scratch && takes_one_launch(shape, stride, swizzle, vec, di.sms)) {
    const int e = launch_quantize_resident(out, sf, g_out, scratch, in, max_scale, shape, stride, swizzle, sf_layout, stream);
    if (e != kResidentDeclined) return e;
  }
  if (!scratch || numel > (1 << 24)) {
    if (int e = ac4k_global_scale_bf16(in, numel, max_scale, g_out, stream_)) return e;
    src.g = g_out;
    // what the reduction read last is still in L2: begin there
    src.last_first = nbatch == 1;
    return quantize_impl<false>(out, sf, in, src, shape, stride, swizzle, sf_layout, stream);
  }
  // 128 x 256 tiles from one CTA per SM on; below that the flat kernel's 256 blocks per CTA fill the chip better.  Under the
  // flat one the reduction itself may start under the kernel before it (22.9 -> 21.3 us for quantise + GEMM at
  // 666 x 4096 x 4096); on larger tensors the three kernels then compete (55.8 -> 57.6 us at 4096^3).  Letting the GEMM start while the
  // reduction still waits, for the sake of its weight prefetch, costs 2.4 us at 50 x 8192 x 8192 and gains nothing at 1 row.
  const int64_t tiles = ceil_div(Kp, Kp <= 128 ? 128 : 256) * ceil_div(M, kTileRows) * nbatch;
  const bool flat = vec && tiles < di.sms;
  const int64_t blocks = std::min<int64_t>(std::min<int64_t>(ceil_div(ceil_div(numel, 8), 512 * 2), (int64_t)di.sms * 2), AC4K_QUANTIZE_SCRATCH_BYTES / 4);
  src.partial = static_cast<const uint32_t *>(scratch);
  src.n_partial = (int)blocks;
  auto *const launch_amax = flat ? &launch_reduction<true> : &launch_reduction<false>;
  if (int e = launch_amax((unsigned)blocks, static_cast<const uint16_t *>(in), numel, static_cast<uint32_t *>(scratch), stream)) return e;
  if (flat)
    return sf_layout == AC4K_SF_AC4K ? launch_flat<AC4K_SF_AC4K>(out, sf, in, src, shape, stride, items, false, stream)
                                     : launch_flat<AC4K_SF_TILE128X4>(out, sf, in, src, shape, stride, items, false, stream);
  return quantize_impl<true>(out, sf, in, src, shape, stride, swizzle, sf_layout, stream);
}
