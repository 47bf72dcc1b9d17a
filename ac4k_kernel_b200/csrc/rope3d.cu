// 3-D rotary position embedding for sm_100a: out[b, s, n, 2c : 2c + 2] = x[b, s, n, 2c : 2c + 2] * freq (complex), where
// position s of a [F, H, W] grid takes its C = D / 2 complex factors from three rows of one table: pairs [0, c1) from
// row f, [c1, c1 + c2) from row h, the rest from row w (c2 = C / 3, c1 = C - 2 c2).  Stands in for ac4k_kernel's
// lib/cuda/sm120/rope3d.cu:23-129 (kernel) and :133-187 (checks) behind the same binding (lib/cuda_bindings.cc:91-97).
//
// Arithmetic as in the reference: bf16 -> fp64, the four products and two sums in fp64 (no fused multiply-add), -> fp32
// -> bf16, so results equal the reference's Python oracle (test/test_rope_3d_apply.py:14-42) bit for bit.  One
// difference, deliberate: positions behind the grid (s >= F * H * W) are copied through, which is what that oracle
// returns; the reference's kernel leaves them unwritten.
//
// HBM-bound: 4 bytes of traffic per element.  The reference runs one thread per (position, head) row over 256-byte
// rows with scalar loads and re-reads 64 table entries per row; here one CTA walks whole positions (all heads, N * D
// contiguous elements) with 16-byte loads and stores, five of them in flight per thread, and a position's factors are
// fetched while its data are.  (Three dependent loads in a row, of the data one vector at a time, and four fp32 <-> fp64
// conversions a pair bounded the kernel before.)
#include <algorithm>
#include <climits>

#include "common.cuh"

namespace ac4k {

// MODE 0 (see the kernel), many positions: a warp per CTA where its lanes hold a head's factors (D <= 256), else four.
// [1, 75600, 40, 128], bit-identical, calls back to back: 386 us with 256 threads, one vector in flight and fp64 throughout; 322
// with five in flight; 298 with the fp32 form below in its present shape (128 threads); 262 with 64 threads; 252 with 32 (6.1
// TB/s; a call on inputs that are not the last call's takes 271, 5.7 TB/s).
static constexpr int kRopeWarpsPerSm = 24;   // 80 registers per thread
static constexpr int kRopeThreads = 256, kRopeCtasPerSm = 5;     // MODE 1 and 2
static constexpr int kRopeBatch = 5;         // vectors a thread has in flight
static constexpr int kRopeMaxC = 1024;      // complex pairs per head staged in shared memory (D <= 2048)

__device__ __forceinline__ uint32_t rope_pair(uint32_t xy, double2 f) {
  const double xr = (double)__uint_as_float(xy << 16), xi = (double)__uint_as_float(xy & 0xffff0000u);
  const double re = __dsub_rn(__dmul_rn(xr, f.x), __dmul_rn(xi, f.y));
  const double im = __dadd_rn(__dmul_rn(xr, f.y), __dmul_rn(xi, f.x));
  const __nv_bfloat162 o = __floats2bfloat162_rn((float)re, (float)im);
  return *reinterpret_cast<const uint32_t *>(&o);
}

// The same result, bit for bit, mostly without fp64 (whose conversions, 16 per clock and SM, four a pair, are most of what
// the fp64 form costs).  With factors rounded to fp32, t = fma(xr, fx, -RN(xi fy)) is off the exact value by at most
// 2^-24 (|xr fx| + 2 |xi fy| + |t|) (1 + 2^-22) for the factors, the product and the sum; the fp64 result is off by 2^-52 of the
// products.  So the fp64 result lies within t - e .. t + e with e = 2^-22 (|xr| + |xi|) max(|fx|, |fy|), at least a quarter more than
// that, and as rounding to fp32 and then to bf16 is monotonic, it ends on the bf16 value of both ends (themselves rounded
// to fp32) if they agree.  Where they do not (a few pairs in ten thousand: a rounding boundary lies between them), the vector
// is computed in fp64.  So it is where e is not between 2^-122 (lost bits of underflowing products stay far below it) and 2^100
// (nothing overflows), or is NaN.  A pair of zeros has e = 0 and is exact in fp32: it is accepted as it is (by way of fp64, behind
// the fp32 form, a tensor of zeros took 425 us where other values take 250, and 385 in fp64 alone; now 243).
struct RopeFactor { float x, y, e; };
__device__ __forceinline__ RopeFactor rope_factor(const double2 &f) {
  const float x = (float)f.x, y = (float)f.y, m = fmaxf(fabsf(x), fabsf(y));
  // NaN (always fp64) for factors that fp32 holds with fewer bits, infinite ones and NaN
  return {x, y, m >= 7.888609052210118e-31f ? fmaf(0.0f, x + y, m * 2.384185791015625e-7f) : __int_as_float(0x7fffffff)};
}
static constexpr uint32_t kRopeMinE = (127u - 122u) << 23, kRopeRangeE = 222u << 23;      // bits of 2^-122, up to 2^100

// one pair in fp32; diff and out_of_range collect what makes the result unusable
__device__ __forceinline__ uint32_t rope_pair_fast(uint32_t xy, const RopeFactor &f, uint32_t &diff, uint32_t &out_of_range) {
  const float xr = __uint_as_float(xy << 16), xi = __uint_as_float(xy & 0xffff0000u);
  const float re = __fmaf_rn(xr, f.x, -__fmul_rn(xi, f.y)), im = __fmaf_rn(xr, f.y, __fmul_rn(xi, f.x));
  const float a = __fadd_rn(fabsf(xr), fabsf(xi)), e = __fmul_rn(a, f.e);
  const __nv_bfloat162 lo = __floats2bfloat162_rn(__fsub_rn(re, e), __fsub_rn(im, e));
  const __nv_bfloat162 hi = __floats2bfloat162_rn(__fadd_rn(re, e), __fadd_rn(im, e));
  const uint32_t l = *reinterpret_cast<const uint32_t *>(&lo);
  if (a != 0.0f) {          // (a pair of zeros under a good factor is exact, the sign of its zeros included)
    diff |= l ^ *reinterpret_cast<const uint32_t *>(&hi);
    out_of_range = max(out_of_range, __float_as_uint(e) - kRopeMinE);
  }
  return l;
}

// not 0 if one of four factors is for fp64 alone
__device__ __forceinline__ uint32_t rope_unusable(const RopeFactor *ff) {
  const float s = (ff[0].e + ff[1].e) + (ff[2].e + ff[3].e);         // (positive or NaN)
  return s == s ? 0u : 0xffffffffu;
}
// eight elements (four pairs) of a vector; f(i): factor i in fp64
template <typename Exact>
__device__ __forceinline__ uint4 rope_vec(const uint4 &q, const RopeFactor *ff, uint32_t unusable, Exact &&f) {
  uint4 o;
  uint32_t diff = 0, range = unusable;
  o.x = rope_pair_fast(q.x, ff[0], diff, range);
  o.y = rope_pair_fast(q.y, ff[1], diff, range);
  o.z = rope_pair_fast(q.z, ff[2], diff, range);
  o.w = rope_pair_fast(q.w, ff[3], diff, range);
  if (diff != 0 || range >= kRopeRangeE) {
    o.x = rope_pair(q.x, f(0));
    o.y = rope_pair(q.y, f(1));
    o.z = rope_pair(q.z, f(2));
    o.w = rope_pair(q.w, f(3));
  }
  return o;
}

// row of the table that pair c of a position takes
__device__ __forceinline__ int rope_row(int c, int c1, int c2, int fi, int hi, int wi) { return c < c1 ? fi : (c < c1 + c2 ? hi : wi); }

// MODE 0: 16-byte accesses, the vectors of a position dealt to `active` threads, 4 * active a multiple of C, so that a
//         thread meets the same four pairs in each of its vectors: the position's factors live in registers, nothing is
//         shared, warps run free of one another.
// MODE 1: 16-byte accesses, the position's C factors staged in shared memory (two CTA barriers per position): D > 1024
//         (or, 32-bit counts exceeded, more than 2^33 elements per position).
// MODE 2: one pair per access (D % 8 != 0 or tensors not 16-byte aligned), factors in shared memory.
template <int MODE>
__global__ void __launch_bounds__(kRopeThreads, MODE == 0 ? kRopeWarpsPerSm * 32 / kRopeThreads : kRopeCtasPerSm) rope3d_kernel(const uint16_t *__restrict__ x, const int32_t *__restrict__ grid_sizes,
                                                               const double2 *__restrict__ freqs, uint16_t *__restrict__ out,
                                                               int64_t BS, int S, int N, int D, int C, int max_pos, int active) {
  __shared__ double2 sf[MODE == 0 ? 1 : kRopeMaxC];
  __shared__ RopeFactor sff[MODE == 1 ? kRopeMaxC : 1];          // the same rounded to fp32
  const int c2 = C / 3, c1 = C - 2 * c2;
  const int64_t row_elems = (int64_t)N * D;
  const int c0 = (int)((threadIdx.x * 4) % C);                  // MODE 0: this thread's four pairs
  if (MODE == 0 && (int)threadIdx.x >= active) return;          // (no barrier in this mode)
  // position ps = (b, pos), carried along without dividing again
  int b = (int)(blockIdx.x / (uint32_t)S), pos = (int)(blockIdx.x % (uint32_t)S);
  const int step_b = (int)(gridDim.x / (uint32_t)S), step_pos = (int)(gridDim.x % (uint32_t)S);
  auto advance = [&]() {
    b += step_b;
    if (pos >= S - step_pos) { pos -= S - step_pos; ++b; }
    else pos += step_pos;
  };
  for (int64_t ps = blockIdx.x; ps < BS; ps += gridDim.x, advance()) {
    const int F = __ldg(grid_sizes + 3 * b), H = __ldg(grid_sizes + 3 * b + 1), W = __ldg(grid_sizes + 3 * b + 2);
    const uint16_t *src = x + ps * row_elems;
    uint16_t *dst = out + ps * row_elems;
    const bool inside = (int64_t)pos < (int64_t)F * H * W;       // warp- and CTA-uniform
    // rows of the table for this position (an index past the table reads its last row instead of faulting)
    const int hw = max(H * W, 1), wd = max(W, 1);
    const int fi = min(pos / hw, max_pos - 1), hi = min((pos % hw) / wd, max_pos - 1), wi = min(pos % wd, max_pos - 1);
    if (MODE == 0) {
      // the position's first vectors are asked for before its factors
      const int nvec = (int)(row_elems / 8);
      const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
      uint4 *d4 = reinterpret_cast<uint4 *>(dst);
      uint4 q[kRopeBatch];
      auto load_batch = [&](int v0) {
#pragma unroll
        for (int u = 0; u < kRopeBatch; ++u) q[u] = v0 + u * active < nvec ? __ldcs(s4 + v0 + u * active) : make_uint4(0u, 0u, 0u, 0u);
      };
      load_batch(threadIdx.x);
      RopeFactor ff[4];
      uint32_t unusable = 0;
      auto exact = [&](int i) { return __ldg(freqs + (int64_t)rope_row(c0 + i, c1, c2, fi, hi, wi) * C + c0 + i); };
      if (inside) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ff[i] = rope_factor(exact(i));
        unusable = rope_unusable(ff);
      }
      for (int v0 = threadIdx.x; v0 < nvec; v0 += kRopeBatch * active) {
        if (v0 != (int)threadIdx.x) load_batch(v0);
#pragma unroll
        for (int u = 0; u < kRopeBatch; ++u) {
          const int v = v0 + u * active;
          if (v < nvec) __stcs(d4 + v, inside ? rope_vec(q[u], ff, unusable, exact) : q[u]);
        }
      }
      continue;
    }
    if (inside) {
      __syncthreads();                                            // the previous position's factors are no longer read
      for (int c = threadIdx.x; c < C; c += kRopeThreads) {
        const double2 f = __ldg(freqs + (int64_t)rope_row(c, c1, c2, fi, hi, wi) * C + c);
        sf[c] = f;
        if (MODE == 1) sff[c] = rope_factor(f);
      }
      __syncthreads();
    }
    if (MODE == 1) {
      const int64_t nvec = row_elems / 8;
      const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
      uint4 *d4 = reinterpret_cast<uint4 *>(dst);
      for (int64_t v = threadIdx.x; v < nvec; v += kRopeThreads) {
        uint4 q = __ldcs(s4 + v);
        if (inside) {
          const int cv = (int)((v * 4) % C);                      // first of this vector's four pairs
          q = rope_vec(q, sff + cv, rope_unusable(sff + cv), [&](int i) { return sf[cv + i]; });
        }
        __stcs(d4 + v, q);
      }
    } else {
      const int64_t npair = row_elems / 2;
      for (int64_t v = threadIdx.x; v < npair; v += kRopeThreads) {
        uint32_t q = (uint32_t)src[2 * v] | ((uint32_t)src[2 * v + 1] << 16);
        if (inside) q = rope_pair(q, sf[(int)(v % C)]);
        dst[2 * v] = (uint16_t)q;
        dst[2 * v + 1] = (uint16_t)(q >> 16);
      }
    }
  }
  grid_launch_dependents();
}

}  // namespace ac4k

using namespace ac4k;

extern "C" int ac4k_rope3d(void *out, const void *x, const int32_t *grid_sizes, const void *freqs, int64_t B, int64_t S,
                           int64_t N, int64_t D, int64_t max_pos, ac4k_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (B < 0 || S < 0 || N < 0 || D < 0 || max_pos < 0) return fail(AC4K_ERR_SHAPE, "negative dimension");
  if (D % 2) return fail(AC4K_ERR_SHAPE, "the feature dimension must be even (complex pairs), got %lld", (long long)D);
  if (B == 0 || S == 0 || N == 0 || D == 0) return 0;
  if (!out || !x || !grid_sizes || !freqs) return fail(AC4K_ERR_NULL, "a required pointer is NULL");
  if (max_pos == 0) return fail(AC4K_ERR_SHAPE, "the frequency table is empty");
  if (D / 2 > kRopeMaxC) return fail(AC4K_ERR_UNSUPPORTED, "feature dimensions up to %d are built, got %lld", 2 * kRopeMaxC, (long long)D);
  if (S > INT32_MAX || N > INT32_MAX || max_pos > INT32_MAX || B > INT32_MAX) return fail(AC4K_ERR_SHAPE, "dimension too large");
  if ((reinterpret_cast<uintptr_t>(out) & 1) || (reinterpret_cast<uintptr_t>(x) & 1) || (reinterpret_cast<uintptr_t>(grid_sizes) & 3) ||
      (reinterpret_cast<uintptr_t>(freqs) & 15))
    return fail(AC4K_ERR_ALIGN, "x/out must be 2-byte, grid_sizes 4-byte and freqs 16-byte aligned");
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  const int64_t BS = B * S;
  const bool vec = (D % 8 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
  // Threads of a multiple of C / 4 vectors (D % 8 == 0), so that their pairs repeat.  As few as hold them, one warp or four, where
  // there are positions enough for every SM's warps; else more, as long as a position has a vector for each.  (One warp a
  // position alone, of 128 heads x 256: 23.5 us for 100 positions and 39.6 for 1000; 7.8 and 30.2 with 256 threads always; 6.2
  // and 27.0 by this rule.)
  const int64_t round = D / 8, nvec = N * D / 8;
  int threads0 = round <= 32 ? 32 : 128;
  while (threads0 < kRopeThreads && threads0 < nvec && BS * (threads0 / 32) < (int64_t)di.sms * kRopeWarpsPerSm) threads0 *= 2;
  const int active = vec && round <= threads0 ? (int)(threads0 / round * round) : 0;
  const int mode = !vec ? 2 : (active && nvec < (1 << 30) ? 0 : 1);
  const int threads = mode == 0 ? threads0 : kRopeThreads;
  const unsigned blocks = (unsigned)std::min<int64_t>(BS, (int64_t)di.sms * (mode == 0 ? kRopeWarpsPerSm * 32 / threads0 : kRopeCtasPerSm));
  const uint16_t *xp = static_cast<const uint16_t *>(x);
  uint16_t *op = static_cast<uint16_t *>(out);
  const double2 *fp = static_cast<const double2 *>(freqs);
  if (mode == 0)
    rope3d_kernel<0><<<blocks, threads, 0, stream>>>(xp, grid_sizes, fp, op, BS, (int)S, (int)N, (int)D, (int)(D / 2), (int)max_pos, active);
  else if (mode == 1)
    rope3d_kernel<1><<<blocks, threads, 0, stream>>>(xp, grid_sizes, fp, op, BS, (int)S, (int)N, (int)D, (int)(D / 2), (int)max_pos, active);
  else
    rope3d_kernel<2><<<blocks, threads, 0, stream>>>(xp, grid_sizes, fp, op, BS, (int)S, (int)N, (int)D, (int)(D / 2), (int)max_pos, active);
  AC4K_LAUNCH_CHECK("rope3d_kernel");
  return 0;
}
