// BF16 -> NVFP4 with the tensor's own global scale in ONE launch: a cooperative grid of one CTA per SM reduces the tensor to its
// maximum, meets (see below), and quantises.  The tiles that a CTA read last are still in its shared memory then (up to 224 KB
// an SM, 33 MB of the chip), so a tensor of at most that size is read from memory once; of a larger one the rest is read again from
// the end backwards, while the L2 still has what was read last.  Same bits as the two-launch route of quantize_nvfp4.cu (same
// arithmetic; also of a block with a NaN, which is left out of the block's maximum by the kernels for rows of whole blocks, and wins it in the
// others: kRowsAnyK, for a K that is no multiple of 16, and the transposed forms).
// What bounds it: latency.  16 warps an SM (shared memory leaves room for no more) issue 200 thread-instructions per block of 16 in the rows
// form, 172 in the transposed ones, 44 % and 39 % of the issue slots, at 2.3 TB/s; the rest is waits for loads, for the meeting and in the
// chain from a block's words to its codes.  Which sizes take it stands at takes_one_launch() in quantize_nvfp4.cu, with the times of both routes.
//
// A tile is 16 KB, one TMA box with the 128-byte swizzle: 128 rows x 64 K-elements of a tensor whose rows are contiguous along K
// (kRows), or 128 K-elements x 64 rows of one that is contiguous along the rows (kTransposed, kTransposedPermuted: attention's V).
// 16 consumer warps in teams; a team takes every n-th tile of the CTA's contiguous share.  kRows: one team, a thread has one
// 16-element block of the tile, four lanes a row, and conflict-free 16-byte reads.  Transposed: teams of four warps, a thread has two
// rows x 32 K-elements (a warp reads 32 words of one 128-byte line at a time), and the scale bytes meet in shared memory.
//
// The meeting.  Every CTA of a tensor leaves its maximum in a word of its own, {48-bit tag of the launch, maximum}; CTA 0 waits for all
// of them and answers each CTA in a second word of that CTA, with the maximum of all or, where one did not come within the launch's
// limit or gave up on a load, with kNoMaximum; the others wait for that answer, for twice as long.  The words are in the call's scratch,
// whose contents are undefined: a tag is not repeated in a process and starts at a random number, so that a word that has not been written
// yet does not have it (2^-48).  A captured launch is replayed with the same tag, so no word may keep it: each has one reader, which clears
// it, and a CTA without an answer clears what it left itself.  (All CTAs polling all words took 2 - 3 us longer, 148 readers on the same
// ten lines: V of [1, 1000, 16, 128] 9.8 us for 5.1.)
// That all CTAs of the grid are on the chip together is what a cooperative launch promises (it fails otherwise).  Programmatic
// serialisation does not take that away: it lets the grid begin when every CTA of the kernel in front has begun, and those wait for
// nothing of this one.
#include <algorithm>
#include <atomic>
#include <random>

#include "gemm_common.cuh"

namespace ac4k {
using namespace ptx;

namespace resident {
enum { kRows = 0, kTransposed = 1, kTransposedPermuted = 2, kRowsAnyK = 3 };
constexpr bool is_rows(int mode) { return mode == kRows || mode == kRowsAnyK; }
static constexpr int kTileBytes = 128 * 128;
static constexpr int kWarps = 16, kThreads = 32 * (kWarps + 1);      // consumers and one producer warp
static constexpr int kMaxSlots = 14;
// beside the slots: reciprocal table, two words per warp, barriers, scale words of the transposed form (two buffers a team)
static constexpr int kMiscBytes = 128 * 4 + 2 * 32 * 4 + 2 * kMaxSlots * 8, kScaleBytes = 4 * 2 * 128 * 4;
static constexpr uint32_t kNoMaximum = 0xFFFF;        // |x| of bf16 has 15 bits
// a meeting's place in scratch: a maximum and an answer per CTA
constexpr int64_t meeting_words(int64_t ctas) { return 2 * ctas; }
constexpr int teams(int mode) { return is_rows(mode) ? 1 : 4; }
// a slot that is used again belongs to one team (its barriers' parities would be ambiguous to a team that skips a use)
constexpr int max_slots(int mode) { return is_rows(mode) ? kMaxSlots : 12; }
constexpr int smem_bytes(int mode, int slots) { return 1024 + slots * kTileBytes + kMiscBytes + (is_rows(mode) ? 0 : kScaleBytes); }
static_assert(smem_bytes(kRows, max_slots(kRows)) <= 227 * 1024 && smem_bytes(kTransposed, max_slots(kTransposed)) <= 227 * 1024, "shared memory overflow");
static_assert(kWarps < 32, "a lane per warp's maximum");
static_assert(max_slots(kTransposed) % teams(kTransposed) == 0, "a slot belongs to one team");
}  // namespace resident

struct ResidentArgs {
  uint8_t *out;
  uint8_t *sf;
  unsigned long long *maxima, *answers;  // the meeting: one word of each per CTA
  unsigned long long tag;                // 48 bits, not 0
  float *g_out;
  float max_scale;
  int M, K, d1;
  int n_fast, n_mid;       // tiles along the tile order's first and second dimension
  int tiles, slots;
  unsigned int *status;
  unsigned long long wait_ns;            // limit of a wait for a load; CTA 0 waits twice as long for the others' maxima, they four times for its answer
  int dbg;                               // experiment switches (builds with -DAC4K_DEBUG_HOOKS), else 0
};

__device__ __forceinline__ uint4 ld_shared_v4u(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cta.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
// max(|a|, |b|) of two packed pairs, of some sign
__device__ __forceinline__ uint32_t maxabs_bf16x2(uint32_t a, uint32_t b) {
  uint32_t m;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(b));
  return m;
}
__device__ __forceinline__ uint32_t amax_bf16x2(const uint4 &a, const uint4 &b) {
  return abs_bf16x2(maxabs_bf16x2(maxabs_bf16x2(maxabs_bf16x2(a.x, a.y), maxabs_bf16x2(a.z, a.w)),
                                  maxabs_bf16x2(maxabs_bf16x2(b.x, b.y), maxabs_bf16x2(b.z, b.w))));
}
// the same with a NaN above every number: the maximum of the bits
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t m;
  asm("max.u16x2 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(b));
  return m;
}
__device__ __forceinline__ uint32_t amax_bits(const uint4 &a, const uint4 &b) {
  return max_u16x2(max_u16x2(max_u16x2(abs_bf16x2(a.x), abs_bf16x2(a.y)), max_u16x2(abs_bf16x2(a.z), abs_bf16x2(a.w))),
                   max_u16x2(max_u16x2(abs_bf16x2(b.x), abs_bf16x2(b.y)), max_u16x2(abs_bf16x2(b.z), abs_bf16x2(b.w))));
}
// e4m3 scale byte of a block, and the multiplier of its elements
__device__ __forceinline__ uint32_t block_scale_of(float amax, float alpha, const float *s_rcp, float &r) {
  const float s = __fmul_rn(alpha, __fmul_rn(amax, kOneSixth));
  uint16_t pk;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pk) : "f"(0.0f), "f"(s));
  const uint32_t sb = pk & 0x7Fu;
  r = __fmul_rn(alpha, s_rcp[sb]);
  return sb;
}

// Waits for a word with `tag`, clears it, and gives its low 16 bits; false, and `value` left alone, where it did not come within the limit
__device__ __forceinline__ bool wait_tagged(unsigned long long *word, unsigned long long tag, unsigned long long limit_ns, uint32_t &value) {
  unsigned long long w, t0 = 0;
  for (int k = 0; (w = ld_relaxed_gpu_u64(word)) >> 16 != tag; ++k) {
    if (k & 63) continue;
    const unsigned long long now = globaltimer();
    if (k == 0) t0 = now;
    else if (now - t0 > limit_ns) return false;
  }
  st_relaxed_gpu_u64(word, 0);
  value = (uint32_t)w & 0xFFFFu;
  return true;
}

// The way out of a wait that expired: the CTA's copies in flight get another limit to land in, before its shared memory is given back.
// (Waiting for each of them on its barrier, by any count of what was issued, cost 2 - 4 % of every call: 4100 x 4096 15.9 -> 16.6 us.)
__device__ __forceinline__ void land_copies(unsigned long long limit_ns) {
  for (const unsigned long long t0 = globaltimer(); globaltimer() - t0 < limit_ns;) {}
}

// One tensor by `ctas` CTAs of the grid, of which this is number `cta`; false where a wait expired.
template <int SF_LAYOUT, int MODE>
__device__ __forceinline__ bool resident_quantize(const CUtensorMap &tma, const ResidentArgs &p, int cta, int ctas) {
  using namespace resident;
  constexpr int TEAMS = teams(MODE), TEAM_WARPS = kWarps / TEAMS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t tiles_s = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *misc = smem_raw + (tiles_s - smem_u32(smem_raw)) + p.slots * kTileBytes;
  float *s_rcp = reinterpret_cast<float *>(misc);
  uint32_t *s_m = reinterpret_cast<uint32_t *>(misc + 512), *s_all = s_m + 32;
  const uint32_t full = smem_u32(misc + 768), empty = full + 8 * kMaxSlots;
  uint32_t *s_sf = reinterpret_cast<uint32_t *>(misc + kMiscBytes);       // transposed: [team][buffer][K = 64 step][64 rows]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.slots;
  const int first = (int)((int64_t)cta * p.tiles / ctas);
  const int n = (int)((int64_t)(cta + 1) * p.tiles / ctas) - first;

  if (threadIdx.x < 128) {
    // 1 / float(e4m3 byte), correctly rounded; entry 0 is 0 so that a zero scale zeroes the block
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)threadIdx.x, __NV_E4M3);
    s_rcp[threadIdx.x] = threadIdx.x ? __frcp_rn(__half2float(__half(h))) : 0.0f;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, TEAM_WARPS);
    }
    fence_barrier_init();
    prefetch_tmap(&tma);
  }
  __syncthreads();
  grid_dependency_wait();
  grid_launch_dependents();

  // Tiles 0 .. n - 1 go through the slots in turn; the second phase takes the tiles from the last to the first and the slots in turn
  // the other way round, so that the last S tiles are where it looks for them.  Use number u of a slot waits for `full` phase u and
  // ends with `empty` phase u.
  const int s_last = (n - 1) % S, u_last = (n - 1) / S;      // slot and use of the last tile
  // (coordinates are counted, not divided out for each tile: five divisions a tile took longer than its quantisation)
  struct Tile {
    int fast, mid, b;
    __device__ Tile(int t, const ResidentArgs &p) : fast(t % p.n_fast), mid(t / p.n_fast % p.n_mid), b(t / p.n_fast / p.n_mid) {}
    __device__ void next(const ResidentArgs &p) {
      if (++fast == p.n_fast) { fast = 0; if (++mid == p.n_mid) { mid = 0; ++b; } }
    }
    __device__ void back(const ResidentArgs &p) {
      if (--fast < 0) { fast = p.n_fast - 1; if (--mid < 0) { mid = p.n_mid - 1; --b; } }
    }
  };
  auto issue = [&](uint32_t el, const Tile &t, int s) {
    mbar_arrive_expect_tx_if(el, full + 8 * s, kTileBytes);
    if (el) tma_load_4d(tiles_s + s * kTileBytes, &tma, t.fast * 64, t.mid * 128, t.b % p.d1, t.b / p.d1, full + 8 * s);
  };
  bool ok = true;
  uint32_t m2 = 0;
  const int team = warp / TEAM_WARPS, tt = threadIdx.x % (32 * TEAM_WARPS);      // team, thread of the team
  if (warp == kWarps) {
    const uint32_t el = elect_one();
    Tile t(first, p);
    if (AC4K_DBG(p, 0x800) && cta == ctas - 1)
      for (const unsigned long long t0 = globaltimer(); globaltimer() - t0 < p.wait_ns + p.wait_ns / 2;) {}
    for (int i = 0, s = 0, u = 0; i < n && ok; ++i) {
      if (u > 0) ok = warp_all(mbar_wait(empty + 8 * s, (u - 1) & 1, p.wait_ns));
      if (ok) issue(el, t, s);
      t.next(p);
      if (++s == S) { s = 0; ++u; }
    }
  } else {
    for (int i = team, s = team, u = 0; i < n; i += TEAMS) {
      if (s >= S) { s -= S; ++u; }
      ok = warp_all(mbar_wait(full + 8 * s, u & 1, p.wait_ns));
      if (!ok) break;
#pragma unroll
      for (int c = 0; c < TEAMS; ++c) {
        const uint32_t at = tiles_s + s * kTileBytes + (uint32_t)(c * 32 * TEAM_WARPS + tt) * 16;
        m2 = max_bf16x2(m2, amax_bf16x2(ld_shared_v4u(at), ld_shared_v4u(at + kTileBytes / 2)));      // (m2 >= 0 first: NaNs drop out)
      }
      if (i < n - S) {
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * s);
      }
      s += TEAMS;
    }
  }
  // the maximum over the CTA, then over the CTAs of the tensor
  {
    uint32_t m = __reduce_max_sync(0xFFFFFFFFu, max(m2 & 0xFFFFu, m2 >> 16));
    // (a warp that gave up has not seen every tile: what the CTA leaves is not a maximum then, and no CTA goes on)
    if (!ok && lane == 0) atomicExch(p.status, warp == kWarps ? kStatusTimeoutProducer : kStatusTimeoutEpilogue);
    if (lane == 0) s_m[warp] = ok ? m : kNoMaximum;
    __syncthreads();
    if (warp == 0) {
      m = __reduce_max_sync(0xFFFFFFFFu, lane <= kWarps ? s_m[lane] : 0u);
      if (lane == 0) s_all[kWarps] = m;
      if (lane == 0 && cta != 0 && !(AC4K_DBG(p, 0x400) && cta == ctas - 1)) st_relaxed_gpu_u64(p.maxima + cta, p.tag << 16 | m);
    }
    __syncwarp();
  }
  uint32_t m = kNoMaximum;
  if (cta == 0) {
    bool all = true;
    uint32_t mine = 0;
    if (warp < kWarps)
      for (int i = 1 + threadIdx.x; i < ctas; i += 32 * kWarps) {
        uint32_t other;
        if (wait_tagged(p.maxima + i, p.tag, 2 * p.wait_ns, other)) mine = max(mine, other);
        else all = false;
      }
    mine = __reduce_max_sync(0xFFFFFFFFu, mine);
    if (lane == 0 && warp < kWarps) s_all[warp] = mine;
    if (!all) atomicExch(p.status, kStatusTimeoutGrid);
    all = !__syncthreads_or(!all);
    if (all) m = __reduce_max_sync(0xFFFFFFFFu, lane <= kWarps ? s_all[lane] : 0u);
    for (int i = 1 + threadIdx.x; i < ctas; i += kThreads) st_relaxed_gpu_u64(p.answers + i, p.tag << 16 | m);
  } else {
    if (threadIdx.x == 0) {
      if (!wait_tagged(p.answers + cta, p.tag, 4 * p.wait_ns, m)) atomicExch(p.status, kStatusTimeoutGrid);
      if (m == kNoMaximum) st_relaxed_gpu_u64(p.maxima + cta, 0);
      s_all[0] = m;
    }
    __syncthreads();
    m = s_all[0];
  }
  if (m == kNoMaximum) return false;
  if (warp == kWarps) {
    const uint32_t el = elect_one();
    if (n > S) {
      Tile t(first + n - 1 - S, p);
      for (int q = S, s = s_last, u = u_last; q < n && ok; ++q) {      // the load behind use u of slot s
        ok = warp_all(mbar_wait(empty + 8 * s, u & 1, p.wait_ns));
        if (ok) issue(el, t, s);
        t.back(p);
        // from the last tile's slot on, each slot's use is one less below the wrap, and one more a round later
        if (--s < 0) { s = S - 1; --u; }
        if (s == s_last) u += 2;
      }
    }
    if (!ok && lane == 0) atomicExch(p.status, kStatusTimeoutProducer);
    return ok;
  }
  const float g = global_scale_of(m, p.max_scale), alpha = alpha_of(g);
  if ((cta | threadIdx.x) == 0) *p.g_out = g;

  const int Kp = (p.K + 63) / 64 * 64, KT = Kp / 64;
  const int rows_sf = SF_LAYOUT == AC4K_SF_AC4K ? (p.M + 15) / 16 * 16 : (p.M + 127) / 128 * 128;
  auto sf_word = [&](int b, int row, int k64) -> int64_t {
    if (SF_LAYOUT == AC4K_SF_AC4K) return ((int64_t)b * KT + k64) * rows_sf + row;
    return (((int64_t)b * (rows_sf >> 7) + (row >> 7)) * KT + k64) * 128 + (row & 31) * 4 + ((row & 127) >> 5);
  };
  uint32_t *sf_w = reinterpret_cast<uint32_t *>(p.sf);
  if (is_rows(MODE)) {
    // Four lanes have the blocks of one row and K = 64 step.  A warp's eight rows are those whose scale words are neighbours in
    // the layout (a whole 32-byte sector); rows of neighbouring lanes differ in their swizzle, so that eight lanes read eight
    // different 16-byte columns of shared memory.
    const int j = lane >> 2, blk = lane & 3;
    const int row_l = SF_LAYOUT == AC4K_SF_AC4K ? warp * 8 + j : (j >> 1) * 32 + 2 * warp + (j & 1);
    const uint32_t at0 = tiles_s + row_l * 128 + (((2 * blk) ^ (row_l & 7)) << 4), at1 = tiles_s + row_l * 128 + (((2 * blk + 1) ^ (row_l & 7)) << 4);
    // (several tiles side by side in one thread, to fill the chain from a block's words to its codes, gained nothing where the tiles
    // are there already and took half as long again where they are loaded again: 8192 x 8192 86 us against 57)
    Tile t(first + n - 1, p);
    for (int q = 0, s = s_last, u = u_last; q < n; ++q) {
      ok = warp_all(mbar_wait(full + 8 * s, u & 1, p.wait_ns));
      if (!ok) break;
      const uint4 v0 = ld_shared_v4u(at0 + s * kTileBytes), v1 = ld_shared_v4u(at1 + s * kTileBytes);
      if (n > S) {
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * s);
      }
      const int row = t.mid * 128 + row_l;
      float r;
      const uint32_t sb = block_scale_of(hmax_bf16x2_to_f32(MODE == kRows ? amax_bf16x2(v0, v1) : amax_bits(v0, v1)), alpha, s_rcp, r);
      uint32_t word = row < p.M ? sb << (8 * blk) : 0u;
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
      if (row < p.M)
        __stcs(reinterpret_cast<uint2 *>(p.out + ((int64_t)t.b * p.M + row) * (Kp / 2) + t.fast * 32 + blk * 8),
               make_uint2(quantize8_x2(v0.x, v0.y, v0.z, v0.w, r), quantize8_x2(v1.x, v1.y, v1.z, v1.w, r)));
      if (blk == 0 && row < rows_sf) sf_w[sf_word(t.b, row, t.fast)] = word;
      t.back(p);
      if (--s < 0) { s = S - 1; --u; }
      if (s == s_last) u += 2;
    }
  } else {
    const int g32 = tt >> 5;                               // 32 K-elements of the tile; the lane: rows 2 lane, 2 lane + 1
    uint32_t buf = 0;
    Tile t(first + n - 1, p);
    for (int q = 0, s = s_last, u = u_last; q < n; ++q, t.back(p), s == 0 ? (s = S - 1, --u) : --s, u += s == s_last ? 2 : 0) {
      if ((n - 1 - q) % TEAMS != team) continue;
      // (a warp whose wait ran out goes on, so that its team does not hang at the barrier below)
      if (ok) ok = warp_all(mbar_wait(full + 8 * s, u & 1, p.wait_ns));
      uint32_t w[32];                                      // element j of row 2 lane (low half) and of row 2 lane + 1 (high half)
#pragma unroll
      for (int j = 0; j < 32; ++j)
        w[j] = ld_shared_u32(tiles_s + s * kTileBytes + (g32 * 32 + j) * 128 + (((lane >> 2) ^ (j & 7)) << 4) + (lane & 3) * 4);
      if (n > S) {
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * s);
      }
      const int mt = t.fast, kt = t.mid, b = t.b;
      const int row = mt * 64 + 2 * lane, k0 = kt * 128 + 32 * g32;
      uint32_t *sf_t = s_sf + (team * 2 + buf) * 128;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t pr[16];                                   // pairs of consecutive elements, in output order
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int at = MODE == kTransposedPermuted ? 8 * (((2 * j) & 7) >> 1) + 2 * ((2 * j) >> 3) : 2 * j;
          pr[j] = __byte_perm(w[at], w[at + 1], e == 0 ? 0x5410 : 0x7632);
        }
        uint32_t bytes = 0, cw[4];
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const uint32_t *v = pr + 8 * blk;
          float r;
          bytes |= block_scale_of(hmax_bf16x2_to_f32(amax_bits(make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]))), alpha, s_rcp, r) << (8 * blk);
          cw[2 * blk] = quantize8_x2(v[0], v[1], v[2], v[3], r);
          cw[2 * blk + 1] = quantize8_x2(v[4], v[5], v[6], v[7], r);
        }
        const bool live = row + e < p.M;
        if (live && k0 < Kp)
          __stcs(reinterpret_cast<uint4 *>(p.out + ((int64_t)b * p.M + row + e) * (Kp / 2) + k0 / 2), make_uint4(cw[0], cw[1], cw[2], cw[3]));
        reinterpret_cast<uint16_t *>(sf_t + (g32 >> 1) * 64 + 2 * lane + e)[g32 & 1] = (uint16_t)(live ? bytes : 0u);
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
      const int row_o = mt * 64 + (tt & 63), k64 = kt * 2 + (tt >> 6);
      if (row_o < rows_sf && k64 < KT) sf_w[sf_word(b, row_o, k64)] = sf_t[tt];
      buf ^= 1;                                            // (the other buffer's words were read before this barrier)
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, kStatusTimeoutEpilogue);
  return ok;
}

template <int SF_LAYOUT, int MODE>
__global__ void __launch_bounds__(resident::kThreads, 1)
nvfp4_quantize_resident_kernel(const __grid_constant__ CUtensorMap tma, const ResidentArgs p) {
  if (!resident_quantize<SF_LAYOUT, MODE>(tma, p, blockIdx.x, gridDim.x)) land_copies(p.wait_ns);
}
// q, k and v of the attention operator, each with a share of the grid and a meeting of its own, in one launch.
template <int SF_LAYOUT, int ROWS>
__global__ void __launch_bounds__(resident::kThreads, 1)
nvfp4_quantize_attention_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                                const __grid_constant__ CUtensorMap tma_v, const ResidentArgs q, const ResidentArgs k, const ResidentArgs v,
                                int ctas_q, int ctas_k) {
  const int cta = blockIdx.x;
  bool ok;
  if (cta < ctas_q) ok = resident_quantize<SF_LAYOUT, ROWS>(tma_q, q, cta, ctas_q);
  else if (cta < ctas_q + ctas_k) ok = resident_quantize<SF_LAYOUT, ROWS>(tma_k, k, cta - ctas_q, ctas_k);
  else ok = resident_quantize<SF_LAYOUT, resident::kTransposedPermuted>(tma_v, v, cta - ctas_q - ctas_k, (int)gridDim.x - ctas_q - ctas_k);
  if (!ok) land_copies(q.wait_ns);
}

// 48 bits, not 0, not repeated within 2^48 launches of the process
static unsigned long long next_tag() {
  static std::atomic<unsigned long long> next = [] {
    try {
      std::random_device rd;
      return (unsigned long long)rd() << 32 | rd();
    } catch (...) {      // (no source of random numbers)
      return (unsigned long long)reinterpret_cast<uintptr_t>(&next_tag) * 0x9E3779B97F4A7C15ull;
    }
  }();
  for (;;)
    if (const unsigned long long t = next.fetch_add(1, std::memory_order_relaxed) & 0xFFFFFFFFFFFFull) return t;
}

// The place of the next `ctas` CTAs' meeting behind `at`
static void set_meeting(ResidentArgs *a, unsigned long long *&at, int64_t ctas) {
  a->maxima = at;
  a->answers = at + ctas;
  a->tag = next_tag();
  at += resident::meeting_words(ctas);
}
static unsigned long long *first_word(void *scratch) { return reinterpret_cast<unsigned long long *>((reinterpret_cast<uintptr_t>(scratch) + 7) & ~(uintptr_t)7); }
// at most one CTA per SM, behind up to 4 bytes in front of the first word
static bool meetings_fit(int sms) { return 8 * resident::meeting_words(sms) + 4 <= AC4K_QUANTIZE_SCRATCH_BYTES; }

#ifdef AC4K_DEBUG_HOOKS
static std::atomic<int> g_one_launches{0};      // what launch_cooperative launched so far, so that a test can say which route a call took
extern "C" __attribute__((visibility("default"))) int ac4k_debug_one_launches() { return g_one_launches.load(); }
#endif

// Cooperative, and beside the tail of the kernel in front of it; kResidentDeclined where the grid does not fit at once (a context with
// fewer SMs than the device).
template <typename... KArgs, typename... Args>
static int launch_cooperative(void (*kern)(KArgs...), int grid, size_t smem, cudaStream_t stream, const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(resident::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return kResidentDeclined;
  }
  AC4K_CUDA_TRY(e);
#ifdef AC4K_DEBUG_HOOKS
  ++g_one_launches;
#endif
  return 0;
}

template <int SF_LAYOUT, int MODE>
static int launch_resident(const CUtensorMap &tm, ResidentArgs a, void *scratch, int sms, cudaStream_t stream) {
  using namespace resident;
  auto kern = nvfp4_quantize_resident_kernel<SF_LAYOUT, MODE>;
  static PerDevice<int> attr_set;
  int unused = 0;
  if (int e = attr_set.get(&unused, [&](int &v) {
        AC4K_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MODE, max_slots(MODE))));
        v = 1;
        return 0;
      }))
    return e;
  const int grid = std::min(a.tiles, sms);
  unsigned long long *at = first_word(scratch);
  set_meeting(&a, at, grid);
  a.slots = std::min((int)ceil_div(a.tiles, grid), max_slots(MODE));
  return launch_cooperative(kern, grid, smem_bytes(MODE, a.slots), stream, tm, a);
}

// Tensor map and arguments for one tensor; kResidentDeclined where no map can have its strides.
static int resident_plan(void *out, void *sf, float *g_out, const void *in, float max_scale, const int64_t shape[4],
                         const int64_t stride[4], int swizzle, int sf_layout, int *mode, CUtensorMap *tm, ResidentArgs *a) {
  using namespace resident;
  const int64_t nbatch = shape[0] * shape[1], M = shape[2], K = shape[3], Kp = align_up(K, 64);
  int64_t dims[4] = {shape[0], shape[1], M, K}, strides[4] = {stride[0], stride[1], stride[2], stride[3]};
  int64_t n_fast, n_mid;
  if (!swizzle && stride[3] == 1) {
    *mode = K % 16 ? kRowsAnyK : kRows;
    n_fast = Kp / 64;
    n_mid = ceil_div(M, 128);
  } else if (stride[2] == 1) {
    *mode = swizzle ? kTransposedPermuted : kTransposed;
    std::swap(dims[2], dims[3]);
    std::swap(strides[2], strides[3]);
    n_fast = ceil_div(align_up(M, sf_layout == AC4K_SF_AC4K ? 16 : 128), 64);
    n_mid = ceil_div(Kp, 128);
    if (reinterpret_cast<uintptr_t>(out) & 15) return kResidentDeclined;
  } else {
    return kResidentDeclined;
  }
  // what a tensor map takes: 16-byte strides and base; and 32-bit coordinates and counts
  if (reinterpret_cast<uintptr_t>(in) & 15) return kResidentDeclined;
  for (int i = 0; i < 3; ++i) {
    if (dims[i] == 1) strides[i] = 8;                 // (never added to anything)
    else if (strides[i] <= 0 || strides[i] % 8 || strides[i] >= (1ll << 38)) return kResidentDeclined;
  }
  if (M > (1 << 30) || K > (1 << 30) || nbatch > (1 << 30) / (n_fast * n_mid)) return kResidentDeclined;
  *a = ResidentArgs{};
  a->status = device_status_ptr();
  if (!a->status || get_tmap_bf16_tiles(in, dims, strides, tm)) return kResidentDeclined;
  a->out = static_cast<uint8_t *>(out);
  a->sf = static_cast<uint8_t *>(sf);
  a->g_out = g_out;
  a->max_scale = max_scale;
  a->wait_ns = debug_wait_ns() ? debug_wait_ns() : kWaitTimeoutNs;
  a->dbg = debug_flags();
  a->M = (int)M; a->K = (int)K; a->d1 = (int)shape[1];
  a->n_fast = (int)n_fast; a->n_mid = (int)n_mid; a->tiles = (int)(nbatch * n_fast * n_mid);
  return 0;
}

int launch_quantize_resident(void *out, void *sf, float *g_out, void *scratch, const void *in, float max_scale, const int64_t shape[4],
                             const int64_t stride[4], int swizzle, int sf_layout, cudaStream_t stream) {
  using namespace resident;
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  if (di.cc_major != 10 || !meetings_fit(di.sms)) return kResidentDeclined;
  int mode;
  CUtensorMap tm;
  ResidentArgs a;
  if (int e = resident_plan(out, sf, g_out, in, max_scale, shape, stride, swizzle, sf_layout, &mode, &tm, &a)) return e;
  if (sf_layout == AC4K_SF_AC4K) {
    if (mode == kRows) return launch_resident<AC4K_SF_AC4K, kRows>(tm, a, scratch, di.sms, stream);
    if (mode == kRowsAnyK) return launch_resident<AC4K_SF_AC4K, kRowsAnyK>(tm, a, scratch, di.sms, stream);
    if (mode == kTransposed) return launch_resident<AC4K_SF_AC4K, kTransposed>(tm, a, scratch, di.sms, stream);
    return launch_resident<AC4K_SF_AC4K, kTransposedPermuted>(tm, a, scratch, di.sms, stream);
  }
  if (mode == kRows) return launch_resident<AC4K_SF_TILE128X4, kRows>(tm, a, scratch, di.sms, stream);
  if (mode == kRowsAnyK) return launch_resident<AC4K_SF_TILE128X4, kRowsAnyK>(tm, a, scratch, di.sms, stream);
  if (mode == kTransposed) return launch_resident<AC4K_SF_TILE128X4, kTransposed>(tm, a, scratch, di.sms, stream);
  return launch_resident<AC4K_SF_TILE128X4, kTransposedPermuted>(tm, a, scratch, di.sms, stream);
}

// The CTAs are shared out by the tensors' tiles.  ROWS: the form of q and k.
template <int ROWS>
static int launch_attention(void *const out[3], void *const sf[3], float *const g_out[3], void *scratch, const void *const in[3],
                            const int64_t shape[3][4], const int64_t stride[3][4], float max_scale, cudaStream_t stream) {
  using namespace resident;
  DeviceInfo di;
  if (int e = get_device_info(&di)) return e;
  if (di.cc_major != 10 || di.sms < 3 || !meetings_fit(di.sms)) return kResidentDeclined;
  CUtensorMap tm[3];
  ResidentArgs a[3];
  int64_t total = 0;
  for (int i = 0; i < 3; ++i) {
    int mode;
    if (int e = resident_plan(out[i], sf[i], g_out[i], in[i], max_scale, shape[i], stride[i], i == 2, AC4K_SF_TILE128X4, &mode, &tm[i], &a[i])) return e;
    if (mode != (i == 2 ? kTransposedPermuted : ROWS)) return kResidentDeclined;
    total += a[i].tiles;
  }
  int ctas[3], used = 0, smem = 0;
  unsigned long long *at = first_word(scratch);
  for (int i = 0; i < 3; ++i) {
    // (rounded down, so that the three fit; at least one)
    ctas[i] = std::min(a[i].tiles, std::max(1, (int)(total <= di.sms ? a[i].tiles : a[i].tiles * (int64_t)(di.sms - 2) / total)));
    set_meeting(&a[i], at, ctas[i]);
    used += ctas[i];
    const int m = i == 2 ? kTransposedPermuted : ROWS;
    a[i].slots = std::min((int)ceil_div(a[i].tiles, ctas[i]), max_slots(m));
    smem = std::max(smem, smem_bytes(m, a[i].slots));
  }
  auto kern = nvfp4_quantize_attention_kernel<AC4K_SF_TILE128X4, ROWS>;
  static PerDevice<int> attr_set;
  int unused = 0;
  if (int e = attr_set.get(&unused, [&](int &v) {
        AC4K_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(smem_bytes(kRows, max_slots(kRows)), smem_bytes(kTransposed, max_slots(kTransposed)))));
        v = 1;
        return 0;
      }))
    return e;
  return launch_cooperative(kern, used, smem, stream, tm[0], tm[1], tm[2], a[0], a[1], a[2], ctas[0], ctas[1]);
}

}  // namespace ac4k

using namespace ac4k;

// The elements lie side by side in some order of the dimensions: ac4k_quantize_nvfp4_dynamic takes the maximum of as many from `in` on
static bool is_dense(const int64_t shape[4], const int64_t stride[4]) {
  int order[4] = {0, 1, 2, 3};
  std::sort(order, order + 4, [&](int a, int b) { return stride[a] < stride[b]; });
  int64_t next = 1;
  for (int i : order) {
    if (shape[i] == 1) continue;
    if (stride[i] != next) return false;
    next *= shape[i];
  }
  return true;
}

extern "C" int ac4k_attention_quantize_nvfp4(void *const out[3], void *const sf[3], float *const g_out[3], void *scratch, const void *const in[3],
                                             const int64_t stride[3][4], int64_t B, int64_t H, int64_t Nq, int64_t Nkv, int64_t D, int64_t Dv,
                                             ac4k_stream_t stream) {
  if (!out || !sf || !g_out || !in || !stride || !scratch) return fail(AC4K_ERR_NULL, "a required pointer is NULL");
  for (int i = 0; i < 3; ++i)
    if (!out[i] || !sf[i] || !g_out[i] || !in[i]) return fail(AC4K_ERR_NULL, "a required pointer is NULL");
  if (B <= 0 || H <= 0 || Nq <= 0 || Nkv <= 0 || D <= 0 || Dv <= 0) return fail(AC4K_ERR_SHAPE, "dimensions must be positive");
  constexpr float kMaxScale = 6.0f * 448.0f;
  // [outer, outer, cross, reduce]: q and k along the features, v along the keys
  const int64_t shape[3][4] = {{B, H, Nq, D}, {B, H, Nkv, D}, {B, H, Dv, Nkv}};
  int64_t st[3][4];
  for (int i = 0; i < 3; ++i) {
    st[i][0] = stride[i][0]; st[i][1] = stride[i][1];
    st[i][2] = stride[i][i == 2 ? 3 : 2]; st[i][3] = stride[i][i == 2 ? 2 : 3];
  }
  for (int i = 0; i < 3; ++i)
    if ((reinterpret_cast<uintptr_t>(out[i]) & 7) || (reinterpret_cast<uintptr_t>(sf[i]) & 3) || (reinterpret_cast<uintptr_t>(in[i]) & 1))
      return fail(AC4K_ERR_ALIGN, "out must be 8-byte, sf 4-byte and in 2-byte aligned");
  const auto launch = D % 16 ? &launch_attention<resident::kRowsAnyK> : &launch_attention<resident::kRows>;
  const int e = launch(out, sf, g_out, scratch, in, shape, st, kMaxScale, static_cast<cudaStream_t>(stream));
  if (e != kResidentDeclined) return e;
  for (int i = 0; i < 3; ++i)
    if (!is_dense(shape[i], st[i])) return fail(AC4K_ERR_SHAPE, "operand %d is not dense, and the one launch does not take its address or strides", i);
  for (int i = 0; i < 3; ++i)
    if (int rc = ac4k_quantize_nvfp4_dynamic(out[i], sf[i], g_out[i], scratch, in[i], kMaxScale, shape[i], st[i], i == 2, AC4K_SF_TILE128X4, stream)) return rc;
  return 0;
}
