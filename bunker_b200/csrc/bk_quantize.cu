// bk_quantize.cu -- f32 / bf16 weight rows -> Q4_K superblocks on the device: the quantiser behind the weight loader.
//
// bunker uploads its safetensors weights as they are, bf16 (loadWeights, prototypes/decode.ts:64-76); the Q4_K model
// served here needs them quantised once at load time.  A lane takes a sub-block of 32 weights, a warp four superblocks of 256.  The
// arithmetic is the CPU oracle's, operation for operation:
//   sub-block:  lo = min(min x, 0), scale = (max x - lo) / 15, mn = 0 - lo
//   superblock: d = f16_rn(max scale / 63), dmin = f16_rn(max mn / 63), sc = floor(scale * (1/d) + 0.5) (<= 63),
//               m = floor(mn * (1/dmin) + 0.5) (<= 63)
//   weight:     q = clamp(floor((x + dmin*m) / (d*sc) + 0.5), 0, 15)
// Output layout: bytes [0,2) d, [2,4) dmin, [4,16) the twelve 6-bit scale/min bytes, [16,144) quants, every 32 bytes
// serving sub-blocks 2p (low nibbles) and 2p+1 (high nibbles).
#include <algorithm>

#include "bk_common.cuh"
#include "bk_internal.h"

namespace {

constexpr int kQWarps = 4;   // warps of a CTA
constexpr int kQSb = 4;      // superblocks of a warp

// floor(t / dl + 0.5) clamped to 0..15, t = w + ml, the sum, the division and the addition each rounded once.  The quotient is first formed as
// w * r + ml * r with the approximate reciprocal r (off by at most 2^-23 of it) and rounded to the nearest integer.  With ml * r up to 32 it
// is off by less than 4e-6 for r and ml * r and 1e-6 for its own rounding, and the exact one by 2.4e-6 for its three, below 16: unless it
// lies within kTieBand of a half the integer is already the exact one.
constexpr float kTieBand = 1e-5f, kMaxMlr = 32.0f;
BK_DEVINL uint32_t quant4_exact(float t, float dl) { return (uint32_t)max(0, min(15, (int)floorf(__fadd_rn(__fdiv_rn(t, dl), 0.5f)))); }

BK_DEVINL uint32_t min_bf2(uint32_t a, uint32_t b) {   // like fminf: a NaN loses
  uint32_t d;
  asm("min.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
BK_DEVINL uint32_t max_nan_bf2(uint32_t a, uint32_t b) {   // a NaN wins
  uint32_t d;
  asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
BK_DEVINL float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
// chunk c of a row of 16-byte chunks: rows are permuted so that the lanes' reads hit all banks
template <bool BF16>
BK_DEVINL int chunk_slot(int row, int c) {
  return BF16 ? row * 4 + (c ^ ((row >> 1) & 3)) : row * 8 + (c ^ (row & 7));
}
// weight e of sub-block `sub`, for what seldom runs
template <bool BF16>
BK_DEVINL float one_weight(const uint4* rows, int sub, int e) {
  if (BF16) return bk_bf16_to_f32(reinterpret_cast<const uint16_t*>(rows + chunk_slot<BF16>(sub, e >> 3))[e & 7]);
  return reinterpret_cast<const float*>(rows + chunk_slot<BF16>(sub, e >> 2))[e & 3];
}
template <bool BF16>
__device__ __noinline__ float largest_number(const uint4* rows) {
  const int lane = threadIdx.x & 31;
  float hi = one_weight<BF16>(rows, lane, 0);
#pragma unroll 1
  for (int e = 1; e < 32; e++) hi = fmaxf(hi, one_weight<BF16>(rows, lane, e));
  return hi;
}
// q of the lanes in `todo` becomes the exact quants of their weights 8c to 8c + 7, a byte each: eight lanes divide for one.  Of 1,024 weights
// one lies near a tie in 50 cases, and a small launch waits for its slowest warp: with the lane's own eight divisions one after the other 64 x
// 1,536 weights took 4.6 us, 301 x 2,304 5.3.
template <bool BF16>
__device__ __noinline__ uint2 exact_quants(const uint4* rows, int c, uint32_t todo, uint2 q, float ml, float dl) {
  const int lane = threadIdx.x & 31, e = lane & 7;
#pragma unroll 1
  for (; todo; todo &= todo - 1) {
    const int sub = __ffs(todo) - 1;
    const float t = __fadd_rn(one_weight<BF16>(rows, sub, 8 * c + e), __shfl_sync(0xffffffffu, ml, sub));
    const uint32_t v = quant4_exact(t, __shfl_sync(0xffffffffu, dl, sub)) << (8 * (e & 3));
    const uint32_t x = __reduce_or_sync(0xffffffffu, e < 4 ? v : 0u), y = __reduce_or_sync(0xffffffffu, e < 4 ? 0u : v);
    if (lane == sub) q = make_uint2(x, y);
  }
  return q;
}

// The quants of this lane's sub-block, with the neighbour's, into their 32 bytes.  PLAIN: no weight of the warp leaves 0..15, none is a NaN, and
// ml * r is small.  Rounding without conversions: y + 1.5 * 2^23 has the integer in its low bits; two weights per instruction.
template <bool BF16, bool PLAIN>
BK_DEVINL void write_quants(const uint4* rows, uint8_t* quants, float r, float mlr, float ml, float dl) {
  constexpr float kMagic = 12582912.0f;
  const int lane = threadIdx.x & 31;
  const bool odd = lane & 1;
  const float2 magic2 = make_float2(kMagic, kMagic), minus2 = make_float2(-1.0f, -1.0f), r2 = make_float2(r, r), c2 = PLAIN ? make_float2(mlr, mlr) : make_float2(0.0f, 0.0f);
#pragma unroll
  for (int c = 0; c < 4; c++) {   // eight weights, read again: kept in registers since the first pass they cost a third of the warps
    float w[8];
    if (BF16) {
      const uint4 v = rows[chunk_slot<BF16>(lane, c)];
      w[0] = __uint_as_float(v.x << 16); w[1] = __uint_as_float(v.x & 0xffff0000u);
      w[2] = __uint_as_float(v.y << 16); w[3] = __uint_as_float(v.y & 0xffff0000u);
      w[4] = __uint_as_float(v.z << 16); w[5] = __uint_as_float(v.z & 0xffff0000u);
      w[6] = __uint_as_float(v.w << 16); w[7] = __uint_as_float(v.w & 0xffff0000u);
    } else {
      const uint4 v = rows[chunk_slot<BF16>(lane, 2 * c)], u = rows[chunk_slot<BF16>(lane, 2 * c + 1)];
      w[0] = __uint_as_float(v.x); w[1] = __uint_as_float(v.y); w[2] = __uint_as_float(v.z); w[3] = __uint_as_float(v.w);
      w[4] = __uint_as_float(u.x); w[5] = __uint_as_float(u.y); w[6] = __uint_as_float(u.z); w[7] = __uint_as_float(u.w);
    }
    uint32_t t[8];
    float tie = 0.0f;   // largest distance from an integer
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      float2 x = make_float2(w[e], w[e + 1]);
      if (!PLAIN) x = bk_add2(x, make_float2(ml, ml));
      const float2 y = bk_fma2(x, r2, c2);
      float2 f = bk_add2(y, magic2);
      const float2 o = bk_add2(y, bk_fma2(f, minus2, magic2));
      tie = fmaxf(tie, fmaxf(fabsf(o.x), fabsf(o.y)));
      if (!PLAIN) f = make_float2(fminf(fmaxf(f.x, kMagic), kMagic + 15.0f), fminf(fmaxf(f.y, kMagic), kMagic + 15.0f));   // (a NaN becomes 0)
      t[e] = __float_as_uint(f.x);
      t[e + 1] = __float_as_uint(f.y);
    }
    uint2 q;   // a quant per byte
    q.x = __byte_perm(__byte_perm(t[0], t[1], 0x0040), __byte_perm(t[2], t[3], 0x0040), 0x5410);
    q.y = __byte_perm(__byte_perm(t[4], t[5], 0x0040), __byte_perm(t[6], t[7], 0x0040), 0x5410);
    const uint32_t near_tie = __ballot_sync(0xffffffffu, tie > 0.5f - kTieBand);
    if (near_tie) q = exact_quants<BF16>(rows, c, near_tie, q, ml, dl);
    if (!PLAIN && !(dl > 0.0f)) q = make_uint2(0u, 0u);
    // of the pair of lanes the even one writes the first four bytes, the odd one the others
    const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? q.x : q.y, 1);
    *reinterpret_cast<uint32_t*>(quants + 8 * c) = odd ? other | (q.y << 4) : q.x | (other << 4);
  }
}

// the 1,024 weights in `rows` to four superblocks in `stage`; sub-block `lane` is this lane's
template <bool BF16>
BK_DEVINL void quantize_superblocks(const uint4* rows, uint8_t* stage) {
  constexpr int kChunks = BF16 ? 4 : 8;
  const int lane = threadIdx.x & 31, l = lane & 7;
  float lo, hi;
  if (BF16) {
    uint32_t mn2, mx2;   // of the even and of the odd weights, as the bf16 pairs that they are
#pragma unroll
    for (int c = 0; c < kChunks; c++) {
      const uint4 v = rows[chunk_slot<BF16>(lane, c)];
      const uint32_t mn = min_bf2(min_bf2(v.x, v.y), min_bf2(v.z, v.w)), mx = max_nan_bf2(max_nan_bf2(v.x, v.y), max_nan_bf2(v.z, v.w));
      mn2 = c == 0 ? mn : min_bf2(mn2, mn);
      mx2 = c == 0 ? mx : max_nan_bf2(mx2, mx);
    }
    lo = fminf(__uint_as_float(mn2 << 16), __uint_as_float(mn2 & 0xffff0000u));
    hi = max_nan(__uint_as_float(mx2 << 16), __uint_as_float(mx2 & 0xffff0000u));
  } else {
#pragma unroll
    for (int c = 0; c < kChunks; c++) {
      const float4 v = *reinterpret_cast<const float4*>(rows + chunk_slot<BF16>(lane, c));
      const float mn = fminf(fminf(v.x, v.y), fminf(v.z, v.w)), mx = max_nan(max_nan(v.x, v.y), max_nan(v.z, v.w));
      lo = c == 0 ? mn : fminf(lo, mn);
      hi = c == 0 ? mx : max_nan(hi, mx);
    }
  }
  const bool has_nan = hi != hi;   // a NaN counts for neither end and becomes 0
  if (has_nan) hi = largest_number<BF16>(rows);
  if (lo > 0.0f) lo = 0.0f;
  float scale = __fdiv_rn(__fsub_rn(hi, lo), 15.0f);
  if (!(scale > 0.0f)) scale = 0.0f;
  const float mn = __fsub_rn(0.0f, lo);   // 0 - lo, not -lo: a zero minimum stays +0 (its sign would reach the f16 dmin)
  float max_scale = scale, max_min = mn;
#pragma unroll
  for (int off = 1; off <= 4; off <<= 1) {
    max_scale = fmaxf(max_scale, __shfl_xor_sync(0xffffffffu, max_scale, off));
    max_min = fmaxf(max_min, __shfl_xor_sync(0xffffffffu, max_min, off));
  }
  uint16_t dh, mh;
  asm("cvt.rn.f16.f32 %0, %1;" : "=h"(dh) : "f"(__fdiv_rn(max_scale, 63.0f)));
  asm("cvt.rn.f16.f32 %0, %1;" : "=h"(mh) : "f"(__fdiv_rn(max_min, 63.0f)));
  const float d = bk_f16_to_f32(dh), dm = bk_f16_to_f32(mh);
  const float inv_d = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f, inv_dm = dm > 0.0f ? __fdiv_rn(1.0f, dm) : 0.0f;
  const int sc = min(63, (int)floorf(__fadd_rn(__fmul_rn(scale, inv_d), 0.5f)));
  const int m6 = min(63, (int)floorf(__fadd_rn(__fmul_rn(mn, inv_dm), 0.5f)));
  const float dl = __fmul_rn(d, (float)sc), ml = __fmul_rn(dm, (float)m6);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(dl));
  uint8_t* const sb = stage + (lane >> 3) * 144;
  uint8_t* const quants = sb + 16 + (l >> 1) * 32 + (lane & 1 ? 4 : 0);   // 32 bytes hold sub-block 2p in their low and 2p + 1 in their high nibbles
  // The smallest and the largest weight (rounding is monotonic) show whether any lane needs the clamp to 0..15, or t before its product.
  const float mlr = __fmul_rn(ml, r);
  const bool plain = dl > 0.0f && mlr <= kMaxMlr && !has_nan && fmaf(lo, r, mlr) > -0.49f && fmaf(hi, r, mlr) < 15.49f;
  if (__all_sync(0xffffffffu, plain)) write_quants<BF16, true>(rows, quants, r, mlr, ml, dl);
  else write_quants<BF16, false>(rows, quants, r, mlr, ml, dl);
  // header: lanes 0..3 of a superblock assemble bytes j, j+4, j+8 of the twelve
  const int upper = __shfl_down_sync(0xffffffffu, sc | (m6 << 8), 4), sc_hi = upper & 0xff, m_hi = upper >> 8;
  if (l < 4) {
    sb[4 + l] = (uint8_t)(sc | ((sc_hi >> 4) << 6));
    sb[8 + l] = (uint8_t)(m6 | ((m_hi >> 4) << 6));
    sb[12 + l] = (uint8_t)((sc_hi & 0x0f) | ((m_hi & 0x0f) << 4));
  }
  if (l == 0) *reinterpret_cast<uint32_t*>(sb) = (uint32_t)dh | ((uint32_t)mh << 16);
}

// Bound: instruction issue, 79 % of the slots with half a sub-block a lane.  Of the 363 instructions per 512 weights that that took, more than
// half were a sub-block's and a superblock's scalar work (five divisions, the maxima, the header), done by every lane; with a whole sub-block
// a lane each of them serves twice as many weights.  A lane's weights are 64 or 128 contiguous bytes, so they come through shared memory:
// 16-byte chunks by asynchronous copies in the order of memory.  The grid fills the device once and a warp requests its next superblocks
// before it quantises the present ones (24,000 f32 superblocks 11.3 us, so 9.3).  64 registers for bf16, as many as eight CTAs of an SM
// leave: fewer cost more than the warps they allow give (11 CTAs 68 us).  17,408 x 5,120 weights: bf16 73.5 -> 58 us (3.9 TB/s), f32 80 -> 68.
template <bool BF16>
__global__ void __launch_bounds__(kQWarps * 32, BF16 ? 8 : 5) quantize_q4k_kernel(const void* x, size_t n_superblocks, uint8_t* out) {
  constexpr int kChunks = BF16 ? 4 : 8;   // 16-byte chunks of a sub-block
  __shared__ __align__(16) uint4 rows[kQWarps][2][32 * kChunks];   // the weights in use and the next ones
  __shared__ __align__(16) uint8_t stage[kQWarps][kQSb * 144];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto request = [&](size_t first, int buffer) {
    if (first < n_superblocks) {
      const int n_sb = (int)min((size_t)kQSb, n_superblocks - first);
#pragma unroll
      for (int k = 0; k < kChunks; k++) {   // chunk `at` of the warp's weights; superblocks past the end are the last one again, and not stored
        const int at = lane + 32 * k, sb = at / (8 * kChunks);
        const uint8_t* src = static_cast<const uint8_t*>(x) + (first + min(sb, n_sb - 1)) * (8 * kChunks * 16) + (at % (8 * kChunks)) * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&rows[warp][buffer][chunk_slot<BF16>(at / kChunks, at % kChunks)])), "l"(src) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const size_t step = (size_t)gridDim.x * kQWarps * kQSb;
  size_t first = ((size_t)blockIdx.x * kQWarps + warp) * kQSb;
  request(first, 0);
#pragma unroll 1
  for (int buffer = 0; first < n_superblocks; first += step, buffer ^= 1) {
    request(first + step, buffer ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    quantize_superblocks<BF16>(rows[warp][buffer], stage[warp]);
    __syncwarp();
    const int n16 = 9 * (int)min((size_t)kQSb, n_superblocks - first);
    for (int i = lane; i < n16; i += 32) reinterpret_cast<uint4*>(out + first * 144)[i] = reinterpret_cast<const uint4*>(stage[warp])[i];
    __syncwarp();
  }
}

}  // namespace

extern "C" int32_t bkQuantizeQ4K(uint64_t x, int32_t dtype, int64_t n_rows, int32_t K, uint64_t out) {
  BK_REQUIRE_INIT();
  BK_ARG(dtype == BK_DTYPE_F32 || dtype == BK_DTYPE_BF16, "bkQuantizeQ4K: dtype %d (BK_DTYPE_F32 or BK_DTYPE_BF16)", dtype);
  BK_ARG(n_rows > 0 && K > 0 && K % 256 == 0, "bkQuantizeQ4K: bad shape rows=%lld K=%d (K a multiple of 256)", (long long)n_rows, K);
  BK_ARG(x && out && (x & 15) == 0 && (out & 15) == 0, "bkQuantizeQ4K: null or misaligned pointer");
  const size_t nsb = (size_t)n_rows * (K / 256);
  static int resident[2] = {0, 0};   // CTAs of an SM
  int& n = resident[dtype == BK_DTYPE_BF16];
  if (!n) {
    if (dtype == BK_DTYPE_BF16) BK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, quantize_q4k_kernel<true>, kQWarps * 32, 0));
    else BK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, quantize_q4k_kernel<false>, kQWarps * 32, 0));
    if (n < 1) n = 1;
  }
  const size_t ctas = (nsb + kQSb * kQWarps - 1) / (kQSb * kQWarps);
  const unsigned grid = (unsigned)std::min<size_t>(ctas, (size_t)n * bk_ctx().sm_count);
  if (dtype == BK_DTYPE_BF16)
    quantize_q4k_kernel<true><<<grid, kQWarps * 32, 0, bk_ctx().stream>>>(bk_ptr<void>(x), nsb, bk_ptr<uint8_t>(out));
  else
    quantize_q4k_kernel<false><<<grid, kQWarps * 32, 0, bk_ctx().stream>>>(bk_ptr<void>(x), nsb, bk_ptr<uint8_t>(out));
  BK_CHECK_LAUNCH();
  return BK_OK;
}
