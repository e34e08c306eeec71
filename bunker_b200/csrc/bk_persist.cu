// bk_persist.cu -- the batch-1 decode step as ONE cooperative launch of one CTA per SM: a list of phases (projection
// GEMVs, conv1d + gated-DeltaNet steps, attention, lm_head + argmax) that hand their activations to one another inside
// the launch.
//
// Replaces the launch loop of bunker's executor (runGraphDecode, src/runner.ts:133-160: ~287 cuLaunch calls per token,
// LOG.md:580,712) on the single-GPU, single-sequence path.  The arithmetic of every phase is the per-op kernels', operation
// for operation, so results are bit-identical to the per-op step.
//
// What bounds a step at batch 1: about 120 dependent phases, so the latency of a hand-off and of a phase's fixed part; the
// weights alone would take 170 us (24 layers, hidden 2048).  As 123 dependent launches the step takes 726 us (5.9 us
// each: grid completion, flush and dependency wait 2 us, activation prologue 1-2 us, then the rows); as one launch 558 us.
// Of the 4.5 us of a projection phase (2048 wide, 84 rows per SM) 0.7 us are the wait for the hand-off, 1.3 us norm and
// quantisation, 1.5 us dot products, 0.4 us reduction and epilogue.  64 layers of hidden 5120: 4.75 -> 4.6 ms.  There the projections are
// long enough to be streams (gate and up 25 us for 100 MB, 4.0 TB/s; the others 2.6 to 2.9) and neither the dots (1.3 ms) nor HBM (2.2 ms)
// account for the step; the ring holds 120 KB, 2.7 us of an SM's share, so it is full and stands still while a long activation is staged.
//
// Hand-off.  There is no grid barrier.  Every activation word carries the generation it belongs to: bf16 values as 32-bit
// words {value, 16-bit tag}, f32 values as 64-bit words {value, 32-bit tag}.  A producer stores the word; a consumer loads
// the words it needs (past L1) until their tags match -- one L2 store and one L2 load on the critical path, no fence, no
// flag.  A value and its tag are one element of the access on both sides (the elements of a vector access are not ordered among
// themselves, so a 64-bit word is never read as two of 32 bits).  A buffer is rewritten once per layer; a writer of generation g+1 has, through the chain of phases in between,
// waited for every reader of generation g (each full-vector input is complete only when all its writers have finished
// reading the vector before it), so one buffer per activation is enough and a tag can never be skipped or reused early.
//
// Weight stream.  A producer warp walks the launch's row groups in the order the other warps consume them and keeps a
// FIFO ring in shared memory filled with bulk copies (cp.async.bulk, completion on an mbarrier), across phase boundaries:
// weights depend on nothing, so the next phases' rows arrive while the activations of this one are waited for.  It also
// prefetches the small per-layer data (norm weights, recurrent state, conv taps, cached keys and values) into L2.
//
// Every wait -- for words, weights, state slices and free buffers -- is bounded by the same number of polls: one that gives up sets the
// status word and a flag in shared memory, after which no wait of that CTA waits again.  Its consumers run through the remaining
// phases on whatever lies in shared memory (their words keep their tags, so nobody waits for them); its producer requests no more,
// waits until what it has requested has landed, and ends.
#include <string.h>

#include <algorithm>
#include <vector>

#include <cuda.h>   // CUtensorMap

#include "bk_gemv_dp4a.cuh"

namespace {

constexpr int kCW = 8;                // consumer warps: with the producer 288 threads, 168 registers each without a spill (16 warps spill)
constexpr int kBlock = 4;             // rows multiplied together
constexpr int kCT = kCW * 32;
static_assert(kCT == 256, "norms and embedded rows are in the 256-thread order");
constexpr int kPT = kCT + 32;         // and the producer warp
constexpr int kEnt = 64;              // ring entries (row groups requested and not yet freed), eight per consumer warp
constexpr int kGroupMax = 128 / kCW;  // rows of a group
constexpr int kLanesPerRow = 32 / kGroupMax;
constexpr int kAccPitch = 32 + kLanesPerRow;   // floats per row of lane sums: kGroupMax rows times kLanesPerRow lanes hit 32 banks
constexpr int kGdnCols = 32;          // state columns of one GDN item: four items share a value head
constexpr uint32_t kGdnBytes = 128 * kGdnCols * 4;
constexpr int kWin = 4;               // phase descriptors in shared memory
constexpr int kMaxNormK = 8192;       // widest normalised row (four chunks per thread of the 256-thread order)
constexpr int kDefaultPolls = 1 << 20;
constexpr int kHD = 256;

enum { PH_GEMV = 1, PH_GDN, PH_ATTN, PH_MERGE };
enum { IN_EMBED = 0, IN_NORM, IN_PLAIN };
enum { OUT_T16 = 0, OUT_T32, OUT_ADD, OUT_SWIGLU, OUT_LOGITS };

struct PSeg {
  const uint8_t* W;
  const uint8_t* W2;
  void* out;
  int n_rows, epi, vrow_begin, pad;
};
struct GemvPart {
  PSeg segs[4];
};
struct GdnPart {
  const uint32_t *qkv, *z;         // tagged bf16
  const unsigned long long *a, *b; // tagged f32
  const uint16_t* conv_w;
  uint16_t* cs[2];
  const float* A_log;
  const uint16_t* dt_bias;
  float* S;
  const float* norm_w;             // gated norm, f32 [128]
  unsigned long long* sums;        // tagged f32 [Hv][4 items][8]: lane sums of the gated norm
  uint32_t* o;                     // tagged bf16
  const CUtensorMap* map;          // S as [Hv*128][128] f32, box 128 rows x 32 columns
};
struct AttnPart {
  const uint32_t *qg, *k, *v;
  const uint16_t *q_norm_w, *k_norm_w;
  uint16_t *kc, *vc;
};
struct __align__(16) Phase {
  int type, in_kind, K, n_segs;
  int vrows, swiglu, gmax, in_tag;   // tags are offsets to the launch's base
  int out_tag, res_tag;
  int ubase, uextra, rounds;   // split of the rows over the CTAs (cta_share)
  int entry;               // ring entries of the phases before this one
  int buffer;              // which staged activation this phase writes: 0 in phases fed by the residual stream, 1 in the others
  int gdn_index;           // PH_GDN: its number among the GDN phases; PH_GEMV: 1 if the phase follows a GDN phase
  float eps;
  int pad;
  const void* in;          // tagged bf16 [K]
  const void* norm_w;      // bf16 [K]
  const uint32_t* res;     // OUT_ADD: tagged bf16
  uint16_t* plain;         // OUT_ADD: untagged copy, or null
  union {
    GemvPart g;
    GdnPart d;
    AttnPart a;
  };
};
static_assert(sizeof(Phase) % 16 == 0 && sizeof(Phase) / 16 <= 32, "one warp copies a descriptor");

struct StepIO {
  const uint8_t* embed;
  const int32_t* ids_in;
  int token;               // the input token, or -1: ids_in has it
  uint32_t* x_tagged;      // residual stream, tagged
  uint16_t* x0;            // untagged copy of the embedded row
  float* part_v;
  int32_t* part_i;
  unsigned int* counter;
  int32_t* ids_out;
  float* val_out;
  int32_t* pos;
  int32_t* hist;
  int hist_ld, hist_rows;
  int32_t* host_out;
  int H;
};

struct StepParams {
  const Phase* phases;
  int n_phases, tags;              // tags: generations per launch
  unsigned int* epoch;
  int* status;
  int polls;
  int parity;                      // conv-state parity of this step
  unsigned long long* trace;       // 8 slots per phase, or null
  uint32_t ring_bytes, xs0_bytes, xs_bytes, scratch_bytes, gdn_bytes;   // xs0: staged activation of the residual stream
  // GDN
  int Hk, Hv, gdn_slots;           // items a CTA takes, one per four warps
  // attention
  int Hq, Hkv, rot_half, max_len, split_len, max_splits;
  float scale;
  const float *cos_t, *sin_t;
  unsigned long long *po, *pml;    // split partials, tagged f32: [Hq][max_splits][256] and [Hq][max_splits][2]
  uint32_t* attn_out;              // tagged bf16 [Hq*256]
  StepIO io;
};

struct SmemLayout {
  size_t desc, pdesc, xs, scratch, red, full, empty, gfull, gfree, ent, misc, best, accs, gdn, ring, total;
};
__host__ __device__ inline SmemLayout smem_layout(uint32_t xs_bytes, uint32_t scratch_bytes, uint32_t gdn_bytes, uint32_t ring_bytes) {
  SmemLayout L;
  size_t o = 0;
  L.desc = o; o += kWin * sizeof(Phase);
  L.pdesc = o; o += sizeof(Phase);    // the producer's own
  L.red = o; o += 128;
  L.full = o; o += kEnt * 8;
  L.empty = o; o += kEnt * 8;
  L.gfull = o; o += 16;
  L.gfree = o; o += 16;
  L.ent = o; o += kEnt * 4;            // ring offset of an entry
  L.misc = o; o += 256;                // [0] dead flag, [1] last flag, [8..24) argmax values, [24..40) indices
  L.best = o; o += (size_t)kCW * kGroupMax * 8;   // running argmax of the lm_head rows
  o = (o + 127) & ~(size_t)127;
  L.ring = o; o += ring_bytes;         // in front of the rest: a CTA that has given up reads up to a group past any offset in it
  L.accs = o; o += (size_t)kCW * kGroupMax * kAccPitch * 4;   // lane sums of a row group, per warp
  L.xs = o; o += xs_bytes;             // both staged activations
  L.scratch = o; o += scratch_bytes;
  o = (o + 127) & ~(size_t)127;
  L.gdn = o; o += gdn_bytes;           // state slices of the CTA's GDN items
  L.total = o;
  return L;
}
// one staged activation: words, then d8, then s8
__host__ __device__ inline uint32_t xs_bytes_for(int K) { return (uint32_t)(((K / 64) * kUnitWords * 4 + (K / 32) * 8 + 127) & ~127); }

// ---- tagged words ------------------------------------------------------------------
struct Ctl {
  volatile int* dead;
  int* status;
  int polls;
};
BK_DEVINL uint32_t ld_word(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
BK_DEVINL uint4 ld_vec(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
BK_DEVINL uint2 ld_pair(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
// loads of constant data that stay where they are written (an ordinary load may be moved down to its use, which is where
// its latency would be paid)
BK_DEVINL uint4 ld_early(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
BK_DEVINL void st_t16(uint32_t* p, uint16_t h, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"((tag << 16) | h) : "memory");
}
BK_DEVINL void st_t32(unsigned long long* p, float v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | __float_as_uint(v)) : "memory");
}
// whether a wait goes on after its it-th look (0, 1, ...) found a stale word
BK_DEVINL bool keep_polling(const Ctl& c, int it) {
  if (*c.dead) return false;
  if (it < c.polls) return true;
  *c.dead = 1;
  atomicExch(c.status, BK_ERR_TIMEOUT);
  return false;
}
// whether the phase of an mbarrier completed before the wait gave up
BK_DEVINL bool wait_bar(uint32_t bar, uint32_t parity, const Ctl& c) {
  for (int it = 0; !mbar_try_wait(bar, parity); it++)
    if (!keep_polling(c, it)) return false;
  return true;
}
// bits of the upper halves that differ from the tag
BK_DEVINL uint32_t stale16(const uint4& v, uint32_t th) { return ((v.x ^ th) | (v.y ^ th) | (v.z ^ th) | (v.w ^ th)) & 0xffff0000u; }
BK_DEVINL uint32_t wait_word(const uint32_t* p, uint32_t first, uint32_t tag, const Ctl& c) {
  uint32_t w = first;
  for (int it = 0; ((w ^ (tag << 16)) & 0xffff0000u) != 0; it++) {
    if (!keep_polling(c, it)) break;
    w = ld_word(p);
  }
  return w;
}
// A warp that found stale words waits for one word of the 256 it loads, a different one in every CTA, before it loads them all
// again: looking at all of them while they are being produced would keep the L2 slices busy with the looks of 148 SMs.
BK_DEVINL void sentinel16(const uint32_t* p, uint32_t th, const Ctl& c) {
  if ((threadIdx.x & 31) == 0) {
    const uint32_t* w = p + ((blockIdx.x * 37u) & 255u);
    for (int it = 0; ((ld_word(w) ^ th) & 0xffff0000u) != 0; it++)
      if (!keep_polling(c, it)) break;
  }
  __syncwarp();
}
// chunk q (eight words, {a, b}) has been looked at: wait until it is fresh
BK_DEVINL void wait_chunk(const uint32_t* in, int q, uint32_t th, uint4& a, uint4& b, const Ctl& c) {
  for (int it = 0; stale16(a, th) | stale16(b, th); it++) {
    if (!keep_polling(c, it)) break;
    a = ld_vec(in + (size_t)q * 8);
    b = ld_vec(in + (size_t)q * 8 + 4);
  }
  __syncwarp();
}

BK_DEVINL unsigned long long global_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
BK_DEVINL void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCT) : "memory"); }
BK_DEVINL void bf16x8(const uint4& v, float (&y)[8]) {
  y[0] = __uint_as_float(v.x << 16); y[1] = __uint_as_float(v.x & 0xffff0000u);
  y[2] = __uint_as_float(v.y << 16); y[3] = __uint_as_float(v.y & 0xffff0000u);
  y[4] = __uint_as_float(v.z << 16); y[5] = __uint_as_float(v.z & 0xffff0000u);
  y[6] = __uint_as_float(v.w << 16); y[7] = __uint_as_float(v.w & 0xffff0000u);
}

// ---- work split of a GEMV phase --------------------------------------------------------
// CTA c owns ubase units, the first uextra CTAs one more (a unit is a row, or a gate/up row pair); they are taken in R
// rounds, a round's units are split over the consumer warps.  Every share is within one of even.
struct Share {
  int u0, n, R, upr;   // first unit, units, rounds, rows per unit
};
BK_DEVINL Share cta_share(const Phase& ph) {
  Share s;
  const int c = blockIdx.x;
  s.upr = ph.swiglu ? 2 : 1;
  s.u0 = c * ph.ubase + min(c, ph.uextra);
  s.n = ph.ubase + (c < ph.uextra ? 1 : 0);
  s.R = ph.rounds;
  return s;
}
BK_DEVINL void group_range(const Share& s, int round, int w, int& g0, int& g1) {
  const int a0 = s.R == 1 ? 0 : s.n * round / s.R, a1 = s.R == 1 ? s.n : s.n * (round + 1) / s.R;
  g0 = a0 + (a1 - a0) * w / kCW;
  g1 = a0 + (a1 - a0) * (w + 1) / kCW;
}

// ---- producer warp --------------------------------------------------------------------
// copies that have been requested land by themselves; the limit is a last resort
__device__ __noinline__ void wait_landed(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 22) && !mbar_try_wait(bar, parity); it++) {
  }
}
BK_DEVINL void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

BK_DEVINL bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}

// Lane w < kCW serves consumer warp w: it places the group in the FIFO (a prefix sum over the round), waits until the space
// is free and issues the copies.  Entries are freed in order; the lanes look at 32 entries' barriers at a time.
struct Requested {
  uint32_t entries, partial;   // entries of whole rounds; bit i: entry `entries` + i of a round that was given up
  uint32_t slices[2];          // state slices, by slot
};
__device__ __forceinline__ void producer_warp(const StepParams& P, uint8_t* smem, const SmemLayout& L, const Ctl& ctl, int pos, Requested& rq) {
  const int lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(smem + L.full), empty0 = smem_u32(smem + L.empty), ring0 = smem_u32(smem + L.ring);
  volatile uint32_t* ent = reinterpret_cast<volatile uint32_t*>(smem + L.ent);
  const Phase& ph = *reinterpret_cast<const Phase*>(smem + L.pdesc);
  constexpr int kDescVec = (int)(sizeof(Phase) / 16);
  const uint32_t size = P.ring_bytes;
  uint32_t h = 0, A = 0, tail_abs = 0;   // ring position of the head; absolute positions of head and tail
  uint32_t &seq = rq.entries, tail = 0;  // entries issued and freed
  uint32_t end0 = 0, end1 = 0;           // absolute end of the entries e = lane and e = lane + 32 (mod 64)
  const int c = blockIdx.x;
  const uint64_t policy = l2_evict_first();
  uint4 next = make_uint4(0, 0, 0, 0);
  if (lane < kDescVec) next = __ldg(reinterpret_cast<const uint4*>(P.phases) + lane);
  for (int k = 0; k < P.n_phases; k++) {
    if (lane < kDescVec) reinterpret_cast<uint4*>(smem + L.pdesc)[lane] = next;
    __syncwarp();
    if (lane < kDescVec && k + 1 < P.n_phases) next = ld_early(reinterpret_cast<const uint4*>(P.phases + k + 1) + lane);
    if (ph.type == PH_GEMV) {
      if (ph.in_kind == IN_NORM) {
        const uint8_t* nw = static_cast<const uint8_t*>(ph.norm_w);
        for (int i = lane; i < ph.K / 64; i += 32) l2_prefetch(nw + (size_t)i * 128);
      }
      const Share s = cta_share(ph);
      const uint32_t rowb = (uint32_t)(ph.K / 256) * 144;
      for (int r = 0; r < s.R; r++) {
        int g0 = 0, g1 = 0;
        if (lane < kCW) group_range(s, r, lane, g0, g1);
        const int nr = (g1 - g0) * s.upr;
        const uint32_t bytes = (uint32_t)nr * rowb;
        uint32_t incl = bytes;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += o;
        }
        const uint32_t excl = incl - bytes, total = __shfl_sync(0xffffffffu, incl, 31);
        const unsigned over = __ballot_sync(0xffffffffu, h + incl > size);   // the groups from here on start over at 0
        const int w0 = over ? __ffs(over) - 1 : 32;
        const uint32_t excl0 = __shfl_sync(0xffffffffu, excl, w0 & 31), pad = over ? size - (h + excl0) : 0;
        const uint32_t off = lane < w0 ? h + excl : excl - excl0;
        const uint32_t my_end = A + incl + (lane < w0 ? 0 : pad);
        // remember the ends by entry
        const int sh = (int)(seq & 31u);
        const uint32_t moved = __shfl_sync(0xffffffffu, my_end, (lane - sh) & 31);
        if (lane >= sh && lane < sh + kCW) (seq & 32u ? end1 : end0) = moved;
        const uint32_t e = (seq + lane) % kEnt;
        bool todo = lane < kCW;
        for (int it = 0;; it++) {
          if (todo && my_end - tail_abs <= size && seq + lane - tail < (uint32_t)kEnt) {
            todo = false;
            ent[e] = off;
            const uint32_t dst = ring0 + off, bar = full0 + 8 * e;
            mbar_expect_tx(bar, bytes);
            if (nr > 0) {
              if (s.upr == 2) {
                const size_t n0 = (size_t)(s.u0 + g0) * rowb;
                bulk_g2s_stream(dst, ph.g.segs[0].W + n0, bytes >> 1, bar, policy);
                bulk_g2s_stream(dst + (bytes >> 1), ph.g.segs[0].W2 + n0, bytes >> 1, bar, policy);
              } else {
                int v = s.u0 + g0, left = nr, si = 0;
                uint32_t d = dst;
                while (left > 0) {   // one iteration unless the group straddles a segment boundary
                  while (si + 1 < ph.n_segs && v >= ph.g.segs[si + 1].vrow_begin) si++;
                  const PSeg& sg = ph.g.segs[si];
                  const int t = v - sg.vrow_begin, run = min(left, sg.n_rows - t);
                  bulk_g2s_stream(d, sg.W + (size_t)t * rowb, (uint32_t)run * rowb, bar, policy);
                  d += (uint32_t)run * rowb;
                  v += run;
                  left -= run;
                }
              }
            }
          }
          if (!__any_sync(0xffffffffu, todo)) break;
          const uint32_t te = tail + lane;
          const bool freed = (int)(seq - te) > 0 && mbar_test(empty0 + 8 * (te % kEnt), (te / kEnt) & 1u);
          const unsigned m = __ballot_sync(0xffffffffu, freed);
          const int n = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
          if (n > 0) {
            const uint32_t last = (tail + n - 1) % kEnt;
            const uint32_t a0 = __shfl_sync(0xffffffffu, end0, last & 31), a1 = __shfl_sync(0xffffffffu, end1, last & 31);
            tail_abs = last & 32u ? a1 : a0;
            tail += n;
          } else {
            mbar_try_wait(empty0 + 8 * (tail % kEnt), (tail / kEnt) & 1u);   // suspends the warp until the oldest entry is free, or a while
            if (!__all_sync(0xffffffffu, keep_polling(ctl, it))) {
              rq.partial = __ballot_sync(0xffffffffu, lane < kCW && !todo);
              return;
            }
          }
        }
        A += total + pad;
        h = over ? total - excl0 : h + total;
        seq += kCW;
      }
    } else if (ph.type == PH_GDN) {
      // state slices by tensor copy; conv taps and weights into L2
#pragma unroll 1
      for (int i = 0; i < P.gdn_slots; i++) {
        const int item = c + i * gridDim.x;
        if (item >= P.Hv * 4) break;
        const int hv = item >> 2, hk = hv / (P.Hv / P.Hk), Cw = (2 * P.Hk + P.Hv) * 128;
        const uint32_t bar = smem_u32(smem + L.gfull) + 8 * i;
        // the previous layer's slice has left
        const uint32_t n = i ? rq.slices[1] : rq.slices[0];
        if (n > 0 && !__all_sync(0xffffffffu, wait_bar(smem_u32(smem + L.gfree) + 8 * i, (n - 1) & 1u, ctl))) return;
        (i ? rq.slices[1] : rq.slices[0]) = n + 1;
        if (lane == 0) {
          mbar_expect_tx(bar, kGdnBytes);
          asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                           smem_u32(smem + L.gdn) + (uint32_t)i * kGdnBytes),
                       "l"(ph.d.map), "r"((item & 3) * kGdnCols), "r"(hv * 128), "r"(bar)
                       : "memory");
        }
        const uint16_t* st = P.parity ? ph.d.cs[1] : ph.d.cs[0];
#pragma unroll 1
        for (int q = lane; q < 42; q += 32) {   // 3 channel groups: two lines of each of three taps, eight of weights
          const int what = q % 3, k3 = q / 3, ch = what == 0 ? hk * 128 : what == 1 ? (P.Hk + hk) * 128 : (2 * P.Hk + hv) * 128;
          if (k3 < 6) l2_prefetch(st + (size_t)(k3 >> 1) * Cw + ch + (k3 & 1) * 64);
          else l2_prefetch(ph.d.conv_w + (size_t)4 * ch + (k3 - 6) * 64);
        }
      }
    } else if (ph.type == PH_ATTN) {
      const int nsplits = pos / P.split_len + 1;
      if (c < nsplits * P.Hkv) {   // a row block that some CTA will read
        const int kvh = c % P.Hkv, split = c / P.Hkv;
        const size_t base = ((size_t)kvh * P.max_len + (size_t)split * P.split_len) * kHD;
        const int lines = min(min(P.split_len, pos + 1 - split * P.split_len), 64) * 4;
        for (int i = lane; i < lines; i += 32) {
          l2_prefetch(ph.a.kc + base + (size_t)i * 64);
          l2_prefetch(ph.a.vc + base + (size_t)i * 64);
        }
      }
    }
    __syncwarp();   // the descriptor has been read by every lane
    if (__any_sync(0xffffffffu, *ctl.dead)) return;
  }
}
// After a wait of this CTA has given up: the copies of the last entries and slices, before the CTA may end.
__device__ __noinline__ void producer_drain(uint32_t full0, uint32_t gfull0, Requested rq) {
  const int lane = threadIdx.x & 31;
  for (uint32_t slot = lane; slot < (uint32_t)kEnt; slot += 32) {
    const uint32_t i = (slot - rq.entries) % kEnt;   // (kEnt is a power of two)
    uint32_t n = rq.entries + i + 1;                 // the last entry in this slot, counted from one
    if (i >= 32 || !((rq.partial >> i) & 1u)) n = n > (uint32_t)kEnt ? n - kEnt : 0;
    if (n > 0) wait_landed(full0 + 8 * slot, ((n - 1) / kEnt) & 1u);
  }
  const uint32_t s = lane == 0 ? rq.slices[0] : lane == 1 ? rq.slices[1] : 0;
  if (s > 0) wait_landed(gfull0 + 8 * lane, (s - 1) & 1u);
}

// ---- consumer side ------------------------------------------------------------------------
// What cost most here were local-memory accesses: with 227 KB of shared memory there is hardly any L1, and the weight stream
// drives the stack's lines out of L2, so one spilled register in a phase's path is 330 cycles to several thousand (a version
// with spills in the row loop and a register array per query head took 1,100 us per step).  Hence registers few enough that
// nothing spills in the GEMV and GDN phases, loop-carried state in shared memory, and rolled loops with one variant of
// everything (a phase runs each of its instructions once per warp, so unrolled code is fetched anew every time).
struct Stage {
  uint32_t* xs;
  float *d8s, *s8s;
};
BK_DEVINL Stage stage_of(uint8_t* base, int K) {
  Stage s;
  s.xs = reinterpret_cast<uint32_t*>(base);
  s.d8s = reinterpret_cast<float*>(s.xs + (K / 64) * kUnitWords);
  s.s8s = s.d8s + K / 32;
  return s;
}
BK_DEVINL float max_nan(float a, float b) {   // a NaN wins
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}
// A block with a NaN or an infinity, or of values too small for a finite factor, as bk_q8_1_store has it: a NaN does not count for the
// maximum and becomes 0.  Out of line: it is hardly ever fetched.
__device__ __noinline__ uint4 stage8_general(float4 a, float4 c) {
  const float y[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
  const unsigned block = 0xfu << (threadIdx.x & 28u);
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; e++) amax = fmaxf(amax, fabsf(y[e]));
  amax = fmaxf(amax, __shfl_xor_sync(block, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(block, amax, 2));
  const float d = __fdiv_rn(amax, 127.0f), id = (d == 0.0f) ? 1.0f : __fdiv_rn(1.0f, d);
  uint32_t o[2] = {0u, 0u};
#pragma unroll
  for (int e = 0; e < 8; e++) o[e >> 2] |= ((uint32_t)max(-128, min(127, __float2int_rd(fmaf(y[e], id, 0.5f)))) & 0xffu) << (8 * (e & 3));
  return make_uint4(o[0], o[1], __float_as_uint(d), 0u);
}
// Chunk q of eight values -> Q8_1; four neighbouring lanes hold a block.
BK_DEVINL void stage8(const Stage& st, const float (&y)[8], int q) {
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; e++) amax = max_nan(amax, fabsf(y[e]));
  amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  float d = __fdiv_rn(amax, 127.0f);
  const float id = (d == 0.0f) ? 1.0f : __fdiv_rn(1.0f, d);
  // floor(y * id + 0.5), |.| <= 127: rounding down to the unit of 1.5 * 2^23 leaves it in the low byte
  uint32_t b[8];
#pragma unroll
  for (int e = 0; e < 8; e++) b[e] = __float_as_uint(__fadd_rd(fmaf(y[e], id, 0.5f), 12582912.0f));
  uint32_t w0 = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
  uint32_t w1 = __byte_perm(__byte_perm(b[4], b[5], 0x0040), __byte_perm(b[6], b[7], 0x0040), 0x5410);
  if (!(amax < INFINITY && id < INFINITY)) {
    const uint4 g = stage8_general(make_float4(y[0], y[1], y[2], y[3]), make_float4(y[4], y[5], y[6], y[7]));
    w0 = g.x;
    w1 = g.y;
    d = __uint_as_float(g.z);
  }
  int qsum = bk_dp4a_ss(w1, 0x01010101u, bk_dp4a_ss(w0, 0x01010101u, 0));
  qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
  qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
  const int blk = q >> 2;
  *reinterpret_cast<uint2*>(st.xs + (blk >> 1) * kUnitWords + (blk & 1) * 8 + (q & 3) * 2) = make_uint2(w0, w1);
  if ((q & 3) == 0) {
    const float d8 = bk_q8half_to_f32(bk_f32_to_f16_trunc(d));
    st.d8s[blk] = d8;
    st.s8s[blk] = __fmul_rn(d8, (float)qsum);
  }
}
// eight tagged words -> eight packed bf16
BK_DEVINL uint4 pack_words(const uint4& a, const uint4& b) {
  return make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410), __byte_perm(b.x, b.y, 0x5410), __byte_perm(b.z, b.w, 0x5410));
}

// chunk q of a Q4_K row dequantised to bf16 (bk_q4k_unit_to_bf16, eight values)
BK_DEVINL uint4 embed_chunk(const uint8_t* row, int q) {
  const uint8_t* sb = row + (size_t)(q >> 5) * 144;
  const int j = (q & 31) >> 2;
  const uint4 hdr = __ldg(reinterpret_cast<const uint4*>(sb));
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(sb + 16 + (j >> 1) * 32 + (q & 3) * 8));
  int sc, mn;
  bk_q4k_scale_min(hdr.y, hdr.z, hdr.w, j, sc, mn);
  const float dl = __fmul_rn(bk_f16_to_f32((uint16_t)(hdr.x & 0xffffu)), (float)sc), ml = __fmul_rn(bk_f16_to_f32((uint16_t)(hdr.x >> 16)), (float)mn);
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const uint32_t b = ((e < 4 ? w.x : w.y) >> (8 * (e & 3))) >> (4 * (j & 1));
    o[e >> 1] = bk_f32x2_to_bf16x2(__fsub_rn(__fmul_rn(dl, (float)(b & 15u)), ml), __fsub_rn(__fmul_rn(dl, (float)((b >> 8) & 15u)), ml));
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// the row of the token, dequantised by every CTA for itself; CTA 0 also stores it as the residual stream
BK_DEVINL void embed_row(const StepIO& io, uint8_t* xrow, uint32_t tag) {
  const int id = io.token >= 0 ? io.token : io.ids_in[0];
  const uint8_t* row = io.embed + (size_t)id * (io.H / 256) * 144;
  for (int q = threadIdx.x; q < io.H / 8; q += kCT) {
    const uint4 v = embed_chunk(row, q);
    reinterpret_cast<uint4*>(xrow)[q] = v;
    if (blockIdx.x == 0) {
      reinterpret_cast<uint4*>(io.x0)[q] = v;
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      for (int e = 0; e < 8; e++) st_t16(io.x_tagged + q * 8 + e, (uint16_t)(w[e >> 1] >> (16 * (e & 1))), tag);
    }
  }
}

// The activation of a GEMV phase into shared memory as Q8_1, eight values per thread and pass.  A normalised row is kept as
// bf16 in `xrow` while its sum of squares forms, in the canonical 256-thread order (chunk q of eight values belongs to thread
// q mod 256).
BK_DEVINL void stage_activation(const StepParams& P, const Phase& ph, const Stage& st, uint8_t* xrow, float* red, uint32_t base, const Ctl& ctl) {
  const int tid = threadIdx.x, K = ph.K, nchunk = K / 8;
  const bool norm = ph.in_kind != IN_PLAIN, embed = ph.in_kind == IN_EMBED;   // IN_EMBED: the row is in place (embed_row)
  const uint4* nw = static_cast<const uint4*>(ph.norm_w);
  const uint32_t* in = static_cast<const uint32_t*>(ph.in);
  const uint32_t th = (base + ph.in_tag) << 16;
  if (!embed && (tid & ~31) < nchunk) sentinel16(in + (size_t)(tid & ~31) * 8, th, ctl);
  uint4 wv = make_uint4(0, 0, 0, 0);
  if (norm && tid < nchunk) wv = ld_early(nw + tid);
  float rstd = 1.0f, acc = 0.0f;
  uint4 a = make_uint4(0, 0, 0, 0), b = a;   // a plain row's words, one pass ahead, and the first of a normalised one
  if (!embed && tid < nchunk) {
    a = ld_vec(in + (size_t)tid * 8);
    b = ld_vec(in + (size_t)tid * 8 + 4);
  }
  if (norm) {
#pragma unroll 1
    for (int q = tid; q < nchunk; q += kCT) {   // whole warps: nchunk is a multiple of 32
      uint4 v;
      if (!embed) {
        if (q != tid) {
          a = ld_vec(in + (size_t)q * 8);
          b = ld_vec(in + (size_t)q * 8 + 4);
        }
        wait_chunk(in, q, th, a, b, ctl);
        v = pack_words(a, b);
        reinterpret_cast<uint4*>(xrow)[q] = v;
      } else {
        v = reinterpret_cast<const uint4*>(xrow)[q];
      }
      float y[8];
      bf16x8(v, y);
#pragma unroll
      for (int e = 0; e < 8; e++) acc = fmaf(y[e], y[e], acc);
    }
    __syncwarp();
    acc = bk_warp_sum(acc);
    if ((tid & 31) == 0) red[tid >> 5] = acc;
    asm volatile("bar.sync 15, 256;" ::: "memory");
    const float4 r0 = *reinterpret_cast<const float4*>(red), r1 = *reinterpret_cast<const float4*>(red + 4);
    float total = __fadd_rn(__fadd_rn(__fadd_rn(r0.x, r0.y), r0.z), r0.w);
    total = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(total, r1.x), r1.y), r1.z), r1.w);
    rstd = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(total, (float)K), ph.eps));
  }
#pragma unroll 1
  for (int q = tid; q < nchunk; q += kCT) {
    float y[8];
    if (norm) {
      if (q != tid) wv = __ldg(nw + q);
      float w8[8];
      bf16x8(reinterpret_cast<const uint4*>(xrow)[q], y);
      bf16x8(wv, w8);
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const uint32_t pk = bk_f32x2_to_bf16x2(__fmul_rn(__fmul_rn(y[e], rstd), __fadd_rn(1.0f, w8[e])),
                                               __fmul_rn(__fmul_rn(y[e + 1], rstd), __fadd_rn(1.0f, w8[e + 1])));
        y[e] = __uint_as_float(pk << 16);
        y[e + 1] = __uint_as_float(pk & 0xffff0000u);
      }
    } else {
      uint4 na = a, nb = b;
      if (q + kCT < nchunk) {
        na = ld_vec(in + (size_t)(q + kCT) * 8);
        nb = ld_vec(in + (size_t)(q + kCT) * 8 + 4);
      }
      wait_chunk(in, q, th, a, b, ctl);
      bf16x8(pack_words(a, b), y);
      a = na;
      b = nb;
    }
    stage8(st, y, q);
  }
}

struct Best {
  float v;
  int i;
};
BK_DEVINL void best_merge(Best& b, float ov, int oi) {
  if (ov > b.v || (ov == b.v && oi < b.i)) {
    b.v = ov;
    b.i = oi;
  }
}

// One row group (up to 16 rows): dots from the ring kBlock rows at a time, lane sums in `accs` (per-warp shared
// memory), then a few lanes per row add them up in the order of the 16,8,4,2,1 butterfly, and the epilogue.
template <int N>
BK_DEVINL void row_block(const uint8_t* row, uint32_t even, uint32_t odd, uint32_t last, const XRegs& xr, int u, bool first, bool live, float* acc) {
  // rows 2i, 2i+1 of the block at row + i * even (+ odd); the last one, which may be missing, at row + last
  RowRegs q[N];
#pragma unroll
  for (int i = 0; i < N; i++) q[i] = load_unit_smem(row + (i == N - 1 ? last : (i >> 1) * even + (i & 1) * odd), u);
  float old[N];
#pragma unroll
  for (int i = 0; i < N; i++) old[i] = first ? 0.0f : acc[i * kAccPitch];
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float v = unit_val(decode_unit(q[i], u & 3), xr);
    acc[i * kAccPitch] = live ? __fadd_rn(old[i], v) : old[i];
  }
}
BK_DEVINL void group_rows(const StepParams& P, const Phase& ph, const Stage& st, const uint8_t* wbase, uint32_t empty_bar, float* accs, int v0, int nr,
                          uint32_t base, const Ctl& ctl, Best* best) {
  const int lane = threadIdx.x & 31, nunits = ph.K / 64, nblk = ph.K / 32;
  const uint32_t rowb = (uint32_t)(ph.K / 256) * 144;
  const bool swiglu = ph.swiglu != 0;
  // where the row this lane will report goes; its residual is requested before the dots
  const int ri = lane / kLanesPerRow;
  const bool mine = (lane & (kLanesPerRow - 1)) == 0 && ri < nr;
  int n = swiglu ? (v0 + ri) >> 1 : v0 + ri, epi = ph.g.segs[0].epi;
  void* out = ph.g.segs[0].out;
  uint32_t res_word = 0;
  if (mine && epi == OUT_ADD) res_word = ld_word(ph.res + n);
  // gate and up rows of a pair lie half a group apart, other rows follow one another
  const uint32_t even = swiglu ? rowb : 2 * rowb, odd = swiglu ? (uint32_t)(nr >> 1) * rowb : rowb;
  if (nr == 1) {   // one row: two passes over its units side by side
    float sum = 0.0f;
#pragma unroll 1
    for (int u = lane; u - lane < nunits; u += 64) {
      const int u0 = min(u, nunits - 1), u1 = min(u + 32, nunits - 1);
      const RowRegs q0 = load_unit_smem(wbase, u0), q1 = load_unit_smem(wbase, u1);
      const XRegs x0 = load_x(st.xs, st.d8s, st.s8s, 0, u0, nunits, nblk), x1 = load_x(st.xs, st.d8s, st.s8s, 0, u1, nunits, nblk);
      const float f0 = unit_val(decode_unit(q0, u0 & 3), x0), f1 = unit_val(decode_unit(q1, u1 & 3), x1);
      if (u < nunits) sum = __fadd_rn(sum, f0);
      if (u + 32 < nunits) sum = __fadd_rn(sum, f1);
    }
    accs[lane] = sum;
  }
#pragma unroll 1
  for (int u = lane; u - lane < nunits && nr > 1; u += 32) {   // whole warps
    const int uc = min(u, nunits - 1);   // a lane without a unit repeats the last one and adds nothing
    const XRegs xr = load_x(st.xs, st.d8s, st.s8s, 0, uc, nunits, nblk);
    const uint8_t* row = wbase;
    float* acc = accs + lane;
    int r = 0;
#pragma unroll 1
    for (; r + kBlock / 2 < nr; r += kBlock) {   // (for a missing last row the one before is computed again)
      row_block<kBlock>(row, even, odd, (kBlock / 2 - 1) * even + (r + kBlock - 1 < nr ? odd : 0), xr, uc, u == lane, u < nunits, acc);
      row += (kBlock / 2) * even;
      acc += kBlock * kAccPitch;
    }
    if (r < nr) row_block<2>(row, even, odd, r + 1 < nr ? odd : 0, xr, uc, u == lane, u < nunits, acc);
  }
  __syncwarp();   // every lane has read the group
  if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar) : "memory");
  // kLanesPerRow lanes per row
  const uint32_t tag = base + ph.out_tag;
  const float* v = accs + ri * kAccPitch + (lane & (kLanesPerRow - 1));
  constexpr int kT = 16 / kLanesPerRow;
  float t[kT];
#pragma unroll
  for (int i = 0; i < kT; i++) t[i] = __fadd_rn(v[kLanesPerRow * i], v[kLanesPerRow * i + 16]);
#pragma unroll
  for (int n = kT / 2; n >= 1; n >>= 1)
#pragma unroll
    for (int i = 0; i < n; i++) t[i] = __fadd_rn(t[i], t[i + n]);
  float y = t[0];
#pragma unroll
  for (int off = kLanesPerRow / 2; off >= 1; off >>= 1) y = __fadd_rn(y, __shfl_xor_sync(0xffffffffu, y, off));
  const float yup = __shfl_xor_sync(0xffffffffu, y, kLanesPerRow);   // the odd neighbour row
#pragma unroll 1
  for (int s = 1; s < ph.n_segs; s++)
    if (v0 + ri >= ph.g.segs[s].vrow_begin) {
      n = v0 + ri - ph.g.segs[s].vrow_begin;
      epi = ph.g.segs[s].epi;
      out = ph.g.segs[s].out;
    }
  if (mine) {
    if (epi == OUT_LOGITS) {
      static_cast<float*>(out)[n] = y;
      best_merge(best[ri], y, n);
    } else if (epi == OUT_T32) {
      st_t32(static_cast<unsigned long long*>(out) + n, y, tag);
    } else if (!(swiglu && (ri & 1))) {
      float o = y;
      if (swiglu) o = __fmul_rn(__fmul_rn(y, bk_sigmoidf(y)), yup);
      if (epi == OUT_ADD) o = __fadd_rn(y, __uint_as_float(wait_word(ph.res + n, res_word, base + ph.res_tag, ctl) << 16));
      const uint16_t h = bk_f32_to_bf16(o);
      st_t16(static_cast<uint32_t*>(out) + n, h, tag);
      if (epi == OUT_ADD && ph.plain) ph.plain[n] = h;
    }
  }
  __syncwarp();
}

// ---- conv1d + gated DeltaNet -----------------------------------------------------------------
// An item is a quarter of a value head's state columns, taken by four warps (warp r: rows 32r..32r+31, lane: column), so
// that 32 heads spread over 128 SMs; the order within a column is that of gdn_step_body (bk_gdn.cuh).  The q and k
// convolutions and norms of a head are repeated by its four items.  The gated norm needs all 128 columns: the items exchange
// the eight lane sums each of them contributes.  The state slice comes and goes by tensor copies through shared memory: as
// 64 KB of plain stores by 32 SMs it held up everything these SMs stored or loaded next (4 us).
struct GdnScratch {
  float q[128], k[128], v[kGdnCols], zs[kGdnCols];
  float qn[128], kn[128];
  float part[4][kGdnCols], part2[4][kGdnCols];
  float gate[2], pad[2];
};
BK_DEVINL void phase_gdn(const StepParams& P, const Phase& ph, uint8_t* smem, const SmemLayout& L, uint32_t n_gdn, uint32_t base, const Ctl& ctl) {
  const int tid = threadIdx.x, lane = tid & 31, quad = tid >> 7, r = (tid >> 5) & 3, t = tid & 127;
  const int item = blockIdx.x + quad * gridDim.x;
  if (quad >= P.gdn_slots || item >= P.Hv * 4) return;
  GdnScratch& sm = reinterpret_cast<GdnScratch*>(smem + L.scratch)[quad];
  const int ratio = P.Hv / P.Hk, keydim = P.Hk * 128, C = 2 * keydim + P.Hv * 128, hv = item >> 2, cq = item & 3, hk = hv / ratio;
  const uint32_t tag = base + ph.in_tag;
  const GdnPart& d = ph.d;
  const uint16_t* cs_in = P.parity ? d.cs[1] : d.cs[0];
  uint16_t* cs_new = P.parity ? d.cs[0] : d.cs[1];
  auto quad_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(2 + quad) : "memory"); };
  // channels of this thread: a q, a k, and in the first warp a v
  const int ch[3] = {hk * 128 + t, keydim + hk * 128 + t, 2 * keydim + hv * 128 + cq * kGdnCols + lane};
  uint16_t h0[3], h1[3], h2[3];
  uint2 cw[3];
  uint32_t x[3];
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (c < 2 || r == 0) {
      h0[c] = cs_in[ch[c]];
      h1[c] = cs_in[C + ch[c]];
      h2[c] = cs_in[2 * C + ch[c]];
      cw[c] = __ldg(reinterpret_cast<const uint2*>(d.conv_w + 4 * (size_t)ch[c]));
    }
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (c < 2 || r == 0) x[c] = ld_word(d.qkv + ch[c]);
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (c < 2 || r == 0) {
      const uint16_t hx = (uint16_t)wait_word(d.qkv + ch[c], x[c], tag, ctl);
      const float w0 = __uint_as_float(cw[c].x << 16), w1 = __uint_as_float(cw[c].x & 0xffff0000u);
      const float w2 = __uint_as_float(cw[c].y << 16), w3 = __uint_as_float(cw[c].y & 0xffff0000u);
      const float raw = __fadd_rn(__fadd_rn(__fmul_rn(w0, bk_bf16_to_f32(h0[c])), __fmul_rn(w1, bk_bf16_to_f32(h1[c]))),
                                  __fadd_rn(__fmul_rn(w2, bk_bf16_to_f32(h2[c])), __fmul_rn(w3, bk_bf16_to_f32(hx))));
      (c == 0 ? sm.q : c == 1 ? sm.k : sm.v)[c < 2 ? t : lane] = bk_bf16_to_f32(bk_f32_to_bf16(__fmul_rn(raw, bk_sigmoidf(raw))));
      if (c == 2 || (hv % ratio == 0 && cq == 0)) {   // q/k channels are shared: the first item of `ratio` heads writes
        cs_new[ch[c]] = h1[c];
        cs_new[C + ch[c]] = h2[c];
        cs_new[2 * C + ch[c]] = hx;
      }
    }
  if (r == 1) {   // z * sigmoid(z)
    const uint32_t* zp = d.z + hv * 128 + cq * kGdnCols + lane;
    const float zv = __uint_as_float(wait_word(zp, ld_word(zp), tag, ctl) << 16);
    sm.zs[lane] = __fmul_rn(zv, bk_sigmoidf(zv));
  } else if (r == 2) {   // gates
    const float alog = __ldg(d.A_log + hv), dtb = bk_bf16_to_f32(__ldg(d.dt_bias + hv));
    uint2 av, bv;
    for (int it = 0;; it++) {
      av = ld_pair(d.a + hv);
      bv = ld_pair(d.b + hv);
      if (!((av.y ^ tag) | (bv.y ^ tag)) || !keep_polling(ctl, it)) break;
    }
    const float sp = bk_softplusf(__fadd_rn(__uint_as_float(av.x), dtb));
    const float g0 = bk_expf(-__fmul_rn(bk_expf(alog), sp)), g1 = bk_sigmoidf(__uint_as_float(bv.x));
    if (lane == 0) {
      sm.gate[0] = g0;
      sm.gate[1] = g1;
    }
  }
  quad_sync();
  {   // L2 norms, by every warp for itself; its 32 rows of k and q scaled
    const float4 q4 = *reinterpret_cast<const float4*>(sm.q + lane * 4), k4 = *reinterpret_cast<const float4*>(sm.k + lane * 4);
    float aq = 0.0f, ak = 0.0f;
    aq = fmaf(q4.x, q4.x, aq); aq = fmaf(q4.y, q4.y, aq); aq = fmaf(q4.z, q4.z, aq); aq = fmaf(q4.w, q4.w, aq);
    ak = fmaf(k4.x, k4.x, ak); ak = fmaf(k4.y, k4.y, ak); ak = fmaf(k4.z, k4.z, ak); ak = fmaf(k4.w, k4.w, ak);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      aq = __fadd_rn(aq, __shfl_xor_sync(0xffffffffu, aq, off));
      ak = __fadd_rn(ak, __shfl_xor_sync(0xffffffffu, ak, off));
    }
    sm.qn[t] = __fmul_rn(sm.q[t], __fmul_rn(bk_rcp_sqrt(__fadd_rn(aq, 1e-6f)), 0.088388347648318441f));
    sm.kn[t] = __fmul_rn(sm.k[t], bk_rcp_sqrt(__fadd_rn(ak, 1e-6f)));
    __syncwarp();
  }
  wait_bar(smem_u32(smem + L.gfull) + 8 * quad, n_gdn & 1u, ctl);
  float* S = reinterpret_cast<float*>(smem + L.gdn + (size_t)quad * kGdnBytes) + 32 * r * kGdnCols + lane;
  float sd[32];
#pragma unroll
  for (int i = 0; i < 32; i++) sd[i] = S[i * kGdnCols];
  const float4 *kn4 = reinterpret_cast<const float4*>(sm.kn + 32 * r), *qn4 = reinterpret_cast<const float4*>(sm.qn + 32 * r);
  const float decay = sm.gate[0], beta = sm.gate[1];
  float acc = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (i == 4) asm volatile("" ::: "memory");   // bounds the registers
    const float4 k4 = kn4[i];
    sd[4 * i] = __fmul_rn(sd[4 * i], decay);
    sd[4 * i + 1] = __fmul_rn(sd[4 * i + 1], decay);
    sd[4 * i + 2] = __fmul_rn(sd[4 * i + 2], decay);
    sd[4 * i + 3] = __fmul_rn(sd[4 * i + 3], decay);
    acc = fmaf(k4.x, sd[4 * i], acc);
    acc = fmaf(k4.y, sd[4 * i + 1], acc);
    acc = fmaf(k4.z, sd[4 * i + 2], acc);
    acc = fmaf(k4.w, sd[4 * i + 3], acc);
  }
  sm.part[r][lane] = acc;
  quad_sync();
  const float kS = __fadd_rn(__fadd_rn(__fadd_rn(sm.part[0][lane], sm.part[1][lane]), sm.part[2][lane]), sm.part[3][lane]);
  const float delta = __fmul_rn(__fsub_rn(sm.v[lane], kS), beta);
  acc = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if ((i & 1) == 0) asm volatile("" ::: "memory");
    const float4 k4 = kn4[i], q4 = qn4[i];
    sd[4 * i] = fmaf(k4.x, delta, sd[4 * i]);
    sd[4 * i + 1] = fmaf(k4.y, delta, sd[4 * i + 1]);
    sd[4 * i + 2] = fmaf(k4.z, delta, sd[4 * i + 2]);
    sd[4 * i + 3] = fmaf(k4.w, delta, sd[4 * i + 3]);
    acc = fmaf(q4.x, sd[4 * i], acc);
    acc = fmaf(q4.y, sd[4 * i + 1], acc);
    acc = fmaf(q4.z, sd[4 * i + 2], acc);
    acc = fmaf(q4.w, sd[4 * i + 3], acc);
  }
  sm.part2[r][lane] = acc;
#pragma unroll
  for (int i = 0; i < 32; i++) S[i * kGdnCols] = sd[i];
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slice leaves through the async proxy
  quad_sync();
  if (r == 0) {
    const float o = __fadd_rn(__fadd_rn(__fadd_rn(sm.part2[0][lane], sm.part2[1][lane]), sm.part2[2][lane]), sm.part2[3][lane]);
    // canonical lane 8cq + i of the head's norm holds columns 4i..4i+3 of this item; i = lane / 4
    const int i0 = lane & ~3;
    float a2 = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float oe = __shfl_sync(0xffffffffu, o, i0 + e);
      a2 = fmaf(oe, oe, a2);
    }
    unsigned long long* sums = d.sums + (size_t)hv * 32;
    if ((lane & 3) == 0) st_t32(sums + cq * 8 + (lane >> 2), a2, base + ph.out_tag);
    const unsigned long long* sp = sums + (lane & 3) * 8 + (lane >> 2);   // item lane & 3
    uint2 w = ld_pair(sp);
    for (int it = 0; w.y != base + ph.out_tag; it++) {
      if (!keep_polling(ctl, it)) break;
      w = ld_pair(sp);
    }
    __syncwarp();
    const float v = __uint_as_float(w.x);
    const float v0 = __shfl_sync(0xffffffffu, v, i0), v1 = __shfl_sync(0xffffffffu, v, i0 + 1), v2 = __shfl_sync(0xffffffffu, v, i0 + 2),
                v3 = __shfl_sync(0xffffffffu, v, i0 + 3);
    float tot = __fadd_rn(__fadd_rn(v0, v2), __fadd_rn(v1, v3));   // butterfly levels 16 and 8
    tot = __fadd_rn(tot, __shfl_xor_sync(0xffffffffu, tot, 16));   // levels 4, 2, 1
    tot = __fadd_rn(tot, __shfl_xor_sync(0xffffffffu, tot, 8));
    tot = __fadd_rn(tot, __shfl_xor_sync(0xffffffffu, tot, 4));
    const float rstd = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(tot, 128.0f), 1e-6f));
    const int n = cq * kGdnCols + lane;
    const float ow = __fmul_rn(__fmul_rn(o, rstd), __ldg(d.norm_w + n));
    st_t16(d.o + hv * 128 + n, bk_f32_to_bf16(__fmul_rn(ow, sm.zs[lane])), base + ph.out_tag);
  } else if (t == 32) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(d.map), "r"(cq * kGdnCols), "r"(hv * 128),
                 "r"(smem_u32(smem + L.gdn) + (uint32_t)quad * kGdnBytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}

// ---- attention ---------------------------------------------------------------------------------
// An item is (split of the cache rows, KV head, pair of the query heads that share it): short caches are cut by heads as well,
// long ones read their rows once per pair, from L2 after the first.  The orders are those of attn_split_kernel (bk_attn.cu):
// lane l owns dims 8l..8l+7 of a score; rows jj mod 8 form eight classes whose p*V sums are chains, added in class order.
__host__ __device__ constexpr size_t attn_item_bytes(int split_len) { return 2 * 512 + 1024 + (size_t)split_len * 8 + (size_t)8 * 2 * kHD * 4; }

BK_DEVINL void attn_items(const StepParams& P, const Phase& ph, uint8_t* scratch, uint32_t base, const Ctl& ctl, int pos) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = P.Hq / P.Hkv, pairs = (G + 1) / 2, nsplits = pos / P.split_len + 1, n_items = nsplits * P.Hkv * pairs;
  const uint32_t th = (base + ph.in_tag) << 16, tag = base + ph.out_tag;
  uint16_t* q_s = reinterpret_cast<uint16_t*>(scratch);       // [2][256], then the new key and value rows
  const uint16_t *k_st = q_s + 2 * kHD, *v_st = q_s + 3 * kHD;
  float2* s_s = reinterpret_cast<float2*>(q_s + 4 * kHD);     // [split_len] scores of the two heads
  float2* ex = s_s + P.split_len;                             // [8 classes][256 dims] of the two heads
  const AttnPart& a = ph.a;
#pragma unroll 1
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int pr = item % pairs, rest = item / pairs, kvh = rest % P.Hkv, split = rest / P.Hkv;
    const int h0 = kvh * G + 2 * pr, nh = 2 * pr + 1 < G ? 2 : 1;
    const int j0 = split * P.split_len, ns = min(pos + 1, j0 + P.split_len) - j0, jp = pos - j0;
    uint16_t* Kb = a.kc + ((size_t)kvh * P.max_len + j0) * kHD;
    uint16_t* Vb = a.vc + ((size_t)kvh * P.max_len + j0) * kHD;
    // cached rows of earlier steps: requested before this token's projections are waited for
    uint4 kc[4];
    constexpr int kCls = 32 / kCW;
    uint32_t vv[8];
    const int db = warp & 3, cls0 = (warp >> 2) * kCls, dim = 64 * db + 2 * lane;   // 64 dims and kCls row classes
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int jj = warp + kCW * i;
      kc[i] = (jj < ns && jj != jp) ? *reinterpret_cast<const uint4*>(Kb + (size_t)jj * kHD + lane * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {   // class cls0 + i mod kCls, its row i / kCls
      const int jj = cls0 + i % kCls + 8 * (i / kCls);
      vv[i] = (jj < ns && jj != jp) ? *reinterpret_cast<const uint32_t*>(Vb + (size_t)jj * kHD + dim) : 0u;
    }
    const bool owner = jp >= 0 && jp < ns;   // this split holds the new row
    if (warp < nh || (owner && (warp == 2 || warp == 3))) {
      const uint32_t* src = warp < 2 ? a.qg + (size_t)(h0 + warp) * 2 * kHD : (warp == 2 ? a.k : a.v) + (size_t)kvh * kHD;
      uint4 u, v;
      for (int it = 0;; it++) {
        u = ld_vec(src + lane * 8);
        v = ld_vec(src + lane * 8 + 4);
        if (!(stale16(u, th) | stale16(v, th)) || !keep_polling(ctl, it)) break;
      }
      __syncwarp();
      uint4 w = pack_words(u, v);
      uint16_t* stage = q_s + warp * kHD;
      if (warp != 3) {   // head norm and rotary on q and k
        float x[8], wv[8];
        bf16x8(w, x);
        bf16x8(__ldg(reinterpret_cast<const uint4*>((warp < 2 ? a.q_norm_w : a.k_norm_w) + lane * 8)), wv);
        float acc = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; e++) acc = fmaf(x[e], x[e], acc);
        acc = bk_warp_sum(acc);
        const float rstd = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(acc, (float)kHD), 1e-6f));
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 8; e += 2)
          o[e >> 1] = bk_f32x2_to_bf16x2(__fmul_rn(__fmul_rn(x[e], rstd), __fadd_rn(1.0f, wv[e])),
                                         __fmul_rn(__fmul_rn(x[e + 1], rstd), __fadd_rn(1.0f, wv[e + 1])));
        *reinterpret_cast<uint4*>(stage + lane * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        __syncwarp();
#pragma unroll 1
        for (int i = lane; i < P.rot_half; i += 32) {
          const float x1 = bk_bf16_to_f32(stage[i]), x2 = bk_bf16_to_f32(stage[i + P.rot_half]);
          const float c = P.cos_t[(size_t)pos * P.rot_half + i], s = P.sin_t[(size_t)pos * P.rot_half + i];
          stage[i] = bk_f32_to_bf16(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
          stage[i + P.rot_half] = bk_f32_to_bf16(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s)));
        }
        __syncwarp();
        w = *reinterpret_cast<const uint4*>(stage + lane * 8);
      } else {
        *reinterpret_cast<uint4*>(stage + lane * 8) = w;
      }
      if (warp >= 2 && pr == 0) *reinterpret_cast<uint4*>((warp == 2 ? Kb : Vb) + (size_t)jp * kHD + lane * 8) = w;   // append
    }
    consumers_sync();
    {   // scores: one packed FMA advances both heads' chains
      float2 qp[8];
      {
        float q0[8], q1[8];
        bf16x8(*reinterpret_cast<const uint4*>(q_s + lane * 8), q0);
        bf16x8(*reinterpret_cast<const uint4*>(q_s + (nh - 1) * kHD + lane * 8), q1);
#pragma unroll
        for (int e = 0; e < 8; e++) qp[e] = make_float2(q0[e], q1[e]);
      }
#pragma unroll 1
      for (int i0 = 0; warp + kCW * i0 < ns; i0 += 4) {   // four rows at a time
        float2 s2[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          float kf[8];
          bf16x8(warp + kCW * (i0 + i) == jp ? *reinterpret_cast<const uint4*>(k_st + lane * 8) : kc[i], kf);
          const int jn = warp + kCW * (i0 + 4 + i);   // the next four are on their way meanwhile
          kc[i] = (jn < ns && jn != jp) ? *reinterpret_cast<const uint4*>(Kb + (size_t)jn * kHD + lane * 8) : make_uint4(0, 0, 0, 0);
          s2[i] = make_float2(0.0f, 0.0f);
#pragma unroll
          for (int e = 0; e < 8; e++) s2[i] = bk_fma2(qp[e], make_float2(kf[e], kf[e]), s2[i]);
        }
        // eight sums (row i, head) over the warp: value index 4*bit4 + 2*bit3 + bit2 of the lane
        const float v8[8] = {s2[0].x, s2[0].y, s2[1].x, s2[1].y, s2[2].x, s2[2].y, s2[3].x, s2[3].y};
        const float y = warp_sum8(v8);
        const int vi = lane >> 2, jj = warp + kCW * (i0 + (vi >> 1));
        if ((lane & 3) == 0 && jj < ns) reinterpret_cast<float*>(s_s + jj)[vi & 1] = __fmul_rn(y, P.scale);
      }
    }
    consumers_sync();
    if (warp < nh) {   // exact max, p = exp(s - m), class sums of p: one warp per head
      float* sh = reinterpret_cast<float*>(s_s) + warp;
      float m = -INFINITY;
#pragma unroll 1
      for (int jj = lane; jj < ns; jj += 32) m = fmaxf(m, sh[2 * jj]);
      m = bk_warp_max(m);
#pragma unroll 1
      for (int jj = lane; jj < ns; jj += 32) sh[2 * jj] = bk_expf(__fsub_rn(sh[2 * jj], m));
      __syncwarp();
      float lw = 0.0f;
      if (lane < 8) {
#pragma unroll 1
        for (int jj = lane; jj < ns; jj += 8) lw = __fadd_rn(lw, sh[2 * jj]);
      }
      float l = __shfl_sync(0xffffffffu, lw, 0);
#pragma unroll
      for (int c = 1; c < 8; c++) l = __fadd_rn(l, __shfl_sync(0xffffffffu, lw, c));
      if (lane < 2) st_t32(P.pml + ((size_t)(h0 + warp) * P.max_splits + split) * 2 + lane, lane == 0 ? m : l, tag);
    }
    consumers_sync();
    {   // kCls row classes of this warp, two dims per lane, both heads side by side
      float2 acc[kCls][2];   // [class][dim]
#pragma unroll
      for (int c = 0; c < kCls; c++) acc[c][0] = acc[c][1] = make_float2(0.0f, 0.0f);
      constexpr int kRows = 8 / kCls;
#pragma unroll 1
      for (int i0 = 0; cls0 + 8 * i0 < ns; i0 += kRows) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int jj = cls0 + i % kCls + 8 * (i0 + i / kCls), jn = jj + 8 * kRows;
          const uint32_t w = jj == jp ? *reinterpret_cast<const uint32_t*>(v_st + dim) : vv[i];
          vv[i] = (jn < ns && jn != jp) ? *reinterpret_cast<const uint32_t*>(Vb + (size_t)jn * kHD + dim) : 0u;   // the next rows are on their way
          if (jj < ns) {
            const float va = __uint_as_float(w << 16), vb = __uint_as_float(w & 0xffff0000u);
            const float2 p2 = s_s[jj];
            acc[i % kCls][0] = bk_fma2(p2, make_float2(va, va), acc[i % kCls][0]);
            acc[i % kCls][1] = bk_fma2(p2, make_float2(vb, vb), acc[i % kCls][1]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < kCls; c++)
        *reinterpret_cast<float4*>(ex + (size_t)(cls0 + c) * kHD + dim) = make_float4(acc[c][0].x, acc[c][0].y, acc[c][1].x, acc[c][1].y);
    }
    consumers_sync();
    if (tid < kHD) {
      float2 o = ex[tid];
#pragma unroll
      for (int c = 1; c < 8; c++) {
        const float2 e2 = ex[(size_t)c * kHD + tid];
        o = make_float2(__fadd_rn(o.x, e2.x), __fadd_rn(o.y, e2.y));
      }
      unsigned long long* po = P.po + ((size_t)h0 * P.max_splits + split) * kHD + tid;
      st_t32(po, o.x, tag);
      if (nh == 2) st_t32(po + (size_t)P.max_splits * kHD, o.y, tag);
    }
    consumers_sync();   // the scratch belongs to the next item
  }
}

// merge the splits of a head: M = max m_s, w_s = exp(m_s - M), L and O chains in ascending s, out = (O / L) * sigmoid(gate)
BK_DEVINL void phase_merge(const StepParams& P, const Phase& ph, uint8_t* scratch, uint32_t base, const Ctl& ctl, int pos) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int ns = pos / P.split_len + 1;
  const uint32_t tag = base + ph.in_tag;
  float* m_s = reinterpret_cast<float*>(scratch);
  float* l_s = m_s + P.max_splits;
  float* w_s = l_s + P.max_splits;
#pragma unroll 1
  for (int h = (int)gridDim.x - 1 - (int)blockIdx.x; h < P.Hq; h += gridDim.x) {
#pragma unroll 1
    for (int s = tid; s < ns; s += kCT) {
      const unsigned long long* ml = P.pml + ((size_t)h * P.max_splits + s) * 2;
      uint2 m, l;
      for (int it = 0;; it++) {
        m = ld_pair(ml);
        l = ld_pair(ml + 1);
        if (!((m.y ^ tag) | (l.y ^ tag)) || !keep_polling(ctl, it)) break;
      }
      m_s[s] = __uint_as_float(m.x);
      l_s[s] = __uint_as_float(l.x);
    }
    consumers_sync();
    float m = -INFINITY;
#pragma unroll 1
    for (int s = lane; s < ns; s += 32) m = fmaxf(m, m_s[s]);
    const float M = bk_warp_max(m);
#pragma unroll 1
    for (int s = tid; s < ns; s += kCT) w_s[s] = bk_expf(__fsub_rn(m_s[s], M));
    consumers_sync();
    if (tid < kHD) {
      const unsigned long long* po = P.po + (size_t)h * P.max_splits * kHD + tid;
      const uint32_t* gate = ph.a.qg + (size_t)h * 2 * kHD + kHD + tid;
      const uint32_t g0 = ld_word(gate);
      float Ls = 0.0f, O = 0.0f;
#pragma unroll 1
      for (int s0 = 0; s0 < ns; s0 += 4) {
        uint2 v[4];
        for (int it = 0;; it++) {
          uint32_t bad = 0;
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (s0 + i < ns) v[i] = ld_pair(po + (size_t)(s0 + i) * kHD);
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (s0 + i < ns) bad |= v[i].y ^ tag;
          if (!bad || !keep_polling(ctl, it)) break;
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (s0 + i < ns) {
            const float w = w_s[s0 + i];
            Ls = fmaf(w, l_s[s0 + i], Ls);
            O = fmaf(w, __uint_as_float(v[i].x), O);
          }
      }
      const float gf = __uint_as_float(wait_word(gate, g0, tag, ctl) << 16);
      st_t16(P.attn_out + (size_t)h * kHD + tid, bk_f32_to_bf16(__fmul_rn(__fdiv_rn(O, Ls), bk_sigmoidf(gf))), base + ph.out_tag);
    }
    consumers_sync();
  }
}

__global__ void __launch_bounds__(kPT, 1) decode_step_kernel(const __grid_constant__ StepParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const SmemLayout L = smem_layout(P.xs_bytes, P.scratch_bytes, P.gdn_bytes, P.ring_bytes);
  int* misc = reinterpret_cast<int*>(smem + L.misc);
  const Ctl ctl = {misc, P.status, P.polls};
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kDescVec = (int)(sizeof(Phase) / 16);
  if (tid == 0) {
    misc[0] = 0;
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(smem + L.gfull) + 8 * i, 1);
      mbar_init(smem_u32(smem + L.gfree) + 8 * i, 1);
    }
    for (int e = 0; e < kEnt; e++) {
      mbar_init(smem_u32(smem + L.full) + 8 * e, 1);
      mbar_init(smem_u32(smem + L.empty) + 8 * e, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid < kEnt) reinterpret_cast<uint32_t*>(smem + L.ent)[tid] = 0u;
  for (int i = tid; i < 2 * kDescVec && i < P.n_phases * kDescVec; i += kPT)
    reinterpret_cast<uint4*>(smem + L.desc)[i] = __ldg(reinterpret_cast<const uint4*>(P.phases) + i);
  const unsigned int ep = *reinterpret_cast<const volatile unsigned int*>(P.epoch);
  const int pos = *reinterpret_cast<const volatile int*>(P.io.pos);
  const uint32_t base = (ep + 1u) * (uint32_t)P.tags;
  __syncthreads();
  if (warp == kCW) {
    Requested rq = {0, 0, {0, 0}};
    producer_warp(P, smem, L, ctl, pos, rq);
    if (__any_sync(0xffffffffu, *ctl.dead)) producer_drain(smem_u32(smem + L.full), smem_u32(smem + L.gfull), rq);
    return;
  }

  embed_row(P.io, smem + L.scratch, base);
  Best* best_s = reinterpret_cast<Best*>(smem + L.best);
  if (tid < kCW * kGroupMax) best_s[tid] = Best{-INFINITY, 0x7fffffff};
  for (int k = 0; k < P.n_phases; k++) {
    const Phase& ph = *reinterpret_cast<const Phase*>(smem + L.desc + (size_t)(k % kWin) * sizeof(Phase));
    uint4 next_desc = make_uint4(0, 0, 0, 0);
    const bool fetch = warp == 0 && lane < kDescVec && k + 2 < P.n_phases;
    if (fetch) next_desc = ld_early(reinterpret_cast<const uint4*>(P.phases + k + 2) + lane);
    unsigned long long* trec = (P.trace && blockIdx.x == 0 && tid == 0) ? P.trace + (size_t)k * 8 : nullptr;
    if (trec) trec[0] = global_timer();
    if (ph.type == PH_GEMV) {
      const Share s = cta_share(ph);
      const Stage st = stage_of(smem + L.xs + (ph.buffer ? P.xs0_bytes : 0), ph.K);
      float* red = reinterpret_cast<float*>(smem + L.red);
      const uint32_t entry = ph.entry + warp;
      bool landed = mbar_test(smem_u32(smem + L.full) + 8 * (entry % kEnt), (entry / kEnt) & 1u);   // weights are usually there by now
      if (s.n > 0) stage_activation(P, ph, st, smem + L.scratch, red, base, ctl);
      consumers_sync();
      if (trec) trec[1] = global_timer();
#pragma unroll 1
      for (int r = 0; r < s.R; r++) {
        const uint32_t e = (entry + r * kCW) % kEnt, parity = ((entry + r * kCW) / kEnt) & 1u;
        int g0, g1;
        group_range(s, r, warp, g0, g1);
        if (!landed) wait_bar(smem_u32(smem + L.full) + 8 * e, parity, ctl);
        landed = false;
        const uint32_t off = reinterpret_cast<const volatile uint32_t*>(smem + L.ent)[e];   // (after giving up: of any group, or 0)
        group_rows(P, ph, st, smem + L.ring + off, smem_u32(smem + L.empty) + 8 * e, reinterpret_cast<float*>(smem + L.accs) + warp * kGroupMax * kAccPitch,
                                     (s.u0 + g0) * s.upr, (g1 - g0) * s.upr, base, ctl, best_s + warp * kGroupMax);
      }
      if (ph.gdn_index && tid < 256 && (tid & 127) == 32) {   // the thread that sent a state slice gives the buffer back
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(smem + L.gfree) + 8 * (tid >> 7)) : "memory");
      }
    } else if (ph.type == PH_GDN) {
      phase_gdn(P, ph, smem, L, ph.gdn_index, base, ctl);
      consumers_sync();
    } else if (ph.type == PH_ATTN) {
      attn_items(P, ph, smem + L.scratch, base, ctl, pos);
      consumers_sync();
    } else {
      phase_merge(P, ph, smem + L.scratch, base, ctl, pos);
      consumers_sync();
    }
    // the descriptor two phases ahead replaces that of two phases ago (every warp has passed a barrier since it was read)
    if (fetch) reinterpret_cast<uint4*>(smem + L.desc + (size_t)((k + 2) % kWin) * sizeof(Phase))[lane] = next_desc;
    if (trec) trec[2] = global_timer();
    if (P.trace && lane == 0) atomicMax(P.trace + (size_t)k * 8 + 3, global_timer());
  }

  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // the last state slices have been written
  // ---- argmax over the lm_head rows: per CTA, then the CTA that arrives last merges; it also closes the step ----
  __syncwarp();
  Best best = best_s[warp * kGroupMax + (lane & (kGroupMax - 1))];
  for (int off = kGroupMax / 2; off >= 1; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best.v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, best.i, off);
    best_merge(best, ov, oi);
  }
  float* sv = reinterpret_cast<float*>(misc + 8);
  int* si = misc + 8 + kCW;
  if (lane == 0) {
    sv[warp] = best.v;
    si[warp] = best.i;
  }
  consumers_sync();
  if (tid == 0) {
    for (int w = 1; w < kCW; w++) best_merge(best, sv[w], si[w]);
    P.io.part_v[blockIdx.x] = best.v;
    P.io.part_i[blockIdx.x] = best.i;
    __threadfence();
    misc[1] = atomicAdd(P.io.counter, 1u) == gridDim.x - 1;
  }
  consumers_sync();
  if (misc[1] == 0 || warp != 0) return;
  __threadfence();
  best = {-INFINITY, 0x7fffffff};
  for (int c = lane; c < (int)gridDim.x; c += 32) best_merge(best, __ldcg(P.io.part_v + c), __ldcg(P.io.part_i + c));
  for (int off = 16; off >= 1; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best.v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, best.i, off);
    best_merge(best, ov, oi);
  }
  if (lane == 0) {
    const int id = best.v == -INFINITY ? 0 : best.i;   // nothing above it: token 0, as argmax_kernel has it
    P.io.ids_out[0] = id;
    P.io.val_out[0] = best.v;
    if (P.io.host_out) {   // pinned host memory mapped into the device
      P.io.host_out[0] = id;
      P.io.host_out[1] = __float_as_int(best.v);
    }
    *P.io.counter = 0;
    if (P.io.hist && pos < P.io.hist_rows) P.io.hist[(size_t)pos * P.io.hist_ld] = id;
    P.io.pos[0] = pos + 1;
    *P.epoch = ep + 1;
  }
}

struct Plan {
  BkPlanDims dims;
  std::vector<Phase> ph;
  Phase* d_ph = nullptr;
  std::vector<void*> owned;
  uint8_t* tagged = nullptr;         // all tagged buffers, one allocation (cleared by a reset)
  size_t tagged_bytes = 0;
  uint32_t *x = nullptr, *h1 = nullptr, *o = nullptr, *qkv = nullptr, *z = nullptr, *act = nullptr, *qg = nullptr, *kbuf = nullptr, *vbuf = nullptr, *attn_out = nullptr;
  unsigned long long *a = nullptr, *b = nullptr, *sums = nullptr, *po = nullptr, *pml = nullptr;
  unsigned int* words = nullptr;     // epoch, argmax counter
  float* part_v = nullptr;
  int32_t* part_i = nullptr;
  int grid = 0, max_splits = 0, layer = 0;
  uint32_t ring_bytes = 0, scratch_bytes = 0, xs0_bytes = 0, xs_bytes = 0, gdn_bytes = 0;
  int gdn_slots = 0;
  bool maps_ok = true;
  std::vector<CUtensorMap> maps;     // state of the GDN layers, in order
  size_t smem = 0;
  bool finished = false;
};

Plan* as_plan(uint64_t h) { return reinterpret_cast<Plan*>(static_cast<uintptr_t>(h)); }

// rows per warp group: a round of one group per warp takes at most 25/32 of the ring, so that the next one is in flight (as three quarters
// it left hidden 5120 with groups of two rows instead of four when splits of 448 cached rows take 3 KB more scratch: gate and up 29.4 us, not 24.8)
int group_max(const Plan& pl, int K, bool swiglu) {
  const size_t rowb = (size_t)(K / 256) * 144;
  int G = (int)((size_t)pl.ring_bytes * 25 / 32 / kCW / rowb);
  if (G > kGroupMax) G = kGroupMax;
  if (swiglu) G &= ~1;
  if (G < (swiglu ? 2 : 1)) G = swiglu ? 2 : 1;
  return G;
}

Phase& add_gemv(Plan& pl, int in_kind, int K, const void* in, int in_tag, const void* norm_w, int out_tag) {
  Phase ph;
  memset(&ph, 0, sizeof(ph));
  ph.type = PH_GEMV;
  ph.in_kind = in_kind;
  ph.K = K;
  ph.in = in;
  ph.in_tag = in_tag;
  ph.out_tag = out_tag;
  ph.norm_w = norm_w;
  ph.eps = pl.dims.eps;
  pl.ph.push_back(ph);
  return pl.ph.back();
}
void add_seg(const Plan& pl, Phase& ph, uint64_t W, uint64_t W2, void* out, int n_rows, int epi) {
  PSeg& s = ph.g.segs[ph.n_segs++];
  s.W = bk_ptr<uint8_t>(W);
  s.W2 = bk_ptr<uint8_t>(W2);
  s.out = out;
  s.n_rows = n_rows;
  s.epi = epi;
  s.vrow_begin = ph.vrows;
  ph.swiglu = epi == OUT_SWIGLU;
  ph.vrows += ph.swiglu ? 2 * n_rows : n_rows;
  ph.gmax = group_max(pl, ph.K, ph.swiglu);
  const int units = ph.swiglu ? ph.vrows / 2 : ph.vrows, per_round = kCW * (ph.gmax / (ph.swiglu ? 2 : 1));
  ph.ubase = units / pl.grid;
  ph.uextra = units % pl.grid;
  ph.rounds = (ph.ubase + (ph.uextra ? 1 : 0) + per_round - 1) / per_round;
  ph.buffer = ph.in != pl.x && ph.in != pl.h1;
}
void add_out_and_mlp(Plan& pl, const BkPlanLayer& L, Phase& out_proj) {
  const BkPlanDims& D = pl.dims;
  const int t = pl.layer + 1;   // this layer's generation; t - 1 is the residual stream's
  add_seg(pl, out_proj, L.out_proj, 0, pl.h1, D.H, OUT_ADD);
  out_proj.res = pl.x;
  out_proj.res_tag = t - 1;
  Phase& gu = add_gemv(pl, IN_NORM, D.H, pl.h1, t, bk_ptr<void>(L.post_ln), t);
  add_seg(pl, gu, L.gate, L.up, pl.act, D.inter, OUT_SWIGLU);
  Phase& dn = add_gemv(pl, IN_PLAIN, D.inter, pl.act, t, nullptr, t);
  add_seg(pl, dn, L.down, 0, pl.x, D.H, OUT_ADD);
  dn.res = pl.h1;
  dn.res_tag = t;
  dn.plain = bk_ptr<uint16_t>(L.x_out);
  pl.layer++;
}

}  // namespace

int32_t bk_plan_create(uint64_t* out, const BkPlanDims& dims) {
  BkContext& c = bk_ctx();
  *out = 0;
  Plan* pl = new Plan();
  const BkPlanDims& D = pl->dims = dims;
  pl->grid = c.sm_count;
  pl->max_splits = (D.max_len + D.split_len - 1) / D.split_len;
  const int ZD = D.Hv * 128, attn_w = D.Hq * kHD, Cw = (2 * D.Hk + D.Hv) * 128;
  int kmax = D.H;
  for (int K : {ZD, attn_w, D.inter})
    if (K > kmax) kmax = K;
  pl->xs0_bytes = xs_bytes_for(D.H);
  pl->xs_bytes = pl->xs0_bytes + xs_bytes_for(kmax);
  size_t scratch = 2 * sizeof(GdnScratch);
  pl->gdn_slots = (D.Hv * 4 + pl->grid - 1) / pl->grid;
  pl->gdn_bytes = (uint32_t)pl->gdn_slots * kGdnBytes;
  if (attn_item_bytes(D.split_len) > scratch) scratch = attn_item_bytes(D.split_len);
  if ((size_t)D.H * 2 > scratch) scratch = (size_t)D.H * 2;
  if ((size_t)pl->max_splits * 12 > scratch) scratch = (size_t)pl->max_splits * 12;
  pl->scratch_bytes = (uint32_t)((scratch + 127) & ~(size_t)127);
  const size_t fixed = smem_layout(pl->xs_bytes, pl->scratch_bytes, pl->gdn_bytes, 0).total, limit = c.smem_optin;
  // the ring must hold a few groups of the widest row (a gate/up pair is two rows)
  const size_t widest = (size_t)(kmax / 256) * 144;
  const bool fits = D.H % 256 == 0 && D.H <= kMaxNormK && ZD % 256 == 0 && D.inter % 256 == 0 && fixed + 8 * widest + 16384 <= limit &&
                    pl->max_splits <= 1024 && pl->gdn_slots <= 2;
  if (!fits) {
    delete pl;
    return BK_OK;   // the caller keeps one launch per op
  }
  pl->ring_bytes = (uint32_t)((limit - fixed) & ~(size_t)127);
  const SmemLayout lay = smem_layout(pl->xs_bytes, pl->scratch_bytes, pl->gdn_bytes, pl->ring_bytes);
  pl->smem = lay.total;
  if (lay.total - lay.accs < std::max((size_t)pl->ring_bytes * 25 / 32 / kCW, 2 * widest)) {   // a group (group_max) must fit behind the ring
    delete pl;
    return BK_OK;
  }
  // tagged buffers
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t ox = take((size_t)D.H * 4), oh = take((size_t)D.H * 4), oq = take((size_t)Cw * 4), oz = take((size_t)ZD * 4), oa = take((size_t)D.Hv * 8),
               ob = take((size_t)D.Hv * 8), oo = take((size_t)ZD * 4), oact = take((size_t)D.inter * 4), oqg = take((size_t)D.Hq * 2 * kHD * 4),
               ok = take((size_t)D.Hkv * kHD * 4), ov = take((size_t)D.Hkv * kHD * 4), oao = take((size_t)attn_w * 4),
               opo = take((size_t)D.Hq * pl->max_splits * kHD * 8), osum = take((size_t)D.Hv * 32 * 8), oml = take((size_t)D.Hq * pl->max_splits * 16), ow = take(256);
  pl->tagged_bytes = o;
  auto fail = [&](cudaError_t e) {
    bk_plan_destroy((uint64_t)(uintptr_t)pl);
    return bk_fail((int32_t)e, "step plan: %s", cudaGetErrorString(e));
  };
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, o);
  if (e != cudaSuccess) return fail(e);
  pl->owned.push_back(p);
  pl->tagged = static_cast<uint8_t*>(p);
  pl->x = reinterpret_cast<uint32_t*>(pl->tagged + ox);
  pl->h1 = reinterpret_cast<uint32_t*>(pl->tagged + oh);
  pl->qkv = reinterpret_cast<uint32_t*>(pl->tagged + oq);
  pl->z = reinterpret_cast<uint32_t*>(pl->tagged + oz);
  pl->a = reinterpret_cast<unsigned long long*>(pl->tagged + oa);
  pl->b = reinterpret_cast<unsigned long long*>(pl->tagged + ob);
  pl->o = reinterpret_cast<uint32_t*>(pl->tagged + oo);
  pl->sums = reinterpret_cast<unsigned long long*>(pl->tagged + osum);
  pl->act = reinterpret_cast<uint32_t*>(pl->tagged + oact);
  pl->qg = reinterpret_cast<uint32_t*>(pl->tagged + oqg);
  pl->kbuf = reinterpret_cast<uint32_t*>(pl->tagged + ok);
  pl->vbuf = reinterpret_cast<uint32_t*>(pl->tagged + ov);
  pl->attn_out = reinterpret_cast<uint32_t*>(pl->tagged + oao);
  pl->po = reinterpret_cast<unsigned long long*>(pl->tagged + opo);
  pl->pml = reinterpret_cast<unsigned long long*>(pl->tagged + oml);
  pl->words = reinterpret_cast<unsigned int*>(pl->tagged + ow);
  e = cudaMalloc(&p, (size_t)pl->grid * 8);
  if (e != cudaSuccess) return fail(e);
  pl->owned.push_back(p);
  pl->part_v = static_cast<float*>(p);
  pl->part_i = reinterpret_cast<int32_t*>(pl->part_v + pl->grid);
  *out = (uint64_t)(uintptr_t)pl;
  return BK_OK;
}

void bk_plan_add_layer(uint64_t plan, const BkPlanLayer& L) {
  Plan& pl = *as_plan(plan);
  const BkPlanDims& D = pl.dims;
  const int t = pl.layer + 1;
  const int in_kind = pl.layer == 0 ? IN_EMBED : IN_NORM;
  Phase& pr = add_gemv(pl, in_kind, D.H, pl.x, t - 1, bk_ptr<void>(L.in_ln), t);
  if (!L.full) {
    add_seg(pl, pr, L.qkv, 0, pl.qkv, (2 * D.Hk + D.Hv) * 128, OUT_T16);
    add_seg(pl, pr, L.z, 0, pl.z, D.Hv * 128, OUT_T16);
    add_seg(pl, pr, L.a, 0, pl.a, D.Hv, OUT_T32);
    add_seg(pl, pr, L.b, 0, pl.b, D.Hv, OUT_T32);
    Phase g;
    memset(&g, 0, sizeof(g));
    g.type = PH_GDN;
    g.in_tag = g.out_tag = t;
    g.d.qkv = pl.qkv;
    g.d.a = pl.a;
    g.d.b = pl.b;
    g.d.conv_w = bk_ptr<uint16_t>(L.conv_w);
    g.d.cs[0] = bk_ptr<uint16_t>(L.conv_state[0]);
    g.d.cs[1] = bk_ptr<uint16_t>(L.conv_state[1]);
    g.d.A_log = bk_ptr<float>(L.A_log);
    g.d.dt_bias = bk_ptr<uint16_t>(L.dt_bias);
    g.d.S = bk_ptr<float>(L.S);
    g.d.o = pl.o;
    g.d.sums = pl.sums;
    pl.maps.emplace_back();
    pl.maps_ok = pl.maps_ok && bk_encode_map_2d(&pl.maps.back(), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, L.S, 128, (uint64_t)D.Hv * 128, 512, kGdnCols, 128);
    g.d.z = pl.z;
    g.d.norm_w = bk_ptr<float>(L.gnorm);
    pl.ph.push_back(g);
    Phase& po = add_gemv(pl, IN_PLAIN, D.Hv * 128, pl.o, t, nullptr, t);
    add_out_and_mlp(pl, L, po);
  } else {
    add_seg(pl, pr, L.q, 0, pl.qg, D.Hq * 2 * kHD, OUT_T16);
    add_seg(pl, pr, L.k, 0, pl.kbuf, D.Hkv * kHD, OUT_T16);
    add_seg(pl, pr, L.v, 0, pl.vbuf, D.Hkv * kHD, OUT_T16);
    Phase g;
    memset(&g, 0, sizeof(g));
    g.type = PH_ATTN;
    g.in_tag = g.out_tag = t;
    g.a.qg = pl.qg;
    g.a.k = pl.kbuf;
    g.a.v = pl.vbuf;
    g.a.q_norm_w = bk_ptr<uint16_t>(L.q_norm);
    g.a.k_norm_w = bk_ptr<uint16_t>(L.k_norm);
    g.a.kc = bk_ptr<uint16_t>(L.kc);
    g.a.vc = bk_ptr<uint16_t>(L.vc);
    pl.ph.push_back(g);
    g.type = PH_MERGE;
    pl.ph.push_back(g);
    Phase& po = add_gemv(pl, IN_PLAIN, D.Hq * kHD, pl.attn_out, t, nullptr, t);
    add_out_and_mlp(pl, L, po);
  }
}

int32_t bk_plan_finish(uint64_t plan, uint64_t head, uint64_t final_norm, uint64_t logits, int vocab) {
  Plan& pl = *as_plan(plan);
  Phase& lm = add_gemv(pl, pl.layer ? IN_NORM : IN_EMBED, pl.dims.H, pl.x, pl.layer, bk_ptr<void>(final_norm), 0);
  add_seg(pl, lm, head, 0, bk_ptr<void>(logits), vocab, OUT_LOGITS);
  cudaStream_t st = bk_ctx().stream;
  if (!pl.maps_ok) return bk_fail(BK_ERR_UNSUPPORTED, "step plan: the tensor maps of the state could not be encoded");
  void* p = nullptr;
  if (!pl.maps.empty()) {
    BK_CUDA(cudaMalloc(&p, pl.maps.size() * sizeof(CUtensorMap)));
    pl.owned.push_back(p);
    BK_CUDA(cudaMemcpyAsync(p, pl.maps.data(), pl.maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, st));
    const CUtensorMap* m = static_cast<const CUtensorMap*>(p);
    for (Phase& ph : pl.ph)
      if (ph.type == PH_GDN) ph.d.map = m++;
  }
  int entry = 0, n_gdn = 0;
  for (size_t k = 0; k < pl.ph.size(); k++) {
    Phase& ph = pl.ph[k];
    if (ph.type == PH_GEMV) {
      ph.entry = entry;
      entry += ph.rounds * kCW;
      ph.gdn_index = k > 0 && pl.ph[k - 1].type == PH_GDN;
    } else if (ph.type == PH_GDN) {
      ph.gdn_index = n_gdn++;
    }
  }
  const size_t bytes = pl.ph.size() * sizeof(Phase);
  BK_CUDA(cudaMalloc(&p, bytes));
  pl.owned.push_back(p);
  pl.d_ph = static_cast<Phase*>(p);
  BK_CUDA(cudaMemcpyAsync(p, pl.ph.data(), bytes, cudaMemcpyHostToDevice, st));
  BK_CUDA(cudaMemsetAsync(pl.tagged, 0, pl.tagged_bytes, st));
  BK_CUDA(cudaStreamSynchronize(st));
  static size_t configured = 0;
  if (pl.smem > configured) {
    BK_CUDA(cudaFuncSetAttribute(decode_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
    configured = pl.smem;
  }
  int per_sm = 0;
  BK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_step_kernel, kPT, pl.smem));
  if (per_sm < 1) return bk_fail(BK_ERR_UNSUPPORTED, "step plan: the persistent kernel does not fit on an SM");
  pl.finished = true;
  return BK_OK;
}

int32_t bk_plan_launch(uint64_t plan, int parity, const BkStepIO& io) {
  Plan* pl = as_plan(plan);
  BK_ARG(pl && pl->finished, "step plan: not finished");
  BkContext& c = bk_ctx();
  const BkPlanDims& D = pl->dims;
  StepParams P;
  memset(&P, 0, sizeof(P));
  P.phases = pl->d_ph;
  P.n_phases = (int)pl->ph.size();
  P.tags = pl->layer + 2;
  P.epoch = pl->words;
  P.status = c.d_status;
  P.polls = c.spin_limit > 0 ? c.spin_limit : kDefaultPolls;
  P.parity = parity & 1;
  P.trace = (c.step_trace && c.step_trace_phases >= (int)pl->ph.size()) ? c.step_trace : nullptr;
  P.ring_bytes = pl->ring_bytes;
  P.xs0_bytes = pl->xs0_bytes;
  P.xs_bytes = pl->xs_bytes;
  P.scratch_bytes = pl->scratch_bytes;
  P.gdn_bytes = pl->gdn_bytes;
  P.gdn_slots = pl->gdn_slots;
  P.Hk = D.Hk;
  P.Hv = D.Hv;
  P.Hq = D.Hq;
  P.Hkv = D.Hkv;
  P.rot_half = D.rot_half;
  P.max_len = D.max_len;
  P.split_len = D.split_len;
  P.max_splits = pl->max_splits;
  P.scale = D.scale;
  P.cos_t = bk_ptr<float>(D.cos_t);
  P.sin_t = bk_ptr<float>(D.sin_t);
  P.po = pl->po;
  P.pml = pl->pml;
  P.attn_out = pl->attn_out;
  P.io.embed = bk_ptr<uint8_t>(io.embed);
  P.io.ids_in = bk_ptr<int32_t>(io.ids_in);
  P.io.token = io.token;
  P.io.x_tagged = pl->x;
  P.io.x0 = bk_ptr<uint16_t>(io.x0);
  P.io.H = D.H;
  P.io.part_v = pl->part_v;
  P.io.part_i = pl->part_i;
  P.io.counter = pl->words + 1;
  P.io.ids_out = bk_ptr<int32_t>(io.ids_out);
  P.io.val_out = bk_ptr<float>(io.val_out);
  P.io.pos = bk_ptr<int32_t>(io.pos);
  P.io.hist = bk_ptr<int32_t>(io.hist);
  P.io.hist_ld = io.hist_ld;
  P.io.hist_rows = io.hist_rows;
  P.io.host_out = bk_ptr<int32_t>(io.host_out);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl->grid);
  cfg.blockDim = dim3(kPT);
  cfg.dynamicSmemBytes = pl->smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BK_CUDA(cudaLaunchKernelEx(&cfg, decode_step_kernel, P));
  BK_CHECK_LAUNCH();
  return BK_OK;
}

// Tagged words, epoch and argmax counter back to zero (after a launch that gave up they are in an unknown state).  Enqueued on
// the library stream.
int32_t bk_plan_reset(uint64_t plan) {
  Plan* pl = as_plan(plan);
  BK_ARG(pl && pl->finished, "step plan: not finished");
  BK_CUDA(cudaMemsetAsync(pl->tagged, 0, pl->tagged_bytes, bk_ctx().stream));
  return BK_OK;
}

void bk_plan_destroy(uint64_t plan) {
  Plan* pl = as_plan(plan);
  if (!pl) return;
  for (void* p : pl->owned) cudaFree(p);
  delete pl;
}
