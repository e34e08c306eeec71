// bk_gemv_umma.cu -- Q4_K x Q8_1 GEMM for 9 to 64 activation columns on the 5th-generation tensor cores (tcgen05.mma kind::f16,
// operand A and the accumulators in tensor memory).
//
// With so many columns the product is a dense contraction: the weights are streamed ONCE for all columns (the batch 2..8 kernel
// streams them once per group of 8).  The reference's nearest thing is its int8 tensor-core GEMM experiment
// (src/kernel.ts:396-456: 4-bit blocks expanded to int8 tiles, int32 accumulators, scales applied afterwards,
// experiments/q4k_q81_final.ts:217); this is that idea on the 144-byte Q4_K layout.
//
// The integer dots are exact in f16 operands and f32 accumulators: A holds sc*q (a 6-bit scale times a nibble, <= 945, an
// integer below 2^11), B the signed 8-bit quants, and every partial sum of a 32-value sub-block is an integer below 2^22.  So
// an accumulator IS f32(sc*isum), and what is left per (row, column, sub-block) are two fused multiply-adds: d8 * it and
// s8 * m.  (With int8 operands the product sc*isum and its conversion cost an integer multiply, at half rate, and an
// addition per element more, and were what bounded this kernel: 2.2 us per 128 x 256 weights and 32 columns.)
//
// A step is (superblock, sub-block pair p): 128 rows x 64 weights.  A CTA of 640 threads runs as groups of warps that meet only at
// mbarriers:
//   * one PRODUCER warp keeps a ring of stages filled: a stage holds one superblock (or the pairs of it that this CTA handles)
//     of the 128 rows and the activations of that superblock, which are ready-made operand B tiles (see the image below);
//   * eight EXPANDER warps (two per 32 rows, taking turns; thread <-> row) turn a row's 32 bytes into 64 f16 in tensor memory
//     (operand A; the shared-memory bandwidth that it would cost is needed by the scalers) and its header into {d, -dmin, m0, m1};
//   * one MMA warp issues four MMAs (M = 128, N = columns, K = 16) per step into two accumulators of N tensor-memory columns;
//   * eight SCALER warps (two per TMEM lane quarter, half of the columns each) read the accumulators as 16x256b fragments (a thread
//     holds 4 rows x 2 columns of every 8 columns, so that a column's d8 and s8 are loaded once for 4 rows and a row's minima
//     once for all columns) and run the f32 part, two columns per instruction; four such blocks (one step at N = 64, four at
//     N = 16) per wait;
//   * two EPILOGUE warps add up what the scalers hand over and write the outputs while the scalers are at the next tile.
//
// Two orders of the f32 part, both fixed and mirrored by the CPU oracle:
//   LANES (the order of the batch <= 8 kernels, for prompts of many columns and for 9 to 15 sequences): per unit u = (s, p)
//     val = fma(d, fma(d8_1, x1, d8_0*x0), -(dmin * fma(s8_1, m1, s8_0*m0))); class c = s mod 8 of pair p adds its units in
//     ascending s; T_p = ((P0+P4)+(P2+P6)) + ((P1+P5)+(P3+P7)); y = (T0+T2) + (T1+T3).  The classes are walked in the order
//     0,4,2,6,1,5,3,7, so that a stack of three values per (row, column, pair) holds what is still to be added: one in
//     registers, two in shared memory, 64 KB, which is why a CTA takes 2 pairs at N = 32 and one at N = 64.
//   TILE (16 and more sequences): accd = fma(d8, x, accd), accm = fma(s8, m, accm) over the eight sub-blocks; yc += fma(d, accd,
//     -(dmin*accm)); every four superblocks y += yc.
//
// A cluster of CTAs shares a tile: the four pairs (LANES), and where there are few tiles also the classes (LANES) or the
// four-superblock chunks (TILE, by any number of CTAs up to eight).  Every CTA sends each value it ends up with to the CTA of the cluster
// that owns the column (one bulk copy through distributed shared memory per owner; the first 1, 2, 4 or 8 CTAs own columns); the owner adds
// them in the fixed order and runs the epilogue.
//
// Weight feed: one tiled TMA load (cp.async.bulk.tensor.2d) of the tile's 128 rows per stage, two where headers and quants are apart; a SwiGLU
// launch keeps 64 gate rows in tile rows 0..63 and their up rows in 64..127.  A tile with rows of several segments takes boxes of 32,
// 16 or 8 rows, whatever divides the segments' first rows; other shapes (TILE only) copy row by row.  No multicast.  Every wait is
// bounded; TMEM is released on every path out of the kernel.
#include <cuda_fp16.h>

#include <algorithm>

#include "bk_gemv_shared.cuh"

namespace {

constexpr int kTileM = 128;
constexpr int kProducerWarp = 8, kMmaWarp = 9, kEpilogueWarp0 = 10, kScalerWarp0 = 12;
constexpr int kUT = 640;
constexpr int kScalers = 256;
constexpr int kTmemCols = 512;
constexpr int kXPitch = 132;       // floats between columns of the exchange buffers: fragments hit 32 banks
constexpr int kMaxStages = 8;

// per-instance constants: NB = columns / 16
template <int NB, bool LANES>
struct Cfg {
  static constexpr int N = 16 * NB;
  static constexpr int PS = LANES ? 4 / NB : 4;                       // sub-block pairs of a superblock that a CTA handles
  // TMEM: kBatches batches of accumulators (128 columns each) and kA steps of operand A (32 each), handed over kHalf at a time.
  // What a step costs the MMA thread beside its MMAs is mostly waits, so few columns take larger halves and fewer batches -- but in the
  // lane order, whose scalers pause at the end of a class, three batches are better (32 columns, 152k rows, when that took 176 us: with two 199; now 137).
  static constexpr int kBatches = LANES || NB == 4 ? 3 : 2, kA = LANES || NB == 4 ? 4 : 8, kHalf = kA / 2;
  static constexpr int BT = 4 / NB;                                   // steps per batch of the scalers: 128 TMEM columns
  static constexpr int kTabs = kA + kBatches * BT;               // row tables: a step's is read before its successor's is written (see there)
  static constexpr int kWBytes = kTileM * (PS == 4 ? 144 : 16 + 32 * PS);
  static constexpr int kBBytes = N * 128;                             // operand B of a step
  static constexpr int kStage = (kWBytes + PS * kBBytes + 1023) & ~1023;
  // registers of expanders, the single warps, scalers: 640 x 96 at launch = 256 E + 128 M + 256 S at most
  static constexpr int kRegE = 64, kRegM = 64, kRegS = 144;
  static constexpr int kColBytes = PS * N * 16;                       // column factors of a superblock
};

struct UmmaParams {
  GemvParams g;       // K, segments, total_vrows, x = image (see bk_tile_image_bytes), status
  int B;              // activation columns, 1..64
  int groups;         // column groups (N > 32 columns of few rows: two groups of 32, each with its own image and its own tiles)
  int use_maps;       // weights come by tiled TMA loads through maps[] and part[]
  int stages;         // ring stages
  int csplit;         // LANES: CTAs that share the classes of a pair; TILE: CTAs that share the chunks (= cluster size, 1 to 8)
  int levels;         // LANES: stack levels in shared memory
  uint32_t xbuf_bytes, stg_bytes;   // received values; values to send (clusters of more than one)
  CUtensorMap maps[10];   // [2i], [2i+1]: headers and quants of segment i (whole superblocks: only [2i]); i = 4: the up matrix.  Boxes of a tile's rows
  CUtensorMap part[8];    // the same in boxes of part_rows rows, for tiles that more than one segment has rows in
  int part_rows;
};

BK_DEVINL uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  // K-major, no swizzle: 8 rows x 16 bytes contiguous; lbo = bytes between the two 16-byte K chunks of a 32-byte row,
  // sbo = bytes between groups of 8 rows.  Bits [46,48) = 1: the descriptor version of this architecture.
  return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Four registers of a 16x256b fragment (16 lanes x 8 columns): rows lane/4 and lane/4 + 8, columns 2(lane mod 4) and the next;
// complete after tmem_wait.  No memory clobber: they touch tensor memory only and `volatile` keeps their order.
BK_DEVINL void tmem_ld_frag(uint32_t taddr, float (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(taddr));
}
// the registers are operands so that no use of them can be scheduled before the wait
BK_DEVINL void tmem_wait16(float (&a)[4], float (&b)[4], float (&c)[4], float (&d)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(b[0]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3]), "+f"(c[0]), "+f"(c[1]), "+f"(c[2]),
                 "+f"(c[3]), "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]));
}

// Bounded wait whose polls may sleep (a waiting role should not spend issue slots on polling).  The first wait of a CTA that gives
// up sets the status word and a flag in shared memory, after which every other wait of that CTA returns at once -- the kernel
// then runs to its end (results undefined, status BK_ERR_TIMEOUT) instead of timing out step after step.
template <bool CLUSTER = false>
BK_DEVINL bool mbar_poll(uint32_t bar, uint32_t parity, bool may_sleep) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
  else if (may_sleep)
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  else
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
template <bool CLUSTER = false>
BK_DEVINL void mbar_wait_idle(uint32_t bar, uint32_t parity, int* status, volatile int* dead) {
  if (!CLUSTER && mbar_poll(bar, parity, false)) return;
#pragma unroll 1
  for (int it = 0; it < (1 << 22); it++)
    if (mbar_poll<CLUSTER>(bar, parity, true) || *dead) return;
  *dead = 1;
  if (status) atomicExch(status, 10003 /* BK_ERR_TIMEOUT */);
}

BK_DEVINL void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
BK_DEVINL void mbar_arrive_remote(uint32_t bar, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(bar), "r"(rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(r) : "memory");
}
// bytes at src (this CTA) to the same kind of address in another CTA of the cluster, whose barrier counts them
BK_DEVINL void bulk_s2cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar, uint32_t rank) {
  uint32_t d, b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(dst), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(bar), "r"(rank));
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(d), "r"(src), "r"(bytes), "r"(b) : "memory");
}
BK_DEVINL void umma_commit(uint32_t bar) {   // arrives when every MMA issued so far has completed
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool ACC>   // D (+)= A * B, K = 16
BK_DEVINL void umma_f16(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred pz;\n\tsetp.ne.b32 pz, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, pz;\n\t}" ::"r"(d), "r"(a), "l"(bdesc),
               "r"(idesc), "n"(ACC ? 1 : 0)
               : "memory");
}
BK_DEVINL bool elect_one() {
  uint32_t p;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(p));
  return p != 0;
}
// the same wait for a whole warp that stays together, as the roles of one warp do whose instructions take uniform registers
BK_DEVINL void mbar_wait_warp(uint32_t bar, uint32_t parity, int* status, volatile int* dead) {
#pragma unroll 1
  for (int it = 0; it < (1 << 22); it++)
    if (__all_sync(0xffffffffu, mbar_poll(bar, parity, true) || *dead)) return;
  *dead = 1;
  if (status) atomicExch(status, 10003 /* BK_ERR_TIMEOUT */);
}
BK_DEVINL void scalers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kScalers) : "memory"); }
BK_DEVINL void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The superblocks of a tile that a CTA handles, in order.
// LANES: class positions [pos0, pos1) of the order 0,4,2,6,1,5,3,7, within a class ascending.  TILE: [pos0, pos1) themselves.
template <bool LANES>
struct Walk {
  int pos, pos1, s, nsb;
  __host__ __device__ __forceinline__ static int cls(int pos) { return (int)((0x73516240u >> (4 * pos)) & 7u); }
  BK_DEVINL void start(int pos0, int end, int n) {
    nsb = n;
    pos1 = end;
    pos = pos0;
    if (LANES) {
      s = cls(pos);
      settle();
    } else s = pos;
  }
  BK_DEVINL bool done() const { return LANES ? pos >= pos1 : s >= pos1; }
  BK_DEVINL void settle() {   // to the next class that has a superblock
    while (pos < pos1 && s >= nsb) {
      pos++;
      s = cls(pos & 7);
    }
  }
  BK_DEVINL void next() {
    if (LANES) {
      s += 8;
      settle();
    } else s++;
  }
};

BK_DEVINL float2 mul2(float2 a, float2 b) {
  unsigned long long ra, rb, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}
BK_DEVINL float2 dup2(float a) { return make_float2(a, a); }
BK_DEVINL uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
BK_DEVINL uint32_t hbk_add2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
BK_DEVINL uint32_t hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

template <int NB, bool LANES>
__global__ void __launch_bounds__(kUT, 1) gemv_q4k_umma_kernel(const __grid_constant__ UmmaParams P) {
  using C = Cfg<NB, LANES>;
  constexpr int N = C::N, PS = C::PS, BT = C::BT;
  bk_pdl_trigger();
  const GemvParams& p = P.g;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int nst = P.stages;
  uint8_t* raw = smem;                                              // [nst] weights | operand B
  uint8_t* rows = raw + (size_t)nst * C::kStage;                    // [kTabs] float4 {d, -dmin, m0, m1} [128] of a step
  uint8_t* cols = rows + C::kTabs * kTileM * 16;                    // [nst + 3] column factors of a superblock: [pair] float4 {d8, d8', s8, s8'} [2][N/2]
  const int ncols = nst + 3;
  float* xbuf = reinterpret_cast<float*>(cols + ncols * C::kColBytes);   // values received: [value][own column][kXPitch rows]
  uint8_t* stg = reinterpret_cast<uint8_t*>(xbuf) + P.xbuf_bytes;   // values to send: [owner][value][column of the owner][kXPitch rows]
  float2* stack = reinterpret_cast<float2*>(stg + P.stg_bytes);     // [levels][16][256]
  uint64_t* wfull = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(stack) + (size_t)P.levels * 32768);   // [kMaxStages] a stage has landed
  uint64_t* wempty = wfull + kMaxStages;                            // [kMaxStages] its readers are done
  uint64_t* a_full = wempty + kMaxStages;                           // [2] operand A and row tables of half a ring are written
  uint64_t* a_free = a_full + 2;                           // [2] its MMAs have completed
  uint64_t* d_full = a_free + 2;                          // [kBatches] accumulators of a batch complete, tables visible
  uint64_t* d_free = d_full + C::kBatches;                             // [kBatches] the scalers are done with it
  uint64_t* xfull = d_free + C::kBatches;                              // the cluster's values of a tile have arrived
  uint64_t* xempty = xfull + 1;                                     // every owner has read this CTA's values
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xempty + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);   // a bounded wait of this CTA has given up

  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int nsb = p.K / 256;
  constexpr int PSPLIT = 4 / PS;
  const int CS = P.csplit * PSPLIT;
  const int owners = CS >= 8 ? 8 : CS >= 4 ? 4 : CS >= 2 ? 2 : 1;   // CTAs of a cluster that own columns: its size, or the power of two below it
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

  if (t == 0) {
    *dead = 0;
    for (int i = 0; i < nst; i++) {
      mbar_init(smem_u32(wfull + i), 1);
      mbar_init(smem_u32(wempty + i), (PS == 1 ? 4 : 8) + 1);   // expander warps, and the MMAs
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(a_full + i), C::kHalf * kTileM);
      mbar_init(smem_u32(a_free + i), 1);
    }
    for (int i = 0; i < C::kBatches; i++) {
      mbar_init(smem_u32(d_full + i), 2);
      mbar_init(smem_u32(d_free + i), kScalers / 32);
    }
    mbar_init(smem_u32(xfull), 1);
    mbar_init(smem_u32(xempty), owners);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();   // every CTA's barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t tmem_a = tmem + C::kBatches * 128;

  const bool two = NB == 2 && P.groups == 2;   // tile index: row tile * 2 + column group
  const int n_tiles = (p.total_vrows + kTileM - 1) / kTileM * (two ? 2 : 1);
  const int n_chunks = (nsb + 3) / 4;
  const int tile0 = (int)blockIdx.x / CS, tile_step = (int)gridDim.x / CS;   // the cluster's tiles
  const int n_my = (n_tiles - tile0 + tile_step - 1) / tile_step;
  const int p0 = LANES ? ((int)rank % PSPLIT) * PS : 0, part = LANES ? (int)rank / PSPLIT : (int)rank;
  const int pos0 = LANES ? part * 8 / P.csplit : 4 * (part * n_chunks / P.csplit);
  const int pos1 = LANES ? (part + 1) * 8 / P.csplit : min(nsb, 4 * ((part + 1) * n_chunks / P.csplit));
  int n_sb = 0;   // superblocks of a tile that this CTA handles, and of all its tiles
  for (int pos = pos0; pos < pos1; pos++) n_sb += LANES ? max(0, (nsb - Walk<LANES>::cls(pos) + 7) / 8) : 1;
  const int total = n_my * n_sb;
  const int own = N / owners;   // columns of a tile that each of the cluster's first CTAs owns
  const bool swiglu_halves = P.use_maps && p.segs[0].epi == BK_EPI_SWIGLU;   // tile rows 0..63 gate, 64..127 up

  if (warp < kProducerWarp) {
    // ================= expanders: row te of every second step =================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegE));
    const int grp = warp >> 2, te = t & (kTileM - 1);
    int stage = 0, g = grp, tab = grp, sbc = 0;   // g: step
    uint32_t spar = 0;
    const uint32_t ta = tmem_a + ((uint32_t)((warp & 3) * 32) << 16);
    {
      for (; sbc < total; sbc++) {
        if (PS > 1 || (sbc & 1) == grp) {
          mbar_wait_idle(smem_u32(wfull + stage), spar, p.status, dead);
          const uint8_t* base = raw + (size_t)stage * C::kStage;
          uint4 hdr, qv[PS > 1 ? PS : 2];
          if (PS == 4) {
            hdr = *reinterpret_cast<const uint4*>(base + te * 144);
#pragma unroll
            for (int i = 0; i < PS; i++) qv[i] = *reinterpret_cast<const uint4*>(base + te * 144 + 16 + (2 * (i >> 1) + grp) * 32 + (i & 1) * 16);
          } else {
            hdr = *reinterpret_cast<const uint4*>(base + te * 16);
            const uint8_t* qr = base + kTileM * 16 + te * 32 * PS;   // boxes are swizzled: 16-byte chunk c of a row lies at c ^ f(row)
            const int sw = PS == 1 ? (te >> 2) & 1 : (te >> 1) & 3, c0 = PS == 1 ? 0 : 2 * grp;
            qv[0] = *reinterpret_cast<const uint4*>(qr + ((c0 ^ sw) * 16));
            qv[1] = *reinterpret_cast<const uint4*>(qr + (((c0 + 1) ^ sw) * 16));
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(wempty + stage));   // this warp's rows are in registers
          const float d = bk_f16_to_f32((uint16_t)(hdr.x & 0xffffu)), nmin = -bk_f16_to_f32((uint16_t)(hdr.x >> 16));
#pragma unroll
          for (int i = 0; i < (PS > 1 ? PS / 2 : 1); i++) {
            const int pi = PS > 1 ? 2 * i + grp : 0;
            uint32_t sc2, mn2;
            bk_q4k_scale_min_pair(hdr.y, hdr.z, hdr.w, p0 + pi, sc2, mn2);
            // half2 of the scales: (1024 + sc) - 1024; the nibble in the mantissa of 1024: (1024 + q) * sc - 1024 * sc, exact
            const uint32_t s0 = hbk_add2(__byte_perm(sc2, 0x64u, 0x4040), 0xE400E400u), s1 = hbk_add2(__byte_perm(sc2, 0x64u, 0x4141), 0xE400E400u);
            const uint32_t n0 = hmul2(s0, 0xE400E400u), s1s = hmul2(s1, 0x2C002C00u), n1 = hmul2(s1, 0xD400D400u);   // -1024 sc0, sc1 / 16, -64 sc1
            uint32_t a[32];
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const uint4 qq = qv[2 * i + (j >> 2)];
              const uint32_t wv = (j & 3) == 0 ? qq.x : (j & 3) == 1 ? qq.y : (j & 3) == 2 ? qq.z : qq.w, w8 = wv >> 8;
              a[2 * j] = hfma2((wv & 0x000f000fu) | 0x64006400u, s0, n0);            // bytes 0, 2
              a[2 * j + 1] = hfma2((w8 & 0x000f000fu) | 0x64006400u, s0, n0);        // bytes 1, 3
              a[16 + 2 * j] = hfma2((wv & 0x00f000f0u) | 0x64006400u, s1s, n1);
              a[17 + 2 * j] = hfma2((w8 & 0x00f000f0u) | 0x64006400u, s1s, n1);
            }
            if (g >= C::kA) mbar_wait_idle(smem_u32(a_free + ((g / C::kHalf) & 1)), (uint32_t)(g / C::kA - 1) & 1u, p.status, dead);   // step g - kA has been multiplied
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
                "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(ta + (g % C::kA) * 32),
                "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]),
                "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]), "r"(a[19]), "r"(a[20]), "r"(a[21]), "r"(a[22]),
                "r"(a[23]), "r"(a[24]), "r"(a[25]), "r"(a[26]), "r"(a[27]), "r"(a[28]), "r"(a[29]), "r"(a[30]), "r"(a[31])
                : "memory");
            // (step g - kTabs, whose table this was, has been scaled: the MMAs of step g - kA waited for that)
            reinterpret_cast<float4*>(rows + tab * (kTileM * 16))[te] =
                make_float4(d, nmin, __fsub_rn(__uint_as_float(__byte_perm(mn2, 0x4B000000u, 0x7440)), 8388608.0f),
                            __fsub_rn(__uint_as_float(__byte_perm(mn2, 0x4B000000u, 0x7441)), 8388608.0f));
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(smem_u32(a_full + ((g / C::kHalf) & 1)));
            g += 2;
            tab += 2;
            if (tab >= C::kTabs) tab -= C::kTabs;
          }
        }
        if (++stage == nst) {
          stage = 0;
          spar ^= 1u;
        }
      }
    }
    for (const int end = (total * PS + C::kHalf - 1) / C::kHalf * C::kHalf; g < end; g += 2) mbar_arrive(smem_u32(a_full + ((g / C::kHalf) & 1)));   // steps that the last half lacks
  } else if (warp < kScalerWarp0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegM));
    if (warp >= kEpilogueWarp0) {
      // ================= epilogue: the columns this CTA owns, in the fixed order of addition =================
      const int et = t - kEpilogueWarp0 * 32;
      bk_pdl_wait();
      const int vs = own * kXPitch;   // floats between values
      auto value = [&](int c, int r) {
        const float* v = xbuf + c * kXPitch + r;
        if constexpr (!LANES) {
          if (CS == 1) return v[0];
          float y = 0.0f;
          for (int ch = 0; ch < n_chunks; ch++) y = __fadd_rn(y, v[ch * vs]);
          return y;
        } else {
          float T[4];
#pragma unroll
          for (int pp = 0; pp < 4; pp++) {   // value of (part, pair): sent by CTA part * PSPLIT + pair / PS
            const float* vp = v + pp * vs;
            if (P.csplit == 1) T[pp] = vp[0];
            else if (P.csplit == 2) T[pp] = __fadd_rn(vp[0], vp[4 * vs]);
            else if (P.csplit == 4) T[pp] = __fadd_rn(__fadd_rn(vp[0], vp[4 * vs]), __fadd_rn(vp[8 * vs], vp[12 * vs]));
            else
              T[pp] = __fadd_rn(__fadd_rn(__fadd_rn(vp[0], vp[4 * vs]), __fadd_rn(vp[8 * vs], vp[12 * vs])),
                                __fadd_rn(__fadd_rn(vp[16 * vs], vp[20 * vs]), __fadd_rn(vp[24 * vs], vp[28 * vs])));
          }
          return __fadd_rn(__fadd_rn(T[0], T[2]), __fadd_rn(T[1], T[3]));
        }
      };
      const uint32_t xbytes = (uint32_t)((LANES ? 4 * P.csplit : n_chunks) * vs * 4);
      const int b00 = (int)rank * own;
      for (int k = 0; k < ((int)rank < owners ? n_my : 0); k++) {
        const int vt = tile0 + k * tile_step, tile = two ? vt >> 1 : vt, b0 = b00 + (two ? (vt & 1) * N : 0);
        if (CS > 1 && et == 0) mbar_expect_tx(smem_u32(xfull), xbytes);
        mbar_wait_idle(smem_u32(xfull), (uint32_t)k & 1u, p.status, dead);
        for (int h = 0; h < (swiglu_halves ? 1 : 2); h++) {
          const int r = et + 64 * h;
          VRow vr = {nullptr, 0, 0};
          bool have;
          int up = 0;   // distance to the up row of a SwiGLU pair
          if (swiglu_halves) {
            vr.n = tile * 64 + r;
            have = vr.n < p.segs[0].n_rows;
            up = 64;
          } else {
            have = tile * kTileM + r < p.total_vrows;
            if (have) vr = decode_vrow(p, tile * kTileM + r);
            if (p.segs[vr.si].epi == BK_EPI_SWIGLU) {
              up = 1;
              have = have && !(r & 1);
            }
          }
          const SegDev& sg = p.segs[vr.si];
          if (!have) continue;
          const size_t o0 = (size_t)b0 * sg.ld_out + sg.col_off + vr.n, ld = sg.ld_out;
          const int nc = min(own, P.B - b0), epi = sg.epi;
          if (epi == BK_EPI_F32) {
            float* o = static_cast<float*>(sg.out) + o0;
#pragma unroll 4
            for (int c = 0; c < nc; c++) o[c * ld] = value(c, r);
          } else if (epi == BK_EPI_BF16) {
            uint16_t* o = static_cast<uint16_t*>(sg.out) + o0;
#pragma unroll 4
            for (int c = 0; c < nc; c++) o[c * ld] = bk_f32_to_bf16(value(c, r));
          } else if (epi == BK_EPI_SWIGLU) {
            uint16_t* o = static_cast<uint16_t*>(sg.out) + o0;
#pragma unroll 4
            for (int c = 0; c < nc; c++) {
              const float y = value(c, r);
              o[c * ld] = bk_f32_to_bf16(__fmul_rn(__fmul_rn(y, bk_sigmoidf(y)), value(c, r + up)));
            }
          } else {   // BK_EPI_ADD_BF16
            uint16_t* o = static_cast<uint16_t*>(sg.out) + o0;
            const uint16_t* res = sg.res + o0;
#pragma unroll 1
            for (int c0 = 0; c0 < nc; c0 += 8) {   // eight residuals in flight (the outputs may alias them)
              uint16_t rs[8];
#pragma unroll
              for (int j = 0; j < 8; j++) rs[j] = c0 + j < nc ? res[(c0 + j) * ld] : (uint16_t)0;
#pragma unroll
              for (int j = 0; j < 8; j++)
                if (c0 + j < nc) o[(c0 + j) * ld] = bk_f32_to_bf16(__fadd_rn(value(c0 + j, r), bk_bf16_to_f32(rs[j])));
            }
          }
        }
        asm volatile("bar.sync 2, 64;" ::: "memory");
        if (et < CS) mbar_arrive_remote(smem_u32(xempty), et);
      }
    } else if (warp == kMmaWarp) {
      // ================= MMA issue: per step two sub-blocks of K = 32 =================
      // The warp stays together and one elected lane issues, so that addresses and descriptors are uniform values: with one lane that runs
      // alone every MMA first moves its operands there (tile order, 32 columns, 152k rows: 110 us, so 105).
      // f32 accumulators, f16 operands, both K-major
      constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t bd0 = umma_desc(smem_u32(raw) + C::kWBytes, N * 16, 128);
      int stage = 0, batch = 0, g = 0;
      uint32_t spar = 0, bpar = 1;   // a fresh barrier counts as freed
      for (int i = 0; i < total; i++) {
        mbar_wait_warp(smem_u32(wfull + stage), spar, p.status, dead);   // operand B and the column factors
        const uint64_t bs = bd0 + (uint32_t)(stage * (C::kStage >> 4));   // (an address below 256 KB: no carry into the other fields)
#pragma unroll
        for (int pi = 0; pi < PS; pi++, g++) {
          const int bi = pi % BT;
          if (bi == 0) mbar_wait_warp(smem_u32(d_free + batch), bpar, p.status, dead);
          if (g % C::kHalf == 0) mbar_wait_warp(smem_u32(a_full + ((g / C::kHalf) & 1)), (uint32_t)(g / C::kA) & 1u, p.status, dead);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a0 = tm + C::kBatches * 128 + (g % C::kA) * 32, d0 = tm + batch * 128 + bi * 2 * N;
          const uint64_t bd = bs + pi * (N * 8);
          if (elect_one()) {
            umma_f16<false>(d0, a0, bd, idesc);
            umma_f16<true>(d0, a0 + 8, bd + N * 2, idesc);
            umma_f16<false>(d0 + N, a0 + 16, bd + N * 4, idesc);
            umma_f16<true>(d0 + N, a0 + 24, bd + N * 6, idesc);
            if (pi == PS - 1) umma_commit(smem_u32(wempty + stage));   // operand B has been read
            if (bi == BT - 1) {
              umma_commit(smem_u32(d_full + batch));
              mbar_arrive(smem_u32(d_full + batch));   // passes on what the expanders and the copies have written
            }
            if (g % C::kHalf == C::kHalf - 1) umma_commit(smem_u32(a_free + ((g / C::kHalf) & 1)));
          }
          __syncwarp();
          if (bi == BT - 1 && ++batch == C::kBatches) {
            batch = 0;
            bpar ^= 1u;
          }
        }
        if (++stage == nst) {
          stage = 0;
          spar ^= 1u;
        }
      }
      __syncwarp();
    } else {
      // ================= producer: superblock after superblock, tile after tile =================
      // One elected lane issues and few copies make a stage: whatever its size a copy costs the issuing warp about 100 cycles, and with
      // a box per 32 rows, one per lane, the issue bound the whole kernel in the lane order (64 columns: 1,940 of 1,960 cycles a step).
      int cslot = 0;
      Walk<LANES> w, wx;
      const int first = min(total, nst);
      const uint64_t policy = l2_evict_first();
      const uint8_t* img_b = static_cast<const uint8_t*>(p.x) + (size_t)p0 * C::kBBytes;   // image: operand B of all units, then their factors
      const uint8_t* img_c = static_cast<const uint8_t*>(p.x) + (size_t)(p.K / 64) * C::kBBytes + (size_t)p0 * (N * 16);
      const size_t img_bytes = (size_t)(p.K / 64) * (C::kBBytes + N * 16);
      const bool leader = elect_one();
      auto fill_x = [&](int s, int stage, int vt) {
        const size_t go = two ? (size_t)(vt & 1) * img_bytes : 0;
        if (leader) {
          const uint32_t bar = smem_u32(wfull + stage);
          bulk_g2s(smem_u32(raw + (size_t)stage * C::kStage + C::kWBytes), img_b + go + (size_t)s * 4 * C::kBBytes, PS * C::kBBytes, bar);
          bulk_g2s(smem_u32(cols + cslot * C::kColBytes), img_c + go + (size_t)s * (4 * N * 16), C::kColBytes, bar);
        }
        if (++cslot == ncols) cslot = 0;   // (three superblocks more than stages: the scalers are at most that far behind the MMAs)
      };
      constexpr uint32_t kXBytes = PS * C::kBBytes + C::kColBytes;
      constexpr uint32_t kRowW = C::kWBytes / kTileM;   // bytes of a tile row in a stage
      auto load_box = [&](const CUtensorMap* m, uint32_t dst, int x, int row, uint32_t bar) {
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
            "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(row), "r"(bar), "l"(policy)
            : "memory");
      };
      // the segment of the tile's first row, that row in it, and whether the tile has rows of no other segment
      int vt = tile0, tile = 0, mi = 0, row0 = 0;
      bool whole = true;
      auto enter_tile = [&]() {
        tile = two ? vt >> 1 : vt;
        mi = 0;
        int next = p.total_vrows;
#pragma unroll
        for (int si = 3; si >= 1; si--)
          if (si < p.n_segs && mi == 0) {
            if (tile * kTileM >= p.segs[si].vrow_begin) mi = si;
            else next = p.segs[si].vrow_begin;
          }
        row0 = swiglu_halves ? tile * 64 : tile * kTileM - p.segs[mi].vrow_begin;
        whole = next == p.total_vrows || (tile + 1) * kTileM <= next;
      };
      int stage = 0;
      uint32_t spar = 1;   // parity of the readers' arrivals on the previous use
      w.start(pos0, pos1, nsb);
      enter_tile();
      for (int i = 0; i < total; i++) {
        if (i >= nst) mbar_wait_warp(smem_u32(wempty + stage), spar, p.status, dead);
        const uint32_t bar = smem_u32(wfull + stage), dst0 = smem_u32(raw + (size_t)stage * C::kStage);
        const int x = w.s * 144, xq = x + 16 + 32 * p0;
        if (P.use_maps && whole) {   // rows past the last one are filled with zeros
          if (leader) {
            mbar_expect_tx(bar, C::kWBytes + kXBytes);
            const CUtensorMap* m = P.maps + 2 * mi;
            load_box(m, dst0, x, row0, bar);
            if (PS < 4) load_box(m + 1, dst0 + kTileM * 16, xq, row0, bar);
            if (swiglu_halves) {   // the maps' boxes have 64 rows: the gate's, and here the same rows of the up matrix
              load_box(P.maps + 8, dst0 + (PS == 4 ? 64 * 144 : 64 * 16), x, row0, bar);
              if (PS < 4) load_box(P.maps + 9, dst0 + kTileM * 16 + 64 * 32 * PS, xq, row0, bar);
            }
          }
        } else if (P.use_maps) {
          // lanes 0..15: the tile's boxes (whole superblocks, or headers); lanes 16..31: their quants
          const int bx = lane & 15, v0 = tile * kTileM + P.part_rows * bx;
          const bool valid = P.part_rows * bx < kTileM && v0 < p.total_vrows && (PS < 4 || lane < 16);
          int si = 0;
#pragma unroll
          for (int k = 1; k < 4; k++)
            if (k < p.n_segs && v0 >= p.segs[k].vrow_begin) si = k;
          const uint32_t boxes = __popc(__ballot_sync(0xffffffffu, valid && lane < 16));
          if (leader) mbar_expect_tx(bar, boxes * (uint32_t)P.part_rows * kRowW + kXBytes);
          __syncwarp();
          if (valid) {
            const bool quants = lane >= 16;
            const int at = P.part_rows * bx;
            load_box(P.part + 2 * si + (quants ? 1 : 0), dst0 + (PS == 4 ? at * 144 : quants ? kTileM * 16 + at * 32 * PS : at * 16), quants ? xq : x,
                     v0 - p.segs[si].vrow_begin, bar);
          }
        } else {
          const int rows_here = min(kTileM, p.total_vrows - tile * kTileM);
          if (leader) mbar_expect_tx(bar, (uint32_t)rows_here * 144 + kXBytes);
          __syncwarp();
#pragma unroll 1
          for (int r = lane; r < rows_here; r += 32) bulk_g2s(dst0 + r * 144, decode_vrow(p, tile * kTileM + r).row + (size_t)w.s * 144, 144, bar);
        }
        if (i == first - 1) {   // the ring is full of weights, which depend on nothing: now the activations of these stages
          bk_pdl_wait();
          for (int f = 0, vx = tile0; f < first; vx += tile_step)
            for (wx.start(pos0, pos1, nsb); !wx.done() && f < first; wx.next(), f++) fill_x(wx.s, f, vx);
        } else if (i >= first) {
          fill_x(w.s, stage, vt);
        }
        w.next();
        if (w.done()) {
          vt += tile_step;
          w.start(pos0, pos1, nsb);
          enter_tile();
        }
        if (++stage == nst) {
          stage = 0;
          spar ^= 1u;
        }
      }
    }
  } else {
    // ================= scalers: f32 part =================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kRegS));
    const int st = t - kScalerWarp0 * 32, q = warp & 3, half = st >> 7;
    const int row0 = 32 * q + (lane >> 2);              // this thread's rows: row0 + 8i
    const int col0 = half * (N / 2) + 2 * (lane & 3);   // and columns: col0 + 8cb and the next
    const int own_shift = __ffs(own) - 1;
    const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + half * (N / 2);
    int batch = 0, tab = 0, col = 0;
    uint32_t bpar = 0;
    // One batch: BT steps from the current row table and pair pi0 of the current column factors on, as four blocks of 8 columns;
    // f(bi, cb, i, x0, x1, c0, c1, r): step bi, the two columns of block cb, row i, accumulators of both sub-blocks, column factors
    // {d8, d8', s8, s8'} of both, row factors
    auto run_batch = [&](int pi0, auto&& f) {
      mbar_wait_idle(smem_u32(d_full + batch), bpar, p.status, dead);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float4* ct = reinterpret_cast<const float4*>(cols + col * C::kColBytes) + pi0 * N + (col0 >> 1);
      const uint32_t td = ta + batch * 128;
      float x[2][2][2][4];   // [buffer][sub-block][lanes 0..15 / 16..31][fragment]
      auto request = [&](int m) {
#pragma unroll
        for (int j = 0; j < 4; j++)
          tmem_ld_frag(td + (m / NB) * 2 * N + (m % NB) * 8 + (j >> 1) * N + ((uint32_t)(16 * (j & 1)) << 16), x[m & 1][j >> 1][j & 1]);
      };
      request(0);
      float4 r4[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int u = m & 1, cb = m % NB, bi = m / NB;
        if (cb == 0) {
          const float4* rt = reinterpret_cast<const float4*>(rows + tab * (kTileM * 16)) + row0;
#pragma unroll
          for (int i = 0; i < 4; i++) r4[i] = rt[8 * i];
          if (++tab == C::kTabs) tab = 0;
        }
        tmem_wait16(x[u][0][0], x[u][0][1], x[u][1][0], x[u][1][1]);
        if (m < 3) request(m + 1);   // in flight during this block's arithmetic
        const float4 c0 = ct[bi * N + cb * 4], c1 = ct[bi * N + N / 2 + cb * 4];
#pragma unroll
        for (int i = 0; i < 4; i++)
          f(bi, cb, i, make_float2(x[u][0][i >> 1][2 * (i & 1)], x[u][0][i >> 1][2 * (i & 1) + 1]),
            make_float2(x[u][1][i >> 1][2 * (i & 1)], x[u][1][i >> 1][2 * (i & 1) + 1]), c0, c1, r4[i]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(d_free + batch));
      if (++batch == C::kBatches) {
        batch = 0;
        bpar ^= 1u;
      }
    };
    auto next_superblock = [&]() {
      if (++col == ncols) col = 0;
    };
    // value v (of nv that this CTA sends) of column block cb and row i into the buffer the owners read or are sent
    float* const out = CS > 1 ? reinterpret_cast<float*>(stg) : xbuf;
    auto place = [&](int v, int nv, int cb, int i) {
      const int c = col0 + 8 * cb;
      return out + ((((c >> own_shift) * nv + v) << own_shift) + (c & (own - 1))) * kXPitch + row0 + 8 * i;
    };
    auto send = [&](int first, int nv) {   // nv values, the owner's buffer index of the first
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      scalers_sync();
      if (CS == 1) {
        if (st == 0) mbar_arrive(smem_u32(xfull));
      } else if (st < owners && nv > 0) {
        const uint32_t bytes = (uint32_t)(nv * own * kXPitch * 4), dst = (uint32_t)(first * own * kXPitch * 4);
        bulk_s2cluster(smem_u32(xbuf) + dst, smem_u32(stg) + st * bytes, bytes, smem_u32(xfull), st);
      }
    };

    for (int k = 0; k < n_my; k++) {
      if constexpr (LANES) {
        float2 S[16], L0[16];   // [step of the batch = pair][column block][row]
        int sp = 0;
        auto unit = [&](float2 x0, float2 x1, const float4& c0, const float4& c1, const float4& r) {
          float2 a = mul2(make_float2(c0.x, c0.y), x0);
          a = bk_fma2(make_float2(c1.x, c1.y), x1, a);
          float2 mm = mul2(make_float2(c0.z, c0.w), dup2(r.z));
          mm = bk_fma2(make_float2(c1.z, c1.w), dup2(r.w), mm);
          return bk_fma2(dup2(r.x), a, mul2(dup2(r.y), mm));
        };
        auto run_class = [&](int pos, float2 (&T)[16]) {
          int s = Walk<LANES>::cls(pos);
          if (s < nsb) {   // the first superblock of the class, onto zero
            run_batch(0, [&](int bi, int cb, int i, float2 x0, float2 x1, const float4& c0, const float4& c1, const float4& r) {
              T[(bi * NB + cb) * 4 + i] = bk_add2(make_float2(0.0f, 0.0f), unit(x0, x1, c0, c1, r));
            });
            next_superblock();
          } else {
#pragma unroll
            for (int e = 0; e < 16; e++) T[e] = make_float2(0.0f, 0.0f);
          }
          for (s += 8; s < nsb; s += 8) {
            run_batch(0, [&](int bi, int cb, int i, float2 x0, float2 x1, const float4& c0, const float4& c1, const float4& r) {
              const int e = (bi * NB + cb) * 4 + i;
              T[e] = bk_add2(T[e], unit(x0, x1, c0, c1, r));
            });
            next_superblock();
          }
        };
        for (int lp = 0; lp < pos1 - pos0; lp += 2) {   // (classes are shared by powers of two: one, or a whole number of pairs)
          run_class(pos0 + lp, L0);
          if (lp + 1 < pos1 - pos0) {
            run_class(pos0 + lp + 1, S);
#pragma unroll
            for (int e = 0; e < 16; e++) S[e] = bk_add2(L0[e], S[e]);
            for (int m = lp >> 1; m & 1; m >>= 1) {
              sp--;
#pragma unroll
              for (int e = 0; e < 16; e++) S[e] = bk_add2(stack[(sp * 16 + e) * kScalers + st], S[e]);
            }
            if (lp + 2 < pos1 - pos0) {
#pragma unroll
              for (int e = 0; e < 16; e++) stack[(sp * 16 + e) * kScalers + st] = S[e];
              sp++;
            }
          }
        }
        if (k > 0) mbar_wait_idle<true>(smem_u32(xempty), (uint32_t)(k - 1) & 1u, p.status, dead);   // what was sent before has been read
#pragma unroll
        for (int e = 0; e < 16; e++) {
          float* o = place(e / (4 * NB), PS, e / 4 % NB, e & 3);
          o[0] = pos1 - pos0 == 1 ? L0[e].x : S[e].x;
          o[kXPitch] = pos1 - pos0 == 1 ? L0[e].y : S[e].y;
        }
        send((int)rank * PS, PS);
      } else {
        constexpr int E = 4 * NB;
        float2 yc[E];
        const int ch0 = pos0 >> 2, nv = CS > 1 ? (pos1 + 3) / 4 - ch0 : 1;
        if (k > 0 && pos0 >= pos1) mbar_wait_idle<true>(smem_u32(xempty), (uint32_t)(k - 1) & 1u, p.status, dead);
        for (int s = pos0; s < pos1; s++) {
          float2 A[E], M[E];
#pragma unroll
          for (int e = 0; e < E; e++) A[e] = M[e] = make_float2(0.0f, 0.0f);
          float rd[4], rm[4];
#pragma unroll 1
          for (int pi = 0; pi < 4; pi += BT)
            run_batch(pi, [&](int bi, int cb, int i, float2 x0, float2 x1, const float4& c0, const float4& c1, const float4& r) {
              const int e = cb * 4 + i;
              A[e] = bk_fma2(make_float2(c0.x, c0.y), x0, A[e]);
              M[e] = bk_fma2(make_float2(c0.z, c0.w), dup2(r.z), M[e]);
              A[e] = bk_fma2(make_float2(c1.x, c1.y), x1, A[e]);
              M[e] = bk_fma2(make_float2(c1.z, c1.w), dup2(r.w), M[e]);
              rd[i] = r.x;
              rm[i] = r.y;
            });
          next_superblock();
#pragma unroll
          for (int e = 0; e < E; e++)
            yc[e] = bk_add2((s & 3) == 0 ? make_float2(0.0f, 0.0f) : yc[e], bk_fma2(dup2(rd[e & 3]), A[e], mul2(dup2(rm[e & 3]), M[e])));
          if ((s & 3) == 3 || s == nsb - 1) {   // a chunk ends: its own value, or y += yc in place
            if (k > 0 && s - pos0 < 4) mbar_wait_idle<true>(smem_u32(xempty), (uint32_t)(k - 1) & 1u, p.status, dead);
            const bool first = CS > 1 || s < 4;
#pragma unroll
            for (int e = 0; e < E; e++) {
              float* o = place(CS > 1 ? (s >> 2) - ch0 : 0, nv, e / 4, e & 3);
              o[0] = __fadd_rn(first ? 0.0f : o[0], yc[e].x);
              o[kXPitch] = __fadd_rn(first ? 0.0f : o[kXPitch], yc[e].y);
            }
          }
        }
        send(ch0, nv);
      }
    }
  }

  // ---- release tensor memory (every thread gets here, whatever happened above) ----
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
  cluster_sync();   // nobody leaves while another CTA may still reach its shared memory
}

// Q8_1 blocks [B][K/32][36] -> image
__global__ void __launch_bounds__(256) tile_image_kernel(const uint32_t* x, int nblk, const int B_all, uint8_t* img, const bool split) {
  bk_pdl_trigger();
  bk_pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x, blk = i / B_all;
  int b = i % B_all, B = B_all;
  if (blk >= nblk) return;
  const uint32_t* src = x + ((size_t)b * nblk + blk) * 9;
  uint32_t w[9];
#pragma unroll
  for (int k = 0; k < 9; k++) w[k] = __ldg(src + k);
  int qsum = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) qsum = bk_dp4a_ss(w[k], 0x01010101u, qsum);
  if (split) {   // an image per 32 columns
    img += (size_t)(b >> 5) * bk_tile_image_bytes(nblk * 32, 32);
    b &= 31;
    B = 32;
  }
#pragma unroll
  for (int c = 0; c < 4; c++) bk_tile_store_quants(img, B, b, blk, c, w[2 * c], w[2 * c + 1]);
  const float d8 = bk_q8half_to_f32((uint16_t)(w[8] & 0xffffu));
  bk_tile_store_factors(img, nblk * 32, B, b, blk, d8, __fmul_rn(d8, (float)qsum));
}

// Matrix of Q4_K rows; header < 0: whole superblock columns (box rows x 144 bytes), 1: their headers (x 16 bytes), 0: the quants
// of `pairs` sub-block pairs (x 32 * pairs bytes, swizzled so that the expanders' 16-byte reads hit all banks).
bool encode_weight_map(CUtensorMap* m, const uint8_t* W, int n_rows, size_t row_bytes, int box_rows, int header, int pairs) {
  const uint32_t box = header < 0 ? 144 : header ? 16 : 32 * pairs;
  const CUtensorMapSwizzle sw = header == 0 ? (pairs == 1 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B) : CU_TENSOR_MAP_SWIZZLE_NONE;
  return bk_encode_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, (uint64_t)(uintptr_t)W, row_bytes, (uint64_t)n_rows, row_bytes, box, box_rows, sw);
}

// How a launch of `tiles` tiles is cut: CTAs of a cluster that share the classes (or chunks) of a tile.
struct TilePlan {
  int csplit, clusters, rounds, len;   // len: superblocks of the longest CTA
  float cost;                          // superblocks, see plan_tiles
  uint32_t xbuf_bytes, stg_bytes;
  int levels, stages;
  size_t smem;
};
constexpr int kMaxCluster = 8;
int owners_of(int cs) { return cs >= 8 ? 8 : cs >= 4 ? 4 : cs >= 2 ? 2 : 1; }

// clusters of each size that are resident at once (0: that size does not fit)
template <int NB, bool LANES>
int32_t resident_clusters(const int** out) {
  static int clusters[kMaxCluster + 1] = {};
  BkContext& c = bk_ctx();
  if (!clusters[1]) {
    auto kernel = gemv_q4k_umma_kernel<NB, LANES>;
    const size_t limit = c.smem_optin - 1024;
    BK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kUT);
    cfg.dynamicSmemBytes = limit;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    for (int cs = kMaxCluster; cs >= 1; cs--) {
      attr[0].val.clusterDim.x = cs;
      cfg.gridDim = dim3(c.sm_count / cs * cs);
      if (cudaOccupancyMaxActiveClusters(&clusters[cs], kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        clusters[cs] = 0;
      }
    }
    if (clusters[1] < 1) return bk_fail(BK_ERR_UNSUPPORTED, "tile GEMV: the kernel does not fit the device");
  }
  *out = clusters;
  return BK_OK;
}

template <int NB, bool LANES>
int32_t plan_tiles(int tiles, int K, TilePlan* best) {
  // LANES: the cheapest of 1, 2, 4 and 8 parts.  A tile costs the superblocks of its longest CTA, 0.1 for each of that CTA's classes and kEnd for the
  // exchange; its end runs beside the next tile's superblocks, but however few those are no tile after the first takes less than kTile.  Fitted to
  // 1,071 launches of 16, 32 and 64 columns: 14 are 4 to 9 % slower than with the best number of parts.  With eight classes of ceil(K / 2048)
  // superblocks and one for a tile's end 85 were, by up to 62 % (64 columns, 9,472 rows, K 256 29.4 us, so 21.2, K 2048 34.3, so 29.6; 32 columns, 20,480
  // rows, K 256 28.5, so 21.2; 16 columns, 24,576 rows, K 256 19.5, so 14.9).
  // TILE: the same with the steps of the longest CTA and one superblock for a tile; with two stages only, superblocks of one tile after another come
  // half as fast (17 chunks, 48 tiles of 32 columns: 1.8 times, rounds of one tile hardly at all).  The lane order shares its classes by powers of
  // two; other numbers of parts are taken in the tile order where they save 30 % (K 5120, 2,048 rows, 32 columns: five parts of one chunk 15.4 us,
  // four of one or two 20.2): by less they are slower, since fewer CTAs own columns.
  using C = Cfg<NB, LANES>;
  constexpr int PSPLIT = 4 / C::PS;
  constexpr size_t per_stage = C::kStage + C::kColBytes;
  const size_t limit = bk_ctx().smem_optin - 1024;
  const int* clusters = nullptr;
  const int32_t rc = resident_clusters<NB, LANES>(&clusters);
  if (rc != BK_OK) return rc;
  const int nsb = K / 256, n_chunks = (nsb + 3) / 4;
  constexpr float kEnd = NB == 1 ? 0.5f : NB == 2 ? 1.5f : 3.5f, kTile = NB == 1 ? 6.0f : NB == 2 ? 7.0f : 9.0f;
  auto candidate = [&](int s, TilePlan& p) {
    const int cs = s * PSPLIT, n = clusters[cs], own = C::N / owners_of(cs);
    p.csplit = s;
    p.clusters = n;
    p.levels = LANES && s <= 2 ? 2 - __builtin_ctz(s) : 0;
    p.xbuf_bytes = (uint32_t)((LANES ? 64 : cs > 1 ? n_chunks * own : C::N) * kXPitch * 4);
    p.stg_bytes = cs == 1 ? 0 : (uint32_t)((LANES ? 64 : (n_chunks + s - 1) / s * C::N) * kXPitch * 4);
    const size_t fixed = (size_t)C::kTabs * kTileM * 16 + 3 * C::kColBytes + p.xbuf_bytes + p.stg_bytes + (size_t)p.levels * 32768 + 512;
    if (n < 1 || fixed + 2 * per_stage > limit) return false;   // (one CTA a tile always fits)
    p.stages = std::min(kMaxStages, (int)((limit - fixed) / per_stage));
    p.smem = fixed + (size_t)p.stages * per_stage;
    p.rounds = (tiles + n - 1) / n;
    if (LANES) {
      p.len = 0;
      for (int part = 0; part < s; part++) {
        int n_sb = 0;
        for (int pos = part * 8 / s; pos < (part + 1) * 8 / s; pos++) n_sb += std::max(0, (nsb - Walk<true>::cls(pos) + 7) / 8);
        p.len = std::max(p.len, n_sb);
      }
      const float tile = p.len + 0.1f * (8 / s) + kEnd;
      p.cost = tile + (p.rounds - 1) * std::max(tile, kTile);
    } else {
      p.len = 4 * ((n_chunks + s - 1) / s);
      p.cost = p.rounds * (p.len * (p.stages == 2 && p.rounds > 1 ? 1.6f : 1.0f) + 1.0f);
    }
    return true;
  };
  TilePlan p;
  best->cost = 1e30f;
  for (int s = 1; s * PSPLIT <= kMaxCluster; s *= 2)
    if (candidate(s, p) && p.cost < best->cost) *best = p;
  if (!LANES) {
    const float pow2 = best->cost;
    for (int s : {3, 5, 6, 7})
      if (candidate(s, p) && p.cost < 0.7f * pow2 && p.cost < best->cost) *best = p;
  }
  return best->cost < 1e30f ? BK_OK : bk_fail(BK_ERR_UNSUPPORTED, "tile GEMV: K=%d does not fit in shared memory", K);
}

template <int NB, bool LANES>
int32_t launch_tile(UmmaParams& P) {
  using C = Cfg<NB, LANES>;
  BkContext& c = bk_ctx();
  GemvParams& g = P.g;
  // tensor-map feed: boxes that never straddle two segments
  P.part_rows = 32;
  bool ok = true, mixed = false;
  for (int i = 1; i < g.n_segs; i++) {
    while (P.part_rows > 8 && g.segs[i].vrow_begin % P.part_rows != 0) P.part_rows /= 2;
    ok = ok && g.segs[i].vrow_begin % P.part_rows == 0;
    mixed = mixed || g.segs[i].vrow_begin % kTileM != 0;
  }
  const size_t row_bytes = (size_t)(g.K / 256) * 144;
  auto encode = [&](CUtensorMap* m, const uint8_t* W, int n_rows, int box_rows) {
    return C::PS == 4 ? encode_weight_map(m, W, n_rows, row_bytes, box_rows, -1, 4)
                      : encode_weight_map(m, W, n_rows, row_bytes, box_rows, 1, 0) && encode_weight_map(m + 1, W, n_rows, row_bytes, box_rows, 0, C::PS);
  };
  for (int i = 0; ok && i < g.n_segs; i++) {
    const bool swiglu = g.segs[i].epi == BK_EPI_SWIGLU;   // (alone in its launch)
    ok = encode(P.maps + 2 * i, g.segs[i].W, g.segs[i].n_rows, swiglu ? 64 : kTileM);
    if (ok && swiglu) ok = encode(P.maps + 8, g.segs[i].W2, g.segs[i].n_rows, 64);
    if (ok && mixed) ok = encode(P.part + 2 * i, g.segs[i].W, g.segs[i].n_rows, P.part_rows);
  }
  BK_ARG(ok || !LANES, "tile GEMV: the lane order needs segments that begin at multiples of 8 rows");
  P.use_maps = ok ? 1 : 0;

  const int tiles = (g.total_vrows + kTileM - 1) / kTileM * P.groups;
  TilePlan t;
  const int32_t rc = plan_tiles<NB, LANES>(tiles, g.K, &t);
  if (rc != BK_OK) return rc;
  const int cs = t.csplit * (4 / C::PS);
  P.csplit = t.csplit;
  P.levels = t.levels;
  P.xbuf_bytes = t.xbuf_bytes;
  P.stg_bytes = t.stg_bytes;
  P.stages = t.stages;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kUT);
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((tiles < t.clusters ? tiles : t.clusters) * cs);
  cfg.dynamicSmemBytes = t.smem;
  BK_CUDA(cudaLaunchKernelEx(&cfg, gemv_q4k_umma_kernel<NB, LANES>, P));
  BK_CHECK_LAUNCH();
  return BK_OK;
}

}  // namespace

// 16 to 64 columns (9 to 64 in the lane order); p: a filled GemvParams whose x is an image, or Q8_1 blocks (prologue BK_PRO_Q8).
int32_t bk_gemv_umma_launch(void* params, int B, bool lanes) {
  BkContext& c = bk_ctx();
  UmmaParams P;
  P.g = *static_cast<GemvParams*>(params);
  P.B = B;
  const bool split = bk_tile_split(P.g.total_vrows, P.g.K, B, lanes);
  P.groups = split ? 2 : 1;
  if (P.g.prologue == BK_PRO_Q8) {
    const size_t need = bk_tile_image_bytes(P.g.K, B);
    if (c.tile_image_bytes < need) {
      if (c.capturing) return bk_fail(BK_ERR_STATE, "bkGemvQ4K: the tile path's image buffer must be sized by an eager launch before a capture");
      BK_CUDA(cudaStreamSynchronize(c.stream));
      cudaFree(c.tile_image);
      c.tile_image = nullptr;
      c.tile_image_bytes = 0;
      void* q = nullptr;
      BK_CUDA(cudaMalloc(&q, need));
      c.tile_image = static_cast<uint8_t*>(q);
      c.tile_image_bytes = need;
    }
    const int nblk = P.g.K / 32;
    BK_CUDA(bk_launch_pdl(tile_image_kernel, dim3((nblk * B + 255) / 256), dim3(256), 0, static_cast<const uint32_t*>(P.g.x), nblk, B, c.tile_image, split));
    BK_CHECK_LAUNCH();
    P.g.x = c.tile_image;
  }
  if (lanes) return B <= 16 ? launch_tile<1, true>(P) : B <= 32 || split ? launch_tile<2, true>(P) : launch_tile<4, true>(P);   // (nine columns and more)
  return B <= 16 ? launch_tile<1, false>(P) : B <= 32 || split ? launch_tile<2, false>(P) : launch_tile<4, false>(P);
}

// Two groups of 32 columns instead of one of 64, each with its own image and tiles.
// LANES: at 64 columns a tile takes a cluster of four CTAs, so up to 18 tiles leave half of the SMs idle (clusters of eight, which would
// share the classes too, do not fit sixteen times).  As two groups they take twice as many clusters.
// TILE: the values that a cluster exchanges grow with columns and K; at 64 columns and K 17,408 no cluster has room for them, and one CTA walks
// all of K (1,024 rows: 161 us).  A superblock of 64 columns takes 1.7 times one of 32 (K 17,408, 12,352 rows, one CTA a tile: 164 and 96 us).
bool bk_tile_split(int rows, int K, int B, bool lanes) {
  if (B <= 32) return false;
  const int tiles = (rows + kTileM - 1) / kTileM;
  if (lanes) return tiles * 8 <= bk_ctx().sm_count;
  TilePlan one, two;
  if (plan_tiles<4, false>(tiles, K, &one) != BK_OK || plan_tiles<2, false>(2 * tiles, K, &two) != BK_OK) return false;
  // (where two groups need every SM for a few superblocks they are slower all the same: K 1024, 9,472 rows 17 us, as two groups 18 to 22)
  return two.cost < 1.65f * one.cost && (2 * tiles * 4 <= 3 * bk_ctx().sm_count || two.len >= 16);
}
