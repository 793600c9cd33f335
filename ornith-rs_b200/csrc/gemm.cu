// Wide mat-mul on the 5th-generation tensor cores: y[rows, O] = x[rows, K] W^T for rows >= 16,
// with W in any of the library's weight formats.
//
// Replaces kquant::qmm_t / gather_qmm_t (src/ops/kquant.rs:783-812,905-972, kernels/kquant_mm.h:
// 88-360: a tile of weights is dequantised into threadgroup memory and multiplied by simdgroup
// matrices) and the prompt-width side of quantized_matmul / matmul (src/ops/quantized.rs:249-333,
// src/ops/matmul.rs:486-526).  The reference exempts this path from row invariance
// (src/generate.rs:99): a prompt row computed here does not carry the bits of the one-row
// mat-vec, it agrees with it to rounding (weights are rounded to bfloat16 once, products are
// accumulated in float32 by the tensor core).
//
// Shape of the kernel.  The contraction runs with the WEIGHTS as the A operand and the TOKENS as
// the B operand, D[feature, token] = sum_k W[feature, k] x[token, k]: the tensor core's M is always
// a full 128 features, its N is the token-tile width BN (16..128), so a launch with few tokens per
// expert (a routed prompt chunk, a batched decode step) wastes no tensor-core work on padding.
// One persistent CTA per SM walks work items (feature tile of 128, up to BN tokens, a range of K);
// its warps have fixed roles and meet only at mbarriers:
//   warp 0        TMA of the raw weight bytes, one super-block (256 weights along K) of the 128 rows
//                 per slot: the scales of a super-block are fetched once, rows arrive as 128-byte
//                 swizzled boxes that the dequantising threads read without bank conflicts
//   warp 2        TMA of the token tiles [BN, 64] (and of bf16 weights)
//   warps 8..     dequantise: two or three groups of four warps, a group owns every second (third) unit of two K
//                 blocks (128 weights a thread: one feature row), stores them with tcgen05.st into TENSOR MEMORY,
//                 where the MMA takes its A operand from, and hands the unit over with one arrival per
//                 warp.  Fewer, longer steps won over sixteen warps of one K block each (with the
//                 rest of this layout 146 -> 137 us for 1024 routed Q4_K rows): a hand-over costs a warp several hundred cycles of waiting
//                 whatever it carries, and with 128 registers the conversions of a step interleave
//   warp 1        issues 4 tcgen05.mma (128 x BN x 16, bf16 in, f32 accumulate) per K block and one
//                 commit per unit: a commit occupies the issuing thread for about 160 cycles, twice
//                 what the four MMAs of a block take
//   warps 4..7    epilogue: accumulators (two buffers where they fit) to registers, round, store
// bf16 weights need no dequantisation: their box lands swizzled in shared memory and the MMA reads it
// there (8 warps).  Every wait is bounded and reports through the context's device error flag, and
// the CTA frees its tensor memory on every path.
//
// The grouped form serves rows sorted by expert (counting_sort + switch_glu_rows,
// src/ops/moe.rs:283-314,463-508): every CTA derives the work items (expert, rows, feature tile) from
// the experts' row ranges at its start.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <set>
#include <string>
#include <utility>

#include "fused.h"
#include "orn_internal.h"
#include "orn_quant.cuh"

namespace {

constexpr int BM = 128;            // features per tile: the tensor core's M
constexpr int BK = 64;             // weights per K block: one 128-byte swizzle row of bf16
constexpr int kDqWarps = 4;     // dequantising warps of a group: one per quadrant of the 128 features
constexpr int kSB = 4;          // K blocks of a super-block (256 weights), the step of the raw ring
constexpr int U = 2;            // K blocks of a unit, the step of the ring the MMA reads
constexpr int gemm_threads(int groups) { return 256 + 32 * kDqWarps * groups; }
constexpr uint32_t kWCols = BK / 2;     // tensor-memory columns of one dequantised 128 x 64 tile (two bf16 per column)
constexpr int kSplitMaxRows = 512;      // dense products up to this many rows may split K
constexpr int kMaxSplit = 8;            // = the portable cluster size: the splits of a tile are one cluster
constexpr uint32_t kWTileBytes = BM * BK * 2;
constexpr int kMaxRaw = 8;  // raw ring slots (super-blocks)
constexpr int kMaxUnits = 8; // units of the ring the MMA reads (token tiles + dequantised weight tiles)
constexpr int kMaxE = 1024;     // experts of the grouped form
constexpr int kItemCache = 256; // work items a CTA lays out at its start (later ones are derived one by one)
constexpr int kStageLd = BM + 8;  // elements between the rows of the epilogue's staging tile
constexpr uint32_t kGemmSmem = 209 * 1024;     // dynamic shared memory a CTA may take
constexpr uint32_t kGemmWaitLimit = 1u << 16;  // try_wait rounds (each may sleep kGemmHintNs)
constexpr uint32_t kGemmHintNs = 20000;

constexpr int kMaxJobs = 4;  // matrices of one launch (projections that share their input rows)
struct GemmJob {
  int O, tile0;        // output features; first feature tile of this matrix in the launch's tile space
  int ldy;             // elements between output rows
  bf16_t* y;
  float* y_f32;        // non-null: float32 output instead of bfloat16
  int vec8;            // y may be stored eight bfloat16 at a time
  const uint32_t* row_map;  // nullable: output row of (sorted) row p
};
struct GemmParams {
  int njobs;
  GemmJob job[kMaxJobs];
  const int* seg;      // grouped: expert e owns sorted rows seg[e] .. seg[e+1]-1; null = dense
  int E;
  int dense_tiles;     // dense: feature tiles x token groups
  int rows;            // rows of x (dense) / of the sorted row space (grouped)
  int K;
  int BN, f_tiles;
  int raw_slots, units;      // slots of the raw ring, units of the MMA's ring
  uint32_t raw_bytes;        // bytes of one raw slot
  int nacc;                  // sets of accumulators (2 where they fit beside the weight ring)
  uint32_t acc_cols;         // columns of one accumulator
  uint32_t tmem_cols;        // power of two: what the CTA takes of tensor memory
  // dense products over few rows sum their K blocks in `splits` ranges of `per` blocks, each range in an
  // accumulator of its own, the ranges then in order: `seq` of them one after the other in a CTA, the
  // CTAs of a cluster of splits / seq side by side
  int splits, seq, per;
  int* err;
};

ORN_D uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
ORN_D void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
ORN_D void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
ORN_D void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
ORN_D bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kGemmHintNs)
      : "memory");
  return ok != 0;
}
ORN_D bool mbar_test(uint32_t bar, uint32_t parity) {  // does not suspend
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false (and the error flag set) when the phase never completes
ORN_D bool mbar_wait(uint32_t bar, uint32_t parity, int* err) {
  for (uint32_t it = 0; it < kGemmWaitLimit; ++it)
    if (mbar_try(bar, parity)) return true;
  atomicExch(err, 1);
  return false;
}
// Each thread's wait runs out by its own clock, so threads that go on to something they execute together
// (tcgen05.ld and .st by whole warps, a named barrier) agree on the outcome first: they all go on or all leave.
// The vote stands inside the loop, whose branch is then uniform: free, where one vote behind a loop per lane cost
// 1.8 % (97-token prompt 1.74 -> 1.77 ms, 64 sequences 18.17 -> 18.47 ms).
ORN_D bool mbar_wait_warp(uint32_t bar, uint32_t parity, int* err) {
  for (uint32_t it = 0; it < kGemmWaitLimit; ++it)
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  atomicExch(err, 1);
  return false;
}
ORN_D bool mbar_wait_epilogue(uint32_t bar, uint32_t parity, int* err) {  // the four epilogue warps
  uint32_t all;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 q, %1, 0;\n"
      "barrier.red.and.pred p, 1, 128, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(all)
      : "r"(mbar_wait_warp(bar, parity, err) ? 1u : 0u)
      : "memory");
  return all != 0;
}
ORN_D void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
ORN_D void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
ORN_D void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
ORN_D void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// The MMA warp runs its loop with all 32 lanes and one elected lane issues: operands stay in uniform
// registers (a lane-0 branch costs about 100 cycles per instruction in register moves).
ORN_D void tc_commit(uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(bar)
      : "memory");
}
// one K block: D[tmem] (+)= A[smem] * B[smem]^T, four times 128 x N x 16, bf16 in, f32 out; `add` = 0
// starts a new sum
ORN_D void tc_mma_block(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n"
      ".reg .pred e, p;\n"
      ".reg .b64 a1, a2, a3, b1, b2, b3;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "add.u64 a1, %1, 2;\nadd.u64 a2, %1, 4;\nadd.u64 a3, %1, 6;\n"
      "add.u64 b1, %2, 2;\nadd.u64 b2, %2, 4;\nadd.u64 b3, %2, 6;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, 1;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, 1;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, 1;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(add)
      : "memory");
}
// the same with A in tensor memory: 128 lanes x 8 columns (16 bf16 of K per row) per step
ORN_D void tc_mma_block_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n"
      ".reg .pred e, p;\n"
      ".reg .b32 a1, a2, a3;\n"
      ".reg .b64 b1, b2, b3;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "add.u32 a1, %1, 8;\nadd.u32 a2, %1, 16;\nadd.u32 a3, %1, 24;\n"
      "add.u64 b1, %2, 2;\nadd.u64 b2, %2, 4;\nadd.u64 b3, %2, 6;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, 1;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, 1;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(add)
      : "memory");
}
// shared-memory operand descriptor: K-major, 128-byte swizzle, rows of 128 bytes, groups of 8 rows
// 1024 bytes apart (start >> 4 | LBO 1 | SBO 64 | version 1 | layout SWIZZLE_128B)
ORN_D uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
ORN_D void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
ORN_D void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 registers of every lane to 16 columns of the warp's 32 tensor-memory lanes (lane i of the warp = row i)
ORN_D void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
ORN_D void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
ORN_D uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
ORN_D uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
ORN_D uint32_t lds16(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// Codes to floats.  The integer (ALU) pipe is what bounds the dequantising warps: it takes a warp
// instruction every two cycles, the FMA pipe one per cycle.  So a code is never widened on the ALU:
// one logic op (or byte permute) drops TWO codes into the mantissas of a pair of halves, and the mixed
// add f32 = f16 + f32 (one FMA-pipe instruction) turns each into the exact float the product wants.
//   0x6400 | q           is the half 1024 + q   (q in bits 0..3 or a whole byte)
//   0x5400 | (q << 4)    is the half   64 + q   (q in bits 4..7)
// The scale then needs one packed fma per two weights and one conversion packs the bfloat16 pair: 1.1
// ALU instructions per 4-bit weight instead of 2, 1.0 instead of 1.5 per 8-bit weight (with the rest
// of this layout the grouped Q6_K product of 1024 routed rows: 110 -> 74 us).
ORN_D float add_lo(uint32_t h2, float c) {  // low half of h2 + c
  float d;
  asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %1;\nadd.rn.f32.f16 %0, l, %2;\n}\n" : "=f"(d) : "r"(h2), "f"(c));
  return d;
}
ORN_D float add_hi(uint32_t h2, float c) {
  float d;
  asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %1;\nadd.rn.f32.f16 %0, h, %2;\n}\n" : "=f"(d) : "r"(h2), "f"(c));
  return d;
}
ORN_D uint32_t bf2_of(uint64_t p) {  // packed pair of floats -> two bfloat16, the first in the low half
  uint32_t r;
  asm("{\n"
      ".reg .f32 x, y;\n"
      "mov.b64 {x, y}, %1;\n"
      "cvt.rn.bf16x2.f32 %0, y, x;\n"
      "}\n"
      : "=r"(r)
      : "l"(p));
  return r;
}
ORN_D uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
ORN_D uint32_t mask_or(uint32_t w, uint32_t mask, uint32_t magic) { return (w & mask) | magic; }  // one LOP3
// The constants of the conversions, read from shared memory.  As literals they were moved into a register again in
// front of nearly every use (a mixed add takes no immediate, a LOP3 one): 87.5 -> 70.5 million warp instructions for
// 1024 routed Q4_K rows, 137 -> 126 us; the 8-bit and 6-bit formats have fewer of them (no change).
struct Magic {
  uint32_t lo, hi;  // halves that hold a code from bit 0 / bit 4 on (a byte each of a format's 8-bit codes)
  float c0, c4;     // what takes the rest of them away
};
__host__ __device__ constexpr Magic magic_of(int kind) {
  return kind == ORN_A8 ? Magic{0x64646464u, 0u, 31744.0f, 0.0f}
       : kind == ORN_Q6K ? Magic{0x64646464u, 0u, -1056.0f, 0.0f}
                         : Magic{0x64006400u, 0x54005400u, -1008.0f, -48.0f};
}

// The raw bytes of a super-block (4 K blocks, 256 weights along K) of 128 rows arrive by TMA as boxes
// cut out of the row records.  Code boxes are 128 (or 64) bytes wide and swizzled, so that the 8 rows
// that a quarter of a warp reads with one 16-byte load each lie in different banks; scale boxes of 16
// bytes per row need no swizzle.  Bytes past the end of a record (the last, partial super-block) hold
// the next field or the fill value and are never converted.
//
// Slot layout per format and the record offsets (x coordinates, multiples of 16) the boxes are cut at,
// for super-block sb:
//   Q4_K  [0, 16384)      codes, box 128 swizzled:   x = sb*128
//         [16384, 18432)  header, box 16:            x = b0 + sb*16
//   Q6_K  [0, 16384)      ql, box 128 swizzled:      x = sb*192
//         [16384, 24576)  qh, box 64 swizzled:       x = sb*192 + 128
//         [24576, 26624)  scales, box 16:            x = b0 + sb*16
//         [26624, 28672)  d, box 16:                 x = b0 + b1 + ((2 sb) & ~15)
//   A8    [0, 32768)      codes, 2 boxes 128 sw.:    x = sb*256, sb*256 + 128
//         [32768, 34816)  {scale,bias}, box 16:      x = b0 + sb*16
//   A4    [0, 16384)      codes, box 128 swizzled:   x = sb*128
//         [16384, 20480)  {scale,bias}, box 32:      x = b0 + sb*32
//   BF16  none: the [128 x 64] bf16 box lands in the MMA tile itself (128-byte swizzle)
//
// A thread holds the raw bytes of one row and of a pair of K blocks (g = 0: the super-block's first two,
// 1: its last two) in registers: load() reads them, convert() turns them into 64 words of two bfloat16
// each, in K order, 16 words (= 16 tensor-memory columns of the row's lane) at a time through st(h, words).
struct WeightMaps {
  CUtensorMap wide;   // row records as bytes [E*O, rec], box [128 rows, 128 bytes], 128-byte swizzle (bf16: [E*O, K] bf16, box [128, 64])
  CUtensorMap mid;    // Q6_K: box [128, 64], 64-byte swizzle
  CUtensorMap scale;  // box [128, 16] (A4: 32)
};
ORN_D uint4 lds_sw128(uint32_t base, int r, int c) { return lds128(base + r * 128 + (((uint32_t)c ^ ((uint32_t)r & 7u)) << 4)); }
ORN_D uint4 lds_sw64(uint32_t base, int r, int c) { return lds128(base + r * 64 + (((uint32_t)c ^ (((uint32_t)r >> 1) & 3u)) << 4)); }

template <int KIND> struct Fmt;

template <> struct Fmt<ORN_BF16> {
  static constexpr uint32_t kRawBytes = kWTileBytes;
  struct Raw {};
  ORN_D static void issue(const WeightMaps& m, const RecGeom&, int kb, int row, uint32_t raw, uint32_t bar) {
    tma_load_2d(raw, &m.wide, kb * BK, row, bar);
  }
  ORN_D static void load(Raw&, uint32_t, int, int, int) {}
  template <class St> ORN_D static void convert(const Raw&, int, const Magic&, St) {}
};

// affine 8-bit, group 64: w = scale * q + bias (one fma, as the embedding lookup computes it)
template <> struct Fmt<ORN_A8> {
  static constexpr uint32_t kRawBytes = 32768 + 2048;
  struct Raw { uint4 c[8]; uint2 sb; };
  ORN_D static void issue(const WeightMaps& m, const RecGeom& g, int sb, int row, uint32_t raw, uint32_t bar) {
    tma_load_2d(raw, &m.wide, sb * 256, row, bar);
    tma_load_2d(raw + 16384, &m.wide, sb * 256 + 128, row, bar);
    tma_load_2d(raw + 32768, &m.scale, (int)g.b0 + sb * 16, row, bar);
  }
  ORN_D static void load(Raw& R, uint32_t raw, int r, int g, int) {
    R.sb = lds64(raw + 32768 + r * 16 + 8 * g);
#pragma unroll
    for (int i = 0; i < 8; ++i) R.c[i] = lds_sw128(raw + 16384 * g, r, i);
  }
  template <class St> ORN_D static void convert(const Raw& R, int, const Magic& M, St st) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      // w = sc * (32768 + q) + (bias - 32768 sc)
      const uint32_t sb = h < 2 ? R.sb.x : R.sb.y;
      const float sc = bf_lo(sb), bi = fmaf(-32768.0f, sc, bf_hi(sb));
      const uint64_t a2 = pk2(sc, sc), b2 = pk2(bi, bi);
      const uint4 q0 = R.c[2 * h], q1 = R.c[2 * h + 1];
      const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      uint32_t out[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t h01 = __byte_perm(w[i], M.lo, 0x4140), h23 = __byte_perm(w[i], M.lo, 0x4342);
        out[2 * i] = bf2_of(ffma2(a2, pk2(add_lo(h01, M.c0), add_hi(h01, M.c0)), b2));
        out[2 * i + 1] = bf2_of(ffma2(a2, pk2(add_lo(h23, M.c0), add_hi(h23, M.c0)), b2));
      }
      st(h, out);
    }
  }
};

// affine 4-bit, group 32: half a K block is one group; byte b holds weights 2b (low nibble), 2b+1 (high)
template <> struct Fmt<ORN_A4> {
  static constexpr uint32_t kRawBytes = 16384 + 4096;
  struct Raw { uint4 c[4], sb; };
  ORN_D static void issue(const WeightMaps& m, const RecGeom& g, int sb, int row, uint32_t raw, uint32_t bar) {
    tma_load_2d(raw, &m.wide, sb * 128, row, bar);
    tma_load_2d(raw + 16384, &m.scale, (int)g.b0 + sb * 32, row, bar);
  }
  ORN_D static void load(Raw& R, uint32_t raw, int r, int g, int) {
    R.sb = lds128(raw + 16384 + r * 32 + 16 * g);
#pragma unroll
    for (int i = 0; i < 4; ++i) R.c[i] = lds_sw128(raw, r, 4 * g + i);
  }
  template <class St> ORN_D static void convert(const Raw& R, int, const Magic& M, St st) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      // w = sc * (16 + q) + (bias - 16 sc)
      const uint32_t sb = h == 0 ? R.sb.x : h == 1 ? R.sb.y : h == 2 ? R.sb.z : R.sb.w;
      const float sc = bf_lo(sb), bi = fmaf(-16.0f, sc, bf_hi(sb));
      const uint64_t a2 = pk2(sc, sc), b2 = pk2(bi, bi);
      const uint4 q = R.c[h];
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      uint32_t out[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {  // one word = 8 weights = 4 words of bfloat16 pairs (low nibble first)
        const uint32_t w8 = w[c] >> 8;
        const uint32_t l02 = mask_or(w[c], 0x000F000Fu, M.lo), h02 = mask_or(w[c], 0x00F000F0u, M.hi);
        const uint32_t l13 = mask_or(w8, 0x000F000Fu, M.lo), h13 = mask_or(w8, 0x00F000F0u, M.hi);
        out[4 * c] = bf2_of(ffma2(a2, pk2(add_lo(l02, M.c0), add_lo(h02, M.c4)), b2));
        out[4 * c + 1] = bf2_of(ffma2(a2, pk2(add_lo(l13, M.c0), add_lo(h13, M.c4)), b2));
        out[4 * c + 2] = bf2_of(ffma2(a2, pk2(add_hi(l02, M.c0), add_hi(h02, M.c4)), b2));
        out[4 * c + 3] = bf2_of(ffma2(a2, pk2(add_hi(l13, M.c0), add_hi(h13, M.c4)), b2));
      }
      st(h, out);
    }
  }
};

// Q4_K (kernels/q4k.metal:43-96): a K block is 32 code bytes; low nibbles are sub-block 2i (the first
// half of the K block), high nibbles sub-block 2i+1 (the second half); w = (d * sc) * q - dmin * m,
// evaluated as one fma per weight (this path agrees with the mat-vec to rounding, not bit for bit)
template <> struct Fmt<ORN_Q4K> {
  static constexpr uint32_t kRawBytes = 16384 + 2048;
  struct Raw { uint4 c[4], hdr; };
  ORN_D static void issue(const WeightMaps& m, const RecGeom& g, int sb, int row, uint32_t raw, uint32_t bar) {
    tma_load_2d(raw, &m.wide, sb * 128, row, bar);
    tma_load_2d(raw + 16384, &m.scale, (int)g.b0 + sb * 16, row, bar);
  }
  ORN_D static void load(Raw& R, uint32_t raw, int r, int g, int) {
    R.hdr = lds128(raw + 16384 + r * 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) R.c[i] = lds_sw128(raw, r, 4 * g + i);
  }
  template <class St> ORN_D static void convert(const Raw& R, int g, const Magic& M, St st) {
    const float d = h2f((uint16_t)(R.hdr.x & 0xffff)), dmin = h2f((uint16_t)(R.hdr.x >> 16));
    // 6-bit scales and minima of sub-blocks 4 g .. 4 g + 3, a byte each (g is the same for the whole warp)
    uint32_t sc4, mn4;
    if (g == 0) { sc4 = R.hdr.y & 0x3F3F3F3Fu; mn4 = R.hdr.z & 0x3F3F3F3Fu; }
    else {
      sc4 = (R.hdr.w & 0x0F0F0F0Fu) | ((R.hdr.y >> 2) & 0x30303030u);
      mn4 = ((R.hdr.w >> 4) & 0x0F0F0F0Fu) | ((R.hdr.z >> 2) & 0x30303030u);
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      // w = (d sc) * (16 + q) + (-16 d sc - dmin m)
      const float a = d * (float)((sc4 >> (8 * h)) & 0xffu), nb = fmaf(-16.0f, a, -(dmin * (float)((mn4 >> (8 * h)) & 0xffu)));
      const uint64_t a2 = pk2(a, a), b2 = pk2(nb, nb);
      const uint32_t mask = h & 1 ? 0x00F000F0u : 0x000F000Fu, magic = h & 1 ? M.hi : M.lo;
      const float c = h & 1 ? M.c4 : M.c0;
      const uint4 q0 = R.c[h & 2], q1 = R.c[(h & 2) + 1];
      const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      uint32_t out[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t h02 = mask_or(w[i], mask, magic), h13 = mask_or(w[i] >> 8, mask, magic);
        out[2 * i] = bf2_of(ffma2(a2, pk2(add_lo(h02, c), add_lo(h13, c)), b2));
        out[2 * i + 1] = bf2_of(ffma2(a2, pk2(add_hi(h02, c), add_hi(h13, c)), b2));
      }
      st(h, out);
    }
  }
};

// Q6_K (kernels/q6k.metal:47-77): per 128 weights, byte l of ql / qh gives q1 (weight l), q2 (l + 32),
// q3 (l + 64), q4 (l + 96); the pair of K blocks is one such half-block: the first takes the low nibbles
// of ql (q1, q2), the second the high ones (q3, q4); w = (d * sc) * (q - 32)
template <> struct Fmt<ORN_Q6K> {
  static constexpr uint32_t kRawBytes = 16384 + 8192 + 2048 + 2048;
  struct Raw { uint4 l[4], h[2]; uint2 sc; uint32_t d; };
  ORN_D static void issue(const WeightMaps& m, const RecGeom& g, int sb, int row, uint32_t raw, uint32_t bar) {
    tma_load_2d(raw, &m.wide, sb * 192, row, bar);
    tma_load_2d(raw + 16384, &m.mid, sb * 192 + 128, row, bar);
    tma_load_2d(raw + 24576, &m.scale, (int)g.b0 + sb * 16, row, bar);
    tma_load_2d(raw + 26624, &m.scale, (int)(g.b0 + g.b1) + ((2 * sb) & ~15), row, bar);
  }
  ORN_D static void load(Raw& R, uint32_t raw, int r, int g, int sb) {
    R.d = lds16(raw + 26624 + r * 16 + ((2 * sb) & 15));
    R.sc = lds64(raw + 24576 + r * 16 + 8 * g);   // the half-block's eight sub-block scales
#pragma unroll
    for (int i = 0; i < 4; ++i) R.l[i] = lds_sw128(raw, r, 4 * g + i);
#pragma unroll
    for (int i = 0; i < 2; ++i) R.h[i] = lds_sw64(raw + 16384, r, 2 * g + i);
  }
  template <class St> ORN_D static void convert(const Raw& R, int, const Magic& M, St st) {
    const float d = h2f((uint16_t)R.d);
    const uint32_t hw[8] = {R.h[0].x, R.h[0].y, R.h[0].z, R.h[0].w, R.h[1].x, R.h[1].y, R.h[1].z, R.h[1].w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {  // code set h: nibble h >> 1 of ql bytes 32 (h & 1) .., bits 2 h of qh
      const uint32_t s2 = (h < 2 ? R.sc.x : R.sc.y) >> (16 * (h & 1));
      const float s0 = d * (float)(int8_t)(s2 & 0xff), s1 = d * (float)(int8_t)((s2 >> 8) & 0xff);
      // w = s * (q - 32), exact in float32 (18 + 6 bits)
      const uint64_t a20 = pk2(s0, s0), a21 = pk2(s1, s1);
      const uint4 l0 = R.l[2 * (h & 1)], l1 = R.l[2 * (h & 1) + 1];
      const uint32_t lw[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
      uint32_t out[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t hb = h == 0 ? hw[i] << 4 : h == 1 ? hw[i] << 2 : h == 2 ? hw[i] : hw[i] >> 2;
        const uint32_t q = ((h >= 2 ? lw[i] >> 4 : lw[i]) & 0x0F0F0F0Fu) | (hb & 0x30303030u);
        const uint32_t h01 = __byte_perm(q, M.lo, 0x4140), h23 = __byte_perm(q, M.lo, 0x4342);
        const uint64_t a2 = i < 4 ? a20 : a21;
        out[2 * i] = bf2_of(fmul2(a2, pk2(add_lo(h01, M.c0), add_hi(h01, M.c0))));
        out[2 * i + 1] = bf2_of(fmul2(a2, pk2(add_lo(h23, M.c0), add_hi(h23, M.c0))));
      }
      st(h, out);
    }
  }
};

// One work item: 128 feature rows starting at weight row `wrow`, ntok tokens from tok0, K blocks kb0..kb1-1
struct Item {
  int wrow, tok0, ntok, job, ft, kb0, kb1;
};
ORN_D int4 pack_item(const Item& it) {
  return make_int4(it.wrow, it.tok0, it.ntok | (it.job << 12) | (it.ft << 16), it.kb0 | (it.kb1 << 16));
}
ORN_D Item unpack_item(const int4& v) {
  return Item{v.x, v.y, v.z & 0xfff, (v.z >> 12) & 3, (int)((uint32_t)v.z >> 16), v.w & 0xffff, (int)((uint32_t)v.w >> 16)};
}
// item w of the launch (off: the experts' first items, grouped form only)
ORN_D Item derive_item(const GemmParams& P, int w, int split /*rank in the cluster*/, const int* off) {
  Item it;
  int e = 0, ft;
  const int KB = P.K / BK;
  if (off != nullptr) {
    int lo = 0, hi = P.E;  // off[lo] <= w < off[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (off[mid] <= w) lo = mid; else hi = mid;
    }
    e = lo;
    const int in = w - off[e], g = in / P.f_tiles;
    ft = in - g * P.f_tiles;
    it.tok0 = P.seg[e] + g * P.BN;
    it.ntok = min(P.BN, P.seg[e + 1] - it.tok0);
    it.kb0 = 0; it.kb1 = KB;
  } else {
    const int g = w / P.f_tiles;
    ft = w - g * P.f_tiles;
    it.tok0 = g * P.BN;
    it.ntok = min(P.BN, P.rows - it.tok0);
    it.kb0 = split * P.seq * P.per; it.kb1 = min(KB, it.kb0 + P.seq * P.per);
  }
  it.job = 0;
  while (it.job + 1 < P.njobs && ft >= P.job[it.job + 1].tile0) ++it.job;
  it.ft = ft - P.job[it.job].tile0;
  it.wrow = e * P.job[it.job].O + it.ft * BM;
  return it;
}

ORN_D uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
ORN_D void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
ORN_D void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
ORN_D uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes into another CTA's shared memory; its barrier counts them as they land
ORN_D void push_f4(uint32_t dst, const uint32_t* v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(bar)
               : "memory");
}

struct GemmMaps {
  CUtensorMap x;    // tokens [rows, K] bf16, box [BN, 64], 128-byte swizzle
  WeightMaps w[kMaxJobs];
};

// Barriers (every ring position is counted from the CTA's first K block on):
//   raw_full[i]  the boxes of raw slot i arrived            (producer's expect_tx)
//   raw_free[i]  every dequantising warp has read slot i    (one arrival per warp)
//   full[u]      the unit's token tiles landed and its weight tiles are in tensor memory (expect_tx + one arrival per
//                warp of the group that owns the unit)
//   free[u]      the MMAs that read unit slot u are done (tcgen05.commit)
//   acc_full[b]  accumulator b is complete (commit);  acc_free[b]  the epilogue has read it
//   part_full    split-K: the partial sums of this CTA's share of the tokens have arrived from the whole cluster
//   mma_done     used by leave_late only

// What the CTA's last barrier hands to leave_late
struct Leave {
  uint32_t quit;          // the epilogue gave up: it does whenever any role did, since an item then stays undone
  uint32_t raw, x;        // where the producers stopped: ring position | phase << 8
  uint32_t met;           // split-K: the epilogue has been through the cluster's first barrier
};
// A wait has run out.  Before the CTA lets go of its memory everything in flight ends, each wait
// with the same limit again: the boxes requested last, the MMAs, and what the cluster's other CTAs push here: they
// have pushed, given up or left once they reach the second barrier of the cluster or are gone (it counts the
// threads that have not exited), and what was pushed has landed once part_full completes (share: the bytes it
// expects).  The barriers themselves are not bounded, all that stands in front of them is.  Behind the CTA's
// last barrier and fed through shared memory: the same waits at the end of each role, or behind a call, moved the
// registers of the dequantising loop (97-token prompt +2.5 % and +0.8 %; here 1726 -> 1722 us, 64 sequences at
// 4096 +0.4 %).
__device__ __forceinline__ void leave_late(uint32_t b0, int raw_slots, int units, const Leave* L, bool cluster, uint32_t share, int* err) {
  const uint32_t raw_full = b0, full = b0 + 16 * kMaxRaw, part_full = full + 16 * kMaxUnits + 32, mma_done = part_full + 8;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(mma_done, 1);
    fence_async_smem();
  }
  __syncthreads();
  auto landed = [&](uint32_t bars, int n, uint32_t pos) {
    const int at = (int)(pos & 0xffu);
    const uint32_t ph = pos >> 8;
    for (int i = 0; i < n && mbar_wait(bars + 8 * i, i < at ? ph : ph ^ 1u, err); ++i) {}
  };
  if (threadIdx.x == 0) landed(raw_full, raw_slots, L->raw);
  if (threadIdx.x == 64) landed(full, units, L->x);
  __syncwarp();
  if (warp == 1) {
    tc_commit(mma_done);
    mbar_wait_warp(mma_done, 0, err);
  }
  if (cluster) {
    const bool epilogue = warp >= 4 && warp < 8;
    if (threadIdx.x == 128 && !L->met) mbar_expect_tx(part_full, share);
    __syncwarp();
    if (!epilogue || !L->met) cluster_wait();
    cluster_arrive();
    cluster_wait();
    if (threadIdx.x == 128) mbar_wait(part_full, 0, err);
  }
  __syncthreads();
}

template <int KIND, int G /*groups of dequantising warps*/>
__global__ void __launch_bounds__(gemm_threads(G), 1) k_qgemm(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams P) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[2 * kMaxRaw + 2 * kMaxUnits + 6];
  __shared__ int4 s_items[kItemCache];
  __shared__ int s_off[kMaxE + 1];
  __shared__ __align__(16) bf16_t s_stage[2][16][kStageLd];
  __shared__ uint32_t s_tmem;
  __shared__ Leave s_leave;
  __shared__ __align__(16) Magic s_magic;
  using F = Fmt<KIND>;
  constexpr bool kDirect = KIND == ORN_BF16;  // the MMA reads the weight box where TMA put it
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_addr(smem_raw) + 1023u) & ~1023u;  // swizzled tiles want 1024-byte alignment
  const int RS = P.raw_slots;
  const int NU = P.units;
  const uint32_t x_bytes = (uint32_t)P.BN * 128u;
  const uint32_t raw0 = smem0, x0 = raw0 + (uint32_t)RS * P.raw_bytes;
  const uint32_t part0 = x0 + (uint32_t)(U * NU) * x_bytes;  // split-K: where the cluster's partial sums arrive
  const uint32_t b0 = smem_addr(s_bar);
  const uint32_t raw_full = b0, raw_free = b0 + 8 * kMaxRaw, full = b0 + 16 * kMaxRaw, free_ = full + 8 * kMaxUnits;
  const uint32_t acc_full = free_ + 8 * kMaxUnits, acc_free = acc_full + 16, part_full = acc_free + 16;
  const bool grouped = P.seg != nullptr;
  if (threadIdx.x == 0) {
    for (int i = 0; i < (kDirect ? 0 : RS); ++i) {
      mbar_init(raw_full + 8 * i, 1);
      mbar_init(raw_free + 8 * i, G * kDqWarps);
    }
    for (int i = 0; i < NU; ++i) {
      mbar_init(full + 8 * i, kDirect ? 1 : 1 + kDqWarps);
      mbar_init(free_ + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_free + 8 * i, 4);
    }
    mbar_init(part_full, 1);
    s_leave.quit = s_leave.met = 0;
    s_magic = magic_of(KIND);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  __syncwarp();
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(P.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // ---- the CTA's work items
  int n_items;
  if (grouped) {
    // items before expert e: its predecessors' started groups of BN rows times the feature tiles
    for (int e = threadIdx.x; e < P.E; e += blockDim.x) s_off[e + 1] = (P.seg[e + 1] - P.seg[e] + P.BN - 1) / P.BN * P.f_tiles;
    __syncthreads();
    if (warp == 0) {
      int carry = 0;
      for (int e0 = 0; e0 < P.E; e0 += 32) {
        int v = e0 + lane < P.E ? s_off[e0 + lane + 1] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        if (e0 + lane < P.E) s_off[e0 + lane + 1] = carry + v;
        carry += __shfl_sync(0xffffffffu, v, 31);
      }
      if (lane == 0) s_off[0] = 0;
    }
    __syncthreads();
    n_items = s_off[P.E];
  } else {
    n_items = P.dense_tiles;
  }
  const int C = P.splits / P.seq;  // CTAs of a cluster
  const int split = C > 1 ? (int)cluster_rank() : 0;
  const int first = C > 1 ? (int)blockIdx.x / C : (int)blockIdx.x;
  const int stride = C > 1 ? (int)gridDim.x / C : (int)gridDim.x;
  const int* off = grouped ? s_off : nullptr;
  const int mine = n_items > first ? (n_items - first + stride - 1) / stride : 0;
  // (the items of a grouped launch are searched once, here; those of a dense one are derived where they are needed)
  for (int i = threadIdx.x; grouped && i < min(mine, kItemCache); i += blockDim.x) s_items[i] = pack_item(derive_item(P, first + i * stride, split, off));
  auto item = [&](int i) { return grouped && i < kItemCache ? unpack_item(s_items[i]) : derive_item(P, first + i * stride, split, off); };
  tc_fence_before();
  __syncthreads();
  if (C > 1) cluster_arrive();  // this CTA's barriers exist
  tc_fence_after();
  const uint32_t tmem = s_tmem, tmem_w = tmem + P.acc_cols * P.nacc * P.seq;
  const RecGeom geo = rec_geom(KIND, P.K);

  if (warp == 0 && !kDirect) {
    // ---- raw weight boxes, a super-block at a time
    if (lane == 0) {
      int rs = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 0; ok && i < mine; ++i) {
        const Item w = item(i);
        const WeightMaps& wm = maps.w[w.job];
        for (int sb = w.kb0 / kSB; sb <= (w.kb1 - 1) / kSB; ++sb) {
          ok = mbar_wait(raw_free + 8 * rs, ph ^ 1u, P.err);
          if (!ok) break;
          mbar_expect_tx(raw_full + 8 * rs, F::kRawBytes);
          F::issue(wm, geo, sb, w.wrow, raw0 + (uint32_t)rs * P.raw_bytes, raw_full + 8 * rs);
          if (++rs == RS) { rs = 0; ph ^= 1u; }
        }
      }
      s_leave.raw = (uint32_t)rs | ph << 8;
    }
  } else if (warp == 2) {
    // ---- token tiles, a unit at a time (and the weight boxes of a bf16 matrix)
    if (lane == 0) {
      int us = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 0; ok && i < mine; ++i) {
        const Item w = item(i);
        const int k1 = ((w.kb1 - 1) / kSB + 1) * kSB;
        for (int k0 = w.kb0 / kSB * kSB; k0 < k1; k0 += U) {  // every unit of the super-blocks the item touches
          ok = mbar_wait(free_ + 8 * us, ph ^ 1u, P.err);
          if (!ok) break;
          const int lo = max(w.kb0, k0), hi = min(w.kb1, k0 + U);
          mbar_expect_tx(full + 8 * us, (uint32_t)max(0, hi - lo) * (x_bytes + (kDirect ? kWTileBytes : 0u)));
          for (int kb = lo; kb < hi; ++kb) {
            const uint32_t slot = (uint32_t)(us * U + kb % U);
            if (kDirect) F::issue(maps.w[w.job], geo, kb, w.wrow, raw0 + slot * kWTileBytes, full + 8 * us);
            tma_load_2d(x0 + slot * x_bytes, &maps.x, kb * BK, w.tok0, full + 8 * us);
          }
          if (++us == NU) { us = 0; ph ^= 1u; }
        }
      }
      s_leave.x = (uint32_t)us | ph << 8;
    }
  } else if (warp == 1) {
    // ---- MMA issuer (all lanes run the loop, see tc_commit)
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(P.BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    const uint64_t xd0 = smem_desc(x0), wd0 = smem_desc(raw0);
    int us = 0;
    uint32_t ph = 0, ab = 0, aph = 0;
    bool ok = true, ready = false;
    // everything the loop branches on goes through a warp reduction or vote: the compiler then knows it to be
    // uniform and keeps descriptors and addresses in uniform registers
    const int n_mine = __reduce_max_sync(0xffffffffu, mine);
    for (int i = 0; ok && i < n_mine; ++i) {
      const Item w = item(i);
      const int kb0 = __reduce_max_sync(0xffffffffu, w.kb0), kb1 = __reduce_max_sync(0xffffffffu, w.kb1);
      ok = mbar_wait_warp(acc_free + 8 * ab, aph ^ 1u, P.err);  // this buffer's last accumulators were read
      uint32_t acc = tmem + ab * (P.acc_cols * P.seq), add = 0;
      int left = P.per;  // K blocks until the next range and its accumulator
      const int k1 = ((kb1 - 1) / kSB + 1) * kSB;
      for (int k0 = kb0 / kSB * kSB; ok && k0 < k1; k0 += U) {
        if (!ready) ok = mbar_wait_warp(full + 8 * us, ph, P.err);
        if (!ok) break;
        tc_fence_after();
        const int cur = us;
        if (++us == NU) { us = 0; ph ^= 1u; }
        ready = __all_sync(0xffffffffu, mbar_test(full + 8 * us, ph));  // the next unit's barrier, looked at while this one's instructions go out
#pragma unroll
        for (int b = 0; b < U; ++b) {
          if (k0 + b < kb0 || k0 + b >= kb1) continue;
          if (left == 0) { left = P.per; acc += P.acc_cols; add = 0; }
          --left;
          const uint64_t xd = xd0 + (uint32_t)(cur * U + b) * (x_bytes >> 4);
          if (kDirect) tc_mma_block(acc, wd0 + (uint32_t)(cur * U + b) * (kWTileBytes >> 4), xd, idesc, add);
          else tc_mma_block_ts(acc, tmem_w + (uint32_t)(cur * U + b) * kWCols, xd, idesc, add);
          add = 1;
        }
        tc_commit(free_ + 8 * cur);
      }
      if (!ok) break;
      tc_commit(acc_full + 8 * ab);
      if (++ab == (uint32_t)P.nacc) { ab = 0; aph ^= 1u; }
    }
  } else if (warp >= 8) {
    // ---- dequantising warps
    const int g = (warp - 8) >> 2, q = warp & 3, r = 32 * q + lane;
    int c = g, half = 0;  // this group's unit of the next super-block: 0, 1, or 2 for none
    const uint32_t wcol = tmem_w + ((uint32_t)(q * 32) << 16);
    int us = g, rs = 0, i = 0, sb = 0, sb1 = -1;  // the group owns every G-th unit of the ring (at least G long)
    uint32_t uph = 1, rph = 0;
    bool ok = true;
    typename F::Raw R;
    const uint4 mv = lds128(smem_addr(&s_magic));
    const Magic M{mv.x, mv.y, __uint_as_float(mv.z), __uint_as_float(mv.w)};
    // moves on to the next unit of the CTA's items and reads this thread's part of it into R; false when none is left.
    // Every unit is converted whole: blocks outside the item's K range are never multiplied.
    auto next = [&]() {
      for (;;) {
        if (sb > sb1) {
          if (i >= mine) return false;
          const Item w = item(i++);
          sb = w.kb0 / kSB; sb1 = (w.kb1 - 1) / kSB;
        }
        ok = mbar_wait_warp(raw_full + 8 * rs, rph, P.err);
        if (!ok) return false;
        half = c;
        c = G == 2 ? c : c == 2 ? 0 : c + 1;
        if (G == 2 || half < kSB / U) {
          F::load(R, raw0 + (uint32_t)rs * P.raw_bytes, r, half, sb++);
          return true;
        }
        ++sb;  // the other groups have both of its units
        if (lane == 0) mbar_arrive(raw_free + 8 * rs);
        if (++rs == RS) { rs = 0; rph ^= 1u; }
      }
    };
    bool more = next();
    while (more) {
      ok = mbar_wait_warp(free_ + 8 * us, uph, P.err);  // the MMAs that read this unit's last tiles are done
      if (!ok) break;
      tc_fence_after();
      const uint32_t dst = wcol + (uint32_t)us * (U * kWCols), done = full + 8 * us, rfree = raw_free + 8 * rs;
      F::convert(R, half, M, [&](int h, const uint32_t* v) { tmem_st16(dst + 16 * h, v); });
      if ((us += G) >= NU) { us -= NU; uph ^= 1u; }
      if (++rs == RS) { rs = 0; rph ^= 1u; }
      tmem_st_wait();
      tc_fence_before();  // ordered before the MMA warp's reads through the barrier below
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(done);
        mbar_arrive(rfree);
      }
      more = next();
    }
  } else if (warp >= 4) {
    // ---- epilogue: tensor-memory lane = feature of the tile
    const int q = warp & 3;
    uint32_t ab = 0, aph = 0;
    int sbuf = 0;
    bool ok = true;
    for (int i = 0; ok && i < mine; ++i) {
      const Item w = item(i);
      const GemmJob& J = P.job[w.job];
      const int fo = w.ft * BM + q * 32 + lane;
      ok = mbar_wait_epilogue(acc_full + 8 * ab, aph, P.err);  // emit() meets at named barrier 1
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = tmem + ab * (P.acc_cols * P.seq) + ((uint32_t)(q * 32) << 16);
      // results of up to 16 tokens (v: this lane's feature of each; tok(r): which token row r is, >= ntok: none).
      // They go through shared memory, so that a token's 128 features leave in 16-byte pieces (a lane holds one
      // feature: stored from there, every token costs each warp a store of 64 bytes).
      auto emit = [&](const float* v, auto tok) {
        if (J.vec8) {
          const int row = (int)(threadIdx.x & 127) >> 3, piece = threadIdx.x & 7, t = tok(row);
          size_t orow = 0;
          if (t < w.ntok) orow = J.row_map != nullptr ? J.row_map[w.tok0 + t] : (size_t)(w.tok0 + t);
          bf16_t* st = &s_stage[sbuf][0][q * 32 + lane];
#pragma unroll
          for (int r = 0; r < 16; ++r) st[r * kStageLd] = f2bf(v[r]);
          asm volatile("bar.sync 1, 128;" ::: "memory");
          if (t < w.ntok) {
            const uint4 a0 = *reinterpret_cast<const uint4*>(&s_stage[sbuf][row][8 * piece]);
            const uint4 a1 = *reinterpret_cast<const uint4*>(&s_stage[sbuf][row][64 + 8 * piece]);
            bf16_t* y = J.y + orow * J.ldy + w.ft * BM + 8 * piece;
            if (w.ft * BM + 8 * piece < J.O) *reinterpret_cast<uint4*>(y) = a0;
            if (w.ft * BM + 64 + 8 * piece < J.O) *reinterpret_cast<uint4*>(y + 64) = a1;
          }
          sbuf ^= 1;
          return;
        }
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const int t = tok(r);
          if (t < w.ntok && fo < J.O) {
            const size_t orow = J.row_map != nullptr ? J.row_map[w.tok0 + t] : (size_t)(w.tok0 + t);
            const size_t at = orow * J.ldy + fo;
            if (J.y_f32 != nullptr) J.y_f32[at] = v[r];
            else J.y[at] = f2bf(v[r]);
          }
        }
      };
      if (C == 1) {
        for (int c0 = 0; c0 < w.ntok; c0 += 16) {  // warp-uniform
          uint32_t u[16];
          float v[16];
          tmem_ld16(acc + c0, u);
          tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 16; ++t) v[t] = __uint_as_float(u[t]);
          if (P.seq > 1) {  // the ranges of K in order
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = 0.f + v[t];
            for (int d = 1; d < P.seq; ++d) {
              tmem_ld16(acc + d * P.acc_cols + c0, u);
              tmem_ld_wait();
#pragma unroll
              for (int t = 0; t < 16; ++t) v[t] += __uint_as_float(u[t]);
            }
          }
          emit(v, [&](int r) { return c0 + r; });
        }
      } else {
        // Four tokens of a feature at a time go to the CTA of the cluster that owns them (group g of four to
        // rank g mod C), which adds the ranges in order: a fixed order, so the result depends neither on timing
        // nor on the rows beside it.  The sums are pushed, not fetched: the receiver waits on a barrier of its
        // own (reading them from the other CTAs' memory behind remote arrivals took 6700 cycles for 24
        // tokens instead of 2000), and a CTA may leave once its share has arrived.
        const int groups = (w.ntok + 3) / 4, own = groups > split ? (groups - split + C - 1) / C : 0;
        if (threadIdx.x == 128) mbar_expect_tx(part_full, (uint32_t)(own * P.splits) * (BM * 16));
        cluster_wait();  // every CTA's barriers exist
        if (threadIdx.x == 128) s_leave.met = 1;
        const uint32_t mine16 = (uint32_t)(q * 32 + lane) * 16;
        int owner = 0, slot = 0;
        for (int c0 = 0; c0 < w.ntok; c0 += 16) {
          const int owner0 = owner, slot0 = slot;
          for (int d = 0; d < P.seq; ++d) {
            uint32_t v[16];
            tmem_ld16(acc + d * P.acc_cols + c0, v);
            tmem_ld_wait();
            owner = owner0; slot = slot0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if (c0 + 4 * t < w.ntok)
                push_f4(map_to_rank(part0 + (uint32_t)((slot * P.splits + split * P.seq + d) * BM) * 16 + mine16, owner), v + 4 * t,
                        map_to_rank(part_full, owner));
              if (++owner == C) { owner = 0; ++slot; }
            }
          }
        }
        ok = mbar_wait_epilogue(part_full, 0, P.err);
        if (!ok) break;
        for (int sl0 = 0; sl0 < own; sl0 += 4) {
          float v[16];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float* r4 = v + 4 * k;
            r4[0] = r4[1] = r4[2] = r4[3] = 0.f;
            if (sl0 + k >= own) continue;
#pragma unroll
            for (int sp = 0; sp < kMaxSplit; ++sp)
              if (sp < P.splits) {
                const uint4 p = lds128(part0 + (uint32_t)((sl0 + k) * P.splits + sp) * (BM * 16) + mine16);
                r4[0] += __uint_as_float(p.x); r4[1] += __uint_as_float(p.y); r4[2] += __uint_as_float(p.z); r4[3] += __uint_as_float(p.w);
              }
          }
          emit(v, [&](int r) { return 4 * (split + (sl0 + (r >> 2)) * C) + (r & 3); });
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free + 8 * ab);
      if (++ab == (uint32_t)P.nacc) { ab = 0; aph ^= 1u; }
    }
    if (!ok) s_leave.quit = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (s_leave.quit) {
    const int groups = (min(P.BN, P.rows - first / P.f_tiles * P.BN) + 3) / 4, own = groups > split ? (groups - split + C - 1) / C : 0;
    leave_late(smem_addr(s_bar), kDirect ? 0 : RS, NU, &s_leave, C > 1, (uint32_t)(own * P.splits) * (BM * 16), P.err);
  }
  if (warp == 3) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
  }
}

// ---- grouped form: sorting and row movement --------------------------------------------------------
// counts[e] = rows routed to expert e (block-wide histogram), then seg[e] = exclusive scan
__global__ void k_route_count(const uint32_t* rhs, int rows, int E, int* seg /*[E+1]*/, int* cursor /*[E]*/) {
  extern __shared__ int s_cnt[];
  for (int i = threadIdx.x; i < E; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    const uint32_t e = rhs[i];
    if (e < (uint32_t)E) atomicAdd(&s_cnt[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) {
      seg[e] = acc;
      cursor[e] = acc;
      acc += s_cnt[e];
    }
    seg[E] = acc;
  }
}
// stable placement: sorted position of row i = seg[e] + (number of earlier rows with the same expert).
// One warp per expert scans the routing table in order, so the order inside an expert is the
// original order (counting_sort, src/ops/moe.rs:463-508).
__global__ void k_route_place(const uint32_t* rhs, int rows, int E, const int* seg, uint32_t* perm /*[rows]: sorted -> original*/) {
  const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (e >= E) return;
  int pos = seg[e];
  for (int base = 0; base < rows; base += 32) {
    const int i = base + lane;
    const bool mine = i < rows && rhs[i] == (uint32_t)e;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (mine) perm[pos + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
    pos += __popc(m);
  }
}
// the same placement for long tables, one thread per row: the slot inside an expert is taken from a
// cursor, so the order inside an expert is arbitrary (every row's result is independent of its
// neighbours, and results are stored by original row index)
__global__ void k_route_place_atomic(const uint32_t* rhs, int rows, int E, int* cursor, uint32_t* perm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows) return;
  const uint32_t e = rhs[i];
  if (e < (uint32_t)E) perm[atomicAdd(&cursor[e], 1)] = (uint32_t)i;
}
// xs[p] = x[lhs[perm[p]]] (rows of K bf16)
__global__ void k_gather_rows(const bf16_t* x, const uint32_t* lhs, const uint32_t* perm, int rows, int K, bf16_t* xs) {
  const int p = blockIdx.x;
  if (p >= rows) return;
  const uint32_t o = perm[p];
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(lhs ? lhs[o] : o) * K);
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)p * K);
  for (int i = threadIdx.x; i < K / 8; i += blockDim.x) dst[i] = src[i];
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

std::mutex g_gemm_mu;

template <int KIND, int G>
int launch_qgemm(orn_ctx* ctx, cudaStream_t s, const GemmMaps& maps, const GemmParams& P, int grid, size_t smem) {
  int rc = orn_grant_smem(ctx, reinterpret_cast<const void*>(k_qgemm<KIND, G>), kGemmSmem);
  if (rc != ORN_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(gemm_threads(G));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = P.splits / P.seq; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = P.splits > P.seq ? 1 : 0;
  ORN_CHECK_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_qgemm<KIND, G>, maps, P));
  if (ctx->kt == nullptr) return orn_launch_check(ctx, "k_qgemm");
  // per-kernel timing: one label per shape
  static std::set<std::string> pool;
  char buf[96];
  snprintf(buf, sizeof buf, "k_qgemm kind=%d O=%d%s K=%d rows=%d %s", KIND, P.job[0].O, P.njobs > 1 ? "+" : "", P.K, P.rows, P.seg ? "grouped" : "dense");
  std::lock_guard<std::mutex> lock(g_gemm_mu);
  return orn_launch_check(ctx, pool.insert(buf).first->c_str());
}

uint32_t raw_bytes(int kind) {
  switch (kind) {
    case ORN_Q4K: return Fmt<ORN_Q4K>::kRawBytes;
    case ORN_Q6K: return Fmt<ORN_Q6K>::kRawBytes;
    case ORN_A8: return Fmt<ORN_A8>::kRawBytes;
    case ORN_A4: return Fmt<ORN_A4>::kRawBytes;
    default: return Fmt<ORN_BF16>::kRawBytes;
  }
}

}  // namespace

// y[rows, O] (row stride ldy) = x[rows, K] W^T.  grp != null: rows are sorted by expert, expert e
// owns rows seg[e] .. seg[e+1]-1 (device array of E + 1 ints) and multiplies by W[e]; row p of the
// result goes to output row row_map[p] when row_map is given.
// (map0 of f_qgemm_multi: the same for the first matrix of a dense launch.)
int f_qgemm(orn_ctx* ctx, cudaStream_t s, const orn_linear* L, const bf16_t* x, int rows, void* y, int ldy,
            const QGemmGroup* grp, int out_f32) {
  return f_qgemm_multi(ctx, s, &L, &y, &ldy, 1, x, rows, grp, out_f32);
}

// Up to four matrices of one format and row length over the same rows in ONE launch (the projections
// of a layer that share their input): their feature tiles form one tile space.  n == 1 is f_qgemm.
// Dense products over few rows: the K blocks of a tile go to the CTAs of a cluster, which add their
// f32 partials in split order through distributed shared memory.  The number of splits depends on the
// matrices (and on rows only in steps of 256), so that a row's bits do not depend on the rows beside it:
// one round of items over the SMs, two where the tiles alone would leave half of the SMs idle, at
// least 4 K blocks per item, no split empty.
int f_qgemm_splits(const orn_ctx* ctx, int f_tiles, int rows, int K) {
  const int KB = K / BK;
  if (rows > kSplitMaxRows || KB < 8) return 1;
  const int tiles = f_tiles * ((rows + 255) / 256);
  int sp = std::max(1, (tiles > ctx->sm_count / 2 ? 2 * ctx->sm_count : ctx->sm_count) / tiles);
  sp = std::min(sp, std::min(kMaxSplit, KB / 4));
  if (sp > 1) {
    const int per = (KB + sp - 1) / sp;
    sp = (KB + per - 1) / per;
  }
  return sp;
}

int f_qgemm_multi(orn_ctx* ctx, cudaStream_t s, const orn_linear* const* Ls, void* const* ys, const int* ldys, int n,
                  const bf16_t* x, int rows, const QGemmGroup* grp, int out_f32, const uint32_t* map0) {
  if (rows < 1) return ORN_OK;
  if (n < 1 || n > kMaxJobs) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: 1..4 matrices per launch");
  const orn_linear* L = Ls[0];
  for (int j = 1; j < n; ++j)
    if (Ls[j]->kind != L->kind || Ls[j]->K != L->K || Ls[j]->E != L->E)
      ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: the matrices of one launch share format and row length");
  if (L->K % BK) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: K must be a multiple of 64");
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: x must be 16-byte aligned");
  if (grp == nullptr && L->E != 1) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: a routed weight goes through the grouped form");
  if (grp != nullptr && L->E > kMaxE) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: more than 1024 experts");
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) ORN_FAIL(ctx, ORN_ERR_CUDA, "gemm: the driver has no cuTensorMapEncodeTiled");
  GemmParams P;
  memset(&P, 0, sizeof P);
  P.njobs = n;
  for (int j = 0; j < n; ++j) {
    GemmJob& J = P.job[j];
    J.O = Ls[j]->O; J.tile0 = P.f_tiles; J.ldy = ldys[j];
    J.row_map = grp ? grp->row_map : j == 0 ? map0 : nullptr;
    J.y = out_f32 ? nullptr : reinterpret_cast<bf16_t*>(ys[j]);
    J.y_f32 = out_f32 ? reinterpret_cast<float*>(ys[j]) : nullptr;
    J.vec8 = !out_f32 && (ldys[j] & 7) == 0 && (Ls[j]->O & 7) == 0 && (reinterpret_cast<uintptr_t>(ys[j]) & 15) == 0;
    P.f_tiles += (Ls[j]->O + BM - 1) / BM;
  }
  const bool direct = L->kind == ORN_BF16;
  // Groups of dequantising warps.  Dense products that do not split K are tiles of 80 to 128 tokens, whose weight ring is
  // two to four units: a third group keeps a unit more under way (1001 x 2048 -> 8192 affine-8 55.3 -> 48.8 us, a
  // prompt of 6621 rows 14.01 -> 13.67 ms).  Routed rows and split products have long rings and are bound by the
  // instructions of all roles, where four more warps with fewer registers cost (1024 routed Q4_K rows 126 -> 130 us,
  // Q6_K 78 -> 89 us; 64 sequences with split products on three groups 17.8 -> 18.7 ms).
  const int G = grp == nullptr && rows > kSplitMaxRows ? 3 : 2;
  const int KB = L->K / BK;
  P.K = L->K; P.rows = rows; P.err = ctx->dev_err;
  P.seg = grp ? grp->seg : nullptr;
  P.E = L->E;
  P.splits = grp == nullptr ? f_qgemm_splits(ctx, P.f_tiles, rows, L->K) : 1;
  P.seq = 1;
  P.per = (KB + P.splits - 1) / P.splits;
  // Token-tile width.  Few rows: one tile that holds them.  Many rows: the width (at most 128, so that two
  // accumulators and the weight ring fit tensor memory) that finishes first over whole rounds of the SMs.  With two
  // groups a tile of 96 tokens or less costs what 100 do, a wider one its columns.  With three its weights, converted
  // once per tile, are nearly all of it: a round of 128 / 112 / 96 / 80 tokens takes 9.5 / 9.2 / 8.8 / 8.6 us at 6621
  // rows 2048 -> 8192 affine-8 (2048 rows 2048 -> 4096: 48 us at the 128 of that rule, 56 at the 96 of the other).
  // bfloat16 weights, which nothing converts, have a ring of two units beside 96 tokens or more and of four beside 80:
  // 2048 rows 2048 -> 4096 take 61.5 / 63.5 / 69.7 / 51.2 us, 513 rows 4096 -> 2048 36.9 / 34.8 / 34.8 / 24.6.  Routed
  // rows: wide enough for an expert's rows in nearly every case (mean plus three standard deviations), since every
  // further item of an expert dequantises its weights again, while columns up to about 96 hide behind the
  // dequantisation.
  auto up16 = [](int v) { return (v + 15) / 16 * 16; };
  if (grp) {
    const double per = grp->bn_hint > 0 ? grp->bn_hint : std::max(1, (rows + L->E - 1) / L->E);
    const int want = (int)std::ceil(per + 3.0 * std::sqrt(per));
    const int groups = (want + 127) / 128;
    P.BN = std::max(16, up16((want + groups - 1) / groups));
  } else if (rows <= 128 || P.splits > 1) {
    P.BN = std::min(128, up16(rows));
  } else if (direct && rows > kSplitMaxRows) {
    P.BN = 80;
  } else {
    int64_t best = -1;
    for (int bn = 128; bn >= 80; bn -= 16) {
      const int64_t items = (int64_t)P.f_tiles * ((rows + bn - 1) / bn);
      const int64_t cost = (items + ctx->sm_count - 1) / ctx->sm_count * (G == 3 ? bn + 380 : std::max(2 * bn, 200));
      if (best < 0 || cost < best) { best = cost; P.BN = bn; }
    }
  }
  P.acc_cols = ((uint32_t)P.BN + 31u) & ~31u;
  // Two or three ranges: one CTA takes them one after the other (no exchange; the tiles fill at least a third of
  // the SMs).  More: clusters of at most four CTAs where the count and the memory allow (a GPC holds two clusters
  // of eight at most, so eight do not place on every SM), each taking its ranges one after the other.
  const size_t unit_b = (size_t)U * ((size_t)P.BN * 128 + (direct ? kWTileBytes : 0)), room = kGemmSmem - 1024;
  const size_t raw_b = direct ? 0 : raw_bytes(L->kind);
  auto part_bytes = [&](int c) { return c > 1 ? (size_t)((P.BN / 4 + c - 1) / c * P.splits) * (BM * 16) : 0; };
  if (P.splits > 1) {
    const int most = (512 - G * U * (int)kWCols) / (int)P.acc_cols;
    int c = P.splits <= std::min(3, most) ? 1 : P.splits;
    for (int t = std::min(4, P.splits); c > 1 && t >= 2; --t)
      if (P.splits % t == 0 && P.splits / t <= most && part_bytes(t) + G * unit_b + 2 * raw_b <= room) { c = t; break; }
    P.seq = P.splits / c;
  }
  const int C = P.splits / P.seq;
  // Tensor memory: the accumulators (two sets where an item has one) and an even number of units of weight
  // tiles.  Shared memory: the units' token tiles, the partial sums that arrive from a cluster, raw slots.
  P.raw_bytes = raw_bytes(L->kind);
  P.nacc = P.seq == 1 ? 2 : 1;
  const uint32_t accs = P.nacc * P.seq * P.acc_cols;
  const size_t part = part_bytes(C);
  if (direct) {
    P.units = (int)std::min<size_t>(kMaxUnits, (room - part) / unit_b) & ~1;
    P.raw_slots = P.units * U;
    P.raw_bytes = kWTileBytes;
  } else {
    // (two groups own even and odd units, so their ring has an even number; three take a raw slot less for a unit more)
    for (P.units = 6; P.units > G; P.units -= G == 2 ? 2 : 1)
      if (accs + P.units * U * kWCols <= 512 && P.units * unit_b + (G == 2 || P.units > 4 ? 3 : 2) * P.raw_bytes + part <= room) break;
    P.raw_slots = (int)std::min<size_t>(kMaxRaw, (room - part - P.units * unit_b) / P.raw_bytes);
  }
  if (P.units < (direct ? 2 : G) || accs + (direct ? 0 : P.units * U * kWCols) > 512 || P.raw_slots < 1) ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: the rings do not fit into shared memory");
  const size_t rings = P.units * unit_b + (direct ? 0 : (size_t)P.raw_slots * P.raw_bytes) + part;
  P.tmem_cols = 32;
  while (P.tmem_cols < accs + (direct ? 0u : P.units * U * kWCols)) P.tmem_cols <<= 1;
  // one CTA per SM (it may take all of tensor memory): never less than half of the SM's shared memory
  const size_t smem = std::max<size_t>(120 * 1024, 1024 + rings);
  GemmMaps maps;
  memset(&maps, 0, sizeof maps);
  auto encode = [&](CUtensorMap* m, CUtensorMapDataType dt, void* base, uint64_t inner, uint64_t outer, uint64_t stride_bytes,
                    uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw) -> bool {
    const cuuint64_t gdim[2] = {inner, outer};
    const cuuint64_t gstride[1] = {stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, dt, 2, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  bool ok = encode(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, const_cast<bf16_t*>(x), (uint64_t)L->K, (uint64_t)rows,
                   (uint64_t)L->K * 2, BK, (uint32_t)P.BN, CU_TENSOR_MAP_SWIZZLE_128B);
  for (int j = 0; j < n; ++j) {
    const orn_linear* Lj = Ls[j];
    WeightMaps& wm = maps.w[j];
    const uint64_t wrows = (uint64_t)Lj->E * Lj->O;
    auto box = [&](CUtensorMap* m, uint32_t bytes, CUtensorMapSwizzle sw) {
      ok = ok && encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, Lj->w, (uint64_t)Lj->rec, wrows, (uint64_t)Lj->rec, bytes, BM, sw);
    };
    if (direct) {
      ok = ok && encode(&wm.wide, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, Lj->w, (uint64_t)Lj->K, wrows, (uint64_t)Lj->rec, BK, BM,
                        CU_TENSOR_MAP_SWIZZLE_128B);
      continue;
    }
    box(&wm.wide, 128, CU_TENSOR_MAP_SWIZZLE_128B);
    if (L->kind == ORN_Q6K) box(&wm.mid, 64, CU_TENSOR_MAP_SWIZZLE_64B);
    box(&wm.scale, L->kind == ORN_A4 ? 32 : 16, CU_TENSOR_MAP_SWIZZLE_NONE);
  }
  if (!ok) ORN_FAIL(ctx, ORN_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed");
  int grid = ctx->sm_count;
  if (grp == nullptr) {
    P.dense_tiles = P.f_tiles * ((rows + P.BN - 1) / P.BN);
    grid = C > 1 ? P.dense_tiles * C : std::min(P.dense_tiles, ctx->sm_count);  // a cluster has one tile
  }
#define QGEMM(kind) return G == 2 ? launch_qgemm<kind, 2>(ctx, s, maps, P, grid, smem) : launch_qgemm<kind, 3>(ctx, s, maps, P, grid, smem)
  switch (L->kind) {
    case ORN_Q4K: QGEMM(ORN_Q4K);
    case ORN_Q6K: QGEMM(ORN_Q6K);
    case ORN_A8: QGEMM(ORN_A8);
    case ORN_BF16: return launch_qgemm<ORN_BF16, 0>(ctx, s, maps, P, grid, smem);
    case ORN_A4: QGEMM(ORN_A4);
  }
#undef QGEMM
  ORN_FAIL(ctx, ORN_ERR_ARG, "gemm: unknown weight format");
}

// rows sorted by expert: seg[E+1] and perm[rows] (sorted position -> original row)
int f_route_sort(orn_ctx* ctx, cudaStream_t s, const uint32_t* rhs, int rows, int E, int* seg, int* cursor, uint32_t* perm) {
  if (E > 4096) ORN_FAIL(ctx, ORN_ERR_ARG, "route sort: more than 4096 experts");
  int rc = ORN_OK;
  // (400 routes over 256 experts: one launch 4.5 us, count and placement 12)
  if (rows < 4096 && orn_route_small(ctx, s, rhs, rows, E, seg, perm, &rc)) return rc;
  k_route_count<<<1, 1024, E * sizeof(int), s>>>(rhs, rows, E, seg, cursor);
  rc = orn_launch_check(ctx, "k_route_count");
  if (rc != ORN_OK) return rc;
  if (rows >= 4096) k_route_place_atomic<<<(rows + 255) / 256, 256, 0, s>>>(rhs, rows, E, cursor, perm);
  else k_route_place<<<(E + 7) / 8, 256, 0, s>>>(rhs, rows, E, seg, perm);
  return orn_launch_check(ctx, "k_route_place");
}

int f_gather_rows(orn_ctx* ctx, cudaStream_t s, const bf16_t* x, const uint32_t* lhs, const uint32_t* perm, int rows, int K,
                  bf16_t* xs) {
  if (K % 8) ORN_FAIL(ctx, ORN_ERR_ARG, "gather rows: K must be a multiple of 8");
  k_gather_rows<<<rows, 128, 0, s>>>(x, lhs, perm, rows, K, xs);
  return orn_launch_check(ctx, "k_gather_rows");
}
