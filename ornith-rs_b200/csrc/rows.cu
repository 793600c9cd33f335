// The row-invariant mat-vec over many rows at once: y[p] = W[e] x[p] with the bits of the one-row mat-vec, for a
// short prompt, a small batch, a router, the experts of the exact expert-parallel block.
//
// Every result is the sum the one-row kernels define (src/ops/invariant.rs:78-168 is what the reference holds its rows
// to): lane l folds units l, l + 32, .. of the row in ascending order, each through two chains of fused
// multiply-adds, and the lanes meet in the xor-16 .. 1 butterfly.  That rules out the tensor cores, so what counts is
// the FMA pipe: a packed multiply-add takes two cycles of a scheduler, and everything else has to fit beside it.
//   * a lane holds its unit of up to eight rows in registers (128 floats) and takes R features past them: a weight is
//     widened once for all of those rows (1.5 instructions; the four-row windows do it for every four rows);
//   * activations come as bfloat16 through L1 and are widened once per unit for R features;
//   * a warp owns its R features: their records lie behind one another and come by cp.async into the warp's own piece
//     of shared memory.  Warps never meet; two to four CTAs of four warps on an SM cover each other's copies.
// FMA work of a unit of 16 weights, 8 rows x 8 features: 512 packed multiply-adds of 1024 cycles in about 1500.
// 50 rows, 2048 -> 12288 affine-8: 110 us.  Its multiply-adds are 31 % of what the float32 pipe could do in that time (34 %
// with the rows padded to 56), the pipe is active 55 % of the cycles, issue slots are 53 % busy: 255 registers leave two
// warps a scheduler, whose chains of dependent packed multiply-adds leave the rest empty.  What it replaced there
// read the weights once per four rows, 13 launches of about 17 us.
#include <algorithm>

#include "fused.h"
#include "mma_bf16.cuh"
#include "orn_internal.h"
#include "units.cuh"

namespace {

constexpr int kRowWarps = 4;  // per CTA
constexpr size_t kRowSmem = 200 * 1024;
constexpr int kRowMaxO = 65535 * 4 * kRowWarps;  // features of a launch: a grid's y, four features a warp

struct RowsTile {
  const uint8_t* w;
  bf16_t* y;
  int O, tile0;  // features; first warp tile of this matrix
};
struct RowsParams {
  RowsTile job[4];
  int njobs, tiles;          // matrices of one format and row length over the same rows; their warp tiles
  int K, units;
  uint32_t rec, b0, b1, tile_bytes;
  int slots;                 // tiles of a warp in shared memory: 2 where it takes several
  const bf16_t* xs;
  const int* seg;            // nullable (one matrix, rows 0 .. rows - 1); expert e owns rows seg[e] .. seg[e + 1] - 1
  int rows;
  const uint32_t* row_map;   // nullable: output row of row p
};

// activations of unit u, in the order of the unit's weights, and their sums (ascending, from zero)
ORN_D void widen4(const uint2& v, float* f) { f[0] = bf_lo(v.x); f[1] = bf_hi(v.x); f[2] = bf_lo(v.y); f[3] = bf_hi(v.y); }
ORN_D float sum16(const float* f) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) s = s + f[i];
  return s;
}
template <int KIND> ORN_D void unit_x(const bf16_t* x, int u, float* f, float* sm) {
  if (KIND == ORN_Q6K) {
    const bf16_t* p = x + (u >> 4) * 256 + 128 * ((u & 15) >> 3) + 4 * (u & 7);
#pragma unroll
    for (int i = 0; i < 4; ++i) widen4(__ldg(reinterpret_cast<const uint2*>(p + 32 * i)), f + 4 * i);
  } else if (KIND == ORN_Q4K) {
    const bf16_t* p = x + (u >> 3) * 256 + 64 * ((u & 7) >> 1) + 16 * (u & 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) widen8(__ldg(reinterpret_cast<const uint4*>(p + 8 * (i & 1) + 32 * (i >> 1))), f + 8 * i);
    sm[0] = sum16(f);
    sm[1] = sum16(f + 16);
  } else if (KIND == ORN_A8) {
    widen8(__ldg(reinterpret_cast<const uint4*>(x + 16 * u)), f);
    widen8(__ldg(reinterpret_cast<const uint4*>(x + 16 * u + 8)), f + 8);
    sm[0] = sum16(f);
  } else {
    widen8(__ldg(reinterpret_cast<const uint4*>(x + 8 * u)), f);
  }
}

// M rows from row g0 on (of n; past the last one the last one again) against the R features in `tile`
ORN_D void wait_tile(const RowsParams& P) {
  if (P.slots > 1) cp_async_wait<1>();
  else cp_async_wait<0>();
  __syncwarp();
}
// LATE: the tile's records are waited for behind the request of the first activations (few rows, where that latency
// counts; with more rows the branch costs the registers of the loop)
template <int KIND, int R, int M, bool LATE>
ORN_D void rows_group(const RowsParams& P, const RowsTile& J, const uint8_t* tile, int row0, int first, int g0, int n, int lane, bool& landed) {
  using U = WU<KIND>;
  constexpr int NX = Lay<KIND>::P * 4, NS = Lay<KIND>::NS > 0 ? Lay<KIND>::NS : 1, V = R * M < 32 ? R * M : 32;
  float acc[R * M];
#pragma unroll
  for (int i = 0; i < R * M; ++i) acc[i] = 0.f;
#pragma unroll 1
  for (int u = lane; u < (LATE ? (P.units + 31) & ~31 : P.units); u += 32) {
    float x[M][NX], sm[M][NS];
    if (!LATE || u < P.units)
#pragma unroll
      for (int m = 0; m < M; ++m) unit_x<KIND>(P.xs + (size_t)(first + min(g0 + m, n - 1)) * P.K, u, x[m], sm[m]);
    if (LATE && !landed) {
      wait_tile(P);
      landed = true;
    }
    if (LATE && u >= P.units) continue;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      typename U::W w;
      U::lds(tile + r * P.rec, P.b0, P.b0 + P.b1, u, w);
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r * M + m] = U::fold(w, x[m], sm[m], u, acc[r * M + m]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < R * M / V; ++c) {
    int which;
    const float v = rs_butterfly<V>(acc + c * V, lane, which);
    const int r = (c * V + which) / M, m = (c * V + which) % M;
    if ((lane & (32 / V - 1)) != 0 || g0 + m >= n || row0 + r >= J.O) continue;
    const int p = first + g0 + m;
    J.y[(P.row_map != nullptr ? P.row_map[p] : (uint32_t)p) * (size_t)J.O + row0 + r] = f2bf(v);
  }
}

template <int KIND, int R, int MAX>
__global__ void __launch_bounds__(32 * kRowWarps) k_rows(const __grid_constant__ RowsParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.z;
  const int first = P.seg != nullptr ? P.seg[e] : 0, n = P.seg != nullptr ? P.seg[e + 1] - first : P.rows;
  const int stride = gridDim.y * kRowWarps;
  int t = blockIdx.y * kRowWarps + warp;
  if (n <= (int)blockIdx.x * MAX || t >= P.tiles) return;
  uint8_t* buf = smem + (size_t)warp * P.slots * P.tile_bytes;
  auto job_of = [&](int tile) {
    int j = 0;
    while (j + 1 < P.njobs && tile >= P.job[j + 1].tile0) ++j;
    return j;
  };
  auto request = [&](int tile, int slot) {
    if (tile < P.tiles) {
      const RowsTile& J = P.job[job_of(tile)];
      const int row0 = (tile - J.tile0) * R;
      const uint8_t* src = J.w + ((size_t)e * J.O + row0) * P.rec;
      const uint32_t bytes = (uint32_t)min(R, J.O - row0) * P.rec, dst = smem_u32(buf) + slot * P.tile_bytes;
      for (uint32_t i = lane * 16; i < bytes; i += 512) cp_async16(dst + i, src + i, 16);
    }
    cp_async_commit();
  };
  request(t, 0);
  for (int slot = 0; t < P.tiles; t += stride) {
    if (P.slots > 1) request(t + stride, slot ^ 1);
    bool landed = false;
    if (MAX > 2) wait_tile(P);
    const RowsTile& J = P.job[job_of(t)];
    const uint8_t* tile = buf + slot * P.tile_bytes;
    const int row0 = (t - J.tile0) * R;
    for (int g0 = blockIdx.x * MAX; g0 < n; g0 += gridDim.x * MAX) {
      const int c = n - g0;
      if (MAX == 2 || c <= 2) rows_group<KIND, R, 2, MAX == 2>(P, J, tile, row0, first, g0, n, lane, landed);
      else if (MAX == 4 || c <= 4) rows_group<KIND, R, 4, false>(P, J, tile, row0, first, g0, n, lane, landed);
      else rows_group<KIND, R, MAX, false>(P, J, tile, row0, first, g0, n, lane, landed);
    }
    __syncwarp();
    if (P.slots > 1) slot ^= 1;
  }
  cp_async_wait<0>();
}

template <int KIND, int R, int MAX>
int launch_rows(orn_ctx* ctx, cudaStream_t s, RowsParams& P, int E) {
  const int64_t rows = P.rows;
  for (int j = 0; j < P.njobs; ++j) {
    P.job[j].tile0 = P.tiles;
    P.tiles += (P.job[j].O + R - 1) / R;
  }
  P.tile_bytes = R * P.rec;
  P.slots = E > 1 && P.units <= 32 ? 2 : 1;  // short rows: two tiles a warp
  int rc = orn_grant_smem(ctx, reinterpret_cast<const void*>(k_rows<KIND, R, MAX>), kRowSmem);
  if (rc != ORN_OK) return rc;
  const int64_t g = (rows + MAX - 1) / MAX, gx = E > 1 ? 1 : g * P.tiles > 8 * kRowWarps * ctx->sm_count ? (g + 1) / 2 : g;
  const int per = kRowWarps * P.slots;
  k_rows<KIND, R, MAX><<<dim3((unsigned)gx, (P.tiles + per - 1) / per, E), 32 * kRowWarps, (size_t)kRowWarps * P.slots * P.tile_bytes, s>>>(P);
  return orn_launch_check(ctx, "k_rows");
}
// Eight features a warp while their records stay below 18 KB, so that three CTAs fit an SM, four of longer rows.
template <int KIND, int MAX>
int launch_max(orn_ctx* ctx, cudaStream_t s, RowsParams& P, int E, int features) {
  const bool eight = 8 * P.rec <= 18 * 1024;
  if (E > 1) return eight ? launch_rows<KIND, 8, 2>(ctx, s, P, E) : launch_rows<KIND, 4, 2>(ctx, s, P, E);
  // a narrow matrix: four or two rows a CTA, so that the launch reaches more SMs
  const int64_t ctas = (features + 31) / 32;
  const bool full = ctas * ((P.rows + MAX - 1) / MAX) >= ctx->sm_count, half = ctas * ((P.rows + 3) / 4) >= ctx->sm_count;
  if (eight) return full ? launch_rows<KIND, 8, MAX>(ctx, s, P, E) : half ? launch_rows<KIND, 8, 4>(ctx, s, P, E) : launch_rows<KIND, 8, 2>(ctx, s, P, E);
  // Long rows are tiles of 9 to 50 KB a warp, which every further group of rows copies again while few CTAs share an SM.
  // Of affine-8 and bfloat16, the most bytes a weight, two rows a CTA do not pay for that (two / four rows, us: affine-8
  // 2048 x 4096 8 rows 18.7 / 12.3, 2048 x 6144 5 rows 23.3 / 16.4; bfloat16 2048 x 4096 6 rows 27.6 / 16.7, where the
  // mat-vec of four rows at a time takes 18.5), of the k-quants they do (Q6_K 2048 x 4096 5 rows 12.6 / 14.4, Q4_K 2048 x 6144
  // 15.4 / 19.5).  bfloat16 is never better off with eight (four / eight: 8192 x 2048 5 rows 18.5 / 24.7, 50 rows 78 / 88).
  constexpr bool kQuant = KIND == ORN_Q4K || KIND == ORN_Q6K;
  constexpr int kMost = KIND == ORN_BF16 ? 4 : MAX, kLeast = kQuant ? 2 : 4;
  return full ? launch_rows<KIND, 4, kMost>(ctx, s, P, E) : half ? launch_rows<KIND, 4, 4>(ctx, s, P, E) : launch_rows<KIND, 4, kLeast>(ctx, s, P, E);
}

}  // namespace

bool f_rows_ok(const orn_linear* L) {
  return L->kind != ORN_A4 && L->K % 256 == 0 && L->E <= 65535 && L->O <= kRowMaxO && (size_t)(L->E > 1 ? 8 : 4) * kRowWarps * L->rec <= kRowSmem;
}

// Up to four matrices of one format and row length over the same rows, or (seg given) one matrix over rows sorted by
// expert.  Dense rows go eight at a time (a unit of Q4_K is 32 weights: four), two groups a CTA where there are many; an
// expert's rows, one or two as a rule, two at a time in the CTA that holds its features, which leaves registers for twice
// the warps (400 rows over 256 Q4_K experts 87 us four at a time, 76 two; two tiles a warp only where a row is one step
// long: Q6_K of 512 weights 98 -> 95 us, Q4_K of 2048 76 -> 80).
int f_rows(orn_ctx* ctx, cudaStream_t s, const orn_linear* const* Ls, bf16_t* const* ys, int n, const bf16_t* xs, int rows, const int* seg,
           const uint32_t* row_map) {
  if (rows < 1) return ORN_OK;
  if (n < 1 || n > 4 || !f_rows_ok(Ls[0]) || (reinterpret_cast<uintptr_t>(xs) & 15) != 0)
    ORN_FAIL(ctx, ORN_ERR_ARG, "rows: 1..4 matrices of a served format, 16-byte aligned rows");
  const orn_linear* L = Ls[0];
  RowsParams P{};
  for (int j = 0; j < n; ++j) {
    if (Ls[j]->kind != L->kind || Ls[j]->K != L->K || Ls[j]->E != L->E) ORN_FAIL(ctx, ORN_ERR_ARG, "rows: matrices of one launch share format and row length");
    P.job[j] = RowsTile{Ls[j]->w, ys[j], Ls[j]->O, 0};
  }
  if (L->E > 1 && (seg == nullptr || n > 1)) ORN_FAIL(ctx, ORN_ERR_ARG, "rows: experts come one matrix at a time, with their row ranges");
  const RecGeom g = rec_geom(L->kind, L->K);
  P.njobs = n; P.K = L->K; P.rec = g.rec; P.b0 = g.b0; P.b1 = g.b1;
  P.xs = xs; P.seg = seg; P.rows = rows; P.row_map = row_map;
  int features = 0;
  for (int j = 0; j < n; ++j) {
    if (Ls[j]->O > kRowMaxO) ORN_FAIL(ctx, ORN_ERR_ARG, "rows: more features than a launch holds");
    features += Ls[j]->O;
  }
  if (features > kRowMaxO) {  // (n > 1) one matrix after the other
    for (int j = 0; j < n; ++j) {
      const int rc = f_rows(ctx, s, Ls + j, ys + j, 1, xs, rows, seg, row_map);
      if (rc != ORN_OK) return rc;
    }
    return ORN_OK;
  }
  switch (L->kind) {
    case ORN_Q4K: P.units = L->K / 32; return launch_max<ORN_Q4K, 4>(ctx, s, P, L->E, features);
    case ORN_Q6K: P.units = L->K / 16; return launch_max<ORN_Q6K, 8>(ctx, s, P, L->E, features);
    case ORN_A8: P.units = L->K / 16; return launch_max<ORN_A8, 8>(ctx, s, P, L->E, features);
    default: P.units = L->K / 8; return launch_max<ORN_BF16, 8>(ctx, s, P, L->E, features);
  }
}
