// Launchers of the persistent fused kernels (fused.cu).
#pragma once

#include <algorithm>

#include "orn_internal.h"

enum { PRO_ADDNORM = 0, PRO_PLAIN = 1, PRO_GATED = 2, PRO_MTPJOIN = 3 };
enum { EPI_STORE = 0, EPI_SWIGLU = 1 };

// How a kernel rebuilds its input row(s) in shared memory.
struct FusedPrologue {
  int mode = PRO_PLAIN;
  int K = 0;                      // length of the staged row
  const bf16_t* a = nullptr;      // ADDNORM/PLAIN: [M][K]; GATED: y [M][K]; MTPJOIN: trunk hidden [M][K/2]
  const bf16_t* b = nullptr;      // ADDNORM: second addend (nullable); GATED: z [M][K]
  const bf16_t* w = nullptr;      // norm weight (GATED: [128]; MTPJOIN: embedding-side norm)
  const bf16_t* w2 = nullptr;     // MTPJOIN: hidden-side norm
  bf16_t* sum_out = nullptr;      // ADDNORM: bf(a+b) written by CTA 0
  bf16_t* norm_out = nullptr;     // staged row written by CTA 0
  const orn_linear* emb = nullptr;  // MTPJOIN: embedding table
  const uint32_t* ids = nullptr;    // MTPJOIN: token ids (device)
  float eps = 1e-6f;
};

struct FusedJob {
  const orn_linear* lin = nullptr;
  const orn_linear* lin2 = nullptr;  // EPI_SWIGLU: the "up" matrix
  bf16_t* out = nullptr;             // [M][O]
  int epi = EPI_STORE;
};

// Weights that the kernel behind the experts of a layer reads (the next layer's input projections, 27 MB, or
// the head's first rows), requested into L2 by the expert up kernel while it waits for its routing: a hint,
// nothing waits for it.  64 tokens to a 51-token prompt 161.8 -> 159.9 ms.  The same for what follows the recurrence and
// the attention (9 MB) brought nothing.
struct L2Hint {
  const uint8_t* at[4] = {};
  uint32_t bytes[4] = {};
  void add(const orn_linear* L) {
    for (int i = 0; i < 4; ++i)
      if (at[i] == nullptr) {
        at[i] = L->w;
        bytes[i] = (uint32_t)std::min(L->w_bytes, (size_t)24 << 20) & ~15u;
        return;
      }
  }
};

int f_norm_gemv(orn_ctx* ctx, cudaStream_t s, int M, const FusedPrologue& fp, const FusedJob* jobs, int njobs);
int f_moe_up(orn_ctx* ctx, cudaStream_t s, int M, const bf16_t* logits, const bf16_t* x, const orn_linear* gate,
             const orn_linear* up, int k, uint32_t* inds, bf16_t* scores, bf16_t* act, const L2Hint& hint = {});
int f_moe_down(orn_ctx* ctx, cudaStream_t s, int M, const bf16_t* act, const bf16_t* sact, const uint32_t* inds,
               const bf16_t* scores, const bf16_t* gs, const orn_linear* down, const orn_linear* sh_down, int k,
               int normalize, bf16_t* out);
int f_gdn(orn_ctx* ctx, cudaStream_t s, const bf16_t* conv, const bf16_t* cw, const bf16_t* a, const bf16_t* b,
          const bf16_t* a_log, const bf16_t* dt_bias, float* ring, int nring, const int* cur, int final_only, int T,
          int Hk, int Hv, int Kc, float eps, bf16_t* y, const bf16_t* z, const bf16_t* norm_w, float norm_eps,
          bf16_t* gated_out /* nullable: rms_norm_gated(y, z) per head, by the last CTA of the head */,
          int B = 1, int64_t conv_stride = 0 /* sequences of T rows each: conv windows conv_stride elements apart */);
int f_attn(orn_ctx* ctx, cudaStream_t s, const bf16_t* qg, const bf16_t* k, const bf16_t* v, const bf16_t* q_norm,
           const bf16_t* k_norm, bf16_t* kc, bf16_t* vc, const int* pos, int T, int Hq, int Hkv, int hd, int cap,
           int rope_dims, float lnb, float eps, bf16_t* out,
           int long_context = 0 /* the key groups of a (head, row) over four CTAs: same bits, for long caches */,
           int B = 1 /* sequences of T rows each */);
// one warp waits, with a limit of `rounds` tries, for a copy that was never requested: sets the
// context's device error flag; *dev_waited receives 0
int f_wait_probe(orn_ctx* ctx, cudaStream_t s, uint32_t rounds, int* dev_waited);

// ---- gemm.cu: the wide (>= 16 rows) mat-mul on the tensor cores
struct QGemmGroup {
  const int* seg;           // device [E + 1]: expert e owns sorted rows seg[e] .. seg[e+1]-1
  const uint32_t* row_map;  // device [rows] or null: output row of sorted row p
  int bn_hint;              // > 0: expected rows per expert (picks the token-tile width)
};
int f_qgemm(orn_ctx* ctx, cudaStream_t s, const orn_linear* L, const bf16_t* x, int rows, void* y, int ldy,
            const QGemmGroup* grp /*nullable: dense*/, int out_f32 = 0);
// up to four matrices of one format and row length over the same rows in one launch
int f_qgemm_splits(const orn_ctx* ctx, int f_tiles, int rows, int K);  // ranges of K of a dense launch with that many 128-feature tiles
int f_qgemm_multi(orn_ctx* ctx, cudaStream_t s, const orn_linear* const* Ls, void* const* ys, const int* ldys, int n,
                  const bf16_t* x, int rows, const QGemmGroup* grp = nullptr, int out_f32 = 0,
                  const uint32_t* map0 = nullptr /*dense: output rows of the first matrix*/);
int f_route_sort(orn_ctx* ctx, cudaStream_t s, const uint32_t* rhs, int rows, int E, int* seg, int* cursor, uint32_t* perm);
int f_gather_rows(orn_ctx* ctx, cudaStream_t s, const bf16_t* x, const uint32_t* lhs /*nullable*/, const uint32_t* perm,
                  int rows, int K, bf16_t* xs);

// ---- rows.cu: the row-invariant mat-vec over many rows
bool f_rows_ok(const orn_linear* L);
int f_rows(orn_ctx* ctx, cudaStream_t s, const orn_linear* const* Ls, bf16_t* const* ys, int n, const bf16_t* xs, int rows,
           const int* seg = nullptr /*rows sorted by expert: device [E + 1]*/, const uint32_t* row_map = nullptr);
