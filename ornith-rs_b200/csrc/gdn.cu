// Gated-delta (linear attention) kernels: the fused front end and the fp32
// recurrent delta rule.
//
// Replaces kernels/gdn_front.metal:65-190 (conv window + depthwise causal
// conv k=4 + SiLU + q/k RMS norm and scale + beta + decay gate) and
// kernels/gated_delta.metal:36-142 (gated_delta_step_packed_btree), as
// dispatched by src/ops/gdn.rs:191-413.
//
// Recurrence layout: the state of one value head is [Dv=128][Dk=128] fp32
// (64 KB).  Value rows are independent, so the work is cut by (head, 16-row
// slice): a CTA of 64 threads holds a 16 x 128 slice entirely in registers
// (4 lanes per row, 32 consecutive state floats per lane, read and written as
// 128-bit accesses that cover whole 512-byte rows).  Every state element is
// read once and written once per token: the kernel moves exactly the
// algorithmic bytes.  The dot products use the reference's tree: eight chains
// of four fmas per lane, pairwise fold, then xor-1 and xor-2 across the four
// lanes of a row.
#include "orn_internal.h"

namespace {

ORN_D float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
ORN_D float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

struct FrontParams {
  const bf16_t* conv_state;  // [S, D]
  const bf16_t* qkv;         // [T, D]
  const bf16_t* cw;          // [D, Kc]
  const bf16_t* a_in;        // [T, Hv]
  const bf16_t* b_in;        // [T, Hv]
  const bf16_t* a_log;       // [Hv]
  const bf16_t* dt_bias;     // [Hv]
  bf16_t* conv_next;         // [S, D] or null
  bf16_t* conv_input;        // [S+T, D] or null
  bf16_t* q;                 // [T, Hk, Dh]
  bf16_t* k;                 // [T, Hk, Dh]
  bf16_t* v;                 // [T, Hv, Dh]
  bf16_t* beta;              // [T, Hv]
  float* g;                  // [T, Hv]
  int T, S, Kc, D, Dh, Hk, Hv;
  float q_scale, k_scale, eps;
  int Tb;         // > 0: the T rows are Tb-row windows of T / Tb sequences ...
  int64_t seq_stride;  // ... whose conv buffers [S + Tcap, D] lie seq_stride elements apart (qkv = rows S.. of each)
};

// one warp per (token, 128-channel head slot); lane owns 4 channels
__global__ void gdn_front_kernel(FrontParams p) {
  const int lane = threadIdx.x & 31;
  const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int t = blockIdx.y;
  const int slots = p.D / p.Dh;
  if (slot >= slots) return;
  const int c0 = slot * p.Dh + lane * 4;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const int seq = p.Tb > 0 ? t / p.Tb : 0, tl = p.Tb > 0 ? t - seq * p.Tb : t;
  const bf16_t* cs = p.conv_state + seq * p.seq_stride;
  const bf16_t* qk = p.qkv + seq * p.seq_stride;
  for (int i = 0; i < p.Kc; ++i) {
    const int j = tl + i;
    const bf16_t* src = (j < p.S) ? (cs + (int64_t)j * p.D) : (qk + (int64_t)(j - p.S) * p.D);
    uint2 xv = *reinterpret_cast<const uint2*>(src + c0);
    float xs[4] = {bf_lo(xv.x), bf_hi(xv.x), bf_lo(xv.y), bf_hi(xv.y)};
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[r] = fmaf(xs[r], bf2f(p.cw[(int64_t)(c0 + r) * p.Kc + i]), acc[r]);
  }
  float y[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) y[r] = orn_silu_bf(bfr(acc[r]));

  if (t + 1 == p.T && p.conv_next != nullptr) {
    for (int j = 0; j < p.S; ++j) {
      const int row = p.T + j;
      const bf16_t* src = (row < p.S) ? (p.conv_state + (int64_t)row * p.D)
                                      : (p.qkv + (int64_t)(row - p.S) * p.D);
      *reinterpret_cast<uint2*>(p.conv_next + (int64_t)j * p.D + c0) =
          *reinterpret_cast<const uint2*>(src + c0);
    }
  }
  if (p.conv_input != nullptr) {
    *reinterpret_cast<uint2*>(p.conv_input + (int64_t)(p.S + t) * p.D + c0) =
        *reinterpret_cast<const uint2*>(p.qkv + (int64_t)t * p.D + c0);
    if (t == 0)
      for (int j = 0; j < p.S; ++j)
        *reinterpret_cast<uint2*>(p.conv_input + (int64_t)j * p.D + c0) =
            *reinterpret_cast<const uint2*>(p.conv_state + (int64_t)j * p.D + c0);
  }

  const int key_dim = p.Hk * p.Dh;
  if (slot < 2 * p.Hk) {
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) sum = fmaf(y[r], y[r], sum);
    sum = warp_sum(sum);
    const float inv = orn_rsqrtf(sum / (float)p.Dh + p.eps);
    const bool is_q = slot < p.Hk;
    bf16_t* dst = (is_q ? p.q : p.k) + (int64_t)t * key_dim + (is_q ? c0 : c0 - key_dim);
    const float sc = is_q ? p.q_scale : p.k_scale;
#pragma unroll
    for (int r = 0; r < 4; ++r) dst[r] = f2bf(sc * bfr(y[r] * inv));
  } else {
    bf16_t* dst = p.v + (int64_t)t * (p.D - 2 * key_dim) + (c0 - 2 * key_dim);
#pragma unroll
    for (int r = 0; r < 4; ++r) dst[r] = f2bf(y[r]);
  }

  if (slot == 0) {
    for (int h = lane; h < p.Hv; h += 32) {
      const int64_t i = (int64_t)t * p.Hv + h;
      float sp = orn_softplus_bf(bfr(bf2f(p.a_in[i]) + bf2f(p.dt_bias[h])));
      float decay = orn_expf(bf2f(p.a_log[h]));
      p.g[i] = orn_expf((-decay) * sp);
      p.beta[i] = f2bf(orn_sigmoid_bf(bf2f(p.b_in[i])));
    }
  }
}

// The same front end for 4 taps and many rows: a warp owns a 128-channel slot for kFrontRun consecutive
// rows of one sequence, so the taps are read once (32 bytes a lane) and a row of qkv once instead of four
// times.  2048 rows: 92 -> 70 us (53 with the packed silu), 128 rows as 64 pairs: 13 -> 11 us.
constexpr int kFrontRun = 8;
__global__ void __launch_bounds__(128) gdn_front_run_kernel(const __grid_constant__ FrontParams p) {
  const int lane = threadIdx.x & 31;
  const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (slot >= p.D / 128) return;
  const int rows = p.Tb > 0 ? p.Tb : p.T, runs = (rows + kFrontRun - 1) / kFrontRun;  // rows and runs of a sequence
  const int seq = blockIdx.y / runs, t0 = (blockIdx.y - seq * runs) * kFrontRun, n = min(kFrontRun, rows - t0);
  const int c0 = slot * 128 + lane * 4;
  const bf16_t* cs = p.conv_state + seq * p.seq_stride;
  const bf16_t* qk = p.qkv + seq * p.seq_stride;
  auto window = [&](int j) {  // row j of the window [S cached rows | this call's rows]
    return *reinterpret_cast<const uint2*>((j < 3 ? cs + (int64_t)j * p.D : qk + (int64_t)(j - 3) * p.D) + c0);
  };
  float tap[4][4];  // [channel][tap]
  {
    const uint4 wa = ldg128(p.cw + (int64_t)c0 * 4), wb = ldg128(p.cw + (int64_t)c0 * 4 + 8);
    const uint32_t u[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      tap[r][0] = bf_lo(u[2 * r]); tap[r][1] = bf_hi(u[2 * r]); tap[r][2] = bf_lo(u[2 * r + 1]); tap[r][3] = bf_hi(u[2 * r + 1]);
    }
  }
  uint2 x[kFrontRun + 3];
#pragma unroll
  for (int j = 0; j < kFrontRun + 3; ++j) x[j] = j < n + 3 ? window(t0 + j) : make_uint2(0, 0);
  const int key_dim = p.Hk * 128;
#pragma unroll
  for (int i = 0; i < kFrontRun; ++i) {
    if (i >= n) break;
    const int64_t t = (int64_t)seq * rows + t0 + i;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float xs[4] = {bf_lo(x[i + j].x), bf_hi(x[i + j].x), bf_lo(x[i + j].y), bf_hi(x[i + j].y)};
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r] = fmaf(xs[r], tap[r][j], acc[r]);
    }
    uint2 o = make_uint2(orn_silu_bf2(bf2_pack(acc[0], acc[1])), orn_silu_bf2(bf2_pack(acc[2], acc[3])));
    bf16_t* dst;
    if (slot < 2 * p.Hk) {
      const float y[4] = {bf_lo(o.x), bf_hi(o.x), bf_lo(o.y), bf_hi(o.y)};
      float sum = 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) sum = fmaf(y[r], y[r], sum);
      sum = warp_sum(sum);
      const float inv = orn_rsqrtf(sum / 128.0f + p.eps);
      const bool is_q = slot < p.Hk;
      dst = (is_q ? p.q : p.k) + t * key_dim + (is_q ? c0 : c0 - key_dim);
      const float sc = is_q ? p.q_scale : p.k_scale;
      const uint32_t a = bf2_pack(y[0] * inv, y[1] * inv), b = bf2_pack(y[2] * inv, y[3] * inv);
      o = make_uint2(bf2_pack(sc * bf_lo(a), sc * bf_hi(a)), bf2_pack(sc * bf_lo(b), sc * bf_hi(b)));
    } else {
      dst = p.v + t * (p.D - 2 * key_dim) + (c0 - 2 * key_dim);
    }
    *reinterpret_cast<uint2*>(dst) = o;
    if (slot == 0)
      for (int h = lane; h < p.Hv; h += 32) {
        const int64_t at = t * p.Hv + h;
        const float sp = orn_softplus_bf(bfr(bf2f(p.a_in[at]) + bf2f(p.dt_bias[h])));
        const float decay = orn_expf(bf2f(p.a_log[h]));
        p.g[at] = orn_expf((-decay) * sp);
        p.beta[at] = f2bf(orn_sigmoid_bf(bf2f(p.b_in[at])));
      }
  }
  if (p.conv_next != nullptr && p.Tb == 0 && t0 + n == rows)  // the next call's cached rows: the window's last three
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(p.conv_next + (int64_t)j * p.D + c0) = window(rows + j);
}
// Runs pay off as soon as they fill the SMs (four warps each); below that one warp per row has the shorter
// chain.  The run form wants 4 taps and 16-byte rows, and keeps no copy of the conv input.
bool front_runs(const orn_ctx* ctx, const FrontParams& p, dim3* grid) {
  const int rows = p.Tb > 0 ? p.Tb : p.T, seqs = p.Tb > 0 ? p.T / p.Tb : 1, slots = p.D / 128;
  const int64_t runs = (int64_t)seqs * ((rows + kFrontRun - 1) / kFrontRun);
  *grid = dim3((slots + 3) / 4, (unsigned)runs);
  return p.Kc == 4 && p.conv_input == nullptr && p.D % 128 == 0 && rows > 1 &&
         ((reinterpret_cast<uintptr_t>(p.cw) | reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15) == 0 &&
         runs < 65536 && runs * slots >= 4 * ctx->sm_count;
}

struct DeltaParams {
  const bf16_t* q;     // [T, Hk, 128]
  const bf16_t* k;     // [T, Hk, 128]
  const bf16_t* v;     // [T, Hv, 128]
  const float* g;      // [T, Hv]
  const bf16_t* beta;  // [T, Hv]
  float* state;        // in-place mode: [Hv,128,128]
  float* snaps;        // in-place mode: [T][Hv,128,128] or null
  float* ring;         // ring mode: [nring][Hv,128,128]; in = ring[cur%nring], out_t = ring[(cur+1+t)%nring]
  const int* cur;      // ring mode selector (device)
  int nring;           // ring mode: number of state buffers
  int ring_final;      // ring mode: only the state after the last token is kept, in ring[(cur+1)%nring]
  bf16_t* y;           // [T, Hv, 128]
  int T, Hk, Hv;
  int batched;         // ring mode over sequences: blockIdx.z = sequence, a ring and a cursor per sequence, T rows each
};

constexpr int kRowsPerCta = 16;

// AHEAD: the inputs of step t + 1 are requested before step t's arithmetic.  A long window otherwise pays a
// memory round trip per token on top of the recurrence's own chain; a window of a few rows is bound by the
// states' traffic and wants the registers for more warps (AHEAD 181 registers and 10 warps per SM, the other form
// 127 and 16; 64 windows of two rows: 110 us ahead, 86 us not).
template <bool AHEAD>
__global__ void __launch_bounds__(kRowsPerCta * 4, AHEAD ? 1 : 8) gated_delta_kernel(const __grid_constant__ DeltaParams p) {
  const int hv = blockIdx.y;
  const int hk = hv / (p.Hv / p.Hk);
  const int row = blockIdx.x * kRowsPerCta + (threadIdx.x >> 2);
  const int lir = threadIdx.x & 3;  // lane in row
  const size_t ssz = (size_t)p.Hv * 128 * 128;
  const int lane = threadIdx.x & 31;
  __shared__ float4 s_stage[kRowsPerCta / 8][kStateWarp];
  float4* stage = s_stage[threadIdx.x >> 5];
  const size_t off = ((size_t)hv * 128 + blockIdx.x * kRowsPerCta + (threadIdx.x >> 5) * 8) * 128;  // this warp's rows
  const float* sin;
  int cur = 0;
  // batched: this sequence's rows, ring and cursor
  const size_t z = p.batched ? blockIdx.z : 0, row0 = z * p.T;
  float* ring = p.ring != nullptr ? p.ring + z * p.nring * ssz : nullptr;
  if (ring != nullptr) {
    cur = p.cur[z];
    sin = ring + (size_t)(cur % p.nring) * ssz + off;
  } else {
    sin = p.state + off;
  }
  float S[32];
  struct StepIn {
    uint4 kv[4], qv[4];
    float g;
    bf16_t beta, v;
  };
  auto fetch = [&](int t, StepIn& in) {
    const bf16_t* kp = p.k + ((row0 + t) * p.Hk + hk) * 128 + lir * 32;
    const bf16_t* qp = p.q + ((row0 + t) * p.Hk + hk) * 128 + lir * 32;
#pragma unroll
    for (int i = 0; i < 4; ++i) { in.kv[i] = ldg128(kp + 8 * i); in.qv[i] = ldg128(qp + 8 * i); }
    in.g = p.g[(row0 + t) * p.Hv + hv];
    in.beta = p.beta[(row0 + t) * p.Hv + hv];
    in.v = p.v[((row0 + t) * p.Hv + hv) * 128 + row];
  };
  StepIn now, nxt;
  fetch(0, now);
  request_state(sin, lane, S);
  take_state(stage, lane, S);
  for (int t = 0; t < p.T; ++t) {
    if (AHEAD && t + 1 < p.T) fetch(t + 1, nxt);
    if (!AHEAD && t > 0) fetch(t, now);
    // element e of the packed keys and queries, unpacked where it is used
    auto at = [](const uint4 (&w)[4], int e) {
      const uint4 u = w[e >> 3];
      const uint32_t x = (e & 4) ? ((e & 2) ? u.w : u.z) : ((e & 2) ? u.y : u.x);
      return (e & 1) ? bf_hi(x) : bf_lo(x);
    };
    const float gt = now.g;
    const float bt = bf2f(now.beta);
    const float vt = bf2f(now.v);
    float part[8];
#pragma unroll
    for (int pb = 0; pb < 8; ++pb) {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = pb * 4 + i;
        S[e] = S[e] * gt;
        acc = fmaf(S[e], at(now.kv, e), acc);
      }
      part[pb] = acc;
    }
    float kv = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
    kv = kv + __shfl_xor_sync(0xffffffffu, kv, 1);
    kv = kv + __shfl_xor_sync(0xffffffffu, kv, 2);
    const float delta = (vt - kv) * bt;
#pragma unroll
    for (int pb = 0; pb < 8; ++pb) {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = pb * 4 + i;
        S[e] = fmaf(at(now.kv, e), delta, S[e]);
        acc = fmaf(S[e], at(now.qv, e), acc);
      }
      part[pb] = acc;
    }
    float o = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
    o = o + __shfl_xor_sync(0xffffffffu, o, 1);
    o = o + __shfl_xor_sync(0xffffffffu, o, 2);
    if (lir == 0) p.y[((row0 + t) * p.Hv + hv) * 128 + row] = f2bf(o);

    float* sout = nullptr;
    if (ring != nullptr) {
      if (!p.ring_final) sout = ring + (size_t)((cur + 1 + t) % p.nring) * ssz + off;
      else if (t + 1 == p.T) sout = ring + (size_t)((cur + 1) % p.nring) * ssz + off;
    }
    else if (p.snaps != nullptr) sout = p.snaps + (size_t)t * ssz + off;
    else if (t + 1 == p.T) sout = p.state + off;
    if (sout != nullptr) store_state(sout, stage, lane, S);
    if (ring == nullptr && p.snaps != nullptr && t + 1 == p.T) store_state(p.state + off, stage, lane, S);
    if (AHEAD) now = nxt;
  }
}
}  // namespace

int k_gdn_front(orn_ctx* ctx, cudaStream_t s, const bf16_t* conv_state, const bf16_t* qkv,
                const bf16_t* cw, const bf16_t* a, const bf16_t* b, const bf16_t* a_log,
                const bf16_t* dt_bias, int T, int Hk, int Hv, int Dh, int Kc, float eps,
                bf16_t* conv_next, bf16_t* q, bf16_t* k, bf16_t* v, bf16_t* beta, float* g,
                bf16_t* conv_input_keep) {
  if (Dh != 128) ORN_FAIL(ctx, ORN_ERR_ARG, "gdn_front: head dim must be 128");
  if (conv_next == conv_state) ORN_FAIL(ctx, ORN_ERR_ARG, "gdn_front: conv_next must not alias conv_state");
  FrontParams p;
  p.conv_state = conv_state; p.qkv = qkv; p.cw = cw; p.a_in = a; p.b_in = b; p.a_log = a_log;
  p.dt_bias = dt_bias; p.conv_next = conv_next; p.conv_input = conv_input_keep;
  p.q = q; p.k = k; p.v = v; p.beta = beta; p.g = g;
  p.T = T; p.S = Kc - 1; p.Kc = Kc; p.D = 2 * Hk * Dh + Hv * Dh; p.Dh = Dh; p.Hk = Hk; p.Hv = Hv;
  p.Tb = 0; p.seq_stride = 0;
  // powf(dk, -0.5) and its square, cast to bfloat16 (qwen3_5.rs:506,524-525)
  float inv_scale = 1.0f / sqrtf((float)Dh);
  p.q_scale = bfr(inv_scale * inv_scale);
  p.k_scale = bfr(inv_scale);
  p.eps = eps;
  int slots = p.D / Dh;
  dim3 grid;
  if (front_runs(ctx, p, &grid)) {
    gdn_front_run_kernel<<<grid, 128, 0, s>>>(p);
    return orn_launch_check(ctx, "gdn_front");
  }
  grid = dim3((slots + 3) / 4, T);
  gdn_front_kernel<<<grid, 128, 0, s>>>(p);
  return orn_launch_check(ctx, "gdn_front");
}

static int launch_delta(orn_ctx* ctx, cudaStream_t s, DeltaParams& p, int B = 1) {
  if (p.Hv % p.Hk != 0) ORN_FAIL(ctx, ORN_ERR_ARG, "gated_delta: Hv % Hk != 0");
  dim3 grid(128 / kRowsPerCta, p.Hv, B);
  if (p.T > 8) gated_delta_kernel<true><<<grid, kRowsPerCta * 4, 0, s>>>(p);
  else gated_delta_kernel<false><<<grid, kRowsPerCta * 4, 0, s>>>(p);
  return orn_launch_check(ctx, "gated_delta");
}

int k_gated_delta(orn_ctx* ctx, cudaStream_t s, const bf16_t* q, const bf16_t* k, const bf16_t* v,
                  const float* g, const bf16_t* beta, float* state, int T, int Hk, int Hv,
                  bf16_t* y, float* snaps) {
  DeltaParams p;
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.state = state; p.snaps = snaps;
  p.ring = nullptr; p.cur = nullptr; p.nring = 1; p.ring_final = 0; p.y = y; p.T = T; p.Hk = Hk; p.Hv = Hv;
  p.batched = 0;
  return launch_delta(ctx, s, p);
}

// ring mode for the model: nring state buffers per layer, selected by a device
// counter so that accepting `keep` tokens is `cur += keep` and never a copy
int k_gated_delta_ring(orn_ctx* ctx, cudaStream_t s, const bf16_t* q, const bf16_t* k,
                       const bf16_t* v, const float* g, const bf16_t* beta, float* ring,
                       int nring, const int* cur, int final_only, int T, int Hk, int Hv,
                       bf16_t* y) {
  if (T + 1 > nring && !final_only) ORN_FAIL(ctx, ORN_ERR_ARG, "gated_delta ring mode: window wider than the ring");
  DeltaParams p;
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.state = nullptr; p.snaps = nullptr;
  p.ring = ring; p.cur = cur; p.nring = nring; p.ring_final = final_only; p.y = y; p.T = T; p.Hk = Hk; p.Hv = Hv;
  p.batched = 0;
  return launch_delta(ctx, s, p);
}

// ---- B sequences at once: rows sequence-major ([B][Tb] windows); conv buffers [B][S + Tcap, D] with the
// window's qkv rows already in place behind each sequence's S cached rows; state rings [B][nring][Hv,128,128]
// with one cursor per sequence, the state after window row t written to slot (cur + 1 + t) % nring
int k_gdn_front_batched(orn_ctx* ctx, cudaStream_t s, const bf16_t* conv, int64_t seq_stride, const bf16_t* cw,
                        const bf16_t* a, const bf16_t* b, const bf16_t* a_log, const bf16_t* dt_bias, int B, int Tb, int Hk,
                        int Hv, int Dh, int Kc, float eps, bf16_t* q, bf16_t* k, bf16_t* v, bf16_t* beta, float* g) {
  if (Dh != 128) ORN_FAIL(ctx, ORN_ERR_ARG, "gdn_front: head dim must be 128");
  FrontParams p;
  p.D = 2 * Hk * Dh + Hv * Dh;
  p.conv_state = conv; p.qkv = conv + (int64_t)(Kc - 1) * p.D; p.cw = cw; p.a_in = a; p.b_in = b; p.a_log = a_log;
  p.dt_bias = dt_bias; p.conv_next = nullptr; p.conv_input = nullptr;
  p.q = q; p.k = k; p.v = v; p.beta = beta; p.g = g;
  p.T = B * Tb; p.S = Kc - 1; p.Kc = Kc; p.Dh = Dh; p.Hk = Hk; p.Hv = Hv;
  p.Tb = Tb; p.seq_stride = seq_stride;
  const float inv_scale = 1.0f / sqrtf((float)Dh);
  p.q_scale = bfr(inv_scale * inv_scale);
  p.k_scale = bfr(inv_scale);
  p.eps = eps;
  const int slots = p.D / Dh;
  dim3 grid;
  if (front_runs(ctx, p, &grid)) {
    gdn_front_run_kernel<<<grid, 128, 0, s>>>(p);
    return orn_launch_check(ctx, "gdn_front");
  }
  grid = dim3((slots + 3) / 4, B * Tb);
  gdn_front_kernel<<<grid, 128, 0, s>>>(p);
  return orn_launch_check(ctx, "gdn_front");
}
int k_gated_delta_batched(orn_ctx* ctx, cudaStream_t s, const bf16_t* q, const bf16_t* k, const bf16_t* v, const float* g,
                          const bf16_t* beta, float* rings, int nring, const int* cur, int B, int Tb, int Hk, int Hv, bf16_t* y) {
  if (Tb + 1 > nring) ORN_FAIL(ctx, ORN_ERR_ARG, "gated_delta: window wider than the ring");
  DeltaParams p;
  p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.state = nullptr; p.snaps = nullptr;
  p.ring = rings; p.cur = cur; p.nring = nring; p.ring_final = 0; p.y = y; p.T = Tb; p.Hk = Hk; p.Hv = Hv;
  p.batched = 1;
  return launch_delta(ctx, s, p, B);
}
