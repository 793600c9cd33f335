// Weight units of the row-invariant mat-vec, with packed pairs of multiply-adds, and the butterfly that ends a row:
// shared by the fused decode kernels (fused.cu) and the product of many rows (rows.cu).
#pragma once

#include "../../include/ornith_cuda.h"
#include "orn_quant.cuh"

namespace {

// P: pieces of four activations in a unit, WPU: weights of a unit, NS: sums of activations the fold takes
template <int KIND> struct Lay;
template <> struct Lay<ORN_A8>   { static constexpr int P = 4, WPU = 16, NS = 1; };
template <> struct Lay<ORN_Q4K>  { static constexpr int P = 8, WPU = 32, NS = 2; };
template <> struct Lay<ORN_Q6K>  { static constexpr int P = 4, WPU = 16, NS = 0; };
template <> struct Lay<ORN_BF16> { static constexpr int P = 2, WPU = 8,  NS = 0; };


// ---------------------------------------------------------------------------
// weight units (the arithmetic of linear.cu's Fmt<>, activations from registers)
// ---------------------------------------------------------------------------
template <int KIND> struct WU;

template <> struct WU<ORN_A8> {
  struct W { uint4 q; uint32_t sb; };
  // unit u of a row record staged in shared memory: [codes K][{scale, bias} K/64]
  ORN_D static void lds(const uint8_t* rec, uint32_t off1, uint32_t, int u, W& w) {
    w.q = *reinterpret_cast<const uint4*>(rec + 16 * u);
    w.sb = *reinterpret_cast<const uint32_t*>(rec + off1 + 4 * (u >> 2));
  }
  ORN_D static float fold(const W& w, const float* x, const float* sm, int, float acc) {
    const uint32_t qw[4] = {w.q.x, w.q.y, w.q.z, w.q.w};
    const uint64_t nm = pk2(-8388608.0f, -8388608.0f);
    uint64_t s2 = pk2(0.f, 0.f);  // (even chain, odd chain)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s2 = ffma2(pk2(x[4 * k + 0], x[4 * k + 1]), byte2_f<0>(qw[k], nm), s2);
      s2 = ffma2(pk2(x[4 * k + 2], x[4 * k + 3]), byte2_f<2>(qw[k], nm), s2);
    }
    acc = fmaf(bf_lo(w.sb), pk2_sum(s2), acc);
    acc = fmaf(bf_hi(w.sb), sm[0], acc);
    return acc;
  }
};

template <> struct WU<ORN_Q4K> {
  struct W { uint4 q; uint4 meta; };
  // staged row record: [codes nb*128][headers nb*16]
  ORN_D static void lds(const uint8_t* rec, uint32_t off1, uint32_t, int u, W& w) {
    w.q = *reinterpret_cast<const uint4*>(rec + 16 * u);
    w.meta = *reinterpret_cast<const uint4*>(rec + off1 + (u >> 3) * 16);
  }
  ORN_D static float fold(const W& w, const float* x, const float* sm, int u, float acc) {
    const int g = (u & 7) >> 1;
    const uint32_t qw[4] = {w.q.x, w.q.y, w.q.z, w.q.w};
    const uint64_t nm = pk2(-8388608.0f, -8388608.0f);
    uint64_t lo2 = pk2(0.f, 0.f), hi2 = pk2(0.f, 0.f);  // (even chain, odd chain) of the two sub-blocks
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t l4 = qw[k] & 0x0F0F0F0Fu, h4 = (qw[k] >> 4) & 0x0F0F0F0Fu;
      lo2 = ffma2(pk2(x[4 * k + 0], x[4 * k + 1]), byte2_f<0>(l4, nm), lo2);
      lo2 = ffma2(pk2(x[4 * k + 2], x[4 * k + 3]), byte2_f<2>(l4, nm), lo2);
      hi2 = ffma2(pk2(x[16 + 4 * k + 0], x[16 + 4 * k + 1]), byte2_f<0>(h4, nm), hi2);
      hi2 = ffma2(pk2(x[16 + 4 * k + 2], x[16 + 4 * k + 3]), byte2_f<2>(h4, nm), hi2);
    }
    const float lo = pk2_sum(lo2), hi = pk2_sum(hi2);
    const float d = h2f((uint16_t)(w.meta.x & 0xffff)), dmin = h2f((uint16_t)(w.meta.x >> 16));
    // get_scale_min_k4 (kernels/q4k.metal:43-56) for the sub-blocks 2g and 2g+1 at once: their
    // bytes are neighbours in each of the three scale words, so both come out of 16-bit pieces
    // (j < 4: sc = q[j] & 63, m = q[j+4] & 63; else sc = (q[j+4] & 15) | (q[j-4] >> 6 << 4),
    // m = (q[j+4] >> 4) | (q[j] >> 6 << 4))
    const int sh = (g & 1) * 16;
    const uint32_t qa = (w.meta.y >> sh) & 0xffffu, qb = (w.meta.z >> sh) & 0xffffu, qc = (w.meta.w >> sh) & 0xffffu;
    const bool low = g < 2;
    const uint32_t sc2 = low ? (qa & 0x3f3fu) : ((qc & 0x0f0fu) | ((qa >> 2) & 0x3030u));
    const uint32_t mn2 = low ? (qb & 0x3f3fu) : (((qc >> 4) & 0x0f0fu) | ((qb >> 2) & 0x3030u));
    float s1, s2, m1, m2;
    {
      const uint64_t sp = byte2_f<0>(sc2, nm), mp = byte2_f<0>(mn2, nm);
      asm("mov.b64 {%0, %1}, %2;" : "=f"(s1), "=f"(s2) : "l"(sp));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(m1), "=f"(m2) : "l"(mp));
    }
    float t = s1 * lo;
    t = fmaf(s2, hi, t);
    float mt = m1 * sm[0];
    mt = fmaf(m2, sm[1], mt);
    acc = fmaf(d, t, acc);
    acc = fmaf(-dmin, mt, acc);
    return acc;
  }
};

template <> struct WU<ORN_Q6K> {
  struct W { uint32_t qa, qb, qh, sc4; float d; };
  // staged row record: [ql|qh nb*192][scales nb*16][d nb*2]
  ORN_D static void lds(const uint8_t* rec, uint32_t off1, uint32_t off2, int u, W& w) {
    const int blk = u >> 4, j = u & 15, half = j >> 3, l0 = 4 * (j & 7);
    const uint8_t* base = rec + blk * 192;
    w.qa = *reinterpret_cast<const uint32_t*>(base + 64 * half + l0);
    w.qb = *reinterpret_cast<const uint32_t*>(base + 64 * half + 32 + l0);
    w.qh = *reinterpret_cast<const uint32_t*>(base + 128 + 32 * half + l0);
    const uint2 s8 = *reinterpret_cast<const uint2*>(rec + off1 + blk * 16 + 8 * half);
    // scales sc[is + 0, 2, 4, 6] of this half: bytes is, is+2 of either word, one byte permute
    w.sc4 = __byte_perm(s8.x, s8.y, (l0 >> 4) ? 0x7531u : 0x6420u);
    w.d = h2f(*reinterpret_cast<const uint16_t*>(rec + off2 + 2 * blk));
  }
  ORN_D static float fold(const W& w, const float* x, const float*, int, float acc) {
    const uint32_t q1 = (w.qa & 0x0F0F0F0Fu) | ((w.qh & 0x03030303u) << 4);
    const uint32_t q2 = (w.qb & 0x0F0F0F0Fu) | ((w.qh & 0x0C0C0C0Cu) << 2);
    const uint32_t q3 = ((w.qa >> 4) & 0x0F0F0F0Fu) | (w.qh & 0x30303030u);
    const uint32_t q4 = ((w.qb >> 4) & 0x0F0F0F0Fu) | ((w.qh & 0xC0C0C0C0u) >> 2);
    const uint64_t nm = pk2(-8388640.0f, -8388640.0f);  // -(2^23 + 32)
    const uint64_t z = pk2(0.f, 0.f);
    uint64_t p0 = ffma2(pk2(x[0], x[1]), byte2_f<0>(q1, nm), z);
    p0 = ffma2(pk2(x[2], x[3]), byte2_f<2>(q1, nm), p0);
    uint64_t p1 = ffma2(pk2(x[4], x[5]), byte2_f<0>(q2, nm), z);
    p1 = ffma2(pk2(x[6], x[7]), byte2_f<2>(q2, nm), p1);
    uint64_t p2 = ffma2(pk2(x[8], x[9]), byte2_f<0>(q3, nm), z);
    p2 = ffma2(pk2(x[10], x[11]), byte2_f<2>(q3, nm), p2);
    uint64_t p3 = ffma2(pk2(x[12], x[13]), byte2_f<0>(q4, nm), z);
    p3 = ffma2(pk2(x[14], x[15]), byte2_f<2>(q4, nm), p3);
    const float s0 = pk2_sum(p0), s1 = pk2_sum(p1), s2 = pk2_sum(p2), s3 = pk2_sum(p3);
    // four int8 scales -> float: b ^ 0x80 is b + 128 as an unsigned byte, then the exact byte -> float form
    float c0, c1, c2, c3;
    {
      const uint32_t ub = w.sc4 ^ 0x80808080u;
      const uint64_t nb = pk2(-8388736.0f, -8388736.0f);  // -(2^23 + 128)
      const uint64_t c01 = byte2_f<0>(ub, nb), c23 = byte2_f<2>(ub, nb);
      asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(c01));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(c2), "=f"(c3) : "l"(c23));
    }
    float t = c0 * s0;
    t = fmaf(c1, s1, t);
    t = fmaf(c2, s2, t);
    t = fmaf(c3, s3, t);
    return fmaf(w.d, t, acc);
  }
};

template <> struct WU<ORN_BF16> {
  struct W { uint4 q; };
  ORN_D static void lds(const uint8_t* rec, uint32_t, uint32_t, int u, W& w) {
    w.q = *reinterpret_cast<const uint4*>(rec + 16 * u);
  }
  ORN_D static float fold(const W& w, const float* x, const float*, int, float acc) {
    float f[8];
    widen8(w.q, f);
    uint64_t s2 = pk2(0.f, 0.f);  // the unit's (even chain, odd chain); their sum joins the lane's total
#pragma unroll
    for (int i = 0; i < 8; i += 2) s2 = ffma2(pk2(x[i], x[i + 1]), pk2(f[i], f[i + 1]), s2);
    return acc + pk2_sum(s2);
  }
};

// Butterfly over V values per lane (V a power of two <= 32) in reduce-scatter form: at the level
// with xor mask m a lane keeps half of its values and adds its partner's copies of them, so each
// value goes through exactly the additions of the plain xor-16..1 butterfly (a + b is commutative,
// both partners hold the same sum) with V-1 + (5 - log2 V) shuffles instead of 5 V.  Returns the
// lane's value; `which` is its index.  Lanes that differ only in the low 5 - log2 V bits hold copies.
template <int V>
ORN_D float rs_butterfly(float* v, int lane, int& which) {
  int idx = 0;
  int n = V;
#pragma unroll
  for (int mask = 16; mask >= 1; mask >>= 1) {
    if (n > 1) {
      const int h = n >> 1;
      const bool upper = (lane & mask) != 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (i < h) {
          const float send = upper ? v[i] : v[i + h];
          const float keep = upper ? v[i + h] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
        }
      }
      idx = idx * 2 + (upper ? 1 : 0);
      n = h;
    } else {
      v[0] = v[0] + __shfl_xor_sync(0xffffffffu, v[0], mask);
    }
  }
  which = idx;
  return v[0];
}
template <>
ORN_D float rs_butterfly<1>(float* v, int, int& which) {
  which = 0;
  return warp_sum(v[0]);
}

}  // namespace
