// Reconstruction of one PLAID / ColBERTv2 token by a half-warp (16 lanes), shared by the stand-alone
// decompress kernel and by the producer warps of the tensor-core scorer so that both give the same
// bits.  Lane hl of the half-warp owns the eight consecutive features [8 hl, 8 hl + 8):
//   - one 16-byte load of the centroid row slice (fp16 / bf16; two for fp32 centroids),
//   - one load of the nbits bytes that hold the eight bucket codes (feature f sits in byte
//     f / (8/nbits) at bit (f % (8/nbits)) * nbits, little-endian inside the byte, so the eight codes
//     of a lane are eight consecutive nbits-wide fields of one little-endian word),
//   - bucket weights from a table in shared memory, fp32 add, and for the L2 norm a half-warp
//     shuffle reduction in a fixed order.
// Needs: embedding width a multiple of 8, centroid rows 16-byte aligned, residual rows nbits-byte aligned.
#pragma once

#include "lik_common.cuh"

namespace lik {

struct PlaidSrc {
  const int* codes;                // [n_tokens]
  const unsigned char* residuals;  // [n_tokens, packed_dim]
  const void* centroids;           // [n_centroids, dim]
  const float* bucket_weights;     // [1 << nbits]
  int centroid_dtype;              // LIK_F32 / LIK_F16 / LIK_BF16
  int n_centroids;
  int nbits;                       // 2, 4 or 8
  int packed_dim;                  // ceil(dim * nbits / 8)
  int dim;
  int normalize;                   // divide the reconstructed token by max(||x||, 1e-12)
};

// raw loads of one token slice: issued for several tokens before any of them is used
template <bool CF32>
struct PlaidRaw {
  uint4 c0;                 // centroid slice: eight 16-bit values, or the first four fp32 values
  unsigned long long w;     // the lane's eight bucket codes
};
template <>
struct PlaidRaw<true> {
  uint4 c0, c1;             // eight fp32 centroid values
  unsigned long long w;
};

__device__ __forceinline__ int plaid_code(const PlaidSrc& S, long long tok, int* status) {
  int c = __ldg(S.codes + tok);
  if (c < 0 || c >= S.n_centroids) {
    if (status) atomicOr(status, LIK_DEV_CODE_RANGE);
    c = 0;
  }
  return c;
}

template <bool CF32>
__device__ __forceinline__ PlaidRaw<CF32> plaid_load(const PlaidSrc& S, long long tok, int code, int hl, bool on) {
  PlaidRaw<CF32> r;
  r.c0 = make_uint4(0, 0, 0, 0);
  r.w = 0ull;
  if constexpr (CF32) r.c1 = make_uint4(0, 0, 0, 0);
  if (!on) return r;
  const long long off = (long long)code * S.dim + hl * 8;
  if constexpr (CF32) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const float*>(S.centroids) + off);
    r.c0 = __ldg(p);
    r.c1 = __ldg(p + 1);
  } else {
    r.c0 = __ldg(reinterpret_cast<const uint4*>(static_cast<const unsigned short*>(S.centroids) + off));
  }
  const unsigned char* rp = S.residuals + tok * S.packed_dim + hl * S.nbits;
  if (S.nbits == 2)
    r.w = __ldg(reinterpret_cast<const unsigned short*>(rp));
  else if (S.nbits == 4)
    r.w = __ldg(reinterpret_cast<const unsigned int*>(rp));
  else
    r.w = __ldg(reinterpret_cast<const unsigned long long*>(rp));
  return r;
}

// e[i] = centroid + bucket weight for the lane's eight features; bw points at the table in shared memory
template <bool CF32>
__device__ __forceinline__ void plaid_features(const PlaidSrc& S, const PlaidRaw<CF32>& r, const float* bw, float (&e)[8]) {
  float c[8];
  if constexpr (CF32) {
    c[0] = __uint_as_float(r.c0.x); c[1] = __uint_as_float(r.c0.y); c[2] = __uint_as_float(r.c0.z); c[3] = __uint_as_float(r.c0.w);
    c[4] = __uint_as_float(r.c1.x); c[5] = __uint_as_float(r.c1.y); c[6] = __uint_as_float(r.c1.z); c[7] = __uint_as_float(r.c1.w);
  } else if (S.centroid_dtype == LIK_BF16) {
    c[0] = __uint_as_float(r.c0.x << 16); c[1] = __uint_as_float(r.c0.x & 0xffff0000u);
    c[2] = __uint_as_float(r.c0.y << 16); c[3] = __uint_as_float(r.c0.y & 0xffff0000u);
    c[4] = __uint_as_float(r.c0.z << 16); c[5] = __uint_as_float(r.c0.z & 0xffff0000u);
    c[6] = __uint_as_float(r.c0.w << 16); c[7] = __uint_as_float(r.c0.w & 0xffff0000u);
  } else {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.c0.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.c0.y));
    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&r.c0.z)), f = __half22float2(*reinterpret_cast<const __half2*>(&r.c0.w));
    c[0] = a.x; c[1] = a.y; c[2] = b.x; c[3] = b.y; c[4] = d.x; c[5] = d.y; c[6] = f.x; c[7] = f.y;
  }
  const unsigned mask = (1u << S.nbits) - 1u;
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = c[i] + bw[(unsigned)(r.w >> (i * S.nbits)) & mask];
}

// Multiplier that normalises the token: 1 / max(||x||, 1e-12), the same on all 16 lanes of the half-warp
// (lanes whose features lie beyond the width pass zeros).  1.0f when the index is scored un-normalised.
__device__ __forceinline__ float plaid_inv_norm(const PlaidSrc& S, const float (&e)[8]) {
  if (!S.normalize) return 1.f;
  float even = 0.f, odd = 0.f;  // two chains of four
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    even = fmaf(e[i], e[i], even);
    odd = fmaf(e[i + 1], e[i + 1], odd);
  }
  float ss = even + odd;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  return inv_norm(ss, 1e-12f);
}

// A half-warp decodes the `n` consecutive tokens [tok0, tok0 + n) and hands the lane's eight finished values of
// token t (0-based) to sink(t, values).  The centroid codes are read 16 at a time (one per lane, a chunk ahead of
// their use) and passed around with shuffles; U row loads are in flight per half-warp.  Both half-warps of a warp
// must call this with the same n_uniform >= n (the shuffles are warp-wide): tokens past n are computed on zeros and
// dropped.  `lane` is the lane in the warp, `lane_on` whether the lane's features exist (8 * (lane & 15) < dim).
template <bool CF32, int U, typename Sink>
__device__ __forceinline__ void plaid_decode_range(const PlaidSrc& S, const float* bw, long long tok0, int n, int n_uniform, int lane,
                                                   bool lane_on, int* status, Sink sink) {
  const int hl = lane & 15;
  int code_next = hl < n ? plaid_code(S, tok0 + hl, status) : 0;
  for (int c0 = 0; c0 < n_uniform; c0 += 16) {
    const int code_cur = code_next;
    code_next = c0 + 16 + hl < n ? plaid_code(S, tok0 + c0 + 16 + hl, status) : 0;
#pragma unroll 1
    for (int b = 0; b < 16; b += U) {
      PlaidRaw<CF32> r[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = c0 + b + u;
        const int code = __shfl_sync(0xffffffffu, code_cur, (lane & 16) | (b + u));
        r[u] = plaid_load<CF32>(S, tok0 + t, code, hl, t < n && lane_on);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = c0 + b + u;
        float e[8];
        plaid_features<CF32>(S, r[u], bw, e);
        if (!lane_on) {
#pragma unroll
          for (int i = 0; i < 8; ++i) e[i] = 0.f;
        }
        const float inv = plaid_inv_norm(S, e);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] *= inv;
        if (t < n && lane_on) sink(t, e);
      }
    }
  }
}

// The same arithmetic (bit for bit) with everything that varies between indexes known at compile time, for the stand-alone
// decompress kernel.  What the form above spends its instructions on - 64-bit shifts by a run-time width per feature, a
// table look-up per feature, a square root and a division on all sixteen lanes for every token, a branch per load - goes:
// two-bit codes are looked up in pairs (a sixteen-entry table of two floats: one shared-memory bank per word, so no lookup
// conflicts), the norms of four tokens are reduced together (each lane ends with one token's sum and takes one root), and
// loads behind the run's end are clamped to its last token instead of branched around.
template <int NBITS>
struct PlaidTable {
  static constexpr int WORDS = NBITS == 2 ? 32 : (1 << NBITS);  // floats in shared memory
  // bw: the 2^NBITS weights
  static __device__ __forceinline__ void fill(float* tab, const float* bw, int tid, int nt) {
    if (NBITS == 2) {
      for (int x = tid; x < 32; x += nt) tab[x] = bw[(x & 1) ? (x >> 3) & 3 : (x >> 1) & 3];  // entry x / 2 = code | next code << 2
    } else {
      for (int x = tid; x < (1 << NBITS); x += nt) tab[x] = bw[x];
    }
  }
};

template <bool CF32, int NBITS>
struct PlaidPiece {  // one lane's part of a token as it is loaded
  uint4 c0, c1;      // centroid (c1: fp32 centroids only)
  unsigned w0, w1;   // residual codes (w1: eight-bit codes only)
};

// cen / res: the lane's bytes of centroid 0 and of the run's first token; addresses are one 32 x 32 + 64-bit multiply-add each
template <bool CF32, int NBITS>
__device__ __forceinline__ PlaidPiece<CF32, NBITS> plaid_piece(const char* cen, unsigned cen_pitch, unsigned code, const char* res, unsigned res_pitch, unsigned t) {
  PlaidPiece<CF32, NBITS> r;
  const uint4* p = reinterpret_cast<const uint4*>(cen + (unsigned long long)code * cen_pitch);
  r.c0 = __ldg(p);
  if constexpr (CF32) r.c1 = __ldg(p + 1);
  const char* rp = res + (unsigned long long)t * res_pitch;
  if constexpr (NBITS == 2) r.w0 = __ldg(reinterpret_cast<const unsigned short*>(rp));
  else if constexpr (NBITS == 4) r.w0 = __ldg(reinterpret_cast<const unsigned*>(rp));
  else {
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(rp));
    r.w0 = w.x;
    r.w1 = w.y;
  }
  return r;
}

// two-wide forms of the same IEEE operations
__device__ __forceinline__ void plaid_add2(float& a, float& b, float x, float y) {
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\tadd.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}" : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}
__device__ __forceinline__ void plaid_mul2(float& a, float& b, float m) {
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %2};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}" : "+f"(a), "+f"(b) : "f"(m));
}

template <bool CF32, bool CBF16, int NBITS>
__device__ __forceinline__ void plaid_values(const PlaidPiece<CF32, NBITS>& r, const float* tab, float (&e)[8]) {
  if constexpr (CF32) {
    e[0] = __uint_as_float(r.c0.x); e[1] = __uint_as_float(r.c0.y); e[2] = __uint_as_float(r.c0.z); e[3] = __uint_as_float(r.c0.w);
    e[4] = __uint_as_float(r.c1.x); e[5] = __uint_as_float(r.c1.y); e[6] = __uint_as_float(r.c1.z); e[7] = __uint_as_float(r.c1.w);
  } else {
    const unsigned w[4] = {r.c0.x, r.c0.y, r.c0.z, r.c0.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (CBF16) {
        e[2 * i] = __uint_as_float(w[i] << 16);
        e[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      } else {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        e[2 * i] = v.x;
        e[2 * i + 1] = v.y;
      }
    }
  }
  if constexpr (NBITS == 2) {
    const char* t = reinterpret_cast<const char*>(tab);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned at = i == 0 ? (r.w0 << 3) & 0x78u : (r.w0 >> (4 * i - 3)) & 0x78u;  // eight bytes per entry
      const float2 v = *reinterpret_cast<const float2*>(t + at);
      plaid_add2(e[2 * i], e[2 * i + 1], v.x, v.y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned c = NBITS == 4 ? (r.w0 >> (4 * i)) & 15u : ((i < 4 ? r.w0 : r.w1) >> (8 * (i & 3))) & 255u;
      e[i] += tab[c];
    }
  }
}

// `n` >= 0 consecutive tokens from tok0 for each of the two half-warps of a warp (their own tok0 and n); `last` is a token
// that may be read when a half-warp has none.  n_uniform: at least either n, a multiple of 4.
template <bool CF32, bool CBF16, int NBITS, typename Sink>
__device__ __forceinline__ void plaid_decode_run(const PlaidSrc& S, const float* tab, long long tok0, int n, long long last, int n_uniform, int lane,
                                                 bool lane_on, int* status, Sink sink) {
  constexpr int U = 4;
  const int hl = lane & 15, ll = lane_on ? hl : 0;
  const long long first = n > 0 ? tok0 : last;
  const int t_max = n > 0 ? n - 1 : 0;
  const char* cen = static_cast<const char*>(S.centroids) + ll * (CF32 ? 32 : 16);
  const char* res = reinterpret_cast<const char*>(S.residuals) + first * S.packed_dim + ll * NBITS;
  const unsigned cen_pitch = (unsigned)S.dim * (CF32 ? 4u : 2u), res_pitch = (unsigned)S.packed_dim;
  int code_next = plaid_code(S, first + min(hl, t_max), status);
  PlaidPiece<CF32, NBITS> nx[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    nx[u] = plaid_piece<CF32, NBITS>(cen, cen_pitch, __shfl_sync(0xffffffffu, code_next, (lane & 16) | u), res, res_pitch, min(u, t_max));
  for (int c0 = 0; c0 < n_uniform; c0 += 16) {
    const int code_cur = code_next;
    code_next = plaid_code(S, first + min(c0 + 16 + hl, t_max), status);
#pragma unroll
    for (int b = 0; b < 16; b += U) {
      PlaidPiece<CF32, NBITS> cur[U];
#pragma unroll
      for (int u = 0; u < U; ++u) cur[u] = nx[u];
      // the next four tokens' rows are on their way while these four are finished
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int code = b + U < 16 ? __shfl_sync(0xffffffffu, code_cur, (lane & 16) | ((b + U + u) & 15)) : __shfl_sync(0xffffffffu, code_next, (lane & 16) | u);
        nx[u] = plaid_piece<CF32, NBITS>(cen, cen_pitch, code, res, res_pitch, min(c0 + b + U + u, t_max));
      }
      float e[U][8], ss[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        plaid_values<CF32, CBF16, NBITS>(cur[u], tab, e[u]);
        float even = 0.f, odd = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          even = fmaf(e[u][i], e[u][i], even);
          odd = fmaf(e[u][i + 1], e[u][i + 1], odd);
        }
        ss[u] = lane_on ? even + odd : 0.f;
      }
      float inv[U];
      if (S.normalize) {
        // (the sums pair lanes 8, 4, 2 and 1 apart, in that order, as the one-token reduction does)
        const bool h8 = hl & 8, h4 = hl & 4;
        const float a0 = (h8 ? ss[2] : ss[0]) + __shfl_xor_sync(0xffffffffu, h8 ? ss[0] : ss[2], 8);
        const float a1 = (h8 ? ss[3] : ss[1]) + __shfl_xor_sync(0xffffffffu, h8 ? ss[1] : ss[3], 8);
        float t = (h4 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, h4 ? a0 : a1, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        const float mine = inv_norm(t, 1e-12f);  // of token 2 * (bit 3) + (bit 2)
#pragma unroll
        for (int u = 0; u < U; ++u) inv[u] = __shfl_sync(0xffffffffu, mine, (lane & 16) | ((u >> 1) << 3) | ((u & 1) << 2));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (S.normalize) {
#pragma unroll
          for (int i = 0; i < 8; i += 2) plaid_mul2(e[u][i], e[u][i + 1], inv[u]);
        }
        if (c0 + b + u < n && lane_on) sink(c0 + b + u, e[u]);
      }
    }
  }
}

// w's two 16-bit values plus a and b: the conversion and the addition in one instruction each, rounded once
template <bool BF16>
__device__ __forceinline__ void add_16(unsigned w, float& a, float& b) {
  if (BF16)
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %1, h, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(w));
  else
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.f16 %0, l, %0;\n\tadd.rn.f32.f16 %1, h, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(w));
}

// The same values for the scoring kernel that decodes (lik_fwd_plaid.cu), whose decoders are bound by issue: conversion and addition in one
// instruction.  tab: an array in shared memory as such, so that its address is part of the loads.  (The stand-alone kernel above is slower with
// this form: 25 000 documents decoded and scored for eight queries 618 -> 650 us.)
template <bool CF32, bool CBF16, int NBITS>
__device__ __forceinline__ void plaid_values_near(const PlaidPiece<CF32, NBITS>& r, const float* tab, float (&e)[8]) {
  const char* t = reinterpret_cast<const char*>(tab);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (NBITS == 2) {
      const float2 v = *reinterpret_cast<const float2*>(t + (i == 0 ? (r.w0 << 3) & 0x78u : (r.w0 >> (4 * i - 3)) & 0x78u));  // eight bytes per entry
      e[2 * i] = v.x;
      e[2 * i + 1] = v.y;
    } else {
      const unsigned w = NBITS == 4 ? r.w0 : (i < 2 ? r.w0 : r.w1);
      auto at = [&](int k) {  // four times code k of the word
        const int sh = NBITS * k - 2;
        return (sh < 0 ? w << 2 : w >> sh) & (NBITS == 4 ? 0x3cu : 0x3fcu);
      };
      const int k = NBITS == 4 ? 2 * i : 2 * (i & 1);
      e[2 * i] = *reinterpret_cast<const float*>(t + at(k));
      e[2 * i + 1] = *reinterpret_cast<const float*>(t + at(k + 1));
    }
  }
  if constexpr (CF32) {
    const unsigned w[8] = {r.c0.x, r.c0.y, r.c0.z, r.c0.w, r.c1.x, r.c1.y, r.c1.z, r.c1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] += __uint_as_float(w[i]);
  } else {
    add_16<CBF16>(r.c0.x, e[0], e[1]);
    add_16<CBF16>(r.c0.y, e[2], e[3]);
    add_16<CBF16>(r.c0.z, e[4], e[5]);
    add_16<CBF16>(r.c0.w, e[6], e[7]);
  }
}

// Two tokens of a quarter-warp, whose lane l has the features from 8 l and from 64 + 8 l on (e[2 u], e[2 u + 1] of token u), divided by
// their norms, where that is asked for: the sums are the same numbers as above.
__device__ __forceinline__ void plaid_finish2(bool normalize, float (&e)[4][8], int lane, bool on0, bool on1) {
  if (!normalize) return;
  float ss[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float even = 0.f, odd = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      even = fmaf(e[p][i], e[p][i], even);
      odd = fmaf(e[p][i + 1], e[p][i + 1], odd);
    }
    ss[p] = (p & 1 ? on1 : on0) ? even + odd : 0.f;
  }
  const float s0 = ss[0] + ss[1], s1 = ss[2] + ss[3];
  const bool h4 = lane & 4;
  float t = (h4 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, h4 ? s0 : s1, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  const float mine = inv_norm(t, 1e-12f);  // of token (bit 2)
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const float inv = __shfl_sync(0xffffffffu, mine, (lane & 24) | (u << 2));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      e[2 * u][i] *= inv;
      e[2 * u + 1][i] *= inv;
    }
  }
}

// eight fp32 values -> eight 16-bit operand values (bf16 or fp16), round to nearest even
__device__ __forceinline__ uint4 plaid_pack16(const float (&v)[8], bool f16) {
  uint4 o;
  if (f16) {
    __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    __half2 c = __floats2half2_rn(v[4], v[5]), d = __floats2half2_rn(v[6], v[7]);
    o.x = *reinterpret_cast<unsigned*>(&a); o.y = *reinterpret_cast<unsigned*>(&b);
    o.z = *reinterpret_cast<unsigned*>(&c); o.w = *reinterpret_cast<unsigned*>(&d);
  } else {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    __nv_bfloat162 c = __floats2bfloat162_rn(v[4], v[5]), d = __floats2bfloat162_rn(v[6], v[7]);
    o.x = *reinterpret_cast<unsigned*>(&a); o.y = *reinterpret_cast<unsigned*>(&b);
    o.z = *reinterpret_cast<unsigned*>(&c); o.w = *reinterpret_cast<unsigned*>(&d);
  }
  return o;
}

// the index can go through the half-warp path
inline bool plaid_row16_ok(const PlaidSrc& S) {
  const size_t ceb = S.centroid_dtype == LIK_F32 ? 4 : 2;
  return S.dim % 8 == 0 && S.dim <= 128 && ((uintptr_t)S.centroids % 16) == 0 && ((size_t)S.dim * ceb) % 16 == 0 &&
         ((uintptr_t)S.residuals % 8) == 0 && S.packed_dim == S.dim * S.nbits / 8 && (S.packed_dim % S.nbits) == 0;
}

}  // namespace lik
