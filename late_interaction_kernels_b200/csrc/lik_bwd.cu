// Argmax-driven MaxSim backward.
//
//   grad_q[row(i,s)] = sum_p g[p] * d_hat[row(j_p, t*)]          (row-owned gather)
//   grad_d[row(j,t)] = sum_{(p,s): t*(p,s) = t} g[p] * q_hat[row(i_p, s)]
//
// grad_d comes in two flavours: a destination-owned reduction (every CTA owns 32
// document tokens, compacts the winners that point at them in a fixed order and
// reduces them in registers: no atomics, one store per output row, bitwise
// reproducible) and an fp32-atomic scatter followed by a finalise pass.  The
// L2-normalise Jacobian is applied in the same kernels.
#include <mutex>

#include "lik_common.cuh"
#include "lik_prep.cuh"
#include "lik_sort.cuh"

namespace lik {

constexpr float kBwdNormEps = 1e-6f;  // the backward clamps ||x|| at 1e-6

struct BwdParams {
  SeqView q, d;  // inv_norm members hold 1/max(||x||,1e-6) when normalize
  PairMap pm;
  int dim;
  int normalize;
  const float* g;
  const int* argmax;
  int argmax_stride;
  void* grad_q;
  void* grad_d;
  float* gq32;  // atomic path accumulators
  float* gd32;
  int* status;
  // pair lists, deterministic path: the pairs grouped by query and by document (stable sorts of the pair index)
  const int* perm_q;   // [n_pairs] pair indices ordered by query, ties in list order
  const int* start_q;  // [n_q + 1] run of query i in perm_q
  const int* perm_d;   // [n_pairs] pair indices ordered by document
  const int* start_d;  // [n_d + 1]
  // grad_q with few query tokens and many documents: the documents of a query are cut into dq_split ranges, one
  // CTA each, whose fp32 partial rows [dq_split][q rows][dim] are summed in range order by a second kernel
  int dq_split;
  float* dq_partial;
};

// The scores of query i: `count` of them, numbered p0 .. p0 + count - 1 (CROSS, GROUPED: score slots; LIST:
// positions in perm_q).
__device__ __forceinline__ void query_slots(const BwdParams& P, int i, long long& p0, int& count, int& j0) {
  const PairMap& pm = P.pm;
  if (pm.pairing == LIK_PAIR_CROSS) {
    p0 = (long long)i * pm.n_d;
    count = pm.n_d;
    j0 = 0;
  } else if (pm.pairing == LIK_PAIR_GROUPED) {
    p0 = (long long)i * pm.group;
    count = pm.group;
    j0 = i * pm.group;
  } else {
    p0 = P.start_q[i];
    count = P.start_q[i + 1] - (int)p0;
    j0 = 0;
  }
}
// score slot and document of the jj-th score of a query
__device__ __forceinline__ void nth_score(const BwdParams& P, long long p0, int j0, int jj, long long& slot, int& j) {
  if (P.pm.pairing == LIK_PAIR_LIST) {
    slot = P.perm_q[p0 + jj];
    j = P.pm.pair_d[slot];
  } else {
    slot = p0 + jj;
    j = j0 + jj;
  }
}
// The scores of document j: n_qr of them; the ii-th one is score slot doc_slot(ii) of query doc_query(ii, slot).
struct DocScores {
  int n_qr, i_begin;
  long long first;  // LIST: run of the document in perm_d
};
__device__ __forceinline__ DocScores doc_scores(const BwdParams& P, int j) {
  DocScores d{0, 0, 0};
  if (P.pm.pairing == LIK_PAIR_CROSS) {
    d.n_qr = P.pm.n_q;
  } else if (P.pm.pairing == LIK_PAIR_GROUPED) {
    d.n_qr = 1;
    d.i_begin = j / P.pm.group;
  } else {
    d.first = P.start_d[j];
    d.n_qr = P.start_d[j + 1] - (int)d.first;
  }
  return d;
}
__device__ __forceinline__ long long doc_slot(const BwdParams& P, const DocScores& d, int j, int ii) {
  if (P.pm.pairing == LIK_PAIR_CROSS) return (long long)(d.i_begin + ii) * P.pm.n_d + j;
  if (P.pm.pairing == LIK_PAIR_GROUPED) return j;
  return __ldg(P.perm_d + d.first + ii);
}
__device__ __forceinline__ int doc_query(const BwdParams& P, const DocScores& d, int ii, long long slot) {
  return P.pm.pairing == LIK_PAIR_LIST ? __ldg(P.pm.pair_q + slot) : d.i_begin + ii;
}

template <typename G>
__device__ __forceinline__ void store_row(G* out, long long row, int dim, int lane, const float* acc, int cmax) {
  for (int c = 0; c < cmax; ++c) {
    int k = c * 32 + lane;
    if (k < dim) out[row * dim + k] = from_f32<G>(acc[c]);
  }
}

// ---------------------------------------------------------------------------------
// grad_q, row-owned.  grid = (n_q, ceil(max_lq / 8)), 8 warps, warp = query token.
// ---------------------------------------------------------------------------------
template <typename T, typename G, int CMAX>
__global__ void __launch_bounds__(256) bwd_dq_kernel(BwdParams P) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x;
  const int s = blockIdx.y * 8 + warp;
  long long qrow0;
  int qlen;
  seq_bounds(P.q, i, qrow0, qlen, nullptr);
  const int q_rows = P.q.cu ? qlen : P.q.max_len;  // rows this query owns in grad_q
  if (s >= q_rows) return;
  const long long qrow = qrow0 + s;
  float acc[CMAX];
#pragma unroll
  for (int c = 0; c < CMAX; ++c) acc[c] = 0.f;
  const bool active = s < qlen && s < P.argmax_stride && row_valid(P.q, qrow);
  if (active) {
    long long p0;
    int count, j0;
    query_slots(P, i, p0, count, j0);
    const T* __restrict__ Dg = (const T*)P.d.data;
    for (int jj = 0; jj < count; ++jj) {
      long long slot;
      int j;
      nth_score(P, p0, j0, jj, slot, j);
      const int t = P.argmax[slot * P.argmax_stride + s];
      if (t < 0) continue;
      long long drow0;
      int dlen;
      seq_bounds(P.d, j, drow0, dlen, nullptr);
      if (t >= dlen) continue;
      const long long drow = drow0 + t;
      float f = P.g[slot] * row_factor(P.d, drow);
      const T* src = Dg + drow * P.d.row_stride;
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        int k = c * 32 + lane;
        if (k < P.dim) acc[c] = fmaf(f, to_f32(src[k]), acc[c]);
      }
    }
    const float qf = P.q.scale_scalar * (P.q.scale ? P.q.scale[qrow] : 1.f);
    if (P.normalize & LIK_NORM_Q) {
      // acc is the gradient w.r.t. q_hat = q * inv; pull it back through the normalisation
      const float inv = P.q.inv_norm[qrow];
      const T* qsrc = (const T*)P.q.data + qrow * P.q.row_stride;
      float qh[CMAX];
      float dot = 0.f;
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        int k = c * 32 + lane;
        qh[c] = k < P.dim ? to_f32(qsrc[k]) * inv : 0.f;
        dot = fmaf(acc[c], qh[c], dot);
      }
      dot = warp_sum(dot);
#pragma unroll
      for (int c = 0; c < CMAX; ++c) acc[c] = (acc[c] - dot * qh[c]) * inv;
    } else if (qf != 1.f) {
#pragma unroll
      for (int c = 0; c < CMAX; ++c) acc[c] *= qf;
    }
  }
  store_row((G*)P.grad_q, qrow, P.dim, lane, acc, CMAX);
}

// ---------------------------------------------------------------------------------
// grad_d, destination-owned.  grid = (n_d, ceil(max_ld / 32)); 8 warps; warp w owns
// tokens t0 + w*4 .. +3 of the tile.  Winners are streamed in (query, token) order,
// compacted into shared memory in that order, and reduced in that order.
// ---------------------------------------------------------------------------------
constexpr int DD_TOK = 32;     // document tokens per CTA
constexpr int DD_CHUNK = 2048; // winner entries scanned per pass

template <typename T, typename G, int CMAX>
__global__ void __launch_bounds__(256) bwd_dd_owned_kernel(BwdParams P) {
  __shared__ int list_row[DD_CHUNK];   // query row of a matching winner (relative to q.data)
  __shared__ float list_g[DD_CHUNK];   // its weight g[p] * q-row factor
  __shared__ unsigned char list_t[DD_CHUNK];
  __shared__ int warp_cnt[8];
  __shared__ int list_n;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j = blockIdx.x;
  const int t0 = blockIdx.y * DD_TOK;
  long long drow0;
  int dlen;
  seq_bounds(P.d, j, drow0, dlen, nullptr);
  const int d_rows = P.d.cu ? dlen : P.d.max_len;
  if (t0 >= d_rows) return;

  float acc[4][CMAX];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < CMAX; ++c) acc[r][c] = 0.f;

  // queries that score this document
  int i_begin, i_end;
  if (P.pm.pairing == LIK_PAIR_CROSS) {
    i_begin = 0;
    i_end = P.pm.n_q;
  } else {
    i_begin = j / P.pm.group;
    i_end = i_begin + 1;
  }
  const int lq = P.argmax_stride;
  const long long total = (long long)(i_end - i_begin) * lq;
  const T* __restrict__ Qg = (const T*)P.q.data;

  for (long long e0 = 0; e0 < total; e0 += DD_CHUNK) {
    // ---- ordered compaction of the entries whose winner lies in this tile ----
    int my_cnt = 0;
    int my_row[DD_CHUNK / 256];
    float my_g[DD_CHUNK / 256];
    int my_t[DD_CHUNK / 256];
    // thread tid takes entries e0 + tid*8 .. +7 so that order == thread order
#pragma unroll
    for (int u = 0; u < DD_CHUNK / 256; ++u) {
      long long e = e0 + (long long)tid * (DD_CHUNK / 256) + u;
      my_t[u] = -1;
      if (e < total) {
        int i = i_begin + (int)(e / lq);
        int s = (int)(e - (long long)(i - i_begin) * lq);
        long long p = P.pm.pairing == LIK_PAIR_CROSS ? (long long)i * P.pm.n_d + j : (long long)j;
        int t = P.argmax[p * lq + s];
        if (t >= t0 && t < t0 + DD_TOK && t < dlen) {
          long long qrow0;
          int qlen;
          seq_bounds(P.q, i, qrow0, qlen, nullptr);
          long long qrow = qrow0 + s;
          if (s < qlen && row_valid(P.q, qrow)) {
            my_t[u] = t - t0;
            my_row[u] = (int)qrow;
            my_g[u] = P.g[p] * row_factor(P.q, qrow);
            ++my_cnt;
          }
        }
      }
    }
    // block-wide exclusive scan of my_cnt (thread order)
    int incl = my_cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_cnt[warp] = incl;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += warp_cnt[w];
    if (tid == 255) list_n = base + incl;
    int pos = base + incl - my_cnt;
#pragma unroll
    for (int u = 0; u < DD_CHUNK / 256; ++u) {
      if (my_t[u] >= 0) {
        list_row[pos] = my_row[u];
        list_g[pos] = my_g[u];
        list_t[pos] = (unsigned char)my_t[u];
        ++pos;
      }
    }
    __syncthreads();
    const int n = list_n;
    // ---- ordered reduction: warp w handles tokens w*4 .. w*4+3 ----
    for (int e = 0; e < n; ++e) {
      const int tt = list_t[e];
      if ((tt >> 2) != warp) continue;
      const int r = tt & 3;
      const float f = list_g[e];
      const T* src = Qg + (long long)list_row[e] * P.q.row_stride;
      float v[CMAX];
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        int k = c * 32 + lane;
        v[c] = k < P.dim ? to_f32(src[k]) : 0.f;
      }
#pragma unroll
      for (int rr = 0; rr < 4; ++rr)
        if (rr == r) {
#pragma unroll
          for (int c = 0; c < CMAX; ++c) acc[rr][c] = fmaf(f, v[c], acc[rr][c]);
        }
    }
    __syncthreads();
  }

  // ---- Jacobian + store ----
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int t = t0 + warp * 4 + r;
    if (t >= d_rows) continue;
    const long long drow = drow0 + t;
    const float df = P.d.scale_scalar * (P.d.scale ? P.d.scale[drow] : 1.f);
    if (P.normalize & LIK_NORM_D) {
      const float inv = P.d.inv_norm[drow];
      const T* dsrc = (const T*)P.d.data + drow * P.d.row_stride;
      float dh[CMAX];
      float dot = 0.f;
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        int k = c * 32 + lane;
        dh[c] = k < P.dim ? to_f32(dsrc[k]) * inv : 0.f;
        dot = fmaf(acc[r][c], dh[c], dot);
      }
      dot = warp_sum(dot);
#pragma unroll
      for (int c = 0; c < CMAX; ++c) acc[r][c] = (acc[r][c] - dot * dh[c]) * inv;
    } else if (df != 1.f) {
#pragma unroll
      for (int c = 0; c < CMAX; ++c) acc[r][c] *= df;
    }
    store_row((G*)P.grad_d, drow, P.dim, lane, acc[r], CMAX);
  }
}


// =================================================================================
// Fast paths (embedding width a multiple of 4, at most 256): every lane moves 4
// consecutive elements per 128-column chunk with one vector load.
// =================================================================================
template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
  float4 x = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
template <>
__device__ __forceinline__ void load4<__half>(const __half* p, float (&v)[4]) {
  uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
  float2 a = __half22float2(*reinterpret_cast<__half2*>(&x.x)), b = __half22float2(*reinterpret_cast<__half2*>(&x.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
  uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
  v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u);
  v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
}
// Four elements as they sit in memory (two 32-bit words for 16-bit types): gather loops keep several
// of these in flight and unpack only when they multiply, which halves the registers a load in flight costs.
template <typename T>
struct Raw4 {
  uint2 x;
};
template <>
struct Raw4<float> {
  float4 x;
};
template <typename T>
__device__ __forceinline__ Raw4<T> load4_raw(const T* p) {
  Raw4<T> r;
  r.x = __ldg(reinterpret_cast<const decltype(r.x)*>(p));
  return r;
}
template <typename T>
__device__ __forceinline__ Raw4<T> zero4_raw() {
  Raw4<T> r;
  r.x = decltype(r.x){};
  return r;
}
__device__ __forceinline__ void unpack4(const Raw4<float>& r, float (&v)[4]) {
  v[0] = r.x.x; v[1] = r.x.y; v[2] = r.x.z; v[3] = r.x.w;
}
__device__ __forceinline__ void unpack4(const Raw4<__half>& r, float (&v)[4]) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.x.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void unpack4(const Raw4<__nv_bfloat16>& r, float (&v)[4]) {
  v[0] = __uint_as_float(r.x.x << 16); v[1] = __uint_as_float(r.x.x & 0xffff0000u);
  v[2] = __uint_as_float(r.x.y << 16); v[3] = __uint_as_float(r.x.y & 0xffff0000u);
}
template <typename T>
__device__ __forceinline__ void fma4_raw(float (&acc)[4], float w, const Raw4<T>& r) {
  float v[4];
  unpack4(r, v);
#pragma unroll
  for (int x = 0; x < 4; ++x) acc[x] = fmaf(w, v[x], acc[x]);
}

template <typename G>
__device__ __forceinline__ void store4(G* p, const float (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store4<__half>(__half* p, const float (&v)[4]) {
  __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  uint2 x;
  x.x = *reinterpret_cast<unsigned*>(&a);
  x.y = *reinterpret_cast<unsigned*>(&b);
  *reinterpret_cast<uint2*>(p) = x;
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[4]) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  uint2 x;
  x.x = *reinterpret_cast<unsigned*>(&a);
  x.y = *reinterpret_cast<unsigned*>(&b);
  *reinterpret_cast<uint2*>(p) = x;
}

// Pull a gradient w.r.t. x_hat = x * inv back to x:  (g - <g, x_hat> x_hat) * inv.   acc is [CH][4] per lane.
template <typename T, int CH>
__device__ __forceinline__ void normalize_jacobian_row(float (&acc)[CH][4], const T* src, float inv, int dim, int lane) {
  float xh[CH][4];
  float dot = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int k = c * 128 + lane * 4;
    if (k < dim) {
      load4<T>(src + k, xh[c]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        xh[c][e] *= inv;
        dot = fmaf(acc[c][e], xh[c][e], dot);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) xh[c][e] = 0.f;
    }
  }
  dot = warp_sum(dot);
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c][e] = (acc[c][e] - dot * xh[c][e]) * inv;
}

// ---------------------------------------------------------------------------------
// grad_q fast: grid = (n_q, ceil(rows / 8)); warp = query token.  The winners and
// upstream gradients of 32 documents at a time are staged through shared memory
// (coalesced), then every warp gathers its 32 winning rows with independent loads.
// ---------------------------------------------------------------------------------
constexpr int DQ_JC = 32;
#ifndef LIK_DQ_UNROLL
#define LIK_DQ_UNROLL 8
#endif
constexpr int DQ_UNROLL = LIK_DQ_UNROLL;  // row loads in flight per warp of the grad_Q gather
static_assert(DQ_JC % DQ_UNROLL == 0, "the chunk is walked in whole groups");

template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dq_fast_kernel(BwdParams P) {
  // per (document of the chunk, query token of the CTA): winning document row (-1: none) and the weight
  // g * row factor, prepared once by the whole CTA so that the gather loop is load + fma only
  __shared__ int2 s_e[DQ_JC][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = blockIdx.x;
  const int s0 = blockIdx.y * 8;
  const int s = s0 + warp;
  long long qrow0;
  int qlen;
  seq_bounds(P.q, i, qrow0, qlen, nullptr);
  const int q_rows = P.q.cu ? qlen : P.q.max_len;
  if (s0 >= q_rows) return;  // whole CTA out of range
  const long long qrow = qrow0 + s;
  const bool owns = s < q_rows;
  const bool active = owns && s < qlen && s < P.argmax_stride && row_valid(P.q, qrow);
  float acc[CH][4];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c][e] = 0.f;
  long long p0;
  int count, j0;
  query_slots(P, i, p0, count, j0);
  const int lq = P.argmax_stride;
  const long long pitch = P.d.row_stride;
  const T* __restrict__ Dlane = (const T*)P.d.data + lane * 4;
  bool lane_on[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) lane_on[c] = c * 128 + lane * 4 < P.dim;
  const bool d_factor = P.d.inv_norm || P.d.scale || P.d.scale_scalar != 1.f;
  for (int jb = 0; jb < count; jb += DQ_JC) {
    __syncthreads();
    {
      // thread (jj, r): winner of document jb + jj for query token s0 + r
      const int jj = tid >> 3, r = tid & 7;
      int2 e = make_int2(-1, 0);
      if (jb + jj < count && s0 + r < lq) {
        long long slot;
        int j;
        nth_score(P, p0, j0, jb + jj, slot, j);
        const int t = P.argmax[slot * lq + s0 + r];
        if (t >= 0) {
          long long r0;
          int dl;
          seq_bounds(P.d, j, r0, dl, nullptr);
          const long long drow = r0 + t;
          if (t < dl && drow < P.d.n_rows) {  // a saved winner outside its document contributes nothing
            float f = P.g[slot];
            if (d_factor) f *= row_factor(P.d, drow);
            e = make_int2((int)drow, __float_as_int(f));
          }
        }
      }
      s_e[jj][r] = e;
    }
    __syncthreads();
    if (active) {
      // DQ_UNROLL winners at a time: all their row loads are issued before the first one is used (an
      // entry without a winner loads nothing and multiplies zeros)
#pragma unroll 1
      for (int j0g = 0; j0g < DQ_JC; j0g += DQ_UNROLL) {
        int2 e[DQ_UNROLL];
#pragma unroll
        for (int u = 0; u < DQ_UNROLL; ++u) e[u] = s_e[j0g + u][warp];
        Raw4<T> v[DQ_UNROLL][CH];
#pragma unroll
        for (int u = 0; u < DQ_UNROLL; ++u) {
          const bool on = e[u].x >= 0;
          const T* src = Dlane + (on ? e[u].x : 0) * pitch;
#pragma unroll
          for (int c = 0; c < CH; ++c) v[u][c] = (on && lane_on[c]) ? load4_raw<T>(src + c * 128) : zero4_raw<T>();
        }
#pragma unroll
        for (int u = 0; u < DQ_UNROLL; ++u) {
          const float f = e[u].x >= 0 ? __int_as_float(e[u].y) : 0.f;
#pragma unroll
          for (int c = 0; c < CH; ++c) fma4_raw<T>(acc[c], f, v[u][c]);
        }
      }
    }
  }
  if (!owns) return;
  if (active) {
    if (P.normalize & LIK_NORM_Q) {
      normalize_jacobian_row<T, CH>(acc, (const T*)P.q.data + qrow * P.q.row_stride, P.q.inv_norm[qrow], P.dim, lane);
    } else {
      const float qf = P.q.scale_scalar * (P.q.scale ? P.q.scale[qrow] : 1.f);
      if (qf != 1.f) {
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[c][e] *= qf;
      }
    }
  }
  G* out = (G*)P.grad_q + qrow * P.dim;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int k = c * 128 + lane * 4;
    if (k < P.dim) store4<G>(out + k, acc[c]);
  }
}


// =================================================================================
// 16-byte gathers.  A row of the operand matrix is covered by 16 lanes that each move 16 bytes per
// 256-byte chunk, so one warp-wide load instruction fetches two different rows (one per half-warp):
// half the load instructions per gathered byte of the 8-byte version above, and twice the bytes in
// flight per instruction slot.  Every half-warp owns one output row from start to finish, so nothing
// is combined across lanes except the normalisation dot product.
// Needs 16-byte-aligned rows and a width that is a multiple of 16 bytes.
// =================================================================================
template <typename T>
struct Vec16 {
  static constexpr int N = 16 / (int)sizeof(T);  // elements per 16-byte load
};

// volatile: the loads of a round keep their program order, i.e. all of them are issued before the
// first multiply-add that consumes one (the compiler otherwise interleaves them to save registers,
// which serialises the round trips to L2)
template <typename T>
__device__ __forceinline__ uint4 load16_raw(const T* p) {
  uint4 r;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ void unpack16(const uint4& r, float (&v)[4], const float*) {
  v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void unpack16(const uint4& r, float (&v)[8], const __nv_bfloat16*) {
  v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
  v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
  v[4] = __uint_as_float(r.z << 16); v[5] = __uint_as_float(r.z & 0xffff0000u);
  v[6] = __uint_as_float(r.w << 16); v[7] = __uint_as_float(r.w & 0xffff0000u);
}
__device__ __forceinline__ void unpack16(const uint4& r, float (&v)[8], const __half*) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
  const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&r.z)), d = __half22float2(*reinterpret_cast<const __half2*>(&r.w));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
template <typename T>
__device__ __forceinline__ void fma16_raw(float (&acc)[Vec16<T>::N], float w, const uint4& r) {
  float v[Vec16<T>::N];
  unpack16(r, v, (const T*)nullptr);
#pragma unroll
  for (int x = 0; x < Vec16<T>::N; ++x) acc[x] = fmaf(w, v[x], acc[x]);
}
// bf16 rows: two features per 32-bit word, folded in with one two-wide FMA per word (fma.rn.f32x2: the same IEEE
// operation per element as fmaf, half the FMA instructions)
template <>
__device__ __forceinline__ void fma16_raw<__nv_bfloat16>(float (&acc)[8], float w, const uint4& r) {
  unsigned long long ww;
  asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w));
  const unsigned x[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned long long v, a;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(x[i] << 16), "r"(x[i] & 0xffff0000u));
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(acc[2 * i]), "f"(acc[2 * i + 1]));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(ww), "l"(v));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[2 * i]), "=f"(acc[2 * i + 1]) : "l"(a));
  }
}
// (names its own half alone: the other may be in another row, in a branch without a sum, or done)
__device__ __forceinline__ float half_warp_sum(float v) {
  const unsigned half = 0xffffu << (threadIdx.x & 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(half, v, o);
  return v;
}
// element offset of chunk c for lane hl of the half-warp
template <typename T>
__device__ __forceinline__ int elt16(int c, int hl) {
  return (c * 16 + hl) * Vec16<T>::N;
}

// (g - <g, x_hat> x_hat) * inv for a row held by one half-warp
template <typename T, int CH>
__device__ __forceinline__ void normalize_jacobian_row16(float (&acc)[CH][Vec16<T>::N], const T* src, float inv, int dim, int hl) {
  constexpr int N = Vec16<T>::N;
  float xh[CH][N];
  float dot = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int k = elt16<T>(c, hl);
    if (k < dim) {
      unpack16(load16_raw<T>(src + k), xh[c], (const T*)nullptr);
#pragma unroll
      for (int e = 0; e < N; ++e) {
        xh[c][e] *= inv;
        dot = fmaf(acc[c][e], xh[c][e], dot);
      }
    } else {
#pragma unroll
      for (int e = 0; e < N; ++e) xh[c][e] = 0.f;
    }
  }
  dot = half_warp_sum(dot);
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < N; ++e) acc[c][e] = (acc[c][e] - dot * xh[c][e]) * inv;
}

template <typename T, typename G, int CH>
__device__ __forceinline__ void store_row16(G* out, const float (&acc)[CH][Vec16<T>::N], int dim, int hl) {
  constexpr int N = Vec16<T>::N;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int k = elt16<T>(c, hl);
    if (k < dim) {
#pragma unroll
      for (int q = 0; q < N; q += 4) {
        const float v[4] = {acc[c][q], acc[c][q + 1], acc[c][q + 2], acc[c][q + 3]};
        store4<G>(out + k + q, v);
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// grad_q, 16-byte gathers: grid = (n_q, ceil(rows / 16)); half-warp = query token.  The winners and
// weights of 32 documents at a time are staged through shared memory by the whole CTA.
// ---------------------------------------------------------------------------------
constexpr int DQ16_TOK = 16;  // query tokens per CTA (one per half-warp)

// What a grad_q row still needs once its sum over the documents is complete: the normalise Jacobian or the query's
// dequantisation factor, then the store.
template <typename T, typename G, int CH>
__device__ __forceinline__ void dq16_finish_row(const BwdParams& P, float (&acc)[CH][Vec16<T>::N], long long qrow, bool active, int hl) {
  constexpr int N = Vec16<T>::N;
  if (active) {
    if (P.normalize & LIK_NORM_Q) {
      normalize_jacobian_row16<T, CH>(acc, (const T*)P.q.data + qrow * P.q.row_stride, P.q.inv_norm[qrow], P.dim, hl);
    } else {
      const float qf = P.q.scale_scalar * (P.q.scale ? P.q.scale[qrow] : 1.f);
      if (qf != 1.f) {
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
          for (int e = 0; e < N; ++e) acc[c][e] *= qf;
      }
    }
  }
  store_row16<T, G, CH>((G*)P.grad_q + qrow * P.dim, acc, P.dim, hl);
}

// One block of 16 * TOK threads: query tokens [s0, s0 + TOK) of query i, document range z.
// AHEAD: winners and weights of a batch of documents are fetched while the rows of the batch before are gathered.  For launches whose
// blocks have few others beside them (packed 128 x 128 step, backward 71 -> 66 us); with many, the loads only stand in the way of the
// gathers' (512 x 512 step 843 -> 860 us).
template <typename T, typename G, int CH, int TOK, bool AHEAD = false>
__device__ __forceinline__ void dq16_block(const BwdParams& P, int i, int s0, int z, int2 (*s_e)[TOK]) {
  constexpr int N = Vec16<T>::N;
  constexpr int U = 8 / CH;  // rows in flight per half-warp
  const int tid = threadIdx.x, hl = tid & 15, hw = tid >> 4;
  const int s = s0 + hw;
  long long qrow0;
  int qlen;
  seq_bounds(P.q, i, qrow0, qlen, nullptr);
  const int q_rows = P.q.cu ? qlen : P.q.max_len;
  if (s0 >= q_rows) return;  // whole CTA out of range
  const long long qrow = qrow0 + s;
  const bool owns = s < q_rows;
  const bool active = owns && s < qlen && s < P.argmax_stride && row_valid(P.q, qrow);
  float acc[CH][N];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < N; ++e) acc[c][e] = 0.f;
  long long p0;
  int count, j0;
  query_slots(P, i, p0, count, j0);
  const int lq = P.argmax_stride;
  const long long pitch = P.d.row_stride;
  const T* __restrict__ Dlane = (const T*)P.d.data + hl * N;
  bool lane_on[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) lane_on[c] = elt16<T>(c, hl) < P.dim;
  const bool d_factor = P.d.inv_norm || P.d.scale || P.d.scale_scalar != 1.f;
  // this CTA's range of the query's documents (all of them unless the documents are split over blocks)
  int jb_lo = 0, jb_hi = count;
  if (P.dq_split > 1) {
    const int chunk = ((count + DQ_JC - 1) / DQ_JC + P.dq_split - 1) / P.dq_split * DQ_JC;
    jb_lo = min(count, z * chunk);
    jb_hi = min(count, jb_lo + chunk);
  }
  // entry (jj, r) of a batch: winner of document jb + jj for query token s0 + r
  constexpr int PER = AHEAD ? DQ_JC / 16 : 1;  // entries per thread
  int win[PER];
  float wgt[PER];
  auto fetch = [&](int jb) {
#pragma unroll
    for (int y = 0; y < PER; ++y) {
      const int x = tid + y * 16 * TOK, jj = x / TOK, r = x % TOK;
      win[y] = -1;
      wgt[y] = 0.f;
      if (jb + jj < jb_hi && s0 + r < lq) {
        long long slot;
        int j;
        nth_score(P, p0, j0, jb + jj, slot, j);
        win[y] = P.argmax[slot * lq + s0 + r];
        wgt[y] = P.g[slot];
      }
    }
  };
  if (AHEAD) fetch(jb_lo);
  for (int jb = jb_lo; jb < jb_hi; jb += DQ_JC) {
    __syncthreads();
    if constexpr (AHEAD) {
#pragma unroll
      for (int y = 0; y < PER; ++y) {
        const int x = tid + y * 16 * TOK, jj = x / TOK, r = x % TOK, t = win[y];
        int2 e = make_int2(-1, 0);
        if (t >= 0) {
          long long slot, r0;
          int j, dl;
          nth_score(P, p0, j0, jb + jj, slot, j);
          seq_bounds(P.d, j, r0, dl, nullptr);
          const long long drow = r0 + t;
          if (t < dl && drow < P.d.n_rows) {  // a saved winner outside its document contributes nothing
            float f = wgt[y];
            if (d_factor) f *= row_factor(P.d, drow);
            e = make_int2((int)drow, __float_as_int(f));
          }
        }
        s_e[jj][r] = e;
      }
      if (jb + DQ_JC < jb_hi) fetch(jb + DQ_JC);
    } else {
#pragma unroll
      for (int x = tid; x < DQ_JC * TOK; x += 16 * TOK) {
        // entry (jj, r): winner of document jb + jj for query token s0 + r
        const int jj = x / TOK, r = x % TOK;
        int2 e = make_int2(-1, 0);
        if (jb + jj < jb_hi && s0 + r < lq) {
          long long slot;
          int j;
          nth_score(P, p0, j0, jb + jj, slot, j);
          const int t = P.argmax[slot * lq + s0 + r];
          if (t >= 0) {
            long long r0;
            int dl;
            seq_bounds(P.d, j, r0, dl, nullptr);
            const long long drow = r0 + t;
            if (t < dl && drow < P.d.n_rows) {  // a saved winner outside its document contributes nothing
              float f = P.g[slot];
              if (d_factor) f *= row_factor(P.d, drow);
              e = make_int2((int)drow, __float_as_int(f));
            }
          }
        }
        s_e[jj][r] = e;
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll 1
      for (int j0g = 0; j0g < DQ_JC; j0g += U) {
        int2 e[U];
#pragma unroll
        for (int u = 0; u < U; ++u) e[u] = s_e[j0g + u][hw];
        uint4 v[U][CH];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool on = e[u].x >= 0;
          const T* src = Dlane + (on ? e[u].x : 0) * pitch;
#pragma unroll
          for (int c = 0; c < CH; ++c) v[u][c] = (on && lane_on[c]) ? load16_raw<T>(src + c * 16 * N) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float f = e[u].x >= 0 ? __int_as_float(e[u].y) : 0.f;
#pragma unroll
          for (int c = 0; c < CH; ++c) fma16_raw<T>(acc[c], f, v[u][c]);
        }
      }
    }
  }
  if (!owns) return;
  if (P.dq_split > 1) {  // the partial sum of this range; bwd_dq16_sum_kernel finishes the row
    store_row16<T, float, CH>(P.dq_partial + ((long long)z * P.q.n_rows + qrow) * P.dim, acc, P.dim, hl);
    return;
  }
  dq16_finish_row<T, G, CH>(P, acc, qrow, active, hl);
}

template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dq16_kernel(BwdParams P) {
  __shared__ int2 s_e[DQ_JC][DQ16_TOK];
  dq16_block<T, G, CH, DQ16_TOK>(P, blockIdx.x, blockIdx.y * DQ16_TOK, blockIdx.z, s_e);
}

// Second half of the split grad_q: the partial rows of the document ranges, summed in range order.
template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dq16_sum_kernel(BwdParams P) {
  constexpr int N = Vec16<T>::N;
  const int tid = threadIdx.x, hl = tid & 15, hw = tid >> 4;
  const int i = blockIdx.x;
  const int s = blockIdx.y * DQ16_TOK + hw;
  long long qrow0;
  int qlen;
  seq_bounds(P.q, i, qrow0, qlen, nullptr);
  const int q_rows = P.q.cu ? qlen : P.q.max_len;
  if (s >= q_rows) return;
  const long long qrow = qrow0 + s;
  const bool active = s < qlen && s < P.argmax_stride && row_valid(P.q, qrow);
  float acc[CH][N];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < N; ++e) acc[c][e] = 0.f;
  for (int z = 0; z < P.dq_split; ++z) {
    const float* src = P.dq_partial + ((long long)z * P.q.n_rows + qrow) * P.dim;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int k = elt16<T>(c, hl);
      if (k < P.dim) {
#pragma unroll
        for (int q4 = 0; q4 < N; q4 += 4) {
          const float4 v = *reinterpret_cast<const float4*>(src + k + q4);
          acc[c][q4] += v.x;
          acc[c][q4 + 1] += v.y;
          acc[c][q4 + 2] += v.z;
          acc[c][q4 + 3] += v.w;
        }
      }
    }
  }
  dq16_finish_row<T, G, CH>(P, acc, qrow, active, hl);
}

// ---------------------------------------------------------------------------------
// grad_d fast, destination-owned, in two kernels.
//
// bwd_dd_sort_kernel, one CTA (16 warps) per document: a stable counting sort of the document's
// winners by token.
//   1. every warp histograms the winners of its contiguous slice of (query, token) entries;
//   2. a scan turns the histograms into write offsets (token-major, then warp, so the order inside
//      a token's list is the entry order);
//   3. the entries are placed into the document's slice of a global list as (query row, weight).
// bwd_dd_reduce_kernel, one warp per document token: reads its list (coalesced), gathers the query
// rows with independent vector loads, accumulates in list order and stores the row once.
// ---------------------------------------------------------------------------------
constexpr int DDS_WARPS = 16;  // most warps a sort CTA uses
#ifndef LIK_DD_UNROLL
#define LIK_DD_UNROLL 8
#endif
constexpr int DD_UNROLL = LIK_DD_UNROLL;  // independent list entries in flight per warp of the reduce kernel

struct DdSortOut {
  int2* pairs;            // [n_scores * lq] (query row, weight bits), grouped by document then token
  long long* tok_begin;   // [d.n_rows] first list entry of every document row
  int* tok_cnt;           // [d.n_rows] list length
  int clear_rest;         // the sort also clears the counts behind a document's end (else they were cleared before)
};

// A cluster of CTAs shares one document when the documents are fewer than the SMs: each takes a slice of the entries.
struct SortCluster {
  int rank, size;
};
__device__ __forceinline__ SortCluster sort_cluster() {
  SortCluster c;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(c.rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(c.size));
  return c;
}
__device__ __forceinline__ void sort_cluster_sync(const SortCluster& c) {
  if (c.size > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else
    __syncthreads();
}
__device__ __forceinline__ int load_cluster_int(const int* p, int rank) {  // the word at p's place in the shared memory of another CTA
  unsigned a;
  int v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

// Words of shared memory beside the histograms: the offsets and block totals of the scan and, where a cluster shares the
// document, per token its count in this CTA, in the cluster and in the CTAs before this one.  (One CTA has no use for the
// latter; with them a document's limit is 10 240 tokens instead of 25 000.)
__host__ __device__ inline size_t dds_scratch_words(int ld_pad, int cluster) {
  return (size_t)ld_pad + 1 + (ld_pad + 31) / 32 + 1 + (cluster > 1 ? (size_t)3 * ld_pad : 0);
}

// Offsets of the winner sort.  In: hist[w][t] = winners of token t counted by warp w (n_hist of the CTA's n_warps warps
// count).  Out: the token's first list entry and count (global), and hist[w][t] = first write position of warp w for token
// t.  All warps work: each takes whole blocks of 32 tokens (totals, prefix inside the block), warp 0 scans the block
// totals, then every warp finishes its blocks.  The order inside a token's list is (CTA, warp, entry).  All CTAs of a
// cluster call it with the same dlen.
__device__ __forceinline__ void dds_offsets(int* hist, int* scratch, const SortCluster& cl, int n_warps, int n_hist, int ld_pad, int dlen,
                                            long long base, long long drow0, const DdSortOut& O, int warp, int lane) {
  int* tok_off = scratch;                    // [ld_pad + 1]
  int* blk = tok_off + ld_pad + 1;           // [ceil(ld_pad / 32) + 1]
  int* mine = blk + (ld_pad + 31) / 32 + 1;  // clusters: [ld_pad] this CTA's winners of a token
  int* all = mine + ld_pad;                  // [ld_pad] the cluster's
  int* before = all + ld_pad;                // [ld_pad] those of the CTAs before this one
  auto own = [&](int t) {
    int tot = 0;
    for (int w = 0; w < n_hist; ++w) tot += hist[w * ld_pad + t];
    return tot;
  };
  const bool shared = cl.size > 1;
  if (shared) {
    for (int t = warp * 32 + lane; t < dlen; t += n_warps * 32) mine[t] = own(t);
    sort_cluster_sync(cl);
  }
  const int n_blk = (dlen + 31) >> 5;
  for (int b = warp; b < n_blk; b += n_warps) {
    const int t = b * 32 + lane;
    int tot = 0;
    if (t < dlen) {
      if (shared) {
        int bef = 0;
        for (int r = 0; r < cl.size; ++r) {
          const int v = load_cluster_int(mine + t, r);
          tot += v;
          if (r < cl.rank) bef += v;
        }
        all[t] = tot;
        before[t] = bef;
      } else {
        tot = own(t);
      }
    }
    int incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (t < dlen) tok_off[t] = incl - tot;
    if (lane == 31) blk[b] = incl;
  }
  sort_cluster_sync(cl);  // (the other CTAs have read `mine` too: it may go away with this CTA)
  if (warp == 0) {
    int running = 0;
    for (int b0 = 0; b0 < n_blk; b0 += 32) {
      const int b = b0 + lane;
      const int tot = b < n_blk ? blk[b] : 0;
      int incl = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (b < n_blk) blk[b] = running + incl - tot;
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncthreads();
  for (int b = warp; b < n_blk; b += n_warps) {
    const int t = b * 32 + lane;
    if (t < dlen) {
      const int excl = blk[b] + tok_off[t];
      int pos = excl + (shared ? before[t] : 0);
      for (int w = 0; w < n_hist; ++w) {
        const int c = hist[w * ld_pad + t];
        hist[w * ld_pad + t] = pos;
        pos += c;
      }
      if (cl.rank == 0) {
        O.tok_begin[drow0 + t] = base + excl;
        O.tok_cnt[drow0 + t] = shared ? all[t] : pos - excl;
      }
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(DDS_WARPS * 32) bwd_dd_sort_kernel(BwdParams P, DdSortOut O, int ld_pad, int n_hist) {
  // n_hist warps take the entries, one histogram each (the launcher sizes that to the entries per document); the CTA may
  // have more warps than that for the work that goes with the document's length (clearing, offsets)
  const int n_warps = blockDim.x >> 5;
  extern __shared__ int dds_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SortCluster cl = sort_cluster();
  const int j = blockIdx.x / cl.size;  // (all CTAs of a cluster leave together: what decides is the document's)
  long long drow0;
  int dlen;
  seq_bounds(P.d, j, drow0, dlen, nullptr);
  if (O.clear_rest && cl.rank == 0)
    for (int t = (dlen > 0 && dlen < ld_pad ? dlen : 0) + tid; t < P.d.max_len; t += blockDim.x) O.tok_cnt[drow0 + t] = 0;
  if (dlen <= 0) return;
  if (dlen >= ld_pad) {  // max_len understated the longest document: report instead of overrunning shared memory
    if (tid == 0 && P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
    return;
  }
  const DocScores ds = doc_scores(P, j);
  const bool list = P.pm.pairing == LIK_PAIR_LIST;
  const int t_bits = 32 - __clz(ld_pad);  // winners are below ld_pad
  const int lq = P.argmax_stride;
  const int n_ent = ds.n_qr * lq;
  const long long base = list ? ds.first * lq : (long long)j * n_ent;  // first entry of the document's slice of the list
  int* hist = dds_raw;                          // [n_hist][ld_pad]
  int* scratch = hist + n_hist * ld_pad;
  float* gcol = reinterpret_cast<float*>(scratch + dds_scratch_words(ld_pad, cl.size));  // [n_qr] (not for pair lists)

  for (int x = tid; x < n_hist * ld_pad; x += blockDim.x) hist[x] = 0;
  if (!list)
    for (int x = tid; x < ds.n_qr; x += blockDim.x) gcol[x] = P.g[doc_slot(P, ds, j, x)];
  __syncthreads();

  // entry e = ii * lq + s ; slice of this warp (multiple of 32 so rounds stay aligned)
  const int n_slices = n_hist * cl.size;
  const int per_warp = ((n_ent + n_slices - 1) / n_slices + 31) & ~31;
  const int e_lo = min(n_ent, (cl.rank * n_hist + warp) * per_warp), e_hi = warp < n_hist ? min(n_ent, e_lo + per_warp) : e_lo;

  // raw saved winner of entry e (no validation): a plain load that can be issued ahead of its use
  auto raw_winner = [&](int e) -> int {
    if (e >= e_hi) return -1;
    const int ii = e / lq, s = e - ii * lq;
    return __ldg(P.argmax + doc_slot(P, ds, j, ii) * lq + s);
  };
  // validate a raw winner: -1 when the entry contributes nothing
  auto checked = [&](int e, int t, int& qrow_out, float& g_out) -> int {
    if (t < 0 || t >= dlen) return -1;
    const int ii = e / lq, s = e - ii * lq;
    const long long slot = doc_slot(P, ds, j, ii);
    long long qrow0;
    int qlen;
    seq_bounds(P.q, doc_query(P, ds, ii, slot), qrow0, qlen, nullptr);
    if (s >= qlen || !row_valid(P.q, qrow0 + s)) return -1;
    qrow_out = (int)(qrow0 + s);
    g_out = list ? P.g[slot] : gcol[ii];
    return t;
  };

  for (int e = e_lo + lane; e < e_hi; e += 128) {
    int t4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t4[u] = raw_winner(e + 32 * u);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int qr;
      float gg;
      const int t = checked(e + 32 * u, t4[u], qr, gg);
      if (t >= 0) atomicAdd(&hist[warp * ld_pad + t], 1);
    }
  }
  __syncthreads();
  // offsets: warp 0 scans the tokens; hist[w][t] becomes the first write position of warp w for token t
  dds_offsets(hist, scratch, cl, n_warps, n_hist, ld_pad, dlen, base, drow0, O, warp, lane);
  // stable placement
  int t_next = raw_winner(e_lo + lane);
  for (int eb = e_lo; eb < e_hi; eb += 32) {
    const int e = eb + lane;
    int qrow = 0;
    float gg = 0.f;
    const int t_raw = t_next;
    t_next = raw_winner(e + 32);  // in flight while this round is placed
    const int t = e < e_hi ? checked(e, t_raw, qrow, gg) : -1;
    const unsigned peers = warp_peers(t, t_bits);
    if (t >= 0) {
      const int rank = __popc(peers & ((1u << lane) - 1u));
      const int pos = hist[warp * ld_pad + t] + rank;
      O.pairs[base + pos] = make_int2(qrow, __float_as_int(gg * row_factor(P.q, qrow)));
    }
    __syncwarp();
    if (t >= 0 && (peers & ((1u << lane) - 1u)) == 0) hist[warp * ld_pad + t] += __popc(peers);
    __syncwarp();
  }
}

template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dd_reduce_kernel(BwdParams P, DdSortOut O) {
  const int lane = threadIdx.x & 31;
  const long long drow = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (drow >= P.d.n_rows) return;
  float acc[CH][4];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c][e] = 0.f;
  // both loads are issued together; tok_begin is only meaningful when the count is non-zero
  const int cnt = __ldg(O.tok_cnt + drow);
  const long long begin = __ldg(O.tok_begin + drow);
  const T* __restrict__ Qg = (const T*)P.q.data;
  if (cnt > 0) {
    // every lane reads the same list entry (one broadcast transaction), then its own slice of the query row:
    // DD_UNROLL independent entries per round, accumulated in list order
    const int2* __restrict__ list = O.pairs + begin;
    const long long pitch = P.q.row_stride;
    const T* __restrict__ Qlane = Qg + lane * 4;
    bool lane_on[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) lane_on[c] = c * 128 + lane * 4 < P.dim;
    int k = 0;
    for (; k + DD_UNROLL <= cnt; k += DD_UNROLL) {
      int2 e[DD_UNROLL];
#pragma unroll
      for (int u = 0; u < DD_UNROLL; ++u) e[u] = __ldg(list + k + u);
      Raw4<T> v[DD_UNROLL][CH];
#pragma unroll
      for (int u = 0; u < DD_UNROLL; ++u) {
        const T* src = Qlane + e[u].x * pitch;
#pragma unroll
        for (int c = 0; c < CH; ++c) v[u][c] = lane_on[c] ? load4_raw<T>(src + c * 128) : zero4_raw<T>();
      }
#pragma unroll
      for (int u = 0; u < DD_UNROLL; ++u) {
        const float w = __int_as_float(e[u].y);
#pragma unroll
        for (int c = 0; c < CH; ++c) fma4_raw<T>(acc[c], w, v[u][c]);
      }
    }
    for (; k < cnt; ++k) {
      const int2 e = __ldg(list + k);
      const float w = __int_as_float(e.y);
      const T* src = Qlane + e.x * pitch;
#pragma unroll
      for (int c = 0; c < CH; ++c)
        if (lane_on[c]) {
          float v[4];
          load4<T>(src + c * 128, v);
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[c][x] = fmaf(w, v[x], acc[c][x]);
        }
    }
  }
  if (P.normalize & LIK_NORM_D) {
    normalize_jacobian_row<T, CH>(acc, (const T*)P.d.data + drow * P.d.row_stride, P.d.inv_norm[drow], P.dim, lane);
  } else {
    const float df = P.d.scale_scalar * (P.d.scale ? P.d.scale[drow] : 1.f);
    if (df != 1.f) {
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[c][x] *= df;
    }
  }
  G* out = (G*)P.grad_d + drow * P.dim;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int kk = c * 128 + lane * 4;
    if (kk < P.dim) store4<G>(out + kk, acc[c]);
  }
}


// The same sort for argmax strides that are a multiple of four: a lane reads four consecutive winners with
// one 16-byte load and a warp keeps four such loads in flight (eight made the straight-line code twice as long for no gain), so a pass over the document's winners is a
// few round trips to L2 instead of one per 32 entries.  The order inside a token's list is (warp, round,
// load, word, lane): fixed by the data alone, hence reproducible.
constexpr int DDS_LOADS = 4;  // 16-byte loads in flight per lane

__global__ void __launch_bounds__(DDS_WARPS * 32) bwd_dd_sort4_kernel(BwdParams P, DdSortOut O, int ld_pad, int n_hist) {
  // n_hist warps take the entries, one histogram each (the launcher sizes that to the entries per document); the CTA may
  // have more warps than that for the work that goes with the document's length (clearing, offsets)
  const int n_warps = blockDim.x >> 5;
  extern __shared__ int dds_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SortCluster cl = sort_cluster();
  const int j = blockIdx.x / cl.size;  // (all CTAs of a cluster leave together: what decides is the document's)
  long long drow0;
  int dlen;
  seq_bounds(P.d, j, drow0, dlen, nullptr);
  if (O.clear_rest && cl.rank == 0)
    for (int t = (dlen > 0 && dlen < ld_pad ? dlen : 0) + tid; t < P.d.max_len; t += blockDim.x) O.tok_cnt[drow0 + t] = 0;
  if (dlen <= 0) return;
  if (dlen >= ld_pad) {  // max_len understated the longest document: report instead of overrunning shared memory
    if (tid == 0 && P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
    return;
  }
  const DocScores ds = doc_scores(P, j);
  const bool list = P.pm.pairing == LIK_PAIR_LIST;
  const int t_bits = 32 - __clz(ld_pad);  // winners are below ld_pad
  const int lq = P.argmax_stride;          // multiple of 4
  const int qpr = lq >> 2;                 // 16-byte groups per score slot
  const int n_quad = ds.n_qr * qpr;
  const int n_ent = n_quad * 4;
  const long long base = list ? ds.first * lq : (long long)j * n_ent;
  int* hist = dds_raw;                          // [n_hist][ld_pad]
  int* scratch = hist + n_hist * ld_pad;
  float* gcol = reinterpret_cast<float*>(scratch + dds_scratch_words(ld_pad, cl.size));  // [n_qr] (not for pair lists)
  int* q_first = reinterpret_cast<int*>(gcol + ds.n_qr);  // [n_qr] first row and length of every score's query (not for pair lists)
  int* q_len = q_first + ds.n_qr;

  for (int x = tid; x < n_hist * ld_pad; x += blockDim.x) hist[x] = 0;
  if (!list)
    for (int x = tid; x < ds.n_qr; x += blockDim.x) {
      const long long slot = doc_slot(P, ds, j, x);
      gcol[x] = P.g[slot];
      long long r0;
      int len;
      seq_bounds(P.q, doc_query(P, ds, x, slot), r0, len, nullptr);
      q_first[x] = (int)r0;
      q_len[x] = len;
    }
  __syncthreads();

  // slice of this warp in 16-byte groups (whole warp loads); a round is DDS_LOADS loads per lane
  const int round_quads = 32 * DDS_LOADS;
  const int n_slices = n_hist * cl.size;
  const int per_warp = ((n_quad + n_slices - 1) / n_slices + 31) & ~31;
  const int m_lo = min(n_quad, (cl.rank * n_hist + warp) * per_warp), m_hi = warp < n_hist ? min(n_quad, m_lo + per_warp) : m_lo;
  const int4 none = make_int4(-1, -1, -1, -1);

  auto load_quad = [&](int m) -> int4 {
    if (m >= m_hi) return none;
    const int ii = m / qpr, sq = m - ii * qpr;
    return __ldg(reinterpret_cast<const int4*>(P.argmax + doc_slot(P, ds, j, ii) * lq) + sq);
  };
  // first query row and length of the query of score ii (and its upstream gradient)
  auto query_of = [&](int ii, long long& qrow0, int& qlen, float& gg) {
    if (list) {
      const long long slot = doc_slot(P, ds, j, ii);
      seq_bounds(P.q, doc_query(P, ds, ii, slot), qrow0, qlen, nullptr);
      gg = P.g[slot];
    } else {
      qrow0 = q_first[ii];
      qlen = q_len[ii];
      gg = gcol[ii];
    }
  };

  // ---- pass 1: per-warp histogram of the winners per token ----
  for (int mb = m_lo; mb < m_hi; mb += round_quads) {
    int4 w[DDS_LOADS];
#pragma unroll
    for (int u = 0; u < DDS_LOADS; ++u) w[u] = load_quad(mb + u * 32 + lane);
#pragma unroll
    for (int u = 0; u < DDS_LOADS; ++u) {
      const int m = mb + u * 32 + lane;
      if (m >= m_hi) continue;
      const int ii = m / qpr, s4 = (m - ii * qpr) * 4;
      long long qrow0;
      int qlen;
      float gg;
      query_of(ii, qrow0, qlen, gg);
      // (the four winners of a load go through one copy of the code: the kernel runs once per CTA, straight through,
      // and its time is instruction fetch as much as anything)
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        const int t = k == 0 ? w[u].x : (k == 1 ? w[u].y : (k == 2 ? w[u].z : w[u].w));
        if (t >= 0 && t < dlen && s4 + k < qlen && row_valid(P.q, qrow0 + s4 + k)) atomicAdd(&hist[warp * ld_pad + t], 1);
      }
    }
  }
  __syncthreads();
  // ---- offsets: warp 0 scans the per-token totals ----
  dds_offsets(hist, scratch, cl, n_warps, n_hist, ld_pad, dlen, base, drow0, O, warp, lane);
  // ---- pass 2: placement (the winners come from L2 this time) ----
  for (int mb = m_lo; mb < m_hi; mb += round_quads) {
    int4 w[DDS_LOADS];
#pragma unroll
    for (int u = 0; u < DDS_LOADS; ++u) w[u] = load_quad(mb + u * 32 + lane);
#pragma unroll
    for (int u = 0; u < DDS_LOADS; ++u) {
      const int m = mb + u * 32 + lane;
      const bool in = m < m_hi;
      const int ii = in ? m / qpr : 0, s4 = in ? (m - ii * qpr) * 4 : 0;
      long long qrow0 = 0;
      int qlen = 0;
      float gi = 0.f;
      if (in) query_of(ii, qrow0, qlen, gi);
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        int t = k == 0 ? w[u].x : (k == 1 ? w[u].y : (k == 2 ? w[u].z : w[u].w));
        const int qrow = (int)(qrow0 + s4 + k);
        if (!(in && t >= 0 && t < dlen && s4 + k < qlen && row_valid(P.q, qrow))) t = -1;
        const unsigned peers = warp_peers(t, t_bits);
        if (t >= 0) {
          const int rank = __popc(peers & ((1u << lane) - 1u));
          const int pos = hist[warp * ld_pad + t] + rank;
          O.pairs[base + pos] = make_int2(qrow, __float_as_int(gi * row_factor(P.q, qrow)));
        }
        __syncwarp();
        if (t >= 0 && (peers & ((1u << lane) - 1u)) == 0) hist[warp * ld_pad + t] += __popc(peers);
        __syncwarp();
      }
    }
  }
}

// grad_d reduce with 16-byte gathers: one half-warp per document token, 16 tokens per CTA.
// GLOBAL: the list is in device memory (read-only loads), not in shared memory
// LONE: lists of one or two entries, nearly all of them: one by one
template <typename T, typename G, int CH, bool GLOBAL, bool LONE = false>
__device__ __forceinline__ void dd_reduce16_list(const BwdParams& P, const int2* __restrict__ list, int cnt, long long drow, int hl) {
  constexpr int N = Vec16<T>::N;
  constexpr int U = 8 / CH;
  auto entry = [&](int k) {
    if constexpr (GLOBAL) return __ldg(list + k);
    else return list[k];
  };
  float acc[CH][N];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < N; ++e) acc[c][e] = 0.f;
  if (cnt > 0) {
    const long long pitch = P.q.row_stride;
    const T* __restrict__ Qlane = (const T*)P.q.data + hl * N;
    bool lane_on[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) lane_on[c] = elt16<T>(c, hl) < P.dim;
    // `n` entries from k on, their rows in flight together (n < W: the others are left out)
    auto batch = [&](auto w_, int k, int n) {
      constexpr int W = decltype(w_)::value;
      int2 e[W];
#pragma unroll
      for (int u = 0; u < W; ++u) e[u] = entry(k + min(u, n - 1));
      uint4 v[W][CH];
#pragma unroll
      for (int u = 0; u < W; ++u) {
        const T* src = Qlane + e[u].x * pitch;
#pragma unroll
        for (int c = 0; c < CH; ++c) v[u][c] = u < n && lane_on[c] ? load16_raw<T>(src + c * 16 * N) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < W; ++u) {
        const float w = __int_as_float(e[u].y);
        if (u < n) {
#pragma unroll
          for (int c = 0; c < CH; ++c) fma16_raw<T>(acc[c], w, v[u][c]);
        }
      }
    };
    int k = 0;
    for (; k + U <= cnt; k += U) batch(std::integral_constant<int, U>{}, k, U);
    if constexpr (LONE) {
      for (; k < cnt; ++k) {
        const int2 e = entry(k);
        const float w = __int_as_float(e.y);
        const T* src = Qlane + e.x * pitch;
#pragma unroll
        for (int c = 0; c < CH; ++c)
          if (lane_on[c]) fma16_raw<T>(acc[c], w, load16_raw<T>(src + c * 16 * N));
      }
    } else {
      // The rest in one or two trips to L2 instead of one per entry: a token of a small batch has three or four entries in all.
      // (Packed 128 x 128 step, grad_D alone 50 -> 41 us.)
      if (U > 4 && k + 4 <= cnt) {
        batch(std::integral_constant<int, 4>{}, k, 4);
        k += 4;
      }
      if (k < cnt) batch(std::integral_constant<int, 3>{}, k, cnt - k);
    }
  }
  if (P.normalize & LIK_NORM_D) {
    normalize_jacobian_row16<T, CH>(acc, (const T*)P.d.data + drow * P.d.row_stride, P.d.inv_norm[drow], P.dim, hl);
  } else {
    const float df = P.d.scale_scalar * (P.d.scale ? P.d.scale[drow] : 1.f);
    if (df != 1.f) {
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int x = 0; x < N; ++x) acc[c][x] *= df;
    }
  }
  store_row16<T, G, CH>((G*)P.grad_d + drow * P.dim, acc, P.dim, hl);
}

template <typename T, typename G, int CH>
__device__ __forceinline__ void dd_reduce16_row(const BwdParams& P, const DdSortOut& O, long long drow, int hl) {
  const int cnt = __ldg(O.tok_cnt + drow);
  const long long begin = __ldg(O.tok_begin + drow);
  dd_reduce16_list<T, G, CH, true>(P, O.pairs + begin, cnt, drow, hl);
}

template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dd_reduce16_kernel(BwdParams P, DdSortOut O) {
  const int hl = threadIdx.x & 15;
  const long long drow = (long long)blockIdx.x * 16 + (threadIdx.x >> 4);
  if (drow >= P.d.n_rows) return;
  dd_reduce16_row<T, G, CH>(P, O, drow, hl);
}

// The same for very many document tokens (long documents), nearly all of them without a winner: a stream of zero rows.
// One CTA per 16 tokens costs more to schedule than to run there, so a capped grid walks the tokens, and a token without
// a winner stores its zero row without looking at anything else.
template <typename T, typename G, int CH>
__global__ void __launch_bounds__(256) bwd_dd_reduce16_walk_kernel(BwdParams P, DdSortOut O) {
  const int hl = threadIdx.x & 15;
  for (long long drow = (long long)blockIdx.x * 16 + (threadIdx.x >> 4); drow < P.d.n_rows; drow += (long long)gridDim.x * 16) {
    if (__ldg(O.tok_cnt + drow) == 0) {
      float zero[CH][Vec16<T>::N];
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int e = 0; e < Vec16<T>::N; ++e) zero[c][e] = 0.f;
      store_row16<T, G, CH>((G*)P.grad_d + drow * P.dim, zero, P.dim, hl);
    } else {
      dd_reduce16_row<T, G, CH>(P, O, drow, hl);
    }
  }
}

// ---------------------------------------------------------------------------------
// Both gradients in one launch, for problems whose documents have few winners each (small batches, candidate lists):
// the first dq_blocks blocks are grad_q blocks, the others take a document each - the counting sort of its winners stays in
// shared memory and the same block reduces and stores the document's rows (a grad_q whose documents are split into ranges
// brings its partial rows in the same launch: as a launch in front, 64 x 512 documents took 126 us, now 103).  Such problems are
// bound by launches and by the
// zero rows of grad_d, not by gathers: against sort and reduce kernels this saves two launches, the list's round trip
// and a scheduling pass over 16-row blocks.  64 x 32 candidate lists of 300 tokens: 75 -> 45 us; a 16 x 16 batch 26 -> 12 us.
// The order inside a token's list is the sort kernels': the gradients have the same bits whichever launch makes them.
// ---------------------------------------------------------------------------------
constexpr int FUSED_ENT = 4096;     // most winners of a document
constexpr int FUSED_ENT_256 = 512;  // ... of one that a block of 256 threads takes
constexpr int FUSED_SMEM = 112 * 1024;  // two blocks per SM
struct FusedShape {
  int dq_blocks, dq_per_query;  // grad_q blocks of one document range, and how many a query has
  int dq_split;                 // document ranges (0: no grad_q in this launch)
  int ld_pad, n_hist;
  int rounds, quads;            // rows of 32 entries per warp; their order (see the kernel):
  int full_rows, tail;          // ... rows in whole groups of four, and the loads of the last, partial group (256 threads)
  int parts;                    // blocks per document: each sorts all of its winners and stores every parts-th run of rows
};
inline size_t fused_smem(int n_ent, int ld_pad, int n_hist) { return (size_t)n_ent * sizeof(int2) + ((size_t)n_hist + 3) * ld_pad * 4 + 64 * 4; }

template <typename T, typename G, int CH, int NT>
__global__ void __launch_bounds__(NT) bwd_fused16_kernel(BwdParams P, FusedShape F) {
  constexpr int TOK = NT / 16;
  extern __shared__ __align__(16) unsigned char fused_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, hl = tid & 15, hw = tid >> 4;
  const int first_doc = F.dq_blocks * F.dq_split;
  if ((int)blockIdx.x < first_doc) {
    const int z = blockIdx.x / F.dq_blocks, b = blockIdx.x - z * F.dq_blocks, i = b / F.dq_per_query;
    dq16_block<T, G, CH, TOK, (NT > 256)>(P, i, (b - i * F.dq_per_query) * TOK, z, reinterpret_cast<int2(*)[TOK]>(fused_raw));
    return;
  }
  const int j = (blockIdx.x - first_doc) / F.parts, part = (blockIdx.x - first_doc) - j * F.parts;
  long long drow0;
  int dlen;
  seq_bounds(P.d, j, drow0, dlen, nullptr);
  const int d_rows = P.d.cu ? dlen : P.d.max_len;
  if (P.d.cu && part == 0 && (j == 0 || j == P.d.n_seq - 1)) {
    // packed rows that no document owns (in front of the first, behind the last)
    float zero[CH][Vec16<T>::N];
#pragma unroll
    for (int c = 0; c < CH; ++c)
#pragma unroll
      for (int e = 0; e < Vec16<T>::N; ++e) zero[c][e] = 0.f;
    const long long lo = 0, hi = j == 0 ? min((long long)P.d.cu[0], P.d.n_rows) : 0;
    for (long long r = lo + hw; r < hi; r += TOK) store_row16<T, G, CH>((G*)P.grad_d + r * P.dim, zero, P.dim, hl);
    if (j == P.d.n_seq - 1)
      for (long long r = (long long)P.d.cu[j + 1] + hw; r < P.d.n_rows; r += TOK) store_row16<T, G, CH>((G*)P.grad_d + r * P.dim, zero, P.dim, hl);
  }
  if (d_rows <= 0) return;
  const bool fits = dlen < F.ld_pad;  // (otherwise max_len understated the longest document: reported, its rows are zero)
  if (!fits && tid == 0 && P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
  const DocScores ds = doc_scores(P, j);
  const int lq = P.argmax_stride, n_ent = ds.n_qr * lq;
  int2* list = reinterpret_cast<int2*>(fused_raw);            // [n_ent] (query row, weight)
  int* hist = reinterpret_cast<int*>(list + n_ent);           // [n_hist][ld_pad]
  int* begin = hist + F.n_hist * F.ld_pad;                    // [ld_pad]
  int* cnt = begin + F.ld_pad;                                // [ld_pad]
  int* live = cnt + F.ld_pad;                                 // [ld_pad] this block's tokens with a winner
  int* wsum = live + F.ld_pad;                                // [NT / 32 + 1]
  float zero[CH][Vec16<T>::N];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int e = 0; e < Vec16<T>::N; ++e) zero[c][e] = 0.f;
  if (NT == 256 && n_ent <= 32) {
    // At most a warp's worth of winners (a candidate of a 32-token query): every warp sorts them for itself, in registers, and
    // every half-warp first clears its rows and then writes the ones that won, so that nothing is handed over and no warp
    // waits for another.  The order inside a token's list is that of the general path: the entries' order by lane.
    // (Candidate lists, backward: 128 x 32 of 64 tokens 54.7 -> 44.4 us, 64 x 32 of 300 43.2 -> 42.4, where the zeros' 157 MB are
    // what is left; 8-token queries, 128 x 32 of 64, 40.1 -> 31.4.  Looking at every token of the list in every warp instead of its
    // own ones: 43 -> 60.)
    int2* mine = list + warp * 64;  // a list for either half (the launch has room for a grad_q block's 4 KB)
    int e = lane;
    if (F.quads) {
      const int loads = max(F.tail, 1), word = lane / loads;
      e = word < 4 ? (lane - word * loads) * 4 + word : n_ent;
    }
    int t = -1, qrow = 0;
    float w = 0.f;
    if (fits && e < n_ent) {
      const int ii = e / lq, s = e - ii * lq;
      const long long slot = doc_slot(P, ds, j, ii);
      t = __ldg(P.argmax + slot * lq + s);
      long long qrow0;
      int qlen;
      seq_bounds(P.q, ds.i_begin + ii, qrow0, qlen, nullptr);
      if (t < 0 || t >= dlen || s >= qlen || !row_valid(P.q, qrow0 + s)) {
        t = -1;
      } else {
        qrow = (int)(qrow0 + s);
        w = P.g[slot] * row_factor(P.q, qrow0 + s);
      }
    }
    const int stride = TOK * F.parts, own = part * TOK + hw;
    for (int r = own; r < d_rows; r += stride) store_row16<T, G, CH>((G*)P.grad_d + (drow0 + r) * P.dim, zero, P.dim, hl);
    const unsigned peers = warp_peers(t, 32 - __clz(F.ld_pad));
    const unsigned below = (1u << lane) - 1u;
    const bool head = t >= 0 && (peers & below) == 0;
    const int to = head ? t % stride - part * TOK - warp * 2 : -1;  // 0, 1: a row of this warp's first / second half
    unsigned first = __ballot_sync(0xffffffffu, to == 0), second = __ballot_sync(0xffffffffu, to == 1);
    while (first | second) {
      const int a = first ? __ffs(first) - 1 : 0, b = second ? __ffs(second) - 1 : 0;
      const unsigned set_a = first ? __shfl_sync(0xffffffffu, peers, a) : 0u, set_b = second ? __shfl_sync(0xffffffffu, peers, b) : 0u;
      const int tok = __shfl_sync(0xffffffffu, t, lane < 16 ? a : b);
      __syncwarp();
      if ((set_a >> lane) & 1u) mine[__popc(set_a & below)] = make_int2(qrow, __float_as_int(w));
      else if ((set_b >> lane) & 1u) mine[32 + __popc(set_b & below)] = make_int2(qrow, __float_as_int(w));
      __syncwarp();
      const unsigned set = lane < 16 ? set_a : set_b;
      if (set) dd_reduce16_list<T, G, CH, false, true>(P, mine + (lane & 16) * 2, __popc(set), drow0 + tok, hl);
      first &= first - 1;
      second &= second - 1;
    }
    return;
  }
  // Mostly rows without a winner: all are cleared while the winners are on their way, and the few others, listed by the
  // scan below so that every half-warp has its share of them, are written again.
  const bool prefill = n_ent * 2 < d_rows;
  if (fits) {
    for (int x = tid; x < F.n_hist * F.ld_pad; x += NT) hist[x] = 0;
    // The winners of this thread, one of every row of its warp.  A row is 32 entries; bwd_dd_sort4_kernel reads four winners
    // at a time and places first, second, third and fourth words of 32 such loads in turn, so there four rows share 128.  (In
    // small documents the words of the last few loads follow one another without gaps; the division costs more than the empty
    // places of a row where there are many.)
    constexpr int ROUNDS = (NT == 256 ? FUSED_ENT_256 : FUSED_ENT) / NT;
    auto entry_of = [&](int k) {
      const int r = warp * F.rounds + k;
      if (!F.quads) return r * 32 + lane;
      if (NT > 256 || r < F.full_rows) return (r >> 2) * 128 + lane * 4 + (r & 3);
      const int p = (r - F.full_rows) * 32 + lane, loads = max(F.tail, 1), word = p / loads;
      return word < 4 ? F.full_rows * 32 + (p - word * loads) * 4 + word : n_ent;
    };
    int t_r[ROUNDS];
    // (where a thread has whole groups of four rows, the four words of a load are its own)
    const bool by_four = ROUNDS >= 4 && F.quads && (F.rounds & 3) == 0;
    if constexpr (ROUNDS >= 4) {
#pragma unroll
      for (int k = 0; k < ROUNDS; k += 4) {
        int4 w = make_int4(-1, -1, -1, -1);
        const int e = entry_of(k);
        if (by_four && k < F.rounds && e < n_ent) {
          const int ii = e / lq, s = e - ii * lq;
          w = __ldg(reinterpret_cast<const int4*>(P.argmax + doc_slot(P, ds, j, ii) * lq + s));
        }
        t_r[k] = w.x;
        t_r[k + 1] = w.y;
        t_r[k + 2] = w.z;
        t_r[k + 3] = w.w;
      }
    }
#pragma unroll
    for (int k = 0; k < ROUNDS; ++k) {
      if (by_four) continue;
      t_r[k] = -1;
      if (k >= F.rounds) continue;
      const int e = entry_of(k);
      if (e < n_ent) {
        const int ii = e / lq, s = e - ii * lq;
        t_r[k] = __ldg(P.argmax + doc_slot(P, ds, j, ii) * lq + s);
      }
    }
    // the query of a round's entry: its first row and length, and the weight of its score; the four words of a load share theirs, which
    // are fetched while the winners are on their way (per entry and twice before: grad_D alone 54 -> 50 us)
    struct Owner {
      int row0, len, s;  // s: the entry's token of the query (of a load's first word)
      float g;
    };
    auto owner_of = [&](int k, bool weight) {
      Owner o{0, 0, 0, 0.f};
      const int e = entry_of(k);
      if (k < F.rounds && e < n_ent) {
        const int ii = e / lq;
        o.s = e - ii * lq;
        long long r0;
        seq_bounds(P.q, ds.i_begin + ii, r0, o.len, nullptr);
        o.row0 = (int)r0;
        if (weight) o.g = P.g[doc_slot(P, ds, j, ii)];
      }
      return o;
    };
    constexpr int FOURS = ROUNDS >= 4 ? ROUNDS / 4 : 1;
    Owner owner[FOURS];
    if (by_four) {
#pragma unroll
      for (int f = 0; f < FOURS; ++f) owner[f] = owner_of(4 * f, true);
    }
    if (prefill)
      for (int t = part * TOK + hw; t < d_rows; t += TOK * F.parts) store_row16<T, G, CH>((G*)P.grad_d + (drow0 + t) * P.dim, zero, P.dim, hl);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ROUNDS; ++k) {
      if (k >= F.rounds) break;
      int t = t_r[k];
      if (t >= dlen) t = -1;
      if (t >= 0) {
        const Owner o = by_four ? owner[k / 4 < FOURS ? k / 4 : 0] : owner_of(k, false);
        const int s = o.s + (by_four ? k & 3 : 0);
        if (s >= o.len || !row_valid(P.q, (long long)o.row0 + s)) t = -1;
      }
      t_r[k] = t;
      if (t >= 0) atomicAdd(&hist[warp * F.ld_pad + t], 1);
    }
    __syncthreads();
    // offsets: a run of tokens per thread, scanned over the block
    const int per = (dlen + NT - 1) / NT;
    const int t0 = min(dlen, tid * per), t1 = min(dlen, t0 + per);
    int sum = 0;
    for (int t = t0; t < t1; ++t) {
      int c = 0;
      for (int w = 0; w < F.n_hist; ++w) c += hist[w * F.ld_pad + t];
      cnt[t] = c;
      sum += c;
      if (c && (t / TOK) % F.parts == part) sum += 1 << 16;  // (at most 4096 winners and 1536 tokens: one scan for both counts)
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int at = incl - sum;
    for (int w = 0; w < warp; ++w) at += wsum[w];
    if (tid == NT - 1) wsum[NT / 32] = (at + sum) >> 16;
    int pos = at & 0xFFFF, n_live = at >> 16;
    for (int t = t0; t < t1; ++t) {
      if (cnt[t] && (t / TOK) % F.parts == part) live[n_live++] = t;
      begin[t] = pos;
      for (int w = 0; w < F.n_hist; ++w) {
        const int c = hist[w * F.ld_pad + t];
        hist[w * F.ld_pad + t] = pos;
        pos += c;
      }
    }
    __syncthreads();
    const int t_bits = 32 - __clz(F.ld_pad);  // winners are below ld_pad
#pragma unroll
    for (int k = 0; k < ROUNDS; ++k) {
      if (k >= F.rounds) break;
      const int t = t_r[k];
      const unsigned peers = warp_peers(t, t_bits);
      if (t >= 0) {
        const Owner o = by_four ? owner[k / 4 < FOURS ? k / 4 : 0] : owner_of(k, true);
        const long long qrow = (long long)o.row0 + o.s + (by_four ? k & 3 : 0);
        const float w = o.g * row_factor(P.q, qrow);
        list[hist[warp * F.ld_pad + t] + __popc(peers & ((1u << lane) - 1u))] = make_int2((int)qrow, __float_as_int(w));
      }
      __syncwarp();
      if (t >= 0 && (peers & ((1u << lane) - 1u)) == 0) hist[warp * F.ld_pad + t] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
  }
  if (prefill && fits) {
    const int n_live = wsum[NT / 32];
    for (int u = hw; u < n_live; u += TOK) {
      const int t = live[u];
      dd_reduce16_list<T, G, CH, false>(P, list + begin[t], cnt[t], drow0 + t, hl);
    }
    return;
  }
  for (int t = part * TOK + hw; t < d_rows; t += TOK * F.parts) {
    const int c = fits && t < dlen ? cnt[t] : 0;
    if (c == 0) {
      store_row16<T, G, CH>((G*)P.grad_d + (drow0 + t) * P.dim, zero, P.dim, hl);
    } else {
      dd_reduce16_list<T, G, CH, false>(P, list + begin[t], c, drow0 + t, hl);
    }
  }
}

// ---------------------------------------------------------------------------------
// Atomic scatter: one warp per (score slot, query token).  Adds into fp32 buffers.
// WITH_DQ also scatters grad_q (pair lists, where a query's slots are not contiguous).
// ---------------------------------------------------------------------------------
template <typename T, bool WITH_DQ, bool VEC>
__global__ void __launch_bounds__(256) bwd_scatter_kernel(BwdParams P) {
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lq = P.argmax_stride;
  if (w >= P.pm.n_scores * lq) return;
  const long long p = w / lq;
  const int s = (int)(w - p * lq);
  int i, j;
  if (!decode_pair(P.pm, p, i, j, nullptr)) return;
  long long qrow0, drow0;
  int qlen, dlen;
  seq_bounds(P.q, i, qrow0, qlen, nullptr);
  if (s >= qlen) return;
  const long long qrow = qrow0 + s;
  if (!row_valid(P.q, qrow)) return;
  const int t = P.argmax[p * lq + s];
  if (t < 0) return;
  seq_bounds(P.d, j, drow0, dlen, nullptr);
  if (t >= dlen) return;
  const long long drow = drow0 + t;
  const float g = P.g[p];
  const T* qsrc = (const T*)P.q.data + qrow * P.q.row_stride;
  const T* dsrc = (const T*)P.d.data + drow * P.d.row_stride;
  const float fq = g * row_factor(P.q, qrow);
  const float fd = g * row_factor(P.d, drow);
  if (VEC) {
    // four consecutive elements per lane and one 16-byte reduction per lane (rows and width are multiples of 4)
    for (int k = lane * 4; k < P.dim; k += 128) {
      float v[4];
      if (P.gd32) {
        load4<T>(qsrc + k, v);
        atomicAdd(reinterpret_cast<float4*>(P.gd32 + drow * P.dim + k), make_float4(fq * v[0], fq * v[1], fq * v[2], fq * v[3]));
      }
      if (WITH_DQ && P.gq32) {
        load4<T>(dsrc + k, v);
        atomicAdd(reinterpret_cast<float4*>(P.gq32 + qrow * P.dim + k), make_float4(fd * v[0], fd * v[1], fd * v[2], fd * v[3]));
      }
    }
  } else {
    for (int k = lane; k < P.dim; k += 32) {
      if (P.gd32) atomicAdd(P.gd32 + drow * P.dim + k, fq * to_f32(qsrc[k]));
      if (WITH_DQ && P.gq32) atomicAdd(P.gq32 + qrow * P.dim + k, fd * to_f32(dsrc[k]));
    }
  }
}

// Finalise an fp32 accumulator: optional Jacobian, optional scale, cast.  Warp per row.
template <typename T, typename G>
__global__ void __launch_bounds__(256) bwd_finalize_kernel(const float* __restrict__ acc32, SeqView v, int dim, int normalize,
                                                         G* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= v.n_rows) return;
  const float* a = acc32 + row * dim;
  if (normalize) {
    const float inv = v.inv_norm[row];
    const T* src = (const T*)v.data + row * v.row_stride;
    float dot = 0.f;
    for (int k = lane; k < dim; k += 32) dot = fmaf(a[k], to_f32(src[k]) * inv, dot);
    dot = warp_sum(dot);
    for (int k = lane; k < dim; k += 32) out[row * dim + k] = from_f32<G>((a[k] - dot * to_f32(src[k]) * inv) * inv);
  } else {
    const float f = v.scale_scalar * (v.scale ? v.scale[row] : 1.f);
    for (int k = lane; k < dim; k += 32) out[row * dim + k] = from_f32<G>(a[k] * f);
  }
}

// Sort keys of a pair list: the query and the document of every pair (a pair with an index out of range gets the key
// one past the last sequence on both sides, so it sorts behind every run and no gradient kernel visits it), and the
// pair index as the value that travels with them.
__global__ void pair_keys_kernel(const int* __restrict__ pair_q, const int* __restrict__ pair_d, long long n, int n_q, int n_d,
                                 unsigned* __restrict__ kq, unsigned* __restrict__ kd, unsigned* __restrict__ vq,
                                 unsigned* __restrict__ vd, int* status) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int i = pair_q[p], j = pair_d[p];
  const bool ok = i >= 0 && i < n_q && j >= 0 && j < n_d;
  if (!ok && status) atomicOr(status, LIK_DEV_PAIR_RANGE);
  kq[p] = ok ? (unsigned)i : (unsigned)n_q;
  kd[p] = ok ? (unsigned)j : (unsigned)n_d;
  vq[p] = (unsigned)p;
  vd[p] = (unsigned)p;
}

namespace {

struct BwdPlan {
  size_t qn_off, dn_off, gq32_off, gd32_off, pairs_off, begin_off, cnt_off, total;
  size_t kq_off, kd_off, pq_off, pd_off, sq_off, sd_off, sort_off;  // pair lists grouped by query / by document
  bool fast, sorted;
  bool list_sorted;  // pair list on the deterministic kernels
  int sort_warps;    // warps of the winner sort that take entries (a histogram each): at least 256 entries of a document per warp
  int sort_cluster;  // CTAs per document
  bool sort_clears;  // every row belongs to a document: the sort writes all the counts, nothing is cleared in front of it
  int sort_threads;  // threads of its CTAs: more warps than that when the documents are long (clearing and offsets go with the length)
  bool row16;  // 16-byte gathers: rows 16-byte aligned, width a multiple of 16 bytes, at most 1024 bytes
  bool fused;      // both gradients in one launch (bwd_fused16_kernel)
  bool fused_quads;
  int fused_threads, fused_rounds, fused_hist, fused_parts;
  size_t fused_bytes;
  int dq_split;    // grad_q: document ranges per query (1: one CTA walks all the documents of its query tokens)
  size_t dqp_off;  // their partial rows
  int ld_pad;
  size_t sort_smem;
};

bool bwd_fast_ok(const lik_bwd_args& a) {
  // vector fast paths: rows 8/16-byte aligned, width a multiple of 4 and at most 256
  const size_t eb = dtype_size(a.dtype);
  return a.dim % 4 == 0 && a.dim <= 256 && (a.q.row_stride * eb) % (4 * eb) == 0 && (a.d.row_stride * eb) % (4 * eb) == 0 &&
         ((uintptr_t)a.q.data % (4 * eb)) == 0 && ((uintptr_t)a.d.data % (4 * eb)) == 0 && ((uintptr_t)a.grad_q % 16) == 0 &&
         ((uintptr_t)a.grad_d % 16) == 0 && a.q.n_rows < (1ll << 31) && a.d.n_rows < (1ll << 31);  // row indices travel as int
}

bool bwd_row16_ok(const lik_bwd_args& a) {
  const size_t eb = dtype_size(a.dtype);
  return bwd_fast_ok(a) && (a.dim * eb) % 16 == 0 && a.dim * eb <= 1024 && (a.q.row_stride * eb) % 16 == 0 &&
         (a.d.row_stride * eb) % 16 == 0 && ((uintptr_t)a.q.data % 16) == 0 && ((uintptr_t)a.d.data % 16) == 0;
}

// winners of a problem from which grad_Q runs on a second stream beside the sort and reduce kernels of grad_D
constexpr long long kForkEntries = 1ll << 20;

// saved winners that are read (and sorted) four at a time
bool winners_in_quads(const lik_bwd_args& a) { return a.argmax_stride % 4 == 0 && ((uintptr_t)a.argmax % 16) == 0; }

BwdPlan plan_bwd(const lik_bwd_args& a) {
  BwdPlan pl{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  pl.qn_off = pl.dn_off = pl.gq32_off = pl.gd32_off = pl.pairs_off = pl.begin_off = pl.cnt_off = (size_t)-1;
  pl.fast = bwd_fast_ok(a);
  pl.row16 = bwd_row16_ok(a);
  pl.sorted = false;
  pl.fused = false;
  if (a.normalize & LIK_NORM_Q) pl.qn_off = take((size_t)a.q.n_rows * 4);
  if (a.normalize & LIK_NORM_D) pl.dn_off = take((size_t)a.d.n_rows * 4);
  const bool list = a.pairing == LIK_PAIR_LIST;
  pl.kq_off = pl.kd_off = pl.pq_off = pl.pd_off = pl.sq_off = pl.sd_off = pl.sort_off = (size_t)-1;
  // a pair list goes through the same deterministic kernels once its pairs are grouped by query and by document
  pl.list_sorted = list && a.deterministic && pl.fast && a.n_pairs > 0 && a.n_pairs < (1ll << 31) && a.d.max_len > 0 &&
                   a.q.max_len > 0 && a.q.n_seq > 0 && a.d.n_seq > 0;
  if (pl.list_sorted) {
    const size_t ws_sort = ((size_t)(a.d.max_len + 1) + a.d.max_len + 2) * 4;  // one CTA per document, one warp counts
    if (ws_sort > 200 * 1024) pl.list_sorted = false;
  }
  if (pl.list_sorted) {
    pl.kq_off = take((size_t)a.n_pairs * 4);
    pl.kd_off = take((size_t)a.n_pairs * 4);
    pl.pq_off = take((size_t)a.n_pairs * 4);
    pl.pd_off = take((size_t)a.n_pairs * 4);
    pl.sq_off = take((size_t)(a.q.n_seq + 1) * 4);
    pl.sd_off = take((size_t)(a.d.n_seq + 1) * 4);
    pl.sort_off = take(sort_pairs_scratch(a.n_pairs));
  }
  // few query tokens against many documents: one CTA per 16 query tokens would leave most of the GPU idle
  pl.dq_split = 1;
  pl.dqp_off = (size_t)-1;
  if (a.grad_q && pl.row16 && a.pairing == LIK_PAIR_CROSS && a.q.n_seq > 0 && a.q.max_len > 0 && a.dim % 4 == 0) {
    const long long base = (long long)a.q.n_seq * ceil_div(a.q.max_len, DQ16_TOK);
    const long long chunks = ceil_div(a.d.n_seq, DQ_JC);
    long long z = (2ll * sm_count()) / base;
    if (z > chunks / 2) z = chunks / 2;  // at least two rounds of documents per range
    if (z > 64) z = 64;
    if (z >= 2) {
      pl.dq_split = (int)z;
      pl.dqp_off = take((size_t)z * a.q.n_rows * a.dim * 4);
    }
  }
  // Few winners per document, and documents whose histograms fit beside each other: everything in one launch, where the sort
  // and reduce kernels do not run beside the grad_Q kernel on a second stream (kForkEntries).  Backward of bf16 rows of 128,
  // sort route to one launch, queries of 32 tokens against documents of up to 300 unless stated: 8 x 32 34 -> 14 us, 32 x 96
  // 46 -> 28, 128 x 128 84 -> 64, 16 x 1024 108 -> 89, 48 x 512 107 -> 91 (up to 1030 tokens 167 -> 140); a candidate list each for
  // 32 queries, 1024 documents 56 -> 29.  From kForkEntries on the two streams win, 32 x 1024 110 to 132, 32 x 2000 205 to 235,
  // 64 x 512 of 1030 137 to 161, except where a document's rows have many winners each and grad_Q is not split: 128 x 2000 670
  // to 592, 96 x 1024 320 to 293, 128 x 2000 of 100 620 to 533; but 128 x 512 of 1030 211 to 246, hence eight per token.
  // (The limits of 1536 tokens and, for more than 1024 winners, 96 documents are the tested range, not crossings: 64 x 95 would
  // go from 52 to 39, 8 x 32 of 1800 tokens from 38 to 28.)
  {
    const long long ent = a.pairing == LIK_PAIR_CROSS ? (long long)a.q.n_seq * a.argmax_stride : (long long)a.argmax_stride;
    const bool rows_owned = a.d.cu || (a.d.seq_stride == a.d.max_len && a.d.n_rows == (int64_t)a.d.n_seq * a.d.seq_stride);
    if (!list && a.deterministic && pl.row16 && a.grad_d && a.d.n_seq > 0 && a.d.max_len > 0 && a.d.max_len <= 1536 && a.q.n_seq > 0 &&
        a.q.max_len > 0 && ent > 0 && ent <= FUSED_ENT && (ent <= 1024 || a.d.n_seq >= 96) && rows_owned &&
        (n_scores_of(a.pairing, a.q.n_seq, a.d.n_seq, a.n_pairs) * a.argmax_stride < kForkEntries ||
         (pl.dq_split == 1 && ent >= 8ll * a.d.max_len))) {
      pl.fused_threads = ent > FUSED_ENT_256 ? 512 : 256;
      const int warps = pl.fused_threads / 32;
      pl.fused_quads = winners_in_quads(a);
      const long long rows = pl.fused_quads && pl.fused_threads > 256 ? ceil_div(ent, 128) * 4 : ceil_div(ent, 32);
      pl.fused_rounds = (int)ceil_div(rows, warps);
      pl.fused_hist = (int)ceil_div(rows, pl.fused_rounds);
      pl.fused_bytes = fused_smem((int)ent, a.d.max_len + 1, pl.fused_hist);
      const size_t dq_bytes = (size_t)DQ_JC * (pl.fused_threads / 16) * sizeof(int2);
      if (pl.fused_bytes < dq_bytes) pl.fused_bytes = dq_bytes;
      pl.fused = pl.fused_bytes <= FUSED_SMEM;
      // few documents: several blocks each, with at least two rows per half-warp
      const long long parts = 2ll * sm_count() / a.d.n_seq, most = ceil_div(a.d.max_len, pl.fused_threads / 16 * 2);
      pl.fused_parts = (int)(parts < 1 ? 1 : (parts > most ? most : parts));
    }
  }
  const bool scatter = list && !pl.list_sorted;
  if (a.grad_q && scatter) pl.gq32_off = take((size_t)a.q.n_rows * a.dim * 4);
  if (a.grad_d && (scatter || !a.deterministic)) pl.gd32_off = take((size_t)a.d.n_rows * a.dim * 4);
  if (!pl.fused && a.grad_d && !scatter && a.deterministic && pl.fast && a.d.n_seq > 0 && a.d.max_len > 0 && a.d.n_rows < (1ll << 31) &&
      a.q.n_rows < (1ll << 31)) {
    const long long n_qrange = a.pairing == LIK_PAIR_CROSS ? a.q.n_seq : (list ? 0 : 1);
    pl.ld_pad = a.d.max_len + 1;
    // entries (query token, winner) per document: every document has the same number, except in a pair list (average)
    const long long ent = a.pairing == LIK_PAIR_CROSS ? (long long)a.q.n_seq * a.argmax_stride
                          : a.pairing == LIK_PAIR_GROUPED ? (long long)a.argmax_stride
                                                          : ceil_div(a.n_pairs, a.d.n_seq) * a.argmax_stride;
    // fewer documents than SMs: as many CTAs per document as leave each two thousand entries, so that the GPU fills up
    pl.sort_cluster = 1;
    while (pl.sort_cluster < 8 && (long long)a.d.n_seq * pl.sort_cluster * 2 <= 2 * sm_count() && ent >= 4096ll * pl.sort_cluster) pl.sort_cluster *= 2;
    auto smem_for = [&](int w) {
      return ((size_t)w * pl.ld_pad + dds_scratch_words(pl.ld_pad, pl.sort_cluster) + 3 * (size_t)n_qrange) * 4;
    };
    if (pl.sort_cluster > 1 && smem_for(1) > 200 * 1024) pl.sort_cluster = 1;  // a document too long for the cluster's counts
    long long nw = ceil_div(ceil_div(ent, pl.sort_cluster), 256);  // a warp per 256 entries: few, long documents still fill their CTAs
    pl.sort_warps = (int)(nw < 1 ? 1 : (nw > DDS_WARPS ? DDS_WARPS : nw));
    while (pl.sort_warps > 1 && smem_for(pl.sort_warps) > 200 * 1024) pl.sort_warps >>= 1;  // long documents: fewer histograms
    pl.sort_smem = smem_for(pl.sort_warps);
    {
      long long by_len = ceil_div(pl.ld_pad, 512);
      if (by_len > DDS_WARPS) by_len = DDS_WARPS;
      pl.sort_threads = 32 * (int)(by_len > pl.sort_warps ? by_len : pl.sort_warps);
    }
    if (pl.sort_smem <= 200 * 1024) {
      pl.sorted = true;
      pl.sort_clears = !a.d.cu && a.d.seq_stride == a.d.max_len && a.d.n_rows == (int64_t)a.d.n_seq * a.d.seq_stride;
      const long long n_ent = n_scores_of(a.pairing, a.q.n_seq, a.d.n_seq, a.n_pairs) * (long long)a.argmax_stride;
      pl.pairs_off = take((size_t)n_ent * sizeof(int2));
      pl.begin_off = take((size_t)a.d.n_rows * sizeof(long long));
      pl.cnt_off = take((size_t)a.d.n_rows * sizeof(int));
    }
  }
  pl.total = off;
  return pl;
}

// grad_Q and grad_D are independent, and both are bound by gather latency rather than by any
// throughput limit, so when both are wanted the grad_Q kernel runs on a second stream beside the
// grad_D kernels: fork after everything already enqueued on the caller's stream, join before returning
// to it.  One auxiliary stream and two events per device, created on first use; the enqueue sequence
// holds a lock because the events are shared by every caller on that device.
struct ForkJoin {
  cudaStream_t aux = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  bool ok = false;
};
std::mutex g_fork_mutex;
ForkJoin g_fork[64];

ForkJoin* fork_join_locked() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  ForkJoin& f = g_fork[dev];
  if (!f.aux) {
    f.ok = cudaStreamCreateWithFlags(&f.aux, cudaStreamNonBlocking) == cudaSuccess &&
           cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming) == cudaSuccess &&
           cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming) == cudaSuccess;
    if (!f.ok) (void)cudaGetLastError();
  }
  return f.ok ? &f : nullptr;
}

template <typename T, typename G>
int run_bwd(const lik_bwd_args& a, BwdParams& P, const BwdPlan& pl, cudaStream_t st_main) {
  const bool list = a.pairing == LIK_PAIR_LIST && !pl.list_sorted;  // pair list on the atomic path
  if (pl.list_sorted) {
    // group the pairs by query and by document: two stable sorts of the pair index
    char* w = (char*)a.workspace;
    unsigned *kq = (unsigned*)(w + pl.kq_off), *kd = (unsigned*)(w + pl.kd_off);
    unsigned *pq = (unsigned*)(w + pl.pq_off), *pd = (unsigned*)(w + pl.pd_off);
    pair_keys_kernel<<<(unsigned)ceil_div(a.n_pairs, 256), 256, 0, st_main>>>(a.pair_q, a.pair_d, a.n_pairs, a.q.n_seq, a.d.n_seq, kq, kd,
                                                                            pq, pd, a.status), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
    auto bits = [](int n) { int b = 1; while ((1ll << b) <= n) ++b; return b; };
    int rc = stable_sort_pairs(kq, pq, a.n_pairs, bits(a.q.n_seq), w + pl.sort_off, st_main);
    if (rc) return rc;
    rc = stable_sort_pairs(kd, pd, a.n_pairs, bits(a.d.n_seq), w + pl.sort_off, st_main);
    if (rc) return rc;
    rc = run_starts(kq, a.n_pairs, a.q.n_seq, (int*)(w + pl.sq_off), st_main);
    if (rc) return rc;
    rc = run_starts(kd, a.n_pairs, a.d.n_seq, (int*)(w + pl.sd_off), st_main);
    if (rc) return rc;
    P.perm_q = (const int*)pq;
    P.perm_d = (const int*)pd;
    P.start_q = (const int*)(w + pl.sq_off);
    P.start_d = (const int*)(w + pl.sd_off);
  }
  // fork only when both gradients run the gather kernels and the problem is large enough to matter
  const bool want_fork = a.grad_q && a.grad_d && !list && a.deterministic && pl.fast && pl.sorted &&
                         P.pm.n_scores * (long long)a.argmax_stride >= kForkEntries;
  std::unique_lock<std::mutex> fork_lock(g_fork_mutex, std::defer_lock);
  ForkJoin* fj = nullptr;
  if (want_fork) {
    fork_lock.lock();
    fj = fork_join_locked();
    if (fj) {
      LIK_CUDA_OK(cudaEventRecord(fj->fork, st_main));
      LIK_CUDA_OK(cudaStreamWaitEvent(fj->aux, fj->fork, 0));
    } else {
      fork_lock.unlock();
    }
  }
  // Stream of the grad_Q kernel; grad_D switches back below.  The winner sort of grad_D so takes the SMs first and grad_Q fills
  // in beside it and the reduction: the other way round costs 32 x 32 pages of 1030 tokens 300 us a step instead of 281 and
  // 256 x 256 documents of 180 tokens 267 instead of 251.
  cudaStream_t st = fj ? fj->aux : st_main;
  const int cmax = (a.dim + 31) / 32;
  char* ws = (char*)a.workspace;
#define LIK_BY_CMAX(KERNEL, GRID, ...)                                          \
  do {                                                                          \
    if (cmax <= 4)                                                              \
      KERNEL<T, G, 4><<<GRID, 256, 0, st>>>(__VA_ARGS__), ::lik::count_launch();                        \
    else if (cmax <= 8)                                                         \
      KERNEL<T, G, 8><<<GRID, 256, 0, st>>>(__VA_ARGS__), ::lik::count_launch();                        \
    else if (cmax <= 16)                                                        \
      KERNEL<T, G, 16><<<GRID, 256, 0, st>>>(__VA_ARGS__), ::lik::count_launch();                       \
    else                                                                        \
      KERNEL<T, G, 32><<<GRID, 256, 0, st>>>(__VA_ARGS__), ::lik::count_launch();                       \
  } while (0)

  const bool fast = pl.fast;
  const bool dq_fused = pl.fused && a.grad_q;
  if (a.grad_q && !dq_fused && !list && a.q.n_seq > 0 && a.q.max_len > 0) {
    dim3 grid((unsigned)a.q.n_seq, (unsigned)ceil_div(a.q.max_len, 8));
    if (pl.row16) {
      const dim3 grid16((unsigned)a.q.n_seq, (unsigned)ceil_div(a.q.max_len, DQ16_TOK), (unsigned)pl.dq_split);
      const dim3 grid_sum((unsigned)a.q.n_seq, (unsigned)ceil_div(a.q.max_len, DQ16_TOK));
      const size_t row_bytes = (size_t)a.dim * sizeof(T);
#define LIK_DQ16(CH_)                                                                              \
  do {                                                                                             \
    bwd_dq16_kernel<T, G, CH_><<<grid16, 256, 0, st>>>(P), ::lik::count_launch();                  \
    if (pl.dq_split > 1) bwd_dq16_sum_kernel<T, G, CH_><<<grid_sum, 256, 0, st>>>(P), ::lik::count_launch(); \
  } while (0)
      if (row_bytes <= 256) LIK_DQ16(1);
      else if (row_bytes <= 512) LIK_DQ16(2);
      else LIK_DQ16(4);
#undef LIK_DQ16
    } else if (fast) {
      if (a.dim <= 128)
        bwd_dq_fast_kernel<T, G, 1><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
      else
        bwd_dq_fast_kernel<T, G, 2><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
    } else {
      LIK_BY_CMAX(bwd_dq_kernel, grid, P);
    }
    LIK_CUDA_OK(cudaGetLastError());
  }
  if (fj) {
    LIK_CUDA_OK(cudaEventRecord(fj->join, fj->aux));
    st = st_main;
  }
  if (pl.fused) {
    FusedShape F;
    F.ld_pad = a.d.max_len + 1;
    F.n_hist = pl.fused_hist;
    F.dq_per_query = (int)ceil_div(a.q.max_len, pl.fused_threads / 16);
    F.dq_blocks = a.q.n_seq * F.dq_per_query;
    F.dq_split = dq_fused ? pl.dq_split : 0;
    F.rounds = pl.fused_rounds;
    F.quads = pl.fused_quads;
    {
      const long long ent = a.pairing == LIK_PAIR_CROSS ? (long long)a.q.n_seq * a.argmax_stride : (long long)a.argmax_stride;
      F.full_rows = (int)(ent / 128 * 4);
      F.tail = (int)(ent % 128 / 4);
    }
    F.parts = pl.fused_parts;
    const unsigned grid = (unsigned)(F.dq_blocks * F.dq_split + a.d.n_seq * F.parts);
    const dim3 grid_sum((unsigned)a.q.n_seq, (unsigned)ceil_div(a.q.max_len, DQ16_TOK));
    const size_t row_bytes = (size_t)a.dim * sizeof(T);
#define LIK_FUSED(CH_, NT_)                                                                                                          \
  do {                                                                                                                               \
    if (pl.fused_bytes > 48 * 1024)                                                                                                  \
      LIK_CUDA_OK(cudaFuncSetAttribute(bwd_fused16_kernel<T, G, CH_, NT_>, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM)); \
    bwd_fused16_kernel<T, G, CH_, NT_><<<grid, NT_, pl.fused_bytes, st>>>(P, F), ::lik::count_launch();                              \
    if (F.dq_split > 1) bwd_dq16_sum_kernel<T, G, CH_><<<grid_sum, 256, 0, st>>>(P), ::lik::count_launch();                          \
  } while (0)
#define LIK_FUSED_NT(CH_)                               \
  do {                                                  \
    if (pl.fused_threads == 256) LIK_FUSED(CH_, 256);   \
    else LIK_FUSED(CH_, 512);                           \
  } while (0)
    if (row_bytes <= 256) LIK_FUSED_NT(1);
    else if (row_bytes <= 512) LIK_FUSED_NT(2);
    else LIK_FUSED_NT(4);
#undef LIK_FUSED_NT
#undef LIK_FUSED
    LIK_CUDA_OK(cudaGetLastError());
  } else if (a.grad_d && !list && a.deterministic && a.d.n_seq > 0 && a.d.max_len > 0) {
    if (pl.sorted) {
      DdSortOut O;
      O.pairs = (int2*)(ws + pl.pairs_off);
      O.tok_begin = (long long*)(ws + pl.begin_off);
      O.tok_cnt = (int*)(ws + pl.cnt_off);
      O.clear_rest = pl.sort_clears;
      auto kernel = winners_in_quads(a) ? bwd_dd_sort4_kernel : bwd_dd_sort_kernel;
      if (pl.sort_smem > 48 * 1024) LIK_CUDA_OK(winners_in_quads(a) ? allow_smem<bwd_dd_sort4_kernel>() : allow_smem<bwd_dd_sort_kernel>());
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = (unsigned)pl.sort_cluster;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)a.d.n_seq * (unsigned)pl.sort_cluster);
      cfg.blockDim = dim3((unsigned)pl.sort_threads);
      cfg.dynamicSmemBytes = pl.sort_smem;
      cfg.stream = st;
      cfg.attrs = &attr;
      cfg.numAttrs = pl.sort_cluster > 1 ? 1 : 0;  // (a launch with clusters of one took 14 us more over 2048 documents)
      LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, P, O, pl.ld_pad, pl.sort_warps));
      ::lik::count_launch();
      if (pl.row16) {
        // one CTA per 16 tokens, except for very many tokens (long documents): there a capped grid walks them
        const long long rg = ceil_div(a.d.n_rows, 16);
        const bool walk = rg > 65536;
        const unsigned rgrid = (unsigned)(walk ? (long long)sm_count() * 32 : rg);
        const size_t row_bytes = (size_t)a.dim * sizeof(T);
#define LIK_REDUCE16(CH_)                                                                                     \
  do {                                                                                                        \
    if (walk) bwd_dd_reduce16_walk_kernel<T, G, CH_><<<rgrid, 256, 0, st>>>(P, O), ::lik::count_launch();     \
    else bwd_dd_reduce16_kernel<T, G, CH_><<<rgrid, 256, 0, st>>>(P, O), ::lik::count_launch();               \
  } while (0)
        if (row_bytes <= 256) LIK_REDUCE16(1);
        else if (row_bytes <= 512) LIK_REDUCE16(2);
        else LIK_REDUCE16(4);
#undef LIK_REDUCE16
      } else {
        const unsigned rgrid = (unsigned)ceil_div(a.d.n_rows, 8);
        if (a.dim <= 128)
          bwd_dd_reduce_kernel<T, G, 1><<<rgrid, 256, 0, st>>>(P, O), ::lik::count_launch();
        else
          bwd_dd_reduce_kernel<T, G, 2><<<rgrid, 256, 0, st>>>(P, O), ::lik::count_launch();
      }
    } else {
      dim3 grid((unsigned)a.d.n_seq, (unsigned)ceil_div(a.d.max_len, DD_TOK));
      LIK_BY_CMAX(bwd_dd_owned_kernel, grid, P);
    }
    LIK_CUDA_OK(cudaGetLastError());
  }
#undef LIK_BY_CMAX
  const bool scatter_q = a.grad_q && list;
  const bool scatter_d = a.grad_d && (list || !a.deterministic);
  if (scatter_q || scatter_d) {
    P.gq32 = scatter_q ? (float*)(ws + pl.gq32_off) : nullptr;
    P.gd32 = scatter_d ? (float*)(ws + pl.gd32_off) : nullptr;
    if (P.gq32) LIK_CUDA_OK(cudaMemsetAsync(P.gq32, 0, (size_t)a.q.n_rows * a.dim * 4, st));
    if (P.gd32) LIK_CUDA_OK(cudaMemsetAsync(P.gd32, 0, (size_t)a.d.n_rows * a.dim * 4, st));
    long long warps = P.pm.n_scores * (long long)a.argmax_stride;
    if (warps > 0) {
      unsigned grid = (unsigned)ceil_div(warps, 8);
      if (scatter_q && fast)
        bwd_scatter_kernel<T, true, true><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
      else if (scatter_q)
        bwd_scatter_kernel<T, true, false><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
      else if (fast)
        bwd_scatter_kernel<T, false, true><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
      else
        bwd_scatter_kernel<T, false, false><<<grid, 256, 0, st>>>(P), ::lik::count_launch();
      LIK_CUDA_OK(cudaGetLastError());
    }
    if (P.gq32 && a.q.n_rows > 0) {
      bwd_finalize_kernel<T, G><<<(unsigned)ceil_div(a.q.n_rows, 8), 256, 0, st>>>(P.gq32, P.q, a.dim, a.normalize & LIK_NORM_Q, (G*)a.grad_q), ::lik::count_launch();
      LIK_CUDA_OK(cudaGetLastError());
    }
    if (P.gd32 && a.d.n_rows > 0) {
      bwd_finalize_kernel<T, G><<<(unsigned)ceil_div(a.d.n_rows, 8), 256, 0, st>>>(P.gd32, P.d, a.dim, a.normalize & LIK_NORM_D, (G*)a.grad_d), ::lik::count_launch();
      LIK_CUDA_OK(cudaGetLastError());
    }
  }
  if (fj) LIK_CUDA_OK(cudaStreamWaitEvent(st_main, fj->join, 0));
  return LIK_OK;
}

template <typename T>
int run_bwd_g(const lik_bwd_args& a, BwdParams& P, const BwdPlan& pl, cudaStream_t st) {
  switch (a.grad_dtype) {
    case LIK_F32:
      return run_bwd<T, float>(a, P, pl, st);
    case LIK_F16:
      return run_bwd<T, __half>(a, P, pl, st);
    case LIK_BF16:
      return run_bwd<T, __nv_bfloat16>(a, P, pl, st);
  }
  set_error("grad_dtype %d not supported", a.grad_dtype);
  return LIK_ERR_INVALID;
}

}  // namespace
}  // namespace lik

extern "C" size_t lik_maxsim_bwd_workspace(const lik_bwd_args* a) {
  if (!a) return 0;
  return lik::plan_bwd(*a).total;
}

extern "C" int lik_maxsim_bwd(const lik_bwd_args* a, lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(a != nullptr, "args is NULL");
  LIK_REQUIRE(a->dim > 0 && a->dim <= 1024, "dim %d outside (0, 1024]", a->dim);
  LIK_REQUIRE(a->pairing >= 0 && a->pairing <= 2, "unknown pairing %d", a->pairing);
  LIK_REQUIRE(a->pairing != LIK_PAIR_GROUPED || a->group > 0, "group must be positive");
  LIK_REQUIRE(a->grad_scores && a->argmax, "grad_scores and argmax are required");
  LIK_REQUIRE(a->argmax_stride > 0 || a->q.max_len == 0, "argmax_stride must be positive");
  cudaStream_t st = (cudaStream_t)stream;
  BwdPlan pl = plan_bwd(*a);
  if (pl.total > a->workspace_bytes || (pl.total && !a->workspace)) {
    set_error("workspace too small: need %zu bytes, got %zu", pl.total, a->workspace_bytes);
    return LIK_ERR_WORKSPACE;
  }
  const float *qn = nullptr, *dn = nullptr;
  PrepJobs prep;
  if (a->normalize & LIK_NORM_Q) {
    float* w = (float*)((char*)a->workspace + pl.qn_off);
    prep.norm[0] = norm_job(a->q, a->dtype, a->dim, kBwdNormEps, w, false);
    qn = w;
  }
  if (a->normalize & LIK_NORM_D) {
    float* w = (float*)((char*)a->workspace + pl.dn_off);
    prep.norm[1] = norm_job(a->d, a->dtype, a->dim, kBwdNormEps, w, false);
    dn = w;
  }
  if (pl.sorted && !pl.sort_clears) prep.fill[0] = FillJob{(char*)a->workspace + pl.cnt_off, (size_t)a->d.n_rows * sizeof(int), 0};  // no winners yet
  {
    const int rc = launch_prep(prep, st);
    if (rc) return rc;
  }
  BwdParams P;
  P.q = make_view(a->q, qn);
  P.d = make_view(a->d, dn);
  P.pm = PairMap{a->pairing, a->group, a->q.n_seq, a->d.n_seq, a->pair_q, a->pair_d,
                 n_scores_of(a->pairing, a->q.n_seq, a->d.n_seq, a->n_pairs)};
  P.dim = a->dim;
  P.normalize = a->normalize;
  P.g = a->grad_scores;
  P.argmax = a->argmax;
  P.argmax_stride = a->argmax_stride;
  P.grad_q = a->grad_q;
  P.grad_d = a->grad_d;
  P.gq32 = P.gd32 = nullptr;
  P.status = a->status;
  P.perm_q = P.start_q = P.perm_d = P.start_d = nullptr;
  P.dq_split = pl.dq_split;
  P.dq_partial = pl.dq_split > 1 ? (float*)((char*)a->workspace + pl.dqp_off) : nullptr;
  switch (a->dtype) {
    case LIK_F32:
      return run_bwd_g<float>(*a, P, pl, st);
    case LIK_F16:
      return run_bwd_g<__half>(*a, P, pl, st);
    case LIK_BF16:
      return run_bwd_g<__nv_bfloat16>(*a, P, pl, st);
  }
  set_error("dtype %d not supported by the backward", a->dtype);
  return LIK_ERR_UNSUPPORTED;
}
