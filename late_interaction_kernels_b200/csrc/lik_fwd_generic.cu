// Portable fp32-accumulate MaxSim forward: any element type, any embedding
// width, every layout and pairing, fp32 FMA in a fixed order.  It is the home of
// the shapes that the tcgen05 kernels do not take (odd widths; of fp32 inputs also
// pair lists, candidate lists, packed queries and long ones).
#include <atomic>

#include "lik_common.cuh"

namespace lik {

namespace {
thread_local char g_err[512] = "";
std::atomic<unsigned long long> g_launches{0};
}

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
unsigned long long launch_count() { return g_launches.load(std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
const char* get_error() { return g_err; }

int sm_count() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

// y[row] = round_to_T(x[row] / max(||x[row]||, eps)), dense rows of `dim` elements.  One warp per row; the row is
// read once (it stays in registers between the norm and the scaling for widths up to 256).
template <typename T>
__global__ void row_normalize_kernel(const T* __restrict__ x, long long n_rows, int dim, long long stride, float eps,
                                     T* __restrict__ y) {
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  const int lane = threadIdx.x & 31;
  const T* p = x + row * stride;
  T* o = y + row * dim;
  float v[8];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int k = c * 32 + lane;
    v[c] = k < dim ? to_f32(p[k]) : 0.f;
    ss = fmaf(v[c], v[c], ss);
  }
  for (int k = 256 + lane; k < dim; k += 32) {
    const float w = to_f32(p[k]);
    ss = fmaf(w, w, ss);
  }
  ss = warp_sum(ss);
  const float inv = inv_norm(ss, eps);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int k = c * 32 + lane;
    if (k < dim) o[k] = from_f32<T>(v[c] * inv);
  }
  for (int k = 256 + lane; k < dim; k += 32) o[k] = from_f32<T>(to_f32(p[k]) * inv);
}

// Normalised copy of a 16-bit matrix (dense output rows).
int launch_row_normalize(const void* data, int dtype, long long n_rows, int dim, long long stride, float eps, void* out,
                         cudaStream_t st) {
  if (n_rows <= 0) return LIK_OK;
  const int warps = 8;
  dim3 grid((unsigned)ceil_div(n_rows, warps)), block(warps * 32);
  switch (dtype) {
    case LIK_F16:
      row_normalize_kernel<<<grid, block, 0, st>>>((const __half*)data, n_rows, dim, stride, eps, (__half*)out), ::lik::count_launch();
      break;
    case LIK_BF16:
      row_normalize_kernel<<<grid, block, 0, st>>>((const __nv_bfloat16*)data, n_rows, dim, stride, eps, (__nv_bfloat16*)out), ::lik::count_launch();
      break;
    default:
      set_error("normalised copies exist for 16-bit inputs only (dtype %d)", dtype);
      return LIK_ERR_INVALID;
  }
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

// ---------------------------------------------------------------------------------
// Exact forward: fp32 FMA in a fixed order.
//
// A CTA of four warps scores one document against QB queries (QB = 2 for the cross product, where both share the staged
// document; 1 otherwise).  Tile: 32 query tokens of every query x up to 128 document tokens, a quarter per warp; a thread owns
// 4 QB query tokens x up to 8 document tokens and walks the width four features at a time: with QB = 2, sixteen 16-byte
// shared-memory loads feed 256 FMAs, the ratio at which both pipes are busy.  Rows are staged row-major with a pitch of
// KC + 4 floats: the rows that a quarter-warp's load touches lie four banks apart.  Documents are trimmed to their last valid
// token.  32 queries x 32 documents of 36..180 tokens: 91 -> 58 us (a thread per query token before, one 16-byte load per
// four FMAs, padding multiplied); what is left beside the FMAs (23 us of issue) is the uneven documents: the slowest SM is a
// third behind the mean.
// ---------------------------------------------------------------------------------
constexpr int G_QC = 32;   // query tokens per tile
constexpr int G_DC = 128;  // document tokens per tile
constexpr int G_KC = 64;   // features staged at once: 52 KB per CTA
constexpr int G_PITCH = G_KC + 4;
// With few documents every block ranks them by length and takes the one of its place in that order, so that the blocks that
// start last are the shortest and the first ones of an SM add up alike.  (Dealt as they come, the fullest of 148 SMs held 1.35
// times the mean of 512 blocks of 36..180 tokens: 32 x 32 documents 58.7 -> 47.0 us.)  A thread compares two documents with all,
// four lengths per load.  More than eight blocks per SM even out by themselves, and ranking costs a block about 1 us: 64 x 256
// documents of 102..512 tokens 1504 us as they come, 1576 ranked.
constexpr int G_RANKED = 256;

struct GenericFwdParams {
  SeqView q, d;
  PairMap pm;
  int dim;
  int vec4;  // rows start on a boundary of four elements and the width is a multiple of four: staged four at a time
  float* scores;
  int* argmax;
  int argmax_stride;
  int* status;
  long long first;  // number of the launch's first block: a grid holds fewer than 2^31
  int by_length;    // cross product: the blocks of the longest documents come first (n_d <= G_RANKED)
};

__device__ __forceinline__ void cp_async16_zfill(float* dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// four neighbouring elements as floats (the address is a multiple of their size)
__device__ __forceinline__ float4 load4_f32(const __half* p) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 load4_f32(const __nv_bfloat16* p) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ float4 load4_f32(const e4m3_t* p) {
  const unsigned r = __ldg(reinterpret_cast<const unsigned*>(p));
  auto at = [&](int i) { return to_f32(e4m3_t{(uint8_t)(r >> (8 * i))}); };
  return make_float4(at(0), at(1), at(2), at(3));
}

// rows [0, n) of a matrix, features [k0, k0 + kw) -> dst rows of G_PITCH floats; rows past `n` up to `rows` become zeros
template <typename T>
__device__ __forceinline__ void stage_rows(float* dst, const T* src, long long pitch, int rows, int n, int k0, int kw, bool vec4, int tid) {
  const int lane = tid & 31;
  if (vec4) {
    if constexpr (sizeof(T) == 4) {  // a warp per row, sixteen bytes per lane
      const bool col = lane * 4 < kw;
      const float* p = reinterpret_cast<const float*>(src) + k0 + lane * 4;
      for (int r = tid >> 5; r < rows; r += 4) {
        const bool on = r < n;
        if (col) cp_async16_zfill(dst + r * G_PITCH + lane * 4, p + (on ? r : 0) * pitch, on);
      }
    } else {
      // Narrower types are widened on the way: a half-warp per row, four elements per lane, four rows in flight.  (Element by
      // element, two bytes per load, staging took longer than the FMAs: 2000 pairs of up to 200 x 700
      // bf16 tokens 3071 us, now 1410.)
      const int c = (lane & 15) * 4;
      if (c < kw) {
#pragma unroll 4
        for (int r = (tid >> 5) * 2 + (lane >> 4); r < rows; r += 8) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < n) v = load4_f32(src + r * pitch + k0 + c);
          *reinterpret_cast<float4*>(dst + r * G_PITCH + c) = v;
        }
      }
    }
  } else {
    const int kp = (kw + 3) & ~3;
    for (int r = tid >> 5; r < rows; r += 4)
      for (int c = lane; c < kp; c += 32) dst[r * G_PITCH + c] = (r < n && c < kw) ? to_f32(src[r * pitch + k0 + c]) : 0.f;
  }
}

// acc[i][t] += <query token i, document token t> over k_end staged features
template <int QI, int TN>
__device__ __forceinline__ void generic_tile(float (&acc)[QI][8], const float* qp, const float* dp, int k_end) {
#pragma unroll 1
  for (int k = 0; k < k_end; k += 4) {
    float4 q4[QI];
#pragma unroll
    for (int i = 0; i < QI; ++i) q4[i] = *reinterpret_cast<const float4*>(qp + i * 8 * G_PITCH + k);
#pragma unroll
    for (int t = 0; t < TN; t += 2) {
      float4 d4[2];
      d4[0] = *reinterpret_cast<const float4*>(dp + t * 4 * G_PITCH + k);
      d4[1] = *reinterpret_cast<const float4*>(dp + (t + 1) * 4 * G_PITCH + k);
      // feature by feature, so that the FMAs of one accumulator stand apart
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < QI; ++i)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float q = c == 0 ? q4[i].x : (c == 1 ? q4[i].y : (c == 2 ? q4[i].z : q4[i].w));
            const float d = c == 0 ? d4[u].x : (c == 1 ? d4[u].y : (c == 2 ? d4[u].z : d4[u].w));
            acc[i][t + u] = fmaf(q, d, acc[i][t + u]);
          }
    }
  }
}

template <typename T, int QB>
__global__ void __launch_bounds__(128, 3) fwd_generic_kernel(GenericFwdParams P) {
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                            // [QB][32 rows]
  float* Ds = smem + QB * G_QC * G_PITCH;      // [128 rows]
  __shared__ float red_m[QB][4][G_QC];
  __shared__ int red_i[QB][4][G_QC];
  __shared__ __align__(16) int d_len[G_RANKED];
  __shared__ int d_pick;
  __shared__ float col_f[G_DC];  // multiplier of every document token of the tile; NaN: the token does not count

  constexpr int QI = 4 * QB;  // query tokens per thread: qg + 8 i of the staged 32 QB
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int qg = lane & 7, dg = lane >> 3;
  const T* __restrict__ Qg = (const T*)P.q.data;
  const T* __restrict__ Dg = (const T*)P.d.data;
  const int k_chunks = (P.dim + G_KC - 1) / G_KC;

  // this query block's score slot
  long long slot[QB];
  int qi[QB], dj = 0;
  bool ok[QB];
  const long long block = P.first + blockIdx.x;
  int place = -1, picked = 0;  // the block's place in the order of lengths, and the document there
  if (P.by_length) {
    const int n_d = P.pm.n_d, n_qb = (P.pm.n_q + QB - 1) / QB;
    place = (int)(block / n_qb);
    for (int j = tid; j < G_RANKED; j += 128) {
      long long r0;
      int len = -1;
      if (j < n_d) seq_bounds(P.d, j, r0, len, nullptr);
      d_len[j] = len;
    }
    __syncthreads();
    for (int j = tid; j < n_d; j += 128) {
      const int mine = d_len[j];
      int rank = 0;
      for (int i = 0; i < n_d; i += 4) {  // (places past n_d hold -1)
        const int4 l = *reinterpret_cast<const int4*>(&d_len[i]);
        rank += (l.x > mine || (l.x == mine && i < j)) + (l.y > mine || (l.y == mine && i + 1 < j)) + (l.z > mine || (l.z == mine && i + 2 < j)) +
                (l.w > mine || (l.w == mine && i + 3 < j));
      }
      if (rank == place) d_pick = j;
    }
    __syncthreads();
    picked = d_pick;
  }
  if (QB == 1 && place >= 0) {
    qi[0] = (int)(block - (long long)place * P.pm.n_q);
    dj = picked;
    slot[0] = (long long)qi[0] * P.pm.n_d + dj;
    ok[0] = true;
  } else if (QB == 1) {
    slot[0] = block;
    ok[0] = decode_pair(P.pm, slot[0], qi[0], dj, tid == 0 ? P.status : nullptr);
  } else {
    const int n_qb = (P.pm.n_q + QB - 1) / QB;
    dj = (int)(block / n_qb);
    const int q0 = (int)(block - (long long)dj * n_qb) * QB;
    if (place >= 0) dj = picked;
#pragma unroll
    for (int b = 0; b < QB; ++b) {
      qi[b] = q0 + b;
      ok[b] = qi[b] < P.pm.n_q;
      slot[b] = (long long)qi[b] * P.pm.n_d + dj;
    }
  }
  long long qrow0[QB], drow0 = 0;
  int qlen[QB], dlen = 0, qmax = 0;
#pragma unroll
  for (int b = 0; b < QB; ++b) {
    qrow0[b] = 0;
    qlen[b] = 0;
    if (ok[b]) {
      seq_bounds(P.q, qi[b], qrow0[b], qlen[b], P.status);
      seq_bounds(P.d, dj, drow0, dlen, P.status);
    }
    if (P.argmax && qlen[b] > P.argmax_stride) {
      if (tid == 0 && P.status) atomicOr(P.status, LIK_DEV_ARGMAX_STRIDE);
      qlen[b] = P.argmax_stride;
    }
    qmax = max(qmax, qlen[b]);
  }
  // the query that this warp sums at the end of a tile (warps 0 .. QB - 1)
  const int mq = warp < QB ? warp : 0;
  const int my_qlen = QB == 1 || mq == 0 ? qlen[0] : qlen[QB - 1];
  const long long my_qrow0 = QB == 1 || mq == 0 ? qrow0[0] : qrow0[QB - 1];
  const long long my_slot = QB == 1 || mq == 0 ? slot[0] : slot[QB - 1];
  const bool my_ok = QB == 1 || mq == 0 ? ok[0] : ok[QB - 1];

  float score = 0.f;  // meaningful in warps 0 .. QB - 1
  for (int qc = 0; qc < qmax; qc += G_QC) {
    float m[QI];
    int mi[QI];
#pragma unroll
    for (int i = 0; i < QI; ++i) {
      m[i] = -INFINITY;
      mi[i] = -1;
    }
    // the document in chunks of equal size, four warps with an equal part of a chunk each
    const int n_chunk = (dlen + G_DC - 1) / G_DC;
    const int per = n_chunk ? ((dlen + n_chunk - 1) / n_chunk + 31) & ~31 : 0;
    const int T_n = per >> 4;  // document tokens per thread: 2, 4, 6 or 8
    for (int dc = 0; dc < dlen; dc += per) {
      float acc[QI][8];
#pragma unroll
      for (int i = 0; i < QI; ++i)
#pragma unroll
        for (int t = 0; t < 8; ++t) acc[i][t] = 0.f;
      const int ncols = min(per, dlen - dc);
      for (int kc = 0; kc < k_chunks; ++kc) {
        const int k0 = kc * G_KC, kw = min(G_KC, P.dim - k0);
        __syncthreads();
        if (dc == 0 || k_chunks > 1) {
#pragma unroll
          for (int b = 0; b < QB; ++b)
            stage_rows<T>(Qs + b * G_QC * G_PITCH, Qg + (qrow0[b] + qc) * P.q.row_stride, P.q.row_stride, G_QC, min(G_QC, qlen[b] - qc), k0, kw, P.vec4, tid);
        }
        stage_rows<T>(Ds, Dg + (drow0 + dc) * P.d.row_stride, P.d.row_stride, per, ncols, k0, kw, P.vec4, tid);
        if (kc == 0) {  // (one token per thread, in flight with the rows: read token by token behind the FMAs they cost more than those)
          float f = __int_as_float(0x7fffffff);
          if (tid < ncols && row_valid(P.d, drow0 + dc + tid)) f = row_factor(P.d, drow0 + dc + tid);
          col_f[tid] = f;
        }
        cp_async_wait_all();
        __syncthreads();
        const float* qp = Qs + qg * G_PITCH;                      // query tokens qg, qg + 8, ...
        const float* dp = Ds + (warp * 4 * T_n + dg) * G_PITCH;   // document tokens dg, dg + 4, ...
        const int k_end = (kw + 3) & ~3;
        // straight-line code for every even count of document tokens: a test inside the loop keeps the FMAs of its two sides apart
        if (T_n <= 2) generic_tile<QI, 2>(acc, qp, dp, k_end);
        else if (T_n <= 4) generic_tile<QI, 4>(acc, qp, dp, k_end);
        else if (T_n <= 6) generic_tile<QI, 6>(acc, qp, dp, k_end);
        else generic_tile<QI, 8>(acc, qp, dp, k_end);
      }
      {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          if (t >= T_n) break;
          const int tok = dc + warp * 4 * T_n + dg + 4 * t;
          const float f = col_f[warp * 4 * T_n + dg + 4 * t];
#pragma unroll
          for (int i = 0; i < QI; ++i) {
            const float v = acc[i][t] * f;  // (a NaN beats nothing)
            if (v > m[i]) {
              m[i] = v;
              mi[i] = tok;
            }
          }
        }
      }
    }
    // combine the lanes that hold the same query tokens, then the warps (each saw other document tokens; ties: lower token)
    auto better = [](float wm, int wi, float bm, int bi) { return wi >= 0 && (bi < 0 || wm > bm || (wm == bm && wi < bi)); };
#pragma unroll
    for (int i = 0; i < QI; ++i) {
#pragma unroll
      for (int o = 8; o <= 16; o <<= 1) {
        const float wm = __shfl_xor_sync(0xffffffffu, m[i], o);
        const int wi = __shfl_xor_sync(0xffffffffu, mi[i], o);
        if (better(wm, wi, m[i], mi[i])) {
          m[i] = wm;
          mi[i] = wi;
        }
      }
      if (dg == 0) {
        red_m[i >> 2][warp][qg + 8 * (i & 3)] = m[i];
        red_i[i >> 2][warp][qg + 8 * (i & 3)] = mi[i];
      }
    }
    __syncthreads();
    if (warp < QB) {
      float bm = red_m[mq][0][lane];
      int bi = red_i[mq][0][lane];
#pragma unroll
      for (int w = 1; w < 4; ++w)
        if (better(red_m[mq][w][lane], red_i[mq][w][lane], bm, bi)) {
          bm = red_m[mq][w][lane];
          bi = red_i[mq][w][lane];
        }
      const int s = qc + lane;
      float val = 0.f;
      if (s < my_qlen) {
        const long long qrow = my_qrow0 + s;
        if (bi >= 0 && row_valid(P.q, qrow)) val = bm * row_factor(P.q, qrow);
        if (P.argmax) P.argmax[my_slot * P.argmax_stride + s] = bi;
      }
      score += warp_sum(val);
    }
    __syncthreads();  // the next query tokens reuse the hand-over arrays
  }
  if (warp < QB && my_ok) {
    if (lane == 0) P.scores[my_slot] = score;
    if (P.argmax)
      for (int s = max(my_qlen, 0) + lane; s < P.argmax_stride; s += 32) P.argmax[my_slot * P.argmax_stride + s] = -1;
  } else if (QB == 1 && warp == 0) {  // a pair that is out of range scores 0 and has no winners
    if (lane == 0) P.scores[my_slot] = 0.f;
    if (P.argmax)
      for (int s = lane; s < P.argmax_stride; s += 32) P.argmax[my_slot * P.argmax_stride + s] = -1;
  }
}

// Two queries of a cross product share a staged document where that still leaves every SM two blocks; fewer pairs spread better one by one
// (8 x 32 documents of up to 300 tokens 57.6 -> 47.3 us, 4 x 100 of 512 96.7 -> 74.2; at 32 x 32 sharing is ahead, 64.1 to 67.3)
bool fwd_generic_shares(long long n_q, long long n_d) { return n_q > 1 && (n_q + 1) / 2 * n_d >= 2 * sm_count(); }

template <typename T>
static int launch_generic(GenericFwdParams P, cudaStream_t st) {
  const bool cross = P.pm.pairing == LIK_PAIR_CROSS && fwd_generic_shares(P.pm.n_q, P.pm.n_d);
  const long long blocks = cross ? (long long)((P.pm.n_q + 1) / 2) * P.pm.n_d : P.pm.n_scores;
  P.by_length = P.pm.pairing == LIK_PAIR_CROSS && P.pm.n_d <= G_RANKED && (P.d.lens || P.d.cu) && blocks <= 8 * sm_count();
  constexpr long long kMaxGrid = 1ll << 30;
  const size_t smem = (size_t)((cross ? 2 : 1) * G_QC + G_DC) * G_PITCH * sizeof(float);
#define LIK_LAUNCH_GENERIC(QB)                                                                                            \
  do {                                                                                                                    \
    LIK_CUDA_OK(cudaFuncSetAttribute(fwd_generic_kernel<T, QB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    for (P.first = 0; P.first < blocks; P.first += kMaxGrid) {                                                            \
      const long long n = blocks - P.first < kMaxGrid ? blocks - P.first : kMaxGrid;                                      \
      fwd_generic_kernel<T, QB><<<(unsigned)n, 128, smem, st>>>(P), ::lik::count_launch();                                \
    }                                                                                                                     \
  } while (0)
  if (cross) LIK_LAUNCH_GENERIC(2);
  else LIK_LAUNCH_GENERIC(1);
#undef LIK_LAUNCH_GENERIC
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

int launch_fwd_generic(const lik_fwd_args& a, const float* qn, const float* dn, cudaStream_t st) {
  GenericFwdParams P;
  P.q = make_view(a.q, qn);
  P.d = make_view(a.d, dn);
  P.pm = PairMap{a.pairing, a.group, a.q.n_seq, a.d.n_seq, a.pair_q, a.pair_d,
                 n_scores_of(a.pairing, a.q.n_seq, a.d.n_seq, a.n_pairs)};
  P.dim = a.dim;
  const uintptr_t four = 4 * dtype_size(a.dtype) - 1;
  P.first = 0;
  P.vec4 = a.dim % 4 == 0 && a.q.row_stride % 4 == 0 && a.d.row_stride % 4 == 0 && ((uintptr_t)a.q.data & four) == 0 && ((uintptr_t)a.d.data & four) == 0;
  P.scores = a.scores;
  P.argmax = a.argmax;
  P.argmax_stride = a.argmax_stride;
  P.status = a.status;
  if (P.pm.n_scores <= 0) return LIK_OK;
  switch (a.dtype) {
    case LIK_F32:
      return launch_generic<float>(P, st);
    case LIK_F16:
      return launch_generic<__half>(P, st);
    case LIK_BF16:
      return launch_generic<__nv_bfloat16>(P, st);
    case LIK_E4M3:
      return launch_generic<e4m3_t>(P, st);
  }
  set_error("unknown dtype %d", a.dtype);
  return LIK_ERR_INVALID;
}

}  // namespace lik
