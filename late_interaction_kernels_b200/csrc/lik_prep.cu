// One launch in front of a scoring or gradient kernel: inverse norms, effective lengths, cleared words.
//
// The norms are bound by HBM reads of the rows.  A row is covered by a group of 8, 16 or 32 lanes that load 16 bytes each
// (a warp instruction fetches several whole rows), four rows of a group are in flight, and rows behind a document's end
// are not read: 300 000 fp16 rows of 128, 60 % of them valid, two launches of 38 us -> one of 17.  (Before: a warp per row, two bytes per lane
// and load, every row.)  Small problems are launch-bound, hence everything in one grid: the jobs take consecutive ranges
// of blocks.
#include "lik_prep.cuh"

namespace lik {

namespace {

constexpr int PREP_THREADS = 256;
constexpr int NORM_ROWS = 4;                    // rows in flight per group of lanes
constexpr int FILL_PER_BLOCK = PREP_THREADS * 16 * 8;

// Loads under a predicate instead of a branch, so that all of a thread's loads are in flight together.
__device__ __forceinline__ uint4 load16_if(const void* p, bool on) {
  uint4 r;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
               "@q ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "=&r"(r.x), "=&r"(r.y), "=&r"(r.z), "=&r"(r.w) : "l"(p), "r"((int)on));
  return r;
}
__device__ __forceinline__ int load_u8_if(const unsigned char* p, bool on) {
  int r;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.u8 %0, [%1];\n\t}" : "=&r"(r) : "l"(p), "r"((int)on));
  return r;
}

__device__ __forceinline__ bool norm_row_live(const NormJob& J, long long row) {
  if (row >= J.n_rows) return false;
  if (J.lens) {
    // (64-bit divisions are a hundred instructions: only where 32 bits do not hold the row)
    const long long j = J.n_rows < (1ll << 31) ? (long long)((unsigned)row / (unsigned)J.seq_stride) : row / J.seq_stride;
    if (row - j * J.seq_stride >= J.lens[j]) return false;
  }
  return true;
}

template <typename T>
__device__ __forceinline__ float sum_sq16(const uint4& r);
template <>
__device__ __forceinline__ float sum_sq16<float>(const uint4& r) {
  const float a = __uint_as_float(r.x), b = __uint_as_float(r.y), c = __uint_as_float(r.z), d = __uint_as_float(r.w);
  return fmaf(a, a, fmaf(b, b, fmaf(c, c, d * d)));
}
template <>
__device__ __forceinline__ float sum_sq16<__nv_bfloat16>(const uint4& r) {
  float s = 0.f;
  fma_sq_pair<__nv_bfloat16>(r.x, s);
  fma_sq_pair<__nv_bfloat16>(r.y, s);
  fma_sq_pair<__nv_bfloat16>(r.z, s);
  fma_sq_pair<__nv_bfloat16>(r.w, s);
  return s;
}
template <>
__device__ __forceinline__ float sum_sq16<__half>(const uint4& r) {
  float s = 0.f;
  fma_sq_pair<__half>(r.x, s);
  fma_sq_pair<__half>(r.y, s);
  fma_sq_pair<__half>(r.z, s);
  fma_sq_pair<__half>(r.w, s);
  return s;
}
template <>
__device__ __forceinline__ float sum_sq16<e4m3_t>(const uint4& r) {
  const unsigned w[4] = {r.x, r.y, r.z, r.w};
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float v = to_f32(e4m3_t{(uint8_t)(w[i] >> (8 * b))});
      s = fmaf(v, v, s);
    }
  return s;
}

// lanes that cover a row: as many as it has 16-byte pieces, at most a warp
__host__ __device__ inline int norm_lanes(long long row_bytes) { return row_bytes <= 128 ? 8 : (row_bytes <= 256 ? 16 : 32); }

template <typename T, int L>
__device__ __forceinline__ void norm_rows_vec(const NormJob& J, int block) {
  const int row_bytes = J.dim * (int)sizeof(T);
  constexpr int groups = PREP_THREADS / L;
  const int gl = threadIdx.x & (L - 1), g = threadIdx.x / L;
  const long long row0 = (long long)block * groups * NORM_ROWS + g;
  float ss[NORM_ROWS];
  bool live[NORM_ROWS];
#pragma unroll
  for (int u = 0; u < NORM_ROWS; ++u) {
    ss[u] = 0.f;
    live[u] = norm_row_live(J, row0 + u * groups);
  }
  if (J.mask) {
    int mb[NORM_ROWS];
    const unsigned char* m = J.mask + row0;
#pragma unroll
    for (int u = 0; u < NORM_ROWS; ++u) mb[u] = load_u8_if(m + u * groups, live[u]);
#pragma unroll
    for (int u = 0; u < NORM_ROWS; ++u) live[u] = mb[u] != 0;
  }
  const long long pitch = J.stride * (long long)sizeof(T), step = pitch * groups;
  const char* p = static_cast<const char*>(J.data) + row0 * pitch + gl * 16;
  if (__any_sync(0xffffffffu, live[0] | live[1] | live[2] | live[3])) {
    for (int b = gl * 16; b < row_bytes; b += L * 16, p += L * 16) {
      uint4 r[NORM_ROWS];
#pragma unroll
      for (int u = 0; u < NORM_ROWS; ++u) r[u] = load16_if(p + u * step, live[u]);
#pragma unroll
      for (int u = 0; u < NORM_ROWS; ++u) ss[u] += sum_sq16<T>(r[u]);
    }
  }
  // The sums of the four rows in one butterfly: at the first two steps a lane hands over the rows that it will not finish,
  // so that every quarter of the group ends up with one row (a fifth of the shuffles, a quarter of the roots and divisions).
  const bool up2 = gl & (L / 2), up1 = gl & (L / 4);
  float a0 = up2 ? ss[2] : ss[0], a1 = up2 ? ss[3] : ss[1];
  a0 += __shfl_xor_sync(0xffffffffu, up2 ? ss[0] : ss[2], L / 2);
  a1 += __shfl_xor_sync(0xffffffffu, up2 ? ss[1] : ss[3], L / 2);
  float v = up1 ? a1 : a0;
  v += __shfl_xor_sync(0xffffffffu, up1 ? a0 : a1, L / 4);
#pragma unroll
  for (int o = L / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int u = (up2 ? 2 : 0) + (up1 ? 1 : 0);
  const bool on = up2 ? (up1 ? live[3] : live[2]) : (up1 ? live[1] : live[0]);
  const long long row = row0 + u * groups;
  if ((gl & (L / 4 - 1)) == 0 && row < J.n_rows) J.out[row] = on ? inv_norm(v, J.eps) : 0.f;
}

// any width and alignment: a warp per row
template <typename T>
__device__ __forceinline__ void norm_rows_any(const NormJob& J, int block) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)block * (PREP_THREADS / 32) + (threadIdx.x >> 5);
  if (row >= J.n_rows) return;
  const T* p = static_cast<const T*>(J.data) + row * J.stride;
  const bool live = norm_row_live(J, row) && (!J.mask || J.mask[row] != 0);
  float ss = 0.f;
  if (live)
    for (int k = lane; k < J.dim; k += 32) {
      const float v = to_f32(p[k]);
      ss = fmaf(v, v, ss);
    }
  ss = warp_sum(ss);
  if (lane == 0) J.out[row] = live ? inv_norm(ss, J.eps) : 0.f;
}

__host__ __device__ inline int elt_size(int dt) { return dt == LIK_F32 ? 4 : (dt == LIK_E4M3 ? 1 : 2); }
__host__ __device__ inline bool norm_vec_ok(const NormJob& J) {
  const int eb = elt_size(J.dtype);
  return (J.dim * eb) % 16 == 0 && (J.stride * eb) % 16 == 0 && ((uintptr_t)J.data & 15) == 0;
}

template <typename T>
__device__ __forceinline__ void norm_block(const NormJob& J, int block) {
  if (!norm_vec_ok(J)) {
    norm_rows_any<T>(J, block);
    return;
  }
  const int L = norm_lanes((long long)J.dim * (int)sizeof(T));
  if (L == 8) norm_rows_vec<T, 8>(J, block);
  else if (L == 16) norm_rows_vec<T, 16>(J, block);
  else norm_rows_vec<T, 32>(J, block);
}

// a warp per document
__device__ __forceinline__ void mask_lens_block(const MaskLensJob& J, int block) {
  const int lane = threadIdx.x & 31;
  const int j = block * (PREP_THREADS / 32) + (threadIdx.x >> 5);
  if (j >= J.n_seq) return;
  int len0 = J.max_len;
  if (J.lens) {
    const int l = J.lens[j];
    len0 = min(max(l, 0), J.max_len);
    if (l != len0 && lane == 0 && J.status) atomicOr(J.status, LIK_DEV_LEN_RANGE);
  }
  const unsigned char* m = J.mask + (long long)j * J.seq_stride;
  int last = -1, cnt = 0;
  if (((uintptr_t)J.mask | (uintptr_t)J.seq_stride) % 4 == 0) {  // four tokens per load
    for (int t = lane * 4; t < len0; t += 128) {
      unsigned w = __ldg(reinterpret_cast<const unsigned*>(m + t));
      if (t + 4 > len0) w &= (1u << (8 * (len0 - t))) - 1u;
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if ((w >> (8 * b)) & 255u) {
          last = t + b;
          ++cnt;
        }
    }
  } else {
    for (int t = lane; t < len0; t += 32)
      if (m[t]) {
        last = t;
        ++cnt;
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) J.out[j] = (last + 1) | (cnt != last + 1 ? J.flag : 0);
}

__device__ __forceinline__ void fill_block(const FillJob& J, int block) {
  const size_t lo = (size_t)block * FILL_PER_BLOCK, hi = lo + FILL_PER_BLOCK < J.bytes ? lo + FILL_PER_BLOCK : J.bytes;
  const int4 v = make_int4(J.word, J.word, J.word, J.word);
  char* p = static_cast<char*>(J.ptr);
  if ((uintptr_t)p & 15) {  // a caller's buffer may sit anywhere
    for (size_t w = lo + (size_t)threadIdx.x * 4; w + 4 <= hi; w += PREP_THREADS * 4) *reinterpret_cast<int*>(p + w) = J.word;
    return;
  }
  size_t b = lo + (size_t)threadIdx.x * 16;
  for (; b + 16 <= hi; b += PREP_THREADS * 16) *reinterpret_cast<int4*>(p + b) = v;
  if (b < hi)  // the last whole words
    for (size_t w = b; w + 4 <= hi; w += 4) *reinterpret_cast<int*>(p + w) = J.word;
}

struct PrepGrid {
  int end[5];  // one past the last block of every job: mask lengths (a chain of dependent steps, so first), norms, fills
};

// (T: the rows' type, the same on both sides)
template <typename T>
__global__ void __launch_bounds__(PREP_THREADS) prep_kernel(const PrepJobs jobs, const PrepGrid G) {
  const int b = blockIdx.x;
  if (b < G.end[0]) mask_lens_block(jobs.mask_lens, b);
  else if (b < G.end[1]) norm_block<T>(jobs.norm[0], b - G.end[0]);
  else if (b < G.end[2]) norm_block<T>(jobs.norm[1], b - G.end[1]);
  else if (b < G.end[3]) fill_block(jobs.fill[0], b - G.end[2]);
  else fill_block(jobs.fill[1], b - G.end[3]);
}

}  // namespace

// `all_rows`: norms of padding too (the caller asked for the norms themselves)
NormJob norm_job(const lik_seqs& s, int dtype, int dim, float eps, float* out, bool all_rows) {
  NormJob j;
  j.data = s.data;
  j.dtype = dtype;
  j.dim = dim;
  j.n_rows = s.n_rows;
  j.stride = s.row_stride;
  j.eps = eps;
  j.out = out;
  if (!all_rows) {
    j.mask = s.mask;
    if (!s.cu && s.lens && s.seq_stride > 0 && s.n_rows == (int64_t)s.n_seq * s.seq_stride) {
      j.lens = s.lens;
      j.seq_stride = s.seq_stride;
    }
  }
  return j;
}

int launch_prep(const PrepJobs& jobs, cudaStream_t st) {
  PrepGrid G;
  long long n = 0;
  if (jobs.mask_lens.mask && jobs.mask_lens.n_seq > 0) n += ceil_div(jobs.mask_lens.n_seq, PREP_THREADS / 32);
  G.end[0] = (int)n;
  for (int i = 0; i < 2; ++i) {
    const NormJob& J = jobs.norm[i];
    if (J.data && J.n_rows > 0) {
      if (J.dtype < LIK_F32 || J.dtype > LIK_E4M3) {
        set_error("unknown dtype %d", J.dtype);
        return LIK_ERR_INVALID;
      }
      const int eb = elt_size(J.dtype);
      n += ceil_div(J.n_rows, norm_vec_ok(J) ? PREP_THREADS / norm_lanes((long long)J.dim * eb) * NORM_ROWS : PREP_THREADS / 32);
    }
    G.end[1 + i] = (int)n;
  }
  for (int i = 0; i < 2; ++i) {
    if (jobs.fill[i].ptr && jobs.fill[i].bytes) n += ceil_div((int64_t)jobs.fill[i].bytes, FILL_PER_BLOCK);
    G.end[3 + i] = (int)n;
  }
  if (n == 0) return LIK_OK;
  if (n >= (1ll << 31)) {
    set_error("too many rows for one launch");
    return LIK_ERR_UNSUPPORTED;
  }
  const int dt = jobs.norm[0].data ? jobs.norm[0].dtype : jobs.norm[1].dtype;
  if (jobs.norm[1].data && jobs.norm[1].dtype != dt) {
    set_error("both sides' rows must have one type");
    return LIK_ERR_INVALID;
  }
  if (dt == LIK_F16) prep_kernel<__half><<<(unsigned)n, PREP_THREADS, 0, st>>>(jobs, G), ::lik::count_launch();
  else if (dt == LIK_BF16) prep_kernel<__nv_bfloat16><<<(unsigned)n, PREP_THREADS, 0, st>>>(jobs, G), ::lik::count_launch();
  else if (dt == LIK_E4M3) prep_kernel<e4m3_t><<<(unsigned)n, PREP_THREADS, 0, st>>>(jobs, G), ::lik::count_launch();
  else prep_kernel<float><<<(unsigned)n, PREP_THREADS, 0, st>>>(jobs, G), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

}  // namespace lik
