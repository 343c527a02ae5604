// fp32 scores on the tensor cores (sm_100a: tcgen05.mma + TMEM): rows cut into three bf16 parts, eight products of parts to a dot product,
// a bound for what that is off, and dot products in fp32 where the bound says so.
//
// The cut.  Let 2^e be the power of two at or below the largest magnitude of a row a (its size).  a0 = the row rounded to multiples of 2^(e-7),
// a1 = the rest rounded to multiples of 2^(e-15), a2 = what is left, rounded to bf16.  a0 b0 has an accumulator of its own, a0 b1 + a1 b0
// another, the third a0 b2 + a1 b1 + a2 b0 + a1 b2 + a2 b1.  The tensor core adds into fp32 but cuts off below (measured: -0.3 ulp on average per 16
// products of full bf16 values, -1.8 over 128, which would shift every score); in the first two it has nothing to cut, since their terms are
// whole multiples of one unit and their sums stay below 2^24 of it.
// The bound.  A product p~ of rows of sizes 2^e and 2^f and width n can be away from the true p by
//   the cuts       2^(e-25) per feature of a, 2^(f-25) of b                                     2^-25 (2^e |b|_1 + 2^f |a|_1)
//   third sum      40 MMAs, each off by 17 ulp of the sum at most: a1 b1, below n 2^(e+f-16)    n 2^(e+f-29.5)
//                  a0 b2 + a2 b0, |a0| <= 2 |a|, below 2^-15 (2^e |b|_1 + 2^f |a|_1)            a twelfth of the first line
//   left out       a2 b2                                                                        n 2^(e+f-32)
//   sum of three   the second and third, below 2^-7 (2^e |b|_1 + 2^f |a|_1), rounded            2^-6 of the first line
// in all below 1.25 times the first line + n 2^(e+f-29), and two roundings of p~ itself (the last sum, the column's multiplier).  It goes with the rows' sizes, not with p: on rows of even features p~
// is off by two or three roundings, where one feature is 2^16 times the others it may be worth nothing.  Sizes and sums of magnitudes are
// taken with the cut, the largest of them per piece, and the epilogue keeps, per query token, the largest p~ of a document and the columns
// that could be the largest in truth: those within both bounds of it, in up to two groups of sixteen.
// The answer.  One candidate whose bound is below max(4, n / 4) 2^-24 |p~|, a quarter of what a chain of n fused multiply-adds is bound by:
// p~.  (Rows of independent Gaussian features, 128 wide, against the best of thirty: half of that.)  Else the candidates' dot products are
// taken in fp32, eight features per lane, and the largest counts; where more than two groups could hold it, all tokens of the document are
// taken that way, and so they are for rows that the cut does not fit (infinities, NaN, sizes beyond 2^50 or below 2^-40).
//
// A CTA per SM takes an equal run of (query tile, document) units, tile by tile, and walks a document in pieces of 64 tokens.
// Warp roles (800 threads):
//   warps 0..7   epilogue, a thread per query token: two sets of four warps take the pieces in turn; where a document ends, the set
//                of its last piece gets the other's candidates through shared memory
//   warp 8       issues the MMAs of a piece, a part of the query times up to three of the piece at once: five per 16 features
//   warps 9..24  cut the rows of the pieces and, where it changes, of the query tile: a half-warp per row; they take the norms too
// Against fwd_generic_kernel, whose fp32 FMAs bound it (queries of up to 32 tokens, documents a fifth to the whole of the length given, normalised):
// 32 x 32 documents of 180 tokens 52 -> 28 us, 1 x 256 of 512 68 -> 50, 64 x 64 of 300 (48-token queries, 96 features) 421 -> 136, 64 x 256 of
// 512 (48 tokens) 3010 -> 750; that last with a feature of the documents 100 or 1000 times the others, every product in fp32, 1120; with infinities in a query
// of every tile 4700, in every sixteenth document 3500; with two features 2^16 times the others, each where the other side has zeros, so that everything
// is gone through by four warps at a time, 28 ms.  (Products for all rows instead of the bound: 32 x 32 35 us, 64 x 256 of 512 and 32 tokens 454 against 375;
// the same by three warps of their own 54 and 620.  Without a1 b2 + a2 b1 the bound is four times as wide, too much for Gaussian rows.)
// What bounds it: issue (59 % active) and the round trips between its roles; the tensor pipe is busy for 45 %.
// Error of the scores against 64 bits, 2-norm over 24 problems of Gaussian rows: 3.3e-8 to 5.3e-8, the other kernel's 5.0e-8 to 6.4e-8.
// Every wait is bounded: on expiry the CTA raises LIK_DEV_WAIT_TIMEOUT in the status word, sets a shared abort flag, frees TMEM and
// returns.  A warp that goes through a document counts its steps, and who waits for it begins anew while they go on.
#include <cfloat>
#include <cmath>

#include "lik_common.cuh"
#include "lik_tc_ptx.cuh"

namespace lik {

namespace {

constexpr int PIECE = 64;                     // document tokens per MMA group
constexpr int PARTS = 3;
constexpr int CUT_WARPS = 16, CUT_WARP0 = 9, ISSUE_WARP = 8, EPI_WARPS = 8;
constexpr int NUM_THREADS = (CUT_WARP0 + CUT_WARPS) * 32;
constexpr int STAGES = 2, ACCS = 2;
constexpr int ACC_COLS = 256;                 // three accumulators of 64 columns, and a gap
constexpr int RING = 4;                       // column arrays and query arrays: see `columns`
constexpr int ROW_BYTES = 128;                // one swizzle span: 64 bf16
constexpr int B_PART = PIECE * ROW_BYTES, B_SLAB = PARTS * B_PART, B_STAGE = 2 * B_SLAB;  // (the parts of B are one matrix of 192 rows)
constexpr int A_SLAB = TILE_M * ROW_BYTES, A_PART = 2 * A_SLAB;
// Candidates of a query token: columns at + i for bit i of `bits`, at2 + i for bit 16 + i
constexpr int NO_MORE = -1, WHOLE_DOC = -2;  // instead of at2: no second group; all tokens
static_assert(PIECE == 4 * CUT_WARPS && TILE_M == 8 * CUT_WARPS, "a half-warp cuts two rows of a piece and four of a query tile");

struct SplitParams {
  SeqView q, d;        // inv_norm unused: the kernel takes the norms
  int n_q, n_d, dim;
  int q_per_tile, n_tiles;
  int norm_q, norm_d;
  float eps;
  float* scores;
  int* argmax;         // nullptr: no winners
  int argmax_stride;
  int* status;
};

struct SharedCtl {
  unsigned long long a_full, a_empty;
  unsigned long long b_full[STAGES], b_empty[STAGES];
  unsigned long long acc_full[ACCS], acc_empty[ACCS];
  unsigned long long epi_sync[2];
  // candidates of the set without a document's last piece, on their way to the other.  It can be three pieces ahead, so two exchanges.
  unsigned long long x_full[4][4];  // by exchange and quadrant of rows
  uint32_t tmem_base;
  WaitCtl wait;           // (its progress: a scan of a document goes on)
  SplitParams params;     // for `products`
  // A slot is written again four pieces (query tiles) later.  By then the MMAs of the piece two behind it have completed, for the
  // cutters waited for its stage; they had taken the accumulator that the epilogue of this piece gave back after its last look here.
  alignas(16) float col_mul[RING][PIECE], col_add[RING][PIECE];  // 0 or, for columns that are no valid token, -inf
  // of the counted rows that a warp cut, with their multipliers: the largest size (infinity: one does not fit) and the largest sum of magnitudes
  alignas(16) float2 piece_size[RING][CUT_WARPS];
  float q_inv[RING][TILE_M];
  float2 q_size[RING][TILE_M];
  float2 x_size[4][4];
  int4 x_row[4][TILE_M];          // largest p~, at, at2, bits
  float emit[2][2][TILE_M];
};

__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  return wait_bar_all(bar, parity, &ctl->wait, status);
}

// The units of a CTA: unit = tile * n_d + document.
struct Units {
  int left, tile, doc;  // (a CTA's share of the scores fits an int)
  __device__ __forceinline__ Units(const SplitParams& P) {
    const long long n = (long long)P.n_tiles * P.n_d, u = n * blockIdx.x / gridDim.x;
    left = (int)(n * (blockIdx.x + 1) / gridDim.x - u);
    tile = (int)(u / P.n_d);
    doc = (int)(u - (long long)tile * P.n_d);
  }
  __device__ __forceinline__ bool more() const { return left > 0; }
  __device__ __forceinline__ void next(const SplitParams& P) {
    --left;
    if (++doc == P.n_d) {
      doc = 0;
      ++tile;
    }
  }
};
__device__ __forceinline__ int doc_length(const SplitParams& P, int doc, long long& row0, int* status) {
  int len;
  seq_bounds(P.d, doc, row0, len, status);
  return len;
}

struct Row8 {  // a lane's eight features of a row
  float4 a, b;
};
__device__ __forceinline__ Row8 load_row8(const float* p, bool on0, bool on1) {
  Row8 r;
  r.a = r.b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (on0) r.a = __ldg(reinterpret_cast<const float4*>(p));
  if (on1) r.b = __ldg(reinterpret_cast<const float4*>(p + 4));
  return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// Cuts a row that a half-warp holds and stores its three parts at `dst` (+ 1, 2 strides).  Returns the row's size 2^e: 0 for a row of zeros,
// infinity for one that does not fit.
__device__ __forceinline__ float cut_row(const Row8& r, unsigned char* dst, int part_stride) {
  const float x[8] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w};
  // (as bit patterns of magnitudes: NaN lies above infinity)
  unsigned top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(x[i]) & 0x7fffffffu);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  const unsigned ex = top >> 23;  // biased exponent of the largest magnitude
  const bool fits = top == 0 || (ex >= 87 && ex <= 177);
  // adding and taking away 1.5 * 2^(e + 16) rounds to multiples of 2^(e - 7)
  const float m0 = __uint_as_float(((fits ? ex : 127u) + 16u) << 23 | 0x400000u), m1 = m0 * 0x1p-8f;
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a0[2], a1[2], a2[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float v = x[2 * i + k];
      a0[k] = __fsub_rn(__fadd_rn(v, m0), m0);
      const float rest = __fsub_rn(v, a0[k]);
      a1[k] = __fsub_rn(__fadd_rn(rest, m1), m1);
      a2[k] = __fsub_rn(rest, a1[k]);
    }
    w[0][i] = pack_bf16(a0[0], a0[1]);
    w[1][i] = pack_bf16(a1[0], a1[1]);
    w[2][i] = pack_bf16(a2[0], a2[1]);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(dst + p * part_stride) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  return top == 0 ? 0.f : fits ? __uint_as_float(ex << 23) : INFINITY;
}

__device__ __forceinline__ float dot8(const Row8& x, const Row8& y) {
  float s = x.a.x * y.a.x, t = x.a.y * y.a.y;
  s = fmaf(x.a.z, y.a.z, s);
  t = fmaf(x.a.w, y.a.w, t);
  s = fmaf(x.b.x, y.b.x, s);
  t = fmaf(x.b.y, y.b.y, t);
  s = fmaf(x.b.z, y.b.z, s);
  return s + fmaf(x.b.w, y.b.w, t);
}
__device__ __forceinline__ float squares8(const Row8& x) {
  const float s = fmaf(x.b.z, x.b.z, fmaf(x.b.x, x.b.x, fmaf(x.a.z, x.a.z, x.a.x * x.a.x)));
  return s + fmaf(x.b.w, x.b.w, fmaf(x.b.y, x.b.y, fmaf(x.a.w, x.a.w, x.a.y * x.a.y)));
}
__device__ __forceinline__ float magnitudes8(const Row8& x) {
  return ((fabsf(x.a.x) + fabsf(x.a.y)) + (fabsf(x.a.z) + fabsf(x.a.w))) + ((fabsf(x.b.x) + fabsf(x.b.y)) + (fabsf(x.b.z) + fabsf(x.b.w)));
}
// Sums of four values over a half-warp, with the order of a sum over lanes 8, 4, 2 and 1 apart: lane hl gets that of value 2 (hl >> 3) + (hl >> 2 & 1).
__device__ __forceinline__ float half_sums4(float a, float b, float c, float d, int lane) {
  const bool h8 = lane & 8, h4 = lane & 4;
  const float x0 = (h8 ? c : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : c, 8);
  const float x1 = (h8 ? d : b) + __shfl_xor_sync(0xffffffffu, h8 ? b : d, 8);
  float t = (h4 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, h4 ? x0 : x1, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  return t;
}

__device__ __forceinline__ void better(float p, int i, float& best, int& who) {
  if (i >= 0 && (p > best || (p == best && i < who))) {
    best = p;
    who = i;
  }
}
// A document in memory, and what its tokens' products are multiplied by: NaN where a token does not count.
struct Document {
  const float* rows;
  const unsigned char* mask;
  const float* scale;
  long long pitch;
  float scalar, eps;  // eps < 0: no norms
  int dim;
  __device__ __forceinline__ Document(const SplitParams& P, long long row0)
      : rows(static_cast<const float*>(P.d.data) + row0 * P.d.row_stride), mask(P.d.mask ? P.d.mask + row0 : nullptr), scale(P.d.scale ? P.d.scale + row0 : nullptr),
        pitch(P.d.row_stride), scalar(P.d.scale_scalar), eps(P.norm_d ? P.eps : -1.f), dim(P.dim) {}
  __device__ __forceinline__ float scaled(int t) const {
    const float f = scale ? scalar * scale[t] : scalar;
    return mask && !mask[t] ? __int_as_float(0x7fffffff) : f;
  }
  __device__ __forceinline__ float normed(float f, float ss) const { return eps >= 0.f ? f * inv_norm(ss, eps) : f; }
};

// The best of all tokens of a document, in fp32, for the rows of a warp that are set in `rows`: four rows at a time, held in registers, against four
// tokens per step, a half-warp per token.  A lane gets its row's largest product and whose it is, < 0: no token counts, or every product is a NaN
// or -inf.  The sums are those of `products`.
__device__ __noinline__ int2 whole_document(const Document& doc, unsigned rows, const float* q_tile, long long q_off, int len, int* progress) {
  const int lane = threadIdx.x & 31, hl = lane & 15, half = lane >> 4;
  const Document D = doc;
  const bool on0 = hl * 8 < D.dim, on1 = hl * 8 + 4 < D.dim;
  const float* d_lane = D.rows + (on0 ? hl * 8 : 0);
  q_tile += on0 ? hl * 8 : 0;
  int2 mine = make_int2(0, 0);
  while (rows) {
    const unsigned first = rows;  // the four rows: its lowest bits (fewer: the last again)
    Row8 q[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      q[r] = load_row8(q_tile + __shfl_sync(0xffffffffu, q_off, __ffs(rows) - 1), on0, on1);
      if (r == 3 || (rows & (rows - 1))) rows &= rows - 1;
    }
    float best = -INFINITY;  // of row hl >> 2 and this lane's tokens
    int who = -1;
#pragma unroll 1
    for (int t = 0; t < len; t += 4) {
      const int tok = t + 2 * half + (hl >> 1 & 1);
      const Row8 x = load_row8(d_lane + min(t + 2 * half, len - 1) * D.pitch, on0, on1), y = load_row8(d_lane + min(t + 2 * half + 1, len - 1) * D.pitch, on0, on1);
      const float f = D.scaled(min(tok, len - 1));
      float v[8];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        v[2 * r] = dot8(q[r], x);
        v[2 * r + 1] = dot8(q[r], y);
      }
      const float sx = squares8(x), sy = squares8(y);
#pragma unroll
      for (int o = 8; o >= 2; o >>= 1) {  // lane hl ends with the sum of value hl >> 1
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < o / 2; ++k) v[k] = (up ? v[k + o / 2] : v[k]) + __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + o / 2], o);
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
      const float ss = __shfl_sync(0xffffffffu, half_sums4(sx, sy, sx, sy, lane), (lane & 16) | (lane & 2) << 1);
      if (tok < len) better(v[0] * D.normed(f, ss), tok, best, who);
      if ((t & 255) == 0 && lane == 0) atomicAdd(progress, 1);
    }
#pragma unroll
    for (int o = 2; o <= 16; o <<= 3) better(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, who, o), best, who);
    unsigned left = first;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float b = __shfl_sync(0xffffffffu, best, r * 4);
      const int i = __shfl_sync(0xffffffffu, who, r * 4);
      if (left && lane == __ffs(left) - 1) mine = make_int2(__float_as_int(b), i);
      left &= left - 1;
    }
  }
  return mine;
}

// Products in fp32 for the rows of a warp that need them (`what`): a lane gives its row's candidates and gets their largest and who it is.
// (Not inlined: its registers would cost the epilogue's loop over the columns its own.)
enum Need { NOTHING, ONE, MANY, ALL };
__device__ __noinline__ int2 products(SharedCtl* ctl, int what, int tile, int doc, int len, int at, int at2, unsigned bits, int row) {
  const SplitParams& P = ctl->params;
  long long drow0;
  doc_length(P, doc, drow0, nullptr);
  const Document D(P, drow0);
  const int lane = row & 31, hl = lane & 15, ml = P.q.max_len;
  const bool on0 = hl * 8 < D.dim, on1 = hl * 8 + 4 < D.dim;
  const long long pitch = D.pitch, q_stride = P.q.row_stride;
  const float* d_lane = D.rows + (on0 ? hl * 8 : 0);
  const float* q_tile = static_cast<const float*>(P.q.data) + (long long)tile * P.q_per_tile * P.q.seq_stride * q_stride;
  const long long q_off = ((row / ml) * P.q.seq_stride + row % ml) * q_stride;  // of the lane's row in the tile
  const float* q_lane = q_tile + (on0 ? hl * 8 : 0);
  const int tok = at + __ffs(bits) - 1;
  float r = -INFINITY;
  int ri = -1;
  // one candidate: a row per half-warp, two at a time
  const unsigned ones = __ballot_sync(0xffffffffu, what == ONE);
  float dot = 0.f, ss = 0.f;
#pragma unroll 1
  for (unsigned both = (ones | ones >> 16) & 0xffffu; both;) {
    int i[2];
    i[0] = __ffs(both) - 1;
    both &= both - 1;
    i[1] = both ? __ffs(both) - 1 : i[0];
    both &= both - 1;
    Row8 q[2], d[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int from = (lane & 16) | i[k];
      const bool on = ones >> from & 1;
      q[k] = load_row8(q_lane + __shfl_sync(0xffffffffu, q_off, from), on && on0, on && on1);
      d[k] = load_row8(d_lane + __shfl_sync(0xffffffffu, tok, from) * pitch, on && on0, on && on1);
    }
    const float s = half_sums4(dot8(q[0], d[0]), squares8(d[0]), dot8(q[1], d[1]), squares8(d[1]), lane);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float x = __shfl_sync(0xffffffffu, s, (lane & 16) | k * 8), y = __shfl_sync(0xffffffffu, s, (lane & 16) | k * 8 | 4);
      if (hl == i[k]) {
        dot = x;
        ss = y;
      }
    }
  }
  if (what == ONE) {
    r = dot * D.normed(D.scaled(tok), ss);
    ri = tok;
  }
  // several: row by row, four candidates at a time
  for (unsigned rows = __ballot_sync(0xffffffffu, what == MANY); rows; rows &= rows - 1) {
    const int from = __ffs(rows) - 1, a0 = __shfl_sync(0xffffffffu, at, from), a1 = __shfl_sync(0xffffffffu, at2, from) - 16;
    const Row8 q = load_row8(q_lane + __shfl_sync(0xffffffffu, q_off, from), on0, on1);
    float best = -INFINITY;
    int who = -1;
#pragma unroll 1
    for (unsigned left = __shfl_sync(0xffffffffu, bits, from); left;) {
      int t[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int b = __ffs(left) - 1;
        t[k] = b < 0 ? t[0] : b + (b < 16 ? a0 : a1);
        left &= left - 1;
      }
      const int ta = lane & 16 ? t[2] : t[0], tb = lane & 16 ? t[3] : t[1], mine = lane & 8 ? tb : ta;
      const float f = D.scaled(mine);
      const Row8 x = load_row8(d_lane + ta * pitch, on0, on1), y = load_row8(d_lane + tb * pitch, on0, on1);
      const float s = half_sums4(dot8(q, x), squares8(x), dot8(q, y), squares8(y), lane);
      const float p = __shfl_sync(0xffffffffu, s, lane & 24), y2 = __shfl_sync(0xffffffffu, s, (lane & 24) | 4);
      better(p * D.normed(f, y2), mine, best, who);
    }
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) better(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, who, o), best, who);
    if (lane == from) {
      r = best;
      ri = who;
    }
  }
  const unsigned alls = __ballot_sync(0xffffffffu, what == ALL);
  if (alls) {
    const int2 x = whole_document(D, alls, q_tile, q_off, len, const_cast<int*>(&ctl->wait.progress));
    if (what == ALL) {
      r = __int_as_float(x.x);
      ri = x.y;
    }
  }
  return make_int2(__float_as_int(r), ri);
}

template <bool WINNERS>
__global__ void __launch_bounds__(NUM_THREADS, 1) fwd_split_kernel(const __grid_constant__ SplitParams P) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  unsigned char* a_smem = smem;                           // [3 parts][2 slabs][128 rows][128 B]
  unsigned char* b_smem = smem + PARTS * A_PART;          // [stages][2 slabs][3 parts][64 rows][128 B]
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(b_smem + STAGES * B_STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(smem_u32(&ctl->a_full), CUT_WARPS);
    mbar_init(smem_u32(&ctl->a_empty), 1);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&ctl->b_full[i]), CUT_WARPS);
      mbar_init(smem_u32(&ctl->b_empty[i]), 1);
    }
    for (int i = 0; i < ACCS; ++i) {
      mbar_init(smem_u32(&ctl->acc_full[i]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[i]), 4);
    }
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ctl->epi_sync[i]), 4);
    for (int i = 0; i < 16; ++i) mbar_init(smem_u32(&ctl->x_full[i >> 2][i & 3]), 1);
    ctl->wait.init();
    ctl->params = P;
    fence_barrier_init();
  }
  if (warp == ISSUE_WARP) {
    tmem_alloc(smem_u32(&ctl->tmem_base), ACCS * ACC_COLS);
    tmem_relinquish();
  }
  // Launched with programmatic stream serialisation: the set-up above overlaps the kernel in front, nothing below may.
  griddep_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  Units w(P);

  if (warp == ISSUE_WARP) {
    // =========================== MMA issuer ===========================
    const bool issue = elect_one();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const uint32_t a0 = (uint32_t)smem_desc_sw128(smem_u32(a_smem)), b0 = (uint32_t)smem_desc_sw128(smem_u32(b_smem));
    const int k_steps = (P.dim + 15) >> 4;
    uint32_t n = 0, n_tile = 0;  // pieces, query tiles so far
    int cur = -1;
    bool ok = true;
    for (; ok && w.more(); w.next(P)) {
      long long row0;
      const int len = doc_length(P, w.doc, row0, nullptr);
      if (w.tile != cur) {
        cur = w.tile;
        ok = wait_bar(&ctl->a_full, n_tile++ & 1, ctl, P.status);
      }
      const bool tile_ends = w.left == 1 || w.doc + 1 == P.n_d;
      for (int c0 = 0; ok && (c0 == 0 || c0 < len); c0 += PIECE, ++n) {
        const uint32_t st = n % STAGES, acc = n % ACCS;
        ok = wait_bar(&ctl->acc_empty[acc], ((n / ACCS) & 1) ^ 1, ctl, P.status) && wait_bar(&ctl->b_full[st], (n / STAGES) & 1, ctl, P.status);
        if (!ok) break;
        tc_fence_after();
        if (issue) {
          const uint32_t d = tmem_base + acc * ACC_COLS, b = b0 + st * (B_STAGE >> 4);
          // part i of A times parts j .. j + n - 1 of B, into accumulators `to` and on
          auto product = [&](int i, int j, int n, int to, bool first) {
            const uint32_t idesc = instr_desc(1, n * PIECE);
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (k < k_steps)
                tc_mma<false>(d + to * PIECE, a0 + i * (A_PART >> 4) + (k & 3) * 2 + (k >> 2) * (A_SLAB >> 4),
                              b + j * (B_PART >> 4) + (k & 3) * 2 + (k >> 2) * (B_SLAB >> 4), desc_hi, idesc, first && k == 0 ? 0u : 1u);
          };
          product(0, 0, 3, 0, true);
          product(1, 0, 2, 1, false);
          product(1, 2, 1, 2, false);
          product(2, 0, 1, 2, false);
          product(2, 1, 1, 2, false);
          tc_commit(smem_u32(&ctl->b_empty[st]));
          tc_commit(smem_u32(&ctl->acc_full[acc]));
          if (tile_ends && c0 + PIECE >= len) tc_commit(smem_u32(&ctl->a_empty));
        }
        __syncwarp();
      }
    }
  } else if (warp < EPI_WARPS) {
    // =========================== epilogue ===========================
    const int set = warp >> 2, quad = warp & 3, row = quad * 32 + lane;
    bool ok = true;
    uint32_t n = 0, n_tile = 0, n_sync = 0, n_x = 0;
    int cur = -1;
    const int ml = P.q.max_len;
    const int my_slot = row / ml, my_s = row - my_slot * ml;
    bool have = false, counts = false;
    float qf = 0.f;
    for (; ok && w.more(); w.next(P)) {
      long long drow0;
      const int len = doc_length(P, w.doc, drow0, tid == 0 ? P.status : nullptr);
      if (w.tile != cur) {
        const int q0 = w.tile * P.q_per_tile, nq = min(P.q_per_tile, P.n_q - q0);
        cur = w.tile;
        ++n_tile;
        have = my_slot < nq;
        counts = false;
        if (have) {
          long long r0;
          int ql;
          seq_bounds(P.q, q0 + my_slot, r0, ql, P.status);
          if (WINNERS && ql > P.argmax_stride) {
            if (P.status) atomicOr(P.status, LIK_DEV_ARGMAX_STRIDE);
            ql = P.argmax_stride;
          }
          have = my_s < ql;
          if (have) {
            counts = row_valid(P.q, r0 + my_s);
            qf = row_factor(P.q, r0 + my_s);
          }
        }
      }
      const uint32_t ts = (n_tile - 1) % RING;
      const bool any = __any_sync(0xffffffffu, have);
      float r = -FLT_MAX, f = 0.f;  // the largest p~
      float2 q_size = make_float2(0.f, 0.f), d_size = make_float2(0.f, 0.f);
      int at = 0, at2 = NO_MORE;
      unsigned bits = 0;
      // twice the bound for this row and the document so far
      auto bounds = [&]() { return fmaf(q_size.x, fmaf(0x1.4p-24f, d_size.y, (float)P.dim * 0x1p-28f * d_size.x), q_size.y * (0x1.4p-24f * d_size.x)); };
      const int pieces = max(1, (len + PIECE - 1) / PIECE);
      const bool mine = ((n + pieces - 1) & 1) == set;  // the document's last piece
      for (int p = 0; p < pieces; ++p, ++n) {
        if ((n & 1) != set) continue;
        const uint32_t acc = n % ACCS, slot = n % RING;
        const int c0 = p * PIECE;
        ok = wait_bar(&ctl->acc_full[acc], (n / ACCS) & 1, ctl, P.status);
        if (!ok) break;
        tc_fence_after();
        const int cols = min(PIECE, len - c0);
#pragma unroll
        for (int i = 0; i < CUT_WARPS; i += 2) {
          const float4 x = *reinterpret_cast<const float4*>(&ctl->piece_size[slot][i]);
          d_size.x = max3(d_size.x, x.x, x.z);
          d_size.y = max3(d_size.y, x.y, x.w);
        }
        if (any) {
          q_size = ctl->q_size[ts][row];
          const float both = bounds();
#pragma unroll 1
          for (int c = 0; c < cols; c += 16) {
            float v[16], p[16];
            const uint32_t t = tmem_base + ((uint32_t)(quad * 32) << 16) + acc * ACC_COLS + c;
            auto ld16 = [](uint32_t addr, float (&x)[16]) {
              asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                           : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]), "=f"(x[8]), "=f"(x[9]),
                             "=f"(x[10]), "=f"(x[11]), "=f"(x[12]), "=f"(x[13]), "=f"(x[14]), "=f"(x[15])
                           : "r"(addr)
                           : "memory");
            };
            auto held16 = [](float (&x)[16]) {  // no use of the values ahead of the wait
              asm volatile("" : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3]), "+f"(x[4]), "+f"(x[5]), "+f"(x[6]), "+f"(x[7]), "+f"(x[8]), "+f"(x[9]),
                                "+f"(x[10]), "+f"(x[11]), "+f"(x[12]), "+f"(x[13]), "+f"(x[14]), "+f"(x[15]));
            };
            ld16(t + PIECE, v);
            ld16(t + 2 * PIECE, p);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            held16(v);
            held16(p);
#pragma unroll
            for (int i = 0; i < 16; ++i) p[i] += v[i];
            ld16(t, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            held16(v);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 mul = *reinterpret_cast<const float4*>(&ctl->col_mul[slot][c + i]), add = *reinterpret_cast<const float4*>(&ctl->col_add[slot][c + i]);
              // (a NaN beats nothing; columns that are no valid token end as -inf or NaN)
              v[i] = fmaf(v[i] + p[i], mul.x, add.x);
              v[i + 1] = fmaf(v[i + 1] + p[i + 1], mul.y, add.y);
              v[i + 2] = fmaf(v[i + 2] + p[i + 2], mul.z, add.z);
              v[i + 3] = fmaf(v[i + 3] + p[i + 3], mul.w, add.w);
            }
            const float m = fmaxf(max3(max3(v[0], v[1], v[2]), max3(v[3], v[4], v[5]), max3(v[6], v[7], v[8])),
                                  max3(max3(v[9], v[10], v[11]), max3(v[12], v[13], v[14]), v[15]));
            const float gap = fmaf(fabsf(m) + fabsf(r), 0x1p-22f, both);
            const bool candidate = m > r - gap;
            if (__any_sync(0xffffffffu, candidate)) {
              const float least = m - fmaf(fabsf(m), 0x1p-21f, both);
              unsigned near = 0;
#pragma unroll
              for (int i = 0; i < 16; ++i) near |= v[i] >= least ? 1u << i : 0u;
              if (m > r + gap) {
                at = c0 + c;
                at2 = NO_MORE;
                bits = near;
              } else if (candidate) {
                at2 = at2 == NO_MORE ? c0 + c : WHOLE_DOC;
                bits |= near << 16;
              }
            }
            r = fmaxf(r, m);
          }
        }
        // (what the tile's slot holds is looked at before the accumulator goes back)
        if (counts) f = P.norm_q ? qf * ctl->q_inv[ts][row] : qf;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->acc_empty[acc]));
      }
      if (!ok) break;
      if (pieces > 1) {
        const uint32_t x = n_x % 4;
        if (!mine) {
          ctl->x_row[x][row] = make_int4(__float_as_int(r), at, at2, (int)bits);
          if (lane == 0) ctl->x_size[x][quad] = d_size;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl->x_full[x][quad]));
        } else {
          ok = wait_bar(&ctl->x_full[x][quad], (n_x / 4) & 1, ctl, P.status);
          if (!ok) break;
          const int4 o = ctl->x_row[x][row];
          const float2 o_size = ctl->x_size[x][quad];
          d_size = make_float2(fmaxf(d_size.x, o_size.x), fmaxf(d_size.y, o_size.y));
          if (o.w) {
            const float xr = __int_as_float(o.x), gap = fmaf(fabsf(xr) + fabsf(r), 0x1p-22f, bounds());
            if (!bits || xr > r + gap || (xr == r && gap == 0.f && o.y < at)) {
              r = xr;
              at = o.y;
              at2 = o.z;
              bits = (unsigned)o.w;
            } else if (xr > r - gap) {
              at2 = at2 == NO_MORE && o.z == NO_MORE ? o.y : WHOLE_DOC;
              bits |= (unsigned)o.w << 16;
              r = fmaxf(r, xr);
            }
          }
        }
        ++n_x;
      }
      if (!mine) continue;
      int ri = -1;
      {
        const float both = bounds();  // 0: a row of zeros on either side; infinity, NaN: there is no bound
        if (bits) ri = at + __ffs(bits) - 1;
        const bool will_do = bits && both < INFINITY && both <= fabsf(r) * (fmaxf(4.f, (float)P.dim * 0.25f) * 0x1p-23f);  // r is the product as it is
        const bool live = WINNERS ? have : counts && !will_do;
        if (!bits) r = -INFINITY;
        int what = NOTHING;
        if (live && (at2 == WHOLE_DOC || !(both < INFINITY))) what = ALL;
        else if (live && both != 0.f && (bits & (bits - 1))) what = MANY;
        else if (counts && !will_do && both != 0.f && bits) what = ONE;
        if (__any_sync(0xffffffffu, what != NOTHING)) {
          const int2 x = products(ctl, what, w.tile, w.doc, len, at, at2, bits, row);
          if (what != NOTHING) {
            if (!will_do) r = __int_as_float(x.x);
            ri = x.y;
          }
        }
      }
      const float val = counts && r != -INFINITY ? r * f : 0.f;
      const int q0 = w.tile * P.q_per_tile, nq = min(P.q_per_tile, P.n_q - q0);
      if (WINNERS && my_slot < nq) {
        int* out = P.argmax + ((long long)(q0 + my_slot) * P.n_d + w.doc) * P.argmax_stride;
        for (int i = my_s; i < P.argmax_stride; i += ml) out[i] = have && i == my_s ? ri : -1;
      }
      if (ml == 32) {  // a query per warp
        const float sum = warp_sum(val);
        if (lane == 0 && quad < nq) P.scores[(long long)(q0 + quad) * P.n_d + w.doc] = sum;
      } else {
        float* e = ctl->emit[set][n_sync & 1];
        e[row] = val;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->epi_sync[set]));
        ok = wait_bar(&ctl->epi_sync[set], n_sync++ & 1, ctl, P.status);
        if (!ok) break;
        for (int q = quad; q < nq; q += 4) {
          float sum = 0.f;
          for (int i = lane; i < ml; i += 32) sum += e[q * ml + i];
          sum = warp_sum(sum);
          if (lane == 0) P.scores[(long long)(q0 + q) * P.n_d + w.doc] = sum;
        }
      }
    }
  } else if (warp >= CUT_WARP0) {
    // =========================== cutters ===========================
    const int cw = warp - CUT_WARP0, hw = cw * 2 + (lane >> 4), hl = lane & 15;
    const bool on0 = hl * 8 < P.dim, on1 = hl * 8 + 4 < P.dim;
    const float* dbase = static_cast<const float*>(P.d.data) + (on0 ? hl * 8 : 0);
    // the lane's sixteen bytes of row `row` of a part in slabs of `rows` rows
    auto place = [&](unsigned char* part, int row, int slab_bytes) { return part + (hl >> 3) * slab_bytes + row * ROW_BYTES + (((hl & 7) ^ (row & 7)) << 4); };
    uint32_t n = 0, n_tile = 0;
    int cur = -1;
    bool ok = true;
    const int r_lo = hw * 2;  // this half-warp's rows of a piece: r_lo, r_lo + 1
    Row8 nx[2];
    float nx_mul = 0.f;  // multiplier of row r_lo + (hl >> 3); NaN: the token does not count
    auto load_piece = [&](long long row0, int len, int c0) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c = c0 + r_lo + i;
        const bool on = c < len;
        nx[i] = load_row8(dbase + (row0 + (on ? c : 0)) * P.d.row_stride, on && on0, on && on1);
      }
      const int c = c0 + r_lo + (hl >> 3);
      nx_mul = __int_as_float(0x7fffffff);
      if (c < len && row_valid(P.d, row0 + c)) nx_mul = row_factor(P.d, row0 + c);
    };
    long long row0 = 0;
    int len = 0;
    if (w.more()) {
      len = doc_length(P, w.doc, row0, nullptr);
      load_piece(row0, len, 0);
    }
    while (ok && w.more()) {
      if (w.tile != cur) {
        cur = w.tile;
        const uint32_t ts = n_tile % RING;
        if (n_tile > 0) ok = wait_bar(&ctl->a_empty, (n_tile - 1) & 1, ctl, P.status);  // no MMA reads the old tile any more
        if (!ok) break;
        ++n_tile;
        const int q0 = w.tile * P.q_per_tile, nq = min(P.q_per_tile, P.n_q - q0);
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          const int row = hw * 4 + i, slot = row / P.q.max_len, s = row - slot * P.q.max_len;
          Row8 r;
          r.a = r.b = make_float4(0.f, 0.f, 0.f, 0.f);
          bool used = false;
          if (slot < nq) {
            long long r0;
            int ql;
            seq_bounds(P.q, q0 + slot, r0, ql, nullptr);
            if (s < ql) {
              r = load_row8(static_cast<const float*>(P.q.data) + (r0 + s) * P.q.row_stride + (on0 ? hl * 8 : 0), on0, on1);
              used = row_valid(P.q, r0 + s);
            }
          }
          const float size = cut_row(r, place(a_smem, row, A_SLAB), A_PART);
          const float sums = half_sums4(P.norm_q ? squares8(r) : 0.f, magnitudes8(r), 0.f, 0.f, lane), sum = __shfl_xor_sync(0xffffffffu, sums, 4);
          if (hl == 0) {
            ctl->q_inv[ts][row] = P.norm_q ? inv_norm(sums, P.eps) : 1.f;
            // (what padding holds must send nobody through the document)
            ctl->q_size[ts][row] = used || size < INFINITY ? make_float2(size, sum) : make_float2(0.f, 0.f);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->a_full));
      }
      for (int c0 = 0; ok && (c0 == 0 || c0 < len); ++n) {
        const uint32_t st = n % STAGES, slot = n % RING;
        const Row8 x0 = nx[0], x1 = nx[1];
        float mul = nx_mul;
        // the next piece's rows are on their way while these are cut
        c0 += PIECE;
        const bool doc_done = c0 >= len;
        if (doc_done) {
          w.next(P);
          if (w.more()) {
            len = doc_length(P, w.doc, row0, nullptr);
            load_piece(row0, len, 0);
          }
        } else {
          load_piece(row0, len, c0);
        }
        ok = wait_bar(&ctl->b_empty[st], ((n / STAGES) & 1) ^ 1, ctl, P.status);
        if (!ok) break;
        unsigned char* stage = b_smem + st * B_STAGE;
        const float size0 = cut_row(x0, place(stage, r_lo, B_SLAB), B_PART), size1 = cut_row(x1, place(stage, r_lo + 1, B_SLAB), B_PART);
        const float sums = half_sums4(P.norm_d ? squares8(x0) : 0.f, magnitudes8(x0), P.norm_d ? squares8(x1) : 0.f, magnitudes8(x1), lane);
        const float sum = __shfl_xor_sync(0xffffffffu, sums, 4);
        unsigned size = 0, most = 0;
        if ((hl & 7) == 0) {  // a lane per row
          const bool counts = mul == mul;
          if (!counts) mul = 1.f;
          if (P.norm_d) mul *= inv_norm(sums, P.eps);
          ctl->col_mul[slot][r_lo + (hl >> 3)] = mul;
          ctl->col_add[slot][r_lo + (hl >> 3)] = counts ? 0.f : -INFINITY;
          if (counts) {  // (tokens that do not count may hold anything)
            const float x = (hl ? size1 : size0) * fabsf(mul), y = sum * fabsf(mul);
            size = __float_as_uint(x < 0x1p60f ? (x > 0.f ? fmaxf(x, 0x1p-70f) : 0.f) : INFINITY);
            most = __float_as_uint(y < 0x1p60f ? (y > 0.f ? fmaxf(y, 0x1p-70f) : 0.f) : INFINITY);
          }
        }
        size = __reduce_max_sync(0xffffffffu, size);
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) ctl->piece_size[slot][cw] = make_float2(__uint_as_float(size), __uint_as_float(most));
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->b_full[st]));
        if (doc_done) {
          ++n;
          break;
        }
      }
    }
  }

  // ---- teardown (also reached when aborting: every wait above is bounded) ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUE_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACCS * ACC_COLS);
  }
}

constexpr size_t SMEM_BYTES = (size_t)PARTS * A_PART + STAGES * B_STAGE + sizeof(SharedCtl) + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "a block's shared memory");

// The wait of this kernel and of the compressed-index kernel, alone: a warp waits on a barrier that nothing arrives at, first with nobody
// busy, then beside a warp that counts its progress for three limits and stops.
// result[3 * w + ...] = lanes that were told to go on (0: all gave up), the abort flag, cycles spent by the slowest lane.
__global__ void all_lanes_wait_probe_kernel(long long limit, int* status, int* result) {
  __shared__ unsigned long long bar;
  __shared__ WaitCtl ctl;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    fence_barrier_init();
  }
  for (int w = 0; w < 2; ++w) {
    if (threadIdx.x == 0) ctl.init(limit);
    __syncthreads();
    const long long t0 = clock64();
    if (threadIdx.x < 32) {
      const bool got = wait_bar_all(&bar, 0, &ctl, status);
      const long long dt = clock64() - t0;
      const int lanes = __popc(__ballot_sync(0xffffffffu, got));
      const unsigned cycles = __reduce_max_sync(0xffffffffu, dt > 0x7fffffffll ? 0x7fffffffu : (unsigned)dt);
      if (threadIdx.x == 0) {
        result[3 * w] = lanes;
        result[3 * w + 1] = ctl.abort_flag;
        result[3 * w + 2] = (int)cycles;
      }
    } else if (w == 1 && threadIdx.x == 32) {
      while (clock64() - t0 < 3 * limit) atomicAdd(const_cast<int*>(&ctl.progress), 1);
    }
    __syncthreads();
  }
}

}  // namespace

bool fwd_generic_shares(long long n_q, long long n_d);

// Whether this kernel is the faster one, by what either takes in us: a launch, and a CTA's units of so many tokens here; a launch, and an SM's
// blocks of 32 query tokens (of one query or of two) there.  Measured at 1, 4 and 16 queries of 8 to 128 tokens x 1 to 1000 documents of
// up to 16 to 512, 128 and 32 features wide, by graph replay (here / there): 32 tokens x 100 documents of up to 64 15.5 / 13.4, of 180 19.5 / 23.4, of
// 512 31 / 47; x 1000 of 16 41 / 25; 128 tokens x 8 of 16 19 / 24; 16 x 1000 of 512 426 / 1520; 32 wide: 32 x 1000 of 512 109 / 60, 16 x 256 of 512 101 / 149,
// 16 x 100 of 64 27 / 23.  In 350 calls measured the choice is on average 1 % behind the faster one.
static bool split_pays(const lik_fwd_args& a) {
  const float len = a.d.cu ? (float)a.d.n_rows / a.d.n_seq : (float)a.d.max_len, d = (float)a.dim, sms = (float)sm_count();
  const int per_tile = TILE_M / a.q.max_len;
  const float units = (float)ceil_div(a.q.n_seq, per_tile) * a.d.n_seq / sms;
  const float here = 12.f + fmaxf(1.f, units) * ((len <= 32.f ? 4.f : 3.f) + 0.043f * len);  // (short documents: more products in fp32)
  const bool two = fwd_generic_shares(a.q.n_seq, a.d.n_seq);
  const float blocks = (two ? (float)((a.q.n_seq + 1) / 2) : (float)a.q.n_seq) * a.d.n_seq / sms;
  const float block = two ? 1.2f + 0.019f * d + (0.0063f + 0.0005f * d) * len : 0.4f + 0.006f * d + (0.0036f + 0.00054f * d) * len;
  return here < 7.f + (float)ceil_div(a.q.max_len, 32) * fmaxf(1.f, blocks) * block;
}

// fp32 cross products whose queries fit a tile and whose rows can be read sixteen bytes at a time, where it pays (engine 3: wherever it can).
bool fwd_split_supported(const lik_fwd_args& a) {
  if (a.dtype != LIK_F32 || (a.engine != 0 && a.engine != 3) || a.pairing != LIK_PAIR_CROSS) return false;
  if (a.dim % 4 != 0 || a.dim > 128 || a.q.cu || a.q.max_len < 1 || a.q.max_len > TILE_M) return false;
  if (a.q.n_seq <= 0 || a.d.n_seq <= 0 || a.q.n_rows <= 0 || a.d.n_rows <= 0) return false;
  if (a.q.row_stride % 4 != 0 || a.d.row_stride % 4 != 0 || ((uintptr_t)a.q.data & 15) || ((uintptr_t)a.d.data & 15)) return false;
  return (a.engine == 3 || split_pays(a)) && lik_device_supported() != 0;
}

int launch_fwd_split(const lik_fwd_args& a, float eps, cudaStream_t st) {
  SplitParams P{};
  P.q = make_view(a.q, nullptr);
  P.d = make_view(a.d, nullptr);
  P.n_q = a.q.n_seq;
  P.n_d = a.d.n_seq;
  P.dim = a.dim;
  P.q_per_tile = TILE_M / a.q.max_len;
  P.n_tiles = (int)ceil_div(a.q.n_seq, P.q_per_tile);
  P.norm_q = (a.normalize & LIK_NORM_Q) != 0;
  P.norm_d = (a.normalize & LIK_NORM_D) != 0;
  P.eps = eps;
  P.scores = a.scores;
  P.argmax = a.argmax;
  P.argmax_stride = a.argmax_stride;
  P.status = a.status;
  const long long units = (long long)P.n_tiles * P.n_d;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(units < sm_count() ? units : sm_count()));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (a.argmax) {
    LIK_CUDA_OK((allow_smem<fwd_split_kernel<true>>()));
    LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_split_kernel<true>, P));
  } else {
    LIK_CUDA_OK((allow_smem<fwd_split_kernel<false>>()));
    LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_split_kernel<false>, P));
  }
  ::lik::count_launch();
  return LIK_OK;
}

}  // namespace lik

extern "C" int lik_selftest_all_lanes_wait(int64_t limit_cycles, int32_t* status, int32_t* result, lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(result != nullptr, "result is NULL");
  LIK_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000ll, "limit_cycles outside (0, 2e8]");
  all_lanes_wait_probe_kernel<<<1, 64, 0, (cudaStream_t)stream>>>((long long)limit_cycles, status, result), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}
