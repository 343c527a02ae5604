// Exact fp32 scores on the tensor cores (sm_100a: tcgen05.mma + TMEM): every fp32 row is cut into three bf16 parts on its way into
// shared memory, and six products of parts make a dot product.
//
// The cut.  Let 2^e be the power of two at or below the largest magnitude of a row.  a0 = the row rounded to multiples of 2^(e-7),
// a1 = the rest rounded to multiples of 2^(e-15), a2 = what is left, rounded to bf16: at most 2^(e-25) is lost, a quarter of an ulp of the
// largest element.  The tensor core adds into fp32 but cuts off below (measured: -0.3 ulp on average per 16 products of full bf16
// values, -1.8 over 128), which would shift every score.  Here it has nothing to cut: products a0 b0 are whole multiples of one
// unit, at most 2^16 of it, and 128 of them stay below 2^24; so do those of a0 b1 + a1 b0 of theirs; each has an accumulator
// of its own.  The third, a0 b2 + a1 b1 + a2 b0, is 2^-16 of the first and may be cut.  The three are added in fp32, so a dot product
// is rounded twice where a chain of fused multiply-adds rounds 128 times.
// Rows that this does not fit (infinities, NaN, magnitudes beyond 2^50 or all below 2^-50, whose parts or products could leave fp32's range) are marked, and the epilogue takes
// the dot products of a marked piece or query tile with such a chain itself: rare, slow, and what fwd_generic_kernel gives.
//
// A CTA per SM takes an equal run of (query tile, document) units, tile by tile, and walks a document in pieces of 64 tokens.
// Warp roles (800 threads):
//   warps 0..7   epilogue, a thread per query token: two sets of four warps take the pieces in turn; where a document ends, the set
//                of its last piece gets the other's maxima through shared memory
//   warp 8       issues the MMAs of a piece: six products x one per 16 features
//   warps 9..24  cut the rows of the pieces and, where it changes, of the query tile: a half-warp per row; they take the norms too
// Against fwd_generic_kernel, whose fp32 FMAs bound it (queries of up to 32 tokens, documents a fifth to the whole of the length given):
// 32 x 32 documents of 180 tokens 52 -> 25 us, 1 x 256 of 512 58 -> 40, 64 x 64 of 300 (48-token queries, 96 features) 397 -> 110,
// 64 x 256 of 512 2926 -> 558 (one set of epilogue warps: 781); calls of 8 to 16 documents wait for the host either way (21 us).
// Error of the scores against 64 bits, 2-norm over these shapes: 2.6e-8 to 5.2e-8, the other kernel's 4.1e-8 to 6.4e-8.
// What bounds it: instruction issue (68 % active; the tensor pipe 39 %): every document is cut again for each query tile.
// Every wait is bounded: on expiry the CTA raises LIK_DEV_WAIT_TIMEOUT in the status word, sets a shared abort flag, frees TMEM and
// returns.
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
constexpr int B_SLAB = PIECE * ROW_BYTES, B_PART = 2 * B_SLAB, B_STAGE = PARTS * B_PART;
constexpr int A_SLAB = TILE_M * ROW_BYTES, A_PART = 2 * A_SLAB;
constexpr long long WAIT_LIMIT = 4000000000ll;
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
  // maxima of the set without a document's last piece, on their way to the other.  It can be three pieces ahead, so two exchanges.
  unsigned long long x_full[4][4];  // by exchange and quadrant of rows
  uint32_t tmem_base;
  volatile int abort_flag;
  // A slot is written again four pieces (query tiles) later.  By then the MMAs of the piece two behind it have completed, for the
  // cutters waited for its stage; they had taken the accumulator that the epilogue of this piece gave back after its last look here.
  alignas(16) float col_mul[RING][PIECE], col_add[RING][PIECE];  // 0 or, for columns that are no valid token, -inf
  alignas(16) unsigned char piece_odd[RING][CUT_WARPS];            // the rows that a warp cut do not fit
  float q_inv[RING][TILE_M];
  alignas(16) unsigned char tile_odd[RING][CUT_WARPS];
  float emit[2][2][TILE_M];
  float x_max[4][TILE_M];
  int x_idx[4][TILE_M];
};

__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  const uint32_t b = smem_u32(bar);
  if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
  const long long t0 = clock64();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i)
      if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
    if (clock64() - t0 > WAIT_LIMIT) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
    }
    if (__any_sync(0xffffffffu, ctl->abort_flag != 0)) return false;
  }
}

// The units of a CTA: unit = tile * n_d + document.
struct Units {
  long long u, end;
  int tile, doc;
  __device__ __forceinline__ Units(const SplitParams& P) {
    const long long n = (long long)P.n_tiles * P.n_d;
    u = n * blockIdx.x / gridDim.x;
    end = n * (blockIdx.x + 1) / gridDim.x;
    tile = (int)(u / P.n_d);
    doc = (int)(u - (long long)tile * P.n_d);
  }
  __device__ __forceinline__ bool more() const { return u < end; }
  __device__ __forceinline__ void next(const SplitParams& P) {
    ++u;
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
// Cuts a row that a half-warp holds and stores its three parts at `dst` (+ 1, 2 strides).  Returns whether the row fits; ss: sum of
// squares of the whole row, where wanted.
__device__ __forceinline__ bool cut_row(const Row8& r, unsigned char* dst, int part_stride, bool want_ss, float& ss) {
  const float x[8] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w};
  // (as bit patterns of magnitudes: NaN lies above infinity)
  unsigned top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(x[i]) & 0x7fffffffu);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (want_ss) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      s0 = fmaf(x[i], x[i], s0);
      s1 = fmaf(x[i + 1], x[i + 1], s1);
    }
    ss = s0 + s1;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  const unsigned ex = top >> 23;  // biased exponent of the largest magnitude
  const bool fits = top == 0 || (ex >= 77 && ex <= 177);
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
  return fits;
}

// The dot product as fwd_generic_kernel takes it.
__device__ __noinline__ float chain_dot(const float* q, const float* d, int dim) {
  float acc = 0.f;
  for (int k = 0; k < dim; ++k) acc = fmaf(__ldg(q + k), __ldg(d + k), acc);
  return acc;
}

template <bool WINNERS>
__global__ void __launch_bounds__(NUM_THREADS, 1) fwd_split_kernel(const SplitParams P) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  unsigned char* a_smem = smem;                           // [3 parts][2 slabs][128 rows][128 B]
  unsigned char* b_smem = smem + PARTS * A_PART;          // [stages][3 parts][2 slabs][64 rows][128 B]
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
    ctl->abort_flag = 0;
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
      const bool tile_ends = w.u + 1 == w.end || w.doc + 1 == P.n_d;
      for (int c0 = 0; ok && (c0 == 0 || c0 < len); c0 += PIECE, ++n) {
        const uint32_t st = n % STAGES, acc = n % ACCS;
        ok = wait_bar(&ctl->acc_empty[acc], ((n / ACCS) & 1) ^ 1, ctl, P.status) && wait_bar(&ctl->b_full[st], (n / STAGES) & 1, ctl, P.status);
        if (!ok) break;
        tc_fence_after();
        if (issue) {
          const int cols = max(16, (min(PIECE, len - c0) + 15) & ~15);
          const uint32_t idesc = instr_desc(1, cols), d = tmem_base + acc * ACC_COLS, b = b0 + st * (B_STAGE >> 4);
          // product of part i of A and part j of B into accumulator i + j
          auto product = [&](int i, int j, bool first) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (k < k_steps)
                tc_mma<false>(d + (i + j) * PIECE, a0 + i * (A_PART >> 4) + (k & 3) * 2 + (k >> 2) * (A_SLAB >> 4),
                              b + j * (B_PART >> 4) + (k & 3) * 2 + (k >> 2) * (B_SLAB >> 4), desc_hi, idesc, first && k == 0 ? 0u : 1u);
          };
          product(0, 0, true);
          product(0, 1, true);
          product(1, 0, false);
          product(0, 2, true);
          product(1, 1, false);
          product(2, 0, false);
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
    uint32_t n = 0, n_tile = 0, n_sync = 0, n_emit = 0, n_x = 0;
    int cur = -1;
    const int ml = P.q.max_len;
    const bool lone = ml == 32;  // a query per warp
    const int my_slot = row / ml, my_s = row - my_slot * ml;
    bool have = false, counts = false;
    float qf = 0.f;
    const float* q_row = nullptr;
    for (; ok && w.more(); w.next(P)) {
      long long drow0;
      const int len = doc_length(P, w.doc, drow0, tid == 0 ? P.status : nullptr);
      const int q0 = w.tile * P.q_per_tile, nq = min(P.q_per_tile, P.n_q - q0);
      if (w.tile != cur) {
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
            q_row = static_cast<const float*>(P.q.data) + (r0 + my_s) * P.q.row_stride;
            counts = row_valid(P.q, r0 + my_s);
            qf = row_factor(P.q, r0 + my_s);
          }
        }
      }
      const uint32_t ts = (n_tile - 1) % RING;
      const bool any = __any_sync(0xffffffffu, have);
      float r = -INFINITY, f = 0.f;
      int ri = -1;
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
        // (sixteen bytes each: any of the pieces' or the tile's rows that do not fit)
        const uint4 po = *reinterpret_cast<const uint4*>(ctl->piece_odd[slot]), to = *reinterpret_cast<const uint4*>(ctl->tile_odd[ts]);
        const bool odd = (po.x | po.y | po.z | po.w | to.x | to.y | to.z | to.w) != 0;
        if (any && !odd) {
#pragma unroll 1
          for (int c = 0; c < cols; c += 16) {
            float v[16], p1[16], p2[16];
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
            ld16(t, v);
            ld16(t + PIECE, p1);
            ld16(t + 2 * PIECE, p2);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            held16(v);
            held16(p1);
            held16(p2);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 mul = *reinterpret_cast<const float4*>(&ctl->col_mul[slot][c + i]), add = *reinterpret_cast<const float4*>(&ctl->col_add[slot][c + i]);
              // (a NaN beats nothing; columns that are no valid token end as -inf or NaN)
              v[i] = fmaf(v[i] + (p1[i] + p2[i]), mul.x, add.x);
              v[i + 1] = fmaf(v[i + 1] + (p1[i + 1] + p2[i + 1]), mul.y, add.y);
              v[i + 2] = fmaf(v[i + 2] + (p1[i + 2] + p2[i + 2]), mul.z, add.z);
              v[i + 3] = fmaf(v[i + 3] + (p1[i + 3] + p2[i + 3]), mul.w, add.w);
            }
            const float m = fmaxf(max3(max3(v[0], v[1], v[2]), max3(v[3], v[4], v[5]), max3(v[6], v[7], v[8])),
                                  max3(max3(v[9], v[10], v[11]), max3(v[12], v[13], v[14]), v[15]));
            if (WINNERS) {
              const bool better = m > r;
              if (__any_sync(0xffffffffu, better)) {  // the first column that has it
                int at = 0;
#pragma unroll
                for (int i = 15; i >= 0; --i) at = v[i] == m ? i : at;
                ri = better ? c0 + c + at : ri;
              }
            }
            r = fmaxf(r, m);
          }
        } else if (odd && have) {
          for (int c = 0; c < cols; ++c) {
            if (ctl->col_add[slot][c] != 0.f) continue;
            const float x = chain_dot(q_row, static_cast<const float*>(P.d.data) + (drow0 + c0 + c) * P.d.row_stride, P.dim) * ctl->col_mul[slot][c];
            if (x > r) {
              r = x;
              ri = c0 + c;
            }
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
          ctl->x_max[x][row] = r;
          if (WINNERS) ctl->x_idx[x][row] = ri;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl->x_full[x][quad]));
        } else {
          ok = wait_bar(&ctl->x_full[x][quad], (n_x / 4) & 1, ctl, P.status);
          if (!ok) break;
          const float xr = ctl->x_max[x][row];
          if (WINNERS) {
            const int xi = ctl->x_idx[x][row];
            if (xr > r || (xr == r && (unsigned)xi < (unsigned)ri)) ri = xi;
          }
          r = fmaxf(r, xr);
        }
        ++n_x;
      }
      if (!mine) continue;
      const float val = counts && r != -INFINITY ? r * f : 0.f;
      if (WINNERS && my_slot < nq) {
        int* out = P.argmax + ((long long)(q0 + my_slot) * P.n_d + w.doc) * P.argmax_stride;
        for (int i = my_s; i < P.argmax_stride; i += ml) out[i] = have && i == my_s ? ri : -1;
      }
      if (lone) {
        const float sum = warp_sum(val);
        if (lane == 0 && quad < nq) P.scores[(long long)(q0 + quad) * P.n_d + w.doc] = sum;
      } else {
        float* e = ctl->emit[set][n_emit++ & 1];
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
    float nx_mul[2], nx_add[2];
    auto load_piece = [&](long long row0, int len, int c0) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c = c0 + r_lo + i;
        const bool on = c < len;
        const long long dr = row0 + (on ? c : 0);
        nx[i] = load_row8(dbase + dr * P.d.row_stride, on && on0, on && on1);
        nx_mul[i] = 1.f;
        nx_add[i] = -INFINITY;
        if (on && row_valid(P.d, dr)) {
          nx_mul[i] = row_factor(P.d, dr);
          nx_add[i] = 0.f;
        }
      }
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
        bool fits = true;
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
              used = row_valid(P.q, r0 + s);  // (what padding holds must not send the tile to the chain)
            }
          }
          float ss = 0.f;
          fits = (cut_row(r, place(a_smem, row, A_SLAB), A_PART, P.norm_q, ss) || !used) && fits;
          if (hl == 0) ctl->q_inv[ts][row] = P.norm_q ? inv_norm(ss, P.eps) : 1.f;
        }
        const bool all = __all_sync(0xffffffffu, fits);
        if (lane == 0) ctl->tile_odd[ts][cw] = all ? 0 : 1;
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->a_full));
      }
      for (int c0 = 0; ok && (c0 == 0 || c0 < len); ++n) {
        const uint32_t st = n % STAGES, slot = n % RING;
        const Row8 x0 = nx[0], x1 = nx[1];
        const float mul0 = nx_mul[0], mul1 = nx_mul[1], add0 = nx_add[0], add1 = nx_add[1];
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
        float ss0 = 0.f, ss1 = 0.f;
        const bool fits0 = cut_row(x0, place(stage, r_lo, B_SLAB), B_PART, P.norm_d, ss0);
        const bool fits1 = cut_row(x1, place(stage, r_lo + 1, B_SLAB), B_PART, P.norm_d, ss1);
        if (hl < 2) {
          const float mul = hl ? mul1 : mul0;
          ctl->col_mul[slot][r_lo + hl] = P.norm_d ? mul * inv_norm(hl ? ss1 : ss0, P.eps) : mul;
          ctl->col_add[slot][r_lo + hl] = hl ? add1 : add0;
        }
        const bool all = __all_sync(0xffffffffu, (fits0 || add0 != 0.f) && (fits1 || add1 != 0.f));  // (tokens that do not count may hold anything)
        if (lane == 0) ctl->piece_odd[slot][cw] = all ? 0 : 1;
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

}  // namespace

// fp32 cross products whose queries fit a tile and whose rows can be read sixteen bytes at a time; no size is too small (8 documents: even).
bool fwd_split_supported(const lik_fwd_args& a) {
  if (a.dtype != LIK_F32 || a.engine != 0 || a.pairing != LIK_PAIR_CROSS) return false;
  if (a.dim % 4 != 0 || a.dim > 128 || a.q.cu || a.q.max_len < 1 || a.q.max_len > TILE_M) return false;
  if (a.q.n_seq <= 0 || a.d.n_seq <= 0 || a.q.n_rows <= 0 || a.d.n_rows <= 0) return false;
  if (a.q.row_stride % 4 != 0 || a.d.row_stride % 4 != 0 || ((uintptr_t)a.q.data & 15) || ((uintptr_t)a.d.data & 15)) return false;
  return lik_device_supported() != 0;
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
