// Scores of a few queries straight from a compressed (PLAID) index, in one kernel (sm_100a: tcgen05.mma + TMEM): tokens are decoded
// into the operand tiles in shared memory, so that no decoded row is ever written to memory and read back.
//
// GEMM view as in lik_fwd_tc.cu: rows = query tokens (A, one resident tile of 128), columns = document tokens (B), K = width.
// A CTA takes a run of consecutive documents, cut so that every CTA has the same number of tokens, and walks their tokens as one
// stream in tiles of 128: a tile may hold the end of one document, several short ones and the start of the next, so that the
// decoders never wait for a ragged end.
//
// Two CTAs per SM.  Warp roles (448 threads):
//   warps 0..3   epilogue: a thread per query token keeps the running maximum over the columns of a document; where it ends, the
//                score is summed and stored or offered to the query's candidate list
//   warp 4       issues the MMAs of a tile: one per 16 features
//   warp 5       walks the documents: leaves, per tile, token and centroid of every column and the list of document segments in a
//                ring of tables, up to eight tiles ahead, and asks L2 for the tokens' residuals
//   warps 6..13  decode: sixteen columns of every tile each, a quarter-warp per token, the next tokens' rows on their way while these
//                are finished
// 25 000 documents of 60..300 tokens, 2 bits, top-10: one query of 32 tokens 574 -> 387 us, four 581 -> 411 (against decoding the
// rows to memory and scoring them from there); 4 bits 575 -> 408, 8 bits (scores) 698 -> 457; 1000 documents of up to 64 tokens 132 -> 65.
// What bounds it: the decoders (361 us without an epilogue): shared-memory wavefronts (the table look-ups) 74 % of the pipe,
// instruction issue 58 %, and their waits for centroid rows out of L2.  Two CTAs per SM, because every role is a chain of dependent
// steps at some ten cycles each: one CTA with sixteen decoder warps took 642 us, its single epilogue warp 4200 cycles per tile.
// Two query tiles per CTA (five to eight queries) were slower than rows in memory: 820 against 650 us.
// Every wait is bounded: on expiry the CTA raises LIK_DEV_WAIT_TIMEOUT in the status word, sets a shared abort flag, frees TMEM and
// returns.
#include <cuda.h>

#include "lik_fwd_tc.cuh"

namespace lik {

namespace {

constexpr int TILE_T = 128;                   // tokens per tile
constexpr int DEC_WARPS = 8, DEC_COLS = TILE_T / DEC_WARPS;
constexpr int DEC_WARP0 = 6, ISSUE_WARP = 4, WALK_WARP = 5;
constexpr int NUM_THREADS = (DEC_WARP0 + DEC_WARPS) * 32;
constexpr int CTAS_PER_SM = 2;
static_assert(DEC_COLS % 8 == 0, "a decoder warp decodes eight tokens at a time");
constexpr int TABLES = 8;                     // ring of tile tables
constexpr int MAX_SEGS = 48;                  // document segments per tile; a tile with more (empty documents) ends early
constexpr int ACCS = 2;                       // accumulators of 128 columns: half of the tensor memory
constexpr int STAGES = 2;
constexpr int GRANULE = 8;                    // a document starts at a multiple of this many columns; its last token fills the gap behind it
constexpr int SEG_ENDS = 1 << 16;             // the document ends with this segment

struct SharedCtl {
  unsigned long long q_full;
  unsigned long long tab_full[TABLES], tab_empty[TABLES];
  unsigned long long b_full[STAGES], b_empty[STAGES];
  unsigned long long acc_full[ACCS], acc_empty[ACCS];
  unsigned long long epi_sync;
  uint32_t tmem_base;
  WaitCtl wait;
  alignas(16) int2 col[TABLES][TILE_T];       // per column: token, centroid
  int2 seg[TABLES][MAX_SEGS];                 // x = document, y = first granule behind the segment | SEG_ENDS
  int n_seg[TABLES];                          // -1: the stream has ended before this tile
  short row_seg[TILE_M], seg_off[TILE_M], seg_len[TILE_M];
  float emit[2][TILE_M];
  int seg_cnt[TILE_M];                     // candidate lists of a fused top-k
  unsigned seg_thr[TILE_M];
  int seg_list[TILE_M];
};

__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  return wait_bar_all(bar, parity, &ctl->wait, status);
}

// First index in [0, n) whose offset is not below x (n: none), 32 places per step.  For ascending x the results ascend, whatever the
// offsets are, so the CTAs' shares are disjoint and complete even where they are not sorted.
__device__ __forceinline__ int lower_bound_warp(const int* __restrict__ cu, int n, long long x, int lane) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32;
    const long long p = (long long)lo + (long long)(lane + 1) * step - 1;
    const bool ge = p >= hi || (long long)__ldg(cu + p) >= x;
    const unsigned m = __ballot_sync(0xffffffffu, ge);
    const int f = m ? __ffs(m) - 1 : 32;
    const long long end = (long long)lo + (long long)(f + 1) * step - 1;
    lo = (int)min((long long)lo + (long long)f * step, (long long)hi);
    hi = (int)min(end, (long long)hi);
  }
  return lo;
}

// One (query, document) score: stored, or offered to the query's candidate list.  Warp-uniform.
__device__ __forceinline__ void emit_score(const TcParams& P, SharedCtl* ctl, int sg, float value, int doc, int lane) {
  if (P.topk.cand_key == nullptr) {
    if (lane == 0) P.scores[(long long)sg * P.n_d + doc] = value;
    return;
  }
  const float key = (P.topk.largest ? value : -value) + 0.f;
  if (ordered_key(key) <= ctl->seg_thr[sg]) return;
  const int cnt = ctl->seg_cnt[sg], list = ctl->seg_list[sg];
  if ((unsigned)cnt >= (unsigned)TOPK_CAP || (unsigned)list >= (unsigned)P.topk.n_lists) {
    if (lane == 0 && P.status) atomicOr(P.status, LIK_DEV_INTERNAL);
    return;
  }
  if (lane == 0) {
    P.topk.cand_key[(long long)list * TOPK_CAP + cnt] = key;
    P.topk.cand_idx[(long long)list * TOPK_CAP + cnt] = doc + P.topk.doc_base;
    ctl->seg_cnt[sg] = cnt + 1;
  }
  __syncwarp();
}
// Between tiles: a list that another tile could fill is cut back to its k best.  (Not where a score arrives: a call there would have the
// tile's maxima saved around it.)
__device__ __forceinline__ void tidy_list(const TcParams& P, SharedCtl* ctl, int sg, int lane) {
  const int cnt = ctl->seg_cnt[sg], list = ctl->seg_list[sg];
  if (cnt <= TOPK_CAP - MAX_SEGS || (unsigned)list >= (unsigned)P.topk.n_lists) return;
  const unsigned thr = topk_compact<true>(P.topk.cand_key + (long long)list * TOPK_CAP, P.topk.cand_idx + (long long)list * TOPK_CAP, P.topk.k, lane, cnt);
  if (lane == 0) {
    ctl->seg_thr[sg] = thr;
    ctl->seg_cnt[sg] = P.topk.k;
  }
  __syncwarp();
}
static_assert(TOPK_CAP - MAX_SEGS >= TOPK_CAP / 2, "a list that was cut back has room for a tile");

constexpr size_t dynamic_smem(int n_slabs) { return (size_t)n_slabs * (TILE_M + STAGES * TILE_T) * SLAB_BYTES_ROW + sizeof(SharedCtl) + 1024; }
// (an SM has 228 KB and takes 1 KB of them per CTA; 512 bytes more and eight-bit indexes, with the largest table, had one CTA per SM)
static_assert(CTAS_PER_SM * (dynamic_smem(2) + PlaidTable<8>::WORDS * sizeof(float) + 1024) <= 228 * 1024, "two CTAs per SM for every index");

// FULL: 128 features
template <bool CF32, bool CBF16, int NBITS, bool FULL>
__global__ void __launch_bounds__(NUM_THREADS, CTAS_PER_SM) fwd_plaid_kernel(const __grid_constant__ CUtensorMap q_map, const TcParams P) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(16) float tab[PlaidTable<NBITS>::WORDS];  // the bucket weights
  // (Rounded up by an offset and not through an integer, so that the compiler sees shared memory behind every pointer: generic loads of
  // it wait in line behind the gathers, a thousand cycles at a time.)
  unsigned char* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  const int q_tile_bytes = P.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const int stage_bytes = P.n_slabs * TILE_T * SLAB_BYTES_ROW;
  unsigned char* q_smem = smem;                        // [n_slabs][128 rows][128 B]
  unsigned char* b_smem = smem + q_tile_bytes;  // [STAGES][n_slabs][128 rows][128 B]
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(b_smem + (size_t)STAGES * stage_bytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // queries of one warp's 32 rows each (lone): warps without rows leave at once; others need all four for a score
  const bool lone = !P.q.lens && P.q.max_len <= 32 && (P.n_q == 1 || (P.q.seq_stride == 32 && P.n_q <= 4));
  const int epi_warps = lone ? P.n_q : 4;

  if (tid == 0) {
    mbar_init(smem_u32(&ctl->q_full), 1);
    for (int i = 0; i < TABLES; ++i) {
      mbar_init(smem_u32(&ctl->tab_full[i]), 33);  // the copies of the walker's lanes, and the walker
      mbar_init(smem_u32(&ctl->tab_empty[i]), epi_warps);
    }
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&ctl->b_full[i]), DEC_WARPS);
      mbar_init(smem_u32(&ctl->b_empty[i]), 1);
    }
    for (int i = 0; i < ACCS; ++i) {
      mbar_init(smem_u32(&ctl->acc_full[i]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[i]), epi_warps);
    }
    mbar_init(smem_u32(&ctl->epi_sync), 4);
    ctl->wait.init();
    fence_barrier_init();
    prefetch_tmap(&q_map);
  }
  if (warp == ISSUE_WARP) {
    tmem_alloc(smem_u32(&ctl->tmem_base), ACCS * TILE_T);
    tmem_relinquish();
  }
  // Launched with programmatic stream serialisation: the set-up above overlaps the kernel in front, nothing below may.
  griddep_wait();
  PlaidTable<NBITS>::fill(tab, P.plaid.bucket_weights, tid, NUM_THREADS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == ISSUE_WARP) {
    // =========================== MMA issuer ===========================
    const bool issue = elect_one();
    if (issue) {
      mbar_arrive_expect_tx(smem_u32(&ctl->q_full), (uint32_t)q_tile_bytes);
      for (int sl = 0; sl < P.n_slabs; ++sl)
        tma_load_2d(smem_u32(q_smem + sl * TILE_M * SLAB_BYTES_ROW), &q_map, sl * (SLAB_BYTES_ROW / 2), 0, smem_u32(&ctl->q_full));
    }
    __syncwarp();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const uint32_t a_desc0 = (uint32_t)smem_desc_sw128(smem_u32(q_smem)), b_desc0 = (uint32_t)smem_desc_sw128(smem_u32(b_smem));
    const uint32_t idesc = instr_desc(P.ab_format, TILE_T);
    constexpr uint32_t SLAB = (TILE_M * SLAB_BYTES_ROW) >> 4;
    const int k_steps = P.k_steps;
    bool ok = wait_bar(&ctl->q_full, 0, ctl, P.status);
    uint32_t st = 0, ph = 0;
    for (uint32_t t = 0; ok; ++t) {
      ok = wait_bar(&ctl->tab_full[t % TABLES], (t / TABLES) & 1, ctl, P.status);
      if (!ok) break;
      const uint32_t buf = t % ACCS, use = t / ACCS;
      if (ctl->n_seg[t % TABLES] < 0) {  // the epilogue waits for accumulators only
        if (wait_bar(&ctl->acc_empty[buf], (use & 1) ^ 1, ctl, P.status) && issue) mbar_arrive(smem_u32(&ctl->acc_full[buf]));
        break;
      }
      ok = wait_bar(&ctl->acc_empty[buf], (use & 1) ^ 1, ctl, P.status) && wait_bar(&ctl->b_full[st], ph, ctl, P.status);
      if (!ok) break;
      tc_fence_after();
      if (issue) {
        const uint32_t b_stage = b_desc0 + st * (uint32_t)(stage_bytes >> 4);
        const uint32_t d_tmem = tmem_base + buf * TILE_T;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < k_steps)
            tc_mma<false>(d_tmem, a_desc0 + (uint32_t)((k & 3) * 2) + (k >> 2) * SLAB, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * SLAB, desc_hi, idesc, k ? 1u : 0u);
        tc_commit(smem_u32(&ctl->b_empty[st]));
        tc_commit(smem_u32(&ctl->acc_full[buf]));
      }
      __syncwarp();
      if (++st == (uint32_t)STAGES) { st = 0; ph ^= 1; }
    }
    if (issue) {  // the copies must have landed before the CTA goes away, whatever became of the wait for them
      for (int spin = 0; spin < (1 << 16) && !mbar_try_wait_long(smem_u32(&ctl->q_full), 0); ++spin) {
      }
    }
  } else if (warp == WALK_WARP) {
    // =========================== walker ===========================
    int j, j_end;  // this CTA's documents
    const long long c = blockIdx.x, G = gridDim.x;
    if (P.d.cu) {
      const long long t0 = P.d.cu[0], t1 = P.d.cu[P.n_d], n = t1 > t0 ? t1 - t0 : 0;
      j = c == 0 ? 0 : lower_bound_warp(P.d.cu, P.n_d, t0 + n * c / G, lane);
      j_end = c == G - 1 ? P.n_d : lower_bound_warp(P.d.cu, P.n_d, t0 + n * (c + 1) / G, lane);
    } else {
      j = (int)(P.n_d * c / G);
      j_end = (int)(P.n_d * (c + 1) / G);
    }
    int nx_row, nx_len;  // bounds of document j + lane of the next 32
    auto fetch = [&](int first) {
      nx_row = nx_len = 0;
      if (first + lane < j_end) {
        long long r0;
        seq_bounds(P.d, first + lane, r0, nx_len, nullptr);
        nx_row = (int)r0;
        if (r0 < 0) nx_row = nx_len = 0;  // offsets that are none: nothing is read
      }
    };
    fetch(j);
    int cur_row = 0, cur_len = 0, at = 32;  // the 32 documents at hand, and the next of them
    int row = 0, left = 0;                  // the document in work
    bool open = false;
    const unsigned res_pitch = (unsigned)P.plaid.packed_dim;
    for (uint32_t t = 0;; ++t) {
      const uint32_t sl = t % TABLES;
      if (!wait_bar(&ctl->tab_empty[sl], ((t / TABLES) & 1) ^ 1, ctl, P.status)) break;
      int filled = 0, n_seg = 0;
      while (filled < TILE_T && n_seg < MAX_SEGS) {
        if (!open) {
          if (j >= j_end) break;
          if (at == 32) {
            cur_row = nx_row;
            cur_len = nx_len;
            at = 0;
            fetch(j + 32);
          }
          row = __shfl_sync(0xffffffffu, cur_row, at);
          left = __shfl_sync(0xffffffffu, cur_len, at);
          ++at;
          open = true;
        }
        const int n = min(left, TILE_T - filled), cols = (n + GRANULE - 1) & ~(GRANULE - 1);
        for (int i = lane; i < cols; i += 32) ctl->col[sl][filled + i].x = row + min(i, n - 1);
        filled += cols;
        row += n;
        left -= n;
        if (lane == 0) ctl->seg[sl][n_seg] = make_int2(j, filled / GRANULE | (left == 0 ? SEG_ENDS : 0));
        ++n_seg;
        if (left == 0) {
          open = false;
          ++j;
        }
      }
      // (columns behind the last segment decode some token that exists; nobody looks at them)
      for (int i = filled + lane; i < TILE_T; i += 32) ctl->col[sl][i].x = 0;
      if (lane == 0) ctl->n_seg[sl] = n_seg > 0 ? n_seg : -1;
      __syncwarp();
      if (n_seg > 0) {
        // the codes are copied behind the walker's back; the table is announced when all of them have come
#pragma unroll
        for (int u = 0; u < TILE_T / 32; ++u) {
          int2* c = &ctl->col[sl][lane + 32 * u];
          const int tok = c->x;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&c->y)), "l"(P.plaid.codes + tok) : "memory");
          asm volatile("prefetch.global.L2 [%0];" ::"l"(P.plaid.residuals + (long long)tok * res_pitch));
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&ctl->tab_full[sl])) : "memory");
      if (lane == 0) mbar_arrive(smem_u32(&ctl->tab_full[sl]));
      if (n_seg == 0) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // (none may land after the CTA is gone)
  } else if (warp < 4) {
    // =========================== epilogue ===========================
    const int wq = warp, row = wq * 32 + lane, et = row;
    bool ok = true;
    uint32_t n_sync = 0, n_emit = 0;
    auto epi_sync = [&]() {  // bounded rendezvous of the four warps
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->epi_sync));
      ok = wait_bar(&ctl->epi_sync, n_sync++ & 1, ctl, P.status) && ok;
    };
    const bool topk = P.topk.cand_key != nullptr;
    const int nq = P.n_q;  // all queries share the one tile
    ctl->row_seg[et] = -1;
    epi_sync();
    if (ok && et < nq) {
      long long r0;
      int l;
      seq_bounds(P.q, et, r0, l, P.status);
      const int off = (int)r0;
      if (off + l > TILE_M) {
        l = max(0, TILE_M - off);
        if (P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
      }
      ctl->seg_off[et] = (short)off;
      ctl->seg_len[et] = (short)l;
      for (int i = 0; i < l; ++i) ctl->row_seg[off + i] = (short)et;
      if (topk) {
        // the candidate list of (this CTA, this query)
        int list = (int)blockIdx.x * P.topk.qpg + et;
        if ((unsigned)list >= (unsigned)P.topk.n_lists) {
          if (P.status) atomicOr(P.status, LIK_DEV_INTERNAL);
          list = 0;
        }
        const int2 hd = P.topk.hdr[list];
        ctl->seg_list[et] = list;
        ctl->seg_cnt[et] = hd.x;
        ctl->seg_thr[et] = (unsigned)hd.y;
      }
    }
    epi_sync();
    const int my_sg = ok ? ctl->row_seg[row] : -1;
    const bool counts = my_sg >= 0 && row_valid(P.q, row);
    const float my_qf = my_sg >= 0 ? row_factor(P.q, row) : 0.f;
    const bool any = __any_sync(0xffffffffu, my_sg >= 0);
    const uint32_t acc0 = tmem_base + ((uint32_t)(wq * 32) << 16);
    float r = -INFINITY;  // maximum over the document so far
    for (uint32_t t = 0; ok && wq < epi_warps; ++t) {
      const uint32_t sl = t % TABLES, buf = t % ACCS, use = t / ACCS;
      ok = wait_bar(&ctl->acc_full[buf], use & 1, ctl, P.status);  // (behind the last tile: announced without one)
      if (!ok) break;
      const int n_seg = ctl->n_seg[sl];
      if (n_seg < 0) break;
      tc_fence_after();
      if (topk) {
        if (lone) tidy_list(P, ctl, wq, lane);
        else
          for (int q = wq; q < nq; q += 4) tidy_list(P, ctl, q, lane);
      }
      int sgi = 0;
      int2 sg = ctl->seg[sl][0];
#pragma unroll 1
      for (int c = 0; c < TILE_T / GRANULE; c += 4) {  // 32 columns: four granules, each of one document
        float g[4];
        if (lone || any) {
          float v[32];
          tmem_ld32_issue(acc0 + buf * TILE_T + c * GRANULE, v);
          tmem_ld_wait(v);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            g[i] = max3(max3(v[8 * i], v[8 * i + 1], v[8 * i + 2]), max3(v[8 * i + 3], v[8 * i + 4], v[8 * i + 5]), fmaxf(v[8 * i + 6], v[8 * i + 7]));
        }
        if (c + 4 == TILE_T / GRANULE) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl->acc_empty[buf]));
        }
        int at = 0;  // granules of the chunk that are done with
        while (sgi < n_seg) {
          const int end = (sg.y & 0xffff) - c;  // of the segment, in granules of the chunk
          if (at == 0 && end >= 4) {
            r = fmaxf(max3(g[0], g[1], g[2]), fmaxf(g[3], r));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i >= at && i < end) r = fmaxf(r, g[i]);
          }
          at = min(end, 4);
          if (end > 4) break;
          if (sg.y & SEG_ENDS) {
            const float val = counts && r != -INFINITY ? r * my_qf : 0.f;
            r = -INFINITY;
            if (lone) {
              const float sum = warp_sum(val);
              emit_score(P, ctl, wq, sum, sg.x, lane);
            } else {
              float* e = ctl->emit[n_emit++ & 1];
              e[row] = val;
              epi_sync();
              if (!ok) break;
              for (int q = wq; q < nq; q += 4) {
                const int off = ctl->seg_off[q], len = ctl->seg_len[q];
                float sum = 0.f;
                for (int i = lane; i < len; i += 32) sum += e[off + i];
                sum = warp_sum(sum);
                emit_score(P, ctl, q, sum, sg.x, lane);
              }
            }
          }
          if (++sgi >= n_seg) break;
          sg = ctl->seg[sl][sgi];
          if (at == 4 && (sg.y & 0xffff) - c > 4) break;
        }
        if (!ok) break;
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->tab_empty[sl]));
    }
    if (topk && ok) {
      if (!lone) epi_sync();  // every warp is done with the lists
      if (ok && (lone ? lane == 0 && wq < nq : et < nq)) {
        const int q = lone ? wq : et;
        P.topk.hdr[ctl->seg_list[q]] = make_int2(ctl->seg_cnt[q], (int)ctl->seg_thr[q]);
      }
    }
  } else if (warp >= DEC_WARP0) {
    // =========================== decoders ===========================
    const int l = lane & 7, dim = FULL ? 128 : P.plaid.dim;
    const bool on0 = FULL || l * 8 < dim, on1 = FULL || 64 + l * 8 < dim;
    constexpr int GROUPS = DEC_COLS / 8;  // of eight columns, one after the other
    const int col0 = (warp - DEC_WARP0) * DEC_COLS + (lane >> 3) * 2;  // this quarter-warp's columns of the first
    // (lanes behind the width read what lane 0 reads)
    const char* cen0 = static_cast<const char*>(P.plaid.centroids) + (on0 ? l * (CF32 ? 32 : 16) : 0);
    const char* res0 = reinterpret_cast<const char*>(P.plaid.residuals) + (on0 ? l * NBITS : 0);
    const int cen_h = FULL ? (CF32 ? 256 : 128) : on1 ? (CF32 ? 256 : 128) : 0, res_h = FULL ? 8 * NBITS : on1 ? 8 * NBITS : 0;
    const unsigned cen_pitch = (unsigned)dim * (CF32 ? 4u : 2u), res_pitch = FULL ? 16u * NBITS : (unsigned)P.plaid.packed_dim;
    const bool f16 = P.plaid_f16 != 0;
    unsigned char* dst0 = b_smem + col0 * SLAB_BYTES_ROW;
    const unsigned n_centroids = (unsigned)P.plaid.n_centroids;
    bool ok = true;
    auto announced = [&](uint32_t t) {  // whether there is a tile t
      ok = wait_bar(&ctl->tab_full[t % TABLES], (t / TABLES) & 1, ctl, P.status);
      return ok && ctl->n_seg[t % TABLES] >= 0;
    };
    PlaidPiece<CF32, NBITS> nx[4];
    auto load_rows = [&](uint32_t t, int grp) {
      const int4 cc = *reinterpret_cast<const int4*>(&ctl->col[t % TABLES][col0 + grp * 8]);  // two columns
      unsigned c0 = (unsigned)cc.y, c1 = (unsigned)cc.w;
      if (max(c0, c1) >= n_centroids) {
        if (P.status) atomicOr(P.status, LIK_DEV_CODE_RANGE);
        c0 = c0 < n_centroids ? c0 : 0;
        c1 = c1 < n_centroids ? c1 : 0;
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
        nx[p] = plaid_piece<CF32, NBITS>(cen0 + (p & 1 ? cen_h : 0), cen_pitch, p < 2 ? c0 : c1, res0 + (p & 1 ? res_h : 0), res_pitch, (unsigned)(p < 2 ? cc.x : cc.z));
    };
    bool have = announced(0);
    if (have) load_rows(0, 0);
    uint32_t st = 0, ph = 0;
    for (uint32_t t = 0; have && ok; ++t) {
#pragma unroll
      for (int grp = 0; grp < GROUPS; ++grp) {
        // the values of eight tokens; the next eight's rows are on their way while these are finished
        float e[4][8];
#pragma unroll
        for (int p = 0; p < 4; ++p) plaid_values_near<CF32, CBF16, NBITS>(nx[p], tab, e[p]);
        if (grp + 1 < GROUPS) {
          load_rows(t, grp + 1);
        } else {
          have = announced(t + 1);
          if (!ok) break;
          if (have) load_rows(t + 1, 0);
        }
        plaid_finish2(P.plaid.normalize != 0, e, lane, on0, on1);
        if (grp == 0) {
          ok = wait_bar(&ctl->b_empty[st], ph ^ 1, ctl, P.status);
          if (!ok) break;
        }
        unsigned char* dst = dst0 + st * (uint32_t)stage_bytes + grp * (8 * SLAB_BYTES_ROW);
        auto store = [&](auto f16_) {
#pragma unroll
          for (int p = 0; p < 4; ++p)
            if (p & 1 ? on1 : on0)
              *reinterpret_cast<uint4*>(dst + (p & 1) * (TILE_T * SLAB_BYTES_ROW) + (p >> 1) * SLAB_BYTES_ROW + ((l ^ ((col0 + (p >> 1)) & 7)) << 4)) =
                  plaid_pack16(e[p], decltype(f16_)::value);
        };
        if (f16) store(std::true_type{});
        else store(std::false_type{});
      }
      if (!ok) break;
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->b_full[st]));
      if (++st == (uint32_t)STAGES) { st = 0; ph ^= 1; }
    }
  }

  // ---- teardown (also reached when aborting: every wait above is bounded) ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUE_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACCS * TILE_T);
  }
}

}  // namespace

size_t fwd_plaid_smem(int n_slabs) { return dynamic_smem(n_slabs); }
int fwd_plaid_ctas_per_sm() { return CTAS_PER_SM; }

int launch_fwd_plaid(const lik_fwd_args& a, const TcPlan& pl, const TcParams& P, cudaStream_t st) {
  CUtensorMap q_map;
  int rc = make_tmap_rows(&q_map, a.q.data, a.dtype, a.dim, a.q.n_rows, a.q.row_stride, TILE_M);
  if (rc) return rc;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)pl.grid);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = pl.smem_bytes;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
#define LIK_PLAID_LAUNCH(CF, CB, NB)                                            \
  do {                                                                          \
    if (a.dim == 128) {                                                         \
      LIK_CUDA_OK((allow_smem<fwd_plaid_kernel<CF, CB, NB, true>>()));          \
      LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_plaid_kernel<CF, CB, NB, true>, q_map, P)); \
    } else {                                                                    \
      LIK_CUDA_OK((allow_smem<fwd_plaid_kernel<CF, CB, NB, false>>()));         \
      LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_plaid_kernel<CF, CB, NB, false>, q_map, P)); \
    }                                                                           \
  } while (0)
#define LIK_PLAID_BITS(CF, CB)                      \
  do {                                              \
    if (P.plaid.nbits == 2) LIK_PLAID_LAUNCH(CF, CB, 2);      \
    else if (P.plaid.nbits == 4) LIK_PLAID_LAUNCH(CF, CB, 4); \
    else LIK_PLAID_LAUNCH(CF, CB, 8);               \
  } while (0)
  if (P.plaid.centroid_dtype == LIK_F32) LIK_PLAID_BITS(true, false);
  else if (P.plaid.centroid_dtype == LIK_BF16) LIK_PLAID_BITS(false, true);
  else LIK_PLAID_BITS(false, false);
#undef LIK_PLAID_BITS
#undef LIK_PLAID_LAUNCH
  ::lik::count_launch();
  return LIK_OK;
}

}  // namespace lik
