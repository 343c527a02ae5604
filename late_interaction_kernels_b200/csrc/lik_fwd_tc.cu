// Blackwell tensor-core MaxSim forward (sm_100a: TMA + tcgen05.mma + TMEM): the kernel for smaller problems, for norms taken
// from the document tiles and for documents decoded from a PLAID index, and the host side of both tensor-core kernels.
// Larger problems run in lik_fwd_streams.cu (streams_pay has the rule).
//
// GEMM view: rows = query tokens (A operand, K-major, 128 per tile), columns = document tokens (B
// operand, K-major, up to 256 per tile), K = embedding width.  A CTA is persistent: it keeps one or
// two 128-row query tiles resident in shared memory and streams document tiles through a TMA ring.
// Every document tile feeds one MMA group per resident query tile; the fp32 accumulator of query
// tile m lives in TMEM columns [256 m, 256 m + 256).  A tile never spans two documents, so the
// epilogue is: per thread (= one query token = one TMEM lane) a running max over the tile's columns,
// carried across the tiles of a document; at the end of the document the 128 row maxima are summed
// per query (fixed order) into one score.  Scores for a (query, document) pair have exactly one
// writer, so the forward is bitwise reproducible.
//
// Warp roles (640 threads): warp 0 = producer (TMA; the only role that walks the work units, which it publishes in
// a small ring in shared memory); warp 1 = MMA issuer + TMEM owner, driven by one word per ring stage that the
// producer writes; warps 2-9 = epilogue group 0 (accumulator 0), warps 10-17 = epilogue group 1 (accumulator 1);
// warps 18-19 decode tokens beside warp 0 in the PLAID kernels and are idle otherwise (they also round the block up
// to the register-allocation granule).  An accumulator is single-buffered (two 256-column accumulators fill TMEM).
// What bounds the kernel is the chain of dependent steps an epilogue warp runs per (query tile, document): hand-shake,
// three or four TMEM round trips with their folds, the hand-over between the two halves of a group, the emit.  So the
// code on that chain is kept short and free of branches, and paths that are rare (documents whose mask has holes)
// get their own copy of the loop instead of a test inside the common one.
//
// The same kernel scores into a matrix, keeps the winners for the backward, or keeps a per-query top-k (candidate
// lists per CTA and query, merged by a second kernel); documents come from a matrix through TMA or are decoded
// from a PLAID index by the producer warps.
//
// Every mbarrier wait is bounded: on expiry the CTA raises LIK_DEV_WAIT_TIMEOUT in the status word,
// sets a shared abort flag, drains its TMA copies, frees TMEM and returns.
#include <cuda.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "lik_fwd_tc.cuh"

namespace lik {

int topk_merge_parts(int n_ctas, int n_groups, int per_slot);

namespace {

#ifndef LIK_TILE_N
#define LIK_TILE_N 256
#endif
constexpr int TILE_N = LIK_TILE_N;     // document tokens per TMA stage = columns of one accumulator
constexpr int ACC_COLS = 256;          // TMEM columns reserved per accumulator
static_assert(TILE_N <= ACC_COLS && TILE_N % 32 == 0, "a stage must fit one accumulator");
constexpr int N_BOXES = TILE_N / BOX_ROWS;
constexpr int NUM_THREADS = 640;
constexpr int EPI_THREADS = 128;     // threads per half of an epilogue group (one per accumulator row)
constexpr int GROUP_WARPS = 8;
constexpr int UNIT_RING = 8;                  // slots of the producer -> epilogue unit ring
constexpr int LONG_DOC_TOKENS = 2048;         // problems whose documents can be this long run the kernel with the lazy winner scan

// Rings of multiplier slots: two of sc_per = stages + 1 slots, one per accumulator (tiles that feed both use the first).  Slot n
// of an accumulator's ring is refilled for its tile n + sc_per: by then the MMAs of one of the sc_per - 1 tiles between them have
// completed (the producer is at most `stages` tiles ahead of the tensor pipe), which needed the accumulator back from every
// earlier tile - and an epilogue gives it back only after its last read of the multipliers.

// Warps 18 and 19 take the rows' inverse norms from the tiles in shared memory when the launch asks for it: the documents
// are then read once instead of twice, and no norms go through device memory.  Two queries of 128 tokens against 4000
// documents of up to 1030: 484 -> 232 us (146 without normalisation; the two warps' arithmetic is what remains of the gap).
constexpr int NORM_WARPS = 2;
constexpr int PLAID_WARPS = 3;  // warps 0, 18 and 19 decode compressed tokens in the PLAID kernels

struct SharedCtl {
  unsigned long long q_full, q_empty;
  unsigned long long d_full[8], d_empty[8];
  unsigned long long acc_full[2], acc_empty[2];
  uint32_t stage_info[8];
  int4 unit_info[UNIT_RING];    // per work unit: x = document length | LEN_FLAG_MASKED, y = its first row, z = tile group, w = document
  volatile int units_posted;    // units published in unit_info so far
  volatile int units_total;     // all units of this CTA once the producer has walked them (INT_MAX until then)
  uint32_t tmem_base;
  volatile int abort_flag;
  long long wait_limit;         // cycles after which a wait gives up
  int seg_off[2][TILE_M], seg_len[2][TILE_M], seg_q[2][TILE_M];
  short row_seg[2][TILE_M];
  int n_seg[2];
  int warp_aligned[2];  // every query of the tile sits inside one warp's 32 rows, starting at its first row
  float emit[2][2][TILE_M];
  float xch_m[2][2][TILE_M];  // half 1 -> half 0: per-row running maximum and its column
  int xch_i[2][2][TILE_M];
  alignas(16) float col_scale[2][TILE_N];  // read as float4
  alignas(16) float col_bias[2][TILE_N];
  // fused top-k: state of the candidate list of every query of the resident tiles
  int seg_cnt[2][TILE_M];
  unsigned seg_thr[2][TILE_M];
  int seg_list[2][TILE_M];      // list number (slot * qpg + query within the group)
  float plaid_bw[256];          // PLAID kernels: the bucket weights
};

// Bounded wait.  Returns false when the CTA is aborting.  The first probe lets the hardware suspend
// the thread until the phase completes (or the hint expires), so the common case costs two
// instructions; everything else is out of line or, with INLINE, behind it.  A call has registers around it saved to
// local memory.  Only the kernels for e4m3 operands gain from doing without it: 4 x 4096 documents of 256 tokens
// 43.9 -> 41.9 us; with all of them inlined the others lose (1 x 1000 normalised fp16 28.6 -> 31.1 us, 3001 pairs 37.0 -> 37.6).
__device__ __forceinline__ bool wait_bar_loop(uint32_t b, uint32_t parity, SharedCtl* ctl, int* status) {
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait_long(b, parity)) return true;
    if (ctl->abort_flag) return false;
    if (clock64() - t0 > ctl->wait_limit) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
      return false;
    }
  }
}
__device__ __noinline__ bool wait_bar_slow(uint32_t b, uint32_t parity, SharedCtl* ctl, int* status) {
  return wait_bar_loop(b, parity, ctl, status);
}
template <bool INLINE>
__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  const uint32_t b = smem_u32(bar);
  if (mbar_try_wait_long(b, parity)) return true;
  return INLINE ? wait_bar_loop(b, parity, ctl, status) : wait_bar_slow(b, parity, ctl, status);
}
// The same for all lanes of a warp: they leave together, with one answer.
template <bool INLINE>
__device__ __forceinline__ bool wait_bar_warp(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  return __all_sync(0xffffffffu, wait_bar<INLINE>(bar, parity, ctl, status));
}
// Bounded wait until the producer has published unit `uc` of this CTA in the unit ring.
// Returns 1 when the unit is there, 2 when the stream has ended before it, 0 when the CTA is aborting.
__device__ __noinline__ int wait_posted_slow(SharedCtl* ctl, int uc, int* status) {
  const long long t0 = clock64();
  while (true) {
    if (ctl->units_posted > uc) return 1;
    if (ctl->units_total <= uc) return 2;
    if (ctl->abort_flag) return 0;
    if (clock64() - t0 > ctl->wait_limit) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
      return 0;
    }
  }
}
__device__ __forceinline__ int wait_posted(SharedCtl* ctl, int uc, int* status) {
  if (ctl->units_posted > uc) return 1;
  return wait_posted_slow(ctl, uc, status);
}

// ---------------------------------------------------------------------------------------------
// The units of a CTA, in the order every role walks them.
//   CROSS: the documents are cut into super-blocks (one unless the caller asked for more: a super-block is
//   sized to stay in L2 while every tile group passes over it); inside a super-block the units are (tile
//   group, document), group-major, and CTA c of G takes the c-th of G equal shares.  A CTA therefore sees
//   the same one to three groups in every super-block, each with an ascending document range.
//   GROUPED: unit = document, group = its query.  LIST: unit = pair, group = its query (from the table).
// `doc` is the global document index (LIST: the pair).
// ---------------------------------------------------------------------------------------------
struct UnitIter {
  int sb;               // super-block
  int doc_lo, doc_hi;   // its documents
  int left;             // units of this CTA's share of the super-block still to come, this one included
  int grp, doc, in_grp;
};

__device__ __forceinline__ bool iter_enter(const TcParams& P, int n_groups, UnitIter& it) {
  const long long c = blockIdx.x, G = gridDim.x;
  while (it.sb < P.n_sb) {
    long long units;
    if (P.pairing == LIK_PAIR_CROSS) {
      it.doc_lo = (int)min((long long)it.sb * P.sb_docs, (long long)P.n_d);
      it.doc_hi = (int)min((long long)it.doc_lo + P.sb_docs, (long long)P.n_d);
      units = (long long)n_groups * (it.doc_hi - it.doc_lo);
    } else {
      it.doc_lo = 0;
      it.doc_hi = P.n_d;
      units = P.n_flat;
    }
    long long u, u_end;
    if (units < (1ll << 32) / 256) {  // (a 64-bit division is a hundred dependent instructions in front of the first load; grids have at most 256 CTAs)
      u = (unsigned)units * (unsigned)c / (unsigned)G;
      u_end = (unsigned)units * (unsigned)(c + 1) / (unsigned)G;
    } else {
      u = units * c / G;
      u_end = units * (c + 1) / G;
    }
    if (u < u_end) {
      it.left = (int)(u_end - u);
      if (P.pairing == LIK_PAIR_CROSS) {
        const int nd_b = it.doc_hi - it.doc_lo;
        it.grp = u < (1ll << 32) ? (int)((unsigned)u / (unsigned)nd_b) : (int)(u / nd_b);
        it.doc = it.doc_lo + (int)(u - (long long)it.grp * nd_b);
        it.in_grp = 0;
      } else if (P.pairing == LIK_PAIR_GROUPED) {
        it.doc = (int)u;
        it.grp = it.doc / P.group;
        it.in_grp = it.doc - it.grp * P.group;
      } else {
        it.doc = (int)u;
        it.grp = -1;  // comes from the table
        it.in_grp = 0;
      }
      return true;
    }
    ++it.sb;
  }
  return false;
}
__device__ __forceinline__ bool iter_begin(const TcParams& P, int n_groups, UnitIter& it) {
  it.sb = 0;
  return iter_enter(P, n_groups, it);
}
__device__ __forceinline__ bool iter_next(const TcParams& P, int n_groups, UnitIter& it) {
  if (--it.left > 0) {
    ++it.doc;
    if (P.pairing == LIK_PAIR_CROSS) {
      if (it.doc == it.doc_hi) {
        it.doc = it.doc_lo;
        ++it.grp;
      }
    } else if (P.pairing == LIK_PAIR_GROUPED) {
      if (++it.in_grp == P.group) {
        it.in_grp = 0;
        ++it.grp;
      }
    }
    return true;
  }
  ++it.sb;
  return iter_enter(P, n_groups, it);
}

// Length words of a unit's document, loaded one unit ahead of their use.
struct UnitRaw {
  int a, b, q;
};
__device__ __forceinline__ UnitRaw unit_fetch(const TcParams& P, int doc) {
  UnitRaw r{0, 0, 0};
  if (P.pairing == LIK_PAIR_LIST) {
    const int4 t = __ldg(P.list_tab + doc);
    r.q = t.x;
    r.a = t.y;
    r.b = t.z;
  } else if (P.d.cu) {
    r.a = P.d.cu[doc];
    r.b = P.d.cu[doc + 1];
  } else if (P.d.lens) {
    r.a = P.d.lens[doc];
  }
  return r;
}
// First row and column count of the fetched document; `masked` tells whether its mask has holes.
// Lengths come from the caller-validated views, clamped to the padded extent.
__device__ __forceinline__ void unit_resolve(const TcParams& P, int doc, const UnitRaw& r, long long& row0, int& len, bool& masked) {
  masked = false;
  if (P.pairing == LIK_PAIR_LIST) {
    row0 = r.a;
    len = r.b;
  } else if (P.d.cu) {
    const int a = r.a, b = r.b;
    row0 = a;
    len = b > a ? b - a : 0;
    if ((long long)a + len > P.d.n_rows) len = P.d.n_rows > a ? (int)(P.d.n_rows - a) : 0;
  } else {
    row0 = (long long)doc * P.d.seq_stride;
    len = P.d.max_len;
    if (P.d.lens) {
      int l = r.a;
      if (P.d_len_flagged) {
        masked = (l & LEN_FLAG_MASKED) != 0;
        l &= ~LEN_FLAG_MASKED;
      }
      len = l < 0 ? 0 : (l > P.d.max_len ? P.d.max_len : l);
    }
  }
}

// Sum of squares of one row of a stage (lane = row: eight consecutive rows of a swizzled slab lie in different banks).  The
// pieces of 16 bytes are summed and combined in the order of prep_kernel's butterfly, so that the norms of a row are the
// same number wherever they are taken.
template <typename T>
__device__ __forceinline__ float stage_row_sum_sq(const unsigned char* row, int r, bool two_slabs) {
  float half[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // pieces h, h + 2, h + 4, h + 6, each beside its partner eight further: their loads in flight together
    uint4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned char* a = row + (((2 * i + h) ^ (r & 7)) << 4);
      x[i] = *reinterpret_cast<const uint4*>(a);
      y[i] = make_uint4(0, 0, 0, 0);
      if (two_slabs) y[i] = *reinterpret_cast<const uint4*>(a + TILE_N * SLAB_BYTES_ROW);
    }
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        fma_sq_pair<T>(w == 0 ? x[i].x : w == 1 ? x[i].y : w == 2 ? x[i].z : x[i].w, s0[i]);
        fma_sq_pair<T>(w == 0 ? y[i].x : w == 1 ? y[i].y : w == 2 ? y[i].z : y[i].w, s1[i]);
      }
    half[h] = ((s0[0] + s1[0]) + (s0[2] + s1[2])) + ((s0[1] + s1[1]) + (s0[3] + s1[3]));
  }
  return half[0] + half[1];
}

struct DocMaps {
  CUtensorMap m[N_BOXES];  // document boxes of 32, 64, ... rows: one copy per K slab whatever the tile height
};

// Word the producer leaves beside every ring stage for the MMA issuer.
constexpr uint32_t STAGE_COLS_MASK = 0x1FFu;   // valid document rows in the stage
constexpr uint32_t STAGE_ACC0 = 1u << 16;      // feed accumulator 0 / 1
constexpr uint32_t STAGE_ACC1 = 1u << 17;
constexpr uint32_t STAGE_FIRST = 1u << 18;     // first stage of a query-tile group: wait for the tiles
constexpr uint32_t STAGE_LAST = 1u << 19;      // last stage of the group: hand the tiles back afterwards
constexpr uint32_t STAGE_END = 1u << 20;       // no more work

// WINNERS: 0 = scores only, 1 = winners saved, 2 = winners saved and every document takes the lazy winner scan (launched
// for problems whose documents are long, so that the kernels for short documents carry no third copy of the tile loop)
template <bool FP8, int WINNERS, bool SCALED, bool PLAID>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fwd_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ DocMaps d_maps, const TcParams P) {
  constexpr bool ARGMAX = WINNERS != 0;
  extern __shared__ unsigned char smem_raw[];
  // operand tiles need 1024-byte alignment for the 128-byte swizzle
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int q_tile_bytes = P.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const int d_stage_bytes = P.n_slabs * TILE_N * SLAB_BYTES_ROW;
  unsigned char* q_smem = smem;                              // [2][n_slabs][128 rows][128 B]
  unsigned char* d_smem = smem + 2 * q_tile_bytes;           // [stages][n_slabs][256 rows][128 B]
  float* sc_ring = reinterpret_cast<float*>(d_smem + (size_t)P.stages * d_stage_bytes);  // [sc_slots][TILE_N] (kernels with multipliers)
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(d_smem + (size_t)P.stages * d_stage_bytes + (size_t)P.sc_slots * TILE_N * sizeof(float));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const bool list = P.pairing == LIK_PAIR_LIST;
  const bool topk = !ARGMAX && P.topk.cand_key != nullptr;  // the fused top-k never saves winners

  const bool norm_warps = SCALED && !FP8 && !PLAID && P.norm_eps > 0.f;  // (a member of every pipeline barrier then)
  if (tid == 0) {
    mbar_init(smem_u32(&ctl->q_full), 1);
    mbar_init(smem_u32(&ctl->q_empty), 1);
    for (int s = 0; s < P.stages; ++s) {
      mbar_init(smem_u32(&ctl->d_full[s]), PLAID ? PLAID_WARPS : 1);  // the decoder warps, or TMA
      mbar_init(smem_u32(&ctl->d_empty[s]), norm_warps ? 1 + NORM_WARPS : 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ctl->acc_full[a]), norm_warps ? 1 + NORM_WARPS : 1);
      mbar_init(smem_u32(&ctl->acc_empty[a]), GROUP_WARPS);
    }
    ctl->abort_flag = 0;
    ctl->wait_limit = WAIT_LIMIT_CYCLES;
    ctl->units_posted = 0;
    ctl->units_total = 0x7fffffff;
    fence_barrier_init();
    prefetch_tmap(&q_map);
    if (!PLAID)
      for (int i = 0; i < N_BOXES; ++i) prefetch_tmap(&d_maps.m[i]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctl->tmem_base), 512);
    tmem_relinquish();
  }
  // Launched with programmatic stream serialisation: the set-up above overlaps the kernel in front, nothing below may.
  griddep_wait();
  if (PLAID)
    for (int b = tid; b < (1 << P.plaid.nbits); b += NUM_THREADS) ctl->plaid_bw[b] = P.plaid.bucket_weights[b];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  // greedy-packed query tiles are counted on the device (the count sits in front of the table)
  const int n_tiles = P.tile_q0 ? P.tile_q0[-1] : P.n_tiles;
  const int n_groups = (n_tiles + P.mt - 1) / P.mt;

  const bool producer_warp = warp == 0 || (PLAID && warp >= 2 + 2 * GROUP_WARPS);
  if (producer_warp) {
    // =========================== producer ===========================
    // TMA kernels: one thread (warp 0, lane 0) walks the units, loads the query tiles and the document
    // stages with TMA and leaves the stage words and the unit ring.  PLAID kernels: three whole warps walk
    // the units in step; each decodes its share of every stage's tokens into the swizzled operand layout
    // (generic-proxy stores, fenced for the tensor core's reads), and arrives on the stage barrier; the
    // elected thread of warp 0 still does everything else.
    const bool elect = warp == 0 && lane == 0;
    if (PLAID || lane == 0) {
      const int pw = warp == 0 ? 0 : warp - (2 + 2 * GROUP_WARPS) + 1;  // decoder warp number 0..2
      int cur_grp = -1;
      uint32_t n_qload = 0, st = 0, ph = 0, n_dload = 0;
      int sc_cnt[2] = {0, 0};  // next slot in either accumulator's multiplier ring
      long long uc = 0;
      const int x_per_slab = SLAB_BYTES_ROW / P.elt_bytes;
      bool ok = true;
      int tiles_here = 0;
      // the iterator stands one unit ahead: that unit's length words are in flight while this one is produced
      UnitIter it;
      bool have = iter_begin(P, n_groups, it);
      int nx_grp = 0, nx_doc = 0;
      UnitRaw nx_raw{0, 0, 0};
      if (have) {
        nx_grp = it.grp;
        nx_doc = it.doc;
        nx_raw = unit_fetch(P, nx_doc);
      }
      while (have && ok) {
        const int doc = nx_doc;
        const int grp = list ? nx_raw.q : nx_grp;
        long long drow0;
        int dlen;
        bool dmasked;
        unit_resolve(P, doc, nx_raw, drow0, dlen, dmasked);
        have = iter_next(P, n_groups, it);
        int next_grp = -1;
        if (have) {
          nx_grp = it.grp;
          nx_doc = it.doc;
          nx_raw = unit_fetch(P, nx_doc);
          next_grp = list ? nx_raw.q : nx_grp;
        }
        const bool last_unit_of_grp = next_grp != grp;
        uint32_t first = 0;
        if (grp != cur_grp) {
          cur_grp = grp;
          first = STAGE_FIRST;
          const int t0 = grp * P.mt, t1 = min(t0 + P.mt, n_tiles);
          tiles_here = t1 - t0;
          if (elect) {
            // wait until the MMAs that read the previous query tiles are done
            ok = wait_bar<FP8>(&ctl->q_empty, (n_qload & 1) ^ 1, ctl, P.status);
            if (ok) {
              mbar_arrive_expect_tx(smem_u32(&ctl->q_full), (uint32_t)((t1 - t0) * q_tile_bytes));
              for (int t = t0; t < t1; ++t) {
                TileInfo ti = tile_info(P, t);
                for (int sl = 0; sl < P.n_slabs; ++sl)
                  tma_load_2d(smem_u32(q_smem + (t - t0) * q_tile_bytes + sl * TILE_M * SLAB_BYTES_ROW), &q_map, sl * x_per_slab,
                              (int)ti.row0, smem_u32(&ctl->q_full));
              }
            }
          }
          ++n_qload;
          if (PLAID && warp == 0) ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          if (!ok) break;
        }
        // which accumulators this unit feeds: both resident tiles, or (one tile) alternating with the unit count
        const uint32_t acc_bits = P.mt == 2 ? (tiles_here == 2 ? (STAGE_ACC0 | STAGE_ACC1) : STAGE_ACC0)
                                            : ((uc & 1) ? STAGE_ACC1 : STAGE_ACC0);
        const int sc_ring_id = (!SCALED || P.mt == 2 || !(uc & 1)) ? 0 : 1;  // the multiplier ring of the accumulator(s) this unit feeds
        // publish the unit for the epilogue groups, then its stages; an empty document still sends one
        // (empty) stage so that every unit passes through the same hand-shakes
        if (elect) {
          ctl->unit_info[uc & (UNIT_RING - 1)] = make_int4(
              (dlen & UNIT_LEN_MASK) | (SCALED ? (sc_ring_id * P.sc_per + sc_cnt[sc_ring_id]) << UNIT_SLOT_SHIFT : 0) |
                  (dmasked ? LEN_FLAG_MASKED : 0),
              (int)drow0, grp, doc);
          __threadfence_block();
          ctl->units_posted = (int)uc + 1;
        }
        int c0 = 0;
        do {
          const int ncols = max(0, min(TILE_N, dlen - c0));
          ok = wait_bar<FP8>(&ctl->d_empty[st], ph ^ 1, ctl, P.status);
          if (!ok) break;
          const uint32_t full = smem_u32(&ctl->d_full[st]);
          if (elect) {
            uint32_t info = (uint32_t)ncols | acc_bits;
            if (c0 == 0) info |= first;
            if (last_unit_of_grp && c0 + TILE_N >= dlen) info |= STAGE_LAST;
            ctl->stage_info[st] = info;
          }
          if (PLAID) {
            // the stage's tokens in six equal runs, one per half-warp of the three decoder warps
            const int hl = lane & 15;
            const int hw6 = pw * 2 + (lane >> 4);
            const int per = (ncols + 2 * PLAID_WARPS - 1) / (2 * PLAID_WARPS);
            const int t_lo = min(hw6 * per, ncols), n_run = min(per, ncols - t_lo);
            unsigned char* stage = d_smem + (size_t)st * d_stage_bytes + (hl >> 3) * (TILE_N * SLAB_BYTES_ROW);
            const bool f16 = P.plaid_f16 != 0;
            auto sink = [&](int t, const float (&e)[8]) {
              const int row = t_lo + t;
              *reinterpret_cast<uint4*>(stage + row * SLAB_BYTES_ROW + (((hl & 7) ^ (row & 7)) << 4)) = plaid_pack16(e, f16);
            };
            if (P.plaid.centroid_dtype == LIK_F32)
              plaid_decode_range<true, 4>(P.plaid, ctl->plaid_bw, drow0 + c0 + t_lo, n_run, per, lane, hl * 8 < P.plaid.dim, P.status, sink);
            else
              plaid_decode_range<false, 8>(P.plaid, ctl->plaid_bw, drow0 + c0 + t_lo, n_run, per, lane, hl * 8 < P.plaid.dim, P.status, sink);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full);
          } else {
            const int boxes = (ncols + BOX_ROWS - 1) / BOX_ROWS;
            if (boxes > 0) {
              // the tile's multipliers ride on the same barrier: whole groups of four floats, never past the array's end
              uint32_t sc_bytes = 0;
              if (SCALED && P.col_src) {
                const long long r = drow0 + c0;
                sc_bytes = (uint32_t)min((long long)((ncols + 3) & ~3), P.d.n_rows - r) * 4u;
              }
              mbar_arrive_expect_tx(full, (uint32_t)(boxes * BOX_ROWS * SLAB_BYTES_ROW * P.n_slabs) + sc_bytes);
              const CUtensorMap* map = &d_maps.m[boxes - 1];
              for (int sl = 0; sl < P.n_slabs; ++sl)
                tma_load_2d(smem_u32(d_smem + (size_t)st * d_stage_bytes + sl * TILE_N * SLAB_BYTES_ROW), map, sl * x_per_slab,
                            (int)(drow0 + c0), full);
              if (sc_bytes)
                bulk_load_1d(smem_u32(sc_ring + (sc_ring_id * P.sc_per + sc_cnt[sc_ring_id]) * TILE_N), P.col_src + drow0 + c0, sc_bytes, full);
            } else {
              mbar_arrive(full);
            }
          }
          ++n_dload;
          if (++st == (uint32_t)P.stages) { st = 0; ph ^= 1; }
          if (SCALED && ++sc_cnt[sc_ring_id] >= P.sc_per) sc_cnt[sc_ring_id] = 0;
          c0 += TILE_N;
        } while (c0 < dlen);
        ++uc;
      }
      if (ok && elect) {
        // tell the epilogue groups how many units there were
        __threadfence_block();
        ctl->units_total = (int)uc;
      }
      if (ok) {
        // tell the issuer that the stream has ended
        ok = wait_bar<FP8>(&ctl->d_empty[st], ph ^ 1, ctl, P.status);
        if (ok) {
          if (elect) ctl->stage_info[st] = STAGE_END;
          if (lane == 0) mbar_arrive(smem_u32(&ctl->d_full[st]));
        }
      }
      if (elect) {
        // let the copies already issued land before the CTA goes away: an issuer that gives up takes no more of them
        if (!PLAID) {
          // (the end of the stream has completed a phase of slot `st` without a copy: its copy before that has been taken)
          for (uint32_t i = 1; i <= (uint32_t)P.stages - (ok ? 1u : 0u) && i <= n_dload; ++i) {
            const bool wrapped = i > st;  // that use lies before the last wrap of the ring
            const uint32_t slot = wrapped ? st + (uint32_t)P.stages - i : st - i;
            const uint32_t bar = smem_u32(&ctl->d_full[slot]);
            for (int spin = 0; spin < (1 << 16) && !mbar_try_wait_long(bar, wrapped ? ph ^ 1 : ph); ++spin) {
            }
          }
        }
        if (n_qload) {
          const uint32_t bar = smem_u32(&ctl->q_full);
          for (int spin = 0; spin < (1 << 16) && !mbar_try_wait_long(bar, (n_qload - 1) & 1); ++spin) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // =========================== MMA issuer ===========================
    // Driven by the stage words alone.  The whole warp runs the loop on warp-uniform values (the stage word is broadcast from
    // lane 0, which also tells the compiler that it is uniform) and one elected lane issues: tcgen05.mma takes its
    // descriptors from uniform registers, and with the loop under `lane == 0` every MMA paid about 100 cycles for moving
    // them there, whatever its width.
    uint32_t st = 0, ph = 0, q_ph = 0, acc_ph = 0;  // acc_ph: one phase bit per accumulator
    bool ok = true;
    const bool issue = elect_one();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const uint32_t a_desc0 = (uint32_t)smem_desc_sw128(smem_u32(q_smem));
    const uint32_t b_desc0 = (uint32_t)smem_desc_sw128(smem_u32(d_smem));
    const uint32_t stage_desc = (uint32_t)(d_stage_bytes >> 4);
    const uint32_t a_tile1 = P.mt == 2 ? (uint32_t)(q_tile_bytes >> 4) : 0u;  // descriptor offset of the second resident tile
    const uint32_t idesc0 = instr_desc(P.ab_format, 0);
    const int k_steps = P.k_steps;
    constexpr uint32_t A_SLAB = (TILE_M * SLAB_BYTES_ROW) >> 4, B_SLAB = (TILE_N * SLAB_BYTES_ROW) >> 4;
    while (ok) {
      ok = wait_bar_warp<FP8>(&ctl->d_full[st], ph, ctl, P.status);
      if (!ok) break;
      const uint32_t info = __shfl_sync(0xffffffffu, ctl->stage_info[st], 0);
      if (info & STAGE_END) break;
      if (info & STAGE_FIRST) {
        ok = wait_bar_warp<FP8>(&ctl->q_full, q_ph, ctl, P.status);
        if (!ok) break;
        q_ph ^= 1;
      }
      const uint32_t ncols = info & STAGE_COLS_MASK;
      const uint32_t idesc = idesc0 | (((ncols + 15) >> 4) << 18);  // N / 8 in bits 17..22
      const uint32_t b_stage = b_desc0 + st * stage_desc;
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        if (!ok || !(info & (STAGE_ACC0 << a))) continue;
        ok = wait_bar_warp<FP8>(&ctl->acc_empty[a], ((acc_ph >> a) & 1u) ^ 1u, ctl, P.status);
        if (!ok) continue;
        acc_ph ^= 1u << a;
        tc_fence_after();
        if (issue) {
          if (ncols) {  // (an empty document: the accumulator still changes hands so that both sides keep their phase)
            const uint32_t d_tmem = tmem_base + (uint32_t)(a * ACC_COLS);
            const uint32_t a_desc = a_desc0 + (a ? a_tile1 : 0u);
            // descriptors differ only in the start address, in units of 16 bytes
            if (k_steps == 8) {  // the common width (128 two-byte or 256 one-byte elements): straight-line issue
#pragma unroll
              for (int k = 0; k < 8; ++k)
                tc_mma<FP8>(d_tmem, a_desc + (uint32_t)((k & 3) * 2) + (k >> 2) * A_SLAB, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * B_SLAB, desc_hi,
                            idesc, k ? 1u : 0u);
            } else {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (k < k_steps)
                  tc_mma<FP8>(d_tmem, a_desc + (uint32_t)((k & 3) * 2) + (k >> 2) * A_SLAB, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * B_SLAB,
                              desc_hi, idesc, k ? 1u : 0u);
            }
          }
          tc_commit(smem_u32(&ctl->acc_full[a]));
        }
        __syncwarp();
      }
      if (!ok) break;
      if (issue) {
        tc_commit(smem_u32(&ctl->d_empty[st]));                     // ring slot reusable once these MMAs retire
        if (info & STAGE_LAST) tc_commit(smem_u32(&ctl->q_empty));  // and so are the query tiles
      }
      __syncwarp();
      if (++st == (uint32_t)P.stages) { st = 0; ph ^= 1; }
    }
  } else if (warp < 2 + 2 * GROUP_WARPS) {
    // =========================== epilogue groups ===========================
    // Group g (eight warps) drains accumulator g.  Its two halves split the 32-column chunks of a tile
    // between them (even chunks / odd chunks); half 1 hands its per-row result to half 0, which sums
    // the rows of every query and writes the score.  (group, document) advance locally; a document's
    // length and first row come from the producer's unit ring.
    const int e = warp - 2;
    const int wg = e >> 3;                   // accumulator / epilogue group
    const int sub = (e >> 2) & 1;            // half of the group
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int wq = e & 3;                    // warp index inside the half
    const int row = quad * 32 + lane;        // accumulator row == query token slot in the tile
    const int et = wq * 32 + lane;           // thread index inside the half (0..127)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(wg * ACC_COLS);
    const uint32_t acc_empty_bar = smem_u32(&ctl->acc_empty[wg]);
    int cur_grp = -1;
    uint32_t n_acc = 0, n_emit = 0, n_doc = 0;
    int uc = 0;
    bool ok = true;
    // per-row / per-warp state for the resident query tile
    bool have_tile = false, warp_rows = false, in_seg = false, row_ok = false, aligned = false;
    float my_qf = 1.f;
    int tile_id = 0;
    long long arg_off = -1;   // ARGMAX: offset of this row's slot for document 0 (-1: row stores nothing)
    long long warp_out = -1;  // aligned tiles: offset of this warp's query score for document 0
    int my_list = -1;         // top-k: the list whose state thread `et` (half 0) loaded into shared memory
    int warp_seg = -1;        // aligned tiles: the query (segment) of this warp's rows
    // Rendezvous of the whole group / of half 0 on hardware named barriers: a waiting warp issues
    // nothing.  Nobody waits on anything else between two of them, so every warp of the group always
    // arrives; the only bounded waits of a group (for a unit, for the accumulator) are done by its first warp,
    // which tells the others whether to go on through the rendezvous itself: a barrier that counts the
    // threads arriving with a true predicate (0: go on, 1: the wait gave up, 2: the stream has ended).
    const bool leader = (e & 7) == 0;
#define LIK_GRP_SYNC_COUNT(pred_, count_out_)                                                                        \
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\tbar.red.popc.u32 %0, %1, %2, q;\n\t}"              \
               : "=r"(count_out_) : "r"(1 + wg), "r"(2 * EPI_THREADS), "r"((int)(pred_)) : "memory")
#define LIK_GRP_SYNC() asm volatile("bar.sync %0, %1;" ::"r"(1 + wg), "r"(2 * EPI_THREADS) : "memory")
#define LIK_SUB_SYNC() asm volatile("bar.sync %0, %1;" ::"r"(3 + wg), "r"(EPI_THREADS) : "memory")
#define LIK_GROUP_WAIT_ACC()                                                         \
  do {                                                                               \
    bool gave_up_ = false;                                                           \
    if (leader) gave_up_ = !wait_bar<FP8>(&ctl->acc_full[wg], n_acc & 1, ctl, P.status);  \
    int n_;                                                                          \
    LIK_GRP_SYNC_COUNT(gave_up_ && lane == 0, n_);                                   \
    ok = n_ == 0;                                                                    \
  } while (0)
    // top-k: write the state of the lists this thread loaded back to their headers
#define LIK_TOPK_STORE_BACK()                                                                          \
  do {                                                                                                 \
    if (topk && sub == 0 && my_list >= 0) {                                                            \
      P.topk.hdr[my_list] = make_int2(ctl->seg_cnt[wg][et], (int)ctl->seg_thr[wg][et]);                \
      my_list = -1;                                                                                    \
    }                                                                                                  \
  } while (0)
    // one (query, document) score: stored, or offered to the query's candidate list (warp-uniform)
#define LIK_EMIT_SCORE(sg_, value_, offset_)                                                           \
  do {                                                                                                 \
    if (!topk) {                                                                                       \
      if (lane == 0) P.scores[offset_] = (value_);                                                     \
    } else {                                                                                           \
      const float key_ = (P.topk.largest ? (value_) : -(value_)) + 0.f;                                \
      const unsigned ukey_ = ordered_key(key_);                                                        \
      if (ukey_ > ctl->seg_thr[wg][sg_]) {                                                             \
        int cnt_ = ctl->seg_cnt[wg][sg_];                                                              \
        if ((unsigned)cnt_ >= (unsigned)TOPK_CAP || (unsigned)ctl->seg_list[wg][sg_] >= (unsigned)P.topk.n_lists) {  \
          if (lane == 0 && P.status) atomicOr(P.status, LIK_DEV_INTERNAL);                             \
          break;                                                                                       \
        }                                                                                              \
        float* keys_ = P.topk.cand_key + (long long)ctl->seg_list[wg][sg_] * TOPK_CAP;                 \
        int* idx_ = P.topk.cand_idx + (long long)ctl->seg_list[wg][sg_] * TOPK_CAP;                    \
        if (lane == 0) {                                                                               \
          keys_[cnt_] = key_;                                                                          \
          idx_[cnt_] = doc + P.topk.doc_base;                                                          \
        }                                                                                              \
        ++cnt_;                                                                                        \
        __syncwarp();                                                                                  \
        if (cnt_ == TOPK_CAP) {                                                                        \
          const unsigned thr_ = topk_compact(keys_, idx_, P.topk.k, lane);                             \
          cnt_ = P.topk.k;                                                                             \
          if (lane == 0) ctl->seg_thr[wg][sg_] = thr_;                                                 \
        }                                                                                              \
        if (lane == 0) ctl->seg_cnt[wg][sg_] = cnt_;                                                   \
        __syncwarp();                                                                                  \
      }                                                                                                \
    }                                                                                                  \
  } while (0)

    const bool cross = P.pairing == LIK_PAIR_CROSS;
    const bool bulk = SCALED && P.sc_slots != 0;  // the multipliers of a tile arrive with it, or are made from it
    const bool every_group_full = P.mt == 1 || (n_tiles & 1) == 0;
    for (;; ++uc) {
      // with one resident tile the two groups take alternate units
      if (P.mt == 1 && (uc & 1) != wg) continue;
      // The unit (tile group, document, length, first row) comes from the producer's ring.  The group's first warp
      // waits for its publication and - in kernels without per-column multipliers, which have nothing to prepare
      // while the MMAs run - for the unit's first accumulator, when this group has a tile in the unit's tile group.
      int st_ = 1;
      if (leader) {
        st_ = wait_posted(ctl, uc, P.status);
        if (st_ == 1 && !SCALED) {
          // (only the last tile group can lack this group's tile, and only when the tile count is odd)
          const bool mine_ = every_group_full || ctl->unit_info[uc & (UNIT_RING - 1)].z * P.mt + wg < n_tiles;
          if (mine_ && !wait_bar<FP8>(&ctl->acc_full[wg], n_acc & 1, ctl, P.status)) st_ = 0;
        }
      }
      {
        // the first warp arrives with one true predicate when its wait gave up, with two when the stream has ended
        int state_;
        LIK_GRP_SYNC_COUNT((st_ == 0 && lane == 0) || (st_ == 2 && lane < 2), state_);
        ok = state_ != 1;
        if (state_ != 0) break;
      }
      const int4 uinfo = ctl->unit_info[uc & (UNIT_RING - 1)];
      const int grp = uinfo.z;
      const int doc = uinfo.w;
      // (a group number out of range cannot index anything: its tile number fails the range check below)
      if (grp != cur_grp) {
        cur_grp = grp;
        // (re)build the segment table of this group's tile `wg` (mt == 2) or tile 0 (mt == 1: both groups)
        const int m = P.mt == 2 ? wg : 0;
        tile_id = grp * P.mt + m;
        have_tile = (unsigned)tile_id < (unsigned)n_tiles;
        LIK_GRP_SYNC();  // everyone in the group is done reading the old table
        LIK_TOPK_STORE_BACK();
        TileInfo ti{};
        int nseg = 0;
        if (have_tile) {
          ti = tile_info(P, tile_id);
          nseg = ti.qb - ti.qa;
          if (sub == 0) {
            ctl->row_seg[wg][et] = -1;
            if (et == 0) {
              ctl->n_seg[wg] = nseg;
              ctl->warp_aligned[wg] = P.q_chunks == 1 ? 1 : 0;
            }
          }
        }
        LIK_GRP_SYNC();
        if (have_tile && sub == 0 && et < nseg) {
          long long r0;
          int len;
          seq_bounds(P.q, ti.qa + et, r0, len, P.status);
          int off, l;
          if (P.q_chunks == 1) {
            off = (int)(r0 - ti.row0);
            l = len;
            if (off + l > TILE_M) {  // max_len was smaller than a real query: report, stay in bounds
              l = max(0, TILE_M - off);
              if (P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
            }
          } else {
            off = 0;
            l = min(TILE_M, max(0, len - ti.chunk * TILE_M));
            if (len > P.q_chunks * TILE_M && P.status) atomicOr(P.status, LIK_DEV_LEN_RANGE);
          }
          // an empty query owns no accumulator row, so only the per-query pass below can write its zero
          if ((off & 31) != 0 || l > 32 || l == 0) ctl->warp_aligned[wg] = 0;
          if (ARGMAX && len > P.argmax_stride && P.status) atomicOr(P.status, LIK_DEV_ARGMAX_STRIDE);
          ctl->seg_off[wg][et] = off;
          ctl->seg_len[wg][et] = l;
          ctl->seg_q[wg][et] = ti.qa + et;
          for (int i = 0; i < l; ++i) ctl->row_seg[wg][off + i] = (short)et;
          if (topk) {
            // the candidate list of (this CTA, this group, this query)
            // (with one resident tile the two epilogue groups take alternate documents: a list each)
            my_list = ((int)blockIdx.x + grp) * P.topk.qpg + (P.mt == 2 ? m : wg) * P.q_per_tile + et;
            if ((unsigned)my_list >= (unsigned)P.topk.n_lists) {
              if (P.status) atomicOr(P.status, LIK_DEV_INTERNAL);
              my_list = 0;
            }
            const int2 hd = P.topk.hdr[my_list];
            ctl->seg_list[wg][et] = my_list;
            ctl->seg_cnt[wg][et] = hd.x;
            ctl->seg_thr[wg][et] = (unsigned)hd.y;
          }
        }
        LIK_GRP_SYNC();
        in_seg = false;
        row_ok = false;
        arg_off = -1;
        warp_out = -1;
        warp_seg = -1;
        aligned = have_tile && ctl->warp_aligned[wg] != 0;
        if (have_tile) {
          const int sg = ctl->row_seg[wg][row];
          if (sg >= 0) {
            in_seg = true;
            const int my_q = ctl->seg_q[wg][sg];
            const int my_s = row - ctl->seg_off[wg][sg] + ti.chunk * TILE_M;
            const long long qrow = ti.row0 + row;
            row_ok = row_valid(P.q, qrow);
            my_qf = row_factor(P.q, qrow);
            if (ARGMAX && my_s < P.argmax_stride)
              arg_off = (cross ? (long long)my_q * P.n_d : 0ll) * P.argmax_stride + my_s;
          }
          warp_rows = __any_sync(0xffffffffu, in_seg);
          const int sg0 = ctl->row_seg[wg][quad * 32];
          if (aligned && sg0 >= 0) {
            warp_seg = sg0;
            warp_out = cross ? (long long)ctl->seg_q[wg][sg0] * P.n_d : 0ll;
          }
        }
      }
      // a tile group with an odd tile out: the second epilogue group has nothing in it
      if (!have_tile) continue;
      const int dlen = uinfo.x & UNIT_LEN_MASK;
      int sc_slot = SCALED ? (uinfo.x >> UNIT_SLOT_SHIFT) & 31 : 0;  // multiplier slot of the unit's first tile
      const int sc_base = SCALED && sc_slot >= P.sc_per ? P.sc_per : 0;  // first slot of its ring
      const long long drow0 = uinfo.y;
      const bool holes = (uinfo.x & LEN_FLAG_MASKED) != 0;  // the document's mask is not a plain prefix
      // where this unit's results go: CROSS / GROUPED index by document, LIST by pair (== unit)
      const long long out_col = doc;
      float run_m = -INFINITY;
      int run_i = -1;
      int c0 = 0;
      // The tiles of the document.  The body exists twice in the kernels without per-column multipliers: documents whose
      // mask is a plain prefix (nearly all) take the copy that has no column arrays in it, the others the general one -
      // the common path's time goes with its code size, so the rare one stays out of it.
      auto document_tiles = [&](auto general_, auto lazy_) {
      constexpr bool general = decltype(general_)::value;  // the document's mask has holes
      constexpr bool lazy = decltype(lazy_)::value;        // long document: winner scan only when some row of the warp needs it
      constexpr bool use_cols = SCALED || general;          // per-column multiplier / additive mask needed
      do {
        const int ncols = max(0, min(TILE_N, dlen - c0));
        // per-column arrays of this tile.  They may be written once the previous tile's readers are done with them (a
        // rendezvous, unless the one at the top of the unit already stands between), and read after one more rendezvous.
#define LIK_STAGE_COLUMNS(sync_before_)                                                                   \
  do {                                                                                                    \
    if (sync_before_) LIK_GRP_SYNC();                                                                     \
    for (int c = sub * EPI_THREADS + et; c < ((ncols + 31) & ~31); c += 2 * EPI_THREADS) {                \
      float sc = 1.f, bi = -INFINITY;                                                                     \
      if (c < ncols) {                                                                                    \
        const long long drow = drow0 + c0 + c;                                                            \
        sc = norm_warps ? sc_ring[sc_slot * TILE_N + c] : row_factor(P.d, drow);                          \
        bi = row_valid(P.d, drow) ? 0.f : -INFINITY;                                                      \
      }                                                                                                   \
      ctl->col_scale[wg][c] = sc;                                                                         \
      ctl->col_bias[wg][c] = bi;                                                                          \
    }                                                                                                     \
  } while (0)
        // before the accumulator wait: overlaps the MMAs; the wait's rendezvous also publishes the columns
        // (not needed when the multipliers came with the tile and the mask has no holes)
        const bool staged = SCALED && (general || !bulk) && !norm_warps;
        if (staged) LIK_STAGE_COLUMNS(c0 > 0);
        if (SCALED || c0 > 0) {
          LIK_GROUP_WAIT_ACC();
          if (!ok) break;
        }
        ++n_acc;
        if (general && (!SCALED || norm_warps)) {  // a document whose mask has holes: known only now, or its multipliers are
          LIK_STAGE_COLUMNS(true);
          LIK_GRP_SYNC();
        }
#undef LIK_STAGE_COLUMNS
        tc_fence_after();
        // the accumulator goes back to the issuer as soon as this warp's last columns sit in registers
#define LIK_RELEASE_ACC()                                          \
  do {                                                             \
    tc_fence_before();                                             \
    __syncwarp();                                                  \
    if (lane == 0) mbar_arrive(acc_empty_bar);                     \
  } while (0)
        // chunks of this half: cc, cc + 64, ...; only the tile's last chunk can be partial
        // (a warp without a query row, as most have under a single short query, only hands the accumulator on)
        int cc = warp_rows ? sub * 32 : ncols;
        if (cc >= ncols) LIK_RELEASE_ACC();
        if (use_cols && general) {
          // a mask with holes: every chunk takes multiplier and additive mask
          for (; cc < ncols; cc += 64) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (cc + 64 >= ncols) LIK_RELEASE_ACC();
            affine32(v, &ctl->col_scale[wg][cc], &ctl->col_bias[wg][cc]);  // bias is -inf past ncols and in holes
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
        } else if (use_cols) {
          // whole chunks are valid: multiplier only; the partial last chunk also takes the mask (-inf past ncols).
          // Multipliers that came with the tile sit in a ring slot that is refilled once the accumulator has changed
          // hands often enough: there the accumulator goes back after the last read of them, not before.
          const float* sc_arr = bulk ? sc_ring + sc_slot * TILE_N : ctl->col_scale[wg];
          for (; cc + 32 <= ncols; cc += 64) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (!bulk && cc + 64 >= ncols) LIK_RELEASE_ACC();
            scale32(v, sc_arr + cc);
            if (bulk && cc + 64 >= ncols) LIK_RELEASE_ACC();
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
          if (cc < ncols) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (bulk) {
              scale32_first(v, sc_arr + cc, ncols - cc);
              LIK_RELEASE_ACC();
            } else {
              LIK_RELEASE_ACC();
              affine32(v, &ctl->col_scale[wg][cc], &ctl->col_bias[wg][cc]);
            }
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
        } else {
          for (; cc + 32 <= ncols; cc += 64) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (cc + 64 >= ncols) LIK_RELEASE_ACC();
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
          if (cc < ncols) {  // the partial last chunk
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            LIK_RELEASE_ACC();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = cc + i < ncols ? v[i] : -INFINITY;
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
        }
#undef LIK_RELEASE_ACC
        c0 += TILE_N;
        if (SCALED && ++sc_slot >= sc_base + P.sc_per) sc_slot = sc_base;
      } while (c0 < dlen);
      };
      // (long documents, WINNERS == 2: most 32-column chunks past the first few hundred tokens hold no new maximum for any
      // of a warp's rows, and the scan for its column is skipped there)
      if (holes) document_tiles(std::true_type{}, std::false_type{});
      else document_tiles(std::false_type{}, std::integral_constant<bool, WINNERS == 2>{});
      if (!ok) break;
      // ---- end of document: half 1 hands over, half 0 merges (lower column wins a tie) ----
      float* xm = ctl->xch_m[wg][n_doc & 1];
      int* xi = ctl->xch_i[wg][n_doc & 1];
      ++n_doc;
      if (sub == 1) {
        xm[row] = run_m;
        if (ARGMAX) xi[row] = run_i;
      }
      LIK_GRP_SYNC();
      if (sub == 1) continue;
      {
        const float m1 = xm[row];
        if (ARGMAX) {
          const int i1 = xi[row];
          const bool take = (i1 >= 0) & ((run_i < 0) | (m1 > run_m) | ((m1 == run_m) & (i1 < run_i)));
          run_m = take ? m1 : run_m;
          run_i = take ? i1 : run_i;
        } else {
          run_m = fmaxf(run_m, m1);
        }
      }
      // one value per row, summed per query in a fixed order
      const bool has_winner = ARGMAX ? (run_i >= 0) : (run_m != -INFINITY);
      const float val = (in_seg && row_ok && has_winner) ? run_m * my_qf : 0.f;
      if (ARGMAX && arg_off >= 0) P.argmax[arg_off + out_col * P.argmax_stride] = has_winner ? run_i : -1;
      if (aligned) {
        // one query per warp: a shuffle tree (fixed order) replaces the shared-memory pass
        const float sum = warp_sum(val);
        if (warp_out >= 0) LIK_EMIT_SCORE(warp_seg, sum, warp_out + out_col);
        continue;
      }
      float* ebuf = ctl->emit[wg][n_emit & 1];
      ++n_emit;
      ebuf[row] = val;
      LIK_SUB_SYNC();
      const int nseg = ctl->n_seg[wg];
      for (int sg = wq; sg < nseg; sg += 4) {
        const int off = ctl->seg_off[wg][sg], len = ctl->seg_len[wg][sg];
        float sum = 0.f;
        for (int i = lane; i < len; i += 32) sum += ebuf[off + i];
        sum = warp_sum(sum);
        const int qq = ctl->seg_q[wg][sg];
        if (P.q_chunks == 1) {
          const long long o = cross ? (long long)qq * P.n_d + out_col : out_col;
          LIK_EMIT_SCORE(sg, sum, o);
        } else if (lane == 0) {
          P.partial[(long long)tile_id * P.n_d + doc] = sum;
        }
      }
    }
    // top-k: leave the lists' state where the next launch stage (the merge) finds it
    if (sub == 0) {
      LIK_SUB_SYNC();
      LIK_TOPK_STORE_BACK();
    }
#undef LIK_EMIT_SCORE
#undef LIK_TOPK_STORE_BACK
#undef LIK_GROUP_WAIT_ACC
#undef LIK_GRP_SYNC
#undef LIK_GRP_SYNC_COUNT
#undef LIK_SUB_SYNC
  } else if (SCALED && !FP8 && !PLAID && norm_warps) {
    // =========================== inverse norms of the tiles ===========================
    // The multipliers of a tile go into its ring slot, and the arrival that announces them belongs to the phase of the
    // accumulator(s) that the tile feeds: the epilogue waits for both with one wait.  An arrival must not fall into the
    // phase before, hence the wait for that one; it also says that the epilogue is done with the slots three tiles back.
    const int nw = warp - (2 + 2 * GROUP_WARPS);
    uint32_t st = 0, ph = 0, n_acc[2] = {0, 0};
    int sc_cnt[2] = {0, 0};
    bool ok = true;
    const bool bf16 = P.ab_format == 1, two_slabs = P.n_slabs == 2;
    while (ok) {
      ok = wait_bar_warp<FP8>(&ctl->d_full[st], ph, ctl, P.status);
      if (!ok) break;
      const uint32_t info = __shfl_sync(0xffffffffu, ctl->stage_info[st], 0);
      if (info & STAGE_END) break;
      const int ncols = (int)(info & STAGE_COLS_MASK);
      const int ring = (info & STAGE_ACC0) ? 0 : 1;
      float* slot = sc_ring + (ring * P.sc_per + sc_cnt[ring]) * TILE_N;
      const unsigned char* stage = d_smem + (size_t)st * d_stage_bytes;
      for (int r = nw * 32 + lane; r < ncols; r += NORM_WARPS * 32) {
        const float ss = bf16 ? stage_row_sum_sq<__nv_bfloat16>(stage + r * SLAB_BYTES_ROW, r, two_slabs)
                              : stage_row_sum_sq<__half>(stage + r * SLAB_BYTES_ROW, r, two_slabs);
        slot[r] = inv_norm(ss, P.norm_eps);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->d_empty[st]));
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        if (!ok || !(info & (STAGE_ACC0 << a))) continue;
        if (n_acc[a]) ok = wait_bar_warp<FP8>(&ctl->acc_full[a], (n_acc[a] - 1) & 1, ctl, P.status);
        if (ok && lane == 0) mbar_arrive(smem_u32(&ctl->acc_full[a]));
        ++n_acc[a];
      }
      // the odd tile out of a pair feeds one accumulator only: the other's epilogue must be done with the ring they share
      if (ok && P.mt == 2 && !(info & STAGE_ACC1) && n_acc[1]) ok = wait_bar_warp<FP8>(&ctl->acc_empty[1], (n_acc[1] - 1) & 1, ctl, P.status);
      if (++sc_cnt[ring] >= P.sc_per) sc_cnt[ring] = 0;
      if (++st == (uint32_t)P.stages) { st = 0; ph ^= 1; }
    }
  }

  // ---- teardown (also reached when aborting: every wait above is bounded) ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// The bounded wait of the kernel above, alone: one thread waits on a barrier that nothing ever arrives at, with a
// limit the caller chooses.  It must give up after that many cycles, raise LIK_DEV_WAIT_TIMEOUT in the status word,
// set the abort flag and return - the path every role of the scoring kernel takes when a hand-shake never comes.
// result[0] = what the wait returned (0 = gave up), result[1] = the abort flag, result[2] = cycles spent.
template <bool INLINE>
__global__ void wait_probe_kernel(long long limit, int* status, int* result) {
  __shared__ SharedCtl ctl;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctl.q_full), 1);
    ctl.abort_flag = 0;
    ctl.wait_limit = limit;
    fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    const bool got = wait_bar<INLINE>(&ctl.q_full, 0, &ctl, status);
    const long long dt = clock64() - t0;
    result[0] = got ? 1 : 0;
    result[1] = ctl.abort_flag;
    result[2] = dt > 0x7fffffffll ? 0x7fffffff : (int)dt;
  }
}

// One row of the pair-list table per pair: the query (0 when the pair is out of range, which is reported
// through the status word and scores 0 because its document is then empty), the first row and the length of
// the document.
__global__ void list_units_kernel(SeqView q, SeqView d, const int* __restrict__ pair_q, const int* __restrict__ pair_d,
                                  long long n_pairs, int4* __restrict__ tab, int* status) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_pairs) return;
  const int i = pair_q[p], j = pair_d[p];
  int4 t = make_int4(0, 0, 0, 0);
  if (i < 0 || i >= q.n_seq || j < 0 || j >= d.n_seq) {
    if (status) atomicOr(status, LIK_DEV_PAIR_RANGE);
  } else {
    long long r0;
    int len;
    seq_bounds(d, j, r0, len, status);
    t = make_int4(i, (int)r0, len, 0);
  }
  tab[p] = t;
}

constexpr int PACK_MAX_QUERIES = 8192;  // offsets are staged in shared memory; larger batches use fixed groups

// Greedy packing of ragged queries into 128-row tiles: a tile takes whole consecutive queries until the next
// one would not fit (or it holds 128 queries; empty ones take no rows).  out[0] = tile count, out[1 + m] =
// first query of tile m (out[1 + count] = n_q).  One CTA: the offsets go to shared memory, every thread finds
// by bisection where a tile starting at its query would end, then one thread follows those links.
__global__ void __launch_bounds__(256) pack_query_tiles_kernel(const int* __restrict__ cu, int n_q, int* __restrict__ out) {
  __shared__ int s_cu[PACK_MAX_QUERIES + 1];
  __shared__ unsigned char s_span[PACK_MAX_QUERIES];  // queries in the tile that starts at query i (1..128)
  for (int i = threadIdx.x; i <= n_q; i += blockDim.x) s_cu[i] = cu[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n_q; i += blockDim.x) {
    int lo = i + 1, hi = min(i + TILE_M, n_q);  // the tile ends at some j in [lo, hi]; a lone long query still gets one
    const int base = s_cu[i];
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_cu[mid] - base <= TILE_M) lo = mid;
      else hi = mid - 1;
    }
    s_span[i] = (unsigned char)(lo - i - 1);  // stored minus one so that 128 fits a byte
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int tiles = 0, q = 0;
    out[1] = 0;
    while (q < n_q) {
      q += (int)s_span[q] + 1;
      ++tiles;
      out[1 + tiles] = q;
    }
    if (tiles == 0) {  // n_q == 0 cannot reach this kernel; keep the table well formed anyway
      tiles = 1;
      out[2] = n_q;
    }
    out[0] = tiles;
  }
}

// scores[q, j] = sum over the chunks of query q, in chunk order
__global__ void reduce_chunks_kernel(const float* __restrict__ partial, int n_q, int n_d, int q_chunks, float* __restrict__ scores) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n_q * n_d) return;
  const int q = (int)(idx / n_d), j = (int)(idx - (long long)q * n_d);
  float s = 0.f;
  for (int c = 0; c < q_chunks; ++c) s += partial[((long long)q * q_chunks + c) * n_d + j];
  scores[idx] = s;
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int make_map(CUtensorMap* map, const lik_seqs& s, int dtype, int dim, int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled is not available from this driver");
    return LIK_ERR_CUDA;
  }
  const int eb = (int)dtype_size(dtype);
  CUtensorMapDataType dt = dtype == LIK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                           : dtype == LIK_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                              : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  cuuint64_t gdim[2] = {(cuuint64_t)dim, (cuuint64_t)(s.n_rows > 0 ? s.n_rows : 1)};
  cuuint64_t gstride[1] = {(cuuint64_t)s.row_stride * eb};
  cuuint32_t box[2] = {(cuuint32_t)(SLAB_BYTES_ROW / eb), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, dt, 2, const_cast<void*>(s.data), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return LIK_ERR_CUDA;
  }
  return LIK_OK;
}

constexpr size_t SB_WINDOW_BYTES = 48u << 20;   // documents of one super-block: stays in L2 while every group passes
// LIK_SB_WINDOW_MB overrides the window (a tuning knob; document sets below twice the window are walked as one block)
static size_t sb_window_bytes() {
  static size_t v = 0;
  if (!v) {
    const char* e = getenv("LIK_SB_WINDOW_MB");
    const long mb = e ? atol(e) : 0;
    v = mb > 0 ? (size_t)mb << 20 : SB_WINDOW_BYTES;
  }
  return v;
}

// A launch that reads every document up to four times takes the documents' norms from its tiles instead of one pass of
// prep_kernel in front.  A query of 32 tokens against 1000 documents of up to 300 40 -> 30 us; two groups of query tiles (12 x 32
// against 8000 of 300) 407 -> 308, (4 x 128 against 8000 of 1030) 1498 -> 953; 128-token queries against 4000 documents of up
// to 500: three groups 458 -> 394, four 540 -> 484, five 646 -> 611, six 740 -> 724, eight 921 -> 930: the two warps take every
// norm once per group.
bool norms_from_tiles(const lik_fwd_args& a, const TcExtra& x, const TcPlan& pl) {
  if (!(a.normalize & LIK_NORM_D) || x.plaid || (a.dtype != LIK_BF16 && a.dtype != LIK_F16) || a.d.scale || a.d.scale_scalar != 1.0f) return false;
  return a.pairing == LIK_PAIR_GROUPED || (a.pairing == LIK_PAIR_CROSS && pl.n_groups <= 4);
}

// Candidate lists of a fused top-k: a slot per CTA and tile group (see TopkOut).
size_t topk_list_bytes(int n_groups, int per_slot) {
  return (size_t)(sm_count() + n_groups) * per_slot * (TOPK_CAP * (sizeof(float) + sizeof(int)) + sizeof(int2));
}
// The streams kernel keeps twice as many of them, which is a matter of megabytes for the batches that wait for an answer (256
// queries of 32 tokens: 6 MB).  Beyond this the other kernel runs: 100 000 queries would take 414 MB instead of 207.
constexpr size_t STREAMS_LISTS_BYTES = 128u << 20;

// Which kernel takes a problem that both can: true for the one with two streams per CTA.  Times in us, the other kernel / streams,
// bf16, 128 features, queries of 32 tokens, document lengths spread from a fifth of the longest to the longest unless said otherwise;
// "units" are per SM.  What the streams kernel loses by: a longer start (query tiles on their way through shared to tensor memory),
// the same way again with both streams idle whenever the query tiles change, and documents of more than 100 up to 256
// tokens, which are two or three pieces there and one tile in the other kernel.
bool streams_pay(const lik_fwd_args& a, const TcExtra& x, const TcPlan& pl, bool multipliers) {
  const long long sms = sm_count(), len = a.d.max_len;
  const bool two = pl.mt == 2, list = a.pairing == LIK_PAIR_LIST;
  const bool brief = len <= 100, middle = !brief && len <= 256;
  // Plain scores of documents that are all of one length and fill their last tile of 256: 64 queries x 445 documents of 256 tokens
  // 53.7 / 55.2, of 512 84.6 / 87.6 (of 300: 76.2 / 62.5; of 700 even).
  if (!a.argmax && !multipliers && !a.d.cu && !a.d.lens && !a.d.mask && (len - 1) % 256 + 1 > 192) return false;
  // Units.  One query x documents of 64 tokens: 6 units 13.8 / 13.0, 12 17.2 / 14.0; of 192: 12 units 18.5 / 19.2, 24 32.6 / 27.3; of
  // 256: 16 units 26.2 / 26.5, 24 36.8 / 34.9; of 300: 12 1.03 to 1.17.  Two tiles, 64 queries x documents of 256: 8 units 23.4 /
  // 23.9, 12 29.5 / 29.3, with winners 34.4 / 32.2.  A pair list reads its table besides: 256 queries, documents of 300 tokens: 16 units
  // 31.6 / 32.8, 32 47.5 / 46.9, 48 65.2 / 60.8; of 200 tokens 48 units 0.99, 96 1.09; of 256 0.89 and 0.95.
  long long units = middle && !two ? 24 : 12;
  if (list && !brief) units = middle ? 96 : 32;
  // Units per change of the query tiles.  One tile, candidate lists with winners, 12 units, of 300 tokens: 1 per query 49.6 / 56.4, 2 (one for
  // either stream) 40.8 / 40.6 (of 512 1.10), 3 0.93, 4 35.1 / 36.5 (of 512 1.03), 6 1.04, 8 35.6 / 32.8; of 192 tokens, 24 units: 1 62.9 /
  // 77.4, 4 44.0 / 50.5, 8 39.0 / 40.9, 12 37.6 / 38.2, 16 37.6 / 36.4.  Two tiles, 12 units: documents of 64 tokens: 1 42.6 / 48.6, 2 35.7 / 29.8, 3
  // 0.94 to 1.09, 4 29.7 / 25.6; of 300: 2 0.88 to 0.98, 4 0.95 to 1.01, 6 39.9 / 37.7, 8 42.2 / 39.6.
  const long long have = a.pairing == LIK_PAIR_CROSS ? a.d.n_seq : list ? a.n_pairs / a.q.n_seq : a.group;
  const long long run = two ? (brief ? 4 : 8) : brief ? 1 : middle ? 12 : 6;
  if (have < run && !(have == 2 && (two ? brief : !middle))) return false;
  // Twice the candidate lists may need one more pass to merge (about 15 us): 40 queries over 500 documents of 180 tokens (17 units)
  // 51.5 / 59.1, 1000 (34) 77.4 / 79.5, 2000 (68) 126.3 / 108.9; of 1030 tokens 0.91 to 0.98 at any size.
  if (x.topk_k > 0 && topk_merge_parts((int)sms, pl.n_groups, 2 / pl.mt) == 1 && topk_merge_parts((int)sms, pl.n_groups, 4 / pl.mt) > 1) {
    if (len > 512) return false;
    units = 40;
  }
  return pl.n_units_total >= units * sms;
}

TcPlan plan_tc(const lik_fwd_args& a, const TcExtra& x) {
  TcPlan pl{};
  const int eb = (int)dtype_size(a.dtype);
  pl.n_slabs = (a.dim * eb + SLAB_BYTES_ROW - 1) / SLAB_BYTES_ROW;
  pl.k_steps = (a.dim * eb + 31) / 32;
  const int ml = a.q.max_len > 0 ? a.q.max_len : 1;
  pl.n_sb = 1;
  pl.sb_docs = a.d.n_seq > 0 ? a.d.n_seq : 1;
  if (a.pairing != LIK_PAIR_CROSS) {
    pl.q_per_tile = 1;
    pl.q_chunks = 1;
    pl.n_tiles = a.q.n_seq;
    pl.mt = 1;
    pl.n_groups = a.q.n_seq;
    pl.n_flat = a.pairing == LIK_PAIR_GROUPED ? a.d.n_seq : a.n_pairs;
    pl.n_units_total = pl.n_flat;
  } else {
    if (ml <= TILE_M) {
      pl.q_per_tile = TILE_M / ml;
      pl.q_chunks = 1;
      pl.n_tiles = (int)ceil_div(a.q.n_seq, pl.q_per_tile);
    } else {
      pl.q_per_tile = 1;
      pl.q_chunks = (int)ceil_div(ml, TILE_M);
      pl.n_tiles = a.q.n_seq * pl.q_chunks;
    }
    pl.mt = pl.n_tiles >= 2 ? 2 : 1;
    // packed queries shorter than the fixed slot: let the device pack them tightly (n_tiles becomes an upper bound)
    pl.pack_tiles = a.q.cu && ml < TILE_M && pl.q_per_tile > 1 && a.q.n_seq > 1 && a.q.n_seq <= PACK_MAX_QUERIES;
    pl.n_groups = (int)ceil_div(pl.n_tiles, pl.mt);
    pl.n_flat = 0;
    pl.n_units_total = (long long)pl.n_groups * a.d.n_seq;
    // large document sets are walked in L2-sized super-blocks (several tile groups read every document)
    const size_t row_bytes = x.plaid ? (size_t)(4 + x.plaid->packed_dim) : (size_t)a.dim * eb;
    const size_t d_bytes = (size_t)a.d.n_rows * row_bytes;
    if (a.d.n_seq > 0 && pl.n_groups > 1 && d_bytes > 2 * sb_window_bytes()) {
      const size_t per_doc = d_bytes / (size_t)a.d.n_seq + 1;
      long long sb = (long long)(sb_window_bytes() / per_doc);
      if (sb < 64) sb = 64;
      if (sb < a.d.n_seq) {
        pl.sb_docs = (int)sb;
        pl.n_sb = (int)ceil_div(a.d.n_seq, sb);
      }
    }
  }
  const bool norms = norms_from_tiles(a, x, pl);
  const bool multipliers = a.d.scale || ((a.normalize & LIK_NORM_D) && !x.plaid);
  const bool bulk = multipliers && !a.d.cu && a.d.seq_stride % 4 == 0 && a.d.n_rows % 4 == 0;
  // It takes no norms from the tiles and decodes no index; with one resident tile, per-column multipliers that arrive with the tiles
  // are the other kernel's (4 queries x 4096 documents of 256 tokens in e4m3: 43 against 53 us).  The candidate lists of a fused
  // top-k are laid out for one kernel: the pieces of a corpus go where LIK_TOPK_LARGE says, never by a piece's own size.
  const bool pieces = x.topk_flags & (LIK_TOPK_CONTINUE | LIK_TOPK_PARTIAL);
  pl.streams = !x.small_lists && !x.plaid && !norms && !(multipliers && pl.mt == 1 && (bulk || x.topk_k > 0)) &&
               (x.topk_k == 0 || topk_list_bytes(pl.n_groups, 4 * pl.q_per_tile) <= STREAMS_LISTS_BYTES) &&
               (pieces ? (x.topk_flags & LIK_TOPK_LARGE) != 0 : streams_pay(a, x, pl, multipliers));
  const long long g = pl.n_units_total < sm_count() ? pl.n_units_total : sm_count();
  pl.grid = (int)(g < 0 ? 0 : g);
  // the fused top-k numbers its candidate lists by CTA: the same grid whatever the piece of the corpus
  if (x.topk_k > 0 && pl.grid > 0) pl.grid = sm_count();
  const size_t q_bytes = 2 * (size_t)pl.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const size_t stage = pl.streams ? fwd_streams_stage_bytes(pl.n_slabs) : (size_t)pl.n_slabs * TILE_N * SLAB_BYTES_ROW;
  const size_t fixed = pl.streams ? fwd_streams_fixed_smem(pl.n_slabs) : q_bytes + sizeof(SharedCtl) + 1024;
  pl.stage_bytes = stage;
  pl.slot_bytes = pl.streams ? fwd_streams_slot_bytes() : TILE_N * sizeof(float);
  pl.lists = pl.streams ? 4 : 2;
  // Scores or a top-k of one query tile from a compressed index
  pl.decode = x.plaid && a.pairing == LIK_PAIR_CROSS && !a.argmax && !a.q.cu && a.q.max_len <= TILE_M && pl.n_tiles == 1;
  if (pl.decode) {
    pl.lists = 1;
    pl.grid = fwd_plaid_ctas_per_sm() * sm_count();
    pl.smem_bytes = fwd_plaid_smem(pl.n_slabs);
    pl.stages = 1;
    return pl;
  }
  const size_t budget = 227 * 1024;
  int st = (int)((budget - fixed) / stage);
  pl.stages = st > 8 ? 8 : st;
  pl.smem_bytes = fixed + (size_t)pl.stages * stage;
  return pl;
}

}  // namespace

// What the tcgen05 kernel takes.  `plaid`: the documents are a compressed index (a.d.data is NULL).
static bool tc_problem_ok(const lik_fwd_args& a, bool plaid) {
  // per device ordinal: a process may hold GPUs of different architectures
  static signed char dev_ok[64] = {0};  // 0 = not asked yet, 1 = usable, -1 = not usable
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev < 0 || dev >= 64) {
    if (!lik_device_supported()) return false;
  } else {
    if (dev_ok[dev] == 0) dev_ok[dev] = lik_device_supported() ? 1 : -1;
    if (dev_ok[dev] < 0) return false;
  }
  if (a.dtype != LIK_BF16 && a.dtype != LIK_F16 && a.dtype != LIK_E4M3) return false;
  if (plaid && a.dtype == LIK_E4M3) return false;
  if (a.pairing < LIK_PAIR_CROSS || a.pairing > LIK_PAIR_LIST) return false;
  const int eb = (int)dtype_size(a.dtype);
  if ((a.dim * eb) % 16 != 0 || a.dim * eb > MAX_SLABS * SLAB_BYTES_ROW) return false;
  if (a.q.n_seq <= 0 || a.d.n_seq <= 0 || a.q.n_rows <= 0 || a.d.n_rows <= 0) return false;
  if (a.q.max_len <= 0) return false;  // packed queries need their longest length to form tiles
  if (a.pairing != LIK_PAIR_CROSS && a.q.max_len > TILE_M) return false;  // one query per tile
  if (a.pairing == LIK_PAIR_LIST) {
    if (a.n_pairs <= 0 || a.n_pairs >= (1ll << 31) || !a.pair_q || !a.pair_d) return false;
    if (a.d.mask) return false;  // token masks with holes are not carried by the pair table
  }
  if ((a.q.row_stride * eb) % 16 != 0 || ((uintptr_t)a.q.data & 15)) return false;
  if (!plaid && ((a.d.row_stride * eb) % 16 != 0 || ((uintptr_t)a.d.data & 15))) return false;
  if (a.q.n_rows >= (1ll << 31) || a.d.n_rows >= (1ll << 31)) return false;
  if (a.argmax && a.argmax_stride < 0) return false;
  return get_encode_fn() != nullptr;
}

bool fwd_tc_supported(const lik_fwd_args& a) { return tc_problem_ok(a, false); }

// Helpers shared with the document-head kernel: a 128-byte-swizzled TMA map over the rows of a matrix whose box is
// one 128-byte K slab wide and `box_rows` high, and the effective document lengths under a token mask.
int make_tmap_rows(CUtensorMap* map, const void* data, int dtype, long long inner, long long n_rows, long long row_stride,
                   int box_rows) {
  lik_seqs s{};
  s.data = data;
  s.n_rows = n_rows;
  s.row_stride = row_stride;
  return make_map(map, s, dtype, (int)inner, box_rows);
}
bool tmap_available() { return get_encode_fn() != nullptr; }
// The fused top-k needs fixed query slots (padded queries of at most 128 tokens) and k within the list size.
bool fwd_tc_topk_supported(const lik_fwd_args& a, const TcExtra& x) {
  if (!tc_problem_ok(a, x.plaid != nullptr)) return false;
  if (a.pairing != LIK_PAIR_CROSS || a.q.cu || a.q.max_len > TILE_M || a.argmax) return false;
  return x.topk_k >= 1 && x.topk_k <= TOPK_CAP / 2;
}

bool fwd_tc_plaid_supported(const lik_fwd_args& a, const TcExtra& x) {
  if (!x.plaid || !tc_problem_ok(a, true)) return false;
  if (x.plaid->dim != a.dim || a.dim % 16 != 0 || a.dim > 128 || a.d.mask || a.d.scale) return false;
  return plaid_row16_ok(*x.plaid);
}

namespace {
struct TcWs {
  size_t partial, lens, tiles, list, hdr, keys, idx, merge, total;
  long long n_lists;
  int merge_parts;  // the lists of a query are merged in this many parts first (1: in one pass)
};
TcWs tc_ws_layout(const TcPlan& pl, const lik_fwd_args& a, const TcExtra& x) {
  TcWs w{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += align_up(bytes, 256);
    return o;
  };
  // the candidate lists first: their size depends on the queries and the machine only, so they keep their place
  // when the documents come in pieces
  w.n_lists = 0;
  if (x.topk_k > 0) {
    w.n_lists = (long long)(pl.grid + pl.n_groups) * pl.lists * pl.q_per_tile;
    w.hdr = take((size_t)w.n_lists * sizeof(int2));
    w.keys = take((size_t)w.n_lists * TOPK_CAP * sizeof(float));
    w.idx = take((size_t)w.n_lists * TOPK_CAP * sizeof(int));
    // few tile groups: a query has lists from many CTAs, which are merged in parts by as many CTAs first
    w.merge_parts = topk_merge_parts(pl.grid, pl.n_groups, pl.lists / pl.mt);
    w.merge = take(w.merge_parts > 1 ? (size_t)w.merge_parts * a.q.n_seq * x.topk_k * sizeof(long long) : 0);
  }
  w.partial = take(pl.q_chunks > 1 ? (size_t)pl.n_tiles * a.d.n_seq * sizeof(float) : 0);
  w.lens = take((a.d.mask && !a.d.cu) ? (size_t)a.d.n_seq * sizeof(int) : 0);
  w.tiles = take(pl.pack_tiles ? (size_t)(a.q.n_seq + 3) * sizeof(int) : 0);
  w.list = take(a.pairing == LIK_PAIR_LIST ? (size_t)a.n_pairs * sizeof(int4) : 0);
  w.total = off;
  return w;
}
}  // namespace

size_t fwd_tc_workspace(const lik_fwd_args& a, const TcExtra& x, bool* streams) {
  const TcPlan pl = plan_tc(a, x);
  if (streams) *streams = pl.streams;
  return tc_ws_layout(pl, a, x).total;
}

int launch_topk_slots(const float* keys, const int* idx, const int2* hdr, long long n_lists, int cap, int n_ctas, int n_groups,
                      int mt, int lists, int qpt, long long n_q, int k, int largest, long long index_offset, float* out_scores,
                      long long* out_index, int parts, void* part_buf, cudaStream_t st);

bool fwd_tc_norms_in_kernel(const lik_fwd_args& a, const TcExtra& x) {
  const TcPlan pl = plan_tc(a, x);
  return pl.stages >= 2 && norms_from_tiles(a, x, pl);
}

int launch_fwd_tc(const lik_fwd_args& a, const float* qn, const float* dn, float norm_d_eps, PrepJobs prep, void* ws, size_t ws_bytes,
                  cudaStream_t st, const TcExtra& x) {
  TcPlan pl = plan_tc(a, x);
  if (pl.stages < 1) {
    set_error("not enough shared memory for the document ring");
    return LIK_ERR_UNSUPPORTED;
  }
  const TcWs w = tc_ws_layout(pl, a, x);
  if (ws_bytes < w.total || (w.total && !ws)) {  // before anything that writes into the workspace is enqueued
    set_error("tcgen05 forward: workspace too small");
    return LIK_ERR_WORKSPACE;
  }
  if (pl.grid < 1) return LIK_OK;
  const bool plaid = x.plaid != nullptr;
  CUtensorMap q_map;
  DocMaps d_maps;
  memset(&d_maps, 0, sizeof(d_maps));
  int rc = pl.streams || pl.decode ? LIK_OK : make_map(&q_map, a.q, a.dtype, a.dim, TILE_M);
  if (rc) return rc;
  if (!plaid && !pl.streams) {
    for (int i = 0; i < N_BOXES; ++i) {
      rc = make_map(&d_maps.m[i], a.d, a.dtype, a.dim, (i + 1) * BOX_ROWS);
      if (rc) return rc;
    }
  }

  TcParams P{};
  P.q = make_view(a.q, qn);
  P.d = make_view(a.d, dn);
  P.pairing = a.pairing;
  P.group = a.group;
  P.n_q = a.q.n_seq;
  P.n_d = a.d.n_seq;
  P.elt_bytes = (int)dtype_size(a.dtype);
  P.ab_format = a.dtype == LIK_BF16 ? 1 : 0;  // kind::f16: F16 = 0, BF16 = 1; kind::f8f6f4: E4M3 = 0
  P.n_slabs = pl.n_slabs;
  P.k_steps = pl.k_steps;
  P.stages = pl.stages;
  P.q_per_tile = pl.q_per_tile;
  P.q_chunks = pl.q_chunks;
  P.n_tiles = pl.n_tiles;
  P.mt = pl.mt;
  P.n_sb = pl.n_sb;
  P.sb_docs = pl.sb_docs;
  P.n_flat = pl.n_flat;
  P.scores = a.scores;
  P.partial = pl.q_chunks > 1 ? (float*)((char*)ws + w.partial) : nullptr;
  P.d_len_flagged = 0;
  P.tile_q0 = nullptr;
  P.list_tab = nullptr;
  // Per-column multipliers that are exactly one fp32 array over the document rows (inverse norms or per-token scales,
  // not both) travel with the tiles when every tile's run of them starts on a 16-byte boundary and whole groups of four
  // stay inside the array: padded documents whose stride and row count are multiples of four.
  P.col_src = nullptr;
  P.sc_per = P.sc_slots = 0;
  P.norm_eps = norm_d_eps;
  if (norm_d_eps > 0.f || (!plaid && !a.d.cu && a.d.scale_scalar == 1.0f && ((a.d.scale != nullptr) != (dn != nullptr)))) {
    const float* arr = a.d.scale ? a.d.scale : dn;
    // (the streams kernel has a ring per stream, which goes with both accumulators of a stream taking every piece)
    if (norm_d_eps > 0.f || (!(pl.streams && pl.mt == 1) && ((uintptr_t)arr & 15) == 0 && a.d.seq_stride % 4 == 0 && a.d.n_rows % 4 == 0)) {
      const size_t stage = pl.stage_bytes;
      const size_t fixed = pl.smem_bytes - (size_t)pl.stages * stage;
      auto need = [&](int stages) { return fixed + (size_t)stages * stage + (size_t)2 * (stages + 1) * pl.slot_bytes; };
      int stages = pl.stages;
      while (stages > 1 && need(stages) > (size_t)227 * 1024) --stages;
      if (need(stages) <= (size_t)227 * 1024) {
        pl.stages = stages;
        pl.smem_bytes = need(stages);
        P.stages = stages;
        P.col_src = arr;
        P.sc_per = stages + 1;
        P.sc_slots = 2 * P.sc_per;
      }
    }
    if (norm_d_eps > 0.f) P.col_src = nullptr;
    if (norm_d_eps > 0.f && P.sc_per < 3) {
      set_error("not enough shared memory for the documents' norms");
      return LIK_ERR_UNSUPPORTED;
    }
  }
  if (plaid) {
    P.plaid = *x.plaid;
    P.plaid_f16 = a.dtype == LIK_F16;
  }
  if (pl.pack_tiles) {
    int* tbl = (int*)((char*)ws + w.tiles);
    pack_query_tiles_kernel<<<1, 256, 0, st>>>(a.q.cu, a.q.n_seq, tbl), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
    P.tile_q0 = tbl + 1;
  }
  if (a.d.mask && !a.d.cu) {
    // trim every document to its last valid token; only documents with holes pay for per-column masking
    int* eff = (int*)((char*)ws + w.lens);
    prep.mask_lens = MaskLensJob{a.d.mask, a.d.lens, a.d.n_seq, a.d.max_len, a.d.seq_stride, eff, LEN_FLAG_MASKED};
    P.d.lens = eff;
    P.d_len_flagged = 1;
  }
  if (a.pairing == LIK_PAIR_LIST) {
    int4* tab = (int4*)((char*)ws + w.list);
    list_units_kernel<<<(unsigned)ceil_div(a.n_pairs, 256), 256, 0, st>>>(P.q, P.d, a.pair_q, a.pair_d, a.n_pairs, tab, a.status), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
    P.list_tab = tab;
  }
  P.argmax = a.argmax;
  P.argmax_stride = a.argmax_stride;
  P.status = a.status;
  if (x.topk_k > 0) {
    P.topk.hdr = (int2*)((char*)ws + w.hdr);
    P.topk.cand_key = (float*)((char*)ws + w.keys);
    P.topk.cand_idx = (int*)((char*)ws + w.idx);
    P.topk.k = x.topk_k;
    P.topk.qpg = pl.lists * pl.q_per_tile;
    P.topk.largest = x.topk_largest;
    P.topk.doc_base = x.topk_doc_base;
    P.topk.n_lists = (int)w.n_lists;
    if (!(x.topk_flags & LIK_TOPK_CONTINUE))
      prep.fill[0] = FillJob{P.topk.hdr, (size_t)w.n_lists * sizeof(int2), 0};  // empty lists, no threshold
  }
  // positions of the saved argmax that no accumulator row covers (queries shorter than the stride)
  if (a.argmax && (a.q.cu || a.q.lens || a.argmax_stride > a.q.max_len))
    prep.fill[1] = FillJob{a.argmax, (size_t)n_scores_of(a.pairing, a.q.n_seq, a.d.n_seq, a.n_pairs) * a.argmax_stride * sizeof(int), -1};
  rc = launch_prep(prep, st);
  if (rc) return rc;

  const bool fp8 = a.dtype == LIK_E4M3;
  const bool argmax = a.argmax != nullptr;
  const bool affine = a.d.scale || dn || norm_d_eps > 0.f;  // a per-column multiplier for every document
  // LIK_LONG_DOC_TOKENS overrides the length from which the lazy winner scan is used (a tuning knob)
  static int long_doc_tokens = 0;
  if (!long_doc_tokens) {
    const char* e = getenv("LIK_LONG_DOC_TOKENS");
    const int v = e ? atoi(e) : 0;
    long_doc_tokens = v > 0 ? v : LONG_DOC_TOKENS;
  }
  const bool long_docs = argmax && a.d.max_len >= long_doc_tokens;
  if (pl.streams) {
    rc = launch_fwd_streams(a, pl, P, affine, long_docs, st);
    if (rc) return rc;
  } else if (pl.decode) {
    rc = launch_fwd_plaid(a, pl, P, st);
    if (rc) return rc;
  } else {
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
#define LIK_TC_LAUNCH(F, A, X, PL)                                                                                     \
    do {                                                                                                                 \
      LIK_CUDA_OK((allow_smem<fwd_tc_kernel<F, A, X, PL>>()));                                                           \
      LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_tc_kernel<F, A, X, PL>, q_map, d_maps, P));                               \
      ::lik::count_launch();                                                                                             \
    } while (0)
    if (plaid) {
      if (argmax) LIK_TC_LAUNCH(false, 1, false, true);
      else LIK_TC_LAUNCH(false, 0, false, true);
    } else if (fp8) {
      if (argmax && affine) LIK_TC_LAUNCH(true, 1, true, false);
      else if (argmax) LIK_TC_LAUNCH(true, 1, false, false);
      else if (affine) LIK_TC_LAUNCH(true, 0, true, false);
      else LIK_TC_LAUNCH(true, 0, false, false);
    } else {
      if (long_docs && affine) LIK_TC_LAUNCH(false, 2, true, false);
      else if (long_docs) LIK_TC_LAUNCH(false, 2, false, false);
      else if (argmax && affine) LIK_TC_LAUNCH(false, 1, true, false);
      else if (argmax) LIK_TC_LAUNCH(false, 1, false, false);
      else if (affine) LIK_TC_LAUNCH(false, 0, true, false);
      else LIK_TC_LAUNCH(false, 0, false, false);
    }
#undef LIK_TC_LAUNCH
  }
  LIK_CUDA_OK(cudaGetLastError());
  if (pl.q_chunks > 1) {
    const long long n = (long long)a.q.n_seq * a.d.n_seq;
    reduce_chunks_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(P.partial, a.q.n_seq, a.d.n_seq, pl.q_chunks, a.scores), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
  }
  if (x.topk_k > 0 && !(x.topk_flags & LIK_TOPK_PARTIAL)) {
    rc = launch_topk_slots(P.topk.cand_key, P.topk.cand_idx, P.topk.hdr, w.n_lists, TOPK_CAP, pl.grid, pl.n_groups, pl.mt, pl.lists, pl.q_per_tile,
                           a.q.n_seq, x.topk_k, x.topk_largest, x.topk_index_offset, x.topk_scores, (long long*)x.topk_index,
                           w.merge_parts, w.merge_parts > 1 ? (char*)ws + w.merge : nullptr, st);
    if (rc) return rc;
  }
  return LIK_OK;
}

}  // namespace lik

extern "C" int lik_selftest_wait_timeout(int64_t limit_cycles, int32_t* status, int32_t* result, lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(result != nullptr, "result is NULL");
  LIK_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000ll, "limit_cycles outside (0, 2e8]");
  wait_probe_kernel<false><<<1, 32, 0, (cudaStream_t)stream>>>((long long)limit_cycles, status, result), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

extern "C" int lik_selftest_other_waits(int64_t limit_cycles, int32_t* status, int32_t* result, lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(result != nullptr, "result is NULL");
  LIK_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000ll, "limit_cycles outside (0, 2e8]");
  wait_probe_kernel<true><<<1, 32, 0, (cudaStream_t)stream>>>((long long)limit_cycles, status, result), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return launch_streams_wait_probe((long long)limit_cycles, status, result + 3, (cudaStream_t)stream);
}
