// Blackwell tensor-core MaxSim forward (sm_100a: TMA + tcgen05.mma + TMEM).
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

#include "lik_common.cuh"
#include "lik_plaid_row.cuh"
#include "lik_tc.cuh"
#include "lik_tc_ptx.cuh"

namespace lik {

namespace {

constexpr int TILE_N = 96;          // document tokens per piece: rows of a TMA stage, columns of an accumulator
constexpr int SETS = 4;             // accumulators, each with its own set of epilogue warps
constexpr int SET_WARPS = 4;        // one per quadrant of 32 TMEM lanes
constexpr int ACC_COLS = TILE_N;
// The query tiles sit in tensor memory behind the accumulators, 64 columns each: an MMA that reads A from shared memory moves
// 4 KB of it for every 16 features, more than the 3 KB of 96 document rows, and took 56 cycles instead of 48 for that.
constexpr int A_COL0 = SETS * ACC_COLS;
constexpr int A_COLS = 64;
static_assert(A_COL0 + 2 * A_COLS == 512, "accumulators and query tiles fill the tensor memory");
constexpr int BOX_ROWS = 32;        // granule of the document TMA boxes: 32, 64 and 96 rows
constexpr int N_BOXES = TILE_N / BOX_ROWS;
constexpr int SLAB_BYTES_ROW = 128; // one swizzle span: 64 two-byte or 128 one-byte elements
constexpr int MAX_SLABS = 2;
constexpr int NUM_THREADS = 640;
constexpr long long WAIT_LIMIT_CYCLES = 4000000000ll;  // default limit of a wait: about 2 s at 2 GHz
constexpr int UNIT_RING = 16;                 // slots of a lane's producer -> epilogue unit ring: more than ring stages + 2
constexpr int LONG_DOC_TOKENS = 2048;         // problems whose documents can be this long run the kernel with the lazy winner scan
constexpr int UNIT_LEN_MASK = 0xFFFFFF;       // unit_info.x: document length in the low 24 bits,
constexpr int UNIT_SLOT_SHIFT = 24;           // the multiplier slot of its first piece in bits 24..27, LEN_FLAG_MASKED above,
constexpr int UNIT_END = 1 << 31;             // the sign bit in the entries behind the last unit

// ---------------------------------------------------------------------------------------------
// Kernel parameters
// ---------------------------------------------------------------------------------------------
// Fused top-k (retrieve).  Instead of a score matrix the epilogue keeps candidate lists: one list per
// (CTA, query) for every query of the tile groups the CTA works on.  A CTA meets the documents of a
// group in ascending order, so a list is append-only in document order; a score enters when it beats the
// list's threshold (strictly: an equal score that arrives later has a higher index and loses the tie).
// A full list (TOPK_CAP entries) is cut back to its k best by the warp that owns it, which also raises
// the threshold to the k-th best.  The lists of a query are merged by lik::launch_topk_slots afterwards.
// List slot of (CTA c, group g) is c + g: a CTA works on a contiguous range of groups and the ranges of
// consecutive CTAs are ordered, so c + g is unique among the pairs that occur.
constexpr int TOPK_CAP = 256;  // entries per list: eight per lane of the owning warp
struct TopkOut {
  float* cand_key;  // [n_slots * qpg][TOPK_CAP]: score (negated when the smallest are wanted)
  int* cand_idx;    // same shape: document index
  int2* hdr;        // [n_slots * qpg]: x = entries in the list, y = threshold as an ordered key (0: none yet)
  int k;
  int qpg;          // lists per slot: one per accumulator and query of its tile
  int largest;
  int doc_base;     // added to the document index stored with a candidate
  int n_lists;      // lists allocated (the kernel checks every list number against it)
};

// One row of the pair-list table (LIK_PAIR_LIST): written by list_units_kernel, read by the producer.
//   x = query (0 for a pair that is out of range), y = first document row, z = document length, w = unused
struct TcParams {
  SeqView q, d;
  int pairing;       // CROSS, GROUPED or LIST
  int group;         // GROUPED: documents per query
  int n_q, n_d;
  int elt_bytes;     // 1 or 2
  int ab_format;     // instruction-descriptor operand format
  int n_slabs;       // 128-byte K slabs per row
  int k_steps;       // MMA K steps (32 bytes each)
  int stages;        // document ring depth
  int q_per_tile;    // whole queries per 128-row tile (when q_chunks == 1)
  int q_chunks;      // 128-row chunks per query (> 1: one query chunk per tile)
  int n_tiles;       // query tiles
  int mt;            // query tiles resident per CTA (1 or 2)
  int n_sb;          // CROSS: the documents are walked in n_sb super-blocks of sb_docs documents (L2-sized)
  int sb_docs;
  long long n_flat;  // GROUPED / LIST: number of units
  const int4* list_tab;  // LIST: one row per pair
  float* scores;
  float* partial;    // [n_tiles * 4, n_d] when q_chunks > 1: sums of 32 rows
  int* argmax;
  int argmax_stride;
  int* status;
  const int* tile_q0;  // packed queries: tile m holds queries [tile_q0[m], tile_q0[m+1]); tile_q0[-1] is the tile count
  int d_len_flagged;  // d.lens carries LEN_FLAG_MASKED on documents whose mask is not a plain prefix
  // Per-column multipliers that are one fp32 per document row (inverse norms, or per-token scales) and whose layout
  // allows it travel with the tile: the producer copies the tile's run of them into a slot of a small ring in shared
  // memory (bulk copy on the stage's barrier) instead of the epilogue fetching them from device memory per tile.
  const float* col_src;  // nullptr: the epilogue stages the multipliers itself
  // A ring of sc_per = stages + 1 slots per lane.  The slot of a lane's piece n is refilled for its piece n + sc_per: by
  // then the MMAs of the lane's piece n + 1 have completed (the producer is at most `stages` pieces ahead of the tensor
  // pipe), which needed the lane's accumulators back from piece n - and an epilogue gives an accumulator back only
  // after its last read of the multipliers.
  int sc_per;
  int sc_slots;          // lanes * sc_per, or 0
  float norm_eps;     // > 0: the kernel takes the documents' inverse norms from the tiles themselves (NORM_WARPS)
  int d_deep;         // the documents' rows fill their slabs: one copy brings all slabs of a piece
  int d_full_count;   // arrivals that complete a ring stage: 1 (TMA) or the number of decompress warps
  TopkOut topk;       // cand_key == nullptr: scores are written instead
  PlaidSrc plaid;     // PLAID kernels: the compressed documents
  int plaid_f16;      // PLAID kernels: operand type fp16 instead of bf16
};

// Warps 18 and 19 take the rows' inverse norms from the tiles in shared memory when the launch asks for it: the documents
// are then read once instead of twice, and no norms go through device memory.  Two queries of 128 tokens against 4000
// documents of up to 1030: 484 -> 232 us (146 without normalisation; the two warps' arithmetic is what remains of the gap).
constexpr int NORM_WARPS = 2;
constexpr int PLAID_WARPS = 3;  // warps 0, 18 and 19 decode compressed tokens in the PLAID kernels

struct SharedCtl {
  unsigned long long q_full, q_empty;
  unsigned long long a_idle[2];       // an issuer's MMAs on the query tiles in tensor memory are done
  unsigned long long d_full[8], d_empty[8];
  unsigned long long acc_full[SETS], acc_empty[SETS];
  unsigned long long set_sync[SETS];  // rendezvous of an epilogue set
  uint32_t stage_info[8];
  int4 unit_info[SETS][UNIT_RING];    // by lane; per work unit: x = document length | flags, y = its first row, z = tile group, w = document
  volatile int units_posted[SETS];    // entries published in a lane's ring so far
  uint32_t tmem_base;
  volatile int abort_flag;
  long long wait_limit;         // cycles after which a wait gives up
  short seg_off[SETS][TILE_M], seg_len[SETS][TILE_M], row_seg[SETS][TILE_M];
  int seg_q[SETS][TILE_M];
  int n_seg[SETS];
  int warp_aligned[SETS];  // every query of the tile sits inside one warp's 32 rows, starting at its first row
  float emit[SETS][2][TILE_M];
  alignas(16) float col_scale[SETS][2][TILE_N];  // by set and parity of the piece; read as float4
  alignas(16) float col_bias[SETS][2][TILE_N];
  // fused top-k: state of the candidate list of every query of the resident tiles
  int seg_cnt[SETS][TILE_M];
  unsigned seg_thr[SETS][TILE_M];
  int seg_list[SETS][TILE_M];      // list number (slot * qpg + query within the group)
  float plaid_bw[256];          // PLAID kernels: the bucket weights
};

// Bounded wait.  Returns false when the CTA is aborting.  The first probe lets the hardware suspend
// the thread until the phase completes (or the hint expires), so the common case costs two
// instructions; everything else lives in one out-of-line function.
__device__ __noinline__ bool wait_bar_slow(uint32_t b, uint32_t parity, SharedCtl* ctl, int* status) {
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(b, parity)) return true;
    if (ctl->abort_flag) return false;
    if (clock64() - t0 > ctl->wait_limit) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
      return false;
    }
  }
}
__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  const uint32_t b = smem_u32(bar);
  if (mbar_try_wait(b, parity)) return true;
  return wait_bar_slow(b, parity, ctl, status);
}
// The same for all lanes of a warp: they leave together, with one answer.
__device__ __forceinline__ bool wait_bar_warp(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  return __all_sync(0xffffffffu, wait_bar(bar, parity, ctl, status));
}
// Bounded wait until the producer has published entry `uc` of a lane's unit ring.  False when the CTA is aborting.
__device__ __noinline__ bool wait_posted_slow(SharedCtl* ctl, int ln, int uc, int* status) {
  const long long t0 = clock64();
  while (true) {
    if (ctl->units_posted[ln] > uc) return true;
    if (ctl->abort_flag) return false;
    if (clock64() - t0 > ctl->wait_limit) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
      return false;
    }
  }
}
__device__ __forceinline__ bool wait_posted(SharedCtl* ctl, int ln, int uc, int* status) {
  const bool there = ctl->units_posted[ln] > uc;
  return __all_sync(0xffffffffu, there || wait_posted_slow(ctl, ln, uc, status));
}
// Bounded rendezvous of the warps that share `bar` (initialised with their number); `n` counts this warp's uses of it.
__device__ __forceinline__ bool warps_sync(unsigned long long* bar, uint32_t& n, int lane, SharedCtl* ctl, int* status) {
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
  return wait_bar_warp(bar, n++ & 1, ctl, status);
}

// Query tiles of tile-group g: tiles [g*mt, min((g+1)*mt, n_tiles)).
struct TileInfo {
  int qa, qb;        // queries [qa, qb)
  int chunk;         // chunk index when q_chunks > 1
  long long row0;    // first matrix row of the tile
};

__device__ __forceinline__ TileInfo tile_info(const TcParams& P, int tile) {
  TileInfo t;
  if (P.tile_q0) {
    t.qa = P.tile_q0[tile];
    t.qb = P.tile_q0[tile + 1];
    t.chunk = 0;
  } else if (P.q_chunks == 1) {
    t.qa = tile * P.q_per_tile;
    t.qb = min(t.qa + P.q_per_tile, P.n_q);
    t.chunk = 0;
  } else {
    t.qa = tile / P.q_chunks;
    t.qb = t.qa + 1;
    t.chunk = tile - t.qa * P.q_chunks;
  }
  long long r0;
  int len;
  seq_bounds(P.q, t.qa, r0, len, nullptr);
  t.row0 = r0 + (long long)t.chunk * TILE_M;
  return t;
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
struct UnitWalk {
  int sb;               // super-block
  int doc_lo, n_docs;   // its documents
  long long u, u_end;   // what is left of this CTA's share of its units
};

// moves to the next super-block with units for this CTA, unless there are some left in this one
__device__ __forceinline__ void walk_settle(const TcParams& P, int n_groups, UnitWalk& w) {
  const long long c = blockIdx.x, G = gridDim.x;
  while (w.u >= w.u_end && w.sb < P.n_sb) {
    long long units;
    if (P.pairing == LIK_PAIR_CROSS) {
      w.doc_lo = (int)min((long long)w.sb * P.sb_docs, (long long)P.n_d);
      w.n_docs = (int)min((long long)P.sb_docs, (long long)(P.n_d - w.doc_lo));
      units = (long long)n_groups * w.n_docs;
    } else {
      w.doc_lo = 0;
      w.n_docs = P.n_d;
      units = P.n_flat;
    }
    if (units < (1ll << 32) / 256) {  // (a 64-bit division is a hundred dependent instructions in front of the first load; grids have at most 256 CTAs)
      w.u = (unsigned)units * (unsigned)c / (unsigned)G;
      w.u_end = (unsigned)units * (unsigned)(c + 1) / (unsigned)G;
    } else {
      w.u = units * c / G;
      w.u_end = units * (c + 1) / G;
    }
    ++w.sb;
  }
}

// A unit as the producer warp fetches it: the length words of 32 units are loaded at once, a lane each, a batch ahead of their use.
struct UnitRaw {
  int doc, grp, a, b;
};
__device__ __forceinline__ UnitRaw unit_fetch(const TcParams& P, const UnitWalk& w, long long u) {
  UnitRaw r{0, 0, 0, 0};
  if (P.pairing == LIK_PAIR_CROSS) {
    r.grp = u < (1ll << 32) ? (int)((unsigned)u / (unsigned)w.n_docs) : (int)(u / w.n_docs);
    r.doc = w.doc_lo + (int)(u - (long long)r.grp * w.n_docs);
  } else {
    r.doc = (int)u;
    r.grp = P.pairing == LIK_PAIR_GROUPED ? r.doc / P.group : 0;
  }
  if (P.pairing == LIK_PAIR_LIST) {
    const int4 t = __ldg(P.list_tab + r.doc);
    r.grp = t.x;
    r.a = t.y;
    r.b = t.z;
  } else if (P.d.cu) {
    r.a = P.d.cu[r.doc];
    r.b = P.d.cu[r.doc + 1];
  } else if (P.d.lens) {
    r.a = P.d.lens[r.doc];
  }
  return r;
}
// First row and column count of the fetched document; `masked` tells whether its mask has holes.
// Lengths come from the caller-validated views, clamped to the padded extent.
// (the tensor-core path takes fewer than 2^31 rows)
__device__ __forceinline__ void unit_resolve(const TcParams& P, const UnitRaw& r, int& row, int& len, bool& masked) {
  masked = false;
  long long row0;
  if (P.pairing == LIK_PAIR_LIST) {
    row0 = r.a;
    len = r.b;
  } else if (P.d.cu) {
    const int a = r.a, b = r.b;
    row0 = a;
    len = b > a ? b - a : 0;
    if ((long long)a + len > P.d.n_rows) len = P.d.n_rows > a ? (int)(P.d.n_rows - a) : 0;
  } else {
    row0 = (long long)r.doc * P.d.seq_stride;
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
  row = (int)row0;
}

// Sum of squares of one row of a stage whose second slab, if any, lies `slab_rows` rows behind the first (lane = row: eight consecutive rows of a swizzled slab lie in different banks).  The
// pieces of 16 bytes are summed and combined in the order of prep_kernel's butterfly, so that the norms of a row are the
// same number wherever they are taken.
template <typename T>
__device__ __forceinline__ float stage_row_sum_sq(const unsigned char* row, int r, int slab_rows) {
  float half[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // pieces h, h + 2, h + 4, h + 6, each beside its partner eight further: their loads in flight together
    uint4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned char* a = row + (((2 * i + h) ^ (r & 7)) << 4);
      x[i] = *reinterpret_cast<const uint4*>(a);
      y[i] = make_uint4(0, 0, 0, 0);
      if (slab_rows) y[i] = *reinterpret_cast<const uint4*>(a + slab_rows * SLAB_BYTES_ROW);
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
  CUtensorMap flat[N_BOXES];  // document boxes of 32, 64, 96 rows, one 128-byte slab wide
  CUtensorMap deep[N_BOXES];  // the same with all slabs of the rows, slab behind slab (rows that fill their slabs)
};

// Word the producer leaves beside every ring stage for the MMA issuer.
constexpr uint32_t STAGE_COLS_MASK = 0x7Fu;    // rows of the stage that are multiplied: a multiple of 32
constexpr int STAGE_LANE_SHIFT = 16;           // the lane whose accumulator(s) the piece feeds
constexpr uint32_t STAGE_FIRST = 1u << 18;     // first stage of a query-tile group: take the tiles over first
constexpr uint32_t STAGE_END = 1u << 20;       // no more work
constexpr uint32_t STAGE_LONE = 1u << 21;      // the second accumulator has no query tile: it changes hands, nothing is multiplied into it
constexpr uint32_t STAGE_WIDE = 1u << 22;      // the slabs lie a full stage apart instead of right behind each other

// Monotone map float -> unsigned (larger float, larger key); 0 is below every float.
__device__ __forceinline__ unsigned ordered_key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Cut a full candidate list (TOPK_CAP entries, in arrival = ascending document order) back to its k best
// and return the k-th best as an ordered key.  One warp; lane l holds entries l, l + 32, ...  The k-th
// largest key is found by bisection on its bits (32 warp-wide counts); entries above it stay, and of the
// entries equal to it the earliest ones (lowest document indices), so that exactly k remain, in order.
__device__ __noinline__ unsigned topk_compact(float* keys, int* idx, int k, int lane) {
  constexpr int PER = TOPK_CAP / 32;
  unsigned uk[PER];
  float fk[PER];
  int id[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    fk[j] = keys[j * 32 + lane];
    id[j] = idx[j * 32 + lane];
    uk[j] = ordered_key(fk[j]);
  }
  unsigned kth = 0;
  for (int bit = 31; bit >= 0; --bit) {
    const unsigned cand = kth | (1u << bit);
    int c = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) c += uk[j] >= cand ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (c >= k) kth = cand;
  }
  int n_gt = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) n_gt += uk[j] > kth ? 1 : 0;
  n_gt = __reduce_add_sync(0xffffffffu, n_gt);
  const int need = k - n_gt;  // ties to keep (at least one)
  const unsigned lt = (1u << lane) - 1u;
  int out = 0, ties = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const bool eq = uk[j] == kth;
    const unsigned m_eq = __ballot_sync(0xffffffffu, eq);
    const bool keep = uk[j] > kth || (eq && ties + __popc(m_eq & lt) < need);
    const unsigned m_keep = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int pos = out + __popc(m_keep & lt);
      keys[pos] = fk[j];
      idx[pos] = id[j];
    }
    out += __popc(m_keep);
    ties += __popc(m_eq);
  }
  __syncwarp();
  return kth;
}

// WINNERS: 0 = scores only, 1 = winners saved, 2 = winners saved and every document takes the lazy winner scan (launched
// for problems whose documents are long, so that the kernels for short documents carry no third copy of the tile loop)
template <bool FP8, int WINNERS, bool SCALED, bool PLAID>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fwd_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ DocMaps d_maps, const TcParams P) {
  constexpr bool ARGMAX = WINNERS != 0;
  // The last box of a document that is not a multiple of 32 tokens is moved back to end where the document ends: the
  // columns it shares with the box before hold the same dot products twice, which no maximum minds, and no column has to
  // be masked.  (Multipliers per column do not move along, and decoded rows have no boxes.)
  constexpr bool SHIFT = !SCALED && !PLAID;
  extern __shared__ unsigned char smem_raw[];
  // operand tiles need 1024-byte alignment for the 128-byte swizzle
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int q_tile_bytes = P.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const int d_stage_bytes = P.n_slabs * TILE_N * SLAB_BYTES_ROW;
  unsigned char* q_smem = smem;                              // [mt][n_slabs][128 rows][128 B], on their way to tensor memory
  unsigned char* d_smem = smem + P.mt * q_tile_bytes;        // [stages][n_slabs][rows][128 B]
  float* sc_ring = reinterpret_cast<float*>(d_smem + (size_t)P.stages * d_stage_bytes);  // [lanes][sc_per][TILE_N] (kernels with multipliers)
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(d_smem + (size_t)P.stages * d_stage_bytes + (size_t)P.sc_slots * TILE_N * sizeof(float));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const bool list = P.pairing == LIK_PAIR_LIST;
  const bool topk = !ARGMAX && P.topk.cand_key != nullptr;  // the fused top-k never saves winners

  const bool norm_warps = SCALED && !FP8 && !PLAID && P.norm_eps > 0.f;  // (a member of every pipeline barrier then)
  const int n_issuers = PLAID || norm_warps ? 1 : 2;
  if (tid == 0) {
    mbar_init(smem_u32(&ctl->q_full), 1);
    mbar_init(smem_u32(&ctl->q_empty), (uint32_t)n_issuers);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ctl->a_idle[i]), 1);
    for (int s = 0; s < P.stages; ++s) {
      mbar_init(smem_u32(&ctl->d_full[s]), (uint32_t)P.d_full_count);
      mbar_init(smem_u32(&ctl->d_empty[s]), (uint32_t)(norm_warps ? n_issuers + NORM_WARPS : n_issuers));
    }
    for (int a = 0; a < SETS; ++a) {
      mbar_init(smem_u32(&ctl->acc_full[a]), norm_warps ? 1 + NORM_WARPS : 1);
      mbar_init(smem_u32(&ctl->acc_empty[a]), SET_WARPS);
      mbar_init(smem_u32(&ctl->set_sync[a]), SET_WARPS);
    }
    ctl->abort_flag = 0;
    ctl->wait_limit = WAIT_LIMIT_CYCLES;
    for (int i = 0; i < SETS; ++i) ctl->units_posted[i] = 0;
    fence_barrier_init();
    prefetch_tmap(&q_map);
    if (!PLAID)
      for (int i = 0; i < N_BOXES; ++i) prefetch_tmap(P.d_deep ? &d_maps.deep[i] : &d_maps.flat[i]);
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
  const int lanes = SETS / P.mt;  // documents in flight

  const bool producer_warp = warp == 0 || (PLAID && warp >= 2 + SETS * SET_WARPS);
  if (producer_warp) {
    // =========================== producer ===========================
    // One warp walks the units, loads the query tiles and the document pieces with TMA and leaves the stage words and the
    // unit rings.  It runs on warp-uniform values and one elected lane issues, as in the issuer below: TMA instructions, too,
    // take their operands from uniform registers.  In the PLAID kernels three warps walk the units in step; each decodes its
    // share of every piece's tokens into the swizzled operand layout (generic-proxy stores, fenced for the tensor core's
    // reads), and arrives on the stage barrier; the elected lane of warp 0 still does everything else.
    {
      const int pw = warp == 0 ? 0 : warp - (2 + SETS * SET_WARPS) + 1;  // decoder warp number 0..2
      const bool elect = warp == 0 && elect_one();
      int cur_grp = -1;
      uint32_t n_qload = 0, st = 0, ph = 0, n_dload = 0;
      const int x_per_slab = SLAB_BYTES_ROW / P.elt_bytes;
      bool ok = true;
      uint32_t lone = 0, first = 0;
      // the documents in flight, one per lane: what is left of each
      int l_len[SETS], l_c0[SETS], l_uc[SETS], l_sc[SETS], l_row[SETS];
#pragma unroll
      for (int l = 0; l < SETS; ++l) {
        l_len[l] = -1;  // none
        l_c0[l] = l_uc[l] = l_sc[l] = l_row[l] = 0;
      }
      int open = 0;  // lanes with a document
      // 32 units at a time, a lane of the warp each: a batch that is dealt out, and one whose length words are on their way
      UnitWalk walk{0, 0, 0, 0, 0};
      walk_settle(P, n_groups, walk);
      UnitRaw raw{0, 0, 0, 0};
      int n_raw = 0, n_unit = 0, at_unit = 0;
      int u_doc = 0, u_grp = 0, u_row = 0, u_len = 0;  // this lane's unit; u_len carries LEN_FLAG_MASKED
      auto fetch_batch = [&]() {
        n_raw = (int)min(32ll, walk.u_end - walk.u);
        if (n_raw > 0) {
          if (lane < n_raw) raw = unit_fetch(P, walk, walk.u + lane);
          walk.u += n_raw;
          walk_settle(P, n_groups, walk);
        }
      };
      bool have;
      int nx_doc = 0, nx_grp = 0, nx_row = 0, nx_len = 0;
      auto pull = [&]() {
        if (at_unit == n_unit) {
          bool masked = false;
          u_doc = raw.doc;
          u_grp = raw.grp;
          unit_resolve(P, raw, u_row, u_len, masked);
          u_len = (u_len & UNIT_LEN_MASK) | (masked ? LEN_FLAG_MASKED : 0);
          n_unit = n_raw > 0 ? n_raw : 0;
          at_unit = 0;
          fetch_batch();
        }
        have = n_unit > 0;
        if (have) {
          nx_doc = __shfl_sync(0xffffffffu, u_doc, at_unit);
          nx_grp = __shfl_sync(0xffffffffu, u_grp, at_unit);
          nx_row = __shfl_sync(0xffffffffu, u_row, at_unit);
          nx_len = __shfl_sync(0xffffffffu, u_len, at_unit);
          ++at_unit;
        }
      };
      fetch_batch();
      pull();
      while (ok && (have || open)) {
#pragma unroll
        for (int l = 0; l < SETS; ++l) {
          if (l >= lanes || !ok) continue;
          if (l_len[l] < 0) {
            // the lane takes the next unit, unless that belongs to another tile group and this one is not finished yet
            if (!have || (nx_grp != cur_grp && open)) continue;
            const int doc = nx_doc, grp = nx_grp, drow0 = nx_row, dlen = nx_len & UNIT_LEN_MASK;
            const int dmasked = nx_len & LEN_FLAG_MASKED;
            pull();
            if (grp != cur_grp) {
              cur_grp = grp;
              first = STAGE_FIRST;
              const int t0 = grp * P.mt, t1 = min(t0 + P.mt, n_tiles);
              lone = P.mt == 2 && t1 - t0 < 2 ? STAGE_LONE : 0u;
              if (warp == 0) {
                // wait until the issuers have copied the previous query tiles to tensor memory
                ok = wait_bar_warp(&ctl->q_empty, (n_qload & 1) ^ 1, ctl, P.status);
                if (ok && elect) {
                  mbar_arrive_expect_tx(smem_u32(&ctl->q_full), (uint32_t)((t1 - t0) * q_tile_bytes));
                  for (int t = t0; t < t1; ++t) {
                    TileInfo ti = tile_info(P, t);
                    for (int sl = 0; sl < P.n_slabs; ++sl)
                      tma_load_2d(smem_u32(q_smem + (t - t0) * q_tile_bytes + sl * TILE_M * SLAB_BYTES_ROW), &q_map, sl * x_per_slab, (int)ti.row0,
                                  smem_u32(&ctl->q_full));
                  }
                }
                __syncwarp();
              }
              ++n_qload;
              if (!ok) continue;
            }
            // publish the unit for the lane's epilogue sets; an empty document still sends one (empty) piece so that every
            // unit passes through the same hand-shakes
            if (elect) {
              ctl->unit_info[l][l_uc[l] & (UNIT_RING - 1)] = make_int4(dlen | (SCALED ? l_sc[l] << UNIT_SLOT_SHIFT : 0) | dmasked, drow0, grp, doc);
              if (SCALED) {  // (the others learn of it from a full accumulator)
                __threadfence_block();
                ctl->units_posted[l] = l_uc[l] + 1;
              }
            }
            ++l_uc[l];
            ++open;
            l_len[l] = dlen;
            l_c0[l] = 0;
            l_row[l] = drow0;
          }
          // the lane's next piece
          const int c0 = l_c0[l], dlen = l_len[l], drow0 = l_row[l];
          const int ncols = min(TILE_N, dlen - c0);
          const bool ends = c0 + TILE_N >= dlen;
          const int rows = __shfl_sync(0xffffffffu, (ncols + BOX_ROWS - 1) & ~(BOX_ROWS - 1), 0);
          // A short document that is no multiple of 32 tokens takes two boxes, the second moved back to end where the document
          // ends; a longer one's last piece is moved back as a whole.
          const bool split = SHIFT && dlen < rows && dlen > BOX_ROWS;
          ok = wait_bar_warp(&ctl->d_empty[st], ph ^ 1, ctl, P.status);
          if (!ok) continue;
          const uint32_t full = smem_u32(&ctl->d_full[st]);
          if (ends) --open;
          if (elect)
            ctl->stage_info[st] = (uint32_t)rows | ((uint32_t)l << STAGE_LANE_SHIFT) | first | lone | (split || PLAID ? STAGE_WIDE : 0u);
          first = 0;
          if (PLAID) {
            // the piece's tokens in six equal runs, one per half-warp of the three decoder warps
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
            const int row = __shfl_sync(0xffffffffu, drow0 + (SHIFT ? max(min(c0, dlen - rows), 0) : c0), 0);
            // the piece's multipliers ride on the same barrier: whole groups of four floats, never past the array's end
            uint32_t sc_bytes = 0;
            if (SCALED && P.col_src && rows > 0) sc_bytes = (uint32_t)min((long long)((ncols + 3) & ~3), P.d.n_rows - row) * 4u;
            if (elect) {
              const uint32_t dst = smem_u32(d_smem) + st * (uint32_t)d_stage_bytes;
              if (rows > 0) {
                mbar_arrive_expect_tx(full, (uint32_t)(rows * SLAB_BYTES_ROW * P.n_slabs) + sc_bytes);
                const int box = rows / BOX_ROWS - 1;
                if (!split && P.d_deep) {
                  tma_load_3d(dst, &d_maps.deep[box], 0, row, 0, full);
                } else {
                  const uint32_t slab = (uint32_t)((split ? TILE_N : rows) * SLAB_BYTES_ROW);
                  for (int sl = 0; sl < P.n_slabs; ++sl) {
                    tma_load_2d(dst + sl * slab, &d_maps.flat[split ? box - 1 : box], sl * x_per_slab, row, full);
                    if (split) tma_load_2d(dst + sl * slab + box * BOX_ROWS * SLAB_BYTES_ROW, &d_maps.flat[0], sl * x_per_slab, row + dlen - BOX_ROWS, full);
                  }
                }
                if (sc_bytes) bulk_load_1d(smem_u32(sc_ring + (l * P.sc_per + l_sc[l]) * TILE_N), P.col_src + row, sc_bytes, full);
              } else {
                mbar_arrive(full);
              }
            }
            __syncwarp();
          }
          ++n_dload;
          if (++st == (uint32_t)P.stages) { st = 0; ph ^= 1; }
          if (SCALED && ++l_sc[l] >= P.sc_per) l_sc[l] = 0;
          l_c0[l] = c0 + TILE_N;
          if (ends) l_len[l] = -1;
        }
      }
      if (ok) {
        // tell the epilogue sets and the issuer that the stream has ended
        ok = wait_bar_warp(&ctl->d_empty[st], ph ^ 1, ctl, P.status);
        if (ok) {
          if (elect) {
#pragma unroll
            for (int l = 0; l < SETS; ++l) {
              if (l >= lanes) continue;
              ctl->unit_info[l][l_uc[l] & (UNIT_RING - 1)] = make_int4(UNIT_END, 0, 0, 0);
              __threadfence_block();
              ctl->units_posted[l] = l_uc[l] + 1;
            }
            ctl->stage_info[st] = STAGE_END;
          }
          __syncwarp();
          if (PLAID ? lane == 0 : elect) mbar_arrive(smem_u32(&ctl->d_full[st]));
        }
      }
      if (!ok && elect) {
        // aborting: let the copies already issued land before the CTA goes away
        if (!PLAID) {
          for (uint32_t i = 1; i <= (uint32_t)P.stages && i <= n_dload; ++i) {
            const bool wrapped = i > st;  // that use lies before the last wrap of the ring
            const uint32_t slot = wrapped ? st + (uint32_t)P.stages - i : st - i;
            const uint32_t bar = smem_u32(&ctl->d_full[slot]);
            for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(bar, wrapped ? ph ^ 1 : ph); ++spin) {
            }
          }
        }
        if (n_qload) {
          const uint32_t bar = smem_u32(&ctl->q_full);
          for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(bar, (n_qload - 1) & 1); ++spin) {
          }
        }
      }
    }
  } else if (warp == 1 || (warp == 2 + SETS * SET_WARPS && n_issuers == 2)) {
    // =========================== MMA issuers ===========================
    // Driven by the stage words alone.  A whole warp runs the loop on warp-uniform values (the stage word is broadcast from
    // lane 0, which also tells the compiler that it is uniform) and one elected lane issues: tcgen05.mma takes its
    // descriptors from uniform registers, and with the loop under `lane == 0` every MMA paid about 100 cycles for moving
    // them there, whatever its width.
    // Two warps share the work where a warp is free for it: one feeds the even accumulators, the other the odd ones.  The
    // tensor pipe holds about four MMAs ahead, some 250 cycles, and the waits and words of a piece take a warp longer than
    // that; each of the two has the other's MMAs to hide behind.
    const uint32_t me = warp == 1 ? 0u : 1u;
    uint32_t st = 0, ph = 0, n_q = 0, acc_ph = 0;  // acc_ph: one phase bit per accumulator
    bool ok = true;
    const bool issue = elect_one();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const uint32_t a_desc0 = (uint32_t)smem_desc_sw128(smem_u32(q_smem));
    const uint32_t b_desc0 = (uint32_t)smem_desc_sw128(smem_u32(d_smem));
    const uint32_t stage_desc = (uint32_t)(d_stage_bytes >> 4);
    const uint32_t q_desc = (uint32_t)(q_tile_bytes >> 4);
    const uint32_t idesc0 = instr_desc(P.ab_format, 0);
    const int k_steps = P.k_steps;
    const uint32_t mt = (uint32_t)P.mt;
    constexpr uint32_t A_SLAB = (TILE_M * SLAB_BYTES_ROW) >> 4, B_SLAB = (TILE_N * SLAB_BYTES_ROW) >> 4;
    // `step` visits this warp's share of the accumulators [a0, a0 + n)
    const uint32_t step = (uint32_t)n_issuers;
    while (ok) {
      ok = wait_bar_warp(&ctl->d_full[st], ph, ctl, P.status);
      if (!ok) break;
      const uint32_t info = __shfl_sync(0xffffffffu, ctl->stage_info[st], 0);
      if (info & STAGE_END) {
        // the accumulators change hands once more, empty: the sets find the end of the stream in their unit ring
        for (uint32_t a = me; a < SETS; a += step) {
          if (ok) ok = wait_bar_warp(&ctl->acc_empty[a], ((acc_ph >> a) & 1u) ^ 1u, ctl, P.status);
          if (ok && issue) tc_commit(smem_u32(&ctl->acc_full[a]));
          __syncwarp();
        }
        break;
      }
      if (info & STAGE_FIRST) {
        // New query tiles: this warp copies the ones it multiplies with to its place(s) in tensor memory, once its MMAs on the
        // old ones are done.  (A copy and an MMA that follows it run in order.)  With one tile and two issuers either has its own.
        ok = wait_bar_warp(&ctl->q_full, n_q & 1u, ctl, P.status);
        if (ok && n_q) {
          if (issue) tc_commit(smem_u32(&ctl->a_idle[me]));
          __syncwarp();
          ok = wait_bar_warp(&ctl->a_idle[me], (n_q - 1) & 1u, ctl, P.status);
        }
        if (!ok) break;
        ++n_q;
        tc_fence_after();
        if (issue) {
          for (uint32_t t = 0; t < mt; ++t) {
            if (mt == 2 && step == 2 && t != me) continue;
            const uint32_t to = tmem_base + A_COL0 + (mt == 2 ? t : me) * A_COLS;
            for (int k = 0; k < k_steps; ++k) tc_copy_128x256b(to + 8 * k, a_desc0 + t * q_desc + (uint32_t)((k & 3) * 2) + (k >> 2) * A_SLAB, desc_hi);
          }
          tc_commit(smem_u32(&ctl->q_empty));
        }
        __syncwarp();
      }
      const uint32_t rows = info & STAGE_COLS_MASK;
      const uint32_t idesc = idesc0 | (rows << 14);  // N / 8 in bits 17..22
      const uint32_t b_stage = b_desc0 + st * stage_desc;
      const uint32_t b_slab = info & STAGE_WIDE ? B_SLAB : rows * (SLAB_BYTES_ROW >> 4);
      const uint32_t set0 = ((info >> STAGE_LANE_SHIFT) & (SETS - 1)) * mt;
      uint32_t a = set0;
      if (step == 2 && ((a ^ me) & 1u)) ++a;
      bool mine = false;
      for (; a < set0 + mt; a += step) {
        ok = wait_bar_warp(&ctl->acc_empty[a], ((acc_ph >> a) & 1u) ^ 1u, ctl, P.status);
        if (!ok) break;
        acc_ph ^= 1u << a;
        mine = true;
        const uint32_t t = a - set0;
        tc_fence_after();
        if (issue) {
          if (rows && !(t == 1 && (info & STAGE_LONE))) {  // (the accumulator always changes hands, so that both sides keep their phase)
            const uint32_t d_tmem = tmem_base + a * ACC_COLS;
            const uint32_t a_tmem = tmem_base + A_COL0 + (mt == 2 ? t : me) * A_COLS;
            // descriptors differ only in the start address, in units of 16 bytes
            if (k_steps == 8) {  // the common width (128 two-byte or 256 one-byte elements): straight-line issue
#pragma unroll
              for (int k = 0; k < 8; ++k)
                tc_mma_ts<FP8>(d_tmem, a_tmem + 8 * k, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * b_slab, desc_hi, idesc, k ? 1u : 0u);
            } else {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (k < k_steps) tc_mma_ts<FP8>(d_tmem, a_tmem + 8 * k, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * b_slab, desc_hi, idesc, k ? 1u : 0u);
            }
          }
          tc_commit(smem_u32(&ctl->acc_full[a]));
        }
        __syncwarp();
      }
      if (!ok) break;
      if (issue) {
        if (mine) tc_commit(smem_u32(&ctl->d_empty[st]));  // ring slot reusable once these MMAs retire
        else mbar_arrive(smem_u32(&ctl->d_empty[st]));
      }
      __syncwarp();
      if (++st == (uint32_t)P.stages) { st = 0; ph ^= 1; }
    }
  } else if (warp < 2 + SETS * SET_WARPS) {
    // =========================== epilogue sets ===========================
    // Set s (four warps) drains accumulator s: with two resident query tiles, tile s & 1 of lane s >> 1; with one, lane s.
    // A warp owns 32 rows of a document from its first column to its score.  It waits for its accumulator by itself and gives
    // it back by itself; the warps of a set meet only where the query tile changes, where columns are staged by all of them
    // and where a query's rows lie in several warps.  All of these waits are bounded: a warp that gives up leaves the
    // loop, and the others' waits find the abort flag.
    const int e = warp - 2;
    const int set = e >> 2;
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int wq = e & 3;                    // warp index inside the set
    const int row = quad * 32 + lane;        // accumulator row == query token slot in the tile
    const int et = wq * 32 + lane;           // thread index inside the set (0..127)
    const int ln = P.mt == 2 ? set >> 1 : set;
    const int my_tile = P.mt == 2 ? set & 1 : 0;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(set * ACC_COLS);
    const uint32_t acc_empty_bar = smem_u32(&ctl->acc_empty[set]);
    int cur_grp = -1;
    uint32_t n_acc = 0, n_emit = 0, n_sync = 0, n_col = 0;
    bool ok = true;
    // per-row / per-warp state for the resident query tile
    bool have_tile = false, warp_rows = false, in_seg = false, row_ok = false, aligned = false;
    float my_qf = 1.f;
    int tile_id = 0;
    long long arg_off = -1;   // ARGMAX: offset of this row's slot for document 0 (-1: row stores nothing)
    long long warp_out = -1;  // aligned tiles: offset of this warp's query score for document 0
    int my_list = -1;         // top-k: the list whose state thread `et` loaded into shared memory
    int warp_seg = -1;        // aligned tiles: the query (segment) of this warp's rows
#define LIK_SET_SYNC() warps_sync(&ctl->set_sync[set], n_sync, lane, ctl, P.status)
#define LIK_WAIT_ACC() wait_bar_warp(&ctl->acc_full[set], n_acc & 1, ctl, P.status)
    // top-k: write the state of the lists this thread loaded back to their headers
#define LIK_TOPK_STORE_BACK()                                                                          \
  do {                                                                                                 \
    if (topk && my_list >= 0) {                                                                        \
      P.topk.hdr[my_list] = make_int2(ctl->seg_cnt[set][et], (int)ctl->seg_thr[set][et]);              \
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
      if (ukey_ > ctl->seg_thr[set][sg_]) {                                                            \
        int cnt_ = ctl->seg_cnt[set][sg_];                                                             \
        if ((unsigned)cnt_ >= (unsigned)TOPK_CAP || (unsigned)ctl->seg_list[set][sg_] >= (unsigned)P.topk.n_lists) {  \
          if (lane == 0 && P.status) atomicOr(P.status, LIK_DEV_INTERNAL);                             \
          break;                                                                                       \
        }                                                                                              \
        float* keys_ = P.topk.cand_key + (long long)ctl->seg_list[set][sg_] * TOPK_CAP;                \
        int* idx_ = P.topk.cand_idx + (long long)ctl->seg_list[set][sg_] * TOPK_CAP;                   \
        if (lane == 0) {                                                                               \
          keys_[cnt_] = key_;                                                                          \
          idx_[cnt_] = doc + P.topk.doc_base;                                                          \
        }                                                                                              \
        ++cnt_;                                                                                        \
        __syncwarp();                                                                                  \
        if (cnt_ == TOPK_CAP) {                                                                        \
          const unsigned thr_ = topk_compact(keys_, idx_, P.topk.k, lane);                             \
          cnt_ = P.topk.k;                                                                             \
          if (lane == 0) ctl->seg_thr[set][sg_] = thr_;                                                \
        }                                                                                              \
        if (lane == 0) ctl->seg_cnt[set][sg_] = cnt_;                                                  \
        __syncwarp();                                                                                  \
      }                                                                                                \
    }                                                                                                  \
  } while (0)

    const bool cross = P.pairing == LIK_PAIR_CROSS;
    const bool bulk = SCALED && P.sc_slots != 0;  // the multipliers of a piece arrive with it, or are made from it
    // multipliers that the set stages itself are fetched while the MMAs run, so the unit has to be known before the accumulator is full
    const bool early = SCALED && !bulk;
    for (int uc = 0;; ++uc) {
      // The unit (tile group, document, length, first row) comes from the lane's ring, where it stands before its first
      // piece is announced to the issuer, so that a full accumulator says that it is there.
      ok = early ? wait_posted(ctl, ln, uc, P.status) : LIK_WAIT_ACC();
      if (!ok) break;
      const int4 uinfo = ctl->unit_info[ln][uc & (UNIT_RING - 1)];
      if (uinfo.x < 0) break;  // the end of the stream
      const int grp = uinfo.z;
      const int doc = uinfo.w;
      // (a group number out of range cannot index anything: its tile number fails the range check below)
      if (grp != cur_grp) {
        cur_grp = grp;
        // (re)build the segment table of this set's tile
        tile_id = grp * P.mt + my_tile;
        have_tile = (unsigned)tile_id < (unsigned)n_tiles;
        ok = LIK_SET_SYNC();  // everyone in the set is done reading the old table
        if (!ok) break;
        LIK_TOPK_STORE_BACK();
        TileInfo ti{};
        int nseg = 0;
        if (have_tile) {
          ti = tile_info(P, tile_id);
          nseg = ti.qb - ti.qa;
          ctl->row_seg[set][et] = -1;
          if (et == 0) {
            ctl->n_seg[set] = nseg;
            ctl->warp_aligned[set] = P.q_chunks == 1 ? 1 : 0;
          }
        }
        ok = LIK_SET_SYNC();
        if (!ok) break;
        if (have_tile && et < nseg) {
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
          if ((off & 31) != 0 || l > 32 || l == 0) ctl->warp_aligned[set] = 0;
          if (ARGMAX && len > P.argmax_stride && P.status) atomicOr(P.status, LIK_DEV_ARGMAX_STRIDE);
          ctl->seg_off[set][et] = (short)off;
          ctl->seg_len[set][et] = (short)l;
          ctl->seg_q[set][et] = ti.qa + et;
          for (int i = 0; i < l; ++i) ctl->row_seg[set][off + i] = (short)et;
          if (topk) {
            // the candidate list of (this CTA, this group, this lane, this query)
            my_list = ((int)blockIdx.x + grp) * P.topk.qpg + set * P.q_per_tile + et;
            if ((unsigned)my_list >= (unsigned)P.topk.n_lists) {
              if (P.status) atomicOr(P.status, LIK_DEV_INTERNAL);
              my_list = 0;
            }
            const int2 hd = P.topk.hdr[my_list];
            ctl->seg_list[set][et] = my_list;
            ctl->seg_cnt[set][et] = hd.x;
            ctl->seg_thr[set][et] = (unsigned)hd.y;
          }
        }
        ok = LIK_SET_SYNC();
        if (!ok) break;
        in_seg = false;
        row_ok = false;
        warp_rows = false;
        arg_off = -1;
        warp_out = -1;
        warp_seg = -1;
        aligned = have_tile && ctl->warp_aligned[set] != 0;
        if (have_tile) {
          const int sg = ctl->row_seg[set][row];
          if (sg >= 0) {
            in_seg = true;
            const int my_q = ctl->seg_q[set][sg];
            const int my_s = row - ctl->seg_off[set][sg] + ti.chunk * TILE_M;
            const long long qrow = ti.row0 + row;
            row_ok = row_valid(P.q, qrow);
            my_qf = row_factor(P.q, qrow);
            if (ARGMAX && my_s < P.argmax_stride)
              arg_off = (cross ? (long long)my_q * P.n_d : 0ll) * P.argmax_stride + my_s;
          }
          warp_rows = __any_sync(0xffffffffu, in_seg);
          const int sg0 = ctl->row_seg[set][quad * 32];
          if (aligned && sg0 >= 0) {
            warp_seg = sg0;
            warp_out = cross ? (long long)ctl->seg_q[set][sg0] * P.n_d : 0ll;
          }
        }
      }
      const int dlen = uinfo.x & UNIT_LEN_MASK;
      int sc_slot = SCALED ? (uinfo.x >> UNIT_SLOT_SHIFT) & 15 : 0;  // multiplier slot of the unit's first piece, in its lane's ring
      const long long drow0 = uinfo.y;
      const bool holes = (uinfo.x & LEN_FLAG_MASKED) != 0;  // the document's mask is not a plain prefix
      // where this unit's results go: CROSS / GROUPED index by document, LIST by pair (== unit)
      const long long out_col = doc;
      float run_m = -INFINITY;
      int run_i = -1;
      int c0 = 0;
      // The pieces of the document.  The body exists twice in the kernels without per-column multipliers: documents whose
      // mask is a plain prefix (nearly all) take the copy that has no column arrays in it, the others the general one -
      // the common path's time goes with its code size, so the rare one stays out of it.
      auto document_tiles = [&](auto general_, auto lazy_) {
      constexpr bool general = decltype(general_)::value;  // the document's mask has holes
      constexpr bool lazy = decltype(lazy_)::value;        // long document: winner scan only when some row of the warp needs it
      constexpr bool use_cols = SCALED || general;          // per-column multiplier / additive mask needed
      do {
        const int ncols = max(0, min(TILE_N, dlen - c0));
        // SHIFT: the token of the piece's first column; a chunk of 32 columns never reaches behind the document's end
        const int base = SHIFT ? max(min(c0, dlen - ((ncols + 31) & ~31)), 0) : c0;
        // Per-column arrays of this piece, staged by the whole set.  There are two of them, so that the one rendezvous
        // behind the writes also says that everyone is done with the one that the piece after the next will overwrite.
        float* const col_scale = ctl->col_scale[set][n_col & 1];
        float* const col_bias = ctl->col_bias[set][n_col & 1];
        const bool staged = general || (SCALED && !bulk);
        const float* const sc_arr = SCALED && bulk ? sc_ring + (ln * P.sc_per + sc_slot) * TILE_N : col_scale;
        auto stage_columns = [&]() {
          ++n_col;
          const int c = et;  // a thread per column
          if (c < ((ncols + 31) & ~31)) {
            float sc = 1.f, bi = -INFINITY;
            const int tok = SHIFT && dlen >= BOX_ROWS ? min(base + (c & ~31), dlen - BOX_ROWS) + (c & 31) : base + c;  // the token that column c stands for
            if (tok < dlen) {
              const long long drow = drow0 + tok;
              sc = norm_warps ? sc_arr[c] : row_factor(P.d, drow);
              bi = row_valid(P.d, drow) ? 0.f : -INFINITY;
            }
            col_scale[c] = sc;
            col_bias[c] = bi;
          }
        };
        if (staged && early) {  // before the accumulator wait: overlaps the MMAs
          stage_columns();
          ok = LIK_SET_SYNC();
          if (!ok) break;
        }
        if (early || c0 > 0) {
          ok = LIK_WAIT_ACC();
          if (!ok) break;
        }
        ++n_acc;
        if (staged && !early) {
          stage_columns();
          ok = LIK_SET_SYNC();
          if (!ok) break;
        }
        tc_fence_after();
        // the accumulator goes back to the issuer as soon as this warp's last columns sit in registers
#define LIK_RELEASE_ACC()                                          \
  do {                                                             \
    tc_fence_before();                                             \
    __syncwarp();                                                  \
    if (lane == 0) mbar_arrive(acc_empty_bar);                     \
  } while (0)
        // (a warp without a query row, as most have under a single short query, only hands the accumulator on)
        int cc = warp_rows ? 0 : ncols;
        if (cc >= ncols) LIK_RELEASE_ACC();
        if (use_cols && general) {
          // a mask with holes: every chunk takes multiplier and additive mask
          for (; cc < ncols; cc += 32) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            affine32(v, col_scale + cc, col_bias + cc);  // bias is -inf past ncols and in holes
            if (cc + 32 >= ncols) LIK_RELEASE_ACC();
            fold32<ARGMAX, lazy>(v, SHIFT && dlen >= BOX_ROWS ? min(base + cc, dlen - BOX_ROWS) : base + cc, run_m, run_i);
          }
        } else if (use_cols) {
          // whole chunks are valid: multiplier only; the partial last chunk also takes the mask (-inf past ncols).
          // Multipliers that came with the piece sit in a ring slot that is refilled once the accumulator has changed
          // hands often enough: there the accumulator goes back after the last read of them, not before.
          for (; cc < ncols; cc += 32) {
            const bool last = cc + 32 >= ncols;
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (last && !bulk) LIK_RELEASE_ACC();
            if (cc + 32 <= ncols) scale32(v, sc_arr + cc);
            else scale32_first(v, sc_arr + cc, ncols - cc);
            if (last && bulk) LIK_RELEASE_ACC();
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
        } else if (SHIFT) {
          for (; cc < ncols; cc += 32) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (cc + 32 >= ncols) LIK_RELEASE_ACC();
            int at = min(base + cc, dlen - BOX_ROWS);
            if (dlen < BOX_ROWS) {  // a document of fewer than 32 tokens is all that still needs a mask
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = i < ncols ? v[i] : -INFINITY;
              at = 0;
            }
            fold32<ARGMAX, lazy>(v, at, run_m, run_i);
          }
        } else {
          for (; cc < ncols; cc += 32) {
            float v[32];
            tmem_ld32_issue(lane_addr + (uint32_t)cc, v);
            tmem_ld_wait(v);
            if (cc + 32 >= ncols) {
              LIK_RELEASE_ACC();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = cc + i < ncols ? v[i] : -INFINITY;
            }
            fold32<ARGMAX, lazy>(v, c0 + cc, run_m, run_i);
          }
        }
#undef LIK_RELEASE_ACC
        c0 += TILE_N;
        if (SCALED && ++sc_slot >= P.sc_per) sc_slot = 0;
      } while (c0 < dlen);
      };
      // (long documents, WINNERS == 2: most 32-column chunks past the first few hundred tokens hold no new maximum for any
      // of a warp's rows, and the scan for its column is skipped there)
      if (holes) document_tiles(std::true_type{}, std::false_type{});
      else document_tiles(std::false_type{}, std::integral_constant<bool, WINNERS == 2>{});
      if (!ok) break;
      // ---- end of document ----
      if (!have_tile || (aligned && !warp_rows)) continue;
      // one value per row, summed per query in a fixed order
      const bool has_winner = ARGMAX ? (run_i >= 0) : (run_m != -INFINITY);
      const float val = (in_seg && row_ok && has_winner) ? run_m * my_qf : 0.f;
      if (ARGMAX && arg_off >= 0) P.argmax[arg_off + out_col * P.argmax_stride] = has_winner ? run_i : -1;
      if (P.q_chunks > 1) {
        // a piece of a long query: every warp leaves the sum of its 32 rows
        const float sum = warp_sum(val);
        if (lane == 0) P.partial[((long long)tile_id * SET_WARPS + quad) * P.n_d + doc] = sum;
        continue;
      }
      if (aligned) {
        // one query per warp: a shuffle tree (fixed order) replaces the shared-memory pass
        const float sum = warp_sum(val);
        if (warp_out >= 0) LIK_EMIT_SCORE(warp_seg, sum, warp_out + out_col);
        continue;
      }
      float* ebuf = ctl->emit[set][n_emit & 1];
      ++n_emit;
      ebuf[row] = val;
      ok = LIK_SET_SYNC();
      if (!ok) break;
      const int nseg = ctl->n_seg[set];
      for (int sg = wq; sg < nseg; sg += SET_WARPS) {
        const int off = ctl->seg_off[set][sg], len = ctl->seg_len[set][sg];
        float sum = 0.f;
        for (int i = lane; i < len; i += 32) sum += ebuf[off + i];
        sum = warp_sum(sum);
        const int qq = ctl->seg_q[set][sg];
        const long long o = cross ? (long long)qq * P.n_d + out_col : out_col;
        LIK_EMIT_SCORE(sg, sum, o);
      }
    }
    // top-k: leave the lists' state where the next launch stage (the merge) finds it
    if (topk && ok && LIK_SET_SYNC()) LIK_TOPK_STORE_BACK();
#undef LIK_EMIT_SCORE
#undef LIK_TOPK_STORE_BACK
#undef LIK_WAIT_ACC
#undef LIK_SET_SYNC
  } else if (SCALED && !FP8 && !PLAID && norm_warps) {
    // =========================== inverse norms of the pieces ===========================
    // The multipliers of a piece go into its lane's ring, and the arrival that announces them belongs to the phase of the
    // accumulator(s) that the piece feeds: the epilogue waits for both with one wait.  An arrival must not fall into the
    // phase before, hence the wait for that one.
    const int nw = warp - (2 + SETS * SET_WARPS);
    uint32_t st = 0, ph = 0, acc_ph = 0, seen = 0;
    int sc_cnt[SETS] = {0, 0, 0, 0};
    bool ok = true;
    const bool bf16 = P.ab_format == 1, two_slabs = P.n_slabs == 2;
    while (ok) {
      ok = wait_bar_warp(&ctl->d_full[st], ph, ctl, P.status);
      if (!ok) break;
      const uint32_t info = __shfl_sync(0xffffffffu, ctl->stage_info[st], 0);
      // arrives for accumulator a's current phase, once the one before is complete
      auto announce = [&](uint32_t a) {
        if (ok && ((seen >> a) & 1u)) ok = wait_bar_warp(&ctl->acc_full[a], ((acc_ph >> a) & 1u) ^ 1u, ctl, P.status);
        if (ok && lane == 0) mbar_arrive(smem_u32(&ctl->acc_full[a]));
        seen |= 1u << a;
        acc_ph ^= 1u << a;
      };
      if (info & STAGE_END) {  // the accumulators' last phase, which brings nothing
        for (uint32_t a = 0; a < SETS; ++a) announce(a);
        break;
      }
      const int rows = (int)(info & STAGE_COLS_MASK);
      const uint32_t ln = (info >> STAGE_LANE_SHIFT) & (SETS - 1);
      int at = 0;
#pragma unroll
      for (int l = 0; l < SETS; ++l)
        if (l == (int)ln) {
          at = sc_cnt[l];
          if (++sc_cnt[l] >= P.sc_per) sc_cnt[l] = 0;
        }
      float* slot = sc_ring + (ln * P.sc_per + at) * TILE_N;
      const unsigned char* stage = d_smem + (size_t)st * d_stage_bytes;
      for (int r = nw * 32 + lane; r < rows; r += NORM_WARPS * 32) {
        const float ss = bf16 ? stage_row_sum_sq<__nv_bfloat16>(stage + r * SLAB_BYTES_ROW, r, two_slabs ? rows : 0)
                              : stage_row_sum_sq<__half>(stage + r * SLAB_BYTES_ROW, r, two_slabs ? rows : 0);
        slot[r] = inv_norm(ss, P.norm_eps);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->d_empty[st]));
      for (int t = 0; t < P.mt; ++t) announce(ln * (uint32_t)P.mt + t);
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
    const bool got = wait_bar(&ctl.q_full, 0, &ctl, status);
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

// scores[q, j] = sum over the pieces of 32 rows of query q, in order
__global__ void reduce_chunks_kernel(const float* __restrict__ partial, int n_q, int n_d, int pieces, float* __restrict__ scores) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n_q * n_d) return;
  const int q = (int)(idx / n_d), j = (int)(idx - (long long)q * n_d);
  float s = 0.f;
  for (int c = 0; c < pieces; ++c) s += partial[((long long)q * pieces + c) * n_d + j];
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

// `slabs` 0: a map over the rows, one slab wide; otherwise rows x slabs, whose boxes hold all slabs of their rows
int make_map(CUtensorMap* map, const lik_seqs& s, int dtype, int dim, int box_rows, int slabs = 0) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled is not available from this driver");
    return LIK_ERR_CUDA;
  }
  const int eb = (int)dtype_size(dtype);
  CUtensorMapDataType dt = dtype == LIK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                           : dtype == LIK_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                              : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const cuuint32_t slab_elems = (cuuint32_t)(SLAB_BYTES_ROW / eb);
  cuuint64_t gdim[3] = {slabs ? (cuuint64_t)slab_elems : (cuuint64_t)dim, (cuuint64_t)(s.n_rows > 0 ? s.n_rows : 1), (cuuint64_t)slabs};
  cuuint64_t gstride[2] = {(cuuint64_t)s.row_stride * eb, (cuuint64_t)SLAB_BYTES_ROW};
  cuuint32_t box[3] = {slab_elems, (cuuint32_t)box_rows, (cuuint32_t)slabs};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, dt, slabs ? 3 : 2, const_cast<void*>(s.data), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
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

struct TcPlan {
  bool pack_tiles;  // ragged queries packed greedily into tiles by pack_query_tiles_kernel
  int q_per_tile, q_chunks, n_tiles, mt, n_slabs, k_steps, stages;
  int n_sb, sb_docs, n_groups;
  long long n_flat, n_units_total;
  int grid;
  size_t smem_bytes;
};

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
  const long long g = pl.n_units_total < sm_count() ? pl.n_units_total : sm_count();
  pl.grid = (int)(g < 0 ? 0 : g);
  // the fused top-k numbers its candidate lists by CTA: the same grid whatever the piece of the corpus
  if (x.topk_k > 0 && pl.grid > 0) pl.grid = sm_count();
  const size_t q_bytes = (size_t)pl.mt * pl.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const size_t stage = (size_t)pl.n_slabs * TILE_N * SLAB_BYTES_ROW;
  const size_t fixed = q_bytes + sizeof(SharedCtl) + 1024;
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

int topk_merge_parts(int n_ctas, int n_groups, int mt);

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
    w.n_lists = (long long)(pl.grid + pl.n_groups) * SETS * pl.q_per_tile;
    w.hdr = take((size_t)w.n_lists * sizeof(int2));
    w.keys = take((size_t)w.n_lists * TOPK_CAP * sizeof(float));
    w.idx = take((size_t)w.n_lists * TOPK_CAP * sizeof(int));
    // few tile groups: a query has lists from many CTAs, which are merged in parts by as many CTAs first
    w.merge_parts = topk_merge_parts(pl.grid, pl.n_groups, pl.mt);
    w.merge = take(w.merge_parts > 1 ? (size_t)w.merge_parts * a.q.n_seq * x.topk_k * sizeof(long long) : 0);
  }
  w.partial = take(pl.q_chunks > 1 ? (size_t)pl.n_tiles * SET_WARPS * a.d.n_seq * sizeof(float) : 0);
  w.lens = take((a.d.mask && !a.d.cu) ? (size_t)a.d.n_seq * sizeof(int) : 0);
  w.tiles = take(pl.pack_tiles ? (size_t)(a.q.n_seq + 3) * sizeof(int) : 0);
  w.list = take(a.pairing == LIK_PAIR_LIST ? (size_t)a.n_pairs * sizeof(int4) : 0);
  w.total = off;
  return w;
}
}  // namespace

size_t fwd_tc_workspace(const lik_fwd_args& a, const TcExtra& x) { return tc_ws_layout(plan_tc(a, x), a, x).total; }

int launch_topk_slots(const float* keys, const int* idx, const int2* hdr, long long n_lists, int cap, int n_ctas, int n_groups,
                      int mt, int qpt, long long n_q, int k, int largest, long long index_offset, float* out_scores,
                      long long* out_index, int parts, void* part_buf, cudaStream_t st);

// Raise the kernel's dynamic shared memory limit once per device and size instead of on every launch (a host call
// of a microsecond or two that small problems feel).
template <bool F, int A, bool X, bool PL>
static cudaError_t allow_smem(size_t bytes) {
  static size_t allowed[64] = {0};  // by device ordinal
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < 64 && allowed[dev] >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(fwd_tc_kernel<F, A, X, PL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && dev >= 0 && dev < 64) allowed[dev] = bytes;
  return e;
}

// A launch that reads every document up to four times takes the documents' norms from its tiles instead of one pass of
// prep_kernel in front.  A query of 32 tokens against 1000 documents of up to 300 40 -> 30 us; two groups of query tiles (12 x 32
// against 8000 of 300) 407 -> 308, (4 x 128 against 8000 of 1030) 1498 -> 953; 128-token queries against 4000 documents of up
// to 500: three groups 458 -> 394, four 540 -> 484, five 646 -> 611, six 740 -> 724, eight 921 -> 930: the two warps take every
// norm once per group.
bool fwd_tc_norms_in_kernel(const lik_fwd_args& a, const TcExtra& x) {
  if (!(a.normalize & LIK_NORM_D) || x.plaid || (a.dtype != LIK_BF16 && a.dtype != LIK_F16) || a.d.scale || a.d.scale_scalar != 1.0f) return false;
  const TcPlan pl = plan_tc(a, x);
  return pl.stages >= 2 && (a.pairing == LIK_PAIR_GROUPED || (a.pairing == LIK_PAIR_CROSS && pl.n_groups <= 4));
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
  int rc = make_map(&q_map, a.q, a.dtype, a.dim, TILE_M);
  if (rc) return rc;
  const bool deep = a.dim * (int)dtype_size(a.dtype) == pl.n_slabs * SLAB_BYTES_ROW;
  if (!plaid) {
    for (int i = 0; i < N_BOXES; ++i) {
      rc = make_map(&d_maps.flat[i], a.d, a.dtype, a.dim, (i + 1) * BOX_ROWS);
      if (!rc && deep) rc = make_map(&d_maps.deep[i], a.d, a.dtype, a.dim, (i + 1) * BOX_ROWS, pl.n_slabs);
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
  P.d_deep = deep;
  P.d_full_count = plaid ? PLAID_WARPS : 1;
  // Per-column multipliers that are exactly one fp32 array over the document rows (inverse norms or per-token scales,
  // not both) travel with the tiles when every tile's run of them starts on a 16-byte boundary and whole groups of four
  // stay inside the array: padded documents whose stride and row count are multiples of four.
  P.col_src = nullptr;
  P.sc_per = P.sc_slots = 0;
  P.norm_eps = norm_d_eps;
  if (norm_d_eps > 0.f || (!plaid && !a.d.cu && a.d.scale_scalar == 1.0f && ((a.d.scale != nullptr) != (dn != nullptr)))) {
    const float* arr = a.d.scale ? a.d.scale : dn;
    if (norm_d_eps > 0.f || (((uintptr_t)arr & 15) == 0 && a.d.seq_stride % 4 == 0 && a.d.n_rows % 4 == 0)) {
      const size_t stage = (size_t)pl.n_slabs * TILE_N * SLAB_BYTES_ROW;
      const size_t fixed = pl.smem_bytes - (size_t)pl.stages * stage;
      auto need = [&](int stages) { return fixed + (size_t)stages * stage + (size_t)(SETS / pl.mt) * (stages + 1) * TILE_N * sizeof(float); };
      int stages = pl.stages;
      while (stages > 1 && need(stages) > (size_t)227 * 1024) --stages;
      if (need(stages) <= (size_t)227 * 1024) {
        pl.stages = stages;
        pl.smem_bytes = need(stages);
        P.stages = stages;
        P.col_src = arr;
        P.sc_per = stages + 1;
        P.sc_slots = SETS / pl.mt * P.sc_per;
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
    P.topk.qpg = SETS * pl.q_per_tile;
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
    LIK_CUDA_OK((allow_smem<F, A, X, PL>(pl.smem_bytes)));                                                             \
    LIK_CUDA_OK(cudaLaunchKernelEx(&cfg, fwd_tc_kernel<F, A, X, PL>, q_map, d_maps, P));                               \
    ::lik::count_launch();                                                                                             \
  } while (0)
  // LIK_LONG_DOC_TOKENS overrides the length from which the lazy winner scan is used (a tuning knob)
  static int long_doc_tokens = 0;
  if (!long_doc_tokens) {
    const char* e = getenv("LIK_LONG_DOC_TOKENS");
    const int v = e ? atoi(e) : 0;
    long_doc_tokens = v > 0 ? v : LONG_DOC_TOKENS;
  }
  const bool long_docs = argmax && a.d.max_len >= long_doc_tokens;
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
  LIK_CUDA_OK(cudaGetLastError());
  if (pl.q_chunks > 1) {
    const long long n = (long long)a.q.n_seq * a.d.n_seq;
    reduce_chunks_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(P.partial, a.q.n_seq, a.d.n_seq, SET_WARPS * pl.q_chunks, a.scores), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
  }
  if (x.topk_k > 0 && !(x.topk_flags & LIK_TOPK_PARTIAL)) {
    rc = launch_topk_slots(P.topk.cand_key, P.topk.cand_idx, P.topk.hdr, w.n_lists, TOPK_CAP, pl.grid, pl.n_groups, pl.mt, pl.q_per_tile,
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
  wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((long long)limit_cycles, status, result), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}
