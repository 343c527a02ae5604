// What the two tensor-core scoring kernels share (lik_fwd_tc.cu, lik_fwd_streams.cu): parameters, query tiles, candidate lists.
#pragma once

#include "lik_common.cuh"
#include "lik_plaid_row.cuh"
#include "lik_tc.cuh"
#include "lik_tc_ptx.cuh"

namespace lik {

struct TcPlan {
  bool streams;     // the kernel with two streams (lik_fwd_streams.cu)
  bool decode;      // the kernel that decodes a compressed index for one query tile (lik_fwd_plaid.cu)
  bool pack_tiles;  // ragged queries packed greedily into tiles by pack_query_tiles_kernel
  int q_per_tile, q_chunks, n_tiles, mt, n_slabs, k_steps, stages;
  int n_sb, sb_docs, n_groups;
  long long n_flat, n_units_total;
  int grid;
  size_t smem_bytes;
  int lists;        // candidate lists of a query's place per list slot (fused top-k)
  size_t stage_bytes, slot_bytes;  // shared memory per ring stage / per multiplier slot
};

namespace {

constexpr int SLAB_BYTES_ROW = 128; // one swizzle span: 64 two-byte or 128 one-byte elements
constexpr int MAX_SLABS = 2;
constexpr int BOX_ROWS = 32;        // granule of the document TMA boxes (64 read a sixth more rows than ragged documents have)
constexpr int UNIT_LEN_MASK = 0xFFFFFF;       // unit_info.x: document length in the low 24 bits,
constexpr int UNIT_SLOT_SHIFT = 24;           // the multiplier slot of its first tile in bits 24..28, LEN_FLAG_MASKED above

}  // namespace

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
  int qpg;          // lists per slot: two query tiles' worth, of every document that the kernel has in flight for them
  int largest;
  int doc_base;     // added to the document index stored with a candidate
  int n_lists;      // lists allocated (the kernel checks every list number against it)
};

struct TcParams {
  SeqView q, d;
  int pairing;       // CROSS, GROUPED or LIST
  int group;         // GROUPED: documents per query
  int n_q, n_d;
  int elt_bytes;     // 1 or 2
  int ab_format;     // instruction-descriptor operand format
  int n_slabs;       // 128-byte K slabs per row
  int k_steps;       // MMA K steps (32 bytes each)
  int stages;        // document ring depth (of either stream)
  int q_per_tile;    // whole queries per 128-row tile (when q_chunks == 1)
  int q_chunks;      // 128-row chunks per query (> 1: one query chunk per tile)
  int n_tiles;       // query tiles
  int mt;            // query tiles resident per CTA (1 or 2)
  int n_sb;          // CROSS: the documents are walked in n_sb super-blocks of sb_docs documents (L2-sized)
  int sb_docs;
  long long n_flat;  // GROUPED / LIST: number of units
  const int4* list_tab;  // LIST: one row per pair, by list_units_kernel: x = query (0: out of range), y = first document row, z = document length
  float* scores;
  float* partial;    // [n_tiles, n_d] when q_chunks > 1
  int* argmax;
  int argmax_stride;
  int* status;
  const int* tile_q0;  // packed queries: tile m holds queries [tile_q0[m], tile_q0[m+1]); tile_q0[-1] is the tile count
  int d_len_flagged;  // d.lens carries LEN_FLAG_MASKED on documents whose mask is not a plain prefix
  // Per-column multipliers that are one fp32 per document row (inverse norms, or per-token scales) and whose layout
  // allows it travel with the tile: the producer copies the tile's run of them into a slot of a small ring in shared
  // memory (bulk copy on the stage's barrier) instead of the epilogue fetching them from device memory per tile.
  const float* col_src;  // nullptr: the epilogue stages the multipliers itself
  int sc_per, sc_slots;  // slots per ring, and of both rings (0: the epilogue stages the multipliers)
  float norm_eps;     // > 0: the kernel takes the documents' inverse norms from the tiles themselves
  TopkOut topk;       // cand_key == nullptr: scores are written instead
  PlaidSrc plaid;     // PLAID kernels: the compressed documents
  int plaid_f16;      // PLAID kernels: operand type fp16 instead of bf16
};


namespace {

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

// Monotone map float -> unsigned (larger float, larger key); 0 is below every float.
__device__ __forceinline__ unsigned ordered_key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Cut a full candidate list (TOPK_CAP entries, in arrival = ascending document order) back to its k best
// and return the k-th best as an ordered key.  One warp; lane l holds entries l, l + 32, ...  The k-th
// largest key is found by bisection on its bits (32 warp-wide counts); entries above it stay, and of the
// entries equal to it the earliest ones (lowest document indices), so that exactly k remain, in order.
// PARTIAL: the list holds n entries, k at least.
template <bool PARTIAL = false>
__device__ __noinline__ unsigned topk_compact(float* keys, int* idx, int k, int lane, int n = TOPK_CAP) {
  constexpr int PER = TOPK_CAP / 32;
  unsigned uk[PER];
  float fk[PER];
  int id[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    fk[j] = keys[j * 32 + lane];
    id[j] = idx[j * 32 + lane];
    uk[j] = !PARTIAL || j * 32 + lane < n ? ordered_key(fk[j]) : 0u;
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

}  // namespace

// the kernel with two streams
size_t fwd_streams_fixed_smem(int n_slabs);   // shared memory beside its rings
size_t fwd_streams_stage_bytes(int n_slabs);  // a stage of both streams
size_t fwd_streams_slot_bytes();
int launch_fwd_streams(const lik_fwd_args& a, const TcPlan& pl, const TcParams& P, bool affine, bool long_docs, cudaStream_t st);
// the kernel that decodes a compressed index
size_t fwd_plaid_smem(int n_slabs);
int fwd_plaid_ctas_per_sm();
int launch_fwd_plaid(const lik_fwd_args& a, const TcPlan& pl, const TcParams& P, cudaStream_t st);
int launch_streams_wait_probe(long long limit, int* status, int* result, cudaStream_t st);

}  // namespace lik
