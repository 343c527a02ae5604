// Tensor-core MaxSim forward for larger problems (sm_100a: TMA + tcgen05.mma + TMEM): two independent streams per CTA.
//
// The work is that of lik_fwd_tc.cu - rows are query tokens, columns document tokens, the epilogue keeps a running maximum per
// row - and so are the results; what differs is how a CTA is organised.  Traces of that kernel show each of its serial roles, not
// the tensor pipe, setting the pace: a wait on a barrier costs a warp 110 to 150 cycles even when it is complete already, an MMA
// group's hand-shakes some 400, an epilogue warp's document 1000 to 3000.  So here
//   - a CTA has two streams, each with a producer warp, an issuer warp, a ring of stages and two accumulators of its own; they
//     take the CTA's units in turn and share the resident query tiles and the tensor pipe;
//   - documents are cut into pieces of 96 tokens; one accumulator of 96 columns per (stream, query tile), or per every second
//     unit of a stream with one resident tile, each drained by a set of four warps of its own;
//   - an epilogue warp owns its 32 rows of a document from the first column to the score and meets no other warp on the way
//     (two groups of eight warps with rendezvous before: half of all instructions were hand-shakes);
//   - the query tiles are copied to tensor memory (tcgen05.cp): an MMA with A in shared memory moves 4 KB of it per 16 features
//     beside the 3 KB of 96 document rows and took 56 cycles instead of 48 for that;
//   - the last box of a document is moved back to end where the document ends, so that no column needs a mask.
// In-batch 512 x 512 of 32 x 300 tokens 477 -> 326 us with winners, 334 -> 284 us without; 256 x 256 of 16 x 64 tokens 61 -> 41 and
// 57 -> 39 us.
// What bounds it now: the search for the winners' columns (54 instructions on the half-rate pipe per 32 columns and warp, half of
// the pipe's time) and the round trip of an accumulator (MMAs, 3 chunks of TMEM loads and folds, two barriers).
//
// Warp roles (640 threads): warps 0 and 19 load for the two streams, 1 and 18 issue their MMAs, 2 to 17 are the epilogue.
//
// Every wait is bounded: on expiry the CTA raises LIK_DEV_WAIT_TIMEOUT in the status word, sets a shared abort flag, drains its
// TMA copies, frees TMEM and returns.
#include <cuda.h>

#include <cstring>
#include <type_traits>

#include "lik_fwd_tc.cuh"

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
constexpr int N_BOXES = TILE_N / BOX_ROWS;
constexpr int NUM_THREADS = 640;
constexpr int EPI_WARP0 = 2;        // 16 epilogue warps; 0 and 1 load and issue for the first stream, 19 and 18 for the second
constexpr int UNIT_RING = 16;       // slots of a producer -> epilogue unit ring: more than ring stages + 2
constexpr int UNIT_END = 1 << 31;   // unit_info.x, the sign bit: the entry behind the last unit

// Rings of multiplier slots: sc_per = stages + 1 slots per stream (they arrive with the pieces only where both of its accumulators
// take every piece).
// The slot of piece n is refilled for piece n + sc_per: by then the MMAs of piece n + 1 have completed (the producer is at most
// `stages` pieces ahead of the tensor pipe), which needed the accumulator(s) back from piece n - and an epilogue gives an
// accumulator back only after its last read of the multipliers.

struct SharedCtl {
  unsigned long long q_full, q_empty;
  unsigned long long a_idle, a_ready;  // the query tiles in tensor memory: no MMA reads the old ones, the new ones are there
  unsigned long long d_full[2][8], d_empty[2][8];  // by stream
  unsigned long long acc_full[SETS], acc_empty[SETS];
  unsigned long long set_sync[SETS];  // rendezvous of an epilogue set
  uint32_t stage_info[2][8];
  int4 unit_info[SETS][UNIT_RING];    // by accumulator (a stream's first, where both take every unit); per work unit: x = document length | flags, y = its first row, z = tile group, w = document
  volatile int units_posted[SETS];    // entries published in it so far
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
};

// Bounded waits of a whole warp.  They return false when the CTA is aborting.  A probe lets the hardware suspend the threads
// until the phase completes (or some thousands of cycles have passed), so the common case costs a probe and a vote.
// The lanes leave together, with one answer: TMEM loads, shuffles and rendezvous of the full warp follow, and nothing promises
// that two lanes that probe a barrier get the same answer, or read the clock in the same cycle.  What every warp waits for
// cannot pass by unseen: the phase after it needs this warp's arrival first, so an answer "complete" stays true.
template <class Done>
__device__ __forceinline__ bool wait_warp(Done done, SharedCtl* ctl, int* status) {
  if (__all_sync(0xffffffffu, done())) return true;
  const long long t0 = clock64();
  while (!__all_sync(0xffffffffu, done())) {
    if (clock64() - t0 > ctl->wait_limit) {
      ctl->abort_flag = 1;
      if (status) atomicOr(status, LIK_DEV_WAIT_TIMEOUT);
    }
    if (__any_sync(0xffffffffu, ctl->abort_flag != 0)) return false;
  }
  return true;
}
__device__ __noinline__ bool wait_bar_slow(uint32_t b, uint32_t parity, SharedCtl* ctl, int* status) {
  return wait_warp([&] { return mbar_try_wait(b, parity); }, ctl, status);
}
// The loop behind the first probe is out of line, except (INLINE) in the epilogue that looks for winners: there a call would have
// the registers around it saved to local memory, next to 204 KB of shared memory that leave little L1.
template <bool INLINE = false>
__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity, SharedCtl* ctl, int* status) {
  const uint32_t b = smem_u32(bar);
  if (INLINE) return wait_warp([&] { return mbar_try_wait(b, parity); }, ctl, status);
  return __all_sync(0xffffffffu, mbar_try_wait(b, parity)) || wait_bar_slow(b, parity, ctl, status);
}
// until the producer has published entry `uc` of a unit ring
__device__ __forceinline__ bool wait_posted(SharedCtl* ctl, int ln, int uc, int* status) {
  return wait_warp([&] { return ctl->units_posted[ln] > uc; }, ctl, status);
}
// Bounded rendezvous of the warps that share `bar` (initialised with their number); `n` counts this warp's uses of it.
template <bool INLINE = false>
__device__ __forceinline__ bool warps_sync(unsigned long long* bar, uint32_t& n, int lane, SharedCtl* ctl, int* status) {
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
  return wait_bar<INLINE>(bar, n++ & 1, ctl, status);
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

struct DocMaps {
  CUtensorMap m[N_BOXES];  // document boxes of 32, 64, 96 rows, one 128-byte slab wide
};

// Word the producer leaves beside every ring stage for the MMA issuer.
constexpr uint32_t STAGE_COLS_MASK = 0x7Fu;    // rows of the stage that are multiplied: a multiple of 32
constexpr uint32_t STAGE_ACC1 = 1u << 16;      // one resident tile: the piece goes to the stream's second accumulator
constexpr uint32_t STAGE_FIRST = 1u << 18;     // no piece: the query tiles change
constexpr uint32_t STAGE_END = 1u << 20;       // no more work
constexpr uint32_t STAGE_LONE = 1u << 21;      // the second accumulator has no query tile: it changes hands, nothing is multiplied into it
constexpr uint32_t STAGE_SPLIT = 1u << 22;     // the last box of the stage does not follow the others: it ends where the document ends

// WINNERS: 0 = scores only, 1 = winners saved, 2 = winners saved and every document takes the lazy winner scan (launched
// for problems whose documents are long, so that the kernels for short documents carry no third copy of the tile loop)
template <bool FP8, int WINNERS, bool SCALED>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fwd_streams_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ DocMaps d_maps, const TcParams P) {
  constexpr bool ARGMAX = WINNERS != 0;
  // The last box of a document that is not a multiple of 32 tokens is moved back to end where the document ends: the
  // columns it shares with the box before hold the same dot products twice, which no maximum minds, and no column has to
  // be masked.  (Multipliers per column do not move along.)
  constexpr bool SHIFT = !SCALED;
  extern __shared__ unsigned char smem_raw[];
  // operand tiles need 1024-byte alignment for the 128-byte swizzle
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int q_tile_bytes = P.n_slabs * TILE_M * SLAB_BYTES_ROW;
  const int d_stage_bytes = P.n_slabs * TILE_N * SLAB_BYTES_ROW;
  unsigned char* q_smem = smem;                              // [n_slabs][128 rows][128 B], a tile on its way to tensor memory
  unsigned char* d_smem = smem + q_tile_bytes;               // [2 streams][stages][n_slabs][rows][128 B]
  float* sc_ring = reinterpret_cast<float*>(d_smem + (size_t)2 * P.stages * d_stage_bytes);  // [2 streams][sc_per][TILE_N] (kernels with multipliers)
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(d_smem + (size_t)2 * P.stages * d_stage_bytes + (size_t)P.sc_slots * TILE_N * sizeof(float));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const bool list = P.pairing == LIK_PAIR_LIST;
  const bool topk = !ARGMAX && P.topk.cand_key != nullptr;  // the fused top-k never saves winners

  if (tid == 0) {
    mbar_init(smem_u32(&ctl->q_full), 1);
    mbar_init(smem_u32(&ctl->q_empty), 1);
    mbar_init(smem_u32(&ctl->a_idle), 2);
    mbar_init(smem_u32(&ctl->a_ready), 1);
    for (int i = 0; i < 2; ++i)
      for (int s = 0; s < P.stages; ++s) {
        mbar_init(smem_u32(&ctl->d_full[i][s]), 1);
        mbar_init(smem_u32(&ctl->d_empty[i][s]), 1);
      }
    for (int a = 0; a < SETS; ++a) {
      mbar_init(smem_u32(&ctl->acc_full[a]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[a]), SET_WARPS);
      mbar_init(smem_u32(&ctl->set_sync[a]), SET_WARPS);
    }
    ctl->abort_flag = 0;
    ctl->wait_limit = WAIT_LIMIT_CYCLES;
    for (int i = 0; i < SETS; ++i) ctl->units_posted[i] = 0;
    fence_barrier_init();
    prefetch_tmap(&q_map);
    for (int i = 0; i < N_BOXES; ++i) prefetch_tmap(&d_maps.m[i]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctl->tmem_base), 512);
    tmem_relinquish();
  }
  // Launched with programmatic stream serialisation: the set-up above overlaps the kernel in front, nothing below may.
  griddep_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  // greedy-packed query tiles are counted on the device (the count sits in front of the table)
  const int n_tiles = P.tile_q0 ? P.tile_q0[-1] : P.n_tiles;
  const int n_groups = (n_tiles + P.mt - 1) / P.mt;

  if (warp == 0 || warp == 19) {
    // =========================== producers ===========================
    // Two streams, each with a producer and an issuer of its own, share the tensor pipe and the resident query tiles: whatever a
    // warp does for a piece - a wait on a barrier alone takes more than a hundred cycles, also one that is complete already - has
    // the time of two pieces.  A CTA's units go to the streams in turn; both pass through the same tile groups.
    // The warp walks the units (32 are looked up at a time, a thread each), cuts them into pieces, loads these with TMA and
    // publishes units and pieces.  It runs on warp-uniform values and one elected lane issues, as in the issuers below: TMA
    // instructions, too, take their operands from uniform registers.
    const int sm = warp == 0 ? 0 : 1;
    const bool elect = elect_one();
    const int x_per_slab = SLAB_BYTES_ROW / P.elt_bytes, n_slabs = P.n_slabs, stages = P.stages, mt = P.mt;
    unsigned char* const ring = d_smem + (size_t)sm * stages * d_stage_bytes;
    unsigned long long *const d_full = ctl->d_full[sm], *const d_empty = ctl->d_empty[sm];
    int cur_grp = -1;
    uint32_t n_qload = 0, st = 0, ph = 0, n_dload = 0, lone = 0;
    int n_unit[2] = {0, 0}, n_slot = 0, turn = 0;  // units by accumulator (one resident tile) or the first alone (two)
    bool ok = true;
    // One stage: `rows` of `ncols` document rows from `row` on; split: two boxes, the second at row2
    auto stage = [&](uint32_t info, int ncols, int row, int row2, int slot) {
      ok = wait_bar(&d_empty[st], ph ^ 1, ctl, P.status);
      if (!ok) return;
      const uint32_t full = smem_u32(&d_full[st]);
      const int rows = (int)(info & STAGE_COLS_MASK);
      {
        if (elect) {
          ctl->stage_info[sm][st] = info;
          if (rows > 0) {
            const uint32_t dst = smem_u32(ring) + st * (uint32_t)d_stage_bytes;
            // the piece's multipliers ride on the same barrier: whole groups of four floats, never past the array's end
            const uint32_t sc_bytes = SCALED && P.col_src ? (uint32_t)min((long long)((ncols + 3) & ~3), P.d.n_rows - row) * 4u : 0u;
            mbar_arrive_expect_tx(full, (uint32_t)(rows * SLAB_BYTES_ROW * n_slabs) + sc_bytes);
            const int box = rows / BOX_ROWS - 1;
            const bool split = info & STAGE_SPLIT;
            for (int sl = 0; sl < n_slabs; ++sl) {
              const uint32_t at = dst + sl * TILE_N * SLAB_BYTES_ROW;
              tma_load_2d(at, &d_maps.m[split ? box - 1 : box], sl * x_per_slab, row, full);
              if (split) tma_load_2d(at + box * BOX_ROWS * SLAB_BYTES_ROW, &d_maps.m[0], sl * x_per_slab, row2, full);
            }
            if (sc_bytes) bulk_load_1d(smem_u32(sc_ring + slot * TILE_N), P.col_src + row, sc_bytes, full);
          } else {
            mbar_arrive(full);  // an empty document, new query tiles, or the end
          }
        }
        __syncwarp();
      }
      ++n_dload;
      if (++st == (uint32_t)stages) { st = 0; ph ^= 1; }
    };
    // a batch of units that is dealt out, and one whose length words are on their way
    UnitWalk walk{0, 0, 0, 0, 0};
    walk_settle(P, n_groups, walk);
    UnitRaw raw{0, 0, 0, 0};
    int n_raw = 0;
    auto fetch_batch = [&]() {
      n_raw = (int)min(32ll, walk.u_end - walk.u);
      if (n_raw > 0) {
        if (lane < n_raw) raw = unit_fetch(P, walk, walk.u + lane);
        walk.u += n_raw;
        walk_settle(P, n_groups, walk);
      }
    };
    fetch_batch();
    int parity = sm;  // units until this stream's next
    while (ok && n_raw > 0) {
      const int n = n_raw, u_doc = raw.doc, u_grp = raw.grp;  // this thread's unit
      int u_row = 0, u_len = 0;
      bool masked = false;
      unit_resolve(P, raw, u_row, u_len, masked);
      u_len = (u_len & UNIT_LEN_MASK) | (masked ? LEN_FLAG_MASKED : 0);
      fetch_batch();
      for (int i = 0; ok && i < n; ++i) {
        const int grp = __shfl_sync(0xffffffffu, u_grp, i);
        if (grp != cur_grp) {
          cur_grp = grp;
          const int t0 = grp * mt, t1 = min(t0 + mt, n_tiles);
          lone = mt == 2 && t1 - t0 < 2 ? STAGE_LONE : 0u;
          for (int t = t0; t < t1; ++t) {
            if (sm == 0) {
              // one tile at a time through the place in shared memory, which is free when its copy to tensor memory is made
              ok = wait_bar(&ctl->q_empty, (n_qload & 1) ^ 1, ctl, P.status);
              if (!ok) break;
              if (elect) {
                mbar_arrive_expect_tx(smem_u32(&ctl->q_full), (uint32_t)q_tile_bytes);
                const int row = (int)tile_info(P, t).row0;
                for (int sl = 0; sl < n_slabs; ++sl)
                  tma_load_2d(smem_u32(q_smem + sl * TILE_M * SLAB_BYTES_ROW), &q_map, sl * x_per_slab, row, smem_u32(&ctl->q_full));
              }
              __syncwarp();
              ++n_qload;
            }
            // a stage of its own tells the issuers; it goes in front of the second tile, whose load waits for the first one's copy
            if (t == t0) stage(STAGE_FIRST | lone, 0, 0, 0, 0);
            if (!ok) break;
          }
          if (!ok) break;
        }
        if (parity) {
          --parity;
          continue;
        }
        parity = 1;
        const int doc = __shfl_sync(0xffffffffu, u_doc, i), drow0 = __shfl_sync(0xffffffffu, u_row, i), len = __shfl_sync(0xffffffffu, u_len, i);
        const int dlen = len & UNIT_LEN_MASK, j = mt == 2 ? 0 : turn, ln = 2 * sm + j;
        turn ^= 1;
        // publish the unit for the epilogue; an empty document still sends one (empty) piece so that every unit passes through
        // the same hand-shakes
        int slot = n_slot;
        if (elect) {
          const int at = j ? n_unit[1] : n_unit[0];
          ctl->unit_info[ln][at & (UNIT_RING - 1)] = make_int4(dlen | slot << UNIT_SLOT_SHIFT | (len & LEN_FLAG_MASKED), drow0, grp, doc);
          if (SCALED) {  // (the others learn of it from a full accumulator)
            __threadfence_block();
            ctl->units_posted[ln] = at + 1;
          }
        }
        if (j) ++n_unit[1];
        else ++n_unit[0];
        int c0 = 0;
        do {
          const int ncols = min(TILE_N, dlen - c0), rows = __shfl_sync(0xffffffffu, (ncols + BOX_ROWS - 1) & ~(BOX_ROWS - 1), 0);
          // A short document that is no multiple of 32 tokens takes two boxes, the second moved back to end where the document
          // ends; a longer one's last piece is moved back as a whole.
          const bool split = SHIFT && dlen < rows && dlen > BOX_ROWS;
          stage((uint32_t)rows | lone | (j ? STAGE_ACC1 : 0u) | (split ? STAGE_SPLIT : 0u), ncols,
                __shfl_sync(0xffffffffu, drow0 + (SHIFT ? max(min(c0, dlen - rows), 0) : c0), 0), __shfl_sync(0xffffffffu, drow0 + dlen - BOX_ROWS, 0),
                SCALED ? sm * P.sc_per + slot : 0);
          if (SCALED && ++slot >= P.sc_per) slot = 0;
          c0 += TILE_N;
        } while (ok && c0 < dlen);
        n_slot = slot;
      }
    }
    if (ok) {
      // tell the epilogue sets and the issuer that the stream has ended
      if (elect) {
        for (int j = 0; j < 3 - mt; ++j) {
          const int at = j ? n_unit[1] : n_unit[0];
          ctl->unit_info[2 * sm + j][at & (UNIT_RING - 1)] = make_int4(UNIT_END, 0, 0, 0);
          if (SCALED) {
            __threadfence_block();
            ctl->units_posted[2 * sm + j] = at + 1;
          }
        }
      }
      __syncwarp();
      stage(STAGE_END, 0, 0, 0, 0);
    }
    if (elect) {
      // let the copies already issued land before the CTA goes away: an issuer that gives up takes no more of them
      for (uint32_t i = 1; i <= (uint32_t)stages && i <= n_dload; ++i) {
        const bool wrapped = i > st;  // that use lies before the last wrap of the ring
        const uint32_t at = wrapped ? st + (uint32_t)stages - i : st - i;
        const uint32_t bar = smem_u32(&d_full[at]);
        for (int spin = 0; spin < (1 << 16) && !mbar_try_wait_long(bar, wrapped ? ph ^ 1 : ph); ++spin) {
        }
      }
      if (n_qload) {
        const uint32_t bar = smem_u32(&ctl->q_full);
        for (int spin = 0; spin < (1 << 16) && !mbar_try_wait_long(bar, (n_qload - 1) & 1); ++spin) {
        }
      }
    }
  } else if (warp == 1 || warp == 18) {
    // =========================== MMA issuers ===========================
    // Driven by the stage words alone.  A whole warp runs the loop on warp-uniform values and one elected lane issues:
    // tcgen05.mma takes its descriptors from uniform registers, and with the loop under `lane == 0` every MMA paid about 100
    // cycles for moving them there, whatever its width.
    const uint32_t sm = warp == 1 ? 0u : 1u;
    const bool two = P.mt == 2;
    unsigned long long *const d_full = ctl->d_full[sm], *const d_empty = ctl->d_empty[sm], *const acc_empty = &ctl->acc_empty[2 * sm],
                             *const acc_full = &ctl->acc_full[2 * sm];
    uint32_t st = 0, ph = 0, n_q = 0, n_grp = 0, acc_ph = 3;  // acc_ph: one phase bit per accumulator
    const uint32_t stages = (uint32_t)P.stages;
    const bool issue = elect_one();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const uint32_t b_desc0 = (uint32_t)smem_desc_sw128(smem_u32(d_smem + (size_t)sm * P.stages * d_stage_bytes));
    const uint32_t stage_desc = (uint32_t)(d_stage_bytes >> 4);
    const uint32_t idesc0 = instr_desc(P.ab_format, 0);
    const uint32_t d_tmem0 = tmem_base + 2 * sm * ACC_COLS, a_tmem0 = tmem_base + A_COL0;
    const int k_steps = P.k_steps;
    constexpr uint32_t A_SLAB = (TILE_M * SLAB_BYTES_ROW) >> 4, B_SLAB = (TILE_N * SLAB_BYTES_ROW) >> 4;
    // the MMAs of one tile on one stage
    auto multiply = [&](uint32_t acc, uint32_t tile, uint32_t rows, uint32_t b_stage) {
      const uint32_t idesc = idesc0 | (rows << 14);  // N / 8 in bits 17..22
      const uint32_t d_tmem = d_tmem0 + acc * ACC_COLS, a_tmem = a_tmem0 + tile * A_COLS;
      // descriptors differ only in the start address, in units of 16 bytes
      if (k_steps == 8) {  // the common width (128 two-byte or 256 one-byte elements): straight-line issue
#pragma unroll
        for (int k = 0; k < 8; ++k)
          tc_mma_ts<FP8>(d_tmem, a_tmem + 8 * k, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * B_SLAB, desc_hi, idesc, k ? 1u : 0u);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < k_steps) tc_mma_ts<FP8>(d_tmem, a_tmem + 8 * k, b_stage + (uint32_t)((k & 3) * 2) + (k >> 2) * B_SLAB, desc_hi, idesc, k ? 1u : 0u);
      }
    };
    while (true) {
      if (!wait_bar(&d_full[st], ph, ctl, P.status)) break;
      const uint32_t info = __shfl_sync(0xffffffffu, ctl->stage_info[sm][st], 0);
      if (info & (STAGE_FIRST | STAGE_END)) {
        if (info & STAGE_END) {
          // the accumulators change hands once more, empty: the sets find the end of the stream in their unit ring
          for (uint32_t a = 0; a < 2; ++a) {
            if (!wait_bar(&acc_empty[a], (acc_ph >> a) & 1u, ctl, P.status)) break;
            if (issue) tc_commit(smem_u32(&acc_full[a]));
            __syncwarp();
          }
          break;
        }
        // New query tiles: they go to tensor memory when all MMAs of both streams on the old ones are done; the first stream's
        // issuer copies them.
        if (issue) tc_commit(smem_u32(&ctl->a_idle));
        __syncwarp();
        bool ok = true;
        if (sm == 0) {
          ok = wait_bar(&ctl->a_idle, n_grp & 1u, ctl, P.status);
          const uint32_t n_new = two && !(info & STAGE_LONE) ? 2u : 1u;
          for (uint32_t t = 0; ok && t < n_new; ++t, ++n_q) {
            ok = wait_bar(&ctl->q_full, n_q & 1u, ctl, P.status);
            if (!ok) break;
            tc_fence_after();
            if (issue) {
              const uint32_t a_desc = (uint32_t)smem_desc_sw128(smem_u32(q_smem));
              for (int k = 0; k < k_steps; ++k) tc_copy_128x256b(a_tmem0 + t * A_COLS + 8 * k, a_desc + (uint32_t)((k & 3) * 2) + (k >> 2) * A_SLAB, desc_hi);
              tc_commit(smem_u32(&ctl->q_empty));
              if (t + 1 == n_new) tc_commit(smem_u32(&ctl->a_ready));
            }
            __syncwarp();
          }
        }
        ok = ok && wait_bar(&ctl->a_ready, n_grp & 1u, ctl, P.status);
        if (!ok) break;
        ++n_grp;
      }
      const uint32_t rows = info & STAGE_COLS_MASK;
      const uint32_t b_stage = b_desc0 + st * stage_desc;
      if (info & STAGE_FIRST) {
        // (a stage that only announced them: nobody else gives it back)
        if (issue) mbar_arrive(smem_u32(&d_empty[st]));
      } else if (two) {
        // (the accumulators always change hands, so that both sides keep their phase)
        if (!wait_bar(&acc_empty[0], acc_ph & 1u, ctl, P.status)) break;
        tc_fence_after();
        if (issue) {
          if (rows) multiply(0, 0, rows, b_stage);
          tc_commit(smem_u32(&acc_full[0]));
        }
        __syncwarp();
        if (!wait_bar(&acc_empty[1], (acc_ph >> 1) & 1u, ctl, P.status)) break;
        acc_ph ^= 3u;
        tc_fence_after();
        if (issue) {
          if (rows && !(info & STAGE_LONE)) multiply(1, 1, rows, b_stage);
          tc_commit(smem_u32(&acc_full[1]));
          tc_commit(smem_u32(&d_empty[st]));  // ring slot reusable once these MMAs retire
        }
      } else {
        const uint32_t a = info & STAGE_ACC1 ? 1u : 0u;
        if (!wait_bar(&acc_empty[a], (acc_ph >> a) & 1u, ctl, P.status)) break;
        acc_ph ^= 1u << a;
        tc_fence_after();
        if (issue) {
          if (rows) multiply(a, 0, rows, b_stage);
          tc_commit(smem_u32(&acc_full[a]));
          tc_commit(smem_u32(&d_empty[st]));
        }
      }
      __syncwarp();
      if (++st == stages) { st = 0; ph ^= 1; }
    }
  } else if (warp >= EPI_WARP0) {
    // =========================== epilogue sets ===========================
    // Set s (four warps) drains accumulator s, which belongs to stream s >> 1: with two resident query tiles, tile s & 1 of all the
    // stream's units; with one, every second unit.
    // A warp owns 32 rows of a document from its first column to its score.  It waits for its accumulator by itself and gives
    // it back by itself; the warps of a set meet only where the query tile changes, where columns are staged by all of them
    // and where a query's rows lie in several warps.  All of these waits are bounded: a warp that gives up leaves the
    // loop, and the others' waits find the abort flag.
    const int e = warp - EPI_WARP0;
    const int set = e >> 2;
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int wq = e & 3;                    // warp index inside the set
    const int row = quad * 32 + lane;        // accumulator row == query token slot in the tile
    const int et = wq * 32 + lane;           // thread index inside the set (0..127)
    const int sm = set >> 1;                 // stream
    const int ln = P.mt == 2 ? set & 2 : set;  // whose unit ring
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
#define LIK_SET_SYNC() warps_sync<ARGMAX && !SCALED>(&ctl->set_sync[set], n_sync, lane, ctl, P.status)
#define LIK_WAIT_ACC() wait_bar<ARGMAX && !SCALED>(&ctl->acc_full[set], n_acc & 1, ctl, P.status)
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
    const bool bulk = SCALED && P.sc_slots != 0;  // the multipliers of a piece arrive with it
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
            // the candidate list of (this CTA, this group, this set, this query)
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
        const float* const sc_arr = SCALED && bulk ? sc_ring + (sm * P.sc_per + sc_slot) * TILE_N : col_scale;
        auto stage_columns = [&]() {
          ++n_col;
          const int c = et;  // a thread per column
          if (c < ((ncols + 31) & ~31)) {
            float sc = 1.f, bi = -INFINITY;
            const int tok = SHIFT && dlen >= BOX_ROWS ? min(base + (c & ~31), dlen - BOX_ROWS) + (c & 31) : base + c;  // the token that column c stands for
            if (tok < dlen) {
              const long long drow = drow0 + tok;
              sc = row_factor(P.d, drow);
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
        } else {
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
        if (P.q_chunks == 1) {
          const long long o = cross ? (long long)qq * P.n_d + out_col : out_col;
          LIK_EMIT_SCORE(sg, sum, o);
        } else if (lane == 0) {
          P.partial[(long long)tile_id * P.n_d + doc] = sum;  // a piece of a long query
        }
      }
    }
    // top-k: leave the lists' state where the next launch stage (the merge) finds it
    if (topk && ok && LIK_SET_SYNC()) LIK_TOPK_STORE_BACK();
#undef LIK_EMIT_SCORE
#undef LIK_TOPK_STORE_BACK
#undef LIK_WAIT_ACC
#undef LIK_SET_SYNC
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


// The bounded waits of the kernel above, alone (see wait_probe_kernel in lik_fwd_tc.cu): a warp waits on a barrier that nothing
// arrives at, then for a unit that nobody posts, then for a second warp that never comes.
// result[3 * w + ...] = lanes that were told to go on (0: all gave up), the abort flag, cycles spent by the slowest lane.
__global__ void streams_wait_probe_kernel(long long limit, int* status, int* result) {
  __shared__ SharedCtl ctl;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctl.q_full), 1);
    mbar_init(smem_u32(&ctl.set_sync[0]), 2);
    ctl.units_posted[0] = 0;
    ctl.wait_limit = limit;
    fence_barrier_init();
  }
  for (int w = 0; w < 3; ++w) {
    if (threadIdx.x == 0) ctl.abort_flag = 0;
    __syncwarp();
    uint32_t n = 0;
    const long long t0 = clock64();
    const bool got = w == 0   ? wait_bar<true>(&ctl.q_full, 0, &ctl, status)
                     : w == 1 ? wait_posted(&ctl, 0, 0, status)
                              : warps_sync(&ctl.set_sync[0], n, (int)threadIdx.x, &ctl, status);
    const long long dt = clock64() - t0;
    const int lanes = __popc(__ballot_sync(0xffffffffu, got));
    const unsigned cycles = __reduce_max_sync(0xffffffffu, dt > 0x7fffffffll ? 0x7fffffffu : (unsigned)dt);
    if (threadIdx.x == 0) {
      result[3 * w] = lanes;
      result[3 * w + 1] = ctl.abort_flag;
      result[3 * w + 2] = (int)cycles;
    }
    __syncwarp();
  }
}

template <bool F, int A, bool X>
cudaError_t launch_one(const cudaLaunchConfig_t& cfg, const CUtensorMap& q_map, const DocMaps& d_maps, const TcParams& P) {
  cudaError_t e = allow_smem<fwd_streams_kernel<F, A, X>>();
  if (e != cudaSuccess) return e;
  e = cudaLaunchKernelEx(&cfg, fwd_streams_kernel<F, A, X>, q_map, d_maps, P);
  count_launch();
  return e;
}

}  // namespace

size_t fwd_streams_fixed_smem(int n_slabs) { return (size_t)n_slabs * TILE_M * SLAB_BYTES_ROW + sizeof(SharedCtl) + 1024; }
size_t fwd_streams_stage_bytes(int n_slabs) { return 2 * (size_t)n_slabs * TILE_N * SLAB_BYTES_ROW; }
size_t fwd_streams_slot_bytes() { return TILE_N * sizeof(float); }

int launch_streams_wait_probe(long long limit, int* status, int* result, cudaStream_t st) {
  streams_wait_probe_kernel<<<1, 32, 0, st>>>(limit, status, result), count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

int launch_fwd_streams(const lik_fwd_args& a, const TcPlan& pl, const TcParams& P, bool affine, bool long_docs, cudaStream_t st) {
  CUtensorMap q_map;
  DocMaps d_maps;
  memset(&d_maps, 0, sizeof(d_maps));
  int rc = make_tmap_rows(&q_map, a.q.data, a.dtype, a.dim, a.q.n_rows, a.q.row_stride, TILE_M);
  for (int i = 0; i < N_BOXES && !rc; ++i)
    rc = make_tmap_rows(&d_maps.m[i], a.d.data, a.dtype, a.dim, a.d.n_rows, a.d.row_stride, (i + 1) * BOX_ROWS);
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
  const bool fp8 = a.dtype == LIK_E4M3, argmax = a.argmax != nullptr;
#define LIK_STREAMS_LAUNCH(F, A, X) LIK_CUDA_OK((launch_one<F, A, X>(cfg, q_map, d_maps, P)))
  if (fp8) {
    if (argmax && affine) LIK_STREAMS_LAUNCH(true, 1, true);
    else if (argmax) LIK_STREAMS_LAUNCH(true, 1, false);
    else if (affine) LIK_STREAMS_LAUNCH(true, 0, true);
    else LIK_STREAMS_LAUNCH(true, 0, false);
  } else {
    if (long_docs && affine) LIK_STREAMS_LAUNCH(false, 2, true);
    else if (long_docs) LIK_STREAMS_LAUNCH(false, 2, false);
    else if (argmax && affine) LIK_STREAMS_LAUNCH(false, 1, true);
    else if (argmax) LIK_STREAMS_LAUNCH(false, 1, false);
    else if (affine) LIK_STREAMS_LAUNCH(false, 0, true);
    else LIK_STREAMS_LAUNCH(false, 0, false);
  }
#undef LIK_STREAMS_LAUNCH
  return LIK_OK;
}

}  // namespace lik
