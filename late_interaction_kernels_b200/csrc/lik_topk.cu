// Per-query top-k selection and merge.
//
// One CTA per query row keeps the current best KP = pow2(k) candidates sorted in
// shared memory.  New candidates arrive KP at a time (a slice of a score row, or
// one of several already-selected lists), are bitonic-sorted, combined with the
// kept list by the "best of top[i] and block[KP-1-i]" step (which leaves the KP
// best of the union as a bitonic sequence) and re-sorted by a bitonic merge.  Blocks
// of a score row in which nothing beats the current k-th best are skipped after one
// read of their values.
// Order: better score first, ties to the lower document index; padding
// (index < 0) last.
#include <climits>

#include "lik_common.cuh"

namespace lik {

struct Cand {
  float key;  // score for largest=true, -score otherwise
  long long idx;
};

__device__ __forceinline__ bool before(const Cand& a, const Cand& b) {
  return a.key > b.key || (a.key == b.key && a.idx < b.idx);
}

constexpr long long kPadIdx = LLONG_MAX;

// sort KP entries in shared memory, best first
__device__ void bitonic_sort(float* key, long long* idx, int KP, int tid, int nthreads) {
  for (int size = 2; size <= KP; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int t = tid; t < (KP >> 1); t += nthreads) {
        int i = 2 * t - (t & (stride - 1));
        int j = i + stride;
        bool up = (i & size) == 0;  // this sub-sequence is ordered best first
        Cand a{key[i], idx[i]}, b{key[j], idx[j]};
        bool swap = up ? before(b, a) : before(a, b);
        if (swap) {
          key[i] = b.key;
          idx[i] = b.idx;
          key[j] = a.key;
          idx[j] = a.idx;
        }
      }
    }
  }
  __syncthreads();
}

// merge a bitonic sequence of KP entries into best-first order
__device__ void bitonic_merge(float* key, long long* idx, int KP, int tid, int nthreads) {
  for (int stride = KP >> 1; stride > 0; stride >>= 1) {
    __syncthreads();
    for (int t = tid; t < (KP >> 1); t += nthreads) {
      int i = 2 * t - (t & (stride - 1));
      int j = i + stride;
      Cand a{key[i], idx[i]}, b{key[j], idx[j]};
      if (before(b, a)) {
        key[i] = b.key;
        idx[i] = b.idx;
        key[j] = a.key;
        idx[j] = a.idx;
      }
    }
  }
  __syncthreads();
}

struct TopkParams {
  // mode 0: slices of a score row; mode 1: lists [n_lists, n_rows, k]
  int mode;
  const float* scores;
  long long n_cols, ld, index_offset;
  const float* cand_scores;
  const long long* cand_index;
  int n_lists;
  long long n_rows;
  int k, KP, largest, merge;
  float* out_scores;
  long long* out_index;
};

template <int NT, int MIN_CTAS>
__global__ void __launch_bounds__(NT, MIN_CTAS) topk_kernel(TopkParams P) {
  extern __shared__ unsigned char raw[];
  long long* top_i = reinterpret_cast<long long*>(raw);
  long long* blk_i = top_i + P.KP;
  float* top_k = reinterpret_cast<float*>(blk_i + P.KP);
  float* blk_k = top_k + P.KP;
  const int tid = threadIdx.x, nt = blockDim.x;
  const long long row = blockIdx.x;
  const float sgn = P.largest ? 1.f : -1.f;

  for (int t = tid; t < P.KP; t += nt) {
    float key = -INFINITY;
    long long id = kPadIdx;
    if (P.merge && t < P.k) {
      long long o = P.out_index[row * P.k + t];
      if (o >= 0) {
        id = o;
        key = sgn * P.out_scores[row * P.k + t];
      }
    }
    top_k[t] = key;
    top_i[t] = id;
  }
  __syncthreads();
  if (P.merge) bitonic_sort(top_k, top_i, P.KP, tid, nt);

  const long long n_blocks = P.mode == 0 ? (P.n_cols + P.KP - 1) / P.KP : P.n_lists;
  for (long long b = 0; b < n_blocks; ++b) {
    // A block of new candidates matters only if one of them beats the current k-th best: the kept list
    // never gets worse, so anything behind that entry can never reach the output.  Once the list is warm
    // almost every block is dismissed by this one pass over its values.
    if (P.mode == 0) {
      const Cand kth{top_k[P.k - 1], top_i[P.k - 1]};
      int hit = 0;
      for (int t = tid; t < P.KP; t += nt) {
        const long long c = b * P.KP + t;
        if (c < P.n_cols && before(Cand{sgn * P.scores[row * P.ld + c], c + P.index_offset}, kth)) hit = 1;
      }
      if (!__syncthreads_or(hit)) continue;
    }
    for (int t = tid; t < P.KP; t += nt) {
      float key = -INFINITY;
      long long id = kPadIdx;
      if (P.mode == 0) {
        long long c = b * P.KP + t;
        if (c < P.n_cols) {
          key = sgn * P.scores[row * P.ld + c];
          id = c + P.index_offset;
        }
      } else if (t < P.k) {
        long long o = (b * P.n_rows + row) * P.k + t;
        long long ci = P.cand_index[o];
        if (ci >= 0) {
          id = ci;
          key = sgn * P.cand_scores[o];
        }
      }
      blk_k[t] = key;
      blk_i[t] = id;
    }
    bitonic_sort(blk_k, blk_i, P.KP, tid, nt);
    for (int t = tid; t < P.KP; t += nt) {
      Cand a{top_k[t], top_i[t]}, c{blk_k[P.KP - 1 - t], blk_i[P.KP - 1 - t]};
      if (before(c, a)) {
        top_k[t] = c.key;
        top_i[t] = c.idx;
      }
    }
    bitonic_merge(top_k, top_i, P.KP, tid, nt);
  }
  for (int t = tid; t < P.k; t += nt) {
    bool pad = top_i[t] == kPadIdx;
    P.out_scores[row * P.k + t] = pad ? -sgn * INFINITY : sgn * top_k[t];
    P.out_index[row * P.k + t] = pad ? -1 : top_i[t];
  }
}

// Merge of the candidate lists the fused scoring kernels leave (lik_fwd_tc.cuh): list slot of (CTA c, tile
// group g) is c + g, each slot holds `lists` * qpt lists of up to 256 entries (unsorted), and CTA c of n_ctas can
// only have worked on the groups [n_groups * c / n_ctas, n_groups * (c + 1) / n_ctas] (a superset of the ones
// it really met; lists it never touched are empty).  A group is `mt` query tiles of `qpt` queries.  A kernel has lists of its
// own for every document it has in flight: a query has lists / mt of them per slot.
//
// An entry becomes one 64-bit number, larger = better: the score's ordered key above the complement of the document
// index, so that ties need no second look.  A CTA holds the entries of up to 32 lists in registers (sixteen per thread),
// finds the k-th largest by bisection on the bits with a block-wide count per bit - neighbouring scores share their upper
// bits, on which a radix histogram's counters collide - and sorts the k survivors.  A query with more lists (few tile
// groups: lists from every CTA) is cut in parts, whose winners go through the same selection once more.  One query over
// 25 000 documents, 296 lists: 91 -> 26 us in two kernels (list after list through bitonic merges before).
typedef unsigned long long u64;
constexpr int SLOT_CAP = 256;     // entries of a candidate list
constexpr int SLOT_LISTS = 32;    // lists per CTA
constexpr int SLOT_T = 512;
constexpr int SLOT_PER = SLOT_LISTS * SLOT_CAP / SLOT_T;
constexpr int SLOT_K = 128;       // largest k of the fused path
constexpr int SLOT_CTAS = 512;    // largest grid whose lists it takes

struct SlotParams {
  const float* keys;
  const int* idx;
  const int2* hdr;
  int n_ctas, n_groups, mt, lists, qpt;
  long long n_q, index_offset, n_lists;
  int k, largest;
  float* out_scores;
  long long* out_index;
  int parts;   // lists of a query are merged in this many parts first ...
  u64* part;   // ... into [parts, n_q, k] entries (0: none)
};

__device__ __forceinline__ unsigned slot_order(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float slot_unorder(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// The k largest of the block's entries (0: none), written to out[0 .. n) in shared memory, best first; returns n.
__device__ int slot_select(const u64 (&e)[SLOT_PER], int k, u64* out, int* cnt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int WARPS = SLOT_T / 32;
  // block-wide count of the entries at or above a bound (cnt: two rows of WARPS words, used in turn)
  int turn = 0;
  auto count_ge = [&](u64 bound) {
    int c = 0;
#pragma unroll
    for (int j = 0; j < SLOT_PER; ++j) c += e[j] >= bound ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    int* row = cnt + (turn & 1) * WARPS;
    ++turn;
    if (lane == 0) row[warp] = c;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < WARPS ? row[lane] : 0);
  };
  u64 kth = 1;
  const int total = count_ge(1);
  if (total > k) {
    kth = 0;
    for (int bit = 63; bit >= 0; --bit) {
      const u64 cand = kth | (1ull << bit);
      const int c = count_ge(cand);
      if (c >= k) kth = cand;
      if (c == k) break;  // exactly the k best lie at or above it
    }
  }
  const int n = total < k ? total : k;
  int* fill = cnt + 2 * WARPS;
  if (tid == 0) *fill = 0;
  for (int t = tid; t < SLOT_K; t += SLOT_T) out[t] = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SLOT_PER; ++j)
    if (e[j] >= kth && e[j] != 0) {
      const int pos = atomicAdd(fill, 1);
      if (pos < SLOT_K) out[pos] = e[j];
    }
  int KP = 2;
  while (KP < n) KP <<= 1;
  for (int size = 2; size <= KP; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      if (tid < (KP >> 1)) {
        const int i = 2 * tid - (tid & (stride - 1)), j = i + stride;
        const bool up = (i & size) == 0;
        const u64 a = out[i], b = out[j];
        if (up ? b > a : a > b) {
          out[i] = b;
          out[j] = a;
        }
      }
    }
  __syncthreads();
  return n;
}

__device__ __forceinline__ void slot_write(const SlotParams& P, long long q, const u64* top, int n) {
  const float sgn = P.largest ? 1.f : -1.f;
  for (int t = threadIdx.x; t < P.k; t += SLOT_T) {
    const u64 v = t < n ? top[t] : 0;
    P.out_scores[q * P.k + t] = v ? sgn * slot_unorder((unsigned)(v >> 32)) : -sgn * INFINITY;
    P.out_index[q * P.k + t] = v ? (long long)(unsigned)~(unsigned)v + P.index_offset : -1;
  }
}

// grid (n_q, parts)
__global__ void __launch_bounds__(SLOT_T) topk_slots_kernel(SlotParams P) {
  __shared__ u64 top[SLOT_K];
  __shared__ int cnt[2 * SLOT_T / 32 + 1];
  __shared__ int slots[SLOT_CTAS];  // list slots of this query, in CTA order
  __shared__ int n_slots_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long q = blockIdx.x;
  const int tile = (int)(q / P.qpt), et = (int)(q - (long long)tile * P.qpt);
  const int g = tile / P.mt, m = tile - g * P.mt;
  const int n_sub = P.lists / P.mt;
  if (warp == 0) {  // the CTAs that can have met this group
    int n = 0;
    for (int c0 = 0; c0 < P.n_ctas; c0 += 32) {
      const int c = c0 + lane;
      const bool hit = c < P.n_ctas && g >= (long long)P.n_groups * c / P.n_ctas && g <= (long long)P.n_groups * (c + 1) / P.n_ctas;
      const unsigned mask = __ballot_sync(0xffffffffu, hit);
      const int pos = n + __popc(mask & ((1u << lane) - 1u));
      if (hit && pos < SLOT_CTAS) slots[pos] = c + g;
      n += __popc(mask);
    }
    if (lane == 0) n_slots_s = n < SLOT_CTAS ? n : SLOT_CTAS;
  }
  __syncthreads();
  const int n_lists = n_slots_s * n_sub;
  const int lo = (int)((long long)n_lists * blockIdx.y / P.parts), hi = (int)((long long)n_lists * (blockIdx.y + 1) / P.parts);
  u64 e[SLOT_PER];
#pragma unroll
  for (int j = 0; j < SLOT_PER; ++j) e[j] = 0;
  constexpr int PER_LIST = SLOT_CAP / 32;
#pragma unroll
  for (int u = 0; u < SLOT_LISTS / (SLOT_T / 32); ++u) {  // a warp per list
    const int li = lo + u * (SLOT_T / 32) + warp;
    if (li < hi) {
      const int sub = li % n_sub;
      const long long list = (long long)slots[li / n_sub] * (P.lists * P.qpt) + (sub * P.mt + m) * P.qpt + et;
      const int c = list < P.n_lists ? min(P.hdr[list].x, SLOT_CAP) : 0;
#pragma unroll
      for (int x = 0; x < PER_LIST; ++x) {
        const int t = x * 32 + lane;
        if (t < c) {
          const float key = P.keys[list * SLOT_CAP + t];
          if (key == key)  // (a score that is no number beats nothing)
            e[u * PER_LIST + x] = ((u64)slot_order(key) << 32) | (unsigned)~(unsigned)P.idx[list * SLOT_CAP + t];
        }
      }
    }
  }
  const int n = slot_select(e, P.k, top, cnt);
  if (P.parts == 1) {
    slot_write(P, q, top, n);
  } else {
    u64* out = P.part + ((long long)blockIdx.y * P.n_q + q) * P.k;
    for (int t = tid; t < P.k; t += SLOT_T) out[t] = t < n ? top[t] : 0;
  }
}

// the parts' winners: at most SLOT_PER * SLOT_T entries
__global__ void __launch_bounds__(SLOT_T) topk_parts_kernel(SlotParams P) {
  __shared__ u64 top[SLOT_K];
  __shared__ int cnt[2 * SLOT_T / 32 + 1];
  const long long q = blockIdx.x;
  const int n_ent = P.parts * P.k;
  u64 e[SLOT_PER];
#pragma unroll
  for (int j = 0; j < SLOT_PER; ++j) {
    const int x = j * SLOT_T + threadIdx.x;
    const int p = x / P.k;
    e[j] = x < n_ent ? P.part[((long long)p * P.n_q + q) * P.k + (x - p * P.k)] : 0;
  }
  const int n = slot_select(e, P.k, top, cnt);
  slot_write(P, q, top, n);
}

static int launch_topk(TopkParams& P, cudaStream_t st);

// In how many parts the lists of a query are merged first: a CTA holds those of one part.  (The CTAs whose share of the
// units can touch one tile group are at most n_ctas / n_groups + 2.)
int topk_merge_parts(int n_ctas, int n_groups, int per_slot) {
  if (n_ctas <= 0 || n_groups <= 0) return 1;
  return (int)ceil_div((int64_t)(n_ctas / n_groups + 2) * per_slot, SLOT_LISTS);
}

int launch_topk_slots(const float* keys, const int* idx, const int2* hdr, long long n_lists, int cap, int n_ctas, int n_groups,
                      int mt, int lists, int qpt, long long n_q, int k, int largest, long long index_offset, float* out_scores,
                      long long* out_index, int parts, void* part_buf, cudaStream_t st) {
  if (n_q <= 0 || k <= 0) return LIK_OK;
  if (cap != SLOT_CAP || k > SLOT_K || n_ctas > SLOT_CTAS || parts * k > SLOT_PER * SLOT_T || (parts > 1 && !part_buf)) {
    set_error("candidate lists of %d entries from %d CTAs, k = %d: outside what the merge takes", cap, n_ctas, k);
    return LIK_ERR_UNSUPPORTED;
  }
  SlotParams P{keys, idx, hdr, n_ctas, n_groups, mt, lists, qpt, n_q, index_offset, n_lists, k, largest, out_scores, out_index, parts, (u64*)part_buf};
  topk_slots_kernel<<<dim3((unsigned)n_q, (unsigned)parts), SLOT_T, 0, st>>>(P), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  if (parts > 1) {
    topk_parts_kernel<<<(unsigned)n_q, SLOT_T, 0, st>>>(P), ::lik::count_launch();
    LIK_CUDA_OK(cudaGetLastError());
  }
  return LIK_OK;
}


// ---------------------------------------------------------------------------------------------
// Top-k of score rows by selection instead of sorting (mode 0 of TopkParams).
//
// One CTA per row.  The row is taken in slabs of SEL_SLAB columns that live in registers (SEL_PER per thread,
// column = slab + j * threads + thread); the k entries kept so far (the running list, or the list the caller
// merges into) are SEL_OLD more elements per thread.  The k-th best key of all of them is
// found by a radix select on the order-preserving 32-bit image of the float (four passes of 256 shared-memory
// counters); entries above it are kept, and of the entries equal to it the ones with the lowest document
// index (a second select, on the index, only when the equal entries do not all fit).  The kept k are sorted
// once per slab that changed anything (best first, ties to the lower index) - a slab with nothing above the
// current k-th best is dismissed after one pass over its values.
// ---------------------------------------------------------------------------------------------
// Two shapes of the CTA, both with slabs of 4096 columns: 256 threads x (16 slab + 4 kept) elements for k <= 1024
// (three CTAs per SM), 1024 threads x (4 slab + 8 kept) elements for k <= LIK_TOPK_MAX = 8192.
constexpr int SEL_SLAB = 4096;
constexpr int SEL_K_SMALL = 1024;

// Monotone map float -> unsigned (larger float, larger key); 0 is below every float.
__device__ __forceinline__ unsigned sel_key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct SelShared {
  int hist[256];
  int digit, want, n_eq, count;
};

// Radix select over the elements every thread holds: key[e] (larger is better) of the elements with on[e], `nbits`
// wide.  Returns the key of rank `want` (1 = the best) to every thread; *need_eq = how many of the elements equal to
// it belong to the best `want`, *n_eq = how many elements equal it.  All threads of the block call it.
template <typename K, int NE>
__device__ K block_select(const K (&key)[NE], const bool (&on)[NE], int nbits, int want, SelShared* sh, int* need_eq, int* n_eq) {
  const int tid = threadIdx.x, lane = tid & 31;
  K prefix = 0;
  for (int shift = nbits - 8; shift >= 0; shift -= 8) {
    if (tid < 256) sh->hist[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      // bits above this digit must match what is fixed already (nothing in the first pass)
      const bool same = shift + 8 >= nbits || (key[e] >> (shift + 8)) == (prefix >> (shift + 8));
      if (on[e] && same) atomicAdd(&sh->hist[(int)((key[e] >> shift) & 255)], 1);
    }
    __syncthreads();
    if (tid < 32) {
      // lane l owns the bins 255 - 8 l ... 248 - 8 l (best first); find the bin in which the running count reaches `want`
      int c[8], s = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        c[i] = sh->hist[255 - 8 * lane - i];
        s += c[i];
      }
      int incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      int above = incl - s;
      if (above < want && want <= incl) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (above < want && want <= above + c[i]) {
            sh->digit = 255 - 8 * lane - i;
            sh->want = want - above;
            sh->n_eq = c[i];
          }
          above += c[i];
        }
      }
    }
    __syncthreads();
    prefix |= (K)sh->digit << shift;
    want = sh->want;
  }
  *need_eq = want;
  *n_eq = sh->n_eq;
  __syncthreads();  // the shared words may be rewritten by the next call
  return prefix;
}

template <int SEL_T, int SEL_PER, int SEL_OLD, int MIN_CTAS>
__global__ void __launch_bounds__(SEL_T, MIN_CTAS) topk_select_kernel(TopkParams P) {
  static_assert(SEL_T * SEL_PER == SEL_SLAB, "a slab is 4096 columns");
  constexpr int SEL_NE = SEL_PER + SEL_OLD;
  extern __shared__ unsigned char raw[];
  long long* top_i = reinterpret_cast<long long*>(raw);
  float* top_k = reinterpret_cast<float*>(top_i + P.KP);
  __shared__ SelShared sh;
  const int tid = threadIdx.x;
  const long long row = blockIdx.x;
  const float sgn = P.largest ? 1.f : -1.f;

  // the kept list: what the caller merges into, or empty
  for (int t = tid; t < P.KP; t += SEL_T) {
    float key = -INFINITY;
    long long id = kPadIdx;
    if (P.merge && t < P.k) {
      const long long o = P.out_index[row * P.k + t];
      if (o >= 0) {
        id = o;
        key = sgn * P.out_scores[row * P.k + t] + 0.f;
      }
    }
    top_k[t] = key;
    top_i[t] = id;
  }
  if (tid == 0) sh.count = 0;
  __syncthreads();
  bool sorted = !P.merge;  // an empty list is in order; a caller's list is taken as it comes
  // k-th best of the kept list as a key (0: the list is not full) - a slab must beat it to matter
  unsigned kth_key = 0;

  const long long n_slabs = (P.n_cols + SEL_SLAB - 1) / SEL_SLAB;
  for (long long sl = 0; sl < (n_slabs > 0 ? n_slabs : 1); ++sl) {
    float f[SEL_NE];
    unsigned u[SEL_NE];
    bool on[SEL_NE];
    int hit = 0;
#pragma unroll
    for (int j = 0; j < SEL_PER; ++j) {
      const long long c = sl * SEL_SLAB + (long long)j * SEL_T + tid;
      on[j] = c < P.n_cols;
      f[j] = on[j] ? sgn * P.scores[row * P.ld + c] + 0.f : -INFINITY;
      u[j] = on[j] ? sel_key(f[j]) : 0u;
      if (on[j] && u[j] >= kth_key) hit = 1;  // (an equal key only matters against a higher kept index; rare, so let it through)
    }
    const bool last = sl + 1 >= n_slabs;
    if (!__syncthreads_or(hit) && !(last && !sorted)) continue;
#pragma unroll
    for (int m = 0; m < SEL_OLD; ++m) {
      const int t = m * SEL_T + tid;
      on[SEL_PER + m] = t < P.k && top_i[t] != kPadIdx;
      f[SEL_PER + m] = on[SEL_PER + m] ? top_k[t] : -INFINITY;
      u[SEL_PER + m] = on[SEL_PER + m] ? sel_key(f[SEL_PER + m]) : 0u;
    }
    // kept entries carry their document index; a slab element's is its column
    long long my_idx[SEL_OLD];
#pragma unroll
    for (int m = 0; m < SEL_OLD; ++m) my_idx[m] = on[SEL_PER + m] ? top_i[m * SEL_T + tid] : kPadIdx;
    // how many real elements there are: with fewer than k, all of them are kept
    int mine = 0;
#pragma unroll
    for (int e = 0; e < SEL_NE; ++e) mine += on[e] ? 1 : 0;
    // block-wide count of the elements
    {
      int w = mine;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
      if ((tid & 31) == 0 && w) atomicAdd(&sh.count, w);
    }
    __syncthreads();
    const int n_all = sh.count;
    __syncthreads();
    if (tid == 0) sh.count = 0;
    const int want = n_all < P.k ? n_all : P.k;
    unsigned T = 0;
    int need_eq = 0, n_eq = 0;
    unsigned long long Ti = 0;  // ties: the kept ones have ~index >= Ti
    bool all_ties = true;
    if (want > 0 && n_all > P.k) {
      T = block_select<unsigned, SEL_NE>(u, on, 32, want, &sh, &need_eq, &n_eq);
      if (need_eq < n_eq) {
        // more entries equal the k-th best than fit: the lowest document indices win
        unsigned long long ik[SEL_NE];
        bool tie[SEL_NE];
#pragma unroll
        for (int e = 0; e < SEL_NE; ++e) {
          tie[e] = on[e] && u[e] == T;
          const long long id = e < SEL_PER ? sl * SEL_SLAB + (long long)e * SEL_T + tid + P.index_offset : my_idx[e - SEL_PER];
          ik[e] = ~(unsigned long long)id;
        }
        int ne2 = 0, nn2 = 0;
        Ti = block_select<unsigned long long, SEL_NE>(ik, tie, 64, need_eq, &sh, &ne2, &nn2);
        all_ties = false;
      }
    }
    __syncthreads();  // everyone has read the kept list; it is rebuilt now
    // gather the kept elements (any order), pad, sort
    int my_pos[SEL_NE];
#pragma unroll
    for (int e = 0; e < SEL_NE; ++e) {
      bool take = on[e] && (n_all <= P.k || u[e] > T);
      if (on[e] && n_all > P.k && u[e] == T) {
        const long long id = e < SEL_PER ? sl * SEL_SLAB + (long long)e * SEL_T + tid + P.index_offset : my_idx[e - SEL_PER];
        take = all_ties || ~(unsigned long long)id >= Ti;
      }
      my_pos[e] = take ? atomicAdd(&sh.count, 1) : -1;
    }
    __syncthreads();
    const int n_kept = sh.count;
    __syncthreads();
    if (tid == 0) sh.count = 0;
#pragma unroll
    for (int e = 0; e < SEL_NE; ++e) {
      if (my_pos[e] >= 0 && my_pos[e] < P.KP) {
        top_k[my_pos[e]] = f[e];
        top_i[my_pos[e]] = e < SEL_PER ? sl * SEL_SLAB + (long long)e * SEL_T + tid + P.index_offset : my_idx[e - SEL_PER];
      }
    }
    for (int t = n_kept + tid; t < P.KP; t += SEL_T) {
      top_k[t] = -INFINITY;
      top_i[t] = kPadIdx;
    }
    __syncthreads();
    bitonic_sort(top_k, top_i, P.KP, tid, SEL_T);
    sorted = true;
    kth_key = (n_kept >= P.k) ? sel_key(top_k[P.k - 1]) : 0u;
  }
  for (int t = tid; t < P.k; t += SEL_T) {
    const bool pad = top_i[t] == kPadIdx;
    P.out_scores[row * P.k + t] = pad ? -sgn * INFINITY : sgn * top_k[t];
    P.out_index[row * P.k + t] = pad ? -1 : top_i[t];
  }
}

static int launch_topk(TopkParams& P, cudaStream_t st) {
  if (P.n_rows <= 0 || P.k <= 0) return LIK_OK;
  int KP = 1;
  while (KP < P.k) KP <<= 1;
  if (KP < 2) KP = 2;
  P.KP = KP;
  if (P.mode == 0) {
    const size_t smem = (size_t)KP * (sizeof(long long) + sizeof(float));
    if (P.k <= SEL_K_SMALL) {
      topk_select_kernel<256, 16, SEL_K_SMALL / 256, 3><<<(unsigned)P.n_rows, 256, smem, st>>>(P), ::lik::count_launch();
    } else {
      static bool raised[64] = {false};  // by device ordinal: the kept list of a large k needs more than 48 KB
      int dev = 0;
      LIK_CUDA_OK(cudaGetDevice(&dev));
      if (dev < 0 || dev >= 64 || !raised[dev]) {
        LIK_CUDA_OK(cudaFuncSetAttribute(topk_select_kernel<1024, 4, LIK_TOPK_MAX / 1024, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((size_t)LIK_TOPK_MAX * (sizeof(long long) + sizeof(float)))));
        if (dev >= 0 && dev < 64) raised[dev] = true;
      }
      topk_select_kernel<1024, 4, LIK_TOPK_MAX / 1024, 1><<<(unsigned)P.n_rows, 1024, smem, st>>>(P), ::lik::count_launch();
    }
    LIK_CUDA_OK(cudaGetLastError());
    return LIK_OK;
  }
  size_t smem = (size_t)KP * 2 * (sizeof(long long) + sizeof(float));
  if (smem > 48 * 1024) {
    static bool raised[64] = {false};
    int dev = 0;
    LIK_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !raised[dev]) {
      LIK_CUDA_OK(cudaFuncSetAttribute(topk_kernel<1024, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)((size_t)LIK_TOPK_MAX * 2 * (sizeof(long long) + sizeof(float)))));
      if (dev >= 0 && dev < 64) raised[dev] = true;
    }
  }
  if (KP > 1024) topk_kernel<1024, 1><<<(unsigned)P.n_rows, 1024, smem, st>>>(P), ::lik::count_launch();
  else topk_kernel<256, 6><<<(unsigned)P.n_rows, 256, smem, st>>>(P), ::lik::count_launch();
  LIK_CUDA_OK(cudaGetLastError());
  return LIK_OK;
}

}  // namespace lik

extern "C" int lik_topk_rows(const float* scores, int64_t n_rows, int64_t n_cols, int64_t ld, int32_t k, int32_t largest,
                             int64_t index_offset, int32_t merge, float* out_scores, int64_t* out_index,
                             lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(k > 0 && k <= LIK_TOPK_MAX, "k=%d outside [1, %d]", k, LIK_TOPK_MAX);
  LIK_REQUIRE(n_rows >= 0 && n_cols >= 0 && ld >= n_cols, "bad score matrix shape");
  LIK_REQUIRE(out_scores && out_index && (scores || n_cols == 0), "NULL pointer");
  TopkParams P{};
  P.mode = 0;
  P.scores = scores;
  P.n_cols = n_cols;
  P.ld = ld;
  P.index_offset = index_offset;
  P.n_rows = n_rows;
  P.k = k;
  P.largest = largest;
  P.merge = merge;
  P.out_scores = out_scores;
  P.out_index = (long long*)out_index;
  return launch_topk(P, (cudaStream_t)stream);
}

extern "C" int lik_topk_merge(const float* cand_scores, const int64_t* cand_index, int32_t n_lists, int64_t n_rows,
                              int32_t k, int32_t largest, float* out_scores, int64_t* out_index, lik_stream_t stream) {
  using namespace lik;
  LIK_REQUIRE(k > 0 && k <= LIK_TOPK_MAX, "k=%d outside [1, %d]", k, LIK_TOPK_MAX);
  LIK_REQUIRE(n_lists >= 0 && n_rows >= 0, "negative size");
  LIK_REQUIRE(out_scores && out_index && ((cand_scores && cand_index) || n_lists == 0), "NULL pointer");
  TopkParams P{};
  P.mode = 1;
  P.cand_scores = cand_scores;
  P.cand_index = (const long long*)cand_index;
  P.n_lists = n_lists;
  P.n_rows = n_rows;
  P.k = k;
  P.largest = largest;
  P.merge = 0;
  P.out_scores = out_scores;
  P.out_index = (long long*)out_index;
  return launch_topk(P, (cudaStream_t)stream);
}
