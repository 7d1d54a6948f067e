// Result rows: the pair list sorted by (i, j), and the CSR neighbour table.
//
// Reference counterpart: the pairs of each batch are sorted by thrust
// sort_by_key and copied into per-point ranges on the host
// (src/launcher.cu:3468-3488, constructNeighborTable, src/launcher.cu:4-50).
//
// Both results are the accepted pairs grouped by row with ascending ids
// inside each row, so they are built row by row rather than by sorting whole
// packed pairs: count the entries of every row (the atomic's return value is
// the entry's rank in arrival order), scan the counts, put every id at its
// row's offset + rank, and sort each row on its own.  That moves each pair
// about four times; the 8-bit radix sort of the packed pairs it replaces
// moved it three times per digit over 5 to 8 digits, most of them needed only
// to tell rows apart.  Sorted lists, before and after: 1.53e8 pairs of 5M rows
// 17.6 -> 4.6 ms, 1.7e7 pairs of 2M rows 1.90 -> 0.46 ms; the table of 1.6e5
// pairs of 20,011 rows 0.26 -> 0.10 ms.
//
// Bounds: the counting and placing passes by one atomic and one scattered
// 4-byte access an entry, the row sort by HBM.
#include <type_traits>

#include "internal.cuh"

namespace mistic {
namespace {

constexpr int RW_THREADS = 256;
constexpr int RW_ITEMS = 4;                  // pairs a thread has in flight
constexpr uint32_t ROW_REG_MAX = 256;        // rows sorted in a warp's registers
constexpr uint32_t ROW_BLOCK_MAX = 8192;     // rows sorted in a block's registers
constexpr int RL_THREADS = 256;              // block of the long-row kernel
constexpr int RL_BINS = 256;
constexpr int RL_ITEMS = 8;                  // entries a thread ranks between barriers of its radix sort

// BOTH: an entry in either row of the pair (the neighbour table); else one in
// row i (the pair list).
template <bool BOTH>
__global__ void __launch_bounds__(RW_THREADS)
k_row_count(const unsigned long long* __restrict__ pairs, size_t np, uint32_t* __restrict__ cnt,
            uint32_t* __restrict__ rank) {
  const size_t base = (size_t)blockIdx.x * (RW_THREADS * RW_ITEMS) + threadIdx.x;
  uint32_t r[RW_ITEMS], s[RW_ITEMS];
#pragma unroll
  for (int k = 0; k < RW_ITEMS; ++k) {
    const size_t t = base + (size_t)k * RW_THREADS;
    if (t < np) {
      const unsigned long long v = pairs[t];
      r[k] = atomicAdd(&cnt[v >> 32], 1u);
      if (BOTH) s[k] = atomicAdd(&cnt[(uint32_t)v], 1u);
    }
  }
#pragma unroll
  for (int k = 0; k < RW_ITEMS; ++k) {
    const size_t t = base + (size_t)k * RW_THREADS;
    if (t < np) {
      rank[t] = r[k];
      if (BOTH) rank[np + t] = s[k];
    }
  }
}

// off: exclusive scan of the counts.  In the neighbour table every row also
// holds its own id, in front, so row i starts at off[i] + i.
template <bool BOTH>
__global__ void __launch_bounds__(RW_THREADS)
k_row_place(const unsigned long long* __restrict__ pairs, size_t np, size_t n, const uint32_t* __restrict__ off,
            const uint32_t* __restrict__ rank, uint32_t* __restrict__ ids) {
  const size_t base = (size_t)blockIdx.x * (RW_THREADS * RW_ITEMS) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < RW_ITEMS; ++k) {
    const size_t t = base + (size_t)k * RW_THREADS;
    if (t < np) {
      const unsigned long long v = pairs[t];
      const uint32_t i = (uint32_t)(v >> 32), j = (uint32_t)v;
      if (BOTH) {
        ids[(size_t)off[i] + i + 1 + rank[t]] = j;
        ids[(size_t)off[j] + j + 1 + rank[np + t]] = i;
      } else {
        ids[(size_t)off[i] + rank[t]] = j;
      }
    } else if (BOTH && t < np + n) {
      const uint32_t p = (uint32_t)(t - np);
      ids[(size_t)off[p] + p] = p;
    }
  }
}

struct RowOut {
  const uint32_t* off;         // n + 1
  size_t n;
  uint32_t* ids;               // entries, row by row, unsorted
  uint32_t* rank;              // their ranks, no longer needed: scratch, row i's from off[i] on
  int csr;                     // rows hold their own id too (start at off[i] + i)
  unsigned long long* pairs;   // pair list: entry e as (i, j) in memory order
  uint32_t* nbrs;              // neighbour table: ids
  unsigned long long* offs;    // neighbour table: n + 1 row offsets
  const uint32_t* row0;        // fused batch: first global row of each instance (ids become local), else null
  uint32_t n_inst;
  uint32_t* long_rows;         // rows above ROW_REG_MAX entries
  uint32_t* long_n;            // their number, and the claim cursor of the kernel that sorts them
  uint32_t rpw;                // rows a warp of k_row_sort (at most 32)
};

__device__ __forceinline__ size_t row_begin(const RowOut& R, size_t i) {
  return (size_t)R.off[i] + (R.csr ? i : 0);
}

// First global row of row i's instance (0 outside fused batches).
__device__ __forceinline__ uint32_t row_base(const RowOut& R, uint32_t i) {
  if (!R.row0) return 0u;
  uint32_t lo = 0, hi = R.n_inst - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (R.row0[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return R.row0[lo];
}

__device__ __forceinline__ void put(const RowOut& R, size_t e, uint32_t i, uint32_t j, uint32_t r0) {
  if (R.csr)
    R.nbrs[e] = j;
  else
    R.pairs[e] = ((unsigned long long)(j - r0) << 32) | (i - r0);
}

// The steps j = j0, j0 / 2 .. 1 of a bitonic merge of length k inside a warp;
// value idx = base + 32 e + lane is in v[e], base a multiple of 32 E.
template <int E>
__device__ __forceinline__ void warp_merge(uint32_t (&v)[E], uint32_t base, int k, int j0) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 16 * E; j > 0; j >>= 1) {
    if (j > j0) continue;
    if (j >= 32) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int f = e ^ (j >> 5);
        if (f > e) {
          const bool up = ((base + 32 * e) & k) == 0;  // k > j >= 32: the lane has no say in the direction
          const uint32_t a = min(v[e], v[f]), b = max(v[e], v[f]);
          v[e] = up ? a : b;
          v[f] = up ? b : a;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const uint32_t o = __shfl_xor_sync(FULL_MASK, v[e], j);
        const bool up = ((base + 32 * e + lane) & k) == 0, low = (lane & j) == 0;
        v[e] = (up == low) ? min(v[e], o) : max(v[e], o);
      }
    }
  }
}

// Bitonic sort of the warp's 32 E values: ascending, or (base & 32 E) descending.
template <int E>
__device__ __forceinline__ void warp_sort(uint32_t (&v)[E], uint32_t base = 0) {
#pragma unroll
  for (int k = 2; k <= 32 * E; k <<= 1) warp_merge<E>(v, base, k, k >> 1);
}

// Ascending sort of a block's 32 E RL_THREADS / 32 values, warp w's from 32 E w
// on: only the steps between warps go through shared memory (sv), 6 of the 45
// to 91.
template <int E>
__device__ __forceinline__ void block_sort(uint32_t (&v)[E], uint32_t* sv) {
  const uint32_t lane = threadIdx.x & 31, base = (threadIdx.x >> 5) * 32 * E;
  warp_sort<E>(v, base);
#pragma unroll 1
  for (uint32_t k = 64 * E; k <= RL_THREADS * E; k <<= 1) {
#pragma unroll 1
    for (uint32_t j = k >> 1; j >= 32 * E; j >>= 1) {
      __syncthreads();
#pragma unroll
      for (int e = 0; e < E; ++e) sv[base + 32 * e + lane] = v[e];
      __syncthreads();
      const bool keep_min = ((base & k) == 0) == ((base & j) == 0);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const uint32_t o = sv[(base + 32 * e + lane) ^ j];
        v[e] = keep_min ? min(v[e], o) : max(v[e], o);
      }
    }
    warp_merge<E>(v, base, (int)k, 16 * E);
  }
}

template <int E>
__device__ __forceinline__ void sort_one_row(const RowOut& R, size_t b, uint32_t len, uint32_t i) {
  const int lane = threadIdx.x & 31;
  uint32_t v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = 32u * e + lane < len ? R.ids[b + 32 * e + lane] : 0xffffffffu;
  warp_sort<E>(v);
  const uint32_t r0 = row_base(R, i);
#pragma unroll
  for (int e = 0; e < E; ++e)
    if (32u * e + lane < len) put(R, b + 32 * e + lane, i, v[e], r0);
}

// A warp per R.rpw consecutive rows.  Runs of rows with at most 32 entries
// together are sorted at once, one entry a lane: an entry's place in its row
// is the number of smaller ids there (rows of a planar join hold about 8
// entries; a row at a time would leave most lanes idle).  A longer row takes
// the whole warp, one above ROW_REG_MAX entries is left to k_row_sort_long.
__global__ void __launch_bounds__(RW_THREADS) k_row_sort(const RowOut R) {
  const int lane = threadIdx.x & 31;
  const size_t i0 = ((size_t)blockIdx.x * (RW_THREADS / 32) + (threadIdx.x >> 5)) * R.rpw;
  if (i0 >= R.n) return;  // warp-uniform
  const uint32_t rows = (uint32_t)min((size_t)R.rpw, R.n - i0);
  // lane l: begin of row i0 + l and of the row after it
  const size_t beg = (uint32_t)lane < rows ? row_begin(R, i0 + lane) : 0;
  const size_t nxt = (uint32_t)lane < rows ? row_begin(R, i0 + lane + 1) : 0;
  const size_t base = __shfl_sync(FULL_MASK, beg, 0);
  const uint32_t b = (uint32_t)(beg - base), e = (uint32_t)(nxt - base);  // relative to the warp's first entry
  if (R.csr && (uint32_t)lane < rows) {
    R.offs[i0 + lane] = beg;
    if (i0 + lane + 1 == R.n) R.offs[R.n] = nxt;
  }
  for (uint32_t r = 0; r < rows;) {
    const uint32_t rb = __shfl_sync(FULL_MASK, b, r), re = __shfl_sync(FULL_MASK, e, r);
    // rows r .. r + nr - 1 end within 32 entries of row r's begin (ends ascend)
    const uint32_t fit = __ballot_sync(FULL_MASK, (uint32_t)lane >= r && (uint32_t)lane < rows && e - rb <= 32u);
    const uint32_t nr = __popc(fit);
    if (nr == 0) {
      const uint32_t len = re - rb, i = (uint32_t)(i0 + r);
      if (len <= 64)
        sort_one_row<2>(R, base + rb, len, i);
      else if (len <= 128)
        sort_one_row<4>(R, base + rb, len, i);
      else if (len <= ROW_REG_MAX)
        sort_one_row<8>(R, base + rb, len, i);
      else if (lane == 0)
        R.long_rows[atomicAdd(R.long_n, 1u)] = i;
      ++r;
      continue;
    }
    const uint32_t tot = __shfl_sync(FULL_MASK, e, r + nr - 1) - rb;
    if (tot > 0) {
      // lane's row: the begins of rows r + 1 .. that lie at or before this entry
      const uint32_t rel = b - rb;  // begin of row `lane`, meaningful for the rows of the run
      const bool bound = (uint32_t)lane > r && (uint32_t)lane < r + nr && rel < 32u;
      const uint32_t starts = __reduce_or_sync(FULL_MASK, bound ? 1u << rel : 0u);
      // empty rows share a begin with the row after them: count rows, not bits
      uint32_t row = r;
      for (uint32_t q = r + 1; q < r + nr; ++q) row += __shfl_sync(FULL_MASK, rel, q) <= (uint32_t)lane ? 1u : 0u;
      const uint32_t upto = starts & (lane == 31 ? FULL_MASK : ((2u << lane) - 1u));
      const uint32_t sb = upto ? 31 - __clz(upto) : 0u;  // first entry of this entry's row
      const uint32_t above = lane == 31 ? 0u : starts & (FULL_MASK << (lane + 1));
      const uint32_t se = above ? __ffs(above) - 1 : tot;
      const bool ok = (uint32_t)lane < tot;
      const uint32_t v = ok ? R.ids[base + rb + lane] : 0u;
      const uint32_t len = ok ? se - sb : 0u;
      const uint32_t most = __reduce_max_sync(FULL_MASK, len);
      uint32_t k = 0;
      for (uint32_t t = 0; t < most; ++t) {
        const uint32_t o = __shfl_sync(FULL_MASK, v, min(sb + t, 31u));
        k += t < len && o < v ? 1u : 0u;
      }
      if (ok) {
        const uint32_t i = (uint32_t)(i0 + row);
        put(R, base + rb + sb + k, i, v, row_base(R, i));
      }
    }
    r += nr;
  }
}

// A row whose ids, all different, fill a bitmap of n bits: the bits are set,
// then written out in order behind a running count.
__device__ __forceinline__ void sort_by_bitmap(const RowOut& R, size_t b, uint32_t len, uint32_t i, uint32_t r0,
                                            uint32_t* ws) {
  const uint32_t words = (uint32_t)((R.n + 31) / 32);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t* bm = R.rank + R.off[i];
  for (uint32_t t = tid; t < words; t += RL_THREADS) bm[t] = 0u;
  __syncthreads();
#pragma unroll 8
  for (uint32_t t = tid; t < len; t += RL_THREADS) {
    const uint32_t v = R.ids[b + t];
    atomicOr(&bm[v >> 5], 1u << (v & 31));
  }
  __syncthreads();
  uint32_t base = 0;  // entries written before this step's words
  for (uint32_t t0 = 0; t0 < words; t0 += RL_THREADS) {
    uint32_t m = t0 + tid < words ? __ldcg(&bm[t0 + tid]) : 0u;
    uint32_t incl = __popc(m);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t pos = base + incl - __popc(m), total = 0;
    for (int q = 0; q < RL_THREADS / 32; ++q) {
      pos += q < w ? ws[q] : 0u;
      total += ws[q];
    }
    for (; m; m &= m - 1) put(R, b + pos++, i, 32u * (t0 + tid) + __ffs(m) - 1, r0);
    base += total;
    __syncthreads();
  }
}

// Rows above ROW_REG_MAX entries, a block a row, claimed from the list.  Up
// to ROW_BLOCK_MAX entries are sorted in the block's registers (in shared
// memory, a barrier a step, these rows took 2.0 ms of a 5M x 18 join's sorted
// list; now 1.0).  Longer rows: by a bitmap of the n ids in the place of the
// row's ranks where that is large enough (n / 32 entries); shorter ones by a
// stable 8-bit radix sort through global memory, between the unsorted ids and
// the row's own place in the output (which is at least as large).
// One block sorts a row however long, so a lone row of nearly n entries (a point
// amid all others) ends the pass: of 50,000, 200,000 and 1M rows (90 columns,
// joins of 0.4, 5.8 and 143 ms) 0.16, 0.58 and 2.4 ms for the whole sorted list;
// 0.69, 2.7 and 13.6 by a radix sort that ranked an entry a thread.  Where all
// rows are long: 40,000 near duplicates, 8e8 pairs, 37 -> 17.5 ms.
__global__ void __launch_bounds__(RL_THREADS, 4) k_row_sort_long(const RowOut R) {
  extern __shared__ uint32_t sv[];  // ROW_BLOCK_MAX
  __shared__ uint32_t s_claim, wcnt[RL_THREADS / 32][RL_BINS], ws[RL_THREADS / 32], gbase[RL_BINS];
  const uint32_t total = R.long_n[0];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_claim = atomicAdd(R.long_n + 1, 1u);
    __syncthreads();
    if (s_claim >= total) return;
    const uint32_t i = R.long_rows[s_claim], r0 = row_base(R, i);
    const size_t b = row_begin(R, i);
    const uint32_t len = (uint32_t)(row_begin(R, (size_t)i + 1) - b);
    if (len <= ROW_BLOCK_MAX) {
      auto row = [&](auto e_) {
        constexpr int E = decltype(e_)::value;
        uint32_t v[E];
        const uint32_t t0 = w * 32 * E + lane;
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = t0 + 32 * e < len ? R.ids[b + t0 + 32 * e] : 0xffffffffu;
        block_sort<E>(v, sv);
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (t0 + 32 * e < len) put(R, b + t0 + 32 * e, i, v[e], r0);
      };
      if (len <= 2 * RL_THREADS)
        row(std::integral_constant<int, 2>());
      else if (len <= 4 * RL_THREADS)
        row(std::integral_constant<int, 4>());
      else if (len <= 8 * RL_THREADS)
        row(std::integral_constant<int, 8>());
      else if (len <= 16 * RL_THREADS)
        row(std::integral_constant<int, 16>());
      else
        row(std::integral_constant<int, 32>());
      continue;
    }
    if (R.off[i + 1] - R.off[i] >= (R.n + 31) / 32) {
      sort_by_bitmap(R, b, len, i, r0, ws);
      continue;
    }
    uint32_t* src = R.ids + b;
    uint32_t* dst = R.csr ? R.nbrs + b : reinterpret_cast<uint32_t*>(R.pairs + b);
    for (int shift = 0; shift < 32; shift += 8) {
      // digit counts of the row, and their exclusive scan
      gbase[tid] = 0;
      __syncthreads();
      for (uint32_t t = tid; t < len; t += RL_THREADS) atomicAdd(&gbase[(src[t] >> shift) & 255u], 1u);
      __syncthreads();
      uint32_t c = gbase[tid], x = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) ws[w] = x;
      __syncthreads();
      uint32_t pre = 0;
      for (int q = 0; q < w; ++q) pre += ws[q];
      gbase[tid] = pre + x - c;
      // tiles of RL_THREADS x RL_ITEMS entries in order, each warp a run of
      // them: rank among equal digits before it in the warp's run, in the warps
      // before it, then in the tiles before it
      for (uint32_t t0 = 0; t0 < len; t0 += RL_THREADS * RL_ITEMS) {
        for (int q = 0; q < RL_THREADS / 32; ++q) wcnt[q][tid] = 0;
        __syncthreads();
        const uint32_t tw = t0 + w * 32 * RL_ITEMS + lane;
        uint32_t v[RL_ITEMS], rk[RL_ITEMS];
#pragma unroll
        for (int r = 0; r < RL_ITEMS; ++r) v[r] = tw + 32 * r < len ? src[tw + 32 * r] : 0u;
#pragma unroll
        for (int r = 0; r < RL_ITEMS; ++r) {
          const bool ok = tw + 32 * r < len;
          const uint32_t dg = ok ? (v[r] >> shift) & 255u : RL_BINS + lane;
          const uint32_t peers = __match_any_sync(FULL_MASK, dg);
          const uint32_t lt = __popc(peers & ((1u << lane) - 1u));
          const uint32_t before = ok ? wcnt[w][dg] : 0u;
          __syncwarp();
          if (ok && lt == 0) wcnt[w][dg] = before + __popc(peers);
          __syncwarp();
          rk[r] = before + lt;
        }
        __syncthreads();
        uint32_t run = gbase[tid];
        for (int q = 0; q < RL_THREADS / 32; ++q) {
          const uint32_t c = wcnt[q][tid];
          wcnt[q][tid] = run;
          run += c;
        }
        gbase[tid] = run;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RL_ITEMS; ++r)
          if (tw + 32 * r < len) dst[wcnt[w][(v[r] >> shift) & 255u] + rk[r]] = v[r];
        __syncthreads();
      }
      uint32_t* sw = src;
      src = dst;
      dst = sw;
      __syncthreads();  // the block's global stores are visible to its next pass
    }
    // four passes: the sorted ids are back in R.ids
    for (uint32_t t = tid; t < len; t += RL_THREADS) put(R, b + t, i, src[t], r0);
  }
}

}  // namespace

namespace {
struct RowScratch {
  uint32_t *off, *rank, *ids, *lrows;
  size_t max_long;  // at most this many rows can hold more than ROW_REG_MAX entries
};

RowScratch row_scratch(mistic_handle_s* h, size_t np, size_t n, bool both) {
  // 32-bit offsets and ranks
  if (np > 0xffffffffull) throw Error(MISTIC_ERR_TOO_LARGE, "sorting supports < 2^32 pairs");
  const size_t dir = (both ? 2 : 1) * np, entries = dir + (both ? n : 0);
  RowScratch s;
  s.max_long = entries / ROW_REG_MAX + 1;
  s.off = (uint32_t*)h->arena.get("row_off", (n + 1) * sizeof(uint32_t));
  s.rank = (uint32_t*)h->arena.get("row_rank", dir * sizeof(uint32_t));
  s.ids = (uint32_t*)h->arena.get("row_ids", entries * sizeof(uint32_t));
  s.lrows = (uint32_t*)h->arena.get("row_long", (s.max_long + 2) * sizeof(uint32_t));
  return s;
}
}  // namespace

void reserve_row_sort(mistic_handle_s* h, size_t np, size_t n, bool csr) { row_scratch(h, np, n, csr); }

static void sort_rows(mistic_handle_s* h, const unsigned long long* in, size_t np, size_t n, RowOut R) {
  const bool both = R.csr != 0;
  const RowScratch sc = row_scratch(h, np, n, both);
  uint32_t *off = sc.off, *rank = sc.rank, *ids = sc.ids, *lrows = sc.lrows;
  const size_t max_long = sc.max_long;
  MCK(cudaMemsetAsync(off, 0, (n + 1) * sizeof(uint32_t), h->stream));
  MCK(cudaMemsetAsync(lrows, 0, 2 * sizeof(uint32_t), h->stream));
  const size_t tile = RW_THREADS * RW_ITEMS;
  if (np) {
    const unsigned nb = (unsigned)((np + tile - 1) / tile);
    if (both)
      k_row_count<true><<<nb, RW_THREADS, 0, h->stream>>>(in, np, off, rank);
    else
      k_row_count<false><<<nb, RW_THREADS, 0, h->stream>>>(in, np, off, rank);
    launched(h, "row_count");
  }
  exclusive_scan<uint32_t>(h, off, off, n + 1, nullptr);
  const size_t items = np + (both ? n : 0);
  const unsigned nb = (unsigned)((items + tile - 1) / tile);
  if (both)
    k_row_place<true><<<nb, RW_THREADS, 0, h->stream>>>(in, np, n, off, rank, ids);
  else
    k_row_place<false><<<nb, RW_THREADS, 0, h->stream>>>(in, np, n, off, rank, ids);
  launched(h, "row_place");
  R.off = off;
  R.n = n;
  R.ids = ids;
  R.rank = rank;
  R.long_n = lrows;
  R.long_rows = lrows + 2;
  // 32 rows a warp, fewer while that leaves the SMs without 16 warps each
  // (4,000 rows of 16: the whole sort 83 -> 50 us)
  R.rpw = 32;
  while (R.rpw > 4 && n < (size_t)h->sms * 16 * R.rpw) R.rpw /= 2;
  const size_t per_block = (size_t)R.rpw * (RW_THREADS / 32);
  k_row_sort<<<(unsigned)((n + per_block - 1) / per_block), RW_THREADS, 0, h->stream>>>(R);
  launched(h, "row_sort");
  k_row_sort_long<<<(unsigned)std::min<size_t>((size_t)h->sms * 4, max_long), RL_THREADS,
                    ROW_BLOCK_MAX * sizeof(uint32_t), h->stream>>>(R);
  launched(h, "row_sort_long");
}

void sort_pairs_ij(mistic_handle_s* h, const unsigned long long* pairs, unsigned long long* out, size_t np, size_t n,
                   const uint32_t* row0, uint32_t n_inst) {
  if (np == 0) return;
  RowOut R{};
  R.pairs = out;
  R.row0 = row0;
  R.n_inst = n_inst;
  sort_rows(h, pairs, np, n, R);
}

void neighbour_table(mistic_handle_s* h, const unsigned long long* pairs, size_t np, size_t n, uint32_t* nbrs,
                     unsigned long long* offs) {
  RowOut R{};
  R.csr = 1;
  R.nbrs = nbrs;
  R.offs = offs;
  sort_rows(h, pairs, np, n, R);
}

}  // namespace mistic
