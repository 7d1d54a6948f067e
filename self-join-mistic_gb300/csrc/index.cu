// Reference-point bin index and neighbour-bin enumeration on the device.
//
// Reference counterparts (bwd29/self-join-MiSTIC):
//  - binningKernel, src/kernel.cu:880-909: per point, floor(||x - r|| / ε)
//    for each reference point in FP64.  Here the same FP64 distances are
//    taken to k reference points and quantised with a width slightly above ε
//    so the triangle-inequality argument survives rounding (see k_pack_keys).
//  - the host-built node net, src/nodes.cu:5-356, whose neighbour relation is
//    "bins differ by at most one on every layer" (src/nodes.cu:416-435,
//    719-747).  Here the bin keys are packed into one 64-bit key, radix
//    sorted, and non-empty bins become contiguous runs of the sorted order.
//  - the 3^k neighbour search over sorted bin keys, generateRanges /
//    binarySearch in src/tree.cu:596-759,886-996 (device form
//    GPUBinarySearch, src/kernel.cu:164-224).  Here a warp per non-empty bin
//    compares the keys that can be near where bins are few; where they are
//    many, up to 8 threads a bin walk the ±1 neighbourhood depth-first,
//    narrowing a sorted range one key field at a time (the top fields through
//    a direct-address prefix table), so empty prefixes are pruned early.  Only
//    neighbours of index >= the home bin are emitted (each unordered bin pair
//    once).
#include <math.h>

#include "internal.cuh"

namespace mistic {

template <class T>
__device__ __forceinline__ double ld(const T* p, size_t i) {
  return (double)p[i];
}

// ------------------------------------------------------------ column stats
// Per-column min, max and sum over all rows plus a finiteness flag.  Each
// block writes its partials; a second kernel folds them in a fixed order so
// the result (and therefore the reference points) is deterministic.
//
// A block reads its rows as one stream, RG = 256 / cols rows at a time, thread
// t always at column t % cols, so that narrow rows fill the warps too (lanes
// tied to 32 columns left 30 of 32 idle at d = 2); rows above 256 columns are
// cut into column tiles.  FP64 values are compared as order-preserving
// integers: FP64 compares run on the FP64 pipe, whose rate is 1/75 of FP32's,
// and with the sum they bound the pass before HBM did.  The whole phase (this,
// the sample covariance, the reference points): 2M x 2 FP32 0.94 -> 0.15 ms;
// 5M x 18 FP64 1.81 -> 0.56 ms (the rows alone 0.11 ms at HBM's rate).

constexpr int CS_THREADS = 256;

template <class T>
struct ColMinMax;
template <>
struct ColMinMax<float> {
  float mn = INFINITY, mx = -INFINITY;
  __device__ void add(float v) {  // NaN leaves both unchanged
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  __device__ double lo() const { return mn; }
  __device__ double hi() const { return mx; }
};
template <>
struct ColMinMax<double> {
  // bits of a double, the magnitude bits of negative ones flipped: signed
  // integer order is then the order of the values
  static constexpr long long kInf = 0x7ff0000000000000ll;
  long long mn, mx;
  static __device__ long long key(double v) {
    const long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
  }
  static __device__ double val(long long k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll)); }
  __device__ ColMinMax() : mn(key(INFINITY)), mx(key(-INFINITY)) {}
  __device__ void add(double v) {  // NaN leaves both unchanged
    const long long k = key(v);
    const bool num = (__double_as_longlong(v) & 0x7fffffffffffffffll) <= kInf;
    if (num && k < mn) mn = k;
    if (num && k > mx) mx = k;
  }
  __device__ double lo() const { return val(mn); }
  __device__ double hi() const { return val(mx); }
};

__device__ __forceinline__ bool finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite_bits(double v) {
  return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
}

template <class T>
__global__ void __launch_bounds__(CS_THREADS)
k_colstats(const T* __restrict__ x, size_t n, uint32_t d, double* __restrict__ part, unsigned* __restrict__ nonfinite) {
  // part layout: [blockIdx.y][3][d] : min, max, sum of the block's rows, column tile blockIdx.x
  __shared__ double red[3][CS_THREADS];
  const uint32_t c0 = blockIdx.x * CS_THREADS, cols = min((uint32_t)CS_THREADS, d - c0);
  const uint32_t rg = CS_THREADS / cols;                       // rows side by side
  const uint32_t r = threadIdx.x / cols, c = threadIdx.x % cols;
  ColMinMax<T> mm;
  double sm[4] = {0, 0, 0, 0};
  bool bad = false;
  if (r < rg) {
    const size_t step = (size_t)gridDim.y * rg, stride = step * d;
    size_t row = (size_t)blockIdx.y * rg + r;
    const T* p = x + row * d + c0 + c;
    for (; row + 3 * step < n; row += 4 * step, p += 4 * stride) {
      T v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = p[k * stride];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        bad |= !finite_bits(v[k]);
        mm.add(v[k]);
        sm[k] += (double)v[k];
      }
    }
    for (; row < n; row += step, p += stride) {
      const T v = *p;
      bad |= !finite_bits(v);
      mm.add(v);
      sm[0] += (double)v;
    }
  }
  if (bad) atomicOr(nonfinite, 1u);
  red[0][threadIdx.x] = mm.lo();
  red[1][threadIdx.x] = mm.hi();
  red[2][threadIdx.x] = (sm[0] + sm[1]) + (sm[2] + sm[3]);
  __syncthreads();
  if (threadIdx.x < cols) {
    double mn = red[0][c], mx = red[1][c], s = red[2][c];
    for (uint32_t q = 1; q < rg; ++q) {
      mn = fmin(mn, red[0][q * cols + c]);
      mx = fmax(mx, red[1][q * cols + c]);
      s += red[2][q * cols + c];
    }
    double* o = part + (size_t)blockIdx.y * 3 * d + c0 + c;
    o[0] = mn;
    o[d] = mx;
    o[2 * (size_t)d] = s;
  }
}

// A warp per column over the blocks' partials.
__global__ void k_colstats_final(const double* __restrict__ part, uint32_t nparts, uint32_t d,
                                 size_t n, double* __restrict__ out /* mean, min, max */) {
  const uint32_t col = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (col >= d) return;
  double mn = INFINITY, mx = -INFINITY, sm = 0.0;
  for (uint32_t b = lane; b < nparts; b += 32) {
    const double* p = part + (size_t)b * 3 * d + col;
    mn = fmin(mn, p[0]);
    mx = fmax(mx, p[d]);
    sm += p[2 * (size_t)d];
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
    sm += __shfl_xor_sync(FULL_MASK, sm, o);
  }
  if (lane == 0) {
    out[col] = n ? sm / (double)n : 0.0;
    out[d + col] = mn;
    out[2 * (size_t)d + col] = mx;
  }
}

// ------------------------------------------------------------ sample covariance
template <class T>
__global__ void k_gather_sample(const T* __restrict__ x, size_t n, uint32_t d, uint32_t S,
                                double* __restrict__ s) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)S * d) return;
  const size_t row = i / d, col = i % d;
  const size_t src = (size_t)((row * (unsigned long long)n) / S);
  s[i] = ld(x, src * d + col);
}

// Sample covariance about the full-data mean mu: each block accumulates a
// 16 x 16 tile of (a, b) over one chunk of sample rows (staged in shared
// memory); a second kernel adds the chunk partials in a fixed order, so the
// result - and the reference points derived from it - is deterministic.
constexpr int COV_T = 16;
// Rows a chunk: 128, or 32 for rows of at most 32 columns, whose few tiles
// would leave most SMs idle.
constexpr uint32_t cov_chunk(uint32_t d) { return d <= 32 ? 32u : 128u; }

template <int COV_CHUNK>
__global__ void k_sample_cov_part(const double* __restrict__ s, uint32_t S, uint32_t d, const double* __restrict__ mu,
                                  double* __restrict__ part /* [chunks][d][d] */) {
  __shared__ double sa[COV_CHUNK][COV_T + 1], sb[COV_CHUNK][COV_T + 1];
  const uint32_t a0 = blockIdx.y * COV_T, b0 = blockIdx.x * COV_T, r0 = blockIdx.z * COV_CHUNK;
  const int tx = threadIdx.x, ty = threadIdx.y, t = ty * COV_T + tx;
  for (int i = t; i < COV_CHUNK * COV_T; i += COV_T * COV_T) {
    const int rr = i / COV_T, cc = i % COV_T;
    const uint32_t row = r0 + rr;
    double va = 0.0, vb = 0.0;
    if (row < S && a0 + cc < d) va = s[(size_t)row * d + a0 + cc] - mu[a0 + cc];
    if (row < S && b0 + cc < d) vb = s[(size_t)row * d + b0 + cc] - mu[b0 + cc];
    sa[rr][cc] = va;
    sb[rr][cc] = vb;
  }
  __syncthreads();
  double acc = 0.0;
  for (int rr = 0; rr < COV_CHUNK; ++rr) acc = fma(sa[rr][ty], sb[rr][tx], acc);
  const uint32_t a = a0 + ty, b = b0 + tx;
  if (a < d && b < d) part[((size_t)blockIdx.z * d + a) * d + b] = acc;
}

__global__ void k_sample_cov_final(const double* __restrict__ part, uint32_t chunks, uint32_t d, uint32_t S,
                                   double* __restrict__ cov) {
  // four lanes an element, each every fourth chunk
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 4;
  const uint32_t l = threadIdx.x & 3u;
  double acc = 0.0;
  if (i < (size_t)d * d)
    for (uint32_t c = l; c < chunks; c += 4) acc += part[(size_t)c * d * d + i];
  acc += __shfl_xor_sync(FULL_MASK, acc, 1);
  acc += __shfl_xor_sync(FULL_MASK, acc, 2);
  if (i < (size_t)d * d && l == 0) cov[i] = acc / S;
}

// ------------------------------------------------------------ reference-point distances
// D[i][j] = FP64 ||x_i - r_j|| (sequential sum, then sqrt), with per-block
// min/max partials per reference point.  Bound by the FP64 pipe (2 k d
// operations a row).  A block's rows pass through shared memory RPD_COLS
// columns at a time, each value read once for all k sums, so rows of any
// length load coalesced: a thread reading its own row of 384 FP32 values took
// 17.5 ms for 1M rows at k = 8, now 12.1 ms; 515k x 90 4.0 -> 1.7 ms.
constexpr int RPD_COLS = 32;

template <class T, int K, int RPD_THREADS>
__global__ void __launch_bounds__(RPD_THREADS)
k_rp_dist(const T* __restrict__ x, size_t n, uint32_t d, const double* __restrict__ rps, int k,
          double* __restrict__ D, double* __restrict__ part /* [block][2][k] */) {
  extern __shared__ double tile[];  // RPD_THREADS rows x (RPD_COLS + 1), then K x RPD_COLS reference values
  double* srp = tile + RPD_THREADS * (RPD_COLS + 1);
  __shared__ double smn[MAX_K][RPD_THREADS / 32], smx[MAX_K][RPD_THREADS / 32];
  const size_t row0 = (size_t)blockIdx.x * RPD_THREADS;
  const uint32_t rows = (uint32_t)min((size_t)RPD_THREADS, n - row0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double s[K];
#pragma unroll
  for (int j = 0; j < K; ++j) s[j] = 0.0;
  for (uint32_t t0 = 0; t0 < d; t0 += RPD_COLS) {
    const uint32_t nc = min((uint32_t)RPD_COLS, d - t0);
    __syncthreads();
    if (nc == d) {  // whole rows: one contiguous run
      for (uint32_t e = threadIdx.x; e < rows * d; e += RPD_THREADS)
        tile[(e / d) * (RPD_COLS + 1) + e % d] = (double)x[row0 * d + e];
    } else if ((uint32_t)lane < nc) {
      for (uint32_t r = w; r < rows; r += RPD_THREADS / 32)
        tile[r * (RPD_COLS + 1) + lane] = (double)x[(row0 + r) * d + t0 + lane];
    }
    for (uint32_t e = threadIdx.x; e < K * RPD_COLS; e += RPD_THREADS) {
      const uint32_t j = e / RPD_COLS, t = e % RPD_COLS;
      srp[e] = j < (uint32_t)k && t < nc ? rps[(size_t)j * d + t0 + t] : 0.0;
    }
    __syncthreads();
    const double* xr = tile + threadIdx.x * (RPD_COLS + 1);
    for (uint32_t t = 0; t < nc; ++t) {
      const double xv = xr[t];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (j >= k) break;
        const double df = xv - srp[j * RPD_COLS + t];
        s[j] = fma(df, df, s[j]);
      }
    }
  }
  const size_t i = row0 + threadIdx.x;
  const bool valid = i < n;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (j >= k) break;
    const double dist = sqrt(s[j]);
    if (valid) D[i * k + j] = dist;
    double mn = valid ? dist : INFINITY, mx = valid ? dist : -INFINITY;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
      mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
    }
    if (lane == 0) {
      smn[j][w] = mn;
      smx[j][w] = mx;
    }
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)k) {
    const int j = threadIdx.x;
    double mn = INFINITY, mx = -INFINITY;
    for (int ww = 0; ww < RPD_THREADS / 32; ++ww) {
      mn = fmin(mn, smn[j][ww]);
      mx = fmax(mx, smx[j][ww]);
    }
    part[(size_t)blockIdx.x * 2 * k + j] = mn;
    part[(size_t)blockIdx.x * 2 * k + k + j] = mx;
  }
}

__global__ void k_minmax_final(const double* __restrict__ part, uint32_t nparts, int k,
                               double* __restrict__ out /* min[k], max[k] */) {
  // one block per reference point; fixed reduction order (deterministic)
  const int j = blockIdx.x;
  double mn = INFINITY, mx = -INFINITY;
  for (uint32_t b = threadIdx.x; b < nparts; b += blockDim.x) {
    mn = fmin(mn, part[(size_t)b * 2 * k + j]);
    mx = fmax(mx, part[(size_t)b * 2 * k + k + j]);
  }
  __shared__ double smn[32], smx[32];
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    mx = fmax(mx, __shfl_xor_sync(FULL_MASK, mx, o));
  }
  if ((threadIdx.x & 31) == 0) {
    smn[threadIdx.x >> 5] = mn;
    smx[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      mn = fmin(mn, smn[w]);
      mx = fmax(mx, smx[w]);
    }
    out[j] = mn;
    out[k + j] = mx;
  }
}

// ------------------------------------------------------------ key packing
// field_j = floor((D_ij - Dmin_j) / w_j), clamped to [0, maxkey_j].
// Completeness: for any pair in the result, |D_xj - D_yj| (computed) is
// below w_j, so the two fields differ by at most one; w_j = ε(1+δ) with δ
// covering the FP64 rounding of the distances and of the quotient (chosen
// on the host).  Clamping only shrinks differences.
__global__ void k_pack_keys(const double* __restrict__ D, size_t n, PackParams P,
                            uint64_t* __restrict__ keys) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t key = 0;
  for (int j = 0; j < P.k; ++j) {
    double v = floor((D[i * P.kstride + P.col[j]] - P.dmin[j]) / P.w[j]);
    v = fmin(fmax(v, 0.0), (double)P.maxkey[j]);
    key |= (uint64_t)v << P.shift[j];
  }
  keys[i] = key;
}

__global__ void k_iota(uint32_t* v, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = (uint32_t)i;
}

// ------------------------------------------------------------ bins
__global__ void k_bin_flags(const uint64_t* __restrict__ keys, size_t n, uint32_t* __restrict__ flags) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

__global__ void k_bin_starts(const uint64_t* __restrict__ keys, size_t n,
                             const uint32_t* __restrict__ binid /* exclusive scan of flags */,
                             uint32_t* __restrict__ bstart, uint64_t* __restrict__ bkey) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool head = (i == 0 || keys[i] != keys[i - 1]);
  if (head) {
    bstart[binid[i]] = (uint32_t)i;
    bkey[binid[i]] = keys[i];
  }
  if (i == n - 1) bstart[binid[i] + (head ? 1 : 0)] = (uint32_t)n;
}

// ------------------------------------------------------------ point gather
// Sorted-order copies for the join: FP32 centred coordinates (row stride
// dpad, zero padded), the original row ids, and optionally FP64 rows for the
// plain FP64 join.  Also the largest FP32 row norm (for the filter's error
// bound), reduced per block.
template <class T>
__global__ void k_gather_points(const T* __restrict__ x, size_t n, uint32_t d,
                                const uint32_t* __restrict__ perm, const double* __restrict__ center,
                                uint32_t dpad32, float* __restrict__ xf, uint32_t dpad64,
                                double* __restrict__ xd, uint32_t* __restrict__ ids,
                                double* __restrict__ norm_part) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double nrm2 = 0.0;
  if (p < n) {
    const uint32_t src = perm[p];
    ids[p] = src;
    for (uint32_t t = 0; t < dpad32; ++t) {
      float v = 0.f;
      if (t < d) v = (float)(ld(x, (size_t)src * d + t) - center[t]);
      if (xf) xf[p * dpad32 + t] = v;
      nrm2 = fma((double)v, (double)v, nrm2);
    }
    if (xd) {
      for (uint32_t t = 0; t < dpad64; ++t) xd[p * dpad64 + t] = t < d ? ld(x, (size_t)src * d + t) : 0.0;
    }
  }
  // block max of nrm2
#pragma unroll
  for (int o = 16; o; o >>= 1) nrm2 = fmax(nrm2, __shfl_xor_sync(FULL_MASK, nrm2, o));
  __shared__ double sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = nrm2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, sm[w]);
    norm_part[blockIdx.x] = m;
  }
}

__global__ void k_max_final(const double* __restrict__ part, uint32_t nparts, double* out) {
  double m = 0;
  for (uint32_t i = threadIdx.x; i < nparts; i += blockDim.x) m = fmax(m, part[i]);
#pragma unroll
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(FULL_MASK, m, o));
  __shared__ double sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = fmax(r, sm[w]);
    *out = r;
  }
}

// ------------------------------------------------------------ neighbour enumeration
// Up to 8 threads per non-empty bin h.  Depth-first over the key fields: at
// level j the candidate field value is K_j - 1, K_j, K_j + 1; the bins whose
// key starts with the chosen prefix form a contiguous sorted range, found by
// two lower-bound searches inside the parent range.  The first p fields
// skip the searches: a direct-address table (ptab[v] = first bin whose
// p-field prefix, read as a mixed-radix number, is >= v) gives the range of
// each of the 3^p prefixes with two loads, and the walk starts at level p
// inside it.  A range lying wholly below h is skipped (home <= neighbour).
// Leaves come out in ascending bin order, starting with h itself.
//
// Pass 1 (FILL false) counts neighbours and candidate points per home bin;
// k_unit_plan turns them into units; pass 2 writes the neighbour list and the
// units.  The candidate points of h's neighbour list are cut into segments of
// equal length, and the home bin into chunks of `chunk` points; one unit is
// one (chunk, segment) combination.
__device__ __forceinline__ uint32_t lower_bound_u64(const uint64_t* __restrict__ a, uint32_t lo,
                                                    uint32_t hi, uint64_t v) {
  while (lo < hi) {
    uint32_t mid = lo + ((hi - lo) >> 1);
    if (a[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Home-point sample (mistic_opts.home_sample): group g (points
// [512 g, 512 g + 512) of bin h's sorted order) takes part iff a hash of
// (h, g) is 0 mod S.  Every unit chunk size (4 .. 512 points) divides 512,
// so a unit is either wholly in the sample or wholly out of it, in every mode.
constexpr uint32_t SAMPLE_GROUP = 512;
__device__ __forceinline__ bool group_sampled(uint32_t h, uint32_t g, uint32_t S) {
  if (S <= 1) return true;
  uint32_t x = h * 0x9E3779B1u ^ (g + 0x7F4A7C15u) * 0x85EBCA77u;
  x ^= x >> 15;
  x *= 0x2C1B3C6Du;
  x ^= x >> 12;
  return x % S == 0;
}

// Field j of key K: bits [shift[j], shift[j-1]) (shift[-1] = 64).
__device__ __forceinline__ int key_field(uint64_t K, const EnumParams& P, int j) {
  const int hi_bit = j == 0 ? 64 : P.shift[j - 1];
  const int width = hi_bit - P.shift[j];
  const uint64_t mask = width >= 64 ? ~0ull : ((1ull << width) - 1ull);
  return (int)((K >> P.shift[j]) & mask);
}

// The same walk for any depth, with its per-level state in arrays (local
// memory): used below the levels walk_levels keeps in registers.
template <class Leaf>
__device__ __noinline__ void walk_deep(const uint64_t* __restrict__ bkey, uint64_t K, uint32_t hb,
                                       const EnumParams& P, int j0, uint32_t lo0, uint32_t hi0, uint64_t base0,
                                       Leaf& leaf) {
  uint32_t lo[MAX_K + 1], hi[MAX_K + 1];
  uint64_t base[MAX_K + 1];
  int di[MAX_K + 1];
  lo[j0] = lo0;
  hi[j0] = hi0;
  base[j0] = base0;
  di[j0] = 0;
  int j = j0;
  while (j >= j0) {
    if (di[j] == 3) {
      --j;
      if (j >= j0) ++di[j];
      continue;
    }
    const int cv = key_field(K, P, j) + di[j] - 1;
    if (cv < 0 || (long long)cv > (long long)P.maxkey[j]) {
      ++di[j];
      continue;
    }
    const uint64_t lower = base[j] | ((uint64_t)cv << P.shift[j]);
    const uint64_t upper = lower + (1ull << P.shift[j]);
    const uint32_t a = lower_bound_u64(bkey, lo[j], hi[j], lower);
    const uint32_t b = lower_bound_u64(bkey, a, hi[j], upper);
    if (a == b || b <= hb) {
      ++di[j];
      continue;
    }
    if (j == P.k - 1) {
      leaf(a);
      ++di[j];
      continue;
    }
    base[j + 1] = lower;
    lo[j + 1] = a;
    hi[j + 1] = b;
    di[j + 1] = 0;
    ++j;
  }
}

// Ranges of at most this many bins are read through instead of walked: the
// reads do not depend on one another, a search's do.
constexpr uint32_t ENUM_SCAN = 32;

// leaf(a) for the bins a >= hb of [lo, hi) whose fields j .. k-1 are within
// one of the home key's.
template <class Leaf>
__device__ __forceinline__ void scan_range(const uint64_t* __restrict__ bkey, uint64_t K, uint32_t hb,
                                           const EnumParams& P, int j, uint32_t lo, uint32_t hi, Leaf& leaf) {
#pragma unroll 1
  for (uint32_t a = max(lo, hb); a < hi; ++a) {
    bool ok = true;
    if (j < P.k) {
      const uint64_t Ka = bkey[a];
      for (int q = j; q < P.k; ++q) {
        const int df = key_field(Ka, P, q) - key_field(K, P, q);
        ok = ok && df >= -1 && df <= 1;
      }
    }
    if (ok) leaf(a);
  }
}

// Depth-first walk of key fields j .. k-1 of home key K inside the sorted bin
// range [lo, hi) whose keys share the prefix bits `base`: the range of field
// values K_j - 1 .. K_j + 1, read through when it is short, else cut into its
// three values; leaf(a) for every bin a >= hb, in ascending order.  The first
// R levels keep their range and loop state in registers; deeper ones go to
// walk_deep.
template <int R, class Leaf>
__device__ __forceinline__ void walk_levels(const uint64_t* __restrict__ bkey, uint64_t K, uint32_t hb,
                                            const EnumParams& P, int j, uint32_t lo, uint32_t hi, uint64_t base,
                                            Leaf& leaf) {
  const int sh = P.shift[j];
  const int kfj = key_field(K, P, j);
  const int c0 = max(kfj - 1, 0), c1 = (int)min((long long)kfj + 1, (long long)P.maxkey[j]);
  uint32_t a = lower_bound_u64(bkey, lo, hi, base | ((uint64_t)c0 << sh));
  const uint32_t end = lower_bound_u64(bkey, a, hi, (base | ((uint64_t)c1 << sh)) + (1ull << sh));
  if (end <= hb) return;
  if (j == P.k - 1 || end - a <= ENUM_SCAN) {
    scan_range(bkey, K, hb, P, j + 1, a, end, leaf);
    return;
  }
#pragma unroll 1
  for (int cv = c0; cv <= c1; ++cv) {
    const uint64_t lower = base | ((uint64_t)cv << sh);
    const uint32_t b = cv == c1 ? end : lower_bound_u64(bkey, a, end, lower + (1ull << sh));
    if (a < b && b > hb) {
      if constexpr (R > 1)
        walk_levels<R - 1>(bkey, K, hb, P, j + 1, a, b, lower, leaf);
      else
        walk_deep(bkey, K, hb, P, j + 1, a, b, lower, leaf);
    }
    a = b;
  }
}

// The split of a home bin's work into units: home chunks of csz points (nch
// of them, nch_s in the sample) against segments of `seg` candidate points.
// Segment b covers the candidate ranks [b seg, (b + 1) seg) of the bin's
// neighbour list, wherever the bin boundaries fall; the units are ordered by
// segment, then chunk.
struct HomeSplit {
  bool tc;             // tensor-core units
  uint32_t csz, nch, nch_s;
  unsigned long long rows_s, self_s;  // sampled home points, and their pairs inside the bin
};

__device__ __forceinline__ HomeSplit home_split(const EnumParams& P, uint32_t hb, uint32_t asz) {
  HomeSplit s;
  // large home bins go to the tensor-core join (128-row chunks), the rest to the CUDA-core join
  s.tc = P.tc_min > 0 && asz >= P.tc_min;
  s.csz = s.tc ? P.tc_chunk : P.chunk;
  s.nch = (asz + s.csz - 1) / s.csz;
  s.nch_s = s.nch;
  s.rows_s = asz;
  s.self_s = (unsigned long long)asz * (asz - (asz > 0)) / 2;
  if (P.sample > 1) {
    s.nch_s = 0;
    for (uint32_t ch = 0; ch < s.nch; ++ch) s.nch_s += group_sampled(hb, ch * s.csz / SAMPLE_GROUP, P.sample);
    s.rows_s = 0;
    s.self_s = 0;
    for (uint32_t g0 = 0; g0 < asz; g0 += SAMPLE_GROUP) {
      if (!group_sampled(hb, g0 / SAMPLE_GROUP, P.sample)) continue;
      const unsigned long long g1 = min(asz, g0 + SAMPLE_GROUP), c = g1 - g0;
      s.rows_s += c;
      s.self_s += c * (asz - 1) - (g0 + g1 - 1) * c / 2;  // pairs (p, q) of the bin with p in the group, q > p
    }
  }
  return s;
}

// Chunks of the home bin with candidates in segment b: those whose first row
// lies below the segment's end.  The home bin leads its own neighbour list
// and a pair of two of its rows is taken at the smaller one, so chunk c has no
// candidates below rank c * csz (unit_bin skips them); segments are multiples
// of csz long.  Without this half of every home bin's own square was
// evaluated twice: 10 % of the cells of a 1M x 384 join with 62 bins.
__device__ __forceinline__ uint32_t seg_chunks(const HomeSplit& s, uint32_t seg, uint32_t b) {
  return (uint32_t)min((unsigned long long)s.nch, (b + 1ull) * (seg / s.csz));
}

// Units of the first nseg segments of a home bin.
__device__ __forceinline__ unsigned long long count_units(const EnumParams& P, const HomeSplit& s, uint32_t hb,
                                                          uint32_t seg, uint32_t nseg) {
  const uint32_t r = seg / s.csz;
  if (P.sample <= 1) {
    // (b + 1) r chunks while that is at most nch, then nch
    const unsigned long long B = min(nseg, s.nch / r);
    return r * (B * (B + 1) / 2) + (nseg - B) * (unsigned long long)s.nch;
  }
  unsigned long long u = 0;
  for (uint32_t c = 0; c < s.nch; ++c)
    if (c / r < nseg && group_sampled(hb, c * s.csz / SAMPLE_GROUP, P.sample)) u += nseg - c / r;
  return u;
}

// The units of one home bin while its neighbour list is walked: cut() ends
// those of the current segment at (s1, o1) and starts the next segment's at
// (s0, o0).  WARP: a warp's lanes share the chunks; else one thread.
template <bool WARP>
struct UnitWriter {
  Unit* units;   // of the current segment
  uint32_t hb, seg, nseg, b;

  __device__ __forceinline__ uint32_t each(const EnumParams& P, const HomeSplit& s, uint32_t nc, Unit* u, bool start,
                                           uint32_t e, uint32_t o) const {
    uint32_t n = 0;  // sampled chunks so far
    for (uint32_t c0 = 0; c0 < nc; c0 += WARP ? 32u : 1u) {
      const uint32_t c = c0 + (WARP ? (threadIdx.x & 31u) : 0u);
      const bool take = c < nc && group_sampled(hb, c * s.csz / SAMPLE_GROUP, P.sample);
      const uint32_t m = WARP ? __ballot_sync(FULL_MASK, take) : (take ? 1u : 0u);
      if (take) {
        Unit& t = u[n + (WARP ? __popc(m & ((1u << (threadIdx.x & 31u)) - 1u)) : 0)];
        if (start) {
          t.h = hb;
          t.chunk = c;
          t.s0 = e;
          t.o0 = o;
        } else {
          t.s1 = e;
          t.o1 = o;
        }
      }
      n += __popc(m);
    }
    return n;
  }
  __device__ __forceinline__ void begin(const EnumParams& P, const HomeSplit& s, uint32_t s0) {
    b = 0;
    if (nseg) each(P, s, seg_chunks(s, seg, 0), units, true, s0, 0);
  }
  __device__ __forceinline__ void cut(const EnumParams& P, const HomeSplit& s, uint32_t s1, uint32_t o1, uint32_t s0,
                                      uint32_t o0) {
    units += each(P, s, seg_chunks(s, seg, b), units, false, s1, o1);
    if (++b < nseg) each(P, s, seg_chunks(s, seg, b), units, true, s0, o0);
  }
};

// Adds the home bin's candidate points, once per home chunk, to its class's
// total (the segment lengths are chosen from it).
__device__ __forceinline__ void add_work(idx::EnumTotals* tot, unsigned long long v, bool tc) {
  unsigned long long w[2] = {tc ? 0ull : v, tc ? v : 0ull};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int o = 16; o; o >>= 1) w[k] += __shfl_xor_sync(FULL_MASK, w[k], o);
    if ((threadIdx.x & 31) == 0 && w[k]) atomicAdd(&tot->work[k], w[k]);
  }
}

// P.lanes threads (a power of two within a warp) share a home bin when the
// prefix table is used: each takes a run of the prefixes.  Pass 1 leaves each
// one's first neighbour and first candidate rank within the bin in lane_off.
template <bool FILL>
__global__ void __launch_bounds__(128, 8) k_enum(const uint64_t* __restrict__ bkey, const uint32_t* __restrict__ bstart,
                       uint32_t m, EnumParams P, uint32_t* __restrict__ npts, uint32_t* __restrict__ nbr_cnt,
                       uint2* __restrict__ lane_off, idx::EnumTotals* __restrict__ tot,
                       const uint32_t* __restrict__ nbr_off, const uint32_t* __restrict__ unit_off,
                       const uint32_t* __restrict__ unit_off_tc, uint32_t* __restrict__ nbr,
                       Unit* __restrict__ units_simt, Unit* __restrict__ units_tc) {
  const unsigned long long gt = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t hb = (uint32_t)min((unsigned long long)m, gt / P.lanes), part = (uint32_t)gt & (P.lanes - 1);
  unsigned long long work = 0;
  uint32_t cnt = 0, pts = 0;
  bool tc = false;
  if (hb < m) {
    const uint64_t K = bkey[hb];
    const uint32_t asz = bstart[hb + 1] - bstart[hb];
    const HomeSplit hsp = home_split(P, hb, asz);
    tc = hsp.tc;
    const uint32_t n0 = FILL ? nbr_off[hb] : 0u;
    const uint32_t seg = FILL ? tot->seg[tc ? 1 : 0] : 0u;
    const uint32_t total = FILL ? npts[hb] : 0u;
    const uint32_t nseg = FILL ? (uint32_t)(((unsigned long long)total + seg - 1) / seg) : 0u;
    UnitWriter<false> uw{FILL ? (tc ? units_tc + unit_off_tc[hb] : units_simt + unit_off[hb]) : nullptr, hb, seg, nseg, 0};
    unsigned long long cut = seg;  // candidate rank of the next segment boundary
    if (FILL) {
      if (part == 0) {
        uw.begin(P, hsp, n0);
      } else {
        const uint2 lo = lane_off[gt];
        cnt = lo.x;
        pts = lo.y;
        uw.b = pts / seg;  // boundaries up to here belong to the threads before
        uw.units += count_units(P, hsp, hb, seg, uw.b);
        cut = (uw.b + 1ull) * seg;
      }
    }

    // Visits neighbour bin `a` (ascending, a >= hb): its points, and in pass
    // 2 the neighbour list and the segment boundaries that fall inside it.
    auto leaf = [&](uint32_t a) {
      const uint32_t bsz = bstart[a + 1] - bstart[a];
      if (FILL) {
        nbr[n0 + cnt] = a;
        for (; cut <= (unsigned long long)pts + bsz; cut += seg) {
          const uint32_t o = (uint32_t)(cut - pts);  // 1 .. bsz
          uw.cut(P, hsp, n0 + cnt + 1, o, n0 + cnt + (o == bsz), o == bsz ? 0u : o);
        }
        if (pts + bsz == total && uw.b < nseg) uw.cut(P, hsp, n0 + cnt + 1, bsz, 0, 0);  // the list ends in segment b
      }
      pts += bsz;
      ++cnt;
    };

    if (P.k == 0) {
      leaf(hb);  // no key fields: one bin holding every point (lanes is 1)
    } else if (P.p == 0) {
      walk_levels<3>(bkey, K, hb, P, 0, 0u, m, 0ull, leaf);  // lanes is 1
    } else {
      // prefixes in ascending order: field q < p - 1 offset by digit q of cb
      // in base 3 (field 0 most significant).  The values of field p - 1
      // adjoin in the table, so its three prefixes are one range.  The first
      // half of the prefixes lies below the home bin's.
      int n3 = 1;
      for (int q = 0; q + 1 < P.p; ++q) n3 *= 3;
      const int last = P.p - 1;
      const int kl = key_field(K, P, last);
      const int c0 = max(kl - 1, 0), c1 = (int)min((long long)kl + 1, (long long)P.maxkey[last]);
      const int mid = n3 / 2, np = n3 - mid;
      const int cb1 = mid + (int)(np * (part + 1) / P.lanes);
      for (int cb = mid + (int)(np * part / P.lanes); cb < cb1; ++cb) {
        int rem = cb, pw = n3 / 3;
        uint32_t idx = 0;
        uint64_t pre = 0;
        bool ok = true;
        for (int q = 0; q < last; ++q) {
          const int t = rem / pw;
          rem -= t * pw;
          pw /= 3;
          const int cv = key_field(K, P, q) + t - 1;
          if (cv < 0 || (uint32_t)cv > P.maxkey[q]) {
            ok = false;
            break;
          }
          idx += (uint32_t)cv * P.stride[q];
          pre |= (uint64_t)cv << P.shift[q];
        }
        if (!ok) continue;
        const uint32_t r0 = P.ptab[idx + c0], r1 = P.ptab[idx + c1 + 1];
        if (r0 == r1 || r1 <= hb) continue;
        if (P.p == P.k || r1 - r0 <= ENUM_SCAN) {
          scan_range(bkey, K, hb, P, P.p, r0, r1, leaf);
          continue;
        }
        for (int cv = c0; cv <= c1; ++cv) {
          const uint32_t a = P.ptab[idx + cv], b = P.ptab[idx + cv + 1];
          if (a < b && b > hb) walk_levels<3>(bkey, K, hb, P, P.p, a, b, pre | ((uint64_t)cv << P.shift[last]), leaf);
        }
      }
    }
    work = (unsigned long long)hsp.nch_s * pts;
  }
  if (!FILL) {
    add_work(tot, work, tc);
    uint32_t ce = cnt, pe = pts;  // inclusive sums over the bin's threads
    for (uint32_t o = 1; o < P.lanes; o <<= 1) {
      const uint32_t c = __shfl_up_sync(FULL_MASK, ce, o, P.lanes), p = __shfl_up_sync(FULL_MASK, pe, o, P.lanes);
      if (part >= o) {
        ce += c;
        pe += p;
      }
    }
    if (hb < m) {
      if (P.lanes > 1) lane_off[gt] = make_uint2(ce - cnt, pe - pts);
      if (part == P.lanes - 1) {
        nbr_cnt[hb] = ce;
        npts[hb] = pe;
      }
    }
  }
}

// The same enumeration with a warp per home bin: the keys from the bin itself
// up to the last one whose field 0 is within one of its own are read 32 at a
// time and every field is compared.  A thread's walk takes up to 3^k
// dependent steps, and with few bins nothing hides them: at 62 bins, k = 8,
// the two passes took 7.4 ms, at 292 bins, k = 6, 0.8 ms.
constexpr int FLAT_WARPS = 4;
template <bool FILL>
__global__ void __launch_bounds__(FLAT_WARPS * 32)
k_enum_flat(const uint64_t* __restrict__ bkey, const uint32_t* __restrict__ bstart, uint32_t m, EnumParams P,
            uint32_t* __restrict__ npts, uint32_t* __restrict__ nbr_cnt, idx::EnumTotals* __restrict__ tot,
            const uint32_t* __restrict__ nbr_off, const uint32_t* __restrict__ unit_off,
            const uint32_t* __restrict__ unit_off_tc, uint32_t* __restrict__ nbr, Unit* __restrict__ units_simt,
            Unit* __restrict__ units_tc) {
  const uint32_t hb = blockIdx.x * FLAT_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (hb >= m) return;  // warp-uniform
  const uint64_t K = bkey[hb];
  const uint32_t asz = bstart[hb + 1] - bstart[hb];
  const HomeSplit hsp = home_split(P, hb, asz);
  uint32_t end = m;
  if (P.k > 0) {
    const uint64_t f0 = (uint64_t)key_field(K, P, 0) + 2;
    if (f0 <= P.maxkey[0]) end = lower_bound_u64(bkey, hb, m, f0 << P.shift[0]);
  }
  uint32_t cnt = 0, pts = 0;
  const uint32_t n0 = FILL ? nbr_off[hb] : 0u;
  const uint32_t seg = FILL ? tot->seg[hsp.tc ? 1 : 0] : 0u;
  const uint32_t total = FILL ? npts[hb] : 0u;
  const uint32_t nseg = FILL ? (uint32_t)(((unsigned long long)total + seg - 1) / seg) : 0u;
  UnitWriter<true> uw{FILL ? (hsp.tc ? units_tc + unit_off_tc[hb] : units_simt + unit_off[hb]) : nullptr, hb, seg, nseg,
                      0};
  unsigned long long cut = seg;
  if (FILL) uw.begin(P, hsp, n0);
  for (uint32_t c0 = hb; c0 < end; c0 += 32) {
    const uint32_t a = c0 + lane;
    bool ok = a < end;
    const uint64_t Ka = ok ? bkey[a] : 0ull;
    for (int j = 0; j < P.k && __any_sync(FULL_MASK, ok); ++j) {
      const int df = key_field(Ka, P, j) - key_field(K, P, j);
      ok = ok && df >= -1 && df <= 1;
    }
    const uint32_t hit = __ballot_sync(FULL_MASK, ok);
    if (!hit) continue;
    const uint32_t bsz = ok ? bstart[a + 1] - bstart[a] : 0u;
    uint32_t incl = bsz;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    const uint32_t step = __shfl_sync(FULL_MASK, incl, 31);
    if (FILL) {
      const uint32_t pos = n0 + cnt + __popc(hit & ((1u << lane) - 1u));
      if (ok) nbr[pos] = a;
      // segment boundaries among these bins' points (warp-uniform loop)
      for (; cut <= (unsigned long long)pts + step; cut += seg) {
        const uint32_t r = (uint32_t)(cut - pts);  // 1 .. step: inside the first bin whose inclusive end reaches r
        const int src = __ffs(__ballot_sync(FULL_MASK, ok && incl >= r)) - 1;
        const uint32_t e = __shfl_sync(FULL_MASK, pos, src), z = __shfl_sync(FULL_MASK, bsz, src);
        const uint32_t o = r - (__shfl_sync(FULL_MASK, incl, src) - z);
        uw.cut(P, hsp, e + 1, o, e + (o == z), o == z ? 0u : o);
      }
      if (pts + step == total && uw.b < nseg) {  // the list ends in segment b
        const int src = 31 - __clz(hit);
        uw.cut(P, hsp, __shfl_sync(FULL_MASK, pos, src) + 1, __shfl_sync(FULL_MASK, bsz, src), 0, 0);
      }
    }
    pts += step;
    cnt += __popc(hit);
  }
  if (!FILL && lane == 0) {
    nbr_cnt[hb] = cnt;
    npts[hb] = pts;
    const unsigned long long work = (unsigned long long)hsp.nch_s * pts;
    if (work) atomicAdd(&tot->work[hsp.tc ? 1 : 0], work);
  }
}

// Segment lengths from the work totals, and the units and candidate pairs of
// every home bin.  A join of little work gets segments short enough for
// want_units units of each class: with 4096-point segments the 100,000 x 18
// uniform join had 2,145 CUDA-core units on 4,864 resident warps and ran as
// long as its slowest one (1.78 ms).
__global__ void k_unit_plan(const uint32_t* __restrict__ bstart, uint32_t m, EnumParams P,
                            const uint32_t* __restrict__ npts, const uint32_t* __restrict__ nbr_cnt,
                            uint32_t* __restrict__ unit_cnt, uint32_t* __restrict__ unit_cnt_tc,
                            idx::EnumTotals* __restrict__ tot) {
  uint32_t seg[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    seg[c] = P.seg_max[c];
    if (P.want_units[c]) {
      const unsigned long long fair = (tot->work[c] / P.want_units[c] + 127) & ~127ull;
      seg[c] = (uint32_t)min((unsigned long long)P.seg_max[c], max((unsigned long long)P.seg_min[c], fair));
    }
    // A bin of n points holds n^2 / (2 chunk seg) units, so a few very large
    // bins would run past the work lists' 32-bit offsets, and long before that
    // take gigabytes at 24 bytes a unit: 4,096-point segments of 12M points in
    // one bin are 4.4e9 units at chunks of 4.  work / seg + one a chunk bounds
    // the units of a class.
    if (P.max_units) {
      unsigned long long len = min(tot->work[c] / P.max_units + 1, 1ull << 30);
      if (P.seg_to_bin) len = min(len, (unsigned long long)tot->max_bin);
      seg[c] = (uint32_t)max((unsigned long long)seg[c], len);
    }
    const uint32_t csz = c ? P.tc_chunk : P.chunk;  // a multiple of the home chunk (seg_chunks)
    seg[c] = (seg[c] + csz - 1) / csz * csz;
  }
  if (blockIdx.x == 0 && threadIdx.x < 2) tot->seg[threadIdx.x] = seg[threadIdx.x];
  unsigned long long s[4] = {0, 0, 0, 0};
  for (uint32_t hb = blockIdx.x * blockDim.x + threadIdx.x; hb < m; hb += gridDim.x * blockDim.x) {
    const uint32_t asz = bstart[hb + 1] - bstart[hb];
    const HomeSplit h = home_split(P, hb, asz);
    const uint32_t sg = seg[h.tc ? 1 : 0];
    const unsigned long long nu = count_units(P, h, hb, sg, (uint32_t)(((unsigned long long)npts[hb] + sg - 1) / sg));
    // a bin's unit count saturates at 2^32 - 1; the 64-bit totals then exceed
    // the 32-bit offsets the work lists use, and the call fails with
    // MISTIC_ERR_TOO_LARGE
    const uint32_t nu32 = nu > 0xffffffffull ? 0xffffffffu : (uint32_t)nu;
    unit_cnt[hb] = h.tc ? 0u : nu32;
    unit_cnt_tc[hb] = h.tc ? nu32 : 0u;
    s[0] += h.self_s + h.rows_s * (npts[hb] - asz);
    s[1] += nbr_cnt[hb];
    s[2] += h.tc ? 0u : nu32;
    s[3] += h.tc ? nu32 : 0u;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int o = 16; o; o >>= 1) s[k] += __shfl_xor_sync(FULL_MASK, s[k], o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (s[0]) atomicAdd(&tot->cand, s[0]);
    for (int k = 0; k < 3; ++k)
      if (s[k + 1]) atomicAdd(&tot->n[k], s[k + 1]);
  }
}

// Points of the largest bin into *out (zero before).
__global__ void k_max_bin(const uint32_t* __restrict__ bstart, uint32_t m, uint32_t* __restrict__ out) {
  uint32_t v = 0;
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < m; b += gridDim.x * blockDim.x)
    v = max(v, bstart[b + 1] - bstart[b]);
  v = __reduce_max_sync(FULL_MASK, v);
  if ((threadIdx.x & 31) == 0 && v) atomicMax(out, v);
}

// Bins per prefix of the enumeration table: cnt[v] += 1 for each bin whose
// first P.p key fields, as a mixed-radix number with strides P.stride, are v.
__global__ void k_prefix_count(const uint64_t* __restrict__ bkey, uint32_t m, EnumParams P,
                               uint32_t* __restrict__ cnt) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= m) return;
  const uint64_t K = bkey[b];
  uint32_t v = 0;
  for (int j = 0; j < P.p; ++j) {
    const int w = min((j == 0 ? 64 : P.shift[j - 1]) - P.shift[j], 63);
    v += (uint32_t)((K >> P.shift[j]) & ((1ull << w) - 1ull)) * P.stride[j];
  }
  atomicAdd(&cnt[v], 1u);
}

// ------------------------------------------------------------ host launchers
namespace idx {

void colstats(mistic_handle_s* h, const void* x, mistic_dtype dt, size_t n, uint32_t d,
              double* part, uint32_t nparts, double* out, unsigned* nonfinite) {
  const dim3 grd((d + CS_THREADS - 1) / CS_THREADS, nparts);
  if (dt == MISTIC_F64)
    k_colstats<double><<<grd, CS_THREADS, 0, h->stream>>>((const double*)x, n, d, part, nonfinite);
  else
    k_colstats<float><<<grd, CS_THREADS, 0, h->stream>>>((const float*)x, n, d, part, nonfinite);
  launched(h, "colstats");
  k_colstats_final<<<(d + 7) / 8, 256, 0, h->stream>>>(part, nparts, d, n, out);
  launched(h, "colstats_final");
}

size_t cov_parts(uint32_t S, uint32_t d) { return (S + cov_chunk(d) - 1) / cov_chunk(d); }

void sample_cov(mistic_handle_s* h, const void* x, mistic_dtype dt, size_t n, uint32_t d,
                uint32_t S, double* sbuf, const double* mu, double* part, double* cov) {
  const size_t tot = (size_t)S * d;
  const unsigned nb = (unsigned)((tot + 255) / 256);
  if (dt == MISTIC_F64)
    k_gather_sample<double><<<nb, 256, 0, h->stream>>>((const double*)x, n, d, S, sbuf);
  else
    k_gather_sample<float><<<nb, 256, 0, h->stream>>>((const float*)x, n, d, S, sbuf);
  launched(h, "gather_sample");
  const uint32_t chunk = cov_chunk(d), chunks = (S + chunk - 1) / chunk;
  dim3 blk(COV_T, COV_T), grd((d + COV_T - 1) / COV_T, (d + COV_T - 1) / COV_T, chunks);
  if (chunk == 32)
    k_sample_cov_part<32><<<grd, blk, 0, h->stream>>>(sbuf, S, d, mu, part);
  else
    k_sample_cov_part<128><<<grd, blk, 0, h->stream>>>(sbuf, S, d, mu, part);
  launched(h, "sample_cov_part");
  k_sample_cov_final<<<(unsigned)((4 * (size_t)d * d + 255) / 256), 256, 0, h->stream>>>(part, chunks, d, S, cov);
  launched(h, "sample_cov_final");
}

void rp_dist(mistic_handle_s* h, const void* x, mistic_dtype dt, size_t n, uint32_t d,
             const double* rps, int k, double* D, double* part, double* mm) {
  const unsigned tpb = row_block(h, n), nparts = (unsigned)((n + tpb - 1) / tpb);
  auto launch = [&](auto kern, const auto* xs, int K) {
    allow_max_dyn_smem(kern);
    const size_t smem = (tpb * (RPD_COLS + 1) + (size_t)K * RPD_COLS) * sizeof(double);
    kern<<<nparts, tpb, smem, h->stream>>>(xs, n, d, rps, k, D, part);
  };
#define MISTIC_RPD(T, K)                                             \
  tpb == 64 ? launch(k_rp_dist<T, K, 64>, (const T*)x, K) : launch(k_rp_dist<T, K, 256>, (const T*)x, K)
  if (dt == MISTIC_F64) {
    if (k <= 8) MISTIC_RPD(double, 8); else MISTIC_RPD(double, 16);
  } else {
    if (k <= 8) MISTIC_RPD(float, 8); else MISTIC_RPD(float, 16);
  }
#undef MISTIC_RPD
  launched(h, "rp_dist");
  k_minmax_final<<<k, 256, 0, h->stream>>>(part, nparts, k, mm);
  launched(h, "minmax_final");
}

void pack_keys(mistic_handle_s* h, const double* D, size_t n, const PackParams& P, uint64_t* keys) {
  const unsigned tpb = row_block(h, n);
  k_pack_keys<<<(unsigned)((n + tpb - 1) / tpb), tpb, 0, h->stream>>>(D, n, P, keys);
  launched(h, "pack_keys");
}

void iota(mistic_handle_s* h, uint32_t* v, size_t n) {
  k_iota<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(v, n);
  launched(h, "iota");
}

void bins(mistic_handle_s* h, const uint64_t* keys, size_t n, uint32_t* flags, uint32_t* nbins_dev,
          uint32_t* bstart, uint64_t* bkey) {
  const unsigned nb = (unsigned)((n + 255) / 256);
  k_bin_flags<<<nb, 256, 0, h->stream>>>(keys, n, flags);
  launched(h, "bin_flags");
  exclusive_scan<uint32_t>(h, flags, flags, n, nbins_dev);
  k_bin_starts<<<nb, 256, 0, h->stream>>>(keys, n, flags, bstart, bkey);
  launched(h, "bin_starts");
}

void gather(mistic_handle_s* h, const void* x, mistic_dtype dt, size_t n, uint32_t d,
            const uint32_t* perm, const double* center, uint32_t dpad32, float* xf, uint32_t dpad64,
            double* xd, uint32_t* ids, double* norm_part, double* rmax) {
  const unsigned tpb = row_block(h, n), nb = (unsigned)((n + tpb - 1) / tpb);
  if (dt == MISTIC_F64)
    k_gather_points<double><<<nb, tpb, 0, h->stream>>>((const double*)x, n, d, perm, center, dpad32, xf,
                                                      dpad64, xd, ids, norm_part);
  else
    k_gather_points<float><<<nb, tpb, 0, h->stream>>>((const float*)x, n, d, perm, center, dpad32, xf,
                                                     dpad64, xd, ids, norm_part);
  launched(h, "gather_points");
  k_max_final<<<1, 1024, 0, h->stream>>>(norm_part, nb, rmax);
  launched(h, "max_final");
}

void prefix_table(mistic_handle_s* h, const uint64_t* bkey, uint32_t m, const EnumParams& P, uint32_t* ptab,
                  uint32_t entries) {
  MCK(cudaMemsetAsync(ptab, 0, ((size_t)entries + 1) * sizeof(uint32_t), h->stream));
  k_prefix_count<<<(m + 255) / 256, 256, 0, h->stream>>>(bkey, m, P, ptab);
  launched(h, "prefix_count");
  exclusive_scan<uint32_t>(h, ptab, ptab, (size_t)entries + 1, nullptr);
}

// A warp per bin reads every key whose field 0 lies near (m^2 work); threads
// that walk take up to 3^k dependent steps whatever m is.  Both passes and the
// scans, ms, warp / threads per bin: k = 2: 7,131 bins 0.058 / 0.085, 14,921
// 0.078 / 0.077, 21,555 0.099 / 0.087; k = 3: 8,952 bins 0.081 / 0.080, 17,832
// 0.152 / 0.112; k = 4: 7,599 bins 0.090 / 0.105, 12,446 0.140 / 0.118; k = 6:
// 7,824 bins 0.172 / 0.237, 10,061 0.248 / 0.247, 14,894 0.387 / 0.277; k = 8:
// 9,867 bins 0.340 / 0.627, 16,761 0.708 / 0.815, 26,116 1.376 / 1.200.
bool enum_flat(uint32_t m, const EnumParams& P) { return m <= (P.k > 6 ? 20480u : 10240u); }

// Threads a bin: up to 8, while they are 256 K threads in all, or 640 K where
// three levels or more are walked below the table (1.7 and 4.2 times what the
// device holds at once): beyond that the extra searches cost more than the
// shorter chains give.  ms at 1 / 2 / 4 / 8 threads: k = 6: 28,357 bins 0.725 / 0.514
// / 0.403 / 0.359, 76,372 0.926 / 0.691 / 0.719 / 0.752, 136,090 1.061 / 1.042
// / 1.166 / 1.289.  With three levels or more below the table the chains are
// longer: k = 8: 129,896 bins 8.12 / 6.22 / 5.21 / 5.48, 321,117 12.6 / 10.7 /
// 11.8 / 13.6.  Fewer than three table fields make too few prefixes to share.
uint32_t enum_lanes(uint32_t m, const EnumParams& P) {
  if (P.p < 3) return 1;
  const unsigned long long most = P.k - P.p >= 3 ? 640u * 1024u : 256u * 1024u;
  uint32_t l = 8;
  while (l > 1 && (unsigned long long)m * l > most) l >>= 1;
  return l;
}

static unsigned enum_grid(uint32_t m, const EnumParams& P) {
  return (unsigned)(((unsigned long long)m * P.lanes + 127) / 128);
}

void enum_count(mistic_handle_s* h, const uint64_t* bkey, const uint32_t* bstart, uint32_t m, const EnumParams& P,
                uint32_t* npts, uint32_t* nbr_cnt, uint2* lane_off, uint32_t* unit_cnt, uint32_t* unit_cnt_tc,
                EnumTotals* tot) {
  MCK(cudaMemsetAsync(tot, 0, sizeof(EnumTotals), h->stream));
  if (enum_flat(m, P))
    k_enum_flat<false><<<(m + FLAT_WARPS - 1) / FLAT_WARPS, FLAT_WARPS * 32, 0, h->stream>>>(
        bkey, bstart, m, P, npts, nbr_cnt, tot, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
  else
    k_enum<false><<<enum_grid(m, P), 128, 0, h->stream>>>(bkey, bstart, m, P, npts, nbr_cnt, lane_off, tot, nullptr,
                                                          nullptr, nullptr, nullptr, nullptr, nullptr);
  launched(h, "enum_count");
  const unsigned nb = std::max(1u, std::min((m + 255) / 256, 4u * (unsigned)h->sms));
  if (P.seg_to_bin) {
    k_max_bin<<<nb, 256, 0, h->stream>>>(bstart, m, &tot->max_bin);
    launched(h, "max_bin");
  }
  k_unit_plan<<<nb, 256, 0, h->stream>>>(bstart, m, P, npts, nbr_cnt, unit_cnt, unit_cnt_tc, tot);
  launched(h, "unit_plan");
  exclusive_scan3(h, nbr_cnt, unit_cnt, unit_cnt_tc, m);
}

void enum_fill(mistic_handle_s* h, const uint64_t* bkey, const uint32_t* bstart, uint32_t m, const EnumParams& P,
               const uint32_t* npts, const uint2* lane_off, const uint32_t* nbr_off, const uint32_t* unit_off,
               const uint32_t* unit_off_tc, const EnumTotals* tot, uint32_t* nbr, Unit* units, Unit* units_tc) {
  uint32_t* np = const_cast<uint32_t*>(npts);
  EnumTotals* t = const_cast<EnumTotals*>(tot);
  if (enum_flat(m, P))
    k_enum_flat<true><<<(m + FLAT_WARPS - 1) / FLAT_WARPS, FLAT_WARPS * 32, 0, h->stream>>>(
        bkey, bstart, m, P, np, nullptr, t, nbr_off, unit_off, unit_off_tc, nbr, units, units_tc);
  else
    k_enum<true><<<enum_grid(m, P), 128, 0, h->stream>>>(bkey, bstart, m, P, np, nullptr, const_cast<uint2*>(lane_off),
                                                         t, nbr_off, unit_off, unit_off_tc, nbr, units, units_tc);
  launched(h, "enum_fill");
}

// Points per log2 bin-size class: hist[c] += size of every bin with
// floor(log2(size)) == c (c < 32).
__global__ void k_bin_hist(const uint32_t* __restrict__ bstart, uint32_t m, unsigned long long* __restrict__ hist) {
  __shared__ unsigned long long sh[32];
  if (threadIdx.x < 32) sh[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < m; b += gridDim.x * blockDim.x) {
    const uint32_t sz = bstart[b + 1] - bstart[b];
    if (sz) atomicAdd(&sh[31 - __clz(sz)], (unsigned long long)sz);
  }
  __syncthreads();
  if (threadIdx.x < 32 && sh[threadIdx.x]) atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

void bin_hist(mistic_handle_s* h, const uint32_t* bstart, uint32_t m, unsigned long long* hist) {
  MCK(cudaMemsetAsync(hist, 0, 32 * sizeof(unsigned long long), h->stream));
  const unsigned nb = std::max(1u, std::min((m + 255) / 256, 4u * (unsigned)h->sms));
  k_bin_hist<<<nb, 256, 0, h->stream>>>(bstart, m, hist);
  launched(h, "bin_hist");
}

}  // namespace idx
}  // namespace mistic
