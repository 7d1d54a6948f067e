// Tensor-core distance join (tcgen05, sm_103a).
//
// Reference counterpart: the FP64 distance loop of nodeByPoint5 /
// cachedDistanceCheck (src/kernel.cu:992-1046, 833-865).  Here a unit — up to
// 128 points of one large home bin against a segment of its neighbour bins
// (bins >= home) — is evaluated as dense 128 x 128 tiles on the 5th-generation
// tensor cores:
//
//   A row m = [a'_m, |a'_m|^2, 1, 0...]      a' = a~ - c  (c: first home row)
//   B row n = [-2 q'_n, 1, |q'_n|^2, 0...]    q' = q~ - c
//   D[m][n] = sum_k A[m][k] B[n][k] = |a'|^2 + |q'|^2 - 2 a'.q' = ||a' - q'||^2
//
// where a~, q~ are the FP32 globally centred rows.  Each operand is split
// into bf16 hi + lo parts; D = Ahi.Bhi + Ahi.Blo + Alo.Bhi is accumulated in
// FP32 in tensor memory (3 MMAs per K step of 16).  Centering at the unit's
// first row keeps |a'|, |q'| at the size of the local neighbourhood, so the
// cancellation in the Gram form stays small.
//
// Exactness: per row and tile, a rigorous bound E on |D - s64| (s64 = the
// reference FP64 predicate value) gives T_lo = eps2/(1+g64) - E and
// T_hi = eps2/(1-g64) + E: D <= T_lo accepts, D > T_hi rejects, anything in
// between is re-decided with the reference FP64 predicate.  The bound covers
//   - bf16 splitting: each product carries <= 3.02 * 2^-16 |A_k||B_k| (bf16
//     keeps 8 significant bits: |x - hi| <= 2^-8 |x|, |x - hi - lo| <= 2^-16 |x|),
//   - tensor-core FP32 accumulation: taken as <= 2^-19 per MMA instruction
//     relative to the sum of |products| (a generous allowance),
//   - FP32 norms (g_d), the FP32 centring (2uR + u(|a'|+|q'|)),
// with sum_k |A_k||B_k| <= (|a'| + |q'|)^2.  Columns whose bound
// exceeds 16 eps2 are re-decided entirely in FP64 (T_lo = -1, T_hi = inf).
//
// Data movement: operands are converted from the sorted FP32 rows into the
// K-major layouts of chunk_off (tc_common.cuh), elected threads issue the MMAs
// and commit to mbarriers, and the epilogue warps read each 128 x 128 FP32
// accumulator back with tcgen05.ld.  Every mbarrier wait is bounded; on expiry
// the CTA records an error, stops, drains its MMAs and releases its tensor
// memory.
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "emit.cuh"
#include "internal.cuh"
#include "tc_common.cuh"

namespace mistic {
namespace {

using namespace tcu;

constexpr int TM = 128;          // home rows per tile (MMA M)
constexpr int TN = 128;          // candidate columns per tile (MMA N)
constexpr int WIN = 256;         // neighbour bins per candidate window

// ---------------------------------------------------------------- pipeline
// One persistent CTA per SM: 8 producer warps, NEPI epilogue warps, 4 MMA warps.
//   producers  K <= 32: 4 loader warps claim units, walk their neighbour bins
//              and copy each tile's 128 candidate rows (raw FP32, cp.async)
//              into a ring of RAW landing slots; 4 converter warps, a thread
//              a row, turn a slot into the bf16 hi/lo operand rows of one of
//              the NS B stages, with the per-column threshold folded in
//              (column d+1 holds |q'|^2 - T(n)), and stage each unit's home
//              rows (A: G chunks of 128).  A stage's operands go back when its
//              MMAs are done; what the epilogue needs of it sits in a ring of
//              its own.  K >= 48: all 8 warps do both, two
//              threads a row, the raw rows landing in the B stages
//              themselves where no separate slots fit;
//   MMA warps  one lane of each issues 3 * KP/16 tcgen05.mma per (tile, home
//              chunk) into its own of the NACC = 4 TMEM accumulators and
//              commits, the warps taking turns.  With two warps of two
//              accumulators each, a warp that waited for one could not refill
//              the other: 75.3 ms on the 5M x 18 join against 71.9, 1.54
//              against 1.47 on its 250k;
//   epilogue   groups of 4 warps, one per TMEM lane quarter, each group with
//              its own accumulators: tcgen05.ld, sign-bit test (D' < 0 marks
//              a candidate), home-bin rule by column range, sure accepts to
//              the pair list, the error band to the band list.
// Barriers (all waits bounded by a %globaltimer deadline):
//   rawfull[r] loaders    -> converters (each loader thread's copies landed, + 1 for the slot's metadata)
//   rawfree[r] converters -> loaders    (4 arrivals: slot read)
//   ubar       converters among themselves, twice a unit (128 arrivals)
//   full[s]    producers  -> MMA        (128 arrivals, or NPROD)
//   bfree[s]   MMA        -> producers  (a tcgen05.commit by each MMA warp, whether or not the tile holds work
//                                        for it: stage s read, full[s] and the tile's metadata seen)
//   mfree[m]   epilogue   -> producers  (metadata slot m drained; 48 arrivals: 12 / home chunks by each of a
//                                        group's 4 warps)
//   dfull[b]   MMA        -> epilogue   (tcgen05.commit, + 1 for the accumulator's metadata)
//   dfree[b]   epilogue   -> MMA        (4 arrivals; accumulator b reusable)
//   afull      producers  -> MMA        (128 arrivals, or NPROD, per unit: A written)
//   afree      MMA        -> producers  (a tcgen05.commit by each MMA warp after a unit's last tile)
// A stage and its metadata slot are written again after both bfree and mfree.
// mfree alone says only that the warps which own a home chunk of the tile have
// issued it: a warp that owns none may not have waited on full[s] yet, and a
// second completion of full[s] would leave it on the wrong phase, or reading
// the wrong tile's metadata.
constexpr int NPW = 8;     // producer warps: two threads per operand row
constexpr int NPROD = NPW * 32;
constexpr int NLOAD = 128; // K <= 32: threads of the loader warps, and of the converter warps after them
constexpr int NUNIT = 8;   // unit slots between them (at most RAW = 4 units have tiles in flight)
// NEPI epilogue warps (a template parameter: 8 or 16) in groups of 4; the MMA
// warps follow them.
constexpr int EPI0 = NPW;  // first epilogue warp (a multiple of 4: warp % 4 is its lane quarter)
constexpr int NMMA = 4;    // MMA warps
__host__ __device__ constexpr int tc_threads(int nepi) { return (EPI0 + nepi + NMMA) * 32; }
constexpr int NACC = 4;    // TMEM accumulators of 128 columns (512 per CTA, one CTA per SM)
constexpr uint32_t FLAG_FIRST = 1, FLAG_LAST = 2, FLAG_END = 4;

struct __align__(16) TileMeta {
  uint32_t a0, na, flags, ng;  // ng: 128-row MMA tiles of this unit (1..G); the MMA warps read these four as one
  uint32_t inst;               // instance of the unit (fused batch joins; else 0)
  uint32_t ncols;
  uint32_t hcr, hq;  // columns [hcr & 255, hcr >> 8) hold home-bin rows, the first at sorted position hq
};

// What the converters need about a unit, written by a loader.
struct TcUnit {
  const float* X;   // the instance's sorted rows
  uint32_t a0, na, ng, inst;
  TcBound tb;
};

// A raw slot's tile.
struct TcSlot {
  uint32_t ncols, flags, hcr, hq, unit;  // unit: index into TcShared2::units
};

// What an accumulator holds: home chunk g of the tile with metadata slot ms.
struct __align__(16) TcAcc {
  uint32_t ms, g, end;
};

template <int NS, int G, int RAW>
struct TcShared2 {
  // Metadata slots.  Eight where they are apart from the stages: a slot is
  // held until the epilogue is done with its tile, and with four, tiles of one
  // home chunk could not be converted ahead of the four accumulators (250k x
  // 18 1.47 -> 1.44 ms).
  static constexpr int NM = RAW == 4 ? 8 : NS;
  __align__(16) float cadd_a[128];  // -c   (A rows: x - c)
  __align__(16) float cadd_b[128];  // 2c   (B rows: -2 (x - c))
  uint32_t w_home;  // (window generation << 8) | index of the home bin in the window
  uint32_t hx[4][2];  // home column range of issued tiles (producer thread 0 only)
  uint32_t qid[NM][TN];  // original row ids of the candidates
  __align__(16) float dlt[NM][TN];  // accept when D' < -dlt
  TileMeta meta[NM];
  uint32_t rid[RAW > 0 ? RAW : 1][TN];  // candidate ids of the tiles in the raw ring
  uint32_t w_start[WIN];
  uint32_t w_pref[WIN + 1];
  uint32_t scan_ws[NPW];
  unsigned long long unit;
  uint32_t w_total, w_pos, seg_next, w_nb;
  uint32_t ra2max;  // float bits, non-negative
  // K <= 32: [unit parity][A, B] as cadd_a, cadd_b, then the columns d and d + 1 (conv_row) and zeros
  __align__(16) float cadd[2][2][RAW == 4 ? 32 : 4];
  uint32_t ra2[4];                      // K <= 32: largest |a|^2 by unit mod 4, float bits
  TcUnit units[RAW == 4 ? NUNIT : 1];
  TcSlot slot[RAW == 4 ? RAW : 1];
  TcAcc acc[NACC];
  uint32_t abort_flag;
  uint32_t tmem_base;
  uint32_t pflag[2];  // producer-wide decisions, written by producer thread 0
  // [tile parity][K-block parity][row]: partial row norms of the two threads
  // of a row (K >= 48)
  float npart[RAW == 4 ? 1 : 2][2][RAW == 4 ? 1 : TM];
  unsigned long long full[NS], bfree[NS], mfree[NM], dfull[NACC], dfree[NACC], afull, afree;
  unsigned long long rawfull[RAW > 0 ? RAW : 1], rawfree[RAW > 0 ? RAW : 1], ubar;
};

// Barrier of the loader warps that also returns the AND of p over them.
__device__ __forceinline__ bool load_sync_and(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\t"
      "setp.ne.u32 pi, %1, 0;\n\t"
      "bar.red.and.pred po, 2, %2, pi;\n\t"
      "selp.u32 %0, 1, 0, po;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "n"(NLOAD)
      : "memory");
  return r != 0u;
}

// This thread's arrival on `bar` once every cp.async it issued before has landed.
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void prod_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NPROD) : "memory"); }

// Operand rows live in the layout of chunk_off: the 16-byte chunk of row r and
// K block kb (8 bf16) sits at bf16 offset chunk_off(r, kb).  A raw FP32 row is first copied (cp.async) into the
// chunk slots of the row itself -- floats [8kb, 8kb+4) into the hi chunk of
// block kb, [8kb+4, 8kb+8) into its lo chunk -- and then converted in place,
// block by block, into the augmented bf16 hi/lo row.  Two threads share a
// row, one per parity of the K blocks (kb = 2j + half); a thread only touches
// its own chunks.  Blocks wholly beyond the augmented columns (k0 >= d + 2)
// are cleared once when the kernel starts and never written again.
template <int KP>
__device__ __forceinline__ void load_half(__nv_bfloat16* hi, __nv_bfloat16* lo, uint32_t r, uint32_t half,
                                          const float* __restrict__ xr, uint32_t dpad) {
  constexpr int HB = KP / 16;
#pragma unroll
  for (int j = 0; j < HB; ++j) {
    const uint32_t kb = 2 * j + half, k0 = 8 * kb, off = chunk_off<KP>(r, kb);
    if (k0 < dpad) cp_async16(hi + off, xr + k0);
    if (k0 + 4 < dpad) cp_async16(lo + off, xr + k0 + 4);
  }
}

__device__ __forceinline__ void unpack8(const __nv_bfloat16* hi, const __nv_bfloat16* lo, uint32_t off, bool l0,
                                        bool l1, float (&x)[8]) {
  float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
  if (l0) x0 = *reinterpret_cast<const float4*>(hi + off);
  if (l1) x1 = *reinterpret_cast<const float4*>(lo + off);
  x[0] = x0.x, x[1] = x0.y, x[2] = x0.z, x[3] = x0.w;
  x[4] = x1.x, x[5] = x1.y, x[6] = x1.z, x[7] = x1.w;
}

__device__ __forceinline__ void store_split(__nv_bfloat16* hi, __nv_bfloat16* lo, uint32_t off, const float (&v)[8]) {
  uint4 oh, ol;
  uint32_t* ph = reinterpret_cast<uint32_t*>(&oh);
  uint32_t* pl = reinterpret_cast<uint32_t*>(&ol);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 hv = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    const float2 hf = __bfloat1622float2(hv);
    const __nv_bfloat162 lv = __floats2bfloat162_rn(v[2 * i] - hf.x, v[2 * i + 1] - hf.y);
    ph[i] = *reinterpret_cast<const uint32_t*>(&hv);
    pl[i] = *reinterpret_cast<const uint32_t*>(&lv);
  }
  *reinterpret_cast<uint4*>(hi + off) = oh;
  *reinterpret_cast<uint4*>(lo + off) = ol;
}

// Operand values: scale * fl(x[k] - c[k]) = fma(x[k], scale, cadd[k]) with
// cadd = -scale * c, exactly (scale is 1 or -2).  The row norm |x - c|^2 is
// accumulated from the scaled values (fma(v, v, acc) = scale^2 fma(t, t, acc')
// exactly) in K order per half; the halves are added by the caller.
//
// Pass 1 writes every K block of this thread that holds a data or an
// augmented column, with placeholders pd, pd1 in the augmented columns d and
// d + 1, and returns the partial sum of v^2; once the two halves of the norm
// are added, patch_col writes the one augmented value that depends on it
// (|a'|^2 in column d of A, |q'|^2 - T in column d + 1 of B).  A block is
// read before it is written, so the source may be the destination.
template <int KP>
__device__ __forceinline__ float conv_pass1(const __nv_bfloat16* sh, const __nv_bfloat16* sl, __nv_bfloat16* hi,
                                            __nv_bfloat16* lo, uint32_t r, uint32_t half, bool ok, const float* cadd,
                                            float scale, uint32_t d, float pd, float pd1) {
  constexpr int HB = KP / 16;
  float acc = 0.f;
  if (!ok) return acc;  // a column beyond the tile: its stale values are masked by the epilogue
#pragma unroll 2
  for (int j = 0; j < HB; ++j) {
    const uint32_t kb = 2 * j + half, k0 = 8 * kb, off = chunk_off<KP>(r, kb);
    float v[8];
    if (k0 >= d + 2) continue;  // zero block (cleared at the start)
    float x[8];
    unpack8(sh, sl, off, k0 < d, k0 + 4 < d, x);
    if (k0 + 8 <= d) {  // full block
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = fmaf(x[i], scale, cadd[k0 + i]);
        acc = fmaf(v[i], v[i], acc);
      }
    } else {  // holds d or d + 1
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t k = k0 + i;
        float t = 0.f;
        if (k < d) {
          t = fmaf(x[i], scale, cadd[k]);
          acc = fmaf(t, t, acc);
        } else if (k == d) {
          t = pd;
        } else if (k == d + 1) {
          t = pd1;
        }
        v[i] = t;
      }
    }
    store_split(hi, lo, off, v);
  }
  return acc;
}

// Whole-row forms for one thread a row (K <= 32): the raw row's chunks land in
// the row's own slots as in load_half, every K block of the row.
template <int KP>
__device__ __forceinline__ void load_row(__nv_bfloat16* hi, __nv_bfloat16* lo, uint32_t r,
                                         const float* __restrict__ xr, uint32_t dpad) {
#pragma unroll
  for (int kb = 0; kb < KP / 8; ++kb) {
    const uint32_t k0 = 8 * kb, off = chunk_off<KP>(r, kb);
    if (k0 < dpad) cp_async16(hi + off, xr + k0);
    if (k0 + 4 < dpad) cp_async16(lo + off, xr + k0 + 4);
  }
}

// Converts row r, its 8-float blocks given by block(kb, x) (zeros beyond
// column d - 1), into the bf16 hi/lo operand row (hi, lo), K blocks in order;
// returns the row norm |x - c|^2 (times scale^2).  cadd holds the constants of
// the augmented columns d and d + 1 after the data's, so that every column is
// one FMA: with a select by column instead, and cadd read a word at a time,
// the converters were the slowest role of joins with one home chunk a unit
// (5M x 18 69.0 -> 66.0 ms of tensor-core time, 100k x 18 1.45 -> 1.41).
template <int KP, class Block>
__device__ __forceinline__ float conv_row(Block block, __nv_bfloat16* hi, __nv_bfloat16* lo, uint32_t r,
                                          const float* cadd, float scale, uint32_t d) {
  float acc = 0.f;
#pragma unroll
  for (int kb = 0; kb < KP / 8; ++kb) {
    const uint32_t k0 = 8 * kb, off = chunk_off<KP>(r, kb);
    if (k0 >= d + 2) break;  // zero blocks (cleared at the start)
    float x[8], v[8];
    block(kb, x);
    const float4 c0 = *reinterpret_cast<const float4*>(cadd + k0), c1 = *reinterpret_cast<const float4*>(cadd + k0 + 4);
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = fmaf(x[i], scale, c[i]);
      if (k0 + i < d) acc = fmaf(v[i], v[i], acc);
    }
    store_split(hi, lo, off, v);
  }
  return acc;
}

// Column k of row r := v, split into bf16 hi + lo as store_split does.
template <int KP>
__device__ __forceinline__ void patch_col(__nv_bfloat16* hi, __nv_bfloat16* lo, uint32_t r, uint32_t k, float v) {
  const uint32_t off = chunk_off<KP>(r, k >> 3) + (k & 7);
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  hi[off] = h;
  lo[off] = __float2bfloat16_rn(v - __bfloat162float(h));
}

template <int KP, int NS, int G, int RAW, int NEPI>
__global__ void __launch_bounds__(tc_threads(NEPI), 1) k_join_tc(const JoinParams P, const TcParams T) {
  constexpr int MMA_WARP = EPI0 + NEPI;  // the first of NMMA
  extern __shared__ __align__(128) unsigned char tc_raw[];
  using Shared = TcShared2<NS, G, RAW>;
  __shared__ Shared S;
  constexpr int NM = Shared::NM;
  constexpr uint32_t OPB = TM * KP;  // bf16 elements per 128-row operand buffer
  unsigned char* tc_dyn = tc_raw + ((512u - (smem_u32(tc_raw) & 511u)) & 511u);  // swizzle atoms: 512 bytes
  __nv_bfloat16* Ahi = reinterpret_cast<__nv_bfloat16*>(tc_dyn);  // G home chunks of 128 rows
  __nv_bfloat16* Alo = Ahi + G * OPB;
  __nv_bfloat16* Bhi = Alo + G * OPB;  // NS stages of hi, then NS stages of lo
  __nv_bfloat16* Blo = Bhi + NS * OPB;
  __nv_bfloat16* Raw = Blo + NS * OPB;  // RAW landing slots (raw FP32 rows in the chunk layout, 2 * OPB each)
  unsigned long long* pstage = reinterpret_cast<unsigned long long*>(Raw + RAW * 2 * OPB);  // 2 NEPI x PSTAGE
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abort_flag = &S.abort_flag;

  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&S.full[i], RAW == 4 ? NLOAD : NPROD);
      mbar_init(&S.bfree[i], NMMA);
    }
    for (int i = 0; i < NM; ++i) mbar_init(&S.mfree[i], 48);
    for (int i = 0; i < NACC; ++i) {
      mbar_init(&S.dfull[i], 2);
      mbar_init(&S.dfree[i], 4);
    }
    mbar_init(&S.afull, RAW == 4 ? NLOAD : NPROD);
    mbar_init(&S.afree, NMMA);
    if (RAW == 4) {
      for (int i = 0; i < RAW; ++i) {
        mbar_init(&S.rawfull[i], NLOAD + 1);
        mbar_init(&S.rawfree[i], 4);
      }
      mbar_init(&S.ubar, NLOAD);
      for (int i = 0; i < 4; ++i) S.ra2[i] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
    S.abort_flag = 0;
    S.w_home = 0xffffffffu;
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&S.tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  {  // operand buffers start at zero: K blocks beyond the augmented columns are never written
    uint4* z = reinterpret_cast<uint4*>(tc_dyn);
    const uint32_t nz = (2 * G + 2 * NS) * OPB * (uint32_t)sizeof(__nv_bfloat16) / 16;
    for (uint32_t i = tid; i < nz; i += blockDim.x) z[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tbase = S.tmem_base;

  if (warp < NPW) {
    if constexpr (RAW == 4) {
    if (tid < NLOAD) {
      // ============================ loaders (K <= 32)
      // Thread t copies row t of every candidate tile.  The warps meet only to
      // claim a unit and to fill a window of neighbour bins; between those a
      // warp waits for its slots alone, so up to RAW tiles of copies are in
      // flight while the converters work.  A failed wait (abort) is carried in
      // `ok` to the next meeting, where all warps leave together.
      const uint32_t t = (uint32_t)tid;
      uint32_t k = 0, useq = 0, wgen = 0;  // tiles, units and windows so far
      bool ok = true;
      for (;;) {
        if (t == 0) {
          // claim index -> unit: units deferred by the last ring pass first,
          // then the list from main_start (the identity outside ring mode)
          const unsigned long long c = atomicAdd(&T.ctr->next_unit, 1ull);
          const unsigned long long uu =
              c < T.n_def_in ? (unsigned long long)T.def_in[c] : T.main_start + (c - T.n_def_in);
          S.unit = uu;
          bool go = (T.claim_cap == 0 || c < T.claim_cap) && uu < T.n_units && !*abort_flag;
          if (go && P.ring && *(volatile unsigned long long*)&P.ctr->stop) {  // the ring filled: leave it for the next pass
            const RingCtx rc{P.pair_tags, P.deferred, P.def_out, &P.ctr->def_n, &P.ctr->stop};
            ring_defer(&rc, P.tag_base_tc + (uint32_t)uu);
            go = false;
          }
          ok = ok && go;
        }
        if (!load_sync_and(ok)) break;
        const unsigned long long u = S.unit;
        const Unit U = T.units[u];
        // the unit's instance: its arrays and bound constants (fused batch
        // joins), or the launch's own
        const float* X = (const float*)P.xs;
        const uint32_t *bstart = P.bstart, *nbr = P.nbr, *ids = P.ids;
        uint32_t inst = 0;
        if (T.unit_inst) {
          inst = T.unit_inst[u];
          const InstDesc& I = P.insts[inst];
          X = (const float*)I.xs;
          bstart = I.bstart;
          nbr = I.nbr;
          ids = I.ids;
        }
        const uint32_t hs = bstart[U.h], he = bstart[U.h + 1];
        const uint32_t a0 = hs + U.chunk * (TM * G);
        const uint32_t na = min((uint32_t)(TM * G), he - a0);
        // the converters read the home rows when they reach the unit
        for (uint32_t r = t; r < na; r += NLOAD)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(X + (size_t)(a0 + r) * P.dpad));
        if (t == 0) {
          TcUnit& W = S.units[useq % NUNIT];
          W.X = X;
          W.a0 = a0;
          W.na = na;
          W.ng = (na + TM - 1) / TM;
          W.inst = P.ring ? P.tag_base_tc + (uint32_t)u : inst;  // the ring's tag of this unit's pairs
          W.tb = T.unit_inst ? P.insts[inst].tcb : T.b;
        }
        uint32_t flags = FLAG_FIRST;
        for (uint32_t seg = U.s0; seg < U.s1; seg += WIN) {
          // ---- window of up to WIN neighbour bins, two a thread
          const uint32_t nb = min((uint32_t)WIN, U.s1 - seg);
          uint32_t st[2] = {0, 0}, sz[2] = {0, 0}, bn[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (2 * t + q < nb) unit_bin(U, TM * G, nbr, bstart, seg + 2 * t + q, &bn[q], &st[q], &sz[q]);
          const uint32_t incl = warp_scan_incl(sz[0] + sz[1]);
          if (lane == 31) S.scan_ws[warp] = incl;
          ok = load_sync_and(ok);  // also: every warp is done with the window before
          if (!ok) break;
          uint32_t wp = 0;
          for (int w = 0; w < warp; ++w) wp += S.scan_ws[w];
          ++wgen;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (2 * t + q < nb) {
              S.w_start[2 * t + q] = st[q];
              S.w_pref[2 * t + q + 1] = wp + incl - (q == 0 ? sz[1] : 0u);
              if (bn[q] == U.h) S.w_home = ((wgen & 0xffffffu) << 8) | (2 * t + q);
            }
          }
          if (t == 0) S.w_pref[0] = 0;
          ok = load_sync_and(ok);
          if (!ok) break;
          const uint32_t wh = S.w_home, total = S.w_pref[nb];
          const int w_hj = (wh >> 8) == (wgen & 0xffffffu) ? (int)(wh & 255u) : -1;
          for (uint32_t pos = 0; pos < total; pos += TN, ++k) {
            const uint32_t ncols = min((uint32_t)TN, total - pos);
            if (pos + TN >= total && seg + nb >= U.s1) flags |= FLAG_LAST;
            // row of candidate rank pos + t: the warp finds the bin of its
            // first rank (two 32-way probes of the window prefix), then each
            // lane counts the bin boundaries among the next 32 ranks
            uint32_t q = 0xffffffffu;
            {
              const uint32_t r0 = pos + (t & ~31u);
              const uint32_t step = (nb + 31) >> 5;
              const uint32_t c = __popc(__ballot_sync(FULL_MASK, lane * step < nb && S.w_pref[lane * step] <= r0));
              const uint32_t base = (c - 1) * step;  // w_pref[0] = 0 <= r0, so c >= 1
              const uint32_t b0 =
                  base + __popc(__ballot_sync(FULL_MASK, (uint32_t)lane < step && base + lane < nb &&
                                                             S.w_pref[base + lane] <= r0)) - 1;
              const uint32_t e = b0 + 1 + lane;  // boundary after bin b0 + lane
              const uint32_t tt = e <= nb ? S.w_pref[e] - r0 : 32u;
              const uint32_t bounds = __reduce_or_sync(FULL_MASK, tt < 32u ? 1u << tt : 0u);
              if (t < ncols) {
                const uint32_t b = b0 + __popc(bounds & ((2u << lane) - 1u));
                q = S.w_start[b] + (r0 + lane - S.w_pref[b]);
              }
            }
            const uint32_t rs = k % RAW;
            ok = ok && wait_or_abort(&S.rawfree[rs], ((k / RAW) & 1) ^ 1, abort_flag, T.wait_limit);
            if (ok && t < ncols) {
              __nv_bfloat16* dh = Raw + rs * 2 * OPB;
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&S.rid[rs][t])), "l"(ids + q)
                           : "memory");
              load_row<KP>(dh, dh + OPB, t, X + (size_t)q * P.dpad, P.dpad);
            }
            cp_async_arrive(&S.rawfull[rs]);
            if (t == 0) {
              uint32_t hcr = 0, hq = 0;
              if (w_hj >= 0) {
                const uint32_t hr0 = S.w_pref[w_hj], hr1 = S.w_pref[w_hj + 1];
                const uint32_t lo = max(hr0, pos), hi = min(hr1, pos + ncols);
                if (lo < hi) {
                  hcr = (lo - pos) | ((hi - pos) << 8);
                  hq = S.w_start[w_hj] + (lo - hr0);
                }
              }
              if (ok) S.slot[rs] = TcSlot{ncols, flags, hcr, hq, useq % NUNIT};
              mbar_arrive(&S.rawfull[rs]);
            }
            flags = 0;
          }
        }
        ++useq;
      }
      // stop marker: the next slot, with no rows
      const uint32_t rs = k % RAW;
      ok = wait_or_abort(&S.rawfree[rs], ((k / RAW) & 1) ^ 1, abort_flag, T.wait_limit);
      if (t == 0) {
        if (ok) S.slot[rs].flags = FLAG_END;
        mbar_arrive(&S.rawfull[rs]);
      }
      cp_async_arrive(&S.rawfull[rs]);
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
      // ============================ converters (K <= 32): thread c, row c of every tile
      const uint32_t c = (uint32_t)tid - NLOAD;
      uint32_t useq = 0;
      unsigned long long n_tiles = 0, n_cells = 0;
      uint32_t a0 = 0, na = 0, ng = 0, inst = 0;
      TcBound tb = T.b;
      float ra = 0.f;  // bound of the unit's largest |a|
      long long pw_sfree = 0, pw_raw = 0;
      const long long p_start = T.prof ? clock64() : 0;
      for (uint32_t tile = 0;; ++tile) {
        const uint32_t rs = tile % RAW, st = tile % NS, ms = tile % NM;
        const long long c0 = T.prof ? clock64() : 0;
        if (!__all_sync(FULL_MASK, wait_or_abort(&S.rawfull[rs], (tile / RAW) & 1, abort_flag, T.wait_limit))) break;
        const long long c1 = T.prof ? clock64() : 0;
        const TcSlot L = S.slot[rs];
        // the stage and metadata slot this tile goes to
        {
          const bool ok = wait_or_abort(&S.bfree[st], ((tile / NS) & 1) ^ 1, abort_flag, T.wait_limit) &&
                          wait_or_abort(&S.mfree[ms], ((tile / NM) & 1) ^ 1, abort_flag, T.wait_limit);
          if (!__all_sync(FULL_MASK, ok)) break;
        }
        if (T.prof) {
          pw_raw += c1 - c0;
          pw_sfree += clock64() - c1;
        }
        if (L.flags & FLAG_END) {
          if (c == 0) S.meta[ms].flags = FLAG_END;
          mbar_arrive(&S.full[st]);
          break;
        }
        if (L.flags & FLAG_FIRST) {
          // ---- a new unit: its home rows, once the MMAs are done with the last unit's
          const TcUnit& W = S.units[L.unit];
          const float* X = W.X;
          a0 = W.a0, na = W.na, ng = W.ng, inst = W.inst;
          tb = W.tb;
          float* ca = S.cadd[useq & 1][0];
          if (c < KP) {
            const float x = c < P.d ? X[(size_t)a0 * P.dpad + c] : 0.f;
            ca[c] = c == P.d + 1 ? 1.f : -x;
            S.cadd[useq & 1][1][c] = c == P.d ? 1.f : 2.f * x;
          }
          if (c == 0) S.ra2[(useq + 2) & 3] = 0;  // last read two units ago
          mbar_arrive(&S.ubar);
          bool ok = wait_or_abort(&S.ubar, 0, abort_flag, T.wait_limit);  // first of its two phases a unit
          if (ok && useq > 0) ok = wait_or_abort(&S.afree, (useq - 1) & 1, abort_flag, T.wait_limit);
          if (!__all_sync(FULL_MASK, ok)) break;
          float m = 0.f;
          for (uint32_t g = 0; g < ng; ++g) {
            const uint32_t r = g * TM + c;
            if (r < na) {
              const float4* xr = reinterpret_cast<const float4*>(X + (size_t)(a0 + r) * P.dpad);
              float4 f[KP / 4];
#pragma unroll
              for (int q = 0; q < KP / 4; ++q) f[q] = 4u * q < P.dpad ? xr[q] : make_float4(0.f, 0.f, 0.f, 0.f);
              auto block = [&](int kb, float (&x)[8]) {
                x[0] = f[2 * kb].x, x[1] = f[2 * kb].y, x[2] = f[2 * kb].z, x[3] = f[2 * kb].w;
                x[4] = f[2 * kb + 1].x, x[5] = f[2 * kb + 1].y, x[6] = f[2 * kb + 1].z, x[7] = f[2 * kb + 1].w;
              };
              __nv_bfloat16 *ah = Ahi + g * OPB, *al = Alo + g * OPB;
              const float nrm = conv_row<KP>(block, ah, al, c, ca, 1.f, P.d);
              patch_col<KP>(ah, al, c, P.d, nrm);
              m = fmaxf(m, nrm);
            }
          }
#pragma unroll
          for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL_MASK, m, o));
          if (lane == 0) atomicMax(&S.ra2[useq & 3], __float_as_uint(m));
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_arrive(&S.afull);
          mbar_arrive(&S.ubar);
          if (!__all_sync(FULL_MASK, wait_or_abort(&S.ubar, 1, abort_flag, T.wait_limit))) break;
          ra = norm_bound(tb, __uint_as_float(*(volatile uint32_t*)&S.ra2[useq & 3]));
          ++useq;
        }
        __nv_bfloat16 *bh = Bhi + st * OPB, *bl = Blo + st * OPB;
        if (c < L.ncols) {
          const __nv_bfloat16* sh = Raw + rs * 2 * OPB;
          auto block = [&](int kb, float (&x)[8]) {
            unpack8(sh, sh + OPB, chunk_off<KP>(c, kb), 8u * kb < P.d, 8u * kb + 4 < P.d, x);
          };
          S.qid[ms][c] = S.rid[rs][c];
          const float nq2 =
              conv_row<KP>(block, bh, bl, c, S.cadd[(useq - 1) & 1][1], -2.f, P.d) * 0.25f;
          float tcol = 0.f, dl = 0.f;
          if (!column_threshold(tb, ra, nq2, &tcol, &dl)) {
            tcol = 1e30f;   // every row of this column becomes a candidate ...
            dl = INFINITY;  // ... and none is accepted without the FP64 check
          }
          patch_col<KP>(bh, bl, c, P.d + 1, nq2 - tcol);
          S.dlt[ms][c] = dl;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.rawfree[rs]);
        if (c == 0) {
          n_tiles += 1;
          n_cells += (unsigned long long)na * L.ncols;
        }
        if (c == 0) S.meta[ms] = TileMeta{a0, na, L.flags, ng, inst, L.ncols, L.hcr, L.hq};
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(&S.full[st]);
      }
      if (c == 0 && n_tiles) {
        atomicAdd(&T.ctr->tiles, n_tiles);
        atomicAdd(&T.ctr->cells, n_cells);
      }
      if (c == 0 && T.prof) {
        atomicAdd(&T.ctr->prof[0], (unsigned long long)pw_sfree);
        atomicAdd(&T.ctr->prof[14], (unsigned long long)pw_raw);
        atomicAdd(&T.ctr->prof[1], (unsigned long long)(clock64() - p_start));
      }
    }
    } else {
    // ============================ producers (NPW warps, two threads per row)
    // Thread (prow, half): row prow = 32 * (warp % 4) + lane of every operand
    // tile, K blocks kb = 2j + half with half = warp / 4, so the lanes of a
    // warp take the same branches; the two halves of a row norm meet in
    // S.npart (one bar.sync).  Every branch that
    // leads to bar.sync is taken on a value all producer threads hold in
    // registers or read from shared memory after the same bar.sync; barrier
    // waits are done by thread 0 and broadcast through S.pflag[2] (two slots:
    // a thread is at most one bar.sync behind thread 0).
    const uint32_t prow = ((uint32_t)(warp & 3) << 5) | (uint32_t)lane, half = (uint32_t)warp >> 2;
    uint32_t xpar = 0;  // parity of the next S.npart exchange
    // row norm from this thread's part and the other half's (all producer
    // threads call it together)
    auto row_norm = [&](float part) {
      S.npart[xpar][half][prow] = part;
      prod_sync();
      const float o = S.npart[xpar][half ^ 1][prow];
      xpar ^= 1;
      return half == 0 ? part + o : o + part;  // the same sum, in the same order, in both threads
    };
    uint32_t tile = 0, issued = 0, unit_k = 0, pf = 0;
    unsigned long long n_tiles = 0, n_cells = 0;
    long long pw_sfree = 0, pc_unit = 0, pc_win = 0, pc_conv = 0, pc_ldw = 0;
    long long pc_adv = 0, pc_bar = 0, pc_p1 = 0, pc_p2 = 0, pc_fin = 0;
    uint32_t wgen = 0;  // window refills so far (tags S.w_home)
    // tiles in flight: RAW landing slots, or (rows landing in the B stages
    // themselves) NS - 1, so that issuing tile t + LA - 1 waits only on tiles
    // before t
    constexpr uint32_t LA = RAW > 0 ? RAW : (NS - 1 < 3 ? NS - 1 : 3);
    const long long p_start = T.prof ? clock64() : 0;
    // bounded wait until stage k % NS may take tile k (bfree and mfree, see the barrier table)
    auto stage_free = [&](uint32_t k) -> bool {
      const uint32_t st = k % NS, par = ((k / NS) & 1) ^ 1;
      return wait_or_abort(&S.mfree[st], par, abort_flag, T.wait_limit) &&
             wait_or_abort(&S.bfree[st], par, abort_flag, T.wait_limit);
    };
    auto end_marker = [&]() {  // last tile slot: tells the MMA warps and the epilogue to stop
      const uint32_t st = tile % NS;
      if (tid == 0) {
        stage_free(tile);
        S.meta[st].flags = FLAG_END;
      }
      prod_sync();
      mbar_arrive(&S.full[st]);
    };
    for (;;) {
      const long long cu0 = T.prof ? clock64() : 0;
      const uint32_t slot = pf++ & 1;
      if (tid == 0) {
        // claim index -> unit: units deferred by the last ring pass first,
        // then the list from main_start (the identity outside ring mode)
        const unsigned long long t = atomicAdd(&T.ctr->next_unit, 1ull);
        const unsigned long long uu = t < T.n_def_in ? (unsigned long long)T.def_in[t] : T.main_start + (t - T.n_def_in);
        S.unit = uu;
        bool go = (T.claim_cap == 0 || t < T.claim_cap) && uu < T.n_units && !*abort_flag;
        if (go && P.ring && *(volatile unsigned long long*)&P.ctr->stop) {  // the ring filled: leave it for the next pass
          const RingCtx rc{P.pair_tags, P.deferred, P.def_out, &P.ctr->def_n, &P.ctr->stop};
          ring_defer(&rc, P.tag_base_tc + (uint32_t)uu);
          go = false;
        }
        if (go && unit_k > 0) go = wait_or_abort(&S.afree, (unit_k - 1) & 1, abort_flag, T.wait_limit);  // A no longer read
        S.pflag[slot] = go ? 1u : 0u;
      }
      prod_sync();
      if (!S.pflag[slot]) {
        end_marker();
        break;
      }
      const unsigned long long u = S.unit;
      const Unit U = T.units[u];
      // the unit's instance: its arrays and bound constants (fused batch
      // joins), or the launch's own
      const float* X = (const float*)P.xs;
      const uint32_t *bstart = P.bstart, *nbr = P.nbr, *ids = P.ids;
      TcBound tb = T.b;
      uint32_t inst = 0;
      if (T.unit_inst) {
        inst = T.unit_inst[u];
        const InstDesc& I = P.insts[inst];
        X = (const float*)I.xs;
        bstart = I.bstart;
        nbr = I.nbr;
        ids = I.ids;
        tb = I.tcb;
      }
      if (P.ring) inst = P.tag_base_tc + (uint32_t)u;  // the ring's tag of this unit's pairs
      const uint32_t hs = bstart[U.h], he = bstart[U.h + 1];
      const uint32_t a0 = hs + U.chunk * (TM * G);
      const uint32_t na = min((uint32_t)(TM * G), he - a0);
      const uint32_t ng = (na + TM - 1) / TM;
      if (tid < (int)P.dpad) {
        const float c = X[(size_t)a0 * P.dpad + tid];
        S.cadd_a[tid] = -c;
        S.cadd_b[tid] = 2.f * c;
      }
      if (tid == 0) S.ra2max = 0;
      prod_sync();
      {
        for (uint32_t g = 0; g < ng; ++g) {
          const uint32_t r = g * TM + prow;
          if (r < na) load_half<KP>(Ahi + g * OPB, Alo + g * OPB, prow, half, X + (size_t)(a0 + r) * P.dpad, P.dpad);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        float m = 0.f;
        for (uint32_t g = 0; g < ng; ++g) {
          const bool ok = g * TM + prow < na;
          __nv_bfloat16 *ah = Ahi + g * OPB, *al = Alo + g * OPB;
          const float part = conv_pass1<KP>(ah, al, ah, al, prow, half, ok, S.cadd_a, 1.f, P.d, 0.f, 1.f);
          const float nrm = row_norm(part);
          if (ok && ((P.d >> 3) & 1u) == half) patch_col<KP>(ah, al, prow, P.d, nrm);
          m = fmaxf(m, ok ? nrm : 0.f);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL_MASK, m, o));
        if (lane == 0) atomicMax(&S.ra2max, __float_as_uint(m));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&S.afull);
      prod_sync();
      const float ra2max = __uint_as_float(S.ra2max);
      if (T.prof) pc_unit += clock64() - cu0;

      // ---- candidate tiles of this unit: window of up to WIN neighbour bins
      // (state uniform, in registers); the rows of up to LA tiles are in
      // flight (cp.async, one group per tile) while the oldest is converted
      uint32_t seg_next = U.s0, w_nb = 0, w_pos = 0, w_total = 0;
      uint32_t pq = 0;  // (columns | last << 8) of the tiles in flight, 9 bits each, oldest lowest
      int w_hj = -1;    // index of the home bin in the window, or -1
      // 1: tile issued; 2: abort
      auto advance = [&]() -> int {
        while (w_pos >= w_total) {  // the caller checked that the unit has more tiles
          const long long cw0 = T.prof ? clock64() : 0;
          const uint32_t nb = min((uint32_t)WIN, U.s1 - seg_next);
          uint32_t st0 = 0, sz0 = 0, bn = 0xffffffffu;
          if ((uint32_t)tid < nb) unit_bin(U, TM * G, nbr, bstart, seg_next + tid, &bn, &st0, &sz0);
          const uint32_t incl = warp_scan_incl(sz0);
          if (lane == 31) S.scan_ws[warp] = incl;
          prod_sync();
          uint32_t wp = 0;
          for (int w = 0; w < warp; ++w) wp += S.scan_ws[w];
          ++wgen;
          if ((uint32_t)tid < nb) {
            S.w_start[tid] = st0;
            S.w_pref[tid + 1] = wp + incl;
            if (bn == U.h) S.w_home = ((wgen & 0xffffffu) << 8) | (uint32_t)tid;
          }
          if (tid == 0) S.w_pref[0] = 0;
          prod_sync();
          {
            const uint32_t wh = S.w_home;
            w_hj = (wh >> 8) == (wgen & 0xffffffu) ? (int)(wh & 255u) : -1;
          }
          w_nb = nb;
          w_pos = 0;
          w_total = S.w_pref[nb];
          seg_next += nb;
          if (T.prof) pc_win += clock64() - cw0;
        }
        const long long ca0 = T.prof ? clock64() : 0;
        const uint32_t ncols = min((uint32_t)TN, w_total - w_pos);
        const bool last = (w_pos + TN >= w_total) && (seg_next >= U.s1);
        // row of candidate rank w_pos + prow: the warp finds the bin of its
        // first rank (two 32-way probes of the window prefix), then each lane
        // counts the bin boundaries among the next 32 ranks
        uint32_t q = 0xffffffffu;
        {
          const uint32_t r0 = w_pos + (prow & ~31u);
          const uint32_t step = (w_nb + 31) >> 5;
          const uint32_t c = __popc(__ballot_sync(FULL_MASK, lane * step < w_nb && S.w_pref[lane * step] <= r0));
          const uint32_t base = (c - 1) * step;  // w_pref[0] = 0 <= r0, so c >= 1
          const uint32_t b0 =
              base + __popc(__ballot_sync(FULL_MASK, (uint32_t)lane < step && base + lane < w_nb &&
                                                         S.w_pref[base + lane] <= r0)) - 1;
          const uint32_t e = b0 + 1 + lane;  // boundary after bin b0 + lane
          const uint32_t t = e <= w_nb ? S.w_pref[e] - r0 : 32u;
          const uint32_t bounds = __reduce_or_sync(FULL_MASK, t < 32u ? 1u << t : 0u);
          if (prow < ncols) {
            const uint32_t b = b0 + __popc(bounds & ((2u << lane) - 1u));
            q = S.w_start[b] + (r0 + lane - S.w_pref[b]);
          }
        }
        __nv_bfloat16 *dh, *dl;  // landing slot of the raw rows
        uint32_t* iddst;  // candidate ids
        if (RAW > 0) {
          // own-row slots, last read by this thread when it converted tile
          // issued - RAW: no wait needed
          const uint32_t rs = issued % (RAW > 0 ? RAW : 1);
          dh = Raw + rs * 2 * OPB;
          dl = dh + OPB;
          iddst = S.rid[rs];
        } else {
          const uint32_t st = issued % NS;
          const uint32_t sl = pf++ & 1;
          if (tid == 0) {
            const long long c0 = T.prof ? clock64() : 0;
            S.pflag[sl] = stage_free(issued) ? 1u : 0u;
            if (T.prof) pw_sfree += clock64() - c0;
          }
          prod_sync();
          if (!S.pflag[sl]) return 2;
          dh = Bhi + st * OPB;
          dl = Blo + st * OPB;
          iddst = S.qid[st];
        }
        if (prow < ncols) {
          if (half == 0)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&iddst[prow])), "l"(ids + q)
                         : "memory");
          load_half<KP>(dh, dl, prow, half, X + (size_t)q * P.dpad, P.dpad);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        pq |= (ncols | (last ? 0x100u : 0u)) << (9 * (issued - tile));  // uniform queue of (columns, last)
        if (tid == 0) {
          uint32_t hcr = 0, hq = 0;
          if (w_hj >= 0) {
            const uint32_t hr0 = S.w_pref[w_hj], hr1 = S.w_pref[w_hj + 1];
            const uint32_t lo = max(hr0, w_pos) - w_pos, hi = min(hr1, w_pos + ncols) - w_pos;
            if (max(hr0, w_pos) < min(hr1, w_pos + ncols)) {
              hcr = lo | (hi << 8);
              hq = S.w_start[w_hj] + (w_pos + lo - hr0);
            }
          }
          S.hx[issued & 3][0] = hcr;
          S.hx[issued & 3][1] = hq;
        }
        w_pos += TN;
        ++issued;
        if (T.prof) pc_adv += clock64() - ca0;
        return 1;
      };

      bool first = true, aborted = false;
      for (;;) {
        while (issued < tile + LA && (w_pos < w_total || seg_next < U.s1)) {
          if (advance() == 2) {
            aborted = true;
            break;
          }
        }
        if (aborted || issued == tile) break;
        const long long cc0 = T.prof ? clock64() : 0;
        switch (issued - tile - 1) {  // groups newer than this tile's
          case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
          case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
          default: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        }
        if (T.prof) pc_ldw += clock64() - cc0;
        const uint32_t st = tile % NS;
        const uint32_t ncols = pq & 0xffu;
        const bool last = (pq & 0x100u) != 0u;
        pq >>= 9;
        __nv_bfloat16* bh = Bhi + st * OPB;
        __nv_bfloat16* bl = Blo + st * OPB;
        const __nv_bfloat16* sh = bh;  // raw rows: in place, or in the landing slot
        const __nv_bfloat16* sl = bl;
        if (RAW > 0) {
          const uint32_t rs = tile % (RAW > 0 ? RAW : 1);
          const uint32_t id = S.rid[rs][prow];  // own row's id (half 0 copied it)
          sh = Raw + rs * 2 * OPB;
          sl = sh + OPB;
          const uint32_t fl = pf++ & 1;
          const long long cb0 = T.prof ? clock64() : 0;
          if (tid == 0) {
            const long long c0 = T.prof ? clock64() : 0;
            S.pflag[fl] = stage_free(tile) ? 1u : 0u;
            if (T.prof) pw_sfree += clock64() - c0;
          }
          prod_sync();
          if (T.prof) pc_bar += clock64() - cb0;
          if (!S.pflag[fl]) {
            aborted = true;
            break;
          }
          if (half == 0) S.qid[st][prow] = id;
        }
        const bool ok = prow < ncols;
        const long long cp0 = T.prof ? clock64() : 0;
        const float part = conv_pass1<KP>(sh, sl, bh, bl, prow, half, ok, S.cadd_b, -2.f, P.d, 1.f, 0.f);
        const float nq2 = row_norm(part) * 0.25f;
        float tcol = 0.f, dl = 0.f;
        if (ok && !column_threshold(tb, norm_bound(tb, ra2max), nq2, &tcol, &dl)) {
          tcol = 1e30f;   // every row of this column becomes a candidate ...
          dl = INFINITY;  // ... and none is accepted without the FP64 check
        }
        const long long cp1 = T.prof ? clock64() : 0;
        if (ok && (((P.d + 1) >> 3) & 1u) == half) patch_col<KP>(bh, bl, prow, P.d + 1, nq2 - tcol);
        const long long cp2 = T.prof ? clock64() : 0;
        if (T.prof) {
          pc_p1 += cp1 - cp0;
          pc_p2 += cp2 - cp1;
        }
        if (half == 0) S.dlt[st][prow] = dl;
        if (tid == 0) {
          S.meta[st] = TileMeta{a0, na, (first ? FLAG_FIRST : 0u) | (last ? FLAG_LAST : 0u), ng, inst, ncols,
                                S.hx[tile & 3][0], S.hx[tile & 3][1]};
          n_tiles += 1;
          n_cells += (unsigned long long)na * ncols;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(&S.full[st]);
        if (T.prof) {
          const long long ce = clock64();
          pc_fin += ce - cp2;
          pc_conv += ce - cc0;
        }
        first = false;
        ++tile;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      ++unit_k;
      if (aborted) {
        end_marker();
        break;
      }
    }
    if (tid == 0 && n_tiles) {
      atomicAdd(&T.ctr->tiles, n_tiles);
      atomicAdd(&T.ctr->cells, n_cells);
    }
    if (tid == 0 && T.prof) {
      atomicAdd(&T.ctr->prof[0], (unsigned long long)pw_sfree);
      atomicAdd(&T.ctr->prof[1], (unsigned long long)(clock64() - p_start));
      atomicAdd(&T.ctr->prof[7], (unsigned long long)pc_unit);
      atomicAdd(&T.ctr->prof[8], (unsigned long long)pc_win);
      atomicAdd(&T.ctr->prof[9], (unsigned long long)pc_conv);
      atomicAdd(&T.ctr->prof[14], (unsigned long long)pc_ldw);
      atomicAdd(&T.ctr->prof[16], (unsigned long long)pc_adv);
      atomicAdd(&T.ctr->prof[17], (unsigned long long)pc_bar);
      atomicAdd(&T.ctr->prof[18], (unsigned long long)pc_p1);
      atomicAdd(&T.ctr->prof[19], (unsigned long long)pc_p2);
      atomicAdd(&T.ctr->prof[20], (unsigned long long)pc_fin);
    }
    }  // two threads a row
  } else if (warp >= MMA_WARP) {
    // ============================ MMA issuers
    // B tiles come in stage order; each is multiplied with the unit's ng home
    // chunks into a TMEM accumulator (MMA tile counter mt), warp w issuing
    // every mt = w mod NMMA into accumulator w.
    const uint32_t me = (uint32_t)(warp - MMA_WARP), b = me;
    static_assert(NMMA == NACC, "an accumulator a warp");
    if (lane == 0) {
      const uint64_t desc_a = chunk_desc<KP>(smem_u32(Ahi)), desc_b = chunk_desc<KP>(smem_u32(Bhi));
      uint32_t tile = 0, mt = 0, unit_k = 0;
      uint32_t use = 0;  // uses of accumulator me so far
      uint32_t last_par = 0;
      long long mw_full = 0, mw_dfree = 0;
      const long long m_start = T.prof ? clock64() : 0;
      for (;;) {
        const uint32_t st = tile % NS, ms = tile % NM;
        const long long c0 = T.prof ? clock64() : 0;
        const bool fok = wait_or_abort(&S.full[st], (tile / NS) & 1, abort_flag, T.wait_limit);
        if (T.prof) mw_full += clock64() - c0;
        if (!fok) break;
        const uint4 m4 = *reinterpret_cast<const uint4*>(&S.meta[ms]);
        const uint32_t flags = m4.z, ng = m4.w;
        if (flags & FLAG_END) {
          // wake the epilogue group on its next accumulator, but only once
          // the group has taken the accumulator's previous use: an arrival
          // before that would complete a second phase of dfull[b] under a
          // warp still waiting for the first (parity aliasing)
          if (wait_or_abort(&S.dfree[b], (use & 1) ^ 1, abort_flag, T.wait_limit)) {
            S.acc[b].end = 1;
            mbar_arrive_n(&S.dfull[b], 2);
          }
          break;
        }
        bool ok = true;
        if (flags & FLAG_FIRST) ok = wait_or_abort(&S.afull, unit_k & 1, abort_flag, T.wait_limit);
        if (!ok) break;
        // descriptors differ from the buffers' first ones by address / 16 alone
        const uint64_t dbh = desc_b + st * (OPB * 2 / 16), dbl = dbh + NS * (OPB * 2 / 16);
        constexpr uint32_t idesc = umma_idesc(TM, TN);
        for (uint32_t g = (me - mt) % NMMA; g < ng; g += NMMA) {
          const long long c1 = T.prof ? clock64() : 0;
          const uint32_t par = use & 1;
          ok = wait_or_abort(&S.dfree[b], par ^ 1, abort_flag, T.wait_limit);
          if (T.prof) mw_dfree += clock64() - c1;
          if (!ok) break;
          ++use;
          if (T.stall_test) continue;  // failure-detection test: never signal, let the waits run out
          asm volatile("tcgen05.fence::after_thread_sync;");
          S.acc[b] = TcAcc{ms, g, 0u};
          mbar_arrive(&S.dfull[b]);  // releases the metadata; the commit below completes the phase
          const uint64_t dah = desc_a + g * (OPB * 2 / 16), dal = dah + G * (OPB * 2 / 16);
          const uint32_t dt = tbase + b * TN;
#pragma unroll
          for (int ks = 0; ks < KP / 16; ++ks) {
            const uint32_t o = ks * chunk_kstep<KP>();
            mma_bf16(dt, dah + o, dbh + o, idesc, ks > 0 ? 1u : 0u);
            mma_bf16(dt, dah + o, dbl + o, idesc, 1u);
            mma_bf16(dt, dal + o, dbh + o, idesc, 1u);
          }
          tc_commit(&S.dfull[b]);
          last_par = par;
        }
        if (!ok) break;
        mt += ng;
        if (!T.stall_test) tc_commit(&S.bfree[st]);
        if ((flags & FLAG_LAST) && !T.stall_test) {
          tc_commit(&S.afree);
          ++unit_k;
        }
        ++tile;
      }
      if (T.prof) {
        atomicAdd(&T.ctr->prof[2], (unsigned long long)mw_full);
        atomicAdd(&T.ctr->prof[3], (unsigned long long)mw_dfree);
        atomicAdd(&T.ctr->prof[4], (unsigned long long)(clock64() - m_start));
        if (me == 0) atomicAdd(&T.ctr->prof[12], (unsigned long long)mt);
      }
      // an aborting CTA may still have MMAs in flight: wait (bounded) for the
      // last committed tile, MMAs complete in issue order
      if (*abort_flag && use > 0 && !T.stall_test) {
        volatile uint32_t no_abort = 0;
        wait_or_abort(&S.dfull[b], last_par, &no_abort, T.wait_limit);
      }
    }
    __syncwarp();
  } else if (warp >= EPI0 && warp < EPI0 + NEPI) {
    // ============================ epilogue (NEPI warps)
    // Group e of EG = NEPI / 4 drains accumulators e, e + EG, ... in turn; its
    // warp w reads TMEM lane quarter w % 4 (the hardware's access rule), all
    // 128 columns in blocks of 32.  With all 16 warps on one accumulator the
    // waits, the metadata and the slowest block of every accumulator were on
    // every warp's path (2,550 cycles an accumulator on the 5M x 18 join);
    // groups overlap them.  Two groups of 8 with two accumulators each measured
    // 73.2 ms there (T = 66), four of 4 with one each 70.6.
    constexpr uint32_t EG = NEPI / 4;
    const uint32_t grp = (uint32_t)(warp - EPI0) / 4;
    const uint32_t quarter = warp & 3;
    PairStage ps{pstage + (warp - EPI0) * PSTAGE, 0, 0, P.pairs_ij != 0};
    PairStage bs{pstage + (NEPI + warp - EPI0) * PSTAGE, 0};
    const RingCtx rcp_{P.pair_tags, P.deferred, P.def_out, &P.ctr->def_n, &P.ctr->stop};
    const RingCtx rcb_{P.band_tags, P.deferred, P.def_out, &P.ctr->def_n, &P.ctr->stop};
    const RingCtx* rcp = P.ring ? &rcp_ : nullptr;
    const RingCtx* rcb = P.ring ? &rcb_ : nullptr;
    long long ew_dfull = 0;
    const long long e_start = T.prof ? clock64() : 0;
    for (uint32_t n = 0;; ++n) {
      const uint32_t b = grp + EG * (n % (NACC / EG));
      // all lanes wait; the outcome is made warp-uniform (tcgen05.ld is .sync.aligned)
      const long long cw = T.prof ? clock64() : 0;
      const bool ok = __all_sync(FULL_MASK, wait_or_abort(&S.dfull[b], (n / (NACC / EG)) & 1, abort_flag, T.wait_limit));
      if (T.prof) ew_dfull += clock64() - cw;
      if (!ok) break;
      const TcAcc A = S.acc[b];
      if (A.end) break;  // the same in all lanes
      const TileMeta M = S.meta[A.ms];
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t row0 = A.g * TM + quarter * 32, row = row0 + lane;  // row within the unit
      if (row0 < M.na) {
        const bool row_ok = row < M.na;
        const uint32_t a_sorted = M.a0 + row;
        const uint32_t* ids = P.insts ? P.insts[M.inst].ids : P.ids;
        const uint32_t ia = row_ok ? ids[a_sorted] : 0u;
        // home bin: a pair (a, q) of two home rows is kept only for a < q
        // (sorted positions); the home rows of this tile are the columns
        // [hlo, hhi), column c at position hq + c - hlo: those below `drop`
        // have q <= a
        const uint32_t hlo = M.hcr & 255u, hhi = M.hcr >> 8;
        const uint32_t drop = (hlo < hhi && a_sorted >= M.hq) ? min(hhi, hlo + min(a_sorted - M.hq, 255u) + 1) : 0u;
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < M.ncols; c0 += 32) {
          uint32_t v[32];
          tmem_ld32_nowait(tbase + b * TN + ((quarter * 32u) << 16) + c0, v);
          tmem_wait();
          // with the last block in registers the accumulator can be refilled
          // (5M x 18 77.0 -> 75.3 ms, 100k x 18 1.55 -> 1.47)
          if (c0 + 32 >= M.ncols) {
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.dfree[b]);
          }
          // D' < 0 marks a candidate.  Three blocks of four hold none: a tree
          // of three-input ORs over the signs (16 operations) finds those;
          // extracting the 32 sign bits takes a funnel shift each, on a pipe
          // at half the issue rate.
          {
            uint32_t o = v[0] | v[1];
#pragma unroll
            for (int j = 2; j < 32; j += 2) o |= v[j] | v[j + 1];
            if (!__any_sync(FULL_MASK, (int)o < 0)) continue;
          }
          // sign bits, value j at bit j, in four independent chains of 8
          auto signs = [&]() {
            uint32_t m0 = 0, m1 = 0, m2 = 0, m3 = 0;
#pragma unroll
            for (int j = 7; j >= 0; --j) {
              m0 = __funnelshift_l(v[j], m0, 1);
              m1 = __funnelshift_l(v[8 + j], m1, 1);
              m2 = __funnelshift_l(v[16 + j], m2, 1);
              m3 = __funnelshift_l(v[24 + j], m3, 1);
            }
            return m0 | (m1 << 8) | (m2 << 16) | (m3 << 24);
          };
          uint32_t m = signs();
          const uint32_t nvalid = M.ncols - c0;
          if (nvalid < 32) m &= (1u << nvalid) - 1u;
          if (!row_ok) m = 0;
          if (drop > c0 && hlo < c0 + 32) {
            const uint32_t e0 = max(hlo, c0) - c0, e1 = min(drop, c0 + 32) - c0;
            if (e0 < e1) m &= ~((e1 >= 32 ? FULL_MASK : ((1u << e1) - 1u)) & ~((1u << e0) - 1u));
          }
          const float* dlt = &S.dlt[A.ms][c0];
          const uint32_t* qid = &S.qid[A.ms][c0];
          if (!__any_sync(FULL_MASK, (m & (m - 1)) != 0)) {
            // at most one candidate a lane (most blocks that hold any)
            if (!__any_sync(FULL_MASK, m != 0)) continue;
            bool acc = false, band = false;
            unsigned long long pr = 0;
            if (m) {
              const int j = __ffs(m) - 1;
              const uint32_t iq = qid[j];
              acc = pick32(v, j) <= -dlt[j];
              band = !acc;  // decided later in FP64
              pr = ((unsigned long long)min(ia, iq) << 32) | max(ia, iq);
            }
            stage_one(ps, acc, pr, &P.ctr->pairs, P.pairs, P.cap, P.inst_pairs, M.inst, rcp);
            stage_one(bs, band, pr, &P.ctr->band_n, P.band_list, P.band_cap, nullptr, M.inst, rcb);
            continue;
          }
          // D' + dlt < 0: accepted (an infinite dlt accepts nothing)
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(dlt + j);
            v[j] = __float_as_uint(__uint_as_float(v[j]) + d4.x);
            v[j + 1] = __float_as_uint(__uint_as_float(v[j + 1]) + d4.y);
            v[j + 2] = __float_as_uint(__uint_as_float(v[j + 2]) + d4.z);
            v[j + 3] = __float_as_uint(__uint_as_float(v[j + 3]) + d4.w);
          }
          const uint32_t acc_bits = m & signs();
          auto emit = [&](PairStage& stg, uint32_t bits, unsigned long long* counter, unsigned long long* list,
                          unsigned long long lcap, unsigned long long* ip, const RingCtx* rc) {
            stage_pairs(
                stg, __popc(bits),
                [&](uint32_t) {
                  const int j = __ffs(bits) - 1;
                  bits &= bits - 1;
                  const uint32_t iq = qid[j];
                  return ((unsigned long long)min(ia, iq) << 32) | max(ia, iq);
                },
                counter, list, lcap, ip, M.inst, rc);
          };
          emit(ps, acc_bits, &P.ctr->pairs, P.pairs, P.cap, P.inst_pairs, rcp);
          // the band is decided later in FP64
          if (__any_sync(FULL_MASK, m != acc_bits))
            emit(bs, m & ~acc_bits, &P.ctr->band_n, P.band_list, P.band_cap, nullptr, rcb);
        }
      }
      __syncwarp();
      if (lane == 0) {
        if (row0 >= M.na) mbar_arrive(&S.dfree[b]);
        mbar_arrive_n(&S.mfree[A.ms], 12u / M.ng);  // the tile served one of its home chunks
      }
    }
    stage_flush(ps, &P.ctr->pairs, P.pairs, P.cap, P.inst_pairs, rcp);
    stage_flush(bs, &P.ctr->band_n, P.band_list, P.band_cap, nullptr, rcb);
    if (T.prof && lane == 0) {
      atomicAdd(&T.ctr->prof[5], (unsigned long long)ew_dfull);
      atomicAdd(&T.ctr->prof[6], (unsigned long long)(clock64() - e_start));
    }
  }
  // all roles meet here before tensor memory is released
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase));
  if (tid == 0 && S.abort_flag) atomicExch(&P.ctr->error, 1ull);
}

// Stages and home chunks per KP within about 200 KB of operands: one CTA per
// SM (512 TMEM columns).
template <int KP>
struct TcShape {
  static constexpr int G = KP <= 32 ? 4 : (KP <= 64 ? 2 : 1);
  static constexpr int NS = KP <= 32 ? 4 : (KP <= 96 ? 3 : 2);
  // separate landing slots where they fit: four for K <= 32 (tiles on their
  // way to the converters), three for K = 48
  static constexpr int RAW = KP <= 32 ? 4 : (KP <= 48 ? 3 : 0);
  // short rows: many tiles, pairs and hits per converted row -> more epilogue
  // warps (16: 72 registers a thread); long rows: 8 (96 registers)
  static constexpr int NEPI = KP <= 48 ? 16 : 8;
};

template <int KP>
void launch_tc(mistic_handle_s* h, const JoinParams& P, const TcParams& T) {
  constexpr int NS = TcShape<KP>::NS, G = TcShape<KP>::G, RAW = TcShape<KP>::RAW, NEPI = TcShape<KP>::NEPI;
  constexpr int NT = tc_threads(NEPI);
  const size_t dyn = 512 + (2 * G + 2 * NS + 2 * RAW) * (size_t)TM * KP * sizeof(__nv_bfloat16) +
                     (size_t)2 * NEPI * PSTAGE * sizeof(unsigned long long);
  MCK(cudaFuncSetAttribute(k_join_tc<KP, NS, G, RAW, NEPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  MCK(cudaFuncSetAttribute(k_join_tc<KP, NS, G, RAW, NEPI>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int per_sm = 0;
  MCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_join_tc<KP, NS, G, RAW, NEPI>, NT, dyn));
  if (per_sm < 1) throw Error(MISTIC_ERR_TOO_LARGE, "tensor-core join does not fit on an SM");
  unsigned grid = (unsigned)std::min<unsigned long long>((unsigned long long)h->sms, T.n_units);
  if (T.grid_cap) grid = std::min(grid, T.grid_cap);
  if (getenv("MISTIC_DEBUG"))
    fprintf(stderr, "[mistic] join_tc KP=%d NS=%d G=%d RAW=%d NEPI=%d dyn=%zu occupancy=%d grid=%u units=%llu\n", KP,
            NS, G, RAW, NEPI, dyn, per_sm, grid, (unsigned long long)T.n_units);
  k_join_tc<KP, NS, G, RAW, NEPI><<<grid, NT, dyn, h->stream>>>(P, T);
  launched(h, "join_tc");
}

}  // namespace

namespace join {

int tc_kp(uint32_t d) { return (int)(((d + 2) + 15) / 16 * 16); }
// Home rows per tensor-core unit: G chunks of 128 share each converted
// candidate tile, as many as fit beside the stages of one CTA's 200 KB (TcShape).
// Longer rows go to the K-chunked kernel (join_tcw.cu), 256 home rows a unit.
uint32_t tc_rows(uint32_t d) {
  const int kp = tc_kp(d);
  if (kp > 128) return 256;
  return (uint32_t)TM * (kp <= 32 ? 4 : (kp <= 64 ? 2 : 1));
}
bool tc_supported(uint32_t d) { return d >= 1 && d <= MAX_D; }

void run_tc(mistic_handle_s* h, const JoinParams& P, const TcParams& T) {
  if (T.n_units == 0) return;
  switch (tc_kp(P.d)) {
    case 16: launch_tc<16>(h, P, T); break;
    case 32: launch_tc<32>(h, P, T); break;
    case 48: launch_tc<48>(h, P, T); break;
    case 64: launch_tc<64>(h, P, T); break;
    case 80: launch_tc<80>(h, P, T); break;
    case 96: launch_tc<96>(h, P, T); break;
    case 112: launch_tc<112>(h, P, T); break;
    case 128: launch_tc<128>(h, P, T); break;
    default: run_tcw(h, P, T); break;
  }
}

}  // namespace join
}  // namespace mistic
