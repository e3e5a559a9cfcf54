// FP64-accurate complex GEMM on the bf16 tensor cores (tcgen05): the long-K contractions of
// the FP64 mode and every product of GTN_PREC_FP64E.  FP64 runs at about 1.2 TFLOP/s on this
// part, more than a thousand times below the bf16 tensor rate; this kernel trades that for
// exact integer arithmetic.
//
// Method (the fixed-point splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59
// (2012), with exact chunked accumulation):
//   * every row of the real-expanded A (and every complex row of B') is scaled by a power
//     of two so that its entries lie in (-1/2, 1/2), then written as S = 7 signed base-256
//     digits, a = sum_i d_i 2^{-8(i+1)}, |d_i| <= 128 (bf16 holds them exactly);
//   * the digit products d_i e_j of the levels l = i + j < L are summed on the tensor cores,
//     one TMEM accumulator of 64 columns per level: L = 8 (34 products) in the FP64 mode, L = 7
//     (28) in FP64E.  A level gets at most min(l + 1, 13 - l) 2^14 per real k, so the FP32 sums are
//     exact integers (<= 2^24) over 256 real k for the levels 0-3 and over 128 for the others;
//   * the epilogue warps read the levels from 4 on after every 128 k and the levels 0-3 after
//     every 256, and add them with their weights into two 64-bit integers per output (units
//     2^-72 and 2^-40): the sum over all k of the kept digit products is exact.  Its one rounding
//     is the conversion to FP64 at the end, done on the integers' bits.
// In FP64 every output is checked against the bound of an FP64 sum and, where the digits may miss it,
// summed again on the FP64 pipe (f64e_check_kernel, f64e_repair_kernel).  What is left out of the
// others (levels from L on, digits beyond the seventh) does not grow with K, unlike the
// rounding errors of FP64 fused multiply-adds.  Measured against extended precision, relative
// 2-norm, Gaussian operands: K = 65 5.7e-17 (FP64 pipe 3.7e-16), K = 5120 7.1e-17 (3.4e-15),
// rows that decay from 1 to 1e-9 along k 1.3e-16 (5.4e-16) and 1.8e-16 (4.9e-15); L = 7 about
// 3.6e-16 at every K.
// A row with an infinity, a NaN, nothing but subnormals or a magnitude beyond 2^+-450 has no digits:
// what this kernel makes of it is overwritten by f64e_repair_kernel, which looks at the rows' exponents and leaves no trace
// for a later product.
//
// Tile: 128 rows x 64 real columns (32 complex); stages of 16 real k hold all 7 planes of A
// (28 KB) and of B' (14 KB), laid out by the split so that one contiguous bulk copy loads each
// (rows of 32 bytes, SWIZZLE_32B order).  The planes of B' lie behind each other in a stage, so
// digit i of A meets the stack e_0, e_1, .. in MMAs up to 256 wide whose columns run through
// the levels from i on: 10 to 13 instructions a stage instead of 28 or 34 of width 64 (A is read
// from shared memory once per instruction, and 64-wide instructions are bound by that).  One CTA per SM
// walks over the tiles: warp 0 copies, warp 1 issues the MMAs, warps 2-17 drain the levels (warp
// w reads TMEM lanes 32 (w % 4) .. + 31, columns (w - 2) / 4 * 16 .. + 15) and convert and store
// a tile while the next one's MMAs run.  Every mbarrier wait is bounded as in the other tcgen05
// kernels.
#include "gtn_internal.h"
#include "gtn_group.h"
#include "gtn_digits.h"
#include "gtn_tcgen05.h"

#include <algorithm>
#include <cmath>

namespace {
using namespace gtn_tc;

constexpr int kS = kF64eSlices;                  // digits per value
constexpr int kBM = kF64eRowsA;
constexpr int kBN = kF64eRowsB;                  // real columns (32 complex outputs)
constexpr int kPlaneA = kBM * 32;                // 16 real k
constexpr int kPlaneB = kBN * 32;
constexpr int kStageA = kS * kPlaneA, kStageB = kS * kPlaneB;
constexpr int kStageBytes = kStageA + kStageB;
constexpr int kStages = 5;
constexpr int kSmem = kStages * kStageBytes + 1024;
constexpr int kChunkStages = 8;                  // 128 real k between drains of the levels 4-6
constexpr int kHiLevels = 4;                     // levels 0-3: drained every second chunk
constexpr uint32_t kTmemCols = 512;              // up to 8 levels x 64 columns
constexpr int kEpiWarps = 16;                    // four per TMEM lane quarter
constexpr int kCols = kBN / (kEpiWarps / 4);     // real columns per epilogue thread
constexpr int kThreads = 64 + 32 * kEpiWarps;
// Stages of a chunk whose levels 0-3 are multiplied before the other levels are free again: the MMAs
// hide most of their drain (8192 x 1024 x 1024: 1673 -> 1533 us with 34 products, 1468 -> 1353 with 28).
constexpr int kAhead = 4;
constexpr int kGroupM = 8;                       // row tiles walked together (L2 reuse of B')
static_assert(kSmem <= 227 * 1024 - 1024, "operand ring");

// hi 2^-40 + lo 2^-72, times 2^(ea + eb - 2 * 1021) (the rows' scales), rounded once to double.
// |hi| < 2^61, |lo| < 2^63; the exponents keep the result a normal number or zero.
__device__ __forceinline__ double to_double(long long hi, long long lo, int esum) {
  long long th = hi + (lo >> 32);          // value = th 2^-40 + tl 2^-72
  uint32_t tl = (uint32_t)lo;
  const bool neg = th < 0;
  if (neg) {
    tl = 0u - tl;
    th = ~th + (tl == 0u ? 1 : 0);
  }
  int e = esum - 2 * 1021 - 41;            // bit 0 of th is 2^(e + 1), of tl 2^(e - 31)
  unsigned long long m = (unsigned long long)th;
  e += 64;                                 // bit 63
  if (m == 0) {
    if (tl == 0u) return 0.0;
    m = tl;
    tl = 0u;
    e -= 32;
  }
  const int lz = __clzll((long long)m);
  const unsigned long long w = lz == 0 ? m : (lz < 32 ? (m << lz) | (tl >> (32 - lz)) : (m << lz) | ((unsigned long long)tl << (lz - 32)));
  const bool sticky = lz < 32 && (tl << lz) != 0u;
  e -= lz;
  unsigned long long r = w >> 11;
  const uint32_t rem = (uint32_t)w & 0x7ffu;
  if (rem > 0x400u || (rem == 0x400u && (sticky || (r & 1ull)))) ++r;
  const unsigned long long bits = ((unsigned long long)(e + 1022) << 52) + r;  // r's top bit adds one
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// acc[j] += w * (the exact integer in column j).
__device__ __forceinline__ void drain(uint32_t taddr, int w, long long (&acc)[kCols]) {
  static_assert(kCols == 16, "one 16-column load");
  uint32_t v[16];
  tmem_ld16(taddr, v);
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] += (long long)__float2int_rn(__uint_as_float(v[j])) * w;
}

// Tile t -> (row tile, column tile): groups of kGroupM row tiles, rows fastest.
__device__ __forceinline__ void tile_of(int64_t t, int64_t tm, int64_t tn, int64_t* mt, int64_t* nt) {
  const int64_t per = kGroupM * tn, g = t / per, r = t - g * per;
  const int64_t gm = min((int64_t)kGroupM, tm - g * kGroupM);
  *nt = r / gm;
  *mt = g * kGroupM + (r - *nt * gm);
}

// A CTA's share of the product: whole tiles in turn (neighbouring CTAs on neighbouring tiles).  With
// Split the tiles of the last, incomplete wave (from `whole` on) are cut: their chunks, in tile
// order, are dealt evenly, CTA b of G getting [U b / G, U (b+1) / G) of the U chunks.
__device__ __forceinline__ int64_t unit_begin(int64_t U, int64_t b, int64_t G) { return U * b / G; }
template <bool Split>
struct Segments {
  int nchunks;
  int64_t t, whole, u, u0, end;
  int64_t tile = 0;
  int c0 = 0, c1 = 0, slot = 0;  // chunks [c0, c1) of the tile; where its partial sums go
  __device__ Segments(int64_t ntiles, int nch) : nchunks(nch), t(blockIdx.x), whole(ntiles) {
    if (Split) {
      whole = ntiles / gridDim.x * gridDim.x;
      const int64_t U = (ntiles - whole) * nch;
      u0 = u = unit_begin(U, blockIdx.x, gridDim.x);
      end = unit_begin(U, (int64_t)blockIdx.x + 1, gridDim.x);
    }
  }
  __device__ bool next() {
    if (t < whole) {
      tile = t;
      c0 = 0;
      c1 = nchunks;
      t += gridDim.x;
      return true;
    }
    if (!Split || u >= end) return false;
    const int64_t q = u / nchunks;
    tile = whole + q;
    c0 = (int)(u - q * nchunks);
    c1 = (int)(end - u < nchunks - c0 ? c0 + (end - u) : nchunks);
    slot = 2 * (int)blockIdx.x + (u == u0 ? 0 : 1);
    u += c1 - c0;
    return true;
  }
};

template <int L, bool Split>
__global__ void __launch_bounds__(kThreads, 1)
    f64e_gemm_kernel(const unsigned char* __restrict__ A, const unsigned char* __restrict__ B, double2* __restrict__ C,
                     int64_t M, int64_t N, int nkb, int64_t tiles_m, int64_t tiles_n, const float* __restrict__ a_exp,
                     const float* __restrict__ b_exp, longlong2* __restrict__ part, int* __restrict__ errflag) {
  chained_wait();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t chunk_full, hi_empty, lo_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ int n_issued, n_consumed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ntiles = tiles_m * tiles_n;
  const int nchunks = (nkb + kChunkStages - 1) / kChunkStages;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&chunk_full, 1);
    mbar_init(&hi_empty, kEpiWarps);
    mbar_init(&lo_empty, kEpiWarps);
    abort_flag = 0;
    n_issued = 0;
    n_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0 && lane == 0) {
    int it = 0;
    bool stop = false;
    Segments<Split> seg(ntiles, nchunks);
    while (!stop && seg.next()) {
      int64_t mt, nt;
      tile_of(seg.tile, tiles_m, tiles_n, &mt, &nt);
      const unsigned char* a = A + mt * nkb * kStageA;
      const unsigned char* b = B + nt * nkb * kStageB;
      const int kb_end = seg.c1 * kChunkStages < nkb ? seg.c1 * kChunkStages : nkb;
      for (int kb = seg.c0 * kChunkStages; kb < kb_end; ++kb, ++it) {
        const int s = it % kStages;
        const uint32_t ph = (uint32_t)(it / kStages) & 1u;
        if (!mbar_wait(&empty_bar[s], ph ^ 1u, &abort_flag)) {
          abort_flag = 1;
          atomicCAS(errflag, 0, DEVERR_TMA_TIMEOUT);
          stop = true;
          break;
        }
        const uint32_t sa = smem_u32(smem + s * kStageBytes);
        mbar_expect_tx(&full_bar[s], kStageBytes);
        bulk_load(sa, a + (int64_t)kb * kStageA, kStageA, &full_bar[s]);
        bulk_load(sa + kStageA, b + (int64_t)kb * kStageB, kStageB, &full_bar[s]);
      }
    }
    n_issued = it;
  } else if (warp == 1 && lane == 0) {
    int it = 0, ev = 0;      // stages and chunks issued
    uint32_t hi_ev = 0;      // drains of the levels 0-3 waited for
    bool stop = false;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!stop && !mbar_wait(bar, parity, &abort_flag)) {
        abort_flag = 1;
        atomicCAS(errflag, 0, DEVERR_MMA_TIMEOUT);
        stop = true;
      }
      fence_after();
      return !stop;
    };
    Segments<Split> seg(ntiles, nchunks);
    while (!stop && seg.next()) {
      int kb = seg.c0 * kChunkStages;
      for (int c = 0; c < seg.c1 - seg.c0 && !stop; ++c, ++ev) {
        const int n = nkb - kb < kChunkStages ? nkb - kb : kChunkStages;
        // the levels 0-3 run over two chunks: a pair's first one overwrites them
        if (!(c & 1) && !wait(&hi_empty, (hi_ev++ & 1u) ^ 1u)) break;
        // mma(i, j, n): digit i of A times the digits j .. j+n-1 of B', into the levels i+j ..
        // i+j+n-1
        auto mma = [&](uint32_t sa, int i, int j, int nj, uint32_t acc) {
          umma_bf16(tmem_base + (uint32_t)((i + j) * kBN), sdesc32(sa + i * kPlaneA),
                    sdesc32(sa + kStageA + j * kPlaneB), idesc_bf16(kBM, nj * kBN), acc);
        };
        auto stage = [&](int q) { return smem_u32(smem + ((it + q) % kStages) * kStageBytes); };
        auto high = [&](int q) {  // levels 0-3
          const uint32_t sa = stage(q);
          mma(sa, 0, 0, 4, (c & 1) || q > 0 ? 1u : 0u);
          mma(sa, 1, 0, 3, 1u);
          mma(sa, 2, 0, 2, 1u);
          mma(sa, 3, 0, 1, 1u);
        };
        auto low = [&](int q) {   // levels 4 .. L-1; digit 1 comes first, it reaches all of them
          const uint32_t sa = stage(q);
          const uint32_t acc = q > 0 ? 1u : 0u;
          mma(sa, 1, 3, L - 4, acc);
          mma(sa, 0, 4, 3, 1u);
          mma(sa, 2, 2, L - 4, 1u);
          mma(sa, 3, 1, L - 4, 1u);
          mma(sa, 4, 0, L - 4, 1u);
          mma(sa, 5, 0, L - 5, 1u);
          mma(sa, 6, 0, L - 6, 1u);
          umma_commit(&empty_bar[(it + q) % kStages]);
        };
        auto full = [&](int q) { return wait(&full_bar[(it + q) % kStages], (uint32_t)((it + q) / kStages) & 1u); };
        // the first stages' levels 0-3 are multiplied while the previous chunk's other levels
        // are still being drained
        const int ahead = n < kAhead ? n : kAhead;
        int q = 0;
        for (; q < ahead; ++q) {
          if (!full(q)) break;
          high(q);
        }
        if (stop || !wait(&lo_empty, ((uint32_t)ev & 1u) ^ 1u)) break;
        for (q = 0; q < ahead; ++q) low(q);
        for (; q < n; ++q) {
          if (!full(q)) break;
          high(q);
          low(q);
        }
        if (stop) break;
        it += n;
        kb += n;
        umma_commit(&chunk_full);  // the chunk's levels are complete once its MMAs are
      }
    }
    n_consumed = it;
  } else if (warp >= 2) {
    const int q4 = warp & 3;             // TMEM lane quarter
    const int cg = (warp - 2) >> 2;      // column group
    const uint32_t tm0 = tmem_base + (uint32_t)(cg * kCols) + ((uint32_t)(q4 * 32) << 16);
    int ev = 0;
    bool ok = true;
    Segments<Split> seg(ntiles, nchunks);
    while (ok && seg.next()) {
      const int nc = seg.c1 - seg.c0;
      long long hi[kCols], lo[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) hi[j] = lo[j] = 0;
      for (int c = 0; c < nc; ++c, ++ev) {
        if (!mbar_wait(&chunk_full, (uint32_t)ev & 1u, &abort_flag)) {
          if (lane == 0) {
            abort_flag = 1;
            atomicCAS(errflag, 0, DEVERR_EPI_TIMEOUT);
          }
          ok = false;
          break;
        }
        __syncwarp();
        fence_after();
        // weights 2^{-8(l + 2)}: levels 0-3 in units of 2^-40, the others in units of 2^-72
        if ((c & 1) || c == nc - 1) {
#pragma unroll 1
          for (int l = 0; l < kHiLevels; ++l) drain(tm0 + (uint32_t)(l * kBN), 1 << (8 * (3 - l)), hi);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_local(&hi_empty);
        }
#pragma unroll 1
        for (int l = kHiLevels; l < L; ++l) drain(tm0 + (uint32_t)(l * kBN), 1 << (8 * (7 - l)), lo);
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_local(&lo_empty);
      }
      if (!ok) break;
      if (Split && nc < nchunks) {  // part of a tile: f64e_finish_kernel adds the parts and converts
        longlong2* p = part + (int64_t)seg.slot * kBM * kBN + (warp - 2) * 32 + lane;
#pragma unroll
        for (int j = 0; j < kCols; ++j) p[j * 32 * kEpiWarps] = make_longlong2(hi[j], lo[j]);
        continue;
      }
      int64_t mt, nt;
      tile_of(seg.tile, tiles_m, tiles_n, &mt, &nt);
      const int64_t m = mt * kBM + q4 * 32 + lane;
      if (m < M) {
        const int ea = (int)a_exp[m];
        const int64_t nb = nt * (kBN / 2) + cg * (kCols / 2);
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) {
          const int64_t n = nb + j;
          if (n < N) {
            const int es = ea + (int)b_exp[n];
            C[n * M + m] = make_double2(to_double(hi[2 * j], lo[2 * j], es), to_double(hi[2 * j + 1], lo[2 * j + 1], es));
          }
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  if (threadIdx.x == 0) {  // copies issued but never consumed (abort path only) land before exit
    for (int it = n_consumed; it < n_issued; ++it) {
      volatile int no_abort = 0;
      mbar_wait(&full_bar[it % kStages], (uint32_t)(it / kStages) & 1u, &no_abort);
    }
  }
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// The tiles that several CTAs shared: CTA (tile, jp) adds the parts of the column pair jp of each
// epilogue thread (exact integer sums, any order gives the same), rounds and stores.
__global__ void __launch_bounds__(32 * kEpiWarps)
    f64e_finish_kernel(const longlong2* __restrict__ part, double2* __restrict__ C, int64_t M, int64_t N, int nchunks,
                       int64_t tiles_m, int64_t tiles_n, int G, const float* __restrict__ a_exp,
                       const float* __restrict__ b_exp) {
  chained_wait();
  constexpr int kPairs = kCols / 2, kT = 32 * kEpiWarps;
  const int64_t whole = tiles_m * tiles_n / G * G;
  // fewer than G tiles of at most 2^15 chunks are shared: 32 bits hold U b
  const int t = blockIdx.x / kPairs, U = (int)(tiles_m * tiles_n - whole) * nchunks;  // tile whole + t
  const int jp = blockIdx.x % kPairs;
  auto begin = [&](int b) { return (int)((uint32_t)U * (uint32_t)b / (uint32_t)G); };
  auto owner = [&](int u) { return (int)(((uint32_t)(u + 1) * (uint32_t)G + U - 1) / (uint32_t)U) - 1; };  // CTA of u
  const int b0 = owner(t * nchunks), b1 = owner(t * nchunks + nchunks - 1);
  if (b0 == b1) return;
  longlong2 re = make_longlong2(0, 0), im = make_longlong2(0, 0);
  int next = begin(b0);
#pragma unroll 4
  for (int b = b0; b <= b1; ++b) {
    const int ub = next;
    next = begin(b + 1);
    if (ub == next) continue;  // fewer chunks than CTAs: this one had none
    // its first segment where it begins in this tile, else (b == b0) its second
    const int64_t slot = 2 * b + (ub >= t * nchunks ? 0 : 1);
    const longlong2* p = part + slot * kBM * kBN + 2 * jp * kT + threadIdx.x;
    const longlong2 x = p[0], y = p[kT];
    re.x += x.x;
    re.y += x.y;
    im.x += y.x;
    im.y += y.y;
  }
  int64_t mt, nt;
  tile_of(whole + t, tiles_m, tiles_n, &mt, &nt);
  const int warp = (threadIdx.x >> 5) + 2, lane = threadIdx.x & 31;
  const int64_t m = mt * kBM + (warp & 3) * 32 + lane, n = nt * (kBN / 2) + ((warp - 2) >> 2) * kPairs + jp;
  if (m < M && n < N) {
    const int es = (int)a_exp[m] + (int)b_exp[n];
    C[n * M + m] = make_double2(to_double(re.x, re.y, es), to_double(im.x, im.y, es));
  }
}

// ---- outputs that the digit planes cannot give --------------------------------------------------
// A digit holds its entry to 2^-57 of the row's power of two, so an output is as accurate as its
// rows' largest entries, which a sparse or graded sum can be far below.  With E the sum of
//   2^-56 (alpha_k + beta_k) + 2^-62.6
// over the k at which neither factor is zero (alpha, beta: magnitudes max(|re|, |im|) of the scaled
// rows, at most 1/2; the last term for the levels left out), each part of an output is exact to E.
// It stands where E <= 2 K 2^-53 sum alpha beta, the a-priori bound of K complex multiply-adds in
// FP64 (N. J. Higham, Accuracy and Stability of Numerical Algorithms, 2nd ed., section 3.1); the others
// are summed again on the FP64 pipe.
//   * f64e_check_kernel looks for outputs with sum alpha beta below kSureSum, above which the bound
//     holds whatever the entries.  Two rows with L of W entries more than W = 128 together that are at
//     least 0.0508 have L products of 0.0026 in common: 28 are enough, and so the tiles of dense
//     operands are done by counting (a row of 128 Gaussian entries has 110 such).  Of the others the
//     sums are formed from bf16 magnitudes, 64 k at a time until all are above.  A sum of zero means
//     that no two factors meet, and that the digit products are exact.  What remains is listed.
//   * f64e_repair_kernel adds E and the magnitudes' products over the listed outputs' rows.  Where the
//     bound does not hold it adds the products of A's first and B's eighth digits to the output, by
//     which B's entries count to 2^-65 and E becomes the sum of
//       2^-56 beta_k + 2^-64 + min(2^-62.6, 2^-12.6 min(alpha_k, beta_k))
//     (the last for the levels left out: a factor below 2^-50 has few digits to meet them).  That is
//     what the identity channel of an environment wants, one entry of 1 and others of rounding size.
//     Where it is not enough either the output is summed again.  Chunks of 32 listed outputs keep every
//     SM at work where they come from few tiles.
// The sums have half of the digit product's rows, columns and k and one plane: mma.sync, which
// needs no TMEM (the digit levels hold all of it), leaves them a small part of the step.
// One-site map of a 31-site binary tree at D = 128 (M = 163840, N = 640, K = 128, digit product
// 2423 us): the sums take 241 us, 148 us with tiles that end early, and counting 27 us.  Products of the
// two-site map of a DMRG step at D = 96 (M = 384, N = 480, K = 96 and M = 384, N = 96, K = 480) with a
// state of which 7 to 10 % of the outputs miss the bound: check 11 and 19 us, repair 27 and 50 us (with
// a CTA for each tile 1059 and 510 us together); 1 % of a Lanczos vector's: 23 us together.  Environments
// of a random state at D = 128 (M = 163840, N = 640, K = 128; 6.4 % miss it, 2.4 % with eighth digits
// too): 5.9 ms, 10.5 ms with every one of them summed again, 93 ms on the FP64 pipe.
constexpr int kRM = kF64eCheckM, kRN = kF64eCheckN, kRThreads = 256;
constexpr int kRKC = 64, kRStages = 2;              // complex k per stage (rows of 128 bytes)
constexpr int kRStage = (kRM + kRN) * kRKC * 2;
constexpr int kRSmem = kRStages * kRStage;
static_assert(kRM * kRN * 2 + (kRM + kRN) * 4 <= kRSmem, "a tile's list and sums over the stages");
// (2^-56 + 2^-62.6) K <= 2 K 2^-53 s from s = 0.0632 on; the rest covers the rounding of the sums
constexpr float kSureSum = 0.0703f;
constexpr int kSureMeets = 28;  // times 0.05078^2
// E / (2 2^-53): 2^-4 (alpha + beta) and 2^-10.6, with the rounding of the magnitudes and sums
constexpr float kMagError = 0.064f, kLevelError = 0.00066f;
constexpr float kLowError = 0.000247f, kSmallError = 7.35e11f;  // 2^-12, 2^39.4
constexpr int kRowSumBlocks = 512;  // K up to 4096: longer sums are above kSureSum or far below

struct RepairArgs {
  const double2* T;
  const int64_t *om, *ok;  // offset tables, or null
  GroupSpec mg, kg;
  const double2* B;
  double2* C;
  int64_t M, N, K, tiles_m, ntiles;
  const float *a_exp, *b_exp;
  const uint16_t *a_mag, *b_mag;
  const int* b_large;
  const uint32_t* b_low;
  int low_all;
  const unsigned char* planes;  // of A
  uint16_t* lists;             // [tile][kRM kRN]: n_local kRM + m_local
  unsigned long long* chunks;  // tile << 24 | first << 8 | length
  int* count;                  // chunks
};

__global__ void __launch_bounds__(kRThreads, 3) f64e_check_kernel(const __grid_constant__ RepairArgs g) {
  chained_wait();
  extern __shared__ __align__(128) unsigned char rsmem[];
  __shared__ int count, slot, large[kRM], least_row[kRThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
  const int64_t nkb = (g.K + 7) / 8;
  const int nk = (int)((nkb + kRKC / 8 - 1) / (kRKC / 8));
  const uint32_t s0 = smem_u32(rsmem);
  auto ldmatrix = [&](uint32_t addr, uint32_t (&v)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(addr)
                 : "memory");
  };
  // chunk kc of the tile at (m0, n0) into a stage: 16 bytes (8 k) of a row a time, rows on consecutive threads
  auto load = [&](int64_t m0, int64_t n0, int kc, int stage) {
    if (kc < nk) {
      const uint32_t st = s0 + (uint32_t)(stage * kRStage);
      auto put = [&](const uint16_t* mag, int64_t row, int64_t rows, int r, int c) {
        const int64_t kb = (int64_t)kc * (kRKC / 8) + c;
        const bool in = row < rows && kb < nkb;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(st + r * 128 + ((c ^ (r & 7)) << 4)),
                     "l"(mag + (in ? (kb * rows + row) * 8 : 0)), "r"(in ? 16 : 0)
                     : "memory");
      };
#pragma unroll
      for (int i = 0; i < kRM * 8 / kRThreads; ++i) {
        const int e = i * kRThreads + tid, r = e % kRM;
        put(g.a_mag, m0 + r, g.M, r, e / kRM);
      }
#pragma unroll
      for (int i = 0; i < kRN * 8 / kRThreads; ++i) {
        const int e = i * kRThreads + tid, r = e % kRN;
        put(g.b_mag, n0 + r, g.N, kRM + r, e / kRN);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[2][4][4];
  auto multiply = [&](int stage) {
    const uint32_t st = s0 + (uint32_t)(stage * kRStage);
#pragma unroll
    for (int ks = 0; ks < kRKC / 16; ++ks) {
      uint32_t a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + (lane & 15), c = ks * 2 + (lane >> 4);
        ldmatrix(st + r * 128 + ((c ^ (r & 7)) << 4), a[i]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = kRM + wn + j * 16 + (lane & 7) + ((lane >> 4) << 3), c = ks * 2 + ((lane >> 3) & 1);
        ldmatrix(st + r * 128 + ((c ^ (r & 7)) << 4), b[j]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
              "{%0, %1, %2, %3};"
              : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
              : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[j >> 1][(j & 1) * 2]),
                "r"(b[j >> 1][(j & 1) * 2 + 1]));
    }
  };
  auto for_outputs = [&](auto f) {  // f(m_local, n_local, sum)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          f(wm + i * 16 + (lane >> 2) + (e >> 1) * 8, wn + j * 8 + 2 * (lane & 3) + (e & 1), acc[i][j][e]);
  };
  uint16_t* list = reinterpret_cast<uint16_t*>(rsmem);
  float* row_sum = reinterpret_cast<float*>(rsmem + kRM * kRN * 2);  // of the rows of A, then of B
  const int window = (int)min(g.K, (int64_t)kF64eWindow), wkb = (int)min(nkb, (int64_t)(kF64eWindow / 8));
  // a CTA's tiles: a range with the column tiles of a row tile behind each other
  const unsigned tiles_n = (unsigned)(g.ntiles / g.tiles_m);
  const unsigned end = (unsigned)(g.ntiles * (blockIdx.x + 1) / gridDim.x);
  unsigned row = ~0u;
#pragma unroll 1
  for (unsigned t = (unsigned)(g.ntiles * blockIdx.x / gridDim.x); t < end; ++t) {
    const unsigned tm = t / tiles_n, tn = t - tm * tiles_n;
    const int64_t m0 = (int64_t)tm * kRM, n0 = (int64_t)tn * kRN;
    const int mlim = (int)min((int64_t)kRM, g.M - m0), nlim = (int)min((int64_t)kRN, g.N - n0);
    // A CTA of one tile forms the sums at once: counting is worth its latency from the second one on
    // (two-site map of a chain at D = 250, 160 tiles: 287 us with it, 283 without).
    if (g.ntiles > gridDim.x && tm != row) {  // large entries of the row tile, two threads a row
      row = tm;
      if (tid < kRM) large[tid] = 0;
      __syncthreads();
      const int r = tid % kRM;
      int c = 0;
      if (r < mlim)
#pragma unroll 4
        for (int kb = tid / kRM; kb < wkb; kb += 2) {
          const uint4 u = *reinterpret_cast<const uint4*>(g.a_mag + (kb * g.M + m0 + r) * 8);
          const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t lo = x[q] & 0xffffu, hi = x[q] >> 16;
            c += (lo >= kF64eLarge) + (hi >= kF64eLarge);
            if (lo > 0x7f80u) c = kF64eNoCount;
          }
        }
      atomicAdd(&large[r], r < mlim ? c : window);
      __syncthreads();
      int least = large[r];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) least = min(least, __shfl_xor_sync(0xffffffffu, least, o));
      if (lane == 0) least_row[warp] = least;
      __syncthreads();
    }
    if (g.ntiles > gridDim.x) {  // every output of the tile sure by the numbers of large entries?
      int a = least_row[0];
#pragma unroll
      for (int q = 1; q < kRM / 32; ++q) a = min(a, least_row[q]);
      const bool few = tid < nlim && a + g.b_large[n0 + tid] < window + kSureMeets;
      if (!__syncthreads_or(few)) continue;
    }
#pragma unroll
    for (int p = 0; p < kRStages - 1; ++p) load(m0, n0, p, p);
    if (tid == 0) count = 0;
    for_outputs([&](int, int, float& s) { s = 0.f; });
    if (mlim < kRM || nlim < kRN)  // outputs beyond the edges are sure (or NaN)
      for_outputs([&](int ml, int nl, float& s) { s = ml < mlim && nl < nlim ? 0.f : 1.f; });
    bool done = false;
#pragma unroll 1
    for (int kc = 0; kc < nk && !done; ++kc) {
      load(m0, n0, kc + kRStages - 1, (kc + kRStages - 1) % kRStages);  // where chunk kc - 1 was
      asm volatile("cp.async.wait_group %0;" ::"n"(kRStages - 1) : "memory");
      __syncthreads();
      multiply(kc % kRStages);
      bool sure = true;
      for_outputs([&](int, int, float& s) { sure = sure && s >= kSureSum; });  // (never for NaN)
      done = __syncthreads_and(sure);  // and the stage may be written again
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (done) continue;
    // the bound again with the rows' own sums in place of K halves (a thread a row; short sums, and
    // graded rows, gain by it)
    const bool sums = nkb <= kRowSumBlocks;
    if (sums) {
      if (tid < kRM + kRN) {
        const bool is_a = tid < kRM;
        const int64_t rows = is_a ? g.M : g.N, row_at = is_a ? m0 + tid : n0 + tid - kRM;
        const uint16_t* mag = (is_a ? g.a_mag : g.b_mag) + row_at * 8;
        float x = 0.f;
        if (row_at < rows)
#pragma unroll 8
          for (int kb = 0; kb < (int)nkb; ++kb) {
            const uint4 u = *reinterpret_cast<const uint4*>(mag + kb * rows * 8);
            x += ((__uint_as_float(u.x << 16) + __uint_as_float(u.x & 0xffff0000u)) +
                  (__uint_as_float(u.y << 16) + __uint_as_float(u.y & 0xffff0000u))) +
                 ((__uint_as_float(u.z << 16) + __uint_as_float(u.z & 0xffff0000u)) +
                  (__uint_as_float(u.w << 16) + __uint_as_float(u.w & 0xffff0000u)));
          }
        row_sum[tid] = kMagError * x;
      }
      __syncthreads();
    }
    const float levels = kLevelError * (float)g.K;
    uint32_t doubtful = 0, bit = 1;
    for_outputs([&](int ml, int nl, float& s) {
      if (!(s >= kSureSum) && s != 0.f && ml < mlim && nl < nlim &&
          !(sums && s * (float)g.K >= row_sum[ml] + row_sum[kRM + nl] + levels))
        doubtful |= bit;
      bit <<= 1;
    });
    int at = __popc(doubtful), total = at;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, total, o);
      if (lane >= o) total += x;
    }
    at = total - at;  // of the lanes before
    int first = 0;
    if (lane == 31 && total > 0) first = atomicAdd(&count, total);
    at += __shfl_sync(0xffffffffu, first, 31);
    bit = 1;
    for_outputs([&](int ml, int nl, float&) {
      if (doubtful & bit) list[at++] = (uint16_t)(nl * kRM + ml);
      bit <<= 1;
    });
    __syncthreads();
    const int n = count, nch = (n + kF64eCheckChunk - 1) / kF64eCheckChunk;
    if (n > 0) {
      if (tid == 0) slot = atomicAdd(g.count, nch);
      for (int e = tid; e < n; e += kRThreads) g.lists[(int64_t)t * (kRM * kRN) + e] = list[e];
      __syncthreads();
      for (int c = tid; c < nch; c += kRThreads)
        g.chunks[slot + c] = (unsigned long long)t << 24 | (unsigned long long)(c * kF64eCheckChunk) << 8 |
                             (unsigned long long)min(kF64eCheckChunk, n - c * kF64eCheckChunk);
    }
    __syncthreads();
  }
}

constexpr int kRPerWarp = 4;                        // outputs a warp sums at a time
constexpr int kPThreads = 4 * kF64eCheckChunk;      // four threads for each output of a chunk

// Sum the listed outputs (n_local kRM + m_local) of the tile at (m0, n0) again: kRPerWarp a warp, the k
// range over its lanes.  Warps work by themselves: the latency of their loads is what this takes.
template <int Threads>
__device__ __forceinline__ void repair_outputs(const RepairArgs& g, const uint16_t* list, int count, int64_t m0,
                                               int64_t n0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto offset = [&](int64_t k) { return g.ok ? g.ok[k] : decompose(k, g.kg); };
#pragma unroll 1
  for (int base = warp * kRPerWarp; base < count; base += Threads / 32 * kRPerWarp) {
    int64_t om[kRPerWarp];
    const double2* b[kRPerWarp];
    double2 acc[kRPerWarp];
#pragma unroll
    for (int j = 0; j < kRPerWarp; ++j) {
      const int id = list[min(base + j, count - 1)];  // past the end: the last one again
      const int64_t m = m0 + id % kRM;
      om[j] = g.om ? g.om[m] : decompose(m, g.mg);
      b[j] = g.B + (n0 + id / kRM) * g.K;
      acc[j] = make_double2(0.0, 0.0);
    }
    auto add = [&](double2& s, double2 t, double2 v) {
      s.x = fma(t.x, v.x, s.x);
      s.x = fma(-t.y, v.y, s.x);
      s.y = fma(t.x, v.y, s.y);
      s.y = fma(t.y, v.x, s.y);
    };
    int64_t k = lane;
#pragma unroll 1
    for (; k + 32 < g.K; k += 64) {
      const int64_t o0 = offset(k), o1 = offset(k + 32);
      double2 t[2][kRPerWarp], v[2][kRPerWarp];
#pragma unroll
      for (int j = 0; j < kRPerWarp; ++j) {
        t[0][j] = g.T[om[j] + o0];
        v[0][j] = b[j][k];
        t[1][j] = g.T[om[j] + o1];
        v[1][j] = b[j][k + 32];
      }
#pragma unroll
      for (int j = 0; j < kRPerWarp; ++j) {
        add(acc[j], t[0][j], v[0][j]);
        add(acc[j], t[1][j], v[1][j]);
      }
    }
    if (k < g.K) {
      const int64_t o = offset(k);
#pragma unroll
      for (int j = 0; j < kRPerWarp; ++j) add(acc[j], g.T[om[j] + o], b[j][k]);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kRPerWarp; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        acc[j].x += __shfl_xor_sync(0xffffffffu, acc[j].x, o);
        acc[j].y += __shfl_xor_sync(0xffffffffu, acc[j].y, o);
      }
      if (lane == 0 && base + j < count) {
        const int id = list[base + j];
        g.C[(n0 + id / kRM) * g.M + m0 + id % kRM] = acc[j];
      }
    }
  }
}

// Two bf16 in a word: the first (even k, or the real part) and the second.
__device__ __forceinline__ float lo16(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi16(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float sum4(float x) {  // over the four threads of an output
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x + __shfl_xor_sync(0xffffffffu, x, 1);
}

// Checked products: the chunks of f64e_check_kernel, four threads for each output.  Each decides
// between the output as it is, with B's eighth digits, and a sum on the FP64 pipe.
__global__ void __launch_bounds__(kPThreads, 4) f64e_repair_kernel(const __grid_constant__ RepairArgs g) {
  chained_wait();
  __shared__ uint16_t again[kF64eCheckChunk];
  __shared__ int nagain;
  const int nch = *g.count, l = threadIdx.x & 3, e = threadIdx.x >> 2;
  const int64_t nkb = (g.K + 7) / 8, tiles_n = g.ntiles / g.tiles_m;
#pragma unroll 1
  for (int c = blockIdx.x; c < nch; c += gridDim.x) {
    const unsigned long long ch = g.chunks[c];
    const int64_t tile = (int64_t)(ch >> 24);
    const int count = (int)(ch & 0xff), first = (int)(ch >> 8 & 0xffff);
    const int64_t m0 = tile / tiles_n * kRM, n0 = tile % tiles_n * kRN;
    const int id = g.lists[tile * (kRM * kRN) + first + min(e, count - 1)], rr = id % kRM;
    const int64_t m = m0 + rr, n = n0 + id / kRM;
    const unsigned char* a = g.planes + (m0 / kBM * nkb * kS * kBM + rr) * 32;  // A's first digits
    const uint32_t* b = g.b_low + n * 8 * nkb;
    const bool kept = f64e_low_kept(g.b_large[n], g.K, g.low_all);
    const int eb = (int)g.b_exp[n];
    const uint16_t *am = g.a_mag + m * 8, *bm = g.b_mag + n * 8;
    float re = 0.f, im = 0.f, prod = 0.f, alpha = 0.f, beta = 0.f, met = 0.f, left = 0.f;
#pragma unroll 2
    for (int64_t q = l; q < 2 * nkb; q += 4) {  // four k
      const uint4 u = *reinterpret_cast<const uint4*>(a + (q >> 1) * (kS * kPlaneA) + (((int)q ^ (rr >> 2)) & 1) * 16);
      const uint2 x = *reinterpret_cast<const uint2*>(am + (q >> 1) * g.M * 8 + (q & 1) * 4);
      const uint2 y = *reinterpret_cast<const uint2*>(bm + (q >> 1) * g.N * 8 + (q & 1) * 4);
      const uint32_t d[4] = {u.x, u.y, u.z, u.w}, xs[2] = {x.x, x.y}, ys[2] = {y.x, y.y};
      float tr[4], ti[4];
      if (kept) {
        const uint4 v = *reinterpret_cast<const uint4*>(b + q * 4);
        const uint32_t t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          tr[p] = lo16(t[p]);
          ti[p] = hi16(t[p]);
        }
      } else {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const double2 v = q * 4 + p < g.K ? g.B[n * g.K + q * 4 + p] : make_double2(0.0, 0.0);
          tr[p] = (float)low_digit(v.x, eb);
          ti[p] = (float)low_digit(v.y, eb);
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        re = fmaf(lo16(d[p]), tr[p], fmaf(-hi16(d[p]), ti[p], re));
        im = fmaf(lo16(d[p]), ti[p], fmaf(hi16(d[p]), tr[p], im));
        const float al = p & 1 ? hi16(xs[p >> 1]) : lo16(xs[p >> 1]), be = p & 1 ? hi16(ys[p >> 1]) : lo16(ys[p >> 1]);
        const bool both = al != 0.f && be != 0.f;
        prod = fmaf(al, be, prod);
        alpha += both ? al : 0.f;
        beta += both ? be : 0.f;
        met += both ? 1.f : 0.f;
        left += both ? fminf(kLevelError, kSmallError * fminf(al, be)) : 0.f;
      }
    }
    __syncwarp();
    re = sum4(re);
    im = sum4(im);
    prod = sum4(prod) * (float)g.K;
    alpha = sum4(alpha);
    beta = sum4(beta);
    met = sum4(met);
    left = sum4(left);
    __syncthreads();  // the last chunk's list has been used
    if (threadIdx.x == 0) nagain = 0;
    __syncthreads();
    // (no bound holds with NaN, the magnitudes of a row without digits)
    if (l == 0 && e < count && !(prod >= fmaf(kMagError, alpha + beta, kLevelError * met))) {
      if (prod >= fmaf(kMagError, beta, fmaf(kLowError, met, left))) {  // units of 2^-72 of the scaled rows
        const int scale = (int)g.a_exp[m] + (int)g.b_exp[n] - 2 * 1021 - 72;
        double2* y = g.C + n * g.M + m;
        *y = make_double2(y->x + scalbn((double)re, scale), y->y + scalbn((double)im, scale));
      } else {
        again[atomicAdd(&nagain, 1)] = (uint16_t)id;
      }
    }
    __syncthreads();
    repair_outputs<kPThreads>(g, again, nagain, m0, n0);
  }
}

// Others (FP64E): the outputs of rows without digits, found by the rows' exponents tile by tile.
__global__ void __launch_bounds__(kRThreads) f64e_rows_kernel(const __grid_constant__ RepairArgs g) {
  chained_wait();
  __shared__ uint16_t list[kRM * kRN];
  __shared__ uint8_t bad[kRM + kRN];  // rows of A, then of B
  __shared__ int count;
  for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    const int64_t m0 = tile % g.tiles_m * kRM, n0 = tile / g.tiles_m * kRN;
    bool any = false;
    if (threadIdx.x < kRM + kRN) {
      const bool is_a = threadIdx.x < kRM;
      const int64_t r = is_a ? m0 + threadIdx.x : n0 + threadIdx.x - kRM;
      any = r < (is_a ? g.M : g.N) && f64e_no_digits(is_a ? g.a_exp[r] : g.b_exp[r]);
      bad[threadIdx.x] = any;
    }
    if (threadIdx.x == 0) count = 0;
    if (!__syncthreads_or(any)) continue;
    for (int e = threadIdx.x; e < kRM * kRN; e += kRThreads) {
      const int ml = e % kRM, nl = e / kRM;
      if (m0 + ml < g.M && n0 + nl < g.N && (bad[ml] || bad[kRM + nl])) list[atomicAdd(&count, 1)] = (uint16_t)e;
    }
    __syncthreads();
    repair_outputs<kRThreads>(g, list, count, m0, n0);
    __syncthreads();
  }
}

}  // namespace

// Seconds of a chunk (128 real k) and of a tile's end, and whether the last wave's tiles are shared:
// when whole ones would leave more idle than the shared tiles' sums cost (about 10 us: 128 KB a part
// written and read back, one more launch).  Measured, 34 products: M, N, K = 384, 96, 480 (9 tiles)
// 63 -> 25 us, 250, 250, 1250 (16 tiles) 143 -> 39 us.
constexpr double kChunk = 6e-6, kTileEnd = 2.5e-6, kShareCost = 10e-6;
static double f64e_waves(double M, double N, double K, int sms, bool* share) {
  const double tiles = std::ceil(M / kBM) * std::ceil(2 * N / kBN), chunks = std::ceil(K / 64);
  const double tile = std::min(chunks, K / 64 + 0.125) * kChunk + kTileEnd;
  const double rest = tiles - std::floor(tiles / sms) * sms;
  const double cut = std::ceil(rest * chunks / sms) * kChunk + kTileEnd + kShareCost;
  *share = rest > 0 && chunks > 1 && cut < tile;
  return std::floor(tiles / sms) * tile + (rest > 0 ? std::min(tile, cut) : 0.0);
}
// Digit planes: the split, the check and the launches, then the waves of tiles.  FP64 pipe: 1.15
// TFLOP/s.
double f64e_time(double M, double N, double K) {
  bool share;
  return 12e-6 + f64e_waves(M, N, K, 152, &share) + M * K * 60 / 4e12;
}
// CTAs of a product, and whether its last tiles are shared.
static int64_t f64e_grid(int64_t M, int64_t N, int64_t K, int sm_count, bool* share) {
  const int64_t sms = std::max(1, sm_count), tiles = ((M + kBM - 1) / kBM) * ((2 * N + kBN - 1) / kBN);
  f64e_waves((double)M, (double)N, (double)K, (int)sms, share);
  const int64_t chunks = (K + 8 * kChunkStages - 1) / (8 * kChunkStages);
  return std::min(*share && tiles < sms ? tiles * chunks : tiles, sms);
}
size_t f64e_part_bytes(int64_t M, int64_t N, int64_t K, int sm_count) {
  bool share;
  const int64_t grid = f64e_grid(M, N, K, sm_count, &share);
  return share ? (size_t)(2 * grid) * kBM * kBN * sizeof(longlong2) : 0;  // two segments a CTA
}
double f64_pipe_time(double M, double N, double K) { return 4e-6 + 8.0 * M * N * K / 1.15e12; }

cudaError_t launch_f64e_gemm(const F64eGemmArgs& a, int sm_count, int* errflag, cudaStream_t s, std::string* why,
                             int* launches) {
  *launches = 0;
  if (a.M <= 0 || a.N <= 0) return cudaSuccess;
  if (!a.A || !a.B || !a.C || !a.a_exp || !a.b_exp || a.K <= 0 || a.K > kF64eMaxK) {
    if (why) *why = "f64e_gemm: every operand given and K at most 2^21";
    return cudaErrorInvalidValue;
  }
  if (reinterpret_cast<uintptr_t>(a.A) % 16 || reinterpret_cast<uintptr_t>(a.B) % 16) {
    if (why) *why = "f64e_gemm: digit planes must be 16-byte aligned";
    return cudaErrorInvalidValue;
  }
  const int nkb = (int)((a.K + 7) / 8);
  const int64_t tm = (a.M + kBM - 1) / kBM, tn = (2 * a.N + kBN - 1) / kBN;
  const int nchunks = (nkb + kChunkStages - 1) / kChunkStages;
  bool share = false;
  int64_t grid = f64e_grid(a.M, a.N, a.K, sm_count, &share);
  if (share && !a.part) {
    share = false;
    grid = std::min<int64_t>(tm * tn, std::max(1, sm_count));
  }
  using Kern = void (*)(const unsigned char*, const unsigned char*, double2*, int64_t, int64_t, int, int64_t, int64_t,
                        const float*, const float*, longlong2*, int*);
  static const Kern kerns[4] = {f64e_gemm_kernel<8, false>, f64e_gemm_kernel<8, true>, f64e_gemm_kernel<7, false>,
                                f64e_gemm_kernel<7, true>};
  static PerDeviceOnce opt_in[4];
  const int which = (a.levels == 7 ? 2 : 0) + (share ? 1 : 0);
  if (const cudaError_t e = smem_opt_in(opt_in[which], kerns[which], kSmem)) return e;
  launch_chained(kerns[which], dim3((unsigned)grid), dim3(kThreads), kSmem, s, static_cast<const unsigned char*>(a.A), static_cast<const unsigned char*>(a.B), a.C, a.M, a.N, nkb, tm, tn,
      a.a_exp, a.b_exp, share ? static_cast<longlong2*>(a.part) : nullptr, errflag);
  cudaError_t e = cudaGetLastError();
  *launches = 1;
  if (e == cudaSuccess && share) {
    *launches = 2;
    const int64_t rest = tm * tn - tm * tn / grid * grid;
    launch_chained(f64e_finish_kernel, dim3((unsigned)(rest * (kCols / 2))), dim3(32 * kEpiWarps), 0, s, static_cast<const longlong2*>(a.part), a.C, a.M, a.N,
                                                             nchunks, tm, tn, (int)grid, a.a_exp, a.b_exp);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t launch_f64e_repair(const F64eGemmArgs& a, const double2* T, const GatherTab& tab, const GroupSpec& mg,
                               const GroupSpec& kg, const double2* B, int sm_count, cudaStream_t s, int* launches) {
  *launches = 0;
  if (a.M <= 0 || a.N <= 0) return cudaSuccess;
  RepairArgs g = {};
  g.T = T;
  g.om = tab.om;
  g.ok = tab.ok;
  g.mg = mg;
  g.kg = kg;
  g.B = B;
  g.C = a.C;
  g.M = a.M;
  g.N = a.N;
  g.K = a.K;
  g.tiles_m = (a.M + kRM - 1) / kRM;
  g.ntiles = g.tiles_m * ((a.N + kRN - 1) / kRN);
  g.a_exp = a.a_exp;
  g.b_exp = a.b_exp;
  const int sms = std::max(1, sm_count);
  if (!a.a_mag) {
    *launches = 1;
    return launch_chained(f64e_rows_kernel, dim3((unsigned)std::min<int64_t>(g.ntiles, 4 * sms)), dim3(kRThreads), 0, s, g);
  }
  g.a_mag = a.a_mag;
  g.b_mag = a.b_mag;
  g.b_large = a.b_large;
  g.count = a.count;
  g.b_low = a.b_low;
  g.low_all = a.low_all;
  g.planes = static_cast<const unsigned char*>(a.A);
  g.lists = static_cast<uint16_t*>(a.lists);
  g.chunks = reinterpret_cast<unsigned long long*>(g.lists + g.ntiles * kRM * kRN);
  static PerDeviceOnce opt_in;
  if (const cudaError_t e = smem_opt_in(opt_in, f64e_check_kernel, kRSmem)) return e;
  *launches = 2;
  cudaError_t e = launch_chained(f64e_check_kernel, dim3((unsigned)std::min<int64_t>(g.ntiles, 3 * sms)),
                                 dim3(kRThreads), kRSmem, s, g);
  if (e == cudaSuccess) e = launch_chained(f64e_repair_kernel, dim3((unsigned)(4 * sms)), dim3(kPThreads), 0, s, g);
  return e;
}
