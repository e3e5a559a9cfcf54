// Internal declarations shared by the libgrafttn translation units.
#pragma once

#include "gtn_once.h"

#include <utility>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>
#include <map>
#include <memory>
#include <mutex>

#include "../../include/grafttn.h"

#define GTN_MAXG 12   // index groups per gather (a two-site tensor of a 4-ary tree has 10 legs)
#define GTN_BLOCK_MAXG 8  // index groups of a gtn_block_gather (the ABI struct's arrays)

// A multi-index group: index i in [0, prod(dim)) decomposes into digits (outer..inner)
// whose strides (in elements) give the offset into a row-major tensor.
struct GroupSpec {
  int n;
  int64_t dim[GTN_MAXG];
  int64_t str[GTN_MAXG];
};

// Where a product's output (n, m) goes: C[n][m], or the offsets of these groups (on != 0).
struct OutView {
  int on = 0;
  GroupSpec n, m;
};

// Launches of the plans' chains: a kernel may be set up, and its CTAs become resident, while the
// one before it in the stream still runs; its first statement, chained_wait(), returns when that one
// has completed and its writes are visible (CTAs wait without issuing).  The order of the stream is
// kept: whatever is launched without this waits for the whole kernel as usual.  Saves about
// 1.2 us a launch (two-site FP64 map of a chain at bond 250: 11 launches, 268 -> 255 us).
template <class... P, class... A>
inline cudaError_t launch_chained_if(bool chained, void (*kern)(P...), dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  return launch_chained_if(true, kern, grid, block, smem, s, std::forward<A>(args)...);
}
// A kernel's attribute, set once per device (it belongs to the kernel on the current device).
template <class... P>
inline cudaError_t func_attribute(PerDeviceOnce& once, void (*kern)(P...), cudaFuncAttribute attribute, int value) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  return e != cudaSuccess ? e : once(dev, [&] { return cudaFuncSetAttribute(kern, attribute, value); });
}
// Opt in to more than 48 KB of dynamic shared memory.
template <class... P>
inline cudaError_t smem_opt_in(PerDeviceOnce& once, void (*kern)(P...), size_t bytes) {
  return func_attribute(once, kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
#ifdef __CUDACC__
__device__ __forceinline__ void chained_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// Device error codes written to the context's error flag by bounded waits.
enum : int { DEVERR_NONE = 0, DEVERR_TMA_TIMEOUT = 1, DEVERR_MMA_TIMEOUT = 2, DEVERR_EPI_TIMEOUT = 3,
             DEVERR_SELFTEST_TIMEOUT = 4 };
cudaError_t launch_wait_selftest(int* errflag, uint64_t timeout_ns, cudaStream_t s);

struct gtn_ctx_s {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;          // last failure message (any thread), guarded by err_mu
  std::mutex err_mu;
  int64_t launches = 0;
  int* d_errflag = nullptr;
  int sm_count = 0;
  int cc_major = 0, cc_minor = 0;
  // reduction scratch (device + pinned host)
  double2* d_red = nullptr;
  size_t red_cap = 0;
  double2* h_red = nullptr;
  size_t hred_cap = 0;
  cudaEvent_t step_ev[2] = {nullptr, nullptr};  // the Krylov steps in flight
  // transient workspace for one-shot contractions / factorisations
  void* ws = nullptr;
  size_t ws_bytes = 0;
  // bump arena of one-shot contractions (stream-ordered reuse, grown to the largest need)
  char* carena = nullptr;
  size_t carena_cap = 0, carena_need = 0;
  void* cusolver = nullptr;
  // precision of the GEMMs inside the factorisations (Gram SVD route): GTN_PREC_FP64 or
  // GTN_PREC_FP64E (gtn_ctx_set_linalg_precision)
  int linalg_prec = 0;
  // freed map workspace blocks by size, reused in stream order by later maps on this
  // context (maps are built and dropped at every node visit of a sweep; cudaMalloc and the
  // device-synchronising cudaFree made a small map's creation cost about a millisecond)
  std::multimap<size_t, void*> blk_free;
  size_t blk_cached = 0;
};

// ---- status helpers -------------------------------------------------------------
int set_err(gtn_ctx ctx, int code, const std::string& msg);
#define GTN_CUDA_TRY(ctx, expr)                                                       \
  do {                                                                                \
    cudaError_t e__ = (expr);                                                         \
    if (e__ != cudaSuccess)                                                           \
      return set_err((ctx), GTN_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e__)); \
  } while (0)

cudaError_t ctx_workspace(gtn_ctx ctx, size_t bytes, void** out);
// Map workspace blocks through the context's cache: *got is the block's size, to be handed
// back with the block; release returns it to the cache (or frees it past the cache's bound),
// flush frees every cached block.
cudaError_t ctx_blk_alloc(gtn_ctx ctx, size_t bytes, void** out, size_t* got);
void ctx_blk_release(gtn_ctx ctx, void* p, size_t bytes);
void ctx_blk_flush(gtn_ctx ctx);
// Thin QR of a tall-skinny row-major matrix by shifted Cholesky QR with two refinement
// passes (gtn_tsqr.cu); GTN_ERR_UNSUPPORTED when it does not apply or the matrix is too
// ill-conditioned for it (the Householder QR then runs).
bool tsqr_applies(int64_t m, int64_t n);
// Householder QR of a small matrix (m n and m min(m, n) <= 4096) in one CTA, no host sync.
bool small_qr_applies(int64_t m, int64_t n);
// One-sided Jacobi SVD of a small matrix (min(m, n) <= 64, m n <= 4096) in one CTA:
// S (k, descending), U (m x k row-major), Vh (k x n row-major), k = min(m, n), on the device.
bool small_svd_applies(int64_t m, int64_t n);
int svd_small_launch(gtn_ctx ctx, int64_t m, int64_t n, const double2* A, double* S, double2* U, double2* Vh);
// One-sided Jacobi SVD over the whole chip (gtn_jacobi.cu), min(m, n) <= 384 and max(m, n) <= 768:
// run computes all singular values (host, descending), store the leading r vectors from the same
// workspace of jacobi_svd_bytes.
bool jacobi_svd_applies(int64_t m, int64_t n);
size_t jacobi_svd_bytes(int64_t m, int64_t n);
int jacobi_svd_run(gtn_ctx ctx, int64_t m, int64_t n, const double2* A, void* ws, std::vector<double>* S);
int jacobi_svd_store(gtn_ctx ctx, int64_t m, int64_t n, void* ws, int64_t r, int64_t nonzero, double2* U, double2* Vh);
int qr_small(gtn_ctx ctx, int64_t m, int64_t n, const double2* A, double2* Q, double2* R);
int qr_tall_cholesky(gtn_ctx ctx, int64_t m, int64_t n, const double2* A, double2* Q, double2* R);
cudaError_t ctx_red(gtn_ctx ctx, size_t n2);   // ensure d_red/h_red hold n2 double2
void linalg_release(gtn_ctx ctx);               // drop the cuSOLVER handle (gtn_linalg.cu)

// ---- layout kernels (gtn_layout.cu) ----------------------------------------------
// out[m, k] = T[offM(m) + offK(k)] for m < M, k < Kw (zero where k >= K).
cudaError_t launch_gather_c128_to_c128(const double2* T, const GroupSpec& mg, const GroupSpec& kg,
                                       int64_t M, int64_t K, int64_t ldo, double2* out, cudaStream_t s);
cudaError_t launch_gather_c128_to_c64(const double2* T, const GroupSpec& mg, const GroupSpec& kg,
                                      int64_t M, int64_t K, int64_t ldo, float2* out, cudaStream_t s);
cudaError_t launch_gather_c64_to_c64(const float2* T, const GroupSpec& mg, const GroupSpec& kg,
                                     int64_t M, int64_t K, int64_t ldo, float2* out, cudaStream_t s);
cudaError_t launch_gather_c64_to_c128(const float2* T, const GroupSpec& mg, const GroupSpec& kg,
                                      int64_t M, int64_t K, int64_t ldo, double2* out, cudaStream_t s);
// Split into bf16 planes: plane p at out + p*pstride, row m at m*ld2, complex k at 2k.
// Columns K <= k < Kp are written as zero (TMA reads the padded extent).
cudaError_t launch_split_c128(const double2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M,
                              int64_t K, int64_t Kp, int nplanes, int64_t pstride,
                              __nv_bfloat16* out, cudaStream_t s);
cudaError_t launch_split_c64(const float2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M,
                             int64_t K, int64_t Kp, int nplanes, int64_t pstride,
                             __nv_bfloat16* out, cudaStream_t s);
// Expanded real operand of a static B [N][K] (complex, row-major) for the tcgen05 path:
// rows (n, c_out), columns (k, c_in): [[Br, -Bi], [Bi, Br]], split into bf16 planes.
// Precomputed element offsets of a gather's rows and columns (device tables) and the
// lane mapping of its load phase.
struct GatherTab {
  const int64_t* om = nullptr;
  const int64_t* ok = nullptr;
  int m_fast = 0;
};
bool gather_m_fast(const GroupSpec& mg, const GroupSpec& kg);
cudaError_t launch_rowmax_tab(const void* T, int is64, const GatherTab& t, int64_t M, int64_t K, float* amax,
                              cudaStream_t s);
cudaError_t launch_split_tab(const void* T, int is64, const GatherTab& t, int64_t M, int64_t K, int64_t Kp,
                             int nplanes, int64_t pstride, __nv_bfloat16* out, cudaStream_t s);
cudaError_t launch_split16_tab(const void* T, int is64, const GatherTab& t, int64_t M, int64_t K, int64_t Kp,
                               int64_t pstride, const float* amax, __nv_bfloat16* out, cudaStream_t s);
// One pass: row maxima (written to amax) and the slice planes together, a cluster of CTAs
// per block of rows; *done = false when a row does not fit the clusters' shared memory.
cudaError_t launch_split16_rows_tab(const void* T, int is64, const GatherTab& t, int64_t M, int64_t K, int64_t Kp,
                                    int64_t pstride, float* amax, __nv_bfloat16* out, cudaStream_t s, bool* done);
cudaError_t launch_split16_rows_grp(const void* T, int is64, const GroupSpec& mg, const GroupSpec& kg, int64_t M,
                                    int64_t K, int64_t Kp, int64_t pstride, float* amax, __nv_bfloat16* out,
                                    cudaStream_t s, bool* done);
cudaError_t launch_gather_tab_to_c128(const void* T, int is64, const GatherTab& t, int64_t M, int64_t K, int64_t ldo,
                                      double2* out, cudaStream_t s);
// fp16 slice planes (2 planes, hi + lo) of a K-major gather, rows scaled by
// fp16_row_scale(amax[m]); launch_rowmax_* first fills amax[m] = max_k max(|re|, |im|).
cudaError_t launch_rowmax_c128(const double2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M, int64_t K,
                               float* amax, cudaStream_t s);
cudaError_t launch_rowmax_c64(const float2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M, int64_t K,
                              float* amax, cudaStream_t s);
cudaError_t launch_split16_c128(const double2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M, int64_t K,
                                int64_t Kp, int64_t pstride, const float* amax, __nv_bfloat16* out, cudaStream_t s);
cudaError_t launch_split16_c64(const float2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M, int64_t K,
                               int64_t Kp, int64_t pstride, const float* amax, __nv_bfloat16* out, cudaStream_t s);
// Static operand as fp16 planes of B' with per-complex-row maxima written to bmax[N].
cudaError_t launch_pack_b_planes_f16(const double2* B, int64_t N, int64_t K, int64_t Kp, int64_t pstride,
                                     __nv_bfloat16* out, float* bmax, cudaStream_t s);
cudaError_t launch_pack_b_planes(const double2* B, int64_t N, int64_t K, int64_t Kp, int nplanes,
                                 int64_t pstride, __nv_bfloat16* out, cudaStream_t s);

// Grouped variants: independent jobs in one launch (per 48 jobs).
constexpr int kGatherJobMax = 48, kGatherTabJobMax = 128;  // jobs per launch: a 4 to 30 KB parameter
struct GatherJob {
  const void* T;
  GroupSpec mg, kg;
  int64_t M, K, Kw;
  void* out;
  int64_t ld;        // complex output: row pitch
  int64_t pstride;   // split output: plane pitch (bf16 elements)
  int nplanes;       // 0: complex output, 2 or 3: bf16 slice planes (row pitch 2*Kw)
  const float* amax = nullptr;  // with nplanes == 2: fp16 planes scaled by these row maxima
  GatherTab tab;                // offset tables, or none
};
struct SmallJob {
  const void* A;
  GroupSpec mg, kg;
  int64_t M;
  int K, N;
  const void* B;
  void* C;
};
cudaError_t launch_gather_grouped(const GatherJob* jobs, int njobs, int in_is64, int out_is64, cudaStream_t s);
int gather_grouped_launches(const GatherJob* jobs, int njobs);  // that it makes
// out[i] = offset of index i of the group (i < n), computed on the device.
cudaError_t launch_offsets_table(const GroupSpec& g, int64_t n, int64_t* out, cudaStream_t s);
// Row maxima of the jobs that carry amax (zeroed first), for their fp16 splits.
cudaError_t launch_rowmax_grouped(const GatherJob* jobs, int njobs, int in_is64, cudaStream_t s);
// Device-resident gather jobs (block-sparse maps): buffers resolved per launch.
struct BlockBases {
  void* buf[6];  // 0 x, 1 y, 2/3 running buffers, 4 staging, 5 fp16 row maxima
};
struct DevGatherJob {
  GroupSpec mg, kg;
  int64_t src_off, dst_off;
  int64_t M, K, Kw, ld, pstride;
  int src_buf, dst_buf;
  int nplanes;   // > 0: bf16 slice planes (row pitch 2*ld), else complex
  int dst_is64;  // complex output element type
  int tiles_m, m_fast;
  int mode;                      // 0 copy / bf16 split, 2 fp16 split (row maxima: launch_block_rowmax)
  int64_t amax_off;              // row maxima of this job's rows: (float*)bases.buf[5] + amax_off
  int tks;                       // log2 of the tile width in K (tile = (1024 >> tks) x (1 << tks))
  int fast_m;                    // M digits by 32-bit multiply-shift division (M < 2^31)
  uint32_t m_mag[GTN_MAXG];      // round-up multipliers of mg.dim (Granlund-Montgomery)
  uint32_t m_sh[GTN_MAXG];
};
void finish_dev_gather_job(DevGatherJob* J);
// tile_map[b] = (job, tile within the job) of CTA b: one load instead of a search.
cudaError_t launch_block_rowmax(const DevGatherJob* jobs, const int2* tile_map, int ntiles, const BlockBases& bases,
                                int src_is64, cudaStream_t s);
cudaError_t launch_block_gather(const DevGatherJob* jobs, const int2* tile_map, int ntiles, const BlockBases& bases,
                                int src_is64, cudaStream_t s);
// Fused gather + product for coupled-charge problems with few output columns (block maps):
// a band is the rows [row_off, row_off + M) of A_q, read straight from the running tensor,
// C_q[n][row_off + m] = sum_j A_q[row_off + m][bcol_j] * B_q[n][bcol_j] over the band's
// present columns j, with no staged copy of A_q.  Column j lives at
// src_j + sum_t digit_t(m) * rstr[rect_j][t]: the digits of m in the band's common row
// groups (the refinement of every rectangle's row groups) and the strides of column j's
// rectangle (source block) in those groups.
struct DevBandCol {
  int64_t src;   // element offset of the column in bases.buf[src_buf] (block offset + column offset)
  int32_t rect;  // its rectangle within the band
  int32_t bcol;  // its column of B_q
};
constexpr int kBandMaxRects = 24, kBandMaxGroups = 6;
struct DevBand {
  int64_t M;       // rows of the band
  int64_t row_off; // its first row in A_q
  int64_t c_off;   // product bands: element offset of C_q[0][row_off] in bases.buf[c_buf]
  int64_t ldc;     // product bands: M_q, the pitch between output columns n
  const void* B;   // product bands: B_q [N][Kq] in the compute type
  int64_t a_off;   // split bands: element offset (halves) of A_q's plane 0 in bases.buf[4]
  int64_t pstride; // split bands: plane pitch (halves)
  int64_t amax_off;  // split bands, fp16: row maxima of A_q at (float*)bases.buf[5] + amax_off
  int N, Kq, Kp, nplanes, c_buf, src_buf;
  int col0, ncol;  // present columns: cols[col0, col0 + ncol)
  int rs0, nrect;  // row strides: rstr[rs0 + rect * ng + t]
  int ng, m_fast;  // common row groups (slowest first); loads run along rows when m_fast
  uint32_t dim[kBandMaxGroups], mag[kBandMaxGroups], sh[kBandMaxGroups];  // group sizes, division magic
};
// A CTA's share of a band: the rows [m0, m0 + nrows).
struct DevBandWork {
  int band, nrows;
  int64_t m0;
};
bool block_band_fits(int64_t N, int64_t Kq, int fp64);
int block_band_rows_per_pass(int maxn);  // rows a CTA covers per pass (one thread per row)
size_t block_band_smem(int maxn, int Kq, int nrect, int fp64, int wide);
// Split bands: the slice planes of a tensor-core problem's A_q built band by band (rows of
// up to 1024 columns staged whole, row maxima reduced in the CTA for fp16), replacing the
// row-maxima pass, the block moves and the K padding of that problem.
constexpr int kSplitBandMaxKp = 1024;
int block_split_band_rows(int Kp, int src_is64);  // rows per pass
size_t block_split_band_smem(int Kp, int nrect, int ng, int ncol, int src_is64);
cudaError_t launch_block_split_band(const DevBand* bands, const DevBandWork* work, int nwork, const DevBandCol* cols,
                                    const int64_t* rstr, const BlockBases& bases, int src_is64, int fp16,
                                    size_t smem, cudaStream_t s);
// wide: 64-bit element offsets (a source buffer of 2^31 elements or more).
cudaError_t launch_block_band(const DevBand* bands, const DevBandWork* work, int nwork, const DevBandCol* cols,
                              const int64_t* rstr, const BlockBases& bases, int src_is64, int fp64, int maxn, int wide,
                              size_t smem, cudaStream_t s);
cudaError_t launch_small_grouped(const SmallJob* jobs, int njobs, int is64, cudaStream_t s);

// C[n][m] = sum_k T[offM(m) + offK(k)] * B[n][k]   (small K; B in shared memory)
cudaError_t launch_small_contract_c128(const double2* T, const GroupSpec& mg, const GroupSpec& kg,
                                       int64_t M, int K, int N, const double2* B, double2* C,
                                       cudaStream_t s);
cudaError_t launch_small_contract_c64(const float2* T, const GroupSpec& mg, const GroupSpec& kg,
                                      int64_t M, int K, int N, const float2* B, float2* C,
                                      cudaStream_t s);
bool small_contract_fits(int K, int N, size_t elem_bytes);

// ---- SIMT GEMMs (gtn_gemm_simt.cu): C[n][m] = sum_k A[m][k] B[n][k] -----------------
cudaError_t launch_cgemm_simt(const float2* A, const float2* B, float2* C, int64_t M, int64_t N,
                              int64_t K, cudaStream_t s);

constexpr int kGemmJobMax = 64;
struct GemmJob {
  const void* A;
  const void* B;
  void* C;
  int64_t M, N, K;
};
cudaError_t launch_gemm_simt_grouped(const GemmJob* jobs, int njobs, int is64, cudaStream_t s);
// Split-K for GEMMs with few output tiles and a long K: the number of K slices (1 = no
// split), and the launchers with a partial-sum workspace P of slices * M * N elements.
int gemm_splitk_slices(int64_t M, int64_t N, int64_t K);
cudaError_t launch_cgemm_simt_splitk(const float2* A, const float2* B, float2* C, int64_t M, int64_t N, int64_t K,
                                     int S, float2* P, cudaStream_t s);
// Skinny grouped GEMM (same contraction) for N <= 32; every job must pass gemm_skinny_fits.
constexpr int kSkinnyMaxSmem = 96 * 1024;
cudaError_t launch_gemm_skinny_grouped(const GemmJob* jobs, int njobs, int is64, cudaStream_t s);
bool gemm_skinny_fits(int64_t N, int64_t K, int is64);

// ---- tcgen05 GEMM (gtn_gemm_tc.cu) ---------------------------------------------------
// Real GEMM on bf16 slice planes: C (complex fp32, [N][M]) from A planes [P][M][2Kp] and
// B planes [P][2N][2Kp].  prods lists (a_plane, b_plane) pairs accumulated in order.
struct TcGemmArgs {
  const __nv_bfloat16* A;  // planes, pitch 2Kp elements per row
  const __nv_bfloat16* B;
  float2* C;
  int64_t M, N, Kp;        // complex dims; Kp = padded K (multiple of 32)
  int a_planes, b_planes;  // number of planes stored (for the tensor-map extents)
  int nprod;
  int prod_a[9], prod_b[9];
  // fp16 slice planes (the planes hold IEEE half bits): row m of A was scaled by
  // fp16_row_scale(a_max[m]) and complex row n of B by fp16_row_scale(b_max[n]); the
  // epilogue divides both out.  Null maxima and fp16 = 0 for bf16 planes.
  int fp16 = 0;
  const float* a_max = nullptr;
  const float* b_max = nullptr;
};

// Power-of-two scale taking a row maximum mx into [2^14, 2^15) (fp16 holds up to 65504):
// 2^(14 - floor(log2 mx)); 1 for a zero or subnormal maximum.
__host__ __device__ inline float fp16_row_scale(float mx) {
  uint32_t b;
  memcpy(&b, &mx, 4);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0) return 1.0f;
  int te = 268 - e;  // biased exponent of 2^(14 - (e - 127))
  te = te < 1 ? 1 : (te > 254 ? 254 : te);
  const uint32_t o = (uint32_t)te << 23;
  float r;
  memcpy(&r, &o, 4);
  return r;
}
// 1 / fp16_row_scale(mx) exactly (a power of two, 2^-127 at the smallest), without a division.
__host__ __device__ inline float fp16_row_scale_inv(float mx) {
  uint32_t b;
  memcpy(&b, &mx, 4);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0) return 1.0f;
  int te = 268 - e;
  te = te < 1 ? 1 : (te > 254 ? 254 : te);
  const int ie = 254 - te;  // biased exponent of 2^(127 - te)
  const uint32_t o = ie > 0 ? (uint32_t)ie << 23 : 0x00400000u;
  float r;
  memcpy(&r, &o, 4);
  return r;
}
cudaError_t launch_tc_gemm(const TcGemmArgs& a, int* errflag, cudaStream_t s, std::string* why);

// ---- FP64-accurate GEMM on the tensor cores (gtn_gemm_f64e.cu) ---------------------------
// C (complex FP64, [N][M]) = A B^T from integer digit planes (7 base-256 digits): A in blocks
// [row tile of 128][16 real k][plane][128][32 bytes], the real-expanded B' in blocks of 64
// rows; row m of A scaled by 2^(1021 - a_exp[m]), complex row n of B by 2^(1021 - b_exp[n])
// (biased exponents of the rows' largest entries).  A row whose exponent lies outside
// [kF64eMinExp, kF64eMaxExp] (infinities, NaN, subnormals, magnitudes beyond 2^+-450) has no digits:
// its outputs are computed again by launch_f64e_repair.
constexpr int kF64eSlices = 7;
constexpr int kF64eRowsA = 128, kF64eRowsB = 64;
constexpr int64_t kF64eMaxK = int64_t(1) << 21;  // the 64-bit sums hold 2^22 real k
constexpr int kF64eMinExp = 1023 - 450, kF64eMaxExp = 1023 + 450;
__host__ __device__ inline bool f64e_no_digits(float E) {
  return E != 0.f && !(E >= (float)kF64eMinExp && E <= (float)kF64eMaxExp);
}
inline size_t f64e_a_bytes(int64_t M, int64_t K) {
  return (size_t)((M + kF64eRowsA - 1) / kF64eRowsA) * ((K + 7) / 8) * kF64eSlices * kF64eRowsA * 32;
}
// The check of FP64 products: magnitudes of an operand's entries (bf16, [k / 8][row][k % 8]); the
// lists of doubtful outputs, over tiles of kF64eCheckM x kF64eCheckN; the eighth digits of B.
constexpr int kF64eCheckM = 128, kF64eCheckN = 64, kF64eCheckChunk = 32;
// Entries among a row's first kF64eWindow that are at least kF64eLarge (bf16 bits of 0.0508): where two
// rows have L of W entries more than W together, L of them meet.  A row without digits counts as
// far below none.
constexpr int kF64eWindow = 128, kF64eNoCount = -(1 << 20);
constexpr uint32_t kF64eLarge = 0x3d50;
inline size_t f64e_mag_bytes(int64_t rows, int64_t K) { return ((size_t)rows * ((K + 7) / 8) * 16 + 255) / 256 * 256; }
// Whether a row of B with that many large entries keeps its eighth digits (others are formed where
// an output wants them).  A map's statics, packed once, keep all; an operand of a one-shot contraction
// only rows of half as many large entries as they have entries or fewer: the products of dense rows
// are sure, and the digits of all rows took 5 of 156 us of an environment at D = 193.
__host__ __device__ inline bool f64e_low_kept(int large, int64_t K, int all) {
  return all || (large >= 0 && 2 * large < (K < kF64eWindow ? (int)K : kF64eWindow));
}
inline size_t f64e_low_bytes(int64_t N, int64_t K) { return (size_t)N * ((K + 7) / 8) * 32; }
inline size_t f64e_list_bytes(int64_t M, int64_t N) {
  const size_t tiles = (size_t)((M + kF64eCheckM - 1) / kF64eCheckM) * ((N + kF64eCheckN - 1) / kF64eCheckN);
  return tiles * kF64eCheckM * kF64eCheckN / kF64eCheckChunk * (kF64eCheckChunk * 2 + 8);
}
// What an FP64 step keeps in its staging buffer behind A's planes: a count, A's magnitudes, the lists.
inline size_t f64e_check_bytes(int64_t M, int64_t N, int64_t K) {
  return 256 + f64e_mag_bytes(M, K) + f64e_list_bytes(M, N);
}
inline size_t f64e_b_bytes(int64_t N, int64_t K) {
  return (size_t)((2 * N + kF64eRowsB - 1) / kF64eRowsB) * ((K + 7) / 8) * kF64eSlices * kF64eRowsB * 32;
}
// Modelled seconds of an FP64 step (M, N, K) on digit planes (split and GEMM) and on the FP64
// pipe; the step takes the faster one.
double f64e_time(double M, double N, double K);
double f64_pipe_time(double M, double N, double K);
struct F64eGemmArgs {
  const void* A = nullptr;
  const void* B = nullptr;
  double2* C = nullptr;
  int64_t M = 0, N = 0, K = 0;
  const float* a_exp = nullptr;
  const float* b_exp = nullptr;
  const uint16_t* a_mag = nullptr;  // magnitudes: the outputs are checked; null: they are not
  const uint16_t* b_mag = nullptr;
  const int* b_large = nullptr;     // large entries of B's rows
  const uint32_t* b_low = nullptr;  // eighth digits of those that keep them (low_all: of all)
  int low_all = 0;
  int* count = nullptr;             // of the check, zeroed by the split
  void* lists = nullptr;            // of the check
  int levels = 8;               // digit products d_i e_j with i + j < levels (7 or 8)
  void* part = nullptr;         // f64e_part_bytes of the product, or null: no tile is shared
};
cudaError_t launch_f64e_gemm(const F64eGemmArgs& a, int sm_count, int* errflag, cudaStream_t s, std::string* why,
                             int* launches);
// Bytes of partial sums of the tiles that CTAs share in a product (0: none are).
size_t f64e_part_bytes(int64_t M, int64_t N, int64_t K, int sm_count);
// The outputs of rows without digits (of A or of B), and with magnitudes those whose digit products
// may miss the bound 2 K 2^-53 sum_k |a_k| |b_k| of an FP64 sum, each summed again on the FP64 pipe from
// the operands: T read in place (offsets from the tables, or the groups where tab has none), B [N][K].
cudaError_t launch_f64e_repair(const F64eGemmArgs& a, const double2* T, const GatherTab& tab, const GroupSpec& mg,
                               const GroupSpec& kg, const double2* B, int sm_count, cudaStream_t s, int* launches);
// Digit planes and row exponents of the running tensor's K-major view (c128) and of a static B [N][K].
cudaError_t launch_split_digits_tab(const double2* T, const GatherTab& t, int64_t M, int64_t K, float* rexp, void* out,
                                    uint16_t* mag, int* count, cudaStream_t s, int* launches);
cudaError_t launch_split_digits_grp(const double2* T, const GroupSpec& mg, const GroupSpec& kg, int64_t M, int64_t K,
                                    float* rexp, void* out, uint16_t* mag, int* count, cudaStream_t s,
                                    int* launches);
cudaError_t launch_pack_b_digits(const double2* B, int64_t N, int64_t K, void* out, float* bexp, uint16_t* mag,
                                 int* large, uint32_t* low, int low_all, cudaStream_t s);
// C[n][m] = sum_k T[offM(m) + offK(k)] B[n][k] on the FP64 pipe, T read in place.  With slices > 1
// (of zgemm_view_slices: few outputs, long K) the k range is cut into that many partial products
// P[slice][n][m], summed in order.
int zgemm_view_slices(int64_t M, int64_t N, int64_t K);
cudaError_t launch_zgemm_view(const double2* T, const GroupSpec& mg, const GroupSpec& kg, const double2* B, double2* C,
                              int64_t M, int64_t N, int64_t K, cudaStream_t s, int slices = 1, double2* P = nullptr,
                              const OutView& ov = OutView());
bool tc_gemm_supported(int cc_major, int cc_minor);
// Independent problems in one launch per kTcGroupMax problems (same product list for all).
constexpr int kTcGroupMax = 64;
cudaError_t launch_tc_gemm_grouped(const TcGemmArgs* probs, int nprob, int* errflag, cudaStream_t s,
                                   std::string* why);

// ---- vector kernels (gtn_blas.cu) --------------------------------------------------
// scratch holds nblk * J partials; with scratch_cap > 0 (its capacity in entries) the grid
// may widen up to 4 * nblk CTAs where that helps.
cudaError_t launch_multidot(const double2* V, int64_t ldv, int J, const double2* w, int64_t n,
                            double2* out /*[J]*/, double2* scratch, int nblk, cudaStream_t s,
                            int64_t scratch_cap = 0);
cudaError_t launch_lincomb(double2* w, double2 beta, const double2* V, int64_t ldv, int J,
                           const double2* coef /*device [J]*/, double2 cscale, int64_t n,
                           cudaStream_t s);
cudaError_t launch_axpby(int64_t n, double2 a, const double2* x, double2 b, double2* y,
                         cudaStream_t s);
int multidot_launch_count(int J);  // kernels one launch_multidot[_f32] of J vectors issues
// FP32-product variants for reorthogonalisation passes of mixed-precision bases.
cudaError_t launch_multidot_f32(const double2* V, int64_t ldv, int J, const double2* w, int64_t n,
                                double2* out /*[J]*/, double2* scratch, int nblk, cudaStream_t s,
                                int64_t scratch_cap = 0);
// w -= sum_j coef[j] V_j (f32: FP32 products); with nrm2 also nrm2[0] = |w|^2 of the result, by way
// of scratch (blocks as for launch_multidot of one vector), and nrm2[1] = *errflag.
cudaError_t launch_update(double2* w, const double2* V, int64_t ldv, int J, const double2* coef /*device [J]*/,
                          int64_t n, bool f32, double2* nrm2, double2* scratch, int nblk, int64_t scratch_cap,
                          const int* errflag, cudaStream_t s);
// w /= sqrt(nrm2), the squared norm read on the device.
cudaError_t launch_unit_scale(double2* w, const double2* nrm2, int64_t n, cudaStream_t s);
// In place: V_j <- sum_{i<m} Q[i * k + j] V_i for j < k (k <= m <= 64, Q real, device).
cudaError_t launch_basis_rotate(double2* V, int64_t ldv, int m, int k, const double* Q, int64_t n,
                                cudaStream_t s);
cudaError_t launch_c64_to_c128(const float2* x, double2* y, int64_t n, cudaStream_t s);
cudaError_t launch_fill_c128(double2* x, double2 v, int64_t n, cudaStream_t s);
// x[i] = (u, v), u and v uniform in [-1, 1), a fixed function of (seed, i).
cudaError_t launch_fill_uniform_c128(double2* x, int64_t n, uint64_t seed, cudaStream_t s);
cudaError_t launch_conj_inplace(double2* x, int64_t n, cudaStream_t s);
// out[a][j][b] = in[a][idx[j]][b] for j < nsel (idx: device int64, entries < Lin)
cudaError_t launch_restrict_leg(const double2* in, double2* out, int64_t A, int64_t Lin, int64_t nsel, int64_t B,
                                const int64_t* idx, cudaStream_t s);
cudaError_t launch_transpose_c128(const double2* in, int64_t rows, int64_t cols, double2* out,
                                  cudaStream_t s);  // out[c][r] = in[r][c]
cudaError_t launch_zero_lower(double2* R, int64_t rows, int64_t cols, cudaStream_t s);
cudaError_t launch_row_norms(const double2* A, int64_t rows, int64_t cols, double* out, cudaStream_t s);
cudaError_t launch_row_phase_conj(double2* A, int64_t rows, int64_t cols, const double2* ph, cudaStream_t s);
cudaError_t launch_diag_scale(double2* A, int64_t rows, int64_t cols, const double* d, int side,
                              cudaStream_t s);
int multidot_blocks(gtn_ctx ctx);

// ---- plans (gtn_plan.cpp) ----------------------------------------------------------
struct PlanStep {
  int operand;             // static operand absorbed
  bool narrow;             // fits the small-K kernel (no permute), which FP32 and batched steps take then
  bool small;              // and takes it in a single FP64 application
  bool tc;                 // tcgen05 path (mixed precisions only)
  int64_t M, K, N, Kp;
  GroupSpec mg, kg;        // access of the running tensor as [M, K]
  std::vector<int> out_labels;       // labels of C = [N legs..., M legs...]
  std::vector<int64_t> out_dims;
  int64_t out_elems;
  // packed static operand (owned by the map)
  double2* b64 = nullptr;          // [N][K] c128 (conj applied)
  float2* b32 = nullptr;           // [N][K] c64
  __nv_bfloat16* bpl = nullptr;    // [P][2N][2Kp] slice planes
  int bplanes = 0;
  int bfp16 = 0;                   // planes hold fp16 slices scaled per complex row by bmax
  float* bmax = nullptr;           // [N] row maxima of the static (fp16 planes)
  GatherTab tab;                   // offset tables of the running tensor's [M, K] view (tc steps)
  int splitk = 1;                  // K slices of the FP32 SIMT GEMM (few output tiles, long K)
  int vslices = 1;                 // K slices of the FP64 product
  // FP64-accurate digit-plane GEMM (FP64 and FP64E plans): planes, row exponents and
  // out-of-range flag of the static; bdig stays null where the FP64 pipe keeps the step
  bool dg = false;
  void* bdig = nullptr;
  float* bexp = nullptr;
  uint16_t* bmag = nullptr;  // magnitudes of the static and the large ones' number (FP64 applications)
  int* blarge = nullptr;
  uint32_t* blow = nullptr;  // and eighth digits
  double macs = 0;
};

// Entry guard of the public calls that run a map: a map owns its workspace and Krylov
// basis, so like the reference's WorkspaceMap (lib/GraftPlanning/src/Planning/
// types.jl:503-552) it is task-local and non-reentrant; a second concurrent call is refused.
struct MapUse {
  gtn_map_s* m;
  bool ok;
  explicit MapUse(gtn_map_s* map);
  ~MapUse();
};
int map_busy_error(gtn_map_s* map);

struct gtn_map_s {
  gtn_ctx ctx = nullptr;
  std::atomic<int> busy{0};  // set while a public call runs on this map (maps are not reentrant)
  int precision = 0;
  std::vector<int64_t> x_dims, y_dims;
  int64_t x_elems = 0, y_elems = 0;
  std::vector<PlanStep> steps;
  GroupSpec fin_mg, fin_kg;  // final permute of the last C into y order
  GatherTab fin_tab;         // its offset tables
  int64_t fin_M = 0, fin_K = 0;
  OutView out;  // the last step's outputs (n, m) in y
  double flops = 0;        // algorithmic FLOPs of the reference's env-first chain
  double exec_flops = 0;   // FLOPs of the executed (possibly grouped) chain
  int n_groups = 0;
  gtn_map fp64_alt = nullptr;  // FP64-optimal plan sharing this map's workspace
  gtn_map fp64_map = nullptr;  // caller-set map serving this map's FP64 applications (not owned)
  int64_t max_t = 0;       // largest running tensor (elements)
  int64_t max_a = 0;       // largest A operand (elements, for permuted / split staging)
  int64_t max_apl = 0;     // largest split-plane staging (bf16 elements per plane * planes)
  int64_t max_mtc = 0;     // largest M of a tensor-core step (fp16 row maxima, digit row exponents)
  size_t max_adg = 0;      // largest digit-plane operand (bytes)
  void* part = nullptr;    // partial sums of its digit-plane products (or null)
  int64_t max_splitk = 0;  // largest split-K partial-sum workspace (complex elements)
  bool oneshot = false;    // a one-shot contraction (gtn_contract): arena allocations, no tables
  char* arena = nullptr;   // allocations come from here first (one-shot contractions)
  size_t arena_cap = 0, arena_off = 0, arena_spill = 0;
  void* skbuf = nullptr;   // that workspace
  float* amax = nullptr;   // [max_mtc] row maxima of the running operand (fp16 planes)
  // device workspace owned by the map
  void* buf0 = nullptr; void* buf1 = nullptr; void* abuf = nullptr;
  void* dx = nullptr; void* dy = nullptr;     // staging for the host-buffer entry point
  int64_t bytes = 0;
  std::vector<void*> owned;
  std::vector<std::pair<void*, size_t>> blocks;  // workspace from the context's block cache
  struct PendingTab {  // offset tables filled on the device once the plan is admitted
    GroupSpec g;
    int64_t n;
    int64_t* d;
  };
  std::vector<PendingTab> pending_tabs;
  // a Krylov operator backed by block-sparse maps instead of a plan (gtn_blockmap_lanczos_*):
  // applications go to bm (its own precision) or, in FP64, to bm64
  struct gtn_blockmap_s* bm = nullptr;
  struct gtn_blockmap_s* bm64 = nullptr;
  // Krylov scratch
  double2* kv = nullptr; int kv_cap = 0;     // (krylovdim+1) vectors
  double2* kcoef = nullptr; double2* kscratch = nullptr; int kscratch_cap = 0;
};

double plan_step_time(int precision, double M, double K, double N, bool oneshot);
int plan_build(gtn_ctx ctx, int n_operands, const int* ranks, const int64_t* dims,
               const int* labels, const int* conj, const int* order, const void* const* statics,
               int precision, gtn_map map, bool allow_group = true, bool alloc_ws = true);
int map_run(gtn_map map, int precision, const double2* x, double2* y);
// One eager application of a block-sparse map (no graph), in its own precision.
int blockmap_run(struct gtn_blockmap_s* bm, const double2* x, double2* y);
int blockmap_precision(struct gtn_blockmap_s* bm);
int map_run_profiled(gtn_map map, int precision, const double2* x, double2* y, int cap, double* ms,
                     int* kind, double* flops, int* count);
void map_free(gtn_map map);
int map_run_batched(gtn_map* maps, int n, int precision, const double2* const* xs, double2* const* ys);
