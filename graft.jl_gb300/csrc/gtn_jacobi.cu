// Singular value decomposition of a matrix with up to 384 columns by Householder QR and one-sided
// Jacobi rotations (Hestenes) on the whole chip: the truncated splits of sweeps at bond dimensions
// of about 30 to 190, for which bidiagonalisation is a chain of latency-bound column steps.
//
//   W = Q R (W the tall side's matrix: A, or A^H of a wide A), R^H = P T, L = T^H, L J = V S, so
//   that W = (Q V) S (P J)^H.  The triangular factors are what makes the rotations converge: on the
//   columns of W itself a decaying spectrum, the usual one of a split, takes 28 sweeps (they are
//   all nearly parallel), on R^H 12, on T^H 8 or 9 (Gaussian matrices: 12, 11, 10); a third
//   factorisation saves less than it takes.
//
// Both parts are dataflow kernels, one CTA per column or column pair, all resident (cooperative
// launches), that hand columns on through L2 without flags or fences: every 64-bit word travels
// with a sequence number in one 16-byte store (relaxed, single-copy atomic), and a reader polls the
// words it needs until they carry the number of its step.  With a version per column behind a fence
// a hand-over took 6000 of a round's 12000 clocks (write drain, poll, load); FP64 itself, two FMAs
// per clock and SM at a latency of about 60 clocks, is the rest.  Sums are trees for the same
// reason, and a rotation's parameters take two reciprocal square roots and an FP32 tangent.
//   * QR: CTA k holds column k, applies the reflectors 0 .. k-1 as they appear, forms its own.
//   * Jacobi: a round of the round-robin schedule rotates n / 2 disjoint pairs of columns of L, one
//     CTA each; a second CTA per pair applies the same rotations to J a little later.  A sweep ends
//     with a grid barrier, the iteration with a sweep that rotated nothing.
// A pair counts as orthogonal when |a^H b| <= eps sqrt(n) |a| |b| (the rounding of the dot product
// itself).  Cosine and phase of a rotation carry full precision (they keep the columns' norms); the
// tangent is formed in FP32, its error only leaves 1e-7 of the overlap to the next sweep.
// Measured against cuSOLVER's gesvd: singular values 1 .. 1e-8, 192 x 192 38.5 -> 11.8 ms, 300 x 300
// 81 -> 22.7 ms, 96 x 400 with columns 1 .. 1e-6 16.5 -> 4.2 ms (one factorisation: 12.7, 26, 4.6).
// On the 192 x 192 split of a DMRG step the second factorisation takes 1.25 ms and saves 4.4 of
// 14.9 ms of sweeps.
// Every wait is bounded (4 s, then a flag ends all CTAs).
#include "gtn_internal.h"

#include <algorithm>
#include <cmath>

namespace {

constexpr int kT = 128;           // threads per CTA
constexpr int kMaxRows = 768;     // rows of W: six per thread
constexpr int kMaxColumns = 384;  // columns of W, order of L: three per thread
constexpr int kQE = kMaxRows / kT, kJE = kMaxColumns / kT;
constexpr int kMaxSweeps = 60;
constexpr uint64_t kWaitNs = 4000000000ull;

struct JacobiState {
  unsigned arrived;           // sweep barrier: CTAs that have arrived so far
  int stop;                   // a wait timed out
  int max_exp;                // largest binary exponent of the input (biased)
  int sweeps;                 // sweeps done
  int rotated[kMaxSweeps];    // whether sweep s rotated a pair
};

// ---- words with sequence numbers --------------------------------------------------------
struct __align__(16) Word {
  double v;
  unsigned long long seq;
};
__device__ __forceinline__ Word ld_word(const Word* p) {
  unsigned long long a, b;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  return Word{__longlong_as_double((long long)a), b};
}
__device__ __forceinline__ void st_word(Word* p, double v, unsigned long long seq) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(seq)
               : "memory");
}
__device__ __forceinline__ void st_complex(Word* p, double2 a, unsigned long long seq) {
  st_word(p, a.x, seq);
  st_word(p + 1, a.y, seq);
}

// A wait's clock: false once it has lasted 4 s or another wait has given up.
struct Patience {
  uint64_t t0 = 0;
  unsigned it = 0;
  __device__ bool more(JacobiState* st, int* errflag) {
    if ((++it & 63u) != 0u) return true;
    uint64_t now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (t0 == 0) t0 = now;
    if (now - t0 <= kWaitNs && !*(volatile int*)&st->stop) return true;
    *(volatile int*)&st->stop = 1;
    atomicCAS(errflag, 0, DEVERR_EPI_TIMEOUT);
    return false;
  }
};

// Rows tid + k kT < rows (from `from` on) of a column of complex words, once all carry seq.
template <int E>
__device__ __forceinline__ bool load_column(const Word* col, int from, int rows, unsigned long long seq,
                                            double2 (&a)[E], JacobiState* st, int* errflag) {
  Patience wait;
  for (;;) {
    bool ready = true;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int x = threadIdx.x + k * kT;
      a[k] = make_double2(0.0, 0.0);
      if (x >= from && x < rows) {
        const Word re = ld_word(col + 2 * x), im = ld_word(col + 2 * x + 1);
        a[k] = make_double2(re.v, im.v);
        ready = ready && re.seq == seq && im.seq == seq;
      }
    }
    if (ready) return true;
    if (!wait.more(st, errflag)) return false;
  }
}

// Sums of R values over the CTA (value v of every thread in red[v]), pairwise, 32 / R lanes of warp
// 0 each; the result of value v in tot[v] after the caller's barrier.
template <int R>
__device__ __forceinline__ void warp_sums(const double (*red)[kT], double* tot) {
  constexpr int G = 32 / R, C = kT / G;
  const int v = threadIdx.x / G, l = threadIdx.x % G;
  double x[C];
#pragma unroll
  for (int k = 0; k < C; ++k) x[k] = red[v][l + G * k];
#pragma unroll
  for (int o = C / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < o; ++k) x[k] += x[k + o];
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) x[0] += __shfl_down_sync(0xffffffffu, x[0], o, G);
  if (l == 0) tot[v] = x[0];
}

// Squared column norms below this are formed on a scaled column: above it, squares lost to
// underflow (below 2^-1074 each) are less than 2^-160 of the sum, and its reciprocal is in range.
constexpr double kTinySquare = 0x1p-900;
__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

__global__ void jacobi_exponent_kernel(const double2* __restrict__ A, int64_t n, JacobiState* st) {
  int e = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 a = A[i];
    e = max(e, max(exponent_of(a.x), exponent_of(a.y)));
  }
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if ((threadIdx.x & 31) == 0) atomicMax(&st->max_exp, e);
}

// x 2^(1023 - e) for the largest exponent e (two exact factors: 1 / 2^e may leave the range).
__device__ __forceinline__ double scaled(double x, int e) {
  const int s = 1023 - min(max(e, 1), 2046), h = s / 2;
  return (x * __longlong_as_double((long long)(1023 + h) << 52)) * __longlong_as_double((long long)(1023 + s - h) << 52);
}

// ---- Householder QR --------------------------------------------------------------------------
// a -= f (v^H a) v with f = conj(tau) (dagger, the factorisation) or tau (applying Q), v from row
// `from` on.
__device__ __forceinline__ void reflect(double2 (&a)[kQE], const double2 (&v)[kQE], double2 f, double (*red)[kT],
                                        double* tot) {
  double dx = 0.0, dy = 0.0;
#pragma unroll
  for (int k = 0; k < kQE; ++k) {
    dx = fma(v[k].x, a[k].x, fma(v[k].y, a[k].y, dx));   // conj(v) a
    dy = fma(v[k].x, a[k].y, fma(-v[k].y, a[k].x, dy));
  }
  red[0][threadIdx.x] = dx;
  red[1][threadIdx.x] = dy;
  __syncthreads();
  if (threadIdx.x < 32) warp_sums<2>(red, tot);
  __syncthreads();
  const double2 g = make_double2(fma(f.x, tot[0], -f.y * tot[1]), fma(f.x, tot[1], f.y * tot[0]));
#pragma unroll
  for (int k = 0; k < kQE; ++k) {
    a[k].x = fma(-g.x, v[k].x, fma(g.y, v[k].y, a[k].x));
    a[k].y = fma(-g.x, v[k].y, fma(-g.y, v[k].x, a[k].y));
  }
}

// CTA k: column k of W (from the row-major A, scaled) or, without A, of the n x n words X.  Reflector k as words of sequence 1 in
// refl[k * rows ..] (from row k on) and tau[k]; row k of R conjugated as column entries of L, and
// the k-th unit column of J, as words of sequence 0 (both zeroed before; without L neither).
__global__ void __launch_bounds__(kT, 3)
    jacobi_qr_kernel(const double2* __restrict__ A, const Word* __restrict__ X, int tall, int rows, int n, Word* refl,
                     Word* tau, Word* L, Word* J, JacobiState* st, int* errflag) {
  __shared__ double red[2][kT];
  __shared__ double tot[2];
  __shared__ double2 alpha;
  __shared__ int emax;
  const int k = blockIdx.x, tid = threadIdx.x, e = st->max_exp;
  double2 a[kQE], v[kQE];
#pragma unroll
  for (int q = 0; q < kQE; ++q) {
    const int x = tid + q * kT;
    a[q] = make_double2(0.0, 0.0);
    if (x < rows) {
      if (A) {
        const double2 t = tall ? A[(int64_t)x * n + k] : A[(int64_t)k * rows + x];
        a[q] = make_double2(scaled(t.x, e), tall ? scaled(t.y, e) : -scaled(t.y, e));
      } else {
        const Word* w = X + ((int64_t)k * rows + x) * 2;
        a[q] = make_double2(w[0].v, w[1].v);
      }
    }
  }
  for (int j = 0; j < k; ++j) {
    int ok = load_column(refl + (int64_t)j * rows * 2, j, rows, 1, v, st, errflag);
    Word tx = ld_word(tau + 2 * j), ty = ld_word(tau + 2 * j + 1);
    for (Patience wait; ok && (tx.seq != 1 || ty.seq != 1);) {
      tx = ld_word(tau + 2 * j);
      ty = ld_word(tau + 2 * j + 1);
      ok = wait.more(st, errflag);
    }
    if (!__syncthreads_and(ok)) return;
    reflect(a, v, make_double2(tx.v, -ty.v), red, tot);
  }
  double x2 = 0.0;
#pragma unroll
  for (int q = 0; q < kQE; ++q) {
    const int x = tid + q * kT;
    if (x > k) x2 = fma(a[q].x, a[q].x, fma(a[q].y, a[q].y, x2));
    if (x == k) alpha = a[q];
  }
  red[0][tid] = x2;
  red[1][tid] = 0.0;
  __syncthreads();
  if (tid < 32) warp_sums<2>(red, tot);
  __syncthreads();
  // LAPACK's reflector: H = 1 - tau v v^H, H^H a = beta e_k, v_k = 1
  double2 al = alpha;
  double r2 = fma(al.x, al.x, fma(al.y, al.y, tot[0]));
  bool tail = tot[0] != 0.0;
  const bool tiny = r2 < kTinySquare;  // the same for every thread
  int ec = 0;
  if (tiny) {
    // What is left of the column lies so far below the matrix's largest entry that its squares (or
    // the reciprocal of their sum) leave the FP64 range: again on the column scaled by its own
    // largest exponent.  A reflector depends only on the column's direction.
    if (tid == 0) emax = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kQE; ++q) {
      const int x = tid + q * kT;
      if (x >= k && x < rows) atomicMax(&emax, max(exponent_of(a[q].x), exponent_of(a[q].y)));
    }
    __syncthreads();
    ec = emax;
    x2 = 0.0;
#pragma unroll
    for (int q = 0; q < kQE; ++q) {
      const int x = tid + q * kT;
      if (x < k) continue;
      a[q] = make_double2(scaled(a[q].x, ec), scaled(a[q].y, ec));
      if (x > k) x2 = fma(a[q].x, a[q].x, fma(a[q].y, a[q].y, x2));
      if (x == k) alpha = a[q];
    }
    red[0][tid] = x2;
    __syncthreads();
    if (tid < 32) warp_sums<2>(red, tot);
    __syncthreads();
    al = alpha;
    r2 = fma(al.x, al.x, fma(al.y, al.y, tot[0]));
    tail = tot[0] != 0.0;
  }
  double2 tk = make_double2(0.0, 0.0), sc = make_double2(0.0, 0.0);
  double beta = al.x;
  if (tail || al.y != 0.0) {
    beta = al.x >= 0.0 ? -sqrt(r2) : sqrt(r2);
    tk = make_double2((beta - al.x) / beta, -al.y / beta);
    const double2 d = make_double2(al.x - beta, al.y);
    const double i2 = 1.0 / fma(d.x, d.x, d.y * d.y);
    sc = make_double2(d.x * i2, -d.y * i2);
  }
  if (tiny) beta = scalbn(beta, max(ec, 1) - 1023);
  if (tid < 2) st_word(tau + 2 * k + tid, tid == 0 ? tk.x : tk.y, 1);
#pragma unroll
  for (int q = 0; q < kQE; ++q) {
    const int x = tid + q * kT;
    if (x >= rows) continue;
    if (x >= k) {
      const double2 u = x == k ? make_double2(1.0, 0.0)
                               : make_double2(fma(sc.x, a[q].x, -sc.y * a[q].y), fma(sc.x, a[q].y, sc.y * a[q].x));
      st_complex(refl + ((int64_t)k * rows + x) * 2, u, 1);
    }
    if (!L) continue;
    if (x < k) st_complex(L + ((int64_t)x * n + k) * 2, make_double2(a[q].x, -a[q].y), 0);
    if (x == k) {
      st_complex(L + ((int64_t)k * n + k) * 2, make_double2(beta, 0.0), 0);
      st_complex(J + ((int64_t)k * n + k) * 2, make_double2(1.0, 0.0), 0);
    }
  }
}

// ---- Jacobi sweeps -------------------------------------------------------------------------------
// The rotation p' = c p - u q, q' = s p + d q of a column pair; u = s e^{-i phi}, d = c e^{-i phi}.
struct Rotation {
  double c, s;
  double2 u, d;
  int turn;
};
__device__ __forceinline__ void rotate(const Rotation& R, double2& a, double2& b) {
  const double2 x = a, y = b;
  a.x = fma(R.c, x.x, fma(-R.u.x, y.x, R.u.y * y.y));
  a.y = fma(R.c, x.y, fma(-R.u.x, y.y, -R.u.y * y.x));
  b.x = fma(R.s, x.x, fma(R.d.x, y.x, -R.d.y * y.y));
  b.y = fma(R.s, x.y, fma(R.d.x, y.y, R.d.y * y.x));
}

// The rotation that makes the columns with squared norms A2, B2 and overlap g = a^H b orthogonal.
__device__ __forceinline__ void make_rotation(double A2, double B2, double gx, double gy, double tol2, Rotation* R) {
  const double g2 = fma(gx, gx, gy * gy), half = 0.5 * (B2 - A2);
  R->turn = g2 > tol2 * A2 * B2 && g2 > 1e-290;
  R->c = 1.0;
  R->s = 0.0;
  R->u = make_double2(0.0, 0.0);
  R->d = make_double2(1.0, 0.0);
  if (!R->turn) return;
  const double ig = rsqrt(g2);
  // tangent of the smaller rotation, t = sgn / (|z| + sqrt(1 + z^2)), z = half / |g|
  const double zd = fabs(half * ig);
  const float z = (float)zd;
  double t = zd < 1e15 ? (double)__fdividef(1.f, z + __fsqrt_rn(fmaf(z, z, 1.f))) : 0.5 / zd;
  if (half < 0.0) t = -t;
  const double w = fma(t, t, 1.0);
  const double c = rsqrt(w), s = t * c;
  const double2 ph = make_double2(gx * ig, -gy * ig);  // e^{-i phi}
  R->c = c;
  R->s = s;
  R->u = make_double2(s * ph.x, s * ph.y);
  R->d = make_double2(c * ph.x, c * ph.y);
}

// CTAs [0, gw): pairs of L; the others: the same pairs of J.  rots: [round of a sweep][pair][6].
__global__ void __launch_bounds__(kT, 4)
    jacobi_sweeps_kernel(Word* L, Word* J, int n, int gw, Word* rots, JacobiState* st, int* errflag) {
  __shared__ double red[4][kT];
  __shared__ double tot[4];
  __shared__ Rotation rot;
  const int tid = threadIdx.x;
  const int P = (n + 1) & ~1, pairs = P / 2;
  const bool isl = (int)blockIdx.x < gw;
  const int first = isl ? blockIdx.x : blockIdx.x - gw, stride = isl ? gw : gridDim.x - gw;
  Word* M = isl ? L : J;
  const double tol2 = 4.93038065763132e-32 * n;  // (2^-52)^2 n
  unsigned long long round = 0;                  // through all sweeps: the sequence a column carries
  int sweep = 0;
  for (; sweep < kMaxSweeps; ++sweep) {
    for (int r = 0; r < P - 1; ++r, ++round) {
      for (int i = first; i < pairs; i += stride) {
        // round robin: every pair once per sweep, the pairs of a round disjoint
        int p = i == 0 ? P - 1 : (r + i) % (P - 1), q = i == 0 ? r : (r + P - 1 - i) % (P - 1);
        if (p > q) { const int t = p; p = q; q = t; }
        Word* mp = M + (int64_t)p * n * 2;
        Word* mq = M + (int64_t)q * n * 2;
        double2 a[kJE], b[kJE];
        int ok = load_column(mp, 0, n, round, a, st, errflag);
        if (q >= n) {  // the bye of an odd column count: hand the column on
          if (!__syncthreads_and(ok)) return;
#pragma unroll
          for (int k = 0; k < kJE; ++k) {
            const int x = tid + k * kT;
            if (x < n) st_complex(mp + 2 * x, a[k], round + 1);
          }
          continue;
        }
        ok = ok && load_column(mq, 0, n, round, b, st, errflag);
        Word* R = rots + ((int64_t)r * pairs + i) * 6;
        if (isl) {
          double al = 0.0, be = 0.0, gx = 0.0, gy = 0.0;
#pragma unroll
          for (int k = 0; k < kJE; ++k) {
            if (k * kT >= n) break;
            al = fma(a[k].x, a[k].x, fma(a[k].y, a[k].y, al));
            be = fma(b[k].x, b[k].x, fma(b[k].y, b[k].y, be));
            gx = fma(a[k].x, b[k].x, fma(a[k].y, b[k].y, gx));   // conj(a) b
            gy = fma(a[k].x, b[k].y, fma(-a[k].y, b[k].x, gy));
          }
          red[0][tid] = al;
          red[1][tid] = be;
          red[2][tid] = gx;
          red[3][tid] = gy;
          if (!__syncthreads_and(ok)) return;
          if (tid < 32) {
            warp_sums<4>(red, tot);
            __syncwarp();
            if (tid == 0) {
              make_rotation(tot[0], tot[1], tot[2], tot[3], tol2, &rot);
              if (rot.turn) st->rotated[sweep] = 1;
            }
            __syncwarp();
            if (tid < 6) st_word(R + tid, reinterpret_cast<const double*>(&rot)[tid], round + 1);
          }
          __syncthreads();
        } else {
          if (tid < 6) {
            Word w = ld_word(R + tid);
            for (Patience wait; ok && w.seq != round + 1;) {
              w = ld_word(R + tid);
              ok = wait.more(st, errflag);
            }
            reinterpret_cast<double*>(&rot)[tid] = w.v;
          }
          if (!__syncthreads_and(ok)) return;
        }
        const Rotation T = rot;
        const bool turn = T.s != 0.0 || T.u.x != 0.0 || T.u.y != 0.0 || T.c != 1.0;
#pragma unroll
        for (int k = 0; k < kJE; ++k) {
          const int x = tid + k * kT;
          if (x < n) {
            if (turn) rotate(T, a[k], b[k]);
            st_complex(mp + 2 * x, a[k], round + 1);
            st_complex(mq + 2 * x, b[k], round + 1);
          }
        }
        __syncthreads();  // rot and red are written again in the next round
      }
    }
    // sweep barrier: has any pair been rotated?
    int ok = 1;
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(&st->arrived, 1u);
      const unsigned want = (unsigned)(sweep + 1) * gridDim.x;
      for (Patience wait; ok;) {
        unsigned x;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(&st->arrived) : "memory");
        if (x >= want) break;
        ok = wait.more(st, errflag);
      }
    }
    if (!__syncthreads_and(ok)) return;
    if (!*(volatile int*)&st->rotated[sweep]) break;
  }
  if (blockIdx.x == 0 && tid == 0) st->sweeps = sweep;
}

// Column norms of L: the singular values.
__global__ void __launch_bounds__(kT) jacobi_norms_kernel(const Word* __restrict__ L, int n, double* __restrict__ nrm) {
  __shared__ double red[1][kT];
  __shared__ double tot[1];
  double x2 = 0.0;
  for (int x = threadIdx.x; x < n; x += kT) {
    const Word* w = L + ((int64_t)blockIdx.x * n + x) * 2;
    x2 = fma(w[0].v, w[0].v, fma(w[1].v, w[1].v, x2));
  }
  red[0][threadIdx.x] = x2;
  __syncthreads();
  if (threadIdx.x < 32) warp_sums<1>(red, tot);
  __syncthreads();
  if (threadIdx.x == 0) nrm[blockIdx.x] = sqrt(tot[0]);
}

// The unit columns ord[0 .. p - 1] of L as words of sequence 0, then zero columns.
__global__ void __launch_bounds__(kT) jacobi_unit_columns_kernel(const Word* __restrict__ L,
                                                                 const double* __restrict__ nrm,
                                                                 const int* __restrict__ ord, int n, int p,
                                                                 Word* __restrict__ X) {
  const int i = blockIdx.x, c = ord[i];
  const double s = nrm[c];
  for (int x = threadIdx.x; x < n; x += kT) {
    const Word* w = L + ((int64_t)c * n + x) * 2;
    st_complex(X + ((int64_t)i * n + x) * 2, i < p ? make_double2(w[0].v / s, w[1].v / s) : make_double2(0.0, 0.0), 0);
  }
}

// a <- H_0 .. H_{count-1} a for the reflectors refl, tau of a `rows`-row matrix.
__device__ __forceinline__ void apply_reflectors(double2 (&a)[kQE], const Word* __restrict__ refl,
                                                 const Word* __restrict__ tau, int count, int rows, double (*red)[kT],
                                                 double* tot) {
  const int tid = threadIdx.x;
  double2 v[kQE], nv[kQE];
  auto fetch = [&](int j, double2 (&t)[kQE]) {
#pragma unroll
    for (int q = 0; q < kQE; ++q) {
      const int x = tid + q * kT;
      t[q] = make_double2(0.0, 0.0);
      if (j >= 0 && x >= j && x < rows) {
        const Word* w = refl + ((int64_t)j * rows + x) * 2;
        t[q] = make_double2(w[0].v, w[1].v);
      }
    }
  };
  fetch(count - 1, v);
  for (int j = count - 1; j >= 0; --j) {
    fetch(j - 1, nv);  // in flight during the reflection
    reflect(a, v, make_double2(tau[2 * j].v, tau[2 * j + 1].v), red, tot);
#pragma unroll
    for (int q = 0; q < kQE; ++q) v[q] = nv[q];
  }
}

// CTA (i, 0): the long vector of the i-th largest triplet, Q times the unit column ord[i] of L, or
// for i >= p (a value of zero, which leaves no direction) Q times the i-th column of the completion
// refl2, tau2 of the unit columns; CTA (i, 1): its short one, P times that column of J.  Tall A:
// U = long (m x r), Vh = short^H; wide: U = short, Vh = long^H.
__global__ void __launch_bounds__(kT, 3)
    jacobi_vectors_kernel(const Word* __restrict__ refl0, const Word* __restrict__ tau0,
                          const Word* __restrict__ refl1, const Word* __restrict__ tau1,
                          const Word* __restrict__ refl2, const Word* __restrict__ tau2, const Word* __restrict__ L,
                          const Word* __restrict__ J, const double* __restrict__ nrm, const int* __restrict__ ord,
                          int tall, int rows0, int n, int r, int p, double2* __restrict__ U, double2* __restrict__ Vh) {
  __shared__ double red[2][kT];
  __shared__ double tot[2];
  const bool is_long = blockIdx.y == 0;
  const int i = blockIdx.x, c = ord[i], tid = threadIdx.x, rows = is_long ? rows0 : n;
  const bool completed = is_long && i >= p;
  const Word* src = is_long ? L : J;
  const double s = is_long ? nrm[c] : 1.0;
  double2 a[kQE];
#pragma unroll
  for (int q = 0; q < kQE; ++q) {
    const int x = tid + q * kT;
    const Word* w = src + ((int64_t)c * n + x) * 2;
    a[q] = x >= n ? make_double2(0.0, 0.0)
           : completed ? make_double2(x == i ? 1.0 : 0.0, 0.0) : make_double2(w[0].v / s, w[1].v / s);
  }
  if (completed) apply_reflectors(a, refl2, tau2, p, n, red, tot);
  apply_reflectors(a, is_long ? refl0 : refl1, is_long ? tau0 : tau1, n, rows, red, tot);
  const bool to_u = (tall != 0) == is_long;
#pragma unroll
  for (int q = 0; q < kQE; ++q) {
    const int x = tid + q * kT;
    if (x < rows) {
      if (to_u) U[(int64_t)x * r + i] = a[q];
      else Vh[(int64_t)i * rows + x] = make_double2(a[q].x, -a[q].y);
    }
  }
}

inline size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// The workspace's parts; the first `zeroed` bytes start as zero.
struct Parts {
  JacobiState* st;
  Word *refl, *tau, *R, *refl2, *tau2, *L, *J, *rots;  // R: R^H of the first factorisation
  double* nrm;
  int* ord;
  size_t zeroed, bytes;
  Parts(void* ws, int64_t rows, int64_t n) {
    char* p = static_cast<char*>(ws);
    size_t o = 0;
    auto take = [&](size_t b) {
      char* q = p + o;
      o += up256(b);
      return q;
    };
    st = reinterpret_cast<JacobiState*>(take(sizeof(JacobiState)));
    refl = reinterpret_cast<Word*>(take(rows * n * 2 * sizeof(Word)));
    tau = reinterpret_cast<Word*>(take(n * 2 * sizeof(Word)));
    R = reinterpret_cast<Word*>(take(n * n * 2 * sizeof(Word)));
    refl2 = reinterpret_cast<Word*>(take(n * n * 2 * sizeof(Word)));
    tau2 = reinterpret_cast<Word*>(take(n * 2 * sizeof(Word)));
    L = reinterpret_cast<Word*>(take(n * n * 2 * sizeof(Word)));
    J = reinterpret_cast<Word*>(take(n * n * 2 * sizeof(Word)));
    rots = reinterpret_cast<Word*>(take(n * ((n + 1) / 2) * 6 * sizeof(Word)));
    zeroed = o;
    nrm = reinterpret_cast<double*>(take(n * sizeof(double)));
    ord = reinterpret_cast<int*>(take(n * sizeof(int)));
    bytes = o;
  }
};

}  // namespace

bool jacobi_svd_applies(int64_t m, int64_t n) {
  return std::min(m, n) >= 2 && std::min(m, n) <= kMaxColumns && std::max(m, n) <= kMaxRows;
}
size_t jacobi_svd_bytes(int64_t m, int64_t n) { return Parts(nullptr, std::max(m, n), std::min(m, n)).bytes; }

// Factorises and rotates; S (host, descending, k = min(m, n) values).  The workspace
// (jacobi_svd_bytes) then holds what jacobi_svd_store makes the vectors of; those of the values
// from `nonzero` on complete the others to an orthonormal set.
int jacobi_svd_run(gtn_ctx ctx, int64_t m, int64_t n, const double2* A, void* ws, std::vector<double>* S) {
  int tall = m >= n ? 1 : 0, rows = (int)std::max(m, n), k = (int)std::min(m, n);
  Parts w(ws, rows, k);
  cudaStream_t s = ctx->stream;
  int qr_sm = 0, sw_sm = 0;
  GTN_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&qr_sm, jacobi_qr_kernel, kT, 0));
  GTN_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sw_sm, jacobi_sweeps_kernel, kT, 0));
  if (qr_sm * ctx->sm_count < k) return GTN_ERR_UNSUPPORTED;  // every CTA has to be resident
  GTN_CUDA_TRY(ctx, cudaMemsetAsync(ws, 0, w.zeroed, s));
  jacobi_exponent_kernel<<<(unsigned)std::min<int64_t>((m * n + 255) / 256, 152 * 4), 256, 0, s>>>(A, m * n, w.st);
  GTN_CUDA_TRY(ctx, cudaGetLastError());
  int* errflag = ctx->d_errflag;
  const Word* none = nullptr;
  const double2* noA = nullptr;
  void* qargs[] = {&A, &none, &tall, &rows, &k, &w.refl, &w.tau, &w.R, &w.J, &w.st, &errflag};
  GTN_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void*)jacobi_qr_kernel, dim3((unsigned)k), dim3(kT), qargs, 0, s));
  void* pargs[] = {&noA, &w.R, &tall, &k, &k, &w.refl2, &w.tau2, &w.L, &w.J, &w.st, &errflag};
  GTN_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void*)jacobi_qr_kernel, dim3((unsigned)k), dim3(kT), pargs, 0, s));
  // one CTA per pair of L and of J where they fit
  int gw = std::max(1, std::min((k + 1) / 2, sw_sm * ctx->sm_count / 2));
  void* args[] = {&w.L, &w.J, &k, &gw, &w.rots, &w.st, &errflag};
  GTN_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void*)jacobi_sweeps_kernel, dim3((unsigned)(2 * gw)), dim3(kT),
                                                args, 0, s));
  jacobi_norms_kernel<<<(unsigned)k, kT, 0, s>>>(w.L, k, w.nrm);
  GTN_CUDA_TRY(ctx, cudaGetLastError());
  ctx->launches += 5;
  std::vector<double> hn(k);
  JacobiState hst;
  GTN_CUDA_TRY(ctx, cudaMemcpyAsync(hn.data(), w.nrm, k * sizeof(double), cudaMemcpyDeviceToHost, s));
  GTN_CUDA_TRY(ctx, cudaMemcpyAsync(&hst, w.st, sizeof(JacobiState), cudaMemcpyDeviceToHost, s));
  const int rc = gtn_ctx_sync(ctx);
  if (rc != GTN_OK) return rc;
  if (hst.sweeps >= kMaxSweeps) return GTN_ERR_UNSUPPORTED;  // did not converge
  for (double v : hn)
    if (!std::isfinite(v)) return GTN_ERR_UNSUPPORTED;  // an infinity or NaN in the input: cuSOLVER's
  std::vector<int> ho(k);
  for (int i = 0; i < k; ++i) ho[i] = i;
  std::stable_sort(ho.begin(), ho.end(), [&](int a, int b) { return hn[a] > hn[b]; });
  S->resize(k);
  const int e = std::min(std::max(hst.max_exp, 1), 2046) - 1023;
  for (int i = 0; i < k; ++i) (*S)[i] = std::ldexp(hn[ho[i]], e);
  GTN_CUDA_TRY(ctx, cudaMemcpyAsync(w.ord, ho.data(), k * sizeof(int), cudaMemcpyHostToDevice, s));
  GTN_CUDA_TRY(ctx, cudaStreamSynchronize(s));  // ho leaves scope
  return GTN_OK;
}

int jacobi_svd_store(gtn_ctx ctx, int64_t m, int64_t n, void* ws, int64_t r, int64_t nonzero, double2* U, double2* Vh) {
  const int tall = m >= n ? 1 : 0, rows = (int)std::max(m, n);
  int k = (int)std::min(m, n), one = 1;
  const Parts w(ws, rows, k);
  cudaStream_t s = ctx->stream;
  // the completion's reflectors lie where the rotations were, its matrix where R^H was
  Word *refl = w.rots, *tau = w.rots + (int64_t)k * k * 2, *X = w.R, *none = nullptr;
  if (nonzero > 0 && nonzero < r) {
    GTN_CUDA_TRY(ctx, cudaMemsetAsync(refl, 0, (size_t)(k * k + k) * 2 * sizeof(Word), s));
    jacobi_unit_columns_kernel<<<(unsigned)k, kT, 0, s>>>(w.L, w.nrm, w.ord, k, (int)nonzero, X);
    GTN_CUDA_TRY(ctx, cudaGetLastError());
    const double2* noA = nullptr;
    int* errflag = ctx->d_errflag;
    JacobiState* st = w.st;
    void* args[] = {&noA, &X, &one, &k, &k, &refl, &tau, &none, &none, &st, &errflag};
    GTN_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void*)jacobi_qr_kernel, dim3((unsigned)k), dim3(kT), args, 0, s));
    ctx->launches += 2;
  }
  jacobi_vectors_kernel<<<dim3((unsigned)r, 2), kT, 0, s>>>(w.refl, w.tau, w.refl2, w.tau2, refl, tau, w.L, w.J, w.nrm,
                                                            w.ord, tall, rows, k, (int)r, (int)nonzero, U, Vh);
  ctx->launches++;
  GTN_CUDA_TRY(ctx, cudaGetLastError());
  return GTN_OK;
}
