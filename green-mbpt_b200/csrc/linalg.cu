// FP64 batched linear algebra: hermitization and inverses.
//
// Matrices up to 64 (the Dyson inverses of nso x nso, the leaves of the larger ones) are inverted in the
// registers of one CTA each (gj_small_kernel).  The NQ x NQ Hermitian aux-basis matrices of the screened
// interaction, I - P0, are positive definite for every physical polarization: they are split into blocks down to
// such leaves and put together by batched matrix products (invert_large_batched).  A matrix that turns out not to
// be positive definite is inverted instead by Gauss-Jordan with partial pivoting on an augmented [B | I] in a
// global scratch buffer, one CTA per matrix: blocked by panels of 16 pivots when the panel fits shared memory, one
// pivot at a time otherwise.
#include <algorithm>

#include "context.cuh"

namespace gb200 {
namespace {

__global__ void hermitize_kernel(cplx* X, int64_t nmat, int n, double scale) {
  const int64_t npairs = (int64_t)n * (n + 1) / 2;
  const int64_t total = nmat * npairs;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t m = e / npairs;
    int64_t p = e - m * npairs;
    // p -> (i, j) with i >= j
    int i = (int)((sqrt(8.0 * (double)p + 1.0) - 1.0) * 0.5);
    while ((int64_t)i * (i + 1) / 2 > p) --i;
    while ((int64_t)(i + 1) * (i + 2) / 2 <= p) ++i;
    int j = (int)(p - (int64_t)i * (i + 1) / 2);
    cplx* M = X + m * (int64_t)n * n;
    cplx a = cscale(M[(int64_t)i * n + j], scale);
    cplx b = cscale(M[(int64_t)j * n + i], scale);
    cplx h = cscale(cadd(a, cconj(b)), 0.5);
    M[(int64_t)i * n + j] = h;
    M[(int64_t)j * n + i] = cconj(h);
  }
}

__global__ void scale_kernel(cplx* X, int64_t count, double s) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count; e += (int64_t)gridDim.x * blockDim.x) {
    X[e] = cscale(X[e], s);
  }
}

__device__ __forceinline__ cplx crecip(cplx a) {
  double d = a.x * a.x + a.y * a.y;
  return make_double2(a.x / d, -a.y / d);
}

// Block-wide argmax of |aug[i][j]|^2 over i in [j, n).
template <int NT>
__device__ int pivot_search(const cplx* aug, int64_t ld, int j, int n, double* sval, int* sidx) {
  double best = -1.0;
  int bi = j;
  for (int i = j + threadIdx.x; i < n; i += NT) {
    double v = cabs2(aug[(int64_t)i * ld + j]);
    if (v > best) { best = v; bi = i; }
  }
  sval[threadIdx.x] = best;
  sidx[threadIdx.x] = bi;
  __syncthreads();
  for (int s = NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      double o = sval[threadIdx.x + s];
      int oi = sidx[threadIdx.x + s];
      if (o > sval[threadIdx.x] || (o == sval[threadIdx.x] && oi < sidx[threadIdx.x])) {
        sval[threadIdx.x] = o;
        sidx[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  int p = sidx[0];
  __syncthreads();
  return p;
}

// In-place Gauss-Jordan inverse of an n x n matrix in the registers of one CTA: thread (ti, tj) of the TI x 16 grid
// holds the elements (ti + TI a, tj + 16 b).  Step k publishes column k and the scaled pivot row in shared memory and
// every thread updates its elements from them; rows stay where they are and the pivot order is undone when the result
// is stored.  The block of 16 columns that k lies in is a compile-time index, and column k and the pivot row are
// cleared by their holders, so the update is 6 RI CJ FP64 operations and nothing else.  PIVOT: partial pivoting (every
// warp finds the largest unused element of the column by itself, two barriers a step); otherwise the diagonal in order,
// one barrier a step, and a pivot that is not positive is reported.
// Against the augmented matrix in shared memory that it replaced, 15000 matrices of n = 40: 4.96 -> 1.13 ms, with the
// assembly of the matrices and the trace in the same pass (0.12 + 0.55 ms before).
// Many matrices (the Dyson step): 128 threads each, five of them on an SM, which cover one another's barriers and
// pivot searches.  Few matrices (the screened interaction): 256 threads each, because only the latency counts.
template <int NTH>
struct GjGrid {
  static constexpr int TJ = 16, TI = NTH / TJ;
};

struct GjShared {
  cplx col[2][64], row[2][64];
  int order[64];   // order[k]: the row that was pivot k
  int place[64];   // its inverse
};

// x -> 1 / x with one reciprocal
__device__ __forceinline__ cplx gj_recip(cplx a) {
  const double r = __drcp_rn(fma(a.x, a.x, a.y * a.y));
  return cmk(a.x * r, -a.y * r);
}

template <int NTH, int RI, int CJ, bool PIVOT>
__device__ __forceinline__ bool gj_invert(cplx (&m)[RI][CJ], int n, GjShared& sh) {
  constexpr int TI = GjGrid<NTH>::TI, TJ = GjGrid<NTH>::TJ;
  const int tid = threadIdx.x, ti = tid / TJ, tj = tid % TJ, lane = tid % 32;
  uint64_t used = 0;
  bool ok = true;
#pragma unroll
  for (int kb = 0; kb < CJ; ++kb) {
    for (int kk = 0; kk < TJ; ++kk) {
      const int k = kb * TJ + kk, buf = k & 1;
      if (k >= n) break;
      if (tj == kk) {
#pragma unroll
        for (int a = 0; a < RI; ++a) sh.col[buf][ti + TI * a] = m[a][kb];
      }
      int p = k;
      if constexpr (PIVOT) {
        __syncthreads();
        // the high words of non-negative doubles order like the numbers; ties (within 2^-20) go to the lowest lane, and
        // to the smaller row of a lane's two
        int best = -1, row = 0;
#pragma unroll
        for (int h = 0; h < (RI * TI > 32 ? 2 : 1); ++h) {
          const int r = lane + 32 * h;
          if (r < n && !((used >> r) & 1)) {
            const int key = __double2hiint(cabs2(sh.col[buf][r])) & 0x7fffffff;
            if (key > best) {
              best = key;
              row = r;
            }
          }
        }
        const int top = __reduce_max_sync(0xffffffffu, best);
        const unsigned cand = __ballot_sync(0xffffffffu, best == top);
        p = __shfl_sync(0xffffffffu, row, __ffs(cand) - 1);
        if (tid == 0) {
          sh.order[k] = p;
          sh.place[p] = k;
        }
      }
      used |= 1ull << p;
      const int pi = p % TI, pa = p / TI;
      if (tid / 32 == pi * TJ / 32) {  // the warp that holds row p
        cplx r[CJ];
#pragma unroll
        for (int b = 0; b < CJ; ++b) {
          r[b] = m[0][b];
#pragma unroll
          for (int a = 1; a < RI; ++a)
            if (a == pa) r[b] = m[a][b];
        }
        cplx piv;
        if constexpr (PIVOT) {
          piv = sh.col[buf][p];
        } else {
          const int src = (pi * TJ + kk) % 32;
          piv.x = __shfl_sync(0xffffffffu, r[kb].x, src);
          piv.y = __shfl_sync(0xffffffffu, r[kb].y, src);
          ok = ok && piv.x > 0.0;
        }
        const cplx inv = gj_recip(piv);
        if (ti == pi) {
#pragma unroll
          for (int b = 0; b < CJ; ++b) sh.row[buf][tj + TJ * b] = (b == kb && tj == kk) ? inv : cmul(r[b], inv);
#pragma unroll
          for (int a = 0; a < RI; ++a)
            if (a == pa) {
#pragma unroll
              for (int b = 0; b < CJ; ++b) m[a][b] = cmk(0.0, 0.0);
            }
        }
      }
      if (tj == kk) {
#pragma unroll
        for (int a = 0; a < RI; ++a) m[a][kb] = cmk(0.0, 0.0);
      }
      __syncthreads();
      cplx r[CJ];
#pragma unroll
      for (int b = 0; b < CJ; ++b) r[b] = sh.row[buf][tj + TJ * b];
#pragma unroll
      for (int a = 0; a < RI; ++a) {
        cplx f = sh.col[buf][ti + TI * a];
        if (ti + TI * a == p) f = cmk(-1.0, 0.0);
#pragma unroll
        for (int b = 0; b < CJ; ++b) {
          // the product first, then one subtraction: an element much larger than the product is rounded once (two
          // chained FMAs: 1.0 ms instead of 1.13, but an error of 2.4e-15 where the augmented form had 2.0e-15)
          cplx& e = m[a][b];
          e.x += fma(-f.x, r[b].x, f.y * r[b].y);
          e.y -= fma(f.x, r[b].y, f.y * r[b].x);
        }
      }
    }
  }
  __syncthreads();  // the pivot order is complete
  return ok;
}

// What a CTA inverts and what becomes of the result.
enum GjMode {
  GJ_HERM,     // the Hermitian matrix of the lower triangle and real diagonal of A or I - A -> Ainv, with pivoting
  GJ_LEAF,     // a positive definite diagonal block in place; bad[matrix] = 1 if it is not
  GJ_DYSON,    // z S - X -> Ainv, z = mu + i w of the matrix's frequency
  GJ_TRACE,    // z S - X -> sum_ij (inverse)_ij S_ji
};

struct GjJob {
  const cplx* A = nullptr;
  cplx* out = nullptr;
  int64_t stride = 0;  // elements between matrices
  int64_t nmat = 0;
  int ld = 0, n = 0;
  bool identity_minus = false;
  int* bad = nullptr;
  // GJ_DYSON, GJ_TRACE: X is A, S [nsk][n][n], wn [nw]; matrix m has frequency m / nsk and S block m % nsk
  const cplx* S = nullptr;
  const double* wn = nullptr;
  double mu = 0.0;
  int nsk = 1;
};

template <int NTH, int RI, int MODE>
__global__ void __launch_bounds__(NTH, NTH == 128 ? (RI <= 5 ? 5 : 3) : 2) gj_small_kernel(GjJob j) {
  constexpr int TI = GjGrid<NTH>::TI, TJ = GjGrid<NTH>::TJ, CJ = (RI * TI + TJ - 1) / TJ;
  __shared__ GjShared sh;
  __shared__ double red[2][NTH / 32];
  const int n = j.n, ti = threadIdx.x / TJ, tj = threadIdx.x % TJ;
  const int64_t mat = blockIdx.x;
  const cplx* A = j.A + mat * j.stride;
  const cplx* S = (MODE == GJ_DYSON || MODE == GJ_TRACE) ? j.S + (mat % j.nsk) * (int64_t)n * n : nullptr;
  const cplx z = (MODE == GJ_DYSON || MODE == GJ_TRACE) ? cmk(j.mu, j.wn[mat / j.nsk]) : cmk(0.0, 0.0);
  cplx m[RI][CJ];
#pragma unroll
  for (int a = 0; a < RI; ++a)
#pragma unroll
    for (int b = 0; b < CJ; ++b) {
      const int i = ti + TI * a, c = tj + TJ * b;
      cplx v = cmk(0.0, 0.0);
      if (i < n && c < n) {
        if constexpr (MODE == GJ_HERM) {
          v = i >= c ? A[(int64_t)i * j.ld + c] : cconj(A[(int64_t)c * j.ld + i]);
          if (j.identity_minus) v = cmk((i == c ? 1.0 : 0.0) - v.x, -v.y);
          if (i == c) v.y = 0.0;
        } else {
          v = A[(int64_t)i * j.ld + c];
          if constexpr (MODE == GJ_DYSON || MODE == GJ_TRACE) v = csub(cmul(z, S[i * n + c]), v);
        }
      }
      m[a][b] = v;
    }
  const bool ok = gj_invert<NTH, RI, CJ, MODE != GJ_LEAF>(m, n, sh);
  if constexpr (MODE == GJ_LEAF) {
    if (!ok) j.bad[mat] = 1;
  }
  double re = 0.0, im = 0.0;
#pragma unroll
  for (int a = 0; a < RI; ++a)
#pragma unroll
    for (int b = 0; b < CJ; ++b) {
      int i = ti + TI * a, c = tj + TJ * b;
      if (i >= n || c >= n) continue;
      if constexpr (MODE != GJ_LEAF) {
        i = sh.place[i];
        c = sh.order[c];
      }
      if constexpr (MODE == GJ_TRACE) {
        const cplx t = cmul(m[a][b], S[c * n + i]);
        re += t.x;
        im += t.y;
      } else {
        j.out[mat * j.stride + (int64_t)i * j.ld + c] = m[a][b];
      }
    }
  if constexpr (MODE == GJ_TRACE) {
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (threadIdx.x % 32 == 0) {
      red[0][threadIdx.x / 32] = re;
      red[1][threadIdx.x / 32] = im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      re = im = 0.0;
      for (int w = 0; w < NTH / 32; ++w) {
        re += red[0][w];
        im += red[1][w];
      }
      j.out[mat] = cmk(re, im);
    }
  }
}

template <int NTH, int RI, int MODE>
void launch_gj_one(const GjJob& j, cudaStream_t st) {
  gj_small_kernel<NTH, RI, MODE><<<(unsigned)j.nmat, NTH, 0, st>>>(j);
  GB_CHECK_LAUNCH();
}

// The thread count follows what a call has: the Dyson modes invert thousands of matrices, the modes of the screened
// interaction one per frequency.
template <int MODE>
void launch_gj(const GjJob& j, int64_t nmat, cudaStream_t st) {
  constexpr bool many = MODE == GJ_DYSON || MODE == GJ_TRACE;
  for (int64_t off = 0; off < nmat; off += 2147483647LL) {
    GjJob q = j;
    q.nmat = std::min<int64_t>(nmat - off, 2147483647LL);
    q.A += off * j.stride;
    if (MODE != GJ_TRACE) q.out += off * j.stride;
    if constexpr (many) {
      switch ((j.n + 7) / 8) {
        case 1: launch_gj_one<128, 1, MODE>(q, st); break;
        case 2: launch_gj_one<128, 2, MODE>(q, st); break;
        case 3: launch_gj_one<128, 3, MODE>(q, st); break;
        case 4: launch_gj_one<128, 4, MODE>(q, st); break;
        case 5: launch_gj_one<128, 5, MODE>(q, st); break;
        case 6: launch_gj_one<128, 6, MODE>(q, st); break;
        case 7: launch_gj_one<128, 7, MODE>(q, st); break;
        default: launch_gj_one<128, 8, MODE>(q, st); break;
      }
    } else {
      switch ((j.n + 15) / 16) {
        case 1: launch_gj_one<256, 1, MODE>(q, st); break;
        case 2: launch_gj_one<256, 2, MODE>(q, st); break;
        case 3: launch_gj_one<256, 3, MODE>(q, st); break;
        default: launch_gj_one<256, 4, MODE>(q, st); break;
      }
    }
  }
}

// B = the Hermitian matrix of the lower triangle and real diagonal of A or I - A (what Eigen's LDLT reads,
// gw_cpu_kernel.cpp:245-249)
__global__ void herm_from_lower_kernel(const cplx* A, cplx* B, int64_t nmat, int n, bool identity_minus) {
  const int64_t n2 = (int64_t)n * n, total = nmat * n2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = e / n2;
    const int r = (int)(e - m * n2), i = r / n, c = r - i * n;
    cplx v = i >= c ? A[e] : cconj(A[m * n2 + (int64_t)c * n + i]);
    if (identity_minus) v = cmk((i == c ? 1.0 : 0.0) - v.x, -v.y);
    if (i == c) v.y = 0.0;
    B[e] = v;
  }
}

// The block of `size` rows at `off` of each matrix made Hermitian: its two diagonal blocks (n1 and size - n1) by
// averaging, the upper off-diagonal block from the lower one.
__global__ void herm_join_kernel(cplx* B, int64_t nmat, int n, int off, int size, int n1) {
  const int64_t s2 = (int64_t)size * size, total = nmat * s2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = e / s2;
    const int r = (int)(e - m * s2), i = r / size, c = r - i * size;
    if (c > i) continue;
    cplx* M = B + m * (int64_t)n * n + (int64_t)off * n + off;
    cplx* lo = M + (int64_t)i * n + c;
    cplx* up = M + (int64_t)c * n + i;
    cplx v = *lo;
    if (!(i >= n1 && c < n1)) v = cscale(cadd(v, cconj(*up)), 0.5);
    *lo = v;
    if (c != i) *up = cconj(v);
  }
}

constexpr int LARGE_NT = 1024;

__global__ void __launch_bounds__(LARGE_NT) invert_large_kernel(const cplx* A, cplx* Ainv, cplx* augbase, int n,
                                                                 bool identity_minus, const int* bad) {
  if (!bad[blockIdx.x]) return;
  extern __shared__ double2 smem_c[];
  cplx* prow = smem_c;           // 2n (pivot row)
  cplx* fac = prow + 2 * n;      // n
  __shared__ double sval[LARGE_NT];
  __shared__ int sidx[LARGE_NT];
  const int64_t m = blockIdx.x;
  const int ld = 2 * n;
  cplx* aug = augbase + m * (int64_t)n * ld;
  const cplx* Am = A + m * (int64_t)n * n;
  for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += LARGE_NT) {
    int i = (int)(e / n), c = (int)(e % n);
    // B = identity_minus ? I - A : A ; the inverted matrix is the Hermitian one of B's strict lower triangle and real
    // diagonal (what Eigen's LDLT reads, gw_cpu_kernel.cpp:245-249)
    auto Bel = [&](int x, int y) -> cplx {
      cplx a = Am[(int64_t)x * n + y];
      return identity_minus ? cmk((x == y ? 1.0 : 0.0) - a.x, -a.y) : a;
    };
    cplx v;
    if (i > c) v = Bel(i, c);
    else if (i < c) v = cconj(Bel(c, i));
    else v = cmk(Bel(i, i).x, 0.0);
    aug[(int64_t)i * ld + c] = v;
    aug[(int64_t)i * ld + n + c] = (i == c) ? cmk(1.0, 0.0) : cmk(0.0, 0.0);
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    int p = pivot_search<LARGE_NT>(aug, ld, j, n, sval, sidx);
    if (p != j) {
      for (int c = threadIdx.x; c < ld; c += LARGE_NT) {
        cplx t = aug[(int64_t)j * ld + c];
        aug[(int64_t)j * ld + c] = aug[(int64_t)p * ld + c];
        aug[(int64_t)p * ld + c] = t;
      }
      __syncthreads();
    }
    cplx inv = crecip(aug[(int64_t)j * ld + j]);
    for (int c = threadIdx.x; c < ld; c += LARGE_NT) prow[c] = cmul(aug[(int64_t)j * ld + c], inv);
    for (int i = threadIdx.x; i < n; i += LARGE_NT) fac[i] = aug[(int64_t)i * ld + j];
    __syncthreads();
    for (int c = threadIdx.x; c < ld; c += LARGE_NT) aug[(int64_t)j * ld + c] = prow[c];
    const int w = ld - j;
    for (int64_t e = threadIdx.x; e < (int64_t)n * w; e += LARGE_NT) {
      int i = (int)(e / w), c = j + (int)(e % w);
      if (i == j) continue;
      aug[(int64_t)i * ld + c] = csub(aug[(int64_t)i * ld + c], cmul(fac[i], prow[c]));
    }
    __syncthreads();
  }
  cplx* Om = Ainv + m * (int64_t)n * n;
  for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += LARGE_NT) {
    int i = (int)(e / n), c = (int)(e % n);
    Om[e] = aug[(int64_t)i * ld + n + c];
  }
}

// Blocked Gauss-Jordan with partial pivoting, one CTA per matrix (the aux-basis inverses of the
// screened interaction).  The augmented [B | I] lives in a global scratch buffer; rows are kept in
// a logical order through a permutation instead of being swapped.  Per panel of BLK_NB columns:
//   1. the panel is copied to shared memory and eliminated there to choose the pivot rows J
//      (the same choices as unblocked Gauss-Jordan with partial pivoting);
//   2. D = B[J, panel] (original values) is inverted in shared memory;
//   3. the remaining columns are updated in chunks:  R = D^-1 B[J, :],  B[J, :] = R,
//      B[i, :] -= B[i, panel] R for every other row i  (a rank-BLK_NB update, R in registers).
// The traffic through L2 is one read and one write of the remaining columns per panel instead
// of one per pivot.
constexpr int BLK_NB = 16, BLK_NT = 512, BLK_CH = 128;

__device__ __forceinline__ void block_argmax(double v, int idx, double* sval, int* sidx, int& best_idx) {
  // block-wide argmax of v (ties: smaller idx); every thread gets the result
  sval[threadIdx.x] = v;
  sidx[threadIdx.x] = idx;
  __syncthreads();
  for (int s = BLK_NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      const double o = sval[threadIdx.x + s];
      const int oi = sidx[threadIdx.x + s];
      if (o > sval[threadIdx.x] || (o == sval[threadIdx.x] && oi < sidx[threadIdx.x])) {
        sval[threadIdx.x] = o;
        sidx[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  best_idx = sidx[0];
  __syncthreads();
}

__global__ void __launch_bounds__(BLK_NT) invert_blocked_kernel(const cplx* A, cplx* Ainv, cplx* augbase, int n,
                                                                bool identity_minus, const int* bad) {
  if (!bad[blockIdx.x]) return;
  extern __shared__ double2 smem_c[];
  cplx* pan = smem_c;                        // [n][BLK_NB]: panel copy, then the original panel rows
  cplx* dinv = pan + (size_t)n * BLK_NB;     // [BLK_NB][2*BLK_NB]: D | I -> I | D^-1
  cplx* rch = dinv + 2 * BLK_NB * BLK_NB;    // [BLK_NB][BLK_CH]: R for one column chunk
  int* perm = reinterpret_cast<int*>(rch + BLK_NB * BLK_CH);  // logical row -> physical row
  __shared__ double sval[BLK_NT];
  __shared__ int sidx[BLK_NT];
  const int64_t m = blockIdx.x;
  const int ld = 2 * n;
  cplx* aug = augbase + m * (int64_t)n * ld;
  const cplx* Am = A + m * (int64_t)n * n;
  for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += BLK_NT) {
    const int i = (int)(e / n), c = (int)(e % n);
    auto Bel = [&](int x, int y) -> cplx {
      cplx a = Am[(int64_t)x * n + y];
      return identity_minus ? cmk((x == y ? 1.0 : 0.0) - a.x, -a.y) : a;
    };
    cplx v;
    if (i > c) v = Bel(i, c);
    else if (i < c) v = cconj(Bel(c, i));
    else v = cmk(Bel(i, i).x, 0.0);
    aug[(int64_t)i * ld + c] = v;
    aug[(int64_t)i * ld + n + c] = (i == c) ? cmk(1.0, 0.0) : cmk(0.0, 0.0);
  }
  for (int i = threadIdx.x; i < n; i += BLK_NT) perm[i] = i;
  __syncthreads();
  for (int j0 = 0; j0 < n; j0 += BLK_NB) {
    const int nb = min(BLK_NB, n - j0);
    // 1. panel elimination in shared memory (logical row order) to choose the pivots
    for (int e = threadIdx.x; e < n * BLK_NB; e += BLK_NT) {
      const int li = e / BLK_NB, c = e % BLK_NB;
      pan[e] = c < nb ? aug[(int64_t)perm[li] * ld + j0 + c] : cmk(0.0, 0.0);
    }
    __syncthreads();
    for (int c = 0; c < nb; ++c) {
      const int jr = j0 + c;
      double best = -1.0;
      int bi = jr;
      for (int li = jr + threadIdx.x; li < n; li += BLK_NT) {
        const double v = cabs2(pan[li * BLK_NB + c]);
        if (v > best) { best = v; bi = li; }
      }
      int p;
      block_argmax(best, bi, sval, sidx, p);
      if (p != jr) {
        if (threadIdx.x < BLK_NB) {
          const cplx t = pan[jr * BLK_NB + threadIdx.x];
          pan[jr * BLK_NB + threadIdx.x] = pan[p * BLK_NB + threadIdx.x];
          pan[p * BLK_NB + threadIdx.x] = t;
        }
        if (threadIdx.x == 0) {
          const int t = perm[jr];
          perm[jr] = perm[p];
          perm[p] = t;
        }
      }
      __syncthreads();
      const cplx inv = crecip(pan[jr * BLK_NB + c]);
      __syncthreads();
      if (threadIdx.x < BLK_NB) pan[jr * BLK_NB + threadIdx.x] = cmul(pan[jr * BLK_NB + threadIdx.x], inv);
      __syncthreads();
      for (int e = threadIdx.x; e < n * BLK_NB; e += BLK_NT) {
        const int li = e / BLK_NB, cc = e % BLK_NB;
        if (li == jr || cc <= c) continue;
        pan[e] = csub(pan[e], cmul(pan[li * BLK_NB + c], pan[jr * BLK_NB + cc]));
      }
      __syncthreads();
      for (int li = threadIdx.x; li < n; li += BLK_NT)
        if (li != jr) pan[li * BLK_NB + c] = cmk(0.0, 0.0);
      __syncthreads();
    }

    // 2. original panel values in logical row order (pan) and [D | I] for the pivot block
    for (int e = threadIdx.x; e < n * BLK_NB; e += BLK_NT) {
      const int li = e / BLK_NB, c = e % BLK_NB;
      pan[e] = c < nb ? aug[(int64_t)perm[li] * ld + j0 + c] : cmk(0.0, 0.0);
    }
    for (int e = threadIdx.x; e < BLK_NB * 2 * BLK_NB; e += BLK_NT) {
      const int r = e / (2 * BLK_NB), c = e % (2 * BLK_NB);
      cplx v;
      if (c < BLK_NB) v = (r < nb && c < nb) ? aug[(int64_t)perm[j0 + r] * ld + j0 + c] : cmk(r == c ? 1.0 : 0.0, 0.0);
      else v = cmk(c - BLK_NB == r ? 1.0 : 0.0, 0.0);
      dinv[e] = v;
    }
    __syncthreads();
    // D^-1 by Gauss-Jordan with partial pivoting on [D | I] (512 threads = 16 x 32 entries)
    for (int c = 0; c < BLK_NB; ++c) {
      if (threadIdx.x == 0) {
        int pr = c;
        double b = cabs2(dinv[c * 2 * BLK_NB + c]);
        for (int r = c + 1; r < BLK_NB; ++r) {
          const double v = cabs2(dinv[r * 2 * BLK_NB + c]);
          if (v > b) { b = v; pr = r; }
        }
        sidx[0] = pr;
      }
      __syncthreads();
      const int pr = sidx[0];
      if (pr != c && threadIdx.x < 2 * BLK_NB) {
        const cplx t = dinv[c * 2 * BLK_NB + threadIdx.x];
        dinv[c * 2 * BLK_NB + threadIdx.x] = dinv[pr * 2 * BLK_NB + threadIdx.x];
        dinv[pr * 2 * BLK_NB + threadIdx.x] = t;
      }
      __syncthreads();
      const cplx inv = crecip(dinv[c * 2 * BLK_NB + c]);
      __syncthreads();
      if (threadIdx.x < 2 * BLK_NB) dinv[c * 2 * BLK_NB + threadIdx.x] = cmul(dinv[c * 2 * BLK_NB + threadIdx.x], inv);
      __syncthreads();
      {
        const int r = threadIdx.x / (2 * BLK_NB), cc = threadIdx.x % (2 * BLK_NB);
        const cplx f = (r != c) ? dinv[r * 2 * BLK_NB + c] : cmk(0.0, 0.0);
        __syncthreads();
        if (r != c) dinv[r * 2 * BLK_NB + cc] = csub(dinv[r * 2 * BLK_NB + cc], cmul(f, dinv[c * 2 * BLK_NB + cc]));
      }
      __syncthreads();
    }
    // 3. remaining columns in chunks: R = D^-1 B[J, chunk]; B[J, chunk] = R; other rows -= C R
    for (int col0 = j0 + nb; col0 < ld; col0 += BLK_CH) {
      const int cw = min(BLK_CH, ld - col0);
      for (int e = threadIdx.x; e < BLK_NB * BLK_CH; e += BLK_NT) {
        const int r = e / BLK_CH, cc = e % BLK_CH;
        cplx acc = cmk(0.0, 0.0);
        if (r < nb && cc < cw)
          for (int k = 0; k < nb; ++k)
            acc = cadd(acc, cmul(dinv[r * 2 * BLK_NB + BLK_NB + k], aug[(int64_t)perm[j0 + k] * ld + col0 + cc]));
        rch[e] = acc;
      }
      __syncthreads();
      const int cc = threadIdx.x % BLK_CH, grp = threadIdx.x / BLK_CH;
      if (cc < cw) {
        cplx rr[BLK_NB];
#pragma unroll
        for (int k = 0; k < BLK_NB; ++k) rr[k] = rch[k * BLK_CH + cc];
        for (int li = grp; li < n; li += BLK_NT / BLK_CH) {
          cplx* dst = aug + (int64_t)perm[li] * ld + col0 + cc;
          if (li >= j0 && li < j0 + nb) {
            *dst = rch[(li - j0) * BLK_CH + cc];
            continue;
          }
          cplx v = *dst;
          const cplx* cl = pan + li * BLK_NB;
#pragma unroll
          for (int k = 0; k < BLK_NB; ++k) v = csub(v, cmul(cl[k], rr[k]));
          *dst = v;
        }
      }
      __syncthreads();
    }
  }
  cplx* Om = Ainv + m * (int64_t)n * n;
  for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += BLK_NT) {
    const int i = (int)(e / n), c = (int)(e % n);
    Om[e] = aug[(int64_t)perm[i] * ld + n + c];
  }
}

size_t blocked_smem_bytes(int n) {
  return ((size_t)n * BLK_NB + 2 * BLK_NB * BLK_NB + BLK_NB * BLK_CH) * sizeof(cplx) + (size_t)n * sizeof(int);
}
inline unsigned grid_for(int64_t n, int nt) {
  int64_t g = (n + nt - 1) / nt;
  if (g > 148 * 32) g = 148 * 32;
  if (g < 1) g = 1;
  return (unsigned)g;
}

}  // namespace

void hermitize_batched(cplx* X, int64_t nmat, int n, double scale, cudaStream_t st) {
  if (nmat <= 0) return;
  int64_t total = nmat * (int64_t)n * (n + 1) / 2;
  hermitize_kernel<<<grid_for(total, 256), 256, 0, st>>>(X, nmat, n, scale);
  GB_CHECK_LAUNCH();
}

void scale_inplace(cplx* X, int64_t count, double s, cudaStream_t st) {
  if (count <= 0) return;
  scale_kernel<<<grid_for(count, 256), 256, 0, st>>>(X, count, s);
  GB_CHECK_LAUNCH();
}

void invert_dyson_batched(const cplx* X, const cplx* S, const double* wn, double mu, cplx* G, int64_t nw, int64_t nsk,
                          int n, cudaStream_t st) {
  require(n <= 64, GB200_ERR_INVALID, "invert_dyson_batched: n > 64");
  GjJob j;
  j.A = X; j.out = G; j.stride = (int64_t)n * n; j.ld = n; j.n = n;
  j.S = S; j.wn = wn; j.mu = mu; j.nsk = (int)nsk;
  launch_gj<GJ_DYSON>(j, nw * nsk, st);
}

void trace_dyson_batched(const cplx* X, const cplx* S, const double* wn, double mu, cplx* tr, int64_t nw, int64_t nsk,
                         int n, cudaStream_t st) {
  require(n <= 64, GB200_ERR_INVALID, "trace_dyson_batched: n > 64");
  require(nw * nsk < 2147483647LL, GB200_ERR_INVALID, "trace_dyson_batched: too many matrices");
  GjJob j;
  j.A = X; j.out = tr; j.stride = (int64_t)n * n; j.ld = n; j.n = n;
  j.S = S; j.wn = wn; j.mu = mu; j.nsk = (int)nsk;
  launch_gj<GJ_TRACE>(j, nw * nsk, st);
}

namespace {

// Inverse in place of the `size` x `size` Hermitian block at `off` of every n x n matrix of B, all leading blocks
// positive definite (else bad[matrix] = 1 and the block's content is undefined).  With B = [B11 B21^H; B21 B22]:
// X = B11^-1, T = B21 X, Y = (B22 - T B21^H)^-1, and the inverse is [X + T^H Y T, .; -Y T, Y].  The products run on
// the FP64 tensor cores over all matrices at once: 121 matrices of n = 250 take 1.2 ms, one CTA per matrix with panel
// updates through L2 took 4.44.
void invert_posdef_block(cplx* B, cplx* scratch, int* bad, int64_t nmat, int n, int off, int size, cudaStream_t st) {
  const int64_t n2 = (int64_t)n * n;
  if (size <= 64) {
    GjJob j;
    j.A = j.out = B + (int64_t)off * n + off;
    j.stride = n2; j.ld = n; j.n = size; j.bad = bad;
    launch_gj<GJ_LEAF>(j, nmat, st);
    return;
  }
  const int leaves = (size + 63) / 64;
  const int n1 = (size * ((leaves + 1) / 2) / leaves + 7) / 8 * 8, m2 = size - n1;
  cplx* B11 = B + (int64_t)off * n + off;
  cplx* B21 = B11 + (int64_t)n1 * n;
  cplx* B22 = B21 + n1;
  cplx* T = scratch;  // [nmat][m2][n1], kept over the second inverse
  const int64_t t2 = (int64_t)m2 * n1;
  auto op = [&](cplx* p, int64_t row, int64_t col, int64_t batch, bool conj) {
    ZOperand o;
    o.ptr = p;
    o.row = lin(row);
    o.col = lin(col);
    o.bat.s2 = batch;
    o.conj = conj;
    return o;
  };
  auto mul = [&](const ZOperand& a, const ZOperand& b, int M, int N, int K, cplx* c, int64_t ldc, int64_t cbatch,
                 double alpha, double beta) {
    ZGemm g;
    g.M = M; g.N = N; g.K = K; g.nb2 = nmat;
    g.A = a; g.B = b;
    g.C.ptr = c; g.C.row = lin(ldc); g.C.col = lin(1); g.C.bat.s2 = cbatch;
    g.alpha = cmk(alpha, 0.0); g.beta = cmk(beta, 0.0);
    zgemm_fp64(g, st);
  };
  invert_posdef_block(B, scratch, bad, nmat, n, off, n1, st);
  mul(op(B21, n, 1, n2, false), op(B11, n, 1, n2, false), m2, n1, n1, T, n1, t2, 1.0, 0.0);
  mul(op(T, n1, 1, t2, false), op(B21, 1, n, n2, true), m2, m2, n1, B22, n, n2, -1.0, 1.0);
  invert_posdef_block(B, scratch + nmat * t2, bad, nmat, n, off + n1, m2, st);
  mul(op(B22, n, 1, n2, false), op(T, n1, 1, t2, false), m2, n1, m2, B21, n, n2, -1.0, 0.0);
  mul(op(T, 1, n1, t2, true), op(B21, n, 1, n2, false), n1, n1, m2, B11, n, n2, -1.0, 1.0);
  herm_join_kernel<<<grid_for(nmat * (int64_t)size * size, 256), 256, 0, st>>>(B, nmat, n, off, size, n1);
  GB_CHECK_LAUNCH();
}

}  // namespace

void invert_large_batched(const cplx* A, cplx* Ainv, cplx* aug, int* bad, int64_t nmat, int n, bool identity_minus,
                          cudaStream_t st) {
  require(n <= 4096, GB200_ERR_INVALID, "invert_large_batched: n > 4096");
  if (nmat <= 0) return;
  if (n <= 64) {
    GjJob j;
    j.A = A; j.out = Ainv; j.stride = (int64_t)n * n; j.ld = n; j.n = n; j.identity_minus = identity_minus;
    launch_gj<GJ_HERM>(j, nmat, st);
    return;
  }
  GB_CUDA(cudaMemsetAsync(bad, 0, (size_t)nmat * sizeof(int), st));
  herm_from_lower_kernel<<<grid_for(nmat * (int64_t)n * n, 256), 256, 0, st>>>(A, Ainv, nmat, n, identity_minus);
  GB_CHECK_LAUNCH();
  invert_posdef_block(Ainv, aug, bad, nmat, n, 0, n, st);
  // matrices with a pivot that is not positive: Gauss-Jordan with pivoting from the untouched A
  GB_CUDA(cudaFuncSetAttribute(invert_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  GB_CUDA(cudaFuncSetAttribute(invert_blocked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
  const size_t bsmem = blocked_smem_bytes(n);
  if (bsmem <= 220 * 1024) {
    invert_blocked_kernel<<<(unsigned)nmat, BLK_NT, bsmem, st>>>(A, Ainv, aug, n, identity_minus, bad);
  } else {
    const size_t smem = (size_t)(3 * n) * sizeof(cplx);
    invert_large_kernel<<<(unsigned)nmat, LARGE_NT, smem, st>>>(A, Ainv, aug, n, identity_minus, bad);
  }
  GB_CHECK_LAUNCH();
}

}  // namespace gb200
