// FP64 batched complex GEMM over general index maps, on the FP64 tensor cores.
//
// A CTA of 4 warps computes an 8 TM x 8 TN WN complex tile: WN warps side by side along N, each with TM x TN
// tiles of 8 x 8, and WK = 4 / WN groups of them that split the K steps and are summed at the end.  A step of 4
// along K is four mma.sync m8n8k4 per 8 x 8 tile (Re C += Re A Re B - Im A Im B, Im C += Re A Im B + Im A Re B),
// ordered so that two products into the same accumulator lie 2 TM TN instructions apart (back to back they
// wait for one another's latency).  Operands stay interleaved complex in shared memory: 16-byte cp.async
// straight from the index-mapped global element into a ring of STAGES K blocks, zero fill outside the matrix,
// one barrier per block.  K-fastest operands are kept [row][k] with 4 spare elements a row, the others [k][row]
// with 2 spare, so that the 8 lanes of a 128-bit fragment read hit different banks in both.
//
// Two or three CTAs of 128 threads share an SM (255 or 168 registers a thread): one of them stores its tile or fills
// its ring while another multiplies (three instead of two for the smaller tiles: 10.0 -> 9.0 ms on the exchange below,
// 132 -> 122 ms on a two-spin self-energy at nao = 26).  What bounds it is the FP64 tensor pipe (37 TFLOP/s from
// registers): 76 % of its cycles on 250 x 250 x 3200 and 250 x 1600 x 250, 54 to 62 % where K = 40, where the ring's fill,
// the index maps and the stores count.  Copies issued between the products instead of before them were slower (their
// address loads stall the warp that multiplies).
// Exchange of a Fock build at nk = 27, nao = 40, NQ = 250: 29.4 -> 9.0 ms against the 64 x 64 kernel with register
// staging that this one replaced.
// Contractions with few tiles split K over a cluster of up to 8 CTAs and sum the parts through distributed
// shared memory in rank order, so a result never depends on timing.
#include <cooperative_groups.h>

#include <cmath>

#include "common.cuh"

namespace gb200 {
namespace {

namespace cg = cooperative_groups;

constexpr int NT = 128;

struct LoadMode {
  bool a_kfast;  // consecutive threads walk K for A (else walk M)
  bool b_kfast;  // consecutive threads walk K for B (else walk N)
};

template <int TM, int TN, int WN>
struct Tile {
  static constexpr int WK = 4 / WN;
  static constexpr int MT = 8 * TM, NTL = 8 * TN * WN;
  static constexpr int BK = WK == 1 ? 8 : 16;
  static constexpr int A_ELEMS = MT * (BK + 4), B_ELEMS = NTL * (BK + 4);  // [k][row] needs no more: BK <= 2 rows
  static constexpr int STAGE = A_ELEMS + B_ELEMS;
  // CTAs of an SM: three where the warp's accumulators leave the registers for it (170 a thread)
  static constexpr int CTAS = TM * TN <= 10 ? 3 : 2;
  static constexpr int RING_MAX = (CTAS == 3 ? 70 : 106) * 1024 / (STAGE * 16);
  static constexpr int STAGES = RING_MAX > 4 ? 4 : RING_MAX;
  static constexpr int RED = (WK * MT * NTL);  // elements of the partial sums (reuses the ring)
  static constexpr size_t SMEM = (size_t)(STAGES * STAGE > RED ? STAGES * STAGE : RED) * sizeof(cplx);
};

// D = A B + D for one 8 x 8 x 4 FP64 tile (A row-major 8 x 4, B column-major 4 x 8): lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// 16 bytes global -> shared, zeros when !valid (nothing is read then)
__device__ __forceinline__ void cp_async16(cplx* dst, const cplx* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ double flip(double x, uint32_t sign) {
  return __hiloint2double((int)((uint32_t)__double2hiint(x) ^ sign), __double2loint(x));
}

// One operand block [R rows] x [BK] of K block kb (from k0, up to k1) into shared memory.
template <int R, int BK>
__device__ __forceinline__ void load_block(cplx* s, const cplx* base, const IdxMap& kmap, const int64_t* roff, int rlim,
                                           bool kfast, int64_t k0, int64_t k1) {
  constexpr int N = R * BK;
  if (kfast) {
    const int kk = threadIdx.x % BK;
    const int64_t k = k0 + kk;
    const bool kv = k < k1;
    const cplx* p = base + (kv ? kmap(k) : 0);
#pragma unroll
    for (int i = 0; i < (N + NT - 1) / NT; ++i) {
      const int r = threadIdx.x / BK + i * (NT / BK);
      if (N % NT != 0 && r >= R) break;
      cp_async16(s + r * (BK + 4) + kk, p + roff[r], kv && r < rlim);
    }
  } else {
#pragma unroll
    for (int i = 0; i < (N + NT - 1) / NT; ++i) {
      const int e = threadIdx.x + i * NT;
      if (N % NT != 0 && e >= N) break;
      const int kk = e / R, r = e % R;
      const int64_t k = k0 + kk;
      const bool kv = k < k1;
      cp_async16(s + kk * (R + 2) + r, base + (kv ? kmap(k) : 0) + roff[r], kv && r < rlim);
    }
  }
}

template <int TM, int TN, int WN>
__global__ void __launch_bounds__(NT, (Tile<TM, TN, WN>::CTAS))
    zgemm_fp64_kernel(const __grid_constant__ ZGemm g, LoadMode lm, int64_t nbatch, int ksplit) {
  using T = Tile<TM, TN, WN>;
  constexpr int BK = T::BK;
  extern __shared__ __align__(16) uint8_t zsmem[];
  cplx* ring = reinterpret_cast<cplx*>(zsmem);
  __shared__ int64_t rowA[T::MT], colB[T::NTL], rowC[T::MT], colC[T::NTL];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wn = warp % WN, wk = warp / WN;
  const int fr = lane >> 2, fk = lane & 3;  // fragment row (column for B) and K index
  const int64_t m0 = (int64_t)blockIdx.y * T::MT, n0 = (int64_t)blockIdx.x * T::NTL;
  const int mlim = (int)(g.M - m0 < T::MT ? g.M - m0 : T::MT), nlim = (int)(g.N - n0 < T::NTL ? g.N - n0 : T::NTL);
  const int rank = (int)(blockIdx.z % (unsigned)ksplit);  // part of K (the rank within the cluster)

  for (int i = tid; i < T::MT + T::NTL; i += NT) {
    if (i < T::MT) {
      rowA[i] = i < mlim ? g.A.row(m0 + i) : 0;
      rowC[i] = i < mlim ? g.C.row(m0 + i) : 0;
    } else {
      const int c = i - T::MT;
      colB[c] = c < nlim ? g.B.col(n0 + c) : 0;
      colC[c] = c < nlim ? g.C.col(n0 + c) : 0;
    }
  }
  // this CTA's K range, whole blocks of BK
  const int64_t nkb = (g.K + BK - 1) / BK;
  const int64_t kb0 = nkb * rank / ksplit, kb1 = nkb * (rank + 1) / ksplit;
  const int nkt = (int)(kb1 - kb0);
  const int64_t kbeg = kb0 * BK, kend = kb1 * BK < g.K ? kb1 * BK : g.K;

  // fragment strides of the two layouts, in elements
  const int ars = lm.a_kfast ? BK + 4 : 1, aks = lm.a_kfast ? 1 : T::MT + 2;
  const int brs = lm.b_kfast ? BK + 4 : 1, bks = lm.b_kfast ? 1 : T::NTL + 2;
  const uint32_t sga = g.A.conj ? 0x80000000u : 0u, sgb = g.B.conj ? 0x80000000u : 0u;
  const bool has_beta = (g.beta.x != 0.0 || g.beta.y != 0.0);
  __syncthreads();

  for (int64_t b = blockIdx.z / (unsigned)ksplit; b < nbatch; b += gridDim.z / (unsigned)ksplit) {
    const int64_t b2 = b % g.nb2;
    const int64_t b1 = (b / g.nb2) % g.nb1;
    const int64_t b0 = b / (g.nb2 * g.nb1);
    const cplx* Ab = g.A.ptr + g.A.bat(b0, b1, b2);
    const cplx* Bb = g.B.ptr + g.B.bat(b0, b1, b2);
    cplx* Cb = g.C.ptr + g.C.bat(b0, b1, b2);

    double cr[TM][TN][2], ci[TM][TN][2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

    auto load = [&](int kt) {
      if (kt < nkt) {
        cplx* s = ring + (size_t)(kt % T::STAGES) * T::STAGE;
        const int64_t k0 = kbeg + (int64_t)kt * BK;
        load_block<T::MT, BK>(s, Ab, g.A.col, rowA, mlim, lm.a_kfast, k0, kend);
        load_block<T::NTL, BK>(s + T::A_ELEMS, Bb, g.B.row, colB, nlim, lm.b_kfast, k0, kend);
      }
      cp_commit();  // (an empty group past the end keeps the count of groups in flight)
    };
#pragma unroll
    for (int s = 0; s < T::STAGES - 1; ++s) load(s);
    for (int kt = 0; kt < nkt; ++kt) {
      cp_wait<T::STAGES - 2>();
      __syncthreads();  // block kt has landed for every thread, and block kt - 1 has been read
      load(kt + T::STAGES - 1);
      const cplx* s = ring + (size_t)(kt % T::STAGES) * T::STAGE;
      const cplx* sa = s + fr * ars + fk * aks;
      const cplx* sb = s + T::A_ELEMS + (wn * 8 * TN + fr) * brs + fk * bks;
      const int64_t left = kend - kbeg - (int64_t)kt * BK;
      const int ksteps = left >= BK ? BK / 4 : (int)((left + 3) / 4);
#pragma unroll
      for (int kq = 0; kq < BK / 4 / T::WK; ++kq) {
        const int k4 = kq * T::WK + wk;
        if (k4 >= ksteps) break;
        double are[TM], aim[TM], bre[TN], bim[TN], nim[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const cplx v = sb[j * 8 * brs + k4 * 4 * bks];
          bre[j] = v.x;
          bim[j] = flip(v.y, sgb);
          nim[j] = flip(v.y, sgb ^ 0x80000000u);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const cplx v = sa[i * 8 * ars + k4 * 4 * aks];
          are[i] = v.x;
          aim[i] = flip(v.y, sga);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) dmma(cr[i][j], are[i], bre[j]);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) dmma(ci[i][j], are[i], bim[j]);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) dmma(cr[i][j], aim[i], nim[j]);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) dmma(ci[i][j], aim[i], bre[j]);
      }
    }
    cp_wait<0>();
    __syncthreads();  // the ring is free again

    if (T::WK == 1 && ksplit == 1) {
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int r = i * 8 + fr;
        if (r >= mlim) continue;
        cplx* Cr = Cb + rowC[r];
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = (wn * TN + j) * 8 + 2 * fk + h;
            if (c >= nlim) continue;
            cplx* p = Cr + colC[c];
            cplx v = cmul(g.alpha, cmk(cr[i][j][h], ci[i][j][h]));
            if (has_beta) v = cadd(v, cmul(g.beta, *p));
            *p = v;
          }
      }
      continue;
    }
    // partial sums of the WK warp groups and the cluster's CTAs: each CTA finishes its share of the tile
    cplx* red = ring + (size_t)wk * T::MT * T::NTL;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          red[(i * 8 + fr) * T::NTL + (wn * TN + j) * 8 + 2 * fk + h] = cmk(cr[i][j][h], ci[i][j][h]);
    if (ksplit > 1) cg::this_cluster().sync();
    else __syncthreads();
    const bool row_major = (g.C.col.s_in <= g.C.row.s_in && g.C.col.s_in >= -g.C.row.s_in);
    for (int e = tid + rank * NT; e < T::MT * T::NTL; e += NT * ksplit) {
      const int r = row_major ? e / T::NTL : e % T::MT, c = row_major ? e % T::NTL : e / T::MT;
      if (r >= mlim || c >= nlim) continue;
      cplx v = cmk(0.0, 0.0);
      for (int q = 0; q < ksplit; ++q) {
        const cplx* src = ksplit > 1 ? cg::this_cluster().map_shared_rank(ring, q) : ring;
#pragma unroll
        for (int w = 0; w < T::WK; ++w) v = cadd(v, src[(size_t)w * T::MT * T::NTL + r * T::NTL + c]);
      }
      cplx* p = Cb + rowC[r] + colC[c];
      v = cmul(g.alpha, v);
      if (has_beta) v = cadd(v, cmul(g.beta, *p));
      *p = v;
    }
    if (ksplit > 1) cg::this_cluster().sync();
    else __syncthreads();
  }
}

inline int64_t abs64(int64_t v) { return v < 0 ? -v : v; }

struct Variant {
  int tm, tn, wn;
};

// Time of a variant in SM cycles, up to what all variants share.  Per K step of one element a CTA needs MT NTL 4 / 65
// cycles of the FP64 tensor pipe (65 multiply-adds a cycle and SM: 37 TFLOP/s measured from registers) and (MT + NTL) 16
// bytes from L2 at 19 bytes a cycle and SM; 900 cycles a tile are the ring's fill and the stores that the other CTA of the
// SM does not hide.  The last two are not rates of the hardware but the values at which the variants rank as they measure:
// with 12 bytes gw at nao = 26, ns = 2 takes 128.5 ms instead of 122.1, with 33 the adjoint at nao = 20 takes 127.5
// instead of 114.1, and 120.4 with 500 cycles, 115.3 with 1500; Fock builds do not care.  Tiles are spread over 148 SMs.
double variant_cost(const Variant& v, int64_t M, int64_t N, int64_t K, int64_t nbatch, int ks) {
  const double mt = 8.0 * v.tm, nt = 8.0 * v.tn * v.wn;
  const double tiles = std::ceil(M / mt) * std::ceil(N / nt) * (double)nbatch * ks;
  const double pipe = mt * nt * 4.0 / 65.0, l2 = (mt + nt) * 16.0 / 19.0;
  const double perk = (pipe > l2 ? pipe + 0.15 * l2 : l2 + 0.15 * pipe);
  double tile = perk * (double)((K + ks - 1) / ks + 4) + 900.0 + (v.wn < 4 ? 300.0 : 0.0) + (ks > 1 ? 2500.0 : 0.0);
  return std::ceil(tiles / 148.0) * tile;
}

template <int TM, int TN, int WN>
void launch(const ZGemm& g, const LoadMode& lm, int64_t nbatch, int ks, cudaStream_t st) {
  using T = Tile<TM, TN, WN>;
  static_assert(T::STAGES >= 2, "ring");
  auto kern = zgemm_fp64_kernel<TM, TN, WN>;
  // set on every call: the attribute belongs to the current device (a host call of about a microsecond)
  GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM));
  const int64_t nz = nbatch < 65535 / ks ? nbatch : 65535 / ks;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((g.N + T::NTL - 1) / T::NTL), (unsigned)((g.M + T::MT - 1) / T::MT), (unsigned)(nz * ks));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = T::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  if (ks > 1) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = (unsigned)ks;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
  GB_CUDA(cudaLaunchKernelEx(&cfg, kern, g, lm, nbatch, ks));
  GB_CHECK_LAUNCH();
}

template <int TN, int WN>
void launch_tm(int tm, const ZGemm& g, const LoadMode& lm, int64_t nbatch, int ks, cudaStream_t st) {
  switch (tm) {
    case 1: launch<1, TN, WN>(g, lm, nbatch, ks, st); break;
    case 2: launch<2, TN, WN>(g, lm, nbatch, ks, st); break;
    case 3: launch<3, TN, WN>(g, lm, nbatch, ks, st); break;
    case 4: launch<4, TN, WN>(g, lm, nbatch, ks, st); break;
    case 5: launch<5, TN, WN>(g, lm, nbatch, ks, st); break;
    default:
      if constexpr (TN == 2) {
        if (tm == 6) launch<6, TN, WN>(g, lm, nbatch, ks, st);
        else if (tm == 7) launch<7, TN, WN>(g, lm, nbatch, ks, st);
        else launch<8, TN, WN>(g, lm, nbatch, ks, st);
      }
  }
}

template <int TN, int WN, int TM>
void preload_one() {
  if constexpr (TM * TN <= 16) {
    cudaFuncAttributes at;
    GB_CUDA(cudaFuncGetAttributes(&at, zgemm_fp64_kernel<TM, TN, WN>));
  }
}

template <int TN, int WN>
void preload_tn() {
  preload_one<TN, WN, 1>();
  preload_one<TN, WN, 2>();
  preload_one<TN, WN, 3>();
  preload_one<TN, WN, 4>();
  preload_one<TN, WN, 5>();
  preload_one<TN, WN, 6>();
  preload_one<TN, WN, 7>();
  preload_one<TN, WN, 8>();
}

}  // namespace

void zgemm_fp64_preload() {
  preload_tn<2, 4>();
  preload_tn<3, 2>();
  preload_tn<2, 2>();
  preload_tn<2, 1>();
}

void validate(const ZGemm& g) {
  // an outer index with neither a table nor a stride is a set-up error, not a broadcast
  const IdxMap* maps[] = {&g.A.row, &g.A.col, &g.B.row, &g.B.col, &g.C.row, &g.C.col};
  for (const IdxMap* m : maps)
    require(!(m->n_in > 0 && m->tab == nullptr && m->s_out == 0), GB200_ERR_STATE, "zgemm: index map without outer table");
}

void zgemm_fp64(const ZGemm& g0, cudaStream_t st) {
  if (g0.M <= 0 || g0.N <= 0) return;
  validate(g0);
  const int64_t nbatch = g0.nb0 * g0.nb1 * g0.nb2;
  if (nbatch <= 0) return;
  // the cheapest tile, for C = A B or its transpose C^T = B^T A^T (so that a narrow side of either kind takes
  // the M tile of 8 to 64 rows, and 10 to 60 orbitals are not padded to 64), and the number of K parts
  static const int shapes[][2] = {{2, 4}, {3, 2}, {2, 2}, {2, 1}};  // (TN, WN)
  Variant best{8, 2, 4};
  int best_ks = 1;
  bool best_swap = false;
  double best_cost = 1e300;
  for (int swap = 0; swap < 2; ++swap) {
    const int64_t M = swap ? g0.N : g0.M, N = swap ? g0.M : g0.N;
    for (const auto& sh : shapes)
      for (int tm = 1; tm <= 8; ++tm) {
        const Variant v{tm, sh[0], sh[1]};
        if ((M + 8 * tm - 1) / (8 * tm) > 65535) continue;
        if (tm * sh[0] > 16) continue;  // the accumulators of a larger warp tile do not fit the registers
        for (int ks = 1; ks <= 8; ks *= 2) {
          if (ks > 1 && g0.K / ks < 32) break;
          const double c = variant_cost(v, M, N, g0.K, nbatch, ks);
          if (c < best_cost) {
            best_cost = c;
            best = v;
            best_ks = ks;
            best_swap = swap != 0;
          }
        }
      }
  }
  require(best_cost < 1e300, GB200_ERR_INVALID, "zgemm: M too large");
  ZGemm g = g0;
  if (best_swap) {
    g.M = g0.N;
    g.N = g0.M;
    g.A = g0.B;
    g.A.row = g0.B.col;
    g.A.col = g0.B.row;
    g.B = g0.A;
    g.B.row = g0.A.col;
    g.B.col = g0.A.row;
    g.C.row = g0.C.col;
    g.C.col = g0.C.row;
  }
  LoadMode lm;
  // choose the coalescing direction: the index with the smaller inner stride walks fastest
  lm.a_kfast = abs64(g.A.col.s_in) <= abs64(g.A.row.s_in);
  lm.b_kfast = abs64(g.B.row.s_in) <= abs64(g.B.col.s_in);
  if (best.wn == 4) launch_tm<2, 4>(best.tm, g, lm, nbatch, best_ks, st);
  else if (best.tn == 3) launch_tm<3, 2>(best.tm, g, lm, nbatch, best_ks, st);
  else if (best.wn == 2) launch_tm<2, 2>(best.tm, g, lm, nbatch, best_ks, st);
  else launch_tm<2, 1>(best.tm, g, lm, nbatch, best_ks, st);
}

}  // namespace gb200
