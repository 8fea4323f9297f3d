// Split-precision complex contractions: Ozaki slicing into INT8, exact INT32
// products on the 5th-generation tensor cores (tcgen05, kind::i8), FP64
// recombination.
//
// Number format.  Every complex row of the left operand (and every complex column of the right one) gets a
// power-of-two exponent e with max|Re|,|Im| < 2^(e-1) over the contraction range.  Each real part is rounded to an
// integer and cut into S balanced digits, a = 2^(e-7) (q_0 + q_1 B^-1 + ... + q_{S-1} B^-(S-1)) + r, base B = 256 for
// up to six slices and 128 for seven and eight (split_digits.cuh).  Products of slices s and t share the weight
// B^-(s+t); all pairs with s + t = d accumulate into one INT32 accumulator "diagonal" d (pairs with s + t >= S are
// dropped, the usual triangular Ozaki truncation).  Rounding and balanced digits keep the representation error and the
// dropped products zero-mean, so they do not add up in phase along the contraction.  The host splits the contraction
// so that no diagonal can overflow INT32.
//
// Complex arithmetic.  C = A B is computed as its transpose: the rows of the tensor-core tile are the columns n of B
// (the large operand of every contraction), stored as (re, im) pairs along K, and its columns come from the rows m of
// A in the real embedding, 2m: (re, -im) pairs and 2m+1: (im, re) pairs.  Columns 2m and 2m+1 of the result are then Re
// and Im of C(m, n), in the same TMEM lane.  (With the embedding on the row side the two lie in different lanes, and
// exchanging them took a fifth of the epilogue's instructions; the small operand's padding, 40 rows to 64, becomes
// 80 columns of 80.)
//
// Tensor-core kernel.  One CTA computes 128 values of n x BN / 2 values of m for all S diagonals (S * BN <= 512 TMEM
// columns).  Warp 0 streams 64-byte K blocks of every slice plane with TMA (64-byte swizzle) through a multi-stage
// mbarrier ring, warp 1 issues the tcgen05.mma instructions from one thread, warp 2 gathers the index maps and
// exponents of the coming tile into shared memory, and 16 epilogue warps read the accumulators from TMEM (tcgen05.ld),
// recombine in FP64 and store.  Every wait is bounded; on timeout the kernel records an error and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>

#include "split.cuh"
#include "split_digits.cuh"

namespace gb200 {

namespace {

constexpr int KBLK = 64;          // bytes of K per pipeline stage (one 64B swizzle atom)
constexpr int TILE_R = 128;       // rows per CTA: complex columns n of the product
constexpr int SMEM_MAX = 227 * 1024;  // the opt-in limit of a block
constexpr int EPI_WARPS = 16;     // four per TMEM sub-partition: enough warps in flight to hide
                                  // the TMEM, FP64 and store latencies of the recombination
constexpr int EPI_FIRST = 3;      // producer, MMA and table warps before them
constexpr int NWARPS = EPI_FIRST + EPI_WARPS;
constexpr int EPI_CG = 8;         // result columns (4 complex) per TMEM read: one tcgen05.ld of 8 columns
constexpr long long WAIT_LIMIT = 4000000000LL;  // clock64 cycles (~2 s)

enum SplitErr { SERR_NONE = 0, SERR_TIMEOUT_PRODUCER = 1, SERR_TIMEOUT_MMA = 2, SERR_TIMEOUT_EPILOGUE = 3, SERR_TIMEOUT_TABLES = 4 };

// ----------------------------------------------------------------------------
// PTX wrappers
// ----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive_local(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The time hint lets the hardware keep the thread asleep instead of polling: without it the waiting warps issued a third
// of the SM's instructions, in competition with the warps they waited for.
constexpr uint32_t WAIT_HINT_NS = 20000;

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase), "r"(WAIT_HINT_NS)
      : "memory");
  return ok != 0;
}

// Bounded wait: returns false on timeout.  Warps whose lanes all touch what a barrier guards call it from every lane, and
// vote on the outcome: each lane then has its own acquire.  (One lane polling for the others needs a __syncwarp behind it,
// because a shuffle of the outcome orders no memory, and the loop of a single lane was slower: with it gw_split_mid took
// 171.7 ms, iteration_split 51.0 and batch_uneven 255 instead of 160.0, 47.6 and 234.)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, volatile int* abort_flag) {
  if (mbar_try_wait(bar, phase)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, phase)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > WAIT_LIMIT) return false;
  }
  return true;
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// one lane of a converged warp
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t is;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(is));
  return is;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}

// Issued by the one lane with `issue` set.  The whole warp runs the surrounding code, so that the operands, the same in
// every lane, stay in uniform registers: computed by a single diverged thread they cost that thread several
// instructions per operand, in competition with the epilogue warps of its scheduler.
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum,
                                        uint32_t issue) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum), "r"(issue));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar, uint32_t issue) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(issue)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major operand, 64-byte swizzle, rows of
// 64 bytes, 8-row groups 512 bytes apart (SBO), layout version 1 (sm_100).
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;   // stride byte offset
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)4 << 61;            // SWIZZLE_64B
  return d;
}

// Instruction descriptor: S32 accumulate, signed 8-bit A and B, both K-major, M=128, N=bn.
__host__ __device__ constexpr uint32_t idesc_i8(int bn) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(TILE_R >> 4) << 24);
}

// ----------------------------------------------------------------------------
// parameters
// ----------------------------------------------------------------------------
struct GemmParams {
  int S;
  int BN;         // tile columns: real columns of the embedded operand
  int stages;
  int tiles_r, tiles_c;
  int nkb;        // K blocks of KBLK bytes
  int nkk;        // K steps of 32 bytes
  int overlap;    // launch-wide: two accumulator sets and resident row planes (short contractions)
  int64_t M, N;   // complex rows of A (tile columns / 2) and columns of B (tile rows)
  int64_t nb0, nb1, nb2;
  int depA[3], depB[3];
  int64_t rowsA, rowsB;  // rows of a plane: 2 M and N
  int ntile;       // tiles of this problem
  const int32_t* eA;
  const int32_t* eB;
  int64_t eA_ld, eB_ld;
  ZResult C;
  cplx alpha, beta;
  int alpha_pow2;  // alpha is real and a power of two (possibly negative)
  int* err;
  // grouped launch: the problems' entries (tile ranges in order) and the total tile count; the
  // launch-wide fields above (S, BN = the widest tile, stages, err) size the shared ring
  const struct GroupEntry* group;
  int ngroup;
  int64_t ntiles;
};

// one problem of a grouped launch: its tensor maps, parameters and first global tile
struct alignas(64) GroupEntry {
  CUtensorMap mR, mC;  // planes of the tile's rows (operand B) and columns (operand A)
  GemmParams p;
  int64_t tile_begin;
};

__device__ __forceinline__ int64_t reduced_batch(const int dep[3], int64_t b0, int64_t b1, int64_t b2, int64_t n1,
                                                 int64_t n2) {
  int64_t rb = 0;
  if (dep[0]) rb = b0;
  if (dep[1]) rb = rb * n1 + b1;
  if (dep[2]) rb = rb * n2 + b2;
  return rb;
}

// ----------------------------------------------------------------------------
// slicing
// ----------------------------------------------------------------------------
struct SliceJob {
  const cplx* ptr;
  IdxMap rmap, kmap;
  BatchMap bat;
  bool conj;
  int64_t R, K, k0;            // rows, K range [k0, k0 + K)
  int64_t n0, n1, n2;          // batch sizes of the GEMM
  int dep[3];
  int embed;                   // 1: operand A (doubled rows), 0: operand B
  int S;
  int64_t rows_pad;            // real rows per plane (2 R for the embedded operand)
  int64_t rpad;                // complex rows covered (R)
  int64_t kpad, e_ld;
  int8_t* out;
  int32_t* expo;
  bool r_fast;                 // consecutive threads walk rows (else K) when reading
  int single;                  // 1: the whole K range is one tile, exponents found in the same pass
};

constexpr int TR = 32, TK = 64, SL_NT = 256;
// shared tile columns: one spare slot after every 8 complex values, so the 8 threads that
// read consecutive groups of 8 columns of a row hit different banks
constexpr int TKP = TK + TK / 8 + 1;
__device__ __forceinline__ int tcol(int c) { return c + (c >> 3); }
constexpr int EXP_EMPTY = -(1 << 30);

__device__ __forceinline__ void enumerate_batch(const SliceJob& j, int64_t rb, int64_t& b0, int64_t& b1, int64_t& b2) {
  // inverse of reduced_batch with the components the operand does not depend on set to 0
  b0 = b1 = b2 = 0;
  int64_t r = rb;
  if (j.dep[2]) { b2 = r % j.n2; r /= j.n2; }
  if (j.dep[1]) { b1 = r % j.n1; r /= j.n1; }
  if (j.dep[0]) { b0 = r; }
}

// Row and K offsets of a tile (one IdxMap evaluation per row and per K position instead of
// one per element); callers synchronise before using them.
__device__ __forceinline__ void tile_offsets(const SliceJob& j, int64_t r0, int64_t kc, int64_t* roff, int64_t* koff) {
  const int t = threadIdx.x;
  if (t < TR) roff[t] = (r0 + t < j.R) ? j.rmap(r0 + t) : 0;
  else if (t >= 64 && t < 64 + TK) koff[t - 64] = (kc + t - 64 < j.K) ? j.kmap(j.k0 + kc + t - 64) : 0;
}

// Stage a TR x TK tile of the operand in shared memory (zero outside [0,R) x [0,K)); a thread
// issues its loads four at a time before storing them.
__device__ __forceinline__ void load_slice_tile(const SliceJob& j, const cplx* base, const int64_t* roff,
                                                const int64_t* koff, int64_t r0, int64_t kc, cplx (*tile)[TKP]) {
  constexpr int PER = TR * TK / SL_NT, BATCH = 4;
#pragma unroll
  for (int i0 = 0; i0 < PER; i0 += BATCH) {
    cplx v[BATCH];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int e = threadIdx.x + (i0 + i) * SL_NT;
      int rl, kl;
      if (j.r_fast) { rl = e % TR; kl = e / TR; } else { kl = e % TK; rl = e / TK; }
      v[i] = cmk(0.0, 0.0);
      if (r0 + rl < j.R && kc + kl < j.K) v[i] = __ldg(base + roff[rl] + koff[kl]);
    }
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int e = threadIdx.x + (i0 + i) * SL_NT;
      int rl, kl;
      if (j.r_fast) { rl = e % TR; kl = e / TR; } else { kl = e % TK; rl = e / TK; }
      if (j.conj) v[i].y = -v[i].y;
      tile[rl][tcol(kl)] = v[i];
    }
  }
}

// Pass 1: per-row exponent e' = e + 1 (max |Re|,|Im| < 2^e = 2^(e'-1)) by atomicMax over K tiles.
__global__ void __launch_bounds__(SL_NT, 4) slice_expo_kernel(SliceJob j) {
  __shared__ cplx tile[TR][TKP];
  __shared__ int64_t roff[TR], koff[TK];
  const int64_t rb = blockIdx.z, r0 = (int64_t)blockIdx.x * TR, kc = (int64_t)blockIdx.y * TK;
  if (r0 >= j.R || kc >= j.K) return;
  int64_t b0, b1, b2;
  enumerate_batch(j, rb, b0, b1, b2);
  const cplx* base = j.ptr + j.bat(b0, b1, b2);
  tile_offsets(j, r0, kc, roff, koff);
  __syncthreads();
  load_slice_tile(j, base, roff, koff, r0, kc, tile);
  __syncthreads();
  // 8 threads per row, 8 columns each
  const int rl = threadIdx.x / 8, part = threadIdx.x % 8;
  double m = 0.0;
#pragma unroll
  for (int i = 0; i < TK / 8; ++i) {
    cplx v = tile[rl][tcol(part * (TK / 8) + i)];
    m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
  }
  for (int o = 4; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (part == 0 && m > 0.0 && r0 + rl < j.R) {
    int e;
    frexp(m, &e);
    atomicMax(&j.expo[rb * j.e_ld + r0 + rl], e + 1);  // |a| < 2^(e'-1): one bit of headroom
  }
}

// base of the digits of S slices, and the power of two of the lowest diagonal's unit: a product of operands with
// exponents ea, eb is 2^(ea + eb - unit_exp) times sum_d q_d B^(S-1-d)
__host__ __device__ constexpr int digit_bits(int S) { return S <= 6 ? 8 : 7; }
__host__ __device__ constexpr int unit_exp(int S) { return 14 + digit_bits(S) * (S - 1); }

// Write the S digit planes of 8 consecutive K positions (from k) of row r with row exponent e, including the zero
// padding of K.  S is a compile-time constant, so every digit position is one, and a plane's 16 bytes take four
// packed words.
template <int S>
__device__ __forceinline__ void write_digits(const SliceJob& j, const cplx (&vals)[8], int64_t rb, int64_t r, int64_t k,
                                             int e) {
  if (r >= j.rpad || 2 * k >= j.kpad) return;
  constexpr bool WIDE = digit_bits(S) == 8;
  // the scale 2^(8S - 1 - e) (base 128: 2^(7S - e)); as two exact factors where it leaves the double range
  const int ex = (WIDE ? 8 * S - 1 : 7 * S) - e;
  // the integers of the 8 positions, (re, im) in turn, plus the bias that makes their digits unsigned
  uint64_t u[16];
  if (ex >= -1000 && ex <= 1000) {
    const double sc = __longlong_as_double((long long)(ex + 1023) << 52);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      u[2 * i] = WIDE ? wide_input(vals[i].x * sc, S) : balanced_input(vals[i].x * sc, S);
      u[2 * i + 1] = WIDE ? wide_input(vals[i].y * sc, S) : balanced_input(vals[i].y * sc, S);
    }
  } else {
    const int ex1 = max(-1000, min(1000, ex));
    const double sc1 = __longlong_as_double((long long)(ex1 + 1023) << 52);
    const double sc2 = __longlong_as_double((long long)(max(-1022, min(1023, ex - ex1)) + 1023) << 52);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      u[2 * i] = WIDE ? wide_input((vals[i].x * sc1) * sc2, S) : balanced_input((vals[i].x * sc1) * sc2, S);
      u[2 * i + 1] = WIDE ? wide_input((vals[i].y * sc1) * sc2, S) : balanced_input((vals[i].y * sc1) * sc2, S);
    }
  }
  const int64_t plane = j.rows_pad * j.kpad;
  int8_t* outb = j.out + rb * (int64_t)S * plane + (j.embed ? 2 * r : r) * j.kpad + 2 * k;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    uint32_t w[4];  // bytes (re, im) of positions 2h and 2h + 1
#pragma unroll
    for (int h = 0; h < 4; ++h)
      w[h] = WIDE ? wide_digit_word(u[4 * h], u[4 * h + 1], u[4 * h + 2], u[4 * h + 3], S, s)
                  : balanced_digit_word(u[4 * h], u[4 * h + 1], u[4 * h + 2], u[4 * h + 3], S, s);
    int8_t* p = outb + (int64_t)s * plane;
    if (j.embed) {
      // row 2r: (re, -im) pairs; row 2r+1: (im, re) pairs.  (A base-256 digit of -128 has no negative: -im is cut into
      // its own digits.)
      uint32_t w0[4], w1[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t neg = WIDE ? wide_digit_word(u[4 * h], wide_negate(u[4 * h + 1], S), u[4 * h + 2],
                                                    wide_negate(u[4 * h + 3], S), S, s)
                                  : __byte_perm(w[h], negate_bytes(w[h]), 0x7250);
        w0[h] = neg;
        w1[h] = __byte_perm(w[h], 0u, 0x2301);
      }
      *reinterpret_cast<uint4*>(p) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
      *reinterpret_cast<uint4*>(p + j.kpad) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
    } else {
      *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Pass 2: slice planes, including the zero padding of rows and K.
template <int S>
__global__ void __launch_bounds__(SL_NT, 4) slice_write_kernel(SliceJob j) {
  __shared__ cplx tile[TR][TKP];
  __shared__ int64_t roff[TR], koff[TK];
  const int64_t rb = blockIdx.z, r0 = (int64_t)blockIdx.x * TR, kc = (int64_t)blockIdx.y * TK;
  int64_t b0, b1, b2;
  enumerate_batch(j, rb, b0, b1, b2);
  const cplx* base = j.ptr + j.bat(b0, b1, b2);
  tile_offsets(j, r0, kc, roff, koff);
  __syncthreads();
  load_slice_tile(j, base, roff, koff, r0, kc, tile);
  __syncthreads();
  const int rl = threadIdx.x / 8, grp = threadIdx.x % 8;
  const int64_t r = r0 + rl;
  const int64_t k = kc + grp * 8;  // first of 8 complex K positions
  cplx vals[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) vals[i] = tile[rl][tcol(grp * 8 + i)];
  int e = 0;
  if (j.single) {
    // the 8 lanes of a row hold all of its K range: reduce the maximum here (before any lane leaves)
    double m = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmax(m, fmax(fabs(vals[i].x), fabs(vals[i].y)));
    for (int o = 4; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (m > 0.0) {
      frexp(m, &e);
      ++e;  // one bit of headroom, as in slice_expo_kernel
    }
    if (grp == 0 && r < j.R) j.expo[rb * j.e_ld + r] = e;
  } else if (r < j.R) {
    e = j.expo[rb * j.e_ld + r];
    if (e == EXP_EMPTY) e = 0;
  }
  write_digits<S>(j, vals, rb, r, k, e);
}

// One pass for contractions of moderate length (K up to 8 tiles): a block stages RB rows over the
// whole contraction range in shared memory, reduces their exponents there and writes the slices,
// so the operand is read from HBM once.  Row layout in shared memory as in the tile kernels (one
// spare slot after every 8 complex values: the 8 threads reading consecutive groups of a row hit
// different banks).
__host__ __device__ inline int resident_ld(int kt) { return kt + kt / 8 + 1; }

inline size_t resident_smem(int rb, int kt) {
  return (size_t)rb * resident_ld(kt) * sizeof(cplx) + (size_t)(rb + kt) * sizeof(int64_t) + rb * sizeof(double);
}

template <int RB, int S>
__global__ void __launch_bounds__(SL_NT) slice_resident_kernel(SliceJob j, int kt) {
  extern __shared__ __align__(16) uint8_t sl_smem[];
  const int ld = resident_ld(kt);
  cplx* rows = reinterpret_cast<cplx*>(sl_smem);
  int64_t* roff = reinterpret_cast<int64_t*>(rows + RB * ld);
  int64_t* koff = roff + RB;
  double* rmax = reinterpret_cast<double*>(koff + kt);
  const int64_t rb = blockIdx.z, r0 = (int64_t)blockIdx.x * RB;
  int64_t b0, b1, b2;
  enumerate_batch(j, rb, b0, b1, b2);
  const cplx* base = j.ptr + j.bat(b0, b1, b2);
  for (int i = threadIdx.x; i < RB + kt; i += SL_NT) {
    if (i < RB) roff[i] = (r0 + i < j.R) ? j.rmap(r0 + i) : 0;
    else koff[i - RB] = (i - RB < j.K) ? j.kmap(j.k0 + i - RB) : 0;
  }
  __syncthreads();
  // stage the block's rows, eight loads in flight per thread
  const int n = RB * kt;
  for (int e0 = 0; e0 < n; e0 += 8 * SL_NT) {
    cplx v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + threadIdx.x + i * SL_NT;
      int rl, kl;
      if (j.r_fast) { rl = e % RB; kl = e / RB; } else { kl = e % kt; rl = e / kt; }
      v[i] = cmk(0.0, 0.0);
      if (e < n && r0 + rl < j.R && kl < j.K) v[i] = __ldg(base + roff[rl] + koff[kl]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + threadIdx.x + i * SL_NT;
      int rl, kl;
      if (j.r_fast) { rl = e % RB; kl = e / RB; } else { kl = e % kt; rl = e / kt; }
      if (j.conj) v[i].y = -v[i].y;
      if (e < n) rows[rl * ld + tcol(kl)] = v[i];
    }
  }
  __syncthreads();
  // row maxima: SL_NT / RB consecutive threads per row
  constexpr int TPR = SL_NT / RB;
  static_assert(TPR <= 32 && (32 % TPR) == 0, "threads of a row within one warp");
  {
    const int rl = threadIdx.x / TPR, part = threadIdx.x % TPR;
    double m = 0.0;
    for (int k = part; k < kt; k += TPR) {
      const cplx v = rows[rl * ld + tcol(k)];
      m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
    }
    for (int o = TPR / 2; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (part == 0) rmax[rl] = m;
  }
  __syncthreads();
  // digits: one thread per (row, 8 consecutive K positions)
  const int groups = kt / 8;
  for (int it = threadIdx.x; it < RB * groups; it += SL_NT) {
    const int rl = it / groups, g = it % groups;
    const int64_t r = r0 + rl;
    int e = 0;
    if (rmax[rl] > 0.0) {
      frexp(rmax[rl], &e);
      ++e;  // one bit of headroom, as in slice_expo_kernel
    }
    if (g == 0 && r < j.R) j.expo[rb * j.e_ld + r] = e;
    cplx vals[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) vals[i] = rows[rl * ld + tcol(g * 8 + i)];
    write_digits<S>(j, vals, rb, r, (int64_t)g * 8, e);
  }
}

// exponent of a row that was entirely zero -> 0 (its slices are zero)
__global__ void fix_empty_expo_kernel(int32_t* e, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (e[i] == EXP_EMPTY) e[i] = 0;
}

// ----------------------------------------------------------------------------
// recombination epilogue (shared by both cores)
// ----------------------------------------------------------------------------
// 2^e as an exact double (e within the normal range)
__device__ __forceinline__ double pow2(int e) {
  e = max(-1022, min(1023, e));
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// int32 -> double on the FP64 pipe: the double with high word 0x43380000 and low word x + 2^31
// is 1.5*2^52 + 2^31 + x exactly (IEEE-754 bit pattern), so one subtraction gives x.
__device__ __forceinline__ double int_to_double(int32_t x) {
  return __hiloint2double(0x43380000, (int)((uint32_t)x ^ 0x80000000u)) - 6755401588539392.0;
}

// sum_d q_d B^(S-1-d) as a double, the value in units of 2^(ea + eb - unit_exp).  Up to five slices the sum is formed
// exactly in 64-bit integers (|q_d| < 2^31, so it is below 2^63) and rounded once: four multiply-adds and three FP64
// operations where a Horner sum over converted diagonals takes fourteen.  Both engines use this function, so they agree
// bit for bit.
template <int S>
__device__ __forceinline__ double combine_diagonals(const int32_t (&q)[S]) {
  if constexpr (S <= 5) {
    long long t = q[S - 1];
#pragma unroll
    for (int i = 1; i < (S < 4 ? S : 4); ++i) t += (long long)q[S - 1 - i] * (1 << (8 * i));
    int hi = (int)(t >> 32);
    if constexpr (S == 5) hi += q[0];
    const double lo = __hiloint2double(0x43300000, (int)(uint32_t)t) - 4503599627370496.0;  // the low word, unsigned
    return fma(int_to_double(hi), 4294967296.0, lo);
  } else {
    constexpr double B = digit_bits(S) == 8 ? 256.0 : 128.0;
    double v = int_to_double(q[0]);
#pragma unroll
    for (int d = 1; d < S; ++d) v = fma(v, B, int_to_double(q[d]));
    return v;
  }
}

// ----------------------------------------------------------------------------
// tcgen05 core
// ----------------------------------------------------------------------------
// Short contractions (over up to RES_KB K blocks: 64 orbitals) run in overlap mode: two accumulator sets of half the
// width, so that the epilogue of a tile runs beside the MMAs of the next, and the row planes of a tile kept in shared
// memory (two sets) for the column tiles that share them, which halves what a tile reads from L2.
constexpr int RES_KB = 2;
constexpr int OVERLAP_MAX_S = 5;  // (six slices leave no room for two sets of rows)

struct SmemLayout {
  int r_plane_bytes;  // one row plane of a K block
  int rows_bytes;     // resident row planes, [2][S][RES_KB] (0: they are part of the stages)
  int stage_rows;     // row-plane bytes of a stage
  int stage_bytes, stages, ring_bytes;
};

__host__ __device__ inline SmemLayout smem_layout(int S, int BN, int stages, int overlap) {
  SmemLayout L;
  L.r_plane_bytes = TILE_R * KBLK;
  L.rows_bytes = overlap ? 2 * S * RES_KB * L.r_plane_bytes : 0;
  L.stage_rows = overlap ? 0 : S * L.r_plane_bytes;
  L.stage_bytes = L.stage_rows + S * BN * KBLK;
  L.stages = stages;
  L.ring_bytes = L.rows_bytes + stages * L.stage_bytes;
  return L;
}

// What the epilogue needs of a tile: this head, then per complex column its offset in C and factor 2^(eA - unit_exp);
// and, in one of two sets that consecutive tiles on the same rows share, per row its offset and factor 2^eB (alpha).
struct TileHead {
  cplx* C;
  int rlim, clim;  // rows and complex columns inside the result
  int ngroups;     // groups of EPI_CG columns
  int bn;
  int scaled;      // alpha is not in the factors
  int has_beta;
  int rowset;
  int pad[3];
  cplx alpha, beta;
};
static_assert(sizeof(TileHead) % 16 == 0, "tables follow the head");

constexpr int ROW_TABLE_BYTES = TILE_R * 16;
__host__ __device__ inline int table_set_bytes(int BN) { return (int)sizeof(TileHead) + BN / 2 * 16; }

// bytes after the tile ring: barriers, TMEM slot, flags, two sets of row and of per-tile tables
__host__ __device__ inline int misc_bytes(int stages, int BN) {
  return (2 * stages + 12) * 8 + 32 + 2 * (ROW_TABLE_BYTES + table_set_bytes(BN)) + 64;
}

// A CTA's walk over its tiles: its problem's parameters and maps, and the tile's position as digits (column tile, row
// tile, batch; columns fastest, so neighbours share rows), advanced by adding the digits of the step.  Tile and batch
// counts fit 32 bits (the host checks).
template <bool GROUPED>
struct TileWalk {
  const GemmParams* launch;
  const GemmParams* q;
  const CUtensorMap* mR;
  const CUtensorMap* mC;
  uint32_t t, t_end, step;  // tile of the launch
  uint32_t local;           // tile of the problem
  uint32_t bx, by, bz, sx, sy, sz;
  uint32_t b0, b1, b2, rbA, rbB;
  bool new_rows;            // other rows than the tile before (always so at the start of a run of column tiles)

  __device__ __forceinline__ void batch() {
    const uint32_t nb2 = (uint32_t)q->nb2, nb1 = (uint32_t)q->nb1;
    const uint32_t bq = nb2 == 1 ? bz : bz / nb2;
    b2 = bz - bq * nb2;
    b0 = nb1 == 1 ? bq : bq / nb1;
    b1 = bq - b0 * nb1;
    rbA = (uint32_t)reduced_batch(q->depA, b0, b1, b2, nb1, nb2);
    rbB = (uint32_t)reduced_batch(q->depB, b0, b1, b2, nb1, nb2);
  }
  __device__ __forceinline__ void locate() {
    if constexpr (GROUPED) {
      int lo = 0, hi = launch->ngroup - 1;  // last entry with tile_begin <= t
      while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (launch->group[mid].tile_begin <= (int64_t)t) lo = mid;
        else hi = mid - 1;
      }
      const GroupEntry& e = launch->group[lo];
      q = &e.p;
      mR = &e.mR;
      mC = &e.mC;
      local = t - (uint32_t)e.tile_begin;
    } else {
      local = t;
    }
    const uint32_t tc = (uint32_t)q->tiles_c, tr = (uint32_t)q->tiles_r;
    uint32_t x = local / tc;
    bx = local - x * tc;
    bz = x / tr;
    by = x - bz * tr;
    x = step / tc;
    sx = step - x * tc;
    sz = x / tr;
    sy = x - sz * tr;
    batch();
    new_rows = true;
  }
  __device__ __forceinline__ TileWalk(const GemmParams& p, const CUtensorMap* r, const CUtensorMap* c, uint32_t first,
                                      uint32_t end, uint32_t st)
      : launch(&p), q(&p), mR(r), mC(c), t(first), t_end(end), step(st) {
    if (t < t_end) locate();
  }
  __device__ __forceinline__ bool more() const { return t < t_end; }
  __device__ __forceinline__ void next() {
    t += step;
    if (t >= t_end) return;
    local += step;
    if (GROUPED && local >= (uint32_t)q->ntile) {
      locate();
      return;
    }
    const uint32_t tc = (uint32_t)q->tiles_c, tr = (uint32_t)q->tiles_r, oy = by;
    bx += sx;
    by += sy;
    if (bx >= tc) {
      bx -= tc;
      ++by;
    }
    uint32_t dz = sz;
    if (by >= tr) {
      by -= tr;
      ++dz;
    }
    new_rows = by != oy || dz != 0;
    if (dz) {
      bz += dz;
      batch();
    }
  }
  __device__ __forceinline__ int row0() const { return (int)by * TILE_R; }
  __device__ __forceinline__ int col0() const { return (int)bx * q->BN; }
};

// Persistent tensor-core kernel: every CTA walks tiles blockIdx.x, +gridDim.x, ...
//  warp 0       TMA producer (one thread), a ring of `stages` K blocks that runs across tiles
//  warp 1       MMA issuer (one thread), one TMEM accumulator set of S * BN columns
//  warp 2       tables: what the epilogue needs of the next tile, in two alternating sets
//  warps 3..    epilogue (EPI_WARPS): TMEM -> registers -> FP64 recombination -> stores to C
// Bound by the MMAs for long contractions (8192 multiply-adds a cycle and SM) and by the instructions of the epilogue
// for the short ones (K = 40: 3 K steps of 720 cycles a tile against 12 column groups per scheduler), which is why the
// tile's index arithmetic has a warp of its own and no block barrier separates tiles.
template <int SS, bool GROUPED>
__global__ void __launch_bounds__(NWARPS * 32, 1)
    split_gemm_tc_kernel(const __grid_constant__ CUtensorMap mapR, const __grid_constant__ CUtensorMap mapC,
                         const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const SmemLayout L = smem_layout(p.S, p.BN, p.stages, p.overlap);
  uint8_t* rows_smem = smem;
  uint8_t* tiles = smem + L.rows_bytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L.ring_bytes);
  uint64_t* empty_bar = full_bar + L.stages;
  uint64_t* accf_bar = empty_bar + L.stages;   // [2] accumulator set complete
  uint64_t* acce_bar = accf_bar + 2;           // [2] accumulator set read
  uint64_t* tabf_bar = acce_bar + 2;           // [2] table set filled
  uint64_t* tabe_bar = tabf_bar + 2;           // [2] table set read
  uint64_t* rowf_bar = tabe_bar + 2;           // [2] resident rows loaded
  uint64_t* rowe_bar = rowf_bar + 2;           // [2] resident rows no longer read
  uint8_t* misc = reinterpret_cast<uint8_t*>(rowe_bar + 2);
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 4);
  uint8_t* row_tables = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(misc + 8) + 15) & ~uintptr_t(15));
  uint8_t* tables = row_tables + 2 * ROW_TABLE_BYTES;
  const int tsb = table_set_bytes(p.BN);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  constexpr int S = SS;
  const int nbuf = p.overlap ? 2 : 1;
  const uint32_t acc_cols = (uint32_t)(S * p.BN);
  const uint32_t need = acc_cols * (uint32_t)nbuf;
  const uint32_t ncols_alloc = need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512;
  const int64_t ntiles = GROUPED ? p.ntiles : (int64_t)p.tiles_r * p.tiles_c * p.nb0 * p.nb1 * p.nb2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < L.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&rowf_bar[b], 1);
      mbar_init(&rowe_bar[b], 1);
      mbar_init(&accf_bar[b], 1);
      mbar_init(&acce_bar[b], EPI_WARPS);  // every epilogue warp releases the set it has read
      mbar_init(&tabf_bar[b], 1);
      mbar_init(&tabe_bar[b], EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_base_slot, ncols_alloc);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;

  // this CTA's tiles: every gridDim.x-th one, or, in overlap mode, a contiguous range (columns fastest), in which
  // most neighbours share their rows
  const uint32_t t_first = p.overlap ? (uint32_t)(ntiles * blockIdx.x / gridDim.x) : blockIdx.x;
  const uint32_t t_end = p.overlap ? (uint32_t)(ntiles * (blockIdx.x + 1) / gridDim.x) : (uint32_t)ntiles;
  const uint32_t t_step = p.overlap ? 1u : gridDim.x;
  const int nstage = L.stages;

  uint32_t issued = 0;  // producer: K blocks issued in total
  uint32_t nrows = 0;   // producer: row tiles loaded (overlap mode)
  if (warp == 0) {
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 1;  // a fresh barrier's previous phase counts as complete
      const GemmParams* last_q = nullptr;
      for (TileWalk<GROUPED> w(p, &mapR, &mapC, t_first, t_end, t_step); w.more() && !*abort_flag; w.next()) {
        const GemmParams& q = *w.q;
        if constexpr (GROUPED) {
          if (w.q != last_q) {
            // the problem's tensor maps live in global memory that the host rewrites between
            // launches: order those writes before the tensor-map reads of the loads
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(w.mR) : "memory");
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(w.mC) : "memory");
            last_q = w.q;
          }
        }
        // all S planes of a K block in one load each; rows past a plane's end come as zeros
        const uint32_t rbytes = (uint32_t)(S * L.r_plane_bytes);
        const uint32_t tile_stage_bytes = (uint32_t)(S * q.BN * KBLK) + (p.overlap ? 0u : rbytes);
        const int nkb = q.nkb, row0 = w.row0(), col0 = w.col0(), zr = (int)w.rbB * S, zc = (int)w.rbA * S;
        if (p.overlap && w.new_rows) {
          const uint32_t rset = nrows & 1;
          if (!mbar_wait(&rowe_bar[rset], ((nrows >> 1) & 1) ^ 1, abort_flag)) {
            atomicExch(p.err, SERR_TIMEOUT_PRODUCER);
            *abort_flag = 1;
            break;
          }
          ++nrows;
          mbar_expect_tx(&rowf_bar[rset], rbytes * (uint32_t)nkb);
          for (int kb = 0; kb < nkb; ++kb)
            tma_load_3d(rows_smem + (size_t)(rset * RES_KB + kb) * rbytes, w.mR, kb * KBLK, row0, zr, &rowf_bar[rset]);
        }
        bool ok = true;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&empty_bar[st], ph, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* sbase = tiles + (size_t)st * L.stage_bytes;
          mbar_expect_tx(&full_bar[st], tile_stage_bytes);
          if (!p.overlap) tma_load_3d(sbase, w.mR, kb * KBLK, row0, zr, &full_bar[st]);
          tma_load_3d(sbase + L.stage_rows, w.mC, kb * KBLK, col0, zc, &full_bar[st]);
          ++issued;
          if (++st == nstage) {
            st = 0;
            ph ^= 1;
          }
        }
        if (!ok) {
          atomicExch(p.err, SERR_TIMEOUT_PRODUCER);
          *abort_flag = 1;
          break;
        }
      }
    }
  } else if (warp == 1) {
    // Slice plane s of the rows meets the S - s first planes of the columns at once: they lie one after another in the
    // stage, and their products belong to the consecutive diagonals s .. S - 1, so they are one MMA of (S - s) BN
    // columns (two when that is above 256).  For S = 5 and 96 columns a 32-byte K step is 8 MMAs that run at the tensor
    // pipe's 8192 multiply-adds a cycle; one MMA per pair of planes (15 of 96 columns) is bound by the shared-memory
    // reads of its operands (56 cycles for 48 of work).  The descriptors' upper halves and the widths are fixed per
    // tile; per stage only base addresses are added.
    const uint32_t issue = elect_one();
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw64(0) >> 32);
    const uint32_t ring_lo = (uint32_t)smem_desc_sw64(smem_u32(tiles));
    const uint32_t rows_lo = (uint32_t)smem_desc_sw64(smem_u32(rows_smem));
    const uint32_t stage_lo = (uint32_t)L.stage_bytes >> 4, plane_lo = (uint32_t)L.r_plane_bytes >> 4;
    const uint32_t cols_lo = (uint32_t)L.stage_rows >> 4;
    const int overlap = p.overlap;
    int st = 0, buf = 0;
    uint32_t ph = 0, acc_ph = 1, rows_seen = 0;
    for (TileWalk<GROUPED> w(p, &mapR, &mapC, t_first, t_end, t_step); w.more(); w.next()) {
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      const int tbn = w.q->BN, nkb = w.q->nkb;
      int ksteps = w.q->nkk;  // 32-byte K steps left
      bool ok = mbar_wait(&acce_bar[buf], acc_ph, abort_flag);
      if (overlap && w.new_rows) {
        if (rows_seen > 0) umma_commit(&rowe_bar[(rows_seen - 1) & 1], issue);  // the previous rows' MMAs are all issued
        ok = ok && mbar_wait(&rowf_bar[rows_seen & 1], (rows_seen >> 1) & 1, abort_flag);
        ++rows_seen;
      }
      const uint32_t acc = tmem_base + (uint32_t)buf * acc_cols;
      const uint32_t rows_set = rows_lo + ((rows_seen - 1) & 1) * (uint32_t)(RES_KB * S) * plane_lo;
      uint32_t accum = 0;
      for (int kb = 0; kb < nkb; ++kb) {
        ok = ok && mbar_wait(&full_bar[st], ph, abort_flag);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        const uint32_t s_lo = ring_lo + (uint32_t)st * stage_lo;
        const uint32_t a_lo = overlap ? rows_set + (uint32_t)(kb * S) * plane_lo : s_lo;  // row planes of this K block
        const uint32_t b_lo = s_lo + cols_lo;
#pragma unroll
        for (int kk = 0; kk < KBLK / 32; ++kk) {
          if (kk < ksteps) {
            const uint64_t bd = ((uint64_t)desc_hi << 32) | (b_lo + 2 * kk);
#pragma unroll
            for (int s = 0; s < S; ++s) {
              const uint64_t ad = ((uint64_t)desc_hi << 32) | (a_lo + (uint32_t)s * plane_lo + 2 * kk);
              const uint32_t dt = acc + (uint32_t)(s * tbn);
              const int n = (S - s) * tbn;
              if (n <= 256) {
                umma_i8(dt, ad, bd, idesc_i8(n), accum, issue);
              } else {
                const int n0 = (n / 2 + 15) / 16 * 16;
                umma_i8(dt, ad, bd, idesc_i8(n0), accum, issue);
                umma_i8(dt + (uint32_t)n0, ad, bd + (uint32_t)(n0 * (KBLK / 16)), idesc_i8(n - n0), accum, issue);
              }
              accum = 1;
            }
          }
        }
        ksteps -= KBLK / 32;
        umma_commit(&empty_bar[st], issue);
        if (++st == nstage) {
          st = 0;
          ph ^= 1;
        }
      }
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          atomicExch(p.err, SERR_TIMEOUT_MMA);
          *abort_flag = 1;
        }
        break;
      }
      umma_commit(&accf_bar[buf], issue);
      if (++buf == nbuf) {
        buf = 0;
        acc_ph ^= 1;
      }
    }
  } else if (warp == 2) {
    // (this warp works beside four busy epilogue warps, so it keeps to what changes: the problem's constants are written
    // once per set, and 32-bit indices serve wherever a tile's share allows)
    uint32_t tcount = 0, nr = 0;  // tiles, row tables written (the last in set (nr - 1) & 1)
    const GemmParams* head_q[2] = {nullptr, nullptr};
    for (TileWalk<GROUPED> w(p, &mapR, &mapC, t_first, t_end, t_step); w.more(); w.next(), ++tcount) {
      const int set = (int)(tcount & 1);
      const GemmParams& q = *w.q;
      const int64_t row0 = w.row0(), m0 = w.col0() >> 1;
      const int half = q.BN >> 1;
      const int rlim = (int)(q.N - row0 < TILE_R ? q.N - row0 : TILE_R), clim = (int)(q.M - m0 < half ? q.M - m0 : half);
      // this tile's exponents are on their way while the table set is waited for
      const int32_t* eA = q.eA + w.rbA * q.eA_ld + m0;
      const bool cin = lane < clim;
      const int e0 = cin ? eA[lane] : 0;
      const int64_t o0 = cin ? q.C.row(m0 + lane) : 0;
      const bool ok = mbar_wait(&tabe_bar[set], ((tcount >> 1) & 1) ^ 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          atomicExch(p.err, SERR_TIMEOUT_TABLES);
          *abort_flag = 1;
        }
        break;
      }
      uint8_t* tb = tables + set * tsb;
      int64_t* coff = reinterpret_cast<int64_t*>(tb + sizeof(TileHead));
      double* csc = reinterpret_cast<double*>(coff + half);
      if (w.new_rows) {
        // new rows go to the other row set; its last tile lies at least two tiles back and has been stored
        int64_t* roff = reinterpret_cast<int64_t*>(row_tables + (nr & 1) * ROW_TABLE_BYTES);
        double* rsc = reinterpret_cast<double*>(roff + TILE_R);
        ++nr;
        // a real alpha that is a power of two is folded into the row factor (exact, so the result equals the validation
        // engine's alpha * value)
        const double al = q.alpha_pow2 ? q.alpha.x : 1.0;
        const int32_t* eB = q.eB + w.rbB * q.eB_ld + row0;
        int e[TILE_R / 32];
#pragma unroll
        for (int j = 0; j < TILE_R / 32; ++j) e[j] = lane + 32 * j < rlim ? eB[lane + 32 * j] : 0;
#pragma unroll
        for (int j = 0; j < TILE_R / 32; ++j) {
          const int i = lane + 32 * j;
          roff[i] = i < rlim ? q.C.col(row0 + i) : 0;
          rsc[i] = pow2(e[j]) * al;
        }
      }
      if (lane < half) {
        coff[lane] = o0;
        csc[lane] = pow2(e0 - unit_exp(S));
      }
      for (int i = lane + 32; i < half; i += 32) {
        const bool in = i < clim;
        coff[i] = in ? q.C.row(m0 + i) : 0;
        csc[i] = pow2((in ? eA[i] : 0) - unit_exp(S));
      }
      if (lane == 0) {
        TileHead& h = *reinterpret_cast<TileHead*>(tb);
        h.C = q.C.ptr + q.C.bat(w.b0, w.b1, w.b2);
        h.rlim = rlim;
        h.clim = clim;
        h.ngroups = (2 * clim + EPI_CG - 1) / EPI_CG;
        h.rowset = (int)((nr - 1) & 1);
        if (head_q[set] != w.q) {
          h.bn = q.BN;
          h.scaled = !q.alpha_pow2;
          h.has_beta = q.beta.x != 0.0 || q.beta.y != 0.0;
          h.alpha = q.alpha;
          h.beta = q.beta;
        }
      }
      head_q[set] = w.q;
      __syncwarp();
      if (lane == 0) mbar_arrive_local(&tabf_bar[set]);
    }
  } else {
    // epilogue warps: TMEM sub-partition = warp % 4, one row of the tile per lane; the EPI_WARPS / 4 warps of a
    // sub-partition take the groups of EPI_CG columns in turn.
    const int sp = warp % 4;
    const int row = sp * 32 + lane;
    uint32_t tcount = 0, acc_ph = 0, turn = (uint32_t)(warp - EPI_FIRST) / 4;
    int buf = 0;
    for (uint32_t t = t_first; t < t_end; t += t_step, ++tcount) {
      const int set = (int)(tcount & 1);
      const bool ok = mbar_wait(&tabf_bar[set], (tcount >> 1) & 1, abort_flag) && mbar_wait(&accf_bar[buf], acc_ph, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          atomicExch(p.err, SERR_TIMEOUT_EPILOGUE);
          *abort_flag = 1;
        }
        break;
      }
      tc_fence_after();
      const uint8_t* tb = tables + set * tsb;
      const TileHead& h = *reinterpret_cast<const TileHead*>(tb);
      const int64_t* roff = reinterpret_cast<const int64_t*>(row_tables + h.rowset * ROW_TABLE_BYTES);
      const double* rsc = reinterpret_cast<const double*>(roff + TILE_R);
      const int bn = h.bn, clim = h.clim;
      const int64_t* coff = reinterpret_cast<const int64_t*>(tb + sizeof(TileHead));
      const double* csc = reinterpret_cast<const double*>(coff + bn / 2);
      // a warp whose 32 rows all lie outside the result has no groups
      const int ng = sp * 32 < h.rlim ? h.ngroups : 0;
      const bool rok = row < h.rlim;
      const double rs = rsc[row];
      cplx* Crow = h.C + roff[row];
      const bool plain = !h.scaled && !h.has_beta;
      const uint32_t acc = tmem_base + (uint32_t)buf * acc_cols + ((uint32_t)(sp * 32) << 16);
      // the first group rotates, so that a group count that is no multiple of four loads the warps evenly
      const int gfirst = (int)(turn & 3u);
      turn += (uint32_t)(bn / EPI_CG);
      for (int g = gfirst; g < ng; g += EPI_WARPS / 4) {
        // all S diagonals of 8 columns in one TMEM round trip
        int32_t dq[S][EPI_CG];
#pragma unroll
        for (int d = 0; d < S; ++d) tmem_ld8(acc + (uint32_t)(d * bn + g * EPI_CG), dq[d]);
        tmem_wait_ld();
        cplx v[EPI_CG / 2];
#pragma unroll
        for (int j = 0; j < EPI_CG / 2; ++j) {
          int32_t qr[S], qi[S];
#pragma unroll
          for (int d = 0; d < S; ++d) {
            qr[d] = dq[d][2 * j];
            qi[d] = dq[d][2 * j + 1];
          }
          const double sc = rs * csc[g * (EPI_CG / 2) + j];
          v[j] = cmk(combine_diagonals<S>(qr) * sc, combine_diagonals<S>(qi) * sc);
        }
        if (g + EPI_WARPS / 4 >= ng) {
          // this warp's reads of the accumulators are complete: release them to the MMA warp
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_local(&acce_bar[buf]);
        }
        const int c0 = g * (EPI_CG / 2);
        if (rok) {
          if (plain) {
#pragma unroll
            for (int j = 0; j < EPI_CG / 2; ++j)
              if (c0 + j < clim) Crow[coff[c0 + j]] = v[j];
          } else {
#pragma unroll
            for (int j = 0; j < EPI_CG / 2; ++j)
              if (c0 + j < clim) {
                cplx* d = Crow + coff[c0 + j];
                cplx val = h.scaled ? cmul(h.alpha, v[j]) : v[j];
                if (h.has_beta) val = cadd(val, cmul(h.beta, *d));
                *d = val;
              }
          }
        }
      }
      if (gfirst >= ng) {  // no group of this tile was this warp's
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_local(&acce_bar[buf]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive_local(&tabe_bar[set]);
      if (++buf == nbuf) {
        buf = 0;
        acc_ph ^= 1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // after an abort, let in-flight TMA loads land before the shared memory is released
  if (warp == 0 && lane == 0 && *abort_flag) {
    for (uint32_t k = (issued > (uint32_t)nstage ? issued - nstage : 0); k < issued; ++k) {
      const long long t0 = clock64();
      while (!mbar_try_wait(&full_bar[k % nstage], (k / nstage) & 1))
        if (clock64() - t0 > WAIT_LIMIT) break;
    }
    for (uint32_t k = (nrows > 2 ? nrows - 2 : 0); k < nrows; ++k) {
      const long long t0 = clock64();
      while (!mbar_try_wait(&rowf_bar[k & 1], (k >> 1) & 1))
        if (clock64() - t0 > WAIT_LIMIT) break;
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ncols_alloc);
  }
}

// ----------------------------------------------------------------------------
// CUDA-core validation core: the same diagonal INT32 sums from the same planes.
// ----------------------------------------------------------------------------
template <int S>
__global__ void split_gemm_ref_kernel(const int8_t* Ap, const int8_t* Bp, int64_t kpad, GemmParams p) {
  const int64_t bz = blockIdx.z;
  const int64_t b2 = bz % p.nb2, b1 = (bz / p.nb2) % p.nb1, b0 = bz / (p.nb2 * p.nb1);
  const int64_t rbA = reduced_batch(p.depA, b0, b1, b2, p.nb1, p.nb2);
  const int64_t rbB = reduced_batch(p.depB, b0, b1, b2, p.nb1, p.nb2);
  const int64_t m = (int64_t)blockIdx.y * 16 + threadIdx.y;
  const int64_t n = (int64_t)blockIdx.x * 16 + threadIdx.x;
  if (m >= p.M || n >= p.N) return;
  int32_t qr[S], qi[S];
#pragma unroll
  for (int d = 0; d < S; ++d) {
    int32_t accr = 0, acci = 0;
    for (int s = 0; s <= d; ++s) {
      const int8_t* a0 = Ap + ((rbA * S + s) * p.rowsA + 2 * m) * kpad;
      const int8_t* a1 = a0 + kpad;
      const int8_t* bb = Bp + ((rbB * S + d - s) * p.rowsB + n) * kpad;
      for (int64_t k = 0; k < kpad; ++k) {
        accr += (int32_t)a0[k] * (int32_t)bb[k];
        acci += (int32_t)a1[k] * (int32_t)bb[k];
      }
    }
    qr[d] = accr;
    qi[d] = acci;
  }
  const double sc = pow2(p.eB[rbB * p.eB_ld + n]) * pow2(p.eA[rbA * p.eA_ld + m] - unit_exp(S));
  cplx* dst = p.C.ptr + p.C.bat(b0, b1, b2) + p.C.row(m) + p.C.col(n);
  cplx v = cmul(p.alpha, cmk(combine_diagonals<S>(qr) * sc, combine_diagonals<S>(qi) * sc));
  if (p.beta.x != 0.0 || p.beta.y != 0.0) v = cadd(v, cmul(p.beta, *dst));
  *dst = v;
}

// ----------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  require(fn != nullptr, GB200_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  return fn;
}

// planes [nplanes][rows][kpad] of an operand; a load takes box_rows rows of one K block from S planes
CUtensorMap make_map(const int8_t* base, int64_t kpad, int64_t rows, int64_t nplanes, int box_rows, int S) {
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows, (cuuint64_t)nplanes};
  cuuint64_t strides[2] = {(cuuint64_t)kpad, (cuuint64_t)(kpad * rows)};
  cuuint32_t box[3] = {(cuuint32_t)KBLK, (cuuint32_t)box_rows, (cuuint32_t)S};
  cuuint32_t estr[3] = {1, 1, 1};
  require((reinterpret_cast<uintptr_t>(base) & 15) == 0 && kpad % 16 == 0, GB200_ERR_INVALID, "TMA alignment");
  CUresult r = get_encode()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  require(r == CUDA_SUCCESS, GB200_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return m;
}

inline int64_t rup(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

void deps_of(const ZOperand& o, int dep[3]) {
  dep[0] = (o.bat.tab0 != nullptr || o.bat.s0 != 0) ? 1 : 0;
  dep[1] = o.bat.s1 != 0 ? 1 : 0;
  dep[2] = o.bat.s2 != 0 ? 1 : 0;
}

int64_t nrb_of(const int dep[3], const ZGemm& g) {
  int64_t n = 1;
  if (dep[0]) n *= g.nb0;
  if (dep[1]) n *= g.nb1;
  if (dep[2]) n *= g.nb2;
  return n;
}

}  // namespace

struct SplitEngine {
  int core = 0;  // 0: tcgen05, 1: CUDA-core validation core
  DevArray<int8_t> planesA, planesB;
  DevArray<int32_t> expA, expB;
  DevArray<int> err;
  DevArray<GroupEntry> group;  // problems of a grouped launch (tensor maps, parameters, tile ranges)
  bool attr_set = false;
};

SplitEngine* split_engine(Context& c) {
  if (!c.split) c.split = new SplitEngine();
  c.split->core = c.split_core;
  return c.split;
}

void split_release(Context& c) {
  delete c.split;
  c.split = nullptr;
}

namespace {

__global__ void fill_int_kernel(int32_t* e, int64_t n, int32_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) e[i] = v;
}

// widest column tile for S diagonals in `cols` TMEM columns, a multiple of 16
int max_bn(int S, int cols) {
  int bn = (cols / S) / 16 * 16;
  return std::max(16, std::min(bn, 256));
}

unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 8)); }

// the digit-writing kernels for the job's slice count (a template parameter of the kernels)
void launch_write(const SliceJob& j, dim3 g, cudaStream_t st) {
  switch (j.S) {
    case 2: slice_write_kernel<2><<<g, SL_NT, 0, st>>>(j); break;
    case 3: slice_write_kernel<3><<<g, SL_NT, 0, st>>>(j); break;
    case 4: slice_write_kernel<4><<<g, SL_NT, 0, st>>>(j); break;
    case 5: slice_write_kernel<5><<<g, SL_NT, 0, st>>>(j); break;
    case 6: slice_write_kernel<6><<<g, SL_NT, 0, st>>>(j); break;
    case 7: slice_write_kernel<7><<<g, SL_NT, 0, st>>>(j); break;
    default: slice_write_kernel<8><<<g, SL_NT, 0, st>>>(j); break;
  }
  GB_CHECK_LAUNCH();
}

template <int RB>
void launch_resident(const SliceJob& j, dim3 g, size_t sm, int kt, cudaStream_t st) {
  switch (j.S) {
    case 2: slice_resident_kernel<RB, 2><<<g, SL_NT, sm, st>>>(j, kt); break;
    case 3: slice_resident_kernel<RB, 3><<<g, SL_NT, sm, st>>>(j, kt); break;
    case 4: slice_resident_kernel<RB, 4><<<g, SL_NT, sm, st>>>(j, kt); break;
    case 5: slice_resident_kernel<RB, 5><<<g, SL_NT, sm, st>>>(j, kt); break;
    case 6: slice_resident_kernel<RB, 6><<<g, SL_NT, sm, st>>>(j, kt); break;
    case 7: slice_resident_kernel<RB, 7><<<g, SL_NT, sm, st>>>(j, kt); break;
    default: slice_resident_kernel<RB, 8><<<g, SL_NT, sm, st>>>(j, kt); break;
  }
}

// Opt-in shared memory above 48 KB for the kernels that use it (once per engine).
void set_smem_attrs(SplitEngine& se) {
  if (se.attr_set) return;
  const void* fns[] = {
#define GB_TC_ALL(G)                                                                                     \
  (const void*)split_gemm_tc_kernel<2, G>, (const void*)split_gemm_tc_kernel<3, G>,                      \
      (const void*)split_gemm_tc_kernel<4, G>, (const void*)split_gemm_tc_kernel<5, G>,                  \
      (const void*)split_gemm_tc_kernel<6, G>, (const void*)split_gemm_tc_kernel<7, G>,                  \
      (const void*)split_gemm_tc_kernel<8, G>
      GB_TC_ALL(false), GB_TC_ALL(true),
#undef GB_TC_ALL
#define GB_RES_ALL(RB)                                                                        \
  (const void*)slice_resident_kernel<RB, 2>, (const void*)slice_resident_kernel<RB, 3>,       \
      (const void*)slice_resident_kernel<RB, 4>, (const void*)slice_resident_kernel<RB, 5>,   \
      (const void*)slice_resident_kernel<RB, 6>, (const void*)slice_resident_kernel<RB, 7>,   \
      (const void*)slice_resident_kernel<RB, 8>
      GB_RES_ALL(8), GB_RES_ALL(16)
#undef GB_RES_ALL
  };
  for (const void* f : fns) GB_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  se.attr_set = true;
}

// Slice one operand (rows x K) into planes + exponents.
void run_slicer(SliceJob& j, int64_t nrb, cudaStream_t st) {
  const int64_t ne = nrb * j.e_ld;
  require(nrb < 65536, GB200_ERR_INVALID, "split: too many operand batches");
  if (j.kpad / 2 <= TK) {
    // the whole contraction range fits one tile: one pass finds the exponents and writes the slices
    j.single = 1;
    dim3 g((unsigned)((j.rpad + TR - 1) / TR), 1, (unsigned)nrb);
    launch_write(j, g, st);
    return;
  }
  j.single = 0;
  const int64_t nkt = (j.kpad / 2 + TK - 1) / TK;  // K tiles covering the padded range
  if (nkt <= 8) {
    // moderate contraction length: the block's rows stay in shared memory for both steps
    const int kt = (int)nkt * TK;
    if (nkt <= 4) {
      const size_t sm = resident_smem(16, kt);
      dim3 g((unsigned)((j.rpad + 15) / 16), 1, (unsigned)nrb);
      launch_resident<16>(j, g, sm, kt, st);
    } else {
      const size_t sm = resident_smem(8, kt);
      dim3 g((unsigned)((j.rpad + 7) / 8), 1, (unsigned)nrb);
      launch_resident<8>(j, g, sm, kt, st);
    }
    GB_CHECK_LAUNCH();
    return;
  }
  fill_int_kernel<<<blocks_for(ne), 256, 0, st>>>(j.expo, ne, EXP_EMPTY);
  GB_CHECK_LAUNCH();
  require(nrb < 65536, GB200_ERR_INVALID, "split: too many operand batches");
  dim3 g1((unsigned)((j.R + TR - 1) / TR), (unsigned)((j.K + TK - 1) / TK), (unsigned)nrb);
  require(g1.y < 65536, GB200_ERR_INVALID, "split: contraction too long for the slicer grid");
  slice_expo_kernel<<<g1, SL_NT, 0, st>>>(j);
  GB_CHECK_LAUNCH();
  dim3 g2((unsigned)((j.rpad + TR - 1) / TR), (unsigned)((j.kpad / 2 + TK - 1) / TK), (unsigned)nrb);
  launch_write(j, g2, st);
  fix_empty_expo_kernel<<<blocks_for(ne), 256, 0, st>>>(j.expo, ne);
  GB_CHECK_LAUNCH();
}

}  // namespace

namespace {

// largest K chunk for which no INT32 diagonal can overflow: S * 2K * 128^2 < 2^31 (base 128: 64^2 at most)
int64_t kmax_for(int S) {
  int64_t kmax = (int64_t)(2147483647.0 / (2.0 * 128.0 * 128.0 * S));
  return kmax / 32 * 32;
}

// Tile width of a problem, in real columns of the embedded operand (2 M of them): one TMEM accumulator set of up to 512
// columns (two of half that in overlap mode), no more than the context's limit, and below that the multiple of 16 with
// which the tiles cost least: their number times the rows and columns of planes that a K step brings from L2; in overlap
// mode a tile costs its epilogue and about 16 columns' worth of waits.  Five slices at nao = 24 to 48: a limit of 80, 64,
// 48 or 32 columns is 0-6, 0-8, 6-12 or 21-36 % slower than none (gb200/tile_table.json).
int tile_width(const Context& c, int S, int64_t M, bool overlap) {
  int top = max_bn(S, overlap ? 256 : 512);
  if (c.tile_bn > 0) top = std::min(top, std::max(16, c.tile_bn / 16 * 16));
  top = std::min<int>(top, (int)std::min<int64_t>(rup(2 * M, 16), 256));
  int best = top;
  double cost = 1e300;
  for (int bn = top; bn >= 16 && 2 * bn >= top; bn -= 16) {
    const double x = std::ceil(2.0 * (double)M / bn) * (bn + (overlap ? 16.0 : (double)TILE_R));
    if (x < cost) {
      cost = x;
      best = bn;
    }
  }
  return best;
}

// bytes of a plane's row for Kc complex K positions: whole 32-byte K steps of the MMA; a last half block is filled with
// zeros by the TMA load
int64_t row_bytes(int64_t Kc) { return std::max<int64_t>(KBLK, rup(2 * Kc, 32)); }

struct Prepared {
  GemmParams p{};
  CUtensorMap mR{}, mC{};
  int64_t kpad = 0, ntiles = 0;
  double flops = 0.0;
};

// Slice K chunk [k0, k0 + Kc) of both operands into the engine's planes and fill the problem's
// parameters (and, for the tensor-core engine, its tensor maps).
Prepared prepare_chunk(SplitEngine& se, const ZGemm& g0, int S, int BN, int64_t k0, int64_t Kc, cudaStream_t st) {
  Prepared pr;
  set_smem_attrs(se);
  int depA[3], depB[3];
  deps_of(g0.A, depA);
  deps_of(g0.B, depB);
  const int64_t nrbA = nrb_of(depA, g0), nrbB = nrb_of(depB, g0);
  const int64_t rowsA = 2 * g0.M, rowsB = g0.N;
  if (!se.err.p) {
    se.err.alloc(1);
    GB_CUDA(cudaMemsetAsync(se.err.p, 0, sizeof(int), st));
  }
  const int64_t kpad = row_bytes(Kc);
  SplitBuffers buf;
  buf.cover(g0, S);
  se.planesA.alloc(buf.planesA);
  se.planesB.alloc(buf.planesB);
  se.expA.alloc(buf.expA);
  se.expB.alloc(buf.expB);
  auto slice = [&](const ZOperand& o, const IdxMap& rmap, const IdxMap& kmap, const int* dep, int64_t R, int64_t nrb,
                   int embed, int8_t* out, int32_t* expo) {
    SliceJob j{};
    j.ptr = o.ptr; j.rmap = rmap; j.kmap = kmap; j.bat = o.bat; j.conj = o.conj;
    j.R = R; j.K = Kc; j.k0 = k0; j.n0 = g0.nb0; j.n1 = g0.nb1; j.n2 = g0.nb2;
    std::copy(dep, dep + 3, j.dep);
    j.embed = embed; j.S = S; j.rows_pad = embed ? 2 * R : R; j.rpad = R; j.kpad = kpad; j.e_ld = R;
    j.out = out; j.expo = expo;
    j.r_fast = std::abs(rmap.s_in) < std::abs(kmap.s_in);
    run_slicer(j, nrb, st);
  };
  slice(g0.A, g0.A.row, g0.A.col, depA, g0.M, nrbA, 1, se.planesA.p, se.expA.p);
  slice(g0.B, g0.B.col, g0.B.row, depB, g0.N, nrbB, 0, se.planesB.p, se.expB.p);
  GemmParams& p = pr.p;
  p.S = S; p.BN = BN; p.nkb = (int)((kpad + KBLK - 1) / KBLK); p.nkk = (int)(kpad / 32);
  p.M = g0.M; p.N = g0.N; p.nb0 = g0.nb0; p.nb1 = g0.nb1; p.nb2 = g0.nb2;
  std::copy(depA, depA + 3, p.depA);
  std::copy(depB, depB + 3, p.depB);
  p.rowsA = rowsA; p.rowsB = rowsB;
  p.eA = se.expA.p; p.eB = se.expB.p; p.eA_ld = g0.M; p.eB_ld = g0.N;
  p.C = g0.C; p.alpha = g0.alpha; p.beta = (k0 == 0) ? g0.beta : cmk(1.0, 0.0);
  p.err = se.err.p;
  {
    int aexp = 0;
    p.alpha_pow2 = (g0.alpha.y == 0.0 && g0.alpha.x != 0.0 && std::fabs(std::frexp(g0.alpha.x, &aexp)) == 0.5) ? 1 : 0;
  }
  const int64_t nbatch = g0.nb0 * g0.nb1 * g0.nb2;
  require(nbatch < 65536, GB200_ERR_INVALID, "split: too many batches for one launch");
  p.tiles_r = (int)((g0.N + TILE_R - 1) / TILE_R);
  p.tiles_c = (int)((rowsA + BN - 1) / BN);
  pr.kpad = kpad;
  pr.ntiles = (int64_t)p.tiles_r * p.tiles_c * nbatch;
  require(pr.ntiles < (1LL << 31), GB200_ERR_INVALID, "split: too many tiles for one launch");
  p.ntile = (int)pr.ntiles;
  pr.flops = 8.0 * (double)g0.M * (double)g0.N * (double)Kc * (double)nbatch;
  if (se.core == 0) {
    const int64_t totalA = nrbA * S * rowsA, totalB = nrbB * S * rowsB;
    require(totalA < (1LL << 31) && totalB < (1LL << 31), GB200_ERR_INVALID, "split: operand too large for TMA");
    pr.mR = make_map(se.planesB.p, kpad, rowsB, nrbB * S, TILE_R, S);
    pr.mC = make_map(se.planesA.p, kpad, rowsA, nrbA * S, BN, S);
  }
  return pr;
}

template <bool G>
void launch_tc(int S, unsigned grid, size_t smem, cudaStream_t st, const CUtensorMap& mR, const CUtensorMap& mC,
               const GemmParams& p) {
  switch (S) {
    case 2: split_gemm_tc_kernel<2, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    case 3: split_gemm_tc_kernel<3, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    case 4: split_gemm_tc_kernel<4, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    case 5: split_gemm_tc_kernel<5, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    case 6: split_gemm_tc_kernel<6, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    case 7: split_gemm_tc_kernel<7, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
    default: split_gemm_tc_kernel<8, G><<<grid, NWARPS * 32, smem, st>>>(mR, mC, p); break;
  }
  GB_CHECK_LAUNCH();
}

void launch_ref(int S, dim3 grid, cudaStream_t st, const int8_t* A, const int8_t* B, int64_t kpad, const GemmParams& p) {
  const dim3 block(16, 16);
  switch (S) {
    case 2: split_gemm_ref_kernel<2><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    case 3: split_gemm_ref_kernel<3><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    case 4: split_gemm_ref_kernel<4><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    case 5: split_gemm_ref_kernel<5><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    case 6: split_gemm_ref_kernel<6><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    case 7: split_gemm_ref_kernel<7><<<grid, block, 0, st>>>(A, B, kpad, p); break;
    default: split_gemm_ref_kernel<8><<<grid, block, 0, st>>>(A, B, kpad, p); break;
  }
  GB_CHECK_LAUNCH();
}

// Launch-wide layout for tiles up to BN columns: TMA ring depth (what fits, at most 6 K blocks)
// and the dynamic shared memory.
void ring_layout(int S, int BN, GemmParams& p, size_t& smem) {
  const SmemLayout L1 = smem_layout(S, BN, 1, p.overlap);
  const int room = SMEM_MAX - 1024 /*alignment*/ - misc_bytes(6, BN) - L1.rows_bytes;
  p.stages = std::max(1, std::min(room / L1.stage_bytes, 6));
  smem = (size_t)smem_layout(S, BN, p.stages, p.overlap).ring_bytes + 1024 + misc_bytes(p.stages, BN);
  require(smem <= SMEM_MAX, GB200_ERR_INVALID, "split: shared memory budget exceeded");
}

bool overlap_mode(int S, int64_t K) { return S <= OVERLAP_MAX_S && 2 * K <= RES_KB * KBLK; }

KernelRecord* begin_record(Context& c, double flops, cudaStream_t st) {
  if (!c.stats_on) return nullptr;
  if (c.records_used == c.records.size()) {
    KernelRecord r;
    GB_CUDA(cudaEventCreate(&r.start));
    GB_CUDA(cudaEventCreate(&r.stop));
    c.records.push_back(r);
  }
  KernelRecord* rec = &c.records[c.records_used++];
  rec->alg_flops = flops;  // FP64-equivalent work: 8 real flops per complex multiply-add
  GB_CUDA(cudaEventRecord(rec->start, st));
  return rec;
}

unsigned persistent_grid(const Context& c, int64_t ntiles) {
  require(ntiles < (1LL << 31), GB200_ERR_INVALID, "split: too many tiles for one launch");
  int nsm = 148;
  GB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
  return (unsigned)std::min<int64_t>(ntiles, nsm);  // one CTA per SM walks the tiles
}

}  // namespace

void SplitBuffers::cover(const ZGemm& g, int S) {
  int depA[3], depB[3];
  deps_of(g.A, depA);
  deps_of(g.B, depB);
  const int64_t nrbA = nrb_of(depA, g), nrbB = nrb_of(depB, g), kpad = row_bytes(std::min(kmax_for(S), g.K));
  planesA = std::max(planesA, (size_t)(nrbA * S * 2 * g.M * kpad));
  planesB = std::max(planesB, (size_t)(nrbB * S * g.N * kpad));
  expA = std::max(expA, (size_t)(nrbA * g.M));
  expB = std::max(expB, (size_t)(nrbB * g.N));
}

void split_reserve(Context& c, const SplitBuffers& b) {
  SplitEngine& e = *split_engine(c);
  e.planesA.alloc(b.planesA);
  e.planesB.alloc(b.planesB);
  e.expA.alloc(b.expA);
  e.expB.alloc(b.expB);
}

size_t split_held(const Context& c) {
  if (!c.split) return 0;
  const SplitEngine& e = *c.split;
  return e.planesA.n + e.planesB.n + (e.expA.n + e.expB.n) * sizeof(int32_t);
}

void split_gemm(Context& c, SplitEngine& se, const ZGemm& g0, cudaStream_t st, int slices) {
  if (g0.M <= 0 || g0.N <= 0) return;
  validate(g0);
  const int S = slices > 0 ? slices : c.slices;
  require(S >= 2 && S <= 8, GB200_ERR_INVALID, "split: slices out of range");
  require(g0.K > 0, GB200_ERR_INVALID, "split: empty contraction");
  const bool overlap = overlap_mode(S, g0.K);
  const int BN = tile_width(c, S, g0.M, overlap);
  const int64_t kmax = kmax_for(S);
  for (int64_t k0 = 0; k0 < g0.K; k0 += kmax) {
    const int64_t Kc = std::min(kmax, g0.K - k0);
    Prepared pr = prepare_chunk(se, g0, S, BN, k0, Kc, st);
    const int64_t nbatch = g0.nb0 * g0.nb1 * g0.nb2;
    if (se.core == 1) {
      dim3 grid((unsigned)((g0.N + 15) / 16), (unsigned)((g0.M + 15) / 16), (unsigned)nbatch);
      launch_ref(S, grid, st, se.planesA.p, se.planesB.p, pr.kpad, pr.p);
      continue;
    }
    size_t smem = 0;
    pr.p.overlap = overlap ? 1 : 0;
    ring_layout(S, BN, pr.p, smem);
    KernelRecord* rec = begin_record(c, pr.flops, st);
    launch_tc<false>(S, persistent_grid(c, pr.ntiles), smem, st, pr.mR, pr.mC, pr.p);
    if (rec) GB_CUDA(cudaEventRecord(rec->stop, st));
  }
}

void split_gemm_group(const std::vector<Context*>& cs, const std::vector<ZGemm>& gs, cudaStream_t st, int slices) {
  require(cs.size() == gs.size() && !cs.empty(), GB200_ERR_INVALID, "split group: one contraction per context");
  const int S = slices;
  require(S >= 2 && S <= 8, GB200_ERR_INVALID, "split: slices out of range");
  const int64_t kmax = kmax_for(S);
  std::vector<SplitEngine*> ses;
  std::vector<int> bns;
  int64_t nch = 0;
  bool tc_engine = true, overlap = true;
  for (size_t i = 0; i < cs.size(); ++i) {
    for (size_t j = 0; j < i; ++j)
      require(cs[j] != cs[i], GB200_ERR_INVALID, "split group: a context appears twice (its slice buffers are shared)");
    validate(gs[i]);
    require(gs[i].K > 0 && gs[i].M > 0 && gs[i].N > 0, GB200_ERR_INVALID, "split group: empty contraction");
    ses.push_back(split_engine(*cs[i]));
    tc_engine = tc_engine && ses.back()->core == 0;
    overlap = overlap && overlap_mode(S, gs[i].K);
    nch = std::max<int64_t>(nch, (gs[i].K + kmax - 1) / kmax);
  }
  if (!tc_engine) {  // the CUDA-core validation engine has no grouped form
    for (size_t i = 0; i < cs.size(); ++i) split_gemm(*cs[i], *ses[i], gs[i], st, S);
    return;
  }
  for (size_t i = 0; i < cs.size(); ++i) bns.push_back(tile_width(*cs[i], S, gs[i].M, overlap));
  SplitEngine& se0 = *ses[0];
  // K chunk ch of every problem that has one, all in one grouped launch per chunk
  for (int64_t ch = 0; ch < nch; ++ch) {
    std::vector<GroupEntry> entries;
    int BNmax = 16;
    double flops = 0.0;
    int64_t total = 0;
    for (size_t i = 0; i < cs.size(); ++i) {
      const int64_t k0 = ch * kmax;
      if (k0 >= gs[i].K) continue;
      Prepared pr = prepare_chunk(*ses[i], gs[i], S, bns[i], k0, std::min(kmax, gs[i].K - k0), st);
      GroupEntry e;
      e.mR = pr.mR;
      e.mC = pr.mC;
      e.p = pr.p;
      e.tile_begin = total;
      entries.push_back(e);
      total += pr.ntiles;
      BNmax = std::max(BNmax, bns[i]);
      flops += pr.flops;
    }
    GemmParams p{};
    p.S = S;
    p.BN = BNmax;
    p.overlap = overlap ? 1 : 0;
    p.err = se0.err.p;
    size_t smem = 0;
    ring_layout(S, BNmax, p, smem);
    se0.group.alloc(entries.size());
    GB_CUDA(cudaMemcpyAsync(se0.group.p, entries.data(), entries.size() * sizeof(GroupEntry), cudaMemcpyHostToDevice, st));
    p.group = se0.group.p;
    p.ngroup = (int)entries.size();
    p.ntiles = total;
    KernelRecord* rec = begin_record(*cs[0], flops, st);
    launch_tc<true>(S, persistent_grid(*cs[0], total), smem, st, entries[0].mR, entries[0].mC, p);
    if (rec) GB_CUDA(cudaEventRecord(rec->stop, st));
  }
}

int split_check_error(Context& c, cudaStream_t st) {
  if (!c.split || !c.split->err.p) return 0;
  int h = 0;
  GB_CUDA(cudaMemcpyAsync(&h, c.split->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  if (h) GB_CUDA(cudaMemsetAsync(c.split->err.p, 0, sizeof(int), st));
  return h;
}

}  // namespace gb200
