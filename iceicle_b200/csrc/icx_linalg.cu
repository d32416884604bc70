// Device linear algebra for the Newton solver: block-diagonal inversion
// (block-Jacobi preconditioner), block-ILU(0) on the element block pattern,
// deterministic reductions and the multi-vector kernels of GMRES.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "icx_internal.h"
#include "icx_linalg.h"
#include "icx_blockrow.cuh"
#include "icx_blockinv.cuh"
#include "icx_ilu_rows.cuh"

namespace icx {

// ----------------------------------------------------- block inversion
// gj_invert / write_inverse / InvSmem: icx_blockinv.cuh

// inverse of one diagonal block per CTA; a singular block becomes the
// identity and raises *flag (the preconditioner degrades to no-op on it)
template <int BS>
__global__ void __launch_bounds__(256) block_invert_kernel(int nblk, const double* __restrict__ src,
                                                           const int* __restrict__ blk_index,
                                                           double* __restrict__ dst, int* flag) {
  extern __shared__ double sh[];
  double* a = sh;
  double* fcol = a + BS * BS;
  int* perm = reinterpret_cast<int*>(fcol + BS);
  int* colsrc = perm + BS;
  __shared__ int singular;
  int b = blockIdx.x;
  if (b >= nblk) return;
  const double* A = src + (size_t)blk_index[b] * BS * BS;
  for (int t = threadIdx.x; t < BS * BS; t += blockDim.x) a[t] = A[t];
  __syncthreads();
  gj_invert<BS>(a, perm, fcol, &singular);
  __syncthreads();
  if (singular && threadIdx.x == 0) atomicExch(flag, 1);
  write_inverse<BS>(a, perm, colsrc, singular, dst + (size_t)b * BS * BS);
}

// ------------------------------------------------------------ block-ILU(0)
// Block ILU(0) on the element block pattern in natural (element) order, IKJ
// form: for each row e, for each lower block (e, k) in ascending k,
//   A_ek <- A_ek inv(A_kk);  A_ej -= A_ek A_kj  for every (k, j), j > k, with (e, j) in the pattern;
// then inv(A_ee) is stored for the next rows and the backward solve. On the
// structured element grid row (i, j) depends only on (i-1, j) and (i, j-1),
// so the rows of one anti-diagonal i + j = level are independent (in a batch
// of grids, the rows of that level in every grid): one launch per level, one
// CTA per row.

__device__ inline int find_block(const int* rowptr, const int* colidx, int r, int c) {
  for (int k = rowptr[r]; k < rowptr[r + 1]; ++k)
    if (colidx[k] == c) return k;
  return -1;
}

// C = X Y for BS x BS blocks in shared memory, each thread owning 4 x 4
// output tiles; op(r0, c0, acc) consumes every finished tile
template <int BS>
__device__ inline void block_gemm_tile(const double* X, const double* Y, int r0, int c0, double (&acc)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  for (int m = 0; m < BS; ++m) {
    double xa[4], yb[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) xa[a] = (r0 + a < BS) ? X[(r0 + a) * BS + m] : 0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b) yb[b] = (c0 + b < BS) ? Y[m * BS + c0 + b] : 0.0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] += xa[a] * yb[b];
  }
}

// Shapes of the row factorisation and of the block products. Blocks whose size
// is a multiple of 4 (above 4) go through the FP64 matrix instructions
// (8 x 8 x 4): warp w owns rows 8 w .. 8 w + 7 of the result, lane l rows l / 4
// and column pairs 8 t + 2 (l % 4); staged blocks have rows of LD doubles, LD * 8
// bytes = 32 modulo 128, so that neither operand's fragments conflict in shared
// memory. Odd sizes keep a 4 x 4 tile per thread. The rate of the FP64 pipe is
// the same either way (64 multiply-adds per clock and SM); what the matrix form
// saves is shared memory reads: a 64 x 64 product took 10,400 cycles with 4 x 4
// tiles, 4,096 being the pipe's bound.
template <int BS>
struct BlkCfg {
  static constexpr bool MMA = BS % 4 == 0 && BS > 4;
  static constexpr int LD = MMA && BS % 16 != 4 ? (BS / 16 * 16 + 4 < BS ? BS / 16 * 16 + 20 : BS / 16 * 16 + 4) : BS;
  static constexpr int NM = (BS + 7) / 8;                // 8-row tiles: warps of a product
  static constexpr int KS = BS / 4;                      // its steps
  static constexpr int NT4 = (BS + 3) / 4, TILES = NT4 * NT4;
  static constexpr int WORK = MMA ? NM * 32 : TILES;     // threads of a product
  static constexpr int ACC = MMA ? 2 * NM : 16;          // results per thread
};
static_assert(BlkCfg<64>::LD == 68 && BlkCfg<36>::LD == 36 && BlkCfg<16>::LD == 20 && BlkCfg<100>::LD == 100, "strides");

// position (row, column) of a thread's n-th result
template <int BS>
__device__ inline int2 blk_pos(int n) {
  using K = BlkCfg<BS>;
  const int tid = threadIdx.x;
  if constexpr (K::MMA) {
    const int lane = tid & 31;
    return make_int2((tid >> 5) * 8 + lane / 4, (n >> 1) * 8 + (lane % 4) * 2 + (n & 1));
  } else {
    return make_int2(tid / K::NT4 * 4 + n / 4, tid % K::NT4 * 4 + n % 4);
  }
}

// acc = X Y; X and Y in shared memory with rows of LD doubles (whole warps call it)
template <int BS>
__device__ inline void blk_mul(const double* X, const double* Y, double (&acc)[BlkCfg<BS>::ACC]) {
  using K = BlkCfg<BS>;
  const int tid = threadIdx.x;
  if constexpr (K::MMA) {
    const int lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int n = 0; n < K::ACC; ++n) acc[n] = 0.0;
    // rows and columns past the block meet clamped addresses; their results are not used
    const int row = w * 8 + lane / 4;
    const double* x = X + (row < BS ? row : BS - 1) * K::LD + lane % 4;
    const double* y = Y + (lane % 4) * K::LD + lane / 4;
    constexpr int LAST = (K::NM - 1) * 8;
    const int yl = LAST + lane / 4 < BS ? LAST : LAST - (LAST + 8 - BS);
#pragma unroll 4
    for (int m = 0; m < K::KS; ++m) {
      const double av = x[m * 4];
#pragma unroll
      for (int t = 0; t < K::NM; ++t) {
        const double bv = y[m * 4 * K::LD + (t == K::NM - 1 ? yl : t * 8)];
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
            : "+d"(acc[2 * t]), "+d"(acc[2 * t + 1])
            : "d"(av), "d"(bv));
      }
    }
  } else {
    double c[4][4];
    block_gemm_tile<BS>(X, Y, tid / K::NT4 * 4, tid % K::NT4 * 4, c);
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n] = c[n / 4][n % 4];
  }
}

// a thread's results to rows of ld doubles (global or shared); matrix form: pairs of columns
template <int BS>
__device__ inline void blk_store(const double (&acc)[BlkCfg<BS>::ACC], double* dst, int ld) {
  using K = BlkCfg<BS>;
  if constexpr (K::MMA) {
#pragma unroll
    for (int n = 0; n < K::ACC; n += 2) {
      const int2 p = blk_pos<BS>(n);
      if (p.x < BS && p.y < BS) *reinterpret_cast<double2*>(dst + p.x * ld + p.y) = make_double2(acc[n], acc[n + 1]);
    }
  } else {
#pragma unroll
    for (int n = 0; n < K::ACC; ++n) {
      const int2 p = blk_pos<BS>(n);
      if (p.x < BS && p.y < BS) dst[p.x * ld + p.y] = acc[n];
    }
  }
}

// copies a block to shared memory with rows of LD doubles (asynchronously)
template <int BS>
__device__ inline void block_fetch(double* dst, const double* __restrict__ src) {
  constexpr int LD = BlkCfg<BS>::LD;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BS % 2 == 0) {
    for (int t = threadIdx.x; t < BS * BS / 2; t += blockDim.x) {
      const int o = LD == BS ? 2 * t : 2 * t / BS * LD + 2 * t % BS;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + o * 8), "l"(src + 2 * t) : "memory");
    }
  } else {
    for (int t = threadIdx.x; t < BS * BS; t += blockDim.x)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d + t * 8), "l"(src + t) : "memory");
  }
}

// One CTA factors one element's row. Both lower neighbours' operands are
// requested at the start (cp.async) and the diagonal block stays in registers
// through its updates and its inversion.
//
// Inversion: in-place Gauss-Jordan with partial pivoting. Rows are not exchanged:
// the pivot of column k is the largest |a[i][k]| of the rows not yet used (first
// index on ties), and with p_k that row the stored matrix S gives
// inv[k][p_j] = S[p_k][j].
//   matrix form (blk_invert): eight columns at a time. One warp takes the panel
//     of those columns through its eight pivots alone (whole-warp maximum, no
//     barrier, every lane forming its candidate's reciprocal meanwhile); with
//     the panel M that leaves and the eight pivot rows R as they were, every
//     other entry becomes a[i][j] (0 in a pivot row) + M[i] . R[:, j], two matrix
//     instructions per 8 x 8 tile on the tiles the warps hold. Three barriers per
//     eight pivots instead of a barrier and a selection among the warps for each.
//   odd sizes (block_invert_regs): TPR threads per row, thread q holding columns
//     q, q + TPR, ...; every warp offers its best row and all pick the winner.
template <int BS>
struct FacCfg {
  using B = BlkCfg<BS>;
  static constexpr int TPR = BS > 64 ? 4 : 2;
  static constexpr int NC = (BS + TPR - 1) / TPR;        // columns per thread
  static constexpr int NCP = (NC + 3) / 4 * 4 + 2;       // stride of a thread's part of an offer (16-byte reads of
                                                         // the TPR parts fall in different banks)
  static constexpr int GJ = BS * TPR;                    // threads of the inversion
  static constexpr int GW = (GJ + 31) / 32;              // its warps
  static constexpr int THREADS = ((B::WORK > GJ ? B::WORK : GJ) + 31) / 32 * 32;
  static constexpr int B2 = BS * BS;
  static constexpr int B2P = (BS * B::LD + 1) / 2 * 2;   // a staged block
  // operand buffers: A_ek, inv(U_kk), A_ke of two neighbours, or (largest blocks) two buffers used in turn
  static constexpr int NBUF = 6 * B2P * 8 <= 212 * 1024 ? 6 : 2;
  static constexpr int OFFER = GW * TPR * NCP;           // doubles of one pivot's offers
  // scratch of the inversion: the panel and the pivot rows, or the offers and candidates; pivot rows by column,
  // columns by pivot row, flag
  static constexpr int PS = 12, WK = B::MMA ? BS * PS + 8 * B::LD : 2 * OFFER + 4 * GW;
  static constexpr size_t SMEM = sizeof(double) * ((size_t)NBUF * B2P + WK) + sizeof(int) * (2 * BS + 4);
  static_assert(SMEM <= 227 * 1024, "the row's operands exceed the shared memory of one CTA");
};

// dst (global) = inverse of the block in shared memory at `a` (rows of LD), which is overwritten; false (uniform
// over the CTA) if it is singular, dst then the identity
template <int BS>
__device__ inline bool block_invert_regs(double* a, double* offers, uint4* cand, int* perm, double* dst) {
  using K = FacCfg<BS>;
  constexpr int TPR = K::TPR, NC = K::NC, NCP = K::NCP, LD = BlkCfg<BS>::LD;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool singular = false;
  double m[NC];
  const bool mine = tid < K::GJ;
  const int r = mine ? tid / TPR : 0, q = tid % TPR;
  int kr = 0;  // the column whose pivot this row is
  if (warp < K::GW) {
#pragma unroll
    for (int j = 0; j < NC; ++j) m[j] = mine && q + TPR * j < BS ? a[r * LD + q + TPR * j] : 0.0;
    bool used = !mine;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
#pragma unroll
      for (int qq = 0; qq < TPR; ++qq) {
        const int k = qq + TPR * j;
        if (k >= BS || singular) break;
        const int par = k & 1;
        double* offer = offers + par * K::OFFER;
        const double f = __shfl_sync(0xffffffffu, m[j], (lane & ~(TPR - 1)) | qq);  // a[r][k]
        // the warp's largest |a[i][k]| of the rows not used (a NaN counts as zero)
        unsigned hi = 0, lo = 0;
        if (!used && f == f) {
          hi = (unsigned)__double2hiint(f) & 0x7fffffffu;
          lo = (unsigned)__double2loint(f);
        }
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        const unsigned who = __ballot_sync(0xffffffffu, !used && hi == mh && lo == ml);
        const int first = who ? __ffs(who) - 1 : 0;
        if (who && lane / TPR == first / TPR) {
          double2* o = reinterpret_cast<double2*>(offer + (warp * TPR + q) * NCP);
#pragma unroll
          for (int h = 0; h < (NC + 1) / 2; ++h) o[h] = make_double2(m[2 * h], 2 * h + 1 < NC ? m[2 * h + 1] : 0.0);
        }
        unsigned bh = mh, bl = ml, row = (unsigned)(warp * 32 + first) / TPR;
        int bw = warp;
        if constexpr (K::GW == 1) {
          __syncwarp();
        } else {
          if (lane == 0) cand[par * K::GW + warp] = make_uint4(mh, ml, row, 0u);
          asm volatile("bar.sync 1, %0;" ::"n"(K::GW * 32) : "memory");
          // the winner: largest, then lowest warp (rows ascend with the warps)
          bh = bl = 0;
#pragma unroll
          for (int w = 0; w < K::GW; ++w) {
            const uint4 cw = cand[par * K::GW + w];
            if (cw.x > bh || (cw.x == bh && cw.y > bl)) {
              bh = cw.x;
              bl = cw.y;
              row = cw.z;
              bw = w;
            }
          }
        }
        if ((bh | bl) == 0) {  // no nonzero pivot: uniform over the inversion's warps
          singular = true;
        } else {
          if (tid == 0) perm[k] = (int)row;
          const double* o = offer + bw * TPR * NCP;
          const double ri = 1.0 / o[qq * NCP + j];
          const double2* oq = reinterpret_cast<const double2*>(o + q * NCP);
          const bool own = mine && r == (int)row;
          // the pivot row becomes ri times itself, the others lose f ri times it: with z = 0 for the pivot row,
          // both are z a[i] + g a[p]
          const double g = own ? ri : -(f * ri);
#pragma unroll
          for (int h = 0; h < (NC + 1) / 2; ++h) {
            const double2 pr = oq[h];
#pragma unroll
            for (int w = 0; w < 2; ++w)
              if (2 * h + w < NC) m[2 * h + w] = fma(g, w ? pr.y : pr.x, own ? 0.0 : m[2 * h + w]);
          }
          if (q == qq) m[j] = g;
          if (own) {
            used = true;
            kr = k;
          }
          if constexpr (K::GW == 1) __syncwarp();
        }
      }
    }
    if (tid == 0) perm[BS] = singular ? 1 : 0;
  }
  __syncthreads();
  singular = perm[BS] != 0;
  if (mine && !singular) {
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (q + TPR * j < BS) a[kr * LD + perm[q + TPR * j]] = m[j];
  }
  __syncthreads();
  for (int t = tid; t < BS * BS; t += blockDim.x) dst[t] = singular ? (t / BS == t % BS ? 1.0 : 0.0) : a[t / BS * LD + t % BS];
  return !singular;
}

// the inverse of the block whose tiles the warps hold (C, as blk_mul's results) into dst (global), through out
// (shared, rows of LD); work: the inversion's shared scratch; false (uniform over the CTA) if it is singular, dst
// then the identity
template <int BS>
__device__ inline bool blk_invert(double (&C)[BlkCfg<BS>::ACC], double* out, double* work, int* perm, double* dst) {
  using K = FacCfg<BS>;
  using B = BlkCfg<BS>;
  constexpr int LD = B::LD, NM = B::NM, PS = K::PS, RPL = (BS + 31) / 32;
  double* PB = work;             // [BS][PS]: the panel
  double* R = work + BS * PS;    // [8][LD]: its pivot rows before the update
  int* rank = perm + BS;         // the column a row was pivot of (-1: not yet)
  int* fail = rank + BS;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int row = w * 8 + lane / 4, q = lane % 4;
  const bool mine = w < NM && row < BS;
  for (int i = tid; i < BS; i += blockDim.x) rank[i] = -1;
  if (tid == 0) *fail = 0;
#pragma unroll
  for (int t = 0; t < NM; ++t) {
    constexpr int LASTC = BS - (NM - 1) * 8;
    const int nc = t == NM - 1 ? LASTC : 8;  // columns of the panel (4 or 8)
    if (mine && 2 * q < nc) *reinterpret_cast<double2*>(PB + row * PS + 2 * q) = make_double2(C[2 * t], C[2 * t + 1]);
    __syncthreads();
    if (w == 0) {
      // the panel's pivots: lane l holds rows l, l + 32, ...
      double p[RPL][8];
      bool used[RPL];
#pragma unroll
      for (int rr = 0; rr < RPL; ++rr) {
        const int r = lane + 32 * rr;
        used[rr] = r >= BS || rank[r] >= 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) p[rr][c] = r < BS && c < nc ? PB[r * PS + c] : 0.0;
      }
      bool bad = false;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c >= nc || bad) break;
        // the lane's largest candidate (a NaN counts as zero; first row on ties) and its reciprocal
        unsigned long long key = 0;
        int br = 0;
#pragma unroll
        for (int rr = 0; rr < RPL; ++rr) {
          const unsigned long long v = !used[rr] && p[rr][c] == p[rr][c]
                                           ? (unsigned long long)__double_as_longlong(p[rr][c]) & 0x7fffffffffffffffull
                                           : 0ull;
          if (v > key) {
            key = v;
            br = rr;
          }
        }
        double bv = p[0][c];
#pragma unroll
        for (int rr = 1; rr < RPL; ++rr) bv = br == rr ? p[rr][c] : bv;
        const double rl = 1.0 / bv;
        const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        // the lowest row among equal candidates
        const unsigned mr = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)(lane + 32 * br) : ~0u);
        if ((mh | ml) == 0) {
          bad = true;
          break;
        }
        const int src = mr & 31, sr = mr >> 5;  // uniform
        const double ri = __shfl_sync(0xffffffffu, rl, src);
        double pr[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          double v = p[0][k];
#pragma unroll
          for (int rr = 1; rr < RPL; ++rr) v = sr == rr ? p[rr][k] : v;
          pr[k] = __shfl_sync(0xffffffffu, v, src);
        }
#pragma unroll
        for (int rr = 0; rr < RPL; ++rr) {
          const bool own = lane == src && rr == sr;
          const double g = own ? ri : -(p[rr][c] * ri);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k != c) p[rr][k] = fma(g, pr[k], own ? 0.0 : p[rr][k]);
          p[rr][c] = g;
          used[rr] = used[rr] || own;
        }
        if (lane == 0) {
          perm[t * 8 + c] = (int)mr;
          rank[mr] = t * 8 + c;
        }
      }
      if (bad) {
        if (lane == 0) *fail = 1;
      } else {
#pragma unroll
        for (int rr = 0; rr < RPL; ++rr) {
          const int r = lane + 32 * rr;
          if (r < BS) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (c < nc) PB[r * PS + c] = p[rr][c];
          }
        }
      }
    }
    __syncthreads();
    if (*fail) break;  // uniform
    // the pivot rows as they were, then out of the tiles
    if (mine) {
      const int k = rank[row] - t * 8;
      if (k >= 0) {
#pragma unroll
        for (int n = 0; n < NM; ++n) {
          if (n * 8 + 2 * q < BS) *reinterpret_cast<double2*>(R + k * LD + n * 8 + 2 * q) = make_double2(C[2 * n], C[2 * n + 1]);
          C[2 * n] = C[2 * n + 1] = 0.0;
        }
      }
    }
    __syncthreads();
    if (w < NM) {
      const double* a = PB + (row < BS ? row : BS - 1) * PS + q;
      const double a0 = a[0], a1 = nc > 4 ? a[4] : 0.0;
      const double* b = R + q * LD + lane / 4;
      constexpr int LAST = (NM - 1) * 8;
      const int yl = LAST + lane / 4 < BS ? LAST : LAST - (LAST + 8 - BS);
#pragma unroll
      for (int n = 0; n < NM; ++n) {
        if (n == t) continue;
        const int o = n == NM - 1 ? yl : n * 8;
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
            : "+d"(C[2 * n]), "+d"(C[2 * n + 1])
            : "d"(a0), "d"(b[o]));
        if (nc > 4)
          asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
              : "+d"(C[2 * n]), "+d"(C[2 * n + 1])
              : "d"(a1), "d"(b[4 * LD + o]));
      }
      const double2 v = mine && 2 * q < nc ? *reinterpret_cast<const double2*>(PB + row * PS + 2 * q) : make_double2(0.0, 0.0);
      C[2 * t] = v.x;
      C[2 * t + 1] = v.y;
    }
    __syncthreads();  // the panel and the pivot rows are read before the next ones are written
  }
  const bool singular = *fail != 0;
  if (mine && !singular) {
#pragma unroll
    for (int n = 0; n < B::ACC; ++n) {
      const int col = (n >> 1) * 8 + 2 * q + (n & 1);
      if (col < BS) out[rank[row] * LD + perm[col]] = C[n];
    }
  }
  __syncthreads();
  for (int t = tid; t < BS * BS; t += blockDim.x) dst[t] = singular ? (t / BS == t % BS ? 1.0 : 0.0) : out[t / BS * LD + t % BS];
  return !singular;
}

// What bounds it: the chain of BS pivots and the four block products of an inner
// element. Whole factorisation and one apply, before (4 x 4 tiles, three barriers
// per pivot with the block in shared memory) and now: Navier-Stokes 64 x 64 p = 2
// 9.4 and 3.7 ms, p = 3 26.2 and 8.0 ms, 40 x 40 p = 4 50.4 and 17.4 ms; tiles of
// 8, 128 x 128 p = 2 4.9 and 2.1 ms; Burgers 64 x 64 p = 2 2.9 and 1.9 ms.
template <int BS>
__global__ void __launch_bounds__(FacCfg<BS>::THREADS) ilu_level_kernel(int E, int nnzb, const int* __restrict__ elems,
                                                                        const int* __restrict__ rowptr,
                                                                        const int* __restrict__ colidx,
                                                                        double* LU, double* Uinv, int* flag) {
  using K = FacCfg<BS>;
  using B = BlkCfg<BS>;
  constexpr int B2 = K::B2, LD = B::LD;
  extern __shared__ __align__(16) double sh[];
  double* offers = sh + (size_t)K::NBUF * K::B2P;
  int* perm = reinterpret_cast<int*>(offers + K::WK);
  const int tid = threadIdx.x;
  const int e = elems[blockIdx.x];
  // block and element indices are checked before use: a bad one sets
  // *flag = 2 and the CTA leaves (the values are uniform over the CTA)
  if (e < 0 || e >= E || rowptr[e] < 0 || rowptr[e + 1] > nnzb) {
    if (tid == 0) atomicExch(flag, 2);
    return;
  }
  const int b0 = rowptr[e];
  const int kd = find_block(rowptr, colidx, e, e);
  bool bad = kd < 0;
  for (int kl = b0; !bad && kl < kd; ++kl) bad = colidx[kl] < 0 || colidx[kl] >= e;  // columns ascend
  if (bad) {
    if (tid == 0) atomicExch(flag, 2);
    return;
  }
  // neighbour n's operands in buffers 3 n .. 3 n + 2 (A_ek, inv(U_kk), A_ke)
  const int nl = kd - b0;
  auto fetch = [&](int n) {
    const int k = colidx[b0 + n];
    double* buf = sh + (size_t)(K::NBUF == 6 ? 3 * (n & 1) : 0) * K::B2P;
    block_fetch<BS>(buf, LU + (size_t)(b0 + n) * B2);
    block_fetch<BS>(buf + K::B2P, Uinv + (size_t)k * B2);
    if (K::NBUF == 6) {
      const int ke = find_block(rowptr, colidx, k, e);
      if (ke >= 0) block_fetch<BS>(buf + 2 * K::B2P, LU + (size_t)ke * B2);
    }
    cp_async_commit();
  };
  if (nl > 0) fetch(0);
  if (K::NBUF == 6 && nl > 1) fetch(1);
  const bool work = tid < B::WORK;
  double D[B::ACC], acc[B::ACC];
#pragma unroll
  for (int n = 0; n < B::ACC; ++n) {
    const int2 p = blk_pos<BS>(n);
    D[n] = work && p.x < BS && p.y < BS ? LU[(size_t)kd * B2 + p.x * BS + p.y] : 0.0;
  }
  for (int n = 0; n < nl; ++n) {
    const int kl = b0 + n, k = colidx[kl];
    double* X = sh + (size_t)(K::NBUF == 6 ? 3 * (n & 1) : 0) * K::B2P;
    double* Y = X + K::B2P;
    if (K::NBUF == 6 && n + 1 < nl) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    // L_ek = A_ek inv(U_kk) over A_ek (matrix form: a warp reads and writes its own rows only)
    if (work) blk_mul<BS>(X, Y, acc);
    if (B::MMA) __syncwarp();
    else __syncthreads();
    if (work) {
      blk_store<BS>(acc, X, LD);
      blk_store<BS>(acc, LU + (size_t)kl * B2, BS);
    }
    if (B::MMA) __syncwarp();
    else __syncthreads();
    // A_ej -= L_ek U_kj for the upper blocks of row k that lie in row e's pattern (on a quadrilateral grid: e's
    // own diagonal block only)
    bool have_z = K::NBUF == 6;  // A_ke is in its buffer
    for (int kj = rowptr[k]; kj < rowptr[k + 1]; ++kj) {
      const int jc = colidx[kj];
      if (jc <= k) continue;
      const int ej = jc == e ? kd : find_block(rowptr, colidx, e, jc);
      if (ej < 0) continue;  // outside the pattern: dropped (level 0 fill)
      if (kj >= nnzb || ej >= nnzb) {  // uniform over the CTA
        if (tid == 0) atomicExch(flag, 2);
        cp_async_wait<0>();
        return;
      }
      double* Z = K::NBUF == 6 ? X + 2 * K::B2P : Y;
      if (!have_z || jc != e) {
        have_z = false;
        __syncthreads();
        for (int t = tid; t < B2; t += blockDim.x) Z[t / BS * LD + t % BS] = LU[(size_t)kj * B2 + t];
        __syncthreads();
      }
      if (work) {
        blk_mul<BS>(X, Z, acc);
#pragma unroll
        for (int m = 0; m < B::ACC; ++m) {
          const int2 p = blk_pos<BS>(m);
          if (jc == e) D[m] -= acc[m];
          else if (p.x < BS && p.y < BS) LU[(size_t)ej * B2 + p.x * BS + p.y] -= acc[m];
        }
      }
      if (K::NBUF == 6 && jc < e && n + 1 < nl) {  // this may be the next neighbour's A_ek, staged as it was before
        cp_async_wait<0>();
        __syncthreads();
        double* Xn = sh + (size_t)(3 * ((n + 1) & 1)) * K::B2P;
        for (int t = tid; t < B2; t += blockDim.x) Xn[t / BS * LD + t % BS] = LU[(size_t)(kl + 1) * B2 + t];
      }
    }
    // buffers of this neighbour are free
    if (n + (K::NBUF == 6 ? 2 : 1) < nl) {
      __syncthreads();
      fetch(n + (K::NBUF == 6 ? 2 : 1));
    }
  }
  if (work && nl > 0) blk_store<BS>(D, LU + (size_t)kd * B2, BS);
  __syncthreads();
  bool ok;
  if constexpr (B::MMA) {
    ok = blk_invert<BS>(D, sh, offers, perm, Uinv + (size_t)e * B2);
  } else {
    if (work) blk_store<BS>(D, sh, LD);
    __syncthreads();
    ok = block_invert_regs<BS>(sh, offers, reinterpret_cast<uint4*>(offers + 2 * K::OFFER), perm, Uinv + (size_t)e * B2);
  }
  if (!ok && tid == 0) atomicExch(flag, 1);
}

// After the factorisation every upper block is scaled by the inverse of its
// row's diagonal block, U_ek <- inv(U_ee) U_ek (k > e), so that the backward
// substitution y_e = inv(U_ee) (f_e - sum_{k>e} U_ek y_k) becomes
//   y_e = inv(U_ee) f_e - sum_{k>e} (inv(U_ee) U_ek) y_k,
// a plain block-row product whose rows can be split across warps.
// One CTA per row, the operands staged in shared memory.
template <int BS>
struct ScaleCfg {
  static constexpr int THREADS = (BlkCfg<BS>::WORK + 31) / 32 * 32;
  static constexpr int B2P = FacCfg<BS>::B2P;
  static constexpr size_t SMEM = sizeof(double) * 2 * B2P;
};

template <int BS>
__global__ void __launch_bounds__(ScaleCfg<BS>::THREADS) ilu_scale_upper_kernel(int E, const int* __restrict__ rowptr,
                                                                                const int* __restrict__ colidx,
                                                                                double* LU,
                                                                                const double* __restrict__ Uinv) {
  using B = BlkCfg<BS>;
  extern __shared__ __align__(16) double sh[];
  double* D = sh;
  double* U = sh + ScaleCfg<BS>::B2P;
  const int e = blockIdx.x;
  if (e >= E) return;
  block_fetch<BS>(D, Uinv + (size_t)e * BS * BS);
  for (int kb = rowptr[e]; kb < rowptr[e + 1]; ++kb) {
    if (colidx[kb] <= e) continue;
    double* g = LU + (size_t)kb * BS * BS;
    __syncthreads();
    block_fetch<BS>(U, g);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (threadIdx.x < B::WORK) {
      double acc[B::ACC];
      blk_mul<BS>(D, U, acc);
      blk_store<BS>(acc, g, BS);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();  // a row without upper blocks still has its first copy in flight
}

// ------------------------------------------------------------- reductions
// partial[j * nblocks + b] = sum over block b's rows of V_j . x (V_j = V + j*ld;
// an FP32 basis is widened to FP64 before the product), G vectors per pass
// over x: each thread holds x_i once per group of G basis vectors, so x is
// read ceil(nvec / G) times instead of nvec times (the vectors V_j once
// each); per block the sums are reduced by shuffles, then across the warps in
// a fixed order. Few rows per thread make that reduction the larger part, so a
// warp folds its G sums together (9 exchanges for 8 sums instead of 40, the
// same values) and a single vector takes G = 1: 15 FP32 vectors of 589824
// values 19.9 -> 18.3 us, a norm 6.4 -> 3.7 us (both with 1184 blocks). With a ticket the last block to finish adds the blocks'
// partial sums as mdot_final_kernel does, in the same order: for small grids
// and few vectors that is over before a second launch would have begun
template <class TV, int G>
__global__ void __launch_bounds__(256) mdot_grouped_kernel(long long n, const TV* __restrict__ V, long long ld,
                                                           int nvec, const double* __restrict__ x, double* partial,
                                                           unsigned* ticket, double* __restrict__ out) {
  __shared__ double red[G][8];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j0 = 0; j0 < nvec; j0 += G) {
    double acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = 0.0;
#pragma unroll 2
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
      const double xi = x[i];
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (j0 + g < nvec) acc[g] += (double)V[(size_t)(j0 + g) * ld + i] * xi;
    }
    const RowSum<double> sum = warp_row_sums<G>(acc);
    if (sum.owner) red[sum.row][warp] = sum.v;
    __syncthreads();
    if (threadIdx.x < G && j0 + (int)threadIdx.x < nvec) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += red[threadIdx.x][w];
      partial[(size_t)(j0 + threadIdx.x) * gridDim.x + blockIdx.x] = s;
      if (ticket) __threadfence();
    }
    __syncthreads();
  }
  if (!ticket) return;
  // the counter wraps to 0 with the last block: ready for the next launch
  if (threadIdx.x == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int j = warp; j < nvec; j += 8) {
    double v[8];  // what threads lane, lane + 32, ... of mdot_final_kernel hold
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.0;
    for (int b0 = 0; b0 < (int)gridDim.x; b0 += 256)
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int b = b0 + lane + 32 * k;
        if (b < (int)gridDim.x) v[k] += __ldcg(partial + (size_t)j * gridDim.x + b);
      }
#pragma unroll
    for (int h = 4; h > 0; h >>= 1)
#pragma unroll
      for (int k = 0; k < h; ++k) v[k] += v[k + h];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], off);
    if (lane == 0) out[j] = v[0];
  }
}

__global__ void mdot_final_kernel(int nblocks, int nvec, const double* __restrict__ partial, double* __restrict__ out) {
  __shared__ double red[256];
  int j = blockIdx.x;
  double s = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += partial[(size_t)j * nblocks + b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[j] = red[0];
}

// w += sign * sum_j h[j] V_j
template <class TV>
__global__ void maxpy_kernel(long long n, const TV* __restrict__ V, long long ld, int nvec,
                             const double* __restrict__ h, double sign, double* __restrict__ w) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < nvec; ++j) s += h[j] * (double)V[(size_t)j * ld + i];
    w[i] += sign * s;
  }
}

// v32 = a x rounded to FP32
__global__ void scale_to_f32_kernel(long long n, double a, const double* __restrict__ x, float* __restrict__ v32) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v32[i] = (float)(a * x[i]);
}

// v32 = w / sqrt(*h2) rounded to FP32 (w itself when *h2 is not positive)
__global__ void normalize_to_f32_kernel(long long n, const double* __restrict__ h2, const double* __restrict__ w,
                                        float* __restrict__ v32) {
  const double h = *h2;
  const double a = h > 0.0 ? 1.0 / sqrt(h) : 1.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v32[i] = (float)(a * w[i]);
}

// y = a x + b y
__device__ inline double axpby_val(double a, double x, double b, double y) { return a * x + b * y; }

__global__ void axpby_kernel(long long n, double a, const double* __restrict__ x, double b, double* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = axpby_val(a, x[i], b, y[i]);
}

// v /= sqrt(*h2) when *h2 > 0, with the same operations as
// la_axpby(n, 1 / sqrt(h2), v, 0, v) after the host has read h2
__global__ void normalize_kernel(long long n, const double* __restrict__ h2, double* v) {
  const double h = *h2;
  if (!(h > 0.0)) return;
  const double a = 1.0 / sqrt(h);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v[i] = axpby_val(a, v[i], 0.0, v[i]);
}

// z = x + a y
__global__ void xpay_kernel(long long n, const double* __restrict__ x, double a, const double* __restrict__ y,
                            double* __restrict__ z) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    z[i] = x[i] + a * y[i];
}

// ------------------------------------------------------------- launchers
static int grid_for(long long n) {
  long long g = (n + 255) / 256;
  return (int)(g < 148 * 8 ? (g < 1 ? 1 : g) : 148 * 8);
}

// a block per 256 rows up to kMdotBlocks (blocks without a row would add zeros). Up to a block per SM the last one
// sums the partials: a Krylov step of 9216 unknowns 98 us against 107; with 1184 blocks their fences and tickets
// cost more than the second launch (a norm of 589824 values 11.0 us against 6.4 + 2.3)
template <class TV>
static cudaError_t mdot(LinalgWork& w, long long n, const TV* V, long long ld, int nvec, const double* x,
                        double* d_out, cudaStream_t s) {
  const int nb = std::min(grid_for(n), kMdotBlocks);
  const bool fuse = nb <= kMdotFuse;
  unsigned* ticket = fuse ? w.ticket() : nullptr;
  if (nvec == 1) mdot_grouped_kernel<TV, 1><<<nb, 256, 0, s>>>(n, V, ld, nvec, x, w.partial, ticket, d_out);
  else mdot_grouped_kernel<TV, 8><<<nb, 256, 0, s>>>(n, V, ld, nvec, x, w.partial, ticket, d_out);
  if (!fuse) mdot_final_kernel<<<nvec, 256, 0, s>>>(nb, nvec, w.partial, d_out);
  return cudaGetLastError();
}

cudaError_t la_mdot(LinalgWork& w, long long n, const double* V, long long ld, int nvec, const double* x,
                    double* d_out, cudaStream_t s) {
  return mdot(w, n, V, ld, nvec, x, d_out, s);
}

cudaError_t la_mdot32(LinalgWork& w, long long n, const float* V, long long ld, int nvec, const double* x,
                      double* d_out, cudaStream_t s) {
  return mdot(w, n, V, ld, nvec, x, d_out, s);
}

cudaError_t la_mdot_alloc(LinalgWork& w) {
  if (w.partial) return cudaSuccess;
  cudaError_t e = cudaMalloc((void**)&w.partial, sizeof(double) * (64 * kMdotBlocks + 1));
  if (e != cudaSuccess) {
    w.partial = nullptr;
    return e;
  }
  // the ticket is zero before any stream, also one that does not wait for the legacy one, uses it; without that
  // there are no buffers
  e = cudaMemset(w.ticket(), 0, sizeof(double));
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e != cudaSuccess) {
    cudaFree(w.partial);
    w.partial = nullptr;
  }
  return e;
}

cudaError_t la_maxpy(long long n, const double* V, long long ld, int nvec, const double* d_h, double sign, double* w,
                     cudaStream_t s) {
  maxpy_kernel<double><<<grid_for(n), 256, 0, s>>>(n, V, ld, nvec, d_h, sign, w);
  return cudaGetLastError();
}

cudaError_t la_maxpy32(long long n, const float* V, long long ld, int nvec, const double* d_h, double sign, double* w,
                       cudaStream_t s) {
  maxpy_kernel<float><<<grid_for(n), 256, 0, s>>>(n, V, ld, nvec, d_h, sign, w);
  return cudaGetLastError();
}

// matrix-free products: slot = {|v|^2, c}, h = c / |v| (c when v = 0)
__device__ inline double fd_step(const double* slot) {
  const double v2 = slot[0];
  return v2 > 0.0 ? slot[1] / sqrt(v2) : slot[1];
}

__global__ void fd_perturb_kernel(long long n, const double* __restrict__ u, const double* __restrict__ v,
                                  const double* __restrict__ slot, double* __restrict__ up) {
  const double h = fd_step(slot);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    up[i] = u[i] + h * v[i];
}

__global__ void fd_diff_kernel(long long n, const double* __restrict__ rp, const double* __restrict__ r0,
                               const double* __restrict__ slot, double* __restrict__ y) {
  const double h = fd_step(slot);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = (rp[i] - r0[i]) / h;
}

cudaError_t la_fd_perturb(long long n, const double* u, const double* v, const double* slot, double* up,
                          cudaStream_t s) {
  fd_perturb_kernel<<<grid_for(n), 256, 0, s>>>(n, u, v, slot, up);
  return cudaGetLastError();
}

cudaError_t la_fd_diff(long long n, const double* rp, const double* r0, const double* slot, double* y,
                       cudaStream_t s) {
  fd_diff_kernel<<<grid_for(n), 256, 0, s>>>(n, rp, r0, slot, y);
  return cudaGetLastError();
}

__global__ void scale_kernel(long long n, double a, const double* __restrict__ x, double* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = a * x[i];
}

cudaError_t la_scale(long long n, double a, const double* x, double* y, cudaStream_t s) {
  scale_kernel<<<grid_for(n), 256, 0, s>>>(n, a, x, y);
  return cudaGetLastError();
}

cudaError_t la_axpby(long long n, double a, const double* x, double b, double* y, cudaStream_t s) {
  axpby_kernel<<<grid_for(n), 256, 0, s>>>(n, a, x, b, y);
  return cudaGetLastError();
}

cudaError_t la_xpay(long long n, const double* x, double a, const double* y, double* z, cudaStream_t s) {
  xpay_kernel<<<grid_for(n), 256, 0, s>>>(n, x, a, y, z);
  return cudaGetLastError();
}

template <class K>
static cudaError_t smem_attr(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t la_block_invert(int nblk, int bs, const double* src, const int* blk_index, double* dst, int* flag,
                            cudaStream_t s) {
#define ICX_INV_CASE(B)                                                                        \
  if (bs == B) {                                                                               \
    cudaError_t e = smem_attr(block_invert_kernel<B>, InvSmem<B>::BYTES);                      \
    if (e != cudaSuccess) return e;                                                            \
    block_invert_kernel<B><<<nblk, 256, InvSmem<B>::BYTES, s>>>(nblk, src, blk_index, dst, flag); \
    return cudaGetLastError();                                                                 \
  }
  ICX_BLOCK_SIZES(ICX_INV_CASE)
#undef ICX_INV_CASE
  return cudaErrorInvalidValue;
}

template <class TA>
static cudaError_t tri_rows_t(const DeviceMesh& dm, bool lower, const TA* A, const double* v, const double* x0,
                              double sign, double* y, cudaStream_t s) {
  const int bs = dm.nb * dm.neq;
  RowSet rs{0, 0, -1, dm.E};
#define ICX_TRI_CASE(B)                                                                                          \
  if (bs == B)                                                                                                   \
    return lower ? launch_block_rows<B, BR_LOWER, TA>(rs, dm.bsr_rowptr, dm.bsr_colidx, A, v, x0, sign, y, s)    \
                 : launch_block_rows<B, BR_UPPER, TA>(rs, dm.bsr_rowptr, dm.bsr_colidx, A, v, x0, sign, y, s);
  ICX_BLOCK_SIZES(ICX_TRI_CASE)
#undef ICX_TRI_CASE
  return cudaErrorInvalidValue;
}

cudaError_t la_tri_rows(const DeviceMesh& dm, bool lower, const double* A, const double* v, const double* x0,
                        double sign, double* y, cudaStream_t s) {
  return tri_rows_t<double>(dm, lower, A, v, x0, sign, y, s);
}
cudaError_t la_tri_rows_f32(const DeviceMesh& dm, bool lower, const float* A, const double* v, const double* x0,
                            double sign, double* y, cudaStream_t s) {
  return tri_rows_t<float>(dm, lower, A, v, x0, sign, y, s);
}

cudaError_t la_block_diag_apply(int E, int bs, const double* D, const double* x, double* y, cudaStream_t s) {
  RowSet rs{0, 0, -1, E};
#define ICX_DIAG_CASE(B) \
  if (bs == B) return launch_block_rows<B, BR_DIAG>(rs, nullptr, nullptr, D, x, nullptr, 1.0, y, s);
  ICX_BLOCK_SIZES(ICX_DIAG_CASE)
#undef ICX_DIAG_CASE
  return cudaErrorInvalidValue;
}


cudaError_t la_ilu_factor(const DeviceMesh& dm, const int* order, const std::vector<int>& lvl_off, double* LU,
                          double* Uinv, int* flag, cudaStream_t s) {
  const int bs = dm.nb * dm.neq;
#define ICX_ILUF_CASE(B)                                                                               \
  if (bs == B) {                                                                                       \
    cudaError_t e = smem_attr(ilu_level_kernel<B>, FacCfg<B>::SMEM);                                   \
    if (e == cudaSuccess) e = smem_attr(ilu_scale_upper_kernel<B>, ScaleCfg<B>::SMEM);                 \
    if (e != cudaSuccess) return e;                                                                    \
    for (size_t l = 0; l + 1 < lvl_off.size(); ++l) {                                                  \
      const int cnt = lvl_off[l + 1] - lvl_off[l];                                                     \
      if (cnt > 0)                                                                                     \
        ilu_level_kernel<B><<<cnt, FacCfg<B>::THREADS, FacCfg<B>::SMEM, s>>>(                          \
            dm.E, dm.nnzb, order + lvl_off[l], dm.bsr_rowptr, dm.bsr_colidx, LU, Uinv, flag);          \
    }                                                                                                  \
    ilu_scale_upper_kernel<B><<<dm.E, ScaleCfg<B>::THREADS, ScaleCfg<B>::SMEM, s>>>(                   \
        dm.E, dm.bsr_rowptr, dm.bsr_colidx, LU, Uinv);                                                 \
    return cudaGetLastError();                                                                         \
  }
  ICX_BLOCK_SIZES(ICX_ILUF_CASE)
#undef ICX_ILUF_CASE
  return cudaErrorInvalidValue;
}

// rows per task compiled for a block size: at most the block size, and the
// three blocks' rows a task holds (R x column chunks each) at most 24 values
// per lane, which keeps them in registers

template <int B, int R, class TA>
static const void* flow_kernel_if_fit(bool sen) {
  if constexpr (flow_rows_fit(B, (B + 31) / 32, R))
    return sen ? (const void*)ilu_apply_flow_kernel<B, R, TA, true> : (const void*)ilu_apply_flow_kernel<B, R, TA, false>;
  else return nullptr;
}

// the data-flow kernel for `rows` rows per task (0: the default) on the
// counter or the sentinel schedule, or null
template <int B, class TA>
static const void* flow_kernel_for(int rows, bool sen) {
  static_assert(kFlowRows[0] == 2 && kFlowRows[1] == 4 && kFlowRows[2] == 6 && kFlowRows[3] == 8, "tiles");
  switch (rows ? rows : FlowCfg<B>::R_DEFAULT) {
    case 2: return flow_kernel_if_fit<B, 2, TA>(sen);
    case 4: return flow_kernel_if_fit<B, 4, TA>(sen);
    case 6: return flow_kernel_if_fit<B, 6, TA>(sen);
    case 8: return flow_kernel_if_fit<B, 8, TA>(sen);
    default: return nullptr;
  }
}

__global__ void flow_fill_kernel(long long n, double* __restrict__ f, double* __restrict__ y) {
  const double v = __longlong_as_double((long long)FLOW_SENTINEL);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    f[i] = v;
    y[i] = v;
  }
}

template <class TA>
static cudaError_t ilu_apply_flow_t(const DeviceMesh& dm, const int* order, const TA* LU,
                                   const TA* Uinv, const double* x, double* y, double* f, unsigned* cnt_f,
                                   unsigned* cnt_b, unsigned epoch, int* err, cudaStream_t s) {
  const int bs = dm.nb * dm.neq;
  int dev = 0, nsm = 0, coop = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (e != cudaSuccess) return e;
  if (!coop) return cudaErrorNotSupported;
  IluFlowArgs<TA> args{dm.E, dm.nnzb, dm.bsr_rowptr, dm.bsr_colidx, dm.bsr_diag, order, LU, Uinv, x, f, y, cnt_f,
                       cnt_b, epoch, err};
  const int pi = sizeof(TA) == 8 ? 0 : 1;
  const int rows = dm.tile.flow_rows[pi], ctas = dm.tile.flow_ctas[pi];
  if (ctas < 0) return cudaErrorInvalidValue;
  const bool sen = flow_sentinel(dm.tile, pi);
  const void* kern = nullptr;
#define ICX_ILUF2_CASE(B)                                                                  \
  if (bs == B) kern = flow_kernel_for<B, TA>(rows, sen);
  ICX_BLOCK_SIZES(ICX_ILUF2_CASE)
#undef ICX_ILUF2_CASE
  if (!kern) return cudaErrorInvalidValue;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorNotSupported;
  // the whole grid is resident (the tasks wait on one another): at most the
  // occupancy limit per SM; two by default
  const int want = ctas ? ctas : 2;
  const int grid = nsm * (per_sm < want ? per_sm : want);
  if (sen) {
    const long long n = (long long)dm.E * bs;
    flow_fill_kernel<<<grid_for(n), 256, 0, s>>>(n, f, y);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  void* params[] = {&args};
  return cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(256), params, 0, s);
}

int flow_rows_default(int bs) {
#define ICX_FLOWR_CASE(B) \
  if (bs == B) return FlowCfg<B>::R_DEFAULT;
  ICX_BLOCK_SIZES(ICX_FLOWR_CASE)
#undef ICX_FLOWR_CASE
  return 0;
}

bool flow_rows_compiled(int bs, int rows) {
  if (rows == 0) return true;
  const int ns = (bs + 31) / 32;
  for (int r : kFlowRows)
    if (r == rows) return flow_rows_fit(bs, ns, r);
  return false;
}

template <class TA>
static cudaError_t ilu_apply_rows_t(const DeviceMesh& dm, int nx, int ny, const TA* LU, const TA* Uinv,
                                   const double* x, double* y, double* f, unsigned* cnt_f, unsigned* cnt_b,
                                   unsigned epoch, int* err, cudaStream_t s) {
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (nx < 1 || ny < 1 || nx * ny != dm.E) return cudaErrorInvalidValue;
  const int bs = dm.nb * dm.neq;
  IluRowArgs<TA> a{nx, ny, dm.nnzb, dm.bsr_rowptr, dm.bsr_colidx, dm.bsr_diag, LU, Uinv, x, f, y, cnt_f, cnt_b,
                   epoch, err};
  void* params[] = {&a};
#define ICX_ROWS_CASE(B)                                                                              \
  if (bs == B) {                                                                                      \
    using K = IluRowCfg<B, TA>;                                                                       \
    if ((e = smem_attr(ilu_apply_rows_kernel<B, TA>, K::SMEM)) != cudaSuccess) return e;              \
    int per_sm = 0;                                                                                   \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ilu_apply_rows_kernel<B, TA>, 128, K::SMEM); \
    if (e != cudaSuccess) return e;                                                                   \
    if ((long long)per_sm * nsm < ny) return cudaErrorNotSupported;                                   \
    return cudaLaunchCooperativeKernel((const void*)ilu_apply_rows_kernel<B, TA>, dim3(ny), dim3(128), params, \
                                       K::SMEM, s);                                                   \
  }
  ICX_ROWS_CASE(4) ICX_ROWS_CASE(9) ICX_ROWS_CASE(16) ICX_ROWS_CASE(25) ICX_ROWS_CASE(36) ICX_ROWS_CASE(64)
#undef ICX_ROWS_CASE
  return cudaErrorNotSupported;
}

cudaError_t la_ilu_apply_rows(const DeviceMesh& dm, int nx, int ny, const double* LU, const double* Uinv,
                              const double* x, double* y, double* f, unsigned* cnt_f, unsigned* cnt_b, unsigned epoch,
                              int* err, cudaStream_t s) {
  return ilu_apply_rows_t<double>(dm, nx, ny, LU, Uinv, x, y, f, cnt_f, cnt_b, epoch, err, s);
}

cudaError_t la_ilu_apply_rows_f32(const DeviceMesh& dm, int nx, int ny, const float* LU, const float* Uinv,
                                  const double* x, double* y, double* f, unsigned* cnt_f, unsigned* cnt_b,
                                  unsigned epoch, int* err, cudaStream_t s) {
  return ilu_apply_rows_t<float>(dm, nx, ny, LU, Uinv, x, y, f, cnt_f, cnt_b, epoch, err, s);
}

cudaError_t la_ilu_apply_flow(const DeviceMesh& dm, const int* order, const double* LU, const double* Uinv,
                              const double* x, double* y, double* f, unsigned* cnt_f, unsigned* cnt_b, unsigned epoch,
                              int* err, cudaStream_t s) {
  return ilu_apply_flow_t<double>(dm, order, LU, Uinv, x, y, f, cnt_f, cnt_b, epoch, err, s);
}

cudaError_t la_ilu_apply_flow_f32(const DeviceMesh& dm, const int* order, const float* LU, const float* Uinv,
                                  const double* x, double* y, double* f, unsigned* cnt_f, unsigned* cnt_b,
                                  unsigned epoch, int* err, cudaStream_t s) {
  return ilu_apply_flow_t<float>(dm, order, LU, Uinv, x, y, f, cnt_f, cnt_b, epoch, err, s);
}

cudaError_t la_block_diag_correct_f32(int E, int bs, const float* D, const double* y, double* z, cudaStream_t s) {
  RowSet rs{0, 0, -1, E};
#define ICX_CORR_CASE(B) \
  if (bs == B) return launch_block_rows<B, BR_DIAG, float>(rs, nullptr, nullptr, D, y, y, 1.0, z, s);
  ICX_BLOCK_SIZES(ICX_CORR_CASE)
#undef ICX_CORR_CASE
  return cudaErrorInvalidValue;
}

__global__ void dot_to_kernel(long long n, const double* __restrict__ x, const double* __restrict__ y,
                              double* __restrict__ out) {
  __shared__ double red[256];
  double s = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    s += x[i] * y[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(out, red[0]);
}

cudaError_t la_dot_to(long long n, const double* x, const double* y, double* d_out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(double), s);
  if (e != cudaSuccess) return e;
  dot_to_kernel<<<592, 256, 0, s>>>(n, x, y, d_out);
  return cudaGetLastError();
}

cudaError_t la_block_diag_apply_f32(int E, int bs, const float* D, const double* x, double* y, cudaStream_t s) {
  RowSet rs{0, 0, -1, E};
#define ICX_DIAG32_CASE(B) \
  if (bs == B) return launch_block_rows<B, BR_DIAG, float>(rs, nullptr, nullptr, D, x, nullptr, 1.0, y, s);
  ICX_BLOCK_SIZES(ICX_DIAG32_CASE)
#undef ICX_DIAG32_CASE
  return cudaErrorInvalidValue;
}

__global__ void d2f_kernel(long long n, const double* __restrict__ x, float* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = (float)x[i];
}

cudaError_t la_d2f(long long n, const double* x, float* y, cudaStream_t s) {
  d2f_kernel<<<grid_for(n), 256, 0, s>>>(n, x, y);
  return cudaGetLastError();
}

__global__ void d2bf_kernel(long long n, const double* __restrict__ x, __nv_bfloat16* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = __double2bfloat16(x[i]);
}

cudaError_t la_d2bf(long long n, const double* x, __nv_bfloat16* y, cudaStream_t s) {
  d2bf_kernel<<<grid_for(n), 256, 0, s>>>(n, x, y);
  return cudaGetLastError();
}

__global__ void f2d_kernel(long long n, const float* __restrict__ x, double* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = (double)x[i];
}

cudaError_t la_f2d(long long n, const float* x, double* y, cudaStream_t s) {
  f2d_kernel<<<grid_for(n), 256, 0, s>>>(n, x, y);
  return cudaGetLastError();
}

// dst block b = src block map[b]; each CTA copies whole blocks with 16-byte
// vector loads (a block of bs x bs doubles starts on a 16-byte boundary when
// bs * bs is even; odd sizes fall back to 8-byte copies)
__global__ void gather_blocks_kernel(int nblk, int bs2, const double* __restrict__ src, const int* __restrict__ map,
                                     double* __restrict__ dst) {
  for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
    const double* s = src + (size_t)map[b] * bs2;
    double* d = dst + (size_t)b * bs2;
    if ((bs2 & 1) == 0) {
      const double2* s2 = reinterpret_cast<const double2*>(s);
      double2* d2 = reinterpret_cast<double2*>(d);
      for (int t = threadIdx.x; t < bs2 / 2; t += blockDim.x) d2[t] = __ldcs(s2 + t);
    } else {
      for (int t = threadIdx.x; t < bs2; t += blockDim.x) d[t] = __ldcs(s + t);
    }
  }
}

cudaError_t la_gather_blocks(int nblk, int bs, const double* src, const int* map, double* dst, cudaStream_t s) {
  if (nblk <= 0) return cudaSuccess;
  const int grid = nblk < 148 * 16 ? nblk : 148 * 16;
  gather_blocks_kernel<<<grid, 256, 0, s>>>(nblk, bs * bs, src, map, dst);
  return cudaGetLastError();
}

}  // namespace icx

// ------------------------------------------------------------------ GMRES
namespace icx {

double la_norm(LinalgWork& lw, long long n, const double* x, double* d_scratch, cudaStream_t s) {
  // a failed launch or copy gives NaN: callers treat a non-finite norm as an error
  if (la_mdot(lw, n, x, 0, 1, x, d_scratch, s) != cudaSuccess) return NAN;
  double h = 0.0;
  if (cudaMemcpyAsync(&h, d_scratch, sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess) return NAN;
  if (cudaStreamSynchronize(s) != cudaSuccess) return NAN;
  return std::sqrt(h);
}

#define GCK(expr)                                                  \
  do {                                                             \
    cudaError_t _e = (expr);                                       \
    if (_e != cudaSuccess) {                                       \
      if (err) *err = std::string(#expr) + ": " + cudaGetErrorString(_e); \
      return ICX_ERR_CUDA;                                         \
    }                                                              \
  } while (0)

void ArnoldiGraphs::reset() {
  for (cudaGraphExec_t& g : exec)
    if (g) cudaGraphExecDestroy(g), g = nullptr;
  std::fill(seen.begin(), seen.end(), 0);
  failed = false;
}

void ArnoldiGraphs::release() {
  reset();
  exec.clear();
  seen.clear();
  if (cap) cudaStreamDestroy(cap), cap = nullptr;
  if (hp) cudaFreeHost(hp), hp = nullptr;
  for (cudaEvent_t& ev : done)
    if (ev) cudaEventDestroy(ev), ev = nullptr;
  key = 0;
  m = 0;
}

// prepares the graph set for operators `key` and restart length m (drops
// graphs of another key); false when it cannot be used
static bool arnoldi_graphs_ready(ArnoldiGraphs& g, unsigned long long key, int m) {
  if (g.m != m) {
    g.release();
    g.m = m;
    g.exec.assign(m, nullptr);
    g.seen.assign(m, 0);
  }
  if (!g.cap && cudaStreamCreateWithFlags(&g.cap, cudaStreamNonBlocking) != cudaSuccess) return false;
  if (!g.hp && cudaMallocHost((void**)&g.hp, sizeof(double) * 6 * (m + 2)) != cudaSuccess) return false;
  for (cudaEvent_t& ev : g.done)
    if (!ev && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return false;
  if (g.key != key) {
    g.reset();
    g.key = key;
  }
  return !g.failed;
}

// the graph of Arnoldi step j: captured on the step's second eager run under
// the current key (the first run has done every one-time setup of the
// kernels it launches), then replayed; it copies its reductions to host
// half j % 2. Null: run the step eagerly.
template <class Step>
static cudaGraphExec_t arnoldi_graph(ArnoldiGraphs& g, int j, long long n, double* vj1, const double* h2, Step& step,
                                     bool append_normalize) {
  if (g.failed) return nullptr;
  if (g.exec[j]) return g.exec[j];
  if (g.seen[j]++ < 1) return nullptr;
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamBeginCapture(g.cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    cudaError_t es = step(g.cap, g.hp + (size_t)(j & 1) * 3 * (g.m + 2));
    if (es == cudaSuccess && append_normalize) {
      normalize_kernel<<<grid_for(n), 256, 0, g.cap>>>(n, h2, vj1);
      es = cudaGetLastError();
    }
    e = cudaStreamEndCapture(g.cap, &graph);
    if (es != cudaSuccess) e = es;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&g.exec[j], graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    // operators that cannot be captured: eager steps from now on under this key
    (void)cudaGetLastError();
    g.exec[j] = nullptr;
    g.failed = true;
    return nullptr;
  }
  return g.exec[j];
}

icx_status gmres_op(KrylovBuffers& kb, const LinOp& A, const LinOp* M, int maxit, double rtol, const double* b,
                    double* x, int* iters, double* relres, cudaStream_t s, std::string* err) {
  long long n = kb.n;
  int m = kb.m;
  if (b == kb.r || b == kb.w || b == kb.z || x == kb.r || x == kb.w || x == kb.z) {
    if (err) *err = "gmres vectors alias its work buffers";
    return ICX_ERR_INVALID;
  }
  GCK(cudaMemsetAsync(x, 0, sizeof(double) * n, s));
  double bnorm = la_norm(*kb.lw, n, b, kb.dh, s);
  *iters = 0;
  *relres = 0.0;
  if (bnorm == 0.0) return ICX_OK;
  if (!std::isfinite(bnorm)) {
    if (err) *err = "non-finite right-hand side";
    return ICX_ERR_NONFINITE;
  }
  double tol = rtol * bnorm;
  std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), g(m + 1), y(m), hcol(m + 2), hp3(3 * (m + 2));
  kb.graph_launches = 0;
  bool use_graphs = kb.graphs && kb.graph_key != 0 && !kb.samples;
  if (use_graphs && !arnoldi_graphs_ready(*kb.graphs, kb.graph_key, m)) use_graphs = false;
  GCK(cudaMemcpyAsync(kb.r, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  double beta = bnorm;
  int total = 0;
  std::vector<double> cycle_beta{bnorm};
  // FP32 basis: v_j is widened into vt for the operators, w = A M^-1 v_j is
  // formed in kb.w (FP64) and stored rounded into the basis once normalised
  const bool f32 = kb.V32 != nullptr && kb.vt != nullptr;
  while (true) {
    if (f32) {
      scale_to_f32_kernel<<<grid_for(n), 256, 0, s>>>(n, 1.0 / beta, kb.r, kb.V32);
      GCK(cudaGetLastError());
    } else {
      // v_0 = r / beta, written without reading the basis (a fresh
      // allocation may hold NaN bit patterns, and 0 * NaN is NaN)
      GCK(la_scale(n, 1.0 / beta, kb.r, kb.V, s));
    }
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int j = 0;
    double resid = beta;
    // replayed steps run one ahead: step j + 1 (whose inputs the device
    // forms: v_j+1 is normalised inside step j's graph) is launched before
    // the host waits for step j, so the host's rotations overlap it; a step
    // launched past convergence only writes scratch the solve overwrites
    bool ahead = false;
    for (; j < m && total < maxit; ++j) {
      double* vj = f32 ? kb.vt : kb.V + (size_t)j * n;
      double* vj1 = f32 ? kb.w : kb.V + (size_t)(j + 1) * n;
      const float* vj32 = f32 ? kb.V32 + (size_t)j * n : nullptr;
      float* vj1_32 = f32 ? kb.V32 + (size_t)(j + 1) * n : nullptr;
      if (kb.samples && kb.sample_every > 0 && kb.sample_count < kb.sample_cap && j > 0 &&
          total % kb.sample_every == 0) {
        double* dst = kb.samples + (size_t)kb.sample_count++ * n;
        if (f32) GCK(la_f2d(n, vj32, dst, s));
        else GCK(cudaMemcpyAsync(dst, vj, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
      }
      // the step: preconditioner and operator, classical Gram-Schmidt twice
      // (once with cgs_passes = 1) and the norm of the result; the
      // reductions land in separate device slots [pass 1 | pass 2 | |v|^2]
      // and come back in one copy
      auto step = [&](cudaStream_t st, double* host_dst) -> cudaError_t {
        cudaError_t e = f32 ? la_f2d(n, vj32, vj, st) : cudaSuccess;
        if (e == cudaSuccess && M) e = (*M)(vj, kb.z, st);
        if (e == cudaSuccess) e = A(M ? kb.z : vj, vj1, st);
        const int passes = kb.cgs_passes == 1 ? 1 : 2;
        for (int pass = 0; pass < passes && e == cudaSuccess; ++pass) {
          double* slot = kb.dh + (size_t)pass * (m + 2);
          e = f32 ? la_mdot32(*kb.lw, n, kb.V32, n, j + 1, vj1, slot, st)
                  : la_mdot(*kb.lw, n, kb.V, n, j + 1, vj1, slot, st);
          if (e == cudaSuccess)
            e = f32 ? la_maxpy32(n, kb.V32, n, j + 1, slot, -1.0, vj1, st)
                    : la_maxpy(n, kb.V, n, j + 1, slot, -1.0, vj1, st);
        }
        if (e == cudaSuccess) e = la_mdot(*kb.lw, n, vj1, 0, 1, vj1, kb.dh + 2 * (m + 2), st);
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(host_dst, kb.dh, sizeof(double) * 3 * (m + 2), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && f32) {
          normalize_to_f32_kernel<<<grid_for(n), 256, 0, st>>>(n, kb.dh + 2 * (m + 2), vj1, vj1_32);
          e = cudaGetLastError();
        }
        return e;
      };
      // replayed from a CUDA graph (which also normalises v_j+1 on the
      // device), or launched one by one
      cudaGraphExec_t gx =
          use_graphs ? arnoldi_graph(*kb.graphs, j, n, vj1, kb.dh + 2 * (m + 2), step, !f32) : nullptr;
      if (gx) {
        ArnoldiGraphs& ag = *kb.graphs;
        if (!ahead) {
          GCK(cudaGraphLaunch(gx, s));
          GCK(cudaEventRecord(ag.done[j & 1], s));
          ++kb.graph_launches;
        }
        ahead = false;
        if (j + 1 < m && total + 1 < maxit && ag.exec[j + 1]) {
          GCK(cudaGraphLaunch(ag.exec[j + 1], s));
          GCK(cudaEventRecord(ag.done[(j + 1) & 1], s));
          ++kb.graph_launches;
          ahead = true;
        }
        GCK(cudaEventSynchronize(ag.done[j & 1]));
        const double* hj = ag.hp + (size_t)(j & 1) * 3 * (m + 2);
        std::copy(hj, hj + 3 * (m + 2), hp3.begin());
      } else {
        GCK(step(s, hp3.data()));
        GCK(cudaStreamSynchronize(s));
      }
      std::fill(hcol.begin(), hcol.end(), 0.0);
      for (int i = 0; i <= j; ++i) hcol[i] += hp3[i] + (kb.cgs_passes == 1 ? 0.0 : hp3[(m + 2) + i]);
      double hn = std::sqrt(hp3[2 * (m + 2)]);
      hcol[j + 1] = hn;
      if (!std::isfinite(hn)) {
        if (err) *err = "non-finite Krylov vector";
        return ICX_ERR_NONFINITE;
      }
      if (!gx && !f32 && hn > 0.0) GCK(la_axpby(n, 1.0 / hn, vj1, 0.0, vj1, s));
      for (int i = 0; i < j; ++i) {
        double t = cs[i] * hcol[i] + sn[i] * hcol[i + 1];
        hcol[i + 1] = -sn[i] * hcol[i] + cs[i] * hcol[i + 1];
        hcol[i] = t;
      }
      double den = std::hypot(hcol[j], hcol[j + 1]);
      cs[j] = den == 0.0 ? 1.0 : hcol[j] / den;
      sn[j] = den == 0.0 ? 0.0 : hcol[j + 1] / den;
      hcol[j] = den;
      hcol[j + 1] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      for (int i = 0; i <= j; ++i) H[(size_t)i * m + j] = hcol[i];
      ++total;
      resid = std::fabs(g[j + 1]);
      if (resid <= tol || hn == 0.0) { ++j; break; }
    }
    for (int i = j - 1; i >= 0; --i) {
      double sacc = g[i];
      for (int k = i + 1; k < j; ++k) sacc -= H[(size_t)i * m + k] * y[k];
      y[i] = sacc / H[(size_t)i * m + i];
    }
    GCK(cudaMemcpyAsync(kb.dh, y.data(), sizeof(double) * j, cudaMemcpyHostToDevice, s));
    GCK(cudaMemsetAsync(kb.w, 0, sizeof(double) * n, s));
    if (f32) GCK(la_maxpy32(n, kb.V32, n, j, kb.dh, 1.0, kb.w, s));
    else GCK(la_maxpy(n, kb.V, n, j, kb.dh, 1.0, kb.w, s));
    if (M) {
      GCK((*M)(kb.w, kb.z, s));
      GCK(la_axpby(n, 1.0, kb.z, 1.0, x, s));
    } else {
      GCK(la_axpby(n, 1.0, kb.w, 1.0, x, s));
    }
    GCK(A(x, kb.w, s));
    GCK(la_xpay(n, b, -1.0, kb.w, kb.r, s));
    if (kb.samples && kb.sample_count < kb.sample_cap)
      GCK(cudaMemcpyAsync(kb.samples + (size_t)kb.sample_count++ * n, kb.r, sizeof(double) * n,
                          cudaMemcpyDeviceToDevice, s));
    beta = la_norm(*kb.lw, n, kb.r, kb.dh, s);
    *relres = beta / bnorm;
    if (beta <= tol || total >= maxit || resid <= tol) break;
    cycle_beta.push_back(beta);
    const int nc = (int)cycle_beta.size() - 1;
    if (kb.stall_cycles > 0 && nc >= kb.stall_cycles && beta > 0.9 * cycle_beta[nc - kb.stall_cycles]) break;
  }
  *iters = total;
  return ICX_OK;
}

}  // namespace icx
