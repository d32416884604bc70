// Block-ILU(0) apply on element groups (tiles) with the factors streamed
// through shared memory: one CTA per group, a producer warp and NW consumer
// warps.
//
// Bound by the factors' bytes (each block is read once): what has to be hidden
// is the trip to memory of every level. The order in which a group's blocks are
// used is known, so the producer copies them ahead of the levels, one or two
// bulk copies per element (an element's off-diagonal blocks of a sweep are
// adjacent), into a ring of element slots; the consumers never wait for memory
// unless the ring runs dry. A consumer warp takes a whole element: eight rows
// at a time, four lanes to a row, each lane holding its columns of the (up to
// three) vectors the blocks multiply in registers over all rows. x, f and y of
// the group share one vector in shared memory (an element's forward result is
// read by its own warp alone before the backward result takes its place).
//
// The sums (the row kernel's apart) are those of the data-flow apply, value for
// value: 32 partial sums over the columns modulo 32, folded at distance 16, 8,
// 4, 2, 1 (warp_row_sums).
// A lane holds the partial sums (k LPR + g) VEC + i, so distances down to
// LPR VEC fold inside the lane, the next ones across the row's lanes, the last
// ones inside the lane again.
//
// Measured (NS, 8 x 8 tiles, BS = 36; calls on one vector in turn), against the
// forms it replaces:
//                              before      here    factors at 6.45 TB/s
//   FP64   256 x 256            922 us    487 us    474 us
//   FP64   128 x 128            241       136       118
//   FP32   256 x 256            501       278       237
//   FP32   128 x 128            146        72        59
//   BF16   128 x 128 (rows)      95        47        30
// (FP64 256 x 256 with other inputs from call to call 924 and 515.)
// Below some 148 tiles the levels' own latency is left (32 x 32: 54, 41 and 33 us
// for 30 levels; 177, 54 and 58 before).
//
// Every wait ends: the producer fills slots in the order of use and waits only
// for a slot's previous element, whose warp waits for no later element. The
// waits are bounded all the same (ICX_FLOW_SPINS): *err = 1, and a warp that
// gave up goes on through the same barriers without computing and gives no
// slot back, so nothing is filled under another's feet; y of its group is NaN
// then, never what it held before. The producer leaves only after its last
// copies have landed.
#include <cuda_runtime.h>

#include <algorithm>

#include "icx_bulk.cuh"
#include "icx_internal.h"
#include "icx_linalg.h"

namespace icx {

namespace {

template <int BS, class TS>
struct TileCfg {
  using TC = typename ComputeOf<TS>::type;
  static constexpr int LPR = 4;                                      // lanes per row
  static constexpr int LB = group_rows_load_bytes<BS, TS>();         // bytes per load of a factor row
  static constexpr int VEC = LB / (int)sizeof(TS);
  static constexpr int NV = BS / VEC;                                // vectors per row
  static constexpr int XV = VEC * (int)sizeof(TC) > 16 ? 16 / (int)sizeof(TC) : VEC;  // vector values per load
  static constexpr int KPL = (NV + LPR - 1) / LPR;                   // vectors per lane and row
  static constexpr int KN = 32 / (LPR * VEC);                        // partial sums per lane: KN VEC
  static constexpr int NP = (BS + 7) / 8;                            // passes of 8 rows
  static constexpr int BB = BS * BS * (int)sizeof(TS);               // bytes per block
  static constexpr int SLOT = 3 * BB;
  static constexpr bool ALIGNED = BB % 16 == 0;                      // bulk copies move 16-byte units
  // rows that a load's phase holds together lie ROWD apart, so that they fall
  // into different banks (stride of a row: STRIDE words)
  static constexpr int STRIDE = BS * (int)sizeof(TS) / 4;
  static constexpr int ROWD = STRIDE % 32 == 16 ? 1 : (2 * STRIDE) % 32 == 16 ? 2 : 4;
  __device__ static int row_of(int q) {
    return ROWD == 1 ? q : ROWD == 2 ? ((q & 1) << 1 | (q >> 1 & 1) | (q & 4)) : ((q & 1) << 2 | q >> 1);
  }
};

// the row kernel runs BF16 factors of these sizes
template <int BS, class TS>
constexpr bool tile_by_rows() { return sizeof(TS) == 2 && TileCfg<BS, TS>::STRIDE % 32 == 18; }

// sizes and types that the kernels of this file are ahead at, with three slots that fit: not the 4 x 4 blocks of
// FP32 and BF16, nor the 16 x 16 and 100 x 100 ones of BF16 (128 x 128 elements, 8 x 8 tiles: 27 us here against 24;
// 31 against 28; 300 against 302)
template <int BS, class TS>
constexpr bool tile_ahead() {
  return TileCfg<BS, TS>::ALIGNED && 3 * TileCfg<BS, TS>::SLOT < 227 * 1024 &&
         (sizeof(TS) == 8 || (sizeof(TS) == 4 ? BS >= 16 : BS == 36 || BS == 64));
}

// the group's table (an entry per element and sweep) and its vectors: one for x, f and y, the row kernel two
template <int BS, class TS>
size_t tile_fixed_smem(int gmax) {
  const size_t vectors = tile_by_rows<BS, TS>() ? 2 : 1;
  return (size_t)2 * gmax * sizeof(int4) + (vectors * gmax * BS * sizeof(typename ComputeOf<TS>::type) + 15) / 16 * 16;
}

constexpr int kTileSlotsMax = 16;

template <int BS, class TS>
struct TileLane {
  using K = TileCfg<BS, TS>;
  using TC = typename K::TC;
  TC v[K::KPL][K::VEC];
  // this lane's columns of the vector xs[BS]; columns beyond the row are zero
  __device__ inline void load(const TC* xs, int g) {
#pragma unroll
    for (int k = 0; k < K::KPL; ++k) {
      const int j = k * K::LPR + g;
#pragma unroll
      for (int i = 0; i < K::VEC; i += K::XV) {
        using V = typename RawLoad<K::XV * (int)sizeof(TC)>::type;
        V raw = V();
        if ((k + 1) * K::LPR <= K::NV || j < K::NV) raw = *reinterpret_cast<const V*>(xs + j * K::VEC + i);
        const TC* xv = reinterpret_cast<const TC*>(&raw);
#pragma unroll
        for (int t = 0; t < K::XV; ++t) v[k][i + t] = xv[t];
      }
    }
  }
  template <bool NEG>
  __device__ inline void madd(const TS* arow, int g, TC (&acc)[K::KN][K::VEC]) const {
    using V = typename RawLoad<K::LB>::type;
#pragma unroll
    for (int k = 0; k < K::KPL; ++k) {
      const int j = k * K::LPR + g;
      V raw = V();
      if ((k + 1) * K::LPR <= K::NV || j < K::NV) raw = reinterpret_cast<const V*>(arow)[j];
      const TS* av = reinterpret_cast<const TS*>(&raw);
#pragma unroll
      for (int i = 0; i < K::VEC; ++i) {
        const TC aw = widen(av[i]);
        acc[k % K::KN][i] = fused_madd(NEG ? -aw : aw, v[k][i], acc[k % K::KN][i]);
      }
    }
  }
};

// the row's sum, on each of its lanes
template <int BS, class TS>
__device__ inline typename ComputeOf<TS>::type tile_row_sum(
    typename ComputeOf<TS>::type (&acc)[TileCfg<BS, TS>::KN][TileCfg<BS, TS>::VEC]) {
  using K = TileCfg<BS, TS>;
#pragma unroll
  for (int h = K::KN / 2; h >= 1; h /= 2)
#pragma unroll
    for (int k = 0; k < h; ++k)
#pragma unroll
      for (int i = 0; i < K::VEC; ++i) acc[k][i] += acc[k + h][i];
#pragma unroll
  for (int d = K::LPR / 2; d >= 1; d /= 2)
#pragma unroll
    for (int i = 0; i < K::VEC; ++i) acc[0][i] += __shfl_xor_sync(0xffffffffu, acc[0][i], d);
#pragma unroll
  for (int h = K::VEC / 2; h >= 1; h /= 2)
#pragma unroll
    for (int i = 0; i < h; ++i) acc[0][i] += acc[0][i + h];
  return acc[0][0];
}

// row sums of an element: NBK off-diagonal blocks at A (subtracted), then with
// DIAG the inverse of the diagonal one (added). The passes have no branch and
// no store between them, so their loads and folds overlap
template <int BS, class TS, int NBK, bool DIAG>
__device__ inline void tile_rows(const TS* A, const typename ComputeOf<TS>::type* v0,
                                 const typename ComputeOf<TS>::type* v1, const typename ComputeOf<TS>::type* vd, int g,
                                 int rq, typename ComputeOf<TS>::type (&sum)[TileCfg<BS, TS>::NP]) {
  using K = TileCfg<BS, TS>;
  TileLane<BS, TS> x0, x1, xd;
  if constexpr (NBK > 0) x0.load(v0, g);
  if constexpr (NBK > 1) x1.load(v1, g);
  if constexpr (DIAG) xd.load(vd, g);
#pragma unroll
  for (int s = 0; s < K::NP; ++s) {
    const int r = 8 * s + rq, rr = r < BS ? r : BS - 1;
    typename K::TC acc[K::KN][K::VEC] = {};
    if constexpr (NBK > 0) x0.template madd<true>(A + (size_t)rr * BS, g, acc);
    if constexpr (NBK > 1) x1.template madd<true>(A + (size_t)(BS + rr) * BS, g, acc);
    if constexpr (DIAG) xd.template madd<false>(A + (size_t)(NBK * BS + rr) * BS, g, acc);
    sum[s] = tile_row_sum<BS, TS>(acc);
  }
}

// a CTA's view of its group
template <class TS>
struct TileCta {
  int G, nlev;               // elements, levels
  unsigned char* ring;
  const int4* tab;
  typename ComputeOf<TS>::type* vec;  // [gmax][BS], VECS times
  unsigned full, empty;      // barriers of the slots
};
struct TileShared {
  int slev[kGroupLevelsSmem + 1];
  int held[kTileSlotsMax];  // the element of the order of use that a slot is being filled with
  int gave_up;              // a wait ran out
  unsigned long long bars[2 * kTileSlotsMax];
};

// table and barriers of the group; false (uniform over the CTA): a plan out of its bounds
template <int BS, class TS>
__device__ inline bool tile_setup(const IluGroupArgs<TS>& a, int nslot, TileShared& sh, unsigned char* dsm,
                                  TileCta<TS>& c) {
  using K = TileCfg<BS, TS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gid = blockIdx.x, gm = a.plan.gmax;
  const int l0 = a.plan.glev_ptr[gid], l1 = a.plan.glev_ptr[gid + 1];
  const int nlev = l1 - l0 - 1;
  const int pg0 = a.plan.glev[l0], G = a.plan.glev[l1 - 1] - pg0;
  if (nlev > kGroupLevelsSmem || G > gm || G < 0) {
    if (threadIdx.x == 0) atomicExch(a.err, 2);
    return false;
  }
  // per element in the order of use (the forward positions, then the backward ones from the last down):
  // {element (-1: an index out of range), first block, own position | slot << 16 | parity << 24,
  //  positions + 1 of the neighbours, 0 none}
  int4* tab = reinterpret_cast<int4*>(dsm + (size_t)nslot * K::SLOT);  // [2 gmax]
  c.G = G;
  c.nlev = nlev;
  c.ring = dsm;
  c.tab = tab;
  c.vec = reinterpret_cast<typename K::TC*>(tab + 2 * gm);
  c.full = (unsigned)__cvta_generic_to_shared(sh.bars);
  c.empty = c.full + 8 * kTileSlotsMax;
  for (int i = threadIdx.x; i <= nlev; i += blockDim.x) sh.slev[i] = a.plan.glev[l0 + i] - pg0;
  for (int n = threadIdx.x; n < 2 * G; n += blockDim.x) {
    const size_t at = n < G ? (size_t)pg0 + n : (size_t)a.E + pg0 + (2 * G - 1 - n);
    const int4 inf = a.plan.task[at], loc = a.plan.loc[at];
    const int nbk = (inf.z >= 0) + (inf.w >= 0);
    const bool good = group_task_ok<BS, 1, TS>(a, inf) && loc.x >= 0 && loc.x < G && loc.y < G && loc.z < G &&
                      (nbk < 1 || loc.y >= 0) && (nbk < 2 || loc.z >= 0);
    if (!good) atomicExch(a.err, 2);
    tab[n] = make_int4(good ? inf.x : -1, inf.y, (loc.x & 0xffff) | n % nslot << 16 | (n / nslot & 1) << 24,
                       (nbk > 0 ? loc.y + 1 : 0) | (nbk > 1 ? loc.z + 1 : 0) << 16);
  }
  // x on its way into L2: the forward sweep then reads it from there, a task ahead
  for (int i = warp; i < G; i += blockDim.x / 32) {
    const int e = a.plan.task[pg0 + i].x;
    if (e >= 0 && e < a.E)
      for (int k = lane * 16; k < BS; k += 512)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.x + (size_t)e * BS + k));
  }
  if (threadIdx.x == 0) sh.gave_up = 0;
  if (threadIdx.x < nslot) {
    sh.held[threadIdx.x] = -1;
    mbar_init(c.full + 8 * threadIdx.x, 1);
    mbar_init(c.empty + 8 * threadIdx.x, 1);
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  return true;
}

// the producer warp: lane l fills slot l with elements l, l + nslot, ...
template <int BS, class TS>
__device__ inline void tile_produce(const IluGroupArgs<TS>& a, int nslot, TileShared& sh, const TileCta<TS>& c) {
  using K = TileCfg<BS, TS>;
  const int lane = threadIdx.x & 31, N = 2 * c.G;
  int n = lane;
  unsigned phase = 1, spins = 0;  // phase of the slot's empty barrier; its first filling needs no wait
  bool more = lane < nslot && n < N;
  while (__any_sync(0xffffffffu, more)) {
    // every lane asks once and goes on: no lane with a free slot waits for one without
    if (more) {
      if (n < nslot || mbar_test(c.empty + 8 * lane, phase)) {
        const int4 t = c.tab[n];
        const unsigned bar = c.full + 8 * lane;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(c.ring + (size_t)lane * K::SLOT);
        const bool dg = t.x >= 0 && n >= c.G;
        const unsigned nb = t.x >= 0 ? ((t.w & 0xffff ? 1 : 0) + (t.w >> 16 ? 1 : 0)) * K::BB : 0;
        *(volatile int*)(sh.held + lane) = n;
        mbar_expect(bar, nb + (dg ? K::BB : 0));
        if (nb) bulk_copy(dst, a.LU + (size_t)t.y * BS * BS, nb, bar);
        if (dg) bulk_copy(dst + nb, a.Uinv + (size_t)t.x * BS * BS, K::BB, bar);
        n += nslot;
        phase ^= 1;
        spins = 0;
        more = n < N;
      } else if (++spins > ICX_FLOW_SPINS) {
        atomicExch(a.err, 1);
        more = false;
      }
    }
  }
  // the slot's last copies may still be in flight
  n -= nslot;
  if (n >= 0 && lane < nslot) mbar_wait(c.full + 8 * lane, (unsigned)(n / nslot) & 1);
}

// waits until the slot holds element n: a barrier tells only the parity of its phase, so the slot has to be
// this element's before it is asked
__device__ inline bool tile_wait(const TileShared& sh, unsigned full, int slot, int n, unsigned parity) {
  unsigned spins = 0;
  while (*(const volatile int*)(sh.held + slot) != n && ++spins < ICX_FLOW_SPINS) {}
  return spins < ICX_FLOW_SPINS && mbar_wait(full + 8 * slot, parity);
}

// y of a group that was given up, by NT threads after their last barrier
template <int BS, class TS>
__device__ inline void tile_give_up(const IluGroupArgs<TS>& a, const TileCta<TS>& c, int nt) {
  for (int i = threadIdx.x; i < c.G * BS; i += nt) {
    const int e = c.tab[i / BS].x;
    if (e >= 0) a.y[(size_t)e * BS + i % BS] = __longlong_as_double(-1ll);
  }
}

// a warp per element, eight rows at a time
template <int BS, class TS, int NW, int MINB>
__global__ void __launch_bounds__(NW * 32 + 32, MINB) ilu_apply_tile_kernel(IluGroupArgs<TS> a, int nslot) {
  using K = TileCfg<BS, TS>;
  using TC = typename K::TC;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ TileShared sh;
  TileCta<TS> cta;
  if (!tile_setup<BS, TS>(a, nslot, sh, dsm, cta)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == NW) {
    tile_produce<BS, TS>(a, nslot, sh, cta);
    return;
  }
  const int G = cta.G, nlev = cta.nlev;
  const int* slev = sh.slev;
  const int4* tab = cta.tab;
  const unsigned full = cta.full, empty = cta.empty;
  TC* vec = cta.vec;
  const int g = lane & (K::LPR - 1), rq = K::row_of(lane / K::LPR);
  const int nq = 2 * nlev;
  bool ok = true, ready = false;
  // the warp's next task: level step tq (nq: none left), element tk of it, n in the order of use, table entry tn
  int tq = 0, tk = warp, n = 0;
  int4 tn = make_int4(-1, 0, 0, 0);
  double xn[K::NP];  // x of its rows (forward): on its way from L2 while the current task runs
  auto seek = [&]() {
    for (; tq < nq; ++tq, tk = warp) {
      const int lv = tq < nlev ? tq : nq - 1 - tq, b = slev[lv], c = slev[lv + 1];
      if (tk < c - b) {
        n = tq < nlev ? b + tk : 2 * G - c + tk;
        tn = tab[n];
        break;
      }
    }
    if (tq < nlev) {
#pragma unroll
      for (int s = 0; s < K::NP; ++s) {
        const int r = 8 * s + rq;
        if (r < BS && g == 0 && tn.x >= 0) xn[s] = a.x[(size_t)tn.x * BS + r];
      }
    }
  };
  seek();
#pragma unroll 1
  for (int q = 0; q < nq; ++q) {
#pragma unroll 1
    while (tq == q) {
      const int4 t = tn;
      const int m = n, slot = t.z >> 16 & 255;
      double xe[K::NP];
#pragma unroll
      for (int s = 0; s < K::NP; ++s) xe[s] = xn[s];
      tk += NW;
      seek();
      if (!__all_sync(0xffffffffu, ready) && ok) {
        ok = tile_wait(sh, full, slot, m, (unsigned)t.z >> 24);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) {
          atomicExch(a.err, 1);
          sh.gave_up = 1;
        }
      }
      if (ok && t.x >= 0) {
        const TS* A = reinterpret_cast<const TS*>(cta.ring + (size_t)slot * K::SLOT);
        const int k0 = (t.w & 0xffff) - 1, k1 = (int)((unsigned)t.w >> 16) - 1;
        const TC *v0 = vec + (size_t)k0 * BS, *v1 = vec + (size_t)k1 * BS;
        TC* ve = vec + (size_t)(t.z & 0xffff) * BS;
        TC sum[K::NP];
        if (q < nlev) {
          if (k1 >= 0) tile_rows<BS, TS, 2, false>(A, v0, v1, ve, g, rq, sum);
          else if (k0 >= 0) tile_rows<BS, TS, 1, false>(A, v0, v1, ve, g, rq, sum);
          else tile_rows<BS, TS, 0, false>(A, v0, v1, ve, g, rq, sum);
#pragma unroll
          for (int s = 0; s < K::NP; ++s) sum[s] = (TC)(xe[s] + (double)sum[s]);
        } else {
          if (k1 >= 0) tile_rows<BS, TS, 2, true>(A, v0, v1, ve, g, rq, sum);
          else if (k0 >= 0) tile_rows<BS, TS, 1, true>(A, v0, v1, ve, g, rq, sum);
          else tile_rows<BS, TS, 0, true>(A, v0, v1, ve, g, rq, sum);
        }
        __syncwarp();  // f_e is in every lane's registers: y_e takes its place
#pragma unroll
        for (int s = 0; s < K::NP; ++s)
          if (g == 0 && 8 * s + rq < BS) ve[8 * s + rq] = sum[s];
        __syncwarp();
        if (q >= nlev)
          for (int c = lane; c < BS; c += 32) a.y[(size_t)t.x * BS + c] = (double)ve[c];
      }
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(empty + 8 * slot);
      // asked without waiting: another element of its level may have to give its slot back first
      const int sn = tn.z >> 16 & 255;
      ready = tq < nq && *(volatile int*)(sh.held + sn) == n && mbar_test(full + 8 * sn, (unsigned)tn.z >> 24);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
  }
  if (sh.gave_up) tile_give_up<BS, TS>(a, cta, NW * 32);
}

// BF16 factors, rows of half-bank stride (BS = 36): a thread per matrix row,
// the elements of a level side by side over the CTA in chunks of as many as it
// has rows for; the chunk's slots go back after its barrier. What bounds a warp
// per element there is its instructions: widening and the padding of 9 vectors
// over 4 lanes make 800 per element and sweep, against 250 here. A thread's
// 8-byte loads of its own row fall into all banks (the stride is 18 words). A
// row's sums are two pairs of partial sums over the columns modulo 4 (packed
// FP32 arithmetic); this order is not the data-flow apply's.
template <int BS>
struct TileRowCfg {
  static constexpr int C = 288 / BS;  // elements of a chunk
  static constexpr int NT = C * BS;   // row threads, whole warps: eight elements at BS = 36
  static_assert(NT % 32 == 0, "row threads");
};

// c += a b, two FP32 values at once, each rounded once
__device__ inline void madd2(float (&c)[2], float a0, float a1, float b0, float b1) {
  asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%0, %1};\n"
      "fma.rn.f32x2 c, a, b, c;\nmov.b64 {%0, %1}, c;\n}"
      : "+f"(c[0]), "+f"(c[1])
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

template <int BS, class TS>
__device__ inline void tile_row_madd(const TS* arow, const float* xs, float (&acc)[2][2]) {
  using K = TileCfg<BS, TS>;
  using V = typename RawLoad<K::LB>::type;
#pragma unroll
  for (int i = 0; i < K::NV; ++i) {
    const V raw = reinterpret_cast<const V*>(arow)[i];
    const TS* av = reinterpret_cast<const TS*>(&raw);
#pragma unroll
    for (int v = 0; v < K::VEC; v += 4) {
      const float4 x = *reinterpret_cast<const float4*>(xs + i * K::VEC + v);
      madd2(acc[0], widen(av[v]), widen(av[v + 1]), x.x, x.y);
      madd2(acc[1], widen(av[v + 2]), widen(av[v + 3]), x.z, x.w);
    }
  }
}

template <int BS, class TS>
__global__ void __launch_bounds__(TileRowCfg<BS>::NT + 32, 2)
    ilu_apply_tile_rows_kernel(IluGroupArgs<TS> a, int nslot) {
  using K = TileCfg<BS, TS>;
  using R = TileRowCfg<BS>;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ TileShared sh;
  TileCta<TS> cta;
  if (!tile_setup<BS, TS>(a, nslot, sh, dsm, cta)) return;
  if (threadIdx.x >= R::NT) {
    tile_produce<BS, TS>(a, nslot, sh, cta);
    return;
  }
  const int tid = threadIdx.x, G = cta.G, nlev = cta.nlev, nq = 2 * nlev;
  const int* slev = sh.slev;
  const int4* tab = cta.tab;
  float *fs = cta.vec, *ys = fs + (size_t)a.plan.gmax * BS;
  const int C = R::C < nslot ? R::C : nslot;
  const int ei = tid / BS, r = tid - ei * BS;  // this thread's element of a chunk, and its row
  bool ok = true;
  // the next chunk: level step tq, its first element tk, the thread's element n (-1: none) and table entry tn
  int tq = 0, tk = -C, n = -1;
  int4 tn = make_int4(-1, 0, 0, 0);
  double xn = 0.0;
  auto next = [&]() {
    tk += C;
    int b = 0, w = 0;
    for (; tq < nq; ++tq, tk = 0) {
      const int lv = tq < nlev ? tq : nq - 1 - tq;
      b = slev[lv];
      w = slev[lv + 1] - b;
      if (tk < w) break;
    }
    n = -1;
    if (tq < nq && ei < C && tk + ei < w) {
      n = (tq < nlev ? b : 2 * G - b - w) + tk + ei;
      tn = tab[n];
      if (tq < nlev && tn.x >= 0) xn = a.x[(size_t)tn.x * BS + r];
    }
  };
  next();
#pragma unroll 1
  while (tq < nq) {
    const int4 t = tn;
    const int m = n, slot = t.z >> 16 & 255;
    const bool fwd = tq < nlev;
    const double xe = xn;
    next();
    if (m >= 0) {
      if (ok && !tile_wait(sh, cta.full, slot, m, (unsigned)t.z >> 24)) {
        ok = false;
        atomicExch(a.err, 1);
      }
      if (ok && t.x >= 0) {
        const TS* A = reinterpret_cast<const TS*>(cta.ring + (size_t)slot * K::SLOT) + (size_t)r * BS;
        const int k0 = (t.w & 0xffff) - 1, k1 = (int)((unsigned)t.w >> 16) - 1, at = (t.z & 0xffff) * BS;
        const float* vs = fwd ? fs : ys;
        float acc[2][2] = {};
        if (k0 >= 0) {
          tile_row_madd<BS, TS>(A, vs + k0 * BS, acc);
          A += BS * BS;
        }
        if (k1 >= 0) {
          tile_row_madd<BS, TS>(A, vs + k1 * BS, acc);
          A += BS * BS;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int v = 0; v < 2; ++v) acc[i][v] = -acc[i][v];
        if (!fwd) tile_row_madd<BS, TS>(A, fs + at, acc);
        const float sum = (acc[0][0] + acc[1][0]) + (acc[0][1] + acc[1][1]);
        if (fwd) {
          fs[at + r] = (float)(xe + (double)sum);
        } else {
          ys[at + r] = sum;
          a.y[(size_t)t.x * BS + r] = (double)sum;
        }
      }
    }
    // the chunk's rows are done, also those of the other warps: its slots go back, its results are there to read
    {
      int all = ok;
      asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %0, 0;\nbarrier.cta.red.and.pred q, 1, %1, p;\n"
                   "selp.s32 %0, 1, 0, q;\n}"
                   : "+r"(all)
                   : "n"(R::NT)
                   : "memory");
      ok = all;
    }
    if (ok && m >= 0 && r == 0) mbar_arrive(cta.empty + 8 * slot);
  }
  if (!ok) tile_give_up<BS, TS>(a, cta, R::NT);
}

// slots of the ring with `ctas` CTAs on an SM; fewer than three: not by this kernel
template <int BS, class TS>
int tile_slots(int gmax, int nlev_max, int ctas, int optin) {
  using K = TileCfg<BS, TS>;
  if (nlev_max > kGroupLevelsSmem || gmax <= 0 || gmax >= 0xffff) return 0;
  const long long free = ((long long)optin + 1024) / ctas - 1024 - 2048 - (long long)tile_fixed_smem<BS, TS>(gmax);
  const long long n = free < 0 ? 0 : free / K::SLOT;
  return n < 3 ? 0 : (int)(n < kTileSlotsMax ? n : kTileSlotsMax);
}

int device_attr(cudaDeviceAttr attr) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) return 0;
  return v;
}

// Groups for which the forms of before are ahead: a group's table, barriers and first copies are a fixed cost that
// few elements do not repay, and 16 x 16 blocks in FP32 on wide levels run a lane per row on 512 threads there. Both
// sides in us, the form of before first:
//   FP64  groups of less than 96 rows in more than two rounds over the SMs (160 x 160 elements, 2 x 2 tiles: 4 x 4
//         blocks 59 / 80, 16 x 16 125 / 148; single 36 x 36 blocks 471 / 636; from 96 rows on 1.0 to 1.6 times
//         ahead here), and single 4 x 4 blocks (6.0 / 6.3)
//   FP32  single blocks (4.3 / 6.3; 64 x 64 in any number, 11.5 / 13.0) and groups of less than 8 of 36 x 36 (2 x 2
//         tiles 8.4 / 10.5), in up to two rounds; 16 x 16 blocks in groups of more than 256 on up to a quarter of the SMs, where the lane-per-row
//         form fits (one tile of 32 x 32: 186 / 244; 64 tiles of 24 x 24: 190 / 168)
//   BF16  single 36 x 36 blocks (4.3 / 6.3); groups of less than 12 of 64 x 64 (2 x 2 tiles, 160 x 160: 193 / 285;
//         4 x 4 tiles: 244 / 209)
template <int BS, class TS>
bool tile_behind(const IluGroupPlan& plan, int nlev_max, int sms, int optin) {
  const int g = plan.gmax, n = plan.ngroups;
  if (sizeof(TS) == 8) return g * BS < 16 || (g * BS < 96 && n > 2 * sms);
  if (sizeof(TS) == 2) return g < (BS == 36 ? 2 : 12);
  if (g < 2 && (BS == 64 || n <= 2 * sms)) return true;
  if (BS == 36 && g < 8 && n <= 2 * sms) return true;
  return BS == 16 && g > 256 && n <= sms / 4 && nlev_max <= kGroupLevelsSmem &&
         group_rows_smem<float>(g, BS) + 2048 <= (size_t)optin;
}

template <int BS, class TS>
cudaError_t tile_launch(const IluGroupArgs<TS>& args, int nlev_max, cudaStream_t s) {
  using K = TileCfg<BS, TS>;
  const int optin = device_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin);
  const int sms = device_attr(cudaDevAttrMultiProcessorCount);
  if (optin <= 0 || sms <= 0 || tile_behind<BS, TS>(args.plan, nlev_max, sms, optin)) return cudaErrorNotSupported;
  // as many CTAs on an SM as there are groups for (FP32 up to three, the row kernel two; FP64 reaches the copy
  // rate with one) while each keeps a ring worth having: four slots, the row kernel eight, since a chunk takes
  // that many at once (16 x 16 tiles in BF16: 212 us with one CTA of 16 slots, 272 with two of 4). Eight consumer
  // warps where the CTA has the SM to itself, four where three share it (FP32, 128 x 128: 71 us against 77)
  const int gmax = args.plan.gmax, most = sizeof(TS) == 8 ? 1 : tile_by_rows<BS, TS>() ? 2 : 3;
  const int want = std::min(most, (args.plan.ngroups + sms - 1) / sms), ring = tile_by_rows<BS, TS>() ? 8 : 4;
  int c = want, nslot = tile_slots<BS, TS>(gmax, nlev_max, c, optin);
  while (c > 1 && nslot < ring) nslot = tile_slots<BS, TS>(gmax, nlev_max, --c, optin);
  if (nslot < 3) return cudaErrorNotSupported;
  const void* kern;
  int nt;
  if constexpr (tile_by_rows<BS, TS>()) {
    // more than two rounds of groups: the one-lane-per-row form keeps more of them on an SM and is ahead
    // (8 x 8 tiles: 1024 of them 180 us here against 158, 256 of them 49 against 94)
    if (args.plan.ngroups > 2 * c * sms) return cudaErrorNotSupported;
    kern = (const void*)ilu_apply_tile_rows_kernel<BS, TS>;
    nt = TileRowCfg<BS>::NT + 32;
  } else {
    kern = (const void*)ilu_apply_tile_kernel<BS, TS, 8, 1>;
    nt = 8 * 32 + 32;
    if constexpr (sizeof(TS) < 8) {
      if (c > 1) {
        kern = (const void*)ilu_apply_tile_kernel<BS, TS, 4, 3>;
        nt = 4 * 32 + 32;
      }
    }
  }
  const size_t smem = (size_t)nslot * K::SLOT + tile_fixed_smem<BS, TS>(gmax);
  // the limit is a property of the kernel, shared by all threads: always the same value (tile_slots leaves 2048 bytes
  // to the static shared memory)
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 2048);
  if (e != cudaSuccess) return e;
  IluGroupArgs<TS> ka = args;
  void* params[] = {&ka, &nslot};
  return cudaLaunchKernel(kern, dim3(args.plan.ngroups), dim3(nt), params, smem, s);
}

template <class TS>
cudaError_t tile_apply(const DeviceMesh& dm, const IluGroupShape& gs, const int* task, const int* glev,
                       const int* glev_ptr, const TS* LU, const TS* Uinv, const double* x, double* y, int* err,
                       cudaStream_t s) {
  if (gs.ngroups <= 0 || !gs.loc) return cudaErrorInvalidValue;
  const int bs = dm.nb * dm.neq;
  const IluGroupArgs<TS> args{dm.E, dm.nnzb, LU, Uinv, x, nullptr, y, err,
                              IluGroupPlan{gs.ngroups, reinterpret_cast<const int4*>(task), glev, glev_ptr, gs.gmax,
                                           reinterpret_cast<const int4*>(gs.loc)}};
#define ICX_TILE_CASE(B)           \
  if constexpr (tile_ahead<B, TS>()) \
    if (bs == B) return tile_launch<B, TS>(args, gs.nlev_max, s);
  ICX_BLOCK_SIZES(ICX_TILE_CASE)
#undef ICX_TILE_CASE
  return cudaErrorNotSupported;
}

}  // namespace

cudaError_t la_ilu_apply_tiles(const DeviceMesh& dm, const IluGroupShape& gs, const int* task, const int* glev,
                               const int* glev_ptr, const double* LU, const double* Uinv, const double* x,
                               double* y, int* err, cudaStream_t s) {
  return tile_apply<double>(dm, gs, task, glev, glev_ptr, LU, Uinv, x, y, err, s);
}
cudaError_t la_ilu_apply_tiles(const DeviceMesh& dm, const IluGroupShape& gs, const int* task, const int* glev,
                               const int* glev_ptr, const float* LU, const float* Uinv, const double* x,
                               double* y, int* err, cudaStream_t s) {
  return tile_apply<float>(dm, gs, task, glev, glev_ptr, LU, Uinv, x, y, err, s);
}
cudaError_t la_ilu_apply_tiles(const DeviceMesh& dm, const IluGroupShape& gs, const int* task, const int* glev,
                               const int* glev_ptr, const __nv_bfloat16* LU, const __nv_bfloat16* Uinv,
                               const double* x, double* y, int* err, cudaStream_t s) {
  return tile_apply<__nv_bfloat16>(dm, gs, task, glev, glev_ptr, LU, Uinv, x, y, err, s);
}

}  // namespace icx
