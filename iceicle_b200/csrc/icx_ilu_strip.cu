// Block-ILU(0) apply on whole structured grids, by strips of grid rows:
//   forward   f_e = x_e - sum_{k<e} L_ek f_k                      (natural order)
//   backward  y_e = inv(U_ee) f_e - sum_{k>e} (inv(U_ee) U_ek) y_k  (reverse order)
// One CTA owns up to S consecutive rows of a grid and runs along them: in step
// t its row k holds element t - k, so the elements of a step (an anti-diagonal
// of the strip) are independent, and what a step needs was formed one step
// earlier by the same CTA: it passes through shared memory behind one CTA
// barrier. Only the row below (above) the strip comes from another CTA, through
// an exchange buffer in global memory: the producer stores its last row there,
// and one warp of the consumer (the fetcher) reads that row ahead of the steps,
// re-reading slots that still hold a sentinel and putting the sentinel back once
// read, so that a finished apply leaves the buffer ready for the next one (inside
// a cluster the row goes straight into the consumer's shared memory). A strip
// that is given up leaves NaN, never what y held before. A strip follows its
// neighbour at a distance of one hand-over; after that both run at the pace of
// the in-CTA steps.
//
// The factors are repacked once per factorisation in the order in which the
// steps read them: a step's blocks of all rows are one contiguous piece, entry
// by entry in lane order (absent blocks are zeros), which another warp (the
// loader) copies ahead with one bulk copy per step into a ring in shared memory,
// and which the lanes read without bank conflicts, one step ahead, into
// registers. A matrix row is shared by LPR lanes (columns q, q + LPR, ...). The
// sums are taken in the order of the data-flow apply (32 column accumulators
// added pairwise at distances 16, 8, 4, 2, 1), so the results are the same bit
// for bit.
//
// Against the data-flow apply, whose every level is a trip through L2 (FP64 /
// FP32): NS p = 2 256 x 256 1.69 -> 1.03 / 1.56 -> 0.91 ms, 128 x 128 716 -> 448
// us; Burgers p = 2 32 x 32 139 -> 45 us (a Newton solve 132 -> 62 ms, with the
// dot products' steps); also ahead on one row or column of 1000 elements and on
// rows too wide for an inbox (NS p = 2 400 x 400 3.29 -> 3.00 ms).
#include <algorithm>
#include <vector>

#include "icx_bulk.cuh"
#include "icx_internal.h"
#include "icx_linalg.h"
#include "icx_blockrow.cuh"

namespace icx {

namespace {

// lanes per matrix row, rows per strip and the ring of staged steps for a block size
template <int BS, class TA>
struct StripCfg {
  static constexpr int LPR = BS <= 9 ? 2 : 4;
  static constexpr int NCOL = (BS + LPR - 1) / LPR;  // columns per lane
  static constexpr int NA = 32 / LPR;                // its column accumulators
  static constexpr int EL = BS * LPR;                // lanes per element
  static constexpr int S = ilu_strip_rows(BS);
  static constexpr int NL = S * EL;                  // lanes with work
  static constexpr int NW = (NL + 31) / 32;          // worker warps
  static constexpr int NT = NW * 32 + 96;            // and the fetcher, the loader and the vector warp
  // CTAs per SM to compile for: what sets of problems side by side share an SM with (16 x 16 blocks compiled for one:
  // a set of 16 problems, orders 1 to 4, 314 ms instead of 301; left to the compiler 304)
  static constexpr int MINB = BS == 4 ? 4 : BS == 9 || BS == 16 ? 2 : 1;
  static constexpr int NF = 2 * NCOL, NB = 3 * NCOL; // entries per lane and step, forward and backward
  static constexpr int BF = (NF * NL * (int)sizeof(TA) + 15) / 16 * 16;  // bytes of a packed step
  static constexpr int BB = (NB * NL * (int)sizeof(TA) + 15) / 16 * 16;
  // the ring: chunks of two steps' entries, and x or f of VD steps
  static constexpr int CHUNK = 2 * BB, VB = (S * BS * 8 + 15) / 16 * 16, VD = 8;
  static constexpr int DMAX = 6;  // chunks at most (the launch takes what fits, at least 2)
};

template <class TA>
struct StripArgs {
  int nstrips;
  const IluStrip* strips;
  const unsigned char* pk;  // packed factors: strip s's forward steps at pk + strips[s].pk, then its backward steps
  const double* x;
  double* f;
  double* y;
  double* ex;  // exchange rows: strip s, sweep w at ex + strips[s].ex[w]
  int* err;
  int depth;   // chunks in the ring
  int cluster; // CTAs per cluster (1: every hand-over through the exchange rows)
  int inbox;   // values of an inbox: a row of the widest grid (the same in all CTAs of a cluster)
  int sweep;   // 0 both sweeps in one launch (all CTAs resident), 1 the forward one, 2 the backward one
  unsigned long long* ticket;  // sweep 1 and 2: tickets drawn by the clusters so far
};

// a row handed over inside a cluster goes straight into the consumer's shared memory, into an inbox per sweep of the
// launch: a slot is written once, so no store of the backward sweep has to be ordered against the forward one's
__device__ inline unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ inline unsigned cluster_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ inline void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ inline void st_cluster_f64(unsigned addr, double v) {
  asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ inline double ld_cluster_f64(unsigned addr) {
  double v;
  asm volatile("ld.relaxed.cluster.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

// the steps after whose barrier every thread looks whether a wait was given up (the two flags alternate, so
// that none is written while it may still be read)
constexpr int kStripCheck = 16;
__device__ inline bool strip_check(int t, int nsteps) { return t % kStripCheck == kStripCheck - 1 || t == nsteps - 1; }

// all bits set: a NaN in FP64, and two of them in FP32
__device__ inline double strip_nan() { return __longlong_as_double(-1ll); }

// y of a strip whose sweeps were given up: NaN, never what y held before or values of an unfinished sweep
template <int BS>
__device__ inline void strip_give_up(const IluStrip& st, double* y) {
  double* const ys = y + ((size_t)st.e0 + (size_t)st.j0 * st.nx) * BS;
  for (int i = threadIdx.x; i < st.nr * st.nx * BS; i += blockDim.x) ys[i] = strip_nan();
}

template <int BS, class TA>
struct StripShared {
  double vec[2][StripCfg<BS, TA>::S + 1][BS];  // by step parity: the neighbour strip's element, then each row's
  unsigned long long bars[StripCfg<BS, TA>::DMAX];
  int stop[2];
};

// one sweep of one strip; false (uniform over the CTA) when a wait was given up. gch: the chunks used so far
// (slot gch % D of the ring, phase (gch / D) & 1 of its barrier)
template <int BS, class TA, bool FWD>
__device__ inline bool strip_sweep(const StripArgs<TA>& a, int s, StripShared<BS, TA>& sh, unsigned char* ring,
                                   double* inbox, unsigned& gch) {
  using K = StripCfg<BS, TA>;
  constexpr int LPR = K::LPR, NCOL = K::NCOL, NA = K::NA, VD = K::VD, NE = FWD ? K::NF : K::NB;
  constexpr unsigned BYTES = FWD ? K::BF : K::BB;
  const IluStrip st = a.strips[s];
  const int nx = st.nx, nr = st.nr;
  const int nsteps = nx + nr - 1, nch = (nsteps + 1) / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* stop = sh.stop;
  const int D = a.depth;
  const int rank = a.cluster > 1 ? (int)cluster_rank() : 0;
  const bool has_prev = FWD ? st.j0 > 0 : st.j0 + nr < st.ny;

  // absent neighbours are zero blocks: they must meet finite values
  for (int i = tid; i < 2 * (K::S + 1) * BS; i += K::NT) (&sh.vec[0][0][0])[i] = 0.0;
  __syncthreads();

  if (warp == K::NW) {
    // ---- fetcher: the neighbour strip's row, element t in vec[(t + 1) & 1][0] before step t
    constexpr int NP = (BS + 31) / 32, Q = 8;
    double* ein = has_prev ? a.ex + a.strips[FWD ? s - 1 : s + 1].ex[FWD ? 0 : 1] : nullptr;
    double v[Q][NP];
    const bool near = has_prev && a.cluster > 1 && (FWD ? rank > 0 : rank < a.cluster - 1);
    const unsigned in0 = (unsigned)__cvta_generic_to_shared(inbox) + lane * 8;
    auto ask = [&](int c, double (&o)[NP]) {
#pragma unroll
      for (int p = 0; p < NP; ++p)
        if (has_prev && !near && c < nx && lane + 32 * p < BS) o[p] = ld_relaxed_f64(ein + (size_t)c * BS + lane + 32 * p);
    };
    // given up: a NaN in the neighbour's row from here on, so that what is still computed and handed on cannot pass
    // for a result (an element's rows all read all of its neighbours; the step that is running may or may not see it)
    auto poison = [&]() {
      if (lane < 2) *reinterpret_cast<volatile double*>(sh.vec[lane][0]) = strip_nan();
      return false;
    };
    // element c's vector (slot u0 of the window c .. c + Q - 1) into shared memory; false when the wait was
    // given up. A wait asks again for the whole window: a poll's trip covers several of the producer's steps,
    // and a window asked for element by element would cost a trip for each
    auto take = [&](int c, int u0, double* dst) -> bool {
      if (!has_prev || c >= nx) return true;
      unsigned spins = 0;
      if (near) {
        // from the inbox, filled by the neighbouring CTA of the cluster
        double o[NP];
        while (true) {
          bool ready = true;
#pragma unroll
          for (int p = 0; p < NP; ++p)
            if (lane + 32 * p < BS) {
              o[p] = ld_cluster_f64(in0 + (c * BS + 32 * p) * 8);
              if ((unsigned long long)__double_as_longlong(o[p]) == FLOW_SENTINEL) ready = false;
            }
          if (__all_sync(0xffffffffu, ready)) break;
          int quit = 0;
          if (lane == 0 && (++spins & 1023) == 0) {
            if (*reinterpret_cast<volatile int*>(a.err)) quit = 1;
            else if (spins > 8 * ICX_FLOW_SPINS) {
              atomicExch(a.err, 1);
              quit = 1;
            }
          }
          if (__shfl_sync(0xffffffffu, quit, 0)) return poison();
        }
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (lane + 32 * p < BS) dst[lane + 32 * p] = o[p];
        return true;
      }
      while (true) {
        bool ready = true;
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (lane + 32 * p < BS && (unsigned long long)__double_as_longlong(v[u0][p]) == FLOW_SENTINEL) ready = false;
        if (__all_sync(0xffffffffu, ready)) break;
        int quit = 0;
        if (lane == 0) {
          if (*reinterpret_cast<volatile int*>(a.err)) quit = 1;
          else if (++spins > ICX_FLOW_SPINS) {
            atomicExch(a.err, 1);
            quit = 1;
          }
        }
        if (__shfl_sync(0xffffffffu, quit, 0)) return poison();
#pragma unroll
        for (int d = 0; d < Q; ++d) ask(c + d, v[(u0 + d) % Q]);
      }
#pragma unroll
      for (int p = 0; p < NP; ++p)
        if (lane + 32 * p < BS) {
          dst[lane + 32 * p] = v[u0][p];
          ein[(size_t)c * BS + lane + 32 * p] = __longlong_as_double((long long)FLOW_SENTINEL);
        }
      return true;
    };
#pragma unroll
    for (int u = 0; u < Q; ++u) ask(u, v[u]);
    // an apply that was given up leaves *err set: later ones end at once
    bool ok = __all_sync(0xffffffffu, *reinterpret_cast<volatile int*>(a.err) == 0) || poison();
    ok = ok && take(0, 0, sh.vec[1][0]);
    ask(Q, v[0]);
    __syncthreads();
    for (int t0 = 0; t0 < nsteps; t0 += Q) {
#pragma unroll
      for (int u = 0; u < Q; ++u) {
        const int t = t0 + u;
        if (t < nsteps) {
          ok = ok && take(t + 1, (u + 1) % Q, sh.vec[t & 1][0]);
          ask(t + 1 + Q, v[(u + 1) % Q]);
          if (!ok && lane == 0 && strip_check(t, nsteps)) stop[t / kStripCheck & 1] = 1;
          __syncthreads();
          if (strip_check(t, nsteps) && stop[t / kStripCheck & 1]) return false;
        }
      }
    }
    gch += nch;
    return true;
  }
  if (warp == K::NW + 1) {
    // ---- loader: before the barrier that ends an even step t, the chunk of steps t + 2 and t + 3 has landed; a
    // chunk's slot is free once its second step's entries are read, in the chunk's first step
    const unsigned bar0 = (unsigned)__cvta_generic_to_shared(sh.bars);
    const unsigned ring0 = (unsigned)__cvta_generic_to_shared(ring);
    const unsigned char* src = a.pk + st.pk + (FWD ? 0 : (size_t)nsteps * K::BF);
    unsigned islot = gch % D, wslot = gch % D, phase = gch / D & 1;
    int issued = 0, waited = 0;
    bool ok = true;
    auto issue = [&]() {
      if (issued < nch && lane == 0) {
        const unsigned bytes = 2 * issued + 2 <= nsteps ? 2 * BYTES : BYTES;
        mbar_expect(bar0 + 8 * islot, bytes);
        bulk_copy(ring0 + islot * K::CHUNK, src + (size_t)issued * 2 * BYTES, bytes, bar0 + 8 * islot);
      }
      ++issued;
      islot = islot + 1 == D ? 0 : islot + 1;
    };
    auto wait = [&]() {
      if (!__all_sync(0xffffffffu, waited >= nch || mbar_wait(bar0 + 8 * wslot, phase))) {
        // not landed: NaN in its place (a copy that lands after all brings the right entries)
        ok = false;
        for (int i = lane; i < K::CHUNK / 8; i += 32) reinterpret_cast<double*>(ring + wslot * K::CHUNK)[i] = strip_nan();
      }
      ++waited;
      if (++wslot == D) {
        wslot = 0;
        phase ^= 1;
      }
    };
#pragma unroll 1
    for (int u = 0; u < D; ++u) issue();
    wait();
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < nsteps; ++t) {
      if (t & 1) issue();
      else wait();
      if (!ok && lane == 0) atomicExch(a.err, 1);
      if (!ok && lane == 0 && strip_check(t, nsteps)) stop[t / kStripCheck & 1] = 1;
      __syncthreads();
      if (strip_check(t, nsteps) && stop[t / kStripCheck & 1]) {
        // given up: the copies in flight land before the CTA ends
        while (waited < issued && waited < nch) wait();
        return false;
      }
    }
    gch += nch;
    return true;
  }
  unsigned char* const vring = ring + (size_t)D * K::CHUNK;
  if (warp == K::NW + 2) {
    // ---- vector warp: x (forward) or the elements' own f (backward), VD - 1 steps ahead, one value per lane and
    // row of 32
    constexpr int NX = (K::S * BS + 31) / 32;
    const unsigned ring0 = (unsigned)__cvta_generic_to_shared(vring) + lane * 8;
    const double* gV[NX];
    int vk[NX];
#pragma unroll
    for (int u = 0; u < NX; ++u) {
      const int p = lane + 32 * u, k = p / BS;
      vk[u] = p < K::S * BS && k < nr ? k : -1;
      const int j = FWD ? st.j0 + k : st.j0 + nr - 1 - k;
      gV[u] = (FWD ? a.x : a.f) + ((ptrdiff_t)st.e0 + (ptrdiff_t)j * nx + (FWD ? -k : nx - 1 + k)) * BS + (p - k * BS);
    }
    int issued = 0;
    auto issue = [&]() {
#pragma unroll
      for (int u = 0; u < NX; ++u) {
        if (vk[u] >= 0 && (unsigned)(issued - vk[u]) < (unsigned)nx)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(ring0 + issued % VD * K::VB + 32 * u * 8), "l"(gV[u])
                       : "memory");
        gV[u] += FWD ? BS : -BS;
      }
      cp_async_commit();
      ++issued;
    };
#pragma unroll 1
    for (int u = 0; u < VD - 1; ++u) issue();
    cp_async_wait<VD - 2>();
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < nsteps; ++t) {
      issue();  // step t + VD - 1, into the slot read in step t - 1
      cp_async_wait<VD - 2>();
      __syncthreads();
      if (strip_check(t, nsteps) && stop[t / kStripCheck & 1]) {
        cp_async_wait<0>();
        return false;
      }
    }
    cp_async_wait<0>();
    gch += nch;
    return true;
  }

  // ---- workers: lane li of row k's element holds columns q, q + LPR, ... of matrix row r
  const int k = tid / K::EL, li = tid - k * K::EL;
  const int r = li / LPR, q = li % LPR;
  const bool lives = tid < K::NL;
  const int kk = lives ? k : 0;
  const int j = FWD ? st.j0 + kk : st.j0 + nr - 1 - kk;
  const unsigned cnt = lives && k < nr ? nx : 0;  // the row's elements c = 0 .. cnt - 1
  const bool has_next = FWD ? st.j0 + nr < st.ny : st.j0 > 0;
  const bool hand = k == nr - 1 && has_next && q == 0;
  const int e00 = st.e0 + j * nx + (FWD ? 0 : nx - 1);
  constexpr ptrdiff_t SE = FWD ? 1 : -1;
  double* gO = (FWD ? a.f : a.y) + (size_t)e00 * BS + r;
  double* gX = has_next ? a.ex + st.ex[FWD ? 0 : 1] + r : nullptr;
  const bool near_next = has_next && a.cluster > 1 && (FWD ? rank < a.cluster - 1 : rank > 0);
  unsigned nX = near_next ? cluster_map((unsigned)__cvta_generic_to_shared(inbox) + r * 8, FWD ? rank + 1 : rank - 1) : 0;
  // the lane's entries of a step: chunk by chunk, two steps each
  const unsigned char* el = ring + gch % D * K::CHUNK + (lives ? tid : 0) * sizeof(TA);
  const unsigned char* const el_end = ring + (size_t)D * K::CHUNK + (lives ? tid : 0) * sizeof(TA);
  auto read = [&](int par, TA (&m)[NE]) {
    const TA* p = reinterpret_cast<const TA*>(el + (par ? BYTES : 0));
#pragma unroll
    for (int n = 0; n < NE; ++n) m[n] = p[n * K::NL];
    if (par) el = el + K::CHUNK == el_end ? el_end - D * K::CHUNK : el + K::CHUNK;
  };
  const unsigned char* ve = vring + kk * BS * 8;
  const unsigned char* const ve_end = ve + VD * K::VB;
  int c = -kk;
  auto run = [&](int par, const TA (&m)[NE], TA (&mn)[NE]) {
    const bool in = (unsigned)c < cnt;
    const double* prev = &sh.vec[par ^ 1][kk][q];  // row k - 1's vector; row k's own is BS further
    const double* vs = reinterpret_cast<const double*>(ve);
    constexpr int NV = NCOL < NA ? NCOL : NA;  // accumulators in use (the rest would add zeros)
    TA v0[NCOL], v1[NCOL], v2[FWD ? 1 : NCOL];
#pragma unroll
    for (int n = 0; n < NCOL; ++n) {
      const bool col = q + LPR * n < BS;
      v0[n] = col ? (TA)prev[(FWD ? 0 : BS) + LPR * n] : TA(0);  // ascending columns: below, left / right, above
      v1[n] = col ? (TA)prev[(FWD ? BS : 0) + LPR * n] : TA(0);
      if constexpr (!FWD) v2[n] = in && col ? (TA)vs[q + LPR * n] : TA(0);
    }
    const double xv = FWD ? vs[r] : 0.0;
    read(par ^ 1, mn);  // the next step's entries
    TA acc[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) acc[n] = TA(0);
#pragma unroll
    for (int n = 0; n < NCOL; ++n) acc[n % NA] = fused_madd(-m[n], v0[n], acc[n % NA]);
#pragma unroll
    for (int n = 0; n < NCOL; ++n) acc[n % NA] = fused_madd(-m[NCOL + n], v1[n], acc[n % NA]);
    if constexpr (!FWD) {
#pragma unroll
      for (int n = 0; n < NCOL; ++n) acc[n % NA] = fused_madd(m[2 * NCOL + n], v2[n], acc[n % NA]);
    }
    // lane l = q + LPR n of the data-flow apply's warp: distances 16, 8, ... down to LPR here, the rest by shuffles
#pragma unroll
    for (int h = NA / 2; h > 0; h >>= 1)
#pragma unroll
      for (int n = 0; n < NV; ++n)
        if (n < h && n + h < NV) acc[n] = acc[n] + acc[n + h];
    TA sum = acc[0];
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (in && q == 0) {
      const double val = FWD ? xv + (double)sum : (double)sum;
      sh.vec[par][kk + 1][r] = val;
      if (hand) {
        if (near_next) st_cluster_f64(nX, flow_value(val));
        else st_relaxed_f64(gX, flow_value(val));
      }
      *gO = val;
      gX += BS;
      nX += BS * 8;
      gO += SE * BS;
    }
    ++c;
    ve = ve + K::VB == ve_end ? ve_end - VD * K::VB : ve + K::VB;
  };
  TA ma[NE], mb[NE];
  __syncthreads();  // the first chunk has landed
  read(0, ma);
#pragma unroll 1
  for (int t = 0; t < nsteps; t += 2) {
    run(0, ma, mb);
    __syncthreads();
    if (strip_check(t, nsteps) && stop[t / kStripCheck & 1]) return false;
    if (t + 1 >= nsteps) break;
    run(1, mb, ma);
    __syncthreads();
    if (strip_check(t + 1, nsteps) && stop[(t + 1) / kStripCheck & 1]) return false;
  }
  gch += nch;
  return true;
}

// One launch for both sweeps: strips are dealt to the CTAs round-robin in order;
// every CTA runs its forward sweeps in ascending, then its backward sweeps in
// descending order. A strip waits only for the one before (after) it, and the
// whole grid is resident (cooperative launch), so the first unfinished strip can
// always run.
// One launch per sweep: every CTA runs one strip, and the clusters draw tickets
// as they start, ascending strips for the forward, descending ones for the
// backward sweep. A strip then waits only for a CTA of its own cluster or for a
// cluster that drew before it, so nothing needs to be resident: for plans larger
// than the GPU, and for several applies side by side (cooperative launches run
// one after the other).
template <int BS, class TA>
__global__ void __launch_bounds__((StripCfg<BS, TA>::NT), (StripCfg<BS, TA>::MINB)) ilu_apply_strip_kernel(StripArgs<TA> a) {
  using K = StripCfg<BS, TA>;
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ StripShared<BS, TA> sh;
  double* inbox = reinterpret_cast<double*>(ring + (size_t)a.depth * K::CHUNK + K::VD * K::VB);
  int s = blockIdx.x;
  if (threadIdx.x < 2) sh.stop[threadIdx.x] = 0;
  if (threadIdx.x < K::DMAX) mbar_init((unsigned)__cvta_generic_to_shared(sh.bars + threadIdx.x), 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __shared__ unsigned drawn;
  const int ncl = gridDim.x / a.cluster;
  if (a.sweep && cluster_rank() == 0 && threadIdx.x == 0)
    drawn = (unsigned)(atomicAdd(a.ticket, 1ull) % (unsigned long long)ncl);
  if (a.sweep) {
    cluster_sync();
    unsigned t;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(t) : "r"(cluster_map((unsigned)__cvta_generic_to_shared(&drawn), 0)) : "memory");
    s = (int)(a.sweep == 1 ? t : ncl - 1 - t) * a.cluster + (int)cluster_rank();
  }
  if (a.cluster > 1) {
    const int n = a.sweep == 0 ? 2 * a.inbox : a.inbox;
    for (int i = threadIdx.x; i < n; i += K::NT) inbox[i] = __longlong_as_double((long long)FLOW_SENTINEL);
    cluster_sync();
  } else {
    __syncthreads();
  }
  unsigned gch = 0;
  bool ok = true;
  if (a.sweep == 0) {
    for (; ok && s < a.nstrips; s += gridDim.x) ok = strip_sweep<BS, TA, true>(a, s, sh, ring, inbox, gch);
    while (s < a.nstrips) s += gridDim.x;  // given up forwards: none of this CTA's strips is finished
    for (s -= gridDim.x; s >= 0; s -= gridDim.x) {
      ok = ok && strip_sweep<BS, TA, false>(a, s, sh, ring, inbox + a.inbox, gch);
      if (!ok) strip_give_up<BS>(a.strips[s], a.y);
    }
  } else if (s < a.nstrips) {
    // the backward launch after a forward one that was given up ends at once (*err)
    if (a.sweep == 1) strip_sweep<BS, TA, true>(a, s, sh, ring, inbox, gch);
    else if (!strip_sweep<BS, TA, false>(a, s, sh, ring, inbox, gch)) strip_give_up<BS>(a.strips[s], a.y);
  }
  // no CTA of a cluster ends while another may still store into its inbox
  if (a.cluster > 1) cluster_sync();
}

// the factors in the order of the steps: blockIdx.x the strip, blockIdx.y step and sweep (forward steps first)
template <int BS, class TA>
__global__ void __launch_bounds__(256) strip_pack_kernel(const IluStrip* __restrict__ strips,
                                                         const double* __restrict__ LU,
                                                         const double* __restrict__ Uinv, unsigned char* pk) {
  using K = StripCfg<BS, TA>;
  constexpr int LPR = K::LPR, NCOL = K::NCOL, B2 = BS * BS;
  const IluStrip st = strips[blockIdx.x];
  const int nx = st.nx, nsteps = nx + st.nr - 1;
  const bool fwd = (int)blockIdx.y < nsteps;
  const int t = fwd ? blockIdx.y : blockIdx.y - nsteps;
  if (t >= nsteps) return;
  TA* out = reinterpret_cast<TA*>(pk + st.pk + (fwd ? (size_t)t * K::BF : (size_t)nsteps * K::BF + (size_t)t * K::BB));
  const int ne = fwd ? K::NF : K::NB;
  for (int p = threadIdx.x; p < ne * K::NL; p += blockDim.x) {
    const int n = p / K::NL, l = p - n * K::NL;
    const int b = n / NCOL, m = n - b * NCOL;
    const int k = l / K::EL, li = l - k * K::EL, r = li / LPR, col = li % LPR + LPR * m;
    const int c = t - k;
    double v = 0.0;
    if (k < st.nr && c >= 0 && c < nx && col < BS) {
      const int j = fwd ? st.j0 + k : st.j0 + st.nr - 1 - k, i = fwd ? c : nx - 1 - c;
      // blocks of element (i, j) in natural order: below, left, diagonal, right, above
      const int d = 1 + (j > 0) + (j < st.ny - 1);
      const int rp = st.b0 + j * (3 * nx - 2) + nx * ((j > 0 ? j - 1 : 0) + j) + i * d + (i > 0 ? i - 1 : 0) + i;
      const int diag = rp + (j > 0) + (i > 0);
      int blk = -1;  // forward: below, left; backward: right, above, inv(U_ee)
      if (fwd) blk = b == 0 ? (j > 0 ? rp : -1) : (i > 0 ? rp + (j > 0) : -1);
      else if (b < 2) blk = b == 0 ? (i < nx - 1 ? diag + 1 : -1) : (j < st.ny - 1 ? diag + 1 + (i < nx - 1) : -1);
      if (!fwd && b == 2) v = Uinv[((size_t)(st.e0 + j * nx + i) * BS + r) * BS + col];
      else if (blk >= 0) v = LU[(size_t)blk * B2 + r * BS + col];
    }
    out[p] = (TA)v;
  }
}

__global__ void strip_fill_kernel(long long n, double* ex) {
  const double v = __longlong_as_double((long long)FLOW_SENTINEL);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    ex[i] = v;
}

constexpr int kStripSmem = 225 * 1024, kStripCluster = 8;

// a launch by clusters of strips that hand their rows over in shared memory: so many inboxes (a row of the widest
// grid each) beside the ring; side by side with other applies no more than two chunks, so that several CTAs share an
// SM. depth < 2: the inboxes leave no room
template <int BS, class TA>
struct StripClusters {
  using K = StripCfg<BS, TA>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  int depth = 0, resident = 0;  // chunks of the ring, clusters that run at the same time
  static long long fit(const IluStripPlan& p, int inboxes) {
    return (kStripSmem - K::VD * K::VB - (long long)inboxes * p.max_nx * BS * 8) / K::CHUNK;
  }
  StripClusters(const IluStripPlan& p, int inboxes, bool side_by_side, cudaStream_t s) {
    depth = (int)std::min<long long>(side_by_side ? 2 : 4, fit(p, inboxes));
    if (depth < 2) return;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kStripCluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(K::NT);
    cfg.gridDim = dim3((p.nstrips + kStripCluster - 1) / kStripCluster * kStripCluster);
    cfg.dynamicSmemBytes = (size_t)depth * K::CHUNK + K::VD * K::VB + (size_t)inboxes * p.max_nx * BS * 8;
    cfg.stream = s;
    if (cudaOccupancyMaxActiveClusters(&resident, ilu_apply_strip_kernel<BS, TA>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      resident = 0;
    }
  }
  StripClusters(const StripClusters&) = delete;
};

// the kernel's dynamic shared memory limit is its own, shared by all threads: always the same value
template <int BS, class TA>
cudaError_t strip_limit() {
  return cudaFuncSetAttribute(ilu_apply_strip_kernel<BS, TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStripSmem);
}

template <int BS, class TA>
cudaError_t launch_strips(const IluStripPlan& p, const StripArgs<TA>& args, bool side_by_side, cudaStream_t s) {
  using K = StripCfg<BS, TA>;
  using C = StripClusters<BS, TA>;
  constexpr auto kern = ilu_apply_strip_kernel<BS, TA>;
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = strip_limit<BS, TA>();
  if (e != cudaSuccess) return e;
  StripArgs<TA> a = args;
  a.inbox = p.max_nx * BS;
  a.cluster = kStripCluster;
  // one cooperative launch for both sweeps (saves a launch and the tickets) where their inboxes leave the ring three
  // chunks, or as many as one inbox does, and the whole grid is resident
  if (!side_by_side && C::fit(p, 2) >= 2 && C::fit(p, 2) >= std::min<long long>(3, C::fit(p, 1))) {
    C both(p, 2, false, s);
    if ((long long)both.resident * kStripCluster >= both.cfg.gridDim.x) {
      both.cfg.numAttrs = 2;
      a.depth = both.depth;
      a.sweep = 0;
      return cudaLaunchKernelEx(&both.cfg, kern, a);
    }
  }
  C each(p, 1, side_by_side, s);
  if (each.resident > 0) {
    a.depth = each.depth;
    for (a.sweep = 1; a.sweep <= 2; ++a.sweep)
      if ((e = cudaLaunchKernelEx(&each.cfg, kern, a)) != cudaSuccess) return e;
    return cudaSuccess;
  }
  // rows too wide for an inbox: every hand-over through L2
  a.depth = (int)std::min<long long>(K::DMAX, (kStripSmem - K::VD * K::VB) / K::CHUNK);
  a.cluster = 1;
  a.sweep = 0;
  const size_t smem = (size_t)a.depth * K::CHUNK + K::VD * K::VB;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, K::NT, smem)) != cudaSuccess) return e;
  if (per_sm < 1 || a.depth < 2) return cudaErrorNotSupported;
  const int grid = std::min(p.nstrips, nsm * per_sm);
  void* params[] = {&a};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(K::NT), params, smem, s);
}

template <int BS, class TA>
cudaError_t pack_strips(const IluStripPlan& p, const double* LU, const double* Uinv, TA* pk, cudaStream_t s) {
  strip_pack_kernel<BS, TA><<<dim3(p.nstrips, 2 * p.max_steps), 256, 0, s>>>(p.strips, LU, Uinv,
                                                                            reinterpret_cast<unsigned char*>(pk));
  return cudaGetLastError();
}

#define ICX_STRIP_SIZES(X) X(4) X(9) X(16) X(25) X(36)

template <class TA>
cudaError_t apply_strips(int bs, const IluStripPlan& p, const TA* pk, const double* x, double* y, double* f, int* err,
                         bool side_by_side, cudaStream_t s) {
  if (p.nstrips < 1 || !pk) return cudaErrorInvalidValue;
  StripArgs<TA> a{p.nstrips, p.strips, reinterpret_cast<const unsigned char*>(pk), x, f, y, p.ex, err, 0, 1, 0, 0, p.ticket};
#define ICX_STRIP_CASE(B) \
  if (bs == B) return launch_strips<B, TA>(p, a, side_by_side, s);
  ICX_STRIP_SIZES(ICX_STRIP_CASE)
#undef ICX_STRIP_CASE
  return cudaErrorNotSupported;
}

template <class TA>
cudaError_t pack_all(int bs, const IluStripPlan& p, const double* LU, const double* Uinv, TA* pk, cudaStream_t s) {
  if (p.nstrips < 1 || !pk) return cudaErrorInvalidValue;
#define ICX_STRIP_CASE(B) \
  if (bs == B) return pack_strips<B, TA>(p, LU, Uinv, pk, s);
  ICX_STRIP_SIZES(ICX_STRIP_CASE)
#undef ICX_STRIP_CASE
  return cudaErrorNotSupported;
}

}  // namespace

long long ilu_strip_bytes(int bs, int nx, int nr, bool f32) {
  const long long steps = nx + nr - 1;
#define ICX_STRIP_CASE(B)                                                             \
  if (bs == B)                                                                        \
    return steps * (f32 ? (long long)StripCfg<B, float>::BF + StripCfg<B, float>::BB  \
                        : (long long)StripCfg<B, double>::BF + StripCfg<B, double>::BB);
  ICX_STRIP_SIZES(ICX_STRIP_CASE)
#undef ICX_STRIP_CASE
  return 0;
}

bool la_ilu_strips_resident(int bs, const IluStripPlan& p, bool f32) {
#define ICX_STRIP_CASE(B)                                                                                           \
  if (bs == B)                                                                                                      \
    return f32 ? strip_limit<B, float>() != cudaSuccess || StripClusters<B, float>(p, 1, true, 0).resident == 0     \
               : strip_limit<B, double>() != cudaSuccess || StripClusters<B, double>(p, 1, true, 0).resident == 0;
  ICX_STRIP_SIZES(ICX_STRIP_CASE)
#undef ICX_STRIP_CASE
  return true;
}

cudaError_t la_ilu_strip_reset(const IluStripPlan& p, cudaStream_t s) {
  if (p.nex <= 0) return cudaSuccess;
  strip_fill_kernel<<<(int)std::min<long long>((p.nex + 255) / 256, 148 * 8), 256, 0, s>>>(p.nex, p.ex);
  return cudaGetLastError();
}

cudaError_t la_ilu_strip_pack(int bs, const IluStripPlan& p, const double* LU, const double* Uinv, double* pk,
                              cudaStream_t s) {
  return pack_all<double>(bs, p, LU, Uinv, pk, s);
}
cudaError_t la_ilu_strip_pack_f32(int bs, const IluStripPlan& p, const double* LU, const double* Uinv, float* pk,
                                  cudaStream_t s) {
  return pack_all<float>(bs, p, LU, Uinv, pk, s);
}
cudaError_t la_ilu_apply_strips(int bs, const IluStripPlan& p, const double* pk, const double* x, double* y, double* f,
                                int* err, bool side_by_side, cudaStream_t s) {
  return apply_strips<double>(bs, p, pk, x, y, f, err, side_by_side, s);
}
cudaError_t la_ilu_apply_strips_f32(int bs, const IluStripPlan& p, const float* pk, const double* x, double* y,
                                    double* f, int* err, bool side_by_side, cudaStream_t s) {
  return apply_strips<float>(bs, p, pk, x, y, f, err, side_by_side, s);
}

}  // namespace icx
