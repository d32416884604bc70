// Finite-difference Jacobian straight into BSR (form_petsc_jacobian_fd,
// src/solvers/include/iceicle/form_petsc_jacobian.hpp:55-317), with the
// reference's perturbation scheme:
//   * faces: every DOF of a side is perturbed by eps_f = max(eps, eps *
//     max(|R_L^f|_2, |R_R^f|_2)) where R^f are that face's own contributions to
//     the two elements' residuals (boundary faces: |R_L^f|_2), and the face's
//     flux is re-evaluated: J(:, c) += (R^f(u + eps_f e_c) - R^f(u)) / eps_f
//     (FJ:97-285, fd_utils.hpp:11-14);
//   * volume: flux-level FD at each quadrature point with
//     eps_q = max(sqrt(eps), sqrt(eps) |F|_F) over u and grad u, contracted
//     analytically with the basis (domain_integral_jacobian,
//     conservation_law.hpp:316-432).
//
// FP32 form (T = float): coefficient tiles, metrics, tabulations and fluxes
// rounded to FP32 and every product, sum and difference taken in FP32, with
// eps = sqrt(FLT_EPSILON) in place of sqrt(DBL_EPSILON) in both schemes; the
// blocks are written as FP32. The FP64 form is this kernel with T = double.
//
// Element-centric: one CTA per element e perturbs e's own DOFs only. It owns
// the diagonal block (volume + the four faces' e-e couplings) and, for each
// face with a neighbour n, the block (n, e) — the neighbour's residual with
// respect to e's DOFs. Every block of the pattern therefore has exactly one
// writer: no atomics, no zero fill.
#include <cfloat>

#include "icx_dg.cuh"
#include "icx_blockrow.cuh"

namespace icx {

// Work of one CTA, in phases between barriers (N1 = P + 1 one-dimensional
// functions, Q1 = G + P points, both as in the residual's sum factorisation):
//   0  coefficient tiles, metrics, 1D tables
//   A  base states, one (point, side, equation) per thread; base fluxes
//   B  perturbed fluxes. On a nodal basis a face's points see the value of
//      the N1 functions on that face only (the others' traces are exactly 0),
//      so the other NB - N1 functions perturb gradients alone: their
//      convective flux is the base one and only the viscous part is evaluated
//   C  the differences D[lf][q][ie][c] are lifted along the face: a thread owns
//      (lf, ie, c), forms L[j] = sum_q b_j(q) D for the neighbour's and for
//      this element's functions, writes its column of the neighbour block
//      (fix_i L_j: one product per entry) and leaves its own L over D
//   D  volume: the point derivatives become W_ab, the coefficients of
//      d_a phi_i d_b phi_j in reference coordinates; two 1D contractions (over
//      q1 into S, then over q0 in registers, (i0, j0) per thread) give the
//      diagonal block, to which the lifted faces are added.
// What bounds it: instruction issue and latency (35 % of the issue slots, 28 % of the FP64 pipe at two CTAs of
// 128 registers per SM), not memory: 1.25 TB/s of stores. Navier-Stokes, p = 3, 64 x 64, FP64: 0.54 ms, against
// 4.73 ms when each entry summed over all points by itself (its reads of D fell into the same banks, 16 lanes
// deep) and every perturbed point took the whole flux; FP32, p = 2, 131 x 77: 0.44 ms against 1.87 ms; Burgers,
// p = 1, 64 x 64 (64 threads per CTA instead of 256): 34 us against 103 us.
template <int PDE, int P, int G, class T = double>
struct JacCfg {
  using C = Cfg<PDE, P, G>;
  static constexpr int NEQ = C::NEQ, NB = C::NB, BS = C::BS, NQF = C::NQF, NQV = C::NQV;
  static constexpr int N1 = P + 1, Q1 = G + P, NP = 4 * NQF;
  static constexpr int THREADS = BS >= 100 ? 512 : BS >= 32 ? 256 : BS >= 16 ? 128 : 64;
  // resident CTAs per SM of the register bound
  static constexpr int MINB = BS >= 100 ? 1 : BS >= 32 ? 2 : BS >= 16 ? 4 : 8;
  static constexpr int NST = NEQ * 7;           // side state: u, grad, Hessian
  static constexpr int NFP = 24;                // FacePt scalars, in the order of FaceGeoField
  static constexpr int IC = Phys<PDE>::has_ic ? 1 : 0;
  // equations ie per pass of phase D: half of them for the largest blocks, whose S would not fit otherwise
  static constexpr int IEC = BS >= 100 ? NEQ / 2 : NEQ;
  static constexpr int NS = 4 * Q1 * IEC * N1 * N1 * NEQ;  // S[4][q0][ie][i1][j1][je]
  // shared memory layout, in scalars of type T
  static constexpr int al(int n) { return (n + 3) / 4 * 4; }
  static constexpr int O_B = 0;                                      // [Q1][N1] values, [Q1][N1] derivatives
  static constexpr int O_FIX = O_B + 2 * Q1 * N1;                    // [4][N1] along each face's fixed direction
  static constexpr int O_VAR = O_FIX + 4 * N1;                       // [4][2][NQF][N1] along the varying one
  static constexpr int O_W = al(O_VAR + 8 * NQF * N1);                   // [6][ie][je][NQV] point derivatives, then W
  static constexpr int O_JI = O_W + 6 * NEQ * NEQ * NQV;             // [4][NQV]
  static constexpr int O_WD = O_JI + 4 * NQV;                        // [NQV]
  static constexpr int O_DFQ = al(O_WD + NQV);                          // [4][NQF][NEQ][BS], then L[4][N1][NEQ][BS]
  static constexpr int O_DGQ = O_DFQ + 4 * NQF * NEQ * BS;           // [4][NQF][4][BS]
  static constexpr int O_S = al(O_DGQ + IC * 4 * NQF * 4 * BS);          // S over the phases A and B data
  static constexpr int O_COEF = O_S;                                 // [5][BS]
  static constexpr int O_FP = O_COEF + 5 * BS;                       // [4][NQF] FacePt
  static constexpr int O_FST = O_FP + NP * NFP;                      // [4][NQF][2][NST]
  static constexpr int O_FQB = O_FST + NP * 2 * NST;                 // [4][NQF][NEQ] base flux
  static constexpr int O_FAB = O_FQB + NP * NEQ;                     // [4][NQF][NEQ] its convective part
  static constexpr int O_GQB = O_FAB + NP * NEQ;                     // [4][NQF][4]
  static constexpr int O_UQ = O_GQB + IC * NP * 4;                   // [NQV][NEQ]
  static constexpr int O_GQ = O_UQ + NQV * NEQ;                      // [NQV][NEQ][2]
  static constexpr int O_FB = O_GQ + NQV * NEQ * 2;                  // [NQV][NEQ][2]
  static constexpr int O_EPSQ = O_FB + NQV * NEQ * 2;                // [NQV], then the reciprocals
  static constexpr int O_EPSF = O_EPSQ + 2 * NQV;                    // [4], then the reciprocals
  static constexpr int O_NRM = O_EPSF + 8;                           // [8]
  static constexpr int O_END = O_NRM + 8;
  static constexpr int TOTAL = O_END > O_S + NS ? O_END : O_S + NS;
  static constexpr size_t SMEM = sizeof(T) * TOTAL;
  static_assert(SMEM <= 227 * 1024, "Jacobian tile exceeds the shared memory of one CTA");
  static_assert(N1 <= NQF, "the lifted faces overwrite the point differences");
};

template <class T>
__device__ inline void fp_load(const T* s, FacePtT<T>& p) {
  p.n[0] = s[0]; p.n[1] = s[1]; p.wsq = s[2]; p.h = s[3];
#pragma unroll
  for (int a = 0; a < 4; ++a) { p.JiL[a] = s[4 + a]; p.JiR[a] = s[14 + a]; }
#pragma unroll
  for (int a = 0; a < 6; ++a) { p.HL[a] = s[8 + a]; p.HR[a] = s[18 + a]; }
}

template <int PDE, int P, int G, bool DDG, class T>
__global__ void __launch_bounds__((JacCfg<PDE, P, G, T>::THREADS), (JacCfg<PDE, P, G, T>::MINB))
    jac_elem_kernel(DeviceMesh dm, PhysParams pp_in, const double* __restrict__ u, T* __restrict__ vals,
                    double eps_in) {
  // every face of the element joins it to the same problem: one parameter set
  const PhysParams pp = elem_params<PDE>(dm, pp_in, blockIdx.x);
  using J = JacCfg<PDE, P, G, T>;
  constexpr int NEQ = J::NEQ, NB = J::NB, BS = J::BS, NQF = J::NQF, NQV = J::NQV, NST = J::NST;
  constexpr int N1 = J::N1, Q1 = J::Q1, NP = J::NP, NT = J::THREADS;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T* sm = reinterpret_cast<T*>(sm_raw);
  const int e = blockIdx.x;
  const int tid = threadIdx.x;
  const bool ic = Phys<PDE>::has_ic && pp.sigma_ic != 0.0;
  const T sqeps = sizeof(T) == sizeof(double) ? T(sqrt(DBL_EPSILON)) : T(sqrtf(FLT_EPSILON));
  const T eps = T(eps_in);

  // per local face: face index, e's side, neighbour, tabulation slots
  struct FaceRec {
    int f, side, nbr, oe, lfn, on, bct, bidx, lL, lR, oR;
  };
  __shared__ FaceRec rec[4];
  if (tid < 4) {
    FaceRec r;
    r.f = dm.el_face[e * 4 + tid];
    const int* fi = dm.face_info + 8 * r.f;
    const int s = dm.el_side[e * 4 + tid];
    r.side = s;
    r.nbr = fi[1] < 0 ? -1 : (s == 0 ? fi[1] : fi[0]);
    r.oe = s ? fi[4] : 0;    // orientation of e's tabulation
    r.lfn = s ? fi[2] : fi[3];  // neighbour's local face number
    r.on = s ? 0 : fi[4];    // orientation of the neighbour's tabulation
    r.bct = fi[5];
    r.bidx = fi[7];
    r.lL = fi[2];
    r.lR = fi[3];
    r.oR = fi[4];
    rec[tid] = r;
  }
  // 1D tables; whether every face sees one function value along its fixed direction (a nodal basis)
  int fixed_ok = 1;
  for (int t = tid; t < 2 * Q1 * N1; t += NT) sm[J::O_B + t] = T(dm.tab_1d[t]);
  for (int t = tid; t < 4 * N1; t += NT) {
    const double v = dm.tab_f1d[t * 3];
    sm[J::O_FIX + t] = T(v);
    const int lf = t / N1, k = t - lf * N1;
    if (k != (lf < 2 ? 0 : P) && v != 0.0) fixed_ok = 0;
  }
  for (int t = tid; t < 8 * NQF * N1; t += NT) sm[J::O_VAR + t] = T(dm.tab_f1d[(4 * N1 + t) * 3]);
  for (int t = tid; t < 4 * NQV; t += NT) {
    const int a = t / NQV, q = t - a * NQV;
    sm[J::O_JI + t] = T(dm.vgeo[(size_t)a * dm.E * NQV + (size_t)e * NQV + q]);
  }
  for (int t = tid; t < NQV; t += NT) sm[J::O_WD + t] = T(dm.vgeo[(size_t)4 * dm.E * NQV + (size_t)e * NQV + t]);
  const bool nodal = __syncthreads_and(fixed_ok);

  // ---- coefficient tiles: [0] = e, [1 + lf] = neighbour across lf; face metrics
  for (int t = tid; t < 5 * BS; t += NT) {
    const int slot = t / BS, r = t - slot * BS;
    const int el = slot == 0 ? e : rec[slot - 1].nbr;
    sm[J::O_COEF + t] = el >= 0 ? T(u[(size_t)el * BS + r]) : T(0.0);
  }
  for (int t = tid; t < NP * J::NFP; t += NT) {
    const int a = t / NP, pt = t - a * NP;
    const int lf = pt / NQF, q = pt - lf * NQF;
    sm[J::O_FP + pt * J::NFP + a] = T(dm.fgeo[(size_t)a * dm.F * NQF + (size_t)rec[lf].f * NQF + q]);
  }
  __syncthreads();

  // ---- phase A: base states, one (point, side, equation) per thread
  for (int t = tid; t < NP * 2 * NEQ; t += NT) {
    const int eq = t % NEQ, sd = t / NEQ % 2, pt = t / (2 * NEQ);
    const int lf = pt / NQF, q = pt - lf * NQF;
    const FaceRec& r = rec[lf];
    if (sd == 1 && r.nbr < 0) continue;
    const T* cf = sm + J::O_COEF + (r.side == sd ? 0 : 1 + lf) * BS + eq;
    const double* tab =
        dm.tab_face + (size_t)(((sd ? r.lR : r.lL) * 2 + (sd ? r.oR : 0)) * NQF + q) * NB * 6;
    const T* fp = sm + J::O_FP + pt * J::NFP + (sd ? FG_JIR : FG_JIL);
    T v = T(0.0), tt[6] = {T(0.0), T(0.0), T(0.0), T(0.0), T(0.0), T(0.0)};
#pragma unroll 4
    for (int i = 0; i < NB; ++i) {
      const T c = cf[i * NEQ];
      v += c * T(tab[i * 6]);
      tt[1] += c * T(tab[i * 6 + 1]);
      tt[2] += c * T(tab[i * 6 + 2]);
      if (DDG) {
        tt[3] += c * T(tab[i * 6 + 3]);
        tt[4] += c * T(tab[i * 6 + 4]);
        tt[5] += c * T(tab[i * 6 + 5]);
      }
    }
    T* st = sm + J::O_FST + (pt * 2 + sd) * NST;
    T gx[2], hx[4];
    basis_phys<DDG>(tt, fp, fp + 4, gx, hx);
    st[eq] = v;
    st[NEQ + eq * 2] = gx[0];
    st[NEQ + eq * 2 + 1] = gx[1];
    if (DDG) {
#pragma unroll
      for (int a = 0; a < 4; ++a) st[3 * NEQ + eq * 4 + a] = hx[a];
    }
  }
  __syncthreads();
  // base fluxes
  for (int t = tid; t < NP + NQV; t += NT) {
    if (t < NP) {
      const int lf = t / NQF, q = t - lf * NQF;
      const FaceRec& r = rec[lf];
      const bool interior = r.nbr >= 0;
      FacePtT<T> fp;
      fp_load(sm + J::O_FP + t * J::NFP, fp);
      const T* sL = sm + J::O_FST + t * 2 * NST;
      const T* sR = sL + NST;
      const double* bval = interior ? nullptr : dm.bvals + ((size_t)r.bidx * NQF + q) * NEQ;
      T out[NEQ], gq[4], fadv[NEQ], fvis[NEQ];
      face_conv_part<PDE, DDG, T>(pp, fp, interior, r.bct, bval, sL, sR, fadv, gq);
      face_visc_part<PDE, DDG, T>(pp, fp, interior, r.bct, bval, sL, sL + NEQ, sL + 3 * NEQ, sR, sR + NEQ,
                                  sR + 3 * NEQ, fvis);
      face_combine<PDE, T>(fp, fvis, fadv, out);
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        sm[J::O_FQB + t * NEQ + k] = out[k];
        sm[J::O_FAB + t * NEQ + k] = fadv[k];
      }
      if (J::IC && ic) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sm[J::O_GQB + t * 4 + k] = gq[k];
      }
    } else {
      // a volume point's base state and flux
      const int q = t - NP;
      const int nq = dm.E * NQV;
      const size_t kq = (size_t)e * NQV + q;
      T Ji[4] = {T(dm.vgeo[0 * nq + kq]), T(dm.vgeo[1 * nq + kq]), T(dm.vgeo[2 * nq + kq]), T(dm.vgeo[3 * nq + kq])};
      const double* tb = dm.tab_vol + (size_t)q * NB * 3;
      const T* cf = sm + J::O_COEF;
      T uq[NEQ], gxi[NEQ][2];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) { uq[k] = T(0.0); gxi[k][0] = gxi[k][1] = T(0.0); }
      for (int i = 0; i < NB; ++i) {
        T phi = T(tb[i * 3]), d0 = T(tb[i * 3 + 1]), d1 = T(tb[i * 3 + 2]);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          T c = cf[i * NEQ + k];
          uq[k] += c * phi;
          gxi[k][0] += c * d0;
          gxi[k][1] += c * d1;
        }
      }
      T gx[2 * NEQ], F[2 * NEQ];
#pragma unroll
      for (int k = 0; k < NEQ; ++k)
#pragma unroll
        for (int d = 0; d < 2; ++d) gx[k * 2 + d] = gxi[k][0] * Ji[0 * 2 + d] + gxi[k][1] * Ji[1 * 2 + d];
      // The differences divide by eps, so a last bit of the base flux is worth 1 / sqrt(FLT_EPSILON) of them. The
      // FP32 form without second derivatives takes the internal energy fused here, which keeps its values where
      // callers had them; the perturbed flux below is rounded as the compiler contracts it. Fused in both, the blocks
      // would be at most 0.9 % nearer to the FP64 ones (NS, 33 x 21, p = 4: 1.183e-3 of their norm instead of
      // 1.193e-3) and would move by 1.1e-4 of it
      Phys<PDE>::template flux<T, sizeof(T) == 4 && !DDG>(pp, uq, gx, F);
      T fro = T(0.0);
#pragma unroll
      for (int k = 0; k < 2 * NEQ; ++k) fro += F[k] * F[k];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) sm[J::O_UQ + q * NEQ + k] = uq[k];
#pragma unroll
      for (int k = 0; k < 2 * NEQ; ++k) {
        sm[J::O_GQ + q * 2 * NEQ + k] = gx[k];
        sm[J::O_FB + q * 2 * NEQ + k] = F[k];
      }
      const T ev = fmax(sqeps, sqrt(fro) * sqeps);
      sm[J::O_EPSQ + q] = ev;
      sm[J::O_EPSQ + NQV + q] = T(1.0) / ev;
    }
  }
  __syncthreads();

  // ---- face perturbation sizes from the base face residual norms (one warp per face and side)
  for (int w = tid >> 5; w < 8; w += NT / 32) {
    const int lane = tid & 31;
    const int lf = w >> 1, sd = w & 1;  // sd: 0 = left element of the face, 1 = right
    const FaceRec& rc = rec[lf];
    T ss = T(0.0);
    if (sd == 0 || rc.nbr >= 0) {
      const int lfs = sd == 0 ? rc.lL : rc.lR, os = sd == 0 ? 0 : rc.oR;
      const T sgn = sd == 0 ? T(1.0) : T(-1.0);
      for (int r = lane; r < BS; r += 32) {
        const int i = r / NEQ, k = r - i * NEQ;
        T v = T(0.0);
#pragma unroll
        for (int q = 0; q < NQF; ++q) {
          const double* tf = dm.tab_face + ((size_t)((lfs * 2 + os) * NQF + q) * NB + i) * 6;
          v += sgn * T(tf[0]) * sm[J::O_FQB + (lf * NQF + q) * NEQ + k];
          if (J::IC && ic)
            v -= T(tf[1]) * sm[J::O_GQB + (lf * NQF + q) * 4 + sd * 2 + 0] +
                 T(tf[2]) * sm[J::O_GQB + (lf * NQF + q) * 4 + sd * 2 + 1];
        }
        ss += v * v;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (lane == 0) sm[J::O_NRM + w] = sqrt(ss);
  }
  __syncthreads();
  if (tid < 4) {
    const T nL = sm[J::O_NRM + 2 * tid], nR = sm[J::O_NRM + 2 * tid + 1];
    const T ev = fmax(eps, fmax(nL, nR) * eps);
    sm[J::O_EPSF + tid] = ev;
    sm[J::O_EPSF + 4 + tid] = T(1.0) / ev;
  }
  __syncthreads();

  // ---- phase B: perturbed face fluxes (e's DOFs) and perturbed volume fluxes
  const int cf_pt = nodal ? N1 * NEQ : BS;              // full evaluations per face point
  const int nfull = NP * cf_pt;
  const int nvis = nodal ? NP * (NB - N1) * NEQ : 0;    // viscous-only evaluations
  for (int t = tid; t < nfull + nvis + NQV * NEQ * 3; t += NT) {
    if (t < nfull + nvis) {
      const bool full = t < nfull;
      const int per = full ? cf_pt : (NB - N1) * NEQ;
      const int t1 = full ? t : t - nfull;
      const int pt = t1 / per, m = t1 - pt * per;
      const int kc = m % NEQ, jj = m / NEQ;
      const int lf = pt / NQF, q = pt - lf * NQF;
      int j;
      if (!nodal) j = jj;
      else if (full) j = (lf & 1) ? jj * N1 + (lf < 2 ? 0 : P) : (lf < 2 ? 0 : P) * N1 + jj;
      else j = (lf & 1) ? jj / P * N1 + jj % P + (lf < 2 ? 1 : 0) : jj + (lf < 2 ? N1 : 0);
      const int c = j * NEQ + kc;
      const FaceRec& r = rec[lf];
      const bool interior = r.nbr >= 0;
      const int se = r.side;
      FacePtT<T> fp;
      fp_load(sm + J::O_FP + pt * J::NFP, fp);
      const T* st = sm + J::O_FST + pt * 2 * NST;
      const T epsf = sm[J::O_EPSF + lf];
      const double* tfd = dm.tab_face + ((size_t)((lf * 2 + r.oe) * NQF + q) * NB + j) * 6;
      T tf[6];
#pragma unroll
      for (int a = 0; a < (DDG ? 6 : 3); ++a) tf[a] = T(tfd[a]);
      T gphi[2], hphi[4];
      basis_phys<DDG>(tf, se ? fp.JiR : fp.JiL, se ? fp.HR : fp.HL, gphi, hphi);
      // both sides' states, side se perturbed in equation kc (explicit fused operations: a product that the
      // selects below share would be rounded on its own, and the differences amplify that)
      T us[2][NEQ], gs[2][2 * NEQ], hs[2][DDG ? 4 * NEQ : 1];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          const bool hit = s == se && k == kc;
          const T uv = st[s * NST + k];
          us[s][k] = hit && full ? fused_madd(epsf, tf[0], uv) : uv;
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            const T gv = st[s * NST + NEQ + k * 2 + d];
            gs[s][k * 2 + d] = hit ? fused_madd(epsf, gphi[d], gv) : gv;
          }
          if (DDG) {
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const T hv = st[s * NST + 3 * NEQ + k * 4 + a];
              hs[s][k * 4 + a] = hit ? fused_madd(epsf, hphi[a], hv) : hv;
            }
          }
        }
      }
      const double* bval = interior ? nullptr : dm.bvals + ((size_t)r.bidx * NQF + q) * NEQ;
      T out[NEQ], gq[4], fadv[NEQ], fvis[NEQ];
      if (full) {
        face_conv_part<PDE, DDG, T>(pp, fp, interior, r.bct, bval, us[0], us[1], fadv, gq);
      } else {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) fadv[k] = sm[J::O_FAB + pt * NEQ + k];
        if (J::IC && ic) {
#pragma unroll
          for (int k = 0; k < 4; ++k) gq[k] = sm[J::O_GQB + pt * 4 + k];
        }
      }
      face_visc_part<PDE, DDG, T>(pp, fp, interior, r.bct, bval, us[0], gs[0], hs[0], us[1], gs[1], hs[1], fvis);
      face_combine<PDE, T>(fp, fvis, fadv, out);
      const T inv = sm[J::O_EPSF + 4 + lf];
#pragma unroll
      for (int k = 0; k < NEQ; ++k)
        sm[J::O_DFQ + (pt * NEQ + k) * BS + c] = (out[k] - sm[J::O_FQB + pt * NEQ + k]) * inv;
      if (J::IC && ic) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          sm[J::O_DGQ + (pt * 4 + k) * BS + c] = (gq[k] - sm[J::O_GQB + pt * 4 + k]) * inv;
      }
    } else {
      const int t2 = t - nfull - nvis;
      const int pidx = t2 / NQV, q = t2 - pidx * NQV;
      T uq[NEQ], gx[2 * NEQ], F[2 * NEQ];
      const T epsq = sm[J::O_EPSQ + q];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        const T v = sm[J::O_UQ + q * NEQ + k];
        uq[k] = k == pidx ? v + epsq : v;
      }
#pragma unroll
      for (int k = 0; k < 2 * NEQ; ++k) {
        const T v = sm[J::O_GQ + q * 2 * NEQ + k];
        gx[k] = k == pidx - NEQ ? v + epsq : v;
      }
      Phys<PDE>::flux(pp, uq, gx, F);
      const T inv = sm[J::O_EPSQ + NQV + q];
      const T* Fb = sm + J::O_FB + q * 2 * NEQ;
      // W component: 0 .. 1 d / du of F_d, 2 + 2 d + jd d / d(du/dx_jd) of F_d
      const int je = pidx < NEQ ? pidx : (pidx - NEQ) >> 1;
#pragma unroll
      for (int ie = 0; ie < NEQ; ++ie)
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int comp = pidx < NEQ ? d : 2 + 2 * d + ((pidx - NEQ) & 1);
          sm[J::O_W + ((comp * NEQ + ie) * NEQ + je) * NQV + q] = (F[ie * 2 + d] - Fb[ie * 2 + d]) * inv;
        }
    }
  }
  __syncthreads();

  // ---- phase C: lift the face differences; neighbour blocks (n, e)
  for (int t = tid; t < 4 * NEQ * BS; t += NT) {
    const int c = t % BS, ie = t / BS % NEQ, lf = t / (BS * NEQ);
    const FaceRec& r = rec[lf];
    T* D = sm + J::O_DFQ + (lf * NQF * NEQ + ie) * BS + c;
    T dq[NQF];
#pragma unroll
    for (int q = 0; q < NQF; ++q) dq[q] = D[q * NEQ * BS];
    if (r.nbr >= 0) {
      const int se = r.side, sn = 1 - se;
      const int blk = dm.face_blk[r.f * 4 + (se == 0 ? 2 : 1)];
      T* Jn = vals + (size_t)blk * BS * BS + (size_t)ie * BS + c;
      const T* bv = sm + J::O_VAR + (r.lfn * 2 + r.on) * NQF * N1;
      const T* bf = sm + J::O_FIX + r.lfn * N1;
      const T sgn = sn == 0 ? T(1.0) : T(-1.0);
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        T s = T(0.0);
#pragma unroll
        for (int q = 0; q < NQF; ++q) s += bv[q * N1 + j] * dq[q];
        s *= sgn;
#pragma unroll
        for (int k = 0; k < N1; ++k) {
          const int i = (r.lfn & 1) ? j * N1 + k : k * N1 + j;
          T v = bf[k] * s;
          if (J::IC && ic) {
            for (int q = 0; q < NQF; ++q) {
              const double* tf = dm.tab_face + ((size_t)((r.lfn * 2 + r.on) * NQF + q) * NB + i) * 6;
              const T* dg = sm + J::O_DGQ + (lf * NQF + q) * 4 * BS + c;
              v -= T(tf[1]) * dg[(sn * 2 + 0) * BS] + T(tf[2]) * dg[(sn * 2 + 1) * BS];
            }
          }
          Jn[(size_t)i * NEQ * BS] = v;
        }
      }
    }
    const T* bv = sm + J::O_VAR + (lf * 2 + r.oe) * NQF * N1;
    const T sgn = r.side == 0 ? T(1.0) : T(-1.0);
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      T s = T(0.0);
#pragma unroll
      for (int q = 0; q < NQF; ++q) s += bv[q * N1 + j] * dq[q];
      D[j * NEQ * BS] = sgn * s;
    }
  }
  // ---- phase D: W_ab in place of the point derivatives; component (a - 1) * 3 + b
  for (int t = tid; t < NEQ * NEQ * NQV; t += NT) {
    const int q = t % NQV;
    constexpr int ST = NEQ * NEQ * NQV;
    T* w = sm + J::O_W + t;
    const T wd = sm[J::O_WD + q];
    const T* Ji = sm + J::O_JI + q;
    const T Du[2] = {w[0], w[ST]};
    const T Dg[2][2] = {{w[2 * ST], w[3 * ST]}, {w[4 * ST], w[5 * ST]}};
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const T j0 = Ji[(a * 2) * NQV] * wd, j1 = Ji[(a * 2 + 1) * NQV] * wd;
      const T h0 = j0 * Dg[0][0] + j1 * Dg[1][0], h1 = j0 * Dg[0][1] + j1 * Dg[1][1];
      w[(a * 3) * ST] = j0 * Du[0] + j1 * Du[1];
#pragma unroll
      for (int b = 0; b < 2; ++b) w[(a * 3 + 1 + b) * ST] = h0 * Ji[(b * 2) * NQV] + h1 * Ji[(b * 2 + 1) * NQV];
    }
  }
  T* Jd = vals + (size_t)dm.bsr_diag[e] * BS * BS;
  const T* sb = sm + J::O_B;
  const T* sdb = sb + Q1 * N1;
#pragma unroll 1
  for (int ie0 = 0; ie0 < NEQ; ie0 += J::IEC) {
    __syncthreads();
    // over q1: S1 = sum b_i1 (W10 b_j1 + W12 b'_j1), S2 = sum b_i1 W11 b_j1, S3, S4 the same with b'_i1 and W2.
    constexpr int ROW = N1 * NEQ;        // [j1][je]
    constexpr int SQ = J::IEC * N1 * ROW;  // one q0
    for (int t = tid; t < J::IEC * Q1 * ROW; t += NT) {
      const int je = t % NEQ, j1 = t / NEQ % N1, q0 = t / ROW % Q1, il = t / (ROW * Q1);
      const T* w = sm + J::O_W + ((ie0 + il) * NEQ + je) * NQV + q0 * Q1;
      constexpr int ST = NEQ * NEQ * NQV;
      T z[4][Q1];
#pragma unroll
      for (int q1 = 0; q1 < Q1; ++q1) {
        const T b = sb[q1 * N1 + j1], db = sdb[q1 * N1 + j1];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          z[a * 2][q1] = w[(a * 3) * ST + q1] * b + w[(a * 3 + 2) * ST + q1] * db;
          z[a * 2 + 1][q1] = w[(a * 3 + 1) * ST + q1] * b;
        }
      }
      T* S = sm + J::O_S + q0 * SQ + il * N1 * ROW + j1 * NEQ + je;
#pragma unroll
      for (int i1 = 0; i1 < N1; ++i1) {
        T s[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
#pragma unroll
        for (int q1 = 0; q1 < Q1; ++q1) {
          const T b = sb[q1 * N1 + i1], db = sdb[q1 * N1 + i1];
          s[0] += b * z[0][q1];
          s[1] += b * z[1][q1];
          s[2] += db * z[2][q1];
          s[3] += db * z[3][q1];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) S[k * Q1 * SQ + i1 * ROW] = s[k];
      }
    }
    __syncthreads();
    // the lifted faces, and over q0; the (i0, j0) entries of one (ie, i1, j1, je) per thread
    for (int t = tid; t < SQ; t += NT) {
      const int je = t % NEQ, j1 = t / NEQ % N1, i1 = t / ROW % N1, ie = ie0 + t / (ROW * N1);
      T acc[N1][N1];
#pragma unroll
      for (int i0 = 0; i0 < N1; ++i0)
#pragma unroll
        for (int j0 = 0; j0 < N1; ++j0) acc[i0][j0] = T(0.0);
#pragma unroll
      for (int lf = 0; lf < 4; ++lf) {
        const T* L = sm + J::O_DFQ + (lf * NQF * NEQ + ie) * BS + j1 * NEQ + je;
        const T* bf = sm + J::O_FIX + lf * N1;
#pragma unroll
        for (int j0 = 0; j0 < N1; ++j0) {
          if ((lf & 1) == 0) {
            const T l = L[i1 * NEQ * BS + j0 * ROW];
#pragma unroll
            for (int i0 = 0; i0 < N1; ++i0) acc[i0][j0] += bf[i0] * l;
          } else {
            const T fx = bf[i1];
#pragma unroll
            for (int i0 = 0; i0 < N1; ++i0) acc[i0][j0] += fx * L[i0 * NEQ * BS + j0 * ROW];
          }
        }
      }
#pragma unroll
      for (int q0 = 0; q0 < Q1; ++q0) {
        const T* S = sm + J::O_S + q0 * SQ + t;
        const T s0 = S[0], s1 = S[Q1 * SQ], s2 = S[2 * Q1 * SQ], s3 = S[3 * Q1 * SQ];
#pragma unroll
        for (int j0 = 0; j0 < N1; ++j0) {
          const T b = sb[q0 * N1 + j0], db = sdb[q0 * N1 + j0];
          const T pv = b * s0 + db * s1, qv = b * s2 + db * s3;
#pragma unroll
          for (int i0 = 0; i0 < N1; ++i0) acc[i0][j0] += sdb[q0 * N1 + i0] * pv + sb[q0 * N1 + i0] * qv;
        }
      }
#pragma unroll
      for (int i0 = 0; i0 < N1; ++i0)
#pragma unroll
        for (int j0 = 0; j0 < N1; ++j0) {
          const int i = i0 * N1 + i1, c = (j0 * N1 + j1) * NEQ + je;
          if (J::IC && ic) {
            for (int lf = 0; lf < 4; ++lf)
              for (int q = 0; q < NQF; ++q) {
                const double* tf = dm.tab_face + ((size_t)((lf * 2 + rec[lf].oe) * NQF + q) * NB + i) * 6;
                const T* dg = sm + J::O_DGQ + ((lf * NQF + q) * 4 + rec[lf].side * 2) * BS + c;
                acc[i0][j0] -= T(tf[1]) * dg[0] + T(tf[2]) * dg[BS];
              }
          }
          Jd[(size_t)(i * NEQ + ie) * BS + c] = acc[i0][j0];
        }
    }
  }
}

// the element kernel of one (PDE, order, geometry order), with the DDG flux's second derivatives or without
template <int PDE, int P, int G, class T>
static cudaError_t jac_pg(const DeviceMesh& dm, const PhysParams& pp, const double* u, T* vals, double eps,
                          cudaStream_t s) {
  using J = JacCfg<PDE, P, G, T>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e1 = cudaFuncSetAttribute(jac_elem_kernel<PDE, P, G, true, T>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)J::SMEM);
    cudaError_t e2 = cudaFuncSetAttribute(jac_elem_kernel<PDE, P, G, false, T>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)J::SMEM);
    if (e1 != cudaSuccess) return e1;
    if (e2 != cudaSuccess) return e2;
    attr_set = true;
  }
  if (pp.beta1 != 0.0)
    jac_elem_kernel<PDE, P, G, true, T><<<dm.E, J::THREADS, J::SMEM, s>>>(dm, pp, u, vals, eps);
  else
    jac_elem_kernel<PDE, P, G, false, T><<<dm.E, J::THREADS, J::SMEM, s>>>(dm, pp, u, vals, eps);
  return cudaGetLastError();
}

template <class T>
static cudaError_t jac_dispatch(const DeviceMesh& dm, const PhysParams& pp, const double* u, T* vals, double eps,
                                cudaStream_t s) {
#define ICX_JAC_CASE(PDE, PP, GG) \
  if (pp.pde == PDE && dm.P == PP && dm.G == GG) return jac_pg<PDE, PP, GG, T>(dm, pp, u, vals, eps, s);
  ICX_JAC_CASE(0, 1, 1) ICX_JAC_CASE(0, 2, 1) ICX_JAC_CASE(0, 3, 1) ICX_JAC_CASE(0, 4, 1)
  ICX_JAC_CASE(0, 1, 2) ICX_JAC_CASE(0, 2, 2) ICX_JAC_CASE(0, 3, 2) ICX_JAC_CASE(0, 4, 2)
  ICX_JAC_CASE(1, 1, 1) ICX_JAC_CASE(1, 2, 1) ICX_JAC_CASE(1, 3, 1) ICX_JAC_CASE(1, 4, 1)
  ICX_JAC_CASE(1, 1, 2) ICX_JAC_CASE(1, 2, 2) ICX_JAC_CASE(1, 3, 2) ICX_JAC_CASE(1, 4, 2)
#undef ICX_JAC_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_jacobian_fd(const DeviceMesh& dm, const PhysParams& pp, const double* u, double* res,
                               double* vals, double eps, cudaStream_t s) {
  cudaError_t e = launch_residual(dm, pp, u, res, s);
  if (e != cudaSuccess) return e;
  return jac_dispatch<double>(dm, pp, u, vals, eps, s);
}

// the FP64 residual and the FP32-quadrature Jacobian (T = float)
cudaError_t launch_jacobian_fd_f32(const DeviceMesh& dm, const PhysParams& pp, const double* u, double* res,
                                   float* vals, cudaStream_t s) {
  cudaError_t e = launch_residual(dm, pp, u, res, s);
  if (e != cudaSuccess) return e;
  return jac_dispatch<float>(dm, pp, u, vals, std::sqrt((double)FLT_EPSILON), s);
}

// ------------------------------------------------------------------ SpMV
// y = J x; one warp per block row, lanes over the rows of the block
cudaError_t launch_bsr_spmv(const DeviceMesh& dm, const double* vals, const double* x, double* y, cudaStream_t s) {
  int bs = dm.nb * dm.neq;
  RowSet rs{0, 0, -1, dm.E};
#define ICX_SPMV_CASE(B) \
  if (bs == B) return launch_block_rows<B, BR_ALL>(rs, dm.bsr_rowptr, dm.bsr_colidx, vals, x, nullptr, 1.0, y, s);
  ICX_BLOCK_SIZES(ICX_SPMV_CASE)
#undef ICX_SPMV_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_bsr_spmv_f32(const DeviceMesh& dm, const float* vals, const double* x, double* y, cudaStream_t s) {
  int bs = dm.nb * dm.neq;
  RowSet rs{0, 0, -1, dm.E};
#define ICX_SPMV32_CASE(B) \
  if (bs == B) return launch_block_rows<B, BR_ALL, float>(rs, dm.bsr_rowptr, dm.bsr_colidx, vals, x, nullptr, 1.0, y, s);
  ICX_BLOCK_SIZES(ICX_SPMV32_CASE)
#undef ICX_SPMV32_CASE
  return cudaErrorInvalidValue;
}

}  // namespace icx
