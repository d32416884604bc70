// C entries to the block-ILU(0) launchers for tests that hand them what no
// context makes: a set error flag, a plan whose neighbour never runs, block
// patterns of other meshes. Device pointers throughout.
#include <vector>

#include "icx_internal.h"
#include "icx_linalg.h"

namespace {
icx::IluStripPlan plan(int nstrips, int max_steps, int max_nx, void* strips, double* ex, long long nex,
                       unsigned long long* ticket) {
  icx::IluStripPlan p;
  p.nstrips = nstrips;
  p.max_steps = max_steps;
  p.max_nx = max_nx;
  p.strips = static_cast<icx::IluStrip*>(strips);
  p.ex = ex;
  p.nex = nex;
  p.ticket = ticket;
  return p;
}
}  // namespace

extern "C" {

int strip_rows(int bs) { return icx::ilu_strip_rows(bs); }
long long strip_bytes(int bs, int nx, int nr, int f32) { return icx::ilu_strip_bytes(bs, nx, nr, f32 != 0); }

int strip_pack(int bs, int nstrips, int max_steps, int max_nx, void* strips, double* ex, long long nex,
               unsigned long long* ticket, const double* LU, const double* Uinv, void* pk, int f32) {
  const icx::IluStripPlan p = plan(nstrips, max_steps, max_nx, strips, ex, nex, ticket);
  cudaError_t e = icx::la_ilu_strip_reset(p, 0);
  if (e == cudaSuccess)
    e = f32 ? icx::la_ilu_strip_pack_f32(bs, p, LU, Uinv, static_cast<float*>(pk), 0)
            : icx::la_ilu_strip_pack(bs, p, LU, Uinv, static_cast<double*>(pk), 0);
  return (int)e;
}

int strip_apply(int bs, int nstrips, int max_steps, int max_nx, void* strips, double* ex, long long nex,
                unsigned long long* ticket, const void* pk, int f32, const double* x, double* y, double* f, int* err,
                int side_by_side) {
  const icx::IluStripPlan p = plan(nstrips, max_steps, max_nx, strips, ex, nex, ticket);
  return (int)(f32 ? icx::la_ilu_apply_strips_f32(bs, p, static_cast<const float*>(pk), x, y, f, err,
                                                  side_by_side != 0, 0)
                   : icx::la_ilu_apply_strips(bs, p, static_cast<const double*>(pk), x, y, f, err, side_by_side != 0,
                                              0));
}

int ilu_factor(int E, int bs, int nnzb, int* rowptr, int* colidx, const int* order, const int* lvl_off, int n_levels,
               double* LU, double* Uinv, int* flag) {
  icx::DeviceMesh dm{};
  dm.E = E;
  dm.nb = bs;
  dm.neq = 1;
  dm.nnzb = nnzb;
  dm.bsr_rowptr = rowptr;
  dm.bsr_colidx = colidx;
  return (int)icx::la_ilu_factor(dm, order, std::vector<int>(lvl_off, lvl_off + n_levels + 1), LU, Uinv, flag, 0);
}

}  // extern "C"
