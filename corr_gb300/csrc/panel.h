// Panels of (ia|jb) of an occupied block (panel.cu): the plain form's energy
// from the digit GEMM, and the elementwise step of the adjoint.
#pragma once

#include "abi_internal.h"
#include "dgemm_tc.h"

namespace corr {

// Element (i, a), (j, b), i0 <= i < i0 + ni and j >= i0, of the panel at
// p[((i - i0) v + a) ld + (j v + b - col0)].
struct PanelView {
  double* p;
  long long ld, col0;
  int o, v, i0, ni;
};

// Blocks of ni occupied orbitals whose panels stay within `budget` (at least
// one orbital), the column operand's digit planes (col_bytes; 0 where they would
// exceed kDgPlaneBytes: every block's product slices its columns again, 24 bytes
// of traffic per element against 2 ni nvir operations at the digit GEMM's rate),
// the workspace of a block's product, and the partials of all launch_panel calls.
struct PanelPlan {
  int ni, split;
  size_t panel_bytes, col_bytes, product_bytes;
  long long partials;
};
constexpr size_t kPanelBudget = (size_t)512 << 20;
constexpr int kPanelMaxNvir = 6144;  // of the gradient's panels (sums of W in shared memory)
PanelPlan panel_plan(int o, int v, int X, size_t budget);

// panel = B_block^T B over Q, its diagonal (ia|ia) in FP64; cols: the sliced columns of B, or null.
// dws: product_bytes of the plan.
int panel_product(corr_context* c, int o, int v, int X, const double* bia, const DgColumns* cols,
                  int i0, int ni, double* panel, void* dws, PanelView* pv);
// Energy partials ({E_OS, E_SS} per CTA), or with grad the elements replaced by
// the adjoint G, W added to deps and {E, 0} partials.  split (of the plan): CTAs
// per (i, j) block; ni (o - i0) split partials.
int launch_panel(corr_context* c, const PanelView& pv, const double* eps, double* deps,
                 double* part, int split, bool grad);

// The plain form's energy: scratch bytes, and the evaluation on device-resident
// inputs (raises kStatusNeedFp64 for values out of the digit GEMM's range).
size_t energy_panel_bytes(int o, int v, int X);
int energy_from_panels(corr_context* c, Carver& w, int o, int v, int X, const double* bia,
                       const double* eps, double* out_e);

}  // namespace corr
