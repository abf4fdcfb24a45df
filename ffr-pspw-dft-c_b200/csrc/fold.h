// FP64 projector products over pairs (+G, -G) (fold.cu).
#pragma once

#include "common.cuh"
#include "engine.h"

namespace pspw {

// Finds the pairs of a cell's sphere from its grid indices (gi1, gi2, gi3 of
// each G, `order` = the stick lists' G order) and checks on the device that
// EIGR and PKG_A have the symmetry, for every value.  Called once at cell
// creation, after the projector arrays; leaves fold.ok false otherwise.
int fold_prepare(pspw_cell *c, const int *gi1, const int *gi2, const int *gi3, const int *order);

// True when a product over the first ngw G may run over pairs.
inline bool fold_usable(const pspw_cell *c, int ngw) {
  return c->proj.fold.ok && ngw == c->basis.ngw;
}

// wp(p, b) = W_p acc(p, b) for the back-projection, acc the real-matrix sums:
// the projections are acc for even p and i acc for odd p.  With `plain`, the
// unweighted projections themselves.  wp: nproj x nb, column-major.
int fold_project64(pspw_cell *c, const double2 *psi, int ld, int nb, double2 *wp, bool plain);

// out(:, b) += alpha sum_p beta_p (projections of p, b), from fold_project64's wp
int fold_backproject64(pspw_cell *c, const double2 *wp, int nb, double2 *out, int ldo,
                       double alpha);

}  // namespace pspw
