// FP64 projector products over pairs (+G, -G) (fold.cu).
#pragma once

#include <vector>

#include "common.cuh"
#include "engine.h"

namespace pspw {

// Finds the pairs of a cell's sphere from its stick lists (cell_create's:
// sticks in ascending (y, x), their G in ascending z, `order` the G of each
// position) and checks on the device that EIGR and PKG_A have the symmetry, for
// every value.  Called once at cell creation, after the projector arrays;
// leaves fold.ok false otherwise.
int fold_prepare(pspw_cell *c, const std::vector<int> &col_x, const std::vector<int> &col_y,
                 const std::vector<int> &col_of_xy, const std::vector<int> &col_start,
                 const std::vector<int> &sg_z, const std::vector<int> &order);

// Groups that hold a pair with one of the first ngw G (pairs are in ascending
// order of their first G).
int fold_groups(const Fold &f, int ngw);

// wp(p, b) = W_p acc(p, b) for the back-projection, acc the real-matrix sums:
// the projections are acc for even p and i acc for odd p.  With `plain`, the
// unweighted projections themselves.  wp: nproj x nb, column-major.  The sums
// are over the first ngw G (in the stick order: all of them).
int fold_project64(pspw_cell *c, const double2 *psi, int ld, int ngw, int nb, double2 *wp,
                   bool plain);

// out(G, b) += alpha sum_p beta_p(G) (projections of p, b) for the first ngw G,
// from fold_project64's wp
int fold_backproject64(pspw_cell *c, const double2 *wp, int ngw, int nb, double2 *out, int ldo,
                       double alpha);

}  // namespace pspw
