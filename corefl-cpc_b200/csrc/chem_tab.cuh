// A mechanism repacked for the block chemistry kernel and passed to it by value: constants reach
// the FP64 instructions as constant-bank operands and the reaction loop branches uniformly.
// Reactants and products are lists of species (a species with coefficient 2 is listed twice) for the
// products of concentrations; the coefficients are rows of doubles for the sums over species.
#pragma once
#include "common.cuh"

namespace cb2 {

constexpr int kChemTabReac = 24;  // reactions a table holds (the tables of one launch: 11 KB)
constexpr int kChemTabList = 8;   // reactants (or products) of one reaction, with repeats

enum ChemBack { kBackNone = 0, kBackArrhenius = 1, kBackEquilibrium = 2 };

template <int NS>
struct alignas(16) ChemReac {
  double A, b, Ea, A2, b2, Ea2;   // k = A exp(b ln T - Ea / T)
  double order, order_ln;         // products minus reactants, and that times ln(p_atm / R_u 1e-3)
  double alpha, it3, it1, t2;     // Troe: alpha, 1/T3, 1/T1, T2
  double tb[NS];                  // third-body efficiencies
  double nu[NS], f[NS], bk[NS];   // net, reactant and product coefficients
  unsigned flist, blist;          // 4 bits per entry: species, repeated by its coefficient, padded with
  int nf, nb;                     // species NS, whose concentration is 1; entries in use, at least two
  int type, back;                 // the mechanism's reaction type; ChemBack
};

template <int NS>
struct ChemHead {
  int n_reac, need_gibbs, same_mid, list_len;     // list_len: the longest species list
  double t_mid, t_in_low, t_in_high;              // same_mid: the common middle and the range every fit covers
  double c_per_rho_y[NS], w[NS];                  // 1e-3 / W and 1e3 W
  double tl[NS], tm[NS], th[NS];
  double g[2][NS][7];                             // a0, a1/2, a2/6, a3/12, a4/20, a5, a6 of both ranges
};
template <int NS>
struct ChemTab : ChemHead<NS> {
  ChemReac<NS> r[kChemTabReac];
};

// A table of either size (one is filled), kept by the context.
struct ChemTabs {
  int ns = 0;  // 0: the mechanism does not fit a table
  ChemTab<5> t5;
  ChemTab<9> t9;
  void *rows = nullptr;  // device copy of r
};

}  // namespace cb2
