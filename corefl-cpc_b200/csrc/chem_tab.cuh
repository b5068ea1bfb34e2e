// A mechanism repacked for the block chemistry kernel and passed to it by value: constants reach
// the FP64 instructions as constant-bank operands and the reaction loop branches uniformly.
// Reactants and products are lists of species (a species with coefficient 2 is listed twice), so
// that no operation is spent on zero coefficients.
#pragma once
#include "common.cuh"

namespace cb2 {

constexpr int kChemTabReac = 24;  // reactions a table holds (the tables of one launch: 6 KB)
constexpr int kChemTabList = 8;   // reactants (or products) of one reaction, with repeats
constexpr int kChemTabMult = 3;   // largest stoichiometric coefficient

enum ChemBack { kBackNone = 0, kBackArrhenius = 1, kBackEquilibrium = 2 };

struct ChemReac {
  double A, b, Ea, A2, b2, Ea2;   // k = A exp(b ln T - Ea / T)
  double order_ln;                // order x ln(p_atm / R_u 1e-3)
  double order;                   // sum of products minus reactants
  double alpha, it3, it1, t2;     // Troe: alpha, 1/T3, 1/T1, T2
  double tb[kMaxSpec];            // third-body efficiencies
  unsigned flist, blist;          // 4 bits per entry: species index
  int nf, nb;                     // entries in use
  int type, back;                 // the mechanism's reaction type; ChemBack
  unsigned short mf[kChemTabMult], mb[kChemTabMult];  // bit s: coefficient of species s > level
  int levels;                     // largest coefficient
};

template <int NS>
struct ChemTab {
  int n_reac, need_gibbs, same_mid;
  double t_mid, t_in_low, t_in_high;              // same_mid: the common middle and the range every fit covers
  double c_per_rho_y[NS], w[NS];                  // 1e-3 / W and 1e3 W
  double tl[NS], tm[NS], th[NS];
  double g[2][NS][7];                             // a0, a1/2, a2/6, a3/12, a4/20, a5, a6 of both ranges
  ChemReac r[kChemTabReac];
};

// A table of either size (one is filled), kept by the context.
struct ChemTabs {
  int ns = 0;  // 0: the mechanism does not fit a table
  ChemTab<5> t5;
  ChemTab<9> t9;
};

}  // namespace cb2
