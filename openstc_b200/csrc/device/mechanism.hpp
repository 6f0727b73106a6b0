// The stoichiometry of the H2-O2-N2 mechanism the package ships
// (data/chemistry/combustion_mechanism.inp: 9 species, 19 reactions), known
// at compile time so that the chemistry kernels unroll over its reactions:
// a reaction touches 3 to 4 of the 9 species, so dense loops over run-time
// coefficients spend most of their work on zeros and on converting integers.
// Rate constants, third-body efficiencies and thermodynamics stay run-time
// values.  mech::matches says whether a case's mechanism has this
// stoichiometry, whatever its rates; any other mechanism takes the general
// loops.
#pragma once

#include "common.cuh"

namespace ostc {
namespace mech {

struct H2O2 {
  static constexpr int ns = 9, nr = 19;
  // reaction types as the CHEMKIN reader labels them: 1 elementary, 3
  // duplicate (two rates added), 4 third body, 6 Troe falloff
  static constexpr int label[nr] = {1, 1, 1, 1, 4, 4, 4, 4, 6, 1, 1, 1, 1, 3, 6, 1, 1, 1, 3};
  // H2 H O2 O OH HO2 H2O2 H2O N2
  static constexpr int sf[nr][ns] = {
      {0, 1, 1, 0, 0, 0, 0, 0, 0}, {1, 0, 0, 1, 0, 0, 0, 0, 0}, {1, 0, 0, 0, 1, 0, 0, 0, 0},
      {0, 0, 0, 1, 0, 0, 0, 1, 0}, {1, 0, 0, 0, 0, 0, 0, 0, 0}, {0, 0, 0, 2, 0, 0, 0, 0, 0},
      {0, 1, 0, 1, 0, 0, 0, 0, 0}, {0, 1, 0, 0, 1, 0, 0, 0, 0}, {0, 1, 1, 0, 0, 0, 0, 0, 0},
      {0, 1, 0, 0, 0, 1, 0, 0, 0}, {0, 1, 0, 0, 0, 1, 0, 0, 0}, {0, 0, 0, 1, 0, 1, 0, 0, 0},
      {0, 0, 0, 0, 1, 1, 0, 0, 0}, {0, 0, 0, 0, 0, 2, 0, 0, 0}, {0, 0, 0, 0, 0, 0, 1, 0, 0},
      {0, 1, 0, 0, 0, 0, 1, 0, 0}, {0, 1, 0, 0, 0, 0, 1, 0, 0}, {0, 0, 0, 1, 0, 0, 1, 0, 0},
      {0, 0, 0, 0, 1, 0, 1, 0, 0}};
  static constexpr int sb[nr][ns] = {
      {0, 0, 0, 1, 1, 0, 0, 0, 0}, {0, 1, 0, 0, 1, 0, 0, 0, 0}, {0, 1, 0, 0, 0, 0, 0, 1, 0},
      {0, 0, 0, 0, 2, 0, 0, 0, 0}, {0, 2, 0, 0, 0, 0, 0, 0, 0}, {0, 0, 1, 0, 0, 0, 0, 0, 0},
      {0, 0, 0, 0, 1, 0, 0, 0, 0}, {0, 0, 0, 0, 0, 0, 0, 1, 0}, {0, 0, 0, 0, 0, 1, 0, 0, 0},
      {1, 0, 1, 0, 0, 0, 0, 0, 0}, {0, 0, 0, 0, 2, 0, 0, 0, 0}, {0, 0, 1, 0, 1, 0, 0, 0, 0},
      {0, 0, 1, 0, 0, 0, 0, 1, 0}, {0, 0, 1, 0, 0, 0, 1, 0, 0}, {0, 0, 0, 0, 2, 0, 0, 0, 0},
      {0, 0, 0, 0, 1, 0, 0, 1, 0}, {1, 0, 0, 0, 0, 1, 0, 0, 0}, {0, 0, 0, 0, 1, 1, 0, 0, 0},
      {0, 0, 0, 0, 0, 1, 0, 1, 0}};
  static constexpr int nu(int r, int k) { return sb[r][k] - sf[r][k]; }
  static constexpr int order(int r) {
    int o = 0;
    for (int k = 0; k < ns; ++k) o += nu(r, k);
    return o;
  }
};

template <class M>
inline bool matches(const DevParams &p) {
  if (p.ns != M::ns || p.nr != M::nr) return false;
  for (int r = 0; r < M::nr; ++r) {
    if (p.label[r] != M::label[r] || p.order[r] != M::order(r)) return false;
    for (int k = 0; k < M::ns; ++k)
      if (p.sf[r * M::ns + k] != M::sf[r][k] || p.sb[r * M::ns + k] != M::sb[r][k]) return false;
  }
  return true;
}

}  // namespace mech
}  // namespace ostc
