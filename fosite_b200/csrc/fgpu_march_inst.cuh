// fgpu_march_inst.cuh -- instantiation and launch of the marching stage kernels over the compiled-in
// limiters, with and without reductions and sources (included by one translation unit per kernel
// family, so that they compile in parallel).
#pragma once
#include "fgpu_march_launch.h"

namespace fgpu {
namespace {

// Fam<LIM, RED, SRC>::run(args...) launches one kernel, ::configure() opts it into its shared
// memory.  PLAIN: the family has kernels without sources (ideal-gas physics, whose Cartesian
// grids are the common case; isothermal grids are disks with sources).
template <template <int, bool, bool> class Fam, bool PLAIN, int LIM, class... T>
void launch_red(bool red, bool plain, T... a) {
  if constexpr (PLAIN) {
    if (plain) {
      if (red) Fam<LIM, true, false>::run(a...);
      else Fam<LIM, false, false>::run(a...);
      return;
    }
  }
  if (red) Fam<LIM, true, true>::run(a...);
  else Fam<LIM, false, true>::run(a...);
}
template <template <int, bool, bool> class Fam, bool PLAIN, class... T>
void launch_family(int lim, bool red, bool plain, T... a) {
  switch (lim) {
    case LIM_MINMOD: launch_red<Fam, PLAIN, LIM_MINMOD>(red, plain, a...); break;
    case LIM_MC: launch_red<Fam, PLAIN, LIM_MC>(red, plain, a...); break;
    case LIM_VANLEER: launch_red<Fam, PLAIN, LIM_VANLEER>(red, plain, a...); break;
    default: launch_red<Fam, PLAIN, 0>(red, plain, a...); break;
  }
}
template <template <int, bool, bool> class Fam, bool PLAIN, int LIM>
void configure_lim() {
  Fam<LIM, false, true>::configure();
  Fam<LIM, true, true>::configure();
  if constexpr (PLAIN) {
    Fam<LIM, false, false>::configure();
    Fam<LIM, true, false>::configure();
  }
}
template <template <int, bool, bool> class Fam, bool PLAIN>
void configure_family(int lim) {
  switch (lim) {
    case LIM_MINMOD: configure_lim<Fam, PLAIN, LIM_MINMOD>(); break;
    case LIM_MC: configure_lim<Fam, PLAIN, LIM_MC>(); break;
    case LIM_VANLEER: configure_lim<Fam, PLAIN, LIM_VANLEER>(); break;
    default: configure_lim<Fam, PLAIN, 0>(); break;
  }
}

}  // namespace
}  // namespace fgpu
