// The straight-line lattice kernels of (20|11) and (20|20) in register passes, compiled
// apart from the smaller classes.

#include "pfe_lattice_sl.cuh"

namespace pfe {

LatSlFn lattice_sl_launcher_d(int e1, int e2, bool sw) {
  switch (e1 * 8 + e2) {
    case 26: return sw ? &launch_sl_passes<2, 0, 1, 1, true, 4> : &launch_sl_passes<2, 0, 1, 1, false, 5>;
    case 27: return sw ? &launch_sl_passes<2, 0, 2, 0, true, 5> : &launch_sl_passes<2, 0, 2, 0, false, 5>;
    case 33: return lattice_sl_launcher_2110(sw);
    default: return nullptr;
  }
}

}  // namespace pfe
