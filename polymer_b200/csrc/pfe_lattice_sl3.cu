// The straight-line lattice kernels of (21|10) in register passes, compiled apart.

#include "pfe_lattice_sl.cuh"

namespace pfe {

LatSlFn lattice_sl_launcher_2110(bool sw) {
  return sw ? &launch_sl_passes<2, 1, 1, 0, true, 4> : &launch_sl_passes<2, 1, 1, 0, false, 5>;
}

}  // namespace pfe
