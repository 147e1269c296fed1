// The straight-line lattice kernels of classes without d shells and of the small ones
// with them; the launch table of all of them (pfe_lattice_sl2.cu holds the rest).

#include "pfe_lattice_sl.cuh"

namespace pfe {

int lattice_sl_passes(int e1, int e2, bool sw) {
  switch (e1 * 8 + e2) {
    case 18: return 4;               // (11|11)
    case 26:                         // (20|11)
    case 33: return sw ? 4 : 5;      // (21|10)
    case 27: return 5;               // (20|20)
    default: return lattice_sl_launcher(e1, e2, sw) ? 1 : 0;
  }
}

// evaluated class (e1 >= e2) and swap flag -> straight-line launcher, or null
LatSlFn lattice_sl_launcher(int e1, int e2, bool sw) {
#define L2(A, B, C, D) (sw ? &launch_sl<A, B, C, D, true> : &launch_sl<A, B, C, D, false>)
  switch (e1 * 8 + e2) {
    case 0: return L2(0, 0, 0, 0);
    case 8: return L2(1, 0, 0, 0);
    case 9: return L2(1, 0, 1, 0);
    case 16: return L2(1, 1, 0, 0);
    case 17: return L2(1, 1, 1, 0);
    case 18: return sw ? &launch_sl_passes<1, 1, 1, 1, true, 4> : &launch_sl_passes<1, 1, 1, 1, false, 4>;
    case 24: return L2(2, 0, 0, 0);
    case 25: return L2(2, 0, 1, 0);
    case 32: return L2(2, 1, 0, 0);
    default: return lattice_sl_launcher_d(e1, e2, sw);
  }
#undef L2
}

}  // namespace pfe
