// The pass variants of kept components only of (22|20), (21|20), single molecules and batches,
// compiled apart so the build runs them in parallel.

#define PFE_KEPT_UNIT
#include "pfe_mol_kernels.cuh"

namespace pfe {

PFE_KEPT(2, 2, 2, 0, )
PFE_KEPT(2, 1, 2, 0, )

}  // namespace pfe
