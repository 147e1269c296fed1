// The pass variants of kept components only of (22|11), single molecules and batches,
// compiled apart so the build runs them in parallel.

#define PFE_KEPT_UNIT
#include "pfe_mol_kernels.cuh"

namespace pfe {

PFE_KEPT(2, 2, 1, 1, )

}  // namespace pfe
