// smo_form_exact.cu -- the persistent SMO solver of FORM_EXACT (smo_solver.cuh).
#include "smo_resident.cuh"

namespace svmb {

const void *smo_entry_exact() { return (const void *)smo_persistent<FORM_EXACT>; }
const void *smo_rows_exact() { return (const void *)smo_rows<FORM_EXACT>; }
const void *smo_cluster_exact() { return (const void *)smo_cluster<FORM_EXACT>; }

}  // namespace svmb
