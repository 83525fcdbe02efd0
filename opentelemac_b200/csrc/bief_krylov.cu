// bief_krylov.cu -- instantiations of the solver kernels of SLV 2 to 7.
#include "bief_krylov.h"

namespace bief {

void *equnor_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_equnor);
}

void *rescjg_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_rescjg);
}

void *errmin_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_errmin);
}

void *cgsqua_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_cgsqua);
}

void *gmres_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_gmres);
}

void *cgstab_kernel(int td, int sto, bool comp, bool wide) {
  return KSEL(k_cgstab);
}

}  // namespace bief
