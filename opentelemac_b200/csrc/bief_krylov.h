// bief_krylov.h -- the persistent solver kernels by method, TYPDIA, storage,
// dot-product mode and residency.  The methods other than GRACJG are
// compiled in bief_krylov.cu.
#pragma once

#include "bief_kernels.cuh"

namespace bief {

// Kernel of a method for TYPDIA code td, storage sto, dot-product mode
// (comp: MODASS = 3, compensated) and residency (wide: twice the blocks per
// SM, MINB = 2 CG_MIN_BLOCKS)
#define KSEL1(k, STO_, C_, M_)                                                \
  (td == DIA_Q ? (void *)k<DIA_Q, STO_, C_, M_>                                \
               : td == DIA_I ? (void *)k<DIA_I, STO_, C_, M_> : (void *)k<DIA_0, STO_, C_, M_>)
#define KSELM(k, M_)                                                          \
  (sto == 3 ? (comp ? KSEL1(k, 3, true, M_) : KSEL1(k, 3, false, M_))         \
            : (comp ? KSEL1(k, 1, true, M_) : KSEL1(k, 1, false, M_)))
#define KSEL(k) (wide ? KSELM(k, 2 * CG_MIN_BLOCKS) : KSELM(k, CG_MIN_BLOCKS))

void *equnor_kernel(int td, int sto, bool comp = false, bool wide = false);
void *rescjg_kernel(int td, int sto, bool comp = false, bool wide = false);
void *errmin_kernel(int td, int sto, bool comp = false, bool wide = false);
void *cgsqua_kernel(int td, int sto, bool comp = false, bool wide = false);
void *gmres_kernel(int td, int sto, bool comp = false, bool wide = false);
void *cgstab_kernel(int td, int sto, bool comp = false, bool wide = false);

}  // namespace bief
