// The lane-group kernels (kin_group.cuh), one precision (-DSGB_PREC=0, 1 or 4) and one size of
// mechanism (-DSGB_NM: species at most) per compilation: 8, 16 or 32 lanes per cell, Rodas3
// coefficients folded in or read from the launch.

#include <string.h>

#include "group.h"
#include "kin_group.cuh"

#if !defined(SGB_PREC) || !defined(SGB_NM)
#error "compile with -DSGB_PREC=0, 1 or 4 and -DSGB_NM=12, 17, 20 or 32"
#endif

namespace sgb {

namespace {
template <class M> GroupFn of_lanes(uint32_t G) {
    return G == 8 ? kin_group_kernel<M, SGB_PREC, 8, SGB_NM>
                  : G == 16 ? kin_group_kernel<M, SGB_PREC, 16, SGB_NM> : kin_group_kernel<M, SGB_PREC, 32, SGB_NM>;
}
}   // namespace

template <> GroupFn group_kernel<SGB_PREC, SGB_NM>(uint32_t G, bool rodas3) {
#if SGB_NM == 17   // exact n: Rodas3 only (group_kernel_for)
    (void)rodas3;
    return of_lanes<Rodas3Coef>(G);
#else
    return rodas3 ? of_lanes<Rodas3Coef>(G) : of_lanes<RuntimeCoef>(G);
#endif
}

}   // namespace sgb
