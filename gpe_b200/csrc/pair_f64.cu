// pair_f64.cu -- complex128 pair kernels (pair_kernel.cuh).
#include "pair.h"
#include "pair_kernel.cuh"

namespace gpe {
namespace {

template <int R, int KIND>
const void* by_form(int form) {
  if (form == FORM_PLAIN)
    return reinterpret_cast<const void*>(&pair_kernel<double, R, KIND, false, FORM_PLAIN, false>);
  if (form == FORM_TRAP)
    return reinterpret_cast<const void*>(&pair_kernel<double, R, KIND, false, FORM_TRAP, false>);
  return nullptr;
}

template <int R>
const void* by_kind(int kind, int form) {
  return kind == PAIR_RK4_A   ? by_form<R, PAIR_RK4_A>(form)
         : kind == PAIR_RK4_B ? by_form<R, PAIR_RK4_B>(form)
                              : by_form<R, PAIR_RK2>(form);
}

}  // namespace

const void* pair_fn_f64(int R, int kind, int form) {
  return R == 1 ? by_kind<1>(kind, form) : by_kind<2>(kind, form);
}

}  // namespace gpe
