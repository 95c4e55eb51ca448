// pair_batch.cu -- batched rk4 pair kernels (pair_kernel.cuh).
#include "pair.h"
#include "pair_kernel.cuh"

namespace gpe {
namespace {

template <typename T, int R, int KIND, bool KAHAN>
const void* by_form(int form) {
  if (form == FORM_PLAIN)
    return reinterpret_cast<const void*>(&pair_kernel<T, R, KIND, KAHAN, FORM_PLAIN, true>);
  if (form == FORM_TRAP)
    return reinterpret_cast<const void*>(&pair_kernel<T, R, KIND, KAHAN, FORM_TRAP, true>);
  return nullptr;
}

template <typename T, int R>
const void* by_kind(int kind, bool kahan, int form) {
  if (kind == PAIR_RK4_A) return by_form<T, R, PAIR_RK4_A, false>(form);
  if (kind != PAIR_RK4_B) return nullptr;
  if constexpr (std::is_same<T, float>::value)
    if (kahan) return by_form<T, R, PAIR_RK4_B, true>(form);
  return by_form<T, R, PAIR_RK4_B, false>(form);
}

}  // namespace

const void* pair_fn_batch(int es, int R, int kind, bool kahan, int form) {
  if (es == 8) return R == 1 ? by_kind<float, 1>(kind, kahan, form) : by_kind<float, 2>(kind, kahan, form);
  return R == 1 ? by_kind<double, 1>(kind, false, form) : by_kind<double, 2>(kind, false, form);
}

}  // namespace gpe
