// pair_f32.cu -- complex64 pair kernels (pair_kernel.cuh), and the choice
// among all of them.
#include "pair.h"
#include "pair_kernel.cuh"

namespace gpe {
namespace {

template <int R, int KIND, bool KAHAN>
const void* by_form(int form) {
  if (form == FORM_PLAIN)
    return reinterpret_cast<const void*>(&pair_kernel<float, R, KIND, KAHAN, FORM_PLAIN, false>);
  if (form == FORM_TRAP)
    return reinterpret_cast<const void*>(&pair_kernel<float, R, KIND, KAHAN, FORM_TRAP, false>);
  if constexpr (R == 1)
    return reinterpret_cast<const void*>(&pair_kernel<float, R, KIND, KAHAN, FORM_FULL, false>);
  return nullptr;
}

template <int R>
const void* by_kind(int kind, bool kahan, int form) {
  if (kind == PAIR_RK4_A) return by_form<R, PAIR_RK4_A, false>(form);
  if (kind == PAIR_RK4_B)
    return kahan ? by_form<R, PAIR_RK4_B, true>(form) : by_form<R, PAIR_RK4_B, false>(form);
  return kahan ? by_form<R, PAIR_RK2, true>(form) : by_form<R, PAIR_RK2, false>(form);
}

}  // namespace

const void* pair_fn_f32(int R, int kind, bool kahan, int form) {
  return R == 1 ? by_kind<1>(kind, kahan, form) : by_kind<2>(kind, kahan, form);
}

const void* pair_kernel_fn(int es, int R, int kind, bool kahan, int form, bool batch) {
  if (batch) return pair_fn_batch(es, R, kind, kahan, form);
  return es == 8 ? pair_fn_f32(R, kind, kahan, form) : pair_fn_f64(R, kind, form);
}

}  // namespace gpe
