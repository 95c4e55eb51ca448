// pair.h -- the entry points of the pair kernels (pair_kernel.cuh), compiled
// in translation units of their own.
#pragma once

namespace gpe {

// Kernel for fields of es bytes per complex, order 2R, pair `kind`
// (PAIR_*), with or without compensation, right-hand-side form, single-run or
// batched; nullptr where none is built (the full form is, for
// single runs in complex64 at order 2).
const void* pair_kernel_fn(int es, int R, int kind, bool kahan, int form, bool batch);

// The parts of it by translation unit.
const void* pair_fn_f32(int R, int kind, bool kahan, int form);
const void* pair_fn_f64(int R, int kind, int form);
const void* pair_fn_batch(int es, int R, int kind, bool kahan, int form);

}  // namespace gpe
