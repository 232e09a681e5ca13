// Declarations of the per-(word, LOGN) cluster launchers; definitions in
// fhb_runners.cuh, instantiated in fhb_inst_logn.cu (one object per LOGN).
#pragma once
#include <cuda_runtime.h>

#include "fhb_context.h"

namespace fhb {
template <typename T, int LOGN>
int run_forward(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, bool mont,
                cudaStream_t st);
template <typename T, int LOGN>
int run_inverse(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, int kind,
                cudaStream_t st);
template <typename T, int LOGN>
int run_mul_coef(const Context& c, const void* a, const void* b, void* out, int64_t batch, int level,
                 cudaStream_t st);
template <typename T, int LOGN>
int run_ks_core(const Context& c, const void* digits, const void* key, void* acc0, void* acc1, int64_t batch,
                int level, cudaStream_t st, const uint64_t* item_keys, const void* ct3, bool pre,
                int64_t ct3_pitch = 0);
// The key-switch core as launches of column and block stages (fhb_pass.cuh).
// pre: `y` holds the extensions [D_l][B][QP_l][N] already (all rows in one
// go).  Otherwise `y` has room for y_words words (at least one ciphertext's
// digits of one row, ks_pass_min_words) and rows are processed in as few
// groups as that allows.
template <typename T, int LOGN>
int run_ks_pass(const Context& c, const void* digits, void* y, int64_t y_words, const void* key, void* acc0,
                void* acc1, int64_t batch, int level, cudaStream_t st, const uint64_t* item_keys, const void* ct3,
                bool pre, int64_t ct3_pitch = 0);
template <typename T, int LOGN>
int run_ks_sum(const Context& c, const void* digits, const uint64_t* key_ptrs, void* acc0, void* acc1, int giants,
               int64_t batch, int level, cudaStream_t st, bool pre);
// The sum as launches of column and block stages; `y` as for run_ks_pass.
template <typename T, int LOGN>
int run_ks_sum_pass(const Context& c, const void* digits, void* y, int64_t y_words, const uint64_t* key_ptrs,
                    void* acc0, void* acc1, int terms, int64_t batch, int level, cudaStream_t st, bool pre);
// Mixed-level item stages: 0 = forward NTT of the HMult operands, 1 =
// inverse NTT of d2, 2 = key-switch core; `count` units of `units`.  Stage 2
// also takes the column launch's own list (pairs of rows) and the largest
// digit count of the items.
template <typename T, int LOGN>
int run_items(const Context& c, int stage, const void* items, int item_count, int* status, const void* units,
              int64_t count, cudaStream_t st, const void* column_units = nullptr, int64_t column_count = 0,
              int max_digits = 0);
template <typename T, int LOGN>
int run_prepare(const Context& c, const void* digits, void* prepared, int64_t batch, int level, cudaStream_t st);
template <typename T, int LOGN>
int run_apply_prepared(const Context& c, const void* prepared, const void* key, void* acc0, void* acc1,
                       int64_t batch, int level, uint32_t galois, cudaStream_t st);
}  // namespace fhb
