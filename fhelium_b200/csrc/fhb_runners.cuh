// Cluster launchers for the NTT-based kernels.  Each is explicitly
// instantiated per LOGN in its own translation unit (fhb_inst_logn.cu), so
// the kernel templates compile in parallel.
#pragma once
#include <algorithm>
#include "fhb_items.cuh"
#include "fhb_kernels.cuh"
#include "fhb_pass.cuh"

namespace fhb {

// Rows [row_start, row_start + rows) of a transform whose leading k rows
// have primes below 2^42 and may run in FP64 arithmetic (0 when the
// context has no FP64 tables or the form is switched off).
inline int f64_rows(const Context& c, int row_start, int rows) {
  if (!c.f64_core || !c.f64_tables_ok) return 0;
  return std::max(0, std::min(rows, c.f64_prime_end - row_start));
}

// FP64 form of the chain's leading Q rows, how many of them, and its tables.
// FHB_TUNE_F64_CORE is the narrow rows' switch: it reads 0 on chains without
// them, and a caller that puts back what it read must change nothing there.
struct F64Form {
  int form, end;
  const ChainTables<double>* tabs;
};
inline F64Form f64_form(const Context& c) {
  if (c.f64_core && c.f64_tables_ok) return {kNarrowF64, c.f64_prime_end, &c.t64f};
  if (c.wide_tables_ok) return {kWideF64, c.wide_prime_end, &c.t64w};
  return {kNoF64, 0, &c.t64f};
}

template <typename T, int LOGN, int EPT = 0, typename... KArgs, typename... Args>
int launch_cluster(void (*kernel)(KArgs...), int64_t polys, size_t smem, cudaStream_t stream, Args... args) {
  using G = NttGeom<T, LOGN, EPT>;
  if (polys <= 0) return 0;
  if (polys * G::kC > 0x7fffffffLL) return fail(-6, "too many polynomials for one launch");
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), int(smem));
  if (rc != 0) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(polys * G::kC));
  cfg.blockDim = dim3(G::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = G::kC;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = G::kC > 1 ? 1 : 0;
  return cuda_status(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...), "cluster launch");
}

template <typename... KArgs, typename... Args>
int launch_blocks(void (*kernel)(KArgs...), int64_t blocks, int threads, size_t smem, cudaStream_t stream,
                  Args... args) {
  if (blocks <= 0) return 0;
  if (blocks > 0x7fffffffLL) return fail(-6, "too many blocks for one launch");
  if (smem > 48 * 1024) {
    const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), int(smem));
    if (rc != 0) return rc;
  }
  kernel<<<unsigned(blocks), unsigned(threads), smem, stream>>>(static_cast<KArgs>(args)...);
  return cuda_status(cudaGetLastError(), "pass launch");
}

template <typename T, int LOGN>
constexpr size_t ntt_smem() {
  return size_t(NttGeom<T, LOGN>::kSmemElems) * sizeof(T);
}

// ---- per (T, LOGN) launchers --------------------------------------------
// The standalone transforms run as two launches (fhb_pass.cuh) unless the
// context's tuning value for the direction is 16: one cluster per polynomial
// with 16 residues per thread.  (0.40 against 0.86 ms forward for 12 x 2 x 35
// int64 rows of N = 2^16, 0.68 against 1.72 ms inverse for 48 x 2 x 25 int32
// rows; the autotuner times both.)
template <typename T, int LOGN, int EPT>
int run_forward_e(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, bool mont,
                  cudaStream_t st) {
  // the leading rows of primes below 2^42 in FP64 arithmetic (int64 chains), same launch
  const int k = sizeof(T) == 8 ? f64_rows(c, row_start, rows) : 0;
  auto launch = [&](auto kern) {
    return launch_cluster<T, LOGN, EPT>(kern, polys, ntt_smem<T, LOGN>(), st, (const T*)in, (T*)out, rows, row_start,
                                        tables<T>(c), c.t64f, k);
  };
  if constexpr (sizeof(T) == 8) {
    if (k > 0)
      return mont ? launch(k_ntt_forward<T, LOGN, false, EPT, true>) : launch(k_ntt_forward<T, LOGN, true, EPT, true>);
  }
  return mont ? launch(k_ntt_forward<T, LOGN, false, EPT>) : launch(k_ntt_forward<T, LOGN, true, EPT>);
}

// Columns then rows of 256 words, or the reverse, the intermediate in `out`.
template <typename T, int LOGN, int SPLIT>
int run_forward_passes(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, bool mont,
                       int k, cudaStream_t st) {
  using G = ColGeom<T, LOGN>;
  auto columns = [&](auto kern) {
    return launch_blocks(kern, polys * G::kTiles, G::kThreads, G::smem_bytes(), st, (const T*)in, (T*)out, rows,
                         row_start, tables<T>(c), c.t64f, k);
  };
  const int rc = mont ? columns(k_ntt_columns<T, LOGN, false, SPLIT>) : columns(k_ntt_columns<T, LOGN, true, SPLIT>);
  if (rc != 0) return rc;
  const int64_t slots = polys << (LOGN - kBlkLog);
  return launch_blocks(k_ntt_rows<T, LOGN, SPLIT>, (slots + kRowSlots - 1) / kRowSlots, kRowThreads, 0, st, (T*)out,
                       slots, rows, row_start, tables<T>(c), c.t64f, k);
}

template <typename T, int LOGN, int SPLIT>
int run_inverse_passes(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, int kind,
                       int k, cudaStream_t st, const ChainTables<double>& tabs64f) {
  using G = ColGeom<T, LOGN>;
  const int64_t slots = polys << (LOGN - kBlkLog);
  const int rc = launch_blocks(k_ntt_rows_inverse<T, LOGN, SPLIT>, (slots + kRowSlots - 1) / kRowSlots, kRowThreads, 0,
                               st, (const T*)in, (T*)out, slots, rows, row_start, tables<T>(c), tabs64f, k);
  if (rc != 0) return rc;
  return launch_blocks(k_ntt_columns_inverse<T, LOGN, SPLIT>, polys * G::kTiles, G::kThreads, G::smem_bytes(), st,
                       (T*)out, rows, row_start, kind, tables<T>(c), tabs64f, k);
}

template <typename T, int LOGN>
int run_forward(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start,
                bool mont, cudaStream_t st) {
  if (c.ntt_ept_fwd != 16) {
    if constexpr (sizeof(T) == 8) {
      const int k = f64_rows(c, row_start, rows);
      if (k > 0) return run_forward_passes<T, LOGN, kNarrowF64>(c, in, out, polys, rows, row_start, mont, k, st);
    }
    return run_forward_passes<T, LOGN, kNoF64>(c, in, out, polys, rows, row_start, mont, 0, st);
  }
  return run_forward_e<T, LOGN, 16>(c, in, out, polys, rows, row_start, mont, st);
}

template <typename T, int LOGN, int EPT>
int run_inverse_e(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, int kind,
                  cudaStream_t st) {
  const int k = sizeof(T) == 8 ? f64_rows(c, row_start, rows) : 0;
  auto launch = [&](auto kern) {
    return launch_cluster<T, LOGN, EPT>(kern, polys, ntt_smem<T, LOGN>(), st, (const T*)in, (T*)out, rows, row_start,
                                        kind, tables<T>(c), c.t64f, k);
  };
  if constexpr (sizeof(T) == 8) {
    if (k > 0) return launch(k_ntt_inverse<T, LOGN, EPT, true>);
  }
  return launch(k_ntt_inverse<T, LOGN, EPT>);
}

template <typename T, int LOGN>
int run_inverse(const Context& c, const void* in, void* out, int64_t polys, int rows, int row_start, int kind,
                cudaStream_t st) {
  if (c.ntt_ept_inv != 16) {
    if constexpr (sizeof(T) == 8) {
      // the wide rows' words are canonical, so they take the canonical kinds only
      const F64Form f = f64_form(c);
      const int k = std::max(0, std::min(rows, f.end - row_start));
      if (k > 0 && f.form == kNarrowF64)
        return run_inverse_passes<T, LOGN, kNarrowF64>(c, in, out, polys, rows, row_start, kind, k, st, *f.tabs);
      if (k > 0 && f.form == kWideF64 && kind >= kInvStandard)
        return run_inverse_passes<T, LOGN, kWideF64>(c, in, out, polys, rows, row_start, kind, k, st, *f.tabs);
    }
    return run_inverse_passes<T, LOGN, kNoF64>(c, in, out, polys, rows, row_start, kind, 0, st, c.t64f);
  }
  return run_inverse_e<T, LOGN, 16>(c, in, out, polys, rows, row_start, kind, st);
}

template <typename T, int LOGN>
int run_mul_coef(const Context& c, const void* a, const void* b, void* out, int64_t batch, int level,
                 cudaStream_t st) {
  const int limbs = c.num_q - level;
  const int64_t polys = 3 * batch * limbs;
  if (c.ntt_ept_inv == 16)
    return launch_cluster<T, LOGN, 16>(k_mul_to_coefficient<T, LOGN, 16>, polys, ntt_smem<T, LOGN>(), st,
                                       (const T*)a, (const T*)b, (T*)out, batch, limbs, level, tables<T>(c));
  return launch_cluster<T, LOGN>(k_mul_to_coefficient<T, LOGN>, polys, ntt_smem<T, LOGN>(), st, (const T*)a,
                                 (const T*)b, (T*)out, batch, limbs, level, tables<T>(c));
}

template <typename T, int LOGN>
int run_ks_core(const Context& c, const void* digits, const void* key, void* acc0, void* acc1, int64_t batch,
                int level, cudaStream_t st, const uint64_t* item_keys, const void* ct3, bool pre,
                int64_t ct3_pitch) {
  const int ql = c.num_q - level, qpl = ql + c.num_p;
  if (ct3_pitch <= 0) ct3_pitch = batch * ql * int64_t(c.n());  // component pitch of ct3 [3, batch, L, N]
  const auto* ik = reinterpret_cast<const unsigned long long*>(item_keys);
  auto launch_int = [&](auto kern) {
    return launch_cluster<T, LOGN>(kern, batch * qpl, KsAcc<T, LOGN>::smem_bytes(), st, (const T*)digits,
                                   (const T*)key, (T*)acc0, (T*)acc1, batch, ql, qpl, level, c.qp(), c.ks_order, ik,
                                   (const T*)ct3, ct3_pitch, tables<T>(c), level_tables<T>(c, level));
  };
  if constexpr (sizeof(T) == 8) {
    if constexpr (KsAcc<double, LOGN>::kSmem) {
      static_assert(KsAcc<double, LOGN>::smem_bytes() == KsAcc<T, LOGN>::smem_bytes(), "one smem size for both");
      // the leading Q rows whose primes are below 2^42 in FP64 arithmetic,
      // the rest (wider Q primes, the P rows) on the integer body, one launch
      const int f64_rows = c.f64_core && c.f64_tables_ok ? std::max(0, std::min(ql, c.f64_prime_end - level)) : 0;
      if (f64_rows > 0) {
        auto launch_split = [&](auto kern) {
          return launch_cluster<double, LOGN>(kern, batch * qpl, KsAcc<double, LOGN>::smem_bytes(), st,
                                              (const uint64_t*)digits, (const uint64_t*)key, (uint64_t*)acc0,
                                              (uint64_t*)acc1, batch, ql, qpl, level, c.qp(), c.ks_order, ik,
                                              (const uint64_t*)ct3, ct3_pitch, tables<uint64_t>(c),
                                              level_tables<uint64_t>(c, level), c.t64f, f64_rows, c.ext64f,
                                              c.ext64f_digits, c.f64_prime_end);
        };
        return pre ? launch_split(k_keyswitch_core_split<LOGN, true>)
                   : launch_split(k_keyswitch_core_split<LOGN, false>);
      }
    }
    if (pre) return launch_int(k_keyswitch_core<T, LOGN, true>);  // extensions of the tensor-core form
  } else {
    if (pre) return fail(-7, "the tensor-core basis conversion needs an int64 context");
  }
  return launch_int(k_keyswitch_core<T, LOGN>);
}

// What the pass kernels of one level share; all rows in flight.
template <typename T>
KsPass<T> ks_pass_args(const Context& c, int level) {
  KsPass<T> k = {};
  k.q_limbs = c.num_q - level, k.qp_limbs = k.q_limbs + c.num_p, k.level = level, k.qp0 = c.qp();
  const F64Form f = f64_form(c);
  k.f_cnt = sizeof(T) == 8 ? std::max(0, std::min(k.q_limbs, f.end - level)) : 0;
  k.i_lo = k.f_cnt, k.i_cnt = k.qp_limbs - k.f_cnt;
  k.terms = 1;
  k.ext_digits = c.ext64f_digits, k.f64_end = c.f64_prime_end;
  k.tabs = tables<T>(c), k.lt = level_tables<T>(c, level);
  k.tabs64f = *f.tabs, k.ext64f = c.ext64f;
  return k;
}

// Whether the rows launch shares a row's digits among a block's warps (k_ks_rows,
// SHARED): with three digits or more and at most as many half warps as fill
// the GPU once without sharing (half as many 32-bit ones).  Below that line
// warps would be missing; above it the sharing costs its exchange.  Whole
// HMult, without / with (us), by half warps: N = 2^14 (9 rows) 576 105/74,
// 1728 155/121, 2880 177/155, 4608 210/217; N = 2^16, one ciphertext, four
// digits, 3328 193/182, 4096 221/228, two digits, 2048 117/124; 32-bit words
// of N = 2^15 (12 rows) 1536 61/59, 3072 83/87.
template <typename T>
bool shared_rows(int64_t half_warps, int digits) {
  return digits > 2 && half_warps <= 148 * (sizeof(T) == 8 ? 3 : 2) * kRowSlots;
}
inline int64_t rows_blocks(int64_t slots, int rows, bool shared) {
  return slots / (shared ? 2 : kRowSlots) * rows;  // (a polynomial has a multiple of kRowSlots rows of 256 words)
}

// The three launches of one group of rows.
template <typename T, int LOGN, int SPLIT>
int launch_ks_pass(const KsPass<T>& k, int digits, bool pre, cudaStream_t st) {
  using G = ColGeom<T, LOGN>;
  const int64_t units = (k.f_cnt + 1) / 2 + k.i_cnt, blocks = int64_t(digits) * k.batch * units * G::kTiles;
  int rc = pre ? launch_blocks(k_ks_columns<T, LOGN, true, SPLIT>, blocks, G::kThreads, G::smem_bytes(), st, k)
               : launch_blocks(k_ks_columns<T, LOGN, false, SPLIT>, blocks, G::kThreads,
                               ks_columns_smem<T, LOGN>(SPLIT == kNarrowF64), st, k);
  if (rc != 0) return rc;
  const int64_t slots = (int64_t(k.batch) << (LOGN - kBlkLog));
  const bool shared = shared_rows<T>(slots * k.rows(), digits);
  rc = launch_blocks(shared ? k_ks_rows<T, LOGN, SPLIT, true> : k_ks_rows<T, LOGN, SPLIT, false>,
                     rows_blocks(slots, k.rows(), shared), kRowThreads, 0, st, k);
  if (rc != 0) return rc;
  return launch_blocks(k_ks_columns_inverse<T, LOGN, SPLIT>, int64_t(2) * k.batch * k.rows() * G::kTiles, G::kThreads,
                       G::smem_bytes(), st, k);
}

// Launch 1 over the ciphertexts of all terms, then launches 2 and 3 over the sums.
template <typename T, int LOGN, int SPLIT>
int launch_ks_sum(KsPass<T> k, int digits, int terms, bool pre, cudaStream_t st) {
  using G = ColGeom<T, LOGN>;
  const int batch = k.batch;
  k.batch = batch * terms;
  const int64_t units = (k.f_cnt + 1) / 2 + k.i_cnt, blocks = int64_t(digits) * k.batch * units * G::kTiles;
  int rc = pre ? launch_blocks(k_ks_columns<T, LOGN, true, SPLIT>, blocks, G::kThreads, G::smem_bytes(), st, k)
               : launch_blocks(k_ks_columns<T, LOGN, false, SPLIT>, blocks, G::kThreads,
                               ks_columns_smem<T, LOGN>(SPLIT == kNarrowF64), st, k);
  if (rc != 0) return rc;
  k.batch = batch, k.terms = terms;
  const int64_t slots = (int64_t(batch) << (LOGN - kBlkLog));
  const bool shared = terms == 1 && shared_rows<T>(slots * k.rows(), digits);
  rc = launch_blocks(shared ? k_ks_rows<T, LOGN, SPLIT, true> : k_ks_rows<T, LOGN, SPLIT, false>,
                     rows_blocks(slots, k.rows(), shared), kRowThreads, 0, st, k);
  if (rc != 0) return rc;
  return launch_blocks(k_ks_columns_inverse<T, LOGN, SPLIT>, int64_t(2) * batch * k.rows() * G::kTiles, G::kThreads,
                       G::smem_bytes(), st, k);
}

// Sum of the key switches of `terms` x batch ciphertexts, each term with its
// own key, in the groups of rows that `y` has room for (pre: the extensions).
template <typename T, int LOGN>
int run_ks_sum_pass(const Context& c, const void* digits, void* y, int64_t y_words, const uint64_t* key_ptrs,
                    void* acc0, void* acc1, int terms, int64_t batch, int level, cudaStream_t st, bool pre) {
  KsPass<T> k = ks_pass_args<T>(c, level);
  const int qpl = k.qp_limbs, nd = k.lt.num_digits, f64 = k.f_cnt, ints = k.i_cnt;
  const int64_t per_row = int64_t(nd) * terms * batch * c.n();
  if (batch <= 0) return 0;
  if (batch * terms > kMaxPassGroup) return fail(-6, "too many ciphertexts for one launch");
  k.digits = static_cast<const T*>(digits);
  k.y = static_cast<T*>(y);
  k.item_keys = reinterpret_cast<const unsigned long long*>(key_ptrs);
  k.keys_by_term = 1;
  k.acc0 = static_cast<T*>(acc0), k.acc1 = static_cast<T*>(acc1);
  k.by_row = pre, k.batch = int(batch), k.y_batch = int(batch) * terms;
  const int step = pre ? qpl : int(std::min<int64_t>(qpl, y_words / per_row));
  if (step < 1) return fail(-8, "no room for the transform's intermediate");
  for (int lo = 0; lo < qpl; lo += step) {
    const int hi = std::min(qpl, lo + step);
    k.i_lo = f64 + lo * ints / qpl, k.i_cnt = f64 + hi * ints / qpl - k.i_lo;
    k.f_lo = lo - (k.i_lo - f64), k.f_cnt = hi - lo - k.i_cnt;
    k.y_rows = pre ? qpl : hi - lo;
    int rc = 0;
    if constexpr (sizeof(T) == 8) {
      const int form = f64 > 0 ? f64_form(c).form : kNoF64;
      rc = form == kNarrowF64 ? launch_ks_sum<T, LOGN, kNarrowF64>(k, nd, terms, pre, st)
           : form == kWideF64 ? launch_ks_sum<T, LOGN, kWideF64>(k, nd, terms, pre, st)
                              : launch_ks_sum<T, LOGN, kNoF64>(k, nd, terms, pre, st);
    } else {
      if (pre) return fail(-7, "the tensor-core basis conversion needs an int64 context");
      rc = launch_ks_sum<T, LOGN, kNoF64>(k, nd, terms, false, st);
    }
    if (rc != 0) return rc;
  }
  return 0;
}

template <typename T, int LOGN>
int run_ks_pass(const Context& c, const void* digits, void* y, int64_t y_words, const void* key, void* acc0,
                void* acc1, int64_t batch, int level, cudaStream_t st, const uint64_t* item_keys, const void* ct3,
                bool pre, int64_t ct3_pitch) {
  if (batch <= 0) return 0;
  KsPass<T> k = ks_pass_args<T>(c, level);
  const int ql = k.q_limbs, qpl = k.qp_limbs, nd = k.lt.num_digits, f64 = k.f_cnt, ints = k.i_cnt;
  const int64_t n = c.n();
  if (ct3_pitch <= 0) ct3_pitch = batch * ql * n;
  k.y = static_cast<T*>(y);
  k.key = static_cast<const T*>(key);
  k.ct3_stride = ct3_pitch;
  k.by_row = pre;
  // ciphertexts per group: all of them, unless the room holds fewer or the
  // launch would pass the grid's limit
  const int64_t per_row = nd * n;  // words of one ciphertext's row
  int64_t group = std::min(batch, kMaxPassGroup);
  if (!pre) {
    group = std::min(group, y_words / per_row);
    if (group < 1) return fail(-8, "no room for the transform's intermediate");
  }
  for (int64_t b0 = 0; b0 < batch; b0 += group) {
    k.batch = int(std::min(group, batch - b0));
    k.y_batch = pre ? int(batch) : k.batch;
    if (pre) k.y = static_cast<T*>(y) + b0 * qpl * n;
    k.digits = static_cast<const T*>(digits) + b0 * ql * n;
    k.acc0 = static_cast<T*>(acc0) + b0 * qpl * n;
    k.acc1 = static_cast<T*>(acc1) + b0 * qpl * n;
    k.ct3 = ct3 ? static_cast<const T*>(ct3) + b0 * ql * n : nullptr;
    if (item_keys) k.item_keys = reinterpret_cast<const unsigned long long*>(item_keys) + b0;
    const int step = pre ? qpl : int(std::min<int64_t>(qpl, y_words / (per_row * k.batch)));
    for (int lo = 0; lo < qpl; lo += step) {
      // rows lo .. hi of the order that spreads the integer rows evenly
      const int hi = std::min(qpl, lo + step);
      k.i_lo = f64 + lo * ints / qpl, k.i_cnt = f64 + hi * ints / qpl - k.i_lo;
      k.f_lo = lo - (k.i_lo - f64), k.f_cnt = hi - lo - k.i_cnt;
      k.y_rows = pre ? qpl : hi - lo;
      int rc = 0;
      if constexpr (sizeof(T) == 8) {
        const int form = f64 > 0 ? f64_form(c).form : kNoF64;
        rc = form == kNarrowF64 ? launch_ks_pass<T, LOGN, kNarrowF64>(k, nd, pre, st)
             : form == kWideF64 ? launch_ks_pass<T, LOGN, kWideF64>(k, nd, pre, st)
                                : launch_ks_pass<T, LOGN, kNoF64>(k, nd, pre, st);
      } else {
        if (pre) return fail(-7, "the tensor-core basis conversion needs an int64 context");
        rc = launch_ks_pass<T, LOGN, kNoF64>(k, nd, false, st);
      }
      if (rc != 0) return rc;
    }
  }
  return 0;
}

template <typename T, int LOGN>
int run_ks_sum(const Context& c, const void* digits, const uint64_t* key_ptrs, void* acc0, void* acc1, int giants,
               int64_t batch, int level, cudaStream_t st, bool pre) {
  const int ql = c.num_q - level, qpl = ql + c.num_p;
  if (pre) {
    if constexpr (sizeof(T) == 8) {
      return launch_cluster<T, LOGN>(k_keyswitch_sum<T, LOGN, true>, batch * qpl, KsAcc<T, LOGN>::smem_bytes(), st,
                                     (const T*)digits, reinterpret_cast<const unsigned long long*>(key_ptrs),
                                     (T*)acc0, (T*)acc1, giants, batch, ql, qpl, level, c.qp(), c.ks_order,
                                     tables<T>(c), level_tables<T>(c, level));
    } else {
      return fail(-7, "the tensor-core basis conversion needs an int64 context");
    }
  }
  return launch_cluster<T, LOGN>(k_keyswitch_sum<T, LOGN>, batch * qpl, KsAcc<T, LOGN>::smem_bytes(), st,
                                 (const T*)digits, reinterpret_cast<const unsigned long long*>(key_ptrs), (T*)acc0,
                                 (T*)acc1, giants, batch, ql, qpl, level, c.qp(), c.ks_order, tables<T>(c),
                                 level_tables<T>(c, level));
}

// Hoisting stage 1 (fhelium/engine/hybrid_keyswitch.py:373-417): the digits'
// extensions transformed once, [D_l, B, QP_l, N] standard NTT-domain values
// in [0, 2p), as the column launch of the key switch and the row launch of
// the plain transform.
template <typename T, int LOGN>
int run_prepare(const Context& c, const void* digits, void* prepared, int64_t batch, int level,
                cudaStream_t st) {
  KsPass<T> k = ks_pass_args<T>(c, level);
  if (f64_form(c).form == kWideF64) {  // the prepared words are the integer transform's
    k.i_lo = k.f_cnt = 0;
    k.i_cnt = k.qp_limbs;
  }
  const int f64 = k.f_cnt, nd = k.lt.num_digits, qpl = k.qp_limbs;
  const int64_t n = c.n(), units = (k.f_cnt + 1) / 2 + k.i_cnt, polys = int64_t(nd) * batch * qpl;
  k.by_row = 1, k.y_rows = qpl, k.y_batch = int(batch);
  using G = ColGeom<T, LOGN>;
  auto run = [&](auto columns, auto rows, bool split) {
    for (int64_t b0 = 0; b0 < batch; b0 += k.batch) {
      k.batch = int(std::min(batch - b0, kMaxPassGroup));
      k.digits = static_cast<const T*>(digits) + b0 * k.q_limbs * n;
      k.y = static_cast<T*>(prepared) + b0 * qpl * n;
      const int rc = launch_blocks(columns, int64_t(nd) * k.batch * units * G::kTiles, G::kThreads,
                                   ks_columns_smem<T, LOGN>(split), st, k);
      if (rc != 0) return rc;
    }
    const int64_t slots = polys << (LOGN - kBlkLog);
    return launch_blocks(rows, (slots + kRowSlots - 1) / kRowSlots, kRowThreads, 0, st, (T*)prepared, slots, qpl,
                         level, tables<T>(c), c.t64f, f64);
  };
  if constexpr (sizeof(T) == 8) {
    if (f64 > 0) return run(k_ks_columns<T, LOGN, false, kNarrowF64>, k_ntt_rows<T, LOGN, kNarrowF64>, true);
  }
  return run(k_ks_columns<T, LOGN, false, kNoF64>, k_ntt_rows<T, LOGN, kNoF64>, false);
}

template <typename T, int LOGN>
int run_apply_prepared(const Context& c, const void* prepared, const void* key, void* acc0, void* acc1,
                       int64_t batch, int level, uint32_t galois, cudaStream_t st) {
  KsPass<T> k = ks_pass_args<T>(c, level);
  const int64_t n = c.n();
  k.by_row = 1, k.y_rows = k.qp_limbs, k.y_batch = int(batch);
  k.key = static_cast<const T*>(key);
  using G = ColGeom<T, LOGN>;
  auto run = [&](auto rows, auto columns) {
    for (int64_t b0 = 0; b0 < batch; b0 += k.batch) {
      k.batch = int(std::min(batch - b0, kMaxPassGroup));
      k.y = static_cast<T*>(const_cast<void*>(prepared)) + b0 * k.qp_limbs * n;
      k.acc0 = static_cast<T*>(acc0) + b0 * k.qp_limbs * n;
      k.acc1 = static_cast<T*>(acc1) + b0 * k.qp_limbs * n;
      const int64_t slots = int64_t(k.batch) << (LOGN - kBlkLog);
      int rc = launch_blocks(rows, (slots + kRowSlots - 1) / kRowSlots * k.rows(), kRowThreads, 0, st, k,
                             galois == 1 ? 0u : galois);
      if (rc != 0) return rc;
      rc = launch_blocks(columns, int64_t(2) * k.batch * k.rows() * G::kTiles, G::kThreads, G::smem_bytes(), st, k);
      if (rc != 0) return rc;
    }
    return 0;
  };
  if constexpr (sizeof(T) == 8) {
    if (k.f_cnt > 0)
      return f64_form(c).form == kNarrowF64
                 ? run(k_apply_rows<T, LOGN, kNarrowF64>, k_ks_columns_inverse<T, LOGN, kNarrowF64>)
                 : run(k_apply_rows<T, LOGN, kWideF64>, k_ks_columns_inverse<T, LOGN, kWideF64>);
  }
  return run(k_apply_rows<T, LOGN, kNoF64>, k_ks_columns_inverse<T, LOGN, kNoF64>);
}

// ---- mixed-level item stages (fhb_items.cuh) ---------------------------------
template <typename T, int LOGN, int SPLIT>
int run_items_form(const Context& c, int stage, const ItemsView& iv, const ItemUnit* un, int64_t count,
                   const ItemUnit* column_units, int64_t column_count, int max_digits, cudaStream_t st) {
  using G = ColGeom<T, LOGN>;
  const int64_t slots = count << (LOGN - kBlkLog), row_blocks = (slots + kRowSlots - 1) / kRowSlots;
  auto columns = [&](auto kern, int64_t blocks, size_t smem, auto... args) {
    return launch_blocks(kern, blocks, G::kThreads, smem, st, iv, args...);
  };
  auto rows = [&](auto kern, auto... args) {
    return launch_blocks(kern, row_blocks, kRowThreads, 0, st, iv, un, slots, args...);
  };
  if (stage == 0) {
    const int rc = columns(k_items_ntt_columns<T, LOGN, false, SPLIT>, count * G::kTiles, G::smem_bytes(), un, c.num_q,
                           tables<T>(c), c.t64f, c.f64_prime_end);
    return rc ? rc : rows(k_items_ntt_rows<T, LOGN, false, SPLIT>, c.num_q, tables<T>(c), c.t64f, c.f64_prime_end);
  }
  if (stage == 1) {
    const int rc = rows(k_items_ntt_rows<T, LOGN, true, SPLIT>, c.num_q, tables<T>(c), c.t64f, c.f64_prime_end);
    return rc ? rc
              : columns(k_items_ntt_columns<T, LOGN, true, SPLIT>, count * G::kTiles, G::smem_bytes(), un, c.num_q,
                        tables<T>(c), c.t64f, c.f64_prime_end);
  }
  const ItemsCore<T> core{level_tables_dev<T>(c), c.num_q, c.num_p, c.ext64f_digits, c.f64_prime_end, tables<T>(c),
                          c.t64f, c.ext64f};
  int rc = columns(k_items_core_columns<T, LOGN, SPLIT>, column_count * G::kTiles * max_digits,
                   ks_columns_smem<T, LOGN>(SPLIT), column_units, max_digits, core);
  if (rc != 0) return rc;
  rc = rows(k_items_core_rows<T, LOGN, SPLIT>, core);
  if (rc != 0) return rc;
  return columns(k_items_core_columns_inverse<T, LOGN, SPLIT>, 2 * count * G::kTiles, G::smem_bytes(), un, core);
}

template <typename T, int LOGN>
int run_items(const Context& c, int stage, const void* items, int item_count, int* status, const void* units,
              int64_t count, cudaStream_t st, const void* column_units, int64_t column_count, int max_digits) {
  const ItemsView iv{static_cast<const KsItem*>(items), item_count, status};
  const auto* un = static_cast<const ItemUnit*>(units);
  const auto* cu = static_cast<const ItemUnit*>(column_units);
  // int64 chains with FP64 tables: the rows of primes below 2^42 in FP64 arithmetic
  if constexpr (sizeof(T) == 8) {
    if (c.f64_core && c.f64_tables_ok && c.f64_prime_end > 0)
      return run_items_form<T, LOGN, true>(c, stage, iv, un, count, cu, column_count, max_digits, st);
  }
  return run_items_form<T, LOGN, false>(c, stage, iv, un, count, cu, column_count, max_digits, st);
}

// Explicit instantiation of every runner for one (T, LOGN).
#define FHB_INSTANTIATE_RUNNERS(T, LOGN)                                                                       \
  template int run_forward<T, LOGN>(const Context&, const void*, void*, int64_t, int, int, bool, cudaStream_t);   \
  template int run_inverse<T, LOGN>(const Context&, const void*, void*, int64_t, int, int, int, cudaStream_t);    \
  template int run_mul_coef<T, LOGN>(const Context&, const void*, const void*, void*, int64_t, int, cudaStream_t); \
  template int run_ks_core<T, LOGN>(const Context&, const void*, const void*, void*, void*, int64_t, int,        \
                                    cudaStream_t, const uint64_t*, const void*, bool, int64_t);                 \
  template int run_ks_pass<T, LOGN>(const Context&, const void*, void*, int64_t, const void*, void*, void*, int64_t, int, \
                                    cudaStream_t, const uint64_t*, const void*, bool, int64_t);                 \
  template int run_ks_sum_pass<T, LOGN>(const Context&, const void*, void*, int64_t, const uint64_t*, void*, void*, \
                                        int, int64_t, int, cudaStream_t, bool);                                 \
  template int run_ks_sum<T, LOGN>(const Context&, const void*, const uint64_t*, void*, void*, int, int64_t, int, \
                                   cudaStream_t, bool);                                                         \
  template int run_prepare<T, LOGN>(const Context&, const void*, void*, int64_t, int, cudaStream_t);            \
  template int run_items<T, LOGN>(const Context&, int, const void*, int, int*, const void*, int64_t, cudaStream_t, \
                                  const void*, int64_t, int);                                                                     \
  template int run_apply_prepared<T, LOGN>(const Context&, const void*, const void*, void*, void*, int64_t, int, \
                                           uint32_t, cudaStream_t);

}  // namespace fhb
