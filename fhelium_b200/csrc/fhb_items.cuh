// Key switches of ciphertexts at mixed levels, driven by a device table of
// item descriptors: every stage is one launch over all items, whatever their
// levels, instead of one launch sequence per level.
//
// An item is one ciphertext (batch 1) with its own operation:
//   kind 0  HMult + relinearise + rescale of a (lhs) and b (rhs), both
//           [2, L, N] coefficient/standard, with the relinearisation key;
//   kind 1  rotation of a [2, L, N] coefficient/standard by its own Galois
//           element with its own rotation key.
// The stages mirror the fused batch path (forward NTT of the operands, the
// tensor product, the inverse NTT of d2, ModUp digits, the key-switch core
// with c0, c1 folded in for relinearisation, ModDown with the rescale or
// with sigma_g(c0)), and use the same building blocks, so every result is
// integer-equal to the per-level batch calls.  Work lists of (item, row)
// units map the transform kernels' blocks to items; the element-wise kernels
// take the item from the grid's z dimension.
#pragma once
#include "fhb_kernels.cuh"
#include "fhb_moddown.cuh"
#include "fhb_pass.cuh"

namespace fhb {

struct KsItem {
  int32_t kind;         // 0: HMult + relinearise + rescale, 1: rotation
  int32_t level;
  uint32_t galois;      // rotation: Galois element of the step; 1 for HMult
  uint32_t check;       // item_check() of the other fields, written by the planner
  const void* a;        // [2, L, N] coefficient/standard (lhs, or the rotated ciphertext)
  const void* b;        // HMult rhs [2, L, N] coefficient/standard; null for a rotation
  const void* key;      // [D, 2, QP0, N] NTT/Montgomery key
  void* out;            // HMult [2, L - 1, N]; rotation [2, L, N]; coefficient/standard
  void* ab;             // scratch: HMult [2 operands][2][L][N] NTT/Montgomery, then (and for rotations)
                        // the core's intermediate [D][L + P][N]
  void* coef;           // scratch: HMult ct3 [3, L, N] NTT/Montgomery
  void* digits;         // scratch: [L, N] ModUp digits
  void* t0;             // scratch: [L + P, N] (d2 in the coefficient domain, then accumulator 0)
  void* t1;             // scratch: [L + P, N] accumulator 1
};

struct ItemUnit {
  int32_t item;
  int32_t row;          // forward NTT: operand * 2 L + component * L + row
};

// Check word of a descriptor: FNV-1a over every field but the check itself.
// The planner validates the fields on the host and stores the word; every
// kernel recomputes it before it uses the item, so a descriptor changed in
// device memory after planning is skipped (and reported) instead of being
// trusted for addressing.
__host__ __device__ __forceinline__ uint32_t fnv_mix(uint32_t h, uint64_t w) {
  h = (h ^ uint32_t(w)) * 16777619u;
  return (h ^ uint32_t(w >> 32)) * 16777619u;
}

__host__ __device__ __forceinline__ uint32_t item_check(const KsItem& it) {
  uint32_t h = 2166136261u;
  h = fnv_mix(h, (uint64_t(uint32_t(it.kind)) << 32) | uint32_t(it.level));
  h = fnv_mix(h, it.galois);
  const void* const ptrs[9] = {it.a, it.b, it.key, it.out, it.ab, it.coef, it.digits, it.t0, it.t1};
#pragma unroll
  for (int i = 0; i < 9; ++i) h = fnv_mix(h, uint64_t(reinterpret_cast<uintptr_t>(ptrs[i])));
  return h;
}

// Status codes of a run (the first one raised is kept).
enum ItemsStatus : int {
  kItemsOk = 0,
  kItemsBadIndex = 1,    // a work list names an item outside the plan
  kItemsBadCheck = 2,    // a descriptor no longer matches its check word
  kItemsBadRow = 3,      // a work-list row outside the item's rows
  kItemsBadKind = 4,     // the HMult list names a rotation
};

struct ItemsView {
  const KsItem* items;
  int32_t count;
  int* status;
};

__device__ __forceinline__ void items_raise(int* status, int code) {
  if (*reinterpret_cast<volatile int*>(status) == 0) atomicCAS(status, 0, code);
}

// Fetches item `idx` into `it`; false (status raised) when the index or the
// descriptor is not the planned one.
__device__ __forceinline__ bool items_fetch(const ItemsView& v, int idx, KsItem& it) {
  if (idx < 0 || idx >= v.count) {
    items_raise(v.status, kItemsBadIndex);
    return false;
  }
  it = v.items[idx];
  if (it.check != item_check(it)) {
    items_raise(v.status, kItemsBadCheck);
    return false;
  }
  return true;
}

// Tensor product of the HMult items (k_mul_ntt per item): grid (N / (256 V),
// rows, HMult items), rows past an item's level return.
template <typename T, int V>
__global__ void k_items_mul(ItemsView iv, const int32_t* __restrict__ hmult, int num_q, int log_n,
                            ChainTables<T> tabs) {
  KsItem it;
  if (!items_fetch(iv, hmult[blockIdx.z], it)) return;
  if (it.kind != 0) {
    items_raise(iv.status, kItemsBadKind);
    return;
  }
  const int limbs = num_q - it.level;
  const int row = blockIdx.y;
  const int64_t n = int64_t(1) << log_n;
  const int64_t k = (int64_t(blockIdx.x) * kEwThreads + threadIdx.x) * V;
  if (row >= limbs || k >= n) return;
  const PrimeInfo<T>& pp = tabs.prime[it.level + row];
  const T q = pp.q, ni = pp.neg_inv, tq = pp.twice_q;
  const T* ab = static_cast<const T*>(it.ab);
  const int64_t comp = int64_t(limbs) * n, i = int64_t(row) * n + k;
  const EwVec<T, V> x0 = ew_load<T, V>(ab + i), x1 = ew_load<T, V>(ab + comp + i);
  const EwVec<T, V> y0 = ew_load<T, V>(ab + 2 * comp + i), y1 = ew_load<T, V>(ab + 3 * comp + i);
  EwVec<T, V> d0, d1, d2;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    d0.v[e] = Word<T>::mont(x0.v[e], y0.v[e], q, ni);
    d1.v[e] = csub(Word<T>::mont(x0.v[e], y1.v[e], q, ni) + Word<T>::mont(x1.v[e], y0.v[e], q, ni), tq);
    d2.v[e] = Word<T>::mont(x1.v[e], y1.v[e], q, ni);
  }
  T* out = static_cast<T*>(it.coef);
  ew_store<T, V>(out + i, d0);
  ew_store<T, V>(out + comp + i, d1);
  ew_store<T, V>(out + 2 * comp + i, d2);
}

// ModUp digits of every item (k_modup_digits per item): the source is d2 in
// the coefficient domain (t0) for HMult, c1 through sigma_g for a rotation.
// Grid (N / (256 V), digits, items), digits past an item's level return.
template <typename T, int V, int WIDTH>
__global__ void k_items_modup(ItemsView iv, const LevelTables<T>* __restrict__ levels, int num_q, int log_n,
                              ChainTables<T> tabs) {
  KsItem it;
  if (!items_fetch(iv, int(blockIdx.z), it)) return;
  const LevelTables<T> lt = levels[it.level];
  if (int(blockIdx.y) >= lt.num_digits) return;
  const int64_t n = int64_t(1) << log_n;
  const int64_t k0 = (int64_t(blockIdx.x) * kEwThreads + threadIdx.x) * V;
  if (k0 >= n) return;
  using W = Word<T>;
  const int limbs = num_q - it.level;
  const DigitDesc d = lt.digits[blockIdx.y];
  const TwPair<T>* g = lt.garner + blockIdx.y * kMaxDigitWidth * kMaxDigitWidth;
  const uint32_t gi = (it.kind == 0 || it.galois == 1) ? 0u : galois_inverse_dev(it.galois, log_n);
  const T* src = it.kind == 0 ? static_cast<const T*>(it.t0) : static_cast<const T*>(it.a) + int64_t(limbs) * n;
  T* dst = static_cast<T*>(it.digits);
  EwVec<T, V> dig[WIDTH];
#pragma unroll
  for (int r = 0; r < WIDTH; ++r) {
    if (r >= d.alpha) break;
    const int row = d.prime0 - it.level + r;
    const T q = tabs.prime[d.prime0 + r].q;
    EwVec<T, V> x;
    if (gi == 0) {
      x = ew_load<T, V>(src + row * n + k0);
#pragma unroll
      for (int e = 0; e < V; ++e) x.v[e] = csub(x.v[e], q);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        bool neg = false;
        const int srck = galois_source(int(k0) + e, log_n, gi, neg);
        T y = csub(src[row * n + srck], q);
        x.v[e] = (neg && y) ? q - y : y;
      }
    }
    if (r > 0) {
      const TwPair<T> inv = g[r * kMaxDigitWidth + r];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        T acc = 0;
#pragma unroll
        for (int i = 0; i < r; ++i) {
          const TwPair<T> c = g[r * kMaxDigitWidth + i];
          acc = csub(acc + csub(W::shoup(dig[i].v[e], c.w, c.wp, q), q), q);
        }
        x.v[e] = csub(W::shoup(csub(x.v[e] + q - acc, q), inv.w, inv.wp, q), q);
      }
    }
    dig[r] = x;
    ew_store<T, V>(dst + row * n + k0, x);
  }
}

// ModDown of every item (k_moddown per item): HMult items rescale by the
// leading prime (c0, c1 are already in the accumulators); rotations add
// sigma_g(c0).  Blocks (coefficients, component, group of rows) on x, items on y.
template <typename T, int NP, bool SPLIT>
__global__ void __launch_bounds__(kMdThreads, 2)
k_items_moddown(ItemsView iv, const __grid_constant__ MdArgs<T> args, int groups) {
  __shared__ double staged[md_staged<SPLIT>()];
  KsItem it;
  if (!items_fetch(iv, int(blockIdx.y), it)) return;
  unsigned idx = blockIdx.x;
  const int g = int(idx % unsigned(groups));
  idx /= unsigned(groups);
  const int c = int(idx & 1), k0 = int((idx >> 1) * kMdThreads + threadIdx.x) * 2;
  MdArgs<T> a = args;
  a.level = it.level;
  a.rescale = it.kind == 0 ? 1 : 0;
  const int ql = a.num_q - a.level, out_limbs = ql - a.rescale;
  const bool add = it.kind == 1 && c == 0;
  const uint32_t gi = !add || it.galois == 1 ? 0u : galois_inverse_dev(it.galois, a.log_n);
  moddown_rows<T, NP, SPLIT>(a, static_cast<const T*>(c ? it.t1 : it.t0), add ? static_cast<const T*>(it.a) : nullptr,
                             gi, static_cast<T*>(it.out) + ((int64_t(c) * out_limbs) << a.log_n), k0,
                             ql * g / groups, ql * (g + 1) / groups, staged);
}

// The transform stages take their (item, row) from a work list.  Every thread
// of a block reads the same unit in the column kernels, every half warp its
// own in the row kernels (all warps of one unit have an even number of rows
// of 256 words, so a warp never splits).  Rows of primes below 2^42 (prime id
// < f64_end) run in FP64 arithmetic; their lazy words may differ from the
// integer transform's by q, which the later stages (all modular, canonical at
// the end) do not see.

// Forward NTT of the HMult operands, unit row operand * 2 L + component * L +
// row: coefficient/standard -> NTT/Montgomery (x R), into the item's `ab`.
template <typename T>
__device__ __forceinline__ bool items_forward_unit(const ItemsView& iv, const ItemUnit& u, int num_q, int64_t n,
                                                   KsItem& it, const T*& in, T*& out, int& pid) {
  if (!items_fetch(iv, u.item, it)) return false;
  const int limbs = num_q - it.level;
  if (it.kind != 0) {
    items_raise(iv.status, kItemsBadKind);
    return false;
  }
  if (u.row < 0 || u.row >= 4 * limbs) {
    items_raise(iv.status, kItemsBadRow);
    return false;
  }
  const int op = u.row / (2 * limbs), rem = u.row - op * 2 * limbs;  // rem = component L + row
  pid = it.level + rem % limbs;
  in = static_cast<const T*>(op == 0 ? it.a : it.b) + int64_t(rem) * n;
  out = static_cast<T*>(it.ab) + int64_t(u.row) * n;
  return true;
}

// Inverse NTT of d2 of the HMult items, unit row a Q_l row: NTT/Montgomery ->
// coefficient/standard canonical, into the item's t0.
template <typename T>
__device__ __forceinline__ bool items_inverse_unit(const ItemsView& iv, const ItemUnit& u, int num_q, int64_t n,
                                                   KsItem& it, const T*& in, T*& out, int& pid) {
  if (!items_fetch(iv, u.item, it)) return false;
  const int limbs = num_q - it.level;
  if (it.kind != 0) {
    items_raise(iv.status, kItemsBadKind);
    return false;
  }
  if (u.row < 0 || u.row >= limbs) {
    items_raise(iv.status, kItemsBadRow);
    return false;
  }
  pid = it.level + u.row;
  in = static_cast<const T*>(it.coef) + int64_t(2 * limbs + u.row) * n;
  out = static_cast<T*>(it.t0) + int64_t(u.row) * n;
  return true;
}

template <typename T, int LOGN, bool INVERSE, bool SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(false))
k_items_ntt_columns(ItemsView iv, const ItemUnit* __restrict__ units, int num_q, ChainTables<T> tabs,
                    ChainTables<double> tabs64f, int f64_end) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KsItem it;
  const T* in;
  T* out;
  int pid;
  const ItemUnit u = units[blockIdx.x / G::kTiles];
  const int col0 = int(blockIdx.x % G::kTiles) * G::kCols;
  if constexpr (INVERSE) {
    if (!items_inverse_unit<T>(iv, u, num_q, int64_t(1) << LOGN, it, in, out, pid)) return;
    ntt_columns_inverse<T, LOGN, SPLIT>(out, pid, pid < f64_end, kInvStandard, tabs, tabs64f, col0, smem_raw);
  } else {
    if (!items_forward_unit<T>(iv, u, num_q, int64_t(1) << LOGN, it, in, out, pid)) return;
    ntt_columns<T, LOGN, true, SPLIT>(in, out, pid, pid < f64_end, tabs, tabs64f, col0, smem_raw);
  }
}

template <typename T, int LOGN, bool INVERSE, bool SPLIT>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 5 : 8)
k_items_ntt_rows(ItemsView iv, const ItemUnit* __restrict__ units, int64_t slots, int num_q, ChainTables<T> tabs,
                 ChainTables<double> tabs64f, int f64_end) {
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  __shared__ __align__(16) unsigned char smem[exchange_smem<T>()];
  const int64_t slot = int64_t(blockIdx.x) * kRowSlots + (threadIdx.x >> 4);
  if (slot >= slots) return;
  KsItem it;
  const T* in;
  T* out;
  int pid;
  const ItemUnit u = units[slot / kBlks];
  const int blk = int(slot % kBlks);
  if constexpr (INVERSE) {
    if (!items_inverse_unit<T>(iv, u, num_q, int64_t(1) << LOGN, it, in, out, pid)) return;
    ntt_rows_inverse<T, LOGN, SPLIT>(in, out, pid, pid < f64_end, tabs, tabs64f, blk, smem);
  } else {
    if (!items_forward_unit<T>(iv, u, num_q, int64_t(1) << LOGN, it, in, out, pid)) return;
    ntt_rows<T, LOGN, SPLIT>(out, pid, pid < f64_end, tabs, tabs64f, blk, smem);
  }
}

// Key-switch core of every item: the three launches of fhb_pass.cuh over
// units (item, destination row of Q_l P); the column launch's units name two
// adjacent rows with kItemPair (both in FP64 arithmetic when the form is on).
// For HMult items the NTT-domain ct3 is folded in (c0, c1 as P c_k, own-digit
// rows from c2).
constexpr int32_t kItemPair = 1 << 24;
constexpr int32_t kItemNone = -1;  // fills the column launch's list

// False (status raised) for a unit outside its item's rows.
__device__ __forceinline__ bool items_core_unit(const ItemsView& iv, int item, int row, int rows_named, int num_q,
                                                int num_p, KsItem& it) {
  if (!items_fetch(iv, item, it)) return false;
  if (row < 0 || row + rows_named > num_q - it.level + num_p) {
    items_raise(iv.status, kItemsBadRow);
    return false;
  }
  return true;
}

template <typename T>
struct ItemsCore {
  const LevelTables<T>* levels;
  int num_q, num_p, ext_digits, f64_end;
  ChainTables<T> tabs;
  ChainTables<double> tabs64f;
  const TwPair<double>* ext64f;
  // The item as a batch of one, every row's intermediate in `ab`.
  __device__ __forceinline__ KsPass<T> pass(const KsItem& it, int64_t n) const {
    KsPass<T> k;
    k.digits = static_cast<const T*>(it.digits);
    k.y = static_cast<T*>(it.ab);
    k.key = static_cast<const T*>(it.key);
    k.item_keys = nullptr;
    k.acc0 = static_cast<T*>(it.t0), k.acc1 = static_cast<T*>(it.t1);
    k.q_limbs = num_q - it.level, k.qp_limbs = k.q_limbs + num_p, k.level = it.level, k.qp0 = num_q + num_p;
    k.ct3 = it.kind == 0 ? static_cast<const T*>(it.coef) : nullptr;
    k.ct3_stride = int64_t(k.q_limbs) * n;
    k.batch = k.y_batch = k.by_row = k.terms = 1;
    k.keys_by_term = 0;
    k.y_rows = k.qp_limbs;
    k.f_lo = k.f_cnt = k.i_lo = k.i_cnt = 0;
    k.ext_digits = ext_digits, k.f64_end = f64_end;
    k.tabs = tabs, k.lt = levels[it.level], k.tabs64f = tabs64f, k.ext64f = ext64f;
    return k;
  }
};

// The item of a block's unit as key-switch arguments in shared memory (every
// thread of a block works on one unit: a polynomial has a multiple of
// kRowSlots rows of 256 words).  One thread fetches and checks the
// descriptor; null (status raised) for a unit that is not the plan's.
template <typename T>
__device__ __forceinline__ const KsPass<T>* items_core_pass(const ItemsView& iv, int item, int row, int rows_named,
                                                            const ItemsCore<T>& core, int64_t n) {
  __shared__ __align__(16) unsigned char held[sizeof(KsPass<T>)];
  __shared__ bool ok;
  if (threadIdx.x == 0) {
    KsItem it;
    ok = items_core_unit(iv, item, row, rows_named, core.num_q, core.num_p, it);
    if (ok) *reinterpret_cast<KsPass<T>*>(held) = core.pass(it, n);
  }
  __syncthreads();
  return ok ? reinterpret_cast<const KsPass<T>*>(held) : nullptr;
}

// Blocks (unit, column tile, digit), digits fastest; digits past an item's level return.
template <typename T, int LOGN, bool SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(SPLIT))
k_items_core_columns(ItemsView iv, const ItemUnit* __restrict__ units, int max_digits,
                     const __grid_constant__ ItemsCore<T> core) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned idx = blockIdx.x;
  const int a = int(idx % unsigned(max_digits));
  idx /= unsigned(max_digits);
  const int col0 = int(idx % G::kTiles) * G::kCols;
  const ItemUnit u = units[idx / G::kTiles];
  if (u.item == kItemNone && u.row == kItemNone) return;
  const int named = u.row >= kItemPair ? 2 : 1, j0 = u.row >= kItemPair ? u.row - kItemPair : u.row;
  const KsPass<T>* held = items_core_pass(iv, u.item, j0, named, core, int64_t(1) << LOGN);
  if (!held) return;
  const KsPass<T>& k = *held;
  if (a >= k.lt.num_digits) return;
  if constexpr (SPLIT) {
    if (k.level + j0 < core.f64_end) {
      const bool two = named == 2 && k.level + j0 + 1 < core.f64_end;
      const DigitDesc d = k.lt.digits[a];
      ks_columns_f64<LOGN, false, false>(k, a, 0, col0, j0, j0 + 1, !ks_own(k, d, j0), two && !ks_own(k, d, j0 + 1),
                                  smem_raw);
      return;
    }
  }
  for (int i = 0; i < named; ++i) {
    if (i) __syncthreads();
    ks_columns_int<T, LOGN, false>(k, a, 0, col0, j0 + i, smem_raw);
  }
}

template <typename T, int LOGN, bool SPLIT>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 3 : 4)
k_items_core_rows(ItemsView iv, const ItemUnit* __restrict__ units, int64_t slots,
                  const __grid_constant__ ItemsCore<T> core) {
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  __shared__ __align__(16) unsigned char smem[row_smem<T>()];
  static_assert(kBlks % kRowSlots == 0, "a block's rows belong to one unit");
  const int64_t slot = int64_t(blockIdx.x) * kRowSlots + (threadIdx.x >> 4);
  if (slot >= slots) return;  // whole blocks
  const ItemUnit u = units[slot / kBlks];
  const int blk = int(slot % kBlks);
  const KsPass<T>* held = items_core_pass(iv, u.item, u.row, 1, core, int64_t(1) << LOGN);
  if (!held) return;
  const KsPass<T>& k = *held;
  if constexpr (SPLIT) {
    if (k.level + u.row < core.f64_end) {
      ks_rows_f64<LOGN, false, false>(k, u.row, 0, blk, smem);
      return;
    }
  }
  ks_rows_int<T, LOGN, false>(k, u.row, 0, blk, smem);
}

// Blocks (unit, component, column tile).
template <typename T, int LOGN, bool SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(false))
k_items_core_columns_inverse(ItemsView iv, const ItemUnit* __restrict__ units,
                             const __grid_constant__ ItemsCore<T> core) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned idx = blockIdx.x;
  const int col0 = int(idx % G::kTiles) * G::kCols;
  idx /= G::kTiles;
  const ItemUnit u = units[idx / 2];
  KsItem it;
  if (!items_core_unit(iv, u.item, u.row, 1, core.num_q, core.num_p, it)) return;
  T* z = static_cast<T*>(idx & 1 ? it.t1 : it.t0) + (int64_t(u.row) << LOGN);
  const int pid = it.level + u.row;
  ks_columns_inverse<T, LOGN, SPLIT>(z, pid, SPLIT && pid < core.f64_end, core.tabs, core.tabs64f, col0, smem_raw);
}

}  // namespace fhb
