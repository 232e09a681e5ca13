// ModDown by P (device code).
//
// Per coefficient, with e_r the Garner digits of the P part, row i of Q_l
// (prime q) of the result is, fused with the addend and the rescale by the
// leading prime q_0:
//   v_i   = (t_i - sum_r e_r M_r) P^{-1} + add_i                     (mod q)
//   out_i = v_i,  or with rescale  (v_i - v_0) q_0^{-1} + [v_0 > q_0/2]
// which is one sum of products with per-row constants,
//   out_i = t_i A + sum_r e_r B_r + add_i C + v_0 D (+ 1),
//   C = 1 or q_0^{-1},  A = P^{-1} C,  B_r = -M_r A,  D = -C,
// so a row takes num_p + 2 (or 3) products and one reduction.  Equal to the
// sequential divide-by-p_j chain of csrc/ops/ckks/cpu/ckks_cpu.cpp:474-601
// and the nearest-rounded division of csrc/ops/ckks/cpu/ckks_cpu.cpp:203-262:
// every result is the canonical residue of the same value.
//
// Integer rows add the double-width products and reduce once by 2^W (W the
// word's bits; the constants carry 2^W): x < 2^60, c < q keep eleven
// products' sum below q 2^64 (28-bit primes: below q 2^32).  FP64 rows
// (primes below 2^42) split the digits, which reach 60 bits, into 30-bit
// halves with their own constants and add every product exactly on top of
// 1.5 2^88 (ext_chain in fhb_pass.cuh): at most 19 products of less than
// 2^84 (three of them) or 2^72 stay below 2^87.  With a reduction per product
// the kernel was bound by those: 1.93 -> 0.80 ms with the rescale for 32
// ciphertexts of 35 + 4 rows at N = 2^16 (1.02 ms before the FP64 constants
// were staged in shared memory).
#pragma once
#include <algorithm>
#include <type_traits>

#include "fhb_kernels.cuh"

namespace fhb {

// One sum of products modulo a prime.
struct MdSumF64 {
  static constexpr double kBig = 1.5 * 309485009821345068724781056.0;  // 1.5 2^88
  double t = kBig, low = 0.0;
  __device__ __forceinline__ void add(double x, double c) {
    const double next = fma(x, c, t);
    low += fma(x, c, t - next);
    t = next;
  }
  __device__ __forceinline__ double balanced(double q, double qinv) const {  // (-0.51 q, 0.51 q)
    const double h = t - kBig;
    return Word<double>::reduce_bal(fma(-Word<double>::mul_round(h, qinv), q, h) + low, q, qinv);
  }
};
struct MdSum64 {
  unsigned __int128 s = 0;
  __device__ __forceinline__ void add(uint64_t x, uint64_t c) { s += static_cast<unsigned __int128>(x) * c; }
  __device__ __forceinline__ uint64_t reduced(uint64_t q, uint64_t qi) const {  // (0, 2q)
    return uint64_t(s >> 64) - __umul64hi(uint64_t(s) * qi, q) + q;
  }
};
struct MdSum32 {
  uint64_t s = 0;
  __device__ __forceinline__ void add(uint32_t x, uint32_t c) { s += static_cast<uint64_t>(x) * c; }
  __device__ __forceinline__ uint32_t reduced(uint32_t q, uint32_t qi) const {
    return uint32_t(s >> 32) - __umulhi(uint32_t(s) * qi, q) + q;
  }
};
template <typename T>
using MdSum = std::conditional_t<sizeof(T) == 8, MdSum64, MdSum32>;

constexpr int kMdThreads = 256;  // two coefficients each

template <typename T>
struct MdArgs {
  int log_n, level, num_q, num_p, rescale, f64_end;
  ChainTables<T> tabs;
  MdTables<T> md;
};

// The FP64 rows' constants of one block in shared memory (q, 1/q, then the
// table's): read from device memory they cost a row thirteen dependent loads,
// more latency than its products cover.  At most kMdRows rows per block.
constexpr int kMdRows = 96;
constexpr int kMdStaged = kMdDoubles + 2;
template <bool SPLIT>
constexpr int md_staged() {
  return SPLIT ? kMdRows * kMdStaged : 1;
}

// Rows [i0, i1) of Q_l at coefficients k0, k0 + 1 of one component: t
// [QP_l][N], add [Q_l][N] or null (through sigma_g with inverse gi when gi is
// not 0), out [Q_l (- 1)][N].  NP = num_p (8: any).  `staged`: md_staged
// doubles of shared memory; every thread of the block calls this.
template <typename T, int NP, bool SPLIT>
__device__ __forceinline__ void moddown_rows(const MdArgs<T>& a, const T* __restrict__ t, const T* __restrict__ add,
                                             uint32_t gi, T* __restrict__ out, int k0, int i0, int i1,
                                             double* staged) {
  using W = Word<T>;
  struct alignas(2 * sizeof(T)) Two {
    T v[2];
  };
  const int log_n = a.log_n, ql = a.num_q - a.level, qp0 = a.num_q + a.num_p;
  auto two = [&](const T* row) {
    return *reinterpret_cast<const Two*>(row + k0);
  };
  const int64_t base = int64_t(a.rescale ? a.level + 1 : 0) * qp0 + a.level;  // table 0: no rescale
  const int first = i0;
  if constexpr (SPLIT) {
    constexpr int kUsed = 5 + 2 * NP;
    const int rows = min(i1, a.f64_end - a.level) - first;
    for (int w = threadIdx.x; w < rows * kUsed; w += kMdThreads) {
      const int r = w / kUsed, c = w % kUsed, pid = a.level + first + r;
      staged[r * kMdStaged + c] = c == 0   ? a.md.prime[pid].q
                                  : c == 1 ? a.md.prime[pid].one_s
                                           : a.md.f[(base + first + r) * kMdDoubles + c - 2];
    }
    __syncthreads();
  }
  // Garner digits of the P part
  T e[NP][2];
#pragma unroll
  for (int r = 0; r < NP; ++r) {
    if (NP == kMaxDigitWidth && r >= a.num_p) {
      e[r][0] = e[r][1] = 0;
      continue;
    }
    const T q = a.tabs.prime[a.num_q + r].q;
    const Two x = two(t + (int64_t(ql + r) << log_n));
    const TwPair<T> inv = a.tabs.p_garner[r * kMaxDigitWidth + r];
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      T acc = 0, y = x.v[z];
#pragma unroll
      for (int i = 0; i < r; ++i) {
        const TwPair<T> g = a.tabs.p_garner[r * kMaxDigitWidth + i];
        acc = csub(acc + csub(W::shoup(e[i][z], g.w, g.wp, q), q), q);
      }
      if (r > 0) y = csub(W::shoup(csub(y + q - acc, q), inv.w, inv.wp, q), q);
      e[r][z] = y;
    }
  }
  int ak[2] = {k0, k0 + 1};
  bool neg[2] = {false, false};
  if (add && gi) {
#pragma unroll
    for (int z = 0; z < 2; ++z) ak[z] = galois_source(k0 + z, log_n, gi, neg[z]);
  }
  auto addend = [&](int i, int z, T q) {
    T x = csub(add[(int64_t(i) << log_n) + ak[z]], q);
    return neg[z] && x ? q - x : x;
  };
  // one row's canonical value; c: its constants; v0 added through D unless null
  auto row_int = [&](int i, const T* __restrict__ c, const T* v0, T (&r)[2]) {
    const PrimeInfo<T>& p = a.tabs.prime[a.level + i];
    const T q = p.q, x = T(0) - p.neg_inv, qi = x * (T(2) - q * x);  // q^{-1} mod 2^W
    const Two tv = two(t + (int64_t(i) << log_n));
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      MdSum<T> s;
      s.add(tv.v[z], c[0]);
      if (add) s.add(addend(i, z, q), c[1]);
      if (v0) s.add(v0[z], c[2]);
#pragma unroll
      for (int d = 0; d < NP; ++d)
        if (NP != kMaxDigitWidth || d < a.num_p) s.add(e[d][z], c[3 + d]);
      r[z] = csub(s.reduced(q, qi), q);
    }
  };
  double eh[SPLIT ? NP : 1][2], el[SPLIT ? NP : 1][2];
  if constexpr (SPLIT) {
#pragma unroll
    for (int d = 0; d < NP; ++d)
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        eh[d][z] = Word<double>::from_word(e[d][z] >> 30);
        el[d][z] = Word<double>::from_word(e[d][z] & ((uint64_t{1} << 30) - 1));
      }
  }
  // the balanced value, not yet canonical
  auto row_f64 = [&](int i, const Two& tv, const double* c, const double* v0, double q, double qinv, double (&r)[2]) {
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      MdSumF64 s;
      s.add(Word<double>::from_word(tv.v[z]), c[0]);
      if (add) s.add(Word<double>::from_word(addend(i, z, a.tabs.prime[a.level + i].q)), c[1]);
      if (v0) s.add(v0[z], c[2]);
#pragma unroll
      for (int d = 0; d < NP; ++d)
        if (NP != kMaxDigitWidth || d < a.num_p) {
          s.add(eh[d][z], c[3 + 2 * d]);
          s.add(el[d][z], c[4 + 2 * d]);
        }
      r[z] = s.balanced(q, qinv);
    }
  };
  T v0[2] = {0, 0};
  double v0d[2] = {0.0, 0.0};
  T bit[2] = {0, 0};
  if (a.rescale) {  // v_0, by the constants without rescale
    if (SPLIT && a.level < a.f64_end) {
      if constexpr (SPLIT) {
        const double q = a.md.prime[a.level].q, qinv = a.md.prime[a.level].one_s;
        row_f64(0, two(t), a.md.f + int64_t(a.level) * kMdDoubles, nullptr, q, qinv, v0d);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          if (v0d[z] < 0.0) v0d[z] += q;
          v0[z] = Word<double>::to_word(v0d[z]);
        }
      }
    } else {
      row_int(0, a.md.w + int64_t(a.level) * kMdWords, nullptr, v0);
    }
    const T half = a.tabs.prime[a.level].q >> 1;
#pragma unroll
    for (int z = 0; z < 2; ++z) bit[z] = v0[z] > half ? 1 : 0;
    if (i0 == 0) i0 = 1;
  }
  T* o = out - (a.rescale ? int64_t(1) << log_n : 0) + k0;
  int i = i0;
  if constexpr (SPLIT) {
    const int f1 = min(i1, a.f64_end - a.level);
    Two next = i < f1 ? two(t + (int64_t(i) << log_n)) : Two{};
    for (; i < f1; ++i) {
      const Two tv = next;
      if (i + 1 < f1) next = two(t + (int64_t(i + 1) << log_n));
      const double* c = staged + (i - first) * kMdStaged;
      const double q = c[0], qinv = c[1];
      double r[2];
      row_f64(i, tv, c + 2, a.rescale ? v0d : nullptr, q, qinv, r);
      Two w;
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        double x = r[z] + (bit[z] ? 1.0 : 0.0);  // at most 0.51 q + 1
        if (x < 0.0) x += q;
        w.v[z] = Word<double>::to_word(x);
      }
      *reinterpret_cast<Two*>(o + (int64_t(i) << log_n)) = w;
    }
  }
  for (; i < i1; ++i) {
    const T q = a.tabs.prime[a.level + i].q;
    T r[2];
    row_int(i, a.md.w + (base + i) * kMdWords, a.rescale ? v0 : nullptr, r);
    Two w;
#pragma unroll
    for (int z = 0; z < 2; ++z) w.v[z] = csub(T(r[z] + bit[z]), q);
    *reinterpret_cast<Two*>(o + (int64_t(i) << log_n)) = w;
  }
}

template <typename T>
MdArgs<T> moddown_args(const Context& c, int level, int rescale) {
  const bool f64 = sizeof(T) == 8 && c.f64_core && c.f64_tables_ok;
  return MdArgs<T>{c.log_n, level, c.num_q, c.num_p, rescale, f64 ? c.f64_prime_end : 0, tables<T>(c),
                   md_tables<T>(c)};
}

// Groups of rows per coefficient tile, so that a few ciphertexts fill the GPU.
// Each group forms the digits (and v_0) again, about num_p / 2 rows' work:
// * as many as give two blocks per SM, which hide one another's loads, with at
//   least 1 + num_p / 2 rows each;
// * up to fourteen blocks per SM where the rows are many (2 + 2 num_p, 6 more
//   with the rescale, whose v_0 is a row's sum that nothing hides): shorter
//   blocks leave a smaller last wave.
// Measured, by groups (us): N = 2^14, 8 + 1 rows, 1 ciphertext (64 tiles) 1:
// 6.4, 2: 4.7, 4: 4.2, 8: 5.2; 16 ciphertexts of 2 + 1 rows (1024 tiles) 1: 11.6,
// 2: 14.2 (one group for all rows and both components, before the sums of
// products: 10.5); N = 2^16, 29 + 4 rows through sigma_g, 3 ciphertexts (768
// tiles) 1: 106.6, 2: 100.9, 3: 110.0, 4 of them 1: 132.1, 2: 134.4; 32-bit words
// of N = 2^15, 30 + 2 rows, 7 ciphertexts (896 tiles) 1: 49.7, 2: 42.8, 3: 42.1,
// with the rescale 44.9, 40.7, 41.3.  Over 1041 calls (1 to 24 ciphertexts, both
// words, with and without addends and rescale) the choice is 0.9 % from the best
// on average, 16 % at most.  And few enough rows in each for the staged
// constants.
inline int moddown_groups(int64_t tiles, int q_limbs, int num_p, int rescale) {
  const int64_t fill = std::min<int64_t>(2 * 148 / tiles, q_limbs / (1 + num_p / 2));
  const int64_t tail = std::min<int64_t>(14 * 148 / tiles, q_limbs / (2 + 2 * num_p + (rescale ? 6 : 0)));
  const int64_t least = (q_limbs + kMdRows - 2) / (kMdRows - 1);
  return int(std::max({least, int64_t(1), fill, tail}));
}

// t0/t1: [B, QP_l, N] canonical coefficient rows; add0/add1 (nullable):
// [B, Q_l, N] canonical, add0 optionally read through sigma_g (rotation of
// c0); out: [2, B, Q_l (- 1), N] canonical, components out_pitch words apart.
// Blocks (coefficients, component, ciphertext, group of rows), groups
// fastest: they share the P rows in L2.  Every group forms the digits (and
// v_0) itself.
template <typename T, int NP, bool SPLIT>
__global__ void __launch_bounds__(kMdThreads, 2)
k_moddown(const __grid_constant__ MdArgs<T> a, const T* __restrict__ t0, const T* __restrict__ t1,
          const T* __restrict__ add0, const T* __restrict__ add1, T* __restrict__ out, int64_t out_pitch, int groups,
          uint32_t add0_ginv, const uint32_t* __restrict__ item_galois) {
  __shared__ double staged[md_staged<SPLIT>()];
  unsigned idx = blockIdx.x;
  const int g = int(idx % unsigned(groups));
  idx /= unsigned(groups);
  const unsigned tiles = 1u << (a.log_n - 9);
  const int k0 = int((idx % tiles) * kMdThreads + threadIdx.x) * 2;
  idx /= tiles;
  const int c = int(idx & 1), bi = int(idx >> 1);
  const int ql = a.num_q - a.level;
  const T* add = c ? add1 : add0;
  uint32_t gi = 0;
  if (c == 0) gi = item_galois ? (item_galois[bi] == 1 ? 0u : galois_inverse_dev(item_galois[bi], a.log_n)) : add0_ginv;
  moddown_rows<T, NP, SPLIT>(a, (c ? t1 : t0) + ((int64_t(bi) * (ql + a.num_p)) << a.log_n),
                             add ? add + ((int64_t(bi) * ql) << a.log_n) : nullptr, gi,
                             out + c * out_pitch + ((int64_t(bi) * (ql - (a.rescale ? 1 : 0))) << a.log_n), k0,
                             ql * g / groups, ql * (g + 1) / groups, staged);
}

// Standalone rescale of coefficient/standard components: in [K, L, N] ->
// out [K, L-1, N] (csrc/ops/ckks/cpu/ckks_cpu.cpp:203-262): row i is
// (v_i - v_0) C (+ 1) with C = q_0^{-1}.  A thread takes two coefficients of
// up to kRescaleRows rows, so v_0 and its rounding are read and formed once
// for them.  Blocks (row group, coefficients, polynomial).  Bound by HBM:
// 73 -> 36 us for 2 x 3 x 29 rows of N = 2^16, 25 us at the copy rate.
constexpr int kRescaleRows = 6;

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(kMdThreads)
k_rescale(const __grid_constant__ MdArgs<T> a, const T* __restrict__ in, T* __restrict__ out, int groups, int nearest) {
  struct alignas(2 * sizeof(T)) Two {
    T v[2];
  };
  unsigned idx = blockIdx.x;
  const int g = int(idx % unsigned(groups));
  idx /= unsigned(groups);
  const unsigned tiles = 1u << (a.log_n - 9);
  const int k0 = int((idx % tiles) * kMdThreads + threadIdx.x) * 2;
  const int64_t poly = idx / tiles;
  const int limbs = a.num_q - a.level, qp0 = a.num_q + a.num_p;
  const T* src = in + ((poly * limbs) << a.log_n) + k0;
  T* dst = out + ((poly * (limbs - 1)) << a.log_n) + k0;
  const Two v0 = *reinterpret_cast<const Two*>(src);
  const T half = a.tabs.prime[a.level].q >> 1;
  T bit[2];
#pragma unroll
  for (int z = 0; z < 2; ++z) bit[z] = nearest && v0.v[z] > half ? 1 : 0;
  const int i0 = 1 + g * kRescaleRows, i1 = min(limbs, i0 + kRescaleRows);
#pragma unroll 2
  for (int i = i0; i < i1; ++i) {
    const int pid = a.level + i;
    const int64_t c = int64_t(a.level + 1) * qp0 + pid;
    const Two v = *reinterpret_cast<const Two*>(src + (int64_t(i) << a.log_n));
    Two o;
    if (SPLIT && pid < a.f64_end) {
      if constexpr (SPLIT) {
        const double q = a.md.prime[pid].q, qinv = a.md.prime[pid].one_s, f = a.md.f[c * kMdDoubles + 1];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const double d = Word<double>::from_word(v.v[z]) - Word<double>::from_word(v0.v[z]);
          double x = Word<double>::mul_qinv_bal(d, f, q, qinv) + (bit[z] ? 1.0 : 0.0);
          if (x < 0.0) x += q;
          o.v[z] = Word<double>::to_word(x);
        }
      }
    } else {
      const PrimeInfo<T>& p = a.tabs.prime[pid];
      const T q = p.q, y = T(0) - p.neg_inv, qi = y * (T(2) - q * y);
      const T cc = a.md.w[c * kMdWords + 1], dd = a.md.w[c * kMdWords + 2];
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        MdSum<T> s;
        s.add(v.v[z], cc);
        s.add(v0.v[z], dd);
        o.v[z] = csub(T(csub(s.reduced(q, qi), q) + bit[z]), q);
      }
    }
    *reinterpret_cast<Two*>(dst + (int64_t(i - 1) << a.log_n)) = o;
  }
}

}  // namespace fhb
