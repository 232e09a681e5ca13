// Negacyclic transforms in two launches, and the key switch built on them.
//
// N = 2^LOGN is taken as 2^(LOGN - 8) rows of 256 words.  The column stages
// (half spans N/2 .. 256) pair words of one column in different rows; the
// block stages (half spans 128 .. 1) stay inside one row.  The intermediate
// crosses device memory (L2 where it fits), so no cluster, no distributed
// shared memory and no whole-SM block is needed: column tiles are blocks of
// 256 threads with one barrier, and a row of 256 words is transformed by half
// a warp, 16 words per thread, whose only exchanges are warp-local.  Every SM
// can hold several such blocks, so one block's loads run under another's
// products; the one-launch cluster transform (fhb_ntt.cuh) holds a whole SM
// per block, meets a cluster barrier before and after its cross-block stages,
// and leaves 28 of the 148 SMs without a cluster.  Measured on the key-switch
// core at N = 2^16, L = 35 + 4, 32 ciphertexts: cluster core 20.4 ms (FP64
// pipe 33 % busy, long scoreboard and barriers), these launches 10.9 ms
// (FP64 pipe 52-56 % busy: columns 5.1, rows 5.2, inverse columns 0.65 ms);
// at N = 2^14, one ciphertext, 6 rows: 217 -> 117 us for the whole HMult.
//
// Butterflies, twiddles and ranges are those of fhb_ntt.cuh: integer words
// see the same operations in the same order, so even lazy results are the
// same words; FP64 rows (primes below 2^42) hold balanced integers in
// doubles, which is also how they cross memory between the two launches.
#pragma once
#include "fhb_kernels.cuh"

namespace fhb {

// Twiddles by table index: (w, companion) pairs for integer words; values
// alone for the FP64 rows, whose butterflies take the quotient from the
// product and 1/q.
template <typename T>
struct TwAt {
  static constexpr bool kQFromProduct = false;
  const TwPair<T>* g;
  __device__ __forceinline__ TwPair<T> at(int i) const { return ldtw(g, i); }
};
struct TwAtQ {
  static constexpr bool kQFromProduct = true;
  const double* g;
  double qinv;
  __device__ __forceinline__ TwPair<double> at(int i) const { return TwPair<double>{__ldg(g + i), qinv}; }
};

constexpr int kBlkLog = 8;           // words per row: the block stages' length
constexpr int kBlk = 1 << kBlkLog;

// Bounds of the balanced FP64 inverse: a pass of K Gentleman-Sande stages
// over inputs below 2.4 q leaves word i of a group of 2^K grown by one
// doubling per stage after the last stage that took it as a product: word 0
// by 2^K, word 1 to 0.6 q 2^(K-1), words 2 and 3 to at most 2.4 q, the others
// less.  Reducing words 0 and (K = 4) 1 keeps every pass's inputs below
// 2.4 q and every product operand below 2 x 19.2 q < 2^48 (q < 2^42).
template <typename T, int K>
__device__ __forceinline__ void reduce_grown(T (&x)[1 << K], T q, T qinv) {
  if constexpr (std::is_same<T, double>::value) {
    x[0] = Word<double>::reduce_bal(x[0], q, qinv);
    if constexpr (K >= 4) x[1] = Word<double>::reduce_bal(x[1], q, qinv);
  }
}

// ---- column stages ---------------------------------------------------------
// A block transforms kCols adjacent columns (at least 128 contiguous bytes of
// every row where the ring allows it), 16 words per thread.
template <typename T, int LOGN>
struct ColGeom {
  static constexpr int kA = LOGN - kBlkLog;  // column stages
  static constexpr int kRows = 1 << kA;
  static constexpr int kThreads = (kA > 8 || (sizeof(T) == 4 && kA == 8)) ? 512 : 256;
  static constexpr int kTile = kThreads * 16;
  static constexpr int kCols = kTile >> kA;
  static constexpr int kTiles = (1 << LOGN) / kTile;
  static_assert(kCols <= kBlk && kTiles >= 1, "a tile is at most a whole polynomial");
  static constexpr int kPasses = kA <= 4 ? 1 : (kA <= 8 ? 2 : 3);
  static constexpr int pass_k(int j) { return kA == 9 ? 3 : (j == 0 ? (kA < 4 ? kA : 4) : kA - 4); }
  static constexpr int pass_a(int j) { return j == 0 ? 0 : pass_a(j - 1) + pass_k(j - 1); }
  static constexpr size_t smem_bytes() { return kPasses > 1 ? size_t(kTile) * sizeof(T) : 0; }
};

template <typename T, int LOGN, class TW>
struct Cols {
  using G = ColGeom<T, LOGN>;
  using B = Ntt<T, LOGN, TW>;

  // One group of 2^K words: row0 the row of its first word, hi the stage
  // group it belongs to.
  template <int K, int R>
  __device__ __forceinline__ static void group(int u, int& row0, int& hi, int& col) {
    const int gid = u * G::kThreads + int(threadIdx.x);
    col = gid & (G::kCols - 1);
    const int rest = gid / G::kCols;
    hi = rest >> R;
    row0 = (hi << (K + R)) | (rest & ((1 << R) - 1));
  }

  template <int J, class Src, class Sink>
  __device__ __forceinline__ static void fwd(Src& src, Sink& sink, T* s, const TW& tw, T q, T m2, int col0) {
    constexpr int K = G::pass_k(J), A = G::pass_a(J), R = G::kA - A - K, kGs = 1 << K;
    constexpr bool kLast = J == G::kPasses - 1;
#pragma unroll
    for (int u = 0; u < (16 >> K); ++u) {
      int row0, hi, col;
      group<K, R>(u, row0, hi, col);
      T x[kGs];
      if constexpr (J == 0) {
        src.template column<kGs>(row0 * kBlk + col0 + col, kBlk << R, x);
      } else {
#pragma unroll
        for (int k = 0; k < kGs; ++k) x[k] = s[(row0 + (k << R)) * G::kCols + col];
      }
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int h = kGs >> (b + 1);
#pragma unroll
        for (int i = 0; i < kGs; ++i)
          if (!(i & h)) B::fwd_bfly(x[i], x[i + h], tw.at((1 << (A + b)) + (hi << b) + (i >> (K - b))), q, m2);
      }
      if constexpr (kLast) {
        sink.template column<kGs>(row0 * kBlk + col0 + col, kBlk << R, x);
      } else {
#pragma unroll
        for (int k = 0; k < kGs; ++k) s[(row0 + (k << R)) * G::kCols + col] = x[k];
      }
    }
    if constexpr (!kLast) {
      __syncthreads();
      fwd<J + 1>(src, sink, s, tw, q, m2, col0);
    }
  }

  template <int J, class Src, class Epi>
  __device__ __forceinline__ static void inv(Src& src, Epi& epi, T* s, const TW& tw, T q, T m2, int col0) {
    constexpr int F = G::kPasses - 1 - J;  // the forward pass it undoes
    constexpr int K = G::pass_k(F), A = G::pass_a(F), R = G::kA - A - K, kGs = 1 << K;
    constexpr bool kLast = J == G::kPasses - 1;
#pragma unroll
    for (int u = 0; u < (16 >> K); ++u) {
      int row0, hi, col;
      group<K, R>(u, row0, hi, col);
      const int at = row0 * kBlk + col0 + col;
      T x[kGs];
      if constexpr (J == 0) {
        src.template column<kGs>(at, kBlk << R, x);
      } else {
#pragma unroll
        for (int k = 0; k < kGs; ++k) x[k] = s[(row0 + (k << R)) * G::kCols + col];
      }
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int j = kBlkLog + R + b, h = 1 << b;
#pragma unroll
        for (int i = 0; i < kGs; ++i)
          if (!(i & h))
            B::inv_bfly(x[i], x[i + h], tw.at(((1 << LOGN) >> (j + 1)) + (hi << (K - 1 - b)) + (i >> (b + 1))), q, m2);
      }
      if constexpr (kLast) {
#pragma unroll
        for (int k = 0; k < kGs; ++k) epi(at + k * (kBlk << R), x[k]);
      } else {
        reduce_grown<T, K>(x, q, m2);
#pragma unroll
        for (int k = 0; k < kGs; ++k) s[(row0 + (k << R)) * G::kCols + col] = x[k];
      }
    }
    if constexpr (!kLast) {
      __syncthreads();
      inv<J + 1>(src, epi, s, tw, q, m2, col0);
    }
  }
};

// Plain column source and sink over a polynomial held as T (FP64 rows:
// doubles over the words).  Every word of a tile is read before it is written
// by the thread that read it, or after a barrier: in place is fine.
template <typename T>
struct ColSource {
  const T* p;
  template <int C>
  __device__ __forceinline__ void column(int m, int stride, T (&x)[C]) const {
#pragma unroll
    for (int k = 0; k < C; ++k) x[k] = p[m + k * stride];
  }
};
template <typename T>
struct ColSink {
  T* p;
  template <int C>
  __device__ __forceinline__ void column(int m, int stride, const T (&x)[C]) const {
#pragma unroll
    for (int k = 0; k < C; ++k) p[m + k * stride] = x[k];
  }
};

// ---- block stages ----------------------------------------------------------
// Half a warp holds one row of 256 words, 16 per thread t of 16, in one of
// three layouts: strided (word t + 16 k), contiguous (16 t + k) and vector
// (16-byte vectors of V words: 16 V k + V t + i, coalesced in global memory).
// Exchanges go through 256 words of shared memory per half warp, swizzled in
// 16-byte pieces so that every access below is free of bank conflicts.
constexpr int kRowThreads = 128;                 // four warps, eight half warps
constexpr int kRowSlots = kRowThreads / 16;

template <typename T>
struct RowX {
  static constexpr int V = 16 / int(sizeof(T));  // words per 16-byte piece
  static constexpr int kVec = 16 / V;            // pieces per thread
  struct alignas(16) Piece {
    T v[V];
  };
  unsigned char* w;  // this warp's 512 words
  int half, t;
  __device__ __forceinline__ explicit RowX(unsigned char* smem)
      : w(smem + (threadIdx.x >> 5) * (2 * kBlk * sizeof(T))), half((threadIdx.x >> 4) & 1), t(threadIdx.x & 15) {}
  // byte offset of 16-byte piece p of the 16 words [16 r, 16 r + 16)
  __device__ __forceinline__ int at(int r, int p) const {
    if constexpr (sizeof(T) == 8) {
      return half * 2048 + r * 128 + ((p ^ (r & 7)) << 4);
    } else {
      return r * 128 + (((half * 4 + p) ^ (r & 7)) << 4);
    }
  }
  __device__ __forceinline__ T* word(int r, int c) const {
    return reinterpret_cast<T*>(w + at(r, c / V)) + (c & (V - 1));
  }
  __device__ __forceinline__ void put_strided(const T (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) *word(k, t) = v[k];
  }
  __device__ __forceinline__ void get_strided(T (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = *word(k, t);
  }
  __device__ __forceinline__ void put_contiguous(const T (&v)[16]) const {
#pragma unroll
    for (int p = 0; p < kVec; ++p) {
      Piece x;
#pragma unroll
      for (int i = 0; i < V; ++i) x.v[i] = v[p * V + i];
      *reinterpret_cast<Piece*>(w + at(t, p)) = x;
    }
  }
  __device__ __forceinline__ void get_contiguous(T (&v)[16]) const {
#pragma unroll
    for (int p = 0; p < kVec; ++p) {
      const Piece x = *reinterpret_cast<const Piece*>(w + at(t, p));
#pragma unroll
      for (int i = 0; i < V; ++i) v[p * V + i] = x.v[i];
    }
  }
  __device__ __forceinline__ void put_vector(const T (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
      Piece x;
#pragma unroll
      for (int i = 0; i < V; ++i) x.v[i] = v[k * V + i];
      *reinterpret_cast<Piece*>(w + at(V * k + ((V * t) >> 4), ((V * t) & 15) / V)) = x;
    }
  }
  __device__ __forceinline__ void get_vector(T (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
      const Piece x = *reinterpret_cast<const Piece*>(w + at(V * k + ((V * t) >> 4), ((V * t) & 15) / V));
#pragma unroll
      for (int i = 0; i < V; ++i) v[k * V + i] = x.v[i];
    }
  }
};

template <typename T, int LOGN, class TW>
struct Rows {
  using B = Ntt<T, LOGN, TW>;
  static constexpr int kA = LOGN - kBlkLog;

  // strided -> contiguous
  __device__ __forceinline__ static void fwd(T (&v)[16], const RowX<T>& x, const TW& tw, T q, T m2, int blk) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int h = 8 >> b;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) B::fwd_bfly(v[i], v[i + h], tw.at((1 << (kA + b)) + (blk << b) + (i >> (4 - b))), q, m2);
    }
    __syncwarp();
    x.put_strided(v);
    __syncwarp();
    x.get_contiguous(v);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int h = 8 >> b;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h))
          B::fwd_bfly(v[i], v[i + h], tw.at((1 << (kA + 4 + b)) + ((blk * 16 + x.t) << b) + (i >> (4 - b))), q, m2);
    }
  }
  __device__ __forceinline__ static void contiguous_to_vector(T (&v)[16], const RowX<T>& x) {
    __syncwarp();
    x.put_contiguous(v);
    __syncwarp();
    x.get_vector(v);
  }
  __device__ __forceinline__ static void vector_to_contiguous(T (&v)[16], const RowX<T>& x) {
    __syncwarp();
    x.put_vector(v);
    __syncwarp();
    x.get_contiguous(v);
  }
  __device__ __forceinline__ static void strided_to_contiguous(T (&v)[16], const RowX<T>& x) {
    __syncwarp();
    x.put_strided(v);
    __syncwarp();
    x.get_contiguous(v);
  }

  // contiguous -> strided
  __device__ __forceinline__ static void inv(T (&v)[16], const RowX<T>& x, const TW& tw, T q, T m2, int blk) {
    constexpr int kN = 1 << LOGN;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int h = 1 << j;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h))
          B::inv_bfly(v[i], v[i + h], tw.at((kN >> (j + 1)) + ((blk * 16 + x.t) << (3 - j)) + (i >> (j + 1))), q, m2);
    }
    reduce_grown<T, 4>(v, q, m2);
    __syncwarp();
    x.put_contiguous(v);
    __syncwarp();
    x.get_strided(v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int h = 1 << j;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h))
          B::inv_bfly(v[i], v[i + h], tw.at((kN >> (j + 5)) + (blk << (3 - j)) + (i >> (j + 1))), q, m2);
    }
    reduce_grown<T, 4>(v, q, m2);
  }
};

// ---------------------------------------------------------------------------
// Key switch.  Y holds, per (digit a, ciphertext b, row j) of the rows
// [row_lo, row_lo + rows) in flight, the polynomial between the launches:
// Y[(a y_batch + b) rows + j - row_lo][N].
template <typename T>
struct KsPass {
  const T* digits;      // ModUp digits [B, L, N]
  T* y;
  const T* key;         // [D, 2, QP0, N]
  const unsigned long long* item_keys;  // per-ciphertext keys instead of `key` (nullable)
  T* acc0;              // [B, QP_l, N]
  T* acc1;
  const T* ct3;         // relinearisation addends (nullable), components ct3_stride words apart
  int64_t ct3_stride;
  int batch, y_batch, q_limbs, qp_limbs, level, qp0, row_lo, rows, f64_rows, ext_digits, f64_end;
  ChainTables<T> tabs;
  LevelTables<T> lt;
  ChainTables<double> tabs64f;
  const TwPair<double>* ext64f;
};

// True when row pid's own digit residue replaces the transform (relinearisation).
template <typename T>
__device__ __forceinline__ bool ks_own(const KsPass<T>& k, const DigitDesc& d, int jrow) {
  const int pid = k.level + jrow;
  return k.ct3 != nullptr && jrow < k.q_limbs && pid >= d.prime0 && pid < d.prime0 + d.alpha;
}

// Launch 1: extension of a digit to a row's prime and the column stages of
// its forward transform.  One block per (digit, ciphertext, column tile, row),
// rows fastest, so the blocks in flight share the digit's words in L2.  PRE:
// Y already holds the extensions (tensor-core basis conversion), transformed
// in place.
template <typename T, int LOGN, bool PRE, bool SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads)
k_ks_columns(const __grid_constant__ KsPass<T> k) {
  using G = ColGeom<T, LOGN>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned idx = blockIdx.x;
  const int jrow = k.row_lo + k.rows - 1 - int(idx % unsigned(k.rows));
  idx /= unsigned(k.rows);
  const int col0 = int(idx % G::kTiles) * G::kCols;
  idx /= G::kTiles;
  const int bi = int(idx % unsigned(k.batch)), a = int(idx / unsigned(k.batch));
  const DigitDesc d = k.lt.digits[a];
  if (ks_own(k, d, jrow)) return;
  const int pid = k.level + jrow;
  T* y = k.y + ((int64_t(a) * k.y_batch + bi) * k.rows + (jrow - k.row_lo)) * kN;
  const T* dig = k.digits + (int64_t(bi) * k.q_limbs + (d.prime0 - k.level)) * kN;
  if constexpr (SPLIT) {
    static_assert(sizeof(T) == 8, "FP64 rows exist in int64 chains only");
    if (jrow < k.f64_rows) {
      using C = Cols<double, LOGN, TwAtQ>;
      const double q = k.tabs64f.prime[pid].q, qinv = k.tabs64f.prime[pid].one_s;
      ColSink<double> sink{reinterpret_cast<double*>(y)};
      double* s = reinterpret_cast<double*>(smem_raw);
      const TwAtQ tw{k.tabs64f.twv_fwd + int64_t(pid) * kN, qinv};
      if constexpr (PRE) {
        U64RowSource src{reinterpret_cast<const uint64_t*>(y)};
        C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
      } else {
        ExtSourceF64 src{reinterpret_cast<const uint64_t*>(dig),
                         k.ext64f + (((int64_t(k.level) * k.ext_digits + a) * kMaxDigitWidth) * 2) * k.qp0 + pid,
                         k.qp0, d.alpha, LOGN, d.prime0 + d.alpha > k.f64_end, q, qinv};
        C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
      }
      return;
    }
  }
  using C = Cols<T, LOGN, TwAt<T>>;
  const T q = k.tabs.prime[pid].q, twoq = k.tabs.prime[pid].twice_q;
  ColSink<T> sink{y};
  T* s = reinterpret_cast<T*>(smem_raw);
  const TwAt<T> tw{k.tabs.tw_fwd + int64_t(pid) * kN};
  if constexpr (PRE) {
    ColSource<T> src{y};
    C::template fwd<0>(src, sink, s, tw, q, twoq, col0);
  } else {
    ExtSource<T> src{dig, k.lt.ext + int64_t(a) * kMaxDigitWidth * k.qp0 + pid, k.qp0, d.alpha, LOGN, q, twoq};
    C::template fwd<0>(src, sink, s, tw, q, twoq, col0);
  }
}

// Launch 2: for one row of 256 words of (ciphertext, row j): the block stages
// of every digit's forward transform, the products with both key components
// summed in registers, and the block stages of both inverse transforms.  Half
// a warp per (ciphertext, 256 words), ciphertexts fastest, so that the half
// warps of a block read the same key words and twiddles.
template <int LOGN>
__device__ __forceinline__ void ks_rows_f64(const KsPass<uint64_t>& k, int jrow, int bi, int blk, bool live,
                                            unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  using W = Word<double>;
  using R = Rows<double, LOGN, TwAtQ>;
  const int pid = k.level + jrow;
  const PrimeInfo<double>& p = k.tabs64f.prime[pid];
  const double q = p.q, qinv = p.one_s;
  const RowX<double> x(smem);
  const int vec = blk * kBlk + 2 * x.t;  // this thread's first word, vector layout
  const uint64_t* key = k.item_keys ? reinterpret_cast<const uint64_t*>(k.item_keys[bi]) : k.key;
  const uint64_t* ct3 = k.ct3 ? k.ct3 + (int64_t(bi) * k.q_limbs + jrow) * kN + vec : nullptr;
  const TwAtQ twf{k.tabs64f.twv_fwd + int64_t(pid) * kN, qinv};
  double a0[16], a1[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) a0[e] = a1[e] = 0.0;
  for (int a = 0; a < k.lt.num_digits; ++a) {
    const DigitDesc d = k.lt.digits[a];
    double v[16];
    if (ks_own(k, d, jrow)) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(ct3 + 2 * k.ct3_stride + 32 * e));
        v[2 * e] = W::shoup_bal(W::from_word(w.x), p.rinv, p.rinv_s, q);
        v[2 * e + 1] = W::shoup_bal(W::from_word(w.y), p.rinv, p.rinv_s, q);
      }
    } else {
      const double* y = reinterpret_cast<const double*>(k.y) +
                        ((int64_t(a) * k.y_batch + bi) * k.rows + (jrow - k.row_lo)) * kN + blk * kBlk + x.t;
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = __ldg(y + 16 * e);
      R::fwd(v, x, twf, q, qinv, blk);
      R::contiguous_to_vector(v, x);
    }
    const uint64_t* key0 = key + ((int64_t(d.key_digit) * 2) * k.qp0 + pid) * kN + vec;
    const uint64_t* key1 = key0 + k.qp0 * kN;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const ulonglong2 u0 = __ldg(reinterpret_cast<const ulonglong2*>(key0 + 32 * e));
      const ulonglong2 u1 = __ldg(reinterpret_cast<const ulonglong2*>(key1 + 32 * e));
      a0[2 * e] += W::mul_qinv_bal(v[2 * e], W::from_word(u0.x), q, qinv);
      a0[2 * e + 1] += W::mul_qinv_bal(v[2 * e + 1], W::from_word(u0.y), q, qinv);
      a1[2 * e] += W::mul_qinv_bal(v[2 * e], W::from_word(u1.x), q, qinv);
      a1[2 * e + 1] += W::mul_qinv_bal(v[2 * e + 1], W::from_word(u1.y), q, qinv);
    }
  }
  const TwAtQ twi{k.tabs64f.twv_inv + int64_t(pid) * kN, qinv};
  auto finish = [&](double (&v)[16], const uint64_t* add, uint64_t* out) {
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = W::reduce_bal(v[e], q, qinv);
    if (add) {  // P c_k, carrying R like the sums
      const TwPair<double> pc = k.tabs64f.p_rinv[pid];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(add + 32 * e));
        v[2 * e] += W::shoup_bal(W::from_word(w.x), pc.w, pc.wp, q);
        v[2 * e + 1] += W::shoup_bal(W::from_word(w.y), pc.w, pc.wp, q);
      }
    }
    R::vector_to_contiguous(v, x);
    R::inv(v, x, twi, q, qinv, blk);
    double* o = reinterpret_cast<double*>(out) + (int64_t(bi) * k.qp_limbs + jrow) * kN + blk * kBlk + x.t;
    if (live) {
#pragma unroll
      for (int e = 0; e < 16; ++e) o[16 * e] = v[e];
    }
  };
  finish(a0, ct3, k.acc0);
  finish(a1, ct3 ? ct3 + k.ct3_stride : nullptr, k.acc1);
}

template <typename T, int LOGN>
__device__ __forceinline__ void ks_rows_int(const KsPass<T>& k, int jrow, int bi, int blk, bool live,
                                            unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  using W = Word<T>;
  using R = Rows<T, LOGN, TwAt<T>>;
  using X = RowX<T>;
  using Piece = typename X::Piece;
  const int pid = k.level + jrow;
  const PrimeInfo<T>& p = k.tabs.prime[pid];
  const T q = p.q, twoq = p.twice_q, ni = p.neg_inv;
  const X x(smem);
  const int vec = blk * kBlk + X::V * x.t;
  const T* key = k.item_keys ? reinterpret_cast<const T*>(k.item_keys[bi]) : k.key;
  const T* ct3 = k.ct3 && jrow < k.q_limbs ? k.ct3 + (int64_t(bi) * k.q_limbs + jrow) * kN + vec : nullptr;
  auto piece = [](const T* at) {
    Piece r;
    *reinterpret_cast<uint4*>(r.v) = __ldg(reinterpret_cast<const uint4*>(at));
    return r;
  };
  const TwAt<T> twf{k.tabs.tw_fwd + int64_t(pid) * kN};
  T a0[16], a1[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) a0[e] = a1[e] = 0;
  for (int a = 0; a < k.lt.num_digits; ++a) {
    const DigitDesc d = k.lt.digits[a];
    T v[16];
    if (ks_own(k, d, jrow)) {
#pragma unroll
      for (int e = 0; e < X::kVec; ++e) {
        const Piece w = piece(ct3 + 2 * k.ct3_stride + 16 * X::V * e);
#pragma unroll
        for (int i = 0; i < X::V; ++i) v[e * X::V + i] = W::shoup(w.v[i], p.rinv, p.rinv_s, q);
      }
    } else {
      const T* y =
          k.y + ((int64_t(a) * k.y_batch + bi) * k.rows + (jrow - k.row_lo)) * kN + blk * kBlk + x.t;
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = __ldg(y + 16 * e);
      R::fwd(v, x, twf, q, twoq, blk);
      R::contiguous_to_vector(v, x);
    }
    const T* key0 = key + ((int64_t(d.key_digit) * 2) * k.qp0 + pid) * kN + vec;
    const T* key1 = key0 + k.qp0 * kN;
#pragma unroll
    for (int e = 0; e < X::kVec; ++e) {
      const Piece u0 = piece(key0 + 16 * X::V * e), u1 = piece(key1 + 16 * X::V * e);
#pragma unroll
      for (int i = 0; i < X::V; ++i) {
        const int at = e * X::V + i;
        const T y = csub(v[at], twoq);
        a0[at] = csub(a0[at] + W::mont(y, u0.v[i], q, ni), twoq);
        a1[at] = csub(a1[at] + W::mont(y, u1.v[i], q, ni), twoq);
      }
    }
  }
  const TwAt<T> twi{k.tabs.tw_inv + int64_t(pid) * kN};
  auto finish = [&](T (&v)[16], const T* add, T* out) {
    if (add) {
      const TwPair<T> ps = k.tabs.p_rinv[pid];
#pragma unroll
      for (int e = 0; e < X::kVec; ++e) {
        const Piece w = piece(add + 16 * X::V * e);
#pragma unroll
        for (int i = 0; i < X::V; ++i) {
          const int at = e * X::V + i;
          v[at] = csub(v[at] + W::shoup(w.v[i], ps.w, ps.wp, q), twoq);
        }
      }
    }
    R::vector_to_contiguous(v, x);
    R::inv(v, x, twi, q, twoq, blk);
    T* o = out + (int64_t(bi) * k.qp_limbs + jrow) * kN + blk * kBlk + x.t;
    if (live) {
#pragma unroll
      for (int e = 0; e < 16; ++e) o[16 * e] = v[e];
    }
  };
  finish(a0, ct3, k.acc0);
  finish(a1, ct3 ? ct3 + k.ct3_stride : nullptr, k.acc1);
}

template <typename T>
constexpr size_t row_smem() {
  return size_t(kRowSlots) * kBlk * sizeof(T);
}

template <typename T, int LOGN, bool SPLIT>
__global__ void __launch_bounds__(kRowThreads, 4)
k_ks_rows(const __grid_constant__ KsPass<T> k) {
  __shared__ __align__(16) unsigned char smem[row_smem<T>()];
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  const unsigned slots = unsigned(kBlks) * unsigned(k.batch);
  const unsigned per_row = (slots + kRowSlots - 1) / kRowSlots;
  const int jrow = k.row_lo + k.rows - 1 - int(blockIdx.x / per_row);
  unsigned slot = (blockIdx.x % per_row) * kRowSlots + (threadIdx.x >> 4);
  const bool live = slot < slots;
  if (!live) slot = slots - 1;  // the last block's spare half warps repeat a row and store nothing
  const int bi = int(slot % unsigned(k.batch)), blk = int(slot / unsigned(k.batch));
  if constexpr (SPLIT) {
    static_assert(sizeof(T) == 8, "FP64 rows exist in int64 chains only");
    if (jrow < k.f64_rows) {
      ks_rows_f64<LOGN>(k, jrow, bi, blk, live, smem);
      return;
    }
  }
  ks_rows_int<T, LOGN>(k, jrow, bi, blk, live, smem);
}

// Launch 3: the column stages of the inverse transforms, in place over the
// accumulator rows, to canonical coefficients.  One block per (component,
// ciphertext, row, column tile).
template <typename T, int LOGN, bool SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads)
k_ks_columns_inverse(const __grid_constant__ KsPass<T> k) {
  using G = ColGeom<T, LOGN>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned idx = blockIdx.x;
  const int col0 = int(idx % G::kTiles) * G::kCols;
  idx /= G::kTiles;
  const int jrow = k.row_lo + k.rows - 1 - int(idx % unsigned(k.rows));
  idx /= unsigned(k.rows);
  const int bi = int(idx % unsigned(k.batch));
  T* z = (idx / unsigned(k.batch) ? k.acc1 : k.acc0) + (int64_t(bi) * k.qp_limbs + jrow) * kN;
  const int pid = k.level + jrow;
  if constexpr (SPLIT) {
    if (jrow < k.f64_rows) {
      const PrimeInfo<double>& p = k.tabs64f.prime[pid];
      ColSource<double> src{reinterpret_cast<double*>(z)};
      F64InvEpilogue epi{reinterpret_cast<uint64_t*>(z), p.q, p.ninv_rinv, p.ninv_rinv_s};
      Cols<double, LOGN, TwAtQ>::template inv<0>(src, epi, reinterpret_cast<double*>(smem_raw),
                                                 TwAtQ{k.tabs64f.twv_inv + int64_t(pid) * kN, p.one_s}, p.q, p.one_s,
                                                 col0);
      return;
    }
  }
  const PrimeInfo<T>& p = k.tabs.prime[pid];
  ColSource<T> src{z};
  InvEpilogue<T> epi{z, p.q, p.ninv, p.ninv_s, kInvStandard};
  Cols<T, LOGN, TwAt<T>>::template inv<0>(src, epi, reinterpret_cast<T*>(smem_raw),
                                          TwAt<T>{k.tabs.tw_inv + int64_t(pid) * kN}, p.q, p.twice_q, col0);
}

}  // namespace fhb
