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
// pipe 33 % busy, long scoreboard and barriers), these launches 8.9 ms
// (columns 3.9, rows 4.4, inverse columns 0.64 ms; FP64 pipe 65-73 % busy
// over the FP64 rows, 46-54 % with the five integer rows); at N = 2^14, one ciphertext: 217 -> 69 us for the whole
// HMult.  The standalone transforms: 0.86 -> 0.40 ms forward for 12 x 2 x 35
// int64 rows of N = 2^16, 1.72 -> 0.68 ms inverse for 48 x 2 x 25 int32 rows.
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
  static constexpr bool kWide = false;
  const TwPair<T>* g;
  __device__ __forceinline__ TwPair<T> at(int i) const { return ldtw(g, i); }
};
template <bool WIDE>
struct TwQ {
  static constexpr bool kQFromProduct = true;
  static constexpr bool kWide = WIDE;
  const double* g;
  double qinv;
  __device__ __forceinline__ TwPair<double> at(int i) const { return TwPair<double>{__ldg(g + i), qinv}; }
};

using TwAtQ = TwQ<false>;

// Forms of the FP64 rows (the kernels' FORM): none; narrow, primes below
// 2^42; or wide, primes below 1.1 2^50 (kWidePrimeEnd), on chains without
// narrow rows (the 50-bit chains).  Wide rows use the same butterfly with
// twiddles balanced to (-q/2, q/2) and keep less headroom.  The quotient of a
// product x w comes from the rounded product and the rounded 1/q, each off by
// 2^-53 of it, besides the rounding to an integer; with q < 1.1 2^50 and |w| <=
// q/2 that is at most (1.1/8) |x/q|, so a product leaves (0.5 + 0.1375 |x/q|) q.
// Every value stays exact below 2^53 = 7.2 q as long as each pass of at most
// four stages starts from reduced words: forward from 1.0 q, 1.64, 2.37, 3.19
// to 4.13 q; inverse from 0.51 q, sums double, so the words that were sums
// twice are reduced after two stages (2.04 q) and reach 3.12 q after four.
// Operands stay below 3.2 q, quotients below 1.6 q < 2^51.  Words enter as
// u - q (lazy words below 2q, so |x| <= q).
constexpr int kNoF64 = 0, kNarrowF64 = 1, kWideF64 = 2;

template <bool WIDE>
__device__ __forceinline__ double f64_word(uint64_t u, double q) {
  if constexpr (WIDE) return Word<double>::from_word_minus(u, q);
  return Word<double>::from_word(u);
}

template <class TW, typename T, int COUNT>
__device__ __forceinline__ void reduce_wide(T (&x)[COUNT], T q, T qinv) {
  if constexpr (TW::kWide) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) x[i] = Word<double>::reduce_bal(x[i], q, qinv);
  }
}
// after the second of an inverse pass's stages: the words summed in both
template <class TW, typename T, int COUNT>
__device__ __forceinline__ void reduce_wide_sums(T (&x)[COUNT], T q, T qinv) {
  if constexpr (TW::kWide) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i)
      if ((i & 3) < 2) x[i] = Word<double>::reduce_bal(x[i], q, qinv);
  }
}

constexpr int kBlkLog = 8;           // words per row: the block stages' length
constexpr int kBlk = 1 << kBlkLog;

// Bounds of the balanced FP64 inverse: a pass of K Gentleman-Sande stages
// over inputs below 2.4 q leaves word i of a group of 2^K grown by one
// doubling per stage after the last stage that took it as a product: word 0
// by 2^K, word 1 to 0.6 q 2^(K-1), words 2 and 3 to at most 2.4 q, the others
// less.  Reducing words 0 and (K = 4) 1 keeps every pass's inputs below
// 2.4 q and every product operand below 2 x 19.2 q < 2^48 (q < 2^42).
template <class TW, typename T, int K>
__device__ __forceinline__ void reduce_grown(T (&x)[1 << K], T q, T qinv) {
  reduce_wide<TW>(x, q, qinv);
  if constexpr (std::is_same<T, double>::value && !TW::kWide) {
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

// Blocks per SM the column kernels are compiled for: two of 256 threads where
// a thread holds the words of two rows (128 registers), otherwise 768 threads
// (80 registers) for 64-bit words and 1024 for 32-bit words.  (Left to itself
// the compiler takes 150 registers and the kernel 1.4 times as long.)
template <typename T, int LOGN>
constexpr int col_blocks(bool pairs) {
  constexpr int kThreads = ColGeom<T, LOGN>::kThreads;
  if (sizeof(T) == 4) return 1024 / kThreads;
  return pairs ? 512 / kThreads : (kThreads > 256 ? 1 : 3);
}

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

  template <int A, int K>
  __device__ __forceinline__ static void fwd_stages(T (&x)[1 << K], const TW& tw, T q, T m2, int hi) {
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const int h = (1 << K) >> (b + 1);
#pragma unroll
      for (int i = 0; i < (1 << K); ++i)
        if (!(i & h)) B::fwd_bfly(x[i], x[i + h], tw.at((1 << (A + b)) + (hi << b) + (i >> (K - b))), q, m2);
    }
    reduce_wide<TW>(x, q, m2);
  }

  // Pass J: words from `src` (J = 0) or shared memory, to shared memory or (the last pass) to `sink`.
  template <int J, class Src, class Sink>
  __device__ __forceinline__ static void fwd_pass(Src& src, Sink& sink, T* s, const TW& tw, T q, T m2, int col0) {
    constexpr int K = G::pass_k(J), A = G::pass_a(J), R = G::kA - A - K, kGs = 1 << K;
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
      fwd_stages<A, K>(x, tw, q, m2, hi);
      if constexpr (J == G::kPasses - 1) {
        sink.template column<kGs>(row0 * kBlk + col0 + col, kBlk << R, x);
      } else {
#pragma unroll
        for (int k = 0; k < kGs; ++k) s[(row0 + (k << R)) * G::kCols + col] = x[k];
      }
    }
  }

  template <int J, class Src, class Sink>
  __device__ __forceinline__ static void fwd(Src& src, Sink& sink, T* s, const TW& tw, T q, T m2, int col0) {
    fwd_pass<J>(src, sink, s, tw, q, m2, col0);
    if constexpr (J + 1 < G::kPasses) {
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
        if (b == 1 && K > 2) reduce_wide_sums<TW>(x, q, m2);
      }
      if constexpr (kLast) {
        reduce_wide<TW>(x, q, m2);
#pragma unroll
        for (int k = 0; k < kGs; ++k) epi(at + k * (kBlk << R), x[k]);
      } else {
        reduce_grown<TW, T, K>(x, q, m2);
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
constexpr int kRowWarps = kRowThreads / 32;

template <typename T>
constexpr size_t exchange_smem() {
  return size_t(kRowSlots) * kBlk * sizeof(T);
}

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

// The next row of 256 words on its way into shared memory (cp.async, 16 bytes
// a thread and piece) while the current one is transformed: half a warp owns
// 256 words here, read back in the strided layout without bank conflicts.
// Asks L2 for 256 words (a digit ahead of their use; one thread of a half warp).
template <typename T>
__device__ __forceinline__ void prefetch_row(const T* row) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row), "r"(int(kBlk * sizeof(T))) : "memory");
}
// A 16-byte load that stays where it is written: issued ahead of the stages
// that run while it is under way.
__device__ __forceinline__ uint4 load_ahead(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

template <typename T>
struct RowStage {
  unsigned char* w;
  int half, t;
  __device__ __forceinline__ explicit RowStage(unsigned char* smem)
      : w(smem + (threadIdx.x >> 5) * (2 * kBlk * sizeof(T))), half((threadIdx.x >> 4) & 1), t(threadIdx.x & 15) {}
  __device__ __forceinline__ unsigned char* at(int word) const {
    if constexpr (sizeof(T) == 8) return w + half * 2048 + word * 8;
    return w + (word >> 4) * 128 + half * 64 + (word & 15) * 4;
  }
  __device__ __forceinline__ void request(const T* row) const {
    constexpr int V = 16 / int(sizeof(T));
#pragma unroll
    for (int i = 0; i < 16 / V; ++i) {
      const int word = (i * 16 + t) * V;
      const unsigned dst = unsigned(__cvta_generic_to_shared(at(word)));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(row + word) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // Every thread's words of the requested row, strided layout.  The caller
  // may request the next row afterwards.
  __device__ __forceinline__ void take(T (&v)[16]) const {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = *reinterpret_cast<const T*>(at(16 * k + t));
    __syncwarp();
  }
};

template <typename T, int LOGN, class TW>
struct Rows {
  using B = Ntt<T, LOGN, TW>;
  static constexpr int kA = LOGN - kBlkLog;

  // Twiddle j of row blk's stage b of the strided layout's four (a) and of
  // thread t's stage b of the contiguous layout's four (b); the inverse
  // stages mirror them (b = 3 first).  From the block tables (ChainTables::
  // twr_*), where a row's 255 twiddles lie together and those of the
  // contiguous layout's stages have the thread fastest: a load is one or two
  // whole lines (in bit-reversed order a thread's twiddles lie together, and
  // a load touches up to eight lines).
  __device__ __forceinline__ static TwPair<T> tw_a(const TW& tw, int b, int blk, int j) {
    return tw.at(blk * kBlk + (1 << b) + j);
  }
  __device__ __forceinline__ static TwPair<T> tw_b(const TW& tw, int b, int blk, int t, int j) {
    return tw.at(blk * kBlk + (16 << b) + 16 * j + t);
  }

  // strided -> contiguous: the strided layout's stages and the exchange, then
  // the contiguous layout's stages
  __device__ __forceinline__ static void fwd_a(T (&v)[16], const RowX<T>& x, const TW& tw, T q, T m2, int blk) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int h = 8 >> b;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) B::fwd_bfly(v[i], v[i + h], tw_a(tw, b, blk, i >> (4 - b)), q, m2);
    }
    reduce_wide<TW>(v, q, m2);
    __syncwarp();
    x.put_strided(v);
    __syncwarp();
    x.get_contiguous(v);
  }
  __device__ __forceinline__ static void fwd_b(T (&v)[16], const RowX<T>& x, const TW& tw, T q, T m2, int blk) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int h = 8 >> b;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) B::fwd_bfly(v[i], v[i + h], tw_b(tw, b, blk, x.t, i >> (4 - b)), q, m2);
    }
    reduce_wide<TW>(v, q, m2);
  }
  __device__ __forceinline__ static void fwd(T (&v)[16], const RowX<T>& x, const TW& tw, T q, T m2, int blk) {
    fwd_a(v, x, tw, q, m2, blk);
    fwd_b(v, x, tw, q, m2, blk);
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
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int h = 1 << j;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) B::inv_bfly(v[i], v[i + h], tw_b(tw, 3 - j, blk, x.t, i >> (j + 1)), q, m2);
      if (j == 1) reduce_wide_sums<TW>(v, q, m2);
    }
    reduce_grown<TW, T, 4>(v, q, m2);
    __syncwarp();
    x.put_contiguous(v);
    __syncwarp();
    x.get_strided(v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int h = 1 << j;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) B::inv_bfly(v[i], v[i + h], tw_a(tw, 3 - j, blk, i >> (j + 1)), q, m2);
      if (j == 1) reduce_wide_sums<TW>(v, q, m2);
    }
    reduce_grown<TW, T, 4>(v, q, m2);
  }
};

// ---------------------------------------------------------------------------
// Key switch.  The rows in flight are f_cnt FP64 rows from f_lo and i_cnt
// integer rows from i_lo, the integer ones spread evenly among the others
// (ks_unit).  In the columns launch neighbouring blocks are of both kinds, so
// that the FP64 and the integer pipe work side by side; the rows launch takes
// row after row.  Y holds, per (digit a, ciphertext b, row), the polynomial
// between the launches: Y[(a y_batch + b) y_rows + slot][N], slot the row
// itself (by_row: Y covers every row) or its place among the rows in flight.
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
  int batch, y_batch, y_rows, by_row, q_limbs, qp_limbs, level, qp0, ext_digits, f64_end;
  int f_lo, f_cnt, i_lo, i_cnt;
  int terms;            // > 1: accumulator bi sums the key switches of ciphertexts g batch + bi of Y
                        // (g < terms), each with the key item_keys[g]
  int keys_by_term;     // item_keys holds one key per term (also a single one) instead of one per ciphertext
  ChainTables<T> tabs;
  LevelTables<T> lt;
  ChainTables<double> tabs64f;
  const TwPair<double>* ext64f;
  __host__ __device__ int rows() const { return f_cnt + i_cnt; }
  __device__ __forceinline__ T* y_poly(int a, int bi, int jrow, bool f64, int log_n) const {
    const int slot = by_row ? jrow : (f64 ? jrow - f_lo : f_cnt + jrow - i_lo);
    return y + (((int64_t(a) * y_batch + bi) * y_rows + slot) << log_n);
  }
};

// Unit p of `total` of which `ints` are integer ones, spread evenly: true and
// the index among the integer ones, or false and the index among the others.
__device__ __forceinline__ bool ks_unit(int p, int total, int ints, int& index) {
  const int before = int(unsigned(p * ints) / unsigned(total)), after = int(unsigned((p + 1) * ints) / unsigned(total));
  index = after > before ? before : p - before;
  return after > before;
}

// True when row pid's own digit residue replaces the transform (relinearisation).
template <typename T>
__device__ __forceinline__ bool ks_own(const KsPass<T>& k, const DigitDesc& d, int jrow) {
  const int pid = k.level + jrow;
  return k.ct3 != nullptr && jrow < k.q_limbs && pid >= d.prime0 && pid < d.prime0 + d.alpha;
}

// Exact extension of a digit of at most four primes below 2^42 to a prime
// p < 2^42, in FP64: d_0 + sum_{r >= 1} d_r M_r (M_0 = 1) with one reduction.
// The products are summed in T on top of 1.5 2^88, so every T is a multiple
// of 2^36 in one binade (the sum stays below 2^87): the differences of
// successive T are exact, and d_r M_r minus that difference, at most 2^35 in
// magnitude, is exact too (fma).  With H the sum of the differences,
// H - rint(H / p) p lies in (-0.51 p, 0.51 p) and the result below
// 0.51 p + 2^42 + 2^37.  14 operations for four primes, where a reduction per
// product takes 27.
template <int ALPHA>
__device__ __forceinline__ double ext_chain(const double (&d)[ALPHA], const double (&m)[4], double q, double qinv) {
  if constexpr (ALPHA == 1) return d[0];
  constexpr double kBig = 1.5 * 309485009821345068724781056.0;  // 1.5 2^88
  double t = kBig, low = d[0];
#pragma unroll
  for (int r = 1; r < ALPHA; ++r) {
    const double next = fma(d[r], m[r], t);
    low += fma(d[r], m[r], t - next);
    t = next;
  }
  const double h = t - kBig;
  return fma(-Word<double>::mul_round(h, qinv), q, h) + low;
}

// The extensions to two primes of 16 words `stride` apart.
template <int ALPHA, int LOGN>
__device__ __forceinline__ void ext_pair(const uint64_t* __restrict__ p, int stride, const double (&m0)[4],
                                         const double (&m1)[4], double q0, double qi0, double q1, double qi1,
                                         double (&x0)[16], double (&x1)[16]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint64_t w[ALPHA][8];
#pragma unroll
    for (int r = 0; r < ALPHA; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e) w[r][e] = __ldg(p + (int64_t(r) << LOGN) + (h * 8 + e) * stride);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      double d[ALPHA];
#pragma unroll
      for (int r = 0; r < ALPHA; ++r) d[r] = Word<double>::from_word(w[r][e]);
      x0[h * 8 + e] = ext_chain<ALPHA>(d, m0, q0, qi0);
      x1[h * 8 + e] = ext_chain<ALPHA>(d, m1, q1, qi1);
    }
  }
}

// A column source that hands out 16 words already in registers.
struct RegSource {
  const double (&v)[16];
  template <int C>
  __device__ __forceinline__ void column(int, int, double (&x)[C]) const {
    static_assert(C == 16, "one group of 16 words per thread");
#pragma unroll
    for (int k = 0; k < C; ++k) x[k] = v[k];
  }
};

// Two FP64 rows of one (digit, ciphertext, column tile): the digit's words
// are loaded and converted once for both.  Rows not live (own-digit rows, the
// missing partner of an odd row) are not transformed.
template <int LOGN>
__device__ __forceinline__ void ks_columns_pair(const KsPass<uint64_t>& k, const DigitDesc& d, int a, int bi, int col0,
                                                int j0, int j1, bool live0, bool live1, double* s) {
  using G = ColGeom<uint64_t, LOGN>;
  using C = Cols<double, LOGN, TwAtQ>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  if (!live0) j0 = j1;
  if (!live1) j1 = j0;
  const int p0 = k.level + j0, p1 = k.level + j1;
  const double q0 = k.tabs64f.prime[p0].q, qi0 = k.tabs64f.prime[p0].one_s;
  const double q1 = k.tabs64f.prime[p1].q, qi1 = k.tabs64f.prime[p1].one_s;
  const TwPair<double>* ext = k.ext64f + (((int64_t(k.level) * k.ext_digits + a) * kMaxDigitWidth) * 2 + 1) * k.qp0;
  double m0[4], m1[4];
#pragma unroll
  for (int r = 1; r < 4; ++r) {
    m0[r] = r < d.alpha ? ext[int64_t(2 * r) * k.qp0 + p0].w : 0.0;
    m1[r] = r < d.alpha ? ext[int64_t(2 * r) * k.qp0 + p1].w : 0.0;
  }
  m0[0] = m1[0] = 1.0;
  int row0, hi, col;
  C::template group<4, G::kA - 4>(0, row0, hi, col);
  const uint64_t* p = k.digits + (int64_t(bi) * k.q_limbs + (d.prime0 - k.level)) * kN + row0 * kBlk + col0 + col;
  constexpr int kStride = kBlk << (G::kA - 4);
  double x0[16], x1[16];
  if (d.alpha == 4) {
    ext_pair<4, LOGN>(p, kStride, m0, m1, q0, qi0, q1, qi1, x0, x1);
  } else if (d.alpha == 3) {
    ext_pair<3, LOGN>(p, kStride, m0, m1, q0, qi0, q1, qi1, x0, x1);
  } else if (d.alpha == 2) {
    ext_pair<2, LOGN>(p, kStride, m0, m1, q0, qi0, q1, qi1, x0, x1);
  } else {
    ext_pair<1, LOGN>(p, kStride, m0, m1, q0, qi0, q1, qi1, x0, x1);
  }
  const TwAtQ tw0{k.tabs64f.twv_fwd + int64_t(p0) * kN, qi0}, tw1{k.tabs64f.twv_fwd + int64_t(p1) * kN, qi1};
  ColSink<double> sink0{reinterpret_cast<double*>(k.y_poly(a, bi, j0, true, LOGN))};
  ColSink<double> sink1{reinterpret_cast<double*>(k.y_poly(a, bi, j1, true, LOGN))};
  RegSource r0{x0}, r1{x1};
  double* s1 = s + G::kTile;
  if (live0) C::template fwd_pass<0>(r0, sink0, s, tw0, q0, qi0, col0);
  if (live1) C::template fwd_pass<0>(r1, sink1, s1, tw1, q1, qi1, col0);
  if constexpr (G::kPasses > 1) {
    __syncthreads();
    if (live0) C::template fwd_pass<1>(r0, sink0, s, tw0, q0, qi0, col0);
    if (live1) C::template fwd_pass<1>(r1, sink1, s1, tw1, q1, qi1, col0);
  }
}

template <typename T, int LOGN>
constexpr size_t ks_columns_smem(bool split) {
  return ColGeom<T, LOGN>::smem_bytes() * (split && ColGeom<T, LOGN>::kPasses <= 2 ? 2 : 1);
}

struct WideRowSource {
  const uint64_t* in;
  double q;
  template <int C>
  __device__ __forceinline__ void column(int m, int stride, double (&x)[C]) const {
#pragma unroll
    for (int k = 0; k < C; ++k) x[k] = Word<double>::from_word_minus(in[k * stride + m], q);
  }
};
struct WideExtSource {
  ExtSource<uint64_t> ext;
  double q;
  template <int C>
  __device__ __forceinline__ void column(int m, int stride, double (&x)[C]) const {
    uint64_t w[C];
    ext.column(m, stride, w);
#pragma unroll
    for (int k = 0; k < C; ++k) x[k] = Word<double>::from_word_minus(w[k], q);
  }
};

// Launch 1, one column tile: extension of digit a of ciphertext bi to the
// primes of FP64 rows j0, j1 (each if live) and the column stages of their
// forward transforms.  PRE: Y already holds the extensions (tensor-core basis
// conversion), transformed in place.
template <int LOGN, bool PRE, bool WIDE>
__device__ __forceinline__ void ks_columns_f64(const KsPass<uint64_t>& k, int a, int bi, int col0, int j0, int j1,
                                               bool live0, bool live1, unsigned char* smem) {
  using G = ColGeom<uint64_t, LOGN>;
  using TW = TwQ<WIDE>;
  using C = Cols<double, LOGN, TW>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  if (!live0 && !live1) return;
  const DigitDesc d = k.lt.digits[a];
  double* s = reinterpret_cast<double*>(smem);
  if constexpr (!PRE && !WIDE && G::kPasses <= 2) {
    if (d.alpha <= 4 && d.prime0 + d.alpha <= k.f64_end) {
      ks_columns_pair<LOGN>(k, d, a, bi, col0, j0, j1, live0, live1, s);
      return;
    }
  }
  for (int i = 0; i < 2; ++i) {
    const int jrow = i ? j1 : j0, pid = k.level + jrow;
    if (!(i ? live1 : live0)) continue;
    if (i) __syncthreads();  // the first row's words have been read
    const double q = k.tabs64f.prime[pid].q, qinv = k.tabs64f.prime[pid].one_s;
    uint64_t* y = k.y_poly(a, bi, jrow, true, LOGN);
    ColSink<double> sink{reinterpret_cast<double*>(y)};
    const TW tw{k.tabs64f.twv_fwd + int64_t(pid) * kN, qinv};
    if constexpr (PRE && WIDE) {
      WideRowSource src{y, q};
      C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
    } else if constexpr (WIDE) {  // the integer extension, below 2q
      const PrimeInfo<uint64_t>& p = k.tabs.prime[pid];
      WideExtSource src{ExtSource<uint64_t>{k.digits + (int64_t(bi) * k.q_limbs + (d.prime0 - k.level)) * kN,
                                            k.lt.ext + int64_t(a) * kMaxDigitWidth * k.qp0 + pid, k.qp0, d.alpha, LOGN,
                                            p.q, p.twice_q},
                        q};
      C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
    } else if constexpr (PRE) {
      U64RowSource src{y};
      C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
    } else {
      ExtSourceF64 src{k.digits + (int64_t(bi) * k.q_limbs + (d.prime0 - k.level)) * kN,
                       k.ext64f + (((int64_t(k.level) * k.ext_digits + a) * kMaxDigitWidth) * 2) * k.qp0 + pid, k.qp0,
                       d.alpha, LOGN, d.prime0 + d.alpha > k.f64_end, q, qinv};
      C::template fwd<0>(src, sink, s, tw, q, qinv, col0);
    }
  }
}

// The same for one integer row.
template <typename T, int LOGN, bool PRE>
__device__ __forceinline__ void ks_columns_int(const KsPass<T>& k, int a, int bi, int col0, int jrow,
                                               unsigned char* smem) {
  using C = Cols<T, LOGN, TwAt<T>>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  const DigitDesc d = k.lt.digits[a];
  if (ks_own(k, d, jrow)) return;
  const int pid = k.level + jrow;
  const T q = k.tabs.prime[pid].q, twoq = k.tabs.prime[pid].twice_q;
  T* y = k.y_poly(a, bi, jrow, false, LOGN);
  ColSink<T> sink{y};
  T* s = reinterpret_cast<T*>(smem);
  const TwAt<T> tw{k.tabs.tw_fwd + int64_t(pid) * kN};
  if constexpr (PRE) {
    ColSource<T> src{y};
    C::template fwd<0>(src, sink, s, tw, q, twoq, col0);
  } else {
    ExtSource<T> src{k.digits + (int64_t(bi) * k.q_limbs + (d.prime0 - k.level)) * kN,
                     k.lt.ext + int64_t(a) * kMaxDigitWidth * k.qp0 + pid, k.qp0, d.alpha, LOGN, q, twoq};
    C::template fwd<0>(src, sink, s, tw, q, twoq, col0);
  }
}

// One block per (digit, ciphertext, column tile, two FP64 rows or one integer
// row), rows fastest, so the blocks in flight share the digit's words in L2.
template <typename T, int LOGN, bool PRE, int SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(SPLIT == kNarrowF64 && !PRE))
k_ks_columns(const __grid_constant__ KsPass<T> k) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int units = (k.f_cnt + 1) / 2 + k.i_cnt;
  unsigned idx = blockIdx.x;
  int at;
  const bool is_int = ks_unit(int(idx % unsigned(units)), units, k.i_cnt, at);
  idx /= unsigned(units);
  const int col0 = int(idx % G::kTiles) * G::kCols;
  idx /= G::kTiles;
  const int bi = int(idx % unsigned(k.batch)), a = int(idx / unsigned(k.batch));
  if constexpr (SPLIT) {
    static_assert(sizeof(T) == 8, "FP64 rows exist in int64 chains only");
    if (!is_int) {
      const DigitDesc d = k.lt.digits[a];
      const int j0 = k.f_lo + 2 * at, j1 = j0 + 1;
      ks_columns_f64<LOGN, PRE, SPLIT == kWideF64>(k, a, bi, col0, j0, j1, !ks_own(k, d, j0),
                                2 * at + 1 < k.f_cnt && !ks_own(k, d, j1), smem_raw);
      return;
    }
  }
  ks_columns_int<T, LOGN, PRE>(k, a, bi, col0, k.i_lo + at, smem_raw);
}

// x k 2^-W mod q (W the word's bits) in (0, 2q) for x < 4q, k < 2q: one
// high product and a subtraction instead of the masked carries of a
// reduction by R = 2^(W - 2); qi = q^{-1} mod 2^W.
__device__ __forceinline__ uint64_t redc_word(uint64_t x, uint64_t k, uint64_t q, uint64_t qi) {
  const unsigned __int128 p = static_cast<unsigned __int128>(x) * k;
  return uint64_t(p >> 64) - __umul64hi(uint64_t(p) * qi, q) + q;
}
__device__ __forceinline__ uint32_t redc_word(uint32_t x, uint32_t k, uint32_t q, uint32_t qi) {
  const uint64_t p = static_cast<uint64_t>(x) * k;
  return uint32_t(p >> 32) - __umulhi(uint32_t(p) * qi, q) + q;
}
// q^{-1} mod 2^W from -q^{-1} mod 2^(W - 2) (one Newton step doubles the bits)
template <typename T>
__device__ __forceinline__ T inverse_pow2(T q, T neg_inv) {
  const T x = T(0) - neg_inv;
  return x * (T(2) - q * x);
}

// Launch 2: for one row of 256 words of (ciphertext, row j): the block stages
// of every digit's forward transform, the products with both key components
// summed in registers, and the block stages of both inverse transforms.  Half
// a warp per (ciphertext, 256 words), ciphertexts fastest, so that the half
// warps of a block read the same key words and twiddles.
template <int LOGN, bool WIDE, bool SHARED>
__device__ __forceinline__ void ks_rows_f64(const KsPass<uint64_t>& k, int jrow, int bi, int blk,
                                            unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  using W = Word<double>;
  using TW = TwQ<WIDE>;
  using R = Rows<double, LOGN, TW>;
  const int pid = k.level + jrow;
  const PrimeInfo<double>& p = k.tabs64f.prime[pid];
  const double q = p.q, qinv = p.one_s;
  const RowX<double> x(smem);
  const int vec = blk * kBlk + 2 * x.t;  // this thread's first word, vector layout
  const uint64_t* ct3 = k.ct3 ? k.ct3 + (int64_t(bi) * k.q_limbs + jrow) * kN + vec : nullptr;
  const TW twf{k.tabs64f.twrv_fwd + int64_t(pid) * kN, qinv};
  const RowStage<double> stage(smem + kRowSlots * kBlk * sizeof(double));
  int next = 0;  // the term whose row is requested next
  auto request = [&](int a) {  // digit a's row, unless its residue is the ciphertext's own
    if (!SHARED && a == k.lt.num_digits && ++next < k.terms) a = 0;
    if (a < k.lt.num_digits && x.t == 0) {  // and its keys
      const uint64_t* key = k.item_keys ? reinterpret_cast<const uint64_t*>(k.item_keys[k.keys_by_term ? next : bi]) : k.key;
      key += (int64_t(k.lt.digits[a].key_digit) * 2 * k.qp0 + pid) * kN + blk * kBlk;
      prefetch_row(key);
      prefetch_row(key + k.qp0 * kN);
    }
    if (a < k.lt.num_digits && !ks_own(k, k.lt.digits[a], jrow))
      stage.request(reinterpret_cast<const double*>(k.y_poly(a, next * k.batch + bi, jrow, true, LOGN)) + blk * kBlk);
  };
  const int warp = int(threadIdx.x >> 5), a_first = SHARED ? warp : 0, a_step = SHARED ? kRowWarps : 1;
  request(a_first);
  double a0[16], a1[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) a0[e] = a1[e] = 0.0;
  for (int g = 0; g < k.terms; ++g) {
    const uint64_t* key = k.item_keys ? reinterpret_cast<const uint64_t*>(k.item_keys[k.keys_by_term ? g : bi]) : k.key;
#pragma unroll 1
    for (int a = a_first; a < k.lt.num_digits; a += a_step) {
      const DigitDesc d = k.lt.digits[a];
      const uint64_t* key0 = key + ((int64_t(d.key_digit) * 2) * k.qp0 + pid) * kN + vec;
      const uint64_t* key1 = key0 + k.qp0 * kN;
      double v[16];
      uint4 u[8];  // the first component's key words, then the second's, loaded ahead
      auto load = [&](const uint64_t* key) {
#pragma unroll
        for (int e = 0; e < 8; ++e) u[e] = load_ahead(key + 32 * e);
      };
      auto lo = [&](const uint4& w) { return f64_word<WIDE>(uint64_t(w.y) << 32 | w.x, q); };
      auto hi = [&](const uint4& w) { return f64_word<WIDE>(uint64_t(w.w) << 32 | w.z, q); };
      if (ks_own(k, d, jrow)) {
        load(key0);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(ct3 + 2 * k.ct3_stride + 32 * e));
          v[2 * e] = W::shoup_bal(f64_word<WIDE>(w.x, q), p.rinv, p.rinv_s, q);
          v[2 * e + 1] = W::shoup_bal(f64_word<WIDE>(w.y, q), p.rinv, p.rinv_s, q);
        }
        request(a + a_step);
      } else {
        stage.take(v);
        request(a + a_step);
        R::fwd_a(v, x, twf, q, qinv, blk);
        load(key0);
        R::fwd_b(v, x, twf, q, qinv, blk);
        R::contiguous_to_vector(v, x);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        a0[2 * e] += W::mul_qinv_bal(v[2 * e], lo(u[e]), q, qinv);
        a0[2 * e + 1] += W::mul_qinv_bal(v[2 * e + 1], hi(u[e]), q, qinv);
        u[e] = load_ahead(key1 + 32 * e);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        a1[2 * e] += W::mul_qinv_bal(v[2 * e], lo(u[e]), q, qinv);
        a1[2 * e + 1] += W::mul_qinv_bal(v[2 * e + 1], hi(u[e]), q, qinv);
      }
      if (WIDE && (SHARED || (a & 3) == 3 || a + 1 == k.lt.num_digits)) {  // at most four terms of 0.68 q
        reduce_wide<TW>(a0, q, qinv);
        reduce_wide<TW>(a1, q, qinv);
      }
    }
    if (!WIDE && k.terms > 1) {  // at most 17 digits a term: the sums stay below 2^48
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        a0[e] = W::reduce_bal(a0[e], q, qinv);
        a1[e] = W::reduce_bal(a1[e], q, qinv);
      }
    }
  }
  const TW twi{k.tabs64f.twrv_inv + int64_t(pid) * kN, qinv};
  auto finish = [&](double (&v)[16], const uint64_t* add, uint64_t* out) {
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = W::reduce_bal(v[e], q, qinv);
    if (add) {  // P c_k, carrying R like the sums
      const TwPair<double> pc = k.tabs64f.p_rinv[pid];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(add + 32 * e));
        v[2 * e] += W::shoup_bal(f64_word<WIDE>(w.x, q), pc.w, pc.wp, q);
        v[2 * e + 1] += W::shoup_bal(f64_word<WIDE>(w.y, q), pc.w, pc.wp, q);
      }
      reduce_wide<TW>(v, q, qinv);
    }
    R::vector_to_contiguous(v, x);
    R::inv(v, x, twi, q, qinv, blk);
    double* o = reinterpret_cast<double*>(out) + (int64_t(bi) * k.qp_limbs + jrow) * kN + blk * kBlk + x.t;
#pragma unroll
    for (int e = 0; e < 16; ++e) o[16 * e] = v[e];
  };
  if constexpr (SHARED) {  // the warps' partial sums: warp 0 takes component 0, warp 1 component 1
    double* part = reinterpret_cast<double*>(smem);
    constexpr int kWarpWords = 2 * kBlk;
    const int lane = int(threadIdx.x & 31), mine = warp & 1;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      part[(warp * 2) * kWarpWords + e * 32 + lane] = a0[e];
      part[(warp * 2 + 1) * kWarpWords + e * 32 + lane] = a1[e];
      a0[e] = 0;
    }
    __syncthreads();
    for (int w = 0; w < kRowWarps; ++w)
#pragma unroll
      for (int e = 0; e < 16; ++e) a0[e] += part[(w * 2 + mine) * kWarpWords + e * 32 + lane];
    __syncthreads();
    if (warp < 2) finish(a0, mine && ct3 ? ct3 + k.ct3_stride : ct3, mine ? k.acc1 : k.acc0);
  } else {
    finish(a0, ct3, k.acc0);
    finish(a1, ct3 ? ct3 + k.ct3_stride : nullptr, k.acc1);
  }
}

template <typename T, int LOGN, bool SHARED>
__device__ __forceinline__ void ks_rows_int(const KsPass<T>& k, int jrow, int bi, int blk,
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
  const T* ct3 = k.ct3 && jrow < k.q_limbs ? k.ct3 + (int64_t(bi) * k.q_limbs + jrow) * kN + vec : nullptr;
  auto piece = [](const T* at) {
    Piece r;
    *reinterpret_cast<uint4*>(r.v) = __ldg(reinterpret_cast<const uint4*>(at));
    return r;
  };
  const TwAt<T> twf{k.tabs.twr_fwd + int64_t(pid) * kN};
  const RowStage<T> stage(smem + kRowSlots * kBlk * sizeof(T));
  int next = 0;
  auto request = [&](int a) {
    if (!SHARED && a == k.lt.num_digits && ++next < k.terms) a = 0;
    if (a < k.lt.num_digits && x.t == 0) {
      const T* key = k.item_keys ? reinterpret_cast<const T*>(k.item_keys[k.keys_by_term ? next : bi]) : k.key;
      key += (int64_t(k.lt.digits[a].key_digit) * 2 * k.qp0 + pid) * kN + blk * kBlk;
      prefetch_row(key);
      prefetch_row(key + k.qp0 * kN);
    }
    if (a < k.lt.num_digits && !ks_own(k, k.lt.digits[a], jrow))
      stage.request(k.y_poly(a, next * k.batch + bi, jrow, false, LOGN) + blk * kBlk);
  };
  const int warp = int(threadIdx.x >> 5), a_first = SHARED ? warp : 0, a_step = SHARED ? kRowWarps : 1;
  request(a_first);
  const T qi = inverse_pow2(q, ni);
  T a0[16], a1[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) a0[e] = a1[e] = 0;
  for (int g = 0; g < k.terms; ++g) {
    const T* key = k.item_keys ? reinterpret_cast<const T*>(k.item_keys[k.keys_by_term ? g : bi]) : k.key;
#pragma unroll 1
    for (int a = a_first; a < k.lt.num_digits; a += a_step) {
      const DigitDesc d = k.lt.digits[a];
      T v[16];
      if (ks_own(k, d, jrow)) {
#pragma unroll
        for (int e = 0; e < X::kVec; ++e) {
          const Piece w = piece(ct3 + 2 * k.ct3_stride + 16 * X::V * e);
#pragma unroll
          for (int i = 0; i < X::V; ++i) v[e * X::V + i] = W::shoup(w.v[i], p.rinv, p.rinv_s, q);
        }
        request(a + a_step);
      } else {
        stage.take(v);
        request(a + a_step);
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
          a0[at] = csub(a0[at] + redc_word(v[at], u0.v[i], q, qi), twoq);
          a1[at] = csub(a1[at] + redc_word(v[at], u1.v[i], q, qi), twoq);
        }
      }
    }
  }
  const TwAt<T> twi{k.tabs.twr_inv + int64_t(pid) * kN};
  auto finish = [&](T (&v)[16], const T* add, T* out) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {  // x 4: the products were reduced by 2^W, not by R = 2^(W - 2)
      v[e] = csub(v[e] + v[e], twoq);
      v[e] = csub(v[e] + v[e], twoq);
    }
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
#pragma unroll
    for (int e = 0; e < 16; ++e) o[16 * e] = v[e];
  };
  if constexpr (SHARED) {  // the warps' partial sums: warp 0 takes component 0, warp 1 component 1
    T* part = reinterpret_cast<T*>(smem);
    constexpr int kWarpWords = 2 * kBlk;
    const int lane = int(threadIdx.x & 31), mine = warp & 1;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      part[(warp * 2) * kWarpWords + e * 32 + lane] = a0[e];
      part[(warp * 2 + 1) * kWarpWords + e * 32 + lane] = a1[e];
      a0[e] = 0;
    }
    __syncthreads();
    for (int w = 0; w < kRowWarps; ++w)
#pragma unroll
      for (int e = 0; e < 16; ++e) a0[e] = csub(a0[e] + part[(w * 2 + mine) * kWarpWords + e * 32 + lane], twoq);
    __syncthreads();
    if (warp < 2) finish(a0, mine && ct3 ? ct3 + k.ct3_stride : ct3, mine ? k.acc1 : k.acc0);
  } else {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {  // one copy of the code: 348 -> 327 us for 5 rows, batch 8; FP64 rows lose (763 -> 795)
      finish(a0, c && ct3 ? ct3 + k.ct3_stride : ct3, c ? k.acc1 : k.acc0);
#pragma unroll
      for (int e = 0; e < 16; ++e) a0[e] = a1[e];
    }
  }
}

template <typename T>
constexpr size_t row_smem() {
  return size_t(2 * kRowSlots) * kBlk * sizeof(T);  // exchanges and the next rows
}

// SHARED: a block takes the rows of one warp only and deals the digits to its
// four warps, whose sums meet in shared memory; two warps then finish a
// component each.  For launches that do not fill the GPU: the
// digits are a serial chain of loads and exchanges otherwise (N = 2^14, one
// ciphertext: 47.9 -> 25.6 us).
template <typename T, int LOGN, int SPLIT, bool SHARED>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 3 : 4)
k_ks_rows(const __grid_constant__ KsPass<T> k) {
  __shared__ __align__(16) unsigned char smem[row_smem<T>()];
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  const unsigned slots = unsigned(kBlks) * unsigned(k.batch);
  // Rows one after the other: the blocks in flight share a row's keys and
  // twiddles, and an SM runs one of the two bodies at a time (integer blocks
  // dealt out among the FP64 ones measured 25 % slower: the bodies evict each
  // other from the instruction caches).
  static_assert(kBlks % kRowSlots == 0, "a block's half warps all have a row");
  const unsigned per_block = SHARED ? 2 : kRowSlots, per_row = slots / per_block;
  int at;
  const bool is_int = ks_unit(int(blockIdx.x / per_row), k.rows(), k.i_cnt, at);
  const int jrow = at + (is_int ? k.i_lo : k.f_lo);
  const unsigned slot = blockIdx.x % per_row * per_block + ((threadIdx.x >> 4) & (per_block - 1));
  const int bi = int(slot % unsigned(k.batch)), blk = int(slot / unsigned(k.batch));
  if constexpr (SPLIT) {
    static_assert(sizeof(T) == 8, "FP64 rows exist in int64 chains only");
    if (!is_int) {
      ks_rows_f64<LOGN, SPLIT == kWideF64, SHARED>(k, jrow, bi, blk, smem);
      return;
    }
  }
  ks_rows_int<T, LOGN, SHARED>(k, jrow, bi, blk, smem);
}

// Launch 3: one column tile of the inverse transform of the accumulator row z
// of prime pid, in place, to canonical coefficients.
template <typename T, int LOGN, int SPLIT>
__device__ __forceinline__ void ks_columns_inverse(T* z, int pid, bool f64, const ChainTables<T>& tabs,
                                                   const ChainTables<double>& tabs64f, int col0,
                                                   unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  if constexpr (SPLIT) {
    if (f64) {
      const PrimeInfo<double>& p = tabs64f.prime[pid];
      ColSource<double> src{reinterpret_cast<double*>(z)};
      F64InvEpilogue epi{reinterpret_cast<uint64_t*>(z), p.q, p.ninv_rinv, p.ninv_rinv_s};
      Cols<double, LOGN, TwQ<SPLIT == kWideF64>>::template inv<0>(src, epi, reinterpret_cast<double*>(smem),
                                                 TwQ<SPLIT == kWideF64>{tabs64f.twv_inv + int64_t(pid) * kN, p.one_s}, p.q, p.one_s,
                                                 col0);
      return;
    }
  }
  const PrimeInfo<T>& p = tabs.prime[pid];
  ColSource<T> src{z};
  InvEpilogue<T> epi{z, p.q, p.ninv, p.ninv_s, kInvStandard};
  Cols<T, LOGN, TwAt<T>>::template inv<0>(src, epi, reinterpret_cast<T*>(smem),
                                          TwAt<T>{tabs.tw_inv + int64_t(pid) * kN}, p.q, p.twice_q, col0);
}

// One block per (component, ciphertext, row, column tile).
template <typename T, int LOGN, int SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(false))
k_ks_columns_inverse(const __grid_constant__ KsPass<T> k) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned idx = blockIdx.x;
  const int col0 = int(idx % G::kTiles) * G::kCols;
  idx /= G::kTiles;
  int at;
  const bool is_int = ks_unit(int(idx % unsigned(k.rows())), k.rows(), k.i_cnt, at);
  const int jrow = at + (is_int ? k.i_lo : k.f_lo);
  idx /= unsigned(k.rows());
  const int bi = int(idx % unsigned(k.batch));
  T* z = (idx / unsigned(k.batch) ? k.acc1 : k.acc0) + ((int64_t(bi) * k.qp_limbs + jrow) << LOGN);
  ks_columns_inverse<T, LOGN, SPLIT>(z, k.level + jrow, !is_int, k.tabs, k.tabs64f, col0, smem_raw);
}

// ---------------------------------------------------------------------------
// Standalone transforms of polynomials [polys][N], poly p of row p mod rows
// (prime row_start + row); the leading f64_rows rows of every group in FP64.
// Both directions hold the intermediate in `out`.
template <bool TO_MONT>
struct WordSource {  // 64-bit words of a prime below 2^42 as balanced doubles
  const uint64_t* in;
  double c, cs, q;
  template <int C>
  __device__ __forceinline__ void column(int m, int stride, double (&x)[C]) const {
#pragma unroll
    for (int k = 0; k < C; ++k) {
      x[k] = Word<double>::from_word(in[k * stride + m]);
      if constexpr (TO_MONT) x[k] = Word<double>::shoup_bal(x[k], c, cs, q);
    }
  }
};

// One column tile of the forward transform of the polynomial `in` of prime
// pid into `out` (f64: FP64 arithmetic, the intermediate in doubles).
template <typename T, int LOGN, bool TO_MONT, int SPLIT>
__device__ __forceinline__ void ntt_columns(const T* in, T* out, int pid, bool f64, const ChainTables<T>& tabs,
                                            const ChainTables<double>& tabs64f, int col0, unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  if constexpr (SPLIT) {
    if (f64) {
      const PrimeInfo<double>& p = tabs64f.prime[pid];
      WordSource<TO_MONT> src{in, p.rmod, p.rmod_s, p.q};
      ColSink<double> sink{reinterpret_cast<double*>(out)};
      Cols<double, LOGN, TwAtQ>::template fwd<0>(src, sink, reinterpret_cast<double*>(smem),
                                                 TwAtQ{tabs64f.twv_fwd + int64_t(pid) * kN, p.one_s}, p.q, p.one_s,
                                                 col0);
      return;
    }
  }
  const PrimeInfo<T>& p = tabs.prime[pid];
  RowSource<T, TO_MONT> src{in, p.rmod, p.rmod_s, p.q};
  ColSink<T> sink{out};
  Cols<T, LOGN, TwAt<T>>::template fwd<0>(src, sink, reinterpret_cast<T*>(smem),
                                          TwAt<T>{tabs.tw_fwd + int64_t(pid) * kN}, p.q, p.twice_q, col0);
}

// The block stages of the forward transform of row blk of `poly`, in place,
// to lazy words in [0, 2q).  Half a warp per row of 256 words.
template <typename T, int LOGN, int SPLIT>
__device__ __forceinline__ void ntt_rows(T* poly, int pid, bool f64, const ChainTables<T>& tabs,
                                         const ChainTables<double>& tabs64f, int blk, unsigned char* smem) {
  using X = RowX<T>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  const X x(smem);
  T* at = poly + blk * kBlk;
  T* dst = at + X::V * x.t;
  if constexpr (SPLIT) {
    if (f64) {
      const double q = tabs64f.prime[pid].q, qinv = tabs64f.prime[pid].one_s;
      const double* src = reinterpret_cast<const double*>(at) + x.t;
      const RowX<double> xd(smem);
      using R = Rows<double, LOGN, TwAtQ>;
      double v[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = src[16 * e];
      R::fwd(v, xd, TwAtQ{tabs64f.twrv_fwd + int64_t(pid) * kN, qinv}, q, qinv, blk);
      R::contiguous_to_vector(v, xd);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        reinterpret_cast<ulonglong2*>(dst)[16 * e] =
            make_ulonglong2(Word<double>::to_word(Word<double>::to_lazy(v[2 * e], q, qinv)),
                            Word<double>::to_word(Word<double>::to_lazy(v[2 * e + 1], q, qinv)));
      return;
    }
  }
  const T q = tabs.prime[pid].q, twoq = tabs.prime[pid].twice_q;
  using R = Rows<T, LOGN, TwAt<T>>;
  T v[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] = at[x.t + 16 * e];
  R::fwd(v, x, TwAt<T>{tabs.twr_fwd + int64_t(pid) * kN}, q, twoq, blk);
  R::contiguous_to_vector(v, x);
#pragma unroll
  for (int e = 0; e < X::kVec; ++e) {
    typename X::Piece w;
#pragma unroll
    for (int i = 0; i < X::V; ++i) w.v[i] = csub(v[e * X::V + i], twoq);
    reinterpret_cast<typename X::Piece*>(dst)[16 * e] = w;
  }
}

// The block stages of the inverse transform of row blk, `in` to `out` (which
// may be the same buffer).
template <typename T, int LOGN, int SPLIT>
__device__ __forceinline__ void ntt_rows_inverse(const T* in, T* out, int pid, bool f64, const ChainTables<T>& tabs,
                                                 const ChainTables<double>& tabs64f, int blk, unsigned char* smem) {
  using X = RowX<T>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  const X x(smem);
  const typename X::Piece* src = reinterpret_cast<const typename X::Piece*>(in + blk * kBlk + X::V * x.t);
  T* dst = out + blk * kBlk + x.t;
  if constexpr (SPLIT) {
    if (f64) {
      const double q = tabs64f.prime[pid].q, qinv = tabs64f.prime[pid].one_s;
      const RowX<double> xd(smem);
      using TW = TwQ<SPLIT == kWideF64>;
      using R = Rows<double, LOGN, TW>;
      double v[16];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const typename X::Piece w = src[16 * e];
        v[2 * e] = f64_word<TW::kWide>(w.v[0], q);
        v[2 * e + 1] = f64_word<TW::kWide>(w.v[1], q);
      }
      reduce_wide<TW>(v, q, qinv);
      R::vector_to_contiguous(v, xd);
      R::inv(v, xd, TW{tabs64f.twrv_inv + int64_t(pid) * kN, qinv}, q, qinv, blk);
#pragma unroll
      for (int e = 0; e < 16; ++e) reinterpret_cast<double*>(dst)[16 * e] = v[e];
      return;
    }
  }
  using R = Rows<T, LOGN, TwAt<T>>;
  T v[16];
#pragma unroll
  for (int e = 0; e < X::kVec; ++e) {
    const typename X::Piece w = src[16 * e];
#pragma unroll
    for (int i = 0; i < X::V; ++i) v[e * X::V + i] = w.v[i];
  }
  R::vector_to_contiguous(v, x);
  R::inv(v, x, TwAt<T>{tabs.twr_inv + int64_t(pid) * kN}, tabs.prime[pid].q, tabs.prime[pid].twice_q, blk);
#pragma unroll
  for (int e = 0; e < 16; ++e) dst[16 * e] = v[e];
}

// Canonical (centred: signed) word of a balanced inverse transform's output.
// The lazy kinds get the canonical word too: their range is [0, 2q).
struct WordOutEpilogue {
  uint64_t* dst;
  double q, c, cs;
  bool centred;
  __device__ __forceinline__ void operator()(int pos, double v) const {
    v = Word<double>::shoup_bal(v, c, cs, q);  // (-0.6 q, 0.6 q)
    if (v < 0.0) v += q;
    const uint64_t w = Word<double>::to_word(v);
    dst[pos] = centred && v > floor(0.5 * q) ? w - uint64_t(q) : w;
  }
};

// One column tile of the inverse transform, in place.
template <typename T, int LOGN, int SPLIT>
__device__ __forceinline__ void ntt_columns_inverse(T* out, int pid, bool f64, int kind, const ChainTables<T>& tabs,
                                                    const ChainTables<double>& tabs64f, int col0,
                                                    unsigned char* smem) {
  constexpr int64_t kN = int64_t(1) << LOGN;
  if constexpr (SPLIT) {
    if (f64) {
      const PrimeInfo<double>& p = tabs64f.prime[pid];
      const bool std_out = kind != kInvMontgomery;  // N^-1 R^-1 unless the output stays Montgomery
      ColSource<double> src{reinterpret_cast<const double*>(out)};
      WordOutEpilogue epi{out, p.q, std_out ? p.ninv_rinv : p.ninv, std_out ? p.ninv_rinv_s : p.ninv_s,
                          kind == kInvCentered};
      Cols<double, LOGN, TwQ<SPLIT == kWideF64>>::template inv<0>(src, epi, reinterpret_cast<double*>(smem),
                                                 TwQ<SPLIT == kWideF64>{tabs64f.twv_inv + int64_t(pid) * kN, p.one_s}, p.q, p.one_s,
                                                 col0);
      return;
    }
  }
  const PrimeInfo<T>& p = tabs.prime[pid];
  ColSource<T> src{out};
  InvEpilogue<T> epi = make_inv_epilogue<T>(out, p, kind, true);
  Cols<T, LOGN, TwAt<T>>::template inv<0>(src, epi, reinterpret_cast<T*>(smem),
                                          TwAt<T>{tabs.tw_inv + int64_t(pid) * kN}, p.q, p.twice_q, col0);
}

template <typename T, int LOGN, bool TO_MONT, int SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(false))
k_ntt_columns(const T* in, T* out, int rows, int row_start, ChainTables<T> tabs, ChainTables<double> tabs64f,
              int f64_rows) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t poly = blockIdx.x / G::kTiles, at = poly << LOGN;
  const int row = int(poly % rows);
  ntt_columns<T, LOGN, TO_MONT, SPLIT>(in + at, out + at, row_start + row, row < f64_rows, tabs, tabs64f,
                                       int(blockIdx.x % G::kTiles) * G::kCols, smem_raw);
}

template <typename T, int LOGN, int SPLIT>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 5 : 8)
k_ntt_rows(T* out, int64_t slots, int rows, int row_start, ChainTables<T> tabs, ChainTables<double> tabs64f,
           int f64_rows) {
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  __shared__ __align__(16) unsigned char smem[exchange_smem<T>()];
  const int64_t slot = int64_t(blockIdx.x) * kRowSlots + (threadIdx.x >> 4);
  if (slot >= slots) return;  // a whole warp: a polynomial has an even number of rows of 256 words
  const int64_t poly = slot / kBlks;
  const int row = int(poly % rows);
  ntt_rows<T, LOGN, SPLIT>(out + (poly << LOGN), row_start + row, row < f64_rows, tabs, tabs64f, int(slot % kBlks),
                           smem);
}

template <typename T, int LOGN, int SPLIT>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 5 : 8)
k_ntt_rows_inverse(const T* in, T* out, int64_t slots, int rows, int row_start, ChainTables<T> tabs,
                   ChainTables<double> tabs64f, int f64_rows) {
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  __shared__ __align__(16) unsigned char smem[exchange_smem<T>()];
  const int64_t slot = int64_t(blockIdx.x) * kRowSlots + (threadIdx.x >> 4);
  if (slot >= slots) return;
  const int64_t poly = slot / kBlks, at = poly << LOGN;
  const int row = int(poly % rows);
  ntt_rows_inverse<T, LOGN, SPLIT>(in + at, out + at, row_start + row, row < f64_rows, tabs, tabs64f,
                                   int(slot % kBlks), smem);
}

template <typename T, int LOGN, int SPLIT>
__global__ void __launch_bounds__(ColGeom<T, LOGN>::kThreads, col_blocks<T, LOGN>(false))
k_ntt_columns_inverse(T* out, int rows, int row_start, int kind, ChainTables<T> tabs, ChainTables<double> tabs64f,
                      int f64_rows) {
  using G = ColGeom<T, LOGN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t poly = blockIdx.x / G::kTiles;
  const int row = int(poly % rows);
  ntt_columns_inverse<T, LOGN, SPLIT>(out + (poly << LOGN), row_start + row, row < f64_rows, kind, tabs, tabs64f,
                                      int(blockIdx.x % G::kTiles) * G::kCols, smem_raw);
}

// ---------------------------------------------------------------------------
// Hoisting stage 2, per rotation step: NTT-domain automorphism of the prepared
// digits, products with both key components, block stages of both inverse
// transforms (fhelium/engine/hybrid_keyswitch.py:419-469); the column stages
// follow in k_ks_columns_inverse.  The sources of 16 aligned destinations
// under the NTT-domain automorphism are a permutation of 16 aligned words
// (the low bits of k are the top bits of br(k), which the odd g permutes), so
// in the strided layout the gathers, like the key loads, are whole 128-byte
// lines.  y: the prepared digits [D_l, B, QP_l, N].  A thread takes its 16
// words in two halves, so that a digit's 24 loads fit the registers and can
// all be in flight (33 rows, three ciphertexts, 8 digits at N = 2^16:
// 350 -> 287 us a step).  Bound by the loads' latency: four blocks per SM
// spill (333 us), asking the next digit's lines into L2 adds instructions and
// no overlap (371 us).
template <typename T, int LOGN, int SPLIT>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 8 ? 3 : 4)
k_apply_rows(const __grid_constant__ KsPass<T> k, uint32_t galois) {
  using X = RowX<T>;
  constexpr int64_t kN = int64_t(1) << LOGN;
  constexpr int kBlks = 1 << (LOGN - kBlkLog);
  __shared__ __align__(16) unsigned char smem[exchange_smem<T>()];
  const unsigned slots = unsigned(kBlks) * unsigned(k.batch);  // even: whole warps
  const unsigned per_row = (slots + kRowSlots - 1) / kRowSlots;
  int at;
  const bool is_int = ks_unit(int(blockIdx.x / per_row), k.rows(), k.i_cnt, at);
  const int jrow = at + (is_int ? k.i_lo : k.f_lo), pid = k.level + jrow;
  const unsigned slot = blockIdx.x % per_row * kRowSlots + (threadIdx.x >> 4);
  if (slot >= slots) return;
  const int bi = int(slot % unsigned(k.batch)), blk = int(slot / unsigned(k.batch));
  const X x(smem);
  auto source = [&](int e) {  // the word gathered for this thread's word t + 16 e
    const int dst = blk * kBlk + x.t + 16 * e;
    return galois ? galois_ntt_source(dst, LOGN, galois) : dst;
  };
  const T* key = k.key + int64_t(pid) * kN + blk * kBlk + x.t;
  const int64_t o = (int64_t(bi) * k.qp_limbs + jrow) * kN + blk * kBlk + x.t;
  if constexpr (SPLIT) {
    if (!is_int) {
      using W = Word<double>;
      using TW = TwQ<SPLIT == kWideF64>;
      using R = Rows<double, LOGN, TW>;
      const RowX<double> xd(smem);
      const double q = k.tabs64f.prime[pid].q, qinv = k.tabs64f.prime[pid].one_s;
      double a0[16], a1[16];
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        int src[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) src[e] = source(h + e), a0[h + e] = a1[h + e] = 0.0;
#pragma unroll 1
        for (int a = 0; a < k.lt.num_digits; ++a) {
          const T* y = k.y_poly(a, bi, jrow, true, LOGN);
          const T* key0 = key + int64_t(k.lt.digits[a].key_digit) * 2 * k.qp0 * kN + 16 * h;
          const T* key1 = key0 + k.qp0 * kN;
          T w[8], k0[8], k1[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = __ldg(y + src[e]), k0[e] = __ldg(key0 + 16 * e), k1[e] = __ldg(key1 + 16 * e);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const double v = f64_word<TW::kWide>(w[e], q);
            a0[h + e] += W::mul_qinv_bal(v, f64_word<TW::kWide>(k0[e], q), q, qinv);
            a1[h + e] += W::mul_qinv_bal(v, f64_word<TW::kWide>(k1[e], q), q, qinv);
            if (TW::kWide && (a & 3) == 3) {  // four terms of at most 0.78 q
              a0[h + e] = W::reduce_bal(a0[h + e], q, qinv);
              a1[h + e] = W::reduce_bal(a1[h + e], q, qinv);
            }
          }
        }
      }
      const TW tw{k.tabs64f.twrv_inv + int64_t(pid) * kN, qinv};
      auto finish = [&](double (&v)[16], T* out) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = W::reduce_bal(v[e], q, qinv);
        R::strided_to_contiguous(v, xd);
        R::inv(v, xd, tw, q, qinv, blk);
#pragma unroll
        for (int e = 0; e < 16; ++e) reinterpret_cast<double*>(out + o)[16 * e] = v[e];
      };
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        finish(a0, c ? k.acc1 : k.acc0);
#pragma unroll
        for (int e = 0; e < 16; ++e) a0[e] = a1[e];
      }
      return;
    }
  }
  using R = Rows<T, LOGN, TwAt<T>>;
  const T q = k.tabs.prime[pid].q, twoq = k.tabs.prime[pid].twice_q;
  const T qi = inverse_pow2(q, k.tabs.prime[pid].neg_inv);
  T a0[16], a1[16];
#pragma unroll
  for (int h = 0; h < 16; h += 8) {
    int src[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) src[e] = source(h + e), a0[h + e] = a1[h + e] = 0;
#pragma unroll 1
    for (int a = 0; a < k.lt.num_digits; ++a) {
      const T* y = k.y_poly(a, bi, jrow, false, LOGN);
      const T* key0 = key + int64_t(k.lt.digits[a].key_digit) * 2 * k.qp0 * kN + 16 * h;
      const T* key1 = key0 + k.qp0 * kN;
      T w[8], k0[8], k1[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = __ldg(y + src[e]), k0[e] = __ldg(key0 + 16 * e), k1[e] = __ldg(key1 + 16 * e);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        a0[h + e] = csub(a0[h + e] + redc_word(w[e], k0[e], q, qi), twoq);
        a1[h + e] = csub(a1[h + e] + redc_word(w[e], k1[e], q, qi), twoq);
      }
    }
  }
  const TwAt<T> tw{k.tabs.twr_inv + int64_t(pid) * kN};
  auto finish = [&](T (&v)[16], T* out) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {  // x 4, as in ks_rows_int
      v[e] = csub(v[e] + v[e], twoq);
      v[e] = csub(v[e] + v[e], twoq);
    }
    R::strided_to_contiguous(v, x);
    R::inv(v, x, tw, q, twoq, blk);
#pragma unroll
    for (int e = 0; e < 16; ++e) out[o + 16 * e] = v[e];
  };
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    finish(a0, c ? k.acc1 : k.acc0);
#pragma unroll
    for (int e = 0; e < 16; ++e) a0[e] = a1[e];
  }
}

}  // namespace fhb
