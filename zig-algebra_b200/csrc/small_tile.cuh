// small_tile.cuh -- one tile of one pass of the small fields' transforms on
// sixteen elements per thread.
//
// The network and the pass structure are small.cu's.  A pass of K stages runs
// on whole tiles of 2^12 elements in CTAs of 256 threads, each thread holding
// the sixteen elements whose rows differ in four bits (the window): up to four
// stages in registers, then an exchange through shared memory to the next
// window.  The first window reads global memory and the last one writes it, so
// a pass of up to eight stages exchanges once, where groups of four elements
// staged by the tile exchanged five times; K and the windows are compile-time
// constants, and an address serves sixteen elements.  On radix-4 groups staged by
// the tile a butterfly took 48 instructions (BabyBear) and 77 (Goldilocks); here 16
// and 45.  BabyBear is bound by memory (2^24: three passes of 268 MB in 0.160 ms,
// 5.0 TB/s; 0.362 before), Goldilocks by its arithmetic on the ALU and multiply
// pipes (2^24 0.524 -> 0.382 ms; B200).
#pragma once

#include <cstdint>

#include "small_field.cuh"

namespace zntt {

struct SmallPass {
  const uint64_t* src;
  uint64_t* dst;
  const uint64_t* tw;  // table entries (SF::entry), stage s at entry 2^s - 1
  uint32_t log_n, S, k, c, first, inverse, tw0_one, scale;
  uint64_t scale_val;  // twiddle form
  uint32_t src_len;    // column launches' first pass: natural index >= src_len reads as zero
  const uint64_t* coset_pw;  // when not null: output i is scaled by shift^i from these power tables
};

__device__ __forceinline__ uint32_t rev_bits_small(uint32_t x, uint32_t bits) {
  return bits == 0 ? 0u : (__brev(x) >> (32 - bits));
}

constexpr int kTileLog = 12;
constexpr int kTileThreads = 256;

template <class SF, int K, bool FIRST, bool INV>
struct SmallTile {
  using word = typename SF::word;
  static constexpr int c = kTileLog - K;  // log2 of the columns of a tile
  static_assert(K >= 6 && K <= 10, "two or three windows");
  // Shared memory is padded by one element in sixteen, so that threads whose
  // elements lie 2^(c + 4) apart use different banks.
  static constexpr int kWords = (1 << kTileLog) + (1 << (kTileLog - 4));

  const SmallPass& pp;
  word* const sm;
  const uint64_t* src;
  uint64_t* dst;
  uint32_t hi_base = 0, m0 = 0, col0 = 0;

  __device__ __forceinline__ SmallTile(const SmallPass& p, const uint64_t* s, uint64_t* d, uint32_t blk, word* shared)
      : pp(p), sm(shared), src(s), dst(d) {
    if constexpr (FIRST) {
      col0 = blk << c;
    } else {
      const uint32_t mlog = pp.S - c;
      hi_base = (blk >> mlog) << (pp.S + K);
      m0 = (blk & ((1u << mlog) - 1)) << c;
    }
  }

  static __device__ __forceinline__ constexpr uint32_t rev4(uint32_t r) {
    return ((r & 1) << 3) | ((r & 2) << 1) | ((r & 4) >> 1) | (r >> 3);
  }

  // Stages LO+1 .. HI of the pass on the window of row bits [W, W + 4).
  template <int W, int LO, int HI, bool IN, bool OUT>
  __device__ __forceinline__ void window() const {
    constexpr int B = c + W;  // the window's lowest bit in a tile index
    const uint32_t tid = threadIdx.x;
    uint32_t eb;  // the thread's tile index with the window bits zero
    if constexpr (OUT && FIRST) {
      // Rows fastest: the first pass writes consecutive rows of a column.
      eb = ((tid & ((1u << (K - 4)) - 1)) << c) | (tid >> (K - 4));
    } else {
      eb = (tid & ((1u << B) - 1)) | ((tid >> B) << (B + 4));
    }
    const uint32_t col = eb & ((1u << c) - 1), row = eb >> c;
    const uint32_t sb = eb + (eb >> 4);
    word x[16];
    if constexpr (IN && FIRST) {
      const uint32_t g = (rev_bits_small(row, K) << (pp.log_n - K)) + col0 + col;
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t gr = g + (rev4(r) << (pp.log_n - 4));
        x[r] = gr >= pp.src_len ? (word)0 : (word)src[gr];
      }
    } else if constexpr (IN) {
      const uint64_t* p = src + (hi_base + (row << pp.S) + m0 + col);
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) x[r] = (word)p[(uint64_t)r << pp.S];
    } else {
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) x[r] = sm[sb + (r << B) + ((r << B) >> 4)];
    }
    const uint32_t jl = row & ((1u << W) - 1);
#pragma unroll
    for (int st = LO; st < HI; st++) {
      const int b = st - W;
      const uint32_t S = FIRST ? 0 : pp.S;
      const uint32_t half = 1u << (S + st);
      const uint64_t* tw = pp.tw + (half - 1);
      const uint32_t j0 = FIRST ? jl : (jl << S) + m0 + col;
#pragma unroll
      for (uint32_t q = 0; q < (1u << b); q++) {
        // Butterfly index j0 + q 2^(W + S): the inverse's factor is one for
        // index 0, else minus the mirrored entry.
        const bool one = FIRST && W == 0 && q == 0;
        uint64_t w = 0;
        if (!one) {
          const uint32_t j = j0 + (q << (W + S));
          if constexpr (INV) {
            if (q == 0) {
              w = __ldg(tw + (j == 0 ? 0u : half - j));
              w = j == 0 ? SF::kOneEntry : SF::neg_entry(w);
            } else {
              w = SF::neg_entry(__ldg(tw + (half - j)));
            }
          } else {
            w = __ldg(tw + j);
          }
        }
#pragma unroll
        for (uint32_t h = 0; h < (8u >> b); h++) {
          const uint32_t i = q + (h << (b + 1)), k = i + (1u << b);
          // The first stage's inputs are canonical.
          const word t = !one ? (word)SF::mul_entry(w, x[k]) : st == 0 ? x[k] : (word)SF::canonical(x[k]);
          SF::butterfly(x[i], t, x[i], x[k]);
        }
      }
    }
    if constexpr (OUT) {
      const uint32_t g = (FIRST ? rev_bits_small(col0 + col, pp.log_n - K) << K : hi_base + m0 + col) +
                         (FIRST ? row : row << pp.S);
      const uint32_t step = FIRST ? W : W + pp.S;
      const bool last = (FIRST ? 0 : pp.S) + K == pp.log_n;
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t gr = g + (r << step);
        uint64_t y = x[r];
        if (pp.scale) y = SF::mul(pp.scale_val, y);
        else if (last) y = SF::canonical(y);
        if (pp.coset_pw) {
          const uint64_t v = SF::mul(__ldg(pp.coset_pw + (gr & 1023)), __ldg(pp.coset_pw + 1024 + ((gr >> 10) & 1023)));
          y = SF::mul(SF::mul(v, __ldg(pp.coset_pw + 2048 + (gr >> 20))), y);
        }
        dst[gr] = y;
      }
    } else {
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) sm[sb + (r << B) + ((r << B) >> 4)] = x[r];
    }
  }

  __device__ __forceinline__ void run() const {
    window<0, 0, 4, true, false>();
    __syncthreads();
    if constexpr (K > 8) {
      window<4, 4, 8, false, false>();
      __syncthreads();
      window<K - 4, 8, K, false, true>();
    } else {
      window<K - 4, 4, K, false, true>();
    }
  }
};

}  // namespace zntt
