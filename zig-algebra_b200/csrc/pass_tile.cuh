// pass_tile.cuh -- one tile of one fused DIT pass, shared by the plain pass
// kernel and the batched persistent kernel.
//
// The network is zig-ntt's (libs/ntt/src/root.zig:148-212): stage s pairs
// DIT positions q and q + 2^(s-1) inside blocks of 2^s with twiddle
// tw[s-1][q mod 2^(s-1)].  A tile holds the 2^k positions that differ only in
// bits [S, S+k) of q, times 2^c neighbouring low-bit positions, in shared
// memory as two planes of 16-byte halves (half h of tile element e at
// sm[h * TILE + e]); stages run two at a time on four elements in registers.
#pragma once

#include "field.cuh"
#include "kernels.cuh"
#include "shoup.cuh"

namespace zntt {

__device__ __forceinline__ uint32_t rev_bits(uint32_t x, uint32_t bits) {
  return bits == 0 ? 0u : (__brev(x) >> (32 - bits));
}

template <uint32_t TILE>
__device__ __forceinline__ fe sm_load(const uint4* sm, uint32_t e) {
  uint4 lo = sm[e], hi = sm[TILE + e];
  fe r;
  r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = lo.z; r.v[3] = lo.w;
  r.v[4] = hi.x; r.v[5] = hi.y; r.v[6] = hi.z; r.v[7] = hi.w;
  return r;
}
template <uint32_t TILE>
__device__ __forceinline__ void sm_store(uint4* sm, uint32_t e, const fe& a) {
  sm[e] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
  sm[TILE + e] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

// t = w v for the table entry `idx` of a stage (mul), or v itself: below 2 p for
// lazy fields, below p for the others.
template <class F>
__device__ __forceinline__ fe times_factor(bool mul, const uint4* stw, uint32_t idx, const fe& v) {
  if (!mul) return fe_weak<F>(v);
  const uint4* f = stw + 4ull * idx;
  const fe t = fe_mul_fixed<F>(v, ld_fe32(f), ld_fe32(f + 2));
  if constexpr (F::kLazy) return t;
  else return fe_reduce<F>(t);
}

// Global access to tile data, one element (32 bytes) per thread.  `wide`: the
// vectors are 32-byte aligned, and an element moves in one instruction; else in
// two of 16 bytes.  COHERENT reads through L2 only, for data other SMs wrote
// earlier in the same launch (the batched kernel).
template <bool COHERENT>
__device__ __forceinline__ fe load_data(const uint4* p, bool wide) {
  fe r;
  if (wide) {
    if constexpr (COHERENT)
      asm volatile("ld.global.cg.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                     "=r"(r.v[7])
                   : "l"(p));
    else
      asm volatile("ld.global.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                     "=r"(r.v[7])
                   : "l"(p));
    return r;
  }
  uint4 lo, hi;
  if constexpr (COHERENT) {
    lo = __ldcg(p);
    hi = __ldcg(p + 1);
  } else {
    lo = p[0];
    hi = p[1];
  }
  r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = lo.z; r.v[3] = lo.w;
  r.v[4] = hi.x; r.v[5] = hi.y; r.v[6] = hi.z; r.v[7] = hi.w;
  return r;
}
__device__ __forceinline__ void store_data(uint4* p, const fe& a, bool wide) {
  if (wide)
    asm volatile("st.global.v8.u32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.v[0]), "r"(a.v[1]),
                 "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7])
                 : "memory");
  else
    fe_store(p, a);
}

// A pass's launch may overlap the pass before it (launch_pass_kernel): it reads
// and writes no vector before the one it follows has completed.  The radix-2
// passes let the next one's launch begin at once; the others, which fill the
// chip, only as their CTAs end (begun earlier, the next pass's waiting CTAs are
// dealt out unevenly: 2^18 BN254-Fr 0.052 -> 0.061 ms, B200).
__device__ __forceinline__ void pass_start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pass_wait_input() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// EXT enables the extension features: zero padding of the first pass's input
// from index src_len, a per-position scale table, and storing only the output
// positions below dst_len.  Plain transforms compile without them (fewer live
// registers in the hot loop).  FULL: the tile is the shape's whole tile
// (k + c == LOG_TILE, every pass of a transform larger than one tile), so no
// thread needs a bound check; without the checks the pass runs about 5% faster
// (2^24 BN254-Fr, B200).  SCALE compiles the output scaling (the inverse's
// 1/n, the extension's factor table); a pass launched without it must not ask
// for scaling (pp.scale == 0).  STRIDED: the twiddle table may be a strided one.
//
// The first stages read their elements straight from global memory and the last
// ones write theirs there (an element is one 32-byte sector, so a thread's own
// element moves as efficiently as a coalesced row); shared memory only carries
// the exchanges between stage pairs.
template <class F, int LOG_TILE, int THREADS, bool COHERENT, bool EXT, bool FULL = false, bool SCALE = true,
          bool STRIDED = false>
struct TilePass {
  static constexpr uint32_t TILE_MAX = 1u << LOG_TILE;
  const PassParams& pp;
  uint4* const sm;
  // The fields the stage loop reads, read once (for parameters held in
  // memory rather than in the kernel's parameter space, each later read would
  // be a load re-issued after every barrier).
  const uint32_t k, c, C, S;
  const bool first, inverse, unit0, wide;
  const uint4* const tw;
  // Indices fit 32 bits: transforms and tables hold at most 2^31 elements, so
  // an element's 16-byte-half offset is below 2^32.
  uint32_t hi_base = 0, m0 = 0, col0 = 0;

  __device__ __forceinline__ TilePass(const PassParams& p, uint32_t b, uint4* s)
      : pp(p), sm(s), k(p.k), c(p.c), C(1u << p.c), S(p.S), first(p.first), inverse(p.inverse),
        unit0(p.inverse | p.tw0_one), wide(p.wide), tw(p.tw) {
    if (first) {
      col0 = b << c;
    } else {
      const uint32_t mlog = S - c;
      hi_base = (b >> mlog) << (S + k);
      m0 = (b & ((1u << mlog) - 1)) << c;
    }
  }

  // Element (row t, column col) of the input (`rev`: t bit-reversed in k bits,
  // the natural-order row the first pass gathers) and of the output.
  __device__ __forceinline__ fe load(uint32_t t, uint32_t rev, uint32_t col) const {
    uint32_t g;
    if (first) {
      g = (rev << (pp.log_n - k)) + col0 + col;
      if (EXT && g >= pp.src_len) {
        fe z;
#pragma unroll
        for (int q = 0; q < 8; q++) z.v[q] = 0;
        return z;
      }
    } else {
      g = hi_base + (t << S) + m0 + col;
    }
    return load_data<COHERENT>(pp.src + ((uint64_t)g << 1), wide);
  }
  __device__ __forceinline__ uint32_t out_base(uint32_t col) const {
    return first ? rev_bits(col0 + col, pp.log_n - k) << k : hi_base + m0 + col;
  }
  __device__ __forceinline__ void store(uint32_t base, uint32_t t, const fe& x, bool last) const {
    const uint32_t g = base + (t << S);  // S == 0 in the first pass
    fe y = x;
    if (SCALE && pp.scale) {
      const uint4* f = pp.scale_tab;
      if (EXT && pp.scale != kScaleFixed) f += (pp.scale == kScaleElements ? 2ull : 4ull) * g;
      // Elements are the other transform's output: in a batch other CTAs of this launch
      // wrote them (so they go through L2, as the tile's data does), elsewhere an earlier
      // launch that this one may overlap (so not through the read-only path).  The factors
      // are constant.
      if (EXT && pp.scale == kScaleElements) y = fe_mul<F>(load_data<COHERENT>(f, false), x);
      else y = fe_reduce<F>(fe_mul_fixed<F>(x, ld_fe32(f), ld_fe32(f + 2)));
    } else if (last) {
      y = fe_canonical<F>(x);
    }
    if (!EXT || g < pp.dst_len) store_data(pp.dst + ((uint64_t)g << 1), y, wide);
  }

  // The table entries of the stage with `half` butterflies, and the place of its entry
  // idx among them (strided: below 2^(log_n - 1)).
  __device__ __forceinline__ const uint4* stage_entries(uint32_t half) const {
    if constexpr (STRIDED) {
      if (half >> pp.tw_flat) return tw + (4ull << pp.tw_flat);
    }
    return tw + 4ull * (half - 1);
  }
  __device__ __forceinline__ uint32_t entry(uint32_t half, uint32_t idx) const {
    if constexpr (STRIDED) {
      if (half >> pp.tw_flat) return idx << (pp.log_n - 32 + __clz(half));
    }
    return idx;
  }

  // Stages i and i+1 on four elements in registers (rows t0 + {0, h, 2h, 3h}).
  // With u, v -> u + t, u - t, t = tw[j] v, the inverse (inttWithTwiddles: factor
  // one for j = 0, else -tw[2^(s-1) - j]) is the same butterfly with the two
  // results exchanged, so it reads the mirrored entry and exchanges where they
  // go: the first stage's through the choice of the second stage's factors,
  // the second's through the rows.
  template <bool IN, bool OUT>
  __device__ __forceinline__ void pair(uint32_t i, uint32_t ga, bool last) const {
    const uint32_t h = IN ? 1u : 1u << (i - 1);
    const uint32_t half1 = 1u << (S + i - 1);  // stage S+i
    const uint32_t half2 = half1 << 1;         // stage S+i+1
    const uint4* stw1 = stage_entries(half1);
    const uint4* stw2 = stage_entries(half2);
    const uint32_t col = ga & (C - 1), g = ga >> c;
    const uint32_t j = g & (h - 1);
    const uint32_t t0 = IN ? g << 2 : ((g >> (i - 1)) << (i + 1)) | j;
    const uint32_t e0 = (t0 << c) | col, eh = h << c;
    uint32_t jg1, jg3;
    if (first) {
      jg1 = j;
      jg3 = j + h;
    } else {
      jg1 = (j << S) + m0 + col;
      jg3 = jg1 + (h << S);
    }
    const bool mul = !(jg1 == 0 && unit0);
    const bool swap = inverse && jg1 != 0;  // first-stage results exchanged
    const uint32_t i1 = entry(half1, inverse ? half1 - jg1 : jg1);
    // Second stage: the sums' pair and the differences' pair.
    const uint32_t jp = swap ? jg3 : jg1, jm = swap ? jg1 : jg3;
    const uint32_t ip = entry(half2, inverse ? half2 - jp : jp), im = entry(half2, inverse ? half2 - jm : jm);
    fe x0, x1, x2, x3;
    if constexpr (IN) {
      const uint32_t rv = first ? rev_bits(t0, k) : 0;  // t0 is a multiple of 4
      x1 = load(t0 + 1, rv + (1u << (k - 1)), col);
      x0 = load(t0, rv, col);
      x3 = load(t0 + 3, rv + (3u << (k - 2)), col);
      x2 = load(t0 + 2, rv + (1u << (k - 2)), col);
    }
    fe p0, d0, p2, d2, y, z;
    {
      if constexpr (!IN) x1 = sm_load<TILE_MAX>(sm, e0 + eh);
      const fe t = times_factor<F>(mul, stw1, i1, x1);
      if constexpr (!IN) x0 = sm_load<TILE_MAX>(sm, e0);
      fe_butterfly<F>(fe_weak<F>(x0), t, p0, d0);
    }
    {
      if constexpr (!IN) x3 = sm_load<TILE_MAX>(sm, e0 + 3 * eh);
      const fe t = times_factor<F>(mul, stw1, i1, x3);
      if constexpr (!IN) x2 = sm_load<TILE_MAX>(sm, e0 + 2 * eh);
      fe_butterfly<F>(fe_weak<F>(x2), t, p2, d2);
    }
    const uint32_t base = OUT ? out_base(col) : 0;
    {
      const fe t = times_factor<F>(mul, stw2, ip, p2);
      if constexpr (!F::kLazy) p0 = fe_weak<F>(p0);
      fe_butterfly<F>(p0, t, y, z);
      const uint32_t a = swap ? 3 : 0, b = swap ? 1 : 2;  // rows of the sum and of the difference
      if constexpr (OUT) {
        store(base, t0 + a * h, y, last);
        store(base, t0 + b * h, z, last);
      } else {
        sm_store<TILE_MAX>(sm, e0 + a * eh, y);
        sm_store<TILE_MAX>(sm, e0 + b * eh, z);
      }
    }
    {
      const fe t = times_factor<F>(true, stw2, im, d2);
      if constexpr (!F::kLazy) d0 = fe_weak<F>(d0);
      fe_butterfly<F>(d0, t, y, z);
      const uint32_t a0 = swap ? 0 : 1;
      const uint32_t a = inverse ? a0 + 2 : a0, b = inverse ? a0 : a0 + 2;
      if constexpr (OUT) {
        store(base, t0 + a * h, y, last);
        store(base, t0 + b * h, z, last);
      } else {
        sm_store<TILE_MAX>(sm, e0 + a * eh, y);
        sm_store<TILE_MAX>(sm, e0 + b * eh, z);
      }
    }
  }

  // Stage k alone, at the end of a pass of odd k: rows t0 and t0 + 2^(k-1).
  template <bool IN>
  __device__ __forceinline__ void single(uint32_t ga, bool last) const {
    const uint32_t h = 1u << (k - 1);
    const uint32_t half = 1u << (S + k - 1);  // stage S+k
    const uint4* stw = stage_entries(half);
    const uint32_t col = ga & (C - 1), j = ga >> c;
    const uint32_t jg = first ? j : (j << S) + m0 + col;
    const bool swap = inverse && jg != 0;
    const uint32_t e0 = (j << c) | col;
    fe u, v, y, z;
    if constexpr (IN) {
      v = load(1, 1, col);
      u = load(0, 0, col);
    } else {
      v = sm_load<TILE_MAX>(sm, e0 + (h << c));
    }
    const fe t = times_factor<F>(!(jg == 0 && unit0), stw, entry(half, inverse ? half - jg : jg), v);
    if constexpr (!IN) u = sm_load<TILE_MAX>(sm, e0);
    fe_butterfly<F>(fe_weak<F>(u), t, y, z);
    const uint32_t base = out_base(col);
    store(base, swap ? j + h : j, y, last);
    store(base, swap ? j : j + h, z, last);
  }

  __device__ __forceinline__ void run() const {
    const uint32_t tile = FULL ? TILE_MAX : 1u << (k + c);
    const uint32_t tid = threadIdx.x;
    const bool last = S + k == pp.log_n;  // the transform's last stages: canonical results
    if (k <= 2) {
      // One group, straight from input to output (k == 0: a length-1 vector).
      if (k == 2) {
        for (uint32_t ga = tid; ga < tile / 4; ga += THREADS) pair<true, true>(1, ga, last);
      } else if (k == 1) {
        for (uint32_t ga = tid; ga < tile / 2; ga += THREADS) single<true>(ga, last);
      } else if (tid == 0) {
        store(0, 0, load(0, 0, 0), false);
      }
      return;
    }
    // Warp w's groups of a pair of span 4 h C <= 128 elements are the same
    // 128-element slices of the tile: such pairs exchange data only inside the
    // warp and synchronise with __syncwarp, the others with a CTA barrier
    // (2^24: two of the three exchanges of every pass are warp-local).
#pragma unroll
    for (uint32_t q = 0; q < TILE_MAX / 4 / THREADS; q++) {
      const uint32_t ga = tid + q * THREADS;
      if (FULL || ga < tile / 4) pair<true, false>(1, ga, false);
    }
    uint32_t i = 3;
    for (;; i += 2) {
      // Stages i, i+1 next: their span is 2^(i+1) C.
      if (((2u << i) << c) <= 128u) __syncwarp();
      else __syncthreads();
      if (i + 1 >= k) break;
#pragma unroll
      for (uint32_t q = 0; q < TILE_MAX / 4 / THREADS; q++) {
        const uint32_t ga = tid + q * THREADS;
        if (FULL || ga < tile / 4) pair<false, false>(i, ga, false);
      }
    }
    if (i + 1 == k) {
#pragma unroll
      for (uint32_t q = 0; q < TILE_MAX / 4 / THREADS; q++) {
        const uint32_t ga = tid + q * THREADS;
        if (FULL || ga < tile / 4) pair<false, true>(i, ga, last);
      }
    } else {
      // An odd stage count ends with one radix-2 stage.  Last rather than
      // first: in a transform's first pass the first stage pair then holds the
      // factors that are one (stage 1, and stage 2's j = 0), so the pass skips
      // their products in whole warps (2^20 first pass 8% faster, B200).
#pragma unroll
      for (uint32_t q = 0; q < TILE_MAX / 2 / THREADS; q++) {
        const uint32_t ga = tid + q * THREADS;
        if (FULL || ga < tile / 2) single<false>(ga, last);
      }
    }
  }
};

// A pass on one butterfly per thread (tile / 2 threads), for transforms that do
// not fill the chip: what counts there is the length of each thread's chain of
// products, one per stage instead of the radix-4 groups' four per two stages.
// Bound by that chain (about 1,400 cycles a stage for a warp alone on its
// scheduler) and the launches: 2^12 BN254-Fr forward and inverse 0.0226 -> 0.0143
// ms each, 2^14 0.0256 -> 0.0159, 2^16 0.0280 -> 0.0215 (B200).
// Each stage's factor is loaded a stage ahead, and the exchange alternates
// between two buffers of a tile, so that one barrier a stage suffices.
template <class F, int LOG_TILE>
__device__ __forceinline__ void ntt_tile_radix2(const PassParams& pp, uint32_t blk, uint4* sm) {
  constexpr uint32_t TILE = 1u << LOG_TILE, THREADS = TILE / 2;
  const TilePass<F, LOG_TILE, THREADS, false, true> tp(pp, blk, sm);
  const uint32_t k = tp.k, c = tp.c, S = tp.S;
  const bool inverse = tp.inverse;
  const uint32_t ga = threadIdx.x;
  const bool on = ga < (1u << (k + c)) / 2;
  const bool last = S + k == pp.log_n;
  const uint32_t col = ga & (tp.C - 1), g = ga >> c;
  // The factor of stage i: its table entry, and whether it multiplies at all.
  const auto entry = [&](uint32_t i, bool& mul, bool& swap) {
    const uint32_t half = 1u << (S + i - 1), j = g & ((1u << (i - 1)) - 1);
    const uint32_t jg = tp.first ? j : (j << S) + tp.m0 + col;
    mul = on && !(jg == 0 && tp.unit0);
    swap = inverse && jg != 0;
    return tp.tw + 4ull * (half - 1 + (inverse ? half - jg : jg));
  };
  struct Factor {
    fe w, q;
    bool mul, swap;
  };
  const auto fetch = [&](Factor& f, uint32_t i) {
    const uint4* p = entry(i, f.mul, f.swap);
    if (f.mul) {
      f.w = ld_fe32(p);
      f.q = ld_fe32(p + 2);
    }
  };
  Factor even, odd;  // of the stages with even and with odd number
  fetch(odd, 1);
  pass_wait_input();
  fe u, v;
  if (on) {
    const uint32_t rv = tp.first ? rev_bits(2 * g, k) : 0;
    v = tp.load(2 * g + 1, rv + (1u << (k - 1)), col);
    u = tp.load(2 * g, rv, col);
  }
  // Stage i with its factor f, fetching the next one into fn; true after the last.
  const auto stage = [&](uint32_t i, const Factor& f, Factor& fn, uint4* buf) {
    const uint32_t h = 1u << (i - 1);
    const uint32_t t0 = ((g >> (i - 1)) << i) | (g & (h - 1));
    if (i < k) fetch(fn, i + 1);
    fe t, y, z;
    if (f.mul) {
      t = fe_mul_fixed<F>(v, f.w, f.q);
      if constexpr (!F::kLazy) t = fe_reduce<F>(t);
    } else {
      t = fe_weak<F>(v);
    }
    fe_butterfly<F>(fe_weak<F>(u), t, y, z);
    const uint32_t a = f.swap ? t0 + h : t0, b = f.swap ? t0 : t0 + h;  // rows of the sum and of the difference
    if (i == k) {
      if (on) {
        const uint32_t base = tp.out_base(col);
        tp.store(base, a, y, last);
        tp.store(base, b, z, last);
      }
      return true;
    }
    if (on) {
      sm_store<TILE>(buf, (a << c) | col, y);
      sm_store<TILE>(buf, (b << c) | col, z);
    }
    if (THREADS <= 32) __syncwarp();
    else __syncthreads();
    if (on) {
      const uint32_t t1 = ((g >> i) << (i + 1)) | (g & (2 * h - 1));
      u = sm_load<TILE>(buf, (t1 << c) | col);
      v = sm_load<TILE>(buf, ((t1 + 2 * h) << c) | col);
    }
    return false;
  };
  for (uint32_t i = 1; i <= k; i += 2) {
    if (stage(i, odd, even, sm)) break;
    if (stage(i + 1, even, odd, sm + 2 * TILE)) break;
  }
}

template <class F, int LOG_TILE, int THREADS, bool COHERENT, bool EXT, bool FULL = false, bool SCALE = true,
          bool STRIDED = false>
__device__ __forceinline__ void ntt_tile(const PassParams& pp, uint32_t blk, uint4* sm) {
  TilePass<F, LOG_TILE, THREADS, COHERENT, EXT, FULL, SCALE, STRIDED>(pp, blk, sm).run();
}

}  // namespace zntt
