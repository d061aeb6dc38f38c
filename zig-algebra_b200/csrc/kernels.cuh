// kernels.cuh -- launch interface between the host runtime and the sm_100a kernels.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace zntt {

// Field identifiers shared with the C ABI (include/zntt.h).
// 0 and 1: 256-bit Montgomery fields (32-byte elements, this file's kernels);
// 2 and 3: SmallField's Goldilocks and BabyBear (8-byte elements, small.cu).
enum FieldId : int { kBn254Fr = 0, kBls12381Fr = 1, kGoldilocksField = 2, kBabyBearField = 3 };

// The output scaling of a pass: none, one fixed factor (the inverse's 1/n), a
// table of fixed factors (a coset extension's n^-1 g^q), or a table of elements
// (the other transform of a polynomial product).
enum ScaleKind : uint32_t { kScaleNone = 0, kScaleFixed = 1, kScaleFixedTab = 2, kScaleElements = 3 };

// One fused radix-2^k pass of the decimation-in-time network.
//
// The network is zig-ntt's (libs/ntt/src/root.zig:148-212): bit-reverse the
// input, then stages s = 1..log_n; stage s pairs positions q and q + 2^(s-1)
// inside blocks of 2^s and uses twiddle tw[s-1][q mod 2^(s-1)].  A pass runs
// stages S+1..S+k on tiles of 2^k positions that differ only in bits
// [S, S+k) of q, with 2^c neighbouring low-bit positions per tile so global
// rows are 2^c * 32 contiguous bytes.  The first pass (S == 0) gathers its
// tile from the natural-order input, which folds the bit reversal into the
// load: permuted block rev(col) holds input column col of the 2^k x 2^(L-k)
// row-major view, row r landing at tile row rev_k(r).
struct PassParams {
  const uint4* src;   // 2 uint4 per element
  uint4* dst;
  const uint4* tw;    // zig-ntt twiddle table as fixed factors (shoup.cuh), 4 uint4 each, stage s at entry 2^s - 1
  uint32_t log_n;     // L
  uint32_t S;         // stages already applied
  uint32_t k;         // stages in this pass
  uint32_t c;         // log2 of contiguous positions per tile row
  uint32_t first;     // gather the input through the bit reversal
  uint32_t inverse;   // inttWithTwiddles mapping: w = 1 (j = 0) or -tw[s-1][2^(s-1) - j]
  uint32_t wide;      // src and dst are 32-byte aligned
  uint32_t tw0_one;   // every stage's entry 0 is one (j = 0 needs no multiply)
  uint32_t scale;     // what the outputs are multiplied by after the last stage (ScaleKind)
  const uint4* scale_tab;  // the factor, or the table whose entry q multiplies output position q
  uint64_t src_len;   // first pass: natural input index >= src_len reads as zero (zero padding)
  uint64_t dst_len;   // output positions >= dst_len are not stored
  uint32_t tw_flat;   // stages from here on share the last one's table entries (log_n but in strided tables)
};

// Pass kernel shapes.  Each shape is a compiled kernel: a tile of 2^log_tile
// elements (32 bytes each in shared memory), `threads` per CTA, `min_blocks`
// CTAs per SM for the register budget.  The autotuner picks a shape and a
// stage count per pass for each (field, log n).
struct PassShape {
  int log_tile, threads, min_blocks;
};
// 2^11 and 2^10 tiles in CTAs of 256 threads (3 per SM), and the same 24 warps
// per SM in smaller CTAs: 2^9 tiles in 128 threads (6 per SM) and 2^8 tiles in
// 64 threads (12 per SM), where each barrier waits on fewer warps.  The last
// shape trades a 72-register budget (a few spilled words) for 28 warps per SM.
// 2^24 BN254-Fr in ms, B200: 2^10 tiles 2.88, 2^9 at 7 CTAs 2.71 (and at 8 CTAs,
// 64 registers, 2.80: not compiled), 2^8 tiles 3.09.
constexpr int kNumShapes = 5;
// Behind the tunable shapes, two of one butterfly per thread (ntt_tile_radix2),
// kRadix2Shape with 2^7-element tiles and the next with 2^8.
constexpr PassShape kShapes[kNumShapes + 2] = {{11, 256, 3}, {10, 256, 3}, {9, 128, 6}, {8, 64, 12},
                                               {9, 128, 7},  {7, 64, 8},   {8, 128, 4}};
constexpr int kRadix2Shape = kNumShapes;
// Plain transforms up to this size run on the radix-2 shapes, unless the tuning table
// holds a faster plan.  Both ways, two transforms (forward and inverse) of BN254-Fr in
// us, B200: 2^10 24.6 against 38.9 with the tuned radix-4 passes, 2^14 30.9 / 47.2,
// 2^16 42.7 / 51.3 (BLS12-381-Fr 22.6 / 35.9, 28.7 / 45.1, 41.0 / 51.2), and from 2^17
// on the radix-4 passes are as fast or faster (BN254-Fr 63.5 / 63.6, 2^18 106 / 102).
constexpr uint32_t kRadix2MaxLog = 16;
// The shape of persistent launches (batches and the server's slices): the
// 7-CTA 2^9 tile runs the mixed 520-transform batch in 2.22 ms, the 2^11 tile in
// 2.26, the 6-CTA 2^9 tile 2.27, the 2^10 tile 2.37, the 2^8 tile 2.42; 64 coset
// extensions 2^18 -> 2^20 (BLS12-381-Fr) 11.9 / 11.9 / 12.1 / 12.6 / 13.0 (B200).
constexpr int kBatchShape = 4;
// Root-derived tables from this size on are strided: the last stage's 2^(log_n - 1)
// entries also serve the five stages before it, whose entries are every second, every
// fourth, ... of them, and only the stages below have entries of their own.  That is 33
// bytes an element instead of 64, about what 32-byte entries took: a BLS12-381-Fr
// extension 2^29 -> 2^30 takes 130 GiB with its tables, 192 with flat ones.  The passes
// on strided tables have their own kernels on one shape (2^29 forward 109.8 ms, 109.9 on
// a flat table; B200): below, the tables stay flat and the hot kernels without the stride,
// which cost them 0.3 to 0.9%.
constexpr uint32_t kStridedLog = 29;
constexpr uint32_t kStridedStages = 6;
constexpr int kStridedShape = 2;
inline uint32_t table_flat_stages(uint32_t log_n) { return log_n < kStridedLog ? log_n : log_n - kStridedStages; }
// Entries of a table, 1/n among them (entry 2^flat - 1).
inline uint64_t table_entries(uint32_t log_n, uint32_t flat) {
  return flat == log_n ? 1ull << log_n : (1ull << flat) + (1ull << (log_n - 1));
}
// Tables of one factor per element (an extension's, a fold's) of 2^29 entries and more
// hold 32-byte elements, whose product is a Montgomery product, for the same reason (of
// the two fields only BLS12-381-Fr has folds that large).
inline bool narrow_factors(uint64_t count) { return count >= 1ull << kStridedLog; }
constexpr int kLogTile = 11;  // the largest tile of any shape
constexpr int kDefaultShape = 0;

inline int shape_smem_bytes(int shape) { return (1 << kShapes[shape].log_tile) * 32; }

// A pass that pads its input with zeros, scales by a table or stores a prefix
// of its output runs the extension variant of the kernels.
inline bool pass_needs_ext(const PassParams& pp) {
  const uint64_t n = 1ull << pp.log_n;
  return (pp.first && pp.src_len < n) || pp.scale >= kScaleFixedTab || pp.dst_len < n;
}

// PassParams::wide of a pass between the two vectors.
inline uint32_t pass_wide(const uint4* src, const uint4* dst) {
  return ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 31) == 0;
}

cudaError_t launch_ntt_pass(int field, int shape, const PassParams& pp, uint64_t num_tiles, cudaStream_t st);
cudaError_t configure_kernels();
cudaError_t configure_batch_kernels();

// ---- batched persistent launch ----------------------------------------------
// One pass of one job inside a batch, and one unit of work (a tile of a pass).
struct BatchPass {
  PassParams pp;
  uint32_t tiles;  // tiles in this pass
  uint32_t dep;    // pass that must finish first (kNoDep: none)
};
constexpr uint32_t kNoDep = 0xffffffffu;
struct BatchItem {
  uint32_t pass;
  uint32_t tile;
};
// ctl[0]: next item, ctl[1]: error flag, ctl[2 + p]: finished tiles of pass p.
// Every wait for a finished pass spins at most `spin_limit` rounds of ~1 us,
// then raises the error flag; every CTA stops at the next item once it is set.
// `full`: every pass has whole tiles (batch_all_full), so no bound checks.
// strided: some pass's twiddle table is strided (kStridedShape only).
cudaError_t launch_batch(int field, int shape, bool ext, bool full, bool strided, const BatchPass* passes, const BatchItem* items,
                         uint32_t n_items, uint32_t* ctl, uint32_t spin_limit, int grid, cudaStream_t st);
// True when every pass's tile is the shape's whole tile (k + c == log_tile).
inline bool batch_all_full(int shape, const BatchPass* passes, size_t n) {
  for (size_t i = 0; i < n; i++)
    if (passes[i].pp.k + passes[i].pp.c != (uint32_t)kShapes[shape].log_tile) return false;
  return true;
}
int batch_grid(int field, int shape, bool ext);

// zig-ntt twiddle table for one (field, log_n, root), as fixed factors: entry
// 2^s - 1 + j of stage s < flat is root^(j * 2^(log_n-1-s)), entry 2^flat - 1 is 1/n,
// given in Montgomery form, and in a strided table (flat < log_n) entry 2^flat + j is
// root^j, j < 2^(log_n - 1).  The powers are assembled from three
// small host-made tables: pw[0][i] = root^i, pw[1][i] = root^(1024 i),
// pw[2][i] = root^(2^20 i), i < 1024 (each 1024 x 32 bytes, contiguous).
cudaError_t launch_twiddle_table(int field, const uint4* d_pw, const uint64_t* n_inv, uint4* d_table, uint32_t log_n,
                                 uint32_t flat, cudaStream_t st);
// A flat table from its 2^log_n - 1 entries in Montgomery form.
cudaError_t launch_twiddle_pairs(int field, const uint4* d_entries, const uint64_t* n_inv, uint4* d_table,
                                 uint32_t log_n, cudaStream_t st);
// `count` fixed factors from d_pairs on, every 2^step-th one, back in Montgomery form.
cudaError_t launch_pair_entries(int field, const uint4* d_pairs, uint32_t step, uint4* d_entries, uint64_t count,
                                cudaStream_t st);

// out[i] = c * base^i for i < count (count <= 2^30), from the three power
// tables of `base` laid out as for launch_twiddle_table; `pairs`: as fixed factors.
cudaError_t launch_powers(int field, const uint4* d_pw, const uint64_t* c, uint4* out, uint64_t count, bool pairs,
                          cudaStream_t st);

// dst[rev(i)] = src[i] for 2^log_n elements (out of place).
cudaError_t launch_bit_reverse(const uint4* src, uint4* dst, uint32_t log_n, cudaStream_t st);

// Elementwise device arithmetic for tests: op 0 mul, 1 add, 2 sub, 3 neg.
cudaError_t launch_elementwise(int field, int op, const uint4* a, const uint4* b, uint4* out,
                               uint64_t count, cudaStream_t st);

// Multiply-throughput probe: `iters` rounds of 8-long mad.lo/madc.hi carry
// chains per thread; returns through `sink` so nothing is optimised away.
cudaError_t launch_imad_probe(uint32_t* sink, uint32_t iters, int blocks, int threads, cudaStream_t st);
// Independent 32x32->64 multiply-adds per thread (8 per iteration).
cudaError_t launch_imad_wide_probe(unsigned long long* sink, uint32_t iters, int blocks, int threads,
                                   cudaStream_t st);
// Independent modular products per thread, to time the field multiply alone.
cudaError_t launch_modmul_probe(int field, uint4* sink, uint32_t iters, int blocks, int threads,
                                cudaStream_t st);

}  // namespace zntt
