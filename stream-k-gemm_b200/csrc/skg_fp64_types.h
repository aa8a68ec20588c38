// Constants, enums and launch parameters of the native FP64 Stream-K kernel,
// shared by the kernel and its host-side users.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace skg {

constexpr int kBM = 128;
constexpr int kBN = 128;
constexpr int kBK = 16;
constexpr int kStages = 6;
constexpr int kChunkBytes = kBK * 16 * 8;           // [BK][16] doubles = 2 KB
constexpr int kTileABytes = (kBM / 16) * kChunkBytes;  // 16 KB
constexpr int kTileBBytes = (kBN / 16) * kChunkBytes;  // 16 KB
constexpr int kStageBytes = kTileABytes + kTileBBytes;
constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;

// Output-tile shape of one kernel instantiation: WM x WN consumer warps, each
// owning (BM/WM) x (BN/WN) outputs = MI m16 blocks x NJ n8 blocks, fed by MI A
// chunks and NQ = NJ/2 B chunks of 16 columns; one more warp issues the loads.
template <int BM_, int BN_, int WM_, int WN_>
struct TileShape {
  static constexpr int BM = BM_;
  static constexpr int BN = BN_;
  static constexpr int WM = WM_;
  static constexpr int WN = WN_;
  static constexpr int kWarps = WM * WN;        // consumer warps
  static constexpr int kCons = kWarps * 32;     // consumer threads
  static constexpr int kThreads = kCons + 32;   // + one producer warp
  static constexpr int MI = BM / (16 * WM);
  static constexpr int NJ = BN / (8 * WN);
  static constexpr int NQ = NJ / 2;
  static constexpr int kABytes = (BM / 16) * kChunkBytes;
  static constexpr int kBBytes = (BN / 16) * kChunkBytes;
  static constexpr int kStage = kABytes + kBBytes;
  static constexpr int kSmem = kStages * kStage + 1024 /*align*/ + 256 /*barriers*/;
  // CTAs per SM the launch bounds ask for: one 197 KB ring for 128 x 128,
  // two 97 KB rings for 64 x 64, four 49 KB rings for 32 x 32.
  static constexpr int kMinBlocks = BM >= 128 ? 1 : (BM >= 64 ? 2 : 4);
};
using Tile128 = TileShape<128, 128, 2, 4>;
using Tile64 = TileShape<64, 64, 2, 4>;
using Tile32 = TileShape<32, 32, 2, 2>;
static_assert(Tile128::kStage == kStageBytes && Tile128::kSmem == kSmemBytes, "tile constants");

enum OperandKind : int {
  kOpPacked16 = 0,  // [ceil(R/16)][K][16]; 3-D map {16, K, tiles}, one box per stage
  kOpPacked32 = 1,  // [ceil(R/32)][K][32]; 3-D map {32, K, tiles}, two half-width boxes
                    // per stage -> shared memory [half][tile][BK][16]
  kOpDense = 2,     // R contiguous, k stride ld; 2-D map {R, K}, one box per 16-chunk
  kOpBandK = 3,     // K-major [K/16][R][16] (band-packed Psi as the rotation's A:
                    // element (r, k) at (k/16)*R*16 + r*16 + k%16); 3-D map
                    // {16, R, K/16}, one box {16, BM, 1} per stage (BK = 16) ->
                    // shared memory [BM][16 k]; A operand of the single-problem
                    // kernels only, K % 16 == 0
};

enum OutKind : int { kOutRowMajor = 0, kOutSyrkUpper = 1, kOutBand16 = 2 };

enum TileOrder : int { kTilesAll = 0, kTilesUpper = 1 };

// The even split of `total` iterations over `grid` CTAs: CTA c covers
// [begin(c), begin(c + 1)), begin(c) = floor(c total / grid), held as quotient
// and remainder so that the kernels divide 32-bit numbers only.
struct IterSplit {
  int64_t q;     // total / grid
  int r;         // total % grid
  int grid;
  double inv;    // ~ grid / total, to guess the CTA of an iteration
#ifdef __CUDACC__
  __host__ __device__
#endif
  int64_t begin(int c) const {
    return (int64_t)c * q + (uint32_t)c * (uint32_t)r / (uint32_t)grid;
  }
  // The CTA whose range holds iteration i (0 <= i < total).
#ifdef __CUDACC__
  __host__ __device__
#endif
  int cta_of(int64_t i) const {
    int c = (int)((double)i * inv);
    c = c < grid - 1 ? c : grid - 1;
    while (begin(c) > i) --c;
    while (begin(c + 1) <= i) ++c;
    return c;
  }
};

inline IterSplit make_split(int64_t total, int grid) {
  IterSplit s;
  s.grid = grid > 0 ? grid : 1;
  s.q = total / s.grid;
  s.r = (int)(total % s.grid);
  s.inv = total > 0 ? (double)s.grid / (double)total : 0.0;
  return s;
}

struct Fp64Params {
  int64_t M, N, K;
  int tiles_m, tiles_n;
  int num_tiles;
  int iters_per_tile;  // ceil(K / BK)
  int64_t total_iters;
  int a_kind, b_kind;
  int tile_order;
  int out_kind;
  double* D;
  int64_t ldd;  // row stride (row-major) / column stride (SYRK); unused for band16
  double alpha;
  double gamma;  // GEMM: added scalar; SYRK: beta
  int beta_zero;
  double* workspace;  // partial tiles: BM*BN doubles per slot, slots(spread, grid)
  uint32_t* flags;    // one per slot
  uint32_t epoch;     // value a published flag carries for this launch
  IterSplit split;    // the launch's CTA ranges (single-problem launches)
  int spread;         // shared fix-up (2 slots per CTA); 0: the owner adds the partials
  uint32_t* err;      // device error word
};

// Partial-tile slots (and flags) of a launch of `grid` CTAs. A CTA publishes
// its first segment's partial in slot `cta`; with the shared fix-up the owner
// of a tile publishes its own part too, in slot grid + cta.
inline int64_t fixup_slots(int grid, int spread) { return (int64_t)grid * (spread ? 2 : 1); }

// Grouped launch: many independent problems in one persistent Stream-K
// launch. Their MAC-loop iterations are concatenated (problem p owns
// [iter_begin[p], iter_begin[p+1])) and split evenly over the CTAs; a CTA's
// range may cross tile and problem boundaries. Per-problem fields of
// Fp64Params used: M, N, K, tiles_m, tiles_n, num_tiles, iters_per_tile,
// a_kind, b_kind, tile_order, out_kind, D, ldd, alpha, gamma, beta_zero.
// Flags are cleared by the launcher before every launch (a memset in the same
// stream or graph) and published as 1, so the pair can be replayed from a
// CUDA graph.
struct Fp64Group {
  const Fp64Params* probs;
  const CUtensorMap* maps;     // 2 per problem (A, B), 64-byte aligned
  const int64_t* iter_begin;   // num_problems + 1 entries
  int num_problems;
  int64_t total_iters;
  int grid;
  int max_tile_iters;  // the longest tile's iterations
  IterSplit split;    // make_split(total_iters, grid)
  double* workspace;  // grid slots of BM*BN doubles, 2 * grid with the shared fix-up
  uint32_t* flags;    // 2 * grid flags, zero at launch
  uint32_t* err;
};

}  // namespace skg
