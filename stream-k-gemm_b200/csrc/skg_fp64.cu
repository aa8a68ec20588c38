// Host launcher of the native FP64 Stream-K kernel: operand descriptors ->
// TMA tensor maps, Stream-K schedule, cooperative persistent launch.
#include <algorithm>
#include <cmath>

#include "skg_fp64_kernel.cuh"
#include "skg_runtime.h"

namespace skg {

int make_operand_map(CUtensorMap* map, const Fp64Operand& op, int64_t K, int rows_per_tile) {
  if (op.ptr == nullptr) return fail(SKGEMM_ERR_INVALID_ARG, "null operand pointer");
  if ((reinterpret_cast<uintptr_t>(op.ptr) & 15) != 0)
    return fail(SKGEMM_ERR_INVALID_ARG, "operand base must be 16-byte aligned");
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B;
  if (op.kind == kOpPacked16) {
    uint64_t dims[3] = {16, (uint64_t)K, (uint64_t)((op.rows + 15) / 16)};
    uint64_t strides[2] = {16 * 8, (uint64_t)K * 16 * 8};
    uint32_t box[3] = {16, (uint32_t)kBK, (uint32_t)(rows_per_tile / 16)};
    return encode_tiled(map, 3, op.ptr, dims, strides, box, dt, sw);
  }
  if (op.kind == kOpPacked32) {
    uint64_t dims[3] = {32, (uint64_t)K, (uint64_t)((op.rows + 31) / 32)};
    uint64_t strides[2] = {32 * 8, (uint64_t)K * 32 * 8};
    uint32_t box[3] = {16, (uint32_t)kBK, (uint32_t)(rows_per_tile / 32)};
    return encode_tiled(map, 3, op.ptr, dims, strides, box, dt, sw);
  }
  if (op.kind == kOpBandK) {
    if (K % 16) return fail(SKGEMM_ERR_INVALID_ARG, "K-major operand needs K a multiple of 16");
    uint64_t dims[3] = {16, (uint64_t)op.rows, (uint64_t)(K / 16)};
    uint64_t strides[2] = {16 * 8, (uint64_t)op.rows * 16 * 8};
    uint32_t box[3] = {16, (uint32_t)rows_per_tile, 1};
    return encode_tiled(map, 3, op.ptr, dims, strides, box, dt, sw);
  }
  if (op.kind == kOpDense) {
    if (op.ld < op.rows || ((op.ld * 8) % 16) != 0)
      return fail(SKGEMM_ERR_INVALID_ARG, "dense operand leading dimension must be even and >= rows");
    uint64_t dims[2] = {(uint64_t)op.rows, (uint64_t)K};
    uint64_t strides[1] = {(uint64_t)op.ld * 8};
    uint32_t box[2] = {16, (uint32_t)kBK};
    return encode_tiled(map, 2, op.ptr, dims, strides, box, dt, sw);
  }
  return fail(SKGEMM_ERR_INVALID_ARG, "unknown operand kind");
}

namespace {

struct Schedule {
  int tiles_m, tiles_n, num_tiles, ipt;
  int64_t total;
  int grid;
};

// Persistent CTAs of a single-problem launch: every resident CTA, fewer where that
// cuts tiles into more parts than their sum pays for. Measured (us, grid at full
// occupancy / here):
//  * half of the resident CTAs where a tile is in many parts and a CTA's share
//    short: SYRK 10000 x 96 on 32 x 32 tiles 24 / 15, GEMM 32768 x 96 37 / 31,
//    rotation 1008 x 256 15 / 13; SYRK 10000 x 128 on 64 x 64 22 / 21, GEMM 23 /
//    19; equal from about 230 (32 x 32) and 60 iterations a CTA (64 x 64), where
//    the multiplications want all of them. 64 x 64 tiles in fewer than eight
//    parts keep the full grid: half of it costs dense operands 7-12% (700 x 500 x
//    900 31 / 33, 800^3 43 / 47, 1024^3 74 / 82, 500 x 500 x 2500 50 / 56) and
//    gains packed ones little (GEMM 1000 x 512 27 / 25, 2500 x 512 47 / 47).
//  * at most sqrt(14 iterations) parts a tile: an iteration costs about as much
//    as the sums of 14 parts in the fix-up. SYRK 10000 x 32 17 / 11 (94 parts
//    instead of 592), 32768 x 32 25 / 14.
int schedule_grid(DeviceState* dev, const Schedule& sc, int tile, int per_sm) {
  const int64_t full = (int64_t)dev->num_sms * per_sm;
  int64_t g = std::min(full, sc.total);
  if ((tile == 32 && sc.num_tiles < full && sc.total < 230 * full) ||
      (tile == 64 && 8 * (int64_t)sc.num_tiles <= full && sc.total < 60 * full))
    g = std::min(g, full / 2);
  const int64_t parts = (int64_t)std::ceil(std::sqrt(14.0 * sc.ipt));
  return (int)std::max<int64_t>(1, std::min(g, sc.num_tiles * parts));
}

Schedule make_schedule(DeviceState* dev, const Fp64Problem& prob, int tile, int per_sm) {
  Schedule sc;
  sc.tiles_m = (int)((prob.M + tile - 1) / tile);
  sc.tiles_n = (int)((prob.N + tile - 1) / tile);
  sc.num_tiles = prob.tile_order == kTilesUpper ? sc.tiles_n * (sc.tiles_n + 1) / 2
                                                : sc.tiles_m * sc.tiles_n;
  sc.ipt = (int)((prob.K + kBK - 1) / kBK);
  sc.total = (int64_t)sc.num_tiles * sc.ipt;
  sc.grid = schedule_grid(dev, sc, tile, per_sm);
  return sc;
}

// Issued MACs (padding included) of `prob` on tile x tile outputs.
double issued_macs(const Fp64Problem& prob, int tile) {
  const double tm = (double)((prob.M + tile - 1) / tile), tn = (double)((prob.N + tile - 1) / tile);
  const double tiles = prob.tile_order == kTilesUpper ? tn * (tn + 1) / 2 : tm * tn;
  return tiles * tile * tile * (double)((prob.K + kBK - 1) / kBK * kBK);
}

// Tile of a single-problem launch, by the MACs it issues (padding included) and
// how much work a CTA gets. Measured on B200 (us on 128 / 64 / 32 tiles):
//  * 32 x 32 where it saves enough padding: its operand traffic (half a byte a
//    MAC) holds it to 0.8 of the 64 x 64 rate. SYRK / GEMM 110592 x 96: 117 /
//    91 / 62, 118 / 116 / 88; SYRK 110592 x 224: 323 / 269 / 218; not GEMM
//    110592 x 128 (0 saved): 119 / 117 / 132. Dense operands take more, smaller
//    loads a tile (2000^3: 494 / 531 / 696) and need 0.7.
//  * 32 x 32 where the output has fewer 64 x 64 iterations than eight a CTA and
//    a short reduction, so that latency counts: GEMM 1008 x 128: 23 / 14 / 12,
//    rotation 1008 x 256: 21 / 16 / 15.
//  * 64 x 64 where it issues fewer MACs than 128 x 128 (triangles, edges) or
//    the output has >= 4 tiles of 128 x 128 per SM, so that two CTAs per SM
//    pay off: SYRK 110592 x 512 1018 / 925.
//  * 64 x 64 too where a CTA would get few 128 x 128 iterations (the last part
//    and the fix-up of a tile are a quarter as long): under 200 with packed
//    operands (GEMM 10000 x 512 (67): 162 / 158, 110592 x 128 (47): 119 / 117;
//    equal at 187-221), under 60 with a dense one (1000^3 (27): 81 / 76,
//    rotation 32768 x 256 (55): 155 / 137; 1500^3 (91): 218 / 228).
int single_tile(DeviceState* dev, const Fp64Problem& prob) {
  const double i32 = issued_macs(prob, 32), i64 = issued_macs(prob, 64),
               i128 = issued_macs(prob, 128);
  const bool dense_a = prob.a.kind == kOpDense, dense = dense_a || prob.b.kind == kOpDense;
  if (i32 < (dense_a ? 0.7 : 0.8) * i64) return 32;
  const double ipt = (double)((prob.K + kBK - 1) / kBK);
  const double it64 = i64 / (64.0 * 64.0 * kBK), it128 = i128 / (128.0 * 128.0 * kBK);
  if (!dense_a && ipt <= 128 && it64 < 16.0 * dev->num_sms) return 32;
  if (i64 < i128 || it128 / ipt >= 4.0 * dev->num_sms) return 64;
  return it128 < (dense ? 60.0 : 200.0) * dev->num_sms ? 64 : 128;
}

// CTAs per SM of the single-problem kernel of `tile` and A layout (its
// shared-memory attribute set once per device).
template <class TS>
int single_setup(int device, const void* kernel, bool akm, int* per_sm) {
  static int occ[2][64] = {};  // per tile shape: one array per instantiation
  int& o = occ[akm ? 1 : 0][device];
  if (!o) {
    SKG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  TS::kSmem));
    int n = 0;
    SKG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, TS::kThreads, TS::kSmem));
    if (n < 1) return fail(SKGEMM_ERR_CUDA, "FP64 kernel does not fit on an SM");
    o = std::min(n, TS::kMinBlocks);
  }
  *per_sm = o;
  return SKGEMM_OK;
}

}  // namespace

int fp64_preload(DeviceState* dev) {
  int per_sm = 0;
  return single_setup<Tile128>(dev->device, (const void*)fp64_streamk_kernel, false, &per_sm);
}

int fp64_grid_for(DeviceState* dev, const Fp64Problem& prob) {
  if (prob.M <= 0 || prob.N <= 0 || prob.K <= 0) return 0;
  return make_schedule(dev, prob, 128, 1).grid;
}

int launch_fp64(DeviceState* dev, const Fp64Problem& prob, cudaStream_t s,
                StreamWorkspace* ws_override, int tile) {
  if (prob.M < 0 || prob.N < 0 || prob.K < 0)
    return fail(SKGEMM_ERR_INVALID_ARG, "negative dimension");
  if (prob.tile_order == kTilesUpper && prob.M != prob.N)
    return fail(SKGEMM_ERR_INVALID_ARG, "SYRK tiles need a square output");
  if (prob.K > (int64_t)INT32_MAX - kBK || prob.M > ((int64_t)1 << 31) ||
      prob.N > ((int64_t)1 << 31))
    return fail(SKGEMM_ERR_INVALID_ARG, "dimension too large");
  if (prob.M == 0 || prob.N == 0) return SKGEMM_OK;
  if (prob.D == nullptr) return fail(SKGEMM_ERR_INVALID_ARG, "null output pointer");
  if (prob.K == 0) {
    // Empty reduction: D = gamma (GEMM), C = beta*C (SYRK), D = 0 (rotation).
    return fail(SKGEMM_ERR_UNSUPPORTED, "K == 0 is handled by the caller");
  }
  if (tile == 0) tile = single_tile(dev, prob);

  if (tile != 128 && tile != 64 && tile != 32)
    return fail(SKGEMM_ERR_INVALID_ARG, "tile must be 128, 64 or 32");
  const bool akm = prob.a.kind == kOpBandK;
  if (prob.b.kind == kOpBandK || (akm && prob.b.kind == kOpPacked32))
    return fail(SKGEMM_ERR_INVALID_ARG, "operand layouts not supported together");
  using Kernel = void (*)(CUtensorMap, CUtensorMap, Fp64Params);
  struct Variant {
    Kernel kernel;
    const char* name;
  };
  static const Variant variants[3][2] = {
      {{fp64_streamk_kernel, "fp64_streamk_kernel"},
       {fp64_streamk_kernel_ak, "fp64_streamk_kernel_ak"}},
      {{fp64_streamk_kernel64, "fp64_streamk_kernel64"},
       {fp64_streamk_kernel64_ak, "fp64_streamk_kernel64_ak"}},
      {{fp64_streamk_kernel32, "fp64_streamk_kernel32"},
       {fp64_streamk_kernel32_ak, "fp64_streamk_kernel32_ak"}}};
  const Variant& var = variants[tile == 128 ? 0 : (tile == 64 ? 1 : 2)][akm ? 1 : 0];
  const void* kernel = (const void*)var.kernel;
  int per_sm = 1, st = SKGEMM_OK;
  if ((st = tile == 128  ? single_setup<Tile128>(dev->device, kernel, akm, &per_sm)
            : tile == 64 ? single_setup<Tile64>(dev->device, kernel, akm, &per_sm)
                         : single_setup<Tile32>(dev->device, kernel, akm, &per_sm)))
    return st;
  Schedule sc = make_schedule(dev, prob, tile, per_sm);
  if ((int64_t)sc.num_tiles * sc.ipt > ((int64_t)1 << 40))
    return fail(SKGEMM_ERR_INVALID_ARG, "problem too large");

  // Slots in units of 128 x 128 partial tiles (a 64 x 64 slot is a quarter, a
  // 32 x 32 slot a sixteenth).
  auto big_slots = [&](int spread) {
    const int64_t n = fixup_slots(sc.grid, spread);
    const int64_t per = (128 / tile) * (128 / tile);
    return (size_t)((n + per - 1) / per);
  };
  int spread = 1;
  StreamWorkspace* ws = ws_override ? ws_override
                                    : stream_workspace(dev, s, big_slots(1), &st,
                                                       (size_t)fixup_slots(sc.grid, 1));
  if (!ws) return st;
  if (ws_override && (ws->partial_slots < big_slots(1) ||
                      ws->num_flags < (size_t)fixup_slots(sc.grid, 1)))
    spread = 0;
  if (ws->partial_slots < big_slots(spread) ||
      ws->num_flags < (size_t)fixup_slots(sc.grid, spread))
    return fail(SKGEMM_ERR_INVALID_ARG, "workspace has fewer partial slots than the grid");

  CUtensorMap mapA, mapB;
  if ((st = make_operand_map(&mapA, prob.a, prob.K, tile)) != SKGEMM_OK) return st;
  if ((st = make_operand_map(&mapB, prob.b, prob.K, tile)) != SKGEMM_OK) return st;

  Fp64Params p;
  p.M = prob.M;
  p.N = prob.N;
  p.K = prob.K;
  p.tiles_m = sc.tiles_m;
  p.tiles_n = sc.tiles_n;
  p.num_tiles = sc.num_tiles;
  p.iters_per_tile = sc.ipt;
  p.total_iters = sc.total;
  p.split = make_split(sc.total, sc.grid);
  p.a_kind = prob.a.kind;
  p.b_kind = prob.b.kind;
  p.tile_order = prob.tile_order;
  p.out_kind = prob.out_kind;
  p.D = prob.D;
  p.ldd = prob.ldd;
  p.alpha = prob.alpha;
  p.gamma = prob.gamma;
  p.beta_zero = prob.beta_zero ? 1 : 0;
  p.workspace = ws->partials;
  p.flags = ws->flags;
  p.epoch = ++ws->epoch;
  if (p.epoch == 0) p.epoch = ++ws->epoch;  // 0 is the value of a fresh flag
  p.spread = spread;
  p.err = ws->err;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sc.grid);
  cfg.blockDim = dim3(tile == 32 ? Tile32::kThreads : Tile64::kThreads);
  cfg.dynamicSmemBytes = tile == 128 ? Tile128::kSmem : tile == 64 ? Tile64::kSmem : Tile32::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  KernelTimer kt_(s, var.name);
  SKG_CUDA(cudaLaunchKernelEx(&cfg, var.kernel, mapA, mapB, p));
  return SKGEMM_OK;
}

}  // namespace skg

// ------------------------------------------------------------ grouped launch
namespace skg {

namespace {

template <class TS, bool SPREAD>
int grouped_occupancy(int* n) {
  SKG_CUDA(cudaFuncSetAttribute(fp64_grouped_kernel<TS, SPREAD>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, TS::kSmem));
  SKG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, fp64_grouped_kernel<TS, SPREAD>,
                                                         TS::kThreads, TS::kSmem));
  if (*n < 1) return fail(SKGEMM_ERR_UNSUPPORTED, "grouped kernel does not fit on an SM");
  return SKGEMM_OK;
}

template <class TS>
int grouped_setup(int device, int* blocks_per_sm) {
  static int occ[64] = {0};
  if (device < 0 || device >= 64) return fail(SKGEMM_ERR_INVALID_ARG, "device index");
  if (!occ[device]) {
    int a = 0, b = 0, st;
    if ((st = grouped_occupancy<TS, false>(&a)) || (st = grouped_occupancy<TS, true>(&b))) return st;
    occ[device] = std::min(a, b);
  }
  *blocks_per_sm = occ[device];
  return SKGEMM_OK;
}

template <class TS>
int grouped_launch(const Fp64Group& g, cudaStream_t s) {
  // Flags start at zero for every launch (a stream-ordered memset, captured
  // together with the kernel when the pair is recorded into a graph).
  SKG_CUDA(cudaMemsetAsync(g.flags, 0, (size_t)fixup_slots(g.grid, 1) * sizeof(uint32_t), s));
  if (!fp64_group_spread(g)) {
    // Only owners wait, for CTAs that never do: any number of CTAs may be resident.
    fp64_grouped_kernel<TS, false><<<g.grid, TS::kThreads, TS::kSmem, s>>>(g);
    SKG_CUDA(cudaGetLastError());
    return SKGEMM_OK;
  }
  // Cooperative: the CTAs that finish a tile wait for every other CTA of the tile
  // (shared_fixup), so all of the grid has to be resident, also beside another
  // stream's grouped launch.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.grid);
  cfg.blockDim = dim3(TS::kThreads);
  cfg.dynamicSmemBytes = TS::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SKG_CUDA(cudaLaunchKernelEx(&cfg, fp64_grouped_kernel<TS, true>, g));
  return SKGEMM_OK;
}

}  // namespace

// The shared fix-up needs a tile that can be in kSharedParts parts: its first and last
// part and kSharedParts - 2 whole CTA ranges of q iterations between them. Its code
// slows the loop of all tiles by 3% (the compiler's schedule; serving's launches of 25
// problems 28.2 -> 27.7 TFLOP/s without such tiles), 0.03 (64 x 64 tiles) or 0.06 us an
// iteration, and takes the owner 1.1 or 3 us a part off the longest tile: it pays from
// about q / 40 parts.
bool fp64_group_spread(const Fp64Group& g) {
  const int64_t q = std::max<int64_t>(1, g.total_iters / g.grid);
  return g.max_tile_iters >= (kSharedParts - 2) * q + 2 && 40 * (g.max_tile_iters / q) >= q;
}

int fp64_group_occupancy(DeviceState* dev, int tile, int* blocks_per_sm) {
  if (tile == 128) return grouped_setup<Tile128>(dev->device, blocks_per_sm);
  if (tile == 64) return grouped_setup<Tile64>(dev->device, blocks_per_sm);
  return fail(SKGEMM_ERR_INVALID_ARG, "tile must be 128 or 64");
}

int launch_fp64_group(int tile, const Fp64Group& group, cudaStream_t s) {
  if (group.grid <= 0 || group.total_iters <= 0) return SKGEMM_OK;
  Fp64Group g = group;
  g.split = make_split(g.total_iters, g.grid);
  if (tile == 128) return grouped_launch<Tile128>(g, s);
  if (tile == 64) return grouped_launch<Tile64>(g, s);
  return fail(SKGEMM_ERR_INVALID_ARG, "tile must be 128 or 64");
}

}  // namespace skg
