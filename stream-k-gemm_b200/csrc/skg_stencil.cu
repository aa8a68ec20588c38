// The H Psi producer of a CheFSI step on device: the 6th-order finite-
// difference stencil on extended (halo-padded) band-packed Psi, output in the
// 32-band-packed layout that the GEMM reads as B (Hs = Psi^T H Psi) or in the
// 16-band-packed layout (calc_laplacian_extended_packed_16to32 / _16to16,
// include/stencil_extended_packed.hpp:47-181, :276-), and the single-rank
// periodic halo that extends band-packed Psi (copy_interior_to_extended_packed,
// include/halo_packed.hpp:93-124, and the no-MPI wrap of :350-393).
//
// Per grid point g = i + j ni + k ni nj (extended index g_ex, offset FDn on
// each axis) and band b:
//   res = psi(g_ex) (A[g] + c0)
//   for r = 1 .. 6: res = fma(psi(g_ex + r) + psi(g_ex - r), cx[r], res), then
//                   the same along y (stride ni_ex) and z (ni_ex nj_ex)
// in the reference SVE kernels' order (x, y, z for each r; FMLA is fused),
// so the results equal those kernels bit for bit.
#include <algorithm>

#include "skg_common.cuh"
#include "skg_runtime.h"

namespace skg {

namespace {

constexpr int kFDn = 6;
constexpr int kZq = 2 * kFDn + 1;  // planes k - 6 .. k + 6

struct StencilCoef {
  double cx[kFDn + 1], cy[kFDn + 1], cz[kFDn + 1];
  double c0;
};

// Tile = one 8-band slab (bands 8 q .. 8 q + 7: 64 bytes per point) of 16 x 8
// columns. One CTA per SM takes whole tiles, nk planes each, and then an even
// share of the planes that are left (StWork). A producer warp streams one stage
// per plane k into a ring of kStRing shared-memory stages, on through the tiles:
//   the tile's plane k with its x / y halo, 28 x 20 points x 8 bands, by TMA;
//   the tile's 16 x 8 points of plane k + 6 (the z queue's new entry), by TMA;
//   A[g] of the tile's points of plane k, by 8-byte asynchronous copies (a row
//   of A starts at any multiple of 8 bytes).
// A piece begins with kStFills stages that hold planes k0 - 6 .. k0 + 5 for the
// queues, so that they too are loaded while the piece before is computed.
// Consumer thread = two columns (i, j) and (i, j + 1) and a band pair: a
// quarter-warp reads 2 consecutive points (128 contiguous bytes); the 14
// staged values j - 6 .. j + 7 serve the y neighbours of both columns; the
// 12 z neighbours come from the columns' 13-slot register queues (slot of
// plane k + d at step u of a 13-step period: (u + d + 6) mod 13). No global
// load waits inside the k loop. Same arithmetic in the same order as the
// reference kernels: the output equals theirs bit for bit. Every wait is
// bounded; on expiry the CTA records the error and skips the remaining waits.
//
// Bound by the shared-memory pipe, 89% busy: 20 16-byte loads per column and
// band pair, and the stage itself is written through it. TMA moves one box row per
// 1.3 cycles whatever its length, so the 32-byte rows of a 4-band slab on 16 x 16
// columns took 297 us without any arithmetic against 225 us for these 64-byte rows
// (400 us and 351 us in all).
// Whole launches, one CTA per tile with its queues loaded at its start, 4-band
// slabs -> this: 48^3 x 512 400 -> 351 us, 33 x 35 x 41 x 512 362 -> 243 us,
// 56^3 x 318 475 -> 394 us, 48^3 x 72 86 -> 60 us, 24^3 x 24 31 -> 15 us.
// Five stages took 353 us.
constexpr int kStI = 16;                 // columns per CTA along x
constexpr int kStJ = 8;                  // columns per CTA along y
constexpr int kSlab = 8;                 // bands per CTA
constexpr int kBP = kSlab / 2;           // band pairs
constexpr int kStHI = kStI + 2 * kFDn;   // staged points along x
constexpr int kStHJ = kStJ + 2 * kFDn;   // staged points along y
constexpr int kStPlane = kStHI * kStHJ * kSlab;  // doubles: halo plane
constexpr int kStCenter = kStI * kStJ * kSlab;   // doubles: plane k + 6
constexpr int kStA = kStI * kStJ;                // doubles: A of plane k
constexpr int kStStage = kStPlane + kStCenter + kStA;  // doubles per stage
constexpr int kStRing = 4;
constexpr int kStConsumerWarps = kStI * kStJ * kSlab / 128;  // 4 outputs a thread
constexpr int kStThreads = (kStConsumerWarps + 1) * 32;
constexpr int kStFill = 4;               // planes of a queue-filling stage
constexpr int kStFills = 2 * kFDn / kStFill;
constexpr int kStTxBytes = (kStPlane + kStCenter) * 8;
constexpr int kStMinSteps = 8;           // planes a CTA should have at least: each piece
                                         // costs 12 planes' queue entries on top
constexpr int kStSmem = kStRing * kStStage * 8 + 2 * kStRing * 8 + 16 + 128;
static_assert((kStPlane * 8) % 128 == 0 && (kStCenter * 8) % 128 == 0, "stage alignment");
static_assert((kStStage * 8) % 128 == 0 && (2 * kFDn) % kStFill == 0, "stage layout");
static_assert(kStFill * kStCenter <= kStStage, "queue-filling stage");
static_assert(kStSmem <= 232448, "stencil stages exceed 227 KB of shared memory");

// Arrives at a barrier once all this thread's asynchronous copies have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The work of one CTA: tiles c, c + G, .. of the full waves, then its share of
// the remaining tiles' planes, cut evenly over all G CTAs (a share is shorter
// than a tile's nk planes: at most two pieces).
struct StWork {
  int waves, first, ka, len;  // whole tiles; the share's first tile, first plane and planes
};
// Piece n: its tile and planes [k0, k1); false when there is none.
__device__ __forceinline__ bool st_piece(const volatile StWork* w, int n, int nk, int* tile, int* k0,
                                         int* k1) {
  const int m = n - w->waves;
  if (m < 0) {
    *tile = blockIdx.x + n * gridDim.x;
    *k0 = 0;
    *k1 = nk;
    return true;
  }
  const int end = w->ka + w->len - m * nk;  // the share's end, from this tile's plane 0
  *tile = w->first + m;
  *k0 = m == 0 ? w->ka : 0;
  *k1 = min(nk, end);
  return w->len > 0 && end > 0;
}

template <int OT>
__global__ void __launch_bounds__(kStThreads, 1) stencil_staged_kernel(
    const __grid_constant__ CUtensorMap mapP, const __grid_constant__ CUtensorMap mapC,
    const __grid_constant__ CUtensorMap mapF, int ni, int nj, int nk, int nb, int tiles,
    const double* __restrict__ A, const __grid_constant__ StencilCoef cf,
    double* __restrict__ out, uint32_t* __restrict__ err) {
  extern __shared__ uint8_t sraw[];
  double* stages =
      reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(sraw) + 127) & ~uintptr_t(127));
  uint64_t* full = reinterpret_cast<uint64_t*>(stages + kStRing * kStStage);
  uint64_t* empty = full + kStRing;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kStRing);
  const int itiles = (ni + kStI - 1) / kStI;
  const int64_t nkx = nk + 2 * kFDn;
  const int64_t plane_pts = (int64_t)ni * nj;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cols = itiles * ((nj + kStJ - 1) / kStJ);
  __shared__ StWork work;
  if (threadIdx.x == 0) {
    const int G = gridDim.x, full_tiles = tiles / G * G;
    const int64_t rest = (int64_t)(tiles - full_tiles) * nk;
    const int lo = (int)(blockIdx.x * rest / G), hi = (int)((blockIdx.x + 1) * rest / G);
    work.waves = tiles / G;
    work.first = full_tiles + lo / nk;
    work.ka = lo % nk;
    work.len = hi - lo;
    for (int b = 0; b < kStRing; ++b) {
      mbar_init(&full[b], 33);  // the TMA loads and 32 lanes' copies of A
      mbar_init(&empty[b], kStConsumerWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();

  int tile, k0, k1;
  if (warp == kStConsumerWarps) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      tma_prefetch_desc(&mapP);
      tma_prefetch_desc(&mapC);
      tma_prefetch_desc(&mapF);
    }
    uint32_t it = 0;
    bool ok = true;
    for (int n = 0; ok && st_piece(&work, n, nk, &tile, &k0, &k1); ++n) {
      const int col = tile % cols, q = tile / cols;
      const int i0 = col % itiles * kStI, j0 = col / itiles * kStJ;
      const int t = q / (16 / kSlab), b0 = q % (16 / kSlab) * kSlab;
      const int jl = lane / kStI, i = i0 + lane % kStI;
      const double* Ak = A + i + (int64_t)(j0 + jl) * ni + k0 * plane_pts;
      for (int u = -kStFills; u < k1 - k0; ++u, ++it) {
        const uint32_t b = it % kStRing;
        if (it >= kStRing && (*abort_flag || !mbar_wait(&empty[b], (it / kStRing - 1) & 1, err, kDevErrStencil)))
          ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          *abort_flag = 1;
          break;
        }
        double* st = stages + b * kStStage;
        if (u < 0) {  // planes k0 - 6 .. k0 + 5 for the queues, kStFill a stage
          if (lane == 0) {
            mbar_arrive_expect_tx(&full[b], kStFill * kStCenter * 8);
            tma_load_4d(st, &mapF, &full[b], b0, i0 + kFDn, j0 + kFDn,
                        (int)(t * nkx + k0 + (u + kStFills) * kStFill));
          }
        } else {
          if (lane == 0) {
            mbar_arrive_expect_tx(&full[b], kStTxBytes);
            tma_load_4d(st, &mapP, &full[b], b0, i0, j0, (int)(t * nkx + k0 + u + kFDn));
            tma_load_4d(st + kStPlane, &mapC, &full[b], b0, i0 + kFDn, j0 + kFDn,
                        (int)(t * nkx + k0 + u + 2 * kFDn));
          }
          double* As = st + kStPlane + kStCenter + lane;
#pragma unroll
          for (int m = 0; m < kStJ; m += 32 / kStI)
            if (i < ni && j0 + jl + m < nj) cp_async8(As + m * kStI, Ak + (int64_t)m * ni, 8);
          Ak += plane_pts;
        }
        cp_async_arrive(&full[b]);
      }
    }
    // The CTA leaves only after its last loads have landed (immediate on
    // the normal path: the consumers waited for every one of them).
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (uint32_t v = it > kStRing ? it - kStRing : 0; v < it; ++v)
      mbar_wait(&full[v % kStRing], (v / kStRing) & 1, err, kDevErrStencil);
    return;
  }

  // -------------------------------------------------------------- consumers
  const int bp = lane % kBP;
  const int il = warp % (kStI * kBP / 32) * (32 / kBP) + lane / kBP;
  const int jA = warp / (kStI * kBP / 32) * 2;  // tile rows jA, jA + 1
  // Lane pair (il, row) offsets in a stage, in double2 units.
  const int pA = ((jA + kFDn) * kStHI + il + kFDn) * kBP + bp;  // halo plane, row jA
  const int yA = (jA * kStHI + il + kFDn) * kBP + bp;            // halo plane, row jA - 6
  const int cA = (jA * kStI + il) * kBP + bp;                     // center box, row jA
  const int64_t K = plane_pts * nk;
  uint32_t buf = 0, ph = 0;
  for (int n = 0; st_piece(&work, n, nk, &tile, &k0, &k1); ++n) {
    const int col = tile % cols, q = tile / cols;
    const int i = col % itiles * kStI + il, j = col / itiles * kStJ + jA;
    const int b = q * kSlab + 2 * bp;
    const bool actA = i < ni && j < nj && b < nb;
    const bool actB = i < ni && j + 1 < nj && b < nb;
    double2 zqA[kZq], zqB[kZq];
#pragma unroll
    for (int f = 0; f < kStFills; ++f) {  // planes k0 - 6 .. k0 + 5
      if (!*abort_flag && !mbar_wait(&full[buf], ph, err, kDevErrStencil)) *abort_flag = 1;
      const double2* C = reinterpret_cast<const double2*>(stages + buf * kStStage);
#pragma unroll
      for (int d = 0; d < kStFill; ++d) {
        zqA[f * kStFill + d] = C[d * (kStCenter / 2) + cA];
        zqB[f * kStFill + d] = C[d * (kStCenter / 2) + cA + kStI * kBP];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[buf]);
      if (++buf == kStRing) {
        buf = 0;
        ph ^= 1;
      }
    }
    double* o = out + ((int64_t)(b / OT) * K + i + (int64_t)j * ni + k0 * plane_pts) * OT + b % OT;
    for (int kb = k0; kb < k1; kb += kZq) {
#pragma unroll
      for (int u = 0; u < kZq; ++u) {
        if (kb + u >= k1) break;
        if (!*abort_flag && !mbar_wait(&full[buf], ph, err, kDevErrStencil)) *abort_flag = 1;
        const double* st = stages + buf * kStStage;
        const double2* P = reinterpret_cast<const double2*>(st);
        const double2* C = reinterpret_cast<const double2*>(st + kStPlane);
        const double* As = st + kStPlane + kStCenter + jA * kStI + il;
        zqA[(u + 2 * kFDn) % kZq] = C[cA];
        zqB[(u + 2 * kFDn) % kZq] = C[cA + kStI * kBP];
        if (actA) {
          const double aA = As[0] + cf.c0;
          const double aB = As[kStI] + cf.c0;
          double2 Y[2 * kFDn + 2];  // rows jA - 6 .. jA + 7
#pragma unroll
          for (int d = 0; d < 2 * kFDn + 2; ++d) Y[d] = P[yA + d * kStHI * kBP];
          const double2 ca = zqA[(u + kFDn) % kZq], cb = zqB[(u + kFDn) % kZq];
          double a0 = ca.x * aA, a1 = ca.y * aA;
          double b0 = cb.x * aB, b1 = cb.y * aB;
#pragma unroll
          for (int r = 1; r <= kFDn; ++r) {
            const double2 xpA = P[pA + kBP * r], xmA = P[pA - kBP * r];
            const double2 xpB = P[pA + kBP * (kStHI + r)], xmB = P[pA + kBP * (kStHI - r)];
            a0 = fma(xpA.x + xmA.x, cf.cx[r], a0);
            a1 = fma(xpA.y + xmA.y, cf.cx[r], a1);
            b0 = fma(xpB.x + xmB.x, cf.cx[r], b0);
            b1 = fma(xpB.y + xmB.y, cf.cx[r], b1);
            a0 = fma(Y[kFDn + r].x + Y[kFDn - r].x, cf.cy[r], a0);
            a1 = fma(Y[kFDn + r].y + Y[kFDn - r].y, cf.cy[r], a1);
            b0 = fma(Y[kFDn + 1 + r].x + Y[kFDn + 1 - r].x, cf.cy[r], b0);
            b1 = fma(Y[kFDn + 1 + r].y + Y[kFDn + 1 - r].y, cf.cy[r], b1);
            const double2 zpA = zqA[(u + kFDn + r) % kZq], zmA = zqA[(u + kFDn - r + kZq) % kZq];
            const double2 zpB = zqB[(u + kFDn + r) % kZq], zmB = zqB[(u + kFDn - r + kZq) % kZq];
            a0 = fma(zpA.x + zmA.x, cf.cz[r], a0);
            a1 = fma(zpA.y + zmA.y, cf.cz[r], a1);
            b0 = fma(zpB.x + zmB.x, cf.cz[r], b0);
            b1 = fma(zpB.y + zmB.y, cf.cz[r], b1);
          }
          if (b + 1 < nb)
            *reinterpret_cast<double2*>(o) = make_double2(a0, a1);
          else
            o[0] = a0;  // lane b + 1 is padding: left untouched
          if (actB) {
            double* o2 = o + (int64_t)ni * OT;
            if (b + 1 < nb)
              *reinterpret_cast<double2*>(o2) = make_double2(b0, b1);
            else
              o2[0] = b0;
          }
        }
        o += plane_pts * OT;
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[buf]);
        if (++buf == kStRing) {
          buf = 0;
          ph ^= 1;
        }
      }
    }
  }
}

// One warp per extended row (tile t, k_ex, j_ex): ext[(t K_ex + g_ex) 16 + l] =
// local[(t K + g) 16 + l], g the periodic image of g_ex's interior point; 16-byte
// lane pairs. Bound by memory once enough of it is asked for: kHaloLoads loads
// stand before the first store (a 48-point row with its halo at once), and the
// stores stream past L2. One 256-thread CTA per row, a load and a store at a time
// -> this: 48^3 x 506 229 -> 199 us (6.7 TB/s, a plain copy's rate), 24^3 x 512
// 64 -> 42 us, 48^3 x 72 40 -> 35 us, 33 x 35 x 41 x 512 130 -> 101 us. Longer rows
// take a second round: 49^3 x 480 232 -> 200 us, 56^3 x 318 211 -> 189 us, 80^3 x 112
// 197 -> 185 us; rounds of equal length are slower (207, 193 and 188 us). 4 loads in
// 8 warps: 204, 42 and 36 us; 8 loads took 260 us on 48^3; without the streaming hint
// 234 us.
constexpr int kHaloLoads = 15;
constexpr int kHaloWarps = 4;
__global__ void __launch_bounds__(kHaloWarps * 32) halo_periodic_kernel(
    int64_t rows, int ni, int nj, int nk, int FDn, const double* __restrict__ local,
    double* __restrict__ ext) {
  const int64_t nix = ni + 2 * FDn, njx = nj + 2 * FDn, nkx = nk + 2 * FDn;
  // row = (t * nkx + kx) * njx + jx
  const int64_t row = (int64_t)blockIdx.x * kHaloWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int64_t jx = row % njx, kx = (row / njx) % nkx, t = row / (njx * nkx);
  int jl = (int)jx - FDn, kl = (int)kx - FDn;
  jl += jl < 0 ? nj : (jl >= nj ? -nj : 0);
  kl += kl < 0 ? nk : (kl >= nk ? -nk : 0);
  const int64_t K = (int64_t)ni * nj * nk;
  const double2* src = reinterpret_cast<const double2*>(local) +
                       (t * K + (int64_t)jl * ni + (int64_t)kl * ni * nj) * 8;
  double2* dst = reinterpret_cast<double2*>(ext) + row * nix * 8;
  const int n = (int)nix * 8;
  for (int e0 = threadIdx.x & 31; e0 < n; e0 += 32 * kHaloLoads) {
    double2 v[kHaloLoads];
#pragma unroll
    for (int x = 0; x < kHaloLoads; ++x) {
      const int e = e0 + 32 * x;
      int il = (e >> 3) - FDn;
      il += il < 0 ? ni : (il >= ni ? -ni : 0);
      if (e < n) v[x] = __ldg(src + il * 8 + (e & 7));
    }
#pragma unroll
    for (int x = 0; x < kHaloLoads; ++x)
      if (e0 + 32 * x < n) __stcs(dst + e0 + 32 * x, v[x]);
  }
}

}  // namespace

namespace {

template <int OT>
int launch_staged(const CUtensorMap& mapP, const CUtensorMap& mapC, const CUtensorMap& mapF, int ni,
                  int nj, int nk, int nb, int tiles, int grid, const double* A,
                  const StencilCoef& cf, double* out, uint32_t* err, cudaStream_t s) {
  static bool attr_set[64] = {};  // function attributes are per device
  int d = 0;
  SKG_CUDA(cudaGetDevice(&d));
  if (d < 0 || d >= 64) return fail(SKGEMM_ERR_INVALID_ARG, "device index");
  if (!attr_set[d]) {
    SKG_CUDA(cudaFuncSetAttribute(stencil_staged_kernel<OT>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, kStSmem));
    attr_set[d] = true;
  }
  KernelTimer kt_(s, "stencil_staged_kernel");
  stencil_staged_kernel<OT><<<grid, kStThreads, kStSmem, s>>>(mapP, mapC, mapF, ni, nj, nk, nb,
                                                              tiles, A, cf, out, err);
  SKG_CUDA(cudaGetLastError());
  return SKGEMM_OK;
}

}  // namespace

int launch_stencil_ext(int64_t ni, int64_t nj, int64_t nk, int64_t nb, int FDn,
                       const double* ext, const double* A, const double* cx, const double* cy,
                       const double* cz, double c0, double* out, int out_tile, int num_sms,
                       uint32_t* err, cudaStream_t s) {
  if (ni < 0 || nj < 0 || nk < 0 || nb < 0) return fail(SKGEMM_ERR_INVALID_ARG, "negative extent");
  if (FDn != kFDn)
    return fail(SKGEMM_ERR_UNSUPPORTED, "stencil radius FDn must be 6 (the reference's kernels)");
  if (out_tile != 16 && out_tile != 32) return fail(SKGEMM_ERR_INVALID_ARG, "out_tile must be 16 or 32");
  if (ni == 0 || nj == 0 || nk == 0 || nb == 0) return SKGEMM_OK;
  if (!ext || !A || !cx || !cy || !cz || !out) return fail(SKGEMM_ERR_INVALID_ARG, "null pointer");
  if (ni > (1 << 20) || nj > (1 << 20) || nk > (1 << 20) || ni * nj * nk > ((int64_t)1 << 40))
    return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  StencilCoef cf;
  for (int r = 0; r <= kFDn; ++r) {
    cf.cx[r] = cx[r];
    cf.cy[r] = cy[r];
    cf.cz[r] = cz[r];
  }
  cf.c0 = c0;
  if ((reinterpret_cast<uintptr_t>(ext) | reinterpret_cast<uintptr_t>(out)) & 15)
    return fail(SKGEMM_ERR_INVALID_ARG, "stencil arrays must be 16-byte aligned");
  if ((reinterpret_cast<uintptr_t>(A) & 15) != 0)
    return fail(SKGEMM_ERR_INVALID_ARG, "stencil A_diag must be 16-byte aligned");
  const int64_t cols = ((ni + kStI - 1) / kStI) * ((nj + kStJ - 1) / kStJ);
  const int64_t tiles = (nb + 15) / 16;
  if (cols > INT32_MAX || tiles > 16383) return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  const int64_t nix = ni + 2 * kFDn, njx = nj + 2 * kFDn, nkx = nk + 2 * kFDn;
  if (tiles * nkx > INT32_MAX || ni * nj * nk + 2 >= INT32_MAX)
    return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  // Extended Psi as a 4-D tensor [tiles * nkx][njx][nix][16 lanes]: boxes of
  // 8 lanes x 28 x 20 points (halo planes), 8 lanes x 16 x 8 points (z
  // entries) and 4 such planes (filling the z queues). Zero fill outside.
  CUtensorMap mapP, mapC, mapF;
  const uint64_t dims[4] = {16, (uint64_t)nix, (uint64_t)njx, (uint64_t)(tiles * nkx)};
  const uint64_t strides[3] = {16 * 8, (uint64_t)nix * 16 * 8, (uint64_t)(nix * njx) * 16 * 8};
  const uint32_t boxP[4] = {(uint32_t)kSlab, (uint32_t)kStHI, (uint32_t)kStHJ, 1};
  const uint32_t boxC[4] = {(uint32_t)kSlab, (uint32_t)kStI, (uint32_t)kStJ, 1};
  const uint32_t boxF[4] = {(uint32_t)kSlab, (uint32_t)kStI, (uint32_t)kStJ, (uint32_t)kStFill};
  int st;
  if ((st = encode_tiled(&mapP, 4, ext, dims, strides, boxP, CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         CU_TENSOR_MAP_SWIZZLE_NONE)) ||
      (st = encode_tiled(&mapC, 4, ext, dims, strides, boxC, CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         CU_TENSOR_MAP_SWIZZLE_NONE)) ||
      (st = encode_tiled(&mapF, 4, ext, dims, strides, boxF, CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         CU_TENSOR_MAP_SWIZZLE_NONE)))
    return st;
  // One CTA per SM; slabs past nb have no work.
  const int64_t work = cols * ((nb + kSlab - 1) / kSlab);
  if (work > INT32_MAX) return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  // A CTA per tile at least, where tiles have fewer planes than that (6^3 x 512: 12.8
  // -> 12.2 us).
  const int grid = (int)std::min<int64_t>(num_sms, std::max<int64_t>(work, work * nk / kStMinSteps));
  if (out_tile == 32)
    return launch_staged<32>(mapP, mapC, mapF, (int)ni, (int)nj, (int)nk, (int)nb, (int)work, grid, A,
                             cf, out, err, s);
  return launch_staged<16>(mapP, mapC, mapF, (int)ni, (int)nj, (int)nk, (int)nb, (int)work, grid, A,
                           cf, out, err, s);
}

int launch_halo_periodic(int64_t ni, int64_t nj, int64_t nk, int64_t nb, int FDn,
                         const double* local, double* ext, cudaStream_t s) {
  if (ni < 0 || nj < 0 || nk < 0 || nb < 0 || FDn < 0)
    return fail(SKGEMM_ERR_INVALID_ARG, "negative extent");
  if (ni == 0 || nj == 0 || nk == 0 || nb == 0) return SKGEMM_OK;
  if (FDn > ni || FDn > nj || FDn > nk)
    return fail(SKGEMM_ERR_INVALID_ARG, "periodic halo wider than the domain");
  if (!local || !ext) return fail(SKGEMM_ERR_INVALID_ARG, "null pointer");
  if ((reinterpret_cast<uintptr_t>(local) | reinterpret_cast<uintptr_t>(ext)) & 15)
    return fail(SKGEMM_ERR_INVALID_ARG, "halo arrays must be 16-byte aligned");
  if (ni > (1 << 20) || nj > (1 << 20) || nk > (1 << 20))
    return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  const int64_t rows = ((nb + 15) / 16) * (nk + 2 * FDn) * (nj + 2 * FDn);
  if (rows > INT32_MAX) return fail(SKGEMM_ERR_INVALID_ARG, "grid too large");
  KernelTimer kt_(s, "halo_periodic_kernel");
  halo_periodic_kernel<<<(unsigned)((rows + kHaloWarps - 1) / kHaloWarps), kHaloWarps * 32, 0, s>>>(
      rows, (int)ni, (int)nj, (int)nk, FDn, local, ext);
  SKG_CUDA(cudaGetLastError());
  return SKGEMM_OK;
}

}  // namespace skg
