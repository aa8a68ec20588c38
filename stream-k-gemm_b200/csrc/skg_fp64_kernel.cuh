// Persistent Stream-K FP64 GEMM kernel for sm_100a (native-precision path).
//
// Computes, over a set of BM x BN output tiles, acc(m,n) = sum_k A(m,k) B(k,n)
// and applies one of three epilogues:
//   kOutRowMajor  D[m*ldd + n]                     = alpha*acc + gamma
//                 (gemm<double>::compute_packed, gemm_opt.cpp:314; gamma is a
//                  scalar added to every element, gemm_opt.cpp:201-204)
//   kOutSyrkUpper C[m + n*ldd], m <= n only        = alpha*acc + beta*C
//                 (sme_syrk<double>::compute, sme_syrk.hpp:137; upper triangle of
//                  a column-major M x M matrix)
//   kOutBand16    D[(n/16)*M*16 + m*16 + n%16]     = acc
//                 (sme_gemm_trp_3d<double>::compute, sme_trp_3d.hpp:194; the
//                  rotation writes band-packed output, no scaling)
//
// Work decomposition (Stream-K): the MAC-loop iterations of all tiles
// (tiles * ceil(K/BK)) are split evenly over the persistent CTAs. A CTA whose
// range starts inside a tile stores its partial accumulator to a workspace slot
// and publishes a flag. A tile of fewer than kSharedParts parts is finished by the
// CTA that owns its k = 0 segment: it waits (with a time budget) for the flags, adds
// the partials and runs the epilogue. A tile of more parts is finished by all the
// CTAs whose range ends in it (shared_fixup below), each a slice of the
// elements. The reduction order is a pure function of the schedule, so results
// are bitwise reproducible run to run.
//
// The same body serves one problem (fp64_streamk_kernel, fp64_streamk_kernel64 and
// fp64_streamk_kernel32: BM = BN = 128, 64 and 32) and a group of problems in one
// launch (fp64_grouped_kernel<TileShape>, 128 or 64, the batched path: iterations of
// all problems concatenated, see Fp64Group).
//
// Data movement: one producer warp issues TMA tile loads (128B-swizzled boxes
// of 16 doubles x BK rows) into a ring of kStages; 8 consumer warps (4 on 32 x 32
// tiles) run FP64 DMMA (m16n8k8) from shared memory. Every operand tile in shared memory is a set of
// "chunks" [BK][16] doubles (16 rows/columns of the output, k-major rows of
// 128 B), which is exactly the reference's packed panel layout
// ([tiles][K][16], gemm_opt.cpp:342-354) restricted to a BK slice.
//
// Fragment mapping: lane (g = lane/4, t = lane%4) reads one 16-byte unit per
// (chunk, k-row) with ld.shared.v2.f64. MMA row r maps to chunk row 2r (r<8)
// or 2(r-8)+1, MMA column c of the even/odd n8 block of a pair maps to chunk
// column 2c / 2c+1, and MMA k index t / t+4 maps to k-row 2t / 2t+1 of the k8
// step. With the 128B swizzle (16B unit ^= k-row mod 8) every quarter-warp hits
// eight distinct bank groups, so fragment loads are conflict-free.
#pragma once

#include "skg_common.cuh"

#include "skg_fp64_types.h"

namespace skg {

// Tile index -> (tm, tn). kTilesAll: row-major over (tm, tn) so that
// consecutive tiles of one CTA share the A panel (L2 reuse). kTilesUpper:
// row-major over the upper triangle tm <= tn.
__device__ __forceinline__ void tile_coords(const Fp64Params& p, int tile, int& tm, int& tn) {
  if (p.tile_order == kTilesAll) {
    tm = tile / p.tiles_n;
    tn = tile - tm * p.tiles_n;
  } else {
    int T = p.tiles_n;
    int r = 0, rem = tile;
    while (rem >= T - r) {
      rem -= T - r;
      ++r;
    }
    tm = r;
    tn = r + rem;
  }
}

__device__ __forceinline__ void load_operand(int kind, const CUtensorMap* map, uint8_t* dst,
                                             uint64_t* bar, int tile_idx, int rows_per_tile,
                                             int k0) {
  if (kind == kOpPacked16) {
    tma_load_3d(dst, map, bar, 0, k0, tile_idx * (rows_per_tile / 16));
  } else if (kind == kOpBandK) {
    tma_load_3d(dst, map, bar, 0, tile_idx * rows_per_tile, k0 / 16);
  } else if (kind == kOpPacked32) {
    const int per = rows_per_tile / 32;
    tma_load_3d(dst, map, bar, 0, k0, tile_idx * per);
    tma_load_3d(dst + per * kChunkBytes, map, bar, 16, k0, tile_idx * per);
  } else {
#pragma unroll 1
    for (int c = 0; c < rows_per_tile / 16; ++c)
      tma_load_2d(dst + c * kChunkBytes, map, bar, tile_idx * rows_per_tile + c * 16, k0);
  }
}

__device__ __forceinline__ void store_row4(const Fp64Params& p, int64_t m, int64_t n, double v0,
                                           double v1, double v2, double v3) {
  // Four consecutive columns n..n+3 of output row m.
  if (m >= p.M) return;
  double v[4] = {v0, v1, v2, v3};
  if (p.out_kind == kOutRowMajor) {
    double* row = p.D + m * p.ldd;
    bool vec_ok = (n + 3 < p.N) && ((((uintptr_t)(row + n)) & 15) == 0);
    if (vec_ok) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = p.alpha * v[i] + p.gamma;
      *reinterpret_cast<double2*>(row + n) = make_double2(v[0], v[1]);
      *reinterpret_cast<double2*>(row + n + 2) = make_double2(v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < p.N) row[n + i] = p.alpha * v[i] + p.gamma;
    }
  } else if (p.out_kind == kOutSyrkUpper) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int64_t col = n + i;
      if (col < p.N && m <= col) {
        double* c = p.D + m + col * p.ldd;
        double r = p.alpha * v[i];
        if (!p.beta_zero) r += p.gamma * (*c);
        *c = r;
      }
    }
  } else {  // kOutBand16
    double* dst = p.D + (n >> 4) * (p.M * 16) + m * 16 + (n & 15);
    if (n + 3 < p.N) {
      *reinterpret_cast<double2*>(dst) = make_double2(v[0], v[1]);
      *reinterpret_cast<double2*>(dst + 2) = make_double2(v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < p.N) dst[i] = v[i];
    }
  }
}

// One problem: its parameters and tensor maps are kernel parameters; flags
// carry the host-side epoch of the launch.
struct SingleSched {
  const Fp64Params& p;
  const CUtensorMap* mA;
  const CUtensorMap* mB;
  __device__ __forceinline__ const IterSplit& split() const { return p.split; }
  __device__ __forceinline__ const Fp64Params& prob(int) const { return p; }
  __device__ __forceinline__ const CUtensorMap* map_a(int) const { return mA; }
  __device__ __forceinline__ const CUtensorMap* map_b(int) const { return mB; }
  __device__ __forceinline__ int64_t begin(int) const { return 0; }
  __device__ __forceinline__ int locate(int64_t, int) const { return 0; }
  __device__ __forceinline__ double* workspace() const { return p.workspace; }
  __device__ __forceinline__ uint32_t* flags() const { return p.flags; }
  __device__ __forceinline__ uint32_t* err() const { return p.err; }
  __device__ __forceinline__ uint32_t pub() const { return p.epoch; }
  __device__ __forceinline__ bool spread() const { return p.spread != 0; }
  static constexpr bool kOwnersOnly = false;
  __device__ __forceinline__ int64_t cta_begin(int c) const { return p.split.begin(c); }
};

// A group of problems: descriptors and tensor maps in global memory.
template <bool SPREAD>
struct GroupSched {
  const Fp64Group& g;
  __device__ __forceinline__ const IterSplit& split() const { return g.split; }
  __device__ __forceinline__ const Fp64Params& prob(int i) const { return g.probs[i]; }
  __device__ __forceinline__ const CUtensorMap* map_a(int i) const { return g.maps + 2 * i; }
  __device__ __forceinline__ const CUtensorMap* map_b(int i) const { return g.maps + 2 * i + 1; }
  __device__ __forceinline__ int64_t begin(int i) const { return g.iter_begin[i]; }
  // Problem containing iteration `it`; `hint` is a problem at or before it.
  __device__ __forceinline__ int locate(int64_t it, int hint) const {
    int i = hint;
    if (g.iter_begin[i + 1] <= it) {
      int lo = i + 1, hi = g.num_problems - 1;  // invariant: answer in [lo, hi]
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g.iter_begin[mid] <= it) lo = mid; else hi = mid - 1;
      }
      i = lo;
    }
    return i;
  }
  __device__ __forceinline__ double* workspace() const { return g.workspace; }
  __device__ __forceinline__ uint32_t* flags() const { return g.flags; }
  __device__ __forceinline__ uint32_t* err() const { return g.err; }
  __device__ __forceinline__ uint32_t pub() const { return 1u; }
  __device__ __forceinline__ bool spread() const { return SPREAD; }
  // Without the shared fix-up the ranges are divided in 64 bits, and a tile's end is
  // found where it is needed: the compiler's schedule of the whole loop follows (16
  // sets of three problems 1198 -> 1170 us, rotations 4 x 65536 x 32 and 2 x 65536 x
  // 256 792 -> 774).
  static constexpr bool kOwnersOnly = !SPREAD;
  __device__ __forceinline__ int64_t cta_begin(int c) const {
    return kOwnersOnly ? (int64_t)c * g.total_iters / g.grid : g.split.begin(c);
  }
};

// Where iteration `it` (< it_end) falls: problem, tile, k-block range of this
// CTA inside the tile and the tile coordinates.
struct Seg {
  int pid, tile, kb, ke, tm, tn;
};

template <class Sched>
__device__ __forceinline__ Seg locate_seg(const Sched& S, int64_t it, int64_t it_end, int hint) {
  Seg sg;
  sg.pid = S.locate(it, hint);
  const Fp64Params& q = S.prob(sg.pid);
  const int ipt = q.iters_per_tile;
  const int64_t local = it - S.begin(sg.pid);
  sg.tile = (int)(local / ipt);
  sg.kb = (int)(local - (int64_t)sg.tile * ipt);
  sg.ke = (int)((int64_t)ipt < sg.kb + (it_end - it) ? (int64_t)ipt : sg.kb + (it_end - it));
  tile_coords(q, sg.tile, sg.tm, sg.tn);
  return sg;
}

// One output element (m, n) of the finished sum v.
__device__ __forceinline__ void store_one(const Fp64Params& p, int64_t m, int64_t n, double v) {
  if (m >= p.M || n >= p.N) return;
  if (p.out_kind == kOutRowMajor) {
    p.D[m * p.ldd + n] = p.alpha * v + p.gamma;
  } else if (p.out_kind == kOutSyrkUpper) {
    if (m > n) return;
    double* c = p.D + m + n * p.ldd;
    double r = p.alpha * v;
    if (!p.beta_zero) r += p.gamma * (*c);
    *c = r;
  } else {  // kOutBand16
    p.D[(n >> 4) * (p.M * 16) + m * 16 + (n & 15)] = v;
  }
}

// Parts from which a tile's fix-up is shared. Fewer are added by the owner
// alone, which needs no exchange of its own part: with 2 / 3 / 4 as the line a
// 10000 x 32 rotation (3 parts) takes 14.7 / 10.7 / 10.7 us (10.6 with the
// owner) and a dense 1000^3 product (4 parts) 87.7 / 88.3 / 85.0 us (82.2);
// with 5 both stay, and the tiles cut into more parts are faster shared.
constexpr int kSharedParts = 5;

// CTAs of the tile [tile_begin, tile_end) in iterations: first .. last hold a
// part of it, first .. red_last finish it (their ranges end in it).
struct FixupSpan {
  int first, last, red_last;
};

template <class Sched>
__device__ __forceinline__ FixupSpan fixup_span(const Sched& S, int64_t tile_begin,
                                                int64_t tile_end) {
  const IterSplit& sp = S.split();
  FixupSpan f;
  f.first = sp.cta_of(tile_begin);
  f.last = sp.cta_of(tile_end - 1);
  f.red_last = sp.begin(f.last + 1) <= tile_end ? f.last : f.last - 1;
  return f;
}

// Named barrier 1 over the consumer threads; true if `v` holds on all of them.
template <int kThreads>
__device__ __forceinline__ bool bar_and(bool v) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"((uint32_t)v), "n"(kThreads)
      : "memory");
  return all != 0;
}

// Shared fix-up of a tile of kSharedParts parts or more. All parts are in
// workspace slots (the owner's in slot grid + first); CTA `cta` of first ..
// red_last sums its slice of the tile's elements over the parts and stores
// them. Added by the owner alone, the parts are a serial chain of
// last - first reads of a whole tile by one SM: a 10000 x 32 SYRK (295 parts
// of 32 KB) took 334 us and a 13824 x 128 GEMM (147 of 128 KB) 445 us, with this
// alone 21 and 29 us. Here every SM reads one tile's worth.
// Slices of fewer elements than threads are summed by several threads an element,
// each over a contiguous run of parts, and the runs added in order. The CTAs
// of a tile finish together (equal ranges), so nobody waits long; all CTAs
// are co-resident (cooperative launches). A flag that does not arrive within the
// budget is recorded in the error word, and the slice is not stored: the missing
// part's slot holds an earlier tile's sums.
template <class TS, bool AKM, class Sched>
__device__ __forceinline__ void shared_fixup(const Sched& S, const Fp64Params& q, FixupSpan f,
                                          int cta, int tm, int tn, uint32_t pubval, double* red) {
  constexpr int kSlot = TS::BM * TS::BN;
  constexpr int NJ = TS::NJ;
  const int tid = threadIdx.x;  // 0 .. TS::kCons - 1
  const int n = f.last - f.first + 1, nred = f.red_last - f.first + 1;
  bool here = true;
  for (int j = tid; j < n; j += TS::kCons)
    here &= fixup_flag_wait(S.flags() + (j == 0 ? S.split().grid + f.first : f.first + j), pubval,
                            S.err(), kFixupBudgetNs);
  if (!bar_and<TS::kCons>(here)) return;
  const int idx = cta - f.first;
  const int e0 = (int)((int64_t)idx * kSlot / nred), e1 = (int)((int64_t)(idx + 1) * kSlot / nred);
  const int ne = e1 - e0;
  // part(j): slot of the j-th part in ascending k.
  const double* own = S.workspace() + ((int64_t)S.split().grid + f.first) * kSlot;
  const double* others = S.workspace() + (int64_t)f.first * kSlot;
  const int64_t mb = (int64_t)tm * TS::BM, nbase = (int64_t)tn * TS::BN;
  auto finish = [&](int e, double v) {
    // Slot element e = reg * kCons + thread: the accumulator layout.
    const int reg = e / TS::kCons, th = e % TS::kCons;
    const int r = reg & 3, j = (reg >> 2) % NJ, i = (reg >> 2) / NJ;
    const int w = th >> 5, l = th & 31, g = l >> 2, t = l & 3;
    const int row = (w / TS::WN) * (TS::BM / TS::WM) + i * 16 +
                    (AKM ? 4 * (g & 1) + (g >> 1) + 8 * (r >> 1) : 2 * g + (r >> 1));
    const int col = (w % TS::WN) * (TS::BN / TS::WN) + (j >> 1) * 16 + 4 * t + (j & 1) + 2 * (r & 1);
    store_one(q, mb + row, nbase + col, v);
  };
  const int P = ne > 0 ? min(TS::kCons / ne, n) : 0;
  if (P <= 1) {
    // Eight elements a thread at a time: the loads of one part are in flight
    // together (the sums are bound by their latency).
    constexpr int U = 8;
    for (int eb = e0 + tid; eb < e1; eb += U * TS::kCons) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = eb + u * TS::kCons;
        v[u] = e < e1 ? __ldcg(own + e) : 0.0;
      }
#pragma unroll 2
      for (int j = 1; j < n; ++j) {
        const double* part = others + (int64_t)j * kSlot + eb;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (eb + u * TS::kCons < e1) v[u] += __ldcg(part + u * TS::kCons);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (eb + u * TS::kCons < e1) finish(eb + u * TS::kCons, v[u]);
    }
    return;
  }
  const int grp = tid / ne, e = e0 + tid % ne;
  if (grp < P) {
    const int j0 = (int)((int64_t)grp * n / P), j1 = (int)((int64_t)(grp + 1) * n / P);
    double v = j0 == 0 ? __ldcg(own + e) : __ldcg(others + (int64_t)j0 * kSlot + e);
#pragma unroll 8
    for (int j = j0 + 1; j < j1; ++j) v += __ldcg(others + (int64_t)j * kSlot + e);
    red[grp * ne + tid % ne] = v;
  }
  asm volatile("bar.sync 1, %0;" ::"n"(TS::kCons) : "memory");
  if (tid < ne) {
    double v = red[tid];
    for (int p = 1; p < P; ++p) v += red[p * ne + tid];
    finish(e0 + tid, v);
  }
}

template <class TS, bool AKM = false, class Sched>
__device__ __forceinline__ void streamk_body(const Sched& S) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * TS::kStage);
  uint64_t* empty_bar = full_bar + kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty_bar + kStages);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cta = blockIdx.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], TS::kWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();

  const int64_t it_begin = S.cta_begin(cta);
  const int64_t it_end = S.cta_begin(cta + 1);

  if (warp == TS::kWarps) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int hint = S.locate(it_begin < it_end ? it_begin : 0, 0);
      int prefetched = -1;
      for (int64_t it = it_begin; it < it_end;) {
        const Seg sg = locate_seg(S, it, it_end, hint);
        hint = sg.pid;
        const Fp64Params& q = S.prob(sg.pid);
        const CUtensorMap* mA = S.map_a(sg.pid);
        const CUtensorMap* mB = S.map_b(sg.pid);
        if (prefetched != sg.pid) {
          tma_prefetch_desc(mA);
          tma_prefetch_desc(mB);
          prefetched = sg.pid;
        }
        for (int k = sg.kb; k < sg.ke; ++k) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, S.err(), kDevErrFp64)) *abort_flag = 1;
          if (*abort_flag) break;
          uint8_t* sa = smem + stage * TS::kStage;
          uint8_t* sb = sa + TS::kABytes;
          mbar_arrive_expect_tx(&full_bar[stage], TS::kStage);
          load_operand(q.a_kind, mA, sa, &full_bar[stage], sg.tm, TS::BM, k * kBK);
          load_operand(q.b_kind, mB, sb, &full_bar[stage], sg.tn, TS::BN, k * kBK);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (*abort_flag) break;
        it += sg.ke - sg.kb;
      }
    }
    return;
  }

  // -------------------------------------------------------------- consumers
  constexpr int MI = TS::MI, NJ = TS::NJ, NQ = TS::NQ;
  const int wm = warp / TS::WN;  // rows wm*BM/WM ..
  const int wn = warp % TS::WN;  // cols wn*BN/WN ..
  const int g = lane >> 2;
  const int t = lane & 3;
  // Byte offsets inside a chunk of the two k-rows this lane reads per k8 step.
  // Row 2t holds MMA k index t, row 2t+1 holds MMA k index t+4; the 16-byte
  // unit g is XOR-swizzled with the row index (TMA SWIZZLE_128B).
  const uint32_t off_r0 = (2 * t) * 128 + ((g ^ (2 * t)) << 4);
  const uint32_t off_r1 = (2 * t + 1) * 128 + ((g ^ (2 * t + 1)) << 4);
  // K-major A (AKM): output row r holds its 16 k in one 128-byte row, the
  // 16-byte unit u at u ^ (r mod 8). MMA rows g and g + 8 are fed from tile
  // rows q(g) and 8 + q(g), q(g) = 4 (g % 2) + g / 2 (the epilogue stores
  // them there): the two g of a quarter-warp then differ in bit 2 of the
  // swizzle, so its 16-byte loads of unit 4s + t (k = 8s + 2t, 8s + 2t + 1)
  // hit 8 distinct units (conflict-free). Each load holds (a0, a2) or
  // (a1, a3) of the fragment and is transposed into its order. Step s's
  // unit is step 0's with bit 2 flipped: offset ^ (s << 6).
  const int qg = 4 * (g & 1) + (g >> 1);
  const uint32_t offk0 = qg * 128 + ((t ^ qg) << 4);
  const uint32_t smem_base = smem_u32(smem);
  __shared__ int fixup_ok;
  __shared__ double fixup_red[TS::kCons];

  double acc[MI][NJ][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

  int stage = 0;
  uint32_t phase = 0;
  bool aborted = false;
  int hint = S.locate(it_begin < it_end ? it_begin : 0, 0);
  const uint32_t pubval = S.pub();

  bool published = false;  // the last segment's partial sum went to a slot
  for (int64_t it = it_begin; it < it_end;) {
    const Seg sg = locate_seg(S, it, it_end, hint);
    hint = sg.pid;
    const Fp64Params& q = S.prob(sg.pid);
    // Shared-memory chunk of this warp's B column chunks (logical wn*NQ+qq).
    // A packed32 operand lands as [half][tile32][BK][16]: logical chunk c
    // sits at (c % 2) * (BN/32) + c / 2.
    uint32_t b_chunk[NQ];
    const bool b32 = !AKM && (q.b_kind == kOpPacked32);  // AKM: B never packed32
#pragma unroll
    for (int qq = 0; qq < NQ; ++qq) {
      const int c = wn * NQ + qq;
      b_chunk[qq] = b32 ? (uint32_t)((c & 1) * (TS::BN / 32) + (c >> 1)) : (uint32_t)c;
    }

    // Three iterations a trip (half the ring), so that the loop's own work
    // spreads over 48 k: GEMM 512 x 512 x 110592 1.670 -> 1.617 ms, SYRK 0.933
    // -> 0.921, rotation 110592 x 512 1.710 -> 1.680 (two, four, six a trip:
    // 1.617, 1.617, 1.616 / 0.930, 0.923, 0.923 / 1.685, 1.680, 1.681). Two in
    // groups of 64 x 64 tiles without long ones, many of them rotations of few
    // iterations: 16 sets of three problems 1170 -> 1140 us, their rotations 420 -> 408.
#pragma unroll (Sched::kOwnersOnly && TS::BM == 64 ? 2 : 3)
    for (int k = sg.kb; k < sg.ke && !aborted; ++k) {
      if (!mbar_wait(&full_bar[stage], phase, S.err(), kDevErrFp64)) {
        aborted = true;
        *abort_flag = 1;
        break;
      }
      const uint32_t sa = smem_base + stage * TS::kStage + (wm * MI) * kChunkBytes;
      const uint32_t sb = smem_base + stage * TS::kStage + TS::kABytes;
#pragma unroll
      for (int s = 0; s < kBK / 8; ++s) {
        const uint32_t ks = s * 8 * 128;  // k8 step = 8 rows of 128 B
        double2 a_lo[MI], a_hi[MI], b_lo[NQ], b_hi[NQ];
        auto load_b = [&]() {
#pragma unroll
          for (int qq = 0; qq < NQ; ++qq) {
            b_lo[qq] = lds128(sb + b_chunk[qq] * kChunkBytes + ks + off_r0);
            b_hi[qq] = lds128(sb + b_chunk[qq] * kChunkBytes + ks + off_r1);
          }
        };
        if constexpr (AKM) load_b();
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          if constexpr (AKM) {
            const uint32_t o = sa + i * kChunkBytes + (offk0 ^ (s << 6));
            const double2 r0 = lds128(o), r1 = lds128(o + 8 * 128);
            a_lo[i] = make_double2(r0.x, r1.x);
            a_hi[i] = make_double2(r0.y, r1.y);
          } else {
            a_lo[i] = lds128(sa + i * kChunkBytes + ks + off_r0);
            a_hi[i] = lds128(sa + i * kChunkBytes + ks + off_r1);
          }
        }
        if constexpr (!AKM) load_b();
        // The column direction turns at each row of MMAs (a neighbour shares
        // A or B) where that measured faster: GEMM 512 x 512 x 110592 on
        // 128 x 128 tiles 1.618 against 1.628 ms, the K-major rotation of
        // 13824 x 512 0.233 against 0.242 ms; no gain on 64 x 64 packed tiles.
        constexpr bool kTurn = TS::BM == 128 || AKM;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
#pragma unroll
          for (int j = 0; j < NQ; ++j) {
            const bool back = kTurn && (i & 1);
            const int qq = back ? NQ - 1 - j : j;
            auto even = [&]() {
              dmma_16x8x8(acc[i][2 * qq], a_lo[i].x, a_lo[i].y, a_hi[i].x, a_hi[i].y, b_lo[qq].x,
                          b_hi[qq].x);
            };
            if (!back) even();
            dmma_16x8x8(acc[i][2 * qq + 1], a_lo[i].x, a_lo[i].y, a_hi[i].x, a_hi[i].y,
                        b_lo[qq].y, b_hi[qq].y);
            if (back) even();
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[stage]);
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (aborted) break;

    // ---------------------------------------------------------- epilogue
    const bool owner = (sg.kb == 0);
    const bool complete = owner && (sg.ke == q.iters_per_tile);
    const int ctid = threadIdx.x;  // 0 .. TS::kCons - 1
    constexpr int kSlot = TS::BM * TS::BN;
    auto tile_end_of = [&]() -> int64_t {
      if constexpr (Sched::kOwnersOnly)
        return S.begin(sg.pid) + (int64_t)(sg.tile + 1) * q.iters_per_tile;
      return it - sg.kb + q.iters_per_tile;
    };
    // An owner without the whole tile is in its last segment. It adds the
    // other parts itself if they are few.
    const bool shared = owner && !complete && S.spread() && cta + kSharedParts <= S.split().grid &&
                        S.cta_begin(cta + kSharedParts - 1) < tile_end_of();
    if (!owner || shared) {
      // Publish this CTA's partial tile (layout [reg][thread], coalesced).
      const int slot_id = owner ? S.split().grid + cta : cta;
      double* slot = S.workspace() + (int64_t)slot_id * kSlot;
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r)
            __stcg(slot + ((i * NJ + j) * 4 + r) * TS::kCons + ctid, acc[i][j][r]);
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(TS::kCons));
      if (ctid == 0) st_release_gpu(S.flags() + slot_id, pubval);
      published = true;
    } else {
      published = false;
      if (!complete) {
        // Add the partials of the later CTAs that cover the rest of this tile,
        // in ascending k order. A flag that does not arrive within the budget
        // is recorded in the error word and its partial is skipped; the CTA
        // keeps consuming its pipeline so no copy is left in flight.
        const int64_t tile_end = tile_end_of();
        for (int c2 = cta + 1; c2 < S.split().grid; ++c2) {
          if (S.cta_begin(c2) >= tile_end) break;
          if (ctid == 0)
            fixup_ok = fixup_flag_wait(S.flags() + c2, pubval, S.err(), kFixupBudgetNs) ? 1 : 0;
          asm volatile("bar.sync 1, %0;" ::"n"(TS::kCons));
          const bool have = fixup_ok != 0;
          asm volatile("bar.sync 1, %0;" ::"n"(TS::kCons));
          if (!have) continue;
          const double* slot = S.workspace() + (int64_t)c2 * kSlot;
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
              for (int r = 0; r < 4; ++r)
                acc[i][j][r] += __ldcg(slot + ((i * NJ + j) * 4 + r) * TS::kCons + ctid);
        }
      }
      // Final epilogue for tile (tm, tn).
      const int64_t mbase = (int64_t)sg.tm * TS::BM + wm * (TS::BM / TS::WM);
      const int64_t nbase = (int64_t)sg.tn * TS::BN + wn * (TS::BN / TS::WN);
      const bool syrk_skip = (q.out_kind == kOutSyrkUpper) && (mbase > nbase + TS::BN / TS::WN - 1);
      if (!syrk_skip) {
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          // MMA rows g, g + 8 sit at tile rows 2g, 2g + 1 (AKM: q(g), 8 + q(g)).
          const int64_t m0 = mbase + i * 16 + (AKM ? qg : 2 * g);
          const int64_t m1 = m0 + (AKM ? 8 : 1);
#pragma unroll
          for (int qq = 0; qq < NQ; ++qq) {
            const int64_t n0 = nbase + qq * 16 + 4 * t;
            store_row4(q, m0, n0, acc[i][2 * qq][0], acc[i][2 * qq + 1][0], acc[i][2 * qq][1],
                       acc[i][2 * qq + 1][1]);
            store_row4(q, m1, n0, acc[i][2 * qq][2], acc[i][2 * qq + 1][2],
                       acc[i][2 * qq][3], acc[i][2 * qq + 1][3]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;
    it += sg.ke - sg.kb;
  }
  // The tile this CTA's range ends in, if its part of it went to a slot.
  if (published && S.spread() && !aborted) {
    const Seg sg = locate_seg(S, it_end - 1, it_end, 0);
    const Fp64Params& q = S.prob(sg.pid);
    const int64_t tb = S.begin(sg.pid) + (int64_t)sg.tile * q.iters_per_tile;
    const FixupSpan f = fixup_span(S, tb, tb + q.iters_per_tile);
    if (f.last - f.first + 1 >= kSharedParts)
      shared_fixup<TS, AKM>(S, q, f, cta, sg.tm, sg.tn, pubval, fixup_red);
  }
}

__global__ void __launch_bounds__(Tile128::kThreads, 1)
    fp64_streamk_kernel(const __grid_constant__ CUtensorMap mapA,
                        const __grid_constant__ CUtensorMap mapB,
                        const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile128>(S);
}

// One problem on 64 x 64 tiles, two CTAs per SM.
__global__ void __launch_bounds__(Tile64::kThreads, Tile64::kMinBlocks)
    fp64_streamk_kernel64(const __grid_constant__ CUtensorMap mapA,
                          const __grid_constant__ CUtensorMap mapB,
                          const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile64>(S);
}

// One problem on 32 x 32 tiles, four CTAs of four MMA warps per SM.
__global__ void __launch_bounds__(Tile32::kThreads, Tile32::kMinBlocks)
    fp64_streamk_kernel32(const __grid_constant__ CUtensorMap mapA,
                          const __grid_constant__ CUtensorMap mapB,
                          const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile32>(S);
}

// The same kernels on a K-major A (kOpBandK: the rotation reading
// band-packed Psi, the band -> grid transposition folded into the loads).
__global__ void __launch_bounds__(Tile128::kThreads, 1)
    fp64_streamk_kernel_ak(const __grid_constant__ CUtensorMap mapA,
                           const __grid_constant__ CUtensorMap mapB,
                           const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile128, true>(S);
}

__global__ void __launch_bounds__(Tile64::kThreads, Tile64::kMinBlocks)
    fp64_streamk_kernel64_ak(const __grid_constant__ CUtensorMap mapA,
                             const __grid_constant__ CUtensorMap mapB,
                             const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile64, true>(S);
}

__global__ void __launch_bounds__(Tile32::kThreads, Tile32::kMinBlocks)
    fp64_streamk_kernel32_ak(const __grid_constant__ CUtensorMap mapA,
                             const __grid_constant__ CUtensorMap mapB,
                             const __grid_constant__ Fp64Params p) {
  const SingleSched S{p, &mapA, &mapB};
  streamk_body<Tile32, true>(S);
}

// SPREAD: with the shared fix-up (tiles of kSharedParts parts or more in the group).
template <class TS, bool SPREAD>
__global__ void __launch_bounds__(TS::kThreads, TS::kMinBlocks)
    fp64_grouped_kernel(const __grid_constant__ Fp64Group g) {
  const GroupSched<SPREAD> S{g};
  streamk_body<TS>(S);
}

}  // namespace skg
