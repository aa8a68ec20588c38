// The nonlocal part of H on device: Hamiltonian::nloc_project_vectors_packed
// (16-band-packed Psi -> 32-band-packed H Psi) and _16to16
// (include/nloc_packed_opt2.hpp:226-445). Per projector p (grid rows
// index_p, coefficients chi_p column-major nrow x ncol, coefficient block at
// offsets[p], shared by the projectors of one atom's periodic images):
//   C_p[j, b] = C_p + dv * sum_r chi_p[r, j] psi[index_p[r], b]  (gather + chi^T psi)
//   C_p *= gamma_p per column, on every change of atom index in projector order
//   out[index_p[r], b] += sum_j chi_p[r, j] C_p[j, b]             (chi C + scatter)
// The single-rank all-reduce of the coefficients is the identity here.
//
// Three kernels, no atomics, the reference's loop and rounding order (as its
// C++ compiles: the forward dot products unfused, the block update fused, the
// back-projection sums fused), so results equal it bit for bit:
//  * nloc_forward_kernel: CTA per (block, 32 bands, 16 columns) — for each of
//    the block's projectors in order, gathered psi rows staged in shared
//    memory (asynchronous copies, chunks ahead), each thread summing its (column,
//    band) products in row order; then the block's gamma scalings in order;
//  * nloc_chi_c_kernel: the back-projection rows chi_p C_p of every projector
//    (spans of 64-row tiles x 64 bands, C in registers, chi in shared memory),
//    into a scratch of total rows x nb;
//  * nloc_backward_kernel: thread per (touched grid point, band pair) — walks
//    the point's (projector, row) entries in projector order (an inverse index
//    built at creation, each entry stored as its scratch row), so the
//    scatter-adds keep the reference's order.
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "skg_common.cuh"
#include "skg_runtime.h"

struct skgemm_nloc {
  int device = 0;
  int64_t P = 0, K = 0, nblk = 0, ntouch = 0, total_cols = 0;
  // device arrays
  uint32_t *d_nrow = nullptr, *d_ncol = nullptr, *d_index = nullptr;
  int64_t *d_row_off = nullptr, *d_chi_off = nullptr;
  double *d_chi = nullptr, *d_gamma = nullptr;
  // blocks: column base, width, projectors (CSR), gamma scalings (CSR)
  int64_t* d_blk = nullptr;  // [nblk][4]: col base, ncol, proj begin, scale begin
  int64_t* d_blk_end = nullptr;  // [nblk][2]: proj end, scale end
  int32_t* d_blk_proj = nullptr;
  int64_t* d_blk_scale = nullptr;  // gamma offsets
  int64_t* d_proj_blk_col = nullptr;  // per projector: its block's column base
  // touched points: grid index, entries (CSR of (projector, row))
  uint32_t* d_touch = nullptr;
  int64_t* d_touch_off = nullptr;
  int64_t* d_ent_off = nullptr;  // per entry: its temp row (projector's row_off + row)
  // back-projection row tiles (projector, first row)
  int64_t ntiles = 0;
  int64_t *d_tile_proj = nullptr, *d_tile_r0 = nullptr;
  int64_t total_rows = 0;
  // scratch: the coefficient blocks ([column][band], total_cols x nb), then
  // the back-projection rows (total_rows x nb)
  double* d_coef = nullptr;
  int64_t coef_cap = 0;
  std::vector<int64_t> blk_width;  // host copy of each block's ncol
  std::mutex mu;
};

namespace skg {

namespace {

// chi on the device: each projector's columns in groups of kNlocCols, a group
// row-major [nrow][group_pitch], a chunk of rows then contiguous, for whole 16-byte
// copies. An odd last column has a zero one beside it.
__host__ __device__ inline int group_pitch(int ncol, int k0) {  // the group from column k0
  const int w = ncol - k0;
  return w < 16 ? (w + 1) & ~1 : 16;
}

// Forward CTA: (block q, 32 bands, 16 columns); thread (bands bl, bl + 1, columns
// jl, jl + 1). The CTA walks the block's projectors in order and each projector's
// rows in chunks of kNlocRows: a chunk's gathered rows x 32 bands of psi and its
// rows x 16 columns of chi land in shared memory by asynchronous copies,
// kNlocRing - 1 chunks ahead, the gathered row numbers one chunk before that (24
// KB a CTA: all CTAs of 64 atoms x 512 bands are resident at once). Every thread
// adds its products over a chunk's rows in row order — the reference's order, so
// the sums are exact to it — and folds each projector's sum into the block
// coefficient with fma(dv, sum, C). Coefficients stored [column][band].
// Bound by the latency of gathers and the adds' order (a projector's rows are one
// chain per output) at small sizes, by the shared-memory pipe (90%) at large ones:
// two bands x four columns in 64 threads took 89 us at 512 bands but 5-20% longer
// where few CTAs run; one band x four columns took the same 98 us. Before: 32-row
// chunks, one ahead, their row numbers loaded just before the copies, chi copied 8
// bytes at a time from its columns, five 8-byte shared loads for four sums.
// 64 balls of ~800 points x 16 columns x 512 bands 137 -> 99 us, 37 bands 105 -> 46
// us; 20 balls of ~380 points x 9 columns x 100 bands 50 -> 25 us.
constexpr int kNlocBands = 32;
constexpr int kNlocCols = 16;
constexpr int kNlocRows = 16;
constexpr int kNlocRing = 4;
constexpr int kNlocThreads = kNlocBands * kNlocCols / 4;
static_assert(kNlocCols == 16, "group_pitch");
static_assert(kNlocRows * kNlocCols == 2 * kNlocThreads, "one 16-byte piece of chi a thread");
static_assert(kNlocRows * kNlocBands == 4 * kNlocThreads, "two 16-byte pieces of psi a thread");

__global__ void __launch_bounds__(kNlocThreads) nloc_forward_kernel(
    int64_t nb, int64_t K, double dv, const int64_t* __restrict__ blk,
    const int64_t* __restrict__ blk_end, const int32_t* __restrict__ blk_proj,
    const int64_t* __restrict__ blk_scale, const uint32_t* __restrict__ nrow,
    const int64_t* __restrict__ row_off, const int64_t* __restrict__ chi_off,
    const uint32_t* __restrict__ index, const double* __restrict__ chi,
    const double* __restrict__ gamma, const double* __restrict__ psi16,
    double* __restrict__ coef) {
  __shared__ __align__(16) double rows[kNlocRing][kNlocRows][kNlocBands];
  __shared__ __align__(16) double xs[kNlocRing][kNlocRows][kNlocCols];
  const int64_t q = blockIdx.x;
  const int64_t b0 = (int64_t)blockIdx.y * kNlocBands;
  const int64_t jb = (int64_t)blockIdx.z * kNlocCols;  // the CTA's first column
  const int bl = 2 * (threadIdx.x % (kNlocBands / 2));
  const int jl = 2 * (threadIdx.x / (kNlocBands / 2));
  const int64_t col0 = blk[4 * q], nc = blk[4 * q + 1];
  if (jb >= nc) return;  // the whole CTA past the block
  const int64_t e_begin = blk[4 * q + 2], e_end = blk_end[2 * q];
  const int64_t b = b0 + bl;
  // This thread's copies: bands bl, bl + 1 of rows cr and cr + kNlocRows / 2, and
  // 16 bytes of chi.
  const int cr = threadIdx.x / (kNlocBands / 2);
  const int pitch = group_pitch((int)nc, (int)jb);
  const int xr = threadIdx.x / (kNlocCols / 2), xc = 2 * (threadIdx.x % (kNlocCols / 2));
  const bool band_ok = b < nb;
  const double* pb = psi16 + (band_ok ? (b / 16) * K * 16 + b % 16 : 0);

  // Issuing cursor: a projector entry, its rows and the chunk's first row; the
  // chunk's row numbers for this thread's copies.
  int64_t ie = e_begin, ib = 0;
  int ir0 = 0, inr = 0;
  const double* ix = chi;
  uint32_t n0 = 0, n1 = 0;
  auto enter = [&]() {  // entry ie
    if (ie < e_end) {
      const int p = blk_proj[ie];
      inr = (int)nrow[p];
      ib = row_off[p];
      ix = chi + chi_off[p] + jb * inr;
    }
  };
  auto numbers = [&]() {
    if (ie < e_end) {
      const uint32_t* idx = index + ib + ir0 + cr;
      if (ir0 + cr < inr) n0 = __ldg(idx);
      if (ir0 + cr + kNlocRows / 2 < inr) n1 = __ldg(idx + kNlocRows / 2);
    }
  };
  auto issue = [&](int buf) {
    if (ie < e_end) {
      const int left = inr - ir0;
      if (band_ok && cr < left) cp_async16(&rows[buf][cr][bl], pb + (int64_t)n0 * 16, 16u);
      if (band_ok && cr + kNlocRows / 2 < left)
        cp_async16(&rows[buf][cr + kNlocRows / 2][bl], pb + (int64_t)n1 * 16, 16u);
      if (xr < left && xc < pitch)
        cp_async16(&xs[buf][xr][xc], ix + (int64_t)(ir0 + xr) * pitch + xc, 16u);
      ir0 += kNlocRows;
      if (ir0 >= inr) {
        ++ie;
        ir0 = 0;
        enter();
      }
    }
    cp_async_commit();
  };
  enter();
  for (int s = 0; s < kNlocRing - 1; ++s) {
    numbers();
    issue(s);
  }
  numbers();

  double acc[4] = {};
  double sum[4] = {};
  int buf = 0;
  for (int64_t e = e_begin; e < e_end; ++e) {
    const int nr = (int)nrow[blk_proj[e]];
    for (int r0 = 0; r0 < nr; r0 += kNlocRows) {
      cp_async_wait<kNlocRing - 2>();
      __syncthreads();  // the chunk has landed; the one before it is consumed
      issue((buf + kNlocRing - 1) % kNlocRing);
      numbers();
      const double* rb = &rows[buf][0][bl];
      const double* xb = &xs[buf][0][jl];
      auto row = [&](int rr) {
        const double2 v = *reinterpret_cast<const double2*>(rb + rr * kNlocBands);
        const double2 x = *reinterpret_cast<const double2*>(xb + rr * kNlocCols);
        sum[0] = __dadd_rn(sum[0], __dmul_rn(x.x, v.x));
        sum[1] = __dadd_rn(sum[1], __dmul_rn(x.x, v.y));
        sum[2] = __dadd_rn(sum[2], __dmul_rn(x.y, v.x));
        sum[3] = __dadd_rn(sum[3], __dmul_rn(x.y, v.y));
      };
      if (nr - r0 >= kNlocRows) {
#pragma unroll
        for (int rr = 0; rr < kNlocRows; ++rr) row(rr);
      } else {
        for (int rr = 0; rr < nr - r0; ++rr) row(rr);
      }
      buf = (buf + 1) % kNlocRing;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // projector e into the block
      acc[i] = fma(dv, sum[i], acc[i]);
      sum[i] = 0.0;
    }
  }
  if (b >= nb) return;
#pragma unroll
  for (int jj = 0; jj < 2; ++jj) {
    const int64_t j = jb + jl + jj;
    if (j >= nc) break;
    double a0 = acc[2 * jj], a1 = acc[2 * jj + 1];
    for (int64_t f = blk[4 * q + 3]; f < blk_end[2 * q + 1]; ++f) {
      const double gm = __ldg(gamma + blk_scale[f] + j);
      a0 = __dmul_rn(a0, gm);
      a1 = __dmul_rn(a1, gm);
    }
    coef[(col0 + j) * nb + b] = a0;
    if (b + 1 < nb) coef[(col0 + j) * nb + b + 1] = a1;
  }
}

// Back-projection, step 1: temp_p[r, b] = sum_k chi_p[r, k] C_p[k, b] (fused,
// k ascending: the reference's gemm_ab order) for every projector row, into
// temp[(row_off_p + r) * nb + b]. CTA = (a span of up to kNlocSpan row tiles
// of 64 rows of one projector, 64 bands); thread = a band pair and every
// kNlocWarps-th group of 4 rows. A column group's C stays in registers, its chi rows
// are copied to shared memory ahead of their use and read as broadcasts. Further
// column groups continue from the stored sums, so the order is the same for any
// number of columns.
// Was: C and chi staged in shared memory behind one barrier, a row tile at a time.
// 64 balls of ~800 points x 16 columns x 512 bands 90 -> 65 us (writing temp alone
// takes 32 us), 37 bands 25 -> 17 us. Spans of 4 tiles: 64 and 21 us. A second and
// third column group cost a pass over temp each: 40 columns 57 -> 65 us, with the
// forward kernel 168 -> 148 us.
constexpr int kNlocTileR = 64;
constexpr int kNlocTileB = 64;
constexpr int kNlocMaxCols = 64;
constexpr int kNlocSpan = 2;
constexpr int kNlocWarps = 4;
static_assert(kNlocSpan == 2, "the waits of nloc_chi_c_kernel");

__global__ void __launch_bounds__(kNlocWarps * 32) nloc_chi_c_kernel(
    int64_t nb, const int64_t* __restrict__ tile_proj, const int64_t* __restrict__ tile_r0,
    const uint32_t* __restrict__ nrow, const uint32_t* __restrict__ ncol,
    const int64_t* __restrict__ row_off, const int64_t* __restrict__ chi_off,
    const int64_t* __restrict__ proj_col, const double* __restrict__ chi,
    const double* __restrict__ coef, double* __restrict__ temp) {
  __shared__ __align__(16) double xs[kNlocSpan][kNlocTileR][kNlocCols];
  const int64_t tile = blockIdx.x;
  const int p = (int)tile_proj[tile];
  const int64_t span0 = tile_r0[tile];
  const int nr = (int)min((int64_t)nrow[p] - span0, (int64_t)kNlocSpan * kNlocTileR);
  const int nc = (int)ncol[p];
  const int64_t b = (int64_t)blockIdx.y * kNlocTileB + 2 * (threadIdx.x % 32);
  const int warp = threadIdx.x / 32;
  const bool one = b < nb, two = b + 1 < nb;
  // 16-byte accesses where every row of temp starts on 16 bytes.
  const bool wide = two && nb % 2 == 0 && (reinterpret_cast<uintptr_t>(temp) & 15) == 0;
  double* out = temp + (row_off[p] + span0) * nb + b;
  for (int k0 = 0; k0 < nc; k0 += kNlocCols) {
    if (k0 > 0) __syncthreads();  // the group before is consumed
    const int pitch = group_pitch(nc, k0);
    const double* x = chi + chi_off[p] + (int64_t)k0 * nrow[p] + span0 * pitch;
#pragma unroll
    for (int t = 0; t < kNlocSpan; ++t) {
#pragma unroll
      for (int i = 0; i < kNlocTileR * kNlocCols / 2; i += kNlocWarps * 32) {
        const int o = t * kNlocTileR * kNlocCols + 2 * (i + (int)threadIdx.x);
        const int r = o / kNlocCols, c = o % kNlocCols;
        if (r < nr && c < pitch) cp_async16(&xs[0][0][0] + o, x + r * pitch + c, 16u);
      }
      cp_async_commit();
    }
    const int ncg = min(kNlocCols, nc - k0);
    const double* c = coef + (proj_col[p] + k0) * nb + b;
    double c0[kNlocCols], c1[kNlocCols];
#pragma unroll
    for (int k = 0; k < kNlocCols; ++k) {
      c0[k] = k < ncg && one ? c[k * nb] : 0.0;
      c1[k] = k < ncg && two ? c[k * nb + 1] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < kNlocSpan; ++t) {
      if (t * kNlocTileR >= nr) break;
      if (t == 0)
        cp_async_wait<kNlocSpan - 1>();
      else
        cp_async_wait<0>();
      __syncthreads();
      for (int r0 = 4 * warp; r0 < kNlocTileR; r0 += 4 * kNlocWarps) {
        const int r = t * kNlocTileR + r0;
        if (r >= nr || !one) break;
        double t0[4] = {}, t1[4] = {};
        if (k0 > 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (r + i < nr) {
              t0[i] = out[(r + i) * nb];
              if (two) t1[i] = out[(r + i) * nb + 1];
            }
        }
#pragma unroll
        for (int k = 0; k < kNlocCols; k += 2) {
          if (k >= ncg) break;
          double2 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            v[i] = *reinterpret_cast<const double2*>(&xs[t][r0 + i][k]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            t0[i] = fma(v[i].x, c0[k], t0[i]);
            t1[i] = fma(v[i].x, c1[k], t1[i]);
          }
          if (k + 1 < ncg) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              t0[i] = fma(v[i].y, c0[k + 1], t0[i]);
              t1[i] = fma(v[i].y, c1[k + 1], t1[i]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (r + i >= nr) break;
          double* o = out + (int64_t)(r + i) * nb;
          if (wide) {
            *reinterpret_cast<double2*>(o) = make_double2(t0[i], t1[i]);
          } else {
            o[0] = t0[i];
            if (two) o[1] = t1[i];
          }
        }
      }
    }
    cp_async_wait<0>();
  }
}

// Back-projection, step 2: thread per (touched grid point, band pair): the
// point's (projector, row) entries added to out in projector order.
template <int OT>
__global__ void __launch_bounds__(256) nloc_backward_kernel(
    int64_t ntouch, int64_t nb, int64_t K, const uint32_t* __restrict__ touch,
    const int64_t* __restrict__ touch_off, const int64_t* __restrict__ ent_off,
    const double* __restrict__ temp, double* __restrict__ out) {
  const int64_t nbp = (nb + 1) / 2;  // band pairs
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntouch * nbp) return;
  const int64_t b = 2 * (t % nbp), s = t / nbp;
  const bool two = b + 1 < nb;
  const int64_t g = touch[s];
  double* o = out + ((b / OT) * K + g) * OT + (b % OT);  // b + 1 in the same tile (OT even)
  double v0 = o[0], v1 = two ? o[1] : 0.0;
  for (int64_t e = touch_off[s]; e < touch_off[s + 1]; ++e) {
    const double* tr = temp + __ldg(ent_off + e) * nb + b;
    v0 = __dadd_rn(v0, __ldg(tr));
    if (two) v1 = __dadd_rn(v1, __ldg(tr + 1));
  }
  o[0] = v0;
  if (two) o[1] = v1;
}

// Allocates *dst for v and adds its upload to `copies`.
template <typename T>
int stage(T** dst, const std::vector<T>& v, std::vector<TableCopy>& copies) {
  if (v.empty()) return SKGEMM_OK;
  SKG_CUDA(cudaMalloc(dst, v.size() * sizeof(T)));
  copies.push_back({*dst, v.data(), v.size() * sizeof(T)});
  return SKGEMM_OK;
}

// Uploads `copies` and chi (projector p's columns one after the other from in_off[p])
// into d_chi (total doubles) in the kernels' layout, row by row: the reads are as many
// streams as the group has columns, the writes one.
int upload_chi(skgemm_nloc* h, const double* chi, const uint32_t* nrow, const uint32_t* ncol,
               const std::vector<int64_t>& in_off, int64_t total, std::vector<TableCopy>& copies) {
  std::unique_ptr<double[]> buf(new double[total]);
  double* out = buf.get();
  for (int64_t p = 0; p < (int64_t)in_off.size(); ++p) {
    const int64_t nr = nrow[p];
    const int nc = (int)ncol[p];
    for (int k0 = 0; k0 < nc; k0 += kNlocCols) {
      const int w = std::min(kNlocCols, nc - k0), pitch = group_pitch(nc, k0);
      const double* in = chi + in_off[p] + k0 * nr;
      for (int64_t r = 0; r < nr; ++r, out += pitch) {
        for (int j = 0; j < w; ++j) out[j] = in[j * nr + r];
        if (w < pitch) out[w] = 0.0;
      }
    }
  }
  if (total > 0) {
    SKG_CUDA(cudaMalloc(&h->d_chi, (size_t)total * sizeof(double)));
    copies.push_back({h->d_chi, buf.get(), (size_t)total * sizeof(double)});
  }
  return upload_tables(copies);
}

// Sorts `rows` (ascending) by their index, rows of one index in their order: two stable
// passes over 16 bits. A map of lists took most of a creation's time.
void sort_by_index(const uint32_t* index, std::vector<int64_t>& rows) {
  std::vector<int64_t> other(rows.size());
  for (int shift = 0; shift < 32; shift += 16) {
    std::vector<int64_t> at(65537, 0);
    for (int64_t r : rows) ++at[((index[r] >> shift) & 0xFFFFu) + 1];
    for (int v = 0; v < 65536; ++v) at[v + 1] += at[v];
    for (int64_t r : rows) other[at[(index[r] >> shift) & 0xFFFFu]++] = r;
    rows.swap(other);
  }
}

void release(skgemm_nloc* h) {
  void* ptrs[] = {h->d_nrow, h->d_ncol, h->d_index, h->d_row_off, h->d_chi_off, h->d_chi,
                  h->d_gamma, h->d_blk, h->d_blk_end, h->d_blk_proj, h->d_blk_scale,
                  h->d_proj_blk_col, h->d_touch, h->d_touch_off, h->d_ent_off,
                  h->d_tile_proj, h->d_tile_r0, h->d_coef};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

}  // namespace

// Builds the device form of a projector set (see skgemm_nloc_create).
int nloc_create(int64_t P, const uint32_t* nrow, const uint32_t* ncol, const int32_t* atom,
                const uint32_t* offsets, const uint32_t* index, const double* chi,
                const double* gamma, int64_t K, skgemm_nloc** out) {
  if (!out) return fail(SKGEMM_ERR_INVALID_ARG, "null handle pointer");
  *out = nullptr;
  if (P < 0 || P > INT32_MAX || K <= 0 || K > ((int64_t)1 << 32))
    return fail(SKGEMM_ERR_INVALID_ARG, "projector count or grid size out of range");
  if (P > 0 && (!nrow || !ncol || !atom || !offsets))
    return fail(SKGEMM_ERR_INVALID_ARG, "null projector array");
  int st;
  DeviceState* dev = current_device(&st);
  if (!dev) return st;
  std::vector<int64_t> row_off(P), chi_off(P);
  int64_t rows = 0, chis = 0, gams = 0, chi_in = 0;
  std::vector<int64_t> gam_off(P), in_off(P);
  const int64_t total = P > 0 ? offsets[P] : 0;
  for (int64_t p = 0; p < P; ++p) {
    row_off[p] = rows;
    chi_off[p] = chis;
    gam_off[p] = gams;
    rows += nrow[p];
    in_off[p] = chi_in;
    chi_in += (int64_t)nrow[p] * ncol[p];
    chis += (int64_t)nrow[p] * ((ncol[p] + 1) / 2 * 2);  // all groups at their pitch
    gams += ncol[p];
    if ((int64_t)offsets[p] + ncol[p] > total)
      return fail(SKGEMM_ERR_INVALID_ARG, "projector block past the total column count");
    if (ncol[p] > kNlocMaxCols)
      return fail(SKGEMM_ERR_UNSUPPORTED, "projectors of more than 64 columns");
  }
  if (rows > 0 && !index) return fail(SKGEMM_ERR_INVALID_ARG, "null index array");
  if ((chi_in > 0 && !chi) || (gams > 0 && !gamma))
    return fail(SKGEMM_ERR_INVALID_ARG, "null coefficient array");
  for (int64_t i = 0; i < rows; ++i)
    if (index[i] >= (uint64_t)K) return fail(SKGEMM_ERR_INVALID_ARG, "grid index out of range");
  // Blocks by offset, in order of first use; projectors sharing one must
  // share its width, and distinct blocks must not overlap.
  std::map<uint32_t, int64_t> blk_of;
  std::vector<int64_t> bcol, bnc;
  std::vector<std::vector<int32_t>> bproj;
  std::vector<std::vector<int64_t>> bscale;
  std::vector<int64_t> proj_col(P);
  for (int64_t p = 0; p < P; ++p) {
    auto it = blk_of.find(offsets[p]);
    int64_t q;
    if (it == blk_of.end()) {
      q = (int64_t)bcol.size();
      blk_of[offsets[p]] = q;
      bcol.push_back(offsets[p]);
      bnc.push_back(ncol[p]);
      bproj.emplace_back();
      bscale.emplace_back();
    } else {
      q = it->second;
      if (bnc[q] != ncol[p])
        return fail(SKGEMM_ERR_INVALID_ARG, "projectors sharing a block differ in width");
    }
    proj_col[p] = offsets[p];
    if (nrow[p] > 0 && ncol[p] > 0) bproj[q].push_back((int32_t)p);
  }
  {
    int64_t end = 0;
    for (const auto& kv : blk_of) {
      const int64_t q = kv.second;
      if (bcol[q] < end) return fail(SKGEMM_ERR_INVALID_ARG, "projector blocks overlap");
      end = bcol[q] + bnc[q];
    }
  }
  if (P > 0) {  // gamma on each change of atom index, in projector order
    int32_t a = atom[0] - 1;
    for (int64_t p = 0; p < P; ++p) {
      if (a == atom[p]) continue;
      a = atom[p];
      bscale[blk_of[offsets[p]]].push_back(gam_off[p]);
    }
  }
  // Inverse index: grid point -> its rows (of all projectors, in projector order).
  std::vector<int64_t> ent_off;
  ent_off.reserve(rows);
  for (int64_t p = 0; p < P; ++p)
    for (int64_t r = 0; ncol[p] > 0 && r < nrow[p]; ++r) ent_off.push_back(row_off[p] + r);
  sort_by_index(index, ent_off);
  auto* h = new skgemm_nloc();
  h->device = dev->device;
  h->P = P;
  h->K = K;
  h->nblk = (int64_t)bcol.size();
  h->total_cols = total;
  h->blk_width = bnc;
  std::vector<int64_t> blk(4 * h->nblk), blk_end(2 * h->nblk);
  std::vector<int32_t> blk_proj;
  std::vector<int64_t> blk_scale;
  for (int64_t q = 0; q < h->nblk; ++q) {
    blk[4 * q] = bcol[q];
    blk[4 * q + 1] = bnc[q];
    blk[4 * q + 2] = (int64_t)blk_proj.size();
    blk[4 * q + 3] = (int64_t)blk_scale.size();
    blk_proj.insert(blk_proj.end(), bproj[q].begin(), bproj[q].end());
    blk_scale.insert(blk_scale.end(), bscale[q].begin(), bscale[q].end());
    blk_end[2 * q] = (int64_t)blk_proj.size();
    blk_end[2 * q + 1] = (int64_t)blk_scale.size();
  }
  std::vector<uint32_t> touch;
  std::vector<int64_t> touch_off;
  for (size_t e = 0; e < ent_off.size(); ++e)
    if (e == 0 || index[ent_off[e]] != touch.back()) {
      touch.push_back(index[ent_off[e]]);
      touch_off.push_back((int64_t)e);
    }
  touch_off.push_back((int64_t)ent_off.size());
  h->ntouch = (int64_t)touch.size();
  h->total_rows = rows;
  std::vector<int64_t> tile_proj, tile_r0;
  for (int64_t p = 0; p < P; ++p) {
    if (nrow[p] == 0 || ncol[p] == 0) continue;
    for (int64_t r0 = 0; r0 < nrow[p]; r0 += kNlocTileR * kNlocSpan) {
      tile_proj.push_back(p);
      tile_r0.push_back(r0);
    }
  }
  h->ntiles = (int64_t)tile_proj.size();
  std::vector<uint32_t> vnrow(nrow, nrow + P), vncol(ncol, ncol + P);
  std::vector<uint32_t> vindex(index, index + rows);
  std::vector<double> vgam(gamma, gamma + gams);
  std::vector<TableCopy> up;
  if ((st = stage(&h->d_nrow, vnrow, up)) ||
      (st = stage(&h->d_ncol, vncol, up)) ||
      (st = stage(&h->d_index, vindex, up)) ||
      (st = stage(&h->d_row_off, row_off, up)) ||
      (st = stage(&h->d_chi_off, chi_off, up)) ||
      (st = stage(&h->d_gamma, vgam, up)) ||
      (st = stage(&h->d_blk, blk, up)) ||
      (st = stage(&h->d_blk_end, blk_end, up)) ||
      (st = stage(&h->d_blk_proj, blk_proj, up)) ||
      (st = stage(&h->d_blk_scale, blk_scale, up)) ||
      (st = stage(&h->d_proj_blk_col, proj_col, up)) ||
      (st = stage(&h->d_touch, touch, up)) ||
      (st = stage(&h->d_touch_off, touch_off, up)) ||
      (st = stage(&h->d_ent_off, ent_off, up)) ||
      (st = stage(&h->d_tile_proj, tile_proj, up)) ||
      (st = stage(&h->d_tile_r0, tile_r0, up)) ||
      (st = upload_chi(h, chi, nrow, ncol, in_off, chis, up))) {
    release(h);
    delete h;
    return st;
  }
  *out = h;
  return SKGEMM_OK;
}

int nloc_apply(skgemm_nloc* h, int64_t nb, double dv, const double* psi16, double* out,
               int out_tile, cudaStream_t s) {
  if (!h) return fail(SKGEMM_ERR_INVALID_ARG, "null projector handle");
  if (nb < 0) return fail(SKGEMM_ERR_INVALID_ARG, "negative band count");
  if (out_tile != 16 && out_tile != 32) return fail(SKGEMM_ERR_INVALID_ARG, "out_tile must be 16 or 32");
  if (nb == 0 || h->nblk == 0 || h->total_cols == 0) return SKGEMM_OK;
  if (!psi16 || !out) return fail(SKGEMM_ERR_INVALID_ARG, "null pointer");
  int st;
  DeviceState* dev = current_device(&st);
  if (!dev) return st;
  if (dev->device != h->device) return fail(SKGEMM_ERR_INVALID_ARG, "handle of another device");
  std::lock_guard<std::mutex> lk(h->mu);
  // Scratch: coefficients (total columns x nb), then back-projection rows
  // (total rows x nb); grown on demand.
  const int64_t need = (h->total_cols + h->total_rows) * nb;
  if (need > h->coef_cap) {
    if (h->d_coef) {
      SKG_CUDA(cudaStreamSynchronize(s));
      cudaFree(h->d_coef);
      h->d_coef = nullptr;
      h->coef_cap = 0;
    }
    SKG_CUDA(cudaMalloc(&h->d_coef, need * sizeof(double)));
    h->coef_cap = need;
  }
  // Debug mode: the coefficient and scratch rows start as 0xFF bytes.
  if ((st = debug_poison(h->d_coef, (size_t)h->coef_cap * sizeof(double), s))) return st;
  const int64_t maxw = *std::max_element(h->blk_width.begin(), h->blk_width.end());
  if (maxw > 0) {
    dim3 grid((unsigned)h->nblk, (unsigned)((nb + kNlocBands - 1) / kNlocBands),
              (unsigned)((maxw + kNlocCols - 1) / kNlocCols));
    if (grid.y > 65535u || grid.z > 65535u)
      return fail(SKGEMM_ERR_INVALID_ARG, "too many bands or projector columns");
    KernelTimer kt_(s, "nloc_forward_kernel");
    nloc_forward_kernel<<<grid, kNlocThreads, 0, s>>>(
        nb, h->K, dv, h->d_blk, h->d_blk_end, h->d_blk_proj, h->d_blk_scale, h->d_nrow,
        h->d_row_off, h->d_chi_off, h->d_index, h->d_chi, h->d_gamma, psi16, h->d_coef);
    SKG_CUDA(cudaGetLastError());
  }
  double* temp = h->d_coef + h->total_cols * nb;
  if (h->ntiles > 0) {
    dim3 grid((unsigned)h->ntiles, (unsigned)((nb + kNlocTileB - 1) / kNlocTileB));
    if (h->ntiles > INT32_MAX || grid.y > 65535u)
      return fail(SKGEMM_ERR_INVALID_ARG, "too many projector rows or bands");
    KernelTimer kt_(s, "nloc_chi_c_kernel");
    nloc_chi_c_kernel<<<grid, kNlocWarps * 32, 0, s>>>(
        nb, h->d_tile_proj, h->d_tile_r0, h->d_nrow, h->d_ncol, h->d_row_off, h->d_chi_off,
        h->d_proj_blk_col, h->d_chi, h->d_coef, temp);
    SKG_CUDA(cudaGetLastError());
  }
  const int64_t nbk = h->ntouch * ((nb + 1) / 2);  // threads: (touched point, band pair)
  if (nbk > 0) {
    if ((nbk + 255) / 256 > INT32_MAX)
      return fail(SKGEMM_ERR_INVALID_ARG, "too many touched points x bands");
    KernelTimer kt_(s, "nloc_backward_kernel");
    if (out_tile == 32)
      nloc_backward_kernel<32><<<(unsigned)((nbk + 255) / 256), 256, 0, s>>>(
          h->ntouch, nb, h->K, h->d_touch, h->d_touch_off, h->d_ent_off, temp, out);
    else
      nloc_backward_kernel<16><<<(unsigned)((nbk + 255) / 256), 256, 0, s>>>(
          h->ntouch, nb, h->K, h->d_touch, h->d_touch_off, h->d_ent_off, temp, out);
    SKG_CUDA(cudaGetLastError());
  }
  return SKGEMM_OK;
}

void nloc_destroy(skgemm_nloc* h) {
  if (!h) return;
  release(h);
  delete h;
}

}  // namespace skg
