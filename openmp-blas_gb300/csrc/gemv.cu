// gemv.cu - matrix x vector kernels behind amt::mtv and amt::vtm.
//
// Two access shapes cover both layouts and both products:
//
//   gemv_rows  every output is the dot of one CONTIGUOUS row with x:
//              y[r] (+)= sum_c A[r*lda + c] * x[c].
//              mtv with row-major A (reference include/mtv.hpp:72-98,
//              simd_loop.hpp:21-35, overwrites y) and vtm with column-major
//              A (columns of A are the contiguous rows of A^T).
//   gemv_cols  the axpy form over CONTIGUOUS columns:
//              y[r] (+)= sum_c A[r + c*lda] * x[c].
//              mtv with column-major A (reference include/mtv.hpp:15-70,
//              simd_loop.hpp:52-78, accumulates into y) and vtm with
//              row-major A.
//
// Both stream A from HBM once, with 128-bit read-only loads (columns off the
// 16-byte grid: of single elements, except for large float matrices), and keep x
// in L1 / shared memory.  When the grid would be too
// small to fill the 152 SMs the reduction dimension is split across CTAs.
// Up to 8 splits of a small matrix run as one thread-block cluster per row
// block: each CTA leaves its partials in its shared memory and the
// cluster's rank 0 adds them in split order through distributed shared
// memory.  Otherwise the partials go to per-stream scratch and a second small
// kernel, chained to the first, adds them.  Either way the order of additions
// is fixed by the shape and the alignment (no atomics).
// Roofline: HBM, (rows*cols + rows + cols) * sizeof(T) bytes per call; for
// double the FP64 pipes (2 multiply-adds per clock and SM: 4.6 TB/s of A),
// so that sums over threads are kept few.  us per call, cold, before (scalar
// loads at odd leading dimensions, a CTA per four rows, a thread per row of a
// column) and now: rows f32 16384^2 153.9 -> 148, 8191 x 6001 48.3 -> 35.4,
// 25596 x 256 16.4 -> 8.5; f64 18652 x 947 86 -> 45, 25596 x 256 82 -> 20;
// columns f32 16384^2 156.4 -> 154, 10001 x 10003 166 -> 69, 256 x 25596 36 -> 11;
// f64 8191 x 6001 95 -> 92, 10001 x 10003 205 -> 177, 512 x 6552 33 -> 15.
#include <algorithm>
#include <type_traits>
#include <utility>

#include "common.cuh"

namespace gbblas {
namespace {

template <typename T>
struct V;
template <>
struct V<float> {
  using t = float4;
  static constexpr int w = 4;
};
template <>
struct V<double> {
  using t = double2;
  static constexpr int w = 2;
};

__device__ __forceinline__ float vdot(float4 a, float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc);
  acc = fmaf(a.y, b.y, acc);
  acc = fmaf(a.z, b.z, acc);
  return fmaf(a.w, b.w, acc);
}
__device__ __forceinline__ double vdot(double2 a, double2 b, double acc) {
  acc = fma(a.x, b.x, acc);
  return fma(a.y, b.y, acc);
}
__device__ __forceinline__ float4 ldg_vec(const float4* p) { return __ldg(p); }
__device__ __forceinline__ double2 ldg_vec(const double2* p) { return __ldg(p); }

constexpr int kRowsThreads = 256;
constexpr int kWarps = kRowsThreads / 32;

constexpr int kMaxClusterSplits = 8;  // portable cluster size

// Whether the ksplit CTAs of a row block reduce as one cluster: on a small
// matrix, where a second launch is a good part of the call (512 x 512
// column-major: f32 4.1 us, 5.2 through scratch; f64 6.2 and 7.3).  On larger
// ones the CTAs of a cluster waiting for one another cost more than the
// chained finish (20069 x 264 f64: 20.4 us in clusters, 17.7 through scratch;
// 256 x 25596 f32 12.3 and 10.7).
inline bool cluster_splits(int64_t ksplit, int64_t rows, int64_t cols, size_t elem) {
  return ksplit >= 2 && ksplit <= kMaxClusterSplits && (double)rows * cols * elem <= 8.0e6;
}

// The sums of a warp's R values per lane: lane 32 / R * j ends up with the
// total of value j.  The halves of the warp first trade values, so R = 4 takes
// 6 additions where a butterfly per value takes 20 (the same pairs are added,
// so the same bits) - on the FP64 pipes 96 cycles against 320.
template <typename T>
__device__ __forceinline__ T warp_totals(const T (&v)[1], int) {
  return dev::warp_sum(v[0]);
}
template <typename T>
__device__ __forceinline__ T warp_totals(const T (&v)[4], int lane) {
  const bool h = lane & 16, q = lane & 8;
  T a = (h ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
  T b = (h ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
  T t = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Row-streaming form.  A CTA's 8 warps are 8 / wc row groups of wc warps; a
// group computes R rows, its warps sharing the columns out 32 vectors at a
// time.  The R rows of a group lie `period` apart, the distance at which every
// row starts at the same offset from a 16-byte boundary: the group's `head`
// elements up to it and its last few are added one by one, everything between
// by 128-bit loads, and x is read once for all R rows (by vectors where it
// shares their alignment).  grid = (groups / groups per CTA, ksplit); split p
// covers vectors p * vps .. + vps - 1.  The last vectors of a row, fewer than U
// a lane, are loaded together too: one after another they cost a round trip to
// memory each (f32 4096 x 512, four vectors a row and lane: 5.8 us, 4.3 so).
// AL: every row and x start on 16-byte boundaries; CTAS: resident CTAs an SM.
// CL: the ksplit CTAs of a row block form a cluster (1, ksplit, 1).
template <typename T, int R, bool AL, bool CL, int CTAS>
__global__ void __launch_bounds__(kRowsThreads, CTAS)
    gemv_rows_kernel(int64_t rows, int64_t cols, const T* __restrict__ A, int64_t lda, const T* __restrict__ x,
                     T* __restrict__ y, bool accumulate, T* __restrict__ partials, int64_t vps, int lp, int lwc) {
  const int lperiod = AL ? 0 : lp;
  using VT = typename V<T>::t;
  constexpr int W = V<T>::w;
  constexpr int U = R == 4 ? 2 : 4;  // vectors per row and lane in flight
  __shared__ T red[kWarps][R];
  __shared__ T split_part[kWarps * R];  // CL: this split's row sums, read by the cluster's rank 0
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int period = 1 << lperiod, wc = 1 << lwc;  // powers of two: no division on the way to the first load
  const int wr = warp >> lwc, wi = warp & (wc - 1);
  const int groups = kWarps >> lwc;  // of this CTA
  // first row of a group (its others follow `period` apart)
  auto first_row = [&](int w) {
    const int64_t g = (int64_t)blockIdx.x * groups + w;
    return ((g >> lperiod) * R << lperiod) + (g & (period - 1));
  };
  const int64_t r0 = first_row(wr);
  const int nr = r0 < rows ? (int)min((rows - r0 + period - 1) >> lperiod, (int64_t)R) : 0;
  const T* __restrict__ row = A + (nr > 0 ? r0 : 0) * lda;
  const int64_t rstep = lda << lperiod;
  int64_t head = AL ? 0 : (int64_t)(((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) / sizeof(T));
  if (head > cols) head = cols;
  const int64_t nv = (cols - head) / W;
  const int64_t v1 = min(((int64_t)blockIdx.y + 1) * vps, nv);
  const T* __restrict__ xb = x + head;
  const bool xvec = AL || (reinterpret_cast<uintptr_t>(xb) & 15) == 0;
  // the elements before the first vector and after the last (R = 1, whose
  // calls are short: loaded ahead of the rest)
  T ex = T(0), ea[R];
  int64_t edge = -1;
  auto load_edge = [&]() {
    if (blockIdx.y == 0 && wi == 0) {
      const int64_t tail = cols - head - nv * W;
      edge = lane < head ? lane : (lane >= 8 && lane - 8 < tail ? head + nv * W + lane - 8 : -1);
      if (edge >= 0) {
        ex = __ldg(x + edge);
#pragma unroll
        for (int j = 0; j < R; ++j)
          if (j < nr) ea[j] = dev::ld_stream(row + j * rstep + edge);
      }
    }
  };
  if (R == 1) load_edge();

  T acc[R];
#pragma unroll
  for (int j = 0; j < R; ++j) acc[j] = T(0);
  const int step = 32 * wc;
  const int64_t v = (int64_t)blockIdx.y * vps + wi * 32 + lane;
  const VT* q = reinterpret_cast<const VT*>(row + head) + v;  // this lane's next vector of the first row
  const T* xq = xb + v * W;                                    // and of x
  const int64_t rv = rstep / W;                                // the next row's vectors lie this far on
  int left = (int)(v1 - v) + lane;                             // of the warp's range (32 vectors every `step`), from lane 0 on
  auto xload = [&](int u) {
    VT r;
    if (xvec) {
      r = ldg_vec(reinterpret_cast<const VT*>(xq) + u * step);
    } else {
      T* e = reinterpret_cast<T*>(&r);
#pragma unroll
      for (int i = 0; i < W; ++i) e[i] = __ldg(xq + u * step * W + i);
    }
    return r;
  };
  if (nr == R) {
    for (; left > (U - 1) * step + 31; left -= U * step, q += U * step, xq += U * step * W) {
      VT a[U][R], xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < R; ++j) a[u][j] = dev::ld_stream(q + j * rv + u * step);
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = xload(u);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[j] = vdot(a[u][j], xv[u], acc[j]);
    }
  }
  // what is left (of all rows, where they are fewer than R): under predicates,
  // with its loads in flight together
  for (; left > 0; left -= U * step, q += U * step, xq += U * step * W) {
    VT a[U][R], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (j < nr && left - lane > u * step) a[u][j] = dev::ld_stream(q + j * rv + u * step);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (left - lane > u * step) xv[u] = xload(u);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (left <= u * step) break;  // (the whole warp: no FP64 work on absent vectors)
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (j < nr && left - lane > u * step) acc[j] = vdot(a[u][j], xv[u], acc[j]);
    }
  }
  if (R > 1) load_edge();
  if (edge >= 0) {
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j < nr) acc[j] = fma(ea[j], ex, acc[j]);
  }
  dev::grid_release();  // a chained finish_splits_kernel may be set up

  const T t = warp_totals(acc, lane);
  if (lane % (32 / R) == 0) red[warp][lane / (32 / R)] = t;
  __syncthreads();
  const int fw = (int)threadIdx.x / R, fj = (int)threadIdx.x % R;  // this thread's group and row of it
  const int64_t r = fw < groups ? first_row(fw) + (int64_t)fj * period : rows;
  T sum = T(0);
  if (r < rows) {
    for (int w = 0; w < wc; ++w) sum += red[fw * wc + w][fj];
    if (CL)
      split_part[threadIdx.x] = sum;
    else if (gridDim.y == 1)
      y[r] = accumulate ? y[r] + sum : sum;
    else
      partials[(int64_t)blockIdx.y * rows + r] = sum;
  }
  if constexpr (CL) {
    dev::cluster_sync();
    if (blockIdx.y == 0 && r < rows) {  // rank 0 of the cluster: splits in order
      T s = T(0);
      for (unsigned k = 0; k < gridDim.y; ++k) s += dev::dsmem_ld(&split_part[threadIdx.x], k);
      y[r] = accumulate ? y[r] + s : s;
    }
    dev::cluster_sync();  // the other splits stay resident until rank 0 has read them
  }
}

// Row-streaming form of a small matrix, all latency: a warp per row, every load
// of the row in flight at once - vectors (AL: rows and x on 16-byte boundaries)
// or elements - and no barrier.  cols at most kShortCols.  us back to back in a
// graph, by the general form (before its remainder had its loads in flight
// together) and here: f32 310 x 448 4.1 and 1.7, 64 x 67 2.0 and 1.1, 1000 x 512
// 2.3 and 1.9; f64 64 x 67 2.5 and 1.8.
template <typename T>
constexpr int kShortCols = sizeof(T) == 4 ? 512 : 256;
template <typename T, bool AL>
__global__ void __launch_bounds__(kRowsThreads) gemv_rows_short_kernel(int rows, int cols, const T* __restrict__ A,
                                                                       int64_t lda, const T* __restrict__ x,
                                                                       T* __restrict__ y, bool accumulate) {
  using VT = std::conditional_t<AL, typename V<T>::t, T>;
  constexpr int W = AL ? V<T>::w : 1, U = kShortCols<T> / (32 * W);
  const int lane = threadIdx.x & 31, r = (int)blockIdx.x * kWarps + (int)(threadIdx.x >> 5);
  if (r >= rows) return;
  const T* __restrict__ row = A + r * lda;
  VT a[U], xv[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (lane + 32 * u < cols / W) {
      a[u] = dev::ld_stream(reinterpret_cast<const VT*>(row) + lane + 32 * u);
      xv[u] = __ldg(reinterpret_cast<const VT*>(x) + lane + 32 * u);
    }
  const int c = cols / W * W + lane;  // AL: the elements after the last vector
  T ea = T(0), ex = T(0);
  if (AL && c < cols) {
    ea = dev::ld_stream(row + c);
    ex = __ldg(x + c);
  }
  T s = T(0);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (lane + 32 * u < cols / W) {
      if constexpr (AL)
        s = vdot(a[u], xv[u], s);
      else
        s = fma(a[u], xv[u], s);
    }
  if (AL && c < cols) s = fma(ea, ex, s);
  s = dev::warp_sum(s);
  if (lane == 0) y[r] = accumulate ? y[r] + s : s;
}

// y[r] = (accumulate ? y[r] : 0) + sum_s partials[s*rows + r].  Up to 16
// splits: a thread per row, in split order.  More: 8 threads per row, thread
// g adding splits g, g + 8, ..., their sums then added in order of g (a
// thread alone waited for one load after another: 8191 rows of 38 splits took
// 10.6 us).
__device__ __forceinline__ int finish_group(int ksplit) { return ksplit > 16 ? 8 : 1; }

template <typename T>
__global__ void __launch_bounds__(256) finish_splits_kernel(int64_t rows, int ksplit, const T* partials,
                                                            T* __restrict__ y, bool accumulate) {
  dev::grid_wait();
  __shared__ T part[256];
  const int groups = finish_group(ksplit), per = 256 / groups;
  const int g = (int)threadIdx.x / per;
  const int64_t r = (int64_t)blockIdx.x * per + threadIdx.x % per;
  T s = T(0);
  if (r < rows) {
    const T* p = partials + r;
    int k = g;
    for (; k + 7 * groups < ksplit; k += 8 * groups) {
      T v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcg(p + (int64_t)(k + u * groups) * rows);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; k < ksplit; k += groups) s += __ldcg(p + (int64_t)k * rows);
  }
  if (groups > 1) {
    part[threadIdx.x] = s;
    __syncthreads();
    if (g > 0) return;
    for (int i = 1; i < groups; ++i) s += part[i * per + threadIdx.x];
  }
  if (r < rows) y[r] = accumulate ? y[r] + s : s;
}

// Column-streaming form.  A warp owns 32 VW consecutive rows (a 16-byte
// vector of VW rows a lane, or one row), a CTA's 8 warps take the columns of
// its range 8 at a time in turn, and their sums meet in shared memory.
// SHIFT (VW > 1, columns that do not all start on a 16-byte boundary): column
// c is read from the boundary at or before its first row of the block, m(c)
// elements early; columns 4 apart share m, so a lane keeps one set of sums
// per c % 4 and the sets are shifted back when they meet.  A block then owns
// the 32 VW - 4 rows that every shift covers.
// grid = (row blocks, ksplit); split p covers cps columns (a multiple of 64).
// CL: the ksplit CTAs of a row block form a cluster (1, ksplit, 1).
constexpr int kColsUnroll = 8;

template <int VW, bool SHIFT>
struct ColsCfg {
  static constexpr int kSpan = 32 * VW;                    // rows a warp reads
  static constexpr int kRows = SHIFT ? kSpan - 4 : kSpan;  // rows a block owns
  static constexpr int kSets = SHIFT ? 4 : 1;
};

template <typename T, int VW, bool SHIFT, bool CL>
__global__ void __launch_bounds__(256, 3)
    gemv_cols_kernel(int64_t rows, int64_t cols, const T* __restrict__ A, int64_t lda, const T* __restrict__ x,
                     T* __restrict__ y, bool accumulate, T* __restrict__ partials, int64_t cps, int rw) {
  using VT = std::conditional_t<VW == 1, T, typename V<T>::t>;
  using CF = ColsCfg<VW, SHIFT>;
  constexpr int U = kColsUnroll, SETS = CF::kSets, SPAN = CF::kSpan;
  static_assert(VW == 1 || VW == V<T>::w, "one row or a 16-byte vector of rows");
  __shared__ T part[kWarps][SETS][SPAN];
  __shared__ T split_part[CL ? kWarps * SPAN : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wc = kWarps / rw;  // warps that share a row block's columns
  const int64_t cta_rb = (int64_t)blockIdx.x * rw * CF::kRows;   // the CTA's first row
  const int64_t rb = cta_rb + (int64_t)(warp % rw) * CF::kRows;  // this warp's
  const int64_t c0 = (int64_t)blockIdx.y * cps;
  const int64_t c1 = min(c0 + cps, cols);
  T acc[SETS][VW];
#pragma unroll
  for (int q = 0; q < SETS; ++q)
#pragma unroll
    for (int i = 0; i < VW; ++i) acc[q][i] = T(0);
  // elements from the 16-byte boundary to column c's row rb (columns 4 apart agree)
  auto shift_of = [&](int64_t c) {
    return SHIFT ? (int)((reinterpret_cast<uintptr_t>(A + rb + c * lda) & 15) / sizeof(T)) : 0;
  };
  int m[SETS];
#pragma unroll
  for (int q = 0; q < SETS; ++q) m[q] = shift_of(c0 + q);  // c0 is a multiple of 4

  // a block whose every vector lies inside its column (not the first or last)
  const bool inside = (rb >= 4 || !SHIFT) && rb + SPAN <= rows;
  for (int64_t c = c0 + warp / rw * U; c < c1; c += wc * U) {
    const T* p = A + rb + VW * lane + c * lda;
    if (inside && c + U <= c1) {
      VT a[U];
      T xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) a[u] = dev::ld_stream(reinterpret_cast<const VT*>(p + u * lda - m[u % SETS]));
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = __ldg(x + c + u);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T* e = reinterpret_cast<const T*>(&a[u]);
#pragma unroll
        for (int i = 0; i < VW; ++i) acc[u % SETS][i] = fma(e[i], xv[u], acc[u % SETS][i]);
      }
    } else {
      T a[U][VW];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t rv = rb + VW * lane - m[u % SETS];  // the vector's first row
#pragma unroll
        for (int i = 0; i < VW; ++i)
          a[u][i] = (c + u < c1 && rv + i >= 0 && rv + i < rows) ? dev::ld_stream(p + u * lda - m[u % SETS] + i) : T(0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c + u < c1) {
          const T xc = __ldg(x + c + u);
#pragma unroll
          for (int i = 0; i < VW; ++i) acc[u % SETS][i] = fma(a[u][i], xc, acc[u % SETS][i]);
        }
    }
  }
  dev::grid_release();  // a chained finish_splits_kernel may be set up
#pragma unroll
  for (int q = 0; q < SETS; ++q)
#pragma unroll
    for (int i = 0; i < VW; ++i) part[warp][q][VW * lane + i] = acc[q][i];
  __syncthreads();
  // the CTA's rows: their sums over the column warps and sets, in order
  for (int t = threadIdx.x; t < rw * CF::kRows; t += kRowsThreads) {
    const int64_t r = cta_rb + t;
    if (r >= rows) break;
    const int blk = t / CF::kRows, i = t % CF::kRows;
    const int64_t brow = cta_rb + (int64_t)blk * CF::kRows;
    T sum = T(0);
#pragma unroll
    for (int q = 0; q < SETS; ++q) {
      const int mq = SHIFT ? (int)((reinterpret_cast<uintptr_t>(A + brow + (c0 + q) * lda) & 15) / sizeof(T)) : 0;
      for (int w = 0; w < wc; ++w) {
        const T v = part[w * rw + blk][q][i + mq];
        sum = q + w == 0 ? v : sum + v;
      }
    }
    if (CL)
      split_part[t] = sum;
    else if (gridDim.y == 1)
      y[r] = accumulate ? y[r] + sum : sum;
    else
      partials[(int64_t)blockIdx.y * rows + r] = sum;
  }
  if constexpr (CL) {
    dev::cluster_sync();
    if (blockIdx.y == 0) {  // rank 0 of the cluster: splits in order
      for (int t = threadIdx.x; t < rw * CF::kRows && cta_rb + t < rows; t += kRowsThreads) {
        T s = T(0);
        for (unsigned k = 0; k < gridDim.y; ++k) s += dev::dsmem_ld(&split_part[t], k);
        y[cta_rb + t] = accumulate ? y[cta_rb + t] + s : s;
      }
    }
    dev::cluster_sync();  // the other splits stay resident until rank 0 has read them
  }
}

inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Launch with clusters of (1, grid.y, 1): the splits of one row block.
template <typename... P, typename... A>
cudaError_t launch_split_clusters(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = grid.y;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace

namespace {

// The kernel over `grid` with its splits as clusters, or with partials in
// scratch and the finish behind it.
template <typename T, typename K, typename... A>
gbblas_status launch_split(DeviceCtx* c, K clustered, K plain, dim3 grid, int64_t rows, int64_t cols, T* y,
                           bool accumulate, cudaStream_t stream, const char* what, const T* mat, int64_t lda,
                           const T* x, A... more) {
  const int64_t ksplit = grid.y;
  T* partials = nullptr;
  if (cluster_splits(ksplit, rows, cols, sizeof(T))) {
    if (launch_split_clusters(clustered, grid, kRowsThreads, stream, rows, cols, mat, lda, x, y, accumulate, partials,
                              more...) == cudaSuccess)
      return check_launch(what);
    cudaGetLastError();  // the cluster launch was refused: partials in scratch instead
  }
  if (ksplit > 1) {
    void* s = nullptr;
    GB_TRY(get_scratch(c, stream, kScratchZeroBytes + sizeof(T) * ksplit * rows, &s));
    partials = reinterpret_cast<T*>(static_cast<char*>(s) + kScratchZeroBytes);
  }
  plain<<<grid, kRowsThreads, 0, stream>>>(rows, cols, mat, lda, x, y, accumulate, partials, more...);
  GB_TRY(check_launch(what));
  if (ksplit > 1) {
    const int64_t per = 256 / (ksplit > 16 ? 8 : 1);
    GB_CUDA_TRY(launch_after(finish_splits_kernel<T>, dim3((unsigned)cdiv(rows, per)), 256, 0, stream, rows,
                             (int)ksplit, (const T*)partials, y, accumulate));
    GB_TRY(check_launch("finish_splits_kernel"));
  }
  return GBBLAS_STATUS_SUCCESS;
}

// Log2 of the number of rows after which a row starts at the same offset from
// a 16-byte boundary again: 1, 2 or 4 rows.
template <typename T>
int align_period(int64_t lda) {
  const int64_t off = lda * (int64_t)sizeof(T) % 16;
  return off == 0 ? 0 : (off == 8 ? 1 : 2);
}

}  // namespace

template <typename T>
gbblas_status launch_gemv_rows(DeviceCtx* c, int64_t rows, int64_t cols, const T* A, int64_t lda, const T* x,
                               T* y, bool accumulate, cudaStream_t stream) {
  if (rows <= 0) return GBBLAS_STATUS_SUCCESS;
  constexpr int W = V<T>::w;
  const int64_t nv = cols / W, sms = c->num_sms;
  const int odd = align_period<T>(lda);
  const bool al = odd == 0 && aligned16(A) && aligned16(x);
  if (rows <= 1024 && cols <= kShortCols<T>) {
    const dim3 grid((unsigned)cdiv(rows, kWarps));
    if (al)
      gemv_rows_short_kernel<T, true><<<grid, kRowsThreads, 0, stream>>>((int)rows, (int)cols, A, lda, x, y, accumulate);
    else
      gemv_rows_short_kernel<T, false><<<grid, kRowsThreads, 0, stream>>>((int)rows, (int)cols, A, lda, x, y, accumulate);
    return check_launch("gemv_rows_short_kernel");
  }
  // Rows per group, warps per group (2^lwc) and column ranges, from a sweep of
  // 300 shapes of 48 .. 32768 rows and columns, both types, aligned and not, over
  // every choice, on cold operands back to back in a graph (calls timed from the
  // host start 4 us apart at best, which hid what small ones take): 2.5-4 % off
  // the best choice of each shape in the mean.  Four rows a group once the rows
  // make enough of them; more warps a group while a warp has more than `most`
  // vectors of a row, or there are few warps and each keeps 32 vectors; fewer
  // again where the CTAs would be one round of four an SM and a part of another
  // (double, bound by its FP64 work, up to several); then the columns in ranges
  // while the CTAs do not fill the SMs and a warp keeps 256 vectors (128, float
  // and under half a CTA an SM).  us, a CTA per row group / the rule that left
  // each warp 64 or 128 vectors / now: f32 707 x 3824 4.0 / 5.1 / 4.4, 4096 x 512
  // 4.1 / 5.7 / 3.4, 32768 x 2048 39.3 / 42.7 / 40.4; f64 740 x 2083 7.3 / 9.8 /
  // 7.4, 4096 x 1024 21.5 / 15.9 / 12.1, 32768 x 1024 146 / 95 / 66.
  constexpr bool kF32 = sizeof(T) == 4;
  const int R = rows >= (kF32 ? 1024 : 3000) ? 4 : 1;
  const int lperiod = R == 1 ? 0 : odd;
  const int64_t groups = cdiv(rows, (int64_t)R << lperiod) << lperiod;
  const int64_t most = kF32 ? 128 : 256, few = (kF32 ? 8 : 4) * sms;
  int lwc = 0;
  while (lwc < 3 && ((nv >> lwc) > most || ((nv >> (lwc + 1)) >= 32 && (groups << lwc) < few))) ++lwc;
  auto ctas_of = [&](int l) { return cdiv(groups, kWarps >> l); };
  const int64_t over = (kF32 ? 4 : (R == 1 ? 3 : 8)) * sms, upto = (kF32 ? 6 : 20) * sms;
  while (lwc > 0 && ctas_of(lwc) > over && ctas_of(lwc) <= upto && (nv >> (lwc - 1)) <= (kF32 ? 2048 : 1024)) --lwc;
  const int64_t ctas = ctas_of(lwc);
  // (single rows beyond 60 MB: an incomplete round of CTAs costs more than the
  // second kernel: f32 312 x 200001 57 us in ranges and 64 whole, 312 x 23256 17.4
  // and 14.3; f64 312 x 50000 42 and 47, 312 x 8192 17.2 and 14.4)
  const double bytes = (double)rows * cols * sizeof(T);
  const int64_t enough = R == 1 && bytes > 60.0e6 ? 5 * sms / 2 : (kF32 ? 3 * sms / 2 : sms);
  int64_t ksplit = 1;
  if (ctas < enough) ksplit = std::min(cdiv(4 * sms, ctas), nv >> (lwc + (kF32 && ctas < sms / 2 ? 7 : 8)));
  ksplit = std::max<int64_t>(1, std::min<int64_t>(ksplit, 65535));
  const int64_t vps = cdiv(cdiv(nv, ksplit), 32) * 32;
  if (vps > 0) ksplit = std::max<int64_t>(1, cdiv(nv, vps));
  const dim3 grid((unsigned)ctas, (unsigned)ksplit);
  // (CTAs an SM: float's four rows on boundaries fit four, and take them except
  // from 300 MB on, where three read DRAM better: 16384^2 157 us with four, 151
  // with three; 16384 x 8192 81 and 78; 2048 x 32768 42 and 47, 8192 x 1024 7.0 and 7.9)
  const bool huge = kF32 && bytes > 300.0e6;
#define GB_ROWS(R_, AL_, CTAS_)                                                                                   \
  launch_split<T>(c, gemv_rows_kernel<T, R_, AL_, true, CTAS_>, gemv_rows_kernel<T, R_, AL_, false, CTAS_>, grid, \
                  rows, cols, y, accumulate, stream, "gemv_rows_kernel", A, lda, x, vps, lperiod, lwc)
  if (R == 4) return !al ? GB_ROWS(4, false, 3) : (kF32 && !huge ? GB_ROWS(4, true, (kF32 ? 4 : 3)) : GB_ROWS(4, true, 3));
  return al ? GB_ROWS(1, true, 4) : GB_ROWS(1, false, 4);
#undef GB_ROWS
}

template <typename T>
gbblas_status launch_gemv_cols(DeviceCtx* c, int64_t rows, int64_t cols, const T* A, int64_t lda, const T* x,
                               T* y, bool accumulate, cudaStream_t stream) {
  if (rows <= 0) return GBBLAS_STATUS_SUCCESS;
  constexpr int W = V<T>::w;
  const bool vec = aligned16(A) && (lda % W) == 0;
  // unaligned columns: one row a lane, or, for a float matrix beyond 100 MB,
  // shifted vectors (16387 x 4096 48 us, 53 by elements; 8195 x 256 6.6 and 5.1,
  // 259 x 128 4.0 and 2.7: their four sets of sums weigh there); double is bound
  // by the FP64 pipes, and no row is to be computed twice
  constexpr bool kF32 = sizeof(T) == 4;
  const double bytes = (double)rows * cols * sizeof(T);
  const bool shift = kF32 && !vec && bytes > 100.0e6;
  const int64_t span = vec ? ColsCfg<W, false>::kRows : (shift ? ColsCfg<W, true>::kRows : 32);
  // two row blocks a CTA from 2048 rows (their pieces of a column adjoin: at
  // 16384^2 f32 159 us with one, 154-156 with two, 160 with eight), one below
  const int rw = rows > 2048 ? 2 : 1;
  const int64_t blocks = cdiv(rows, span * rw);
  // columns per CTA: enough CTAs for 16 per SM (5 of single rows up to 20 MB: shapes
  // of 8 .. 20 MB 6 % faster in the mean), at least 64 columns, a whole
  // number of rounds (8 columns a warp); double, whose time is its FP64 work,
  // shares short rows out evenly instead (20069 x 264: 20 us, 23 in 64s and a
  // rest; float 11.0 and 10.3)
  const int64_t per_sm = kF32 && !vec && bytes < 20.0e6 ? 5 : 16;
  const int64_t want = std::min<int64_t>(cdiv(per_sm * c->num_sms, blocks), 65535), round = 8 * (kWarps / rw);
  const int64_t even = cdiv(cols, std::max<int64_t>(1, std::min(want, cols / 64)));
  const int64_t cps = cdiv(!kF32 ? even : std::max<int64_t>(cdiv(cols, want), 64), round) * round;
  const dim3 grid((unsigned)blocks, (unsigned)std::max<int64_t>(1, cdiv(cols, cps)));
  if (vec)
    return launch_split<T>(c, gemv_cols_kernel<T, W, false, true>, gemv_cols_kernel<T, W, false, false>, grid, rows,
                           cols, y, accumulate, stream, "gemv_cols_kernel", A, lda, x, cps, rw);
  if constexpr (kF32)
    if (shift)
      return launch_split<T>(c, gemv_cols_kernel<T, W, true, true>, gemv_cols_kernel<T, W, true, false>, grid, rows,
                             cols, y, accumulate, stream, "gemv_cols_kernel", A, lda, x, cps, rw);
  return launch_split<T>(c, gemv_cols_kernel<T, 1, false, true>, gemv_cols_kernel<T, 1, false, false>, grid, rows,
                         cols, y, accumulate, stream, "gemv_cols_kernel", A, lda, x, cps, rw);
}

#define GB_INST(T)                                                                                          \
  template gbblas_status launch_gemv_rows<T>(DeviceCtx*, int64_t, int64_t, const T*, int64_t, const T*, T*, \
                                             bool, cudaStream_t);                                            \
  template gbblas_status launch_gemv_cols<T>(DeviceCtx*, int64_t, int64_t, const T*, int64_t, const T*, T*, \
                                             bool, cudaStream_t);
GB_INST(float)
GB_INST(double)
#undef GB_INST

}  // namespace gbblas
