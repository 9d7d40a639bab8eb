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
// Both stream A from HBM once with 128-bit read-only loads at any leading
// dimension and keep x in L1 / shared memory.  When the grid would be too
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
// columns f32 16384^2 156.4 -> 154, 10001 x 10003 166 -> 69, 256 x 25596 36 -> 12;
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
// covers vectors p * vps .. + vps - 1.
// CL: the ksplit CTAs of a row block form a cluster (1, ksplit, 1).
template <typename T, int R, bool CL>
__global__ void __launch_bounds__(kRowsThreads, R == 4 ? 3 : 4)
    gemv_rows_kernel(int64_t rows, int64_t cols, const T* __restrict__ A, int64_t lda, const T* __restrict__ x,
                     T* __restrict__ y, bool accumulate, T* __restrict__ partials, int64_t vps, int lperiod, int lwc) {
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
  int64_t head = (int64_t)(((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) / sizeof(T));
  if (head > cols) head = cols;
  const int64_t nv = (cols - head) / W;
  const int64_t v1 = min(((int64_t)blockIdx.y + 1) * vps, nv);
  const T* __restrict__ xb = x + head;
  const bool xvec = (reinterpret_cast<uintptr_t>(xb) & 15) == 0;
  auto xload = [&](int64_t v) {
    VT r;
    if (xvec) {
      r = ldg_vec(reinterpret_cast<const VT*>(xb) + v);
    } else {
      T* e = reinterpret_cast<T*>(&r);
#pragma unroll
      for (int i = 0; i < W; ++i) e[i] = __ldg(xb + v * W + i);
    }
    return r;
  };
  T acc[R];
#pragma unroll
  for (int j = 0; j < R; ++j) acc[j] = T(0);

  const int64_t step = 32 * wc;
  int64_t v = (int64_t)blockIdx.y * vps + wi * 32 + lane;
  if (nr == R) {
    for (; v + (U - 1) * step < v1; v += U * step) {
      VT a[U][R], xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < R; ++j)
          a[u][j] = dev::ld_stream(reinterpret_cast<const VT*>(row + head + j * rstep) + v + u * step);
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = xload(v + u * step);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[j] = vdot(a[u][j], xv[u], acc[j]);
    }
  }
  for (; v < v1; v += step) {
    const VT xv = xload(v);
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j < nr) acc[j] = vdot(dev::ld_stream(reinterpret_cast<const VT*>(row + head + j * rstep) + v), xv, acc[j]);
  }
  if (blockIdx.y == 0 && wi == 0) {  // the elements before the first vector and after the last
    const int64_t tail = cols - head - nv * W;
    const int64_t c = lane < head ? lane : (lane >= 8 && lane - 8 < tail ? head + nv * W + lane - 8 : -1);
    if (c >= 0) {
      const T xc = __ldg(x + c);
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (j < nr) acc[j] = fma(dev::ld_stream(row + j * rstep + c), xc, acc[j]);
    }
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
  // warps per row group: as many as leave each 2 vectors a lane (4 where the
  // rows are few and the call is all latency: 944 x 1024 f32 4.1 us, 6.2 with 1)
  const int64_t least = rows >= 16 * sms ? 64 : 128;
  int lwc = 3;
  while (lwc > 0 && (nv >> lwc) < least) --lwc;
  // 4 rows a group once those groups make 3 CTAs per SM (2 where the 4 rows
  // share x read element by element, or the FP64 additions of their sums):
  // 1488 x 16384 f32 takes 21 us as 372 CTAs of 4 rows, 18-20 as 1488 of one
  const int R = (rows << lwc) >= (odd > 0 || sizeof(T) == 8 ? 64 : 96) * sms ? 4 : 1;
  const int lperiod = R == 1 ? 0 : odd;
  const int64_t groups = cdiv(rows, (int64_t)R << lperiod) << lperiod;
  const int64_t ctas = cdiv(groups, kWarps >> lwc);
  // split the columns while the CTAs do not fill the SMs and each warp has
  // more than 8 vectors a lane
  // (up to 60 MB only where they are fewer than two an SM, 1.5 for double: the
  // finish of a split in two costs more than the idle warps do.  Split and not,
  // us, f32 312 x 23256 17.4 and 14.3, 600 x 23256 21.2 and 18.4, 312 x 200001
  // 57 and 64; f64 312 x 8192 17.2 and 14.4, 256 x 16000 22.5 and 18.4, 312 x
  // 50000 42 and 47)
  int64_t ksplit = 1;
  const int64_t warps_enough = (double)rows * cols * sizeof(T) > 60.0e6 ? 32 : (sizeof(T) == 8 ? 12 : 16);
  if (ctas * kWarps < warps_enough * sms) ksplit = std::min(cdiv(48 * sms, ctas * kWarps), nv >> (lwc + 8));
  ksplit = std::max<int64_t>(1, std::min<int64_t>(ksplit, 65535));
  const int64_t vps = cdiv(cdiv(nv, ksplit), 32) * 32;
  if (vps > 0) ksplit = std::max<int64_t>(1, cdiv(nv, vps));
  const dim3 grid((unsigned)ctas, (unsigned)ksplit);
  if (R == 4)
    return launch_split<T>(c, gemv_rows_kernel<T, 4, true>, gemv_rows_kernel<T, 4, false>, grid, rows, cols, y,
                           accumulate, stream, "gemv_rows_kernel", A, lda, x, vps, lperiod, lwc);
  return launch_split<T>(c, gemv_rows_kernel<T, 1, true>, gemv_rows_kernel<T, 1, false>, grid, rows, cols, y,
                         accumulate, stream, "gemv_rows_kernel", A, lda, x, vps, lperiod, lwc);
}

template <typename T>
gbblas_status launch_gemv_cols(DeviceCtx* c, int64_t rows, int64_t cols, const T* A, int64_t lda, const T* x,
                               T* y, bool accumulate, cudaStream_t stream) {
  if (rows <= 0) return GBBLAS_STATUS_SUCCESS;
  constexpr int W = V<T>::w;
  const bool vec = aligned16(A) && (lda % W) == 0;
  // unaligned columns: shifted vectors for float; for double, bound by the
  // FP64 pipes, one row a lane (no row is computed twice)
  constexpr bool kShift = sizeof(T) == 4;
  using Odd = ColsCfg<kShift ? W : 1, kShift>;
  // two row blocks a CTA from 2048 rows (their pieces of a column adjoin: at
  // 16384^2 f32 159 us with one, 154-156 with two, 160 with eight), one below
  const int rw = rows > 2048 ? 2 : 1;
  const int64_t blocks = cdiv(rows, (vec ? ColsCfg<W, false>::kRows : Odd::kRows) * (int64_t)rw);
  // columns per CTA: enough CTAs for 16 per SM, at least 64 columns, a whole
  // number of rounds (8 columns a warp); double, whose time is its FP64 work,
  // shares short rows out evenly instead (20069 x 264: 20 us, 23 in 64s and a
  // rest; float 11.0 and 10.3)
  const int64_t want = std::min<int64_t>(cdiv(16 * (int64_t)c->num_sms, blocks), 65535), round = 8 * (kWarps / rw);
  const int64_t even = cdiv(cols, std::max<int64_t>(1, std::min(want, cols / 64)));
  const int64_t cps = cdiv(sizeof(T) == 8 ? even : std::max<int64_t>(cdiv(cols, want), 64), round) * round;
  const dim3 grid((unsigned)blocks, (unsigned)std::max<int64_t>(1, cdiv(cols, cps)));
  if (vec)
    return launch_split<T>(c, gemv_cols_kernel<T, W, false, true>, gemv_cols_kernel<T, W, false, false>, grid, rows,
                           cols, y, accumulate, stream, "gemv_cols_kernel", A, lda, x, cps, rw);
  if constexpr (kShift)
    return launch_split<T>(c, gemv_cols_kernel<T, W, true, true>, gemv_cols_kernel<T, W, true, false>, grid, rows,
                           cols, y, accumulate, stream, "gemv_cols_kernel", A, lda, x, cps, rw);
  else
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
