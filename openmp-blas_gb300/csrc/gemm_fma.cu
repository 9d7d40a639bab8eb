// gemm_fma.cu - C += A*B on the CUDA cores (FP32 FMA / FP64 DFMA).
//
// Replaces the reference's Goto/BLIS GEMM (include/mtm.hpp:116-206 with the
// MR x NR micro-kernel include/simd_loop.hpp:80-192).  The GPU keeps the
// same three-level idea with GPU-sized levels:
//   * a CTA owns a BM x BN tile of C (the reference's MB x NB cache block),
//   * K is walked in BK slices that cp.async brings into a ring of kStages
//     shared-memory buffers (the reference's packed A/B panels,
//     include/utils.hpp:99-141), so three slices' loads are in flight during
//     the FMAs on the current one,
//   * each thread owns a TM x TN register tile (the reference's MR x NR
//     `buff`), accumulates over its K from zero in k order with FMA, and the
//     tile is finally added into C - like copy_from_buff, C is accumulated.
// Every (C, A, B) layout mix is served.  Operands reach one K-major
// shared-memory layout element by element (4- / 8-byte cp.async, coalesced
// along whichever dimension is contiguous, zero-filled outside the matrix),
// or as 16-byte cp.async where rows (columns) along M (N) start on 16-byte
// boundaries; the inner loop does not change.  The finished tile goes through
// shared memory, so C is read and written along its contiguous rows at any
// alignment (a column-major 8192 x 3328 C over K = 72 was bound by its
// scattered update: 440 us, now 127); a column-major C is computed as C^T = B^T A^T (the same products
// in the same order, so the same bits).
//
// Split-K: where the tiles leave SMs idle, the CTAs of a thread-block cluster
// (1, s, 1) each take 1/s of a tile's K slices and leave their sums in their
// shared memory; rank r then adds rows r / s of all s sums in rank order
// through distributed shared memory and updates that part of C.  One launch,
// no scratch, a fixed order.
//
// Bound by the FMA pipes at large sizes (4097 x 4099 x 1025: 48 TFLOP/s, 41
// with register staging before the ring), by latency at one CTA per SM - a
// slice then takes 0.6 us, three times its FMAs - hence the cut of K.  64 x
// 64 tiles take 128 threads of 8 x 4 outputs: 256 threads of 4 x 4 spend more
// of their issue slots on shared-memory loads (1023 x 1021 x 1025: 80 against
// 70 us).
#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace gbblas {
namespace {

// How an operand's elements are fetched (mn: the M or N index).
enum : int {
  kLoadVec = 0,  // mn contiguous, 16-byte aligned: 16 bytes along mn
  kLoadMN = 1,   // one element at a time, consecutive threads along mn (also general strides)
  kLoadK = 2     // one element at a time, consecutive threads along k
};

constexpr int kBK = 16;
constexpr int kStages = 4;
constexpr int kMaxSplit = 8;  // portable cluster size

template <typename T, int BM, int BN, int TM, int TN>
struct Cfg {
  static constexpr int W = 16 / (int)sizeof(T);  // elements of a 16-byte vector
  static constexpr int NT = (BM / TM) * (BN / TN);
  static constexpr int LDA = BM + 4, LDB = BN + 4;  // padded: 16-byte rows, k-strided stores two to a bank
  static constexpr int TM4 = TM / 4, TN4 = TN / 4;
  static_assert(TM % 4 == 0 && TN % 4 == 0, "register tile in groups of 4");
  static_assert(NT % BM == 0 && NT % BN == 0, "the loaders' thread maps");
  // registers: 128 a thread at most
  static constexpr int kMinCtas = 65536 / (NT * 128);
  static constexpr size_t kRing = (size_t)kStages * kBK * (LDA + LDB) * sizeof(T);
  static constexpr size_t kTile = (size_t)BM * BN * sizeof(T);  // the finished tile, in the ring's place
  static constexpr size_t kSmem = kRing > kTile ? kRing : kTile;
};

// 4 consecutive T from shared memory (16-byte aligned).
__device__ __forceinline__ void lds4(const float* p, float (&o)[4]) {
  float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void lds4(const double* p, double (&o)[4]) {
  double2 v0 = reinterpret_cast<const double2*>(p)[0];
  double2 v1 = reinterpret_cast<const double2*>(p)[1];
  o[0] = v0.x; o[1] = v0.y; o[2] = v1.x; o[3] = v1.y;
}
__device__ __forceinline__ void sts4(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void sts4(double* p, const double* v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// Asynchronous copy of one element / of 16 bytes into shared memory; bytes
// beyond `n` are not read and arrive as zero (n = 0: src is not touched).
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, int n) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One thread's share of an operand's slices: elements (mn, k), mn0 <= mn <
// mn0 + B, of 16 consecutive k at a time, into dst[k][mn] (row pitch LD).
// Element (mn, k) at src[mn * smn + k * sk]; those at mn >= MN or k >= K read
// as zero.
template <typename T, int B, int LD, int NT>
struct Loader {
  static constexpr int W = 16 / (int)sizeof(T);
  static constexpr int kPer = B / W;                  // 16-byte vectors per k
  static constexpr int kVecs = kPer * kBK / NT;       // of them per thread
  static constexpr int kElems = B * kBK / NT;         // elements per thread
  static_assert(NT % kPer == 0 && kVecs >= 1, "whole vectors per thread");
  const T* p;        // this thread's first element of the next slice
  int64_t step;      // its next element (vector) lies this far on
  int k;             // the first element's k within the slice
  int n;             // bytes of a vector that exist / elements along mn that exist
  int off, dstep;    // their places in the slice buffer
  int mode;

  __device__ __forceinline__ void init(const T* src, int mode_, int64_t mn0, int64_t MN, int64_t k0, int64_t smn,
                                       int64_t sk) {
    mode = mode_;
    const int tid = threadIdx.x;
    k = mode == kLoadVec ? tid / kPer : (mode == kLoadK ? tid % kBK : tid / B);
    const int mn = mode == kLoadVec ? tid % kPer * W : (mode == kLoadK ? tid / kBK : tid % B);
    const int64_t left = MN - mn0 - mn;
    p = src + (mn0 + mn) * smn + (k0 + k) * sk;
    off = k * LD + mn;
    if (mode == kLoadVec) {
      n = left >= W ? 16 : (left > 0 ? (int)left * (int)sizeof(T) : 0);
      step = NT / kPer * sk;
      dstep = NT / kPer * LD;
    } else if (mode == kLoadK) {
      n = left <= 0 ? 0 : (left >= B ? kElems : (int)((left + NT / kBK - 1) / (NT / kBK)));
      step = NT / kBK * smn;
      dstep = NT / kBK;
    } else {
      n = left > 0 ? kElems : 0;
      step = NT / B * sk;
      dstep = NT / B * LD;
    }
  }
  // queue the next slice's copies, of which k < kr exist
  __device__ __forceinline__ void load(T* dst, int64_t sk, int kr) {
    T* d = dst + off;
    if (mode == kLoadVec) {
#pragma unroll
      for (int i = 0; i < kVecs; ++i)
        cp_async<16>(d + i * dstep, p + i * step, k + i * (NT / kPer) < kr ? n : 0);
    } else {
      const int cnt = mode == kLoadK ? (k < kr ? n : 0) : min(n, (kr - k + NT / B - 1) / (NT / B));
#pragma unroll
      for (int i = 0; i < kElems; ++i)
        cp_async<(int)sizeof(T)>(d + i * dstep, p + i * step, i < cnt ? (int)sizeof(T) : 0);
    }
    p += kBK * sk;
  }
};

// grid = (CTAs walking the tiles, K parts); K parts > 1: clusters (1, parts, 1).
// A: element (m, k) at A[m*rsa + k*csa]; B: (k, n) at B[k*rsb + n*csb].
template <typename T, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), Cfg<T, BM, BN, TM, TN>::kMinCtas)
    gemm_fma_kernel(int64_t M, int64_t N, int64_t K, const T* __restrict__ A, int64_t rsa, int64_t csa,
                    const T* __restrict__ B, int64_t rsb, int64_t csb, T* __restrict__ C, int64_t rsc,
                    int64_t csc, int la, int lb, int64_t tiles_n, int64_t ntiles) {
  using CF = Cfg<T, BM, BN, TM, TN>;
  constexpr int NT = CF::NT, LDA = CF::LDA, LDB = CF::LDB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* As = reinterpret_cast<T*>(smem_raw);  // [kStages][kBK][LDA]
  T* Bs = As + kStages * kBK * LDA;        // [kStages][kBK][LDB]
  T* Cs = reinterpret_cast<T*>(smem_raw);  // the finished tile [BM][BN], once the ring is idle

  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  // this CTA's part of K, whole slices
  const int parts = (int)gridDim.y, part = (int)blockIdx.y;
  const int64_t slices = (K + kBK - 1) / kBK;
  const int64_t s0 = slices * part / parts;
  const int ns = (int)(slices * (part + 1) / parts - s0);

  // Tiles are handed out grid-stride, so a grid capped below the tile count
  // (a caller sharing the GPU with latency-sensitive work) still covers C.
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = T(0);

    Loader<T, BM, LDA, NT> ldA;
    Loader<T, BN, LDB, NT> ldB;
    ldA.init(A, la, m0, M, s0 * kBK, rsa, csa);
    ldB.init(B, lb, n0, N, s0 * kBK, csb, rsb);
    auto load = [&](int s) {  // slice s of this part into its ring buffer (one commit group, empty past the end)
      if (s < ns) {
        const int buf = s % kStages;
        const int64_t rest = K - (s0 + s) * kBK;
        const int kr = rest < kBK ? (int)rest : kBK;
        ldA.load(As + buf * kBK * LDA, csa, kr);
        ldB.load(Bs + buf * kBK * LDB, rsb, kr);
      }
      cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) load(s);
    for (int s = 0; s < ns; ++s) {
      cp_async_wait<kStages - 2>();  // slice s has landed (this thread's copies) ...
      __syncthreads();               // ... everyone's, and buffer (s - 1) % kStages is free again
      load(s + kStages - 1);
      const T* as = As + s % kStages * kBK * LDA + ty * 4;
      const T* bs = Bs + s % kStages * kBK * LDB + tx * 4;
      // double: only the k that exist, since on the FP64 pipes those of the
      // last slice that do not would take as long as the others (2048 x 2048 x 1
      // 126 us, 26 so; 304 x 34 x 20 39.3, 26.9; 1024 x 147 x 37 55.7, 43.7)
      const int kn = (int)min((int64_t)kBK, K - (s0 + s) * kBK);
#pragma unroll
      for (int k = 0; k < kBK; ++k) {
        if (sizeof(T) == 8 && k >= kn) break;
        T a[TM], b[TN];
#pragma unroll
        for (int g = 0; g < CF::TM4; ++g) {
          T t[4];
          lds4(as + k * LDA + g * (BM / CF::TM4), t);
#pragma unroll
          for (int i = 0; i < 4; ++i) a[g * 4 + i] = t[i];
        }
#pragma unroll
        for (int g = 0; g < CF::TN4; ++g) {
          T t[4];
          lds4(bs + k * LDB + g * (BN / CF::TN4), t);
#pragma unroll
          for (int j = 0; j < 4; ++j) b[g * 4 + j] = t[j];
        }
        if constexpr (sizeof(T) == 4) {
          // packed FP32x2 FMAs: two columns per instruction, each lane an IEEE
          // fmaf (bit-identical to the scalar form), half the issue slots
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const float2 ai = make_float2(a[i], a[i]);
#pragma unroll
            for (int j = 0; j < TN; j += 2) {
              const float2 r = __ffma2_rn(ai, make_float2(b[j], b[j + 1]), make_float2(acc[i][j], acc[i][j + 1]));
              acc[i][j] = r.x;
              acc[i][j + 1] = r.y;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
      }
    }

    // ---- C += the tile (the reference's copy_from_buff, include/simd_loop.hpp:160-190)
    // this part's rows of the tile, consecutive threads along n: column
    // tid % BN, every kRowStep-th row; a batch's loads are issued before its
    // stores (the compiler cannot see that runtime strides keep the outputs
    // apart), the first batch's before the sums are exchanged
    constexpr int kRowStep = NT / BN, UN = 16;
    const int r1 = BM * (part + 1) / parts, col = tid % BN;
    int r = BM * part / parts + tid / BN;
    const int rows = n0 + col < N ? (int)min((int64_t)r1, M - m0) : 0;  // rows r < rows exist
    T* cp = C + (m0 + r) * rsc + (n0 + col) * csc;
    T old[UN];
    auto load_old = [&]() {
#pragma unroll
      for (int u = 0; u < UN; ++u) old[u] = r + u * kRowStep < rows ? cp[u * kRowStep * rsc] : T(0);
    };
    load_old();
    cp_async_wait<0>();
    __syncthreads();  // the ring is idle: the tile takes its place
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      T* row = Cs + ((i / 4) * (BM / CF::TM4) + ty * 4 + (i % 4)) * BN + tx * 4;
#pragma unroll
      for (int g = 0; g < CF::TN4; ++g) sts4(row + g * (BN / CF::TN4), &acc[i][g * 4]);
    }
    if (parts > 1)
      dev::cluster_sync();
    else
      __syncthreads();
    while (r < rows) {
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int ru = r + u * kRowStep;
        if (ru < rows) {
          const T* sp = Cs + ru * BN + col;
          T v;
          if (parts == 1) {
            v = *sp;
          } else {
            v = dev::dsmem_ld(sp, 0);
            for (int q = 1; q < parts; ++q) v += dev::dsmem_ld(sp, (unsigned)q);
          }
          cp[u * kRowStep * rsc] = old[u] + v;
        }
      }
      r += UN * kRowStep;
      cp += UN * kRowStep * rsc;
      load_old();
    }
    // the next tile's copies overwrite Cs: not before everyone has read it
    // (and a CTA of a cluster leaves only then)
    if (parts > 1)
      dev::cluster_sync();
    else
      __syncthreads();
  }  // tile loop
}

template <typename T, int BM, int BN, int TM, int TN>
void set_attributes(DeviceCtx* c) {
  static std::mutex mu;
  static bool done[64] = {false};
  std::lock_guard<std::mutex> lk(mu);
  if (done[c->device & 63]) return;
  cudaFuncSetAttribute(gemm_fma_kernel<T, BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Cfg<T, BM, BN, TM, TN>::kSmem);
  done[c->device & 63] = true;
}

// K parts of a split launch: as many as bring the CTAs to two per SM, each
// part at least two slices, at most a portable cluster; none below eight
// slices, where the cluster's barriers cost more than the slices they save
// (64^3: 8.2 us in one part, 10.3 in two; 211 x 190 x 173: 14.4 us before,
// 8.2 in five parts; 649 x 47 x 8192: 304 us in one part, 45 in eight).
template <int BM, int BN>
int split_parts(const DeviceCtx* c, int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int64_t slices = (K + kBK - 1) / kBK;
  if (slices < 8) return 1;
  const int64_t s = std::min<int64_t>({(int64_t)kMaxSplit, 2 * (int64_t)c->num_sms / tiles, slices / 2});
  return s > 1 ? (int)s : 1;
}

template <typename T, int BM, int BN, int TM, int TN>
gbblas_status launch_cfg(DeviceCtx* c, int64_t M, int64_t N, int64_t K, const T* A, int64_t rsa, int64_t csa,
                         const T* B, int64_t rsb, int64_t csb, T* C, int64_t rsc, int64_t csc,
                         cudaStream_t stream, int max_ctas, int parts) {
  using CF = Cfg<T, BM, BN, TM, TN>;
  // how each operand is fetched (mn stride, k stride)
  auto mode = [](const T* p, int64_t smn, int64_t sk) {
    if (smn == 1 && aligned16(p) && sk % CF::W == 0) return (int)kLoadVec;
    return (sk == 1 && smn != 1) ? (int)kLoadK : (int)kLoadMN;
  };
  const int la = mode(A, rsa, csa), lb = mode(B, csb, rsb);
  const int64_t tiles_n = (N + BN - 1) / BN, ntiles = tiles_n * ((M + BM - 1) / BM);
  int64_t g = ntiles;
  if (max_ctas > 0) {
    parts = std::min(parts, max_ctas);
    g = std::min<int64_t>(g, max_ctas / parts);
  }
  if (g > 0x7fffffff) g = 0x7fffffff;
  set_attributes<T, BM, BN, TM, TN>(c);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g, (unsigned)parts);
  cfg.blockDim = dim3(CF::NT);
  cfg.dynamicSmemBytes = CF::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = (unsigned)parts;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_fma_kernel<T, BM, BN, TM, TN>, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc,
                                 csc, la, lb, tiles_n, ntiles));
  return check_launch("gemm_fma_kernel");
}

}  // namespace

void gemm_fma_prepare(DeviceCtx* c) {
  set_attributes<float, 128, 128, 8, 8>(c);
  set_attributes<float, 64, 64, 8, 4>(c);
  set_attributes<double, 64, 64, 4, 4>(c);
}

template <typename T>
gbblas_status launch_gemm_fma(DeviceCtx* c, int64_t M, int64_t N, int64_t K, const T* A, int64_t rsa,
                              int64_t csa, const T* B, int64_t rsb, int64_t csb, T* C, int64_t rsc, int64_t csc,
                              cudaStream_t stream, int max_ctas, int tile) {
  if (M == 0 || N == 0 || K == 0) return GBBLAS_STATUS_SUCCESS;
  if (csc != 1 && rsc == 1) {  // column-major C: C^T += B^T A^T, the same products and sums
    std::swap(M, N);
    std::swap(A, B);
    std::swap(rsa, csb);
    std::swap(csa, rsb);
    std::swap(rsc, csc);
  }
  if constexpr (sizeof(T) == 4) {
    const int64_t big_tiles = ((M + 127) / 128) * ((N + 127) / 128);
    const bool tma = sgemm_tma_eligible(M, N, K, A, rsa, csa, B, rsb, csb);
    // default: TMA-fed where B is row-major (at 8192^3: 63.8 / 58.7 TFLOP/s
    // with A column- / row-major against 58.9 / 57.5 register-tiled; with B
    // column-major its FMA pairs need register moves and it trails)
    if (tile < 0)
      tile = (tma && csb == 1 && big_tiles >= (int64_t)c->num_sms) ? 2
                                                                   : (big_tiles >= 2 * (int64_t)c->num_sms ? 1 : 5);
    if (tile == 4 && tma)
      return launch_sgemm_tma(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas, 2);
    if (tile == 3 && tma)
      return launch_sgemm_tma(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas, 1);
    if (tile >= 2 && tile <= 4 && tma)
      return launch_sgemm_tma(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas);
    if (tile == 6 || (tile >= 1 && tile <= 4))
      return launch_cfg<float, 128, 128, 8, 8>(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas,
                                               tile == 6 ? split_parts<128, 128>(c, M, N, K) : 1);
    return launch_cfg<float, 64, 64, 8, 4>(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas,
                                           tile == 5 ? split_parts<64, 64>(c, M, N, K) : 1);
  } else {
    return launch_cfg<double, 64, 64, 4, 4>(c, M, N, K, A, rsa, csa, B, rsb, csb, C, rsc, csc, stream, max_ctas,
                                            split_parts<64, 64>(c, M, N, K));
  }
}

template gbblas_status launch_gemm_fma<float>(DeviceCtx*, int64_t, int64_t, int64_t, const float*, int64_t,
                                              int64_t, const float*, int64_t, int64_t, float*, int64_t, int64_t,
                                              cudaStream_t, int, int);
template gbblas_status launch_gemm_fma<double>(DeviceCtx*, int64_t, int64_t, int64_t, const double*, int64_t,
                                               int64_t, const double*, int64_t, int64_t, double*, int64_t,
                                               int64_t, cudaStream_t, int, int);

}  // namespace gbblas
