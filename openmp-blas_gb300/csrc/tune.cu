// tune.cu - the autotuner.
//
// The reference picks its blocking once per process from the CPU's cache
// geometry and a hard-coded FMA latency table (include/mtm.hpp:19-81,
// include/cpuinfo.hpp:167-223, include/cache_manager.hpp:107-150).  On the
// GPU the choices are kernel variants, and they are picked by measurement:
// the first time a (device, operation, shape bucket, dtype, accuracy) key is
// seen, every candidate is timed with CUDA events on scratch outputs and the
// fastest is remembered - in memory, and in a JSON file so later processes
// start tuned.
//
//   GBBLAS_AUTOTUNE=0      use the built-in defaults, time nothing
//   GBBLAS_TUNE_CACHE=path cache file (default $XDG_CACHE_HOME/gbblas/tune.json
//                          or ~/.cache/gbblas/tune.json); unwritable = memory only
//
// Tuned choices:
//   gemv_group_rows  rows per warp item of the grouped row-streaming GEMV
//                    (1, 2, 4, 8), bucketed by median log2 rows / cols;
//   gemm_auto        for GBBLAS_ACCURACY_AUTO, FP32 FMA kernel or the guarded
//                    FP16 split (three products) - both FP32-accurate -
//                    bucketed by log2 M, N, K;
//   gemm_tc          per split-BF16 mode and log2 M, N, K bucket: the CTA form
//                    (single CTAs, with split-K by rule, or CTA pairs);
//                    GBBLAS_TC_SPLITK=n forces n parts;
//   gemm_fma_tile    FP32 FMA kernel and CTA tile per bucket, operand
//                    layouts and alignment: 64 x 64 or 128 x 128 (K cut over
//                    a cluster's CTAs where those leave SMs idle), the TMA-fed
//                    128 x 128, that in stream-K form where whole tiles fill
//                    the SMs badly, or in cluster pairs;
//                    GBBLAS_FMA_TILE=0 .. 6 forces one (launch_gemm_fma's list).
// Nothing is timed while the caller's stream is being captured into a graph
// (the defaults apply); single-call paths consult the tuner, grouped,
// batched and served launches use the defaults.
#include <sys/stat.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <fstream>
#include <map>
#include <regex>
#include <sstream>
#include <string>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace gbblas {

gbblas_status time_gemv_group_variant(DeviceCtx* c, const gbblas_gemv_desc* d, int64_t count, int R, float* ms);

namespace {

class Tuner {
 public:
  static Tuner& get() {
    static Tuner t;
    return t;
  }

  bool enabled() const { return enabled_; }

  // Choices this process has looked up or made, by a packed key: every call
  // asks, and building the text key and searching for it took 1.5 us of a
  // call's host time.
  int recall(uint64_t packed) {
    std::lock_guard<std::mutex> lk(mu_);
    auto it = memo_.find(packed);
    return it == memo_.end() ? -1 : it->second;
  }
  int remember(uint64_t packed, int value) {
    std::lock_guard<std::mutex> lk(mu_);
    memo_[packed] = value;
    return value;
  }

  // Cached choice for `key`, or -1.
  int lookup(const std::string& key) {
    std::lock_guard<std::mutex> lk(mu_);
    load_locked();
    auto it = cache_.find(key);
    return it == cache_.end() ? -1 : it->second;
  }

  void store(const std::string& key, int value) {
    std::lock_guard<std::mutex> lk(mu_);
    load_locked();
    cache_[key] = value;
    save_locked();
  }

 private:
  Tuner() {
    const char* e = std::getenv("GBBLAS_AUTOTUNE");
    enabled_ = !(e && std::string(e) == "0");
    if (const char* p = std::getenv("GBBLAS_TUNE_CACHE")) {
      path_ = p;
    } else if (const char* x = std::getenv("XDG_CACHE_HOME")) {
      path_ = std::string(x) + "/gbblas/tune.json";
    } else if (const char* h = std::getenv("HOME")) {
      path_ = std::string(h) + "/.cache/gbblas/tune.json";
    }
  }

  void load_locked() {
    if (loaded_) return;
    loaded_ = true;
    if (path_.empty()) return;
    std::ifstream f(path_);
    if (!f) return;
    std::stringstream ss;
    ss << f.rdbuf();
    const std::string text = ss.str();
    static const std::regex kv("\"([^\"]+)\"\\s*:\\s*(-?[0-9]+)");
    for (auto it = std::sregex_iterator(text.begin(), text.end(), kv); it != std::sregex_iterator(); ++it) {
      const std::string key = (*it)[1];
      if (key == "version") continue;
      cache_[key] = std::atoi((*it)[2].str().c_str());
    }
  }

  void save_locked() {
    if (path_.empty()) return;
    const auto slash = path_.find_last_of('/');
    if (slash != std::string::npos) {
      std::string dir = path_.substr(0, slash);
      for (size_t i = 1; i <= dir.size(); ++i)
        if (i == dir.size() || dir[i] == '/') ::mkdir(dir.substr(0, i).c_str(), 0755);
    }
    const std::string tmp = path_ + ".tmp";
    std::ofstream f(tmp);
    if (!f) return;
    f << "{\n  \"version\": 1";
    for (const auto& kv : cache_) f << ",\n  \"" << kv.first << "\": " << kv.second;
    f << "\n}\n";
    f.close();
    std::rename(tmp.c_str(), path_.c_str());
  }

  std::mutex mu_;
  std::map<std::string, int> cache_;
  std::unordered_map<uint64_t, int> memo_;  // bounded by the number of keys
  bool loaded_ = false;
  bool enabled_ = true;
  std::string path_;
};

std::string device_tag(DeviceCtx* c) {
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, c->device) != cudaSuccess) return "unknown";
  std::string name = p.name;
  std::replace(name.begin(), name.end(), ' ', '_');
  return name + "_sm" + std::to_string(c->num_sms);
}

// Packed form of a key: what is chosen (op), mode or layout flags, device, buckets.
uint64_t pack_key(int op, int flags, DeviceCtx* c, int bm, int bn, int bk) {
  return (uint64_t)op | (uint64_t)flags << 4 | (uint64_t)c->device << 12 | (uint64_t)bm << 20 | (uint64_t)bn << 28 |
         (uint64_t)bk << 36;
}
enum : int { kOpAuto = 1, kOpPair = 2, kOpFma = 3 };

int log2_bucket(int64_t v) { return v <= 1 ? 0 : (int)std::lround(std::log2((double)v)); }

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();
    return true;  // unknown: do not time
  }
  return st != cudaStreamCaptureStatusNone;
}

// Scratch FP32 operands (zeros) for timing one GEMM shape on the tuner's own
// stream; each candidate runs once to warm up, then 3 times between events.
// a_col / b_col: column-major operands (C is row-major); pad: leading
// dimensions that much longer than they need be.
class GemmBench {
 public:
  GemmBench(DeviceCtx* c, int64_t m, int64_t n, int64_t k, bool a_col = false, bool b_col = false, int64_t pad = 0)
      : c_(c), m_(m), n_(n), k_(k), a_col_(a_col), b_col_(b_col), pad_(pad) {
    if (cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking) != cudaSuccess) return;
    const size_t bytes = sizeof(float) * (size_t)(a_elems() + b_elems() + m * n);
    if (cudaMallocAsync(&mem_, bytes, s_) != cudaSuccess) {
      mem_ = nullptr;
      return;
    }
    cudaMemsetAsync(mem_, 0, bytes, s_);
    cudaEventCreate(&e0_);
    cudaEventCreate(&e1_);
  }
  ~GemmBench() {
    if (mem_) cudaFreeAsync(mem_, s_);
    if (s_) {
      cudaStreamSynchronize(s_);
      release_scratch(c_, s_);
      cudaStreamDestroy(s_);
    }
    if (e0_) cudaEventDestroy(e0_);
    if (e1_) cudaEventDestroy(e1_);
  }
  bool ok() const { return mem_ != nullptr; }
  gbblas_gemm_desc desc() const {
    float* A = static_cast<float*>(mem_);
    float* B = A + a_elems();
    float* C = B + b_elems();
    const int64_t lda = (a_col_ ? m_ : k_) + pad_, ldb = (b_col_ ? k_ : n_) + pad_;
    return gbblas_gemm_desc{m_, n_, k_, A, a_col_ ? 1 : lda, a_col_ ? lda : 1, B, b_col_ ? 1 : ldb, b_col_ ? ldb : 1,
                            C, n_, 1};
  }
  cudaStream_t stream() const { return s_; }
  // ms per call of run(stream), or a huge value if it failed
  template <typename F>
  float time(F&& run) {
    if (run(s_) != GBBLAS_STATUS_SUCCESS) return 1e30f;
    cudaEventRecord(e0_, s_);
    for (int i = 0; i < 3; ++i)
      if (run(s_) != GBBLAS_STATUS_SUCCESS) return 1e30f;
    cudaEventRecord(e1_, s_);
    if (cudaEventSynchronize(e1_) != cudaSuccess) return 1e30f;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0_, e1_);
    return ms;
  }

 private:
  // (rounded so that B and C start on 16-byte boundaries)
  int64_t a_elems() const { return ((a_col_ ? k_ * (m_ + pad_) : m_ * (k_ + pad_)) + 3) / 4 * 4; }
  int64_t b_elems() const { return ((b_col_ ? n_ * (k_ + pad_) : k_ * (n_ + pad_)) + 3) / 4 * 4; }

  DeviceCtx* c_;
  int64_t m_, n_, k_;
  bool a_col_, b_col_;
  int64_t pad_;
  cudaStream_t s_ = nullptr;
  void* mem_ = nullptr;
  cudaEvent_t e0_ = nullptr, e1_ = nullptr;
};

// Representative shape of a log2 bucket: 2^b per dimension, M and N at most
// 8192, K at most 2^16, and the operands at most 2^28 elements.
void bucket_shape(int bm, int bn, int bk, int64_t& m, int64_t& n, int64_t& k) {
  m = std::min<int64_t>(int64_t(1) << bm, 8192);
  n = std::min<int64_t>(int64_t(1) << bn, 8192);
  k = std::min<int64_t>(int64_t(1) << bk, 65536);
  while ((m + n) * k > (int64_t(1) << 28) && k > 64) k >>= 1;
}

}  // namespace

int tuned_gemv_group_rows(DeviceCtx* c, const gbblas_gemv_desc* d, int64_t count) {
  constexpr int kDefault = 4;
  Tuner& t = Tuner::get();
  std::vector<int64_t> rows, cols;
  for (int64_t i = 0; i < count; ++i) {
    const bool tr = d[i].transpose != 0;
    const bool rows_contig = (d[i].layout == GBBLAS_LAST_ORDER) != tr;
    if (!rows_contig || d[i].M <= 0 || d[i].N <= 0) continue;
    rows.push_back(tr ? d[i].N : d[i].M);
    cols.push_back(tr ? d[i].M : d[i].N);
  }
  if (rows.empty()) return kDefault;
  std::nth_element(rows.begin(), rows.begin() + rows.size() / 2, rows.end());
  std::nth_element(cols.begin(), cols.begin() + cols.size() / 2, cols.end());
  const std::string key = "gemv_group_rows|" + device_tag(c) + "|r" + std::to_string(log2_bucket(rows[rows.size() / 2])) +
                          "|c" + std::to_string(log2_bucket(cols[cols.size() / 2])) + "|n" +
                          std::to_string(log2_bucket((int64_t)rows.size())) + "|f32";
  int v = t.lookup(key);
  if (v > 0) return v;
  if (!t.enabled()) return kDefault;
  int best = kDefault;
  float best_ms = 1e30f;
  for (int R : {1, 2, 4, 8}) {
    float ms = 0.f;
    if (time_gemv_group_variant(c, d, count, R, &ms) != GBBLAS_STATUS_SUCCESS) return kDefault;
    if (ms < best_ms) {
      best_ms = ms;
      best = R;
    }
  }
  t.store(key, best);
  return best;
}

// 1 = the guarded FP16 split, 0 = FP32 FMA, for an AUTO-accuracy GEMM of this
// shape on `stream`.  Without tuning: the tensor cores once the work fills them.
int tuned_gemm_auto(DeviceCtx* c, int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
  if (const char* e = std::getenv("GBBLAS_GEMM_AUTO"); e && (e[0] == '0' || e[0] == '1')) return e[0] - '0';
  const int fallback = (M >= 256 && N >= 256 && K >= 256 && (double)M * N * K >= 1.0e9) ? 1 : 0;
  Tuner& t = Tuner::get();
  const int bm = log2_bucket(M), bn = log2_bucket(N), bk = log2_bucket(K);
  const uint64_t packed = pack_key(kOpAuto, 0, c, bm, bn, bk);
  if (const int m = t.recall(packed); m >= 0) return m;
  const std::string key = "gemm_auto_f16s|" + device_tag(c) + "|m" + std::to_string(bm) + "|n" + std::to_string(bn) +
                          "|k" + std::to_string(bk) + "|f32";
  int v = t.lookup(key);
  if (v >= 0) return t.remember(packed, v);
  if (!t.enabled() || capturing(stream)) return fallback;
  // representative shape of the bucket, capped so tuning stays cheap
  const int64_t m = std::min<int64_t>(int64_t(1) << bm, 8192), n = std::min<int64_t>(int64_t(1) << bn, 8192),
                k = std::min<int64_t>(int64_t(1) << bk, 8192);
  cudaStream_t s;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return fallback;
  void* mem = nullptr;
  const size_t bytes = sizeof(float) * (size_t)(m * k + k * n + m * n);
  if (cudaMallocAsync(&mem, bytes, s) != cudaSuccess) {
    cudaStreamDestroy(s);
    return fallback;
  }
  cudaMemsetAsync(mem, 0, bytes, s);
  float* A = static_cast<float*>(mem);
  float* B = A + m * k;
  float* C = B + k * n;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  // What three FMA calls take at the pipe's peak (128 multiply-adds per clock
  // and SM): no tile need be timed, nor FMA's own choice of tile made, where the
  // tensor cores are faster than that.  First AUTO call, ms, with FMA's tile
  // tuned for every size, with one fixed tile timed, and so: 8192^3 316, 87, 15;
  // 4096^3 43, 12.4, 3.5; 1024^3 2.5, 0.9, 3.5; 512^3 1.2, 1.6, 1.9.
  int khz = 0;
  if (cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, c->device) != cudaSuccess) khz = 0;
  const float fma_least_ms = khz > 0 ? (float)(3.0 * m * n * k / (128.0 * c->num_sms * khz)) : 0.f;
  int fma_tile = -1;
  float best_ms[2] = {1e30f, 1e30f};
  for (int choice = 1; choice >= 0; --choice) {
    if (choice == 0) {
      if (best_ms[1] < fma_least_ms) break;
      fma_tile = tuned_fma_tile(c, {m, n, k, A, k, 1, B, n, 1, C, n, 1}, s);
    }
    auto run = [&]() {
      return choice == 1 ? launch_gemm_tc(c, kTcModeF16Guard, m, n, k, A, k, 1, B, n, 1, C, n, 1, s)
                         : launch_gemm_fma<float>(c, m, n, k, A, k, 1, B, n, 1, C, n, 1, s, 0, fma_tile);
    };
    if (run() != GBBLAS_STATUS_SUCCESS) continue;  // warm-up
    cudaEventRecord(e0, s);
    bool ok = true;
    for (int i = 0; i < 3 && ok; ++i) ok = run() == GBBLAS_STATUS_SUCCESS;
    cudaEventRecord(e1, s);
    if (!ok || cudaEventSynchronize(e1) != cudaSuccess) continue;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    best_ms[choice] = ms;
  }
  cudaFreeAsync(mem, s);
  cudaStreamSynchronize(s);
  release_scratch(c, s);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(s);
  if (best_ms[0] >= 1e30f && best_ms[1] >= 1e30f) return fallback;
  const int best = best_ms[1] < best_ms[0] ? 1 : 0;
  t.store(key, best);
  return t.remember(packed, best);
}

// Split-K parts of an M x N x K tensor-core GEMM on single CTAs: the number
// with the least estimated time, waves of tiles x K stages each (us per stage
// as measured at 8192^3) plus, for more than one part, the reduction (its
// launch, and the partials' bytes at about 3 TB/s).  A rule and not a
// measurement per bucket: whether tiles x parts fit the SMs in one wave turns
// on the shape itself (4880 x 249 x 4096, 78 tiles: 137 us unsplit, 178 in the
// two parts that suit its bucket's 64 tiles).  The BF16 splits and FP8 keep to
// K at least four times the larger output side, so that a product of ordinary
// proportions gives the same bits alone as in a group (whose problems are not
// split); AUTO, whose arithmetic is the library's choice per shape, splits any
// of them, and the FP16 split it stands for goes with it.
static int split_parts(DeviceCtx* c, int mode, int64_t M, int64_t N, int64_t K) {
  const int64_t sms = c->num_sms;
  const int64_t tiles = ((M + 127) / 128) * ((N + 127) / 128);
  const int64_t stages = (K + tc_stage_k(mode) - 1) / tc_stage_k(mode);
  const bool f16 = mode == kTcModeF16Guard || mode == tc_mode(GBBLAS_ACCURACY_FP16X3);
  if (tiles >= sms || (!f16 && K < 4 * std::max(M, N))) return 1;
  const double stage_us = mode == tc_mode(GBBLAS_ACCURACY_BF16X6) ? 1.25 : 0.7;
  int best = 1;
  double best_us = 1e30;
  for (int s : {1, 2, 3, 4, 6, 8, 12, 16}) {
    if (s > 1 && stages < 4 * s) break;
    const int64_t waves = (tiles * s + sms - 1) / sms;
    const double us = (double)waves * (double)((stages + s - 1) / s) * stage_us +
                      (s > 1 ? 3.0 + (double)(s + 1) * (double)M * (double)N * 4.0 / 3e6 : 0.0);
    if (us < (s > 1 ? 0.9 : 1.0) * best_us) {  // (each step up has to be worth 10 %)
      best_us = us;
      best = s;
    }
  }
  return best;
}

TcLaunchOpts tuned_tc_opts(DeviceCtx* c, int mode, const gbblas_gemm_desc& g, cudaStream_t stream) {
  const int64_t M = g.M, N = g.N, K = g.K;
  TcLaunchOpts def;
  if (const char* e = std::getenv("GBBLAS_TC_SPLITK"); e && std::atoi(e) > 0) {
    def.split = std::atoi(e);
    return def;
  }
  def.split = split_parts(c, mode, M, N, K);
  // GBBLAS_TC_PAIR, when set, fixes the CTA form; otherwise the tuner picks it
  // (pairs only where padding M to 256 rows adds at most 10 % of the work, and
  // where C admits them: elsewhere the plan would drop the pairs and the split
  // with them)
  const char* pe = std::getenv("GBBLAS_TC_PAIR");
  const bool pair_env = pe && pe[0];
  def.pair = pair_env ? -1 : 0;
  const bool pairs = !pair_env && mode != tc_mode(GBBLAS_ACCURACY_FP8) && mode != tc_mode(GBBLAS_ACCURACY_FP16X3) &&
                     mode != kTcModeF16Guard && tc_c_on_grid(g) && M >= 256 &&
                     (double)((M + 255) / 256 * 256) <= 1.1 * (double)((M + 127) / 128 * 128);
  if (!pairs) return def;
  Tuner& t = Tuner::get();
  const int bm = log2_bucket(M), bn = log2_bucket(N), bk = log2_bucket(K);
  const uint64_t packed = pack_key(kOpPair, mode, c, bm, bn, bk);
  if (const int m = t.recall(packed); m >= 0) return m == 1 ? TcLaunchOpts{1, 1} : def;
  const std::string key = "gemm_tc|" + device_tag(c) + "|mode" + std::to_string(mode) + "|m" + std::to_string(bm) +
                          "|n" + std::to_string(bn) + "|k" + std::to_string(bk) + "|pair";
  const int v = t.lookup(key);
  if (v >= 0) return t.remember(packed, v) == 1 ? TcLaunchOpts{1, 1} : def;
  if (!t.enabled() || capturing(stream)) return def;
  int64_t m, n, k;
  bucket_shape(bm, bn, bk, m, n, k);
  if (m < 256) return def;
  GemmBench b(c, m, n, k);
  if (!b.ok()) return def;
  const gbblas_gemm_desc d = b.desc();
  float ms[2];
  const TcLaunchOpts cands[2] = {TcLaunchOpts{split_parts(c, mode, m, n, k), 0}, TcLaunchOpts{1, 1}};
  for (int i = 0; i < 2; ++i)
    ms[i] = b.time([&](cudaStream_t s) { return launch_gemm_tc_opts(c, mode, d, cands[i], s); });
  if (ms[0] >= 1e30f && ms[1] >= 1e30f) return def;
  const int best = ms[1] < ms[0] ? 1 : 0;
  t.store(key, best);
  return t.remember(packed, best) == 1 ? cands[1] : def;
}

int tuned_fma_tile(DeviceCtx* c, const gbblas_gemm_desc& g, cudaStream_t stream) {
  if (const char* e = std::getenv("GBBLAS_FMA_TILE"); e && e[0] >= '0' && e[0] <= '6') return e[0] - '0';
  if ((double)g.M * g.N * g.K < 1.0e8) return -1;  // small: the tile-count rule
  // a column-major C runs as its transpose (launch_gemm_fma): tune that
  const bool flip = g.csc != 1 && g.rsc == 1;
  const int64_t M = flip ? g.N : g.M, N = flip ? g.M : g.N, K = g.K;
  const int64_t rsa = flip ? g.csb : g.rsa, csa = flip ? g.rsb : g.csa;
  const int64_t rsb = flip ? g.csa : g.rsb, csb = flip ? g.rsa : g.csb;
  const float *A = flip ? g.B : g.A, *B = flip ? g.A : g.B;
  const bool a_col = rsa == 1 && csa != 1, b_col = rsb == 1 && csb != 1;
  // operands TMA cannot fetch never take its kernels, and are timed with
  // leading dimensions off the 16-byte grid
  const bool tma = sgemm_tma_eligible(M, N, K, A, rsa, csa, B, rsb, csb);
  Tuner& t = Tuner::get();
  const int bm = log2_bucket(M), bn = log2_bucket(N), bk = log2_bucket(K);
  const uint64_t packed = pack_key(kOpFma, (a_col ? 1 : 0) | (b_col ? 2 : 0) | (tma ? 4 : 0), c, bm, bn, bk);
  if (const int m = t.recall(packed); m >= 0) return m;
  const std::string key = "gemm_fma_tile|" + device_tag(c) + "|m" + std::to_string(bm) + "|n" + std::to_string(bn) +
                          "|k" + std::to_string(bk) + (a_col ? "|ac" : "|ar") + (b_col ? "|bc" : "|br") +
                          (tma ? "|t" : "|u") + "|f32";
  const int v = t.lookup(key);
  if (v >= 0) return t.remember(packed, v);
  if (!t.enabled() || capturing(stream)) return -1;
  int64_t m, n, k;
  bucket_shape(bm, bn, bk, m, n, k);
  GemmBench b(c, m, n, k, a_col, b_col, tma ? 0 : 1);
  if (!b.ok()) return -1;
  const gbblas_gemm_desc d = b.desc();
  // 5 / 6 = 64 x 64 / 128 x 128 CTA tiles, K cut over the CTAs of a cluster
  // where they leave SMs idle; 2 = TMA-fed 128 x 128, 3 = TMA-fed stream-K,
  // offered where whole tiles fill the SMs badly, 4 = TMA-fed cluster pairs,
  // offered where two CTAs per tile fill the SMs in one wave
  std::vector<int> tiles{5, 6};
  if (tma) {
    tiles.push_back(2);
    if (sgemm_tma_streamk_useful(c, m, n, k)) tiles.push_back(3);
    if (sgemm_tma_pairs_useful(c, m, n, k)) tiles.push_back(4);
  }
  int best = -1;
  float best_ms = 1e30f;
  for (int tile : tiles) {
    const float ms = b.time([&](cudaStream_t s) {
      return launch_gemm_fma<float>(c, d.M, d.N, d.K, d.A, d.rsa, d.csa, d.B, d.rsb, d.csb, d.C, d.rsc, d.csc, s, 0,
                                    tile);
    });
    if (ms < best_ms) {
      best_ms = ms;
      best = tile;
    }
  }
  if (best < 0) return -1;
  t.store(key, best);
  return t.remember(packed, best);
}

}  // namespace gbblas
