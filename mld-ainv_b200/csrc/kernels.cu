// sm_100a kernels for the factor sweeps of the AINV apply and the A SpMV.
//
// Layout: 32-row slices (see internal.h).  One warp owns one slice, one lane
// one row; slot k of a slice is a 32-wide contiguous run of values, so each
// value load of the warp is one coalesced 256 B (FP64) request.  Slices of
// stencil-derived factors store one shared list of column offsets instead of
// per-entry indices, so the streamed bytes are essentially the values alone
// and the gathers of a warp are contiguous.  Factor values are read exactly
// once per apply and use the streaming (evict-first) hint, so the gathered
// vectors (x and t: 64 MB at n = 8M, inside the 126 MB L2) stay resident
// between the two sweeps.
//
// Epilogues are fused: sweep 1 writes t = D^-1 .* (W^T x), sweep 2 writes
// y = alpha*Z t + beta*y, so the reference's three passes
// (src/impl/mld_d_base_ainv_solver_apply_vect.f90:114-119) become two.
// `stop` (optional) is a device flag set by the Krylov loop once it has
// converged; kernels launched after that return immediately.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <map>
#include <utility>

#include "stream.cuh"

namespace ainv {
namespace {

using namespace dev;

// Slices [s0, s1) of a sweep (all of them, or a range of the host-array
// pipeline).  HBM-bound: at 200^3 in FP64 sweep 1 moves 453 MB and sweep 2 389 MB,
// together in 134-140 us on different boards, 6.0-6.3 TB/s (a copy: 6.5).
template <class V, class T, int P, int K>
__global__ void __launch_bounds__(kBlock, info_blocks<V, K>())
    k_sweep_dscale(InfoView<V> m, const double *x, const V *d, T *t, int s0, int s1,
                   const int *stop) {
  for_each_info<P, K>(
      m, x, s0, s1, [&] { return !stop || !ld_now(stop); }, [&](int row) { return ldd_now(d + row); },
      [&](int row, auto acc, auto dr) { t[row] = (T)(dr * acc); }, [](int) {});
}

// Every sweep-2 epilogue (here and in the host-array pipeline kernel) uses
// axpby_row, so all forms give the same bits.
template <class V, class T, int P, int K>
__global__ void __launch_bounds__(kBlock, info_blocks<V, K>())
    k_sweep_axpby(InfoView<V> m, const T *t, double alpha, double beta, double *y, int s0, int s1,
                  const int *stop) {
  for_each_info<P, K>(
      m, t, s0, s1, [&] { return !stop || !ld_now(stop); },
      [&](int row) { return beta == 0.0 ? 0.0 : ld_now(y + row); },
      [&](int row, auto acc, double yr) { y[row] = axpby_row(alpha, (double)acc, beta, yr); },
      [](int) {});
}

// Both sweeps of a small apply in one launch.  Block b owns a tile of slices of
// the second sweep; it computes every row of t that the tile gathers into
// shared memory (Z and W are upper triangular: from the tile's first row to
// `span` rows past its last slice's first), so blocks share nothing and rows of
// t are computed several times over instead of crossing a grid barrier or a
// second launch.  The owner also stores its rows of t, as the sweeps do.
constexpr int kTileBlock = 1024;
constexpr int kTilePack = 4;  // packs up to which there is such a kernel
template <class V, class T, int P, int K>
__global__ void __launch_bounds__(kTileBlock)
    k_apply_tile(InfoView<V> m1, InfoView<V> m2, const double *x, const V *d, T *t, double alpha,
                 double beta, double *y, int tile, int span) {
  using A = typename Acc<V>::type;
  constexpr int kStep = kTileBlock / 32;
  extern __shared__ __align__(16) unsigned char tile_smem[];
  T *tw = reinterpret_cast<T *>(tile_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x * tile, e = min(m1.nslices, a + tile);
  const int lo = a * kSlice, hi = min(m1.n, (e - 1) * kSlice + span + 1);
  const int we = (hi + kSlice - 1) / kSlice;  // window: slices [a, we)
  dep_start();
  InfoSlab<V, P, K> b;
  int4 f = make_int4(0, 0, 0, 0);
  if (a + warp < we) f = __ldg(m1.info + a + warp);
  info_load(m1, f, 0, b);
  dep_wait();
  const auto gx = [&](int c) { return (unsigned)c < (unsigned)m1.n ? ld_now(x + c) : 0.0; };
  for (int s = a + warp; s < we; s += kStep) {
    const int row = s * kSlice + lane;
    const A dr = ldd_now(d + min(row, m1.n - 1));
    int4 fn = f;
    if (s + kStep < we) fn = __ldg(m1.info + s + kStep);
    A acc = A(0);
    info_sum<double>(b, f.w ? row : 0, gx, acc);
    for (int k0 = K; k0 < f.z; k0 += K) {
      info_load(m1, f, k0, b);
      info_sum<double>(b, f.w ? row : 0, gx, acc);
    }
    f = fn;
    if (s + kStep < we) info_load(m1, f, 0, b);
    if (row < hi) {
      const T tr = (T)(dr * acc);
      tw[row - lo] = tr;
      if (s < e) t[row] = tr;
    }
  }
  const int s = a + warp;
  if (s < e) {
    f = __ldg(m2.info + s);
    info_load(m2, f, 0, b);
  }
  __syncthreads();
  const auto gt = [&](int c) {
    const int i = c - lo;
    return (unsigned)i < (unsigned)(hi - lo) ? tw[i] : T(0);
  };
  for (int q = s; q < e; q += kStep) {
    const int row = q * kSlice + lane;
    if (q != s) {
      f = __ldg(m2.info + q);
      info_load(m2, f, 0, b);
    }
    const double yr = beta == 0.0 ? 0.0 : ld_now(y + min(row, m2.n - 1));
    A acc = A(0);
    info_sum<T>(b, f.w ? row : 0, gt, acc);
    for (int k0 = K; k0 < f.z; k0 += K) {
      info_load(m2, f, k0, b);
      info_sum<T>(b, f.w ? row : 0, gt, acc);
    }
    if (row < m2.n) y[row] = axpby_row(alpha, (double)acc, beta, yr);
  }
}

inline int check_launch(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s launch failed: %s", what, cudaGetErrorString(e));
    return AINV_ERR_CUDA;
  }
  return AINV_SUCCESS;
}

}  // namespace

namespace dev {
int sm_count() {
  static int sms[64] = {};
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) d = 0;
  if (sms[d] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || v <= 0)
      v = 148;
    sms[d] = v;
  }
  return sms[d];
}

bool set_smem_attr(const void *kernel, size_t bytes) {
  // opt in to the dynamic shared memory this launch needs (kept per kernel
  // and device); a refusal leaves no error pending and reports false
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> granted;
  int d = 0;
  cudaGetDevice(&d);
  std::lock_guard<std::mutex> lock(mu);
  size_t &g = granted[{kernel, d}];
  if (bytes <= g || bytes <= 48 * 1024) return true;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  g = bytes;
  return true;
}

int stream_plan(const DevSell &m, int xs, int nrv, StreamLayout &L, size_t &smem_bytes) {
  if (m.nstages <= 0 || !m.stages || m.stage_slices <= 0) return 0;
  if (m.stage_slices % kConsumerWarps != 0 || m.stage_slices > kMaxStageSlices) return 0;
  auto r128 = [](long long b) { return (int)((b + 127) / 128 * 128); };
  L.R = m.stage_slices / kConsumerWarps;
  L.vb = r128(m.stage_vmax);
  L.ib = r128(m.stage_imax);
  // a window: the stage's rows, its offset cluster's span and granule slack
  L.xw = (int)(((long long)(m.stage_slices * kSlice + kWindowSpan) * xs + 32 + 15) / 16 * 16);
  L.nwin = m.stage_nwin_max;
  L.nrv = std::max(0, std::min(kMaxRowVecs, nrv));
  L.rw = (int)(((long long)m.stage_slices * kSlice * 8 + 15) / 16 * 16);
  L.stage = r128((long long)kHeaderBytes + L.vb + L.ib + (long long)L.nwin * L.xw +
                 (long long)L.nrv * L.rw);
  if (L.stage > kStreamStageMax) return 0;
  // shared memory per block (tunable: AINV_STREAM_SMEM_KB); a smaller budget
  // means fewer buffers per block but more blocks (producers) per SM
  static const int budget = [] {
    const char *e = std::getenv("AINV_STREAM_SMEM_KB");
    const int v = e ? std::atoi(e) : 0;
    return v >= 16 && v <= 220 ? v * 1024 : kStreamBlockBudget;
  }();
  L.D = std::max(2, std::min(8, budget / L.stage));
  smem_bytes = 128 + (size_t)L.D * L.stage;
  if (smem_bytes > (size_t)kStreamSmemMax) return 0;
  const int per_sm = std::max(1, std::min(4, (int)(kStreamSmemSM / (smem_bytes + 1024))));
  return std::min(m.nstages, per_sm * sm_count());
}

int wave_grid(const void *kernel, long long rows) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, int> cache;
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) d = 0;
  int wave;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find({d, kernel});
    if (it != cache.end()) {
      wave = it->second;
    } else {
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0) !=
              cudaSuccess ||
          per_sm <= 0) {
        cudaGetLastError();
        per_sm = 1;
      }
      wave = per_sm * sm_count();
      cache[{d, kernel}] = wave;
    }
  }
  const long long units = (rows + kBlock - 1) / kBlock;
  return (int)std::max(1LL, std::min(units, (long long)wave));
}

int reduction_grid(long long rows) {
  static int sms[64] = {};
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) d = 0;
  if (sms[d] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || v <= 0)
      v = 148;
    sms[d] = v;
  }
  const long long units = (rows + kBlock - 1) / kBlock;
  const long long wave = 8LL * sms[d];
  return (int)std::max(1LL, std::min(units, wave));
}
}  // namespace dev

namespace {

template <class V, class T>
struct DscaleLaunch {
  const DevSell &m;
  const void *d;
  const double *x;
  void *t;
  int s0, s1;
  cudaStream_t s;
  const int *stop;
  template <int P, int K>
  void run() const {
    auto kern = k_sweep_dscale<V, T, P, K>;
    launch_dep(kern, wave_grid((const void *)kern, (long long)(s1 - s0) * kSlice), kBlock, 0, s,
           info_view<V>(m), x, (const V *)d, (T *)t, s0, s1, stop);
  }
};

template <class V, class T>
struct AxpbyLaunch {
  const DevSell &m;
  const void *t;
  double alpha, beta;
  double *y;
  int s0, s1;
  cudaStream_t s;
  const int *stop;
  template <int P, int K>
  void run() const {
    auto kern = k_sweep_axpby<V, T, P, K>;
    launch_dep(kern, wave_grid((const void *)kern, (long long)(s1 - s0) * kSlice), kBlock, 0, s,
           info_view<V>(m), (const T *)t, alpha, beta, y, s0, s1, stop);
  }
};

template <class V, class T>
struct TileLaunch {
  const ainv_handle *h;
  const DevSell &m1, &m2;
  double alpha, beta;
  const double *x;
  double *y;
  int tile, window;  // slices
  cudaStream_t s;
  template <int P>
  void run() const {
    if constexpr (P <= kTilePack)
      launch_dep(k_apply_tile<V, T, P, 4>, (m1.nslices + tile - 1) / tile, kTileBlock,
                 sizeof(T) * kSlice * (size_t)window, s, info_view<V>(m1), info_view<V>(m2), x,
                 (const V *)h->d, (T *)h->t, alpha, beta, y, tile, m2.span);
  }
};

// Storage type V and intermediate type T of a precision, as a tag.
template <class V_, class T_>
struct Types {
  using V = V_;
  using T = T_;
};
template <class F>
int by_prec(int prec, F &&f) {
  switch (prec) {
    case AINV_PREC_FP64: f(Types<double, double>()); break;
    case AINV_PREC_FP32: f(Types<float, float>()); break;
    case AINV_PREC_BF16: f(Types<__nv_bfloat16, float>()); break;
    case AINV_PREC_FP32_ACC64: f(Types<f32w, double>()); break;
    case AINV_PREC_BF16_ACC64: f(Types<b16w, double>()); break;
    default:
      set_error("unknown precision %d", prec);
      return AINV_ERR_ARG;
  }
  return AINV_SUCCESS;
}

int check_range(const DevSell &m, int s0, int s1) {
  if (s0 < 0 || s1 > m.nslices || s0 > s1) {
    set_error("slice range [%d, %d) invalid for %d slices", s0, s1, m.nslices);
    return AINV_ERR_ARG;
  }
  return AINV_SUCCESS;
}

int sweep_dscale(const DevSell &m, const void *d, const double *x, void *t, int s0, int s1,
                 cudaStream_t s, const int *stop, const char *what) {
  if (s0 == s1) return AINV_SUCCESS;
  AINV_TRY(by_prec(m.prec, [&](auto ty) {
    using Ty = decltype(ty);
    with_info<typename Ty::V>(
        m, DscaleLaunch<typename Ty::V, typename Ty::T>{m, d, x, t, s0, s1, s, stop});
  }));
  return check_launch(what);
}

int sweep_axpby(const DevSell &m, const void *t, double alpha, double beta, double *y, int s0,
                int s1, cudaStream_t s, const int *stop, const char *what) {
  if (s0 == s1) return AINV_SUCCESS;
  AINV_TRY(by_prec(m.prec, [&](auto ty) {
    using Ty = decltype(ty);
    with_info<typename Ty::V>(m, AxpbyLaunch<typename Ty::V, typename Ty::T>{
                                     m, t, alpha, beta, y, s0, s1, s, stop});
  }));
  return check_launch(what);
}

}  // namespace

int launch_sweep_dscale(const DevSell &m, const void *d, const double *x, void *t,
                        cudaStream_t s, const int *stop) {
  return sweep_dscale(m, d, x, t, 0, m.nslices, s, stop, "sweep_dscale");
}

int launch_sweep_axpby(const DevSell &m, const void *t, double alpha, double beta,
                       double *y, cudaStream_t s, const int *stop) {
  return sweep_axpby(m, t, alpha, beta, y, 0, m.nslices, s, stop, "sweep_axpby");
}

int launch_sweep_dscale_slices(const DevSell &m, const void *d, const double *x, void *t,
                               int s0, int s1, cudaStream_t s) {
  AINV_TRY(check_range(m, s0, s1));
  return sweep_dscale(m, d, x, t, s0, s1, s, nullptr, "sweep_dscale (slices)");
}

int launch_sweep_axpby_slices(const DevSell &m, const void *t, double alpha, double beta,
                              double *y, int s0, int s1, cudaStream_t s) {
  AINV_TRY(check_range(m, s0, s1));
  return sweep_axpby(m, t, alpha, beta, y, s0, s1, s, nullptr, "sweep_axpby (slices)");
}

int launch_spmv(const DevSell &a, double alpha, const double *x, double beta, double *y,
                cudaStream_t s) {
  if (a.prec != AINV_PREC_FP64) {
    set_error("operator A must be stored in FP64");
    return AINV_ERR_ARG;
  }
  return sweep_axpby(a, x, alpha, beta, y, 0, a.nslices, s, nullptr, "spmv");
}

// Slices of t that a block of k_apply_tile computes at most: four rounds of
// its 32 warps.  GPU time here / as two launches, FP64: 24^3 (22 slices) 2.3 /
// 3.9 us, 40^3 (64) 3.3 / 4.9, 46^3 (88) 4.1 / 5.1, 52^3 (115) 5.0 / 5.7; and a
// launch less costs the host 1.8 us less per call.  Rows of more than 4 entries
// are not worth computing several times: INVK(1,1) at 24^3 8.5 / 6.5, at 40^3
// 19.4 / 9.7.
constexpr int kTileWindow = 128;

// An apply whose tiles (one per SM) gather few enough rows of t goes out as
// one launch.  x and y must not overlap: a block reads rows of x that another
// one owns.  A BF16 matrix without entries has pack 8 and width 0; it takes
// the two sweeps.
static bool apply_tile(const ainv_handle *h, const DevSell &m1, const DevSell &m2, double alpha,
                       const double *x, double beta, double *y, cudaStream_t s) {
  const int tile = (m1.nslices + sm_count() - 1) / sm_count();
  const long long window = (long long)tile + m2.span / kSlice + 1;
  if (window > kTileWindow || m1.pack != m2.pack || m1.pack > kTilePack || m1.wmax > 4 ||
      m2.wmax > 4)
    return false;
  const uintptr_t xa = (uintptr_t)x, ya = (uintptr_t)y, nb = sizeof(double) * (uintptr_t)h->n;
  if (xa < ya + nb && ya < xa + nb) return false;
  by_prec(m1.prec, [&](auto ty) {
    using Ty = decltype(ty);
    with_pack<typename Ty::V>(m1.pack, TileLaunch<typename Ty::V, typename Ty::T>{
                                           h, m1, m2, alpha, beta, x, y, tile, (int)window, s});
  });
  return true;
}

int ainv_apply_async(const ainv_handle *h, char trans, double alpha, const double *x,
                     double beta, double *y, cudaStream_t s, const int *stop) {
  bool tr = false;
  switch (trans) {
    case 'N': case 'n': break;
    case 'T': case 't': case 'C': case 'c': tr = true; break;
    default:
      // psb_err_iarg_invalid_i_ (src/impl/mld_d_base_ainv_solver_apply_vect.f90:64-71)
      set_error("invalid trans '%c'", trans);
      return AINV_ERR_ARG;
  }
  const DevSell &m1 = tr ? h->zt : h->wt, &m2 = tr ? h->w : h->z;
  if (!stop && apply_tile(h, m1, m2, alpha, x, beta, y, s)) return check_launch("apply");
  AINV_TRY(launch_sweep_dscale(m1, h->d, x, h->t, s, stop));
  return launch_sweep_axpby(m2, h->t, alpha, beta, y, s, stop);
}

}  // namespace ainv
