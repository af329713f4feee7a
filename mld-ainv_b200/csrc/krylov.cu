// Krylov loop on the device: preconditioned CG and BiCGSTAB in the form of
// PSBLAS psb_dcg / psb_dbicgstab with istop=2 (stop when ||r|| <= eps*||b||),
// as driven at tests/pdegen/ppde3d.f90:280-281.
//
// Small systems run as one persistent kernel (persist.cuh); what follows is
// the form of the larger ones.  Both give the same iterates.
//
// Every scalar of the recurrence (rho, alpha, omega, beta, norms, status)
// lives in device memory and is produced by the fold kernel that completes
// the corresponding reduction, so one iteration is a fixed sequence of
// launches with no host round trip.  Iterations are issued in chunks
// captured once into a CUDA graph; when the loop has converged (or broken
// down) a device flag makes every later kernel of the chunk return at once,
// and the host inspects the state once per chunk.
//
// Reproducible iterates.  Every dot is summed in the canonical order of
// sell_device.cuh (slice trees, groups of 8 slices, ranges of 256 groups,
// then the ranges),
// which does not depend on the grid, the kernel that computes the products
// or the device: the producing kernel stores one sum per 32-row slice and a
// small fold kernel (k_fold) reduces them.  The library is compiled without
// floating-point contraction, so every FP64 product and sum of the vector
// updates rounds once, as in the reference's Fortran on a target without
// fused multiply-add, and the row sums of the sweeps and of A use the same
// unfused order (madd).  With FP64 factors the iterates therefore equal,
// bit for bit, those of the oracle's ordered-dot Krylov loop.
//
// Fused steps: the A product and the dots that consume it (p.q, rt.v, t.t
// and t.s) share one kernel; the Z sweep of the preconditioner and the CG
// dot r.z share one kernel; x/r updates and the residual norm (plus rt.r
// for BiCGSTAB) share one kernel.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "kstate.cuh"
#include "krylov_epi.cuh"
#include "persist.cuh"

namespace ainv {

constexpr int kRecheck = 50;  // true-residual period for FP32/BF16 factors

namespace {

using namespace dev;
using namespace kstate;

// Iterations per captured graph launch: a divisor of the true-residual period.
constexpr int kChunk = 10;
static_assert(kRecheck % kChunk == 0, "periodic checks fall on chunk ends");
constexpr int kHistCap = 8192;  // iterations whose residual is recorded
// Arrival counters of the persistent loop, on cache lines of their own.
constexpr int kBarLine = 32, kBarWords = 2 * kBarLine;
constexpr int kPersistIters = 1024;  // iterations per launch of it

// Where a reduction kernel stores its sums: dot k of slice s at sp[k*ld + s].
struct SliceOut {
  double *sp;
  int ld, ns;
};

// ---- the fold ----------------------------------------------------------------
// Block j takes range j (kFoldRange groups of 8 slices): thread t forms the
// sum of group t from its 8 slice sums in slice order, the block folds
// them (block_sum) and stores the range sum; the last block to finish
// (atomic ticket, no waiting) folds the range sums and hands the totals to
// fin.  fin.skip(st) repeats the producing kernel's early-exit test, so a
// reduction that did not run is not folded.
template <int NV, class Fin>
__global__ void __launch_bounds__(kFoldThreads)
    k_fold(const double *sp, int ld, int ns, int ng, double *rs, int ldr, KState *st, Fin fin) {
  dep_start();
  dep_wait();
  if (fin.skip(st)) return;
  __shared__ bool is_last;
  const int nr = gridDim.x;
  double v[NV];
  fold_range<NV>(sp, ld, ns, ng, blockIdx.x, v);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) rs[(size_t)k * ldr + blockIdx.x] = v[k];
    __threadfence();
    is_last = atomicAdd(&st->ticket[3], 1u) == (unsigned)nr - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  fold_total<NV>(rs, ldr, nr, v);
  if (threadIdx.x == 0) {
    st->ticket[3] = 0u;
    fin(st, v);
  }
}

// Early-exit test of the reductions that stop once the loop is done.
struct UntilDone {
  __device__ __forceinline__ bool skip(const KState *st) const { return st->done != 0; }
};

struct FinBnorm {
  __device__ __forceinline__ bool skip(const KState *) const { return false; }
  __device__ __forceinline__ void operator()(KState *st, const double (&v)[1]) const {
    const double bn = sqrt(v[0]);
    st->bn2 = (bn == 0.0) ? 1.0 : bn;
  }
};

__device__ __forceinline__ bool true_res_verify(const KState *st) {
  return st->done && st->status == AINV_SUCCESS && !st->verified;
}
__device__ __forceinline__ bool true_res_periodic(const KState *st) {
  return !st->done && st->check_every > 0 && st->iter > 0 && st->iter % st->check_every == 0;
}

// Scalar step of an SpMV-with-dots reduction (w2: rt for BiCGSTAB, else
// null, as finish_dots expects).
template <int MODE>
struct FinDots {
  const double *w2;
  __device__ __forceinline__ bool skip(const KState *st) const {
    if (MODE == kTrueRes) return !true_res_verify(st) && !true_res_periodic(st);
    return st->done != 0;
  }
  __device__ __forceinline__ void operator()(KState *st, const double (&v)[dots_of(MODE)]) const {
    double pr[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < dots_of(MODE); k++) pr[k] = v[k];
    finish_dots<MODE>(st, pr, MODE == kTrueRes && true_res_verify(st), w2);
  }
};

struct FinCgRho : UntilDone {
  __device__ __forceinline__ void operator()(KState *st, const double (&v)[1]) const {
    cg_take_rho(st, v[0]);
  }
};

struct FinCgXr : UntilDone {
  __device__ __forceinline__ void operator()(KState *st, const double (&v)[1]) const {
    finish_iteration(st, v[0]);
  }
};

struct FinBicgXr : UntilDone {
  __device__ __forceinline__ void operator()(KState *st, const double (&v)[2]) const {
    finish_iteration(st, v[0]);
    bicg_next_rho(st, v[1]);
  }
};

// ---- reduction kernels ---------------------------------------------------------
// Vector-only kernels walk warp-per-slice (lane = row), so the slice trees
// see the same lane order as in the SpMV kernels.
__device__ __forceinline__ int nslices_of(int n) { return (n + kSlice - 1) / kSlice; }

// ||b||_2 (istop=2 denominator).
__global__ void __launch_bounds__(kBlock)
    k_bnorm(int n, const double *b, SliceOut o) {
  dep_start();
  dep_wait();
  SliceSums<1> ss{o.sp, o.ld, {0.0}};
  const int ns = nslices_of(n), lane = threadIdx.x & 31;
  for (int s = first_slice(); s < ns; s += slice_stride()) {
    const int i = s * kSlice + lane;
    if (i < n) ss.v[0] = b[i] * b[i];
    ss.end(s);
  }
}

template <int MODE>
__device__ __forceinline__ bool dots_skip(const KState *st) {
  if (MODE == kTrueRes) return !true_res_verify(st) && !true_res_periodic(st);
  return st->done != 0;
}

template <int MODE, int P, int K>
__global__ void __launch_bounds__(kBlock, info_blocks<double, K>())
    k_spmv_dots(InfoView<double> m, const double *x, double *y, const double *w1, double *w2,
                const double *w3, const KState *st, SliceOut o) {
  SliceSums<dots_of(MODE)> ss{o.sp, o.ld, {}};
  const double *a = dots_operand<MODE>(x, w1);
  for_each_info<P, K>(
      m, x, 0, m.nslices, [&] { return !dots_skip<MODE>(st); }, [&](int i) { return a[i]; },
      [&](int i, double acc, double ai) { dots_row<MODE>(i, acc, ai, y, w2, w3, ss); },
      [&](int s) { ss.end(s); });
}

// r := b - A x when the last true-residual check asked for it.
__global__ void __launch_bounds__(kBlock)
    k_replace_r(int n, const double *rtrue, double *r, const KState *st) {
  dep_start();
  dep_wait();
  if (!st->replace) return;
  for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) r[i] = rtrue[i];
}

// CG: z = Z t (sweep 2 of the AINV apply) fused with rho = r.z.
template <class V, class T, int P, int K>
__global__ void __launch_bounds__(kBlock, info_blocks<V, K>())
    k_cg_sweep2(InfoView<V> m, const T *t, const double *r, double *z, const KState *st,
                SliceOut o) {
  SliceSums<1> ss{o.sp, o.ld, {0.0}};
  for_each_info<P, K>(
      m, t, 0, m.nslices, [&] { return !st->done; }, [&](int i) { return r[i]; },
      [&](int i, auto acc, double ri) {
        const double zi = (double)acc;
        z[i] = zi;
        ss.v[0] = ri * zi;
      },
      [&](int s) { ss.end(s); });
}

// CG without preconditioner: z = r, rho = r.r.
__global__ void __launch_bounds__(kBlock)
    k_cg_ident(int n, const double *r, double *z, const KState *st, SliceOut o) {
  dep_start();
  dep_wait();
  if (st->done) return;
  SliceSums<1> ss{o.sp, o.ld, {0.0}};
  const int ns = nslices_of(n), lane = threadIdx.x & 31;
  for (int s = first_slice(); s < ns; s += slice_stride()) {
    const int i = s * kSlice + lane;
    if (i < n) {
      z[i] = r[i];
      ss.v[0] = r[i] * r[i];
    }
    ss.end(s);
  }
}

// CG: p = z (first iteration) or p = z + beta p.
__global__ void __launch_bounds__(kBlock)
    k_cg_p(int n, const double *z, double *p, const KState *st) {
  dep_start();
  dep_wait();
  if (st->done) return;
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  p[i] = (st->iter == 0) ? z[i] : z[i] + st->beta * p[i];
}

// CG: x += alpha p, r -= alpha q, rn2 = r.r.
__global__ void __launch_bounds__(kBlock)
    k_cg_xr(int n, const double *p, const double *q, double *x, double *r, const KState *st,
            SliceOut o) {
  dep_start();
  dep_wait();
  if (st->done) return;
  const double alpha = st->alpha;
  SliceSums<1> ss{o.sp, o.ld, {0.0}};
  const int ns = nslices_of(n), lane = threadIdx.x & 31;
  for (int s = first_slice(); s < ns; s += slice_stride()) {
    const int i = s * kSlice + lane;
    if (i < n) {
      x[i] = x[i] + alpha * p[i];
      const double ri = r[i] - alpha * q[i];
      r[i] = ri;
      ss.v[0] = ri * ri;
    }
    ss.end(s);
  }
}

// BiCGSTAB: p = r (first iteration) or p = r + beta (p - omega v).
__global__ void __launch_bounds__(kBlock)
    k_bicg_p(int n, const double *r, const double *v, double *p, const KState *st) {
  dep_start();
  dep_wait();
  if (st->done) return;
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  p[i] = (st->iter == 0) ? r[i] : r[i] + st->beta * (p[i] - st->omega * v[i]);
}

// BiCGSTAB: s = r - alpha v.
__global__ void __launch_bounds__(kBlock)
    k_bicg_s(int n, const double *r, const double *v, double *s, const KState *st) {
  dep_start();
  dep_wait();
  if (st->done) return;
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  s[i] = r[i] - st->alpha * v[i];
}

// BiCGSTAB: x += alpha f + omega z, r = s - omega t, rn2 = r.r, rho' = rt.r.
__global__ void __launch_bounds__(kBlock)
    k_bicg_xr(int n, const double *f, const double *z, const double *s, const double *t,
              const double *rt, double *x, double *r, const KState *st, SliceOut o) {
  dep_start();
  dep_wait();
  if (st->done) return;
  const double alpha = st->alpha, omega = st->omega;
  SliceSums<2> ss{o.sp, o.ld, {0.0, 0.0}};
  const int ns = nslices_of(n), lane = threadIdx.x & 31;
  for (int sl = first_slice(); sl < ns; sl += slice_stride()) {
    const int i = sl * kSlice + lane;
    if (i < n) {
      x[i] = (x[i] + alpha * f[i]) + omega * z[i];
      const double ri = s[i] - omega * t[i];
      r[i] = ri;
      ss.v[0] = ri * ri;
      ss.v[1] = rt[i] * ri;
    }
    ss.end(sl);
  }
}


template <class V, class T>
struct CgSweep2Launch {
  const DevSell &m;
  const void *t;
  const double *r;
  double *z;
  KState *st;
  SliceOut o;
  cudaStream_t s;
  template <int P, int K>
  void run() const {
    auto kern = k_cg_sweep2<V, T, P, K>;
    launch_dep(kern, wave_grid((const void *)kern, m.n), kBlock, 0, s, info_view<V>(m), (const T *)t,
           r, z, st, o);
  }
};

template <class V, class T>
void launch_cg_sweep2(const DevSell &m, const void *t, const double *r, double *z, KState *st,
                      SliceOut o, cudaStream_t s) {
  with_info<V>(m, CgSweep2Launch<V, T>{m, t, r, z, st, o, s});
}

template <int MODE>
struct SpmvDotsLaunch {
  const DevSell &A;
  cudaStream_t s;
  const double *x;
  double *y;
  const double *w1;
  double *w2;
  const double *w3;
  KState *st;
  SliceOut pp;
  template <int P, int K>
  void run() const {
    auto kern = k_spmv_dots<MODE, P, K>;
    launch_dep(kern, wave_grid((const void *)kern, A.n), kBlock, 0, s, info_view<double>(A), x, y, w1,
           w2, w3, st, pp);
  }
};

// y = A x with the dots of MODE.
template <int MODE>
void spmv_dots(const DevSell &A, cudaStream_t s, const double *x, double *y, const double *w1,
               double *w2, const double *w3, KState *st, SliceOut pp) {
  with_info<double>(A, SpmvDotsLaunch<MODE>{A, s, x, y, w1, w2, w3, st, pp});
}

std::atomic<unsigned long long> g_serial{1};

// What the host reads of a loop: its state, and the persistent loop's abort word.
struct LoopState {
  KState k;
  int abort;
};

}  // namespace

unsigned wait_limit_us() {
  const char *e = std::getenv("AINV_WAIT_MS");
  const long long ms = e ? std::atoll(e) : 2000;
  return (unsigned)(std::min(std::max(ms, 0ll), 1000000ll) * 1000);
}

unsigned long long next_serial() { return g_serial.fetch_add(1); }

// ------------------------------------------------------------ workspace --
struct KrylovWs {
  int n = 0, G = 0;
  size_t stride = 0;      // doubles between vectors (n rounded up to 32: 256 B aligned)
  char *mem = nullptr, *hmem = nullptr;  // one device and one page-locked allocation
  double *vec = nullptr;  // 11 vectors of n
  // canonical-order reductions: up to 3 dots' slice sums (ld per dot) and
  // range sums (ldr per dot)
  int ns = 0, ng = 0, ld = 0, nr = 0, ldr = 0;
  double *sp = nullptr, *rs = nullptr;
  // relative residual per iteration of the last solve (device, host copy)
  double *hist = nullptr;
  double *hist_h = nullptr;  // page-locked
  std::vector<double> hhist;
  int hcount = 0;
  // persistent loop: two arrival counters used in turn
  unsigned *bar = nullptr;
  unsigned turn = 0;
  LoopState *loop = nullptr;
  KState *st = nullptr;       // &loop->k
  LoopState *hloop = nullptr;  // page-locked mirror
  KState *hst = nullptr;      // &hloop->k
  cudaStream_t s = nullptr;
  cudaEvent_t ev = nullptr;
  cudaGraphExec_t exec = nullptr;
  unsigned long long key_serial = 0;
  int key_method = -1;
  bool key_each = false;
  KState last{};  // final state of the last solve (statistics)
  double *v(int i) const { return vec + (size_t)i * stride; }
  SliceOut out() const { return SliceOut{sp, ld, ns}; }
  // Fold the slice sums of the reduction just enqueued (NV dots).
  template <int NV, class Fin>
  void fold(const Fin &fin) const {
    launch_dep(k_fold<NV, Fin>, nr, kFoldThreads, 0, s, sp, ld, ns, ng, rs, ldr, st, fin);
  }
};

void destroy_ws(KrylovWs *w) {
  if (!w) return;
  if (w->exec) cudaGraphExecDestroy(w->exec);
  if (w->mem) cudaFree(w->mem);
  if (w->hmem) cudaFreeHost(w->hmem);
  if (w->ev) cudaEventDestroy(w->ev);
  if (w->s) cudaStreamDestroy(w->s);
  delete w;
}

namespace {

enum { XW = 0, BW, R, RT, P, V_, F, S, Z, T_, RTRUE, kNumVec };

int get_ws(ainv_csr *a, KrylovWs **out) {
  if (a->ws) {
    *out = a->ws;
    return AINV_SUCCESS;
  }
  KrylovWs *w = new (std::nothrow) KrylovWs;
  if (!w) {
    set_error("krylov workspace: host allocation failed");
    return AINV_ERR_ALLOC;
  }
  w->n = a->n;
  w->stride = ((size_t)a->n + 31) / 32 * 32;
  w->G = reduction_grid(a->n);
  w->ns = (a->n + kSlice - 1) / kSlice;
  w->ld = (w->ns + 31) / 32 * 32;
  w->ng = (w->ns + kGroupSlices - 1) / kGroupSlices;
  w->nr = (w->ng + kFoldRange - 1) / kFoldRange;
  w->ldr = (w->nr + 31) / 32 * 32;
  size_t at = 0;
  auto part = [&at](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) / 256 * 256;
    return o;
  };
  const size_t vec = part(sizeof(double) * kNumVec * w->stride);
  const size_t sp = part(sizeof(double) * 3 * (size_t)w->ld);
  const size_t rs = part(sizeof(double) * 3 * (size_t)w->ldr);
  const size_t hist = part(sizeof(double) * kHistCap);
  const size_t bar = part(sizeof(unsigned) * kBarWords), loop = part(sizeof(LoopState));
  cudaError_t e = cudaMalloc(&w->mem, at);
  w->vec = reinterpret_cast<double *>(w->mem + vec);
  w->sp = reinterpret_cast<double *>(w->mem + sp);
  w->rs = reinterpret_cast<double *>(w->mem + rs);
  w->hist = reinterpret_cast<double *>(w->mem + hist);
  w->bar = reinterpret_cast<unsigned *>(w->mem + bar);
  w->loop = reinterpret_cast<LoopState *>(w->mem + loop);
  w->st = &w->loop->k;
  const size_t hh = (sizeof(LoopState) + 255) / 256 * 256;
  if (e == cudaSuccess) e = cudaMallocHost(&w->hmem, hh + sizeof(double) * kHistCap);
  w->hloop = reinterpret_cast<LoopState *>(w->hmem);
  w->hst = &w->hloop->k;
  w->hist_h = reinterpret_cast<double *>(w->hmem + hh);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&w->s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(w->mem, 0, at, w->s);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w->ev, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    destroy_ws(w);
    set_error("krylov workspace allocation failed: %s", cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? AINV_ERR_ALLOC : AINV_ERR_CUDA;
  }
  a->ws = w;
  *out = w;
  return AINV_SUCCESS;
}

void precond_sweep2_cg(const ainv_handle *h, const double *r, double *z, KState *st,
                       SliceOut o, cudaStream_t s) {
  switch (h->prec) {
    case AINV_PREC_FP64: return launch_cg_sweep2<double, double>(h->z, h->t, r, z, st, o, s);
    case AINV_PREC_FP32: return launch_cg_sweep2<float, float>(h->z, h->t, r, z, st, o, s);
    case AINV_PREC_FP32_ACC64: return launch_cg_sweep2<f32w, double>(h->z, h->t, r, z, st, o, s);
    case AINV_PREC_BF16_ACC64: return launch_cg_sweep2<b16w, double>(h->z, h->t, r, z, st, o, s);
    default: return launch_cg_sweep2<__nv_bfloat16, float>(h->z, h->t, r, z, st, o, s);
  }
}

// One iteration, enqueued on ws->s.  Kernels ending in a reduction run on
// the reduction grid G (one resident wave, grid-stride loops); the plain
// vector updates use one thread per row.  check: with the true-residual check
// (three launches that return at once unless convergence is claimed or the
// period has passed).
int enqueue_iteration(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, int method,
                      bool check) {
  const int n = w->n, G = w->G;
  const int Gv = (n + kBlock - 1) / kBlock;
  const DevSell &A = a->a;
  KState *st = w->st;
  const SliceOut pp = w->out();
  cudaStream_t s = w->s;
  const int *stop = &st->done;
  if (method == AINV_KRYLOV_CG) {
    double *r = w->v(R), *z = w->v(Z), *p = w->v(P), *q = w->v(V_), *x = w->v(XW);
    if (h) {
      AINV_TRY(launch_sweep_dscale(h->wt, h->d, r, h->t, s, stop));
      precond_sweep2_cg(h, r, z, st, pp, s);
    } else {
      launch_dep(k_cg_ident, std::min(G, wave_grid((const void *)k_cg_ident, n)), kBlock, 0, s, n, r, z,
             st, pp);
    }
    w->fold<1>(FinCgRho{});
    launch_dep(k_cg_p, Gv, kBlock, 0, s, n, z, p, st);
    spmv_dots<kCgSigma>(A, s, p, q, nullptr, nullptr, nullptr, st, pp);
    w->fold<1>(FinDots<kCgSigma>{nullptr});
    launch_dep(k_cg_xr, std::min(G, wave_grid((const void *)k_cg_xr, n)), kBlock, 0, s, n, p, q, x, r,
           st, pp);
    w->fold<1>(FinCgXr{});
    if (check) {
      spmv_dots<kTrueRes>(A, s, x, w->v(RTRUE), w->v(BW), nullptr, r, st, pp);
      w->fold<3>(FinDots<kTrueRes>{nullptr});
      launch_dep(k_replace_r, wave_grid((const void *)k_replace_r, n), kBlock, 0, s, n,
                 w->v(RTRUE), r, st);
    }
  } else {
    double *r = w->v(R), *rt = w->v(RT), *p = w->v(P), *v = w->v(V_), *f = w->v(F),
           *sv = w->v(S), *z = w->v(Z), *t = w->v(T_), *x = w->v(XW);
    launch_dep(k_bicg_p, Gv, kBlock, 0, s, n, r, v, p, st);
    if (h) {
      AINV_TRY(ainv_apply_async(h, 'N', 1.0, p, 0.0, f, s, stop));
    } else {
      AINV_CUDA_TRY(cudaMemcpyAsync(f, p, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    }
    spmv_dots<kBicgSigma>(A, s, f, v, rt, nullptr, nullptr, st, pp);
    w->fold<1>(FinDots<kBicgSigma>{rt});
    launch_dep(k_bicg_s, Gv, kBlock, 0, s, n, r, v, sv, st);
    if (h) {
      AINV_TRY(ainv_apply_async(h, 'N', 1.0, sv, 0.0, z, s, stop));
    } else {
      AINV_CUDA_TRY(cudaMemcpyAsync(z, sv, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    }
    spmv_dots<kBicgOmega>(A, s, z, t, sv, nullptr, nullptr, st, pp);
    w->fold<2>(FinDots<kBicgOmega>{rt});
    launch_dep(k_bicg_xr, std::min(G, wave_grid((const void *)k_bicg_xr, n)), kBlock, 0, s, n, f, z, sv,
           t, rt, x, r, st, pp);
    w->fold<2>(FinBicgXr{});
    if (check) {
      spmv_dots<kTrueRes>(A, s, x, w->v(RTRUE), w->v(BW), rt, r, st, pp);
      w->fold<3>(FinDots<kTrueRes>{rt});
      launch_dep(k_replace_r, wave_grid((const void *)k_replace_r, n), kBlock, 0, s, n,
                 w->v(RTRUE), r, st);
    }
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("krylov launch failed: %s", cudaGetErrorString(e));
    return AINV_ERR_CUDA;
  }
  return AINV_SUCCESS;
}

// Once the loop is done, nothing of it runs until the check, so a convergence
// claim can wait for the chunk's end; and as long as no check has failed,
// chunks start at multiples of kChunk, so the periodic checks fall on their
// ends.  After a failed claim every iteration is followed by the check.
int enqueue_chunk(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, int method, bool each) {
  for (int k = 0; k < kChunk; k++)
    AINV_TRY(enqueue_iteration(w, h, a, method, each || k == kChunk - 1));
  return AINV_SUCCESS;
}

int ensure_graph(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, int method, bool each) {
  const unsigned long long key = h ? h->serial : 0ull;
  if (w->exec && w->key_serial == key && w->key_method == method && w->key_each == each)
    return AINV_SUCCESS;
  if (w->exec) {
    cudaGraphExecDestroy(w->exec);
    w->exec = nullptr;
  }
  AINV_CUDA_TRY(cudaStreamBeginCapture(w->s, cudaStreamCaptureModeThreadLocal));
  const int rc = enqueue_chunk(w, h, a, method, each);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(w->s, &g);
  if (rc != AINV_SUCCESS) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) {
    set_error("graph capture failed: %s", cudaGetErrorString(e));
    return AINV_ERR_CUDA;
  }
  e = cudaGraphInstantiate(&w->exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    w->exec = nullptr;
    set_error("graph instantiate failed: %s", cudaGetErrorString(e));
    return AINV_ERR_CUDA;
  }
  w->key_serial = key;
  w->key_method = method;
  w->key_each = each;
  return AINV_SUCCESS;
}

// ---- the persistent loop (persist.cuh) -----------------------------------------
int log2i(int v) {
  int l = 0;
  while ((1 << l) < v) l++;
  return l;
}
template <class V>
PMat<V> pmat(const DevSell &m) {
  return PMat<V>{info_view<V>(m), log2i(m.pack)};
}

template <class V, class T, int PK, int K, int METHOD, int MB>
int persist_launch_mb(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, const double *b,
                   double *x, int resume) {
  PArgs<V, T> p;
  p.wt = pmat<V>(h->wt);
  p.z = pmat<V>(h->z);
  p.a = pmat<double>(a->a);
  p.d = (const V *)h->d;
  p.t = (T *)h->t;
  // CG leaves rt and f free, and BiCGSTAB's check needs no vector of its own
  // (it uses the p buffer that the next iteration writes)
  if (METHOD == AINV_KRYLOV_CG)
    p.w = PVecs{w->v(XW), w->v(BW), {w->v(R), w->v(RT)}, nullptr, {w->v(P), w->v(F)},
                w->v(V_), nullptr, nullptr, w->v(Z), nullptr};
  else
    p.w = PVecs{w->v(XW), w->v(BW), {w->v(R), nullptr}, w->v(RT), {w->v(P), w->v(RTRUE)},
                w->v(V_), w->v(F), w->v(S), w->v(Z), w->v(T_)};
  p.xin = x;
  p.bin = b;
  p.xout = x;
  p.gs = w->sp;
  p.n = w->n;
  p.ns = w->ns;
  p.ng = w->ng;
  p.bar = w->bar + (w->turn & 1u) * kBarLine;
  p.bar_next = w->bar + ((w->turn + 1) & 1u) * kBarLine;
  p.abort = &w->loop->abort;
  p.wait_us = wait_limit_us();
  p.st = w->st;
  p.resume = resume;
  p.max_iters = kPersistIters;
  auto kern = k_persist<V, T, PK, K, METHOD, MB>;
  static const int per_sm = [&] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kern, kPBlock, 0) != cudaSuccess) v = 0;
    cudaGetLastError();
    return v;
  }();
  if (per_sm < 1) return AINV_ERR_UNSUPPORTED;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = std::min((w->ng + kPTeams - 1) / kPTeams,
                         std::min(per_sm, MB) * sm_count());
  cfg.blockDim = kPBlock;
  cfg.stream = w->s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) {
    cudaGetLastError();
    return AINV_ERR_UNSUPPORTED;
  }
  w->turn++;
  return AINV_SUCCESS;
}

template <class V, class T, int K, int METHOD>
int persist_launch(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, const double *b,
                   double *x, int resume) {
  constexpr int PK = fast_pack<V, K>();
  const bool one = w->ng <= kPTeams * sm_count();  // a group per team, a block per SM
  if (h->wt.pack == PK && h->z.pack == PK && a->a.pack == 1)
    return one ? persist_launch_mb<V, T, PK, K, METHOD, 1>(w, h, a, b, x, resume)
               : persist_launch_mb<V, T, PK, K, METHOD, 2>(w, h, a, b, x, resume);
  return persist_launch_mb<V, T, 0, K, METHOD, 2>(w, h, a, b, x, resume);
}

template <int K, int METHOD>
int persist_prec(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, const double *b, double *x,
                 int resume) {
  switch (h->prec) {
    case AINV_PREC_FP64: return persist_launch<double, double, K, METHOD>(w, h, a, b, x, resume);
    case AINV_PREC_FP32: return persist_launch<float, float, K, METHOD>(w, h, a, b, x, resume);
    case AINV_PREC_FP32_ACC64: return persist_launch<f32w, double, K, METHOD>(w, h, a, b, x, resume);
    case AINV_PREC_BF16_ACC64: return persist_launch<b16w, double, K, METHOD>(w, h, a, b, x, resume);
    default: return persist_launch<__nv_bfloat16, float, K, METHOD>(w, h, a, b, x, resume);
  }
}

bool narrow_factors(const ainv_handle *h) { return h->wt.wmax <= 4 && h->z.wmax <= 4; }

// Whether a solve runs there: few enough groups per team for its rows' slots.
bool persist_fits(const KrylovWs *w, const ainv_handle *h, const ainv_csr *a) {
  const int teams = kPTeams * 2 * sm_count();
  const long long rounds = (w->ng + teams - 1) / teams, rows = (long long)w->ns * kSlice;
  const int p = fast_pack(prec_size(h->prec), narrow_factors(h));
  const bool fast = h->wt.pack == p && h->z.pack == p && a->a.pack == 1;
  return w->n <= kPMaxRows && rounds <= kPMaxPerTeam &&
         rounds * (h->wt.slots + h->z.slots) <= persist_limit(h->prec, fast) * rows &&
         rounds * a->a.slots <= kPMaxASlots * rows;
}

int persist(KrylovWs *w, const ainv_handle *h, const ainv_csr *a, const double *b, double *x,
            int method, int resume) {
  const bool narrow = narrow_factors(h);
  if (method == AINV_KRYLOV_CG)
    return narrow ? persist_prec<4, AINV_KRYLOV_CG>(w, h, a, b, x, resume)
                  : persist_prec<8, AINV_KRYLOV_CG>(w, h, a, b, x, resume);
  return narrow ? persist_prec<4, AINV_KRYLOV_BICGSTAB>(w, h, a, b, x, resume)
                : persist_prec<8, AINV_KRYLOV_BICGSTAB>(w, h, a, b, x, resume);
}

// What a finished solve reports (state and residuals are in page-locked memory).
int finish_solve(KrylovWs *w, int itmax, int *iter, double *err) {
  const KState &f = *w->hst;
  w->last = f;
  w->hcount = std::min(std::max(f.iter, 0), kHistCap);
  w->hhist.assign(w->hist_h, w->hist_h + w->hcount);
  if (iter) *iter = f.iter;
  if (err) *err = sqrt(f.rn2) / f.bn2;
  if (f.timeout) {
    set_error("a device wait of the Krylov loop ran past its time limit");
    return AINV_ERR_TIMEOUT;
  }
  if (!f.done) {
    set_error("krylov loop did not terminate");
    return AINV_ERR_INTERNAL;
  }
  if (f.status != AINV_SUCCESS) {
    switch (f.status) {
      case AINV_ERR_NOCONV: set_error("itmax (%d) reached, err %.3e", itmax, sqrt(f.rn2) / f.bn2); break;
      case AINV_ERR_BREAKDOWN: set_error("Krylov breakdown at iteration %d", f.iter); break;
      default: set_error("non-finite residual at iteration %d", f.iter); break;
    }
  }
  return f.status;
}

}  // namespace

int krylov_solve(const ainv_handle *h, ainv_csr *a, const double *b, double *x, int method,
                 double eps, int itmax, int replace_every, int *iter, double *err,
                 cudaStream_t user) {
  KrylovWs *w = nullptr;
  AINV_TRY(get_ws(a, &w));
  const int n = w->n;
  const size_t bytes = sizeof(double) * (size_t)n;
  // order after the caller's stream
  AINV_CUDA_TRY(cudaEventRecord(w->ev, user));
  AINV_CUDA_TRY(cudaStreamWaitEvent(w->s, w->ev, 0));
  KState init{};
  init.eps = eps;
  init.itmax = itmax;
  init.check_every = replace_every;
  init.method = method;
  init.hist = w->hist;
  init.hist_cap = kHistCap;
  *w->hloop = LoopState{init, 0};
  AINV_CUDA_TRY(cudaMemcpyAsync(w->loop, w->hloop, sizeof(LoopState), cudaMemcpyHostToDevice, w->s));
  if (h && persist_fits(w, h, a)) {
    for (int resume = 0;; resume = 1) {
      const int rc = persist(w, h, a, b, x, method, resume);
      if (rc == AINV_ERR_UNSUPPORTED && !resume) break;  // no cooperative launch: plain loop
      AINV_TRY(rc);
      AINV_CUDA_TRY(cudaMemcpyAsync(w->hloop, w->loop, sizeof(LoopState), cudaMemcpyDeviceToHost,
                                    w->s));
      AINV_CUDA_TRY(cudaMemcpyAsync(w->hist_h, w->hist,
                                    sizeof(double) * (size_t)std::min(itmax, kHistCap),
                                    cudaMemcpyDeviceToHost, w->s));
      AINV_CUDA_TRY(cudaStreamSynchronize(w->s));
      if (w->hloop->abort) {
        w->hst->timeout = 1;
        AINV_CUDA_TRY(cudaMemsetAsync(w->bar, 0, sizeof(unsigned) * kBarWords, w->s));
      }
      if (w->hst->done || w->hst->timeout) {
        AINV_CUDA_TRY(cudaEventRecord(w->ev, w->s));
        AINV_CUDA_TRY(cudaStreamWaitEvent(user, w->ev, 0));
        return finish_solve(w, itmax, iter, err);
      }
    }
  }
  AINV_CUDA_TRY(cudaMemcpyAsync(w->v(XW), x, bytes, cudaMemcpyDeviceToDevice, w->s));
  AINV_CUDA_TRY(cudaMemcpyAsync(w->v(BW), b, bytes, cudaMemcpyDeviceToDevice, w->s));
  const DevSell &A = a->a;
  launch_dep(k_bnorm, std::min(w->G, wave_grid((const void *)k_bnorm, n)), kBlock, 0, w->s, n, w->v(BW),
         w->out());
  w->fold<1>(FinBnorm{});
  double *rt0 = method == AINV_KRYLOV_BICGSTAB ? w->v(RT) : nullptr;
  spmv_dots<kInit>(A, w->s, w->v(XW), w->v(R), w->v(BW), rt0, nullptr, w->st, w->out());
  w->fold<2>(FinDots<kInit>{rt0});
  AINV_CUDA_TRY(cudaGetLastError());

  // The first chunk always runs as plain launches (kernel attributes are
  // settled outside any capture); later chunks replay one captured graph.
  const bool use_graph = getenv("AINV_NO_GRAPH") == nullptr;
  const long max_chunks = (long)itmax / kChunk + 2 + kMaxVerifyFails;
  for (long c = 0; c < max_chunks; c++) {
    AINV_CUDA_TRY(cudaMemcpyAsync(w->hst, w->st, sizeof(KState), cudaMemcpyDeviceToHost, w->s));
    AINV_CUDA_TRY(cudaStreamSynchronize(w->s));
    if (w->hst->done) break;
    const bool each = w->hst->fails > 0;
    if (use_graph && c > 0) {
      AINV_TRY(ensure_graph(w, h, a, method, each));
      AINV_CUDA_TRY(cudaGraphLaunch(w->exec, w->s));
    } else {
      AINV_TRY(enqueue_chunk(w, h, a, method, each));
    }
  }
  AINV_CUDA_TRY(cudaMemcpyAsync(x, w->v(XW), bytes, cudaMemcpyDeviceToDevice, w->s));
  AINV_CUDA_TRY(cudaMemcpyAsync(w->hst, w->st, sizeof(KState), cudaMemcpyDeviceToHost, w->s));
  AINV_CUDA_TRY(cudaMemcpyAsync(w->hist_h, w->hist,
                                sizeof(double) * (size_t)std::min(itmax, kHistCap),
                                cudaMemcpyDeviceToHost, w->s));
  AINV_CUDA_TRY(cudaStreamSynchronize(w->s));
  AINV_CUDA_TRY(cudaEventRecord(w->ev, w->s));
  AINV_CUDA_TRY(cudaStreamWaitEvent(user, w->ev, 0));
  return finish_solve(w, itmax, iter, err);
}

}  // namespace ainv

extern "C" int ainv_csr_solve_info(const ainv_csr *a, int *verify_fails, int *replacements) {
  if (!a) {
    ainv::set_error("ainv_csr_solve_info: null operator");
    return AINV_ERR_ARG;
  }
  const ainv::KState *s = a->ws ? &a->ws->last : nullptr;
  if (verify_fails) *verify_fails = s ? s->fails : 0;
  if (replacements) *replacements = s ? s->replacements : 0;
  return AINV_SUCCESS;
}

extern "C" int ainv_csr_solve_history(const ainv_csr *a, double *rel_res, int cap,
                                      int *count) {
  if (!a || cap < 0 || (cap > 0 && !rel_res)) {
    ainv::set_error("ainv_csr_solve_history: invalid argument");
    return AINV_ERR_ARG;
  }
  const int have = a->ws ? a->ws->hcount : 0;
  const int k = std::min(have, cap);
  if (k > 0) std::memcpy(rel_res, a->ws->hhist.data(), sizeof(double) * (size_t)k);
  if (count) *count = have;
  return AINV_SUCCESS;
}

extern "C" int ainv_gpu_solve(ainv_handle *h, const ainv_csr *a, const double *b_dev,
                              double *x_dev, int method, double eps, int itmax, int *iter,
                              double *err, void *stream) {
  if (!a || !b_dev || !x_dev) {
    ainv::set_error("ainv_gpu_solve: null argument");
    return AINV_ERR_ARG;
  }
  if (method != AINV_KRYLOV_CG && method != AINV_KRYLOV_BICGSTAB) {
    ainv::set_error("ainv_gpu_solve: unknown method %d", method);
    return AINV_ERR_ARG;
  }
  if (h && h->n != a->n) {
    ainv::set_error("ainv_gpu_solve: preconditioner size %d != operator size %d", h->n, a->n);
    return AINV_ERR_ARG;
  }
  if (!(eps > 0.0) || itmax < 0) {
    ainv::set_error("ainv_gpu_solve: invalid eps/itmax");
    return AINV_ERR_ARG;
  }
  // Every solve confirms convergence on the true residual b - A x.  With
  // FP32/BF16 factors the true residual is also checked every 50 iterations
  // and replaces the recurrence residual if the two have drifted apart.
  const int replace = (h && h->prec != AINV_PREC_FP64) ? ainv::kRecheck : 0;
  return ainv::krylov_solve(h, const_cast<ainv_csr *>(a), b_dev, x_dev, method, eps, itmax,
                            replace, iter, err, (cudaStream_t)stream);
}
