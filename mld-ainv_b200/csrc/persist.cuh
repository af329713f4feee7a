// The Krylov loops as one persistent kernel.
//
// Below about 600,000 rows an iteration is bound by its launches, not
// by its bytes: at 40^3 a CG iteration was 11 launches of 2.3-5.5 us (34 us)
// for 1.7 us of L2 traffic, a BiCGSTAB iteration 20 (52 us).  As phases of
// one kernel they take 11.0 and 18.9 us: per phase about 0.8 us from the
// first gather to the group sums, 1.0 us at the barrier and, where a dot is
// folded, 1.2 us.  Here the blocks of one cooperative grid run whole
// iterations, with a grid barrier where one phase reads what another block
// wrote in the phase before:
//
//   CG        z = Z t, rho | p = z + beta p, q = A p, sigma |
//             x += alpha p, r -= alpha q, ||r||, t = D^-1 W^T r |
//   BiCGSTAB  p = r + beta (p - omega v), t = D^-1 W^T p | f = Z t |
//             v = A f, sigma | s = r - alpha v, t = D^-1 W^T s | z = Z t |
//             t' = A z, omega | x += alpha f + omega z, r = s - omega t',
//             ||r||, rho |
//
// A vector update feeds the product that follows it without a barrier in
// between: the product forms the updated element of every column it gathers
// (the same two roundings that the row's owner stores), so p, s and CG's r
// are never gathered from memory in the phase that writes them (p and CG's
// r alternate between two buffers).
//
// Sums keep the canonical order (sell_device.cuh).  A team of 8 warps takes
// the 8 slices of a group together and stores the group's sum; after the
// barrier every block folds all group sums itself and performs the scalar
// step on its own copy of the state, so a reduction costs no second barrier.
// Iterates are therefore those of the multi-kernel loop, bit for bit.
//
// Matrix words do not change during the loop.  Up to one group per team the
// blocks run one per SM with 128 registers, and a warp keeps its slices of
// the three matrices in them (12.4 -> 11.0 us per CG iteration at 40^3);
// above that, two blocks per SM with 64 registers read them in each phase.
//
// Every wait is bounded (wait_limit_us); a block that gives up sets the abort
// word, which ends the others' waits.  Other blocks, the one that stores the
// state among them, may still pass their last barrier, so the abort word goes
// to the host with the state and decides whether the loop timed out.
#pragma once

#include "krylov_epi.cuh"

namespace ainv {
namespace dev {

constexpr int kPTeams = 2;  // groups per block and step
constexpr int kPBufs = 4;   // group-sum buffers used in turn
constexpr int kPBlock = kPTeams * kFoldThreads;
constexpr int kPWarps = kPBlock / 32;
// Groups per team up to which a solve runs here.  Past it a phase is bound by
// the bytes it moves, and the plain kernels, with 48 warps per SM against 32,
// move them faster: us per iteration here / there at 52^3 CG 15.1 / 28.6,
// 64^3 CG 20.0 / 34.0, 64^3 BiCGSTAB 35.4 / 52.3 (2 groups), 80^3 CG 37.4 /
// 42.9, 84^3 BiCGSTAB 81.7 / 85.4 (4 groups), 90^3 BiCGSTAB 92.9 / 85.9,
// 100^3 BiCGSTAB 120 / 112.  These have factors of 4 slots and an A of 7; wider
// ones end earlier (persist_limit).
constexpr int kPMaxPerTeam = 4;
// Limits on slots per row times groups per team, for both factors together and
// for A.  A phase takes a row's slots 8 at a time one after the other, with up
// to three gathers per slot and registers that spill, so that wide rows cost
// here what the launches cost there; how much depends on the values' loads
// (fast: the packs with kernels of their own).  us per iteration here / there,
// the last size kept and the first one left to the plain loop:
//   INVK(1,1), 23 slots: FP64 BiCGSTAB 52^3 (1 group) 43.7 / 58.5, 60^3 (2) 87.6 /
//   78.8; FP32 66^3 (2) 68.3 / 78.8, 69^3 (3) 91.3 / 85.0; FP32_ACC64 63^3 (2) 68.3 /
//   73.5, 69^3 98.2 / 83.4; BF16_ACC64 fast 66^3 (2) 68.0 / 75.3, 69^3 88.2 / 77.8,
//   not fast (56^3: the rows' average is 22) 94.4 / 59.9; BF16 not fast 52^3 (1) 54.4 /
//   57.8, 56^3 (2) 87.1 / 60.3.
//   11 slots, not fast: FP64 CG 84^3 (4) 80.9 / 83.3; FP32_ACC64 72^3 (3) 67.6 / 68.5,
//   84^3 (4) 115 / 83.1.
//   131 slots, not fast: FP64 BiCGSTAB 20^3 137 / 101, 46^3 254 / 178.
//   A of 27 slots with factors of 1: CG 66^3 (2) 44.4 / 50.7, 68^3 (3) 57.9 / 52.9.
constexpr int kPMaxASlots = 56;
constexpr int persist_limit(int prec, bool fast) {
  if (fast) return prec == AINV_PREC_FP64 ? 64 : 96;
  return prec == AINV_PREC_BF16_ACC64 ? 44 : prec == AINV_PREC_FP32_ACC64 ? 66 : 88;
}
// Ranges a block folds in one step (one lane each): 32 ranges of 256 groups.
constexpr int kPMaxRanges = 32;
constexpr long long kPMaxRows = (long long)kPMaxRanges * kFoldRange * kGroupSlices * kSlice;

template <class V>
struct PMat {
  InfoView<V> m;
  int lg;  // log2 of the pack
};

// The vectors of a loop.  CG alternates r and p: iteration k reads [k & 1] and
// writes [(k + 1) & 1].  BiCGSTAB keeps r in r[0] and alternates p, which is in
// p[0] where a launch starts and ends; p[1] then holds the true residual of a
// replacement that is still to be done.
struct PVecs {
  double *x, *b, *r[2], *rt, *p[2], *v, *f, *s, *z, *t;
};

template <class V, class T>
struct PArgs {
  PMat<V> wt, z;
  PMat<double> a;
  const V *d;
  T *t;  // apply intermediate
  PVecs w;
  const double *xin, *bin;  // start: x0 and b (first launch of a solve)
  double *xout;             // the solution goes here when the loop ends
  double *gs;               // group sums: kPBufs buffers of 3 x ng
  int n, ns, ng;
  unsigned *bar, *bar_next;  // this launch's arrival counter; the next one's, cleared here
  int *abort;        // 0 at the launch; set by a block that gives up
  unsigned wait_us;  // limit of a wait; 0: any wait is given up
  KState *st;
  int resume;     // continue from *st
  int max_iters;  // iterations of this launch at most
};

struct PShared {
  KState k;
  double tree[3][kPMaxRanges * 8];
  double slice[kPTeams][2][3][kGroupSlices];
  double rho;
  int dead;
};

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kFoldThreads) : "memory");
}
__device__ __forceinline__ void red_release(unsigned *p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Arrivals of nb blocks at a counter that only grows.
struct GridBarrier {
  unsigned *ctr;
  int *abort;
  unsigned nb, target;
  // Called by every thread of the block; false once a wait was given up
  // (by any block).
  __device__ __forceinline__ bool wait(PShared &sh, unsigned wait_us) {
    // The block's writes reach the other blocks by the release of thread 0
    // (the block barrier orders them before it), theirs this block by its
    // acquire.
    __syncthreads();
    target += nb;
    if (threadIdx.x == 0 && nb > 1) {
      red_release(ctr, 1u);
      if (ld_acquire(ctr) < target) {
        const unsigned long long t0 = global_ns();
        for (unsigned it = 1;; ++it) {
          if (ld_acquire(ctr) >= target) break;
          if (((it & 63u) == 0 || wait_us == 0) &&
              (*(volatile int *)abort != 0 || global_ns() - t0 >= wait_us * 1000ull ||
               it > (1u << 30))) {
            *(volatile int *)abort = 1;
            sh.dead = 1;
            break;
          }
        }
      }
    }
    __syncthreads();
    return sh.dead == 0;
  }
};

// ---- a slice's static words ------------------------------------------------
// The first K slots of the lane's row.  P: the pack (vector loads), or 0 for
// any pack (a load per slot, position from the matrix's pack): the phases are
// bound by the instructions they issue as much as by latency (with P = 0 368
// per slice and phase at 64^3, 43% of the issue slots; vector loads take the
// 64^3 BiCGSTAB iteration from 42.5 to 35.4 us).  Copying the values ahead into
// shared memory (cp.async) cost more instructions than it hid latency: 50 us.
template <class V, int P, int K>
struct Slab {
  static constexpr int kP = P > 0 ? P : 1;
  InfoSlab<V, kP, K> b;  // columns relative to the row in offset mode
  int4 f;
};

__device__ __forceinline__ double ldk(const double *p) { return __ldg(p); }
template <class V>
__device__ __forceinline__ typename Acc<V>::type ldk(const V *p) { return ldd(p); }

template <class V, int P, int K>
__device__ __forceinline__ void slab_slots(const PMat<V> &a, const int4 &f, int k0,
                                           InfoSlab<V, Slab<V, P, K>::kP, K> &b) {
  if constexpr (P > 0) {
    info_load(a.m, f, k0, b);
  } else {
    const int lane = threadIdx.x & 31;
    const int pm = (1 << a.lg) - 1;
#pragma unroll
    for (int j = 0; j < K; j++) {
      const int k = k0 + j;
      if (k < f.z) {
        const int pos = ((k >> a.lg) << (5 + a.lg)) + (lane << a.lg) + (k & pm);
        b.v[j][0] = ldk(a.m.val + f.x + pos);
        b.c[j][0] = f.w ? __ldg(a.m.pidx + f.y + k) : __ldg(a.m.idx + f.y + pos);
      } else {
        b.v[j][0] = 0;
        b.c[j][0] = INT_MIN;
      }
    }
  }
}

template <class V>
__device__ __forceinline__ int4 slice_info(const PMat<V> &a, int s) {
  return s < a.m.nslices ? __ldg(a.m.info + s) : make_int4(0, 0, 0, 1);
}
template <class V, int P, int K>
__device__ __forceinline__ void slab_load(const PMat<V> &a, const int4 &f, Slab<V, P, K> &b) {
  b.f = f;
  slab_slots<V, P, K>(a, f, 0, b.b);
}

// The lane's row dotted with the gathered vector g (g(column) gives an
// element), G::kBatch gathers in flight; slots in order, zero slots add 0.
template <class V, int P, int K, class G>
__device__ __forceinline__ void slab_sum(const PMat<V> &a, const InfoSlab<V, P, K> &b, int base,
                                         const G &g, typename Acc<V>::type &acc) {
  using A = typename Acc<V>::type;
  constexpr int B = G::kBatch < K ? G::kBatch : K;
#pragma unroll
  for (int j0 = 0; j0 < K; j0 += B) {
    A xv[B];
#pragma unroll
    for (int j = 0; j < B; j++) {
      const int c = b.c[(j0 + j) / P][(j0 + j) % P] + base;
      xv[j] = (unsigned)c < (unsigned)a.m.n ? (A)g(c) : A(0);
    }
#pragma unroll
    for (int j = 0; j < B; j++) {
      const A v = b.v[(j0 + j) / P][(j0 + j) % P];
      acc = madd(v, v != A(0) ? xv[j] : A(0), acc);
    }
  }
}

template <class V, int P, int K, class G>
__device__ __forceinline__ typename Acc<V>::type slab_dot(const PMat<V> &a,
                                                          const Slab<V, P, K> &b, int row,
                                                          const G &g) {
  typename Acc<V>::type acc = 0;
  const int base = b.f.w ? row : 0;
  slab_sum(a, b.b, base, g, acc);
  for (int k0 = K; k0 < b.f.z; k0 += K) {
    InfoSlab<V, Slab<V, P, K>::kP, K> r;
    slab_slots<V, P, K>(a, b.f, k0, r);
    slab_sum(a, r, base, g, acc);
  }
  return acc;
}

// ---- gathered vectors ---------------------------------------------------------
// These vectors are written while the kernel runs: ordinary, volatile loads.
template <class X>
struct GVec {
  static constexpr int kBatch = 8;
  const X *x;
  __device__ __forceinline__ X operator()(int c) const { return ld_now(x + c); }
};
// CG: p = z (first iteration) or z + beta p.
template <int B>
struct GCgP {
  static constexpr int kBatch = B;
  const double *z, *p;
  double beta;
  bool first;
  __device__ __forceinline__ double operator()(int c) const {
    const double zc = ld_now(z + c);
    return first ? zc : zc + beta * ld_now(p + c);
  }
};
// r - alpha q (CG's r, BiCGSTAB's s).
template <int B>
struct GSub {
  static constexpr int kBatch = B;
  const double *r, *q;
  double alpha;
  __device__ __forceinline__ double operator()(int c) const {
    return ld_now(r + c) - alpha * ld_now(q + c);
  }
};
// BiCGSTAB: p = r (first iteration) or r + beta (p - omega v).
template <int B>
struct GBiP {
  static constexpr int kBatch = B;
  const double *r, *p, *v;
  double beta, omega;
  bool first;
  __device__ __forceinline__ double operator()(int c) const {
    const double rc = ld_now(r + c);
    return first ? rc : rc + beta * (ld_now(p + c) - omega * ld_now(v + c));
  }
};

// ---- phases ---------------------------------------------------------------------
// Blocks lb of nb walk the groups, a team per group, a warp per slice:
// body(s, row, v) with the warp's slice and the lane's row (which may be past
// n), then, for NV > 0, the group sums of v[0..NV) go to gs.
template <int NV, class Body>
__device__ __forceinline__ void for_groups(int n, int ns, int ng, int lb, int nb, PShared &sh,
                                           double *gs, Body &&body) {
  const int team = threadIdx.x / kFoldThreads, lane = threadIdx.x & 31;
  const int warp = (threadIdx.x / 32) % kGroupSlices;
  int buf = 0;
  for (int g = lb * kPTeams + team; g < ng; g += nb * kPTeams) {
    const int s = g * kGroupSlices + warp;
    double v[NV > 0 ? NV : 1] = {};
    if (s < ns) body(s, s * kSlice + lane, v);
    if constexpr (NV > 0) {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const double w = warp_tree(v[k]);
        if (lane == 0) sh.slice[team][buf][k][warp] = w;
      }
      team_sync(team);
      const int t = threadIdx.x % kFoldThreads;
      if (t < NV) {
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < kGroupSlices; j++)
          if (g * kGroupSlices + j < ns) sum = __dadd_rn(sum, sh.slice[team][buf][t][j]);
        gs[(size_t)t * ng + g] = sum;
      }
      buf ^= 1;
    }
  }
}

// Every block folds the group sums (steps 3 and 4 of the canonical order;
// at most kPMaxRanges ranges) and runs fin on its copy of the state.
// dot k's group sums are at src[k].
template <int NV, class Fin>
__device__ __forceinline__ void fold_groups(const double *const (&src)[NV], int ng, PShared &sh,
                                            Fin &&fin) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int nt = (ng + 31) / 32;  // warp trees with groups
  for (int u0 = warp; u0 < nt; u0 += 4 * kPWarps) {
    double v[4][NV];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int g = (u0 + q * kPWarps) * 32 + lane;
#pragma unroll
      for (int k = 0; k < NV; k++) v[q][k] = g < ng ? ld_now(src[k] + g) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int u = u0 + q * kPWarps;
      if (u < nt) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
          const double t = warp_tree(__dadd_rn(0.0, v[q][k]));
          if (lane == 0) sh.tree[k][u] = t;
        }
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    double tot[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double r = 0.0;
#pragma unroll
      for (int w = 0; w < 8; w++)
        if (lane * 8 + w < nt) r = __dadd_rn(r, sh.tree[k][lane * 8 + w]);
      r = __dadd_rn(0.0, r);
      // one range: the tree over the ranges would add zeros to it
      if (nt > 8) r = warp_tree(r);
      tot[k] = __dadd_rn(0.0, r);
    }
    if (lane == 0) fin(tot);
  }
  __syncthreads();
}

__device__ __forceinline__ bool periodic_check(const KState &k) {
  return !k.done && k.check_every > 0 && k.iter > 0 && k.iter % k.check_every == 0;
}

// P: the pack of W^T and Z with A's pack 1, or 0 for any packs.
template <class V, class T, int P, int K, int METHOD, int MB>
struct PLoop {
  static constexpr int KA = 8;  // slots of A per step
  static constexpr int PA = P > 0 ? 1 : 0;
  static constexpr bool kKeep = MB == 1 && K <= 4;
  static constexpr int kB = MB == 1 ? 8 : 4;  // formed elements in flight
  const PArgs<V, T> &a;
  PShared &sh;
  GridBarrier bar;
  int lb, nb;
  Slab<V, P, K> hw, hz;     // the warp's first slice of W^T, Z
  Slab<double, PA, KA> ha;  // and of A
  int par = 0;     // group-sum buffer

  __device__ __forceinline__ PLoop(const PArgs<V, T> &args, PShared &shared, int lb_, int nb_)
      : a(args), sh(shared), bar{args.bar, args.abort, (unsigned)nb_, 0u}, lb(lb_), nb(nb_) {
    const int team = threadIdx.x / kFoldThreads;
    const int s0 =
        (lb * kPTeams + team) * kGroupSlices + (int)(threadIdx.x / 32) % kGroupSlices;
    hw.f = slice_info(a.wt, s0);
    hz.f = slice_info(a.z, s0);
    ha.f = slice_info(a.a, s0);
    if constexpr (kKeep) {
      slab_load(a.wt, hw.f, hw);
      slab_load(a.z, hz.f, hz);
      slab_load(a.a, ha.f, ha);
    }
  }
  __device__ __forceinline__ double *gs() const { return a.gs + (size_t)par * 3 * a.ng; }
  __device__ __forceinline__ void next_buf() { par = (par + 1) % kPBufs; }
  template <int NV, class Fin>
  __device__ __forceinline__ void fold_at(const double *sums, Fin &&fin) {
    const double *src[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) src[k] = sums + (size_t)k * a.ng;
    fold_groups<NV>(src, a.ng, sh, fin);
  }
  __device__ __forceinline__ bool sync() { return bar.wait(sh, a.wait_us); }
  template <int NV, class Body>
  __device__ __forceinline__ void groups(Body &&body) {
    for_groups<NV>(a.n, a.ns, a.ng, lb, nb, sh, gs(), body);
  }
  template <int NV, class Fin>
  __device__ __forceinline__ void fold(Fin &&fin) {
    fold_at<NV>(gs(), fin);
    next_buf();
  }

  // Row `row` (of a row past the end, the last one: its loads are in bounds).
  __device__ __forceinline__ int clamp(int row) const { return row < a.n ? row : a.n - 1; }

  // body(row, slab, v) for the warp's slice of every group.  The first slice
  // (h) is kept in registers through the loop where they suffice (kKeep:
  // most systems have one group per team there), else its word group is;
  // the next slice's word group is loaded while this slice is summed.
  template <int NV, class U, int PP, int KK, class Body>
  __device__ __forceinline__ void slabs(const PMat<U> &m, const Slab<U, PP, KK> &h, Body &&body) {
    int4 f = h.f;
    bool head = true;
    groups<NV>([&](int s, int row, auto &v) {
      const int4 fn = slice_info(m, s + nb * kPTeams * kGroupSlices);
      if (kKeep && head) {
        body(row, h, v);
      } else {
        Slab<U, PP, KK> b;
        slab_load(m, f, b);
        body(row, b, v);
      }
      head = false;
      f = fn;
    });
  }

  // In each of the three, pre(row) loads what the row's owner needs besides
  // the gathers, so that both are in flight together, and post stores.
  // t = D^-1 W^T g.
  template <int NV, class G, class Pre, class Post>
  __device__ __forceinline__ void sweep1(const G &g, Pre &&pre, Post &&post) {
    slabs<NV>(a.wt, hw, [&](int row, const auto &b, auto &v) {
      const auto o = pre(clamp(row));
      const auto d = ldk(a.d + clamp(row));
      const auto acc = slab_dot(a.wt, b, row, g);
      if (row < a.n) {
        a.t[row] = (T)(d * acc);
        post(row, o, v);
      }
    });
  }
  // dst = Z t.
  template <int NV, class Pre, class Post>
  __device__ __forceinline__ void sweep2(double *dst, Pre &&pre, Post &&post) {
    const GVec<T> g{a.t};
    slabs<NV>(a.z, hz, [&](int row, const auto &b, auto &v) {
      const auto o = pre(clamp(row));
      const auto acc = slab_dot(a.z, b, row, g);
      if (row < a.n) {
        const double z = (double)acc;
        dst[row] = z;
        post(row, z, o, v);
      }
    });
  }
  // (A g)[row] for post.
  template <int NV, class G, class Pre, class Post>
  __device__ __forceinline__ void product(const G &g, Pre &&pre, Post &&post) {
    slabs<NV>(a.a, ha, [&](int row, const auto &b, auto &v) {
      const auto o = pre(clamp(row));
      const double acc = slab_dot(a.a, b, row, g);
      if (row < a.n) post(row, acc, o, v);
    });
  }

  // x = x0, b, r = b - A x0 (and rt = r), ||b||, ||r||.
  __device__ __forceinline__ bool init() {
    product<2>(
        GVec<double>{a.xin}, [&](int i) { return make_double2(a.bin[i], a.xin[i]); },
        [&](int i, double acc, double2 o, double (&v)[2]) {
          const double r = o.x - acc;
          a.w.x[i] = o.y;
          a.w.b[i] = o.x;
          a.w.r[0][i] = r;
          if (METHOD == AINV_KRYLOV_BICGSTAB) a.w.rt[i] = r;
          v[0] = o.x * o.x;
          v[1] = r * r;
        });
    if (!sync()) return false;
    fold<2>([&](const double (&v)[2]) {
      const double bn = sqrt(v[0]);
      sh.k.bn2 = (bn == 0.0) ? 1.0 : bn;
      const double pr[3] = {v[1], METHOD == AINV_KRYLOV_BICGSTAB ? v[1] : 0.0, 0.0};
      kstate::finish_dots<kInit>(&sh.k, pr, false, nullptr);
    });
    return true;
  }

  // The true-residual check at the end of an iteration (r: the current
  // residual, scratch: a dead vector).  *replaced: r changed (a barrier
  // follows the change).
  __device__ __forceinline__ bool check(double *r, double *scratch, bool *replaced) {
    *replaced = false;
    const KState &k = sh.k;
    const bool verify = k.done && k.status == AINV_SUCCESS && !k.verified;
    if (!verify && !periodic_check(k)) return true;
    const double *rt = METHOD == AINV_KRYLOV_BICGSTAB ? a.w.rt : nullptr;
    product<3>(
        GVec<double>{a.w.x}, [&](int i) { return make_double2(a.w.b[i], r[i]); },
        [&](int i, double acc, double2 o, double (&v)[3]) {
          const double ri = o.x - acc, g = ri - o.y;
          scratch[i] = ri;
          v[0] = ri * ri;
          v[1] = g * g;
          if (rt) v[2] = rt[i] * ri;
        });
    if (!sync()) return false;
    fold<3>([&](const double (&v)[3]) {
      kstate::finish_dots<kTrueRes>(&sh.k, v, verify, rt);
    });
    if (k.replace) {
      *replaced = true;
      return take_r(r, scratch);
    }
    return true;
  }

  // r := from, the replacement that the state asks for.
  __device__ __forceinline__ bool take_r(double *r, const double *from) {
    groups<0>([&](int, int row, auto &) {
      if (row < a.n) r[row] = from[row];
    });
    const bool ok = sync();
    if (threadIdx.x == 0) sh.k.replace = 0;
    return ok;
  }

  // The solve server's start: x = 0, r = rt = b.
  __device__ __forceinline__ bool init_zero() {
    groups<1>([&](int, int i, double (&v)[1]) {
      if (i >= a.n) return;
      const double b = a.w.b[i];
      a.w.x[i] = 0.0;
      a.w.r[0][i] = b;
      a.w.rt[i] = b;
      v[0] = b * b;
    });
    if (!sync()) return false;
    fold<1>([&](const double (&v)[1]) {
      const double bn = sqrt(v[0]);
      sh.k.bn2 = (bn == 0.0) ? 1.0 : bn;
      const double pr[3] = {v[0], v[0], 0.0};
      kstate::finish_dots<kInit>(&sh.k, pr, false, nullptr);
    });
    return true;
  }

  // The residual norm of an iteration is folded together with rho of the next
  // one, after the Z sweep that both need the barrier for; when the norm ends
  // the loop, that sweep's result is not used.
  __device__ __forceinline__ bool cg() {
    const KState &k = sh.k;
    auto plain_sweep1 = [&](double *r) {
      sweep1<0>(
          GVec<double>{r}, [](int) { return 0; }, [](int, int, auto &) {});
    };
    plain_sweep1(a.w.r[k.iter & 1]);
    if (!sync()) return false;
    bool pending = false;  // the last iteration's norm is not folded yet
    for (int it = 0; it < a.max_iters || pending;) {
      const int c = (k.iter + (pending ? 1 : 0)) & 1;
      double *r = a.w.r[c], *rn = a.w.r[c ^ 1], *p = a.w.p[c], *pn = a.w.p[c ^ 1];
      const double *norm = gs();
      if (pending) next_buf();
      sweep2<1>(
          a.w.z, [&](int i) { return r[i]; },
          [&](int, double z, double ri, double (&v)[1]) { v[0] = ri * z; });
      const double *rho = gs();
      next_buf();
      if (!sync()) return false;
      if (pending) {
        pending = false;
        const double *const src[2] = {norm, rho};
        const bool last = it >= a.max_iters;
        fold_groups<2>(src, a.ng, sh, [&](const double (&v)[2]) {
          kstate::finish_iteration(&sh.k, v[0]);
          sh.rho = v[1];
          if (!sh.k.done && !periodic_check(sh.k) && !last) kstate::cg_take_rho(&sh.k, v[1]);
        });
        if (k.done || periodic_check(k)) {
          bool replaced;
          if (!check(r, rn, &replaced)) return false;
          if (k.done || last) break;
          if (replaced) {  // t and rho belong to the old r
            plain_sweep1(r);
            if (!sync()) return false;
            continue;
          }
          __syncthreads();  // all have read done, which thread 0 may set now
          if (threadIdx.x == 0) kstate::cg_take_rho(&sh.k, sh.rho);
          __syncthreads();
        } else if (last) {
          break;
        }
      } else {
        fold_at<1>(rho, [&](const double (&v)[1]) { kstate::cg_take_rho(&sh.k, v[0]); });
      }
      if (k.done) break;
      const GCgP<kB> gp{a.w.z, p, k.beta, k.iter == 0};
      product<1>(
          gp, [&](int i) { return gp(i); },
          [&](int i, double acc, double pi, double (&v)[1]) {
            pn[i] = pi;
            a.w.v[i] = acc;
            v[0] = pi * acc;
          });
      if (!sync()) return false;
      fold<1>([&](const double (&v)[1]) {
        const double pr[3] = {v[0], 0.0, 0.0};
        kstate::finish_dots<kCgSigma>(&sh.k, pr, false, nullptr);
      });
      if (k.done) break;
      const double alpha = k.alpha;
      const GSub<kB> gr{r, a.w.v, alpha};
      sweep1<1>(
          gr,
          [&](int i) { return make_double2(gr(i), a.w.x[i] + alpha * pn[i]); },
          [&](int i, double2 o, double (&v)[1]) {
            a.w.x[i] = o.y;
            rn[i] = o.x;
            v[0] = o.x * o.x;
          });
      if (!sync()) return false;
      pending = true;
      it++;
    }
    return true;
  }

  __device__ __forceinline__ bool bicgstab() {
    const KState &k = sh.k;
    double *r = a.w.r[0];
    const auto none = [](int) { return 0; };
    if (k.replace && !take_r(r, a.w.p[1])) return false;
    int it = 0;
    for (; it < a.max_iters && !k.done; it++) {
      const int c = it & 1;
      double *p = a.w.p[c], *pn = a.w.p[c ^ 1];
      const GBiP<kB> gp{r, p, a.w.v, k.beta, k.omega, k.iter == 0};
      sweep1<0>(
          gp, [&](int i) { return gp(i); }, [&](int i, double pi, auto &) { pn[i] = pi; });
      if (!sync()) return false;
      sweep2<0>(a.w.f, none, [](int, double, int, auto &) {});
      if (!sync()) return false;
      product<1>(
          GVec<double>{a.w.f}, [&](int i) { return a.w.rt[i]; },
          [&](int i, double acc, double o, double (&v)[1]) {
            a.w.v[i] = acc;
            v[0] = o * acc;
          });
      if (!sync()) return false;
      fold<1>([&](const double (&v)[1]) {
        const double pr[3] = {v[0], 0.0, 0.0};
        kstate::finish_dots<kBicgSigma>(&sh.k, pr, false, a.w.rt);
      });
      if (k.done) break;
      const double alpha = k.alpha;
      const GSub<kB> gsv{r, a.w.v, alpha};
      sweep1<0>(
          gsv, [&](int i) { return gsv(i); },
          [&](int i, double si, auto &) { a.w.s[i] = si; });
      if (!sync()) return false;
      sweep2<0>(a.w.z, none, [](int, double, int, auto &) {});
      if (!sync()) return false;
      product<2>(
          GVec<double>{a.w.z}, [&](int i) { return a.w.s[i]; },
          [&](int i, double acc, double o, double (&v)[2]) {
            a.w.t[i] = acc;
            v[0] = acc * acc;
            v[1] = acc * o;
          });
      if (!sync()) return false;
      fold<2>([&](const double (&v)[2]) {
        const double pr[3] = {v[0], v[1], 0.0};
        kstate::finish_dots<kBicgOmega>(&sh.k, pr, false, a.w.rt);
      });
      if (k.done) break;
      const double omega = k.omega;
      groups<2>([&](int, int i, double (&v)[2]) {
        if (i >= a.n) return;
        const double xi = (a.w.x[i] + alpha * a.w.f[i]) + omega * a.w.z[i];
        const double ri = a.w.s[i] - omega * a.w.t[i], rti = a.w.rt[i];
        a.w.x[i] = xi;
        r[i] = ri;
        v[0] = ri * ri;
        v[1] = rti * ri;
      });
      if (!sync()) return false;
      fold<2>([&](const double (&v)[2]) {
        kstate::finish_iteration(&sh.k, v[0]);
        kstate::bicg_next_rho(&sh.k, v[1]);
      });
      bool replaced;
      if (!check(r, p, &replaced)) return false;
    }
    // the next launch finds p in p[0]
    if (!k.done && (it & 1))
      groups<0>([&](int, int row, auto &) {
        if (row < a.n) a.w.p[0][row] = a.w.p[1][row];
      });
    return true;
  }
};

// The pack that most matrices of a width class (at most 4 slots, or more) get
// (layout.cpp), the one with kernels of its own.
constexpr int fast_pack(size_t value_bytes, bool narrow) {
  return value_bytes == 8 ? 2 : value_bytes == 4 || narrow ? 4 : 8;
}
template <class V, int K>
constexpr int fast_pack() {
  return fast_pack(sizeof(V), K <= 4);
}

// One solve (or max_iters iterations of it) by the whole grid.
template <class V, class T, int P, int K, int METHOD, int MB>
__global__ void __launch_bounds__(kPBlock, MB) k_persist(PArgs<V, T> a) {
  __shared__ PShared sh;
  const int lb = blockIdx.x, nb = gridDim.x;
  if (threadIdx.x == 0) {
    sh.k = *a.st;
    sh.dead = 0;
    if (lb != 0) sh.k.hist = nullptr;  // block 0 records the residuals
    if (lb == 0) *a.bar_next = 0u;
  }
  __syncthreads();
  PLoop<V, T, P, K, METHOD, MB> loop(a, sh, lb, nb);
  bool ok = a.resume ? true : loop.init();
  if (ok && !sh.k.done) ok = METHOD == AINV_KRYLOV_CG ? loop.cg() : loop.bicgstab();
  __syncthreads();
  if (ok && sh.k.done)
    loop.template groups<0>([&](int, int row, auto &) {
      if (row < a.n) a.xout[row] = a.w.x[row];
    });
  if (lb == 0 && threadIdx.x == 0) {
    if (!ok) sh.k.timeout = 1;
    *a.st = sh.k;
  }
}

}  // namespace dev
}  // namespace ainv
