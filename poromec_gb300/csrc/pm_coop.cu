// pm_coop.cu -- a whole FP64 PCG or rpsqmr solve as one cooperative kernel.
//
// What bounds it.  With one kernel per phase an iteration of a small system is
// launches, gaps and last-block reductions: 25 us for the 2,702 equations of
// the 2 x 2 x 40 column, whose 273 k panel values take the FP64 pipe 0.5 us.
// Here a CTA on each SM stays on for the whole solve.  A CTA owns a set of nodes:
// it multiplies their rows and keeps their entries of x, r, p, m and q in
// shared memory, so only the direction p, gathered by all, goes through L2.
// An iteration has three exchanges between the CTAs: (p, q), (r, z), and the
// new direction's visibility.  The last one is saved where the panels have few
// columns (FUSE): each gather then forms p = z + beta p_old itself, one more
// FP64 instruction per column.
//
// Exchanges.  Every CTA stores its partial sum with an epoch, 16 bytes, into
// its slot of kReplicas arrays; one warp of each CTA polls one array, all its
// slots in flight together, and adds them: each lane its senders in order, then
// the lanes by a butterfly.  The sum is the same in every CTA, so all take the same
// decisions, and it does not depend on the order of arrival.  Clocks of an exchange of 152 CTAs: 3,530 with 32
// arrays, 3,780 with one per CTA, 4,070 with 8, 7,470 with one for all (its
// readers queue at the same L2 slices); 1,470 of them are the FP64 adds.
//
// FP64 instructions set the rest: a dependent add takes 66 clocks and occupies
// the scheduler's pipe for 64 whatever its mask, a division 1,430.  So the
// reductions and the scalar recurrences run in one warp, the quotients come from
// a reciprocal by Newton's iteration, formed ahead where the divisor is known, and
// a correction, and the results are broadcast.  The scalars stay in shared memory: in
// registers they cost every thread some 20.  The panels come from L2 in every
// iteration (L1 hits 3 to 14 % of the sectors, L2 84 to 96 %).
//
// The recurrences and tests are those of the kernels in pm_sparse.cu
// (k_pcg_update, k_sqmr_r, k_sqmr_x; Iters.f:299-595 and 6100-6439).  Every
// wait is bounded: a CTA that gives up sets ks->fault and leaves, the others then
// give up as well, and the host solves again with the phase kernels.
#include <cuda_runtime.h>

#include <algorithm>

#include "pm_krylov.h"
#include "pm_reduce.h"

namespace pm {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCoopMaxCtas = 160;            // senders and receivers of an exchange
constexpr int kReplicas = 32;                // arrays of slots (at most one per lane)

// A form of the solve: LANES per node; FUSE, the exchange saved; THREADS per CTA, of
// which CTAS are resident per SM; CHUNK columns per lane whose loads are in flight.
template <int LANES, bool FUSE, int THREADS, int CTAS, int CHUNK>
struct Form {
  static constexpr int L = LANES, T = THREADS, kCtas = CTAS, kChunk = CHUNK;
  static constexpr bool fuse = FUSE;
};

struct alignas(16) Slot {
  double v;
  unsigned long long epoch;
};

__device__ __forceinline__ void slot_store(Slot* s, double v, unsigned long long epoch) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(s),
      "l"(__double_as_longlong(v)), "l"(epoch)
      : "memory");
}
__device__ __forceinline__ void slot_load(const Slot* s, double& v, unsigned long long& epoch) {
  long long b;
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
      : "=l"(b), "=l"(epoch)
      : "l"(s)
      : "memory");
  v = __longlong_as_double(b);
}

struct CoopArgs {
  int nloc;             // nodes per CTA (rounded up)
  const double* m;
  double *x, *r, *p;
  double *p2, *z;       // FUSE: the other direction buffer, and z for the gathers
  KrylovScalars* ks;
  Slot* slots;
  unsigned long long epoch;  // the slots' last epoch
  int polls;                 // of one exchange, before a CTA gives up
};

// The CTA's shared memory: partial sums, the recurrence's scalars (thread 0 keeps
// them, the others read what their phase needs), then the nodes it owns and their
// entries, four per node.
template <int T>
struct CoopShared {
  double part[2][T];
  double alpha, beta, t1, t2;
  double d, rd, pq;          // (rpsqmr: rho, 1 / rho, sigma)
  double dn;                 // rpsqmr's next rho
  double tau, rtau, vj, nr;  // rpsqmr only
  double conv, far;
  int iter, maxit, flag, stop;
};
struct CoopLocal {
  double *x, *r, *p, *m, *q, *d;
  int64_t* vo;
  int64_t* co;
  int* e0;
  int* dw;   // d | W << 3
  int rows;  // 4 x nodes of this CTA
};
__host__ __device__ constexpr int coop_local_bytes(bool sqmr, int nloc) {
  return nloc * (4 * (sqmr ? 6 : 5) * (int)sizeof(double) + 2 * (int)sizeof(int64_t) +
                 2 * (int)sizeof(int));
}

// Group i of 32 / L nodes belongs to CTA i % G, whose warps take its groups in
// turn, so all schedulers get equal shares of the sorted visiting order.
template <typename F>
__device__ CoopLocal coop_setup(const PanelView& P, const CoopArgs& A, bool sqmr, double* dyn) {
  constexpr int NPW = 32 / F::L;
  CoopLocal S;
  const size_t n4 = 4 * (size_t)A.nloc;
  S.x = dyn;
  S.r = S.x + n4;
  S.p = S.r + n4;
  S.m = S.p + n4;
  S.q = S.m + n4;
  S.d = S.q + n4;  // rpsqmr only
  S.vo = reinterpret_cast<int64_t*>(sqmr ? S.d + n4 : S.d);
  S.co = S.vo + A.nloc;
  S.e0 = reinterpret_cast<int*>(S.co + A.nloc);
  S.dw = S.e0 + A.nloc;
  const int groups = (P.nact + NPW - 1) / NPW;
  const int mine = (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  S.rows = 4 * NPW * mine;
  for (int k = threadIdx.x; k < NPW * mine; k += F::T) {
    const int slot = ((int)blockIdx.x + (k / NPW) * (int)gridDim.x) * NPW + k % NPW;
    const NodeRef nr = node_ref(P, slot);
    S.vo[k] = nr.vo;
    S.co[k] = nr.co;
    S.e0[k] = nr.e0;
    S.dw[k] = nr.d | (nr.W << 3);
    for (int j = 0; j < 4; ++j) {
      const bool on = j < nr.d;
      S.x[4 * k + j] = 0.0;
      S.r[4 * k + j] = on ? A.r[nr.e0 + j] : 0.0;
      S.p[4 * k + j] = on ? A.p[nr.e0 + j] : 0.0;
      S.m[4 * k + j] = on ? A.m[nr.e0 + j] : 0.0;
      S.q[4 * k + j] = 0.0;
      if (sqmr) S.d[4 * k + j] = 0.0;
    }
  }
  return S;
}

// q = A p on the CTA's nodes, L lanes per node; p (FUSE: z + beta p) is read
// from L2 (other CTAs wrote it).  A lane's loads are issued kChunk columns at a time.
template <int D, typename F, bool FUSE>
__device__ __forceinline__ void coop_rows(const double* __restrict__ v,
                                          const int32_t* __restrict__ cols, const double* p,
                                          const double* z, double beta, int W, int t,
                                          double (&a)[4]) {
  constexpr int kChunk = F::kChunk, L = F::L;
  for (int c0 = 0; c0 < W; c0 += kChunk * L) {
    double xv[kChunk], zv[FUSE ? kChunk : 1];
    // columns past the last one repeat it and count zero: no branch holds back
    // a load
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int c = cols[min(c0 + u * L + t, W - 1)];
      xv[u] = __ldcg(&p[c]);
      if (FUSE) zv[u] = __ldcg(&z[c]);
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      if (c0 + u * L >= W) break;
      const int c = c0 + u * L + t;
      const bool on = c < W;
      if (FUSE) xv[u] = zv[u] + beta * xv[u];
      const double x = on ? xv[u] : 0.0;
      const double* vc = v + (on ? c : W - 1);
#pragma unroll
      for (int r = 0; r < D; ++r) a[r] += (on ? vc[r * W] : 0.0) * x;
    }
  }
}

template <typename F, bool FUSE>
__device__ void coop_spmv(const CoopLocal& S, const double* __restrict__ val,
                          const int32_t* __restrict__ cols, const double* p, const double* z,
                          double beta) {
  constexpr int L = F::L, NPW = 32 / L;
  const int lane = threadIdx.x & 31, t = lane & (L - 1);
  for (int g = threadIdx.x >> 5; g < S.rows / (4 * NPW); g += F::T / 32) {
    const int k = g * NPW + lane / L;
    const int d = S.dw[k] & 7, W = S.dw[k] >> 3;
    const double* v = val + S.vo[k];
    const int32_t* cl = cols + S.co[k];
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    if (d == 4) coop_rows<4, F, FUSE>(v, cl, p, z, beta, W, t, a);
    else if (d == 3) coop_rows<3, F, FUSE>(v, cl, p, z, beta, W, t, a);
    else if (d == 2) coop_rows<2, F, FUSE>(v, cl, p, z, beta, W, t, a);
    else if (d == 1) coop_rows<1, F, FUSE>(v, cl, p, z, beta, W, t, a);
    // transposed butterfly over the L lanes (k_spmv)
    constexpr int o1 = L / 2, o2 = L / 4;
    const bool h1 = (t & o1) != 0, h2 = (t & o2) != 0;
    double k0 = h1 ? a[2] : a[0], k1 = h1 ? a[3] : a[1];
    k0 += __shfl_xor_sync(kFull, h1 ? a[0] : a[2], o1);
    k1 += __shfl_xor_sync(kFull, h1 ? a[1] : a[3], o1);
    double kk = h2 ? k1 : k0;
    kk += __shfl_xor_sync(kFull, h2 ? k0 : k1, o2);
#pragma unroll
    for (int o = L / 8; o > 0; o >>= 1) kk += __shfl_xor_sync(kFull, kk, o);
    const int r = (h1 ? 2 : 0) + (h2 ? 1 : 0);
    if ((t & (o2 - 1)) == 0 && r < d) S.q[4 * k + r] = kk;
  }
}

// 1 / a by Newton's iteration x <- x + x (1 - a x) from the hardware's
// approximation (20 bits: two steps); the division where that could leave the
// normal range.
__device__ __forceinline__ double recip(double a) {
  const int e = (__double2hiint(a) >> 20) & 0x7ff;
  if (e < 100 || e > 1946) return 1.0 / a;
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  x = fma(x, fma(-a, x, 1.0), x);
  return fma(x, fma(-a, x, 1.0), x);
}
// b / a from x = recip(a), formed ahead or not, with one correction by the
// remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990): the quotient's own rounding
// is what is left of its error, as in the division.  The division itself where x,
// the quotient or the remainder could leave the normal range.
__device__ __forceinline__ double quotient(double b, double a, double x) {
  const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
  if (ea < 100 || ea > 1946 || eb < 200 || eb > 1846 || abs(eb - ea) > 900) return b / a;
  const double q = b * x;
  return fma(fma(-a, q, b), x, q);
}

// One exchange.  part[k][i], i < min(rows, T), are the CTA's terms of value k; VIS
// (and NV = 0) makes the writes before it visible to all CTAs after it.  Warp k sums,
// sends and polls value k (warp 0 where there is none) and has its total in all its
// lanes; the other warps return at once.  The caller broadcasts what follows.
template <int NV, bool VIS = NV == 0, int T>
__device__ __forceinline__ bool exchange(CoopShared<T>& S, const CoopArgs& A, int rows,
                                         unsigned long long epoch, double& tot) {
  constexpr int N1 = NV > 0 ? NV : 1;
  __syncthreads();
  if (threadIdx.x >= 32 * N1) return true;
  const int lane = N1 == 1 ? threadIdx.x : threadIdx.x & 31, k = N1 == 1 ? 0 : threadIdx.x >> 5;
  const int G = gridDim.x;
  double mine = 0.0;
  if (NV > 0) {
    const int n = min(rows, T);
#pragma unroll 4
    for (int i = (n - 1 - lane); i >= 0; i -= 32) mine += S.part[k][i];
    mine = warp_sum(mine);
  }
  if (VIS) __threadfence();
  Slot* buf = A.slots + ((size_t)(epoch & 1) * N1 * kReplicas + k) * kCoopMaxCtas;
  if (lane < kReplicas)
    slot_store(buf + (size_t)lane * N1 * kCoopMaxCtas + blockIdx.x, mine, epoch);
  const Slot* in = buf + (size_t)(blockIdx.x % kReplicas) * N1 * kCoopMaxCtas;
  constexpr int kPer = kCoopMaxCtas / 32;
  double got[kPer];
  // all of a lane's slots in flight together: an exchange then costs one or two
  // load latencies, not one per slot
  bool late;
  int left = A.polls;
  do {
    unsigned long long e[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      got[j] = 0.0;
      e[j] = epoch;
      if (lane + 32 * j < G) slot_load(in + lane + 32 * j, got[j], e[j]);
    }
    late = false;
#pragma unroll
    for (int j = 0; j < kPer; ++j) late |= e[j] != epoch;
  } while (late && --left > 0);
  if (__any_sync(kFull, late || A.polls <= 0)) return false;
  if (VIS) __threadfence();
  if (NV > 0) {
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (32 * j < G) sum += got[j];
    tot = warp_sum(sum);
  }
  return true;
}

// Terms of a dot product over the CTA's rows: term(i) for row i, one partial
// per thread.
template <int T, typename Term>
__device__ __forceinline__ void coop_terms(double (&part)[T], int rows, Term term) {
  if ((int)threadIdx.x < rows) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < rows; i += T) acc += term(i);
    part[threadIdx.x] = acc;
  }
}

#define COOP_SYNC()     \
  do {                  \
    __syncthreads();    \
    if (S.stop) return; \
  } while (0)

// PCG: r = b, p = z = M r, d = (r, z) are k_pcg_init's.
template <typename F>
__global__ void __launch_bounds__(F::T, F::kCtas)
    k_pcg_coop(PanelView P, const double* __restrict__ val, CoopArgs A) {
  constexpr bool FUSE = F::fuse;
  extern __shared__ double coop_dyn[];
  __shared__ CoopShared<F::T> S;
  const CoopLocal X = coop_setup<F>(P, A, false, coop_dyn);
  unsigned long long epoch = A.epoch;
  double *pn = A.p, *po = A.p2;  // FUSE: the direction's buffers, newest first
  if (threadIdx.x == 0) {
    const double conv = A.ks->conv, d = A.ks->d;
    S.conv = conv;
    // |d| at or above this is not converged whatever the rounding of the root (where
    // the square has all its bits: below, the root decides)
    S.far = conv * conv >= 1e-280 ? conv * conv * (1.0 + 1e-9) : INFINITY;
    S.d = d;
    S.rd = recip(d);
    S.pq = S.alpha = S.beta = 0.0;
    S.maxit = A.ks->maxit;
    S.iter = S.stop = 0;
  }
  __syncthreads();
  coop_spmv<F, false>(X, val, P.cols, A.p, nullptr, 0.0);
  for (;;) {
    __syncthreads();
    coop_terms(S.part[0], X.rows, [&](int i) { return X.p[i] * X.q[i]; });
    double tot = 0.0;
    bool ok = exchange<1>(S, A, X.rows, ++epoch, tot);
    if (threadIdx.x == 0) {
      const double alpha = quotient(S.d, tot, recip(tot));
      S.pq = tot;
      S.alpha = alpha;
      S.flag = isfinite(alpha) ? 0 : 3;  // (p, A p) = 0: x stays as it is
      if (!ok) S.stop = A.ks->fault = 1;
    }
    COOP_SYNC();
    if (S.flag) break;
    const double al = S.alpha;
    coop_terms(S.part[0], X.rows, [&](int i) {
      X.x[i] = X.x[i] + al * X.p[i];
      const double ri = X.r[i] - al * X.q[i];
      X.r[i] = ri;
      const double zi = ri * X.m[i];
      X.q[i] = zi;  // q is done with: z
      if (FUSE && (i & 3) < (X.dw[i >> 2] & 7)) A.z[X.e0[i >> 2] + (i & 3)] = zi;
      return ri * zi;
    });
    ok = exchange<1, FUSE>(S, A, X.rows, ++epoch, tot);
    if (threadIdx.x == 0) {
      const double di = tot;
      S.beta = quotient(di, S.d, S.rd);
      S.d = di;
      const int iter = S.iter + 1;
      S.iter = iter;
      int f = 0;
      if (!(fabs(di) >= S.far) && sqrt(fabs(di)) < S.conv) f = 1;
      else if (!isfinite(di)) f = 3;
      else if (iter >= S.maxit) f = 2;
      S.flag = f;
      if (!ok) S.stop = A.ks->fault = 1;
    }
    COOP_SYNC();
    if (S.flag) break;
    const double be = S.beta;
    double* to = FUSE ? po : A.p;
    for (int i = threadIdx.x; i < X.rows; i += F::T) {
      const double pi = X.q[i] + be * X.p[i];
      X.p[i] = pi;
      if ((i & 3) < (X.dw[i >> 2] & 7)) to[X.e0[i >> 2] + (i & 3)] = pi;
    }
    if (FUSE) {
      __syncthreads();  // z in X.q is read: the product overwrites it
      coop_spmv<F, true>(X, val, P.cols, pn, A.z, be);
      to = pn;
      pn = po;
      po = to;
    } else {
      ok = exchange<0>(S, A, X.rows, ++epoch, tot);
      if (threadIdx.x == 0 && !ok) S.stop = A.ks->fault = 1;
      COOP_SYNC();
      coop_spmv<F, false>(X, val, P.cols, A.p, nullptr, 0.0);
    }
    if (threadIdx.x == 0) S.rd = recip(S.d);
  }
  for (int i = threadIdx.x; i < X.rows; i += F::T)
    if ((i & 3) < (X.dw[i >> 2] & 7)) A.x[X.e0[i >> 2] + (i & 3)] = X.x[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    KrylovScalars* ks = A.ks;
    ks->d = S.d;
    ks->pq = S.pq;
    ks->alpha = S.alpha;
    ks->beta = S.beta;
    ks->iter = S.iter;
    ks->conv_flag = S.flag;
    ks->done = 1;
  }
}

// rpsqmr: p = the direction q of the method, q = t = A q, d = d; k_sqmr_init's
// start.  (r, M r) is summed with ||r||^2, so an iteration has PCG's exchanges.
template <typename F>
__global__ void __launch_bounds__(F::T, F::kCtas)
    k_sqmr_coop(PanelView P, const double* __restrict__ val, CoopArgs A) {
  constexpr bool FUSE = F::fuse;
  extern __shared__ double coop_dyn[];
  __shared__ CoopShared<F::T> S;
  const CoopLocal X = coop_setup<F>(P, A, true, coop_dyn);
  unsigned long long epoch = A.epoch;
  double *pn = A.p, *po = A.p2;
  // both values of the second exchange in slots apart from the one-value ones
  CoopArgs A2 = A;
  A2.slots = A.slots + 2 * (size_t)kReplicas * kCoopMaxCtas;
  if (threadIdx.x == 0) {
    const double rho = A.ks->d, tau = A.ks->normr;
    S.conv = A.ks->conv;
    S.d = rho;
    S.rd = recip(rho);
    S.tau = tau;
    S.rtau = recip(tau);
    S.vj = A.ks->neta;
    S.pq = S.nr = S.alpha = 0.0;
    S.maxit = A.ks->maxit;
    S.iter = S.stop = 0;
  }
  __syncthreads();
  coop_spmv<F, false>(X, val, P.cols, A.p, nullptr, 0.0);
  for (;;) {
    __syncthreads();
    coop_terms(S.part[0], X.rows, [&](int i) { return X.p[i] * X.q[i]; });
    double tot = 0.0;
    bool ok = exchange<1>(S, A, X.rows, ++epoch, tot);
    if (threadIdx.x == 0) {
      S.pq = tot;
      S.alpha = quotient(S.d, tot, recip(tot));
      if (!ok) S.stop = A.ks->fault = 1;
    }
    COOP_SYNC();
    const double al = S.alpha;
    if ((int)threadIdx.x < X.rows) {
      double rr = 0.0, rt = 0.0;
      for (int i = threadIdx.x; i < X.rows; i += F::T) {
        const double ri = X.r[i] - al * X.q[i];
        X.r[i] = ri;
        const double ti = ri * X.m[i];
        X.q[i] = ti;  // A q is done with: M r
        if (FUSE && (i & 3) < (X.dw[i >> 2] & 7)) A.z[X.e0[i >> 2] + (i & 3)] = ti;
        rr += ri * ri;
        rt += ri * ti;
      }
      S.part[0][threadIdx.x] = rr;
      S.part[1][threadIdx.x] = rt;
    }
    ok = exchange<2, FUSE>(S, A2, X.rows, ++epoch, tot);
    if (threadIdx.x == 0) {
      const double nr = sqrt(tot), alpha = S.alpha, vj = S.vj, tau = S.tau;
      const double vn = quotient(nr, tau, S.rtau);
      const double cn2 = recip(1.0 + vn * vn);
      S.tau = tau * vn * sqrt(cn2);
      S.t1 = cn2 * vj * vj;
      S.t2 = cn2 * alpha;
      S.vj = vn;
      S.nr = nr;
      const int iter = S.iter + 1;
      S.iter = iter;
      int f = 0;
      if (S.pq == 0.0 || !isfinite(alpha)) f = 3;
      else if (nr < S.conv) f = 1;
      else if (!isfinite(nr)) f = 3;
      else if (iter >= S.maxit) f = 2;
      else if (S.d == 0.0) f = 3;
      S.flag = f;
      if (!ok) S.stop = A.ks->fault = 1;
    } else if (threadIdx.x == 32) {
      S.beta = quotient(tot, S.d, S.rd);
      S.dn = tot;
      if (!ok) S.stop = A.ks->fault = 1;
    }
    COOP_SYNC();
    const double t1 = S.t1, t2 = S.t2, be = S.beta;
    const bool go = S.flag == 0;
    double* to = FUSE ? po : A.p;
    for (int i = threadIdx.x; i < X.rows; i += F::T) {
      const double qi = X.p[i], di = t1 * X.d[i] + t2 * qi;
      X.d[i] = di;
      X.x[i] = X.x[i] + di;
      if (go) {
        const double qn = X.q[i] + be * qi;
        X.p[i] = qn;
        if ((i & 3) < (X.dw[i >> 2] & 7)) to[X.e0[i >> 2] + (i & 3)] = qn;
      }
    }
    if (threadIdx.x == 0) S.d = S.dn;
    if (!go) break;
    if (FUSE) {
      __syncthreads();
      coop_spmv<F, true>(X, val, P.cols, pn, A.z, be);
      to = pn;
      pn = po;
      po = to;
    } else {
      ok = exchange<0>(S, A, X.rows, ++epoch, tot);
      if (threadIdx.x == 0 && !ok) S.stop = A.ks->fault = 1;
      COOP_SYNC();
      coop_spmv<F, false>(X, val, P.cols, A.p, nullptr, 0.0);
    }
    if (threadIdx.x == 0) {
      S.rd = recip(S.d);
      S.rtau = recip(S.tau);
    }
  }
  for (int i = threadIdx.x; i < X.rows; i += F::T)
    if ((i & 3) < (X.dw[i >> 2] & 7)) A.x[X.e0[i >> 2] + (i & 3)] = X.x[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    KrylovScalars* ks = A.ks;
    ks->d = S.d;
    ks->pq = S.pq;
    ks->normr = S.tau;
    ks->neta = S.vj;
    ks->ro1 = S.nr;
    ks->iter = S.iter;
    ks->conv_flag = S.flag;
    ks->done = 1;
  }
}
#undef COOP_SYNC

template <bool SQMR, typename F>
cudaError_t launch(const PanelView& P, const double* val, CoopArgs A, int grid, cudaStream_t s) {
  constexpr int NPW = 32 / F::L;
  const int groups = (P.nact + NPW - 1) / NPW;
  A.nloc = NPW * ((groups + grid - 1) / grid);
  const int smem = coop_local_bytes(SQMR, A.nloc);
  const void* k = SQMR ? (const void*)k_sqmr_coop<F> : (const void*)k_pcg_coop<F>;
  // the cap of every mesh, not this one's size: handles of other threads launch too
  cudaError_t e =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoopMaxSmem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&P, (void*)&val, (void*)&A};
  return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(F::T), args, smem, s);
}

// Two forms.  Up to 32 nodes per CTA: a warp per node and the exchange saved by
// FUSE.  Above: two nodes per warp (fewer FP64 adds per node), where the extra FP64
// instruction per column costs more than the exchange.  Microseconds per iteration
// (fused / two nodes per warp): cube 8^3 14.4 / 15.5, cube 10^3 (31 nodes per CTA) PCG
// 18.0 / 16.7, rpsqmr 19.5 / 20.2, tetra 8^3 (30) 15.4 / 16.0, tetra 9^3 (38) 18.9 / 17.6.
//
// Two CTAs per SM, so that the solves of two host threads share the SMs: one waits in
// an exchange while the other computes.  With the whole register file for one CTA
// (512 threads of up to 128 registers) they ran one after the other.  Microseconds
// per PCG solve to 1e-10 with 1, 2, 4 and 8 host threads, here / one CTA per SM /
// phase kernels:
//   column       2,700  1,490  1,430  1,480 /  2,690  2,610  2,550  2,620 /  6,450  3,350  1,720  1,750
//   cube 5^3     3,250  1,740  1,670  1,690 /  3,180  3,140  3,120  3,120 /  6,600  3,410  1,770  1,750
//   cube 8^3     6,490  3,870  3,870  3,820 /  6,420  6,350  6,370  6,370 / 10,560  5,720  3,300  3,310
//   cube 10^3    9,630  6,040  5,980  6,000 /  9,280  9,330  9,230  9,300 / 12,460  8,120  5,730  5,720
//   tetra 11^3  11,100  7,270  7,330  7,240 / 11,000 11,000 11,200 11,200 / 15,200  9,300  7,250  7,260
//   cube 12^3   13,400  9,690  9,600  9,750 / 13,300 13,700 14,000 14,000 / 17,500 12,400  9,140  9,370
//   cube 14^3   19,700 16,400 16,600 16,700 / 19,600 19,400 19,900 19,700 / 24,600 18,200 14,100 14,200
// Three CTAs of 384 threads (56 registers) or four of 256 take less with many threads
// (cube 8^3 3,190 and 2,870) and more with one (16.8 and 16.9 us per iteration).
using Fused = Form<32, true, 384, 2, 5>;
using Pairs = Form<16, false, 512, 2, 9>;
constexpr int kFuseNodes = 32;
// Above this many panel values per CTA the FP64 pipe hides the phase kernels'
// launches and feeds better from their many CTAs.  Microseconds per iteration, here
// and there: cube 14^3 (47 k values per CTA) 26.8 and 33.5, tetra 16^3 (63 k) 39.7 and
// 45.5, cube 16^3 (70 k) 44.5 and 44.6.
constexpr int64_t kCoopValues = 65000;

// at least a node per scheduler
int coop_grid(const PanelView& P, int sms) {
  return std::max(1, std::min({sms, kCoopMaxCtas, (P.nact + 3) / 4}));
}

}  // namespace

size_t coop_scratch_bytes() {
  return 6 * (size_t)kReplicas * kCoopMaxCtas * sizeof(Slot);
}

int coop_form(const PanelView& P, int sms) {
  return P.nact <= kFuseNodes * coop_grid(P, sms) ? 1 : 2;
}

bool coop_fits(const PanelView& P, int64_t nnz, int sms) {
  if (sms < 1 || P.nact < 1) return false;
  const int grid = coop_grid(P, sms);
  return nnz <= kCoopValues * grid &&
         coop_local_bytes(true, 2 * (P.nact / (2 * grid) + 1)) <= kCoopMaxSmem;
}

cudaError_t krylov_coop(bool sqmr, const PanelView& P, const double* val, const double* m,
                        KrylovVecs& V, KrylovScalars* ks, void* scratch,
                        unsigned long long epoch, int polls, int sms, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(&ks->fault, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  CoopArgs A{};
  A.m = m;
  A.x = V.x;
  A.r = V.r;
  A.p = V.p;
  A.p2 = V.q;
  A.z = V.z;
  A.ks = ks;
  A.slots = static_cast<Slot*>(scratch);
  A.epoch = epoch;
  A.polls = polls;
  const int grid = coop_grid(P, sms);
  if (coop_form(P, sms) == 1)
    return sqmr ? launch<true, Fused>(P, val, A, grid, s) : launch<false, Fused>(P, val, A, grid, s);
  return sqmr ? launch<true, Pairs>(P, val, A, grid, s) : launch<false, Pairs>(P, val, A, grid, s);
}

}  // namespace pm
