// krylov.cu -- unpreconditioned CG (cel_cgalg) and restarted GMRES(m) with
// right Jacobi preconditioning (cel_gmresalg_2jacobi).  The vector sweeps
// run on the device with the fixed-order reductions.  CG's scalar recurrence
// runs on the host; GMRES runs entirely on the device: the Hessenberg column,
// the Givens rotations, the convergence test, the back substitution and the
// restart decisions are one-thread kernels between the sweeps, in the
// reference's operation order, so that a whole solve is one CUDA graph (a
// WHILE node over restart cycles) with no host synchronisation inside.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "graph.cuh"
#include "pcg_internal.cuh"

namespace celg {

// ---- device sweeps ------------------------------------------------------------

// r = b - (0 + r); d = r   (cel_fop_vec_distr_calc_r_and_d, :54-56)
struct OpCalcRD {
  static constexpr int NRED = 0;
  struct Regs { double b, r; };
  const double* b;
  double* r;
  double* d;
  __device__ bool prepare() { return true; }
  __device__ void load(long i, Regs& g) const { g.b = __ldg(b + i); g.r = r[i]; }
  __device__ void compute(long i, Regs& g, double*) const {
    const double ri = __dsub_rn(g.b, dadd(0.0, g.r));
    r[i] = ri;
    d[i] = ri;
  }
  __device__ void finish(double*) const {}
};

// x = x + a d ; r = r + (-a) q     (cel_fop_vec_distr_scale, :862-864)
struct OpXR {
  static constexpr int NRED = 0;
  struct Regs { double x, d, r, q; };
  double* x;
  const double* d;
  double* r;
  const double* q;
  double a;
  __device__ bool prepare() { return true; }
  __device__ void load(long i, Regs& g) const {
    g.x = x[i]; g.d = __ldg(d + i); g.r = r[i]; g.q = __ldg(q + i);
  }
  __device__ void compute(long i, Regs& g, double*) const {
    x[i] = dadd(g.x, dmul(a, g.d));
    r[i] = dadd(g.r, dmul(-a, g.q));
  }
  __device__ void finish(double*) const {}
};

// v = r * inv ; z = v * J     (scale_inv :94-97 and vec_mult_distr_jacobi :364-366)
struct OpV1 {
  static constexpr int NRED = 0;
  struct Regs { double r, J; };
  const double* r;
  double* v;
  double* z;
  const double* J;
  const double* rn;   // ||r|| (device): v = r * (1 / ||r||)
  double inv = 0.0;
  __device__ bool prepare() {
    inv = 1.0 / *(volatile const double*)rn;
    return true;
  }
  __device__ void load(long i, Regs& g) const { g.r = __ldg(r + i); g.J = __ldg(J + i); }
  __device__ void compute(long i, Regs& g, double*) const {
    const double vi = dmul(g.r, inv);
    v[i] = vi;
    z[i] = dmul(vi, g.J);
  }
  __device__ void finish(double*) const {}
};

// v_{j+1} = w / h ; z_{j+1} = v_{j+1} * J   (:774-777, :683)
struct OpVNext {
  static constexpr int NRED = 0;
  struct Regs { double w, J; };
  const double* w;
  double* v;
  double* z;
  const double* J;
  const double* hd;   // h(j+1, j) before the rotations (device)
  const int* act;     // the cycle's Arnoldi steps go on (device)
  double hdiv = 0.0;
  __device__ bool prepare() {
    if (!*(volatile const int*)act) return false;
    hdiv = *hd;
    return true;
  }
  __device__ void load(long i, Regs& g) const { g.w = __ldg(w + i); g.J = __ldg(J + i); }
  __device__ void compute(long i, Regs& g, double*) const {
    const double vi = __ddiv_rn(g.w, hdiv);
    v[i] = vi;
    z[i] = dmul(vi, g.J);
  }
  __device__ void finish(double*) const {}
};

// modified Gram-Schmidt step i: w = w - h_ij v_i (h_ij read from device
// memory), then the next coefficient v_{i+1}.w or, after the last step,
// ||w|| (:699-717)
struct OpMgs {
  static constexpr int NRED = 1;
  struct Regs { double w, v, vn; };
  double* w;
  const double* vi;
  const double* vnext;  // null: norm of w
  const double* hij;
  double* out;
  const int* act;     // the cycle's Arnoldi steps go on (device)
  double h = 0.0;
  __device__ bool prepare() {
    if (!*(volatile const int*)act) return false;
    h = *hij;
    return true;
  }
  __device__ void load(long i, Regs& g) const {
    g.w = w[i];
    g.v = __ldg(vi + i);
    g.vn = vnext ? __ldg(vnext + i) : 0.0;
  }
  __device__ void compute(long i, Regs& g, double* acc) const {
    const double wn = __dsub_rn(g.w, dmul(h, g.v));
    w[i] = wn;
    acc[0] = dadd(acc[0], vnext ? dmul(g.vn, wn) : dmul(wn, wn));
  }
  __device__ void finish(double* tot) const { *out = vnext ? tot[0] : sqrt(tot[0]); }
};

// v_0 . w -> h(0, j), skipped when the cycle has ended
struct OpDotIf {
  static constexpr int NRED = 1;
  struct Regs { double a, b; };
  const double* a;
  const double* b;
  double* out;
  const int* act;
  __device__ bool prepare() { return *(volatile const int*)act != 0; }
  __device__ void load(long i, Regs& r) const { r.a = __ldg(a + i); r.b = __ldg(b + i); }
  __device__ void compute(long, Regs& r, double* acc) const { acc[0] = dadd(acc[0], dmul(r.a, r.b)); }
  __device__ void finish(double* tot) const { *out = tot[0]; }
};

// w = 0 + A z_j, skipped when the cycle has ended
struct EpiStoreIf {
  static constexpr int NRED = 0;
  double* y;
  const int* act;
  __device__ bool active() const { return *(volatile const int*)act != 0; }
  __device__ void row(long r, double s, double*) const { y[r] = dadd(0.0, s); }
  __device__ void finish(double*) const {}
};

// ---- GMRES device state and its one-thread kernels -----------------------------

constexpr int kMaxRestart = 128;

struct GmState {
  double eps, bnorm, resnorm, local;
  int iter, steps, restart, hpos, jdone, conv, act, go;
  double hn[kMaxRestart];   // h(j+1, j) before the rotations: v_{j+1} = w / hn[j]
  double cc[kMaxRestart], ss[kMaxRestart], gam[kMaxRestart + 1], al[kMaxRestart];
};

struct GmArgs {
  GmState* st;
  double* H;     // (M+1) x M Hessenberg, column-major: H(i, j) = H[j (M+1) + i]
  int M;
  double* hist;  // |gamma| history (device, hist_cap entries) or null
  int hist_cap;
  int iter_max;
  int literal;   // the reference's unrotated Givens update (:722-727)
  cudaGraphConditionalHandle cond;
  const int* errw;
  __device__ double& h(int i, int j) const { return H[(size_t)j * (M + 1) + i]; }
  __device__ void push_hist(double v) const {
    if (hist && st->hpos < hist_cap) hist[st->hpos] = v;
    st->hpos += 1;
  }
};

// after ||b||: the tolerance and the counters of the first outer iteration
__global__ void gm_setup_kernel(GmArgs a, double eps_abs, double eps_rel) {
  GmState* s = a.st;
  double e = eps_abs;
  if (eps_rel > 0.0 && eps_rel * s->bnorm > e) e = eps_rel * s->bnorm;
  s->eps = e;
  s->iter = 1;  // the outer loop's first ++iter (:643)
  s->steps = 0;
  s->restart = 0;
  s->hpos = 0;
  s->conv = 0;
  s->act = 0;
  s->go = 1;
}

// after the first residual: its norm opens the history
__global__ void gm_begin_kernel(GmArgs a) {
  GmState* s = a.st;
  a.push_hist(s->resnorm);
  s->local = s->resnorm;
}

// a restart cycle begins: gamma_0 = ||r|| (:669-672)
__global__ void gm_cycle_start_kernel(GmArgs a) {
  GmState* s = a.st;
  s->gam[0] = s->resnorm;
  s->jdone = a.M;
  s->act = 1;
}

// Arnoldi step j after the Gram-Schmidt sweeps left the raw column
// h(0..j+1, j): the previous rotations, the new rotation, gamma and the
// convergence test (:722-737), in the host restatement's operation order.
__device__ void gm_givens(const GmArgs& a, int j) {
  GmState* s = a.st;
  s->steps += 1;
  for (int i = 0; i < j; ++i) {
    if (a.literal) {
      const double t = dadd(dmul(a.h(i, j), s->cc[i]), dmul(a.h(i + 1, j), s->ss[i]));
      a.h(i, j) = dadd(dmul(-t, s->ss[i]), dmul(a.h(i + 1, j), s->cc[i]));
    } else {
      const double top = dadd(dmul(a.h(i, j), s->cc[i]), dmul(a.h(i + 1, j), s->ss[i]));
      const double bot = dadd(dmul(-a.h(i, j), s->ss[i]), dmul(a.h(i + 1, j), s->cc[i]));
      a.h(i, j) = top;
      a.h(i + 1, j) = bot;
    }
  }
  const double hjj = a.h(j, j), hn = a.h(j + 1, j);
  s->hn[j] = hn;
  const double beta = sqrt(dadd(dmul(hjj, hjj), dmul(hn, hn)));
  s->ss[j] = hn / beta;
  s->cc[j] = hjj / beta;
  a.h(j, j) = beta;
  s->gam[j + 1] = dmul(-s->ss[j], s->gam[j]);
  s->gam[j] = dmul(s->cc[j], s->gam[j]);
  const double g = fabs(s->gam[j + 1]);
  a.push_hist(g);
  if (g <= s->eps) {
    s->jdone = j + 1;
    s->conv = 1;
    s->act = 0;
  }
}

__global__ void gm_givens_kernel(GmArgs a, int j) {
  if (a.st->act) gm_givens(a, j);
}

// ---- one Arnoldi step's orthogonalisation in one cooperative kernel ----------------
//
// As one sweep per basis vector, modified Gram-Schmidt reads w, v_i and
// v_i+1 and writes w, 32 n bytes, for each of the j+1 vectors of step j: at
// 128^3 and 15 vectors on average 210 us a step, all of it memory time.  Here
// each CTA keeps its share of w in registers for the whole step and each v_i
// in shared memory between its use as the next and as the current vector, so
// that an MGS step reads 8 n bytes, and the vector after next is on its way
// (bulk copy) while the coefficient is being summed.  The tiles, the order
// within a tile and the tree over the tile sums are those of tile_kernel.
//
// Exchange: a CTA publishes its tile sums, CTA 0 polls and folds them and
// publishes the coefficient, all as 16-byte words of a value and the number
// of the exchange, written and read whole, so that a word needs no reset.  A
// tile's word is not written again before its CTA has the coefficient that
// was made from it.  (Eight CTAs folding a group each: twice as slow, 148
// pollers of eight words hold up the writers.)  Waits are bounded.
//
// The copies of the vector after next start when the pass over the current
// one is done, a few at a time: all at once they queue the exchange's words
// behind 14 MB of data.  (Tile by tile within the pass, with a barrier per
// tile, the pass took 5800 cycles instead of 2400.)
constexpr int kGmThreads = 512;            // 128 registers each (a 17th warp would leave 96)
constexpr int kGmHalf = 7;                 // tiles of w in a thread's registers (4 rows of each)
constexpr int kGmTiles = 2 * kGmHalf;      // tiles of a CTA, alternating between its two 256-thread halves
constexpr int kGmStaged = kGmTiles - 2;    // tiles of v that fit shared memory twice; the others come from L2
constexpr int kGmPolls = 5;                // tile sums a thread of CTA 0 polls
constexpr int kGmMaxTiles = 2112;
constexpr int kGmSmem = (2 * kGmStaged * kTile + kGmMaxTiles) * 8;

struct GmExch {
  ulonglong2* word;           // the coefficient's, then one per tile
  unsigned long long* count;  // exchanges so far (device)
};

__device__ __forceinline__ void put_word(ulonglong2* p, double v, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ bool get_word(const ulonglong2* p, unsigned long long tag, double* v) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  *v = __longlong_as_double((long long)lo);
  return hi == tag;
}
__device__ __forceinline__ double wait_word(const ulonglong2* p, unsigned long long tag, int* abort_) {
  double v;
  unsigned long long t0 = 0;
  for (unsigned i = 0; !get_word(p, tag, &v) && poll_more(i, t0, abort_); ++i) {
  }
  return v;
}

// The butterfly sums (warp_fold) of 8 values per lane at once: at each step
// the lanes of one half of the butterfly take over one half of the values, so
// that 9 exchanges do what 40 would.  Every sum adds the same pairs (operands
// in either order) as warp_fold.  Lane 4 u gets the sum of value u.
__device__ __forceinline__ double warp_fold8(const double (&v)[8], int lane) {
  double a[4], b[2], c;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool up = lane & 16;
    const double mine = up ? v[k + 4] : v[k], other = up ? v[k] : v[k + 4];
    a[k] = dadd(mine, __shfl_xor_sync(0xffffffffu, other, 16));
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const bool up = lane & 8;
    const double mine = up ? a[k + 2] : a[k], other = up ? a[k] : a[k + 2];
    b[k] = dadd(mine, __shfl_xor_sync(0xffffffffu, other, 8));
  }
  {
    const bool up = lane & 4;
    const double mine = up ? b[1] : b[0], other = up ? b[0] : b[1];
    c = dadd(mine, __shfl_xor_sync(0xffffffffu, other, 4));
  }
  c = dadd(c, __shfl_xor_sync(0xffffffffu, c, 2));
  return dadd(c, __shfl_xor_sync(0xffffffffu, c, 1));
}

// One pass over the thread's rows: f(value of w, v_i, v_i+1) -> the new w and
// the term to sum.  FULL: every row exists.
template <bool FULL, class F>
__device__ __forceinline__ void gm_pass(double (&wr)[kGmHalf][4], double (&acc)[8], const double* cur, const double* nxt,
                                        const double* gcur, const double* gnxt, int half, int T, int rows, F f) {
  constexpr int kLast = kGmHalf - 1;
  acc[kGmHalf] = 0.0;
  // the tile that is not staged comes straight from memory
  double e0[4], e1[4];
  if (2 * kLast + half < T) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int o = kLast * 2 * kTile + q * kLanes;
      const bool in = FULL || o < rows;
      e0[q] = in ? __ldg(gcur + o) : 0.0;
      e1[q] = in ? __ldg(gnxt + o) : 0.0;
    }
  }
#pragma unroll
  for (int s = 0; s < kGmHalf; ++s) {
    double t = 0.0;
    if (2 * s + half < T) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = s * 2 * kTile + q * kLanes;
        if (FULL || o < rows) {
          const double a = s == kLast ? e0[q] : cur[o];
          const double b = s == kLast ? e1[q] : nxt[o];
          t = dadd(t, f(wr[s][q], a, b));
        }
      }
    }
    acc[s] = t;
  }
}

__global__ void __launch_bounds__(kGmThreads, 1)
    gm_orth_kernel(GmArgs a, int j, long n, const double* __restrict__ w, double* V, double* Z, size_t nn,
                   const double* __restrict__ J, GmExch ex, int per_cta, int* err) {
  extern __shared__ __align__(128) double vbuf[];  // [2][kGmStaged][kTile], then the tile sums (CTA 0)
  double* tsum = vbuf + 2 * kGmStaged * kTile;
  __shared__ double part[kGmTiles][8];
  __shared__ double red[8];
  __shared__ double s_tot;
  __shared__ int abort_;
  __shared__ uint64_t full[2];
  if (!*(volatile const int*)&a.st->act) return;
  const int tid = threadIdx.x, half = (tid >> 8) & 1, lane256 = tid & 255;
  const long ntiles = (n + kTile - 1) / kTile;
  const long t0 = (long)blockIdx.x * per_cta;
  const int T = (int)max(0L, min((long)per_cta, ntiles - t0));
  unsigned long long tag = *(volatile unsigned long long*)ex.count;
  if (tid == 0) {
    abort_ = 0;
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // offsets of a thread's rows: s 2 kTile + q kLanes from its first
  const long first = (t0 + half) * kTile + lane256;
  const long mine = half * kTile + lane256;  // the same within the CTA's share
  const int rows = (int)min(n - first, 1L << 30);
  const bool all = (t0 + T) * kTile <= n;
  // v_i into buffer i & 1, by one thread (vectors start on 128-byte
  // boundaries and have room to the next 16 bytes)
  auto fetch = [&](int i, bool spread) {
    const long bytes = (min((long)min(T, kGmStaged) * kTile, n - t0 * kTile) * 8 + 15) & ~15L;
    double* dst = vbuf + (size_t)(i & 1) * kGmStaged * kTile;
    const double* src = V + nn * (size_t)i + t0 * kTile;
    mbar_arrive_expect_tx(&full[i & 1], (uint32_t)bytes);
    for (long o = 0; o < bytes; o += 16384) {
      if (spread && o) __nanosleep(150);
      bulk_g2s(dst + o / 8, src + o / 8, (uint32_t)min(16384L, bytes - o), &full[i & 1]);
    }
  };
  if (tid == kGmThreads - 1) {
    fetch(0, false);
    if (j > 0) fetch(1, false);
  }
  auto wait_for = [&](int i) {
    if (!mbar_wait_bounded(&full[i & 1], (uint32_t)((i >> 1) & 1), err)) *(volatile int*)&abort_ = 1;
  };
  auto buf = [&](int i) { return vbuf + (size_t)(i & 1) * kGmStaged * kTile + mine; };
  auto vec = [&](int i) { return V + nn * (size_t)i + first; };
  // the sum of the tiles' lane sums acc[s], the same in every thread; after
  // its first barrier vector `next` is fetched (none: -1)
  auto total = [&](const double (&acc)[8], int next) -> double {
    ++tag;
    const double f = warp_fold8(acc, tid & 31);
    const int s = (tid & 31) >> 2, l = 2 * s + half;
    if ((tid & 3) == 0 && s < kGmHalf && l < T) part[l][lane256 >> 5] = f;
    __syncthreads();
    if (tid < T) {
      double g = part[tid][0];
#pragma unroll
      for (int k = 1; k < 8; ++k) g = dadd(g, part[tid][k]);
      put_word(ex.word + 1 + t0 + tid, g, tag);
    }
    if (next >= 0 && tid == kGmThreads - 1) fetch(next, true);
    if (blockIdx.x == 0) {
      // a thread's words are polled together: one round trip, not one each
      double v[kGmPolls];
      unsigned long long t0w = 0;
      for (unsigned i = 0;; ++i) {
        bool ok = true;
#pragma unroll
        for (int u = 0; u < kGmPolls; ++u) {
          const int k = tid + u * kGmThreads;
          if (k < ntiles) ok = get_word(ex.word + 1 + k, tag, &v[u]) && ok;
        }
        if (ok || !poll_more(i, t0w, &abort_)) break;
      }
#pragma unroll
      for (int u = 0; u < kGmPolls; ++u)
        if (tid + u * kGmThreads < ntiles) tsum[tid + u * kGmThreads] = v[u];
      __syncthreads();
      if (tid < kLanes) {
        double g = 0.0;
        for (int k = tid; k < ntiles; k += kLanes) g = dadd(g, tsum[k]);
        g = warp_fold(g);
        if ((tid & 31) == 0) red[tid >> 5] = g;
      }
      __syncthreads();
      if (tid == 0) {
        double g = red[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) g = dadd(g, red[k]);
        put_word(ex.word, g, tag);
        s_tot = g;
      }
    } else if (tid == 0) {
      s_tot = wait_word(ex.word, tag, &abort_);
    }
    __syncthreads();
    return s_tot;
  };

  double wr[kGmHalf][4], acc[8];
#pragma unroll
  for (int s = 0; s < kGmHalf; ++s)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int o = s * 2 * kTile + q * kLanes;
      wr[s][q] = 2 * s + half < T && o < rows ? __ldg(w + first + o) : 0.0;
    }
  wait_for(0);
  const auto dot = [](double x, double v, double) { return dmul(v, x); };
  if (all) gm_pass<true>(wr, acc, buf(0), buf(0), vec(0), vec(0), half, T, rows, dot);
  else gm_pass<false>(wr, acc, buf(0), buf(0), vec(0), vec(0), half, T, rows, dot);
  double h = total(acc, -1);
  if (blockIdx.x == 0 && tid == 0) a.h(0, j) = h;
  for (int i = 0; i < j; ++i) {
    wait_for(i + 1);
    const auto step = [h](double& x, double v, double vn) {
      x = __dsub_rn(x, dmul(h, v));
      return dmul(vn, x);
    };
    if (all) gm_pass<true>(wr, acc, buf(i), buf(i + 1), vec(i), vec(i + 1), half, T, rows, step);
    else gm_pass<false>(wr, acc, buf(i), buf(i + 1), vec(i), vec(i + 1), half, T, rows, step);
    h = total(acc, i + 2 <= j ? i + 2 : -1);
    if (blockIdx.x == 0 && tid == 0) a.h(i + 1, j) = h;
    if (*(volatile int*)&abort_) break;
  }
  const auto last = [h](double& x, double v, double) {
    x = __dsub_rn(x, dmul(h, v));
    return dmul(x, x);
  };
  if (all) gm_pass<true>(wr, acc, buf(j), buf(j), vec(j), vec(j), half, T, rows, last);
  else gm_pass<false>(wr, acc, buf(j), buf(j), vec(j), vec(j), half, T, rows, last);
  h = sqrt(total(acc, -1));
  if (blockIdx.x == 0 && tid == 0) a.h(j + 1, j) = h;
  // v_{j+1} = w / h(j+1, j), z_{j+1} = J v_{j+1}: not read when the cycle ends here
  if (j + 1 < a.M) {
    double* v = V + nn * (size_t)(j + 1) + first;
    double* z = Z + nn * (size_t)(j + 1) + first;
#pragma unroll
    for (int s = 0; s < kGmHalf; ++s)
      if (2 * s + half < T)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int o = s * 2 * kTile + q * kLanes;
          if (o < rows) {
            const double x = __ddiv_rn(wr[s][q], h);
            v[o] = x;
            z[o] = dmul(x, __ldg(J + first + o));
          }
        }
  }
  if (tid == 0 && *(volatile int*)&abort_) atomicExch(err, kErrTimeout);
  if (blockIdx.x == 0 && tid == 0) {
    *ex.count = tag;
    gm_givens(a, j);
    if (*(volatile int*)&abort_) a.st->act = 0;
  }
}

// al = H^-1 gamma over the cycle's jdone steps (:739-747, :784-792)
__global__ void gm_backsub_kernel(GmArgs a) {
  GmState* s = a.st;
  const int k = s->jdone;
  for (int i = k - 1; i >= 0; --i) {
    double acc = 0.0;
    for (int t = i + 1; t < k; ++t) acc = dadd(acc, dmul(a.h(i, t), s->al[t]));
    s->al[i] = dmul(1.0 / a.h(i, i), __dsub_rn(s->gam[i], acc));
  }
  s->act = 0;
}

// after the cycle's residual: the restart and outer-loop decisions
// (:643, :664-668, :824-830); sets the WHILE node's condition
__global__ void gm_cycle_end_kernel(GmArgs a) {
  GmState* s = a.st;
  s->local = s->resnorm;
  s->restart += 1;
  int go = 1;
  if (s->conv || *(volatile const int*)a.errw) {
    go = 0;
  } else if (s->restart > a.M) {
    // the inner while ends; the outer one goes on while iter <= iter_max
    // (its residual is the one just computed, x being unchanged)
    if (s->iter <= a.iter_max) {
      s->iter += 1;
      s->restart = 0;
    } else {
      go = 0;
    }
  }
  s->go = go;
  if (a.cond) cudaGraphSetConditional(a.cond, (unsigned)go);
}

// x = x + sum_i al_i z_i over the cycle's steps, terms added in order
// i = 0..k-1 (:755-760, :799-803)
__global__ void x_update_kernel(long n, double* __restrict__ x, const double* __restrict__ Z,
                                size_t nn, const GmState* __restrict__ st) {
  const int k = st->jdone;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double xi = x[i];
    for (int t = 0; t < k; ++t) xi = dadd(xi, dmul(st->al[t], __ldg(Z + nn * (size_t)t + i)));
    x[i] = xi;
  }
}

// ---- helpers --------------------------------------------------------------------

static int read_scalar(celg_handle* h, const double* d, double* out) {
  CELG_CUDA(cudaMemcpyAsync(h->scal_h, d, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  *out = h->scal_h[0];
  return CELG_OK;
}

static int spmv_fmt(celg_handle* h, celg_mat* m, int fmt, const double* x, double* y) {
  if (fmt == CELG_FMT_JAD) return launch_spmv_jad(h, m->csr, m->jad, x, y);
  return launch_spmv_csr(h, m->csr, x, y, 0);
}

struct OpFillOne {
  static constexpr int NRED = 0;
  struct Regs { int unused; };
  double* x;
  __device__ bool prepare() { return true; }
  __device__ void load(long, Regs&) const {}
  __device__ void compute(long i, Regs&, double*) const { x[i] = 1.0; }
  __device__ void finish(double*) const {}
};

static int set_x0(celg_handle* h, long n, int mode, double* x) {
  if (mode == CELG_X0_USER || n == 0) return CELG_OK;
  if (mode == CELG_X0_ZERO) {
    CELG_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * (size_t)n, h->stream));
    return CELG_OK;
  }
  return launch_tile(h, n, OpFillOne{x});
}

static void store_hist(celg_result* res, int idx, double v) {
  if (res && res->history && idx < res->history_cap) {
    res->history[idx] = v;
    res->history_len = std::max(res->history_len, idx + 1);
  }
}

// ---- CG: cel_cgalg, src/fcgalg/cel_cgalg_module.f90:34-175 --------------------------

int cg_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
             celg_result* res) {
  const long n = m->csr.n;
  const int fmt = p->fmt;
  if (fmt == CELG_FMT_JAD && m->jad.mmax < 0) return CELG_ERR_STATE;
  int st = ensure_work(h, (size_t)n);
  if (st) return st;
  if (res) res->history_len = 0;
  double* r = h->wr;
  double* d = h->wp;
  double* q = h->wv;
  double* sd = h->scal_d;
  cudaEventRecord(h->ev0, h->stream);
  if ((st = set_x0(h, n, p->x0_mode, x))) return st;
  double bnorm, norm, sigma_new, sigma_old, alpha = 1.0, dq;
  if ((st = launch_dot(h, n, b, b, sd, 1)) || (st = read_scalar(h, sd, &bnorm))) return st;
  double eps = p->eps_abs;
  if (p->eps_rel > 0.0 && p->eps_rel * bnorm > eps) eps = p->eps_rel * bnorm;
  // r = 0 + A x; ||A x|| (:67-77)
  if ((st = spmv_fmt(h, m, fmt, x, r))) return st;
  if ((st = launch_dot(h, n, r, r, sd, 1)) || (st = read_scalar(h, sd, &norm))) return st;
  if ((st = launch_tile(h, n, OpCalcRD{b, r, d}))) return st;
  if ((st = launch_dot(h, n, r, r, sd, 0)) || (st = read_scalar(h, sd, &sigma_new))) return st;
  sigma_old = sigma_new;
  if (!p->literal_ref_bugs) norm = std::sqrt(sigma_new);
  store_hist(res, 0, norm);
  int ii = 0, err = CELG_OK;
  for (;;) {
    bool go;
    if (p->literal_ref_bugs)
      go = ii < p->iter_max && sigma_new > sigma_old * p->eps_abs * p->eps_abs &&
           std::fabs(sigma_new) > kRealSmall;
    else
      go = ii < p->iter_max && norm > eps && std::fabs(sigma_new) > kRealSmall;
    if (!go) break;
    if ((st = spmv_fmt(h, m, fmt, d, q))) return st;
    ++ii;
    if ((st = launch_dot(h, n, d, q, sd, 0)) || (st = read_scalar(h, sd, &dq))) return st;
    alpha = sigma_new / dq;
    if (!std::isfinite(alpha)) {
      err = CELG_ERR_BREAKDOWN;
      break;
    }
    if ((st = launch_tile(h, n, OpXR{x, d, r, q, alpha}))) return st;
    sigma_old = sigma_new;
    if ((st = launch_dot(h, n, r, r, sd, 0)) || (st = read_scalar(h, sd, &sigma_new))) return st;
    const double beta = p->literal_ref_bugs ? alpha : sigma_new / sigma_old;  // :151
    if ((st = launch_xpby(h, n, r, beta, d))) return st;
    norm = std::sqrt(sigma_new);
    store_hist(res, ii, norm);
  }
  // verification
  double vres = 0.0;
  if ((st = launch_residual(h, m, fmt, b, x, q, sd)) || (st = read_scalar(h, sd, &vres))) return st;
  cudaEventRecord(h->ev1, h->stream);
  cudaEventSynchronize(h->ev1);
  cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1);
  h->last_iters = ii;
  int ret = err;
  if (!ret && !p->literal_ref_bugs && norm > eps && ii >= p->iter_max) ret = CELG_ERR_NOCONV;
  if (res) {
    res->iter_done = ii;
    res->final_norm2 = norm;
    res->bnorm = bnorm;
    res->verified_relres = bnorm > 0 ? vres / bnorm : vres;
    res->err = ret;
    res->arnoldi_steps = 0;
  }
  return ret;
}

// ---- GMRES(m): cel_gmresalg_2jacobi, src/fcgalg/cel_gmresalg_module.f90:570-851 -------

// The work space of a GMRES(M) solve on n rows, kept by the handle:
// V[0..M], Z[0..M-1] and H ((M+1) x M), plus the device state.
static int ensure_gmres_work(celg_handle* h, size_t nn, int M) {
  const size_t need = nn * (size_t)(2 * M + 1) + (size_t)(M + 1) * M + 8;
  if (!h->gm_state_d) CELG_CUDA(raw_alloc(h, &h->gm_state_d, sizeof(GmState)));
  if (!h->gm_state_h) CELG_CUDA(cudaMallocHost(&h->gm_state_h, sizeof(GmState)));
  if (need <= h->gm_cap && h->gm_work) return CELG_OK;
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  graph_cache_clear(h);
  cudaFree(h->gm_work);
  h->gm_work = nullptr;
  h->gm_cap = 0;
  CELG_CUDA(raw_alloc(h, &h->gm_work, sizeof(double) * need));
  h->gm_cap = need;
  return CELG_OK;
}

struct GmPlan {
  celg_mat* m;
  int fmt;
  long n;
  size_t nn;
  const double* b;
  double* x;
  const celg_params* p;
  double* V;
  double* Z;
  double* r;
  double* w;
  GmArgs a;
  GmExch ex;      // exchange words of gm_orth_kernel
  int per_cta;    // its tiles per CTA; 0: the graph of sweeps
  double* Vp(int i) const { return V + nn * (size_t)i; }
  double* Zp(int i) const { return Z + nn * (size_t)i; }
  double* Hp(int i, int j) const { return a.H + (size_t)j * (a.M + 1) + i; }
};

// w = A z in the matrix's most compact form
static int gm_spmv(celg_handle* h, const GmPlan& g, const double* x, double* y) {
  const EpiStoreIf epi{y, &g.a.st->act};
  if (g.fmt == CELG_FMT_JAD) return launch_jad(h, g.m->csr, g.m->jad, x, epi);
  return launch_csr<double>(h, g.m->csr, g.m->csr.v, x, epi);
}

// x0, ||b||, the tolerance and the first residual
static int gm_record_setup(celg_handle* h, const GmPlan& g) {
  int st = set_x0(h, g.n, g.p->x0_mode, g.x);
  if (!st) st = launch_dot(h, g.n, g.b, g.b, &g.a.st->bnorm, 1);
  if (st) return st;
  gm_setup_kernel<<<1, 1, 0, h->stream>>>(g.a, g.p->eps_abs, g.p->eps_rel);
  CELG_CUDA(cudaGetLastError());
  st = launch_residual(h, g.m, g.fmt, g.b, g.x, g.r, &g.a.st->resnorm);
  if (st) return st;
  gm_begin_kernel<<<1, 1, 0, h->stream>>>(g.a);
  CELG_CUDA(cudaGetLastError());
  return CELG_OK;
}

static int gm_orth(celg_handle* h, const GmPlan& g, int j) {
  GmArgs a = g.a;
  long n = g.n;
  const double* w = g.w;
  double *V = g.V, *Z = g.Z;
  size_t nn = g.nn;
  const double* J = g.m->jacobi;
  GmExch ex = g.ex;
  int per = g.per_cta;
  int* err = h->err_d;
  void* params[] = {&a, &j, &n, &w, &V, &Z, &nn, &J, &ex, &per, &err};
  const int grid = (int)((ntiles_of(n) + per - 1) / per);
  CELG_CUDA(cudaLaunchCooperativeKernel((const void*)gm_orth_kernel, dim3(grid), dim3(kGmThreads), params, kGmSmem,
                                        h->stream));
  return CELG_OK;
}

// Tiles per CTA of gm_orth_kernel, 0 when w does not fit the registers of the
// resident CTAs, the driver refuses the grid or there is no memory for its
// words (then the graph of sweeps runs; CELG_ONCHIP_ROWS as for PCG).
static int gm_plan_orth(celg_handle* h, GmPlan* g) {
  g->per_cta = 0;
  const long nt = ntiles_of(g->n);
  const char* e = std::getenv("CELG_ONCHIP_ROWS");
  if (g->n < 1 || nt > std::min((long)kGmTiles * h->sms, (long)kGmMaxTiles) || (e && g->n > std::atol(e))) return CELG_OK;
  const int per = (int)((nt + h->sms - 1) / h->sms);
  bool fits = false;
  if (const int st = coop_fits(h, (int)((nt + per - 1) / per), &fits)) return st;
  if (!fits) return CELG_OK;
  if (const int st = allow_dynamic_smem<gm_orth_kernel>(kGmSmem)) return st;
  const size_t bytes = 256 + sizeof(ulonglong2) * (size_t)(kGmMaxTiles + 1);
  if (!h->gm_exch) {
    const cudaError_t em = raw_alloc(h, &h->gm_exch, bytes);
    if (out_of_memory(em)) return CELG_OK;
    CELG_CUDA(em);
  }
  CELG_CUDA(cudaMemsetAsync(h->gm_exch, 0, bytes, h->stream));
  g->ex.count = static_cast<unsigned long long*>(h->gm_exch);
  g->ex.word = static_cast<ulonglong2*>(h->gm_exch) + 15;
  g->per_cta = per;
  return CELG_OK;
}

// One restart cycle: M Arnoldi steps (the kernels of the steps after
// convergence return at once), back substitution, x update, the new
// residual and the loop decision.
static int gm_record_cycle(celg_handle* h, const GmPlan& g) {
  const int M = g.a.M;
  const int* act = &g.a.st->act;
  const double* J = g.m->jacobi;
  gm_cycle_start_kernel<<<1, 1, 0, h->stream>>>(g.a);
  CELG_CUDA(cudaGetLastError());
  // v_0 = r * (1/||r||); z_0 = J v_0 (:669, :683)
  int st = launch_tile(h, g.n, OpV1{g.r, g.Vp(0), g.Zp(0), J, &g.a.st->local});
  for (int j = 0; !st && j < M; ++j) {
    // w = 0 + A z_j (:680-697)
    st = gm_spmv(h, g, g.Zp(j), g.w);
    if (!st && g.per_cta > 0) {
      st = gm_orth(h, g, j);
      if (st) break;
      continue;
    }
    // h_0j = v_0 . w, then modified Gram-Schmidt with the next coefficient fused
    if (!st) st = launch_tile(h, g.n, OpDotIf{g.Vp(0), g.w, g.Hp(0, j), act});
    for (int i = 0; !st && i <= j; ++i) {
      const bool last = i == j;
      st = launch_tile(h, g.n, OpMgs{g.w, g.Vp(i), last ? nullptr : g.Vp(i + 1), g.Hp(i, j),
                                     last ? g.Hp(j + 1, j) : g.Hp(i + 1, j), act});
    }
    if (st) break;
    gm_givens_kernel<<<1, 1, 0, h->stream>>>(g.a, j);
    CELG_CUDA(cudaGetLastError());
    // v_{j+1} = w / h(j+1,j); z_{j+1} = J v_{j+1}
    if (j + 1 < M)
      st = launch_tile(h, g.n, OpVNext{g.w, g.Vp(j + 1), g.Zp(j + 1), J, &g.a.st->hn[j], act});
  }
  if (st) return st;
  gm_backsub_kernel<<<1, 1, 0, h->stream>>>(g.a);
  CELG_CUDA(cudaGetLastError());
  if (g.n > 0) {
    const int grid = (int)std::max(1L, std::min((g.n + 255) / 256, (long)h->sms * 16));
    x_update_kernel<<<grid, 256, 0, h->stream>>>(g.n, g.x, g.Z, g.nn, g.a.st);
    CELG_CUDA(cudaGetLastError());
  }
  // r = b - A x ; ||r|| (:808-824)
  st = launch_residual(h, g.m, g.fmt, g.b, g.x, g.r, &g.a.st->resnorm);
  if (st) return st;
  gm_cycle_end_kernel<<<1, 1, 0, h->stream>>>(g.a);
  CELG_CUDA(cudaGetLastError());
  return CELG_OK;
}

int gmres_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
                celg_result* res) {
  const long n = m->csr.n;
  const int fmt = p->fmt;
  const int M = p->restart;
  if (M <= 0 || M > kMaxRestart) return CELG_ERR_ARG;
  if (p->iter_max < 0) return CELG_ERR_ARG;
  if (!m->jacobi) return CELG_ERR_STATE;
  if (fmt == CELG_FMT_JAD && m->jad.mmax < 0) return CELG_ERR_STATE;
  // distance of the basis vectors: each starts on a 128-byte boundary
  const size_t nn = ((size_t)std::max(1L, n) + 15) & ~(size_t)15;
  int st = ensure_work(h, (size_t)n);
  if (!st) st = ensure_offset_dict(h, m);
  if (!st) st = ensure_gmres_work(h, nn, M);
  if (!st) st = ensure_partials(h, ntiles_of(n), 2);
  const int hist_cap = (res && res->history && res->history_cap > 0) ? res->history_cap : 0;
  if (!st && hist_cap) st = ensure_state(h, hist_cap);
  if (st) return st;
  if (res) res->history_len = 0;
  GmPlan g;
  g.m = m;
  g.fmt = fmt;
  g.n = n;
  g.nn = nn;
  g.b = b;
  g.x = x;
  g.p = p;
  g.V = h->gm_work;
  g.Z = g.V + nn * (size_t)(M + 1);
  g.r = h->wr;
  g.w = h->wv;
  GmState* sd = static_cast<GmState*>(h->gm_state_d);
  g.a = GmArgs{sd, g.Z + nn * (size_t)M, M, hist_cap ? h->hist_d : nullptr, hist_cap, p->iter_max,
               p->literal_ref_bugs, 0, h->err_d};
  CELG_CUDA(cudaMemsetAsync(h->err_d, 0, sizeof(int), h->stream));
  if ((st = gm_plan_orth(h, &g))) return st;
  if (!graphs_enabled()) {
    // host-driven (profiling): one poll of the loop flag per restart cycle
    CELG_CUDA(cudaEventRecord(h->ev0, h->stream));
    st = gm_record_setup(h, g);
    GmState* sh = static_cast<GmState*>(h->gm_state_h);
    while (!st) {
      st = gm_record_cycle(h, g);
      if (st) break;
      CELG_CUDA(cudaMemcpyAsync(&sh->go, &sd->go, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
      CELG_CUDA(cudaStreamSynchronize(h->stream));
      if (!sh->go) break;
    }
    if (st) return st;
    CELG_CUDA(cudaEventRecord(h->ev1, h->stream));
  } else {
    char kb[512];
    std::snprintf(kb, sizeof(kb), "gmres|%p|%d|%d|%p|%p|%d|%d|%d|%.17g|%.17g|%d|%d|%d", (const void*)m,
                  m->csr.n, fmt, (const void*)b, (const void*)x, M, p->x0_mode, p->literal_ref_bugs,
                  p->eps_abs, p->eps_rel, p->iter_max, hist_cap, g.per_cta);
    const std::string key(kb);
    GraphEntry* ge = graph_cache_find(h, key);
    if (!ge) {
      st = graph_build(h, key, [&](cudaGraphConditionalHandle cond) -> int {
        GmPlan gc = g;
        gc.a.cond = cond;
        int s2 = gm_record_setup(h, gc);
        if (!s2) s2 = capture_while(h, cond, [&]() -> int { return gm_record_cycle(h, gc); });
        return s2;
      }, &ge);
      if (st) return st;
    }
    CELG_CUDA(cudaEventRecord(h->ev0, h->stream));
    CELG_CUDA(cudaGraphLaunch(ge->exec, h->stream));
    CELG_CUDA(cudaEventRecord(h->ev1, h->stream));
  }
  GmState* sh = static_cast<GmState*>(h->gm_state_h);
  CELG_CUDA(cudaMemcpyAsync(sh, sd, sizeof(GmState), cudaMemcpyDeviceToHost, h->stream));
  int err_word = 0;
  CELG_CUDA(cudaMemcpyAsync(h->scal_h + 8, h->err_d, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  std::memcpy(&err_word, h->scal_h + 8, sizeof(int));
  cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1);
  h->last_iters = sh->steps;
  int ret = sh->conv ? CELG_OK : CELG_ERR_NOCONV;
  if (err_word) ret = err_word;
  if (res) {
    res->iter_done = sh->iter;
    res->final_norm2 = sh->resnorm;
    res->bnorm = sh->bnorm;
    res->verified_relres = sh->bnorm > 0 ? sh->resnorm / sh->bnorm : sh->resnorm;
    res->err = ret;
    res->arnoldi_steps = sh->steps;
    if (hist_cap) {
      st = copy_history(h, std::min(sh->hpos, hist_cap), res);
      if (st) return st;
    }
  }
  return ret;
}

}  // namespace celg
