// pcg_onchip.cu -- the whole Jacobi-PCG solve of a small or medium system in
// one cooperative kernel (the loop of pcg.cu, same arithmetic, same bits).
//
// What bounds a small solve is not memory but the chain of dependent steps:
// as three graph kernels an iteration of a 32^3 system took 20 us, of which
// the work is under one.  Here one CTA per SM keeps its rows' r, p, x, v and
// J in shared memory for the whole solve; only p (gathered by other CTAs)
// and the reduction terms go through L2, and an iteration is three grid-wide
// exchanges instead of three kernels and a loop node.
//
// Work split.  A unit is what one warp contributes to the reduction tree of
// celg_device.cuh: rows 1024 t + 32 w + lane + 256 k (k = 0..3) of tile t,
// warp w.  Its warp sum depends on nothing else, so units (8 per tile) are
// dealt to the CTAs in equal contiguous runs, one warp per unit at a time,
// and every SM gets the same share to within 128 rows (whole 1024-row tiles
// leave a system of 200 tiles 148 SMs with two tiles on some and one on
// most).
//
// Exchanges.  A warp sum is published by storing it over a sentinel (a NaN
// pattern that no published value has); CTA 0 polls the slots, folds them in
// the tree's order and publishes the totals the same way, and every other
// CTA polls that one word: two trips through L2 with the data in them.
// (All CTAs polling all slots needs one trip, but 128 CTAs spinning on the
// same 2 KB hold up the stores: 9100 cycles an exchange against 2000.)  The
// slots of an iteration are set back to the sentinel once they are known to
// have been read.  p is published by a release of one arrival counter, which
// a thread of each CTA acquires (2400 cycles; a flag per CTA: 4200).  Every
// wait is bounded (kWaitLimitNs).
//
// Matrix.  Values in slices of 32 rows, entry e of the slice's lane l at
// e * 32 + l, so that a warp's loads are whole lines (row-major values would
// touch 14 lines per load for 7 entries a row, 32 for 16 and more).  With
// row patterns (spmv_kernels.cuh) the columns come from the pattern table
// and the slices are kPatLen wide; units whose values fit keep them in
// shared memory.  Otherwise int32 columns are stored like the values.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "graph.cuh"
#include "pcg_internal.cuh"

namespace celg {

// 16 warps at 128 registers: at 32 warps and 64 registers the gathers in
// flight per lane are fewer and every barrier costs more (53^3: 10.1 against
// 8.7 us an iteration; 200k unstructured rows: 32 against 22)
constexpr int kOcThreads = 512;
constexpr int kUnitRows = 128;
constexpr int kOcMaxSmem = 227 * 1024;
constexpr int kOcTail = 64;  // doubles after the slots: the totals (kSlotSets), the arrival counter
// slot sets: p.v, (r.z, r.r) twice, ||b||^2, set-up (r.z, r.r), verification
// (pairs at even positions)
enum OcSlot { kSlotUpd0 = 0, kSlotUpd1 = 2, kSlotInit = 4, kSlotPv = 6, kSlotB = 7, kSlotVer = 8, kSlotSets = 9 };
// longest row of a sliced matrix: with at most 4 kOcMaxUnits slices the sum of
// the slice widths stays within an int
constexpr int kMaxWidth = 31000;
constexpr long kOcMaxUnits = 8 * 2112;
constexpr unsigned long long kSentinel = ~0ull;

template <typename VT>
struct OcArgs {
  int n, ntiles, slots, ncache;
  const VT* sv;       // sliced values
  const int* sc;      // sliced columns (no row patterns)
  const int* sbase;   // first entry of each slice / 32 (no row patterns)
  const int* rp;
  const uint8_t* pid;
  const int* pat;
  int pat_ints;
  const int* plen;
  const VT* rowv;     // row table (then no sliced values), or null
  int juni;           // one Jacobi value, jval, for all rows
  VT jval;
  const VT* b;
  VT* x;
  const VT* J;
  VT* p;
  double* slot;       // kSlotSets x 8 ntiles
  double* total;      // kSlotSets + 1, pairs 16-byte aligned
  unsigned* arrive;
  PcgState* out;      // pinned host memory
  double* hist;
  int hist_cap, iter_max, x0_mode, verify;
  double eps_abs, eps_rel;
};

__device__ __forceinline__ void publish(double* q, double v) {
  unsigned long long u = (unsigned long long)__double_as_longlong(v);
  if (u == kSentinel) u = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(q), "l"(u) : "memory");
}

__device__ __forceinline__ void load2(const double* q, unsigned long long& a, unsigned long long& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(q) : "memory");
}

// The eight warp sums of a tile, waited for, added in warp order.
__device__ __forceinline__ double tile_sum(const double* q, int* abort_) {
  unsigned long long w[8];
  unsigned long long t0 = 0;
  for (unsigned i = 0;; ++i) {
#pragma unroll
    for (int u = 0; u < 8; u += 2) load2(q + u, w[u], w[u + 1]);
    bool ok = true;
#pragma unroll
    for (int u = 0; u < 8; ++u) ok = ok && w[u] != kSentinel;
    if (ok || !poll_more(i, t0, abort_)) break;
  }
  double s = __longlong_as_double((long long)w[0]);
#pragma unroll
  for (int u = 1; u < 8; ++u) s = dadd(s, __longlong_as_double((long long)w[u]));
  return s;
}

// Shared memory of a CTA: fold scratch, the tile sums of up to two
// reductions, the pattern table, then per unit slot the row data.
template <typename VT>
struct OcSmem {
  double* red;   // 16
  int* abort_;
  double* tp;    // 2 ntiles
  int* pat;
  int* meta;     // row length (and pattern index << 16)
  VT *r, *p, *x, *J, *v, *val;
  size_t bytes;
  __host__ __device__ OcSmem(unsigned char* base, int ntiles, int pat_ints, int slots, int ncache) {
    size_t o = 0;
    auto take = [&](size_t b) {
      unsigned char* q = base + o;
      o += (b + 15) & ~(size_t)15;
      return q;
    };
    red = (double*)take(16 * sizeof(double));
    abort_ = (int*)take(16);
    tp = (double*)take(2 * sizeof(double) * (size_t)ntiles);
    pat = (int*)take(sizeof(int) * (size_t)pat_ints);
    const size_t rows = (size_t)slots * kUnitRows;
    meta = (int*)take(sizeof(int) * rows);
    r = (VT*)take(sizeof(VT) * rows);
    p = (VT*)take(sizeof(VT) * rows);
    x = (VT*)take(sizeof(VT) * rows);
    J = (VT*)take(sizeof(VT) * rows);
    v = (VT*)take(sizeof(VT) * rows);
    val = (VT*)take(sizeof(VT) * (size_t)ncache * kUnitRows * kPatLen);
    bytes = o;
  }
};

// values stream from L2 once an iteration; kept out of the small L1 that the
// gathers live in
__device__ __forceinline__ double ld_stream(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_stream(const int* p) {
  int v;
  asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Row sum of one row of a lane (row k of unit slot `slot`), 0 + v0 x0 + v1 x1
// + ... in stored order.  The gathers are ordinary loads: src is written by
// other CTAs between two calls.
template <typename VT, bool PAT>
__device__ __forceinline__ VT row_sum(const OcArgs<VT>& a, const OcSmem<VT>& sm, const VT* src, int slot, int k,
                                      int unit, int lane) {
  const int tile = unit >> 3, w = unit & 7;
  const int meta = sm.meta[slot * kUnitRows + k * 32 + lane];
  VT t = VT(0);
  if constexpr (PAT) {
    const int len = meta & 0xffff;
    const VT* xr = src + (tile * kTile + k * 256 + w * 32 + lane);
    const int4* pq = reinterpret_cast<const int4*>(sm.pat + (meta >> 16) * kPatLen);
    VT xv[kPatLen], vv[kPatLen];
    if (len > 0) {  // the pattern's padding reads src[row]
      const int4 q0 = pq[0], q1 = pq[1];
      xv[0] = xr[q0.x];
      xv[1] = xr[q0.y];
      xv[2] = xr[q0.z];
      xv[3] = xr[q0.w];
      xv[4] = xr[q1.x];
      xv[5] = xr[q1.y];
      xv[6] = xr[q1.z];
      xv[7] = xr[q1.w];
    }
    if (slot < a.ncache) {
      const VT* cv = sm.val + (size_t)(slot * 4 + k) * (kPatLen * 32) + lane;
#pragma unroll
      for (int e = 0; e < kPatLen; ++e)
        if (e < len) vv[e] = cv[e * 32];
    } else {
      const VT* gv = a.sv + (size_t)(tile * 32 + k * 8 + w) * (kPatLen * 32) + lane;
#pragma unroll
      for (int e = 0; e < kPatLen; ++e)
        if (e < len) vv[e] = ld_stream(gv + e * 32);
    }
#pragma unroll
    for (int e = 0; e < kPatLen; ++e)
      if (e < len) t = vadd(t, vmul(vv[e], xv[e]));
  } else {
    constexpr int C = 8;  // entries per round
    const size_t at = (size_t)__ldg(a.sbase + tile * 32 + k * 8 + w) * 32 + lane;
    for (int e0 = 0; e0 < meta; e0 += C) {
      int c[C];
      VT xv[C], vv[C];
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < meta) {
          c[e] = ld_stream(a.sc + at + (e0 + e) * 32);
          vv[e] = ld_stream(a.sv + at + (e0 + e) * 32);
        }
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < meta) xv[e] = src[c[e]];
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < meta) t = vadd(t, vmul(vv[e], xv[e]));
    }
  }
  return t;
}

// Row sums of all of the CTA's rows into sm.v (one 32-row group per warp at
// a time), then a barrier.
template <typename VT, bool PAT>
__device__ __forceinline__ void cta_spmv(const OcArgs<VT>& a, const OcSmem<VT>& sm, const VT* src, int u0, int nu) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int g = warp; g < 4 * nu; g += blockDim.x >> 5)
    sm.v[g * 32 + lane] = row_sum<VT, PAT>(a, sm, src, g >> 2, g & 3, u0 + (g >> 2), lane);
  __syncthreads();
}

// All CTAs' stores so far become visible to all CTAs.  The counter starts at
// -1 (the 0xff fill), so after `epoch` exchanges (from 1) it is epoch G - 1.
template <typename VT>
__device__ __forceinline__ void grid_exchange(const OcArgs<VT>& a, const OcSmem<VT>& sm, unsigned epoch) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.arrive) : "memory");
    unsigned long long t0 = 0;
    for (unsigned i = 0;; ++i) {
      unsigned f;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(a.arrive) : "memory");
      if ((int)(f + 1u - epoch * gridDim.x) >= 0 || !poll_more(i, t0, sm.abort_)) break;
    }
  }
  __syncthreads();
}

// The NR sums whose warp terms are in slot set `set`, in the order of
// grid_finish; the same value in every thread of every CTA.
template <int NR, typename VT>
__device__ __forceinline__ void grid_sum(const OcArgs<VT>& a, const OcSmem<VT>& sm, int set, double (&tot)[NR]) {
  if (blockIdx.x == 0) {
    const double* q = a.slot + (size_t)set * 8 * a.ntiles;
    for (int t = threadIdx.x; t < NR * a.ntiles; t += blockDim.x) sm.tp[t] = tile_sum(q + (size_t)t * 8, sm.abort_);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 8 * NR) {
      const double* tp = sm.tp + (warp >> 3) * a.ntiles;
      double s = 0.0;
      for (int k = (warp & 7) * 32 + lane; k < a.ntiles; k += kLanes) s = dadd(s, tp[k]);
      s = warp_fold(s);
      if (lane == 0) sm.red[warp] = s;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      tot[r] = sm.red[8 * r];
#pragma unroll
      for (int g = 1; g < 8; ++g) tot[r] = dadd(tot[r], sm.red[8 * r + g]);
    }
    if (threadIdx.x < NR) publish(a.total + set + threadIdx.x, threadIdx.x ? tot[NR - 1] : tot[0]);
  } else {
    if (threadIdx.x == 0) {
      unsigned long long t0 = 0, w0, w1;
      for (unsigned i = 0;; ++i) {
        if constexpr (NR == 2) {
          load2(a.total + set, w0, w1);
        } else {
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w0) : "l"(a.total + set) : "memory");
          w1 = 0;
        }
        if ((w0 != kSentinel && w1 != kSentinel) || !poll_more(i, t0, sm.abort_)) break;
      }
      sm.red[0] = __longlong_as_double((long long)w0);
      sm.red[1] = __longlong_as_double((long long)w1);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NR; ++r) tot[r] = sm.red[r];
    __syncthreads();  // before the next sum writes red
  }
}

template <typename VT, bool PAT>
__global__ void __launch_bounds__(kOcThreads, 1) pcg_onchip_kernel(OcArgs<VT> a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const OcSmem<VT> sm(smem, a.ntiles, a.pat_ints, a.slots, a.ncache);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kOcThreads / 32;
  const int nunits = a.ntiles * 8;
  const int u0 = blockIdx.x * a.slots;
  const int nu = max(0, min(a.slots, nunits - u0));
  double* slot_of = a.slot;
  auto slots = [&](int set) { return slot_of + (size_t)set * nunits; };
  unsigned epoch = 1;
  if (threadIdx.x == 0) *sm.abort_ = 0;
  for (int q = threadIdx.x; q < a.pat_ints; q += kOcThreads) sm.pat[q] = a.pat[q];

  // ---- x0, ||b||, row lengths, values --------------------------------------
  for (int sl = warp; sl < nu; sl += nwarps) {
    const int unit = u0 + sl, tile = unit >> 3, w = unit & 7;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = sl * kUnitRows + k * 32 + lane;
      const int row = tile * kTile + k * 256 + w * 32 + lane;
      int meta = 0;
      VT x0 = VT(0), J = VT(0);
      if (row < a.n) {
        meta = a.rp[row + 1] - a.rp[row];
        if constexpr (PAT) meta |= (int)a.pid[row] << 16;
        const VT bi = a.b[row];
        acc = dadd(acc, dmul(D(bi), D(bi)));
        J = a.J[row];
        if (a.x0_mode == CELG_X0_USER) {
          x0 = a.x[row];
        } else {
          x0 = a.x0_mode == CELG_X0_REF_ONES ? VT(1) : VT(0);
          a.x[row] = x0;
        }
      }
      sm.meta[i] = meta;
      sm.x[i] = x0;
      sm.J[i] = J;
      sm.p[i] = sm.r[i] = sm.v[i] = VT(0);
      if constexpr (PAT) {
        if (sl < a.ncache) {
          const size_t s = (size_t)(tile * 32 + k * 8 + w) * (kPatLen * 32) + lane;
          for (int e = 0; e < (meta & 0xffff); ++e)
            sm.val[(size_t)(sl * 4 + k) * (kPatLen * 32) + e * 32 + lane] = a.sv[s + e * 32];
        }
      }
    }
    acc = warp_fold(acc);
    if (lane == 0) publish(slots(kSlotB) + unit, acc);
  }
  grid_exchange(a, sm, epoch++);
  double one[1], two[2];
  grid_sum<1>(a, sm, kSlotB, one);
  const double bnorm = sqrt(one[0]);
  double eps = a.eps_abs;
  if (a.eps_rel > 0.0 && a.eps_rel * bnorm > eps) eps = a.eps_rel * bnorm;

  // ---- r = b - A x, p = J r -------------------------------------------------
  cta_spmv<VT, PAT>(a, sm, a.x, u0, nu);
  for (int sl = warp; sl < nu; sl += nwarps) {
    const int unit = u0 + sl, tile = unit >> 3, w = unit & 7;
    double rp = 0.0, rr = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = sl * kUnitRows + k * 32 + lane;
      const int row = tile * kTile + k * 256 + w * 32 + lane;
      if (row < a.n) {
        const VT ri = R<VT>(__dsub_rn(D(a.b[row]), D(vadd(VT(0), sm.v[i]))));
        const double z = dmul(D(ri), D(sm.J[i]));
        const VT pi = R<VT>(z);
        sm.r[i] = ri;
        sm.p[i] = pi;
        a.p[row] = pi;
        rp = dadd(rp, dmul(D(ri), z));
        rr = dadd(rr, dmul(D(ri), D(ri)));
      }
    }
    rp = warp_fold(rp);
    rr = warp_fold(rr);
    if (lane == 0) {
      publish(slots(kSlotInit) + unit, rp);
      publish(slots(kSlotInit + 1) + unit, rr);
    }
  }
  grid_exchange(a, sm, epoch++);
  grid_sum<2>(a, sm, kSlotInit, two);
  double alpha = two[0], norm = sqrt(two[1]), sigma = 0.0, beta = 0.0, pvd = 0.0, rz = 0.0;
  int iter = 0, err = 0;
  const bool scribe = blockIdx.x == 0 && threadIdx.x == 0;
  if (scribe && a.hist && a.hist_cap > 0) a.hist[0] = norm;
  bool act = iter < a.iter_max && fabs(alpha) > kRealSmall && norm > eps;
  int stop = *(volatile int*)sm.abort_;

  while (act && !stop) {
    // v = A p, p.v
    cta_spmv<VT, PAT>(a, sm, a.p, u0, nu);
    for (int sl = warp; sl < nu; sl += nwarps) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = sl * kUnitRows + k * 32 + lane;
        const VT vi = vadd(VT(0), sm.v[i]);
        sm.v[i] = vi;
        acc = dacc_prod(acc, vi, sm.p[i]);
      }
      acc = warp_fold(acc);
      if (lane == 0) publish(slots(kSlotPv) + u0 + sl, acc);
    }
    grid_sum<1>(a, sm, kSlotPv, one);
    pvd = one[0];
    sigma = alpha / pvd;
    if (!isfinite(sigma)) {
      err = kErrBreakdown;
      act = false;
      break;
    }
    // r += (-sigma) v, r.z, r.r
    const int us = (iter & 1) ? kSlotUpd1 : kSlotUpd0, uo = (iter & 1) ? kSlotUpd0 : kSlotUpd1;
    for (int sl = warp; sl < nu; sl += nwarps) {
      double t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = sl * kUnitRows + k * 32 + lane;
        const VT ri = R<VT>(dadd(D(sm.r[i]), dmul(-sigma, D(sm.v[i]))));
        sm.r[i] = ri;
        const double z = dmul(D(ri), D(sm.J[i]));
        t0 = dadd(t0, dmul(D(ri), z));
        t1 = dadd(t1, dmul(D(ri), D(ri)));
      }
      t0 = warp_fold(t0);
      t1 = warp_fold(t1);
      if (lane == 0) {
        publish(slots(us) + u0 + sl, t0);
        publish(slots(us + 1) + u0 + sl, t1);
      }
    }
    grid_sum<2>(a, sm, us, two);
    rz = two[0];
    beta = rz / alpha;
    alpha = rz;
    norm = sqrt(two[1]);
    ++iter;
    if (scribe && a.hist && iter < a.hist_cap) a.hist[iter] = norm;
    act = iter < a.iter_max && fabs(alpha) > kRealSmall && norm > eps;
    // x += sigma p, p = beta p + J r.  Every CTA has read this iteration's
    // p.v slots and the last iteration's r.z, r.r slots: back to the
    // sentinel, ordered before their next use by the exchange below.
    for (int sl = warp; sl < nu; sl += nwarps) {
      const int unit = u0 + sl, tile = unit >> 3, w = unit & 7;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = sl * kUnitRows + k * 32 + lane;
        const int row = tile * kTile + k * 256 + w * 32 + lane;
        const double pi = D(sm.p[i]);
        sm.x[i] = R<VT>(dadd(D(sm.x[i]), dmul(sigma, pi)));
        if (act) {
          const VT pn = R<VT>(dadd(dmul(beta, pi), dmul(D(sm.r[i]), D(sm.J[i]))));
          sm.p[i] = pn;
          if (row < a.n) a.p[row] = pn;
        }
      }
      if (lane < 3) {
        double* q = slots(lane == 0 ? kSlotPv : uo + lane - 1) + unit;
        *reinterpret_cast<unsigned long long*>(q) = kSentinel;
      }
    }
    if (blockIdx.x == 0 && threadIdx.x < 3) {
      double* q = a.total + (threadIdx.x == 0 ? kSlotPv : uo + threadIdx.x - 1);
      *reinterpret_cast<unsigned long long*>(q) = kSentinel;
    }
    stop = *(volatile int*)sm.abort_;
    if (act) {
      grid_exchange(a, sm, epoch++);
      stop = *(volatile int*)sm.abort_;
    }
  }

  // ---- x out, ||b - A x|| ------------------------------------------------------
  for (int sl = warp; sl < nu; sl += nwarps) {
    const int unit = u0 + sl, tile = unit >> 3, w = unit & 7;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = tile * kTile + k * 256 + w * 32 + lane;
      if (row < a.n) a.x[row] = sm.x[sl * kUnitRows + k * 32 + lane];
    }
  }
  double vres = 0.0;
  if (a.verify && !stop) {
    grid_exchange(a, sm, epoch++);
    cta_spmv<VT, PAT>(a, sm, a.x, u0, nu);
    for (int sl = warp; sl < nu; sl += nwarps) {
      const int unit = u0 + sl, tile = unit >> 3, w = unit & 7;
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = tile * kTile + k * 256 + w * 32 + lane;
        if (row < a.n) {
          const double ri = __dsub_rn(D(a.b[row]), dadd(0.0, D(sm.v[sl * kUnitRows + k * 32 + lane])));
          acc = dadd(acc, dmul(ri, ri));
        }
      }
      acc = warp_fold(acc);
      if (lane == 0) publish(slots(kSlotVer) + unit, acc);
    }
    grid_sum<1>(a, sm, kSlotVer, one);
    vres = bnorm > 0.0 ? sqrt(one[0]) / bnorm : sqrt(one[0]);
  }
  if (scribe) {
    PcgState* o = a.out;
    o->alpha = alpha;
    o->sigma = sigma;
    o->beta = beta;
    o->norm = norm;
    o->bnorm = bnorm;
    o->eps = eps;
    o->pvd = pvd;
    o->rz = rz;
    o->vres = vres;
    o->iter = iter;
    o->active = act ? 1 : 0;
    o->err = *(volatile int*)sm.abort_ ? kErrTimeout : err;
    o->hist_len = iter + 1;
    o->xpend = o->xprev = 0;
    o->sigprev = 0.0;
  }
}

// ---- systems of 0.7 to 2.1 million rows ------------------------------------------
//
// The same loop where only r and p fit on the chip.  As three sweeps a 128^3
// system took 60 us an iteration: 140 bytes a row cross from L2 to the SMs,
// at about 7 TB/s, plus three launches.  With r and p in shared memory it is
// the values, the gathers, v, J (twice) and x.  A CTA has whole tiles, its
// two halves alternate between them (warp w of a half has the tile's rows 32
// w + lane + 256 k), and it publishes tile sums; CTA 0, which folds them all,
// has kWideLess tiles less and their room for the sums where both do not fit.
// us an iteration, sweeps : this kernel (variable coefficients, FP64): 90^3
// 34.8 : 21.9, 104^3 41.3 : 27.0, 120^3 54.8 : 38.4, 128^3 61.3 : 51.5 (the
// working set leaves L2); constant coefficients 128^3 43.8 : 32.9.
constexpr int kWideTiles = 14;  // r and p of 14 tiles: 224 of 227 KB
constexpr int kWideLess = 4;    // 64 KB: two sums of up to 2112 tiles
constexpr int kWidePolls = 9;
constexpr int kWideStatic = (2 * kWideTiles * 8 + 16) * 8 + 64;  // its static shared memory

struct WideArgs {
  OcArgs<double> o;  // slot: kSlotSets x ntiles
  double* v;
  int per;           // tiles of a CTA
  int less;          // of them CTA 0 has not: 0 or kWideLess
};

__host__ __device__ inline int wide_table_bytes(int pat_ints) {
  return ((pat_ints + pat_ints / kPatLen) * 4 + 127) & ~127;
}

// the matrix: int32 columns, row patterns, row table
enum { kFormCols, kFormPat, kFormTable };

// row sum as row_sum, the row's length and pattern from memory
template <int FORM>
__device__ __forceinline__ double wide_row_sum(const OcArgs<double>& a, const int* s_pat, const int* s_len,
                                               const double* src, int row, int lane, int id) {
  double t = 0.0;
  if constexpr (FORM != kFormCols) {
    const int len = s_len[id];
    const double* xr = src + row;
    const int4* pq = reinterpret_cast<const int4*>(s_pat + id * kPatLen);
    double xv[kPatLen], vv[kPatLen];
    if constexpr (FORM == kFormTable) {
      // (the lanes of one pattern share the loads; the table stays in L1)
      const double2* tv = reinterpret_cast<const double2*>(a.rowv + id * kPatLen);
#pragma unroll
      for (int e = 0; e < kPatLen; e += 2) {
        const double2 t2 = __ldg(tv + e / 2);
        vv[e] = t2.x;
        vv[e + 1] = t2.y;
      }
    } else {
      const double* gv = a.sv + (size_t)(row >> 5) * (kPatLen * 32) + lane;
#pragma unroll
      for (int e = 0; e < kPatLen; ++e)
        if (e < len) vv[e] = ld_stream(gv + e * 32);
    }
    const int4 q0 = pq[0], q1 = pq[1];
    xv[0] = xr[q0.x];
    xv[1] = xr[q0.y];
    xv[2] = xr[q0.z];
    xv[3] = xr[q0.w];
    xv[4] = xr[q1.x];
    xv[5] = xr[q1.y];
    xv[6] = xr[q1.z];
    if (len == kPatLen) xv[7] = xr[q1.w];
#pragma unroll
    for (int e = 0; e < kPatLen; ++e)
      if (e < len) t = dadd(t, dmul(vv[e], xv[e]));
  } else {
    constexpr int C = 8;
    const int len = __ldg(a.rp + row + 1) - __ldg(a.rp + row);
    const size_t at = (size_t)__ldg(a.sbase + (row >> 5)) * 32 + lane;
    for (int e0 = 0; e0 < len; e0 += C) {
      int c[C];
      double xv[C], vv[C];
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < len) {
          c[e] = ld_stream(a.sc + at + (e0 + e) * 32);
          vv[e] = ld_stream(a.sv + at + (e0 + e) * 32);
        }
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < len) xv[e] = src[c[e]];
#pragma unroll
      for (int e = 0; e < C; ++e)
        if (e0 + e < len) t = dadd(t, dmul(vv[e], xv[e]));
    }
  }
  return t;
}

template <int FORM>
__device__ __forceinline__ double wide_J(const OcArgs<double>& a, int row) {
  if constexpr (FORM == kFormTable)
    if (a.juni) return a.jval;
  return __ldg(a.J + row);
}

template <int FORM>
__global__ void __launch_bounds__(kOcThreads, 1) pcg_wide_kernel(WideArgs wa) {
  const OcArgs<double>& a = wa.o;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double part[2][kWideTiles][8];
  __shared__ double red[16];
  __shared__ int abort_;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = tid >> 8, w = warp & 7;
  const int nt = a.ntiles, per = wa.per;
  const int own = blockIdx.x == 0 ? per - wa.less : per;
  const int t0 = blockIdx.x == 0 ? 0 : (int)blockIdx.x * per - wa.less;
  const int T = max(0, min(own, nt - t0));
  int* s_pat = reinterpret_cast<int*>(smem);
  int* s_len = s_pat + a.pat_ints;
  double* s_r = reinterpret_cast<double*>(smem + wide_table_bytes(a.pat_ints));
  double* s_p = s_r + (size_t)own * kTile;
  double* s_tp = s_r + (size_t)2 * own * kTile;  // CTA 0
  if (tid == 0) abort_ = 0;
  for (int q = tid; q < a.pat_ints; q += kOcThreads) s_pat[q] = a.pat[q];
  for (int q = tid; q < a.pat_ints / kPatLen; q += kOcThreads) s_len[q] = a.plen[q];
  __syncthreads();
  auto slots = [&](int set) { return a.slot + (size_t)set * nt; };
  OcSmem<double> ex(nullptr, 0, 0, 0, 0);  // grid_exchange wants the flag only
  ex.abort_ = &abort_;
  unsigned epoch = 1;

  // the tile sums of NR warp sums per tile in part[], published
  auto publish_tiles = [&](auto nr, int set) {
    constexpr int NR = decltype(nr)::value;
    __syncthreads();
    for (int q = tid; q < NR * T; q += kOcThreads) {
      const int r = q / T, l = q % T;
      double f = part[r][l][0];
#pragma unroll
      for (int g = 1; g < 8; ++g) f = dadd(f, part[r][l][g]);
      publish(slots(set + r) + t0 + l, f);
    }
  };
  // grid_sum over tile sums
  auto sum = [&](auto nr, int set, double* tot) {
    constexpr int NR = decltype(nr)::value;
    if (blockIdx.x == 0) {
      const double* q = slots(set);
      unsigned long long v[kWidePolls], c0 = 0;
      for (unsigned i = 0;; ++i) {
        bool ok = true;
#pragma unroll
        for (int u = 0; u < kWidePolls; ++u) {
          const int k = tid + u * kOcThreads;
          if (k < NR * nt) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[u]) : "l"(q + k) : "memory");
            ok = ok && v[u] != kSentinel;
          }
        }
        if (ok || !poll_more(i, c0, &abort_)) break;
      }
#pragma unroll
      for (int u = 0; u < kWidePolls; ++u)
        if (tid + u * kOcThreads < NR * nt) s_tp[tid + u * kOcThreads] = __longlong_as_double((long long)v[u]);
      __syncthreads();
      if (warp < 8 * NR) {
        const double* tp = s_tp + (warp >> 3) * nt;
        double s = 0.0;
        for (int k = (warp & 7) * 32 + lane; k < nt; k += kLanes) s = dadd(s, tp[k]);
        s = warp_fold(s);
        if (lane == 0) red[warp] = s;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        tot[r] = red[8 * r];
#pragma unroll
        for (int g = 1; g < 8; ++g) tot[r] = dadd(tot[r], red[8 * r + g]);
      }
      if (tid < NR) publish(a.total + set + tid, tid ? tot[NR - 1] : tot[0]);
      __syncthreads();
    } else {
      if (tid == 0) {
        unsigned long long c0 = 0, w0, w1 = 0;
        for (unsigned i = 0;; ++i) {
          if constexpr (NR == 2) load2(a.total + set, w0, w1);
          else asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w0) : "l"(a.total + set) : "memory");
          if ((w0 != kSentinel && w1 != kSentinel) || !poll_more(i, c0, &abort_)) break;
        }
        red[0] = __longlong_as_double((long long)w0);
        red[1] = __longlong_as_double((long long)w1);
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < NR; ++r) tot[r] = red[r];
      __syncthreads();
    }
  };
  using One = std::integral_constant<int, 1>;
  using Two = std::integral_constant<int, 2>;
  double tot[2];

  // ---- x0, ||b|| ------------------------------------------------------------
  for (int l = half; l < T; l += 2) {
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
      const int i = l * kTile + k * kLanes + w * 32 + lane;
      s_r[i] = s_p[i] = 0.0;
      if (row < a.n) {
        const double bi = a.b[row];
        acc = dadd(acc, dmul(bi, bi));
        if (a.x0_mode != CELG_X0_USER) a.x[row] = a.x0_mode == CELG_X0_REF_ONES ? 1.0 : 0.0;
      }
    }
    acc = warp_fold(acc);
    if (lane == 0) part[0][l][w] = acc;
  }
  publish_tiles(One(), kSlotB);
  grid_exchange(a, ex, epoch++);
  sum(One(), kSlotB, tot);
  const double bnorm = sqrt(tot[0]);
  double eps = a.eps_abs;
  if (a.eps_rel > 0.0 && a.eps_rel * bnorm > eps) eps = a.eps_rel * bnorm;

  // ---- r = b - A x, p = J r -------------------------------------------------
  for (int l = half; l < T; l += 2) {
    double rp = 0.0, rr = 0.0;
    for (int k = 0; k < 4; ++k) {
      const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
      const int i = l * kTile + k * kLanes + w * 32 + lane;
      if (row < a.n) {
        const double s = wide_row_sum<FORM>(a, s_pat, s_len, a.x, row, lane, FORM == kFormCols ? 0 : (int)__ldg(a.pid + row));
        const double ri = __dsub_rn(a.b[row], dadd(0.0, s));
        const double z = dmul(ri, wide_J<FORM>(a, row));
        s_r[i] = ri;
        s_p[i] = z;
        a.p[row] = z;
        rp = dadd(rp, dmul(ri, z));
        rr = dadd(rr, dmul(ri, ri));
      }
    }
    rp = warp_fold(rp);
    rr = warp_fold(rr);
    if (lane == 0) {
      part[0][l][w] = rp;
      part[1][l][w] = rr;
    }
  }
  publish_tiles(Two(), kSlotInit);
  grid_exchange(a, ex, epoch++);
  sum(Two(), kSlotInit, tot);
  double alpha = tot[0], norm = sqrt(tot[1]), sigma = 0.0, beta = 0.0, pvd = 0.0, rz = 0.0;
  int iter = 0, err = 0;
  const bool scribe = blockIdx.x == 0 && tid == 0;
  if (scribe && a.hist && a.hist_cap > 0) a.hist[0] = norm;
  bool act = iter < a.iter_max && fabs(alpha) > kRealSmall && norm > eps;
  int stop = *(volatile int*)&abort_;

  while (act && !stop) {
    // v = A p, p.v; the pattern bytes come a tile ahead
    int id[4];
    auto ids = [&](int l) {
      if constexpr (FORM != kFormCols)
        if (l < T)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            id[k] = (int)__ldg(a.pid + min((t0 + l) * kTile + k * kLanes + w * 32 + lane, a.n - 1));
    };
    ids(half);
    for (int l = half; l < T; l += 2) {
      double acc = 0.0;
      const int now[4] = {id[0], id[1], id[2], id[3]};
      ids(l + 2);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
        if (row < a.n) {
          const double vi = dadd(0.0, wide_row_sum<FORM>(a, s_pat, s_len, a.p, row, lane, now[k]));
          wa.v[row] = vi;
          acc = dadd(acc, dmul(vi, s_p[l * kTile + k * kLanes + w * 32 + lane]));
        }
      }
      acc = warp_fold(acc);
      if (lane == 0) part[0][l][w] = acc;
    }
    publish_tiles(One(), kSlotPv);
    sum(One(), kSlotPv, tot);
    pvd = tot[0];
    sigma = alpha / pvd;
    if (!isfinite(sigma)) {
      err = kErrBreakdown;
      act = false;
      break;
    }
    // r += (-sigma) v, r.z, r.r
    const int us = (iter & 1) ? kSlotUpd1 : kSlotUpd0, uo = (iter & 1) ? kSlotUpd0 : kSlotUpd1;
    for (int l = half; l < T; l += 2) {
      double f0 = 0.0, f1 = 0.0, v[4], J[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
        v[k] = row < a.n ? wa.v[row] : 0.0;
        J[k] = row < a.n ? wide_J<FORM>(a, row) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = l * kTile + k * kLanes + w * 32 + lane;
        const double ri = dadd(s_r[i], dmul(-sigma, v[k]));
        s_r[i] = ri;
        const double z = dmul(ri, J[k]);
        f0 = dadd(f0, dmul(ri, z));
        f1 = dadd(f1, dmul(ri, ri));
      }
      f0 = warp_fold(f0);
      f1 = warp_fold(f1);
      if (lane == 0) {
        part[0][l][w] = f0;
        part[1][l][w] = f1;
      }
    }
    publish_tiles(Two(), us);
    sum(Two(), us, tot);
    rz = tot[0];
    beta = rz / alpha;
    alpha = rz;
    norm = sqrt(tot[1]);
    ++iter;
    if (scribe && a.hist && iter < a.hist_cap) a.hist[iter] = norm;
    act = iter < a.iter_max && fabs(alpha) > kRealSmall && norm > eps;
    // x += sigma p, p = beta p + J r; slots back to the sentinel as in
    // pcg_onchip_kernel
    for (int l = half; l < T; l += 2) {
      double x[4], J[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
        x[k] = row < a.n ? a.x[row] : 0.0;
        J[k] = row < a.n ? wide_J<FORM>(a, row) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
        const int i = l * kTile + k * kLanes + w * 32 + lane;
        if (row < a.n) {
          const double pi = s_p[i];
          a.x[row] = dadd(x[k], dmul(sigma, pi));
          if (act) {
            const double pn = dadd(dmul(beta, pi), dmul(s_r[i], J[k]));
            s_p[i] = pn;
            a.p[row] = pn;
          }
        }
      }
    }
    for (int q = tid; q < 3 * T; q += kOcThreads) {
      const int r = q / T;
      *reinterpret_cast<unsigned long long*>(slots(r == 0 ? kSlotPv : uo + r - 1) + t0 + q % T) = kSentinel;
    }
    if (blockIdx.x == 0 && tid < 3)
      *reinterpret_cast<unsigned long long*>(a.total + (tid == 0 ? kSlotPv : uo + tid - 1)) = kSentinel;
    stop = *(volatile int*)&abort_;
    if (act) {
      grid_exchange(a, ex, epoch++);
      stop = *(volatile int*)&abort_;
    }
  }

  // ---- ||b - A x|| -------------------------------------------------------------
  double vres = 0.0;
  if (a.verify && !stop) {
    grid_exchange(a, ex, epoch++);
    for (int l = half; l < T; l += 2) {
      double acc = 0.0;
      for (int k = 0; k < 4; ++k) {
        const int row = (t0 + l) * kTile + k * kLanes + w * 32 + lane;
        if (row < a.n) {
          const double ri = __dsub_rn(a.b[row], dadd(0.0, wide_row_sum<FORM>(a, s_pat, s_len, a.x, row, lane, FORM == kFormCols ? 0 : (int)__ldg(a.pid + row))));
          acc = dadd(acc, dmul(ri, ri));
        }
      }
      acc = warp_fold(acc);
      if (lane == 0) part[0][l][w] = acc;
    }
    publish_tiles(One(), kSlotVer);
    sum(One(), kSlotVer, tot);
    vres = bnorm > 0.0 ? sqrt(tot[0]) / bnorm : sqrt(tot[0]);
  }
  if (scribe) {
    PcgState* o = a.out;
    o->alpha = alpha;
    o->sigma = sigma;
    o->beta = beta;
    o->norm = norm;
    o->bnorm = bnorm;
    o->eps = eps;
    o->pvd = pvd;
    o->rz = rz;
    o->vres = vres;
    o->iter = iter;
    o->active = act ? 1 : 0;
    o->err = *(volatile int*)&abort_ ? kErrTimeout : err;
    o->hist_len = iter + 1;
    o->xpend = o->xprev = 0;
    o->sigprev = 0.0;
  }
}

// ---- sliced matrix copy -----------------------------------------------------------

// longest row of each slice of 32 rows, and of the matrix
__global__ void slice_width_kernel(int n, long nslices, const int* __restrict__ rp, int* __restrict__ width,
                                   int* __restrict__ longest) {
  const int lane = threadIdx.x & 31;
  for (long s = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5; s < nslices;
       s += ((long)gridDim.x * blockDim.x) >> 5) {
    const long row = s * 32 + lane;
    int len = row < n ? rp[row + 1] - rp[row] : 0;
    for (int off = 16; off >= 1; off >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, off));
    if (lane == 0) {
      width[s] = min(len, kMaxWidth);
      atomicMax(longest, len);
    }
  }
}

// base == nullptr: slices of kPatLen entries a row
template <typename VT>
__global__ void slice_fill_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                  const VT* __restrict__ v, const int* __restrict__ base,
                                  VT* __restrict__ sv, int* __restrict__ sc) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int b = rp[i], len = rp[i + 1] - b;
    const size_t at = (base ? (size_t)base[i >> 5] : (size_t)(i >> 5) * kPatLen) * 32 + (i & 31);
    for (int e = 0; e < len; ++e) {
      sv[at + (size_t)e * 32] = v[b + e];
      if (sc) sc[at + (size_t)e * 32] = ci[b + e];
    }
  }
}

void sell_free(celg_handle* h, CsrDev& A) {
  dev_free(h, A.sell_v);
  dev_free(h, A.sell_v32);
  dev_free(h, A.sell_c);
  dev_free(h, A.sell_base);
  A.sell_v = nullptr;
  A.sell_v32 = nullptr;
  A.sell_c = A.sell_base = nullptr;
  A.sell_total = -1;
}

static double*& sell_vals(CsrDev& A, const double*) { return A.sell_v; }
static float*& sell_vals(CsrDev& A, const float*) { return A.sell_v32; }

// Builds the sliced copy once; *ok = false when its padding is not worth it
// (more than twice the entries plus one slice row per slice: a few very long
// rows among short ones) or there is no memory for it, which leaves the
// matrix to the graph of sweeps.
template <typename VT>
static int ensure_sell(celg_handle* h, CsrDev& A, const VT* vals, bool* ok) {
  *ok = false;
  const bool pat = A.pid != nullptr;
  const long nslices = ntiles_of(A.n) * (kTile / 32);
  if (A.sell_total < 0) {
    if (pat) {
      A.sell_total = nslices * kPatLen * 32;
    } else {
      int *width = nullptr, *base = nullptr;
      void* tmp = nullptr;
      size_t tmp_bytes = 0;
      cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, width, base, (int)nslices + 1, h->stream);
      cudaError_t e = dev_alloc(h, &width, sizeof(int) * (nslices + 1));
      if (e == cudaSuccess) e = dev_alloc(h, &base, sizeof(int) * (nslices + 1));
      if (e == cudaSuccess) e = dev_alloc(h, &tmp, std::max<size_t>(tmp_bytes, 16));
      if (e == cudaSuccess) e = cudaMemsetAsync(width + nslices, 0, sizeof(int), h->stream);
      int total = 0, longest = 0;
      int* longest_d = h->err_d + 5;
      if (e == cudaSuccess) e = cudaMemsetAsync(longest_d, 0, sizeof(int), h->stream);
      if (e == cudaSuccess) {
        slice_width_kernel<<<(int)std::min(nslices / 8 + 1, 2048L), 256, 0, h->stream>>>(A.n, nslices, A.rp, width,
                                                                                        longest_d);
        e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, width, base, (int)nslices + 1, h->stream);
      }
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(&total, base + nslices, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(&longest, longest_d, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
      dev_free(h, width);
      dev_free(h, tmp);
      if (e != cudaSuccess || longest > kMaxWidth || 32L * total > 2L * A.nnz + 32 * nslices) {
        dev_free(h, base);
        if (out_of_memory(e)) return CELG_OK;
        A.sell_total = 0;
        return e != cudaSuccess ? cuda_status(e, "sliced matrix") : CELG_OK;
      }
      A.sell_base = base;
      A.sell_total = 32L * total;
    }
  }
  if (A.sell_total == 0) return CELG_OK;
  VT*& sv = sell_vals(A, vals);
  const bool need_c = !pat && !A.sell_c;
  if (!sv) {
    cudaError_t e = dev_alloc(h, &sv, sizeof(VT) * (size_t)A.sell_total);
    if (e == cudaSuccess && need_c) e = dev_alloc(h, &A.sell_c, sizeof(int) * (size_t)A.sell_total);
    if (e == cudaSuccess) {
      slice_fill_kernel<VT><<<(int)std::min(((long)A.n + 255) / 256, (long)h->sms * 8), 256, 0, h->stream>>>(
          A.n, A.rp, A.ci, vals, pat ? nullptr : A.sell_base, sv, need_c ? A.sell_c : nullptr);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
      sell_free(h, A);
      return out_of_memory(e) ? CELG_OK : cuda_status(e, "sliced matrix");
    }
  }
  *ok = true;
  return CELG_OK;
}

// Most rows a system may have for the one-kernel solve (CELG_ONCHIP_ROWS
// overrides: 0 sends every solve through the graph of sweeps).
static long onchip_max_rows() {
  const char* e = std::getenv("CELG_ONCHIP_ROWS");
  return e ? std::atol(e) : 1L << 30;
}

// A process or a stream can have fewer SMs at its disposal than the device
// reports.  The driver then refuses cooperative grids that cannot all be
// resident, but says so only at a launch (for a captured one, at the graph's),
// and a batch must not be refused half way.  So an empty kernel that fills an
// SM per CTA, as those that matter do, is launched for every new largest grid.
__global__ void __launch_bounds__(kOcThreads, 1) coop_probe_kernel() {}

int coop_fits(celg_handle* h, int grid, bool* fits) {
  *fits = grid <= h->coop_ok;
  if (*fits || (h->coop_no && grid >= h->coop_no)) return CELG_OK;
  const int smem = kOcMaxSmem - 1024;
  if (const int st = allow_dynamic_smem<coop_probe_kernel>(smem)) return st;
  const cudaError_t e =
      cudaLaunchCooperativeKernel((const void*)coop_probe_kernel, dim3(grid), dim3(kOcThreads), nullptr, smem, h->stream);
  *fits = e == cudaSuccess;
  if (*fits) {
    h->coop_ok = grid;
  } else if (e == cudaErrorCooperativeLaunchTooLarge) {
    (void)cudaGetLastError();
    h->coop_no = grid;
  } else {
    CELG_CUDA(e);
  }
  return CELG_OK;
}

template <typename VT, bool PAT>
static int launch_onchip(cudaStream_t stream, const OcArgs<VT>& a, int grid, size_t smem) {
  if (const int st = allow_dynamic_smem<pcg_onchip_kernel<VT, PAT>>((int)smem)) return st;
  OcArgs<VT> arg = a;
  void* params[] = {&arg};
  CELG_CUDA(cudaLaunchCooperativeKernel((const void*)pcg_onchip_kernel<VT, PAT>, dim3(grid), dim3(kOcThreads), params,
                                        smem, stream));
  return CELG_OK;
}

template <int FORM>
static int launch_wide(cudaStream_t stream, const OcArgs<double>& o, double* v, int per, int less, int grid,
                       size_t smem) {
  if (const int st = allow_dynamic_smem<pcg_wide_kernel<FORM>>((int)smem)) return st;
  WideArgs arg{o, v, per, less};
  void* params[] = {&arg};
  CELG_CUDA(cudaLaunchCooperativeKernel((const void*)pcg_wide_kernel<FORM>, dim3(grid), dim3(kOcThreads), params, smem,
                                        stream));
  return CELG_OK;
}

// How a system runs on `sms` SMs, and the doubles of exchange words it needs.
struct OnchipPlan {
  bool wide = false;
  int slots = 0, grid = 0, per = 0, less = 0, ncache = 0;
  size_t smem = 0, nslot = 0;
  size_t words() const { return nslot + (nslot & 1) + kOcTail; }
};

// false: the system does not fit
template <typename VT>
static bool onchip_plan(const CsrDev& A, int sms, OnchipPlan* out) {
  const long n = A.n;
  if (n < 1 || n > onchip_max_rows()) return false;
  const long nt = ntiles_of(n), nunits = nt * 8;
  if (nunits > kOcMaxUnits) return false;
  OnchipPlan q;
  q.slots = (int)((nunits + sms - 1) / sms);
  q.grid = (int)((nunits + q.slots - 1) / q.slots);
  const bool pat = A.pid != nullptr;
  const int pat_ints = pat ? A.npat * kPatLen : 0;
  const size_t base = OcSmem<VT>(nullptr, (int)nt, pat_ints, q.slots, 0).bytes;
  // the wide form, where r and p fit
  q.wide = base > (size_t)kOcMaxSmem;
  if (q.wide) {
    if (sizeof(VT) != 8 || 2 * nt > kWidePolls * kOcThreads) return false;
    // CTA 0's room for the sums: beside its tiles, else in place of some
    for (q.less = 0;; q.less = kWideLess) {
      q.per = (int)((nt + q.less + sms - 1) / sms);
      q.smem = wide_table_bytes(pat_ints) + (size_t)2 * q.per * kTile * 8 + (q.less ? 0 : 2 * nt * 8);
      if (q.per <= kWideTiles && q.per > q.less && q.smem + kWideStatic <= (size_t)kOcMaxSmem) break;
      if (q.less) return false;
    }
    q.grid = (int)((nt + q.less + q.per - 1) / q.per);
    q.nslot = (size_t)kSlotSets * (nt + (nt & 1));
  } else {
    const size_t per_cached = sizeof(VT) * kUnitRows * kPatLen;
    q.ncache = pat ? (int)std::min<size_t>((size_t)q.slots, (kOcMaxSmem - base) / per_cached) : 0;
    q.smem = OcSmem<VT>(nullptr, (int)nt, pat_ints, q.slots, q.ncache).bytes;
    q.nslot = (size_t)kSlotSets * nunits;
  }
  *out = q;
  return true;
}

// What an iteration of such a kernel moves between the SMs and L2: p stored and
// gathered, and the matrix, but for the units whose values are kept; the wide
// form v, x and J too, and (int32 columns) two words of the row pointer.
template <typename VT>
static double onchip_bytes(const CsrDev& A, const OnchipPlan& q) {
  const double vt = sizeof(VT), n = A.n, nnz = A.nnz;
  if (!q.wide) return 2 * vt * n + (A.pid ? vt * nnz * (q.slots - q.ncache) / q.slots : (vt + 4) * nnz);
  const double J = A.rowv && A.juni ? 0.0 : 2 * vt * n;
  return 6 * vt * n + J + (A.rowv ? n : A.pid ? vt * nnz + n : (vt + 4) * nnz + 8 * n);
}

// the sliced values, where the kernel reads them
template <typename VT>
static int onchip_matrix(celg_handle* h, CsrDev& A, const VT* vals, const OnchipPlan& q, bool* ok) {
  *ok = q.wide && row_values<VT>(A);
  return *ok ? CELG_OK : ensure_sell<VT>(h, A, vals, ok);
}

// words: q.words() doubles set to 0xff
template <typename VT>
static int onchip_launch(cudaStream_t stream, CsrDev& A, const PcgBind<VT>& B, const celg_params* p, const OnchipPlan& q,
                         double* words, PcgState* out, double* hist, int hist_cap) {
  OcArgs<VT> a;
  a.n = A.n;
  a.ntiles = (int)ntiles_of(A.n);
  a.slots = q.slots;
  a.ncache = q.ncache;
  a.sv = sell_vals(A, B.vals);
  a.sc = A.sell_c;
  a.sbase = A.sell_base;
  a.rp = A.rp;
  a.pid = A.pid;
  a.pat = A.pat;
  a.pat_ints = A.pid ? A.npat * kPatLen : 0;
  a.plen = A.plen;
  a.rowv = q.wide ? row_values<VT>(A) : nullptr;
  a.juni = B.juni;
  a.jval = B.jval;
  a.b = B.b;
  a.x = B.x;
  a.J = B.J;
  a.p = B.p;
  a.slot = words;
  a.total = words + (q.nslot + (q.nslot & 1));
  a.arrive = reinterpret_cast<unsigned*>(a.total + kSlotSets + 7);
  a.out = out;
  a.hist = hist;
  a.hist_cap = hist_cap;
  a.iter_max = p->iter_max;
  a.x0_mode = p->x0_mode;
  a.verify = B.verify_vals != nullptr;
  a.eps_abs = p->eps_abs;
  a.eps_rel = p->eps_rel;
  if constexpr (sizeof(VT) == 8) {
    if (q.wide) {
      if (a.rowv) return launch_wide<kFormTable>(stream, a, B.v, q.per, q.less, q.grid, q.smem);
      return A.pid ? launch_wide<kFormPat>(stream, a, B.v, q.per, q.less, q.grid, q.smem)
                   : launch_wide<kFormCols>(stream, a, B.v, q.per, q.less, q.grid, q.smem);
    }
  }
  return A.pid ? launch_onchip<VT, true>(stream, a, q.grid, q.smem) : launch_onchip<VT, false>(stream, a, q.grid, q.smem);
}

// *ok = false: no memory for a buffer of the handle's that has to grow to
// `need` doubles
static int onchip_grow(celg_handle* h, double** buf, size_t* cap, size_t need, bool* ok) {
  *ok = true;
  if (need <= *cap) return CELG_OK;
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  cudaFree(*buf);
  *buf = nullptr;
  *cap = 0;
  const cudaError_t e = raw_alloc(h, buf, sizeof(double) * need);
  *ok = !out_of_memory(e);
  if (!*ok) return CELG_OK;
  CELG_CUDA(e);
  *cap = need;
  return CELG_OK;
}

static int onchip_words(celg_handle* h, size_t words, bool* ok) {
  const int st = onchip_grow(h, &h->oc_slots, &h->oc_cap, words, ok);
  if (st || !*ok) return st;
  CELG_CUDA(cudaMemsetAsync(h->oc_slots, 0xff, sizeof(double) * words, h->stream));
  return CELG_OK;
}

template <typename VT>
int pcg_onchip(celg_handle* h, CsrDev& A, const PcgBind<VT>& B, const celg_params* p, int hist_cap, bool* done) {
  *done = false;
  OnchipPlan q;
  if (!onchip_plan<VT>(A, h->sms, &q)) return CELG_OK;
  bool ok = false;
  int st = coop_fits(h, q.grid, &ok);
  if (st || !ok) return st;
  st = onchip_matrix<VT>(h, A, B.vals, q, &ok);
  if (st || !ok) return st;
  st = onchip_words(h, q.words(), &ok);
  if (st || !ok) return st;
  st = onchip_launch<VT>(h->stream, A, B, p, q, h->oc_slots, h->state_h, h->hist_d, hist_cap);
  *done = !st;
  h->last_bytes_per_iter = onchip_bytes<VT>(A, q);
  return st;
}

// ---- many systems ------------------------------------------------------------------
//
// Independent systems as such kernels side by side, each on a share of the
// SMs: the SMs' time goes into exchanges when one small system has them all,
// and about 1.3 million rows at once keep their working set in L2.  1, 2, 4
// or 8 lanes (streams) share the SMs; the largest systems come first, and
// when a lane is through with its class it divides into two of the next, so
// that no lane waits for another.  ms, in common sweeps (batched.cu) : these
// classes : classes of 303k, 151k, 74k rows : of 600k, 300k, 150k : of 1.3M,
// 700k, 350k:
//   64 systems of sides 16..96   170 : 125 : 160 : 149 : 124
//   24 of 84..90                 126 : 100 : 144 : 141 : 100
//   32 of 60..75                76.6 : 57.8 : 83.1 : 66.4 : 60.2
//   16 of 40..100               73.1 : 59.1 : 68.4 : 65.1 : 58.6
//   6 of 88..110                70.4 : 56.4 : 56.4 : 56.4 : 61.8
//   8 of 80..96                 55.9 : 41.9 : 48.9 : 50.8 : 41.9
//   64 of 30..50                26.0 : 20.5 : 22.6 : 20.5 : 20.5
//   12 of 50..56                14.1 : 10.1 : 11.9 : 10.9 : 10.1
//   4 of 60..64                 10.8 : 5.1 : 6.0 : 5.1 : 8.8
constexpr int kOcLanes = 8;
static long lane_rows(int lanes) { return lanes == 1 ? 1L << 30 : lanes == 2 ? 900000 : lanes == 4 ? 500000 : 200000; }

int pcg_onchip_many(celg_handle* h, int count, celg_mat* const* mats, const double* const* b, double* const* x,
                    const celg_params* p, const PcgState** states, bool* done) {
  *done = false;
  struct Job {
    int sys, lanes;
    OnchipPlan q;
    size_t words;
  };
  std::vector<Job> jobs;
  size_t words = 0;
  for (int s = 0; s < count; ++s) {
    CsrDev& A = mats[s]->csr;
    if (A.n == 0) continue;
    Job j;
    j.sys = s;
    j.lanes = 0;
    for (int lanes = kOcLanes; lanes >= 1 && !j.lanes; lanes /= 2)
      if (A.n <= lane_rows(lanes) && onchip_plan<double>(A, std::max(1, h->sms / lanes), &j.q)) j.lanes = lanes;
    if (!j.lanes) return CELG_OK;
    j.words = words;
    words += j.q.words();
    jobs.push_back(j);
  }
  // Which way is faster, from us an iteration of each and iterations that grow
  // with the side: the sweeps take 24 us and the rows of all live systems at
  // 26k a us for as many iterations as the slowest needs; a kernel takes 7 us
  // and its rows at its lane's share of 36k a us.  (64 systems of sides 8..16:
  // 2.2 : 3.1 ms, the sweeps; 8..40 8.9 : 8.1, 16..60 32 : 26.)
  double sweeps = 0.0, slowest = 0.0, kernels = 0.0, longest = 0.0;
  for (const Job& j : jobs) {
    const double n = (double)mats[j.sys]->csr.n, its = std::cbrt(n), t = its * (7.0 + n * j.lanes / 36000.0);
    slowest = std::max(slowest, its);
    sweeps += its * n / 26000.0;
    kernels += t / j.lanes;
    longest = std::max(longest, t);
  }
  if (std::max(kernels, longest) >= sweeps + 24.0 * slowest) return CELG_OK;
  bool ok = true;
  int largest = 0;
  for (const Job& j : jobs) largest = std::max(largest, j.q.grid);
  int st = largest ? coop_fits(h, largest, &ok) : CELG_OK;
  if (st || !ok) return st;
  std::vector<CsrDev*> built;
  for (const Job& j : jobs) {
    CsrDev& A = mats[j.sys]->csr;
    const bool had = A.sell_v != nullptr;
    st = onchip_matrix<double>(h, A, A.v, j.q, &ok);
    if (!had && A.sell_v) built.push_back(&A);
    if (!st && ok) continue;
    // one has none: the sweeps need no copy of the others
    if (!st) CELG_CUDA(cudaStreamSynchronize(h->stream));
    for (CsrDev* B : built) sell_free(h, *B);
    return st;
  }
  // work vectors p and v of every lane, as long as the largest system
  size_t room = 32;
  for (const Job& j : jobs) room = std::max(room, ((size_t)mats[j.sys]->csr.n + 31) & ~(size_t)31);
  const size_t work = 2 * kOcLanes * room;
  st = onchip_grow(h, &h->oc_work, &h->oc_work_cap, work, &ok);
  if (st || !ok) return st;
  if (count > h->oc_states_cap) {
    cudaFreeHost(h->oc_states);
    h->oc_states = nullptr;
    h->oc_states_cap = 0;
    const cudaError_t e = cudaMallocHost(&h->oc_states, sizeof(PcgState) * (size_t)count);
    if (out_of_memory(e)) return CELG_OK;
    CELG_CUDA(e);
    h->oc_states_cap = count;
  }
  for (int l = 0; l < kOcLanes; ++l) {
    if (l && !h->oc_lane[l]) CELG_CUDA(cudaStreamCreateWithFlags(&h->oc_lane[l], cudaStreamNonBlocking));
    if (!h->oc_event[l]) CELG_CUDA(cudaEventCreateWithFlags(&h->oc_event[l], cudaEventDisableTiming));
  }
  st = onchip_words(h, std::max<size_t>(words, 1), &ok);
  if (st || !ok) return st;
  std::stable_sort(jobs.begin(), jobs.end(),
                   [&](const Job& a, const Job& c) { return mats[a.sys]->csr.n > mats[c.sys]->csr.n; });
  double load[kOcLanes] = {};
  auto stream_of = [&](int l) { return l ? h->oc_lane[l] : h->stream; };
  // what stream l does next comes after what stream `from` has been given
  auto follow = [&](int l, int from, cudaEvent_t ev) {
    cudaError_t e = cudaEventRecord(ev, stream_of(from));
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream_of(l), ev, 0);
    if (e != cudaSuccess && !st) st = cuda_status(e, "batch lanes");
  };
  for (int lanes = 1; lanes <= kOcLanes && !st; lanes *= 2) {
    // lane l of the upper half starts where lane l - lanes / 2 is now
    for (int l = lanes / 2; l < lanes && lanes > 1; ++l) {
      const int from = l - lanes / 2;
      if (!st) follow(l, from, h->oc_event[l]);
      load[l] = load[from];
    }
    for (const Job& j : jobs) {
      if (j.lanes != lanes || st) continue;
      celg_mat* m = mats[j.sys];
      int l = 0;
      for (int k = 1; k < lanes; ++k)
        if (load[k] < load[l]) l = k;
      // (iterations grow with the side; an iteration is a fixed part and the
      // rows' share of the memory)
      load[l] += std::cbrt((double)m->csr.n) * (200000.0 + (double)lanes * m->csr.n);
      PcgBind<double> B;
      B.A = &m->csr;
      B.vals = B.verify_vals = m->csr.v;
      B.b = b[j.sys];
      B.x = x[j.sys];
      B.p = h->oc_work + (size_t)(2 * l) * room;
      B.v = h->oc_work + (size_t)(2 * l + 1) * room;
      B.J = m->jacobi;
      B.juni = m->csr.juni;
      B.jval = m->csr.jval;
      st = onchip_launch<double>(stream_of(l), m->csr, B, p, j.q, h->oc_slots + j.words, h->oc_states + j.sys, nullptr, 0);
    }
  }
  for (int l = 1; l < kOcLanes && !st; ++l) follow(0, l, h->oc_event[l]);
  if (st) {
    // the kernels under way use the handle's buffers and the caller's vectors:
    // they end before the error is reported
    for (int l = 0; l < kOcLanes; ++l) cudaStreamSynchronize(stream_of(l));
    (void)cudaGetLastError();
  }
  *states = h->oc_states;
  *done = !st;
  return st;
}

template int pcg_onchip<double>(celg_handle*, CsrDev&, const PcgBind<double>&, const celg_params*, int, bool*);
template int pcg_onchip<float>(celg_handle*, CsrDev&, const PcgBind<float>&, const celg_params*, int, bool*);

}  // namespace celg
