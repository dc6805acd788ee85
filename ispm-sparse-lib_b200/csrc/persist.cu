// Whole PCG solves in one cooperative launch.
//
// A system whose matrices and vectors stay in L2 is not bound by bytes: the
// step kernels of its iteration run a few microseconds each, and most of an
// iteration is launch latency, the ramp and tail of each grid, iterations of
// a captured chunk that run past the stop, and the host's look at the flags
// between chunks.  Here a group of CTAs takes a lane (one system, one
// right-hand side) from b to x: the iteration, its stop test, the FP64
// reliable updates and the restarts all run on the device, the CTAs of a
// group meeting at a counter in global memory between steps that read one
// another's rows.  The lanes of a batch have groups of their own, sized by
// their work, and never wait for one another.
//
// What bounds it: a meeting costs about 1.7 us on 7-point 24^3 (the release waits
// 0.6 us for the step's stores, the count is seen 0.6 us later, the others' sums
// take 0.4) and 2.2 on 27-point 56^3, three a pipelined and five a classic
// iteration: over half of a solve's cycles up to there.  Past it CTAs wait for
// the slowest one's loads (3.5 us on 72^3).  A step's loads come from L2 in a few
// dependent rounds.  So a step's loads go out in blocks
// before the first is used, the slice headers stay in shared memory for the
// whole solve, and a thread takes whole rows with lanes on consecutive ones:
// a diagonal step is one element load, one x load and one multiply-add a row
// with addresses shared by up to four rows (the step kernels' four
// consecutive rows a thread spend most instructions on realigning x windows,
// which pays where HBM sets the pace).
//
// Waits are bounded: a CTA that has polled for PersistParams::wait_cycles sets an
// abort flag that every other wait sees, all CTAs return, and the host reports
// ISPM_ERR_TIMEOUT.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <queue>
#include <type_traits>

#include "cuda_util.cuh"
#include "pcg_state.h"
#include "persist.h"

namespace ispm {
namespace {

constexpr int kSums = 3;

// Matrix words: read once an iteration, kept out of L1 (x lives there).
__device__ __forceinline__ float ld_raw(const float *p)
{
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_raw(const double *p)
{
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ __half ld_raw(const __half *p)
{
  unsigned short v;
  asm("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return __ushort_as_half(v);
}
// Predicated forms (0 where !on): no branch, so a block's loads all issue.
__device__ __forceinline__ float ld_raw_if(const float *p, bool on)
{
  float v;
  asm("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.f32 %0, 0f00000000;\n"
      "@q ld.global.nc.L1::no_allocate.f32 %0, [%1];\n}\n"
      : "=f"(v)
      : "l"(p), "r"((unsigned)on));
  return v;
}
__device__ __forceinline__ double ld_raw_if(const double *p, bool on)
{
  double v;
  asm("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n"
      "@q ld.global.nc.L1::no_allocate.f64 %0, [%1];\n}\n"
      : "=d"(v)
      : "l"(p), "r"((unsigned)on));
  return v;
}
__device__ __forceinline__ __half ld_raw_if(const __half *p, bool on)
{
  unsigned short v;
  asm("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.u16 %0, 0;\n"
      "@q ld.global.nc.L1::no_allocate.u16 %0, [%1];\n}\n"
      : "=h"(v)
      : "l"(p), "r"((unsigned)on));
  return __ushort_as_half(v);
}
__device__ __forceinline__ unsigned ld_col_if(const unsigned *p, bool on)
{
  unsigned v;
  asm("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.u32 %0, 0;\n@q ld.global.nc.u32 %0, [%1];\n}\n"
      : "=r"(v)
      : "l"(p), "r"((unsigned)on));
  return v;
}
// x changes between meetings: volatile, so that no load moves across one.
__device__ __forceinline__ float ld_x(const float *p)
{
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_x(const double *p)
{
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_x_if(const float *p, bool on)
{
  float v;
  asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.f32 %0, 0f00000000;\n"
               "@q ld.global.f32 %0, [%1];\n}\n"
               : "=f"(v)
               : "l"(p), "r"((unsigned)on));
  return v;
}
__device__ __forceinline__ double ld_x_if(const double *p, bool on)
{
  double v;
  asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n"
               "@q ld.global.f64 %0, [%1];\n}\n"
               : "=d"(v)
               : "l"(p), "r"((unsigned)on));
  return v;
}
template <class T, class E> __device__ __forceinline__ T widen(E v)
{
  if constexpr (std::is_same<E, __half>::value)
    return T(__half2float(v));
  else
    return T(v);
}

// What a walk multiplies: a vector, or a combination of two formed as it is
// read (the same value each time, so rows agree on it without it being
// stored first).
template <class T> struct Plain {
  const T *x;
  __device__ __forceinline__ T at(unsigned c) const { return ld_x(x + c); }
  __device__ __forceinline__ T at_if(unsigned c, bool on) const { return ld_x_if(x + c, on); }
};
// x + a y
template <class T> struct Axpy {
  const T *x, *y;
  T a;
  __device__ __forceinline__ T at(unsigned c) const { return fma(a, ld_x(y + c), ld_x(x + c)); }
  __device__ __forceinline__ T at_if(unsigned c, bool on) const
  {
    return fma(a, ld_x_if(y + c, on), ld_x_if(x + c, on));
  }
};

// A tile's header as the walk needs it, kept in shared memory for the whole
// solve: where its entries start, how many there are, and the column (in the
// lane) that its first row meets under each diagonal.
struct Tile {
  unsigned e0, c0, nc, nd;  // elements and columns of the tile's first row
  unsigned inside;          // diagonals whose columns all lie in the lane
  unsigned pos[kPersistMaxDiag];
};

// One group's view of itself and the sums its CTAs agree on.
template <int V, int LP, bool WIDE> struct Group {
  const PersistParams &P;
  const PersistLane &L;  // in shared memory
  double *sh;            // shared: kSums x 32 warp sums, then as many of the readers
  int *ok;               // shared: a word per reading warp
  Tile *tiles;           // shared: A, G, Ht of each of the CTA's tiles
  int cta = 0;           // this CTA's place in the group
  int r0 = 0, r1 = 0;    // its rows
  unsigned *bar = nullptr;  // the group's count of arrivals
  unsigned epoch = 0;       // meetings so far
  bool dead = false;     // a wait ran out (uniform over the CTA)

  __device__ Group(const PersistParams &p, const PersistLane &l, double *s, int *o, Tile *t)
      : P(p), L(l), sh(s), ok(o), tiles(t)
  {
  }

  static constexpr int kTileRows = 32 * V >> LP;

  __device__ void start(int slot)
  {
    cta = (int)blockIdx.x - L.cta0;
    bar = P.bar + slot;
    const int units = L.rows / 32;
    // in whole tiles of the walk where rows allow it (r0 sits on a tile)
    const int strips = (units + V - 1) / V;
    r0 = min(units, (int)((long long)strips * cta / L.ncta) * V) * 32;
    r1 = min(units, (int)((long long)strips * (cta + 1) / L.ncta) * V) * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_tiles = (r1 - r0 + kTileRows - 1) / kTileRows;
    for (int k = warp; k < 3 * n_tiles; k += nw) {
      const int which = k / n_tiles, t = k - which * n_tiles;
      if (which > 0 && !P.have_prec)
        break;
      const PersistOp &op = which == 0 ? L.A : which == 1 ? L.G : L.Ht;
      tile_header(op, r0 + t * kTileRows, tiles[which * P.max_tiles + t], lane);
    }
    __syncthreads();
  }

  __device__ void tile_header(const PersistOp &op, int base, Tile &t, int lane)
  {
    const unsigned lh = op.log2h, S = 1u << lh, n = (unsigned)L.rows;
    const unsigned slice = op.slice0 + ((unsigned)base >> lh), r = (unsigned)base & (S - 1);
    unsigned e0, c0, nc, nd = 0, d0 = 0;
    if (op.diag) {
      const unsigned *rec = op.sp + 3 * (size_t)slice;
      e0 = __ldg(rec), c0 = __ldg(rec + 1), d0 = __ldg(rec + 2);
      nc = (__ldg(rec + 4) - c0) >> lh;
      nd = ((__ldg(rec + 3) - e0) >> lh) - nc;
    } else {
      c0 = e0 = __ldg(op.sp + slice);
      nc = (__ldg(op.sp + slice + 1) - e0) >> lh;
    }
    unsigned inside = 0;
    for (unsigned kb = 0; kb < nd; kb += 32) {
      const bool have = kb + lane < nd;
      const unsigned w0 = have ? __ldg(op.sp + d0 + kb + lane) - S - op.col0 + r : 0u;
      if (kb + lane < (unsigned)kPersistMaxDiag)
        t.pos[kb + lane] = w0;
      if (kb == 0)
        inside = __ballot_sync(0xffffffffu, have && w0 < n && n - w0 >= (unsigned)kTileRows);
    }
    if (lane == 0) {
      t.e0 = e0 + r;
      t.c0 = c0 + r;
      t.nc = nc;
      t.nd = nd;
      t.inside = inside;
    }
  }

  // The CTAs of a group meet: each leaves its N partial sums, counts itself in
  // and waits for the count; then every CTA adds all CTAs' partials, a thread
  // a CTA.  What was written before a meeting is visible after it.  (Polling
  // every CTA's own word instead of one count floods L2: 148 x 148 words.)
  // v: in, this thread's part; out, the group's sums, the same bits in every
  // thread (warp sums, the CTA's, then all CTAs' in a fixed order).
  template <int N> __device__ __forceinline__ void meet_sum(double (&v)[N > 0 ? N : 1])
  {
    constexpr int M = N > 0 ? N : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // sums over the warp's lanes; several at once share the exchanges (each
    // half of the lanes goes on with half of the sums)
    auto warp_sum = [lane](double (&a)[M]) {
      constexpr unsigned full = 0xffffffffu;
      if constexpr (M == 1) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
          a[0] += __shfl_xor_sync(full, a[0], off);
      } else {
        const bool hi = lane & 16, hi2 = lane & 8;
        double b = (hi ? a[1] : a[0]) + __shfl_xor_sync(full, hi ? a[0] : a[1], 16);
        if constexpr (M == 3) {
          const double c = a[2] + __shfl_xor_sync(full, a[2], 16);
          b = (hi2 ? c : b) + __shfl_xor_sync(full, hi2 ? b : c, 8);
        } else {
          b += __shfl_xor_sync(full, b, 8);
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1)
          b += __shfl_xor_sync(full, b, off);
        a[0] = __shfl_sync(full, b, 0);
        a[1] = __shfl_sync(full, b, 16);
        if constexpr (M == 3)
          a[2] = __shfl_sync(full, b, 8);
      }
    };
    if constexpr (N > 0) {
      warp_sum(v);
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; k++)
          sh[32 * k + warp] = v[k];
    }
    epoch++;
    __syncthreads();
    if (L.ncta == 1) {
      if constexpr (N > 0) {
        double a[M];
#pragma unroll
        for (int k = 0; k < N; k++)
          a[k] = lane < nw ? sh[32 * k + lane] : 0.0;
        warp_sum(a);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < N; k++)
          v[k] = a[k];
      }
      return;
    }
    // two sets of partials in turn: a CTA may still read the last meeting's
    double *part = P.part + ((size_t)(epoch & 1) * P.n_ctas + L.cta0) * kSums;
    if (warp == 0) {
      if constexpr (N > 0) {
        double a[M];
#pragma unroll
        for (int k = 0; k < N; k++)
          a[k] = lane < nw ? sh[32 * k + lane] : 0.0;
        warp_sum(a);
        if (lane == 0)
#pragma unroll
          for (int k = 0; k < N; k++)
            part[cta * kSums + k] = a[k];
      }
      if (lane == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
    const unsigned target = epoch * (unsigned)L.ncta;
    const int readers = N > 0 ? min((L.ncta + 31) >> 5, nw) : 1;  // warps that wait
    if (warp < readers) {
      int good = 1;
      const long long t0 = clock64();
      for (;;) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
        if (__all_sync(0xffffffffu, (int)(c - target) >= 0))
          break;
        const long long waited = clock64() - t0;
        if (waited > P.wait_cycles) {
          atomicExch(P.abort, 1u);
          good = 0;
        } else if (waited > P.wait_cycles / 1000) {
          unsigned stop;
          asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];"
                       : "=r"(stop)
                       : "l"(P.abort)
                       : "memory");
          good = !stop;
        }
        good = __all_sync(0xffffffffu, good);
        if (!good)
          break;
      }
      if constexpr (N > 0) {
        double s[M];
#pragma unroll
        for (int k = 0; k < N; k++)
          s[k] = 0.0;
        for (int c = threadIdx.x; c < L.ncta; c += 32 * readers)
#pragma unroll
          for (int k = 0; k < N; k++)
            s[k] += __ldcg(part + c * kSums + k);
        warp_sum(s);
        if (lane == 0)
#pragma unroll
          for (int k = 0; k < N; k++)
            sh[32 * (kSums + k) + warp] = s[k];
      }
      if (lane == 0)
        ok[warp] = good;
    }
    __syncthreads();
    int good = 1;
    for (int q = 0; q < readers; q++)
      good &= ok[q];
    dead = dead || !good;
    if constexpr (N > 0) {
#pragma unroll
      for (int k = 0; k < N; k++) {
        double a = 0.0;
        for (int q = 0; q < readers; q++)
          a += sh[32 * (kSums + k) + q];
        v[k] = a;
      }
    }
  }

  __device__ __forceinline__ void meet()
  {
    double none[1];
    meet_sum<0>(none);
  }

  template <int N> __device__ __forceinline__ void sum(double (&v)[N]) { meet_sum<N>(v); }

  template <class F> __device__ __forceinline__ void rows(F f)
  {
    for (int i = r0 + (int)threadIdx.x; i < r1; i += (int)blockDim.x)
      f(i);
  }

  // f(row, (op x)_row) for this CTA's rows.  x: coherent loads (the group
  // writes it between meetings).
  //
  // V > 1: a warp takes 32 V consecutive rows, lane l rows l, l + 32, ...: one
  // column and one pair of addresses serve V element and V x loads.  V = 1
  // with 2^LP threads a row where rows are few.  Entries go in blocks whose
  // loads are all issued before the first is used.
  // `which`: the operator's set of tile headers (0 A, 1 G, 2 Ht), or -1 to
  // read them anew (A64, once a phase).
  template <class T, class E, class F>
  __device__ __forceinline__ void spmv(const PersistOp &op, int which, const T *x, F f)
  {
    spmv<T, E>(op, which, Plain<T>{x}, [](int) { return 0; }, [&](int i, T v, int) { f(i, v); });
  }

  // pre(row): what f needs of the row besides the product, loaded before the
  // walk where a thread has one row (its latency then overlaps the walk's).
  template <class T, class E, class X, class Pre, class F>
  __device__ __forceinline__ void spmv(const PersistOp &op, int which, const X x, Pre pre, F f)
  {
    constexpr int rpw = kTileRows;         // rows a warp takes at once
    constexpr int U = (WIDE ? 16 : 8) / V;  // entries a block
    constexpr unsigned np = 1u << LP;
    const unsigned *cols = op.cols;
    const E *elms = static_cast<const E *>(op.elms);
    const unsigned lh = op.log2h, n = (unsigned)L.rows, col0 = op.col0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned mine = LP ? lane & (rpw - 1) : lane, part = LP ? lane / rpw : 0;
    for (int base = r0 + warp * rpw; base < r1; base += nw * rpw) {
      // (the last tile of a CTA may be short: rows in whole groups of 32)
      const int live = LP ? 1 : min(V, (r1 - base) >> 5);
      const Tile *tp = tiles + 3 * P.max_tiles + warp;
      if (which >= 0) {
        tp = tiles + which * P.max_tiles + (base - r0) / rpw;
      } else {
        __syncwarp();
        tile_header(op, base, tiles[3 * P.max_tiles + warp], lane);
        __syncwarp();
      }
      const Tile &t = *tp;
      const unsigned nc = t.nc, nd = t.nd, inside = t.inside;
      decltype(pre(0)) own;
      if (V == 1 && part == 0)
        own = pre(base + (int)mine);
      T acc[V];
#pragma unroll
      for (int v = 0; v < V; v++)
        acc[v] = T(0);
      const E *e = elms + t.e0 + mine;
      if (nc) {
        const unsigned *cc = cols + t.c0 + mine;
        for (unsigned k = 0; k < nc; k += U * np) {
          unsigned cv[U][V];
          E ev[U][V];
          T xv[U][V];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const unsigned kk = k + u * np + part, at = kk << lh;
#pragma unroll
            for (int v = 0; v < V; v++) {
              const bool have = kk < nc && v < live;
              cv[u][v] = ld_col_if(cc + at + 32 * v, have) - col0;
              ev[u][v] = ld_raw_if(e + at + 32 * v, have);
              cv[u][v] = have ? cv[u][v] : 0xffffffffu;
            }
          }
#pragma unroll
          for (int u = 0; u < U; u++)
#pragma unroll
            for (int v = 0; v < V; v++)
              xv[u][v] = x.at_if(cv[u][v], cv[u][v] < n);
#pragma unroll
          for (int u = 0; u < U; u++)
#pragma unroll
            for (int v = 0; v < V; v++)
              acc[v] = fma(widen<T>(ev[u][v]), xv[u][v], acc[v]);
        }
        e += nc << lh;
      }
      auto block = [&](auto width, bool whole, unsigned k) {
        constexpr int N = decltype(width)::value;
        E ev[N][V];
        T xv[N][V];
        if (whole) {
#pragma unroll
          for (int u = 0; u < N; u++) {
            const unsigned kk = k + u * np + part;
            const unsigned c = t.pos[kk] + mine;
            const E *ep = e + (kk << lh);
#pragma unroll
            for (int v = 0; v < V; v++) {
              ev[u][v] = ld_raw(ep + 32 * v);
              xv[u][v] = x.at(c + 32u * v);
            }
          }
        } else {
#pragma unroll
          for (int u = 0; u < N; u++) {
            const unsigned kk = k + u * np + part;
            const unsigned c = t.pos[kk < nd ? kk : 0u] + mine;
            const E *ep = e + (kk << lh);
#pragma unroll
            for (int v = 0; v < V; v++) {
              // (32-bit: c wraps below the lane's first column)
              const unsigned cv = c + 32u * v;
              const bool in = kk < nd && v < live && cv < n;
              ev[u][v] = ld_raw_if(ep + 32 * v, in);
              xv[u][v] = x.at_if(cv, in);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < N; u++)
#pragma unroll
          for (int v = 0; v < V; v++)
            acc[v] = fma(widen<T>(ev[u][v]), xv[u][v], acc[v]);
      };
      constexpr int N2 = U > 2 ? U / 2 : 1;
      // (uniform over the warp: k, nd and the mask are; the mask covers the
      // first 32 diagonals)
      for (unsigned k = 0; k < nd;) {
        const unsigned left = nd - k;
        if (left >= U * np) {
          constexpr unsigned want = U * np >= 32 ? ~0u : (1u << (U * np % 32)) - 1;
          block(std::integral_constant<int, U>(),
                live == V && k + U * np <= 32 && ((inside >> k) & want) == want, k);
          k += U * np;
        } else {
          constexpr unsigned want = N2 * np >= 32 ? ~0u : (1u << (N2 * np % 32)) - 1;
          block(std::integral_constant<int, N2>(),
                live == V && left >= N2 * np && k + N2 * np <= 32 &&
                    ((inside >> k) & want) == want,
                k);
          k += N2 * np;
        }
      }
      if constexpr (LP > 0)
        for (int off = rpw; off < 32; off <<= 1)
          acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
#pragma unroll
      for (int v = 0; v < V; v++)
        if (part == 0 && v < live) {
          if constexpr (std::is_same<E, __half>::value)
            acc[v] *= op.inv_scale;
          const int row = base + (int)mine + 32 * v;
          if constexpr (V == 1)
            f(row, acc[v], own);
          else
            f(row, acc[v], pre(row));
        }
    }
  }
};

// How a phase of iterations ended, from the recursive residual (cg_flags).
__device__ __forceinline__ int stop_of(double rr, double thresh2, double ru2ref, int it, int max_it)
{
  return !isfinite(rr)    ? kBreakdown
         : rr <= thresh2  ? kConverged
         : rr < ru2ref    ? kReplace
         : it >= max_it   ? kCap
                          : kRunning;
}

// The outer loop around phases of an inner recurrence: x = 0, r = b; then a
// phase from the true residual, x += d, r = b - A x in FP64, until the true
// residual meets the tolerance or the accounting stops it.  phase(restart,
// thresh2, max_it, it, rr) runs one and returns how it ended.
template <class T, class G, class Phase>
__device__ __forceinline__ void outer(G &g, int slot, const T *d, Phase phase)
{
  const PersistParams &P = g.P;
  const PersistLane &L = g.L;
  double *r64 = P.r64 + L.row0, *x = P.x + L.row0;
  const double *b = P.b + L.row0;
  const int n = L.n;
  double v[1] = {0.0};
  g.rows([&](int i) {
    const double bi = i < n ? b[i] : 0.0;
    x[i] = 0.0;
    r64[i] = bi;
    v[0] = fma(bi, bi, v[0]);
  });
  g.sum(v);
  PersistOut o{};
  o.bnorm = sqrt(v[0]);
  o.status = ISPM_OK;
  o.rel = o.bnorm > 0.0 ? 1.0 : 0.0;
  const bool usable = isfinite(o.bnorm);
  if (!usable) {
    o.rel = o.bnorm;
    o.status = ISPM_ERR_INVALID;
  }
  const double target = P.tol * o.bnorm, thresh2 = 0.25 * target * target;
  bool restart = true;
  int it = 0, since = 0;
  while (usable && (P.batch ? o.bnorm > 0.0 : o.rel > P.tol)) {
    if (!P.batch && (o.replacements + o.restarts >= P.max_refinements ||
                     o.iterations >= P.max_iters)) {
      o.status = ISPM_ERR_NOT_CONVERGED;
      break;
    }
    const int max_it = P.batch ? P.max_iters
                               : P.max_iters - o.iterations + (restart ? 0 : since);
    if (restart && !P.batch)
      it = since = 0;
    double rr = 0.0;
    const int done = phase(restart, thresh2, max_it, it, rr);
    if (g.dead)
      return;
    o.iterations += it - since;
    since = it;
    g.rows([&](int i) {
      if (i < n)
        x[i] += (double)d[i];
    });
    g.meet();
    v[0] = 0.0;
    g.template spmv<double, double>(L.A64, -1, x, [&](int i, double ax) {
      const double r = i < n ? b[i] - ax : 0.0;
      r64[i] = r;
      v[0] = fma(r, r, v[0]);
    });
    g.sum(v);
    if (g.dead)
      return;
    const double rel = sqrt(v[0]) / o.bnorm, before = o.rel;
    if (P.history && g.cta == 0 && threadIdx.x == 0 && o.n_history < P.history_cap)
      P.history[o.n_history] = rel;
    o.n_history++;
    o.rel = rel;
    if (P.batch) {
      if (rel <= P.tol)
        break;
      if (done == kCap || it >= P.max_iters ||
          o.replacements + o.restarts >= P.max_refinements) {
        o.status = ISPM_ERR_NOT_CONVERGED;
        break;
      }
      restart = done == kBreakdown;
      if (restart) {
        o.restarts++;
        if (!(rel < before) && o.restarts > 2) {
          o.status = ISPM_ERR_BREAKDOWN;
          break;
        }
      } else {
        o.replacements++;
        // the recursive residual ran far below the true one: the old
        // direction no longer fits
        restart = !(v[0] <= 4.0 * rr);
      }
    } else if (done == kBreakdown) {
      o.restarts++;
      restart = true;
      if (!(rel < before) && o.restarts > 2) {
        o.status = ISPM_ERR_BREAKDOWN;
        break;
      }
    } else if (done == kCap) {
      o.status = ISPM_ERR_NOT_CONVERGED;
      break;
    } else {
      o.replacements++;
      restart = false;
    }
  }
  if (g.cta == 0 && threadIdx.x == 0)
    P.out[slot] = o;
}

// Classic PCG (the recurrence of pcg.cu's cg_* kernels).
template <class T, class E, class G>
__device__ __forceinline__ void solve_classic(G &g, int slot)
{
  const PersistParams &P = g.P;
  const PersistLane &L = g.L;
  auto vec = [&](int k) { return static_cast<T *>(P.vec[k]) + L.row0; };
  T *R = vec(0), *Pv = vec(1), *Q = vec(2), *D = vec(3), *Z = vec(4), *TT = vec(5);
  const double *r64 = P.r64 + L.row0;
  const bool prec = P.have_prec != 0;
  double rz = 0.0;  // r.z of the current direction
  bool fresh = true;
  outer<T>(g, slot, D, [&](bool restart, double thresh2, int max_it, int &it, double &rr) {
    double v1[1] = {0.0};
    g.rows([&](int i) {
      const T ri = (T)r64[i];
      R[i] = ri;
      D[i] = T(0);
      v1[0] = fma((double)ri, (double)ri, v1[0]);
    });
    g.sum(v1);
    rr = v1[0];
    const double ru2ref = P.ru2 * rr;
    if (restart)
      fresh = true;
    int done = rr <= thresh2 ? kConverged : kRunning;
    double rzn = rr;
    while (!done && !g.dead) {
      if (prec) {  // z = G^T (G r), r.z and r.r
        g.template spmv<T, E>(L.G, 1, R, [&](int i, T v) { TT[i] = v; });
        g.meet();
        double v2[2] = {0.0, 0.0};
        g.template spmv<T, E>(L.Ht, 2, Plain<T>{TT}, [&](int i) { return R[i]; }, [&](int i, T v, T r) {
          const double ri = (double)r;
          Z[i] = v;
          v2[0] = fma((double)v, ri, v2[0]);
          v2[1] = fma(ri, ri, v2[1]);
        });
        g.sum(v2);
        rzn = v2[0];
        rr = v2[1];
        done = stop_of(rr, thresh2, ru2ref, it, max_it);
        if (done)
          break;
      }
      const double beta = fresh ? 0.0 : rzn / rz;
      if (!(rzn > 0.0) || !isfinite(beta)) {
        done = rzn == 0.0 ? kConverged : kBreakdown;
        break;
      }
      const T bt = (T)beta;
      const T *z = prec ? Z : R;
      if (fresh)
        g.rows([&](int i) { Pv[i] = z[i]; });
      else
        g.rows([&](int i) { Pv[i] = fma(bt, Pv[i], z[i]); });
      g.meet();
      double pq[1] = {0.0};
      g.template spmv<T, T>(L.A, 0, Plain<T>{Pv}, [&](int i) { return Pv[i]; }, [&](int i, T v, T pi) {
        Q[i] = v;
        pq[0] = fma((double)v, (double)pi, pq[0]);
      });
      g.sum(pq);
      const double alpha = rzn / pq[0];
      if (!(alpha > 0.0) || !isfinite(alpha)) {
        done = kBreakdown;
        break;
      }
      rz = rzn;
      fresh = false;
      it++;
      const T a = (T)alpha;
      v1[0] = 0.0;
      g.rows([&](int i) {
        const T ri = fma(-a, Q[i], R[i]);
        R[i] = ri;
        D[i] = fma(a, Pv[i], D[i]);
        v1[0] = fma((double)ri, (double)ri, v1[0]);
      });
      if (prec) {
        g.meet();
      } else {
        g.sum(v1);
        rzn = rr = v1[0];
        done = stop_of(rr, thresh2, ru2ref, it, max_it);
      }
    }
    return done;
  });
}

// The same for systems of few rows, where meetings are most of the time: the
// new direction and the new residual are formed where they are gathered (p =
// z + beta p in A p, r - alpha q in G r), each row stored by its owner beside
// the old ones, so an iteration has three meetings instead of five.  4,096
// rows: 0.55 against 0.63 ms a solve; at 64,000 rows and more the second
// gather costs more than the meetings (0.83 against 0.80 ms, 27-point 40^3).
template <class T, class E, class G> __device__ __forceinline__ void solve_classic_few(G &g, int slot)
{
  const PersistParams &P = g.P;
  const PersistLane &L = g.L;
  auto vec = [&](int k) { return static_cast<T *>(P.vec[k]) + L.row0; };
  T *R = vec(0), *Pv = vec(1), *Q = vec(2), *D = vec(3), *Z = vec(4), *TT = vec(5);
  T *Rn = vec(6), *Pn = vec(7);
  const double *r64 = P.r64 + L.row0;
  const bool prec = P.have_prec != 0;
  double rz = 0.0;  // r.z of the current direction
  bool fresh = true;
  outer<T>(g, slot, D, [&](bool restart, double thresh2, int max_it, int &it, double &rr) {
    double v1[1] = {0.0};
    g.rows([&](int i) {
      const T ri = (T)r64[i];
      R[i] = ri;
      D[i] = T(0);
      v1[0] = fma((double)ri, (double)ri, v1[0]);
    });
    g.sum(v1);
    rr = v1[0];
    const double ru2ref = P.ru2 * rr;
    if (restart)
      fresh = true;
    int done = rr <= thresh2 ? kConverged : kRunning;
    double rzn = rr;
    if (prec && !done) {
      g.template spmv<T, E>(L.G, 1, R, [&](int i, T v) { TT[i] = v; });
      g.meet();
    }
    while (!done && !g.dead) {
      if (prec) {  // z = G^T (G r), r.z and r.r
        double v2[2] = {0.0, 0.0};
        g.template spmv<T, E>(L.Ht, 2, Plain<T>{TT}, [&](int i) { return R[i]; },
                              [&](int i, T v, T r) {
                                const double ri = (double)r;
                                Z[i] = v;
                                v2[0] = fma((double)v, ri, v2[0]);
                                v2[1] = fma(ri, ri, v2[1]);
                              });
        g.sum(v2);
        rzn = v2[0];
        rr = v2[1];
        done = stop_of(rr, thresh2, ru2ref, it, max_it);
        if (done)
          break;
      }
      const double beta = fresh ? 0.0 : rzn / rz;
      if (!(rzn > 0.0) || !isfinite(beta)) {
        done = rzn == 0.0 ? kConverged : kBreakdown;
        break;
      }
      // p = z + beta p, q = A p, p.q
      double pq[1] = {0.0};
      const T *z = prec ? Z : R;
      const T bt = (T)beta;
      if (fresh) {
        g.template spmv<T, T>(L.A, 0, Plain<T>{z}, [&](int i) { return z[i]; },
                              [&](int i, T v, T pi) {
                                Q[i] = v;
                                Pn[i] = pi;
                                pq[0] = fma((double)v, (double)pi, pq[0]);
                              });
      } else {
        g.template spmv<T, T>(L.A, 0, Axpy<T>{z, Pv, bt},
                              [&](int i) { return fma(bt, Pv[i], z[i]); },
                              [&](int i, T v, T pi) {
                                Q[i] = v;
                                Pn[i] = pi;
                                pq[0] = fma((double)v, (double)pi, pq[0]);
                              });
      }
      {
        T *const old = Pv;
        Pv = Pn;
        Pn = old;
      }
      g.sum(pq);
      const double alpha = rzn / pq[0];
      if (!(alpha > 0.0) || !isfinite(alpha)) {
        done = kBreakdown;
        break;
      }
      rz = rzn;
      fresh = false;
      it++;
      const T a = (T)alpha;
      if (prec) {  // r -= alpha q, d += alpha p, t = G r
        struct Own {
          T r, d;
        };
        g.template spmv<T, E>(
            L.G, 1, Axpy<T>{R, Q, -a},
            [&](int i) { return Own{fma(-a, Q[i], R[i]), fma(a, Pv[i], D[i])}; },
            [&](int i, T v, const Own &o) {
              TT[i] = v;
              Rn[i] = o.r;
              D[i] = o.d;
            });
        T *const old = R;
        R = Rn;
        Rn = old;
        g.meet();
      } else {
        v1[0] = 0.0;
        g.rows([&](int i) {
          const T ri = fma(-a, Q[i], R[i]);
          R[i] = ri;
          D[i] = fma(a, Pv[i], D[i]);
          v1[0] = fma((double)ri, (double)ri, v1[0]);
        });
        g.sum(v1);
        rzn = rr = v1[0];
        done = stop_of(rr, thresh2, ru2ref, it, max_it);
      }
    }
    return done;
  });
}

// Pipelined PCG (the recurrence of pcg.cu's pcg_step_kernel; after a reliable
// update the auxiliaries are derived again from the directions).
template <class T, class E, class G>
__device__ __forceinline__ void solve_pipelined(G &g, int slot)
{
  const PersistParams &P = g.P;
  const PersistLane &L = g.L;
  auto vec = [&](int k) { return static_cast<T *>(P.vec[k]) + L.row0; };
  T *R = vec(0), *U = vec(1), *W = vec(2), *M = vec(3), *Pv = vec(4), *Sv = vec(5), *Q = vec(6),
    *Z = vec(7), *D = vec(8), *TT = vec(9);
  const double *r64 = P.r64 + L.row0;
  const bool prec = P.have_prec != 0;
  double gammaold = 0.0, alpha_old = 0.0;
  // out = M in
  auto apply_m = [&](const T *in, T *out) {
    if (!prec) {
      g.rows([&](int i) { out[i] = in[i]; });
    } else {
      g.template spmv<T, E>(L.G, 1, in, [&](int i, T v) { TT[i] = v; });
      g.meet();
      g.template spmv<T, E>(L.Ht, 2, TT, [&](int i, T v) { out[i] = v; });
    }
    g.meet();
  };
  auto apply_a = [&](const T *in, T *out) {
    g.template spmv<T, T>(L.A, 0, in, [&](int i, T v) { out[i] = v; });
  };
  outer<T>(g, slot, D, [&](bool restart, double thresh2, int max_it, int &it, double &rr) {
    g.rows([&](int i) {
      R[i] = (T)r64[i];
      D[i] = T(0);
      if (restart)
        Pv[i] = Sv[i] = Q[i] = Z[i] = T(0);
    });
    g.meet();
    apply_m(R, U);
    apply_a(U, W);
    if (!restart) {
      apply_a(Pv, Sv);
      g.meet();
      apply_m(Sv, Q);
      apply_a(Q, Z);
    }
    double v[3] = {0.0, 0.0, 0.0};
    __syncthreads();  // rows() and spmv() give a row to different threads
    g.rows([&](int i) {
      const double ri = R[i], ui = U[i], wi = W[i];
      v[0] = fma(ri, ui, v[0]);
      v[1] = fma(wi, ui, v[1]);
      v[2] = fma(ri, ri, v[2]);
    });
    g.sum(v);
    const double ru2ref = P.ru2 * v[2];
    bool first = restart || it == 0;
    if (restart)
      gammaold = alpha_old = 0.0;
    int done = v[2] <= thresh2 ? kConverged : kRunning;
    while (!done && !g.dead) {
      const double gamma = v[0], delta = v[1];
      const double beta = first ? 0.0 : gamma / gammaold;
      const double alpha = first ? gamma / delta : gamma / (delta - beta * gamma / alpha_old);
      if (!(alpha > 0.0) || !isfinite(alpha) || !isfinite(beta)) {
        done = kBreakdown;
        break;
      }
      apply_m(W, M);
      const T a = (T)alpha, b = (T)beta;
      v[0] = v[1] = v[2] = 0.0;
      struct Own {
        T w, u, z, q, m, s, p, r, d;
      };
      auto own = [&](int i) {
        return Own{W[i], U[i], Z[i], Q[i], M[i], Sv[i], Pv[i], R[i], D[i]};
      };
      g.template spmv<T, T>(L.A, 0, Plain<T>{M}, own, [&](int i, T nv, const Own &o) {
        T wi = o.w, ui = o.u;
        const T zi = fma(b, o.z, nv), qi = fma(b, o.q, o.m);
        const T si = fma(b, o.s, wi), pi = fma(b, o.p, ui);
        ui = fma(-a, qi, ui);
        wi = fma(-a, zi, wi);
        const T ri = fma(-a, si, o.r);
        D[i] = fma(a, pi, o.d);
        Z[i] = zi;
        Q[i] = qi;
        Sv[i] = si;
        Pv[i] = pi;
        U[i] = ui;
        W[i] = wi;
        R[i] = ri;
        v[0] = fma((double)ri, (double)ui, v[0]);
        v[1] = fma((double)wi, (double)ui, v[1]);
        v[2] = fma((double)ri, (double)ri, v[2]);
      });
      g.sum(v);
      gammaold = gamma;
      alpha_old = alpha;
      first = false;
      it++;
      rr = v[2];
      if (!isfinite(v[0]))
        done = kBreakdown;
      else
        done = stop_of(rr, thresh2, ru2ref, it, max_it);
    }
    return done;
  });
}

// WIDE: at most 640 threads a CTA (96 registers each) with sixteen entries'
// loads of a row in flight; else 1024 threads with eight.
template <class T, class E, bool PIPE, int V, int LP, bool WIDE>
__global__ void __launch_bounds__(WIDE ? kPersistWideThreads : 1024, 1) persist_kernel(const __grid_constant__ PersistParams P)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[2 * kSums * 32];
  __shared__ PersistLane lane;
  __shared__ int ok[32];
  const int first = P.cta_lane[blockIdx.x], count = P.lane_count[first];
  for (int k = 0; k < count; k++) {
    __syncthreads();
    for (int w = threadIdx.x; w < (int)(sizeof(PersistLane) / 4); w += blockDim.x)
      reinterpret_cast<unsigned *>(&lane)[w] =
          reinterpret_cast<const unsigned *>(P.lanes + first + k)[w];
    __syncthreads();
    Group<V, LP, WIDE> g(P, lane, sh, ok, reinterpret_cast<Tile *>(smem_raw));
    g.start(first + k);
    if constexpr (PIPE)
      solve_pipelined<T, E>(g, first + k);
    else if constexpr (LP > 0)
      solve_classic_few<T, E>(g, first + k);
    else
      solve_classic<T, E>(g, first + k);
    if (g.dead)
      return;
  }
}

using Kernel = void (*)(PersistParams);

template <class T, class E, bool PIPE, bool WIDE> Kernel pick_shape(PersistShape w)
{
  switch (w) {
  case kRow4: return persist_kernel<T, E, PIPE, 4, 0, WIDE>;
  case kRow2: return persist_kernel<T, E, PIPE, 2, 0, WIDE>;
  case kRow1: return persist_kernel<T, E, PIPE, 1, 0, WIDE>;
  default: return persist_kernel<T, E, PIPE, 1, 2, WIDE>;
  }
}

// (FP32 pipelined solves stay on the step kernels: no default takes them)
Kernel pick(const PersistKind &k)
{
  if (!k.wide)  // batches
    return k.pipelined || k.factor_f16 ? nullptr
           : k.inner == ISPM_F64       ? pick_shape<double, double, false, false>(k.shape)
                                       : pick_shape<float, float, false, false>(k.shape);
  if (k.inner == ISPM_F64)
    return k.pipelined ? pick_shape<double, double, true, true>(k.shape)
                       : pick_shape<double, double, false, true>(k.shape);
  if (k.pipelined)
    return nullptr;
  return k.factor_f16 ? pick_shape<float, __half, false, true>(k.shape)
                      : pick_shape<float, float, false, true>(k.shape);
}

}  // namespace

bool persist_op(const Operator &op, long long row0, PersistOp &out)
{
  const ispm_slell_view m = op.dev.view();
  const unsigned S = m.slice_height;
  if (op.max_diags > kPersistMaxDiag)
    return false;
  if (m.var_height || m.hblock != 1 || S < 32 || !is_pow2(S) || row0 % S || op.diag ||
      m.n_elms >= 0xffffffffLL)
    return false;
  out.sp = m.slice_ptr;
  out.cols = m.cols;
  out.elms = m.elms;
  out.log2h = (unsigned)ilog2(S);
  out.slice0 = (unsigned)(row0 / S);
  out.col0 = (unsigned)row0;
  out.diag = m.diags != 0;
  out.inv_scale = op.inv_scale;
  return true;
}

size_t persist_smem(int max_tiles, int threads)
{
  return (3 * (size_t)max_tiles + threads / 32) * sizeof(Tile);
}

int persist_tiles(const PersistKind &k, int rows, int ncta)
{
  const int v = k.shape == kRow4 ? 4 : k.shape == kRow2 ? 2 : 1;
  const int per = k.shape == kQuarter ? 8 : 32 * v;
  const int strips = (rows / 32 + v - 1) / v;
  return ((strips + ncta - 1) / ncta * v * 32 + per - 1) / per;
}

int persist_capacity(const PersistKind &k, int threads, int max_tiles, int &ctas)
{
  ctas = 0;
  const Kernel kernel = pick(k);
  const size_t smem = persist_smem(max_tiles, threads);
  if (!kernel || smem > kPersistMaxSmem)
    return ISPM_OK;
  ISPM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kPersistMaxSmem));
  int per_sm = 0;
  ISPM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  ctas = per_sm * device_sm_count();
  return ISPM_OK;
}

PersistShape persist_shape(double rows, double threads, double width, unsigned min_height)
{
  if (rows > 2 * threads && min_height >= 128)
    return kRow4;
  if (rows > threads && min_height >= 64)
    return kRow2;
  return 10 * rows <= threads && width >= 4 ? kQuarter : kRow1;
}

int persist_launch(const PersistParams &p, const PersistKind &k, int ctas, int threads,
                   cudaStream_t s, cudaError_t fault, bool &refused)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = persist_smem(p.max_tiles, threads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = fault != cudaSuccess ? fault : cudaLaunchKernelEx(&cfg, pick(k), p);
  refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources ||
            e == cudaErrorNotSupported;
  if (refused) {
    cudaGetLastError();
    return ISPM_OK;
  }
  return e == cudaSuccess ? ISPM_OK
                          : fail(ISPM_ERR_CUDA, "persistent solve: %s", cudaGetErrorString(e));
}

int persist_assign(std::vector<PersistLane> &lanes, const std::vector<double> &work, int ctas,
                   std::vector<int> &order, std::vector<int> &cta_lane,
                   std::vector<int> &lane_count)
{
  const int n = (int)lanes.size();
  order.resize(n);
  std::iota(order.begin(), order.end(), 0);
  // heaviest first (ties by index)
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[a] > work[b]; });
  lane_count.assign(n, 0);
  cta_lane.clear();
  if (n > ctas) {
    // one CTA a group: the heaviest remaining lane to the least loaded one
    using Load = std::pair<double, int>;
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> q;
    std::vector<std::vector<int>> list(ctas);
    for (int c = 0; c < ctas; c++)
      q.push({0.0, c});
    for (int l : order) {
      Load t = q.top();
      q.pop();
      list[t.second].push_back(l);
      t.first += work[l];
      q.push(t);
    }
    order.clear();
    for (int c = 0; c < ctas; c++) {
      cta_lane.push_back((int)order.size());
      lane_count[order.size()] = (int)list[c].size();
      for (int l : list[c]) {
        lanes[l].cta0 = c;
        lanes[l].ncta = 1;
        order.push_back(l);
      }
    }
    return ctas;
  }
  for (PersistLane &l : lanes)
    l.ncta = 1;
  // the rest one by one to the lane with the most work a CTA
  std::priority_queue<std::pair<double, int>> q;
  for (int l : order)
    q.push({work[l], l});
  for (int left = ctas - n; left > 0 && !q.empty(); left--) {
    const int l = q.top().second;
    q.pop();
    lanes[l].ncta++;
    if (lanes[l].ncta < lanes[l].rows / 32)
      q.push({work[l] / lanes[l].ncta, l});
  }
  int at = 0;
  for (int k = 0; k < n; k++) {
    PersistLane &l = lanes[order[k]];
    l.cta0 = at;
    at += l.ncta;
    cta_lane.insert(cta_lane.end(), l.ncta, k);
    lane_count[k] = 1;
  }
  return at;
}

}  // namespace ispm
