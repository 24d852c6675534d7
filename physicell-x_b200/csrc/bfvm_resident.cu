// bfvm_resident.cu -- whole runs of steps of a small grid in one launch.
//
// Reference: as bfvm_sweeps.cu (the 3-D step, BioFVM/BioFVM_solvers.cpp:
// 102-780 with the pins of BioFVM_microenvironment.cpp:348-446 and the agents
// of BioFVM_basic_agent.cpp:509-559) and bfvm_lod2d.cu (the 2-D step): the
// same operations on every line in the same order, so the same bits.
//
// A small grid's step is bound by latencies, not by work: a launch per stage
// (sources, x, y, z), each with its first memory round trip and one serial
// chain per line.  Here one cooperative launch runs all the steps of a call:
// every warp owns 32 lines per sweep, the sweeps of a step follow one another
// behind a grid-wide barrier, the sources (and a 2-D step's Dirichlet nodes)
// are applied by the warp whose x lines hold them, and coefficients and code
// stay on the SMs from the first step to the last.  Where there are more tiles
// than warps, and for a batch's solves side by side, resident_many_kernel does
// the same with several tiles per warp.
//
// What a step takes, in cycles at 50x50x50x2 FP64 (156 tiles): per sweep a
// tile's copy in 1,200-1,500 (one memory latency), forward 2,500 (50 values of
// 32 dependent cycles and the loads about them), back 1,100-1,300, the x rows
// out 1,900, then the barrier 2,500-3,400 (two memory latencies and what the
// CTAs differ by); the sources 900.  Against a launch per stage, us per step in
// calls of 10 steps (of 64, where those replay a captured graph), one solve alone:
//   20x20x20x2    FP64 26.3 -> 12.7 (16.7 -> 10.8)
//   50x50x50x2    FP64 32.3 -> 15.5 (24.8 -> 13.9)  FP32 34.2 -> 15.3 (25.5 -> 13.5)
//   64x64x64x8    FP64 38.6 -> 22.9 (29.7 -> 21.2), seven warps to an SM
//   100x100x100x2 FP64 50.8 -> 28.7 (40.6 -> 26.6)  FP32 49.3 -> 26.2 (40.3 -> 23.9)
//   128x128x128x1 FP64 52.9 -> 28.8 (43.4 -> 27.0)
//   300x260 2-D x3 FP64 50.7 -> 30.3 (49.4 -> 27.5); with 10,000 agents and a
//                 rim of nodes 62.1 -> 43.7 (60.6 -> 41.2)
// With one tile per warp it won at every size it takes, up to what an SM holds:
// eight warps of 254 registers, or 227 KB of line buffers and coefficients.
// With several, the next tile's lines prefetched to the L2: see resident_wins;
// 24 uneven solves of edges 24 to 128: FP32 (247 MB) 580 -> 411 us a step, FP64
// 912 -> 673.  Where it gives way to a launch per stage: resident_shares.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "biofvm_b200.h"
#include "bfvm_ctx.h"
#include "bfvm_internal.h"
#include "bfvm_prefetch_lines.h"
#include "bfvm_ptx.cuh"
#include "bfvm_sweep_common.cuh"

namespace bfvm {

namespace {

constexpr int kResidentMembers = 48;  // solves per launch at most (their parameters are the launch's: 20 of 32 KB)
constexpr int kResidentWarps = 8;  // warps per CTA at most
constexpr int kSpreadThreads = 128;  // at least, of a CTA that takes part in the sources ahead of the x sweep
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kAgentBytes = 3 * sizeof(double) + sizeof(int);
constexpr int kResidentSteps = 64;  // steps per launch at most, about a millisecond: other streams' kernels get a turn

// The grid-wide barrier: arrivals counted up from 0 for the whole launch.
// False once a wait has run out (bounded as every device-side wait here).
struct GridBarrier {
  unsigned long long* count;
  unsigned ctas;
  unsigned long long target = 0;
  bool ok = true;
  __device__ __forceinline__ bool sync(int* status) {
    __syncthreads();
    if (threadIdx.x == 0) {
      target += ctas;
      // this CTA's stores (ordered before by the barrier above) with the arrival
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(count), "l"(1ull) : "memory");
      unsigned long long t0 = 0;
      for (;;) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(count) : "memory");
        if (v >= target) break;
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > g_wait_limit_ns) {
          atomicExch(status, kDevTimeout);
          ok = false;
          break;
        }
      }
    }
    ok = __syncthreads_and(threadIdx.x != 0 || ok);
    return ok;
  }
};

// The run's shape; every warp of the grid has at most one tile per axis.
struct ResidentPlan {
  int warps;
  int line;       // values of the longest line: sizes a warp's buffer
  int nsteps;
  int two_d;
  int face_rows;  // y and z face lines of one activated substrate
  int dr_off[3];  // staged coefficient rows of each axis, in doubles from the coefficients' start
  int cu_off[3];
  int rows[3];    // rows per substrate of each axis
  // a warp's part of shared memory: the line buffer, then what the run reads
  // again every step, kept from its start: agents and nodes (x, y) in lists of
  // these lengths
  int agents, nodes[2];
  int own;     // one warp: the coefficients of its own tiles' substrates only
  int spread;  // the sources ahead of the x sweep, by every thread of the run
  int crowd;   // so too where some x tile holds more agents than this
  int warp_bytes;  // (a multiple of 16, as each list is)
};

// A warp's line buffer: an x tile's 32 lines lie at an odd pitch of 16-byte
// units, so that eight lanes' units lie in different banks.
template <typename T>
__host__ __device__ constexpr int resident_pitch(int n) {
  constexpr int W = 16 / sizeof(T);
  return ((n + W - 1) / W | 1) * W;
}

template <typename T, int U>
struct alignas(U * sizeof(T)) ResidentUnit {
  T v[U];
};

// 16 bytes global -> shared memory, asynchronously.
template <typename T>
__device__ __forceinline__ void copy_async16(T* dst, const T* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// This lane's line of a warp's tile of one axis, set up once for the run.
template <typename T>
struct ResidentLine {
  T* line;            // its first value
  T* tile;            // the tile's first value
  int rows;           // x: the tile's rows; y, z: its lines, the pad's counted
  double c1, shift;
  double x0, x1;      // x: an activated substrate's pinned ends
  int s;
  bool act, on, any;  // on: the lane has a line that the recurrence writes; any: some lane has
};

template <typename T, int AXIS>
__device__ __forceinline__ size_t resident_stride(const SweepParams<T>& p) {
  return AXIS == 0 ? 1 : (AXIS == 1 ? static_cast<size_t>(p.nxp) : static_cast<size_t>(p.nxp) * p.ny);
}

template <typename T, int AXIS>
__device__ __forceinline__ ResidentLine<T> resident_line(const SweepParams<T>& p, int tile) {
  constexpr bool F32 = sizeof(T) == 4;
  const int t = threadIdx.x & 31;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int per_s = AXIS == 0 ? (ny * nz + 31) / 32 : (nx + 31) / 32 * (AXIS == 1 ? nz : ny);
  ResidentLine<T> l{};
  l.line = p.f;
  if (tile >= per_s * p.S) return l;
  const int s = tile / per_s, q0 = tile - s * per_s;
  l.s = s;
  l.act = p.active[s] != 0;
  l.c1 = __ldg(p.c1 + s);
  l.shift = F32 ? __ldg(p.shift + s) : 0.0;
  bool inr, face;
  size_t first;
  if (AXIS == 0) {
    const int row = q0 * 32 + t;
    inr = row < ny * nz;
    const int k = inr ? row / ny : 0, j = inr ? row - k * ny : 0;
    face = l.act && (j == 0 || j == ny - 1 || k == 0 || k == nz - 1);
    first = (static_cast<size_t>(s) * ny * nz + (inr ? row : 0)) * p.nxp;
    if (l.act && inr) {
      const double off = F32 ? p.off[s] : 0.0;
      const double a = __ldg(p.xface + static_cast<size_t>(s) * ny * nz + row);
      const double b = __ldg(p.xface + (static_cast<size_t>(p.S) + s) * ny * nz + row);
      l.x0 = F32 ? a - off : a;
      l.x1 = F32 ? b - off : b;
    }
  } else {
    const int xt = (nx + 31) / 32, m = q0 / xt, i = (q0 - m * xt) * 32 + t, nm = AXIS == 1 ? nz : ny;
    inr = i < nx;  // (a lane past the rows' end runs along on the rows' first value)
    face = l.act && (i == 0 || i == nx - 1 || m == 0 || m == nm - 1);
    first = (AXIS == 1 ? (static_cast<size_t>(s) * nz + m) * ny * p.nxp
                       : (static_cast<size_t>(s) * nz * ny + m) * p.nxp) + (inr ? i : 0);
    l.tile = p.f + first - (inr ? t : 0) + (inr ? 0 : i - t);
    l.rows = p.nxp - (i - t);
  }
  l.line = p.f + first;
  if (AXIS == 0) {
    l.tile = p.f + (static_cast<size_t>(s) * ny * nz + q0 * 32) * p.nxp;
    l.rows = min(32, ny * nz - q0 * 32);
  }
  l.on = inr && !face;
  l.any = __any_sync(0xffffffffu, l.on);
  return l;
}

// One sweep of one 32-line tile by one warp.  An x sweep's `before` changes
// the tile in shared memory, and in the field, ahead of the sweep (sources and
// nodes); its `after` does before the rows go out.
template <typename T, int AXIS, typename Meanwhile, typename Before, typename After>
__device__ __forceinline__ void resident_tile(const SweepParams<T>& p, const ResidentPlan& pl, const double* coef,
                                              T* buf, const ResidentLine<T>& l, Meanwhile meanwhile, Before before,
                                              After after) {
  using DR = typename Coef<T>::DR;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int R = kRowBatch, kAhead = 4;  // (kUnits: as many values by units)
  if (!l.any) return;
  const int t = threadIdx.x & 31;
  const int n = AXIS == 0 ? p.nx : (AXIS == 1 ? p.ny : p.nz);
  const size_t stride = resident_stride<T, AXIS>(p);
  T* const line = l.line;
  const int s = l.s;
  const bool act = l.act, on = l.on, fast = p.screen == kScreenFast;
  const double c1 = l.c1, shift = l.shift, x0 = l.x0, x1 = l.x1;
  const size_t set = pl.own ? 0 : static_cast<size_t>(s) * pl.rows[AXIS];
  const DR* dr = reinterpret_cast<const DR*>(coef + pl.dr_off[AXIS]) + set;
  const double* cu = coef + pl.cu_off[AXIS] + set;

  // ---- the tile in: every copy under way at once (one memory latency for
  // the tile, 1,200 cycles), 16 bytes a lane (8 took three times as long for
  // 50 rows) and each row's side by side at both ends (the field's rows start
  // on 16 bytes and are padded to them).  A line's values go by units: 16
  // bytes of a row for x, one value for y and z; unit q of lane t's line lies
  // at col[q * kStep].
  constexpr int W = 16 / sizeof(T), U = AXIS == 0 ? W : 1;
  constexpr int kUnits = kAhead / U;
  using Unit = ResidentUnit<T, U>;
  constexpr int kStep = AXIS == 0 ? 1 : 32;
  const int pitch = AXIS == 0 ? resident_pitch<T>(n) : 32;
  Unit* const col = reinterpret_cast<Unit*>(AXIS == 0 ? buf + t * pitch : buf + t);
  T* const values = reinterpret_cast<T*>(col);
  // lanes per row, rows per instruction, this lane's first row and value
  const int lanes = AXIS == 0 ? (n <= 8 * W ? 8 : (n <= 16 * W ? 16 : 32)) : 32 / W;
  const int rows = 32 / lanes, r0 = t / lanes, i0 = (t % lanes) * W;
  if (AXIS == 0) {
    for (int i = i0; i < n; i += 32 * W) {
      const T* at = l.tile + static_cast<size_t>(r0) * p.nxp + i;
      T* to = buf + r0 * pitch + i;
      const size_t step = static_cast<size_t>(rows) * p.nxp;
#pragma unroll 8
      for (int r = r0; r < l.rows; r += rows, at += step, to += rows * pitch) copy_async16(to, at);
    }
  } else if (i0 < l.rows) {
    const T* at = l.tile + r0 * stride + i0;
    T* to = buf + r0 * 32 + i0;
#pragma unroll 8
    for (int q = r0; q < n; q += rows, at += rows * stride, to += rows * 32) copy_async16(to, at);
  }
  meanwhile();
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  if (AXIS == 0) {
    before();
    if (act) {  // the pin before the sweep
      values[0] = static_cast<T>(x0);
      values[n - 1] = static_cast<T>(x1);
    }
  }

  // ---- forward, in place.  Inputs and coefficients are read kAhead values
  // early, as the stores between keep the compiler from doing so.
  double y = -0.0;
  int hwmin = INT_MAX;
  auto eliminate = [&](const DR e, const T v) __attribute__((always_inline)) {
    if constexpr (F32) {
      const double in = static_cast<double>(v) - shift;
      if (fast)
        y = __fma_rn(__dmul_rn(c1, e), y, __dmul_rn(in, e));
      else
        y = __dmul_rn(__fma_rn(c1, y, in), e);
    } else {
      if (fast) {
        y = __fma_rn(e.x, y, __dmul_rn(v, e.y));
      } else {
        hwmin = min(hwmin, __double2hiint(v));
        y = markstein(__fma_rn(c1, y, v), e.x, e.y);
      }
    }
    return static_cast<T>(y);
  };
  const int whole = n / R * R;
  {
    const DR* d = dr;
    Unit* c = col;
    for (int b0 = 0; b0 < whole; b0 += R, d += R, c += R / U * kStep) {
      DR dq[kAhead];
      Unit vq[kUnits];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) dq[q] = d[q];
#pragma unroll
      for (int g = 0; g < kUnits; ++g) vq[g] = c[g * kStep];
#pragma unroll
      for (int g = 0; g < R / U; ++g) {
        Unit v = vq[g % kUnits];
        if (g + kUnits < R / U) vq[g % kUnits] = c[(g + kUnits) * kStep];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int q = g * U + u;
          const DR e = dq[q % kAhead];
          if (q + kAhead < R) dq[q % kAhead] = d[q + kAhead];
          v.v[u] = eliminate(e, v.v[u]);
        }
        c[g * kStep] = v;
      }
    }
    for (int q = whole; q < n; ++q, ++d) values[q * kStep] = eliminate(*d, values[q * kStep]);
  }
  if constexpr (!F32) {
    // The screen, once per line: one with an input below 2^-960 (or negative)
    // anywhere is redone from its inputs, which the field still holds.
    if (!fast && on && !screen_clean(p.screen, hwmin)) {
      y = -0.0;
      for (int b0 = 0; b0 < n; b0 += R) {
        double v[R];
        double2 cf[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          v[q] = b0 + q < n ? __ldcg(line + static_cast<size_t>(b0 + q) * stride) : 1.0;
          if (AXIS == 0 && act) {
            if (b0 + q == 0) v[q] = x0;
            if (b0 + q == n - 1) v[q] = x1;
          }
          cf[q] = dr[b0 + q];
        }
        y = forward_checked<R>(v, cf, c1, y, [&](int q, double val) {
          if (b0 + q < n) values[(b0 + q) * kStep] = val;
        });
      }
    }
  }

  // ---- back, over an activated substrate's first and last rows without a
  // store: they keep their pinned input
  double xn = -0.0;
  T* at = line + static_cast<size_t>(n - 1) * stride;
  for (int q = n - 1; q >= whole; --q, at -= stride) {
    T* const v = values + q * kStep;
    xn = back_elem(cu[q], xn, static_cast<double>(*v));
    if (AXIS == 0)
      *v = static_cast<T>(xn);
    else if (on && !(act && (q == n - 1 || q == 0)))
      *at = static_cast<T>(xn);
  }
  const double2* w2 = reinterpret_cast<const double2*>(cu + whole);
  Unit* c = col + whole / U * kStep;
  for (int b0 = whole - R; b0 >= 0; b0 -= R) {
    w2 -= R / 2;
    c -= R / U * kStep;
    const bool first = on && !(act && b0 == 0), end = on && !(act && b0 + R == n);
    double2 wq[kAhead / 2];
    Unit oq[kUnits];
#pragma unroll
    for (int e = 0; e < kUnits; ++e) oq[e] = c[(R / U - 1 - e) * kStep];
#pragma unroll
    for (int e = 0; e < kAhead / 2; ++e) wq[e] = w2[R / 2 - 1 - e];
#pragma unroll
    for (int g = R / U - 1; g >= 0; --g) {
      const int slot = (R / U - 1 - g) % kUnits;
      Unit o = oq[slot];
      if (g - kUnits >= 0) oq[slot] = c[(g - kUnits) * kStep];
#pragma unroll
      for (int u = U - 1; u >= 0; --u) {
        const int q = g * U + u, h = (R / 2 - 1 - q / 2) % (kAhead / 2);
        const double w = (q & 1) ? wq[h].y : wq[h].x;
        if ((q & 1) == 0 && q / 2 - kAhead / 2 >= 0) wq[h] = w2[q / 2 - kAhead / 2];
        xn = back_elem(w, xn, static_cast<double>(o.v[u]));
        o.v[u] = static_cast<T>(xn);
        if (AXIS != 0) {
          if (q == R - 1 ? end : (q == 0 ? first : on)) *at = static_cast<T>(xn);
          at -= stride;
        }
      }
      if (AXIS == 0) c[g * kStep] = o;
    }
  }
  if (AXIS == 0) {  // the rows out as they came in, the pad with them
    if (act) {      // the pin after the sweep
      values[0] = static_cast<T>(x0);
      values[n - 1] = static_cast<T>(x1);
    }
    const unsigned write = __ballot_sync(0xffffffffu, on);
    constexpr int kOut = 8;  // (read ahead: the compiler keeps the reads behind earlier stores)
    __syncwarp();
    after();
    for (int i = i0; i < n; i += 32 * W) {
      T* to = l.tile + static_cast<size_t>(r0) * p.nxp + i;
      const T* from = buf + r0 * pitch + i;
      const size_t step = static_cast<size_t>(rows) * p.nxp;
      for (int r = r0; r < 32; r += kOut * rows) {
        int4 v[kOut];
#pragma unroll
        for (int e = 0; e < kOut; ++e, from += rows * pitch) v[e] = *reinterpret_cast<const int4*>(from);
#pragma unroll
        for (int e = 0; e < kOut; ++e, to += step)
          if ((write >> (r + e * rows)) & 1u) *reinterpret_cast<int4*>(to) = v[e];
      }
    }
  }
  __syncwarp();
}

// The agents of an x tile's rows and substrate, in list order per voxel: lane t
// takes agents a0 + t, a0 + t + 32, ..., the first of each voxel's run going on
// through it.  The first `kept` agents' data lie in shared memory for the run,
// as do a plane's nodes: 300x260x3 FP64 with 10,000 agents and a rim of nodes,
// three solves at once, took 26 us a step with both read from memory each time
// and takes 15.  Agents in a face line of an activated substrate are
// left out: the line is pinned before anything reads it (no agents are tracked
// here).
struct ResidentAgent {
  int at;  // its place in the tile: row of 32 << 16 | value; negative: not a run's first, or in a face line
  double k1, k2, k3;
};
constexpr int kStacked = 1 << 30;  // ... | this, where the next agent is in the same voxel

template <typename T>
struct ResidentAgents {
  int a0, a1, kept;  // the tile's agents in the sorted list
  const double *c1, *c2, *e2;
  double off;
  int r0, s;
  bool act;
  double* k;  // shared memory: k1, k2 and k3 of the kept agents, `cap` apart, and their places
  int* at;
  int cap;
};

template <typename T>
__device__ __forceinline__ ResidentAgent resident_agent(const SweepParams<T>& p, const ResidentAgents<T>& g, int q) {
  ResidentAgent a;
  const unsigned key = __ldg(p.a_key + q);  // one latency for all six
  const unsigned before = __ldg(p.a_key + max(q - 1, g.a0)), after = __ldg(p.a_key + min(q + 1, g.a1 - 1));
  a.k1 = __ldg(g.c1 + q);
  a.k2 = __ldg(g.c2 + q);
  a.k3 = __ldg(g.e2 + q);
  a.at = INT_MIN | (q + 1 < g.a1 && after == key ? kStacked : 0);
  if (q > g.a0 && before == key) return a;
  const int row = static_cast<int>(key / p.nx), i = static_cast<int>(key - static_cast<unsigned>(row) * p.nx);
  const int k = row / p.ny, j = row - k * p.ny;
  if (g.act && (j == 0 || j == p.ny - 1 || k == 0 || k == p.nz - 1)) return a;
  a.at = (a.at & kStacked) | (row - g.r0) << 16 | i;
  return a;
}

template <int ROUNDS, typename T>
__device__ __forceinline__ ResidentAgents<T> resident_agents(const SweepParams<T>& p, int tile, int cap, double* keep) {
  ResidentAgents<T> g{};
  const int rows = p.ny * p.nz, per_s = (rows + 31) / 32, t = threadIdx.x & 31;
  if (p.line_off == nullptr || tile >= per_s * p.S) return g;
  const int s = tile / per_s, r0 = (tile - s * per_s) * 32;
  g.s = s;
  g.r0 = r0;
  g.act = p.active[s] != 0;
  g.a0 = __ldg(p.line_off + r0);
  g.a1 = __ldg(p.line_off + min(rows, r0 + 32));
  g.kept = min(cap, g.a1 - g.a0);
  const size_t sn = static_cast<size_t>(s) * p.n_sorted;
  g.c1 = p.ac1 + sn;
  g.c2 = p.ac2 + sn;
  g.e2 = p.ae2 + sn;
  g.off = sizeof(T) == 4 ? p.off[s] : 0.0;
  g.cap = cap;
  g.k = keep;
  g.at = reinterpret_cast<int*>(keep + 3 * cap);
  constexpr int kRounds = ROUNDS;  // read together: one memory latency
  for (int e0 = t; e0 < g.kept; e0 += 32 * kRounds) {
    ResidentAgent a[kRounds];
#pragma unroll
    for (int u = 0; u < kRounds; ++u) a[u] = resident_agent(p, g, g.a0 + min(e0 + 32 * u, g.kept - 1));
#pragma unroll
    for (int u = 0; u < kRounds; ++u) {
      const int e = e0 + 32 * u;
      if (e >= g.kept) break;
      g.k[e] = a[u].k1;
      g.k[e + cap] = a[u].k2;
      g.k[e + 2 * cap] = a[u].k3;
      g.at[e] = a[u].at;
    }
  }
  return g;
}

// To the tile in shared memory, and to the field for a line that is redone
// from it.
template <typename T>
__device__ __forceinline__ void resident_sources(const SweepParams<T>& p, const ResidentAgents<T>& g, T* buf, int pitch,
                                                 T* tile) {
  const int n = g.a1 - g.a0;
  auto agent = [&](int e) __attribute__((always_inline)) {
    if (e >= g.kept) return resident_agent(p, g, g.a0 + e);
    return ResidentAgent{g.at[e], g.k[e], g.k[e + g.cap], g.k[e + 2 * g.cap]};
  };
  for (int e = threadIdx.x & 31; e < n; e += 32) {
    ResidentAgent a = agent(e);
    if (a.at < 0) continue;
    const int row = (a.at >> 16) & 31, i = a.at & 0xffff;
    T* const rho = buf + row * pitch + i;
    double r = static_cast<double>(*rho);
    if constexpr (kF32<T>) r += g.off;
    r = agent_update(r, a.k1, a.k2, a.k3, g.a0 + e, g.s, p.track);
    for (int q = e + 1; (a.at & kStacked) != 0; ++q) {
      a = agent(q);
      r = agent_update(r, a.k1, a.k2, a.k3, g.a0 + q, g.s, p.track);
    }
    if constexpr (kF32<T>) r -= g.off;
    const T x = static_cast<T>(r);
    *rho = x;
    tile[static_cast<size_t>(row) * p.nxp + i] = x;
  }
  __syncwarp();
}

// The sources by all of the run's threads, thread `id` of `threads`, ahead of
// the x sweep and a barrier: where many agents lie in a tile.  Four agents a
// thread at a time, two memory latencies for the four.
template <typename T>
__device__ __forceinline__ void resident_spread(const SweepParams<T>& p, unsigned id, unsigned threads) {
  constexpr int kAgents = 4;
  const int rows = p.ny * p.nz, n = __ldg(p.line_off + rows);
  const unsigned total = static_cast<unsigned>(n) * p.S;  // (below 2^31: resident_spreads)
  for (unsigned e0 = id; e0 < total; e0 += kAgents * threads) {
    unsigned key[kAgents], before[kAgents], after[kAgents];
    double k1[kAgents], k2[kAgents], k3[kAgents];
    T* rho[kAgents];
    T x[kAgents];
#pragma unroll
    for (int u = 0; u < kAgents; ++u) {
      const unsigned e = min(e0 + u * threads, total - 1);
      const int s = static_cast<int>(e / n), q = static_cast<int>(e - s * n);
      const size_t at = static_cast<size_t>(s) * p.n_sorted + q;
      key[u] = __ldg(p.a_key + q);
      before[u] = __ldg(p.a_key + max(q - 1, 0));
      after[u] = __ldg(p.a_key + min(q + 1, n - 1));
      k1[u] = __ldg(p.ac1 + at);
      k2[u] = __ldg(p.ac2 + at);
      k3[u] = __ldg(p.ae2 + at);
    }
#pragma unroll
    for (int u = 0; u < kAgents; ++u) {
      const unsigned e = e0 + u * threads;
      const int s = static_cast<int>(e / n), q = static_cast<int>(e - s * n);
      const int row = static_cast<int>(key[u] / p.nx), i = static_cast<int>(key[u] - static_cast<unsigned>(row) * p.nx);
      const int k = row / p.ny, j = row - k * p.ny;
      rho[u] = nullptr;
      x[u] = T(0);
      if (e >= total || (q > 0 && before[u] == key[u]) ||
          (p.active[s] != 0 && (j == 0 || j == p.ny - 1 || k == 0 || k == p.nz - 1)))
        continue;
      rho[u] = p.f + (static_cast<size_t>(s) * rows + row) * p.nxp + i;
      x[u] = __ldcg(rho[u]);
    }
    // The first agent of each run; then what the runs go on to, where agents are
    // stacked, one by one: a lane's first run, then its second.  (Stacks leave
    // most of a warp's agents without a run of their own: taking the runs by the
    // agents' places, a warp waited four times for the longest of its lanes:
    // 50x50x50x2 FP64, 70,000 agents in a ball of 12 voxels 43 -> 37 us a step, a
    // plane of 300x260x3, 10,000 in a disc of 20 54 -> 48, 30,000 81 -> 67.)
    double r[kAgents];
    unsigned more = 0;
#pragma unroll
    for (int u = 0; u < kAgents; ++u) {
      if (rho[u] == nullptr) continue;
      const unsigned e = e0 + u * threads;
      const int s = static_cast<int>(e / n), q = static_cast<int>(e - s * n);
      const double off = sizeof(T) == 4 ? p.off[s] : 0.0;
      r[u] = static_cast<double>(x[u]);
      if constexpr (kF32<T>) r[u] += off;
      r[u] = agent_update(r[u], k1[u], k2[u], k3[u], q, s, p.track);
      if (q + 1 < n && after[u] == key[u]) {
        more |= 1u << u;
      } else {
        if constexpr (kF32<T>) r[u] -= off;
        *rho[u] = static_cast<T>(r[u]);
      }
    }
    while (more != 0) {
      const int pick = __ffs(more) - 1;
      more &= more - 1;
      T* at = rho[0];
      double v = r[0];
      unsigned mine = key[0];
#pragma unroll
      for (int u = 1; u < kAgents; ++u) {
        if (pick != u) continue;
        at = rho[u];
        v = r[u];
        mine = key[u];
      }
      const unsigned e = e0 + pick * threads;
      const int s = static_cast<int>(e / n);
      const size_t sn = static_cast<size_t>(s) * p.n_sorted;
      for (int q = static_cast<int>(e - s * n) + 1; q < n && __ldg(p.a_key + q) == mine; ++q)
        v = agent_update(v, __ldg(p.ac1 + sn + q), __ldg(p.ac2 + sn + q), __ldg(p.ae2 + sn + q), q, s, p.track);
      if constexpr (kF32<T>) v -= p.off[s];
      *at = static_cast<T>(v);
    }
  }
}

// What a launch looks up for the two below, read before the rest of its set-up,
// which hides the latency.
struct ResidentLook {
  int from, to;  // this thread's first x tile in the sorted agents
  int on;        // activation of substrate `lane`
};

template <typename T>
__device__ __forceinline__ ResidentLook resident_look(const SweepParams<T>& p, const ResidentPlan& pl) {
  ResidentLook l{};
  const int rows = p.ny * p.nz, r = 32 * threadIdx.x, s = threadIdx.x & 31;
  if (p.line_off != nullptr && !pl.spread && r < rows) {
    l.from = __ldg(p.line_off + r);
    l.to = __ldg(p.line_off + min(rows, r + 32));
  }
  if (s < p.S) l.on = __ldg(p.active + s);
  return l;
}

// The face lines of all activated substrates.  How many are activated is read
// when the launch runs: a captured launch outlives the activation it was
// captured under, and the lines it leaves out of the sweeps follow the device's.
template <typename T>
__device__ __forceinline__ int resident_face_rows(const SweepParams<T>& p, const ResidentPlan& pl,
                                                  const ResidentLook& l) {
  if (pl.face_rows == 0) return 0;
  int on = __popc(__ballot_sync(0xffffffffu, l.on != 0));
  for (int s0 = 32; s0 < p.S; s0 += 32) {
    const int s = s0 + (threadIdx.x & 31);
    on += __popc(__ballot_sync(0xffffffffu, s < p.S && p.active[s] != 0));
  }
  return on * pl.face_rows;
}

// Whether some x tile that this thread looks at holds more than pl.crowd agents
// (the threads of a CTA look at all of them between them, so every CTA of the
// run comes to the same answer).
template <typename T>
__device__ __forceinline__ bool resident_crowded(const SweepParams<T>& p, const ResidentPlan& pl,
                                                 const ResidentLook& l) {
  if (p.line_off == nullptr || pl.spread) return false;
  const int rows = p.ny * p.nz;
  int worst = l.to - l.from;
  for (int r = 32 * (threadIdx.x + blockDim.x); r < rows; r += 32 * blockDim.x)
    worst = max(worst, __ldg(p.line_off + min(rows, r + 32)) - __ldg(p.line_off + r));
  return worst > pl.crowd;
}

// The y and z face lines of activated substrates take their face's values
// (their ends, the x faces') in the x sweep's place: row number `at` of all
// of them, by one warp, coalesced.
template <typename T>
struct ResidentFace {
  T* row;  // null: none
  const double *fv, *x0, *x1;
  double off;
  T v[4];  // the row's first 128 values, this lane's, read once for the run
};

template <typename T>
__device__ __forceinline__ T resident_face_value(const ResidentFace<T>& r, int nx, int i) {
  const double f = i < nx ? __ldg(i == nx - 1 ? r.x1 : (i == 0 ? r.x0 : r.fv + i)) : 0.0;
  return static_cast<T>(sizeof(T) == 4 ? f - r.off : f);
}

template <typename T>
__device__ __forceinline__ ResidentFace<T> resident_face(const SweepParams<T>& p, int at) {
  ResidentFace<T> r{};
  const int nx = p.nx, ny = p.ny, nz = p.nz, t = threadIdx.x & 31;
  const int zrows = (nz > 1 ? 2 : 1) * ny, yrows = (ny > 1 ? 2 : 1) * (nz > 2 ? nz - 2 : 0), per = zrows + yrows;
  int s = 0;
  for (;; ++s) {
    if (s >= p.S) return r;
    if (p.active[s] == 0) continue;
    if (at < per) break;
    at -= per;
  }
  int k, j;
  const double* fv;
  if (at < zrows) {
    const int side = at >= ny ? 1 : 0;
    j = at - side * ny;
    k = side == 0 ? 0 : nz - 1;
    fv = p.zface + ((static_cast<size_t>(side) * p.S + s) * ny + j) * nx;
  } else {
    const int side = at - zrows >= nz - 2 ? 1 : 0;
    k = 1 + at - zrows - side * (nz - 2);
    j = side == 0 ? 0 : ny - 1;
    fv = p.yface + ((static_cast<size_t>(side) * p.S + s) * nz + k) * nx;
  }
  const size_t row = (static_cast<size_t>(s) * nz + k) * ny + j;
  r.row = p.f + row * p.nxp;
  r.fv = fv;
  r.x0 = p.xface + row;
  r.x1 = p.xface + static_cast<size_t>(p.S) * ny * nz + row;
  r.off = sizeof(T) == 4 ? p.off[s] : 0.0;
#pragma unroll
  for (int e = 0; e < 4; ++e) r.v[e] = resident_face_value(r, nx, t + 32 * e);
  return r;
}

template <typename T>
__device__ __forceinline__ void resident_face_store(const ResidentFace<T>& r, int nx) {
  if (r.row == nullptr) return;
  const int t = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (t + 32 * e < nx) r.row[t + 32 * e] = r.v[e];
  for (int i = t + 128; i < nx; i += 32) r.row[i] = resident_face_value(r, nx, i);
}

// A 2-D step's Dirichlet nodes of one tile: the activated ones of lines
// [l0, l0 + 32), in shared memory from the run's start.
template <typename T>
struct ResidentNodes {
  int n;
  T* v;
  int* at;  // row of the plane << 16 | column; -1: not activated
  T* plane;
};

template <typename T>
__device__ __forceinline__ ResidentNodes<T> resident_nodes(const SweepParams<T>& p, const NodeLines& nd, int axis,
                                                           int tile, int cap, void* keep) {
  ResidentNodes<T> g{};
  const int lines = axis == 0 ? p.ny : p.nx, per_s = (lines + 31) / 32, t = threadIdx.x & 31;
  if (nd.n == 0 || tile >= per_s * p.S) return g;
  const int s = tile / per_s, l0 = (tile - s * per_s) * 32;
  const int a0 = __ldg(nd.first[axis] + l0);
  g.n = __ldg(nd.first[axis] + min(lines, l0 + 32)) - a0;
  g.v = static_cast<T*>(keep);
  g.at = reinterpret_cast<int*>(g.v + cap);
  g.plane = p.f + static_cast<size_t>(s) * p.nxp * p.ny;
  const double off = sizeof(T) == 4 ? p.off[s] : 0.0;
  for (int q = t; q < g.n; q += 32) {
    const int a = __ldg(nd.order[axis] + a0 + q);
    const size_t e = static_cast<size_t>(a) * p.S + s;
    const long long at = nd.off[a];
    const int row = static_cast<int>(at / p.nxp);
    g.v[q] = static_cast<T>(sizeof(T) == 4 ? nd.val[e] - off : nd.val[e]);
    g.at[q] = nd.act[e] ? row << 16 | static_cast<int>(at - static_cast<long long>(row) * p.nxp) : -1;
  }
  return g;
}

// The nodes' values to the field, and to the x tile in shared memory whose
// rows start at l0 (buf given).
template <typename T>
__device__ __forceinline__ void resident_pin(const SweepParams<T>& p, const ResidentNodes<T>& g, bool field, T* buf,
                                             int pitch, int l0) {
  __syncwarp();
  for (int q = threadIdx.x & 31; q < g.n; q += 32) {
    const int at = g.at[q];
    if (at < 0) continue;
    const int row = at >> 16, i = at & 0xffff;
    if (field) g.plane[static_cast<size_t>(row) * p.nxp + i] = g.v[q];
    if (buf != nullptr) buf[(row - l0) * pitch + i] = g.v[q];
  }
  __syncwarp();
}

// A tile's 128-byte lines (a row's start on them) on their way to the L2.
template <typename T, int AXIS>
__device__ __forceinline__ void resident_prefetch(const SweepParams<T>& p, int tile, int tiles) {
  if (tile >= tiles) return;
  const int t = threadIdx.x & 31;
  const PrefetchLines l = prefetch_lines<AXIS, 128 / static_cast<int>(sizeof(T))>(p.nx, p.ny, p.nz, p.nxp, tile, t);
  const T* at = p.f + l.at;
  for (int q = t; q < l.count; q += 32, at += l.step) asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
}

// A run's coefficients to shared memory, every copy under way at once (a plane's
// CTA has one warp: with a loop of loads a call of one step of 300x260x3 took
// 67 us, its steps 39).
template <typename T>
__device__ __forceinline__ double* resident_coefs(const SweepParams<T>& p, const ResidentPlan& pl, unsigned char* smem,
                                                  int sx, int sy, int sz) {
  constexpr int kDR = sizeof(typename Coef<T>::DR) / sizeof(double);
  double* const coef = reinterpret_cast<double*>(smem + static_cast<size_t>(pl.warps) * pl.warp_bytes);
  const AxisCoefs<T>* axes[3] = {&p.ax, &p.ay, &p.az};
  const int naxes = pl.two_d ? 2 : 3;
  for (int a = 0; a < naxes; ++a) {
    const int rows = pl.rows[a];  // (even, and the padded rows too: 16 bytes are whole)
    const int s0 = pl.own ? (a == 0 ? sx : (a == 1 ? sy : sz)) : 0, ns = pl.own ? 1 : p.S;
    for (int q0 = 0; q0 < ns; ++q0) {
      const int s = s0 + q0;
      const double* dr = reinterpret_cast<const double*>(axes[a]->dr + static_cast<size_t>(s) * axes[a]->npad);
      const double* cu = axes[a]->cu + static_cast<size_t>(s) * axes[a]->npad;
      double* const to = coef + pl.dr_off[a] + q0 * rows * kDR;
      for (int q = 2 * threadIdx.x; q < rows * kDR; q += 2 * blockDim.x) copy_async16(to + q, dr + q);
      for (int q = 2 * threadIdx.x; q < rows; q += 2 * blockDim.x)
        copy_async16(coef + pl.cu_off[a] + q0 * rows + q, cu + q);
    }
  }
  return coef;  // (there once the caller has waited for its copies)
}

// The last of the run's CTAs leaves the counters at zero for the next run.
__device__ __forceinline__ void resident_leave(unsigned long long* barrier, int ctas) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(barrier + 1, 1ull) == ctas - 1) {
      barrier[0] = 0;
      barrier[1] = 0;
    }
  }
}

// One tile per warp and axis: all that does not change from step to step is
// set up once.
template <typename T>
__global__ void __launch_bounds__(32 * kResidentWarps, 1)
    resident_kernel(const SweepParams<T> p, const ResidentPlan pl, const NodeLines nd, unsigned long long* barrier) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const ResidentLook look = resident_look(p, pl);
  // Neighbouring tiles on different SMs.  (Warps past the plan's, there for the
  // sources, find no tile.)
  const int w0 = blockIdx.x + gridDim.x * warp, nw = gridDim.x * (blockDim.x >> 5);
  unsigned char* keep = smem_raw + static_cast<size_t>(warp) * pl.warp_bytes;
  T* const buf = reinterpret_cast<T*>(keep);
  const int pitch = resident_pitch<T>(p.nx);
  keep += static_cast<size_t>(32) * resident_pitch<T>(pl.line) * sizeof(T);
  const ResidentLine<T> lx = resident_line<T, 0>(p, w0), ly = resident_line<T, 1>(p, w0);
  ResidentLine<T> lz{};
  if (!pl.two_d) lz = resident_line<T, 2>(p, w0);
  // (own: warp 0's tiles are the CTA's)
  const int cta = blockIdx.x, xt = (p.nx + 31) / 32;
  const double* const coef =
      resident_coefs(p, pl, smem_raw, min(cta / ((p.ny * p.nz + 31) / 32), p.S - 1), min(cta / (xt * p.nz), p.S - 1),
                     min(cta / (xt * p.ny), p.S - 1));
  ResidentAgents<T> ag{};
  if (!pl.spread) ag = resident_agents<4>(p, w0, pl.agents, reinterpret_cast<double*>(keep));
  keep += static_cast<size_t>(pl.agents) * kAgentBytes;
  const ResidentNodes<T> xn = resident_nodes(p, nd, 0, w0, pl.nodes[0], keep);
  keep += static_cast<size_t>(pl.nodes[0]) * (sizeof(T) + sizeof(int));
  const ResidentNodes<T> yn = resident_nodes(p, nd, 1, w0, pl.nodes[1], keep);
  const int l0 = w0 % ((p.ny + 31) / 32) * 32;  // (of a plane)
  __syncwarp();
  const bool crowded = resident_crowded(p, pl, look);
  const int face_rows = resident_face_rows(p, pl, look);
  ResidentFace<T> face{};
  if (w0 < face_rows) face = resident_face(p, w0);
  asm volatile("cp.async.wait_all;" ::: "memory");
  const bool spread = __syncthreads_or(crowded) || pl.spread;
  if (spread) ag.a1 = ag.a0;
  const auto none = [] {};
  GridBarrier bar{barrier, gridDim.x};
  for (int step = 0; step < pl.nsteps; ++step) {
    if (spread) {
      resident_spread(p, w0 * 32 + (threadIdx.x & 31), nw * 32);
      if (!bar.sync(p.status)) break;
    }
    resident_tile<T, 0>(
        p, pl, coef, buf, lx, none,
        [&] {
          if (ag.a1 > ag.a0) resident_sources(p, ag, buf, pitch, lx.tile);
          if (xn.n > 0) resident_pin(p, xn, true, buf, pitch, l0);
        },
        [&] {
          if (xn.n > 0) resident_pin(p, xn, false, buf, pitch, l0);
        });
    resident_face_store(face, p.nx);
    for (int q = w0 + nw; q < face_rows; q += nw) resident_face_store(resident_face(p, q), p.nx);
    if (!bar.sync(p.status)) break;
    resident_tile<T, 1>(p, pl, coef, buf, ly, none, none, none);
    if (yn.n > 0) resident_pin<T>(p, yn, true, nullptr, 0, 0);
    if (!pl.two_d) {
      if (!bar.sync(p.status)) break;
      resident_tile<T, 2>(p, pl, coef, buf, lz, none, none, none);
    }
    if (step + 1 < pl.nsteps && !bar.sync(p.status)) break;
  }
  resident_leave(barrier, gridDim.x);
}

// Several tiles per warp and axis, and several solves side by side: each has
// CTAs cta0 .. cta0 + ctas - 1 and a barrier of its own, so a batch's solves
// go through their steps independently.
template <typename T>
struct ResidentSolve {
  SweepParams<T> p;
  ResidentPlan pl;
  int cta0, ctas;
  unsigned long long* barrier;
};

template <typename T, int N>
struct ResidentBatch {
  int n, nsteps;
  ResidentSolve<T> solve[N];
};

// Warps per CTA at most: FP32's eight and sixteen were no faster (24 solves
// side by side: 420 us a step with any; 100 smaller ones 642 with 8 and 12, 725
// with 16), FP64's twelve neither, as shared memory holds fewer from 100 values
// a line on.
template <typename T>
constexpr int kManyWarps = sizeof(T) == 4 ? 12 : 8;

template <typename T, int N>
__global__ void __launch_bounds__(32 * kManyWarps<T>, 1)
    resident_many_kernel(const __grid_constant__ ResidentBatch<T, N> b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int m = 0;
  if constexpr (N > 1) {
    while (m + 1 < b.n && static_cast<int>(blockIdx.x) >= b.solve[m + 1].cta0) ++m;
  }
  const SweepParams<T>& p = b.solve[m].p;
  const ResidentPlan& pl = b.solve[m].pl;
  const int ctas = b.solve[m].ctas;
  const ResidentLook look = resident_look(p, pl);
  const double* const coef = resident_coefs(p, pl, smem_raw, 0, 0, 0);
  const int warp = threadIdx.x >> 5;
  const int nw = ctas * pl.warps;
  // (a warp past the solve's takes part in the barriers only)
  const int w0 = warp < pl.warps ? static_cast<int>(blockIdx.x) - b.solve[m].cta0 + ctas * warp : INT_MAX / 2;
  unsigned char* const keep = smem_raw + static_cast<size_t>(warp) * pl.warp_bytes;
  T* const buf = reinterpret_cast<T*>(keep);
  double* const agents =
      reinterpret_cast<double*>(keep + static_cast<size_t>(32) * resident_pitch<T>(pl.line) * sizeof(T));
  const int pitch = resident_pitch<T>(p.nx);
  const int xt = (p.nx + 31) / 32;
  const int face_rows = resident_face_rows(p, pl, look);
  const bool crowded = resident_crowded(p, pl, look);
  const int ntx = (p.ny * p.nz + 31) / 32 * p.S, nty = xt * p.nz * p.S, ntz = xt * p.ny * p.S;
  asm volatile("cp.async.wait_all;" ::: "memory");
  const bool spread = __syncthreads_or(crowded) || pl.spread;
  const auto none = [] {};
  GridBarrier bar{b.solve[m].barrier, static_cast<unsigned>(ctas)};
  for (int step = 0; step < b.nsteps; ++step) {
    for (int q = w0; q < face_rows; q += nw) resident_face_store(resident_face(p, q), p.nx);
    if (spread) {
      resident_spread(p, (blockIdx.x - b.solve[m].cta0) * blockDim.x + threadIdx.x, ctas * blockDim.x);
      if (!bar.sync(p.status)) break;
    }
    for (int tile = w0; tile < ntx; tile += nw) {
      ResidentAgents<T> ag{};
      const ResidentLine<T> l = resident_line<T, 0>(p, tile);
      resident_tile<T, 0>(
          p, pl, coef, buf, l, [&] {
            resident_prefetch<T, 0>(p, tile + nw, ntx);
            if (!spread) ag = resident_agents<1>(p, tile, pl.agents, agents);
          },
          [&] {
            if (ag.a1 > ag.a0) resident_sources(p, ag, buf, pitch, l.tile);
          },
          none);
    }
    if (!bar.sync(p.status)) break;
    for (int tile = w0; tile < nty; tile += nw)
      resident_tile<T, 1>(p, pl, coef, buf, resident_line<T, 1>(p, tile),
                          [&] { resident_prefetch<T, 1>(p, tile + nw, nty); }, none, none);
    if (!bar.sync(p.status)) break;
    for (int tile = w0; tile < ntz; tile += nw)
      resident_tile<T, 2>(p, pl, coef, buf, resident_line<T, 2>(p, tile),
                          [&] { resident_prefetch<T, 2>(p, tile + nw, ntz); }, none, none);
    if (step + 1 < b.nsteps && !bar.sync(p.status)) break;
  }
  resident_leave(b.solve[m].barrier, ctas);
}

// Whether the sources go ahead of the x sweep, spread over `threads` threads.
// x tiles take them 32 at a time, about 1,000 cycles (an exact division, then
// the runs of stacked agents), `rounds` tiles one after another; the spread
// phase takes a barrier and up to 2,000 cycles for each agent of a thread.
// us per step, FP64, 10 steps, in the tiles -> spread: a plane of 300x260x3 with
// 10,000 agents and a rim of nodes 63 -> 41, of 537x74x3 with 8,000 (83 rounds)
// 100 -> 37; 200x200x200x1 with 1.6 million (3 x 40 rounds, 42 spread) 250 -> 182;
// but 64x64x64x8 FP32 with 52,000 (13 rounds, 11 spread) 25 -> 36, and spread at
// half these lines 24 uneven FP32 solves side by side 427 -> 470.
template <typename T>
bool resident_spreads(const bfvm_ctx* c, const SweepParams<T>& p, long long rounds, long long threads) {
  if (p.line_off == nullptr || static_cast<long long>(c->n_agents) * c->S > INT_MAX / 2) return false;
  const long long tiles = (static_cast<long long>(c->ny) * c->nz + 31) / 32;
  const long long in_tiles = rounds * ((c->n_agents / tiles + 31) / 32);
  return in_tiles > 8 + 2 * ((static_cast<long long>(c->n_agents) * c->S + threads - 1) / threads);
}

// ResidentPlan::crowd: as many as no tile of agents spread evenly holds, and as
// cost a tile of them more than the spread phase of `threads` threads.  us per
// step, FP64, 10 steps, by averages alone -> with this (a launch per stage):
//   50x50x50x2, 7,000 agents in a ball of 12 voxels' radius 29 -> 20 (32), 35,000
//     156 -> 27 (34), 10,000 in one of 6 158 -> 25 (37), 2,000 in one of 2 189 ->
//     32 (46), in eight voxels 279 -> 79 (87)
//   100x100x100x2, 20,000 in a ball of 12 94 -> 34 (52); 128x128x128x1, 30,000 in
//     one of 10 125 -> 37 (52); a plane of 300x260x3, 2,000 in a disc of 6 230 ->
//     39 (55)
// Slower than a launch per stage, which has more threads for them, where stacks
// are deep over a whole crowd: 30,000 in a disc of 20 of the plane (24 a voxel)
// 67 (57), FP32 65 (52); 64x64x64x2 FP32, 100,000 in a ball of 24 41 (37).
template <typename T>
int resident_crowd(const bfvm_ctx* c, const SweepParams<T>& p, long long threads) {
  if (p.line_off == nullptr || static_cast<long long>(c->n_agents) * c->S > INT_MAX / 2) return INT_MAX;
  const long long tiles = (static_cast<long long>(c->ny) * c->nz + 31) / 32;
  const long long each = (static_cast<long long>(c->n_agents) * c->S + threads - 1) / threads;
  return static_cast<int>(std::max(2 * (c->n_agents / tiles) + 32, 32 * (4 + 2 * each)));
}

// Shapes and shared memory of a solve's run, with one tile per warp (many
// false) or several; false where it does not fit.
template <typename T>
bool resident_plan(const bfvm_ctx* c, const SweepParams<T>& p, const NodeLines& nodes, bool two_d, bool many, int sms,
                   ResidentPlan* plan, long long* tiles, size_t* smem) {
  const SweepConfig& g = c->cfg;
  if (c->timing || c->sources_set || (p.line_off != nullptr && c->track) || c->sub_streams != 1 ||
      g.persistent != 1 || g.tmem != 1 || g.x_lines != 32 || g.yz_tile != 32)
    return false;
  if (!two_d && (partitioned<T, 1>(c, p) || partitioned<T, 2>(c, p))) return false;  // (serial lines here)
  const int n[3] = {c->nx, c->ny, c->nz}, S = c->S;
  const int naxes = two_d ? 2 : 3;
  ResidentPlan pl{};
  pl.two_d = two_d ? 1 : 0;
  if (!two_d) {
    const int zrows = (c->nz > 1 ? 2 : 1) * c->ny, yrows = (c->ny > 1 ? 2 : 1) * (c->nz > 2 ? c->nz - 2 : 0);
    pl.face_rows = zrows + yrows;
  }
  const long long xt = (c->nx + 31) / 32, xrows = (static_cast<long long>(c->ny) * c->nz + 31) / 32;
  tiles[0] = xrows * S;
  tiles[1] = xt * c->nz * S;
  tiles[2] = two_d ? 0 : xt * c->ny * S;
  const long long most = std::max(tiles[0], std::max(tiles[1], tiles[2]));
  if (most >= INT_MAX / 2) return false;
  const long long ctas = std::min<long long>(most, sms), per_cta = (most + ctas - 1) / ctas;
  pl.own = !many && per_cta == 1 ? 1 : 0;
  const size_t sets = pl.own ? 1 : S;
  size_t doubles = 0;
  const int drd = sizeof(typename Coef<T>::DR) / 8;
  for (int a = 0; a < naxes; ++a) {
    pl.rows[a] = (n[a] + kRowBatch - 1) / kRowBatch * kRowBatch;
    pl.line = std::max(pl.line, n[a]);
    pl.dr_off[a] = static_cast<int>(doubles);
    doubles += static_cast<size_t>(drd) * pl.rows[a] * sets;
    pl.cu_off[a] = static_cast<int>(doubles);
    doubles += static_cast<size_t>(pl.rows[a]) * sets;
    if (doubles * sizeof(double) > kSmemMax) return false;
  }
  const size_t coefs = doubles * sizeof(double);
  size_t each = static_cast<size_t>(32) * resident_pitch<T>(pl.line) * sizeof(T);
  for (int a = 0; a < 2 && nodes.n > 0; ++a) {
    pl.nodes[a] = (nodes.most[a] + 3) / 4 * 4;
    each += static_cast<size_t>(pl.nodes[a]) * (sizeof(T) + sizeof(int));
  }
  if (many) {
    pl.agents = p.line_off != nullptr ? 32 : 0;
    each += static_cast<size_t>(pl.agents) * kAgentBytes;
    pl.warps = static_cast<int>(std::min<size_t>(kManyWarps<T>, (kSmemMax - coefs) / each));
    if (pl.warps < 1) return false;
  } else {
    if (per_cta > kResidentWarps || per_cta * each + coefs > kSmemMax) return false;
    pl.warps = static_cast<int>(per_cta);
    pl.spread = resident_spreads(c, p, 1, static_cast<long long>(sms) * kSpreadThreads) ? 1 : 0;
    if (p.line_off != nullptr && !pl.spread) {  // room for a tile of twice the average, or what there is
      const long long fit = static_cast<long long>((kSmemMax - coefs) / pl.warps - each) / kAgentBytes;
      pl.agents = static_cast<int>(std::min<long long>(fit, 2 * (c->n_agents / xrows) + 32) / 4 * 4);
      each += static_cast<size_t>(pl.agents) * kAgentBytes;
    }
  }
  pl.warp_bytes = static_cast<int>(each);
  *plan = pl;
  *smem = pl.warps * each + coefs;
  return true;
}

template <typename T, int N>
cudaError_t launch_many(ResidentBatch<T, N>& b, int grid, size_t smem, int warps, int nsteps, cudaStream_t st,
                        int* launches) {
  int blocks = 0;
  cudaError_t e = persistent_grid(resident_many_kernel<T, N>, smem, grid, &blocks, 32 * warps);
  if (e != cudaSuccess) return e;
  if (blocks < grid) return cudaErrorLaunchOutOfResources;
  for (int done = 0; done < nsteps && e == cudaSuccess; done += b.nsteps) {
    b.nsteps = std::min(kResidentSteps, nsteps - done);
    void* args[] = {&b};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(resident_many_kernel<T, N>), dim3(grid),
                                    dim3(32 * warps), args, smem, st);
    if (e == cudaSuccess) ++*launches;
  }
  return e;
}

// Whether a solve with several tiles per warp is faster this way than with a
// launch per stage.  us per step, 10 steps a call, a launch per stage -> this:
//   FP64 100x100x100x3 71.9 -> 43.5   128x128x128x4 114 -> 78   200x200x200x1 136 -> 104
//        100x100x100x10 (80 MB) 130 -> 126, 64 steps 119 -> 123; 160x160x160x3
//        (98 MB) 152 -> 152, 140 -> 150; 200x200x200x4 (256 MB) 336 -> 428
//   FP32 100x100x100x3 54.6 -> 31.2   128x128x128x8 132 -> 89   200x200x200x2 169 -> 112
//        300x300x300x1 (108 MB) 264 -> 242, 200x200x200x4 (128 MB) 254 -> 236,
//        300x300x300x2 (216 MB) 409 -> 458
// Its warps hide an L2 latency, not DRAM's: the field has to stay in the L2, in
// FP64, with half the warps, well inside it.  And lines that leave room for
// fewer than three warps an SM are a serial chain with nothing beside it: FP64
// 256x128x128 (three) 98 -> 70, 300x100x100 (two) 73 -> 75, 400x64x64x2 (two)
// 81 -> 120.
template <typename T>
constexpr double kL2Share = sizeof(T) == 4 ? 1.0 : 0.55;

template <typename T>
bool resident_wins(const bfvm_ctx* c, const ResidentPlan& pl) {
  int l2 = 0;
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, c->device) != cudaSuccess) return false;
  const double bytes = static_cast<double>(sizeof(T)) * c->nx * c->ny * c->nz * c->S;
  return pl.warps >= 3 && bytes <= kL2Share<T> * l2;
}

// And for a solve that has the GPU to itself or shares it with others on
// streams of their own, which a launch per stage leaves more room for.  us per
// call, a launch per stage -> this, alone and three at once:
//   two CTAs to an SM: 50x50x50x2 FP64 1 step 32 -> 22 and 22 -> 10, 10 steps
//     309 -> 147 and 153 -> 54; 33x47x61x3 FP64 10 steps 319 -> 149 and 152 -> 80
//   one: 64x64x64x8 FP32 (seven warps an SM) 1 step 37 -> 28 and 19 -> 24, 4 steps
//     143 -> 78 and 71 -> 75
//   with agents in 1 voxel of 17: 100x100x100x3 FP64 702 -> 499 and 437 -> 502,
//     120x30x30x6 370 -> 205 and 163 -> 203: a tile takes them 32 at a time, a
//     launch of its own with all threads
// A run that fills the SMs is 1.3 to 2.2 times as fast alone, but others wait for
// it, and its idle warps are theirs.  Per call and solve, three at once:
//   10 steps, a tile per warp, FP32: 50x50x50x8 176 -> 160, 64x64x64x8 191 -> 178,
//     100x100x100x2 236 -> 230, 128x128x128x2 275 -> 280, 160x160x160x1 313 -> 330;
//     FP64: 50x50x50x8 184 -> 175, 64x64x64x8 211 -> 225, 80x80x80x4 234 -> 250,
//     100x100x100x2 256 -> 261, 112x112x112x2 283 -> 304; but fewer warps or lines
//     too short to hide the barriers in: 96x96x96x2 FP64 (four) 198 -> 234,
//     60x60x60x6 FP32 (five) 0.93 of it, 32x32x32x24 (lines of 32) 0.86; and lanes
//     or warps that idle: 58x25x184x2 FP32 (busy 0.25) 163 -> 182, 120x60x60x4
//     (0.65) 189 -> 201
//   20 steps, where a launch per stage replays its graph: FP32 50x50x50x8 293 ->
//     312, 100x100x100x2 395 -> 454; FP64 97x102x98x2 464 -> 525, 64x64x64x6 323 ->
//     387, 96x96x96x3 465 -> 549: FP64 gives way
//   several tiles per warp, either: FP64 50x50x50x20 (2.5 million values) 1.14 times
//     as fast, 64x64x64x12 0.95, 128x128x128x2 474 -> 479, 160x160x160x1 552 -> 533,
//     128x128x128x4 1025 -> 755, but 120x60x60x4 (1.7 million) 216 -> 280, 128x64x64x4
//     0.79 and 256x128x128x1 (busy 0.69) 0.91; FP32 64x64x64x16 0.89, 256x128x128x1
//     0.84, 200x200x100x1 355 -> 397: gives way; from 6 million values on, past the L2
//     three at once, all of them 0.95 to 1.7 (busy 0.70 and more; 100x100x100x3 FP64,
//     0.63, 402 -> 416)
//   planes, few tiles of long lines: 600x600x4 FP64 0.76, 400x700x4 0.62: gives way
template <typename T>
bool resident_shares(const bfvm_ctx* c, const SweepParams<T>& p, const long long* tiles, int sms, long long warps,
                     bool two_d, int nsteps) {
  const long long voxels = static_cast<long long>(c->nx) * c->ny * c->nz, values = voxels * c->S;
  if (two_d || nsteps < 4 || (p.line_off != nullptr && 32ll * c->n_agents > voxels)) return false;
  const long long n[3] = {c->nx, c->ny, c->nz};
  const long long most = std::max(tiles[0], std::max(tiles[1], tiles[2])), line = std::max(n[0], std::max(n[1], n[2]));
  double slots = 0;  // values that the warps' lanes could take meanwhile
  for (int a = 0; a < 3; ++a) slots += static_cast<double>((tiles[a] + warps - 1) / warps * warps) * 32 * n[a];
  const double busy = 3.0 * values / slots;
  if (values >= 6000000) return busy >= 0.65;
  if (most <= warps) return warps > 5ll * sms && busy >= 0.67 && line >= 40 && (sizeof(T) == 4 || nsteps <= 16);
  return sizeof(T) == 8 && values >= 2500000 && busy >= 0.75;
}

int sm_count(int device, int* sms) {
  BFVM_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device));
  return BFVM_OK;
}

}  // namespace

template <typename T>
int run_resident(bfvm_ctx* c, const SweepParams<T>& p, const NodeLines& nodes, bool two_d, int nsteps, cudaStream_t st,
                 int* launches) {
  *launches = 0;
  if (nsteps < 1) return BFVM_OK;
  int sms = 0;
  const int rc = sm_count(c->device, &sms);
  if (rc != BFVM_OK) return rc;
  ResidentPlan pl;
  long long tiles[3];
  size_t smem = 0;
  unsigned long long* barrier = c->d_tile_counter + 4;
  if (resident_plan(c, p, nodes, two_d, false, sms, &pl, tiles, &smem)) {
    int grid = static_cast<int>(std::min<long long>(std::max(tiles[0], std::max(tiles[1], tiles[2])), sms));
    int threads = 32 * pl.warps;
    // Eight warps an SM take that many agents' chains of divisions slower than a
    // launch of their own: 50x50x50x2 FP64, us per step of this and of a launch
    // per stage, 100,000 agents (11 a thread) 30 and 35, 200,000 (21) 48 and 38.
    if (p.line_off != nullptr && static_cast<long long>(c->n_agents) * c->S > 12ll * sms * kSpreadThreads)
      return BFVM_OK;
    if (pl.spread) {
      // Eight agents a thread, and two CTAs to an SM where their lines allow it:
      // a small grid leaves SMs to others' work (600x500x4 FP32 with 18,000
      // agents, 10 steps, three solves at once: 469 us a call on all SMs).
      const long long ctas =
          (static_cast<long long>(c->n_agents) * c->S + 8 * kSpreadThreads - 1) / (8 * kSpreadThreads);
      grid = static_cast<int>(std::max<long long>(grid, std::min<long long>(ctas, sms)));
      threads = std::max(threads, kSpreadThreads);
    } else if (p.line_off != nullptr && static_cast<long long>(c->n_agents) * c->S > 4ll * grid * threads) {
      threads = std::max(threads, kSpreadThreads);  // in case they crowd (resident_crowd)
    }
    // whether another such run finds room beside this one: 227 KB and eight warps an SM
    const long long per_sm = std::min<long long>(kSmemMax / smem, kResidentWarps / std::max(pl.warps, threads / 32));
    const long long all = static_cast<long long>(grid) * pl.warps;
    if (2 * grid > per_sm * sms && !resident_shares(c, p, tiles, sms, all, two_d, nsteps)) return BFVM_OK;
    pl.crowd = resident_crowd(c, p, static_cast<long long>(grid) * threads);
    int blocks = 0;
    BFVM_CUDA(persistent_grid(resident_kernel<T>, smem, grid, &blocks, threads));
    if (blocks < grid) return BFVM_OK;
    for (int done = 0; done < nsteps; done += pl.nsteps) {
      pl.nsteps = std::min(kResidentSteps, nsteps - done);
      void* args[] = {const_cast<SweepParams<T>*>(&p), &pl, const_cast<NodeLines*>(&nodes), &barrier};
      BFVM_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(resident_kernel<T>), dim3(grid),
                                            dim3(threads), args, smem, st));
      ++*launches;
    }
    return BFVM_OK;
  }
  if (!two_d && resident_plan(c, p, nodes, false, true, sms, &pl, tiles, &smem)) {
    const long long most = std::max(tiles[0], std::max(tiles[1], tiles[2]));
    const int grid = static_cast<int>(std::min<long long>(most, sms));
    const long long all = static_cast<long long>(grid) * pl.warps, rounds = (most + all - 1) / all;
    // no more warps than that many rounds need
    const int warps = static_cast<int>((most + grid * rounds - 1) / (grid * rounds));
    if (!resident_wins<T>(c, pl) || !resident_shares(c, p, tiles, sms, static_cast<long long>(grid) * warps, false, nsteps))
      return BFVM_OK;
    smem -= static_cast<size_t>(pl.warps - warps) * pl.warp_bytes;
    pl.warps = warps;
    const long long all_x = static_cast<long long>(grid) * warps;
    pl.spread = resident_spreads(c, p, (tiles[0] + all_x - 1) / all_x, 32ll * grid * kManyWarps<T>) ? 1 : 0;
    pl.crowd = resident_crowd(c, p, 32 * all_x);
    ResidentBatch<T, 1> b{};
    b.n = 1;
    b.solve[0] = {p, pl, 0, grid, barrier};
    BFVM_CUDA(launch_many(b, grid, smem, pl.spread ? kManyWarps<T> : warps, nsteps, st, launches));
  }
  return BFVM_OK;
}

// ---- a batch's solves ------------------------------------------------------

template <typename T>
bool resident_member(bfvm_ctx* c, bool sources) {
  int sms = 0;
  ResidentPlan pl;
  long long tiles[3];
  size_t smem;
  return sm_count(c->device, &sms) == BFVM_OK &&
         resident_plan(c, make_params<T>(c, sources), NodeLines{}, false, true, sms, &pl, tiles, &smem) &&
         resident_wins<T>(c, pl);
}

template <typename T>
cudaError_t run_resident_members(bfvm_ctx* const* members, int count, bool sources, int nsteps, cudaStream_t st,
                                 int* launches) {
  ResidentBatch<T, kResidentMembers> b{};
  int sms = 0;
  if (count == 0 || sm_count(members[0]->device, &sms) != BFVM_OK) return cudaGetLastError();
  // FP64 members go in launches of about equal bytes that stay in the L2 (what
  // resident_wins asks of one): 24 of edges 24 to 128 (490 MB) 792 -> 700 us a
  // step, 20 of edges to 110 421 -> 397; FP32's were as fast all at once (428
  // and 436).
  auto bytes = [&](int m) {
    const bfvm_ctx* c = members[m];
    return static_cast<double>(sizeof(T)) * c->nx * c->ny * c->nz * c->S;
  };
  int l2 = 0;
  cudaError_t e = cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, members[0]->device);
  if (e != cudaSuccess) return e;
  double total = 0;
  for (int m = 0; m < count; ++m) {
    // all or none: what some members' launches took would be steps ahead
    if (!resident_member<T>(members[m], sources)) return cudaErrorInvalidValue;
    total += bytes(m);
  }
  const double share = total / std::ceil(total / (kL2Share<T> * l2));
  for (int m0 = 0; m0 < count; m0 += b.n) {
    b.n = std::min(count - m0, std::min(kResidentMembers, sms));
    if (sizeof(T) == 8) {
      double taken = 0;
      int k = 0;
      for (; k < b.n && (k == 0 || taken + 0.5 * bytes(m0 + k) <= share); ++k) taken += bytes(m0 + k);
      b.n = k;
    }
    long long tiles[kResidentMembers][3];
    size_t smem = 0;
    int warps = 0;
    for (int m = 0; m < b.n; ++m) {
      bfvm_ctx* c = members[m0 + m];
      ResidentSolve<T>& s = b.solve[m];
      size_t need = 0;
      s.p = make_params<T>(c, sources);
      if (!resident_plan(c, s.p, NodeLines{}, false, true, sms, &s.pl, tiles[m], &need)) return cudaErrorInvalidValue;
      s.barrier = c->d_tile_counter + 4;
      s.ctas = 1;
      smem = std::max(smem, need);
      warps = std::max(warps, s.pl.warps);
    }
    // The SMs to the solves, one by one to the one that would take longest: a
    // tile's time goes with its line (cycles measured at 50 to 128 values).
    auto time = [&](int m) {
      const bfvm_ctx* c = members[m0 + m];
      const ResidentSolve<T>& s = b.solve[m];
      const int n[3] = {c->nx, c->ny, c->nz};
      const long long w = static_cast<long long>(s.ctas) * s.pl.warps;
      long long t = 0;
      for (int a = 0; a < 3; ++a) t += (tiles[m][a] + w - 1) / w * (2000 + 100 * n[a]) + 2500;
      return t;
    };
    long long took[kResidentMembers];
    for (int m = 0; m < b.n; ++m) took[m] = time(m);
    int grid = b.n;
    for (; grid < sms; ++grid) {
      const int worst = static_cast<int>(std::max_element(took, took + b.n) - took);
      ++b.solve[worst].ctas;
      took[worst] = time(worst);
    }
    int cta = 0;
    for (int m = 0; m < b.n; ++m) {
      b.solve[m].cta0 = cta;
      const long long w = static_cast<long long>(b.solve[m].ctas) * b.solve[m].pl.warps;
      b.solve[m].pl.spread =
          resident_spreads(members[m0 + m], b.solve[m].p, (tiles[m][0] + w - 1) / w, 32ll * warps * b.solve[m].ctas)
              ? 1
              : 0;
      b.solve[m].pl.crowd = resident_crowd(members[m0 + m], b.solve[m].p, 32ll * warps * b.solve[m].ctas);
      cta += b.solve[m].ctas;
    }
    e = launch_many(b, grid, smem, warps, nsteps, st, launches);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template bool resident_member<double>(bfvm_ctx*, bool);
template bool resident_member<float>(bfvm_ctx*, bool);
template cudaError_t run_resident_members<double>(bfvm_ctx* const*, int, bool, int, cudaStream_t, int*);
template cudaError_t run_resident_members<float>(bfvm_ctx* const*, int, bool, int, cudaStream_t, int*);
template int run_resident<double>(bfvm_ctx*, const SweepParams<double>&, const NodeLines&, bool, int, cudaStream_t,
                                  int*);
template int run_resident<float>(bfvm_ctx*, const SweepParams<float>&, const NodeLines&, bool, int, cudaStream_t,
                                 int*);

cudaError_t resident_set_wait_limit(unsigned long long ns) { return set_module_wait_limit(ns); }

}  // namespace bfvm
