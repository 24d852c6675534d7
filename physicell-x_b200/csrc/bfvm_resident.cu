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
// stay on the SMs from the first step to the last.
//
// What a step takes, in cycles at 50x50x50x2 FP64 (156 tiles): per sweep a
// tile's copy in 1,200-1,500 (one memory latency), forward 2,500 (50 values of
// 32 dependent cycles and the loads about them), back 1,100-1,300, the x rows
// out 1,900, then the barrier 2,500-3,400 (two memory latencies and what the
// CTAs differ by); the sources 900.  Against a launch per stage, us per step in
// calls of 10 steps (of 64, where those replay a captured graph):
//   20x20x20x2    FP64 26.3 -> 12.7 (16.7 -> 10.8)
//   50x50x50x2    FP64 32.3 -> 15.5 (24.8 -> 13.9)  FP32 34.2 -> 15.3 (25.5 -> 13.5)
//   64x64x64x8    FP64 38.6 -> 22.9 (29.7 -> 21.2), seven warps to an SM
//   100x100x100x2 FP64 50.8 -> 28.7 (40.6 -> 26.6)  FP32 49.3 -> 26.2 (40.3 -> 23.9)
//   128x128x128x1 FP64 52.9 -> 28.8 (43.4 -> 27.0)
//   300x260 2-D x3 FP64 50.7 -> 30.3 (49.4 -> 27.5); with 10,000 agents and a
//                 rim of nodes 62.1 -> 51.3 (60.7 -> 46.7)
// It won at every size it takes, up to what an SM holds: eight warps of 248
// registers, or 227 KB of line buffers and coefficients.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "biofvm_b200.h"
#include "bfvm_ctx.h"
#include "bfvm_internal.h"
#include "bfvm_ptx.cuh"
#include "bfvm_sweep_common.cuh"

namespace bfvm {

namespace {

constexpr int kResidentWarps = 8;  // warps per CTA at most
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kAgentBytes = 3 * sizeof(double) + sizeof(int);
constexpr int kResidentSteps = 64;  // steps per launch at most, about a millisecond: other streams' kernels get a turn

// The grid-wide barrier: arrivals counted up from 0 for the whole launch.
// False once a wait has run out (bounded as every device-side wait here).
struct GridBarrier {
  unsigned long long* count;
  unsigned long long target = 0;
  bool ok = true;
  __device__ __forceinline__ bool sync(int* status) {
    __syncthreads();
    if (threadIdx.x == 0) {
      target += gridDim.x;
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
  int face_rows;  // y and z face lines of all activated substrates
  int dr_off[3];  // staged coefficient rows of each axis, in doubles from the coefficients' start
  int cu_off[3];
  int rows[3];    // rows per substrate of each axis
  // a warp's part of shared memory: the line buffer, then what the run reads
  // again every step, kept from its start: agents and nodes (x, y) in lists of
  // these lengths
  int agents, nodes[2];
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
template <typename T, int AXIS, typename Before, typename After>
__device__ __forceinline__ void resident_tile(const SweepParams<T>& p, const ResidentPlan& pl, const double* coef,
                                              T* buf, const ResidentLine<T>& l, Before before, After after) {
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
  const DR* dr = reinterpret_cast<const DR*>(coef + pl.dr_off[AXIS]) + static_cast<size_t>(s) * pl.rows[AXIS];
  const double* cu = coef + pl.cu_off[AXIS] + static_cast<size_t>(s) * pl.rows[AXIS];

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
// and takes 17.  Agents in a face line of an activated substrate are
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

template <typename T>
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
  for (int e = t; e < g.kept; e += 32) {
    const ResidentAgent a = resident_agent(p, g, g.a0 + e);
    g.k[e] = a.k1;
    g.k[e + cap] = a.k2;
    g.k[e + 2 * cap] = a.k3;
    g.at[e] = a.at;
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

template <typename T>
__global__ void __launch_bounds__(32 * kResidentWarps, 1)
    resident_kernel(const SweepParams<T> p, const ResidentPlan pl, const NodeLines nd, unsigned long long* barrier) {
  using DR = typename Coef<T>::DR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* const coef = reinterpret_cast<double*>(smem_raw + static_cast<size_t>(pl.warps) * pl.warp_bytes);
  const AxisCoefs<T>* axes[3] = {&p.ax, &p.ay, &p.az};
  const int naxes = pl.two_d ? 2 : 3;
  for (int a = 0; a < naxes; ++a) {
    const int rows = pl.rows[a], npad = axes[a]->npad;
    DR* dr = reinterpret_cast<DR*>(coef + pl.dr_off[a]);
    for (int q = threadIdx.x; q < rows * p.S; q += blockDim.x) {
      const int s = q / rows, r = q - s * rows;
      dr[q] = __ldg(axes[a]->dr + static_cast<size_t>(s) * npad + r);
      coef[pl.cu_off[a] + q] = __ldg(axes[a]->cu + static_cast<size_t>(s) * npad + r);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  const int w0 = blockIdx.x + gridDim.x * warp, nw = gridDim.x * pl.warps;  // neighbouring tiles on different SMs
  unsigned char* keep = smem_raw + static_cast<size_t>(warp) * pl.warp_bytes;
  T* const buf = reinterpret_cast<T*>(keep);
  const int pitch = resident_pitch<T>(p.nx);
  keep += static_cast<size_t>(32) * resident_pitch<T>(pl.line) * sizeof(T);
  const ResidentLine<T> lx = resident_line<T, 0>(p, w0), ly = resident_line<T, 1>(p, w0);
  ResidentLine<T> lz{};
  if (!pl.two_d) lz = resident_line<T, 2>(p, w0);
  const ResidentAgents<T> ag = resident_agents(p, w0, pl.agents, reinterpret_cast<double*>(keep));
  keep += static_cast<size_t>(pl.agents) * kAgentBytes;
  const ResidentNodes<T> xn = resident_nodes(p, nd, 0, w0, pl.nodes[0], keep);
  keep += static_cast<size_t>(pl.nodes[0]) * (sizeof(T) + sizeof(int));
  const ResidentNodes<T> yn = resident_nodes(p, nd, 1, w0, pl.nodes[1], keep);
  const int l0 = w0 % ((p.ny + 31) / 32) * 32;  // (of a plane)
  __syncwarp();
  ResidentFace<T> face{};
  if (w0 < pl.face_rows) face = resident_face(p, w0);
  const auto none = [] {};
  GridBarrier bar{barrier};
  for (int step = 0; step < pl.nsteps; ++step) {
    resident_tile<T, 0>(
        p, pl, coef, buf, lx,
        [&] {
          if (ag.a1 > ag.a0) resident_sources(p, ag, buf, pitch, lx.tile);
          if (xn.n > 0) resident_pin(p, xn, true, buf, pitch, l0);
        },
        [&] {
          if (xn.n > 0) resident_pin(p, xn, false, buf, pitch, l0);
        });
    resident_face_store(face, p.nx);
    for (int q = w0 + nw; q < pl.face_rows; q += nw) resident_face_store(resident_face(p, q), p.nx);
    if (!bar.sync(p.status)) break;
    resident_tile<T, 1>(p, pl, coef, buf, ly, none, none);
    if (yn.n > 0) resident_pin<T>(p, yn, true, nullptr, 0, 0);
    if (!pl.two_d) {
      if (!bar.sync(p.status)) break;
      resident_tile<T, 2>(p, pl, coef, buf, lz, none, none);
    }
    if (step + 1 < pl.nsteps && !bar.sync(p.status)) break;
  }
  // the launch's last CTA leaves the counters at zero for the next one
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(barrier + 1, 1ull) == gridDim.x - 1) {
      barrier[0] = 0;
      barrier[1] = 0;
    }
  }
}

}  // namespace

template <typename T>
int run_resident(bfvm_ctx* c, const SweepParams<T>& p, const NodeLines& nodes, bool two_d, int nsteps, cudaStream_t st,
                 bool* launched) {
  *launched = false;
  const SweepConfig& g = c->cfg;
  if (nsteps < 1 || c->timing || (p.line_off != nullptr && c->track) || c->sub_streams != 1 || g.persistent != 1 ||
      g.tmem != 1 || g.x_lines != 32 || g.yz_tile != 32)
    return BFVM_OK;
  const int n[3] = {c->nx, c->ny, c->nz}, S = c->S;
  const int naxes = two_d ? 2 : 3;
  ResidentPlan pl{};
  pl.two_d = two_d ? 1 : 0;
  size_t doubles = 0;
  const int drd = sizeof(typename Coef<T>::DR) / 8;
  for (int a = 0; a < naxes; ++a) {
    pl.rows[a] = (n[a] + kRowBatch - 1) / kRowBatch * kRowBatch;
    pl.line = std::max(pl.line, n[a]);
    pl.dr_off[a] = static_cast<int>(doubles);
    doubles += static_cast<size_t>(drd) * pl.rows[a] * S;
    pl.cu_off[a] = static_cast<int>(doubles);
    doubles += static_cast<size_t>(pl.rows[a]) * S;
    if (doubles * sizeof(double) > kSmemMax) return BFVM_OK;
  }
  if (!two_d) {
    int on = 0;
    for (int s = 0; s < S; ++s) on += c->active[s] ? 1 : 0;
    const int zrows = (c->nz > 1 ? 2 : 1) * c->ny, yrows = (c->ny > 1 ? 2 : 1) * (c->nz > 2 ? c->nz - 2 : 0);
    pl.face_rows = on * (zrows + yrows);
  }
  const long long xt = (c->nx + 31) / 32;
  long long tiles = (static_cast<long long>(c->ny) * c->nz + 31) / 32;
  tiles = std::max(tiles, xt * c->nz);
  if (!two_d) tiles = std::max(tiles, xt * c->ny);
  tiles *= S;
  int sms = 0;
  BFVM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  const int grid = static_cast<int>(std::min<long long>(tiles, sms));
  const long long warps = (tiles + grid - 1) / grid;
  if (warps > kResidentWarps) return BFVM_OK;
  pl.warps = static_cast<int>(warps);
  const size_t coefs = doubles * sizeof(double);
  size_t each = static_cast<size_t>(32) * resident_pitch<T>(pl.line) * sizeof(T);
  for (int a = 0; a < 2 && nodes.n > 0; ++a) {
    pl.nodes[a] = (nodes.most[a] + 3) / 4 * 4;
    each += static_cast<size_t>(pl.nodes[a]) * (sizeof(T) + sizeof(int));
  }
  if (warps * each + coefs > kSmemMax) return BFVM_OK;
  if (p.line_off != nullptr) {  // room for the agents of a tile with twice the average, or what there is
    const long long rows = (static_cast<long long>(c->ny) * c->nz + 31) / 32;
    const long long fit = static_cast<long long>((kSmemMax - coefs) / warps - each) / kAgentBytes;
    pl.agents = static_cast<int>(std::min<long long>(fit, 2 * (c->n_agents / rows) + 32) / 4 * 4);
    each += static_cast<size_t>(pl.agents) * kAgentBytes;
  }
  pl.warp_bytes = static_cast<int>(each);
  const size_t smem = warps * each + coefs;
  int blocks = 0;
  BFVM_CUDA(persistent_grid(resident_kernel<T>, smem, grid, &blocks, 32 * pl.warps));
  if (blocks < grid) return BFVM_OK;
  unsigned long long* barrier = c->d_tile_counter + 4;
  for (int done = 0; done < nsteps; done += pl.nsteps) {
    pl.nsteps = std::min(kResidentSteps, nsteps - done);
    void* args[] = {const_cast<SweepParams<T>*>(&p), &pl, const_cast<NodeLines*>(&nodes), &barrier};
    BFVM_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(resident_kernel<T>), dim3(grid),
                                          dim3(32 * pl.warps), args, smem, st));
  }
  *launched = true;
  return BFVM_OK;
}

template int run_resident<double>(bfvm_ctx*, const SweepParams<double>&, const NodeLines&, bool, int, cudaStream_t,
                                  bool*);
template int run_resident<float>(bfvm_ctx*, const SweepParams<float>&, const NodeLines&, bool, int, cudaStream_t,
                                 bool*);

cudaError_t resident_set_wait_limit(unsigned long long ns) { return set_module_wait_limit(ns); }

}  // namespace bfvm
