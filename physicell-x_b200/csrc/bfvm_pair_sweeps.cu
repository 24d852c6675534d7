// bfvm_pair_sweeps.cu -- the persistent sweeps whose warps run two tiles at
// once: the forward elimination of one tile beside the back substitution of
// the tile before it.
//
// Reference: the x, y and z sweeps of
// diffusion_decay_solver__constant_coefficients_LOD_3D_BLOCKING
// (BioFVM/BioFVM_solvers.cpp:352-777, one rank) with the Dirichlet pins of
// Microenvironment::apply_dirichlet_boundaries_conditions
// (BioFVM/BioFVM_microenvironment.cpp:348-446): the same operations in the
// same order on every line, so the same bits as the other sweep kernels.
//
// What bounds a sweep is the serial chain of each line: 4 dependent FP64
// operations forward (8 cycles each: 32 per value) and one back, with the
// line's forward results held on chip in between.  A warp that runs the two
// passes one after the other (bfvm_tmem_sweeps.cu) spends most of a tile's
// time in latencies of its own: per 16 values about 520 cycles of chain and,
// measured by clock reads, twice that in TMA issue (350), the barrier (70),
// shared-memory loads and stores (8 cycles each per warp), coefficient loads
// and register moves.  Here
//   * a warp runs tile B forward and tile A back in one instruction stream, so
//     the two chains and the loads and stores between them overlap, and a
//     tile's storage is filled again by the very step that empties it;
//   * a second warp per ring issues its TMA loads and stores and takes its
//     tiles; a slot carries an input in and a result out;
//   * a step reads the next step's inputs and writes its results within the
//     chains, and keeps the coefficients in registers where both chunks lie
//     past the factorization's fixed point.
// One step (16 FP64 values of 32 lines forward and back) takes about 1,270
// cycles of its warp; four warps per SM then move a field at the rate of the
// tiles' own copies (6.1 TB/s in the steady state of 200^3 x 16: 20.8 us per
// substrate and sweep), and what is left at 200^3 x 4 is the first tile's
// forward pass and the last one's back pass, with nothing beside them.
//
// Measured on one B200, us per sweep, single-tile rings before -> this form
// (FP64, 200^3 x 4: x 115 -> 110, y 119 -> 108, z 120 -> 108; with all four
// substrates activated x 160 -> 131; 256^3 x 2: y 114 -> 104; 300^3 x 2: x
// 241 -> 172, y 204 -> 172; 400^3: y 284 -> 223; 640^3: x 2222 -> 1614, y 2330
// -> 1579; 128^3 x 6: y 51.6 -> 47.3; FP32, 224^3 x 3: y 79 -> 72; 640^3: x
// 1157 -> 572, y 1153 -> 495).
#include <climits>
#include <type_traits>

#include "biofvm_b200.h"
#include "bfvm_internal.h"
#include "bfvm_pair_coefs.h"
#include "bfvm_ptx.cuh"
#include "bfvm_sweep_common.cuh"

namespace bfvm {

// The forms of one sweep.
template <typename T, int AXIS>
struct PairForm {
  static constexpr bool X = AXIS == 0;
  static constexpr int R = 128 / static_cast<int>(sizeof(T));                  // values of a line per chunk
  static constexpr int kCols = R * static_cast<int>(sizeof(T)) / 4;            // TMEM columns of a unit
  static constexpr uint32_t kChunkBytes = 32u * R * sizeof(T);
  using DR = typename Coef<T>::DR;
};

constexpr int kPairMaxSlots = 16;
constexpr int kPairLagSlots = 4;  // a slot refills one step late where there are more of them

// The launch's shape, the same for all its rings.
struct PairPlan {
  int C;      // chunks per line
  int rings;  // compute warps 0 .. rings-1; the CTA's second half of warps copies for them
  int D;      // slots of a ring (<= C)
  int KC;     // staged coefficient chunks a ring has room for,
  int conv;   // for lines whose rows are constant from this entry on
  int pw;     // packed partial tiles of the y/z sweeps (FieldMaps::pyz_w)
  int TU;     // units of a ring in TMEM; the other C - TU in shared memory
  uint32_t ring_bytes;
};

// Tiles of an x sweep per substrate: 32 consecutive rows of the planes
// 1 .. nz - 2 (running on across the ends of y rows), then of each z face.
__host__ __device__ __forceinline__ unsigned pair_x_tiles(int ny, int nz) {
  const unsigned face = (static_cast<unsigned>(ny) + 31) / 32;
  return (nz > 2 ? (static_cast<unsigned>(ny) * (nz - 2) + 31) / 32 : 0u) + (nz > 1 ? 2 : 1) * face;
}

// The x sweep's maps: rows of the planes 1 .. nz - 2, of plane 0 and of plane
// nz - 1, so that a tile's load and store end with its planes.  y/z sweeps:
// the regular tiles' map and the packed ones'.
struct PairMaps {
  CUtensorMap m[3];
};

struct PairTile {
  double c1, shift;  // the substrate's (shift: FP32)
  int a, b, s;       // x: first row of its map b; y/z: first x, plane
  int has;           // 0: no tile; bit 1: y/z packed tile (b its first plane); bit 2: activated substrate
};

// An x tile's first row (k * ny + j), and the rows of its map.
__device__ __forceinline__ int pair_x_row(const PairTile& q, int ny, int nz) {
  return q.a + (q.b == 0 ? ny : (q.b == 1 ? 0 : (nz - 1) * ny));
}
__device__ __forceinline__ int pair_x_rows(const PairTile& q, int ny, int nz) { return q.b == 0 ? (nz - 2) * ny : ny; }

// A ring's shared memory: slots | units past TMEM | forward coefficients |
// upper diagonal | full barriers | done barriers | tile queue.
template <typename T, int AXIS>
struct PairRing {
  using F = PairForm<T, AXIS>;
  unsigned char *slots, *units;
  typename F::DR* drs;
  double* cus;
  uint64_t *full, *done;
  PairTile* queue;  // [4]: the tile of round r in entry r & 3
  T* pins;          // x: [4][2][32] the lines' pinned ends, as the queue
  __device__ __forceinline__ PairRing(unsigned char* base, const PairPlan& pl) {
    slots = base;
    units = slots + static_cast<size_t>(pl.D) * F::kChunkBytes;
    drs = reinterpret_cast<typename F::DR*>(units + static_cast<size_t>(pl.C - pl.TU) * F::kChunkBytes);
    cus = reinterpret_cast<double*>(drs + static_cast<size_t>(pl.KC) * F::R);
    full = reinterpret_cast<uint64_t*>(cus + static_cast<size_t>(pl.KC) * F::R);
    done = full + kPairMaxSlots;
    queue = reinterpret_cast<PairTile*>(done + kPairMaxSlots);
    pins = reinterpret_cast<T*>(queue + 4);
  }
  static size_t bytes(const PairPlan& pl) {
    const size_t b = static_cast<size_t>(pl.D + pl.C - pl.TU) * F::kChunkBytes +
                     static_cast<size_t>(pl.KC) * F::R * (sizeof(typename F::DR) + 8) + 2 * kPairMaxSlots * 8 +
                     4 * sizeof(PairTile) + (F::X ? 4 * 2 * 32 * sizeof(T) : 0);
    return (b + 1023) / 1024 * 1024;
  }
};

// Wait of a copy thread, which has time: it sleeps in the barrier (up to a
// microsecond at a time) instead of taking issue slots from the compute warps.
__device__ __forceinline__ bool mbar_wait_idle(uint32_t bar, uint32_t parity) {
  unsigned long long t0 = 0;
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    const unsigned long long now = global_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > g_wait_limit_ns) return false;
  }
}

// The compute warps' wait: one test, and the bounded loop out of line.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) { return mbar_wait(bar, parity); }
enum { kPlain, kConst, kFace, kFull };
enum { kTmem, kShared, kEither };  // where a step's unit is

// The copies of one ring, by lane 0 of a warp.  Round r eliminates tile r forward
// and substitutes tile r - 1 back, in steps j = 0 .. C - 1: step j takes
// chunk j of the one in and gives chunk C - 1 - j of the other out, through
// one and the same slot.  A slot's full barrier completes when its input has
// landed (or, in the last round, when it is free); its done barrier when the
// compute warp has left the output there.
template <typename T, int AXIS>
__device__ __forceinline__ void pair_copy(const CUtensorMap* map, const SweepParams<T>& p,
                                          const PairPlan& pl, const PairRing<T, AXIS>& g) {
  using F = PairForm<T, AXIS>;
  constexpr bool X = F::X;
  const int C = pl.C, D = pl.D;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int nm = AXIS == 1 ? nz : ny;
  const int P = pl.pw > 0 ? 32 / pl.pw : 1;
  const unsigned ntr = pl.pw > 0 ? nx / 32 : (nx + 31) / 32;
  const unsigned nreg = X ? pair_x_tiles(ny, nz) : ntr * nm;
  const unsigned per_s = (!X && pl.pw > 0) ? nreg + (nm + P - 1) / P : nreg;
  const unsigned long long ntiles = static_cast<unsigned long long>(per_s) * (p.s_hi - p.s_lo);
  // x: tiles of 32 rows of the planes 1 .. nz - 2, and of each z face
  const unsigned nface = (static_cast<unsigned>(ny) + 31) / 32;
  const unsigned nmid = nz > 2 ? (static_cast<unsigned>(ny) * (nz - 2) + 31) / 32 : 0u;
  // The next tile for this ring.  A y/z tile whose lines all lie in an
  // activated face is final already; an x tile all of whose rows lie in a z
  // face is written by pair_z_faces.
  const int t = threadIdx.x & 31;
  auto grab_one = [&]() {
    PairTile r{};
    for (;;) {
      const unsigned long long v = atomicAdd(p.tile_counter, 1ull);
      if (v >= ntiles) return r;
      const unsigned sg = ntiles <= 0xffffffffull ? static_cast<unsigned>(v) / per_s : static_cast<unsigned>(v / per_s);
      const unsigned q = static_cast<unsigned>(v - static_cast<unsigned long long>(sg) * per_s);
      r.s = p.s_lo + static_cast<int>(sg);
      const int act = p.active[r.s] != 0;
      if (X) {
        // the planes between the z faces first, then the two z faces', which
        // an activated substrate leaves out (pair_z_faces writes them)
        r.b = q < nmid ? 0 : (q < nmid + nface ? 1 : 2);
        if (r.b != 0 && act) continue;
        r.a = static_cast<int>(r.b == 0 ? q : q - nmid - (r.b - 1) * nface) * 32;
      } else if (q >= nreg) {
        r.has = 2;
        r.b = static_cast<int>(q - nreg) * P;
        r.a = static_cast<int>(ntr) * 32;
      } else {
        r.b = static_cast<int>(q / ntr);
        r.a = static_cast<int>(q - static_cast<unsigned>(r.b) * ntr) * 32;
        if (act && (r.b == 0 || r.b == nm - 1)) continue;
      }
      r.has |= 1 | (act << 2);
      r.c1 = p.c1[r.s];
      r.shift = sizeof(T) == 4 ? p.shift[r.s] : 0.0;
      return r;
    }
  };
  // Tile of round r into the queue (whole warp).
  auto grab = [&](int r) {
    PairTile q{};
    if (t == 0) {
      q = grab_one();
      g.queue[r & 3] = q;
    }
    __syncwarp();
    q = g.queue[r & 3];
    if (X && (q.has & 4)) {  // the pinned ends of its lines
      const int rl = pair_x_row(q, ny, nz) + t;
      if (q.a + t < pair_x_rows(q, ny, nz)) {
        const double o = sizeof(T) == 4 ? p.off[q.s] : 0.0;
        const size_t at = static_cast<size_t>(q.s) * ny * nz + rl;
        const double a = __ldg(p.xface + at), b = __ldg(p.xface + static_cast<size_t>(p.S) * ny * nz + at);
        g.pins[(r & 3) * 64 + t] = static_cast<T>(sizeof(T) == 4 ? a - o : a);
        g.pins[(r & 3) * 64 + 32 + t] = static_cast<T>(sizeof(T) == 4 ? b - o : b);
      }
    }
    __syncwarp();
    return q;
  };
  auto slot_at = [&](int sl) { return smem_u32(g.slots + static_cast<size_t>(sl) * F::kChunkBytes); };
  auto load = [&](const PairTile& q, int c, int sl) {
    if (t != 0) return;
    const uint32_t bar = smem_u32(&g.full[sl]);
    if (!q.has) {  // no input: the slot is free
      mbar_arrive(bar);
      return;
    }
    mbar_expect_tx(bar, F::kChunkBytes);
    if (X)
      tma_load_3d(slot_at(sl), map + q.b, bar, c * F::R, q.a, q.s);
    else if (q.has & 2)  // the packed map's dimensions: x, planes, rows along the line, substrate
      tma_load_4d(slot_at(sl), map + 1, bar, q.a, q.b, c * F::R, q.s);
    else if (AXIS == 1)
      tma_load_4d(slot_at(sl), map, bar, q.a, c * F::R, q.b, q.s);
    else
      tma_load_4d(slot_at(sl), map, bar, q.a, q.b, c * F::R, q.s);
  };
  auto store = [&](const PairTile& q, int c, int sl) {
    if (X)
      tma_store_3d(map + q.b, slot_at(sl), c * F::R, q.a, q.s);
    else if (q.has & 2)
      tma_store_4d(map + 1, slot_at(sl), q.a, q.b, c * F::R, q.s);
    else if (AXIS == 1)
      tma_store_4d(map, slot_at(sl), q.a, c * F::R, q.b, q.s);
    else
      tma_store_4d(map, slot_at(sl), q.a, q.b, c * F::R, q.s);
  };

  PairTile tl = grab(0);               // the tile being loaded (round lr, next chunk lj)
  PairTile td{}, tn = tl;    // the tile being stored; the one after it
  int lr = 0, lj = 0, lsl = 0;
  bool loading = tl.has != 0;
  if (!loading) {  // nothing for this ring
    if (t == 0) mbar_arrive(smem_u32(&g.full[0]));
    return;
  }
  for (int c = 0; c < D; ++c) load(tl, c, c);
  lj = D;
  unsigned nload = D;
  // Step m is done: its output leaves, and the slot of step m - 1, whose
  // output has been read by then, takes the input D - 1 steps on (with few
  // slots: step m's own, after a wait, the input D steps on).
  const bool lag = D > kPairLagSlots;
  int sj = 0, ssl = 0;
  uint32_t spar = 0;
  bool first = true, ok = true;
  for (;;) {
    if (t == 0) ok = mbar_wait_idle(smem_u32(&g.done[ssl]), spar);
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    if (!ok) break;
    if (t == 0) {
      if (td.has) store(td, C - 1 - sj, ssl);
      tma_store_commit();
    }
    if (loading && !(first && lag)) {
      if (lj == C) {  // the next round's tile; a round without one follows the last
        lj = 0;
        ++lr;
        if (!tl.has) {
          loading = false;
        } else {
          tl = grab(lr);
        }
      }
      if (loading) {
        if (t == 0) {
          if (lag)
            tma_store_wait_read_1();
          else
            tma_store_wait_read();
        }
        load(tl, lj, lsl);
        ++nload;
        ++lj;
        if (++lsl == D) lsl = 0;
      }
    }
    first = false;
    if (++ssl == D) {
      ssl = 0;
      spar ^= 1u;
    }
    if (++sj == C) {  // the next round stores the tile that this one eliminated
      sj = 0;
      if (!tn.has) break;  // that was the round without a tile
      td = tn;
      tn = tl;  // the loads are at most one round ahead
    }
  }
  if (t == 0) tma_store_wait_read();
  if (!ok && t == 0) {
    // A wait gave up: loads still in flight land before the CTA ends (the
    // last phase of every full barrier, with the same bound).
    atomicExch(p.status, kDevTimeout);
    for (int q = 0; q < D; ++q) mbar_wait(smem_u32(&g.full[q]), (nload / D + (q < static_cast<int>(nload % D) ? 1 : 0) - 1) & 1);
  }
}

// One compute warp.  At step j of a round it runs two chains side by side,
// element by element: tile B's forward elimination over chunk j and tile A's
// back substitution over chunk C - 1 - j.
template <typename T, int AXIS, bool FAST, bool LONG>
__device__ __forceinline__ void pair_compute(const SweepParams<T>& p, const PairPlan& pl, const PairRing<T, AXIS>& g,
                                             uint32_t tbase) {
  using F = PairForm<T, AXIS>;
  using DR = typename F::DR;
  constexpr bool X = F::X;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int R = F::R;
  constexpr int kElems = 32 * R;
  constexpr unsigned kAll = 0xffffffffu;
  const int t = threadIdx.x & 31;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int n = X ? nx : (AXIS == 1 ? ny : nz);
  const int C = pl.C, D = pl.D;
  const int rows = ny * nz;  // x: lines of a substrate, row k * ny + j
  const int nm = AXIS == 1 ? nz : ny;
  const int pw = pl.pw, pw_log = pw > 0 ? 31 - __clz(pw) : 0;

  // ---- coefficient rows, staged per substrate ----
  const AxisCoefs<T>& ac = X ? p.ax : (AXIS == 1 ? p.ay : p.az);
  auto conv_of = [&](int s) {
    return pair_conv(C, R, n, ac.conv != nullptr ? __ldg(ac.conv + s) : n, pl.conv);
  };
  auto stage_chunks = [&](auto* dst, const auto* src, const PairConv& cv) {
    const int sh = cv.sh(), m = (C - sh) * R;
    __syncwarp();
    for (int q = t; q < m; q += 32) dst[q] = __ldg(src + q + (q / R > cv.k0 ? sh * R : 0));
    __syncwarp();
  };
  int dr_s = -1, cu_s = -1;
  PairConv dr_cv{0, C}, cu_cv{0, C};  // before the first tile: chunk 0 throughout
  DR dk{};          // B's converged forward coefficients
  double ck = 0.0;  // A's converged upper diagonal

  // ---- the lines of a tile, this lane's ----
  struct Line {
    T p0, p1;  // an activated substrate: the line's pinned ends
    unsigned off;  // x: the lanes whose line lies in a y or z face
    bool on;   // the recurrence writes this lane's line
    bool act;  // the substrate's faces are pinned
    bool edge; // some lane of the tile is not on
  };
  auto lines = [&](const PairTile& q, [[maybe_unused]] int r) {
    Line l;
    l.act = (q.has & 4) != 0;
    l.p0 = l.p1 = T(0);
    if constexpr (X) {
      const int rl = pair_x_row(q, ny, nz) + t;
      const bool valid = q.a + t < pair_x_rows(q, ny, nz);
      const int k = valid ? rl / ny : 0, j = valid ? rl - k * ny : 0;
      l.on = valid && !(l.act && (j == 0 || j == ny - 1 || k == 0 || k == nz - 1));
      if (l.act) {  // (a lane without a line reads what nothing uses)
        l.p0 = g.pins[(r & 3) * 64 + t];
        l.p1 = g.pins[(r & 3) * 64 + 32 + t];
      }
    } else {
      const int i = (q.has & 2) ? q.a + (t & (pw - 1)) : q.a + t;
      const int m = (q.has & 2) ? q.b + (t >> pw_log) : q.b;
      l.on = i < nx && m < nm && !(l.act && (i == 0 || i == nx - 1 || m == 0 || m == nm - 1));
    }
    l.edge = __any_sync(kAll, !l.on);
    l.off = X && l.act ? __ballot_sync(kAll, !l.on && q.a + t < pair_x_rows(q, ny, nz)) : 0u;
    return l;
  };

  // ---- units: where a chunk's forward results wait for the back
  // substitution.  A tile keeps chunk c in unit c, the next one in unit
  // C - 1 - c, and so on in turn: at step j the back substitution of tile A
  // empties the very unit that the forward elimination of tile B fills.
  constexpr int kRegs = F::kCols;
  static_assert(kRegs == 32, "a unit fills one 32-column load");
  T* const my_units = reinterpret_cast<T*>(g.units) + t;
  auto st_unit = [&](int u, const T (&yv)[R], bool in_tmem) {
    if (in_tmem) {
      __syncwarp();
      if constexpr (!F32)
        tmem_st16d(tbase + static_cast<uint32_t>(u) * F::kCols, yv);
      else
        tmem_st32f(tbase + static_cast<uint32_t>(u) * F::kCols, yv);
    } else {
      T* b = my_units + static_cast<size_t>(u - pl.TU) * kElems;
#pragma unroll
      for (int q = 0; q < R; ++q) b[q * 32] = yv[q];
    }
  };

  bool hasA = false, flip = false;
  PairTile ta{};
  Line la{};  // (no lane in a face)
  int sl = 0;
  uint32_t par = 0;
  // the chunk of this lane's line in a slot, element by element or whole
  auto slot_at = [&](int q) { return g.slots + static_cast<size_t>(q) * F::kChunkBytes; };
  auto elem = [&](unsigned char* slot, int q) -> T* {
    if constexpr (X)
      return swz_elem<T>(slot + t * 128, q, t & 7);
    else
      return reinterpret_cast<T*>(slot) + t + q * 32;
  };
  unsigned char* slot_p = g.slots;
  T v[R];  // the inputs of B's next chunk
  bool ok = mbar_wait(smem_u32(&g.full[0]), 0u);
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = *elem(slot_at(0), q);
  for (int r = 0;; ++r) {
    if (!__all_sync(kAll, ok)) {
      if (t == 0) atomicExch(p.status, kDevTimeout);
      return;
    }
    const PairTile tb = g.queue[r & 3];
    const bool hasB = tb.has != 0;
    if (!hasA && !hasB) return;
    Line lb = la;
    if (hasB) {
      lb = lines(tb, r);
      if (tb.s != dr_s) {
        dr_s = tb.s;
        dr_cv = conv_of(tb.s);
        stage_chunks(g.drs, ac.dr + static_cast<size_t>(tb.s) * ac.npad, dr_cv);
        dk = __ldg(ac.dr + static_cast<size_t>(tb.s) * ac.npad + max(n - 2, 0));
      }
    }
    const double c1 = tb.c1, shift = tb.shift;
    if (hasA && ta.s != cu_s) {
      cu_s = ta.s;
      cu_cv = conv_of(ta.s);
      stage_chunks(g.cus, ac.cu + static_cast<size_t>(ta.s) * ac.npad, cu_cv);
      ck = __ldg(ac.cu + static_cast<size_t>(ta.s) * ac.npad + max(n - 2, 0));
    }
    double y = -0.0, xn = -0.0;
    int hwmin = INT_MAX;
    // One step.  kPlain: whole chunks of lines that are all on; kConst: the
    // same where both chunks' coefficients are the factorization's fixed
    // point, kept in registers; kFace: kPlain with one or two lines of A in a y
    // face (x); kFull: everything else.
    auto step = [&](auto form, auto where, int j) __attribute__((always_inline)) {
      constexpr int FORM = decltype(form)::value, UNIT = decltype(where)::value;
      const int uu = flip ? C - 1 - j : j;
      const bool in_tmem = UNIT == kTmem || (UNIT == kEither && (!LONG || uu < pl.TU));
      constexpr bool FULL = FORM == kFull, CONST = FORM == kConst;
      constexpr bool FACE = X && (FULL || FORM == kFace);
      const int ca = C - 1 - j, u = flip ? ca : j;
      unsigned char* const slot = slot_p;
      const bool wrap = sl + 1 == D;
      const int nsl = wrap ? 0 : sl + 1;
      const uint32_t npar = par ^ (wrap ? 1u : 0u);
      unsigned char* const next = wrap ? g.slots : slot + F::kChunkBytes;
      uint32_t tr[kRegs];
      if (in_tmem) {
        __syncwarp();
        tmem_ld32_issue(tbase + static_cast<uint32_t>(u) * F::kCols, tr);
      }
      // ---- B's next inputs have landed; the slot's output may go in ----
      if (!FULL || hasB) {
        if (!mbar_try_wait(smem_u32(&g.full[nsl]), npar)) ok = ok && mbar_wait_slow(smem_u32(&g.full[nsl]), npar);
      } else if (j > 0) {
        if (!mbar_try_wait(smem_u32(&g.full[sl]), par)) ok = ok && mbar_wait_slow(smem_u32(&g.full[sl]), par);
      }
      if (FULL && hasB) {
        const int rb = j * R;
        if (lb.act) {
          // x: the pin before the sweep; y/z: the ends are pinned already and kept
          if (j == 0) {
            if (X)
              v[0] = lb.p0;
            else
              lb.p0 = v[0];
          }
          if (rb + R >= n) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
              if (rb + q == n - 1) {
                if (X)
                  v[q] = lb.p1;
                else
                  lb.p1 = v[q];
              }
            }
          }
        }
        if (rb + R > n) {  // past the line's end (TMA fill): any clean value
#pragma unroll
          for (int q = 0; q < R; ++q)
            if (rb + q >= n) v[q] = T(1);
        }
      }
      // x: lines in a y face leave as their pinned values: up to two of them (the
      // rows about the end of a plane) by coalesced loads that are under way
      // during the chains
      const unsigned faces = FACE ? la.off : 0u;
      const bool few_faces = __popc(faces) <= 2;
      constexpr int kVals = 2 * R / 32;  // FP64: half a warp per row
      [[maybe_unused]] int face_row[kVals];
      [[maybe_unused]] T face_val[kVals];
      auto face_plane = [&](int row) {  // the face plane's row of the tile's line `row`
        const int rl = pair_x_row(ta, ny, nz) + row, k = rl / ny, jj = rl - k * ny;
        return (k == 0 || k == nz - 1) ? p.zface + ((static_cast<size_t>(k == 0 ? 0 : 1) * p.S + ta.s) * ny + jj) * nx
                                       : p.yface + ((static_cast<size_t>(jj == 0 ? 0 : 1) * p.S + ta.s) * nz + k) * nx;
      };
      if (FACE && faces != 0 && few_faces) {
        const unsigned rest = faces & (faces - 1);
#pragma unroll
        for (int e = 0; e < kVals; ++e) {
          face_row[e] = __ffs((e == 1 || t >= R) && rest != 0 ? rest : faces) - 1;
          const int i = ca * R + (t & (R - 1));
          const double f = i < nx ? __ldg(face_plane(face_row[e]) + i) : 0.0;
          face_val[e] = static_cast<T>(F32 ? f - p.off[ta.s] : f);
        }
      }
      // ---- A's forward results of chunk ca ----
      T a[R];
      if (in_tmem) {
        __syncwarp();
        tmem_wait_ld32(tr);
#pragma unroll
        for (int q = 0; q < R; ++q) {
          if constexpr (F32)
            a[q] = __uint_as_float(tr[q]);
          else
            a[q] = __hiloint2double(static_cast<int>(tr[2 * q + 1]), static_cast<int>(tr[2 * q]));
        }
      } else {
        const T* b = my_units + static_cast<size_t>(u - pl.TU) * kElems;
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = b[q * 32];
      }
      // ---- the two chains, element by element side by side, with the
      // loads of B's next chunk and the stores of A's results among them ----
      const DR* __restrict__ df = g.drs + dr_cv.at(j) * R;
      const double2* __restrict__ cw = reinterpret_cast<const double2*>(g.cus + cu_cv.at(ca) * R);
      T yv[R];
      [[maybe_unused]] T ob[X ? 16 / sizeof(T) : 1];  // x: a 16-byte unit of results on its way out
      // coefficients, loaded kAhead elements early: the stores between them
      // keep the compiler from doing so
      constexpr int kAhead = 4;
      DR dq[kAhead];
      double2 cq[kAhead / 2];
      if constexpr (!CONST) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q) dq[q] = df[q];
#pragma unroll
        for (int q = 0; q < kAhead / 2; ++q) cq[q] = cw[R / 2 - 1 - q];
      }
      auto back = [&](int w) {
        double c2 = ck;
        if constexpr (!CONST) {
          const int e = R - 1 - w, h = (e / 2) % (kAhead / 2);
          c2 = (w & 1) ? cq[h].y : cq[h].x;
          if ((w & 1) == 0 && w / 2 - kAhead / 2 >= 0) cq[h] = cw[w / 2 - kAhead / 2];
        }
        xn = back_elem(c2, xn, static_cast<double>(a[w]));
        const T o = (FULL && !X && !la.on) ? a[w] : static_cast<T>(xn);
        if constexpr (X) {
          constexpr int U = 16 / sizeof(T);
          ob[w % U] = o;
          if (w % U == 0) {
            using Unit = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
            Unit uv;
            T* ev = reinterpret_cast<T*>(&uv);
#pragma unroll
            for (int e = 0; e < U; ++e) ev[e] = ob[e];
            *reinterpret_cast<Unit*>(slot + t * 128 + (((w / U) ^ (t & 7)) << 4)) = uv;
          }
        } else {
          *elem(slot, w) = o;
        }
      };
      if (!FULL || hasB) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          DR d = dk;
          if constexpr (!CONST) {
            d = dq[q % kAhead];
            if (q + kAhead < R) dq[q % kAhead] = df[q + kAhead];
          }
          if constexpr (F32) {
            if constexpr (FAST)
              y = __fma_rn(__dmul_rn(c1, d), y, __dmul_rn(static_cast<double>(v[q]) - shift, d));
            else
              y = __dmul_rn(__fma_rn(c1, y, static_cast<double>(v[q]) - shift), d);
            yv[q] = static_cast<float>(y);
          } else {
            if constexpr (FAST) {
              y = __fma_rn(d.x, y, __dmul_rn(v[q], d.y));
            } else {
              hwmin = min(hwmin, __double2hiint(v[q]));
              y = markstein(__fma_rn(c1, y, v[q]), d.x, d.y);
            }
            yv[q] = y;
          }
          // a line in a face keeps its input: it waits in the unit as it came
          if (FULL && !X && !lb.on) yv[q] = v[q];
          if constexpr (X) {
            constexpr int U = 16 / sizeof(T);
            if (q % U == U - 1) {
              using Unit = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
              const Unit uv = *reinterpret_cast<const Unit*>(next + t * 128 + (((q / U) ^ (t & 7)) << 4));
              const T* ev = reinterpret_cast<const T*>(&uv);
#pragma unroll
              for (int e = 0; e < U; ++e) v[q - (U - 1) + e] = ev[e];
            }
          } else {
            v[q] = *elem(next, q);
          }
          back(R - 1 - q);
        }
      } else {
#pragma unroll
        for (int q = R - 1; q >= 0; --q) back(q);
      }
      if (FACE && faces != 0) {
        __syncwarp();
        if (few_faces) {
#pragma unroll
          for (int e = 0; e < kVals; ++e)
            *swz_elem<T>(slot + face_row[e] * 128, t & (R - 1), face_row[e] & 7) = face_val[e];
        } else if (FULL && ((faces >> t) & 1u)) {
          const int ra = ca * R;
          const double* fv = face_plane(t);
          const double o = F32 ? p.off[ta.s] : 0.0;
#pragma unroll 4
          for (int q = 0; q < R; ++q) {
            const double f = ra + q < nx ? __ldg(fv + ra + q) : 0.0;
            *elem(slot, q) = static_cast<T>(F32 ? f - o : f);
          }
        }
        __syncwarp();
      }
      if (FULL && hasA) {
        const int ra = ca * R;
        if (la.act) {  // the pinned ends
          if (ca == 0) *elem(slot, 0) = la.p0;
          if (j == 0) *elem(slot, n - 1 - ra) = la.p1;
        }
      }
      fence_async_smem();
      __syncwarp();
      if (t == 0) mbar_arrive(smem_u32(&g.done[sl]));
      // ---- B's results take A's unit ----
      if (FULL && j * R + R > n) {
        // rows past the end: -0, which the back substitution carries down to
        // the line's last row unchanged (their upper diagonal is -0 too)
#pragma unroll
        for (int q = 0; q < R; ++q)
          if (j * R + q >= n) yv[q] = T(-0.0);
      }
      if (!FULL || hasB) st_unit(u, yv, in_tmem);
      sl = nsl;
      par = npar;
      slot_p = next;
    };
    // steps j0 .. j1 are not full ones; ka .. kb of them have both chunks'
    // coefficients converged
    const bool ends = lb.act || (hasA && la.act), all_full = !hasB || (X ? __popc(la.off) > 2 : lb.edge || (hasA && la.edge));
    const int j0 = all_full ? C : (ends ? 1 : 0), j1 = (n % R != 0 || ends) ? C - 2 : C - 1;
    const int ka = max(dr_cv.k0, C - 1 - cu_cv.k1), kb = min(dr_cv.k1, C - 1 - cu_cv.k0);
    // Runs of steps of one form, each in a loop of its own (one loop that
    // chose the form at every step had cost 0.2 of a step in register moves).
    const int jt = flip ? C - pl.TU : pl.TU;  // LONG: the first step past the change of units
    for (int j = 0; j < C;) {
      const bool full = j < j0 || j > j1, konst = !F32 && j >= ka && j <= kb;
      const bool shared = LONG && (flip ? j < jt : j >= jt);
      int end = j < j0 ? j0 : (j > j1 ? C : min(C, j1 + 1));
      if (!full) {
        if (!F32 && !(X && la.off != 0)) end = min(end, konst ? kb + 1 : (j < ka && kb >= ka ? ka : C));
        if (LONG && j < jt) end = min(end, jt);
      }
      using In = std::integral_constant<int, kTmem>;
      using Out = std::integral_constant<int, LONG ? kShared : kTmem>;
      if (full) {
        for (; j < end; ++j)
          step(std::integral_constant<int, kFull>{}, std::integral_constant<int, LONG ? kEither : kTmem>{}, j);
      } else if (X && la.off != 0) {
        using Form = std::integral_constant<int, X ? kFace : kPlain>;
        if (shared)
          for (; j < end; ++j) step(Form{}, Out{}, j);
        else
          for (; j < end; ++j) step(Form{}, In{}, j);
      } else if (konst) {
        using Form = std::integral_constant<int, F32 ? kPlain : kConst>;
        if (shared)
          for (; j < end; ++j) step(Form{}, Out{}, j);
        else
          for (; j < end; ++j) step(Form{}, In{}, j);
      } else {
        using Form = std::integral_constant<int, kPlain>;
        if (shared)
          for (; j < end; ++j) step(Form{}, Out{}, j);
        else
          for (; j < end; ++j) step(Form{}, In{}, j);
      }
    }
    __syncwarp();
    tmem_wait_st();
    if (!__all_sync(kAll, ok)) {
      if (t == 0) atomicExch(p.status, kDevTimeout);
      return;
    }
    if (!hasB) return;
    if constexpr (!F32 && !FAST) {
      // The screen, once per tile: a line with an input below 2^-960 (or
      // negative) anywhere is redone from its inputs, which are still in the
      // field (this tile's results leave only in the next round).
      if (__any_sync(kAll, lb.on && !screen_clean(p.screen, hwmin))) {
        const int i = X ? 0 : ((tb.has & 2) ? tb.a + (t & (pw - 1)) : tb.a + t);
        const int m = X ? 0 : ((tb.has & 2) ? tb.b + (t >> pw_log) : tb.b);
        const size_t stride = X ? 1 : (AXIS == 1 ? static_cast<size_t>(p.nxp) : static_cast<size_t>(p.nxp) * ny);
        const T* in = p.f + (X ? (static_cast<size_t>(tb.s) * rows + pair_x_row(tb, ny, nz) + t) * p.nxp
                               : (AXIS == 1 ? (static_cast<size_t>(tb.s) * nz + m) * ny * p.nxp
                                            : (static_cast<size_t>(tb.s) * nz * ny + m) * p.nxp) + i);
        y = -0.0;
        for (int c = 0; c < C; ++c) {
          double v[R], yv[R];
          double2 cf[R];
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const int row = c * R + q;
            v[q] = (lb.on && row < n) ? in[static_cast<size_t>(row) * stride] : 1.0;
            if (X && lb.act) {
              if (row == 0) v[q] = lb.p0;
              if (row == n - 1) v[q] = lb.p1;
            }
            cf[q] = g.drs[dr_cv.at(c) * R + q];
            yv[q] = 0.0;
          }
          if (lb.on) {
            y = forward_checked<R>(v, cf, c1, y, [&](int q, double val) { yv[q] = val; });
          } else if (!X && (i < nx && m < nm)) {  // a face's line, as it came
#pragma unroll
            for (int q = 0; q < R; ++q)
              if (c * R + q < n) yv[q] = in[static_cast<size_t>(c * R + q) * stride];
          }
#pragma unroll
          for (int q = 0; q < R; ++q)
            if (c * R + q >= n) yv[q] = -0.0;
          const int u = flip ? C - 1 - c : c;
          st_unit(u, yv, !LONG || u < pl.TU);
        }
        __syncwarp();
        tmem_wait_st();
      }
    }
    ta = tb;
    la = lb;
    hasA = true;
    flip = !flip;
  }
}

// The z faces of activated substrates, which the x sweep's tiles leave out:
// every row takes the face's values (its ends, the x faces').  A row per warp
// at a time, by all compute warps of the launch, while the first loads are
// under way.
template <typename T>
__device__ __forceinline__ void pair_z_faces(const SweepParams<T>& p, int warps) {
  const int nx = p.nx, ny = p.ny, nz = p.nz, t = threadIdx.x & 31;
  const size_t rows = static_cast<size_t>(ny) * nz;
  const int w0 = blockIdx.x * warps + (threadIdx.x >> 5), nw = gridDim.x * warps;
  const int nrow = (nz > 1 ? 2 : 1) * ny;  // rows per substrate: plane 0's, plane nz - 1's
  int at = w0;                             // this warp's next row, counted over the activated substrates
  for (int s = p.s_lo; s < p.s_hi; ++s) {
    if (p.active[s] == 0) continue;
    const double o = sizeof(T) == 4 ? p.off[s] : 0.0;
    for (; at < nrow; at += nw) {
      const int side = at >= ny ? 1 : 0, j = at - side * ny;
      const size_t row = side == 0 ? j : rows - ny + j;
      const double* src = p.zface + ((static_cast<size_t>(side) * p.S + s) * ny + j) * nx;
      const double* x0 = p.xface + static_cast<size_t>(s) * rows + row;
      T* dst = p.f + (static_cast<size_t>(s) * rows + row) * p.nxp;
      for (int i0 = t; i0 < nx; i0 += 8 * 32) {
        double f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = i0 + 32 * e;
          const double* q = i == nx - 1 ? x0 + static_cast<size_t>(p.S) * rows : (i == 0 ? x0 : src + i);
          f[e] = i < nx ? __ldg(q) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (i0 + 32 * e < nx) dst[i0 + 32 * e] = static_cast<T>(sizeof(T) == 4 ? f[e] - o : f[e]);
      }
    }
    at -= nrow;
  }
}

// RQ: rings per TMEM lane quarter, 1 or 2 (each then has half its columns).
template <typename T, int AXIS, bool FAST, bool LONG, int RQ>
__global__ void __launch_bounds__(64 * 4 * RQ, 1)
    sweep_pair_kernel(const __grid_constant__ PairMaps maps, const SweepParams<T> p, const PairPlan pl) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + smem_align_pad(smem_raw, 1024);
  const int warp = threadIdx.x >> 5, t = threadIdx.x & 31;
  constexpr int kMax = 4 * RQ;  // rings at most
  const int w = warp & (kMax - 1);  // the ring
  const PairRing<T, AXIS> g(base + static_cast<size_t>(w) * pl.ring_bytes, pl);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base + static_cast<size_t>(pl.rings) * pl.ring_bytes);
  if (threadIdx.x == 0) {
    prefetch_tmap(&maps.m[0]);
    if (AXIS == 0 || pl.pw > 0) prefetch_tmap(&maps.m[1]);
  }
  if (warp < pl.rings && t < pl.D) {
    mbar_init(smem_u32(&g.full[t]), 1);
    mbar_init(smem_u32(&g.done[t]), 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
    tmem_fence_before();
  }
  __syncthreads();
  tmem_fence_after();
  if (warp < kMax) {
    if constexpr (RQ == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    if (AXIS == 0) pair_z_faces(p, kMax);
    if (w < pl.rings)
      pair_compute<T, AXIS, FAST, LONG>(p, pl, g, *tmem_slot + (static_cast<uint32_t>(32 * (w & 3)) << 16) +
                                                      static_cast<uint32_t>((w >> 2) * (512 / RQ)));
    __syncwarp();
    tmem_wait_st();
    tmem_fence_before();
  } else {
    if constexpr (RQ == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    if (w < pl.rings) pair_copy<T, AXIS>(maps.m, p, pl, g);
  }
  __syncthreads();
  if (warp == 0) {
    tmem_fence_after();
    tmem_dealloc(*tmem_slot, 512);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(p.tile_counter + 1, 1ull) == gridDim.x - 1) {
      p.tile_counter[0] = 0;
      p.tile_counter[1] = 0;
    }
  }
}

// ---- launch policy ----

// alignment pad, the rings, the TMEM address word
static size_t pair_smem(const PairPlan& pl) {
  return 1024 + static_cast<size_t>(pl.rings) * pl.ring_bytes + 128;
}

// The launch's plan; false where no ring fits.  Lines of at most 8 chunks fit
// twice into a lane quarter's 512 columns and run two rings per quarter (the
// register file then split by setmaxnreg); longer ones one ring per quarter,
// chunks past TMEM's 16 in shared memory.  Slots: as many as fit up to 8
// (200^3 x 4, y: 121, 112, 108 and 107 us with 5, 6, 8 and 10), at least 3, as
// a step waits for the next step's input.
template <typename T, int AXIS>
static bool pair_plan(int n, int conv_max, int pw, PairPlan* out) {
  using F = PairForm<T, AXIS>;
  PairPlan pl{};
  pl.C = (n + F::R - 1) / F::R;
  pl.pw = pw;
  pl.conv = conv_max;
  pl.KC = pl.C - pair_conv(pl.C, F::R, n, conv_max).sh();
  const int rq = pl.C <= 256 / F::kCols ? 2 : 1;
  pl.TU = pl.C < 512 / rq / F::kCols ? pl.C : 512 / rq / F::kCols;
  for (pl.rings = 4 * rq; pl.rings >= 1; --pl.rings) {
    for (pl.D = pl.C < 8 ? pl.C : 8; pl.D >= 3; --pl.D) {
      pl.ring_bytes = static_cast<uint32_t>(PairRing<T, AXIS>::bytes(pl));
      if (pair_smem(pl) <= 227 * 1024) {
        *out = pl;
        return true;
      }
    }
  }
  return false;
}

// Whether this form is the faster one for lines of n values (measured on one
// B200 against the single-tile rings and, where those do not launch, the
// per-tile sweeps; time of this form over theirs):
//   FP64, more than 10 chunks: 0.79-0.95 from 2 tiles per ring on (176^3 x 2
//     to 256^3 x 2), 0.68-0.86 past 16 chunks; below 2 tiles per ring 1.08 at
//     200 x 60^2 x 2 but 0.5-0.7 past 16 chunks (500 x 60^2, 300 x 100^2);
//     9 and 10 chunks: 1.0-1.06 (144^3), so not taken; 4 to 8 chunks, two
//     rings per quarter: 0.88-0.99 from 2 tiles per ring on, 1.15-1.28 below;
//   FP32 (chunks of 32 values, two conversions per value each way): 0.43-0.9
//     past 8 chunks; up to 8 where the last chunk is nearly full and rings
//     get 4 tiles: 0.89-0.96 at 128^3 x 16 and 224^3 x 3, but 1.04 at 200^3 x 4
//     (224 values' work per line), 1.35 at 100^3 x 8.
// Past 16 chunks the plan must hold as many rings as the single-tile one
// (coefficients that converge late leave no room: then those rings run).
template <typename T>
static bool pair_wins(int n, const PairPlan& pl, long long tiles, int sms, bool any_count, int single_rings) {
  const long long rings = static_cast<long long>(sms) * pl.rings;
  const bool two = any_count || tiles >= 2 * rings;
  if (sizeof(T) == 8) {
    if (pl.C > 16) return pl.rings >= single_rings && (any_count || tiles >= 2 * sms);
    if (pl.C > 10) return two;
    return pl.C >= 4 && pl.C <= 8 && two;
  }
  if (pl.C > 8) return pl.rings * 2 >= single_rings && (any_count || tiles >= 2 * sms);
  return pl.C >= 4 && n * 100 >= 93 * 32 * pl.C && (any_count || tiles >= 4 * rings);
}

// The plan of the launch for this solve; false where another form runs.
template <typename T, int AXIS>
static cudaError_t pair_choose(int pw, const SweepParams<T>& p, const SweepConfig& cfg, PairPlan* pl, long long* tiles,
                               bool* takes) {
  *takes = false;
  const int n = AXIS == 0 ? p.nx : (AXIS == 1 ? p.ny : p.nz);
  if (cfg.persistent < 1 || cfg.tmem == 0 || (AXIS == 0 ? cfg.x_lines : cfg.yz_tile) != 32 ||
      (AXIS == 0 && p.line_off != nullptr))
    return cudaSuccess;
  const AxisCoefs<T>& ac = AXIS == 0 ? p.ax : (AXIS == 1 ? p.ay : p.az);
  if (!pair_plan<T, AXIS>(n, ac.conv ? ac.conv_max : n, pw, pl)) return cudaSuccess;
  long long per_s;
  if (AXIS == 0) {
    per_s = pair_x_tiles(p.ny, p.nz);
  } else {
    const int nm = AXIS == 1 ? p.nz : p.ny, P = pw > 0 ? 32 / pw : 1;
    per_s = pw > 0 ? static_cast<long long>(p.nx / 32) * nm + (nm + P - 1) / P
                   : static_cast<long long>((p.nx + 31) / 32) * nm;
  }
  *tiles = per_s * (p.s_hi - p.s_lo);
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  *takes = pair_wins<T>(n, *pl, *tiles, sms, cfg.persistent >= 2, tmem_single_rings(sizeof(T), AXIS, n, cfg));
  // few tiles: a tile or two per SM rather than full CTAs on some
  if (*tiles < static_cast<long long>(sms) * pl->rings) pl->rings = static_cast<int>((*tiles + sms - 1) / sms);
  return cudaSuccess;
}

template <typename T, int AXIS>
bool pair_takes(int pw, const SweepParams<T>& p, const SweepConfig& cfg) {
  PairPlan pl{};
  long long tiles = 0;
  bool takes = false;
  return pair_choose<T, AXIS>(pw, p, cfg, &pl, &tiles, &takes) == cudaSuccess && takes;
}

template <typename T, int AXIS>
cudaError_t launch_pair(const CUtensorMap* const (&map)[3], int pw, const SweepParams<T>& p, const SweepConfig& cfg,
                        cudaStream_t st, bool* launched) {
  *launched = false;
  PairPlan pl{};
  long long tiles = 0;
  bool takes = false;
  cudaError_t e = pair_choose<T, AXIS>(pw, p, cfg, &pl, &tiles, &takes);
  if (e != cudaSuccess || !takes) return e;
  // more than half of an SM's, so that one CTA has the SM's tensor memory
  size_t smem = pair_smem(pl);
  if (smem < 116 * 1024) smem = 116 * 1024;
  const bool fast = p.screen == kScreenFast, lng = pl.C > pl.TU;
  const bool two = pl.TU * 2 * PairForm<T, AXIS>::kCols <= 512;
  auto kern = two ? (fast ? sweep_pair_kernel<T, AXIS, true, false, 2> : sweep_pair_kernel<T, AXIS, false, false, 2>)
                  : (fast ? (lng ? sweep_pair_kernel<T, AXIS, true, true, 1> : sweep_pair_kernel<T, AXIS, true, false, 1>)
                          : (lng ? sweep_pair_kernel<T, AXIS, false, true, 1> : sweep_pair_kernel<T, AXIS, false, false, 1>));
  const int threads = two ? 512 : 256;
  PairMaps maps;
  for (int q = 0; q < 3; ++q) maps.m[q] = *map[q];
  int grid = 0;
  e = persistent_grid(kern, smem, (tiles + pl.rings - 1) / pl.rings, &grid, threads);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, st>>>(maps, p, pl);
  *launched = true;
  return cudaGetLastError();
}

#define BFVM_PAIR_INST(T, AXIS)                                                                                   \
  template cudaError_t launch_pair<T, AXIS>(const CUtensorMap* const (&)[3], int, const SweepParams<T>&,          \
                                            const SweepConfig&, cudaStream_t, bool*);                            \
  template bool pair_takes<T, AXIS>(int, const SweepParams<T>&, const SweepConfig&);
BFVM_PAIR_INST(double, 0)
BFVM_PAIR_INST(double, 1)
BFVM_PAIR_INST(double, 2)
BFVM_PAIR_INST(float, 0)
BFVM_PAIR_INST(float, 1)
BFVM_PAIR_INST(float, 2)

cudaError_t pair_sweeps_set_wait_limit(unsigned long long ns) { return set_module_wait_limit(ns); }

}  // namespace bfvm
