// Line-by-line TDMA sweeps and the transport residual on the device.
//
// tdma_3d_mpi (src/mod_solver_3d.f90:252-366, serial branch) solves, per
// sweep, every r line (loop k, then j), every theta line (k, then i) and
// every z line (j, then i) with the Thomas algorithm `tdma` (:22-46),
// refreshing the theta halos before each direction. Each line solve reads
// phi in place, so a line sees the NEW values of the lines solved before it
// (Gauss-Seidel between lines) and the OLD values of the lines after it. The
// kernels keep exactly that: the result is bit-identical to the sequential
// sweep.
//
// Schedule. In a direction the lines form a grid (a, b) and line (a, b)
// needs the new values of (a-1, b) and (a, b-1) only, so the critical path is
// A + B - 1 dependent line solves. One warp (the solver of owner b) solves
// its chain a = 0..A-1 in order, keeping its previous line in registers; the
// line of the previous owner arrives through a hand-over slot whose value is
// its own signal (slots hold a signalling NaN, which arithmetic never
// produces, until written, and the consumer marks them empty again). G
// adjacent owners share a block and hand over through shared memory; only
// every G-th hand-over crosses blocks, through global memory (the mail warp
// of the consuming block fetches it ahead of the solver). A loader warp per
// solver copies the next lines' operands into a ring of buffers. The owner is
// the shorter of the two line indices, never theta (its periodic halo must
// keep the old values until its chain ends).
//
// A line solve. Both halves of the Thomas solve that depend on phi,
//   dp_i = (d_i - a_i dp_{i-1}) / m_i,   x_i = dp_i - cp_i x_{i+1},
// are first-order recurrences of correctly rounded operations, sequential in
// i. One lane running them took 95 ns an element, all of it latency. Here
// each lane owns K = ceil(L/32) consecutive elements and needs only the
// value entering its segment. A prefix scan of the segments' affine maps
// gives that to a few ulps; then every lane runs its segment with the
// sequential operations and hands its last value on, and the warp repeats
// until no entering value changes by a single bit. Then, by induction from
// lane 0, whose input is exact, every value is the sequential recurrence's,
// whatever the scan delivered. Two passes are the rule, because a segment
// contracts an error of a few ulps below a rounding; a line without
// contraction takes up to 32, about the sequential cost. Per line of 120
// elements the recurrences are 2 x 8 dependent elements long instead of
// 2 x 120.
//
// What does not depend on phi -- the guarded pivots m_i, cp_i, y_i = 1/m_i
// and the scan's segment products -- is computed once per call, by the same
// fixed-point passes, in a record per line and direction that also holds the
// line's coefficients in the order the solver's lanes read them, so a line
// is one bulk copy plus the old neighbour values.
// Built with -fmad=false like the CG unit.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "cg_common.cuh"
#include "cg_kernels.h"
#include "cluster_red.cuh"
#include "recipdiv.cuh"
#include "stencil.cuh"
#include "stream_stage.cuh"
#include "eafcg.h"

namespace eaf {
namespace {

__device__ __forceinline__ double sign_small(double v) {
  return fabs(v) < kSmall ? copysign(kSmall, v) : v;
}

constexpr int kTdmaMaxLine = 1024;
constexpr unsigned kAllLanes = 0xffffffffu;

// Record of one line: nine arrays of W = 32 K doubles, element lane*K + k of
// the line at [k][lane]; the scan's products, [step][lane], forward then
// backward; four scalars.
enum { kRSu, kR1m, kR1p, kR2m, kR2p, kRLo, kRM, kRY, kRCp, kRArrays };
constexpr int kScanSteps = 5;
enum { kRE0, kRE1, kRNf, kRNb, kRScalars };  // end links, scan steps needed

// Sizes for K elements a lane: owners per block, operand buffers per owner
// and hand-over slots per ring, as many as 220 KB of shared memory hold (at
// least three buffers before a further owner).
template <int K>
struct LineGeo {
  static constexpr int W = 32 * K;
  static constexpr int kScanF = kRArrays * W;
  static constexpr int kScanB = kScanF + 32 * kScanSteps;
  static constexpr int kScalars = kScanB + 32 * kScanSteps;
  static constexpr int kRec = kScalars + kRScalars;
  static constexpr int kP1 = kRec, kP2 = kRec + W, kEnds = kRec + 2 * W;
  static constexpr int kBuf = kEnds + 4;
  static constexpr int kSlots = K <= 16 ? 4 : 2;
  static constexpr int kLimit = 220 * 1024 / 8;
  static constexpr int need(int g, int nb) { return g * (nb * kBuf + kSlots * W); }
  static constexpr int owners() {
    for (int g = 8; g > 1; --g)
      if ((g <= 4 || K <= 2) && need(g, 3) <= kLimit) return g;
    return 1;
  }
  static constexpr int G = owners();
  static constexpr int NB = need(G, 4) <= kLimit ? 4 : need(G, 3) <= kLimit ? 3 : 2;
  static constexpr int kThreads = 32 * (2 * G + 1);
  static constexpr size_t kSmem = (size_t)need(G, NB) * sizeof(double);
  static_assert(need(G, NB) <= kLimit, "line buffers exceed the shared memory");
};

// One direction. Cell (a, b, e) sits at halo index base + a*sa + b*sb + e*se;
// pair 1 and pair 2 are the neighbour pairs of the right-hand side
//   d = (Su + c1m*n1m) + c1p*n1p;  d = (d + c2m*n2m) + c2p*n2p
// in the reference's order (strides s1, s2); the chain runs along pair 1
// (chain1) or pair 2.
struct Dir {
  int A, B, L;
  long long base, sa, sb, se, s1, s2;
  const double *c1m, *c1p, *c2m, *c2p, *lm, *lp, *aP, *Su;
  bool chain1;
  bool b_fast;  // the owner index is the unit-stride one
  int wrap;     // refresh theta halos: 0 no, 1 theta is the chain, 2 the line
  long long sx;
};

struct FactorArgs {
  Dir d;
  double* rec;
  double* mail;       // hand-over slots between blocks, marked empty here
  double* phi;        // non-null: refresh the theta halos (first direction)
  int nr, nth, nz;
  int* err;
};

struct SweepArgs {
  Dir d;
  const double* rec;
  double* mail;
  double* phi;
  int* err;
  uint64_t timeout_ns;
};

// Empty hand-over slot: a signalling NaN (IEEE arithmetic only delivers
// quiet NaNs, so no solution value has this pattern).
constexpr unsigned long long kEmptyBits = 0x7ff000017ff00001ull;
__device__ __forceinline__ double empty_slot() {
  return __longlong_as_double((long long)kEmptyBits);
}
__device__ __forceinline__ bool is_empty(double v) {
  return (unsigned long long)__double_as_longlong(v) == kEmptyBits;
}
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// Serial theta-periodic halo copy (src/mod_mpi_topology.f90:303-311) over
// all (i, k) columns of the halo layout; with nth == 1 the second and fourth
// statements read the columns that the first and third just wrote.
__device__ void theta_wrap(double* phi, int nr, int nth, int nz) {
  const long long sx = nr + 4, sxy = sx * (nth + 4);
  const long long ncol = sx * (nz + 4);
  for (long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
       col += (long long)gridDim.x * blockDim.x) {
    double* p = phi + col % sx + sxy * (col / sx);
    auto J = [&](int j) { return (long long)(j + 1) * sx; };
    const double v0 = p[J(nth)], v1 = p[J(1)];
    const double vm = nth == 1 ? v0 : p[J(nth - 1)], v2 = nth == 1 ? v1 : p[J(2)];
    p[J(0)] = v0;
    p[J(-1)] = vm;
    p[J(nth + 1)] = v1;
    p[J(nth + 2)] = v2;
  }
}

// ---------------------------------------------------------------------------
// Line records: one warp per line. The pivots' recurrence (:30-38)
//   m_i = guard(b_i - a_i cp_{i-1}),  cp_i = c_i / m_i
// runs in the lanes' segments from the previous pass's entering values until
// none changes (the first pass starts from zero: the recurrence forgets its
// start within a few elements). Padding elements and the line's ends carry
// values that leave the solver's recurrences untouched: lo = 0 in the first
// element, cp = 0 in the last, and m = y = 1 with zero links beyond.
// Bound by its stores: 60x120x84, 200 MB of records.
// ---------------------------------------------------------------------------
constexpr int kFactorBlock = 256;

template <int K>
__global__ void __launch_bounds__(kFactorBlock) tdma_factor_kernel(FactorArgs a) {
  using Geo = LineGeo<K>;
  const Dir& d = a.d;
  const int lane = threadIdx.x & 31;
  const long long lines = (long long)d.A * d.B;
  const long long warps = (long long)gridDim.x * (kFactorBlock / 32);
  if (a.phi) theta_wrap(a.phi, a.nr, a.nth, a.nz);
  if (a.err && blockIdx.x == 0 && threadIdx.x == 0) *a.err = 0;
  for (long long t = (long long)blockIdx.x * (kFactorBlock / 32) + (threadIdx.x >> 5); t < lines;
       t += warps) {
    const int ch = d.b_fast ? (int)(t / d.B) : (int)(t % d.A);
    const int b = d.b_fast ? (int)(t % d.B) : (int)(t / d.A);
    const long long q0 = d.base + ch * d.sa + b * d.sb;
    double* rec = a.rec + ((long long)b * d.A + ch) * Geo::kRec;
    double lo[K], bb[K], cc[K], mm[K], cp[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      const long long q = q0 + e * d.se;
      const bool live = e < d.L;
      lo[k] = live && e > 0 ? -d.lm[q] : 0.0;
      bb[k] = live ? d.aP[q] : 1.0;
      cc[k] = live ? -d.lp[q] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      const long long q = q0 + e * d.se;
      const bool live = e < d.L;
      const int o = k * 32 + lane;
      rec[kRSu * Geo::W + o] = live ? d.Su[q] : 0.0;
      rec[kR1m * Geo::W + o] = live ? d.c1m[q] : 0.0;
      rec[kR1p * Geo::W + o] = live ? d.c1p[q] : 0.0;
      rec[kR2m * Geo::W + o] = live ? d.c2m[q] : 0.0;
      rec[kR2p * Geo::W + o] = live ? d.c2p[q] : 0.0;
    }
    double in = 0.0;
    for (int pass = 0; pass <= 32; ++pass) {
      double c = in;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        mm[k] = sign_small(bb[k] - lo[k] * c);
        c = cc[k] / mm[k];
        cp[k] = c;
      }
      double nin = __shfl_up_sync(kAllLanes, c, 1);
      if (lane == 0) nin = 0.0;
      if (__all_sync(kAllLanes, same_bits(nin, in))) break;
      in = nin;
    }
    double pf = 1.0, pb = 1.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      const int o = k * 32 + lane;
      const double y = exp_in_safe_range(mm[k]) ? 1.0 / mm[k] : 0.0;
      const double cpe = e < d.L - 1 ? cp[k] : 0.0;
      rec[kRLo * Geo::W + o] = lo[k];
      rec[kRM * Geo::W + o] = mm[k];
      rec[kRY * Geo::W + o] = y;
      rec[kRCp * Geo::W + o] = cpe;
      pf = pf * (-lo[k] * y);
      pb = pb * -cpe;
    }
    // Scan products: step s adds the value 2^s lanes away times the product
    // over the 2^s segments in between; a step whose products are all below
    // 2^-56 (and those after it) would change nothing and is left out.
    int nf = 0, nb = 0;
#pragma unroll
    for (int s = 0; s < kScanSteps; ++s) {
      rec[Geo::kScanF + 32 * s + lane] = pf;
      rec[Geo::kScanB + 32 * s + lane] = pb;
      if (nf == s && __any_sync(kAllLanes, !(fabs(pf) < 0x1p-56))) nf = s + 1;
      if (nb == s && __any_sync(kAllLanes, !(fabs(pb) < 0x1p-56))) nb = s + 1;
      pf = pf * __shfl_up_sync(kAllLanes, pf, 1 << s);
      pb = pb * __shfl_down_sync(kAllLanes, pb, 1 << s);
    }
    if (lane == 0) {
      double* sc = rec + Geo::kScalars;
      sc[kRE0] = d.lm[q0];
      sc[kRE1] = d.lp[q0 + (long long)(d.L - 1) * d.se];
      sc[kRNf] = (double)nf;
      sc[kRNb] = (double)nb;
    }
    if (b % Geo::G == 0) {
      double* slot = a.mail + ((long long)(b / Geo::G) * d.A + ch) * Geo::W;
#pragma unroll
      for (int k = 0; k < K; ++k) slot[k * 32 + lane] = empty_slot();
    }
  }
}

// ---------------------------------------------------------------------------
// Sweep of one direction.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double ld_volatile_f64(const double* p) {
  return *(const volatile double*)p;
}
__device__ __forceinline__ void st_volatile_f64(double* p, double v) {
  *(volatile double*)p = v;
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Bound of a polling loop; warp-uniform, true when the wait gives up (the
// error word is set, by this wait's expiry or by another's).
struct Patience {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  __device__ __forceinline__ bool gives_up(int* err, uint64_t timeout_ns) {
    if ((++spins & 63u) != 0) return false;
    int stop = 0;
    if ((threadIdx.x & 31) == 0) {
      if (spins == 64u) t0 = global_ns();
      if (ld_volatile_i32(err) != 0) {
        stop = 1;
      } else if (global_ns() - t0 > timeout_ns) {
        atomicCAS(err, 0, (int)EAF_ETIMEOUT);
        stop = 1;
      }
    }
    return __shfl_sync(kAllLanes, stop, 0) != 0;
  }
};

// Takes this lane's K values of a hand-over slot in shared memory once all
// have arrived, and marks them empty; with `next`, also waits until the lane's
// values of that slot (the one this line goes to) have been taken.
template <int K>
__device__ __forceinline__ bool take_slot(const SweepArgs& a, double* slot, const double* next,
                                          int lane, double (&v)[K]) {
  Patience w;
  for (;;) {
    bool ready = true;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      v[k] = ld_volatile_f64(slot + k * 32 + lane);
      ready = ready && !is_empty(v[k]);
    }
    if (next) {
#pragma unroll
      for (int k = 0; k < K; ++k) ready = ready && is_empty(ld_volatile_f64(next + k * 32 + lane));
    }
    if (__all_sync(kAllLanes, ready)) break;
    if (w.gives_up(a.err, a.timeout_ns)) return false;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) st_volatile_f64(slot + k * 32 + lane, empty_slot());
  return true;
}

// Writes a solved line from its buffer to phi, and the theta halos that it
// completes: its own where the line is a theta column; where theta is the
// chain, at the chain's end, the owner's columns (their old halo values are
// no longer needed; the lane reads back values that it wrote).
template <int K>
__device__ __forceinline__ void write_line(const SweepArgs& a, const double* buf, int b, int ch,
                                           int lane) {
  using Geo = LineGeo<K>;
  const Dir& d = a.d;
  double* p = a.phi + d.base + ch * d.sa + b * d.sb;
  double x[K];
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] = buf[Geo::kP1 + k * 32 + lane];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int e = lane * K + k;
    if (e < d.L) p[e * d.se] = x[k];
  }
  if (d.wrap == 2) {
    const int n = d.L, n2 = n > 1 ? n - 2 : 0, one = n > 1 ? 1 : 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      if (e == n - 1) p[-d.se] = x[k];
      if (e == n2) p[-2 * d.se] = x[k];
      if (e == 0) p[n * d.se] = x[k];
      if (e == one) p[(n + 1) * d.se] = x[k];
    }
  } else if (d.wrap == 1 && ch == d.A - 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      if (e >= d.L) continue;
      double* c = a.phi + d.base + b * d.sb + e * d.se;  // (e, j = 1)
      const int n = d.A;
      const double v0 = x[k], v1 = c[0];
      const double vm = n == 1 ? v0 : c[(n - 2) * d.sx], v2 = n == 1 ? v1 : c[d.sx];
      c[-d.sx] = v0;
      c[-2 * d.sx] = vm;
      c[n * d.sx] = v1;
      c[(n + 1) * d.sx] = v2;
    }
  }
}

// Position of a warp in its owners' lines, with the buffer it is in.
template <int K>
struct LineAt {
  int b, ch = 0, st = 0;
  uint32_t phase = 0;
  __device__ explicit LineAt(int w) : b(blockIdx.x * LineGeo<K>::G + w) {}
  __device__ __forceinline__ void next(int A) {
    if (++st == LineGeo<K>::NB) {
      st = 0;
      phase ^= 1u;
    }
    if (++ch == A) {
      ch = 0;
      b += gridDim.x * LineGeo<K>::G;
    }
  }
};

// Copies the operands of the owner's lines into its ring of buffers, as far
// ahead as the solver has finished with them, and writes each finished line
// out of its buffer before that is filled again. The old neighbour values may
// be read at any time before the line is solved: a line's plus-side
// neighbours are solved, and written, after it.
template <int K>
__device__ void load_lines(const SweepArgs& a, int w, double* bufs, uint64_t* full,
                           uint64_t* empty, int lane) {
  using Geo = LineGeo<K>;
  const Dir& d = a.d;
  LineAt<K> at(w), done(w);
  int ahead = 0;  // lines issued and not yet written out
  bool ok = true;
  while (ok && done.b < d.B) {
    if (ahead == Geo::NB || at.b >= d.B) {
      ok = mbar_wait(&empty[done.st], done.phase, a.err, a.timeout_ns);
      ok = __all_sync(kAllLanes, ok);
      if (!ok) break;
      write_line<K>(a, bufs + (size_t)done.st * Geo::kBuf, done.b, done.ch, lane);
      done.next(d.A);
      --ahead;
    }
    if (at.b >= d.B) continue;
    double* buf = bufs + (size_t)at.st * Geo::kBuf;
    const double* p = a.phi + d.base + at.ch * d.sa + at.b * d.sb;
    if (lane == 0) {
      mbar_arrive_expect(&full[at.st], Geo::kRec * 8);
      bulk_copy_g2s(buf, a.rec + ((long long)at.b * d.A + at.ch) * Geo::kRec, Geo::kRec * 8,
                    &full[at.st]);
      cp_async8(buf + Geo::kEnds, p - d.se);
      cp_async8(buf + Geo::kEnds + 1, p + d.L * d.se);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      if (e < d.L) {
        cp_async8(buf + Geo::kP1 + k * 32 + lane, p + e * d.se + d.s1);
        cp_async8(buf + Geo::kP2 + k * 32 + lane, p + e * d.se + d.s2);
      }
    }
    cp_async_arrive(&full[at.st]);
    at.next(d.A);
    ++ahead;
  }
  // After a wait gave up: no copy may still be in flight into this block's
  // memory when it leaves.
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (; ahead > 0; --ahead) {
    for (int n = 0; n < (1 << 20) && !mbar_test(&full[done.st], done.phase); ++n) {
    }
    done.next(d.A);
  }
}

// Fetches the lines that the block's first owner needs -- the previous
// block's last owner's, or the halo -- into the first ring.
template <int K>
__device__ void fetch_mail(const SweepArgs& a, double* ring, int lane) {
  using Geo = LineGeo<K>;
  const Dir& d = a.d;
  const long long so = d.chain1 ? d.s2 : d.s1;
  int sl = 0;
  for (int b = blockIdx.x * Geo::G; b < d.B; b += gridDim.x * Geo::G) {
    for (int ch = 0; ch < d.A; ++ch) {
      double v[K];
      if (b == 0) {
        const double* p = a.phi + d.base + ch * d.sa - so;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int e = lane * K + k;
          v[k] = e < d.L ? __ldcg(p + e * d.se) : 0.0;
        }
      } else {
        double* slot = a.mail + ((long long)(b / Geo::G) * d.A + ch) * Geo::W;
        Patience w;
        for (;;) {
          bool got = true;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            v[k] = ld_relaxed_f64(slot + k * 32 + lane);
            got = got && !is_empty(v[k]);
          }
          if (__all_sync(kAllLanes, got)) break;
          if (w.gives_up(a.err, a.timeout_ns)) return;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) st_relaxed_f64(slot + k * 32 + lane, empty_slot());
      }
      double* to = ring + (size_t)sl * Geo::W;
      sl = sl + 1 == Geo::kSlots ? 0 : sl + 1;
      Patience w;
      for (;;) {
        bool free = true;
#pragma unroll
        for (int k = 0; k < K; ++k) free = free && is_empty(ld_volatile_f64(to + k * 32 + lane));
        if (__all_sync(kAllLanes, free)) break;
        if (w.gives_up(a.err, a.timeout_ns)) return;
      }
#pragma unroll
      for (int k = 0; k < K; ++k) st_volatile_f64(to + k * 32 + lane, v[k]);
    }
  }
}

// One lane's segment of the forward recurrence from the entering value, in
// the sequential operations (division by the stored reciprocal and one
// correction, which is the correctly rounded quotient: recipdiv.cuh). A
// segment with an operand outside its range, or a numerator of -0 (the
// correction would turn it into +0), is redone with `/`; the empty asm keeps
// that division in a branch of its own (speculated, it doubled a pass).
template <int K>
__device__ __forceinline__ double forward_segment(const double (&dd)[K], const double (&lo)[K],
                                                  const double (&m)[K], const double (&y)[K],
                                                  bool y_ok, double in, double (&dp)[K]) {
  bool ok = y_ok;
  double p = in;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double t = dd[k] - lo[k] * p;
    const double q = t * y[k];
    p = __fma_rn(__fma_rn(-q, m[k], t), y[k], q);
    ok = ok && (__double_as_longlong(t) == 0 || exp_in_safe_range(t));
    dp[k] = p;
  }
  if (!ok) {
    asm volatile("" ::: "memory");
    p = in;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      p = (dd[k] - lo[k] * p) / m[k];
      dp[k] = p;
    }
  }
  return p;
}

template <int K>
__device__ __forceinline__ double backward_segment(const double (&dp)[K], const double (&cp)[K],
                                                   double in, double (&x)[K]) {
  double p = in;
#pragma unroll
  for (int k = K - 1; k >= 0; --k) {
    p = dp[k] - cp[k] * p;
    x[k] = p;
  }
  return p;
}

// Passes run before the first look at the fixed point, from the scan steps
// that the line needs (a measure of its segments' contraction): the scan
// leaves a few ulps, which two passes absorb where a segment contracts by
// 2^-7 or more.
__device__ __forceinline__ int first_passes(int scan_steps) {
  return scan_steps <= 3 ? 2 : scan_steps;
}

template <int K, bool CHAIN1>
__device__ void solve_lines(const SweepArgs& a, int w, double* bufs, uint64_t* full,
                            uint64_t* empty, double* ring, double* next_ring, int lane) {
  using Geo = LineGeo<K>;
  const Dir& d = a.d;
  const long long sc = CHAIN1 ? d.s1 : d.s2;
  const int last_lane = (d.L - 1) / K;
  int sl = 0;
  double x[K];
  for (LineAt<K> at(w); at.b < d.B; at.next(d.A)) {
    const bool feeds = at.b + 1 < d.B;
    const bool in_block = w + 1 < Geo::G;
    if (at.ch == 0) {  // the chain starts from the halo
      const double* p = a.phi + d.base + at.b * d.sb - sc;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int e = lane * K + k;
        x[k] = e < d.L ? __ldcg(p + e * d.se) : 0.0;
      }
    }
    const bool here = mbar_wait(&full[at.st], at.phase, a.err, a.timeout_ns);
    if (!__all_sync(kAllLanes, here)) return;
    double* buf = bufs + (size_t)at.st * Geo::kBuf;
    auto op = [buf, lane](int arr, int k) { return buf[arr * Geo::W + k * 32 + lane]; };
    double lo[K], m[K], y[K], cp[K], dd[K], t2[K];
    bool y_ok = true;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      lo[k] = op(kRLo, k);
      m[k] = op(kRM, k);
      y[k] = op(kRY, k);
      cp[k] = op(kRCp, k);
      y_ok = y_ok && y[k] != 0.0;
    }
    const double end0 = buf[Geo::kScalars + kRE0] * buf[Geo::kEnds];
    const double end1 = buf[Geo::kScalars + kRE1] * buf[Geo::kEnds + 1];
    const int nf = (int)buf[Geo::kScalars + kRNf], nb = (int)buf[Geo::kScalars + kRNb];
    double sf[kScanSteps], sb[kScanSteps];
#pragma unroll
    for (int s = 0; s < kScanSteps; ++s) {
      sf[s] = buf[Geo::kScanF + 32 * s + lane];
      sb[s] = buf[Geo::kScanB + 32 * s + lane];
    }
    double* to = next_ring + (size_t)sl * Geo::W;
    if (!take_slot<K>(a, ring + (size_t)sl * Geo::W, feeds && in_block ? to : nullptr, lane, t2))
      return;
    sl = sl + 1 == Geo::kSlots ? 0 : sl + 1;
    // right-hand side, the reference's order; the lagged couplings of the
    // segment ends come last (:299-302, :325-328, :352-355)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = lane * K + k;
      const double n1 = CHAIN1 ? x[k] : t2[k], n2 = CHAIN1 ? t2[k] : x[k];
      double t = op(kRSu, k) + op(kR1m, k) * n1;
      t = t + op(kR1p, k) * buf[Geo::kP1 + k * 32 + lane];
      t = t + op(kR2m, k) * n2;
      t = t + op(kR2p, k) * buf[Geo::kP2 + k * 32 + lane];
      if (e == 0) t = t + end0;
      if (e == d.L - 1) t = t + end1;
      dd[k] = t;
    }
    // Forward: entering values from the scan, then the passes.
    double dp[K];
    double u = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) u = __fma_rn(-lo[k] * y[k], u, dd[k] * y[k]);
#pragma unroll
    for (int s = 0; s < kScanSteps; ++s)
      if (s < nf) u = __fma_rn(sf[s], __shfl_up_sync(kAllLanes, u, 1 << s), u);
    auto enter_f = [lane](double out) {
      const double v = __shfl_up_sync(kAllLanes, out, 1);
      return lane == 0 ? 0.0 : v;
    };
    double inf = enter_f(u), nin = inf;
    for (int n = first_passes(nf); n > 0; --n) {
      inf = nin;
      nin = enter_f(forward_segment<K>(dd, lo, m, y, y_ok, inf, dp));
    }
    bool settled = same_bits(nin, inf);
    inf = nin;
    // Backward, likewise; padding elements enter it as zeros whatever the
    // forward passes left in them (0 * Inf), so the last element is dp itself.
    auto clear_pads = [&] {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (lane * K + k >= d.L) dp[k] = 0.0;
    };
    clear_pads();
    u = 0.0;
#pragma unroll
    for (int k = K - 1; k >= 0; --k) u = __fma_rn(-cp[k], u, dp[k]);
#pragma unroll
    for (int s = 0; s < kScanSteps; ++s)
      if (s < nb) u = __fma_rn(sb[s], __shfl_down_sync(kAllLanes, u, 1 << s), u);
    auto enter_b = [lane, last_lane](double out) {
      const double v = __shfl_down_sync(kAllLanes, out, 1);
      return lane >= last_lane ? 0.0 : v;
    };
    double inb = enter_b(u);
    nin = inb;
    for (int n = first_passes(nb); n > 0; --n) {
      inb = nin;
      nin = enter_b(backward_segment<K>(dp, cp, inb, x));
    }
    settled = settled && same_bits(nin, inb);
    inb = nin;
    if (!__all_sync(kAllLanes, settled)) {  // on to the fixed points, each at most 32 passes away
      for (int n = 0; n <= 32; ++n) {
        nin = enter_f(forward_segment<K>(dd, lo, m, y, y_ok, inf, dp));
        if (__all_sync(kAllLanes, same_bits(nin, inf))) break;
        inf = nin;
      }
      clear_pads();
      for (int n = 0; n <= 32; ++n) {
        nin = enter_b(backward_segment<K>(dp, cp, inb, x));
        if (__all_sync(kAllLanes, same_bits(nin, inb))) break;
        inb = nin;
      }
    }
    if (feeds && in_block) {
#pragma unroll
      for (int k = 0; k < K; ++k) st_volatile_f64(to + k * 32 + lane, x[k]);
    } else if (feeds) {
      double* mail = a.mail + ((long long)((at.b + 1) / Geo::G) * d.A + at.ch) * Geo::W;
#pragma unroll
      for (int k = 0; k < K; ++k) st_relaxed_f64(mail + k * 32 + lane, x[k]);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) buf[Geo::kP1 + k * 32 + lane] = x[k];
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[at.st]);
  }
}

// Warps 0..G-1 solve, G..2G-1 load and write, 2G fetches the mail. A warp whose wait
// gave up leaves; the others' waits see the error word and leave too.
template <int K, bool CHAIN1>
__global__ void __launch_bounds__(LineGeo<K>::kThreads, 1) tdma_sweep_kernel(SweepArgs a) {
  using Geo = LineGeo<K>;
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(8) uint64_t full[Geo::G][Geo::NB], empty[Geo::G][Geo::NB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* rings = sm + (size_t)Geo::G * Geo::NB * Geo::kBuf;
  for (int i = threadIdx.x; i < Geo::G * Geo::kSlots * Geo::W; i += Geo::kThreads)
    rings[i] = empty_slot();
  // padding elements' neighbour values are never loaded
  for (int i = threadIdx.x; i < Geo::G * Geo::NB * 2 * Geo::W; i += Geo::kThreads)
    sm[(size_t)(i / (2 * Geo::W)) * Geo::kBuf + Geo::kP1 + i % (2 * Geo::W)] = 0.0;
  if (threadIdx.x == 0) {
    for (int g = 0; g < Geo::G; ++g)
      for (int n = 0; n < Geo::NB; ++n) {
        mbar_init(&full[g][n], 33);  // the bulk copy's expect and 32 lanes' copies
        mbar_init(&empty[g][n], 1);
      }
    mbar_fence_init();
  }
  __syncthreads();
  if (warp < Geo::G) {
    solve_lines<K, CHAIN1>(a, warp, sm + (size_t)warp * Geo::NB * Geo::kBuf, full[warp],
                           empty[warp], rings + (size_t)warp * Geo::kSlots * Geo::W,
                           rings + (size_t)(warp + 1) * Geo::kSlots * Geo::W, lane);
  } else if (warp < 2 * Geo::G) {
    const int w = warp - Geo::G;
    load_lines<K>(a, w, sm + (size_t)w * Geo::NB * Geo::kBuf, full[w], empty[w], lane);
  } else {
    fetch_mail<K>(a, rings, lane);
  }
}

// ---------------------------------------------------------------------------
// compute_residual_3d_mpi (src/mod_solver_3d.f90:625-694), serial: one pass
// over the interior in the blocks' contiguous slices, the two sums reduced
// with the deterministic group all-reduce (the CG dots' association).
// ---------------------------------------------------------------------------
struct ResArgs {
  HaloInputs in;
  const double* phi;
  MeshDims d;
  long long sx, sxy;
  GroupWs ws;
  uint64_t timeout_ns;
};

__global__ void __launch_bounds__(1024) residual_kernel(ResArgs a) {
  Group g;
  g.counter = a.ws.counter;
  g.err = a.ws.err;
  g.part = a.ws.part;
  g.stage = group_stage_smem();
  g.nb = gridDim.x;
  g.bid = blockIdx.x;
  g.timeout_ns = a.timeout_ns;
  g.epoch = 0;
  const Slice own = own_slice(a.d.n, g.nb, g.bid);
  double v[2] = {0.0, 0.0};
  const HaloInputs& in = a.in;
  for (int c = own.begin + (int)threadIdx.x; c < own.end; c += blockDim.x) {
    int i, j, k;
    cell_ijk(a.d, c, i, j, k);
    const long long q = (i + 2) + a.sx * (j + 2) + a.sxy * (k + 2);
    const double P = in.aP[q], W = in.aW[q], E = in.aE[q], S = in.aS[q], N = in.aN[q],
                 B = in.aB[q], T = in.aT[q], U = in.Su[q];
    if (P == 1.0 && W == 0.0 && E == 0.0 && S == 0.0 && N == 0.0 && B == 0.0 &&
        T == 0.0) {
      v[0] = v[0] + 0.0;
      v[1] = v[1] + 0.0;
      continue;
    }
    const double* ph = a.phi;
    const double pc = ph[q];
    double r = U - P * pc + S * ph[q - a.sx] + N * ph[q + a.sx];
    r = r + W * ph[q - 1] + E * ph[q + 1];
    r = r + B * ph[q - a.sxy] + T * ph[q + a.sxy];
    const double t = fabs(U) + fabs(P * pc) + kSmall;
    v[0] = v[0] + r * r;
    v[1] = v[1] + t * t;
  }
  const bool ok = group_allsum<2>(v, g, 0);
  if (g.bid == 0 && threadIdx.x == 0) {
    SolveResult* res = a.ws.result;
    const int err = ld_volatile_i32(a.ws.err);
    res->status = err != 0 ? err : (ok ? EAF_OK : EAF_ETIMEOUT);
    res->n_iter = 0;
    res->n_outer = 0;
    res->sym = 0;
    res->residual = sqrt(v[0]) / (sqrt(v[1]) + kSmall);
    res->bnorm = 0.0;
  }
}

// Diagnostic: div_by_recip against `/`, bit for bit, on generated pairs.
// Case mix per index: random sign, mantissa and exponent in [-540, 540]
// (both paths); t = m * k for small integers k (exact quotients); t one ulp
// off m * k (quotients next to halfway points); zeros, infinities, NaN.
__device__ __forceinline__ unsigned long long splitmix(unsigned long long x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__device__ double gen_double(unsigned long long r, int emin, int emax) {
  const unsigned long long mant = r & 0xfffffffffffffull;
  const int span = emax - emin + 1;
  const int ex = emin + (int)((r >> 52) % (unsigned long long)span);
  const unsigned long long sign = (r >> 63) << 63;
  return __longlong_as_double((long long)(sign | ((unsigned long long)(ex + 1023) << 52) | mant));
}

__global__ void div_check_kernel(long long n, unsigned long long seed,
                                 unsigned long long* counts) {
  unsigned long long bad = 0, fast = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long r1 = splitmix(seed ^ (2 * (unsigned long long)i));
    const unsigned long long r2 = splitmix(seed ^ (2 * (unsigned long long)i + 1));
    double t, m;
    switch ((int)(i & 7)) {
      case 0: case 1: case 2:
        t = gen_double(r1, -540, 540);
        m = gen_double(r2, -540, 540);
        break;
      case 3: case 4: {
        m = gen_double(r2, -400, 400);
        const double k = (double)((long long)(r1 % 2000001ull) - 1000000);
        t = m * k;
        break;
      }
      case 5: case 6: {
        m = gen_double(r2, -400, 400);
        const double k = (double)((long long)(r1 % 2001ull) - 1000) + 0.5;
        const double p = m * k;
        t = (r1 >> 40) & 1 ? nextafter(p, 1e308) : nextafter(p, -1e308);
        break;
      }
      default: {
        const double specials[6] = {0.0, -0.0, __longlong_as_double(0x7ff0000000000000ll),
                                    __longlong_as_double((long long)0xfff0000000000000ull),
                                    __longlong_as_double(0x7ff8000000000000ll), 1e-310};
        t = (r1 & 1) ? specials[(r1 >> 1) % 6] : gen_double(r1, -540, 540);
        m = (r2 & 1) ? specials[(r2 >> 1) % 6] : gen_double(r2, -540, 540);
        break;
      }
    }
    const bool m_ok = exp_in_safe_range(m);
    const double y = m_ok ? 1.0 / m : 0.0;
    const double a = div_by_recip(t, m, y, m_ok);
    const double b = t / m;
    const bool same = (__double_as_longlong(a) == __double_as_longlong(b)) ||
                      (a != a && b != b);
    bad += same ? 0 : 1;
    fast += (m_ok && (t == 0.0 || exp_in_safe_range(t))) ? 1 : 0;
  }
  atomicAdd(counts, bad);
  atomicAdd(counts + 1, fast);
}

// Elements per lane of a line of L: the next instantiated size.
int line_k(int L) {
  const int k = (L + 31) / 32;
  return k <= 8 ? k : k <= 12 ? 12 : k <= 16 ? 16 : k <= 24 ? 24 : 32;
}

template <class F>
auto with_k(int k, F f) {
  switch (k) {
    case 1: return f(std::integral_constant<int, 1>());
    case 2: return f(std::integral_constant<int, 2>());
    case 3: return f(std::integral_constant<int, 3>());
    case 4: return f(std::integral_constant<int, 4>());
    case 5: return f(std::integral_constant<int, 5>());
    case 6: return f(std::integral_constant<int, 6>());
    case 7: return f(std::integral_constant<int, 7>());
    case 8: return f(std::integral_constant<int, 8>());
    case 12: return f(std::integral_constant<int, 12>());
    case 16: return f(std::integral_constant<int, 16>());
    case 24: return f(std::integral_constant<int, 24>());
    default: return f(std::integral_constant<int, 32>());
  }
}

// The three directions' geometry (r, theta, z lines). The chain of the r and
// z lines is theta; the theta lines' chain is the longer of r and z, since a
// hand-over between owners costs more than a step along the chain.
Dir make_dir(const HaloInputs& in, int nr, int nth, int nz, int dir) {
  const long long sx = nr + 4, sxy = sx * (nth + 4);
  Dir d;
  d.base = 2 + 2 * sx + 2 * sxy;  // cell (1, 1, 1)
  d.aP = in.aP;
  d.Su = in.Su;
  d.sx = sx;
  d.wrap = dir == 1 ? 2 : 1;
  d.b_fast = false;
  d.chain1 = true;
  if (dir == 0) {
    d.A = nth; d.B = nz; d.L = nr;
    d.sa = sx; d.sb = sxy; d.se = 1;
    d.s1 = sx; d.c1m = in.aS; d.c1p = in.aN;
    d.s2 = sxy; d.c2m = in.aB; d.c2p = in.aT;
    d.lm = in.aW; d.lp = in.aE;
  } else if (dir == 1) {
    d.L = nth;
    d.se = sx;
    d.s1 = 1; d.c1m = in.aW; d.c1p = in.aE;
    d.s2 = sxy; d.c2m = in.aB; d.c2p = in.aT;
    d.lm = in.aS; d.lp = in.aN;
    d.chain1 = nr >= nz;
    d.A = d.chain1 ? nr : nz; d.B = d.chain1 ? nz : nr;
    d.sa = d.chain1 ? 1 : sxy; d.sb = d.chain1 ? sxy : 1;
    d.b_fast = !d.chain1;
  } else {
    d.A = nth; d.B = nr; d.L = nz;
    d.sa = sx; d.sb = 1; d.se = sxy;
    d.s1 = sx; d.c1m = in.aS; d.c1p = in.aN;
    d.s2 = 1; d.c2m = in.aW; d.c2p = in.aE;
    d.lm = in.aB; d.lp = in.aT;
    d.b_fast = true;
  }
  return d;
}

struct DirSizes {
  size_t rec, mail;  // doubles
  int blocks, threads;
};

DirSizes dir_sizes(const Dir& d) {
  return with_k(line_k(d.L), [&d](auto k) {
    using Geo = LineGeo<decltype(k)::value>;
    const int blocks = (d.B + Geo::G - 1) / Geo::G;
    return DirSizes{(size_t)d.A * d.B * Geo::kRec, (size_t)blocks * d.A * Geo::W, blocks,
                    Geo::kThreads};
  });
}

template <int K, bool CHAIN1>
cudaError_t launch_sweep(const SweepArgs& a, int sms, cudaStream_t st) {
  using Geo = LineGeo<K>;
  const void* k = (const void*)tdma_sweep_kernel<K, CHAIN1>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)Geo::kSmem);
  if (e != cudaSuccess) return e;
  // One block per SM; further owners follow in rounds.
  const int blocks = (a.d.B + Geo::G - 1) / Geo::G;
  SweepArgs copy = a;
  void* args[] = {&copy};
  return cudaLaunchCooperativeKernel(k, dim3(blocks < sms ? blocks : sms), dim3(Geo::kThreads),
                                     args, Geo::kSmem, st);
}

}  // namespace

size_t tdma_mailbox_doubles(int nr, int nth, int nz) {
  size_t most = 0;
  for (int dir = 0; dir < 3; ++dir) {
    const size_t n = dir_sizes(make_dir(HaloInputs{}, nr, nth, nz, dir)).mail;
    if (n > most) most = n;
  }
  return most;
}

size_t tdma_factor_doubles(int nr, int nth, int nz) {
  size_t sum = 0;
  for (int dir = 0; dir < 3; ++dir)
    sum += dir_sizes(make_dir(HaloInputs{}, nr, nth, nz, dir)).rec;
  return sum;
}

void tdma_launch_shape(int nr, int nth, int nz, int sms, int* grid, int* block) {
  *grid = 1;
  *block = 1;
  for (int dir = 0; dir < 3; ++dir) {
    const DirSizes s = dir_sizes(make_dir(HaloInputs{}, nr, nth, nz, dir));
    if (s.blocks > *grid) *grid = s.blocks;
    if (s.threads > *block) *block = s.threads;
  }
  if (*grid > sms) *grid = sms;
}

cudaError_t launch_tdma_f64(const HaloInputs& in, double* phi, int nr, int nth, int nz,
                            int n_sweep, double* mbox, double* fac, int sms, const GroupWs& ws,
                            uint64_t timeout_ns, cudaStream_t st) {
  if (nr > kTdmaMaxLine || nth > kTdmaMaxLine || nz > kTdmaMaxLine)
    return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> attr_lock(launch_attr_mutex());
  (void)cudaGetLastError();  // report these launches' errors, not an older one
  const double* rec[3];
  for (int dir = 0; dir < 3; ++dir) {
    FactorArgs f;
    f.d = make_dir(in, nr, nth, nz, dir);
    f.rec = fac;
    f.mail = mbox;
    f.phi = dir == 0 ? phi : nullptr;
    f.err = dir == 0 ? ws.err : nullptr;
    f.nr = nr;
    f.nth = nth;
    f.nz = nz;
    rec[dir] = fac;
    fac += dir_sizes(f.d).rec;
    const long long lines = (long long)f.d.A * f.d.B;
    long long grid = (lines + kFactorBlock / 32 - 1) / (kFactorBlock / 32);
    if (grid > 8LL * sms) grid = 8LL * sms;
    with_k(line_k(f.d.L), [&](auto k) {
      tdma_factor_kernel<decltype(k)::value><<<(unsigned)grid, kFactorBlock, 0, st>>>(f);
      return 0;
    });
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  for (int sweep = 1; sweep <= n_sweep; ++sweep) {
    for (int dir = 0; dir < 3; ++dir) {
      SweepArgs a;
      a.d = make_dir(in, nr, nth, nz, dir);
      if (dir == 2 && sweep == n_sweep) a.d.wrap = 0;  // no refresh after the last direction
      a.rec = rec[dir];
      a.mail = mbox;
      a.phi = phi;
      a.err = ws.err;
      a.timeout_ns = timeout_ns;
      const cudaError_t e = with_k(line_k(a.d.L), [&](auto k) {
        constexpr int K = decltype(k)::value;
        return a.d.chain1 ? launch_sweep<K, true>(a, sms, st) : launch_sweep<K, false>(a, sms, st);
      });
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

cudaError_t launch_residual_f64(const HaloInputs& in, const double* phi, const MeshDims& d,
                                const GroupWs& ws, uint64_t timeout_ns, int grid, int block,
                                cudaStream_t st) {
  ResArgs a;
  a.in = in;
  a.phi = phi;
  a.d = d;
  a.sx = d.nr + 4;
  a.sxy = (long long)(d.nr + 4) * (d.nth + 4);
  a.ws = ws;
  a.timeout_ns = timeout_ns;
  cudaError_t e = cudaMemsetAsync(ws.counter, 0, sizeof(unsigned long long), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ws.err, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel((const void*)residual_kernel, dim3(grid), dim3(block),
                                     args, 0, st);
}

const void* residual_kernel_ptr() { return (const void*)residual_kernel; }

cudaError_t run_div_check(long long n, unsigned long long seed, unsigned long long* counts,
                          cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  div_check_kernel<<<592, 256, 0, st>>>(n, seed, counts);
  return cudaGetLastError();
}

}  // namespace eaf
