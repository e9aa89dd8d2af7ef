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
// every G-th hand-over crosses blocks, through global memory (the consuming
// block's mail warp fetches it ahead of the solver). A loader warp per solver
// copies the next lines' operands into a ring of buffers and writes the
// solved lines to phi. The owner is
// the shorter of the two line indices, never theta (its periodic halo must
// keep the old values until its chain ends).
//
// A line solve. Both halves of the Thomas solve that depend on phi,
//   dp_i = (d_i - a_i dp_{i-1}) / m_i,   x_i = dp_i - cp_i x_{i+1},
// are first-order recurrences of correctly rounded operations, sequential in
// i. One lane running them took 95 ns an element, all of it latency. Here a
// lane owns K consecutive elements and needs only the value entering its
// segment. A prefix scan of the segments' affine maps gives that to a few
// ulps; then every lane runs its segment with the sequential operations and
// hands its last value on, and the warp repeats until no entering value
// changes by a single bit. Then, by induction from lane 0, whose input is
// exact, every value is the sequential recurrence's, whatever the scan
// delivered. Two passes are the rule, because a segment contracts an error of
// a few ulps below a rounding; a line without contraction takes up to 32,
// about the sequential cost. (60x120x84, two sweeps, ms, a lane a line 8.5 on
// all: random links 1.62, conduction on the cylinder with a sink of 1e-2 of the
// links 1.84, of 1e-6 2.05, links of one direction 1e6 times the others' 3.29.) A pass costs 42 cycles an element (five
// dependent FP64 operations) plus a shuffle, so the passes needed times K is
// what counts: K = 4 on as few lanes as the line fills, more only beyond 128
// elements (one element a lane needs four to five passes and five scan steps).
//
// Layout. The sweep itself is bound by latency, so the transposing work is
// left to parallel kernels before it: what does not depend on phi -- the
// guarded pivots m_i, cp_i, y_i = 1/m_i (by the same fixed-point passes) and
// the scan's segment products -- is computed once per call (before a direction's
// sweep where the records of only one have room) into a record per
// line and direction, lane by lane; what a direction takes from the old phi
// (its plus-side neighbours, which no line changes before it is solved) goes
// into an old-value record per line before each direction. A line is then two
// bulk copies. (Gathering the old values in the sweep cost a third of it:
// every element of a theta or z line is a sector of its own.)
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

// Record of one line: four scalars, then per lane seven arrays of its K
// elements and the scan's products, forward and backward in turn. K is even
// and the lane strides are 2 mod 4, so that the lanes read 16 bytes at a time
// without bank conflicts.
enum { kRSu, kR1m, kR2m, kRLo, kRM, kRY, kRCp, kRArrays };
constexpr int kScanSteps = 5;
enum { kRE0, kRE1, kRNf, kRNb, kRScalars };  // end links, scan steps needed (and kUnsafe)
// Old values of one line: the two halo values beyond its ends (and two words
// of padding), then per lane the products of the plus-side neighbours of pairs
// 1 and 2 and the coupling of the line's far end (-0.0 elsewhere).
enum { kO1 = 0, kO2 = 1, kOEnd = 2, kOArrays = 3, kOScalars = 4 };
constexpr int kUnsafe = 8;  // added to the forward steps: a pivot outside the reciprocal's range

constexpr int lane_stride(int doubles) { return doubles + (6 - doubles % 4) % 4; }

template <int K>
struct Lanes {
  static_assert(K % 2 == 0, "16-byte reads");
  static constexpr int kScan = kRArrays * K;
  static constexpr int kRec = lane_stride(kScan + 2 * kScanSteps);  // in a record
  static constexpr int kOld = lane_stride(kOArrays * K);  // in old values
  static constexpr int kRing = lane_stride(K);     // of a hand-over slot
  static constexpr int kMail = 32 * K;             // slot between blocks
  // One owner per scheduler; long lines leave registers for fewer.
  static constexpr int kMaxOwners = K <= 8 ? 4 : K <= 16 ? 2 : 1;
  static constexpr int kMaxThreads = 32 * (2 * kMaxOwners + 1);
};

// Sizes for lines of L elements (doubles): lanes in use, record, old values,
// buffer (both), and owners per block, buffers per owner and hand-over slots
// per ring, as many as 220 KB of shared memory hold (three buffers before a
// further owner).
struct LineGeo {
  int n, rec, old, buf, G, NB, slots, ring;
  size_t smem;
};

template <int K>
LineGeo line_geo(int L) {
  using Ln = Lanes<K>;
  constexpr int limit = 220 * 1024 / 8;
  LineGeo g;
  g.n = (L + K - 1) / K;
  g.rec = (kRScalars + g.n * Ln::kRec + 1) & ~1;
  g.old = kOScalars + g.n * Ln::kOld;
  g.buf = g.rec + g.old;  // (all even: 16-byte copies and reads)
  g.ring = 32 * Ln::kRing;
  g.slots = K <= 16 ? 4 : 2;
  auto need = [&g](int owners, int nb) {
    return owners * (nb * g.buf + g.slots * g.ring) + Ln::kRec + Ln::kOld;
  };
  g.G = Ln::kMaxOwners;
  while (g.G > 1 && need(g.G, 3) > limit) --g.G;
  g.NB = need(g.G, 4) <= limit ? 4 : need(g.G, 3) <= limit ? 3 : 2;
  g.smem = (size_t)need(g.G, g.NB) * sizeof(double);
  return g;
}

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
  LineGeo g;
  int tile;           // lines per block
  double* rec;
  double* mail;       // hand-over slots between blocks, marked empty here
  double* phi;        // non-null: refresh the theta halos (first direction)
  int nr, nth, nz;
  int* err;
};

struct OldArgs {
  Dir d;
  LineGeo g;
  int tile;
  const double* phi;
  double* old;
};

struct SweepArgs {
  Dir d;
  LineGeo g;
  const double *rec, *old;
  double* mail;
  double* phi;
  int* err;
  uint64_t timeout_ns;
};

// Empty hand-over slot: a signalling NaN (IEEE arithmetic only delivers
// quiet NaNs, so no solution value has this high word).
constexpr int kEmptyHigh = 0x7ff00001;
__device__ __forceinline__ double empty_slot() { return __hiloint2double(kEmptyHigh, kEmptyHigh); }
__device__ __forceinline__ bool is_empty(double v) { return __double2hiint(v) == kEmptyHigh; }
// A caller's value as a slot may carry it: one with the mark's bits becomes the
// quiet NaN that any operation on it makes of it.
__device__ __forceinline__ double unmarked(double v) {
  return is_empty(v) ? __hiloint2double(kEmptyHigh | 0x00080000, __double2loint(v)) : v;
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
// Line records. A block builds the records of `tile` lines that are adjacent
// in the unit-stride index (r lines: adjacent rows) in shared memory: all
// threads gather the coefficients, neighbouring threads neighbouring
// addresses, then a warp per line computes its factors in place, and one bulk
// store writes each record. (A warp gathering its own line with strides of a
// row or a plane between lanes was bound by its 32 sectors a load: 1280 us at
// 120x240x168 against the bytes' 330.) The pivots' recurrence (:30-38)
//   m_i = guard(b_i - a_i cp_{i-1}),  cp_i = c_i / m_i
// runs in the lanes' segments from the previous pass's entering values until
// none changes (the first pass starts from zero: the recurrence forgets its
// start within a few elements). Padding elements and the line's ends carry
// values that leave the solver's recurrences untouched: cp = 0 in the last
// element, and m = y = 1 with zero links beyond. The first element's lo takes
// no part in the pivots: with it the solver adds the lagged coupling of the
// line's near end (see solve_lines).
// ---------------------------------------------------------------------------
constexpr int kTileBlock = 256;

// A block's lines: `tile` adjacent ones in the unit-stride line index u (r
// lines: in the chain's) at one value v of the other.
struct Tile {
  int u0, v, lines;
  __device__ Tile(const Dir& d, int tile) {
    const int U = d.b_fast ? d.B : d.A;
    const int tiles = (U + tile - 1) / tile;
    u0 = (int)(blockIdx.x % tiles) * tile;
    v = (int)(blockIdx.x / tiles);
    lines = min(tile, U - u0);
  }
  __device__ __forceinline__ int a_of(const Dir& d, int u) const { return d.b_fast ? v : u0 + u; }
  __device__ __forceinline__ int b_of(const Dir& d, int u) const { return d.b_fast ? u0 + u : v; }
  // Halo index of element 0 of the tile's line u.
  __device__ __forceinline__ long long cell(const Dir& d, int u) const {
    return d.base + a_of(d, u) * d.sa + b_of(d, u) * d.sb;
  }
  // Work item t of lines x E elements, neighbouring items at neighbouring
  // addresses.
  __device__ __forceinline__ void split(const Dir& d, int t, int E, int& u, int& e) const {
    u = d.se == 1 ? t / E : t % lines;
    e = d.se == 1 ? t % E : t / lines;
  }
};

__device__ __forceinline__ void bulk_copy_s2g(double* dst, const double* src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_addr(src)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Orders this thread's view of shared memory (generic proxy) before bulk copies
// (async proxy) that are issued behind it.
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_copies_done() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

template <int K>
__device__ __forceinline__ void factor_line(const Dir& d, const LineGeo& g, double* rec,
                                            int lane) {
  using Ln = Lanes<K>;
  double* r = rec + kRScalars + lane * Ln::kRec;
  const bool on = lane < g.n;
  double lo[K], bb[K], cc[K], mm[K], cp[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    lo[k] = on && lane + k > 0 ? r[kRLo * K + k] : 0.0;
    bb[k] = on ? r[kRM * K + k] : 1.0;
    cc[k] = on ? r[kRCp * K + k] : 0.0;
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
    if (lane == 0 || !on) nin = 0.0;
    if (__all_sync(kAllLanes, same_bits(nin, in))) break;
    in = nin;
  }
  double pf = on ? 1.0 : 0.0, pb = pf;
  bool safe = true;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const bool in_range = exp_in_safe_range(mm[k]);
    const double y = in_range ? 1.0 / mm[k] : 0.0;
    safe = safe && in_range;
    const double cpe = lane * K + k < d.L - 1 ? cp[k] : 0.0;
    if (on) {
      r[kRM * K + k] = mm[k];
      r[kRY * K + k] = y;
      r[kRCp * K + k] = cpe;
    }
    pf = pf * (-lo[k] * y);
    pb = pb * -cpe;
  }
  // Scan products: step s adds the value 2^s lanes away times the product
  // over the 2^s segments in between; a step whose products are all below
  // 2^-56 (and those after it) would change nothing and is left out.
  int nf = 0, nb = 0;
#pragma unroll
  for (int s = 0; s < kScanSteps; ++s) {
    if (on) {
      r[Ln::kScan + 2 * s] = pf;
      r[Ln::kScan + 2 * s + 1] = pb;
    }
    if (nf == s && __any_sync(kAllLanes, !(fabs(pf) < 0x1p-56))) nf = s + 1;
    if (nb == s && __any_sync(kAllLanes, !(fabs(pb) < 0x1p-56))) nb = s + 1;
    pf = pf * __shfl_up_sync(kAllLanes, pf, 1 << s);
    pb = pb * __shfl_down_sync(kAllLanes, pb, 1 << s);
  }
  safe = __all_sync(kAllLanes, safe);
  if (lane == 0) {
    rec[kRNf] = (double)(safe ? nf : nf + kUnsafe);
    rec[kRNb] = (double)nb;
  }
}

template <int K>
__global__ void __launch_bounds__(kTileBlock) tdma_factor_kernel(FactorArgs a) {
  using Ln = Lanes<K>;
  extern __shared__ __align__(128) double sm[];
  const Dir& d = a.d;
  const LineGeo& g = a.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (a.phi) theta_wrap(a.phi, a.nr, a.nth, a.nz);
  if (a.err && blockIdx.x == 0 && threadIdx.x == 0) *a.err = 0;
  const Tile tl(d, a.tile);
  const int E = g.n * K;  // elements with padding
  for (int t = threadIdx.x; t < tl.lines * E; t += kTileBlock) {
    int u, e;
    tl.split(d, t, E, u, e);
    double* rec = sm + (size_t)u * g.rec;
    double* r = rec + kRScalars + (e / K) * Ln::kRec + e % K;
    if (e < d.L) {
      const long long q = tl.cell(d, u) + e * d.se;
      const double lm = d.lm[q], lp = d.lp[q], ap = d.aP[q], s0 = d.Su[q], c1m = d.c1m[q],
                   c2m = d.c2m[q];
      r[kRSu * K] = s0;
      r[kR1m * K] = c1m;
      r[kR2m * K] = c2m;
      r[kRLo * K] = d.L > 1 ? -lm : 0.0;
      r[kRM * K] = ap;
      r[kRCp * K] = -lp;
      if (e == 0) rec[kRE0] = lm;
      if (e == d.L - 1) rec[kRE1] = lp;
    } else {
#pragma unroll
      for (int arr = 0; arr < kRArrays; ++arr) r[arr * K] = arr == kRM ? 1.0 : 0.0;
    }
  }
  fence_proxy_async();  // before the bulk stores
  __syncthreads();
  for (int u = warp; u < tl.lines; u += kTileBlock / 32) {
    double* rec = sm + (size_t)u * g.rec;
    const int ch = tl.a_of(d, u), b = tl.b_of(d, u);
    factor_line<K>(d, g, rec, lane);
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) bulk_copy_s2g(a.rec + ((long long)b * d.A + ch) * g.rec, rec, g.rec * 8);
    if (b % g.G == 0) {
      double* slot = a.mail + ((long long)(b / g.G) * d.A + ch) * Ln::kMail;
#pragma unroll
      for (int k = 0; k < K; ++k) slot[k * 32 + lane] = empty_slot();
    }
  }
  if (lane == 0) bulk_copies_done();
}

// Old-value records of one direction, in the factor kernel's tiles.
template <int K>
__global__ void __launch_bounds__(kTileBlock) tdma_old_kernel(OldArgs a) {
  using Ln = Lanes<K>;
  extern __shared__ __align__(128) double sm[];
  const Dir& d = a.d;
  const LineGeo& g = a.g;
  const Tile tl(d, a.tile);
  const int E = g.n * K;
  const double* __restrict__ phi = a.phi;
  for (int t = threadIdx.x; t < tl.lines * E; t += kTileBlock) {
    int u, e;
    tl.split(d, t, E, u, e);
    double* rec = sm + (size_t)u * g.old;
    double* r = rec + kOScalars + (e / K) * Ln::kOld + e % K;
    double o1 = 0.0, o2 = 0.0, end = -0.0;
    if (e < d.L) {
      const long long q = tl.cell(d, u) + e * d.se;
      o1 = d.c1p[q] * phi[q + d.s1];
      o2 = d.c2p[q] * phi[q + d.s2];
      if (e == 0) rec[0] = phi[q - d.se];
      if (e == d.L - 1) {
        const double far = phi[q + d.se];
        rec[1] = far;
        if (d.L > 1) end = d.lp[q] * far;
      }
    }
    r[kO1 * K] = o1;
    r[kO2 * K] = o2;
    r[kOEnd * K] = end;
  }
  fence_proxy_async();
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int u = 0; u < tl.lines; ++u)
      bulk_copy_s2g(a.old + ((long long)tl.b_of(d, u) * d.A + tl.a_of(d, u)) * g.old,
                    sm + (size_t)u * g.old, g.old * 8);
    bulk_copies_done();
  }
}

// ---------------------------------------------------------------------------
// Sweep of one direction.
// ---------------------------------------------------------------------------
// Shared memory by its 32-bit addresses: a solver's line is short of issue
// slots, and generic 64-bit addresses cost it a third more instructions.
using saddr = uint32_t;
__device__ __forceinline__ void ld_pair(saddr p, double& v, double& w) {
  asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v), "=d"(w) : "r"(p));
}
__device__ __forceinline__ void st_pair(saddr p, double v, double w) {
  asm volatile("st.volatile.shared.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(v), "d"(w) : "memory");
}
template <int N>
__device__ __forceinline__ void ld_pairs(saddr p, double (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) ld_pair(p + 8 * i, v[i], v[i + 1]);
}
template <int N>
__device__ __forceinline__ void st_pairs(saddr p, const double (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) st_pair(p + 8 * i, v[i], v[i + 1]);
}
// (mbar_test may suspend the warp; this looks and returns)
__device__ __forceinline__ bool mbar_look(saddr bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(saddr bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
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

// A lane's K values in a hand-over slot in shared memory.
template <int K>
__device__ __forceinline__ bool slot_full(saddr slot, double (&v)[K]) {
  ld_pairs(slot, v);
  bool all = true;
#pragma unroll
  for (int k = 0; k < K; ++k) all = all & !is_empty(v[k]);
  return all;
}
template <int K>
__device__ __forceinline__ bool slot_free(saddr slot) {
  double v[K];
  ld_pairs(slot, v);
  bool all = true;
#pragma unroll
  for (int k = 0; k < K; ++k) all = all & is_empty(v[k]);
  return all;
}

// Writes a solved line from its buffer to phi, and the theta halos that it
// completes: its own where the line is a theta column; where theta is the
// chain, at the chain's end, the owner's columns (their old halo values are
// no longer needed; the lane reads back values that it wrote).
template <int K>
__device__ __forceinline__ void write_line(const SweepArgs& a, const double* old, int b, int ch,
                                           int lane) {
  const Dir& d = a.d;
  if (lane >= a.g.n) return;
  double* p = a.phi + d.base + ch * d.sa + b * d.sb;
  double x[K];
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] = old[k];
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
struct LineAt {
  int b, ch = 0, st = 0;
  uint32_t phase = 0;
  __device__ LineAt(const LineGeo& g, int w) : b(blockIdx.x * g.G + w) {}
  __device__ __forceinline__ void next(const Dir& d, const LineGeo& g) {
    if (++st == g.NB) {
      st = 0;
      phase ^= 1u;
    }
    if (++ch == d.A) {
      ch = 0;
      b += gridDim.x * g.G;
    }
  }
};

// Copies the operands of the owner's lines into its ring of buffers, as far
// ahead as the solver has finished with them, and writes each finished line
// out of its buffer before that is filled again.
template <int K>
__device__ void load_lines(const SweepArgs& a, int w, double* bufs, uint64_t* full,
                           uint64_t* empty, int lane) {
  using Ln = Lanes<K>;
  const Dir& d = a.d;
  const LineGeo& g = a.g;
  LineAt at(g, w), done(g, w);
  int ahead = 0;  // lines issued and not yet written out
  Patience wait;
  while (done.b < d.B) {
    if (ahead < g.NB && at.b < d.B) {
      if (lane == 0) {
        const long long line = (long long)at.b * d.A + at.ch;
        double* buf = bufs + (size_t)at.st * g.buf;
        mbar_arrive_expect(&full[at.st], g.buf * 8);
        bulk_copy_g2s(buf, a.rec + line * g.rec, g.rec * 8, &full[at.st]);
        bulk_copy_g2s(buf + g.rec, a.old + line * g.old, g.old * 8, &full[at.st]);
      }
      at.next(d, g);
      ++ahead;
    } else if (__all_sync(kAllLanes, mbar_look(smem_addr(&empty[done.st]), done.phase))) {
      write_line<K>(a, bufs + (size_t)done.st * g.buf + g.rec + kOScalars + lane * Ln::kOld,
                    done.b, done.ch, lane);
      // The solver wrote its values, and the lanes here read them, by the generic
      // proxy; the copy that fills the buffer again writes by the async one, after
      // every lane's fence.
      fence_proxy_async();
      __syncwarp();
      done.next(d, g);
      --ahead;
      wait = Patience();
    } else {
      if (wait.gives_up(a.err, a.timeout_ns)) break;
      __nanosleep(100);  // leave the issue slots to the solver
    }
  }
  // After a wait gave up: no copy may still be in flight into this block's
  // memory when it leaves.
  for (; ahead > 0; --ahead) {
    for (int n = 0; n < (1 << 20) && !mbar_test(&full[done.st], done.phase); ++n) {
    }
    done.next(d, g);
  }
}

// Fetches the lines that the block's first owner needs -- the previous
// block's last owner's, or the halo -- into the first ring, as far ahead as
// it has room, so that the solver never waits for global memory itself.
template <int K>
__device__ void fetch_mail(const SweepArgs& a, double* ring, int lane) {
  using Ln = Lanes<K>;
  const Dir& d = a.d;
  const LineGeo& g = a.g;
  int sl = 0;
  for (int b = blockIdx.x * g.G; b < d.B; b += gridDim.x * g.G) {
    double* m = a.mail + (long long)(b / g.G) * d.A * Ln::kMail + lane;
    for (int ch = 0; ch < d.A; ++ch, m += Ln::kMail) {
      double v[K];
      if (b == 0) {
        const double* p = a.phi + d.base + ch * d.sa - (d.chain1 ? d.s2 : d.s1);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int e = lane * K + k;
          v[k] = e < d.L ? __ldcg(p + e * d.se) : 0.0;
        }
      } else {
        Patience wait;
        for (;;) {
          bool got = true;
#pragma unroll
          for (int k = 0; k < K; ++k) v[k] = ld_relaxed_f64(m + k * 32);
#pragma unroll
          for (int k = 0; k < K; ++k) got = got & !is_empty(v[k]);
          if (__all_sync(kAllLanes, got)) break;
          if (wait.gives_up(a.err, a.timeout_ns)) return;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) st_relaxed_f64(m + k * 32, empty_slot());
      }
      const saddr to = smem_addr(ring + (size_t)sl * g.ring + lane * Ln::kRing);
      sl = sl + 1 == g.slots ? 0 : sl + 1;
      Patience wait;
      while (!__all_sync(kAllLanes, slot_free<K>(to)))
        if (wait.gives_up(a.err, a.timeout_ns)) return;
      // (looked at here, not as they are loaded: a look waits for its load)
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = unmarked(v[k]);
      st_pairs(to, v);
    }
  }
}

// One lane's segment of the forward recurrence from the entering value, in
// the sequential operations (division by the stored reciprocal and one
// correction, which is the correctly rounded quotient: recipdiv.cuh). CHECKED,
// for the pass whose values are kept: a segment with an operand outside the
// correction's range, or a numerator of -0 (the correction would turn it into
// +0), is redone with `/`, and its padding elements, which an infinity would
// reach as 0 * Inf, are cleared. The empty asm keeps that division in a
// branch of its own (speculated, it doubled a pass).
template <int K, bool CHECKED>
__device__ __forceinline__ double forward_segment(const double (&dd)[K], const double (&lo)[K],
                                                  const double (&m)[K], const double (&y)[K],
                                                  bool y_ok, double in, double (&dp)[K],
                                                  int elements) {
  bool ok = y_ok;
  double p = in;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double t = dd[k] - lo[k] * p;
    const double q = t * y[k];
    p = __fma_rn(__fma_rn(-q, m[k], t), y[k], q);
    if (CHECKED) {
      const int hi = __double2hiint(t);
      const unsigned e = (unsigned)(hi & 0x7ff00000) - (523u << 20);
      ok = ok & ((e <= (1000u << 20)) | ((hi | __double2loint(t)) == 0));
    }
    dp[k] = p;
  }
  if (CHECKED && !ok) {
    asm volatile("" ::: "memory");
    p = in;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      p = (dd[k] - lo[k] * p) / m[k];
      dp[k] = k < elements ? p : 0.0;
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
// 2^-7 or more (at most three steps).
__device__ __forceinline__ int first_passes(int scan_steps) {
  return scan_steps <= 3 ? 2 : scan_steps - 1;
}

// A line's dependent operations take about 1000 cycles with K = 4 and the
// instructions around them cost one warp as much again, so everything that
// can be looked up early is: the next line's hand-over, the state of the slot
// it goes to and of its buffer are read between this line's two recurrences
// and settled by a vote beside the vote on the fixed point; only when they
// were not ready does the warp poll. All 32 lanes take part; those beyond the
// line read a neutral record (zeros, unit pivots), and their hand-over values
// are zeros.
//
// The lagged coupling of the line's near end, d_1 + a_1 phi_0 (:299-302,
// :325-328, :352-355), is the recurrence's own step from an entering value
// phi_0 (d - (-a) phi rounds as d + a phi); the far end's is added to the
// right-hand side last (-0.0 in the other elements: x + -0.0 is x).
template <int K, bool CHAIN1>
__device__ void solve_lines(const SweepArgs& a, int w, saddr bufs, saddr full, saddr empty,
                            saddr ring, saddr next_ring, saddr neutral, int lane) {
  using Ln = Lanes<K>;
  const Dir& d = a.d;
  const LineGeo& g = a.g;
  const long long sc = CHAIN1 ? d.s1 : d.s2;
  const bool on = lane < g.n;
  const bool first = lane == 0 || !on, last = lane >= g.n - 1;
  const bool near_end = lane == 0 && d.L > 1;
  const bool in_block = w + 1 < g.G;
  const int elements = d.L - lane * K;  // this lane's, if less than K
  const saddr buf_bytes = 8u * g.buf, bufs_end = bufs + g.NB * buf_bytes;
  const saddr slot_bytes = 8u * g.ring, slots_bytes = g.slots * slot_bytes;
  const saddr rec_at = 8u * (kRScalars + lane * Ln::kRec);
  const saddr old_at = 8u * (g.rec + kOScalars + lane * Ln::kOld);
  ring += 8u * lane * Ln::kRing;
  next_ring += 8u * lane * Ln::kRing;
  saddr buf = bufs, bar = 0, slot = 0;  // this line's buffer, barriers and slots
  uint32_t phase = 0;
  double x[K], t2[K];
  bool go = false;  // the hand-over, its target slot and the buffer are ready
  for (int b = blockIdx.x * g.G + w; b < d.B; b += gridDim.x * g.G) {
    const bool feeds = b + 1 < d.B;
    double* mail =
        a.mail + (long long)((b + 1) / g.G) * d.A * Ln::kMail + lane;  // of the next block
    {  // the chain starts from the halo
      const double* p = a.phi + d.base + b * d.sb - sc;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int e = lane * K + k;
        x[k] = e < d.L ? __ldcg(p + e * d.se) : 0.0;
      }
    }
    for (int ch = 0; ch < d.A; ++ch) {
      if (!go) {
        Patience wait;
        for (;;) {
          bool ready = slot_full<K>(ring + slot, t2);
          if (feeds && in_block) ready = ready & slot_free<K>(next_ring + slot);
          ready = ready & mbar_look(full + bar, phase);
          if (__all_sync(kAllLanes, ready)) break;
          if (wait.gives_up(a.err, a.timeout_ns)) return;
        }
      }
      const saddr r = on ? buf + rec_at : neutral;
      const saddr old = on ? buf + old_at : neutral + 8u * Ln::kRec;
      // Right-hand side, in the reference's order.
      double dd[K], lo[K], m[K], y[K], cp[K], scan[2 * kScanSteps], scalars[kRScalars], ends[2];
      {
        double su[K], c1m[K], c2m[K], ov[kOArrays * K];
        ld_pairs(r + 8 * kRSu * K, su);
        ld_pairs(r + 8 * kR1m * K, c1m);
        ld_pairs(old, ov);
        ld_pairs(r + 8 * kR2m * K, c2m);
        ld_pairs(r + 8 * kRLo * K, lo);
        ld_pairs(r + 8 * kRY * K, y);
        ld_pairs(buf, scalars);
        ld_pairs(buf + 8 * g.rec, ends);
        ld_pairs(r + 8 * Ln::kScan, scan);
        ld_pairs(r + 8 * kRM * K, m);
        ld_pairs(r + 8 * kRCp * K, cp);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const double n1 = CHAIN1 ? x[k] : t2[k], n2 = CHAIN1 ? t2[k] : x[k];
          double t = su[k] + c1m[k] * n1;
          t = t + ov[kO1 * K + k];
          t = t + c2m[k] * n2;
          t = t + ov[kO2 * K + k];
          dd[k] = t + ov[kOEnd * K + k];
        }
      }
      if (d.L == 1 && lane == 0)  // both ends in one element
        dd[0] = (dd[0] + scalars[kRE0] * ends[0]) + scalars[kRE1] * ends[1];
#pragma unroll
      for (int k = 0; k < K; k += 2) st_pair(ring + slot + 8 * k, empty_slot(), empty_slot());
      // Forward: entering values from the scan, then the passes.
      const int nfu = (int)scalars[kRNf], nf = nfu & (kUnsafe - 1), nb = (int)scalars[kRNb];
      const bool y_ok = nfu < kUnsafe;
      const double enter = near_end ? ends[0] : 0.0;
      double dp[K];
      double u = enter;
#pragma unroll
      for (int k = 0; k < K; ++k) u = __fma_rn(-lo[k] * y[k], u, dd[k] * y[k]);
      constexpr int kFew = 3;  // steps taken without a look at the count
#pragma unroll
      for (int s = 0; s < kFew; ++s)
        u = __fma_rn(scan[2 * s], __shfl_up_sync(kAllLanes, u, 1 << s), u);
      if (nf > kFew) {
#pragma unroll
        for (int s = kFew; s < kScanSteps; ++s)
          u = __fma_rn(scan[2 * s], __shfl_up_sync(kAllLanes, u, 1 << s), u);
      }
      auto enter_f = [first, enter](double out) {
        const double v = __shfl_up_sync(kAllLanes, out, 1);
        return first ? enter : v;
      };
      auto forward = [&](double in) {
        return enter_f(forward_segment<K, true>(dd, lo, m, y, y_ok, in, dp, elements));
      };
      double inf = enter_f(u);
      inf = enter_f(forward_segment<K, false>(dd, lo, m, y, y_ok, inf, dp, elements));
      for (int n = first_passes(nf); n > 2; --n)
        inf = enter_f(forward_segment<K, false>(dd, lo, m, y, y_ok, inf, dp, elements));
      double nin = forward(inf);
      bool settled = same_bits(nin, inf);
      inf = nin;
      // A first look at what the next line needs.
      const saddr this_to = next_ring + slot, this_old = old, this_empty = empty + bar;
      slot = slot + slot_bytes == slots_bytes ? 0 : slot + slot_bytes;
      buf += buf_bytes;
      bar += 8;
      if (buf == bufs_end) {
        buf = bufs;
        bar = 0;
        phase ^= 1u;
      }
      bool ready = slot_full<K>(ring + slot, t2);
      if (in_block) ready = ready & slot_free<K>(next_ring + slot);
      ready = ready & mbar_look(full + bar, phase);
      // Backward, likewise.
      u = 0.0;
#pragma unroll
      for (int k = K - 1; k >= 0; --k) u = __fma_rn(-cp[k], u, dp[k]);
#pragma unroll
      for (int s = 0; s < kFew; ++s)
        u = __fma_rn(scan[2 * s + 1], __shfl_down_sync(kAllLanes, u, 1 << s), u);
      if (nb > kFew) {
#pragma unroll
        for (int s = kFew; s < kScanSteps; ++s)
          u = __fma_rn(scan[2 * s + 1], __shfl_down_sync(kAllLanes, u, 1 << s), u);
      }
      auto enter_b = [last](double out) {
        const double v = __shfl_down_sync(kAllLanes, out, 1);
        return last ? 0.0 : v;
      };
      double inb = enter_b(u);
      inb = enter_b(backward_segment<K>(dp, cp, inb, x));
      for (int n = first_passes(nb); n > 2; --n)
        inb = enter_b(backward_segment<K>(dp, cp, inb, x));
      nin = enter_b(backward_segment<K>(dp, cp, inb, x));
      settled = settled & same_bits(nin, inb);
      inb = nin;
      go = __all_sync(kAllLanes, ready);
      if (!__all_sync(kAllLanes, settled)) {  // on to the fixed points, at most 32 passes away
        for (int n = 0; n <= 32; ++n) {
          nin = forward(inf);
          if (__all_sync(kAllLanes, same_bits(nin, inf))) break;
          inf = nin;
        }
        for (int n = 0; n <= 32; ++n) {
          nin = enter_b(backward_segment<K>(dp, cp, inb, x));
          if (__all_sync(kAllLanes, same_bits(nin, inb))) break;
          inb = nin;
        }
      }
      if (feeds && in_block) {
        st_pairs(this_to, x);
      } else if (feeds) {
#pragma unroll
        for (int k = 0; k < K; ++k) st_relaxed_f64(mail + k * 32, x[k]);
        mail += Ln::kMail;
      }
      if (on) st_pairs(this_old, x);
      __syncwarp();
      if (lane == 0) mbar_arrive(this_empty);
    }
  }
}

// Warps 0..G-1 solve, G..2G-1 load and write, 2G fetches the mail. A warp
// whose wait gave up leaves; the others' waits see the error word and leave
// too.
template <int K, bool CHAIN1>
__global__ void __launch_bounds__(Lanes<K>::kMaxThreads, 1) tdma_sweep_kernel(SweepArgs a) {
  using Ln = Lanes<K>;
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(8) uint64_t full[Ln::kMaxOwners][4], empty[Ln::kMaxOwners][4];
  const LineGeo& g = a.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* rings = sm + (size_t)g.G * g.NB * g.buf;
  const int ring = g.slots * g.ring;
  double* neutral = rings + g.G * ring;
  for (int i = threadIdx.x; i < g.G * ring; i += blockDim.x) rings[i] = empty_slot();
  for (int i = threadIdx.x; i < Ln::kRec + Ln::kOld; i += blockDim.x)
    neutral[i] = i >= kRM * K && i < (kRY + 1) * K ? 1.0 : 0.0;
  if (threadIdx.x == 0) {
    for (int o = 0; o < g.G; ++o)
      for (int n = 0; n < g.NB; ++n) {
        mbar_init(&full[o][n], 1);
        mbar_init(&empty[o][n], 1);
      }
    mbar_fence_init();
  }
  __syncthreads();
  if (warp < g.G) {
    solve_lines<K, CHAIN1>(a, warp, smem_addr(sm + (size_t)warp * g.NB * g.buf),
                           smem_addr(full[warp]), smem_addr(empty[warp]),
                           smem_addr(rings + (size_t)warp * ring),
                           smem_addr(rings + (size_t)(warp + 1) * ring), smem_addr(neutral), lane);
  } else if (warp < 2 * g.G) {
    const int w = warp - g.G;
    load_lines<K>(a, w, sm + (size_t)w * g.NB * g.buf, full[w], empty[w], lane);
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

// Bound by memory: every load of a cell (the identity-row test needs the
// coefficients, the residual also seven values of phi) is issued before the
// first decision, and 64 registers a thread leave room for two blocks of 512
// on an SM.
constexpr int kResBlock = 512;

__global__ void __launch_bounds__(kResBlock, 2) residual_kernel(ResArgs a) {
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
  const double* __restrict__ ph = a.phi;
  for (int c = own.begin + (int)threadIdx.x; c < own.end; c += kResBlock) {
    int i, j, k;
    cell_ijk(a.d, c, i, j, k);
    const long long q = (i + 2) + a.sx * (j + 2) + a.sxy * (k + 2);
    const double P = __ldg(in.aP + q), W = __ldg(in.aW + q), E = __ldg(in.aE + q),
                 S = __ldg(in.aS + q), N = __ldg(in.aN + q), B = __ldg(in.aB + q),
                 T = __ldg(in.aT + q), U = __ldg(in.Su + q);
    const double pc = ph[q], pw = ph[q - 1], pe = ph[q + 1], ps = ph[q - a.sx],
                 pn = ph[q + a.sx], pb = ph[q - a.sxy], pt = ph[q + a.sxy];
    const bool trivial = (P == 1.0) & (W == 0.0) & (E == 0.0) & (S == 0.0) & (N == 0.0) &
                         (B == 0.0) & (T == 0.0);
    double r = U - P * pc + S * ps + N * pn;
    r = r + W * pw + E * pe;
    r = r + B * pb + T * pt;
    const double t = fabs(U) + fabs(P * pc) + kSmall;
    v[0] = v[0] + (trivial ? 0.0 : r * r);
    v[1] = v[1] + (trivial ? 0.0 : t * t);
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

// Elements per lane of a line of L: four (see the file comment), beyond 128 the
// next instantiated size. A lane pays for K elements whether the line fills them
// or not, and the sizes between the powers of two save a part of that (two sweeps,
// ms, with / without them: z lines of 160 1.76 / 1.96, 300 2.75 / 3.19, 700 4.20 /
// 4.71). From 16 on the 255 registers do not hold a lane's arrays (K = 32 spills
// 3.7 KB), and still no length is slower than a lane a line was: 200 10.2 -> 2.1,
// 300 15.0 -> 2.75, theta lines of 512 7.1 -> 2.6, of 1024 13.9 -> 5.2.
int line_k(int L) {
  const int k = (L + 31) / 32;
  return k <= 4 ? 4 : k <= 6 ? 6 : k <= 8 ? 8 : k <= 12 ? 12 : k <= 16 ? 16 : k <= 24 ? 24 : 32;
}

template <class F>
auto with_k(int L, F f) {
  switch (line_k(L)) {
    case 4: return f(std::integral_constant<int, 4>());
    case 6: return f(std::integral_constant<int, 6>());
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
  size_t rec, old, mail;  // doubles
  int blocks, threads;
};

DirSizes dir_sizes(const Dir& d) {
  return with_k(d.L, [&d](auto k) {
    constexpr int K = decltype(k)::value;
    const LineGeo g = line_geo<K>(d.L);
    const int blocks = (d.B + g.G - 1) / g.G;
    return DirSizes{(size_t)d.A * d.B * g.rec, (size_t)d.A * d.B * g.old, (size_t)blocks * d.A * Lanes<K>::kMail, blocks,
                    32 * (2 * g.G + 1)};
  });
}

cudaError_t allow_smem(const void* kernel, size_t bytes) {
  return bytes <= 48 * 1024
             ? cudaSuccess
             : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)bytes);
}

// Launches a kernel over tiles of lines whose records of `rec` doubles are
// built in shared memory: eight lines a block (64-byte rows, a warp a line),
// fewer where three blocks' records would not fit an SM.
template <class Args>
cudaError_t launch_tiles(void (*kernel)(Args), Args a, int rec, cudaStream_t st) {
  const size_t bytes = (size_t)rec * sizeof(double);
  a.tile = 8;
  while (a.tile > 1 && a.tile * bytes > 75 * 1024) a.tile /= 2;
  const int U = a.d.b_fast ? a.d.B : a.d.A, V = a.d.b_fast ? a.d.A : a.d.B;
  const long long grid = (long long)((U + a.tile - 1) / a.tile) * V;
  const cudaError_t e = allow_smem((const void*)kernel, a.tile * bytes);
  if (e != cudaSuccess) return e;
  kernel<<<(unsigned)grid, kTileBlock, a.tile * bytes, st>>>(a);
  return cudaGetLastError();
}

template <int K, bool CHAIN1>
cudaError_t launch_sweep(SweepArgs a, int sms, cudaStream_t st) {
  const void* k = (const void*)tdma_sweep_kernel<K, CHAIN1>;
  const cudaError_t e = allow_smem(k, a.g.smem);
  if (e != cudaSuccess) return e;
  // At most one block per SM; further owners follow in rounds.
  const int blocks = (a.d.B + a.g.G - 1) / a.g.G;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(k, dim3(blocks < sms ? blocks : sms),
                                     dim3(32 * (2 * a.g.G + 1)), args, a.g.smem, st);
}

}  // namespace

TdmaSizes tdma_sizes(int nr, int nth, int nz) {
  TdmaSizes z = {};
  auto rounded = [](size_t n) { return (n + 31) / 32 * 32; };
  for (int dir = 0; dir < 3; ++dir) {
    const DirSizes s = dir_sizes(make_dir(HaloInputs{}, nr, nth, nz, dir));
    z.rec[dir] = rounded(s.rec);
    if (s.mail > z.mail) z.mail = rounded(s.mail);
    if (s.old > z.old) z.old = rounded(s.old);
  }
  return z;
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
                            int n_sweep, const TdmaScratch& w, int sms, const GroupWs& ws,
                            uint64_t timeout_ns, cudaStream_t st) {
  if (nr > kTdmaMaxLine || nth > kTdmaMaxLine || nz > kTdmaMaxLine)
    return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> attr_lock(launch_attr_mutex());
  (void)cudaGetLastError();  // report these launches' errors, not an older one
  // A direction's records; the call's first launch also refreshes phi's theta
  // halos and clears the error word.
  auto build = [&](int dir, bool first) {
    FactorArgs f;
    f.d = make_dir(in, nr, nth, nz, dir);
    f.rec = w.rec[dir];
    f.mail = w.mail;
    f.phi = first ? phi : nullptr;
    f.err = first ? ws.err : nullptr;
    f.nr = nr;
    f.nth = nth;
    f.nz = nz;
    return with_k(f.d.L, [&](auto k) {
      constexpr int K = decltype(k)::value;
      f.g = line_geo<K>(f.d.L);
      return launch_tiles(tdma_factor_kernel<K>, f, f.g.rec, st);
    });
  };
  for (int dir = 0; dir < 3 && !w.rebuild; ++dir) {
    const cudaError_t e = build(dir, dir == 0);
    if (e != cudaSuccess) return e;
  }
  for (int sweep = 1; sweep <= n_sweep; ++sweep) {
    for (int dir = 0; dir < 3; ++dir) {
      if (w.rebuild) {
        const cudaError_t e = build(dir, sweep == 1 && dir == 0);
        if (e != cudaSuccess) return e;
      }
      OldArgs o;
      o.d = make_dir(in, nr, nth, nz, dir);
      o.phi = phi;
      o.old = w.old;
      SweepArgs a;
      a.d = o.d;
      if (dir == 2 && sweep == n_sweep) a.d.wrap = 0;  // no refresh after the last direction
      a.rec = w.rec[dir];
      a.old = w.old;
      a.mail = w.mail;
      a.phi = phi;
      a.err = ws.err;
      a.timeout_ns = timeout_ns;
      const cudaError_t e = with_k(a.d.L, [&](auto k) {
        constexpr int K = decltype(k)::value;
        o.g = a.g = line_geo<K>(a.d.L);
        const cudaError_t e2 = launch_tiles(tdma_old_kernel<K>, o, o.g.old, st);
        if (e2 != cudaSuccess) return e2;
        return a.d.chain1 ? launch_sweep<K, true>(a, sms, st) : launch_sweep<K, false>(a, sms, st);
      });
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

// A cell a thread up to two blocks per SM (more cells in turn beyond).
void residual_launch_shape(long long n, int sms, int* grid, int* block) {
  const long long g = (n + kResBlock - 1) / kResBlock;
  *grid = (int)(g < 2 * sms ? g : 2 * sms);
  *block = kResBlock;
}

cudaError_t launch_residual_f64(const HaloInputs& in, const double* phi, const MeshDims& d,
                                const GroupWs& ws, uint64_t timeout_ns, int grid,
                                cudaStream_t st) {
  ResArgs a;
  a.in = in;
  a.phi = phi;
  a.d = d;
  a.sx = d.nr + 4;
  a.sxy = (long long)(d.nr + 4) * (d.nth + 4);
  a.ws = ws;
  a.timeout_ns = timeout_ns;
  const cudaError_t e = launch_group_init(ws, st);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel((const void*)residual_kernel, dim3(grid), dim3(kResBlock),
                                     args, 0, st);
}


cudaError_t run_div_check(long long n, unsigned long long seed, unsigned long long* counts,
                          cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  div_check_kernel<<<592, 256, 0, st>>>(n, seed, counts);
  return cudaGetLastError();
}

}  // namespace eaf
