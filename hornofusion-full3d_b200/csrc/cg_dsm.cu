// Cluster-resident FP64 CG for small systems: ONE thread-block cluster of C
// blocks (up to 16) holds the whole system in distributed shared memory for
// the whole solve, so an iteration touches global memory not at all.
//
// The solver is cg_3d_mpi (src/mod_solver_3d.f90:485-620) exactly as the
// persistent kernels of cg_f64.cu run it -- same slices (block b owns compact
// cells [b*ceil(n/C), ...)), same thread-to-cell assignment, same per-cell
// arithmetic in the reference's expression order (built with -fmad=false),
// same exit tests and NaN outcome -- with two differences in where data
// lives:
//   * each block keeps its slice of the seven coefficients (the symmetric
//     form's west, south and bottom links copied from the neighbours' east,
//     north and top links once, at load), of x, r, z, q and of the
//     double-buffered direction in its shared memory; a neighbour cell that
//     another block owns is read from that block's shared memory
//     (ld.shared::cluster);
//   * an all-reduce is one exchange: every block writes its partial into
//     every block's shared memory and signals it, and then every thread
//     folds the C partials in rank order. The association is that of the
//     cluster all-reduce with one cluster (the oracle's plan (C, B, C)), so
//     the solve is bit-identical to cg_cluster_kernel on the same launch
//     shape and to the oracle. The signal is either a full cluster barrier
//     (3.4 us per iteration at 12x24x16) or a remote arrival on an mbarrier of
//     each block (release at cluster scope, one arrival per block and phase,
//     barriers double-buffered by all-reduce parity; 3.9 us).
// Where a thread's cells fit its registers, the default is the pushed form
// (cg_push_kernel, below): 1.8 us.
//
// Global memory is read once (the packed system) and written once (x and
// the result). There is no global synchronisation and no wait that another
// block could leave unfinished: every block of a cluster is co-scheduled
// and reaches every cluster barrier on every path (the exit decisions depend
// only on the totals, which all blocks fold identically).
#include <math.h>
#include <stddef.h>

#include "cg_kernels.h"
#include "cluster_red.cuh"
#include "recipdiv.cuh"
#include "stencil.cuh"

namespace eaf {
namespace {

// Shared-memory arrays of a slice, in this order:
//   coefficients aP aW aE aS aN aB aT, then x r z p0 p1 q, then the six
//   neighbour addresses of every cell (32-bit shared-window addresses of the
//   neighbour's element of array 0 in its owner block, or kNoNeighbour at an
//   r or z wall), which occupy the room of three more arrays.
constexpr int kDsmArrays = 16;
enum { kAP, kAW, kAE, kAS, kAN, kAB, kAT, kX, kR, kZ, kP0, kP1, kQ, kNB };
enum { kW, kE, kS, kN, kB, kT };  // neighbour directions, stencil order
constexpr uint32_t kNoNeighbour = 0xFFFFFFFFu;

struct DsmArgs {
  MeshDims d;
  SysF64 s;      // the packed compact system (read) and x (written back)
  GroupWs ws;    // result and error word
  int max_iter;
  double tol;
  uint64_t timeout_ns;
  int chunk;     // cells per block
  int reach;     // blocks on either side that hold neighbours (pushed form)
  FastDiv fd_chunk;
};

struct PartSmem {
  double part[2][kMaxClusterSize][kClusterSlotsNV];  // by parity, by rank
  double warp[kClusterSlotsNV][32];
  uint64_t bar[2];  // arrivals of the C blocks' partials, by parity
};

// Signalling of the exchange: mbarrier arrivals (MB) or a cluster barrier.
struct Exchange {
  int C, rank, parity;
  uint32_t phase;  // completion parity expected next, bit per barrier
  int* err;
  uint64_t timeout_ns;
};

__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                   cluster_addr)
               : "memory");
}
__device__ __forceinline__ bool mbar_test_cluster(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ double ld_cluster_f64(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

struct Dsm {
  double* base;      // this block's arrays
  uint32_t base_sa;  // its shared-window address
  int chunk, rank;
  FastDiv fd;
  __device__ __forceinline__ double* arr(int k) const { return base + (size_t)k * chunk; }
  __device__ __forceinline__ uint32_t* nb(int dir) const {
    return reinterpret_cast<uint32_t*>(base + (size_t)kNB * chunk) + (size_t)dir * chunk;
  }
  // Address (in the cluster's shared window) of array 0 at compact cell cc.
  __device__ __forceinline__ uint32_t where(int cc) const {
    const int owner = (int)fd.div((uint32_t)cc);
    const int off = cc - owner * chunk;
    return cluster_map(base_sa + 8u * (uint32_t)off, (uint32_t)owner);
  }
  // Value of array k at the neighbour whose array-0 address is a.
  __device__ __forceinline__ double at(int k, uint32_t a) const {
    return ld_cluster_f64(a + 8u * (uint32_t)k * (uint32_t)chunk);
  }
};

// Every block's partials go to every block, then each thread folds them in
// rank order (starting from rank 0's). Returns false if a bounded wait gave
// up (then every thread of the block returns false).
template <int NV, bool MB>
__device__ __forceinline__ bool dsm_allsum(double (&v)[NV], PartSmem& ps, Exchange& x) {
  const int C = x.C, rank = x.rank, parity = x.parity;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nthreads = blockDim.x;
#pragma unroll
  for (int m = 0; m < NV; ++m) v[m] = warp_allsum(v[m]);
  if (w != 0) {
    if (lane == 0) {
#pragma unroll
      for (int m = 0; m < NV; ++m) ps.warp[m][w] = v[m];
    }
    named_arrive(kBarPosted, nthreads);
  } else {
    if (lane == 0) {
#pragma unroll
      for (int m = 0; m < NV; ++m) ps.warp[m][0] = v[m];
    }
    named_sync(kBarPosted, nthreads);
    const int nw = (nthreads + 31) >> 5;
    double blk[NV];
#pragma unroll
    for (int m = 0; m < NV; ++m) blk[m] = warp_allsum(lane < nw ? ps.warp[m][lane] : 0.0);
    if (lane < C) {
      const uint32_t dst = cluster_map(smem_addr(&ps.part[parity][rank][0]), (uint32_t)lane);
#pragma unroll
      for (int m = 0; m < NV; ++m) st_cluster_f64(dst + 8u * m, blk[m]);
      if (MB) mbar_arrive_remote(cluster_map(smem_addr(&ps.bar[parity]), (uint32_t)lane));
    }
    __syncwarp();
  }
  bool ok = true;
  if (MB) {
    // Every thread acquires the C arrivals itself (bounded wait).
    const uint32_t a = smem_addr(&ps.bar[parity]);
    const uint32_t want = (x.phase >> parity) & 1u;
    if (!mbar_test_cluster(a, want)) {
      const uint64_t t0 = global_ns();
      uint32_t spins = 0;
      while (!mbar_test_cluster(a, want)) {
        if ((++spins & 255u) == 0) {
          if (ld_volatile_i32(x.err) != 0) { ok = false; break; }
          if (global_ns() - t0 > x.timeout_ns) {
            atomicCAS(x.err, 0, (int)EAF_ETIMEOUT);
            ok = false;
            break;
          }
        }
      }
    }
    x.phase ^= 1u << parity;
    ok = __syncthreads_and(ok) != 0;
  } else {
    cluster_sync_all();
  }
  x.parity ^= 1;
#pragma unroll
  for (int m = 0; m < NV; ++m) {
    double t = ps.part[parity][0][m];
    for (int r = 1; r < C; ++r) t = t + ps.part[parity][r][m];
    v[m] = t;
  }
  return ok;
}

// y = A x at own cell o, the reference's expression order; the coefficients
// are this block's copies, neighbour values come from xv(neighbour address)
// (a missing neighbour -- r or z wall -- is skipped in the symmetric form and
// multiplies a zero value in the general form, as in apply_row_with).
template <bool SYM, typename XF>
__device__ __forceinline__ double dsm_row(const Dsm& m, int o, double xc, XF xv) {
  const uint32_t w = m.nb(kW)[o], e = m.nb(kE)[o], so = m.nb(kS)[o];
  const uint32_t no = m.nb(kN)[o], bo = m.nb(kB)[o], t = m.nb(kT)[o];
  double y = m.arr(kAP)[o] * xc;
  if (SYM) {
    if (w != kNoNeighbour) y = y - m.arr(kAW)[o] * xv(w);
    if (e != kNoNeighbour) y = y - m.arr(kAE)[o] * xv(e);
    y = y - m.arr(kAS)[o] * xv(so);
    y = y - m.arr(kAN)[o] * xv(no);
    if (bo != kNoNeighbour) y = y - m.arr(kAB)[o] * xv(bo);
    if (t != kNoNeighbour) y = y - m.arr(kAT)[o] * xv(t);
  } else {
    const double xw = w != kNoNeighbour ? xv(w) : 0.0;
    const double xe = e != kNoNeighbour ? xv(e) : 0.0;
    const double xb = bo != kNoNeighbour ? xv(bo) : 0.0;
    const double xt = t != kNoNeighbour ? xv(t) : 0.0;
    y = y - m.arr(kAW)[o] * xw;
    y = y - m.arr(kAE)[o] * xe;
    y = y - m.arr(kAS)[o] * xv(so);
    y = y - m.arr(kAN)[o] * xv(no);
    y = y - m.arr(kAB)[o] * xb;
    y = y - m.arr(kAT)[o] * xt;
  }
  return y;
}

template <bool SYM, bool MB>
__device__ void dsm_body(const DsmArgs& a, const Dsm& m, PartSmem& ps, int C) {
  const MeshDims& d = a.d;
  const SysF64& s = a.s;
  const int rank = m.rank;
  Exchange xc;
  xc.C = C;
  xc.rank = rank;
  xc.parity = 0;
  xc.phase = 0;
  xc.err = a.ws.err;
  xc.timeout_ns = a.timeout_ns;
  const int begin = min(d.n, rank * a.chunk);
  const int end = min(d.n, begin + a.chunk);
  const int B = blockDim.x;

  // Load the slice; the symmetric form's west/south/bottom links are the
  // neighbours' east/north/top links (zero at the r and z walls, where the
  // solver skips them).
  for (int c = begin + (int)threadIdx.x; c < end; c += B) {
    const int o = c - begin;
    int i, j, k;
    cell_ijk(d, c, i, j, k);
    const int cs = j > 0 ? c - d.nr : c + (d.nth - 1) * d.nr;
    m.arr(kAP)[o] = s.aP[c];
    m.arr(kAE)[o] = s.aE[c];
    m.arr(kAN)[o] = s.aN[c];
    m.arr(kAT)[o] = s.aT[c];
    if (SYM) {
      m.arr(kAW)[o] = i > 0 ? s.aE[c - 1] : 0.0;
      m.arr(kAS)[o] = s.aN[cs];
      m.arr(kAB)[o] = k > 0 ? s.aT[c - d.plane] : 0.0;
    } else {
      m.arr(kAW)[o] = s.aW[c];
      m.arr(kAS)[o] = s.aS[c];
      m.arr(kAB)[o] = s.aB[c];
    }
    m.arr(kX)[o] = s.x[c];
    const int cn = j < d.nth - 1 ? c + d.nr : c - (d.nth - 1) * d.nr;
    m.nb(kW)[o] = i > 0 ? m.where(c - 1) : kNoNeighbour;
    m.nb(kE)[o] = i < d.nr - 1 ? m.where(c + 1) : kNoNeighbour;
    m.nb(kS)[o] = m.where(cs);
    m.nb(kN)[o] = m.where(cn);
    m.nb(kB)[o] = k > 0 ? m.where(c - d.plane) : kNoNeighbour;
    m.nb(kT)[o] = k < d.nz - 1 ? m.where(c + d.plane) : kNoNeighbour;
  }
  // Preamble (src/mod_solver_3d.f90:515-530): ||Su||, z = r/max(|aP|,SMALL),
  // p = z, r.z and r.r.
  double v3[3] = {0.0, 0.0, 0.0};
  for (int c = begin + (int)threadIdx.x; c < end; c += B) {
    const int o = c - begin;
    const double bv = s.b[c], rv = s.r[c];
    const double zv = rv / guard_small(fabs(s.aP[c]));
    m.arr(kR)[o] = rv;
    m.arr(kZ)[o] = zv;
    m.arr(kP0)[o] = zv;
    v3[0] = v3[0] + bv * bv;
    v3[1] = v3[1] + rv * rv;
    v3[2] = v3[2] + rv * zv;
  }
  bool ok = dsm_allsum<3, MB>(v3, ps, xc);
  const double bnorm = sqrt(v3[0]);
  double residual = 0.0;
  int n_iter = 0;
  bool nan_fill = false;
  if (ok && !(bnorm < kSmall)) {
    double rz = v3[2];
    double beta = 0.0;
    residual = sqrt(v3[1]) / bnorm;
    if (residual != residual && a.max_iter >= 1) nan_fill = true;
    for (int iter = 1; iter <= a.max_iter && !nan_fill; ++iter) {
      // Phase A: p = z + beta p_old fused with q = A p and p.q.
      const int kcur = (iter & 1) ? kP0 : kP1;
      const int kold = (iter & 1) ? kP1 : kP0;
      double* pcur = m.arr(kcur);
      double* q = m.arr(kQ);
      double v1[1] = {0.0};
      if (iter == 1) {
        auto xv = [&m, kcur](uint32_t na) { return m.at(kcur, na); };
        for (int c = begin + (int)threadIdx.x; c < end; c += B) {
          const int o = c - begin;
          const double pc = pcur[o];
          const double qv = dsm_row<SYM>(m, o, pc, xv);
          q[o] = qv;
          v1[0] = v1[0] + pc * qv;
        }
      } else {
        const double bt = beta;
        auto pnew = [&m, kold, bt](uint32_t na) { return m.at(kZ, na) + bt * m.at(kold, na); };
        const double* z = m.arr(kZ);
        const double* pold = m.arr(kold);
        for (int c = begin + (int)threadIdx.x; c < end; c += B) {
          const int o = c - begin;
          const double pc = z[o] + bt * pold[o];
          const double qv = dsm_row<SYM>(m, o, pc, pnew);
          pcur[o] = pc;
          q[o] = qv;
          v1[0] = v1[0] + pc * qv;
        }
      }
      if (!(ok = dsm_allsum<1, MB>(v1, ps, xc))) break;
      const double pq = v1[0];
      if (fabs(pq) < kSmall) break;
      const double alpha = rz / pq;
      // Phase B: phi += alpha p; r -= alpha q; r.r; z and r.z (:538-553)
      double v2[2] = {0.0, 0.0};
      {
        double* x = m.arr(kX);
        double* r = m.arr(kR);
        double* z = m.arr(kZ);
        const double* aP = m.arr(kAP);
        for (int c = begin + (int)threadIdx.x; c < end; c += B) {
          const int o = c - begin;
          const double xn = x[o] + alpha * pcur[o];
          const double rn = r[o] - alpha * q[o];
          const double zv = rn / guard_small(fabs(aP[o]));
          x[o] = xn;
          r[o] = rn;
          z[o] = zv;
          v2[0] = v2[0] + rn * rn;
          v2[1] = v2[1] + rn * zv;
        }
      }
      if (!(ok = dsm_allsum<2, MB>(v2, ps, xc))) break;
      residual = sqrt(v2[0]) / bnorm;
      n_iter = iter;
      if (residual < a.tol) break;
      if (residual != residual && iter < a.max_iter) { nan_fill = true; break; }
      beta = v2[1] / guard_small(rz);
      rz = v2[1];
    }
  }
  // x back to global memory for the unpack kernel.
  const double qnan = __longlong_as_double(0x7ff8000000000000ll);
  for (int c = begin + (int)threadIdx.x; c < end; c += B)
    s.x[c] = nan_fill ? qnan : m.arr(kX)[c - begin];
  if (nan_fill) {
    residual = qnan;
    n_iter = a.max_iter;
  }
  if (rank == 0 && threadIdx.x == 0) {
    SolveResult* res = a.ws.result;
    const int err = ld_volatile_i32(a.ws.err);
    res->status = err != 0 ? err : (isfinite(residual) ? EAF_OK : EAF_ENONFINITE);
    res->n_iter = n_iter;
    res->n_outer = 0;
    res->sym = SYM ? 1 : 0;
    res->residual = residual;
    res->bnorm = bnorm;
  }
}

template <bool MB>
__global__ void __launch_bounds__(1024, 1) cg_dsm_kernel(DsmArgs a) {
  extern __shared__ __align__(16) double dsm_smem[];
  __shared__ __align__(8) PartSmem ps;
  Dsm m;
  m.base = dsm_smem;
  m.base_sa = smem_addr(dsm_smem);
  m.chunk = a.chunk;
  m.rank = (int)cluster_ctarank();
  m.fd = a.fd_chunk;
  const int C = (int)cluster_nctarank();
  if (MB && threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ps.bar[0])), "r"(C)
                 : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ps.bar[1])), "r"(C)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Every block has started (and initialised its barriers) before any
  // block addresses another's memory.
  cluster_sync_all();
  if (*a.s.asym == 0)
    dsm_body<true, MB>(a, m, ps, C);
  else
    dsm_body<false, MB>(a, m, ps, C);
  // No block leaves while another may still address its shared memory.
  cluster_sync_all();
}

// ---------------------------------------------------------------------------
// Pushed form: a thread holds its one or two cells in registers for the whole
// solve -- coefficients, x, r, z, q, its direction and, instead of re-reading
// z and the old direction of the six neighbours, their directions, which it
// advances itself (p_nb = z_nb + beta p_nb, the owner's own operation). What an
// iteration exchanges is the new z and the blocks' partials, and both are
// PUSHED, completing bytes on an mbarrier of the receiving block: the partials
// by st.async, a block's slice of z by one bulk copy to each block within a
// z-plane of it (every neighbour of a cell is less than a plane away). A block
// keeps the slices it receives beside its own, so all its reads are local.
// Measured on 16 blocks of 288 threads, cycles: remote stores and a releasing
// cluster barrier 1035, pushed exchange 370; six remote loads a thread 930.
// (z by one st.async per cell and remote neighbour was no faster than the
// bulk copies and needs the addresses in registers.) us per iteration, cluster
// barrier -> pushed: 10x20x12 2.9 -> 1.6, 12x24x16 3.4 -> 1.8, 18x36x24
// 4.5 -> 2.8. What is left is latency: two reductions of two butterflies each,
// two exchanges and one division chain an iteration.
//
// Order. Two exchanges an iteration, each on its own barrier: p.q after the
// stencil phase, (r.r, r.z) and z after the update phase. A block's partial
// and its copies follow a block barrier behind everything its threads read
// and wrote, so: received slices and partial slots are overwritten, and the
// own z behind an earlier copy rewritten, only after every block has this
// block's next partial; a barrier's next phase cannot receive bytes before
// this one was waited for by every thread here (a block two exchanges ahead
// would need this block's partial between). The arithmetic and the
// association are dsm_body's.
// ---------------------------------------------------------------------------
struct PushSmem {
  // Block partials by rank, as many doubles each as the sums they carry
  // (preamble: three and a pad).
  double pq[kMaxClusterSize], rz[kMaxClusterSize][2], pre[kMaxClusterSize][4];
  double warp[kClusterSlotsNV][32];
  double zero;       // z of a missing neighbour
  double dummy;      // where cells beyond the slice leave theirs
  uint64_t bar[2];
  int gave_up;       // a block of the cluster left an exchange unfinished
};
static_assert(offsetof(PushSmem, rz) == 8 * kMaxClusterSize &&
                  offsetof(PushSmem, pre) == 24 * kMaxClusterSize &&
                  offsetof(PushSmem, warp) == 56 * kMaxClusterSize,
              "the offsets that push_allsum uses");

// What a block's all-reduces need, set up once (shared-memory addresses).
struct Pusher {
  int rank;
  uint32_t phases;             // completion parity expected next, bit per barrier
  uint32_t smem, bar;          // this block's PushSmem and barriers
  uint32_t to_smem, to_bar;    // those of lane's target block (lane & 15)
  uint32_t z_bytes;            // bytes of z a block receives per exchange
  uint32_t z_src, z_dst, z_len, z_bar;  // last warp: lane's copy of z
  int* err;
  uint64_t timeout_ns;
};

__device__ __forceinline__ void st_async_f64(uint32_t dst, double v, uint32_t bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
      "l"(__double_as_longlong(v)), "r"(bar)
      : "memory");
}
// (the writers of the source have passed a proxy fence and a block barrier)
__device__ __forceinline__ void push_bulk(uint32_t dst, uint32_t src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, "
      "[%3];" ::"r"(dst),
      "r"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// The slices of z in a block's shared memory: slot s holds that of block
// rank - reach + s; a slot is `pad` doubles (the slice, to 16 bytes).
struct Slices {
  int reach, pad;
  uint32_t base;
  __device__ __forceinline__ uint32_t slot(int rank, int owner) const {
    return base + 8u * (uint32_t)((owner - rank + reach) * pad);
  }
  __device__ __forceinline__ uint32_t bytes(const DsmArgs& a, int owner) const {
    const int cells = max(0, min(a.chunk, a.d.n - owner * a.chunk));
    return 8u * (uint32_t)((cells + 1) & ~1);
  }
};
__device__ __forceinline__ Pusher make_pusher(const DsmArgs& a, const Slices& zs, PushSmem& ps,
                                              int C, int rank) {
  Pusher px;
  const int lane = threadIdx.x & 31, to = rank - zs.reach + lane;
  px.rank = rank;
  px.phases = 0;
  px.smem = smem_addr(&ps);
  px.bar = smem_addr(&ps.bar[0]);
  px.to_smem = cluster_map(px.smem, (uint32_t)min(lane & 15, C - 1));
  px.to_bar = cluster_map(px.bar, (uint32_t)min(lane & 15, C - 1));
  px.z_bytes = 0;
  for (int b = max(0, rank - zs.reach); b <= min(C - 1, rank + zs.reach); ++b)
    if (b != rank) px.z_bytes += zs.bytes(a, b);
  const bool sends = lane <= 2 * zs.reach && to >= 0 && to < C && to != rank;
  px.z_len = sends ? zs.bytes(a, rank) : 0u;
  px.z_src = zs.slot(rank, rank);
  px.z_dst = sends ? cluster_map(zs.slot(to, rank), (uint32_t)to) : 0u;
  px.z_bar = sends ? cluster_map(px.bar + 8u, (uint32_t)to) : 0u;
  px.err = a.ws.err;
  px.timeout_ns = a.timeout_ns;
  return px;
}
__device__ __forceinline__ double ld_shared_f64(uint32_t a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

// Sums of the warp's NV values, by the xor butterfly (steps 16, 8, 4, 2, 1);
// HALF: only lanes 0..15 hold values, the others zeros, and step 16, which
// would add them, is left out (x + 0 is x for every sum but -0, and no sum
// here is -0 where it matters). Two values share the steps after the first:
// each half of the warp goes on with one of them. Value m is valid in lane
// 16 m (one value: every lane).
template <int NV, bool HALF>
__device__ __forceinline__ double warp_sums(const double (&v)[NV], int lane) {
  static_assert(NV <= 2, "one value per half");
  const unsigned all = 0xffffffffu;
  double t;
  if (NV == 1) {
    t = v[0];
    if (!HALF) t = t + __shfl_xor_sync(all, t, 16);
  } else {
    const bool up = lane >= 16;
    const double got = __shfl_xor_sync(all, up ? v[0] : v[NV - 1], 16);
    const double mine = up ? v[NV - 1] : v[0];
    t = HALF ? (up ? got : mine) : mine + got;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t = t + __shfl_xor_sync(all, t, o);
  return t;
}

// Opens the next phase of a barrier: it completes with `bytes` pushed.
__device__ __forceinline__ void push_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void ld_shared_pair(uint32_t a, double& v, double& w) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v), "=d"(w) : "r"(a) : "memory");
}
__device__ __forceinline__ void st_shared_f64(uint32_t a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

constexpr uint64_t kPushDrainNs = 1000000;  // bound of the wait for copies in flight

// Offsets in a PushSmem, and the doubles a block's sums take there.
constexpr uint32_t kAtPq = 0, kAtRz = 8 * kMaxClusterSize, kAtPre = 24 * kMaxClusterSize,
                   kAtWarp = 56 * kMaxClusterSize;

// All-reduce of NV sums over the cluster: warp sums, block sums (warp 0)
// pushed to every block, with KIND 1 also z (the last warp); then every thread
// waits for the partials of the (at most) CMAX blocks, whose slots beyond the
// cluster's size hold zeros, and folds them in rank order. Two values are
// pushed by the two halves of warp 0. The barrier's next phase, which will
// carry `next` bytes, is opened by a thread that has seen this one complete (the
// others still find it so: nothing pushes into the next before this block's
// threads have met). False if the wait gave up; that thread then leaves the open
// phase alone, which an arrival more would corrupt. A block leaves as one: before
// the fold (EARLY) or behind it, whichever the registers bear better (50
// iterations: two cells a thread, 18x36x24, 157.6 us before, 159.8 behind; one cell,
// 10x20x12, 92.2 before, 90.1 behind).
template <int NV, int KIND, int CMAX, bool EARLY = false>
__device__ __forceinline__ bool push_allsum(double (&v)[NV], int C, uint32_t next, Pusher& x) {
  constexpr int kPairs = (NV + 1) / 2;  // values go two by two
  constexpr int kTwo = NV >= 2 ? 2 : 1;
  constexpr uint32_t kStride = 8 * (NV <= 2 ? NV : 4);
  constexpr uint32_t kAt = NV == 1 ? kAtPq : NV == 2 ? kAtRz : kAtPre;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int h = 0; h < kPairs; ++h) {
    double in[kTwo];
#pragma unroll
    for (int m = 0; m < kTwo; ++m) in[m] = 2 * h + m < NV ? v[2 * h + m < NV ? 2 * h + m : 0] : 0.0;
    const double t = warp_sums<kTwo, false>(in, lane);
    if ((lane & 15) == 0)
      st_shared_f64(x.smem + kAtWarp + 8u * (uint32_t)(32 * (2 * h + (kTwo - 1) * (lane >> 4)) + w), t);
  }
  if (KIND == 1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (KIND == 1 && w == nw - 1) {
    if (x.z_len) push_bulk(x.z_dst, x.z_src, x.z_len, x.z_bar);
    __syncwarp();
  }
  if (w == 0) {
    const uint32_t dst = x.to_smem + kAt + kStride * (uint32_t)x.rank + 8u * (kTwo - 1) * (lane >> 4);
    const bool pushes = (lane & 15) < C && (kTwo == 2 || lane < 16);
#pragma unroll
    for (int h = 0; h < kPairs; ++h) {
      double in[kTwo];
#pragma unroll
      for (int m = 0; m < kTwo; ++m)
        in[m] = lane < nw && 2 * h + m < NV
                    ? ld_shared_f64(x.smem + kAtWarp + 8u * (uint32_t)(32 * (2 * h + m) + lane))
                    : 0.0;
      const double t = nw <= 16 ? warp_sums<kTwo, true>(in, lane) : warp_sums<kTwo, false>(in, lane);
      if (pushes && (2 * h + 1 < NV || lane < 16))
        st_async_f64(dst + 16u * h, t, x.to_bar + 8u * KIND);
    }
    __syncwarp();
  }
  const uint32_t bar = x.bar + 8u * KIND;
  const uint32_t want = (x.phases >> KIND) & 1u;
  x.phases ^= 1u << KIND;
  bool ok = true;
  if (!mbar_test_cluster(bar, want)) {
    const uint64_t t0 = global_ns();
    uint32_t spins = 0;
    while (!mbar_test_cluster(bar, want)) {
      if ((++spins & 255u) == 0) {
        if (ld_volatile_i32(x.err) != 0) { ok = false; break; }
        if (global_ns() - t0 > x.timeout_ns) {
          atomicCAS(x.err, 0, (int)EAF_ETIMEOUT);
          ok = false;
          break;
        }
      }
    }
  }
  if (threadIdx.x == blockDim.x - 1 && ok) push_expect(bar, next);
  ok = __syncthreads_and(ok) != 0;
  if (EARLY && !ok) return false;
  const uint32_t part = x.smem + kAt;
  if (NV == 1) {
    double t[CMAX];
#pragma unroll
    for (int r = 0; r < CMAX; r += 2) ld_shared_pair(part + 8u * r, t[r], t[r + 1]);
    v[0] = t[0];
#pragma unroll
    for (int r = 1; r < CMAX; ++r) v[0] = v[0] + t[r];
  } else if (NV == 2) {
    ld_shared_pair(part, v[0], v[NV - 1]);
#pragma unroll
    for (int r0 = 1; r0 < CMAX; r0 += 8) {
      double t[8], u[8];
#pragma unroll
      for (int r = r0; r < r0 + 8 && r < CMAX; ++r)
        ld_shared_pair(part + 16u * r, t[r - r0], u[r - r0]);
#pragma unroll
      for (int r = r0; r < r0 + 8 && r < CMAX; ++r) {
        v[0] = v[0] + t[r - r0];
        v[NV - 1] = v[NV - 1] + u[r - r0];
      }
    }
  } else {
    for (int m = 0; m < NV; ++m) {
      double t = ld_shared_f64(part + 8u * m);
#pragma unroll 1
      for (int r = 1; r < CMAX; ++r) t = t + ld_shared_f64(part + kStride * r + 8u * m);
      v[m] = t;
    }
  }
  return ok;
}

// The end of a solve, every thread of the cluster: no block leaves while another
// may still push into its memory. After complete exchanges a barrier says so,
// since every block has waited for all that was pushed to it. If a wait gave up,
// pushes may be in flight behind the barrier, which all blocks' pushes precede;
// each block then waits for the bytes that its open phases lack, with a limit far
// beyond a copy's time because a block that gave up may never have sent them,
// before any of them leaves.
__device__ __forceinline__ void push_leave(PushSmem& ps, const Pusher& x, int C, bool ok) {
  if (!ok && threadIdx.x < C) {
    const uint32_t to = cluster_map(smem_addr(&ps.gave_up), threadIdx.x);
    asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(to) : "memory");
  }
  __syncwarp();
  cluster_sync_all();
  if (*(volatile int*)&ps.gave_up == 0) return;
  const uint64_t t0 = global_ns();
  for (int b = 0; b < 2; ++b) {
    // (of the two parities, the open phase's is the one that has not completed)
    const uint32_t bar = x.bar + 8u * b, open = mbar_test_cluster(bar, 0u) ? 1u : 0u;
    for (int n = 0; n < 4096 && !mbar_test_cluster(bar, open); ++n)
      if (global_ns() - t0 > kPushDrainNs) break;
  }
  __syncthreads();
  cluster_sync_all();
}

// Neighbour in direction d (kW..kT) of compact cell (i, j, k), or -1 at an r
// or z wall; its direction back is d ^ 1.
__device__ __forceinline__ int neighbour(const MeshDims& d, int c, int i, int j, int k, int dir) {
  switch (dir) {
    case kW: return i > 0 ? c - 1 : -1;
    case kE: return i < d.nr - 1 ? c + 1 : -1;
    case kS: return j > 0 ? c - d.nr : c + (d.nth - 1) * d.nr;
    case kN: return j < d.nth - 1 ? c + d.nr : c - (d.nth - 1) * d.nr;
    case kB: return k > 0 ? c - d.plane : -1;
    default: return k < d.nz - 1 ? c + d.plane : -1;
  }
}

// What only the update phase uses of a thread's cells: x, the Jacobi divisor
// and its reciprocal; in registers for one cell, in shared memory for two,
// whose 128 registers would spill.
template <int R>
struct Own {
  double v[3];
  __device__ __forceinline__ void init(uint32_t) {}
  __device__ __forceinline__ void set(int, double x, double d, double y) {
    v[0] = x; v[1] = d; v[2] = y;
  }
  __device__ __forceinline__ double x(int) const { return v[0]; }
  __device__ __forceinline__ double dv(int) const { return v[1]; }
  __device__ __forceinline__ double dy(int) const { return v[2]; }
  __device__ __forceinline__ void set_x(int, double x) { v[0] = x; }
};
template <>
struct Own<2> {
  uint32_t at, row;  // three rows of 2 B doubles
  __device__ __forceinline__ void init(uint32_t base) {
    at = base + 8u * threadIdx.x;
    row = 16u * blockDim.x;
  }
  __device__ __forceinline__ uint32_t cell(int m) const { return at + (m ? row / 2 : 0u); }
  __device__ __forceinline__ void set(int m, double x, double d, double y) {
    st_shared_f64(cell(m), x);
    st_shared_f64(cell(m) + row, d);
    st_shared_f64(cell(m) + 2 * row, y);
  }
  __device__ __forceinline__ double x(int m) const { return ld_shared_f64(cell(m)); }
  __device__ __forceinline__ double dv(int m) const { return ld_shared_f64(cell(m) + row); }
  __device__ __forceinline__ double dy(int m) const { return ld_shared_f64(cell(m) + 2 * row); }
  __device__ __forceinline__ void set_x(int m, double x) { st_shared_f64(cell(m), x); }
};

template <bool SYM, int R, int CMAX>
__device__ void push_body(const DsmArgs& a, double* sm, PushSmem& ps, int C, int rank) {
  const uint32_t own_smem =
      smem_addr(sm + (size_t)(2 * a.reach + 1) * ((a.chunk + 1) & ~1));
  const MeshDims& d = a.d;
  const SysF64& s = a.s;
  const int begin = min(d.n, rank * a.chunk), end = min(d.n, begin + a.chunk);
  const int B = blockDim.x;
  int* err = a.ws.err;
  Slices zs;
  zs.reach = a.reach;
  zs.pad = (a.chunk + 1) & ~1;
  zs.base = smem_addr(sm);
  const uint32_t own_z = zs.slot(rank, rank);
  Pusher px = make_pusher(a, zs, ps, C, rank);
  const uint32_t zero = smem_addr(&ps.zero);
  const uint32_t pq_bytes = 8u * (uint32_t)C, rz_bytes = 16u * (uint32_t)C + px.z_bytes;
  if (threadIdx.x == 0) {
    push_expect(px.bar, pq_bytes);
    push_expect(px.bar + 8u, 24u * (uint32_t)C + px.z_bytes);
  }
  // Every cell of this thread; a dead one (beyond the slice) sums zeros.
  double ap[R], al[R][6], r[R], z[R], p[R], q[R], pn[R][6];
  Own<R> own;
  own.init(own_smem);
  uint32_t from[R][6], z_at[R];
  bool live[R], d_ok[R];
#pragma unroll
  for (int m = 0; m < R; ++m) {
    const int c = begin + (int)threadIdx.x + m * B;
    live[m] = c < end;
    ap[m] = r[m] = z[m] = p[m] = q[m] = 0.0;
    double xv = 0.0, dv = 1.0, dy = 1.0;
    d_ok[m] = true;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      al[m][e] = pn[m][e] = 0.0;
      from[m][e] = zero;
    }
    z_at[m] = smem_addr(&ps.dummy);
    if (live[m]) {
      z_at[m] = own_z + 8u * (uint32_t)(c - begin);
      int i, j, k;
      cell_ijk(d, c, i, j, k);
      ap[m] = s.aP[c];
      xv = s.x[c];
      r[m] = s.r[c];
      dv = guard_small(fabs(ap[m]));
      d_ok[m] = exp_in_safe_range(dv);
      dy = d_ok[m] ? 1.0 / dv : 0.0;
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const int nb = neighbour(d, c, i, j, k, e);
        const double* lower = e == kW ? s.aE : e == kS ? s.aN : s.aT;  // symmetric form
        const double* own = e == kW   ? s.aW
                            : e == kE ? s.aE
                            : e == kS ? s.aS
                            : e == kN ? s.aN
                            : e == kB ? s.aB
                                      : s.aT;
        if (SYM)
          al[m][e] = nb < 0 ? 0.0 : (e & 1) ? own[c] : lower[nb];
        else
          al[m][e] = own[c];
        if (nb < 0) continue;
        const int owner = (int)a.fd_chunk.div((uint32_t)nb);
        from[m][e] = zs.slot(rank, owner) + 8u * (uint32_t)(nb - owner * a.chunk);
      }
    }
    own.set(m, xv, dv, dy);
  }
  // z = r / max(|aP|, SMALL) of the thread's cells, kept and stored; the
  // quotient by the stored reciprocal (recipdiv.cuh), `/` outside its range.
  auto precondition = [&](int m) {
    const double dv = own.dv(m), dy = own.dy(m);
    const double t = r[m], q0 = t * dy;
    double zv = __fma_rn(__fma_rn(-q0, dv, t), dy, q0);
    if (!(d_ok[m] & (exp_in_safe_range(t) | (__double_as_longlong(t) == 0)))) {
      asm volatile("" ::: "memory");  // (keeps the division in its own branch)
      zv = t / dv;
    }
    z[m] = zv;
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(z_at[m]), "d"(zv) : "memory");
  };

  // Preamble (src/mod_solver_3d.f90:515-530).
  double v3[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int m = 0; m < R; ++m) {
    precondition(m);
    const double bv = live[m] ? s.b[begin + threadIdx.x + m * B] : 0.0;
    v3[0] = v3[0] + bv * bv;
    v3[1] = v3[1] + r[m] * r[m];
    v3[2] = v3[2] + r[m] * z[m];
  }
  bool ok = push_allsum<3, 1, CMAX, R == 2>(v3, C, rz_bytes, px);
  const double bnorm = sqrt(v3[0]);
  double residual = 0.0, rr = 0.0;
  int n_iter = 0;
  bool nan_fill = false;
  if (ok && !(bnorm < kSmall)) {
    double rz = v3[2], beta = 0.0;
    rr = v3[1];
    residual = sqrt(rr) / bnorm;
    // A r.r above this cannot give a residual below tol (the square root and
    // the quotient of the exit test, some 250 cycles, are then left out); out
    // of range, the test is always made.
    const double lim = (a.tol * bnorm) * (a.tol * bnorm) * (1.0 + 1e-12);
    const double surely_above = lim > 1e-290 && lim < 1e290 ? lim : lim == 0.0 && a.tol == 0.0
                                                                        ? 0.0
                                                                        : HUGE_VAL;
    if (residual != residual && a.max_iter >= 1) nan_fill = true;
    for (int iter = 1; iter <= a.max_iter && !nan_fill; ++iter) {
      // p = z + beta p (own and neighbours), q = A p, p.q. A missing
      // neighbour's direction stays zero: the symmetric form's link to it is
      // zero too (the term the reference's loop does not have changes
      // nothing), the general form's multiplies a zero. Only a beta that is
      // not finite would turn it into NaN.
      double v1[1] = {0.0};
      const bool first = iter == 1, finite = isfinite(beta);
#pragma unroll
      for (int m = 0; m < R; ++m) {
        double zn[6];
#pragma unroll
        for (int e = 0; e < 6; ++e) zn[e] = ld_shared_f64(from[m][e]);
        if (first) {
          p[m] = z[m];
#pragma unroll
          for (int e = 0; e < 6; ++e) pn[m][e] = zn[e];
        } else {
          p[m] = z[m] + beta * p[m];
#pragma unroll
          for (int e = 0; e < 6; ++e) pn[m][e] = zn[e] + beta * pn[m][e];
          if (!finite) {
            asm volatile("" ::: "memory");
#pragma unroll
            for (int e = 0; e < 6; ++e)
              if (from[m][e] == zero) pn[m][e] = 0.0;
            if (!live[m]) p[m] = 0.0;
          }
        }
        double y = ap[m] * p[m];
#pragma unroll
        for (int e = 0; e < 6; ++e) y = y - al[m][e] * pn[m][e];
        q[m] = y;
        v1[0] = v1[0] + p[m] * y;
      }
      if (!(ok = push_allsum<1, 0, CMAX, R == 2>(v1, C, pq_bytes, px))) break;
      const double pq = v1[0];
      if (fabs(pq) < kSmall) break;
      const double alpha = rz / pq;
      // beta's reciprocal, beside that division and off its own chain
      const double rz_g = guard_small(rz);
      const bool rz_ok = exp_in_safe_range(rz_g);
      const double rz_y = rz_ok ? 1.0 / rz_g : 0.0;
      const bool steps = isfinite(alpha);
      double v2[2] = {0.0, 0.0};
#pragma unroll
      for (int m = 0; m < R; ++m) {
        own.set_x(m, own.x(m) + alpha * p[m]);
        r[m] = r[m] - alpha * q[m];
        if (!steps && !live[m]) r[m] = 0.0;  // (0 * Inf)
        precondition(m);
        v2[0] = v2[0] + r[m] * r[m];
        v2[1] = v2[1] + r[m] * z[m];
      }
      if (!(ok = push_allsum<2, 1, CMAX, R == 2>(v2, C, rz_bytes, px))) break;
      rr = v2[0];
      n_iter = iter;
      if (!(rr > surely_above)) {
        residual = sqrt(rr) / bnorm;
        if (residual < a.tol) break;
        if (residual != residual && iter < a.max_iter) { nan_fill = true; break; }
      }
      beta = div_by_recip(v2[1], rz_g, rz_y, rz_ok);
      rz = v2[1];
    }
  }
  if (n_iter > 0) residual = sqrt(rr) / bnorm;
  const double qnan = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
  for (int m = 0; m < R; ++m)
    if (live[m]) s.x[begin + threadIdx.x + m * B] = nan_fill ? qnan : own.x(m);
  if (nan_fill) {
    residual = qnan;
    n_iter = a.max_iter;
  }
  if (rank == 0 && threadIdx.x == 0) {
    SolveResult* res = a.ws.result;
    const int e = ld_volatile_i32(err);
    res->status = e != 0 ? e : (isfinite(residual) ? EAF_OK : EAF_ENONFINITE);
    res->n_iter = n_iter;
    res->n_outer = 0;
    res->sym = SYM ? 1 : 0;
    res->residual = residual;
    res->bnorm = bnorm;
  }
  push_leave(ps, px, C, ok);
}

// Threads of a block whose cells (one or two each) fit its registers: one
// cell in 96 (640 threads) or more, two in 128.
constexpr int kPushBlock1 = 640, kPushBlock2 = 512, kPushSmall = 384;

__device__ __forceinline__ void push_init(PushSmem& ps) {
  for (int i = threadIdx.x; i < 7 * kMaxClusterSize; i += blockDim.x)
    ps.pq[i] = 0.0;  // (and rz, pre behind it)
  if (threadIdx.x == 0) {
    ps.zero = 0.0;
    ps.gave_up = 0;
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&ps.bar[b]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Every block's barriers exist before any block pushes.
  cluster_sync_all();
}

template <int R, int MAXB, int CMAX>
__global__ void __launch_bounds__(MAXB, 1) cg_push_kernel(DsmArgs a) {
  extern __shared__ __align__(16) double push_smem[];
  __shared__ __align__(16) PushSmem ps;
  const int rank = (int)cluster_ctarank(), C = (int)cluster_nctarank();
  push_init(ps);
  if (*a.s.asym == 0)
    push_body<true, R, CMAX>(a, push_smem, ps, C, rank);
  else
    push_body<false, R, CMAX>(a, push_smem, ps, C, rank);
}

// Self-test of an exchange that a block leaves out: two blocks of one cluster
// complete an exchange of partials, then only block 0 enters one with z. Its wait
// runs out, while its own partial and slice are on their way to block 1, and
// both blocks leave through push_leave.
constexpr int kPushTestCells = 256;  // per block
__global__ void __launch_bounds__(64, 1) push_selftest_kernel(DsmArgs a) {
  __shared__ __align__(16) double slices[3 * kPushTestCells];
  __shared__ __align__(16) PushSmem ps;
  const int rank = (int)cluster_ctarank(), C = (int)cluster_nctarank();
  push_init(ps);
  Slices zs;
  zs.reach = a.reach;
  zs.pad = a.chunk;
  zs.base = smem_addr(slices);
  Pusher px = make_pusher(a, zs, ps, C, rank);
  for (int i = threadIdx.x; i < a.chunk; i += blockDim.x) slices[a.chunk + i] = 1.0;
  const uint32_t pq_bytes = 8u * (uint32_t)C, rz_bytes = 16u * (uint32_t)C + px.z_bytes;
  if (threadIdx.x == 0) {
    push_expect(px.bar, pq_bytes);
    push_expect(px.bar + 8u, rz_bytes);
  }
  double v[1] = {1.0}, w[2] = {1.0, 2.0};
  bool ok = push_allsum<1, 0, 2>(v, C, pq_bytes, px) && v[0] == C * (double)blockDim.x;
  if (ok && rank == 0) ok = push_allsum<2, 1, 2>(w, C, rz_bytes, px);
  push_leave(ps, px, C, ok);
}

// Cells per thread of the pushed form for blocks of `block` threads, 0 where
// it does not apply: more cells than registers, or slices much thinner than a
// plane, whose z would go to too many blocks.
constexpr int kPushReach = 3;
int push_reach(const MeshDims& d, int chunk) { return (d.plane + chunk - 1) / chunk; }
int push_cells(const MeshDims& d, int chunk, int block) {
  const int r = (chunk + block - 1) / block;
  if (push_reach(d, chunk) > kPushReach) return 0;
  return r == 1 && block <= kPushBlock1 ? 1 : r == 2 && block <= kPushBlock2 ? 2 : 0;
}
template <int CMAX>
const void* push_kernel_of(int cells, int block) {
  if (cells == 1)
    return block <= kPushSmall ? (const void*)cg_push_kernel<1, kPushSmall, CMAX>
                               : (const void*)cg_push_kernel<1, kPushBlock1, CMAX>;
  return block <= kPushSmall ? (const void*)cg_push_kernel<2, kPushSmall, CMAX>
                             : (const void*)cg_push_kernel<2, kPushBlock2, CMAX>;
}
const void* push_kernel(int cells, int block, int cluster) {
  return cluster <= 8 ? push_kernel_of<8>(cells, block)
                      : push_kernel_of<kMaxClusterSize>(cells, block);
}
size_t push_smem_bytes(int reach, int chunk, int cells, int block) {
  const size_t slices = (size_t)(2 * reach + 1) * ((chunk + 1) & ~1);
  return (slices + (cells == 2 ? (size_t)6 * block : 0)) * sizeof(double);
}

size_t dsm_smem_bytes(int chunk) { return (size_t)kDsmArrays * chunk * sizeof(double); }

}  // namespace

int dsm_max_cells(int cluster) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
      cudaSuccess)
    return 0;
  const long long avail = (long long)optin - (long long)sizeof(PartSmem) - 1024;
  if (avail <= 0) return 0;
  const long long per_block = avail / (kDsmArrays * (long long)sizeof(double));
  return (int)(per_block * cluster);
}

bool dsm_can_launch(long long n, int block, int cluster) {
  if (cluster < 1 || cluster > kMaxClusterSize || block < 32 || block > 1024 ||
      block % 32 != 0 || n > dsm_max_cells(cluster))
    return false;
  const int chunk = (int)((n + cluster - 1) / cluster);
  const size_t smem = dsm_smem_bytes(chunk);
  const void* k = (const void*)cg_dsm_kernel<false>;
  std::lock_guard<std::mutex> attr_lock(launch_attr_mutex());
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess ||
      (cluster > 8 &&
       cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
           cudaSuccess)) {
    (void)cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int count = 0;
  if (cudaOccupancyMaxActiveClusters(&count, k, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return count >= 1;
}

cudaError_t launch_push_selftest(const GroupWs& ws, uint64_t timeout_ns, cudaStream_t st) {
  DsmArgs a = {};
  a.d.n = 2 * kPushTestCells;
  a.ws = ws;
  a.timeout_ns = timeout_ns;
  a.chunk = kPushTestCells;
  a.reach = 1;
  cudaError_t e = cudaMemsetAsync(ws.err, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(64);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, push_selftest_kernel, a);
}

cudaError_t launch_cg_f64_dsm(const MeshDims& d, const SysF64& s, const GroupWs& ws,
                              int max_iter, double tol, int block, int cluster,
                              cudaStream_t st, int signal, uint64_t timeout_ns, int* ran) {
  if (cluster < 1 || cluster > kMaxClusterSize || block < 32 || block > 1024 ||
      block % 32 != 0 || d.n > dsm_max_cells(cluster))
    return cudaErrorInvalidValue;
  DsmArgs a;
  a.d = d;
  a.s = s;
  a.ws = ws;
  a.max_iter = max_iter;
  a.tol = tol;
  a.timeout_ns = timeout_ns;
  a.chunk = (d.n + cluster - 1) / cluster;
  a.fd_chunk = FastDiv((uint32_t)a.chunk);
  // The default signalling pushes where a thread's cells fit its registers.
  const int cells = signal == kDsmSignalMbarrier ? 0 : push_cells(d, a.chunk, block);
  a.reach = push_reach(d, a.chunk);
  if (ran)
    *ran = cells ? EAF_CG_RESIDENT_PUSHED
           : signal == kDsmSignalMbarrier ? EAF_CG_RESIDENT_MBARRIER : EAF_CG_RESIDENT_BARRIER;
  const size_t smem = cells ? push_smem_bytes(a.reach, a.chunk, cells, block) : dsm_smem_bytes(a.chunk);
  const void* k = cells ? push_kernel(cells, block, cluster)
                  : signal == kDsmSignalMbarrier ? (const void*)cg_dsm_kernel<true>
                                                 : (const void*)cg_dsm_kernel<false>;
  std::lock_guard<std::mutex> attr_lock(launch_attr_mutex());
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e == cudaSuccess) e = cudaMemsetAsync(ws.err, 0, sizeof(int), st);
  if (e == cudaSuccess && cluster > 8)
    e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  (void)cudaGetLastError();  // report this launch's error, not an older one
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  return cudaLaunchKernelExC(&cfg, k, args);
}

}  // namespace eaf
