// common.cuh -- shared device helpers and data layout of the B200 step.
//
// Data layout in HBM (one context = one scene):
//   positions / velocities / targets        : double[3V]   (AoS xyz per vertex)
//   Newton gradient                         : double[3V]
//   PCG vectors (b, x, r, z, p ping-pong, Ap): float[3V]
//   BSR Hessian values                      : float[9*nnzb] (row-major 3x3 blocks)
//   BSR pattern                             : rowptr int[V+1], cols int[nnzb], slot_row int[nnzb]
//   block-Jacobi inverse                    : float[9V]
// The BSR pattern is static (self + mesh-edge blocks); contact blocks between
// non-adjacent vertices live in a per-step "extra" segment sorted by row.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ando {

// ----------------------------------------------------------------- vectors
struct d3 { double x, y, z; };
__host__ __device__ inline d3 mk(double a, double b, double c) { return d3{a, b, c}; }
__host__ __device__ inline d3 operator+(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__host__ __device__ inline d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__host__ __device__ inline d3 operator-(d3 a) { return {-a.x, -a.y, -a.z}; }
__host__ __device__ inline d3 operator*(d3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__host__ __device__ inline d3 operator/(d3 a, double s) { return {a.x / s, a.y / s, a.z / s}; }
__host__ __device__ inline double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__host__ __device__ inline double sqn(d3 a) { return a.x * a.x + a.y * a.y + a.z * a.z; }
__host__ __device__ inline double nrm(d3 a) { return sqrt(sqn(a)); }
__host__ __device__ inline d3 cross(d3 a, d3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__host__ __device__ inline double comp(d3 a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }
__host__ __device__ inline d3 normalized(d3 a) { double n2 = sqn(a); return n2 > 0.0 ? a / sqrt(n2) : a; }
__device__ inline d3 ld3(const double* p, int i) { return {p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ inline void st3(double* p, int i, d3 v) { p[3 * i] = v.x; p[3 * i + 1] = v.y; p[3 * i + 2] = v.z; }

// --------------------------------------------------- cubic barrier (barrier.cpp:29-65)
__host__ __device__ inline double bar_energy(double g, double gm, double k) {
  if (gm <= 0.0 || g >= gm) return 0.0;
  double d = gm - g; if (d <= 0.0) return 0.0;
  return 0.5 * k * (1.0 / gm) * d * d * d;
}
__host__ __device__ inline double bar_grad(double g, double gm, double k) {
  if (gm <= 0.0 || g >= gm) return 0.0;
  double d = gm - g; return -1.5 * k * (1.0 / gm) * d * d;
}
__host__ __device__ inline double bar_hess(double g, double gm, double k) {
  if (gm <= 0.0 || g >= gm) return 0.0;
  double d = gm - g; return 3.0 * k * (1.0 / gm) * d;
}
__host__ __device__ inline bool in_domain(double g, double gm) { return gm > 0.0 && g <= gm; }
__host__ __device__ inline d3 normalize_or_default(d3 n, double eps) { return sqn(n) > eps * eps ? normalized(n) : mk(0.0, 1.0, 0.0); }

// CORRECTED pin stiffness: kappa = PIN_SCALE (m / dt^2 + a) with a the
// vertex's elastic diagonal coefficient; a pinned vertex then follows its
// target within about 1 % of the elastic load on it.
constexpr double PIN_SCALE = 100.0;

// -------------------------------------------------------------- parameters
struct WallDev { double n[3]; double offset, gap; int active; };

struct StepParams {
  double dt, dt2inv, contact_gap_max, wall_gap, normal_eps, barrier_tol, min_gap;
  double friction_mu, friction_eps, friction_thresh;
  int enable_friction, enable_strain, semantics;
  double strain_tau, strain_eps, svd_eps;  // already converted by to_fraction
  int num_walls;
  int first_wall;                          // index of the first active wall, -1 if none
};

// --------------------------------------------------------------- contacts
struct ContactDev {
  int type, idx[4], rigid, count;
  double gap, n[3], wp[3], wq[3], bary[3], w[4];
  // per-step constants (frozen gap, frozen normal)
  double kbar, dV, d2V, nn[3];
  int in_dom;
};

// The fields up to the weights, as the public ando_contact holds them.
constexpr int CONTACT_OUT_BYTES = 168;

// What the block sums read of a contact: 96 bytes (three sectors; the merged
// off-diagonal blocks read the first two) in place of ContactDev's 224, so a
// contact met from its four vertices and twelve blocks costs a third.
struct alignas(32) ContactRec {
  double nn[3], w[4], d2V;
  int idx[4];
  double dV;
  unsigned mask;   // bit i: vertex i carries a weight; REC_HESS, REC_GRAD: a Hessian / gradient to add
  unsigned pad;
};
static_assert(sizeof(ContactRec) == 96 && offsetof(ContactRec, idx) % 16 == 0, "records are read in 16-byte pieces");
constexpr unsigned REC_HESS = 16u, REC_GRAD = 32u;

// Contact entries, sorted by vertex and in contact order within one: 4 * contact
// + local vertex, with ENTRY_FRICTION where the vertex takes the contact's friction.
constexpr int ENTRY_FRICTION = 1 << 30;

// --------------------------------------------------------- mesh on device
struct MeshDev {
  int V, T, nnzb;
  double mu, thickness, density;   // material: mu = E / (2 (1 + nu))
  const int* tris;          // 3T
  const double* rest_area;  // T
  const double* dm_inv;     // 4T (a b c d row-major)
  const double* mass;       // V
  const int* rowptr;        // V+1
  const int* cols;          // nnzb
  const int* slot_row;      // nnzb
  const int* diag_slot;     // V
  const int* face_slot;     // 9T  slot of block (a,b) of face f at f*9+a*3+b
  const int* slot_cptr;     // nnzb+1
  const int* slot_contrib;  // 9T   entries f*9+a*3+b, sorted by face within a slot
  const int* vf_ptr;        // V+1
  const int* vf;            // 3T   entries f*3+a, sorted by face within a vertex
  const double* el_a;       // nnzb elastic in-plane coefficient of the diag(a,a,b) block
  const double* el_b;       // nnzb elastic third-axis coefficient
  const double* g_elastic;  // 3V  elastic gradient on the mesh vertices (constant)
  // nnzb coefficient q of the quadratic bending Hessian q I3 per slot
  // (CORRECTED semantics, bending_stiffness > 0; null without bending)
  const double* bend_q;
  // 13 per face (R0, R1, n, a_t, W00, W01, W11) of the projected exact membrane
  // Hessian at the current positions (CORRECTED, membrane_hessian projected;
  // null otherwise): the assembly subtracts its correction of the constant
  // fixed-rotation blocks
  const double* mface;
};
constexpr int MFACE = 13;

// Strain-limit data of one face and one singular value.
struct StrainSV { double J[9]; double dV, d2V; };

// Lower-triangular 3x3 (Cholesky factor or its inverse), row-major packed.
struct Tri3 { double l00, l10, l11, l20, l21, l22; };

// -------------------------------------------------------- device control
struct Ctrl {
  unsigned long long gnorm_bits;  // max |g| as IEEE bits (non-negative doubles order as integers)
  unsigned int ls_mask;           // AND over all feasibility masks, bit j = level j feasible
  int converged;                  // gradient-norm test passed this Newton iteration
  int pcg_iters, pcg_converged, pcg_status;
  double pcg_rel;
  double alpha;
  int strain_active;
  int bar_err;                    // a bounded wait of the PCG gave up
  int tc_err;                     // a tensor-core GEMM's bounded wait gave up (sticky)
  int toi_overflow;               // > 0: a time-of-impact candidate list needed this many slots; the move was not applied
  int learned_iters;              // iterations of this Newton iteration's learned solve
  int fallback_ran;               // block-Jacobi redid this Newton iteration's learned solve
  int xs_blocks;                  // block places of the contact blocks' SELL-32 copy (-1: too uneven)
  unsigned long long bar_arrivals;  // xr_reduce (and grid_sync_ar): arrivals since the launcher zeroed it
};

// PCG_NOT_SPD: |p^T A p| < 1e-16, or p^T A p or a residual that is not finite.
// PCG_PRECOND: the learned preconditioner lost positive definiteness
// (r^T z <= 0); PCG_STALL: its residual stopped improving. All three hand a
// learned solve back to block-Jacobi.
enum PcgStatus { PCG_OK = 0, PCG_MAXIT = 1, PCG_NOT_SPD = 2, PCG_TIMEOUT = 3, PCG_SKIPPED = 4, PCG_PRECOND = 5, PCG_STALL = 6 };

// Device-side control of one step (integrator.cpp:98-121 and 152-236) when the
// whole frame runs as one CUDA graph: the beta loop, the error-reduction pass
// and the Newton loop are decided on the device between graph iterations.
struct StepCtl {
  double beta, ret, last_alpha;
  int bi, phase, newton_it, max_it;   // phase 0: beta loop, 1: error-reduction pass, 2: done
  int newton_iters, pcg_iters, pcg_max, pcg_not_converged, line_search_fail, strain_active, error;
  int iterations_run;                 // Newton bodies executed (launch accounting)
  int arrived;                        // blocks of the iteration's last kernel
};

// Bounded grid barrier with acquire/release atomics: every CTA adds one
// arrival to a 64-bit counter that the launcher zeroed (release: the CTA's
// writes, ordered before the arrival by __syncthreads, are published) and
// polls with acquire loads until all nblocks CTAs have arrived `epoch` times.
// The polling thread hands
// its verdict to the CTA through shared memory, so the other threads leave
// the barrier without another L2 round trip. A CTA that passed a barrier
// while another CTA was giving up on it meets the error flag in the poll of
// the next barrier (every wait stays bounded), and the host reads the flag
// after the launch.
__device__ inline bool grid_sync_ar(unsigned long long* arrivals, unsigned int nblocks, unsigned int& epoch, int* err) {
  __shared__ int passed;
  __syncthreads();  // also orders the previous call's reads of `passed` before this call's write
  ++epoch;
  if (threadIdx.x == 0) {
    const unsigned long long target = (unsigned long long)epoch * nblocks;
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(arrivals) : "memory");
    long long polls = 0;
    int ok = 1;
    while (true) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(arrivals) : "memory");
      if (v >= target) break;
      if (*(volatile int*)err) { ok = 0; break; }
      if (++polls > (1ll << 24)) { atomicExch(err, 1); ok = 0; break; }
      if (polls > 1024) __nanosleep(32);
    }
    passed = ok;
  }
  __syncthreads();
  return passed != 0;
}

// ------------------------------------------------ PCG reductions across CTAs
// A PCG iteration is two dot products with a barrier each. These reductions
// are the barrier: every CTA hands over its partial sum (and maximum) with its
// arrival and leaves with the total of one partial per CTA.
//
// Grid form (cooperative launch, at most XR_MAX_CTAS CTAs): a CTA writes its
// partial and adds one arrival to a 64-bit counter that the launcher zeroed
// (release: the CTA's writes, ordered before the arrival by __syncthreads, are
// published); one thread polls the counter (acquire) and its warp then reads
// all partials. They alternate between two sets: a CTA writes set s again only
// after a reduction that every CTA has entered, so nobody still reads it. The
// polls are bounded; on timeout the error flag makes the other CTAs leave
// their next wait, and the host reads the flag after the launch. Measured
// alone, 148 CTAs of 896 threads: 2.25 us; polling one flagged slot per CTA
// instead of the counter 3.4 us (148 x 148 reads of the same lines), two
// levels of such slots 2.0 us without and 2.8 us with the publication,
// clusters of 8 handing one partial each 2.6 us.
//
// Cluster form (cl_reduce, the whole launch is one cluster of at most 16
// CTAs): each CTA leaves its partial in its own shared memory, the cluster
// barrier follows, and one warp of each CTA reads the others'. The barrier's
// release waits for every outstanding store of the thread: 360 to 500 cycles
// with shared-memory stores, 900 to 2,000 behind global ones; with a release
// restricted to the CTA's own shared memory it takes 100 to 280. So the
// cluster form publishes its vectors in shared memory and writes no global
// memory between its barriers.
//
// In both forms one thread of each CTA turns the total into the iteration's
// scalar (`tail`) and the others read that from shared memory: the FP64
// divisions and the state of the stopping test take no registers of theirs.
// The partials are added in an order that depends on the numbers of CTAs and
// slices only.
constexpr int XR_MAX_CTAS = 160;
constexpr int XR_MAX_SLICES = 96;   // 32-row slices of one CTA whose partials fit its shared array
struct alignas(16) XrSlot { double v; unsigned m, pad; };
constexpr size_t XR_SLOTS = 2ull * XR_MAX_CTAS;

struct XrSmem {
  double part[XR_MAX_SLICES];
  unsigned pmax[XR_MAX_SLICES];
  XrSlot mine[2];                   // cluster form: this CTA's partial
};

__device__ inline double xr_warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// |v| as bits whose unsigned order is the order of the magnitudes, with a NaN
// above infinity: the maximum of a vector that holds one is not a small residual
__device__ inline unsigned xr_mag(float v) { return __float_as_uint(fabsf(v)); }
constexpr unsigned XR_NOT_FINITE = 0x7f800000u;   // xr_mag of infinity; a NaN's is above

// Sum of part[0, n) and max of pmax[0, n) over the calling warp's lanes; the
// total is lane 0's. (Lanes past n hold zeros, so up to 32 entries need only
// log2(n) exchanges.)
__device__ inline void xr_block_total(const XrSmem& sh, int n, double& v, unsigned& m) {
  const int l = threadIdx.x & 31;
  v = 0.0; m = 0u;
  for (int k = l; k < n; k += 32) { v += sh.part[k]; m = max(m, sh.pmax[k]); }
  for (int o = n > 16 ? 16 : n > 8 ? 8 : n > 4 ? 4 : n > 2 ? 2 : n > 1 ? 1 : 0; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  m = __reduce_max_sync(0xffffffffu, m);
}

// Total over all CTAs of the partials that the warps left in sh.part / sh.pmax
// (n slices of this CTA; written before this call, no barrier needed). Writes
// to global memory made by any thread of the grid before the call are visible
// to every thread after it. `epoch`: this is the epoch-th reduction of the
// launch, from 1. One thread calls tail(ok, sum, max); what it writes to
// shared memory is visible to the CTA afterwards. ok: no wait gave up. Called
// by all threads.
template <class Tail>
__device__ inline void xr_reduce(XrSmem& sh, int n, unsigned epoch, XrSlot* slots, unsigned long long* arrivals, int* err, Tail tail) {
  __syncthreads();
  const int nb = gridDim.x;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    double v; unsigned m;
    xr_block_total(sh, n, v, m);
    XrSlot* set = slots + (epoch & 1u) * XR_MAX_CTAS;
    bool good = true;
    if (lane == 0) {
      *reinterpret_cast<uint4*>(set + blockIdx.x) = make_uint4((unsigned)__double2loint(v), (unsigned)__double2hiint(v), m, 0u);
      const unsigned long long target = (unsigned long long)epoch * (unsigned)nb;
      asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(arrivals) : "memory");
      long long polls = 0;
      while (true) {
        unsigned long long c;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(arrivals) : "memory");
        if (c >= target) break;
        if ((++polls & 1023) == 0) {
          if (*(volatile int*)err) { good = false; break; }
          if (polls > (1ll << 24)) { atomicExch(err, 1); good = false; break; }
        }
      }
    }
    __syncwarp();
    v = 0.0; m = 0u;
#pragma unroll
    for (int k = 0; k < XR_MAX_CTAS / 32; ++k) {
      const int s = lane + 32 * k;
      if (s < nb) {
        const uint4 q = __ldcg(reinterpret_cast<const uint4*>(set + s));   // written by other CTAs: read from L2
        v += __hiloint2double((int)q.y, (int)q.x);
        m = max(m, q.z);
      }
    }
    v = xr_warp_sum(v);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) tail(good, v, m);
  }
  __syncthreads();
}

__device__ inline unsigned cl_size() { unsigned r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
// Cluster barrier that orders the CTAs' own shared-memory writes before it with any CTA's reads of them after it.
__device__ inline void cl_sync_shared() {
  asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\t"
               "barrier.cluster.arrive.relaxed;\n\t"
               "barrier.cluster.wait.acquire;\n\t"
               "fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
}
// shared::cluster address of a location of this CTA's shared memory in CTA `rank`
__device__ inline unsigned cl_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// xr_reduce over a cluster: shared-memory writes of any thread of the cluster
// before the call are visible to every thread after it. No CTA may leave the
// kernel before a further cl_sync_shared (others still read its partial).
template <class Tail>
__device__ inline void cl_reduce(XrSmem& sh, int n, unsigned epoch, Tail tail) {
  __syncthreads();
  const int lane = threadIdx.x & 31, par = epoch & 1u;
  if (threadIdx.x < 32) {
    double v; unsigned m;
    xr_block_total(sh, n, v, m);
    if (lane == 0) sh.mine[par] = XrSlot{v, m, 0u};
  }
  cl_sync_shared();
  if (threadIdx.x < 32) {
    const int C = (int)cl_size();
    double v = 0.0;
    unsigned m = 0u;
    if (lane < C) {
      unsigned lo, hi, z;
      const unsigned at = cl_map((unsigned)__cvta_generic_to_shared(&sh.mine[par]), lane);
      asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(lo), "=r"(hi), "=r"(m), "=r"(z) : "r"(at) : "memory");
      v = __hiloint2double((int)hi, (int)lo);
    }
    for (int o = C > 8 ? 8 : C > 4 ? 4 : C > 2 ? 2 : C > 1 ? 1 : 0; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) tail(true, v, m);
  }
  __syncthreads();
}

}  // namespace ando
