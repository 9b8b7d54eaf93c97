// pcg.cu -- block-Jacobi preconditioned conjugate gradients as one persistent
// cooperative kernel (replaces PCGSolver::solve, pcg_solver.cpp:8-146).
//
// Same iteration as the reference: x0 = 0, r = b, block-Jacobi z = P r,
// stop when |r|_inf / |b|_inf < tol (or |r|_inf when |b|_inf < 1e-16), fail
// when |p^T A p| < 1e-16 or a NaN or infinity appears. Vectors and the BSR
// matrix are FP32; every dot product and norm is accumulated in FP64 and reduced
// in a fixed order, so results are bitwise reproducible run to run.
//
// Per iteration there are two barriers over the launch's CTAs:
//   A: p_new = z + beta p_old (recomputed on the fly for gathered columns),
//      Ap = A p_new, partial p^T Ap
//   B: x += alpha p, r -= alpha Ap, z = P r, partial r^T z and |r|_inf
// The barriers are bounded (common.cuh): on timeout the kernel reports
// PCG_TIMEOUT instead of spinning forever.
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "copy_pieces.cuh"
#include "kernels.cuh"

namespace ando {

namespace {

// ---------------------------------------------------------- unscaled PCG
// What bounds it: a small system by the two dependent reductions of an
// iteration, a large one by reading the matrix and its neighbours' vectors from
// L2. So
//  - each warp owns whole 32-row slices, one thread per row. A warp with one
//    slice (ONE) keeps its rows' r, z, p, A p, P and x in registers for the
//    whole solve; only z and p are published, for the neighbours' products. With
//    more slices to a warp the rows' state stays in the caller's vectors (two
//    or three rows' state per thread spilled: 26 us an iteration at 262,144
//    rows against 20);
//  - a warp copies a slice's blocks and columns, contiguous in the CSR arrays,
//    into its own shared-memory buffer with 16-byte asynchronous copies: once
//    per solve if it has one slice; otherwise it walks its slices up and down in
//    turn, so that one of them is always still there. The row stride of 9 x 7
//    floats reads without bank conflicts;
//  - the barrier of each dot product carries the sum (xr_reduce).
constexpr int PCG_WARPS = 24;                 // 24 x 9.4 KB of shared memory: a slice of 32 rows of 7 blocks each
// (a launch of up to 20 warps takes the kernel compiled for 20, with 96 registers
// to a thread in place of 80: 90,000 rows 7.8 us an iteration in place of 8.6)
// With several slices to a warp the buffers leave room in the L1 for the
// gathers, and the slices divide evenly: 262,144 rows on 19 warps with 9.1 KB
// each 20.5 us an iteration, on 24 warps 28.4, on 12 26.9 (with a row's sum in
// one part; in eight, 21.8 on 19 warps).
constexpr int PCG_WARPS_MANY = 20, PCG_BUF_MANY = 9344;
constexpr int PCG_CLUSTER_TPB = 512;
constexpr int PCG_SMEM = 224 * 1024;          // all warps' buffers

// The solve's scalars, in shared memory: written by the thread that ends a
// reduction, read by the CTA after it (coef: alpha after phase A, beta after
// phase B).
struct PcgScalars {
  double rz, binf, rel, best;
  int status, iters, since;
  float coef;
  // max |b| and r^T z of the initial residual
  __device__ void start(bool ok, double rz0, unsigned mx, float tol, bool learned) {
    rz = rz0; binf = double(__uint_as_float(mx)); rel = 0.0; iters = 0; since = 0; coef = 0.f; status = PCG_MAXIT;
    if (!ok) { status = PCG_TIMEOUT; return; }
    best = rel = binf < 1e-16 ? binf : 1.0;
    if (mx >= XR_NOT_FINITE) status = PCG_NOT_SPD;
    else if (rel < double(tol)) status = PCG_OK;
    else if (learned && !(rz > 0.0)) status = PCG_PRECOND;
  }
  __device__ void after_product(bool ok, double pap) {
    if (!ok) { status = PCG_TIMEOUT; return; }
    ++iters;
    if (!(fabs(pap) >= 1e-16)) status = PCG_NOT_SPD;   // a NaN too
    else coef = float(rz / pap);
  }
  __device__ void after_update(bool ok, double rz_new, unsigned mx, float tol, int stall_window) {
    if (!ok) { status = PCG_TIMEOUT; return; }
    const double rinf = double(__uint_as_float(mx));
    rel = binf < 1e-16 ? rinf : rinf / binf;
    if (mx >= XR_NOT_FINITE) { status = PCG_NOT_SPD; return; }
    if (rel < double(tol)) { status = PCG_OK; return; }
    if (stall_window > 0) {   // learned preconditioner
      if (!(rz_new > 0.0)) { status = PCG_PRECOND; return; }
      if (rel < best) { best = rel; since = 0; }
      else if (++since >= stall_window) { status = PCG_STALL; return; }
    }
    coef = float(rz_new / rz);
    rz = rz_new;
  }
  __device__ void report(Ctrl* ctrl) const {
    ctrl->pcg_iters = iters;
    ctrl->pcg_status = status;
    ctrl->pcg_converged = status == PCG_OK ? 1 : 0;
    ctrl->pcg_rel = rel;
  }
};

// Row stride of z and p: float4 rows where the state is in registers, packed
// rows where the caller's work buffer also holds r and A p.
template <int S> __device__ inline float4 ld4(const float* v, int j) {
  if (S == 4) return reinterpret_cast<const float4*>(v)[j];
  return make_float4(v[3 * j], v[3 * j + 1], v[3 * j + 2], 0.f);
}
template <int S> __device__ inline void st4(float* v, int j, float a, float b, float c) {
  if (S == 4) reinterpret_cast<float4*>(v)[j] = make_float4(a, b, c, 0.f);
  else { v[3 * j] = a; v[3 * j + 1] = b; v[3 * j + 2] = c; }
}

// Asynchronous copy of n 4-byte elements from src into 16-byte aligned shared
// memory, by the calling warp, in whole 16-byte pieces of global memory and the
// elements beside them one by one (the array may be a caller's, and its
// neighbours another's). Returns the element offset of src[0] in dst.
__device__ inline int warp_copy_async(void* dst, const void* src, int n) {
  const int off = int(reinterpret_cast<size_t>(src) & 15) >> 2;
  const char* g = reinterpret_cast<const char*>(src) - 4 * off;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const CopyPieces p = copy_pieces(off, n);
  const int lane = threadIdx.x & 31;
  for (int q = p.q0 + lane; q < p.q1; q += 32)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * q), "l"(g + 16ll * q) : "memory");
  const int e = off + (lane < 4 ? lane : n - p.tail + lane - 4);   // lanes 0 to 2: the head, 4 to 6: the tail
  if (lane < 4 ? lane < p.head : lane - 4 < p.tail)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4u * e), "l"(g + 4ll * e) : "memory");
  return off;
}

// The roundings of the unscaled PCG are written out, so that its forms agree:
// y + a x, and a . b with the middle product rounded first.
__device__ inline float axpy(float a, float x, float y) { return __fmaf_rn(a, x, y); }
__device__ inline float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
  return __fmaf_rn(a2, b2, __fmaf_rn(a0, b0, __fmul_rn(a1, b1)));
}
// t += block h times q
__device__ inline void block_product(const float* h, const float (&q)[3], float (&t)[3]) {
  for (int c = 0; c < 3; ++c) t[c] = __fadd_rn(t[c], dot3(h[3 * c], h[3 * c + 1], h[3 * c + 2], q[0], q[1], q[2]));
}

// A row's product is summed in eight parts, block e into part e mod 8, and the
// parts by halves: ((0 + 4) + (2 + 6)) + ((1 + 5) + (3 + 7)), the sum of a
// butterfly over eight lanes. One block after the other rounds 15 to 35 % worse
// (root mean square, against 64 bits), and on systems whose blocks span eleven
// orders of magnitude (a strain limit met by an irregular mesh) that decides
// whether a solve takes 8 iterations or none of 1,000 suffices.
// Blocks of half h in the order of its four parts: 0 4 2 6 and 1 5 3 7.
__device__ inline int half_block(int h, int u) { return h + (u == 1 ? 4 : u == 2 ? 2 : u == 3 ? 6 : 0); }
__device__ inline void add_half(const float (&t)[4][3], float (&y)[3]) {
  for (int c = 0; c < 3; ++c) y[c] += __fadd_rn(__fadd_rn(t[0][c], t[1][c]), __fadd_rn(t[2][c], t[3][c]));
}
// One half's blocks among [0, n), B of them gathered at once (4 or 2), added to
// its parts. col(e): the block's column or its handle.
template <int B, class Col, class Vec>
__device__ inline void add_parts(int h, int n, const Col& col, const float* val, const Vec& vec, float (&t)[4][3]) {
  for (int e0 = h; e0 < n; e0 += 8) {
#pragma unroll
    for (int b = 0; b < 4; b += B) {
      typename Vec::Raw raw[B];
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (half_block(e0, b + u) < n) vec.load(col(half_block(e0, b + u)), raw[u]);
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (half_block(e0, b + u) < n) {
          float q[3];
          vec.value(raw[u], q);
          block_product(val + 9 * half_block(e0, b + u), q, t[b + u]);
        }
    }
  }
}

// Rows of more than PCG_WIDE blocks are summed by their warp, one row after
// another with a block to each lane. By its thread alone a row of 900 blocks took
// 220 us an iteration and one of 8,000 2.4 ms (15 and 60 so), and rows of 81
// throughout 569 us at 90,000 rows (110 so), which their threads read from memory
// in pieces. Rows of 27 throughout are the faster by thread, 38 us against 65
// with a warp to a row at 8,100 rows; of 41, 103 against 50.
constexpr int PCG_WIDE = 32;

// y += the row of n blocks from k0 on, for the lanes whose n is above PCG_WIDE. Called by the whole warp.
template <class Vec>
__device__ inline void add_wide(int k0, int n, const int* cols, const float* val, const Vec& vec, float (&y)[3]) {
  const int lane = threadIdx.x & 31;
  for (unsigned left = __ballot_sync(0xffffffffu, n > PCG_WIDE); left; left &= left - 1) {
    const int src = __ffs(left) - 1;
    const int first = __shfl_sync(0xffffffffu, k0, src), last = first + __shfl_sync(0xffffffffu, n, src);
    float t[3] = {0.f, 0.f, 0.f};
#pragma unroll 2
    for (int k = first + lane; k < last; k += 32) {
      typename Vec::Raw raw;
      float q[3];
      vec.load(vec.handle(cols[k]), raw);
      vec.value(raw, q);
      block_product(val + 9ll * k, q, t);
    }
    for (int c = 0; c < 3; ++c) {
      for (int o = 16; o; o >>= 1) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
      if (lane == src) y[c] += t[c];
    }
  }
}

// The lane's row in general: its first `held` blocks (8 | held, or all) from the
// buffer, the others and the extra segment's from memory. One copy of the code
// for the three: a register spilled is a store that every barrier waits for.
struct RowAt { int row, k0, n, held; const int* cols; const float* val; };   // cols, val: in the buffer
template <int B, class Vec>
__device__ inline void add_row(const PcgArgs& a, const RowAt r, const Vec& vec, float (&y)[3]) {
  const int xb = a.xbegin && r.row < a.V ? a.xbegin[r.row] : 0, xn = a.xbegin && r.row < a.V ? a.xend[r.row] - xb : 0;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float t[4][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll 1
    for (int s = 0; s < (a.xbegin ? 3 : 2); ++s) {
      const int* cols = s == 0 ? r.cols : s == 1 ? a.cols + r.k0 + r.held : a.xcols + xb;
      const float* val = s == 0 ? r.val : s == 1 ? a.val + 9ll * (r.k0 + r.held) : a.xval + 9ll * xb;
      const int n = s == 0 ? r.held : s == 1 ? (r.n > PCG_WIDE ? 0 : r.n - r.held) : xn;
      add_parts<B>(h, n, [&](int e) { return s == 0 ? vec.held(cols[e]) : vec.handle(cols[e]); }, val, vec, t);
    }
    add_half(t, y);
  }
  if (__any_sync(0xffffffffu, r.n > PCG_WIDE)) add_wide(r.k0, r.n, a.cols, a.val, vec, y);
}

// p_new = z + beta p_old of a column: from the published rows
template <int S> struct NewP {
  const float* z; const float* pold; float beta; bool first;
  struct Raw { float4 z, p; };
  __device__ int handle(int col) const { return col; }
  __device__ int held(int c) const { return c; }   // of a column entry in the buffer
  __device__ void load(int c, Raw& r) const { r.z = ld4<S>(z, c); r.p = first ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4<S>(pold, c); }
  __device__ void value(const Raw& r, float (&v)[3]) const {
    v[0] = first ? r.z.x : axpy(beta, r.p.x, r.z.x); v[1] = first ? r.z.y : axpy(beta, r.p.y, r.z.y); v[2] = first ? r.z.z : axpy(beta, r.p.z, r.z.z);
  }
};

// ALL: the CTA's rows have all their blocks in the buffers, and none elsewhere.
template <bool ONE, bool ALL>
__device__ __forceinline__ void pcg_solve(const PcgArgs& a, XrSmem& sh, PcgScalars& st) {
  Ctrl* ctrl = a.ctrl;
  extern __shared__ __align__(16) unsigned char pcg_dyn[];
  constexpr int S = ONE ? 4 : 3;
  // P and x of the row too, whose registers the other copy needs: a register
  // spilled is a store that each barrier waits for (1 to 2 us an iteration)
  constexpr bool KEEP = ONE && ALL;
  const int V = a.V, ns = (V + 31) >> 5, spc = (ns + (int)gridDim.x - 1) / (int)gridDim.x;
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  const int s0 = blockIdx.x * spc, sn = max(0, min(spc, ns - s0));   // slices [s0, s0 + sn)
  const int wbuf = (a.smem / nw) & ~15, cap = (wbuf - 64) / 40;      // blocks that a warp's buffer holds
  unsigned char* buf = pcg_dyn + (size_t)w * wbuf;
  float* bval = reinterpret_cast<float*>(buf);
  int* bcol = reinterpret_cast<int*>(buf + ((36 * cap + 16 + 15) & ~15));
  float r[3], z[3], p[3], q[3], x[3], Pm[9];   // ONE: the row's state
  int kb = 0, cnt = 0;
  int held = -1, vo = 0, co = 0, hk0 = 0;   // slice in the buffer, element offsets of its first block and column, that block
  auto row_of = [&](int j) { return 32 * (s0 + j) + lane; };
  auto load_P = [&](int row, float (&m)[9]) {
    for (int e = 0; e < 9; ++e) m[e] = a.P[9ll * row + e];
  };
  auto apply_P = [&](const float (&m)[9], const float (&v)[3], float (&o)[3]) {
    for (int c = 0; c < 3; ++c) o[c] = dot3(m[3 * c], m[3 * c + 1], m[3 * c + 2], v[0], v[1], v[2]);
  };
  // slice j's partials of the next reduction: the warp's, of all its slices in turn
  auto hand_over = [&](double v, float m0, float m1, float m2) {
    v = xr_warp_sum(v);
    const unsigned m = __reduce_max_sync(0xffffffffu, max(xr_mag(m0), max(xr_mag(m1), xr_mag(m2))));
    if (lane == 0) { sh.part[w] += v; sh.pmax[w] = max(sh.pmax[w], m); }
  };
  auto begin = [&]() { if (lane == 0) { sh.part[w] = 0.0; sh.pmax[w] = 0u; } __syncwarp(); };
  auto reduce = [&](unsigned epoch, auto tail) { xr_reduce(sh, nw, epoch, a.slots, &ctrl->bar_arrivals, &ctrl->bar_err, tail); };

  // init: x = 0, r = b, z = P r
  begin();
  for (int j = w; j < sn; j += nw) {
    const int row = row_of(j);
    double rz_loc = 0.0;
    float b[3] = {0.f, 0.f, 0.f}, zz[3];
    if (row < V) {
      for (int e = 0; e < 3; ++e) b[e] = a.b[3 * row + e];
      float m[9];
      load_P(row, m);
      apply_P(m, b, zz);
      st4<S>(a.z, row, zz[0], zz[1], zz[2]);
      rz_loc = double(b[0]) * zz[0] + double(b[1]) * zz[1] + double(b[2]) * zz[2];
      if (ONE) {
        kb = a.rowptr[row]; cnt = a.rowptr[row + 1] - kb;
        if (KEEP) for (int e = 0; e < 9; ++e) Pm[e] = m[e];
        for (int e = 0; e < 3; ++e) { r[e] = b[e]; z[e] = zz[e]; x[e] = 0.f; p[e] = 0.f; if (!KEEP) a.x[3 * row + e] = 0.f; }
      } else {
        for (int e = 0; e < 3; ++e) { a.x[3 * row + e] = 0.f; a.r[3 * row + e] = b[e]; }
      }
    }
    hand_over(rz_loc, b[0], b[1], b[2]);
  }
  reduce(1, [&](bool ok, double rz, unsigned mx) { st.start(ok, rz, mx, a.tol, false); });
  float beta = 0.f;
  float* pold = a.p0;
  float* pnew = a.p1;
  bool first = true;
  for (int it = 0; st.status == PCG_MAXIT && it < a.max_iters; ++it) {
    // ---- phase A: p_new = z + beta p_old, Ap = A p_new, p^T Ap
    begin();
    const int slices = w < sn ? (sn - 1 - w) / nw + 1 : 0;
    for (int t = 0; t < slices; ++t) {
      const int j = w + nw * ((it & 1) == 0 ? t : slices - 1 - t), row = row_of(j);   // up and down in turn
      int k0 = kb, n = cnt;
      if (!ONE) {
        k0 = 0; n = 0;
        if (row < V) { k0 = a.rowptr[row]; n = a.rowptr[row + 1] - k0; }
      }
      if (held != j) {
        const int first_block = __shfl_sync(0xffffffffu, k0, 0);
        const int nb = __reduce_max_sync(0xffffffffu, n > 0 ? k0 + n - first_block : 0);
        __syncwarp();
        hk0 = first_block;
        vo = warp_copy_async(bval, a.val + 9ll * first_block, 9 * min(nb, cap));
        co = warp_copy_async(bcol, a.cols + first_block, min(nb, cap));
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        held = j;
      }
      const int lo = k0 - hk0;
      const int* bc = bcol + co + lo;
      float y[3] = {0.f, 0.f, 0.f};
      const NewP<S> vec{a.z, pold, beta, first};
      const float* bv = bval + vo + 9 * lo;
      if constexpr (ALL) {
#pragma unroll 1
        for (int h = 0; h < min(n, 2); ++h) {
          float t[4][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
          add_parts<4>(h, n, [&](int e) { return bc[e]; }, bv, vec, t);
          add_half(t, y);
        }
      } else {
        const int held = n > PCG_WIDE ? 0 : n <= cap - lo ? n : max(0, cap - lo) & ~7;
        add_row<ONE ? 2 : 4>(a, RowAt{row, k0, n, held, bc, bv}, vec, y);
      }
      double pap_loc = 0.0;
      if (row < V) {
        float pv[3];
        if (ONE) {
          for (int e = 0; e < 3; ++e) { pv[e] = p[e] = first ? z[e] : axpy(beta, p[e], z[e]); q[e] = y[e]; }
        } else {
          typename NewP<S>::Raw own;
          vec.load(row, own);
          vec.value(own, pv);
          for (int e = 0; e < 3; ++e) a.Ap[3 * row + e] = y[e];
        }
        st4<S>(pnew, row, pv[0], pv[1], pv[2]);
        pap_loc = double(pv[0]) * y[0] + double(pv[1]) * y[1] + double(pv[2]) * y[2];
      }
      hand_over(pap_loc, 0.f, 0.f, 0.f);
    }
    reduce(2 + 2 * it, [&](bool ok, double pap, unsigned) { st.after_product(ok, pap); });
    if (st.status != PCG_MAXIT) break;
    const float alpha = st.coef;
    // ---- phase B: x, r, z, r^T z, |r|_inf
    begin();
    for (int j = w; j < sn; j += nw) {
      const int row = row_of(j);
      double rz_loc = 0.0;
      float rv[3] = {0.f, 0.f, 0.f}, zv[3];
      if (row < V) {
        if (ONE) {
          for (int e = 0; e < 3; ++e) {
            float& xe = KEEP ? x[e] : a.x[3 * row + e];
            xe = axpy(alpha, p[e], xe);
            rv[e] = r[e] = axpy(-alpha, q[e], r[e]);
          }
          if (!KEEP) load_P(row, Pm);
          apply_P(Pm, rv, zv);
          for (int e = 0; e < 3; ++e) z[e] = zv[e];
        } else {
          float m[9];
          load_P(row, m);
          const float4 pp = ld4<S>(pnew, row);
          const float pv[3] = {pp.x, pp.y, pp.z};
          for (int e = 0; e < 3; ++e) {
            a.x[3 * row + e] = axpy(alpha, pv[e], a.x[3 * row + e]);
            rv[e] = a.r[3 * row + e] = axpy(-alpha, a.Ap[3 * row + e], a.r[3 * row + e]);
          }
          apply_P(m, rv, zv);
        }
        st4<S>(a.z, row, zv[0], zv[1], zv[2]);
        rz_loc = double(rv[0]) * zv[0] + double(rv[1]) * zv[1] + double(rv[2]) * zv[2];
      }
      hand_over(rz_loc, rv[0], rv[1], rv[2]);
    }
    reduce(3 + 2 * it, [&](bool ok, double rz, unsigned mx) { st.after_update(ok, rz, mx, a.tol, 0); });
    if (st.status != PCG_MAXIT) break;
    beta = st.coef;
    first = false;
    float* t = pold; pold = pnew; pnew = t;
  }
  if (KEEP) {
    const int row = row_of(w);
    if (w < sn && row < V) for (int e = 0; e < 3; ++e) a.x[3 * row + e] = x[e];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) st.report(ctrl);
}

// At most WARPS to a CTA. Both copies of the loop are inlined: a call in the
// kernel costs the common one 4 us an iteration.
template <bool ONE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 1) k_pcg(const __grid_constant__ PcgArgs a) {
  if (a.ctrl->converged) return;
  __shared__ XrSmem sh;
  __shared__ PcgScalars st;
  const int ns = (a.V + 31) >> 5, spc = (ns + (int)gridDim.x - 1) / (int)gridDim.x, s0 = blockIdx.x * spc;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, cap = (((a.smem / nw) & ~15) - 64) / 40;
  bool rest = false;
  for (int j = threadIdx.x >> 5; j < min(spc, ns - s0); j += nw) {
    const int row = 32 * (s0 + j) + lane, first = a.rowptr[32 * (s0 + j)];
    if (row >= a.V) continue;
    const int k0 = a.rowptr[row], k1 = a.rowptr[row + 1];
    rest |= k1 - k0 > PCG_WIDE || k1 - first > cap || (a.xbegin && a.xend[row] > a.xbegin[row]);
  }
  if (__syncthreads_or(rest)) pcg_solve<ONE, false>(a, sh, st);
  else pcg_solve<ONE, true>(a, sh, st);
}

// The same solve for a small system, as one cluster of at most 16 CTAs with
// one row per thread (512 rows to a CTA): z and p are published in shared
// memory and read from the CTA that owns the row, so an iteration touches no
// global memory and its two barriers are the cluster's. A row's first PCG_KQ
// neighbours' p stay in registers (p_new_j = z_j + beta p_j is what the
// thread computed for them one iteration ago). 1,024 rows: 34.9 us per
// iteration with a warp per row and two grid barriers through L2.
constexpr int PCG_KQ = 8;   // one block in each of a row's eight parts

__device__ inline float4 cl_ld4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// p_new of a column from the CTA that owns it (handle: the address of its z);
// in the first iteration p_old is not there yet, and z is read for it with beta 0
struct ClusterP {
  unsigned z0; int rows; unsigned pold; float beta;
  struct Raw { float4 z, p; };
  __device__ unsigned handle(int col) const { const int c = col / rows; return cl_map(z0 + 16u * (col - c * rows), c); }
  __device__ unsigned held(int c) const { return (unsigned)c; }
  __device__ void load(unsigned at, Raw& r) const { r.z = cl_ld4(at); r.p = cl_ld4(at + pold); }
  __device__ void value(const Raw& r, float (&v)[3]) const {
    v[0] = axpy(beta, r.p.x, r.z.x); v[1] = axpy(beta, r.p.y, r.z.y); v[2] = axpy(beta, r.p.z, r.z.z);
  }
};

// ALL: the CTA's rows have at most PCG_KQ blocks, all in the buffers, and none elsewhere.
template <bool ALL>
__device__ __forceinline__ void pcg_solve_cluster(const PcgArgs& a, XrSmem& sh, PcgScalars& st) {
  extern __shared__ __align__(16) unsigned char pcg_dyn[];   // z, p, p' of the CTA's rows (float4), then each warp's matrix buffer
  const int V = a.V, rows = blockDim.x, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int row = blockIdx.x * rows + threadIdx.x;
  const bool live = row < V;
  float4* const pub = reinterpret_cast<float4*>(pcg_dyn);
  const unsigned pub0 = (unsigned)__cvta_generic_to_shared(pub);
  const unsigned array = 16u * rows;                         // bytes of one published vector: z, then the two p
  const int wbuf = ((a.smem - 48 * rows) / nw) & ~15, cap = (wbuf - 64) / 40;
  unsigned char* buf = pcg_dyn + 48 * rows + (size_t)w * wbuf;
  float* bval = reinterpret_cast<float*>(buf);
  int* bcol = reinterpret_cast<int*>(buf + ((36 * cap + 16 + 15) & ~15));
  auto handle = [&](int col) { const int c = col / rows; return cl_map(pub0 + 16u * (col - c * rows), c); };   // z of row col

  const int kb = live ? a.rowptr[row] : 0, n = live ? a.rowptr[row + 1] - kb : 0;
  const int k0 = __shfl_sync(0xffffffffu, kb, 0), nb = __reduce_max_sync(0xffffffffu, n > 0 ? kb + n - k0 : 0);
  const int vo = warp_copy_async(bval, a.val + 9ll * k0, 9 * min(nb, cap));
  const int co = warp_copy_async(bcol, a.cols + k0, min(nb, cap));
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  const int lo = kb - k0, held = ALL || n <= min(PCG_WIDE, cap - lo) ? n : n > PCG_WIDE ? 0 : max(0, cap - lo) & ~7;
  int* const bc = bcol + co + lo;
  const float* const bv = bval + vo + 9 * lo;
  for (int e = 0; e < held; ++e) bc[e] = (int)handle(bc[e]);   // columns -> addresses of their z

  float P[9], r[3] = {0.f, 0.f, 0.f}, z[3] = {0.f, 0.f, 0.f}, p[3] = {0.f, 0.f, 0.f}, x[3] = {0.f, 0.f, 0.f}, q[ALL ? PCG_KQ : 1][3];
  for (int e = 0; e < 9; ++e) P[e] = live ? a.P[9ll * row + e] : 0.f;
  for (int e = 0; e < (ALL ? PCG_KQ : 1); ++e) q[e][0] = q[e][1] = q[e][2] = 0.f;
  if (live) for (int e = 0; e < 3; ++e) r[e] = a.b[3 * row + e];
  auto put = [&](unsigned off, const float (&v)[3]) { *reinterpret_cast<float4*>(pcg_dyn + off + 16 * threadIdx.x) = make_float4(v[0], v[1], v[2], 0.f); };
  auto apply_P = [&]() {
    for (int c = 0; c < 3; ++c) z[c] = dot3(P[3 * c], P[3 * c + 1], P[3 * c + 2], r[0], r[1], r[2]);
    put(0, z);
    return double(r[0]) * z[0] + double(r[1]) * z[1] + double(r[2]) * z[2];
  };
  auto mag = [&]() { return max(xr_mag(r[0]), max(xr_mag(r[1]), xr_mag(r[2]))); };
  auto reduce = [&](unsigned epoch, double v, unsigned m, auto tail) {
    v = xr_warp_sum(v);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) { sh.part[w] = v; sh.pmax[w] = m; }
    cl_reduce(sh, nw, epoch, tail);
  };
  double rz0 = apply_P();
  reduce(1, rz0, mag(), [&](bool ok, double rz, unsigned mx) { st.start(ok, rz, mx, a.tol, false); });
  unsigned pold = array, pnew = 2 * array;
  float beta = 0.f;
  for (int it = 0; st.status == PCG_MAXIT && it < a.max_iters; ++it) {
    // ---- phase A: p_new = z + beta p_old, Ap = A p_new, p^T Ap
    float y[3] = {0.f, 0.f, 0.f};
    if constexpr (ALL) {
      float4 zz[PCG_KQ];
#pragma unroll
      for (int e = 0; e < PCG_KQ; ++e) if (e < n) zz[e] = cl_ld4((unsigned)bc[e]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float t[4][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = half_block(h, u);
          if (e < n) {
            q[e][0] = axpy(beta, q[e][0], zz[e].x); q[e][1] = axpy(beta, q[e][1], zz[e].y); q[e][2] = axpy(beta, q[e][2], zz[e].z);
            block_product(bv + 9 * e, q[e], t[u]);
          }
        }
        add_half(t, y);
      }
    } else {
      add_row<4>(a, RowAt{row, kb, n, held, bc, bv}, ClusterP{pub0, rows, it ? pold : 0u, it ? beta : 0.f}, y);
    }
    for (int e = 0; e < 3; ++e) p[e] = axpy(beta, p[e], z[e]);
    put(pnew, p);
    reduce(2 + 2 * it, double(p[0]) * y[0] + double(p[1]) * y[1] + double(p[2]) * y[2], 0u,
           [&](bool ok, double pap, unsigned) { st.after_product(ok, pap); });
    if (st.status != PCG_MAXIT) break;
    const float alpha = st.coef;
    // ---- phase B: x, r, z, r^T z, |r|_inf
    for (int e = 0; e < 3; ++e) { x[e] = axpy(alpha, p[e], x[e]); r[e] = axpy(-alpha, y[e], r[e]); }
    rz0 = apply_P();
    reduce(3 + 2 * it, rz0, mag(), [&](bool ok, double rz, unsigned mx) { st.after_update(ok, rz, mx, a.tol, 0); });
    if (st.status != PCG_MAXIT) break;
    beta = st.coef;
    const unsigned t = pold; pold = pnew; pnew = t;
  }
  if (live) for (int e = 0; e < 3; ++e) a.x[3 * row + e] = x[e];
  if (row == 0) st.report(a.ctrl);
  cl_sync_shared();   // the others have read this CTA's last partial
}

__global__ void __launch_bounds__(PCG_CLUSTER_TPB, 1) k_pcg_cluster(const __grid_constant__ PcgArgs a) {
  if (a.ctrl->converged) return;
  __shared__ XrSmem sh;
  __shared__ PcgScalars st;
  const int rows = blockDim.x, nw = rows >> 5, cap = ((((a.smem - 48 * rows) / nw) & ~15) - 64) / 40;
  const int row = blockIdx.x * rows + threadIdx.x;
  bool rest = false;
  if (row < a.V) {
    const int k0 = a.rowptr[row], k1 = a.rowptr[row + 1];
    rest = k1 - k0 > PCG_KQ || k1 - a.rowptr[row & ~31] > cap || (a.xbegin && a.xend[row] > a.xbegin[row]);
  }
  if (__syncthreads_or(rest)) pcg_solve_cluster<false>(a, sh, st);
  else pcg_solve_cluster<true>(a, sh, st);
}

// ------------------------------------------------------------ scaled PCG
// CG on the block-scaled system A^ = L^-1 A L^-T (A_ii = L_i L_i^T), used by
// the CORRECTED step. With the identity as preconditioner on A^ this is the
// block-Jacobi PCG of the reference, iterate for iterate in exact arithmetic:
// x = L^-T x^, r = L r^. The stopping test is relative like the reference's
// (pcg_solver.cpp:8-75) but taken on the block-scaled residual,
// max_i |r^_i| < tol * max_i |b^_i|: on the unscaled residual a few contact or
// pin rows whose forces are orders of magnitude above the rest set the
// tolerance for every other row, and the solve stops with a direction that is
// poor everywhere else. Scaled by L^-1, rows are compared in displacement-
// like units. The learned and block-Jacobi solves stop on the same test.
//
// LEARNED: z = S r with S a symmetric positive definite block matrix on the
// static pattern (the learned approximate inverse of A^), applied as
// S_ij = coef_ij A^_ij off the diagonal plus its diagonal blocks. Phase B then
// is a second row product over A^'s values; it gathers r - alpha Ap from the
// neighbours, so
// the iteration still needs only two grid barriers (r ping-pongs between two
// buffers because neighbours read the old values). r^T z <= 0 (S lost
// definiteness) or no new best residual for `stall_window` iterations ends
// the solve with PCG_PRECOND / PCG_STALL, and the caller redoes it with
// block-Jacobi.

// Sliced-ELL layout of the static pattern (SELL-32): rows in chunks of 32,
// chunk c holding W_c = (chunk_off[c+1] - chunk_off[c]) / 32 block slots per
// row; slot k of row lane l sits at block index chunk_off[c] + 32 k + l, its
// column in sell_col (-1 pads a short row) and its 9 values at
// 9 (chunk_off[c] + 32 k) + 32 q + l, q = 0..8. One thread per block row: a
// warp's 32 rows read every value and column load as one coalesced 128-byte
// line, and 32 rows' gathers are in flight at once (sell_row_u below).

// Row stride S of the scaled PCG's vectors r, r2, z, p0, p1 and Ap: 4 (one
// float4 per row, the fourth lane unused, so a neighbour's entry is one
// 16-byte load) in the block-Jacobi solve, 3 in the learned one, where the
// larger vectors measured slower (19.5 against 18.7 us per iteration at
// C4). Each solve initialises its vectors, so the two layouts share buffers
// of 4V floats.
template <int S> struct GatherP {  // p = z + beta p_old
  const float* z; const float* pold; float beta; bool first;
  __device__ void operator()(int j, float& q0, float& q1, float& q2) const {
    const float4 zz = ld4<S>(z, j);
    if (first) { q0 = zz.x; q1 = zz.y; q2 = zz.z; return; }
    const float4 pp = ld4<S>(pold, j);
    q0 = zz.x + beta * pp.x; q1 = zz.y + beta * pp.y; q2 = zz.z + beta * pp.z;
  }
};
struct GatherV {  // plain vector
  const float* v;
  __device__ void operator()(int j, float& q0, float& q1, float& q2) const { q0 = v[3 * j]; q1 = v[3 * j + 1]; q2 = v[3 * j + 2]; }
};
template <int S> struct GatherR {  // r - alpha Ap
  const float* r; const float* Ap; float alpha;
  __device__ void operator()(int j, float& q0, float& q1, float& q2) const {
    const float4 rr = ld4<S>(r, j), aa = ld4<S>(Ap, j);
    q0 = rr.x - alpha * aa.x; q1 = rr.y - alpha * aa.y; q2 = rr.z - alpha * aa.z;
  }
};

// Fixed-order reductions over per-slice partials. Each warp owns whole
// 32-row slices and writes one partial per slice (a xor butterfly, whose
// result is the same in every lane); after the grid barrier every CTA adds
// the partials in one order that does not depend on the launch shape:
// s_t = sum_k part[t + 1024 k] for t < 1024, then butterflies over 32 groups
// of 32. So the tuned launch shape never changes a result bit.
__device__ inline double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// the larger of two magnitudes, a NaN above all (fmax would drop it, and a
// residual that is NaN throughout would count as 0)
__device__ inline double mag_max(double a, double b) { return b > a || b != b ? b : a; }
__device__ inline double warp_max(double v) {
  for (int o = 16; o; o >>= 1) v = mag_max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
constexpr int RED_T = 1024;
struct RedSmem { double s[RED_T + 32]; double m[RED_T + 32]; };

// sum of part[0, n) and (with MAX) max of pm[0, n), identical in every CTA
template <bool MAX>
__device__ inline void fixed_reduce(const double* part, const double* pm, int n, RedSmem& sh, double& sum, double& mx) {
  for (int t = threadIdx.x; t < RED_T; t += blockDim.x) {
    double s = 0.0, m = 0.0;
    for (int k = t; k < n; k += RED_T) {
      s += __ldcg(part + k);  // written by other CTAs before the barrier: read from L2
      if (MAX) m = mag_max(m, __ldcg(pm + k));
    }
    sh.s[t] = s;
    if (MAX) sh.m[t] = m;
  }
  __syncthreads();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int g = w; g < 32; g += nw) {
    double v = warp_sum(sh.s[32 * g + l]);
    if (l == 0) sh.s[RED_T + g] = v;
    if (MAX) {
      double u = warp_max(sh.m[32 * g + l]);
      if (l == 0) sh.m[RED_T + g] = u;
    }
  }
  __syncthreads();
  sum = warp_sum(sh.s[RED_T + l]);
  mx = MAX ? warp_max(sh.m[RED_T + l]) : 0.0;
  __syncthreads();  // sh is reused by the next reduction
}

// a += H q for one 3x3 block (row-major, entries h(e) = h[e * stride]), with
// the FMA order written out so that every product variant rounds alike.
template <int STRIDE>
__device__ inline void block_fma(const float* h, float q0, float q1, float q2, float& a0, float& a1, float& a2) {
  a0 = __fmaf_rn(h[2 * STRIDE], q2, __fmaf_rn(h[1 * STRIDE], q1, __fmaf_rn(h[0], q0, a0)));
  a1 = __fmaf_rn(h[5 * STRIDE], q2, __fmaf_rn(h[4 * STRIDE], q1, __fmaf_rn(h[3 * STRIDE], q0, a1)));
  a2 = __fmaf_rn(h[8 * STRIDE], q2, __fmaf_rn(h[7 * STRIDE], q1, __fmaf_rn(h[6 * STRIDE], q0, a2)));
}

// One row of the SELL-32 product. U > 1 loads the column indices of U slots
// ahead of their gathers (more loads in flight per thread, more registers);
// the sum runs over k = 0, 1, ... with the same FMAs for every U.
template <int U, class Vec>
__device__ inline void sell_row_u(int row, const int* chunk_off, const int* sell_col, const float* val, const int* xbegin, const int* xend,
                                  const int* xcols, const float* xval, const Vec& vec, float& y0, float& y1, float& y2) {
  const int c = row >> 5, l = row & 31;
  const int b0 = chunk_off[c], w = (chunk_off[c + 1] - b0) >> 5;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f;
  if (U == 1) {
    for (int k = 0; k < w; ++k) {
      const int slot = b0 + 32 * k;
      const int col = sell_col[slot + l];
      if (col < 0) continue;
      float q0, q1, q2; vec(col, q0, q1, q2);
      block_fma<32>(val + 9ll * slot + l, q0, q1, q2, a0, a1, a2);
    }
  } else {
#pragma unroll 1
    for (int k = 0; k < w; k += U) {
      int col[U];
#pragma unroll
      for (int u = 0; u < U; ++u) col[u] = k + u < w ? sell_col[b0 + 32 * (k + u) + l] : -1;
      float q[U][3];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (col[u] >= 0) vec(col[u], q[u][0], q[u][1], q[u][2]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (col[u] >= 0) block_fma<32>(val + 9ll * (b0 + 32 * (k + u)) + l, q[u][0], q[u][1], q[u][2], a0, a1, a2);
    }
  }
  if (xbegin) {
    for (int e = xbegin[row]; e < xend[row]; ++e) {
      float q0, q1, q2; vec(xcols[e], q0, q1, q2);
      block_fma<1>(xval + 9ll * e, q0, q1, q2, a0, a1, a2);
    }
  }
  y0 = a0; y1 = a1; y2 = a2;
}

// One row of z = S g with S_ij = coef_ij A^_ij off the diagonal and S_ii =
// Sdiag_i: the SELL-32 product over A^'s static slots (the values phase A
// has just read) with each gathered g_j scaled by its slot's coefficient,
// the row's own slot skipped, then the diagonal block. The same FMA order
// for every U.
template <int U, class Vec>
__device__ inline void sell_row_S(int row, const int* chunk_off, const int* sell_col, const float* val, const float* coef, const float* Sdiag,
                                  const Vec& vec, float& y0, float& y1, float& y2) {
  const int c = row >> 5, l = row & 31;
  const int b0 = chunk_off[c], w = (chunk_off[c + 1] - b0) >> 5;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f;
  if (U == 1) {
    for (int k = 0; k < w; ++k) {
      const int slot = b0 + 32 * k;
      const int col = sell_col[slot + l];
      if (col < 0 || col == row) continue;
      const float cf = coef[slot + l];
      float q0, q1, q2; vec(col, q0, q1, q2);
      block_fma<32>(val + 9ll * slot + l, cf * q0, cf * q1, cf * q2, a0, a1, a2);
    }
  } else {
#pragma unroll 1
    for (int k = 0; k < w; k += U) {
      int col[U];
      float cf[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        col[u] = k + u < w ? sell_col[b0 + 32 * (k + u) + l] : -1;
        if (col[u] == row) col[u] = -1;
        cf[u] = col[u] >= 0 ? coef[b0 + 32 * (k + u) + l] : 0.f;
      }
      float q[U][3];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (col[u] >= 0) vec(col[u], q[u][0], q[u][1], q[u][2]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (col[u] >= 0) block_fma<32>(val + 9ll * (b0 + 32 * (k + u)) + l, cf[u] * q[u][0], cf[u] * q[u][1], cf[u] * q[u][2], a0, a1, a2);
    }
  }
  float g0, g1, g2; vec(row, g0, g1, g2);
  block_fma<32>(Sdiag + 288ll * (row >> 5) + (row & 31), g0, g1, g2, a0, a1, a2);
  y0 = a0; y1 = a1; y2 = a2;
}

constexpr int SCALED_MAX_TPB = 1024;

template <bool LEARNED, int U>
__global__ void __launch_bounds__(SCALED_MAX_TPB) k_pcg_scaled(PcgScaledArgs a) {
  Ctrl* ctrl = a.ctrl;
  if (ctrl->converged) return;
  if (!LEARNED && a.fallback) {
    // every CTA reads the learned solve's status before the first grid
    // barrier; it is rewritten only after one
    const int st = ctrl->pcg_status;
    if (st == PCG_OK || st == PCG_TIMEOUT) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->fallback_ran = 1;
  }
  __shared__ RedSmem sh;
  constexpr int S = LEARNED ? 3 : 4;  // row stride of r, z, p, Ap
  const int V = a.V, ns = (V + 31) >> 5;
  const unsigned nb = gridDim.x;
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, W = (gridDim.x * blockDim.x) >> 5;
  double* part_pap = a.partials;
  double* part_rz = a.partials + ns;
  double* part_rinf = a.partials + 2 * ns;
  float* r = a.r;
  float* rn = a.r2;
  const float* zsrc = LEARNED ? a.z : a.r;
  double dummy;
  unsigned int epoch = 0;  // grid barriers passed (the launcher zeroes the arrival counter)

  // init: x^ = 0, r = b^, z = S b^, max |b^|
  for (int sl = gw; sl < ns; sl += W) {
    const int i = 32 * sl + lane;
    double rz_loc = 0.0, binf_loc = 0.0;
    if (i < V) {
      float b0 = a.bhat[3 * i], b1 = a.bhat[3 * i + 1], b2 = a.bhat[3 * i + 2];
      binf_loc = mag_max(fabs(double(b0)), mag_max(fabs(double(b1)), fabs(double(b2))));
      a.xh[3 * i] = 0.0; a.xh[3 * i + 1] = 0.0; a.xh[3 * i + 2] = 0.0;
      st4<S>(r, i, b0, b1, b2);
      if (LEARNED) {
        float y0, y1, y2;
        sell_row_S<U>(i, a.chunk_off, a.sell_col, a.valh, a.coef, a.Sdiag, GatherV{a.bhat}, y0, y1, y2);
        st4<S>(a.z, i, y0, y1, y2);
        rz_loc = double(b0) * y0 + double(b1) * y1 + double(b2) * y2;
      } else {
        rz_loc = double(b0) * b0 + double(b1) * b1 + double(b2) * b2;
        if (a.snap_r && a.snap_max > 0) {
          a.snap_r[3 * i] = b0; a.snap_r[3 * i + 1] = b1; a.snap_r[3 * i + 2] = b2;
          a.snap_x[3 * i] = 0.0; a.snap_x[3 * i + 1] = 0.0; a.snap_x[3 * i + 2] = 0.0;
        }
      }
    }
    rz_loc = warp_sum(rz_loc);
    binf_loc = warp_max(binf_loc);
    if (lane == 0) { part_rz[sl] = rz_loc; part_rinf[sl] = binf_loc; }
  }
  bool ok = grid_sync_ar(&ctrl->bar_arrivals, nb, epoch, &ctrl->bar_err);
  int status = PCG_MAXIT, iters = 0;
  double rel = 0.0, rz = 0.0, binf = 0.0;
  if (!ok) status = PCG_TIMEOUT;
  else fixed_reduce<true>(part_rz, part_rinf, ns, sh, rz, binf);
  if (ok) {
    rel = binf < 1e-16 ? binf : 1.0;
    if (!(binf <= FLT_MAX)) status = PCG_NOT_SPD;
    else if (rel < double(a.tol)) status = PCG_OK;
    else if (LEARNED && !(rz > 0.0)) status = PCG_PRECOND;
  }
  float* pold = a.p0;
  float* pnew = a.p1;
  float beta = 0.f;
  bool first = true;
  double best = rel;
  int since = 0;
  for (int it = 0; ok && status == PCG_MAXIT && it < a.max_iters; ++it) {
    // ---- phase A: p_new = z + beta p_old, Ap = A^ p_new, p^T Ap
    GatherP<S> gp{zsrc, pold, beta, first};
    for (int sl = gw; sl < ns; sl += W) {
      const int row = 32 * sl + lane;
      double pap_loc = 0.0;
      if (row < V) {
        float y0, y1, y2;
        sell_row_u<U>(row, a.chunk_off, a.sell_col, a.valh, a.xbegin, a.xend, a.xcols, a.xvalh, gp, y0, y1, y2);
        float q0, q1, q2; gp(row, q0, q1, q2);
        st4<S>(pnew, row, q0, q1, q2);
        st4<S>(a.Ap, row, y0, y1, y2);
        pap_loc = double(q0) * y0 + double(q1) * y1 + double(q2) * y2;
      }
      pap_loc = warp_sum(pap_loc);
      if (lane == 0) part_pap[sl] = pap_loc;
    }
    ok = grid_sync_ar(&ctrl->bar_arrivals, nb, epoch, &ctrl->bar_err);
    if (!ok) { status = PCG_TIMEOUT; break; }
    double pap;
    fixed_reduce<false>(part_pap, nullptr, ns, sh, pap, dummy);
    iters = it + 1;
    if (!(fabs(pap) >= 1e-16)) { status = PCG_NOT_SPD; break; }   // a NaN too
    float alpha = float(rz / pap);
    // ---- phase B: x^ += alpha p, r -= alpha Ap, z = S r, r^T z, |L r|_inf
    if (!LEARNED) {
      // snapshot k of (r^, x^) after 2^k - 1 iterations (training probes)
      const int done = it + 1;
      const int snap = (a.snap_r && ((done & (done + 1)) == 0)) ? __ffs(done + 1) - 1 : -1;
      float* sr = (snap >= 0 && snap < a.snap_max) ? a.snap_r + 3ll * V * snap : nullptr;
      double* sx = sr ? a.snap_x + 3ll * V * snap : nullptr;
      for (int sl = gw; sl < ns; sl += W) {
        const int i = 32 * sl + lane;
        double rz_new_loc = 0.0, rinf_loc = 0.0;
        if (i < V) {
          const float4 pv = ld4<S>(pnew, i), rv = ld4<S>(r, i), av = ld4<S>(a.Ap, i);
          const float p0 = pv.x, p1 = pv.y, p2 = pv.z;
          a.xh[3 * i] += double(alpha) * p0; a.xh[3 * i + 1] += double(alpha) * p1; a.xh[3 * i + 2] += double(alpha) * p2;
          float r0 = rv.x - alpha * av.x, r1 = rv.y - alpha * av.y, r2 = rv.z - alpha * av.z;
          st4<S>(r, i, r0, r1, r2);
          if (sr) {
            sr[3 * i] = r0; sr[3 * i + 1] = r1; sr[3 * i + 2] = r2;
            sx[3 * i] = a.xh[3 * i]; sx[3 * i + 1] = a.xh[3 * i + 1]; sx[3 * i + 2] = a.xh[3 * i + 2];
          }
          rz_new_loc = double(r0) * r0 + double(r1) * r1 + double(r2) * r2;
          rinf_loc = mag_max(fabs(double(r0)), mag_max(fabs(double(r1)), fabs(double(r2))));
        }
        rz_new_loc = warp_sum(rz_new_loc);
        rinf_loc = warp_max(rinf_loc);
        if (lane == 0) { part_rz[sl] = rz_new_loc; part_rinf[sl] = rinf_loc; }
      }
    } else {
      GatherR<S> gr{r, a.Ap, alpha};
      for (int sl = gw; sl < ns; sl += W) {
        const int row = 32 * sl + lane;
        double rz_new_loc = 0.0, rinf_loc = 0.0;
        if (row < V) {
          float y0, y1, y2;
          sell_row_S<U>(row, a.chunk_off, a.sell_col, a.valh, a.coef, a.Sdiag, gr, y0, y1, y2);
          float r0, r1, r2; gr(row, r0, r1, r2);
          const float4 pv = ld4<S>(pnew, row);
          a.xh[3 * row] += double(alpha) * pv.x; a.xh[3 * row + 1] += double(alpha) * pv.y;
          a.xh[3 * row + 2] += double(alpha) * pv.z;
          st4<S>(rn, row, r0, r1, r2);
          st4<S>(a.z, row, y0, y1, y2);
          rz_new_loc = double(r0) * y0 + double(r1) * y1 + double(r2) * y2;
          rinf_loc = mag_max(fabs(double(r0)), mag_max(fabs(double(r1)), fabs(double(r2))));
        }
        rz_new_loc = warp_sum(rz_new_loc);
        rinf_loc = warp_max(rinf_loc);
        if (lane == 0) { part_rz[sl] = rz_new_loc; part_rinf[sl] = rinf_loc; }
      }
    }
    ok = grid_sync_ar(&ctrl->bar_arrivals, nb, epoch, &ctrl->bar_err);
    if (!ok) { status = PCG_TIMEOUT; break; }
    double rz_new, rinf;
    fixed_reduce<true>(part_rz, part_rinf, ns, sh, rz_new, rinf);
    rel = binf < 1e-16 ? rinf : rinf / binf;
    if (LEARNED) { float* t = r; r = rn; rn = t; }
    if (!(rinf <= FLT_MAX)) { status = PCG_NOT_SPD; break; }
    if (rel < double(a.tol)) { status = PCG_OK; break; }
    if (LEARNED) {
      if (!(rz_new > 0.0)) { status = PCG_PRECOND; break; }
      if (rel < best) { best = rel; since = 0; }
      else if (++since >= a.stall_window) { status = PCG_STALL; break; }
    }
    beta = float(rz_new / rz);
    rz = rz_new;
    first = false;
    float* t = pold; pold = pnew; pnew = t;
  }
  // d = L^-T x^ (every x^ write precedes the last grid barrier); x^ is FP64:
  // rounding it to FP32 would cost up to cond(L_i) x 6e-8 of d_i at stiff vertices
  if (ok) {
    for (int sl = gw; sl < ns; sl += W) {
      const int i = 32 * sl + lane;
      if (i >= V) continue;
      const double* q = a.Linv + 6 * (long long)i;
      double x0 = a.xh[3 * i], x1 = a.xh[3 * i + 1], x2 = a.xh[3 * i + 2];
      a.d[3 * i] = float(q[0] * x0 + q[1] * x1 + q[3] * x2);
      a.d[3 * i + 1] = float(q[2] * x1 + q[4] * x2);
      a.d[3 * i + 2] = float(q[5] * x2);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (LEARNED) ctrl->learned_iters = iters;
    ctrl->pcg_iters = iters;
    ctrl->pcg_status = status;
    ctrl->pcg_converged = status == PCG_OK ? 1 : 0;
    ctrl->pcg_rel = rel;
  }
}

// ------------------------------------------- scaled PCG, resident form
// The same solve, bit for bit in its vectors, for meshes of at most one row
// per thread of the GPU (1,024 rows per CTA, one CTA on each SM): each warp
// owns one 32-row slice, one thread per row, for the whole solve.
//  - r^, p, A^ p and x^ of a row are registers; r^ (learned: z, r^ and A^ p)
//    is published as float4 rows for the neighbours' products.
//  - With KQ > 0 the neighbours' p of a row's first KQ slots stay in registers
//    too: p_new_j = z_j + beta p_j is what the thread computed for column j
//    one iteration ago, so a product gathers one vector instead of two. The
//    shapes whose registers do not hold them (KQ = 0) publish p as well.
//  - A^ is constant over the solve, so a slice's blocks are copied into shared
//    memory once, in the SELL-32 order (9 planes of 32 lanes: no bank
//    conflicts). A row's own block is exactly I unless its factorisation was
//    shifted, so in CTAs of more than 512 threads it takes no space: a
//    curtain's 6 remaining blocks at 886 rows per SM just fit. FAR: meshes with
//    wider rows and systems with contact blocks; slots past the capacity
//    (`slots` per row) are read from L2.
//  - The barrier of each dot product carries the sum: one partial per CTA
//    through L2 (xr_reduce), or, for systems of at most 16,384 rows, one
//    cluster whose CTAs publish everything through shared memory (cl_reduce).
// Contact blocks come in a SELL-32 copy of their own (xs_*), so a warp reads
// them as whole lines; without one (rows of very uneven contact counts) they
// are walked row by row.
constexpr int RES_KQ = PCG_NEAR_SLOTS;
constexpr int RES_SMEM = 224 * 1024;   // dynamic shared memory of a CTA, at most
constexpr int RES_CLUSTER_SLOTS = 72;  // slots of a slice of the cluster form, at most (res_layout)
// float4 vectors that a CTA of the cluster form publishes in shared memory
constexpr int res_vectors(bool learned, bool far, int kq) { return (learned ? 4 : 1) + (far || kq == 0 ? 2 : 0); }
// CTAs of more than 512 threads have no room for the rows' own blocks
constexpr bool res_compact(bool far, int max_threads) { return !far && max_threads > 512; }
inline int res_warp_bytes(int slots) { return slots * 1152 + (slots + 1) * 128; }

template <bool LEARNED, bool FAR, bool CLUSTER, int KQ, int NB, int U, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_pcg_res(const __grid_constant__ PcgScaledArgs a) {
  Ctrl* const ctrl = a.ctrl;
  if (ctrl->converged) return;
  if (!LEARNED && a.fallback) {
    // every CTA reads the learned solve's status before the first barrier; it
    // is rewritten only after one
    const int st = ctrl->pcg_status;
    if (st == PCG_OK || st == PCG_TIMEOUT) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->fallback_ran = 1;
  }
  constexpr bool COMPACT = res_compact(FAR, MAXT);
  constexpr int PUB = CLUSTER ? res_vectors(LEARNED, FAR, KQ) : 0;
  constexpr bool PUB_P = FAR || KQ == 0;
  extern __shared__ __align__(16) float res_dyn[];   // cluster form: the published vectors; then each warp's blocks and columns
  __shared__ XrSmem sh;
  __shared__ PcgScalars st;
  const int V = a.V, ns = (V + 31) >> 5, nw = blockDim.x >> 5, rows = blockDim.x;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sn = max(0, min(nw, ns - (int)blockIdx.x * nw));   // slices of this CTA
  const int slice = blockIdx.x * nw + w, row = 32 * slice + lane;
  const bool own = w < sn, live = own && row < V;
  const int Kc = a.slots;
  float* const sm = res_dyn + 4 * PUB * rows + w * (Kc * 288 + (Kc + 1) * 32) + lane;   // the lane's entries of the warp's blocks
  int* const smc = reinterpret_cast<int*>(sm + Kc * 288);                                // and columns

  // Published vectors: global float4 rows, or this CTA's shared memory. A
  // column's handle is its row, or the address of its row's first vector in
  // the CTA that owns it; -1: padding.
  using Vec = std::conditional_t<CLUSTER, unsigned, float*>;
  const unsigned pub0 = (unsigned)__cvta_generic_to_shared(res_dyn), array = 16u * rows;
  auto vec_z = [&]() -> Vec { if constexpr (CLUSTER) return 0u; else return LEARNED ? a.z : a.r; };
  auto vec_r = [&](int odd) -> Vec { if constexpr (CLUSTER) return (odd ? 2u : 1u) * array; else return odd ? a.r2 : a.r; };
  auto vec_ap = [&]() -> Vec { if constexpr (CLUSTER) return 3u * array; else return a.Ap; };
  auto vec_p = [&](int odd) -> Vec { if constexpr (CLUSTER) return ((LEARNED ? 4u : 1u) + (odd ? 1u : 0u)) * array; else return odd ? a.p1 : a.p0; };
  auto get = [&](Vec v, int h) -> float4 {
    if constexpr (CLUSTER) return cl_ld4((unsigned)h + v);
    else return ld4<4>(v, h);
  };
  auto put = [&](Vec v, const float (&f)[3]) {
    if constexpr (CLUSTER) *reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(res_dyn) + v + 16 * threadIdx.x) = make_float4(f[0], f[1], f[2], 0.f);
    else if (live) st4<4>(v, row, f[0], f[1], f[2]);
  };
  auto handle = [&](int col) -> int {
    if constexpr (CLUSTER) {
      if (col < 0) return -1;
      const int c = col / rows;
      return (int)cl_map(pub0 + 16u * (col - c * rows), c);
    } else return col;
  };

  // The slice's columns and blocks: static slots, then contact blocks. In the
  // compact layout the row's own block (slot kd) takes no place and the blocks
  // after it move up one.
  const int b0 = own ? a.chunk_off[slice] : 0, wd = own ? (a.chunk_off[slice + 1] - b0) >> 5 : 0;
  const int xb0 = FAR && own && a.xs_off ? a.xs_off[slice] : 0, xw = FAR && own && a.xs_off ? (a.xs_off[slice + 1] - xb0) >> 5 : 0;
  const int nk = wd + xw, own_h = handle(min(row, V - 1));   // a row past the end reads the last one's vectors, unused
  const float* const gv = a.valh + 9ll * b0 + lane;   // slot k: 288 k floats on
  auto global_block = [&](int k) -> const float* {
    return !FAR || k < wd ? gv + 288 * k : a.xs_val + 9ll * (xb0 + 32 * (k - wd)) + lane;
  };
  auto global_col = [&](int k) { return handle(!FAR || k < wd ? a.sell_col[b0 + 32 * k + lane] : a.xs_col[xb0 + 32 * (k - wd) + lane]); };
  int kd = 1 << 20;
  bool ident = true;
  for (int k = 0; k < min(nk, Kc + 1); ++k) {
    const int h = global_col(k);
    smc[32 * k] = h;
    if (COMPACT && h == own_h) kd = k;
  }
  for (int k = 0; k < min(nk, Kc + 1); ++k) {
    const float* g = global_block(k);
    const int t = COMPACT ? k - (k > kd) : k;
    if (COMPACT && k == kd) { for (int e = 0; e < 9; ++e) ident = ident && g[32 * e] == ((e & 3) == 0 ? 1.f : 0.f); }
    else if (t < Kc) for (int e = 0; e < 9; ++e) sm[288 * t + 32 * e] = g[32 * e];
  }
  // h = block k (on chip), entries of a lane without that slot undefined
  auto near_block = [&](int k, float (&h)[9]) {
    const float* s = sm + 288 * min(COMPACT ? k - (k > kd) : k, Kc - 1);
#pragma unroll
    for (int e = 0; e < 9; ++e) h[e] = s[32 * e];
    if (COMPACT && k == kd) {
      if (ident) { for (int e = 0; e < 9; ++e) h[e] = (e & 3) == 0 ? 1.f : 0.f; }
      else { for (int e = 0; e < 9; ++e) h[e] = gv[288 * k + 32 * e]; }
    }
  };
  auto fma9 = [&](const float (&h)[9], float q0, float q1, float q2, float (&y)[3]) { block_fma<1>(h, q0, q1, q2, y[0], y[1], y[2]); };
  auto reduce = [&](unsigned epoch, double v, float m0, float m1, float m2, auto tail) {
    v = xr_warp_sum(v);
    const unsigned m = __reduce_max_sync(0xffffffffu, max(xr_mag(m0), max(xr_mag(m1), xr_mag(m2))));
    if (lane == 0 && own) { sh.part[w] = v; sh.pmax[w] = m; }
    if constexpr (CLUSTER) cl_reduce(sh, sn, epoch, tail);
    else xr_reduce(sh, sn, epoch, a.slots_red, &ctrl->bar_arrivals, &ctrl->bar_err, tail);
  };

  // init: x^ = 0, r = b^, z = S b^, max |b^|
  float r[3] = {0.f, 0.f, 0.f}, z[3] = {0.f, 0.f, 0.f}, p[3] = {0.f, 0.f, 0.f}, q[KQ > 0 ? KQ : 1][3];
  double x[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < KQ; ++k) q[k][0] = q[k][1] = q[k][2] = 0.f;
  if (live) for (int e = 0; e < 3; ++e) r[e] = a.bhat[3 * row + e];
  if (LEARNED) {
    for (int k = 0; k < wd; ++k) {
      const int c = a.sell_col[b0 + 32 * k + lane];
      if (c < 0 || c == row) continue;
      const float cf = a.coef[b0 + 32 * k + lane];
      block_fma<32>(gv + 288 * k, cf * a.bhat[3 * c], cf * a.bhat[3 * c + 1], cf * a.bhat[3 * c + 2], z[0], z[1], z[2]);
    }
    if (live) block_fma<32>(a.Sdiag + 288ll * slice + lane, r[0], r[1], r[2], z[0], z[1], z[2]);
    put(vec_r(0), r);
  } else {
    for (int e = 0; e < 3; ++e) z[e] = r[e];
    if (live && a.snap_r && a.snap_max > 0)
      for (int e = 0; e < 3; ++e) { a.snap_r[3 * row + e] = r[e]; a.snap_x[3 * row + e] = 0.0; }
  }
  put(vec_z(), z);
  reduce(1, double(r[0]) * z[0] + double(r[1]) * z[1] + double(r[2]) * z[2], r[0], r[1], r[2],
         [&](bool ok, double rz, unsigned mx) { st.start(ok, rz, mx, a.tol, LEARNED); });
  float beta = 0.f;
  int it = 0;
  for (; st.status == PCG_MAXIT && it < a.max_iters; ++it) {
    // ---- phase A: p_new = z + beta p_old, Ap = A^ p_new, p^T Ap
    float y[3] = {0.f, 0.f, 0.f};
    // slots whose neighbours' p the thread keeps. Loads are unconditional (a
    // lane without the slot reads its own row), so a batch's are all in flight
    // together; only the products are predicated.
#pragma unroll
    for (int k0 = 0; k0 < KQ; k0 += NB) {
      if (k0 >= nk) break;
      int c[NB];
      float4 zz[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k0 + u < KQ) {
          c[u] = k0 + u < nk ? (!FAR || k0 + u <= Kc ? smc[32 * (k0 + u)] : global_col(k0 + u)) : -1;
          zz[u] = get(vec_z(), c[u] != -1 ? c[u] : own_h);
        }
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k0 + u < KQ) {
          float (&qk)[3] = q[KQ > 0 ? k0 + u : 0];
          qk[0] = zz[u].x + beta * qk[0]; qk[1] = zz[u].y + beta * qk[1]; qk[2] = zz[u].z + beta * qk[2];
          float h[9];
          if (!FAR || k0 + u < Kc) near_block(k0 + u, h);
          else if (k0 + u < nk) for (int e = 0; e < 9; ++e) h[e] = global_block(k0 + u)[32 * e];
          if (c[u] != -1) fma9(h, qk[0], qk[1], qk[2], y);
        }
    }
    if (PUB_P) {   // further slots: both vectors gathered
      const Vec pold = vec_p(it & 1);
#pragma unroll 1
      for (int k0 = KQ; k0 < nk; k0 += U) {
        int c[U];
        float4 zz[U], pp[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          c[u] = k0 + u < nk ? (!FAR || k0 + u <= Kc ? smc[32 * (k0 + u)] : global_col(k0 + u)) : -1;
          const int at = c[u] != -1 ? c[u] : own_h;
          zz[u] = get(vec_z(), at);
          pp[u] = it ? get(pold, at) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float h[9];
          if (!FAR || k0 + u < Kc) near_block(min(k0 + u, nk - 1), h);
          else if (k0 + u < nk) for (int e = 0; e < 9; ++e) h[e] = global_block(k0 + u)[32 * e];
          if (c[u] != -1) fma9(h, zz[u].x + beta * pp[u].x, zz[u].y + beta * pp[u].y, zz[u].z + beta * pp[u].z, y);
        }
      }
      if (FAR && a.xbegin && !a.xs_off && live)
        for (int e = a.xbegin[row]; e < a.xend[row]; ++e) {
          const int c = handle(a.xcols[e]);
          const float4 zf = get(vec_z(), c), pf = it ? get(pold, c) : make_float4(0.f, 0.f, 0.f, 0.f);
          block_fma<1>(a.xvalh + 9ll * e, zf.x + beta * pf.x, zf.y + beta * pf.y, zf.z + beta * pf.z, y[0], y[1], y[2]);
        }
    }
    for (int e = 0; e < 3; ++e) p[e] = z[e] + beta * p[e];
    if (PUB_P) put(vec_p(~it & 1), p);
    if (LEARNED) put(vec_ap(), y);
    reduce(2 + 2 * it, double(p[0]) * y[0] + double(p[1]) * y[1] + double(p[2]) * y[2], 0.f, 0.f, 0.f,
           [&](bool ok, double pap, unsigned) { st.after_product(ok, pap); });
    if (st.status != PCG_MAXIT) break;
    const float alpha = st.coef;
    // ---- phase B: x^ += alpha p, r -= alpha Ap, z = S r, r^T z, |r|_inf
    for (int e = 0; e < 3; ++e) { x[e] += double(alpha) * p[e]; r[e] = r[e] - alpha * y[e]; }
    if (LEARNED) {
      z[0] = z[1] = z[2] = 0.f;
#pragma unroll 1
      for (int k0 = 0; k0 < wd; k0 += U) {
        int c[U];
        float cf[U];
        float4 rr[U], aa[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          c[u] = k0 + u < wd ? (!FAR || k0 + u <= Kc ? smc[32 * (k0 + u)] : global_col(k0 + u)) : -1;
          if (c[u] == own_h) c[u] = -1;
          const int at = c[u] != -1 ? c[u] : own_h;
          cf[u] = c[u] != -1 ? a.coef[b0 + 32 * (k0 + u) + lane] : 0.f;
          rr[u] = get(vec_r(it & 1), at);
          aa[u] = get(vec_ap(), at);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float h[9];
          if (!FAR || k0 + u < Kc) near_block(min(k0 + u, wd - 1), h);
          else if (k0 + u < wd) for (int e = 0; e < 9; ++e) h[e] = gv[288 * (k0 + u) + 32 * e];
          const float g0 = rr[u].x - alpha * aa[u].x, g1 = rr[u].y - alpha * aa[u].y, g2 = rr[u].z - alpha * aa[u].z;
          if (c[u] != -1) fma9(h, cf[u] * g0, cf[u] * g1, cf[u] * g2, z);
        }
      }
      if (live) block_fma<32>(a.Sdiag + 288ll * slice + lane, r[0], r[1], r[2], z[0], z[1], z[2]);
      put(vec_r(~it & 1), r);   // neighbours still read the old r
    } else {
      for (int e = 0; e < 3; ++e) z[e] = r[e];
      if (live && a.snap_r) {
        // snapshot k of (r^, x^) after 2^k - 1 iterations (training probes)
        const int done = it + 1, snap = (done & (done + 1)) == 0 ? __ffs(done + 1) - 1 : -1;
        if (snap >= 0 && snap < a.snap_max)
          for (int e = 0; e < 3; ++e) {
            a.snap_r[3ll * V * snap + 3 * row + e] = r[e];
            a.snap_x[3ll * V * snap + 3 * row + e] = x[e];
          }
      }
    }
    put(vec_z(), z);
    reduce(3 + 2 * it, double(r[0]) * z[0] + double(r[1]) * z[1] + double(r[2]) * z[2], r[0], r[1], r[2],
           [&](bool ok, double rz, unsigned mx) { st.after_update(ok, rz, mx, a.tol, LEARNED ? a.stall_window : 0); });
    if (st.status != PCG_MAXIT) break;
    beta = st.coef;
  }
  // d = L^-T x^; x^ is FP64: rounding it to FP32 would cost up to cond(L_i) x
  // 6e-8 of d_i at stiff vertices
  if (live) {
    for (int e = 0; e < 3; ++e) a.xh[3 * row + e] = x[e];
    if (st.status != PCG_TIMEOUT) {
      const double* l = a.Linv + 6 * (long long)row;
      a.d[3 * row] = float(l[0] * x[0] + l[1] * x[1] + l[3] * x[2]);
      a.d[3 * row + 1] = float(l[2] * x[1] + l[4] * x[2]);
      a.d[3 * row + 2] = float(l[5] * x[2]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (LEARNED) ctrl->learned_iters = st.iters;
    st.report(ctrl);
  }
  if constexpr (CLUSTER) cl_sync_shared();   // the others have read this CTA's last partial
}

using ScaledKernel = void (*)(PcgScaledArgs);
ScaledKernel scaled_kernel(bool learned, int unroll) {
  if (learned) return unroll >= 2 ? k_pcg_scaled<true, 2> : k_pcg_scaled<true, 1>;
  return unroll >= 2 ? k_pcg_scaled<false, 2> : k_pcg_scaled<false, 1>;
}

}  // namespace

size_t pcg_scaled_partials(int V) { return 3ull * (size_t)((V + 31) / 32 + 1); }

namespace {
using PcgKernel = void (*)(PcgArgs);
PcgKernel pcg_kernel(bool one, int warps) {
  if (!one) return k_pcg<false, PCG_WARPS_MANY>;
  return warps <= PCG_WARPS_MANY ? k_pcg<true, PCG_WARPS_MANY> : k_pcg<true, PCG_WARPS>;
}

// Resident kernel of a shape: threads per CTA rounded up to a compiled bound,
// and with it the registers, which decide how many neighbours' p are kept
// and how many slots are gathered at once.
struct ResKernel { const void* f; int kq; bool compact; };
template <bool L, bool F, bool C> ResKernel res_pick(int tpb) {
  constexpr int KW = F ? 24 : RES_KQ;   // 256 threads leave registers for contact blocks' neighbours as well
  // a grid's CTAs have 16 slices without contact blocks (fewer only where no cluster can be had)
  if constexpr (F || C) if (tpb <= 256) return {(const void*)k_pcg_res<L, F, C, KW, F ? 8 : RES_KQ, 4, 256>, KW, res_compact(F, 256)};
  // a cluster's CTAs have at most 16 slices, with contact blocks 4
  if constexpr (!(F && C)) if (tpb <= 512) return {(const void*)k_pcg_res<L, F, C, RES_KQ, 4, L ? 3 : 4, 512>, RES_KQ, res_compact(F, 512)};
  if constexpr (!C) {
    if constexpr (!F) if (tpb <= 896) return {(const void*)k_pcg_res<L, F, C, L ? 0 : RES_KQ, 4, L ? 2 : 3, 896>, L ? 0 : RES_KQ, res_compact(F, 896)};
    return {(const void*)k_pcg_res<L, F, C, 0, 1, 2, 1024>, 0, res_compact(F, 1024)};
  }
  return {nullptr, 0, false};
}
ResKernel res_kernel(bool learned, bool far, bool cluster, int tpb) {
  if (cluster) {
    if (learned) return far ? res_pick<true, true, true>(tpb) : res_pick<true, false, true>(tpb);
    return far ? res_pick<false, true, true>(tpb) : res_pick<false, false, true>(tpb);
  }
  if (learned) return far ? res_pick<true, true, false>(tpb) : res_pick<true, false, false>(tpb);
  return far ? res_pick<false, true, false>(tpb) : res_pick<false, false, false>(tpb);
}

// Shared-memory and cluster attributes of a kernel, set on its first launch on
// a device: setting them loads the kernel, and a process uses few of them.
// Host-side calls only, so a first launch may be under stream capture.
cudaError_t kernel_ready(const void* f, int smem, bool cluster) {
  static std::mutex mu;
  static std::vector<std::pair<int, const void*>> ready;
  int d = 0;
  cudaGetDevice(&d);
  std::lock_guard<std::mutex> lock(mu);
  for (const auto& r : ready) if (r.first == d && r.second == f) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (!e && cluster) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (!e) ready.push_back({d, f});
  return e;
}

// SMs of the current device, and whether a cluster of 16 CTAs of the cluster
// kernels' size (one to an SM) can run on it.
struct PcgDevice { int sms = 0; bool cluster = false; };
PcgDevice pcg_device() {
  static std::mutex mu;
  static PcgDevice dev[64];
  int d = 0, sms = 0, n = 0;
  cudaGetDevice(&d);
  std::lock_guard<std::mutex> lock(mu);
  PcgDevice& D = dev[d & 63];
  if (D.sms) return D;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
  const void* f = (const void*)k_pcg_cluster;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(16); cfg.blockDim = dim3(PCG_CLUSTER_TPB); cfg.dynamicSmemBytes = RES_SMEM; cfg.attrs = at; cfg.numAttrs = 1;
  D.cluster = kernel_ready(f, RES_SMEM, true) == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n >= 1;
  cudaGetLastError();
  D.sms = sms > 0 ? sms : 148;
  return D;
}

// One cluster of `ctas` CTAs, or a cooperative grid of them.
cudaError_t launch_ctas(const void* f, bool cluster, int ctas, int tpb, int smem, int smem_max, void** args, cudaStream_t s) {
  cudaError_t e = kernel_ready(f, smem_max, cluster);
  if (e) return e;
  if (!cluster) return cudaLaunchCooperativeKernel(f, dim3(ctas), dim3(tpb), args, smem, s);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(tpb); cfg.dynamicSmemBytes = smem; cfg.stream = s; cfg.attrs = at; cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, f, args);
}

// Launch shapes of the looping form (more rows than the resident form takes):
//  - balanced: the 32-row slices spread evenly over the SMs (one or two
//    CTAs per SM, each warp one slice per pass);
//  - fixed CTA sizes of 256 and 512 threads up to the co-resident grid;
// each with one and two column slots loaded ahead per thread.
int streamed_shapes(int device, int V, bool learned, PcgShape* out, int max) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (sms < 1) sms = 1;
  const int ns = (V + 31) / 32 > 0 ? (V + 31) / 32 : 1;
  int n = 0;
  auto occ = [&](int unroll, int tpb) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, scaled_kernel(learned, unroll), tpb, 0);
    return per;
  };
  for (int unroll = 1; unroll <= 2; ++unroll) {
    const int wps = (ns + sms - 1) / sms;  // warps needed per SM for one pass
    int k = (wps + 31) / 32;               // CTAs per SM
    int tpb = 32 * ((wps + k - 1) / k);
    while (k > 1 && occ(unroll, tpb) < k) {
      --k;
      tpb = 32 * ((wps + k - 1) / k);
      if (tpb > SCALED_MAX_TPB) { tpb = SCALED_MAX_TPB; break; }
    }
    if (tpb > SCALED_MAX_TPB) tpb = SCALED_MAX_TPB;
    int per = occ(unroll, tpb);
    if (per >= 1 && n < max) {
      int grid = (ns + tpb / 32 - 1) / (tpb / 32);
      if (grid > sms * per) grid = sms * per;
      out[n++] = PcgShape{tpb, grid, unroll};
    }
    // fewer, larger CTAs: fewer arrivals at each grid barrier and fewer
    // copies of the per-slice partials read after it; the last two
    // candidates give every warp two slices
    for (int t : {256, 512, 768, 1024}) {
      int p = occ(unroll, t);
      if (p < 1 || n >= max) continue;
      int grid = (ns + t / 32 - 1) / (t / 32);
      if (grid > sms * p) grid = sms * p;
      out[n++] = PcgShape{t, grid, unroll};
      if (t >= 768 && grid > 1 && n < max) out[n++] = PcgShape{t, (grid + 1) / 2, unroll};
    }
  }
  return n;
}

// CTAs and slices per CTA of the resident form; false when V has more rows
// than it takes.
//  - Up to 8,192 rows without contact blocks (1,024 with): one cluster. Its
//    barriers cost a third of the grid's, but a row of another CTA is read at
//    an eighth of the local shared-memory rate, which many-block rows or more
//    rows to a CTA make the longer part. A slice as wide as a hub's row is walked
//    slot by slot, each with a column to turn into an address: on discs about a
//    hub of 64, 80, 128 and 512 neighbours the cluster takes 16, 24, 49 and 252 us
//    an iteration, the grid 16, 21, 44 and 194, so wider meshes go to the grid, and
//    so do contact blocks that are walked row by row (rows of 680 blocks: 209 and 148).
//  - Above: CTAs of 16 slices (8 with contact blocks, whose registers then
//    hold 24 neighbours' p), so that a small system leaves SMs to other
//    contexts' solves, and more slices once every SM has a CTA.
bool res_layout(int V, bool far, int wmax, bool& cluster, int& ctas, int& spc) {
  const PcgDevice D = pcg_device();
  const int ns = std::max(1, (V + 31) / 32), sms = std::min(D.sms, XR_MAX_CTAS);
  cluster = D.cluster && ns <= (far ? 32 : 256) && wmax <= RES_CLUSTER_SLOTS;
  if (cluster) {
    ctas = 1;
    while (ctas < 16 && ctas * 4 < ns) ctas *= 2;   // four warps to an SM while there are CTAs left
    spc = (ns + ctas - 1) / ctas;
    return true;
  }
  const int wide = far ? 8 : 16;
  spc = std::max(std::min(wide, ns), (ns + sms - 1) / sms);
  ctas = (ns + spc - 1) / spc;
  return spc <= 32;
}

}  // namespace

bool pcg_resident(int V) {
  bool cluster; int ctas, spc;
  return res_layout(V, true, 1, cluster, ctas, spc) && res_layout(V, false, 1, cluster, ctas, spc);
}

namespace {
// The resident launch of a system. far: contact blocks, rows of more than RES_KQ
// slots, or blocks that do not all fit on the chip.
struct ResPlan { ResKernel k; bool far, cluster; int ctas, spc, pub, near; };
ResPlan res_plan(int V, int wmax, bool contact, bool walked, bool learned) {
  ResPlan p{};
  if (walked) wmax = std::max(wmax, RES_CLUSTER_SLOTS + 1);
  p.far = contact || wmax > RES_KQ;
  while (true) {
    res_layout(V, p.far, wmax, p.cluster, p.ctas, p.spc);
    p.k = res_kernel(learned, p.far, p.cluster, 32 * p.spc);
    p.near = std::max(wmax - (p.k.compact ? 1 : 0), 1);
    p.pub = p.cluster ? 16 * 32 * p.spc * res_vectors(learned, p.far, p.k.kq) : 0;
    if (p.far || p.pub + p.spc * res_warp_bytes(p.near) <= RES_SMEM) return p;
    p.far = true;
  }
}
}  // namespace

// Candidate launch shapes of the scaled PCG for V rows of at most wmax slots,
// with or without contact blocks (walked: row by row), on `device`; shape 0 is the default. Every
// shape gives the same result bits. The resident form's CTAs and warps follow
// from those three; its candidates are the shared memory (KiB) for the blocks of
// a system that does not fit whole: all of it, or less, which leaves more to the
// L1 for the gathers. *same: the system fits, and they are one launch.
int pcg_scaled_shapes(int device, int V, int wmax, bool contact, bool walked, bool learned, PcgShape* out, int max, bool* same) {
  *same = false;
  if (!pcg_resident(V)) return streamed_shapes(device, V, learned, out, max);
  const ResPlan p = res_plan(V, wmax, contact, walked, learned);
  *same = !p.far;
  int n = 0;
  for (int kb : {RES_SMEM / 1024, 160, 96})
    if (n < max) out[n++] = PcgShape{32 * p.spc, p.ctas, kb};
  return n;
}

cudaError_t launch_pcg_scaled(const PcgScaledArgs& args, bool learned, const PcgShape& sh, cudaStream_t s) {
  if (sh.tpb < 32 || sh.tpb > SCALED_MAX_TPB || (sh.tpb & 31) || sh.grid < 1) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaMemsetAsync(&args.ctrl->bar_arrivals, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  PcgScaledArgs a = args;
  void* p[] = {(void*)&a};
  if (!pcg_resident(a.V)) return cudaLaunchCooperativeKernel((void*)scaled_kernel(learned, sh.unroll), dim3(sh.grid), dim3(sh.tpb), p, 0, s);
  const ResPlan q = res_plan(a.V, a.wmax, a.xbegin != nullptr, a.xbegin && !a.xs_off, learned);
  const int room = std::max(std::min(sh.unroll * 1024, RES_SMEM) - q.pub - 128 * q.spc, 0);
  a.slots = q.far ? std::min(room / (1280 * q.spc), 64) : q.near;
  const int smem = q.pub + q.spc * res_warp_bytes(a.slots);
  return launch_ctas(q.k.f, q.cluster, q.ctas, 32 * q.spc, smem, RES_SMEM, p, s);
}

bool pcg_packed_rows(int V) {
  const int ns = (V + 31) / 32, ctas = std::min(pcg_device().sms, XR_MAX_CTAS);
  return (ns + ctas - 1) / ctas > PCG_WARPS;
}

// Form of a solve, by its rows alone: one cluster up to 8,192 (3.8 us an
// iteration there, 6.5 over every SM at 8,281), then one CTA on each SM with a
// slice to each of its warps, from 113,665 rows on with several.
cudaError_t launch_pcg(const PcgArgs& args, cudaStream_t s) {
  const PcgDevice D = pcg_device();
  PcgArgs a = args;
  const int ns = (a.V + 31) / 32;
  if (D.cluster && a.V <= 16 * PCG_CLUSTER_TPB) {
    int C = 1;
    while (C < 16 && C * 4 < ns) C *= 2;   // four warps to an SM while there are CTAs left
    const int spc = (ns + C - 1) / C;
    a.smem = 48 * 32 * spc + spc * std::min((RES_SMEM - 48 * 32 * spc) / spc, 16 * 1024);
    void* p[] = {(void*)&a};
    return launch_ctas((const void*)k_pcg_cluster, true, C, 32 * spc, a.smem, RES_SMEM, p, s);
  }
  const int ctas = std::min(D.sms, XR_MAX_CTAS);
  const int spc = (ns + ctas - 1) / ctas, grid = (ns + spc - 1) / spc;
  const bool one = spc <= PCG_WARPS;   // as pcg_packed_rows
  const int each = one ? 1 : (spc + PCG_WARPS_MANY - 1) / PCG_WARPS_MANY, nw = (spc + each - 1) / each;
  a.smem = nw * std::min(PCG_SMEM / nw, one ? 24 * 1024 : PCG_BUF_MANY);
  void* p[] = {(void*)&a};
  return launch_ctas((const void*)pcg_kernel(one, nw), false, grid, 32 * nw, a.smem, PCG_SMEM, p, s);
}

}  // namespace ando
