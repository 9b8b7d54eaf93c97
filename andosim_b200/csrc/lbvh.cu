// lbvh.cu -- linear BVH broad phase (replaces Collision::build_*_bvh and
// broad_phase_triangles / broad_phase_edges, collision.cpp:65-276).
//
// Boxes are FP32, built from the FP32-rounded positions exactly as the
// reference's Real=float AABBs are (collision.cpp:48-62), optionally inflated
// by `pad`. The candidate predicate is the reference's inclusive overlap test
// (collision.h:37-41) with a +-1e-4 point box, the incident-face exclusion
// (collision.cpp:221) and, for edges, e1 < e2 and no shared vertex
// (collision.cpp:259-266). Any correct hierarchy returns exactly the set of
// primitive pairs whose boxes pass that test, so the result equals the
// brute-force query bit for bit once sorted.
//
// Pipeline: scene bounds -> 30-bit Morton codes of box centres -> stable radix
// sort (equal codes stay in index order, so code and index together are unique
// sorted keys) -> Karras hierarchy (one thread per internal node) -> boxes in
// shared memory (cut subtrees, then the nodes above the cut) -> one descent for
// the 32 queries of a warp, whose hits are queued and appended in batches; the
// pair list is then sorted so its order does not depend on scheduling.
#include <atomic>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>

#include "lbvh.cuh"
#include "narrow.cuh"

namespace ando {

namespace {

constexpr int TPB = 256;
inline int nblk(long long n, int tpb = TPB) { return int((n + tpb - 1) / tpb); }

using Box = LbvhBox;

__device__ inline float3 xf(const double* x, int i) { return make_float3(float(x[3 * i]), float(x[3 * i + 1]), float(x[3 * i + 2])); }

__device__ inline void grow(Box& b, float3 q) {
  b.lo[0] = fminf(b.lo[0], q.x); b.lo[1] = fminf(b.lo[1], q.y); b.lo[2] = fminf(b.lo[2], q.z);
  b.hi[0] = fmaxf(b.hi[0], q.x); b.hi[1] = fmaxf(b.hi[1], q.y); b.hi[2] = fmaxf(b.hi[2], q.z);
}

// Box of primitive i at positions x, or swept over x -> x1 when x1 is given.
__device__ inline Box prim_box(const double* x, const double* x1, const int* prims, int arity, int i, float pad) {
  float3 p = xf(x, prims[arity * i]);
  Box b; b.lo[0] = b.hi[0] = p.x; b.lo[1] = b.hi[1] = p.y; b.lo[2] = b.hi[2] = p.z;
  for (int k = 1; k < arity; ++k) grow(b, xf(x, prims[arity * i + k]));
  if (x1) for (int k = 0; k < arity; ++k) grow(b, xf(x1, prims[arity * i + k]));
  if (pad > 0.f) for (int k = 0; k < 3; ++k) { b.lo[k] -= pad; b.hi[k] += pad; }
  return b;
}

// Centre of a primitive's box, as the bounds and the codes take it.
__device__ inline float3 box_centre(const Box& b) {
  return make_float3(0.5f * (b.lo[0] + b.hi[0]), 0.5f * (b.lo[1] + b.hi[1]), 0.5f * (b.lo[2] + b.hi[2]));
}

// Scene bounds: min/max over box centres, on the ordered-int encoding (exact
// in any order). A block reduces its primitives first: one atomic per warp and
// axis of all primitives met at six addresses (18.7 us for 145,000 edges).
__device__ inline int f2ord(float f) { int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7fffffff; }
__device__ inline float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void k_bounds_init(int* b) {
  if (threadIdx.x < 3) { b[threadIdx.x] = 0x7fffffff; b[3 + threadIdx.x] = (int)0x80000000; }
}
__global__ void __launch_bounds__(TPB) k_bounds(const double* x, const double* x1, const int* prims, int arity, int n, float pad, int* bounds) {
  __shared__ int part[TPB / 32][6];
  int b[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000, (int)0x80000000};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float3 c = box_centre(prim_box(x, x1, prims, arity, i, pad));
    const int q[3] = {f2ord(c.x), f2ord(c.y), f2ord(c.z)};
    for (int k = 0; k < 3; ++k) { b[k] = min(b[k], q[k]); b[3 + k] = max(b[3 + k], q[k]); }
  }
  for (int k = 0; k < 6; ++k) b[k] = k < 3 ? __reduce_min_sync(0xffffffffu, b[k]) : __reduce_max_sync(0xffffffffu, b[k]);
  if ((threadIdx.x & 31) == 0) for (int k = 0; k < 6; ++k) part[threadIdx.x >> 5][k] = b[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    const int k = threadIdx.x;
    int v = part[0][k];
    for (int w = 1; w < TPB / 32; ++w) v = k < 3 ? min(v, part[w][k]) : max(v, part[w][k]);
    if (k < 3) atomicMin(&bounds[k], v); else atomicMax(&bounds[k], v);
  }
}

__device__ inline unsigned expand10(unsigned v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__global__ void k_morton(const double* x, const double* x1, const int* prims, int arity, int n, float pad, const int* bounds, unsigned* keys, int* vals) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 ctr = box_centre(prim_box(x, x1, prims, arity, i, pad));
  const float cc[3] = {ctr.x, ctr.y, ctr.z};
  unsigned m = 0;
  unsigned q[3];
  for (int k = 0; k < 3; ++k) {
    float lo = ord2f(bounds[k]), hi = ord2f(bounds[3 + k]);
    float c = cc[k];
    float t = hi > lo ? (c - lo) / (hi - lo) : 0.5f;
    t = fminf(fmaxf(t, 0.f), 1.f);
    q[k] = min(1023u, (unsigned)(t * 1024.f));
  }
  m = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
  keys[i] = m;
  vals[i] = i;
}

// The sorted keys: code then index.
struct SortedKeys {
  const unsigned* code; const int* index;
  __device__ unsigned long long operator[](int i) const { return ((unsigned long long)code[i] << 32) | (unsigned)index[i]; }
};
__device__ inline int delta(const SortedKeys& k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  return __clzll(k[i] ^ k[j]);
}

// Karras 2012: internal node i covers a key range found from the common
// prefix lengths of its neighbours. Nodes [0, n-1) are internal, leaves are
// encoded as n-1 + sorted position.
// topo[i] = {first leaf, last leaf of the left child, last leaf, parent} in
// sorted leaf positions (parent -1 at the root); the parent component is
// written by the parent's thread. The same thread fills sorted position i of
// the leaf arrays (rank; leafv: {primitive, its vertices, -1 past the arity},
// so a query's leaf test is one 16-byte load) and clears what the build and the
// refit start from (arrival counters, box slots).
__global__ void k_karras(SortedKeys keys, const int* prims, int arity, int n, int* parent, LbvhInner* inner, int4* topo, int* rank, int4* leafv,
                         int* arrive, int* wslot) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int prim = keys.index[i];
  const int* pv = prims + (long long)arity * prim;
  rank[prim] = i;
  leafv[i] = make_int4(prim, pv[0], arity > 1 ? pv[1] : -1, arity > 2 ? pv[2] : -1);
  wslot[n - 1 + i] = -1;
  if (i >= n - 1) return;
  arrive[i] = 0;
  wslot[i] = -1;
  if (i == 0) parent[0] = -1;
  int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = delta(keys, n, i, j);
  int s = 0;
  int t = l;
  do {
    t = (t + 1) >> 1;
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  int gamma = i + s * d + min(d, 0);
  int lo = min(i, j), hi = max(i, j);
  int lc = (lo == gamma) ? (n - 1 + gamma) : gamma;
  int rc = (hi == gamma + 1) ? (n - 1 + gamma + 1) : gamma + 1;
  inner[i].lc = lc; inner[i].rc = rc;
  inner[i].lmax = gamma; inner[i].rmax = hi;  // leaf ranges [lo, gamma] and [gamma + 1, hi]
  parent[lc] = i; parent[rc] = i;
  int* tw = reinterpret_cast<int*>(topo);
  tw[4 * i] = lo; tw[4 * i + 1] = gamma; tw[4 * i + 2] = hi;
  if (i == 0) tw[3] = -1;
  if (lc < n - 1) tw[4 * lc + 3] = i;
  if (rc < n - 1) tw[4 * rc + 3] = i;
}

__device__ inline Box ld_box_volatile(const Box* b) {
  const volatile float* v = reinterpret_cast<const volatile float*>(b);
  Box r;
  for (int k = 0; k < 3; ++k) { r.lo[k] = v[k]; r.hi[k] = v[3 + k]; }
  return r;
}

__device__ inline Box ld_box_cg(const Box* b) {
  const float* v = reinterpret_cast<const float*>(b);
  Box r;
  for (int k = 0; k < 3; ++k) { r.lo[k] = __ldcg(v + k); r.hi[k] = __ldcg(v + 3 + k); }
  return r;
}

__device__ inline Box unite(const Box& a, const Box& b) {
  Box u;
  for (int k = 0; k < 3; ++k) { u.lo[k] = fminf(a.lo[k], b.lo[k]); u.hi[k] = fmaxf(a.hi[k], b.hi[k]); }
  return u;
}

// Tiled bottom-up refit in two launches over a cut of the hierarchy made at
// build time. Below the cut: every subtree of at most RF_CUT leaves whose
// parent has more ("cut subtree"). Above it: the top nodes (more than RF_CUT
// leaves), numbered compactly.
//
// k_refit_cut: one CTA per cut subtree (grid-stride over the cut list). A
// node covers a run of leaves, so its box is a minimum over that run: the CTA
// builds the boxes of 2, 4, 8, ... leaves from each position (ten rounds of one
// unite a leaf, one barrier each), and after the round that fits its length each
// node unites the two runs that cover its own. Nothing waits for a child and all
// lanes work in every round; climbing from the leaves with arrival counters
// took a chain of some fifteen shared-memory atomics and fences at 14 active
// lanes of 32, and its staged topology left room for three CTAs of 512 on an SM.
// Boxes go to the four-wide records only; of the binary nodes' boxes just the
// subtree's root is read again. The leaf boxes are computed from the positions
// here. Shared-memory bandwidth bounds it now (some 18 accesses a leaf and round).
// A frame's refits: two curtains of 151^2 499 -> 280 us, of 256^2 818 -> 627, four
// sheets of 96^2 276 -> 169; one cloth of 97^2 31 -> 19. Two leaves to a thread,
// three CTAs of 512: 564 for the largest but 327 and 187 for the others.
//
// k_refit_top: one CTA finishes the top nodes in shared memory, each by the second
// of its children to arrive (block-scope arrival counters),
// reading the cut subtrees' boxes from nodes[], and writes them in one pass.
//
// When the top has more nodes than one CTA holds (or than the caller's
// capacity, Lbvh::top_cap), thread 0 of each cut subtree carries on through
// the top nodes with global arrival counters (acquire/release atomics; the
// second arrival zeroes the counter for the next refit) and k_refit_top does
// nothing. Min/max are exact, so every box has the same bits in any arrival
// order.
constexpr int RF_CUT = 1024;   // leaves of a subtree, and threads of its CTA
constexpr int TOP_TPB = 1024, TOP_MAX = 4096;
// top node: {node index, parent's top number (-1 at the root), left, right};
// a child is its top number (>= 0) or -(1 + its nodes[] index) below the cut
struct TopSmem { int4 rec[TOP_MAX]; Box box[TOP_MAX]; int arr[TOP_MAX]; };

__device__ inline bool is_top(const int4& t) { return t.z - t.x + 1 > RF_CUT; }

// Build time, per internal node: bit 0 for a top node, bit 32 for a node at
// even depth, the nodes of the four-wide hierarchy (the root is node 0 at depth
// 0); one exclusive scan numbers both. Karras depth is at most about 64 with
// unique 64-bit keys; the climb is bounded at 256 regardless.
__global__ void k_node_flags(const int4* topo, int n, unsigned long long* flag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int4 t = topo[i];
  int d = 0, p = t.w;
  while (p >= 0 && d < 256) { ++d; p = topo[p].w; }
  flag[i] = (is_top(t) ? 1ull : 0ull) | ((d & 1) == 0 ? 1ull << 32 : 0ull);
}

// Build time: the top records and the cut list (entries 2k, 2k+1: the
// below-cut children of top node k as leaf ranges, {-1, -1} for a top child).
__device__ inline void top_record(const int4* topo, const LbvhInner* inner, const unsigned long long* num, int n, int i, int4* rec, int2* cuts) {
  const int4 t = topo[i];
  if (!is_top(t)) return;
  const int k = int(num[i] & 0xffffffffull);
  const int lc = inner[i].lc, rc = inner[i].rc;
  const bool ltop = lc < n - 1 && is_top(topo[lc]), rtop = rc < n - 1 && is_top(topo[rc]);
  auto top_no = [&](int q) { return int(num[q] & 0xffffffffull); };
  rec[k] = make_int4(i, t.w >= 0 ? top_no(t.w) : -1, ltop ? top_no(lc) : -(1 + lc), rtop ? top_no(rc) : -(1 + rc));
  cuts[2 * k] = ltop ? make_int2(-1, -1) : make_int2(t.x, t.y);
  cuts[2 * k + 1] = rtop ? make_int2(-1, -1) : make_int2(t.y + 1, t.z);
}

// A node's final box into its four-wide slot (ws = 4 * node + slot; the
// slot's six floats start on an 8-byte boundary).
__device__ inline void store_slot(LbvhWide* wide, int ws, const Box& b) {
  float2* d = reinterpret_cast<float2*>(&wide[ws >> 2].box[ws & 3][0]);
  d[0] = make_float2(b.lo[0], b.lo[1]);
  d[1] = make_float2(b.lo[2], b.hi[0]);
  d[2] = make_float2(b.hi[1], b.hi[2]);
}

__global__ void __launch_bounds__(RF_CUT, 2) k_refit_cut(const double* x, const double* x1, const int* prims, int arity, float pad,
                                                         const int* order, int n, const int* parent, const int4* topo, const int2* cuts,
                                                         const int* meta, int top_cap, Box* nodes, int* arrive, const int* wslot, LbvhWide* wide) {
  __shared__ float run[2][6][RF_CUT];   // boxes of runs of 2^k leaves from each position, even and odd k
  const int ncut = meta[1], t = threadIdx.x;
  const bool top_global = meta[0] > top_cap;
  auto load = [&](int k, int i) {
    Box b;
    for (int e = 0; e < 3; ++e) { b.lo[e] = run[k & 1][e][i]; b.hi[e] = run[k & 1][3 + e][i]; }
    return b;
  };
  auto store = [&](int k, const Box& b) {
    for (int e = 0; e < 3; ++e) { run[k & 1][e][t] = b.lo[e]; run[k & 1][3 + e][t] = b.hi[e]; }
  };
  for (int cb = blockIdx.x; cb < ncut; cb += gridDim.x) {
    const int2 cut = cuts[cb];
    if (cut.x < 0) continue;  // uniform over the CTA
    const int c0 = cut.x, m = cut.y - c0 + 1, q = c0 + t;
    const bool leaf = t < m, inner = leaf && q < n - 1;
    const int prim = leaf ? order[q] : -1, wl = leaf ? wslot[n - 1 + q] : -1, wn = inner ? wslot[q] : -1;
    int first = 0, length = 0;
    if (inner) {
      const int4 tp = topo[q];
      // a node that is not wholly in this subtree is another's, or a top node
      if (tp.x >= c0 && tp.z < c0 + m) { first = tp.x - c0; length = tp.z - tp.x + 1; }
    }
    __syncthreads();  // the previous subtree's boxes are no longer read
    Box box;
    if (leaf) {
      box = prim_box(x, x1, prims, arity, prim, pad);
      store(0, box);
      if (wl >= 0) store_slot(wide, wl, box);
      if (m == 1) nodes[n - 1 + c0] = box;
    }
    __syncthreads();
    for (int k = 1; (1 << k) <= m; ++k) {
      if (t + (1 << k) <= m) {   // there is such a run
        box = unite(box, load(k - 1, t + (1 << (k - 1))));
        store(k, box);
      }
      __syncthreads();
      if (length >> k == 1) {
        const Box b = unite(load(k, first), load(k, first + length - (1 << k)));
        if (wn >= 0) store_slot(wide, wn, b);
        if (length == m) nodes[q] = b;
      }
    }
    // with more top nodes than k_refit_top holds, thread 0 carries on from
    // the subtree's root (index c0 or c1, or the leaf) through the top nodes,
    // once the root's box is published
    if (top_global) {
      __threadfence();
      __syncthreads();
    }
    if (top_global && threadIdx.x == 0) {
      const int c1 = cut.y;
      int root = -1;  // internal root index, -1: a single leaf
      if (m > 1) root = c0 < n - 1 && topo[c0].x == c0 && topo[c0].z == c1 ? c0 : c1;
      Box up = ld_box_cg(nodes + (root < 0 ? n - 1 + c0 : root));
      int p = root < 0 ? (n > 1 ? parent[n - 1 + c0] : -1) : topo[root].w;
      int chi = c1;
      while (p >= 0) {
        const int4 tp = __ldg(topo + p);
        const bool from_left = chi == tp.y;
        int prior;
        asm volatile("atom.add.acq_rel.gpu.s32 %0, [%1], 1;" : "=r"(prior) : "l"(arrive + p) : "memory");
        if (prior == 0) break;
        arrive[p] = 0;
        const int sl = from_left ? tp.y + 1 : tp.x, sh = from_left ? tp.z : tp.y, sidx = from_left ? tp.y + 1 : tp.y;
        up = unite(up, ld_box_cg(nodes + (sl == sh ? n - 1 + sl : sidx)));
        nodes[p] = up;
        const int wp = wslot[p];
        if (wp >= 0) store_slot(wide, wp, up);
        chi = tp.z;
        p = tp.w;
      }
    }
  }
}

__global__ void __launch_bounds__(TOP_TPB) k_refit_top(const int* meta, int top_cap, const int4* rec, Box* nodes, const int* wslot, LbvhWide* wide) {
  extern __shared__ __align__(16) unsigned char rt_raw[];
  TopSmem& S = *reinterpret_cast<TopSmem*>(rt_raw);
  const int m = meta[0];
  if (m <= 0 || m > top_cap) return;
  for (int k = threadIdx.x; k < m; k += TOP_TPB) {
    const int4 r = rec[k];
    S.rec[k] = r;
    S.arr[k] = (r.z < 0) + (r.w < 0);  // below-cut children have arrived already
  }
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += TOP_TPB) {
    int4 r = S.rec[k];
    if (r.z >= 0 || r.w >= 0) continue;  // starts only where both children are below the cut
    int cur = k;
    Box box = unite(ld_box_cg(nodes + (-r.z - 1)), ld_box_cg(nodes + (-r.w - 1)));
    while (true) {
      S.box[cur] = box;
      const int pc = r.y;
      if (pc < 0) break;
      const int4 pr = S.rec[pc];
      const bool from_left = pr.z == cur;
      __threadfence_block();
      if (atomicAdd(&S.arr[pc], 1) == 0) break;
      __threadfence_block();
      const int sib = from_left ? pr.w : pr.z;
      box = unite(box, sib >= 0 ? ld_box_volatile(&S.box[sib]) : ld_box_cg(nodes + (-sib - 1)));
      cur = pc;
      r = pr;
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += TOP_TPB) {
    const int4 r = S.rec[k];
    nodes[r.x] = S.box[k];
    const int ws = wslot[r.x];
    if (ws >= 0) store_slot(wide, ws, S.box[k]);
  }
}

// Build time: the refit schedule and the four-wide topology. Per internal node
// its top record; for a node of the four-wide hierarchy its children, leaf
// bounds and empty slots, and the slot of every binary node whose box it keeps:
// a leaf child, or a child of a folded node (k_karras set wslot to -1; the root
// and the folded nodes keep that). meta = {top nodes, cut entries}; with no top
// node the whole hierarchy is one cut subtree.
__global__ void k_schedule(const int4* topo, const LbvhInner* inner, const unsigned long long* flag, const unsigned long long* num, int n, int4* rec,
                           int2* cuts, int* meta, LbvhWide* wide, int* wslot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    const int m = n > 1 ? int((num[n - 2] + flag[n - 2]) & 0xffffffffull) : 0;
    meta[0] = m;
    meta[1] = m > 0 ? 2 * m : 1;
    if (m == 0) cuts[0] = make_int2(0, n - 1);
  }
  if (i >= n - 1) return;
  top_record(topo, inner, num, n, i, rec, cuts);
  if (!(flag[i] >> 32)) return;
  auto wide_no = [&](int q) { return int(num[q] >> 32); };
  const int leaf0 = n - 1, w = wide_no(i);
  LbvhWide& W = wide[w];
  const LbvhInner r = inner[i];
  auto enc = [&](int c) { return c >= leaf0 ? -(c - leaf0) - 1 : wide_no(c); };
  for (int sd = 0; sd < 2; ++sd) {
    const int c = sd ? r.rc : r.lc;
    const int k = 2 * sd;
    if (c >= leaf0) {
      W.child[k] = enc(c); W.cmax[k] = sd ? r.rmax : r.lmax; wslot[c] = 4 * w + k;
      for (int e = 0; e < 3; ++e) { W.box[k + 1][e] = FLT_MAX; W.box[k + 1][3 + e] = -FLT_MAX; }
      W.child[k + 1] = 0; W.cmax[k + 1] = INT_MIN;
    } else {
      const LbvhInner g = inner[c];
      W.child[k] = enc(g.lc); W.cmax[k] = g.lmax; wslot[g.lc] = 4 * w + k;
      W.child[k + 1] = enc(g.rc); W.cmax[k + 1] = g.rmax; wslot[g.rc] = 4 * w + k + 1;
    }
  }
}

__device__ inline bool overlap(const Box& a, const Box& b) {
  return a.lo[0] <= b.hi[0] && a.hi[0] >= b.lo[0] && a.lo[1] <= b.hi[1] && a.hi[1] >= b.lo[1] && a.lo[2] <= b.hi[2] && a.hi[2] >= b.lo[2];
}

// Warp-ballot append: one atomic per warp per round of hits.
__device__ inline void emit(bool hit, int q, int prim, int2* out, int* count, int cap) {
  unsigned mask = __ballot_sync(0xffffffffu, hit);
  if (!mask) return;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (hit) {
    int slot = base + __popc(mask & ((1u << lane) - 1u));
    if (slot < cap) out[slot] = make_int2(q, prim);
  }
}

// One lane per query. kind 0: query = vertex (point box +-1e-4 inflated by
// pad), prims = triangles, skip incident triangles. kind 1: query = edge,
// prims = edges, keep e1 < e2 without shared vertex. kind 2: query = edge,
// prims = triangles, skip triangles that hold either end of the edge.
//
// A descent is a chain of dependent node loads, and with one to a query there
// were about a hundred of them to a warp, half the lanes idle in each. The queries
// of a warp are neighbours (Morton order at rest), so the warp descends once for
// all of them: per step it takes up to eight nodes from its stack, a lane to each
// child box, and keeps the children that meet one of the warp's group boxes; the
// leaves found are then tested against every lane's own box, 32 tests a
// broadcast. A group is the largest aligned run of lanes whose common box is no
// larger than GROUP_SPREAD (runs of up to four: FOUR_SPREAD) times the patch that
// as many boxes of their size, or of a primitive's where that is larger (the
// root's box over sqrt(n)), fill. A run that spans a seam of the order, or sheets
// that have moved apart, so falls into smaller groups, down to single lanes, in
// place of descending through all that lies between. The tests that decide are
// each query's own: the pairs are those of one descent per query.
//
// Hits that are not incident (the leaves' vertices are loaded beside the tests)
// gather in a shared-memory queue of the warp and leave it with one atomic for up
// to QUEUE of them.
//
// Two curtains of 256^2 (swept boxes; 50 to 57 thousand cycles of a warp go to 20
// steps, half of them, and the rest to 130 leaves and 70 hits): the edge-edge
// query 156 -> 135 us, vertex-triangle 140 -> 87; four sheets of 96^2, a frame's
// eight queries 1296 -> 850; one hanging cloth of 97^2, both 117 -> 44. The spread:
// at 2.0 the sheets' edges take 180 us in place of 166 (long tails of leaves), at
// 1.0 the curtains' vertices 98 in place of 87 (22 groups a step); runs of up to
// four lanes may spread twice as far, which halves the groups there and adds no
// leaves. 64 registers instead of 76 spill and cost a third.
constexpr int QUEUE = 256;                        // hits per warp
constexpr int QSTACK = 256, QSTACK_WIDE = 128;    // nodes per warp; above QSTACK_WIDE one node is taken at a time
constexpr int QLEAVES = 64;                       // leaves per warp; a step adds at most 32
constexpr int Q_TPB = 128;
constexpr float GROUP_SPREAD = 1.5f, FOUR_SPREAD = 3.f;
struct QueryWarp {
  float4 box[32][2];        // group boxes: lo, hi and the smallest leaf position that concerns the group
  float4 leaf[QLEAVES][2];  // leaf boxes: lo, hi, position
  int4 prim[32];            // of the leaves under test: primitive and vertices
  int2 hits[QUEUE];
  int stack[QSTACK];
};
__global__ void __launch_bounds__(Q_TPB) k_query(const double* x, const double* x1, const int* qprims, const int* qorder, int kind, int nq, float pad, int n,
                        const int4* leafv, const int* rank, const LbvhWide* wide, const Box* nodes, int2* out, int* count, int cap) {
  __shared__ __align__(16) QueryWarp warps[Q_TPB / 32];
  QueryWarp& W = warps[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  int held = 0;   // entries in the queue (this and the other counts are uniform over the warp)
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  bool active = t < nq;
  const int q = active && qorder ? qorder[t] : t;
  Box qb;
  qb.lo[0] = qb.lo[1] = qb.lo[2] = FLT_MAX; qb.hi[0] = qb.hi[1] = qb.hi[2] = -FLT_MAX;
  int qa = -1, qc = -1;
  if (active) {
    if (kind == 0) {
      float3 p = xf(x, q);
      float e = 1e-4f;
      qb.lo[0] = p.x - e; qb.lo[1] = p.y - e; qb.lo[2] = p.z - e;
      qb.hi[0] = p.x + e; qb.hi[1] = p.y + e; qb.hi[2] = p.z + e;
      if (x1) {
        float3 p1 = xf(x1, q);
        qb.lo[0] = fminf(qb.lo[0], p1.x - e); qb.lo[1] = fminf(qb.lo[1], p1.y - e); qb.lo[2] = fminf(qb.lo[2], p1.z - e);
        qb.hi[0] = fmaxf(qb.hi[0], p1.x + e); qb.hi[1] = fmaxf(qb.hi[1], p1.y + e); qb.hi[2] = fmaxf(qb.hi[2], p1.z + e);
      }
      if (pad > 0.f) for (int k = 0; k < 3; ++k) { qb.lo[k] -= pad; qb.hi[k] += pad; }
    } else {
      qa = qprims[2 * q]; qc = qprims[2 * q + 1];
      float3 a = xf(x, qa), b = xf(x, qc);
      qb.lo[0] = fminf(a.x, b.x); qb.lo[1] = fminf(a.y, b.y); qb.lo[2] = fminf(a.z, b.z);
      qb.hi[0] = fmaxf(a.x, b.x); qb.hi[1] = fmaxf(a.y, b.y); qb.hi[2] = fmaxf(a.z, b.z);
      if (x1) { grow(qb, xf(x1, qa)); grow(qb, xf(x1, qc)); }
      if (pad > 0.f) for (int k = 0; k < 3; ++k) { qb.lo[k] -= pad; qb.hi[k] += pad; }
    }
  }
  // The edge-edge query is a self query: each pair is found from the edge
  // that comes first in the tree's sorted leaf order (children whose leaves
  // all come before the query's own position are skipped) and reported with
  // the lower edge index first, which is the set the q < prim rule of a full
  // query gives.
  const int qpos = !active ? INT_MAX : kind == 1 ? rank[q] : -1;
  // group boxes: level by level the box of the lane's aligned run of 2^l lanes
  int groups = 0;
  {
    Box u = qb, best = qb;
    int first = qpos, best_first = qpos, level = 0;
    const Box root = nodes[0];
    const float prim = ((root.hi[0] - root.lo[0]) + (root.hi[1] - root.lo[1]) + (root.hi[2] - root.lo[2])) * rsqrtf(float(n));
    float sum = active ? fmaxf((qb.hi[0] - qb.lo[0]) + (qb.hi[1] - qb.lo[1]) + (qb.hi[2] - qb.lo[2]), prim) : 0.f;
    int members = active;
#pragma unroll
    for (int l = 1; l <= 5; ++l) {
      const int o = 1 << (l - 1);
      for (int e = 0; e < 3; ++e) {
        u.lo[e] = fminf(u.lo[e], __shfl_xor_sync(0xffffffffu, u.lo[e], o));
        u.hi[e] = fmaxf(u.hi[e], __shfl_xor_sync(0xffffffffu, u.hi[e], o));
      }
      first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      members += __shfl_xor_sync(0xffffffffu, members, o);
      if ((u.hi[0] - u.lo[0]) + (u.hi[1] - u.lo[1]) + (u.hi[2] - u.lo[2]) <= (l <= 2 ? FOUR_SPREAD : GROUP_SPREAD) * sum * rsqrtf(float(max(members, 1)))) {
        level = l; best = u; best_first = first;
      }
    }
    const bool lead = active && (lane & ((1 << level) - 1)) == 0;   // lane 0 of a run is active where any is
    const unsigned mask = __ballot_sync(0xffffffffu, lead);
    if (lead) {
      const int g = __popc(mask & ((1u << lane) - 1u));
      W.box[g][0] = make_float4(best.lo[0], best.lo[1], best.lo[2], best.hi[0]);
      W.box[g][1] = make_float4(best.hi[1], best.hi[2], __int_as_float(best_first), 0.f);
    }
    groups = __popc(mask);
  }
  auto flush = [&]() {
    int base = 0;
    __syncwarp();
    if (lane == 0) base = atomicAdd(count, held);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int k = lane; k < held; k += 32)
      if (base + k < cap) out[base + k] = W.hits[k];
    held = 0;
    __syncwarp();
  };
  // The binary hierarchy is at most 64 levels deep with unique 64-bit keys, the
  // four-wide one half that. Eight nodes at a time are taken from a stack of up to
  // QSTACK_WIDE nodes and add at most 24; one at a time then adds three a level:
  // 128 + 24 + 96 nodes. An overflow would be reported through count[1] instead
  // of dropping candidates silently.
  int sp = 0, nl = 0;
  if (groups > 0) {
    if (n > 1) {
      sp = 1;
      if (lane == 0) W.stack[0] = 0;
    } else {       // one primitive: the root (node 0) is its leaf
      nl = 1;
      if (lane == 0) {
        const Box b = nodes[0];
        W.leaf[0][0] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.hi[0]);
        W.leaf[0][1] = make_float4(b.hi[1], b.hi[2], __int_as_float(0), 0.f);
      }
    }
  }
  __syncwarp();
  while (sp > 0 || nl > 0) {
    if (sp > 0) {
      const int take = sp <= QSTACK_WIDE ? min(8, sp) : 1;
      const int node = (lane >> 2) < take ? W.stack[sp - 1 - (lane >> 2)] : -1, k = lane & 3;
      sp -= take;
      float2 a = make_float2(FLT_MAX, FLT_MAX), b = make_float2(FLT_MAX, -FLT_MAX), c = make_float2(-FLT_MAX, -FLT_MAX);
      int child = 0, last = INT_MIN;
      if (node >= 0) {
        const float2* r = reinterpret_cast<const float2*>(wide + node) + 3 * k;
        a = __ldg(r); b = __ldg(r + 1); c = __ldg(r + 2);
        child = __ldg(reinterpret_cast<const int*>(wide + node) + 24 + k);
        last = __ldg(reinterpret_cast<const int*>(wide + node) + 28 + k);
      }
      bool hit = false;
      for (int g = 0; g < groups; ++g) {
        const float4 u = W.box[g][0], w = W.box[g][1];
        hit |= (last > __float_as_int(w.z)) & (u.x <= b.y) & (u.w >= a.x) & (u.y <= c.x) & (w.x >= a.y) & (u.z <= c.y) & (w.y >= b.x);
      }
      const unsigned inner = __ballot_sync(0xffffffffu, hit && child >= 0), leaves = __ballot_sync(0xffffffffu, hit && child < 0);
      if (hit && child >= 0) {
        const int at = sp + __popc(inner & ((1u << lane) - 1u));
        if (at < QSTACK) W.stack[at] = child;
        else atomicAdd(count + 1, 1);
      }
      if (hit && child < 0) {
        const int at = nl + __popc(leaves & ((1u << lane) - 1u));
        W.leaf[at][0] = make_float4(a.x, a.y, b.x, b.y);
        W.leaf[at][1] = make_float4(c.x, c.y, __int_as_float(-child - 1), 0.f);
      }
      sp = min(sp + __popc(inner), QSTACK);
      nl += __popc(leaves);
      __syncwarp();
    }
    while (nl >= 32 || (sp == 0 && nl > 0)) {
      const int m = min(nl, 32);
      nl -= m;
      int4 mine = make_int4(0, 0, 0, 0);
      if (lane < m) mine = leafv[__float_as_int(W.leaf[nl + lane][1].z)];
      unsigned met = 0;   // bit e: the lane's box meets leaf nl + e
#pragma unroll 8
      for (int e = 0; e < m; ++e) {
        const float4 u = W.leaf[nl + e][0], w = W.leaf[nl + e][1];
        const bool h = (__float_as_int(w.z) > qpos) & (qb.lo[0] <= u.w) & (qb.hi[0] >= u.x) & (qb.lo[1] <= w.x) & (qb.hi[1] >= u.y) &
                       (qb.lo[2] <= w.y) & (qb.hi[2] >= u.z);
        met |= unsigned(h) << e;
      }
      W.prim[lane] = mine;
      __syncwarp();
      for (unsigned left = met; left; left &= left - 1) {
        const int e = __ffs(left) - 1;
        const int4 lv = W.prim[e];
        const bool incident = kind == 0 ? (lv.y == q) | (lv.z == q) | (lv.w == q)
                                        : (lv.y == qa) | (lv.y == qc) | (lv.z == qa) | (lv.z == qc) | (kind == 2 && (lv.w == qa || lv.w == qc));
        met ^= unsigned(incident) << e;
      }
      while (__any_sync(0xffffffffu, met != 0)) {
        // as many of each lane's hits as the queue takes from all lanes
        const int room = QUEUE - held;
        int mineto = __popc(met), upto = mineto;
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += v; }
        const int total = __shfl_sync(0xffffffffu, upto, 31);
        int at = upto - mineto;
        for (; met && at < room; met &= met - 1, ++at) {
          const int prim = W.prim[__ffs(met) - 1].x;
          // (lower, higher) edge index for the self query
          W.hits[held + at] = kind == 1 ? make_int2(min(q, prim), max(q, prim)) : make_int2(q, prim);
        }
        held += min(total, room);
        if (held == QUEUE) flush();
      }
      __syncwarp();
    }
  }
  if (held) flush();
}

// The four vertices of candidate pair (q, prim): kind 0 vertex q against
// triangle prim; kind 1 edge q against edge prim.
__device__ inline void pair_ids(int kind, int2 pr, const int* prims, const int* qprims, int id[4]) {
  if (kind == 0) { id[0] = pr.x; id[1] = prims[3 * pr.y]; id[2] = prims[3 * pr.y + 1]; id[3] = prims[3 * pr.y + 2]; }
  else { id[0] = qprims[2 * pr.x]; id[1] = qprims[2 * pr.x + 1]; id[2] = prims[2 * pr.y]; id[3] = prims[2 * pr.y + 1]; }
}

// Narrow phase over the candidate list of the last traversal. The count
// stays on the device (count[0]); a list that overflowed its capacity sets
// *overflow instead of being used, so the caller grows it and runs again.
constexpr int NARROW_GRID = 148 * 8;

// candidates whose FP64 distance at x is below gap -> surv (count[2])
__global__ void k_pairs_gap(const int2* cand, const int* count, int cap, int kind, const int* prims, const int* qprims, const double* x,
                            double gap, int2* surv, int* scount) {
  const int n = min(count[0], cap);
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    bool keep = false;
    int2 pr = make_int2(0, 0);
    if (i < n) {
      pr = cand[i];
      int id[4];
      pair_ids(kind, pr, prims, qprims, id);
      keep = pair_gap(kind, id, x) < gap;
    }
    emit(keep, pr.x, pr.y, surv, scount, cap);
  }
}

// min over the candidates of the conservative time of impact along ext. With
// `pad` > 0 the traversal ran on boxes inflated by pad (so that the list also
// holds every pair that can come within the contact distance at any position
// on the way): only the pairs whose boxes overlap without the pad, built and
// compared exactly as an unpadded traversal does, bound the step.
__global__ void k_pairs_toi(const int2* cand, const int* count, int cap, int kind, const int* prims, const int* qprims, const double* x,
                            const double* x1, const double* ext, float pad, double eta_min, double near, unsigned long long* toi,
                            int* overflow) {
  if (count[0] > cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(overflow, count[0]);  // the capacity that is needed
    return;
  }
  const int n = count[0];
  double t = 1.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int2 pr = cand[i];
    if (pad > 0.f) {
      Box qb;
      if (kind == 0) {
        const float3 p = xf(x, pr.x), p1 = xf(x1, pr.x);
        const float e = 1e-4f;
        qb.lo[0] = fminf(p.x - e, p1.x - e); qb.lo[1] = fminf(p.y - e, p1.y - e); qb.lo[2] = fminf(p.z - e, p1.z - e);
        qb.hi[0] = fmaxf(p.x + e, p1.x + e); qb.hi[1] = fmaxf(p.y + e, p1.y + e); qb.hi[2] = fmaxf(p.z + e, p1.z + e);
      } else {
        qb = prim_box(x, x1, qprims, 2, pr.x, 0.f);
      }
      if (!overlap(qb, prim_box(x, x1, prims, kind == 0 ? 3 : 2, pr.y, 0.f))) continue;
    }
    int id[4];
    pair_ids(kind, pr, prims, qprims, id);
    t = fmin(t, pair_toi(kind, id, x, ext, eta_min, near));
  }
  t = warp_min(t);
  if ((threadIdx.x & 31) == 0 && t < 1.0) atomic_min_pos(toi, t);
}

// Exact segment-triangle crossing test in FP64: the segment's ends lie
// strictly on opposite sides of the triangle's plane and the crossing point
// has barycentric coordinates in [0, 1]. Every product, sum and quotient is
// rounded on its own (no fused multiply-add), in the order written, so the
// test takes the same decision as the same formula in plain IEEE double
// arithmetic on the host.
__device__ inline bool segment_crosses_triangle(const double* x, int p, int q, int a, int b, int c) {
  auto mul = [](double u, double v) { return __dmul_rn(u, v); };
  auto add = [](double u, double v) { return __dadd_rn(u, v); };
  auto sub = [](double u, double v) { return __dsub_rn(u, v); };
  double A[3], u[3], w[3], P[3], Q[3];
  for (int k = 0; k < 3; ++k) {
    A[k] = x[3 * a + k];
    u[k] = sub(x[3 * b + k], A[k]);
    w[k] = sub(x[3 * c + k], A[k]);
    P[k] = x[3 * p + k];
    Q[k] = x[3 * q + k];
  }
  const double n0 = sub(mul(u[1], w[2]), mul(u[2], w[1]));
  const double n1 = sub(mul(u[2], w[0]), mul(u[0], w[2]));
  const double n2 = sub(mul(u[0], w[1]), mul(u[1], w[0]));
  const double s0 = add(add(mul(n0, sub(P[0], A[0])), mul(n1, sub(P[1], A[1]))), mul(n2, sub(P[2], A[2])));
  const double s1 = add(add(mul(n0, sub(Q[0], A[0])), mul(n1, sub(Q[1], A[1]))), mul(n2, sub(Q[2], A[2])));
  if (!((s0 > 0.0 && s1 < 0.0) || (s0 < 0.0 && s1 > 0.0))) return false;
  const double t = __ddiv_rn(s0, sub(s0, s1));
  double X[3];
  for (int k = 0; k < 3; ++k) X[k] = sub(add(P[k], mul(t, sub(Q[k], P[k]))), A[k]);
  auto dot3 = [&](const double* e, const double* f) { return add(add(mul(e[0], f[0]), mul(e[1], f[1])), mul(e[2], f[2])); };
  const double uu = dot3(u, u), uw = dot3(u, w), ww = dot3(w, w), xu = dot3(X, u), xw = dot3(X, w);
  const double den = sub(mul(uu, ww), mul(uw, uw));
  if (!(fabs(den) > 0.0)) return false;
  const double bv = __ddiv_rn(sub(mul(ww, xu), mul(uw, xw)), den);
  const double bw = __ddiv_rn(sub(mul(uu, xw), mul(uw, xu)), den);
  return bv >= 0.0 && bw >= 0.0 && add(bv, bw) <= 1.0;
}

// Crossings among the (edge, triangle) candidates of a kind-2 traversal,
// summed into *crossings; nothing when the list overflowed its capacity (the
// caller reads count[0], grows the list and runs again).
__global__ void k_pairs_cross(const int2* cand, const int* count, int cap, const int* tris, const int* edges, const double* x,
                              unsigned long long* crossings) {
  if (count[0] > cap) return;
  const int n = count[0];
  unsigned long long mine = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int2 pr = cand[i];
    mine += segment_crosses_triangle(x, edges[2 * pr.x], edges[2 * pr.x + 1], tris[3 * pr.y], tris[3 * pr.y + 1], tris[3 * pr.y + 2]);
  }
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(crossings, mine);
}

// Candidate pairs are sorted as one key each, query above primitive (`pbits`
// bits), which is all there is to move: no payload, and only the bits that the
// two index ranges need.
__global__ void k_pair_keys(const int2* pairs, int n, int pbits, unsigned long long* keys) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = ((unsigned long long)(unsigned)pairs[i].x << pbits) | (unsigned)pairs[i].y;
}
__global__ void k_key_pairs(const unsigned long long* keys, int n, int pbits, int2* pairs) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) pairs[i] = make_int2(int(keys[i] >> pbits), int(keys[i] & ((1ull << pbits) - 1ull)));
}
inline int index_bits(int n) { int b = 1; while (b < 31 && (1 << b) < n) ++b; return b; }

// `out` = the m pairs of `in` (query < nq, primitive < n) sorted by (query, primitive).
cudaError_t sort_pairs(const int2* in, int m, int nq, int n, DevBuf<int2>& out, DevBuf<unsigned long long>& k0, DevBuf<unsigned long long>& k1,
                       DevBuf<unsigned char>& tmp, cudaStream_t s) {
  cudaError_t e;
  if ((e = k0.reserve(m))) return e;
  if ((e = k1.reserve(m))) return e;
  if ((e = out.reserve(m))) return e;
  const int pbits = index_bits(n), bits = pbits + index_bits(nq);
  k_pair_keys<<<nblk(m), TPB, 0, s>>>(in, m, pbits, k0.p);
  size_t bytes = 0;
  if ((e = cub::DeviceRadixSort::SortKeys(nullptr, bytes, k0.p, k1.p, m, 0, bits, s))) return e;
  if ((e = tmp.reserve(bytes))) return e;
  if ((e = cub::DeviceRadixSort::SortKeys(tmp.p, bytes, k0.p, k1.p, m, 0, bits, s))) return e;
  k_key_pairs<<<nblk(m), TPB, 0, s>>>(k1.p, m, pbits, out.p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t Lbvh::reserve_prims(int n) {
  cudaError_t e;
  size_t N = n > 0 ? n : 1;
  if ((e = codes.reserve(N))) return e;
  if ((e = codes_sorted.reserve(N))) return e;
  if ((e = idx.reserve(N))) return e;
  if ((e = nflag.reserve(N))) return e;
  if ((e = nnum.reserve(N))) return e;
  if ((e = order.reserve(N))) return e;
  if ((e = parent.reserve(2 * N))) return e;
  if ((e = nodes.reserve(2 * N))) return e;
  if ((e = inner.reserve(N))) return e;
  if ((e = wide.reserve(N))) return e;
  if ((e = wslot.reserve(2 * N))) return e;
  if ((e = rank.reserve(N))) return e;
  if ((e = arrive.reserve(N))) return e;
  if ((e = topo.reserve(N))) return e;
  if ((e = leafv.reserve(N))) return e;
  if ((e = toprec.reserve(N))) return e;
  if ((e = cuts.reserve(2 * N))) return e;
  if ((e = meta.reserve(2))) return e;
  if ((e = bounds.reserve(6))) return e;
  return cudaSuccess;
}

// Build the hierarchy over `n` primitives of `arity` vertex indices each.
cudaError_t Lbvh::build(const double* x, const double* x1, const int* prims_, int arity_, int n_, float pad, DevBuf<unsigned char>& tmp, cudaStream_t s) {
  n = n_;
  prims = prims_;
  arity = arity_;
  cudaError_t e = reserve_prims(n);
  if (e) return e;
  if (n == 0) return cudaSuccess;
  k_bounds_init<<<1, 32, 0, s>>>(bounds.p);
  k_bounds<<<std::min(nblk(n), 296), TPB, 0, s>>>(x, x1, prims, arity, n, pad, bounds.p);
  k_morton<<<nblk(n), TPB, 0, s>>>(x, x1, prims, arity, n, pad, bounds.p, codes.p, idx.p);
  // 30 code bits: half the passes that sorting by code and index took, and half the key
  size_t bytes = 0;
  if ((e = cub::DeviceRadixSort::SortPairs(nullptr, bytes, codes.p, codes_sorted.p, idx.p, order.p, n, 0, 30, s))) return e;
  if ((e = tmp.reserve(bytes))) return e;
  if ((e = cub::DeviceRadixSort::SortPairs(tmp.p, bytes, codes.p, codes_sorted.p, idx.p, order.p, n, 0, 30, s))) return e;
  k_karras<<<nblk(n), TPB, 0, s>>>(SortedKeys{codes_sorted.p, order.p}, prims, arity, n, parent.p, inner.p, topo.p, rank.p, leafv.p, arrive.p, wslot.p);
  if (n > 1) {
    k_node_flags<<<nblk(n - 1), TPB, 0, s>>>(topo.p, n, nflag.p);
    bytes = 0;
    if ((e = cub::DeviceScan::ExclusiveSum(nullptr, bytes, nflag.p, nnum.p, n - 1, s))) return e;
    if ((e = tmp.reserve(bytes))) return e;
    if ((e = cub::DeviceScan::ExclusiveSum(tmp.p, bytes, nflag.p, nnum.p, n - 1, s))) return e;
  }
  k_schedule<<<std::max(1, nblk(n - 1)), TPB, 0, s>>>(topo.p, inner.p, nflag.p, nnum.p, n, toprec.p, cuts.p, meta.p, wide.p, wslot.p);
  if ((e = launch_refit(x, x1, pad, s))) return e;
  launches += (n > 1 ? 7 : 6) + (n > RF_CUT ? 1 : 0);
  return cudaGetLastError();
}

// Update the boxes of the last build for new positions (same primitives):
// primitive boxes, then the bottom-up node boxes over the existing topology.
// The candidate set of a query does not depend on the topology, only the
// traversal cost does, so the Morton order of an earlier build stays valid.
cudaError_t Lbvh::refit(const double* x, const double* x1, float pad, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  cudaError_t e = launch_refit(x, x1, pad, s);
  launches += n > RF_CUT ? 2 : 1;
  return e;
}

// The global arrival counters are zero between refits: the build zeroes them
// and every refit leaves them zero (each node's second arrival resets it).
cudaError_t Lbvh::launch_refit(const double* x, const double* x1, float pad, cudaStream_t s) {
  static_assert(sizeof(TopSmem) <= 227 * 1024, "refit tile exceeds shared memory");
  // Set once per device: the call is 0.3 us from one thread and 200 us when sixteen
  // contexts step at once, for it waits there for the others' launches.
  static std::atomic<unsigned> attr{0};
  cudaError_t e = cudaSuccess;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 32 || !(attr.load() & (1u << dev))) {
    e = cudaFuncSetAttribute(k_refit_top, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TopSmem)));
    if (e) return e;
    if (dev < 32) attr.fetch_or(1u << dev);
  }
  // SMs of the device (contexts of a batch step on host threads: the
  // function-local static is initialised once, thread-safely; 148 if the
  // query fails)
  static const int sms = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return 148;
    }
    return n;
  }();
  // grid-stride over the cut list (its length stays on the device): about
  // two subtrees per SM resident at once
  const int grid = std::max(1, std::min(2 * sms, 2 * ((n + 255) / 256)));
  const int cap = top_cap < 0 || top_cap > TOP_MAX ? TOP_MAX : top_cap;
  k_refit_cut<<<grid, RF_CUT, 0, s>>>(x, x1, prims, arity, pad, order.p, n, parent.p, topo.p, cuts.p, meta.p, cap,
                                                      nodes.p, arrive.p, wslot.p, wide.p);
  if (n > RF_CUT) k_refit_top<<<1, TOP_TPB, sizeof(TopSmem), s>>>(meta.p, cap, toprec.p, nodes.p, wslot.p, wide.p);
  return cudaGetLastError();
}

cudaError_t Lbvh::update(const double* x, const double* x1, const int* prims_, int arity_, int n_, float pad, long long epoch_,
                         DevBuf<unsigned char>& tmp, cudaStream_t s) {
  if (epoch_ == epoch && n_ == n && prims_ == prims && arity_ == arity && n > 0) return refit(x, x1, pad, s);
  epoch = epoch_;
  return build(x, x1, prims_, arity_, n_, pad, tmp, s);
}

namespace {
// Sorted box-candidate pairs of a query (capacity grown as needed).
cudaError_t run_query(Lbvh& B, const double* x, const double* x1, int kind, const int* qprims, int nq, float pad, DevBuf<int2>& out,
                      DevBuf<int2>& scratch, DevBuf<unsigned long long>& k0, DevBuf<unsigned long long>& k1, DevBuf<int>& counter,
                      DevBuf<unsigned char>& tmp, int* npairs, cudaStream_t s) {
  cudaError_t e;
  *npairs = 0;
  if (B.n == 0 || nq == 0) return cudaSuccess;
  if ((e = counter.reserve(3))) return e;
  if (scratch.n < 1024) if ((e = scratch.reserve(1024))) return e;
  for (int attempt = 0; attempt < 2; ++attempt) {
    int cap = int(scratch.n);
    if ((e = cudaMemsetAsync(counter.p, 0, 3 * sizeof(int), s))) return e;
    k_query<<<nblk(nq, Q_TPB), Q_TPB, 0, s>>>(x, x1, qprims, B.qorder, kind, nq, pad, B.n, B.leafv.p, B.rank.p, B.wide.p, B.nodes.p,
                                     scratch.p, counter.p, cap);
    B.launches += 1;
    int cnt2[2] = {0, 0};
    if ((e = cudaMemcpyAsync(cnt2, counter.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    if (cnt2[1]) return cudaErrorLaunchOutOfResources;  // traversal stack overflow (cannot happen with unique keys)
    int cnt = cnt2[0];
    if (cnt < 0 || cnt > (1 << 26)) return cudaErrorMemoryAllocation;  // > 64M candidate pairs: refuse instead of exhausting memory
    if (cnt <= cap) { *npairs = cnt; break; }
    if ((e = scratch.reserve(size_t(cnt) + size_t(cnt) / 4))) return e;
  }
  const int m = *npairs;
  if (m == 0) return cudaSuccess;
  B.launches += 2;
  return sort_pairs(scratch.p, m, nq, B.n, out, k0, k1, tmp, s);
}
}  // namespace

// Query the hierarchy; returns the sorted (query, primitive) pairs in `out`
// (capacity grown as needed) and their number in *npairs.
cudaError_t Lbvh::query(const double* x, const double* x1, int kind, const int* qprims, int nq, float pad, DevBuf<int2>& out,
                        DevBuf<int2>& scratch, DevBuf<unsigned long long>& k0, DevBuf<unsigned long long>& k1,
                        DevBuf<int>& counter, DevBuf<unsigned char>& tmp, int* npairs, cudaStream_t s) {
  return run_query(*this, x, x1, kind, qprims, nq, pad, out, scratch, k0, k1, counter, tmp, npairs, s);
}

cudaError_t Lbvh::contacts_launch(const double* x, int kind, const int* qprims, int nq, float pad, double gap, DevBuf<int2>& scratch,
                                  DevBuf<int>& counter, cudaStream_t s) {
  cudaError_t e;
  if ((e = counter.reserve(3))) return e;
  if ((e = cudaMemsetAsync(counter.p, 0, 3 * sizeof(int), s))) return e;
  if (n == 0 || nq == 0) return cudaSuccess;
  if (scratch.n < 1024) if ((e = scratch.reserve(1024))) return e;
  if ((e = surv.reserve(scratch.n))) return e;
  const int cap = int(scratch.n);
  k_query<<<nblk(nq, Q_TPB), Q_TPB, 0, s>>>(x, nullptr, qprims, qorder, kind, nq, pad, n, leafv.p, rank.p, wide.p, nodes.p, scratch.p, counter.p, cap);
  k_pairs_gap<<<NARROW_GRID, TPB, 0, s>>>(scratch.p, counter.p, cap, kind, prims, qprims, x, gap, surv.p, counter.p + 2);
  launches += 2;
  return cudaGetLastError();
}

cudaError_t Lbvh::contacts_finish(const int count[3], int nq, DevBuf<int2>& out, DevBuf<unsigned long long>& k0, DevBuf<unsigned long long>& k1,
                                  DevBuf<unsigned char>& tmp, int* npairs, cudaStream_t s) {
  cudaError_t e;
  *npairs = 0;
  if (count[1]) return cudaErrorLaunchOutOfResources;  // traversal stack overflow (cannot happen with unique keys)
  const int m = count[2];
  if (m < 0 || m > int(surv.n)) return cudaErrorInvalidValue;
  if (m == 0) return cudaSuccess;
  launches += 2;
  if ((e = sort_pairs(surv.p, m, nq, n, out, k0, k1, tmp, s))) return e;
  *npairs = m;
  return cudaSuccess;
}

cudaError_t Lbvh::query_toi(const double* x, const double* x1, const double* ext, int kind, const int* qprims, int nq, float pad,
                            double eta_min, double near, unsigned long long* toi, DevBuf<int2>& scratch, DevBuf<int>& counter,
                            int* overflow, cudaStream_t s) {
  if (n == 0 || nq == 0) return cudaSuccess;
  cudaError_t e;
  if ((e = counter.reserve(3))) return e;
  if (scratch.n < 1024) if ((e = scratch.reserve(1024))) return e;
  const int cap = int(scratch.n);
  if ((e = cudaMemsetAsync(counter.p, 0, 3 * sizeof(int), s))) return e;
  k_query<<<nblk(nq, Q_TPB), Q_TPB, 0, s>>>(x, x1, qprims, qorder, kind, nq, pad, n, leafv.p, rank.p, wide.p, nodes.p, scratch.p, counter.p, cap);
  k_pairs_toi<<<NARROW_GRID, TPB, 0, s>>>(scratch.p, counter.p, cap, kind, prims, qprims, x, x1, ext, pad, eta_min, near, toi, overflow);
  launches += 2;
  return cudaGetLastError();
}

cudaError_t Lbvh::contacts_from(const double* x, int kind, const int* qprims, double gap, DevBuf<int2>& cand, DevBuf<int>& counter,
                                cudaStream_t s) {
  cudaError_t e;
  if ((e = counter.reserve(3))) return e;
  if (n == 0 || cand.n == 0) return cudaMemsetAsync(counter.p, 0, 3 * sizeof(int), s);
  if ((e = cudaMemsetAsync(counter.p + 2, 0, sizeof(int), s))) return e;
  if ((e = surv.reserve(cand.n))) return e;
  k_pairs_gap<<<NARROW_GRID, TPB, 0, s>>>(cand.p, counter.p, int(cand.n), kind, prims, qprims, x, gap, surv.p, counter.p + 2);
  launches += 1;
  return cudaGetLastError();
}

// Edge-triangle crossings at x over this triangle hierarchy (built at x):
// queries are the ne edges (their boxes inflated by pad, which only adds
// candidates for the exact test). One host round trip per attempt; the
// candidate list grows once if it overflowed.
cudaError_t Lbvh::count_crossings(const double* x, const int* edges, int ne, float pad, DevBuf<int2>& scratch, DevBuf<int>& counter,
                                  DevBuf<unsigned long long>& total, long long* crossings, cudaStream_t s) {
  cudaError_t e;
  *crossings = 0;
  if (n == 0 || ne == 0) return cudaSuccess;
  if ((e = counter.reserve(3))) return e;
  if ((e = total.reserve(1))) return e;
  if (scratch.n < 1024) if ((e = scratch.reserve(1024))) return e;
  for (int attempt = 0; attempt < 2; ++attempt) {
    const int cap = int(scratch.n);
    if ((e = cudaMemsetAsync(counter.p, 0, 3 * sizeof(int), s))) return e;
    if ((e = cudaMemsetAsync(total.p, 0, sizeof(unsigned long long), s))) return e;
    k_query<<<nblk(ne, Q_TPB), Q_TPB, 0, s>>>(x, nullptr, edges, qorder, 2, ne, pad, n, leafv.p, rank.p, wide.p, nodes.p, scratch.p, counter.p, cap);
    k_pairs_cross<<<NARROW_GRID, TPB, 0, s>>>(scratch.p, counter.p, cap, prims, edges, x, total.p);
    launches += 2;
    int cnt2[2] = {0, 0};
    unsigned long long got = 0;
    if ((e = cudaMemcpyAsync(cnt2, counter.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaMemcpyAsync(&got, total.p, sizeof(got), cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    if (cnt2[1]) return cudaErrorLaunchOutOfResources;  // traversal stack overflow (cannot happen with unique keys)
    if (cnt2[0] < 0 || cnt2[0] > (1 << 26)) return cudaErrorMemoryAllocation;
    if (cnt2[0] <= cap) { *crossings = (long long)got; return cudaSuccess; }
    if ((e = scratch.reserve(size_t(cnt2[0]) + size_t(cnt2[0]) / 4))) return e;
  }
  return cudaErrorMemoryAllocation;
}

}  // namespace ando
