// Time-tree operations around the likelihood, batched over samples:
//
// * node-height ratio transform and its log-determinant
//   (torchtree/evolution/tree_height_transform.py:7-99, GeneralNodeHeightTransform):
//     h[root] = x[root];  h[v] = lb[v] + x[v] (h[parent v] - lb[v]) in pre-order,
//     log|J| = sum over non-root internal v of log(h[parent v] - lb[v]),
//   with lb[v] the largest sampling time below v, plus branch lengths
//   h[parent] - h[child] (tree_model.py:23-40);
// * constant-size coalescent log-density
//   (torchtree/evolution/coalescent.py:86-134, ConstantCoalescent.log_prob):
//     log p = -sum_i C(l_i, 2) (t_(i+1) - t_i) / theta - (T - 1) log theta
//   over the sorted node heights t with l_i lineages between t_i and t_(i+1).
//
// One CTA per sample.  The transform walks the tree level by level (all nodes
// of one depth in parallel, a barrier between depths) on the sample's row in
// shared memory, loaded and stored coalesced; its adjoint walks the levels
// back, each parent gathering its internal children's terms (fixed order, no
// atomics).  The coalescent sorts the sample's internal heights in registers
// and walks their merge with the tip times (sorted once at set-up).
//
// FP64 instructions take 16 cycles of an SM each here, so they are what the
// kernels save: log|J| is the logarithm of one running product (a
// multiplication per node instead of a logarithm of ~40), the sort and the
// merge compare heights as integers, and the pair counts C(l, 2) come from a
// table.  1,000 tips x 16,384 samples, before (logarithm per node; bitonic sort
// and binary searches on doubles in shared memory) -> now: transform
// 1,489 -> 297 us, coalescent 4,422 -> 403 us, adjoint 1,077 -> 647 us.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/torchtree_gb300.h"
#include "tt_common.cuh"
#include "tt_launch.h"

struct tt_time_tree {
  int device = 0;
  int T = 0;
  int levels = 0;               // depths of internal nodes (root: depth 0)
  int4 *d_lvl = nullptr;        // [T-1] internal nodes by depth, root first: node, parent (indices - T), lower bound
  int4 *d_lvl_kids = nullptr;   // [T-1] in the same order: node, left, right (index - T, negative: tip)
  int *d_lvl_off = nullptr;     // [levels + 1] offsets into the two
  int2 *d_kids = nullptr;       // [T-1] children (node indices) of internal node index - T
  int *d_parent = nullptr;      // [2T-2] parent node index of every non-root node
  double *d_lb = nullptr;       // [T-1] lower bounds of internal nodes
  double *d_times = nullptr;    // [T] sampling times
  unsigned long long *d_tip_key = nullptr;  // [T] sampling times in ascending order, as ordered integers
  double *d_pairs = nullptr;    // [2T+1] C(l, 2) for l = -T .. T lineages
};

namespace {

constexpr int kTimeTreeThreads = 128;  // threads of the per-sample transform CTAs

int tfail(int code, const std::string &m) { return tt::record_error(code, m.c_str()); }

// A product kept as mantissa and exponent: factors in (0, inf) multiply the
// mantissa (in [1, 2) after each step) and add to the exponent; any other factor
// goes through its logarithm.
struct LogProduct {
  double m = 1.0, rest = 0.0;
  int e = 0;
  __device__ __forceinline__ void renorm() {
    const int hi = __double2hiint(m);
    e += (hi >> 20) - 1023;
    m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(m));
  }
  __device__ __forceinline__ void times(double x) {
    const int hi = __double2hiint(x), be = hi >> 20;
    if (be > 0 && be < 0x7ff) {  // positive, normal, finite
      e += be - 1023;
      m *= __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
      renorm();
    } else {
      rest += log(x);
    }
  }
  __device__ __forceinline__ void join(double om, int oe, double orest) {
    m *= om;
    e += oe;
    renorm();
    rest += orest;
  }
  __device__ __forceinline__ double value() const { return fma(double(e), 0.69314718055994530942, log(m)) + rest; }
};

__global__ void __launch_bounds__(kTimeTreeThreads)
    ratio_forward_kernel(const int4 *lvl, const int *lvl_off, int levels, const int *parent, const double *times,
                         const double *x, double *h, double *bl, double *logdet, int T) {
  extern __shared__ __align__(16) double rs[];
  __shared__ double wm[32], wr[32];
  __shared__ int we[32];
  const int b = blockIdx.x, tid = threadIdx.x, NT = blockDim.x, I = T - 1;
  double *hs = rs;  // this sample's ratios, each overwritten by its node's height
  const double *xb = x + size_t(b) * I;
#pragma unroll 4
  for (int v = tid; v < I; v += NT) hs[v] = xb[v];
  // the level table does not depend on the sample's values: each thread reads its next entry a level ahead
  int off = 1, end = levels > 1 ? lvl_off[2] : 1;
  int4 nxt = make_int4(0, 0, 0, 0);
  if (off + tid < end) nxt = lvl[off + tid];
  __syncthreads();  // the root's ratio is its height
  LogProduct ld;
  for (int d = 1; d < levels; ++d) {  // one depth at a time, parents before children
    const int off2 = end, end2 = d + 1 < levels ? lvl_off[d + 2] : end;
    int4 r = nxt;
    if (off2 + tid < end2) nxt = lvl[off2 + tid];
    for (int e = off + tid; e < end; e += NT) {
      if (e != off + tid) r = lvl[e];
      const double lb = __hiloint2double(r.w, r.z), span = hs[r.y] - lb;
      hs[r.x] = lb + hs[r.x] * span;
      ld.times(span);
    }
    off = off2;
    end = end2;
    __syncthreads();
  }
  // the product over the CTA in a fixed order (warps, then warp totals)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    ld.join(__shfl_down_sync(0xffffffffu, ld.m, o), __shfl_down_sync(0xffffffffu, ld.e, o),
            __shfl_down_sync(0xffffffffu, ld.rest, o));
  if ((tid & 31) == 0) wm[tid >> 5] = ld.m, we[tid >> 5] = ld.e, wr[tid >> 5] = ld.rest;
  double *hb = h + size_t(b) * I;
#pragma unroll 4
  for (int v = tid; v < I; v += NT) hb[v] = hs[v];
  if (bl) {
    double *blb = bl + size_t(b) * (2 * T - 2);
#pragma unroll 4
    for (int n = tid; n < 2 * T - 2; n += NT) {
      const double hn = n < T ? times[n] : hs[n - T];
      blb[n] = hs[parent[n] - T] - hn;
    }
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < (NT + 31) >> 5; ++w) ld.join(wm[w], we[w], wr[w]);
    logdet[b] = ld.value();
  }
}

// dlnL/dx from dlnL/dh, dlnL/dbranch lengths and dlnL/dlog|J|
//
// What does not depend on the children's gradients (the spans, their divisions,
// the branch lengths' terms) is done for every node at once, all lanes busy; the
// walk over the depths, where a level of a few nodes costs a whole warp
// instruction, keeps one multiplication and one FMA per child.  The two row
// buffers are used in turn: branch-length gradients, heights, then spans and
// log-span terms, then spans and ratios.  1,000 tips x 16,384 samples: 1,050
// (division inside the walk, branch-length gradients gathered from global
// memory) -> 647 us.
constexpr int kNodesPerThread = 10;  // 9,600 tips at 1,024 threads

__global__ void ratio_backward_kernel(const int4 *lvl_kids, const int *lvl_off, int levels, const int2 *kids,
                                      const int *parent, const double *lb, const double *x, const double *h,
                                      const double *gh_in, const double *gbl, const double *gld, double *gx, int T) {
  extern __shared__ __align__(16) double rs[];
  const int b = blockIdx.x, tid = threadIdx.x, NT = blockDim.x, I = T - 1, B = 2 * T - 2;
  double *xs = rs, *hs = rs + I, *g = rs + 2 * I;
  if (gbl) {
#pragma unroll 4
    for (int c = tid; c < B; c += NT) rs[c] = gbl[size_t(b) * B + c];  // B = 2 I: both row buffers
    __syncthreads();
  }
#pragma unroll 2
  for (int v = tid; v < I; v += NT) {
    double gv = gh_in ? gh_in[size_t(b) * I + v] : 0.0;
    if (gbl) {  // branch c above node c has length h[parent c] - h[c]
      const int2 k = kids[v];
      gv += rs[k.x] + rs[k.y];
      if (v < I - 1) gv -= rs[v + T];
    }
    g[v] = gv;
  }
  __syncthreads();
#pragma unroll 4
  for (int v = tid; v < I; v += NT) hs[v] = h[size_t(b) * I + v];
  __syncthreads();
  const double gl = gld ? gld[b] : 0.0;
  double span[kNodesPerThread];
#pragma unroll
  for (int i = 0; i < kNodesPerThread; ++i) {
    const int v = tid + i * NT;
    if (v < I - 1) span[i] = hs[parent[v + T] - T] - lb[v];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kNodesPerThread; ++i) {
    const int v = tid + i * NT;
    if (v < I - 1) {
      hs[v] = span[i];
      xs[v] = gl / span[i];  // d log(span)/dh_parent
    }
  }
  __syncthreads();
#pragma unroll 2
  for (int v = tid; v < I; v += NT) {
    const int2 k = kids[v];
    double gv = g[v];
    if (k.x >= T) gv += xs[k.x - T];
    if (k.y >= T) gv += xs[k.y - T];
    g[v] = gv;
  }
  __syncthreads();
#pragma unroll 4
  for (int v = tid; v < I; v += NT) xs[v] = x[size_t(b) * I + v];
  // deepest parents first: a parent gathers d/dh of its internal children,
  // which are final, then turns them into d/dx.  Each thread reads its next
  // table entry a level ahead.
  int off = 0, end = 0;
  int4 nxt = make_int4(0, 0, 0, 0);
  if (levels > 1) {
    off = lvl_off[levels - 2];
    end = lvl_off[levels - 1];
    if (off + tid < end) nxt = lvl_kids[off + tid];
  }
  __syncthreads();
  for (int d = levels - 2; d >= 0; --d) {
    const int end2 = off, off2 = d > 0 ? lvl_off[d - 1] : off;
    int4 r = nxt;
    if (off2 + tid < end2) nxt = lvl_kids[off2 + tid];
    for (int e = off + tid; e < end; e += NT) {
      if (e != off + tid) r = lvl_kids[e];
      double gp = g[r.x];
      const int c2[2] = {r.y, r.z};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int cv = c2[c];
        if (cv < 0) continue;
        const double gc = g[cv];
        g[cv] = gc * hs[cv];        // dh_c/dx_c = span
        gp = fma(gc, xs[cv], gp);   // dh_c/dh_p = x_c
      }
      g[r.x] = gp;
    }
    off = off2;
    end = end2;
    __syncthreads();
  }
  // the root entry keeps d/dh[root] (h_root = x_root)
#pragma unroll 4
  for (int v = tid; v < I; v += NT) gx[size_t(b) * I + v] = g[v];
}

// Doubles as integers of the same order (-0 as +0), and back.
__host__ __device__ inline unsigned long long ordered_key(double v) {
  long long bits;
#ifdef __CUDA_ARCH__
  bits = __double_as_longlong(v);
#else
  std::memcpy(&bits, &v, 8);
#endif
  if (bits == (long long)0x8000000000000000ull) bits = 0;
  return (unsigned long long)bits ^ ((unsigned long long)(bits >> 63) | 0x8000000000000000ull);
}
__device__ __forceinline__ double ordered_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k ^ 0x8000000000000000ull : ~k));
}

constexpr int kSortPerThread = 8, kSortIndexBits = 12;  // up to 4,096 heights

// One compare-exchange stage (partner e ^ j, ascending where (e & k) == 0) of a
// bitonic sort of 8 keys per thread, element e = 8 tid + r: within the thread, by
// warp shuffles, or through shared memory (buf, keys stored [r][thread]).
__device__ __forceinline__ void sort_stage(unsigned long long (&key)[8], int k, int j, unsigned long long *buf) {
  const int tid = threadIdx.x, NT = blockDim.x;
  if (j < 8) {
#pragma unroll
    for (int jj = 4; jj > 0; jj >>= 1)
      if (jj == j) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (!(r & jj)) {
            const bool up = ((8 * tid + r) & k) == 0;
            const unsigned long long a = key[r], c = key[r | jj];
            const bool keep = (a < c) == up;
            key[r] = keep ? a : c;
            key[r | jj] = keep ? c : a;
          }
      }
    return;
  }
  const int jt = j >> 3;
  const bool low = ((tid & jt) == 0) == (((8 * tid) & k) == 0);  // keep the smaller key
  if (jt < 32) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, key[r], jt);
      key[r] = (key[r] < o) == low ? key[r] : o;
    }
    return;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) buf[r * NT + tid] = key[r];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const unsigned long long o = buf[r * NT + (tid ^ jt)];
    key[r] = (key[r] < o) == low ? key[r] : o;
  }
}

// One CTA per sample, 8 internal heights per thread (m2 = 8 blockDim.x >= T - 1).
// 1. Sort: a 64-bit key holds the ordered height without its lowest 12 bits and
//    the node's index in their place (so ties sort by node index, one compare and
//    two selects per key).  Heights that differ in those 12 bits only (2^-40
//    relative) may come out in index order; if any neighbours do, the CTA sorts
//    again in shared memory on the whole height.
// 2. Merge: thread t takes merged positions [t E, (t+1) E) (its start by a binary
//    search along the diagonal; a tip precedes an internal node of equal height).
//    The lineages through position p are L_p = (tips - internal nodes at or before
//    p); with c_p = C(L_p, 2) for p < n - 1 (0 at the last):
//      log p = -sum_p c_p (t_{p+1} - t_p) / theta - (T - 1) log theta,
//      d/dt_p = (c_p - c_{p-1}) / theta  (each internal node written once),
//      d/dtheta = sum_p c_p (t_{p+1} - t_p) / theta^2 - (T - 1) / theta.
//    The sum runs in a fixed order (per-thread runs, then warps, then warp totals).
__global__ void coalescent_kernel(const unsigned long long *tip_key, const double *pairs, const double *hint,
                                  const double *theta, int T, double *logp, double *gh, double *gtheta) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int b = blockIdx.x, tid = threadIdx.x, NT = blockDim.x, m2 = 8 * NT;
  const int n = 2 * T - 1, I = T - 1;
  unsigned long long *raw = reinterpret_cast<unsigned long long *>(sm);  // [m2] ordered heights by node; then gradients
  unsigned long long *sk = raw + m2;                                     // [m2] ordered heights, sorted
  unsigned short *si = reinterpret_cast<unsigned short *>(sk + m2);      // [m2] their nodes (index - T)
  const double *hb = hint + size_t(b) * I;
#pragma unroll 4
  for (int e = tid; e < m2; e += NT) raw[e] = e < I ? ordered_key(hb[e]) : ~0ull;
  __syncthreads();
  constexpr unsigned long long kIdx = (1ull << kSortIndexBits) - 1;
  unsigned long long key[kSortPerThread];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int e = 8 * tid + r;
    key[r] = e < I ? (raw[e] & ~kIdx) | unsigned(e) : ~0ull;  // (no height's key is all ones: that is a NaN's)
  }
#pragma unroll
  for (int k = 2; k <= 8; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) sort_stage(key, k, j, sk);
  for (int k = 16; k <= m2; k <<= 1) {
    for (int j = k >> 1; j >= 8; j >>= 1) sort_stage(key, k, j, sk);
#pragma unroll
    for (int j = 4; j > 0; j >>= 1) sort_stage(key, k, j, sk);
  }
  __syncthreads();  // sk's last exchange has been read
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int e = 8 * tid + r, node = int(key[r] & kIdx);
    si[e] = static_cast<unsigned short>(node);
    sk[e] = e < I && node < I ? raw[node] : ~0ull;
  }
  __syncthreads();
  bool unsorted = false;
  for (int e = tid; e + 1 < I; e += NT) unsorted |= sk[e] > sk[e + 1];
  if (__syncthreads_or(unsorted)) {  // close heights: sort on the whole key, ties by node
    for (int k = 2; k <= m2; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int e = tid; e < m2; e += NT) {
          const int o = e ^ j;
          if (o > e) {
            const unsigned long long ke = sk[e], ko = sk[o];
            const unsigned short ie = si[e], io = si[o];
            if ((ke > ko || (ke == ko && ie > io)) == ((e & k) == 0)) {
              sk[e] = ko, sk[o] = ke;
              si[e] = io, si[o] = ie;
            }
          }
        }
        __syncthreads();
      }
  }
  double *g = reinterpret_cast<double *>(raw);  // [I] d/dheight by node
  const double th = theta[b], inv_th = 1.0 / th;
  const int E = (n + NT - 1) / NT;
  const int p0 = min(n, tid * E), p1 = min(n, p0 + E);
  int lo = max(0, p0 - I), hi = min(p0, T);  // tips among the first p0 positions
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (tip_key[mid] <= sk[p0 - 1 - mid]) lo = mid + 1;
    else hi = mid;
  }
  int jt = lo, ji = p0 - lo, L = jt - ji;
  double acc = 0.0;
  unsigned long long kt = jt < T ? tip_key[jt] : ~0ull, ki = ji < I ? sk[ji] : ~0ull;
  bool tip = jt < T && (ji >= I || kt <= ki);
  double cur = ordered_value(tip ? kt : ki), c_prev = p0 > 0 ? pairs[L + T] : 0.0;
  for (int p = p0; p < p1; ++p) {
    const int node = tip ? -1 : si[ji];
    if (tip) {
      ++L;
      kt = ++jt < T ? tip_key[jt] : ~0ull;
    } else {
      --L;
      ki = ++ji < I ? sk[ji] : ~0ull;
    }
    const double c = p < n - 1 ? pairs[L + T] : 0.0;
    tip = jt < T && (ji >= I || kt <= ki);
    const double next = ordered_value(tip ? kt : ki);
    if (p < n - 1) acc = fma(c, next - cur, acc);
    if (node >= 0) g[node] = (c - c_prev) * inv_th;
    c_prev = c;
    cur = next;
  }
  __shared__ double wacc[32];
  const int lane = tid & 31, warp = tid >> 5, NW = (NT + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0) wacc[warp] = acc;
  __syncthreads();
  if (gh) {
#pragma unroll 4
    for (int v = tid; v < I; v += NT) gh[size_t(b) * I + v] = g[v];
  }
  if (tid == 0) {
    double total = 0.0;
    for (int w = 0; w < NW; ++w) total += wacc[w];
    logp[b] = -total * inv_th - double(T - 1) * log(th);
    if (gtheta) gtheta[b] = total * inv_th * inv_th - double(T - 1) * inv_th;
  }
}

}  // namespace

extern "C" {

int tt_time_tree_create(tt_time_tree **tree, int32_t tip_count, const int32_t *postorder,
                        const double *sampling_times) {
  if (!tree || !postorder || !sampling_times) return tfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  *tree = nullptr;
  const int T = tip_count, I = T - 1, NN = 2 * T - 1;
  if (T < 2) return tfail(TT_ERR_INVALID_ARGUMENT, "a tree needs at least 2 tips");
  std::vector<int> parent(NN, -1), left(NN, -1), right(NN, -1);
  std::vector<char> done(NN, 0);
  for (int t = 0; t < T; ++t) done[t] = 1;
  for (int s = 0; s < I; ++s) {
    const int v = postorder[3 * s], l = postorder[3 * s + 1], r = postorder[3 * s + 2];
    if (v < T || v >= NN || l < 0 || l >= NN || r < 0 || r >= NN || done[v] || !done[l] || !done[r] ||
        parent[l] >= 0 || parent[r] >= 0 || l == r)
      return tfail(TT_ERR_INVALID_ARGUMENT, "postorder is not a valid post-order of a binary tree");
    parent[l] = v, parent[r] = v, left[v] = l, right[v] = r, done[v] = 1;
  }
  if (postorder[3 * (I - 1)] != NN - 1) return tfail(TT_ERR_INVALID_ARGUMENT, "the root must be node 2T-2, last");
  std::vector<double> lb(I, 0.0);
  for (int s = 0; s < I; ++s) {
    const int v = postorder[3 * s];
    auto h = [&](int c) { return c < T ? sampling_times[c] : lb[c - T]; };
    lb[v - T] = std::max(h(left[v]), h(right[v]));
  }
  // internal nodes by depth (root at depth 0; a parent precedes its children)
  std::vector<int> depth(NN, 0);
  int levels = 1;
  for (int s = I - 1; s >= 0; --s) {  // reversed post-order: parents first
    const int v = postorder[3 * s];
    if (v != NN - 1) depth[v] = depth[parent[v]] + 1;
    levels = std::max(levels, depth[v] + 1);
  }
  std::vector<int> lvl_off(levels + 1, 0), lvl_nodes;
  lvl_nodes.reserve(I);
  for (int d = 0; d < levels; ++d) {
    lvl_off[d] = int(lvl_nodes.size());
    for (int v = T; v < NN; ++v)
      if (depth[v] == d) lvl_nodes.push_back(v - T);
  }
  lvl_off[levels] = int(lvl_nodes.size());
  std::vector<int2> kids(I);
  for (int v = T; v < NN; ++v) kids[v - T] = make_int2(left[v], right[v]);
  std::vector<int4> lvl(I), lvl_kids(I);
  for (int e = 0; e < I; ++e) {
    const int v = lvl_nodes[e], pv = v + T == NN - 1 ? 0 : parent[v + T] - T;
    int2 bits;
    std::memcpy(&bits, &lb[v], 8);
    lvl[e] = make_int4(v, pv, bits.x, bits.y);
    lvl_kids[e] = make_int4(v, left[v + T] - T, right[v + T] - T, 0);
  }
  std::vector<unsigned long long> tip_key(T);  // sampling times in ascending order
  for (int i = 0; i < T; ++i) tip_key[i] = ordered_key(sampling_times[i]);
  std::sort(tip_key.begin(), tip_key.end());
  std::vector<double> pairs(2 * size_t(T) + 1);  // lineages lie in [-(T - 1), T]
  for (int l = -T; l <= T; ++l) pairs[l + T] = 0.5 * double(l) * double(l - 1);
  tt_time_tree *t = new tt_time_tree();
  cudaGetDevice(&t->device);
  t->T = T;
  t->levels = levels;
  cudaError_t e = cudaSuccess;
  auto up = [&](auto **dst, const auto *src, size_t n) {
    if (e != cudaSuccess) return;
    e = cudaMalloc(reinterpret_cast<void **>(dst), std::max<size_t>(n, 1) * sizeof(**dst));
    if (e == cudaSuccess && n) e = cudaMemcpy(*dst, src, n * sizeof(**dst), cudaMemcpyHostToDevice);
  };
  up(&t->d_lvl, lvl.data(), lvl.size());
  up(&t->d_lvl_kids, lvl_kids.data(), lvl_kids.size());
  up(&t->d_lvl_off, lvl_off.data(), lvl_off.size());
  up(&t->d_kids, kids.data(), kids.size());
  up(&t->d_parent, parent.data(), size_t(2 * T - 2));
  up(&t->d_lb, lb.data(), lb.size());
  up(&t->d_times, sampling_times, size_t(T));
  up(&t->d_tip_key, tip_key.data(), tip_key.size());
  up(&t->d_pairs, pairs.data(), pairs.size());
  if (e != cudaSuccess) {
    tt_time_tree_destroy(t);
    return tfail(TT_ERR_OUT_OF_MEMORY, std::string("time-tree upload: ") + cudaGetErrorString(e));
  }
  *tree = t;
  return TT_OK;
}

int tt_time_tree_destroy(tt_time_tree *t) {
  if (!t) return TT_OK;
  void *bufs[] = {t->d_lvl, t->d_lvl_kids, t->d_lvl_off, t->d_kids, t->d_parent, t->d_lb, t->d_times, t->d_tip_key,
                  t->d_pairs};
  for (void *p : bufs)
    if (p) cudaFree(p);
  delete t;
  return TT_OK;
}

int tt_ratio_transform(tt_time_tree *t, int32_t batch, const double *ratios, double *heights,
                       double *branch_lengths, double *log_det_jacobian, void *stream) {
  if (!t || !ratios || !heights || !log_det_jacobian || batch < 1)
    return tfail(TT_ERR_INVALID_ARGUMENT, "NULL argument or empty batch");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t smem = size_t(t->T - 1) * sizeof(double);
  if (3 * size_t(t->T - 1) * sizeof(double) > 227 * 1024)
    return tfail(TT_ERR_UNSUPPORTED, "the ratio transform holds a sample's rows in shared memory: at most 9,600 tips");
  cudaError_t e = tt::kernel_smem(ratio_forward_kernel, smem);
  if (e == cudaSuccess) {
    ratio_forward_kernel<<<batch, kTimeTreeThreads, smem, s>>>(t->d_lvl, t->d_lvl_off, t->levels, t->d_parent,
                                                               t->d_times, ratios, heights, branch_lengths,
                                                               log_det_jacobian, t->T);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? TT_OK : tfail(TT_ERR_CUDA, std::string("ratio transform launch: ") + cudaGetErrorString(e));
}

int tt_ratio_transform_backward(tt_time_tree *t, int32_t batch, const double *ratios, const double *heights,
                                const double *grad_heights, const double *grad_branch_lengths,
                                const double *grad_log_det, double *grad_ratios, void *stream) {
  if (!t || !ratios || !heights || !grad_ratios || batch < 1)
    return tfail(TT_ERR_INVALID_ARGUMENT, "NULL argument or empty batch");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t smem = 3 * size_t(t->T - 1) * sizeof(double);
  if (smem > 227 * 1024)
    return tfail(TT_ERR_UNSUPPORTED, "the ratio transform holds a sample's rows in shared memory: at most 9,600 tips");
  cudaError_t e = tt::kernel_smem(ratio_backward_kernel, smem);
  if (e == cudaSuccess) {
    int threads = kTimeTreeThreads;
    while (threads * kNodesPerThread < t->T - 1) threads *= 2;  // at most 1,024: the rows fit up to 9,600 tips
    ratio_backward_kernel<<<batch, threads, smem, s>>>(t->d_lvl_kids, t->d_lvl_off, t->levels, t->d_kids, t->d_parent,
                                                       t->d_lb, ratios, heights, grad_heights, grad_branch_lengths,
                                                       grad_log_det, grad_ratios, t->T);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? TT_OK
                          : tfail(TT_ERR_CUDA, std::string("ratio transform backward launch: ") + cudaGetErrorString(e));
}

int tt_constant_coalescent(tt_time_tree *t, int32_t batch, const double *heights, const double *theta,
                           double *log_prob, double *grad_heights, double *grad_theta, void *stream) {
  if (!t || !heights || !theta || !log_prob || batch < 1)
    return tfail(TT_ERR_INVALID_ARGUMENT, "NULL argument or empty batch");
  const int T = t->T, I = T - 1;
  if (T > 4096) return tfail(TT_ERR_UNSUPPORTED, "the coalescent kernel sorts at most 4,096 tips");
  int m2 = 32 * kSortPerThread;
  while (m2 < I) m2 <<= 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t smem = size_t(m2) * (2 * sizeof(unsigned long long) + sizeof(unsigned short));
  cudaError_t e = tt::kernel_smem(coalescent_kernel, smem);
  if (e == cudaSuccess) {  // every internal node's gradient is written once: no clearing needed
    coalescent_kernel<<<batch, m2 / kSortPerThread, smem, s>>>(t->d_tip_key, t->d_pairs, heights, theta, T, log_prob,
                                                               grad_heights, grad_theta);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? TT_OK : tfail(TT_ERR_CUDA, std::string("coalescent launch: ") + cudaGetErrorString(e));
}

}  // extern "C"
