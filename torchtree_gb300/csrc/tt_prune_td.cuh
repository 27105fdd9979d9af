// FP64 pruning kernels of 4-state plans: the drop-in precision.
//
// Bound by the FP64 pipe: one warp instruction per 64 cycles and SM quarter
// (measured: 31 ns for DFMA, DADD and DMUL alike, whatever the number of
// chains; fmax 3.4 and a division 9 of those), so the count of FP64
// instructions is the time and everything else hides behind it.  Hence:
//  * a tile of 32 / KP patterns (KP = categories padded to 1, 2, 4 or 8), one thread
//    per (pattern, category), on a CTA of two warps: one walks the tree, the other
//    stages the steps and, in the adjoint, sums the gradients, so that little but FP64
//    instructions is on the walk, which is all the time of a small alignment;
//  * a tip with an unambiguous state takes its matrix's column (no product), and
//    its gradient is one addition per pattern and row, its state picking the
//    accumulator by selects;
//  * maxima, power-of-two scaling and exponents run on the integer pipe;
//  * the adjoint divides once per pattern, at the root: the outside partial of
//    the root carries w / L, and stored exponents keep every later product's
//    scale, so no node forms its own denominator.
// The adjoint's warps each walk several tiles and add into one gradient block
// per (branch, warp), so the blocks stay few at a tile of 8 patterns.
//
// Lane = category * PW + pattern (PW = 32 / KP): a category's lanes read one
// matrix (broadcast) and a contiguous run of partials.  Per step a lane copies
// its share of the matrices, its own child vectors, the tip codes and exponents
// into a ring by cp.async, two or three steps ahead.
//
// Measured (GB300), post-order / adjoint: 64-pattern CTAs, one thread per pattern, all
// categories, tips as products -> one warp per tile -> two warps per tile:
//   69 taxa x 238 patterns x 1:                         109 / 283 ->    95 / 179 us
//   87 taxa x 611 patterns x 3:      681 / 1,847 ->     135 / 355 ->   118 / 230 us
//   500 taxa x 6,584 patterns x 4: 4,996 / 31,916 -> 2,526 / 7,385 -> 2,394 / 7,000 us
#pragma once

#include "tt_common.cuh"
#include "tt_prune.cuh"

namespace tt {

// lanes per pattern: the category count padded to a power of two
__host__ __device__ inline int td_lanes(int K) { return K <= 1 ? 1 : (K <= 2 ? 2 : (K <= 4 ? 4 : 8)); }
// patterns per warp
__host__ __device__ inline int td_tile(int K) { return 32 / td_lanes(K); }

constexpr int kTdFwdStages = 4, kTdBwdStages = 3;

struct TdLayout {
  // within a stage
  int rec, codes, expo, pm, kids, stage;
  // whole CTA
  int stages, table, onehot, stack, sexp, ubuf, total;
};

__host__ __device__ inline TdLayout td_layout(int K, int C, int slots, bool backward) {
  const int KP = td_lanes(K), PW = 32 / KP;
  TdLayout L;
  int off = 0;
  L.rec = off, off += 48;
  L.codes = off, off += 2 * 32;
  L.expo = off, off += 2 * PW * 4;
  off = int(align16(off));
  L.pm = off, off += 2 * K * 128;
  L.kids = off;
  if (backward) off += 2 * KP * (PW * 32 + 16);
  L.stage = off;
  off = 0;
  L.stages = off, off += (backward ? kTdBwdStages : kTdFwdStages) * L.stage;
  L.table = off, off += C * 32;
  L.onehot = off, off = int(align16(off + C));
  L.stack = off, off += slots * 32 * 32;
  L.sexp = off;
  if (backward) off += slots * 32 * 4;
  L.ubuf = off;
  if (backward) off += 2 * 8 * KP * (PW * 8 + 16);
  L.total = off;
  return L;
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
// 16 bytes, or zeros when !on (src is not read)
__device__ __forceinline__ void cp_async16_or_zero(void *dst, const void *src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// What one step reads, into a stage: its record, matrices, tip codes and, in
// the adjoint, the lane's own child vectors and the children's exponents.
template <int KP, bool BACKWARD>
__device__ __forceinline__ void td_issue(const PruneArgs<double> &a, const TdLayout &L, unsigned char *stg,
                                         const int4 (&rec)[3], int s, int b, int tile, int lane) {
  constexpr int PW = 32 / KP;
  const int k = lane / PW, p = lane % PW, n = tile * PW + p;
  const bool on = n < a.N && k < a.K;
  if (lane == 0) {
    int4 *r = reinterpret_cast<int4 *>(stg + L.rec);
    r[0] = rec[0], r[1] = rec[1], r[2] = rec[2];
  }
  const char *pm = reinterpret_cast<const char *>(a.pmat + (size_t(b) * a.n_steps + s) * 2 * a.K * 16);
  for (int c = lane; c < 2 * a.K * 8; c += 32) cp_async<16>(stg + L.pm + c * 16, pm + c * 16);
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int child = side ? rec[0].z : rec[0].y;
    if (child < a.tip_count) {
      constexpr int CB = PW < 16 ? PW : 16;  // tip codes: rows are padded past the last tile
      if (lane < PW / CB)
        cp_async<CB>(stg + L.codes + side * 32 + lane * CB, a.codes + size_t(child) * a.code_stride + tile * PW + lane * CB);
    } else if (BACKWARD) {
      const size_t node = size_t(b) * (a.n_steps - 1) + (child - a.tip_count);
      const double *src = on ? a.partials + ((node * a.K + k) * size_t(a.N) + n) * 4 : a.partials;
      unsigned char *dst = stg + L.kids + (side * KP + k) * (PW * 32 + 16) + p * 32;
      cp_async16_or_zero(dst, src, on);
      cp_async16_or_zero(dst + 16, src + 2, on);
      if (k == 0 && n < a.N) cp_async<4>(stg + L.expo + (side * PW + p) * 4, a.expo + node * a.N + n);
    }
  }
}

// largest of the pattern's 4 KP values (its lanes' v): the exponent that scales
// it into [1, 2), 0 when there is no positive finite value (scale_exponent)
template <int KP>
__device__ __forceinline__ int td_exponent(const double (&v)[4]) {
  constexpr int PW = 32 / KP;
  // positive doubles order as their high words; negative ones fall below zero
  int m = max(max(__double2hiint(v[0]), __double2hiint(v[1])), max(__double2hiint(v[2]), __double2hiint(v[3])));
#pragma unroll
  for (int o = PW; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int be = m >> 20;
  if (__any_sync(0xffffffffu, be <= 0 || be == 0x7ff)) {  // zero, subnormal or not finite: the exact rule
    double x = fmax(fmax(fmax(0.0, v[0]), v[1]), fmax(v[2], v[3]));
#pragma unroll
    for (int o = PW; o < 32; o <<= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
    return scale_exponent(x);
  }
  return be - 1023;
}

// v * 2^-e, exact; on the integer pipe while every value stays normal
__device__ __forceinline__ void td_scale(double (&v)[4], int e) {
  if (e == 0) return;
  bool plain = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int be = (__double2hiint(v[i]) >> 20) & 0x7ff, nb = be - e;
    plain = plain && ((be > 0 && be < 0x7ff && nb > 0 && nb < 0x7ff) || v[i] == 0.0);
  }
  if (plain) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int hi = __double2hiint(v[i]), lo = __double2loint(v[i]);
      v[i] = __hiloint2double((hi & 0x7fffffff) | lo ? hi - (e << 20) : hi, lo);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = times_pow2_neg(v[i], e);
  }
}

// P x of one child: a product for an internal child or an ambiguous tip, the
// state's column for an unambiguous one (the same bits: the other terms are 0)
__device__ __forceinline__ void td_product(double (&out)[4], const double *P, bool tip, int code,
                                           const unsigned char *onehot, const double *tab, double (&v)[4]) {
  if (tip) {
    const int s = onehot[code];
    if (s < 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) out[i] = P[i * 4 + s];
      return;
    }
    load_vec<double, 4>(v, tab + code * 4);
  }
  matvec<double, 4>(out, P, v);
}

__device__ __forceinline__ void td_stack_load(double (&v)[4], const unsigned char *stack, int slot, int lane) {
  const double2 x = reinterpret_cast<const double2 *>(stack)[(slot * 2) * 32 + lane];
  const double2 y = reinterpret_cast<const double2 *>(stack)[(slot * 2 + 1) * 32 + lane];
  v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
}
__device__ __forceinline__ void td_stack_store(const double (&v)[4], unsigned char *stack, int slot, int lane) {
  reinterpret_cast<double2 *>(stack)[(slot * 2) * 32 + lane] = make_double2(v[0], v[1]);
  reinterpret_cast<double2 *>(stack)[(slot * 2 + 1) * 32 + lane] = make_double2(v[2], v[3]);
}

// code table and its one-hot states (255: not a unit vector) into shared memory
__device__ __forceinline__ void td_load_table(const PruneArgs<double> &a, double *tab, unsigned char *onehot, int lane) {
  for (int c = lane; c < a.C; c += 32) {
    int s = 255, ones = 0, zeros = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double x = a.table[c * 4 + j];
      tab[c * 4 + j] = x;
      if (x == 1.0) s = j, ++ones;
      else zeros += x == 0.0;
    }
    onehot[c] = static_cast<unsigned char>(ones == 1 && zeros == 3 ? s : 255);
  }
}

// The two warps of a CTA pass stages and u by named barriers, two of each kind in turn
// (one warp may be a step ahead); every arrival has its wait.  (Immediate barrier
// numbers: a number in a register would take all sixteen, and CTAs per SM with them.)
constexpr int kTdBarFull = 1, kTdBarU = 3, kTdBarFree = 5;  // stage landed, u written, stage read
template <int BAR>
__device__ __forceinline__ void td_arrive(int j) {
  __syncwarp();
  if (j & 1) asm volatile("bar.arrive %0, 64;" ::"n"(BAR + 1) : "memory");
  else asm volatile("bar.arrive %0, 64;" ::"n"(BAR) : "memory");
}
template <int BAR>
__device__ __forceinline__ void td_await(int j) {
  __syncwarp();
  if (j & 1) asm volatile("bar.sync %0, 64;" ::"n"(BAR + 1) : "memory");
  else asm volatile("bar.sync %0, 64;" ::"n"(BAR) : "memory");
}
// -------------------------------------------------------------- post-order
// The first warp walks the tree, the second stages its steps.
template <int KP>
__global__ void __launch_bounds__(64) td_forward_kernel(const PruneArgs<double> a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int PW = 32 / KP, NST = kTdFwdStages;
  const int lane = threadIdx.x % 32, k = lane / PW, p = lane % PW;
  const int tile = blockIdx.x, b = blockIdx.y, n = tile * PW + p, K = a.K, nst = a.n_steps;
  const bool act = n < a.N, kact = k < K;
  const int kk = kact ? k : 0;  // padded lanes read category 0 and contribute zeros
  const TdLayout L = td_layout(K, a.C, a.slots, false);
  double *tab = reinterpret_cast<double *>(smem + L.table);
  unsigned char *onehot = smem + L.onehot, *stack = smem + L.stack;
  if (threadIdx.x >= 32) {
    int4 nxt[3];
    load_rec(nxt, a.steps_ws, 0);
    auto issue = [&](int t) {  // step t, and its group (empty past the last)
      if (t < nst) {
        const int4 cur[3] = {nxt[0], nxt[1], nxt[2]};
        if (t + 1 < nst) load_rec(nxt, a.steps_ws, t + 1);
        td_issue<KP, false>(a, L, smem + L.stages + (t % NST) * L.stage, cur, t, b, tile, lane);
      }
      cp_async_commit();
    };
    for (int s = 0; s < NST; ++s) issue(s);
    cp_async_wait<NST - 1>();
    td_arrive<kTdBarFull>(0);
    for (int s = 0; s < nst; ++s) {
      if (s + 1 < nst) {
        cp_async_wait<NST - 2>();
        td_arrive<kTdBarFull>(s + 1);
      }
      td_await<kTdBarFree>(s);
      issue(s + NST);
    }
    return;
  }
  td_load_table(a, tab, onehot, lane);
  __syncwarp();
  double carry[4] = {0.0, 0.0, 0.0, 0.0};  // the previous step's partial
  int E = 0;
  double ll = 0.0;
  for (int s = 0; s < nst; ++s) {
    td_await<kTdBarFull>(s);
    const unsigned char *stg = smem + L.stages + (s % NST) * L.stage;
    const int4 r0 = reinterpret_cast<const int4 *>(stg + L.rec)[0], r1 = reinterpret_cast<const int4 *>(stg + L.rec)[1];
    const double *Pl = reinterpret_cast<const double *>(stg + L.pm) + kk * 16, *Pr = Pl + K * 16;
    double v[4], prod[4], ar[4];
    if (r0.w >= 0) td_stack_load(v, stack, r0.w, lane);
    if (r0.w == kWsCarry) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = carry[i];
    }
    td_product(prod, Pl, r0.w == -1, stg[L.codes + p], onehot, tab, v);
    if (r1.x >= 0) td_stack_load(v, stack, r1.x, lane);
    if (r1.x == kWsCarry) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = carry[i];
    }
    td_product(ar, Pr, r1.x == -1, stg[L.codes + 32 + p], onehot, tab, v);
    td_arrive<kTdBarFree>(s);
#pragma unroll
    for (int i = 0; i < 4; ++i) prod[i] = kact ? prod[i] * ar[i] : 0.0;
    int e = 0;
    if (a.rescale) {
      e = td_exponent<KP>(prod);
      td_scale(prod, e);
      E += e;
    }
    if (r1.y != -1) {
      if (r1.y >= 0) td_stack_store(prod, stack, r1.y, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) carry[i] = prod[i];
      if (a.partials && act) {
        const size_t node = size_t(b) * (nst - 1) + (r0.x - a.tip_count);
        if (kact) store_vec_stream<double, 4>(a.partials + ((node * K + k) * size_t(a.N) + n) * 4, prod);
        if (k == 0) a.expo[node * a.N + n] = e;
      }
    } else {  // root: fold categories and frequencies, categories in order
      double sk = 0.0, site = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) sk = fma(a.freqs[b * 4 + i], prod[i], sk);
      for (int c = 0; c < K; ++c) site = fma(a.props[b * K + c], __shfl_sync(0xffffffffu, sk, c * PW + p), site);
      ll = log(site) + double(E) * 0.69314718055994530942;
    }
  }
  if (k == 0 && act && a.site_lnl) a.site_lnl[size_t(b) * a.N + n] = ll;
  const double tot = warp_sum(k == 0 && act ? a.weights[n] * ll : 0.0);
  if (lane == 0) a.tile_lnl[size_t(b) * a.ntiles + tile] = tot;
}

// ----------------------------------------------------------------- adjoint
// u = pre o (the other side's product), each branch's gradient block the sum
// over patterns of u x^T.  The partials stored for child c are 2^-e_c times the
// product at its node, so with q_v the exponent for which
//   sum_i pre_v[i] 2^q_v (P_l x_l)[i] (P_r x_r)[i] = w  (per pattern, over categories)
// holds, a child whose outside partial was scaled by 2^-e has q_c = q_v - e_c + e.
// The root's pre is props freqs w / L with L the same sum, and q = 0.
//
// The gradient's sum runs with lanes as rows (side, category, state) of u:
//  A  both children internal (or an ambiguous tip): 4 FMAs per row and pattern;
//  B  two unambiguous tips: 1 addition per row and pattern;
//  C  one of each: every lane takes half (8 / KP-th) of the patterns of both a
//     row of the internal child and one of the tip, then the halves are joined.
//
// The second warp of the CTA also sums the gradients, of the step before while the
// first is at the next one's products: a step's copies and a third of its FP64
// instructions leave the walk.  u passes between them in two buffers.
template <int KP>
__global__ void __launch_bounds__(64) td_backward_kernel(const PruneArgs<double> a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int PW = 32 / KP, NST = kTdBwdStages;
  constexpr int ROWS = 4 * KP;                       // rows of one side
  constexpr int USTR = PW + 2;                       // u row stride (16-byte rows, spread over the banks)
  constexpr int KSTR = PW * 4 + 2;                   // category stride of a staged child tile
  constexpr int RP = ROWS == 32 ? 2 : 1;             // A, B: row passes (one side each when ROWS = 32)
  constexpr int QA = 2 * ROWS < 32 ? 16 / ROWS : 1;  // A, B: pattern chunks per row
  constexpr int CA = PW / QA;                        // patterns per chunk
  constexpr int QC = 32 / ROWS, CC = PW / QC;        // C: chunks per row, patterns per chunk (4)
  const int lane = threadIdx.x % 32, k = lane / PW, p = lane % PW;
  const bool walks = threadIdx.x < 32;  // the other warp stages and sums
  const int b = blockIdx.y, slot = blockIdx.x, K = a.K, nst = a.n_steps, KSS = K * 16;
  const bool kact = k < K;
  const int kk = kact ? k : 0;
  const TdLayout L = td_layout(K, a.C, a.slots, true);
  double *tab = reinterpret_cast<double *>(smem + L.table), *const ubuf = reinterpret_cast<double *>(smem + L.ubuf);
  unsigned char *onehot = smem + L.onehot, *stack = smem + L.stack;
  int *sexp = reinterpret_cast<int *>(smem + L.sexp);
  if (walks) td_load_table(a, tab, onehot, lane);
  __syncthreads();
  double pk = kact ? a.props[b * K + k] : 0.0, fr[4], rpi[4] = {0.0, 0.0, 0.0, 0.0}, rc = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) fr[i] = a.freqs[b * 4 + i];
  bool first = true;
  for (int tile = slot; tile < a.ntiles; tile += a.nslots, first = false) {
    const int n = tile * PW + p;
    const bool act = n < a.N;
    const double w = act ? a.weights[n] : 0.0;
    __syncwarp();  // the ring of the previous tile is free
    int4 nxt[3];
    auto issue = [&](int t) {  // reversed step t, and its group (empty past the last)
      if (t < nst) {
        const int4 cur[3] = {nxt[0], nxt[1], nxt[2]};
        if (t + 1 < nst) load_rec(nxt, a.steps, nst - 2 - t);
        td_issue<KP, true>(a, L, smem + L.stages + (t % NST) * L.stage, cur, nst - 1 - t, b, tile, lane);
      }
      cp_async_commit();
    };
    if (!walks) {
      load_rec(nxt, a.steps, nst - 1);
      for (int j = 0; j < NST; ++j) issue(j);
      cp_async_wait<NST - 1>();
      td_arrive<kTdBarFull>(0);
    }
    for (int j = 0; j < nst; ++j) {
      const unsigned char *stg = smem + L.stages + (j % NST) * L.stage;
      const int4 *rec = reinterpret_cast<const int4 *>(stg + L.rec);
      double *const ub = ubuf + (j & 1 ? 2 * ROWS * USTR : 0);
      if (walks) {
        td_await<kTdBarFull>(j);
        const int4 r0 = rec[0], r1 = rec[1], r2 = rec[2];
        const int slot_in = r1.z, slot_l = r1.w, slot_r = r2.x;
        const bool ltip = r0.y < a.tip_count, rtip = r0.z < a.tip_count;
        const double *Pl = reinterpret_cast<const double *>(stg + L.pm) + kk * 16, *Pr = Pl + K * 16;
        const double *kids = reinterpret_cast<const double *>(stg + L.kids);
        const int cl = stg[L.codes + p], cr = stg[L.codes + 32 + p];
        double pre[4], al[4], ar[4], v[4];
        if (!ltip) load_vec<double, 4>(v, kids + k * KSTR + p * 4);
        td_product(al, Pl, ltip, cl, onehot, tab, v);
        if (!rtip) load_vec<double, 4>(v, kids + (KP + k) * KSTR + p * 4);
        td_product(ar, Pr, rtip, cr, onehot, tab, v);
        int q = 0;
        if (slot_in >= 0) {
          td_stack_load(pre, stack, slot_in, lane);
          q = sexp[slot_in * 32 + lane];
        } else {  // root: L of the pattern over all categories, and the root gradients
          double den = 0.0, r[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            r[i] = kact ? al[i] * ar[i] : 0.0;
            pre[i] = pk * fr[i];
            den = fma(pre[i], r[i], den);
          }
#pragma unroll
          for (int o = PW; o < 32; o <<= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
          const double coef = act && den > 0.0 ? w / den : 0.0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            pre[i] *= coef;
            if (act) {
              rpi[i] = fma(coef * pk, r[i], rpi[i]);
              rc = fma(coef * fr[i], r[i], rc);
            }
          }
        }
        // u of both sides to shared memory as rows, the children's outside partials to the stack
        double ul[4], ur[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ul[i] = kact && act ? pre[i] * ar[i] : 0.0;
          ur[i] = kact && act ? pre[i] * al[i] : 0.0;
        }
        // the rows the gradients sum, at the pattern's true scale
        {
          double sl[4], sr[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) sl[i] = ul[i], sr[i] = ur[i];
          td_scale(sl, -q);
          td_scale(sr, -q);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            ub[(k * 4 + i) * USTR + p] = sl[i];
            ub[(ROWS + k * 4 + i) * USTR + p] = sr[i];
          }
        }
        td_arrive<kTdBarU>(j);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          if (side ? rtip : ltip) continue;
          const double *P = side ? Pr : Pl;
          double o[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            double row[4];
            load_vec<double, 4>(row, P + i * 4);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) o[jj] = fma(row[jj], side ? ur[i] : ul[i], o[jj]);
          }
          const int e = td_exponent<KP>(o), to = side ? slot_r : slot_l;
          td_scale(o, e);
          td_stack_store(o, stack, to, lane);
          sexp[to * 32 + lane] = q + e - (act ? reinterpret_cast<const int *>(stg + L.expo)[side * PW + p] : 0);
        }
        td_arrive<kTdBarFree>(j);
        continue;
      }
      if (j + 1 < nst) {
        cp_async_wait<NST - 2>();
        td_arrive<kTdBarFull>(j + 1);
      }
      td_await<kTdBarU>(j);
      const int left = rec[0].y, right = rec[0].z;
      const bool ltip = left < a.tip_count, rtip = right < a.tip_count;
      const double *kids = reinterpret_cast<const double *>(stg + L.kids);
      const int cl = stg[L.codes + p], cr = stg[L.codes + 32 + p];
      const unsigned amb = __ballot_sync(0xffffffffu, (ltip && onehot[cl] > 3) || (rtip && onehot[cr] > 3));
      double *gl = a.gpart + ((size_t(b) * a.branch_count + left) * a.nslots + slot) * KSS;
      double *gr = a.gpart + ((size_t(b) * a.branch_count + right) * a.nslots + slot) * KSS;
      if (amb == 0 && ltip != rtip) {  // C
        const int row = lane % ROWS, m0 = (lane / ROWS) * CC;
        const int si = ltip;  // the internal side
        const double *ui = ub + (si * ROWS + row) * USTR + m0, *ut = ub + ((1 - si) * ROWS + row) * USTR + m0;
        const double *vi = kids + (si * KP + row / 4) * KSTR + m0 * 4;
        const unsigned char *ct = stg + L.codes + (1 - si) * 32 + m0;
        double *gi = si ? gr : gl, *gt = si ? gl : gr;
        // the lane's result: both rows when there is one chunk, else internal (low lanes) or tip (lanes 16-31)
        const bool hi = QC > 1 && lane >= 16, writer = (QC == 1 || lane % 16 < ROWS) && row / 4 < K;
        double old[4] = {0.0, 0.0, 0.0, 0.0}, old2[4] = {0.0, 0.0, 0.0, 0.0};
        double *dst = (hi ? gt : gi) + row * 4, *dst2 = gt + row * 4;
        if (!first && writer) {
          load_vec<double, 4>(old, dst);
          if (QC == 1) load_vec<double, 4>(old2, dst2);
        }
        double ai[4] = {0.0, 0.0, 0.0, 0.0}, at[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int m = 0; m < CC; ++m) {
          double x[4];
          load_vec<double, 4>(x, vi + m * 4);
          const double um = ui[m], ux = ut[m];
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) ai[jj] = fma(um, x[jj], ai[jj]);
          const int s = onehot[ct[m]];
          const double sum = (s == 0 ? at[0] : s == 1 ? at[1] : s == 2 ? at[2] : at[3]) + ux;
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) at[jj] = s == jj ? sum : at[jj];
        }
#pragma unroll
        for (int o = ROWS; o < 16; o <<= 1)
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            ai[jj] += __shfl_xor_sync(0xffffffffu, ai[jj], o);
            at[jj] += __shfl_xor_sync(0xffffffffu, at[jj], o);
          }
        if constexpr (QC > 1) {  // low lanes keep the internal rows, high lanes the tip's
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const double got = __shfl_xor_sync(0xffffffffu, hi ? ai[jj] : at[jj], 16);
            ai[jj] = (hi ? at[jj] : ai[jj]) + got;
          }
        }
        if (writer) {
          if (!first) {
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) ai[jj] += old[jj];
          }
          store_vec<double, 4>(dst, ai);
          if (QC == 1) {
            if (!first) {
#pragma unroll
              for (int jj = 0; jj < 4; ++jj) at[jj] += old2[jj];
            }
            store_vec<double, 4>(dst2, at);
          }
        }
      } else {  // A, B
        const bool tips = amb == 0 && ltip && rtip;
#pragma unroll
        for (int rp = 0; rp < RP; ++rp) {
          const int rr = (RP == 2 ? rp * 32 + lane : lane / QA), q0 = (RP == 2 ? 0 : lane % QA) * CA;
          const int side = rr / ROWS, row = rr % ROWS;
          const bool writer = lane % QA == 0 && row / 4 < K;
          const bool tip = side ? rtip : ltip;
          const double *ur0 = ub + rr * USTR + q0;
          const double *vs = kids + (side * KP + row / 4) * KSTR;
          const unsigned char *cs = stg + L.codes + side * 32;
          double *dst = (side ? gr : gl) + row * 4;
          double old[4] = {0.0, 0.0, 0.0, 0.0}, acc[4] = {0.0, 0.0, 0.0, 0.0};
          if (!first && writer) load_vec<double, 4>(old, dst);
          if (tips) {
#pragma unroll
            for (int m = 0; m < CA; ++m) {
              const int s = onehot[cs[q0 + m]];
              const double sum = (s == 0 ? acc[0] : s == 1 ? acc[1] : s == 2 ? acc[2] : acc[3]) + ur0[m];
#pragma unroll
              for (int jj = 0; jj < 4; ++jj) acc[jj] = s == jj ? sum : acc[jj];
            }
          } else {
#pragma unroll
            for (int m = 0; m < CA; ++m) {
              double x[4];
              load_vec<double, 4>(x, tip ? tab + cs[q0 + m] * 4 : vs + (q0 + m) * 4);
              const double um = ur0[m];
#pragma unroll
              for (int jj = 0; jj < 4; ++jj) acc[jj] = fma(um, x[jj], acc[jj]);
            }
          }
#pragma unroll
          for (int o = 1; o < QA; o <<= 1)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) acc[jj] += __shfl_xor_sync(0xffffffffu, acc[jj], o);
          if (writer) {
            if (!first) {
#pragma unroll
              for (int jj = 0; jj < 4; ++jj) acc[jj] += old[jj];
            }
            store_vec<double, 4>(dst, acc);
          }
        }
      }
      td_await<kTdBarFree>(j);
      issue(j + NST);
    }
  }
  if (!walks) return;
  // root gradients: frequencies over every lane, category weights over a category's lanes
#pragma unroll
  for (int i = 0; i < 4; ++i) rpi[i] = warp_sum(rpi[i]);
#pragma unroll
  for (int o = 1; o < PW; o <<= 1) rc += __shfl_xor_sync(0xffffffffu, rc, o);
  double *rp = a.rootpart + (size_t(b) * a.nslots + slot) * (4 + K);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) rp[i] = rpi[i];
  }
  if (p == 0 && kact) rp[4 + k] = rc;
}

}  // namespace tt
