// Host side of the wide-state path (S != 4: amino acids, codons): level
// schedule, workspace and launch sequences behind the C entry points.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <string>
#include <vector>

#include <cudaTypedefs.h>

#include "../../include/torchtree_gb300.h"
#include "tt_plan.h"
#include "tt_wide.cuh"
#include "tt_wide_col.cuh"
#include "tt_wide_tc.cuh"
#include "tt_wide_tc_bwd.cuh"

namespace tt {

__global__ void wide_pmatrix_grad_reduce_kernel(const double *part, int nchunks, int S, int K, double *dlam,
                                                double *dU, double *dW, double *drates) {
  const int b = blockIdx.x;
  const int width = 2 * S * S + S + K;
  for (int e = threadIdx.x; e < width; e += blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < nchunks; ++c) s += part[(size_t(b) * nchunks + c) * width + e];
    if (e < S * S) {
      if (dU) dU[size_t(b) * S * S + e] = s;
    } else if (e < 2 * S * S) {
      if (dW) dW[size_t(b) * S * S + e - S * S] = s;
    } else if (e < 2 * S * S + S) {
      if (dlam) dlam[size_t(b) * S + e - 2 * S * S] = s;
    } else if (drates) {
      drates[size_t(b) * K + e - 2 * S * S - S] = s;
    }
  }
}

struct WideState {
  int SP = 0, PTf = 0, PTb = 0;
  int Npad = 0;  // whole alignment padded to 128 patterns: the tip-code row stride
  int bchunk = 8, nbchunks = 1;
  bool tc = false;  // FP32 codon post-order on the tensor cores
  bool store_products = false;  // FP32 codon: the adjoint reads the post-order's children's products
  bool room_products = false;   // FP64: ... of internal children, where there is room (product_room)
  bool tc_bwd = false;  // FP32 codon adjoint on the tensor cores (needs the stored products)
  float *d_pimg = nullptr;  // its GEMM2 operands: split P^T images [b][B][K][2][64][64]
  float *d_pimg_f = nullptr;  // the tensor-core post-order's B operands: split P images, same shape
  // the images hold the current transition matrices (written right after them, in one pass)
  bool img_f_valid = false, img_b_valid = false;
  // tip products of the tensor-core post-order, [b][tips][K][64 or 128 codes][64]: one for either
  // capacity, allocated with the first tips whose passes use it (tip_table) and kept (a captured pass may
  // hold it); a plan with more codes, or without the memory, sends its tips through the MMAs
  float *d_tprod[2] = {nullptr, nullptr};
  // pattern slabs (p->slab != 0): the pattern-sized buffers below hold one
  // slab; tail_valid = they still hold the last slab's post-order (from a
  // tt_log_likelihood with keep_partials), which the gradient then reuses
  bool tail_valid = false;
  size_t slab_bytes = 0;     // of p->bytes: the pattern-sized buffers
  double *d_site = nullptr;  // slab mode: one slab's site log-likelihoods [b][slab]
  std::vector<int> fwd_off, bwd_off;  // level boundaries in d_fwd / d_bwd
  int *d_left = nullptr, *d_right = nullptr, *d_fwd = nullptr, *d_bwd = nullptr;
  int *d_branch_lvn = nullptr;  // [B] node count of each branch's parent level (adjoint chunking)
  void *d_part = nullptr;
  int *d_expo = nullptr;
  double *d_root_site = nullptr;
  int *d_root_expo = nullptr;
  void *d_coef = nullptr;  // the adjoint's per-pattern coefficients and exponents
  int *d_cexp = nullptr;
  double *d_block_lnl = nullptr;
  void *d_gpart = nullptr;
  void *d_rootpart = nullptr;
  double *d_pgpart = nullptr;
  uint8_t *d_tip_row = nullptr;  // [259] code -> row of the staged P^T (WideArgs::tip_row)
  void *d_tip_amb = nullptr;     // [kTipRows][SP] the ambiguous code vectors
  void *d_prod = nullptr;  // the children's products of the post-order, read by the adjoint
};

namespace {

int wfail(int code, const std::string &m) { return record_error(code, m.c_str()); }

// Launch geometry of a pass over `n` patterns (the whole alignment or one
// slab): padded width, tiles of the two passes, root blocks, and the
// adjoint's chunks of tiles (about two CTAs per SM over batch x categories;
// cmax bounds the chunk count of any pass over at most n patterns).
struct WideGeo {
  int Npad, ntiles_f, ntiles_b, nblk, nchunks, tpc, cmax;
  bool fine;  // FP64 codon passes whose levels choose between tiles of 32 and 16 patterns
};

WideGeo wide_geo(const tt_plan *p, int n) {
  const WideState &w = *p->wide;
  WideGeo g;
  g.Npad = (n + 127) / 128 * 128;
  // FP64 plans skip the tiles past the last pattern
  const int last = p->precision == TT_PRECISION_F64 ? n : g.Npad;
  g.ntiles_f = (last + w.PTf - 1) / w.PTf;
  g.ntiles_b = (last + w.PTb - 1) / w.PTb;
  g.nblk = (n + 255) / 256;
  const int want = (2 * 152 + p->batch * p->K - 1) / (p->batch * p->K);
  g.cmax = std::max(1, std::min({want, g.ntiles_b, 64}));
  g.tpc = (g.ntiles_b + g.cmax - 1) / g.cmax;
  g.nchunks = (g.ntiles_b + g.tpc - 1) / g.tpc;
  // (whole alignments of up to 512 patterns, a chunk per tile: the gradient chunks stay small)
  const int t16 = (n + 15) / 16;
  g.fine = p->precision == TT_PRECISION_F64 && w.SP == 64 && n == p->N && t16 <= std::min(want, 32);
  if (g.fine) {
    g.cmax = g.nchunks = t16;
    g.tpc = 1;
  }
  return g;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}

// A row-major FP32 array [rows][cols] (cols a multiple of 4) as a 2-D tensor
// map with bx x by boxes, no swizzle.
bool encode_rows(CUtensorMap *m, const float *base, uint64_t rows, uint64_t cols, uint32_t bx, uint32_t by,
                 CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE) {
  const PFN_cuTensorMapEncodeTiled_v12000 fn = tensor_map_encoder();
  if (!fn) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * sizeof(float)};
  const cuuint32_t box[2] = {bx, by};
  const cuuint32_t elem[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Both split images of the FP32 codon transition matrices that the tensor-core
// kernels use, from d_pmat in one pass (either may be skipped).
cudaError_t launch_pimages(tt_plan *p, bool fwd, bool bwd, cudaStream_t s) {
  WideState &w = *p->wide;
  float *f = fwd ? w.d_pimg_f : nullptr, *b = bwd ? w.d_pimg : nullptr;
  if (!f && !b) return cudaSuccess;
  const long long count = (long long)p->batch * p->B * p->K;
  wide_pimages_kernel<<<unsigned(count), 256, 0, s>>>(static_cast<const float *>(p->d_pmat), f, b);
  p->launches += 1;
  if (f) w.img_f_valid = true;
  if (b) w.img_b_valid = true;
  return cudaGetLastError();
}

int wcuda(cudaError_t e, const char *where) {
  return wfail(e == cudaErrorMemoryAllocation ? TT_ERR_OUT_OF_MEMORY : TT_ERR_CUDA,
               std::string(where) + ": " + cudaGetErrorString(e));
}

template <typename P>
int walloc(tt_plan *p, P **ptr, size_t bytes, const char *what) {
  if (bytes == 0) bytes = 16;
  cudaError_t e = cudaMalloc(reinterpret_cast<void **>(ptr), bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return wfail(TT_ERR_OUT_OF_MEMORY, std::string("cudaMalloc of ") + what + " (" + std::to_string(bytes) +
                                           " bytes) failed: " + cudaGetErrorString(e));
  }
  p->bytes += bytes;
  return TT_OK;
}

// Whether an FP32 codon pass of ntf 128-pattern tiles takes its tips' products from a table by
// code: it costs each tip one tile and the pass a launch, and saves the products of all the tip's
// tiles.  Up to 64 codes, 4 categories, post-order that keeps its products, without and with it: 40 taxa x
// 1,000 patterns x 2 samples 224, 224 us; 200 x 800 x 1 410, 401; 200 x 1,500 x 1 551, 504; 100 x 800 x 4
// 590, 567; 200 x 2,608 x 8 5,203, 4,349.  Up to 128 (the lowest level's two tables then take 70 KB of a CTA):
// 200 x 800 x 1 387, 416; 200 x 1,500 x 1 537, 535; 100 x 800 x 4 569, 596; 200 x 800 x 8 1,841, 1,809; 100 x
// 2,600 x 1 472, 461.
bool tip_table_pays(const tt_plan *p, int codes, int samples, int ntf) {
  const size_t products = size_t(p->T) * samples * p->K * ntf;
  if (codes > 64) return codes <= 128 && ntf >= 6 && products >= (ntf >= 12 ? 8192 : 32768);
  return ntf >= 6 && products >= 2048;
}

// compiled (precision, padded states) -> pattern tiles of the two passes
void tiles_for(bool f32, int SP, int &ptf, int &ptb) {
  if (SP == 20) {
    ptf = ptb = 128;
  } else {
    ptf = ptb = f32 ? 64 : 32;
  }
}

template <typename T, int SP, int PTF, int PTB>
struct Wide {
  static cudaError_t prepare() {
    cudaError_t e = cudaFuncSetAttribute(wide_forward_kernel<T, SP, PTF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(wide_fwd_smem<T, SP, PTF>()));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_backward_kernel<T, SP, PTB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(wide_bwd_smem<T, SP, PTB>()));
    if constexpr (std::is_same<T, double>::value && SP == 64) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wide_forward_kernel<T, SP, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(wide_fwd_smem<T, SP, 16>()));
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wide_backward_kernel<T, SP, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(wide_bwd_smem<T, SP, 16>()));
    }
    if (e == cudaSuccess)  // the CTAs the shared memory allows per SM all resident
      e = cudaFuncSetAttribute(wide_backward_kernel<T, SP, PTB>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               int(cudaSharedmemCarveoutMaxShared));
    for (auto kernel : {wide_forward_tc_kernel<false>, wide_forward_tc_kernel<true>}) {
      if (std::is_same<T, float>::value && SP == 64 && e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmem);
      if (std::is_same<T, float>::value && SP == 64 && e == cudaSuccess)  // two CTAs per SM
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 int(cudaSharedmemCarveoutMaxShared));
    }
    if (std::is_same<T, float>::value && SP == 64 && e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_tip_products_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmem);
    if (std::is_same<T, float>::value && SP == 64 && e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_backward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tcb::kSmem);
    if (std::is_same<T, float>::value && SP == 64 && e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_backward_tc_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                               int(cudaSharedmemCarveoutMaxShared));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_pmatrix_kernel<T, SP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(3 * SP * SP * sizeof(T) + SP * sizeof(T)));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(wide_pmatrix_backward_kernel<double, SP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(Wide<double, SP, PTF, PTB>::pback_smem()));
    return e;
  }
  static size_t pback_smem() { return 4 * SP * SP * sizeof(T) + (SP / 4 * SP + 3 * SP + 8) * sizeof(double); }

  // arguments of a pass over patterns [p0, p0 + n) with geometry g: tip
  // codes and weights from the slab's first pattern, every pattern-sized
  // buffer with the slab's own width
  static WideArgs<T> args(tt_plan *p, const double *props, const double *freqs, int rescale, const WideGeo &g,
                          int p0, int n) {
    WideState &w = *p->wide;
    WideArgs<T> a;
    a.tips = p->T;
    a.N = n;
    a.Npad = g.Npad;
    a.K = p->K;
    a.B = p->B;
    a.I = p->I;
    a.S = p->S;
    a.code_stride = p->code_stride;
    a.rescale = rescale;
    a.nchunks = g.nchunks;
    a.tiles_per_chunk = g.tpc;
    a.ntiles = g.ntiles_b;
    a.nodes = nullptr;
    a.left = w.d_left;
    a.right = w.d_right;
    a.codes = p->d_codes + p0;
    a.table = static_cast<const T *>(p->d_table);
    a.tip_row = w.d_tip_row;
    a.tip_amb = static_cast<const T *>(w.d_tip_amb);
    a.pmat = static_cast<const T *>(p->d_pmat);
    a.part = static_cast<T *>(w.d_part);
    a.expo = w.d_expo;
    a.props = props;
    a.freqs = freqs;
    a.weights = p->d_weights + p0;
    a.root_site = w.d_root_site;
    a.root_expo = w.d_root_expo;
    a.coef = static_cast<const T *>(w.d_coef);
    a.cexp = w.d_cexp;
    a.gpart = static_cast<T *>(w.d_gpart);
    a.rootpart = static_cast<T *>(w.d_rootpart);
    a.prod = nullptr;
    return a;
  }

  // post-order over patterns [p0, p0 + n), root sums, and lnL (added to
  // lnl when accumulate; no lnL when lnl is NULL).  site_lnl [b][n].
  static cudaError_t forward(tt_plan *p, const double *props, const double *freqs, int rescale, bool keep,
                             double *lnl, double *site_lnl, int p0, int n, int accumulate, cudaStream_t s) {
    WideState &w = *p->wide;
    const WideGeo g = wide_geo(p, n);
    WideArgs<T> a = args(p, props, freqs, rescale, g, p0, n);
    if (keep) a.prod = static_cast<T *>(w.d_prod);
    constexpr int NT = WideCfg<T, SP, PTF>::NT;
    const size_t smem = wide_fwd_smem<T, SP, PTF>();
    if constexpr (std::is_same<T, float>::value && SP == 64) {
      if (w.tc && w.d_pimg_f && !w.img_f_valid) {  // the post-order's split P images, if not written with P
        const cudaError_t e = launch_pimages(p, true, false, s);
        if (e != cudaSuccess) return e;
      }
    }
    const float *tprod = nullptr;
    const int tcodes = p->C <= 64 ? 64 : 128;
    if constexpr (std::is_same<T, float>::value && SP == 64) {
      // the tips' products by code, with every pass (a captured one has to follow the matrices)
      if (w.tc && w.d_pimg_f && tip_table_pays(p, p->C, plan_run_samples(p), g.Npad / tc::kPT))
        tprod = w.d_tprod[tcodes / 128];
      if (tprod) {
        wide_tip_products_tc_kernel<<<dim3(p->T, plan_run_samples(p) * p->K), tc::kThreads, tc::kSmem, s>>>(
            a, w.d_pimg_f, tcodes, w.d_tprod[tcodes / 128], p->d_status, 2000000000ull);
        p->launches += 1;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
      }
    }
    for (size_t lv = 0; lv + 1 < w.fwd_off.size(); ++lv) {
      a.nodes = w.d_fwd + w.fwd_off[lv];
      if constexpr (std::is_same<T, float>::value && SP == 64) {
        if (w.tc) {  // tiles per CTA by level: about sixteen waves of two CTAs per SM
          const int nodes = w.fwd_off[lv + 1] - w.fwd_off[lv], ntf = g.Npad / tc::kPT;
          if (lv == 0 && p->I > 1 && tprod) {  // two tips each (and not the root)
            static_assert(kTipPairThreads == tc::kPT, "the tiles are alike");
            const size_t sm = tip_pair_smem(tcodes);
            const cudaError_t e = kernel_smem(wide_tip_pair_kernel, sm, true);
            if (e != cudaSuccess) return e;
            const int chunks = tc_level_chunks(nodes, p->batch * p->K, ntf, ntf, 8 * 152 * 5);
            WideArgs<T> at = a;
            at.ntiles = ntf;
            at.tiles_per_chunk = (ntf + chunks - 1) / chunks;
            wide_tip_pair_kernel<<<dim3(chunks, nodes, plan_run_samples(p) * p->K), kTipPairThreads, sm, s>>>(
                at, tprod, tcodes);
            p->launches += 1;
            continue;
          }
          const int chunks = tc_level_chunks(nodes, p->batch * p->K, ntf, ntf, 16 * 152 * 2);
          WideArgs<T> at = a;
          at.ntiles = ntf;
          at.tiles_per_chunk = (ntf + chunks - 1) / chunks;
          const dim3 grid(chunks, nodes, plan_run_samples(p) * p->K);
          (tprod ? wide_forward_tc_kernel<true> : wide_forward_tc_kernel<false>)<<<grid, tc::kThreads, tc::kSmem, s>>>(
              at, w.d_pimg_f, tprod, tcodes, p->d_status, 2000000000ull);
          p->launches += 1;
          continue;
        }
      }
      const int nodes = w.fwd_off[lv + 1] - w.fwd_off[lv];
      if constexpr (SP == kColStates) {
        // Every level but the root's, in FP32 those that fill the GPU: below 256 (node, sample, category, 128
        // patterns) the table of every CTA is on the level's chain.  32 levels of one node with a tip, without and
        // with it: 32 units 316, 373 us, 128 units 316, 372, 256 units 374, 375, 512 units 438, 439; levels of
        // internal children, 16 to 2 nodes: 16 units a node 108, 105, 512 units a node 437, 340.
        const bool fills = sizeof(T) == 8 || size_t(nodes) * p->batch * p->K * (g.Npad / 128) >= 256;
        if (lv + 2 < w.fwd_off.size() && fills) {  // about eight waves of three CTAs per SM
          constexpr int tile = kColThreads * kColPatterns<T>;
          WideArgs<T> ac = a;
          ac.ntiles = (g.Npad + tile - 1) / tile;
          const int chunks = tc_level_chunks(nodes, p->batch * p->K, ac.ntiles, ac.ntiles, 8 * 152 * 3);
          ac.tiles_per_chunk = (ac.ntiles + chunks - 1) / chunks;
          const size_t sm = col_fwd_smem<T>(p->C);
          const cudaError_t e = kernel_smem(wide_col_forward_kernel<T>, sm, true);
          if (e != cudaSuccess) return e;
          wide_col_forward_kernel<T><<<dim3(chunks, nodes, plan_run_samples(p) * p->K), kColThreads, sm, s>>>(ac, p->C);
          p->launches += 1;
          continue;
        }
      }
      if constexpr (std::is_same<T, double>::value && SP == 64) {
        if (g.fine && wide_fine_level(nodes, p->batch * p->K, n)) {
          wide_forward_kernel<T, SP, 16><<<dim3(2 * g.ntiles_f, nodes, plan_run_samples(p) * p->K),
                                           WideCfg<T, SP, 16>::NT, wide_fwd_smem<T, SP, 16>(), s>>>(a);
          p->launches += 1;
          continue;
        }
      }
      const dim3 grid(g.ntiles_f, nodes, plan_run_samples(p) * p->K);
      wide_forward_kernel<T, SP, PTF><<<grid, NT, smem, s>>>(a);
      p->launches += 1;
    }
    wide_root_kernel<T><<<dim3(g.nblk, plan_run_samples(p)), 256, 0, s>>>(
        w.d_root_site, w.d_root_expo, props, a.weights, site_lnl, static_cast<T *>(w.d_coef), w.d_cexp, w.d_block_lnl,
        p->K, n, g.Npad);
    p->launches += 1;
    cudaError_t e = cudaSuccess;
    if (lnl) {
      e = launch_reduce_lnl(w.d_block_lnl, lnl, plan_run_samples(p), g.nblk, accumulate, s);
      p->launches += 1;
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
  }

  // adjoint over patterns [p0, p0 + n) after that range's post-order; the
  // chunk sums are added to the previous slabs' when accumulate
  static cudaError_t backward(tt_plan *p, const double *props, const double *freqs, int p0, int n, int accumulate,
                              cudaStream_t s) {
    WideState &w = *p->wide;
    const WideGeo g = wide_geo(p, n);
    WideArgs<T> a = args(p, props, freqs, 1, g, p0, n);
    a.prod = static_cast<T *>(w.d_prod);
    if constexpr (std::is_same<T, float>::value && SP == 64) {
      if (w.tc_bwd && a.prod && w.d_pimg) return backward_tc(p, a, g, accumulate, s);
    }
    constexpr int NT = WideCfg<T, SP, PTB>::NT;
    const size_t smem = wide_bwd_smem<T, SP, PTB>(!kChildProducts<T> && a.prod);
    // FP32 20-state plans: a chunk count per level (three CTAs per SM), as the tensor-core adjoint does
    constexpr bool per_level = std::is_same<T, float>::value && SP == 20;
    const int bk = p->batch * p->K, target = 8 * 152 * 3;
    for (size_t lv = 0; lv + 1 < w.bwd_off.size(); ++lv) {
      const int nodes = w.bwd_off[lv + 1] - w.bwd_off[lv];
      a.nodes = w.d_bwd + w.bwd_off[lv];
      if constexpr (std::is_same<T, double>::value && SP == 64) {
        if (g.fine && wide_fine_level(nodes, bk, n)) {
          WideArgs<T> af = a;
          af.ntiles = (n + 15) / 16;
          wide_backward_kernel<T, SP, 16><<<dim3(2 * g.ntiles_b, nodes, plan_run_samples(p) * p->K),
                                            WideCfg<T, SP, 16>::NT, wide_bwd_smem<T, SP, 16>(), s>>>(af);
          p->launches += 1;
          continue;
        }
      }
      const int chunks = per_level ? tc_level_chunks(nodes, bk, g.ntiles_b, g.cmax, target)
                         : g.fine  ? g.ntiles_b
                                   : g.nchunks;
      a.tiles_per_chunk = per_level ? (g.ntiles_b + chunks - 1) / chunks : g.tpc;
      const dim3 grid(chunks, nodes, plan_run_samples(p) * p->K);
      wide_backward_kernel<T, SP, PTB><<<grid, NT, smem, s>>>(a);
      p->launches += 1;
    }
    const int spread = p->B * plan_run_samples(p) < 8 * 152 ? 4 : 1;
    wide_grad_reduce_kernel<T><<<dim3(p->B, plan_run_samples(p), spread), 256, 0, s>>>(
        static_cast<const T *>(w.d_gpart), p->d_G, p->B, g.nchunks, p->K, p->S, SP, accumulate,
        per_level || g.fine ? w.d_branch_lvn : nullptr, bk, g.ntiles_b, g.cmax, target, g.fine ? n : 0);
    const int root_used = g.fine && !wide_fine_level(1, bk, n) ? g.ntiles_b : g.nchunks;
    wide_root_reduce_kernel<T><<<plan_run_samples(p), 64, 0, s>>>(static_cast<const T *>(w.d_rootpart), p->d_rootgrad,
                                                       p->d_rootgrad + size_t(p->batch) * p->S, g.nchunks, p->K,
                                                       p->S, SP, accumulate, root_used);
    p->launches += 2;
    return cudaGetLastError();
  }

  // the tensor-core adjoint (FP32 codon plans): split P^T images, then one
  // launch per depth level over chunks of 128-pattern tiles
  static cudaError_t backward_tc(tt_plan *p, WideArgs<float> a, const WideGeo &g, int accumulate, cudaStream_t s) {
    WideState &w = *p->wide;
    if (!w.img_b_valid) {  // the split P^T images, if not written with P
      const cudaError_t e = launch_pimages(p, false, true, s);
      if (e != cudaSuccess) return e;
    }
    const int ntc = g.Npad / tcb::kPT;
    const int want = (2 * 152 + p->batch * p->K - 1) / (p->batch * p->K);
    const int cmax = std::max(1, std::min({want, ntc, g.cmax}));
    const int tpc = (ntc + cmax - 1) / cmax;
    a.ntiles = ntc;
    a.tiles_per_chunk = tpc;
    a.nchunks = (ntc + tpc - 1) / tpc;
    // The encoder is a driver call: it needs a current context, which a thread that has made no
    // runtime call yet (autograd's) gets from cudaSetDevice.  The plan's device is current already.
    const cudaError_t ctx = cudaSetDevice(p->device);
    if (ctx != cudaSuccess) return ctx;
    // the raw rows as 2-D tensors: partials [b I K 64][Npad], products [b I K 128][Npad]
    TcbMaps maps;
    const uint64_t blocks = uint64_t(p->batch) * p->I * p->K;
    if (!encode_rows(&maps.part32, a.part, blocks * 64, uint64_t(g.Npad), 32, 64, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_rows(&maps.prod32, a.prod, blocks * 128, uint64_t(g.Npad), 32, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_rows(&maps.part128, a.part, blocks * 64, uint64_t(g.Npad), 128, 32) ||
        !encode_rows(&maps.prod128, a.prod, blocks * 128, uint64_t(g.Npad), 128, 32))
      return cudaErrorInvalidValue;
    // a.nchunks stays the chunk stride of the gradient blocks; each level launches
    // tc_level_chunks(...) <= a.nchunks chunks (the root's level all of them)
    const int bk = p->batch * p->K;
    for (size_t lv = 0; lv + 1 < w.bwd_off.size(); ++lv) {
      const int nodes = w.bwd_off[lv + 1] - w.bwd_off[lv];
      const int chunks = tc_level_chunks(nodes, bk, ntc, cmax);
      a.nodes = w.d_bwd + w.bwd_off[lv];
      a.tiles_per_chunk = (ntc + chunks - 1) / chunks;
      const dim3 grid(chunks, nodes, plan_run_samples(p) * p->K);
      wide_backward_tc_kernel<<<grid, tcb::kThreads, tcb::kSmem, s>>>(a, maps, w.d_pimg, p->d_status,
                                                                       2000000000ull);
      p->launches += 1;
    }
    wide_grad_reduce_kernel<float><<<dim3(p->B, plan_run_samples(p)), 256, 0, s>>>(static_cast<const float *>(w.d_gpart),
                                                                         p->d_G, p->B, a.nchunks, p->K, p->S, 64,
                                                                         accumulate, w.d_branch_lvn, bk, ntc, cmax);
    wide_root_reduce_kernel<float><<<plan_run_samples(p), 64, 0, s>>>(static_cast<const float *>(w.d_rootpart), p->d_rootgrad,
                                                           p->d_rootgrad + size_t(p->batch) * p->S, a.nchunks, p->K,
                                                           p->S, 64, accumulate, a.nchunks);
    p->launches += 2;
    return cudaGetLastError();
  }

  static cudaError_t pmatrix(tt_plan *p, const double *lam, const double *U, const double *W, const double *bl,
                             const double *rates, cudaStream_t s) {
    wide_pmatrix_kernel<T, SP><<<dim3(p->B, p->batch), 256, 3 * SP * SP * sizeof(T) + SP * sizeof(T), s>>>(
        lam, U, W, bl, rates, static_cast<T *>(p->d_pmat), p->S, p->B, p->K);
    p->launches += 1;
    p->wide->img_f_valid = p->wide->img_b_valid = false;
    if constexpr (std::is_same<T, float>::value && SP == 64) {  // the tensor-core kernels' images with P
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      return launch_pimages(p, p->wide->tc, p->wide->tc_bwd, s);
    }
    return cudaGetLastError();
  }

  static cudaError_t pmatrix_backward(tt_plan *p, const double *lam, const double *U, const double *W,
                                      const double *bl, const double *rates, double *dlam, double *dU, double *dW,
                                      double *dbl, double *drates, cudaStream_t s) {
    WideState &w = *p->wide;
    wide_pmatrix_backward_kernel<double, SP><<<dim3(w.nbchunks, p->batch), 256, Wide<double, SP, PTF, PTB>::pback_smem(), s>>>(
        p->d_G, lam, U, W, bl, rates, p->S, p->B, p->K, w.bchunk, dbl, w.d_pgpart);
    wide_pmatrix_grad_reduce_kernel<<<p->batch, 256, 0, s>>>(w.d_pgpart, w.nbchunks, p->S, p->K, dlam, dU, dW,
                                                             drates);
    p->launches += 2;
    return cudaGetLastError();
  }
};

// dispatch on (precision, SP)
template <typename F>
cudaError_t dispatch(tt_plan *p, F &&f) {
  const bool f32 = p->precision == TT_PRECISION_F32;
  if (p->wide->SP == 20) {
    if (f32) return f(Wide<float, 20, 128, 128>());
    return f(Wide<double, 20, 128, 128>());
  }
  if (f32) return f(Wide<float, 64, 64, 64>());
  return f(Wide<double, 64, 32, 32>());
}

}  // namespace

int wide_create(tt_plan *p) {
  if (p->S < 2 || p->S > 64) return wfail(TT_ERR_UNSUPPORTED, "state_count must be in [2, 64]");
  WideState *w = new WideState();
  p->wide = w;
  const bool f32 = p->precision == TT_PRECISION_F32;
  w->SP = p->S <= 20 ? 20 : 64;
  tiles_for(f32, w->SP, w->PTf, w->PTb);
  w->Npad = (p->N + 127) / 128 * 128;
  if (size_t(p->batch) * p->K > 65535) return wfail(TT_ERR_INVALID_ARGUMENT, "batch * category_count must be <= 65535");
  w->nbchunks = (p->B + w->bchunk - 1) / w->bchunk;
  {  // tensor-core post-order for FP32 codon plans (TT_WIDE_TC=0 selects the CUDA-core kernel)
    const char *env = getenv("TT_WIDE_TC");
    w->tc = f32 && w->SP == 64 && !(env && atoi(env) == 0);
  }
  p->code_stride = w->Npad;

  // children, levels by height (forward) and by depth (adjoint); the postorder
  // was validated by build_schedule
  const int T = p->T, I = p->I, NN = 2 * T - 1;
  std::vector<int> left(I), right(I), height(NN, 0), depth(NN, 0);
  // the schedule holds (node, left, right) in an evaluation order that is a post-order
  for (int s = 0; s < I; ++s) {
    const int *rec = &p->steps[size_t(s) * kStepInts];
    const int v = rec[0], l = rec[1], r = rec[2];
    left[v - T] = l;
    right[v - T] = r;
    height[v] = 1 + std::max(height[l], height[r]);
  }
  for (int s = I - 1; s >= 0; --s) {
    const int *rec = &p->steps[size_t(s) * kStepInts];
    depth[rec[1]] = depth[rec[0]] + 1;
    depth[rec[2]] = depth[rec[0]] + 1;
  }
  int H = 0, D = 0;
  for (int v = T; v < NN; ++v) {
    H = std::max(H, height[v]);
    D = std::max(D, depth[v]);
  }
  std::vector<int> fwd, bwd;
  w->fwd_off.push_back(0);
  for (int h = 1; h <= H; ++h) {
    for (int v = T; v < NN; ++v)
      if (height[v] == h) fwd.push_back(v);
    w->fwd_off.push_back(int(fwd.size()));
  }
  w->bwd_off.push_back(0);
  std::vector<int> branch_lvn(size_t(p->B), 1);
  for (int d = 0; d <= D; ++d) {
    const size_t first = bwd.size();
    for (int v = T; v < NN; ++v)
      if (depth[v] == d) bwd.push_back(v);
    const int n = int(bwd.size() - first);
    for (size_t i = first; i < bwd.size(); ++i) {
      const int v = bwd[i];
      branch_lvn[left[v - T]] = n;
      branch_lvn[right[v - T]] = n;
    }
    w->bwd_off.push_back(int(bwd.size()));
  }
  const size_t es = p->elem, SP = size_t(w->SP), b = size_t(p->batch), K = size_t(p->K);
  int rc = TT_OK;
  if (!rc) rc = walloc(p, &w->d_left, I * sizeof(int), "children");
  if (!rc) rc = walloc(p, &w->d_right, I * sizeof(int), "children");
  if (!rc) rc = walloc(p, &w->d_fwd, I * sizeof(int), "levels");
  if (!rc) rc = walloc(p, &w->d_bwd, I * sizeof(int), "levels");
  if (!rc) rc = walloc(p, &w->d_branch_lvn, size_t(p->B) * sizeof(int), "branch levels");
  if (!rc) rc = walloc(p, &p->d_codes, size_t(T) * p->code_stride, "tip codes");
  if (!rc) rc = walloc(p, &p->d_table, 256 * SP * es, "code table");
  if (!rc) rc = walloc(p, &w->d_tip_row, 259, "tip rows");
  if (!rc) rc = walloc(p, &w->d_tip_amb, kTipRows * SP * es, "ambiguous code vectors");
  if (!rc) rc = walloc(p, &p->d_weights, size_t(p->N) * sizeof(double), "weights");
  if (!rc) rc = walloc(p, &p->d_pmat, b * p->B * K * SP * SP * es, "transition matrices");
  {  // FP32 codon plans keep the children's products for the adjoint (TT_WIDE_STORE_PRODUCTS=0
     // recomputes them): 84.1 -> 80.2 ms per call at 200 tips x 2,608 codon patterns x 16; with 20
     // states the extra stores cost more than the products they save
    const char *env = getenv("TT_WIDE_STORE_PRODUCTS");
    w->store_products = f32 && SP == 64 && !(env && atoi(env) == 0);
    w->room_products = !f32 && !(env && atoi(env) == 0);
  }
  {  // tensor-core adjoint for those plans (TT_WIDE_TC_BWD=0 selects the CUDA-core kernel)
    const char *env = getenv("TT_WIDE_TC_BWD");
    if (!rc && w->store_products && !(env && atoi(env) == 0)) rc = wide_set_tensor_core_adjoint(p, true);
  }
  if (!rc && w->tc) rc = wide_set_tensor_cores(p, true);  // its split P images
  // the pattern-sized buffers (partials, exponents, products, root and
  // gradient chunks) come from wide_alloc_slab once the slab size is chosen
  if (!rc)
    rc = walloc(p, &w->d_pgpart, b * w->nbchunks * (2 * p->S * p->S + p->S + K) * sizeof(double),
                "matrix gradient chunks");
  if (!rc) rc = walloc(p, &p->d_G, b * p->B * K * p->S * p->S * sizeof(double), "dlnL/dP");
  if (!rc) rc = walloc(p, &p->d_rootgrad, b * (p->S + K) * sizeof(double), "root grads");
  if (!rc) rc = walloc(p, &p->d_status, sizeof(int), "status");
  if (rc) return rc;
  cudaError_t e = cudaMemcpy(w->d_left, left.data(), I * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(w->d_right, right.data(), I * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(w->d_fwd, fwd.data(), I * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(w->d_bwd, bwd.data(), I * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(w->d_branch_lvn, branch_lvn.data(), size_t(p->B) * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(p->d_status, 0, sizeof(int));
  if (e == cudaSuccess)
    e = dispatch(p, [](auto W) { return decltype(W)::prepare(); });
  if (e != cudaSuccess) return wcuda(e, "wide-state plan set-up");
  return TT_OK;
}

namespace {

struct SlabBuffers {
  size_t part, expo, prod, root_site, root_expo, coef, cexp, block, gpart, rootpart, site;
  size_t total() const {
    size_t t = 0;
    for (size_t x : {part, expo, prod, root_site, root_expo, coef, cexp, block, gpart, rootpart, site})
      t += x ? std::max(x, size_t(16)) : 0;
    return t;
  }
};

// Pattern-sized buffers for passes over at most n patterns (slab = n when
// the plan works in slabs, 0 for the whole alignment).
SlabBuffers slab_buffers(const tt_plan *p, int n, bool slab) {
  const WideState &w = *p->wide;
  const WideGeo g = wide_geo(p, n);
  const size_t es = p->elem, SP = size_t(w.SP), b = size_t(p->batch), K = size_t(p->K), I = size_t(p->I);
  SlabBuffers x;
  x.part = b * I * K * SP * g.Npad * es;
  x.expo = b * I * K * g.Npad * sizeof(int);
  x.prod = w.store_products ? b * I * K * 2 * SP * g.Npad * es : 0;
  x.root_site = b * K * g.Npad * sizeof(double);
  x.root_expo = b * K * g.Npad * sizeof(int);
  x.coef = b * g.Npad * es;
  x.cexp = b * g.Npad * sizeof(int);
  x.block = b * g.nblk * sizeof(double);
  x.gpart = b * p->B * g.cmax * K * SP * SP * es;
  x.rootpart = b * g.cmax * K * (SP + 1) * es;
  x.site = slab ? b * size_t(n) * sizeof(double) : 0;
  return x;
}

// Whether there is room for `bytes` beside pattern buffers of `total` bytes, for what a plan can do without:
// FP64 plans' products of internal children (they save the adjoint a third of its products and are as large
// as the partials) and FP32 codon plans' tip products.  Neither is a reason for slabs (choose_slab does not
// count them): kept if they take at most a quarter of the device's free memory and stay within
// TT_GRADIENT_BUDGET_BYTES.
bool product_room(size_t bytes, size_t total) {
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (const char *env = getenv("TT_GRADIENT_BUDGET_BYTES"))
    if (total + bytes > size_t(atoll(env))) return false;
  return bytes <= free_b / 4;
}

void free_slab_buffers(tt_plan *p) {
  WideState &w = *p->wide;
  for (void **x : {reinterpret_cast<void **>(&w.d_part), reinterpret_cast<void **>(&w.d_expo),
                   reinterpret_cast<void **>(&w.d_prod), reinterpret_cast<void **>(&w.d_root_site),
                   reinterpret_cast<void **>(&w.d_root_expo), reinterpret_cast<void **>(&w.d_coef), reinterpret_cast<void **>(&w.d_cexp),
                   reinterpret_cast<void **>(&w.d_block_lnl), reinterpret_cast<void **>(&w.d_gpart),
                   reinterpret_cast<void **>(&w.d_rootpart), reinterpret_cast<void **>(&w.d_site)})
    if (*x) {
      cudaFree(*x);
      *x = nullptr;
    }
  p->bytes -= std::min(p->bytes, w.slab_bytes);
  w.slab_bytes = 0;
}

}  // namespace

namespace {

// The table of tip products of an FP32 codon plan with `codes` tip codes, where its passes use one and there
// is room (without it the tips take products).  Never given back before the plan: a captured pass may hold it.
void tip_table(tt_plan *p, int codes) {
  WideState &w = *p->wide;
  if (p->precision != TT_PRECISION_F32 || w.SP != 64) return;
  const int cap = codes <= 64 ? 64 : 128;
  float *&tprod = w.d_tprod[cap / 128];
  const size_t bytes = size_t(p->batch) * p->T * p->K * cap * w.SP * sizeof(float);
  if (tprod || !tip_table_pays(p, codes, p->batch, ((p->slab ? p->slab : p->N) + tc::kPT - 1) / tc::kPT) ||
      !product_room(bytes, w.slab_bytes))
    return;
  if (walloc(p, &tprod, bytes, "tip products")) tprod = nullptr;
}

}  // namespace

size_t wide_pattern_bytes(const tt_plan *p, int n) { return slab_buffers(p, n, false).total(); }

int wide_alloc_slab(tt_plan *p, int slab) {
  WideState &w = *p->wide;
  free_slab_buffers(p);
  p->partials_valid = false;
  p->grads_valid = false;
  w.tail_valid = false;
  const SlabBuffers x = slab_buffers(p, slab ? slab : p->N, slab != 0);
  const size_t before = p->bytes;
  int rc = walloc(p, &w.d_part, x.part, "partials");
  if (!rc) rc = walloc(p, &w.d_expo, x.expo, "scale exponents");
  if (!rc && x.prod) rc = walloc(p, &w.d_prod, x.prod, "children's products");
  if (!rc) rc = walloc(p, &w.d_root_site, x.root_site, "root sums");
  if (!rc) rc = walloc(p, &w.d_root_expo, x.root_expo, "root exponents");
  if (!rc) rc = walloc(p, &w.d_coef, x.coef, "pattern coefficients");
  if (!rc) rc = walloc(p, &w.d_cexp, x.cexp, "pattern exponents");
  if (!rc) rc = walloc(p, &w.d_block_lnl, x.block, "block sums");
  if (!rc) rc = walloc(p, &w.d_gpart, x.gpart, "gradient chunks");
  if (!rc) rc = walloc(p, &w.d_rootpart, x.rootpart, "root gradient chunks");
  if (!rc && x.site) rc = walloc(p, &w.d_site, x.site, "slab site log-likelihoods");
  if (!rc && w.room_products && product_room(x.part, x.total())) {
    if (walloc(p, &w.d_prod, x.part, "children's products")) w.d_prod = nullptr;  // the adjoint forms them
  }
  w.slab_bytes = p->bytes - before;
  if (rc) {
    free_slab_buffers(p);
    return rc;
  }
  p->slab = slab;
  if (p->tips_set) tip_table(p, p->C);
  return TT_OK;
}

bool wide_has_buffers(const tt_plan *p) { return p->wide && p->wide->d_part; }

int wide_set_tensor_cores(tt_plan *p, bool on) {
  WideState *w = p->wide;
  if (!w || p->precision != TT_PRECISION_F32 || w->SP != 64)
    return on ? wfail(TT_ERR_UNSUPPORTED, "the tensor-core post-order serves FP32 codon (> 20-state) plans") : TT_OK;
  const size_t bytes = size_t(p->batch) * p->B * p->K * tcb::kImgFloats * sizeof(float);
  if (on && !w->d_pimg_f) {  // the split P images: 32 KB per (sample, branch, category)
    const int rc = walloc(p, &w->d_pimg_f, bytes, "split transition-matrix images");
    if (rc) return rc;
    w->img_f_valid = false;
  } else if (!on && w->d_pimg_f) {
    cudaFree(w->d_pimg_f);
    w->d_pimg_f = nullptr;
    p->bytes -= std::min(p->bytes, bytes);
  }
  w->tc = on;
  return TT_OK;
}

bool wide_tensor_cores(const tt_plan *p) { return p->wide && p->wide->tc; }

int wide_set_tensor_core_adjoint(tt_plan *p, bool on) {
  WideState *w = p->wide;
  if (!w || p->precision != TT_PRECISION_F32 || w->SP != 64 || !w->store_products)
    return on ? wfail(TT_ERR_UNSUPPORTED,
                      "the tensor-core adjoint serves FP32 codon (> 20-state) plans that keep the children's products")
              : TT_OK;
  if (on && !w->d_pimg) {  // the split P^T images: 32 KB per (sample, branch, category)
    const size_t bytes = size_t(p->batch) * p->B * p->K * tcb::kImgFloats * sizeof(float);
    const int rc = walloc(p, &w->d_pimg, bytes, "split transition-matrix images");
    if (rc) return rc;
    w->img_b_valid = false;
  } else if (!on && w->d_pimg) {
    cudaFree(w->d_pimg);
    w->d_pimg = nullptr;
    p->bytes -= std::min(p->bytes, size_t(p->batch) * p->B * p->K * tcb::kImgFloats * sizeof(float));
  }
  w->tc_bwd = on;
  return TT_OK;
}

bool wide_tensor_core_adjoint(const tt_plan *p) { return p->wide && p->wide->tc_bwd; }

void wide_destroy(tt_plan *p) {
  WideState *w = p->wide;
  if (!w) return;
  void *bufs[] = {w->d_left, w->d_right, w->d_fwd, w->d_bwd, w->d_branch_lvn, w->d_part, w->d_expo, w->d_root_site, w->d_root_expo,
                  w->d_coef, w->d_cexp, w->d_block_lnl, w->d_gpart, w->d_rootpart, w->d_pgpart, w->d_prod, w->d_site,
                  w->d_pimg, w->d_pimg_f, w->d_tip_row, w->d_tip_amb, w->d_tprod[0], w->d_tprod[1]};
  for (void *x : bufs)
    if (x) cudaFree(x);
  delete w;
  p->wide = nullptr;
}

int wide_set_tips(tt_plan *p, const uint8_t *codes, const double *code_table, int code_count,
                  const double *weights) {
  const int SP = p->wide->SP;
  std::vector<unsigned char> table(size_t(code_count) * SP * p->elem, 0);
  for (int c = 0; c < code_count; ++c)
    for (int j = 0; j < p->S; ++j) {
      const double v = code_table[size_t(c) * p->S + j];
      if (p->precision == TT_PRECISION_F32) {
        const float f = float(v);
        std::memcpy(&table[(size_t(c) * SP + j) * 4], &f, 4);
      } else {
        std::memcpy(&table[(size_t(c) * SP + j) * 8], &v, 8);
      }
    }
  // codes whose product is a row of the staged P^T: unit vectors, and the first kTipRows others
  WideState &w = *p->wide;
  std::vector<uint8_t> rows(259, 0);
  std::vector<unsigned char> amb(size_t(kTipRows) * SP * p->elem, 0);
  int ambs = 0;
  bool ok = true;
  for (int c = 0; c < code_count; ++c) {
    int ones = 0, zeros = 0, s = 0;
    for (int j = 0; j < p->S; ++j) {
      const double v = code_table[size_t(c) * p->S + j];
      if (v == 1.0) s = j, ++ones;
      else zeros += v == 0.0;
    }
    if (ones == 1 && zeros == p->S - 1) {
      rows[c] = uint8_t(s);
    } else if (ambs < kTipRows) {
      rows[c] = uint8_t(SP + ambs);
      std::memcpy(&amb[size_t(ambs) * SP * p->elem], &table[size_t(c) * SP * p->elem], SP * p->elem);
      ++ambs;
    } else {
      ok = false;
    }
  }
  tip_table(p, code_count);
  rows[256] = ok;
  rows[257] = uint8_t(ambs);
  rows[258] = uint8_t(code_count - 1);
  cudaError_t e = cudaMemset(p->d_codes, 0, size_t(p->T) * p->code_stride);
  if (e == cudaSuccess) e = cudaMemcpy(w.d_tip_row, rows.data(), rows.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(w.d_tip_amb, amb.data(), amb.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy2D(p->d_codes, p->code_stride, codes, p->N, p->N, p->T, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p->d_table, table.data(), table.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(p->d_weights, weights, size_t(p->N) * sizeof(double), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return wcuda(e, "tt_plan_set_tips upload");
  return TT_OK;
}

int wide_update_matrices(tt_plan *p, const double *lam, const double *U, const double *W, const double *bl,
                         const double *rates, cudaStream_t s) {
  cudaError_t e = dispatch(p, [&](auto X) { return decltype(X)::pmatrix(p, lam, U, W, bl, rates, s); });
  return e == cudaSuccess ? TT_OK : wcuda(e, "transition-matrix launch");
}

int wide_set_matrices(tt_plan *p, const double *matrices, cudaStream_t s) {
  const int SP = p->wide->SP;
  const long long count = (long long)p->batch * p->B * p->K * SP * SP;
  const unsigned blocks = unsigned((count + 255) / 256);
  if (p->precision == TT_PRECISION_F32)
    wide_pmatrix_copy_kernel<float><<<blocks, 256, 0, s>>>(matrices, static_cast<float *>(p->d_pmat), p->S, SP, count);
  else
    wide_pmatrix_copy_kernel<double><<<blocks, 256, 0, s>>>(matrices, static_cast<double *>(p->d_pmat), p->S, SP,
                                                            count);
  p->launches += 1;
  p->wide->img_f_valid = p->wide->img_b_valid = false;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && p->precision == TT_PRECISION_F32 && SP == 64)  // the tensor-core kernels' images
    e = launch_pimages(p, p->wide->tc, p->wide->tc_bwd, s);
  return e == cudaSuccess ? TT_OK : wcuda(e, "transition-matrix copy launch");
}

int wide_log_likelihood(tt_plan *p, const double *props, const double *freqs, int rescale, bool keep, double *lnl,
                        double *site_lnl, cudaStream_t s) {
  WideState &w = *p->wide;
  if (!p->slab) {
    cudaError_t e = dispatch(
        p, [&](auto X) { return decltype(X)::forward(p, props, freqs, rescale, keep, lnl, site_lnl, 0, p->N, 0, s); });
    return e == cudaSuccess ? TT_OK : wcuda(e, "wide-state post-order launch");
  }
  // slab by slab, lnL summed over slabs; the last slab's post-order stays in
  // the buffers for the gradient
  cudaError_t e = cudaSuccess;
  for (int p0 = 0; p0 < p->N && e == cudaSuccess; p0 += p->slab) {
    const int n = std::min(p->slab, p->N - p0);
    const bool last = p0 + n == p->N;
    e = dispatch(p, [&](auto X) {
      return decltype(X)::forward(p, props, freqs, rescale, keep && last, lnl, site_lnl ? w.d_site : nullptr, p0, n,
                                  p0 > 0, s);
    });
    if (e == cudaSuccess && site_lnl)  // [b][n] rows into columns p0.. of [b][N]
      e = cudaMemcpy2DAsync(site_lnl + p0, size_t(p->N) * sizeof(double), w.d_site, size_t(n) * sizeof(double),
                            size_t(n) * sizeof(double), p->batch, cudaMemcpyDeviceToDevice, s);
  }
  if (e != cudaSuccess) return wcuda(e, "wide-state post-order launch");
  w.tail_valid = keep;
  return TT_OK;
}

int wide_gradient(tt_plan *p, const double *props, const double *freqs, double *grad_matrices,
                  double *grad_frequencies, double *grad_weights, cudaStream_t s) {
  WideState &w = *p->wide;
  cudaError_t e = cudaSuccess;
  if (!p->slab) {
    e = dispatch(p, [&](auto X) { return decltype(X)::backward(p, props, freqs, 0, p->N, 0, s); });
  } else {
    // slabs from the last: its post-order is still in the buffers after a
    // tt_log_likelihood with keep_partials; every other slab's is recomputed
    const int nslab = (p->N + p->slab - 1) / p->slab;
    for (int j = nslab - 1; j >= 0 && e == cudaSuccess; --j) {
      const int p0 = j * p->slab, n = std::min(p->slab, p->N - p0);
      if (!(j == nslab - 1 && w.tail_valid)) {
        e = dispatch(p, [&](auto X) {
          return decltype(X)::forward(p, props, freqs, p->last_rescale, true, nullptr, nullptr, p0, n, 0, s);
        });
        if (e != cudaSuccess) break;
      }
      e = dispatch(p, [&](auto X) { return decltype(X)::backward(p, props, freqs, p0, n, j != nslab - 1, s); });
    }
    w.tail_valid = false;  // the adjoint wrote over the partials
  }
  if (e != cudaSuccess) return wcuda(e, "wide-state adjoint launch");
  const size_t kss = size_t(p->K) * p->S * p->S;
  if (grad_matrices)
    e = cudaMemcpyAsync(grad_matrices, p->d_G, size_t(p->batch) * p->B * kss * sizeof(double),
                        cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess && grad_frequencies)
    e = cudaMemcpyAsync(grad_frequencies, p->d_rootgrad, size_t(p->batch) * p->S * sizeof(double),
                        cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess && grad_weights)
    e = cudaMemcpyAsync(grad_weights, p->d_rootgrad + size_t(p->batch) * p->S,
                        size_t(p->batch) * p->K * sizeof(double), cudaMemcpyDeviceToDevice, s);
  return e == cudaSuccess ? TT_OK : wcuda(e, "gradient copy");
}

int wide_matrices_gradient(tt_plan *p, const double *lam, const double *U, const double *W, const double *bl,
                           const double *rates, double *dlam, double *dU, double *dW, double *dbl, double *drates,
                           cudaStream_t s) {
  cudaError_t e = dispatch(p, [&](auto X) {
    return decltype(X)::pmatrix_backward(p, lam, U, W, bl, rates, dlam, dU, dW, dbl, drates, s);
  });
  return e == cudaSuccess ? TT_OK : wcuda(e, "transition-matrix gradient launch");
}

}  // namespace tt
