// cvo_internal.h -- internal types shared by the CUDA translation units.
//
// Data layout in HBM (replaces the reference's 176-240 B AoS CvoPoint records,
// include/UnifiedCvo/utils/PointSegmentedDistribution.hpp:51-144):
//   positions : float4 {x, y, z, w}   (w = ||p|| for sources, original index bits for targets)
//   features  : n * FP floats, FP = F rounded up to 4 (float4 loads)
//   labels    : n * CP floats, CP = C rounded up to 4
//   geom_type : float2
// Every cloud is additionally kept in "tile order" (Morton order): 32 consecutive points
// are a source tile of the association and a target group of it, with a bounding box in
// position and features; 32 consecutive groups are a supergroup, with a box of its own.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <utility>
#include <vector>
#include <map>
#include <new>
#include <nvtx3/nvToolsExt.h>
#include "../../include/cvo_gb300.h"

namespace cvo_gb {

constexpr int kWarp = 32;
constexpr int kMaxIndicatorWindow = 128;
constexpr int kMaxTargetBits = 22;          // targets per cloud <= 4M
// A row of an align or a window edge that keeps more than cap + order_cap pairs stays in index order
// (order_cap: kOrderCap, or less in large windows).
constexpr int kOrderCap = 4096;
constexpr int kGroup = 32;                  // points of a group, groups of a supergroup

inline int group_count(int n) { return (n + kGroup - 1) / kGroup; }
// Feature chunks (float4) of a bounding box: the association takes at most two.
inline int box_chunks(int FP) { return FP / 4 < 2 ? FP / 4 : 2; }

struct Handle;

// An order of a target cloud's points: by the cells of a lattice over the bounding box (z, then
// y, then x), inside a cell by index.  The align loop and the window solve keep the entries
// of a kernel-matrix row in this order and add them up in it, with the lattice that follows
// the search radius.
struct RankLevel {
  float h;                // cell size
  int *index;             // rank -> original index
  int *of_index;          // original index -> rank
  int *of_tile;           // tile-order position -> rank
};

// Device arrays that share one allocation, each on a 256-byte boundary: take() notes an array's
// pointer and size, allocate() sets the pointers.
struct Pieces {
  size_t bytes = 0;
  std::vector<std::pair<void *, size_t>> at;
  template <class T>
  void take(T **p, size_t count) {
    at.emplace_back(static_cast<void *>(p), bytes);
    bytes += (sizeof(T) * count + 255) & ~(size_t)255;
  }
  int allocate(Handle *h, char **base);      // the status of the allocation; base owns it
};

struct DevCloud {
  char *base = nullptr;          // of the arrays below
  int n = 0, F = 0, C = 0, FP = 0, CP = 0;
  bool has_geo = false;
  float bbmin[3] = {0, 0, 0}, bbmax[3] = {0, 0, 0};
  float max_norm = 0.f;
  float tile_ext = 0.f;          // mean bounding-box diagonal of 128 consecutive tile-order points
  // original order
  float4 *pos = nullptr;
  float *feat = nullptr;
  float *lab = nullptr;
  float2 *geo = nullptr;
  // tile order
  int *sperm = nullptr;          // tile-order position -> original index
  float4 *spos = nullptr;
  float *sfeat = nullptr;
  float *slab = nullptr;
  float2 *sgeo = nullptr;
  // bounding boxes of the groups, then of the supergroups: float4 planes (position low,
  // high, feature low, feature high; box_planes of them) of one entry per group
  float4 *gbox = nullptr, *sbox = nullptr;
  int2 *grange = nullptr;        // lowest and highest original index of a group's points
  std::map<int, RankLevel> ranks;          // by quantised cell size 2^(e/2), device arrays
  std::vector<void *> rank_allocs;
};

// ----------------------------------------------------------- kernel params
// Per-call kernel constants (identical for all pairs of a batch).
struct KParams {
  float sigma2, c2, c_sigma2, s_ell, s_sigma2, s_sigma_sq, sp_thres;
  float log_geo;         // logf(sp_thres / sigma2), evaluated on the host
  float d2_c_thres, d2_s_thres;
  float c, d;            // so(3) / R^3 inner-product scales
  float eps, eps_2, min_step, max_step;
  float ell_decay_rate, ell_min, indicator_stable_threshold;
  int ell_decay_start, indicator_window_size, max_iter, nn_max, use_range_ell_step;
  int use_geo, use_int, use_sem, use_gtype;
  float inv2c2;          // 1 / (2 c_ell^2), rounded once (IEEE division)
  // Candidate test: a kept pair needs d2/(2l^2) + d2c/(2c_ell^2) < mma_tau
  // (mma_tau = ln(sigma^2 c_sigma^2 s_sigma^2 / sp_thres) + slack), see k_cand.
  float mma_tau;
  int use_mma;
  // Pairs with the exponent below this are kept (0: semantic or geometric-type terms decide, too).
  float sure_tau;
  // Value scale (1 on the two-view path; c_sigma for the adaptive path's geometric-only
  // values s^2 exp(-d2/2l^2) c_sigma) and the colour denominator 2 c_ell^2 of the exact
  // (double) value as each path rounds it.
  float val_scale;
  double two_c2;
};

// Groups of the FP64 sums over a pair's rows (k_gradient, k_step): units of 32 rows in a slot,
// slots of the pair, slots of a block.
struct SumGroups {
  int slot_units, slots, block_slots;
};

// Per-pair device state.  One struct per pair, in device memory.
struct PairDev {
  // problem
  int n, m;                       // source rows, target points
  SumGroups sums;
  const float4 *xs;               // source, tile order (x,y,z,||x||)
  const float *xf, *xl;
  const float2 *xg;
  const float4 *sbox;             // source tiles' boxes
  // target, tile order
  const float4 *tpos;
  const int *tperm;               // tile-order position -> original index
  const float *tfs;
  const float4 *tbox, *tsup;      // boxes of groups and supergroups
  const int2 *trange;             // lowest and highest original index of a group's points
  int groups;
  float4 *ycur;                   // transformed targets, tile order
  float4 *yorig;                  // transformed targets, original order
  int *A_j; float *A_v;           // ELL, row-major: entry c of row s at [s * ld + c] (original target index)
  int ld;                         // ELL row pitch (capmax rounded up to a multiple of 4)
  // candidates: entry e of split q of row s at [s * cand_pitch + q * cap_split + e] =
  // {group, bits of its 32 points}; cand_cnt[q * n + s] = {entries and pairs surely kept,
  // candidates} (see kSureShift; more than cap_split entries: not all stored)
  uint2 *cand;
  int2 *cand_cnt;
  int splits, cap_split, cand_pitch;
  const float *tf, *tl;           // target features / labels, original order (float4 chunks)
  const float2 *tg;               // target geometric types, original order
  int *nnz_row;                   // n
  // align and edges: orders of the target's points, finest lattice first, and the largest search radius
  // each serves; order_cap as at kOrderCap, 0 for single passes (all rows in index order)
  const RankLevel *levels;
  float level_r[24];
  int nlevels, level, order_cap;
  float src_norm;                 // largest |x| of the source
  uint2 *long_rows;               // room to order rows of more than kRowOrdered entries (see build_batch)
  int long_pitch;
  double *part;                   // block partials
  unsigned int *counter;          // last-block counters [2]
  unsigned long long run_nnz;     // kept pairs and longest row of the pass so far
  unsigned int run_max;
  int F, C;                       // feature / label dimensions (source and target agree)
  int capmax;
  int mode;                       // 0 align, 1 inner product, 2 export, 3 edges of a window
  // iteration state
  float R[9], T[3];               // internal pose
  float Ri[9], Ti[3];             // target transform R^T, -R^T T
  float ell;
  int cap;
  int iter, done, ret;
  float xi[6];
  double grad[6];
  double asum;
  long long nnz_sum;
  int max_row;
  double bcde[4];
  double step, dist;
  // indicator queues (ring buffers)
  float qs[kMaxIndicatorWindow], qe[kMaxIndicatorWindow];
  int qs_head, qs_len, qe_head, qe_len;
  float ssum, esum;
};


// Batch of pairs processed together by every kernel launch.
struct BatchDev {
  int npairs;
  int total_items;                // work items of k_cand over all pairs (tiles x splits)
  int total_targets;              // sum of m
  PairDev *pairs;                 // device array
  const int *item_off;            // npairs + 1 (prefix of work items)
  const int *tgt_off;             // npairs + 1 (prefix of m)
  int *err;                       // error word (0 ok; no kernel of the engine sets it)
  const int *rblk_off;            // row-pass blocks per pair (prefix)
  const int *sblk_off;            // k_gradient and k_step blocks per pair (prefix)
  int total_rblocks, total_sblocks;
  int *heavy, *heavy_ctr;         // groups of long rows (see k_rows); their number, the next one
  int *active;                    // number of pairs not done
  int *active_iters;              // iterations that started with an active pair
  double *assoc_bytes;            // algorithmic bytes of the association passes
  int record_bytes;               // packed bytes of one target record
};

// Kernels of the association for a batch's feature and label strides (cvo_assoc_*.cu).
using CandFn = void (*)(BatchDev, KParams);
using RowsFn = void (*)(BatchDev, KParams, int);

struct AssocKernels {
  CandFn cand = nullptr;
  RowsFn rows[2] = {nullptr, nullptr}, ordered_rows[2] = {nullptr, nullptr};      // ROWS_ALL, ROWS_LIGHT
};

int assoc_kernels_no_labels(int fch, bool gt, AssocKernels *a);
int assoc_kernels_labels5(int fch, bool gt, AssocKernels *a);
int assoc_kernels_labels9(int fch, bool gt, AssocKernels *a);

// ------------------------------------------------------------- host side
struct Workspace;

struct Profile {
  bool on = false;
  double assoc_ms = 0.0;
  double kernel_ms[5] = {0, 0, 0, 0, 0};   // transform, assoc, reduce, step, all four
  double assoc_split_ms[3] = {0, 0, 0};    // candidate test, row pass, 0 (row sums: part of reduce)
  long long assoc_launches = 0;
  double assoc_bytes = 0.0;
  long long iterations = 0;
};

// Association tuning: how finely the candidate test divides the targets among warps.
// The splits per source tile scale with (cell_div_r / 4) (cell_div_ext / 8), and
// blocks_per_sm > 0 asks for that many times four work items per SM instead of the
// default.  Results do not depend on any of them (k_rows orders the candidates), only how
// the work spreads over the SMs does.
struct TuneConfig {
  float cell_div_r = 4.f;
  float cell_div_ext = 8.f;
  int blocks_per_sm = 0;
};

struct Handle {
  cvo_params params;
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;
  Profile prof;
  int device = 0;
  int num_sms = 0;
  long long launches = 0;
  std::string last_error;
  Workspace *ws = nullptr;
  std::map<long long, TuneConfig> tuned;    // (F, C, log2 rows) -> fastest division
  std::map<long long, int> tuned_bps;       // (F, C, log2 work items of a batch) -> blocks per SM
  const TuneConfig *tune_force = nullptr;   // set while the autotuner times a configuration
};

long long tune_key(int F, int C, long long rows);
// Association work items (128 source rows each) of a pair of `rows` source points.
long long tune_items(long long rows);
// Times one association pass of (src, tgt) at pose T and lengthscale ell for every
// candidate configuration and records the fastest for the batches that match its key.
int autotune_association(Handle *h, DevCloud *src, DevCloud *tgt, const float T[16], float ell, int reps,
                         std::vector<TuneConfig> *configs, std::vector<float> *ms, int *best);

// Label rows are padded to 5 float4 chunks (C <= 20) or 9 chunks (C <= 36).
inline int label_chunks(int C) { return C <= 0 ? 0 : (C <= 20 ? 5 : (C <= 36 ? 9 : (C + 3) / 4)); }

// RGB-D frame -> device cloud, device cloud -> host arrays (cvo_frontend.cu)
int cloud_from_rgbd(Handle *h, const uint8_t *image, int rows, int cols, int channels, const float *depth,
                    const float intrinsic[4], float scaling_factor, const int *uv, int n_sel, const float *geom_type,
                    int num_classes, const float *semantics, DevCloud **out);
int cloud_download(Handle *h, const DevCloud *d, float *xyz, float *features, float *labels, float *geom_type);

// grid / cloud management (cvo_grid.cu)
int cloud_upload(Handle *h, const cvo_cloud *c, DevCloud **out);
// A cloud from device arrays (xyz n x 3, features n x F, labels n x C, geometric
// types n float2 or null); the arrays stay owned by the caller.
int cloud_from_device(Handle *h, int n, int F, int C, const float *xyz_d, const float *feat_d, const float *lab_d,
                      const float2 *geo_d, DevCloud **out);
void cloud_free(DevCloud *c);
float level_cell_size(int level_exp);
int level_for_radius(float r);
// Orders of the cloud by the lattices of the given exponents (built once per cloud).
int cloud_ranks(Handle *h, DevCloud *c, const std::vector<int> &exps);

// radix sort / scan (cvo_sort.cu)
int radix_sort_pairs(Handle *h, unsigned int *keys, int *vals, unsigned int *keys_tmp, int *vals_tmp,
                     int n, int key_bits);
void exclusive_scan_int(Handle *h, const int *in, int *out, int n, int *scratch, int scratch_n);
size_t scan_scratch_ints(int n);

// engine (cvo_engine.cu)
KParams make_kparams(const cvo_params &p);
struct BatchResult {
  std::vector<float> T_out;     // 16 per pair, column-major [R^T, -R^T T]
  std::vector<int> ret, iters;
  std::vector<double> asum;
  std::vector<long long> nnz;
};
int run_align_batch(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                    const std::vector<float> &T_init, BatchResult *res, double *secs,
                    bool export_assoc, std::vector<std::vector<int>> *a_rows,
                    std::vector<std::vector<int>> *a_cols, std::vector<std::vector<float>> *a_vals);
int run_inner_product_batch(Handle *h, DevCloud *src, DevCloud *tgt, const std::vector<float> &T, float ell,
                            int cap, std::vector<double> *asum, std::vector<long long> *nnz,
                            bool export_assoc, std::vector<int> *a_rowptr_host, std::vector<int> *a_cols,
                            std::vector<float> *a_vals);

// Inner products of independent (source, target, pose) triples in one batch.
int run_inner_product_pairs(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                            const std::vector<float> &T, float ell, int cap, std::vector<double> *asum);

// One association pass per edge between world-frame clouds (multi-frame solver).
// src_world: per edge, the source frame's points already in world coordinates in
// tile order ({x, y, z, ||x||}) and an upper bound of their norms; tgt_pose: per edge 12 floats, the target frame's
// pose (row-major 3x4, frame -> world) applied to the target points.  The result
// arrays stay valid until the next batch is built on the handle.
struct EdgeAssoc {
  const int *A_j;        // ELL, row-major over tile-ordered rows (pitch ld), original target indices
  const float *A_v;
  int ld;
  const int *nnz_row;
  int n, m;
  long long nnz;
  int max_row;
};
// Replayable launch sequence of an edge-association batch: the upload of the pair
// records, the association kernels, and the read-back of the records and of the error
// word, captured once as a CUDA graph and relaunched while the batch's launch
// parameters are byte-identical.  The pair records travel through pinned staging
// buffers, whose addresses the graph's copy nodes hold.  One object serves the
// successive batches of one caller (the outer iterations of a window solve).
struct AssocGraph {
  cudaGraphExec_t exec = nullptr;
  std::vector<unsigned char> key;
  long long launches = 0;       // kernel launches of one replay
  PairDev *pin_in = nullptr, *pin_out = nullptr;
  int *pin_err = nullptr;
  int pin_pairs = 0;
  AssocGraph() = default;
  AssocGraph(const AssocGraph &) = delete;
  AssocGraph &operator=(const AssocGraph &) = delete;
  ~AssocGraph();
};
int run_association_edges(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                          const std::vector<const float4 *> &src_world, const std::vector<float> &src_world_norm,
                          const std::vector<float> &tgt_pose, const std::vector<float> &ells,
                          const std::vector<int> &caps, int capmax, std::vector<EdgeAssoc> *out,
                          const KParams *kparams = nullptr, AssocGraph *graph = nullptr);

// ELL rows on the device (ELL row s is row perm[s], or s if perm is null; nnz[s] entries at s * ld)
// to CSR on the host.
int csr_to_host(Handle *h, int n, const int *nnz, const int *perm, int ld, const int *ell_j, const float *ell_v,
                std::vector<int> *rowptr, std::vector<int> *col, std::vector<float> *val);

// Non-isotropic association (cvo_aniso.cu): CSR of the kernel matrix with a 3x3
// geometric kernel (column-major), first `cap` pairs per row in index order.
void kernel_inverse3(const float K[9], float Ki[9]);
int run_association_aniso(Handle *h, DevCloud *src, DevCloud *tgt, const float T[16], const float kernel[9],
                          int cap, std::vector<int> *rowptr, std::vector<int> *col, std::vector<float> *val);

// Adaptive-lengthscale CVO (cvo_adaptive.cu).  trace (optional): per iteration
// {ell, dl, step, nnz A, nnz Axx, nnz Ayy}.
int run_association_adaptive(Handle *h, DevCloud *src, DevCloud *tgt, const float T[16], float ell,
                             std::vector<int> *rowptr, std::vector<int> *col, std::vector<float> *val);
int run_align_adaptive(Handle *h, DevCloud *src, DevCloud *tgt, const float T_init[16], float T_out[16],
                       double *secs, int *iters_out, double *trace, int trace_len);

// IRLS (cvo_irls.cu)
int run_align_multi(Handle *h, int n_frames, DevCloud *const *clouds, double *poses, const uint8_t *hold_const,
                    int n_edges, const int *edges, double *secs, int *iters);

// Learned pose proposal (cvo_learn.cu)
struct NetDev;
size_t net_num_params();
int net_create(Handle *h, int P, unsigned seed, NetDev **out);
void net_destroy(NetDev *n);
int net_points(const NetDev *n);
int net_forward_pool(Handle *h, NetDev *n, int n_scenes, int n_pts, const float *src, const float *tgt, int Bn,
                     const int *scene, const float *T_tgt, uint32_t seed, float *raw_out, float *T_out);
int net_hypotheses(Handle *h, NetDev *n, int Bn, DevCloud *const *src, DevCloud *const *tgt, uint32_t seed,
                   float *T_out);
int net_train_pool(Handle *h, NetDev *n, int n_scenes, int n_pts, const float *src, const float *tgt, int Bn,
                   const int *scene, const float *T_label, float lr, uint32_t seed, float *loss_out);
int net_get(Handle *h, NetDev *n, int which, float *out);
int net_set(Handle *h, NetDev *n, const float *in);
int net_set_gemm(NetDev *n, int kind);

// error helpers
int set_cuda_error(Handle *h, cudaError_t e, const char *where);
#define CVO_CUDA_TRY(h, call)                                      \
  do {                                                             \
    cudaError_t e__ = (call);                                      \
    if (e__ != cudaSuccess) return set_cuda_error((h), e__, #call); \
  } while (0)

// NVTX range over a host phase (no-op unless a profiler is attached): ncu can select
// launches by phase with --nvtx --nvtx-include "<name>/".
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// Status of the exception being handled: the C entry points catch everything, so no
// C++ exception crosses the C ABI (host allocation failure -> out of memory).
inline int status_from_exception() {
  try {
    throw;
  } catch (const std::bad_alloc &) {
    return CVO_ERR_OUT_OF_MEMORY;
  } catch (...) {
    return CVO_ERR_INVALID_ARG;
  }
}

}  // namespace cvo_gb
