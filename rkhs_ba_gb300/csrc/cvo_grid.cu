// cvo_grid.cu -- device clouds: packed SoA upload, tile (Morton) order, and bounding
// boxes of the groups of 32 tile-order points.
//
// Replaces CvoPointCloud_to_gpu (src/cvo/CvoGPU_impl.cu:220-289) and the kd-tree
// association structure (thirdparty/cugicp/cukdtree/cukdtree.cuh:236-509): the boxes do
// not depend on the lengthscale, so one build serves every call, and they bound the
// features as well as the positions.
#include <cmath>
#include <cstring>
#include <algorithm>
#include "cvo_internal.h"
#include "cvo_device.cuh"

namespace cvo_gb {

float level_cell_size(int e) { return exp2f(0.5f * (float)e); }

// Smallest quantised cell size h = 2^(e/2) with h >= r.
int level_for_radius(float r) {
  if (!(r > 0.f)) return -60;
  if (!std::isfinite(r)) return 1000;
  int e = (int)std::ceil(2.0 * std::log2((double)r));
  while (level_cell_size(e) < r) e++;
  while (e > -60 && level_cell_size(e - 1) >= r) e--;
  return e;
}

namespace {

__global__ void k_pack_positions(const float *xyz, int stride, int n, float4 *pos) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x = xyz[(size_t)i * stride], y = xyz[(size_t)i * stride + 1], z = xyz[(size_t)i * stride + 2];
  pos[i] = make_float4(x, y, z, range_norm(x, y, z));
}

__global__ void k_pad_rows(const float *in, int n, int F, int FP, float *out) {
  size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)n * FP) return;
  int i = (int)(t / FP), k = (int)(t % FP);
  out[t] = (k < F) ? in[(size_t)i * F + k] : 0.f;
}

__device__ __forceinline__ unsigned int spread10(unsigned int v) {
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__global__ void k_morton(const float4 *pos, int n, float ox, float oy, float oz, float inv, unsigned int *keys,
                         int *vals) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = pos[i];
  auto q = [&](float v, float o) {
    float c = (v - o) * inv;
    c = fminf(fmaxf(c, 0.f), 1023.f);
    return (unsigned int)c;
  };
  keys[i] = spread10(q(p.x, ox)) | (spread10(q(p.y, oy)) << 1) | (spread10(q(p.z, oz)) << 2);
  vals[i] = i;
}

__global__ void k_gather_source(const int *perm, int n, const float4 *pos, const float *feat, int FP, const float *lab,
                                int CP, const float2 *geo, float4 *spos, float *sfeat, float *slab, float2 *sgeo) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int i = perm[s];
  spos[s] = pos[i];
  for (int k = 0; k < FP; k++) sfeat[(size_t)s * FP + k] = feat[(size_t)i * FP + k];
  for (int k = 0; k < CP; k++) slab[(size_t)s * CP + k] = lab[(size_t)i * CP + k];
  if (geo) sgeo[s] = geo[i];
}

// Bounding boxes of 32 consecutive items, one warp per box.  LEVEL 0: points (tile-order
// positions and features); LEVEL 1: boxes of LEVEL 0.  Planes as in cvo_kernels.cuh.
template <int LEVEL>
__global__ void __launch_bounds__(128) k_boxes(const float4 *pos, const float4 *feat, int stride, int count, int chunks,
                                               float4 *out, int boxes) {
  const int lane = threadIdx.x & 31, g = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (g >= boxes) return;
  const int i = min(32 * g + lane, count - 1);      // spare lanes repeat the last item
  for (int k = 0; k < 1 + chunks; k++) {
    float4 lo, hi;
    if (LEVEL == 0) {
      lo = hi = k == 0 ? pos[i] : feat[(size_t)i * stride + k - 1];
    } else {
      lo = pos[(size_t)(k == 0 ? 0 : 1 + k) * count + i];
      hi = pos[(size_t)(k == 0 ? 1 : 1 + chunks + k) * count + i];
    }
    lo = make_float4(warp_fmin(lo.x), warp_fmin(lo.y), warp_fmin(lo.z), warp_fmin(lo.w));
    hi = make_float4(warp_fmax(hi.x), warp_fmax(hi.y), warp_fmax(hi.z), warp_fmax(hi.w));
    if (lane == 0) {
      out[(size_t)(k == 0 ? 0 : 1 + k) * boxes + g] = lo;
      out[(size_t)(k == 0 ? 1 : 1 + chunks + k) * boxes + g] = hi;
    }
  }
}

// Bounding-box diagonals of 128 consecutive tile-order points (four groups).
__global__ void k_tile_extent(const float4 *box, int groups, int tiles, float *ext) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= tiles) return;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int g = 4 * t; g < min(4 * t + 4, groups); g++) {
    const float4 a = box[g], b = box[groups + g];
    lo[0] = fminf(lo[0], a.x); lo[1] = fminf(lo[1], a.y); lo[2] = fminf(lo[2], a.z);
    hi[0] = fmaxf(hi[0], b.x); hi[1] = fmaxf(hi[1], b.y); hi[2] = fmaxf(hi[2], b.z);
  }
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  ext[t] = sqrtf(dx * dx + dy * dy + dz * dz);
}

// A lattice of rank level q of a joint build: cell c of axis k covers [o + c h, o + (c + 1) h).
struct Lattice {
  float ox, oy, oz, inv_h;
  int dimx, dimy, dimz;
};
constexpr int kMaxLattices = 24;
struct Lattices {
  Lattice l[kMaxLattices];
};

__device__ __forceinline__ unsigned long long lattice_cell(const Lattice &L, const float4 &p) {
  const int cx = min(max((int)floorf((p.x - L.ox) * L.inv_h), 0), L.dimx - 1);
  const int cy = min(max((int)floorf((p.y - L.oy) * L.inv_h), 0), L.dimy - 1);
  const int cz = min(max((int)floorf((p.z - L.oz) * L.inv_h), 0), L.dimz - 1);
  return ((unsigned long long)cz * L.dimy + cy) * L.dimx + cx;
}

// Sort keys of `count` lattices at once: the lattice's number above `bits` bits of the cell.
// hi (single lattice of more than 32 bits): the upper half of the cell number.
__global__ void k_rank_keys(const float4 *pos, int n, Lattices L, int count, int bits, unsigned int *key, unsigned int *hi,
                            int *val) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * count) return;
  const int q = t / n, j = t - q * n;
  const unsigned long long c = lattice_cell(L.l[q], pos[j]);
  key[t] = hi ? (unsigned int)c : ((unsigned int)q << bits) | (unsigned int)c;
  if (hi) hi[t] = (unsigned int)(c >> 32);
  val[t] = j;
}

__global__ void k_rank_upper(const unsigned int *hi, const int *val, int n, unsigned int *key) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) key[t] = hi[val[t]];
}

// Sorted indices of `count` lattices -> the arrays of each (3 n ints: index, of_index, of_tile).
__global__ void k_rank_arrays(const int *val, int n, int count, int *out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * count) return;
  const int q = t / n, r = t - q * n, j = val[t];
  int *o = out + 3 * (size_t)q * n;
  o[r] = j;
  o[n + j] = r;
}
__global__ void k_rank_tiles(const int *sperm, int n, int count, int *out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * count) return;
  const int q = t / n, s = t - q * n;
  int *o = out + 3 * (size_t)q * n;
  o[2 * (size_t)n + s] = o[n + sperm[s]];
}

template <typename T>
int dalloc(Handle *h, T **p, size_t count) {
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc((void **)p, sizeof(T) * count);
  if (e != cudaSuccess) {
    set_cuda_error(h, e, "cudaMalloc");
    return e == cudaErrorMemoryAllocation ? CVO_ERR_OUT_OF_MEMORY : CVO_ERR_CUDA;
  }
  return 0;
}

// Lowest and highest original index of each group's points, a warp per group.
__global__ void k_group_range(const int *sperm, int n, int ng, int2 *range) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, i = 32 * g + (threadIdx.x & 31);
  if (g >= ng) return;
  const int j = i < n ? sperm[i] : sperm[n - 1];
  const int lo = __reduce_min_sync(0xFFFFFFFFu, j), hi = __reduce_max_sync(0xFFFFFFFFu, j);
  if ((threadIdx.x & 31) == 0) range[g] = make_int2(lo, hi);
}

}  // namespace

int Pieces::allocate(Handle *h, char **base) {
  CVO_CUDA_TRY(h, cudaMalloc((void **)base, bytes > 0 ? bytes : 256));
  for (auto &p : at) {
    char *q = *base + p.second;
    memcpy(p.first, &q, sizeof(q));
  }
  return 0;
}

// Device part of a cloud's construction from staged device arrays (xyz with stride
// 3 or 4, features n x F, labels n x C, geometric types n float2 or null) and its
// bounding box: packed original-order records, Morton tile order, tile extents.
static int cloud_build(Handle *h, DevCloud *d, const float *xyz_d, int stride, const float *feat_in,
                       const float *lab_in, const float2 *geo_in, const float mn[3], const float mx[3]) {
  const int n = d->n;
  int rc = 0;
  // one allocation for everything that the cloud keeps and one for the sort: an allocation or a
  // release costs as much as several of the kernels below
  const int ng = group_count(n), ns = group_count(ng), ch = box_chunks(d->FP);
  Pieces keep, tmp;
  keep.take(&d->pos, n);
  keep.take(&d->feat, (size_t)n * d->FP);
  keep.take(&d->lab, (size_t)n * d->CP);
  keep.take(&d->sperm, n);
  keep.take(&d->spos, n);
  keep.take(&d->sfeat, (size_t)n * d->FP);
  keep.take(&d->slab, (size_t)n * d->CP);
  if (d->has_geo) {
    keep.take(&d->geo, n);
    keep.take(&d->sgeo, n);
  }
  keep.take(&d->gbox, (size_t)(2 + 2 * ch) * ng);
  keep.take(&d->sbox, (size_t)(2 + 2 * ch) * ns);
  keep.take(&d->grange, ng);
  if ((rc = keep.allocate(h, &d->base))) return rc;
  unsigned int *keys = nullptr, *keys_tmp = nullptr;
  int *perm_tmp = nullptr;
  char *tmp_d = nullptr;
  tmp.take(&keys, n);
  tmp.take(&keys_tmp, n);
  tmp.take(&perm_tmp, n);
  if ((rc = tmp.allocate(h, &tmp_d))) return rc;
  k_pack_positions<<<(n + 255) / 256, 256, 0, h->stream>>>(xyz_d, stride, n, d->pos);
  h->launches++;
  if (d->FP > 0) {
    size_t tot = (size_t)n * d->FP;
    k_pad_rows<<<(unsigned)((tot + 255) / 256), 256, 0, h->stream>>>(feat_in, n, d->F, d->FP, d->feat);
    h->launches++;
  }
  if (d->CP > 0) {
    size_t tot = (size_t)n * d->CP;
    k_pad_rows<<<(unsigned)((tot + 255) / 256), 256, 0, h->stream>>>(lab_in, n, d->C, d->CP, d->lab);
    h->launches++;
  }
  if (d->has_geo)
    CVO_CUDA_TRY(h, cudaMemcpyAsync(d->geo, geo_in, sizeof(float2) * n, cudaMemcpyDeviceToDevice, h->stream));

  // tile order: Morton order of a 1024^3 lattice over the bounding box
  float ext = std::max(std::max(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]);
  float inv = ext > 0 ? 1023.999f / ext : 0.f;
  k_morton<<<(n + 255) / 256, 256, 0, h->stream>>>(d->pos, n, mn[0], mn[1], mn[2], inv, keys, d->sperm);
  h->launches++;
  if ((rc = radix_sort_pairs(h, keys, d->sperm, keys_tmp, perm_tmp, n, 30))) {
    cudaFree(tmp_d);
    return rc;
  }
  k_gather_source<<<(n + 255) / 256, 256, 0, h->stream>>>(d->sperm, n, d->pos, d->feat, d->FP, d->lab, d->CP, d->geo,
                                                         d->spos, d->sfeat, d->slab, d->sgeo);
  h->launches++;
  // boxes of the groups and supergroups
  k_group_range<<<(ng + 3) / 4, 128, 0, h->stream>>>(d->sperm, n, ng, d->grange);
  k_boxes<0><<<(ng + 3) / 4, 128, 0, h->stream>>>(d->spos, reinterpret_cast<const float4 *>(d->sfeat), d->FP / 4, n, ch,
                                                  d->gbox, ng);
  k_boxes<1><<<(ns + 3) / 4, 128, 0, h->stream>>>(d->gbox, nullptr, 0, ng, ch, d->sbox, ns);
  const int tiles = (n + 127) / 128;
  float *ext_d = reinterpret_cast<float *>(keys);
  k_tile_extent<<<(tiles + 127) / 128, 128, 0, h->stream>>>(d->gbox, ng, tiles, ext_d);
  h->launches += 4;
  std::vector<float> ext_h(tiles);
  CVO_CUDA_TRY(h, cudaMemcpyAsync(ext_h.data(), ext_d, sizeof(float) * tiles, cudaMemcpyDeviceToHost, h->stream));
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  double es = 0.0;
  for (float e : ext_h) es += e;
  d->tile_ext = tiles > 0 ? (float)(es / tiles) : 0.f;
  cudaFree(tmp_d);
  return 0;
}

static DevCloud *new_cloud(int n, int F, int C, bool has_geo) {
  DevCloud *d = new DevCloud();
  d->n = n; d->F = F; d->C = C;
  d->FP = (F + 3) / 4 * 4;
  d->CP = 4 * label_chunks(C);
  d->has_geo = has_geo;
  return d;
}

static void set_extent(DevCloud *d, const float mn[3], const float mx[3], double maxn2) {
  for (int k = 0; k < 3; k++) { d->bbmin[k] = mn[k]; d->bbmax[k] = mx[k]; }
  d->max_norm = (float)std::sqrt(maxn2) * (1.f + 1e-6f);
}

int cloud_upload(Handle *h, const cvo_cloud *c, DevCloud **out) {
  NvtxRange nvtx_range("cloud_upload");
  if (!c || !out) return CVO_ERR_INVALID_ARG;
  if (c->n < 0 || c->F < 0 || c->C < 0) return CVO_ERR_INVALID_ARG;
  if (c->n > 0 && (!c->xyz || (c->xyz_stride != 3 && c->xyz_stride != 4))) return CVO_ERR_INVALID_ARG;
  if (c->F > 0 && c->n > 0 && !c->features) return CVO_ERR_INVALID_ARG;
  if (c->C > 0 && c->n > 0 && !c->labels) return CVO_ERR_INVALID_ARG;
  if (c->n > (1 << kMaxTargetBits)) return CVO_ERR_CAPACITY;
  int n = c->n;
  // bounding box and largest range on the host (input is host memory)
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  double maxn2 = 0;
  for (int i = 0; i < n; i++) {
    const float *p = c->xyz + (size_t)i * c->xyz_stride;
    for (int k = 0; k < 3; k++) {
      if (!std::isfinite(p[k])) return CVO_ERR_INVALID_ARG;
      mn[k] = std::min(mn[k], p[k]);
      mx[k] = std::max(mx[k], p[k]);
    }
    double n2 = (double)p[0] * p[0] + (double)p[1] * p[1] + (double)p[2] * p[2];
    maxn2 = std::max(maxn2, n2);
  }
  if (n == 0) { for (int k = 0; k < 3; k++) mn[k] = mx[k] = 0.f; }
  DevCloud *d = new_cloud(n, c->F, c->C, c->geom_type != nullptr);
  set_extent(d, mn, mx, maxn2);
  *out = d;
  if (n == 0) return 0;

  float *xyz_d = nullptr, *feat_in = nullptr, *lab_in = nullptr;
  float2 *geo_in = nullptr;
  char *staged = nullptr;
  int rc = 0;
  Pieces in;
  in.take(&xyz_d, (size_t)n * c->xyz_stride);
  in.take(&feat_in, (size_t)n * c->F);
  in.take(&lab_in, (size_t)n * c->C);
  if (d->has_geo) in.take(&geo_in, n);
  if ((rc = in.allocate(h, &staged))) return rc;
  auto release = [&]() { cudaFree(staged); };
  CVO_CUDA_TRY(h, cudaMemcpyAsync(xyz_d, c->xyz, sizeof(float) * (size_t)n * c->xyz_stride, cudaMemcpyHostToDevice,
                                  h->stream));
  if (d->FP > 0)
    CVO_CUDA_TRY(h, cudaMemcpyAsync(feat_in, c->features, sizeof(float) * (size_t)n * c->F, cudaMemcpyHostToDevice,
                                    h->stream));
  if (d->CP > 0)
    CVO_CUDA_TRY(h, cudaMemcpyAsync(lab_in, c->labels, sizeof(float) * (size_t)n * c->C, cudaMemcpyHostToDevice,
                                    h->stream));
  if (d->has_geo)
    CVO_CUDA_TRY(h, cudaMemcpyAsync(geo_in, c->geom_type, sizeof(float2) * n, cudaMemcpyHostToDevice, h->stream));
  rc = cloud_build(h, d, xyz_d, c->xyz_stride, feat_in, lab_in, geo_in, mn, mx);
  release();
  return rc;
}

// Bounding box (min, max per axis) and largest squared norm of n device points
// (xyz stride 3), one block.
__global__ void k_extent(const float *xyz, int n, float *box, double *maxn2) {
  __shared__ float sl[3][256], sh[3][256];
  __shared__ double sn[256];
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  double m2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float *p = xyz + 3 * (size_t)i;
    for (int k = 0; k < 3; k++) { lo[k] = fminf(lo[k], p[k]); hi[k] = fmaxf(hi[k], p[k]); }
    m2 = fmax(m2, (double)p[0] * p[0] + (double)p[1] * p[1] + (double)p[2] * p[2]);
  }
  for (int k = 0; k < 3; k++) { sl[k][threadIdx.x] = lo[k]; sh[k][threadIdx.x] = hi[k]; }
  sn[threadIdx.x] = m2;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int t = 1; t < blockDim.x; t++) {
      for (int k = 0; k < 3; k++) { lo[k] = fminf(lo[k], sl[k][t]); hi[k] = fmaxf(hi[k], sh[k][t]); }
      m2 = fmax(m2, sn[t]);
    }
    for (int k = 0; k < 3; k++) { box[k] = lo[k]; box[3 + k] = hi[k]; }
    *maxn2 = m2;
  }
}

int cloud_from_device(Handle *h, int n, int F, int C, const float *xyz_d, const float *feat_d, const float *lab_d,
                      const float2 *geo_d, DevCloud **out) {
  if (n < 0 || F < 0 || C < 0 || !out) return CVO_ERR_INVALID_ARG;
  if (n > (1 << kMaxTargetBits)) return CVO_ERR_CAPACITY;
  float mn[3] = {0.f, 0.f, 0.f}, mx[3] = {0.f, 0.f, 0.f};
  double maxn2 = 0.0;
  if (n > 0) {
    float *box = nullptr;
    double *m2 = nullptr;
    int rc = 0;
    if ((rc = dalloc(h, &box, 6)) || (rc = dalloc(h, &m2, 1))) { cudaFree(box); return rc; }
    k_extent<<<1, 256, 0, h->stream>>>(xyz_d, n, box, m2);
    h->launches++;
    float bh[6];
    cudaError_t e = cudaMemcpyAsync(bh, box, sizeof(bh), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&maxn2, m2, sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    cudaFree(box);
    cudaFree(m2);
    if (e != cudaSuccess) return set_cuda_error(h, e, "cloud extent");
    for (int k = 0; k < 3; k++) { mn[k] = bh[k]; mx[k] = bh[3 + k]; }
  }
  DevCloud *d = new_cloud(n, F, C, geo_d != nullptr);
  set_extent(d, mn, mx, maxn2);
  *out = d;
  if (n == 0) return 0;
  return cloud_build(h, d, xyz_d, 3, feat_d, lab_d, geo_d, mn, mx);
}

void cloud_free(DevCloud *d) {
  if (!d) return;
  cudaFree(d->base);
  for (void *p : d->rank_allocs) cudaFree(p);
  delete d;
}

// Lattices whose cell numbers fit are sorted together (one radix sort over all of them, the
// lattice's number in the top bits): an align wants the orders of every lengthscale it may
// reach, and a sort of some 10^4 keys is launches, not work.
int cloud_ranks(Handle *h, DevCloud *d, const std::vector<int> &exps) {
  const int n = d->n;
  if (n == 0) return 0;
  struct Want { int e, bits; Lattice l; float h; };
  std::vector<Want> joint, single;
  for (int e : exps) {
    if (d->ranks.count(e)) continue;
    Want w;
    w.e = e;
    float ext[3];
    for (int k = 0; k < 3; k++) ext[k] = d->bbmax[k] - d->bbmin[k];
    float hsz = (e >= 1000) ? INFINITY : level_cell_size(e);
    // keep at most 2^20 cells per axis
    float emax = std::max(std::max(ext[0], ext[1]), ext[2]);
    if (std::isfinite(hsz) && emax / hsz > 1048000.f) hsz = emax / 1048000.f;
    w.h = hsz;
    w.l.inv_h = std::isfinite(hsz) ? 1.f / hsz : 0.f;
    w.l.ox = d->bbmin[0]; w.l.oy = d->bbmin[1]; w.l.oz = d->bbmin[2];
    w.l.dimx = std::isfinite(hsz) ? (int)std::floor(ext[0] * w.l.inv_h) + 1 : 1;
    w.l.dimy = std::isfinite(hsz) ? (int)std::floor(ext[1] * w.l.inv_h) + 1 : 1;
    w.l.dimz = std::isfinite(hsz) ? (int)std::floor(ext[2] * w.l.inv_h) + 1 : 1;
    const double cells = (double)w.l.dimx * w.l.dimy * w.l.dimz;
    w.bits = 1;
    while (w.bits < 63 && std::ldexp(1.0, w.bits) < cells) w.bits++;
    (w.bits <= 27 ? joint : single).push_back(w);
  }
  auto build = [&](const Want *w, int count) -> int {
    int bits = 1, lattice_bits = 0;
    for (int q = 0; q < count; q++) bits = std::max(bits, w[q].bits);
    while ((1 << lattice_bits) < count) lattice_bits++;
    const bool wide = bits + lattice_bits > 32;
    const size_t N = (size_t)n * count;
    unsigned int *key = nullptr;
    int *arrays = nullptr;
    CVO_CUDA_TRY(h, cudaMalloc((void **)&arrays, sizeof(int) * 3 * N));
    d->rank_allocs.push_back(arrays);
    CVO_CUDA_TRY(h, cudaMallocAsync((void **)&key, sizeof(int) * 5 * N, h->stream));
    unsigned int *key_tmp = key + N, *hi = key_tmp + N;
    int *val = reinterpret_cast<int *>(hi + N), *val_tmp = val + N;
    Lattices L;
    memset(&L, 0, sizeof(L));
    for (int q = 0; q < count; q++) L.l[q] = w[q].l;
    const unsigned blocks = (unsigned)((N + 255) / 256);
    k_rank_keys<<<blocks, 256, 0, h->stream>>>(d->pos, n, L, count, bits, key, wide ? hi : nullptr, val);
    int rc = radix_sort_pairs(h, key, val, key_tmp, val_tmp, (int)N, wide ? 32 : bits + lattice_bits);
    if (!rc && wide) {
      k_rank_upper<<<blocks, 256, 0, h->stream>>>(hi, val, n, key);
      h->launches++;
      rc = radix_sort_pairs(h, key, val, key_tmp, val_tmp, n, bits - 32);
    }
    if (!rc) {
      k_rank_arrays<<<blocks, 256, 0, h->stream>>>(val, n, count, arrays);
      k_rank_tiles<<<blocks, 256, 0, h->stream>>>(d->sperm, n, count, arrays);
    }
    h->launches += 3;
    CVO_CUDA_TRY(h, cudaFreeAsync(key, h->stream));
    if (rc) return rc;
    for (int q = 0; q < count; q++) {
      int *a = arrays + 3 * (size_t)q * n;
      d->ranks[w[q].e] = RankLevel{w[q].h, a, a + n, a + 2 * (size_t)n};
    }
    return 0;
  };
  // at most 2^25 keys in one sort
  const int most = std::max(1, std::min({kMaxLattices, 16, (1 << 25) / n}));
  for (size_t q = 0; q < joint.size(); q += most)
    if (int rc = build(&joint[q], (int)std::min<size_t>(most, joint.size() - q))) return rc;
  for (const Want &w : single)
    if (int rc = build(&w, 1)) return rc;
  return 0;
}

}  // namespace cvo_gb
