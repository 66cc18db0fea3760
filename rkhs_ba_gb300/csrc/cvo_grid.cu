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

}  // namespace

// Device part of a cloud's construction from staged device arrays (xyz with stride
// 3 or 4, features n x F, labels n x C, geometric types n float2 or null) and its
// bounding box: packed original-order records, Morton tile order, tile extents.
static int cloud_build(Handle *h, DevCloud *d, const float *xyz_d, int stride, const float *feat_in,
                       const float *lab_in, const float2 *geo_in, const float mn[3], const float mx[3]) {
  const int n = d->n;
  int rc = 0;
  int *perm_vals = nullptr, *perm_tmp = nullptr;
  unsigned int *keys = nullptr, *keys_tmp = nullptr;
  if ((rc = dalloc(h, &d->pos, n)) || (rc = dalloc(h, &d->feat, (size_t)n * d->FP)) ||
      (rc = dalloc(h, &d->lab, (size_t)n * d->CP)) || (rc = dalloc(h, &d->sperm, n)) ||
      (rc = dalloc(h, &d->spos, n)) || (rc = dalloc(h, &d->sfeat, (size_t)n * d->FP)) ||
      (rc = dalloc(h, &d->slab, (size_t)n * d->CP)))
    return rc;
  if (d->has_geo) {
    if ((rc = dalloc(h, &d->geo, n)) || (rc = dalloc(h, &d->sgeo, n))) return rc;
  }
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
  if ((rc = dalloc(h, &keys, n)) || (rc = dalloc(h, &keys_tmp, n)) || (rc = dalloc(h, &perm_vals, n)) ||
      (rc = dalloc(h, &perm_tmp, n)))
    return rc;
  float ext = std::max(std::max(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]);
  float inv = ext > 0 ? 1023.999f / ext : 0.f;
  k_morton<<<(n + 255) / 256, 256, 0, h->stream>>>(d->pos, n, mn[0], mn[1], mn[2], inv, keys, perm_vals);
  h->launches++;
  if ((rc = radix_sort_pairs(h, keys, perm_vals, keys_tmp, perm_tmp, n, 30))) return rc;
  CVO_CUDA_TRY(h, cudaMemcpyAsync(d->sperm, perm_vals, sizeof(int) * n, cudaMemcpyDeviceToDevice, h->stream));
  k_gather_source<<<(n + 255) / 256, 256, 0, h->stream>>>(d->sperm, n, d->pos, d->feat, d->FP, d->lab, d->CP, d->geo,
                                                         d->spos, d->sfeat, d->slab, d->sgeo);
  h->launches++;
  // boxes of the groups and supergroups
  const int ng = group_count(n), ns = group_count(ng), ch = box_chunks(d->FP);
  if ((rc = dalloc(h, &d->gbox, (size_t)(2 + 2 * ch) * ng)) || (rc = dalloc(h, &d->sbox, (size_t)(2 + 2 * ch) * ns))) return rc;
  k_boxes<0><<<(ng + 3) / 4, 128, 0, h->stream>>>(d->spos, reinterpret_cast<const float4 *>(d->sfeat), d->FP / 4, n, ch,
                                                  d->gbox, ng);
  k_boxes<1><<<(ns + 3) / 4, 128, 0, h->stream>>>(d->gbox, nullptr, 0, ng, ch, d->sbox, ns);
  h->launches += 2;
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  cudaFree(keys); cudaFree(keys_tmp); cudaFree(perm_vals); cudaFree(perm_tmp);
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
  int rc = 0;
  auto release = [&]() { cudaFree(xyz_d); cudaFree(feat_in); cudaFree(lab_in); cudaFree(geo_in); };
  if ((rc = dalloc(h, &xyz_d, (size_t)n * c->xyz_stride))) { release(); return rc; }
  CVO_CUDA_TRY(h, cudaMemcpyAsync(xyz_d, c->xyz, sizeof(float) * (size_t)n * c->xyz_stride, cudaMemcpyHostToDevice,
                                  h->stream));
  if (d->FP > 0) {
    if ((rc = dalloc(h, &feat_in, (size_t)n * c->F))) { release(); return rc; }
    CVO_CUDA_TRY(h, cudaMemcpyAsync(feat_in, c->features, sizeof(float) * (size_t)n * c->F, cudaMemcpyHostToDevice,
                                    h->stream));
  }
  if (d->CP > 0) {
    if ((rc = dalloc(h, &lab_in, (size_t)n * c->C))) { release(); return rc; }
    CVO_CUDA_TRY(h, cudaMemcpyAsync(lab_in, c->labels, sizeof(float) * (size_t)n * c->C, cudaMemcpyHostToDevice,
                                    h->stream));
  }
  if (d->has_geo) {
    if ((rc = dalloc(h, &geo_in, n))) { release(); return rc; }
    CVO_CUDA_TRY(h, cudaMemcpyAsync(geo_in, c->geom_type, sizeof(float2) * n, cudaMemcpyHostToDevice, h->stream));
  }
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
  cudaFree(d->pos); cudaFree(d->feat); cudaFree(d->lab); cudaFree(d->geo);
  cudaFree(d->sperm); cudaFree(d->spos); cudaFree(d->sfeat); cudaFree(d->slab); cudaFree(d->sgeo);
  cudaFree(d->gbox); cudaFree(d->sbox);
  delete d;
}

}  // namespace cvo_gb
