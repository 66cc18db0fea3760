// cvo_aniso.cu -- association with a non-isotropic (3x3) geometric kernel.
//
// CvoGPU::compute_association_gpu(source, target, T, non_isotropic_kernel, association)
// (src/cvo/CvoGPU.cu:1936-1950 -> inner_product_non_isotropic_impl, :1873-1934):
// the kernel is inverted once on the host; for every source point a the inverse is
// rotated into a frame built from the point's direction (rotate_kernel_and_inverse,
// :135-160: z = a/|a|, x = (1, 1, -(z0+z1)/z2), y = z cross x, neither x nor y
// normalised, M = U K^-1 U^T with U = [x y z]), and the geometric factor of a pair is
// sigma^2 exp(-(a-b)^T M (a-b) / 2) (mahananobis_distance, :165-183) -- no distance
// threshold and no range-scaled lengthscale.  Colour and semantic factors keep their
// thresholds; the geometric type is off.  Each row keeps its first `cap` pairs in
// ascending target index (fill_in_A_mat_gpu_dense_mat_kernel, :719-830).
//
// There is no distance threshold and an indefinite kernel has no bound by position, so this is an
// index-ordered scan of all targets per source row (a positive-definite kernel would have one:
// the columns of U are orthogonal and no shorter than 1, so that (a-b)^T M (a-b) is at least the
// smallest eigenvalue of K^-1 times |a-b|^2; not used).  A warp takes four rows and tests them
// against 32 targets at a time, one a lane, colour first (few pairs pass it); a row's kept pairs
// are the set bits in order, and the warp stops as soon as its rows hold `cap` pairs.  A thread
// per row left five warps in six of the SMs' slots empty and ran every pair's whole arithmetic in
// some lane.
#include <cmath>
#include <cstring>
#include <vector>
#include "cvo_internal.h"
#include "cvo_device.cuh"

namespace cvo_gb {
namespace {

constexpr int kAnisoWarps = 4, kAnisoRows = 4;      // warps of a block, rows of a warp

struct AnisoParams {
  KParams K;
  float Ki[9];        // inverse kernel, column-major
  float Ri[9], Ti[3]; // target transform
  int n, m, cap, F, C;
};

__global__ void k_aniso_transform(const float4 *pos, int m, AnisoParams A, float4 *ytr) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const float4 y = pos[j];
  ytr[j] = make_float4(xform_row(&A.Ri[0], A.Ti[0], y.x, y.y, y.z), xform_row(&A.Ri[3], A.Ti[1], y.x, y.y, y.z),
                       xform_row(&A.Ri[6], A.Ti[2], y.x, y.y, y.z), 0.f);
}

// M (row-major) = U Ki U^T for source point x, in the oracle's order.
__device__ __forceinline__ void aniso_row_matrix(const float *Ki, float x0, float x1, float x2, float (&M)[9]) {
  const float nrm = __fsqrt_rn(fa(fa(fm(x0, x0), fm(x1, x1)), fm(x2, x2)));
  const float z[3] = {__fdiv_rn(x0, nrm), __fdiv_rn(x1, nrm), __fdiv_rn(x2, nrm)};
  const float t = __fdiv_rn(-1.f, z[2]);
  const float xv[3] = {1.f, 1.f, fm(t, fa(z[0], z[1]))};
  const float yv[3] = {fs(fm(z[1], xv[2]), fm(z[2], xv[1])), fs(fm(z[2], xv[0]), fm(z[0], xv[2])),
                       fs(fm(z[0], xv[1]), fm(z[1], xv[0]))};
  float U[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++) { U[i][0] = xv[i]; U[i][1] = yv[i]; U[i][2] = z[i]; }
  float P[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      P[i][j] = fa(fa(fm(U[i][0], Ki[3 * j + 0]), fm(U[i][1], Ki[3 * j + 1])), fm(U[i][2], Ki[3 * j + 2]));
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) M[3 * i + j] = fa(fa(fm(P[i][0], U[j][0]), fm(P[i][1], U[j][1])), fm(P[i][2], U[j][2]));
}

// Bounds: issue, some 25 instructions per row and 32 targets, and 80 more where a colour passes.
template <int FCH, int LCH>
__global__ void __launch_bounds__(32 * kAnisoWarps) k_assoc_aniso(AnisoParams A, const float4 *xpos, const float *xfeat,
                                                                  const float *xlab, const float4 *ytr, const float *yfeat,
                                                                  const float *ylab, int *ell_j, float *ell_v, int *nnz) {
  constexpr int FP = FCH > 0 ? FCH : 1;
  __shared__ float4 sh_x[kAnisoWarps][kAnisoRows], sh_f[kAnisoWarps][kAnisoRows][FP];
  __shared__ float sh_M[kAnisoWarps][kAnisoRows][9];
  const KParams &K = A.K;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * kAnisoWarps + w) * kAnisoRows;
  if (i0 >= A.n) return;
  if (lane < kAnisoRows) {
    const int i = min(i0 + lane, A.n - 1);
    const float4 x = xpos[i];
    sh_x[w][lane] = x;
#pragma unroll
    for (int q = 0; q < FCH; q++) sh_f[w][lane][q] = reinterpret_cast<const float4 *>(xfeat)[(size_t)i * FCH + q];
    float M[9];
    aniso_row_matrix(A.Ki, x.x, x.y, x.z, M);
#pragma unroll
    for (int k = 0; k < 9; k++) sh_M[w][lane][k] = M[k];
  }
  __syncwarp();
  int cnt[kAnisoRows];
#pragma unroll
  for (int r = 0; r < kAnisoRows; r++) cnt[r] = i0 + r < A.n ? 0 : A.cap;
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f), yf[FP];
#pragma unroll
  for (int q = 0; q < FP; q++) yf[q] = y;
  auto load = [&](int j) {
    if (j >= A.m) return;
    y = __ldg(&ytr[j]);
#pragma unroll
    for (int q = 0; q < FCH; q++) yf[q] = __ldg(reinterpret_cast<const float4 *>(yfeat) + (size_t)j * FCH + q);
  };
  load(lane);
  for (int j0 = 0; j0 < A.m; j0 += 32) {
    const int j = j0 + lane;
    const float4 yc = y;
    float4 fc[FP];
#pragma unroll
    for (int q = 0; q < FP; q++) fc[q] = yf[q];
    load(j + 32);
    bool full = true;
#pragma unroll
    for (int r = 0; r < kAnisoRows; r++) {
      if (cnt[r] >= A.cap) continue;
      full = false;
      bool pass = j < A.m;
      float d2c = 0.f;
      if (K.use_int) {
#pragma unroll
        for (int q = 0; q < FCH; q++) {
          const float4 f = sh_f[w][r][q];
          const float av[4] = {f.x, f.y, f.z, f.w}, bv[4] = {fc[q].x, fc[q].y, fc[q].z, fc[q].w};
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (4 * q + k < A.F) { const float t = fs(av[k], bv[k]); d2c = fa(d2c, fm(t, t)); }
        }
        pass = pass && d2c < K.d2_c_thres;
      }
      if (!__any_sync(0xFFFFFFFFu, pass)) continue;
      float d2s = 0.f;
      if (K.use_sem) {
#pragma unroll
        for (int q = 0; q < LCH; q++) {
          const float4 l = __ldg(reinterpret_cast<const float4 *>(xlab) + (size_t)(i0 + r) * LCH + q);
          const float4 o = pass ? __ldg(reinterpret_cast<const float4 *>(ylab) + (size_t)j * LCH + q) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float av[4] = {l.x, l.y, l.z, l.w}, bv[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (4 * q + k < A.C) { const float t = fs(av[k], bv[k]); d2s = fa(d2s, fm(t, t)); }
        }
        pass = pass && d2s < K.d2_s_thres;
      }
      float d2 = 0.f;
      if (K.use_geo) {
        const float4 x = sh_x[w][r];
        const float *M = sh_M[w][r];
        const float d0 = fs(x.x, yc.x), d1 = fs(x.y, yc.y), dd = fs(x.z, yc.z);
        float v[3];
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] = fa(fa(fm(d0, M[k]), fm(d1, M[3 + k])), fm(dd, M[6 + k]));
        d2 = fa(fa(fm(v[0], d0), fm(v[1], d1)), fm(v[2], dd));
      }
      const float kf = K.use_geo ? fm(K.sigma2, __expf(fm(-d2, 0.5f))) : 1.f;
      const float ckf = K.use_int ? fm(K.c_sigma2, __expf(fm(-d2c, K.inv2c2))) : 1.f;
      const float skf = K.use_sem ? fm(K.s_sigma_sq, __expf(fm(-d2s, __frcp_rn(fm(fm(2.f, K.s_ell), K.s_ell))))) : 1.f;
      float af = fm(fm(fm(ckf, kf), skf), 1.f);
      // sigma^2 exp(-d2 / 2) is the isotropic value with l = 1
      if (pass && fabsf(fs(af, K.sp_thres)) <= kBand * K.sp_thres) af = exact_value(K, 1.f, d2, d2c, d2s, 1.f);
      pass = pass && af > K.sp_thres;
      const unsigned kept = __ballot_sync(0xFFFFFFFFu, pass);
      const int c = cnt[r] + __popc(kept & ((1u << lane) - 1u));
      if (pass && c < A.cap) {
        ell_j[(size_t)(i0 + r) * A.cap + c] = j;
        ell_v[(size_t)(i0 + r) * A.cap + c] = af;
      }
      cnt[r] = min(cnt[r] + __popc(kept), A.cap);
    }
    if (full) break;
  }
#pragma unroll
  for (int r = 0; r < kAnisoRows; r++)
    if (lane == 0 && i0 + r < A.n) nnz[i0 + r] = cnt[r];
}

using AnisoFn = void (*)(AnisoParams, const float4 *, const float *, const float *, const float4 *, const float *,
                         const float *, int *, float *, int *);

AnisoFn pick_aniso(int fch, int lch) {
#define CVO_ANISO(FC, LC) \
  if (fch == FC && lch == LC) return k_assoc_aniso<FC, LC>;
  CVO_ANISO(0, 0) CVO_ANISO(1, 0) CVO_ANISO(2, 0)
  CVO_ANISO(0, 5) CVO_ANISO(1, 5) CVO_ANISO(2, 5)
  CVO_ANISO(0, 9) CVO_ANISO(1, 9) CVO_ANISO(2, 9)
#undef CVO_ANISO
  return nullptr;
}

}  // namespace

// Float 3x3 inverse of a column-major matrix: cofactors of column 0, det = their
// dot product with column 0, every entry times 1/det (the order of Eigen's 3x3 inverse).
void kernel_inverse3(const float K[9], float Ki[9]) {
  auto km = [&](int r, int c) { return K[3 * c + r]; };
  float cof[3][3];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
      const float u = km(i1, j1) * km(i2, j2), v = km(i1, j2) * km(i2, j1);
      cof[i][j] = u - v;
    }
  const float d0 = cof[0][0] * km(0, 0), d1 = cof[1][0] * km(1, 0), d2 = cof[2][0] * km(2, 0);
  const float det = (d0 + d1) + d2;
  const float invdet = 1.f / det;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) Ki[3 * j + i] = cof[j][i] * invdet;
}

int run_association_aniso(Handle *h, DevCloud *src, DevCloud *tgt, const float T[16], const float kernel[9],
                          int cap, std::vector<int> *rowptr, std::vector<int> *col, std::vector<float> *val) {
  NvtxRange nvtx_range("aniso_association");
  const int n = src->n, m = tgt->n;
  if (src->F != tgt->F || src->C != tgt->C) return CVO_ERR_INVALID_ARG;
  rowptr->assign((size_t)n + 1, 0);
  col->clear();
  val->clear();
  if (n == 0 || m == 0 || cap <= 0) return CVO_OK;
  AnisoParams A;
  memset(&A, 0, sizeof(A));
  A.K = make_kparams(h->params);
  kernel_inverse3(kernel, A.Ki);
  // target moved by T^-1 (update_tf, src/cvo/CvoGPU.cu:98-130): Ri = R^T, Ti = -R^T t
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) A.Ri[3 * r + c] = T[4 * r + c];   // (R^T)(r, c) = R(c, r) = T[4 r + c]
  for (int r = 0; r < 3; r++) {
    const float a = A.Ri[3 * r] * T[12], b = A.Ri[3 * r + 1] * T[13], c = A.Ri[3 * r + 2] * T[14];
    A.Ti[r] = -((a + b) + c);
  }
  A.n = n; A.m = m; A.cap = cap; A.F = src->F; A.C = src->C;
  const int fch = A.K.use_int ? (src->F + 3) / 4 : 0;
  const int lch = A.K.use_sem ? label_chunks(src->C) : 0;
  AnisoFn fn = pick_aniso(fch, lch);
  if (!fn) return CVO_ERR_UNSUPPORTED;
  float4 *ytr = nullptr;
  int *ej = nullptr, *nz = nullptr;
  float *ev = nullptr;
  auto release = [&]() { cudaFree(ytr); cudaFree(ej); cudaFree(ev); cudaFree(nz); };
  if (cudaMalloc((void **)&ytr, sizeof(float4) * m) != cudaSuccess ||
      cudaMalloc((void **)&ej, sizeof(int) * (size_t)n * cap) != cudaSuccess ||
      cudaMalloc((void **)&ev, sizeof(float) * (size_t)n * cap) != cudaSuccess ||
      cudaMalloc((void **)&nz, sizeof(int) * n) != cudaSuccess) {
    cudaGetLastError();
    release();
    return CVO_ERR_OUT_OF_MEMORY;
  }
  k_aniso_transform<<<(m + 255) / 256, 256, 0, h->stream>>>(tgt->pos, m, A, ytr);
  constexpr int rows = kAnisoRows * kAnisoWarps;
  fn<<<(n + rows - 1) / rows, 32 * kAnisoWarps, 0, h->stream>>>(A, src->pos, src->feat, src->lab, ytr, tgt->feat,
                                                                      tgt->lab, ej, ev, nz);
  h->launches += 2;
  const int rc = csr_to_host(h, n, nz, nullptr, cap, ej, ev, rowptr, col, val);
  release();
  return rc;
}

}  // namespace cvo_gb
