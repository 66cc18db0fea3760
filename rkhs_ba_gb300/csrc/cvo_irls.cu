// cvo_irls.cu -- multi-frame RKHS-BA window (CvoBatchIRLS::solve, src/cvo/IRLS.cpp:148-367).
//
// Per outer iteration: every frame is moved to world coordinates with its float
// pose (CvoFrameGPU::transform_pointcloud, src/cvo/CvoFrameGPU.cu:130-149); every
// edge gets its sparse kernel matrix between the two world-frame clouds in one
// batched association launch (BinaryStateGPU::update_inner_product,
// src/cvo/IRLS_State_GPU.cu:144-336); the poses are then refined by a
// Levenberg-Marquardt solve over the residuals r = a |T1 p1 - T2 p2|^2 with the
// reference's analytic Jacobian (IRLS_Cost_CPU.hpp:260-371) composed with the SE(3)
// local parameterisation (local_parameterization_se3.hpp:13-100).  The reference
// hands that solve to Ceres (LM, SPARSE_NORMAL_CHOLESKY, IRLS.cpp:273-290); here the
// normal equations are accumulated on the GPU (the kernel-matrix entries are read once per
// outer iteration and reduced to moments per row) and the 6F x 6F system is solved on the host, with the LM iteration
// stated in oracle/cvo_oracle.c (lm_solve).
#include <cmath>
#include <cstring>
#include <algorithm>
#include <chrono>
#include <vector>
#include "cvo_internal.h"
#include "cvo_device.cuh"
#include "cvo_lie.cuh"

namespace cvo_gb {
namespace {

constexpr int kIrlsWarps = 4;
constexpr int kIrlsRows = 32 * kIrlsWarps;   // rows per block: one tile of 32 per warp
constexpr int kNormTerms = 28;   // S (6), S K^T (9), K S K^T (6), q (3), K q (3), cost
constexpr int kMoments = 40;     // floats a row's entries are reduced to, see k_irls_moments

// frame points (tile order, local) -> world with the float pose, canonical order
__global__ void k_world(const float4 *local, int n, const float *pose, float4 *world) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  float4 p = local[s];
  // rows of the 3x4 pose: [r00 r01 r02 t0 | r10 r11 r12 t1 | r20 r21 r22 t2]
  float R[9] = {pose[0], pose[1], pose[2], pose[4], pose[5], pose[6], pose[8], pose[9], pose[10]};
  float o0 = xform_row(&R[0], pose[3], p.x, p.y, p.z);
  float o1 = xform_row(&R[3], pose[7], p.x, p.y, p.z);
  float o2 = xform_row(&R[6], pose[11], p.x, p.y, p.z);
  world[s] = make_float4(o0, o1, o2, range_norm(o0, o1, o2));
}

struct IrlsEdge {
  const int *A_j;     // ELL, row-major with pitch ld
  const float *A_v;
  const int *nnz_row;
  int ld;
  const float4 *p1;   // frame-1 local points, tile order (rows of A)
  const float4 *p2;   // frame-2 local points, original order (columns of A)
  int n, lim;         // rows, entries used per row
  int f1, f2;
  int blk0;           // first block of this edge
  float *mom;         // kMoments planes of n floats
};

// The edge of a block.
__device__ __forceinline__ IrlsEdge edge_of(const IrlsEdge *E, int ne, int blk) {
  int lo = 0, hi = ne - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (E[mid].blk0 <= blk) lo = mid; else hi = mid - 1;
  }
  return E[lo];
}

// The row's point in the target frame, p' = R2^T (T1 p1 - t2), in double.
__device__ __forceinline__ void row_point(const double *poses, const IrlsEdge &ed, int s, double (&pd)[3]) {
  const double *T1 = poses + 12 * ed.f1, *T2 = poses + 12 * ed.f2;
  const float4 a1 = __ldg(&ed.p1[s]);
  const double p1[3] = {a1.x, a1.y, a1.z};
  double q1[3];
  for (int r = 0; r < 3; r++) q1[r] = T1[4 * r] * p1[0] + T1[4 * r + 1] * p1[1] + T1[4 * r + 2] * p1[2] + T1[4 * r + 3];
  for (int r = 0; r < 3; r++)
    pd[r] = T2[r] * (q1[0] - T2[3]) + T2[4 + r] * (q1[1] - T2[7]) + T2[8 + r] * (q1[2] - T2[11]);
}

// A row's share of the normal equations is a polynomial in its point p': with c = p' when
// the kernel matrix was made, e = p2 - c per entry and x = p' - c, an entry's difference is
// d = x - e and, with r = a |d|^2,
//   sum d d^T   = n x x^T - x N1^T - N1 x^T + N2
//   sum r d     = |x|^2 x A0 - |x|^2 A1 - 2 (x.A1) x + 2 A2 x + tr(A2) x - A3
//   sum r^2     = |x|^4 M0 + 4 x^T M2 x + M4 - 4 |x|^2 x.M1 + 2 |x|^2 tr(M2) - 4 x.M3
// with N, A, M the moments of e weighted by 1, a and a^2 (N2 = sum e e^T, A3 = sum a |e|^2 e,
// ...).  So the entries are read once per outer iteration (37 sums) and every evaluation of
// the solve, some forty per outer iteration, reads 40 floats a row.  e and x are small
// against the coordinates (c is the rounded double p', e is exact to its own rounding), so
// the sums keep the accuracy of summing each entry's r anew.
// Planes: c (3), n, N1 (3), N2 (6), A0, A1 (3), A2 (6), A3 (3), M0, M1 (3), M2 (6), M3 (3), M4.
// Eight lanes share a row and a warp runs four rows at a time: the rows' entries differ
// widely (0 to cap), and one row per warp left too few gathers in flight.
// Bounds: L2 latency of entry -> point.
__global__ void __launch_bounds__(32 * kIrlsWarps) k_irls_moments(const IrlsEdge *E, int ne, const double *poses) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane & 7;
  const IrlsEdge ed = edge_of(E, ne, blockIdx.x);
  const int t0 = ((int)blockIdx.x - ed.blk0) * kIrlsRows + 32 * w;
  const int s = t0 + lane;
  const int z = s < ed.n ? min(__ldg(&ed.nnz_row[s]), ed.lim) : 0;
  if (s < ed.n) ed.mom[3 * (size_t)ed.n + s] = (float)z;
  if (!__any_sync(FULLMASK, z > 0)) return;
  float c[3] = {0.f, 0.f, 0.f};
  if (z > 0) {
    double pd[3];
    row_point(poses, ed, s, pd);
    for (int r = 0; r < 3; r++) {
      c[r] = (float)pd[r];
      ed.mom[r * (size_t)ed.n + s] = c[r];
    }
  }
  for (int r0 = 0; r0 < 32; r0 += 4) {
    const int r = r0 + (lane >> 3);
    const int zr = __shfl_sync(FULLMASK, z, r);
    if (!__any_sync(FULLMASK, zr > 0)) continue;
    const float c0 = __shfl_sync(FULLMASK, c[0], r), c1 = __shfl_sync(FULLMASK, c[1], r), c2 = __shfl_sync(FULLMASK, c[2], r);
    const int *__restrict__ Aj = ed.A_j + (size_t)(t0 + r) * ed.ld;
    const float *__restrict__ Av = ed.A_v + (size_t)(t0 + r) * ed.ld;
    float v[36];      // all but n
#pragma unroll
    for (int k = 0; k < 36; k++) v[k] = 0.f;
#pragma unroll 4
    for (int i = sub; i < zr; i += 8) {
      const float a = __ldg(Av + i);
      const float4 b2 = __ldg(&ed.p2[__ldg(Aj + i)]);
      const float e[3] = {b2.x - c0, b2.y - c1, b2.z - c2};
      const float e2 = e[0] * e[0] + e[1] * e[1] + e[2] * e[2];
      const float ae[3] = {a * e[0], a * e[1], a * e[2]};
      const float be[3] = {a * ae[0], a * ae[1], a * ae[2]}, be2 = a * a * e2;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        v[k] += e[k];
        v[10 + k] += ae[k];
        v[19 + k] = fmaf(e2, ae[k], v[19 + k]);
        v[23 + k] += be[k];
        v[32 + k] = fmaf(e2, be[k], v[32 + k]);
      }
      v[9] += a;
      v[22] = fmaf(a, a, v[22]);
      v[35] = fmaf(be2, e2, v[35]);
      int k = 0;
#pragma unroll
      for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = p; q < 3; q++, k++) {
          v[3 + k] = fmaf(e[p], e[q], v[3 + k]);
          v[13 + k] = fmaf(ae[p], e[q], v[13 + k]);
          v[26 + k] = fmaf(be[p], e[q], v[26 + k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 36; k++) {
      v[k] += __shfl_xor_sync(FULLMASK, v[k], 4);
      v[k] += __shfl_xor_sync(FULLMASK, v[k], 2);
      v[k] += __shfl_xor_sync(FULLMASK, v[k], 1);
    }
    if (sub == 0 && zr > 0) {
#pragma unroll
      for (int k = 0; k < 36; k++) ed.mom[(4 + k) * (size_t)ed.n + t0 + r] = v[k];
    }
  }
}

// Sums of the normal equations of one edge, per block.  With p' = R2^T (T1 p1 - t2) (the
// row's point in the target frame), d = p' - p2, r = a |d|^2, K = [p']x and t' = R2^T (t1 - t2),
// the Jacobian row of the residual is linear in d,
//   J = [R12 d, p1 x R12 d, -d, -p2 x d] = B [d, p' x d],   R12 = R1^T R2,
//   B = [R12 0; -R12 [t']x R12; -I 0; 0 -I]   (p2 x d = p' x d, p1 x R12 d = R12 ((p' - t') x d)),
// and B is the edge's, p' the row's.  So a row adds G = [I; K] S [I; K]^T and [q; K q] with
// S = sum d d^T, q = sum r d (27 terms), and the host forms J^T J = B G B^T and J^T r once
// per edge, in FP64.  S, q and the cost come from the row's moments.  FP32 per row, FP64
// over rows.
// Bounds: reading 160 bytes a row, and the FP64 sums.  Summing 91 FP32 terms per entry in
// one thread per row took 468 us an evaluation with the Jacobian and 250 without for 28
// edges of 20k-60k rows.
template <bool WANT_J>
__global__ void __launch_bounds__(32 * kIrlsWarps) k_irls_accum(const IrlsEdge *E, int ne, const double *poses,
                                                                double *partial) {
  constexpr int NT = WANT_J ? kNormTerms : 1;
  __shared__ double red[NT][32 * kIrlsWarps + 1];
  const IrlsEdge ed = edge_of(E, ne, blockIdx.x);
  const int s = ((int)blockIdx.x - ed.blk0) * kIrlsRows + threadIdx.x;
  const size_t n = ed.n;
  const float *__restrict__ m = ed.mom + s;
  const float z = s < ed.n ? __ldg(m + 3 * n) : 0.f;
  if (!__syncthreads_or(z > 0.f)) {
    for (int k = threadIdx.x; k < NT; k += blockDim.x) partial[(size_t)blockIdx.x * kNormTerms + k] = 0.0;
    return;
  }
  double acc[NT];
#pragma unroll
  for (int k = 0; k < NT; k++) acc[k] = 0.0;
  if (z > 0.f) {
    double pd[3];
    row_point(poses, ed, s, pd);
    auto M = [&](int k) { return __ldg(m + k * n); };
    const float x[3] = {(float)(pd[0] - (double)M(0)), (float)(pd[1] - (double)M(1)), (float)(pd[2] - (double)M(2))};
    const float x2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
    const float B[6] = {M(30), M(31), M(32), M(33), M(34), M(35)};
    const float Bx[3] = {B[0] * x[0] + B[1] * x[1] + B[2] * x[2], B[1] * x[0] + B[3] * x[1] + B[4] * x[2],
                         B[2] * x[0] + B[4] * x[1] + B[5] * x[2]};
    const float c2 = 4.f * (x[0] * Bx[0] + x[1] * Bx[1] + x[2] * Bx[2]) + 2.f * x2 * (B[0] + B[3] + B[5]);
    const float c1 = x[0] * M(36) + x[1] * M(37) + x[2] * M(38), c3 = x[0] * M(27) + x[1] * M(28) + x[2] * M(29);
    const float cost = 0.5f * (M(39) - 4.f * c1 + c2 - 4.f * x2 * c3 + x2 * x2 * M(26));
    if (WANT_J) {
      const float n1[3] = {M(4), M(5), M(6)}, A[6] = {M(17), M(18), M(19), M(20), M(21), M(22)}, a1[3] = {M(14), M(15), M(16)};
      float S[3][3];
      S[0][0] = M(7) - 2.f * x[0] * n1[0] + z * x[0] * x[0];
      S[0][1] = S[1][0] = M(8) - x[0] * n1[1] - x[1] * n1[0] + z * x[0] * x[1];
      S[0][2] = S[2][0] = M(9) - x[0] * n1[2] - x[2] * n1[0] + z * x[0] * x[2];
      S[1][1] = M(10) - 2.f * x[1] * n1[1] + z * x[1] * x[1];
      S[1][2] = S[2][1] = M(11) - x[1] * n1[2] - x[2] * n1[1] + z * x[1] * x[2];
      S[2][2] = M(12) - 2.f * x[2] * n1[2] + z * x[2] * x[2];
      const float xa = x[0] * a1[0] + x[1] * a1[1] + x[2] * a1[2], tr = A[0] + A[3] + A[5], a0 = M(13);
      const float Ax[3] = {A[0] * x[0] + A[1] * x[1] + A[2] * x[2], A[1] * x[0] + A[3] * x[1] + A[4] * x[2],
                           A[2] * x[0] + A[4] * x[1] + A[5] * x[2]};
      float q[3];
#pragma unroll
      for (int k = 0; k < 3; k++) q[k] = (2.f * Ax[k] + tr * x[k] - M(23 + k)) + (x2 * (x[k] * a0 - a1[k]) - 2.f * xa * x[k]);
      const float px = (float)pd[0], py = (float)pd[1], pz = (float)pd[2];
      // K v = p' x v; W = S K^T has rows p' x (row of S), X = K S K^T columns p' x (column of W)
      float W[3][3], X[3][3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        W[i][0] = py * S[i][2] - pz * S[i][1];
        W[i][1] = pz * S[i][0] - px * S[i][2];
        W[i][2] = px * S[i][1] - py * S[i][0];
      }
#pragma unroll
      for (int j = 0; j < 3; j++) {
        X[0][j] = py * W[2][j] - pz * W[1][j];
        X[1][j] = pz * W[0][j] - px * W[2][j];
        X[2][j] = px * W[1][j] - py * W[0][j];
      }
      const float t[kNormTerms] = {S[0][0], S[0][1], S[0][2], S[1][1], S[1][2], S[2][2],
                                   W[0][0], W[0][1], W[0][2], W[1][0], W[1][1], W[1][2], W[2][0], W[2][1], W[2][2],
                                   X[0][0], X[0][1], X[0][2], X[1][1], X[1][2], X[2][2],
                                   q[0], q[1], q[2], py * q[2] - pz * q[1], pz * q[0] - px * q[2], px * q[1] - py * q[0], cost};
#pragma unroll
      for (int k = 0; k < NT; k++) acc[k] = (double)t[k];
    } else {
      acc[0] = (double)cost;
    }
  }
#pragma unroll
  for (int k = 0; k < NT; k++) red[k][threadIdx.x] = acc[k];
  __syncthreads();
  // four threads per term, 32 rows each
  if (threadIdx.x < 4 * NT) {
    double t = 0.0;
    const int k = threadIdx.x >> 2, q = threadIdx.x & 3;
#pragma unroll 8
    for (int i = 0; i < 32; i++) t += red[k][32 * q + i];
    red[k][32 * q] = t;
  }
  __syncthreads();
  if (threadIdx.x < NT)
    partial[(size_t)blockIdx.x * kNormTerms + threadIdx.x] =
        (red[threadIdx.x][0] + red[threadIdx.x][32]) + (red[threadIdx.x][64] + red[threadIdx.x][96]);
}

// per edge: sum of its blocks' partials, eight threads per term in a fixed order
__global__ void __launch_bounds__(256) k_irls_sum(const IrlsEdge *E, int ne, int total_blocks, int nt, const double *partial,
                                                  double *out) {
  __shared__ double sh[8][32];
  const int e = blockIdx.x;
  if (e >= ne) return;
  const int b0 = E[e].blk0, b1 = (e + 1 < ne) ? E[e + 1].blk0 : total_blocks;
  const int k = threadIdx.x & 31, g = threadIdx.x >> 5;
  double t = 0.0;
  if (k < nt)
#pragma unroll 4
    for (int b = b0 + g; b < b1; b += 8) t += partial[(size_t)b * kNormTerms + k];
  sh[g][k] = t;
  __syncthreads();
  if (g == 0 && k < nt) {
    for (int q = 1; q < 8; q++) t += sh[q][k];
    out[(size_t)e * kNormTerms + k] = t;
  }
}

// ------------------------------------------------------------- host LM
void se3_exp(const double d[6], double X[12]) {
  // Exp_SE3(v, is_wu = false) (src/cvo/LieGroup.cpp:169-192): u = v.head(3), w = v.tail(3)
  const double *u = d, *w = d + 3;
  double th = std::sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
  double A[9] = {0, -w[2], w[1], w[2], 0, -w[0], -w[1], w[0], 0}, A2[9], R[9], J[9];
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) A2[3 * r + c] = A[3 * r] * A[c] + A[3 * r + 1] * A[3 + c] + A[3 * r + 2] * A[6 + c];
  if (th < (double)1e-6f) {
    for (int t = 0; t < 9; t++) R[t] = J[t] = (t % 4 == 0) ? 1.0 : 0.0;
  } else {
    double s1 = std::sin(th) / th, c1 = (1.0 - std::cos(th)) / (th * th), c2 = (th - std::sin(th)) / (th * th * th);
    for (int t = 0; t < 9; t++) {
      double I = (t % 4 == 0) ? 1.0 : 0.0;
      R[t] = I + s1 * A[t] + c1 * A2[t];
      J[t] = I + c1 * A[t] + c2 * A2[t];
    }
  }
  for (int r = 0; r < 3; r++) {
    for (int c = 0; c < 3; c++) X[4 * r + c] = R[3 * r + c];
    X[4 * r + 3] = J[3 * r] * u[0] + J[3 * r + 1] * u[1] + J[3 * r + 2] * u[2];
  }
}

void compose(const double A[12], const double B[12], double out[12]) {
  double o[12];
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 4; c++) {
      double s = A[4 * r] * B[c] + A[4 * r + 1] * B[4 + c] + A[4 * r + 2] * B[8 + c];
      if (c == 3) s += A[4 * r + 3];
      o[4 * r + c] = s;
    }
  memcpy(out, o, sizeof(o));
}

double pose_change(const double A[12], const double B[12]) {
  double Ai[12], M[12];
  for (int r = 0; r < 3; r++) {
    for (int c = 0; c < 3; c++) Ai[4 * r + c] = A[4 * c + r];
    Ai[4 * r + 3] = -(A[r] * A[3] + A[4 + r] * A[7] + A[8 + r] * A[11]);
  }
  compose(Ai, B, M);
  double R[9] = {M[0], M[1], M[2], M[4], M[5], M[6], M[8], M[9], M[10]}, t[3] = {M[3], M[7], M[11]};
  return dist_se3(R, t);
}

bool chol_solve(int n, std::vector<double> &A, std::vector<double> &b) {
  for (int j = 0; j < n; j++) {
    double s = A[(size_t)j * n + j];
    for (int k = 0; k < j; k++) s -= A[(size_t)j * n + k] * A[(size_t)j * n + k];
    if (!(s > 0.0)) return false;
    double d = std::sqrt(s);
    A[(size_t)j * n + j] = d;
    for (int i = j + 1; i < n; i++) {
      double t = A[(size_t)i * n + j];
      for (int k = 0; k < j; k++) t -= A[(size_t)i * n + k] * A[(size_t)j * n + k];
      A[(size_t)i * n + j] = t / d;
    }
  }
  for (int i = 0; i < n; i++) {
    double t = b[i];
    for (int k = 0; k < i; k++) t -= A[(size_t)i * n + k] * b[k];
    b[i] = t / A[(size_t)i * n + i];
  }
  for (int i = n - 1; i >= 0; i--) {
    double t = b[i];
    for (int k = i + 1; k < n; k++) t -= A[(size_t)k * n + i] * b[k];
    b[i] = t / A[(size_t)i * n + i];
  }
  return true;
}

// Normal equations of the window's residuals at given poses.  One evaluation is the
// upload of the poses, the accumulation over every kernel-matrix entry of every edge, the
// per-edge sums and their read-back; it runs as a CUDA graph (one per kind: with or
// without H and g) that is captured once and replayed by every evaluation of the LM
// solves until the edges' layout changes.  The poses and sums travel through pinned
// buffers, whose addresses the graph's copy nodes hold.
struct Normal {
  Handle *h;
  int nf;
  std::vector<IrlsEdge> edges;    // edges with residuals
  IrlsEdge *edges_d = nullptr;
  double *poses_d = nullptr;
  double *partial_d = nullptr;
  double *out_d = nullptr;
  float *mom_d = nullptr;         // moments of every edge's rows
  size_t mom_cap = 0;
  double *poses_pin = nullptr;    // 12 nf
  double *out_pin = nullptr;      // kNormTerms per edge
  int out_pin_edges = 0;
  int total_blocks = 0;
  cudaGraphExec_t exec[2] = {nullptr, nullptr};
  std::vector<unsigned char> key[2];

  Normal() = default;
  Normal(const Normal &) = delete;
  Normal &operator=(const Normal &) = delete;
  ~Normal() {
    for (auto &e : exec)
      if (e) cudaGraphExecDestroy(e);
    cudaFree(partial_d);
    cudaFree(out_d);
    cudaFree(mom_d);
    cudaFree(edges_d);
    cudaFree(poses_d);
    cudaFreeHost(poses_pin);
    cudaFreeHost(out_pin);
  }

  int record(bool want) {
    const int ne = (int)edges.size();
    const int w = want ? 1 : 0;
    std::vector<unsigned char> k;
    auto add = [&](const void *p, size_t n) {
      const unsigned char *c = static_cast<const unsigned char *>(p);
      k.insert(k.end(), c, c + n);
    };
    const void *ptrs[6] = {edges_d, poses_d, partial_d, out_d, poses_pin, out_pin};
    add(ptrs, sizeof(ptrs));
    add(&ne, sizeof(ne));
    add(&total_blocks, sizeof(total_blocks));
    add(&nf, sizeof(nf));
    add(&h->stream, sizeof(h->stream));
    if (exec[w] && key[w] == k) return 0;
    if (exec[w]) cudaGraphExecDestroy(exec[w]);
    exec[w] = nullptr;
    CVO_CUDA_TRY(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t e1 = cudaMemcpyAsync(poses_d, poses_pin, sizeof(double) * 12 * nf, cudaMemcpyHostToDevice, h->stream);
    if (want) k_irls_accum<true><<<total_blocks, 32 * kIrlsWarps, 0, h->stream>>>(edges_d, ne, poses_d, partial_d);
    else k_irls_accum<false><<<total_blocks, 32 * kIrlsWarps, 0, h->stream>>>(edges_d, ne, poses_d, partial_d);
    k_irls_sum<<<ne, 256, 0, h->stream>>>(edges_d, ne, total_blocks, want ? kNormTerms : 1, partial_d, out_d);
    cudaError_t e2 = cudaMemcpyAsync(out_pin, out_d, sizeof(double) * ne * kNormTerms, cudaMemcpyDeviceToHost,
                                     h->stream);
    cudaGraph_t g = nullptr;
    cudaError_t e3 = cudaStreamEndCapture(h->stream, &g);
    cudaError_t e4 = cudaSuccess;
    if (e1 == cudaSuccess && e2 == cudaSuccess && e3 == cudaSuccess) e4 = cudaGraphInstantiate(&exec[w], g, 0);
    if (g) cudaGraphDestroy(g);
    for (cudaError_t e : {e1, e2, e3, e4})
      if (e != cudaSuccess) {
        exec[w] = nullptr;
        return set_cuda_error(h, e, "normal-equation graph capture");
      }
    key[w] = k;
    return 0;
  }

  // the rows' moments at the poses of the kernel matrices
  int moments(const double *poses) {
    if (edges.empty()) return 0;
    memcpy(poses_pin, poses, sizeof(double) * 12 * nf);
    CVO_CUDA_TRY(h, cudaMemcpyAsync(poses_d, poses_pin, sizeof(double) * 12 * nf, cudaMemcpyHostToDevice, h->stream));
    k_irls_moments<<<total_blocks, 32 * kIrlsWarps, 0, h->stream>>>(edges_d, (int)edges.size(), poses_d);
    h->launches++;
    CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));   // poses_pin is rewritten by the first evaluation
    return 0;
  }

  // J^T J = B G B^T and J^T r = B [q; K q] of one edge (see k_irls_accum) into H and g
  static void add_edge(const double *T1, const double *T2, const double *o, int o1, int o2, int D, std::vector<double> *H,
                       std::vector<double> *g) {
    double R12[3][3], tp[3], B[12][6] = {}, G[6][6];
    for (int r = 0; r < 3; r++) {
      for (int c = 0; c < 3; c++) R12[r][c] = T1[r] * T2[c] + T1[4 + r] * T2[4 + c] + T1[8 + r] * T2[8 + c];
      tp[r] = T2[r] * (T1[3] - T2[3]) + T2[4 + r] * (T1[7] - T2[7]) + T2[8 + r] * (T1[11] - T2[11]);
    }
    for (int r = 0; r < 3; r++) {
      // row r of R12 [t']x is R12's row x t'
      const double cr[3] = {R12[r][1] * tp[2] - R12[r][2] * tp[1], R12[r][2] * tp[0] - R12[r][0] * tp[2],
                            R12[r][0] * tp[1] - R12[r][1] * tp[0]};
      for (int c = 0; c < 3; c++) {
        B[r][c] = B[3 + r][3 + c] = R12[r][c];
        B[3 + r][c] = -cr[c];
      }
      B[6 + r][r] = B[9 + r][3 + r] = -1.0;
    }
    const int tri[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) {
        G[i][j] = o[tri[i][j]];
        G[i][3 + j] = G[3 + j][i] = o[6 + 3 * i + j];
        G[3 + i][3 + j] = o[15 + tri[i][j]];
      }
    double BG[12][6];
    for (int p = 0; p < 12; p++)
      for (int j = 0; j < 6; j++) {
        BG[p][j] = 0.0;
        for (int k = 0; k < 6; k++) BG[p][j] += B[p][k] * G[k][j];
      }
    for (int p = 0; p < 12; p++) {
      const int ip = (p < 6 ? o1 : o2) + p % 6;
      for (int q = p; q < 12; q++) {
        const int iq = (q < 6 ? o1 : o2) + q % 6;
        double v = 0.0;
        for (int k = 0; k < 6; k++) v += BG[p][k] * B[q][k];
        (*H)[(size_t)ip * D + iq] += v;
        if (ip != iq || p != q) (*H)[(size_t)iq * D + ip] += v;
      }
      double v = 0.0;
      for (int k = 0; k < 6; k++) v += B[p][k] * o[21 + k];
      (*g)[ip] += v;
    }
  }

  // cost (and, if want, H and g over all 6 nf parameters) at `poses`
  int eval(const double *poses, bool want, std::vector<double> *H, std::vector<double> *g, double *cost) {
    const int ne = (int)edges.size();
    *cost = 0.0;
    if (want) {
      H->assign((size_t)36 * nf * nf, 0.0);
      g->assign((size_t)6 * nf, 0.0);
    }
    if (ne == 0) return 0;
    if (int rc = record(want)) return rc;
    memcpy(poses_pin, poses, sizeof(double) * 12 * nf);
    CVO_CUDA_TRY(h, cudaGraphLaunch(exec[want ? 1 : 0], h->stream));
    h->launches += 2;
    CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    const double *out_h = out_pin;
    const int D = 6 * nf;
    for (int e = 0; e < ne; e++) {
      const double *o = &out_h[(size_t)e * kNormTerms];
      if (!want) { *cost += o[0]; continue; }
      *cost += o[27];
      add_edge(poses + 12 * edges[e].f1, poses + 12 * edges[e].f2, o, 6 * edges[e].f1, 6 * edges[e].f2, D, H, g);
    }
    return 0;
  }
};

// One Levenberg-Marquardt solve (the iteration stated in oracle/cvo_oracle.c, lm_solve).
int lm_solve(Normal &N, int nf, double *poses, const uint8_t *hold, int max_iter, int *successes) {
  const int D = 6 * nf;
  std::vector<int> idx(D);
  int nfree = 0;
  for (int f = 0; f < nf; f++)
    for (int k = 0; k < 6; k++) idx[6 * f + k] = hold[f] ? -1 : nfree++;
  std::vector<double> H, g, Hf((size_t)std::max(nfree, 1) * std::max(nfree, 1)), gf(std::max(nfree, 1)), A, b,
      cand(12 * (size_t)nf);
  double radius = 1e4, nu = 2.0, cost = 0.0;
  int rc = N.eval(poses, true, &H, &g, &cost);
  if (rc) return rc;
  for (int it = 0; it < max_iter && nfree > 0; it++) {
    for (int i = 0; i < D; i++) {
      if (idx[i] < 0) continue;
      gf[idx[i]] = g[i];
      for (int j = 0; j < D; j++)
        if (idx[j] >= 0) Hf[(size_t)idx[i] * nfree + idx[j]] = H[(size_t)i * D + j];
    }
    double gmax = 0.0;
    for (int i = 0; i < nfree; i++) gmax = std::max(gmax, std::fabs(gf[i]));
    if (gmax <= 1e-5) break;
    A = Hf;
    b.assign(nfree, 0.0);
    for (int i = 0; i < nfree; i++) {
      double dg = Hf[(size_t)i * nfree + i];
      dg = dg < 1e-6 ? 1e-6 : (dg > 1e32 ? 1e32 : dg);
      A[(size_t)i * nfree + i] += dg / radius;
      b[i] = -gf[i];
    }
    if (!chol_solve(nfree, A, b)) { radius /= nu; nu *= 2.0; continue; }
    double dn = 0.0, xn = 0.0;
    for (int i = 0; i < nfree; i++) dn += b[i] * b[i];
    for (int t = 0; t < 12 * nf; t++) xn += poses[t] * poses[t];
    if (std::sqrt(dn) <= 1e-5 * (std::sqrt(xn) + 1e-5)) break;
    double model = 0.0;
    for (int i = 0; i < nfree; i++) {
      double hd = 0.0;
      for (int j = 0; j < nfree; j++) hd += Hf[(size_t)i * nfree + j] * b[j];
      model += gf[i] * b[i] + 0.5 * b[i] * hd;
    }
    model = -model;
    memcpy(cand.data(), poses, sizeof(double) * 12 * nf);
    for (int f = 0; f < nf; f++) {
      if (hold[f]) continue;
      double d6[6], X[12];
      for (int k = 0; k < 6; k++) d6[k] = b[idx[6 * f + k]];
      se3_exp(d6, X);
      compose(poses + 12 * f, X, &cand[12 * f]);
    }
    double cnew = 0.0;
    if ((rc = N.eval(cand.data(), false, nullptr, nullptr, &cnew))) return rc;
    double rho = model > 0.0 ? (cost - cnew) / model : -1.0;
    if (rho > 1e-3) {
      memcpy(poses, cand.data(), sizeof(double) * 12 * nf);
      (*successes)++;
      double rel = std::fabs(cost - cnew);
      double fac = 1.0 - std::pow(2.0 * rho - 1.0, 3.0);
      radius = radius / (fac > 1.0 / 3.0 ? fac : 1.0 / 3.0);
      nu = 2.0;
      bool stop = rel <= 1e-5 * cost;
      cost = cnew;
      if (stop) break;
      if ((rc = N.eval(poses, true, &H, &g, &cost))) return rc;
    } else {
      radius /= nu;
      nu *= 2.0;
    }
  }
  return 0;
}

}  // namespace

int run_align_multi(Handle *h, int nf, DevCloud *const *clouds, double *poses, const uint8_t *hold, int ne,
                    const int *edges, double *secs, int *iters) {
  NvtxRange nvtx_range("align_multi");
  auto t0 = std::chrono::steady_clock::now();
  const cvo_params &p = h->params;
  if (p.multiframe_is_optimizing_ell) return CVO_ERR_UNSUPPORTED;
  for (int f = 0; f < nf; f++)
    if (clouds[f]->F != clouds[0]->F || clouds[f]->C != clouds[0]->C) return CVO_ERR_INVALID_ARG;
  if (ne == 0) {   // no edge has pairs: the first outer iteration stops (counter == 0)
    if (iters) *iters = 0;
    if (secs) *secs = 0.0;
    return CVO_OK;
  }
  // world-frame copies of every frame (tile order) and the frames' float poses
  std::vector<float4 *> world(nf, nullptr);
  float *pose_d = nullptr;
  int rc = 0;
  auto cleanup = [&]() {
    for (auto *w : world) cudaFree(w);
    cudaFree(pose_d);
  };
  for (int f = 0; f < nf; f++) {
    if (cudaMalloc((void **)&world[f], sizeof(float4) * std::max(clouds[f]->n, 1)) != cudaSuccess) {
      cleanup();
      return CVO_ERR_OUT_OF_MEMORY;
    }
  }
  if (cudaMalloc((void **)&pose_d, sizeof(float) * 12 * nf) != cudaSuccess) { cleanup(); return CVO_ERR_OUT_OF_MEMORY; }
  Normal N;
  N.h = h;
  N.nf = nf;
  if (cudaMallocHost((void **)&N.poses_pin, sizeof(double) * 12 * nf) != cudaSuccess ||
      cudaMallocHost((void **)&N.out_pin, sizeof(double) * kNormTerms * ne) != cudaSuccess) {
    cudaGetLastError();
    cleanup();
    return CVO_ERR_OUT_OF_MEMORY;
  }
  // the edge association of every outer iteration replays one captured graph while its
  // launch parameters stay the same
  AssocGraph ag;
  // per-edge state (BinaryStateGPU members)
  std::vector<double> ell(ne, (double)p.multiframe_ell_init);
  std::vector<int> nn(ne, p.multiframe_num_neighbors), prev_max(ne, 0), iters_per_ell(ne, 0);
  std::vector<long long> prev_nnz(ne, 0), nz_last(ne, 0);
  const int init_nn = p.multiframe_num_neighbors;
  const double ell_min = p.multiframe_ell_min, ell_max = (double)p.multiframe_ell_init * 1.2;
  std::vector<double> old(12 * (size_t)nf);
  int iter = 0, steps = 0;
  size_t max_blocks = 0;
  for (;;) {
    memcpy(old.data(), poses, sizeof(double) * 12 * nf);
    std::vector<float> fpose(12 * (size_t)nf);
    for (int t = 0; t < 12 * nf; t++) fpose[t] = (float)poses[t];
    if (cudaMemcpyAsync(pose_d, fpose.data(), sizeof(float) * 12 * nf, cudaMemcpyHostToDevice, h->stream) !=
        cudaSuccess) { cleanup(); return CVO_ERR_CUDA; }
    for (int f = 0; f < nf; f++) {
      int n = clouds[f]->n;
      if (n > 0) {
        k_world<<<(n + 255) / 256, 256, 0, h->stream>>>(clouds[f]->spos, n, pose_d + 12 * f, world[f]);
        h->launches++;
      }
    }
    // association of every edge in one batch
    std::vector<DevCloud *> es(ne), et(ne);
    std::vector<const float4 *> ew(ne);
    std::vector<float> epose(12 * (size_t)ne), eell(ne);
    for (int e = 0; e < ne; e++) {
      int f1 = edges[2 * e], f2 = edges[2 * e + 1];
      nz_last[e] = prev_nnz[e];
      if (prev_max[e] > 0) nn[e] = std::min(init_nn, (int)((double)prev_max[e] * 1.1));
      es[e] = clouds[f1];
      et[e] = clouds[f2];
      ew[e] = world[f1];
      for (int t = 0; t < 12; t++) epose[12 * e + t] = fpose[12 * f2 + t];
      eell[e] = (float)ell[e];
    }
    std::vector<EdgeAssoc> EA;
    if ((rc = run_association_edges(h, es, et, ew, epose, eell, nn, init_nn, &EA, nullptr, &ag))) {
      cleanup();
      return rc;
    }
    int counter = 0;
    N.edges.clear();
    int blk = 0;
    for (int e = 0; e < ne; e++) {
      prev_nnz[e] = EA[e].nnz;
      prev_max[e] = EA[e].max_row;
      if (EA[e].nnz > p.multiframe_min_nonzeros) counter++;
      // add_residual_to_problem (IRLS_State_GPU.cpp:17-20): edges with too few pairs add nothing
      if (EA[e].nnz != 0 && EA[e].nnz >= p.multiframe_min_nonzeros) {
        IrlsEdge E;
        E.A_j = EA[e].A_j; E.A_v = EA[e].A_v; E.nnz_row = EA[e].nnz_row;
        E.ld = EA[e].ld;
        E.p1 = clouds[edges[2 * e]]->spos;
        E.p2 = clouds[edges[2 * e + 1]]->pos;
        E.n = EA[e].n;
        E.lim = std::min(p.nearest_neighbors_max, nn[e]);
        E.f1 = edges[2 * e]; E.f2 = edges[2 * e + 1];
        E.blk0 = blk;
        blk += (E.n + kIrlsRows - 1) / kIrlsRows;
        N.edges.push_back(E);
      }
    }
    if (counter == 0) break;
    N.total_blocks = blk;
    if ((size_t)blk > max_blocks || !N.partial_d) {
      cudaFree(N.partial_d); cudaFree(N.out_d); cudaFree(N.edges_d); cudaFree(N.poses_d);
      N.partial_d = N.out_d = N.poses_d = nullptr;
      N.edges_d = nullptr;
      max_blocks = std::max<size_t>(blk, 1) * 2;
      if (cudaMalloc((void **)&N.partial_d, sizeof(double) * kNormTerms * max_blocks) != cudaSuccess ||
          cudaMalloc((void **)&N.out_d, sizeof(double) * kNormTerms * std::max(ne, 1)) != cudaSuccess ||
          cudaMalloc((void **)&N.edges_d, sizeof(IrlsEdge) * std::max(ne, 1)) != cudaSuccess ||
          cudaMalloc((void **)&N.poses_d, sizeof(double) * 12 * nf) != cudaSuccess) {
        cleanup();
        return CVO_ERR_OUT_OF_MEMORY;
      }
    }
    size_t rows = 0;
    for (const IrlsEdge &E : N.edges) rows += E.n;
    if (rows > N.mom_cap) {
      cudaFree(N.mom_d);
      N.mom_d = nullptr;
      N.mom_cap = 0;
      if (cudaMalloc((void **)&N.mom_d, sizeof(float) * kMoments * rows) != cudaSuccess) {
        cudaGetLastError();
        cleanup();
        return CVO_ERR_OUT_OF_MEMORY;
      }
      N.mom_cap = rows;
    }
    float *mom = N.mom_d;
    for (IrlsEdge &E : N.edges) {
      E.mom = mom;
      mom += (size_t)kMoments * E.n;
    }
    if (!N.edges.empty() && cudaMemcpyAsync(N.edges_d, N.edges.data(), sizeof(IrlsEdge) * N.edges.size(),
                                            cudaMemcpyHostToDevice, h->stream) != cudaSuccess) {
      cleanup();
      return CVO_ERR_CUDA;
    }
    if ((rc = N.moments(poses))) { cleanup(); return rc; }
    if ((rc = lm_solve(N, nf, poses, hold, p.multiframe_iterations_per_solve, &steps))) { cleanup(); return rc; }
    double change = 0.0;
    for (int f = 0; f < nf; f++) change += pose_change(&old[12 * f], poses + 12 * f);
    bool all_min = true;
    for (int e = 0; e < ne; e++) {
      // BinaryStateGPU::update_ell (IRLS_State_GPU.cpp:117-146)
      iters_per_ell[e]++;
      if (nz_last[e] > 0 && prev_nnz[e] <= nz_last[e] && iters_per_ell[e] / p.multiframe_iter_per_ell > 0) {
        ell[e] = ell[e] * (double)p.multiframe_ell_decay_rate;
        nz_last[e] = 0;
        iters_per_ell[e] = 0;
      }
      if (ell[e] < ell_min) ell[e] = ell_min;
      else if (ell[e] > ell_max) ell[e] = ell_max;
      all_min = all_min && std::fabs((double)(float)ell[e] - ell_min) < 1e-4;
    }
    iter++;
    if (all_min && change < 1e-5) break;
    if (iter >= p.multiframe_max_iters) break;
  }
  cleanup();
  if (iters) *iters = iter;
  auto t1 = std::chrono::steady_clock::now();
  if (secs) *secs = std::chrono::duration<double>(t1 - t0).count();
  return CVO_OK;
}

}  // namespace cvo_gb
