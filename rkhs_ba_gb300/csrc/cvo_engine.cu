// cvo_engine.cu -- batched, device-resident CVO iteration engine.
//
// The reference's align loop (align_impl, src/cvo/CvoGPU.cu:1239-1477) runs on
// the host with about ten blocking host<->device crossings per iteration.  Here
// the whole iteration, including its scalar tail (step size, pose update,
// lengthscale schedule, neighbour-cap update, stopping tests), runs on the GPU
// for every pair of a batch; the host only relaunches a captured CUDA graph of
// `kChunk` iterations and reads one counter of unfinished pairs per chunk.
#include <cmath>
#include <cstring>
#include <algorithm>
#include <chrono>
#include <cstdio>
#include "cvo_internal.h"
#include "cvo_kernels.cuh"
#include "cvo_lie.cuh"

namespace cvo_gb {

namespace {

constexpr int kChunk = 8;

// ------------------------------------------------------------- transform
// Writes the transformed targets twice: in tile order (read by k_cand) and in
// original order (gathered by index by k_rows and k_step).
__global__ void k_transform(BatchDev B) {
  int gt = blockIdx.x * blockDim.x + threadIdx.x;
  if (gt == 0 && *B.active > 0) *B.active_iters += 1;
  if (gt < 2) B.heavy_ctr[gt] = 0;
  if (gt >= B.total_targets) return;
  int p = find_segment(B.tgt_off, B.npairs, gt);
  PairDev *P = &B.pairs[p];
  if (P->done) return;
  int t = gt - B.tgt_off[p];
  float4 y = __ldg(&P->tpos[t]);
  float o0 = xform_row(&P->Ri[0], P->Ti[0], y.x, y.y, y.z);
  float o1 = xform_row(&P->Ri[3], P->Ti[1], y.x, y.y, y.z);
  float o2 = xform_row(&P->Ri[6], P->Ti[2], y.x, y.y, y.z);
  float4 o = make_float4(o0, o1, o2, 0.f);
  P->ycur[t] = o;
  P->yorig[__ldg(&P->tperm[t])] = o;
}

// Totals of the single passes whose rows took two launches, a block per pair.
__global__ void __launch_bounds__(32 * kRowWarps) k_rows_total(BatchDev B) {
  PairDev *P = &B.pairs[blockIdx.x];
  if (P->done) return;
  sum_slots(B, P, 0, kRowSlots * (B.rblk_off[blockIdx.x + 1] - B.rblk_off[blockIdx.x]));
}

// ---------------------------------------------------------------- row sums
// Sums over the z entries of ELL row s of NV terms: X[t] of an entry from term(y, X),
// acc[t] = a X[t] + acc[t], one entry after the other in slot order.  The order is part of the
// result (see k_rows), so a sum is one lane's chain of fused multiply-adds; but what is added
// does not depend on it.  G lanes share a row: they compute the terms of G entries, one each,
// and lane t < NV then adds the G entries' X[t].  A thread per row was as slow as the longest
// of its warp's 32 rows and left most of the chip without a warp.
// The positions of the next entries and the indices of those after them are in flight.
// buf: the warp's; per row NV + 1 lists (the last: a) of G floats, spaced so that the lanes'
// stores hit distinct banks.  Returns acc[lane % G].  All lanes call it; z is the own row's.
template <int G>
struct RowLists {
  static constexpr int kPitch = G == 8 ? 12 : 4;       // floats from list to list
  static constexpr int kRow = G == 8 ? 104 : 20;       // from row to row
  static constexpr int kWarp = 32 / G * kRow;
};

template <int G, int NV, class Term>
__device__ __forceinline__ float row_sums(const PairDev *P, int s, int z, float *buf, Term term) {
  using L = RowLists<G>;
  const int lane = threadIdx.x & 31, sub = lane % G;
  const int *__restrict__ Aj = P->A_j + (size_t)s * P->ld;
  const float *__restrict__ Av = P->A_v + (size_t)s * P->ld;
  const float4 *__restrict__ yorig = P->yorig;
  float *row = buf + lane / G * L::kRow;
  const float4 *mine = reinterpret_cast<const float4 *>(row + min(sub, NV) * L::kPitch);
  const float4 *val = reinterpret_cast<const float4 *>(row + NV * L::kPitch);
  const int most = __reduce_max_sync(FULLMASK, z);
  int j1 = 0;
  float a0 = 0.f, a1 = 0.f, acc = 0.f;
  float4 y0 = make_float4(0.f, 0.f, 0.f, 0.f), y1 = y0;
  if (sub < z) {
    y0 = __ldg(&yorig[Aj[sub]]);
    a0 = Av[sub];
  }
  if (G + sub < z) {
    j1 = Aj[G + sub];
    a1 = Av[G + sub];
  }
  for (int c = 0; c < most; c += G) {
    if (c + G + sub < z) y1 = __ldg(&yorig[j1]);
    float a2 = 0.f;
    if (c + 2 * G + sub < z) {
      j1 = Aj[c + 2 * G + sub];
      a2 = Av[c + 2 * G + sub];
    }
    float X[NV];
    term(y0, X);
    __syncwarp();
#pragma unroll
    for (int t = 0; t < NV; t++) row[t * L::kPitch + sub] = X[t];
    row[NV * L::kPitch + sub] = a0;
    __syncwarp();
    const int here = z - c;
#pragma unroll
    for (int e = 0; e < G; e += 4) {
      const float4 v = mine[e / 4], a = val[e / 4];
      if (e < here) acc = fmaf(a.x, v.x, acc);
      if (e + 1 < here) acc = fmaf(a.y, v.y, acc);
      if (e + 2 < here) acc = fmaf(a.z, v.z, acc);
      if (e + 3 < here) acc = fmaf(a.w, v.w, acc);
    }
    y0 = y1;
    a0 = a1;
    a1 = a2;
  }
  __syncwarp();
  return acc;
}

// FP64 sums over a pair's rows.  Four rows, 32 (a unit) and the units of a slot are added up in a
// fixed tree, and the slots' sums by the last block: how many slots a block takes and how many
// lanes a row follow the batch, the sums do not, so that a pair's result is the same alone and
// in a batch.
// Units of a block.  60 iterations on 8 pairs of 20k-50k colour points, gradient and step: 20.1 ms
// with 4, 25.7 with 8, 18.9 with 2, which takes a seventh longer on 128k scans.
constexpr int kMostUnits = 4;

// One pass of the block over its rows (lane t < NV of G holds term t of its row in v): the sums
// of four rows each -> quads.
template <int G, int NV>
__device__ __forceinline__ void keep_quads(double v, int pass, double (*quads)[8][NV]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v += __shfl_xor_sync(FULLMASK, v, G);
  v += __shfl_xor_sync(FULLMASK, v, 2 * G);
  constexpr int L = 4 * G;              // lanes of four rows: a warp, or half of one
  const int quad = 32 / L * w + lane / L;
  if (lane % L < NV) quads[(32 / L) * pass + quad / 8][quad % 8][lane % L] = v;
}

// The sums of the block's `rows` rows -> part; whether this is the pair's last block, whose tot
// then holds the sums over all rows.  The groups g are read before the rows: a load after a
// fence waits for L2.
template <int NV>
__device__ __forceinline__ bool sum_blocks(PairDev *P, double (*quads)[8][NV], SumGroups g, int rows, int b, int nb,
                                           unsigned int *counter, double *tot) {
  __shared__ double sh[kStepThreads / 32][8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int units = (rows + kUnitRows - 1) / kUnitRows;
  const int unit = threadIdx.x / NV, k0 = threadIdx.x % NV;
  double t = 0.0;
  __syncthreads();
  if (unit < units) {
    t = quads[unit][0][k0];
    for (int i = 1; i < 8; i++) t += quads[unit][i][k0];
    if (g.slot_units > 1) quads[unit][0][k0] = t;
  }
  if (g.slot_units > 1) {
    if (units * NV > 32) __syncthreads();
    else __syncwarp();                  // one warp has them all
    const int u0 = unit * g.slot_units, u1 = min(units, u0 + g.slot_units);
    if (u0 < u1) {
      t = quads[u0][0][k0];
      for (int u = u0 + 1; u < u1; u++) t += quads[u][0][k0];
    }
  }
  if (unit * g.slot_units < units) {
    P->part[(size_t)(b * g.block_slots + unit) * kPartStride + k0] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == (unsigned)(nb - 1);
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // lane t of eight takes term t of every 32nd slot
  double acc = 0.0;
  const int k = threadIdx.x & 7;
  if (k < NV)
#pragma unroll 8
    for (int q = threadIdx.x >> 3; q < g.slots; q += kStepThreads / 8) acc += __ldcg(P->part + (size_t)q * kPartStride + k);
  acc += __shfl_xor_sync(FULLMASK, acc, 8);
  acc += __shfl_xor_sync(FULLMASK, acc, 16);
  if (lane < 8) sh[w][lane] = acc;
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = sh[0][threadIdx.x];
    for (int q = 1; q < kStepThreads / 32; q++) t += sh[q][threadIdx.x];
    tot[threadIdx.x] = t;
  }
  __syncthreads();
  return true;
}

// The gradient from the final ELL entries: omega = sum a (x cross y) / c, v = sum a (y - x) / d
// and sum a, FP32 per row, FP64 over rows (CvoGPU.cu:2001-2120 computes the same sums from the
// sparse kernel matrix).  The last block of a pair finishes the pass and normalises.
// Bounds: issue and L2 latency of index -> position, see row_sums.
__global__ void __launch_bounds__(kStepThreads) k_gradient(BatchDev B, KParams K) {
  constexpr int G = 8;
  __shared__ __align__(16) float buf[kStepThreads / 32][RowLists<G>::kWarp];
  __shared__ double quads[kMostUnits][8][7], tot[7];
  const int blk = blockIdx.x;
  if (blk >= B.total_sblocks) return;
  const int p = find_segment(B.sblk_off, B.npairs, blk);
  PairDev *P = &B.pairs[p];
  if (P->done) return;
  const int b = blk - B.sblk_off[p], nb = B.sblk_off[p + 1] - B.sblk_off[p], n = P->n;
  const SumGroups g = P->sums;
  const int block_rows = g.block_slots * g.slot_units * kUnitRows, s0 = b * block_rows, rows = min(n - s0, block_rows);
  const int sub = threadIdx.x % G;
  int nnz = 0, mx = 0;
  for (int pass = 0; pass * (kStepThreads / G) < rows; pass++) {
    const int s = s0 + pass * (kStepThreads / G) + (int)threadIdx.x / G;
    const bool has = s < n;
    const int z = has ? P->nnz_row[s] : 0;
    const float4 x = has ? __ldg(&P->xs[s]) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float t = row_sums<G, 7>(P, has ? s : 0, z, buf[threadIdx.x >> 5], [&](const float4 &y, float (&X)[7]) {
      X[0] = fs(fm(x.y, y.z), fm(x.z, y.y));
      X[1] = fs(fm(x.z, y.x), fm(x.x, y.z));
      X[2] = fs(fm(x.x, y.y), fm(x.y, y.x));
      X[3] = y.x - x.x;
      X[4] = y.y - x.y;
      X[5] = y.z - x.z;
      X[6] = 1.f;
    });
    keep_quads<G, 7>((double)(sub < 3 ? __fdiv_rn(t, K.c) : sub < 6 ? __fdiv_rn(t, K.d) : t), pass, quads);
    if (sub == 0) nnz += z;
    mx = max(mx, z);
  }
  // kept pairs and the longest row
  __shared__ unsigned int sh_nnz, sh_mx;
  if (threadIdx.x == 0) sh_nnz = sh_mx = 0u;
  __syncthreads();
  nnz = __reduce_add_sync(FULLMASK, nnz);
  mx = __reduce_max_sync(FULLMASK, mx);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sh_nnz, (unsigned)nnz);
    atomicMax(&sh_mx, (unsigned)mx);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&P->run_nnz, (unsigned long long)sh_nnz);
    atomicMax(&P->run_max, sh_mx);
  }
  if (!sum_blocks<7>(P, quads, g, rows, b, nb, &P->counter[0], tot)) return;
  if (threadIdx.x != 0) return;
  P->counter[0] = 0;
  pass_finished(B, P, tot[6], (double)__ldcg(&P->run_nnz), (double)__ldcg(&P->run_max));
  P->run_nnz = 0ull;
  P->run_max = 0u;
  for (int k = 0; k < 6; k++) P->grad[k] = tot[k];
  // float normalisation of the stacked gradient (CvoGPU.cu:2096-2104)
  float f[6];
  for (int k = 0; k < 6; k++) f[k] = (float)tot[k];
  float s = 0.f;
  for (int k = 0; k < 6; k++) s = fa(s, fm(f[k], f[k]));
  if (s > 0.f) {
    float nr = __fsqrt_rn(s);
    for (int k = 0; k < 6; k++) f[k] = __fdiv_rn(f[k], nr);
  }
  for (int k = 0; k < 6; k++) P->xi[k] = f[k];
}

// Picks the finest lattice whose cells serve the largest search radius.
__device__ void choose_level(PairDev *P, const KParams &K) {
  float l = range_ell(P->ell, P->src_norm);
  float r = K.use_geo ? sqrtf(geo_d2_thres(l, K.log_geo)) : 0.f;
  int lv = P->nlevels - 1;
  for (int i = 0; i < P->nlevels; i++)
    if (P->level_r[i] >= r) { lv = i; break; }
  P->level = lv;
}

__device__ void pose_to_rinv(PairDev *P) {
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) P->Ri[3 * r + c] = P->R[3 * c + r];
  for (int r = 0; r < 3; r++) {
    float a = fm(P->Ri[3 * r], P->T[0]), b = fm(P->Ri[3 * r + 1], P->T[1]), c = fm(P->Ri[3 * r + 2], P->T[2]);
    P->Ti[r] = -fa(fa(a, b), c);
  }
}

// A_sparsity_indicator_ell_update (src/cvo/CvoGPU.cu:547-665) on ring buffers.
__device__ bool indicator_update(PairDev *P, const KParams &K, float ind) {
  const int L = K.indicator_window_size;
  const int Q = kMaxIndicatorWindow;
  bool decrease = false;
  auto push = [&](float *q, int &head, int &len, float v) { q[(head + len) % Q] = v; len++; };
  if (P->qs_len < L) { push(P->qs, P->qs_head, P->qs_len, ind); P->ssum = fa(P->ssum, ind); }
  if (P->qs_len >= L && P->qe_len < L) { push(P->qe, P->qe_head, P->qe_len, ind); P->esum = fa(P->esum, ind); }
  if (P->qs_len >= L && P->qe_len >= L) {
    float ratio = __fdiv_rn(P->esum, P->ssum);
    if (ratio > fs(1.f, K.indicator_stable_threshold) && ratio < fa(1.f, K.indicator_stable_threshold)) {
      decrease = true;
      P->qs_head = P->qs_len = P->qe_head = P->qe_len = 0;
      P->ssum = 0.f; P->esum = 0.f;
    } else {
      float f = P->qe[P->qe_head % Q];
      P->esum = fs(P->esum, f);
      P->ssum = fa(P->ssum, f);
      push(P->qs, P->qs_head, P->qs_len, f);
      P->qe_head = (P->qe_head + 1) % Q; P->qe_len--;
      P->ssum = fs(P->ssum, P->qs[P->qs_head % Q]);
      P->qs_head = (P->qs_head + 1) % Q; P->qs_len--;
      push(P->qe, P->qe_head, P->qe_len, ind);
      P->esum = fa(P->esum, ind);
    }
  }
  return decrease;
}

// Scalar tail of one iteration of align_impl (src/cvo/CvoGPU.cu:1339-1433).
__device__ void finalize_iteration(BatchDev &B, PairDev *P, const KParams &K) {
  const int k = P->iter;
  double step = step_from_terms(P->bcde, (double)K.min_step, (double)K.max_step);
  P->step = step;
  const float *xi = P->xi;
  float wn = __fsqrt_rn(fa(fa(fm(xi[0], xi[0]), fm(xi[1], xi[1])), fm(xi[2], xi[2])));
  float vn = __fsqrt_rn(fa(fa(fm(xi[3], xi[3]), fm(xi[4], xi[4])), fm(xi[5], xi[5])));
  if ((double)wn < (double)K.eps && (double)vn < (double)K.eps) {
    if (wn < 1e-8f && vn < 1e-8f) P->ret = -1;
    P->done = 1;
    atomicSub(B.active, 1);
    return;
  }
  float X[12];
  exp_sek3(xi, (float)step, X);
  double dR[9], dT[3];
  for (int r = 0; r < 3; r++) {
    for (int c = 0; c < 3; c++) dR[3 * r + c] = X[4 * r + c];
    dT[r] = X[4 * r + 3];
  }
  double Rd[9], Td[3];
  for (int t = 0; t < 9; t++) Rd[t] = P->R[t];
  for (int t = 0; t < 3; t++) Td[t] = P->T[t];
  for (int r = 0; r < 3; r++) {
    double s = dm(Rd[3 * r], dT[0]);
    s = da(s, dm(Rd[3 * r + 1], dT[1]));
    s = da(s, dm(Rd[3 * r + 2], dT[2]));
    P->T[r] = __double2float_rn(da(s, Td[r]));
  }
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) {
      double s = dm(Rd[3 * r], dR[c]);
      s = da(s, dm(Rd[3 * r + 1], dR[3 + c]));
      s = da(s, dm(Rd[3 * r + 2], dR[6 + c]));
      P->R[3 * r + c] = __double2float_rn(s);
    }
  double dist = dist_se3(dR, dT);
  P->dist = dist;
  float ip_curr = __double2float_rn(__ddiv_rn((double)P->nnz_sum, sqrt(dm((double)P->n, (double)P->m))));
  bool need_decay = indicator_update(P, K, ip_curr);
  pose_to_rinv(P);
  if (dist < (double)K.eps_2) {
    P->done = 1;
    atomicSub(B.active, 1);
    return;
  }
  if (k > K.ell_decay_start && need_decay) {
    P->ell = fm(P->ell, K.ell_decay_rate);
    if (P->ell < K.ell_min) P->ell = K.ell_min;
  }
  int nc = (int)((double)P->max_row * 1.2);
  P->cap = min(P->capmax, nc);
  P->iter = k + 1;
  if (P->iter >= K.max_iter) {
    P->done = 1;
    atomicSub(B.active, 1);
    return;
  }
  choose_level(P, K);
}

// -------------------------------------------------------------------- step
// 1 / (2 l^2), rounded from double.
__device__ __forceinline__ float step_coef(float l) {
  return __double2float_rn(__ddiv_rn(1.0, dm(dm(2.0, (double)l), (double)l)));
}

// Taylor step-size terms (compute_step_size_xi + compute_step_size_poly_coeff,
// src/cvo/CvoGPU.cu:333-462) per ELL row in FP32, one entry after the other (see row_sums),
// FP64 across rows; the last block of a pair adds the blocks' sums and finishes the iteration.
// Bounds: issue (some 100 instructions per 32 entries), then the scalar tail.
template <int G>
__global__ void __launch_bounds__(kStepThreads, 4) k_step(BatchDev B, KParams K) {
  __shared__ __align__(16) float buf[kStepThreads / 32][RowLists<G>::kWarp];
  __shared__ double quads[kMostUnits][8][4], tot[4];
  __shared__ float sh_coef;
  const int blk = blockIdx.x;
  if (blk >= B.total_sblocks) return;
  const int p = find_segment(B.sblk_off, B.npairs, blk);
  PairDev *P = &B.pairs[p];
  if (P->done) return;
  const int b = blk - B.sblk_off[p], nb = B.sblk_off[p + 1] - B.sblk_off[p], n = P->n;
  const float w0 = P->xi[0], w1 = P->xi[1], w2 = P->xi[2];
  const float u0v = P->xi[3], u1v = P->xi[4], u2v = P->xi[5];
  if (threadIdx.x == 0) sh_coef = step_coef(P->ell);
  __syncthreads();
  const float coef0 = sh_coef;
  const SumGroups g = P->sums;
  const int block_rows = g.block_slots * g.slot_units * kUnitRows, s0 = b * block_rows, rows = min(n - s0, block_rows);
  for (int pass = 0; pass * (kStepThreads / G) < rows; pass++) {
    const int s = s0 + pass * (kStepThreads / G) + (int)threadIdx.x / G;
    const bool has = s < n;
    const int z = has ? P->nnz_row[s] : 0;
    const float4 x = has ? __ldg(&P->xs[s]) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float coef = K.use_range_ell_step ? step_coef(range_ell(P->ell, x.w)) : coef0;
    const float t = row_sums<G, 4>(P, has ? s : 0, z, buf[threadIdx.x >> 5], [&](const float4 &y, float (&X)[4]) {
      float ux = w1 * y.z - w2 * y.y + u0v, uy = w2 * y.x - w0 * y.z + u1v, uz = w0 * y.y - w1 * y.x + u2v;
      float px = w1 * uz - w2 * uy, py = w2 * ux - w0 * uz, pz = w0 * uy - w1 * ux;          // xi^2 z
      float qx = w1 * pz - w2 * py, qy = w2 * px - w0 * pz, qz = w0 * py - w1 * px;          // xi^3 z
      float rx = w1 * qz - w2 * qy, ry = w2 * qx - w0 * qz, rz = w0 * qy - w1 * qx;          // xi^4 z
      float dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
      float normxiz2 = ux * ux + uy * uy + uz * uz;
      float xiz_dot_xi2z = -(ux * px + uy * py + uz * pz);
      float epsil_const = (px * px + py * py + pz * pz) + 2.f * (ux * qx + uy * qy + uz * qz);
      float beta = -2.f * coef * (ux * dx + uy * dy + uz * dz);
      float gamma = -coef * (normxiz2 + 2.f * (px * dx + py * dy + pz * dz));
      float delta = 2.f * coef * (xiz_dot_xi2z - (qx * dx + qy * dy + qz * dz));
      float epsil = -coef * (epsil_const + 2.f * (rx * dx + ry * dy + rz * dz));
      float b2 = beta * beta;
      X[0] = beta;
      X[1] = gamma + 0.5f * b2;
      X[2] = delta + beta * gamma + b2 * beta * (1.f / 6.f);
      X[3] = epsil + beta * delta + 0.5f * b2 * gamma + 0.5f * gamma * gamma + b2 * b2 * (1.f / 24.f);
    });
    keep_quads<G, 4>((double)t, pass, quads);
  }
  if (!sum_blocks<4>(P, quads, g, rows, b, nb, &P->counter[1], tot)) return;
  // The scalar tail is one thread's chain of dependent reads and writes of the pair's state:
  // in shared memory they cost 30 cycles instead of an L2 round trip each.
  __shared__ PairDev state;
  static_assert(sizeof(PairDev) % 4 == 0, "copied by words");
  for (int i = threadIdx.x; i < (int)(sizeof(PairDev) / 4); i += kStepThreads)
    reinterpret_cast<int *>(&state)[i] = reinterpret_cast<const int *>(P)[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    state.counter[1] = 0;
    for (int k = 0; k < 4; k++) state.bcde[k] = tot[k];
    finalize_iteration(B, &state, K);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (int)(sizeof(PairDev) / 4); i += kStepThreads)
    reinterpret_cast<int *>(P)[i] = reinterpret_cast<const int *>(&state)[i];
}

// ----------------------------------------------------- association export
// Entries of each row (ELL row s is row perm[s], or s), and 0 after the last.
__global__ void k_csr_counts(int n, const int *nnz, const int *perm, int *count) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) count[perm ? perm[s] : s] = nnz[s];
  if (s == 0) count[n] = 0;
}

// ELL rows to CSR, a warp per row.
__global__ void __launch_bounds__(128) k_csr_rows(int n, const int *nnz, const int *perm, int ld, const int *ell_j, const float *ell_v,
                                                  const int *rowptr, int *col, float *val) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= n) return;
  const int z = nnz[s], o = rowptr[perm ? perm[s] : s];
  for (int c = lane; c < z; c += 32) {
    col[o + c] = ell_j[(size_t)s * ld + c];
    val[o + c] = ell_v[(size_t)s * ld + c];
  }
}

// --------------------------------------------------------- template dispatch
int select_kernels(const KParams &K, int F, int C, AssocKernels *a) {
  int fch = K.use_int ? (F + 3) / 4 : 0;
  int lch = K.use_sem ? label_chunks(C) : 0;
  bool gt = K.use_gtype != 0;
  if (fch > 2 || lch > 9) return CVO_ERR_UNSUPPORTED;
  // the feature and label chunk counts are the storage strides of the clouds
  if (lch == 0) return assoc_kernels_no_labels(fch, gt, a);
  if (lch == 5) return assoc_kernels_labels5(fch, gt, a);
  return lch == 9 ? assoc_kernels_labels9(fch, gt, a) : CVO_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------ device arena
struct Arena {
  char *base = nullptr;
  size_t cap = 0, off = 0;
  template <typename T>
  T *take(size_t count) {
    size_t bytes = (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
    T *p = reinterpret_cast<T *>(base + off);
    off += bytes;
    return p;
  }
};

}  // namespace

struct Workspace {
  char *dev = nullptr;
  size_t dev_cap = 0;
  int *pinned = nullptr;
  // the last align batch's instantiated graph of kChunk iterations, and the launch
  // parameters it was captured with: a later batch with the same parameters (same
  // shapes in the same workspace) relaunches it without capturing again
  cudaGraphExec_t align_exec = nullptr;
  std::vector<unsigned char> align_key;
  long long align_per_chunk = 0;
};

static int ensure_workspace(Handle *h, size_t bytes) {
  if (!h->ws) h->ws = new Workspace();
  Workspace *w = h->ws;
  if (!w->pinned) CVO_CUDA_TRY(h, cudaMallocHost((void **)&w->pinned, 4096));
  if (w->dev_cap >= bytes) return 0;
  if (w->dev) { cudaStreamSynchronize(h->stream); cudaFree(w->dev); w->dev = nullptr; w->dev_cap = 0; }
  // a cached graph's kernels point into the old workspace
  if (w->align_exec) { cudaGraphExecDestroy(w->align_exec); w->align_exec = nullptr; w->align_key.clear(); }
  size_t want = bytes + bytes / 4 + (1 << 20);
  cudaError_t e = cudaMalloc((void **)&w->dev, want);
  if (e == cudaErrorMemoryAllocation) {      // without room to grow
    cudaGetLastError();
    want = bytes;
    e = cudaMalloc((void **)&w->dev, want);
  }
  if (e != cudaSuccess) {
    set_cuda_error(h, e, "workspace");
    return e == cudaErrorMemoryAllocation ? CVO_ERR_OUT_OF_MEMORY : CVO_ERR_CUDA;
  }
  w->dev_cap = want;
  return 0;
}

void free_workspace(Handle *h) {
  if (!h->ws) return;
  if (h->ws->align_exec) cudaGraphExecDestroy(h->ws->align_exec);
  if (h->ws->dev) cudaFree(h->ws->dev);
  if (h->ws->pinned) cudaFreeHost(h->ws->pinned);
  delete h->ws;
  h->ws = nullptr;
}

KParams make_kparams(const cvo_params &p) {
  KParams k;
  memset(&k, 0, sizeof(k));
  k.sigma2 = p.sigma * p.sigma;
  k.c2 = p.c_ell * p.c_ell;
  k.c_sigma2 = p.c_sigma * p.c_sigma;
  k.s_ell = p.s_ell;
  k.s_sigma2 = p.s_sigma * p.s_sigma;
  k.s_sigma_sq = p.s_sigma * p.s_sigma;
  k.sp_thres = p.sp_thres;
  k.log_geo = logf(p.sp_thres / k.sigma2);
  k.d2_c_thres = 1.f;
  k.d2_s_thres = 1.f;
  if (p.is_using_intensity) k.d2_c_thres = (float)(-2.0 * (double)k.c2 * (double)logf(p.sp_thres / k.c_sigma2));
  if (p.is_using_semantics)
    k.d2_s_thres = (float)(-2.0 * (double)k.s_ell * (double)k.s_ell * (double)logf(p.sp_thres / k.s_sigma2));
  k.c = p.c; k.d = p.d;
  k.eps = p.eps; k.eps_2 = p.eps_2; k.min_step = p.min_step; k.max_step = p.max_step;
  k.ell_decay_rate = p.ell_decay_rate; k.ell_min = p.ell_min;
  k.indicator_stable_threshold = p.indicator_stable_threshold;
  k.ell_decay_start = p.ell_decay_start;
  k.indicator_window_size = p.indicator_window_size;
  k.max_iter = p.MAX_ITER;
  k.nn_max = p.nearest_neighbors_max;
  k.use_range_ell_step = p.is_using_range_ell;
  k.use_geo = p.is_using_geometry;
  k.use_int = p.is_using_intensity;
  k.use_sem = p.is_using_semantics;
  k.use_gtype = p.is_using_geometric_type;
  {
    float t = 2.f * k.c2;
    k.inv2c2 = 1.f / t;
  }
  k.val_scale = 1.f;
  k.two_c2 = 2.0 * (double)k.c2;
  // Kernel value bound: a <= sigma^2 c_sigma^2 s_sigma^2 exp(-(d2/(2l^2) + d2c/(2c^2))) (the geometric-type
  // factor is <= 1), so a > sp_thres needs the exponent below ln(sigma^2 c_sigma^2 s_sigma^2 / sp_thres).
  // Without the geometric kernel the colour term alone bounds the value.
  k.use_mma = 0;
  k.mma_tau = 0.f;
  if ((k.use_geo || k.use_int) && p.sp_thres > 0.f && (!k.use_geo || k.sigma2 > 0.f) && (!k.use_int || k.c_sigma2 > 0.f) &&
      (!k.use_sem || k.s_sigma_sq > 0.f)) {
    double lb = -std::log((double)p.sp_thres);
    if (k.use_geo) lb += std::log((double)k.sigma2);
    if (k.use_int) lb += std::log((double)k.c_sigma2);
    if (k.use_sem) lb += std::log((double)k.s_sigma_sq);
    if (k.val_scale > 0.f) lb += std::log((double)k.val_scale);
    k.mma_tau = (float)(lb + 1e-3);
    k.use_mma = 1;
    // below this the value and each of its terms pass their thresholds
    if (!k.use_sem && !k.use_gtype) {
      if (k.use_geo) lb = std::min(lb, -(double)k.log_geo);
      if (k.use_int) lb = std::min(lb, (double)k.d2_c_thres * (double)k.inv2c2);
      k.sure_tau = (float)(lb - 2e-3);
    }
  }
  return k;
}

// The lattice for search radius r and source blocks of diagonal ext: cells small against r, a
// block's box about 8 of them along each axis.
static float cell_for_radius(float r, float ext) { return std::max(r / 4.f, (ext + 2.f * r) / 8.f); }
// Largest radius a cell of size hc serves (inverse of cell_for_radius).
static float radius_for_cell(float hc, float ext) { return std::max(0.f, std::min(4.f * hc, 0.5f * (8.f * hc - ext))); }
static float host_range_ell(float ell, float dist) { return (float)(((double)dist / 500.0 + 1.0) * (double)ell); }
static float host_radius(const KParams &K, float ell, float norm) {
  if (!K.use_geo) return INFINITY;
  float l = host_range_ell(ell, norm);
  float d2t = (float)(-2.0 * (double)l * (double)l * (double)K.log_geo);
  return std::sqrt(std::max(d2t, 0.f));
}

// The finest of the pair's lattices that serves search radius r.
static int level_for(const PairDev &P, float r) {
  for (int i = 0; i < P.nlevels; i++)
    if (P.level_r[i] >= r) return i;
  return P.nlevels - 1;
}

long long tune_items(long long rows) { return (rows + 127) / 128; }

long long tune_key(int F, int C, long long rows) {
  int b = 0;
  while ((1LL << (b + 1)) <= rows && b < 40) b++;
  return ((long long)F << 32) | ((long long)C << 16) | b;
}

// ------------------------------------------------------------ batch setup
namespace {

struct BatchHost {
  BatchDev B;
  std::vector<PairDev> pairs;
  std::vector<int> item_off, tgt_off, rblk_off, sblk_off;
  AssocKernels fn;
  int cand_blocks = 0, xform_blocks = 0, rows_blocks = 0;
  bool split_rows = false;          // rows of few candidates in a launch of their own
  bool few_rows = false;            // k_step with eight lanes a row
  bool ordered = false;             // rows in the order of the targets' lattice (RankLevel)
};

// Work items that keep the candidate test's warps busy: about two per resident warp slot,
// so that tiles of uneven cost even out.  Fewer tiles than that are split over their
// targets (each split repeats the tile's setup, some 400 instructions against 5,000 or
// more for a tile of a 50k cloud).
constexpr long long kCandItems = 10240;

// Lays out every device buffer of a batch in the handle's workspace.
int lay_out_batch(Handle *h, const KParams &K, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                  const std::vector<float> &T_init, int mode, int capmax, const std::vector<float> &ell0, BatchHost *bh) {
  const int np = (int)srcs.size();
  int F = srcs[0]->F, C = srcs[0]->C;
  for (int p = 0; p < np; p++) {
    if (srcs[p]->F != F || tgts[p]->F != F || srcs[p]->C != C || tgts[p]->C != C) return CVO_ERR_INVALID_ARG;
    if (K.use_gtype && (!srcs[p]->has_geo || !tgts[p]->has_geo)) return CVO_ERR_INVALID_ARG;
  }
  int rc = select_kernels(K, F, C, &bh->fn);
  if (rc) return rc;
  // division of the candidate test: forced by the autotuner, else the tuned one for this
  // key, else the default.  The splits are keyed by the pairs' size (it sets the work per
  // tile); the items per SM by the batch's number of work items (it sets how they spread
  // over the SMs), so a value tuned on one pair does not carry over to a batch of many.
  TuneConfig tc;
  long long tiles = 0, maxn = 0;
  int maxm = 1;
  for (int p = 0; p < np; p++) {
    tiles += group_count(srcs[p]->n);
    maxn = std::max<long long>(maxn, srcs[p]->n);
    maxm = std::max(maxm, tgts[p]->n);
  }
  if (h->tune_force) {
    tc = *h->tune_force;
  } else {
    long long items = 0;
    for (int p = 0; p < np; p++) items += tune_items(srcs[p]->n);
    auto it = h->tuned.find(tune_key(F, C, maxn));
    if (it != h->tuned.end()) tc = it->second;
    tc.blocks_per_sm = 0;
    auto ib = h->tuned_bps.find(tune_key(F, C, items));
    if (ib != h->tuned_bps.end()) tc.blocks_per_sm = ib->second;
  }
  const int sms = h->num_sms > 0 ? h->num_sms : 152;
  const double want = (tc.blocks_per_sm > 0 ? 4.0 * tc.blocks_per_sm * sms : (double)kCandItems) *
                      (tc.cell_div_r / 4.0) * (tc.cell_div_ext / 8.0);
  const int splits = (int)std::min<double>(kMaxSplits, std::max(1.0, std::ceil(want / (double)std::max<long long>(tiles, 1))));
  // orders of the targets (align and edges): the lattices of every radius the lengthscale may reach
  bh->ordered = mode == MODE_ALIGN || mode == MODE_EDGES;
  std::vector<std::vector<RankLevel>> lv(np);
  std::vector<std::vector<float>> lr(np);
  for (int p = 0; p < np && bh->ordered; p++) {
    const float ext = srcs[p]->tile_ext;
    std::vector<int> exps;
    if (!K.use_geo) {
      exps.push_back(1000);
    } else {
      const float ell_hi = ell0[p], ell_lo = mode == MODE_ALIGN ? std::min(K.ell_min, ell_hi) : ell_hi;
      const float r_hi = host_radius(K, ell_hi, srcs[p]->max_norm), r_lo = host_radius(K, ell_lo, 0.f);
      int e_hi = level_for_radius(cell_for_radius(r_hi, ext)), e_lo = level_for_radius(cell_for_radius(r_lo, ext));
      if (e_lo > e_hi) std::swap(e_lo, e_hi);      // a negative ell_min: its square counts
      if (e_hi - e_lo + 1 > 24) e_lo = e_hi - 23;
      for (int e = e_lo; e <= e_hi; e++) exps.push_back(e);
    }
    if (tgts[p]->n == 0) continue;
    if ((rc = cloud_ranks(h, tgts[p], exps))) return rc;
    for (int e : exps) {
      lv[p].push_back(tgts[p]->ranks[e]);
      lr[p].push_back(e >= 1000 ? INFINITY : radius_for_cell(lv[p].back().h, ext));
    }
  }
  // sizes
  bh->item_off.assign(np + 1, 0);
  bh->tgt_off.assign(np + 1, 0);
  bh->rblk_off.assign(np + 1, 0);
  bh->sblk_off.assign(np + 1, 0);
  size_t bytes = 0;
  auto add = [&](size_t b) { bytes += (b + 255) & ~(size_t)255; };
  long long rows_all = 0;
  for (int p = 0; p < np; p++) rows_all += srcs[p]->n;
  const int ell_ld = (std::max(capmax, 1) + 3) & ~3;   // 16-byte aligned ELL rows
  // An ordered row that keeps more than cap + order_cap pairs stays in index order.  A pair of an
  // align batch has one rule whatever the batch, so that its pose is the same alone.  A window is
  // one problem, and another order of some rows moves its poses by up to 3e-5: there the value
  // shrinks beyond 524,288 rows, as it always has.
  const int order_cap = mode != MODE_EDGES || rows_all == 0 ? kOrderCap
                                                            : (int)std::min<long long>(kOrderCap, (16ll << 30) / (8ll * rows_all)) & ~3;
  const bool ell = mode != MODE_IP;                    // an inner product needs no kernel matrix
  std::vector<int> sp(np), caps(np);
  // Rows of a k_gradient or k_step block: 32 (four to a warp), or of large batches multiples of
  // 64, up to kMostUnits units, so that some eight blocks per SM leave their sums to the last
  // one.  A pair's slots (groups of its FP64 sums) are the blocks that its own rows ask for.
  auto share = [&](long long rows) {
    const long long per_block = rows / (8ll * sms);
    return per_block <= kUnitRows ? kUnitRows : (int)std::min<long long>(64 * ((per_block + 63) / 64), kMostUnits * kUnitRows);
  };
  auto groups_of = [&](int n) {
    const int slot = share(n);
    return SumGroups{slot / kUnitRows, (n + slot - 1) / slot, share(rows_all) / slot};
  };
  bh->few_rows = share(rows_all) == kUnitRows;
  for (int p = 0; p < np; p++) {
    int n = srcs[p]->n, m = tgts[p]->n;
    const int ns = group_count(group_count(m));
    sp[p] = std::max(1, std::min(splits, ns));
    if (!K.use_mma) sp[p] = 1;
    bh->item_off[p + 1] = bh->item_off[p] + group_count(n) * sp[p];
    bh->tgt_off[p + 1] = bh->tgt_off[p] + m;
    const SumGroups g = groups_of(n);
    int rb = (n + kRowsPerBlock - 1) / kRowsPerBlock, sb = (g.slots + g.block_slots - 1) / g.block_slots;
    bh->rblk_off[p + 1] = bh->rblk_off[p] + rb;
    bh->sblk_off[p + 1] = bh->sblk_off[p] + sb;
    add(sizeof(float4) * m);                                     // ycur
    add(sizeof(float4) * m);                                     // yorig
    add(ell ? sizeof(int) * (size_t)n * ell_ld : 0);             // ELL
    add(ell ? sizeof(float) * (size_t)n * ell_ld : 0);
    add(sizeof(RankLevel) * lv[p].size());
    add(sizeof(int2) * (size_t)n * sp[p]);                       // entry counts
    add(sizeof(int) * n);                                        // nnz_row
    add(sizeof(double) * kPartStride * (size_t)std::max(kRowSlots * rb, g.slots)); // partials
    add(sizeof(unsigned) * 2);
    bytes += 12 * 256;                                           // room for empty pieces
  }
  add(sizeof(PairDev) * np);
  add(sizeof(int) * (np + 1) * 4);
  add(sizeof(int) * 8);
  const int groups = (kRowsPerBlock / kRowsHeavy) * bh->rblk_off[np];
  add(sizeof(int) * (size_t)groups);                                               // groups of long rows
  // Ordered rows of more than kRowOrdered entries pass through room of their own: each row's, or
  // beyond kRowRoom (room in every row would double the kernel matrix) each resident warp's, with
  // the rows listed as those of large targets are.  Listing them anyway is up to a fourth slower
  // (20 iterations on 8k colour points at a cap of 2,000: 4.8 against 6.0 ms).
  const int longest = std::min(capmax, maxm);
  const bool long_rows = bh->ordered && longest > kRowOrdered;
  bh->split_rows = (K.use_mma && maxm > kRowSplitTargets) || (long_rows && sizeof(uint2) * rows_all * longest > kRowRoom);
  bh->rows_blocks = std::max(1, bh->split_rows ? std::min(groups, 5 * sms) : groups);
  const size_t long_room = !long_rows ? 0 : (size_t)longest * (bh->split_rows ? (long long)bh->rows_blocks * kRowWarps : rows_all);
  add(sizeof(uint2) * long_room);
  add(sizeof(double));
  // Candidate entries per row: one per target group, at most 16 GB for the batch, and fewer if the
  // device has no such room (a row that needs more is evaluated by an index-ordered scan of the
  // targets).
  auto candidates = [&](long long most) {
    size_t sum = 0;
    for (int p = 0; p < np; p++) {
      const int ns = group_count(group_count(tgts[p]->n));
      caps[p] = !K.use_mma ? 1 : std::max(1, (int)std::min<long long>(kGroup * ((ns + sp[p] - 1) / sp[p]), most / sp[p]));
      sum += (sizeof(uint2) * (size_t)srcs[p]->n * sp[p] * caps[p] + 255) & ~(size_t)255;
    }
    return sum;
  };
  long long most = std::min<long long>(group_count(maxm) + kGroup * kMaxSplits, (16ll << 30) / (8ll * std::max(rows_all, 1ll)));
  const std::string error = h->last_error;
  rc = ensure_workspace(h, bytes + candidates(most));
  while (rc == CVO_ERR_OUT_OF_MEMORY && K.use_mma && most > kGroup) rc = ensure_workspace(h, bytes + candidates(most /= 2));
  if (rc) return rc;
  h->last_error = error;
  Arena ar;
  ar.base = h->ws->dev;
  ar.cap = h->ws->dev_cap;
  bh->pairs.assign(np, PairDev());
  int active = 0;
  for (int p = 0; p < np; p++) {
    PairDev &P = bh->pairs[p];
    memset(&P, 0, sizeof(P));
    DevCloud *s = srcs[p], *t = tgts[p];
    P.n = s->n; P.m = t->n; P.F = F; P.C = C;
    P.xs = s->spos; P.xf = s->sfeat; P.xl = s->slab; P.xg = s->sgeo; P.sbox = s->gbox;
    P.tpos = t->spos; P.tperm = t->sperm; P.tfs = t->sfeat; P.tbox = t->gbox; P.tsup = t->sbox; P.trange = t->grange;
    P.groups = group_count(t->n);
    P.ycur = ar.take<float4>(t->n);
    P.yorig = ar.take<float4>(t->n);
    P.A_j = ar.take<int>(ell ? (size_t)s->n * ell_ld : 0);
    P.A_v = ar.take<float>(ell ? (size_t)s->n * ell_ld : 0);
    P.ld = ell_ld;
    P.splits = sp[p];
    P.cap_split = caps[p];
    P.cand_pitch = sp[p] * caps[p];
    P.cand = ar.take<uint2>((size_t)s->n * P.cand_pitch);
    P.cand_cnt = ar.take<int2>((size_t)s->n * sp[p]);
    P.tf = t->feat; P.tl = t->lab; P.tg = t->geo;
    P.nnz_row = ar.take<int>(s->n);
    P.sums = groups_of(s->n);
    const int rb = bh->rblk_off[p + 1] - bh->rblk_off[p];
    P.part = ar.take<double>(kPartStride * (size_t)std::max(kRowSlots * rb, P.sums.slots));
    P.counter = ar.take<unsigned>(2);
    P.capmax = capmax;
    P.mode = mode;
    for (int r = 0; r < 3; r++) {
      for (int c = 0; c < 3; c++) P.R[3 * r + c] = T_init[16 * p + c * 4 + r];
      P.T[r] = T_init[16 * p + 12 + r];
    }
    // target transform R^T, -R^T T (canonical order)
    for (int r = 0; r < 3; r++)
      for (int c = 0; c < 3; c++) P.Ri[3 * r + c] = P.R[3 * c + r];
    for (int r = 0; r < 3; r++) {
      float a = P.Ri[3 * r] * P.T[0], b = P.Ri[3 * r + 1] * P.T[1], c = P.Ri[3 * r + 2] * P.T[2];
      P.Ti[r] = -((a + b) + c);
    }
    P.ell = ell0[p];
    P.cap = capmax;
    P.order_cap = bh->ordered ? order_cap : 0;
    P.src_norm = s->max_norm;
    if (bh->ordered) {
      RankLevel *levels = ar.take<RankLevel>(lv[p].size());
      CVO_CUDA_TRY(h, cudaMemcpyAsync(levels, lv[p].data(), sizeof(RankLevel) * lv[p].size(), cudaMemcpyHostToDevice, h->stream));
      P.levels = levels;
      P.nlevels = (int)lv[p].size();
      for (int i = 0; i < P.nlevels && i < 24; i++) P.level_r[i] = lr[p][i];
      P.level = level_for(P, host_radius(K, P.ell, s->max_norm));
    }
    P.done = (s->n == 0 || t->n == 0) ? 1 : 0;
    if (!P.done) active++;
  }
  PairDev *pairs_d = ar.take<PairDev>(np);
  int *offs_d = ar.take<int>((size_t)(np + 1) * 4);
  int *ctr_d = ar.take<int>(8);
  int *heavy_d = ar.take<int>(groups);
  uint2 *long_d = ar.take<uint2>(long_room);
  if (long_rows)
    for (int p = 0, row = 0; p < np; row += bh->pairs[p++].n) {
      bh->pairs[p].long_rows = long_d + (bh->split_rows ? 0 : (size_t)row * longest);
      bh->pairs[p].long_pitch = longest;
    }
  double *bytes_d = ar.take<double>(1);
  // zero counters of every pair
  for (int p = 0; p < np; p++) CVO_CUDA_TRY(h, cudaMemsetAsync(bh->pairs[p].counter, 0, 2 * sizeof(unsigned), h->stream));
  CVO_CUDA_TRY(h, cudaMemcpyAsync(pairs_d, bh->pairs.data(), sizeof(PairDev) * np, cudaMemcpyHostToDevice, h->stream));
  std::vector<int> offs;
  for (auto *v : {&bh->item_off, &bh->tgt_off, &bh->rblk_off, &bh->sblk_off}) offs.insert(offs.end(), v->begin(), v->end());
  CVO_CUDA_TRY(h, cudaMemcpyAsync(offs_d, offs.data(), sizeof(int) * offs.size(), cudaMemcpyHostToDevice, h->stream));
  int ctr_h[8] = {0, 0, active, 0, 0, 0, 0, 0};
  CVO_CUDA_TRY(h, cudaMemcpyAsync(ctr_d, ctr_h, sizeof(ctr_h), cudaMemcpyHostToDevice, h->stream));
  CVO_CUDA_TRY(h, cudaMemsetAsync(bytes_d, 0, sizeof(double), h->stream));
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  BatchDev &B = bh->B;
  memset(&B, 0, sizeof(B));
  B.npairs = np;
  B.total_items = bh->item_off[np];
  B.total_targets = bh->tgt_off[np];
  B.pairs = pairs_d;
  B.item_off = offs_d;
  B.tgt_off = offs_d + (np + 1);
  B.rblk_off = offs_d + 2 * (np + 1);
  B.sblk_off = offs_d + 3 * (np + 1);
  B.total_rblocks = bh->rblk_off[np];
  B.total_sblocks = bh->sblk_off[np];
  B.err = ctr_d + 1;
  B.active = ctr_d + 2;
  B.active_iters = ctr_d + 3;
  B.heavy = heavy_d;
  B.heavy_ctr = ctr_d + 4;
  B.assoc_bytes = bytes_d;
  {
    int fch = K.use_int ? (F + 3) / 4 : 0, lch = K.use_sem ? label_chunks(C) : 0;
    B.record_bytes = 16 + 16 * fch + 16 * lch + (K.use_gtype ? 8 : 0);
  }
  bh->cand_blocks = K.use_mma ? (B.total_items + kCandWarps - 1) / kCandWarps : 0;
  bh->xform_blocks = (B.total_targets + 255) / 256;
  return 0;
}

// A batch that is refused may have built orders of a target already, which the cloud keeps: they
// are complete when it returns, since the next batch may run on another handle's stream.
int build_batch(Handle *h, const KParams &K, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                const std::vector<float> &T_init, int mode, int capmax, const std::vector<float> &ell0, BatchHost *bh) {
  const int rc = lay_out_batch(h, K, srcs, tgts, T_init, mode, capmax, ell0, bh);
  if (rc) cudaStreamSynchronize(h->stream);
  return rc;
}

// Inside stream capture an event becomes a record node of the graph only with
// cudaEventRecordExternal (a plain cudaEventRecord only adds a dependency).
inline void mark(Handle *h, const cudaEvent_t *ev, int k) {
  if (ev) cudaEventRecordWithFlags(ev[k], h->stream, cudaEventRecordExternal);
}

// ev (optional): 7 events: 0-4 bracket transform, association phase, reduce and step; 5 and 6
// split the association phase into the candidate test, the row pass and the row sums (align
// only: single passes sum in the row pass).
void launch_association(Handle *h, BatchHost *bh, const KParams &K, bool align = false, const cudaEvent_t *ev = nullptr) {
  BatchDev &B = bh->B;
  mark(h, ev, 0);
  k_transform<<<std::max(bh->xform_blocks, 1), 256, 0, h->stream>>>(B);
  mark(h, ev, 1);
  if (bh->cand_blocks > 0) {
    bh->fn.cand<<<bh->cand_blocks, 32 * kCandWarps, 0, h->stream>>>(B, K);
    h->launches++;
  }
  mark(h, ev, 5);
  const RowsFn *rows = bh->ordered ? bh->fn.ordered_rows : bh->fn.rows;
  const int split = bh->split_rows ? 1 : 0, blocks = std::max(B.total_rblocks, 1);
  if (split) {
    rows[ROWS_LIGHT]<<<blocks, 32 * kRowWarps, 0, h->stream>>>(B, K, 1);
    h->launches++;
  }
  rows[ROWS_ALL]<<<bh->rows_blocks, 32 * kRowWarps, 0, h->stream>>>(B, K, split);
  h->launches += 2;
  if (split && !align) {
    k_rows_total<<<B.npairs, 32 * kRowWarps, 0, h->stream>>>(B);
    h->launches++;
  }
  mark(h, ev, 6);
  if (align) {
    mark(h, ev, 2);
    k_gradient<<<std::max(B.total_sblocks, 1), kStepThreads, 0, h->stream>>>(B, K);
    h->launches++;
  }
  mark(h, ev, 3);
}

void launch_iteration(Handle *h, BatchHost *bh, const KParams &K, const cudaEvent_t *ev = nullptr) {
  launch_association(h, bh, K, true, ev);
  // Four lanes a row take fewer instructions per entry (lane t adds term t, and there are four);
  // eight lanes keep the SMs busy when the rows are few.
  (bh->few_rows ? k_step<8> : k_step<4>)<<<std::max(bh->B.total_sblocks, 1), kStepThreads, 0, h->stream>>>(bh->B, K);
  mark(h, ev, 4);
  h->launches += 1;
}

// What a captured launch sequence of a batch depends on.
void append_launch_key(const Handle *h, const BatchHost &bh, const KParams &K, std::vector<unsigned char> *key) {
  auto add = [&](const void *p, size_t n) {
    const unsigned char *c = static_cast<const unsigned char *>(p);
    key->insert(key->end(), c, c + n);
  };
  add(&bh.B, sizeof(bh.B));
  add(&K, sizeof(K));
  add(&bh.fn, sizeof(bh.fn));
  add(&bh.cand_blocks, sizeof(bh.cand_blocks));
  add(&bh.xform_blocks, sizeof(bh.xform_blocks));
  add(&bh.split_rows, sizeof(bh.split_rows));
  add(&bh.rows_blocks, sizeof(bh.rows_blocks));
  add(&bh.few_rows, sizeof(bh.few_rows));
  add(&h->stream, sizeof(h->stream));
}

int read_pairs(Handle *h, BatchHost *bh) {
  CVO_CUDA_TRY(h, cudaMemcpyAsync(bh->pairs.data(), bh->B.pairs, sizeof(PairDev) * bh->B.npairs,
                                  cudaMemcpyDeviceToHost, h->stream));
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  return 0;
}

int check_err(Handle *h, BatchHost *bh) {
  int e = 0;
  CVO_CUDA_TRY(h, cudaMemcpyAsync(&e, bh->B.err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  return e ? e : 0;
}

// Exports the association of pair p into per-row CSR on the host (rows =
// original source indices, columns ascending).
int export_pair(Handle *h, BatchHost *bh, int p, DevCloud *src, std::vector<int> *rowptr, std::vector<int> *cols,
                std::vector<float> *vals) {
  const PairDev &P = bh->pairs[p];
  if (P.n == 0 || P.m == 0) {      // nothing was associated
    rowptr->assign((size_t)P.n + 1, 0);
    cols->clear();
    vals->clear();
    return 0;
  }
  if (int rc = csr_to_host(h, P.n, P.nnz_row, src->sperm, P.ld, P.A_j, P.A_v, rowptr, cols, vals)) return rc;
  if (!bh->ordered) return 0;
  // rows in the order of the lattice: by column
  std::vector<std::pair<int, float>> tmp;
  for (int i = 0; i < P.n; i++) {
    const int o = (*rowptr)[i], z = (*rowptr)[i + 1] - o;
    tmp.resize(z);
    for (int k = 0; k < z; k++) tmp[k] = {(*cols)[o + k], (*vals)[o + k]};
    std::sort(tmp.begin(), tmp.end(), [](const std::pair<int, float> &a, const std::pair<int, float> &b) { return a.first < b.first; });
    for (int k = 0; k < z; k++) { (*cols)[o + k] = tmp[k].first; (*vals)[o + k] = tmp[k].second; }
  }
  return 0;
}

}  // namespace

// Only the kept entries cross to the host, in place: copying whole ELL rows and laying out the
// CSR there took most of an export.
int csr_to_host(Handle *h, int n, const int *nnz, const int *perm, int ld, const int *ell_j, const float *ell_v,
                std::vector<int> *rowptr, std::vector<int> *col, std::vector<float> *val) {
  rowptr->assign((size_t)n + 1, 0);
  col->clear();
  val->clear();
  if (n == 0) return 0;
  const size_t scr = scan_scratch_ints(n + 1);
  int *buf = nullptr, *out = nullptr;
  CVO_CUDA_TRY(h, cudaMallocAsync((void **)&buf, sizeof(int) * (2 * (size_t)(n + 1) + scr), h->stream));
  int *count = buf, *start = buf + n + 1;
  k_csr_counts<<<(n + 255) / 256, 256, 0, h->stream>>>(n, nnz, perm, count);
  exclusive_scan_int(h, count, start, n + 1, start + n + 1, (int)scr);
  h->launches++;
  cudaError_t e = cudaMemcpyAsync(rowptr->data(), start, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  const size_t total = e == cudaSuccess ? (*rowptr)[n] : 0;
  if (total > 0) e = cudaMallocAsync((void **)&out, sizeof(int) * 2 * total, h->stream);
  if (e == cudaSuccess && total > 0) {
    float *out_v = reinterpret_cast<float *>(out + total);
    k_csr_rows<<<(n + 3) / 4, 128, 0, h->stream>>>(n, nnz, perm, ld, ell_j, ell_v, start, out, out_v);
    h->launches++;
    col->resize(total);
    val->resize(total);
    e = cudaMemcpyAsync(col->data(), out, sizeof(int) * total, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(val->data(), out_v, sizeof(float) * total, cudaMemcpyDeviceToHost, h->stream);
  }
  if (out) cudaFreeAsync(out, h->stream);
  cudaFreeAsync(buf, h->stream);
  const cudaError_t es = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = es;
  return e == cudaSuccess ? 0 : set_cuda_error(h, e, "association export");
}

// Runs the align loop for every pair of the batch until all pairs stop.
int run_align_batch(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                    const std::vector<float> &T_init, BatchResult *res, double *secs, bool export_assoc,
                    std::vector<std::vector<int>> *a_rows, std::vector<std::vector<int>> *a_cols,
                    std::vector<std::vector<float>> *a_vals) {
  NvtxRange nvtx_range("align_batch");
  const int np = (int)srcs.size();
  if (np == 0) return 0;
  KParams K = make_kparams(h->params);
  if (K.indicator_window_size > kMaxIndicatorWindow || K.indicator_window_size < 1) return CVO_ERR_UNSUPPORTED;
  int capmax = std::max(h->params.nearest_neighbors_max, 0);
  BatchHost bh;
  std::vector<float> ell0(np, h->params.ell_init);
  int rc = build_batch(h, K, srcs, tgts, T_init, MODE_ALIGN, capmax, ell0, &bh);
  if (rc) return rc;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, h->stream);
  // capture one chunk of iterations as a CUDA graph and relaunch it; without profiling
  // events the instantiated graph is kept in the workspace and reused by a later batch
  // whose launch parameters are byte-identical
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  long long before = h->launches;
  // with profiling on, every kernel launch of the chunk is bracketed by
  // event-record nodes of the graph
  constexpr int kEv = 7;
  std::vector<cudaEvent_t> pev;
  std::vector<unsigned char> key;
  append_launch_key(h, bh, K, &key);
  Workspace *ws = h->ws;
  const bool reuse = !h->prof.on && ws->align_exec && ws->align_key == key;
  long long per_chunk = 0;
  if (reuse) {
    exec = ws->align_exec;
    per_chunk = ws->align_per_chunk;
  } else {
    if (h->prof.on) {
      pev.resize(kEv * kChunk);
      for (auto &e : pev) cudaEventCreate(&e);
    }
    CVO_CUDA_TRY(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    for (int it = 0; it < kChunk; it++) launch_iteration(h, &bh, K, h->prof.on ? &pev[kEv * it] : nullptr);
    CVO_CUDA_TRY(h, cudaStreamEndCapture(h->stream, &graph));
    per_chunk = h->launches - before;
    h->launches = before;
    CVO_CUDA_TRY(h, cudaGraphInstantiate(&exec, graph, 0));
    cudaGraphDestroy(graph);
    graph = nullptr;
    if (!h->prof.on) {
      if (ws->align_exec) cudaGraphExecDestroy(ws->align_exec);
      ws->align_exec = exec;
      ws->align_key = key;
      ws->align_per_chunk = per_chunk;
    }
  }
  int *active_h = h->ws->pinned;
  long long max_chunks = (long long)h->params.MAX_ITER / kChunk + 2;
  long long iters_seen = 0;
  for (long long ch = 0; ch < max_chunks; ch++) {
    CVO_CUDA_TRY(h, cudaGraphLaunch(exec, h->stream));
    h->launches += per_chunk;
    CVO_CUDA_TRY(h, cudaMemcpyAsync(active_h, bh.B.active, 2 * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    if (h->prof.on) {
      // active_h[1]: iterations (so far) that started with at least one active pair
      long long act = active_h[1];
      for (int it = 0; it < kChunk; it++) {
        if (ch * kChunk + it >= act) break;
        for (int k = 0; k < 4; k++) {
          float ms = 0.f;
          if (cudaEventElapsedTime(&ms, pev[kEv * it + k], pev[kEv * it + k + 1]) == cudaSuccess) {
            h->prof.kernel_ms[k] += ms;
            h->prof.kernel_ms[4] += ms;
          }
        }
        // association phase: candidate test (ev 1 -> 5), row pass (5 -> 6), nothing (6 -> 2)
        const int split[4] = {1, 5, 6, 2};
        for (int k = 0; k < 3; k++) {
          float ms = 0.f;
          if (cudaEventElapsedTime(&ms, pev[kEv * it + split[k]], pev[kEv * it + split[k + 1]]) == cudaSuccess)
            h->prof.assoc_split_ms[k] += ms;
        }
        h->prof.assoc_launches++;
      }
      iters_seen = act;
    }
    if (*active_h <= 0) break;
  }
  if (h->prof.on) {
    double bytes = 0;
    CVO_CUDA_TRY(h, cudaMemcpyAsync(&bytes, bh.B.assoc_bytes, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    h->prof.assoc_bytes += bytes;
    h->prof.iterations += iters_seen;
    h->prof.assoc_ms = h->prof.kernel_ms[1];
    for (auto &e : pev) cudaEventDestroy(e);
  }
  cudaEventRecord(e1, h->stream);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (exec != ws->align_exec) cudaGraphExecDestroy(exec);   // profiled graphs are not kept
  if (secs) *secs = ms / 1000.0;
  if ((rc = check_err(h, &bh))) return rc;
  if ((rc = read_pairs(h, &bh))) return rc;
  res->T_out.assign(16 * np, 0.f);
  res->ret.assign(np, 0);
  res->iters.assign(np, 0);
  res->asum.assign(np, 0.0);
  res->nnz.assign(np, 0);
  for (int p = 0; p < np; p++) {
    PairDev &P = bh.pairs[p];
    float *T = &res->T_out[16 * p];
    for (int r = 0; r < 3; r++) {
      for (int c = 0; c < 3; c++) T[c * 4 + r] = P.R[3 * c + r];
      float a = P.R[r] * P.T[0], b = P.R[3 + r] * P.T[1], c = P.R[6 + r] * P.T[2];
      T[12 + r] = -((a + b) + c);
    }
    T[15] = 1.f;
    res->ret[p] = P.ret;
    res->iters[p] = P.iter;
    res->asum[p] = P.asum;
    res->nnz[p] = P.nnz_sum;
    if (srcs[p]->n == 0 || tgts[p]->n == 0) {
      for (int t = 0; t < 16; t++) T[t] = (t % 5 == 0) ? 1.f : 0.f;
      for (int r = 0; r < 3; r++) { for (int c = 0; c < 3; c++) T[c * 4 + r] = T_init[16 * p + r * 4 + c]; }
    }
  }
  if (export_assoc && a_rows) {
    a_rows->resize(np); a_cols->resize(np); a_vals->resize(np);
    for (int p = 0; p < np; p++)
      if ((rc = export_pair(h, &bh, p, srcs[p], &(*a_rows)[p], &(*a_cols)[p], &(*a_vals)[p]))) return rc;
  }
  return 0;
}

// One association pass (no iteration) of one source/target pair under each of
// the given poses (inner_product_impl, src/cvo/CvoGPU.cu:1673-1732).
int run_inner_product_pairs(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                            const std::vector<float> &T, float ell, int cap, std::vector<double> *asum) {
  NvtxRange nvtx_range("inner_product_pairs");
  const int np = (int)srcs.size();
  asum->assign(np, 0.0);
  if (np == 0) return 0;
  KParams K = make_kparams(h->params);
  BatchHost bh;
  std::vector<float> ell0(np, ell);
  int rc = build_batch(h, K, srcs, tgts, T, MODE_IP, std::max(cap, 0), ell0, &bh);
  if (rc) return rc;
  launch_association(h, &bh, K);
  if ((rc = check_err(h, &bh))) return rc;
  if ((rc = read_pairs(h, &bh))) return rc;
  for (int p = 0; p < np; p++) (*asum)[p] = bh.pairs[p].asum;
  return 0;
}

int autotune_association(Handle *h, DevCloud *src, DevCloud *tgt, const float T[16], float ell, int reps,
                         std::vector<TuneConfig> *configs, std::vector<float> *ms, int *best) {
  NvtxRange nvtx_range("autotune");
  // candidates: 1/4 .. 3 times the default division of the targets among warps, then 4 to
  // 12 work items per SM with the fastest one's divisors
  const float div_r[] = {2.f, 3.f, 4.f, 6.f};
  const float div_ext[] = {4.f, 8.f, 16.f};
  configs->clear();
  for (float a : div_r)
    for (float b : div_ext) {
      TuneConfig c;
      c.cell_div_r = a;
      c.cell_div_ext = b;
      configs->push_back(c);
    }
  ms->assign(configs->size(), INFINITY);
  if (src->n == 0 || tgt->n == 0) return CVO_ERR_EMPTY_CLOUD;
  reps = std::max(1, reps);
  std::vector<float> Tv(T, T + 16);
  const int cap = h->params.nearest_neighbors_max;
  cudaEvent_t e0, e1;
  CVO_CUDA_TRY(h, cudaEventCreate(&e0));
  CVO_CUDA_TRY(h, cudaEventCreate(&e1));
  int rc = 0, bi = 0;
  for (size_t k = 0; k < configs->size() && !rc; k++) {
    h->tune_force = &(*configs)[k];
    std::vector<double> asum;
    rc = run_inner_product_pairs(h, {src}, {tgt}, Tv, ell, cap, &asum);   // sizes the workspace
    std::vector<float> t;
    for (int r = 0; r < reps && !rc; r++) {
      cudaEventRecord(e0, h->stream);
      rc = run_inner_product_pairs(h, {src}, {tgt}, Tv, ell, cap, &asum);
      cudaEventRecord(e1, h->stream);
      cudaEventSynchronize(e1);
      float dt = 0.f;
      cudaEventElapsedTime(&dt, e0, e1);
      t.push_back(dt);
    }
    if (!rc) {
      std::sort(t.begin(), t.end());
      (*ms)[k] = t[t.size() / 2];
      if ((*ms)[k] < (*ms)[bi]) bi = (int)k;
    }
  }
  // then the launch: few work items per SM (less setup, but tiles of uneven cost even out less)
  const int per_sm_max = 4;
  for (int bps = 1; bps < per_sm_max && !rc; bps++) {
    TuneConfig c = (*configs)[bi];
    c.blocks_per_sm = bps;
    configs->push_back(c);
    ms->push_back(INFINITY);
    const size_t k = configs->size() - 1;
    h->tune_force = &(*configs)[k];
    std::vector<double> asum;
    std::vector<float> t;
    for (int r = 0; r < reps && !rc; r++) {
      cudaEventRecord(e0, h->stream);
      rc = run_inner_product_pairs(h, {src}, {tgt}, Tv, ell, cap, &asum);
      cudaEventRecord(e1, h->stream);
      cudaEventSynchronize(e1);
      float dt = 0.f;
      cudaEventElapsedTime(&dt, e0, e1);
      t.push_back(dt);
    }
    if (!rc) {
      std::sort(t.begin(), t.end());
      (*ms)[k] = t[t.size() / 2];
      if ((*ms)[k] < (*ms)[bi]) bi = (int)k;
    }
  }
  h->tune_force = nullptr;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  TuneConfig cell = (*configs)[bi];
  h->tuned_bps[tune_key(src->F, src->C, tune_items(src->n))] = cell.blocks_per_sm;
  cell.blocks_per_sm = 0;
  h->tuned[tune_key(src->F, src->C, src->n)] = cell;
  if (best) *best = bi;
  return CVO_OK;
}

int run_inner_product_batch(Handle *h, DevCloud *src, DevCloud *tgt, const std::vector<float> &T, float ell, int cap,
                            std::vector<double> *asum, std::vector<long long> *nnz, bool export_assoc,
                            std::vector<int> *a_rowptr, std::vector<int> *a_cols, std::vector<float> *a_vals) {
  NvtxRange nvtx_range("inner_product_batch");
  const int np = (int)(T.size() / 16);
  KParams K = make_kparams(h->params);
  BatchHost bh;
  std::vector<DevCloud *> srcs(np, src), tgts(np, tgt);
  std::vector<float> ell0(np, ell);
  int rc = build_batch(h, K, srcs, tgts, T, export_assoc ? MODE_EXPORT : MODE_IP, std::max(cap, 0), ell0, &bh);
  if (rc) return rc;
  launch_association(h, &bh, K);
  if ((rc = check_err(h, &bh))) return rc;
  if ((rc = read_pairs(h, &bh))) return rc;
  asum->assign(np, 0.0);
  nnz->assign(np, 0);
  for (int p = 0; p < np; p++) { (*asum)[p] = bh.pairs[p].asum; (*nnz)[p] = bh.pairs[p].nnz_sum; }
  if (export_assoc && np == 1)
    if ((rc = export_pair(h, &bh, 0, src, a_rowptr, a_cols, a_vals))) return rc;
  return 0;
}

AssocGraph::~AssocGraph() {
  if (exec) cudaGraphExecDestroy(exec);
  cudaFreeHost(pin_in);
  cudaFreeHost(pin_out);
  cudaFreeHost(pin_err);
}

namespace {

// Uploads bh's pair records, runs the association and reads the records and the error
// word back, through g's graph (captured anew when the launch parameters changed).
int replay_association(Handle *h, BatchHost *bh, const KParams &K, AssocGraph *g) {
  const int np = bh->B.npairs;
  if (g->pin_pairs < np) {
    if (g->exec) cudaGraphExecDestroy(g->exec);
    g->exec = nullptr;
    cudaFreeHost(g->pin_in);
    cudaFreeHost(g->pin_out);
    cudaFreeHost(g->pin_err);
    g->pin_in = g->pin_out = nullptr;
    g->pin_err = nullptr;
    g->pin_pairs = 0;
    if (cudaMallocHost((void **)&g->pin_in, sizeof(PairDev) * np) != cudaSuccess ||
        cudaMallocHost((void **)&g->pin_out, sizeof(PairDev) * np) != cudaSuccess ||
        cudaMallocHost((void **)&g->pin_err, sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      return CVO_ERR_OUT_OF_MEMORY;
    }
    g->pin_pairs = np;
  }
  std::vector<unsigned char> key;
  append_launch_key(h, *bh, K, &key);
  key.insert(key.end(), reinterpret_cast<const unsigned char *>(&g->pin_in),
             reinterpret_cast<const unsigned char *>(&g->pin_in) + sizeof(g->pin_in));
  if (!g->exec || g->key != key) {
    if (g->exec) cudaGraphExecDestroy(g->exec);
    g->exec = nullptr;
    const long long before = h->launches;
    CVO_CUDA_TRY(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t e1 = cudaMemcpyAsync(bh->B.pairs, g->pin_in, sizeof(PairDev) * np, cudaMemcpyHostToDevice, h->stream);
    launch_association(h, bh, K);
    cudaError_t e2 = cudaMemcpyAsync(g->pin_out, bh->B.pairs, sizeof(PairDev) * np, cudaMemcpyDeviceToHost, h->stream);
    cudaError_t e3 = cudaMemcpyAsync(g->pin_err, bh->B.err, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
    cudaGraph_t graph = nullptr;
    cudaError_t e4 = cudaStreamEndCapture(h->stream, &graph);
    g->launches = h->launches - before;
    h->launches = before;
    cudaError_t e5 = cudaSuccess;
    if (e1 == cudaSuccess && e2 == cudaSuccess && e3 == cudaSuccess && e4 == cudaSuccess)
      e5 = cudaGraphInstantiate(&g->exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    for (cudaError_t e : {e1, e2, e3, e4, e5})
      if (e != cudaSuccess) {
        g->exec = nullptr;
        return set_cuda_error(h, e, "association graph capture");
      }
    g->key = key;
  }
  memcpy(g->pin_in, bh->pairs.data(), sizeof(PairDev) * np);
  CVO_CUDA_TRY(h, cudaGraphLaunch(g->exec, h->stream));
  h->launches += g->launches;
  CVO_CUDA_TRY(h, cudaStreamSynchronize(h->stream));
  if (*g->pin_err) return *g->pin_err;
  memcpy(bh->pairs.data(), g->pin_out, sizeof(PairDev) * np);
  return 0;
}

}  // namespace

int run_association_edges(Handle *h, const std::vector<DevCloud *> &srcs, const std::vector<DevCloud *> &tgts,
                          const std::vector<const float4 *> &src_world, const std::vector<float> &src_world_norm,
                          const std::vector<float> &tgt_pose, const std::vector<float> &ells,
                          const std::vector<int> &caps, int capmax, std::vector<EdgeAssoc> *out,
                          const KParams *kparams, AssocGraph *graph) {
  NvtxRange nvtx_range("association_edges");
  const int ne = (int)srcs.size();
  out->assign(ne, EdgeAssoc());
  if (ne == 0) return 0;
  KParams K = kparams ? *kparams : make_kparams(h->params);
  std::vector<float> Tid(16 * (size_t)ne, 0.f);
  for (int e = 0; e < ne; e++) Tid[16 * e] = Tid[16 * e + 5] = Tid[16 * e + 10] = Tid[16 * e + 15] = 1.f;
  BatchHost bh;
  int rc = build_batch(h, K, srcs, tgts, Tid, MODE_EDGES, capmax, ells, &bh);
  if (rc) return rc;
  for (int e = 0; e < ne; e++) {
    PairDev &P = bh.pairs[e];
    if (P.done) continue;
    P.xs = src_world[e];
    P.cap = caps[e];
    const float *Q = &tgt_pose[12 * e];
    for (int r = 0; r < 3; r++) {
      for (int c = 0; c < 3; c++) P.Ri[3 * r + c] = Q[4 * r + c];   // target moved by its own pose
      P.Ti[r] = Q[4 * r + 3];
    }
    // inverse (only used to place the query box in the target's own frame)
    for (int r = 0; r < 3; r++)
      for (int c = 0; c < 3; c++) P.R[3 * r + c] = Q[4 * c + r];
    for (int r = 0; r < 3; r++) P.T[r] = -(P.R[3 * r] * Q[3] + P.R[3 * r + 1] * Q[7] + P.R[3 * r + 2] * Q[11]);
    P.level = level_for(P, host_radius(K, ells[e], src_world_norm[e]));
  }
  if (graph && !h->prof.on) {
    if ((rc = replay_association(h, &bh, K, graph))) return rc;
  } else {
    CVO_CUDA_TRY(h, cudaMemcpyAsync(bh.B.pairs, bh.pairs.data(), sizeof(PairDev) * ne, cudaMemcpyHostToDevice,
                                    h->stream));
    launch_association(h, &bh, K);
    if ((rc = check_err(h, &bh))) return rc;
    if ((rc = read_pairs(h, &bh))) return rc;
  }
  for (int e = 0; e < ne; e++) {
    const PairDev &P = bh.pairs[e];
    EdgeAssoc &A = (*out)[e];
    A.A_j = P.A_j; A.A_v = P.A_v; A.nnz_row = P.nnz_row;
    A.ld = P.ld;
    A.n = P.n; A.m = P.m;
    A.nnz = P.done ? 0 : P.nnz_sum;
    A.max_row = P.done ? 0 : P.max_row;
  }
  return 0;
}

int set_cuda_error(Handle *h, cudaError_t e, const char *where) {
  if (h) {
    h->last_error = std::string(where) + ": " + cudaGetErrorString(e);
  }
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? CVO_ERR_OUT_OF_MEMORY : CVO_ERR_CUDA;
}

}  // namespace cvo_gb
