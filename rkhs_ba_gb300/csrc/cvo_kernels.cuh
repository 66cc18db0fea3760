// cvo_kernels.cuh -- association kernels of the batched CVO engine.
//
// One iteration of the reference's align loop (src/cvo/CvoGPU.cu:1303-1433) is a
// fixed sequence of launches over every active pair of a batch:
//   k_transform  target transform y' = R^T (y - T)            (CvoGPU_impl.cu:32-83)
//   k_cand       candidates: source tiles against target groups by bounding boxes in
//                position and colour, then a tensor-core test of the 32 x 32 pairs of
//                the groups that remain; one bit per pair that may be kept
//   k_rows       each row's candidates in ascending target index: exact kernel value,
//                threshold, the first cap kept ones to the ELL row    (CvoGPU.cu:951-1099)
//   k_gradient   gradient sums of the rows and of the pair (CvoGPU.cu:2001-2120);
//                single passes sum in k_rows instead
//   k_step       Taylor step-size terms over the ELL rows; the last block of each pair
//                runs the scalar tail of the iteration: cubic roots, step clamp,
//                Exp_SEK3 pose update, SE(3) distance, lengthscale schedule, cap update
//                                                               (CvoGPU.cu:333-544, 547-665, 1339-1433)
#pragma once
#include <climits>
#include <cuda_fp16.h>
#include "cvo_device.cuh"

namespace cvo_gb {

enum { MODE_ALIGN = 0, MODE_IP = 1, MODE_EXPORT = 2, MODE_EDGES = 3 };
constexpr int kStepThreads = 256;
constexpr int kUnitRows = 32;           // fewest rows of a block of the gradient and step kernels
constexpr int kPartStride = 12;

// ------------------------------------------------------------ pair value
// Kernel value of one (source, target) pair with the semantics of
// fill_in_A_mat_gpu (src/cvo/CvoGPU.cu:996-1075).  `pre` is the lane's
// participation; returns whether the pair is kept and its value in a.
// All lanes of the warp must call it together.
template <int FCH, int LCH, bool GT>
__device__ __forceinline__ bool eval_pair(const KParams &K, int F, int C, bool pre, float l, float d2t, float inv2l2,
                                          const float4 &x, const float4 (&xf)[FCH > 0 ? FCH : 1],
                                          const float4 *xl, float2 xg, const float4 &y,
                                          const float4 (&yf)[FCH > 0 ? FCH : 1], const float4 *ylp, float2 yg, float &a) {
  bool pass = pre;
  float d2 = 0.f;
  if (K.use_geo) {
    d2 = sqdist3(y.x, y.y, y.z, x.x, x.y, x.z);
    pass = pass && (d2 < d2t);
  }
  if (!__any_sync(FULLMASK, pass)) return false;
  float geo = 1.f;
  if (GT) {
    float n2a = fa(fm(xg.x, xg.x), fm(xg.y, xg.y));
    float n2b = fa(fm(yg.x, yg.x), fm(yg.y, yg.y));
    float dab = fa(fm(xg.x, yg.x), fm(xg.y, yg.y));
    geo = __fdiv_rn(fm(dab, dab), fm(n2a, n2b));
    pass = pass && !((double)geo < 0.01);
  }
  float d2c = 0.f;
  if (FCH > 0 && K.use_int) {
#pragma unroll
    for (int q = 0; q < FCH; q++) {
      float av[4] = {xf[q].x, xf[q].y, xf[q].z, xf[q].w};
      float bv[4] = {yf[q].x, yf[q].y, yf[q].z, yf[q].w};
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (4 * q + r < F) { float t = fs(av[r], bv[r]); d2c = fa(d2c, fm(t, t)); }
    }
    pass = pass && (d2c < K.d2_c_thres);
  } else if (K.use_int) {
    pass = pass && (d2c < K.d2_c_thres);
  }
  float d2s = 0.f;
  if (LCH > 0 && K.use_sem) {
#pragma unroll
    for (int q = 0; q < LCH; q++) {
      float4 yl = pass ? __ldg(ylp + q) : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 xq = xl[q];
      float av[4] = {xq.x, xq.y, xq.z, xq.w};
      float bv[4] = {yl.x, yl.y, yl.z, yl.w};
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (4 * q + r < C) { float t = fs(av[r], bv[r]); d2s = fa(d2s, fm(t, t)); }
    }
    pass = pass && (d2s < K.d2_s_thres);
  } else if (K.use_sem) {
    pass = pass && (d2s < K.d2_s_thres);
  }
  if (!__any_sync(FULLMASK, pass)) return false;
  // fast FP32 value
  float kf = K.use_geo ? fm(K.sigma2, __expf(fm(-d2, inv2l2))) : 1.f;
  float ckf = K.use_int ? fm(K.c_sigma2, __expf(fm(-d2c, K.inv2c2))) : 1.f;
  float skf = K.use_sem ? fm(K.s_sigma_sq, __expf(fm(-d2s, __frcp_rn(fm(fm(2.f, K.s_ell), K.s_ell))))) : 1.f;
  float af = fm(fm(fm(fm(ckf, kf), skf), geo), K.val_scale);
  if (pass && fabsf(fs(af, K.sp_thres)) <= kBand * K.sp_thres) af = exact_value(K, l, d2, d2c, d2s, geo);
  a = af;
  return pass && (af > K.sp_thres);
}

// Per-source-point kernel constants.
struct RowConst {
  float l, d2t, inv2l2;
};

__device__ __forceinline__ RowConst row_const(const KParams &K, float ell, float norm) {
  RowConst rc;
  rc.l = range_ell(ell, norm);
  rc.d2t = K.use_geo ? geo_d2_thres(rc.l, K.log_geo) : INFINITY;
  rc.inv2l2 = __frcp_rn(fm(fm(2.f, rc.l), rc.l));
  return rc;
}

// ---------------------------------------------------------- candidate test
// A kept pair satisfies  u = g_s |x - y|^2 + c |xc - yc|^2 < tau  with
// g_s = 1/(2 l_s^2), c = 1/(2 c_ell^2), tau = ln(sigma^2 c_sigma^2 s_sigma^2 / sp_thres)
// (+ slack): the kernel value is at most the product of the three scales times
// exp(-u), and the geometric-type factor is at most 1.  With g the smallest g_s of a
// tile of 32 source rows, a = [sqrt(g) (x - p), sqrt(c) (xc - q)] and b likewise for a
// candidate (p, q: a point near the tile), u >= |a - b|^2.  a and b are rounded to
// f16 (a^, b^); then |a^ - b^| <= |a - b| + 2^-11 (|a| + |b|), and a kept pair has
// |b| <= |a| + sqrt(tau), so with A the largest |a^| of the tile the test
//   |a^ - b^|^2 < (sqrt(tau) + 2^-11 (2 A + sqrt(tau)))^2 + rounding
// never rejects a kept pair.  |a^ - b^|^2 minus that bound is one 16-wide product:
//   [-2 a^ (11) | (|a^|^2 - bound) hi | lo | 1 | 1 | 0] . [b^ | 1 | 1 | |b^|^2 hi | lo | 0]
// (squares split into two f16), one mma.sync.m16n8k16 per 16 x 8 pairs, and the sign
// of the accumulator is the answer.  The bound is within 1-2 % of tau for tiles a few
// lengthscales wide.  Only candidates go through the exact per-pair arithmetic
// (eval_pair), so the kernel matrix does not depend on the test.
// The same accumulators answer the opposite question: |a^ - b^|^2 below
//   (sqrt(tau') - 2^-11 (2 A + sqrt(tau)))^2 - rounding,   tau' = K.sure_tau g_min / g_max,
// means that the pair is kept (no term but position and colour, and u below the thresholds of
// both: K.sure_tau > 0).  k_cand counts such pairs of dense groups, see k_rows.
constexpr float kCandWide = 200.f;      // largest |a^| the f16 squares serve
constexpr float kCandFar = 60000.f;     // |b^|^2 beyond which a candidate is rejected outright
// cand_cnt's x: entries (a row has at most 2^17, one per target group), then the pairs that are
// surely kept, as far as they were counted
constexpr int kSureShift = 18, kSureMost = (1 << 13) - 1;

__device__ __forceinline__ float f4_at(const float4 &v, int i) {
  return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

__device__ __forceinline__ uint32_t pack_h2(__half a, __half b) {
  return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}

__device__ __forceinline__ void ldsm_x4(const void *p, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_addr(p))
               : "memory");
}

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %10, %10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c));
}

// The operand of one point: scaled coordinates v[11] rounded to f16, and the four
// square / one columns.  Planes 0 and 1 hold k 0-7 and 8-15 (16 bytes each).
__device__ __forceinline__ void cand_store(const __half (&v)[11], __half c11, __half c12, __half c13, __half c14,
                                           uint4 (*pl)[32], int idx) {
  pl[0][idx] = make_uint4(pack_h2(v[0], v[1]), pack_h2(v[2], v[3]), pack_h2(v[4], v[5]), pack_h2(v[6], v[7]));
  pl[1][idx] = make_uint4(pack_h2(v[8], v[9]), pack_h2(v[10], c11), pack_h2(c12, c13), pack_h2(c14, __float2half_rn(0.f)));
}

// Scaled coordinates of a point relative to the tile's centre.
template <int FCH>
__device__ __forceinline__ void cand_coords(float (&v)[11], const float4 &y, const float4 (&yf)[FCH > 0 ? FCH : 1],
                                            const float (&pc)[3], const float (&fc)[8], float sg, float sc) {
  v[0] = (y.x - pc[0]) * sg;
  v[1] = (y.y - pc[1]) * sg;
  v[2] = (y.z - pc[2]) * sg;
#pragma unroll
  for (int f = 0; f < 8; f++) v[3 + f] = FCH * 4 > f ? (f4_at(yf[FCH > 0 ? (f >> 2) % FCH : 0], f & 3) - fc[f]) * sc : 0.f;
}

// Column of the 32 x 32 tile that answers for bit p of a row's mask: the sign bits of
// the accumulators are shifted together in this order (see k_cand), so candidate p is
// staged in column cand_col(p).
__device__ __forceinline__ int cand_col(int p) {
  const int q = 7 - (p & 7);
  return 8 * (q >> 1) + 2 * (p >> 3) + (q & 1);
}

// Squared distance of the intervals [alo, ahi] and [blo, bhi] (0 if they meet).
__device__ __forceinline__ float gap2(float alo, float ahi, float blo, float bhi) {
  const float d = fmaxf(fmaxf(blo - ahi, alo - bhi), 0.f);
  return d * d;
}

// Bounding boxes of groups (or of 32 groups): float4 planes of `count` entries each --
// position low, high, feature low (FCH chunks), feature high (FCH chunks).
// Whether some pair between the tile and box i may be kept.
template <int FCH>
__device__ __forceinline__ bool box_near(const float4 *box, int count, int i, const float (&qlo)[3], const float (&qhi)[3],
                                         const float (&flo)[8], const float (&fhi)[8], float g, float cw, float tau,
                                         float dc_max) {
  const float4 lo = __ldg(box + i), hi = __ldg(box + count + i);
  const float dp = gap2(qlo[0], qhi[0], lo.x, hi.x) + gap2(qlo[1], qhi[1], lo.y, hi.y) + gap2(qlo[2], qhi[2], lo.z, hi.z);
  float dc = 0.f;
#pragma unroll
  for (int q = 0; q < FCH; q++) {
    const float4 a = __ldg(box + (size_t)(2 + q) * count + i), b = __ldg(box + (size_t)(2 + FCH + q) * count + i);
    dc += gap2(flo[4 * q], fhi[4 * q], a.x, b.x) + gap2(flo[4 * q + 1], fhi[4 * q + 1], a.y, b.y) +
          gap2(flo[4 * q + 2], fhi[4 * q + 2], a.z, b.z) + gap2(flo[4 * q + 3], fhi[4 * q + 3], a.w, b.w);
  }
  // written so that a NaN bound keeps the group
  return !(g * dp + cw * dc > tau) && !(dc > dc_max);
}

// One warp per work item: a tile of 32 source rows (Morton order) and every S-th of the
// target's supergroups (32 groups of 32 points).  The warp tests the supergroups' boxes,
// then the groups' boxes of those near it (one box per lane), and runs the tensor-core
// test on the groups that remain.  A row's answer for a group is a 32-bit mask, appended
// to the row's entries {group, mask} of this split; k_rows puts the entries in index
// order, so neither the number of splits nor their order matters.
// Bounds: issue (box tests 25-45 instructions per 32 groups, 70 to stage a group's 32
// candidates, 60 for the product and its mask).  Boxes in position and colour leave
// 3-14 % of all 32 x 32 tiles on the stereo scenes, four times fewer than boxes in
// position alone, which is why the cells of a position grid are not used here.
constexpr int kCandWarps = 4;

template <int FCH>
__global__ void __launch_bounds__(32 * kCandWarps, 4) k_cand(BatchDev B, KParams K) {
  __shared__ __align__(16) uint4 apl_all[kCandWarps][2][32];
  __shared__ __align__(16) uint4 bpl_all[kCandWarps][2][32];
  constexpr int FP = FCH > 0 ? FCH : 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint4(*apl)[32] = apl_all[w];
  uint4(*bpl)[32] = bpl_all[w];
  const int gw = blockIdx.x * kCandWarps + w;
  if (gw >= B.total_items) return;
  const int p = find_segment(B.item_off, B.npairs, gw);
  const PairDev *P = &B.pairs[p];
  if (P->done) return;
  const int S = P->splits, it = gw - B.item_off[p];
  const int tile = it / S, sp = it - tile * S;
  const int n = P->n, m = P->m;
  const int s = tile * 32 + lane;
  const bool valid = s < n;
  const int si = valid ? s : n - 1;      // spare lanes repeat the last row for the boxes
  const float4 x = __ldg(&P->xs[si]);
  float4 xf[FP];
#pragma unroll
  for (int q = 0; q < FP; q++)
    xf[q] = FCH > 0 ? __ldg(reinterpret_cast<const float4 *>(P->xf) + (size_t)si * FCH + q) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float tau = K.mma_tau;
  const float cw = K.use_int ? K.inv2c2 : 0.f;
  // the tile's smallest 1 / (2 l^2), and how far rounding can move a point between frames
  const float l = range_ell(P->ell, x.w);
  const float lmax = warp_fmax(l);
  const float g = K.use_geo ? 1.f / (2.f * lmax * lmax) : 0.f;
  const float Tn = fabsf(P->T[0]) + fabsf(P->T[1]) + fabsf(P->T[2]);
  const float xn = warp_fmax(sqrtf(x.x * x.x + x.y * x.y + x.z * x.z));
  const float slack = K.use_geo ? 4e-5f * (xn + Tn + lmax * sqrtf(2.f * fmaxf(tau, 0.f))) + 1e-6f : 0.f;
  // box of the rows' positions in the target's own frame (q = R x + T)
  const float *R = P->R;
  const float qx = fmaf(R[0], x.x, fmaf(R[1], x.y, fmaf(R[2], x.z, P->T[0])));
  const float qy = fmaf(R[3], x.x, fmaf(R[4], x.y, fmaf(R[5], x.z, P->T[1])));
  const float qz = fmaf(R[6], x.x, fmaf(R[7], x.y, fmaf(R[8], x.z, P->T[2])));
  const float qlo[3] = {warp_fmin(qx) - slack, warp_fmin(qy) - slack, warp_fmin(qz) - slack};
  const float qhi[3] = {warp_fmax(qx) + slack, warp_fmax(qy) + slack, warp_fmax(qz) + slack};
  // box of the rows' features (kept with the cloud) and the tile's centre
  float flo[8], fhi[8], fc[8];
#pragma unroll
  for (int f = 0; f < 8; f++) flo[f] = fhi[f] = fc[f] = 0.f;
  const int st = (n + 31) >> 5;
#pragma unroll
  for (int q = 0; q < FCH; q++) {
    const float4 a = __ldg(P->sbox + (size_t)(2 + q) * st + tile), b = __ldg(P->sbox + (size_t)(2 + FCH + q) * st + tile);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      flo[4 * q + r] = f4_at(a, r);
      fhi[4 * q + r] = f4_at(b, r);
      fc[4 * q + r] = 0.5f * (flo[4 * q + r] + fhi[4 * q + r]);
    }
  }
  const float pc[3] = {__shfl_sync(FULLMASK, x.x, 0), __shfl_sync(FULLMASK, x.y, 0), __shfl_sync(FULLMASK, x.z, 0)};
  const float sg = sqrtf(g), sc = sqrtf(cw);
  // the rows' operands
  bool wide, spread;
  float sure_at = INFINITY;      // accumulators below -sure_at are kept pairs
  {
    float v[11];
    cand_coords<FCH>(v, x, xf, pc, fc, sg, sc);
    __half h[11];
    float sa = 0.f;
#pragma unroll
    for (int k = 0; k < 11; k++) {
      h[k] = __float2half_rn(v[k]);
      const float r = __half2float(h[k]);
      sa = fmaf(r, r, sa);
      h[k] = __float2half_rn(-2.f * r);
    }
    const float A = sqrtf(warp_fmax(sa)), rt = sqrtf(fmaxf(tau, 0.f));
    wide = !(A <= kCandWide);
    const float lmin = -warp_fmax(-l), rs = K.use_geo ? lmin / lmax : 1.f;
    const float rv = sqrtf(fmaxf(K.sure_tau, 0.f)) * rs - 4.95e-4f * (2.f * A + rt) - 2e-6f;
    spread = K.use_geo && A > 3.f * rt;
    const float reach = 2.f * A + rt;
    const float rb = rt + 4.95e-4f * reach + 2e-6f;
    const float bound = rb * rb * 1.00001f + 4e-6f * reach * reach + 1e-6f;
    const float inner = rv * rv * 0.9999f - 4e-6f * reach * reach - 1e-6f;
    if (P->order_cap > 0 && K.sure_tau > 0.f && rv > 0.f && inner > 0.f) sure_at = bound - inner;
    const float d = valid ? sa - bound : kCandFar;
    const __half hi = __float2half_rn(d), one = __float2half_rn(1.f);
    cand_store(h, hi, __float2half_rn(d - __half2float(hi)), one, one, apl, lane);
  }
  __syncwarp();
  uint32_t af[2][4];
#pragma unroll
  for (int mm = 0; mm < 2; mm++)
    ldsm_x4(&apl[lane >> 4][16 * mm + (lane & 15)], af[mm][0], af[mm][1], af[mm][2], af[mm][3]);
  const float box_tau = tau * 1.0001f + 1e-5f, dc_max = K.use_int ? K.d2_c_thres * 1.0001f : INFINITY;
  const int caps = P->cap_split;
  uint2 *out = P->cand + (size_t)si * P->cand_pitch + (size_t)sp * caps;
  const int ng = P->groups, ns = (ng + 31) >> 5;
  int cnt = 0, cands = 0, sure = 0;
  const int my_col = cand_col(lane);
  const int src0 = 4 * (lane & 7);
  const uint32_t sel = (uint32_t)(lane >> 3) | ((uint32_t)((lane >> 3) + 4) << 4);
  const float4 *__restrict__ ycur = P->ycur;
  const float4 *__restrict__ tfs = reinterpret_cast<const float4 *>(P->tfs);
  // A tile much wider than the search radius (the Morton order jumps within it) has a box
  // that meets almost everything: such a tile also asks whether a box is near one of its rows.
  auto row_near = [&](const float4 *box, int count, int i) {
    const float4 lo = __ldg(box + i), hi = __ldg(box + count + i);
    const float d = gap2(qx - slack, qx + slack, lo.x, hi.x) + gap2(qy - slack, qy + slack, lo.y, hi.y) +
                    gap2(qz - slack, qz + slack, lo.z, hi.z);
    return __any_sync(FULLMASK, !(g * d > box_tau));
  };
  const int mine = sp < ns ? (ns - sp + S - 1) / S : 0;      // supergroups sp, sp + S, ...
  for (int u0 = 0; u0 < mine && tau > 0.f; u0 += 32) {
    const int su = sp + S * (u0 + lane);
    const bool snear = u0 + lane < mine && box_near<FCH>(P->tsup, ns, su, qlo, qhi, flo, fhi, g, cw, box_tau, dc_max);
    uint32_t sm = __ballot_sync(FULLMASK, snear);
    while (sm) {
      const int g0 = 32 * (sp + S * (u0 + __ffs(sm) - 1));
      sm &= sm - 1;
      if (spread && !row_near(P->tsup, ns, g0 >> 5)) continue;
      const bool gnear = g0 + lane < ng && box_near<FCH>(P->tbox, ng, g0 + lane, qlo, qhi, flo, fhi, g, cw, box_tau, dc_max);
      uint32_t gm = __ballot_sync(FULLMASK, gnear);
      if (spread)
        for (uint32_t left = gm; left; left &= left - 1) {
          const int k = __ffs(left) - 1;
          if (!row_near(P->tbox, ng, g0 + k)) gm &= ~(1u << k);
        }
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f), yf[FP];
#pragma unroll
      for (int q = 0; q < FP; q++) yf[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      auto load = [&](uint32_t mk) {      // the next group's candidates, in flight while this one is tested
        if (!mk) return;
        const int t = min(32 * (g0 + __ffs(mk) - 1) + lane, m - 1);
        y = __ldg(&ycur[t]);
#pragma unroll
        for (int q = 0; q < FCH; q++) yf[q] = __ldg(tfs + (size_t)t * FCH + q);
      };
      load(gm);
      while (gm) {
        const int gi = g0 + __ffs(gm) - 1;
        const bool has = 32 * gi + lane < m;
        uint32_t mask = 0;
        gm &= gm - 1;
        if (!wide) {
          float v[11];
          cand_coords<FCH>(v, y, yf, pc, fc, sg, sc);
          load(gm);
          __half h[11];
          float sb = 0.f;
#pragma unroll
          for (int k = 0; k < 11; k++) {
            h[k] = __float2half_rn(v[k]);
            const float r = __half2float(h[k]);
            sb = fmaf(r, r, sb);
          }
          const bool far = !has || !(sb <= kCandFar);
          const __half zero = __float2half_rn(0.f), one = __float2half_rn(1.f);
          if (far) {
#pragma unroll
            for (int k = 0; k < 11; k++) h[k] = zero;
            sb = kCandFar;
          }
          const __half hi = __float2half_rn(sb);
          __syncwarp();      // the previous group's operands have been read
          cand_store(h, one, one, hi, __float2half_rn(sb - __half2float(hi)), bpl, my_col);
          __syncwarp();
          uint32_t b0[4], b1[4];
          ldsm_x4(&bpl[(lane >> 3) & 1][8 * (lane >> 4) + (lane & 7)], b0[0], b0[1], b0[2], b0[3]);
          ldsm_x4(&bpl[(lane >> 3) & 1][16 + 8 * (lane >> 4) + (lane & 7)], b1[0], b1[1], b1[2], b1[3]);
          // signs of the accumulators plus `at`: byte 2 mm + hh of a lane's word holds its
          // columns of row 16 mm + 8 hh + lane / 4
          auto signs = [&](float at) {
            uint32_t wb[4];
#pragma unroll
            for (int mm = 0; mm < 2; mm++) {
              uint32_t w0 = 0, w1 = 0;
#pragma unroll
              for (int nn = 0; nn < 4; nn++) {
                float d[4];
                mma_16816(d, af[mm], nn < 2 ? b0[2 * nn] : b1[2 * nn - 4], nn < 2 ? b0[2 * nn + 1] : b1[2 * nn - 3], at);
                w0 = __funnelshift_l(__float_as_uint(d[0]), w0, 1);
                w0 = __funnelshift_l(__float_as_uint(d[1]), w0, 1);
                w1 = __funnelshift_l(__float_as_uint(d[2]), w1, 1);
                w1 = __funnelshift_l(__float_as_uint(d[3]), w1, 1);
              }
              wb[2 * mm] = w0;
              wb[2 * mm + 1] = w1;
            }
            return __byte_perm(__byte_perm(wb[0], wb[1], 0x0040), __byte_perm(wb[2], wb[3], 0x0040), 0x5410);
          };
          // the word of row `lane`: its 32 columns in the candidates' order
          auto row_mask = [&](uint32_t word) {
            uint32_t q4[4];
#pragma unroll
            for (int t = 0; t < 4; t++) q4[t] = __shfl_sync(FULLMASK, word, src0 + t);
            return __byte_perm(__byte_perm(q4[0], q4[1], sel), __byte_perm(q4[2], q4[3], sel), 0x5410);
          };
          const uint32_t word = signs(0.f);
          if (!__any_sync(FULLMASK, word != 0)) continue;
          mask = row_mask(word);
          // rows of thousands of candidates are made of dense groups
          if (sure_at < INFINITY && __any_sync(FULLMASK, __popc(mask) >= 16)) sure += __popc(row_mask(signs(sure_at)));
        } else {
          // a tile many lengthscales wide: the same test in FP32, candidate by candidate
#pragma unroll 1
          for (int k = 0; k < 32; k++) {
            float d = 0.f, e = 0.f;
            const float yx = __shfl_sync(FULLMASK, y.x, k), yy = __shfl_sync(FULLMASK, y.y, k), yz = __shfl_sync(FULLMASK, y.z, k);
            d = (x.x - yx) * (x.x - yx) + (x.y - yy) * (x.y - yy) + (x.z - yz) * (x.z - yz);
#pragma unroll
            for (int f = 0; f < 4 * FCH; f++) {
              const float t = f4_at(xf[FCH > 0 ? (f >> 2) % FCH : 0], f & 3) -
                              __shfl_sync(FULLMASK, f4_at(yf[FCH > 0 ? (f >> 2) % FCH : 0], f & 3), k);
              e += t * t;
            }
            if (!(g * d + cw * e > box_tau)) mask |= 1u << k;
          }
          const uint32_t there = __ballot_sync(FULLMASK, has);
          mask &= there;
          load(gm);
        }
        if (valid && mask) {
          if (cnt < caps) out[cnt] = make_uint2((uint32_t)gi, mask);
          cnt++;
          cands += __popc(mask);
        }
      }
    }
  }
  if (valid) P->cand_cnt[(size_t)sp * n + s] = make_int2(cnt | (min(sure, kSureMost) << kSureShift), cands);
}

// --------------------------------------------------------------- row pass
__device__ __forceinline__ int warp_excl_scan(int v, int lane, int &total) {
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULLMASK, incl, o);
    if (lane >= o) incl += t;
  }
  total = __shfl_sync(FULLMASK, incl, 31);
  return incl - v;
}

// One warp per row.  The row's candidates (entries of k_cand) are put in ascending target index
// -- up to 256 of them by a sorting network over the lanes, more through a bitmap over a window
// of target indices in shared memory -- and evaluated 32 at a time with the exact arithmetic,
// the next 32 records in flight.  The reference scans the targets by index and stops at cap kept
// pairs (src/cvo/CvoGPU.cu:994-996): here the row stops there too, and no pair beyond cap is
// stored (nor, but for some rows of ROWS_ORDERED, evaluated).  A row whose entries did not fit,
// or a call without a candidate test, scans all targets in index order instead.
// Sums (all but align): FP32 per lane and row, over the lanes, FP64 from there; the last block
// of a pair adds the blocks' sums in a fixed order.
// ROWS_ORDERED: the entries of a row go to the order of the pair's level (RankLevel), in which
// k_gradient, k_step and k_irls_accum add them one by one.  The align loop and the window solve
// turn a different last bit of the gradient into a visibly different pose some tens of
// iterations later, so the order is part of the result and is kept whatever finds the pairs.
// A row of up to 256 candidates and no more than cap is sorted and evaluated by rank from the
// start; another is cut by index first and its kept entries are then put in order.  One that kept
// more than cap + order_cap pairs stays in index order: nearly all such rows are told by the
// pairs that k_cand is sure of; the rest are evaluated that far (eight pairs of 20k-50k
// points had 7 % of the rows evaluated to 4,353 pairs, 60 % of all evaluations).
// Two instances share the rows of large targets: ROWS_LIGHT those of up to 128 candidates, with
// hardly any shared memory, 32 rows to a block; ROWS_ALL the others, which ROWS_LIGHT lists by
// groups of eight rows, or all rows of targets whose bitmap is small anyway.  Its blocks take
// eight rows at a time and hand them to their warps one by one (rows of 0 to cap pairs lie in
// clusters: blocks of 32 rows left a tail of a third of the launch).
// Bounds: latency of the dependent steps entry -> permutation -> bitmap -> record, hidden by
// the resident warps.  The rows' FP64 constants are computed up to 32 rows at a time: once per
// warp and row they took most of a pass over rows without candidates.
constexpr int kRowWarps = 4;
constexpr int kRowsPerBlock = kGroup;
constexpr int kRowsHeavy = 8;           // rows of a ROWS_ALL block
constexpr int kRowSlots = 1 + kRowsPerBlock / kRowsHeavy;      // partial sums of 32 rows: ROWS_LIGHT, ROWS_ALL
constexpr int kMaxSplits = 16;
// Target indices of one bitmap window.  Only the groups whose indices meet the window are
// entered, and a row that is cut needs the first windows alone.  Small: 20 bitmaps of 60k
// targets left the SM 6 KB of L1, and neighbouring rows read the same targets.
constexpr int kRowWindow = 20 * 1024;
constexpr int kRowBatch = 256;          // candidates taken from the bitmap before they are evaluated
constexpr int kRowSorted = 256;         // most candidates a sorting network puts in order
constexpr int kRowLight = 128;          // most candidates of a row of ROWS_LIGHT
constexpr int kRowSplitTargets = 8192;  // larger targets: ROWS_LIGHT and ROWS_ALL
constexpr int kRowOrdered = 512;        // most entries that order_row puts in order
constexpr size_t kRowRoom = 1ull << 30; // most bytes to order longer rows with, see build_batch

// Whether a kernel instance leaves the rows' entries in index order (single passes) or puts
// them in the order of the pair's level (the align loop, the edges of a window).
enum { ROWS_SUM = 0, ROWS_ORDERED = 1 };
enum { ROWS_ALL = 0, ROWS_LIGHT = 1 };

// A warp's bitmap: four times an odd number of words per lane, so that 16-byte loads of the
// lanes' runs meet distinct banks.  Its queue: 16 bits an index, a batch and the 1024 of one step
// more; also sorted candidates, and a 16-bit count before every four words of the bitmap.
constexpr int kRowWindowWords = kRowWindow / 32;
constexpr int kRowQueueWords = (kRowBatch + 1024) / 2;
static_assert(kRowWindow <= 65536 && kRowWindowWords / 32 % 8 == 4, "16-bit queue, banks");

// Sorts v: element 32 r + lane in register r of each lane, ascending, by a bitonic network.
template <int R, class T>
__device__ __forceinline__ void warp_sort(T (&v)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1)
#pragma unroll
    for (int d = k >> 1; d > 0; d >>= 1) {
      if (d >= 32) {
#pragma unroll
        for (int r = 0; r < R; r++)
          if ((r & (d >> 5)) == 0) {
            const T a = v[r], b = v[r | (d >> 5)];
            const bool up = ((32 * r) & k) == 0;
            v[r] = up ? min(a, b) : max(a, b);
            v[r | (d >> 5)] = up ? max(a, b) : min(a, b);
          }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          const T o = __shfl_xor_sync(FULLMASK, v[r], d);
          const bool up = ((32 * r + lane) & k) == 0;
          v[r] = ((lane & d) == 0) == up ? min(v[r], o) : max(v[r], o);
        }
      }
    }
}

// Sorts list[0 .. count), count <= 32 R.
template <int R>
__device__ __forceinline__ void sort_list(int *list, int count, int lane) {
  int v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = 32 * r + lane < count ? list[32 * r + lane] : 0x7FFFFFFF;
  warp_sort<R>(v, lane);
#pragma unroll
  for (int r = 0; r < R; r++) list[32 * r + lane] = v[r];
}

// Puts the z <= 32 R <= kRowOrdered entries of an ELL row, which are in index order, in the order of the
// ranks: rank (22 bits) and slot sorted as one key.
template <int R>
__device__ __forceinline__ void order_row(int *Aj, float *Av, int z, const int *rank, int lane) {
  uint32_t v[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int c = 32 * r + lane;
    v[r] = c < z ? (uint32_t)__ldg(&rank[Aj[c]]) << 9 | (uint32_t)c : 0xFFFFFFFFu;
  }
  warp_sort<R>(v, lane);
  int j[R];
  float a[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const bool has = 32 * r + lane < z;
    j[r] = has ? Aj[v[r] & 511u] : 0;
    a[r] = has ? Av[v[r] & 511u] : 0.f;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; r++)
    if (32 * r + lane < z) {
      Aj[32 * r + lane] = j[r];
      Av[32 * r + lane] = a[r];
    }
}

// The same for rows of more entries:
// their bits in a bitmap over the ranks, a count before every four words, and each entry's slot is
// the number of bits below its own.  tmp: z entries of the warp's own.  All lanes call it.
__device__ __forceinline__ void order_long_row(int *Aj, float *Av, int z, const int *rank, int m, uint32_t *bits,
                                               unsigned short *before, uint2 *tmp, int lane) {
  constexpr int window_words = kRowWindowWords, wl = window_words >> 5;
  int base = 0;
  for (int w0 = 0; w0 < m && base < z; w0 += 32 * window_words) {
    __syncwarp();
    for (int i = lane; i < window_words / 4; i += 32) reinterpret_cast<uint4 *>(bits)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    for (int c = lane; c < z; c += 32) {
      const uint32_t k = (uint32_t)(__ldg(&rank[Aj[c]]) - w0);
      if (k < 32u * (uint32_t)window_words) atomicOr(&bits[k >> 5], 1u << (k & 31));
    }
    __syncwarp();
    const uint4 *run_bits = reinterpret_cast<const uint4 *>(bits + lane * wl);
    int run = 0, total;
    for (int i = 0; i < wl / 4; i++) {
      const uint4 v = run_bits[i];
      run += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    run = warp_excl_scan(run, lane, total);
    for (int i = 0; i < wl / 4; i++) {
      const uint4 v = run_bits[i];
      before[lane * (wl / 4) + i] = (unsigned short)run;      // below 65536
      run += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    __syncwarp();
    for (int c = lane; c < z; c += 32) {
      const int j = Aj[c];
      const uint32_t k = (uint32_t)(__ldg(&rank[j]) - w0);
      if (k < 32u * (uint32_t)window_words) {
        const uint4 v = reinterpret_cast<const uint4 *>(bits)[k >> 7];
        const uint32_t w = (k >> 5) & 3u, own = w == 0 ? v.x : w == 1 ? v.y : w == 2 ? v.z : v.w;
        const int lower = (w > 0 ? __popc(v.x) : 0) + (w > 1 ? __popc(v.y) : 0) + (w > 2 ? __popc(v.z) : 0);
        tmp[base + before[k >> 7] + lower + __popc(own & ((1u << (k & 31)) - 1u))] = make_uint2((uint32_t)j, __float_as_uint(Av[c]));
      }
    }
    base += total;
  }
  __syncwarp();
  for (int c = lane; c < z; c += 32) {
    const uint2 v = tmp[c];
    Aj[c] = (int)v.x;
    Av[c] = __uint_as_float(v.y);
  }
}

// Totals of an association pass.  Algorithmic bytes: every source and target record once, the
// per-row count, and the ELL entries when they are written.
__device__ __forceinline__ void pass_finished(const BatchDev &B, PairDev *P, double asum, double nnz, double mx) {
  atomicAdd(B.assoc_bytes, (double)(P->n + P->m) * B.record_bytes + 4.0 * P->n + (P->mode != MODE_IP ? 8.0 * nnz : 0.0));
  P->asum = asum;
  P->nnz_sum = (long long)nnz;
  P->max_row = (int)mx;
}

// Sums of a single pass (value, kept pairs, longest row) of one block -> slot; sum_slots adds the
// slots first .. first + slots - 1 and finishes the pass.
__device__ __forceinline__ void rows_partial(PairDev *P, int slot, const double (&t)[3]) {
  for (int k = 0; k < 3; k++) P->part[(size_t)slot * kPartStride + k] = t[k];
}
__device__ __forceinline__ void sum_slots(const BatchDev &B, PairDev *P, int first, int slots) {
  __shared__ double sh[kRowWarps][3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double t[3] = {0, 0, 0};
#pragma unroll 8
  for (int q = threadIdx.x; q < slots; q += 32 * kRowWarps) {
    const double *pv = P->part + (size_t)(first + q) * kPartStride;
    t[0] += __ldcg(pv);
    t[1] += __ldcg(pv + 1);
    t[2] = fmax(t[2], __ldcg(pv + 2));
  }
  t[0] = warp_sum(t[0]);
  t[1] = warp_sum(t[1]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t[2] = fmax(t[2], __shfl_xor_sync(FULLMASK, t[2], o));
  if (lane == 0)
    for (int k = 0; k < 3; k++) sh[w][k] = t[k];
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < 3; k++) {
    t[k] = sh[0][k];
    for (int q = 1; q < kRowWarps; q++) t[k] = k < 2 ? t[k] + sh[q][k] : fmax(t[k], sh[q][k]);
  }
  pass_finished(B, P, t[0], t[1], t[2]);
}
// Without ROWS_LIGHT: the last of the pair's nb blocks.
__device__ __forceinline__ void rows_finish(const BatchDev &B, PairDev *P, int nb, int first, int slots) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&P->counter[0], 1u) == (unsigned)(nb - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  sum_slots(B, P, first, slots);
  if (threadIdx.x == 0) P->counter[0] = 0;
}

// split: ROWS_LIGHT has taken the rows of up to 128 candidates.
template <int FCH, int LCH, bool GT, int KIND, int PART>
__global__ void __launch_bounds__(32 * kRowWarps, PART == ROWS_LIGHT && LCH == 0 ? 6 : 5)
    k_rows(BatchDev B, KParams K, int split) {
  constexpr int RB = PART == ROWS_LIGHT ? kRowsPerBlock : kRowsHeavy;
  constexpr int kWords = PART == ROWS_LIGHT ? kRowLight : kRowWindowWords + kRowQueueWords;
  __shared__ __align__(16) uint32_t row_smem[kRowWarps][kWords];      // bitmap and queue
  __shared__ float4 sh_rc[RB];                             // l, d2 threshold, 1 / (2 l^2)
  __shared__ int2 sh_cnt[kMaxSplits][RB];                  // entries and candidates per split
  __shared__ int4 sh_tot[RB];                              // of the row, and pairs surely kept; entries < 0: scan all targets
  __shared__ double sh_sum[RB];                            // the rows' sums and kept pairs
  __shared__ int sh_kept[RB];
  __shared__ int next_row, item;
  __shared__ float4 sh_keep[kRowWarps][64];                // kept pairs by slot: y and value
  __shared__ int sh_keepj[kRowWarps][64];
  constexpr int FP = FCH > 0 ? FCH : 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int SUBS = kRowsPerBlock / RB;                 // blocks of a source tile
  uint32_t *bits = row_smem[w];
  int *sorted = reinterpret_cast<int *>(PART == ROWS_LIGHT ? bits : bits + kRowWindowWords);
  unsigned short *queue = reinterpret_cast<unsigned short *>(sorted);
  while (true) {
  // ROWS_ALL after ROWS_LIGHT: the next listed group of rows; otherwise the block's own
  int group = blockIdx.x;
  if (PART == ROWS_ALL && split) {
    __syncthreads();      // the last item's shared memory has been read
    if (threadIdx.x == 0) item = atomicAdd(&B.heavy_ctr[1], 1);
    __syncthreads();
    if (item >= __ldcg(&B.heavy_ctr[0])) return;
    group = __ldcg(&B.heavy[item]);
  }
  const int blk = group / SUBS, part = group % SUBS;
  if (blk >= B.total_rblocks) return;
  const int p = find_segment(B.rblk_off, B.npairs, blk);
  PairDev *P = &B.pairs[p];
  if (P->done) return;
  const int b = blk - B.rblk_off[p], nb = B.rblk_off[p + 1] - B.rblk_off[p];
  const int n = P->n, m = P->m, F = P->F, C = P->C, cap = P->cap, mode = P->mode, S = P->splits, caps = P->cap_split;
  const float4 *__restrict__ yorig = P->yorig;
  const float4 *__restrict__ tf = reinterpret_cast<const float4 *>(P->tf);
  const float4 *__restrict__ tl = reinterpret_cast<const float4 *>(P->tl);
  const int *__restrict__ tperm = P->tperm;
  const int2 *__restrict__ trange = P->trange;
  const int s0 = b * kRowsPerBlock + part * RB;
  {
    if (K.use_mma)
      for (int i = threadIdx.x; i < S * RB; i += 32 * kRowWarps) {
        const int q = i / RB, s = s0 + i % RB;
        sh_cnt[q][i % RB] = s < n ? __ldg(&P->cand_cnt[(size_t)q * n + s]) : make_int2(0, 0);
      }
    if (threadIdx.x == 0) next_row = 0;
    __syncthreads();
    bool here = false;
    if (threadIdx.x < RB) {
      const int s = s0 + lane;
      int4 t = make_int4(K.use_mma ? 0 : -1, 0, 0, 0);
      bool fits = true;
      for (int q = 0; q < S && K.use_mma; q++) {
        int2 c = sh_cnt[q][lane];
        t.z += c.x >> kSureShift;
        c.x &= (1 << kSureShift) - 1;
        sh_cnt[q][lane].x = c.x;
        fits = fits && c.x <= caps;
        t.x += c.x;
        t.y += c.y;
      }
      if (!fits) t.x = -1;
      if (cap <= 0 || s >= n) t.x = 0;
      const bool light = t.x >= 0 && t.y <= kRowLight;
      if (PART == ROWS_LIGHT) {
        constexpr int groups = kRowsPerBlock / kRowsHeavy;
        const unsigned heavy = __ballot_sync(FULLMASK, t.x != 0 && !light);
        if (lane < groups) {
          if (heavy >> (kRowsHeavy * lane) & ((1u << kRowsHeavy) - 1u))
            B.heavy[atomicAdd(&B.heavy_ctr[0], 1)] = groups * blk + lane;
          else if (mode != MODE_ALIGN)
            for (int k = 0; k < 3; k++) P->part[(size_t)(nb + groups * b + lane) * kPartStride + k] = 0.0;
        }
      }
      if (s < n && t.x == 0 && (PART == ROWS_LIGHT || !split)) P->nnz_row[s] = 0;
      if (PART == ROWS_LIGHT ? !light : split && light) t.x = 0;      // the other instance's
      here = t.x != 0;
      sh_tot[lane] = t;
      sh_sum[lane] = 0.0;
      sh_kept[lane] = 0;
    }
    const bool any = __syncthreads_or(here);
    if (any && threadIdx.x < RB) {
      const int s = s0 + lane;
      const RowConst rc = row_const(K, P->ell, s < n ? __ldg(&P->xs[s]).w : 0.f);
      sh_rc[lane] = make_float4(rc.l, rc.d2t, rc.inv2l2, 0.f);
    }
    if (any) __syncthreads();
    else if (KIND == ROWS_ORDERED && mode == MODE_ALIGN) return;
  }
  const int order_cap = KIND == ROWS_ORDERED ? P->order_cap : 0;
  const RankLevel *lv = KIND == ROWS_ORDERED ? P->levels + P->level : nullptr;
  for (int r = w;; r += kRowWarps) {
    if (PART == ROWS_ALL) {
      if (lane == 0) r = atomicAdd(&next_row, 1);
      r = __shfl_sync(FULLMASK, r, 0);
    }
    if (r >= RB) break;
    const int entries = sh_tot[r].x, cands = sh_tot[r].y;
    if (entries == 0) continue;
    const int s = s0 + r;
    const float4 x = __ldg(&P->xs[s]);
    float4 xf[FP];
#pragma unroll
    for (int q = 0; q < FP; q++)
      xf[q] = FCH > 0 ? __ldg(reinterpret_cast<const float4 *>(P->xf) + (size_t)s * FCH + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 *xl = reinterpret_cast<const float4 *>(P->xl) + (size_t)s * LCH;
    const float2 xg = GT ? __ldg(&P->xg[s]) : make_float2(0.f, 0.f);
    const float4 rc = sh_rc[r];
    const uint2 *ent = P->cand + (size_t)s * P->cand_pitch;
    // entry e of the row, the splits' entries one after the other
    auto entry = [&](int e) {
      const uint2 *at = nullptr;
      for (int q = 0; q < S; q++) {
        const int c = sh_cnt[q][r].x;
        if (e >= 0 && e < c) at = ent + (size_t)q * caps + e;
        e -= c;
      }
      return at ? __ldg(at) : make_uint2(0u, 0u);
    };
    // by rank from the start if the row cannot be cut; otherwise by index, and on past cap only
    // to tell whether the row keeps more than cap + order_cap (it may, and is not sure to)
    const bool ranked = KIND == ROWS_ORDERED && entries > 0 && cands <= min(cap, kRowSorted);
    const int *perm = ranked ? lv->of_tile : tperm;
    const bool over = KIND == ROWS_ORDERED && sh_tot[r].z > cap + order_cap;
    const int stop = KIND == ROWS_ORDERED && !over && (entries < 0 || cands > cap + order_cap) ? cap + order_cap + 1 : cap;
    int kept = 0;
    float acc = 0.f;
    // 32 kept pairs to the ELL row and the sum: lane l takes slots l, l + 32, ..., so the
    // sum depends on the kept pairs alone, not on the candidates beside them
    int flushed = 0;
    float4 *keep = sh_keep[w];
    int *keepj = sh_keepj[w];
    auto flush = [&](bool on) {
      const float4 v = keep[(flushed + lane) & 63];
      if (on) {
        if (KIND == ROWS_ORDERED || mode != MODE_IP) {
          P->A_j[(size_t)s * P->ld + flushed + lane] = keepj[(flushed + lane) & 63];
          P->A_v[(size_t)s * P->ld + flushed + lane] = v.w;
        }
        acc += v.w;
      }
      flushed += 32;
      __syncwarp();
    };
    // Rounds of n candidates in order: all of a sorted list, all targets, or a queue (relative to
    // w0) taken from the bitmap 32 words at a time, one a lane: the indices of a row lie in
    // clusters, and a run of words per lane left most lanes idle.
    const bool direct = entries < 0, listed = !direct && cands <= kRowSorted;
    int w0 = -1, w1 = 0, pos = 0, qn = 0;      // window, the next one, words read, queue
    bool filled = false;
    while (true) {
      int n = m;
      if (PART == ROWS_LIGHT || listed) {
        // one to four candidates in a lane, sorted by a bitonic network
        n = 0;
        for (int e0 = 0; e0 < entries; e0 += 32) {
          const uint2 v = entry(e0 + lane);
          int o, add;
          o = n + warp_excl_scan(__popc(v.y), lane, add);
          for (uint32_t mk = v.y; mk; mk &= mk - 1) sorted[o++] = 32 * (int)v.x + __ffs(mk) - 1;
          n += add;
        }
        __syncwarp();
        for (int i = lane; i < n; i += 32) sorted[i] = __ldg(&perm[sorted[i]]);      // not in the loop over bits: a chain of loads
        __syncwarp();
        if (n <= 32) sort_list<1>(sorted, n, lane);
        else if (n <= 64) sort_list<2>(sorted, n, lane);
        else if (PART == ROWS_LIGHT || n <= 128) sort_list<4>(sorted, n, lane);
        else sort_list<8>(sorted, n, lane);
        __syncwarp();
      } else if (!direct) {
        if (!filled) {
          if (w0 < 0) {      // the first window starts at the row's lowest index
            int low = INT_MAX;
            for (int e0 = 0; e0 < entries; e0 += 32) {
              const uint2 v = entry(e0 + lane);
              if (v.y) low = min(low, __ldg(&trange[v.x]).x);
            }
            w0 = __reduce_min_sync(FULLMASK, low) & ~31;
          }
          for (int i = lane; i < kRowWindowWords / 4; i += 32) reinterpret_cast<uint4 *>(bits)[i] = make_uint4(0u, 0u, 0u, 0u);
          __syncwarp();
          w1 = INT_MAX;
          for (int e0 = 0; e0 < entries; e0 += 32) {
            const uint2 v = entry(e0 + lane);
            const int2 range = v.y ? __ldg(&trange[v.x]) : make_int2(0, -1);
            if (range.y >= w0 + kRowWindow) w1 = min(w1, max(range.x, w0 + kRowWindow));
            uint32_t todo = __ballot_sync(FULLMASK, range.y >= w0 && range.x < w0 + kRowWindow);
            while (todo) {
              // eight groups' indices in flight: a load under its own branch waits for the last one
              uint32_t k[8];
#pragma unroll
              for (int u = 0; u < 8; u++) {
                const int src = todo ? __ffs(todo) - 1 : 0;
                const int g = __shfl_sync(FULLMASK, (int)v.x, src);
                const uint32_t mk = __shfl_sync(FULLMASK, todo ? v.y : 0u, src);
                const uint32_t at = (uint32_t)(__ldg(&tperm[min(32 * g + lane, m - 1)]) - w0);
                k[u] = (mk >> lane) & 1u ? at : 0xFFFFFFFFu;
                todo &= todo - 1;
              }
#pragma unroll
              for (int u = 0; u < 8; u++)
                if (k[u] < (uint32_t)kRowWindow) atomicOr(&bits[k[u] >> 5], 1u << (k[u] & 31));
            }
          }
          w1 = __reduce_min_sync(FULLMASK, w1);
          __syncwarp();
          filled = true;
          pos = qn = 0;
        }
        for (; pos < kRowWindowWords && qn < kRowBatch; pos += 32) {
          uint32_t mk = bits[pos + lane];
          if (!__any_sync(FULLMASK, mk != 0)) continue;
          int add, o = qn + warp_excl_scan(__popc(mk), lane, add);
          uint32_t words = __ballot_sync(FULLMASK, mk != 0);
          if (__popc(words) <= __reduce_max_sync(FULLMASK, __popc(mk))) {
            // few words, some of them dense: word by word, a bit a lane
            for (; words; words &= words - 1) {
              const int src = __ffs(words) - 1;
              const uint32_t v = __shfl_sync(FULLMASK, mk, src);
              const int at = __shfl_sync(FULLMASK, o, src);
              if ((v >> lane) & 1u) queue[at + __popc(v & ((1u << lane) - 1u))] = (unsigned short)(32 * (pos + src) + lane);
            }
          } else {
            for (; mk; mk &= mk - 1) queue[o++] = (unsigned short)(32 * (pos + lane) + __ffs(mk) - 1);
          }
          qn += add;
        }
        __syncwarp();
        n = pos < kRowWindowWords ? qn & ~31 : qn;      // whole rounds of 32, and the rest when the window ends
      }
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f), yf[FP];
#pragma unroll
      for (int q = 0; q < FP; q++) yf[q] = y;
      int j = 0;
      auto load = [&](int i) {
        if (i >= n) return;
        if (PART == ROWS_LIGHT || listed) j = sorted[i];
        else j = direct ? i : w0 + queue[i];
        if (ranked) j = __ldg(&lv->index[j]);
        y = __ldg(&yorig[j]);
#pragma unroll
        for (int q = 0; q < FCH; q++) yf[q] = __ldg(tf + (size_t)j * FCH + q);
      };
      load(lane);
      for (int i0 = 0; i0 < n && kept < stop; i0 += 32) {
        const bool has = i0 + lane < n;
        const float4 yc = y;
        float4 fc[FP];
#pragma unroll
        for (int q = 0; q < FP; q++) fc[q] = yf[q];
        const int jc = j;
        load(i0 + 32 + lane);
        const float2 yg = GT && has ? __ldg(&P->tg[jc]) : make_float2(0.f, 0.f);
        float a = 0.f;
        const bool k = eval_pair<FCH, LCH, GT>(K, F, C, has, rc.x, rc.y, rc.z, x, xf, xl, xg, yc, fc,
                                               tl + (size_t)jc * LCH, yg, a);
        const unsigned bal = __ballot_sync(FULLMASK, k);
        const int c = kept + __popc(bal & ((1u << lane) - 1u));
        if (k && c < cap) {
          keep[c & 63] = make_float4(yc.x, yc.y, yc.z, a);
          keepj[c & 63] = jc;
        }
        kept += __popc(bal);
        __syncwarp();
        if (min(kept, cap) - flushed >= 32) flush(true);
      }
      __syncwarp();
      if (PART == ROWS_LIGHT || listed || direct || kept >= stop) break;
      if (pos < kRowWindowWords) {
        const unsigned short rest = n + lane < qn ? queue[n + lane] : (unsigned short)0;
        __syncwarp();
        queue[lane] = rest;
        qn -= n;
        __syncwarp();
      } else {
        if (w1 == INT_MAX) break;
        w0 = w1 & ~31;
        filled = false;
      }
    }
    const int z = min(kept, cap);
    if (flushed < z) flush(lane < z - flushed);
    if (lane == 0) P->nnz_row[s] = z;
    if (KIND == ROWS_ORDERED) {
      if (!ranked && z > 1 && !over && kept <= cap + order_cap && K.use_geo) {
        int *Aj = P->A_j + (size_t)s * P->ld;
        float *Av = P->A_v + (size_t)s * P->ld;
        __syncwarp();
        if (PART == ROWS_LIGHT) order_row<4>(Aj, Av, z, lv->of_index, lane);
        else if (z <= 256) order_row<8>(Aj, Av, z, lv->of_index, lane);
        else if (z <= kRowOrdered) order_row<16>(Aj, Av, z, lv->of_index, lane);
        else order_long_row(Aj, Av, z, lv->of_index, m, bits, queue, P->long_rows + (size_t)(split ? blockIdx.x * kRowWarps + w : s) * P->long_pitch, lane);
      }
      __syncwarp();
      if (mode == MODE_ALIGN) continue;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULLMASK, acc, o);
    if (lane == 0) {
      sh_sum[r] = (double)acc;
      sh_kept[r] = z;
    }
  }
  if (KIND == ROWS_ORDERED && mode == MODE_ALIGN) {
    if (PART == ROWS_ALL && split) continue;
    return;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[3] = {0.0, 0.0, 0.0};
    for (int r = 0; r < RB; r++) {
      t[0] += sh_sum[r];
      t[1] += (double)sh_kept[r];
      t[2] = fmax(t[2], (double)sh_kept[r]);
    }
    rows_partial(P, PART == ROWS_LIGHT ? b : nb + SUBS * b + part, t);
  }
  if (PART == ROWS_ALL && split) continue;      // k_rows_total adds the slots
  if (PART == ROWS_ALL) rows_finish(B, P, SUBS * nb, nb, (kRowSlots - 1) * nb);
  return;
  }
}

}  // namespace cvo_gb
