// k_align.cu -- projective ICP kernels (AlignerProjective::align and its parts).
//
//   k_zbuffer    PinholePointProjector::project (pinholepointprojector.cpp:33-66):
//                one thread per point, 64-bit atomicMin of (depth key << 32 | index)
//                into a per-pair z-buffer.  The serial reference keeps the first
//                point with the strictly smallest depth, i.e. the minimum of
//                (depth, index) -- exactly what the packed minimum keeps.
//   k_resolve    z-buffer -> index image (+ depth image), resetting the z-buffer.
//   k_corr_lin   fused CorrespondenceFinderProjective::_computeSingle
//                (correspondencefinderprojective.cpp:23-115) and Linearizer::update
//                (linearizer.cpp:21-134): per pixel, gate the pair, and if accepted
//                add its 21 H + 6 b + chi2 + inlier terms.  Per-thread sums in FP32
//                over 8 pixels, then FP64: transposed through shared memory, one
//                partial per 1024-pixel tile (fixed tile -> partial mapping).
//   k_corr_tile  the same pass, the same sums in the same order, one CTA per
//                tile: loops of few tiles.
//   k_corr_count / k_corr_write
//                the same gates with ordered compaction into the reference's
//                row-major correspondence list (parity / list mode).
//   k_lin_list   Linearizer::update over a correspondence list (with the
//                reference's K % T drop when T > 1).
//   k_begin_loop / k_publish
//                descriptors and poses from pinned host memory, states, tables and
//                empty z-buffers; the states back to pinned host memory.
//   k_solve      per pair: fixed-order FP64 sum of the tile partials, H + lambda I,
//                6x6 LDL^T, pose update and renormalisation (alignerprojective.cpp:
//                72-100), early exit, and the float matrices of the next iteration.
#include <cuda_runtime.h>

#include <type_traits>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "kernels.hpp"

namespace nicp {

// The pair whose pixel tiles hold tile `key` (largest i with tile_base <= key).
__device__ __forceinline__ int find_pair(const PairDev *pairs, int n, int key) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    int b = pairs[mid].tile_base;
    if (b <= key) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------ z-buffer
// mode 0: project the current cloud with pair.KRt_cur-equivalent `explicit_KRt`
// (one matrix for all pairs, host-computed); mode 1: the reference cloud with
// the pair state's KRt.
// A CTA covers kPointsPerCta points with kPointsPerCta / PPT threads, PPT
// independent points per thread (their loads and atomics overlap); the
// result does not depend on PPT (atomicMin is order-free).  Grid: (point
// tile, pair) -- the pair comes from blockIdx.y, with no search, so a CTA's
// first loads are its pose and its points.
template <int PPT>
__global__ void __launch_bounds__(kPointsPerCta / PPT)
    k_zbuffer(const PairDev *__restrict__ pairs, int npairs, int mode, const float *__restrict__ explicit_KRt,
              int pair0) {
  constexpr int kThreads = kPointsPerCta / PPT;
  const int pi = pair0 + (int)blockIdx.y;
  if (pi >= npairs) return;
  const PairDev &pd = pairs[pi];
  const PairState *st = pd.state;
  // the clouds are older than the loop: the points are fetched while the
  // kernel before (the solve that sets KRt and done) finishes
  const int i0 = blockIdx.x * kPointsPerCta + threadIdx.x;
  const float4 *pts = mode ? pd.ref_pts : pd.cur_pts;
  const int n = mode ? *pd.ref_count : *pd.cur_count;
  float4 p[PPT];
#pragma unroll
  for (int k = 0; k < PPT; k++) {
    int i = i0 + k * kThreads;
    p[k] = (i < n) ? pts[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  chain();
  if (mode == 1 && st->done) return;
  if (i0 >= n) return;
  float K[12];
  const float *src = mode ? st->KRt : explicit_KRt + 12 * pi;
#pragma unroll
  for (int k = 0; k < 12; k++) K[k] = src[k];
#pragma unroll
  for (int k = 0; k < PPT; k++) {
    int i = i0 + k * kThreads;
    int x, y;
    float d;
    if (i >= n || !project_pixel(K, p[k], pd.rows, pd.cols, pd.min_d, pd.max_d, x, y, d)) continue;
    unsigned long long key =
        ((unsigned long long)float_key(d) << 32) | ((unsigned)i << 1) | (point_has_normal(p[k].w) ? 0u : 1u);
    atomicMin(pd.zbuf + (size_t)y * pd.cols + x, key);
  }
}

// Decodes a z-buffer word: the point index, or -1 when empty -- or, with
// drop_no_normal, when the point has no normal (such a pixel can never pass
// the correspondence gates unless they are demoted to GICP).
__device__ __forceinline__ int zbuf_index(unsigned long long z, bool drop_no_normal) {
  if (z == ~0ull) return -1;
  unsigned lo = (unsigned)(z & 0xffffffffull);
  if (drop_no_normal && (lo & 1u)) return -1;
  return (int)(lo >> 1);
}

// z-buffer -> int index image (and optional depth image, FLT_MAX where empty);
// the z-buffer is left all ones for its next use.  Thread t handles pixels
// t, t + 256, ... of its tile: every warp access is one contiguous run.
// Grid (pixel tile, pair): the pair is pair0 + blockIdx.y, no search.
__global__ void k_resolve(const PairDev *__restrict__ pairs, int npairs, int to_ref, float *depth_out,
                          int drop_no_normal, int pair0) {
  const int pi = pair0 + (int)blockIdx.y;
  if (pi >= npairs) return;
  const PairDev &pd = pairs[pi];
  const int P = pd.rows * pd.cols;
  const int pix0 = blockIdx.x * kCorrTilePixels + threadIdx.x;
  int32_t *dst = to_ref ? pd.ref_index : pd.cur_index;
  chain();
  unsigned long long z[kCorrTilePixels / kCorrThreads];
#pragma unroll
  for (int k = 0; k < kCorrTilePixels / kCorrThreads; k++) {
    const int p = pix0 + k * kCorrThreads;
    z[k] = p < P ? pd.zbuf[p] : ~0ull;
  }
#pragma unroll
  for (int k = 0; k < kCorrTilePixels / kCorrThreads; k++) {
    const int p = pix0 + k * kCorrThreads;
    if (p < P) {
      pd.zbuf[p] = ~0ull;
      dst[p] = zbuf_index(z[k], drop_no_normal != 0);
      if (depth_out) depth_out[p] = (z[k] == ~0ull) ? 3.402823466e+38f : key_float((uint32_t)(z[k] >> 32));
    }
  }
}

// ------------------------------------------------------------ gates + terms
struct Acc {
  // 0..5 Htt lower (00 10 11 20 21 22), 6..14 Htr row-major, 15..20 Hrr lower,
  // 21..23 bt, 24..26 br, 27 chi2, 28 inliers, 29 candidates, 30 accepted.
  // The rotational Jacobian block is skew(2 p) (linearizer.cpp:59-100); the
  // per-pixel terms use skew(p), so Htr and br hold half and Hrr a quarter of
  // their values, and the reductions scale the FP64 tile sums by 2 and 4
  // (exact: powers of two).  The three counts (28 inliers, 29 candidates,
  // 30 accepted) share one integer, 10 bits each (a thread adds at most 8
  // pixels or 4 list entries to a tile partial).
  float v[28];
  unsigned cnt;
  static constexpr unsigned kInlier = 1u, kCandidate = 1u << 10, kAccepted = 1u << 20;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < 28; k++) v[k] = 0.0f;
    cnt = 0u;
  }
  // element k of the partial (0..30) as a float
  __device__ __forceinline__ float get(int k) const {
    return k < 28 ? v[k] : (float)((cnt >> (10 * (k - 28))) & 1023u);
  }
};
// Power-of-two factor of each Acc element (see Acc).
__device__ __forceinline__ double acc_scale(int k) {
  return (k >= 15 && k <= 20) ? 4.0 : ((k >= 6 && k <= 14) || (k >= 24 && k <= 26)) ? 2.0 : 1.0;
}

// The gate's arithmetic: dot3x and xform_normal without the reference's
// zero w terms ("+ 0 * 0" of the 4-vector dot products, "+ A3 * 0" of the
// normal transform), which change at most the sign of a zero -- no
// comparison of the gates can tell, so the decisions stay bitwise the
// reference's -- and xform_point with its "+ A3 * 1" written as "+ A3".
__device__ __forceinline__ float dot3g(float ax, float ay, float az, float bx, float by, float bz) {
  float s = fm(ax, bx);
  s = fa(s, fm(ay, by));
  return fa(s, fm(az, bz));
}
// The reference's "normal.squaredNorm() == 0" (correspondencefinderprojective.cpp:69,
// the normal's w is 0): a sum of non-negative float squares is zero exactly
// when every square rounds to zero, and x * x rounds to zero (round to
// nearest even, subnormals kept) exactly when |x| <= 2^-75, since 2^-150 is
// the tie between 0 and the smallest subnormal 2^-149.  A NaN component
// makes the squared norm NaN, not zero, and every comparison below false.
// Three compares instead of three products and two sums.
__device__ __forceinline__ bool normal_is_zero(float x, float y, float z) {
  constexpr float t = 0x1p-75f;
  return fabsf(x) <= t && fabsf(y) <= t && fabsf(z) <= t;
}
__device__ __forceinline__ float rowg(const float *A, float x, float y, float z) {
  float s = fm(A[0], x);
  s = fa(s, fm(A[1], y));
  return fa(s, fm(A[2], z));
}
// rowg with its first two products in one packed multiply (sm_100 FMUL2;
// each half is rounded as __fmul_rn rounds it, so the sum is bitwise rowg's):
// ((A0 x + A1 y) + A2 z).  A is read element by element (it may be a
// thread's register array as well as a shared row).
__device__ __forceinline__ float rowg2(const float *A, float2 xy, float z) {
  const float2 m = __fmul2_rn(make_float2(A[0], A[1]), xy);
  return fa(fa(m.x, m.y), fm(A[2], z));
}
__device__ __forceinline__ float3 xform_point_g2(const float *A, float4 p) {
  const float2 xy = make_float2(p.x, p.y);
  return make_float3(fa(rowg2(A, xy, p.z), A[3]), fa(rowg2(A + 4, xy, p.z), A[7]), fa(rowg2(A + 8, xy, p.z), A[11]));
}
__device__ __forceinline__ float3 xform_normal_g2(const float *A, float4 n) {
  const float2 xy = make_float2(n.x, n.y);
  return make_float3(rowg2(A, xy, n.z), rowg2(A + 4, xy, n.z), rowg2(A + 8, xy, n.z));
}
__device__ __forceinline__ float3 xform_normal_g(const float *A, float4 n) {
  return make_float3(rowg(A, n.x, n.y, n.z), rowg(A + 4, n.x, n.y, n.z), rowg(A + 8, n.x, n.y, n.z));
}
// row4 with w = 1: "+ A3 * 1" adds A3 exactly
__device__ __forceinline__ float3 xform_point_g(const float *A, float4 p) {
  return make_float3(fa(rowg(A, p.x, p.y, p.z), A[3]), fa(rowg(A + 4, p.x, p.y, p.z), A[7]),
                     fa(rowg(A + 8, p.x, p.y, p.z), A[11]));
}

// correspondencefinderprojective.cpp:59-101.  T12: rows 0..2 of the gating
// transform (the aligner passes _T.inverse()).
// The transformed reference point and normal are returned in rp / rn (rn
// only when the normal gates run, i.e. not demoted).
template <bool kPlain = false>
__device__ __forceinline__ bool gate_t(const CorrParams &cp, const float *T12, float4 rp0, float4 rn0, float4 cpt,
                                       float4 cn, float3 &rp, float3 &rn) {
  if (kPlain || !cp.demoted) {
    if (normal_is_zero(cn.x, cn.y, cn.z)) return false;
    if (normal_is_zero(rn0.x, rn0.y, rn0.z)) return false;
  }
  rp = xform_point_g2(T12, rp0);
  float dx = fsb(cpt.x, rp.x), dy = fsb(cpt.y, rp.y), dz = fsb(cpt.z, rp.z);
  if (dot3g(dx, dy, dz, dx, dy, dz) > cp.sq_thr) return false;
  if (kPlain || !cp.demoted) {
    rn = xform_normal_g2(T12, rn0);
    if (dot3g(cn.x, cn.y, cn.z, rn.x, rn.y, rn.z) < cp.cos_thr) return false;
    float kr = rn0.w, kc = cn.w;
    if (kr < cp.flat_thr) kr = cp.flat_thr;
    if (kc < cp.flat_thr) kc = cp.flat_thr;
    // equal curvatures (in particular both below the flat threshold) give a
    // ratio of exactly 1: skip the division
    float ratio =
        (kr == kc) ? 1.0f : __double2float_rn(__ddiv_rn(__dadd_rn((double)kr, 1e-5), __dadd_rn((double)kc, 1e-5)));
    if (ratio < cp.min_ratio || ratio > cp.max_ratio) return false;
  }
  return true;
}

__device__ __forceinline__ bool gate(const CorrParams &cp, const float *T12, float4 rp0, float4 rn0, float4 cpt,
                                     float4 cn) {
  float3 rp, rn;
  return gate_t(cp, T12, rp0, rn0, cpt, cn, rp, rn);
}

// linearizer.cpp:59-100 for one correspondence, FP32.
__device__ __forceinline__ void lin_terms(const LinParams &lp, const float *T12, float4 rp0, float4 rn0, float4 cpt,
                                         float4 cn, float4 o0, float4 o1, float4 o2, Acc &acc) {
  float3 rp = xform_point_g(T12, rp0);
  float3 rn = xform_normal_g(T12, rn0);
  // symmetric 3x3 as (00 01 02 11 12 22)
  float Op[6] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y};
  float On[6] = {o1.z, o1.w, o2.x, o2.y, o2.z, o2.w};
#pragma unroll
  for (int k = 0; k < 6; k++) On[k] = lp.scale * On[k];
  if (lp.z_scaling) {
    float f = 1.0f / fabsf(cpt.z);
#pragma unroll
    for (int k = 0; k < 6; k++) { Op[k] *= f; On[k] *= f; }
  }
  if (lp.demoted) {
#pragma unroll
    for (int k = 0; k < 6; k++) On[k] = 0.0f;
  }
  float pe[3] = {rp.x - cpt.x, rp.y - cpt.y, rp.z - cpt.z};
  float ne[3] = {rn.x - cn.x, rn.y - cn.y, rn.z - cn.z};
  float ep[3] = {Op[0] * pe[0] + Op[1] * pe[1] + Op[2] * pe[2], Op[1] * pe[0] + Op[3] * pe[1] + Op[4] * pe[2],
                 Op[2] * pe[0] + Op[4] * pe[1] + Op[5] * pe[2]};
  float en[3] = {On[0] * ne[0] + On[1] * ne[1] + On[2] * ne[2], On[1] * ne[0] + On[3] * ne[1] + On[4] * ne[2],
                 On[2] * ne[0] + On[4] * ne[1] + On[5] * ne[2]};
  float le = (pe[0] * ep[0] + pe[1] * ep[1] + pe[2] * ep[2]) + (ne[0] * en[0] + ne[1] * en[1] + ne[2] * en[2]);
  float ks = 1.0f;
  if (le > lp.max_chi2) {
    if (lp.robust) ks = lp.max_chi2 / le;
    else return;
  }
  acc.v[27] += ks * le;
  acc.cnt += Acc::kInlier;
  // skew(v) = [[0, c, -b], [-c, 0, a], [b, -a, 0]], (a, b, c) = v (the
  // Jacobian's factor 2 is applied to the tile sums, see Acc)
  float a = rp.x, b = rp.y, c = rp.z;
  float an = rn.x, bn = rn.y, cn2 = rn.z;
  // Htt += Op * ks
  acc.v[0] += Op[0] * ks; acc.v[1] += Op[1] * ks; acc.v[2] += Op[3] * ks;
  acc.v[3] += Op[2] * ks; acc.v[4] += Op[4] * ks; acc.v[5] += Op[5] * ks;
  // Htr += (Op Sp) ks: (Op S)_i0 = -c Op_i1 + b Op_i2; _i1 = c Op_i0 - a Op_i2; _i2 = -b Op_i0 + a Op_i1
  const float Om[3][3] = {{Op[0], Op[1], Op[2]}, {Op[1], Op[3], Op[4]}, {Op[2], Op[4], Op[5]}};
#pragma unroll
  for (int i = 0; i < 3; i++) {
    acc.v[6 + i * 3 + 0] += (-c * Om[i][1] + b * Om[i][2]) * ks;
    acc.v[6 + i * 3 + 1] += (c * Om[i][0] - a * Om[i][2]) * ks;
    acc.v[6 + i * 3 + 2] += (-b * Om[i][0] + a * Om[i][1]) * ks;
  }
  // Hrr += (S^T O S) for the point and the normal terms
  const float Nm[3][3] = {{On[0], On[1], On[2]}, {On[1], On[3], On[4]}, {On[2], On[4], On[5]}};
  float Ap[3][3], An[3][3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    Ap[0][j] = -c * Om[1][j] + b * Om[2][j];
    Ap[1][j] = c * Om[0][j] - a * Om[2][j];
    Ap[2][j] = -b * Om[0][j] + a * Om[1][j];
    An[0][j] = -cn2 * Nm[1][j] + bn * Nm[2][j];
    An[1][j] = cn2 * Nm[0][j] - an * Nm[2][j];
    An[2][j] = -bn * Nm[0][j] + an * Nm[1][j];
  }
  float R[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    R[i][0] = (-c * Ap[i][1] + b * Ap[i][2]) + (-cn2 * An[i][1] + bn * An[i][2]);
    R[i][1] = (c * Ap[i][0] - a * Ap[i][2]) + (cn2 * An[i][0] - an * An[i][2]);
    R[i][2] = (-b * Ap[i][0] + a * Ap[i][1]) + (-bn * An[i][0] + an * An[i][1]);
  }
  acc.v[15] += R[0][0] * ks; acc.v[16] += R[1][0] * ks; acc.v[17] += R[1][1] * ks;
  acc.v[18] += R[2][0] * ks; acc.v[19] += R[2][1] * ks; acc.v[20] += R[2][2] * ks;
  // bt += ks ep; br += ks (Sp^T ep + Sn^T en), S^T e = v x e
  acc.v[21] += ks * ep[0]; acc.v[22] += ks * ep[1]; acc.v[23] += ks * ep[2];
  float u0 = b * ep[2] - c * ep[1], u1 = c * ep[0] - a * ep[2], u2 = a * ep[1] - b * ep[0];
  float w0 = bn * en[2] - cn2 * en[1], w1 = cn2 * en[0] - an * en[2], w2 = an * en[1] - bn * en[0];
  acc.v[24] += ks * (u0 + w0); acc.v[25] += ks * (u1 + w1); acc.v[26] += ks * (u2 + w2);
}

// lin_terms for a current point whose information matrices have the
// converter's structure Omega = d1 I + (d0 - d1) u u^T, u its normal (the
// smallest-eigenvalue eigenvector; Omega = U diag(d0, d1, d1) U^T,
// informationmatrixcalculator.cpp:9-57).  With S = skew(v) (S x = x cross v,
// v the moved point; the Jacobian's factor 2 is applied to the tile sums, see
// Acc) and w = S^T u:  Omega e = a e + b (u.e) u,  Omega S = a S + b u w^T,
// S^T Omega S = a (|v|^2 I - v v^T) + b w w^T.  The class code in the
// point's w selects (d0, d1); omd holds them for the four classes.
// rp, rn: the reference point and normal already moved by the linearizer's
// transform.  Every accumulator update is one fused chain of FMAs; the
// robust kernel's weight ks (linearizer.cpp:83-89) is folded into the
// weights and residual terms only for the pixels beyond the chi2 bound.
// A pixel's part is what the sums need of it (PixelTerms); two disjoint sets
// of accumulators take it up (add_pose_terms, add_rotation_terms), so that
// k_corr_tile can give them to different warps.
struct PixelTerms {
  float ux, uy, uz, be;   // current normal, beta of Omega_p
  float a, b, c, al;      // moved reference point, alpha of Omega_p
  float an, bn, cn, aln;  // moved reference normal, alpha of Omega_n
  float ep0, ep1, ep2, ben;  // Omega_p times the point residual, beta of Omega_n
  float en0, en1, en2, le;   // Omega_n times the normal residual, chi2
};

// (alpha, beta) of Omega_p and Omega_n for a class code, scaled as the
// linearizer scales them.
__device__ __forceinline__ float4 class_weights(const LinParams &lp, const float *omd, int cls) {
  const float *dp = omd + 2 * (cls & 1), *dn = omd + 4 + 2 * ((cls >> 1) & 1);
  float4 w;
  w.x = dp[1];
  w.y = dp[0] - dp[1];
  w.z = lp.scale * dn[1];
  w.w = lp.scale * dn[0] - w.z;
  return w;
}
// Weights by the code in a point's w (kNoNormalW, 1, 2, 3, 4): entry
// weight_entry(w) of a table of kWeightEntries, so that the lookup is a shift
// and one 128-bit read instead of a conversion, four reads and their sums.
constexpr int kWeightEntries = 7;
__device__ __forceinline__ int weight_entry(float w) {
  return (int)min((__float_as_uint(w) >> 22) - 0xFCu, (unsigned)kWeightEntries - 1u);
}
// Entry e of that table: the codes' floats lie at 0 (0.5), 2 (1.0), 4 (2.0), 5 (3.0) and 6 (4.0).
__device__ __forceinline__ float4 table_weights(const LinParams &lp, const float *omd, int e) {
  const int cls = e == 2 ? 0 : e - 3;
  return e < 2 || e == 3 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : class_weights(lp, omd, cls);
}

// w: the point's weights (class_weights; zero without a normal).  kPlain: the
// defaults (robust kernel, no z scaling, not demoted).  False when the pixel
// adds nothing (an outlier without the robust kernel).
template <bool kPlain>
__device__ __forceinline__ bool pixel_terms(const LinParams &lp, float4 w, float3 rp, float3 rn, float4 cpt, float4 cn,
                                            PixelTerms &o) {
  float alp = w.x, bep = w.y, aln = w.z, ben = w.w;
  if (!kPlain && lp.z_scaling) {
    float f = 1.0f / fabsf(cpt.z);
    alp *= f; bep *= f; aln *= f; ben *= f;
  }
  if (!kPlain && lp.demoted) { aln = 0.0f; ben = 0.0f; }
  const float ux = cn.x, uy = cn.y, uz = cn.z;
  float pe0 = rp.x - cpt.x, pe1 = rp.y - cpt.y, pe2 = rp.z - cpt.z;
  float ne0 = rn.x - cn.x, ne1 = rn.y - cn.y, ne2 = rn.z - cn.z;
  const float bu = bep * fmaf(uz, pe2, fmaf(uy, pe1, ux * pe0));
  const float bv = ben * fmaf(uz, ne2, fmaf(uy, ne1, ux * ne0));
  float ep0 = fmaf(bu, ux, alp * pe0), ep1 = fmaf(bu, uy, alp * pe1), ep2 = fmaf(bu, uz, alp * pe2);
  float en0 = fmaf(bv, ux, aln * ne0), en1 = fmaf(bv, uy, aln * ne1), en2 = fmaf(bv, uz, aln * ne2);
  float le = fmaf(ne2, en2, fmaf(ne1, en1, fmaf(ne0, en0, fmaf(pe2, ep2, fmaf(pe1, ep1, pe0 * ep0)))));
  if (le > lp.max_chi2) {
    if (!kPlain && !lp.robust) return false;
    const float ks = lp.max_chi2 / le;
    le *= ks;
    alp *= ks; bep *= ks; aln *= ks; ben *= ks;
    ep0 *= ks; ep1 *= ks; ep2 *= ks;
    en0 *= ks; en1 *= ks; en2 *= ks;
  }
  o.ux = ux; o.uy = uy; o.uz = uz; o.be = bep;
  o.a = rp.x; o.b = rp.y; o.c = rp.z; o.al = alp;
  o.an = rn.x; o.bn = rn.y; o.cn = rn.z; o.aln = aln;
  o.ep0 = ep0; o.ep1 = ep1; o.ep2 = ep2; o.ben = ben;
  o.en0 = en0; o.en1 = en1; o.en2 = en2; o.le = le;
  return true;
}

// Htt, Htr, bt and br (v[0..14], v[21..26])
__device__ __forceinline__ void add_pose_terms(const PixelTerms &p, float *v) {
  // Htt += Omega_p
  const float t0 = p.be * p.ux, t1 = p.be * p.uy, t2 = p.be * p.uz;
  v[0] = fmaf(t0, p.ux, v[0] + p.al);
  v[1] = fmaf(t0, p.uy, v[1]);
  v[2] = fmaf(t1, p.uy, v[2] + p.al);
  v[3] = fmaf(t0, p.uz, v[3]);
  v[4] = fmaf(t1, p.uz, v[4]);
  v[5] = fmaf(t2, p.uz, v[5] + p.al);
  // Htr += Omega_p S = alp S + bep u wp^T, S = [[0, c, -b], [-c, 0, a], [b, -a, 0]]
  const float wp0 = fmaf(p.b, p.uz, -p.c * p.uy), wp1 = fmaf(p.c, p.ux, -p.a * p.uz),
              wp2 = fmaf(p.a, p.uy, -p.b * p.ux);
  v[6] = fmaf(t0, wp0, v[6]);
  v[7] = fmaf(t0, wp1, fmaf(p.al, p.c, v[7]));
  v[8] = fmaf(t0, wp2, fmaf(-p.al, p.b, v[8]));
  v[9] = fmaf(t1, wp0, fmaf(-p.al, p.c, v[9]));
  v[10] = fmaf(t1, wp1, v[10]);
  v[11] = fmaf(t1, wp2, fmaf(p.al, p.a, v[11]));
  v[12] = fmaf(t2, wp0, fmaf(p.al, p.b, v[12]));
  v[13] = fmaf(t2, wp1, fmaf(-p.al, p.a, v[13]));
  v[14] = fmaf(t2, wp2, v[14]);
  // bt += ep; br += Sp^T ep + Sn^T en (S^T e = v x e)
  v[21] += p.ep0; v[22] += p.ep1; v[23] += p.ep2;
  v[24] = fmaf(p.bn, p.en2, fmaf(-p.cn, p.en1, fmaf(p.b, p.ep2, fmaf(-p.c, p.ep1, v[24]))));
  v[25] = fmaf(p.cn, p.en0, fmaf(-p.an, p.en2, fmaf(p.c, p.ep0, fmaf(-p.a, p.ep2, v[25]))));
  v[26] = fmaf(p.an, p.en1, fmaf(-p.bn, p.en0, fmaf(p.a, p.ep1, fmaf(-p.b, p.ep0, v[26]))));
}

// Hrr and chi2 (v[15..20], v[27]):
// Hrr += S^T Omega_p S + Sn^T Omega_n Sn
//      = alp (|v|^2 I - v v^T) + aln (|vn|^2 I - vn vn^T) + bep wp wp^T + ben wn wn^T
__device__ __forceinline__ void add_rotation_terms(const PixelTerms &p, float *v) {
  v[27] += p.le;
  const float a = p.a, b = p.b, c = p.c, an = p.an, bn = p.bn, cn2 = p.cn;
  const float wp0 = fmaf(b, p.uz, -c * p.uy), wp1 = fmaf(c, p.ux, -a * p.uz), wp2 = fmaf(a, p.uy, -b * p.ux);
  const float wn0 = fmaf(bn, p.uz, -cn2 * p.uy), wn1 = fmaf(cn2, p.ux, -an * p.uz), wn2 = fmaf(an, p.uy, -bn * p.ux);
  const float qa = p.al * a, qb = p.al * b, qc = p.al * c;
  const float qan = p.aln * an, qbn = p.aln * bn, qcn = p.aln * cn2;
  const float pw0 = p.be * wp0, pw1 = p.be * wp1, pw2 = p.be * wp2;
  const float nw0 = p.ben * wn0, nw1 = p.ben * wn1, nw2 = p.ben * wn2;
  v[15] = fmaf(nw0, wn0, fmaf(pw0, wp0, fmaf(qcn, cn2, fmaf(qbn, bn, fmaf(qc, c, fmaf(qb, b, v[15]))))));
  v[16] = fmaf(nw1, wn0, fmaf(pw1, wp0, fmaf(-qbn, an, fmaf(-qb, a, v[16]))));
  v[17] = fmaf(nw1, wn1, fmaf(pw1, wp1, fmaf(qcn, cn2, fmaf(qan, an, fmaf(qc, c, fmaf(qa, a, v[17]))))));
  v[18] = fmaf(nw2, wn0, fmaf(pw2, wp0, fmaf(-qcn, an, fmaf(-qc, a, v[18]))));
  v[19] = fmaf(nw2, wn1, fmaf(pw2, wp1, fmaf(-qcn, bn, fmaf(-qc, b, v[19]))));
  v[20] = fmaf(nw2, wn2, fmaf(pw2, wp2, fmaf(qbn, bn, fmaf(qan, an, fmaf(qb, b, fmaf(qa, a, v[20]))))));
}

template <bool kPlain>
__device__ __forceinline__ void lin_terms_structured_xf(const LinParams &lp, float4 w, float3 rp, float3 rn, float4 cpt,
                                                       float4 cn, Acc &acc) {
  PixelTerms p;
  if (!pixel_terms<kPlain>(lp, w, rp, rn, cpt, cn, p)) return;
  acc.cnt += Acc::kInlier;
  add_pose_terms(p, acc.v);
  add_rotation_terms(p, acc.v);
}

// Reduces every thread's Acc to one FP64 partial of the CTA (fixed order).
// (A pairwise FP32 tree inside the warp measured 3 % faster but moved an
// ill-conditioned pose -- a frame against a subscene rendered from a merged
// scene -- from 1e-5 to 2e-5 rad of the FP64 oracle: the warp sums stay FP64.)
template <int kThreads>
__device__ __forceinline__ void block_reduce_store(const Acc &acc, double *out) {
  __shared__ double wsum[kThreads / 32][32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double v[32];
#pragma unroll
  for (int k = 0; k < 31; k++) v[k] = (double)acc.get(k);
  v[31] = 0.0;
  // butterfly reduce-scatter: lane L ends with the warp total of element L
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < off; j++) {
      double send = upper ? v[j] : v[j + off];
      double keep = upper ? v[j + off] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  wsum[wid][lane] = v[0];
  __syncthreads();
  if (wid == 0) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) s += wsum[w][lane];
    out[lane] = s * acc_scale(lane);
  }
}

// ---- fused correspondence + linearizer: persistent, cp.async-pipelined.
// A pair image is cut into tiles of kCorrTilePixels; every tile yields one
// FP64 partial, so results do not depend on the grid or the batch.  A CTA
// walks its tiles (blockIdx.x, +gridDim.x, ...) in sub-tiles of 256 pixels
// (kFusedPX per thread, at slots t and t + kFusedThreads, so that every
// access of one slot row is coalesced; the per-sub-tile bookkeeping and the
// per-tile reduction are shared by a thread's pixels).  For each pixel the
// thread reads the two indices, then
// stages the 7 gathered float4 (reference point and normal, current point
// and normal, 3 x Omega) into its own shared-memory slot with cp.async;
// kCorrStages sub-tiles are in flight while the oldest one is gated and
// linearized.  Each thread reads back only what it copied itself, so the
// gathered data needs no barrier.
constexpr int kFusedThreads = 128;
constexpr int kFusedPX = 2;
constexpr int kSubPix = kFusedThreads * kFusedPX;        // pixels per sub-tile
constexpr int kSubsPerTile = kCorrTilePixels / kSubPix;  // 4
constexpr int kCorrStages = 3;  // general Omega: gather, gate + Omega gather, linearize
// The only data threads share are a tile's constants (transforms, Omega
// parameters, pair, skip flags) and the per-tile reduction.  The constants
// live in a ring of kConstSlots tiles and the CTA meets at a barrier once per
// tile, in the iteration that writes the next tile's constants: tile U's are
// written before the barrier of iteration 4U - 1 (4U - 2 with three stages)
// and read in iterations up to 4U + 3, and their slot is rewritten for tile
// U + kConstSlots only after the barrier of iteration 4U + 4 kConstSlots - 5
// (- 6), which every thread reaches after its iteration 4U + 3 when
// kConstSlots >= 3.  The reduction's own barrier orders its shared sums.
constexpr int kConstSlots = 4;
#ifndef NICP_CORR_S_STAGES
#define NICP_CORR_S_STAGES 2      // structured Omega: gather, gate + linearize
#endif

// Structure-of-arrays stage: thread t owns slots t + k kFusedThreads of
// every array, so a warp's accesses to one field are consecutive 16-byte
// words (no bank conflicts).
struct GatherStageS {  // structured Omega: rebuilt from the current normal
  float4 rp[kSubPix], rn[kSubPix], cp[kSubPix], cn[kSubPix];
};
struct GatherStageG : GatherStageS {  // general Omega: gathered for accepted pixels
  float4 o0[kSubPix], o1[kSubPix], o2[kSubPix];
  int valid[kSubPix], ci[kSubPix];
};
#ifndef NICP_CORR_S_CTAS
#define NICP_CORR_S_CTAS 5
#endif
template <bool kStructured>
using GatherStage = typename std::conditional<kStructured, GatherStageS, GatherStageG>::type;

// block_reduce_store for the fused kernel, with the warp's step done
// through shared memory instead of a shuffle butterfly: the warp's 32 x 31
// partial sums are written to the warp's own slots of the stage it has just
// consumed (rp, rn, cp, cn at slots 32w.. and 128 + 32w..: eight runs of
// four 32-float rows), and lane L < 31 then sums row L -- the 32 lanes'
// partials of element L -- in FP64, in a fixed order (each lane starts its
// row at another 16-byte column, so that the eight lanes of a quarter-warp
// read eight different bank groups).  The warps' totals are added in FP64
// as in block_reduce_store.  The barrier inside also orders the row reads
// before the next gathers into these slots.
template <int kThreads, class StageT>
__device__ __forceinline__ void block_reduce_store_staged(const Acc &acc, double *out, StageT &g) {
  __shared__ double wsum[kThreads / 32][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float *base = reinterpret_cast<float *>(&g.rp[0]);
  auto row_of = [&](int k) {  // element k: run k / 4, row k % 4 of the warp's region
    const int run = k >> 2;
    return base + 4 * ((run >> 1) * kSubPix + (run & 1) * kFusedThreads + 32 * wid) + 32 * (k & 3);
  };
  __syncwarp();  // every lane of the warp is done with its slots of this stage
#pragma unroll
  for (int k = 0; k < 31; k++) row_of(k)[lane] = acc.get(k);
  __syncwarp();
  double v = 0.0;
  if (lane < 31) {
    const float4 *r4 = reinterpret_cast<const float4 *>(row_of(lane));
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float4 x = r4[(q + lane) & 7];
      v += (double)x.x;
      v += (double)x.y;
      v += (double)x.z;
      v += (double)x.w;
    }
  }
  wsum[wid][lane] = v;
  __syncthreads();
  if (wid == 0) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) s += wsum[w][lane];
    out[lane] = s * acc_scale(lane);
  }
}
template <bool kStructured>
__host__ __device__ constexpr int corr_stages() { return kStructured ? NICP_CORR_S_STAGES : kCorrStages; }
template <bool kStructured>
constexpr int corr_smem() { return corr_stages<kStructured>() * (int)sizeof(GatherStage<kStructured>); }

// 16-byte gather into shared memory through L2 only (.cg): a gathered point
// or normal is read about once per pass, so caching it in L1 only displaces
// the index and descriptor lines the pipeline does reuse (0.97 against 1.02
// ms per launch with .ca).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// flags: bit0 read the reference index from the z-buffer (else ref_index),
// bit1 reset the z-buffer after reading, bit2 keep the resolved reference
// index image, bit3 statistics pass (gate with Tgate_used; ignores `done`).
// kStructured: every pair's current cloud has structured information
// matrices (no Omega gathers, smaller stages).  kPlain (structured): the
// options' defaults, decided on the host; kFirst: bits 0 and 1 of flags.  The
// pass is bound by the instructions it issues, a good part of which asked for
// options pixel by pixel.
template <bool kStructured, bool kPlain, bool kFirst>
__global__ void __launch_bounds__(kFusedThreads, kStructured ? NICP_CORR_S_CTAS : 3)
    k_corr_lin(const PairDev *__restrict__ pairs, int npairs, const int *__restrict__ tile_pair, int first_tile,
               int total_tiles, CorrParams cp, LinParams lp, int flags) {
  extern __shared__ __align__(16) unsigned char corr_smem_raw[];
  using Stage = GatherStage<kStructured>;
  Stage *stages = reinterpret_cast<Stage *>(corr_smem_raw);
  const int t = threadIdx.x;
  // per-tile constants for the two tiles the pipeline can span:
  // [0..11] gating T, [12..23] linearizer T, the Omega weights by point code,
  // then pair index, skip flag and structured-Omega flag
  __shared__ float sT[kConstSlots][24];
  __shared__ float4 sW[kConstSlots][kWeightEntries];
  __shared__ int sPair[kConstSlots], sSkip[kConstSlots], sStruct[kConstSlots], sSame[kConstSlots];
  const bool stats_pass = flags & 8;
  chain_next();  // the solve's CTAs
  if ((int)blockIdx.x >= total_tiles) return;
  const int ntiles = (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int nsub = ntiles * kSubsPerTile;
  const bool drop_no_normal = kPlain || !cp.demoted;
  const bool first = kPlain ? kFirst : (flags & 1) != 0, reset = kPlain ? kFirst : (flags & 2) != 0;
  auto tile_of = [&](int j) { return first_tile + (int)blockIdx.x + (j / kSubsPerTile) * (int)gridDim.x; };
  auto stage_of = [&](int j) -> Stage & { return stages[j % corr_stages<kStructured>()]; };

  // Tile -> pair lookups, cached per pipeline stage (a stage's tile changes
  // once every kSubsPerTile sub-tiles).
  int lt_tile = -1, lt_pi = 0, gt_tile = -1, gt_pi = 0, gt_ctile = -1, gt_rc = 0, gt_cc = 0;
  bool lt_skip = false, gt_skip = false;
  auto lookup = [&](int tile, int &ctile, int &cpi, bool &cskip) {
    if (tile != ctile) {
      ctile = tile;
      cpi = tile_pair[tile];  // filled once per alignment by k_begin_loop
      cskip = !stats_pass && pairs[cpi].state->done;
    }
  };

  // Phase I (one iteration ahead, plain loads into registers): the two index
  // words of the thread's pixels of sub-tile j.
  unsigned long long zI[kFusedPX];
  int cI[kFusedPX];
  auto load_indices = [&](int j) {
#pragma unroll
    for (int k = 0; k < kFusedPX; k++) {
      zI[k] = ~0ull;
      cI[k] = -1;
    }
    if (j >= nsub) return;
    int tile = tile_of(j);
    lookup(tile, lt_tile, lt_pi, lt_skip);
    if (lt_skip) return;
    const PairDev &pd = pairs[lt_pi];
    const int P = pd.rows * pd.cols;
    const int p0 = (tile - pd.tile_base) * kCorrTilePixels + (j % kSubsPerTile) * kSubPix + t;
#pragma unroll
    for (int k = 0; k < kFusedPX; k++) {
      const int p = p0 + k * kFusedThreads;
      if (p < P) {
        if (first) zI[k] = pd.zbuf[p];
        else cI[k] = pd.ref_index[p];  // stashed in cI until phase G1 reads the current index
        if (first) cI[k] = pd.cur_index[p];
        else zI[k] = (unsigned long long)(unsigned)pd.cur_index[p];
      }
    }
  };

  // Phase G1 (two sub-tiles ahead): decode the indices, reset the z-buffer,
  // gather points and normals of both clouds.
  // Returns the valid pixels (bit k) of a structured pass.
  auto issue_g1 = [&](int j) {
    Stage &g = stage_of(j);
    int ci[kFusedPX], valid[kFusedPX];
#pragma unroll
    for (int k = 0; k < kFusedPX; k++) {
      ci[k] = -1;
      valid[k] = 0;
    }
    if (j < nsub) {
      int tile = tile_of(j);
      lookup(tile, gt_tile, gt_pi, gt_skip);
      const PairDev &pd = pairs[gt_pi];
      if (!gt_skip) {
        if (gt_ctile != tile) {  // point counts, read once per tile
          gt_ctile = tile;
          gt_rc = *pd.ref_count;
          gt_cc = *pd.cur_count;
        }
        const int P = pd.rows * pd.cols;
        const int p0 = (tile - pd.tile_base) * kCorrTilePixels + (j % kSubsPerTile) * kSubPix + t;
#pragma unroll
        for (int k = 0; k < kFusedPX; k++) {
          const int p = p0 + k * kFusedThreads, sl = t + k * kFusedThreads;
          if (p < P) {
            int ri;
            if (first) {
              // an empty word (all ones) decodes to -1 with drop_no_normal
              // and to 2^31 - 1 without, which the bounds test below rejects
              const unsigned lo = (unsigned)zI[k];
              ri = (drop_no_normal && (lo & 1u)) ? -1 : (int)(lo >> 1);
              ci[k] = cI[k];
              // evict-first: the word is read again only by the next
              // projection, long after it would have left L2, where it
              // would displace the gathered clouds
              if (reset) __stcs(pd.zbuf + p, ~0ull);
              if (flags & 4) pd.ref_index[p] = ri;
            } else {
              ri = cI[k];
              ci[k] = (int)(unsigned)zI[k];
            }
            valid[k] = (unsigned)ri < (unsigned)gt_rc && (unsigned)ci[k] < (unsigned)gt_cc;
            if (!kPlain && valid[k] && cp.row_limit_threads > 1)
              valid[k] = p / pd.cols < (pd.rows / cp.row_limit_threads) * cp.row_limit_threads;
            if (valid[k]) {
              cp_async16(&g.rp[sl], pd.ref_pts + ri);
              cp_async16(&g.rn[sl], pd.ref_nrm + ri);
              cp_async16(&g.cp[sl], pd.cur_pts + ci[k]);
              cp_async16(&g.cn[sl], pd.cur_nrm + ci[k]);
            }
          }
        }
      }
    }
    unsigned bits = 0;
#pragma unroll
    for (int k = 0; k < kFusedPX; k++) {
      if constexpr (!kStructured) {
        g.ci[t + k * kFusedThreads] = ci[k];
        g.valid[t + k * kFusedThreads] = valid[k];
      } else {
        bits |= (valid[k] ? 1u : 0u) << k;
      }
    }
    cp_async_commit();
    return bits;
  };

  // Per-tile constants, written when the tile's first sub-tile enters G1.
  auto tile_constants = [&](int j) {
    if (j >= nsub || j % kSubsPerTile) return;
    int e = (j / kSubsPerTile) % kConstSlots;
    lookup(tile_of(j), gt_tile, gt_pi, gt_skip);
    const int pi = gt_pi;
    const PairState *st = pairs[pi].state;
    if (threadIdx.x < 24)
      sT[e][threadIdx.x] = threadIdx.x < 12 ? (stats_pass ? st->Tgate_used : st->Tgate)[threadIdx.x]
                                            : st->Tlin[threadIdx.x - 12];
    else if (threadIdx.x >= 32 && threadIdx.x < 32 + kWeightEntries)
      sW[e][threadIdx.x - 32] = table_weights(lp, pairs[pi].cur_omd, threadIdx.x - 32);
    if (threadIdx.x == 0) {
      sPair[e] = pi;
      sSkip[e] = st->done && !stats_pass;
      sStruct[e] = pairs[pi].cur_structured;
      // gating and linearizer transforms equal (first inner iteration): the
      // linearizer reuses the gate's transformed point and normal
      const float *tg = stats_pass ? st->Tgate_used : st->Tgate;
      int same = 1;
      for (int k = 0; k < 12; k++) same &= (tg[k] == st->Tlin[k]);
      sSame[e] = same;
    }
  };

  // Gate (one sub-tile ahead), then gather Omega only for accepted pairs.
  auto gate_g2 = [&](int j) {
    if (j < nsub) {
      Stage &g = stage_of(j);
      int e = (j / kSubsPerTile) % kConstSlots;
      if constexpr (kStructured) {
        // structured: nothing to gather after the gate; it runs with the
        // linearizer in the main step
        (void)g;
        (void)e;
      } else {
#pragma unroll
        for (int k = 0; k < kFusedPX; k++) {
          const int sl = t + k * kFusedThreads;
          int acc_ok = 0;
          if (g.valid[sl] && !sSkip[e]) {
            acc_ok = gate(cp, sT[e], g.rp[sl], g.rn[sl], g.cp[sl], g.cn[sl]) ? 2 : 1;
            if (acc_ok == 2 && !sStruct[e]) {
              const float4 *o = pairs[sPair[e]].cur_omg + 3 * (size_t)g.ci[sl];
              cp_async16(&g.o0[sl], o);
              cp_async16(&g.o1[sl], o + 1);
              cp_async16(&g.o2[sl], o + 2);
            }
          }
          g.valid[sl] = acc_ok;  // 0 none, 1 candidate rejected, 2 accepted
        }
      }
    }
    cp_async_commit();
  };

  Acc acc;
  acc.zero();
  // Linearizes sub-tile j (its gather -- and, for general Omega, its gate --
  // complete); at a tile's last sub-tile the CTA stores the tile's partial.
  auto consume = [&](int j, unsigned bits) {
    const int e = (j / kSubsPerTile) % kConstSlots;
    const int sub = j % kSubsPerTile;
    if (sub == 0) {
      acc.zero();
    }
    if (!sSkip[e]) {
      const Stage &g = stage_of(j);
#pragma unroll
      for (int k = 0; k < kFusedPX; k++) {
        const int sl = t + k * kFusedThreads;
        if constexpr (kStructured) {
          if ((bits >> k) & 1u) {
            acc.cnt += Acc::kCandidate;
            const float4 rp0 = g.rp[sl], rn0 = g.rn[sl], cpt = g.cp[sl], cn = g.cn[sl];
            float3 rp, rn;
            if (gate_t<kPlain>(cp, sT[e], rp0, rn0, cpt, cn, rp, rn)) {
              acc.cnt += Acc::kAccepted;
              if (!sSame[e] || (!kPlain && cp.demoted)) {
                rp = xform_point_g(sT[e] + 12, rp0);
                rn = xform_normal_g(sT[e] + 12, rn0);
              }
              lin_terms_structured_xf<kPlain>(lp, sW[e][weight_entry(cpt.w)], rp, rn, cpt, cn, acc);
            }
          }
        } else {
          const int v = g.valid[sl];
          if (v) acc.cnt += Acc::kCandidate;
          if (v == 2) {
            acc.cnt += Acc::kAccepted;
            if (sStruct[e])
              lin_terms_structured_xf<false>(lp, sW[e][weight_entry(g.cp[sl].w)], xform_point_g(sT[e] + 12, g.rp[sl]),
                                             xform_normal_g(sT[e] + 12, g.rn[sl]), g.cp[sl], g.cn[sl], acc);
            else
              lin_terms(lp, sT[e] + 12, g.rp[sl], g.rn[sl], g.cp[sl], g.cn[sl], g.o0[sl], g.o1[sl], g.o2[sl],
                        acc);
          }
        }
      }
      if (sub == kSubsPerTile - 1) {
        const PairDev &pd = pairs[sPair[e]];
        block_reduce_store_staged<kFusedThreads>(acc, pd.partials + (size_t)(tile_of(j) - pd.tile_base) * kPartialWords,
                                                 stage_of(j));
      }
    }
  };
  if constexpr (corr_stages<kStructured>() == 2) {
    // two stages: sub-tile j+1 is gathered while j is gated and linearized
    load_indices(0);
    tile_constants(0);
    unsigned bits = issue_g1(0);
    load_indices(1);
    __syncthreads();          // tile 0's constants visible
    for (int j = 0; j < nsub; j++) {
      tile_constants(j + 1);
      const unsigned next = issue_g1(j + 1);  // uses the indices loaded in the previous iteration
      load_indices(j + 2);
      if ((j + 1) % kSubsPerTile == 0) __syncthreads();  // the next tile's constants visible
      cp_async_wait<1>();     // G1(j) complete (G1(j+1) may be in flight)
      consume(j, bits);
      bits = next;
    }
  } else {
    // prologue: sub-tile 0 through G1 and the gate, sub-tile 1 through G1
    load_indices(0);
    tile_constants(0);
    issue_g1(0);
    load_indices(1);
    tile_constants(1);
    issue_g1(1);
    load_indices(2);
    __syncthreads();
    cp_async_wait<1>();
    gate_g2(0);
    for (int j = 0; j < nsub; j++) {
      tile_constants(j + 2);
      issue_g1(j + 2);          // uses the indices loaded in the previous iteration
      load_indices(j + 3);
      if ((j + 2) % kSubsPerTile == 0) __syncthreads();  // the constants of j + 2's tile visible
      cp_async_wait<2>();       // G1(j+1) complete (groups after it: G2(j), G1(j+2))
      gate_g2(j + 1);
      cp_async_wait<2>();       // G2(j) complete (groups after it: G1(j+2), G2(j+1))
      consume(j, 0u);
    }
  }
  cp_async_wait<0>();
}

// ---- the same pass for few tiles: one CTA per tile, everything in flight.
// With one tile per CTA the pipeline above has nothing to overlap: a launch
// of 19 to 300 tiles took 9 to 11 us, the latency of one tile -- eight pixels
// one after the other in each of 128 threads, their indices and points
// fetched sub-tile by sub-tile.  Here 256 threads take a tile: all indices,
// then all gathers are issued at once; a thread gates and forms the terms of
// four pixels (PixelTerms, left in place of the gathered points), and the
// sums of a slot -- the slot t, t + 128, ... of the thread t above -- are
// taken over by two warps, one for each set of accumulators.  Every sum has
// the terms and the order of k_corr_lin, so both give the same bits.  Loops
// stay rolled: each instruction runs once or twice per launch, and fetching
// them is a good part of its time.
constexpr int kTileThreads = 256;
constexpr int kTileRows = kCorrTilePixels / kFusedThreads;  // pixels of a slot: 8
constexpr int kTileHalf = kCorrTilePixels / 2;
constexpr int kTileCtas = 3;
struct TileSmem {
  float4 px[2][4][kTileHalf];  // per half tile: points and normals of both clouds, then four parts of the terms
  float4 last[kTileHalf];      // the fifth part of the half at hand; then the sums' rows
};

// Grid (tiles of the largest pair image, pairs).
__global__ void __launch_bounds__(kTileThreads, kTileCtas)
    k_corr_tile(const PairDev *__restrict__ pairs, CorrParams cp, LinParams lp, int flags) {
  extern __shared__ __align__(16) unsigned char tile_smem_raw[];
  TileSmem &sm = *reinterpret_cast<TileSmem *>(tile_smem_raw);
  __shared__ float sT[24];
  __shared__ float4 sW[kWeightEntries];
  __shared__ unsigned counts[kTileThreads / 32];
  __shared__ double wsum[4][32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const bool stats_pass = flags & 8;
  const bool drop_no_normal = !cp.demoted;
  const PairDev &pd = pairs[blockIdx.y];
  const PairState *st = pd.state;
  const int rows = pd.rows, cols = pd.cols, P = rows * cols;
  const int p0 = (int)blockIdx.x * kCorrTilePixels + t;
  if ((int)blockIdx.x * kCorrTilePixels >= P) return;
  const int nref = *pd.ref_count, ncur = *pd.cur_count;
  const float4 *ref_pts = pd.ref_pts, *ref_nrm = pd.ref_nrm, *cur_pts = pd.cur_pts, *cur_nrm = pd.cur_nrm;
  unsigned long long *zbuf = pd.zbuf;
  int32_t *ref_index = pd.ref_index;
  int ci[4], ri[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + k * kTileThreads;
    ci[k] = p < P ? pd.cur_index[p] : -1;  // written before the loop
  }
  if (t >= 32 && t < 32 + kWeightEntries) sW[t - 32] = table_weights(lp, pd.cur_omd, t - 32);
  chain();
  // one round trip: the pair's flag and transforms, the pixels' indices
  const int done = __ldcg(&st->done);
  unsigned long long z[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + k * kTileThreads;
    z[k] = ~0ull;
    if (p < P) z[k] = (flags & 1) ? __ldcg(zbuf + p) : (unsigned long long)(unsigned)__ldcg(ref_index + p);
  }
  bool same_t = true;
  if (t < 12) {
    const float a = __ldcg((stats_pass ? st->Tgate_used : st->Tgate) + t), b = __ldcg(st->Tlin + t);
    sT[t] = a;
    sT[12 + t] = b;
    same_t = a == b;
  }
  if (!stats_pass && done) return;
  unsigned cnt = 0;
  unsigned valid = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = p0 + k * kTileThreads;
    ri[k] = (int)(unsigned)z[k];
    if (flags & 1) {
      // (an empty word decodes to an index beyond every cloud, or to -1)
      const unsigned lo = (unsigned)z[k];
      ri[k] = (drop_no_normal && (lo & 1u)) ? -1 : (int)(lo >> 1);
      if (p < P && (flags & 2)) __stcs(zbuf + p, ~0ull);
      if (p < P && (flags & 4)) ref_index[p] = ri[k];
    }
    bool ok = p < P && (unsigned)ri[k] < (unsigned)nref && (unsigned)ci[k] < (unsigned)ncur;
    if (ok && cp.row_limit_threads > 1) ok = p / cols < (rows / cp.row_limit_threads) * cp.row_limit_threads;
    if (ok) {
      const int at = t + (k & 1) * kTileThreads;
      cp_async16(&sm.px[k >> 1][0][at], ref_pts + ri[k]);
      cp_async16(&sm.px[k >> 1][1][at], ref_nrm + ri[k]);
      cp_async16(&sm.px[k >> 1][2][at], cur_pts + ci[k]);
      cp_async16(&sm.px[k >> 1][3][at], cur_nrm + ci[k]);
      cnt += Acc::kCandidate;
      valid |= 1u << k;
    }
    if (k & 1) cp_async_commit();
  }
  float v[28];
#pragma unroll
  for (int k = 0; k < 28; k++) v[k] = 0.0f;
  const int group = wid & 3;       // slots 32 group .. 32 group + 31
  const bool rotation = wid >= 4;  // the set of accumulators (uniform in the warp)
  const bool same = __syncthreads_and(same_t) != 0;  // and the constants are visible
  cp_async_wait<1>();
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    // gates and terms of a thread's two pixels (each reads what it copied itself)
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
      const int at = t + k * kTileThreads;
      PixelTerms o = {};
      if ((valid >> (2 * h + k)) & 1u) {
        const float4 rp0 = sm.px[h][0][at], rn0 = sm.px[h][1][at], cpt = sm.px[h][2][at], cn = sm.px[h][3][at];
        float3 rp, rn;
        if (gate_t(cp, sT, rp0, rn0, cpt, cn, rp, rn)) {
          cnt += Acc::kAccepted;
          if (!same || cp.demoted) {
            rp = xform_point_g(sT + 12, rp0);
            rn = xform_normal_g(sT + 12, rn0);
          }
          PixelTerms q;
          if (pixel_terms<false>(lp, sW[weight_entry(cpt.w)], rp, rn, cpt, cn, q)) {
            cnt += Acc::kInlier;
            o = q;
          }
        }
      }
      sm.px[h][0][at] = make_float4(o.ux, o.uy, o.uz, o.be);
      sm.px[h][1][at] = make_float4(o.a, o.b, o.c, o.al);
      sm.px[h][2][at] = make_float4(o.an, o.bn, o.cn, o.aln);
      sm.px[h][3][at] = make_float4(o.ep0, o.ep1, o.ep2, o.ben);
      sm.last[at] = make_float4(o.en0, o.en1, o.en2, o.le);
    }
    __syncthreads();
#pragma unroll 1
    for (int m = 0; m < kTileRows / 2; m++) {
      const int at = m * kFusedThreads + 32 * group + lane;
      const float4 r0 = sm.px[h][0][at], r1 = sm.px[h][1][at], r2 = sm.px[h][2][at], r3 = sm.px[h][3][at],
                   r4 = sm.last[at];
      const PixelTerms o = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y,
                            r2.z, r2.w, r3.x, r3.y, r3.z, r3.w, r4.x, r4.y, r4.z, r4.w};
      if (rotation) add_rotation_terms(o, v);
      else add_pose_terms(o, v);
    }
    cp_async_wait<0>();
    __syncthreads();  // sm.last has been read
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);  // (10 bits each: at most 128 pixels a warp)
  if (lane == 0) counts[wid] = cnt;
  // rows of 32 slots per group and element; lane L adds row L in FP64, in
  // block_reduce_store_staged's order
  float *row0 = reinterpret_cast<float *>(sm.px) + group * 28 * 32;
#pragma unroll
  for (int k = 0; k < 28; k++) {
    const bool rot = (k >= 15 && k <= 20) || k == 27;
    if (rot == rotation) row0[32 * k + lane] = v[k];
  }
  __syncthreads();
  if (wid < 4) {
    double d = 0.0;
    if (lane < 28) {
      const float4 *r4 = reinterpret_cast<const float4 *>(row0 + 32 * lane);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float4 x = r4[(q + lane) & 7];
        d += (double)x.x;
        d += (double)x.y;
        d += (double)x.z;
        d += (double)x.w;
      }
    }
    wsum[wid][lane] = d;
  }
  __syncthreads();
  if (wid == 0) {
    double d = 0.0;
    if (lane < 28) {
#pragma unroll
      for (int w = 0; w < 4; w++) d += wsum[w][lane];
    } else if (lane < 31) {
      int n = 0;
#pragma unroll
      for (int w = 0; w < kTileThreads / 32; w++) n += (int)((counts[w] >> (10 * (lane - 28))) & 1023u);
      d = (double)n;
    }
    pd.partials[(size_t)blockIdx.x * kPartialWords + lane] = d * acc_scale(lane);
  }
}

// ------------------------------------------------------------ list mode
// CorrespondenceFinderProjective::_computeMulti for reference pixel p
// (correspondencefinderprojective.cpp:150-240): the best current point of
// the window of rows [r - R, r + R] x cols [c - C, c + C] (clamped), scanned
// row-major with the reference's gate order and its replacement rule
// (strictly closer AND strictly better aligned); -1 when none passes.
__device__ int multi_best(const PairDev &pd, const CorrParams &cp, const float *Tg, int p, int ri, int ncur) {
  const float4 rn0 = pd.ref_nrm[ri];
  if (normal_is_zero(rn0.x, rn0.y, rn0.z)) return -1;
  const float3 rp = xform_point_g(Tg, pd.ref_pts[ri]);
  const float3 rn = xform_normal_g(Tg, rn0);
  float kr = rn0.w;
  if (kr < cp.flat_thr) kr = cp.flat_thr;
  const int r = p / pd.cols, c = p - r * pd.cols;
  const int r0 = max(r - cp.row_search, 0), r1 = min(r + cp.row_search + 1, pd.rows);
  const int c0 = max(c - cp.col_search, 0), c1 = min(c + cp.col_search + 1, pd.cols);
  int best = -1;
  float bestN = 0.0f, bestD = 1e20f;
  for (int r2 = r0; r2 < r1; r2++)
    for (int c2 = c0; c2 < c1; c2++) {
      const int ci = pd.cur_index[r2 * pd.cols + c2];
      if (ci < 0 || ci >= ncur) continue;
      const float4 cn = pd.cur_nrm[ci];
      if (normal_is_zero(cn.x, cn.y, cn.z)) continue;
      const float nd = dot3g(cn.x, cn.y, cn.z, rn.x, rn.y, rn.z);
      if (nd < cp.cos_thr) continue;
      const float4 cpt = pd.cur_pts[ci];
      const float dx = fsb(cpt.x, rp.x), dy = fsb(cpt.y, rp.y), dz = fsb(cpt.z, rp.z);
      const float d = dot3g(dx, dy, dz, dx, dy, dz);
      if (d > cp.sq_thr) continue;
      float kc = cn.w;
      if (kc < cp.flat_thr) kc = cp.flat_thr;
      const float ratio = __double2float_rn(__ddiv_rn(__dadd_rn((double)kr, 1e-5), __dadd_rn((double)kc, 1e-5)));
      if (ratio < cp.min_ratio || ratio > cp.max_ratio) continue;
      if (best == -1 || (d < bestD && nd > bestN)) {
        best = ci;
        bestN = nd;
        bestD = d;
      }
    }
  return best;
}

// Gate decisions of four consecutive pixels (bit k: pixel pix0 + k has a
// correspondence) and the current point each one takes.
__device__ __forceinline__ unsigned list_mask(const PairDev &pd, const CorrParams &cp, const float *Tg, int pix0,
                                              int P, int rmax, int *cur_of) {
  unsigned m = 0;
  const int nref = *pd.ref_count, ncur = *pd.cur_count;
  const bool multi = cp.row_search > 0 || cp.col_search > 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    cur_of[k] = -1;
    int p = pix0 + k;
    if (p >= P) break;
    int ri = pd.ref_index[p];
    if (ri < 0 || ri >= nref || p / pd.cols >= rmax) continue;
    if (multi) {
      cur_of[k] = multi_best(pd, cp, Tg, p, ri, ncur);
      if (cur_of[k] >= 0) m |= 1u << k;
      continue;
    }
    int ci = pd.cur_index[p];
    if (ci < 0 || ci >= ncur) continue;
    cur_of[k] = ci;
    if (gate(cp, Tg, pd.ref_pts[ri], pd.ref_nrm[ri], pd.cur_pts[ci], pd.cur_nrm[ci])) m |= 1u << k;
  }
  return m;
}

__global__ void __launch_bounds__(kCorrThreads) k_corr_count(const PairDev *__restrict__ pairs, int npairs, CorrParams cp,
                                                             int use_state_T, const float *__restrict__ explicit_T) {
  __shared__ int red[32];
  int pi = find_pair(pairs, npairs, blockIdx.x);
  const PairDev &pd = pairs[pi];
  if (use_state_T && pd.state->done) return;
  int tile = blockIdx.x - pd.tile_base;
  int P = pd.rows * pd.cols;
  int rmax = pd.rows;
  if (cp.row_limit_threads > 1) rmax = (pd.rows / cp.row_limit_threads) * cp.row_limit_threads;
  float Tg[12];
  const float *src = use_state_T ? pd.state->Tgate : explicit_T + 12 * pi;
#pragma unroll
  for (int k = 0; k < 12; k++) Tg[k] = src[k];
  int cur_of[4];
  unsigned m = list_mask(pd, cp, Tg, tile * kCorrTilePixels + threadIdx.x * 4, P, rmax, cur_of);
  int v = __popc(m);
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < kCorrThreads / 32; i++) t += red[i];
    pd.list_tile_counts[tile] = t;
  }
}

__global__ void __launch_bounds__(kCorrThreads) k_corr_write(const PairDev *__restrict__ pairs, int npairs, CorrParams cp,
                                                             int use_state_T, const float *__restrict__ explicit_T) {
  __shared__ int red[32];
  __shared__ int wsum[kCorrThreads / 32];
  int pi = find_pair(pairs, npairs, blockIdx.x);
  const PairDev &pd = pairs[pi];
  if (use_state_T && pd.state->done) return;
  int tile = blockIdx.x - pd.tile_base;
  int P = pd.rows * pd.cols;
  int ntiles = (P + kCorrTilePixels - 1) / kCorrTilePixels;
  int rmax = pd.rows;
  if (cp.row_limit_threads > 1) rmax = (pd.rows / cp.row_limit_threads) * cp.row_limit_threads;
  float Tg[12];
  const float *src = use_state_T ? pd.state->Tgate : explicit_T + 12 * pi;
#pragma unroll
  for (int k = 0; k < 12; k++) Tg[k] = src[k];
  int before = 0;
  for (int t = threadIdx.x; t < tile; t += blockDim.x) before += pd.list_tile_counts[t];
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = before;
  __syncthreads();
  before = 0;
  for (int i = 0; i < kCorrThreads / 32; i++) before += red[i];
  int pix0 = tile * kCorrTilePixels + threadIdx.x * 4;
  int cur_of[4];
  unsigned m = list_mask(pd, cp, Tg, pix0, P, rmax, cur_of);
  int cnt = __popc(m);
  int inc = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  int woff = 0, btot = 0;
  for (int i = 0; i < kCorrThreads / 32; i++) {
    if (i < wid) woff += wsum[i];
    btot += wsum[i];
  }
  int o = before + woff + inc - cnt;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (m & (1u << k)) {
      int p = pix0 + k;
      pd.pairs[2 * o] = pd.ref_index[p];
      pd.pairs[2 * o + 1] = cur_of[k];
      o++;
    }
  if (tile == ntiles - 1 && threadIdx.x == 0) *pd.num_pairs = before + btot;
}

// Linearizer::update over pd.pairs[0, K - K % T).  Tiles cover list slots.
// use_state_T: 0 explicit T, 1 the pair state's Tlin (skipping converged
// pairs), 2 the state's Tlin for every pair (statistics pass).
__global__ void __launch_bounds__(kCorrThreads) k_lin_list(const PairDev *__restrict__ pairs, int npairs, LinParams lp,
                                                           int parity_threads, int use_state_T,
                                                           const float *__restrict__ explicit_T) {
  int pi = find_pair(pairs, npairs, blockIdx.x);
  const PairDev &pd = pairs[pi];
  chain();
  if (use_state_T == 1 && pd.state->done) return;
  int tile = blockIdx.x - pd.tile_base;
  int K = *pd.num_pairs;
  if (parity_threads > 1) K = (K / parity_threads) * parity_threads;
  float Tl[12];
  const float *src = use_state_T ? pd.state->Tlin : explicit_T + 12 * pi;
#pragma unroll
  for (int k = 0; k < 12; k++) Tl[k] = src[k];
  const int nref = *pd.ref_count, ncur = *pd.cur_count;
  Acc acc;
  acc.zero();
  int i0 = tile * kCorrTilePixels + threadIdx.x * 4;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int i = i0 + k;
    if (i >= K) break;
    int ri = pd.pairs[2 * i], ci = pd.pairs[2 * i + 1];
    if (ri < 0 || ci < 0 || ri >= nref || ci >= ncur) continue;
    acc.cnt += Acc::kCandidate;
    acc.cnt += Acc::kAccepted;
    const float4 *o = pd.cur_omg + 3 * (size_t)ci;
    lin_terms(lp, Tl, pd.ref_pts[ri], pd.ref_nrm[ri], pd.cur_pts[ci], pd.cur_nrm[ci], o[0], o[1], o[2], acc);
  }
  block_reduce_store<kCorrThreads>(acc, pd.partials + (size_t)tile * kPartialWords);
}

// ------------------------------------------------------------ solve
// ---- the 6x6 solve and the pose update, by one warp.
// The chain of divisions, square roots and 4x4 products is short on work and
// long on latency, so a lane owns an entry, independent divisions run in
// different lanes and code stays short.  Every entry is formed by the same
// operations in the same order as one thread would form it.
struct SolveScratch {
  double L[36];  // factor: row = unknown, column = step
  double x[6];
  double T[16], invT[16], Tstart[16], off[16], dT[16], A[16], B[16];
};

__device__ __forceinline__ int nibble(unsigned w, int i) { return (int)((w >> (4 * i)) & 15u); }
// Lane that owns the unordered entry (i, j): the lower triangle row by row.
__device__ __forceinline__ int tri(int i, int j) {
  const int hi = max(i, j), lo = min(i, j);
  return hi * (hi + 1) / 2 + lo;
}

// M x = b by LDL^T with symmetric diagonal pivoting (Golub & Van Loan 4.2);
// lane tri(i, j) < 21 holds m = M_ij, lane i < 6 holds rhs = b_i; x to
// s.x.  Unknowns are never moved: `perm` (position -> unknown) and `pos`
// (unknown -> position) hold the order, six packed nibbles each, uniform in
// the warp.  A step is a maximum over the remaining diagonal (one integer
// reduction), three exchanges, one division and one FMA.
__device__ __forceinline__ void warp_ldlt_solve6(double m, double rhs, SolveScratch &s, int lane) {
  const unsigned kAll = 0xffffffffu;
  unsigned perm = 0x543210u, pos = 0x543210u;
  const int a = lane >= 21 ? 6 : lane >= 15 ? 5 : lane >= 10 ? 4 : lane >= 6 ? 3 : lane >= 3 ? 2 : lane >= 1 ? 1 : 0;
  const int b = a == 6 ? 6 : lane - a * (a + 1) / 2;
  double dpos = 1.0;  // lane i < 6: the pivot of position i
#pragma unroll
  for (int k = 0; k < 6; k++) {
    if (k < 5) {
      // lane = position: the first of the largest remaining diagonal entries
      const int u = nibble(perm, lane < 6 ? lane : 5);
      const double dl = fabs(__shfl_sync(kAll, m, tri(u, u)));
      const bool in = lane >= k && lane < 6;
      const unsigned nan = __ballot_sync(kAll, in && dl != dl);
      const unsigned hi = in && dl == dl ? (unsigned)__double2hiint(dl) : 0u;
      const unsigned top = __reduce_max_sync(kAll, hi);
      unsigned who = __ballot_sync(kAll, in && dl == dl && hi == top);
      if (__popc(who) > 1) {  // equal upper words: the lower ones decide
        const bool cand = (who >> lane) & 1u;
        const unsigned lo = cand ? (unsigned)__double2loint(dl) : 0u;
        const unsigned top_lo = __reduce_max_sync(kAll, lo);
        who = __ballot_sync(kAll, cand && lo == top_lo);
      }
      // a NaN never beats another entry and is never beaten in its own place
      const int piv = ((nan >> k) & 1u) || !who ? k : __ffs(who) - 1;
      const unsigned uk = nibble(perm, k), up = nibble(perm, piv);
      perm ^= ((uk ^ up) << (4 * k)) | ((uk ^ up) << (4 * piv));
      if (uk != up) pos ^= ((unsigned)(k ^ piv) << (4 * uk)) | ((unsigned)(k ^ piv) << (4 * up));
    }
    const int u = nibble(perm, k);
    const double d = __shfl_sync(kAll, m, tri(u, u));
    if (lane == k) dpos = d;
    if (k < 5) {
      const int pa = nibble(pos, a), pb = nibble(pos, b);
      const int hi = pa >= pb ? a : b, lo = pa >= pb ? b : a;
      const double ch = __shfl_sync(kAll, m, tri(hi, u)), cl = __shfl_sync(kAll, m, tri(lo, u));
      const bool left = a < 6 && pa > k && pb > k;
      const double l = (left ? ch : d) / d;  // (a lane that is done divides d by itself)
      if (left) m = m - l * cl;
      if (left && a == b) s.L[a * 6 + k] = l;
    }
  }
  __syncwarp();
  // L y = b, lane = unknown
  const int row = lane < 6 ? lane : 5, at = nibble(pos, row);
  double y = rhs;
#pragma unroll
  for (int j = 0; j < 5; j++) {
    const double yj = __shfl_sync(kAll, y, nibble(perm, j));
    if (at > j) y = y - s.L[row * 6 + j] * yj;
  }
  y = y / __shfl_sync(kAll, dpos, at);
  // L^T x = y, every lane the same, by position
  double x[6], l[6][6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    x[i] = __shfl_sync(kAll, y, nibble(perm, i));
#pragma unroll
    for (int j = 0; j < i; j++) l[i][j] = s.L[nibble(perm, i) * 6 + j];
  }
#pragma unroll
  for (int i = 4; i >= 0; i--)
#pragma unroll
    for (int j = i + 1; j < 6; j++) x[i] = x[i] - l[j][i] * x[j];
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 6; i++) s.x[nibble(perm, i)] = x[i];
  __syncwarp();
}

// C = A B (rows 0..3), lane < 16 an entry; C is another array than A and B.
__device__ __forceinline__ void warp_mm4(const double *A, const double *B, double *C, int lane) {
  if (lane < 16) {
    const double *r = A + (lane & 12), *c = B + (lane & 3);
    C[lane] = r[0] * c[0] + r[1] * c[4] + r[2] * c[8] + r[3] * c[12];
  }
  __syncwarp();
}
// R = T^-1 of an isometry, R another array than T.
__device__ __forceinline__ void warp_iso_inverse(const double *T, double *R, int lane) {
  if (lane < 16) {
    const int i = lane >> 2, j = lane & 3;
    double v = lane == 15 ? 1.0 : 0.0;
    if (i < 3) v = j < 3 ? T[j * 4 + i] : -(T[i] * T[3] + T[4 + i] * T[7] + T[8 + i] * T[11]);
    R[lane] = v;
  }
  __syncwarp();
}
// v2t by every lane; lane 0 stores.
__device__ __forceinline__ void warp_v2t(const double *x, double *T, int lane) {
  double t[16];
  d_v2t(x, t);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 16; k++) T[k] = t[k];
  __syncwarp();
}
// t2v by every lane, the quaternion's four divisions in four lanes.
__device__ __forceinline__ void warp_t2v(const double *T, double *x, int lane) {
  double q[4], n;
  d_quaternion(T, q, n);
  const double v = (lane == 0 ? q[0] : lane == 1 ? q[1] : lane == 2 ? q[2] : q[3]) / n;
  const bool flip = __shfl_sync(0xffffffffu, v, 3) < 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double c = __shfl_sync(0xffffffffu, v, k);
    x[3 + k] = flip ? -c : c;
    x[k] = T[4 * k + 3];
  }
}

// The matrices of an outer iteration that starts from sc.T (rows 0..3 of the
// pose), by one warp: T and its inverse, the projector's KRt for the pose
// T ref_offset (pinholepointprojector.cpp:16-31), the float transforms of the
// gates and the linearizer.  K: lane < 12 the row lane / 4 of the camera matrix.
__device__ __forceinline__ void warp_begin_outer(PairState *st, SolveScratch &sc, const double K[3], int lane) {
  warp_mm4(sc.T, sc.off, sc.A, lane);
  warp_iso_inverse(sc.A, sc.B, lane);  // the projector's inverse pose
  warp_iso_inverse(sc.T, sc.A, lane);  // invT
  if (lane < 16) {
    st->T[lane] = sc.T[lane];
    st->Tstart[lane] = sc.T[lane];
    st->invT[lane] = sc.A[lane];
  }
  if (lane < 12) {
    const int j = lane & 3;
    st->KRt[lane] = (float)(K[0] * sc.B[j] + K[1] * sc.B[4 + j] + K[2] * sc.B[8 + j]);
    const float f = (float)sc.A[lane];
    st->Tgate[lane] = f;
    st->Tlin[lane] = f;
  }
}

// ---- the sum of a pair's tile partials: kSumGroups warps take the tiles
// t = g, g + kSumGroups, ... each, then the groups are added; a fixed order,
// whatever the batch.  (Four groups, as before, left one SM with 75 partials
// a thread at 640x480: 4800 cycles of a 12500-cycle launch; 16 groups have
// all their loads in flight at once.)
constexpr int kSumGroups = 16, kSumThreads = 32 * kSumGroups;

__device__ __forceinline__ void sum_tile_partials(const double *src, int nt, bool f32, double (*part)[32]) {
  constexpr int kAhead = 8;
  const int e = threadIdx.x & 31, g = threadIdx.x >> 5;
  src += e;
  double s = 0.0;
  float s32 = 0.0f;
  for (int t = g; t < nt; t += kSumGroups * kAhead) {
    double v[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; q++) {
      const int u = t + kSumGroups * q;
      v[q] = u < nt ? __ldcg(src + (size_t)u * kPartialWords) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kAhead; q++) {
      if (f32) s32 += (float)v[q];  // precision study: the same order, in FP32
      else s += v[q];
    }
  }
  part[g][e] = f32 ? (double)s32 : s;
  __syncthreads();
}
__device__ __forceinline__ double sum_groups(double (*part)[32], bool f32, int e) {
  if (f32) {
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < kSumGroups; k++) t += (float)part[k][e];
    return (double)t;
  }
  double q[4];
#pragma unroll
  for (int k = 0; k < 4; k++)
    q[k] = ((part[4 * k][e] + part[4 * k + 1][e]) + part[4 * k + 2][e]) + part[4 * k + 3][e];
  return (q[0] + q[1]) + (q[2] + q[3]);
}

// mode: bit0 last inner iteration of the outer loop, bit1 reduce only (no
// pose update: Linearizer results of a list pass), bit2 statistics pass
// (reduce into Hstat only), kSolveCrossF32 sum the tile partials in FP32.
// The other warps only help to add the partials up; one of them writes the
// sums out while warp 0 solves.
__global__ void __launch_bounds__(kSumThreads) k_solve(const PairDev *__restrict__ pairs, int npairs, float lambda,
                                                      int mode, double early_eps, int ignore_done) {
  __shared__ double part[kSumGroups][32];
  __shared__ SolveScratch sc;
  const PairDev &pd = pairs[blockIdx.x];
  PairState *st = pd.state;
  const double *src = pd.partials;
  const int P = pd.rows * pd.cols;
  const int nt = (P + kCorrTilePixels - 1) / kCorrTilePixels;
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  // (the pose is older than the linearization that this launch waits for)
  if (g >= 2 && threadIdx.x < 64 + 48) {
    const int q = threadIdx.x - 64;
    const double *from = q < 16 ? st->invT : q < 32 ? st->Tstart : st->ref_offset;
    double *to = q < 16 ? sc.invT : q < 32 ? sc.Tstart : sc.off;
    to[q & 15] = from[q & 15];
  }
  const int iterations = st->iterations;
  const float gate_used = lane < 12 ? st->Tgate[lane] : 0.0f;
  double K[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 3; k++)
    if (lane < 12) K[k] = (double)pd.K[(lane >> 2) * 3 + k];
  chain();
  if (st->done && !ignore_done) return;
  sum_tile_partials(src, nt, (mode & kSolveCrossF32) != 0, part);
  const double tot = sum_groups(part, (mode & kSolveCrossF32) != 0, lane);
  // H's entry (i, j) in the sums: 0..5 Htt lower, 6..14 Htr row by row, 15..20 Hrr lower
  auto element = [](int i, int j) {
    const int hi = max(i, j), lo = min(i, j);
    return hi < 3 ? tri(hi, lo) : lo >= 3 ? 15 + tri(hi - 3, lo - 3) : 6 + lo * 3 + hi - 3;
  };
  if (g == 1) {
    double *H = (mode & 4) ? st->Hstat : st->H;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int k = min(lane + 32 * r, 35), i = k / 6, j = k - 6 * i;
      const double h = __shfl_sync(0xffffffffu, tot, element(i, j));
      if (lane + 32 * r < 36) H[k] = h;
    }
    if (!(mode & 4)) {
      if (lane >= 21 && lane < 27) st->b[lane - 21] = tot;
      if (lane == 27) st->error = (float)tot;
      if (lane == 28) st->inliers = (int)tot;
      if (lane == 29) st->candidates = (int)tot;
      if (lane == 30) st->num_corr = (int)tot;
    }
  }
  if (g != 0 || (mode & 6)) return;
  // H += lambda I; dx = H^-1 (-b); invT = v2t(dx) invT  (alignerprojective.cpp:72-95)
  {
    const int a = lane >= 15 ? 5 : lane >= 10 ? 4 : lane >= 6 ? 3 : lane >= 3 ? 2 : lane >= 1 ? 1 : 0;
    const int b = min(lane - a * (a + 1) / 2, 5);
    double m = __shfl_sync(0xffffffffu, tot, element(a, b));
    if (a == b) m = m + (double)lambda;
    const double rhs = -__shfl_sync(0xffffffffu, tot, 21 + (lane < 6 ? lane : 5));
    warp_ldlt_solve6(m, rhs, sc, lane);
  }
  warp_v2t(sc.x, sc.dT, lane);
  warp_mm4(sc.dT, sc.invT, sc.A, lane);  // the new invT
  if (lane >= 12 && lane < 16) sc.A[lane] = lane == 15 ? 1.0 : 0.0;
  __syncwarp();
  if (!(mode & 1)) {
    if (lane < 16) st->invT[lane] = sc.A[lane];
    if (lane < 12) st->Tlin[lane] = (float)sc.A[lane];
    return;
  }
  // T = invT^-1, renormalised through t2v/v2t (alignerprojective.cpp:98-100)
  double v[6];
  warp_iso_inverse(sc.A, sc.B, lane);
  warp_t2v(sc.B, v, lane);
  warp_v2t(v, sc.T, lane);
  if (lane == 0) st->iterations = iterations + 1;
  if (lane < 12) st->Tgate_used[lane] = gate_used;
  if (early_eps > 0) {
    warp_iso_inverse(sc.Tstart, sc.A, lane);
    warp_mm4(sc.T, sc.A, sc.B, lane);
    warp_t2v(sc.B, v, lane);
    double m = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) m = fmax(m, fabs(v[k]));
    if (lane == 0 && m < early_eps) st->done = 1;
    __syncwarp();
  }
  warp_begin_outer(st, sc, K, lane);  // the next outer iteration starts from T
}

// Everything a loop starts from, in one launch (four uploads, a memset and two
// small kernels took 28 us in front of a 20 us iteration): the descriptors,
// projection matrices and poses are read where the host wrote them (pinned
// memory), the pairs' states initialised, the tile -> pair table filled
// (tile_pair[tile] = the pair whose pixel image holds the tile, so that the
// persistent fused kernel finds it with one load) and the z-buffers emptied.
// CTA b: pairs b, b + gridDim.x, ..., and its share of the z-buffers.
__global__ void __launch_bounds__(256) k_begin_loop(BeginArgs a) {
  __shared__ SolveScratch sc;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (int pi = blockIdx.x; pi < a.npairs; pi += gridDim.x) {
    const PairDev &src = a.pairs[pi];
    if (wid == 0) {
      PairState *st = src.state;
      double K[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (lane < 12) K[k] = (double)src.K[(lane >> 2) * 3 + k];
      __syncwarp();  // (the pair before is done with sc)
      if (lane < 16) {
        sc.T[lane] = lane < 12 ? a.guess[16 * (size_t)pi + lane] : lane == 15 ? 1.0 : 0.0;
        const double r = a.roff[16 * (size_t)pi + lane];
        sc.off[lane] = r;
        st->ref_offset[lane] = r;
      }
      __syncwarp();
      warp_begin_outer(st, sc, K, lane);
      if (lane < 12) st->Tgate_used[lane] = st->Tgate[lane];
      for (int k = lane; k < 36; k += 32) st->H[k] = 0.0;
      if (lane < 6) st->b[lane] = 0.0;
      if (lane == 0) {
        st->error = 0;
        st->inliers = st->num_corr = st->candidates = st->iterations = st->done = st->status = 0;
      }
    } else if (wid == 1) {
      const unsigned *from = reinterpret_cast<const unsigned *>(&src);
      unsigned *to = reinterpret_cast<unsigned *>(a.dev_pairs + pi);
      for (int k = lane; k < (int)(sizeof(PairDev) / 4); k += 32) to[k] = from[k];
      if (a.dev_krt && lane < 12) a.dev_krt[12 * (size_t)pi + lane] = a.krt[12 * (size_t)pi + lane];
    } else if (a.tile_pair) {
      const int ntiles = (src.rows * src.cols + kCorrTilePixels - 1) / kCorrTilePixels;
      for (int k = t - 64; k < ntiles; k += 192) a.tile_pair[src.tile_base + k] = pi;
    }
  }
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (size_t k = (size_t)blockIdx.x * 256 + t; k < a.zbuf16; k += (size_t)gridDim.x * 256) a.zbuf[k] = ones;
}

// The pairs' states to the host (pinned memory), chained to the loop's last
// solve, which still writes them when this starts (no __restrict__).
__global__ void __launch_bounds__(256) k_publish(const uint4 *states, uint4 *host, size_t n) {
  chain();
  for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < n; k += (size_t)gridDim.x * 256)
    host[k] = __ldcg(states + k);
}
static_assert(sizeof(PairState) % 16 == 0 && sizeof(PairDev) % 4 == 0, "copied by words");

// ------------------------------------------------------------ launchers
// An SM changes its split of shared memory and L1 only while it is empty.
// The loop's kernels are chained, so all of them ask for the split of the
// fused kernel (its gather stages): otherwise its CTAs find SMs still set up
// for the projection's small need and fewer of them fit.  Once per device
// (std::call_once: host threads on other contexts wait rather than race).
static void configure_loop() {
  constexpr int kMaxDevices = 64;
  static std::once_flag once[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  auto set = [] {
    auto most_shared = [](auto *kernel) {
      cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    };
    most_shared(k_zbuffer<4>);
    most_shared(k_solve);
    most_shared(k_corr_tile);
    cudaFuncSetAttribute(k_corr_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem));
  };
  if (dev >= 0 && dev < kMaxDevices)
    std::call_once(once[dev], set);
  else
    set();
}

void launch_zbuffer(const PairDev *d_pairs, int npairs, int max_pt_tiles, int mode, const float *explicit_KRt,
                    int ppt, bool chained, cudaStream_t s, Profiler *prof) {
  if (max_pt_tiles <= 0 || npairs <= 0) return;
  configure_loop();
  prof->begin(NICP_K_ZBUFFER, s);
  const int kMaxGridY = 65535;
  for (int p0 = 0; p0 < npairs; p0 += kMaxGridY) {
    const dim3 g(max_pt_tiles, std::min(kMaxGridY, npairs - p0));
    switch (ppt) {
      case 1: launch(chained, k_zbuffer<1>, g, kPointsPerCta, 0, s, d_pairs, npairs, mode, explicit_KRt, p0); break;
      case 2: launch(chained, k_zbuffer<2>, g, kPointsPerCta / 2, 0, s, d_pairs, npairs, mode, explicit_KRt, p0); break;
      case 8: launch(chained, k_zbuffer<8>, g, kPointsPerCta / 8, 0, s, d_pairs, npairs, mode, explicit_KRt, p0); break;
      default: launch(chained, k_zbuffer<4>, g, kPointsPerCta / 4, 0, s, d_pairs, npairs, mode, explicit_KRt, p0); break;
    }
  }
  prof->end(NICP_K_ZBUFFER, s);
}

void launch_resolve(const PairDev *d_pairs, int npairs, int max_tiles, int to_ref, float *depth_out,
                    int drop_no_normal, bool chained, cudaStream_t s, Profiler *prof) {
  if (max_tiles <= 0 || npairs <= 0) return;
  configure_loop();
  prof->begin(NICP_K_RESOLVE, s);
  const int kMaxGridY = 65535;
  for (int p0 = 0; p0 < npairs; p0 += kMaxGridY)
    launch(chained, k_resolve, dim3(max_tiles, std::min(kMaxGridY, npairs - p0)), kCorrThreads, 0, s, d_pairs, npairs,
                   to_ref, depth_out, drop_no_normal, p0);
  prof->end(NICP_K_RESOLVE, s);
}

// Persistent grid: as many CTAs as fit on the device at once, never more
// than there are tiles.
// The shared-memory opt-in holds for the device that was current when it was
// set, and the occupancy is that device's: both are taken once per device
// (std::call_once: host threads on other contexts wait rather than race).
template <bool kStructured, bool kPlain, bool kFirst>
static int corr_lin_grid(int total_tiles, int ctas_per_sm) {
  struct Occupancy {
    int sm_count = 1, per_sm_max = 1;
  };
  constexpr int kMaxDevices = 64;
  static Occupancy occ[kMaxDevices];
  static std::once_flag once[kMaxDevices];
  auto query = [](int dev, Occupancy *o) {
    cudaFuncSetAttribute(k_corr_lin<kStructured, kPlain, kFirst>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         corr_smem<kStructured>());
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_corr_lin<kStructured, kPlain, kFirst>, kFusedThreads,
                                                  corr_smem<kStructured>());
    o->per_sm_max = std::max(1, per_sm);
    o->sm_count = std::max(1, sms);
  };
  int dev = 0;
  cudaGetDevice(&dev);
  Occupancy local;
  const Occupancy *o = &local;
  if (dev >= 0 && dev < kMaxDevices) {
    std::call_once(once[dev], query, dev, &occ[dev]);
    o = &occ[dev];
  } else {
    query(dev, &local);
  }
  const int resident = o->sm_count * o->per_sm_max;
  const int grid = (ctas_per_sm > 0 && ctas_per_sm < o->per_sm_max) ? o->sm_count * ctas_per_sm : resident;
  return std::min(total_tiles, grid);
}

template <bool kStructured, bool kPlain, bool kFirst>
static void corr_lin(const PairDev *d_pairs, int npairs, int first_tile, int total_tiles, const CorrParams &cp,
                     const LinParams &lp, int flags, int ctas_per_sm, const int *tile_pair, cudaStream_t s) {
  const int grid = corr_lin_grid<kStructured, kPlain, kFirst>(total_tiles, ctas_per_sm);
  k_corr_lin<kStructured, kPlain, kFirst><<<grid, kFusedThreads, corr_smem<kStructured>(), s>>>(
      d_pairs, npairs, tile_pair, first_tile, total_tiles, cp, lp, flags);
}

// Three CTAs of k_corr_tile fit on an SM.  Up to there the pass takes less
// than with k_corr_lin (19 tiles 9.3 -> 6.8 us, 300 tiles 11.3 -> 9.2 us after
// the projection's end); at 900 tiles, two waves, it takes more (22.4 us
// against 19.7), and over many tiles k_corr_lin's pipeline does 1.6 times the
// tiles per second.
bool few_tiles(int npairs, int max_tiles) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  return npairs <= 65535 && (long long)max_tiles * npairs <= (long long)kTileCtas * sms;
}

void launch_corr_tile(const PairDev *d_pairs, int npairs, int max_tiles, const CorrParams &cp, const LinParams &lp,
                      int flags, cudaStream_t s, Profiler *prof) {
  if (max_tiles <= 0 || npairs <= 0) return;
  configure_loop();
  prof->begin(NICP_K_CORR_LIN, s);
  launch(true, k_corr_tile, dim3(max_tiles, npairs), kTileThreads, sizeof(TileSmem), s, d_pairs, cp, lp, flags);
  prof->end(NICP_K_CORR_LIN, s);
}

void launch_corr_lin(const PairDev *d_pairs, int npairs, int first_tile, int total_tiles, const CorrParams &cp,
                     const LinParams &lp, int flags, bool structured, int ctas_per_sm, const int *tile_pair,
                     cudaStream_t s, Profiler *prof) {
  if (total_tiles <= 0) return;
  configure_loop();
  prof->begin(NICP_K_CORR_LIN, s);
  if (structured) {
    // (the reset goes with the first pass)
    const bool plain = !cp.demoted && cp.row_limit_threads <= 1 && !lp.demoted && !lp.z_scaling && lp.robust &&
                       ((flags & 3) == 0 || (flags & 3) == 3);
    if (plain && (flags & 1)) corr_lin<true, true, true>(d_pairs, npairs, first_tile, total_tiles, cp, lp, flags, ctas_per_sm, tile_pair, s);
    else if (plain) corr_lin<true, true, false>(d_pairs, npairs, first_tile, total_tiles, cp, lp, flags, ctas_per_sm, tile_pair, s);
    else corr_lin<true, false, false>(d_pairs, npairs, first_tile, total_tiles, cp, lp, flags, ctas_per_sm, tile_pair, s);
  } else {
    corr_lin<false, false, false>(d_pairs, npairs, first_tile, total_tiles, cp, lp, flags, ctas_per_sm, tile_pair, s);
  }
  prof->end(NICP_K_CORR_LIN, s);
}

void launch_corr_list(const PairDev *d_pairs, int npairs, int total_tiles, const CorrParams &cp, int use_state_T,
                      const float *explicit_T, cudaStream_t s, Profiler *prof) {
  prof->begin(NICP_K_CORR_LIST, s);
  k_corr_count<<<total_tiles, kCorrThreads, 0, s>>>(d_pairs, npairs, cp, use_state_T, explicit_T);
  k_corr_write<<<total_tiles, kCorrThreads, 0, s>>>(d_pairs, npairs, cp, use_state_T, explicit_T);
  prof->end(NICP_K_CORR_LIST, s, 2);
}

void launch_lin_list(const PairDev *d_pairs, int npairs, int total_tiles, const LinParams &lp, int parity_threads,
                     int use_state_T, const float *explicit_T, bool chained, cudaStream_t s, Profiler *prof) {
  prof->begin(NICP_K_LIN_LIST, s);
  launch(chained, k_lin_list, total_tiles, kCorrThreads, 0, s, d_pairs, npairs, lp, parity_threads, use_state_T,
         explicit_T);
  prof->end(NICP_K_LIN_LIST, s);
}

void launch_begin_loop(const BeginArgs &a, cudaStream_t s, Profiler *prof) {
  configure_loop();
  prof->begin(NICP_K_SOLVE, s);
  // a CTA per pair, and for the z-buffers 16 stores per thread up to eight CTAs per SM
  const size_t want = std::max<size_t>(a.npairs, (a.zbuf16 + 16 * 256 - 1) / (16 * 256));
  k_begin_loop<<<(unsigned)std::min<size_t>(want, 8 * 148), 256, 0, s>>>(a);
  prof->end(NICP_K_SOLVE, s);
}

void launch_publish(const PairState *states, PairState *host, int npairs, bool chained, cudaStream_t s,
                    Profiler *prof) {
  prof->begin(NICP_K_SOLVE, s);
  const size_t n = (size_t)npairs * (sizeof(PairState) / 16);
  launch(chained, k_publish, (unsigned)std::min<size_t>((n + 255) / 256, 148), 256, 0, s, (const uint4 *)states,
         (uint4 *)host, n);
  prof->end(NICP_K_SOLVE, s);
}

void launch_solve(const PairDev *d_pairs, int npairs, float lambda, int mode, double early_eps, int ignore_done,
                  cudaStream_t s, Profiler *prof) {
  configure_loop();
  prof->begin(NICP_K_SOLVE, s);
  launch(true, k_solve, npairs, kSumThreads, 0, s, d_pairs, npairs, lambda, mode, early_eps, ignore_done);
  prof->end(NICP_K_SOLVE, s);
}

// ------------------------------------------------------------ scratch-free linearizer
// The linearizer of nicp_linearize, for callers that must not allocate
// device memory: the per-tile FP64 partials go to this fixed array instead
// of the context workspace.  The array is part of the library's device
// image, so it exists on every GPU that loads the library, from the first
// load until the process exits.  Every call uses the same array: calls whose
// kernels overlap on the GPU (different streams, or different host threads
// on one device) race on it.  Nothing in it needs clearing -- each call
// writes every partial it later reads.
constexpr int kNoAllocMaxTiles = NICP_LINEARIZE_NOALLOC_MAX_PAIRS / kCorrTilePixels;
static __device__ __align__(256) double g_noalloc_partials[kNoAllocMaxTiles * kPartialWords];

__global__ void __launch_bounds__(kCorrThreads) k_lin_noalloc(NoAllocLinArgs a, double *__restrict__ partials) {
  const int tile = blockIdx.x;
  if (tile >= kNoAllocMaxTiles) return;  // the host refuses longer lists; never write past the array
  int K = a.num_pairs;
  if (a.parity_threads > 1) K = (K / a.parity_threads) * a.parity_threads;
  const int nref = *a.ref_count, ncur = *a.cur_count;
  Acc acc;
  acc.zero();
  const int i0 = tile * kCorrTilePixels + threadIdx.x * 4;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int i = i0 + k;
    if (i >= K) break;
    const int ri = a.pairs[2 * i], ci = a.pairs[2 * i + 1];
    if (ri < 0 || ci < 0 || ri >= nref || ci >= ncur) continue;
    acc.cnt += Acc::kCandidate;
    acc.cnt += Acc::kAccepted;
    const float4 *o = a.cur_omg + 3 * (size_t)ci;
    lin_terms(a.lp, a.T, a.ref_pts[ri], a.ref_nrm[ri], a.cur_pts[ci], a.cur_nrm[ci], o[0], o[1], o[2], acc);
  }
  block_reduce_store<kCorrThreads>(acc, partials + (size_t)tile * kPartialWords);
}

// Sums the tile partials in the same fixed order as k_solve and writes
// H (36, row-major), b (6), error, inliers to out.
__global__ void __launch_bounds__(kSumThreads) k_lin_noalloc_sum(int ntiles, const double *__restrict__ partials,
                                                                 double *__restrict__ out) {
  __shared__ double part[kSumGroups][32];
  __shared__ double tot[32];
  sum_tile_partials(partials, min(ntiles, kNoAllocMaxTiles), false, part);
  if (threadIdx.x < 32) tot[threadIdx.x] = sum_groups(part, false, threadIdx.x);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const int li[6][2] = {{0, 0}, {1, 0}, {1, 1}, {2, 0}, {2, 1}, {2, 2}};
  for (int q = 0; q < 6; q++) {
    const int i = li[q][0], j = li[q][1];
    out[i * 6 + j] = out[j * 6 + i] = tot[q];
    out[(3 + i) * 6 + 3 + j] = out[(3 + j) * 6 + 3 + i] = tot[15 + q];
  }
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) out[i * 6 + 3 + j] = out[(3 + j) * 6 + i] = tot[6 + i * 3 + j];
  for (int i = 0; i < 3; i++) {
    out[36 + i] = tot[21 + i];
    out[39 + i] = tot[24 + i];
  }
  out[42] = (double)(float)tot[27];  // Linearizer::error() is a float
  out[43] = (double)(int)tot[28];
}

// Device address of g_noalloc_partials, looked up once per device with that
// device current (host code must not use the symbol itself as an address).
static double *noalloc_partials_on(int device, cudaError_t *err) {
  constexpr int kMaxDevices = 64;
  static double *addr[kMaxDevices] = {};
  static std::mutex m;
  *err = cudaSuccess;
  if (device < 0 || device >= kMaxDevices) {
    *err = cudaErrorInvalidDevice;
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(m);
  if (!addr[device]) {
    double *p = nullptr;
    *err = cudaGetSymbolAddress((void **)&p, g_noalloc_partials);
    if (*err != cudaSuccess) return nullptr;
    addr[device] = p;
  }
  return addr[device];
}

int lin_noalloc(const NoAllocLinArgs &args, double *out_dev, cudaStream_t s) {
  if (args.num_pairs < 0 || args.num_pairs > NICP_LINEARIZE_NOALLOC_MAX_PAIRS) return NICP_EINVAL;
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) return NICP_ECUDA;
  cudaError_t err;
  double *partials = noalloc_partials_on(device, &err);
  if (!partials) return NICP_ECUDA;
  const int ntiles = std::max(1, (args.num_pairs + kCorrTilePixels - 1) / kCorrTilePixels);
  k_lin_noalloc<<<ntiles, kCorrThreads, 0, s>>>(args, partials);
  k_lin_noalloc_sum<<<1, kSumThreads, 0, s>>>(ntiles, partials, out_dev);
  return cudaGetLastError() == cudaSuccess ? NICP_OK : NICP_ECUDA;
}

}  // namespace nicp
