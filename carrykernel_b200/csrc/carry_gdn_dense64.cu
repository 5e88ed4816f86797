// Statequant layout [K][V] with 64-wide heads (K = V = 64): the quantized step with an int8, a packed int4 or no residual,
// and the unquantised fp32 step.
//
// A warp owns 32 whole columns: lane = 4 columns x 16 rows (rows rg, rg + 4, ...; rg = lane / 8), so a column's sums and
// maxima over K stay among the 4 lanes of a column group -- shuffles, no shared memory and no meeting, except for a
// scale per head, over which the tile's two warps meet.  Every load of a tile is in flight at once, straight into
// registers (a row of a warp is 32 bytes of codes, a whole sector), and results go back the same way.  One CTA of two
// warps per (request, head), six or eight to an SM, so that one tile's loads run under another's arithmetic.
//
// A NaN or an infinity leaves the codes and scales that the generic kernel leaves: a warp whose columns
// it reaches goes element by element.  (Looking for them takes 4 to 6 %: 15.4 -> 16.0 us at 100 requests x 32 heads, int8 residual.)
//
// The generic kernel, which took these shapes, stages a tile as fp32 in shared memory and walks columns with a quarter
// of its threads: 215 us at 100 requests x 32 heads with an int8 residual; this one 16 us.
#include "carry_gdn_tile128.cuh"

namespace carry {
namespace {

constexpr int kN = 64;
constexpr int kPair = 64;
constexpr unsigned kAll = 0xffffffffu;

// x[b], y[b] (b = the lane's 4 columns) summed over the 4 lanes of a column group: lane group g = lane / 8 ends up with
// t[j] = total of column 2 (g & 1) + j, of x where g < 2 and of y otherwise
__device__ __forceinline__ void column_sums(const float (&x)[4], const float (&y)[4], int g, float (&t)[2]) {
  const bool up2 = g & 2, up1 = g & 1;
  float a[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float keep = up2 ? y[i] : x[i], send = up2 ? x[i] : y[i];
    a[i] = keep + __shfl_xor_sync(kAll, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float keep = up1 ? a[2 + i] : a[i], send = up1 ? a[i] : a[2 + i];
    t[i] = keep + __shfl_xor_sync(kAll, send, 8);
  }
}
// ... and maxima: lane group g ends up with column g's
__device__ __forceinline__ float column_max(const float (&x)[4], int g) {
  const bool up2 = g & 2, up1 = g & 1;
  float a[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float keep = up2 ? x[2 + i] : x[i], send = up2 ? x[i] : x[2 + i];
    a[i] = fmaxf(keep, __shfl_xor_sync(kAll, send, 16));
  }
  const float keep = up1 ? a[1] : a[0], send = up1 ? a[0] : a[1];
  return fmaxf(keep, __shfl_xor_sync(kAll, send, 8));
}

// the largest magnitude of three, a NaN if one of them is (fmaxf passes a NaN over)
__device__ __forceinline__ float max3abs_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// What both kernels start with: k and q of the tile as {k, k, q, q} rows (a copy per warp), <k, q>
template <int QDT>
__device__ __forceinline__ float spread_kq(const void* q, const void* k, long long at, float4* rows, int lane) {
  float kq = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float a = raw_to_float(load_raw(k, at + lane + 32 * i, QDT), QDT), b = raw_to_float(load_raw(q, at + lane + 32 * i, QDT), QDT);
    rows[lane + 32 * i] = make_float4(a, a, b, b);
    kq = fmaf(a, b, kq);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) kq += __shfl_xor_sync(kAll, kq, o);
  return kq;
}

// The codes of a lane's 16 elements x[0], x[4], ... of a column to bytes `pitch` apart, and their remainders in place, by the
// true quotient and the clamp as the generic kernel does it: for columns that hold a NaN or an infinity, or whose scale is one
// (the reciprocal makes NaNs of all its quotients).  nibble: 0 whole bytes, 1 the low half of each, 2 the high half
// behind it.  Returns the largest remainder.
__device__ __noinline__ float quantize_column_plainly(float* x, float s, float qmax, int8_t* to, int pitch, int nibble) {
  float worst = 0.f;
#pragma unroll 1
  for (int i = 0; i < 16; ++i, to += pitch) {
    const float code = quantize_div(x[4 * i], s, qmax);
    x[4 * i] = fmaf(code, -s, x[4 * i]);
    worst = fmaxf(worst, fabsf(x[4 * i]));
    const int c = (int)code;
    *to = (int8_t)(nibble == 0 ? c : nibble == 1 ? (c & 15) : (*to | (c << 4)));
  }
  return worst;
}

// RSCALE: granularity of the residual's scale, or of the state's where there is no residual
template <int RES, int RSCALE, int QDT>
__global__ void __launch_bounds__(kPair, RES == CARRY_RES_NONE ? 8 : 6) gdn_dense64_kernel(const __grid_constant__ KParams p) {
  constexpr bool kNone = RES == CARRY_RES_NONE, kInt4 = RES == CARRY_RES_INT4;
  constexpr bool kHeadState = kNone && RSCALE == CARRY_SCALE_PER_HEAD, kHeadResid = !kNone && RSCALE == CARRY_SCALE_PER_HEAD;
  constexpr bool kFold = kInt4 || kNone;                 // sums over the bare codes, the scale on the totals
  constexpr int kRow = kInt4 ? kN / 2 : kN;              // bytes of a residual row
  __shared__ __align__(16) float4 kq_rows[2][kN];
  __shared__ float head_red[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 3;
  const int c0 = 32 * warp + 4 * (lane & 7);
  const long long nh = blockIdx.x;
  const int8_t* cin = p.codes_in + nh * kN * kN + g * kN + c0;
  const uint8_t* ein = reinterpret_cast<const uint8_t*>(p.resid_in) + nh * kN * kRow + g * kRow + (kInt4 ? c0 / 2 : c0);

  depend_release();
  depend_wait();
  uint32_t cw[16], ew[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) cw[i] = __ldcg(reinterpret_cast<const uint32_t*>(cin + 4 * i * kN));
  if constexpr (!kNone) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      ew[i] = kInt4 ? (uint32_t)__ldcg(reinterpret_cast<const uint16_t*>(ein + 4 * i * kRow)) : __ldcg(reinterpret_cast<const uint32_t*>(ein + 4 * i * kRow));
  }
  const float alpha = __ldcg(p.alpha + nh), beta = __ldcg(p.beta + nh);
  float scol[4], es_col[4] = {0.f, 0.f, 0.f, 0.f}, v[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    scol[b] = __ldcg(p.sscale_in + (kHeadState ? nh : nh * kN + c0 + b));
    if constexpr (!kNone) es_col[b] = __ldcg(p.rscale_in + (kHeadResid ? nh : nh * kN + c0 + b));
    v[b] = raw_to_float(load_raw(p.v, nh * kN + c0 + b, QDT), QDT);
  }
  float4* rows = kq_rows[warp];
  const float kq = spread_kq<QDT>(p.q, p.k, nh * kN, rows, lane);
  __syncwarp();

  // dequantise, decay, partial column sums
  const float2 sA = make_float2(scol[0], scol[1]), sB = make_float2(scol[2], scol[3]), alpha2 = splat(alpha);
  float2 saA = mul2(sA, alpha2), saB = mul2(sB, alpha2);
  if constexpr (kFold) {                // an infinite scale makes NaNs, as 0 * scale does; the folded sum alone would not
    saA = fma2(saA, splat(0.f), saA); saB = fma2(saB, splat(0.f), saB);
  }
  float2 hA[16], hB[16], dkA = splat(0.f), dkB = dkA, dqA = dkA, dqB = dkA;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float2 a = s8x2_cvt<0, 1>(cw[i]), b = s8x2_to_float<2, 3>(cw[i] ^ 0x80808080u);
    if constexpr (!kFold) { a = mul2(mul2(a, sA), alpha2); b = mul2(mul2(b, sB), alpha2); }
    hA[i] = a; hB[i] = b;
    const float4 r4 = rows[g + 4 * i];
    const float2 kr = make_float2(r4.x, r4.y), qr = make_float2(r4.z, r4.w);
    dkA = fma2(a, kr, dkA); dkB = fma2(b, kr, dkB);
    dqA = fma2(a, qr, dqA); dqB = fma2(b, qr, dqB);
  }
  if constexpr (kFold) { dkA = mul2(dkA, saA); dkB = mul2(dkB, saB); dqA = mul2(dqA, saA); dqB = mul2(dqB, saB); }
  float dv[4];
  {
    const float dk[4] = {dkA.x, dkA.y, dkB.x, dkB.y}, dq[4] = {dqA.x, dqA.y, dqB.x, dqB.y};
    float mine[2];
    column_sums(dk, dq, g, mine);
#pragma unroll
    for (int b = 0; b < 4; ++b)
      dv[b] = __fmul_rn(beta, __fadd_rn(v[b], -__shfl_sync(kAll, mine[b & 1], (lane & 7) + 8 * (b >> 1))));
    if (g >= 2) {                       // the lanes that hold q totals finish their two columns' output
      const bool up = g & 1;
      const long long at = nh * kN + c0 + (up ? 2 : 0);
      const float d0 = up ? dv[2] : dv[0], d1 = up ? dv[3] : dv[1];
      // (0 * d: the sum over rows of an infinite write has both signs in it)
      store_from_float(p.out, at, p.o_dtype, fmaf(d0, kq, fmaf(0.f, d0, mine[0])));
      store_from_float(p.out, at + 1, p.o_dtype, fmaf(d1, kq, fmaf(0.f, d1, mine[1])));
    }
  }
  // rank-1 write, residual, column maxima
  const float2 dvA = make_float2(dv[0], dv[1]), dvB = make_float2(dv[2], dv[3]);
  const float2 esA = make_float2(es_col[0], es_col[1]), esB = make_float2(es_col[2], es_col[3]);
  float amax[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 kr = *reinterpret_cast<const float2*>(rows + g + 4 * i);
    if constexpr (kNone) {
      hA[i] = fma2(hA[i], saA, mul2(kr, dvA)); hB[i] = fma2(hB[i], saB, mul2(kr, dvB));
    } else if constexpr (kInt4) {
      float2 nA, nB;
      s4x4_pairs(ew[i], nA, nB);
      hA[i] = fma2(nA, esA, fma2(hA[i], saA, mul2(kr, dvA)));
      hB[i] = fma2(nB, esB, fma2(hB[i], saB, mul2(kr, dvB)));
    } else {
      const uint32_t w = ew[i] ^ 0x80808080u;
      hA[i] = fma2(s8x2_to_float<0, 1>(w), esA, fma2(kr, dvA, hA[i]));
      hB[i] = fma2(s8x2_to_float<2, 3>(w), esB, fma2(kr, dvB, hB[i]));
    }
    if (i & 1) {                        // two rows per three-operand maximum; it keeps a NaN
      amax[0] = max3abs_nan(amax[0], hA[i - 1].x, hA[i].x); amax[1] = max3abs_nan(amax[1], hA[i - 1].y, hA[i].y);
      amax[2] = max3abs_nan(amax[2], hB[i - 1].x, hB[i].x); amax[3] = max3abs_nan(amax[3], hB[i - 1].y, hB[i].y);
    }
  }
  const float inf = __int_as_float(0x7f800000);
  const bool finite = max3abs_nan(max3abs_nan(amax[0], amax[1], amax[2]), amax[3], 0.f) < inf;
  if (!finite) {                        // a scale passes NaNs over
#pragma unroll
    for (int b = 0; b < 4; ++b) amax[b] = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      amax[0] = fmaxf(amax[0], fabsf(hA[i].x)); amax[1] = fmaxf(amax[1], fabsf(hA[i].y));
      amax[2] = fmaxf(amax[2], fabsf(hB[i].x)); amax[3] = fmaxf(amax[3], fabsf(hB[i].y));
    }
  }
  // a scale per column (its lane group's g-th lane works it out), or one for the matrix
  auto scales = [&](const float (&m)[4], bool per_head, float qmax, float (&s)[4], float (&inv)[4]) {
    float top;
    if (per_head) {
      top = warp_max_nonneg(fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])));
      if (lane == 0) head_red[warp] = top;
      __syncthreads();
      top = fmaxf(head_red[0], head_red[1]);
    } else {
      top = column_max(m, g);
    }
    const float s_mine = scale_from_amax(top, qmax, p.eps_mode), i_mine = rcp_refined(s_mine);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      s[b] = per_head ? s_mine : __shfl_sync(kAll, s_mine, (lane & 7) + 8 * b);
      inv[b] = per_head ? i_mine : __shfl_sync(kAll, i_mine, (lane & 7) + 8 * b);
    }
  };
  float snew[4], sinv[4];
  scales(amax, kHeadState, p.qmax, snew, sinv);
  if (kHeadState) {
    if (tid == 0) p.sscale_out[nh] = snew[0];
  } else if (g == 0) {
#pragma unroll
    for (int b = 0; b < 4; ++b) p.sscale_out[nh * kN + c0 + b] = snew[b];
  }
  int8_t* cout = p.codes_out + nh * kN * kN + g * kN + c0;
  uint8_t* eout = reinterpret_cast<uint8_t*>(p.resid_out) + nh * kN * kRow + g * kRow + (kInt4 ? c0 / 2 : c0);
  constexpr float rqmax = kInt4 ? 7.0f : 127.0f;
  float eamax[4] = {0.f, 0.f, 0.f, 0.f}, es[4], ei[4];
  auto put_resid_scales = [&](const float (&s)[4]) {
    if (kHeadResid) {
      if (tid == 0) p.rscale_out[nh] = s[0];
    } else if (g == 0) {
#pragma unroll
      for (int b = 0; b < 4; ++b) p.rscale_out[nh * kN + c0 + b] = s[b];
    }
  };
  if (__any_sync(kAll, !finite || !(snew[0] + snew[1] + snew[2] + snew[3] < inf))) {      // (one vote per warp: scales() meets)
    float plain[64];
#pragma unroll
    for (int i = 0; i < 16; ++i) { plain[4 * i] = hA[i].x; plain[4 * i + 1] = hA[i].y; plain[4 * i + 2] = hB[i].x; plain[4 * i + 3] = hB[i].y; }
#pragma unroll
    for (int b = 0; b < 4; ++b) eamax[b] = quantize_column_plainly(plain + b, snew[b], p.qmax, cout + b, 4 * kN, 0);
    if constexpr (!kNone) {
      scales(eamax, kHeadResid, rqmax, es, ei);
      put_resid_scales(es);
#pragma unroll
      for (int b = 0; b < 4; ++b)
        quantize_column_plainly(plain + b, es[b], rqmax, reinterpret_cast<int8_t*>(eout) + (kInt4 ? b / 2 : b), 4 * kRow, kInt4 ? 1 + (b & 1) : 0);
    }
    return;
  }
  // codes; remainders in place of the targets
  const float2 invA = make_float2(sinv[0], sinv[1]), invB = make_float2(sinv[2], sinv[3]);
  const float2 nsA = make_float2(-snew[0], -snew[1]), nsB = make_float2(-snew[2], -snew[3]);
  const float2 magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);
  const float thr[4] = {snew[0] * kTieGuard, snew[1] * kTieGuard, snew[2] * kTieGuard, snew[3] * kTieGuard};
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float2 yA = fma2(hA[i], invA, magic2), yB = fma2(hB[i], invB, magic2);
    hA[i] = fma2(add2(yA, nmagic2), nsA, hA[i]);
    hB[i] = fma2(add2(yB, nmagic2), nsB, hB[i]);
    if (fmaxf(fmaxf(fabsf(hA[i].x) - thr[0], fabsf(hA[i].y) - thr[1]), fmaxf(fabsf(hB[i].x) - thr[2], fabsf(hB[i].y) - thr[3])) > 0.f) {
      redecide_rec(hA[i].x, yA.x, snew[0], thr[0]); redecide_rec(hA[i].y, yA.y, snew[1], thr[1]);
      redecide_rec(hB[i].x, yB.x, snew[2], thr[2]); redecide_rec(hB[i].y, yB.y, snew[3], thr[3]);
    }
    *reinterpret_cast<uint32_t*>(cout + 4 * i * kN) = pack4(__float_as_uint(yA.x), __float_as_uint(yA.y), __float_as_uint(yB.x), __float_as_uint(yB.y));
    eamax[0] = fmaxf(eamax[0], fabsf(hA[i].x)); eamax[1] = fmaxf(eamax[1], fabsf(hA[i].y));
    eamax[2] = fmaxf(eamax[2], fabsf(hB[i].x)); eamax[3] = fmaxf(eamax[3], fabsf(hB[i].y));
  }
  if constexpr (!kNone) {
    scales(eamax, kHeadResid, rqmax, es, ei);
    put_resid_scales(es);
    if (kHeadResid && !(es[0] < inf)) ei[0] = ei[1] = ei[2] = ei[3] = 0.f;      // from the other warp's columns
    const float2 ieA = make_float2(ei[0], ei[1]), ieB = make_float2(ei[2], ei[3]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 rA = fma2(hA[i], ieA, magic2), rB = fma2(hB[i], ieB, magic2);
      const uint32_t r[4] = {__float_as_uint(rA.x), __float_as_uint(rA.y), __float_as_uint(rB.x), __float_as_uint(rB.y)};
      if constexpr (kInt4) *reinterpret_cast<uint16_t*>(eout + 4 * i * kRow) = (uint16_t)pack_s4x4(r[0], r[1], r[2], r[3]);
      else *reinterpret_cast<uint32_t*>(eout + 4 * i * kRow) = pack4(r[0], r[1], r[2], r[3]);
    }
  }
}

template <int QDT>
__global__ void __launch_bounds__(kPair, 8) gdn_fp32_64_kernel(const __grid_constant__ CarryGdnFp32Args a) {
  __shared__ __align__(16) float4 kq_rows[2][kN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 3;
  const int c0 = 32 * warp + 4 * (lane & 7);
  const long long nh = blockIdx.x;
  const float* hin = a.h_in + nh * kN * kN + g * kN + c0;
  float* hout = a.h_out + nh * kN * kN + g * kN + c0;
  depend_release();
  depend_wait();
  float4 h[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) h[i] = *reinterpret_cast<const float4*>(hin + 4 * i * kN);
  const float alpha = __ldcg(a.alpha + nh), beta = __ldcg(a.beta + nh);
  float v[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) v[b] = raw_to_float(load_raw(a.v, nh * kN + c0 + b, QDT), QDT);
  float4* rows = kq_rows[warp];
  spread_kq<QDT>(a.q, a.k, nh * kN, rows, lane);
  __syncwarp();
  float dk[4] = {0.f, 0.f, 0.f, 0.f}, dq[4] = {0.f, 0.f, 0.f, 0.f}, dv[4], mine[2];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float k = rows[g + 4 * i].x;
    h[i].x = __fmul_rn(alpha, h[i].x); h[i].y = __fmul_rn(alpha, h[i].y); h[i].z = __fmul_rn(alpha, h[i].z); h[i].w = __fmul_rn(alpha, h[i].w);
    dk[0] = fmaf(h[i].x, k, dk[0]); dk[1] = fmaf(h[i].y, k, dk[1]); dk[2] = fmaf(h[i].z, k, dk[2]); dk[3] = fmaf(h[i].w, k, dk[3]);
  }
  column_sums(dk, dq, g, mine);
#pragma unroll
  for (int b = 0; b < 4; ++b)
    dv[b] = __fmul_rn(beta, __fadd_rn(v[b], -__shfl_sync(kAll, mine[b & 1], (lane & 7) + 8 * (b >> 1))));
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float4 r4 = rows[g + 4 * i];
    h[i].x = __fadd_rn(h[i].x, __fmul_rn(r4.x, dv[0])); h[i].y = __fadd_rn(h[i].y, __fmul_rn(r4.x, dv[1]));
    h[i].z = __fadd_rn(h[i].z, __fmul_rn(r4.x, dv[2])); h[i].w = __fadd_rn(h[i].w, __fmul_rn(r4.x, dv[3]));
    dq[0] = fmaf(h[i].x, r4.z, dq[0]); dq[1] = fmaf(h[i].y, r4.z, dq[1]); dq[2] = fmaf(h[i].z, r4.z, dq[2]); dq[3] = fmaf(h[i].w, r4.z, dq[3]);
    *reinterpret_cast<float4*>(hout + 4 * i * kN) = h[i];
  }
  column_sums(dk, dq, g, mine);
  if (g >= 2) {
    const long long at = nh * kN + c0 + 2 * (g & 1);
    store_from_float(a.o, at, a.o_dtype, mine[0]);
    store_from_float(a.o, at + 1, a.o_dtype, mine[1]);
  }
}

template <int RES, int RSCALE>
int launch_dtype64(const KParams& p, cudaStream_t stream) {
  const dim3 grid((unsigned)((long long)p.B * p.HV));
  if (p.qkv_dtype == CARRY_F32) return launch_dependent(gdn_dense64_kernel<RES, RSCALE, CARRY_F32>, grid, kPair, 0, stream, p);
  if (p.qkv_dtype == CARRY_BF16) return launch_dependent(gdn_dense64_kernel<RES, RSCALE, CARRY_BF16>, grid, kPair, 0, stream, p);
  return launch_dependent(gdn_dense64_kernel<RES, RSCALE, CARRY_F16>, grid, kPair, 0, stream, p);
}

bool aligned(const void* p, unsigned bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

}  // namespace

// K = V = 64 with codes (and an int8 residual) on a 4-byte boundary, an int4 one on 2; scales and activations are read
// element by element.  Int formats need per-V state scales (every lane holds its columns' scale only).
bool dense64_eligible(const KParams& p) {
  if (p.packed || p.K != kN || p.V != kN || (long long)p.B * p.HV > 0x7fffffffLL) return false;
  if (!aligned(p.codes_in, 4) || !aligned(p.codes_out, 4)) return false;
  if (p.res_fmt == CARRY_RES_NONE) return true;
  if (p.sscale_mode != CARRY_SCALE_PER_V) return false;
  if (p.res_fmt == CARRY_RES_INT8) return aligned(p.resid_in, 4) && aligned(p.resid_out, 4);
  return p.res_fmt == CARRY_RES_INT4 && aligned(p.resid_in, 2) && aligned(p.resid_out, 2);
}

int launch_dense64(const KParams& p, cudaStream_t stream) {
  if (p.res_fmt == CARRY_RES_NONE)
    return p.sscale_mode == CARRY_SCALE_PER_V ? launch_dtype64<CARRY_RES_NONE, CARRY_SCALE_PER_V>(p, stream)
                                              : launch_dtype64<CARRY_RES_NONE, CARRY_SCALE_PER_HEAD>(p, stream);
  const bool i4 = p.res_fmt == CARRY_RES_INT4, pv = p.rscale_mode == CARRY_SCALE_PER_V;
  if (i4) return pv ? launch_dtype64<CARRY_RES_INT4, CARRY_SCALE_PER_V>(p, stream)
                    : launch_dtype64<CARRY_RES_INT4, CARRY_SCALE_PER_HEAD>(p, stream);
  return pv ? launch_dtype64<CARRY_RES_INT8, CARRY_SCALE_PER_V>(p, stream)
            : launch_dtype64<CARRY_RES_INT8, CARRY_SCALE_PER_HEAD>(p, stream);
}

bool fp32_64_eligible(const CarryGdnFp32Args& a) {
  return a.K == kN && a.V == kN && aligned(a.h_in, 16) && aligned(a.h_out, 16) && (long long)a.B * a.HV <= 0x7fffffffLL;
}

int launch_fp32_64(const CarryGdnFp32Args& a, cudaStream_t stream) {
  const dim3 grid((unsigned)((long long)a.B * a.HV));
  if (a.qkv_dtype == CARRY_F32) return launch_dependent(gdn_fp32_64_kernel<CARRY_F32>, grid, kPair, 0, stream, a);
  if (a.qkv_dtype == CARRY_BF16) return launch_dependent(gdn_fp32_64_kernel<CARRY_BF16>, grid, kPair, 0, stream, a);
  return launch_dependent(gdn_fp32_64_kernel<CARRY_F16>, grid, kPair, 0, stream, a);
}

}  // namespace carry
