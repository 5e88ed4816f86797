// T chained steps of the statequant layout [K][V] in one launch, from a floating-point state: K = V = 128, a residual in
// fp32, fp16 or fp8, per-V state scales.  A (request, head) tile is read once as h0, quantised, carried through its
// T tokens on chip and written once as codes, scales and residual; each token is the full step of the streaming kernel
// (carry_gdn_tile128.cuh, statequant layout), operation for operation, so the results are those of T separate steps.
//
// What it saves: 8 tokens of 64 requests x 32 heads with an fp32 residual were nine passes of eager kernels for the
// initial state (0.4 ms) and 8 launches that each move 10 bytes per element (0.54 ms, at 85 % of the copy rate).  Here the
// state crosses HBM once, 9 bytes per element in all, and the arithmetic bounds: 1021 -> 241 us.
//
// One CTA of 8 warps per tile, two per SM.  Lane = 4 columns x the warp's 16 rows.  A column's sums and its maximum are
// finished by one lane, through shared memory, and handed to the others the same way: four meetings per token.  (Every
// warp finishing all 128 columns for itself needs two, but took 306 us where this took 254.)  Codes stay in registers from
// token to token, the residual in shared memory in its own format; a token's k and q are spread per warp as {k, k, q, q}
// rows so that packed instructions read them as they are.
#include "carry_gdn_tile128.cuh"

namespace carry {
namespace {

struct ChainExtra {
  const float* h0;        // [B, HV, K, V]; null: carry on from the state in p
  int T;
  int first_token;        // tokens already applied by earlier launches (offset into q, k, v, alpha, beta, o)
};

constexpr int kChainChunk = 8;           // tokens whose activations and facts are fetched together

template <int RES, int QDT>
struct ChainShared {
  static constexpr int kElem = RES == CARRY_RES_FP32 ? 4 : RES == CARRY_RES_FP16 ? 2 : 1;
  static constexpr int kVec = kT * (QDT == CARRY_F32 ? 4 : 2);
  static constexpr int kResid = 0;                                    // [K][V] in the residual's format
  static constexpr int kVecs = kT * kT * kElem;                       // [chunk][q | k | v]
  static constexpr int kDot = kVecs + kChainChunk * 3 * kVec;         // [warp][col][2]
  static constexpr int kMax = kDot + kWarps * kT * 8;                 // [warp][col]
  static constexpr int kRows = kMax + kWarps * kT * 4;                // [warp][16] {k, k, q, q}
  static constexpr int kCol = kRows + kWarps * 16 * 16;               // per column: delta; scale; its reciprocal
  static constexpr int kMeta = kCol + 3 * kT * 4;
  static constexpr int kBytes = kMeta + kChainChunk * (int)sizeof(TileMeta);
};

template <int RES>
__device__ __forceinline__ void chain_put_resid(void* base, int at, float2 a, float2 b) {
  if constexpr (RES == CARRY_RES_FP32) {
    reinterpret_cast<float4*>(base)[at / 4] = make_float4(a.x, a.y, b.x, b.y);
  } else if constexpr (RES == CARRY_RES_FP16) {
    const __half2 a2 = __floats2half2_rn(a.x, a.y), b2 = __floats2half2_rn(b.x, b.y);
    reinterpret_cast<uint2*>(base)[at / 4] = make_uint2(*reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&b2));
  } else {
    reinterpret_cast<uint32_t*>(base)[at / 4] = float4_to_e5m2x4(a, b);
  }
}
template <int RES>
__device__ __forceinline__ void chain_get_resid(const void* base, int at, float2& a, float2& b) {
  if constexpr (RES == CARRY_RES_FP32) {
    const float4 e = reinterpret_cast<const float4*>(base)[at / 4];
    a = make_float2(e.x, e.y); b = make_float2(e.z, e.w);
  } else if constexpr (RES == CARRY_RES_FP16) {
    const uint2 e = reinterpret_cast<const uint2*>(base)[at / 4];
    a = __half22float2(*reinterpret_cast<const __half2*>(&e.x)); b = __half22float2(*reinterpret_cast<const __half2*>(&e.y));
  } else {
    e5m2x4_to_float(reinterpret_cast<const uint32_t*>(base)[at / 4], a, b);
  }
}

template <int RES, int QDT>
__global__ void __launch_bounds__(kThreads, 2) gdn_chain_kernel(const __grid_constant__ KParams p, const __grid_constant__ ChainExtra x) {
  using S = ChainShared<RES, QDT>;
  constexpr int qes = (QDT == CARRY_F32) ? 4 : 2;
  extern __shared__ __align__(128) uint8_t sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = 16 * warp, c0 = 4 * lane;
  float* red_dot = reinterpret_cast<float*>(sm + S::kDot);
  float* red_max = reinterpret_cast<float*>(sm + S::kMax);
  float4* kq_row = reinterpret_cast<float4*>(sm + S::kRows) + warp * 16;
  float* delta = reinterpret_cast<float*>(sm + S::kCol);
  float *scale_of = delta + kT, *inv_of = delta + 2 * kT;
  TileMeta* meta = reinterpret_cast<TileMeta*>(sm + S::kMeta);
  const int tile = (int)blockIdx.x;                       // request * HV + head
  const long long el0 = (long long)tile * kT * kT;
  const long long step_rows = (long long)p.B * p.HV;      // (request, head) pairs of one token
  const float2 magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);

  // a NaN in the initial state has to reach its column's scale, as it does through torch's maximum; fmaxf drops it
  auto max_or_nan = [](float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
  };
  // ... column maxima of all warps -> every lane's four columns
  auto column_max = [&](float (&m)[4]) {
    *reinterpret_cast<float4*>(red_max + warp * kT + c0) = make_float4(m[0], m[1], m[2], m[3]);
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float4 y = *reinterpret_cast<const float4*>(red_max + w * kT + c0);
      m[0] = max_or_nan(m[0], y.x); m[1] = max_or_nan(m[1], y.y); m[2] = max_or_nan(m[2], y.z); m[3] = max_or_nan(m[3], y.w);
    }
  };
  uint32_t cw[16];                                        // codes of my 4 columns x 16 rows
  float scol[4];                                          // their scales
  float2 hA[16], hB[16];
  depend_release();
  depend_wait();
  if (x.h0) {
    // the initial state: scale = max(amax, 1e-12) * (1 / qmax), the product that torch's division by a host scalar
    // makes of it; codes round_half_even(h0 / scale), clamped; no residual
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float4 h4 = *reinterpret_cast<const float4*>(x.h0 + el0 + (r0 + i) * kT + c0);
      hA[i] = make_float2(h4.x, h4.y); hB[i] = make_float2(h4.z, h4.w);
    }
    float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      m[0] = max_or_nan(m[0], fabsf(hA[i].x)); m[1] = max_or_nan(m[1], fabsf(hA[i].y));
      m[2] = max_or_nan(m[2], fabsf(hB[i].x)); m[3] = max_or_nan(m[3], fabsf(hB[i].y));
    }
    column_max(m);
    float inv[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) { scol[b] = __fmul_rn(max_or_nan(m[b], kEps), p.inv_qmax); inv[b] = rcp_refined(scol[b]); }
    auto code = [&](float v, int b) {                     // code + kMagicRound
      float y = fmaf(v, inv[b], kMagicRound);
      if (fabsf(fmaf(__fadd_rn(y, -kMagicRound), -scol[b], v)) > scol[b] * kTieGuard) y = __fadd_rn(exact_code(v, scol[b]), kMagicRound);
      if (!(y == y)) y = kMagicRound;                     // a column with a NaN or an infinity: the conversion to int8 makes 0 of a NaN
      return __float_as_uint(fminf(fmaxf(y, kMagicRound - p.qmax), kMagicRound + p.qmax));
    };
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      cw[i] = pack4(code(hA[i].x, 0), code(hA[i].y, 1), code(hB[i].x, 2), code(hB[i].y, 3));
      chain_put_resid<RES>(sm + S::kResid, (r0 + i) * kT + c0, splat(0.f), splat(0.f));
    }
    __syncthreads();                                      // red_max is free again
  } else {
    const uint8_t* e = reinterpret_cast<const uint8_t*>(p.resid_in) + el0 * S::kElem;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      cw[i] = *reinterpret_cast<const uint32_t*>(p.codes_in + el0 + (r0 + i) * kT + c0);
      float2 a, b;
      chain_get_resid<RES>(e, (r0 + i) * kT + c0, a, b);
      chain_put_resid<RES>(sm + S::kResid, (r0 + i) * kT + c0, a, b);
    }
    const float4 s4 = *reinterpret_cast<const float4*>(p.sscale_in + (long long)tile * kT + c0);
    scol[0] = s4.x; scol[1] = s4.y; scol[2] = s4.z; scol[3] = s4.w;
  }

  for (int t = 0; t < x.T; ++t) {
    const int tc = t % kChainChunk;
    if (tc == 0) {
      // the next chunk of tokens: q, k, v into shared memory, 16 bytes per thread and step, gates and <k, q> by one
      // warp per token
      const int nt = (x.T - t < kChainChunk) ? (x.T - t) : kChainChunk;
      constexpr int kPer = S::kVec / 16;
      __syncthreads();                                    // everybody is done with the previous chunk
      for (int i = tid; i < nt * 3 * kPer; i += kThreads) {
        const int tt = i / (3 * kPer), c = i - tt * 3 * kPer, which = c / kPer;
        const void* src = which == 0 ? p.q : which == 1 ? p.k : p.v;
        const long long row = (x.first_token + t + tt) * step_rows + tile;
        *reinterpret_cast<uint4*>(sm + S::kVecs + tt * 3 * S::kVec + 16 * c) =
            __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(src) + row * kT * qes) + (c - which * kPer));
      }
      if (warp < nt) {
        const long long rows = (x.first_token + t + warp) * step_rows;
        tile_meta<RES, CARRY_SCALE_PER_V, QDT, 32>(p, tile, lane, true, &meta[warp], nullptr, rows * kT, rows, rows);
      }
      __syncthreads();
    }
    const uint8_t* vec = sm + S::kVecs + tc * 3 * S::kVec;
    const uint4 tm0 = lds_v4(&meta[tc]), tm1 = lds_v4(reinterpret_cast<const uint8_t*>(&meta[tc]) + 16);
    const float alpha = __uint_as_float(tm0.w), beta = __uint_as_float(tm1.x), kq = __uint_as_float(tm1.w);
    const float2 alpha2 = splat(alpha);
    {
      const float y = act<QDT>(vec + (lane < 16 ? S::kVec : 0), r0 + (lane & 15));
      *reinterpret_cast<float2*>(reinterpret_cast<float*>(kq_row + (lane & 15)) + (lane < 16 ? 0 : 2)) = splat(y);
    }
    __syncwarp();

    // dequantise, decay, column sums over my rows
    const float2 sA = make_float2(scol[0], scol[1]), sB = make_float2(scol[2], scol[3]);
    float2 dkA = make_float2(0.f, 0.f), dkB = dkA, dqA = dkA, dqB = dkA;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 a = mul2(mul2(s8x2_cvt<0, 1>(cw[i]), sA), alpha2);
      const float2 b = mul2(mul2(s8x2_to_float<2, 3>(cw[i] ^ 0x80808080u), sB), alpha2);
      hA[i] = a; hB[i] = b;
      const float4 kq4 = kq_row[i];
      const float2 kr = make_float2(kq4.x, kq4.y), qr = make_float2(kq4.z, kq4.w);
      dkA = fma2(a, kr, dkA); dkB = fma2(b, kr, dkB);
      dqA = fma2(a, qr, dqA); dqB = fma2(b, qr, dqB);
    }
    // a column's reductions are finished by its lane of the first four warps, in the order of the streaming kernel
    {
      float4* dst = reinterpret_cast<float4*>(red_dot + (warp * kT + c0) * 2);
      dst[0] = make_float4(dkA.x, dqA.x, dkA.y, dqA.y);
      dst[1] = make_float4(dkB.x, dqB.x, dkB.y, dqB.y);
      __syncthreads();
      if (tid < kT) {
        float2 d = splat(0.f);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) d = add2(d, *reinterpret_cast<const float2*>(red_dot + (w * kT + tid) * 2));
        const float dv = __fmul_rn(beta, __fadd_rn(act<QDT>(vec + 2 * S::kVec, tid), -d.x));
        delta[tid] = dv;
        store_from_float(p.out, ((x.first_token + t) * step_rows + tile) * kT + tid, p.o_dtype, fmaf(dv, kq, d.y));
      }
      __syncthreads();
    }

    // rank-1 write, residual, column maxima
    const float4 dv4 = *reinterpret_cast<const float4*>(delta + c0);
    const float2 dvA = make_float2(dv4.x, dv4.y), dvB = make_float2(dv4.z, dv4.w);
    float amax[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 kr = *reinterpret_cast<const float2*>(kq_row + i);
      float2 eA, eB;
      chain_get_resid<RES>(sm + S::kResid, (r0 + i) * kT + c0, eA, eB);
      hA[i] = add2(fma2(kr, dvA, hA[i]), eA);
      hB[i] = add2(fma2(kr, dvB, hB[i]), eB);
      if (i & 1) {
        amax[0] = fmaxf(fmaxf(amax[0], fabsf(hA[i - 1].x)), fabsf(hA[i].x)); amax[1] = fmaxf(fmaxf(amax[1], fabsf(hA[i - 1].y)), fabsf(hA[i].y));
        amax[2] = fmaxf(fmaxf(amax[2], fabsf(hB[i - 1].x)), fabsf(hB[i].x)); amax[3] = fmaxf(fmaxf(amax[3], fabsf(hB[i - 1].y)), fabsf(hB[i].y));
      }
    }
    *reinterpret_cast<float4*>(red_max + warp * kT + c0) = make_float4(amax[0], amax[1], amax[2], amax[3]);
    __syncthreads();
    if (tid < kT) {
      float m = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; w += 2) m = fmaxf(fmaxf(m, red_max[w * kT + tid]), red_max[(w + 1) * kT + tid]);
      const float sc = scale_fast(m, p.qmax, p.inv_qmax, p.eps_mode);
      scale_of[tid] = sc;
      inv_of[tid] = rcp_refined(sc);
    }
    __syncthreads();

    // new scales, codes, residual
    const float4 s4 = *reinterpret_cast<const float4*>(scale_of + c0), i4 = *reinterpret_cast<const float4*>(inv_of + c0);
    scol[0] = s4.x; scol[1] = s4.y; scol[2] = s4.z; scol[3] = s4.w;
    const float thr[4] = {s4.x * kTieGuardExact, s4.y * kTieGuardExact, s4.z * kTieGuardExact, s4.w * kTieGuardExact};
    const float2 invA = make_float2(i4.x, i4.y), invB = make_float2(i4.z, i4.w);
    const float2 nsA = make_float2(-scol[0], -scol[1]), nsB = make_float2(-scol[2], -scol[3]);
    float eamax[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 yA = fma2(hA[i], invA, magic2), yB = fma2(hB[i], invB, magic2);
      hA[i] = fma2(add2(yA, nmagic2), nsA, hA[i]);
      hB[i] = fma2(add2(yB, nmagic2), nsB, hB[i]);
      cw[i] = pack4(__float_as_uint(yA.x), __float_as_uint(yA.y), __float_as_uint(yB.x), __float_as_uint(yB.y));
      if (i & 1) {
        eamax[0] = fmaxf(fmaxf(eamax[0], fabsf(hA[i - 1].x)), fabsf(hA[i].x)); eamax[1] = fmaxf(fmaxf(eamax[1], fabsf(hA[i - 1].y)), fabsf(hA[i].y));
        eamax[2] = fmaxf(fmaxf(eamax[2], fabsf(hB[i - 1].x)), fabsf(hB[i].x)); eamax[3] = fmaxf(fmaxf(eamax[3], fabsf(hB[i - 1].y)), fabsf(hB[i].y));
      }
    }
    if (fmaxf(fmaxf(eamax[0] - thr[0], eamax[1] - thr[1]), fmaxf(eamax[2] - thr[2], eamax[3] - thr[3])) > 0.f) {
      // a quotient within the tie guard: only its quad is gone through again (whole columns: 251 us instead of 241)
#pragma unroll
      for (int i = 0; i < 16; ++i) redecide_quad(hA[i], hB[i], cw[i], scol, thr);
    }
    if (t + 1 < x.T) {
#pragma unroll
      for (int i = 0; i < 16; ++i) chain_put_resid<RES>(sm + S::kResid, (r0 + i) * kT + c0, hA[i], hB[i]);
    }
  }

  uint8_t* e_out = reinterpret_cast<uint8_t*>(p.resid_out) + el0 * S::kElem;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    *reinterpret_cast<uint32_t*>(p.codes_out + el0 + (r0 + i) * kT + c0) = cw[i];
    chain_put_resid<RES>(e_out, (r0 + i) * kT + c0, hA[i], hB[i]);
  }
  if (warp == 0) *reinterpret_cast<float4*>(p.sscale_out + (long long)tile * kT + c0) = make_float4(scol[0], scol[1], scol[2], scol[3]);
}

template <int RES, int QDT>
int launch_chain_variant(const KParams& p, const ChainExtra& x, cudaStream_t stream) {
  auto kern = gdn_chain_kernel<RES, QDT>;
  constexpr int smem = ChainShared<RES, QDT>::kBytes;
  static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs per SM");
  static thread_local bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return CARRY_GDN_ERR_NO_DEVICE;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return CARRY_GDN_ERR_NO_DEVICE;
    }
    configured[dev] = true;
  }
  return launch_dependent(kern, dim3((unsigned)(p.B * p.HV)), kThreads, smem, stream, p, x);
}

template <int RES>
int launch_chain_dtype(const KParams& p, const ChainExtra& x, cudaStream_t stream) {
  if (p.qkv_dtype == CARRY_F32) return launch_chain_variant<RES, CARRY_F32>(p, x, stream);
  if (p.qkv_dtype == CARRY_BF16) return launch_chain_variant<RES, CARRY_BF16>(p, x, stream);
  return launch_chain_variant<RES, CARRY_F16>(p, x, stream);
}

}  // namespace

// The streaming kernel's conditions (the arithmetic is its own), a residual in floating point, a 16-byte-aligned h0.
bool chain_eligible(const KParams& p, const float* h0) {
  const bool float_resid = p.res_fmt == CARRY_RES_FP32 || p.res_fmt == CARRY_RES_FP16 || p.res_fmt == CARRY_RES_FP8;
  return !p.packed && float_resid && tile128_eligible(p) && (reinterpret_cast<uintptr_t>(h0) & 15u) == 0;
}

int launch_chain(const KParams& p_in, const float* h0, int T, cudaStream_t stream) {
  KParams p = p_in;
  fill_shifts(p);
  constexpr int kTokensPerLaunch = 1024;                  // a launch on few tiles stays within a few milliseconds
  for (int t = 0; t < T; t += kTokensPerLaunch) {
    ChainExtra x = {t == 0 ? h0 : nullptr, T - t < kTokensPerLaunch ? T - t : kTokensPerLaunch, t};
    const int rc = p.res_fmt == CARRY_RES_FP32   ? launch_chain_dtype<CARRY_RES_FP32>(p, x, stream)
                   : p.res_fmt == CARRY_RES_FP16 ? launch_chain_dtype<CARRY_RES_FP16>(p, x, stream)
                                                 : launch_chain_dtype<CARRY_RES_FP8>(p, x, stream);
    if (rc != CARRY_GDN_OK) return rc;
  }
  return CARRY_GDN_OK;
}

}  // namespace carry
