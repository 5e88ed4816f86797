// The slot-indexed decode step for 64-wide heads: K = V = 64, int8 or packed int4 residual.
//
// A row of the slot layout [V][K] is 64 elements, which one lane can hold: lane = one V row.  Sums and maxima over K
// are then chains inside a lane, every scale is a lane's own, outputs and scales leave coalesced, and nothing is
// exchanged between lanes except the per-head residual maximum.  (Every operation is rounded where the generic
// kernel rounds it and in its order, so the two agree bit for bit;
// rows with a NaN or an infinity, of which the reciprocal would make other codes, go through the true quotients.)
//
// Bound: a tile is 4 KB of codes and 2 or 4 KB of residual, and a batch of 48 requests x 16 heads is 5 tiles per
// SM -- latency and instruction issue, not bandwidth.  So no ring and no roles: one CTA of two warps per
// (request, head), 32 rows to a warp, and with 6 CTAs on an SM one tile's loads run under another's arithmetic.
// Codes and residual come in by coalesced 16-byte asynchronous copies into rows padded against bank conflicts, while
// gates and norms are worked out, and go out the same way.
//
// Measured (48 requests x 16 heads, int8 residual, 12 layers back to back): 7.7 us per launch with the state in the L2, 8.0
// out of it, 8.3 where inputs that repeat hold the state at a fixed point (ties in every row); the generic kernel 79 us.
// 512 requests: 58 us (2.4 TB/s) against 540.  168 registers and 6 CTAs per SM, since the row is 64 of them: at 128
// registers and 8 CTAs 140 bytes spill and the launch takes 10 us.
//
// Nothing touches memory ahead of the dependency wait.  Hints to the L2 for the slot that the index names then and for
// q, k and v take the 8.3 us to 8.0 and the 8.0 to 7.9, but the wait waits for them too: behind a kernel that does not release
// its dependents, as most of an engine's, a launch takes 0.9 us more (48 requests, 12 layers with another kernel ahead of each:
// 156 -> 166 us; int4 146 -> 157), and back to back with the state in the L2 0.1 to 0.3 us more.
#include "carry_gdn_tile128.cuh"

namespace carry {
namespace {

constexpr int kN = 64;                  // tile edge
constexpr int kPair = 64;               // threads of a CTA
constexpr int kRows = 32;               // rows of a warp
constexpr int kPitch = kN + 16;         // bytes of a staged row of int8: 8 lanes' 16-byte reads cover all banks
constexpr int kPitch4 = kN / 2 + 16;    // ... of int4

__device__ __forceinline__ void async_copy16(void* dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A product that is rounded before it is added to anything: a packed multiplication and the packed addition of its
// result come out of the assembler as one fused multiply-add, -fmad=false or not
__device__ __forceinline__ float2 product2(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }

// A warp's rows between global memory (dense, BYTES per row) and its stage (PITCH), 16 bytes per lane and step
template <int BYTES, int PITCH>
__device__ __forceinline__ void fetch_rows(uint8_t* stage, const void* src, int lane) {
#pragma unroll
  for (int i = 0; i < kRows * BYTES / 512; ++i) {
    const int c = lane + 32 * i;
    async_copy16(stage + (c / (BYTES / 16)) * PITCH + (c % (BYTES / 16)) * 16, static_cast<const uint8_t*>(src) + 16 * c);
  }
}
template <int BYTES, int PITCH>
__device__ __forceinline__ void put_rows(void* dst, const uint8_t* stage, int lane) {
#pragma unroll
  for (int i = 0; i < kRows * BYTES / 512; ++i) {
    const int c = lane + 32 * i;
    *reinterpret_cast<uint4*>(static_cast<uint8_t*>(dst) + 16 * c) =
        *reinterpret_cast<const uint4*>(stage + (c / (BYTES / 16)) * PITCH + (c % (BYTES / 16)) * 16);
  }
}

// the four codes of a word as two pairs
__device__ __forceinline__ void s8x4(uint32_t w, float2& a, float2& b) {
  a = s8x2_cvt<0, 1>(w);
  b = s8x2_to_float<2, 3>(w ^ 0x80808080u);
}
// the eight int4 codes of a word as four pairs
__device__ __forceinline__ void s4x8(uint32_t w, float2 (&e)[4]) {
  const uint32_t lo = (w ^ 0x88888888u) & 0x0F0F0F0Fu, hi = ((w ^ 0x88888888u) >> 4) & 0x0F0F0F0Fu;
  const float2 bias = splat(-kMagicNib);
  auto pair = [&](uint32_t sel) {
    return add2(make_float2(__uint_as_float(__byte_perm(lo, 0x4B000000u, sel)), __uint_as_float(__byte_perm(hi, 0x4B000000u, sel))), bias);
  };
  e[0] = pair(0x7440); e[1] = pair(0x7441); e[2] = pair(0x7442); e[3] = pair(0x7443);
}

// One element whose remainder lies within the tie guard, by the true quotient.  Element by element: a state that its
// inputs hold at a fixed point has remainders near half a step in every row, so a word of codes often has one.
__device__ __forceinline__ void redecide(float x, float& e, float& y, float s, float thr) {
  if (fabsf(e) > thr) {
    const float code = exact_code(x, s);
    y = __fadd_rn(code, kMagicRound);
    e = __fadd_rn(x, -__fmul_rn(code, s));
  }
}

// round_half_even(x / s) of a row of 64 by the reciprocal (exact: see the tie guard in carry_gdn_tile128.cuh), handed to
// `put` pair by pair as code + kMagicRound; KEEP: the remainders x - code * s, the product rounded first, stay in x.
// Returns the largest remainder.
template <bool KEEP, class Put>
__device__ __forceinline__ float quantize_row(float2 (&x)[kN / 2], float s, Put&& put) {
  const float2 inv2 = splat(rcp_refined(s)), ns2 = splat(-s), magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);
  const float thr = s * kTieGuard;
  float worst = 0.f;
#pragma unroll
  for (int j = 0; j < kN / 2; j += 4) {
    float2 y[4], e[4];
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = fma2(x[j + i], inv2, magic2);
      e[i] = add2(x[j + i], product2(add2(y[i], nmagic2), ns2));
      m = max3abs(m, e[i]);
    }
    if (m > thr) {                      // a quotient that the reciprocal may have tipped over a tie
      m = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        redecide(x[j + i].x, e[i].x, y[i].x, s, thr); redecide(x[j + i].y, e[i].y, y[i].y, s, thr);
        m = max3abs(m, e[i]);
      }
    }
    worst = fmaxf(worst, m);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      if (KEEP) { x[j + i] = e[i]; x[j + i + 1] = e[i + 1]; }
      put(j + i, y[i], y[i + 1]);
    }
  }
  return worst;
}

// The same for a row that holds a NaN or an infinity, or whose scale is one (the reciprocal makes NaNs of all its quotients):
// element by element as the generic kernel does it, codes straight into the lane's staged row.
__device__ __noinline__ float quantize_row_plainly(float* x, float s, float qmax, uint8_t* to, bool nibbles) {
  float worst = 0.f;
#pragma unroll 1
  for (int i = 0; i < kN; ++i) {
    const float code = quantize_div(x[i], s, qmax);
    x[i] = __fadd_rn(x[i], -__fmul_rn(code, s));
    worst = fmaxf(worst, fabsf(x[i]));
    const uint32_t c = (uint32_t)(int)code;
    if (!nibbles) to[i] = (uint8_t)c;
    else to[i / 2] = (uint8_t)((i & 1) ? (to[i / 2] | (c << 4)) : (c & 15u));
  }
  return worst;
}

template <int RES, int RSCALE, int QDT>
__global__ void __launch_bounds__(kPair, 6) gdn_narrow_kernel(const __grid_constant__ KParams p) {
  constexpr bool kInt4 = RES == CARRY_RES_INT4, kPerV = RSCALE == CARRY_SCALE_PER_V;
  constexpr int kRowR = kInt4 ? kN / 2 : kN, kPitchR = kInt4 ? kPitch4 : kPitch;   // residual: bytes of a row, and staged
  __shared__ __align__(16) uint8_t codes_all[2][kRows * kPitch];
  __shared__ __align__(16) uint8_t resid_all[2][kRows * kPitchR];
  __shared__ __align__(16) float kq_all[2][2][kN];       // per warp: k and q, normalised and scaled
  __shared__ float head_red[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint8_t *st_codes = codes_all[warp], *st_resid = resid_all[warp];
  int n, hv, h;
  split_tile(p, (int)blockIdx.x, n, hv, h);

  depend_release();
  depend_wait();
  const int slot_id = p.slot_idx[(long long)n * p.stride_idx];
  const GateRaw raw = gate_loads(p, n, hv, 0, 0);
  const long long row = (long long)n * p.stride_mixed_tok;
  auto raw_at = [&](long long i) { return load_raw(p.q, row + i, QDT); };
  uint32_t rq[2], rk[2];                                 // elements lane and lane + 32
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    rq[i] = raw_at((long long)h * kN + lane + 32 * i);
    rk[i] = raw_at(((long long)p.H + h) * kN + lane + 32 * i);
  }
  const uint32_t rv = raw_at(2LL * p.H * kN + (long long)hv * kN + tid);
  const long long out_at = ((long long)n * p.HV + hv) * kN + tid;
  if (slot_id <= 0 || slot_id >= p.num_slots) {          // padding (or a bad id, which is reported): the pool stays as it is
    if (slot_id > 0 && tid == 0 && p.status) atomicOr(p.status, CARRY_GDN_STATUS_BAD_SLOT);
    store_from_float(p.out, out_at, p.o_dtype, 0.f);
    return;
  }
  const long long slot = slot_id;
  int8_t* codes = p.codes_out + slot * p.stride_state_slot + ((long long)hv * kN + kRows * warp) * kN;
  uint8_t* resid = reinterpret_cast<uint8_t*>(p.resid_out) + slot * p.stride_resid_slot + ((long long)hv * kN + kRows * warp) * kRowR;
  float* sscale = p.sscale_out + slot * p.stride_sscale_slot + (long long)hv * kN + tid;
  float* rscale = p.rscale_out + slot * p.stride_rscale_slot + (kPerV ? (long long)hv * kN + tid : (long long)hv);
  fetch_rows<kN, kPitch>(st_codes, codes, lane);
  fetch_rows<kRowR, kPitchR>(st_resid, resid, lane);
  const float s = __ldcg(sscale), es = __ldcg(rscale);

  float alpha, beta;
  gates_from(p, raw, alpha, beta);
  float* sk = kq_all[warp][0];
  float* sq = kq_all[warp][1];
  {
    float qf[2], kf[2], qs[2], ks[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      qf[i] = raw_to_float(rq[i], QDT); kf[i] = raw_to_float(rk[i], QDT);
      qs[i] = __fmul_rn(qf[i], qf[i]); ks[i] = __fmul_rn(kf[i], kf[i]);
    }
    if (p.l2norm) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          qs[i] = __fadd_rn(qs[i], __shfl_xor_sync(0xffffffffu, qs[i], o));
          ks[i] = __fadd_rn(ks[i], __shfl_xor_sync(0xffffffffu, ks[i], o));
        }
      const float qn = sqrtf(__fadd_rn(__fadd_rn(qs[0], qs[1]), 1e-6f)), kn = sqrtf(__fadd_rn(__fadd_rn(ks[0], ks[1]), 1e-6f));
#pragma unroll
      for (int i = 0; i < 2; ++i) { qf[i] = __fdiv_rn(qf[i], qn); kf[i] = __fdiv_rn(kf[i], kn); }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) { sq[lane + 32 * i] = __fmul_rn(qf[i], p.qscale); sk[lane + 32 * i] = kf[i]; }
  }
  async_copies_landed();
  __syncwarp();                         // the rows were fetched, k and q written, by other lanes of this warp

  // dequantise, decay, <row, k>
  const uint8_t* my_codes = st_codes + lane * kPitch;
  const uint8_t* my_resid = st_resid + lane * kPitchR;
  float2 x[kN / 2];
  float dot = 0.f;
#pragma unroll
  for (int c = 0; c < kN / 16; ++c) {
    const uint4 w4 = lds_v4(my_codes + 16 * c);
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float2 a, b;
      s8x4(w[m], a, b);
      a = product2(mul2(a, splat(s)), splat(alpha)); b = product2(mul2(b, splat(s)), splat(alpha));
      const float4 k4 = *reinterpret_cast<const float4*>(sk + 16 * c + 4 * m);
      dot = fmaf(a.x, k4.x, dot); dot = fmaf(a.y, k4.y, dot); dot = fmaf(b.x, k4.z, dot); dot = fmaf(b.y, k4.w, dot);
      x[8 * c + 2 * m] = a; x[8 * c + 2 * m + 1] = b;
    }
  }
  // rank-1 write, <row, q>, residual; the row's maximum
  const float2 dv2 = splat(__fmul_rn(beta, __fadd_rn(raw_to_float(rv, QDT), -dot))), es2 = splat(es);
  float o = 0.f, amax = 0.f;
  auto advance = [&](int j, float2 e) {                   // the pair j of the row; e: its residual codes
    const float2 k2 = *reinterpret_cast<const float2*>(sk + 2 * j), q2 = *reinterpret_cast<const float2*>(sq + 2 * j);
    const float2 hn = add2(x[j], product2(k2, dv2));
    o = fmaf(hn.x, q2.x, o); o = fmaf(hn.y, q2.y, o);
    x[j] = add2(hn, product2(e, es2));
    amax = max3abs(amax, x[j]);
  };
#pragma unroll
  for (int c = 0; c < kRowR / 16; ++c) {
    const uint4 w4 = lds_v4(my_resid + 16 * c);
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if constexpr (kInt4) {
        float2 e[4];
        s4x8(w[m], e);
#pragma unroll
        for (int i = 0; i < 4; ++i) advance(16 * c + 4 * m + i, e[i]);
      } else {
        float2 a, b;
        s8x4(w[m], a, b);
        advance(8 * c + 2 * m, a);
        advance(8 * c + 2 * m + 1, b);
      }
    }
  }
  store_from_float(p.out, out_at, p.o_dtype, o);

  // state codes into the stage (a lane's own row), remainders in place of the targets
  const float snew = scale_from_amax(amax, p.qmax, p.eps_mode);
  *sscale = snew;
  // maxima pass a NaN over; the sum for the output keeps the state's, and those of the residual come from its scale
  const float inf = __int_as_float(0x7f800000);
  const bool finite = fabsf(o) < inf && snew < inf && fabsf(es) < inf;
  float plain[kN];                      // the row of a lane that has to go element by element
  auto take_plain = [&]() {
#pragma unroll
    for (int j = 0; j < kN / 2; ++j) { plain[2 * j] = x[j].x; plain[2 * j + 1] = x[j].y; }
  };
  uint32_t word[4];
  float emax;
  if (finite) {
    emax = quantize_row<true>(x, snew, [&](int j, float2 a, float2 b) {
      word[(j / 2) & 3] = pack4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
      if ((j & 7) == 6) *reinterpret_cast<uint4*>(st_codes + lane * kPitch + (j / 8) * 16) = make_uint4(word[0], word[1], word[2], word[3]);
    });
  } else {
    take_plain();
    emax = quantize_row_plainly(plain, snew, p.qmax, st_codes + lane * kPitch, false);
  }
  // residual scale and codes
  constexpr float rqmax = kInt4 ? 7.0f : 127.0f;
  float top = emax;
  if constexpr (!kPerV) {
    top = warp_max_nonneg(emax);
    if (lane == 0) head_red[warp] = top;
    __syncthreads();
    top = fmaxf(head_red[0], head_red[1]);
  }
  const float esn = scale_from_amax(top, rqmax, p.eps_mode);
  if (kPerV || tid == 0) *rscale = esn;
  if (!finite || !(esn < inf)) {
    if (finite) take_plain();
    quantize_row_plainly(plain, esn, rqmax, st_resid + lane * kPitchR, kInt4);
  } else if constexpr (kInt4) {
    uint32_t by[4];
    quantize_row<false>(x, esn, [&](int j, float2 a, float2 b) {
      // 16 * odd + even in one float whose low byte is the pair, each nibble offset by 8
      by[(j & 3)] = __float_as_uint(fmaf(__fadd_rn(a.y, -kMagicRound), 16.0f, __fadd_rn(a.x, 136.0f)));
      by[(j & 3) + 1] = __float_as_uint(fmaf(__fadd_rn(b.y, -kMagicRound), 16.0f, __fadd_rn(b.x, 136.0f)));
      if ((j & 3) == 2) word[(j / 4) & 3] = pack4(by[0], by[1], by[2], by[3]) ^ 0x88888888u;
      if ((j & 15) == 14) *reinterpret_cast<uint4*>(st_resid + lane * kPitchR + (j / 16) * 16) = make_uint4(word[0], word[1], word[2], word[3]);
    });
  } else {
    quantize_row<false>(x, esn, [&](int j, float2 a, float2 b) {
      word[(j / 2) & 3] = pack4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
      if ((j & 7) == 6) *reinterpret_cast<uint4*>(st_resid + lane * kPitchR + (j / 8) * 16) = make_uint4(word[0], word[1], word[2], word[3]);
    });
  }
  __syncwarp();
  put_rows<kN, kPitch>(codes, st_codes, lane);
  put_rows<kRowR, kPitchR>(resid, st_resid, lane);
}

template <int RES, int RSCALE>
int launch_dtype64(const KParams& p, cudaStream_t stream) {
  const dim3 grid((unsigned)((long long)p.B * p.HV));
  if (p.qkv_dtype == CARRY_F32) return launch_dependent(gdn_narrow_kernel<RES, RSCALE, CARRY_F32>, grid, kPair, 0, stream, p);
  if (p.qkv_dtype == CARRY_BF16) return launch_dependent(gdn_narrow_kernel<RES, RSCALE, CARRY_BF16>, grid, kPair, 0, stream, p);
  return launch_dependent(gdn_narrow_kernel<RES, RSCALE, CARRY_F16>, grid, kPair, 0, stream, p);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

// K = V = 64 and every row of codes and residual on a 16-byte boundary (copies and stores are 16 bytes wide; scales
// and activations are read element by element)
bool narrow64_eligible(const KParams& p) {
  if (!p.packed || p.K != kN || p.V != kN) return false;
  if (p.res_fmt != CARRY_RES_INT8 && p.res_fmt != CARRY_RES_INT4) return false;
  if ((long long)p.B * p.HV > 0x7fffffffLL) return false;
  return aligned16(p.codes_out) && aligned16(p.resid_out) && p.stride_state_slot % 16 == 0 && p.stride_resid_slot % 16 == 0;
}

int launch_narrow64(const KParams& p_in, cudaStream_t stream) {
  KParams p = p_in;
  fill_shifts(p);
  const bool i4 = p.res_fmt == CARRY_RES_INT4, pv = p.rscale_mode == CARRY_SCALE_PER_V;
  if (i4) return pv ? launch_dtype64<CARRY_RES_INT4, CARRY_SCALE_PER_V>(p, stream)
                    : launch_dtype64<CARRY_RES_INT4, CARRY_SCALE_PER_HEAD>(p, stream);
  return pv ? launch_dtype64<CARRY_RES_INT8, CARRY_SCALE_PER_V>(p, stream)
            : launch_dtype64<CARRY_RES_INT8, CARRY_SCALE_PER_HEAD>(p, stream);
}

}  // namespace carry
