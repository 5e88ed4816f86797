// Statequant layout [K][V] with 128-wide heads (K = V = 128): the quantized step with an int8, a packed int4 or no residual.
//
// What bounds it is the issue of instructions, and with 8 warps per tile (lane = 4 columns x 16 rows, 128 registers, 16
// warps per SM; the shape of carry_gdn_tile128.cuh) a scheduler issued in 43 % of its cycles: too few warps to cover the
// latencies of a tile's chain of column reductions, and every warp finished all 128 columns' sums and scales for itself.
// Here 16 warps share a tile, lane = 4 columns x 8 rows in 64 registers, so that an SM holds 32 warps in two CTAs.  A
// column's reduction is finished once, by its lane of the first four warps, which leaves what the others need (the
// delta, the scales and their reciprocals) in shared memory (four lanes per column, over all 16 warps, measured 5 % slower:
// more instructions in all); a scale per head needs one maximum per warp
// only.  256 requests x 32 heads, against that shape: no residual, one scale per head 129 -> 96 us, per V 133 -> 101; int8
// residual 164 -> 138, int4 172 -> 145 (one scale per head); 16 requests, int8 16.7 -> 13.2.
//
// A CTA is persistent (tile = blockIdx.x + number * gridDim.x) and loads with bulk copies into a ring of up to 4 stages; a
// stage is requested again after the meeting behind the last read of it.  Addresses follow from the tile's index, the
// gates are loaded one tile ahead and <k, q> is one warp's work meanwhile, so a launch begins with its first tile's
// copies and nothing ahead of them.
//
// Without a residual there is a second form (LOOSE) for calls that the bulk copies or the division shortcut do not take:
// activations and scales that start off a 16-byte boundary, a qmax that is not 2^(bits-1) - 1 for 3..8 bits.  It copies
// the codes alone and reads the vectors where they are used: 256 requests x 32 heads on 2 bits 113 us with one scale per head
// (133 per V), where the generic kernel takes 3.3 ms.
#include "carry_gdn_tile128.cuh"

namespace carry {
namespace {

constexpr int kWide = 512;              // threads of a CTA
constexpr int kWideWarps = kWide / 32;
constexpr int kLaneRows = kT / kWideWarps;

template <int RES, int RSCALE, int QDT, bool LOOSE>
struct Dense128 {
  static_assert(!LOOSE || RES == CARRY_RES_NONE, "the other formats have the generic kernel");
  static constexpr bool kNone = RES == CARRY_RES_NONE, kInt4 = RES == CARRY_RES_INT4;
  static constexpr bool kHeadState = kNone && RSCALE == CARRY_SCALE_PER_HEAD;     // RSCALE: the state's granularity then
  static constexpr bool kHeadResid = !kNone && RSCALE == CARRY_SCALE_PER_HEAD;
  static constexpr bool kColState = !kHeadState, kColResid = !kNone && !kHeadResid;
  static constexpr int kVec = kT * (QDT == CARRY_F32 ? 4 : 2);
  // a stage
  static constexpr int kResidBytes = kNone ? 0 : kInt4 ? kT * kT / 2 : kT * kT;
  static constexpr int kResid = kT * kT;
  static constexpr int kSScale = kResid + kResidBytes;
  static constexpr int kRScale = kSScale + (kColState && !LOOSE ? 512 : 0);
  static constexpr int kQ = kRScale + (kColResid ? 512 : 0);
  static constexpr int kK = kQ + kVec;
  static constexpr int kV = kK + kVec;
  static constexpr int kStage = LOOSE ? kQ : kV + kVec;
  static_assert(kStage % 128 == 0, "stages keep the ring's alignment");
  // behind the ring; partial results lie [warp][column]
  static constexpr int kDotRow = kT * 8, kMaxRow = kT * 4;
  static constexpr int kRed = 0;                                     // sums, then maxima in the same place
  static constexpr int kRows = kRed + kWideWarps * kDotRow;          // {k, k, q, q} per row
  static constexpr int kDelta = kRows + kT * 16;                     // per column: delta; scale; reciprocal
  static constexpr int kScale = kDelta + kT * 4;
  static constexpr int kInv = kScale + kT * 4;
  static constexpr int kKq = kInv + kT * 4;                          // <k, q>
  static constexpr int kHead = kKq + 16;                             // per warp: its maximum
  static constexpr int kScratch = kHead + kWideWarps * 4;
  static constexpr int kFit = (113 * 1024 - kScratch - 128) / kStage;    // two CTAs per SM, 1 KB each for the system
  static constexpr int kStages = kFit < 4 ? kFit : 4;
  static_assert(kStages >= 2, "one tile in hand, one on the way");
  static constexpr int kBytes = kStages * kStage + kScratch;
};

// One thread requests a tile: the bytes to come are announced, then copied.
template <int RES, int RSCALE, int QDT, bool LOOSE>
__device__ __forceinline__ void request_tile(const KParams& p, uint8_t* sb, uint64_t* bar, int tile) {
  using D = Dense128<RES, RSCALE, QDT, LOOSE>;
  const long long nh = tile;
  if constexpr (LOOSE) {
    mbar_arrive_expect_tx(bar, kT * kT + test_extra_tx(tile));
    bulk_load(sb, p.codes_in + nh * kT * kT, kT * kT, bar);
    return;
  }
  mbar_arrive_expect_tx(bar, kT * kT + D::kResidBytes + (D::kColState ? 512 : 0) + (D::kColResid ? 512 : 0) + 3 * D::kVec + test_extra_tx(tile));
  bulk_load(sb, p.codes_in + nh * kT * kT, kT * kT, bar);
  if constexpr (D::kColState) bulk_load(sb + D::kSScale, p.sscale_in + nh * kT, 512, bar);
  bulk_load(sb + D::kK, reinterpret_cast<const uint8_t*>(p.k) + nh * D::kVec, D::kVec, bar);
  bulk_load(sb + D::kQ, reinterpret_cast<const uint8_t*>(p.q) + nh * D::kVec, D::kVec, bar);
  bulk_load(sb + D::kV, reinterpret_cast<const uint8_t*>(p.v) + nh * D::kVec, D::kVec, bar);
  if constexpr (!D::kNone) bulk_load(sb + D::kResid, reinterpret_cast<const uint8_t*>(p.resid_in) + nh * D::kResidBytes, D::kResidBytes, bar);
  if constexpr (D::kColResid) bulk_load(sb + D::kRScale, p.rscale_in + nh * kT, 512, bar);
}

template <int RES, int RSCALE, int QDT, bool LOOSE>
__global__ void __launch_bounds__(kWide, 2) gdn_dense128_kernel(const __grid_constant__ KParams p) {
  using D = Dense128<RES, RSCALE, QDT, LOOSE>;
  constexpr int S = D::kStages;
  constexpr bool kFold = D::kInt4 || D::kNone;           // sums over the bare codes, the column's scale on the totals
  constexpr float rqmax = D::kInt4 ? 7.0f : 127.0f, rrqmax = 1.0f / rqmax;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t full_bar[S];
  __shared__ int poison_flag;
  volatile int* poison = &poison_flag;
  uint8_t* scratch = smem + S * D::kStage;
  float* delta = reinterpret_cast<float*>(scratch + D::kDelta);
  float* scale_of = reinterpret_cast<float*>(scratch + D::kScale);
  float* inv_of = reinterpret_cast<float*>(scratch + D::kInv);
  float* kq_sum = reinterpret_cast<float*>(scratch + D::kKq);
  float* head_max = reinterpret_cast<float*>(scratch + D::kHead);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = kLaneRows * warp, c0 = 4 * lane;        // my rows and columns
  const int col = tid;                                   // the column whose reductions I finish, in the first four warps
  const bool finisher = warp < kT / 32;
  float4* kq_row = reinterpret_cast<float4*>(scratch + D::kRows) + r0;
  const int total = p.B * p.HV, step = (int)gridDim.x;

  depend_release();
  if (tid == 0) {
    poison_flag = 0;
    for (int s = 0; s < S; ++s) mbar_init(&full_bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  depend_wait();
  if (tid == 0)
    for (int s = 0; s < S && (int)blockIdx.x + s * step < total; ++s)
      request_tile<RES, RSCALE, QDT, LOOSE>(p, smem + s * D::kStage, &full_bar[s], (int)blockIdx.x + s * step);
  // gates (and a scale per head) of the tile in hand and of the next one
  float alpha_next = __ldcg(p.alpha + blockIdx.x), beta_next = __ldcg(p.beta + blockIdx.x), head_next = 0.f;
  const float* head_scale = D::kHeadState ? p.sscale_in : p.rscale_in;
  if constexpr (D::kHeadState || D::kHeadResid) head_next = __ldcg(head_scale + blockIdx.x);

  // partial maxima of my columns -> the whole maximum of column `col`
  auto put_max = [&](const float (&m)[4]) {
    *reinterpret_cast<float4*>(scratch + D::kRed + warp * D::kMaxRow + 16 * lane) = make_float4(m[0], m[1], m[2], m[3]);
  };
  auto col_max = [&]() {
    const float* x = reinterpret_cast<const float*>(scratch + D::kRed) + col;
    float m = 0.f;
#pragma unroll
    for (int w = 0; w < kWideWarps; w += 2) m = fmaxf(fmaxf(m, x[w * kT]), x[(w + 1) * kT]);
    return m;
  };
  auto head_of = [&](const float (&m)[4]) {              // one warp's maximum, for all
    const float top = warp_max_nonneg(fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])));
    if (lane == 0) head_max[warp] = top;
  };
  auto new_scale = [&](float m) {
    if constexpr (LOOSE) return scale_from_amax(m, p.qmax, p.eps_mode);
    return scale_fast(m, p.qmax, p.inv_qmax, p.eps_mode);
  };
  // ... and as it is written out: the shortcut makes a NaN of an infinite maximum, whose quotient is infinite
  auto put_scale = [&](float* to, float m, float sn) { *to = D::kNone && m == __int_as_float(0x7f800000) ? m : sn; };
  auto all_heads = [&]() { return warp_max_nonneg(head_max[lane & (kWideWarps - 1)]); };

  int s = 0;
  uint32_t parity = 0;
  bool healthy = true;
  for (int tile = blockIdx.x; tile < total; tile += step) {
    const float alpha = alpha_next, beta = beta_next, head_in = head_next;
    if (tile + step < total) {
      alpha_next = __ldcg(p.alpha + tile + step); beta_next = __ldcg(p.beta + tile + step);
      if constexpr (D::kHeadState || D::kHeadResid) head_next = __ldcg(head_scale + tile + step);
    }
    uint8_t* sb = smem + s * D::kStage;
    healthy = mbar_wait(&full_bar[s], parity, poison, p.status);
    const long long vec0 = (long long)tile * kT;         // where this tile's vectors start
    auto vec_at = [&](const void* x, int stage_off, int i) {
      if constexpr (LOOSE) return raw_to_float(load_raw(x, vec0 + i, QDT), QDT);
      return act<QDT>(sb + stage_off, i);
    };

    // k and q of my warp's rows, each twice side by side
    {
      const float x = vec_at((lane & 8) ? p.q : p.k, (lane & 8) ? D::kQ : D::kK, r0 + (lane & 7));
      if (lane < 16) *reinterpret_cast<float2*>(reinterpret_cast<float*>(kq_row + (lane & 7)) + ((lane & 8) ? 2 : 0)) = splat(x);
      __syncwarp();
    }
    if (warp == kWideWarps - 1) {
      float4 k4, q4;
      if constexpr (LOOSE) {
        auto four = [&](const void* x) {
          return make_float4(vec_at(x, 0, 4 * lane), vec_at(x, 0, 4 * lane + 1), vec_at(x, 0, 4 * lane + 2), vec_at(x, 0, 4 * lane + 3));
        };
        k4 = four(p.k); q4 = four(p.q);
      } else {
        k4 = act4<QDT>(sb + D::kK, 4 * lane); q4 = act4<QDT>(sb + D::kQ, 4 * lane);
      }
      float y = fmaf(k4.w, q4.w, fmaf(k4.z, q4.z, fmaf(k4.y, q4.y, k4.x * q4.x)));
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (lane == 0) *kq_sum = y;
    }
    // dequantise, decay, column sums over my rows
    const float2 alpha2 = splat(alpha);
    float2 hA[kLaneRows], hB[kLaneRows], saA, saB;
    {
      float2 sA, sB;
      if constexpr (D::kHeadState) {
        sA = sB = splat(head_in);
      } else if constexpr (LOOSE) {
        const float* x = p.sscale_in + vec0 + c0;
        sA = make_float2(__ldcg(x), __ldcg(x + 1)); sB = make_float2(__ldcg(x + 2), __ldcg(x + 3));
      } else {
        const float4 s4 = *reinterpret_cast<const float4*>(sb + D::kSScale + 4 * c0);
        sA = make_float2(s4.x, s4.y); sB = make_float2(s4.z, s4.w);
      }
      saA = mul2(sA, alpha2); saB = mul2(sB, alpha2);
      float2 dkA = splat(0.f), dkB = dkA, dqA = dkA, dqB = dkA;
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(sb + (r0 + i) * kT + c0);
        float2 a = s8x2_cvt<0, 1>(w), b = s8x2_to_float<2, 3>(w ^ 0x80808080u);
        if constexpr (!kFold) { a = mul2(mul2(a, sA), alpha2); b = mul2(mul2(b, sB), alpha2); }
        hA[i] = a; hB[i] = b;
        const float4 kq4 = kq_row[i];
        const float2 kr = make_float2(kq4.x, kq4.y), qr = make_float2(kq4.z, kq4.w);
        dkA = fma2(a, kr, dkA); dkB = fma2(b, kr, dkB);
        dqA = fma2(a, qr, dqA); dqB = fma2(b, qr, dqB);
      }
      if constexpr (kFold) { dkA = mul2(dkA, saA); dkB = mul2(dkB, saB); dqA = mul2(dqA, saA); dqB = mul2(dqB, saB); }
      float4* dst = reinterpret_cast<float4*>(scratch + D::kRed + warp * D::kDotRow + 8 * c0);
      dst[0] = make_float4(dkA.x, dqA.x, dkA.y, dqA.y);
      dst[1] = make_float4(dkB.x, dqB.x, dkB.y, dqB.y);
    }
    if (!__syncthreads_and(healthy)) { healthy = false; break; }      // nothing of this tile has been written
    if (finisher) {
      const float2* x = reinterpret_cast<const float2*>(scratch + D::kRed) + col;
      float2 d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) d[j] = x[j * kT];
#pragma unroll
      for (int w = 4; w < kWideWarps; ++w) d[w & 3] = add2(d[w & 3], x[w * kT]);
      const float2 sum = add2(add2(d[0], d[1]), add2(d[2], d[3]));
      const float dv = __fmul_rn(beta, __fadd_rn(vec_at(p.v, D::kV, col), -sum.x));
      delta[col] = dv;
      // (0 * dv: the sum over rows of an infinite write has both signs in it; the folded sum alone would not show that)
      const float hq = D::kNone ? fmaf(0.f, dv, sum.y) : sum.y;
      store_from_float(p.out, (long long)tile * kT + col, p.o_dtype, fmaf(dv, *kq_sum, hq));
    }
    __syncthreads();
    // rank-1 write, residual, column maxima
    float m[4] = {0.f, 0.f, 0.f, 0.f};
    {
      const float4 d4 = *reinterpret_cast<const float4*>(delta + c0);
      const float2 dvA = make_float2(d4.x, d4.y), dvB = make_float2(d4.z, d4.w);
      float2 esA = splat(head_in), esB = esA;
      if constexpr (D::kColResid) {
        const float4 e4 = *reinterpret_cast<const float4*>(sb + D::kRScale + 4 * c0);
        esA = make_float2(e4.x, e4.y); esB = make_float2(e4.z, e4.w);
      }
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) {
        const float2 kr = *reinterpret_cast<const float2*>(kq_row + i);
        if constexpr (D::kNone) {
          hA[i] = fma2(hA[i], saA, mul2(kr, dvA)); hB[i] = fma2(hB[i], saB, mul2(kr, dvB));
        } else if constexpr (D::kInt4) {
          float2 nA, nB;
          s4x4_pairs(*reinterpret_cast<const uint16_t*>(sb + D::kResid + (r0 + i) * (kT / 2) + c0 / 2), nA, nB);
          hA[i] = fma2(nA, esA, fma2(hA[i], saA, mul2(kr, dvA)));
          hB[i] = fma2(nB, esB, fma2(hB[i], saB, mul2(kr, dvB)));
        } else {
          const uint32_t w = *reinterpret_cast<const uint32_t*>(sb + D::kResid + (r0 + i) * kT + c0) ^ 0x80808080u;
          hA[i] = fma2(s8x2_to_float<0, 1>(w), esA, fma2(kr, dvA, hA[i]));
          hB[i] = fma2(s8x2_to_float<2, 3>(w), esB, fma2(kr, dvB, hB[i]));
        }
        if (i & 1) {                                     // two rows per three-operand maximum
          m[0] = fmaxf(fmaxf(m[0], fabsf(hA[i - 1].x)), fabsf(hA[i].x)); m[1] = fmaxf(fmaxf(m[1], fabsf(hA[i - 1].y)), fabsf(hA[i].y));
          m[2] = fmaxf(fmaxf(m[2], fabsf(hB[i - 1].x)), fabsf(hB[i].x)); m[3] = fmaxf(fmaxf(m[3], fabsf(hB[i - 1].y)), fabsf(hB[i].y));
        }
      }
    }
    if constexpr (D::kHeadState) head_of(m); else put_max(m);
    __syncthreads();
    if (tid == 0 && tile + S * step < total) request_tile<RES, RSCALE, QDT, LOOSE>(p, sb, &full_bar[s], tile + S * step);   // the stage has been read
    // new state scales
    float2 snA, snB, inA, inB;
    if constexpr (D::kHeadState) {
      const float top = all_heads(), sn = new_scale(top);
      snA = snB = splat(sn);
      inA = inB = splat(rcp_refined(sn));
      if (tid == 0) put_scale(p.sscale_out + tile, top, sn);
    } else {
      if (finisher) {
        const float top = col_max(), sn = new_scale(top);
        scale_of[col] = sn;
        inv_of[col] = rcp_refined(sn);
        put_scale(p.sscale_out + (long long)tile * kT + col, top, sn);
      }
      __syncthreads();
      const float4 s4 = *reinterpret_cast<const float4*>(scale_of + c0), i4 = *reinterpret_cast<const float4*>(inv_of + c0);
      snA = make_float2(s4.x, s4.y); snB = make_float2(s4.z, s4.w);
      inA = make_float2(i4.x, i4.y); inB = make_float2(i4.z, i4.w);
    }
    // codes; remainders in place of the targets
    const float2 magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);
    uint32_t cw[kLaneRows];
    {
      const float2 nsA = mul2(snA, splat(-1.0f)), nsB = mul2(snB, splat(-1.0f));
#pragma unroll
      for (int b = 0; b < 4; ++b) m[b] = 0.f;
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) {
        const float2 yA = fma2(hA[i], inA, magic2), yB = fma2(hB[i], inB, magic2);
        hA[i] = fma2(add2(yA, nmagic2), nsA, hA[i]);
        hB[i] = fma2(add2(yB, nmagic2), nsB, hB[i]);
        cw[i] = pack4(__float_as_uint(yA.x), __float_as_uint(yA.y), __float_as_uint(yB.x), __float_as_uint(yB.y));
        if (i & 1) {
          m[0] = fmaxf(fmaxf(m[0], fabsf(hA[i - 1].x)), fabsf(hA[i].x)); m[1] = fmaxf(fmaxf(m[1], fabsf(hA[i - 1].y)), fabsf(hA[i].y));
          m[2] = fmaxf(fmaxf(m[2], fabsf(hB[i - 1].x)), fabsf(hB[i].x)); m[3] = fmaxf(fmaxf(m[3], fabsf(hB[i - 1].y)), fabsf(hB[i].y));
        }
      }
      const float2 thA = mul2(snA, splat(kTieGuardExact)), thB = mul2(snB, splat(kTieGuardExact));
      // One warp in 40 has a quotient within the tie guard, and all sixteen wait for it at the next meeting: only the quads with
      // such an element are gone through again (all eight: 97.0 us instead of 95.9 for 256 requests x 32 heads without a
      // residual, 144.8 instead of 138.1 with int8 and one scale per head).
      if (fmaxf(fmaxf(m[0] - thA.x, m[1] - thA.y), fmaxf(m[2] - thB.x, m[3] - thB.y)) > 0.f) {
        const float sn[4] = {snA.x, snA.y, snB.x, snB.y}, thr[4] = {thA.x, thA.y, thB.x, thB.y};
        m[0] = m[1] = m[2] = m[3] = 0.f;
#pragma unroll
        for (int i = 0; i < kLaneRows; ++i) {
          redecide_quad(hA[i], hB[i], cw[i], sn, thr);
          m[0] = fmaxf(m[0], fabsf(hA[i].x)); m[1] = fmaxf(m[1], fabsf(hA[i].y));
          m[2] = fmaxf(m[2], fabsf(hB[i].x)); m[3] = fmaxf(m[3], fabsf(hB[i].y));
        }
      }
      int8_t* dst = p.codes_out + (long long)tile * kT * kT + r0 * kT + c0;
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) *reinterpret_cast<uint32_t*>(dst + i * kT) = cw[i];
    }
    if constexpr (!D::kNone) {
      if constexpr (D::kHeadResid) head_of(m); else put_max(m);
      __syncthreads();
      if constexpr (D::kHeadResid) {
        const float es = scale_fast(all_heads(), rqmax, rrqmax, p.eps_mode);
        inA = inB = splat(rcp_refined(es));
        if (tid == 0) p.rscale_out[tile] = es;
      } else {
        if (finisher) {
          const float es = scale_fast(col_max(), rqmax, rrqmax, p.eps_mode);
          inv_of[col] = rcp_refined(es);
          p.rscale_out[(long long)tile * kT + col] = es;
        }
        __syncthreads();
        const float4 i4 = *reinterpret_cast<const float4*>(inv_of + c0);
        inA = make_float2(i4.x, i4.y); inB = make_float2(i4.z, i4.w);
      }
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.resid_out) + (long long)tile * D::kResidBytes + (D::kInt4 ? r0 * (kT / 2) + c0 / 2 : r0 * kT + c0);
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) {
        const float2 rA = fma2(hA[i], inA, magic2), rB = fma2(hB[i], inB, magic2);
        if constexpr (D::kInt4) {
          *reinterpret_cast<uint16_t*>(dst + i * (kT / 2)) =
              (uint16_t)pack_s4x4(__float_as_uint(rA.x), __float_as_uint(rA.y), __float_as_uint(rB.x), __float_as_uint(rB.y));
        } else {
          *reinterpret_cast<uint32_t*>(dst + i * kT) = pack4(__float_as_uint(rA.x), __float_as_uint(rA.y), __float_as_uint(rB.x), __float_as_uint(rB.y));
        }
      }
    }
    if (++s == S) { s = 0; parity ^= 1u; }
  }
  // A CTA whose wait ran out leaves copies it has requested a bounded while to land before it gives its memory up.
  if (!healthy) {
#pragma unroll 1
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
}

template <int RES, int RSCALE, int QDT, bool LOOSE>
int launch_wide(const KParams& p, cudaStream_t stream, int sms) {
  auto kern = gdn_dense128_kernel<RES, RSCALE, QDT, LOOSE>;
  constexpr int smem = Dense128<RES, RSCALE, QDT, LOOSE>::kBytes;
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
  const long long tiles = (long long)p.B * p.HV;
  return launch_dependent(kern, dim3((unsigned)(tiles < 2LL * sms ? tiles : 2LL * sms)), kWide, smem, stream, p);
}

template <int RES, int RSCALE, bool LOOSE = false>
int launch_wide_dtype(const KParams& p, cudaStream_t stream, int sms) {
  if (p.qkv_dtype == CARRY_F32) return launch_wide<RES, RSCALE, CARRY_F32, LOOSE>(p, stream, sms);
  if (p.qkv_dtype == CARRY_BF16) return launch_wide<RES, RSCALE, CARRY_BF16, LOOSE>(p, stream, sms);
  return launch_wide<RES, RSCALE, CARRY_F16, LOOSE>(p, stream, sms);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

// Without a residual: any qmax, any number of heads, either granularity, as long as the codes start on a 16-byte boundary.
bool noresid128_eligible(const KParams& p) {
  return !p.packed && p.res_fmt == CARRY_RES_NONE && p.K == kT && p.V == kT && (long long)p.B * p.HV <= 0x7fffffffLL &&
         aligned16(p.codes_in) && aligned16(p.codes_out);
}

int launch_dense128(const KParams& p, cudaStream_t stream, int sms) {
  if (p.res_fmt == CARRY_RES_NONE) {
    const bool per_v = p.sscale_mode == CARRY_SCALE_PER_V;
    const bool loose = !div_qmax_exact(p.qmax) || !aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || (per_v && !aligned16(p.sscale_in));
    if (loose) return per_v ? launch_wide_dtype<CARRY_RES_NONE, CARRY_SCALE_PER_V, true>(p, stream, sms)
                            : launch_wide_dtype<CARRY_RES_NONE, CARRY_SCALE_PER_HEAD, true>(p, stream, sms);
    return per_v ? launch_wide_dtype<CARRY_RES_NONE, CARRY_SCALE_PER_V>(p, stream, sms)
                 : launch_wide_dtype<CARRY_RES_NONE, CARRY_SCALE_PER_HEAD>(p, stream, sms);
  }
  const bool i4 = p.res_fmt == CARRY_RES_INT4, pv = p.rscale_mode == CARRY_SCALE_PER_V;
  if (i4) return pv ? launch_wide_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_V>(p, stream, sms)
                    : launch_wide_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_HEAD>(p, stream, sms);
  return pv ? launch_wide_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_V>(p, stream, sms)
            : launch_wide_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_HEAD>(p, stream, sms);
}

}  // namespace carry
