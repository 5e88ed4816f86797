// Multi-token variant of the slot-indexed decode step: T consecutive tokens of
// every request in one launch.  A (request, head) tile is fetched from the pool
// once, stays in shared memory while its T tokens are applied one after the
// other -- each token is the full step, requantisation and error feedback
// included, exactly as T single-token launches would do it -- and goes back to
// the pool once.  State traffic per token is 1/T of the single-token kernel's.
//
// One CTA (8 warps) per tile, two CTAs per SM.  The per-token arithmetic is that of the streaming kernel
// (carry_gdn_slot_tile.inc), operation for operation and sum for sum, over another split: a lane holds 32 columns (two runs of 16)
// of 2 rows, 8 apart, where it holds 16 columns of 4 rows there.  Sums and maxima then go over 4 lanes instead of 8 and every
// lane has two rows' scalars to work out instead of four.  k and q of a token, scaled, are laid out once for all warps instead
// of once per warp, and the output's store has no branches.  32 requests x 32 heads, us a launch of 4 tokens with the other split
// and with this one: int4, one residual scale per head 64.5 / 62.4, per V row 61.5 / 56.2, int8 per V row 61.0 / 57.8; fp32 activations
// 71.4 / 63.3, 67.3 / 59.5 (int8).  One token, 16-bit activations: 30.9 / 30.8, 31.0 / 30.3, 32.9 / 32.4; up to 16 requests
// level to 1.5 % or ahead.
// Bound: the FMA and ALU pipes, busy for 37 and 38 % of the cycles -- their times add up for most of these instructions, which read
// more than two or three registers -- and, with one scale per head, the meeting of the 8 warps at every token.
// The split's price: rows lie 128 bytes apart (64 for int4), so that the lanes of a 16-byte phase meet on half of the banks: 50 conflicts
// per warp and token, 1.65 M of 6.6 M shared-memory wavefronts of a launch.
// (The streaming kernel has no register left for this split: 60 bytes spill in its loop, 843 us for 24 layers of 64 requests
// instead of 740.)
//
// A warp only ever reads and writes its own 16 rows of the tile, so tokens need no ordering between warps beyond that meeting, which
// is there only with one residual scale per head.  That scale is carried in a register; read back from the staged tile it takes a block
// barrier per token, which is 62.4 us just the same.  With a scale per V row a barrier would hold warps together that need
// nothing from one another: 60.6 instead of 56.2 us for int4, 64.2 instead of 59.7 for int8 (whose re-decision was a call then).
// Activation vectors, gates and norms of up to 8 tokens are fetched together, one trip to global memory per chunk of
// tokens instead of one per token.
#include "carry_gdn_tile128.cuh"

namespace carry {

int launch_multi(const KParams& p, int T, long long stride_mixed_t, long long stride_a_t, long long stride_b_t,
                 cudaStream_t stream);

namespace {

// k and q of a tile as every warp reads them: fp32, times k_mul and q_mul, each quad of columns as {0, 2, 1, 3}.  Quad `Q`
// (columns 4Q..4Q+3) is quad m = 4 * (Q / 16) + Q % 4 of lane t = Q / 4 % 4, since lane t of a row holds columns 16t..16t+15
// (m < 4) and 64+16t..64+16t+15, and lies at 4 * m + t.
struct __align__(16) KqBuf { float4 k[32], q[32]; };
// A lane's place in a tile: the offset of its codes (first row * 128 + first column)
struct SlotLane {
  int codes;
  __device__ __forceinline__ int row() const { return codes >> 7; }
  __device__ __forceinline__ int k() const { return codes & 127; }                   // offset of its first quad of k
};
__device__ __forceinline__ SlotLane slot_lane(int warp, int lane) {
  SlotLane at = {(16 * warp + (lane >> 2)) * kT + 16 * (lane & 3)};
  // kept in a register: worked out again from the thread index wherever it is used it costs 40 instructions per tile
  asm volatile("" : "+r"(at.codes));
  return at;
}
// quad m of k (q: 512 bytes on) from shared memory, read again for each use on purpose: they must not stay in registers
template <int TAG, int VEC>
__device__ __forceinline__ float4 slot_quad(uint32_t addr, int m) {
  constexpr int B = 512 * VEC;
  return (m == 0) ? lds_f4_at<B, TAG>(addr) : (m == 1) ? lds_f4_at<B + 64, TAG>(addr) : (m == 2) ? lds_f4_at<B + 128, TAG>(addr)
         : (m == 3) ? lds_f4_at<B + 192, TAG>(addr) : (m == 4) ? lds_f4_at<B + 256, TAG>(addr) : (m == 5) ? lds_f4_at<B + 320, TAG>(addr)
         : (m == 6) ? lds_f4_at<B + 384, TAG>(addr) : lds_f4_at<B + 448, TAG>(addr);
}
// one vector, k or q, by one warp, lane = quad
__device__ __forceinline__ void put_quad(float4 x, int Q, float mul, float4* to) {
  to[4 * (4 * (Q >> 4) + (Q & 3)) + ((Q >> 2) & 3)] = make_float4(x.x * mul, x.z * mul, x.y * mul, x.w * mul);
}
template <int QDT>
__device__ __forceinline__ void prepare_vector(const uint8_t* vec, int Q, float mul, float4* to) { put_quad(act4<QDT>(vec, 4 * Q), Q, mul, to); }
// Four sums over a row's 4 lanes: lane t ends up with x[t]'s
__device__ __forceinline__ float row_sums4(const float (&x)[4], int t) {
  const bool up2 = t & 2, up1 = t & 1;
  float a[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) a[i] = (up2 ? x[2 + i] : x[i]) + __shfl_xor_sync(0xffffffffu, up2 ? x[i] : x[2 + i], 2);
  return (up1 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, up1 ? a[0] : a[1], 1);
}

// max over the 4 lanes of a row, in each of them
__device__ __forceinline__ float row_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}

__device__ __forceinline__ void shared_max_if(bool on, uint32_t* word, uint32_t v) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %0, 0;\n@p red.shared.max.u32 [%1], %2;\n}\n" ::"r"((int)on), "r"(smem_u32(word)), "r"(v) : "memory");
}
// redecide_rec for the elements of a quad.  It is rarely needed, and written out at every quad it is a third of the kernel's code,
// so that it is a call -- except with an int8 residual and a scale per V row, where the compiler's code around the call costs more
// than the call saves.  Call / in line, us a launch of 32 requests x 32 heads, 4 tokens: int4, one scale per head 62.4 / 63.0;
// int4, per V row 56.2 / 57.3; int8, one scale per head 63.5 / 63.9; int8, per V row 59.7 / 57.8 (fp32 activations 61.3 / 59.5;
// 8 requests of 2 tokens 12.7 / 12.4).  New activations at every token or the same ones: alike.
struct QuadCodes { float2 E, O; uint32_t cw; };
__device__ __forceinline__ QuadCodes redecide_here(QuadCodes x, float s, float thr) {
  float2 yE = add2(s8x2_to_float<0, 2>(x.cw ^ 0x80808080u), splat(kMagicRound));
  float2 yO = add2(s8x2_to_float<1, 3>(x.cw ^ 0x80808080u), splat(kMagicRound));
  redecide_rec(x.E.x, yE.x, s, thr); redecide_rec(x.E.y, yE.y, s, thr);
  redecide_rec(x.O.x, yO.x, s, thr); redecide_rec(x.O.y, yO.y, s, thr);
  x.cw = pack4(__float_as_uint(yE.x), __float_as_uint(yO.x), __float_as_uint(yE.y), __float_as_uint(yO.y));
  return x;
}
__device__ __noinline__ QuadCodes redecide_shared(QuadCodes x, float s, float thr) { return redecide_here(x, s, thr); }

// the codes of a quad's even and odd columns
__device__ __forceinline__ float2 slot_codes_even(uint32_t w) { return s8x2_cvt<0, 2>(w); }
__device__ __forceinline__ float2 slot_codes_odd(uint32_t w) { return s8x2_to_float<1, 3>(w ^ 0x80808080u); }
// store_from_float without a branch on the type, for lanes with `on` set: what is not theirs to write is converted as well.
__device__ __forceinline__ void store_from_float_if(bool on, uint8_t* p, int i, int dtype, float x) {
  const bool wide = dtype == CARRY_F32;
  const unsigned short half = (dtype == CARRY_BF16) ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
  asm volatile(
      "{\n"
      ".reg .pred w, n;\n"
      "setp.ne.u32 w, %0, 0;\n"
      "setp.ne.u32 n, %1, 0;\n"
      "@w st.global.f32 [%2], %3;\n"
      "@n st.global.u16 [%2], %4;\n"
      "}\n" ::"r"((int)(on && wide)), "r"((int)(on && !wide)),
      "l"(p + i * (wide ? 4 : 2)), "f"(x), "h"(half)
      : "memory");
}

struct MultiExtra {
  int T;
  long long stride_mixed_t, stride_a_t, stride_b_t;   // elements from one token of a request to the next
  int first_wave;                                     // CTAs that the device holds at once
};

template <int RES, int RSCALE, int QDT>
__global__ void __launch_bounds__(kThreads, 2) gdn_multi_kernel(const __grid_constant__ KParams p,
                                                               const __grid_constant__ MultiExtra x) {
  using L = StageLayout<RES, LAYOUT_VK, QDT, RSCALE>;
  constexpr int qes = (QDT == CARRY_F32) ? 4 : 2;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t full_bar;
  __shared__ int poison_flag;
  __shared__ uint32_t head_max[4];                    // largest new residual of a token, as bits, by token mod 4
  constexpr int kChunk = 8;                           // tokens whose activations and facts are fetched together
  __shared__ TileMeta meta_t[kChunk];
  __shared__ __align__(16) uint8_t vec_t[kChunk][3 * L::kVecBytes];   // raw q | k | v per token
  __shared__ KqBuf kq_t[kChunk];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* sb = smem;
  volatile int* poison = &poison_flag;
  const int tile = (int)blockIdx.x;
  int n, hv, h;
  split_tile(p, tile, n, hv, h);
  // CTAs that the launch ahead leaves room for start while its last ones run.  What they may do before it has finished
  // is ask the L2 for the state of the slot that the index names now.  32 requests x 32 heads, 4 tokens (1 token): 62.4 us a launch
  // (30.7); launches that start when the one ahead has ended 63.3 (31.3), an early start without hints 63.1 (31.1).  The CTAs
  // behind the first wave find the launch ahead finished, and the look at the index is in their way: hints from all
  // of them, 62.9 (31.0).
  depend_release();
  if (tid == 0 && (int)blockIdx.x < x.first_wave) {
    const long long guess = __ldcg(p.slot_idx + (long long)n * p.stride_idx);
    if (guess > 0 && guess < p.num_slots) {
      unsigned long long a8[8];
      tile_addresses<RES, RSCALE, QDT>(p, n, hv, h, guess, a8);
      l2_prefetch_bulk(reinterpret_cast<const void*>(a8[D_CODES]), kT * kT);
      l2_prefetch_bulk(reinterpret_cast<const void*>(a8[D_RESID]), L::kResidBytes);
    }
  }
  depend_wait();
  long long slot = __ldcg(p.slot_idx + (long long)n * p.stride_idx);
  if (slot >= p.num_slots) {
    if (tid == 0 && p.status) atomicOr(p.status, CARRY_GDN_STATUS_BAD_SLOT);
    slot = 0;
  }
  const long long out_tok0 = ((long long)n * x.T * p.HV + hv) * kT;      // out is [B, T, HV, V]
  const long long out_tok_stride = (long long)p.HV * kT;
  if (slot <= 0) {                                   // padding request: zeros for every token, pool untouched
    for (int i = tid; i < x.T * kT; i += kThreads)
      store_from_float(p.out, out_tok0 + (long long)(i / kT) * out_tok_stride + (i % kT), p.o_dtype, 0.f);
    return;
  }

  __shared__ unsigned long long addr[8];            // where the tile and its activations live (see TileDesc)
  if (tid == 0) {
    unsigned long long a8[8];
    tile_addresses<RES, RSCALE, QDT>(p, n, hv, h, slot, a8);
#pragma unroll
    for (int i = 0; i < 8; ++i) addr[i] = a8[i];
    poison_flag = 0;
    head_max[0] = head_max[1] = head_max[2] = head_max[3] = 0u;
    mbar_init(&full_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // the state of the tile: codes, residual, state scales, residual scale(s)
    mbar_arrive_expect_tx(&full_bar, kT * kT + L::kResidBytes + 512 + L::kRScaleBytes + test_extra_tx(tile));
    bulk_load(sb + L::kCodes, reinterpret_cast<const void*>(a8[D_CODES]), kT * kT, &full_bar);
    bulk_load(sb + L::kResid, reinterpret_cast<const void*>(a8[D_RESID]), L::kResidBytes, &full_bar);
    bulk_load(sb + L::kSScale, reinterpret_cast<const void*>(a8[D_SSCALE]), 512, &full_bar);
    bulk_load(sb + L::kRScale, reinterpret_cast<const void*>(a8[D_RSCALE_IN]), L::kRScaleBytes, &full_bar);
  }
  constexpr float rqmax = (RES == CARRY_RES_INT4) ? 7.0f : 127.0f;
  constexpr float rrqmax = 1.0f / rqmax;             // rounded to nearest, like the host's p.inv_qmax
  const float rqmax_state = p.inv_qmax;
  bool healthy = true;

  const SlotLane at = slot_lane(warp, lane);
  float es_head = 0.f;                               // one residual scale per head: carried from token to token
  for (int t = 0; t < x.T; ++t) {
    const int tc = t % kChunk;
    if (tc == 0) {
      __syncthreads();                               // everybody is done with the previous chunk
      // the next chunk of tokens: q, k, v into shared memory (16 bytes per thread and step), gates and
      // norms by one warp per token
      const int nt = (x.T - t < kChunk) ? (x.T - t) : kChunk;
      constexpr int kVecChunks = 3 * L::kVecBytes / 16;
      for (int i = tid; i < nt * kVecChunks; i += kThreads) {
        const int tt = i / kVecChunks, c = i - tt * kVecChunks;
        const int which = c / (L::kVecBytes / 16), cc = c - which * (L::kVecBytes / 16);
        const uint8_t* src = reinterpret_cast<const uint8_t*>(addr[D_Q + which]) + (long long)(t + tt) * x.stride_mixed_t * qes;
        *reinterpret_cast<uint4*>(&vec_t[tt][16 * c]) = __ldcg(reinterpret_cast<const uint4*>(src) + cc);
      }
      if (warp < nt)
        tile_meta<RES, RSCALE, QDT, 32>(p, tile, lane, true, &meta_t[warp], nullptr,
                                     (long long)(t + warp) * x.stride_mixed_t, (long long)(t + warp) * x.stride_a_t,
                                     (long long)(t + warp) * x.stride_b_t);
      __syncthreads();
      if (warp < nt) {
        prepare_vector<QDT>(&vec_t[warp][0], lane, meta_t[warp].q_mul, kq_t[warp].q);
        prepare_vector<QDT>(&vec_t[warp][L::kVecBytes], lane, meta_t[warp].k_mul, kq_t[warp].k);
      }
      __syncthreads();
    }
    if (t == 0) {                                    // the tile has to be there; the verdict is the CTA's, not a warp's
      mbar_wait(&full_bar, 0u, poison, p.status);
      __syncthreads();
      healthy = !*poison;
      if constexpr (RSCALE == CARRY_SCALE_PER_HEAD) es_head = reinterpret_cast<const float*>(sb + L::kRScale)[hv & 3];
    }
    if (!healthy) break;

    const uint4 tm0 = lds_v4(&meta_t[tc]), tm1 = lds_v4(reinterpret_cast<const uint8_t*>(&meta_t[tc]) + 16);
    const float alpha = __uint_as_float(tm0.w), beta = __uint_as_float(tm1.x), kq = __uint_as_float(tm1.w);
    const float2 alpha2 = splat(alpha);
    const float2 magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);
    uint8_t* out_to = reinterpret_cast<uint8_t*>(p.out) + (out_tok0 + (long long)t * out_tok_stride) * (p.o_dtype == CARRY_F32 ? 4 : 2);

    auto put_out = [&](bool on, int idx, float value) { store_from_float_if(on, out_to, idx, p.o_dtype, value); };
    auto put_sscale = [&](bool on, int r, uint32_t bits) { if (on) *reinterpret_cast<uint32_t*>(sb + L::kSScale + r * 4) = bits; };
    auto put_rscale = [&](bool on, int r, uint32_t bits) { if (on) *reinterpret_cast<uint32_t*>(sb + L::kRScale + r * 4) = bits; };
    auto put16 = [](uint8_t* to, int offset, uint4 v) { *reinterpret_cast<uint4*>(to + offset) = v; };
    auto put8 = [](uint8_t* to, int offset, uint2 v) { *reinterpret_cast<uint2*>(to + offset) = v; };
    // A quad of columns (one 32-bit word of codes) is held as two pairs: E = {col 0, col 2}, O = {col 1, col 3}.
    // Int4 residual: the dot products run over the bare codes (the row's scale * decay goes on the
    // totals) and the target is three fused multiply-adds per pair (phase 2).  Against the int8-residual
    // form below, which keeps the reference's order of roundings, a target moves by a few units in the
    // last place: measured 2e-6 of the state codes and 3e-5 of the int4 residual codes differ from the
    // oracle's, each by one step (limit 1e-3).  An int8 residual code is 18 times finer and already
    // differs in 3e-4 of the elements from reduction order alone, so that format keeps the exact order.
    constexpr bool kFold = (RES == CARRY_RES_INT4);
    const bool odd = lane & 1;
    const uint8_t* codes_at = sb + L::kCodes + at.codes;
    const uint8_t* resid_at = sb + L::kResid + (RES == CARRY_RES_INT4 ? at.codes / 2 : at.codes);
    const float* sscale_at = reinterpret_cast<const float*>(sb + L::kSScale) + at.row();
    const uint32_t k_addr = smem_u32(&kq_t[tc]) + at.k() + order_token();
    float2 hE[2][8], hO[2][8];            // [row][quad]
    // phase 1: dequantise, decay, dot products: per 16 columns one chain for each half of a pair, then over the 8 runs of 16
    const float srow[2] = {sscale_at[0], sscale_at[8]};
    float dot_mine;      // lanes 0..3 of a row pair: <row, k>, <row + 8, k>, <row, q>, <row + 8, q>
    {
      float part[4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t w[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 x = *reinterpret_cast<const uint4*>(codes_at + 8 * kT * i + 64 * j);
          w[i][0] = x.x; w[i][1] = x.y; w[i][2] = x.z; w[i][3] = x.w;
        }
        float2 acc[4] = {};
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const int m = 4 * j + n;
          const float4 kk = slot_quad<2, 0>(k_addr, m), qq = slot_quad<2, 1>(k_addr, m);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            // half of the bytes through the conversion pipe, half through byte permutes (all through either: no gain
            // for int4, 5 % slower for int8)
            float2 e = slot_codes_even(w[i][n]), o = slot_codes_odd(w[i][n]);
            if constexpr (!kFold) { e = mul2(mul2(e, splat(srow[i])), alpha2); o = mul2(mul2(o, splat(srow[i])), alpha2); }
            hE[i][m] = e; hO[i][m] = o;
            acc[i] = fma2(o, make_float2(kk.z, kk.w), fma2(e, make_float2(kk.x, kk.y), acc[i]));
            acc[2 + i] = fma2(o, make_float2(qq.z, qq.w), fma2(e, make_float2(qq.x, qq.y), acc[2 + i]));
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) part[v] = j ? part[v] + (acc[v].x + acc[v].y) : acc[v].x + acc[v].y;
      }
      dot_mine = row_sums4(part, lane & 3);
      // folded form: the sums ran over the bare codes; the row's scale * decay goes on the total
      if constexpr (kFold) dot_mine *= (odd ? srow[1] : srow[0]) * alpha;
    }
    float dv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
      dv[i] = __fmul_rn(beta, __fadd_rn(act<QDT>(&vec_t[tc][2 * L::kVecBytes], at.row() + 8 * i), -__shfl_sync(0xffffffffu, dot_mine, (lane & 28) + i)));
    // the lanes that hold a q total finish that row's output
    put_out(lane & 2, at.row() + (odd ? 8 : 0), fmaf(odd ? dv[1] : dv[0], kq, dot_mine));
    // The two rows one after the other, so that the first one's exchange of maxima hides behind the second one's arithmetic.
    float snew[2], emax[2];
    uint32_t cw[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      // phase 2: dequantise, decay, rank-1 write and residual, each one fused multiply-add; row maximum
      const float es = (RSCALE == CARRY_SCALE_PER_V) ? reinterpret_cast<const float*>(sb + L::kRScale)[at.row() + 8 * i] : es_head;
      const float2 dv2 = splat(dv[i]), es2 = splat(es);
      float amax = 0.f;
      if constexpr (kFold) {
        // target = code * (scale * decay) + k * dv + nibble * es, as three fused multiply-adds.  A
        // nibble (offset binary, 0..15) lands in the byte above a float's low half-word under the
        // exponent of 128, which reads 136 + code; the 136 * es goes into the innermost addend, so the
        // decode costs no arithmetic beyond the byte permute.
        const float2 nb2 = splat(-136.0f * es), sa2 = splat(srow[i] * alpha);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint2 rw = *reinterpret_cast<const uint2*>(resid_at + 8 * (kT / 2) * i + 32 * j);
          const uint32_t wl[2] = {(rw.x ^ 0x88888888u) & 0x0F0F0F0Fu, (rw.y ^ 0x88888888u) & 0x0F0F0F0Fu};
          const uint32_t wh[2] = {((rw.x ^ 0x88888888u) >> 4) & 0x0F0F0F0Fu, ((rw.y ^ 0x88888888u) >> 4) & 0x0F0F0F0Fu};
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            const int m = 4 * j + n;
            const float2 lo = (n & 1) ? nib2_biased<2, 3>(wl[n >> 1]) : nib2_biased<0, 1>(wl[n >> 1]);
            const float2 hi = (n & 1) ? nib2_biased<2, 3>(wh[n >> 1]) : nib2_biased<0, 1>(wh[n >> 1]);
            const float4 kk = i ? slot_quad<1, 0>(k_addr, m) : slot_quad<0, 0>(k_addr, m);
            hE[i][m] = fma2(lo, es2, fma2(hE[i][m], sa2, fma2(make_float2(kk.x, kk.y), dv2, nb2)));
            hO[i][m] = fma2(hi, es2, fma2(hO[i][m], sa2, fma2(make_float2(kk.z, kk.w), dv2, nb2)));
            amax = max3abs(max3abs(amax, hE[i][m]), hO[i][m]);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint4 rw = *reinterpret_cast<const uint4*>(resid_at + 8 * kT * i + 64 * j);
          const uint32_t r[4] = {rw.x, rw.y, rw.z, rw.w};
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            const int m = 4 * j + n;
            const float4 kk = i ? slot_quad<1, 0>(k_addr, m) : slot_quad<0, 0>(k_addr, m);
            hE[i][m] = fma2(slot_codes_even(r[n]), es2, fma2(make_float2(kk.x, kk.y), dv2, hE[i][m]));
            hO[i][m] = fma2(slot_codes_odd(r[n]), es2, fma2(make_float2(kk.z, kk.w), dv2, hO[i][m]));
            amax = max3abs(max3abs(amax, hE[i][m]), hO[i][m]);
          }
        }
      }
      // phase 3: state scale and codes, new residual.  target - code * scale is one fused multiply-add, which is
      // exact here (the difference of two nearly equal numbers), so the target can be rebuilt from the
      // remainder when an element has to be re-decided.  No branch until both rows are done.
      snew[i] = scale_fast(row_max(amax), p.qmax, rqmax_state, p.eps_mode);
      const float2 inv2 = splat(rcp_refined(snew[i])), ns2 = splat(-snew[i]);
      float em = 0.f;
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const float2 yE = fma2(hE[i][m], inv2, magic2);
        const float2 yO = fma2(hO[i][m], inv2, magic2);
        hE[i][m] = fma2(add2(yE, nmagic2), ns2, hE[i][m]);
        hO[i][m] = fma2(add2(yO, nmagic2), ns2, hO[i][m]);
        em = max3abs(max3abs(em, hE[i][m]), hO[i][m]);
        cw[i][m] = pack4(__float_as_uint(yE.x), __float_as_uint(yO.x), __float_as_uint(yE.y), __float_as_uint(yO.y));
      }
      emax[i] = em;
    }
    put_sscale((lane & 2) == 0, at.row() + (odd ? 8 : 0), __float_as_uint(odd ? snew[1] : snew[0]));
    // Some quotient within the tie guard: on activations that change, one warp in 20 per tile; on ones that repeat for 100
    // steps and more an int8 residual settles where a third to half of the warps have one.  The others wait for that warp at
    // the meeting.  Only the quads with such an element are gone through again.
    constexpr bool kInLine = RES == CARRY_RES_INT8 && RSCALE == CARRY_SCALE_PER_V;
    if (fmaxf(fmaf(-snew[0], kTieGuardExact, emax[0]), fmaf(-snew[1], kTieGuardExact, emax[1])) > 0.f) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float thr = snew[i] * kTieGuardExact;
        if (emax[i] > thr) {
          float em = 0.f;
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            if (max3abs(max3abs(0.f, hE[i][m]), hO[i][m]) > thr) {
              const QuadCodes q = {hE[i][m], hO[i][m], cw[i][m]};
              const QuadCodes x = kInLine ? redecide_here(q, snew[i], thr) : redecide_shared(q, snew[i], thr);
              hE[i][m] = x.E; hO[i][m] = x.O; cw[i][m] = x.cw;
            }
            em = max3abs(max3abs(em, hE[i][m]), hO[i][m]);
          }
          emax[i] = em;
        }
      }
    }
    {
      const auto to = (sb + L::kCodes) + at.codes;
      put16(to, 0, make_uint4(cw[0][0], cw[0][1], cw[0][2], cw[0][3]));
      put16(to, 64, make_uint4(cw[0][4], cw[0][5], cw[0][6], cw[0][7]));
      put16(to, 8 * kT, make_uint4(cw[1][0], cw[1][1], cw[1][2], cw[1][3]));
      put16(to, 8 * kT + 64, make_uint4(cw[1][4], cw[1][5], cw[1][6], cw[1][7]));
    }
    // phase 4: residual scale and codes
    float esn[2];
    if constexpr (RSCALE == CARRY_SCALE_PER_V) {
      // no data crosses warps here
#pragma unroll
      for (int i = 0; i < 2; ++i) esn[i] = scale_fast(row_max(emax[i]), rqmax, rrqmax, p.eps_mode);
    } else {
      const uint32_t warp_max = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(emax[0], emax[1])));
      shared_max_if(lane == 0, &head_max[t & 3], warp_max);
      if (tid == 0) head_max[(t + 2) & 3] = 0u;        // last read two meetings ago
      __syncthreads();
      esn[0] = esn[1] = scale_fast(__uint_as_float(*const_cast<volatile uint32_t*>(&head_max[t & 3])), rqmax, rrqmax, p.eps_mode);
    }
    const auto resid_to = (sb + L::kResid) + (RES == CARRY_RES_INT4 ? at.codes / 2 : at.codes);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 inv2 = splat(rcp_refined(esn[i]));
      if constexpr (RES == CARRY_RES_INT4) {
        // even columns: rint(e/es) + 8 + 128 lands in the low mantissa bits; 16 * rint(e/es) of the odd
        // column is added on top, so the low byte of the sum is (odd + 8) << 4 | (even + 8); the final
        // XOR removes the bias of both nibbles.
        const float2 mE = splat(kMagicRound + 136.0f), sixteen = splat(16.0f);
        uint32_t word[4];
#pragma unroll
        for (int m = 0; m < 8; m += 2) {
          const float2 a = fma2(add2(fma2(hO[i][m], inv2, magic2), nmagic2), sixteen, fma2(hE[i][m], inv2, mE));
          const float2 b = fma2(add2(fma2(hO[i][m + 1], inv2, magic2), nmagic2), sixteen, fma2(hE[i][m + 1], inv2, mE));
          word[m / 2] = pack4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y)) ^ 0x88888888u;
        }
        put8(resid_to, 8 * (kT / 2) * i, make_uint2(word[0], word[1]));
        put8(resid_to, 8 * (kT / 2) * i + 32, make_uint2(word[2], word[3]));
      } else {
        uint32_t word[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
          const float2 ye = fma2(hE[i][m], inv2, magic2), yo = fma2(hO[i][m], inv2, magic2);
          word[m] = pack4(__float_as_uint(ye.x), __float_as_uint(yo.x), __float_as_uint(ye.y), __float_as_uint(yo.y));
        }
        put16(resid_to, 8 * kT * i, make_uint4(word[0], word[1], word[2], word[3]));
        put16(resid_to, 8 * kT * i + 64, make_uint4(word[4], word[5], word[6], word[7]));
      }
    }
    if (RSCALE == CARRY_SCALE_PER_V)
      put_rscale((lane & 2) == 0, at.row() + (odd ? 8 : 0), __float_as_uint(odd ? esn[1] : esn[0]));
    if (RSCALE == CARRY_SCALE_PER_HEAD && tid == 0) reinterpret_cast<uint32_t*>(sb + L::kRScale)[hv & 3] = __float_as_uint(esn[0]);
    if constexpr (RSCALE == CARRY_SCALE_PER_HEAD) es_head = esn[0];
    __syncwarp();                                    // a warp's rows are its own: written by one lane, read by another
  }

  __syncthreads();
  if (!healthy || *poison) {                         // the copies never arrived: leave the pool as it was,
#pragma unroll 1
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // after a bounded while for whatever is still on its way
    return;
  }
  // the tile goes back to the pool: 16 bytes per thread and step, whole lines
  for (int i = tid; i < kT * kT / 16; i += kThreads)
    stg_v4(addr[D_CODES] + 16ull * i, *reinterpret_cast<const uint4*>(sb + L::kCodes + 16 * i));
  for (int i = tid; i < L::kResidBytes / 16; i += kThreads)
    stg_v4(addr[D_RESID] + 16ull * i, *reinterpret_cast<const uint4*>(sb + L::kResid + 16 * i));
  if (tid < 32) stg_v4(addr[D_SSCALE] + 16ull * tid, *reinterpret_cast<const uint4*>(sb + L::kSScale + 16 * tid));
  if (RSCALE == CARRY_SCALE_PER_V) {
    if (tid >= 32 && tid < 64)
      stg_v4(addr[D_RSCALE] + 16ull * (tid - 32), *reinterpret_cast<const uint4*>(sb + L::kRScale + 16 * (tid - 32)));
  } else if (tid == 64) {
    stg_b32(addr[D_RSCALE], reinterpret_cast<const uint32_t*>(sb + L::kRScale)[hv & 3]);
  }
}

template <int RES, int RSCALE, int QDT>
int launch_multi_variant(const KParams& p, const MultiExtra& x, cudaStream_t stream) {
  using L = StageLayout<RES, LAYOUT_VK, QDT, RSCALE>;
  auto kern = gdn_multi_kernel<RES, RSCALE, QDT>;
  const size_t smem = (size_t)L::kBytes;
  static thread_local bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return CARRY_GDN_ERR_NO_DEVICE;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      cudaGetLastError();
      return CARRY_GDN_ERR_NO_DEVICE;
    }
    configured[dev] = true;
  }
  return launch_dependent(kern, dim3((unsigned)((long long)p.B * p.HV)), kThreads, smem, stream, p, x);
}

template <int RES, int RSCALE>
int launch_multi_dtype(const KParams& p, const MultiExtra& x, cudaStream_t stream) {
  if (p.qkv_dtype == CARRY_F32) return launch_multi_variant<RES, RSCALE, CARRY_F32>(p, x, stream);
  if (p.qkv_dtype == CARRY_BF16) return launch_multi_variant<RES, RSCALE, CARRY_BF16>(p, x, stream);
  return launch_multi_variant<RES, RSCALE, CARRY_F16>(p, x, stream);
}

}  // namespace

// p describes token 0 of every request exactly as for the single-token call; the caller has checked
// tile128_eligible(p) and that the per-token strides keep every row 16-byte aligned.
int launch_multi(const KParams& p_in, int T, long long stride_mixed_t, long long stride_a_t, long long stride_b_t,
                 cudaStream_t stream) {
  KParams p = p_in;
  fill_shifts(p);
  const int sms = sm_count();
  if (sms == 0) return CARRY_GDN_ERR_NO_DEVICE;
  MultiExtra x = {T, stride_mixed_t, stride_a_t, stride_b_t, 2 * sms};
  const bool i4 = p.res_fmt == CARRY_RES_INT4, pv = p.rscale_mode == CARRY_SCALE_PER_V;
  if (i4) return pv ? launch_multi_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_V>(p, x, stream)
                    : launch_multi_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_HEAD>(p, x, stream);
  return pv ? launch_multi_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_V>(p, x, stream)
            : launch_multi_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_HEAD>(p, x, stream);
}

}  // namespace carry
