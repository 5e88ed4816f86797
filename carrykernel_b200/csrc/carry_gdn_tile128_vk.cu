// Streaming kernel of the serving path: slot layout [V][K], K = V = 128, int8 state, int8 or packed int4 residual with either
// scale mode, every activation type.  (carry_gdn_tile128.cuh has the helpers and says how the arithmetic is ordered.)
//
// A persistent CTA of 8 warps takes one tile after the other, two CTAs per SM: tiles blockIdx.x, + gridDim.x, ...  Tiles come
// in by bulk copies through a ring of stages that stay ahead of the one in hand, results leave from registers.  One meeting
// of the warps per tile (for the residual scale of the head; with scales per V row it only hands the stage on), after which
// one warp requests the tile that will use the stage next and two prepare the dot products (DotBuf) of the tile after the next.
//
// What bounds it: the arithmetic pipes.  The FMA pipe's and the ALU's busy cycles add up to 86 % of all cycles (92 % in the
// kernel before this one) and do not overlap: packed multiply-adds and byte permutes, logic or maxima next to one another
// take the sum of their times, about 0.6 cycles per register operand read.  So a step pays by what it takes off either: the
// dot products on the tensor cores, stores and floors without branches.  Per warp and tile 1009 instructions, 1155 before (one
// CTA of two groups of 8 warps per SM, sums over 8 lanes, groups taking tiles as they go).  Measured, int4 residual with one
// scale per head, 64 / 512 requests x 32 heads: 28.8 / 213 us per launch, 30.8 / 220 before; 1 request 4.9, 5.3 before; int8
// with scales per V row, 40 requests 22.2, 24.1 before.  Not kept: 16 warps per tile of one row per lane in 64 registers
// (851 us for 24 layers of 64 requests, against 691); counting barriers in shared memory in the meeting's place with the next
// tile's dot products behind the arrival (692, and 302 instead of 266 for int8: the polls and moves eat what the wait
// gives); dot products prepared an element per thread by all warps (729) or by one warp alone (730).
#include "carry_gdn_tile128.cuh"

namespace carry {
namespace {

constexpr int kSlotThreads = 256, kSlotWarps = kSlotThreads / 32;

template <int RES, int RSCALE, int QDT>
struct SlotShape {
  using L = StageLayout<RES, LAYOUT_VK, QDT, RSCALE>;
  // Shared memory of two CTAs per SM: at least 3 stages (prepare() waits for a tile that was requested a meeting ago or more),
  // facts and addresses of the CTA's first 64 tiles, worked out when it starts, or of as many as there is room for, and
  // a fourth stage if that fits.
  static constexpr int kBudget = 115712, kFixed = 2 * (int)sizeof(DotBuf) + 192, kEntry = (int)(sizeof(TileMeta) + sizeof(TileDesc));
  static constexpr int kRoom = (kBudget - kFixed - 3 * L::kBytes) / kEntry - 4;
  static constexpr int kCache = kRoom > 64 ? 64 : kRoom / 8 * 8;
  static constexpr int kStatic = kFixed + (kCache + 4) * kEntry;
  static constexpr int kStages = (kBudget - kStatic) / L::kBytes > 3 ? 4 : 3;
  static_assert(kCache >= 32, "room for the first tiles' facts");
};

template <int RES, int RSCALE, int QDT>
__global__ void __launch_bounds__(kSlotThreads, 2) gdn_slot128_kernel(const __grid_constant__ KParams p) {
  using Shape = SlotShape<RES, RSCALE, QDT>;
  using L = typename Shape::L;
  constexpr int S = Shape::kStages, kCache = Shape::kCache;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ TileMeta meta_cache[kCache + 4];    // this CTA's first tiles; spare entries for later ones, by number mod 4
  __shared__ TileDesc desc_cache[kCache + 4];    // their addresses
  __shared__ DotBuf dot_buf[2];                      // of the tile in hand and the next one, by parity
  __shared__ __align__(8) uint64_t full_bar[S];
  __shared__ uint32_t head_max[4];                   // largest new residual of a tile, as bits, by tile count mod 4
  __shared__ int poison_flag;
  static_assert(sizeof(meta_cache) + sizeof(desc_cache) + sizeof(dot_buf) + sizeof(full_bar) + sizeof(head_max) + 64 <= Shape::kStatic,
                "static shared memory exceeds what the stage ring was sized for");

  const int tid = threadIdx.x, gw = tid >> 5, lane = tid & 31, gtid = tid;
  const int total = p.B * p.HV;
  const int my_tiles = (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int cached = my_tiles < kCache ? my_tiles : kCache;
  volatile int* poison = &poison_flag;

  depend_release();
  if (tid == kSlotThreads - 1) {
    poison_flag = 0;
    head_max[0] = head_max[1] = head_max[2] = head_max[3] = 0u;
    for (int s = 0; s < S; ++s) mbar_init(&full_bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Set-up of the CTA's first tiles (up to the cache's size) by all threads, 32, 8 or 4 lanes per tile -- as many as the tile
  // count leaves room for in one pass -- in two halves around the dependency wait:
  //   before it, while the kernel ahead in the stream finishes: load the tiles' inputs past the L1, work
  //     out slot id, gates and norms from whatever they hold, keep both in registers; hint the L2 at the
  //     state of the first tiles and at the v rows.  Nothing here writes memory or hands a value on.
  //   after it: the same loads again, now ordered after every write of that kernel.  Equal words mean the
  //     figures worked out beforehand are the ones this launch must use: the first tile is
  //     requested at once, from the addresses already in registers (the rest of the ring only after all
  //     threads have met, so that it is not queued behind them), and the figures go to the
  //     cache.  A warp that sees a difference runs the whole routine again.
  // Right after a kernel that left tens of MB of results in the L2 a first touch of memory takes some 2 us
  // and the routine's arithmetic, fetched cold, another microsecond: this way both pass while the CTA would
  // otherwise sit in the wait, and what is left behind it is one trip to the L2.
  auto setup = [&](auto lanes_per_tile) {
    constexpr int LPT = decltype(lanes_per_tile)::value;
    constexpr int qes = (QDT == CARRY_F32) ? 4 : 2;
    const int num = tid / LPT, sub = tid % LPT;          // the tile these lanes prepare
    const bool valid = num < cached;
    const bool busy = gw * (32 / LPT) < cached;          // warps without a tile to prepare stay out of the way
    const int tile = (int)blockIdx.x + (valid ? num : 0) * (int)gridDim.x;
    const int entry = valid ? num : 0;
    TileMeta m;
    MetaRaw<QDT, LPT> before;
    unsigned long long a[8];
    bool bad = false;
    int hv = 0, h = 0;
    if (busy) {
      split_tile(p, tile, m.n, hv, h);
      m.hv = hv;
      meta_load<QDT, LPT>(p, m.n, hv, h, sub, 0, 0, 0, before);
      m.slot = before.slot;
      bad = meta_addresses<RES, RSCALE, QDT>(p, m, hv, h, a);
      if (sub == 0 && valid && m.slot > 0) {
        l2_prefetch_line(reinterpret_cast<const void*>(a[D_V]));
        l2_prefetch_line(reinterpret_cast<const void*>(a[D_V] + kT * qes - 16));
        if (num < 2) {
          l2_prefetch_bulk(reinterpret_cast<const void*>(a[D_CODES]), kT * kT);
          l2_prefetch_bulk(reinterpret_cast<const void*>(a[D_RESID]), L::kResidBytes);
          l2_prefetch_bulk(reinterpret_cast<const void*>(a[D_SSCALE]), 512);
        }
      }
      meta_math<QDT, LPT>(p, before, m);
    }
    // nothing before this line hands on what it read from global memory, or writes it; everything after it
    // sees the results of the kernels that precede this one in the stream
    __syncthreads();
    depend_wait();
    if (busy) {
      const bool same = meta_unchanged<QDT, LPT>(p, m.n, hv, h, sub, before);
      test_note_changed(p.status, same);
      if (__all_sync(0xffffffffu, same && !test_inputs_changed(tile))) {
        if (num == 0 && sub == 0) {
          if (m.slot <= 0) mbar_arrive(&full_bar[0]);
          else issue_copies<LAYOUT_VK, RES, RSCALE, QDT>(p, smem, &full_bar[0], a, tile);
        }
        if (valid) meta_put(p, m, a, bad, sub, &meta_cache[entry], &desc_cache[entry]);
        if constexpr (LPT == 32) {                       // lane = quad: straight from the registers
          if (valid && num < 2 && m.slot > 0) {
            RawQuad<QDT> r;
#pragma unroll
            for (int i = 0; i < MetaRaw<QDT, LPT>::kWords; ++i) { r.k[i] = before.kw[i]; r.q[i] = before.qw[i]; }
            prepare_quad<QDT>(r, lane, m, dot_buf[num]);
          }
        }
      } else {
        tile_meta<RES, RSCALE, QDT, LPT>(p, tile, sub, valid, &meta_cache[entry], &desc_cache[entry]);
        __syncwarp();
        if (num == 0 && sub == 0)
          issue_cached<LAYOUT_VK, RES, RSCALE, QDT>(p, smem, &full_bar[0], &desc_cache[0], meta_cache[0].slot, tile);
        if constexpr (LPT == 32) {
          if (valid && num < 2 && meta_cache[num].slot > 0)
            prepare_dots<QDT>(reinterpret_cast<const uint8_t*>(desc_cache[num].a[D_K]), reinterpret_cast<const uint8_t*>(desc_cache[num].a[D_Q]),
                              lane, &meta_cache[num], &dot_buf[num]);
        }
      }
    }
  };
  static_assert(kSlotThreads / 4 >= kCache, "at four lanes per tile one pass covers the whole cache");
  const bool wide = cached <= kSlotWarps;
  if (wide) setup(LanesPerTile<32>{});
  else if (cached <= kSlotThreads / 8) setup(LanesPerTile<8>{});
  else setup(LanesPerTile<4>{});
  __syncthreads();

  constexpr float rqmax = (RES == CARRY_RES_INT4) ? 7.0f : 127.0f;
  constexpr float rrqmax = 1.0f / rqmax;             // rounded to nearest, like the host's p.inv_qmax
  const float rqmax_state = p.inv_qmax;
  auto load_tile = [&](int num, int stage) {         // one thread requests tile `num`
    uint8_t* to = smem + (size_t)stage * L::kBytes;
    const int tile = (int)blockIdx.x + num * (int)gridDim.x;
    if (num < kCache) {
      issue_cached<LAYOUT_VK, RES, RSCALE, QDT>(p, to, &full_bar[stage], &desc_cache[num], meta_cache[num].slot, tile);
    } else {
      int tn, thv, th;
      split_tile(p, tile, tn, thv, th);
      issue_tile<LAYOUT_VK, RES, RSCALE, QDT>(p, to, &full_bar[stage], tn, thv, th, p.slot_idx[(long long)tn * p.stride_idx]);
    }
  };
  // Digits and scaled k of tile `num`, k by warp `who`, q by the one half the CTA on.  (A quad of each per lane of one warp is
  // 75 instructions for the others to wait for at the meeting; an element per thread of all warps is 40 for each.)
  auto prepare = [&](int num, int stage, uint32_t parity, int who) {
    if ((gw ^ who) & (kSlotWarps / 2 - 1)) return;
    const TileMeta& m = meta_cache[num < kCache ? num : kCache + (num & 3)];
    if (m.slot <= 0 || !mbar_wait(&full_bar[stage], parity, poison, p.status)) return;
    const uint8_t* st = smem + (size_t)stage * L::kBytes;
    if (gw == who) prepare_vector<QDT, true>(st + L::kK, lane, m, dot_buf[num & 1]);
    else prepare_vector<QDT, false>(st + L::kQ, lane, m, dot_buf[num & 1]);
  };
  if (lane == 0 && gw >= 1 && gw < S && gw < my_tiles) load_tile(gw, gw);
  __syncwarp();
  if (!wide) {                                       // more than 8 tiles: from the stage
    prepare(0, 0, 0u, 0);
    __syncthreads();
    prepare(1, 1, 0u, 1);                               // published by the first tile's meeting
  }

  const SlotLane at = slot_lane(gw, lane);
  int stage = 0;
  uint32_t parity = 0u;
#pragma unroll 1
  for (int it = 0; it < my_tiles; ++it) {
    const int tile = (int)blockIdx.x + it * (int)gridDim.x;
    uint8_t* sb = smem + (size_t)stage * L::kBytes;
    const int entry = it < kCache ? it : kCache + (it & 3);
    const TileMeta* tm = &meta_cache[entry];
    const uint4 tm0 = lds_v4(tm);
    const int slot = (int)tm0.z;
    // A stage's next tile is requested after its last one's meeting, and the barrier of the tile after that is not looked at
    // before: only a wait that ran out could mistake a phase, and then the CTA is poisoned.
    const bool landed = mbar_try_wait(&full_bar[stage], parity);
    bool healthy = !*poison;
    if (!landed && healthy) {
      mbar_wait_slow(&full_bar[stage], parity, poison, p.status);
      healthy = !*poison;
    }
    auto claim = [&]() {                             // after the meeting: the stage goes on
      if (gw == (it & (kSlotWarps - 1)) && lane == 0) {
        head_max[(it + 2) & 3] = 0u;                 // last read two meetings ago
        if (it + S < my_tiles && !*poison) load_tile(it + S, stage);
      }
    };
    // where results go: read from the tile's cached addresses right before each use, not held in registers
    auto dst_of = [&](int which) -> unsigned long long {
      unsigned long long v;
      asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(smem_u32(&desc_cache[entry].a[which])));
      return v;
    };
    uint8_t* out_to = reinterpret_cast<uint8_t*>(p.out) + (long long)tile * kT * (p.o_dtype == CARRY_F32 ? 4 : 2);
    if (slot <= 0 || !healthy) {
      if (slot <= 0 && tid < kT) store_from_float(p.out, (long long)tile * kT + tid, p.o_dtype, 0.f);
      __syncthreads();
    } else {
      const uint4 tm1 = lds_v4(reinterpret_cast<const uint8_t*>(tm) + 16), tm2 = lds_v4(reinterpret_cast<const uint8_t*>(tm) + 32);
      const float alpha = __uint_as_float(tm0.w), beta = __uint_as_float(tm1.x), k_mul = __uint_as_float(tm1.y),
                  q_mul = __uint_as_float(tm1.z), kq = __uint_as_float(tm1.w);
      const bool dot_fixed = __uint_as_float(tm2.x) != 0.0f;
      const float dot_mul = __uint_as_float((lane & 2) ? tm2.w : tm2.z);
      const float* sscale = reinterpret_cast<const float*>(sb + L::kSScale);
      const float* rscale = reinterpret_cast<const float*>(sb + L::kRScale);
      const float es_head = (RSCALE == CARRY_SCALE_PER_HEAD) ? rscale[tile & 3] : 0.f;   // HV is a multiple of 4 then
      const float2 alpha2 = splat(alpha);
      const float2 magic2 = splat(kMagicRound), nmagic2 = splat(-kMagicRound);
#define CARRY_SLOT_DOTS dot_buf[it & 1]
#define CARRY_SLOT_VEC_Q (sb + L::kQ)
#define CARRY_SLOT_VEC_K (sb + L::kK)
#define CARRY_SLOT_VEC_V (sb + L::kV)
#define CARRY_SLOT_OUT(on, idx, value) store_from_float_if(on, out_to, (idx), p.o_dtype, (value))
#define CARRY_SLOT_PUT_SSCALE(on, row_, bits_) stg_b32_if(on, dst_of(D_SSCALE) + (row_) * 4, (bits_))
#define CARRY_SLOT_CODES_TO dst_of(D_CODES)
#define CARRY_SLOT_RESID_TO dst_of(D_RESID)
#define CARRY_SLOT_PUT16(base, offset, v) stg_v4((base) + (offset), (v))
#define CARRY_SLOT_PUT8(base, offset, v) stg_v2_at<0>((base) + (offset), (v))
#define CARRY_SLOT_HEAD_MAX head_max[it & 3]
#define CARRY_SLOT_MEET(statement)                             \
  statement;                      \
  __syncthreads()
#define CARRY_SLOT_PUT_RSCALE_V(on, row_, bits_) stg_b32_if(on, dst_of(D_RSCALE) + (row_) * 4, (bits_))
#define CARRY_SLOT_PUT_RSCALE_HEAD(bits_) stg_b32(dst_of(D_RSCALE), (bits_))
#include "carry_gdn_slot_tile.inc"
    }
    claim();
    const bool wrap = stage + 1 == S;
    // tile it + 2, whose buffer was this tile's, two stages on; and the facts of the one after it, if they are not cached
    if (it + 2 < my_tiles) {
      const bool over = stage + 2 >= S;
      prepare(it + 2, over ? stage + 2 - S : stage + 2, over ? parity ^ 1u : parity, (it + 1) & (kSlotWarps - 1));
      const int num = it + 3;
      if (num >= kCache && num < my_tiles && gw == ((it + kSlotWarps / 2) & (kSlotWarps - 1)))
        tile_meta<RES, RSCALE, QDT, 32>(p, (int)blockIdx.x + num * (int)gridDim.x, lane, true, &meta_cache[kCache + (num & 3)],
                                        &desc_cache[kCache + (num & 3)]);
    }
    stage = wrap ? 0 : stage + 1;
    parity ^= wrap ? 1u : 0u;
  }
  __syncthreads();
  // A CTA whose wait ran out has stopped requesting tiles, but copies it requested earlier may still be on
  // their way into its shared memory: give them a bounded while to land before the CTA leaves the SM.
  if (*poison) {
#pragma unroll 1
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
}

template <int RES, int RSCALE, int QDT>
int launch_slot_variant(const KParams& p, cudaStream_t stream, int sms) {
  using Shape = SlotShape<RES, RSCALE, QDT>;
  auto kern = gdn_slot128_kernel<RES, RSCALE, QDT>;
  const size_t smem = (size_t)Shape::L::kBytes * Shape::kStages;
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
  const long long tiles = (long long)p.B * p.HV;
  return launch_dependent(kern, dim3((unsigned)(tiles < 2LL * sms ? tiles : 2LL * sms)), kSlotThreads, smem, stream, p);
}

template <int RES, int RSCALE>
int launch_slot_dtype(const KParams& p, cudaStream_t stream, int sms) {
  if (p.qkv_dtype == CARRY_F32) return launch_slot_variant<RES, RSCALE, CARRY_F32>(p, stream, sms);
  if (p.qkv_dtype == CARRY_BF16) return launch_slot_variant<RES, RSCALE, CARRY_BF16>(p, stream, sms);
  return launch_slot_variant<RES, RSCALE, CARRY_F16>(p, stream, sms);
}

}  // namespace

int launch_tile128_vk(const KParams& p, cudaStream_t stream, int sms) {
  const bool i4 = p.res_fmt == CARRY_RES_INT4, pv = p.rscale_mode == CARRY_SCALE_PER_V;
  if (i4) return pv ? launch_slot_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_V>(p, stream, sms)
                    : launch_slot_dtype<CARRY_RES_INT4, CARRY_SCALE_PER_HEAD>(p, stream, sms);
  return pv ? launch_slot_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_V>(p, stream, sms)
            : launch_slot_dtype<CARRY_RES_INT8, CARRY_SCALE_PER_HEAD>(p, stream, sms);
}

}  // namespace carry

#ifdef CARRY_TEST_WAIT_EXPIRY
// Test-only (twin library): a kernel that lets the launch behind it in the stream start at once, idles for
// `delay_ns` (at most 0.2 ms), and only then copies `bytes` (a multiple of 16) from src to dst -- a
// predecessor that is still writing the streaming kernel's inputs while that kernel takes its first look
// at them ahead of its dependency wait.
namespace carry {
namespace {
__global__ void late_writer_kernel(uint4* dst, const uint4* src, long long n16, unsigned delay_ns) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (unsigned waited = 0; waited < delay_ns; waited += 1000) __nanosleep(1000);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}
}  // namespace
}  // namespace carry
extern "C" int carry_gdn_test_late_writer(void* dst, const void* src, long long bytes, unsigned delay_ns, void* stream) {
  if (bytes < 0 || bytes % 16 != 0 || (reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) % 16 != 0)
    return CARRY_GDN_ERR_SHAPE;
  if (delay_ns > 200000u) delay_ns = 200000u;
  carry::late_writer_kernel<<<8, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<uint4*>(dst), static_cast<const uint4*>(src), bytes / 16, delay_ns);
  return cudaGetLastError() == cudaSuccess ? CARRY_GDN_OK : CARRY_GDN_ERR_LAUNCH;
}
#endif
