// Fused activation quantizer + LoRA-down for sm_100a: one pass over x.
//
//   act, ascales = nvfp4( x / smooth )        bit-exact with the reference oracle
//   lora_act     = x @ lora_down              fp32, tcgen05 dense 16-bit MMA
//
// Replaces the reference's Triton kernel
// (triton_kernels/quantize_w4a4_act_fuse_lora/kernel.py:115-286); results
// follow baseline/kernels/quantize_w4a4_act_fuse_lora/ref.py:19-50.
//
// Decomposition.  A cluster of KS (1 to 16) CTAs owns one tile of 64 rows; CTA k
// owns a contiguous range of 64-column slabs of K.  Per slab one producer warp
// TMA-loads the x tile (64 x 64, 128-byte swizzle) with the slab's 64 entries of
// the smoothing table (one bulk copy) into a stage of the x ring, a
// second one the matching lora_down slab (64 x R) into a ring of its own.
// Two kinds of consumers read an x stage: two MMA-issuing warps (even and odd
// slabs) accumulate x_tile @ lora_down_slab into [64 x R] fp32 accumulators in
// tensor memory, one each, and sixteen quantize warps turn the tile into codes
// and scales.  x is read from HBM exactly once.  With KS > 1 the partial
// accumulators are summed in a fixed order, brought together by the copy engine (two ranks: halves, into the partner's
// shared memory; more: every rank's share of the tile): no atomics, no zero-fill, no scratch in global
// memory.  Large inputs run with KS = 2; larger clusters are for inputs of
// a few hundred to two thousand rows, where pairs would leave most SMs idle (256 x 10240:
// 36.0 -> 5.8 us, rank 32), and are taken only if all of them are resident at once.
// (64-row tiles with pairs, not 128-row tiles with quads: a B200 keeps
// at most 33 four-CTA clusters of this size resident, one short of the 34 row
// tiles of a 4352-row activation, while 68 pairs fit in one wave.  128-row tiles
// whose K ranks meet through global memory were measured too: what they save in
// lora_down traffic and MMA count, the 9 MB of partial sums that all CTAs write
// at the same moment costs again.)
//
// Lane mapping.  The four lanes of a quad hold one row's four 16-column groups
// of the slab, so their 8-byte code stores fill one 32-byte sector and their
// scale bytes are adjacent in the atom layout; with a lane per row and a warp
// per group the same stores touched 32 sectors each and cost 4 us more.
//
// Arithmetic: one multiplication per element in the place of each division, exact in every decision; see
// quantize_math.cuh.
#include "nvfp4_math.cuh"
#include "quantize_math.cuh"
#include "sm100.cuh"
#include "svdq_internal.h"

#include <type_traits>

namespace svdq {
namespace qf {

constexpr int TILE_M = 64;
constexpr int SLAB_K = 64;                 // columns per ring stage (128 bytes of 16-bit x)
constexpr int X_BYTES = TILE_M * 128;      // 8 KB
#ifndef SVDQ_QUANT_GROUPS
#define SVDQ_QUANT_GROUPS 4
#endif
constexpr int QUANT_GROUPS = SVDQ_QUANT_GROUPS;   // groups of 4 warps take slabs round-robin
constexpr int QUANT_WARPS = 4 * QUANT_GROUPS;
constexpr int AUX_WARPS = 4;                // x producer, MMA issuer (even slabs), lora_down producer, MMA issuer (odd slabs); with two K ranks they exchange the LoRA sums
constexpr int NUM_THREADS = (AUX_WARPS + QUANT_WARPS) * 32;
constexpr int TB_BYTES = SLAB_K * 4;       // smoothing-table entries of a slab's columns
constexpr int kMaxKSplit = 16;             // CTAs of a cluster

// PUSH: clusters of more than two CTAs (see the exchange of LoRA sums below)
template <int RP, bool PUSH>
struct Cfg {
  // Two rings.  An x stage holds a 64 x 64 tile of x (8 KB) and, in an area of their own, the slab's 64 table
  // entries; it is read by the MMA and by one quantize group and released by both.  A lora_down slab (64 x RP, 16 KB at
  // rank 128) would make that stage three times as large and the ring a third as deep, and the stage would stay
  // held for the slab's four MMAs; in a ring of its own, which only the MMA reads, a few stages are enough
  // (the slabs come out of L2) and the x ring gets the rest of the shared memory.
  static constexpr int W_BYTES = SLAB_K * RP * 2;                 // lora_down slab
  // Six lora_down stages: a slab comes out of L2 in about 1.7 us while x streams in beside it, and slabs pass at
  // 0.3 us (2 / 4 / 6 / 8 stages, 4352 rows: K = 3840 22.0 / 16.2 / 14.9 / 15.6 us, K = 10240 42.5 / 30.3 / 29.0 / 29.5);
  // at rank 256 three are what fits.
  static constexpr int W_STAGES = RP > 128 ? 3 : 6;
  // MMA-issuing warps.  Two take the slabs by turns; then both rings must be even, so that an issuer meets only slabs
  // of its own in a stage: one that went on to slab i could otherwise look at the stage while slab i - W_STAGES,
  // the other issuer's, is still on its way into it, and a one-bit parity would tell it that slab i is there.
  static constexpr int ISSUERS = W_STAGES % 2 == 0 ? 2 : 1;
  static constexpr int W_RING_BYTES = W_STAGES * W_BYTES;
  // Receive buffer for partial sums: of the peer for this CTA's 32 rows (two K ranks), of the other ranks for this CTA's
  // share of the tile (PUSH; shares are rounded up to whole float4s).  With room for this rank's own part too the x ring lost a
  // third of its stages at rank 128 and the lora_down ring one of three above it: rank 256, fp16, 512 x 10240 14.2 us instead
  // of 11.9, 1003 x 3840 10.4 / 9.6, 2000 x 15360 43.3 / 34.0; rank 128, 2000 x 10240 16.4 / 16.1, elsewhere the same.
  static constexpr int RECV_BYTES = PUSH ? TILE_M * RP * 4 / kMaxKSplit * (kMaxKSplit - 1) + kMaxKSplit * 16 : (TILE_M / 2) * RP * 4;
  static constexpr int STAGES_RAW = (232448 - 1024 - 512 - RECV_BYTES - W_RING_BYTES) / (X_BYTES + TB_BYTES);
  // A multiple of the group count: a group then always meets the same stages, and the slab it waits
  // for is the direct successor (in that stage) of one it consumed itself.  A one-bit phase parity
  // cannot tell "one revolution behind" from "one ahead"; this rule makes the second impossible.
  static constexpr int STAGES = ((STAGES_RAW > 16 ? 16 : STAGES_RAW) / QUANT_GROUPS) * QUANT_GROUPS;
  static constexpr int RING_BYTES = STAGES * X_BYTES;
  static constexpr int TB_OFF = RING_BYTES + W_RING_BYTES;
  static constexpr int BARS_OFF = TB_OFF + STAGES * TB_BYTES;
  static constexpr int SMEM_BYTES = 1024 + BARS_OFF + 512 + RECV_BYTES;          // rings, table entries, barriers, receive buffer
  static constexpr int TMEM_COLS = ISSUERS * RP;                  // an accumulator per issuer; a power of two >= 64
  static constexpr int EPI_COLS = RP / 4 < 32 ? 32 : RP / 4;      // accumulator columns per epilogue warp
  static_assert(!PUSH || TILE_M * RP * 4 <= RING_BYTES, "the sums must fit in the x ring");
  static_assert(STAGES >= QUANT_GROUPS && STAGES % QUANT_GROUPS == 0 && (ISSUERS == 1 || STAGES % 2 == 0), "ring depth");
  static_assert((2 * STAGES + 2 * W_STAGES + 3) * 8 + 64 <= 512, "barrier block");
  static_assert(PUSH || 2 * RECV_BYTES <= W_RING_BYTES, "the exchange stages both halves of the accumulator in the lora_down ring");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};
template <int RP> constexpr bool kPushKeepsTheRings =
    Cfg<RP, true>::STAGES >= Cfg<RP, false>::STAGES && Cfg<RP, true>::W_STAGES >= Cfg<RP, false>::W_STAGES;
static_assert(kPushKeepsTheRings<64> && kPushKeepsTheRings<128> && kPushKeepsTheRings<256>, "the receive buffer takes stages from the rings");

struct Params {
  const float* table;     // smoothing table (layout in quantize_math.cuh), or null (no smoothing)
  uint8_t* act;           // [M_pad, K/2]
  uint8_t* scales;        // [K/16, M_pad]
  uint8_t* scales_swz;    // atom order or null
  float* lora;            // [M_pad, R]
  void* lora16;           // 16-bit form of lora (fp16 [M_pad, R] or bf16 [2, M_pad, R]) or null
  int M, K, R, M_pad;
};

// float4 slot of (row, c4) in the partial-accumulator buffer; the XOR spreads the
// rows a warp writes at once over all bank groups.
__device__ __forceinline__ uint32_t partial_slot(uint32_t row, uint32_t c4, uint32_t rp4) {
  return row * rp4 + (c4 ^ (row & 7u));
}

using qmath::unpack_group;

template <typename T, int RP, bool PUSH>
__global__ void __launch_bounds__(NUM_THREADS, 1)
quantize_fused_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Params p) {
  using C = Cfg<RP, PUSH>;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;

  extern __shared__ uint8_t smem_raw[];
  // 1 KB alignment by pointer arithmetic (not an integer round trip) so that the compiler keeps
  // the shared address space and emits shared-memory loads and stores
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* wring = smem + C::RING_BYTES;       // lora_down slabs
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BARS_OFF);
  uint64_t* full = bars;                       // [STAGES]    x stage filled
  uint64_t* empty = bars + C::STAGES;          // [STAGES]    x stage consumed (MMA + one quantize group)
  uint64_t* wfull = bars + 2 * C::STAGES;      // [W_STAGES]  lora_down slab landed
  uint64_t* wempty = wfull + C::W_STAGES;      // [W_STAGES]  lora_down slab consumed (MMA)
  uint64_t* acc_done = wempty + C::W_STAGES;   // MMA -> epilogue
  uint64_t* recv_bar = acc_done + 1;           // the other ranks' partial sums have landed in `recv`
  uint64_t* ack_bar = recv_bar + 1;            // two K ranks: the peer has received what this CTA sent
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ack_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* lora_unfit = tmem_slot + 2;        // bf16 form: some LoRA value this CTA wrote does not fit fp16 (one rank: a bit per 32 rows)
  float4* recv = reinterpret_cast<float4*>(smem + C::BARS_OFF + 512);        // [32 rows][RP / 4], slots as partial_slot; PUSH: [following rank][share]
  const WaitCtx ctx{abort_flag};

  // warp index through a shuffle: provably warp-uniform, so the role branches are convergent code
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  auto uwait = [&](uint64_t* bar, uint32_t parity, unsigned int code, unsigned int tag) -> bool {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, ctx, code, tag)) != 0;
  };
  const uint32_t ks = gridDim.y;               // cluster = (1, KS, 1): blockIdx.y is the rank along K
  const uint32_t krank = blockIdx.y;
  const int m0 = blockIdx.x * TILE_M;
  const bool has_lora = p.R > 0;
  const bool has_table = p.table != nullptr;

  // slabs owned by this CTA
  const int n_slabs = p.K / SLAB_K;
  const int base = n_slabs / static_cast<int>(ks), rem = n_slabs % static_cast<int>(ks);
  const int slab_begin = static_cast<int>(krank) * base + (static_cast<int>(krank) < rem ? static_cast<int>(krank) : rem);
  const int my_slabs = base + (static_cast<int>(krank) < rem ? 1 : 0);
  const int k_begin = slab_begin * SLAB_K;

  // PUSH: the tile's sums as float4s, row by row, the ranks' columns rounded up to whole chunks of 32 and, inside a chunk of
  // eight float4s, XORed by the row (for the banks).  Rank k sums numbers [k T / KS, (k + 1) T / KS) of the T.
  const uint32_t row4 = (static_cast<uint32_t>(p.R) + 31u) / 32u * 8u, tile4 = TILE_M * row4;
  auto share_begin = [&](uint32_t rank) -> uint32_t { return rank * tile4 / ks; };
  const uint32_t item_lo = share_begin(krank), item_hi = share_begin(krank + 1), share = (tile4 + ks - 1) / ks;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *lora_unfit = 0u;
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1 + QUANT_WARPS / QUANT_GROUPS); }
    for (int s = 0; s < C::W_STAGES; ++s) { mbar_init(&wfull[s], 1); mbar_init(&wempty[s], 1); }
    mbar_init(acc_done, C::ISSUERS == 2 && my_slabs > 1 ? 2 : 1);     // one arrival per MMA issuer that has slabs
    mbar_init(recv_bar, 1);                    // armed here with all the bytes that will come
    mbar_init(ack_bar, 1);
    if (PUSH && has_lora) mbar_arrive_expect_tx(recv_bar, (ks - 1) * 16u * (item_hi - item_lo));
    else if (!PUSH && ks == 2 && has_lora) mbar_arrive_expect_tx(recv_bar, C::RECV_BYTES);
    fence_barrier_init();
    tma_prefetch_desc(&tmX);
    if (has_lora) tma_prefetch_desc(&tmW);
  }
  __syncthreads();
  // Two K ranks hand their partial sums to each other through the copy engine, counted on the partner's
  // barrier, so that barrier must exist (and be armed) before either touches it: whoever touches it waits for this.
  if (!PUSH && ks == 2 && has_lora) cluster_arrive_relaxed();       // (fence_barrier_init is what releases the barriers)
  // Tensor memory: the issuers wait for it (loads are under way by then), the epilogue reads the address once the sums are complete.
  if (has_lora && (warp == 1 || warp == 3)) {
    if (warp == 1) {
      tmem_alloc(tmem_slot, C::TMEM_COLS);
      tmem_relinquish();
    }
    tc_fence_before_sync();
    asm volatile("bar.sync 4, 64;" ::: "memory");
    tc_fence_after_sync();
  }
  auto tmem_base = [&]() -> uint32_t { return __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0); };   // warp-uniform, like the warp index
  // set-up done; what follows reads and writes global memory
  pdl_wait();
  if constexpr (PUSH) {
    if (has_lora) {
      // bf16: no value of the tile is known not to fit fp16; a rank that meets one says so after the cluster barrier begun here
      if (kBf16 && p.lora16 != nullptr && krank == 0 && warp == AUX_WARPS + QUANT_WARPS - 1) {
        if (lane < 2) lora16_flags(p.lora16, static_cast<size_t>(p.M_pad) * p.R)[m0 / 32 + lane] = 0u;
        __syncwarp();
        cluster_arrive();
      } else {
        cluster_arrive_relaxed();                              // (a releasing one took 0.4 us here)
      }
    }
  }

  // Out-of-range smooth anywhere in K (flag word behind the table) selects the IEEE divide by the factors.  Asked for where it is
  // out of the way of the first loads: as a condition of those it stood, 0.7 us, in front of everything.  So the first round of
  // the ring holds reciprocals in any case and a flagged launch reads that round's factors where they are, which makes it slower
  // than with factors in the ring throughout (4352 rows, x 3840 22.2 us instead of 20.2, x 10240 48 / 44.6, x 15360 69 / 66; with
  // every round's factors read from global memory 25.4 / 59 / 87).
  auto table_flagged = [&]() -> bool { return has_table && *reinterpret_cast<const volatile uint32_t*>(p.table + 2 * p.K) != 0u; };

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    const uint32_t stage_bytes = X_BYTES + (has_table ? TB_BYTES : 0);
    const float* table = p.table;              // reciprocals; a flagged launch (below): factors, from the second round of the ring on
    for (int i = 0; i < my_slabs; ++i) {
      const uint32_t s = i % C::STAGES, ph = (i / C::STAGES) & 1;
      if (!uwait(&empty[s], ph ^ 1, kDevWaitEmpty, i)) break;
      if (i == C::STAGES && table_flagged()) table += p.K;
      const int k0 = k_begin + i * SLAB_K;
      if (elect_one()) {
        mbar_arrive_expect_tx(&full[s], stage_bytes);
        tma_load_2d(smem + s * X_BYTES, &tmX, k0, m0, &full[s]);
        if (has_table) bulk_load_1d(smem + C::TB_OFF + s * TB_BYTES, table + k0, TB_BYTES, &full[s]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // ------------------------------ lora_down producer ------------------------------
    if (has_lora) {
      for (int i = 0; i < my_slabs; ++i) {
        const uint32_t s = i % C::W_STAGES, ph = (i / C::W_STAGES) & 1;
        if (!uwait(&wempty[s], ph ^ 1, kDevWaitEmpty, 0x50000 + i)) break;
        uint8_t* st = wring + s * C::W_BYTES;
        const int k0 = k_begin + i * SLAB_K;
        if (elect_one()) {
          mbar_arrive_expect_tx(&wfull[s], C::W_BYTES);
#pragma unroll
          for (int b = 0; b < RP / 64; ++b) tma_load_2d(st + b * (SLAB_K * 128), &tmW, b * 64, k0, &wfull[s]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1 || (warp == 3 && C::ISSUERS == 2)) {
    // ------------------------------ MMA issuers ------------------------------
    // Two warps, even and odd slabs, each into an accumulator of its own (added up in the epilogue, always in
    // the same order).  One thread's loop - two barrier waits, four MMAs, three commits - takes longer than the tensor
    // pipe has to do for a slab, which made a single issuer the slowest agent of the kernel: the x ring ran full
    // behind it and the epilogue started late.  Operands are constants added to warp-uniform values.
    constexpr uint64_t kDescA = smem_desc_base(0, 1024, kSwizzle128B);               // x tile, K-major
    constexpr uint64_t kDescB = smem_desc_base(SLAB_K * 128, 1024, kSwizzle128B);    // lora_down slab, R-major (its own ring)
    // As many columns as the rank needs of the RP that a slab holds (what the accumulator's others hold is never used): at rank
    // 32 half of the tensor core's time and of its reads of lora_down (when it came, 256 x 10240 6.03 -> 5.92 us, 4352 x 10240 28.4 -> 28.2).
    const uint32_t idesc = idesc_f16(kBf16, kBf16, TILE_M, (static_cast<uint32_t>(p.R) + 15u) & ~15u, false, true);
    const int issuer = warp >> 1;                                  // 0 or 1
    const uint32_t acc = (has_lora ? tmem_base() : 0u) + issuer * RP;
    const int last = C::ISSUERS == 1 ? my_slabs - 1 : ((my_slabs - 1 - issuer) & ~1) + issuer;   // this issuer's last slab (negative: none)
    const uint32_t x16 = smem_desc_addr(smem), w16 = smem_desc_addr(wring);
    uint32_t s = issuer, ph = 0, sw = issuer, phw = 0;
    for (int i = issuer; i < my_slabs; i += C::ISSUERS) {
      if (!uwait(&full[s], ph, kDevWaitFull, i)) break;
      if (i == 0) pdl_trigger();                 // the first loads have landed: see pdl_trigger
      if (has_lora && !uwait(&wfull[sw], phw, kDevWaitFull, 0x50000 + i)) break;
      tc_fence_after_sync();
      const uint64_t da = kDescA + (x16 + s * (X_BYTES / 16)), db = kDescB + (w16 + sw * (C::W_BYTES / 16));
      if (elect_one()) {
        if (has_lora) {
#pragma unroll
          for (int j = 0; j < SLAB_K / 16; ++j) mma_f16<1>(acc, da + j * 2, db + j * 128, idesc, j != 0 || i != issuer ? 1u : 0u);
          tc_commit(&empty[s]);
          tc_commit(&wempty[sw]);
          if (i == last) tc_commit(acc_done);
        } else {
          mbar_arrive(&empty[s]);
        }
      }
      __syncwarp();
      s += C::ISSUERS; if (s >= C::STAGES) { s -= C::STAGES; ph ^= 1; }
      sw += C::ISSUERS; if (sw >= C::W_STAGES) { sw -= C::W_STAGES; phw ^= 1; }
    }
  } else if (warp >= AUX_WARPS) {
    // ------------------------------ quantize warps ------------------------------
    // Group grp takes slabs grp, grp + QUANT_GROUPS, ...; its warp wq owns rows 16 wq .. 16 wq + 15 of the
    // tile.  Lane l works on 16-column group l % 4 of rows l / 4 and l / 4 + 8 of those, so the four
    // lanes of a quad hold one row's whole 64-column stretch of the slab: their 8-byte code stores
    // fill one 32-byte sector, and their scale bytes are adjacent in the atom layout.
    const int qw = warp - AUX_WARPS;
    const int grp = qw >> 2;
    const int wq = qw & 3;
    const int g = lane & 3;                   // 16-column group inside the slab
    const int row_base = 16 * wq + (lane >> 2);
    const int groups = p.K >> 4;
    uint8_t* const act_base = p.act + static_cast<size_t>(m0) * (p.K >> 1);
    const bool use_fdiv = table_flagged();     // while the first slab is on its way
    for (int i = grp; i < my_slabs; i += QUANT_GROUPS) {
      const uint32_t s = i % C::STAGES, ph = (i / C::STAGES) & 1;
      if (!mbar_wait(&full[s], ph, ctx, kDevWaitFull, 0x10000 + i)) break;
      const uint8_t* st = smem + s * X_BYTES;
      uint4 raw[2][2];
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const uint32_t row = row_base + 8 * rr;
        const uint8_t* xrow = st + row * 128;
        raw[rr][0] = *reinterpret_cast<const uint4*>(xrow + (((2 * g) ^ (row & 7)) << 4));
        raw[rr][1] = *reinterpret_cast<const uint4*>(xrow + (((2 * g + 1) ^ (row & 7)) << 4));
      }
      float2 f[2][8];
      if (has_table) {
        unpack_group<T, false>(raw[0][0], raw[0][1], f[0]);
        unpack_group<T, false>(raw[1][0], raw[1][1], f[1]);
        // this lane's 16 columns' reciprocals, or factors, landed with the slab
        const float4* landed = reinterpret_cast<const float4*>(smem + C::TB_OFF + s * TB_BYTES);
        if (!use_fdiv) qmath::smooth_multiply2(f[0], f[1], landed + g);
        else qmath::smooth_divide2(f[0], f[1], (i < C::STAGES ? reinterpret_cast<const float4*>(p.table + p.K + k_begin + i * SLAB_K) : landed) + g);
      } else {
        unpack_group<T, true>(raw[0][0], raw[0][1], f[0]);
        unpack_group<T, true>(raw[1][0], raw[1][1], f[1]);
      }
      // Hand the stage back once what was read from it is here: both groups' maxima depend on every value of the tile and
      // the table that this warp loads, and the arrival on them.  (Behind a fence, which also waits for the stores of the
      // slab before, 4352 x 15360 took 52.0 us instead of 48.9, 256 x 15360 9.5 instead of 8.7.)
      const float amax[2] = {qmath::group_amax(f[0]), qmath::group_amax(f[1])};
      __syncwarp();
      if (lane == 0) mbar_arrive_after(&empty[s], amax[0], amax[1]);

      const int k0 = k_begin + i * SLAB_K + g * 16;
      const int gi = k0 >> 4;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int row = row_base + 8 * rr;
        // one group after the other, each stored as soon as it is done: running both groups' scale chains
        // side by side and keeping their results in registers until the end measured 5-8 % slower
        uint32_t c_lo, c_hi, s_b;
        qmath::quantize_group_near(f[rr], amax[rr], c_lo, c_hi, s_b);
        *reinterpret_cast<uint2*>(act_base + static_cast<size_t>(row) * (p.K >> 1) + (k0 >> 1)) = make_uint2(c_lo, c_hi);
        p.scales[static_cast<size_t>(gi) * p.M_pad + m0 + row] = static_cast<uint8_t>(s_b);
        if (p.scales_swz != nullptr) p.scales_swz[sf_swizzled_offset(m0 + row, gi, groups)] = static_cast<uint8_t>(s_b);
      }
    }
    // PUSH: every quantize warp is done reading the x ring before it is used again below
    if constexpr (PUSH) asm volatile("bar.sync 2, %0;" ::"n"(QUANT_WARPS * 32) : "memory");
  }

  bool tmem_held = has_lora && warp == 1;
  auto free_tmem = [&]() {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base(), C::TMEM_COLS);
    tmem_held = false;
  };
  // 32 accumulator columns of this warp's lanes: the even slabs' accumulator plus, if there is more than one
  // slab, the odd slabs' (always in this order)
  auto acc_ld = [&](uint32_t taddr, uint32_t (&v)[32]) {
    tmem_ld_32x32(taddr, v);
    if (C::ISSUERS == 2 && my_slabs > 1) {
      uint32_t w[32];
      tmem_ld_32x32(taddr + RP, w);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(w[j])));
    } else {
      tmem_ld_wait();
    }
  };

  // ------------------------------ LoRA epilogue ------------------------------
  // The 64 accumulator rows live in lanes 0-15 of each 32-lane quarter of tensor memory:
  // row r is lane (r % 16) + 32 * (r / 16).
  if (!PUSH && has_lora && ks == 2) {
    // Two K ranks (the form for tall activations): CTA k owns rows [32 k, 32 k + 32) of the tile.  The four
    // auxiliary warps do the whole exchange while the quantize warps are still busy with the last slabs:
    // warp w reads rows 16 w .. 16 w + 15 of the accumulator (lanes 0-15 of its quarter of tensor
    // memory) into the lora_down ring, which is free once the last MMA has retired.  Rows of the partner
    // then go to the partner's receive buffer with one copy-engine transfer per warp, counted on the
    // partner's barrier (remote stores by the 16 lanes took 1.3 us of issue slots that the quantize warps
    // wanted); own rows wait there for the partner's.  Then all four warps add the two partial sums (two
    // terms: the order does not matter) and write the finished rows out, consecutive lanes taking
    // consecutive 16 bytes of a row.
    __syncwarp();
    cluster_wait();
    if (warp < AUX_WARPS) {
      constexpr uint32_t RP4 = RP / 4;
      constexpr uint32_t HALF_BYTES = 16u * RP * 4u;                 // one warp's 16 rows
      const bool ok = __all_sync(0xffffffffu, mbar_wait(acc_done, 0, ctx, kDevWaitAcc, 0)) != 0;
      tc_fence_after_sync();
      const bool mine = static_cast<uint32_t>(warp >> 1) == krank;
      const uint32_t row_local = 16u * (warp & 1) + (lane & 15);     // row within the owner's 32
      const uint32_t taddr = tmem_base() + (static_cast<uint32_t>(warp * 32) << 16);
      float4* send = reinterpret_cast<float4*>(wring);                // [32 rows][RP / 4], slots as partial_slot
      float4* own = reinterpret_cast<float4*>(wring + C::RECV_BYTES);
      float4* dst = mine ? own : send;
#pragma unroll 1
      for (int c0 = 0; c0 < RP; c0 += 32) {
        uint32_t v[32];
        acc_ld(taddr + c0, v);
        if (lane < 16) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            dst[partial_slot(row_local, (c0 >> 2) + j, RP4)] =
                make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
      }
      if (!mine) {
        fence_proxy_async_smem();                                     // the copy engine reads what the lanes wrote
        __syncwarp();
        if (lane == 0 && ok) {
          const uint32_t off = (warp & 1) * HALF_BYTES;
          bulk_copy_smem_to_cluster(map_to_cta(smem_u32(recv) + off, krank ^ 1u), smem_u32(send) + off, HALF_BYTES,
                                    map_to_cta(smem_u32(recv_bar), krank ^ 1u));
        }
      }
      tc_fence_before_sync();
      asm volatile("bar.sync 3, %0;" ::"n"(AUX_WARPS * 32) : "memory");       // own rows are staged
      // Every thread that will read the receive buffer observes the barrier itself: that is what makes
      // the copy engine's writes visible to it.
      const bool got = __all_sync(0xffffffffu, mbar_wait(recv_bar, 0, ctx, kDevWaitMisc, 0x40000)) != 0;
      // both halves are here: the partner may give up the memory they were copied from
      if (warp == 0 && lane == 0 && got) mbar_arrive_cluster(ack_bar, krank ^ 1u);
      if (*abort_flag == 0) {
        const uint32_t r4 = static_cast<uint32_t>(p.R) >> 2;
        const size_t row0 = static_cast<size_t>(m0) + 32u * krank;
        for (uint32_t it = threadIdx.x; it < 32u * r4; it += AUX_WARPS * 32) {
          const uint32_t row = it / r4, c4 = it - row * r4;
          const uint32_t slot = partial_slot(row, c4, RP4);
          const float4 a = own[slot], b = recv[slot];
          const float4 o = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
          const size_t idx = (row0 + row) * p.R + 4u * c4;
          *reinterpret_cast<float4*>(p.lora + idx) = o;
          if (p.lora16 != nullptr) {
            store_lora16x4<T>(p.lora16, idx, static_cast<size_t>(p.M_pad) * p.R, o);
            if (kBf16 && !fits_f16(o)) atomicOr(lora_unfit, 1u);
          }
        }
      }
      if (kBf16 && p.lora16 != nullptr) {
        asm volatile("bar.sync 3, %0;" ::"n"(AUX_WARPS * 32) : "memory");
        if (threadIdx.x == 0) lora16_flags(p.lora16, static_cast<size_t>(p.M_pad) * p.R)[m0 / 32 + krank] = *lora_unfit;
      }
      // tensor memory goes back while the quantize warps are still busy
      if (warp == 1 && *abort_flag == 0) free_tmem();
      // the partner has everything this CTA sent: only then may the memory it was copied from go away
      if (warp == 0) (void)__all_sync(0xffffffffu, mbar_wait_cluster(ack_bar, 0, ctx, kDevWaitMisc, 0x41000));
    }
  } else if (has_lora) {
    // One rank writes its sums out.  More than two (PUSH) lay them out in the x ring, which nobody needs any more, and the
    // copy engine brings every rank its share of them, counted on that rank's barrier: one trip.  (Ranks that fetched their
    // shares themselves, behind a cluster barrier, took 0.8 us for the barrier and three trips of 0.4 us.  Now the
    // transfer is the bound, 30 KB into every CTA at some 16 bytes a cycle at rank 128; 16-byte st.async from the registers
    // need no staging but arrive one by one: 5.8 instead of 6.0 us at rank 32, 6.5 instead of 5.8 at rank 128.  When it came, 256 x
    // 15360 9.6 -> 9.3 us, 256 x 10240 6.5 -> 6.1, 256 x 3840 5.9 -> 5.8; now 8.9, 5.8 and 5.6.)  A rank's share is cut out of the
    // float4s as they lie here, so which rank adds an element, and with that the order of its sum, goes by R and the number of
    // ranks; it is the same from call to call.
    float4* const stage = reinterpret_cast<float4*>(smem);
    if constexpr (PUSH) { __syncwarp(); cluster_wait(); }     // all ranks' barriers exist
    if (warp >= AUX_WARPS) {
      const int qw = warp - AUX_WARPS;
      const int quarter = warp & 3;                           // TMEM lanes this warp may read
      const int cpart = qw >> 2;                              // column part
      // PUSH, worked out before the sums are there: the copy that this warp issues (one each: fifteen lanes of one warp took
      // 0.7 us to issue theirs; each rank starts with its neighbour) and the first float4 that this thread sums
      [[maybe_unused]] const uint32_t to = krank + 1 + qw < ks ? krank + 1 + qw : krank + 1 + qw - ks;
      [[maybe_unused]] uint32_t copy_lo = 0, copy_bytes = 0, copy_to = 0, copy_bar = 0, row_first = 0;
      [[maybe_unused]] const uint32_t first = item_lo + (NUM_THREADS - 1 - threadIdx.x);
      if constexpr (PUSH) {
        if (static_cast<uint32_t>(qw) + 1 < ks) {
          copy_lo = share_begin(to);
          copy_bytes = (share_begin(to + 1) - copy_lo) * 16u;
          copy_to = map_to_cta(smem_u32(recv + (ks - 2 - qw) * share), to);      // seen from there, this rank is number ks - 1 - qw after it
          copy_bar = map_to_cta(smem_u32(recv_bar), to);
        }
        row_first = first / row4;
      }
      if (cpart * C::EPI_COLS < RP) {
        const bool ok = mbar_wait(acc_done, 0, ctx, kDevWaitAcc, 0);
        tc_fence_after_sync();
        const uint32_t row = quarter * 16 + (lane & 15);
#pragma unroll 1
        for (int c0 = cpart * C::EPI_COLS; c0 < (cpart + 1) * C::EPI_COLS && c0 < p.R; c0 += 32) {
          uint32_t v[32];
          acc_ld(tmem_base() + (static_cast<uint32_t>(quarter * 32) << 16) + c0, v);
          if (lane < 16) {
            if constexpr (PUSH) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                stage[partial_slot(row, (c0 >> 2) + j, row4)] =
                    make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
            } else if (ok) {
              const size_t gm = static_cast<size_t>(m0 + row);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int c = c0 + 4 * j;
                if (c < p.R) {
                  const float4 o = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                               __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                  *reinterpret_cast<float4*>(p.lora + gm * p.R + c) = o;
                  if (p.lora16 != nullptr) {
                    store_lora16x4<T>(p.lora16, gm * p.R + c, static_cast<size_t>(p.M_pad) * p.R, o);
                    if (kBf16 && !fits_f16(o)) atomicOr(lora_unfit, 1u << (row / 32));
                  }
                }
              }
            }
          }
        }
      }
      if constexpr (PUSH) {
        tc_fence_before_sync();
        fence_proxy_async_smem();                             // the copy engine reads what the lanes wrote
        asm volatile("bar.sync 2, %0;" ::"n"(QUANT_WARPS * 32) : "memory");
        if (copy_bytes != 0 && elect_one()) bulk_copy_smem_to_cluster(copy_to, smem_u32(stage + copy_lo), copy_bytes, copy_bar);
        __syncwarp();
        const bool got = first < item_hi && mbar_wait_cluster(recv_bar, 0, ctx, kDevWaitMisc, 0x40000);
        __syncwarp();
        cluster_arrive_relaxed();                             // this rank's share has come: nobody need keep it for it
        if (got) {
          for (uint32_t item = first; item < item_hi; item += QUANT_WARPS * 32) {
            const uint32_t row = item == first ? row_first : item / row4, c = 4 * ((item - row * row4) ^ (row & 7u));
            if (c >= static_cast<uint32_t>(p.R)) continue;
            // this rank's part first, then the following ranks' in turn: a fixed order for every element
            float4 acc = stage[item];
            const float4* part = recv + (item - item_lo);
#pragma unroll 4
            for (uint32_t r = 1; r < ks; ++r, part += share) { const float4 t = *part; acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w; }
            const size_t idx = static_cast<size_t>(m0 + row) * p.R + c;
            *reinterpret_cast<float4*>(p.lora + idx) = acc;
            if (p.lora16 != nullptr) {
              store_lora16x4<T>(p.lora16, idx, static_cast<size_t>(p.M_pad) * p.R, acc);
              if (kBf16 && !fits_f16(acc)) lora16_flags(p.lora16, static_cast<size_t>(p.M_pad) * p.R)[(m0 + row) / 32] = 1u;
            }
          }
        }
        __syncwarp();
      }
    } else if constexpr (PUSH) {
      cluster_arrive_relaxed();
    }
    if constexpr (PUSH) {
      cluster_wait();                                         // no CTA leaves before its copies have been read
      if (warp == 1 && *abort_flag == 0) free_tmem();
    }
  }

  if (ks == 1) {
    tc_fence_before_sync();
    __syncthreads();
    if (kBf16 && has_lora && p.lora16 != nullptr && threadIdx.x == 0) {
      // one word per 32 rows: this CTA wrote rows [m0, m0 + 64) alone
      uint32_t* flags = lora16_flags(p.lora16, static_cast<size_t>(p.M_pad) * p.R);
      const uint32_t unfit = *lora_unfit;
      flags[m0 / 32] = unfit & 1u; flags[m0 / 32 + 1] = (unfit >> 1) & 1u;
    }
  }
  if (*abort_flag) {
    // give copies that were already in flight time to land before the CTA's memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) { __nanosleep(1000); }
  }
  if (tmem_held) free_tmem();
}

// The smoothing table: K reciprocals, K factors, one flag word: 1 if any smooth value lies outside [2^-60, 2^60]
// (2^16 for bf16; negative, zero and NaN count as outside), where the multiplications could over- or underflow or
// leave a zero with the wrong sign; the kernels then divide by the factors with __fdiv_rn.  (K not a multiple of 64
// is outside the fused kernels' contract: no slabs, no permutation.)
template <typename T>
__global__ void smooth_table_kernel(const T* __restrict__ smooth, float* __restrict__ table, int K) {
  // upper bound: 2^60 for fp16 inputs; 2^16 for bf16 inputs, whose smallest subnormal (2^-133)
  // divided by anything larger would underflow to a signed zero
  constexpr float kMaxSmooth = std::is_same<T, __nv_bfloat16>::value ? 65536.0f : 1.1529215e18f;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < K; i += blockDim.x) {
    const float s = to_f32(smooth[i]);
    if (!(s >= 8.6736174e-19f && s <= kMaxSmooth)) bad = 1;      // also: negative, zero or NaN
    const int slot = K % 64 == 0 ? qmath::smooth_table_slot(i) : i;
    table[slot] = qmath::smooth_reciprocal(s);
    table[K + slot] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) *reinterpret_cast<uint2*>(table + 2 * K) = make_uint2(bad != 0 ? 1u : 0u, 0u);
}

}  // namespace qf

// How many CTAs share one row tile along K (0 = no admissible split).
// Clusters of more than two serve inputs of a few hundred to a couple of thousand rows, where two CTAs per row
// tile would leave most SMs idle; they are taken only if all of them can be resident at once (max_clusters(ks):
// clusters of that size the device can hold; 33 of four CTAs, 22 of six, 15 of eight, 11 of ten, 7 of sixteen).
// Cost in slabs (0.24 us); the constants are the ways of bringing the LoRA partial sums together, which hardly depend
// on the cluster size (256 x 3840: 4 / 6 / 8 / 10 / 16 CTAs 7.5 / 6.3 / 5.7 / 5.3 / 5.4 us; 256 x 15360: 8 / 12 / 16 CTAs
// 11.4 / 9.4 / 8.7 us; 1003 x 3840, rank 64: 2 / 4 / 6 CTAs 10.5 / 6.5 / 6.1 us, seven, which are not all resident, 10.8; 2048 x
// 3840: 2 / 3 / 4 CTAs 11.6 / 9.8 / 8.5).
template <typename MaxClusters>
static int pick_k_split(int M_pad, int K, MaxClusters max_clusters) {
  const int tiles = M_pad / qf::TILE_M;
  const int slabs = K / qf::SLAB_K;
  const int sms = sm_count();
  int best = 0;
  double best_cost = 1e30;
  for (int ks : {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16}) {
    if (ks > slabs) continue;
    const int ctas = tiles * ks;
    if (ks > 2 && ctas > sms) continue;
    const int waves = (ctas + sms - 1) / sms;
    const double cost = static_cast<double>(waves) * ((slabs + ks - 1) / ks) + (ks == 1 ? 0.0 : ks == 2 ? 2.0 : 3.0 + 0.05 * ks);
    if (cost < best_cost && (ks <= 2 || tiles <= max_clusters(ks))) { best_cost = cost; best = ks; }
  }
  return best;
}

template <typename T, int RP, bool PUSH> static int max_clusters_t(int ks);

bool quantize_fused_supported(int M, int K, int R, int M_pad) {
  if (M <= 0 || K <= 0 || M_pad < M) return false;
  if (M_pad % qf::TILE_M != 0 || K % qf::SLAB_K != 0) return false;
  if (R < 0 || R > 256 || R % 8 != 0) return false;
  return K >= qf::SLAB_K;
}

int launch_smooth_table(const void* smooth, void* table, int K, int dtype, cudaStream_t stream) {
  if (dtype == SVDQ_DTYPE_F16)
    qf::smooth_table_kernel<__half><<<1, 1024, 0, stream>>>(static_cast<const __half*>(smooth), static_cast<float*>(table), K);
  else if (dtype == SVDQ_DTYPE_BF16)
    qf::smooth_table_kernel<__nv_bfloat16><<<1, 1024, 0, stream>>>(static_cast<const __nv_bfloat16*>(smooth), static_cast<float*>(table), K);
  else
    return SVDQ_ERR_DTYPE;
  return cudaGetLastError() == cudaSuccess ? SVDQ_OK : SVDQ_ERR_LAUNCH;
}

template <typename T, int RP, bool PUSH>
static int launch_qf_form(const void* x, const void* w, const qf::Params& p, int ks, int dev, cudaStream_t stream) {
  using C = qf::Cfg<RP, PUSH>;
  CUtensorMap tmX, tmW;
  int rc;
  if ((rc = make_tmap_2d(&tmX, x, 2, p.M, p.K, static_cast<uint64_t>(p.K) * 2, qf::TILE_M, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
  if (p.R > 0) {
    if ((rc = make_tmap_2d(&tmW, w, 2, p.K, p.R, static_cast<uint64_t>(p.R) * 2, qf::SLAB_K, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
  } else {
    tmW = tmX;
  }
  auto kern = qf::quantize_fused_kernel<T, RP, PUSH>;
  // the attribute is per device: remember which devices of this process have it
  static bool configured[64] = {};
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) return SVDQ_ERR_LAUNCH;
    // clusters of more than eight
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return SVDQ_ERR_LAUNCH;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.M_pad / qf::TILE_M, ks, 1);
  cfg.blockDim = dim3(qf::NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = ks;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kern, tmX, tmW, p) != cudaSuccess) return SVDQ_ERR_LAUNCH;
  return SVDQ_OK;
}

template <typename T, int RP>
static int launch_qf(const void* x, const void* w, const qf::Params& p, cudaStream_t stream, int split_rows) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SVDQ_ERR_CUDA;
  // clusters the device can hold, by size and device, asked for when first needed (value + 2; 0: not asked yet)
  static int caps[64][qf::kMaxKSplit + 1];
  auto max_clusters = [&](int k) -> int {
    if (dev < 0 || dev >= 64) return 0;
    if (caps[dev][k] == 0) caps[dev][k] = max_clusters_t<T, RP, true>(k) + 2;
    return caps[dev][k] - 2;
  };
  const int ks = pick_k_split(split_rows > p.M_pad ? split_rows : p.M_pad, p.K, max_clusters);
  return ks > 2 ? launch_qf_form<T, RP, true>(x, w, p, ks, dev, stream) : launch_qf_form<T, RP, false>(x, w, p, ks, dev, stream);
}

template <typename T, int RP, bool PUSH>
static int max_clusters_t(int ks) {
  using C = qf::Cfg<RP, PUSH>;
  auto kern = qf::quantize_fused_kernel<T, RP, PUSH>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(64, ks, 1);
  cfg.blockDim = dim3(qf::NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = ks; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); return -1; }
  return n;
}

template <typename T>
static int max_clusters_r(int R, int ks) {
  auto form = [&](auto push) {
    constexpr bool P = decltype(push)::value;
    return R <= 64 ? max_clusters_t<T, 64, P>(ks) : R <= 128 ? max_clusters_t<T, 128, P>(ks) : max_clusters_t<T, 256, P>(ks);
  };
  return ks > 2 ? form(std::true_type{}) : form(std::false_type{});
}
int quantize_fused_max_clusters(int R, int ks, int dtype) {
  return dtype == SVDQ_DTYPE_F16 ? max_clusters_r<__half>(R, ks) : max_clusters_r<__nv_bfloat16>(R, ks);
}

int launch_quantize_fused(const void* x, const void* lora_down, const void* smooth_table, void* act, void* ascales,
                          float* lora_act, void* ascales_swz, void* lora_act16, int M, int K, int R, int M_pad,
                          int dtype, cudaStream_t stream, int split_rows) {
  if (!quantize_fused_supported(M, K, R, M_pad)) return SVDQ_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(smooth_table) % 16 != 0) return SVDQ_ERR_ALIGN;   // bulk copies start on 16-byte boundaries
  qf::Params p;
  p.table = static_cast<const float*>(smooth_table);
  p.act = static_cast<uint8_t*>(act);
  p.scales = static_cast<uint8_t*>(ascales);
  p.scales_swz = static_cast<uint8_t*>(ascales_swz);
  p.lora = lora_act;
  p.lora16 = lora_act16;
  p.M = M; p.K = K; p.R = R; p.M_pad = M_pad;
  const int rp = R <= 64 ? 64 : (R <= 128 ? 128 : 256);
  if (dtype == SVDQ_DTYPE_F16) {
    if (rp == 64) return launch_qf<__half, 64>(x, lora_down, p, stream, split_rows);
    if (rp == 128) return launch_qf<__half, 128>(x, lora_down, p, stream, split_rows);
    return launch_qf<__half, 256>(x, lora_down, p, stream, split_rows);
  } else if (dtype == SVDQ_DTYPE_BF16) {
    if (rp == 64) return launch_qf<__nv_bfloat16, 64>(x, lora_down, p, stream, split_rows);
    if (rp == 128) return launch_qf<__nv_bfloat16, 128>(x, lora_down, p, stream, split_rows);
    return launch_qf<__nv_bfloat16, 256>(x, lora_down, p, stream, split_rows);
  }
  return SVDQ_ERR_DTYPE;
}

}  // namespace svdq
