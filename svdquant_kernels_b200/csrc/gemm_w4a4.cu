// Persistent, warp-specialised NVFP4 block-scaled GEMM with the LoRA-up product
// accumulated into the same tensor-memory accumulator and the per-column
// affine fused into the epilogue.
//
//   y = cast( (deq(act) deq(wgt)^T + lora_act lora_up^T) * wcscales + bias )
//
// Math order follows baseline/kernels/gemm_w4a4/ref.py:61-78 of the reference
// (LoRA added before the affine; multiply and add rounded separately in fp32).
// The reference's own kernel for this op is
// cute_kernels/gemm_w4a4/kernel_v2_fa4.py:841-1589.
//
// Work decomposition (320 threads per CTA, one CTA per SM):
//   warps 0-7  epilogue: tensor memory -> registers -> affine -> 16 bit -> y, a
//              32-row x 64-column strip per warp at a time
//   warp  8    producer: TMA loads into a ring of shared-memory stages
//   warp  9    issuer: tcgen05.cp of a slab's scale atoms into tensor memory, its
//              tcgen05.mma's, and the commits
// Copies and MMAs of one thread run in its order, so the issuer waits for one
// barrier per slab and never for the copies; two scale buffers let a slab's
// copies run beside the MMAs of the slab before.  A 256 x 256 x 256 slab keeps the
// tensor pipe busy for 512 cycles, and its 12 copies, 4 MMAs and commits go out
// in about 270 (8 cycles a copy, 40 an MMA) plus 160 for the wait and the loop, as
// long as descriptors and addresses live in uniform registers: the issuing code
// stays converged, elects one lane per slab and builds every operand by adding
// constants to warp-uniform values.  (With address arithmetic and predicates per
// k-block the same slab took 640 cycles to issue, more than it takes to run;
// copies in warps of their own cost a barrier handshake per slab and left the
// issuer at about 600.)
//
// Accumulators.  Tensor memory (512 columns) does not hold two 256-column
// accumulators beside the scales, but it holds three halves: tile t of a CTA uses
// columns [0, 256) or [128, 384) by turns.  The epilogue drains the half that the
// next tile needs too first, which takes about 300 cycles, hands it back, and has
// the whole of the next tile for the rest.  The hand-back is a relaxed remote
// arrival: as a releasing one it waited for everything the thread had under way,
// 1500 cycles per strip, and held up both the next tile and the epilogue.
// 4352 x 3840 -> 3072 / -> 15360, x 15360 -> 3840, x 10240 -> 3072 with all this:
// 30.4 / 118.9 / 102.8 / 56.3 -> 28.2 / 109.7 / 95.9 / 52.4 us.
//
// CG = 1: a CTA computes a 128 x BN tile.
// CG = 2: two CTAs of a cluster compute a 256 x BN tile with cta_group::2
//         MMAs.  Each CTA loads its own 128 rows of A and its own BN/2 rows of
//         B (nothing is fetched twice), its own activation scales, and the
//         weight scales of all BN columns.  Loads of both CTAs complete on the
//         leader's "full" barrier; the leader issues the MMAs and its commits
//         arrive on the barriers of both CTAs.
//
// A stage holds one 256-element K slab: A 128 x 128 B, B rows x 128 B (both
// 128-byte swizzled, K-major, two E2M1 codes per byte) and their scale atoms.
// The LoRA-up product reuses the very same ring: a slab of 64 rank elements of
// lora_act (128 rows x 128 B) and lora_up (B rows x 128 B) has exactly the byte
// footprint of a main slab, so it is ceil(R/64) more ring passes per output
// tile, issued as dense 16-bit MMAs into the same accumulator.  Both operands
// of a dense MMA must have the same 16-bit format (an fp16 x bf16 pair is an
// illegal instruction on this part), so lora_act arrives in the output type:
// fp16 as one rounded copy, bf16 as a hi + lo pair (lora_act = hi + lo to 16
// significant bits) that takes two passes over the same lora_up slab - a single
// bf16 copy would put the LoRA term's 2^-9 rounding error above the 1e-3 bound.
// For bf16 the quantizer also provides lora_act as an fp16 plane with a word per 32
// rows telling whether those rows fit fp16; given an fp16 copy of lora_up, a tile
// whose rows all fit takes a single fp16 pass instead (decided per tile by every
// role from the same words, so all agree on the tile's slab count).
//
// Column-sharded form (TP): the launch fills N columns of a wider result that every
// GPU holds in full; each finished strip goes through a staging buffer in shared
// memory and leaves it as one TMA store into the local copy and one per peer, into
// the peers' copies over NVLink (lane stores of 16 bytes measured the same there: the
// link, not the store path, sets the pace).
//
// Split-K within clusters (SK = kClusterSplit): for problems with few tiles and a long K, the S pairs
// of a cluster share a 256 x 128 tile's slabs and add their partial tiles up through distributed shared memory.
//
// Split-K through a workspace (SK = kWorkspaceSplit, one CTA per 128 x 128 tile part; row counts that are an odd multiple
// of 128, or on request): S CTAs share a tile's slabs.  Each parks its fp32 partial tile in a caller-owned
// workspace (thread t writes float4 j at [j][t], so every access is a whole line per warp and a
// thread later reads back exactly the places its namesakes wrote), fences, and draws a ticket
// from the tile's counter; the CTA that draws ticket S - 1 adds the S partials in split order -
// the result does not depend on who finished first - runs the epilogue and zeroes the counter.
// No CTA waits for another, so nothing depends on the CTAs of a tile running together.
#include "nvfp4_math.cuh"
#include "quantize_math.cuh"
#include "sm100.cuh"
#include "svdq_internal.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdlib>
#include <type_traits>

namespace svdq {

namespace gemm {

constexpr int BM = 128;          // rows of y per CTA
constexpr int BK = 256;          // K elements per stage (128 bytes of codes per row)
constexpr int A_BYTES = BM * 128;
constexpr int SFA_BYTES = BM * (BK / 16);  // 2048
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = (EPI_WARPS + 2) * 32;
constexpr int STORE_BUF_BYTES = 32 * 128;  // one 32-row x 64-column strip of y
template <int CG, int BN, bool NEXT = false, bool TP = false>
struct Cfg {
  static constexpr int B_ROWS = BN / CG;                           // rows of B this CTA loads
  static constexpr int B_BYTES = B_ROWS * 128;
  static constexpr int SFB_BYTES = BN * (BK / 16);
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;
  // Accumulators: tile t of a CTA starts at column 128 (t % 2).  128-column tiles simply alternate; 256-column
  // tiles share the middle 128 columns with their neighbours.
  static constexpr bool SHARED_ACC = BN == 256;
  static constexpr int ACC_COLS = 128 + BN;
  static constexpr int STORE_BYTES = TP ? EPI_WARPS * STORE_BUF_BYTES : 0;
  // per-column rows of the current tile: wcscales, bias and, for the next layer's quantisation, -smooth_next and
  // 1 / smooth_next
  static constexpr int AFFINE_BYTES = (NEXT ? 4 : 2) * BN * 4;
  static constexpr int LUT_BYTES = NEXT ? qmath::kScaleLutEntries * 4 : 0;    // the multiplier of each scale byte
  static constexpr int TAIL_BYTES = AFFINE_BYTES + LUT_BYTES + 512 /*barriers*/;
  static constexpr int STAGES_RAW = (232448 - 1024 - STORE_BYTES - TAIL_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_RAW > 8 ? 8 : STAGES_RAW;
  static constexpr int SFA_COLS = 16;                 // 4 k-blocks x 4 columns
  static constexpr int SFB_COLS = 4 * (BN / 32);      // 4 k-blocks x BN/32 columns
  static constexpr int SF_COLS = SFA_COLS + SFB_COLS; // one scale buffer
  // Scale buffers in tensor memory.  Copies into them and the MMAs that read them are issued by one thread and run
  // in its order; a second buffer lets a slab's copies run beside the MMAs of the slab before.
  static constexpr int SF_BUFS_FIT = (512 - ACC_COLS) / SF_COLS;
  static constexpr int SF_BUFS = SF_BUFS_FIT > 4 ? 4 : SF_BUFS_FIT;
  static constexpr int TMEM_COLS = 512;
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + STORE_BYTES + TAIL_BYTES;
  static_assert(ACC_COLS + SF_BUFS * SF_COLS <= TMEM_COLS && SF_BUFS >= 2, "tensor memory budget");
  static_assert(STAGES >= 3 && STAGES * STAGE_BYTES >= BN / 128 * EPI_WARPS * STORE_BUF_BYTES, "ring too shallow");
  static_assert((2 * STAGES + 6) * 8 + 16 <= 512, "barrier block");
};

// Column-sharded form: tensor maps of this GPU's copy of the result and of the peers' (same geometry).
struct PeerMaps {
  CUtensorMap y, m[7];
};
struct NoMaps {};
// bf16: tensor maps of lora_act's fp16 plane and of lora_up's fp16 copy.  (fp16 kernels do without: a launch costs the host
// 0.6 us per KB of parameters.)
struct LoraF16Maps {
  CUtensorMap la, lu;
};

struct Params {
  void* y;              // [M, N] (column-sharded form: through the tensor maps instead)
  int y_wide;           // y is 32-byte aligned: one store instruction per 16 columns instead of two
  const void* wc;       // [N] or null
  const void* bias;     // [N] or null
  const uint32_t* la_flags;   // bf16 only: per 32 rows of lora_act, non-zero = does not fit fp16; null = always two-pass
  int M, N, K, R;
  int tiles_m, tiles_n; // in units of (CG*128) x BN
  int whole_tiles;      // tiles from this one on are worked on as two halves of BN / 2 columns (see launch_gemm_t)
  // Column-sharded (tensor-parallel) form: this launch computes columns [col0, col0 + N) of a
  // [M, y_ld] result that every rank holds in full.  The local copy is written through a tensor map (built over
  // the local full matrix); each finished strip is also stored, by TMA from the same staging buffer,
  // into the same place of every peer's matrix (peer-mapped memory, one tensor map per peer).
  int col0, n_peers;
  // Split-K forms (SK kernels only): a tile's slabs are shared by `splits` CTAs or pairs.  Workspace form: each writes its fp32
  // partial tile to ws_partials[(tile * splits + split) * BM * BN], takes a ticket from
  // ws_tickets[tile], and the CTA that draws the last ticket adds the partials in split order, runs
  // the epilogue and puts the ticket counter back to zero.
  int splits;
  int interleave;       // 1: LoRA slabs spread evenly among the main slabs of a tile; 0: after them
  int stride1, stride2; // interleaved: positions between LoRA slabs of a tile with one / two LoRA passes
  float4* ws_partials;
  unsigned int* ws_tickets;
  // Next-layer quantisation (NEXT kernels only): the fp32 result, before its cast, divided by
  // smooth_next [N] and packed as NVFP4 rows: qout [M, N/2], oscales [N/16, M] (+ the tensor-core twin).
  const void* smooth_next;
  uint8_t* qout;
  uint8_t* oscales;
  uint8_t* oscales_swz;
};

template <typename T> __device__ __forceinline__ uint32_t pack2f(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2f<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2f<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ float as_f32(T v);
template <> __device__ __forceinline__ float as_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float as_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Next layer's quantisation of one 16-column group of one row: the 16 fp32 results (already scaled and
// biased) are divided by smooth_next and packed as NVFP4.  ns4: the group's four entries of the -smooth_next row.
// Returns {codes 0-7, codes 8-15, scale byte, -}.  This form takes every case, by IEEE division of the uncast fp32
// values, as the reference does; + 0 turns a -0 quotient into +0 (the reference gives a zero the sign bit only when the
// value tests < 0).  Not inlined: it is for the rare ones (next_two_groups).
__device__ __noinline__ uint4 next_group_any(float2 a0, float2 a1, float2 a2, float2 a3, float2 a4, float2 a5, float2 a6, float2 a7,
                                             const float4* ns4, const float* lut) {
  const float2 a[8] = {a0, a1, a2, a3, a4, a5, a6, a7};
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) bits |= __float_as_uint(a[j].x) | __float_as_uint(a[j].y);
  if ((bits & 0x7FFFFFFFu) == 0u) return make_uint4(0u, 0u, 0u, 0u);        // a group of zeros, as rows of the padding can be
  float2 q[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 ns = ns4[j];
    q[2 * j] = make_float2(__fadd_rn(__fdiv_rn(a[2 * j].x, -ns.x), 0.0f), __fadd_rn(__fdiv_rn(a[2 * j].y, -ns.y), 0.0f));
    q[2 * j + 1] = make_float2(__fadd_rn(__fdiv_rn(a[2 * j + 1].x, -ns.z), 0.0f), __fadd_rn(__fdiv_rn(a[2 * j + 1].y, -ns.w), 0.0f));
  }
  const uint32_t sb = qmath::group_scale_byte(q);
  uint32_t lo, hi;
  const float c = lut[sb];
  if (c != 0.0f) qmath::group_codes_cut(q, c, lo, hi);
  else qmath::group_codes_compare(q, sb, lo, hi);
  return make_uint4(lo, hi, sb, 0u);
}
// Two neighbouring groups of one row, the same quotients in three packed instructions per pair
// (qmath::divide_by_constant2).  Side by side and inline, so that one's chain of dependent steps fills the other's gaps: an
// epilogue warp has only one other on its scheduler (a call per group: 4352 x 1024 -> 3072 bf16, both kernels, 30.0 -> 27.8 us,
// 4352 x 3840 -> 3072 fp16 47.4 -> 46.5).  Groups that the three steps do not settle go to next_group_any: tile_fdiv, and a
// scale byte of 0 or 448, a group of tiny or of huge values, where a quotient may have under- or overflowed on the way.
// (With a byte in between, the group's largest quotient lies in [2^-10, 2700): every operand that can reach a rounding bound
// of a code is far from both ends of the range, and the quotients that matter are exact.)
__device__ __forceinline__ void next_two_groups(const float2 (&a)[16], const float4* ns4, const float4* r4, const float* lut, bool tile_fdiv,
                                                uint32_t (&codes)[4], uint32_t (&sb)[2]) {
  const float2 zero = make_float2(0.0f, 0.0f);
  float2 q[2][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float4 ns = ns4[j], r = r4[j];
    q[j >> 2][2 * (j & 3)] = __fadd2_rn(qmath::divide_by_constant2(a[2 * j], make_float2(ns.x, ns.y), make_float2(r.x, r.y)), zero);
    q[j >> 2][2 * (j & 3) + 1] = __fadd2_rn(qmath::divide_by_constant2(a[2 * j + 1], make_float2(ns.z, ns.w), make_float2(r.z, r.w)), zero);
  }
  sb[0] = qmath::group_scale_byte(q[0]);
  sb[1] = qmath::group_scale_byte(q[1]);
  const float c0 = lut[sb[0]], c1 = lut[sb[1]];
  if (!tile_fdiv && c0 != 0.0f && c1 != 0.0f) {
    qmath::group_codes_cut(q[0], c0, codes[0], codes[1]);
    qmath::group_codes_cut(q[1], c1, codes[2], codes[3]);
  } else {
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const uint4 t = next_group_any(a[8 * g], a[8 * g + 1], a[8 * g + 2], a[8 * g + 3], a[8 * g + 4], a[8 * g + 5], a[8 * g + 6], a[8 * g + 7],
                                     ns4 + 4 * g, lut);
      codes[2 * g] = t.x; codes[2 * g + 1] = t.y; sb[g] = t.z;
    }
  }
}

// How a tile's K loop is split over CTAs (see the header comment): not at all, through a workspace, within a cluster
enum SplitForm : int { kNoSplit = 0, kWorkspaceSplit = 1, kClusterSplit = 2 };

// HALVES: the last round's tiles are worked on as two halves of BN / 2 columns each (see gemm_halved_tiles).  A form of its
// own: with the choice in the issuing loop of every launch, those without halves took 1 % longer.
template <int CG, int BN, typename OutT, int SK = kNoSplit, bool NEXT = false, bool TP = false, bool HALVES = false>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_w4a4_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmLA, const __grid_constant__ CUtensorMap tmLU,
                 const __grid_constant__ CUtensorMap tmSFA, const __grid_constant__ CUtensorMap tmSFB,
                 const __grid_constant__ typename std::conditional<std::is_same<OutT, __nv_bfloat16>::value, LoraF16Maps, NoMaps>::type lora_f16,
                 const __grid_constant__ typename std::conditional<TP, PeerMaps, NoMaps>::type maps, const Params p) {
  using C = Cfg<CG, BN, NEXT, TP>;
  constexpr bool kBf16 = std::is_same<OutT, __nv_bfloat16>::value;

  extern __shared__ uint8_t smem_raw[];
  // 1 KB alignment by pointer arithmetic (not an integer round trip) so that the compiler keeps
  // the shared address space and emits shared-memory loads and stores
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  [[maybe_unused]] uint8_t* store_bufs = smem + C::STAGES * C::STAGE_BYTES;   // TP; 1024-aligned: every stage is a multiple of 1 KB
  uint8_t* tail = smem + C::STAGES * C::STAGE_BYTES + C::STORE_BYTES;
  float* affine = reinterpret_cast<float*>(tail);                 // [2 or 4][BN] : wcscales, bias, -smooth_next, 1/smooth_next of the current tile
  [[maybe_unused]] float* scale_lut = reinterpret_cast<float*>(tail + C::AFFINE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail + C::AFFINE_BYTES + C::LUT_BYTES);
  uint64_t* full = bars;                                          // [STAGES] operands and scales landed (leader CTA's copy is used)
  uint64_t* empty = bars + C::STAGES;                             // [STAGES] stage consumed by the MMAs (per CTA)
  uint64_t* acc_full = bars + 2 * C::STAGES;                      // [2]      accumulator complete (per CTA)
  uint64_t* acc_empty = acc_full + 2;                             // [2]      accumulator drained (leader's copy is used)
  uint64_t* acc_shared = acc_empty + 2;                           // its columns that the next tile uses too are drained (leader's copy)
  uint64_t* tmem_ready = acc_shared + 1;                          // tensor memory allocated (leader's copy: in both CTAs)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile uint32_t* sk_ticket = tmem_slot + 2;                   // split-K through a workspace: the ticket this CTA drew for its tile
  [[maybe_unused]] volatile uint32_t* ahead_done = tmem_slot + 3; // split-K within clusters: the kernel ahead has finished
  const WaitCtx ctx{abort_flag};
  // bounded wait whose verdict is the same in all lanes of the calling (converged) warp
  auto uwait = [&](uint64_t* bar, uint32_t parity, const WaitCtx& c, unsigned int code, unsigned int tag) -> bool {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, c, code, tag)) != 0;
  };

  // The warp index is taken through a shuffle so that the compiler can prove it warp-uniform: only
  // then do the role branches below count as convergent code, where descriptors and addresses stay
  // in uniform registers.  Single-lane roles also vote on every wait result for the same reason.
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  // rank 0 = leader of the pair; where in the cluster the leader is: a constant wherever the cluster is the pair, else a
  // warp-uniform value (the issuing loop must not lose its uniform registers to it: 0.2 instead of 0.17 us per slab)
  const uint32_t cta = (CG == 1) ? 0u : SK == kClusterSplit ? __shfl_sync(0xffffffffu, cluster_ctarank(), 0) : cluster_ctarank();
  const uint32_t rank = SK == kClusterSplit ? (cta & 1u) : cta;
  const uint32_t leader = SK == kClusterSplit ? (cta & ~1u) : 0u;
  const int pair = blockIdx.x / CG;
  const int num_pairs = gridDim.x / CG;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *ahead_done = 0;
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], EPI_WARPS * CG); }
    mbar_init(acc_shared, EPI_WARPS * CG);
    mbar_init(tmem_ready, CG);
    fence_barrier_init();
  }
  if (warp == EPI_WARPS && lane == 0) {
    tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
    if constexpr (TP) tma_prefetch_desc(&maps.y);
    tma_prefetch_desc(&tmSFA); tma_prefetch_desc(&tmSFB);
    if (p.R > 0) { tma_prefetch_desc(&tmLA); tma_prefetch_desc(&tmLU); }
    if constexpr (kBf16) {
      if (p.R > 0 && p.la_flags != nullptr) { tma_prefetch_desc(&lora_f16.la); tma_prefetch_desc(&lora_f16.lu); }
    }
  }
  if constexpr (NEXT) qmath::fill_near_lut(scale_lut, threadIdx.x, NUM_THREADS);
  __syncthreads();
  if constexpr (CG == 2) cluster_arrive_relaxed();       // (fence_barrier_init is what releases the barriers)
  // Tensor memory: only the issuer waits for it (its loads are under way by then), the epilogue reads the address once an
  // accumulator is complete.
  if (warp == EPI_WARPS + 1) {
    if constexpr (CG == 1) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
    else { tmem_alloc_pair(tmem_slot, C::TMEM_COLS); tmem_relinquish_pair(); }
  }
  if constexpr (CG == 2) cluster_wait();       // both CTAs' barriers exist before anything remote touches them
  if (warp == EPI_WARPS + 1) {
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) { if constexpr (CG == 2) mbar_arrive_cluster(tmem_ready, leader); else mbar_arrive(tmem_ready); }
  }
  // Everything above touched only this CTA's shared and tensor memory, so it may overlap the tail of the kernel before this
  // one in the stream.  Each role waits for that kernel (pdl_wait) before it reads what may be its outputs; the producer
  // has its first tile and addresses worked out by then.  (With the wait here they took it another 0.25 us, and bf16
  // tiles' words 0.8 us more, before the first load: 256 x 3840 -> 3072 6.4 -> 6.2 us, 1003 x 3840 -> 3072 bf16 10.1 -> 9.7.)
  const int kt_main = (p.K + BK - 1) / BK;   // the last slab may hold fewer than four 64-element k-blocks
  const int lora_slabs = (p.R + 63) / 64;
  // bf16 output: lora_act comes as hi and lo bf16 planes (two passes over the same lora_up slab) and
  // as an fp16 plane; a tile whose 32-row blocks all carry a zero "does not fit fp16" word takes
  // the fp16 plane and the fp16 copy of lora_up in a single pass.  Every role of both CTAs
  // evaluates this per tile from the same words, so they agree on the number of slabs.
  // The words come from L2, so a role asks for the next tile's while it works on this one's.
  // Work items: tiles, tile halves after the first `whole_tiles` of them, or (tile, split) pairs.
  static_assert(!HALVES || (CG == 2 && BN == 256 && SK == kNoSplit && !TP), "halved tiles");
  const int total_tiles = p.tiles_m * p.tiles_n;
  const int S = SK ? p.splits : 1;
  const int total_work = HALVES ? 2 * total_tiles - p.whole_tiles : total_tiles * S;
  auto is_half = [&](int work) -> bool { return HALVES && work >= p.whole_tiles; };
  auto tile_of = [&](int work) -> int { return SK ? work / S : is_half(work) ? (work + p.whole_tiles) >> 1 : work; };
  auto lora_words = [&](int work) -> uint32_t {
    if (!kBf16 || p.R == 0 || p.la_flags == nullptr || work >= total_work) return 1u;
    constexpr int kWords = CG * BM / 32;
    return lane < kWords ? __ldg(p.la_flags + tile_of(work) % p.tiles_m * kWords + lane) : 0u;
  };
  auto lora_fp16 = [&](uint32_t words) -> bool { return kBf16 && __all_sync(0xffffffffu, words == 0u) != 0; };
  auto lora_parts = [&](bool fp16_pass) -> int { return (kBf16 && !fp16_pass) ? 2 : 1; };
  const int k_groups4 = p.K / 64;            // scale atoms along K
  // (tile, split) pairs are numbered tile-major so that the CTAs sharing a tile run at the same time.  Split i of a
  // tile with n slabs (LoRA slabs of one pass included, at the end) takes slabs [i n / S, (i + 1) n / S); a second LoRA
  // pass is the last split's.  So where a range begins, and all of it before the LoRA slabs, does not depend on the
  // number of passes, and no role waits for the words before its first slab.
  auto slab_range = [&](int split, int& lo, int& hi) {
    const int n = kt_main + lora_slabs;
    if (SK) { lo = split * n / S; hi = (split + 1) * n / S; } else { lo = 0; hi = n; }
  };
  auto slabs_end = [&](int split, int hi, bool fp16_pass) -> int { return split == S - 1 ? kt_main + lora_parts(fp16_pass) * lora_slabs : hi; };
  // Which slab runs at position pos of a tile's kt_all = kt_main + n_lora slabs.  Slab numbers below
  // kt_main are main slabs, the others LoRA slabs.  End-grouped: position = number.  Interleaved (the
  // reference's schedule, cute_kernels/gemm_w4a4/kernel_v2_fa4.py:299-303): LoRA slab j sits at position
  // (j + 1) * stride - 1 with stride = kt_all / n_lora, the main slabs fill the rest in order.  Every
  // role walks the positions with one of these and the same arguments, so all agree.  No division in
  // the per-slab step: the issuing threads have a few hundred cycles per slab for everything.
  struct SlabWalk {
    int kt_main, n_lora, stride, lora_done, next_lora;
    __device__ __forceinline__ void start(int kt_main_, int kt_all, int interleave, int stride_, int first_pos) {
      kt_main = kt_main_;
      n_lora = interleave ? kt_all - kt_main_ : 0;
      stride = stride_;
      lora_done = 0;
      if (n_lora > 0 && first_pos > 0) { lora_done = first_pos / stride; if (lora_done > n_lora) lora_done = n_lora; }
      next_lora = (lora_done + 1) * stride - 1;
    }
    __device__ __forceinline__ int at(int pos) {
      if (lora_done < n_lora && pos == next_lora) { const int kt = kt_main + lora_done; ++lora_done; next_lora += stride; return kt; }
      return pos - lora_done;
    }
  };
  // stride of a tile with one / two LoRA passes (worked out on the host)
  auto lora_stride = [&](bool fp16_pass) -> int { return (kBf16 && !fp16_pass) ? p.stride2 : p.stride1; };
  bool tmem_held = true;
  auto free_tmem = [&]() {
    tc_fence_after_sync();
    const uint32_t base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    if constexpr (CG == 1) tmem_dealloc(base, C::TMEM_COLS); else tmem_dealloc_pair(base, C::TMEM_COLS);
  };
  // End of a warp's part in what the CTA pair shares (barriers, operands, tensor memory); see the teardown.
  auto leave = [&]() {
    if constexpr (CG == 2) cluster_arrive_relaxed();
    else if (warp < EPI_WARPS) asm volatile("bar.arrive 2, %0;" ::"n"((EPI_WARPS + 1) * 32) : "memory");
  };
  if (warp == EPI_WARPS) {
    // ------------------------------ producer (both CTAs) ------------------------------
    uint32_t s = 0, ph = 1, it = 0;
    bool ok = true;
    uint32_t words = 1u;
    bool waited = false;
    auto wait_ahead = [&]() {
      if (!waited) {
        pdl_wait();
        if (SK == kClusterSplit) *ahead_done = 1;
        words = lora_words(pair);
        waited = true;
      }
    };
    for (int w = pair; w < total_work && ok; w += num_pairs) {
      const int tile = tile_of(w), split = SK ? w - tile * S : 0;
      const int mb = tile % p.tiles_m, nb = tile / p.tiles_m;
      const int m0 = (mb * CG + rank) * BM;
      // a half: 128 columns, half of them this CTA's rows of B
      const bool half = is_half(w);
      const int hsel = half ? (w - p.whole_tiles) & 1 : 0;
      const int nrow0 = nb * BN + hsel * (BN / 2) + static_cast<int>(rank) * (half ? C::B_ROWS / 2 : C::B_ROWS);
      int kt_lo, kt_hi;
      slab_range(split, kt_lo, kt_hi);
      // The number of LoRA passes: of the first tile only when its first LoRA slab is due (unless they are interleaved).
      bool la_fp16 = false, la_known = !kBf16;
      SlabWalk walk;
      auto lora_verdict = [&]() {
        wait_ahead();
        la_fp16 = lora_fp16(words);
        words = lora_words(w + num_pairs);
        kt_hi = slabs_end(split, kt_hi, la_fp16);
        la_known = true;
      };
      if (it > 0 || p.interleave) lora_verdict();
      walk.start(kt_main, kt_main + lora_parts(la_fp16) * lora_slabs, p.interleave, lora_stride(la_fp16), kt_lo);
      for (int pos = kt_lo; pos < kt_hi && ok;) {
        if (!la_known && pos >= kt_main) lora_verdict();
        const int stop = la_known || kt_hi < kt_main ? kt_hi : kt_main;
        for (; pos < stop; ++pos, ++it) {
          const int kt = walk.at(pos);
          if (!uwait(&empty[s], ph, ctx, kDevWaitEmpty, it)) { ok = false; break; }
          if (it == C::STAGES) pdl_trigger();       // the first stage has been consumed: see pdl_trigger
          uint8_t* st = smem + s * C::STAGE_BYTES;
          // the barrier that counts this CTA's bytes: its own for CG = 1, the leader's for a pair
          const uint32_t bar = (CG == 2) ? map_to_cta(smem_u32(&full[s]), leader) : smem_u32(&full[s]);
          // Codes past K are zero-filled by TMA.  The scale atoms of a (128-row block, slab) are four
          // consecutive 512-byte rows of the swizzled scale buffer seen as a [blocks * K/64, 512 B] matrix;
          // a short last slab just fetches (and never uses) the rows that follow.  Every byte of a box
          // counts toward the barrier whether it was in bounds or not.
          const uint32_t kSfBytes = SFA_BYTES + (half ? C::SFB_BYTES / 2 : C::SFB_BYTES), kAbBytes = A_BYTES + (half ? C::B_BYTES / 2 : C::B_BYTES);
          // B rows: one box, or with HALVES two, of which a half takes one
          auto load_b = [&](const CUtensorMap* m, int x) {
            tma_load_2d_bar<CG>(st + A_BYTES, m, x, nrow0, bar);
            if (HALVES && !half) tma_load_2d_bar<CG>(st + A_BYTES + C::B_BYTES / 2, m, x, nrow0 + C::B_ROWS / 2, bar);
          };
          wait_ahead();
          if (elect_one()) {
            if (kt < kt_main) {
              if (rank == 0) mbar_arrive_expect_tx(&full[s], (kSfBytes + kAbBytes) * CG);
              tma_load_2d_bar<CG>(st + A_BYTES + C::B_BYTES, &tmSFA, 0, (mb * CG + rank) * k_groups4 + kt * 4, bar);
#pragma unroll
              for (int h = 0; h < BN / 128; ++h)
                if (h == 0 || !half)
                  tma_load_2d_bar<CG>(st + A_BYTES + C::B_BYTES + SFA_BYTES + h * 2048, &tmSFB, 0,
                                      (nb * (BN / 128) + hsel + h) * k_groups4 + kt * 4, bar);
              tma_load_2d_bar<CG>(st, &tmA, kt * 128, m0, bar);
              load_b(&tmB, kt * 128);
            } else {
              if (rank == 0) mbar_arrive_expect_tx(&full[s], kAbBytes * CG);
              const int lt = kt - kt_main;
              const int part = lt / lora_slabs, r0 = (lt % lora_slabs) * 64;
              const CUtensorMap *la_map = &tmLA, *lu_map = &tmLU;
              int la_row = part * p.M + m0;                                  // lora_act parts are stacked along rows
              if constexpr (kBf16) {
                if (la_fp16) { la_map = &lora_f16.la; lu_map = &lora_f16.lu; la_row = m0; }
              }
              tma_load_2d_bar<CG>(st, la_map, r0, la_row, bar);
              load_b(lu_map, r0);
            }
          }
          __syncwarp();
          if (++s == C::STAGES) { s = 0; ph ^= 1; }
        }
      }
      if (!la_known) words = lora_words(w + num_pairs);
    }
    if (it <= C::STAGES) pdl_trigger();
  } else if (warp == EPI_WARPS + 1) {
    // ------------------------------ MMA issuer (leader CTA only) ------------------------------
    if (rank == 0) {
      constexpr uint64_t kDescAB = smem_desc_base(0, 1024, kSwizzle128B);   // K-major, 8-row groups 1024 B apart
      constexpr uint64_t kDescSF = smem_desc_base(0, 128, kSwizzleNone);    // 8 x 16 B core matrices, 128 B apart
      constexpr uint32_t kIdescHalf = (BN / 2 >> 3) << 17;      // off a descriptor's columns for a half tile
      constexpr uint32_t kIdescLora = idesc_f16(kBf16, kBf16, BM * CG, BN, false, false);
      constexpr uint32_t kIdescLoraF16 = idesc_f16(false, false, BM * CG, BN, false, false);
      const uint16_t mask = static_cast<uint16_t>((CG == 2 ? 3u : 1u) << leader);     // both CTAs of the pair
      const uint32_t smem16 = smem_desc_addr(smem);
      uint32_t s = 0, ph = 0, tcount = 0, sb = 0, it = 0;
      bool ok = uwait(tmem_ready, 0, ctx, kDevWaitTmem, 0);
      tc_fence_after_sync();
      const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0);   // warp-uniform, for the same reason as the warp index
      const uint32_t tmem_sf = tmem_base + C::ACC_COLS;              // SF_BUFS buffers of [SFA 16 | SFB] columns
      pdl_wait();
      uint32_t words = lora_words(pair);
      for (int w = pair; w < total_work && ok; w += num_pairs, ++tcount) {
        const int split = SK ? w - tile_of(w) * S : 0;
        const bool half = is_half(w);
        const uint32_t as = tcount & 1;
        int kt_lo, kt_hi;
        slab_range(split, kt_lo, kt_hi);
        bool la_fp16 = false, la_known = !kBf16;
        SlabWalk walk;
        auto lora_verdict = [&]() {
          la_fp16 = lora_fp16(words);
          words = lora_words(w + num_pairs);
          kt_hi = slabs_end(split, kt_hi, la_fp16);
          la_known = true;
        };
        if (tcount > 0 || p.interleave) lora_verdict();
        walk.start(kt_main, kt_main + lora_parts(la_fp16) * lora_slabs, p.interleave, lora_stride(la_fp16), kt_lo);
        if (!uwait(&acc_empty[as], ((tcount >> 1) & 1) ^ 1, ctx, kDevWaitAccFree, tcount)) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + as * 128;
        // 256-column tiles: the half shared with the tile before (in 128-column tiles acc_empty covers everything)
        if (C::SHARED_ACC && tcount > 0) {
          if (!uwait(acc_shared, (tcount - 1) & 1, ctx, kDevWaitAccFree, 0x20000 + tcount)) break;
          tc_fence_after_sync();
        }
        for (int pos = kt_lo; pos < kt_hi && ok;) {
          if (!la_known && pos >= kt_main) lora_verdict();
          const int stop = la_known || kt_hi < kt_main ? kt_hi : kt_main;
          const int last = stop == kt_hi ? kt_hi - 1 : -1;          // the tile's last position, if it is in this stretch
          for (; pos < stop; ++pos, ++it) {
            const int kt = walk.at(pos);
            if (!uwait(&full[s], ph, ctx, kDevWaitFull, it)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t stage16 = smem16 + s * (C::STAGE_BYTES / 16);
            const uint64_t da = kDescAB + stage16, db = da + A_BYTES / 16;
            const uint32_t accumulate = pos == kt_lo ? 0u : 1u;
            if (elect_one()) {
              if (kt < kt_main) {
                const uint64_t dsa = kDescSF + stage16 + (A_BYTES + C::B_BYTES) / 16, dsb = dsa + SFA_BYTES / 16;
                const uint32_t tsfa = tmem_sf + sb * C::SF_COLS, tsfb = tsfa + C::SFA_COLS;
                // the slab's k-blocks: all their scales, then their MMAs (a tile's columns, or a half's)
                auto k_blocks = [&](int nkb, auto cols) {
                  constexpr int COLS = decltype(cols)::value;
#pragma unroll
                  for (int j = 0; j < 4; ++j)
                    if (j < nkb) {
                      tmem_cp_scales<CG>(tsfa + j * 4, dsa + j * 32);
#pragma unroll
                      for (int h = 0; h < COLS / 128; ++h) tmem_cp_scales<CG>(tsfb + j * (BN / 32) + h * 4, dsb + h * 128 + j * 32);
                    }
#pragma unroll
                  for (int j = 0; j < 4; ++j)
                    if (j < nkb)
                      mma_nvfp4<CG>(acc, da + j * 2, db + j * 2, idesc_nvfp4(BM * CG, COLS), tsfa + j * 4, tsfb + j * (BN / 32), j != 0 ? 1u : accumulate);
                };
                const int nkb = k_groups4 - kt * 4;
                const std::integral_constant<int, BN> all_cols;
                const std::integral_constant<int, HALVES ? BN / 2 : BN> half_cols;
                if (HALVES && half) k_blocks(nkb >= 4 ? 4 : nkb, half_cols);
                else if (nkb >= 4) k_blocks(4, all_cols);
                else k_blocks(nkb, all_cols);                       // the last slab may be short
              } else {
                const uint32_t idesc = (la_fp16 ? kIdescLoraF16 : kIdescLora) - (half ? kIdescHalf : 0u);
                const int nkb = (p.R - ((kt - kt_main) % lora_slabs) * 64) / 16;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  if (j < nkb) mma_f16<CG>(acc, da + j * 2, db + j * 2, idesc, j != 0 ? 1u : accumulate);
              }
              tc_commit_mask<CG>(&empty[s], mask);          // stage reusable (in both CTAs) once these MMAs have read it
              if (pos == last) tc_commit_mask<CG>(&acc_full[as], mask);    // accumulator complete
            }
            __syncwarp();
            if (++sb == C::SF_BUFS) sb = 0;
            if (++s == C::STAGES) { s = 0; ph ^= 1; }
          }
        }
        if (!la_known) words = lora_words(w + num_pairs);
      }
    }
  } else {
    // ------------------------------ epilogue (warps 0-7, both CTAs) ------------------------------
    // Warp w drains the 32 accumulator rows of lane quarter w % 4, in strips of 64 columns: half w / 4 of each 128.
    const OutT* wc = static_cast<const OutT*>(p.wc);
    const OutT* bias = static_cast<const OutT*>(p.bias);
    const int quarter = warp & 3, chalf = warp >> 2;
    uint32_t tcount = 0;
    bool ok = true, drained = false;
    if (SK == kClusterSplit && warp == 0) {
      // Long K loops over weights that come from DRAM: a CTA that is here while the kernel ahead is still at work (the quantizer
      // leaves half of the SMs to half of these CTAs) asks for its slabs of them, into L2, until that has ended.  Not before a
      // moment has passed, and at a pace, or the hints stand in the copy engine in front of the loads: without either, and in
      // every form, 256 x 15360 -> 3840 took 25.3 us instead of 23.8 for both kernels, and forms with a short K loop gain
      // nothing this way either (256 x 3840 -> 3072 11.7 -> 11.8).  Both kernels without / with the hints, us, over eight to
      // twelve sets of weights, more than L2 holds, as in a model whose layers run in turn: 256 x 15360 -> 3840 22.58 / 22.40,
      // -> 3072 22.28 / 21.89, -> 1536 17.52 / 17.48, 256 x 12800 -> 4608 20.31 / 20.31, 256 x 10240 -> 3072 16.69 / 16.35, 256 x
      // 7680 -> 2304 14.85 / 14.89, 512 x 12288 -> 1536 20.01 / 19.76, 768 x 6592 -> 512 14.58 / 14.48; none of the other splits
      // lost either.  Weights that are in L2 already have nothing to gain, and pay for it: over two sets 22.26 / 22.27, 21.58 /
      // 21.7, 16.39 / 16.48, 19.5 / 19.6, 15.72 / 15.82, 13.72 / 13.96, 19.24 / 19.4, 13.84 / 13.88.
      __nanosleep(300);
      const int tile = tile_of(pair), nb = tile / p.tiles_m;
      int lo, hi;
      slab_range(pair - tile * S, lo, hi);
      for (int kt = lo; kt < hi && kt < kt_main && *ahead_done == 0; ++kt) {
        if (elect_one()) {
          tma_prefetch_2d(&tmB, kt * 128, nb * BN + static_cast<int>(rank) * C::B_ROWS);
          if (rank == 0) tma_prefetch_2d(&tmSFB, 0, nb * (BN / 128) * k_groups4 + kt * 4);
        }
        __syncwarp();
        __nanosleep(40);
      }
    }
    pdl_wait();
    for (int w = pair; w < total_work && ok; w += num_pairs, ++tcount) {
      const int tile = tile_of(w), split = SK ? w - tile * S : 0;
      const int mb = tile % p.tiles_m, nb = tile / p.tiles_m;
      const bool half_tile = is_half(w);
      const int cols = half_tile ? BN / 2 : BN;
      const int m0 = (mb * CG + rank) * BM, n0 = nb * BN + (half_tile ? ((w - p.whole_tiles) & 1) * (BN / 2) : 0);
      const uint32_t as = tcount & 1, aph = (tcount >> 1) & 1;
      // stage this tile's per-column affine terms (the previous tile's readers are past the barrier below)
      [[maybe_unused]] bool odd_smooth = false;     // NEXT: some smooth_next of this tile is outside [2^-20, 2^20]
      for (int c = threadIdx.x; c < cols; c += EPI_WARPS * 32) {
        affine[c] = wc != nullptr ? as_f32<OutT>(wc[n0 + c]) : 1.0f;
        affine[BN + c] = bias != nullptr ? as_f32<OutT>(bias[n0 + c]) : 0.0f;
        if constexpr (NEXT) {
          const float sv = as_f32<OutT>(static_cast<const OutT*>(p.smooth_next)[n0 + c]);
          affine[2 * BN + c] = -sv;
          affine[3 * BN + c] = __frcp_rn(sv);
          odd_smooth |= !(sv >= 9.5367431640625e-07f && sv <= 1048576.0f);      // also zero, negative, NaN
        }
      }
      // NEXT: the tile divides with __fdiv_rn if any of its columns asks for it (the same verdict in all warps)
      [[maybe_unused]] bool tile_fdiv = false;
      if constexpr (NEXT) {
        uint32_t any_odd;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
            "bar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(any_odd) : "r"(odd_smooth ? 1u : 0u), "n"(EPI_WARPS * 32) : "memory");
        tile_fdiv = any_odd != 0;
      } else {
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
      }
      // One strip: 64 columns from column cbase of the tile, the 64 accumulator values of this lane's row in v.
      // STAGED: y through shared memory (the TP form's strips; the last tile's, see below).
      auto strip = [&](uint32_t (&v)[64], int cbase, [[maybe_unused]] uint8_t* buf, auto staged) {
        constexpr bool STAGED = decltype(staged)::value;
        if constexpr (TP) {
          // the TMA store that last read this warp's buffer must be done with it
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
        }
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          const float4* wc4 = reinterpret_cast<const float4*>(affine + cbase + hc * 32);
          const float4* bs4 = reinterpret_cast<const float4*>(affine + BN + cbase + hc * 32);
          uint32_t o[16];
          [[maybe_unused]] float2 qf[16];     // NEXT: the 32 values of this half strip
          [[maybe_unused]] uint32_t qcodes[4], qscales[2];
          // the four fp32 results of columns 4 i .. 4 i + 3 of this half strip
          auto affine_at = [&](int i, float& a0, float& a1, float& a2, float& a3) {
            a0 = __uint_as_float(v[hc * 32 + 4 * i]); a1 = __uint_as_float(v[hc * 32 + 4 * i + 1]);
            a2 = __uint_as_float(v[hc * 32 + 4 * i + 2]); a3 = __uint_as_float(v[hc * 32 + 4 * i + 3]);
            if (wc != nullptr) {
              const float4 w4 = wc4[i];
              a0 = __fmul_rn(a0, w4.x); a1 = __fmul_rn(a1, w4.y); a2 = __fmul_rn(a2, w4.z); a3 = __fmul_rn(a3, w4.w);
            }
            if (bias != nullptr) {
              const float4 b4 = bs4[i];
              a0 = __fadd_rn(a0, b4.x); a1 = __fadd_rn(a1, b4.y); a2 = __fadd_rn(a2, b4.z); a3 = __fadd_rn(a3, b4.w);
            }
          };
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float a0, a1, a2, a3;
            affine_at(i, a0, a1, a2, a3);
            o[2 * i] = pack2f<OutT>(a0, a1);
            o[2 * i + 1] = pack2f<OutT>(a2, a3);
            if constexpr (NEXT) {
              qf[2 * i] = make_float2(a0, a1);
              qf[2 * i + 1] = make_float2(a2, a3);
            }
          }
          if constexpr (NEXT) {
            const int e4 = (cbase + hc * 32) / 4;
            next_two_groups(qf, reinterpret_cast<const float4*>(affine + 2 * BN) + e4, reinterpret_cast<const float4*>(affine + 3 * BN) + e4, scale_lut,
                            tile_fdiv, qcodes, qscales);
          }
          if constexpr (NEXT) {
            if (ok) {
              // this thread's row: 32 columns = 16 code bytes and two scale bytes
              const uint32_t row = static_cast<uint32_t>(m0 + quarter * 32 + lane);
              const uint32_t col = static_cast<uint32_t>(n0 + cbase + hc * 32);
              *reinterpret_cast<uint4*>(p.qout + static_cast<size_t>(row) * (p.N >> 1) + (col >> 1)) =
                  make_uint4(qcodes[0], qcodes[1], qcodes[2], qcodes[3]);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint32_t gcol = (col >> 4) + h;
                p.oscales[static_cast<size_t>(gcol) * p.M + row] = static_cast<uint8_t>(qscales[h]);
                if (p.oscales_swz != nullptr) p.oscales_swz[sf_swizzled_offset(row, gcol, p.N >> 4)] = static_cast<uint8_t>(qscales[h]);
              }
            }
          }
          if constexpr (STAGED) {
            // row `lane` of the strip: 16-byte chunks hc*4 .. hc*4+3, XOR-swizzled like the TMA box
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t chunk = static_cast<uint32_t>(hc * 4 + i) ^ static_cast<uint32_t>(lane & 7);
              *reinterpret_cast<uint4*>(buf + lane * 128 + chunk * 16) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            }
          } else {
            // Straight from the registers, whole 32-byte sectors: by TMA from shared memory the strips of the eight
            // warps, all ready at once, held up the operand loads behind them in the same engine for some 500 cycles,
            // twice a tile (4352 x 3840 -> 3072 28.2 -> 26.6 us, -> 15360 110.9 -> 108.1, x 15360 96.6 -> 95.5).
            OutT* dst = static_cast<OutT*>(p.y) + static_cast<size_t>(m0 + quarter * 32 + lane) * p.N + n0 + cbase + hc * 32;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (p.y_wide) {
                st_global_v8(dst + 16 * i, o + 8 * i);
              } else {
                *reinterpret_cast<uint4*>(dst + 16 * i) = make_uint4(o[8 * i], o[8 * i + 1], o[8 * i + 2], o[8 * i + 3]);
                *reinterpret_cast<uint4*>(dst + 16 * i + 8) = make_uint4(o[8 * i + 4], o[8 * i + 5], o[8 * i + 6], o[8 * i + 7]);
              }
            }
          }
        }
        if constexpr (STAGED && !TP) {
          // The CTA's last tile, whose stores nothing hides: out of the ring, which is free by now, eight lanes a row, so that an
          // instruction touches 4 lines instead of 32 (an SM takes a line in some two cycles: the last stores of a
          // 256-column tile ended 1.4 us earlier).  256 x 3840 -> 3072 6.2 -> 6.0 us, 1003 x 3840 -> 3072 9.8 -> 9.4,
          // 4352 x 3840 -> 3072 28.7 -> 28.2, 4352 x 3840 -> 15360 126.3 -> 125.6.
          __syncwarp();
          OutT* dst = static_cast<OutT*>(p.y) + static_cast<size_t>(m0 + quarter * 32 + (lane >> 3)) * p.N + n0 + cbase + (lane & 7) * 8;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = 4 * i + (lane >> 3);
            const uint4 t = *reinterpret_cast<const uint4*>(buf + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
            *reinterpret_cast<uint4*>(dst + static_cast<size_t>(4 * i) * p.N) = t;
          }
        }
        if constexpr (TP) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&maps.y, buf, p.col0 + n0 + cbase, m0 + quarter * 32);
            // the same strip into every peer's matrix: the copy engine sends it over NVLink while the warp goes on
            for (int d = 0; d < p.n_peers; ++d) tma_store_2d(&maps.m[d], buf, p.col0 + n0 + cbase, m0 + quarter * 32);
            tma_store_commit();
          }
        }
      };
      if (!mbar_wait(&acc_full[as], aph, ctx, kDevWaitAcc, tcount)) ok = false;
      tc_fence_after_sync();
      const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
#pragma unroll 1
      for (int q = 0; q < cols / 128; ++q) {
      // A 256-column tile's shared half first: the next tile is waiting for those columns.
      const int half = C::SHARED_ACC && !half_tile ? (q == 0 ? 1 - static_cast<int>(as) : static_cast<int>(as)) : 0;
      const int cbase = half * 128 + chalf * 64;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + as * 128 + cbase;
      // Drain: the strip goes to registers in one burst, its columns are handed back at once, and only then do the
      // affine, the packing and the store happen.
      uint32_t v[64];
      tmem_ld_32x32_x64(taddr, v);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (w + num_pairs < total_work) {
        if (lane == 0) {
          uint64_t* bar = (C::SHARED_ACC && q == 0) ? acc_shared : &acc_empty[as];
          if constexpr (CG == 2) mbar_arrive_cluster_relaxed(bar, leader); else mbar_arrive(bar);
        }
      } else if (q == cols / 128 - 1 && SK != kClusterSplit) {
        // the last accumulator is in registers: nothing is left to hand back, and the tensor memory may go
        leave();
        drained = true;
      }
      bool finish = true;                       // this CTA writes the tile's rows of y
      if constexpr (SK == kWorkspaceSplit) {
        if (S > 1) {
          // Each thread parks its 16 float4s at [j][thread] of the CTA's partial tile
          // (consecutive threads, consecutive 16 bytes) and later reads the same places of the other
          // partials, so no thread ever needs another thread's accumulator values.
          static_assert(BN == 128, "a thread parks one strip");
          constexpr int kVec = 16;
          constexpr int kTileVec = BM * BN / 4;
          const int tid = threadIdx.x;
          float4* mine = p.ws_partials + static_cast<size_t>(tile * S + split) * kTileVec;
          const uint32_t* vf = v;
#pragma unroll
          for (int j = 0; j < kVec; ++j)
            __stcg(mine + j * (EPI_WARPS * 32) + tid,
                   make_float4(__uint_as_float(vf[4 * j]), __uint_as_float(vf[4 * j + 1]), __uint_as_float(vf[4 * j + 2]),
                               __uint_as_float(vf[4 * j + 3])));
          __threadfence();
          asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
          if (tid == 0) *sk_ticket = atomicAdd(p.ws_tickets + tile, 1u);
          asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
          finish = *sk_ticket == static_cast<uint32_t>(S - 1);
          if (finish) {
            __threadfence();
            // Partial sp is added as a whole before partial sp + 1 is looked at: one round trip to L2
            // per partial with all of a thread's loads in flight together, and the same order of
            // additions whatever order the CTAs finished in.
            const float4* first = p.ws_partials + static_cast<size_t>(tile * S) * kTileVec + tid;
            uint32_t* vw = v;
#pragma unroll
            for (int j = 0; j < kVec; ++j) {
              const float4 t = __ldcg(first + j * (EPI_WARPS * 32));
              vw[4 * j] = __float_as_uint(t.x); vw[4 * j + 1] = __float_as_uint(t.y);
              vw[4 * j + 2] = __float_as_uint(t.z); vw[4 * j + 3] = __float_as_uint(t.w);
            }
#pragma unroll 1
            for (int sp = 1; sp < S; ++sp) {
              const float4* part = first + static_cast<size_t>(sp) * kTileVec;
#pragma unroll
              for (int h = 0; h < kVec; h += 8) {
                float4 t[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) t[j] = __ldcg(part + (h + j) * (EPI_WARPS * 32));
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  vw[4 * (h + j)] = __float_as_uint(__uint_as_float(vw[4 * (h + j)]) + t[j].x);
                  vw[4 * (h + j) + 1] = __float_as_uint(__uint_as_float(vw[4 * (h + j) + 1]) + t[j].y);
                  vw[4 * (h + j) + 2] = __float_as_uint(__uint_as_float(vw[4 * (h + j) + 2]) + t[j].z);
                  vw[4 * (h + j) + 3] = __float_as_uint(__uint_as_float(vw[4 * (h + j) + 3]) + t[j].w);
                }
              }
            }
            if (tid == 0) p.ws_tickets[tile] = 0u;      // every split has drawn its ticket: ready for the next launch
          }
        }
      }
      if constexpr (SK == kClusterSplit) {
        // The CTA's partial tile, 128 rows of 128 fp32, into the ring (all its loads have been consumed); 16-byte slots
        // XOR-swizzled by the row, so that neither these stores nor the sums below meet a bank conflict.
        float4* part = reinterpret_cast<float4*>(smem);
        const int row = quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          part[row * 32 + ((chalf * 16 + j) ^ (row & 7))] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                                     __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        finish = false;
      }
      if constexpr (TP) {
        if (finish) strip(v, cbase, store_bufs + warp * STORE_BUF_BYTES, std::true_type{});      // this warp's staging strip
      } else if (finish) {
        if (w + num_pairs < total_work) strip(v, cbase, nullptr, std::false_type{});
        else strip(v, cbase, smem + (q * EPI_WARPS + warp) * STORE_BUF_BYTES, std::true_type{});
      }
      }
      // affine[] may be overwritten after this barrier; it also makes the eight warps agree on whether to go on
      uint32_t any_failed;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.eq.u32 p, %1, 0;\n\t"
          "bar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
          : "=r"(any_failed) : "r"(ok ? 1u : 0u), "n"(EPI_WARPS * 32) : "memory");
      ok = any_failed == 0;
    }
    if (!drained && SK != kClusterSplit) leave();
    if constexpr (TP) {
      if (lane == 0) tma_store_wait_all<0>();   // global writes of this warp are complete before the CTA ends
      __syncwarp();
    }
  }

  if constexpr (SK == kClusterSplit) {
    // ------------------------------ split-K sums (every thread of the cluster) ------------------------------
    // The cluster's S pairs hold partial tiles; of the 128 rows of either side, pair i sums and writes out rows
    // [128 i / S, 128 (i + 1) / S), its own part first and then the other pairs' in turn: a fixed order for every element,
    // and no two pairs ask the same one at the same time.  A warp takes a row at a time, a lane four of its columns: with
    // 512 consecutive bytes per load 2 / 4 pairs take 3400 / 4200 cycles for it (lanes 32 bytes apart 4900 / 6800; the
    // copy engine pushing the same bytes into the owners' rings measured 0.1 us more).
    static_assert(CG == 2 && BN == 128 && !NEXT && !TP && C::STAGES * C::STAGE_BYTES >= BM * BN * 4, "cluster split");
    __syncwarp();
    tc_fence_before_sync();
    cluster_sync_all();
    if (warp == EPI_WARPS + 1 && *abort_flag == 0) { free_tmem(); tmem_held = false; }
    if (warp < EPI_WARPS && *abort_flag == 0) {
      const int tile = pair / S, me = static_cast<int>(cta >> 1);
      const int m0 = ((tile % p.tiles_m) * CG + rank) * BM, n0 = tile / p.tiles_m * BN;
      const int row_lo = me * BM / S, row_hi = (me + 1) * BM / S;
      const float4 w4 = reinterpret_cast<const float4*>(affine)[lane], b4 = reinterpret_cast<const float4*>(affine + BN)[lane];
      const bool has_wc = p.wc != nullptr, has_bias = p.bias != nullptr;
      const float4* part = reinterpret_cast<const float4*>(smem);
      constexpr int RB = 8;                                         // rows of a warp in flight
      for (int row0 = row_lo + warp; row0 < row_hi; row0 += EPI_WARPS * RB) {
        float4 acc[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int row = row0 + k * EPI_WARPS;
          if (row < row_hi) acc[k] = part[row * 32 + (lane ^ (row & 7))];
        }
#pragma unroll 1
        for (int j = 1; j < S; ++j) {
          const int r = me + j;
          const uint32_t from = map_to_cta(smem_u32(part), 2u * static_cast<uint32_t>(r < S ? r : r - S) + rank);
          float4 t[RB];
#pragma unroll
          for (int k = 0; k < RB; ++k) {
            const int row = row0 + k * EPI_WARPS;
            if (row < row_hi) t[k] = ld_cluster_f4(from + (row * 32 + (lane ^ (row & 7))) * 16);
          }
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if (row0 + k * EPI_WARPS < row_hi) { acc[k].x += t[k].x; acc[k].y += t[k].y; acc[k].z += t[k].z; acc[k].w += t[k].w; }
        }
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int row = row0 + k * EPI_WARPS;
          if (row < row_hi) {
            float4 f = acc[k];
            if (has_wc) f = make_float4(__fmul_rn(f.x, w4.x), __fmul_rn(f.y, w4.y), __fmul_rn(f.z, w4.z), __fmul_rn(f.w, w4.w));
            if (has_bias) f = make_float4(__fadd_rn(f.x, b4.x), __fadd_rn(f.y, b4.y), __fadd_rn(f.z, b4.z), __fadd_rn(f.w, b4.w));
            *reinterpret_cast<uint2*>(static_cast<OutT*>(p.y) + static_cast<size_t>(m0 + row) * p.N + n0 + 4 * lane) =
                make_uint2(pack2f<OutT>(f.x, f.y), pack2f<OutT>(f.z, f.w));
          }
        }
      }
    }
  }

  // ------------------------------ teardown ------------------------------
  // What a CTA holds is given back as early as it can be, so that only the stores of the last strips lie between the last
  // accumulator and the end: a pair's barrier (the partner may still signal this one's barriers or read its shared memory;
  // relaxed, for nothing that was written has to be visible to it) completes, and tensor memory is freed, while those
  // stores are on their way.  (A chain of kernels showed 0.27 us for freeing tensor memory and 0.2 to 0.36 for the barrier
  // at the end of each.  With the quantizer's set-up and end done likewise, both kernels from a stream: 256 x 3840 -> 3072
  // 12.7 -> 12.4 us, 64 x 128 -> 128 in a graph 6.5 -> 6.1.)
  if constexpr (SK == kClusterSplit) leave();
  else if (warp >= EPI_WARPS) leave();
  __syncwarp();
  if constexpr (CG == 2) cluster_wait();
  else if (warp == EPI_WARPS + 1) asm volatile("bar.sync 2, %0;" ::"n"((EPI_WARPS + 1) * 32) : "memory");
  if (*abort_flag) {
    // give copies that were already in flight time to land before the CTA's memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) { __nanosleep(1000); }
  }
  if (warp == EPI_WARPS + 1 && tmem_held) free_tmem();
}

}  // namespace gemm

bool gemm_supported(int M, int N, int K, int R) {
  return M > 0 && N > 0 && K > 0 && M % 128 == 0 && N % 128 == 0 && K % 64 == 0 && R >= 0 && R % 16 == 0;
}

// 256-column pair tiles of a last round that leaves at least half of the pairs without one: they are worked on as two halves,
// and the round takes 0.65 of a tile's time, the same sums in the same order.  Sustained, bf16, rank 64, 74 pairs:
// 1536 x 3840 -> 3840 (16 tiles in the second round) 15.2 -> 14.2 us, 1024 x 3840 -> 5888 (18; 128-column tiles before) 16.2 ->
// 15.0, 1280 x 6144 -> 5120 (26) 24.2 -> 22.7, 2048 x 512 -> 3072 (22) 7.9 -> 7.6, 4352 x 15360 -> 3840 (33 in the fourth)
// 95.3 -> 93.6 in short runs, 109.8 -> 108.0 at the power cap.
static int gemm_halved_tiles(long long tiles, long long pairs) {
  const long long left = tiles % pairs;
  return tiles > pairs && 2 * left <= pairs ? static_cast<int>(left) : 0;
}

template <int CG, int BN, typename OutT, int SK = gemm::kNoSplit, bool NEXT = false, bool TP = false, bool HALVES = false>
static int launch_gemm_t(const void* act, const void* wgt, const void* sfa, const void* sfb, const void* la,
                         const void* lu, const void* lu_f16, const void* wc, const void* bias, void* y, int M, int N,
                         int K, int R, const GemmTp& tp, cudaStream_t stream, int splits = 1) {
  using C = gemm::Cfg<CG, BN, NEXT, TP>;
  constexpr bool kBf16 = std::is_same<OutT, __nv_bfloat16>::value;
  constexpr int kBoxRows = HALVES ? C::B_ROWS / 2 : C::B_ROWS;
  CUtensorMap tmA, tmB, tmLA, tmLU, tmSFA, tmSFB;
  typename std::conditional<kBf16, gemm::LoraF16Maps, gemm::NoMaps>::type lora_f16;
  int rc;
  const uint64_t atoms_k = K / 64;
  if ((rc = make_tmap_2d(&tmSFA, sfa, 4, (M / 128) * atoms_k, 128, 512, 4, 128, kTmapSwizzleNone)) != SVDQ_OK) return rc;
  if ((rc = make_tmap_2d(&tmSFB, sfb, 4, (N / 128) * atoms_k, 128, 512, 4, 128, kTmapSwizzleNone)) != SVDQ_OK) return rc;
  if ((rc = make_tmap_2d(&tmA, act, 1, M, K / 2, K / 2, gemm::BM, 128, kTmapSwizzle128)) != SVDQ_OK) return rc;
  if ((rc = make_tmap_2d(&tmB, wgt, 1, N, K / 2, K / 2, kBoxRows, 128, kTmapSwizzle128)) != SVDQ_OK) return rc;
  if (R > 0) {
    const uint64_t la_rows = static_cast<uint64_t>(M) * (std::is_same<OutT, __nv_bfloat16>::value ? 2 : 1);
    if ((rc = make_tmap_2d(&tmLA, la, 2, la_rows, R, static_cast<uint64_t>(R) * 2, gemm::BM, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
    if ((rc = make_tmap_2d(&tmLU, lu, 2, N, R, static_cast<uint64_t>(R) * 2, kBoxRows, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
  } else {
    tmLA = tmA; tmLU = tmB;
  }
  gemm::Params p;
  p.la_flags = nullptr;
  if constexpr (kBf16) {
    lora_f16.la = tmLA; lora_f16.lu = tmLU;
    if (R > 0 && lu_f16 != nullptr) {
      // bf16 form of lora_act: planes hi, lo, fp16, then the per-32-row flag words
      const size_t plane = static_cast<size_t>(M) * R;
      const void* la_f16 = static_cast<const uint16_t*>(la) + 2 * plane;
      if ((rc = make_tmap_2d(&lora_f16.la, la_f16, 2, M, R, static_cast<uint64_t>(R) * 2, gemm::BM, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
      if ((rc = make_tmap_2d(&lora_f16.lu, lu_f16, 2, N, R, static_cast<uint64_t>(R) * 2, kBoxRows, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
      p.la_flags = lora16_flags(la, plane);
    }
  }
  p.wc = wc; p.bias = bias;
  p.M = M; p.N = N; p.K = K; p.R = R;
  p.tiles_m = M / (gemm::BM * CG); p.tiles_n = N / BN;
  p.y = y;
  p.y_wide = reinterpret_cast<uintptr_t>(y) % 32 == 0 ? 1 : 0;
  p.col0 = tp.col0; p.n_peers = tp.n_peers;
  typename std::conditional<TP, gemm::PeerMaps, gemm::NoMaps>::type maps;
  if constexpr (TP) {
    // the [M, y_ld] matrix this launch fills N columns of, here and on the peers
    const uint64_t pitch = static_cast<uint64_t>(tp.y_ld) * 2;
    if ((rc = make_tmap_2d(&maps.y, y, 2, M, tp.y_ld, pitch, 32, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
    for (int d = 0; d < 7; ++d) maps.m[d] = maps.y;
    for (int d = 0; d < tp.n_peers; ++d)
      if ((rc = make_tmap_2d(&maps.m[d], tp.y_peer[d], 2, M, tp.y_ld, pitch, 32, 64, kTmapSwizzle128)) != SVDQ_OK) return rc;
  }
  p.splits = SK != gemm::kNoSplit ? splits : 1;
  p.interleave = tp.interleave;
  {
    const int kt_main = (K + gemm::BK - 1) / gemm::BK, ls = (R + 63) / 64;
    p.stride1 = ls > 0 ? (kt_main + ls) / ls : 1;
    p.stride2 = ls > 0 ? (kt_main + 2 * ls) / (2 * ls) : 1;
  }
  p.ws_tickets = static_cast<unsigned int*>(tp.ws);
  p.ws_partials = tp.ws != nullptr ? reinterpret_cast<float4*>(static_cast<uint8_t*>(tp.ws) + kSplitTicketBytes) : nullptr;
  p.smooth_next = tp.smooth_next;
  p.qout = static_cast<uint8_t*>(tp.qout);
  p.oscales = static_cast<uint8_t*>(tp.oscales);
  p.oscales_swz = static_cast<uint8_t*>(tp.oscales_swz);
  auto kern = gemm::gemm_w4a4_kernel<CG, BN, OutT, SK, NEXT, TP, HALVES>;
  // the attribute is per device: remember which devices of this process have it
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SVDQ_ERR_CUDA;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) return SVDQ_ERR_LAUNCH;
    if (SK == gemm::kClusterSplit && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return SVDQ_ERR_LAUNCH;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int max_pairs = sm_count() / CG;
  p.whole_tiles = p.tiles_m * p.tiles_n;
  if (HALVES) p.whole_tiles -= gemm_halved_tiles(p.whole_tiles, max_pairs);
  const int tiles = p.tiles_m * p.tiles_n * p.splits;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pairs * CG, 1, 1);
  cfg.blockDim = dim3(gemm::NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = SK == gemm::kClusterSplit ? CG * splits : CG; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kern, tmA, tmB, tmLA, tmLU, tmSFA, tmSFB, lora_f16, maps, p) != cudaSuccess) return SVDQ_ERR_LAUNCH;
  return SVDQ_OK;
}

template <typename OutT, bool NEXT, bool TP>
static int launch_gemm_dt(int cg, int bn, const void* act, const void* wgt, const void* sfa, const void* sfb,
                          const void* la, const void* lu, const void* lu_f16, const void* wc, const void* bias, void* y,
                          int M, int N, int K, int R, const GemmTp& tp, cudaStream_t stream) {
  if constexpr (!TP) {
    if (cg == 2 && bn == 256 && gemm_halved_tiles(static_cast<long long>(M / 256) * (N / 256), sm_count() / 2) > 0)
      return launch_gemm_t<2, 256, OutT, gemm::kNoSplit, NEXT, TP, true>(act, wgt, sfa, sfb, la, lu, lu_f16, wc, bias, y, M, N, K, R, tp, stream);
  }
  if (cg == 2 && bn == 256) return launch_gemm_t<2, 256, OutT, gemm::kNoSplit, NEXT, TP>(act, wgt, sfa, sfb, la, lu, lu_f16, wc, bias, y, M, N, K, R, tp, stream);
  if (cg == 2 && bn == 128) return launch_gemm_t<2, 128, OutT, gemm::kNoSplit, NEXT, TP>(act, wgt, sfa, sfb, la, lu, lu_f16, wc, bias, y, M, N, K, R, tp, stream);
  if (cg == 1 && bn == 256) return launch_gemm_t<1, 256, OutT, gemm::kNoSplit, NEXT, TP>(act, wgt, sfa, sfb, la, lu, lu_f16, wc, bias, y, M, N, K, R, tp, stream);
  return launch_gemm_t<1, 128, OutT, gemm::kNoSplit, NEXT, TP>(act, wgt, sfa, sfb, la, lu, lu_f16, wc, bias, y, M, N, K, R, tp, stream);
}

// Clusters of `ctas` CTAs of the cluster-split kernel that the current device can hold at once, asked for when first
// needed (all instantiations have the same block and shared-memory size).
static int gemm_max_clusters(int ctas) {
  static int caps[64][17];                          // value + 2; 0: not asked yet
  int dev = 0;
  if (ctas < 1 || ctas > 16 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (caps[dev][ctas] == 0) {
    using C = gemm::Cfg<2, 128>;
    auto kern = gemm::gemm_w4a4_kernel<2, 128, __half, gemm::kClusterSplit>;
    int n = -1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64 * ctas, 1, 1);
    cfg.blockDim = dim3(gemm::NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = -1;
    }
    caps[dev][ctas] = n + 2;
  }
  return caps[dev][ctas] - 2;
}

// Pairs that share each 256 x 128 tile's K loop within a cluster (1: no split).  A pair streams a slab in about 0.17 us;
// the cluster's sums and its barriers cost about 2.7 us, which n slabs repay from n (1 - 1 / S) = 18 on (256 rows, sustained:
// 3072 columns, K = 3840 / 10240 with S = 2 6.6 -> 7.6 / 10.5 -> 10.0 us; 3840 columns, K = 15360, S = 2 16.1 -> 14.1;
// 1792 columns, K = 9408, S = 4 12.1 -> 8.8; 1280 columns, K = 11520, S = 4 11.2 -> 8.4; 1024 columns, K = 5120, S = 4
// 7.1 -> 7.0).  At least six slabs per pair; all clusters resident at once.
int gemm_cluster_split(int M, int N, int K, int R) {
  if (!gemm_supported(M, N, K, R) || M % 256 != 0) return 1;
  const long long tiles = static_cast<long long>(M / 256) * (N / 128);
  const int n = (K + gemm::BK - 1) / gemm::BK + (R + 63) / 64;
  for (int s = 8; s >= 2; --s)
    if (n >= 6 * s && n * (s - 1) >= 18 * s && tiles * 2 * s <= sm_count() && tiles <= gemm_max_clusters(2 * s)) return s;
  return 1;
}

// Workspace form.  The library runs this plan for row counts that are an odd multiple of 128; for whole 256-row tiles
// (split within clusters above) it only tells a caller who forces the form how much room that takes.
// Split-K plan for a problem with few tiles: 128 x 128 tiles, each tile's slabs shared by S CTAs that
// all run at once (tiles * S <= SMs).  One CTA streams a tile's slabs at about 0.235 us each however
// few tiles there are (32 KB per slab through one SM's load path), so with a few dozen tiles most
// SMs idle and the run time is one tile's K loop.  Splitting costs about 2.8 + 0.5 S us (partials to
// L2, a fence, the ticket, one read per partial), 12 + 2 S slabs, against the n (1 - 1 / S) slabs that
// it saves.  Plain / S = 2 / 3 / 4 in us, 128 rows x 3072 columns, K = 3840 7.5 / 9.4 / 9.5 / 9.8,
// K = 6144 9.4 / 10.4 / 10.0 / 10.4, K = 7680 10.9 / 11.2 / 10.6 / 10.7, K = 10240 13.2 / 12.4 / 11.5 / 11.6,
// K = 15360 18.0 / 15.0 / 13.2 / 12.6; 384 rows, which fit two CTAs a tile, K = 7680 11.2 / 11.8, K = 10240
// 13.6 / 13.0.  Returns S (1 = no split).
int gemm_split_plan(int M, int N, int K, int R) {
  if (!gemm_supported(M, N, K, R)) return 1;
  const long long tiles = static_cast<long long>(M / 128) * (N / 128);
  const int slabs = (K + gemm::BK - 1) / gemm::BK, n = slabs + (R + 63) / 64;
  const int sms = sm_count();
  if (tiles * 2 > sms || tiles > kSplitMaxTiles) return 1;
  int best = 1;
  double best_cost = 0.0;                         // of a split, in slabs, over not splitting
  for (int s = 2; s <= 4 && tiles * s <= sms && s <= slabs / 6; ++s) {      // at least six slabs per split
    const double cost = 12.0 + 2.0 * s - n * (1.0 - 1.0 / s);
    if (cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

size_t gemm_split_workspace_bytes(int M, int N, int K, int R) {
  const int s = gemm_split_plan(M, N, K, R);
  if (s < 2) return 0;
  return kSplitTicketBytes + static_cast<size_t>(M / 128) * (N / 128) * s * (128 * 128 * 4);
}

// Default LoRA schedule: after the main slabs.  Same-box A/B on the four benchmark shapes: interleaved
// 27.1 / 121.0 / 102.4 / 55.0 us against 27.4 / 120.5 / 102.6 / 55.0 us at the end (within run-to-run noise; the
// reference measured +0.5 % for its interleave, docs/gotchas/cute_dsl.md:368-377).
constexpr int kLoraInterleaveDefault = 0;

// variant: 0 = choose; 128 / 256 = one CTA per tile with that N tile; 2128 / 2256 = CTA pairs (256-row tiles);
// 10000 * S + 128 = split-K with S CTAs per 128 x 128 tile (needs the workspace); 10000 * S + 2128 = split-K with the S
// pairs of a cluster per 256 x 128 tile
int launch_gemm_w4a4(const void* act, const void* wgt, const void* ascales_swz, const void* wscales_swz,
                     const void* lora_act16, const void* lora_up, const void* lora_up_f16, const void* wcscales,
                     const void* bias, void* y, int M, int N, int K, int R, int dtype, int variant,
                     const GemmTp& tp_in, cudaStream_t stream) {
  if (!gemm_supported(M, N, K, R)) return SVDQ_ERR_SHAPE;
  // LoRA schedule bits of `variant`: interleaved, end-grouped, or (neither) the library's default
  GemmTp tp = tp_in;
  if (variant & SVDQ_GEMM_LORA_INTERLEAVE) tp.interleave = 1;
  else if (variant & SVDQ_GEMM_LORA_AT_END) tp.interleave = 0;
  else tp.interleave = kLoraInterleaveDefault;
  const bool may_split = (variant & kGemmNoSplit) == 0;
  variant &= ~(SVDQ_GEMM_LORA_INTERLEAVE | SVDQ_GEMM_LORA_AT_END | kGemmNoSplit);
  if (tp.n_peers < 0 || tp.n_peers > 7) return SVDQ_ERR_SHAPE;
  if (tp.y_ld > 0 && (tp.col0 < 0 || tp.col0 % 64 != 0 || tp.col0 + N > tp.y_ld || tp.y_ld % 8 != 0)) return SVDQ_ERR_SHAPE;
  if (tp.y_ld <= 0 && tp.n_peers > 0) return SVDQ_ERR_SHAPE;
  const bool next = tp.smooth_next != nullptr;
  if (next && (tp.qout == nullptr || tp.oscales == nullptr || tp.y_ld > 0 || variant >= 10000)) return SVDQ_ERR_UNSUPPORTED;
  int cg, bn;
  if (!next && tp.y_ld <= 0 && ((variant == 0 && may_split) || (variant >= 10000 && variant % 10000 == 2128))) {
    // split-K within clusters: planned, or forced by the caller
    const int s = variant == 0 ? gemm_cluster_split(M, N, K, R) : variant / 10000;
    if (variant >= 10000) {
      const long long tiles = static_cast<long long>(M / 256) * (N / 128);
      if (M % 256 != 0 || s < 2 || s > 8 || s > (K + gemm::BK - 1) / gemm::BK || tiles > gemm_max_clusters(2 * s)) return SVDQ_ERR_UNSUPPORTED;
    }
    if (s >= 2) {
      if (dtype == SVDQ_DTYPE_F16)
        return launch_gemm_t<2, 128, __half, gemm::kClusterSplit>(act, wgt, ascales_swz, wscales_swz, lora_act16, lora_up, nullptr, wcscales, bias, y, M, N, K, R, tp, stream, s);
      if (dtype == SVDQ_DTYPE_BF16)
        return launch_gemm_t<2, 128, __nv_bfloat16, gemm::kClusterSplit>(act, wgt, ascales_swz, wscales_swz, lora_act16, lora_up, lora_up_f16, wcscales, bias, y, M, N, K, R, tp, stream, s);
      return SVDQ_ERR_DTYPE;
    }
  }
  if (!next && (variant == 0 || (variant >= 10000 && variant % 10000 == 128))) {
    // split-K: planned (variant 0, plain form, workspace large enough) or forced by the caller
    int s = 1;
    if (variant == 0 && may_split && M % 256 != 0 && tp.y_ld <= 0 && tp.ws != nullptr) {
      s = gemm_split_plan(M, N, K, R);
      if (s >= 2 && tp.ws_bytes < gemm_split_workspace_bytes(M, N, K, R)) s = 1;
    } else if (variant >= 10000) {
      s = variant / 10000;
      const long long tiles = static_cast<long long>(M / 128) * (N / 128);
      if (variant % 10000 != 128 || s < 2 || s > kSplitMax || tiles > kSplitMaxTiles || tp.ws == nullptr || tp.y_ld > 0 ||
          s > (K + gemm::BK - 1) / gemm::BK || tiles * s > sm_count() ||
          tp.ws_bytes < kSplitTicketBytes + static_cast<size_t>(tiles) * s * (128 * 128 * 4))
        return SVDQ_ERR_UNSUPPORTED;
    }
    if (s >= 2) {
      if (dtype == SVDQ_DTYPE_F16)
        return launch_gemm_t<1, 128, __half, gemm::kWorkspaceSplit>(act, wgt, ascales_swz, wscales_swz, lora_act16, lora_up, nullptr, wcscales, bias, y, M, N, K, R, tp, stream, s);
      if (dtype == SVDQ_DTYPE_BF16)
        return launch_gemm_t<1, 128, __nv_bfloat16, gemm::kWorkspaceSplit>(act, wgt, ascales_swz, wscales_swz, lora_act16, lora_up, lora_up_f16, wcscales, bias, y, M, N, K, R, tp, stream, s);
      return SVDQ_ERR_DTYPE;
    }
  }
  if (variant == 0) {
    // Pairs wherever the rows allow them: single CTAs, which load all of B themselves, are slower at every size that
    // both take (256 x 3840 x 3072 6.3 / 7.5 us, 1536 x 3840 x 3840 13.1 / 16.1, 4352 x 3840 x 3072 21.3 / 24.1).
    // The tile's width by the least estimated time, rounds of tiles over the pairs (or SMs) times the relative time of
    // a tile.  A 128-column tile takes more than half of a 256-column one, for it moves more operand bytes per flop:
    // 0.65 of it for a pair (one round at 256 x 15360 x 3840 16.3 / 24.8 us, at 256 x 3840 x 3072 6.3 / 9.2), 0.84 for a
    // single CTA (21.3 / 25.5).  So narrow tiles where both widths take one round, and with pairs where three narrow
    // rounds replace two wide ones of which the second is more than half empty, but not a round that can be halved
    // (gemm_halved_tiles; it counts as a narrow one).  Further up the line is flat: two rounds against one 9.73 / 9.83
    // (1024 x 3840 x 3072), five against three 21.2 / 20.2 (3072 x 3840 x 3840).  The column-sharded form stores
    // through shared memory, which narrow tiles do more often: three rounds against two 14.9 / 14.4 (1536 x 3840 x
    // 3840), 31.6 / 29.4 (4352 x 10240 x 1536).
    cg = M % 256 == 0 ? 2 : 1;
    const long long units = sm_count() / cg;
    double best = 1e30;
    bn = 128;
    for (int b : {256, 128}) {
      if (N % b != 0) continue;
      const long long tiles = static_cast<long long>(M / (128 * cg)) * (N / b);
      double cost = static_cast<double>((tiles + units - 1) / units) * (b == 256 ? 1.0 : tp.y_ld > 0 ? 0.72 : cg == 2 ? 0.65 : 0.84);
      if (b == 256 && cg == 2 && tp.y_ld <= 0 && gemm_halved_tiles(tiles, units) > 0) cost -= 0.35;
      if (cost < best) { best = cost; bn = b; }
    }
  } else if (variant == 128 || variant == 256) {
    cg = 1; bn = variant;
  } else {
    cg = variant / 1000; bn = variant % 1000;
  }
  if ((cg != 1 && cg != 2) || (bn != 128 && bn != 256)) return SVDQ_ERR_UNSUPPORTED;
  if (M % (128 * cg) != 0 || N % bn != 0) return SVDQ_ERR_SHAPE;
  const bool sharded = tp.y_ld > 0;
  auto launch = [&](auto dt) {
    using T = decltype(dt);
    const void* lu16 = std::is_same<T, __half>::value ? nullptr : lora_up_f16;
    auto go = [&](auto next_c, auto tp_c) {
      return launch_gemm_dt<T, decltype(next_c)::value, decltype(tp_c)::value>(cg, bn, act, wgt, ascales_swz, wscales_swz, lora_act16, lora_up, lu16,
                                                                              wcscales, bias, y, M, N, K, R, tp, stream);
    };
    if (next) return go(std::true_type{}, std::false_type{});
    return sharded ? go(std::false_type{}, std::true_type{}) : go(std::false_type{}, std::false_type{});
  };
  if (dtype == SVDQ_DTYPE_F16) return launch(__half{});
  if (dtype == SVDQ_DTYPE_BF16) return launch(__nv_bfloat16{});
  return SVDQ_ERR_DTYPE;
}

}  // namespace svdq
