// Implicit-GEMM convolution on the Blackwell tensor cores (CCT_ALGO_UMMA_3XTF32).
//
// All three contractions of the convolution bridge run on tcgen05.mma (kind::tf32, M = 128, fp32 accumulators in
// tensor memory).  The lowered matrix of the reference (type-1 lowering, one row of k*k*D values per output pixel)
// is never written to global memory: producer threads gather each 128 x 32 tile of it straight from the NCHW
// tensors, splitting every fp32 value into hi = its tf32 part and lo = x - hi on the way.  Three MMAs per k-step
// (hi*hi + hi*lo + lo*hi) recover fp32-level accuracy ("3xTF32"); flops are counted once.  Larger contractions split
// scaled values into two fp16 parts instead, at twice the rate, where the operands' values allow it (operand_scale.cuh).
//
//   forward        Y[pix][o]   = sum_k  Lowered(X)[pix][k] * W[o][k]            (+ bias, optional ReLU)
//   data gradient  dX[q][(d,py,px)] = sum_kk Gathered(dY)[q][kk] * Wd[(d,py,px)][kk]   kk = (filter, jy, jx)
//                  - the inverse lowering (col2im) written as a gather over s x s blocks of input pixels q: every
//                  block sums the taps that touch it inside the accumulator and the epilogue scatters the columns
//                  (depth to space), so there is no atomics and the result is deterministic.
//   weight gradient dW[kk][o]  = sum_pix Lowered(X)[pix][kk] * dY[pix][o]        split over pixel ranges across
//                  CTAs, partial sums to scratch, fixed-order reduction.
//
// gather_conv_kernel serves the forward pass, the data gradient and (lanes = rows of the lowered matrix, dY as the
// pre-split TMA operand) the weight gradient of larger layers: gathered operand in tensor memory, the other operand
// streamed by TMA into swizzled shared memory, warp-specialised roles.  Shorter lowered matrices have their own weight-
// gradient kernels: wgrad_ts_kernel (257 .. 384 rows: dY through tensor memory, the lowered rows staged in shared memory)
// and wgrad_kernel (anything shorter, and the allocation-free entry point: both operands staged in shared memory).
// Every kernel is launched with launch_pdl and calls pdl_wait() before it touches anything but its plan's tables (cct_internal.h).
// Every mbarrier wait is bounded: when it runs out the thread
// sets the context's status word, stops waiting on anything else, and the kernel still frees its tensor memory.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include <cuda.h>

#include "cct_internal.h"
#include "operand_scale.cuh"
#include "umma_ptx.cuh"

namespace {

constexpr int kMaxTapsPerAxis = 15;
// Longest accumulation chain of a weight-gradient partial sum, in k-blocks of 32 pixels.  Measured against a
// double-accumulating CPU reference, AlexNet conv1's dW was off by 7.7e-5 (max-norm relative) with chains of 327
// k-blocks, the error pointing towards zero (truncating accumulate), and it shrinks in proportion to the chain.
constexpr int kMaxChainKblocks = 176;
constexpr uint32_t kPadBit = 0x80000000u;  // never set in a pixel's validity mask: marks padding entries

// One entry per reduction index of a gathered operand: element offset from the pixel's tap origin, and the tap's
// row / column as mask bits.  The tap is in bounds for a pixel iff (pixel_mask & bits) == bits, where bit i (rows) and
// bit 16+j (columns) of the pixel's mask say whether tap row i / tap column j falls inside the gathered plane.
struct alignas(8) MaskTap {
  int off;
  uint32_t bits;
};

// Bits [lo, hi) set; 0 <= lo, hi <= 15.
__device__ __forceinline__ uint32_t bit_range(int lo, int hi) {
  lo = max(lo, 0);
  hi = min(hi, kMaxTapsPerAxis);
  return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// v = ((mask & bits) == bits) ? *p : 0 as straight-line predicated code: written through the compiler, each guarded
// load becomes a branch around the load, and the branch bookkeeping costs more issue slots than the load itself.
__device__ __forceinline__ float ldg_if_bits(const float* p, uint32_t mask, uint32_t bits) {
  float v;
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b32 t;\n\t"
      "and.b32 t, %2, %3;\n\t"
      "setp.eq.u32 q, t, %3;\n\t"
      "mov.f32 %0, 0f00000000;\n\t"
      "@q ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"(mask), "r"(bits));
  return v;
}
// v = ((a & b) == 0) ? *p : 0, same form (a, b: "what is out of bounds here" against "what this entry needs").
__device__ __forceinline__ float ldg_if_clear(const float* p, uint32_t a, uint32_t b) {
  float v;
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b32 t;\n\t"
      "and.b32 t, %2, %3;\n\t"
      "setp.eq.u32 q, t, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\t"
      "@q ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"(a), "r"(b));
  return v;
}
// v = flag ? *p : 0, same form.
__device__ __forceinline__ float ldg_if(const float* p, uint32_t flag) {
  float v;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.u32 q, %2, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\t"
      "@q ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"(flag));
  return v;
}

// if (flag) *p = v, as one predicated st.global.
__device__ __forceinline__ void stg_if(float* p, float v, uint32_t flag) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.u32 q, %2, 0;\n\t"
      "@q st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"(flag)
      : "memory");
}

// ------------------------------------------------------------------------------ gather kernel (forward, dgrad)
//
// Persistent, warp-specialised: one CTA per SM walks over (channel tile, 128-pixel tile) pairs.
//   producers   (4 * SETS warps) thread = one pixel of the tile = one TMEM lane.  Per k-block a thread gathers its
//               32 lowered values, splits them hi/lo and writes them with tcgen05.st into an A slot in tensor memory
//               (sets of four warps; set g takes the k-blocks with running index == g mod SETS, each set covers
//               all 128 lanes).
//   MMA warp    issues the MMAs (see elect_one): A from tensor memory, B from shared memory.
//   TMA warp    one thread streams the pre-split weight tiles (B) into shared memory with TMA (128-byte swizzle).
//   epilogue    (4 warps) tcgen05.ld the finished accumulator, add bias / clamp, store NCHW (or depth-to-space for
//               the strided data gradient); overlaps the next tile's MMAs when two accumulators fit.
// Tensor memory: [accumulator(s) | A slots of 64 columns: 32 hi + 32 lo].
// The tensor core truncates every sum it writes to the accumulator, so an accumulator loses about half a place in the last
// per MMA.  Tiles of at most kCrossCols columns therefore have a second one for the cross terms (lo*hi + hi*lo, a factor of
// 2^11 smaller), which the epilogue adds: one truncation at full magnitude per eight products instead of three.  Wider tiles
// have no tensor memory to spare for it next to their A slots.  Error against 64-bit sums, 5x5, 96 -> 41 channels, positive
// data: forward 3.8e-5 with one accumulator, 1.7e-5 with two; the price is an A slot (two instead of three at 48 and 64
// columns) and a second tcgen05.ld in the epilogue: CaffeNet conv2's data gradient (48 columns) 531 -> 545 us.
// The kernel comes in two shapes.  SETS = 4: sixteen producer warps (four sets of four; set g fills the k-blocks with
// running index == g mod 4), 704 threads, one CTA per SM with all 512 tensor-memory columns.  SETS = 2: eight producer
// warps, 448 threads, 256 columns, two or three A slots, one accumulator - two such CTAs share an SM, so that one CTA's
// hand-overs and epilogue overlap the other's MMAs (CaffeNet conv2's data gradient, 48 columns: 525 us, one CTA with four
// sets 660).
constexpr int kEpiWarps = 4;
__host__ __device__ constexpr int gather_threads(int sets) { return (4 * sets + 2 + kEpiWarps) * 32; }  // 704 or 448
constexpr int kMaxAStages = 4, kMaxAccBufs = 2, kCrossCols = 64;
// Columns of one accumulator buffer: hi*hi and behind it, on narrow tiles, the cross terms.
__host__ __device__ constexpr int acc_columns(int n_pad) { return n_pad <= kCrossCols ? 2 * n_pad : n_pad; }

// Channels per table entry where the gathered tensor's channels per group are a multiple of it.  One table read, one bounds
// test and one branch then serve kRun loads of consecutive channels, and the taps of the same kRun channels follow one
// another, so that they still find their lines in L1 (the channels of two CTAs' tiles all at once would not fit it).
constexpr int kRun = 8;

struct alignas(8) ColEnt {  // one accumulator column -> where it lands in the output
  int off;       // element offset from the pixel's output origin
  short cy, cx;  // displacement of the output pixel (depth-to-space), for the bounds test
};

struct GatherParams {
  const float* in;    // gathered tensor: X (forward) or dY (data gradient)
  float* out;         // Y or dX
  const MaskTap* taps; // [k_pad]
  const ColEnt* cols;  // [n_pad]
  const float* bias;  // indexed by output channel, or null
  int n_pix, q_h, q_w;                 // pixels = batch * q_h * q_w
  int iy_mul, iy_add, ix_mul, ix_add;  // tap origin in the gathered tensor: iy0 = qy*iy_mul + iy_add
  int in_lim;                          // gathered tensor is in_lim x in_lim per channel
  int tap_sign, taps_per_axis;         // tap i of an axis sits at coordinate origin + tap_sign * i
  long long in_batch_stride;
  int in_group_stride;   // elements between the channel blocks of consecutive groups
  int tiles_per_group;   // virtual groups per real group (channel tiles)
  int oy_mul, oy_add, ox_mul, ox_add;  // output origin of a pixel: oy0 = qy*oy_mul + oy_add
  int out_lim, check_out;              // output plane is out_lim x out_lim; check_out: columns may fall outside
  int out_pitch, out_plane;
  long long out_batch_stride;
  int out_group_channels, out_tile_channels;  // output channels per real group / per channel tile
  int n, n_pad, k_pad;     // real / padded accumulator columns per virtual group, padded reduction length of one tile
  int cols_per_channel;    // accumulator columns per output channel: 1, or the block of pixels of the data gradient
  // Split reduction (forward, data gradient): a tile covers k_pad of the reduction, `splits` tiles share an accumulator's
  // place and write raw sums to `partial` [split][vg][n_pad][pix_pad], which gather_reduce_kernel adds in order.
  int splits, pix_pad;
  float* partial;
  int n_pix_tiles, total_tiles;
  int a_stages, b_stages, acc_bufs;
  int tmem_cols;           // tensor-memory columns this CTA allocates: 512, or 256 when two CTAs share an SM
  int n_bias;              // entries of `bias` (all output channels), staged in shared memory
  int lo_row_offset;       // first row of the "lo" half inside the packed-weight tensor map
  int relu;
  // Weight-gradient mode: the TMEM lanes are rows of the lowered matrix (taps), the reduction runs over pixels.
  // `taps` then points to a table in global memory with one entry per pixel (offset of the pixel's tap origin and
  // the set of tap rows / columns that fall outside the plane there), `out` to the split partial sums.
  int wg_mtiles, wg_vgroups;  // tiles = splits x channel tiles x M-tiles (M-tile fastest)
  int wg_rows_pad;            // rows of one split's partial-sum slice (M-tiles * 128)
  int wg_k, wg_kreal;         // kernel size, real rows of the lowered matrix
  // HALF: the scales of the plan's operands, which two of them this contraction has (gathered, packed), the first row of the packed
  // operand in pairs of fp16, and the stages that there is room for then.
  const HalfScales* half;
  int half_row_offset;
  uint16_t acc_cols_half;
  uint8_t half_gathered, half_packed, a_stages_half, b_stages_half, acc_bufs_half;
  uint8_t taps_x;             // taps along a row (taps_per_axis: along a column)
  // A data gradient by tall blocks of pixels is two launches, of which one returns at once: kOnlyHalf takes the tall blocks in pairs of fp16, kOnlyTf32
  // the others.  `bad_geom`: the layer, for values that are not finite.
  uint8_t only;
  struct { uint8_t kernel, stride; short pad, size; int channels, group_channels; } bad_geom;
  int taps_smem;              // entries of `taps` staged in shared memory (0 in weight-gradient mode)
  const float* zero;          // kByRun: what lanes whose tap is out of bounds read
  int run_stride;             // kByRun: elements between consecutive channels of the gathered tensor
  int* status;
};

enum { kAny = 0, kOnlyHalf = 1, kOnlyTf32 = 2 };

// Which tile a persistent CTA works on: channel tile, pixel tile (or M-tile), first k-block, split.
struct TileId {
  int vg, ptile, kb0, split;
};
template <bool WG>
__device__ __forceinline__ TileId decode_tile(const GatherParams& P, int t, int kblocks) {
  TileId id;
  if (!WG) {
    const int r = t / P.n_pix_tiles, vgroups = P.total_tiles / (P.n_pix_tiles * P.splits);
    id.ptile = t - r * P.n_pix_tiles;
    id.split = P.splits == 1 ? 0 : r / vgroups;
    id.vg = r - id.split * vgroups;
    id.kb0 = id.split * kblocks;
  } else {
    const int r = t / P.wg_mtiles;
    id.ptile = t - r * P.wg_mtiles;
    id.split = r / P.wg_vgroups;
    id.vg = r - id.split * P.wg_vgroups;
    id.kb0 = id.split * kblocks;
  }
  return id;
}

constexpr int kBiasPad = 256;  // zeros behind the staged bias: every accumulator column of a tile reads an entry
struct GatherSmem {
  uint32_t b_stage_bytes, taps_off, cols_off, bias_off, ptab_off, bars_off, total;
};
// ptab_warps: producer warps that keep a double-buffered 32-entry slice of the per-pixel table (weight-gradient mode).
__host__ __device__ inline GatherSmem gather_smem(int n_pad, int k_pad, int b_stages, int n_bias, int ptab_warps = 0) {
  GatherSmem L;
  L.b_stage_bytes = 2u * (uint32_t)n_pad * 128u;
  L.taps_off = (uint32_t)b_stages * L.b_stage_bytes;
  L.cols_off = L.taps_off + (uint32_t)k_pad * 8u;
  L.bias_off = L.cols_off + (uint32_t)n_pad * 8u;
  L.ptab_off = (L.bias_off + (uint32_t)(n_bias + kBiasPad) * 4u + 15u) & ~15u;
  L.bars_off = L.ptab_off + (uint32_t)ptab_warps * 512u;
  L.total = L.bars_off + 8u * (2 * kMaxAStages + 2 * kMaxAccBufs) + 16u;
  return L;
}

// MODE: what the lanes gather - one table entry per reduction index, one per kRun of them, or (weight gradient) rows of the
// lowered matrix over pixels.
// kInside: one offset per reduction index (four to a shared-memory read) and no bounds test - a forward pass without padding,
// whose windows lie inside the plane: 5.3 instructions per value instead of 9, AlexNet conv1 at batch 256 320 -> 293 us.  (Entries
// behind the last real index read the window's first element against a weight of zero; lanes behind the last pixel read the last
// pixel's window, their columns are not stored.)
// FORM: one of these, + kHalf (HALF), + kTall (with it: tall blocks of pixels, GatherProblem::rows)
enum { kByTap = 0, kByRun = 1, kWeightGrad = 2, kInside = 3, kHalf = 4, kTall = 8 };
// ONE: every CTA has one tile, a short one (kOneKblocks).  There is no next tile then for the epilogue to overlap with, and the producers,
// who are through, take their share of its columns (six chunks of 16 took four warps 1.2 us); in front of the first k-block stood three
// trips to L2 for the tables and the bias, one behind the other, and the allocation of tensor memory (1.3 us in all), now one trip
// beside the allocation.  conv3 of one image 13.6 -> 13.0 us, 37 images of 50 -> 75 channels both ways 36.3 -> 34.9.  Not for the
// persistent kernels' last tiles, nor for the other two modes: the registers it takes spill (AlexNet conv1 at batch 256 1 211 -> 1 227
// us both ways; LeNet conv2's forward kernel 9.9 -> 11.1).  Where a tile is long it gains nothing (CaffeNet at batch 32 1 238 -> 1 245 us).
// Data gradients with a stride, which store every other word and further apart, only up to kOneScattered columns per SM (stride 2; half as many
// above: 4 -> 12 channels 148 x 148, 11 x 11 by 4, 8 images, 37 columns per SM, 7.7 -> 7.7 us, 23 images, 106, 10.3 -> 11.5): beyond, all warps storing
// at once are slower than the persistent kernel's four in turn (64 -> 8 channels 21 x 21, 3 x 3 by 2: 78 images, 296 tiles of 64 columns, 8.5 -> 8.3
// us, 148 images, 280 of 128, 10.9 -> 11.8; 256 -> 51 channels 13 x 13, 48 images, 133 of 160, 13.1 -> 13.5).
constexpr int kOneKblocks = 32, kOneScattered = 128;
// HALF: the operands as pairs of fp16 where the scales of this call say so (operand_scale.cuh), of tf32 otherwise: an A slot has 32 columns
// then (16 of hi, 16 of lo, two values to a column), a weight slot one row of 128 bytes per column, 32 hi and 32 lo.  Half the MMAs:
// CaffeNet at batch 256, conv2 forward 387 -> 280 us, conv3 256 / 253 / 273 (forward, weight, data gradient) -> 150 / 165 / 176, conv4 213 /
// 210 / 211 -> 116 / 138 / 119, conv5 141 / 159 / 149 -> 98 / 138 / 85, 14 - 26 us for each look at the operands; what is left is the gather of the
// producers (tensor pipe and load-store unit wait for it).  Errors against 64 bits are half as large (conv3, 64 images of 14 x 14, positive
// data: Y 1.44e-5 -> 7.9e-6, dX 7.8e-6 -> 4.6e-6, dW 2.2e-5 -> 1.1e-5), since the accumulator is truncated half as often.
template <int SETS, int FORM, bool ONE>
__global__ void __launch_bounds__(gather_threads(SETS), SETS == 2 ? 2 : 1)
    gather_conv_kernel(const __grid_constant__ GatherParams P, const __grid_constant__ CUtensorMap w_map) {
  constexpr int MODE = FORM % kHalf;
  constexpr bool HALF = FORM >= kHalf, TALL = FORM >= kTall;
  constexpr int kProducerWarps = 4 * SETS, kMmaWarp = kProducerWarps, kTmaWarp = kMmaWarp + 1;
  constexpr int kGatherThreads = gather_threads(SETS);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const GatherSmem L = gather_smem(P.n_pad, P.taps_smem, P.b_stages, P.n_bias, MODE == kWeightGrad ? kProducerWarps : 0);
  const uint32_t bars = base + L.bars_off;
  // K-block i (running index over this CTA's tiles) uses A slot i % a_stages, weight slot i % b_stages and the
  // barrier pair i % 4: "ready" completes when the four producer warps of the block's set and the weight tile's TMA
  // bytes have arrived, "done" when the block's MMAs have finished (one tcgen05.commit), which frees both slots.
  // Rings of different depth share the barriers because no waiter can fall a whole barrier phase (4 blocks) behind:
  // block i + 4 cannot finish before the slots of block i + 3 were refilled, which waits for block i.
  const uint32_t ready_bar = bars, done_bar = ready_bar + 8u * kMaxAStages, acc_full = done_bar + 8u * kMaxAStages,
                 acc_empty = acc_full + 8u * kMaxAccBufs, tmem_slot = acc_empty + 8u * kMaxAccBufs;
  MaskTap* s_taps = reinterpret_cast<MaskTap*>(base_ptr + L.taps_off);
  ColEnt* s_cols = reinterpret_cast<ColEnt*>(base_ptr + L.cols_off);
  float* s_bias = reinterpret_cast<float*>(base_ptr + L.bias_off);
  const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;

  // HALF: the gathered operand's scale (0: tf32 instead), what takes both operands' scales back, how many values are not finite
  float* s_scale = reinterpret_cast<float*>(base_ptr + (tmem_slot + 4 - base));
  int* s_offsets = reinterpret_cast<int*>(s_taps);  // kInside: the offsets alone
  if (HALF && P.only != kAny) {
    pdl_wait();
    if (tall_route(P.half) != (P.only == kOnlyHalf)) return;
  }
  auto init_barriers = [&]() {
    for (int s = 0; s < kMaxAStages; ++s) { mbar_init(ready_bar + 8u * s, 5); mbar_init(done_bar + 8u * s, 1); }  // 4 producer warps + the TMA thread
    for (int s = 0; s < kMaxAccBufs; ++s) { mbar_init(acc_full + 8u * s, 1); mbar_init(acc_empty + 8u * s, kEpiWarps); }
    fence_mbar_init();
  };
  if constexpr (ONE) {
    static_assert(MODE == kByTap || MODE == kByRun, "the other modes have no registers to spare");
    if (warp == 0) tmem_alloc(tmem_slot, (uint32_t)P.tmem_cols);
    else if (tid == 32) init_barriers();
    if (warp == kTmaWarp) prefetch_map(&w_map);
    MaskTap tap0{};
    ColEnt col0{};
    if (tid < P.taps_smem) tap0 = P.taps[tid];
    if (tid < P.n_pad) col0 = P.cols[tid];
    pdl_wait();  // so far the plan's tables alone have been read
    const float bias0 = tid < P.n_bias ? P.bias[tid] : 0.f;
    if (tid < P.taps_smem) s_taps[tid] = tap0;
    if (tid < P.n_pad) s_cols[tid] = col0;
    if (tid < P.n_bias + kBiasPad) s_bias[tid] = bias0;
#pragma unroll 4
    for (int i = tid + kGatherThreads; i < P.taps_smem; i += kGatherThreads) s_taps[i] = P.taps[i];
    for (int i = tid + kGatherThreads; i < P.n_bias + kBiasPad; i += kGatherThreads) s_bias[i] = i < P.n_bias ? P.bias[i] : 0.f;
  } else {
    for (int i = tid; i < P.taps_smem; i += kGatherThreads) {
      if (MODE == kInside) s_offsets[i] = P.taps[i].off;
      else s_taps[i] = P.taps[i];
    }
    if (P.cols)
      for (int i = tid; i < P.n_pad; i += kGatherThreads) s_cols[i] = P.cols[i];
    if (tid == 0) init_barriers();
    if (warp == 0) tmem_alloc(tmem_slot, (uint32_t)P.tmem_cols);
    if (warp == kTmaWarp) prefetch_map(&w_map);
    pdl_wait();  // so far the plan's tables alone have been read: set-up beside the end of the kernel before (15.6 -> 15.35 us for conv3 of one image)
    for (int i = tid; i < P.n_bias + kBiasPad; i += kGatherThreads) s_bias[i] = i < P.n_bias ? P.bias[i] : 0.f;
    if (HALF && tid == 0) {
      const HalfScale a = P.half->of[P.half_gathered], b = P.half->of[P.half_packed];
      s_scale[0] = a.ok && b.ok && P.only != kOnlyTf32 ? a.scale : 0.f;
      s_scale[1] = a.inverse * b.inverse;
      reinterpret_cast<int*>(s_scale)[2] = a.bad;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const uint32_t acc_cols = (uint32_t)acc_columns(P.n_pad), cross = acc_cols - (uint32_t)P.n_pad;  // cross: 0 = one accumulator
  const int kblocks = P.k_pad / kBlockK;
  bool failed = false;
  // The roles' text stands in a file of its own because the half kernels need it twice, each time with `half` known: by a flag in one text
  // <2, kWeightGrad> spilled (CaffeNet conv2's weight gradient 332 -> 372 us); as a function or a lambda the kernels of single tiles
  // came out with more registers (37 images of 50 -> 75 channels both ways 35.0 -> 36.4).
  if constexpr (HALF) {
    if (TALL || s_scale[0] != 0.f) {
      constexpr bool half = true;
      const uint32_t acc_cols = (uint32_t)P.acc_cols_half, cross = acc_cols - (uint32_t)P.n_pad;
#include "gather_roles.inc"
    } else {
      constexpr bool half = false;
#include "gather_roles.inc"
    }
  } else {
    constexpr bool half = false;
#include "gather_roles.inc"
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, (uint32_t)P.tmem_cols);
}

// Adds the split sums of gather_conv_kernel in split order, then does what its epilogue does: bias, ReLU, the scatter of
// the data gradient.  Lanes along the pixels (both sides coalesced), a thread owns COLS columns of its pixel: eight where
// there are plenty of pixels (one decode of the pixel for eight columns: CaffeNet conv5 at batch 32, 11 MB of L2-resident
// sums, 14 -> 6 us against one column per thread), one where there are few and the splits' loads have to be in flight
// together (conv3 of one image, 12 splits: 8 -> 4 us against eight).
// ONLY: returns at once where the data gradient has gone by tall blocks.
template <int COLS, bool ONLY>
__global__ void __launch_bounds__(128) gather_reduce_kernel(const __grid_constant__ GatherParams P, int col_tiles) {
  pdl_wait();
  if (ONLY && tall_route(P.half)) return;
  const int pix = blockIdx.x * 128 + threadIdx.x;
  const int vg = blockIdx.y / col_tiles, col0 = (blockIdx.y - vg * col_tiles) * COLS, vgroups = gridDim.y / col_tiles;
  const int grp = vg / P.tiles_per_group, ntile = vg - grp * P.tiles_per_group;
  const int live = min(COLS, min(P.n, (P.out_group_channels - ntile * P.out_tile_channels) * P.cols_per_channel) - col0);
  if (pix >= P.n_pix || live <= 0) return;
  const float* src = P.partial + ((size_t)vg * P.n_pad + col0) * P.pix_pad + pix;
  const size_t stride = (size_t)vgroups * P.n_pad * P.pix_pad;
  float y[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) y[c] = 0.f;
#pragma unroll(COLS == 1 ? 8 : 2)
  for (int s = 0; s < P.splits; ++s, src += stride)
#pragma unroll
    for (int c = 0; c < COLS; ++c) y[c] += c < live ? __ldg(src + (size_t)c * P.pix_pad) : 0.f;
  const int per_img = P.q_h * P.q_w;
  const int b = pix / per_img, r = pix - b * per_img;
  const int qy = r / P.q_w, qx = r - qy * P.q_w;
  const int oy0 = qy * P.oy_mul + P.oy_add, ox0 = qx * P.ox_mul + P.ox_add;
  const int ch0 = grp * P.out_group_channels + ntile * P.out_tile_channels;
  float* op = P.out + (long long)b * P.out_batch_stride + (long long)ch0 * P.out_plane + (long long)oy0 * P.out_pitch + ox0;
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    if (c < live) {
      const ColEnt ce = P.cols[col0 + c];
      float v = y[c];
      if (P.bias) v += __ldg(P.bias + ch0 + col0 + c);  // the forward pass: one column per channel
      if (P.relu) v = fmaxf(v, 0.f);
      if (!P.check_out || ((unsigned)(oy0 + ce.cy) < (unsigned)P.out_lim && (unsigned)(ox0 + ce.cx) < (unsigned)P.out_lim)) op[ce.off] = v;
    }
  }
}

// ---------------------------------------------------------------------------------- weight-gradient kernel
//
// dW[kk][o] (+ the bias row) = sum over pixels of Lowered(X)[pix][kk] * dY[pix][o], split over pixel ranges.
// Both operands are K-major shared-memory tiles whose rows are 32 consecutive pixels (one 128-byte swizzled row):
// a row of the lowered operand is one tap (d, kr, kc) seen by 32 consecutive output pixels, a row of the other
// operand is one output channel of dY for the same pixels.  With lane = pixel every global load is a coalesced run
// and every shared-memory store fills one row, conflict free.
// One CTA owns up to `subs` M-tiles of 128 taps (accumulators side by side in tensor memory), one channel tile of dY
// and a range of 32-pixel k-blocks; the dY tile of a k-block is staged once for all its M-tiles.
//   warps 0-15  tap producers: warp w stages rows w, w+16, ... of every M-tile of the stage: load, split hi/lo, two
//               st.shared per row; the loads of the next k-block are issued before the warp waits for the stage
//               buffer to drain.
//   warps 16-23 dY producers: warp 16+w stages channel rows w, w+8, ... of the dY tile the same way.
//   warp 24     issues the MMAs (both operands from shared memory).
// The producers run at about one instruction per eight cycles each (latency bound), so their number, not their
// instruction count alone, sets the staging rate.  The finished accumulators are written to the split's slice of the
// scratch buffer by warps 0-15.
constexpr int kWgTapWarps = 16, kWgDyWarps = 8, kWgProdWarps = kWgTapWarps + kWgDyWarps, kWgMmaWarp = kWgProdWarps;
constexpr int kWgThreads = (kWgMmaWarp + 1) * 32;  // 800
constexpr int kWgMaxStages = 4, kWgMaxSubs = 2;
constexpr uint32_t kWgValidBit = 0x80000000u;      // set in a pixel's mask when the pixel exists
constexpr uint32_t kWgPadBit = 0x00008000u;        // never set in a pixel's mask: rows beyond the lowered matrix
constexpr uint32_t kWgOnesBits = kWgValidBit | kWgPadBit;  // the all-ones row: never loaded, patched in by its warp

struct WgradParams {
  const float* x;
  const float* dy;
  float* partial;       // [splits][vgroups][m_tiles*128][n_pad]
  const MaskTap* taps;  // [m_tiles*128]; row k_real is the all-ones row, rows beyond it are padding
  int n_pix, m, mm, n, s, p, k;
  long long x_batch_stride;
  int x_group_stride;
  long long dy_batch_stride;
  int dy_group_channels;  // output channels per real group
  int tiles_per_group;
  int n_real, n_pad;
  int m_tiles, subs, stages;
  int x_count;            // elements of x from the first group's on (wgrad_ts_kernel with wide loads)
  int ones_row;           // index of the all-ones row among the lowered-matrix rows
  int kblocks_total, kblocks_per_split;  // end of this launch's k-block range, k-blocks per split
  int kb_first;                          // first k-block of this launch (a later round of a launch sequence starts further in)
  int* status;
  const HalfScales* half = nullptr;      // wgrad_ts_kernel<true>: returns at once where wgrad_half_kernel takes the call
};

struct WgSmem {
  uint32_t a_tile_bytes, b_tile_bytes, stage_bytes, taps_off, bars_off, total;
};
__host__ __device__ inline WgSmem wg_smem(int n_pad, int subs, int stages) {
  WgSmem L;
  L.a_tile_bytes = kTileM * 128u;           // one of hi / lo of one M-tile
  L.b_tile_bytes = (uint32_t)n_pad * 128u;  // one of hi / lo of the dY tile
  L.stage_bytes = 2u * (uint32_t)subs * L.a_tile_bytes + 2u * L.b_tile_bytes;
  L.taps_off = (uint32_t)stages * L.stage_bytes;
  L.bars_off = L.taps_off + (uint32_t)subs * kTileM * 8u;
  L.total = L.bars_off + 8u * (2 * kWgMaxStages + 1) + 16u;
  return L;
}


// SUBS: M-tiles per CTA (accumulators), NB: dY-tile rows per producer warp (= n_pad / 16).  With both fixed at
// compile time every warp stages exactly 8*SUBS tap rows and NB channel rows per k-block, all loads of a k-block are
// in flight together, and the shared-memory addresses are one per-warp base plus immediates: row warp+16*i of a
// 128-byte-swizzled tile has the same swizzle phase ((warp+16*i) & 7 == warp & 7) for every i.
template <int SUBS, int NB>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_kernel(const __grid_constant__ WgradParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const WgSmem L = wg_smem(NB * 16, SUBS, P.stages);
  const uint32_t bars = base + L.bars_off;
  const uint32_t full = bars, empty = full + 8u * kWgMaxStages, acc_full = empty + 8u * kWgMaxStages,
                 tmem_slot = acc_full + 8u;
  MaskTap* s_taps = reinterpret_cast<MaskTap*>(base_ptr + L.taps_off);
  const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
  const int mgroup = blockIdx.x, split = blockIdx.y, vg = blockIdx.z;
  const int grp = vg / P.tiles_per_group, ntile = vg % P.tiles_per_group;
  const int subs = min(SUBS, P.m_tiles - mgroup * SUBS);  // M-tiles this CTA really has
  constexpr int kARows = 8 * SUBS;                        // tap rows per producer warp and k-block
  constexpr uint32_t kATile = kTileM * 128u, kBTile = NB * 16u * 128u;
  constexpr int kNPad = NB * 16;
  // Narrow dY tiles run "dual": the lo tile sits right behind the hi tile, one MMA of width 2*kNPad covers both (an
  // MMA pays some 43 cycles for reading A from shared memory, however narrow it is), and the epilogue adds the two halves of the
  // accumulator.
  constexpr bool kDual = kNPad <= 64;  // operands from shared memory: an MMA wider than 128 is slower than two narrow ones
  constexpr int kAccCols = kDual ? 2 * kNPad : kNPad;

  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
  } else if (tid == 32) {
    for (int s = 0; s < kWgMaxStages; ++s) { mbar_init(full + 8u * s, kWgProdWarps); mbar_init(empty + 8u * s, 1); }
    mbar_init(acc_full, 1);
    fence_mbar_init();
  }
  pdl_wait();  // (the table too may come from a kernel)
  for (int i = tid; i < SUBS * kTileM; i += kWgThreads)
    s_taps[i] = i < subs * kTileM ? P.taps[mgroup * SUBS * kTileM + i] : MaskTap{0, kWgPadBit};
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const int kb_begin = P.kb_first + split * P.kblocks_per_split;
  const int kb_end = min(P.kblocks_total, kb_begin + P.kblocks_per_split);
  const int kblocks = kb_end - kb_begin;  // >= 1 by construction of the grid
  bool failed = false;

  if (warp < kWgProdWarps) {
    // ------------------------------------------------------------------ producers (lane = pixel of the k-block)
    // this lane's pixel, advanced by 32 per k-block
    int pix = kb_begin * kBlockK + lane;
    int pb = pix / P.mm, pr, pc;
    {
      const int pin = pix - pb * P.mm;
      pr = pin / P.m;
      pc = pin - pr * P.m;
    }
    auto next_pixel = [&]() {
      pix += kBlockK;
      pc += kBlockK;
      while (pc >= P.m) { pc -= P.m; ++pr; }
      while (pr >= P.m) { pr -= P.m; ++pb; }
    };
    if (warp < kWgTapWarps) {
      // ---- tap rows: row warp + 16*i of every M-tile
      const float* xg = P.x + (long long)grp * P.x_group_stride;
      // The all-ones row (bias gradient) is one fixed row of one CTA column: its table entry never passes the
      // bounds test (so nothing is loaded for it) and the warp that owns it patches the value in.
      const int ones_local = P.ones_row - mgroup * SUBS * kTileM;
      const bool mine = ones_local >= 0 && ones_local < subs * kTileM && ((ones_local & (kTileM - 1)) % kWgTapWarps) == warp;
      const int ones_i = mine ? (ones_local / kTileM) * 8 + (ones_local & (kTileM - 1)) / kWgTapWarps : -1;
      // This lane's word in row `warp` of a tile; the warp's further rows are 2048 bytes apart.
      uint8_t* lane_ptr = base_ptr + warp * 128 + ((((lane >> 2) ^ (warp & 7)) << 4) + (lane & 3) * 4);
      const MaskTap* my_taps = s_taps + warp;
      float va[kARows];
      auto load_rows = [&]() {
        const bool ok = pix < P.n_pix;
        const int iy0 = pr * P.s - P.p, ix0 = pc * P.s - P.p;
        const float* xsrc = xg + (long long)pb * P.x_batch_stride + (long long)iy0 * P.n + ix0;
        const uint32_t mask =
            ok ? (kWgValidBit | bit_range(-iy0, min(P.k, P.n - iy0)) | (bit_range(-ix0, min(P.k, P.n - ix0)) << 16))
               : 0u;
#pragma unroll
        for (int i = 0; i < kARows; ++i) {
          const MaskTap tap = my_taps[kWgTapWarps * i];
          va[i] = ldg_if_bits(xsrc + tap.off, mask, tap.bits);
        }
        if (ones_i >= 0) {
#pragma unroll
          for (int i = 0; i < kARows; ++i) va[i] = i == ones_i ? (ok ? 1.f : 0.f) : va[i];
        }
      };
      load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(P.stages)) {
        const int s = ring.idx, use = ring.use;
        uint8_t* st = lane_ptr + (size_t)s * L.stage_bytes;
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x10);
#pragma unroll
        for (int i = 0; i < kARows; ++i) {  // tile i/8 (hi then lo), row warp + 16*(i%8)
          uint32_t h, l;
          split_tf32_trunc(va[i], h, l);
          uint8_t* dst = st + (i / 8) * 2 * kATile + (i % 8) * 2048;
          *reinterpret_cast<uint32_t*>(dst) = h;
          *reinterpret_cast<uint32_t*>(dst + kATile) = l;
        }
        if (kbl + 1 < kblocks) {  // the next k-block's loads go in flight before the barrier work
          next_pixel();
          load_rows();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);  // one arrival per warp: same-address arrivals serialise
      }
    } else {
      // ---- dY rows: channel w8 + 8*i of the tile (hi then lo), behind the SUBS tap tiles of the stage
      const int w8 = warp - kWgTapWarps;
      constexpr int kDyRows = kNPad / kWgDyWarps;
      const float* dyg = P.dy + (long long)(grp * P.dy_group_channels + ntile * P.n_real + w8) * P.mm;
      const int dy_step = kWgDyWarps * P.mm;  // elements between consecutive channel rows of this warp
      const int n_live = min(P.n_real, P.dy_group_channels - ntile * P.n_real);  // the last tile of a group may be shorter
      const int b_live = n_live > w8 ? (n_live - w8 + kWgDyWarps - 1) / kWgDyWarps : 0;  // real rows
      uint8_t* lane_ptr = base_ptr + SUBS * 2 * kATile + w8 * 128 + ((((lane >> 2) ^ (w8 & 7)) << 4) + (lane & 3) * 4);
      float vb[kDyRows];
      auto load_rows = [&]() {
        const bool ok = pix < P.n_pix;
        const float* dsrc = dyg + (long long)pb * P.dy_batch_stride + pr * P.m + pc;
#pragma unroll
        for (int i = 0; i < kDyRows; ++i) vb[i] = ldg_if(dsrc + i * dy_step, (ok && i < b_live) ? 1u : 0u);
      };
      load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(P.stages)) {
        const int s = ring.idx, use = ring.use;
        uint8_t* st = lane_ptr + (size_t)s * L.stage_bytes;
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x11);
#pragma unroll
        for (int i = 0; i < kDyRows; ++i) {
          uint32_t h, l;
          split_tf32_trunc(vb[i], h, l);
          uint8_t* dst = st + i * (kWgDyWarps * 128);
          *reinterpret_cast<uint32_t*>(dst) = h;
          *reinterpret_cast<uint32_t*>(dst + kBTile) = l;
        }
        if (kbl + 1 < kblocks) {
          next_pixel();
          load_rows();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
    }
    if (warp < kWgTapWarps) {
    // ---- epilogue: accumulator u, columns in chunks of 16; warp w takes lanes 32*(w%4).. and the (u, chunk) pairs
    //      with index == w/4 (mod 4)
    mbar_wait(acc_full, 0u, failed, P.status, 0x2000);
    tc_fence_after();
    const int quarter = warp & 3, row = quarter * 32 + lane;
    for (int w = warp >> 2; w < subs * NB; w += 4) {
      const int u = w / NB, c = w - u * NB;
      float acc[16];
      const uint32_t col = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(u * kAccCols + c * 16);
      tmem_ld16(col, acc);
      if (kDual) {
        float lo_part[16];
        tmem_ld16(col + kNPad, lo_part);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] += lo_part[j];
      }
      float* op = P.partial + (((size_t)split * gridDim.z + vg) * P.m_tiles * kTileM +
                               (size_t)(mgroup * SUBS + u) * kTileM + row) * kNPad + c * 16;
      if (!failed) {
        float4* o4 = reinterpret_cast<float4*>(op);
#pragma unroll
        for (int j = 0; j < 4; ++j) o4[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
      }
    }
    }
  } else {
    // ------------------------------------------------------------------ MMA issue (see elect_one)
    const uint32_t idesc = make_idesc(kAccCols), tmem = warp_uniform(tmem_base);
    const int n_subs = (int)warp_uniform((uint32_t)subs);
    Ring ring;
    for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(P.stages)) {
      const int s = ring.idx;
      mbar_wait(full + 8u * s, (uint32_t)ring.use & 1u, failed, P.status, 0x40);  // parked: this warp mostly waits for the producers
      tc_fence_after();
      const uint32_t st = base + (uint32_t)s * L.stage_bytes;
      const uint32_t b_hi = st + SUBS * 2u * kATile, b_lo = b_hi + kBTile;
      const uint64_t dbh = make_desc(b_hi), dbl = make_desc(b_lo);
      if (elect_one()) {
        for (int u = 0; u < n_subs; ++u) {
          const uint32_t d_tmem = tmem + (uint32_t)(u * kAccCols);
          const uint32_t a_hi = st + (uint32_t)u * 2u * kATile;
          const uint64_t dah = make_desc(a_hi), dal = make_desc(a_hi + kATile);
#pragma unroll
          for (int j = 0; j < kBlockK / 8; ++j) {
            const uint64_t adv = (uint64_t)(j * 2);
            umma_tf32_ss(d_tmem, dal + adv, dbh + adv, idesc, (kbl == 0 && j == 0) ? 0u : 1u);
            if (!kDual) umma_tf32_ss(d_tmem, dah + adv, dbl + adv, idesc, 1u);
            umma_tf32_ss(d_tmem, dah + adv, dbh + adv, idesc, 1u);
          }
        }
        umma_commit(empty + 8u * s);
        if (kbl == kblocks - 1) umma_commit(acc_full);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// ---------------------------------------------------------------------------------------------------------------
// The same weight gradient with the operands' roles exchanged, for lowered matrices of 257 .. 384 rows (with the
// all-ones row) and at most 128 output channels per tile - AlexNet / CaffeNet conv1:
//     D[channel][row] = sum over pixels of dY[channel][pixel] * lowered[row][pixel].
// The small operand (dY: 128 lanes = channels, 32 pixels per k-block) goes through TENSOR memory, so the MMAs read only
// the lowered rows from shared memory, 192 of them per instruction (two accumulators of 192 columns): per k-block 24
// MMAs of 96 cycles each, none paying the shared-memory-A surcharge, where wgrad_kernel issues 36 of 91, and one CTA
// covers all rows, so dY is staged once per k-block for the whole SM.
//   warps 0-23  tap producers: warp w stages rows w, w+24, ... (16 rows) of the 384-row tile exactly as wgrad_kernel's
//               (WIDE: warps 0-17, two window rows each).
//   warps 24-27 dY (WIDE: 18-25, two per quadrant): the warp of quadrant q owns channels 32q .. 32q+31 (= the tensor-memory
//               lanes it reaches): coalesced loads with lane = pixel,
//               a turn through a private 32 x 33 shared-memory tile, then lane = channel: split and tcgen05.st.
//               After the last k-block the same warps write the accumulators out (lane = channel = fastest index of the
//               partial-sum buffer).
//   last warp   issues the MMAs.
// The partial sums have wgrad_kernel's layout ([split][tile][row][channel]), so the same reduction kernels follow.
__host__ __device__ constexpr int ts_tap_warps(bool wide) { return wide ? 18 : 24; }
__host__ __device__ constexpr int ts_dy_warps(bool wide) { return wide ? 8 : 4; }
__host__ __device__ constexpr int ts_threads(bool wide) { return (ts_tap_warps(wide) + ts_dy_warps(wide) + 1) * 32; }  // 864 or 928
constexpr int kTsRows = 384, kTsNTile = 192, kTsStages = 2;
constexpr uint32_t kTsTile = kTsRows * 128u;       // one of hi / lo of the lowered rows of a k-block
constexpr uint32_t kTsStage = 2u * kTsTile;
constexpr uint32_t kTsTapsOff = kTsStages * kTsStage, kTsTurnOff = kTsTapsOff + kTsRows * 8u,
                   kTsBarsOff = kTsTurnOff + 4u * 32u * 33u * 4u, kTsSmem = kTsBarsOff + 8u * (2 * kTsStages + 1) + 16u;

//
// WIDE (stride a multiple of four, no padding): a tap warp stages whole window rows (input channel, kernel row).  The pixels of
// an image then lie at the same place in their 16-byte blocks, so the k consecutive elements that a pixel needs come with
// three or four aligned loads, and which loaded word is which tap is the same for the whole warp: a branch, no selects.  A
// load per element touched sixteen sectors for the four it used, and the load pipe bound the kernel.  A k-block that crosses
// images, or the tensor's ends, loads element by element.  18 tap warps and 8 dY warps then: with four the turn of dY was the
// longest chain of a k-block.  AlexNet conv1 at batch 256 393 -> 358 us (the MMAs alone would take 205), 16 images of
// 100 x 100 30.4 -> 18.0; what is left is the round of loads, stores and barriers that two stages cannot hide.
constexpr int kTsWideTaps = 13, kTsWideRows = 2;  // taps that four blocks cover at any alignment; window rows per warp

__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Splits taps 0 .. k - 1, which start at w[SHIFT], and stores them as lowered rows: row r at dst + off[r & 7] + (r & ~7) * 128.
template <int SHIFT>
__device__ __forceinline__ void store_wide(const float* w, int k, uint8_t* dst, const uint32_t* off) {
#pragma unroll
  for (int r = 0; r < kTsWideTaps; ++r) {
    if (r >= k) break;
    uint32_t h, l;
    split_tf32_trunc(w[SHIFT + r], h, l);
    uint8_t* at = dst + off[r & 7] + (r & ~7) * 128;
    *reinterpret_cast<uint32_t*>(at) = h;
    *reinterpret_cast<uint32_t*>(at + kTsTile) = l;
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(ts_threads(WIDE), 1) wgrad_ts_kernel(const __grid_constant__ WgradParams P) {
  constexpr int kTsTapWarps = ts_tap_warps(WIDE), kTsDyWarps = ts_dy_warps(WIDE), kTsMmaWarp = kTsTapWarps + kTsDyWarps;
  constexpr int kTsThreads = ts_threads(WIDE), kTsRowsPerWarp = kTsRows / 24;  // 16
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + kTsBarsOff;
  const uint32_t full = bars, empty = full + 8u * kTsStages, acc_full = empty + 8u * kTsStages, tmem_slot = acc_full + 8u;
  MaskTap* s_taps = reinterpret_cast<MaskTap*>(base_ptr + kTsTapsOff);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.y, vg = blockIdx.z;
  const int grp = vg / P.tiles_per_group, ntile = vg % P.tiles_per_group;
  constexpr uint32_t kACol0 = 2 * kTsNTile;  // tensor memory: two accumulators of 192 columns, then 2 x 64 columns of A

  if (WIDE && P.half) {
    pdl_wait();
    if (half_route(P.half, kHalfX, kHalfDy)) return;
  }
  if (WIDE) {  // lowered rows that no warp stages: zeros
    const int words = (kTsRows - P.ones_row - 1) * 32;
    for (int i = tid; i < words * 2 * kTsStages; i += kTsThreads) {
      const int part = i / words;
      reinterpret_cast<uint32_t*>(base_ptr + (size_t)part * kTsTile + (size_t)(P.ones_row + 1) * 128)[i - part * words] = 0u;
    }
    fence_proxy_async_smem();
  } else {
    for (int i = tid; i < kTsRows; i += kTsThreads) s_taps[i] = P.taps[i];
  }
  if (tid == 0) {
    for (int s = 0; s < kTsStages; ++s) { mbar_init(full + 8u * s, kTsTapWarps + kTsDyWarps); mbar_init(empty + 8u * s, 1); }
    mbar_init(acc_full, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  pdl_wait();  // so far the plan's table alone has been read
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const int kb_begin = P.kb_first + split * P.kblocks_per_split;
  const int kb_end = min(P.kblocks_total, kb_begin + P.kblocks_per_split);
  const int kblocks = kb_end - kb_begin;
  bool failed = false;

  if (warp < kTsMmaWarp) {
    // this lane's pixel, advanced by 32 per k-block
    int pix = kb_begin * kBlockK + lane;
    int pb = pix / P.mm, pr, pc;
    {
      const int pin = pix - pb * P.mm;
      pr = pin / P.m;
      pc = pin - pr * P.m;
    }
    auto next_pixel = [&]() {
      pix += kBlockK;
      pc += kBlockK;
      while (pc >= P.m) { pc -= P.m; ++pr; }
      while (pr >= P.m) { pr -= P.m; ++pb; }
    };
    if (WIDE && warp < kTsTapWarps) {
      // ---- window rows u = 2 warp and 2 warp + 1: lowered rows u * k + kc, whose swizzle phases repeat after eight
      const int k = P.k, units = P.ones_row / k, mine = min(kTsWideRows, max(0, units - kTsWideRows * warp));
      const float* x = P.x + (long long)grp * P.x_group_stride;
      int unit_at[kTsWideRows];
      uint32_t lane_off[kTsWideRows][8];
#pragma unroll
      for (int i = 0; i < kTsWideRows; ++i) {
        const int u = kTsWideRows * warp + i, d = u / k;
        unit_at[i] = d * P.n * P.n + (u - d * k) * P.n;
#pragma unroll
        for (int r = 0; r < 8; ++r) lane_off[i][r] = (uint32_t)((u * k + r) * 128 + (((lane >> 2) ^ ((u * k + r) & 7)) << 4) + (lane & 3) * 4);
      }
      const int ones = warp == kTsTapWarps - 1 ? P.ones_row : -1;
      const int misaligned = (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3);  // words between x and its 16-byte block
      float w[kTsWideRows][16];
      int shift[kTsWideRows] = {0, 0};
      bool ok = false;
      auto load_rows = [&]() {
        ok = pix < P.n_pix;
        const int at0 = pb * (int)P.x_batch_stride + pr * P.s * P.n + pc * P.s;
        // The lines of the k-block after the next one (if it lies in the same image), every eighth lane one line: with one
        // k-block's loads in flight a trip to HBM was longer than the MMAs it hid behind.
        int far_r = pr, far_c = pc + 2 * kBlockK;
        while (far_c >= P.m) { far_c -= P.m; ++far_r; }
        const bool far_in = far_r < P.m && (lane & 7) == 0;
        const int far0 = pb * (int)P.x_batch_stride + far_r * P.s * P.n + far_c * P.s;
        const int pb0 = __shfl_sync(0xffffffffu, pb, 0);
        const bool one_image = __all_sync(0xffffffffu, ok && pb == pb0);
#pragma unroll
        for (int i = 0; i < kTsWideRows; ++i) {
          if (i >= mine) break;
          const int at = at0 + unit_at[i];
          if (far_in && ok) prefetch_l2(x + far0 + unit_at[i]);
          shift[i] = (at + misaligned) & 3;  // of this lane; of every lane where the pixels are one image's
          const int first = at - shift[i];
          if (__all_sync(0xffffffffu, one_image && first >= 0 && first + 16 <= P.x_count)) {
            const float4* block = reinterpret_cast<const float4*>(x + first);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (4 * j >= k + shift[i]) break;
              const float4 v = __ldg(block + j);
              w[i][4 * j] = v.x; w[i][4 * j + 1] = v.y; w[i][4 * j + 2] = v.z; w[i][4 * j + 3] = v.w;
            }
          } else {
            shift[i] = 0;
#pragma unroll
            for (int r = 0; r < kTsWideTaps; ++r) {
              if (r >= k) break;
              w[i][r] = ok ? __ldg(x + at + r) : 0.f;
            }
          }
        }
      };
      load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
        const int s = ring.idx, use = ring.use;
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3010);
#pragma unroll
        for (int i = 0; i < kTsWideRows; ++i) {
          if (i >= mine) break;
          uint8_t* dst = base_ptr + (size_t)s * kTsStage;
          switch ((int)warp_uniform((uint32_t)shift[i])) {
            case 0: store_wide<0>(w[i], k, dst, lane_off[i]); break;
            case 1: store_wide<1>(w[i], k, dst, lane_off[i]); break;
            case 2: store_wide<2>(w[i], k, dst, lane_off[i]); break;
            default: store_wide<3>(w[i], k, dst, lane_off[i]); break;
          }
        }
        if (ones >= 0) {
          uint8_t* dst = base_ptr + (size_t)s * kTsStage + ones * 128 + (((lane >> 2) ^ (ones & 7)) << 4) + (lane & 3) * 4;
          *reinterpret_cast<float*>(dst) = ok ? 1.f : 0.f;
          *reinterpret_cast<float*>(dst + kTsTile) = 0.f;
        }
        if (kbl + 1 < kblocks) {  // the next k-block's loads go in flight before the barrier work
          next_pixel();
          load_rows();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
    } else if (warp < kTsTapWarps) {
      // ---- lowered rows warp + 24*i: row offsets 3072 bytes apart, all with the swizzle phase of row `warp`
      const float* xg = P.x + (long long)grp * P.x_group_stride;
      const bool mine = P.ones_row % kTsTapWarps == warp;
      const int ones_i = mine ? P.ones_row / kTsTapWarps : -1;
      uint8_t* lane_ptr = base_ptr + warp * 128 + ((((lane >> 2) ^ (warp & 7)) << 4) + (lane & 3) * 4);
      const MaskTap* my_taps = s_taps + warp;
      float va[kTsRowsPerWarp];
      auto load_rows = [&]() {
        const bool ok = pix < P.n_pix;
        const int iy0 = pr * P.s - P.p, ix0 = pc * P.s - P.p;
        const float* xsrc = xg + (long long)pb * P.x_batch_stride + (long long)iy0 * P.n + ix0;
        const uint32_t mask =
            ok ? (kWgValidBit | bit_range(-iy0, min(P.k, P.n - iy0)) | (bit_range(-ix0, min(P.k, P.n - ix0)) << 16))
               : 0u;
#pragma unroll
        for (int i = 0; i < kTsRowsPerWarp; ++i) {
          const MaskTap tap = my_taps[kTsTapWarps * i];
          va[i] = ldg_if_bits(xsrc + tap.off, mask, tap.bits);
        }
        if (ones_i >= 0) {
#pragma unroll
          for (int i = 0; i < kTsRowsPerWarp; ++i) va[i] = i == ones_i ? (ok ? 1.f : 0.f) : va[i];
        }
      };
      load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
        const int s = ring.idx, use = ring.use;
        uint8_t* st = lane_ptr + (size_t)s * kTsStage;
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3010);
#pragma unroll
        for (int i = 0; i < kTsRowsPerWarp; ++i) {
          uint32_t h, l;
          split_tf32_trunc(va[i], h, l);
          uint8_t* dst = st + i * (kTsTapWarps * 128);
          *reinterpret_cast<uint32_t*>(dst) = h;
          *reinterpret_cast<uint32_t*>(dst + kTsTile) = l;
        }
        if (kbl + 1 < kblocks) {  // the next k-block's loads go in flight before the barrier work
          next_pixel();
          load_rows();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
    } else {
      // ---- dY: channels 32q .. 32q+31 of the tile; tensor-memory lanes of the same numbers.  With eight warps two share a
      // quadrant: each loads half of its channels and stores half of the pixels.
      constexpr int kHalves = kTsDyWarps / 4, kChannels = 32 / kHalves;
      const int q = warp & 3, half = (warp - kTsTapWarps) >> 2;  // a warp reaches the tensor-memory lanes of its number mod 4
      const int ch0 = q * 32 + half * kChannels;
      const float* dyg = P.dy + (long long)(grp * P.dy_group_channels + ntile * P.n_real + ch0) * P.mm;
      const int n_live = min(P.n_real, P.dy_group_channels - ntile * P.n_real);  // the last tile of a group may be shorter
      const int live = min(kChannels, max(0, n_live - ch0));  // real channels of this warp
      float* turn = reinterpret_cast<float*>(base_ptr + kTsTurnOff) + q * (32 * 33);
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + kACol0 + (uint32_t)(half * kChannels);
      auto quadrant_sync = [&]() {
        if (kHalves == 1) __syncwarp();
        else asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
      };
      float vb[kChannels];
      auto load_rows = [&]() {
        const bool ok = pix < P.n_pix;
        const float* dsrc = dyg + (long long)pb * P.dy_batch_stride + pr * P.m + pc;
        // one lane per channel: the line two k-blocks on
        if (WIDE && lane < live && pr * P.m + pc + 2 * kBlockK < P.mm && ok) prefetch_l2(dsrc + (long long)lane * P.mm + 2 * kBlockK - lane);
#pragma unroll
        for (int i = 0; i < kChannels; ++i) {
          if (WIDE) {
            vb[i] = ok && i < live ? __ldg(dsrc) : 0.f;
            dsrc += P.mm;
          } else {
            vb[i] = ldg_if(dsrc + (long long)i * P.mm, (ok && i < live) ? 1u : 0u);
          }
        }
      };
      load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
        const int s = ring.idx, use = ring.use;
#pragma unroll
        for (int i = 0; i < kChannels; ++i) turn[(half * kChannels + i) * 33 + lane] = vb[i];  // row = channel, column = pixel
        quadrant_sync();
        if (kbl + 1 < kblocks) {
          next_pixel();
          load_rows();
        }
        // The stage's 64 tensor-memory columns were last read by the MMAs of k-block kbl - 2.
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3011);
        tc_fence_after();
        const uint32_t st_addr = lane_addr + (uint32_t)(s * 64);
#pragma unroll
        for (int c = 0; c < kChannels / 8; ++c) {  // lane = channel now: its pixels, eight at a time
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) split_tf32_trunc(turn[lane * 33 + half * kChannels + c * 8 + e], hi[e], lo[e]);
          tmem_st8(st_addr + (uint32_t)(c * 8), hi);
          tmem_st8(st_addr + 32u + (uint32_t)(c * 8), lo);
        }
        tmem_wait_st();
        tc_fence_before();
        quadrant_sync();  // also: every lane has read the tile before the next k-block overwrites it
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
      // ---- epilogue: lane = channel, one accumulator column = one lowered row
      mbar_wait(acc_full, 0u, failed, P.status, 0x3020);
      tc_fence_after();
      const int ch = q * 32 + lane;
      float* op = P.partial + ((size_t)split * gridDim.z + vg) * kTsRows * P.n_pad + ch;
      for (int c = half; c < kTsRows / 16; c += kHalves) {
        float acc[16];
        tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 16), acc);
        if (!failed && ch < P.n_pad) {
#pragma unroll
          for (int j = 0; j < 16; ++j) op[(size_t)(c * 16 + j) * P.n_pad] = acc[j];
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ MMA issue (see elect_one)
    const uint32_t idesc = make_idesc(kTsNTile), tmem = warp_uniform(tmem_base);
    Ring ring;
    for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
      const int s = ring.idx;
      mbar_wait(full + 8u * s, (uint32_t)ring.use & 1u, failed, P.status, 0x3040);
      tc_fence_after();
      const uint32_t st = base + (uint32_t)s * kTsStage;
      const uint32_t a_hi = tmem + kACol0 + (uint32_t)(s * 64), a_lo = a_hi + 32u;
      if (elect_one()) {
#pragma unroll
        for (int u = 0; u < kTsRows / kTsNTile; ++u) {
          const uint32_t d_tmem = tmem + (uint32_t)(u * kTsNTile);
          const uint64_t dbh = make_desc(st + (uint32_t)u * kTsNTile * 128u), dbl = make_desc(st + kTsTile + (uint32_t)u * kTsNTile * 128u);
#pragma unroll
          for (int j = 0; j < kBlockK / 8; ++j) {
            const uint64_t adv = (uint64_t)(j * 2);
            umma_tf32_ts(d_tmem, a_lo + (uint32_t)(j * 8), dbh + adv, idesc, (kbl == 0 && j == 0) ? 0u : 1u);
            umma_tf32_ts(d_tmem, a_hi + (uint32_t)(j * 8), dbl + adv, idesc, 1u);
            umma_tf32_ts(d_tmem, a_hi + (uint32_t)(j * 8), dbh + adv, idesc, 1u);
          }
        }
        umma_commit(empty + 8u * s);
        if (kbl == kblocks - 1) umma_commit(acc_full);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// The same in pairs of fp16, for stride 4 (AlexNet / CaffeNet conv1).  A stage is 64 pixels: one row of 128 bytes per lowered row for the hi
// halves and one for the lo halves, so that a lane stores a whole word: it owns two neighbouring pixels, whose windows overlap - 15 of 22 elements
// of a window row, at most five aligned 16-byte loads for both where each alone took three or four.  24 MMAs of 96 cycles per 64 pixels instead of per
// 32, and half the stores.  Rows of an odd number of pixels have one more, so that neighbours are neighbours in memory: the last pair is the last two
// pixels, the first of them a second time with a dY of 0 (its window is that of a real pixel: a value that is not finite in it stays in its
// rows).  AlexNet conv1 at batch 256 358 -> 245 us (and 98 for the scales, which the data gradient shares).  The load-store pipe is 68 % busy then, a third
// of it the MMAs' reads, issue 58 %: with the kernel size known at run time there were twice the instructions for a tap (285 us); stages of 32 pixels,
// four of them, with half a warp to a window row, were slower (270: bank conflicts, registers).  The row of ones is not scaled.
constexpr int kThTapWarps = 18, kThDyWarps = 8, kThThreads = (kThTapWarps + kThDyWarps + 1) * 32, kThPixels = 64;  // 864
constexpr int kThWords = 20;  // five blocks: 13 taps and the neighbour's 4 more, at any alignment

// Taps 0 .. K - 1 of two pixels, which start at w[SHIFT] and four words on, to lowered rows `row`, `row` + 1 ..; at[x]: the lane's word in a row whose
// swizzle phase is x past that of the warp's first row, with `row`'s 128 bytes left to add.
template <int K, int SHIFT, int PHASE>
__device__ __forceinline__ void store_pairs(const float* w, uint8_t* row, const uint32_t* at, float scale) {
#pragma unroll
  for (int r = 0; r < K; ++r) {
    uint32_t h, l;
    split_half2(w[SHIFT + r] * scale, w[SHIFT + 4 + r] * scale, h, l);
    uint8_t* dst = row + at[(PHASE + r) & 7] + r * 128;
    *reinterpret_cast<uint32_t*>(dst) = h;
    *reinterpret_cast<uint32_t*>(dst + kTsTile) = l;
  }
}
template <int K, int PHASE>
__device__ __forceinline__ void store_shifted(const float* w, int shift, uint8_t* row, const uint32_t* at, float scale) {
  switch ((int)warp_uniform((uint32_t)shift)) {
    case 0: store_pairs<K, 0, PHASE>(w, row, at, scale); break;
    case 1: store_pairs<K, 1, PHASE>(w, row, at, scale); break;
    case 2: store_pairs<K, 2, PHASE>(w, row, at, scale); break;
    default: store_pairs<K, 3, PHASE>(w, row, at, scale); break;
  }
}

template <int K>
__global__ void __launch_bounds__(kThThreads, 1) wgrad_half_kernel(const __grid_constant__ WgradParams P) {
  constexpr int kMmaWarp = kThTapWarps + kThDyWarps;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t full = base + kTsBarsOff, empty = full + 8u * kTsStages, acc_full = empty + 8u * kTsStages, tmem_slot = acc_full + 8u;
  const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
  const int split = blockIdx.y, vg = blockIdx.z;
  const int grp = vg / P.tiles_per_group, ntile = vg % P.tiles_per_group;
  constexpr uint32_t kACol0 = 2 * kTsNTile;  // tensor memory: two accumulators of 192 columns, then 2 x 64 columns of A

  pdl_wait();
  if (!half_route(P.half, kHalfX, kHalfDy)) return;
  const HalfScale sx = P.half->of[kHalfX], sy = P.half->of[kHalfDy];
  for (int i = tid; i < (kTsRows - P.ones_row - 1) * 32 * 2 * kTsStages; i += kThThreads) {  // lowered rows that no warp stages: zeros
    const int words = (kTsRows - P.ones_row - 1) * 32, part = i / words;
    reinterpret_cast<uint32_t*>(base_ptr + (size_t)part * kTsTile + (size_t)(P.ones_row + 1) * 128)[i - part * words] = 0u;
  }
  for (int i = tid; i < 32 * kTsStages; i += kThThreads) {  // the row of ones (in pairs of fp16), which needs no swizzle
    uint8_t* at = base_ptr + (size_t)(i >> 5) * kTsStage + P.ones_row * 128 + (i & 31) * 4;
    *reinterpret_cast<uint32_t*>(at) = 0x3c003c00u;
    *reinterpret_cast<uint32_t*>(at + kTsTile) = 0u;
  }
  fence_proxy_async_smem();
  if (tid == 0) {
    for (int s = 0; s < kTsStages; ++s) { mbar_init(full + 8u * s, kThTapWarps + kThDyWarps); mbar_init(empty + 8u * s, 1); }
    mbar_init(acc_full, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  // k-blocks of 64 pixels over rows of `pitch`
  const int pitch = P.m + (P.m & 1), per_image = P.m * pitch, images = P.n_pix / P.mm;
  const int total = (images * per_image + kThPixels - 1) / kThPixels, per_split = (total + (int)gridDim.y - 1) / (int)gridDim.y;
  const int kb_begin = split * per_split, kblocks = max(0, min(total, kb_begin + per_split) - kb_begin);
  bool failed = false;

  if (warp < kMmaWarp) {
    // this lane's pixel (tap warps: the first of two), advanced by `step`
    int pb, pr, pc;
    auto set_pixel = [&](int pix) {
      pb = pix / per_image;
      const int in = pix - pb * per_image;
      pr = in / pitch;
      pc = in - pr * pitch;
    };
    auto next_pixel = [&](int step) {
      pc += step;
      while (pc >= pitch) { pc -= pitch; ++pr; }
      while (pr >= P.m) { pr -= P.m; ++pb; }
    };
    if (warp < kThTapWarps) {
      // ---- window rows u = 2 warp and 2 warp + 1: lowered rows u * K + kc
      set_pixel(kb_begin * kThPixels + 2 * lane);
      const int units = P.ones_row / K, mine = min(kTsWideRows, max(0, units - kTsWideRows * warp));
      const float* x = P.x + (long long)grp * P.x_group_stride;
      int unit_at[kTsWideRows];
#pragma unroll
      for (int i = 0; i < kTsWideRows; ++i) {
        const int u = kTsWideRows * warp + i, d = u / K;
        unit_at[i] = d * P.n * P.n + (u - d * K) * P.n;
      }
      uint32_t at[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) at[r] = (uint32_t)lane * 4u ^ (uint32_t)(((kTsWideRows * warp * K + r) & 7) << 4);
      uint8_t* row0 = base_ptr + kTsWideRows * warp * K * 128;
      const float scale = __uint_as_float(warp_uniform(__float_as_uint(sx.scale)));
      const int misaligned = (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3);  // words between x and its 16-byte block
      float w[kTsWideRows][kThWords];
      int shift[kTsWideRows] = {0, 0};
      auto load_rows = [&]() {
        const bool ok = pb < images;
        const int col = pc + 1 < P.m ? pc : pc - 1;  // the last pair of an odd row
        const int at0 = pb * (int)P.x_batch_stride + pr * 4 * P.n + col * 4;
        const int pb0 = __shfl_sync(0xffffffffu, pb, 0);
        const bool one_image = __all_sync(0xffffffffu, ok && pb == pb0);
        int far_r = pr, far_c = pc + 2 * kThPixels;  // the lines of the k-block after the next one, if it lies in the same image
        while (far_c >= pitch) { far_c -= pitch; ++far_r; }
        const bool far_in = ok && far_r < P.m && (lane & 3) == 0;
        const int far0 = pb * (int)P.x_batch_stride + far_r * 4 * P.n + far_c * 4;
#pragma unroll
        for (int i = 0; i < kTsWideRows; ++i) {
          if (i >= mine) break;
          const int from = at0 + unit_at[i];
          if (far_in) prefetch_l2(x + far0 + unit_at[i]);
          shift[i] = (from + misaligned) & 3;  // of this lane; of every lane where the pixels are one image's
          const int first = from - shift[i];
          if (__all_sync(0xffffffffu, one_image && first >= 0 && first + kThWords <= P.x_count)) {
            const float4* block = reinterpret_cast<const float4*>(x + first);
#pragma unroll
            for (int j = 0; j < (K + 4 + 3 + 3) / 4; ++j) {
              if (4 * j >= K + 4 && 4 * j >= K + 4 + shift[i]) break;
              const float4 v = __ldg(block + j);
              w[i][4 * j] = v.x; w[i][4 * j + 1] = v.y; w[i][4 * j + 2] = v.z; w[i][4 * j + 3] = v.w;
            }
          } else {
            shift[i] = 0;
#pragma unroll
            for (int r = 0; r < K + 4; ++r) w[i][r] = ok && from + r < P.x_count ? __ldg(x + from + r) : 0.f;
          }
        }
      };
      if (kblocks > 0) load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
        const int s = ring.idx, use = ring.use;
        if (use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3110);
        uint8_t* row = row0 + (size_t)s * kTsStage;
        if (mine > 0) store_shifted<K, 0>(w[0], shift[0], row, at, scale);
        if (mine > 1) store_shifted<K, K>(w[1], shift[1], row + K * 128, at, scale);
        if (kbl + 1 < kblocks) {  // the next k-block's loads go in flight before the barrier work
          next_pixel(kThPixels);
          load_rows();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
    } else {
      // ---- dY: two warps per quadrant of channels (= the tensor-memory lanes a warp reaches, its number mod 4); each loads half of the channels and
      // stores half of the pixels, 32 pixels at a time.
      constexpr int kChannels = 16;
      const int q = warp & 3, half = (warp - kThTapWarps) >> 2;
      set_pixel(kb_begin * kThPixels + lane);
      const int ch0 = q * 32 + half * kChannels;
      const float* dyg = P.dy + (long long)(grp * P.dy_group_channels + ntile * P.n_real + ch0) * P.mm;
      const int n_live = min(P.n_real, P.dy_group_channels - ntile * P.n_real);  // the last tile of a group may be shorter
      const int live = min(kChannels, max(0, n_live - ch0));  // real channels of this warp
      const bool any = n_live > q * 32;                       // of the quadrant
      float* turn = reinterpret_cast<float*>(base_ptr + kTsTurnOff) + q * (32 * 33);
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + kACol0 + (uint32_t)(half * 8);
      if (!any) {  // zeros, once
        const uint32_t zeros[8] = {};
        for (int c = 0; c < kTsStages * 4; ++c) tmem_st8(lane_addr + (uint32_t)(c * 16), zeros);
        tmem_wait_st();
      }
      auto quadrant_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory"); };
      float vb[kChannels];
      auto load_rows = [&]() {
        // of the last pair of an odd row the second is the last pixel
        const bool ok = pb < images && !(pc + 1 == P.m && pitch > P.m);
        const int col = pc == P.m ? pc - 1 : pc;
        const float* dsrc = dyg + (long long)pb * P.dy_batch_stride + pr * P.m + col;
        // one lane per channel: the line four blocks of 32 on
        if (lane < live && pr * P.m + col + 4 * kBlockK < P.mm && ok) prefetch_l2(dsrc + (long long)lane * P.mm + 4 * kBlockK - lane);
#pragma unroll
        for (int i = 0; i < kChannels; ++i) vb[i] = 0.f;
        if (ok && live == kChannels) {
#pragma unroll
          for (int i = 0; i < kChannels; ++i) vb[i] = __ldg(dsrc + (size_t)i * P.mm);
        } else if (ok) {
#pragma unroll
          for (int i = 0; i < kChannels; ++i)
            if (i < live) vb[i] = __ldg(dsrc + (size_t)i * P.mm);
        }
      };
      if (kblocks > 0 && any) load_rows();
      Ring ring;
      for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
        const int s = ring.idx, use = ring.use;
#pragma unroll 1
        for (int part = 0; any && part < 2; ++part) {  // 32 of the 64 pixels
#pragma unroll
          for (int i = 0; i < kChannels; ++i) turn[(half * kChannels + i) * 33 + lane] = vb[i];  // row = channel, column = pixel
          quadrant_sync();
          if (part == 0 || kbl + 1 < kblocks) {
            next_pixel(kBlockK);
            load_rows();
          }
          // The stage's 64 tensor-memory columns were last read by the MMAs of k-block kbl - 2.
          if (part == 0 && use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3111);
          tc_fence_after();
          uint32_t hi[8], lo[8];  // lane = channel now: sixteen of its pixels
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float* t = turn + lane * 33 + half * 16 + 2 * e;
            split_half2(t[0] * sy.scale, t[1] * sy.scale, hi[e], lo[e]);
          }
          const uint32_t st_addr = lane_addr + (uint32_t)(s * 64 + part * 16);
          tmem_st8(st_addr, hi);
          tmem_st8(st_addr + 32u, lo);
          quadrant_sync();  // every lane has read the tile before the next 32 pixels overwrite it
        }
        if (!any && use > 0) mbar_wait(empty + 8u * s, (uint32_t)(use - 1) & 1u, failed, P.status, 0x3112);  // (or the barrier would run ahead)
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8u * s);
      }
      // ---- epilogue: lane = channel, one accumulator column = one lowered row
      if (kblocks > 0) mbar_wait(acc_full, 0u, failed, P.status, 0x3120);
      tc_fence_after();
      const int ch = q * 32 + lane;
      float* op = P.partial + ((size_t)split * gridDim.z + vg) * kTsRows * P.n_pad + ch;
      for (int c = half; c < kTsRows / 16; c += 2) {
        float acc[16];
        tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 16), acc);
        if (!failed && ch < P.n_pad) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            op[(size_t)(c * 16 + j) * P.n_pad] = kblocks > 0 ? acc[j] * (c * 16 + j == P.ones_row ? sy.inverse : sx.inverse * sy.inverse) : 0.f;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ MMA issue (see elect_one)
    const uint32_t idesc = make_idesc_f16(kTsNTile), tmem = warp_uniform(tmem_base);
    Ring ring;
    for (int kbl = 0; kbl < kblocks; ++kbl, ring.advance(kTsStages)) {
      const int s = ring.idx;
      mbar_wait(full + 8u * s, (uint32_t)ring.use & 1u, failed, P.status, 0x3140);
      tc_fence_after();
      const uint32_t st = base + (uint32_t)s * kTsStage;
      const uint32_t a_hi = tmem + kACol0 + (uint32_t)(s * 64), a_lo = a_hi + 32u;
      if (elect_one()) {
#pragma unroll
        for (int u = 0; u < kTsRows / kTsNTile; ++u) {
          const uint32_t d_tmem = tmem + (uint32_t)(u * kTsNTile);
          const uint64_t dbh = make_desc(st + (uint32_t)u * kTsNTile * 128u), dbl = make_desc(st + kTsTile + (uint32_t)u * kTsNTile * 128u);
#pragma unroll
          for (int j = 0; j < kThPixels / 16; ++j) {
            const uint64_t adv = (uint64_t)(j * 2);
            umma_f16_ts(d_tmem, a_lo + (uint32_t)(j * 8), dbh + adv, idesc, (kbl == 0 && j == 0) ? 0u : 1u);
            umma_f16_ts(d_tmem, a_hi + (uint32_t)(j * 8), dbl + adv, idesc, 1u);
            umma_f16_ts(d_tmem, a_hi + (uint32_t)(j * 8), dbh + adv, idesc, 1u);
          }
        }
        umma_commit(empty + 8u * s);
        if (kbl == kblocks - 1) umma_commit(acc_full);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

typedef void (*WgradKernel)(const WgradParams);
template <int SUBS>
WgradKernel wgrad_pick_nb(int nb) {
  switch (nb) {
    case 1: return wgrad_kernel<SUBS, 1>;   case 2: return wgrad_kernel<SUBS, 2>;
    case 3: return wgrad_kernel<SUBS, 3>;   case 4: return wgrad_kernel<SUBS, 4>;
    case 5: return wgrad_kernel<SUBS, 5>;   case 6: return wgrad_kernel<SUBS, 6>;
    case 7: return wgrad_kernel<SUBS, 7>;   case 8: return wgrad_kernel<SUBS, 8>;
    case 9: return wgrad_kernel<SUBS, 9>;   case 10: return wgrad_kernel<SUBS, 10>;
    case 11: return wgrad_kernel<SUBS, 11>; case 12: return wgrad_kernel<SUBS, 12>;
    case 13: return wgrad_kernel<SUBS, 13>; case 14: return wgrad_kernel<SUBS, 14>;
    case 15: return wgrad_kernel<SUBS, 15>; case 16: return wgrad_kernel<SUBS, 16>;
  }
  return nullptr;
}
WgradKernel wgrad_pick(int subs, int n_pad) {
  return subs == 2 ? wgrad_pick_nb<2>(n_pad / 16) : wgrad_pick_nb<1>(n_pad / 16);
}

}  // namespace
#include "conv_small.cuh"
namespace {

// ------------------------------------------------------------------------------------------ weight packing
// A block writes one row of the packed operand (blockIdx.x = (vg, j): there may be more than 65 535 of them), four consecutive
// reduction indices per thread and step: one decode per four elements and 16-byte stores (a flat grid-stride loop spent most of its time dividing: CaffeNet
// conv3's 0.9 M weights 8.0 / 11.6 us for the two operands, bound by neither memory nor launch).
constexpr int kPackThreads = 128;

// Into the packed operand: pairs of tf32 in two halves, or (PAIRS, scale != 0) pairs of fp16 in the first (half_word).
template <bool PAIRS>
__device__ __forceinline__ void store_split4(float* hi, float* lo, size_t at, const float* v, float scale) {
  if (PAIRS && scale != 0.f) {
    uint2 h, l;
    split_half2(v[0] * scale, v[1] * scale, h.x, l.x);
    split_half2(v[2] * scale, v[3] * scale, h.y, l.y);
    *reinterpret_cast<uint2*>(hi + half_word(at)) = h;
    *reinterpret_cast<uint2*>(hi + half_word(at) + kHalfLo) = l;
    return;
  }
  float h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split_tf32(v[e], h[e], l[e]);
  *reinterpret_cast<float4*>(hi + at) = make_float4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4*>(lo + at) = make_float4(l[0], l[1], l[2], l[3]);
}

// Data-gradient B operand: [2][vg][n_pad][k_pad]; row j = (d, py, px) of channel tile nt of group g (py, px: position
// inside a block of s x s input pixels), column kk = (oc, jy, jx) <- W[g*og + oc][d][py + jy*s][px + jx*s], zero where the tap
// index is outside the kernel.
struct PackDgrad {
  const float* W;
  float *hi, *lo;
  int tiles_per_group, og, Dg, k, s, taps, d_tile, n_real, n_pad, k_real, k_pad, run;
  int parts;   // blocks per row
  int blocks;  // rows * parts
  const HalfScales* half;  // null: no data gradient by pairs of fp16
  int rows = 1;            // stride periods of a block of pixels along a column (GatherProblem)
  int only = kAny;
};
// The scale of weights that are packed as pairs of fp16 for a contraction with operand `other`, or 0.  (PAIRS, here and in the kernels below: a
// plan without them takes kernels without that code, whose registers the small ones would feel.)
template <bool PAIRS>
__device__ __forceinline__ float pack_scale(const HalfScales* half, int other) {
  return PAIRS && half_route(half, other, kHalfW) ? half->of[kHalfW].scale : 0.f;
}
template <bool PAIRS>
__device__ __forceinline__ void pack_dgrad_block(const PackDgrad& J, int block) {
  if (PAIRS && J.only != kAny && tall_route(J.half) != (J.only == kOnlyHalf)) return;
  const int periods = PAIRS ? J.rows : 1;
  const int r0 = block / J.parts, part = block - r0 * J.parts;
  const int vg = r0 / J.n_pad, j = r0 - vg * J.n_pad;
  const int grp = vg / J.tiles_per_group, d = (vg - grp * J.tiles_per_group) * J.d_tile + j / (periods * J.s * J.s);
  const int py = (j / J.s) % (periods * J.s) - (periods - 1) * J.s, px = j % J.s, window = (J.taps + periods - 1) * J.taps;
  const bool live = j < J.n_real && d < J.Dg;
  const float* src = J.W + ((size_t)grp * J.og * J.Dg + d) * J.k * J.k;
  const float scale = PAIRS && J.only == kOnlyTf32 ? 0.f : pack_scale<PAIRS>(J.half, kHalfDy);
  const size_t row = (size_t)r0 * J.k_pad;
  for (int kk = (part * (int)blockDim.x + (int)threadIdx.x) * 4; kk < J.k_pad; kk += J.parts * (int)blockDim.x * 4) {
    // reduction index -> (filter / run, jy, jx, filter % run); four in a row are four filters of one tap where run is kRun, and
    // one decode serves them (with one each the divisions bound the packing kernels)
    float v[4];
    const size_t filter = (size_t)J.Dg * J.k * J.k;
    if (J.run == kRun) {
      const int r = kk / kRun, chunk = r / window, tap = r - chunk * window;
      const int jy = tap / J.taps, kr = py + jy * J.s, kc = px + (tap - jy * J.taps) * J.s;
      const bool in = live && kk < J.k_real && (!PAIRS || kr >= 0) && kr < J.k && kc < J.k;
      const float* at = src + (size_t)(chunk * kRun + (kk & (kRun - 1))) * filter + kr * J.k + kc;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = in ? __ldg(at + e * filter) : 0.f;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int oc = (kk + e) / window, tap = kk + e - oc * window, jy = tap / J.taps;
        const int kr = py + jy * J.s, kc = px + (tap - jy * J.taps) * J.s;
        v[e] = (live && kk + e < J.k_real && (!PAIRS || kr >= 0) && kr < J.k && kc < J.k) ? __ldg(src + oc * filter + kr * J.k + kc) : 0.f;
      }
    }
    store_split4<PAIRS>(J.hi, J.lo, row + kk, v, scale);
  }
}
__global__ void __launch_bounds__(kPackThreads) pack_dgrad_kernel(const __grid_constant__ PackDgrad J) {
  pdl_wait();
  pack_dgrad_block<false>(J, blockIdx.x);
}

// db[c] = sum over the batch of the plane sums (ConvolutionBridge_impl.hxx:575-599), in a fixed order.
struct BiasSum {
  const float* plane_sums;
  float* db;
  int batch, channels;
  int blocks;
};
__device__ __forceinline__ void bias_grad_block(const BiasSum& J, int block) {
  // one warp per channel: lane l adds images l, l + 32, ... in order, then a fixed shuffle tree
  const int c = (int)((block * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (c >= J.channels) return;
  float t = 0.f;
  for (int b = lane; b < J.batch; b += 32) t += J.plane_sums[(size_t)b * J.channels + c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) J.db[c] = t;
}

// What else goes between the weight gradient and the data gradient of a layer, in blocks behind those that add the split sums:
// the weights are packed for the data gradient, the plane sums of dY are added to the bias gradient.  In launches of their own
// they were 2 - 7 and 2 - 3 us each, most of it the launch: ragged layer of 37 images 42.5 -> 40.5 us, CaffeNet's iteration at
// batch 32 1 214 -> 1 196.
struct ReduceExtras {
  PackDgrad pack;
  BiasSum bias;
};
struct HalfExtras : ReduceExtras {  // pairs of fp16; `tall`: the weights for tall blocks of pixels, if the data gradient has them
  PackDgrad tall;
};
// True if this block was one of them; `first` of the grid's x are not.
template <bool PAIRS>
__device__ __forceinline__ bool extra_block_of(const ReduceExtras& E, int first) {
  int block = (int)blockIdx.x - first;
  if (block < 0) return false;
  if (block < E.pack.blocks) {
    pack_dgrad_block<PAIRS>(E.pack, block);
    return true;
  }
  block -= E.pack.blocks;
  if (block < E.bias.blocks) bias_grad_block(E.bias, block);
  return true;
}
// A reduction with nothing beside it (small layers, whose gradients need neither) is a kernel without that code: with it a network
// of 10 images, two such reductions of 4 us in its iteration, took 88.0 us instead of 86.2.
struct NoExtras {};
__device__ __forceinline__ bool extra_block(const ReduceExtras& E, int first) { return extra_block_of<false>(E, first); }
__device__ __forceinline__ bool extra_block(const HalfExtras& E, int first) {
  const int block = (int)blockIdx.x - first;
  if (block < 0) return false;
  if (block < E.tall.blocks) pack_dgrad_block<true>(E.tall, block);
  else extra_block_of<true>(E, first + E.tall.blocks);
  return true;
}
__device__ __forceinline__ bool extra_block(const NoExtras&, int) { return false; }

// dW[o][kk] and db[o] from the split partial sums, added in split order (deterministic).  One block per 32 x 32
// tile of (kk, channel): the partial sums are read along the channels (their fastest index), the tile is turned in
// shared memory, and dW is written along kk (its fastest index) - both sides coalesced, no division per element.
template <class Extras>
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial, float* __restrict__ dW,
                                                           float* __restrict__ db, int splits, int vgroups,
                                                           int tiles_per_group, int rows_pad, int n_real, int n_pad,
                                                           int k_real, int og, int accumulate, int row_tiles, int col_tiles,
                                                           const __grid_constant__ Extras extras) {
  pdl_wait();
  __shared__ float tile[32][33];
  if (extra_block(extras, row_tiles * col_tiles * vgroups)) return;
  const int across = blockIdx.x / row_tiles, vg = across / col_tiles;
  const int kk0 = (blockIdx.x - across * row_tiles) * 32, j0 = (across - vg * col_tiles) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const int ch0 = (vg / tiles_per_group) * og + (vg % tiles_per_group) * n_real;
  n_real = min(n_real, og - (vg % tiles_per_group) * n_real);  // the last channel tile of a group may be shorter
  const size_t split_stride = (size_t)vgroups * rows_pad * n_pad;
  const int last = db ? k_real : k_real - 1;  // the bias row exists only where the kernel produced it
  // Eight splits of all four rows in flight: row by row each thread had four trips to L2 one behind the other.  With the blocks of
  // ReduceExtras, batch 256: CaffeNet conv2 59 -> 25 us, conv3 20 -> 15, conv4 20 -> 13, conv5 16 -> 10; batch 32 49 -> 38 for the four.
  const int j = min(j0 + tx, n_real - 1);  // a column or row too many repeats the last one's sums; they are not stored
  const float* src[4];
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int r = 0; r < 4; ++r) src[r] = partial + ((size_t)vg * rows_pad + min(kk0 + ty + 8 * r, last)) * n_pad + j;
#pragma unroll 8
  for (int s = 0; s < splits; ++s)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      acc[r] += __ldg(src[r]);
      src[r] += split_stride;
    }
#pragma unroll
  for (int r = 0; r < 4; ++r) tile[ty + 8 * r][tx] = acc[r];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int j = j0 + ty + 8 * r, kk = kk0 + tx;
    if (j < n_real && kk <= last) {
      const float v = tile[tx][ty + 8 * r];
      float* dst = kk < k_real ? dW + (size_t)(ch0 + j) * k_real + kk : db + ch0 + j;
      *dst = accumulate ? *dst + v : v;  // accumulate: a later round of splits adds to what the earlier rounds left
    }
  }
}

// The same reduction for small outputs, where 32 x 32 tiles would leave most SMs idle: a block owns 32 consecutive
// elements of the partial sums' (row, channel) plane and SLICES interleaved slices of the splits, the slice sums added in a
// fixed order - the result does not depend on the grid, and a thread's chain is splits / SLICES long.  dW is written
// without coalescing (a few ten thousand elements).
template <int SLICES, class Extras>
__global__ void __launch_bounds__(32 * SLICES) wgrad_reduce_flat_kernel(const float* __restrict__ partial,
                                                                        float* __restrict__ dW, float* __restrict__ db,
                                                                        int splits, int vgroups, int tiles_per_group,
                                                                        int rows_pad, int n_real, int n_pad, int k_real,
                                                                        int og, int accumulate, int per_group,
                                                                        const __grid_constant__ Extras extras) {
  pdl_wait();
  __shared__ float part[SLICES][33];
  if (extra_block(extras, per_group * vgroups)) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int vg = blockIdx.x / per_group, e = (blockIdx.x - vg * per_group) * 32 + tx;  // e = kk * n_pad + channel
  const size_t split_stride = (size_t)vgroups * rows_pad * n_pad;
  const bool in = e < (k_real + 1) * n_pad;
  float acc = 0.f;
  if (in) {
    const float* src = partial + (size_t)vg * rows_pad * n_pad + e;
#pragma unroll 8
    for (int s = ty; s < splits; s += SLICES) acc += src[(size_t)s * split_stride];
  }
  part[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && in) {
    const int kk = e / n_pad, j = e - kk * n_pad, first = (vg % tiles_per_group) * n_real;
    // the last channel tile of a group may be shorter; the bias row exists only where the kernel produced it
    if (j < min(n_real, og - first) && (kk < k_real || db)) {
      float t[4] = {0.f, 0.f, 0.f, 0.f};  // four short chains
#pragma unroll
      for (int y = 0; y < SLICES; ++y) t[y & 3] += part[y][tx];
      const int ch = (vg / tiles_per_group) * og + first + j;
      float* dst = kk < k_real ? dW + (size_t)ch * k_real + kk : db + ch;
      const float sum = (t[0] + t[1]) + (t[2] + t[3]);
      *dst = accumulate ? *dst + sum : sum;
    }
  }
}

// ------------------------------------------------------------------- dY as a pre-split TMA operand, bias sums
// dY[b][c][pix] -> hi / lo [row of channel c][b * mm + pix] with row = channel tile * n_pad + channel inside the
// tile (K-major rows of `row_len` floats, so a TMA box is 32 consecutive pixels x one channel tile), and the plane
// sum of dY[b][c] for the bias gradient.  One block per plane at a time; every access is a coalesced run.
__global__ void __launch_bounds__(256) split_dy_kernel(const float* __restrict__ dY, float* __restrict__ hi,
                                                       float* __restrict__ lo, float* __restrict__ plane_sums,
                                                       int planes, int channels, int mm, int og, int ch_tile,
                                                       int tiles_per_group, int n_pad, size_t row_len) {
  pdl_wait();
  // One warp per plane at a time in chunks of 256 elements, the next chunk's loads (of this plane or the warp's next one) in
  // flight while the current one is stored; no block-wide synchronisation.  One chunk at a time left planes of 169 elements at
  // 4.0 TB/s (CaffeNet conv3 at batch 256 50.0 -> 45.6 us, conv5 32.7 -> 30.5, conv2 at batch 32 11.7 -> 10.4; planes of 729 at batch 256
  // stay at 102 us, 5.6 TB/s).
  const int lane = threadIdx.x & 31;
  const int warp0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  if (warp0 >= planes) return;
  // Lane l takes the plane's elements whose DESTINATION is l floats into a 128-byte line (rows of the operand are
  // multiples of 32 floats, so only the image's offset b * mm matters): every warp-wide store then fills whole lines.
  // Stores that straddle lines run at about two thirds of the bandwidth on this part; loads do not care.
  struct Place {
    const float* src;
    size_t at;   // in hi and lo
    int i0, plane;
  };
  auto place = [&](int turn) {
    Place q;
    q.plane = planes - 1 - turn;  // what the kernel before wrote last is still in L2
    const int b = q.plane / channels, c = q.plane - b * channels;
    const int grp = c / og, j = c - grp * og;
    const int tile = j / ch_tile, within = j - tile * ch_tile;
    q.src = dY + (size_t)q.plane * mm;
    q.at = ((size_t)(grp * tiles_per_group + tile) * n_pad + within) * row_len + (size_t)b * mm;
    q.i0 = -(int)(((size_t)b * mm) & 31);
    return q;
  };
  float x[8], y[8];
  auto load = [&](const Place& q, float* v) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = q.i0 + u * 32 + lane;
      v[u] = (i >= 0 && i < mm) ? __ldg(q.src + i) : 0.f;
    }
  };
  Place q = place(warp0);
  load(q, x);
  float sum = 0.f;
  for (int turn = warp0;;) {
    Place next = q;
    const bool plane_ends = q.i0 + 256 >= mm;
    if (plane_ends) {
      turn += nwarps;
      if (turn < planes) next = place(turn);
    } else {
      next.i0 += 256;
    }
    if (turn < planes) load(next, y);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = q.i0 + u * 32 + lane;
      uint32_t h, l;
      split_tf32_trunc(x[u], h, l);
      if (i >= 0 && i < mm) {
        hi[q.at + i] = __uint_as_float(h);
        lo[q.at + i] = __uint_as_float(l);
      }
      sum += x[u];
    }
    if (plane_ends) {
      if (plane_sums) {  // fixed-shape reduction: the result does not depend on the grid
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) plane_sums[q.plane] = sum;
      }
      sum = 0.f;
      if (turn >= planes) break;
    }
    q = next;
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = y[u];
  }
}

// The same by runs of a channel's row, whatever images they are of: a warp writes `len` consecutive elements, two to a lane - whole lines of the rows and no
// lane without work (by planes of 169 elements a third had none: CaffeNet conv3, batch 256, in pairs of fp16 48 -> 25 us), and as many warps as there
// are runs (2 images, 64 channels 112 x 112: 128 planes 29.1 us, runs 5.3).  With `half`, and X and dY ok, pairs of fp16 in place of the low parts, and no
// values.  The sums for the bias gradient are those of the runs, [run][channel].  The rows' ends behind the last image are written too (0): what another
// form has left there meets zeros, but may read as Inf.
// Many large planes stay with the other kernel where there are no pairs: 32 images, 256 channels 27 x 27 13.0 us, here 13.8; and so do layers whose gradient a
// pooling layer could write (tiles of channels without padding).
constexpr int kSplitRun = 1024, kSplitAhead = 4, kSplitRunLeast = 64 * kSplitAhead;
bool split_by_planes(int planes, int mm) { return planes >= 4096 && mm >= 512; }
int split_run(int channels, size_t row_len, int sms) {
  int len = kSplitRun;  // shorter ones until every SM has sixteen warps
  while (len > kSplitRunLeast && channels * (double)row_len < 16.0 * sms * len) len /= 2;
  return len;
}
__global__ void __launch_bounds__(256) split_dy_runs_kernel(const float* __restrict__ dY, float* __restrict__ hi, float* __restrict__ lo,
                                                            float* __restrict__ run_sums, int batch, int channels, int mm, int og,
                                                            int ch_tile, int tiles_per_group, int n_pad, size_t row_len, int runs, int len,
                                                            const HalfScales* half) {
  pdl_wait();
  const bool pairs = half_route(half, kHalfX, kHalfDy);
  const float scale = pairs ? half->of[kHalfDy].scale : 1.f;
  const int lane = threadIdx.x & 31, item = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (item >= channels * runs) return;
  const int c = item / runs, run = item - c * runs;
  const int grp = c / og, j = c - grp * og, tile = j / ch_tile;
  const size_t row = ((size_t)(grp * tiles_per_group + tile) * n_pad + (j - tile * ch_tile)) * row_len;
  const unsigned first = (unsigned)run * len + 2u * lane, end = (unsigned)min((size_t)(run + 1) * len, row_len);
  // this lane's first element: image, place in the plane
  int b = (int)(first / (unsigned)mm), r = (int)(first - (unsigned)b * mm);
  const size_t image = (size_t)channels * mm;
  const float* src = dY + (size_t)b * image + (size_t)c * mm;
  float sum = 0.f;
  for (unsigned q = first; q - 2u * lane < end; q += 64 * kSplitAhead) {
    float x[kSplitAhead][2];
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      const bool wraps = r + 1 == mm;  // the second element is the next image's first
      x[u][0] = b < batch ? __ldg(src + r) : 0.f;
      x[u][1] = b + (wraps ? 1 : 0) < batch ? __ldg(wraps ? src + image : src + r + 1) : 0.f;
      r += 64;
      while (r >= mm) { r -= mm; ++b; src += image; }
    }
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      const unsigned at = q + 64u * u;
      if (at >= end) continue;  // (whole rows of 32: both elements, half a warp)
      if (pairs) {
        uint32_t h, l;
        split_half2(x[u][0] * scale, x[u][1] * scale, h, l);
        uint32_t* word = reinterpret_cast<uint32_t*>(lo + row + half_word(at));
        word[0] = h;
        word[kHalfLo] = l;
      } else {
        uint32_t h[2], l[2];
        split_tf32_trunc(x[u][0], h[0], l[0]);
        split_tf32_trunc(x[u][1], h[1], l[1]);
        *reinterpret_cast<uint2*>(hi + row + at) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2*>(lo + row + at) = make_uint2(l[0], l[1]);
      }
      sum += x[u][0];
      sum += x[u][1];
    }
  }
  if (run_sums) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) run_sums[(size_t)run * channels + c] = sum;
  }
}

// Forward B operand: [2 (hi, lo)][vg][n_pad][k_pad] <- W[o][Dg*k*k], zero padded.
template <bool PAIRS>
__global__ void __launch_bounds__(kPackThreads) pack_fwd_kernel(const float* __restrict__ W, float* __restrict__ hi,
                                                                float* __restrict__ lo, int tiles_per_group, int og,
                                                                int n_real, int n_pad, int k_real, int k_pad, int run,
                                                                int window, const HalfScales* half) {
  pdl_wait();
  const float scale = pack_scale<PAIRS>(half, kHalfX);
  const int vg = blockIdx.x / n_pad, j = blockIdx.x - vg * n_pad;
  const int ch = (vg % tiles_per_group) * n_real + j;  // inside the group
  const bool live = j < n_real && ch < og;
  const float* src = W + (size_t)((vg / tiles_per_group) * og + ch) * k_real;
  const size_t row = (size_t)blockIdx.x * k_pad;
  for (int kk = (blockIdx.y * kPackThreads + threadIdx.x) * 4; kk < k_pad; kk += gridDim.y * kPackThreads * 4) {
    // reduction index -> (channel / run, tap, channel % run) -> element (channel, tap) of the filter, one decode for four
    float v[4];
    const int r = kk / kRun, chunk = r / window;
    const int at = run == 1 ? kk : (chunk * kRun + (kk & (kRun - 1))) * window + (r - chunk * window), step = run == 1 ? 1 : window;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = (live && kk + e < k_real) ? __ldg(src + at + e * step) : 0.f;
    store_split4<PAIRS>(hi, lo, row + kk, v, scale);
  }
}

size_t elements_x(const ConvGeom& G) { return (size_t)G.B * G.D * G.n * G.n; }
size_t elements_y(const ConvGeom& G) { return (size_t)G.B * G.o * G.m * G.m; }
size_t elements_w(const ConvGeom& G) { return (size_t)G.o * G.Dg * G.k * G.k; }

int round_up(int v, int a) { return (v + a - 1) / a * a; }

// Fewest channel tiles of at most 256 accumulator columns each (0: one channel alone is wider).
int channel_tiles(int channels, int cols_per_channel) {
  return cols_per_channel > 256 ? 0 : (channels + 256 / cols_per_channel - 1) / (256 / cols_per_channel);
}

// Fewest equal channel tiles of at most 256 accumulator columns each (`channels` where there is nothing better).
int even_tiles(int channels, int cols_per_channel) {
  int t = 1;
  while (t < channels && (channels % t || channels / t * cols_per_channel > 256)) ++t;
  return t;
}
// Channel tiles of the weight gradient, and the longest accumulation chain of its partial sums in k-blocks: the widest tiles,
// even ones unless they are many - uneven tiles are wider and leave fewer splits (375 channels: three tiles of 125 with chains
// of 38 k-blocks against two of 188 with 50).  Where only narrow even tiles exist (337 channels: 337 of one) the wide uneven
// ones, with three additions per eight products, get chains a third as long.
int weight_grad_tiles(int channels, int* chain) {
  const int even = even_tiles(channels, 1), widest = channel_tiles(channels, 1);
  *chain = even <= 2 * widest ? kMaxChainKblocks : kMaxChainKblocks / 3;
  return even <= 2 * widest ? even : widest;
}
// How long an accumulation chain of the forward pass or the data gradient may get, in k-blocks with one truncating addition
// at full magnitude per eight products (a tile of more than kCrossCols columns has three): twice the reduction's k-blocks
// where even channel tiles have at most kCrossCols columns, three times otherwise.  Tilings are chosen by time among those
// that stay within it: no layer is computed less accurately for the sake of a faster tile.
double chain_limit(int channels, int cols_per_channel, int kblocks) {
  return kblocks * (round_up(channels / even_tiles(channels, cols_per_channel) * cols_per_channel, 16) <= kCrossCols ? 2.0 : 3.0);
}

// Weight slots (hi and lo tile each) of a gather problem in shared memory: up to four.
int gather_slots(int n_pad, int taps_smem, int n_bias, int ptab, size_t limit) {
  int b = 4;
  while (b > 1 && gather_smem(n_pad, taps_smem, b, n_bias, ptab).total + 1024 > limit) --b;
  return b;
}
// Accumulators of at most 128 columns leave room for two CTAs per SM: 256 columns each (accumulator + two A slots) and half
// the shared memory (the SM holds 228 KB, 1 KB of it reserved per resident CTA).  Three weight slots per CTA, or two when
// the accumulator is the full 128 columns (each MMA then lasts long enough to cover the refill: CaffeNet conv5 forward
// 0.189 -> 0.153 ms).
bool two_ctas_per_sm(int n_pad, int taps_smem, int n_bias, int ptab, int* slots) {
  *slots = gather_slots(n_pad, taps_smem, n_bias, ptab, 113 * 1024);
  return n_pad <= 128 && (*slots >= 3 || (*slots == 2 && n_pad == 128));
}

// Channel tiles and splits of the reduction for the forward pass and the data gradient, by an estimate of the kernel's
// time in microseconds.  A work unit is (pixel tile, channel tile, split); units are spread over the resident CTAs in whole
// rounds.  The constants are a fit to 754 measured combinations of tiles and splits (CaffeNet's layers at batch 1 to 128 and
// layers of 20 to 384 channels; 6 % rms): what a k-block takes grows with the accumulator's columns, below that stands what the
// gather takes; a unit adds its set-up and epilogue, a split reduction one more kernel and the traffic of the sums.  So: a
// last round that is nearly empty (CaffeNet conv3 at batch 256: 2 x 338 units on 148 CTAs are five rounds, 3 x 338 half-width
// ones on 296 are 3.4) asks for narrower tiles, a layer of few pixels (43 tiles at batch 32, 2 at batch 1) for narrower tiles
// and splits.  A candidate has to win by 1 % and to keep its accumulation chain within `limit` (chain_limit).
// `half`: the same for operands in pairs of fp16, from 654 measured combinations (layers of 20 to 384 channels, batch 16 to 256; 6 % rms): a
// k-block of a tile of up to 128 columns is bound by its gather, so wide tiles are the better ones (CaffeNet conv3 at batch 256, 384
// columns in three tiles 167 us, in two 150); an MMA of more takes the time of the next multiple of 64.
struct GatherTiling {
  int tiles = 0, splits = 1, kps = 0;
  double us = 0.0;
  double chain = 0.0;  // additions at full magnitude, a quarter of them: one per eight products or three (chain_limit); pairs of fp16 have half as many
  bool cross = false;  // pairs of fp16: a second accumulator for the cross terms
};
GatherTiling choose_gather_tiling(int sms, long long pixel_tiles, int groups, int channels, int cols_per_channel, int kblocks,
                                  int run, int lane_stride, int n_bias, double limit, bool half, double half_limit = 0.0,
                                  int most_splits = 32) {
  GatherTiling best;
  const int t0 = channel_tiles(channels, cols_per_channel);
  for (int t = t0; t > 0 && t <= channels; ++t) {
    const int n_pad = round_up((channels + t - 1) / t * cols_per_channel, 16);
    if (t > t0 && n_pad < 32) break;
    if ((channels + t - 1) / t * (t - 1) >= channels) continue;  // the last tile would be empty
    int slots_unused;
    const bool two = two_ctas_per_sm(n_pad, kblocks * kBlockK / run, n_bias, 0, &slots_unused);
    // a k-block of a CTA that shares its SM, of one that has the SM to itself, of the shape with one CTA per SM
    const double far = lane_stride > 2 ? 1.7 : 1.0;  // lanes 16 bytes and more apart: four wavefronts and more per load
    const double shared = 2 * (half ? std::max(0.241 + 0.00053 * n_pad, (run > 1 ? 0.24 : 0.318) * far)
                                    : std::max(0.11 + 0.0028 * n_pad, (run > 1 ? 0.235 : 0.30) * far));
    const double alone = half ? (run > 1 ? 0.279 : 0.348) * far : std::max(0.19 + 0.0018 * n_pad, 0.27 * far);
    const double one = half ? std::max(0.00191 * round_up(n_pad, 64) - 0.039, (run > 1 ? 0.25 : 0.312) * far) : std::max(0.0035 * n_pad, 0.42 * far);
    const double epilogue = half ? 2.1 + 0.0184 * n_pad : 4.0 + 0.004 * n_pad, start = half ? 5.9 : 2.6;
    for (int s = 1; s <= std::max(1, std::min(most_splits, kblocks / 2)); ++s) {
      const int kps = (kblocks + s - 1) / s;
      const double chain = kps * (n_pad <= kCrossCols ? 1.0 : 3.0);
      if ((kblocks + kps - 1) / kps != s || (limit && chain > limit)) continue;
      // Pairs of fp16 are no less accurate than what tf32 would do here: wide tiles take a second accumulator where they have to and there is
      // room for it beside four A slots (two of a CTA that shares its SM).
      const bool cross = half && n_pad > kCrossCols && chain / 2 > half_limit;
      if (half && chain / (cross ? 6 : 2) > half_limit) continue;
      if (cross && 2 * n_pad > (two ? 256 - 64 : 512 - 128)) continue;
      const long long units = pixel_tiles * groups * t * s, slots = (long long)sms * (two ? 2 : 1), tail = units % slots;
      const double overlapped = cross ? 1.0 : half ? 0.65 : 0.4;  // of the epilogue that is not (cross: one accumulator buffer)
      double us = (double)(units / slots) * (kps * (two ? shared : one) + overlapped * epilogue) +
                  (tail ? kps * (!two ? one : tail > sms ? shared : alone) + epilogue : (1 - overlapped) * epilogue) + start;
      if (s > 1) us += (half ? 1.4 : 3.8) + units * 128.0 * n_pad * 4.0 * (half ? 0.284e-6 : 0.18e-6);
      if (!best.tiles || us < 0.99 * best.us) best = GatherTiling{t, s, kps, us, chain, cross};
    }
  }
  return best;
}

// What a launch of operand_scale_kernel over `elements` takes: 5.6 us for CaffeNet conv3's X and W at batch 32 (9 MB), 8.4 for X, dY and W
// of conv4 (14 MB), 58 for those of conv2 at batch 256 (265 MB).
// A contraction takes pairs of fp16 from kHalfMinUs on, if by the estimates (6 % rms) they save 1 - kHalfGain of it and kHalfLeastUs: operands that do not
// lie close enough together pay for the look at them and gain nothing.
// Blocks of several stride periods: for at least 1 - kTallGain of the data gradient; kTallUs: one launch more, which returns at once.
constexpr int kMaxTallRows = 4;
constexpr double kTallUs = 4.0, kTallGain = 0.93;
constexpr double kHalfMinUs = 25.0, kHalfGain = 0.95, kHalfLeastUs = 5.0;
bool half_pays(double us, double saves) { return us > kHalfMinUs && saves > (1 - kHalfGain) * us && saves > kHalfLeastUs; }
// Lowered matrices of 257 .. 384 rows (with the row of ones) and tiles of at most 128 filters: wgrad_ts_kernel; its wide loads: see there.  Below
// eight taps a window row has fewer than three blocks' worth.  With stride 4 wgrad_half_kernel.
bool ts_rows(int rows, int columns) { return round_up(rows + 1, kTileM) == kTsRows && columns <= kTileM; }
bool ts_wide(const ConvGeom& G) {
  return G.s % 4 == 0 && G.p == 0 && G.k >= 8 && G.k <= kTsWideTaps && G.Dg * G.k <= kTsWideRows * ts_tap_warps(true);
}
WgradKernel half_ts_kernel(int k) {
  switch (k) {
    case 8: return wgrad_half_kernel<8>;    case 9: return wgrad_half_kernel<9>;    case 10: return wgrad_half_kernel<10>;
    case 11: return wgrad_half_kernel<11>;  case 12: return wgrad_half_kernel<12>;  default: return wgrad_half_kernel<13>;
  }
}
bool half_ts(const ConvGeom& G, int rows, int columns) { return ts_rows(rows, columns) && ts_wide(G) && G.s == 4 && G.m > 1; }
int wgrad_columns(const ConvGeom& G) {
  int chain;
  const int tiles = weight_grad_tiles(G.og, &chain);
  return round_up((G.og + tiles - 1) / tiles, 16);
}
// From how many lowered rows on the weight gradient goes through the gather kernel, which needs dY in rows: see umma_plan_create; and in pairs of
// fp16, whose MMAs the short kernels' staging from shared memory would not keep up with.
constexpr int kGatherRows = 512, kGatherHalfRows = 320;
bool half_gather(const ConvGeom& G, int rows, int columns) { return rows >= kGatherRows || (rows >= kGatherHalfRows && !ts_rows(rows, columns) && columns > 96); }
// What the weight gradient takes (us), and what pairs of fp16 save of it.  By the gather kernel, more than 128 columns: conv3, conv4 at batch 256 253 -> 165
// us, 210 -> 138, at batch 32 44 -> 31; 128 columns, bound by the gather: conv2 425 -> 345, conv5 159 -> 138, at batch 32 65 -> 62, 64 -> 128
// channels 56 x 56 50 -> 45.  With fewer rows than kGatherRows dY is turned into rows for it: 48 -> 192 channels 28 x 28, 64 images (432 rows) 73 -> 34 + 16,
// 40 -> 370 30 x 30, 50 images (360) 97 -> 44 + 24, 16 -> 128 40 x 40 5 x 5, 100 images (400) 127 -> 69 + 28; 24 -> 296, 72 x 72 by 2, 30 images (216)
// 51 -> 34 + 17: no.  wgrad_half_kernel: AlexNet conv1 at batch 256 358 -> 245.
struct WgradTime {
  double us, saves;
};
WgradTime weight_gradient_time(const ConvGeom& G, int rows, int columns) {
  const double flops = 2.0 * elements_w(G) * G.B * G.m * G.m;
  if (half_ts(G, rows, columns)) return {flops / 152e6, 0.31 * flops / 152e6};
  if (rows >= kGatherRows) return {flops / 230e6, (columns > 128 ? 0.3 : columns > 96 ? 0.1 : 0.0) * flops / 230e6};
  const double us = flops / 125e6;
  return {us, half_gather(G, rows, columns) ? 0.45 * us - 3.0 - elements_y(G) * 8.0 / 5e6 : 0.0};
}
double scales_us(double elements) { return 4.0 + 4.0 * elements / 4.8e6; }

}  // namespace

// One gather problem (forward, or the data gradient): tables, packed weights and their tensor map.
struct GatherProblem {
  int tiles = 1, ch_tile = 0;  // channel tiles per group, channels per tile
  int n = 0, n_pad = 0, k_real = 0, k_pad = 0;
  MaskTap* taps = nullptr;
  ColEnt* cols = nullptr;
  float* w = nullptr;  // [2][vgroups][n_pad][k_pad]
  size_t w_half = 0;   // elements in one half
  CUtensorMap map;
  int a_stages = 4, b_stages = 4, acc_bufs = 1;
  int sets = 4, tmem_cols = 512;  // kernel shape: 4 producer sets and one CTA per SM, or 2 sets and two CTAs per SM
  int taps_smem = -1;             // tap-table entries staged in shared memory (-1: k_pad)
  size_t map_k = 0;               // extent of the packed operand along the reduction (0: k_pad)
  size_t smem = 0;
  bool half = false;              // HALF
  // Data gradient: stride periods of rows in a block of pixels that share what they gather (their columns stand side by side in the
  // accumulator).  Taps that one of the pixels does not have are products with zero weights, so blocks of several periods take finite values alone
  // (tall_route), and only in pairs of fp16, whose MMAs have the time for that.  CaffeNet conv2 (48 columns, three rows 144) at batch 256 502 -> 380 us,
  // at 128 268 -> 205; 20 -> 50 channels 24 x 24, 256 images, four rows 108 -> 55.  Bound by the MMAs then (tensor pipe 71 % active; 144 columns take
  // the time of 192, the zero weights 2 / 7 of it) and a last round of units.
  int rows = 1;
  bool half_cross = false;        // a second accumulator for the cross terms there too
  int a_stages_half = 4, b_stages_half = 4, acc_bufs_half = 1, acc_cols_half = 0;
  float* zero = nullptr;          // one 0.f, read by taps out of bounds
  bool inside = false;            // kInside
  bool one = false;               // ONE: the tiles of the whole batch are short and have a slot each, if no SMs are kept
  int run = 1, run_stride = 0;    // reduction order: 1 = (channel, tap); kRun = (channel / kRun, tap, channel % kRun)
  int splits = 1, split_k = 0;    // splits of the reduction and the length of one (a multiple of 32; k_pad without splits)
  float* partial = nullptr;       // split sums
  size_t pix_pad = 0;
  int taps_y = 0, q_h = 0, q0 = 0;  // rows > 1: taps along a column, blocks of pixels along it and the first that holds a pixel
  int small_ct = 0;               // > 0: small_conv_kernel with this many channels per block instead of gather_conv_kernel
};

struct UmmaPlan {
  ConvGeom G;
  GatherProblem fwd, dgr;
  GatherProblem tall;  // the data gradient by blocks of several stride periods (rows > 1), where that is faster: dgr is for the calls it does not take
  MaskTap* tall_row_taps = nullptr;  // as dgr_row_taps
  // data gradient: taps per axis of one stride period; super-pixels of s x s pixels, how many per axis and the first that
  // holds a pixel
  int dgr_taps = 0, dgr_q = 0, dgr_q0 = 0;
  // weight gradient: channel tiles per group, channels per tile (the last one may be shorter), padded to 16; longest
  // accumulation chain in k-blocks
  int wt_tiles = 1, wt_n = 0, w_chain = kMaxChainKblocks;
  int w_mtiles, w_subs, w_stages, w_mgroups, w_splits, w_kblocks_total, w_kblocks_per_split, w_npad;
  size_t w_smem = 0;
  bool w_small = false;             // weight gradient by small_wgrad_kernel
  int ws_rows = 0, ws_cols = 0, ws_pix = 0;  // its row tiles, channel tiles and pixels per split
  bool w_half = false;              // weight gradient in pairs of fp16 (wgp.half, or wgrad_half_kernel in place of wgrad_ts_kernel)
  bool w_ts = false;  // weight gradient by wgrad_ts_kernel (dY through tensor memory) instead of wgrad_kernel
  MaskTap* w_taps = nullptr;
  float* w_partial = nullptr;
  // weight gradient through the gather kernel: lanes = rows of the lowered matrix, reduction over pixels, dY as the
  // pre-split TMA operand [hi|lo][channel tile][channel][pixel]
  bool wg_gather = false;
  GatherProblem wgp;
  MaskTap* dgr_row_taps = nullptr; // the data gradient's table for a dY in rows (DyRows), where that can be
  MaskTap* wg_pix = nullptr;       // per pixel: offset of the tap origin, taps out of bounds (padded to splits * kps * 32)
  float* wg_plane_sums = nullptr;  // [batch][channel] sums of dY for the bias gradient
  int wg_splits = 1, wg_kps = 1, wg_mtiles = 1;
  HalfScales* half = nullptr;      // scales of the operands, by kHalfX and so on
  uint2* half_parts = nullptr;
  uint32_t* half_ticket = nullptr;
  void* memory = nullptr;          // everything above that lives on the device (PlanMemory)
  size_t bytes = 0;
};

namespace {
typedef void (*GatherKernel)(const GatherParams, const CUtensorMap);
template <int FORM, bool ONE = false>
GatherKernel gather_kernel_of(const GatherProblem& gp) {
  return gp.sets == 2 ? gather_conv_kernel<2, FORM, ONE> : gather_conv_kernel<4, FORM, ONE>;
}
GatherKernel gather_kernel(const GatherProblem& gp, bool weight_grad, bool one, bool half) {
  if (half) {
    if (weight_grad) return gather_kernel_of<kHalf + kWeightGrad>(gp);
    if (gp.rows > 1) return gp.run == kRun ? gather_kernel_of<kTall + kHalf + kByRun>(gp) : gather_kernel_of<kTall + kHalf + kByTap>(gp);
    return gp.run == kRun ? gather_kernel_of<kHalf + kByRun>(gp) : gather_kernel_of<kHalf + kByTap>(gp);
  }
  if (weight_grad) return gather_kernel_of<kWeightGrad>(gp);
  if (gp.run == kRun) return one ? gather_kernel_of<kByRun, true>(gp) : gather_kernel_of<kByRun>(gp);
  if (gp.inside) return gather_kernel_of<kInside>(gp);
  return one ? gather_kernel_of<kByTap, true>(gp) : gather_kernel_of<kByTap>(gp);
}
int gather_smem_limit(const GatherProblem& gp) { return gp.sets == 2 ? 113 * 1024 : kSmemLimit; }
WgradKernel short_wgrad_kernel(const UmmaPlan* p) {
  if (!p->w_ts) return wgrad_pick(p->w_subs, p->w_npad);
  return ts_wide(p->G) ? wgrad_ts_kernel<true> : wgrad_ts_kernel<false>;
}
}  // namespace

bool umma_supported(const ConvGeom& G) {
  if (channel_tiles(G.og, 1) == 0 || channel_tiles(G.Dg, G.s * G.s) == 0) return false;
  if (G.k > kMaxTapsPerAxis || G.n > 8000) return false;  // tap rows / columns are bits of a 32-bit validity mask
  const int taps = (G.k + G.s - 1) / G.s;
  const long long kf = (long long)G.Dg * G.k * G.k, kd = (long long)G.og * taps * taps;
  if (kf > 16384 || kd > 16384) return false;  // the tap table lives in shared memory next to the weight stages
  return true;
}

namespace {

// The plan's device memory: everything a plan owns is one allocation (an allocation and its release cost some eighty
// microseconds each, a plan has up to eleven buffers), laid out first and obtained at the end.
struct PlanMemory {
  struct Part { void** slot; size_t off; bool table; };
  std::vector<Part> parts;
  std::vector<unsigned char> tables;  // contents of the tables, in their layout
  size_t room_bytes = 0;
  static size_t aligned(size_t v) { return (v + 255) & ~(size_t)255; }
  template <class T>
  void table(T** slot, const std::vector<T>& host) {
    const size_t at = tables.size();
    tables.resize(aligned(at + host.size() * sizeof(T)));
    std::copy_n(reinterpret_cast<const unsigned char*>(host.data()), host.size() * sizeof(T), tables.data() + at);
    parts.push_back({(void**)slot, at, true});
  }
  template <class T>
  void room(T** slot, size_t count) {
    parts.push_back({(void**)slot, room_bytes, false});
    room_bytes = aligned(room_bytes + count * sizeof(T));
  }
  int obtain(cct_ctx* ctx, void** memory, size_t* bytes) {
    unsigned char* base = nullptr;
    CCT_CUDA(ctx, cudaMalloc((void**)&base, tables.size() + room_bytes));
    *memory = base;
    *bytes = tables.size() + room_bytes;
    CCT_CUDA(ctx, cudaMemcpy(base, tables.data(), tables.size(), cudaMemcpyHostToDevice));
    for (const Part& p : parts) *p.slot = base + (p.table ? 0 : tables.size()) + p.off;
    return CCT_OK;
  }
};

template <class K>
int set_smem(cct_ctx* ctx, K kernel, size_t bytes) {
  CCT_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return CCT_OK;
}

// Blocks that go with a reduction; those of the bias gradient are counted here, for the block size that is taken.
int extra_blocks(ReduceExtras& E, int threads) {
  if (E.bias.db) E.bias.blocks = (E.bias.channels + threads / 32 - 1) / (threads / 32);
  return E.pack.blocks + E.bias.blocks;
}
int extra_blocks(HalfExtras& E, int threads) { return E.tall.blocks + extra_blocks(static_cast<ReduceExtras&>(E), threads); }
int extra_blocks(NoExtras&, int) { return 0; }

// Split reduction: tiles when they fill the machine, the flat form otherwise (both add in a fixed order).
template <class Extras>
void launch_wgrad_reduce(cct_ctx* ctx, const float* partial, float* dW, float* db, int splits, int vgroups, int tiles_per_group,
                         int rows_pad, int n_real, int n_pad, int k_real, int og, int accumulate, Extras extras) {
  auto go = [&](auto kernel, int threads, int blocks, auto... shape) {
    blocks += extra_blocks(extras, threads);
    launch_pdl(kernel, dim3(blocks), dim3(threads), 0, ctx->stream, partial, dW, db, splits, vgroups, tiles_per_group, rows_pad, n_real,
               n_pad, k_real, og, accumulate, shape..., extras);
  };
  const int row_tiles = (k_real + 1 + 31) / 32, col_tiles = (n_real + 31) / 32, per_group = ((k_real + 1) * n_pad + 31) / 32;
  const int tiles = row_tiles * col_tiles * vgroups, flat = per_group * vgroups;
  if (tiles >= ctx->sm_count) go(wgrad_reduce_kernel<Extras>, 256, tiles, row_tiles, col_tiles);
  else if (splits < 16) go(wgrad_reduce_flat_kernel<4, Extras>, 128, flat, per_group);
  else if (splits < 64 || flat > 2 * ctx->sm_count) go(wgrad_reduce_flat_kernel<8, Extras>, 256, flat, per_group);
  else go(wgrad_reduce_flat_kernel<32, Extras>, 1024, flat, per_group);
}
void launch_wgrad_reduce(cct_ctx* ctx, const float* partial, float* dW, float* db, int splits, int vgroups, int tiles_per_group,
                         int rows_pad, int n_real, int n_pad, int k_real, int og, int accumulate = 0,
                         const ReduceExtras& extras = ReduceExtras(), const PackDgrad& tall = PackDgrad()) {
  if (extras.pack.half)
    launch_wgrad_reduce<HalfExtras>(ctx, partial, dW, db, splits, vgroups, tiles_per_group, rows_pad, n_real, n_pad, k_real, og, accumulate,
                                    HalfExtras{extras, tall});
  else if (extras.pack.blocks || extras.bias.db)
    launch_wgrad_reduce<ReduceExtras>(ctx, partial, dW, db, splits, vgroups, tiles_per_group, rows_pad, n_real, n_pad, k_real, og, accumulate,
                                      extras);
  else
    launch_wgrad_reduce<NoExtras>(ctx, partial, dW, db, splits, vgroups, tiles_per_group, rows_pad, n_real, n_pad, k_real, og, accumulate,
                                  NoExtras());
}

dim3 pack_grid(int rows, int k_pad) { return dim3(rows, (k_pad / 4 + kPackThreads - 1) / kPackThreads); }

// Where the fp32 kernels of conv_small.cuh are the faster ones (measured, kernels alone, tensor cores -> fp32): forward of
// 37 MFLOP (LeNet conv1, batch 64) 9.7 -> 5.0 us, 58 MFLOP (64 channels, 14 x 14, 3 x 3) 13.7 -> 6.8, 148 MFLOP 17 -> 12,
// 231 MFLOP 14.8 -> 15.4; windows of 7 and 11 (too many window columns for the register pipeline) 94 MFLOP 10.1 -> 10.4,
// 211 MFLOP 14.3 -> 23.  Weight gradient: 58 MFLOP 26 -> 9 us, 205 MFLOP 17.7 -> 19.  Flops count a multiply-add as two and
// the idle channels and rows of the blocks with the others.
constexpr double kSmallConvFlops = 1.5e8, kSmallWideFlops = 8e7, kSmallWgradFlops = 1.7e8;

// Channels per block of small_conv_kernel for one pass (0: the tensor-core kernel).
int use_small_conv(int k, int s, long long out_pixels, int groups, int ci, int co) {
  const int ct = small_conv_ct(co);
  if (!small_conv_pick(k, s, ct) || small_conv_smem(k, small_rows(k), ct, ci, 0) > 48 * 1024) return 0;
  if ((long long)groups * ((co + 3) / 4) > 65535) return 0;  // channel tiles (of four at least) are a grid's y
  const double flops = 2.0 * out_pixels * groups * ((co + ct - 1) / ct * ct) * ci * k * k;
  return flops <= (k >= 7 ? kSmallWideFlops : kSmallConvFlops) ? ct : 0;
}
bool use_small_wgrad(long long pixels, int vgroups, int n, int k_real) {
  const double flops = 2.0 * pixels * vgroups * ((n + kSwTile - 1) / kSwTile * kSwTile) * ((k_real + kSwTile) / kSwTile * kSwTile);
  return flops <= kSmallWgradFlops;
}

// Tensor-memory and shared-memory budget of a gather problem, room for its packed operand.
void finish_problem(PlanMemory& mem, GatherProblem& gp, int vgroups, int n_bias, int sms, long long tiles, bool half) {
  // Tensor memory (512 columns) = accumulator buffers + A stages of 64 columns.  Two accumulator buffers let the epilogue
  // overlap the next tile.
  const int acc = acc_columns(gp.n_pad);
  const int taps_smem = gp.taps_smem < 0 ? gp.splits * gp.split_k / gp.run : gp.taps_smem;
  const size_t map_k = gp.map_k ? gp.map_k : (size_t)gp.k_pad;
  if (2 * acc + 4 * 64 <= 512) { gp.acc_bufs = 2; gp.a_stages = 4; }
  else if (2 * acc + 2 * 64 <= 512 && (gp.split_k ? gp.split_k : gp.k_pad) / kBlockK <= 16) { gp.acc_bufs = 2; gp.a_stages = 2; }  // short K: the epilogue matters more
  else { gp.acc_bufs = 1; gp.a_stages = std::min(4, (512 - acc) / 64); }
  const int ptab = gp.taps_smem == 0 ? 16 : 0;  // weight-gradient mode: per-warp table slices (sized for 16 warps)
  gp.b_stages = gather_slots(gp.n_pad, taps_smem, n_bias, ptab, kSmemLimit);
  int b_two;
  if (two_ctas_per_sm(gp.n_pad, taps_smem, n_bias, ptab, &b_two)) {
    gp.sets = 2; gp.tmem_cols = 256; gp.acc_bufs = 1; gp.a_stages = acc <= 64 && !ptab ? 3 : 2; gp.b_stages = b_two;
  }
  // As pairs of fp16: A slots of 32 columns, weight slots of half the size.  Four of those are two of tf32: where two CTAs share the SM the rest of
  // the memory is worth more as L1, from which the producers gather (CaffeNet conv2's weight gradient 341 -> 332 us, conv5's 137 -> 130; one CTA per
  // SM is slower then, conv3's 162 -> 187).
  gp.half = half;
  if (half && gp.sets == 2) gp.b_stages = std::min(gp.b_stages, 2);
  gp.acc_cols_half = gp.half_cross || gp.n_pad <= kCrossCols ? 2 * gp.n_pad : gp.n_pad;
  gp.acc_bufs_half = gp.sets == 4 && 2 * gp.acc_cols_half + 4 * 32 <= 512 ? 2 : 1;
  gp.a_stages_half = std::min(4, (gp.tmem_cols - gp.acc_bufs_half * gp.acc_cols_half) / 32);
  gp.b_stages_half = std::min(4, 2 * gp.b_stages);
  gp.smem = gather_smem(gp.n_pad, taps_smem, gp.b_stages, n_bias, gp.taps_smem == 0 ? 4 * gp.sets : 0).total + 1024;
  const int period = gp.splits == 1 ? gp.n / gp.ch_tile : 1;  // pixels of a stride period, which are columns, where they are stored as such
  gp.one = gp.taps_smem && !gp.inside && gp.split_k <= kOneKblocks * kBlockK && tiles <= (long long)sms * (gp.sets == 2 ? 2 : 1) &&
           (period == 1 || tiles * gp.n_pad <= (long long)sms * (period <= 4 ? kOneScattered : kOneScattered / 2));
  gp.w_half = (size_t)vgroups * gp.n_pad * map_k;
  mem.room(&gp.w, 2 * gp.w_half);
}

// The tensor map of a gather problem's packed operand.
int encode_problem(cct_ctx* ctx, GatherProblem& gp, int vgroups) {
  const size_t map_k = gp.map_k ? gp.map_k : (size_t)gp.k_pad;
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) {
    ctx->last_error = "cuTensorMapEncodeTiled is not available from this driver";
    return CCT_ERR_CUDA;
  }
  const cuuint64_t gdim[2] = {(cuuint64_t)map_k, (cuuint64_t)(2 * vgroups * gp.n_pad)};
  const cuuint64_t gstride[1] = {(cuuint64_t)map_k * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)kBlockK, (cuuint32_t)gp.n_pad};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(&gp.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, gp.w, gdim, gstride, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    ctx->last_error = "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r);
    return CCT_ERR_CUDA;
  }
  return CCT_OK;
}

}  // namespace

int umma_plan_create(cct_ctx* ctx, const ConvGeom& G, bool tensor_only, UmmaPlan** out) {
  UmmaPlan* p = new UmmaPlan();
  p->G = G;
  PlanMemory mem;
  // Floats of the split sums: one buffer for all passes.  A pass therefore ends with its own reduction - no entry point may
  // leave sums there while another pass of the plan is launched.
  size_t sums = 0;
  const int kk = G.k * G.k;
  // ---- forward: accumulator columns = output channels of a tile, reduction = (d, kr, kc)
  {
    GatherProblem& f = p->fwd;
    f.k_real = G.Dg * kk;
    f.k_pad = round_up(f.k_real, kBlockK);
    f.run = G.Dg % kRun == 0 ? kRun : 1; f.run_stride = G.n * G.n;
    f.inside = f.run == 1 && G.p == 0;
    const long long pixel_tiles = ((long long)G.B * G.m * G.m + kTileM - 1) / kTileM;
    auto tiling = [&](bool half, double half_limit) {
      return choose_gather_tiling(ctx->planning_sms(), pixel_tiles, G.g, G.og, 1, f.k_pad / kBlockK, f.run, G.s, G.bias ? G.o : 0,
                                  chain_limit(G.og, 1, f.k_pad / kBlockK), half, half_limit);
    };
    GatherTiling tl = tiling(false, 0.0);
    // Pairs of fp16 where that makes up for a look at the operands.
    const GatherTiling paired = tiling(true, tl.chain);
    const bool half = !f.inside && paired.tiles && half_pays(tl.us, tl.us - paired.us - scales_us(elements_x(G) + elements_w(G)));
    if (half) tl = paired;
    f.half_cross = tl.cross;
    f.tiles = tl.tiles;
    f.ch_tile = f.n = (G.og + f.tiles - 1) / f.tiles;
    f.n_pad = round_up(f.n, 16);
    f.splits = tl.splits; f.split_k = tl.kps * kBlockK; f.pix_pad = (size_t)pixel_tiles * kTileM;
    std::vector<MaskTap> t((size_t)f.splits * f.split_k / f.run);  // padding entries behind the last split's real ones
    for (int i = 0; i < (int)t.size(); ++i) {
      if (i * f.run < f.k_real) {
        const int d = i / kk * f.run, kr = (i / G.k) % G.k, kc = i % G.k;
        t[i] = MaskTap{d * G.n * G.n + kr * G.n + kc, (1u << kr) | (1u << (16 + kc))};
      } else {
        t[i] = MaskTap{0, kPadBit};
      }
    }
    std::vector<ColEnt> c(f.n_pad);
    for (int j = 0; j < f.n_pad; ++j) c[j] = ColEnt{j * G.m * G.m, 0, 0};
    if (!tensor_only) f.small_ct = use_small_conv(G.k, G.s, (long long)G.B * G.m * G.m, G.g, G.Dg, G.og);
    if (!f.small_ct) {
      mem.table(&f.taps, t);
      mem.table(&f.cols, c);
      mem.table(&f.zero, std::vector<float>(1, 0.f));
      finish_problem(mem, f, G.g * f.tiles, G.bias ? G.o : 0, ctx->planning_sms(), pixel_tiles * G.g * f.tiles * f.splits, half);
      if (f.splits > 1) sums = std::max(sums, (size_t)f.splits * G.g * f.tiles * f.n_pad * f.pix_pad);
    }
  }
  bool wgrad_half = false;
  // ---- data gradient as a stride-1 gather over dY: one "super pixel" = an s x s block of input pixels; accumulator
  //      columns = (d, py, px), reduction = (oc, jy, jx) with jy, jx < ceil(k/s); depth-to-space in the epilogue.
  {
    GatherProblem& d = p->dgr;
    const int J = p->dgr_taps = (G.k + G.s - 1) / G.s;
    p->dgr_q0 = G.p / G.s;
    p->dgr_q = (G.n - 1 + G.p) / G.s + 1 - p->dgr_q0;
    d.run = G.og % kRun == 0 ? kRun : 1; d.run_stride = G.m * G.m;
    d.k_real = G.og * J * J;
    // One stride period of rows per super pixel: a taller one gathers less per pixel, but the taps that one of its pixels does
    // not have would be products with a zero weight, and a dY that is not finite would reach pixels whose window does not hold it.
    const int ss = G.s * G.s;
    const long long pixel_tiles = ((long long)G.B * p->dgr_q * p->dgr_q + kTileM - 1) / kTileM;
    const int kblocks = round_up(d.k_real, kBlockK) / kBlockK;
    auto tiling = [&](bool half, double half_limit) {
      return choose_gather_tiling(ctx->planning_sms(), pixel_tiles, G.g, G.Dg, ss, kblocks, d.run, 1, 0, chain_limit(G.Dg, ss, kblocks), half, half_limit);
    };
    GatherTiling tl = tiling(false, 0.0);
    // Narrow tiles are bound by what they gather: blocks of `rows` stride periods gather it for more columns at once.
    struct Tall { int rows, taps_y, q, q0, k_real; long long tiles; };
    auto tall_of = [&](int rows) {
      Tall b{rows, J + rows - 1, 0, G.p / (rows * G.s), 0, 0};
      b.q = (G.n - 1 + G.p) / (rows * G.s) + 1 - b.q0;
      b.k_real = G.og * J * b.taps_y;
      b.tiles = ((long long)G.B * b.q * p->dgr_q + kTileM - 1) / kTileM;
      return b;
    };
    GatherTiling paired = tiling(true, tl.chain);
    if (!paired.tiles) paired.us = tl.us;
    Tall tall = tall_of(1);
    for (int rows = 2; rows <= kMaxTallRows; ++rows) {
      const Tall b = tall_of(rows);
      if (b.taps_y > kMaxTapsPerAxis || b.k_real > 16384 || rows * ss > 256) break;
      const GatherTiling t = choose_gather_tiling(ctx->planning_sms(), b.tiles, G.g, G.Dg, rows * ss, round_up(b.k_real, kBlockK) / kBlockK, d.run, 1, 0,
                                                  0.0, true, tl.chain, 1);
      if (t.tiles && t.us + kTallUs < kTallGain * paired.us) { paired = t; paired.us += kTallUs; tall = b; }
    }
    // The two gradients share the look at dY: both in pairs of fp16, or one of them, or none.
    const WgradTime wgrad = weight_gradient_time(G, p->fwd.k_real, wgrad_columns(G));
    const double wgrad_us = wgrad.us, wgrad_saves = wgrad.saves;
    const double dgrad_saves = tl.us - paired.us, dy = elements_y(G) + elements_w(G), x = elements_x(G);
    const double best = std::max(dgrad_saves - scales_us(dy), std::max(wgrad_saves - scales_us(dy + x), dgrad_saves + wgrad_saves - scales_us(dy + x)));
    const bool worth = half_pays(tl.us + wgrad_us, best);
    const bool half = worth && paired.tiles && dgrad_saves > 0;
    wgrad_half = worth && wgrad_saves - scales_us(dy + x) + (half ? scales_us(dy) : 0) > 0;
    if (half && tall.rows == 1) tl = paired;
    d.half_cross = tl.cross;
    d.k_pad = round_up(d.k_real, kBlockK);
    d.tiles = tl.tiles;
    d.ch_tile = (G.Dg + d.tiles - 1) / d.tiles;
    d.n = d.ch_tile * ss;
    d.n_pad = round_up(d.n, 16);
    d.splits = tl.splits; d.split_k = tl.kps * kBlockK; d.pix_pad = (size_t)pixel_tiles * kTileM;
    std::vector<MaskTap> t((size_t)d.splits * d.split_k / d.run);
    for (int i = 0; i < (int)t.size(); ++i) {
      if (i * d.run < d.k_real) {
        const int jx = i % J, jy = (i / J) % J, oc = i / (J * J) * d.run;
        t[i] = MaskTap{oc * G.m * G.m - jy * G.m - jx, (1u << jy) | (1u << (16 + jx))};
      } else {
        t[i] = MaskTap{0, kPadBit};
      }
    }
    std::vector<ColEnt> c(d.n_pad);
    for (int j = 0; j < d.n_pad; ++j) {
      const int dl = j / ss, py = (j / G.s) % G.s, px = j % G.s;
      c[j] = ColEnt{dl * G.n * G.n + py * G.n + px, (short)py, (short)px};
    }
    if (!tensor_only && G.s == 1) d.small_ct = use_small_conv(G.k, 1, (long long)G.B * G.n * G.n, G.g, G.og, G.Dg);
    if (!d.small_ct) {
      mem.table(&d.taps, t);
      mem.table(&d.cols, c);
      mem.table(&d.zero, std::vector<float>(1, 0.f));
      finish_problem(mem, d, G.g * d.tiles, 0, ctx->planning_sms(), pixel_tiles * G.g * d.tiles * d.splits, half);
      if (half && tall.rows > 1) {
        GatherProblem& b = p->tall;
        b.rows = tall.rows; b.run = d.run; b.run_stride = d.run_stride;
        b.taps_y = tall.taps_y; b.q_h = tall.q; b.q0 = tall.q0;
        b.k_real = tall.k_real; b.k_pad = round_up(tall.k_real, kBlockK);
        b.tiles = paired.tiles; b.ch_tile = (G.Dg + b.tiles - 1) / b.tiles;
        b.n = b.ch_tile * tall.rows * ss; b.n_pad = round_up(b.n, 16);
        b.half_cross = paired.cross;
        b.split_k = b.k_pad; b.pix_pad = (size_t)tall.tiles * kTileM;
        std::vector<MaskTap> bt((size_t)b.k_pad / b.run, MaskTap{0, kPadBit});
        for (int i = 0; i * b.run < b.k_real; ++i) {
          const int jx = i % J, jy = (i / J) % b.taps_y, oc = i / (J * b.taps_y) * b.run;
          bt[i] = MaskTap{oc * G.m * G.m - jy * G.m - jx, (1u << jy) | (1u << (16 + jx))};
        }
        std::vector<ColEnt> bc(b.n_pad);
        for (int j = 0; j < b.n_pad; ++j) {
          const int dl = j / (tall.rows * ss), py = (j / G.s) % (tall.rows * G.s), px = j % G.s;
          bc[j] = ColEnt{dl * G.n * G.n + py * G.n + px, (short)py, (short)px};
        }
        mem.table(&b.taps, bt);
        mem.table(&b.cols, bc);
        mem.table(&b.zero, std::vector<float>(1, 0.f));
        finish_problem(mem, b, G.g * b.tiles, 0, ctx->planning_sms(), tall.tiles * G.g * b.tiles, true);
        b.one = false;
      }
      if (d.splits > 1) sums = std::max(sums, (size_t)d.splits * G.g * d.tiles * d.n_pad * d.pix_pad);
    }
  }
  // ---- weight gradient: rows = (d, kr, kc) plus the all-ones row, columns = output channels of a tile
  {
    GatherProblem f;  // its own channel tiles, whatever the forward pass takes
    f.k_real = p->fwd.k_real;
    f.tiles = p->wt_tiles = weight_grad_tiles(G.og, &p->w_chain);
    f.n = p->wt_n = (G.og + f.tiles - 1) / f.tiles;
    f.n_pad = p->w_npad = round_up(f.n, 16);
    p->w_mtiles = (f.k_real + 1 + kTileM - 1) / kTileM;
    // M-tiles per CTA: as many as leave room for two stages in shared memory (and whose accumulators fit in tensor
    // memory); the dY tile of a k-block is staged once for all of them.
    int subs = 1;
    for (int u = 2; u <= kWgMaxSubs; ++u)
      if (u <= p->w_mtiles && u * (f.n_pad <= 64 ? 2 : 1) * f.n_pad <= 512 && 2 * wg_smem(f.n_pad, u, 2).stage_bytes + 8192 <= (uint32_t)kSmemLimit)
        subs = u;
    // 257 .. 384 rows and one channel tile of at most 128: the role-exchanged kernel, one CTA for all rows
    p->w_ts = ts_rows(f.k_real, f.n_pad);
    const int n_pix = G.B * G.m * G.m;
    p->w_kblocks_total = (n_pix + kBlockK - 1) / kBlockK;
    for (;; subs = 1) {
      p->w_mgroups = p->w_ts ? 1 : (p->w_mtiles + subs - 1) / subs;
      const int out_tiles = p->w_mgroups * G.g * f.tiles;
      // Whole waves of CTAs (one CTA per SM), as few as keep a partial sum's accumulation chain within
      // kMaxChainKblocks: the tensor core's fp32 accumulation truncates, so the error of a partial sum grows with the
      // length of its chain, while the reduction over splits adds with proper rounding.
      int splits = 1;
      for (int waves = 1; waves <= 64; ++waves) {
        splits = std::max(1, waves * ctx->sm_count / out_tiles);
        if ((p->w_kblocks_total + splits - 1) / splits <= p->w_chain) break;
      }
      splits = std::min(splits, std::max(1, p->w_kblocks_total / 3));  // at least 3 k-blocks per CTA
      p->w_kblocks_per_split = (p->w_kblocks_total + splits - 1) / splits;
      p->w_splits = (p->w_kblocks_total + p->w_kblocks_per_split - 1) / p->w_kblocks_per_split;
      // Few pixels: where a CTA for every M-tile has an SM of its own, the same splits with half the MMAs in a row (about 1 us per
      // k-block of two M-tiles): 37 images, 50 -> 75 channels 21 x 21, kernel 14.1 -> 10.0 us, LeNet conv2 at batch 64 12.6 -> 9.1.
      if (subs == 1 || p->w_ts || p->w_mtiles * G.g * f.tiles * p->w_splits > ctx->sm_count) break;
    }
    p->w_subs = subs;
    const uint32_t stage_bytes = wg_smem(f.n_pad, subs, 2).stage_bytes;
    p->w_stages = std::max(2, std::min(kWgMaxStages, (int)((kSmemLimit - 8192) / stage_bytes)));
    p->w_smem = p->w_ts ? kTsSmem + 1024 : wg_smem(f.n_pad, subs, p->w_stages).total + 1024;
    p->w_small = !tensor_only && use_small_wgrad(n_pix, G.g * f.tiles, f.n, f.k_real);
    if (p->w_small) {
      // About one block per SM (two where a block keeps at least two chunks of pixels).
      p->ws_rows = (f.k_real + 1 + kSwTile - 1) / kSwTile;
      p->ws_cols = (f.n + kSwTile - 1) / kSwTile;
      const int tiles = p->ws_rows * p->ws_cols * G.g * f.tiles;
      const int want = std::max(1, ctx->sm_count * 2 / tiles);
      p->ws_pix = std::max(kSwPix, round_up((n_pix + want - 1) / want, kSwPix));
      p->w_splits = (n_pix + p->ws_pix - 1) / p->ws_pix;
      sums = std::max(sums, (size_t)p->w_splits * G.g * f.tiles * p->ws_rows * kSwTile * p->ws_cols * kSwTile);
    }
    p->wg_gather = !p->w_small && (f.k_real >= kGatherRows || (wgrad_half && half_gather(G, f.k_real, f.n_pad)));  // see below
    p->w_half = wgrad_half && !p->w_small && (p->wg_gather || half_ts(G, f.k_real, f.n_pad));
    if (!p->w_small && !p->wg_gather)
      sums = std::max(sums, (size_t)p->w_splits * G.g * f.tiles * p->w_mtiles * kTileM * f.n_pad);
    if (!p->wg_gather) {
      std::vector<MaskTap> t((size_t)p->w_mtiles * kTileM);
      for (size_t i = 0; i < t.size(); ++i) {
        if ((int)i < f.k_real) {
          const int d = (int)i / kk, kr = ((int)i / G.k) % G.k, kc = (int)i % G.k;
          t[i] = MaskTap{d * G.n * G.n + kr * G.n + kc, kWgValidBit | (1u << kr) | (1u << (16 + kc))};
        } else if ((int)i == f.k_real) {
          t[i] = MaskTap{0, kWgOnesBits};
        } else {
          t[i] = MaskTap{0, kWgPadBit};
        }
      }
      mem.table(&p->w_taps, t);
    }
  }
  // ---- weight gradient through the gather kernel (the default): tiles = splits x channel tiles x M-tiles
  // It needs one extra pass over dY (split into hi / lo, 12 bytes moved per element), which pays when every dY
  // element takes part in many multiply-adds: measured faster from CaffeNet conv2 (1200 lowered rows) upwards,
  // slower for AlexNet conv1 (363 rows), so short lowered matrices keep the shared-memory kernel above.
  if (p->wg_gather) {
    GatherProblem& w = p->wgp;
    struct { int tiles, n, n_pad, k_real; } f = {p->wt_tiles, p->wt_n, p->w_npad, p->fwd.k_real};
    const int n_pix = G.B * G.m * G.m;
    const int kb_total = (n_pix + kBlockK - 1) / kBlockK;
    const int vgroups = G.g * f.tiles;
    w.tiles = f.tiles; w.ch_tile = f.n; w.n = f.n; w.n_pad = f.n_pad;
    w.k_real = n_pix;
    p->wg_mtiles = (f.k_real + kTileM - 1) / kTileM;  // no all-ones row here: the bias gradient comes from the dY pass
    const int base_tiles = vgroups * p->wg_mtiles;
    // Splits of the pixel range: all work units (base tiles x splits) cost the same, so the kernel's time is
    // (rounds of units over the resident CTAs) x (k-blocks per unit) - pick the split count that minimises it, plus the
    // traffic of the partial sums it creates (written once, read once by the reduction).  Chains stay bounded
    // (kMaxChainKblocks); a unit's set-up and epilogue cost about five k-blocks.  A last round that fills at most half of the slots of
    // the two-CTAs-per-SM shape costs about half a round: its CTAs have their SM's tensor pipe to themselves.
    {
      const bool two_per_sm = f.n_pad <= 128;  // the shape finish_problem() will pick for this accumulator width
      const int slots = ctx->planning_sms() * (two_per_sm ? 2 : 1);
      const double us_per_kblock = 12.0 * (f.n_pad / 2.0) / 1900.0 * (two_per_sm ? 2.0 : 1.0);
      // (half the additions per k-block in pairs of fp16: no less accurate than the short kernels that would have taken the layer)
      const int chain = f.k_real >= kGatherRows ? p->w_chain : std::min(p->w_chain, 2 * p->w_kblocks_per_split);
      const int s_min = std::max(1, (kb_total + chain - 1) / chain);
      // First without the set-up, among units of at least sixteen k-blocks; then with it, among units no longer than that:
      // a set-up would rather have fewer splits, whose longer chains are less accurate.
      for (const int setup : {0, 5}) {
        double best = 0.0;
        int best_kps = 0;
        for (int s = s_min; s <= std::max(s_min, 8 * slots / base_tiles + 1); ++s) {
          const int kps = (kb_total + s - 1) / s;
          if (setup && kps > p->wg_kps) continue;
          if (kps < (setup ? 4 : 16) && best_kps) break;
          const int units = base_tiles * ((kb_total + kps - 1) / kps);
          const int tail = units % slots;
          const double rounds = units / slots + (tail == 0 ? 0.0 : (two_per_sm && 2 * tail <= slots) ? 0.55 : 1.0);
          const double reduce = 1.5 * units * (double)kTileM * f.n_pad * 8.0 / 6.5e6 / us_per_kblock;
          const double cost = rounds * (kps + setup) + reduce;
          if (!best_kps || cost < best - 1e-9) { best = cost; best_kps = kps; }
        }
        if (best_kps) p->wg_kps = best_kps;
      }
    }
    p->wg_splits = (kb_total + p->wg_kps - 1) / p->wg_kps;
    w.k_pad = p->wg_kps * kBlockK;
    w.taps_smem = 0;
    w.map_k = (size_t)kb_total * kBlockK;
    // dY in rows serves the data gradient too, where rows are channels and the offsets fit.  (Its table goes before the next one, which
    // is long: behind it, it made the tables grow, and the long one was copied once more.)
    if (w.n == w.n_pad && w.tiles * w.n == G.og && !p->dgr.small_ct && (double)G.o * w.map_k < 2147483648.0) {
      const GatherProblem& d = p->dgr;
      const int J = p->dgr_taps;
      std::vector<MaskTap> rt((size_t)d.splits * d.split_k / d.run, MaskTap{0, kPadBit});
      for (int i = 0; i * d.run < d.k_real; ++i) {
        const int jx = i % J, jy = (i / J) % J, oc = i / (J * J) * d.run;
        rt[i] = MaskTap{(int)(oc * w.map_k) - jy * G.m - jx, (1u << jy) | (1u << (16 + jx))};
      }
      mem.table(&p->dgr_row_taps, rt);
      const GatherProblem& b = p->tall;
      if (b.rows > 1) {
        std::vector<MaskTap> bt((size_t)b.k_pad / b.run, MaskTap{0, kPadBit});
        for (int i = 0; i * b.run < b.k_real; ++i) {
          const int jx = i % J, jy = (i / J) % b.taps_y, oc = i / (J * b.taps_y) * b.run;
          bt[i] = MaskTap{(int)(oc * w.map_k) - jy * G.m - jx, (1u << jy) | (1u << (16 + jx))};
        }
        mem.table(&p->tall_row_taps, bt);
      }
    }
    // Per-pixel table: where the pixel's window starts, and which of its rows and columns lie outside the plane.
    std::vector<uint32_t> outside(G.m);  // the same for rows and columns: bit a = window row a of output row r is outside
    for (int r = 0; r < G.m; ++r)
      for (int a = 0; a < kMaxTapsPerAxis; ++a)
        if (a >= G.k || r * G.s - G.p + a < 0 || r * G.s - G.p + a >= G.n) outside[r] |= 1u << a;
    std::vector<MaskTap> t((size_t)p->wg_splits * p->wg_kps * kBlockK, MaskTap{0, 0xffffffffu});
    size_t i = 0;
    for (int b = 0; b < G.B; ++b)
      for (int r = 0; r < G.m; ++r) {
        const int row = (int)((long long)b * G.D * G.n * G.n) + (r * G.s - G.p) * G.n - G.p;
        for (int q = 0; q < G.m; ++q, ++i) t[i] = MaskTap{row + q * G.s, outside[r] | (outside[q] << 16) | 0x80008000u};
      }
    mem.table(&p->wg_pix, t);
    finish_problem(mem, w, vgroups, 0, ctx->planning_sms(), (long long)base_tiles * p->wg_splits, wgrad_half);
    if (G.bias) mem.room(&p->wg_plane_sums, std::max<size_t>(G.B, (w.map_k + kSplitRunLeast - 1) / kSplitRunLeast) * G.o);
    sums = std::max(sums, (size_t)p->wg_splits * vgroups * p->wg_mtiles * kTileM * f.n_pad);
  }
  if (p->fwd.half || p->dgr.half || p->w_half) {
    mem.table(&p->half_ticket, std::vector<uint32_t>(2, 0u));
    mem.room(&p->half, 1);
    mem.room(&p->half_parts, (size_t)ctx->sm_count * kScaleBlocksPerSm);
  }
  float* sum_memory = nullptr;
  mem.room(&sum_memory, sums);
  int rc = mem.obtain(ctx, &p->memory, &p->bytes);
  p->fwd.partial = p->dgr.partial = p->w_partial = sum_memory;
  if (rc == CCT_OK && p->fwd.w) rc = encode_problem(ctx, p->fwd, G.g * p->fwd.tiles);
  if (rc == CCT_OK && p->dgr.w) rc = encode_problem(ctx, p->dgr, G.g * p->dgr.tiles);
  if (rc == CCT_OK && p->tall.w) rc = encode_problem(ctx, p->tall, G.g * p->tall.tiles);
  if (rc == CCT_OK && p->wg_gather) {
    rc = encode_problem(ctx, p->wgp, G.g * p->wt_tiles);
    if (rc == CCT_OK && cudaMemsetAsync(p->wgp.w, 0, 2 * p->wgp.w_half * sizeof(float), ctx->stream) != cudaSuccess) {  // padded channel rows stay zero
      ctx->last_error = "cudaMemsetAsync of the pre-split dY buffer failed";
      rc = CCT_ERR_CUDA;
    }
  }
  // The kernels that this plan launches, and no others: each is one to load at its first use.
  for (const GatherProblem* gp : {&p->fwd, &p->dgr, &p->wgp, &p->tall})
    if (rc == CCT_OK && gp->w) rc = set_smem(ctx, gather_kernel(*gp, gp == &p->wgp, gp->one, gp->half), gather_smem_limit(*gp));
  if (rc == CCT_OK && !p->w_small && !p->wg_gather) rc = set_smem(ctx, short_wgrad_kernel(p), kSmemLimit);
  if (rc == CCT_OK && p->w_half && !p->wg_gather) rc = set_smem(ctx, half_ts_kernel(G.k), kSmemLimit);
  if (rc != CCT_OK) {
    umma_plan_destroy(ctx, p);
    return rc;
  }
  *out = p;
  return CCT_OK;
}

void umma_plan_destroy(cct_ctx* ctx, UmmaPlan* p) {
  if (!p) return;
  cudaFree(p->memory);
  delete p;
}

size_t umma_plan_workspace_bytes(const UmmaPlan* p) { return p->bytes; }

namespace {

void fill_common(GatherParams& P, const GatherProblem& gp, cct_ctx* ctx, int vgroups, int n_bias) {
  P.taps = gp.taps; P.cols = gp.cols;
  P.tiles_per_group = gp.tiles;
  P.out_tile_channels = gp.ch_tile;
  P.n = gp.n; P.n_pad = gp.n_pad; P.k_pad = gp.split_k ? gp.split_k : gp.k_pad;
  P.cols_per_channel = gp.n / gp.ch_tile;
  P.splits = gp.splits; P.partial = gp.partial; P.pix_pad = (int)gp.pix_pad;
  P.taps_smem = gp.taps_smem < 0 ? gp.splits * gp.split_k / gp.run : gp.taps_smem;
  P.run_stride = gp.run_stride; P.zero = gp.zero;
  P.n_pix_tiles = (P.n_pix + kTileM - 1) / kTileM;
  P.total_tiles = P.n_pix_tiles * vgroups * gp.splits;
  P.a_stages = gp.a_stages; P.b_stages = gp.b_stages; P.acc_bufs = gp.acc_bufs;
  P.tmem_cols = gp.tmem_cols;
  P.n_bias = P.bias ? n_bias : 0;
  P.lo_row_offset = vgroups * gp.n_pad;
  P.a_stages_half = (uint8_t)gp.a_stages_half; P.b_stages_half = (uint8_t)gp.b_stages_half; P.acc_bufs_half = (uint8_t)gp.acc_bufs_half; P.acc_cols_half = (uint16_t)gp.acc_cols_half;
  P.status = ctx->status_dev;
}

PackDgrad pack_dgrad_job(const UmmaPlan* p, const GatherProblem& d, const float* W, bool half) {
  const ConvGeom& G = p->G;
  PackDgrad J{W, d.w, d.w + d.w_half, d.tiles, G.og, G.Dg, G.k, G.s, p->dgr_taps, d.ch_tile, d.n, d.n_pad, d.k_real, d.k_pad, d.run, 0, 0,
               half ? p->half : nullptr, d.rows, half && p->tall.rows > 1 ? (d.rows > 1 ? kOnlyHalf : kOnlyTf32) : kAny};
  J.parts = (d.k_pad / 4 + kPackThreads - 1) / kPackThreads;
  J.blocks = G.g * d.tiles * d.n_pad * J.parts;
  return J;
}

// Grid of a pass by small_conv_kernel, and its shared memory; `block_warps` > 0: that many per block, which
// may go beside a weight gradient.
struct SmallConvShape {
  int ct, rows, warps, x, y;
  size_t smem;
};
SmallConvShape shape_small_conv(cct_ctx* ctx, SmallConv& P, int k, int s, int ct, int block_warps = 0) {
  // Tall lanes: see small_rows().
  auto lots_of = [&](int rows) { return ((long long)P.batch * ((P.n_out + rows - 1) / rows) * P.n_out + 31) / 32; };
  const long long few = lots_of(small_rows(k)), tall = lots_of(kSmallTall), sms = ctx->launch_sms();
  const bool eight = k == 5 && s == 1 && ct == 1 && few > sms && (tall < sms || 40 * tall <= (block_warps ? 23 : 22) * few);
  const int rows = eight ? kSmallTall : small_rows(k);
  P.row_groups = (P.n_out + rows - 1) / rows;
  P.positions = P.batch * P.row_groups * P.n_out;
  // Narrower channel tiles and more warps on the input channels until the SMs have about sixteen warps each.
  const long long lots = (P.positions + 31) / 32, want = 16ll * sms;
  if (ct == 8 && lots * P.groups * ((P.co + 7) / 8) * std::min(16, std::max(1, P.ci / 2)) < want) ct = 4;
  P.col_tiles = (P.co + ct - 1) / ct;
  P.share = P.ci >= 4 && lots * P.groups * P.col_tiles < want;
  int warps = block_warps ? block_warps : 4;
  while (!block_warps && P.share && warps < 16 && P.ci >= 4 * warps && lots * P.groups * P.col_tiles * warps < want &&
         small_conv_smem(k, rows, ct, P.ci, 2 * warps) <= 48 * 1024)
    warps *= 2;
  const int per_block = P.share ? 32 : 32 * warps;
  return SmallConvShape{ct, rows, warps, (P.positions + per_block - 1) / per_block, P.groups * P.col_tiles,
                        small_conv_smem(k, rows, ct, P.ci, P.share ? warps : 0)};
}
void launch_small_conv(cct_ctx* ctx, SmallConv& P, int k, int s, int ct, int block_warps = 0) {
  const SmallConvShape g = shape_small_conv(ctx, P, k, s, ct, block_warps);
  launch_pdl(small_conv_pick(k, s, g.ct, g.rows), dim3(g.x, g.y), dim3(32 * g.warps), g.smem, ctx->stream, P);
}
// The data gradient of a stride-1 layer as a convolution of dY.
SmallConv small_dgrad(const ConvGeom& G, const float* dY, const float* W, float* dX, int batch) {
  return SmallConv{dY, W, nullptr, dX, batch, G.m, G.n, G.k - 1 - G.p, G.og, G.Dg, G.g, 1, 0};
}

// Whether both gradients of a small layer go in one launch (kSmallRounds and so on).
bool small_together(cct_ctx* ctx, const UmmaPlan* p) {
  const ConvGeom& G = p->G;
  if (!p->w_small || !p->dgr.small_ct) return false;
  SmallConv d = small_dgrad(G, nullptr, nullptr, nullptr, G.B);
  if (shape_small_conv(ctx, d, G.k, 1, p->dgr.small_ct).warps > kSwWarps) return false;
  const SmallConvShape g = shape_small_conv(ctx, d, G.k, 1, p->dgr.small_ct, kSwWarps);
  const long long blocks = (long long)p->ws_rows * p->ws_cols * G.g * p->wt_tiles * p->w_splits + (long long)g.x * g.y;
  const long long slots = (long long)SmallBackward::blocks(g.ct) * ctx->sm_count;
  return blocks <= kSmallRounds * slots && (g.rows != kSmallTall || G.og >= kSmallTallChannels || blocks <= slots);
}

// A CTA per tile where each has a slot (ONE), or a persistent grid: one CTA per SM (4 producer sets) or two (2 sets); then the reduction over
// the splits, if any.  A plan whose tiles all had slots takes the persistent kernel while a reduction in flight keeps some of them; its
// attribute is set then, since a plan made beside a communicator never comes here.
void launch_gather(cct_ctx* ctx, const GatherParams& P, const GatherProblem& gp, bool weight_grad = false) {
  const int slots = (gp.sets == 2 ? 2 : 1) * ctx->launch_sms();
  const bool one = gp.one && P.total_tiles <= slots;
  const GatherKernel kernel = gather_kernel(gp, weight_grad, one, P.half != nullptr);
  if ((gp.one && !one) || (gp.half && !P.half)) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gather_smem_limit(gp));  // (or the launch fails)
  launch_pdl(kernel, dim3(std::min(P.total_tiles, slots)), dim3(gather_threads(gp.sets)), gp.smem, ctx->stream, P, gp.map);
  if (P.splits > 1) {
    const int vgroups = P.total_tiles / (P.n_pix_tiles * P.splits), cols = P.n_pix_tiles * vgroups * P.n > 32 * ctx->sm_count ? 8 : 1;
    const int col_tiles = (P.n + cols - 1) / cols;
    auto kernel = P.only == kOnlyTf32 ? (cols == 8 ? gather_reduce_kernel<8, true> : gather_reduce_kernel<1, true>)
                                      : (cols == 8 ? gather_reduce_kernel<8, false> : gather_reduce_kernel<1, false>);
    launch_pdl(kernel, dim3((P.n_pix + 127) / 128, vgroups * col_tiles), dim3(128),
               0, ctx->stream, P, col_tiles);
  }
}

// The scales of a call's operands (a = null: not needed) in one launch.
struct ScaleOf {
  const float *a, *mask;
  size_t n;
  int slot, headroom;
  const int32_t* where = nullptr;
  int pooled = 1, plane = 1;
};
void launch_scales(cct_ctx* ctx, const UmmaPlan* p, std::initializer_list<ScaleOf> operands) {
  ScaleJobs J{};
  J.out = p->half; J.parts = p->half_parts; J.ticket = p->half_ticket;
  size_t total = 0;
  for (const ScaleOf& o : operands) total += o.a ? o.n : 0;
  const size_t blocks = (size_t)ctx->sm_count * kScaleBlocksPerSm - 3;  // rounded up for each of three
  const size_t per_block = (std::max<size_t>(kScaleChunk, (total + blocks - 1) / blocks) + 1023) & ~(size_t)1023;
  int grid = 0;
  for (const ScaleOf& o : operands) {
    if (!o.a) continue;
    ScaleJob& job = J.job[J.jobs++];
    job.a = o.a; job.mask = o.mask; job.n = o.n; job.per_block = per_block; job.slot = o.slot; job.headroom = o.headroom;
    job.where = o.where; job.pooled = o.pooled; job.plane = o.plane;
    job.first = grid;
    job.blocks = (int)((o.n + per_block - 1) / per_block);
    grid += job.blocks;
  }
  launch_pdl(operand_scale_kernel, dim3(grid), dim3(kScaleThreads), 0, ctx->stream, J);
}

}  // namespace

int umma_conv_forward(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* bias, float* Y,
                      int relu, PhaseTimer* t, int batch, bool repack) {
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;  // an earlier bounded wait gave up: do not pile up behind it
  const ConvGeom& G = p->G;
  GatherProblem& f = p->fwd;
  const int vgroups = G.g * f.tiles;
  const int B = batch > 0 ? batch : G.B;  // a leading slice of the batch (host-buffer calls pipeline over slices)
  if (f.small_ct) {
    SmallConv P{X, W, G.bias ? bias : nullptr, Y, B, G.n, G.m, G.p, G.Dg, G.og, G.g, 0, relu};
    t->begin(0, ctx->stream);
    launch_small_conv(ctx, P, G.k, G.s, f.small_ct);
    t->end(0, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
    return CCT_OK;
  }
  const bool half = f.half && batch == 0;
  if (repack) {
    t->begin(4, ctx->stream);
    if (half) launch_scales(ctx, p, {ScaleOf{X, nullptr, elements_x(G), kHalfX, 0}, ScaleOf{W, nullptr, elements_w(G), kHalfW, 0}});
    launch_pdl(half ? pack_fwd_kernel<true> : pack_fwd_kernel<false>, pack_grid(vgroups * f.n_pad, f.k_pad), dim3(kPackThreads), 0, ctx->stream, W, f.w,
               f.w + f.w_half, f.tiles, G.og, f.n, f.n_pad, f.k_real, f.k_pad, f.run, G.k * G.k, half ? p->half : nullptr);
    t->end(4, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
  }
  GatherParams P{};
  P.in = X; P.out = Y;
  P.bias = G.bias ? bias : nullptr;
  P.n_pix = B * G.m * G.m; P.q_h = G.m; P.q_w = G.m;
  P.iy_mul = G.s; P.iy_add = -G.p; P.ix_mul = G.s; P.ix_add = -G.p;
  P.in_lim = G.n;
  P.tap_sign = 1; P.taps_per_axis = G.k;
  P.in_batch_stride = (long long)G.D * G.n * G.n;
  P.in_group_stride = G.Dg * G.n * G.n;
  P.oy_mul = 1; P.oy_add = 0; P.ox_mul = 1; P.ox_add = 0;
  P.out_lim = G.m; P.check_out = 0;
  P.out_pitch = G.m; P.out_plane = G.m * G.m;
  P.out_batch_stride = (long long)G.o * G.m * G.m;
  P.out_group_channels = G.og;
  P.relu = relu;
  fill_common(P, f, ctx, vgroups, G.o);
  if (half) { P.half = p->half; P.half_gathered = kHalfX; P.half_packed = kHalfW; P.taps_x = (uint8_t)G.k; }
  t->begin(0, ctx->stream);
  launch_gather(ctx, P, f);
  t->end(0, ctx->stream);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

bool umma_dy_rows(const UmmaPlan* p, DyRows* rows) {
  if (!p->wg_gather || !p->dgr_row_taps) return false;
  *rows = DyRows{p->wgp.w, p->wgp.w_half, p->wgp.map_k, p->G.bias ? p->wg_plane_sums : nullptr, p->G.o, p->G.B,
                 p->wgp.half ? p->half : nullptr};
  return true;
}

int umma_pooled_scales(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* dP, const float* P, const int32_t* idx, int k, int s,
                       bool dgrad) {
  const ConvGeom& G = p->G;
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  if (!p->w_half && !(p->dgr.half && dgrad)) return CCT_OK;
  const int pooled = (G.m - k) / s + 1, windows = (k + s - 1) / s;
  int headroom = 0;  // an element is in up to windows^2 of them
  while ((1 << headroom) < windows * windows) ++headroom;
  launch_scales(ctx, p, {ScaleOf{p->w_half ? X : nullptr, nullptr, elements_x(G), kHalfX, 0},
                         ScaleOf{p->dgr.half && dgrad ? W : nullptr, nullptr, elements_w(G), kHalfW, 0},
                         ScaleOf{dP, P, (size_t)G.B * G.o * pooled * pooled, kHalfDy, headroom, idx, pooled * pooled, G.m * G.m}});
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

namespace {
int weight_gradient(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* dY, float* dW, float* db, PhaseTimer* t, const float* pack_W,
                    SmallConv* with, bool half);
int data_gradient(cct_ctx* ctx, UmmaPlan* p, const float* W, const float* dY, float* dX, PhaseTimer* t, int batch, bool repack, bool half);
}

int umma_conv_backward(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* dY, float* dX,
                       float* dW, float* db, PhaseTimer* t, bool scaled) {
  const ConvGeom& G = p->G;
  const size_t nx = elements_x(G), ny = elements_y(G), nw = elements_w(G);
  // Small layers: the data gradient goes with the weight gradient, unless one writes where the other reads.
  if (dX && p->w_small && p->dgr.small_ct && !t->enabled && apart(dX, nx, {{X, nx}, {dY, ny}, {dW, nw}, {db, G.o}}) &&
      apart(dW, nw, {{W, nw}, {dY, ny}}) && (!G.bias || apart(db, G.o, {{W, nw}, {dY, ny}}))) {
    SmallConv d = small_dgrad(G, dY, W, dX, G.B);
    if (small_together(ctx, p)) return weight_gradient(ctx, p, X, dY, dW, db, t, nullptr, &d, false);
  }
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  if (!scaled && (p->w_half || (p->dgr.half && dX))) {
    launch_scales(ctx, p, {ScaleOf{p->w_half ? X : nullptr, nullptr, nx, kHalfX, 0}, ScaleOf{p->dgr.half && dX ? W : nullptr, nullptr, nw, kHalfW, 0},
                           ScaleOf{dY, nullptr, ny, kHalfDy, 0}});
    CCT_CHECK_LAUNCH(ctx);
  }
  int rc = weight_gradient(ctx, p, X, dY, dW, db, t, dX ? W : nullptr, nullptr, true);
  if (rc == CCT_OK && dX) rc = data_gradient(ctx, p, W, dY, dX, t, 0, false, true);
  return rc;
}

// Weight + bias gradient over the whole batch; `pack_W`: the weights to pack for the data gradient on the way; `with`: the data
// gradient of a small layer, in the same launch.
namespace {
int weight_gradient(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* dY, float* dW, float* db, PhaseTimer* t, const float* pack_W,
                    SmallConv* with, bool half) {
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  const ConvGeom& G = p->G;
  ReduceExtras extras{};
  PackDgrad tall{};
  if (pack_W && !p->dgr.small_ct) {
    extras.pack = pack_dgrad_job(p, p->dgr, pack_W, half && p->dgr.half);
    if (half && p->tall.rows > 1) tall = pack_dgrad_job(p, p->tall, pack_W, true);
  }
  if (p->wg_gather) {
    struct { int tiles, n, n_pad, k_real; } f = {p->wt_tiles, p->wt_n, p->w_npad, p->fwd.k_real};
    GatherProblem& w = p->wgp;
    const int vgroups = G.g * f.tiles, mm = G.m * G.m;
    t->begin(1, ctx->stream);
    float* sums = G.bias ? p->wg_plane_sums : nullptr;
    // Without dY the kernel that made it has written the rows, whose sums are those of planes: where it could, a dY of its own gives the same sums.
    const bool planes = !dY || (!w.half && (p->dgr_row_taps || split_by_planes(G.B * G.o, mm)));
    const int len = split_run(G.o, w.map_k, ctx->sm_count), runs = (int)((w.map_k + len - 1) / len);
    if (!planes)
      launch_pdl(split_dy_runs_kernel, dim3((G.o * runs + 7) / 8), dim3(256), 0, ctx->stream, dY, w.w, w.w + w.w_half, sums, G.B, G.o, mm, G.og, f.n,
                 f.tiles, f.n_pad, w.map_k, runs, len,
                 half && w.half ? p->half : nullptr);
    else if (dY)
      launch_pdl(split_dy_kernel, dim3(std::min((G.B * G.o + 7) / 8, ctx->sm_count * 8)), dim3(256), 0, ctx->stream, dY, w.w, w.w + w.w_half, sums,
                 G.B * G.o, G.o, mm, G.og, f.n, f.tiles, f.n_pad, w.map_k);
    CCT_CHECK_LAUNCH(ctx);
    GatherParams P{};
    P.in = X; P.out = p->w_partial; P.bias = nullptr;
    P.n_pix = p->wg_mtiles * kTileM;  // lanes = rows of the lowered matrix
    P.in_lim = G.n;
    P.in_group_stride = G.Dg * G.n * G.n;
    P.wg_mtiles = p->wg_mtiles; P.wg_vgroups = vgroups; P.wg_rows_pad = p->wg_mtiles * kTileM;
    P.wg_k = G.k; P.wg_kreal = f.k_real;
    fill_common(P, w, ctx, vgroups, 0);
    P.taps = p->wg_pix; P.cols = nullptr;
    if (half && w.half) { P.half = p->half; P.half_gathered = kHalfX; P.half_packed = kHalfDy; P.half_row_offset = P.lo_row_offset; }
    P.total_tiles = p->wg_splits * vgroups * p->wg_mtiles;
    launch_gather(ctx, P, w, true);
    t->end(1, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
    if (G.bias) extras.bias = BiasSum{p->wg_plane_sums, db, planes ? G.B : runs, G.o, 0};
    t->begin(2, ctx->stream);
    launch_wgrad_reduce(ctx, p->w_partial, dW, nullptr, p->wg_splits, vgroups, f.tiles, p->wg_mtiles * kTileM, f.n,
                        f.n_pad, f.k_real, G.og, 0, extras, tall);
    t->end(2, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
  } else {
    struct { int tiles, n, n_pad, k_real; } f = {p->wt_tiles, p->wt_n, p->w_npad, p->fwd.k_real};
    WgradParams P{};
    P.x = X; P.dy = dY; P.partial = p->w_partial; P.taps = p->w_taps;
    P.n_pix = G.B * G.m * G.m; P.m = G.m; P.mm = G.m * G.m; P.n = G.n; P.s = G.s; P.p = G.p; P.k = G.k;
    P.x_batch_stride = (long long)G.D * G.n * G.n;
    P.x_group_stride = G.Dg * G.n * G.n;
    P.dy_batch_stride = (long long)G.o * G.m * G.m;
    P.dy_group_channels = G.og;
    P.tiles_per_group = f.tiles;
    P.n_real = f.n; P.n_pad = f.n_pad;
    P.m_tiles = p->w_mtiles; P.subs = p->w_subs; P.stages = p->w_stages;
    P.ones_row = f.k_real;
    P.kblocks_total = p->w_kblocks_total; P.kblocks_per_split = p->w_kblocks_per_split;
    P.status = ctx->status_dev;
    const int vgroups = G.g * f.tiles;
    dim3 grid(p->w_mgroups, p->w_splits, vgroups);
    int rows_pad = p->w_mtiles * kTileM;
    t->begin(1, ctx->stream);
    if (p->w_small) {
      P.n_pad = p->ws_cols * kSwTile;
      rows_pad = p->ws_rows * kSwTile;
      const SmallWgrad J{P, rows_pad, p->ws_rows, p->ws_cols, p->ws_pix, p->ws_rows * p->ws_cols * vgroups};
      const int blocks = J.tiles * p->w_splits;
      if (with) {
        const SmallConvShape g = shape_small_conv(ctx, *with, G.k, 1, p->dgr.small_ct, kSwWarps);
        const int others = g.x * g.y;
        const bool one_round = blocks + others <= SmallBackward::blocks(g.ct) * ctx->sm_count;
        const bool conv_first = with->ci > 2 * kSwWarps ? p->ws_pix == kSwPix && (g.ct == 1 || one_round) : g.rows == kSmallTall && !one_round;
        launch_pdl(small_backward_pick(G.k, g.ct, g.rows), dim3(blocks + others), dim3(kSwThreads), std::max(kSwSmem, g.smem), ctx->stream,
                   SmallBackward{*with, J, g.x, conv_first ? 0 : blocks, conv_first ? others : 0, blocks});
      } else {
        launch_pdl(small_wgrad_kernel, dim3(blocks), dim3(kSwThreads), kSwSmem, ctx->stream, J);
      }
    } else {
      if (p->w_ts) P.x_count = (int)((long long)G.B * G.D * G.n * G.n - (G.g - 1) * P.x_group_stride);
      if (half && p->w_half) {
        P.half = p->half;
        launch_pdl(half_ts_kernel(G.k), dim3(grid), dim3(kThThreads), p->w_smem, ctx->stream, P);
      }
      launch_pdl(short_wgrad_kernel(p), dim3(grid), dim3(p->w_ts ? ts_threads(ts_wide(G)) : kWgThreads), p->w_smem, ctx->stream, P);
    }
    t->end(1, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
    t->begin(2, ctx->stream);
    launch_wgrad_reduce(ctx, p->w_partial, dW, G.bias ? db : nullptr, p->w_splits, vgroups, f.tiles, rows_pad, f.n, P.n_pad,
                        f.k_real, G.og, 0, extras, tall);
    t->end(2, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
  }
  return CCT_OK;
}

}  // namespace
int umma_conv_wgrad(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* dY, float* dW, float* db, PhaseTimer* t, const float* pack_W) {
  return weight_gradient(ctx, p, X, dY, dW, db, t, pack_W, nullptr, false);
}

// Data gradient of the first `batch` images (0: all of them); `repack` rewrites the packed weights from W first; `half`: the scales are
// those of this call's operands.
int umma_conv_dgrad(cct_ctx* ctx, UmmaPlan* p, const float* W, const float* dY, float* dX, PhaseTimer* t, int batch,
                    bool repack) {
  return data_gradient(ctx, p, W, dY, dX, t, batch, repack, false);
}
namespace {
int data_gradient(cct_ctx* ctx, UmmaPlan* p, const float* W, const float* dY, float* dX, PhaseTimer* t, int batch,
                  bool repack, bool half) {
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  const ConvGeom& G = p->G;
  const int B = batch > 0 ? batch : G.B;
  {
    GatherProblem& d = p->dgr;
    const int vgroups = G.g * d.tiles;
    t->begin(3, ctx->stream);
    if (d.small_ct) {
      SmallConv P = small_dgrad(G, dY, W, dX, B);
      launch_small_conv(ctx, P, G.k, 1, d.small_ct, small_together(ctx, p) ? kSwWarps : 0);  // the same sums with and without company
      t->end(3, ctx->stream);
      CCT_CHECK_LAUNCH(ctx);
      return CCT_OK;
    }
    if (repack) {
      const PackDgrad J = pack_dgrad_job(p, d, W, half);
      launch_pdl(pack_dgrad_kernel, dim3(J.blocks), dim3(kPackThreads), 0, ctx->stream, J);
      CCT_CHECK_LAUNCH(ctx);
    }
    GatherParams P{};
    P.in = dY; P.out = dX; P.bias = nullptr;
    P.n_pix = B * p->dgr_q * p->dgr_q; P.q_h = p->dgr_q; P.q_w = p->dgr_q;
    P.iy_mul = 1; P.iy_add = p->dgr_q0; P.ix_mul = 1; P.ix_add = p->dgr_q0;
    P.in_lim = G.m;
    P.tap_sign = -1; P.taps_per_axis = p->dgr_taps;
    P.in_batch_stride = (long long)G.o * G.m * G.m;
    P.in_group_stride = G.og * G.m * G.m;
    const bool rows = !dY;
    if (rows) {  // DyRows
      P.in = p->wgp.w;
      P.in_batch_stride = G.m * G.m;
      P.in_group_stride = (int)(G.og * p->wgp.map_k);
    }
    P.oy_mul = G.s; P.oy_add = p->dgr_q0 * G.s - G.p; P.ox_mul = G.s; P.ox_add = p->dgr_q0 * G.s - G.p;
    P.out_lim = G.n; P.check_out = 1;
    P.out_pitch = G.n; P.out_plane = G.n * G.n;
    P.out_batch_stride = (long long)G.D * G.n * G.n;
    P.out_group_channels = G.Dg;
    P.relu = 0;
    fill_common(P, d, ctx, vgroups, 0);
    if (rows) {
      P.taps = p->dgr_row_taps;
      P.run_stride = (int)p->wgp.map_k;
    }
    if (half && d.half) { P.half = p->half; P.half_gathered = kHalfDy; P.half_packed = kHalfW; P.taps_x = (uint8_t)p->dgr_taps; }
    if (half && p->tall.rows > 1) {
      const GatherProblem& b = p->tall;
      GatherParams Q = P;
      Q.n_pix = B * b.q_h * p->dgr_q; Q.q_h = b.q_h;
      Q.iy_mul = b.rows; Q.iy_add = b.q0 * b.rows + b.rows - 1;
      Q.taps_per_axis = b.taps_y;
      Q.oy_mul = b.rows * G.s; Q.oy_add = b.q0 * b.rows * G.s - G.p;
      fill_common(Q, b, ctx, G.g * b.tiles, 0);
      if (rows) {
        Q.taps = p->tall_row_taps;
        Q.run_stride = (int)p->wgp.map_k;
      }
      Q.only = kOnlyHalf;
      Q.bad_geom = {(uint8_t)G.k, (uint8_t)G.s, (short)G.p, (short)G.m, G.o, G.og};
      P.only = kOnlyTf32;
      launch_gather(ctx, Q, b);
    }
    launch_gather(ctx, P, d);
    t->end(3, ctx->stream);
    CCT_CHECK_LAUNCH(ctx);
  }
  return CCT_OK;
}
}  // namespace

// ------------------------------------------------------------------ weight gradient without any allocation
// Scratch for cct_conv_weight_grad_noalloc: the lowered-matrix row table followed by the split partial sums.  It is a
// fixed part of the library image: every device that loads the library holds these 16 MiB until the process exits.
constexpr size_t kNoAllocScratchBytes = 16u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// Device address of the array above, per device ordinal, looked up once.  In host code the array's name is only a
// handle for the runtime, never an address a kernel may be given.
static void* g_noalloc_dev_ptr[64] = {};

namespace {

// Fills the weight-gradient row table on the device (the plan-based path builds it on the host and uploads it).
__global__ void noalloc_taps_kernel(MaskTap* taps, int rows, int k_real, int k, int n) {
  pdl_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
    MaskTap t;
    if (i < k_real) {
      const int d = i / (k * k), kr = (i / k) % k, kc = i % k;
      t.off = d * n * n + kr * n + kc;
      t.bits = kWgValidBit | (1u << kr) | (1u << (16 + kc));
    } else {
      t.off = 0;
      t.bits = i == k_real ? kWgOnesBits : kWgPadBit;
    }
    taps[i] = t;
  }
}

}  // namespace

extern "C" int cct_conv_weight_grad_noalloc(cct_ctx* ctx, const cct_conv_desc* desc, const float* X, const float* dY,
                                            float* dW, float* db) {
  if (!ctx || !desc || !X || !dY || !dW) return CCT_ERR_INVALID;
  if (desc->batch <= 0 || desc->in_depth <= 0 || desc->in_size <= 0 || desc->out_depth <= 0 || desc->kernel <= 0 ||
      desc->stride <= 0 || desc->pad < 0 || desc->groups <= 0 || desc->in_depth % desc->groups ||
      desc->out_depth % desc->groups || desc->in_size + 2 * desc->pad < desc->kernel)
    return CCT_ERR_INVALID;
  if (desc->bias_term && !db) return CCT_ERR_INVALID;
  ConvGeom G;
  G.B = desc->batch; G.D = desc->in_depth; G.n = desc->in_size; G.o = desc->out_depth;
  G.k = desc->kernel; G.s = desc->stride; G.p = desc->pad; G.g = desc->groups;
  G.m = (G.n + 2 * G.p - G.k) / G.s + 1;
  G.Dg = G.D / G.g; G.og = G.o / G.g; G.bias = desc->bias_term != 0;
  if ((double)G.B * G.D * G.n * G.n > 2147483647.0 || (double)G.B * G.o * G.m * G.m > 2147483647.0 ||
      !umma_supported(G)) {
    ctx->last_error = "cct_conv_weight_grad_noalloc: shape outside what the tensor-core path supports";
    return CCT_ERR_UNSUPPORTED;
  }
  if (ctx->device < 0 || ctx->device >= 64) return CCT_ERR_UNSUPPORTED;
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  // Set-up, once per device and with that device current: ask the runtime where the array lives on this device.
  if (!g_noalloc_dev_ptr[ctx->device]) {
    void* ptr = nullptr;
    CCT_CUDA(ctx, cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    g_noalloc_dev_ptr[ctx->device] = ptr;
  }
  unsigned char* scratch = static_cast<unsigned char*>(g_noalloc_dev_ptr[ctx->device]);

  // Same tiling rules as the plan-based path.
  int chain;
  const int tiles = weight_grad_tiles(G.og, &chain);
  const int n_real = (G.og + tiles - 1) / tiles, n_pad = round_up(n_real, 16);
  const int k_real = G.Dg * G.k * G.k;
  const int m_tiles = (k_real + 1 + kTileM - 1) / kTileM;
  int subs = 1;
  for (int u = 2; u <= kWgMaxSubs; ++u)
    if (u <= m_tiles && u * (n_pad <= 64 ? 2 : 1) * n_pad <= 512 &&
        2 * wg_smem(n_pad, u, 2).stage_bytes + 8192 <= (uint32_t)kSmemLimit)
      subs = u;
  const int mgroups = (m_tiles + subs - 1) / subs;
  const int stages = std::max(2, std::min(kWgMaxStages, (int)((kSmemLimit - 8192) / wg_smem(n_pad, subs, 2).stage_bytes)));
  const size_t smem = wg_smem(n_pad, subs, stages).total + 1024;
  const int vgroups = G.g * tiles;
  const size_t taps_bytes = ((size_t)m_tiles * kTileM * sizeof(MaskTap) + 255) & ~(size_t)255;
  const size_t split_bytes = (size_t)vgroups * m_tiles * kTileM * n_pad * sizeof(float);
  if (taps_bytes + split_bytes > kNoAllocScratchBytes) {
    char msg[200];
    snprintf(msg, sizeof msg,
             "cct_conv_weight_grad_noalloc: this layer needs %zu bytes of scratch for one split, the built-in buffer "
             "holds %zu",
             taps_bytes + split_bytes, kNoAllocScratchBytes);
    ctx->last_error = msg;
    return CCT_ERR_UNSUPPORTED;
  }
  const int n_pix = G.B * G.m * G.m;
  const int kblocks_total = (n_pix + kBlockK - 1) / kBlockK;
  // Splits: one wave of CTAs, and - as in the plan-based path - enough of them that no partial sum's accumulation
  // chain exceeds kMaxChainKblocks (the tensor core's fp32 accumulate truncates; the split reduction rounds).  When
  // the array cannot hold that many partial-sum slices, the pixel range is covered in several rounds of (weight
  // gradient kernel, reduction), each round reusing the slices and the later reductions adding to dW / db.
  int want = std::max(1, ctx->sm_count / (mgroups * vgroups));
  want = std::max(want, (kblocks_total + chain - 1) / chain);
  want = std::min(want, std::max(1, kblocks_total / 8));  // at least 8 k-blocks per CTA (chain > 8)
  const int kblocks_per_split = (kblocks_total + want - 1) / want;
  const int total_splits = (kblocks_total + kblocks_per_split - 1) / kblocks_per_split;
  const int slots = (int)std::min<size_t>((kNoAllocScratchBytes - taps_bytes) / split_bytes, (size_t)total_splits);

  MaskTap* taps = reinterpret_cast<MaskTap*>(scratch);
  float* partial = reinterpret_cast<float*>(scratch + taps_bytes);
  WgradKernel kernel = wgrad_pick(subs, n_pad);
  CCT_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
  launch_pdl(noalloc_taps_kernel, dim3(8), dim3(256), 0, ctx->stream, taps, m_tiles * kTileM, k_real, G.k, G.n);
  CCT_CHECK_LAUNCH(ctx);
  WgradParams P{};
  P.x = X; P.dy = dY; P.partial = partial; P.taps = taps;
  P.n_pix = n_pix; P.m = G.m; P.mm = G.m * G.m; P.n = G.n; P.s = G.s; P.p = G.p; P.k = G.k;
  P.x_batch_stride = (long long)G.D * G.n * G.n;
  P.x_group_stride = G.Dg * G.n * G.n;
  P.dy_batch_stride = (long long)G.o * G.m * G.m;
  P.dy_group_channels = G.og;
  P.tiles_per_group = tiles;
  P.n_real = n_real; P.n_pad = n_pad;
  P.m_tiles = m_tiles; P.subs = subs; P.stages = stages;
  P.ones_row = k_real;
  P.kblocks_per_split = kblocks_per_split;
  P.status = ctx->status_dev;
  for (int first = 0, round = 0; first < total_splits; first += slots, ++round) {
    const int here = std::min(slots, total_splits - first);
    P.kb_first = first * kblocks_per_split;
    P.kblocks_total = std::min(kblocks_total, P.kb_first + here * kblocks_per_split);
    launch_pdl(kernel, dim3(dim3(mgroups, here, vgroups)), dim3(kWgThreads), smem, ctx->stream, P);
    CCT_CHECK_LAUNCH(ctx);
    launch_wgrad_reduce(ctx, partial, dW, G.bias ? db : nullptr, here, vgroups, tiles, m_tiles * kTileM, n_real, n_pad,
                        k_real, G.og, round > 0);
    CCT_CHECK_LAUNCH(ctx);
  }
  return CCT_OK;
}

// ------------------------------------------------------------------ the bounded wait, exercised on purpose
namespace {
// One warp waits - through the same mbar_wait the convolution kernels use - for a barrier phase that nothing will ever
// complete, with a short limit.  The wait gives up, records `code` in the status word and the kernel returns
// normally: no trap, no fault, the context stays usable.
__global__ void bounded_wait_selftest_kernel(int* status, long long limit_cycles, int code) {
  pdl_wait();
  __shared__ __align__(8) unsigned long long bar_storage;
  const uint32_t bar = smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  bool failed = false;
  mbar_wait(bar, 0u, failed, status, code, limit_cycles);
}
}  // namespace

extern "C" int cct_selftest_bounded_wait(cct_ctx* ctx, long long limit_cycles) {
  if (!ctx || limit_cycles <= 0 || limit_cycles > kWaitLimitCycles) return CCT_ERR_INVALID;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  launch_pdl(bounded_wait_selftest_kernel, dim3(1), dim3(32), 0, ctx->stream, ctx->status_dev, limit_cycles, 0x7e57);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}
