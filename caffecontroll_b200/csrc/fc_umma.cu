// Fully connected layers on the Blackwell tensor cores (FullyConnectedBridge: src/bridges/FullyConnectedBridge_impl.hxx).
//
// The three contractions of the bridge
//   forward        Y[b][o]  = sum_k X[b][k]  * W[o][k]          (:196-215, sgemm_new NoTrans x Trans)
//   data gradient  dX[b][k] = sum_o dY[b][o] * W[o][k]          (:305, NoTrans x NoTrans)
//   weight gradient dW[o][k] = sum_b dY[b][o] * X[b][k]         (:311, Trans x NoTrans)
// are one kernel, fc_gemm_kernel:   out[n][m] = sum_r A(m, r) * B(n, r)   with M = 128 lanes per tile, N <= 256.
// Both operands are fetched from global memory by TMA as raw fp32 tiles of 32 reduction indices.  An operand whose
// reduction index is contiguous in memory ("K-major": W in the forward pass, X, dY) lands as rows of 128 bytes with
// the 128-byte swizzle; an operand whose row index is contiguous ("MN-major": W in the data gradient, X and dY in the
// weight gradient, where the reduction runs over the batch) lands as 32 x 32 boxes with the 128-byte swizzle of
// 32-byte atoms, the only shared-memory layout tcgen05.mma accepts for transposed 32-bit operands.  No operand is ever
// transposed or re-packed in global memory: the weights stream from HBM exactly once per contraction.
//
// 3xTF32: kind::tf32 reads the upper 19 bits of every fp32 operand word, so the raw tile is the "hi" operand as it
// stands; transform warps compute lo = x - hi element-wise into a second tile of the same layout (an element-wise pass
// is layout-agnostic, so it serves both swizzles), and three MMAs per k-step (lo*hi + hi*lo + hi*hi) accumulate in
// fp32 in tensor memory.  Long reductions are split over CTAs (bounded accumulation chains, as in the convolution
// kernels); a small kernel adds the partial sums in split order and applies bias / ReLU / dropout (forward) or the
// masks of the bridges in front of the layer (data gradient).
#include <algorithm>
#include <cstdio>
#include <new>

#include "cct_internal.h"
#include "umma_ptx.cuh"

namespace {

constexpr int kFcEpiWarps = 4, kFcTmaWarp = 4, kFcMmaWarp = 5, kFcXformWarp0 = 6, kFcXformWarps = 8;
constexpr int kFcThreads = (kFcXformWarp0 + kFcXformWarps) * 32;  // 448
constexpr int kFcRing = 4;                    // deepest ring of any kind; the lo and done barriers are a ring of four
constexpr int kFcMaxChainKblocks = 96;        // k-blocks of 32 per partial sum: the tensor core's fp32 accumulate truncates
constexpr uint32_t kFcATile = kTileM * 128u;  // bytes of one 128 x 32 fp32 tile
constexpr uint32_t kFcStoreTile = 32u * 32u * 4u;  // 32 columns x 32 lanes on their way out

struct FcGemmParams {
  int M, N;                 // extents of the output (m fastest in memory)
  int n_pad;                // accumulator columns per tile: N rounded up (a multiple of 32 for MN-major B)
  int m_tiles, n_tiles, splits, kblocks_total, kblocks_per_split;
  int a_mn, b_mn;           // 1: the operand is MN-major (row index contiguous in memory)
  int raw_slots, lo_slots, a_slots, acc_bufs, store_bufs;
  int tmem_cols;            // tensor-memory columns the CTA allocates: 512, or 256 when two CTAs share an SM
  float* direct;            // non-null: plain stores to direct[n * ld_direct + m] (an output no tensor map describes)
  long long ld_direct;
  int* status;
};

// Raw ring (A tile and B tile as TMA delivers them), lo ring (B's lo tiles), the tiles on their way out.
struct FcSmem {
  uint32_t b_tile_bytes, raw_bytes, lo_off, store_off, total;
};
__host__ __device__ inline FcSmem fc_smem(int n_pad, int raw_slots, int lo_slots, int store_bufs) {
  FcSmem L;
  L.b_tile_bytes = (uint32_t)n_pad * 128u;
  L.raw_bytes = kFcATile + L.b_tile_bytes;
  L.lo_off = (uint32_t)raw_slots * L.raw_bytes;
  L.store_off = L.lo_off + (uint32_t)lo_slots * L.b_tile_bytes;
  L.total = L.store_off + (uint32_t)(kFcEpiWarps * store_bufs) * kFcStoreTile;  // the barriers go where the 1 KB of alignment slack leaves room
  return L;
}

// Shared-memory descriptor of an MN-major fp32 operand: 32 x 32 boxes (row = one reduction index, 128 bytes = 32
// consecutive m), 128-byte swizzle with 32-byte atoms (layout type 1).  One MMA reads 8 reduction indices = two atoms
// of four rows, 512 bytes apart; consecutive 32-wide chunks of m are one box (4096 bytes) apart.
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(4096u >> 4) << 16) | ((uint64_t)(512u >> 4) << 32) |
         (1ull << 46) | (1ull << 61);
}

__device__ __forceinline__ void fc_store_3d(const void* tmap, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(tmap), "r"(x), "r"(y), "r"(z),
               "r"(src)
               : "memory");
}

// What bounds it: at batch 256 the tensor pipe (12 MMAs of N / 2 cycles per k-block; fc6's forward pass 84 us, data gradient 76, pipe
// 83 % active on the 128 and 144 SMs with a block, banks of shared memory 40 - 45 % busy), at small batches the stream of W (or,
// for the weight gradient, of dW) - so the same roles in two shapes.
//   N > 128 columns: one CTA per SM, the whole batch in one accumulator, so that a weight tile is split into tensor memory
//   once (two CTAs with half the batch each split it twice and waited for it: 61 % of the tensor pipe).
//   N <= 128: two CTAs per SM, 256 tensor-memory columns each.
// K-block i (running index) uses raw slot i % raw_slots, lo slot i % lo_slots, tensor-memory slot i % a_slots; the raw slot,
// which is also the hi operand, is held for TMA + transform + MMA, the other two only from transform to MMA, so the raw ring
// is the deeper one.  raw[slot] completes when the TMA bytes have landed, lo[i % 4] when the transform warps are through,
// done[i % 4] when the block's MMAs have finished, which frees all three slots (nobody waits more than four blocks back).
// The epilogue turns 32 accumulator columns at a time into a 32 x 32 tile in shared memory (one conflict-free store per
// column) that TMA stores take out, clipping it at the edges: per-lane global stores with their addresses and bounds cost
// about ten instructions each and made the weight gradient of small batches instruction-bound (fc6, batch 32: 70 us, 2.1 TB/s).
// TWO: block `block0` of `blocks` that share the tiles (else the grid's: said of the loops as such, since with variables in their place fc6
// at batch 256 took 308 us both ways instead of 300).
template <bool TWO>
__device__ __forceinline__ void fc_gemm_body(const FcGemmParams& P, const CUtensorMap& a_map, const CUtensorMap& b_map, const CUtensorMap& out_map,
                                             unsigned block0, unsigned blocks) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const FcSmem L = fc_smem(P.n_pad, P.raw_slots, P.lo_slots, P.store_bufs);
  // 1 KB more than L.total is allocated: either in front of the aligned base or behind the tiles there is room for these
  constexpr uint32_t kBarBytes = 8u * (3 * kFcRing + 4) + 24u;
  const uint32_t bars = base - smem_u32(smem_raw) >= kBarBytes ? (smem_u32(smem_raw) + 7u) & ~7u : base + L.total;  // 8-byte aligned
  const uint32_t raw_bar = bars, lo_bar = raw_bar + 8u * kFcRing, done_bar = lo_bar + 8u * kFcRing,
                 acc_full = done_bar + 8u * kFcRing, acc_empty = acc_full + 16u, tmem_slot = acc_empty + 16u;
  const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kFcRing; ++s) {
      mbar_init(raw_bar + 8u * s, 1);
      mbar_init(lo_bar + 8u * s, kFcXformWarps);
      mbar_init(done_bar + 8u * s, 1);
    }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full + 8u * b, 1); mbar_init(acc_empty + 8u * b, kFcEpiWarps); }
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, (uint32_t)P.tmem_cols);
  if (warp == kFcTmaWarp) { prefetch_map(&a_map); prefetch_map(&b_map); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const uint32_t a_col0 = (uint32_t)(P.acc_bufs * P.n_pad);  // A slots (64 columns: 32 hi + 32 lo) behind the accumulators
  const int total_tiles = P.m_tiles * P.n_tiles * P.splits;
  bool failed = false;
  // tile t -> (split, n-tile, m-tile), m-tile fastest; k-blocks [kb0, kb1)
  auto tile_of = [&](int t, int& mt, int& nt, int& split, int& kb0, int& kb1) {
    mt = t % P.m_tiles;
    const int r = t / P.m_tiles;
    nt = r % P.n_tiles;
    split = r / P.n_tiles;
    kb0 = split * P.kblocks_per_split;
    kb1 = min(P.kblocks_total, kb0 + P.kblocks_per_split);
  };
  // the MMAs of the k-block `back` blocks before block i have finished
  auto wait_done = [&](int i, int back, int code) {
    const int j = i - back;
    if (j >= 0) mbar_wait<false>(done_bar + 8u * (j & 3), (uint32_t)(j >> 2) & 1u, failed, P.status, code);
  };

  if (warp == kFcTmaWarp) {
    if (lane == 0) {
      Ring ring;
      int i = 0;
      for (int t = TWO ? block0 : blockIdx.x; t < total_tiles; t += TWO ? blocks : gridDim.x) {
        int mt, nt, split, kb0, kb1;
        tile_of(t, mt, nt, split, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb, ++i, ring.advance(P.raw_slots)) {
          wait_done(i, P.raw_slots, 0x1100);
          const uint32_t a_raw = base + (uint32_t)ring.idx * L.raw_bytes, b_raw = a_raw + kFcATile;
          const uint32_t bar = raw_bar + 8u * ring.idx;
          mbar_expect_tx(bar, kFcATile + L.b_tile_bytes);
          if (P.a_mn) {
#pragma unroll
            for (int j = 0; j < 4; ++j) tma_load_2d(a_raw + j * 4096u, &a_map, mt * kTileM + j * 32, kb * kBlockK, bar);
          } else {
            tma_load_2d(a_raw, &a_map, kb * kBlockK, mt * kTileM, bar);
          }
          if (P.b_mn) {
            for (int j = 0; j < P.n_pad / 32; ++j)
              tma_load_2d(b_raw + j * 4096u, &b_map, nt * P.n_pad + j * 32, kb * kBlockK, bar);
          } else {
            tma_load_2d(b_raw, &b_map, kb * kBlockK, nt * P.n_pad, bar);
          }
        }
      }
    }
  } else if (warp == kFcMmaWarp) {  // see elect_one
    const uint32_t idesc = make_idesc(P.n_pad) | (P.b_mn ? 1u << 16 : 0u);  // A from tensor memory: lanes x K
    const uint32_t tmem = warp_uniform(tmem_base);
    Ring raw, lo, ta;
    int i = 0, tile_iter = 0;
    for (int t = TWO ? block0 : blockIdx.x; t < total_tiles; t += TWO ? blocks : gridDim.x, ++tile_iter) {
      int mt, nt, split, kb0, kb1;
      tile_of(t, mt, nt, split, kb0, kb1);
      const int buf = tile_iter & (P.acc_bufs - 1), use = tile_iter >> (P.acc_bufs - 1);
      if (use > 0) mbar_wait<false>(acc_empty + 8u * buf, (uint32_t)(use - 1) & 1u, failed, P.status, 0x1200);
      tc_fence_after();
      const uint32_t d_tmem = tmem + (uint32_t)(buf * P.n_pad);
      for (int kb = kb0; kb < kb1; ++kb, ++i) {
        mbar_wait<false>(raw_bar + 8u * raw.idx, (uint32_t)raw.use & 1u, failed, P.status, 0x1300);
        mbar_wait<false>(lo_bar + 8u * (i & 3), (uint32_t)(i >> 2) & 1u, failed, P.status, 0x1400);
        tc_fence_after();
        const uint32_t b_raw = base + (uint32_t)raw.idx * L.raw_bytes + kFcATile;
        const uint32_t b_lo = base + L.lo_off + (uint32_t)lo.idx * L.b_tile_bytes;
        const uint32_t t_hi = tmem + a_col0 + (uint32_t)(ta.idx * 64), t_lo = t_hi + 32u;
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < kBlockK / 8; ++j) {
            // K-major: 8 reduction indices = 32 bytes along the swizzled row; MN-major: 8 rows of 128 bytes
            const uint64_t bh = P.b_mn ? make_desc_mn(b_raw + j * 1024u) : make_desc(b_raw) + (uint64_t)(j * 2);
            const uint64_t bl = P.b_mn ? make_desc_mn(b_lo + j * 1024u) : make_desc(b_lo) + (uint64_t)(j * 2);
            umma_tf32_ts(d_tmem, t_lo + (uint32_t)(j * 8), bh, idesc, (kb == kb0 && j == 0) ? 0u : 1u);
            umma_tf32_ts(d_tmem, t_hi + (uint32_t)(j * 8), bl, idesc, 1u);
            umma_tf32_ts(d_tmem, t_hi + (uint32_t)(j * 8), bh, idesc, 1u);
          }
          umma_commit(done_bar + 8u * (i & 3));
          if (kb == kb1 - 1) umma_commit(acc_full + 8u * buf);
        }
        __syncwarp();
        raw.advance(P.raw_slots);
        lo.advance(P.lo_slots);
        ta.advance(P.a_slots);
      }
    }
  } else if (warp >= kFcXformWarp0) {
    // ---- A: hi and lo into tensor memory; B: lo = x - (x with the low 13 mantissa bits cleared), element-wise
    const int xt = tid - kFcXformWarp0 * 32;
    constexpr int kXThreads = kFcXformWarps * 32;
    const int b_vec = (int)(L.b_tile_bytes / 16);
    const int q = warp & 3, half = (warp - kFcXformWarp0) >> 2;
    const int m = q * 32 + lane;  // row of the tile = tensor-memory lane; this thread takes half of the k-block's 32 indices
    const int back = min(P.lo_slots, P.a_slots);
    Ring raw, lo, ta;
    int i = 0;
    for (int t = TWO ? block0 : blockIdx.x; t < total_tiles; t += TWO ? blocks : gridDim.x) {
      int mt, nt, split, kb0, kb1;
      tile_of(t, mt, nt, split, kb0, kb1);
      for (int kb = kb0; kb < kb1; ++kb, ++i) {
        mbar_wait(raw_bar + 8u * raw.idx, (uint32_t)raw.use & 1u, failed, P.status, 0x1500);
        if (i >= back) mbar_wait(done_bar + 8u * ((i - back) & 3), (uint32_t)((i - back) >> 2) & 1u, failed, P.status, 0x1510);
        tc_fence_after();
        const uint8_t* st = base_ptr + (size_t)raw.idx * L.raw_bytes;
        float x[16];
        if (P.a_mn) {
          // 32 x 32 boxes, row = reduction index (128 bytes), 32-byte chunks XORed with the row index mod 4
          const uint8_t* box = st + (size_t)(m >> 5) * 4096u;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const uint32_t k = (uint32_t)(half * 16 + e);
            const uint32_t off = k * 128u + (uint32_t)(m & 31) * 4u;
            x[e] = *reinterpret_cast<const float*>(box + (off ^ ((k & 3u) << 5)));
          }
        } else {
          // rows of 128 bytes, 16-byte chunks XORed with the row index mod 8
          const uint8_t* rowp = st + (size_t)m * 128u;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t c = (uint32_t)(half * 4 + e);
            const float4 v4 = *reinterpret_cast<const float4*>(rowp + ((c ^ (uint32_t)(m & 7)) << 4));
            x[4 * e] = v4.x; x[4 * e + 1] = v4.y; x[4 * e + 2] = v4.z; x[4 * e + 3] = v4.w;
          }
        }
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + a_col0 + (uint32_t)(ta.idx * 64 + half * 16);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t hi[8], l8[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) split_tf32_trunc(x[c * 8 + e], hi[e], l8[e]);
          tmem_st8(taddr + (uint32_t)(c * 8), hi);
          tmem_st8(taddr + 32u + (uint32_t)(c * 8), l8);
        }
        const float4* b_raw = reinterpret_cast<const float4*>(st + kFcATile);
        float4* b_lo = reinterpret_cast<float4*>(base_ptr + L.lo_off + (size_t)lo.idx * L.b_tile_bytes);
#pragma unroll 4
        for (int v = xt; v < b_vec; v += kXThreads) {
          const float4 r = b_raw[v];
          float4 l;
          l.x = r.x - __uint_as_float(__float_as_uint(r.x) & 0xFFFFE000u);
          l.y = r.y - __uint_as_float(__float_as_uint(r.y) & 0xFFFFE000u);
          l.z = r.z - __uint_as_float(__float_as_uint(r.z) & 0xFFFFE000u);
          l.w = r.w - __uint_as_float(__float_as_uint(r.w) & 0xFFFFE000u);
          b_lo[v] = l;
        }
        fence_proxy_async_smem();
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(lo_bar + 8u * (i & 3));
        raw.advance(P.raw_slots);
        lo.advance(P.lo_slots);
        ta.advance(P.a_slots);
      }
    }
  } else {
    // ---- epilogue: lane = m (contiguous in the output), one column = one n
    const int quarter = warp;  // warps 0-3 own tensor-memory lanes 32 * warp ...
    uint8_t* out_ptr = base_ptr + L.store_off + (size_t)(warp * P.store_bufs) * kFcStoreTile;
    const uint32_t out_smem = base + L.store_off + (uint32_t)(warp * P.store_bufs) * kFcStoreTile;
    int tile_iter = 0, stores = 0;
    for (int t = TWO ? block0 : blockIdx.x; t < total_tiles; t += TWO ? blocks : gridDim.x, ++tile_iter) {
      int mt, nt, split, kb0, kb1;
      tile_of(t, mt, nt, split, kb0, kb1);
      const int buf = tile_iter & (P.acc_bufs - 1), use = tile_iter >> (P.acc_bufs - 1);
      mbar_wait(acc_full + 8u * buf, (uint32_t)use & 1u, failed, P.status, 0x1600);
      tc_fence_after();
      const int m0 = mt * kTileM + quarter * 32, n0 = nt * P.n_pad;
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * P.n_pad);
      const int chunks = min(P.n_pad, P.N - n0 + 15) / 16;  // columns behind N are never looked at
      for (int c = 0; c < chunks; c += 2) {  // 32 columns a step: one round of waits, fence and stores for them
        float v[2][16];
        const bool two = c + 1 < chunks;
        tmem_ld16(acc + (uint32_t)(c * 16), v[0]);
        if (two) tmem_ld16(acc + (uint32_t)(c * 16 + 16), v[1]);
        if (failed || m0 >= P.M) continue;
        if (P.direct) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int n = n0 + (c + h) * 16 + j;
              if (m0 + lane < P.M && n < P.N && (h == 0 || two)) P.direct[(long long)n * P.ld_direct + m0 + lane] = v[h][j];
            }
          continue;
        }
        const uint32_t slot = P.store_bufs == 2 ? (uint32_t)(stores++ & 1) * kFcStoreTile : 0u;
        if (lane == 0) {  // the stores that read this tile last have done so
          if (P.store_bufs == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 16; ++j) *reinterpret_cast<float*>(out_ptr + slot + (h * 16 + j) * 128 + lane * 4) = v[h][j];
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          fc_store_3d(&out_map, out_smem + slot, m0, n0 + c * 16, split);
          if (two) fc_store_3d(&out_map, out_smem + slot + 2048u, m0, n0 + c * 16 + 16, split);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8u * buf);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, (uint32_t)P.tmem_cols);
}
__global__ void __launch_bounds__(kFcThreads, 2)
    fc_gemm_kernel(const __grid_constant__ FcGemmParams P, const __grid_constant__ CUtensorMap a_map,
                   const __grid_constant__ CUtensorMap b_map, const __grid_constant__ CUtensorMap out_map) {
  fc_gemm_body<false>(P, a_map, b_map, out_map, 0, 0);
}
// The two contractions of a backward pass of few tiles in one launch: blocks [0, first) work on the weight gradient, those behind them on
// the data gradient.  Each of such a layer's launches is five microseconds of set-up and hand-overs however little it does: 800 -> 500,
// 64 images, both ways 19.4 -> 15.2 us, LeNet's iteration 94.2 -> 89.9.
struct FcJob {
  FcGemmParams P;
  CUtensorMap a, b, out;
};
__global__ void __launch_bounds__(kFcThreads, 2) fc_gemm_two_kernel(const __grid_constant__ FcJob w, const __grid_constant__ FcJob d, unsigned first) {
  const bool second = blockIdx.x >= first;
  const FcGemmParams P = second ? d.P : w.P;
  const FcJob& J = second ? d : w;
  fc_gemm_body<true>(P, J.a, J.b, J.out, blockIdx.x - (second ? first : 0u), second ? gridDim.x - first : first);
}

// db[o] = sum_b dY[b][o] (FullyConnectedBridge_impl.hxx:298: backward_bias_fc).  A block of 32 x 8 threads owns 32
// outputs: thread (x, y) adds the images y, y + 8, ... in order with sixteen loads in flight, then the eight partial sums
// of an output are added in a fixed order - deterministic, and two memory round trips instead of B.
struct FcBiasSum {
  const float* dY;
  float* db;
  int B, O;
};
__device__ __forceinline__ void fc_bias_grad_block(const FcBiasSum& J, int block) {
  __shared__ float part[8][33];
  const float* dY = J.dY;
  const int B = J.B, O = J.O;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int o = block * 32 + tx;
  float acc = 0.f;
  if (o < O) {
    int b = ty;
    for (; b + 8 * 15 < B; b += 8 * 16) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __ldg(dY + (size_t)(b + 8 * j) * O + o);
#pragma unroll
      for (int j = 0; j < 16; ++j) acc += v[j];
    }
    for (; b < B; b += 8) acc += dY[(size_t)b * O + o];
  }
  part[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && o < O) {
    float t = part[0][tx];
#pragma unroll
    for (int y = 1; y < 8; ++y) t += part[y][tx];
    J.db[o] = t;
  }
}
__global__ void __launch_bounds__(256) fc_bias_grad_kernel(const __grid_constant__ FcBiasSum J) {
  pdl_wait();
  fc_bias_grad_block(J, blockIdx.x);
}

// Sums the splits of a contraction in split order and applies what surrounds it, VEC columns of a row per thread.
//   forward        Y[b][o] = act(bias[o] + sum), act = optional ReLU then optional dropout (DropoutBridge forward:
//                  x * mask * scale, src/bridges/DropoutBridge_impl.hxx:71-74)
//   data gradient  dX[b][k] = sum x mask * scale (DropoutBridge::backward) x [X > 0] (the ReLU bridge in front,
//                  src/kernels/relu.hxx:35-43)
struct FcReduceParams {
  const float* partial;      // [splits][rows][pitch]
  float* out;                // [rows][cols]
  const float* bias;         // forward
  const float* X;            // data gradient: the ReLU mask's source, or null
  const uint32_t* drop_mask;
  float drop_scale;
  int rows, cols, pitch, splits, relu;
  // data gradient: the layer's bias gradient in blocks behind the others (a launch less; `sum_blocks` of the grid are not)
  unsigned sum_blocks = 0;
  FcBiasSum bias_sum{};
};
// SLICES > 1: a block's eight warps take interleaved slices of the splits of the same 32 x VEC elements and add them in a
// fixed order - small outputs with many splits, where one thread per element would be a long chain on a few SMs.
// BIAS: blocks behind the others add the layer's bias gradient (data gradient).
template <int VEC, int SLICES, bool BIAS>
__global__ void __launch_bounds__(256) fc_reduce_kernel(const __grid_constant__ FcReduceParams P) {
  pdl_wait();
  if (BIAS && blockIdx.x >= P.sum_blocks) {
    fc_bias_grad_block(P.bias_sum, (int)(blockIdx.x - P.sum_blocks));
    return;
  }
  __shared__ float part[SLICES > 1 ? SLICES : 1][VEC][33];
  const int per_row = (P.cols + VEC - 1) / VEC;
  const int lane = threadIdx.x & 31, slice = SLICES > 1 ? threadIdx.x >> 5 : 0;
  const long long t = SLICES > 1 ? blockIdx.x * 32ll + lane : blockIdx.x * 256ll + threadIdx.x;
  const bool in = t < (long long)P.rows * per_row;
  const int row = !in ? 0 : t <= 0x7fffffffll ? (int)t / per_row : (int)(t / per_row);
  const int col = in ? (int)(t - (long long)row * per_row) * VEC : 0;
  const float* src = P.partial + (size_t)row * P.pitch + col;
  const size_t stride = (size_t)P.rows * P.pitch;
  float acc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
#pragma unroll 4
  for (int s = slice; s < P.splits; s += SLICES) {
    const float* at = src + s * stride;
    if (VEC == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(at));
      acc[0] += v.x; acc[VEC > 1 ? 1 : 0] += v.y; acc[VEC > 2 ? 2 : 0] += v.z; acc[VEC > 3 ? 3 : 0] += v.w;
    } else {
      acc[0] += __ldg(at);
    }
  }
  if (SLICES > 1) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) part[slice][e][lane] = acc[e];
    __syncthreads();
    if (slice) return;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
#pragma unroll
      for (int y = 1; y < SLICES; ++y) acc[e] += part[y][e][lane];
  }
  if (!in) return;
  const size_t at = (size_t)row * P.cols + col;
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    if (P.bias) acc[e] += __ldg(P.bias + col + e);
    if (P.relu) acc[e] = fmaxf(acc[e], 0.f);
    if (P.drop_mask) acc[e] = acc[e] * (float)(P.drop_mask[at + e] != 0u) * P.drop_scale;
    if (P.X) acc[e] = acc[e] * (P.X[at + e] > 0.f ? 1.f : 0.f);
  }
  if (VEC == 4) *reinterpret_cast<float4*>(P.out + at) = make_float4(acc[0], acc[VEC > 1 ? 1 : 0], acc[VEC > 2 ? 2 : 0], acc[VEC > 3 ? 3 : 0]);
  else P.out[at] = acc[0];
}

// A row-major matrix whose rows are no multiple of 16 bytes, copied into rows that are (the tensor maps' pitch rule).
__global__ void __launch_bounds__(256) fc_pad_kernel(const float* __restrict__ src, float* __restrict__ dst, int rows, int cols, int pitch) {
  pdl_wait();
  for (int r = blockIdx.y; r < rows; r += gridDim.y)
    for (int c = blockIdx.x * 256 + threadIdx.x; c < pitch; c += gridDim.x * 256)
      dst[(size_t)r * pitch + c] = c < cols ? __ldg(src + (size_t)r * cols + c) : 0.f;
}

int fc_round_up(int v, int a) { return (v + a - 1) / a * a; }
}  // namespace
#include "fc_small.cuh"
namespace {

int fc_encode(cct_ctx* ctx, CUtensorMap* map, const float* ptr, int rank, const cuuint64_t* dim, const cuuint64_t* stride,
              const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) {
    ctx->last_error = "cuTensorMapEncodeTiled is not available from this driver";
    return CCT_ERR_CUDA;
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank, const_cast<float*>(ptr), dim, stride, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    ctx->last_error = "cuTensorMapEncodeTiled (fully connected operand) failed with code " + std::to_string((int)r);
    return CCT_ERR_CUDA;
  }
  return CCT_OK;
}

// A tensor map and the address it was made for: a training loop passes the same buffers every time.
struct FcMap {
  CUtensorMap map;
  const float* ptr = nullptr;
};

// rows x cols fp32 matrix, cols contiguous, rows `pitch` floats apart.  K-major use: box = 32 cols (reduction) x box_rows,
// 128-byte swizzle.  MN-major use: box = 32 cols (the operand's row index) x 32 rows (reduction), 128-byte swizzle with
// 32-byte atoms.
int fc_operand_map(cct_ctx* ctx, FcMap* m, const float* ptr, size_t rows, size_t cols, size_t pitch, int box_rows, bool mn_major) {
  if (m->ptr == ptr) return CCT_OK;
  const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, stride[1] = {(cuuint64_t)pitch * sizeof(float)};
  const cuuint32_t box[2] = {32u, (cuuint32_t)(mn_major ? 32 : box_rows)};
  const int rc = fc_encode(ctx, &m->map, ptr, 2, dim, stride, box, mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B);
  m->ptr = rc == CCT_OK ? ptr : nullptr;
  return rc;
}

// An output of the contraction: [splits][N][pitch], stored in tiles of 16 rows x 32 columns.
int fc_output_map(cct_ctx* ctx, FcMap* m, const float* ptr, size_t M, size_t N, size_t splits, size_t pitch) {
  if (m->ptr == ptr) return CCT_OK;
  const cuuint64_t dim[3] = {(cuuint64_t)M, (cuuint64_t)N, (cuuint64_t)splits},
                   stride[2] = {(cuuint64_t)pitch * sizeof(float), (cuuint64_t)(N * pitch) * sizeof(float)};
  const cuuint32_t box[3] = {32u, 16u, 1u};
  const int rc = fc_encode(ctx, &m->map, ptr, 3, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE);
  m->ptr = rc == CCT_OK ? ptr : nullptr;
  return rc;
}

// Tile shape, rings and splits of one contraction.
struct FcShape {
  FcGemmParams P{};
  bool pair = false;  // two CTAs per SM
  size_t smem = 0;
};

// Rings that fit: the raw ring first (it holds a slot for TMA + transform + MMA), then the second tile on its way out.
bool fc_fit_rings(FcShape& s) {
  FcGemmParams& P = s.P;
  const size_t budget = s.pair ? 113 * 1024 : kSmemLimit;
  P.tmem_cols = s.pair ? 256 : 512;
  P.a_slots = std::min(kFcRing, (P.tmem_cols - P.acc_bufs * P.n_pad) / 64);
  for (int raw = kFcRing; raw >= 2; --raw)
    for (int st = 2; st >= 1; --st) {
      const int lo = std::min(raw, P.n_pad <= 64 ? 3 : 2);
      const size_t need = fc_smem(P.n_pad, raw, lo, st).total + 1024;
      if (need <= budget) {
        P.raw_slots = raw; P.lo_slots = lo; P.store_bufs = st;
        s.smem = need;
        return P.a_slots >= 2;
      }
    }
  return false;
}

// Forward pass and data gradient: M = the layer's output (input) features, N = batch.  The splits of the reduction are
// chosen by the rounds of (tile, split) units over the resident CTAs: a k-block takes its 12 MMAs, and two CTAs on an SM
// share the tensor pipe; a unit adds set-up and epilogue, a split the traffic of
// one more partial sum.
FcShape fc_batch_shape(int sms, int M, int N, int R) {
  FcShape s;
  FcGemmParams& P = s.P;
  P.M = M; P.N = N;
  P.m_tiles = (M + kTileM - 1) / kTileM;
  P.n_tiles = (N + 255) / 256;
  P.n_pad = fc_round_up((N + P.n_tiles - 1) / P.n_tiles, 16);
  P.acc_bufs = 1;
  s.pair = P.n_pad <= 128;
  P.kblocks_total = (R + kBlockK - 1) / kBlockK;
  // a k-block: its MMAs, or the hand-overs from TMA to transform to MMA (with two raw slots, the room for wide tiles in
  // half an SM, a CTA waits for its own loads: 1.1 us a k-block at 128 columns)
  const double exec = 12 * std::max(P.n_pad / 2.0, 18.0) / 1750.0;
  const double alone = std::max(exec, s.pair && P.n_pad > 64 ? 1.0 : 0.35), shared = std::max(2 * exec, alone);
  const long long slots = (long long)sms * (s.pair ? 2 : 1);
  double best = 0.0;
  for (int n = 1; n <= std::max(1, P.kblocks_total / 2); ++n) {
    const int kps = (P.kblocks_total + n - 1) / n;
    if ((P.kblocks_total + kps - 1) / kps != n || kps > kFcMaxChainKblocks) continue;
    const long long units = (long long)P.m_tiles * P.n_tiles * n, tail = units % slots;
    const double unit = 1.5 + 0.006 * P.n_pad;
    const double us = (units / slots) * (kps * (s.pair ? shared : alone) + unit) +
                      (tail ? kps * (s.pair && tail > sms ? shared : alone) + unit : 0.0) + (double)n * M * N * 8.0 / 4e6;
    if (best == 0.0 || us < best) {
      best = us;
      P.splits = n;
      P.kblocks_per_split = kps;
    }
  }
  return s;
}

// Weight gradient: M = input features, N = output features, reduction over the batch (short): two accumulators, so that
// one is written out while the next is formed.  Widest tiles that do not cost a round.
FcShape fc_weight_shape(int sms, int K, int O, int B) {
  FcShape best;
  double best_us = 0.0;
  for (int n = 192; n >= 32; n -= 32) {
    if (n > 32 && n >= fc_round_up(O, 32) + 32) continue;
    FcShape s;
    FcGemmParams& P = s.P;
    P.M = K; P.N = O;
    P.m_tiles = (K + kTileM - 1) / kTileM;
    P.n_pad = n; P.acc_bufs = 2;
    P.n_tiles = (O + n - 1) / n;
    P.splits = 1;
    P.kblocks_total = P.kblocks_per_split = (B + kBlockK - 1) / kBlockK;
    P.a_mn = P.b_mn = 1;
    const long long rounds = ((long long)P.m_tiles * P.n_tiles + sms - 1) / sms;
    const double mma = P.kblocks_total * std::max(12.0 * n / 2.0 / 1750.0, 0.35), out = 0.2 + 0.006 * n;
    const double us = rounds * std::max(mma, out) + mma + out;
    if (!best.P.n_pad || us < 0.98 * best_us) {
      best = s;
      best_us = us;
    }
  }
  return best;
}

// The weight gradient's shape in half an SM, beside the data gradient's.
FcShape fc_weight_pair_shape(int K, int O, int B) {
  FcShape s;
  FcGemmParams& P = s.P;
  P.M = K; P.N = O;
  P.m_tiles = (K + kTileM - 1) / kTileM;
  P.n_pad = O <= 32 ? 32 : 64; P.acc_bufs = 2;
  P.n_tiles = (O + P.n_pad - 1) / P.n_pad;
  P.splits = 1;
  P.kblocks_total = P.kblocks_per_split = (B + kBlockK - 1) / kBlockK;
  P.a_mn = P.b_mn = 1;
  s.pair = true;
  return s;
}
long long fc_tiles(const FcShape& s) { return (long long)s.P.m_tiles * s.P.n_tiles * s.P.splits; }
// Whether both are faster in one launch.  With a slot for every tile always (272 layers of 8 to 128 images: by 25 - 50 %).  In more rounds not
// where the data gradient's tiles alone have an SM each and more than two k-blocks of images make the weight gradient's wider tiles
// worth while, unless those leave most of a second round empty: 4096 -> 512, 128 images, two launches 18.0 us, one 19.4; 2304 -> 1000 19.2
// and 20.8; 6272 -> 552 22.5 and 23.2; with 64 images 14.7 and 13.8, 15.3 and 14.3, 16.7 and 16.4 (the same layers), but 3136 -> 1000, eight k-blocks
// a tile of the data gradient, 17.7 and 18.4; 128 images, tiles that share SMs alone too: 6272 -> 512 23.2 and 20.6; 215 wide tiles: 5436 -> 400 21.9 and 19.9.
bool fc_pair_faster(int sms, const FcShape& w, const FcShape& d, const FcShape& w_alone) {
  const long long tw = fc_tiles(w), td = fc_tiles(d), alone = fc_tiles(w_alone), slots = 2ll * sms;
  if (!d.pair || !share_slots(slots, tw, td)) return false;
  const bool second_round_empty = alone > sms && 5 * alone < 8 * sms;
  return 20 * (tw + td) <= 21 * slots || td > sms || (w.P.kblocks_total <= 2 && d.P.kblocks_per_split < 8) || second_round_empty;
}

}  // namespace

struct cct_fc_plan {
  cct_ctx* ctx = nullptr;
  int B = 0, K = 0, O = 0, bias = 0;
  int K4 = 0, O4 = 0;        // row pitches: multiples of four floats
  FcShape fwd, dgr, wgr, wgr_pair;  // wgr_pair: the weight gradient's, beside the data gradient in one launch
  bool pair = false;         // both gradients in one launch, where the SMs that a call has can take their tiles
  bool dot = false, dot_narrow = false;  // forward pass by fc_dot_kernel: rows on 16-byte boundaries, and off them
  bool small_forward = false, small = false;  // else the forward pass, and the backward pass, by fc_small_kernel, with these splits (where an
  int small_fwd = 1, small_dgr = 1;           // operand is off a 16-byte boundary too, as far as there is room for their sums)
  float* partial = nullptr;  // split partial sums of the forward pass and of the data gradient
  float *Xp = nullptr, *Wp = nullptr, *dYp = nullptr;  // copies with padded rows, where K or O is no multiple of four
  size_t bytes = 0;
  FcMap w_fwd, x_fwd, w_dgr, dy_dgr, x_wgr, dy_wgr, out_fwd, out_dgr, out_wgr;
  PhaseTimer timer;
};

namespace {

int fc_launch(cct_ctx* ctx, const FcShape& s, const FcMap& a, const FcMap& b, const FcMap& out, float* direct = nullptr,
              long long ld_direct = 0) {
  FcGemmParams P = s.P;
  P.direct = direct; P.ld_direct = ld_direct;
  P.status = ctx->status_dev;
  const int tiles = P.m_tiles * P.n_tiles * P.splits;
  launch_pdl(fc_gemm_kernel, dim3(std::min(tiles, (s.pair ? 2 : 1) * ctx->launch_sms())), dim3(kFcThreads), s.smem, ctx->stream, P,
             a.map, b.map, out.map);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

// `blocks` of the grid are the weight gradient's.  Both jobs give up their share of SMs that a reduction in flight takes: with
// eight fewer 6272 -> 256, 128 images, has 186 blocks for 196 tiles and 94 for 98, not 196 and 84.
int fc_launch_two(cct_ctx* ctx, const cct_fc_plan* plan, int blocks, float* direct, long long ld_direct) {
  FcGemmParams W = plan->wgr_pair.P, D = plan->dgr.P;
  W.direct = direct; W.ld_direct = ld_direct;
  W.status = D.status = ctx->status_dev;
  const int behind = (int)std::min(fc_tiles(plan->dgr), std::max(1ll, 2ll * ctx->launch_sms() - blocks));
  const FcJob w{W, plan->x_wgr.map, plan->dy_wgr.map, (direct ? plan->x_wgr : plan->out_wgr).map};
  const FcJob d{D, plan->w_dgr.map, plan->dy_dgr.map, plan->out_dgr.map};
  launch_pdl(fc_gemm_two_kernel, dim3(blocks + behind), dim3(kFcThreads), std::max(plan->wgr_pair.smem, plan->dgr.smem), ctx->stream, w, d,
             (unsigned)blocks);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

// Flops count the tiles' padding, which is most of the work for a handful of images.
bool use_small_fc(int B, int K, int O) {
  const double flops = 2.0 * fc_round_up(B, kFsTile) * fc_round_up(K, kFsTile) * fc_round_up(O, kFsTile);
  return flops <= (K % 4 || O % 4 ? kSmallFcPaddedFlops : kSmallFcFlops);
}

unsigned fc_small_tiles(const FcSmallParams& P) { return (unsigned)((P.M + kFsTile - 1) / kFsTile) * ((P.N + kFsTile - 1) / kFsTile); }
int fc_small(cct_ctx* ctx, const FcSmallParams& P) {
  launch_pdl(fc_small_kernel, dim3(fc_small_tiles(P), P.splits), dim3(kFsThreads), 0, ctx->stream, P);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}
int fc_small_two(cct_ctx* ctx, const FcSmallParams& first, const FcSmallParams& second) {
  const unsigned blocks = fc_small_tiles(first) * first.splits;
  launch_pdl(fc_small_two_kernel, dim3(blocks + fc_small_tiles(second) * second.splits), dim3(kFsThreads), 0, ctx->stream,
             FcSmallJobs{{first, second}, blocks});
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

bool fc_aligned(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15u) return false;
  return true;
}

int fc_reduce(cct_ctx* ctx, FcReduceParams R) {
  const bool vec = R.cols % 4 == 0 && fc_aligned({R.partial, R.out});
  const long long threads = (long long)R.rows * (vec ? R.cols / 4 : R.cols);
  const bool slices = R.splits >= 8 && threads < 256ll * ctx->sm_count;
  auto pick = [&](auto bias) {
    constexpr bool kBias = decltype(bias)::value;
    return slices ? (vec ? fc_reduce_kernel<4, 8, kBias> : fc_reduce_kernel<1, 8, kBias>)
                  : (vec ? fc_reduce_kernel<4, 1, kBias> : fc_reduce_kernel<1, 1, kBias>);
  };
  auto kernel = R.bias_sum.db ? pick(std::true_type{}) : pick(std::false_type{});
  const long long per_block = slices ? 32 : 256;
  R.sum_blocks = (unsigned)((threads + per_block - 1) / per_block);
  launch_pdl(kernel, dim3(R.sum_blocks + (R.bias_sum.db ? (R.bias_sum.O + 31) / 32 : 0)), dim3(256), 0, ctx->stream, R);
  CCT_CHECK_LAUNCH(ctx);
  return CCT_OK;
}

// Forward pass of a small layer; `vec`: all rows on 16-byte boundaries.  Where Y lies over an operand that other blocks still read, the
// sums go through `scratch`.
int fc_dot(cct_ctx* ctx, bool vec, const float* W, const float* X, int K, FcReduceParams post, float* scratch) {
  FcDotParams P{W, X, post.cols, post.rows, K, post};
  const bool clear = apart(post.out, (size_t)post.rows * post.cols, {{X, (size_t)post.rows * K}, {W, (size_t)post.cols * K}});
  if (!clear) {
    P.post = FcReduceParams{};
    P.post.out = scratch;
    P.post.cols = post.cols;
    post.partial = scratch;
    post.pitch = post.cols;
    post.splits = 1;
  }
  const int steps = (K + (vec ? 127 : 31)) / (vec ? 128 : 32);
  const bool wide = vec && P.N >= 8 && (long long)((P.N + 7) / 8) * ((P.M + kFdM - 1) / kFdM) >= kDotWideBlocks;
  const int nt = wide ? 8 : P.N > 2 ? 4 : P.N;
  launch_pdl(vec ? fc_dot_pick<4>(nt) : fc_dot_pick<1>(nt), dim3((unsigned)((P.M + kFdM - 1) / kFdM) * ((P.N + nt - 1) / nt)),
             dim3(32 * std::min(steps, kFdMaxWarps)), 0, ctx->stream, P);
  CCT_CHECK_LAUNCH(ctx);
  return clear ? CCT_OK : fc_reduce(ctx, post);
}

void fc_pad(cct_ctx* ctx, const float* src, float* dst, int rows, int cols, int pitch) {
  launch_pdl(fc_pad_kernel, dim3(std::min((pitch + 255) / 256, 8), std::min(rows, 8 * ctx->sm_count)), dim3(256), 0, ctx->stream, src, dst,
             rows, cols, pitch);
}

}  // namespace

extern "C" {

int cct_fc_plan_create(cct_ctx* ctx, int batch, int in_features, int out_features, int bias_term, cct_fc_plan** out) {
  if (!ctx || !out) return CCT_ERR_INVALID;
  *out = nullptr;
  if (batch <= 0 || in_features <= 0 || out_features <= 0) return CCT_ERR_INVALID;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  cct_fc_plan* p = new (std::nothrow) cct_fc_plan();
  if (!p) return CCT_ERR_NOMEM;
  p->ctx = ctx; p->B = batch; p->K = in_features; p->O = out_features; p->bias = bias_term != 0;
  p->K4 = fc_round_up(in_features, 4); p->O4 = fc_round_up(out_features, 4);
  p->fwd = fc_batch_shape(ctx->sm_count, out_features, batch, in_features);
  p->dgr = fc_batch_shape(ctx->sm_count, in_features, batch, out_features);
  p->dgr.P.a_mn = 1;
  p->wgr = fc_weight_shape(ctx->sm_count, in_features, out_features, batch);
  if (!fc_fit_rings(p->fwd) || !fc_fit_rings(p->dgr) || !fc_fit_rings(p->wgr)) {
    ctx->last_error = "fully connected tile does not fit in shared memory twice";
    delete p;
    return CCT_ERR_UNSUPPORTED;
  }
  const bool few = use_small_fc(batch, in_features, out_features);
  p->small_forward = few;
  p->wgr_pair = fc_weight_pair_shape(in_features, out_features, batch);
  p->pair = fc_pair_faster(ctx->sm_count, p->wgr_pair, p->dgr, p->wgr) && fc_fit_rings(p->wgr_pair);
  p->small = few || fc_small_faster(ctx->sm_count, batch, in_features, out_features, p->pair);
  p->small_fwd = fc_small_splits(ctx->sm_count, out_features, batch, in_features);
  p->small_dgr = fc_small_splits(ctx->sm_count, in_features, batch, out_features);
  const bool one_launch = few && p->small_fwd == 1;
  p->dot = in_features % 4 == 0 && fc_dot_faster(batch, in_features, out_features, true, one_launch, false);
  p->dot_narrow = fc_dot_faster(batch, in_features, out_features, false, one_launch, !few && in_features % 4);
  // One allocation: split sums, then the padded copies that are needed.
  const int f_splits = few ? p->small_fwd : p->fwd.P.splits, d_splits = p->small ? p->small_dgr : p->dgr.P.splits;
  const size_t sums = std::max((size_t)f_splits * batch * p->O4, (size_t)d_splits * batch * p->K4);
  const bool pad_k = !((p->dot_narrow || few) && p->small) && p->K4 != p->K, pad_o = !p->small && p->O4 != p->O;
  auto room = [](size_t n) { return (n + 63) & ~(size_t)63; };
  const size_t x = pad_k ? room((size_t)batch * p->K4) : 0, w = pad_k ? room((size_t)out_features * p->K4) : 0,
               dy = pad_o ? room((size_t)batch * p->O4) : 0;
  p->bytes = (room(sums) + x + w + dy) * sizeof(float);
  if (cudaMalloc((void**)&p->partial, p->bytes) != cudaSuccess) {
    cudaGetLastError();
    ctx->last_error = "cudaMalloc of the fully connected layer's scratch failed";
    delete p;
    return CCT_ERR_NOMEM;
  }
  float* at = p->partial + room(sums);
  if (pad_k) { p->Xp = at; p->Wp = at + x; }
  if (pad_o) p->dYp = at + x + w;
  cudaError_t e = cudaFuncSetAttribute(fc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  if (e == cudaSuccess && p->pair && !p->small) e = cudaFuncSetAttribute(fc_gemm_two_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 113 * 1024);
  if (e != cudaSuccess) {
    ctx->last_error = std::string("cudaFuncSetAttribute(fc_gemm_kernel): ") + cudaGetErrorString(e);
    cudaFree(p->partial);
    delete p;
    return CCT_ERR_CUDA;
  }
  *out = p;
  return CCT_OK;
}

int cct_fc_plan_destroy(cct_fc_plan* plan) {
  if (!plan) return CCT_ERR_INVALID;
  cudaSetDevice(plan->ctx->device);
  cudaStreamSynchronize(plan->ctx->stream);
  cudaFree(plan->partial);
  plan->ctx->timed_plans -= plan->timer.enabled;
  for (cudaEvent_t e : plan->timer.ev)
    if (e) cudaEventDestroy(e);
  delete plan;
  return CCT_OK;
}

int cct_fc_plan_workspace_bytes(const cct_fc_plan* plan, size_t* bytes) {
  if (!plan || !bytes) return CCT_ERR_INVALID;
  *bytes = plan->bytes;
  return CCT_OK;
}

int cct_fc_forward(cct_fc_plan* plan, const float* X, const float* W, const float* bias, float* Y, int relu,
                   const uint32_t* drop_mask, float drop_scale) {
  if (plan) CCT_RECORD(plan->ctx, cct_fc_forward(plan, X, W, bias, Y, relu, drop_mask, drop_scale))
  if (!plan || !X || !W || !Y || (plan->bias && !bias)) return CCT_ERR_INVALID;
  cct_ctx* ctx = plan->ctx;
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  const int B = plan->B, K = plan->K, O = plan->O, K4 = plan->K4, O4 = plan->O4;
  plan->timer.begin(0, ctx->stream);
  const bool wide = K % 4 == 0 && fc_aligned({X, W});
  if (wide ? plan->dot : plan->dot_narrow) {
    const int rc = fc_dot(ctx, wide, W, X, K, FcReduceParams{nullptr, Y, plan->bias ? bias : nullptr, nullptr, drop_mask, drop_scale, B, O, O4, 1, relu},
                          plan->partial);
    plan->timer.end(0, ctx->stream);
    return rc;
  }
  if (plan->small_forward || !(plan->Wp || fc_aligned({X, W}))) {
    const int splits = plan->small_forward ? plan->small_fwd : std::min(plan->small_fwd, plan->fwd.P.splits);
    // through sums: splits, or an output over an operand that other blocks still read
    const bool sums = splits > 1 || !apart(Y, (size_t)B * O, {{X, (size_t)B * K}, {W, (size_t)O * K}});
    const FcReduceParams post{plan->partial, Y, plan->bias ? bias : nullptr, nullptr, drop_mask, drop_scale, B, O, O4, splits, relu};
    int rc = fc_small(ctx, FcSmallParams{W, X, K, K, 0, 0, O, B, K, splits, fc_round_up((K + splits - 1) / splits, 32),
                                         sums ? plan->partial : Y, sums ? O4 : O, nullptr, sums ? FcReduceParams{} : post});
    if (rc == CCT_OK && sums) rc = fc_reduce(ctx, post);
    plan->timer.end(0, ctx->stream);
    return rc;
  }
  if (plan->Wp) {
    fc_pad(ctx, X, plan->Xp, B, K, K4);
    fc_pad(ctx, W, plan->Wp, O, K, K4);
    X = plan->Xp;
    W = plan->Wp;
  }
  int rc = fc_operand_map(ctx, &plan->w_fwd, W, O, K, K4, kTileM, false);
  if (rc == CCT_OK) rc = fc_operand_map(ctx, &plan->x_fwd, X, B, K, K4, plan->fwd.P.n_pad, false);
  if (rc == CCT_OK) rc = fc_output_map(ctx, &plan->out_fwd, plan->partial, O, B, plan->fwd.P.splits, O4);
  if (rc == CCT_OK) rc = fc_launch(ctx, plan->fwd, plan->w_fwd, plan->x_fwd, plan->out_fwd);
  if (rc == CCT_OK)
    rc = fc_reduce(ctx, FcReduceParams{plan->partial, Y, plan->bias ? bias : nullptr, nullptr, drop_mask, drop_scale, B, O, O4,
                                       plan->fwd.P.splits, relu});
  plan->timer.end(0, ctx->stream);
  return rc;
}

int cct_fc_backward(cct_fc_plan* plan, const float* X, const float* W, const float* dY, float* dX, float* dW, float* db,
                    int in_relu, const uint32_t* in_drop_mask, float in_drop_scale) {
  if (plan) CCT_RECORD(plan->ctx, cct_fc_backward(plan, X, W, dY, dX, dW, db, in_relu, in_drop_mask, in_drop_scale))
  if (!plan || !X || !W || !dY || !dW || (plan->bias && !db)) return CCT_ERR_INVALID;
  cct_ctx* ctx = plan->ctx;
  if (*ctx->status_host != 0) return CCT_ERR_TIMEOUT;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  const int B = plan->B, K = plan->K, O = plan->O, K4 = plan->K4, O4 = plan->O4;
  const bool x_ok = plan->Xp || fc_aligned({X}), w_ok = plan->Wp || fc_aligned({W}), dy_ok = plan->dYp || fc_aligned({dY});
  const bool w_small = plan->small || !(x_ok && dy_ok), d_small = plan->small || !(w_ok && dy_ok);
  const float *Xm = X, *dYm = dY;
  FcBiasSum bias_sum{};
  int rc = CCT_OK;
  // ---- weight gradient: out = dW[o][k] (m = k, n = o), reduction over the batch; both operands MN-major
  plan->timer.begin(1, ctx->stream);
  if (plan->dYp && !(w_small && d_small)) { fc_pad(ctx, dY, plan->dYp, B, O, O4); dYm = plan->dYp; }
  const FcSmallParams W_job{X, dY, K, O, 1, 1, K, O, B, 1, B, dW, K, plan->bias ? db : nullptr, FcReduceParams{}};
  // Both contractions of a layer with few tiles in one launch, where neither writes what the other reads or writes.
  const size_t nx = (size_t)B * K, ny = (size_t)B * O, nw = (size_t)O * K, nb = plan->bias ? O : 0;
  const int d_splits = plan->small ? plan->small_dgr : std::min(plan->small_dgr, plan->dgr.P.splits);
  const bool d_sums = d_splits > 1 || !apart(dX, nx, {{dY, ny}, {W, nw}});  // as in the forward pass
  const bool clear = dX && !plan->timer.enabled && apart(dX, nx, {{X, nx}, {dY, ny}, {dW, nw}, {db, nb}}) &&
                     apart(dW, nw, {{W, nw}, {dY, ny}, {X, nx}, {in_drop_mask, nx}}) && apart(db, nb, {{W, nw}, {dY, ny}, {X, nx}, {in_drop_mask, nx}});
  const bool together = clear && w_small && d_small;
  const int two = clear && plan->pair && !w_small && !d_small ? share_slots(2ll * ctx->launch_sms(), fc_tiles(plan->wgr_pair), fc_tiles(plan->dgr)) : 0;
  const bool direct = K4 != K || !fc_aligned({dW});  // dW: an output no tensor map describes
  if (w_small) {
    if (!together) rc = fc_small(ctx, W_job);
    if (rc != CCT_OK) return rc;
  } else {
    if (plan->Xp) { fc_pad(ctx, X, plan->Xp, B, K, K4); Xm = plan->Xp; }
    rc = fc_operand_map(ctx, &plan->x_wgr, Xm, B, K, K4, 32, true);
    if (rc == CCT_OK) rc = fc_operand_map(ctx, &plan->dy_wgr, dYm, B, O, O4, 32, true);
    if (rc == CCT_OK && !direct) rc = fc_output_map(ctx, &plan->out_wgr, dW, K, O, 1, K);
    if (rc == CCT_OK && !two)
      rc = fc_launch(ctx, plan->wgr, plan->x_wgr, plan->dy_wgr, direct ? plan->x_wgr : plan->out_wgr, direct ? dW : nullptr, K);
    if (rc != CCT_OK) return rc;
    if (plan->bias) {
      // With the data gradient's reduction, unless there is none, or it writes where the sum reads (dX over dY).
      bias_sum = FcBiasSum{dY, db, B, O};
      if (!dX || (d_small && !d_sums) || !apart(dX, nx, {{dY, ny}})) {
        launch_pdl(fc_bias_grad_kernel, dim3((O + 31) / 32), dim3(256), 0, ctx->stream, bias_sum);
        bias_sum = FcBiasSum{};
      }
    }
  }
  plan->timer.end(1, ctx->stream);
  CCT_CHECK_LAUNCH(ctx);
  // ---- data gradient: out = dX[b][k] (m = k, n = b), reduction over o; A = W read MN-major, B = dY K-major
  if (dX && d_small) {
    plan->timer.begin(3, ctx->stream);
    const FcReduceParams post{plan->partial, dX, nullptr, in_relu ? X : nullptr, in_drop_mask, in_drop_scale, B, K, K4, d_splits, 0, 0, bias_sum};
    const FcSmallParams D_job{W, dY, K, O, 1, 0, K, B, O, d_splits, fc_round_up((O + d_splits - 1) / d_splits, 32),
                              d_sums ? plan->partial : dX, d_sums ? K4 : K, nullptr, d_sums ? FcReduceParams{} : post};
    rc = together ? fc_small_two(ctx, W_job, D_job) : fc_small(ctx, D_job);
    if (rc == CCT_OK && d_sums) rc = fc_reduce(ctx, post);
    plan->timer.end(3, ctx->stream);
  } else if (dX) {
    plan->timer.begin(3, ctx->stream);
    if (plan->Wp) { fc_pad(ctx, W, plan->Wp, O, K, K4); W = plan->Wp; }
    rc = fc_operand_map(ctx, &plan->w_dgr, W, O, K, K4, 32, true);
    if (rc == CCT_OK) rc = fc_operand_map(ctx, &plan->dy_dgr, dYm, B, O, O4, plan->dgr.P.n_pad, false);
    if (rc == CCT_OK) rc = fc_output_map(ctx, &plan->out_dgr, plan->partial, K, B, plan->dgr.P.splits, K4);
    if (rc == CCT_OK) rc = two ? fc_launch_two(ctx, plan, two, direct ? dW : nullptr, K) : fc_launch(ctx, plan->dgr, plan->w_dgr, plan->dy_dgr, plan->out_dgr);
    if (rc == CCT_OK)
      rc = fc_reduce(ctx, FcReduceParams{plan->partial, dX, nullptr, in_relu ? X : nullptr, in_drop_mask, in_drop_scale, B, K, K4,
                                         plan->dgr.P.splits, 0, 0, bias_sum});
    plan->timer.end(3, ctx->stream);
  }
  return rc;
}

int cct_fc_plan_enable_timing(cct_fc_plan* plan, int enable) {
  if (!plan) return CCT_ERR_INVALID;
  cct_ctx* ctx = plan->ctx;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  PhaseTimer& t = plan->timer;
  if (enable && !t.ev[0])
    for (cudaEvent_t& e : t.ev) CCT_CUDA(ctx, cudaEventCreate(&e));
  ctx->timed_plans += (enable != 0) - t.enabled;
  t.enabled = enable != 0;
  for (bool& h : t.have) h = false;
  return CCT_OK;
}

int cct_fc_plan_last_timings(cct_fc_plan* plan, float ms[5]) {
  if (!plan || !ms) return CCT_ERR_INVALID;
  cct_ctx* ctx = plan->ctx;
  CCT_CUDA(ctx, cudaSetDevice(ctx->device));
  CCT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int i = 0; i < PhaseTimer::kSlots; ++i) {
    ms[i] = 0.f;
    if (plan->timer.have[i]) CCT_CUDA(ctx, cudaEventElapsedTime(&ms[i], plan->timer.ev[2 * i], plan->timer.ev[2 * i + 1]));
  }
  return CCT_OK;
}

}  // extern "C"
