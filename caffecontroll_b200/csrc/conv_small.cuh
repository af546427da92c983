// Small convolutions in fp32 FMA arithmetic, part of conv_umma.cu (the plan's tables and parameter blocks are shared).
//
// A tensor-core contraction costs about six microseconds before its first k-block is through (weights packed by a kernel of
// their own, tensor-memory allocation, the hand-overs between its roles) and half a microsecond for every further k-block
// of a tile; a layer of a few ten million multiply-adds - LeNet's first layers, a narrow data gradient - is all latency
// there.  These kernels do such a layer in one launch of short blocks: exact fp32 products, fp32 accumulation in a fixed
// order, no packed operand.  use_small_conv() / use_small_wgrad() draw the line.
#pragma once

namespace {

// ------------------------------------------------------------------------------- forward and data gradient
// Direct convolution, window and stride fixed at compile time; the data gradient of a stride-1 layer is the same thing over
// dY with the window turned round and the channel roles exchanged.  A lane owns one column of the output and JR consecutive
// rows of it, for CT output channels: per input channel and window column it loads (JR - 1) S + K values (lanes along the
// row: coalesced, from L1) and uses each for up to min(K, JR) x CT products, with the weights as shared-memory broadcasts
// ([channel][window column][window row][CT]).  With enough input channels the block's warps share the same 32 positions and
// split the input channels, so that even one image of a few hundred pixels spreads over the GPU (a warp's first touch of a
// channel is an L2 round trip: the fewer channels it walks, the shorter the chain); their sums are added in order through
// shared memory.

struct SmallConv {
  const float* in;
  const float* W;
  const float* bias;  // per output channel, or null
  float* out;
  int batch, n_in, n_out, pad;      // input / output plane sizes; pad as seen by this pass
  int ci, co, groups;               // input / output channels per group
  int dgrad;                        // weights: 0 = W[co][ci][kr][kc], 1 = W[ci][co][K-1-kr][K-1-kc]
  int relu;
  int positions, row_groups;        // batch * row_groups * n_out lanes
  int col_tiles;                    // channel tiles of CT per group
  int share;                        // 1: the block's warps split the input channels of the same 32 positions
  static constexpr int kThreads = 512;  // at most
  __host__ __device__ static constexpr int blocks(int) { return 0; }  // per SM at the least: not said (with 1 the compiler takes twice the registers)
};

// Rows per lane (row and column masks share 32 bits).  One channel leaves registers for kSmallTall, with which 3 values of a 5 x 5 window are
// loaded for 2 outputs where four load 2 for 1 (LeNet conv1, both passes, with four: 20.0 us, not 19.3; a 3 x 3 window gains no such
// thing: 44 images 32 x 32, two groups 6.0 us with four, 6.5 with eight).  Taken where four rows are more than one lot of 32 lanes for every
// SM and eight leave as many, or hardly a row behind the plane's last one: backward passes, four rows and eight: one image 28 x 28, 20
// channels 6.5 us and 7.9; 128 images 12 x 12, 32 channels 10.8 and 12.1 (144 lots of four); 16 images 40 x 40, 32 channels 17.5 and 15.3 (200,
// 100 of eight); 64 images 32 x 32, 32 channels 25.4 and 23.5 (512, 256); 64 images 28 x 28, 32 channels, four rows too many 19.9 and 20.4, though not
// beside a weight gradient (20 channels 17.4 and 14.7).
__host__ __device__ constexpr int small_rows(int K) { return K >= 11 ? 2 : 4; }
constexpr int kSmallTall = 8;
// Shared memory: the weights, afterwards the warps' sums.
inline size_t small_conv_smem(int K, int rows, int ct, int ci, int sharing_warps) {
  return std::max((size_t)ci * K * K * ct, (size_t)sharing_warps * rows * ct * 32) * sizeof(float);
}

// JOB: SmallConv, the pass alone, whose grid's x is positions and y channel tiles; or SmallBackward below, both gradients of a layer.  The
// pass's text stands in the kernel: as a function called from two kernels 6 images 16 x 16, 3 -> 8 channels 5 x 5 by 2 took 6.5 us, not 6.0.
template <int K, int S, int CT, typename JOB, int JR = small_rows(K)>
__global__ void __launch_bounds__(JOB::kThreads, JOB::blocks(CT)) small_conv_kernel(const __grid_constant__ JOB J) {
  pdl_wait();
  constexpr bool ALONE = std::is_same<JOB, SmallConv>::value;
  int bx = 0, by = 0;
  if constexpr (!ALONE) {
    if (J.weight_gradient()) return;
    bx = (int)blockIdx.x - J.conv_at; by = bx / J.grid_x, bx -= by * J.grid_x;
  }
  const SmallConv& P = J;
  constexpr int R = (JR - 1) * S + K;
  static_assert(R + K <= 32, "row and column bits share a word");
  extern __shared__ __align__(16) float small_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = (ALONE ? blockIdx.y : by) / P.col_tiles, c0 = ((ALONE ? blockIdx.y : by) - grp * P.col_tiles) * CT;
  const int nwarps = blockDim.x >> 5;
  // weights of this block's channels; consecutive threads read consecutive elements of a channel's window
  for (int e = tid; e < P.ci * K * K; e += blockDim.x) {
    const int d = e / (K * K), kr = (e / K) % K, kc = e % K;
    float wv[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) {
      const size_t at = P.dgrad ? (size_t)(grp * P.ci + d) * P.co + c0 + c : (size_t)(grp * P.co + c0 + c) * P.ci + d;
      wv[c] = c0 + c < P.co ? __ldg(P.W + at * (K * K) + kr * K + kc) : 0.f;
    }
    const int ur = P.dgrad ? K - 1 - kr : kr, uc = P.dgrad ? K - 1 - kc : kc;
#pragma unroll
    for (int c = 0; c < CT; ++c) small_smem[((d * K + uc) * K + ur) * CT + c] = wv[c];
  }
  // where this lane works: image, first row, column
  const int want = P.share ? (ALONE ? blockIdx.x : bx) * 32 + lane : (ALONE ? blockIdx.x : bx) * blockDim.x + tid;
  const int pos = min(want, P.positions - 1);
  const int bg = pos / P.n_out, x = pos - bg * P.n_out;
  const int b = bg / P.row_groups, y0 = (bg - b * P.row_groups) * JR;
  const int iy0 = y0 * S - P.pad, ix0 = x * S - P.pad;
  const int plane = P.n_in * P.n_in;
  uint32_t mask = 0;  // bit r: input row iy0 + r exists; bit R + kc: input column ix0 + kc exists
#pragma unroll
  for (int r = 0; r < R; ++r) mask |= (unsigned)(iy0 + r) < (unsigned)P.n_in ? 1u << r : 0u;
#pragma unroll
  for (int c = 0; c < K; ++c) mask |= (unsigned)(ix0 + c) < (unsigned)P.n_in ? 1u << (R + c) : 0u;
  const int d0 = P.share ? P.ci * warp / nwarps : 0, d1 = P.share ? P.ci * (warp + 1) / nwarps : P.ci;
  const float* src = P.in + ((long long)b * P.groups + grp) * P.ci * plane + (long long)d0 * plane + (long long)iy0 * P.n_in + ix0;
  float acc[JR][CT];
#pragma unroll
  for (int j = 0; j < JR; ++j)
#pragma unroll
    for (int c = 0; c < CT; ++c) acc[j][c] = 0.f;
  __syncthreads();
  const float* w = small_smem + (size_t)d0 * K * K * CT;
  auto fetch = [&](const float* p, int kc, float* dst) {
#pragma unroll
    for (int r = 0; r < R; ++r) dst[r] = ldg_if_bits(p + r * P.n_in + kc, mask, (1u << r) | (1u << (R + kc)));
  };
  auto use = [&](const float* x_col) {
#pragma unroll
    for (int kr = 0; kr < K; ++kr)
#pragma unroll
      for (int c = 0; c < CT; ++c)
#pragma unroll
        for (int j = 0; j < JR; ++j) acc[j][c] = fmaf(x_col[j * S + kr], w[kr * CT + c], acc[j][c]);
    w += K * CT;
  };
  if (K <= 5) {
    // the next window column's values (of this channel or the next) are in flight while the current one's are used
    float v[2][R];
    if (d0 < d1) fetch(src, 0, v[0]);
    for (int d = d0; d < d1; d += 2) {  // two channels a step: K is odd, so the buffers end where they began
#pragma unroll
      for (int i = 0; i < 2 * K; ++i) {
        const int kc = i % K, at = i / K;
        if (at == 1 && d + 1 >= d1) break;
        const bool last = kc == K - 1;
        if (!last) fetch(src + at * plane, kc + 1, v[(i + 1) & 1]);
        else if (d + at + 1 < d1) fetch(src + (at + 1) * plane, 0, v[(i + 1) & 1]);
        use(v[i & 1]);
      }
      src += 2 * plane;
    }
  } else {  // windows of 7 and 11 columns: few channels, many columns - other warps cover the loads
    for (int d = d0; d < d1; ++d, src += plane)
#pragma unroll
      for (int kc = 0; kc < K; ++kc) {
        float v[R];
        fetch(src, kc, v);
        use(v);
      }
  }
  const int live = want < P.positions ? min(CT, P.co - c0) : 0;
  const int oplane = P.n_out * P.n_out, ch0 = grp * P.co + c0;
  float* op = P.out + ((long long)b * P.groups * P.co + ch0) * oplane + (long long)y0 * P.n_out + x;
  auto finish = [&](float y, int j, int c) {
    if (c < live && y0 + j < P.n_out) {
      if (P.bias) y += __ldg(P.bias + ch0 + c);
      if (P.relu) y = fmaxf(y, 0.f);
      op[(long long)c * oplane + j * P.n_out] = y;
    }
  };
  if (!P.share) {
#pragma unroll
    for (int c = 0; c < CT; ++c)
#pragma unroll
      for (int j = 0; j < JR; ++j) finish(acc[j][c], j, c);
    return;
  }
  __syncthreads();  // the weights have been read
#pragma unroll
  for (int j = 0; j < JR; ++j)
#pragma unroll
    for (int c = 0; c < CT; ++c) small_smem[((warp * JR + j) * CT + c) * 32 + lane] = acc[j][c];
  __syncthreads();
  for (int i = warp; i < JR * CT; i += nwarps) {
    float y = 0.f;
    for (int q = 0; q < nwarps; ++q) y += small_smem[(q * JR * CT + i) * 32 + lane];
    finish(y, i / CT, i % CT);
  }
}

typedef void (*SmallConvKernel)(const SmallConv);
template <int CT>
SmallConvKernel small_conv_pick_ks(int k, int s) {
  switch (k * 10 + s) {
    case 11: return small_conv_kernel<1, 1, CT, SmallConv>;
    case 31: return small_conv_kernel<3, 1, CT, SmallConv>;   case 32: return small_conv_kernel<3, 2, CT, SmallConv>;
    case 51: return small_conv_kernel<5, 1, CT, SmallConv>;   case 52: return small_conv_kernel<5, 2, CT, SmallConv>;
    case 71: return small_conv_kernel<7, 1, CT, SmallConv>;   case 72: return small_conv_kernel<7, 2, CT, SmallConv>;
    case 114: return small_conv_kernel<11, 4, CT, SmallConv>;
  }
  return nullptr;
}
SmallConvKernel small_conv_pick(int k, int s, int ct, int rows = 0) {
  if (rows == kSmallTall) return small_conv_kernel<5, 1, 1, SmallConv, kSmallTall>;
  return ct == 8 ? small_conv_pick_ks<8>(k, s) : ct == 4 ? small_conv_pick_ks<4>(k, s) : small_conv_pick_ks<1>(k, s);
}
// Output channels per block: the fewest idle ones, eight where four would leave as many idle.
inline int small_conv_ct(int co) { return co == 1 ? 1 : (co + 7) / 8 * 8 - co <= (co + 3) / 4 * 4 - co ? 8 : 4; }

// ------------------------------------------------------------------------------------------ weight gradient
// dW[kk][channel] (+ the bias row) = sum over pixels of Lowered(X)[pixel][kk] * dY[pixel][channel]: a block owns 32 lowered
// rows x 32 channels and a range of pixels, brought to shared memory 128 pixels at a time ([pixel][row], rows of 36 floats:
// a thread stores four rows of its pixel as 16 bytes, conflict free, and the global loads run along the pixels).  Each of
// the eight warps takes every eighth pixel, 4 x 8 products per lane; the warps' sums are added in order at the end.
constexpr int kSwThreads = 256, kSwWarps = 8, kSwTile = 32, kSwPix = 128, kSwPitch = 36;

struct SmallWgrad {
  WgradParams w;
  int rows_pad, row_tiles, col_tiles, pix_per_split;
  int tiles;  // row tiles x channel tiles x groups
};
constexpr size_t kSwSmem = 2 * kSwPix * kSwPitch * sizeof(float) + kSwTile * sizeof(MaskTap);

__device__ __forceinline__ void small_wgrad_block(const SmallWgrad& J, float* s_ab, int tile, int split) {
  const WgradParams& P = J.w;
  const int rows_pad = J.rows_pad, row_tiles = J.row_tiles, col_tiles = J.col_tiles, pix_per_split = J.pix_per_split;
  MaskTap* s_taps = reinterpret_cast<MaskTap*>(s_ab + 2 * kSwPix * kSwPitch);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rt = tile % row_tiles, rest = tile / row_tiles;
  const int ct = rest % col_tiles, vg = rest / col_tiles;
  const int grp = vg / P.tiles_per_group, ntile = vg - grp * P.tiles_per_group;
  const int pix0 = split * pix_per_split, pix1 = min(P.n_pix, pix0 + pix_per_split);
  if (tid < kSwTile) {
    const int r = rt * kSwTile + tid;
    s_taps[tid] = r <= P.ones_row ? P.taps[r] : MaskTap{0, kWgPadBit};
  }
  float* s_a = s_ab;
  float* s_b = s_ab + kSwPix * kSwPitch;
  const float* xg = P.x + (long long)grp * P.x_group_stride;
  const float* dyg = P.dy + (long long)(grp * P.dy_group_channels + ntile * P.n_real + ct * kSwTile) * P.mm;
  const int live = min(kSwTile, min(P.n_real, P.dy_group_channels - ntile * P.n_real) - ct * kSwTile);
  const int ones = P.ones_row - rt * kSwTile;
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  const int ty = lane >> 2, tx = lane & 3;
  const int p = tid & (kSwPix - 1), half = tid >> 7;  // staging: pixel of the chunk, half of the row / channel quads
  for (int c0 = pix0; c0 < pix1; c0 += kSwPix) {
    __syncthreads();  // the taps are there / the previous chunk has been read
    {
      const int pix = c0 + p;
      const bool ok = pix < pix1;
      const int pb = pix / P.mm, pin = pix - pb * P.mm, pr = pin / P.m, pc = pin - pr * P.m;
      const int iy0 = pr * P.s - P.p, ix0 = pc * P.s - P.p;
      const float* xsrc = xg + (long long)pb * P.x_batch_stride + (long long)iy0 * P.n + ix0;
      const float* dsrc = dyg + (long long)pb * P.dy_batch_stride + pin;
      const uint32_t mask =
          ok ? (kWgValidBit | bit_range(-iy0, min(P.k, P.n - iy0)) | (bit_range(-ix0, min(P.k, P.n - ix0)) << 16)) : 0u;
      float va[4][4], vb[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = (half * 4 + q) * 4 + e;
          va[q][e] = ldg_if_bits(xsrc + s_taps[r].off, mask, s_taps[r].bits);
          vb[q][e] = ldg_if(dsrc + r * P.mm, (ok && r < live) ? 1u : 0u);
          if (r == ones) va[q][e] = ok ? 1.f : 0.f;
        }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int at = p * kSwPitch + (half * 4 + q) * 4;
        *reinterpret_cast<float4*>(s_a + at) = make_float4(va[q][0], va[q][1], va[q][2], va[q][3]);
        *reinterpret_cast<float4*>(s_b + at) = make_float4(vb[q][0], vb[q][1], vb[q][2], vb[q][3]);
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int i = 0; i < kSwPix / kSwWarps; ++i) {
      const int at = (i * kSwWarps + warp) * kSwPitch;
      const float4 a = *reinterpret_cast<const float4*>(s_a + at + 4 * ty);
      const float4 b0 = *reinterpret_cast<const float4*>(s_b + at + 8 * tx), b1 = *reinterpret_cast<const float4*>(s_b + at + 8 * tx + 4);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) s_ab[warp * kSwTile * kSwTile + (4 * ty + u) * kSwTile + 8 * tx + v] = acc[u][v];
  __syncthreads();
  float* out = P.partial + (((size_t)split * J.tiles / (row_tiles * col_tiles) + vg) * rows_pad + rt * kSwTile) * P.n_pad + ct * kSwTile;
  for (int i = tid; i < kSwTile * kSwTile; i += kSwThreads) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kSwWarps; ++w) t += s_ab[w * kSwTile * kSwTile + i];
    out[(size_t)(i / kSwTile) * P.n_pad + (i & (kSwTile - 1))] = t;
  }
}

__global__ void __launch_bounds__(kSwThreads) small_wgrad_kernel(const __grid_constant__ SmallWgrad J) {
  pdl_wait();
  extern __shared__ __align__(16) float small_smem[];
  small_wgrad_block(J, small_smem, blockIdx.x % J.tiles, blockIdx.x / J.tiles);
}

// Both gradients of a layer with stride 1 in one launch: neither reads what the other writes.  LeNet conv1 at batch 64, forward and
// backward: 22.2 -> 19.3 us, three launches instead of four (three blocks per SM for one-channel data gradients, at 80 registers and
// 136 bytes of spills in tall lanes; with two blocks 19.6, with four 20.4).  The weight gradient's blocks go first, since a few of them behind the others are a round of their own (44 images 18 x 18, 7 -> 16
// channels 1 x 1: two launches 9.1 us, the data gradient first 10.5, the weight gradient first 8.1; 32 images 24 x 24, 4 -> 12 channels 3 x 3
// 12.4, 12.8 and 11.0) - unless the data gradient's are the longer ones: three and more channels a warp against one chunk of pixels, in one
// round or with one channel (LeNet conv1's backward pass 14.9 us, the weight gradient first 15.7; 8 images 18 x 18, 7 -> 23 channels 5 x 5 10.2 and 11.6;
// in more rounds 46 x 46, 44 -> 28 channels 3 x 3 12.9 and 11.2), or tall lanes in more than a round (64 images 32 x 32, 12 channels, padding 2 16.5
// and 17.9).  Up to kSmallRounds rounds of blocks: 21 images 18 x 18, 42 -> 24 channels 1 x 1 4.5
// + 5.4 -> 11.7 us (2.6 rounds).  Not where the data gradient alone has more warps per block than go here: 3 images 9 x 9, 3 -> 259
// channels 3 x 3 4.5 + 17.3 -> 23.8.  Nor tall lanes with fewer than kSmallTallChannels in more than a round, which the pass alone shares
// between four warps, not eight (64 images 32 x 32, eight channels, padding 2: 16.1 -> 17.1).
constexpr int kSmallRounds = 2, kSmallTallChannels = 12;
struct SmallBackward : SmallConv {  // the base: the data gradient
  SmallWgrad w;
  int grid_x, conv_at;         // of the data gradient: its grid, and its first block
  int wgrad_at, wgrad_blocks;
  static constexpr int kThreads = kSwThreads;
  __host__ __device__ static constexpr int blocks(int ct) { return ct == 1 ? 3 : 2; }  // per SM
  __device__ bool weight_gradient() const {
    extern __shared__ __align__(16) float small_smem[];
    const unsigned block = blockIdx.x - (unsigned)wgrad_at;
    if (block < (unsigned)wgrad_blocks) small_wgrad_block(w, small_smem, (int)block % w.tiles, (int)block / w.tiles);
    return block < (unsigned)wgrad_blocks;
  }
};
typedef void (*SmallBackwardKernel)(const SmallBackward);
template <int CT>
SmallBackwardKernel small_backward_pick_k(int k) {
  return k == 1   ? small_conv_kernel<1, 1, CT, SmallBackward>
         : k == 3 ? small_conv_kernel<3, 1, CT, SmallBackward>
         : k == 5 ? small_conv_kernel<5, 1, CT, SmallBackward>
                  : small_conv_kernel<7, 1, CT, SmallBackward>;
}
SmallBackwardKernel small_backward_pick(int k, int ct, int rows) {
  if (rows == kSmallTall) return small_conv_kernel<5, 1, 1, SmallBackward, kSmallTall>;
  return ct == 8 ? small_backward_pick_k<8>(k) : ct == 4 ? small_backward_pick_k<4>(k) : small_backward_pick_k<1>(k);
}

}  // namespace
