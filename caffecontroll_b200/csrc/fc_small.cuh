// Small inner products in fp32 FMA arithmetic, part of fc_umma.cu.
//
// A tensor-core contraction of fc_gemm_kernel takes five to six microseconds however small it is; LeNet's inner products
// (51 and 0.6 MFLOP) are nothing but that.  One kernel serves the three contractions out[n][m] = sum_r A(m, r) B(n, r): a
// block owns a 32 x 32 tile of the output and a range of the reduction, brought to shared memory 128 indices at a time as
// [r][32 m] and [r][32 n] (rows of 36 floats: 16-byte stores, conflict free); each of its eight warps takes every eighth
// index, 4 x 8 products per lane, and the warps' sums are added in order.  Without splits the block applies what surrounds
// the contraction itself (bias, ReLU, dropout; the masks of the bridges in front); the weight gradient's blocks of the first
// row of tiles sum the bias gradient on the way.  What bounds these layers is the number of launches (1.5 us each at the least,
// and as long for the host), so both contractions of a backward pass are one, and forward passes have fc_dot_kernel: 4096 -> 10,
// 50 images, both ways 13.4 -> 8.9 us.  Three blocks per SM (80 registers): the backward launch took 7.0 us with two, whose 384
// blocks were two waves, and 6.6 with four; the two launches 3.6 + 4.5.
#pragma once

namespace {

constexpr int kFsThreads = 256, kFsWarps = 8, kFsTile = 32, kFsChunk = 128, kFsPitch = 36;
// Measured against fc_gemm_kernel, forward + backward: 4096 -> 10, 50 images (17 MFLOP with the padding to 32) 23 -> 14 us;
// 512 -> 128, 128 images (17) 24 -> 15; 800 -> 500, 64 images (52) 22 -> 26.  Where feature counts are no multiples of four
// the other path copies its operands first: 999 -> 333, 37 images (46) 42 -> 23.
constexpr double kSmallFcFlops = 4e7, kSmallFcPaddedFlops = 1e8;

struct FcSmallParams {
  const float *a, *b;
  long long a_ld, b_ld;  // elements between rows: K-major: row = m (n), MN-major: row = r
  int a_mn, b_mn;
  int M, N, R, splits, r_per_split;
  float* out;            // splits > 1: [split][N][ld] raw sums; else the output itself
  long long ld;
  float* db;             // weight gradient: column sums of B
  FcReduceParams post;   // splits == 1: bias / ReLU / dropout / masks; `out` and the sizes are not used
};
struct FcSmallJobs {
  FcSmallParams job[2];
  unsigned first;  // blocks [0, first) do job 0, those behind them job 1
};

// 32 rows x 128 reduction indices of one operand into dst[r][kFsPitch].
__device__ __forceinline__ void fs_stage(float* dst, const float* src, long long ld, int mn, int row0, int rows, int r0, int r1, int tid) {
  float v[4][4];
  if (!mn) {  // lanes along the reduction
    const int r = tid & (kFsChunk - 1), half = tid >> 7;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + (half * 4 + q) * 4 + e;
        v[q][e] = (row < rows && r0 + r < r1) ? __ldg(src + (long long)row * ld + r0 + r) : 0.f;
      }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<float4*>(dst + r * kFsPitch + (half * 4 + q) * 4) = make_float4(v[q][0], v[q][1], v[q][2], v[q][3]);
  } else {  // lanes along the rows
    const int quad = (tid & 7) * 4, rr = tid >> 3;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = r0 + rr + 32 * q, row = row0 + quad + e;
        v[q][e] = (row < rows && r < r1) ? __ldg(src + (long long)r * ld + row) : 0.f;
      }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<float4*>(dst + (rr + 32 * q) * kFsPitch + quad) = make_float4(v[q][0], v[q][1], v[q][2], v[q][3]);
  }
}

__global__ void __launch_bounds__(kFsThreads, 3) fc_small_kernel(const __grid_constant__ FcSmallJobs J) {
  pdl_wait();
  const bool second = blockIdx.x >= J.first;
  const FcSmallParams& P = J.job[second];
  const unsigned block = blockIdx.x - (second ? J.first : 0u);
  __shared__ __align__(16) float s_ab[2 * kFsChunk * kFsPitch];
  __shared__ float s_db[kFsWarps][kFsTile];
  float *s_a = s_ab, *s_b = s_ab + kFsChunk * kFsPitch;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = lane >> 2, tx = lane & 3;
  const int m_tiles = (P.M + kFsTile - 1) / kFsTile, split = (int)(block % (unsigned)P.splits), tile = (int)(block / (unsigned)P.splits);
  const int n_tile = tile / m_tiles, m0 = (tile - n_tile * m_tiles) * kFsTile, n0 = n_tile * kFsTile;
  const int r_begin = split * P.r_per_split, r_end = min(P.R, r_begin + P.r_per_split);
  const bool sum_b = P.db != nullptr && m0 == 0;
  float acc[4][8], db = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[u][v] = 0.f;
  for (int r0 = r_begin; r0 < r_end; r0 += kFsChunk) {
    if (r0 != r_begin) __syncthreads();  // the previous chunk has been read
    fs_stage(s_a, P.a, P.a_ld, P.a_mn, m0, P.M, r0, r_end, tid);
    fs_stage(s_b, P.b, P.b_ld, P.b_mn, n0, P.N, r0, r_end, tid);
    __syncthreads();
    const int steps = (min(kFsChunk, r_end - r0) + kFsWarps - 1) / kFsWarps;
#pragma unroll 4
    for (int i = 0; i < steps; ++i) {
      const int at = (i * kFsWarps + warp) * kFsPitch;
      const float4 a = *reinterpret_cast<const float4*>(s_a + at + 4 * ty);
      const float4 b0 = *reinterpret_cast<const float4*>(s_b + at + 8 * tx), b1 = *reinterpret_cast<const float4*>(s_b + at + 8 * tx + 4);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
      if (sum_b) db += s_b[at + lane];
    }
  }
  __syncthreads();
  // [warp][n][m]; rows of 32 floats
#pragma unroll
  for (int v = 0; v < 8; ++v)
    *reinterpret_cast<float4*>(s_ab + warp * kFsTile * kFsTile + (8 * tx + v) * kFsTile + 4 * ty) =
        make_float4(acc[0][v], acc[1][v], acc[2][v], acc[3][v]);
  if (sum_b) s_db[warp][lane] = db;
  __syncthreads();
  const FcReduceParams& F = P.post;
#pragma unroll
  for (int k = 0; k < kFsTile * kFsTile / kFsThreads; ++k) {
    const int i = tid + k * kFsThreads, n = n0 + i / kFsTile, m = m0 + (i & (kFsTile - 1));
    if (n >= P.N || m >= P.M) continue;
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kFsWarps; ++w) t += s_ab[w * kFsTile * kFsTile + i];
    if (P.splits > 1) {
      P.out[((long long)split * P.N + n) * P.ld + m] = t;
      continue;
    }
    const long long at = (long long)n * P.ld + m;
    if (F.bias) t += __ldg(F.bias + m);
    if (F.relu) t = fmaxf(t, 0.f);
    if (F.drop_mask) t = t * (float)(F.drop_mask[at] != 0u) * F.drop_scale;
    if (F.X) t = t * (F.X[at] > 0.f ? 1.f : 0.f);
    P.out[at] = t;
  }
  if (sum_b && tid < kFsTile && n0 + tid < P.N) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kFsWarps; ++w) t += s_db[w][tid];
    P.db[n0 + tid] = t;
  }
}

// Forward pass of a small layer: out[n][m] = sum_r A[m][r] B[n][r], rows along the reduction.  A block owns 4 images x 4 outputs,
// its warps interleaved steps of 32 (x 4 where rows are on 16-byte boundaries) reduction indices; operands go from L2 straight
// to registers, eight loads for sixteen products per lane and index, a warp's sums are added by shuffles and the warps' in
// order.  With the 32 x 32 tiles of fc_small_kernel a few outputs with a long reduction took 32 splits, and a launch to add
// them; with the splits in a cluster, adding through distributed shared memory, 512 indices per block took longer than that
// launch.  4096 -> 10, 50 images: 4.4 + 2.7 -> 3.4 us, 500 -> 10, 64 images: 6.3 + 2.4 -> 2.3.  Traffic is a quarter of a word per product: layers that are not small have other kernels.
constexpr int kFdTile = 4, kFdMaxWarps = 16;
struct FcDotParams {
  const float *a, *b;
  int M, N, R;
  FcReduceParams post;  // out, ld = cols; bias / ReLU / dropout
};
template <int VEC>
__global__ void __launch_bounds__(32 * kFdMaxWarps) fc_dot_kernel(const __grid_constant__ FcDotParams P) {
  pdl_wait();
  __shared__ float s_part[kFdMaxWarps][kFdTile * kFdTile];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  const int m_tiles = (P.M + kFdTile - 1) / kFdTile, n_tile = blockIdx.x / m_tiles;
  const int m0 = (blockIdx.x - n_tile * m_tiles) * kFdTile, n0 = n_tile * kFdTile;
  const float *a[kFdTile], *b[kFdTile];  // rows behind the last one repeat it; their sums are not stored
#pragma unroll
  for (int i = 0; i < kFdTile; ++i) {
    a[i] = P.a + (long long)min(m0 + i, P.M - 1) * P.R;
    b[i] = P.b + (long long)min(n0 + i, P.N - 1) * P.R;
  }
  float acc[kFdTile * kFdTile];
#pragma unroll
  for (int i = 0; i < kFdTile * kFdTile; ++i) acc[i] = 0.f;
#pragma unroll 2
  for (int r = (warp * 32 + lane) * VEC; r < P.R; r += warps * 32 * VEC) {
    float x[kFdTile][VEC], w[kFdTile][VEC];
#pragma unroll
    for (int i = 0; i < kFdTile; ++i) {
      if (VEC == 4) {
        const float4 xv = __ldg(reinterpret_cast<const float4*>(b[i] + r)), wv = __ldg(reinterpret_cast<const float4*>(a[i] + r));
        x[i][0] = xv.x; x[i][VEC > 1 ? 1 : 0] = xv.y; x[i][VEC > 2 ? 2 : 0] = xv.z; x[i][VEC > 3 ? 3 : 0] = xv.w;
        w[i][0] = wv.x; w[i][VEC > 1 ? 1 : 0] = wv.y; w[i][VEC > 2 ? 2 : 0] = wv.z; w[i][VEC > 3 ? 3 : 0] = wv.w;
      } else {
        x[i][0] = __ldg(b[i] + r);
        w[i][0] = __ldg(a[i] + r);
      }
    }
#pragma unroll
    for (int n = 0; n < kFdTile; ++n)
#pragma unroll
      for (int m = 0; m < kFdTile; ++m)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[n * kFdTile + m] = fmaf(w[m][e], x[n][e], acc[n * kFdTile + m]);
  }
  // Sixteen sums over 32 lanes: halves of the sums are exchanged for halves of the lanes, lane l ends with sum l >> 1.
#pragma unroll
  for (int half = 8, o = 16; half > 0; half >>= 1, o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = upper ? acc[i + half] : acc[i], give = upper ? acc[i] : acc[i + half];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
  if (!(lane & 1)) s_part[warp][lane >> 1] = acc[0];
  __syncthreads();
  const int n = n0 + tid / kFdTile, m = m0 + (tid & (kFdTile - 1));
  if (tid >= kFdTile * kFdTile || n >= P.N || m >= P.M) return;
  float t = 0.f;
  for (int w = 0; w < warps; ++w) t += s_part[w][tid];
  const FcReduceParams& F = P.post;
  const long long at = (long long)n * F.cols + m;
  if (F.bias) t += __ldg(F.bias + m);
  if (F.relu) t = fmaxf(t, 0.f);
  if (F.drop_mask) t = t * (float)(F.drop_mask[at] != 0u) * F.drop_scale;
  F.out[at] = t;
}

// Splits of the reduction: about two blocks per SM, at least 64 indices each.
int fc_small_splits(int sms, int M, int N, int R) {
  const int tiles = ((M + kFsTile - 1) / kFsTile) * ((N + kFsTile - 1) / kFsTile);
  return std::max(1, std::min(2 * sms / tiles, R / 128));
}

}  // namespace
