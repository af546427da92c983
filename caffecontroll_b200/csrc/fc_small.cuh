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
// 50 images, both ways 13.4 -> 8.9 us.  Three blocks per SM (80 registers) for two jobs: the backward launch took 7.0 us with two, whose
// 384 blocks were two waves, and 6.6 with four; the two launches 3.6 + 4.5.  One job keeps its registers.
#pragma once

namespace {

constexpr int kFsThreads = 256, kFsWarps = 8, kFsTile = 32, kFsChunk = 128, kFsPitch = 36;
// Measured against fc_gemm_kernel, forward + backward, when each contraction was a launch: 4096 -> 10, 50 images (17 MFLOP with the
// padding to 32) 23 -> 14 us; 512 -> 128, 128 images (17) 24 -> 15; 800 -> 500, 64 images (52) 22 -> 26.  Where feature counts are no
// multiples of four the other path copies its operands first: 999 -> 333, 37 images (46) 42 -> 23.  Layers within these lines stay
// with the fp32 products whatever fc_small_faster() says of their backward pass.
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

// TWO: tile and split of one of two jobs (else the grid's x and y, said as such: with variables in their place 290 -> 1200, 97 images
// forward took 13.4 us instead of 11.3).
template <bool TWO>
__device__ __forceinline__ void fc_small_body(const FcSmallParams& P, unsigned tile, unsigned split) {
  __shared__ __align__(16) float s_ab[2 * kFsChunk * kFsPitch];
  __shared__ float s_db[kFsWarps][kFsTile];
  float *s_a = s_ab, *s_b = s_ab + kFsChunk * kFsPitch;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = lane >> 2, tx = lane & 3;
  const int m_tiles = (P.M + kFsTile - 1) / kFsTile, n_tile = (TWO ? tile : blockIdx.x) / m_tiles;  // one grid axis: y ends at 65 535
  const int m0 = ((TWO ? tile : blockIdx.x) - n_tile * m_tiles) * kFsTile, n0 = n_tile * kFsTile;
  const int r_begin = (TWO ? split : blockIdx.y) * P.r_per_split, r_end = min(P.R, r_begin + P.r_per_split);
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
    if (TWO ? P.splits > 1 : gridDim.y > 1) {
      P.out[((long long)(TWO ? split : blockIdx.y) * P.N + n) * P.ld + m] = t;
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
__global__ void __launch_bounds__(kFsThreads) fc_small_kernel(const __grid_constant__ FcSmallParams P) {
  pdl_wait();
  fc_small_body<false>(P, 0, 0);
}
// Three blocks per SM: see above.
__global__ void __launch_bounds__(kFsThreads, 3) fc_small_two_kernel(const __grid_constant__ FcSmallJobs J) {
  pdl_wait();
  const bool second = blockIdx.x >= J.first;
  const FcSmallParams& P = J.job[second];
  const unsigned block = blockIdx.x - (second ? J.first : 0u);
  fc_small_body<true>(P, block / (unsigned)P.splits, block % (unsigned)P.splits);
}

// Forward pass of a small layer: out[n][m] = sum_r A[m][r] B[n][r], rows along the reduction.  A block owns NT images x 4 outputs,
// its warps interleaved steps of 32 (x 4 where rows are on 16-byte boundaries) reduction indices; operands go from L2 straight
// to registers, a warp's sums are added by shuffles and the warps' in order.  With the 32 x 32 tiles of fc_small_kernel a few outputs
// with a long reduction took 32 splits, and a launch to add them; with the splits in a cluster, adding through distributed shared
// memory, 512 indices per block took longer than that launch.  4096 -> 10, 50 images: 4.4 + 2.7 -> 3.4 us, 500 -> 10, 64 images:
// 6.3 + 2.4 -> 2.3.
// What bounds it is the traffic from L2 (3/8 of a word per product with eight images, 1/2 with four, 5/4 with one); fc_gemm_kernel's two
// launches take five microseconds however little there is to do.  Eight images per block where that leaves kDotWideBlocks blocks (512 -> 512,
// 64 images: four 5.5 us, eight 4.5; 2304 -> 64, 32 images, 64 blocks of eight: 2.9 and 3.1) and the loads are wide (999 -> 333, 32
// images: 6.6 and 7.8); one or two images take fewer registers and loads (4096 -> 1000, one image: 6.2 us with eight).
constexpr int kFdM = 4, kFdMaxWarps = 16;
constexpr int kDotWideBlocks = 128;
struct FcDotParams {
  const float *a, *b;
  int M, N, R;
  FcReduceParams post;  // out, ld = cols; bias / ReLU / dropout
};
template <int VEC, int NT>
__global__ void __launch_bounds__(32 * kFdMaxWarps) fc_dot_kernel(const __grid_constant__ FcDotParams P) {
  pdl_wait();
  constexpr int kSums = NT * kFdM;  // 4 ... 32
  __shared__ float s_part[kFdMaxWarps][kSums];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  const int n_tiles = (P.N + NT - 1) / NT, m_tile = blockIdx.x / n_tiles;
  const int n0 = (blockIdx.x - m_tile * n_tiles) * NT, m0 = m_tile * kFdM;
  const float *a[kFdM], *b[NT];  // rows behind the last one repeat it; their sums are not stored
#pragma unroll
  for (int i = 0; i < kFdM; ++i) a[i] = P.a + (long long)min(m0 + i, P.M - 1) * P.R;
#pragma unroll
  for (int i = 0; i < NT; ++i) b[i] = P.b + (long long)min(n0 + i, P.N - 1) * P.R;
  float acc[kSums];
#pragma unroll
  for (int i = 0; i < kSums; ++i) acc[i] = 0.f;
#pragma unroll 2
  for (int r = (warp * 32 + lane) * VEC; r < P.R; r += warps * 32 * VEC) {
    float x[NT][VEC], w[kFdM][VEC];
    auto load = [&](float (&v)[VEC], const float* p) {
      if (VEC == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p + r));
        v[0] = t.x; v[VEC > 1 ? 1 : 0] = t.y; v[VEC > 2 ? 2 : 0] = t.z; v[VEC > 3 ? 3 : 0] = t.w;
      } else {
        v[0] = __ldg(p + r);
      }
    };
#pragma unroll
    for (int i = 0; i < kFdM; ++i) load(w[i], a[i]);
#pragma unroll
    for (int i = 0; i < NT; ++i) load(x[i], b[i]);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int m = 0; m < kFdM; ++m)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[n * kFdM + m] = fmaf(w[m][e], x[n][e], acc[n * kFdM + m]);
  }
  // kSums sums over 32 lanes: halves of the sums are exchanged for halves of the lanes; lane l ends with sum l / kLanes.
  constexpr int kLanes = 32 / kSums;
#pragma unroll
  for (int half = kSums / 2, o = 16; half > 0; half >>= 1, o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = upper ? acc[i + half] : acc[i], give = upper ? acc[i] : acc[i + half];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
  if (lane % kLanes == 0) s_part[warp][lane / kLanes] = acc[0];
  __syncthreads();
  const int n = n0 + tid / kFdM, m = m0 + (tid & (kFdM - 1));
  if (tid >= kSums || n >= P.N || m >= P.M) return;
  float t = 0.f;
  for (int w = 0; w < warps; ++w) t += s_part[w][tid];
  const FcReduceParams& F = P.post;
  const long long at = (long long)n * F.cols + m;
  if (F.bias) t += __ldg(F.bias + m);
  if (F.relu) t = fmaxf(t, 0.f);
  if (F.drop_mask) t = t * (float)(F.drop_mask[at] != 0u) * F.drop_scale;
  F.out[at] = t;
}
template <int VEC>
void (*fc_dot_pick(int nt))(const FcDotParams) {
  return nt == 1 ? fc_dot_kernel<VEC, 1> : nt == 2 ? fc_dot_kernel<VEC, 2> : nt == 4 ? fc_dot_kernel<VEC, 4> : fc_dot_kernel<VEC, 8>;
}

// Splits of the reduction: about two blocks per SM, about 128 indices each at the least.
int fc_small_splits(int sms, int M, int N, int R) {
  const int tiles = ((M + kFsTile - 1) / kFsTile) * ((N + kFsTile - 1) / kFsTile);
  return std::max(1, std::min(2 * sms / tiles, R / 128));
}

// Whether a forward pass is faster by fc_dot_kernel.  Its time follows the products with the reduction rounded up, since lanes behind its
// end have none (a warp's step is 128 indices, 32 off a 16-byte boundary, where short steps also pay for their blocks: 64 in their place):
// 1.8 us + 0.18 per million by wide loads, 0.35 and more by narrow ones.
// Against one launch of fc_small_kernel (`one_launch`: a small layer without splits; 3.6 us up to 64 indices, 4.0 - 5.5 to 255), us there ->
// here, on both sides of each line: wide 64 -> 512, 128 images (8 M) 4.0 -> 3.2, 256 (17 M) 4.0 -> 5.0; 16 -> 130, 640 (11 M) 3.6 -> 4.0;
// 128 -> 1000, 64 (8 M) 4.5 -> 3.1, 128 (16 M) 4.6 -> 5.0; narrow 16 -> 2048, 32 (4.2 M) 3.7 -> 4.0; 130 -> 500, 64 (6.1 M) 5.4 -> 5.0; 128 ->
// 128, 1024 (17 M) 4.6 -> 11.2.
// Against two launches, of fc_small_kernel with splits or of the tensor cores: wide 512 -> 128, 256 images (17 M) 6.2 -> 4.6; 512 -> 512, 64
// (17 M) 6.7 -> 4.5, 128 (34 M) 8.2 -> 7.7, 256 (67 M) 11.6 -> 13.3; 1024 -> 1000, 20 (20 M) 6.45 -> 6.45; 800 -> 500, 64 (29 M) 7.7 -> 8.0;
// 16 -> 2048, 384 (101 M) 9.6 -> 18.2.  Narrow ones against the tiles, whose splits grow with the reduction: 256 -> 500, 64 images (8.2 M) 6.1 ->
// 6.7; 1024 -> 1000, eight (8.2 M) 7.4 -> 5.2, 16 (16 M) 7.7 -> 8.6; 512 -> 500, 64 (16 M) 6.3 -> 12.8; 2048 -> 100, 64 (13 M) 6.2 -> 6.0; 4096
// -> 100, 50 (20 M) 8.4 -> 8.5.  Up to four images are the stream of the weights, which the tiles read for images that are not there: 4096
// -> 1000, four (16 M) 15.9 -> 5.4; `padded`: the tensor cores' four launches, 4093 -> 1001, four 16.3 -> 5.4.
bool fc_dot_faster(int B, int K, int O, bool wide, bool one_launch, bool padded) {
  const int step = wide ? 128 : 64;
  const double products = (double)B * O * ((K + step - 1) / step) * step;
  if (one_launch) return products <= (wide ? (K <= 64 ? 1e7 : 1.3e7) : (K <= 64 ? 4e6 : 6.4e6));
  return products <= (wide || padded || B <= 4 ? 2.4e7 : std::min(2.4e7, 6.5e6 + 5e3 * K));
}

// Whether a backward pass is faster by fc_small_kernel: a fit to both paths' times (us).  Chunks of 128 indices of the two jobs' blocks,
// 2.0 - 2.9 us for every one that an SM has (0.85 of that beyond 6 us, where blocks overlap), but no less than the chunks
// of the longest block, which walks the whole batch for its tile of the weight gradient; against 8.7 us for five launches of the
// tensor-core path (6.5: `pair`, both contractions in one), the stream of the weights and their gradient, and wider tiles, whose chain over
// the batch is 0.67 us per block of 32.  Us there -> here (estimates): 1000 -> 100, 256 images 18.1 -> 11.8 (16.8, 11.7); 784 -> 128, 256
// images 17.9 -> 10.8 (16.8, 10.2); 64 -> 512, 8192 images 173 -> 147 (187, 169).  Where the tensor cores stay: 800 -> 256, 128 images 8.9
// (10.8 here; 10.8, 11.8); 200 -> 1024, 128 images 8.5 (13.4); 1000 -> 100, 640 images 23.7 (24.3; 25.0, 24.1); 784 -> 128, 4096 images 100 (103;
// 99, 110); 4096 -> 1000, one image 15.6 (60).
bool fc_small_faster(int sms, int B, int K, int O, bool pair) {
  auto up = [](int a, int b) { return (double)((a + b - 1) / b); };
  const int splits = fc_small_splits(sms, K, B, O);
  auto cost = [](double r) { return 2.0 + 0.9 * std::min(1.0, r / kFsChunk); };  // of a chunk with r indices
  const double k = up(K, kFsTile), w = k * up(O, kFsTile) * up(B, kFsChunk) * cost(B);
  const double d = k * up(B, kFsTile) * splits * up((O + splits - 1) / splits, kFsChunk) * cost((double)O / splits), even = (w + d) / sms;
  const double small = 2.6 + std::max(std::min(even, 0.9 + 0.85 * even), 2.6 * up(B, kFsChunk)) + (splits > 1 ? 1.6 : 0.0);
  const double tensor = (pair ? 6.5 : 8.7) + 1.7e-6 * K * O + (B <= 256 ? 0.031 * B : 2.4 + 0.0215 * B) + (K % 4 || O % 4 ? 5.0 : 0.0);
  return small < 0.95 * tensor;
}

}  // namespace
