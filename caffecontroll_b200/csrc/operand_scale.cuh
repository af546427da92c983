// How the operands of a contraction are split into pairs of fp16 (three products of fp16 with fp32 sums in place of three of tf32).
//
// A pair holds 22 bits of a value as a pair of tf32 does - lo is rounded here, cut by the tensor core there - and one instruction takes 16 of
// the reduction instead of 8 in the same time, with half the words of A in tensor memory and of B in shared memory, and with half the
// truncated additions into the accumulator.  What fp16 does not have is fp32's range: an operand is multiplied by a power of two that
// brings its largest finite value to [2^14, 2^15).  A value 18 octaves below that one keeps 21 bits, one further down an error of 2^-40 of the
// largest.  So an operand is `ok` where the values of every stretch of some ten thousand in a row are, by their geometric mean over those
// that are not 0, at most kHalfOctaves below the largest of all (normally distributed values: 3.3 octaves), and the largest lies within
// 2^-45 .. 2^46; a contraction whose operands are not both ok runs on tf32 pairs as before.  Values that are not finite take no part
// in this and are Inf or NaN in the products of their windows either way.
//
// Bound by memory: one read of each operand (CaffeNet conv2's X at batch 256, 72 MB, most of it in L2 behind the kernel that wrote it).
#pragma once

namespace {

constexpr int kHalfOctaves = 18;
constexpr int kScaleThreads = 256, kScaleBlocksPerSm = 6;
constexpr int kScaleChunk = 8192;  // elements of a block at least

struct ScaleJob {
  const float* a = nullptr;
  const float* mask = nullptr;  // set: elements whose mask is not positive count as 0
  size_t n = 0, per_block = 0;
  int first = 0, blocks = 0;    // of the grid
  int slot = 0;
  int headroom = 0;             // octaves that the operand may be larger than `a` (sums of up to four windows' gradients: 2)
  // Of a pooled gradient: which element of its plane of `plane` each is added to, and the pooled planes' size.
  const int32_t* where = nullptr;
  int pooled = 1, plane = 1;
};
struct ScaleJobs {
  ScaleJob job[3];
  int jobs;
  HalfScales* out;
  uint2* parts;       // per block: the largest value's bits, the mean exponent of those that are not 0 (each rounded down to even)
  uint32_t* ticket;   // two words, 0 before and after every launch: blocks that are through, values that are not finite
};

// The largest finite value, the number of those that are not 0 and the sum of their exponents, halved (the top byte: one instruction).
struct ScaleStats {
  uint32_t top = 0, count = 0, halves = 0;
  // 4 * N values; all finite, as nearly always (and said so): four instructions each
  template <int N>
  __device__ __forceinline__ bool add(const float4 (&v)[N]) {
    uint32_t u[4 * N], most = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      u[4 * i] = __float_as_uint(v[i].x) & 0x7fffffffu; u[4 * i + 1] = __float_as_uint(v[i].y) & 0x7fffffffu;
      u[4 * i + 2] = __float_as_uint(v[i].z) & 0x7fffffffu; u[4 * i + 3] = __float_as_uint(v[i].w) & 0x7fffffffu;
    }
#pragma unroll
    for (int i = 0; i < 4 * N; ++i) most = max(most, u[i]);
    const bool finite = most < 0x7f800000u;
    if (!finite) {
      most = 0;
#pragma unroll
      for (int i = 0; i < 4 * N; ++i) {
        u[i] = u[i] < 0x7f800000u ? u[i] : 0u;
        most = max(most, u[i]);
      }
    }
    top = max(top, most);
#pragma unroll
    for (int i = 0; i < 4 * N; ++i) {
      count += min(u[i], 1u);
      halves = __dp4a(u[i], 0x01000000u, halves);
    }
    return finite;
  }
};

// Lists what is not finite of four elements of dY from `i` on.
__device__ __noinline__ void list_bad(const ScaleJobs& J, const ScaleJob& job, size_t i, float4 v) {
  const float x[4] = {v.x, v.y, v.z, v.w};
  for (int e = 0; e < 4; ++e)
    if ((__float_as_uint(x[e]) & 0x7f800000u) == 0x7f800000u) {
      const uint32_t at = atomicAdd(J.ticket + 1, 1u);
      if (at < (uint32_t)kMaxBad) J.out->bad[at] = (int)(job.where ? (i + e) / job.pooled * job.plane + __ldg(job.where + i + e) : i + e);
    }
}

__global__ void __launch_bounds__(kScaleThreads, kScaleBlocksPerSm) operand_scale_kernel(const __grid_constant__ ScaleJobs J) {
  __shared__ uint32_t part[3][kScaleThreads / 32];
  __shared__ bool last;
  pdl_wait();
  int which = 0;
  while (which + 1 < J.jobs && (int)blockIdx.x >= J.job[which + 1].first) ++which;
  const ScaleJob& job = J.job[which];
  const size_t begin = (size_t)(blockIdx.x - job.first) * job.per_block, end = min(job.n, begin + job.per_block);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  ScaleStats s;
  // per_block is a multiple of 1024 floats: a block's part starts on a 16-byte boundary if the tensor does
  const bool wide = ((reinterpret_cast<uintptr_t>(job.a) | reinterpret_cast<uintptr_t>(job.mask)) & 15) == 0;
  size_t i = begin + (size_t)tid * 4;
  if (wide) {
    constexpr int kAhead = 4;
    for (; i + (kAhead - 1) * kScaleThreads * 4 + 4 <= end; i += kAhead * kScaleThreads * 4) {
      float4 v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) v[u] = __ldg(reinterpret_cast<const float4*>(job.a + i + u * kScaleThreads * 4));
      if (job.mask) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const float4 m = __ldg(reinterpret_cast<const float4*>(job.mask + i + u * kScaleThreads * 4));
          v[u] = make_float4(m.x > 0.f ? v[u].x : 0.f, m.y > 0.f ? v[u].y : 0.f, m.z > 0.f ? v[u].z : 0.f, m.w > 0.f ? v[u].w : 0.f);
        }
      }
      if (!s.add(v) && job.slot == kHalfDy)
        for (int u = 0; u < kAhead; ++u) list_bad(J, job, i + u * kScaleThreads * 4, v[u]);
    }
  }
  for (; i < end; i += kScaleThreads * 4) {
    float t[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) t[e] = i + e < end && (!job.mask || __ldg(job.mask + i + e) > 0.f) ? __ldg(job.a + i + e) : 0.f;
    const float4 v[1] = {make_float4(t[0], t[1], t[2], t[3])};
    if (!s.add(v) && job.slot == kHalfDy) list_bad(J, job, i, v[0]);
  }
  s.top = __reduce_max_sync(0xffffffffu, s.top);
  s.count = __reduce_add_sync(0xffffffffu, s.count);
  s.halves = __reduce_add_sync(0xffffffffu, s.halves);
  if (lane == 0) { part[0][warp] = s.top; part[1][warp] = s.count; part[2][warp] = s.halves; }
  __syncthreads();
  if (tid == 0) {
    unsigned long long halves = 0;
    uint32_t top = 0, count = 0;
    for (int w = 0; w < kScaleThreads / 32; ++w) { top = max(top, part[0][w]); count += part[1][w]; halves += part[2][w]; }
    J.parts[blockIdx.x] = make_uint2(top, count ? (uint32_t)(2 * halves / count) : 255u);
    __threadfence();
    last = atomicInc(J.ticket, gridDim.x - 1) == gridDim.x - 1;  // (back to 0 with the last one)
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // The last block reads what the others left, every thread a few, all at once: by a warp for each operand, one read behind the other, the launch took
  // 24 us of which the operands took 8 (CaffeNet conv4 at batch 256).
  uint32_t top[3] = {0, 0, 0}, low[3] = {255, 255, 255};
#pragma unroll 4
  for (int b = tid; b < (int)gridDim.x; b += kScaleThreads) {
    const uint2 p = __ldcg(J.parts + b);
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < J.jobs && b >= J.job[j].first && b < J.job[j].first + J.job[j].blocks) {
        top[j] = max(top[j], p.x);
        low[j] = min(low[j], p.y);
      }
  }
  __shared__ uint32_t tops[3][kScaleThreads / 32], lows[3][kScaleThreads / 32];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    top[j] = __reduce_max_sync(0xffffffffu, top[j]);
    low[j] = __reduce_min_sync(0xffffffffu, low[j]);
    if (lane == 0) { tops[j][warp] = top[j]; lows[j][warp] = low[j]; }
  }
  __syncthreads();
  if (tid < J.jobs) {
    const ScaleJob& mine = J.job[tid];
    uint32_t most = 0, least = 255;
    for (int w = 0; w < kScaleThreads / 32; ++w) { most = max(most, tops[tid][w]); least = min(least, lows[tid][w]); }
    const int e = (int)(most >> 23), up = 14 - mine.headroom - (e - 127);  // the scale is 2^up
    const bool ok = most == 0 || (e >= 127 - 45 && e <= 127 + 45 && (int)least >= e - kHalfOctaves);
    const bool scaled = ok && most != 0;
    J.out->of[mine.slot] = HalfScale{scaled ? __uint_as_float((uint32_t)(127 + up) << 23) : 1.f,
                                     scaled ? __uint_as_float((uint32_t)(127 - up) << 23) : 1.f, ok ? 1 : 0,
                                     mine.slot == kHalfDy ? (int)min(atomicExch(J.ticket + 1, 0u), (uint32_t)kMaxBad + 1u) : 0};
  }
}

}  // namespace
