// Per-Gaussian passes that reuse the renderer's pair loop.
//
// Activity (render.py:417-442, gaussian_activity): each Gaussian's summed raw weight
// visible_weight(q) = max(exp(-q/2) - tail, 0) over the pixels of its clipped support
// rectangle — opacity-free, the pruning diagnostic of the reference fitter.  Every pixel of the
// rectangle is one in-rectangle pair, so the work is P pairs with no image data, bound by the
// exponentials: 16 per SM and clock, 14.5 us for the 67 M pairs of 250k Gaussians on 1024x1024.
//
// A CTA takes 1 to 256 Gaussians, by their number (activity_group), and each is walked by as many lanes
// as its rectangle needs: up to kSmallArea pixels eight lanes, four Gaussians of a warp at a time; up to
// kWarpArea a warp; larger ones the whole CTA, a band of rows per warp.  A lane walks down whole
// columns, so a pixel costs five instructions and its exponential.  Every sum has a fixed order that
// depends on the rectangle's size alone, so the result is deterministic.  (Lanes striding the pixels row
// by row, the same number for every Gaussian of a call chosen from a mean that the host waited for: 94 us.
// Always 32 Gaussians to a warp, large ones in turn: 500 of 301x301 pixels 1,150 us, the same as 5,000.)
#include "ss_common.cuh"

namespace ss {
namespace {

constexpr int kThreads = 256;

constexpr int kSmallArea = 1024, kWarpArea = 8192;

struct Walk {
  float mx, my, qa, qb, qc;
  int x0, y0, w, h;
};

__device__ __forceinline__ Walk walk_of(const Splat& s) {
  return Walk{s.mx, s.my, s.qa, s.qb, s.qc, s.x0, s.y0, s.x1 - s.x0, s.y1 - s.y0};
}

__device__ __forceinline__ Walk from_lane(const Walk& k, int l) {
  const unsigned all = 0xffffffffu;
  Walk o;
  o.mx = __shfl_sync(all, k.mx, l);
  o.my = __shfl_sync(all, k.my, l);
  o.qa = __shfl_sync(all, k.qa, l);
  o.qb = __shfl_sync(all, k.qb, l);
  o.qc = __shfl_sync(all, k.qc, l);
  o.x0 = __shfl_sync(all, k.x0, l);
  o.y0 = __shfl_sync(all, k.y0, l);
  o.w = __shfl_sync(all, k.w, l);
  o.h = __shfl_sync(all, k.h, l);
  return o;
}

// The sum over columns sub, sub + G, … of the rectangle, each from top to bottom, of lane `sub` of
// G; then over the G lanes.
template <int G, bool FADE>
__device__ __forceinline__ float walk(const Walk& k, int sub, float tail) {
  float acc = 0.f;
  for (int c = sub; c < k.w; c += G) {
    const float dx = (float)(k.x0 + c) - k.mx;
    const float bdx = k.qb * dx, adx2 = k.qa * dx * dx;
    float y = (float)k.y0;  // whole numbers: exact
    float col = 0.f;
#pragma unroll 4
    for (int r = 0; r < k.h; ++r, y += 1.0f) {
      const float dy = y - k.my;
      const float raw = fast_exp2(fmaf(dy, fmaf(k.qc, dy, bdx), adx2));
      col += FADE ? fmaxf(raw - tail, 0.0f) : raw;
    }
    acc += col;
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// The activities of a warp's Gaussians of up to kWarpArea pixels: the first lanes hold one each, and each
// gets its own.  Every lane calls it.
template <bool FADE>
__device__ __forceinline__ float warp_activity(const Walk& mine, float tail) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t area = mine.w > 0 && mine.h > 0 ? (int64_t)mine.w * mine.h : 0;
  float result = 0.f;
  unsigned left = __ballot_sync(all, area > 0 && area <= kSmallArea);
  while (left) {  // four at a time: group g takes the g-th of those left
    unsigned rest = left;
    int src = -1;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int l = rest ? __ffs(rest) - 1 : -1;
      if ((lane >> 3) == g) src = l;
      rest &= rest - 1;
    }
    Walk k = from_lane(mine, src < 0 ? 0 : src);
    if (src < 0) k.w = 0;
    const float sum = walk<8, FADE>(k, lane & 7, tail);
    unsigned taken = left & ~rest;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float v = __shfl_sync(all, sum, 8 * g);
      if (taken && lane == __ffs(taken) - 1) result = v;
      taken &= taken - 1;
    }
    left = rest;
  }
  unsigned medium = __ballot_sync(all, area > kSmallArea && area <= kWarpArea);
  while (medium) {
    const int l = __ffs(medium) - 1;
    medium &= medium - 1;
    const float sum = walk<32, FADE>(from_lane(mine, l), lane, tail);
    if (lane == l) result = sum;
  }
  return result;
}

// The activities of a CTA's `group` Gaussians from `first` on (a power of two, the first group / 8, or
// the first one, lanes of each warp hold them), written out.  load(i) gives Gaussian i's Walk.
template <bool FADE, typename Load>
__device__ __forceinline__ void cta_activity(int64_t first, int64_t n, int group, float tail,
                                             float* __restrict__ activity, Load load) {
  constexpr int kWarps = kThreads / 32;
  __shared__ Walk large[kThreads];
  __shared__ int64_t owner[kThreads];
  __shared__ float part[kThreads][kWarps];
  __shared__ int num_large;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = group < kWarps ? 1 : group / kWarps;
  const int64_t i = first + warp * per + lane;
  if (threadIdx.x == 0) num_large = 0;
  __syncthreads();
  Walk mine{};
  const bool have = lane < per && warp * per < group && i < n;
  if (have) mine = load(i);
  const bool is_large = mine.w > 0 && mine.h > 0 && (int64_t)mine.w * mine.h > kWarpArea;
  if (is_large) {
    const int k = atomicAdd(&num_large, 1);
    large[k] = mine;
    owner[k] = i;
  }
  const float v = warp_activity<FADE>(mine, tail);
  if (have && !is_large) activity[i] = v;
  __syncthreads();
  const int todo = num_large;
  for (int k = 0; k < todo; ++k) {
    Walk band = large[k];
    const int y0 = (int)((int64_t)band.h * warp / kWarps), y1 = (int)((int64_t)band.h * (warp + 1) / kWarps);
    band.y0 += y0;
    band.h = y1 - y0;
    const float sum = walk<32, FADE>(band, lane, tail);
    if (lane == 0) part[k][warp] = sum;
  }
  if (todo == 0) return;
  __syncthreads();
  if (threadIdx.x < todo) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += part[threadIdx.x][w];
    activity[owner[threadIdx.x]] = sum;
  }
}

template <bool FADE>
__global__ void __launch_bounds__(kThreads)
    activity_kernel(const Splat* __restrict__ rec, int64_t n, int group, float tail,
                    float* __restrict__ activity) {
  pdl_wait();
  pdl_trigger();
  cta_activity<FADE>((int64_t)blockIdx.x * group, n, group, tail, activity, [&](int64_t i) {
    Splat s;
    const float4* src = reinterpret_cast<const float4*>(rec + i);
    float4* d = reinterpret_cast<float4*>(&s);
    d[0] = src[0];
    d[1] = src[1];
    d[3] = src[3];
    return walk_of(s);
  });
}

// The same from the render inputs, without records in between.
template <bool FADE>
__global__ void __launch_bounds__(kThreads)
    splat_activity_kernel(const float* __restrict__ means, const float* __restrict__ conics,
                          const int64_t* __restrict__ radii, int64_t n, int H, int W, int group,
                          float tail, float* __restrict__ activity) {
  pdl_wait();
  pdl_trigger();
  cta_activity<FADE>((int64_t)blockIdx.x * group, n, group, tail, activity, [&](int64_t i) {
    const float mx = means[2 * i], my = means[2 * i + 1];
    int x0, y0, x1, y1;
    support_rect(mx, my, radii[2 * i], radii[2 * i + 1], H, W, x0, y0, x1, y1);
    return walk_of(make_splat(mx, my, conics[3 * i], conics[3 * i + 1], conics[3 * i + 2], 1.f, 0.f,
                              0.f, 0.f, x0, y0, x1, y1));
  });
}

// Gaussians per CTA: the largest power of two that leaves eight CTAs, the most that are resident, for
// every SM; 1 to 256.
int activity_group(int64_t n) {
  int group = kThreads;
  while (group > 1 && n < (int64_t)group * 148 * 8) group >>= 1;
  return group;
}

}  // namespace
}  // namespace ss

using namespace ss;

extern "C" {

int ss_gaussian_activity(const void* records, int64_t n, float fade_tail, int lanes_per_gaussian,
                         float* activity, ss_stream_t stream) {
  if (n < 0) return fail(SS_ERR_INVALID_ARGUMENT, "negative size");
  if (n == 0) return SS_OK;
  if (!records || !activity) return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  if (lanes_per_gaussian != 8 && lanes_per_gaussian != 32)
    return fail(SS_ERR_INVALID_ARGUMENT, "lanes_per_gaussian must be 8 or 32");
  const Splat* rec = static_cast<const Splat*>(records);
  const int group = activity_group(n);
  const unsigned blocks = (unsigned)((n + group - 1) / group);
  cudaStream_t s = as_stream(stream);
  if (fade_tail > 0.0f)
    launch("activity_kernel", activity_kernel<true>, blocks, kThreads, 0, s, rec, n, group, fade_tail,
           activity);
  else
    launch("activity_kernel", activity_kernel<false>, blocks, kThreads, 0, s, rec, n, group, fade_tail,
           activity);
  return check_launch("gaussian_activity");
}

int ss_splat_activity(const float* means, const float* conics, const int64_t* radii, int64_t n,
                      int height, int width, float fade_tail, float* activity,
                      ss_stream_t stream) {
  if (n < 0 || height < 0 || width < 0) return fail(SS_ERR_INVALID_ARGUMENT, "negative size");
  if (n > (int64_t)INT32_MAX) return fail(SS_ERR_INVALID_ARGUMENT, "n exceeds int32 ids");
  if (n == 0) return SS_OK;
  if (!means || !conics || !radii || !activity)
    return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  const int group = activity_group(n);
  const unsigned blocks = (unsigned)((n + group - 1) / group);
  cudaStream_t s = as_stream(stream);
  if (fade_tail > 0.0f)
    launch("splat_activity_kernel", splat_activity_kernel<true>, blocks, kThreads, 0, s, means,
           conics, radii, n, height, width, group, fade_tail, activity);
  else
    launch("splat_activity_kernel", splat_activity_kernel<false>, blocks, kThreads, 0, s, means,
           conics, radii, n, height, width, group, fade_tail, activity);
  return check_launch("splat_activity");
}

}  // extern "C"
