// Tile binning: count -> exclusive scan -> fill -> per-tile sort.
//
// Result contract (cuda_render.py:177-226, render_ext.cu:858-952): tile t lists every Gaussian
// whose clipped support rectangle touches it, offsets[t]..offsets[t+1]; the lists are sorted by
// ascending Gaussian id, which is the order the reference's stable radix sort leaves and makes
// every downstream sum deterministic.  No sort over all pairs is needed: per-tile counts come
// from atomics, a scan gives the offsets, and each tile's ids are put into ascending order by
// one CTA.  Two forms, by the size of the caller's workspace:
//
//   binned (a workspace of ss_tile_index_binned_workspace_bytes): the count's atomics return each
//     pair's rank in its tile, so the same kernel drops the id into the tile's bin, and
//     bin_sort_kernel orders each bin into the list.  At 100k Gaussians on 1024x1024 (213k pairs)
//     the fill, warp-sort and block-sort launches after the count took 12 + 6.4 + 4.2 us; this one
//     takes their place, and lists the few tiles whose bins overflowed.
//   plain (a workspace of ss_tile_index_workspace_bytes, which depends on the tiles only): the
//     fill enumerates the pairs again and claims slots with per-tile atomic cursors, then a
//     warp or a CTA sorts each list.
#include <climits>

#include <cub/block/block_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "ss_common.cuh"

namespace ss {
namespace {

constexpr int kThreads = 256;
constexpr int kSmallRect = 8;          // tiles a lane enumerates alone; larger rects use the warp
constexpr int kWarpSortMax = 1024;     // per-warp register sort capacity (ints)
constexpr int kBigSortSmem = 16384;    // per-CTA shared-memory sort capacity (ints)
// Per-tile counters sit one per 32-byte sector: a tile receives one atomic per Gaussian that
// touches it, and packing 8 neighbouring tiles' counters into a sector would serialise their
// atomics in the L2.
constexpr int kCounterStride = 8;

struct CounterLoad {
  const int* base;
  __host__ __device__ int operator()(int64_t t) const { return base[t * kCounterStride]; }
};

inline auto counter_iter(const int* base) {
  return thrust::make_transform_iterator(thrust::make_counting_iterator<int64_t>(0),
                                         CounterLoad{base});
}

struct TileGrid {
  int ts, tiles_x, tiles_y;
  int64_t T;
};

inline TileGrid make_grid(int H, int W, int ts) {
  TileGrid g;
  g.ts = ts;
  g.tiles_x = (W + ts - 1) / ts;
  g.tiles_y = (H + ts - 1) / ts;
  g.T = (int64_t)g.tiles_x * g.tiles_y;
  return g;
}

// Workspace layout (each region 256-byte aligned).
struct IndexWorkspace {
  int* tile_count;        // T+1   per-tile counters (fill consumes them back to zero)
  long long* offsets64;   // T+1   exclusive scan in int64
  int* big_tiles;         // T     tiles whose list is too long for the warp sort
  int* big_count;         // 1
  void* scan_temp;
  size_t scan_bytes;
  int32_t* bins;          // T x bin_ids, or NULL: ids by tile in arrival order
  int bin_ids;            // K, ids a bin holds
};

// Ids per bin: 32 times the Gaussians per tile.  Lists of 32-px tiles average 2 to 8 times them, those
// of smaller tiles or wider Gaussians more (ss_tile_index_entries_workspace_bytes then names the plain
// form); a tile beyond its bin is listed by bin_sort_kernel.  0, no bins, without Gaussians or tiles and
// where very many tiles would make them larger than 256 MB + 256 B per Gaussian.
int bin_ids_for(int64_t n, int64_t T) {
  if (n <= 0 || T <= 0) return 0;
  int64_t k = 32 * ((n + T - 1) / T) + 32;
  if (k > n) k = n;
  k = (k + 7) & ~int64_t(7);  // every bin starts on a 32-byte sector
  if (T * k * (int64_t)sizeof(int32_t) > ((int64_t)256 << 20) + 256 * n) return 0;
  return (int)k;
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

size_t scan_temp_bytes(int64_t items) {
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveScan(nullptr, bytes, counter_iter(nullptr), (long long*)nullptr,
                                 ::cuda::std::plus<long long>(), (long long)0, (int)items);
  return bytes;
}

size_t index_workspace_bytes(int64_t T) {
  return align256(sizeof(int) * kCounterStride * (T + 1)) +
         align256(sizeof(long long) * (T + 1)) +
         align256(sizeof(int) * (T > 0 ? T : 1)) + align256(sizeof(int)) +
         align256(scan_temp_bytes(T + 1));
}

size_t binned_workspace_bytes(int64_t n, int64_t T) {
  return index_workspace_bytes(T) +
         align256((size_t)T * (size_t)bin_ids_for(n, T) * sizeof(int32_t));
}

IndexWorkspace carve(void* base, size_t bytes, int64_t n, int64_t T) {
  IndexWorkspace w;
  char* p = static_cast<char*>(base);
  w.tile_count = reinterpret_cast<int*>(p);
  p += align256(sizeof(int) * kCounterStride * (T + 1));
  w.offsets64 = reinterpret_cast<long long*>(p);
  p += align256(sizeof(long long) * (T + 1));
  w.big_tiles = reinterpret_cast<int*>(p);
  p += align256(sizeof(int) * (T > 0 ? T : 1));
  w.big_count = reinterpret_cast<int*>(p);
  p += align256(sizeof(int));
  w.scan_temp = p;
  w.scan_bytes = align256(scan_temp_bytes(T + 1));
  p += w.scan_bytes;
  w.bin_ids = bytes >= binned_workspace_bytes(n, T) ? bin_ids_for(n, T) : 0;
  w.bins = w.bin_ids > 0 ? reinterpret_cast<int32_t*>(p) : nullptr;
  return w;
}

struct TileRect {
  int gx0, gy0, gw, gh;
};

__device__ __forceinline__ TileRect tile_rect(const int4& b, int ts) {
  TileRect r{0, 0, 0, 0};
  if (b.z > b.x && b.w > b.y) {
    r.gx0 = b.x / ts;
    r.gy0 = b.y / ts;
    r.gw = (b.z - 1) / ts - r.gx0 + 1;
    r.gh = (b.w - 1) / ts - r.gy0 + 1;
  }
  return r;
}

__device__ __forceinline__ Splat load_splat(const Splat* rec, int64_t i) {
  Splat s;
  const float4* src = reinterpret_cast<const float4*>(rec + i);
  float4* d = reinterpret_cast<float4*>(&s);
  d[0] = src[0];
  d[1] = src[1];
  d[2] = src[2];
  d[3] = src[3];
  return s;
}

__device__ __forceinline__ TileRect tile_rect_of(const Splat* rec, int64_t i, int ts) {
  return tile_rect(reinterpret_cast<const int4*>(rec + i)[3], ts);
}

// Calls visit(slot, gaussian, tile) for every tile of Gaussian i of each lane of a warp, in any order.
// Each lane enumerates a rectangle of up to kSmallRect tiles itself (unrolled, so independent
// atomics are in flight together); a larger rectangle is enumerated by the whole warp so one
// huge Gaussian cannot serialise a lane.  Tile coordinates advance incrementally (no division).
template <bool CULL, typename Visit>
__device__ __forceinline__ void enumerate_pairs(const Splat* rec, int64_t i, int64_t n, int ts,
                                                const Frames& frames, float cutoff2,
                                                Visit visit) {
  int lane = threadIdx.x & 31;
  TileRect r{0, 0, 0, 0};
  int tiles_x = 0, first_tile = 0;
  if (i < n) {
    r = tile_rect_of(rec, i, ts);
    const Frame fr = frame_of_gaussian(frames, i, n);
    tiles_x = fr.tiles_x;
    first_tile = fr.first_tile;
  }
  int cnt = r.gw * r.gh;
  if (cnt > 0 && cnt <= kSmallRect) {
    Splat s;
    if (CULL) s = load_splat(rec, i);
    int gx = r.gx0, gy = r.gy0;
#pragma unroll
    for (int k = 0; k < kSmallRect; ++k) {
      if (k < cnt) {
        if (!(CULL && culled(s, gx, gy, ts, cutoff2)))
          visit(k, (int)i, first_tile + gy * tiles_x + gx);
        if (++gx == r.gx0 + r.gw) {
          gx = r.gx0;
          ++gy;
        }
      }
    }
  }
  unsigned big = __ballot_sync(0xffffffffu, cnt > kSmallRect);
  while (big) {
    int src = __ffs(big) - 1;
    big &= big - 1;
    int gx0 = __shfl_sync(0xffffffffu, r.gx0, src);
    int gy0 = __shfl_sync(0xffffffffu, r.gy0, src);
    int gw = __shfl_sync(0xffffffffu, r.gw, src);
    int total = __shfl_sync(0xffffffffu, cnt, src);
    const int tx_src = __shfl_sync(0xffffffffu, tiles_x, src);
    const int base_src = __shfl_sync(0xffffffffu, first_tile, src);
    long long gi = __shfl_sync(0xffffffffu, (long long)i, src);
    Splat s;
    if (CULL) s = load_splat(rec, gi);
    const int step_y = 32 / gw, step_x = 32 - step_y * gw;
    int gy = gy0 + lane / gw, gx = gx0 + lane % gw;
    for (int k = lane; k < total; k += 32) {
      if (!(CULL && culled(s, gx, gy, ts, cutoff2)))
        visit(-1, (int)gi, base_src + gy * tx_src + gx);
      gx += step_x;
      gy += step_y;
      if (gx >= gx0 + gw) {
        gx -= gw;
        ++gy;
      }
    }
  }
}

// Whether a tile whose bin does not hold its list of len ids is listed by testing every record of its
// image, or else from the pairs (place_overflow).  The machine tests ~370 records per ns and places ~40
// pairs, so lists of more than 1/8 of the image's Gaussians are sooner found that way (`tests` 8), and all
// of them where the whole set's tests are few (see index_tests).  Either way the work is bounded by the
// pairs or by kFewTests.
constexpr int kSortIds = 4096;                      // most ids sorted in shared memory
constexpr int kWindowIds = 32 * (kSortIds + 1024);  // most ids a bitmap there holds: 163,840
// Few: 45 us if every tile overflowed; or few for each tile and, where some overflow, not many in all
// (3,000 Gaussians of 240 px at 4K in 16-px tiles, most in one clump: a step of 826 us, 883 with them
// placed).
constexpr int64_t kFewTests = 1 << 24;
inline bool few_tests(int64_t n, int64_t T) { return n * T <= kFewTests; }
inline int index_tests(int64_t n, int64_t T) {
  return few_tests(n, T) || (n <= 4096 && n * T <= 8 * kFewTests) ? INT_MAX : 8;
}
__host__ __device__ inline bool listed_from_records(int64_t len, int64_t count, int tests) {
  return len * tests >= count;
}

// Whether the plain form is the better one for about `entries` pairs: where the lists of an even field,
// three deviations above their mean, outgrow their bins, are short (a second walk over the pairs then
// costs more than the bins saved; for long lists the plain form's sorts cost more) and are not found
// from the records.  Count and fill, plain and binned: 100k Gaussians in 4-px tiles on
// 1024x1024, lists of 74 beside bins of 96, 120 and 189 us, of 180 266 and 597; in 16-px tiles 378 beside
// 832 68 and 51, 1,133 beside 832 361 and 318; 250k in 32-px tiles 11,400 beside 7,872 1,346 and 630.
inline bool prefer_plain(int64_t n, int64_t T, int images, int64_t entries) {
  if (T <= 0 || few_tests(n, T)) return false;
  const int64_t mean = entries / T, over = mean - bin_ids_for(n, T);
  return mean < 1024 && (over > 0 || over * over < 9 * mean) &&
         !listed_from_records(mean, n / (images > 0 ? images : 1), 8);
}

// Words in the padding after the counters, zeroed with them.  Of counter 0: the bins' size, whether
// some tile needs place_overflow, and its tickets; of each counter: the slots claimed in its list.
constexpr int kBinsWord = 2, kOverflowWord = 3, kTicketWord = 5, kPlacedWord = 6, kExitWord = 7;
constexpr int kClaimWord = 4;
// Notes that a tile of cnt pairs needs place_overflow.
__device__ __forceinline__ void note_overflow(int64_t cnt, int64_t t, const Frames& frames,
                                              int64_t n, int K, int tests, int* tile_count) {
  if (K > 0 && cnt > K &&
      !listed_from_records(cnt, frame_of_tile(frames, (int)t, n).gauss_count, tests))
    tile_count[kOverflowWord] = 1;
}

// Counts one CTA's pairs: thread l holds Gaussian `first + l` with record s (`in`: there is one).
// The threads share the CTA's pairs evenly, whatever the rectangles' sizes: pair e belongs to
// the last thread whose exclusive prefix of tile counts is <= e.  (Shared by warps only, the warp
// with the widest Gaussians of a heavy-tailed field sets the kernel's time: 69 us for 250k
// Gaussians and 2 M pairs.)  BINS: each pair's rank in its tile, which its atomic returns, is its
// slot in the tile's bin (a full bin drops the id; the count still tells the list's length).  What
// is left is the L2's rate of atomics and of scattered 4-byte stores, ~70 and ~100 per ns.
// Rectangles of more than kHugeRect tiles take the whole CTA one after the other, so the prefix
// stays small.
constexpr int kHugeRect = 1 << 20;

struct PairShare {
  int excl[kThreads], tile0[kThreads], gw[kThreads], gh[kThreads], tiles_x[kThreads];
  int warp_total[kThreads / 32];
  unsigned huge[kThreads / 32];
};
struct CullShare {  // the ellipse cull's inputs
  float mx[kThreads], my[kThreads], a[kThreads], b[kThreads], c[kThreads];
  int4 rect[kThreads];
};

template <bool CULL, bool BINS>
__device__ __forceinline__ void count_pairs(const Splat& s, bool in, int first, int ts,
                                            int tiles_x, int first_tile, float cutoff2,
                                            int* tile_count, int32_t* bins, int K) {
  __shared__ PairShare sh;
  __shared__ CullShare cs[1];
  const unsigned all = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  TileRect r{0, 0, 0, 0};
  if (in) r = tile_rect(make_int4(s.x0, s.y0, s.x1, s.y1), ts);
  const int cnt = r.gw * r.gh;
  const int own = cnt > kHugeRect ? 0 : cnt;
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(all, incl, o);
    if (lane >= o) incl += v;
  }
  const unsigned huge_mask = __ballot_sync(all, cnt > kHugeRect);
  if (lane == 31) sh.warp_total[warp] = incl;
  if (lane == 0) sh.huge[warp] = huge_mask;
  sh.tile0[tid] = first_tile + r.gy0 * tiles_x + r.gx0;
  sh.gw[tid] = r.gw;
  sh.gh[tid] = r.gh;
  sh.tiles_x[tid] = tiles_x;
  if (CULL) {
    cs[0].mx[tid] = s.mx;
    cs[0].my[tid] = s.my;
    cs[0].a[tid] = s.a;
    cs[0].b[tid] = s.b;
    cs[0].c[tid] = s.c;
    cs[0].rect[tid] = make_int4(s.x0, s.y0, s.x1, s.y1);
  }
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    const int t = sh.warp_total[w];
    base += w < warp ? t : 0;
    total += t;
  }
  sh.excl[tid] = base + incl - own;
  __syncthreads();
  auto tile_of = [&](int l, unsigned k) {  // -1: culled
    const unsigned gw = (unsigned)sh.gw[l];
    const int row = (int)(k / gw), col = (int)(k - (unsigned)row * gw);
    if (CULL) {
      Splat o;
      o.mx = cs[0].mx[l];
      o.my = cs[0].my[l];
      o.a = cs[0].a[l];
      o.b = cs[0].b[l];
      o.c = cs[0].c[l];
      const int4 b = cs[0].rect[l];
      o.x0 = b.x;
      o.y0 = b.y;
      o.x1 = b.z;
      o.y1 = b.w;
      if (culled(o, b.x / ts + col, b.y / ts + row, ts, cutoff2)) return -1;
    }
    return sh.tile0[l] + row * sh.tiles_x[l] + col;
  };
  for (int e0 = tid; e0 < total; e0 += 2 * kThreads) {  // two pairs per thread in flight
    int tile[2] = {-1, -1}, owner[2] = {0, 0}, rank[2] = {0, 0};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = e0 + u * kThreads;
      if (e < total) {
        int l = 0;
#pragma unroll
        for (int step = kThreads / 2; step > 0; step >>= 1)
          if (sh.excl[l + step] <= e) l += step;
        owner[u] = l;
        tile[u] = tile_of(l, (unsigned)(e - sh.excl[l]));
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (tile[u] >= 0) rank[u] = atomicAdd(tile_count + (int64_t)tile[u] * kCounterStride, 1);
    if (BINS) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (tile[u] >= 0 && rank[u] < K) bins[(int64_t)tile[u] * K + rank[u]] = first + owner[u];
    }
  }
  for (int w = 0; w < kThreads / 32; ++w) {
    for (unsigned huge = sh.huge[w]; huge; huge &= huge - 1) {
      const int l = 32 * w + __ffs(huge) - 1;
      const unsigned n = (unsigned)sh.gw[l] * (unsigned)sh.gh[l];
      for (unsigned k = tid; k < n; k += kThreads) {
        const int t = tile_of(l, k);
        if (t < 0) continue;
        const int rank = atomicAdd(tile_count + (int64_t)t * kCounterStride, 1);
        if (BINS && rank < K) bins[(int64_t)t * K + rank] = first + l;
      }
    }
  }
}

// Per-tile counts by atomics, and with BINS the bins.  A padding word of counter 0 tells
// bin_sort_kernel that the bins belong to these counts.
template <bool CULL, bool BINS>
__global__ void tile_count_kernel(const Splat* __restrict__ rec, int64_t n, int ts, Frames frames,
                                  float cutoff2, int* __restrict__ tile_count,
                                  int32_t* __restrict__ bins, int K) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (BINS && i == 0) tile_count[kBinsWord] = K;
  Splat s{};
  int tiles_x = 0, first_tile = 0;
  if (i < n) {
    if (CULL) {
      s = load_splat(rec, i);
    } else {
      const int4 b = reinterpret_cast<const int4*>(rec + i)[3];
      s.x0 = b.x;
      s.y0 = b.y;
      s.x1 = b.z;
      s.y1 = b.w;
    }
    const Frame fr = frame_of_gaussian(frames, i, n);
    tiles_x = fr.tiles_x;
    first_tile = fr.first_tile;
  }
  count_pairs<CULL, BINS>(s, i < n, blockIdx.x * kThreads, ts, tiles_x, first_tile, cutoff2,
                          tile_count, bins, K);
}

// The RS projection (rs_project_one, as project_rs_kernel) and the per-tile counts in one pass:
// each thread stores its Gaussian's record and counts its tiles from the registers that hold it.
// BINS as in tile_count_kernel.  The grid also zeroes `clear_vec` 16-byte words at
// `clear` (a caller's per-step scratch, such as the next backward's moments).
template <bool CULL, bool BINS>
__global__ void project_count_kernel(RSField field, int64_t n, int ts, Frames frames,
                                     float cutoff2, Splat* __restrict__ out,
                                     int* __restrict__ tile_count, uint4* __restrict__ clear,
                                     int64_t clear_vec,
                                     int32_t* __restrict__ bins, int K) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (BINS && i == 0) tile_count[kBinsWord] = K;
  for (int64_t v = i; v < clear_vec; v += (int64_t)gridDim.x * blockDim.x)
    clear[v] = make_uint4(0u, 0u, 0u, 0u);
  Splat s{};
  int tiles_x = 0, first_tile = 0;
  if (i < n) {
    const RSParams p = rs_load(field, i);
    const Frame fr = frame_of_gaussian(frames, i, n);
    float rx, ry;
    s = rs_project_one(field, p, fr.H, fr.W, rx, ry);
    store_splat(out + i, s);
    tiles_x = fr.tiles_x;
    first_tile = fr.first_tile;
  }
  count_pairs<CULL, BINS>(s, i < n, blockIdx.x * kThreads, ts, tiles_x, first_tile, cutoff2,
                          tile_count, bins, K);
}

// The render inputs (ss_pack_splats).
struct PackField {
  const float *means, *conics, *colors;
  const int64_t* radii;
  const float* opacities;
};

// Packing and the per-tile counts in one pass, as project_count_kernel.
template <bool CULL, bool BINS>
__global__ void pack_count_kernel(PackField f, int64_t n, int ts, Frames frames, float cutoff2,
                                  Splat* __restrict__ out, int* __restrict__ tile_count,
                                  uint4* __restrict__ clear, int64_t clear_vec,
                                  int32_t* __restrict__ bins, int K) {
  pdl_wait();
  pdl_trigger();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (BINS && i == 0) tile_count[kBinsWord] = K;
  for (int64_t v = i; v < clear_vec; v += (int64_t)gridDim.x * blockDim.x)
    clear[v] = make_uint4(0u, 0u, 0u, 0u);
  Splat s{};
  if (i < n) {
    s = pack_one(f.means, f.conics, f.colors, f.radii, f.opacities, i, frames.H, frames.W);
    store_splat(out + i, s);
  }
  count_pairs<CULL, BINS>(s, i < n, blockIdx.x * kThreads, ts, frames.tiles_x, 0, cutoff2,
                          tile_count, bins, K);
}

// Writes int32 offsets, checks capacity, then claims one slot per pair.  Slots are claimed by
// counting each tile's counter back down, which leaves the counters at zero.  A lane's own
// (small) rectangle claims all its slots first and stores afterwards, so the atomics overlap.
template <bool CULL>
__global__ void tile_fill_kernel(const Splat* __restrict__ rec, int64_t n, int ts, Frames frames,
                                 float cutoff2, int64_t T, const long long* __restrict__ off64,
                                 int* __restrict__ tile_count, int32_t* __restrict__ offsets32,
                                 int32_t* __restrict__ gids, int64_t cap, int* big_count,
                                 uint32_t* status, int K, int tests, int64_t gaussians) {
  pdl_wait();
  pdl_trigger();
  int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  long long total = off64[T];
  for (int64_t t = tid; t <= T; t += stride) {
    offsets32[t] = (int32_t)min(off64[t], 2147483647LL);
    if (t < T) note_overflow(off64[t + 1] - off64[t], t, frames, gaussians, K, tests, tile_count);
  }
  if (tid == 0) {
    *big_count = 0;
    if (total > 2147483647LL) raise_status(status, SS_STATUS_INDEX_INT32);
    if (total > cap) raise_status(status, SS_STATUS_INDEX_OVERFLOW);
  }
  long long pos[kSmallRect];
#pragma unroll
  for (int k = 0; k < kSmallRect; ++k) pos[k] = -1;
  int owner = -1;
  enumerate_pairs<CULL>(rec, tid, n, ts, frames, cutoff2, [&](int k, int g, int t) {
    long long p = off64[t] + (atomicSub(tile_count + (int64_t)t * kCounterStride, 1) - 1);
    if (k < 0) {
      if (p < cap) gids[p] = g;
    } else {
#pragma unroll
      for (int q = 0; q < kSmallRect; ++q)
        if (q == k) pos[q] = p;
      owner = g;
    }
  });
#pragma unroll
  for (int k = 0; k < kSmallRect; ++k)
    if (pos[k] >= 0 && pos[k] < cap) gids[pos[k]] = owner;
}

// Offsets of up to kScanMax tiles in one launch: each CTA sums the counters before its own 1,024
// (coalesced, one sector each, from L2) and scans its own, so no CTA waits for another.  8,161
// counters took 19 us and 13,297 took 26 us in one CTA, and take 6 us here (cold caches); up to
// 4,095 used to be scanned by the count's last CTA, but the fence and ticket that tells it so
// costs every CTA of the count more than this launch: 2 M Gaussians on 2,040 tiles 103 -> 85 us
// together, 100k on 1,024 tiles 16.9 -> 14.8 us.  The re-reads grow with the square of the tile
// count, hence CUB's device scan beyond kScanMax.
constexpr int kScanThreads = 1024;
constexpr int64_t kScanMax = 1 << 16;

__device__ __forceinline__ long long warp_inclusive(long long v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

__global__ void __launch_bounds__(kScanThreads)
    scan_counts_kernel(int* __restrict__ tile_count, int64_t items, long long* __restrict__ off64,
                       int32_t* __restrict__ off32, Frames frames, int64_t n, int K, int tests) {
  pdl_wait();
  pdl_trigger();
  __shared__ long long before[kScanThreads / 32], warp_total[kScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t first = (int64_t)blockIdx.x * kScanThreads, idx = first + tid;
  const long long own = idx < items ? tile_count[idx * kCounterStride] : 0;
  long long pre = 0;
#pragma unroll 4
  for (int64_t k = tid; k < first; k += kScanThreads) pre += tile_count[k * kCounterStride];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pre += __shfl_xor_sync(0xffffffffu, pre, o);
  const long long incl = warp_inclusive(own, lane);
  if (lane == 31) {
    before[warp] = pre;
    warp_total[warp] = incl;
  }
  __syncthreads();
  if (warp == 0) {
    long long b = before[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    const long long v = warp_total[lane];
    warp_total[lane] = b + warp_inclusive(v, lane) - v;  // offset of the warp's first counter
  }
  __syncthreads();
  if (idx < items) {
    const long long o = warp_total[warp] + (incl - own);
    off64[idx] = o;
    off32[idx] = (int32_t)(o < 2147483647LL ? o : 2147483647LL);
    if (idx + 1 < items) note_overflow(own, idx, frames, n, K, tests, tile_count);
  }
}

// Ascending sort of up to 32*K keys held in registers across a warp: key k of lane l is element
// 32k + l, missing elements are INT_MAX.  Standard bitonic network: at block size `size` and
// distance j, elements e and e^j are compared and the block (e & size) == 0 sorts upward.
// Distances below 32 exchange through xor shuffles, larger ones swap registers in-lane.
template <int K>
__device__ __forceinline__ void warp_bitonic(int (&v)[K], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int kp = k ^ (j >> 5);
          if (kp > k) {
            const bool up = ((32 * k + lane) & size) == 0;
            const int lo = min(v[k], v[kp]), hi = max(v[k], v[kp]);
            v[k] = up ? lo : hi;
            v[kp] = up ? hi : lo;
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int other = __shfl_xor_sync(0xffffffffu, v[k], j);
          const bool up = ((32 * k + lane) & size) == 0;
          const bool lower = (lane & j) == 0;
          v[k] = (up == lower) ? min(v[k], other) : max(v[k], other);
        }
      }
    }
  }
}

template <int K>
__device__ __forceinline__ void warp_sort_list(const int32_t* src, int32_t* g, int len, int lane) {
  int v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = 32 * k + lane < len ? src[32 * k + lane] : INT_MAX;
  warp_bitonic<K>(v, lane);
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (32 * k + lane < len) g[32 * k + lane] = v[k];
}

// One warp per tile: lists up to kWarpSortMax ids sort in registers (32 K keys for the smallest
// power-of-two K that holds the list); longer lists are queued for tile_sort_big_kernel.
__global__ void __launch_bounds__(kThreads) tile_sort_kernel(const int32_t* __restrict__ offsets,
                                                             int32_t* __restrict__ gids,
                                                             int64_t cap, int64_t T,
                                                             int* big_tiles, int* big_count) {
  pdl_wait();
  pdl_trigger();
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t t = (int64_t)blockIdx.x * (kThreads / 32) + warp;
  if (t >= T) return;
  int64_t lo = offsets[t], hi = offsets[t + 1];
  if (hi > cap) return;  // truncated list: the renderers scan all Gaussians for this tile
  int len = (int)(hi - lo);
  if (len <= 1) return;
  int32_t* g = gids + lo;
  if (len <= 32) {
    warp_sort_list<1>(g, g, len, lane);
  } else if (len <= 64) {
    warp_sort_list<2>(g, g, len, lane);
  } else if (len <= 128) {
    warp_sort_list<4>(g, g, len, lane);
  } else if (len <= 256) {
    warp_sort_list<8>(g, g, len, lane);
  } else if (len <= 512) {
    warp_sort_list<16>(g, g, len, lane);
  } else if (len <= kWarpSortMax) {
    warp_sort_list<32>(g, g, len, lane);
  } else if (lane == 0) {
    big_tiles[atomicAdd(big_count, 1)] = (int)t;
  }
}

// Long lists: one CTA per list, in shared memory up to kBigSortSmem ids, else in place.
// Lists of up to kRadixSortMax ids sort with CUB's block radix sort over the bits the ids need
// (key_bits: pad keys 2^bits - 1 sort last), with 2, 3 or 4 keys per thread, the fewest that
// hold the list (a radix sort's work grows with its keys, pads included); longer lists with the
// shared-memory bitonic network (the ids of a list are distinct, so every path gives the one
// ascending order).
constexpr int kRadixItems = 4;
constexpr int kRadixSortMax = 1024 * kRadixItems;
template <int K>
using BigRadixSortK = cub::BlockRadixSort<unsigned, 1024, K>;
union BigRadixTemp {
  typename BigRadixSortK<2>::TempStorage k2;
  typename BigRadixSortK<3>::TempStorage k3;
  typename BigRadixSortK<4>::TempStorage k4;
};

template <int K>
__device__ __forceinline__ void radix_sort_list(int32_t* __restrict__ g, int len, unsigned pad,
                                                int key_bits,
                                                typename BigRadixSortK<K>::TempStorage& tmp) {
  unsigned keys[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int e = threadIdx.x * K + i;
    keys[i] = e < len ? (unsigned)g[e] : pad;
  }
  BigRadixSortK<K>(tmp).Sort(keys, 0, key_bits);
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int e = threadIdx.x * K + i;
    if (e < len) g[e] = (int32_t)keys[i];
  }
}

__global__ void __launch_bounds__(1024) tile_sort_big_kernel(const int32_t* __restrict__ offsets,
                                                             int32_t* __restrict__ gids,
                                                             const int* __restrict__ big_tiles,
                                                             const int* __restrict__ big_count,
                                                             int key_bits) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ int sbuf[];
  __shared__ BigRadixTemp radix_temp;
  int count = *big_count;
  const unsigned pad = key_bits >= 32 ? 0xffffffffu : (1u << key_bits) - 1u;
  for (int k = blockIdx.x; k < count; k += gridDim.x) {
    int t = big_tiles[k];
    int64_t lo = offsets[t];
    int len = (int)(offsets[t + 1] - lo);
    auto sync = [] { __syncthreads(); };
    if (len <= 2 * 1024) {  // lists here are longer than the warp sort's 1,024 ids
      radix_sort_list<2>(gids + lo, len, pad, key_bits, radix_temp.k2);
    } else if (len <= 3 * 1024) {
      radix_sort_list<3>(gids + lo, len, pad, key_bits, radix_temp.k3);
    } else if (len <= kRadixSortMax) {
      radix_sort_list<4>(gids + lo, len, pad, key_bits, radix_temp.k4);
    } else if (len <= kBigSortSmem) {
      for (int e = threadIdx.x; e < len; e += blockDim.x) sbuf[e] = gids[lo + e];
      __syncthreads();
      sort_ascending(sbuf, len, threadIdx.x, blockDim.x, sync);
      for (int e = threadIdx.x; e < len; e += blockDim.x) gids[lo + e] = sbuf[e];
    } else {
      sort_ascending(gids + lo, len, threadIdx.x, blockDim.x, sync);
    }
    __syncthreads();
  }
}

// The binned index's second stage puts each bin's ids into ascending order.  The ids of a list are
// distinct, so there is one result whatever the way:
//
//   warp      short lists of a sparse tile set (see bin_sort_kernel): one warp's registers.
//   buckets   up to kSortIds ids: spread over about as many buckets of equal id width (128 to
//             1,024), each bucket finished by insertion, when no bucket holds more than kBucketIds.
//   windows   long lists and clustered ids (a field in Morton order, as decoded ones are, has a
//             tile's ids side by side): a bit per Gaussian of the image in shared memory, set from
//             the bin and read back in order, one window of ids after the other, windows without
//             ids skipped.  Costs the list plus 1/32 of the window, however the ids lie.
//   records   a tile whose bin overflowed with a good part of the image's Gaussians: the windows again,
//             set by testing every record of the image instead.
//   pairs     other tiles whose bin overflowed: place_overflow.
//
// Bound by latency (a few dependent L2 reads and block-wide steps per tile), hence small CTAs, 10 to
// an SM.  Lists of ~1,100 of 2 M ids on 2,040 tiles took 39 + 161 us in the warp and block sorts of
// the plain form, lists of ~2,000 of 250 k on 1,024 tiles 35 + 81 us; here 29 and 22 us.
constexpr int kSortThreads = 128;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kBuckets = 1024;
constexpr int kBucketIds = 24;
constexpr int kWindowWords = kSortIds + kBuckets;
static_assert(kWindowIds == 32 * kWindowWords, "one bitmap");
constexpr int kBitmapIds = 32 * kSortIds;      // a window below the bucket prefixes: 131,072

// Exclusive prefix of v over the CTA's threads (tmp: kSortWarps + 1 words, ends holding the total
// in tmp[kSortWarps]); holds two barriers.
__device__ __forceinline__ int block_exclusive(int v, int* tmp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();  // tmp may still be read from an earlier call
  if (lane == 31) tmp[warp] = incl;
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const int t = tmp[w];
    base += w < warp ? t : 0;
    total += t;
  }
  if (threadIdx.x == 0) tmp[kSortWarps] = total;
  return base + incl - v;
}

// Writes the ids of the set bits of words[0..nw) (bit b of word w is id first + 32 w + b) to g in
// ascending order (at most `room` of them) and returns their number.  An odd run of words per thread
// keeps the warp's reads on distinct banks.  Ends with a barrier.
__device__ __forceinline__ int emit_bits(const uint32_t* words, int nw, int first, int32_t* g,
                                         int room, int* tmp) {
  const int per = ((nw + kSortThreads - 1) / kSortThreads) | 1;
  const int w0 = min(nw, (int)threadIdx.x * per), w1 = min(nw, w0 + per);
  int c = 0;
  for (int w = w0; w < w1; ++w) c += __popc(words[w]);
  int at = block_exclusive(c, tmp);
  for (int w = w0; w < w1; ++w) {
    uint32_t x = words[w];
    while (x) {
      if (at < room) g[at] = first + 32 * w + __ffs(x) - 1;
      ++at;
      x &= x - 1;
    }
  }
  __syncthreads();
  return tmp[kSortWarps];
}

// A list that other CTAs have just placed: not to be read from the L1.
struct PlacedIds {
  const int32_t* p;
  __device__ __forceinline__ int operator[](int e) const { return __ldcg(p + e); }
};

// Orders a bin of len <= kSortIds ids by NB buckets of 2^shift ids and writes it to g; false,
// with nothing written and the buckets' prefixes in hist, when some bucket is too full (the bin may be
// g itself).  Called by every thread.
template <int NB, typename Bin>
__device__ __forceinline__ bool bucket_sort(Bin bin, int len, int first, int count, int* buf,
                                            int* hist, int* tmp, int32_t* g, int& shift) {
  constexpr int kOwn = NB / kSortThreads;
  shift = 0;
  while (((count - 1) >> shift) >= NB) ++shift;
#pragma unroll
  for (int k = 0; k < kOwn; ++k) hist[k * kSortThreads + threadIdx.x] = 0;
  __syncthreads();
  for (int e = threadIdx.x; e < len; e += kSortThreads)
    atomicAdd(&hist[(bin[e] - first) >> shift], 1);
  __syncthreads();
  int own[kOwn], sum = 0, most = 0;
#pragma unroll
  for (int k = 0; k < kOwn; ++k) {
    own[k] = hist[kOwn * threadIdx.x + k];
    sum += own[k];
    most = max(most, own[k]);
  }
  int at = block_exclusive(sum, tmp);
#pragma unroll
  for (int k = 0; k < kOwn; ++k) {
    hist[kOwn * threadIdx.x + k] = at;
    at += own[k];
  }
  at -= sum;
  if (!__syncthreads_and(most <= kBucketIds && len <= kSortIds)) return false;
  for (int e = threadIdx.x; e < len; e += kSortThreads) {
    const int id = bin[e];
    buf[atomicAdd(&hist[(id - first) >> shift], 1)] = id;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kOwn; ++k) {  // the thread's own buckets, each by insertion
    for (int x = at + 1; x < at + own[k]; ++x) {
      const int v = buf[x];
      int y = x;
      for (; y > at && buf[y - 1] > v; --y) buf[y] = buf[y - 1];
      buf[y] = v;
    }
    at += own[k];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < len; e += kSortThreads) g[e] = buf[e];
  return true;
}

// One tile by the whole CTA (see above).  Every thread calls it.
template <bool CULL>
__device__ __forceinline__ void cta_sort_bin(const Splat* __restrict__ rec, int64_t n, int ts,
                                          const Frames& frames, float cutoff2, int t,
                                          long long lo, int len, bool records,
                                          const int32_t* __restrict__ bin,
                                          int32_t* __restrict__ gids, uint32_t* smem, int* tmp) {
  const Frame fr = frame_of_tile(frames, t, n);
  const int first = fr.gauss_first, count = fr.gauss_count;
  int32_t* g = gids + lo;
  auto set_bit = [&](int rel) { atomicOr(&smem[rel >> 5], 1u << (rel & 31)); };
  auto clear = [&](int nw) {
    for (int w = threadIdx.x; w < nw; w += kSortThreads) smem[w] = 0u;
    __syncthreads();
  };
  if (records) {
    const int local = t - fr.first_tile;
    const int gx = local % fr.tiles_x, gy = local / fr.tiles_x;
    const int px0 = gx * ts, py0 = gy * ts;
    int done = 0;
    for (int w0 = 0; w0 < count; w0 += kWindowIds) {
      const int ids = min(count - w0, kWindowIds), nw = (ids + 31) >> 5;
      // a warp tests 32 consecutive records, whose ballot is the bitmap's word; eight words' loads in
      // flight
      constexpr int kWords = 8;
      for (int wa = threadIdx.x >> 5; wa < nw; wa += kWords * kSortWarps) {
        int4 b[kWords];
#pragma unroll
        for (int u = 0; u < kWords; ++u) {
          const int rel = 32 * (wa + u * kSortWarps) + (threadIdx.x & 31);
          b[u] = rel < ids ? reinterpret_cast<const int4*>(rec + first + w0 + rel)[3]
                           : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < kWords; ++u) {
          const int w = wa + u * kSortWarps;
          if (w >= nw) break;
          bool hit = b[u].z > b[u].x && b[u].w > b[u].y && b[u].x < px0 + ts && b[u].z > px0 &&
                     b[u].y < py0 + ts && b[u].w > py0;
          if (CULL && hit)
            hit = !culled(load_splat(rec, (int64_t)first + w0 + 32 * w + (threadIdx.x & 31)), gx, gy,
                          ts, cutoff2);
          const unsigned word = __ballot_sync(0xffffffffu, hit);
          if ((threadIdx.x & 31) == 0) smem[w] = word;
        }
      }
      __syncthreads();
      done += emit_bits(smem, nw, first + w0, g + done, len - done, tmp);
    }
    return;
  }
  int* buf = reinterpret_cast<int*>(smem);
  int* hist = buf + kSortIds;
  int shift = 0;
  if (len <= 128) {
    if (bucket_sort<128>(bin, len, first, count, buf, hist, tmp, g, shift)) return;
  } else if (len <= 256) {
    if (bucket_sort<256>(bin, len, first, count, buf, hist, tmp, g, shift)) return;
  } else if (len <= 512) {
    if (bucket_sort<512>(bin, len, first, count, buf, hist, tmp, g, shift)) return;
  } else {
    if (bucket_sort<kBuckets>(bin, len, first, count, buf, hist, tmp, g, shift)) return;
  }
  if (count <= kWindowIds) {  // one window
    __syncthreads();  // every thread has left the buckets
    const int nw = (count + 31) >> 5;
    clear(nw);
    for (int e = threadIdx.x; e < len; e += kSortThreads) set_bit(bin[e] - first);
    __syncthreads();
    emit_bits(smem, nw, first, g, len, tmp);
    return;
  }
  const int nb = ((count - 1) >> shift) + 1;  // buckets in use
  // windows of whole buckets; the bucket prefixes tell where each one's ids go.  The bitmap takes
  // the shared memory below the buckets.
  const int buckets = max(1, kBitmapIds >> shift);
  for (int b0 = 0; b0 < nb; b0 += buckets) {
    const int b1 = min(nb, b0 + buckets);
    const int beg = hist[b0], end = b1 < nb ? hist[b1] : len;
    if (beg == end) continue;  // the same in every thread
    // a bucket wider than the bitmap (few buckets, or very many Gaussians) is cut in pieces
    const int64_t r0 = (int64_t)b0 << shift, r1 = min((int64_t)count, (int64_t)b1 << shift);
    int done = beg;
    for (int64_t w0 = r0; w0 < r1; w0 += kBitmapIds) {
      const int ids = (int)min(r1 - w0, (int64_t)kBitmapIds), nw = (ids + 31) >> 5;
      clear(nw);
      for (int e = threadIdx.x; e < len; e += kSortThreads) {
        const int64_t rel = (int64_t)(bin[e] - first) - w0;
        if (rel >= 0 && rel < ids) set_bit((int)rel);
      }
      __syncthreads();
      done += emit_bits(smem, nw, first + (int)w0, g + done, len - done, tmp);
    }
  }
}

// Puts g[0, len), a list in arrival order, into ascending order: by buckets, or by windows of the ids as
// in cta_sort_bin, but in place: while a window's bits are set, the ids of later windows move to the end
// of the list, from its end on, and leave the room that the window's ids then take.  Every thread of the
// CTA calls it.
__device__ __noinline__ void sort_placed(int32_t* g, int len, int first, int count, uint32_t* smem,
                                         int* tmp) {
  const PlacedIds list{g};
  int* buf = reinterpret_cast<int*>(smem);
  int shift = 0;
  if (len <= 512) {
    if (bucket_sort<256>(list, len, first, count, buf, buf + kSortIds, tmp, g, shift)) return;
  } else if (len <= kSortIds) {
    if (bucket_sort<kBuckets>(list, len, first, count, buf, buf + kSortIds, tmp, g, shift)) return;
  }
  constexpr int kOwn = 8, kChunk = kOwn * kSortThreads;
  int done = 0;
  for (int w0 = 0; done < len && w0 < count; w0 += kWindowIds) {
    const int ids = min(count - w0, kWindowIds), nw = (ids + 31) >> 5;
    __syncthreads();  // every thread has left the buckets, or the window before
    for (int w = threadIdx.x; w < nw; w += kSortThreads) smem[w] = 0u;
    __syncthreads();
    int end = len;  // the ids of later windows start here
    for (int hi = len; hi > done; hi -= kChunk) {
      const int lo = max(done, hi - kChunk);
      int later[kOwn], num = 0;
#pragma unroll
      for (int u = 0; u < kOwn; ++u) {
        const int e = lo + u * kSortThreads + threadIdx.x;
        later[u] = e < hi ? list[e] : -1;
      }
#pragma unroll
      for (int u = 0; u < kOwn; ++u) {
        const int rel = later[u] - first - w0;
        if (later[u] >= 0 && rel < ids) {
          atomicOr(&smem[rel >> 5], 1u << (rel & 31));
          later[u] = -1;
        }
        num += later[u] >= 0;
      }
      if (w0 + ids == count) continue;  // the last window: nothing is later
      int at = block_exclusive(num, tmp);  // the chunk has been read
      __syncthreads();
      end -= tmp[kSortWarps];
#pragma unroll
      for (int u = 0; u < kOwn; ++u)
        if (later[u] >= 0) g[end + at++] = later[u];
    }
    __syncthreads();
    const int room = w0 + ids == count ? len - done : end - done;
    emit_bits(smem, nw, first + w0, g + done, room, tmp);
    done += room;
  }
}

// The tiles whose bins do not hold their lists.
struct Overflow {
  int K, tests;
  bool trusted;  // the bins belong to the counts
  __device__ __forceinline__ bool beyond(int64_t len) const { return len > K || !trusted; }
  __device__ __forceinline__ bool records(int64_t len, int64_t count) const {
    return listed_from_records(len, count, tests);
  }
};

// Places the ids of the tiles beyond their bins that listed_from_records leaves in their lists, by a
// cursor per tile: share `part` of `parts` of the pairs.  A warp takes `lanes` Gaussians at a time and
// shares their pairs evenly, four per lane in flight (it waits on the offsets and cursors in the L2).
template <bool CULL>
__device__ __noinline__ void place_overflow(const Splat* __restrict__ rec, int64_t n, int ts,
                                            const Frames& frames, float cutoff2,
                                            const long long* __restrict__ off64, int* tile_count,
                                            const Overflow over, int32_t* gids, int64_t cap,
                                            int part, int parts, int lanes) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)part * kSortWarps + (threadIdx.x >> 5);
  for (int64_t b = lanes * warp; b < n; b += (int64_t)lanes * parts * kSortWarps) {
    const int64_t i = b + lane;
    TileRect r{0, 0, 0, 0};
    int tiles_x = 0, first_tile = 0, images = 0;
    if (lane < lanes && i < n) {
      r = tile_rect_of(rec, i, ts);
      const Frame fr = frame_of_gaussian(frames, i, n);
      tiles_x = fr.tiles_x;
      first_tile = fr.first_tile;
      images = fr.gauss_count;
    }
    const int cnt = r.gw * r.gh;
    const int own = cnt > kHugeRect ? 0 : cnt;
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(all, incl, o);
      if (lane >= o) incl += v;
    }
    const int excl = incl - own, total = __shfl_sync(all, incl, 31);
    const int corner = first_tile + r.gy0 * tiles_x + r.gx0;
    // tile k of lane l's rectangle, its list's first slot and length; -1 when not placed here
    auto tile_of = [&](int l, unsigned k, bool some, long long& lo, int& len) {
      const unsigned gw = (unsigned)__shfl_sync(all, r.gw, l);
      const int tx = __shfl_sync(all, tiles_x, l), c = __shfl_sync(all, corner, l);
      const int count = __shfl_sync(all, images, l);
      const int gx0 = __shfl_sync(all, r.gx0, l), gy0 = __shfl_sync(all, r.gy0, l);
      if (!some) return -1;
      const int row = (int)(k / gw), col = (int)(k - (unsigned)row * gw);
      if (CULL && culled(load_splat(rec, b + l), gx0 + col, gy0 + row, ts, cutoff2)) return -1;
      const int t = c + row * tx + col;
      lo = off64[t];
      const long long hi = off64[t + 1];
      len = (int)(hi - lo);
      return hi > cap || !over.beyond(hi - lo) || over.records(hi - lo, count) ? -1 : t;
    };
    // a slot of tile t's list for every lane with t >= 0, one atomic for the lanes of a tile (these are
    // the tiles that many pairs share).  Every lane calls it.
    auto claim = [&](int t) {
      const unsigned peers = __match_any_sync(all, t);
      const int leader = __ffs(peers) - 1;
      int at = 0;
      if (t >= 0 && lane == leader)
        at = atomicAdd(tile_count + (int64_t)t * kCounterStride + kClaimWord, __popc(peers));
      return __shfl_sync(all, at, leader) + __popc(peers & ((1u << lane) - 1u));
    };
    constexpr int kPairs = 2;
    for (int e0 = 0; e0 < total; e0 += 32 * kPairs) {
      int t[kPairs], l[kPairs], len[kPairs], at[kPairs];
      long long lo[kPairs];
#pragma unroll
      for (int u = 0; u < kPairs; ++u) {
        const int e = e0 + 32 * u + lane;
        l[u] = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(all, excl, l[u] + step) <= e) l[u] += step;
        t[u] = tile_of(l[u], (unsigned)(e - __shfl_sync(all, excl, l[u])), e < total, lo[u], len[u]);
      }
#pragma unroll
      for (int u = 0; u < kPairs; ++u) at[u] = claim(t[u]);
#pragma unroll
      for (int u = 0; u < kPairs; ++u)
        if (t[u] >= 0 && at[u] < len[u]) gids[lo[u] + at[u]] = (int32_t)(b + l[u]);
    }
    for (unsigned huge = __ballot_sync(all, cnt > kHugeRect); huge; huge &= huge - 1) {
      const int l = __ffs(huge) - 1, tiles = __shfl_sync(all, cnt, l);
      for (int k0 = 0; k0 < tiles; k0 += 32) {
        long long lo;
        int len;
        const int t = tile_of(l, (unsigned)(k0 + lane), k0 + lane < tiles, lo, len);
        const int at = claim(t);
        if (t >= 0 && at < len) gids[lo + at] = (int32_t)(b + l);
      }
    }
  }
}

// Waits until `parts` shares are placed; false when they are not after about a second.  Every thread
// calls it.
constexpr int kPlacedPolls = 1 << 20;
__device__ __forceinline__ bool wait_placed(const int* placed, int parts) {
  bool ok = true;
  if (threadIdx.x == 0) {
    ok = false;
    for (int k = 0; k < kPlacedPolls && !ok; ++k) {
      int v;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(placed) : "memory");
      ok = v >= parts;
      if (!ok) __nanosleep(200);
    }
  }
  return __syncthreads_and(ok) != 0;
}

// Tiles per CTA: with up to kWarpTilesMax Gaussians per tile on average most lists are short, and a
// CTA takes four tiles, each warp sorting its own in registers (lists up to kWarpIds; bitonic, no
// block-wide step), longer ones then by the whole CTA in turn; beyond that one tile, by the CTA.
// Lists of ~210 on 1,024 and 8,160 tiles: 8.5 and 27 us one tile at a time, 6 and 16 us by fours.
constexpr int kWarpIds = 256;
constexpr int64_t kWarpTilesMax = 128;

// Where some bin overflowed, the CTAs number themselves as they start.  The first `parts` place the
// overflowing tiles' ids (place_overflow) and wait for nobody; the others take the tiles, and wait for
// the first before they sort the placed lists, which they share out singly.  So every wait is for CTAs
// that already run.  Count and fill of 100k Gaussians on 1024x1024: 41 px wide in 4-px tiles (lists of 180
// beside bins of 96) 0.58 ms, 0.27 in the plain form; 97 px in 16-px tiles (1,130 beside 832) 0.32 and
// 0.36; within 40 px of one point in 32-px tiles (10k beside 3,168) 0.14 and 0.17.  When all such tiles
// were tested against every record they took 19.0, 1.09 and 0.45 ms.
// Half the CTAs that the tiles need place pairs, between these numbers; only below twice the first does
// the grid have CTAs for it that leave at once otherwise (222 of them beside 256 cost 0.7 us).
constexpr int64_t kLeastParts = 74, kMostParts = 1184;

struct BinSort {
  const Splat* rec;
  int64_t n;
  int ts;
  float cutoff2;
  int64_t T;
  int tiles_per_cta, parts, lanes, tests;
  const long long* off64;
  int* tile_count;
  const int32_t* bins;
  int K;
  int32_t* gids;
  int64_t cap;
  uint32_t* status;
};

// Sorts the placed lists among tiles first, first + step, …; or lists those tiles from the records when
// their ids did not come.  Every thread calls it.
template <bool CULL>
__device__ __noinline__ void sort_placed_tiles(const BinSort& a, const Frames& frames,
                                               const Overflow over, bool placed, int64_t first,
                                               int64_t step, uint32_t* smem, int* tmp) {
  __shared__ int todo[kSortThreads], num_todo;
  for (int64_t base = first; base < a.T; base += step * kSortThreads) {
    if (threadIdx.x == 0) num_todo = 0;
    __syncthreads();
    const int64_t mine = base + step * threadIdx.x;
    if (mine < a.T) {
      const long long hi = a.off64[mine + 1], len = hi - a.off64[mine];
      if (hi <= a.cap && len > 0 && over.beyond(len) &&
          !over.records(len, frame_of_tile(frames, (int)mine, a.n).gauss_count))
        todo[atomicAdd(&num_todo, 1)] = (int)mine;
    }
    __syncthreads();
    const int count = num_todo;
    for (int k = 0; k < count; ++k) {
      const int t = todo[k];
      const long long lo = a.off64[t];
      const int len = (int)(a.off64[t + 1] - lo);
      const Frame fr = frame_of_tile(frames, t, a.n);
      if (placed)
        sort_placed(a.gids + lo, len, fr.gauss_first, fr.gauss_count, smem, tmp);
      else
        cta_sort_bin<CULL>(a.rec, a.n, a.ts, frames, a.cutoff2, t, lo, len, true, a.bins, a.gids,
                           smem, tmp);
      if (threadIdx.x == 0)
        a.tile_count[(int64_t)t * kCounterStride + kClaimWord] = 0;  // for another fill
      __syncthreads();
    }
  }
}

// Where the list of a warp's tile (with four to a CTA; else of the CTA's) begins and ends.
struct ListEnds {
  long long lo, hi;
};
__device__ __forceinline__ ListEnds ends_of(const BinSort& a, int64_t t0) {
  const int64_t t = t0 + (a.tiles_per_cta > 1 ? threadIdx.x >> 5 : 0);
  return t < a.T ? ListEnds{__ldg(a.off64 + t), __ldg(a.off64 + t + 1)} : ListEnds{0, 0};
}

// Sorts the tiles_per_cta tiles from t0 on, but for those that place_overflow lists (`some` of them).
template <bool CULL>
__device__ __forceinline__ void sort_tiles(const BinSort& a, const Frames& frames, int64_t t0,
                                           const ListEnds& ends, const Overflow& over, bool some,
                                           uint32_t* smem, int* tmp) {
  if (a.tiles_per_cta > 1) {
    const int lane = threadIdx.x & 31;
    const int64_t t = t0 + (threadIdx.x >> 5);
    bool mine = false;  // the CTA takes the tile
    if (t < a.T) {
      const long long lo = ends.lo, hi = ends.hi;
      const int len = (int)(hi - lo);
      if (hi <= a.cap && len > 0) {  // else truncated: the renderers scan all Gaussians
        mine = len > kWarpIds || over.beyond(len);
        if (!mine) {
          const int32_t* bin = a.bins + t * a.K;
          int32_t* g = a.gids + lo;
          if (len <= 32)
            warp_sort_list<1>(bin, g, len, lane);
          else if (len <= 64)
            warp_sort_list<2>(bin, g, len, lane);
          else if (len <= 128)
            warp_sort_list<4>(bin, g, len, lane);
          else
            warp_sort_list<8>(bin, g, len, lane);
        }
      }
    }
    if (!__syncthreads_or(mine)) return;
  }
  for (int u = 0; u < a.tiles_per_cta; ++u) {
    const int64_t t = t0 + u;
    if (t >= a.T) break;
    const bool one = a.tiles_per_cta == 1;
    const long long lo = one ? ends.lo : __ldg(a.off64 + t);
    const long long hi = one ? ends.hi : __ldg(a.off64 + t + 1);
    const int len = (int)(hi - lo);  // at most the image's Gaussians
    if (hi > a.cap || len == 0) continue;
    const bool beyond = over.beyond(len);
    if (a.tiles_per_cta > 1 && len <= kWarpIds && !beyond) continue;  // a warp has sorted it
    if (some && beyond && !over.records(len, frame_of_tile(frames, (int)t, a.n).gauss_count)) continue;
    cta_sort_bin<CULL>(a.rec, a.n, a.ts, frames, a.cutoff2, (int)t, lo, len, beyond,
                       a.bins + t * a.K, a.gids, smem, tmp);
    __syncthreads();
  }
}

// The kernel where some tile's ids are to be placed.
template <bool CULL>
__device__ __noinline__ void sort_and_place(const BinSort& a, const Frames& frames, bool trusted,
                                            uint32_t* smem, int* tmp) {
  const Overflow over{a.K, a.tests, trusted};
  if (threadIdx.x == 0) tmp[0] = atomicAdd(a.tile_count + kTicketWord, 1);
  __syncthreads();
  const int number = tmp[0] - a.parts, tile_ctas = (int)gridDim.x - a.parts;
  __syncthreads();
  if (number < 0) {
    place_overflow<CULL>(a.rec, a.n, a.ts, frames, a.cutoff2, a.off64, a.tile_count, over, a.gids,
                         a.cap, number + a.parts, a.parts, a.lanes);
    __threadfence();  // the ids before the word that tells of them
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(a.tile_count + kPlacedWord, 1);
  } else {
    for (int64_t t0 = (int64_t)number * a.tiles_per_cta; t0 < a.T;
         t0 += (int64_t)tile_ctas * a.tiles_per_cta)
      sort_tiles<CULL>(a, frames, t0, ends_of(a, t0), over, true, smem, tmp);
    const bool placed = wait_placed(a.tile_count + kPlacedWord, a.parts);
    if (!placed && threadIdx.x == 0)
      raise_status(a.status, SS_STATUS_INDEX_OVERFLOW);  // late ids may spoil a list
    sort_placed_tiles<CULL>(a, frames, over, placed, number, tile_ctas, smem, tmp);
  }
  __syncthreads();
  // the last CTA leaves the tickets as they were, for another fill of these counts
  if (threadIdx.x == 0 && atomicAdd(a.tile_count + kExitWord, 1) == (int)gridDim.x - 1)
    a.tile_count[kTicketWord] = a.tile_count[kPlacedWord] = a.tile_count[kExitWord] = 0;
}

template <bool CULL>
__global__ void __launch_bounds__(kSortThreads, 7)
    bin_sort_kernel(__grid_constant__ const BinSort a, __grid_constant__ const Frames frames) {
  pdl_wait();
  pdl_trigger();
  __shared__ __align__(16) uint32_t smem[kWindowWords];  // a bitmap, or ids and buckets
  __shared__ int tmp[kSortWarps + 1];
  const int64_t t0 = (int64_t)blockIdx.x * a.tiles_per_cta;
  const ListEnds ends = ends_of(a, t0);  // on their way while the words below are
  const bool trusted = a.tile_count[kBinsWord] == a.K;  // the bins belong to these counts
  const bool place = a.parts > 0 && (!trusted || a.tile_count[kOverflowWord] != 0);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const long long total = a.off64[a.T];
    if (total > 2147483647LL) raise_status(a.status, SS_STATUS_INDEX_INT32);
    if (total > a.cap) raise_status(a.status, SS_STATUS_INDEX_OVERFLOW);
  }
  if (place) {
    sort_and_place<CULL>(a, frames, trusted, smem, tmp);
    return;
  }
  if (t0 < a.T) sort_tiles<CULL>(a, frames, t0, ends, Overflow{a.K, 0, trusted}, false, smem, tmp);
}

// Bits that hold every id below n and the pad 2^bits - 1 above them.
int sort_key_bits(int64_t n) {
  int b = 1;
  while (b < 32 && ((int64_t)1 << b) <= n) ++b;
  return b;
}

constexpr int kBigSortCtas = 296;  // 2 per SM: long lists are common under heavy-tailed fields

// Opts tile_sort_big_kernel into its dynamic shared memory once per device.
int allow_big_sort_smem() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return check_launch("cudaGetDevice");
  if (dev >= 0 && dev < 64 && done[dev]) return SS_OK;
  if (cudaFuncSetAttribute(tile_sort_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kBigSortSmem * sizeof(int))) != cudaSuccess)
    return check_launch("tile_sort_big smem attribute");
  if (dev >= 0 && dev < 64) done[dev] = true;
  return SS_OK;
}

int check_index_args(int64_t n, int H, int W, int ts) {
  if (n < 0 || H < 0 || W < 0) return fail(SS_ERR_INVALID_ARGUMENT, "negative size");
  if (n > (int64_t)INT32_MAX) return fail(SS_ERR_INVALID_ARGUMENT, "n exceeds int32 ids");
  if (ts <= 0 || ts > 32)  // ts^2 <= 1024, without overflow
    return fail(SS_ERR_INVALID_ARGUMENT, "tile_size must be positive with tile_size^2 <= 1024");
  TileGrid g = make_grid(H, W, ts);
  if (g.T + 1 > (int64_t)INT32_MAX)
    return fail(SS_ERR_INVALID_ARGUMENT, "tile grid exceeds int32 tile ids");
  return SS_OK;
}


// Stage 1 over any tile set (one image or a batch): counts, scan, int32 offsets.
// With `rs`, the records are first projected from that RS field in the same kernel
// (project_count_kernel) and written to `records`; with `pk` (one image) packed from those inputs.
int index_count(const Frames& frames, int ts, int64_t T, const void* records, int64_t n,
                int ellipse_cull, float sigma_cutoff, int32_t* tile_offsets, void* workspace,
                size_t workspace_bytes, uint32_t* status, ss_stream_t stream,
                const RSField* rs = nullptr, void* clear = nullptr, size_t clear_bytes = 0,
                const PackField* pk = nullptr) {
  int rc;
  if (!tile_offsets || !workspace) return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  if (n > 0 && !records) return fail(SS_ERR_INVALID_ARGUMENT, "null records");
  if (workspace_bytes < index_workspace_bytes(T))
    return fail(SS_ERR_INVALID_ARGUMENT, "tile index workspace too small (%zu < %zu)",
                workspace_bytes, index_workspace_bytes(T));
  cudaStream_t s = as_stream(stream);
  IndexWorkspace w = carve(workspace, workspace_bytes, n, T);
  if (cudaMemsetAsync(w.tile_count, 0, sizeof(int) * kCounterStride * (T + 1), s) !=
      cudaSuccess)
    return check_launch("tile_index_count memset");
  const Splat* rec = static_cast<const Splat*>(records);
  float cutoff2 = sigma_cutoff * sigma_cutoff;
  const bool one_scan = T + 1 <= kScanMax;
  const bool binned = w.bins != nullptr;
  if (clear_bytes && (!clear || reinterpret_cast<uintptr_t>(clear) % 16 || clear_bytes % 16))
    return fail(SS_ERR_INVALID_ARGUMENT,
                "clear region must be 16-byte aligned and a multiple of 16 bytes");
  if (clear_bytes && !((rs || pk) && n > 0) && cudaMemsetAsync(clear, 0, clear_bytes, s) != cudaSuccess)
    return check_launch("clear region memset");
  if (pk && n > 0) {  // pack even when the tile set is empty: the records are an output
    if (reinterpret_cast<uintptr_t>(records) % 16)
      return fail(SS_ERR_INVALID_ARGUMENT, "records must be 16-byte aligned");
    int blocks = (int)((n + kThreads - 1) / kThreads);
    Splat* out = static_cast<Splat*>(const_cast<void*>(records));
#define SS_KCOUNT(C, B)                                                                       \
  launch("pack_count_kernel", pack_count_kernel<C, B>, blocks, kThreads, 0, s, *pk, n, ts,      \
         frames, cutoff2, out, w.tile_count, static_cast<uint4*>(clear),                      \
         (int64_t)(clear_bytes / 16), w.bins, w.bin_ids)
    if (ellipse_cull) {
      if (binned) SS_KCOUNT(true, true); else SS_KCOUNT(true, false);
    } else {
      if (binned) SS_KCOUNT(false, true); else SS_KCOUNT(false, false);
    }
#undef SS_KCOUNT
    if ((rc = check_launch("pack_count"))) return rc;
  } else if (rs && n > 0) {  // project even when the tile set is empty
    if (reinterpret_cast<uintptr_t>(records) % 16)
      return fail(SS_ERR_INVALID_ARGUMENT, "records must be 16-byte aligned");
    int blocks = (int)((n + kThreads - 1) / kThreads);
    Splat* out = static_cast<Splat*>(const_cast<void*>(records));
#define SS_PCOUNT(C, B)                                                                       \
  launch("project_count_kernel", project_count_kernel<C, B>, blocks, kThreads, 0, s, *rs, n,   \
         ts, frames, cutoff2, out, w.tile_count, static_cast<uint4*>(clear),                  \
         (int64_t)(clear_bytes / 16), w.bins, w.bin_ids)
    if (ellipse_cull) {
      if (binned) SS_PCOUNT(true, true); else SS_PCOUNT(true, false);
    } else {
      if (binned) SS_PCOUNT(false, true); else SS_PCOUNT(false, false);
    }
#undef SS_PCOUNT
    if ((rc = check_launch("project_count"))) return rc;
  } else if (n > 0 && T > 0) {
    int blocks = (int)((n + kThreads - 1) / kThreads);
#define SS_COUNT(C, B)                                                                        \
  launch("tile_count_kernel", tile_count_kernel<C, B>, blocks, kThreads, 0, s, rec, n, ts,      \
         frames, cutoff2, w.tile_count, w.bins, w.bin_ids)
    if (ellipse_cull) {
      if (binned) SS_COUNT(true, true); else SS_COUNT(true, false);
    } else {
      if (binned) SS_COUNT(false, true); else SS_COUNT(false, false);
    }
#undef SS_COUNT
    if ((rc = check_launch("tile_count"))) return rc;
  }
  (void)status;
  if (one_scan) {
    launch("scan_counts_kernel", scan_counts_kernel,
           (unsigned)((T + kScanThreads) / kScanThreads), kScanThreads, 0, s, w.tile_count, T + 1,
           w.offsets64, tile_offsets, frames, n, w.bin_ids, index_tests(n, T));
    return check_launch("tile_offsets scan");
  }
  size_t sb = w.scan_bytes;
  cudaError_t e = cub::DeviceScan::ExclusiveScan(w.scan_temp, sb, counter_iter(w.tile_count),
                                                 w.offsets64,
                                                 ::cuda::std::plus<long long>(), (long long)0,
                                                 (int)(T + 1), s);
  if (e != cudaSuccess) return fail(SS_ERR_CUDA, "tile offsets scan: %s", cudaGetErrorString(e));
  // int32 offsets for callers that only run stage 1 (the fill rewrites them identically).
  launch("tile_fill_kernel", tile_fill_kernel<false>, (int)((T + 1 + kThreads - 1) / kThreads), kThreads, 0, s, 
      rec, 0, ts, frames, cutoff2, T, w.offsets64, w.tile_count, tile_offsets, nullptr,
      INT64_MAX, w.big_count, nullptr, w.bin_ids, index_tests(n, T), n);
  return check_launch("tile_offsets");
}

// Stage 2 over any tile set: fill, per-tile sort.
int index_fill(const Frames& frames, int ts, int64_t T, const void* records, int64_t n,
               int ellipse_cull, float sigma_cutoff, const int32_t* tile_offsets,
               int32_t* tile_gids, int64_t gid_capacity, void* workspace,
               size_t workspace_bytes, uint32_t* status, ss_stream_t stream) {
  int rc;
  if (!tile_offsets || !workspace) return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  if (gid_capacity < 0) return fail(SS_ERR_INVALID_ARGUMENT, "negative gid capacity");
  if (gid_capacity > 0 && !tile_gids) return fail(SS_ERR_INVALID_ARGUMENT, "null tile_gids");
  if (workspace_bytes < index_workspace_bytes(T))
    return fail(SS_ERR_INVALID_ARGUMENT, "tile index workspace too small");
  if (T == 0) return SS_OK;
  cudaStream_t s = as_stream(stream);
  IndexWorkspace w = carve(workspace, workspace_bytes, n, T);
  const Splat* rec = static_cast<const Splat*>(records);
  float cutoff2 = sigma_cutoff * sigma_cutoff;
  if (w.bins) {  // the count left every tile's ids in its bin
    const int per = n <= kWarpTilesMax * T ? kSortWarps : 1;
    const int64_t ctas = (T + per - 1) / per;
    const int tests = index_tests(n, T);
    int64_t parts = ctas / 2 < kMostParts ? ctas / 2 : kMostParts;
    if (parts < kLeastParts) parts = kLeastParts;
    int lanes = 32;  // a warp's Gaussians at a time
    while (lanes > 1 && n < parts * kSortWarps * lanes) lanes >>= 1;
    const int64_t share = (n + lanes * kSortWarps - 1) / (lanes * kSortWarps);
    if (share < parts) parts = share;
    if (tests == INT_MAX) parts = 0;  // all from the records: nothing is placed
    const int64_t least = parts ? parts + (ctas < kLeastParts ? ctas : kLeastParts) : 0;
    const BinSort a{rec, n, ts, cutoff2, T, per, (int)parts, lanes, tests, w.offsets64,
                    w.tile_count, w.bins, w.bin_ids, tile_gids, gid_capacity, status};
    // the tile kernels that follow take all the shared memory there is (a fit step of 20k Gaussians on
    // 640x480: 51 us with the same split here, 59 without)
    const auto kern = ellipse_cull ? bin_sort_kernel<true> : bin_sort_kernel<false>;
    if ((rc = prefer_shared_memory(reinterpret_cast<const void*>(kern)))) return rc;
    launch("bin_sort_kernel", kern, (unsigned)(ctas > least ? ctas : least), kSortThreads, 0, s, a,
           frames);
    return check_launch("bin_sort");
  }
  int64_t threads_needed = n > T + 1 ? n : T + 1;
  int blocks = (int)((threads_needed + kThreads - 1) / kThreads);
  int32_t* offsets32 = const_cast<int32_t*>(tile_offsets);
  if (ellipse_cull)
    launch("tile_fill_kernel", tile_fill_kernel<true>, blocks, kThreads, 0, s, rec, n, ts, frames, cutoff2, T,
                                                       w.offsets64, w.tile_count, offsets32,
                                                       tile_gids, gid_capacity, w.big_count,
                                                       status, 0, 0, n);
  else
    launch("tile_fill_kernel", tile_fill_kernel<false>, blocks, kThreads, 0, s, rec, n, ts, frames, cutoff2, T,
                                                        w.offsets64, w.tile_count, offsets32,
                                                        tile_gids, gid_capacity, w.big_count,
                                                        status, 0, 0, n);
  if ((rc = check_launch("tile_fill"))) return rc;
  int sort_blocks = (int)((T + (kThreads / 32) - 1) / (kThreads / 32));
  launch("tile_sort_kernel", tile_sort_kernel, sort_blocks, kThreads, 0, s, tile_offsets, tile_gids, gid_capacity, T,
                                                     w.big_tiles, w.big_count);
  if ((rc = check_launch("tile_sort"))) return rc;
  if ((rc = allow_big_sort_smem())) return rc;
  launch("tile_sort_big_kernel", tile_sort_big_kernel, kBigSortCtas, 1024,
         kBigSortSmem * sizeof(int), s, tile_offsets, tile_gids, w.big_tiles, w.big_count,
         sort_key_bits(n));
  return check_launch("tile_sort_big");
}

}  // namespace
}  // namespace ss

using namespace ss;

extern "C" {

int ss_tile_index_workspace_bytes(int64_t n, int height, int width, int tile_size,
                                  size_t* bytes) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  if (!bytes) return fail(SS_ERR_INVALID_ARGUMENT, "null bytes pointer");
  *bytes = index_workspace_bytes(make_grid(height, width, tile_size).T);
  return SS_OK;
}

int ss_tile_index_binned_workspace_bytes(int64_t n, int height, int width, int tile_size,
                                         size_t* bytes) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  if (!bytes) return fail(SS_ERR_INVALID_ARGUMENT, "null bytes pointer");
  *bytes = binned_workspace_bytes(n, make_grid(height, width, tile_size).T);
  return SS_OK;
}

int ss_tile_index_entries_workspace_bytes(int64_t n, int64_t tiles, int images, int64_t entries,
                                          size_t* bytes) {
  if (n < 0 || tiles < 0 || images < 0 || entries < 0)
    return fail(SS_ERR_INVALID_ARGUMENT, "negative size");
  if (!bytes) return fail(SS_ERR_INVALID_ARGUMENT, "null bytes pointer");
  *bytes = prefer_plain(n, tiles, images, entries) ? index_workspace_bytes(tiles)
                                                    : binned_workspace_bytes(n, tiles);
  return SS_OK;
}

int ss_batch_tile_index_binned_workspace_bytes(const ss_batch* batch, int64_t n, size_t* bytes) {
  Frames f;
  int rc = frames_of_batch(batch, n, &f);
  if (rc) return rc;
  if (!bytes) return fail(SS_ERR_INVALID_ARGUMENT, "null bytes pointer");
  *bytes = binned_workspace_bytes(n, batch->tiles);
  return SS_OK;
}

int ss_batch_tile_index_workspace_bytes(const ss_batch* batch, int64_t n, size_t* bytes) {
  Frames f;
  int rc = frames_of_batch(batch, n, &f);
  if (rc) return rc;
  if (!bytes) return fail(SS_ERR_INVALID_ARGUMENT, "null bytes pointer");
  *bytes = index_workspace_bytes(batch->tiles);
  return SS_OK;
}

int ss_tile_index_count(const void* records, int64_t n, int height, int width, int tile_size,
                        int ellipse_cull, float sigma_cutoff, int32_t* tile_offsets,
                        void* workspace, size_t workspace_bytes, uint32_t* status,
                        ss_stream_t stream) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  return index_count(single_frame(height, width, tile_size), tile_size,
                     make_grid(height, width, tile_size).T, records, n, ellipse_cull,
                     sigma_cutoff, tile_offsets, workspace, workspace_bytes, status, stream);
}

int ss_batch_tile_index_count(const ss_batch* batch, const void* records, int64_t n,
                              int ellipse_cull, float sigma_cutoff, int32_t* tile_offsets,
                              void* workspace, size_t workspace_bytes, uint32_t* status,
                              ss_stream_t stream) {
  Frames f;
  int rc = frames_of_batch(batch, n, &f);
  if (rc) return rc;
  return index_count(f, batch->tile_size, batch->tiles, records, n, ellipse_cull, sigma_cutoff,
                     tile_offsets, workspace, workspace_bytes, status, stream);
}

int ss_project_rs_index_count(const float* means, const float* log_scales,
                              const float* rotations, const float* colors,
                              const float* opacity_logits, int64_t n, float dilation,
                              float sigma_cutoff, int height, int width, int tile_size,
                              int ellipse_cull, void* records, int32_t* tile_offsets,
                              void* workspace, size_t workspace_bytes, void* clear,
                              size_t clear_bytes, uint32_t* status, ss_stream_t stream) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  if (n > 0 && (!means || !log_scales || !rotations || !colors))
    return fail(SS_ERR_INVALID_ARGUMENT, "null RS field pointer");
  if (!(dilation >= 0.0f)) return fail(SS_ERR_INVALID_ARGUMENT, "dilation must be >= 0");
  const RSField f{means, log_scales, rotations, colors, opacity_logits, dilation, sigma_cutoff};
  return index_count(single_frame(height, width, tile_size), tile_size,
                     make_grid(height, width, tile_size).T, records, n, ellipse_cull,
                     sigma_cutoff, tile_offsets, workspace, workspace_bytes, status, stream, &f,
                     clear, clear_bytes);
}

int ss_pack_splats_index_count(const float* means, const float* conics, const float* colors,
                               const int64_t* radii, const float* opacities, int64_t n,
                               int height, int width, int tile_size, int ellipse_cull,
                               float sigma_cutoff, void* records, int32_t* tile_offsets,
                               void* workspace, size_t workspace_bytes, void* clear,
                               size_t clear_bytes, uint32_t* status, ss_stream_t stream) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  if (n > 0 && (!means || !conics || !colors || !radii))
    return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  const PackField f{means, conics, colors, radii, opacities};
  return index_count(single_frame(height, width, tile_size), tile_size,
                     make_grid(height, width, tile_size).T, records, n, ellipse_cull,
                     sigma_cutoff, tile_offsets, workspace, workspace_bytes, status, stream,
                     nullptr, clear, clear_bytes, &f);
}

int ss_batch_project_rs_index_count(const ss_batch* batch, const float* means,
                                    const float* log_scales, const float* rotations,
                                    const float* colors, const float* opacity_logits, int64_t n,
                                    float dilation, float sigma_cutoff, int ellipse_cull,
                                    void* records, int32_t* tile_offsets, void* workspace,
                                    size_t workspace_bytes, void* clear, size_t clear_bytes,
                                    uint32_t* status, ss_stream_t stream) {
  Frames fr;
  int rc = frames_of_batch(batch, n, &fr);
  if (rc) return rc;
  if (n > 0 && (!means || !log_scales || !rotations || !colors))
    return fail(SS_ERR_INVALID_ARGUMENT, "null RS field pointer");
  if (!(dilation >= 0.0f)) return fail(SS_ERR_INVALID_ARGUMENT, "dilation must be >= 0");
  const RSField f{means, log_scales, rotations, colors, opacity_logits, dilation, sigma_cutoff};
  return index_count(fr, batch->tile_size, batch->tiles, records, n, ellipse_cull, sigma_cutoff,
                     tile_offsets, workspace, workspace_bytes, status, stream, &f, clear,
                     clear_bytes);
}

int ss_tile_index_fill(const void* records, int64_t n, int height, int width, int tile_size,
                       int ellipse_cull, float sigma_cutoff, const int32_t* tile_offsets,
                       int32_t* tile_gids, int64_t gid_capacity, void* workspace,
                       size_t workspace_bytes, uint32_t* status, ss_stream_t stream) {
  int rc = check_index_args(n, height, width, tile_size);
  if (rc) return rc;
  return index_fill(single_frame(height, width, tile_size), tile_size,
                    make_grid(height, width, tile_size).T, records, n, ellipse_cull,
                    sigma_cutoff, tile_offsets, tile_gids, gid_capacity, workspace,
                    workspace_bytes, status, stream);
}

int ss_batch_tile_index_fill(const ss_batch* batch, const void* records, int64_t n,
                             int ellipse_cull, float sigma_cutoff, const int32_t* tile_offsets,
                             int32_t* tile_gids, int64_t gid_capacity, void* workspace,
                             size_t workspace_bytes, uint32_t* status, ss_stream_t stream) {
  Frames f;
  int rc = frames_of_batch(batch, n, &f);
  if (rc) return rc;
  return index_fill(f, batch->tile_size, batch->tiles, records, n, ellipse_cull, sigma_cutoff,
                    tile_offsets, tile_gids, gid_capacity, workspace, workspace_bytes, status,
                    stream);
}

}  // extern "C"
