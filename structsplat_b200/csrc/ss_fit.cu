// Update of a fit iteration.  Per Gaussian: the render backward's summed moments become conic / mean /
// colour / opacity gradients and the chain rule carries them to the RS field parameters
// (gaussians.py:270-300); the moment accumulators are zeroed for the next iteration.  Per parameter
// element: one Adam step over the five parameter tensors, then the clamp of the log-scales that the
// reference's fit loop applies after opt.step() (fit.py:3033, 3359-3366).
//
// Two passes, fit_grad_kernel and adam_kernel: the gradients pass through the fit workspace, so the
// Adam pass streams four aligned arrays per tensor at full occupancy, as torch's multi-tensor Adam
// does.  Small fields, where a launch counts for more than the traffic, take one,
// fit_update_kernel (see there).
//
// Adam is torch.optim.Adam's multi-tensor step (no weight decay, no amsgrad), element by element:
//   m <- lerp(m, g, 1 - beta1)            = m + (1 - beta1)(g - m)
//   v <- v beta2 + (1 - beta2) g^2
//   p <- p - lr / (1 - beta1^t) * m / (sqrt(v) / sqrt(1 - beta2^t) + eps)
// with the step-dependent factors formed in double and rounded to float as torch's Python-side
// scalars are, so the update reproduces the eager optimizer.
//
// The step count lives on the device (step_state[0]) so the update can be replayed from a CUDA
// graph: every thread of the Adam pass uses t = step_state[0] + 1 and its last CTA to finish
// stores t back (step_state[1] counts finished CTAs and is reset by that CTA).
#include "ss_common.cuh"

namespace ss {
namespace {

constexpr int kThreads = 256;

struct AdamHyper {
  double lr[5];  // means, log_scales, rotations, colors, opacity logits
  double beta1, beta2;
  float eps;
  float log_lo;
  float dilation;
};

struct FieldPtrs {
  float *means, *log_scales, *rotations, *colors, *logits;
};

struct AdamStep {
  float w1, b2, s2, bc2s, eps;  // lerp weight, beta2, 1 - beta2, sqrt(1 - beta2^t), eps
  double bc1;                    // 1 - beta1^t
};

__device__ __forceinline__ float adam(float p, float g, float& m, float& v, float step,
                                      const AdamStep& a) {
  m = fmaf(a.w1, g - m, m);
  v = fmaf(a.s2, g * g, v * a.b2);
  const float denom = sqrtf(v) / a.bc2s + a.eps;
  return fmaf(-step, m / denom, p);
}

// Inputs of one Gaussian's gradients: its nine summed moments, the record's opacity and conic,
// and the current log-scales, rotation and opacity logit.
struct GradIn {
  float m[kMoments];
  float op, a, b, c, ls0, ls1, th, lg;
};

__device__ __forceinline__ void load_grad_in(const Splat* __restrict__ rec,
                                             const float* __restrict__ log_scales,
                                             const float* __restrict__ rotations,
                                             const float* __restrict__ logits, int64_t g,
                                             GradIn& in) {
  const float4 p1 = reinterpret_cast<const float4*>(rec + g)[1];
  const float4 p2 = reinterpret_cast<const float4*>(rec + g)[2];
  in.op = p1.y;
  in.a = p2.y;
  in.b = p2.z;
  in.c = p2.w;
  in.ls0 = log_scales[2 * g];
  in.ls1 = log_scales[2 * g + 1];
  in.th = rotations[g];
  in.lg = logits ? logits[g] : 0.f;
}

// The same arithmetic as the plain backward epilogue, then the RS chain rule.
__device__ __forceinline__ void store_grads(const GradIn& in, int64_t g, float dilation,
                                            bool has_logits, const FieldPtrs& grad) {
  const float* m = in.m;
  float gls0, gls1, grot;
  rs_conic_chain(in.ls0, in.ls1, in.th, dilation, -0.5f * in.op * m[6], -in.op * m[7],
                 -0.5f * in.op * m[8], gls0, gls1, grot);
  grad.means[2 * g] = in.op * (in.a * m[4] + in.b * m[5]);
  grad.means[2 * g + 1] = in.op * (in.b * m[4] + in.c * m[5]);
  grad.log_scales[2 * g] = gls0;
  grad.log_scales[2 * g + 1] = gls1;
  grad.rotations[g] = grot;
  grad.colors[3 * g] = in.op * m[0];
  grad.colors[3 * g + 1] = in.op * m[1];
  grad.colors[3 * g + 2] = in.op * m[2];
  if (has_logits) grad.logits[g] = logit_chain(in.lg, m[3]);
}

// Per-Gaussian gradients of the five parameter groups: the summed moments (fast: the atomic
// accumulators, read and zeroed; deterministic: the entry partials in their fixed order) become
// render-input gradients, and the chain rule carries them to the RS parameters at their current
// values.  Grid-stride, a warp's 32 consecutive Gaussians per round (the deterministic sum is
// warp-collective); fast mode takes two rounds at a time with every load issued before the first
// store, so each thread keeps two Gaussians' loads in flight.  The gradients go to tensors shaped
// like the parameters.
template <bool DETERMINISTIC>
__global__ void __launch_bounds__(kThreads)
    fit_grad_kernel(const Splat* __restrict__ rec, int64_t n, float* __restrict__ moments,
                    const float* __restrict__ partials, const int32_t* __restrict__ order,
                    const int32_t* __restrict__ seg, const float* __restrict__ log_scales,
                    const float* __restrict__ rotations, const float* __restrict__ logits,
                    float dilation, FieldPtrs grad) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x - lane);
  if constexpr (DETERMINISTIC) {
    for (int64_t base = first; base < n; base += stride) {
      const int64_t g = base + lane;
      const bool active = g < n;
      GradIn in;
      sum_entry_partials(partials, order, seg, n, g, active, in.m);
      if (!active) continue;
      load_grad_in(rec, log_scales, rotations, logits, g, in);
      store_grads(in, g, dilation, logits != nullptr, grad);
    }
  } else {
  for (int64_t base = first; base < n; base += 2 * stride) {
    const int64_t g[2] = {base + lane, base + stride + lane};
    GradIn in[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (g[u] >= n) continue;
#pragma unroll
      for (int k = 0; k < kMoments; ++k) in[u].m[k] = moments[k * n + g[u]];
      load_grad_in(rec, log_scales, rotations, logits, g[u], in[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (g[u] >= n) continue;
#pragma unroll
      for (int k = 0; k < kMoments; ++k) moments[k * n + g[u]] = 0.0f;
      store_grads(in[u], g[u], dilation, logits != nullptr, grad);
    }
  }
  }
}

// One parameter tensor of the Adam step: parameters, both moments, gradient and length; its
// position in AdamTensors is its learning-rate group.
struct AdamTensor {
  float *p, *m, *v;
  const float* g;
  int64_t len;
};
struct AdamTensors {
  AdamTensor t[5];  // means, log_scales, rotations, colors, opacity logits (len 0 if absent)
};

__device__ __forceinline__ float clamp_log_scale(float x, float hi, float lo) {
  x = x > hi ? hi : x;  // clamp_(max=hi) then clamp_(min=lo), NaN passing through as in torch
  return x < lo ? lo : x;
}

// The Adam step over the five tensors as flat arrays (four elements per access where every
// pointer allows it), each block taking a grid-stride share of every tensor; log-scales are
// clamped to [log_lo, log_hi[image]] after the step.  The step-dependent factors are formed
// once per thread; the last block to finish advances the device step count.
__global__ void __launch_bounds__(kThreads)
    adam_kernel(AdamTensors ts, AdamHyper h, Frames frames, const float* __restrict__ log_hi,
                int* __restrict__ step_state) {
  pdl_wait();
  pdl_trigger();
  const int t = step_state[0] + 1;
  AdamStep st;
  st.w1 = (float)(1.0 - h.beta1);
  st.b2 = (float)h.beta2;
  st.s2 = (float)(1.0 - h.beta2);
  st.bc2s = (float)sqrt(1.0 - pow(h.beta2, (double)t));
  st.eps = h.eps;
  st.bc1 = 1.0 - pow(h.beta1, (double)t);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  auto hi_of = [&](int64_t e) {  // log-scale element e belongs to Gaussian e / 2
    return log_hi[frames.image ? frames.gauss_image[e >> 1] : 0];
  };
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const AdamTensor T = ts.t[k];
    const float step = (float)(h.lr[k] / st.bc1);
    const bool vec = ((reinterpret_cast<uintptr_t>(T.p) | reinterpret_cast<uintptr_t>(T.m) |
                       reinterpret_cast<uintptr_t>(T.v) | reinterpret_cast<uintptr_t>(T.g)) &
                      15) == 0;
    const int64_t n4 = vec ? T.len / 4 : 0;
    for (int64_t i = tid; i < n4; i += stride) {
      float4 p = reinterpret_cast<float4*>(T.p)[i];
      float4 m = reinterpret_cast<float4*>(T.m)[i];
      float4 v = reinterpret_cast<float4*>(T.v)[i];
      const float4 g = reinterpret_cast<const float4*>(T.g)[i];
      p.x = adam(p.x, g.x, m.x, v.x, step, st);
      p.y = adam(p.y, g.y, m.y, v.y, step, st);
      p.z = adam(p.z, g.z, m.z, v.z, step, st);
      p.w = adam(p.w, g.w, m.w, v.w, step, st);
      if (k == 1) {
        const float h0 = hi_of(4 * i), h1 = hi_of(4 * i + 2);
        p.x = clamp_log_scale(p.x, h0, h.log_lo);
        p.y = clamp_log_scale(p.y, h0, h.log_lo);
        p.z = clamp_log_scale(p.z, h1, h.log_lo);
        p.w = clamp_log_scale(p.w, h1, h.log_lo);
      }
      reinterpret_cast<float4*>(T.p)[i] = p;
      reinterpret_cast<float4*>(T.m)[i] = m;
      reinterpret_cast<float4*>(T.v)[i] = v;
    }
    for (int64_t e = 4 * n4 + tid; e < T.len; e += stride) {
      float m = T.m[e], v = T.v[e];
      float p = adam(T.p[e], T.g[e], m, v, step, st);
      if (k == 1) p = clamp_log_scale(p, hi_of(e), h.log_lo);
      T.p[e] = p;
      T.m[e] = m;
      T.v[e] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(step_state + 1, 1) == (int)gridDim.x - 1) {
      step_state[0] = t;
      step_state[1] = 0;
      __threadfence();
    }
  }
}
constexpr int64_t kOnePassMax = 65536;

struct FieldState {
  FieldPtrs p, m, v;  // parameters and the two Adam moments (logits NULL when absent)
  FieldPtrs g;        // gradients, 256-byte aligned
};

// Gradients of one CTA's Gaussians in shared memory, laid out as the parameter tensors are.
struct GradTile {
  float means[2 * kThreads], log_scales[2 * kThreads], rotations[kThreads], colors[3 * kThreads],
      logits[kThreads];
};

// One float4 of one parameter tensor: where it lies (from: offset in floats), loaded and stepped.
struct AdamSlot {
  float *p, *m, *v, *g;
  const float* grad;  // in shared memory
  float4 pv, mv, vv;
  bool on;
  __device__ __forceinline__ void load() {
    if (!on) return;
    pv = *reinterpret_cast<const float4*>(p);
    mv = *reinterpret_cast<const float4*>(m);
    vv = *reinterpret_cast<const float4*>(v);
  }
  __device__ __forceinline__ void step(float lr, const AdamStep& a) {
    if (!on) return;
    const float4 gv = *reinterpret_cast<const float4*>(grad);
    pv.x = adam(pv.x, gv.x, mv.x, vv.x, lr, a);
    pv.y = adam(pv.y, gv.y, mv.y, vv.y, lr, a);
    pv.z = adam(pv.z, gv.z, mv.z, vv.z, lr, a);
    pv.w = adam(pv.w, gv.w, mv.w, vv.w, lr, a);
    *reinterpret_cast<float4*>(g) = gv;
    *reinterpret_cast<float4*>(m) = mv;
    *reinterpret_cast<float4*>(v) = vv;
  }
  __device__ __forceinline__ void store() {
    if (on) *reinterpret_cast<float4*>(p) = pv;
  }
};

// The whole update of up to kOnePassMax Gaussians in one launch.  A CTA takes 256 consecutive
// Gaussians: their parameters and Adam moments, five contiguous runs, are loaded as float4s before
// anything else; each thread forms one Gaussian's gradients, which change from one Gaussian per
// thread to flat runs through shared memory, and the Adam step follows on the registers loaded at
// the start.  For a 256x256 fit of 4,096 Gaussians the step takes 46.5 us with it, 49 us with two
// launches.  Larger fields stay with two: the one pass keeps some 35 arrays open at once, and from a
// few hundred thousand Gaussians its loads wait on address translation (2 M Gaussians: 577 us, 7%
// of the issue slots, against 52 + 72 us).
// Deterministic mode sums the entry partials in their fixed order (warp-collective); fast mode reads
// and zeroes the atomic accumulators.  vec: every pointer allows 16-byte accesses.
template <bool DETERMINISTIC>
__global__ void __launch_bounds__(kThreads)
    fit_update_kernel(const Splat* __restrict__ rec, int64_t n, float* __restrict__ moments,
                      const float* __restrict__ partials, const int32_t* __restrict__ order,
                      const int32_t* __restrict__ seg, FieldState f, AdamHyper h, Frames frames,
                      const float* __restrict__ log_hi, int* __restrict__ step_state, int vec) {
  pdl_wait();
  pdl_trigger();
  __shared__ __align__(16) GradTile tile;
  __shared__ float lr[5], bc2s;
  const int tid = threadIdx.x;
  const bool logits = f.p.logits != nullptr;
  const int t = step_state[0] + 1;
  const int64_t first = (int64_t)blockIdx.x * kThreads;
  const int count = (int)(n - first < kThreads ? n - first : kThreads);
  const bool flat = vec && count == kThreads;
  // the thread's float4s: of the means or log-scales, of the rotations or colours, of the logits
  AdamSlot s0, s1, s2;
  {
    const bool lo = tid < 128;
    const int64_t at = 2 * first + 4 * (tid & 127);
    s0.p = (lo ? f.p.means : f.p.log_scales) + at;
    s0.m = (lo ? f.m.means : f.m.log_scales) + at;
    s0.v = (lo ? f.v.means : f.v.log_scales) + at;
    s0.g = (lo ? f.g.means : f.g.log_scales) + at;
    s0.grad = (lo ? tile.means : tile.log_scales) + 4 * (tid & 127);
    s0.on = flat;
    const bool rot = tid < 64;
    const int64_t bt = rot ? first + 4 * tid : 3 * first + 4 * (tid - 64);
    s1.p = (rot ? f.p.rotations : f.p.colors) + bt;
    s1.m = (rot ? f.m.rotations : f.m.colors) + bt;
    s1.v = (rot ? f.v.rotations : f.v.colors) + bt;
    s1.g = (rot ? f.g.rotations : f.g.colors) + bt;
    s1.grad = rot ? tile.rotations + 4 * tid : tile.colors + 4 * (tid - 64);
    s1.on = flat;
    const int64_t ct = first + 4 * tid;
    s2.p = f.p.logits + ct;
    s2.m = f.m.logits + ct;
    s2.v = f.v.logits + ct;
    s2.g = f.g.logits + ct;
    s2.grad = tile.logits + 4 * tid;
    s2.on = flat && logits && tid < 64;
  }
  s0.load();
  s1.load();
  s2.load();
  // the step's factors, in double and rounded once, by two threads of different warps
  if (tid == 0) bc2s = (float)sqrt(1.0 - pow(h.beta2, (double)t));
  if (tid == 32) {
    const double bc1 = 1.0 - pow(h.beta1, (double)t);
    for (int k = 0; k < 5; ++k) lr[k] = (float)(h.lr[k] / bc1);
  }
    const int64_t g = first + tid;
  const bool active = tid < count;
  GradIn in;
  if (DETERMINISTIC) {
    sum_entry_partials(partials, order, seg, n, g, active, in.m);
  } else if (active) {
#pragma unroll
    for (int k = 0; k < kMoments; ++k) in.m[k] = moments[k * n + g];
  }
  if (active) {
    load_grad_in(rec, f.p.log_scales, f.p.rotations, f.p.logits, g, in);
    if (!DETERMINISTIC) {
#pragma unroll
      for (int k = 0; k < kMoments; ++k) moments[k * n + g] = 0.0f;
    }
    const FieldPtrs to{tile.means, tile.log_scales, tile.rotations, tile.colors, tile.logits};
    store_grads(in, tid, h.dilation, logits, to);
  }
  __syncthreads();
  AdamStep st;
  st.w1 = (float)(1.0 - h.beta1);
  st.b2 = (float)h.beta2;
  st.s2 = (float)(1.0 - h.beta2);
  st.bc2s = bc2s;
  st.eps = h.eps;
  auto hi_of = [&](int64_t i) { return log_hi[frames.image ? frames.gauss_image[i] : 0]; };
  if (flat) {
    s0.step(lr[tid < 128 ? 0 : 1], st);
    if (tid >= 128) {  // two Gaussians' log-scales
      const float h0 = hi_of(first + 2 * (tid - 128)), h1 = hi_of(first + 2 * (tid - 128) + 1);
      s0.pv.x = clamp_log_scale(s0.pv.x, h0, h.log_lo);
      s0.pv.y = clamp_log_scale(s0.pv.y, h0, h.log_lo);
      s0.pv.z = clamp_log_scale(s0.pv.z, h1, h.log_lo);
      s0.pv.w = clamp_log_scale(s0.pv.w, h1, h.log_lo);
    }
    s0.store();
    s1.step(lr[tid < 64 ? 2 : 3], st);
    s1.store();
    s2.step(lr[4], st);
    s2.store();
  } else {  // the last CTA, or tensors off a 16-byte boundary
    auto run = [&](float* p, float* m, float* v, float* gout, const float* grad, int width, int k) {
      for (int e = tid; e < width * count; e += kThreads) {
        const int64_t at = width * first + e;
        float mv = m[at], vv = v[at];
        float pv = adam(p[at], grad[e], mv, vv, lr[k], st);
        if (k == 1) pv = clamp_log_scale(pv, hi_of(first + (e >> 1)), h.log_lo);
        gout[at] = grad[e];
        p[at] = pv;
        m[at] = mv;
        v[at] = vv;
      }
    };
    run(f.p.means, f.m.means, f.v.means, f.g.means, tile.means, 2, 0);
    run(f.p.log_scales, f.m.log_scales, f.v.log_scales, f.g.log_scales, tile.log_scales, 2, 1);
    run(f.p.rotations, f.m.rotations, f.v.rotations, f.g.rotations, tile.rotations, 1, 2);
    run(f.p.colors, f.m.colors, f.v.colors, f.g.colors, tile.colors, 3, 3);
    if (logits) run(f.p.logits, f.m.logits, f.v.logits, f.g.logits, tile.logits, 1, 4);
  }
  // every thread of this CTA has read step_state[0] (the barriers above); the last CTA advances it
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(step_state + 1, 1) == (int)gridDim.x - 1) {
      step_state[0] = t;
      step_state[1] = 0;
      __threadfence();
    }
  }
}
}  // namespace
}  // namespace ss

using namespace ss;

extern "C" {

int ss_fit_adam_update(const ss_batch* batch, const void* records, int64_t n,
                       const int32_t* tile_gids, int64_t gid_capacity,
                       const int32_t* tile_offsets, int deterministic, void* workspace,
                       float dilation, float* const* params, float* const* exp_avg,
                       float* const* exp_avg_sq, const double* lrs, double beta1, double beta2,
                       double adam_eps, float log_scale_lo, const float* log_scale_hi,
                       int* step_state, ss_stream_t stream) {
  Frames f;
  int rc = frames_of_batch(batch, n, &f);
  if (rc) return rc;
  if (!params || !exp_avg || !exp_avg_sq || !lrs || !step_state || !log_scale_hi)
    return fail(SS_ERR_INVALID_ARGUMENT, "null pointer");
  if (n == 0) return SS_OK;
  if (!records || !workspace) return fail(SS_ERR_INVALID_ARGUMENT, "null records or workspace");
  if (deterministic && (!tile_gids || !tile_offsets))
    return fail(SS_ERR_INVALID_ARGUMENT, "deterministic update needs the tile index");
  for (int k = 0; k < 4; ++k)
    if (!params[k] || !exp_avg[k] || !exp_avg_sq[k])
      return fail(SS_ERR_INVALID_ARGUMENT, "null field tensor %d", k);
  if ((params[4] != nullptr) != (exp_avg[4] != nullptr) ||
      (params[4] != nullptr) != (exp_avg_sq[4] != nullptr))
    return fail(SS_ERR_INVALID_ARGUMENT, "opacity logits and their Adam state go together");
  if (!(beta1 >= 0.0 && beta1 < 1.0 && beta2 >= 0.0 && beta2 < 1.0))
    return fail(SS_ERR_INVALID_ARGUMENT, "Adam betas must lie in [0, 1)");
  FieldPtrs p{params[0], params[1], params[2], params[3], params[4]};
  AdamHyper h;
  for (int k = 0; k < 5; ++k) h.lr[k] = lrs[k];
  h.beta1 = beta1;
  h.beta2 = beta2;
  h.eps = (float)adam_eps;
  h.log_lo = log_scale_lo;
  h.dilation = dilation;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const Splat* rec = static_cast<const Splat*>(records);
  float* ws = static_cast<float*>(workspace);
  const FitGrads fg = fit_grads_layout(
      static_cast<char*>(workspace) + fit_grads_offset(n, gid_capacity, deterministic), n);
  const FieldPtrs gp{fg.means, fg.log_scales, fg.rotations, fg.colors, p.logits ? fg.logits : nullptr};
  cudaStream_t s = as_stream(stream);
  if (n <= kOnePassMax) {
    FieldState fs;
    fs.p = p;
    fs.m = FieldPtrs{exp_avg[0], exp_avg[1], exp_avg[2], exp_avg[3], exp_avg[4]};
    fs.v = FieldPtrs{exp_avg_sq[0], exp_avg_sq[1], exp_avg_sq[2], exp_avg_sq[3], exp_avg_sq[4]};
    fs.g = FieldPtrs{fg.means, fg.log_scales, fg.rotations, fg.colors, fg.logits};
    uintptr_t bits = reinterpret_cast<uintptr_t>(workspace);
    for (int k = 0; k < 5; ++k)
      bits |= reinterpret_cast<uintptr_t>(params[k]) | reinterpret_cast<uintptr_t>(exp_avg[k]) |
              reinterpret_cast<uintptr_t>(exp_avg_sq[k]);
    const int vec = (bits & 15) == 0;
    const unsigned one = (unsigned)((n + kThreads - 1) / kThreads);
    if (deterministic) {
      const EntryOrder eo = entry_order_layout(workspace, n, gid_capacity);
      launch("fit_update_kernel", fit_update_kernel<true>, one, kThreads, 0, s, rec, n, nullptr,
             eo.partials, deterministic == kEntrySlots ? nullptr : eo.order, eo.seg, fs, h, f,
             log_scale_hi, step_state, vec);
    } else {
      launch("fit_update_kernel", fit_update_kernel<false>, one, kThreads, 0, s, rec, n, ws,
             nullptr, nullptr, nullptr, fs, h, f, log_scale_hi, step_state, vec);
    }
    return check_launch("fit update");
  }
  // Both are launched plainly: their grid-stride shares are fixed, so CTAs that started early would
  // crowd on the SMs that the tile kernel left first and finish last there (batched fit step 1,289
  // -> 1,261 us without, 2 M dense Gaussians 1,148 -> 1,114 us).
  // gradients: a grid of at most 8 blocks per SM, grid-stride beyond that
  const int64_t want = (n + kThreads - 1) / kThreads, cap_blocks = (int64_t)sms * 8;
  const unsigned blocks = (unsigned)(want < cap_blocks ? want : cap_blocks);
  if (deterministic) {
    const EntryOrder eo = entry_order_layout(workspace, n, gid_capacity);
    launch_as(false, "fit_grad_kernel", fit_grad_kernel<true>, blocks, kThreads, 0, s, rec, n, nullptr, eo.partials,
                                                      deterministic == kEntrySlots ? nullptr : eo.order,
                                                      eo.seg, p.log_scales, p.rotations,
                                                      p.logits, dilation, gp);
  } else {
    launch_as(false, "fit_grad_kernel", fit_grad_kernel<false>, blocks, kThreads, 0, s, rec, n, ws, nullptr, nullptr, nullptr,
                                                       p.log_scales, p.rotations, p.logits,
                                                       dilation, gp);
  }
  if ((rc = check_launch("fit gradients"))) return rc;
  // the Adam step over the five tensors as flat arrays
  AdamTensors ts;
  const int64_t lens[5] = {2 * n, 2 * n, n, 3 * n, p.logits ? n : 0};
  float* gptr[5] = {fg.means, fg.log_scales, fg.rotations, fg.colors, fg.logits};
  for (int k = 0; k < 5; ++k) {
    ts.t[k].p = params[k];
    ts.t[k].m = exp_avg[k];
    ts.t[k].v = exp_avg_sq[k];
    ts.t[k].g = gptr[k];
    ts.t[k].len = lens[k];
  }
  const int64_t want4 = (3 * n / 4 + kThreads - 1) / kThreads + 1;
  const unsigned ablocks = (unsigned)(want4 < cap_blocks ? want4 : cap_blocks);
  launch_as(false, "adam_kernel", adam_kernel, ablocks, kThreads, 0, s, ts, h, f, log_scale_hi, step_state);
  return check_launch("fit adam step");
}

}  // extern "C"
