// velo_mlp.cu -- the doublet scorer: a 10 -> 32 -> 32 -> 2 ReLU MLP trained in
// FP32 with hand-written forward / backward / Adam kernels; inference
// (velo_mlp_forward and the learned seeding) runs in FP16 on the tensor cores
// (velo_mlp_warp.cuh).
//
// Outputs per (h0, h1) doublet: a keep logit and the half-width (mm) of the
// x window around the straight-line prediction at module f-4 in which the
// doublet's h2 lies.  Loss per sample: binary cross-entropy of the logit
// against the label (1 = the plain seeding chose this doublet for h0 and its
// tracklet survived into an output track) plus, for positives only,
// kWidthWeight * (width - target)^2.
//
// Parameters are one flat FP32 array of VELO_MLP_PARAMS values:
//   W1[32][10] b1[32] W2[32][32] b2[32] W3[2][32] b3[2]
// (row-major, out x in).
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <type_traits>
#include <vector>

#include "velo_internal.h"
#include "velo_mlp_warp.cuh"

namespace velo {

constexpr float kWidthWeight = 0.1f;
constexpr int kTile = 32;             // samples of a CTA's pass: one per lane
constexpr int kTrainWarps = 16;       // each warp owns 2 of the 32 units of a layer
constexpr int kTrainThreads = 32 * kTrainWarps;
constexpr int kUnits = kMlpHidden / kTrainWarps;
static_assert(kUnits == 2 && kMlpOut == 2, "the tile below is laid out for 16 x 2 units and 2 outputs");
// a unit's row over the tile's samples: 36 floats apart, so that 8 lanes
// reading 16 bytes of 8 rows meet no bank twice
constexpr int kRow = kTile + 4;

// BCE-with-logits (stable form) + masked squared width error
__device__ __forceinline__ float sample_loss(const float* out, float label, float target, float* dz, float* dw) {
  const float z = out[0];
  const float p = 1.f / (1.f + expf(-z));
  const float bce = fmaxf(z, 0.f) - z * label + log1pf(expf(-fabsf(z)));
  *dz = p - label;
  const float e = out[1] - target;
  *dw = label * 2.f * kWidthWeight * e;
  return bce + label * kWidthWeight * e * e;
}

// c + a b, the product rounded before the sum.  The step is chaotic in one
// place: a unit whose sum lies within rounding of 0 is live or not by the way
// its terms are rounded, and Adam divides the difference by the gradient's own
// size.  So every term is rounded as a plain FP32 evaluation of the network
// does it, and summed in index order: the decisions are that evaluation's.
// With fused multiply-adds in their place 6 of 240 trainings of 60 steps ended
// more than 2e-5 of the weights' norm away from it (one unit of one sample
// decided otherwise), with these none.
__device__ __forceinline__ float mul_add(float a, float b, float c) { return __fadd_rn(c, __fmul_rn(a, b)); }

// The same where the unit's gradient a is not 0: a unit that is not live adds
// nothing, also where b is infinite or NaN (a feature or a weight is).  kFinite:
// it is known to be neither.
template <bool kFinite>
__device__ __forceinline__ float mul_add_live(float a, float b, float c) {
  return kFinite || a != 0.f ? mul_add(a, b, c) : c;
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= FLT_MAX; }

struct GradTile {
  float w[(VELO_MLP_PARAMS + 3) & ~3];
  float x[kMlpIn][kRow];
  // activations and their gradients by unit and sample
  float a1[kMlpHidden][kRow], d2[kMlpHidden][kRow];
  float a2_d1[kMlpHidden][kRow];   // a2 until the outputs are known, then d1
  float out[kMlpOut][kTile];
};

// Adam (Kingma & Ba), bias-corrected: state and the step's constants.
struct AdamStep {
  float *w, *m, *v;   // null w: no update
  float lr, beta1, beta2, eps, c1, c2;
};

// Floats between two CTAs' rows of partial sums: the gradient, then the loss.
constexpr int kPartialRow = (VELO_MLP_PARAMS + 1 + 31) & ~31;

__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Gradient of the mean loss over n samples (through `index` when given): each
// CTA's share of it, row blockIdx.x of `partial`.
//
// A CTA passes over tiles of 32 samples, one per lane; warp k computes units
// 2k and 2k+1 of each layer, weights broadcast from shared memory, activations
// exchanged through it by unit and sample.  Bias and output-layer gradients
// are summed per lane and reduced once at the end; the two weight matrices
// are products over the tile's samples, each thread holding the same outputs
// for every tile.
//
// The step's floor is 3,904 products and sums a sample, 0.8 us for a batch of
// 4,096 on the whole chip at an instruction each (0.4 if they were fused); what
// bounds it is the chain of launches, gather, six exchanges and reduction.  A
// thread per sample with every product added by a shared-memory atomic, which
// all lanes of a warp aimed at one address, took 1.47 ms a step; this tile with
// its sums added to the gradient by atomics and the update in the last CTA 20.8
// us (128 CTAs waiting on their atomics and a counter); rows of partial sums and
// a second kernel 11.0 us.
__global__ void __launch_bounds__(kTrainThreads) mlp_step_kernel(const float* w,
                                                                 const float* __restrict__ x,
                                                                 const float* __restrict__ label,
                                                                 const float* __restrict__ target,
                                                                 const int64_t* __restrict__ index, int64_t n,
                                                                 float scale, float* __restrict__ partial) {
  __shared__ __align__(16) GradTile t;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, u0 = kUnits * warp;
  const int j2 = tid >> 4, i2 = tid & 15;   // this thread's outputs of W2's gradient: row j2, columns i2 + 16 q
  float gw2[2] = {}, gw1 = 0.f, gw3[kMlpOut][kUnits] = {}, gb1[kUnits] = {}, gb2[kUnits] = {}, gb3[kMlpOut] = {};
  float loss = 0.f;
  bool odd = false;   // a weight is infinite or NaN, or a feature or activation of the tile

  // the samples do not depend on the launch before this one, the weights do
  const int64_t tiles = (n + kTile - 1) / kTile;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t base = tile * kTile;
    if (tile != blockIdx.x) __syncthreads();   // the tile before has been read
    bool odd_tile = false;
    for (int k = tid; k < kTile * kMlpIn; k += kTrainThreads) {
      const int s = k / kMlpIn, i = k % kMlpIn;
      float v = 0.f;
      if (base + s < n) v = x[(index ? index[base + s] : base + s) * kMlpIn + i];
      t.x[i][s] = v;
      odd_tile |= !finite(v);
    }
    const bool in = base + lane < n;
    const int64_t r = in ? (index ? index[base + lane] : base + lane) : 0;
    const float y = in ? label[r] : 0.f, width = in ? target[r] : 0.f;
    if (tile == blockIdx.x) {
      cudaGridDependencySynchronize();
      for (int k = tid; k < VELO_MLP_PARAMS; k += kTrainThreads) {
        const float v = __ldcg(w + k);
        t.w[k] = v;
        odd |= !finite(v);
      }
    }
    __syncthreads();
    // layer 1
    float a1[kUnits], a2[kUnits];
#pragma unroll
    for (int u = 0; u < kUnits; ++u) a1[u] = t.w[kMlpB1 + u0 + u];
#pragma unroll
    for (int i = 0; i < kMlpIn; ++i) {
      const float v = t.x[i][lane];
#pragma unroll
      for (int u = 0; u < kUnits; ++u) a1[u] = mul_add(t.w[kMlpW1 + (u0 + u) * kMlpIn + i], v, a1[u]);
    }
    if (tile == blockIdx.x) cudaTriggerProgrammaticLaunchCompletion();   // the reduction may be set up
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
      a1[u] = in && a1[u] > 0.f ? a1[u] : 0.f;   // no unit of a missing sample is live
      t.a1[u0 + u][lane] = a1[u];
      odd_tile |= !finite(a1[u]);
    }
    const bool careful = __syncthreads_or(odd || odd_tile);
    // layer 2
#pragma unroll
    for (int u = 0; u < kUnits; ++u) a2[u] = t.w[kMlpB2 + u0 + u];
#pragma unroll
    for (int i = 0; i < kMlpHidden; i += 4) {
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = t.a1[i + q][lane];
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const float4 c = *reinterpret_cast<const float4*>(&t.w[kMlpW2 + (u0 + u) * kMlpHidden + i]);
        a2[u] = mul_add(c.w, v[3], mul_add(c.z, v[2], mul_add(c.y, v[1], mul_add(c.x, v[0], a2[u]))));
      }
    }
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
      a2[u] = in && a2[u] > 0.f ? a2[u] : 0.f;
      t.a2_d1[u0 + u][lane] = a2[u];
    }
    __syncthreads();
    // outputs: one warp each, units in order
    if (warp < kMlpOut) {
      float v = t.w[kMlpB3 + warp];
#pragma unroll 8
      for (int i = 0; i < kMlpHidden; ++i) v = mul_add(t.w[kMlpW3 + warp * kMlpHidden + i], t.a2_d1[i][lane], v);
      t.out[warp][lane] = v;
    }
    __syncthreads();
    const float out[kMlpOut] = {t.out[0][lane], t.out[1][lane]};
    float d3[kMlpOut];
    const float l = sample_loss(out, y, width, &d3[0], &d3[1]);
    if (in) {
      loss += l * scale;
      d3[0] *= scale;
      d3[1] *= scale;
    } else {
      d3[0] = d3[1] = 0.f;
    }
    // layers 3 and 2, this warp's units
    gb3[0] += d3[0];
    gb3[1] += d3[1];
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
      gw3[0][u] = mul_add(d3[0], a2[u], gw3[0][u]);
      gw3[1][u] = mul_add(d3[1], a2[u], gw3[1][u]);
      const float d = mul_add(t.w[kMlpW3 + kMlpHidden + u0 + u], d3[1], __fmul_rn(t.w[kMlpW3 + u0 + u], d3[0]));
      const float g = a2[u] > 0.f ? d : 0.f;
      gb2[u] += g;
      t.d2[u0 + u][lane] = g;
    }
    __syncthreads();
    auto backward = [&](auto known_finite) {
      constexpr auto add = mul_add_live<decltype(known_finite)::value>;
      // layer 1: back through W2
      float d1[kUnits] = {};
#pragma unroll 8
      for (int j = 0; j < kMlpHidden; ++j) {
        const float v = t.d2[j][lane];
        const float2 c = *reinterpret_cast<const float2*>(&t.w[kMlpW2 + j * kMlpHidden + u0]);
        d1[0] = add(v, c.x, d1[0]);
        d1[1] = add(v, c.y, d1[1]);
      }
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const float g = a1[u] > 0.f ? d1[u] : 0.f;
        gb1[u] += g;
        t.a2_d1[u0 + u][lane] = g;
      }
      // W2's gradient: sums over the samples of d2[j] a1[i]
#pragma unroll
      for (int k = 0; k < kTile; k += 4) {
        const float4 d = *reinterpret_cast<const float4*>(&t.d2[j2][k]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 a = *reinterpret_cast<const float4*>(&t.a1[i2 + 16 * q][k]);
          gw2[q] = add(d.w, a.w, add(d.z, a.z, add(d.y, a.y, add(d.x, a.x, gw2[q]))));
        }
      }
      __syncthreads();
      // W1's gradient: 320 outputs, d1[j] x[i]
      if (tid < kMlpHidden * kMlpIn) {
        const float* d = t.a2_d1[tid / kMlpIn];
        const float* v = t.x[tid % kMlpIn];
#pragma unroll
        for (int k = 0; k < kTile; k += 4) {
          const float4 a = *reinterpret_cast<const float4*>(&d[k]), b = *reinterpret_cast<const float4*>(&v[k]);
          gw1 = add(a.w, b.w, add(a.z, b.z, add(a.y, b.y, add(a.x, b.x, gw1))));
        }
      }
    };
    if (careful)
      backward(std::false_type{});
    else
      backward(std::true_type{});
  }

  float* row = partial + (size_t)blockIdx.x * kPartialRow;
#pragma unroll
  for (int q = 0; q < 2; ++q) row[kMlpW2 + j2 * kMlpHidden + i2 + 16 * q] = gw2[q];
  if (tid < kMlpHidden * kMlpIn) row[kMlpW1 + tid] = gw1;
  float mine = 0.f;   // lanes 0, 1: b1; 2, 3: b2; 4, 5 and 6, 7: W3's rows; 8, 9: b3; 10: the loss
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const float v1 = lane_sum(gb1[u]), v2 = lane_sum(gb2[u]), v3 = lane_sum(gw3[0][u]), v4 = lane_sum(gw3[1][u]);
    if (lane == u) mine = v1;
    if (lane == 2 + u) mine = v2;
    if (lane == 4 + u) mine = v3;
    if (lane == 6 + u) mine = v4;
  }
  const float vb0 = lane_sum(gb3[0]), vb1 = lane_sum(gb3[1]), vl = lane_sum(loss);
  if (lane == 8) mine = vb0;
  if (lane == 9) mine = vb1;
  if (lane == 10) mine = vl;
  const int u = lane & 1;
  const int to = lane < 2   ? kMlpB1 + u0 + u
                 : lane < 4 ? kMlpB2 + u0 + u
                 : lane < 6 ? kMlpW3 + u0 + u
                 : lane < 8 ? kMlpW3 + kMlpHidden + u0 + u
                            : kMlpB3 + lane - 8;   // the loss after the parameters
  // every warp has the outputs' sums: warp 0 writes them
  if (lane < 8 || (warp == 0 && lane < 11)) row[to] = mine;
}
static_assert(kMlpB3 + 2 == VELO_MLP_PARAMS, "the loss follows the output biases");

// Sums the rows of `partial`, in a fixed order: the gradient (to `grad` when
// given) and the mean loss, and with adam.w the Adam update.  32 parameters
// per CTA, 8 rows at a time.
__global__ void __launch_bounds__(256) mlp_reduce_kernel(const float* __restrict__ partial, int rows, float* grad,
                                                         float* loss, AdamStep adam) {
  __shared__ float sums[8][32];
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();   // the next step may gather its samples
  float v = 0.f;
  if (i <= VELO_MLP_PARAMS) {
#pragma unroll 4
    for (int r = group; r < rows; r += 8) v += __ldcg(partial + (size_t)r * kPartialRow + i);
  }
  sums[group][lane] = v;
  __syncthreads();
  if (group != 0 || i > VELO_MLP_PARAMS) return;
  float gi = 0.f;
#pragma unroll
  for (int g = 0; g < 8; ++g) gi += sums[g][lane];
  if (i == VELO_MLP_PARAMS) {
    if (loss) *loss = gi;
    return;
  }
  if (grad) grad[i] = gi;
  if (!adam.w) return;
  const float mi = adam.beta1 * __ldcg(adam.m + i) + (1.f - adam.beta1) * gi;
  const float vi = adam.beta2 * __ldcg(adam.v + i) + (1.f - adam.beta2) * gi * gi;
  adam.m[i] = mi;
  adam.v[i] = vi;
  adam.w[i] = __ldcg(adam.w + i) - adam.lr * (mi / adam.c1) / (sqrtf(vi / adam.c2) + adam.eps);
}

// Inference as the learned seeding does it (FP16 tensor-core MMA, one warp
// per 32 samples), so the threshold calibrated on its outputs is the one the
// search applies.
__global__ void __launch_bounds__(256) mlp_forward_kernel(const float* __restrict__ w, const float* __restrict__ x,
                                                          int64_t n, float* __restrict__ out) {
  __shared__ MlpFrag frag;
  stage_mlp_fragments(w, &frag);
  __syncthreads();
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;   // whole warps stay in the kernel
  float xi[kMlpIn];
#pragma unroll
  for (int i = 0; i < kMlpIn; ++i) xi[i] = k < n ? x[k * kMlpIn + i] : 0.f;
  float logit, width;
  mlp_eval_warp(frag, xi, &logit, &width);
  if (k < n) {
    out[2 * k] = logit;
    out[2 * k + 1] = width;
  }
}

namespace {

// The device arrays of one call, in one allocation (each cudaMalloc / cudaFree
// pair takes 70 us): reserve them all, then allocate.
struct DevArrays {
  static constexpr size_t kMost = (size_t)1 << 62;
  uint8_t* base = nullptr;
  size_t total = 0;
  cudaStream_t stream = nullptr, aux = nullptr;
  ~DevArrays() {
    if (stream) cudaStreamSynchronize(stream);
    if (aux) cudaStreamSynchronize(aux);
    if (base) cudaFree(base);
    if (stream) cudaStreamDestroy(stream);
    if (aux) cudaStreamDestroy(aux);
  }
  template <typename T>
  size_t reserve(size_t count) {
    const size_t at = total;
    if (count > (kMost - total) / sizeof(T))
      total = kMost;   // no such allocation: allocate() fails
    else
      total += (sizeof(T) * (count ? count : 1) + 255) & ~(size_t)255;
    return at;
  }
  cudaError_t allocate() {
    return total >= kMost ? cudaErrorMemoryAllocation : cudaMalloc(reinterpret_cast<void**>(&base), total);
  }
  template <typename T>
  T* at(size_t offset) const { return reinterpret_cast<T*>(base + offset); }
};

#define MLP_CHECK(call)                      \
  do {                                       \
    cudaError_t e_ = (call);                 \
    if (e_ != cudaSuccess) return VELO_ERR_CUDA; \
  } while (0)

// CTAs (rows of partial sums) of a step over n samples: one per tile of 32
// while the chip has room, at most two per SM.
cudaError_t step_rows(int64_t n, int* rows) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tiles = (n + kTile - 1) / kTile;
  *rows = (int)(tiles < 2 * sms ? tiles : 2 * sms);
  return e;
}

// One step: partial gradients, then their sum and the update.  Each kernel may
// be set up while the one before it finishes; `follows`: so may the first.
cudaError_t launch_step(cudaStream_t stream, bool follows, const float* w, const float* x, const float* label,
                        const float* target, const int64_t* index, int64_t n, float* partial, int rows, float* grad,
                        float* loss, AdamStep adam) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)rows);
  c.blockDim = dim3(kTrainThreads);
  c.stream = stream;
  c.attrs = &attr;
  c.numAttrs = follows ? 1 : 0;
  cudaError_t e =
      cudaLaunchKernelEx(&c, mlp_step_kernel, w, x, label, target, index, n, 1.f / (float)n, partial);
  if (e != cudaSuccess) return e;
  c.gridDim = dim3((VELO_MLP_PARAMS + 1 + 31) / 32);
  c.blockDim = dim3(256);
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, mlp_reduce_kernel, (const float*)partial, rows, grad, loss, adam);
}

// splitmix64: the k-th value (k from 1) of the sequence that starts at `seed`.
__host__ __device__ __forceinline__ uint64_t splitmix(uint64_t seed, uint64_t k) {
  uint64_t z = seed + k * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// The draws of `count` places of the epochs' shuffles from place `first` on:
// an epoch swaps element i (n-1 down to 1) with element value % (i + 1).  The
// 64-bit remainder took the host 5.4 ns a draw, four times the swap itself.
__global__ void shuffle_draws_kernel(uint64_t seed, uint64_t n, uint64_t first, uint64_t count,
                                     uint32_t* __restrict__ out) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = n - 1 - (first + k) % (n - 1);
    out[k] = (uint32_t)(splitmix(seed, first + k + 1) % (i + 1));
  }
}

// Draws made per launch: enough epochs to make the launch worth it.
constexpr uint64_t kDrawsAtOnce = 1u << 20;

}  // namespace
}  // namespace velo

using namespace velo;

extern "C" velo_status velo_mlp_grad(const float* weights, const float* x, const float* label, const float* target,
                                     int64_t n, float* grad_out, float* loss_out) {
  if (!weights || !x || !label || !target || n <= 0 || !grad_out) return VELO_ERR_INVALID_ARGUMENT;
  DevArrays d;
  const size_t ow = d.reserve<float>(VELO_MLP_PARAMS), ox = d.reserve<float>((size_t)n * kMlpIn),
               ol = d.reserve<float>((size_t)n), ot = d.reserve<float>((size_t)n),
               og = d.reserve<float>(VELO_MLP_PARAMS), oloss = d.reserve<float>(1);
  int rows = 0;
  MLP_CHECK(step_rows(n, &rows));
  const size_t op = d.reserve<float>((size_t)rows * kPartialRow);
  MLP_CHECK(d.allocate());
  float *dw = d.at<float>(ow), *dx = d.at<float>(ox), *dl = d.at<float>(ol), *dt = d.at<float>(ot),
        *dg = d.at<float>(og), *dloss = d.at<float>(oloss);
  MLP_CHECK(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
  MLP_CHECK(cudaMemcpyAsync(dw, weights, sizeof(float) * VELO_MLP_PARAMS, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dx, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dl, label, sizeof(float) * n, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dt, target, sizeof(float) * n, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(launch_step(d.stream, false, dw, dx, dl, dt, nullptr, n, d.at<float>(op), rows, dg, dloss, AdamStep{}));
  MLP_CHECK(cudaStreamSynchronize(d.stream));
  MLP_CHECK(cudaMemcpy(grad_out, dg, sizeof(float) * VELO_MLP_PARAMS, cudaMemcpyDeviceToHost));
  if (loss_out) MLP_CHECK(cudaMemcpy(loss_out, dloss, sizeof(float), cudaMemcpyDeviceToHost));
  return VELO_OK;
}

extern "C" velo_status velo_mlp_forward(const float* weights, const float* x, int64_t n, float* out) {
  if (!weights || !x || n <= 0 || !out) return VELO_ERR_INVALID_ARGUMENT;
  DevArrays d;
  const size_t ow = d.reserve<float>(VELO_MLP_PARAMS), ox = d.reserve<float>((size_t)n * kMlpIn),
               oo = d.reserve<float>((size_t)n * 2);
  MLP_CHECK(d.allocate());
  float *dw = d.at<float>(ow), *dx = d.at<float>(ox), *dout = d.at<float>(oo);
  MLP_CHECK(cudaMemcpy(dw, weights, sizeof(float) * VELO_MLP_PARAMS, cudaMemcpyHostToDevice));
  MLP_CHECK(cudaMemcpy(dx, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice));
  mlp_forward_kernel<<<(int)((n + 255) / 256), 256>>>(dw, dx, n, dout);
  MLP_CHECK(cudaGetLastError());
  MLP_CHECK(cudaMemcpy(out, dout, sizeof(float) * n * 2, cudaMemcpyDeviceToHost));
  return VELO_OK;
}

namespace {

velo_status train(const float* x, const float* label, const float* target, int64_t n, int32_t steps, int32_t batch,
                  float lr, uint64_t seed, float* weights_inout, float* loss_per_step) {
  const uint64_t places = (uint64_t)steps * (uint64_t)batch;   // samples drawn in all
  std::vector<int64_t> idx;   // outlives the copies on d.stream
  std::vector<int64_t> order;
  std::vector<uint32_t> draws;
  DevArrays d;
  const bool device_draws = n > 1 && n <= (int64_t)0xffffffff;
  const uint64_t swaps = (uint64_t)n - 1;   // draws of an epoch
  const uint64_t epochs = (places + (uint64_t)n - 1) / (uint64_t)n;
  const uint64_t epochs_at_once =
      device_draws ? std::min(epochs, std::max<uint64_t>(1, kDrawsAtOnce / swaps)) : 1;
  int rows = 0;
  MLP_CHECK(step_rows(batch, &rows));
  const size_t ow = d.reserve<float>(VELO_MLP_PARAMS), ox = d.reserve<float>((size_t)n * kMlpIn),
               ol = d.reserve<float>((size_t)n), ot = d.reserve<float>((size_t)n),
               op = d.reserve<float>((size_t)rows * kPartialRow), om = d.reserve<float>(VELO_MLP_PARAMS),
               ov = d.reserve<float>(VELO_MLP_PARAMS), oloss = d.reserve<float>((size_t)steps),
               oi = d.reserve<int64_t>((size_t)places),
               od = d.reserve<uint32_t>(device_draws ? (size_t)(epochs_at_once * swaps) : 1);
  MLP_CHECK(d.allocate());
  idx.resize((size_t)places);
  order.resize((size_t)n);
  if (device_draws) draws.resize((size_t)(epochs_at_once * swaps));
  float *dw = d.at<float>(ow), *dx = d.at<float>(ox), *dl = d.at<float>(ol), *dt = d.at<float>(ot),
        *dp = d.at<float>(op), *dm = d.at<float>(om), *dv = d.at<float>(ov), *dloss = d.at<float>(oloss);
  int64_t* didx = d.at<int64_t>(oi);
  MLP_CHECK(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
  MLP_CHECK(cudaStreamCreateWithFlags(&d.aux, cudaStreamNonBlocking));
  MLP_CHECK(cudaMemcpyAsync(dw, weights_inout, sizeof(float) * VELO_MLP_PARAMS, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dx, x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dl, label, sizeof(float) * n, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemcpyAsync(dt, target, sizeof(float) * n, cudaMemcpyHostToDevice, d.stream));
  MLP_CHECK(cudaMemsetAsync(dm, 0, oloss - om, d.stream));   // both moments
  for (int64_t i = 0; i < n; ++i) order[(size_t)i] = i;
  const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
  double p1 = 1.0, p2 = 1.0;
  int32_t t = 0;
  uint64_t filled = 0, sent = 0;
  // epoch-wise shuffled sample order: each epoch shuffles the one before it.
  // The steps whose samples are known are launched while the host goes on.
  for (uint64_t e = 0; e < epochs; ++e) {
    if (device_draws && e % epochs_at_once == 0) {
      const uint64_t count = std::min(epochs_at_once, epochs - e) * swaps;
      const unsigned blocks = (unsigned)std::min<uint64_t>((count + 255) / 256, 4096);
      shuffle_draws_kernel<<<blocks, 256, 0, d.aux>>>(seed, (uint64_t)n, e * swaps, count, d.at<uint32_t>(od));
      MLP_CHECK(cudaGetLastError());
      MLP_CHECK(cudaMemcpyAsync(draws.data(), d.at<uint32_t>(od), sizeof(uint32_t) * count, cudaMemcpyDeviceToHost,
                                d.aux));
      MLP_CHECK(cudaStreamSynchronize(d.aux));
    }
    const uint32_t* draw = draws.data() + (e % epochs_at_once) * swaps;
    uint64_t k = e * swaps;
    for (int64_t i = n - 1; i > 0; --i) {
      ++k;
      const uint64_t j = device_draws ? *draw++ : splitmix(seed, k) % (uint64_t)(i + 1);
      std::swap(order[(size_t)i], order[(size_t)j]);
    }
    const uint64_t take = std::min<uint64_t>((uint64_t)n, places - filled);
    std::copy(order.begin(), order.begin() + (ptrdiff_t)take, idx.begin() + (ptrdiff_t)filled);
    filled += take;
    const uint64_t ready = filled / (uint64_t)batch;   // steps
    if (ready < (uint64_t)steps && filled - sent < kDrawsAtOnce) continue;
    MLP_CHECK(cudaMemcpyAsync(didx + sent, idx.data() + sent, sizeof(int64_t) * (filled - sent),
                              cudaMemcpyHostToDevice, d.stream));
    sent = filled;
    for (bool first = true; (uint64_t)t < ready; ++t, first = false) {
      p1 *= beta1;
      p2 *= beta2;
      MLP_CHECK(launch_step(d.stream, !first, dw, dx, dl, dt, didx + (size_t)t * batch, batch, dp, rows, nullptr, dloss + t,
                            AdamStep{dw, dm, dv, lr, beta1, beta2, eps, (float)(1.0 - p1), (float)(1.0 - p2)}));
    }
  }
  MLP_CHECK(cudaStreamSynchronize(d.stream));
  MLP_CHECK(cudaMemcpy(weights_inout, dw, sizeof(float) * VELO_MLP_PARAMS, cudaMemcpyDeviceToHost));
  if (loss_per_step) MLP_CHECK(cudaMemcpy(loss_per_step, dloss, sizeof(float) * steps, cudaMemcpyDeviceToHost));
  return VELO_OK;
}

}  // namespace

extern "C" velo_status velo_mlp_train(const float* x, const float* label, const float* target, int64_t n,
                                      int32_t steps, int32_t batch, float lr, uint64_t seed, float* weights_inout,
                                      float* loss_per_step) {
  if (!x || !label || !target || n <= 0 || steps <= 0 || batch <= 0 || !weights_inout)
    return VELO_ERR_INVALID_ARGUMENT;
  try {
    return train(x, label, target, n, steps, batch, lr, seed, weights_inout, loss_per_step);
  } catch (const std::exception&) {   // the host's sample order does not fit
    return VELO_ERR_OUT_OF_MEMORY;
  }
}
