// lbx_closure.cu — learned lubrication / sub-resolution closure for sphere
// pairs (no counterpart in the reference; it attaches where the reference's
// analytic lubrication branch sits, addHertzian, kernels_fluid_PART.CUF:
// 1463-1501, which stays the fallback and the judge).
//
// Network: 13 -> 64 -> 64 -> 64 -> 12, SiLU, FP32.  Inputs, in the
// lattice-fixed pair frame E of spheres i < j (lattice_frame in
// lbx_closure.h: first axis n = (x_j - x_i)/|x_j - x_i|, transverse axes
// fixed by the cubic symmetry class of n, sign s = det of that class map):
//   gap/R, E (v_j - v_i), s E omega_i, s E omega_j, R, nc_1, nc_2
// (angular velocities in the lab frame; nc the sorted |n| components, which
// with the gap name the pair's lattice class).  Outputs: force and torque
// corrections on i and on j in the same frame (torques carry s).  Inputs and
// outputs are standardised with the mean / std stored after the weights.
// Training decays the Adam step size from lr to 0 as a half cosine over the
// optimiser steps of all epochs.
//
// Kernels
//   k_mlp_train  one thread-block cluster of 8 CTAs runs every epoch of
//                minibatch Adam on the whole data set: each CTA takes 8 of
//                the 64 samples of a minibatch (forward, backward, its
//                gradient in shared memory), the gradient is summed over the
//                cluster in rank order through distributed shared memory,
//                each CTA updates one slice of the parameters and writes it
//                into every CTA's copy.
//   k_mlp_infer  one warp per sample (pair), weights in shared memory.
//   k_pairs (lbx_particles.cu) / k_closure_pairs / k_closure_accum: per
//                step, the close pairs of each sphere (ascending index, listed
//                by the all-pairs force pass), the closure (or the
//                analytic lubrication when the pair leaves the training
//                envelope) and a fixed-order accumulation per sphere.
#include "lbx_device.cuh"
#include "lbx_closure.h"

#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include <type_traits>

namespace lbx {

// ---------------------------------------------------------------------------
// training: a thread-block cluster of NCL CTAs, minibatch TB split over them
// ---------------------------------------------------------------------------
constexpr int TB = 64;              // minibatch
constexpr int TT = 256;             // threads per CTA
constexpr int NCL = 8;              // CTAs of the cluster (portable cluster size)
constexpr int TBC = TB / NCL;       // samples of a minibatch per CTA
constexpr int NC4 = MlpLayout::NPARAM / 4;        // parameters in chunks of 4 (every matrix starts on one)
constexpr int SL4 = (NC4 + NCL - 1) / NCL;        // chunks each CTA reduces and updates
constexpr int SLR = (SL4 + TT - 1) / TT;          // chunks per thread of that slice
// Rows of the 64-wide matrices are 68 words apart in shared memory: eight
// lanes reading four words of eight consecutive rows then touch 32 banks.
constexpr int WS = H + 4;
struct TrainSmem {                  // offsets in floats
  static constexpr int W0 = 0, B0 = W0 + H * DIN, W1 = B0 + H, B1 = W1 + H * WS, W2 = B1 + H, B2 = W2 + H * WS,
                       W3 = B2 + H, B3 = W3 + DOUT * WS, NW = B3 + DOUT;
  static constexpr int GS = NW;                       // [NCL][SL4] chunks: the slice's gradient of each CTA
  static constexpr int X0 = GS + NCL * SL4 * 4;       // TBC x DIN
  static constexpr int T0 = X0 + TBC * DIN;           // TBC x DOUT
  static constexpr int A1 = T0 + TBC * DOUT, A2 = A1 + TBC * H, A3 = A2 + TBC * H;  // activations
  static constexpr int S1 = A3 + TBC * H, S2 = S1 + TBC * H, S3 = S2 + TBC * H;     // silu'
  static constexpr int D = S3 + TBC * H;              // TBC x DOUT: dL/dY
  static constexpr int E = D + TBC * DOUT, F = E + TBC * H;  // TBC x H: dL/dZ of two layers in turn
  static constexpr int TOTAL = F + TBC * H;
  static_assert(NW % 4 == 0 && X0 % 4 == 0 && T0 % 4 == 0 && A1 % 4 == 0 && D % 4 == 0 && E % 4 == 0, "alignment");
};
static_assert(MlpLayout::NPARAM % 4 == 0 && MlpLayout::W1 % 4 == 0 && MlpLayout::W2 % 4 == 0 &&
                  MlpLayout::W3 % 4 == 0 && MlpLayout::B0 % 4 == 0, "chunks of 4 parameters");

struct TrainArgs {
  const float* X;   // n x DIN, standardised
  const float* T;   // n x DOUT, standardised
  int n;
  float* w;         // NPARAM (updated)
  float* loss;      // per epoch (may be null)
  float* grad_out;  // grad-only mode: NPARAM gradient of the first minibatch
  int epochs;
  float lr, beta1, beta2, eps;
  unsigned seed;
};

// place of parameter chunk j (parameters 4 j .. 4 j + 3) in the padded shared copy
__device__ __forceinline__ int chunk_at(int j) {
  using L = MlpLayout;
  using M = TrainSmem;
  const int i = 4 * j;
  if (i < L::W1) return i;
  auto mat = [&](int o, int at) { return at + (o / H) * WS + o % H; };
  if (i < L::B1) return mat(i - L::W1, M::W1);
  if (i < L::W2) return M::B1 + (i - L::B1);
  if (i < L::B2) return mat(i - L::W2, M::W2);
  if (i < L::W3) return M::B2 + (i - L::B2);
  if (i < L::B3) return mat(i - L::W3, M::W3);
  return M::B3 + (i - L::B3);
}

__device__ __forceinline__ float hsum(float4 a) { return (a.x + a.y) + (a.z + a.w); }
__device__ __forceinline__ void fma4(float4& s, float4 a, float4 b) {
  s.x = fmaf(a.x, b.x, s.x);
  s.y = fmaf(a.y, b.y, s.y);
  s.z = fmaf(a.z, b.z, s.z);
  s.w = fmaf(a.w, b.w, s.w);
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void fma1(float4& s, float a, float4 b) {
  s.x = fmaf(a, b.x, s.x);
  s.y = fmaf(a, b.y, s.y);
  s.z = fmaf(a, b.z, s.z);
  s.w = fmaf(a, b.w, s.w);
}

// activation and its derivative
__device__ __forceinline__ void act(float z, float* A, float* S) {
  *A = silu(z);
  *S = dsilu(z);
}

// hidden layer: a thread takes output o of two samples, so a row of W is read
// once for both; four partial sums per output
__device__ __forceinline__ void hidden_fwd(const float* A, const float* W, const float* bias, float* Ao, float* So) {
  const int o = threadIdx.x % H, b = 2 * (threadIdx.x / H);
  float4 s0 = make_float4(bias[o], 0.f, 0.f, 0.f), s1 = s0;
#pragma unroll
  for (int k = 0; k < H; k += 4) {
    const float4 w = ld4(W + o * WS + k);
    fma4(s0, w, ld4(A + b * H + k));
    fma4(s1, w, ld4(A + (b + 1) * H + k));
  }
  act(hsum(s0), Ao + b * H + o, So + b * H + o);
  act(hsum(s1), Ao + (b + 1) * H + o, So + (b + 1) * H + o);
}

// dZp[b][k] = (sum_o dZ[b][o] W[o][k]) silu'(Zp[b][k]), two samples per thread
template <int O>
__device__ __forceinline__ void dense_back(const float* dZ, const float* W, const float* Sp, float* dZp) {
  const int k = threadIdx.x % H, b = 2 * (threadIdx.x / H);
  float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
#pragma unroll
  for (int o = 0; o < O; o += 4) {
    const float4 w = make_float4(W[o * WS + k], W[(o + 1) * WS + k], W[(o + 2) * WS + k], W[(o + 3) * WS + k]);
    fma4(s0, w, ld4(dZ + b * O + o));
    fma4(s1, w, ld4(dZ + (b + 1) * O + o));
  }
  dZp[b * H + k] = hsum(s0) * Sp[b * H + k];
  dZp[(b + 1) * H + k] = hsum(s1) * Sp[(b + 1) * H + k];
}

// Every epoch of minibatch Adam on the whole data set in one launch of one
// cluster.  Each CTA holds the weights and runs forward and backward for its
// TBC samples of the minibatch; each chunk of its gradient goes straight into
// the shared memory of the CTA that owns the chunk (distributed shared
// memory stores, which nobody waits for).  After a cluster barrier CTA r sums
// slice r over the CTAs in rank order, updates it with Adam (moments in
// registers) and writes the new values into every CTA's weights; a second
// barrier ends the step.  The samples of the next minibatch are loaded behind
// the first barrier.
// Bound: the chain of eight small dependent layers and two cluster barriers of
// every step; no unit is busy.  Rows padded by four words, two samples (four
// gradient rows) per thread, the activations in the layer's own pass and the
// gradient pushed instead of fetched took a step from 19.5 us to 9.5 us
// (30,976 samples, 484 steps per epoch).
__global__ void __cluster_dims__(NCL, 1, 1) __launch_bounds__(TT) k_mlp_train(TrainArgs a) {
  namespace cg = cooperative_groups;
  using L = MlpLayout;
  using M = TrainSmem;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = int(cl.block_rank()), tid = int(threadIdx.x);
  extern __shared__ __align__(16) float sm[];
  __shared__ float warp_loss[TT / 32], cta_loss[NCL], rate[3];
  for (int j = tid; j < NC4; j += TT) *reinterpret_cast<float4*>(sm + chunk_at(j)) = ld4(a.w + 4 * j);
  float4 Mo[SLR], Vo[SLR];
#pragma unroll
  for (int r = 0; r < SLR; ++r) Mo[r] = Vo[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int lo = rank * SL4, hi = min(NC4, lo + SL4);
  // the gradient chunk j of this CTA, into the CTA that owns it
  auto push = [&](int j, float4 g) {
    const int r = j / SL4;
    *reinterpret_cast<float4*>(cl.map_shared_rank(sm + M::GS, r) + 4 * (rank * SL4 + j - r * SL4)) = g;
  };
  // weight gradient of a 64-wide matrix: dW[o][k..k+3] of rows o0 .. o0 + N - 1
  auto grad_rows = [&](const float* dZ, int O, const float* A, int base, int o0, int k, auto rows) {
    constexpr int N = decltype(rows)::value;
    float4 g[N];
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int b = 0; b < TBC; ++b) {
      const float4 x = ld4(A + b * H + k);
#pragma unroll
      for (int i = 0; i < N; ++i) fma1(g[i], dZ[b * O + o0 + i], x);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) push((base + (o0 + i) * H + k) / 4, g[i]);
  };
  // bias gradient chunk c of a layer of O outputs
  auto grad_bias = [&](const float* dZ, int O, int base, int c) {
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int b = 0; b < TBC; ++b) fma1(g, 1.f, ld4(dZ + b * O + 4 * c));
    push(base / 4 + c, g);
  };
  using One = std::integral_constant<int, 1>;
  using Four = std::integral_constant<int, 4>;

  const int nb = (a.n + TB - 1) / TB;
  const bool grad_only = a.grad_out != nullptr;
  const int epochs = grad_only ? 1 : a.epochs;
  int off = 0, stride = 1;
  // epoch order: i -> (i * stride + off) mod n with stride coprime to n
  auto epoch_order = [&](int ep) {
    unsigned h = a.seed * 2654435761u + unsigned(ep) * 40503u + 12345u;
    off = int(h % unsigned(a.n));
    stride = 1 + int((h >> 8) % unsigned(a.n));
    while (true) {  // gcd(stride, n) == 1
      int x = stride, y = a.n;
      while (y) { int t = x % y; x = y; y = t; }
      if (x == 1) break;
      stride = stride % a.n + 1;
    }
  };
  // this thread's feature or target of its CTA's samples of minibatch bi
  // (threads 0 .. 103: features, 128 .. 223: targets)
  const bool has_x = tid < TBC * DIN, has_t = tid >= 128 && tid < 128 + TBC * DOUT;
  const int item = has_x ? tid : tid - 128, row = item / (has_x ? DIN : DOUT), col = item % (has_x ? DIN : DOUT);
  auto fetch = [&](int bi) -> float {
    if (!has_x && !has_t) return 0.f;
    const int cnt = min(TB, a.n - bi * TB), gb = rank * TBC + row;  // sample of the minibatch
    const int i = grad_only ? min(gb, a.n - 1)
                            : int((long long)(bi * TB + min(gb, cnt - 1)) * stride % a.n + off) % a.n;
    return has_x ? a.X[size_t(i) * DIN + col] : a.T[size_t(i) * DOUT + col];
  };
  auto keep = [&](float v) {
    if (has_x) sm[M::X0 + item] = v;
    else if (has_t) sm[M::T0 + item] = v;
  };
  epoch_order(0);
  keep(fetch(0));
  cl.sync();
  int t_adam = 0;
  for (int ep = 0; ep < epochs; ++ep) {
    float ep_loss = 0.f;
    for (int bi = 0; bi < (grad_only ? 1 : nb); ++bi) {
      const int cnt = min(TB, a.n - bi * TB);
      // forward: input layer
      {
        const int o = tid % H, b = 2 * (tid / H);
        float s0 = sm[M::B0 + o], s1 = s0;
#pragma unroll
        for (int k = 0; k < DIN; ++k) {
          const float w = sm[M::W0 + o * DIN + k];
          s0 = fmaf(sm[M::X0 + b * DIN + k], w, s0);
          s1 = fmaf(sm[M::X0 + (b + 1) * DIN + k], w, s1);
        }
        act(s0, sm + M::A1 + b * H + o, sm + M::S1 + b * H + o);
        act(s1, sm + M::A1 + (b + 1) * H + o, sm + M::S1 + (b + 1) * H + o);
      }
      __syncthreads();
      hidden_fwd(sm + M::A1, sm + M::W1, sm + M::B1, sm + M::A2, sm + M::S2);
      __syncthreads();
      hidden_fwd(sm + M::A2, sm + M::W2, sm + M::B2, sm + M::A3, sm + M::S3);
      __syncthreads();
      // output layer and the loss: mean over the minibatch's valid samples
      // and outputs of (y - t)^2
      float part = 0.f;
      if (tid < TBC * DOUT) {
        const int b = tid / DOUT, o = tid % DOUT;
        float4 s = make_float4(sm[M::B3 + o], 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < H; k += 4) fma4(s, ld4(sm + M::W3 + o * WS + k), ld4(sm + M::A3 + b * H + k));
        const float d = (rank * TBC + b < cnt) ? hsum(s) - sm[M::T0 + tid] : 0.f;
        part = d * d;
        sm[M::D + tid] = d * (2.0f / float(cnt * DOUT));
      }
#pragma unroll
      for (int st = 16; st > 0; st >>= 1) part += __shfl_xor_sync(0xffffffffu, part, st);
      if (tid % 32 == 0) warp_loss[tid / 32] = part;
      __syncthreads();
      if (tid == TT - 1) {
        float l = 0.f;
        for (int w = 0; w < TT / 32; ++w) l += warp_loss[w];
        cl.map_shared_rank(cta_loss, 0)[rank] = l;
      }
      // backward: output layer, then the three hidden layers
      if (tid < DOUT * H / 4) grad_rows(sm + M::D, DOUT, sm + M::A3, L::W3, tid / 16, 4 * (tid % 16), One{});
      else if (tid < DOUT * H / 4 + DOUT / 4) grad_bias(sm + M::D, DOUT, L::B3, tid - DOUT * H / 4);
      dense_back<DOUT>(sm + M::D, sm + M::W3, sm + M::S3, sm + M::E);
      __syncthreads();
      grad_rows(sm + M::E, H, sm + M::A2, L::W2, 4 * (tid / 16), 4 * (tid % 16), Four{});
      if (tid < H / 4) grad_bias(sm + M::E, H, L::B2, tid);
      dense_back<H>(sm + M::E, sm + M::W2, sm + M::S2, sm + M::F);
      __syncthreads();
      grad_rows(sm + M::F, H, sm + M::A1, L::W1, 4 * (tid / 16), 4 * (tid % 16), Four{});
      if (tid < H / 4) grad_bias(sm + M::F, H, L::B1, tid);
      dense_back<H>(sm + M::F, sm + M::W1, sm + M::S1, sm + M::E);
      __syncthreads();
      if (tid < H * DIN / 4) {
        float g[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int o = (4 * tid + i) / DIN, k = (4 * tid + i) % DIN;
          g[i] = 0.f;
#pragma unroll
          for (int b = 0; b < TBC; ++b) g[i] = fmaf(sm[M::E + b * H + o], sm[M::X0 + b * DIN + k], g[i]);
        }
        push(tid, make_float4(g[0], g[1], g[2], g[3]));
      } else if (tid < H * DIN / 4 + H / 4) {
        grad_bias(sm + M::E, H, L::B0, tid - H * DIN / 4);
      }
      cl.barrier_arrive();  // this CTA's gradient and loss share are on their way
      ++t_adam;
      if (tid == TT - 1) {
        rate[0] = 1.0f - powf(a.beta1, float(t_adam));
        rate[1] = 1.0f - powf(a.beta2, float(t_adam));
        rate[2] = 0.5f * a.lr * (1.0f + cospif(float(t_adam - 1) / float(a.epochs * nb)));
      }
      // the samples of the next minibatch (of the next epoch after the last)
      const bool last = bi + 1 == (grad_only ? 1 : nb);
      float next = 0.f;
      if (!(last && ep + 1 == epochs)) {
        if (last) epoch_order(ep + 1);
        next = fetch(last ? 0 : bi + 1);
      }
      __syncthreads();      // rate[]; every thread has read this minibatch's samples
      cl.barrier_wait();    // every CTA's gradient is here
      keep(next);
      if (rank == 0 && tid == 0)
        for (int r = 0; r < NCL; ++r) ep_loss += cta_loss[r];
      const float c1 = rate[0], c2 = rate[1], lr_t = rate[2];
#pragma unroll
      for (int q = 0; q < SLR; ++q) {
        const int j = lo + tid + q * TT;
        if (j >= hi) continue;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < NCL; ++r) fma1(g, 1.f, ld4(sm + M::GS + 4 * (r * SL4 + j - lo)));
        if (grad_only) {
          *reinterpret_cast<float4*>(a.grad_out + 4 * j) = g;
          continue;
        }
        const int at = chunk_at(j);
        float4 w = ld4(sm + at);
        auto adam = [&](float gi, float& mi, float& vi, float& wi) {
          mi = a.beta1 * mi + (1.0f - a.beta1) * gi;
          vi = a.beta2 * vi + (1.0f - a.beta2) * gi * gi;
          wi = wi - lr_t * (mi / c1) / (sqrtf(vi / c2) + a.eps);
        };
        adam(g.x, Mo[q].x, Vo[q].x, w.x);
        adam(g.y, Mo[q].y, Vo[q].y, w.y);
        adam(g.z, Mo[q].z, Vo[q].z, w.z);
        adam(g.w, Mo[q].w, Vo[q].w, w.w);
#pragma unroll
        for (int r = 0; r < NCL; ++r) *reinterpret_cast<float4*>(cl.map_shared_rank(sm + at, r)) = w;
      }
      cl.sync();  // new weights everywhere; the slices' gradients are free for the next step
    }
    if (rank == 0 && tid == 0 && a.loss && !grad_only) a.loss[ep] = ep_loss / float(a.n * DOUT);
  }
  if (!grad_only && rank == 0)
    for (int j = tid; j < NC4; j += TT) *reinterpret_cast<float4*>(a.w + 4 * j) = ld4(sm + chunk_at(j));
}

// Raw features or targets (rows of D) standardised in place with the blob's
// mean and std: the two roundings of the host loop this replaces (0.45 ms of
// a 15 ms call at 30,976 samples)
__global__ void k_standardise(float* __restrict__ v, size_t n, int D, const float* __restrict__ mean,
                              const float* __restrict__ sd) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    const int k = int(i % unsigned(D));
    v[i] = (v[i] - mean[k]) / sd[k];
  }
}

// ---------------------------------------------------------------------------
// inference: one warp per sample, weights (and normalisation) in shared memory
// ---------------------------------------------------------------------------
__global__ void k_mlp_infer(const float* __restrict__ Wg, const float* __restrict__ X, int n, float* Y) {
  extern __shared__ float sm[];
  float* W = sm;
  float* bufs = W + MlpLayout::TOTAL;
  load_infer_weights(Wg, W);
  __syncthreads();
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* buf = bufs + warp * 2 * H;
  for (int s = blockIdx.x * nw + warp; s < n; s += gridDim.x * nw) {
    float x[DIN], y[DOUT];
    for (int k = 0; k < DIN; ++k) x[k] = X[size_t(s) * DIN + k];
    mlp_warp(W, x, y, buf);
    if ((threadIdx.x & 31) == 0)
      for (int o = 0; o < DOUT; ++o) Y[size_t(s) * DOUT + o] = y[o];
  }
}

// Launch of k_mlp_infer on device buffers (weights, n x DIN features, n x
// DOUT outputs) on the legacy default stream; used by entry points that
// manage their own device memory.
int closure_infer_launch(const float* dW, const float* dX, int n, float* dY) {
  using L = MlpLayout;
  const size_t smem = sizeof(float) * (size_t(L::TOTAL) + 8 * 2 * H);
  if (cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
    return LBX_ERR_CUDA;
  int blocks = (n + 7) / 8;
  if (blocks > 148 * 4) blocks = 148 * 4;
  k_mlp_infer<<<blocks, 256, smem>>>(dW, dX, n, dY);
  return cudaGetLastError() == cudaSuccess ? 0 : LBX_ERR_CUDA;
}

}  // namespace lbx

// ---------------------------------------------------------------------------
// host entry points (C ABI, include/lbx.h)
// ---------------------------------------------------------------------------
namespace {
struct Dev {
  void* p = nullptr;
  explicit Dev(size_t b) {
    if (b && cudaMalloc(&p, b) != cudaSuccess) p = nullptr;
  }
  ~Dev() {
    if (p) cudaFree(p);
  }
};
size_t train_smem() { return sizeof(float) * size_t(lbx::TrainSmem::TOTAL); }
int rc_of(cudaError_t e) { return e == cudaSuccess ? 0 : LBX_ERR_CUDA; }
}  // namespace

extern "C" {

int lbx_closure_init(float* weights, int32_t seed) {
  using L = lbx::MlpLayout;
  if (!weights) return LBX_ERR_ARG;
  // Glorot-uniform weights, zero biases, identity standardisation
  unsigned long long s = 0x9E3779B97F4A7C15ull ^ (unsigned long long)(seed);
  auto rnd = [&]() {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    return double(s >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int fan_out, int fan_in) {
    double lim = std::sqrt(6.0 / double(fan_in + fan_out));
    for (int i = 0; i < fan_out * fan_in; ++i) weights[off + i] = float((2.0 * rnd() - 1.0) * lim);
  };
  for (int i = 0; i < L::TOTAL; ++i) weights[i] = 0.f;
  fill(L::W0, lbx::H, lbx::DIN);
  fill(L::W1, lbx::H, lbx::H);
  fill(L::W2, lbx::H, lbx::H);
  fill(L::W3, lbx::DOUT, lbx::H);
  for (int i = 0; i < lbx::DIN; ++i) weights[L::XSD + i] = 1.f;
  for (int i = 0; i < lbx::DOUT; ++i) weights[L::YSD + i] = 1.f;
  return 0;
}

int lbx_closure_train(float* weights, const float* X, const float* T, int32_t n, int32_t epochs, float lr,
                      int32_t seed, float* loss) {
  using L = lbx::MlpLayout;
  if (!weights || !X || !T || n < 1 || epochs < 1) return LBX_ERR_ARG;
  const size_t nx = size_t(n) * lbx::DIN, nt = size_t(n) * lbx::DOUT;
  Dev dX(nx * 4), dT(nt * 4), dW(size_t(L::TOTAL) * 4), dL(size_t(epochs) * 4);
  if (!dX.p || !dT.p || !dW.p || !dL.p) return LBX_ERR_ALLOC;
  int rc = rc_of(cudaMemcpy(dX.p, X, nx * 4, cudaMemcpyHostToDevice));
  if (!rc) rc = rc_of(cudaMemcpy(dT.p, T, nt * 4, cudaMemcpyHostToDevice));
  if (!rc) rc = rc_of(cudaMemcpy(dW.p, weights, size_t(L::TOTAL) * 4, cudaMemcpyHostToDevice));
  if (!rc) {
    float *x = (float*)dX.p, *t = (float*)dT.p, *w = (float*)dW.p;
    const int bx = int(std::min<size_t>((nx + 255) / 256, 1184)), bt = int(std::min<size_t>((nt + 255) / 256, 1184));
    lbx::k_standardise<<<bx, 256>>>(x, nx, lbx::DIN, w + L::XMU, w + L::XSD);
    lbx::k_standardise<<<bt, 256>>>(t, nt, lbx::DOUT, w + L::YMU, w + L::YSD);
    rc = rc_of(cudaGetLastError());
  }
  if (rc) return rc;
  lbx::TrainArgs a{(const float*)dX.p, (const float*)dT.p, n, (float*)dW.p, (float*)dL.p, nullptr, epochs, lr,
                   0.9f, 0.999f, 1e-8f, unsigned(seed)};
  size_t smem = train_smem();
  rc = rc_of(cudaFuncSetAttribute(lbx::k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  if (rc) return rc;
  lbx::k_mlp_train<<<lbx::NCL, lbx::TT, smem>>>(a);  // one cluster
  rc = rc_of(cudaGetLastError());
  if (!rc) rc = rc_of(cudaDeviceSynchronize());
  if (!rc) rc = rc_of(cudaMemcpy(weights, dW.p, size_t(L::NPARAM) * 4, cudaMemcpyDeviceToHost));
  if (!rc && loss) rc = rc_of(cudaMemcpy(loss, dL.p, size_t(epochs) * 4, cudaMemcpyDeviceToHost));
  return rc;
}

int lbx_closure_grad(const float* weights, const float* Xs, const float* Ts, int32_t n, float* grad) {
  using L = lbx::MlpLayout;
  if (!weights || !Xs || !Ts || !grad || n < 1) return LBX_ERR_ARG;
  const size_t nx = size_t(n) * lbx::DIN, nt = size_t(n) * lbx::DOUT;
  Dev dX(nx * 4), dT(nt * 4), dW(size_t(L::TOTAL) * 4), dG(size_t(L::NPARAM) * 4);
  if (!dX.p || !dT.p || !dW.p || !dG.p) return LBX_ERR_ALLOC;
  int rc = rc_of(cudaMemcpy(dX.p, Xs, nx * 4, cudaMemcpyHostToDevice));
  if (!rc) rc = rc_of(cudaMemcpy(dT.p, Ts, nt * 4, cudaMemcpyHostToDevice));
  if (!rc) rc = rc_of(cudaMemcpy(dW.p, weights, size_t(L::TOTAL) * 4, cudaMemcpyHostToDevice));
  if (rc) return rc;
  lbx::TrainArgs a{(const float*)dX.p, (const float*)dT.p, n, (float*)dW.p, nullptr, (float*)dG.p, 1, 0.f,
                   0.9f, 0.999f, 1e-8f, 0u};
  size_t smem = train_smem();
  rc = rc_of(cudaFuncSetAttribute(lbx::k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  if (rc) return rc;
  lbx::k_mlp_train<<<lbx::NCL, lbx::TT, smem>>>(a);  // one cluster
  rc = rc_of(cudaGetLastError());
  if (!rc) rc = rc_of(cudaDeviceSynchronize());
  if (!rc) rc = rc_of(cudaMemcpy(grad, dG.p, size_t(L::NPARAM) * 4, cudaMemcpyDeviceToHost));
  return rc;
}

int lbx_closure_infer(const float* weights, const float* X, int32_t n, float* Y) {
  using L = lbx::MlpLayout;
  if (!weights || !X || !Y || n < 1) return LBX_ERR_ARG;
  Dev dX(size_t(n) * lbx::DIN * 4), dY(size_t(n) * lbx::DOUT * 4), dW(size_t(L::TOTAL) * 4);
  if (!dX.p || !dY.p || !dW.p) return LBX_ERR_ALLOC;
  int rc = rc_of(cudaMemcpy(dX.p, X, size_t(n) * lbx::DIN * 4, cudaMemcpyHostToDevice));
  if (!rc) rc = rc_of(cudaMemcpy(dW.p, weights, size_t(L::TOTAL) * 4, cudaMemcpyHostToDevice));
  if (rc) return rc;
  size_t smem = sizeof(float) * (size_t(L::TOTAL) + 8 * 2 * lbx::H);
  rc = rc_of(cudaFuncSetAttribute(lbx::k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  if (rc) return rc;
  int blocks = (n + 7) / 8;
  if (blocks > 148 * 4) blocks = 148 * 4;
  lbx::k_mlp_infer<<<blocks, 256, smem>>>((const float*)dW.p, (const float*)dX.p, n, (float*)dY.p);
  rc = rc_of(cudaGetLastError());
  if (!rc) rc = rc_of(cudaDeviceSynchronize());
  if (!rc) rc = rc_of(cudaMemcpy(Y, dY.p, size_t(n) * lbx::DOUT * 4, cudaMemcpyDeviceToHost));
  return rc;
}

}  // extern "C"
