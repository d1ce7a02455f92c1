// cueva_train.cu -- training and batch inference of the learned con2prim
// seed (cueva_mlp.cuh), on the GPU with this file's own kernels:
//   * synthetic (conserved, primitive) pairs from a counter-based generator;
//   * feature extraction and normalisation statistics;
//   * minibatch SGD with Adam: the forward and backward pass of a batch in one
//     kernel (FP32 over bf16-rounded weights, the same rounding the inference
//     kernels read), and one that sums the CTAs' gradients and applies Adam;
//   * batch con2prim for the ablation: Cardano, network seed + Newton, or a
//     given seed + Newton, with the Newton iteration count per state.
// The C-ABI entry points are declared in include/cueva.h.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../include/cueva.h"
#include "cueva_common.cuh"
#include "cueva_launch.h"
#include "cueva_mlp.cuh"

using namespace cueva;

#define TRY(x)                                                                               \
  do {                                                                                       \
    cudaError_t e_ = (x);                                                                    \
    if (e_ != cudaSuccess) return cueva_fail(CUEVA_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

namespace {

// ------------------------------------------------------------ random numbers
// SplitMix64 finaliser (Steele, Lea & Flood 2014) over (seed, index, stream):
// every draw is a pure function of its counter, so the data set does not
// depend on the launch shape.
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double uni(unsigned long long seed, long long i, int k) {
  const unsigned long long h = mix64(seed ^ mix64((unsigned long long)i * 64ull + (unsigned long long)k));
  return (double)(h >> 11) * (1.0 / 9007199254740992.0);   // [0, 1)
}
__device__ __forceinline__ double gauss(unsigned long long seed, long long i, int k) {
  const double u1 = 1.0 - uni(seed, i, k), u2 = uni(seed, i, k + 1);   // Box-Muller
  return sqrt(-2.0 * log(u1)) * cos(2.0 * CUDART_PI * u2);
}
__device__ __forceinline__ void unit_vector(unsigned long long seed, long long i, int k, double& x, double& y,
                                            double& z) {
  const double c = 2.0 * uni(seed, i, k) - 1.0, ph = 2.0 * CUDART_PI * uni(seed, i, k + 1);
  const double s = sqrt(fmax(0.0, 1.0 - c * c));
  x = s * cos(ph); y = s * sin(ph); z = c;
}

// synthetic states: rho log-uniform [1e-3, 10], p log-uniform [1e-4, 10],
// W uniform [1, 20], magnetisation |B|^2 / (rho h) log-uniform [1e-3, 10],
// isotropic directions of v and B, E = -v x B + N(0, 1e-3) per component
__global__ void k_synthetic(long long n, unsigned long long seed, double gamma, double* cons, double* prims) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double rho = pow(10.0, -3.0 + 4.0 * uni(seed, i, 0));
    const double p = pow(10.0, -4.0 + 5.0 * uni(seed, i, 1));
    const double W = 1.0 + 19.0 * uni(seed, i, 2);
    const double sig = pow(10.0, -3.0 + 4.0 * uni(seed, i, 3));
    double ux, uy, uz, bx, by, bz;
    unit_vector(seed, i, 4, ux, uy, uz);
    unit_vector(seed, i, 6, bx, by, bz);
    const double vm = sqrt(1.0 - 1.0 / (W * W));
    const double vx = vm * ux, vy = vm * uy, vz = vm * uz;
    const double h = rho + gamma / (gamma - 1.0) * p;
    const double Bm = sqrt(sig * h);
    const double Bx = Bm * bx, By = Bm * by, Bz = Bm * bz;
    const double Ex = -(vy * Bz - vz * By) + 1.0e-3 * gauss(seed, i, 8);
    const double Ey = -(vz * Bx - vx * Bz) + 1.0e-3 * gauss(seed, i, 10);
    const double Ez = -(vx * By - vy * Bx) + 1.0e-3 * gauss(seed, i, 12);
    const Cons c = startconvar(rho, p, vx, vy, vz, Ex, Ey, Ez, Bx, By, Bz, gamma);
    const double cv[11] = {c.D, c.tau, c.Sx, c.Sy, c.Sz, Ex, Ey, Ez, Bx, By, Bz};
#pragma unroll
    for (int f = 0; f < 11; ++f) cons[f * n + i] = cv[f];
    const double pv[5] = {rho, p, vx, vy, vz};
#pragma unroll
    for (int f = 0; f < 5; ++f) prims[f * n + i] = pv[f];
  }
}

// raw features and target log(p/D) of n states
__global__ void k_features(long long n, const double* cons, const double* p, float* X, float* T) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float f[MLP_IN];
    c2p_features(cons[i], cons[n + i], cons[2 * n + i], cons[3 * n + i], cons[4 * n + i], cons[5 * n + i],
                 cons[6 * n + i], cons[7 * n + i], cons[8 * n + i], cons[9 * n + i], cons[10 * n + i], f);
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k) X[i * MLP_IN + k] = f[k];
    if (T) T[i] = (float)log(p[i] / cons[i]);
  }
}

// sums and sums of squares of the 7 columns (6 features + target)
__global__ void k_moments(long long n, const float* X, const float* T, double* acc) {
  double s[14] = {};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      const double v = (k < MLP_IN) ? (double)X[i * MLP_IN + k] : (double)T[i];
      s[k] += v; s[7 + k] += v * v;
    }
  }
#pragma unroll
  for (int k = 0; k < 14; ++k) {
    double v = s[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&acc[k], v);
  }
}

// One training batch, forward and backward, in one launch.
//
// A CTA takes tiles of 32 rows: features (from the stored ones, or from the
// states themselves), the three hidden layers, the loss and the backward
// pass, with the weights (bf16-rounded, transposed) and every activation of
// the tile in shared memory; its share of the weight gradients stays in
// registers over its tiles and goes to one row of `part`, which
// k_reduce_gradients sums in a fixed order (deterministic).
//
// The passes of a 4096-row batch are 0.1 GFMA: what counts is the number of
// dependent launches and the length of the serial sums, not the arithmetic.
// As 24 launches of small GEMMs, with the weight gradients as one 4096-long
// sum per output on 16 CTAs, a gradient call took 598 us (B200; 170 us in
// each of the four weight-gradient GEMMs).  Split over 128 CTAs of 32 rows the
// longest sum is 32 rows and then 128 partial sums; see k_reduce_gradients
// for the times.  Forward values, dY, dZ and dA keep the order of operations
// of single dot products (ascending index, one FMA each).
constexpr int GT_ROWS = 32;          // rows of a tile
constexpr int GT_THREADS = 256;
constexpr int GT_LD = 68;            // activation row stride: float4 rows, banks shifted by 4
constexpr int GT_LW = MLP_H + 1;     // transposed weight row stride: conflict-free both ways
constexpr int GT_PART = (MLP_NPARAM + 1 + 31) / 32 * 32;   // a partial row: gradients, then the loss sum

struct GradTile {
  float w1t[MLP_IN * GT_LW], w2t[MLP_H * GT_LW], w3t[MLP_H * GT_LW], w4[MLP_H];
  float b1[MLP_H], b2[MLP_H], b3[MLP_H], b4;
  float x[GT_ROWS * 8];              // normalised features
  float t[GT_ROWS], dy[GT_ROWS], d2[GT_ROWS];
  alignas(16) float z1[GT_ROWS * GT_LD], a1[GT_ROWS * GT_LD], z2[GT_ROWS * GT_LD], a2[GT_ROWS * GT_LD],
      z3[GT_ROWS * GT_LD], a3[GT_ROWS * GT_LD], dz[GT_ROWS * GT_LD];
};

// rows 4 w .. 4 w + 3 of C = A B (K = 64) for warp w, lane l holding columns
// l and l + 32: acc[r][c] over ascending k; B(k, n) = bt[k * sk + n * sn]
__device__ __forceinline__ void tile_dot(const float* a, const float* bt, int sk, int sn, float (&acc)[4][2]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float* b0 = bt + lane * sn;
  const float* b1 = bt + (lane + 32) * sn;
#pragma unroll
  for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0.0f;
#pragma unroll 4
  for (int k = 0; k < MLP_H; k += 4) {
    float4 av[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) av[r] = *reinterpret_cast<const float4*>(a + (4 * w + r) * GT_LD + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float u = b0[(k + q) * sk], v = b1[(k + q) * sk];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float x = q == 0 ? av[r].x : q == 1 ? av[r].y : q == 2 ? av[r].z : av[r].w;
        acc[r][0] = fmaf(x, u, acc[r][0]);
        acc[r][1] = fmaf(x, v, acc[r][1]);
      }
    }
  }
}
__device__ __forceinline__ float silu_slope(float z) {
  const float s = sigmoid_fast(z);
  return s * (1.0f + z * (1.0f - s));
}
// hidden layer: z = a W^T + b, act = silu(z)
__device__ __forceinline__ void tile_layer(const float* a, const float* wt, const float* b, float* z, float* act) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float acc[4][2];
  tile_dot(a, wt, GT_LW, 1, acc);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int o = lane + 32 * c, e = (4 * w + r) * GT_LD + o;
      const float v = acc[r][c] + b[o];
      z[e] = v;
      act[e] = silu(v);
    }
}
// dz of the layer below, in place: dz <- (dz W) silu'(z); every warp reads
// and writes its own four rows
__device__ __forceinline__ void tile_back(float* dz, const float* wt, const float* z) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float acc[4][2];
  tile_dot(dz, wt, 1, GT_LW, acc);   // B(o, i) = W(o, i) = wt[i][o]
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int e = (4 * w + r) * GT_LD + lane + 32 * c;
      dz[e] = acc[r][c] * silu_slope(z[e]);
    }
}
// dw[a][b] += sum over the tile's rows of dz(row, to + 16 a) act(row, ti + 16 b)
__device__ __forceinline__ void tile_outer(const float* dz, const float* act, float (&dw)[4][4]) {
  const int ti = threadIdx.x & 15, to = threadIdx.x >> 4;
#pragma unroll 4
  for (int r = 0; r < GT_ROWS; ++r) {
    float u[4], v[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) { u[a] = dz[r * GT_LD + to + 16 * a]; v[a] = act[r * GT_LD + ti + 16 * a]; }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) dw[a][b] = fmaf(u[a], v[b], dw[a][b]);
  }
}

// B rows: row b itself (seed == 0), or drawn uniformly with replacement from
// n.  X, T: stored raw features and targets; with X null they are computed
// from the states (cons, p).
__global__ void __launch_bounds__(GT_THREADS)
k_gradients(long long n, int B, unsigned long long seed, long long step, const float* __restrict__ X,
            const float* __restrict__ T, const double* __restrict__ cons, const double* __restrict__ p,
            const float* __restrict__ norm, const float* __restrict__ wr, float* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char gt_smem[];
  GradTile& S = *reinterpret_cast<GradTile*>(gt_smem);
  const int tid = threadIdx.x;
  for (int e = tid; e < MLP_H * MLP_IN; e += GT_THREADS)
    S.w1t[(e % MLP_IN) * GT_LW + e / MLP_IN] = wr[MLP_OFF_W1 + e];
  for (int e = tid; e < MLP_H * MLP_H; e += GT_THREADS) {
    S.w2t[(e % MLP_H) * GT_LW + e / MLP_H] = wr[MLP_OFF_W2 + e];
    S.w3t[(e % MLP_H) * GT_LW + e / MLP_H] = wr[MLP_OFF_W3 + e];
  }
  if (tid < MLP_H) {
    S.w4[tid] = wr[MLP_OFF_W4 + tid];
    S.b1[tid] = wr[MLP_OFF_B1 + tid];
    S.b2[tid] = wr[MLP_OFF_B2 + tid];
    S.b3[tid] = wr[MLP_OFF_B3 + tid];
    if (tid == 0) S.b4 = wr[MLP_OFF_B4];
  }
  float g3[4][4] = {}, g2[4][4] = {};   // W3, W2: outputs to + 16 a, inputs ti + 16 b
  float g1[2] = {}, gb = 0.0f, gl = 0.0f;   // W1 elements tid, tid + 256; a bias or W4 element; b4 or the loss
  for (long long r0 = (long long)blockIdx.x * GT_ROWS; r0 < B; r0 += (long long)gridDim.x * GT_ROWS) {
    __syncthreads();   // the tile before has been read
    if (tid < GT_ROWS) {
      const long long b = r0 + tid;
      float f[MLP_IN] = {}, t = 0.0f;
      if (b < B) {
        const long long row =
            seed ? (long long)(mix64(seed ^ mix64((unsigned long long)step * 1048576ull + b)) % (unsigned long long)n)
                 : b;
        if (X) {
#pragma unroll
          for (int k = 0; k < MLP_IN; ++k) f[k] = X[row * MLP_IN + k];
          t = T[row];
        } else {
          c2p_features(cons[row], cons[n + row], cons[2 * n + row], cons[3 * n + row], cons[4 * n + row],
                       cons[5 * n + row], cons[6 * n + row], cons[7 * n + row], cons[8 * n + row], cons[9 * n + row],
                       cons[10 * n + row], f);
          t = (float)log(p[row] / cons[row]);
        }
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) f[k] = (f[k] - norm[k]) / norm[MLP_IN + k];
        t = (t - norm[2 * MLP_IN]) / norm[2 * MLP_IN + 1];
      }
#pragma unroll
      for (int k = 0; k < MLP_IN; ++k) S.x[tid * 8 + k] = f[k];
      S.t[tid] = t;
    }
    __syncthreads();
    {   // first layer (K = 6)
      const int lane = tid & 31, w = tid >> 5;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int o = lane + 32 * c, row = 4 * w + r;
          float v = 0.0f;
#pragma unroll
          for (int k = 0; k < MLP_IN; ++k) v = fmaf(S.x[row * 8 + k], S.w1t[k * GT_LW + o], v);
          v += S.b1[o];
          S.z1[row * GT_LD + o] = v;
          S.a1[row * GT_LD + o] = silu(v);
        }
    }
    __syncwarp();   // a warp reads its own four rows only
    tile_layer(S.a1, S.w2t, S.b2, S.z2, S.a2);
    __syncwarp();
    tile_layer(S.a2, S.w3t, S.b3, S.z3, S.a3);
    __syncthreads();
    if (tid < GT_ROWS) {   // output, loss and its gradient (rows past the batch count nothing)
      float y = 0.0f;
#pragma unroll 8
      for (int k = 0; k < MLP_H; ++k) y = fmaf(S.a3[tid * GT_LD + k], S.w4[k], y);
      y += S.b4;
      const float d = r0 + tid < B ? y - S.t[tid] : 0.0f;
      S.dy[tid] = 2.0f * d / (float)B;
      S.d2[tid] = d * d;
    }
    __syncthreads();
    {   // dZ3 = dY W4 silu'(Z3)
      const int lane = tid & 31, w = tid >> 5;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int o = lane + 32 * c, e = (4 * w + r) * GT_LD + o;
          S.dz[e] = (S.dy[4 * w + r] * S.w4[o]) * silu_slope(S.z3[e]);
        }
    }
    __syncthreads();
    // column sums by groups of 64 threads: b3 (dZ3) here, W4 (dY A3), later b2 and b1
    const int col = tid & 63, grp = tid >> 6;
    if (grp == 0) {
      for (int r = 0; r < GT_ROWS; ++r) gb += S.dz[r * GT_LD + col];
    } else if (grp == 3) {
      for (int r = 0; r < GT_ROWS; ++r) gb = fmaf(S.dy[r], S.a3[r * GT_LD + col], gb);
    }
    if (tid == 64)
      for (int r = 0; r < GT_ROWS; ++r) gl += S.dy[r];
    if (tid == 128)
      for (int r = 0; r < GT_ROWS; ++r) gl += S.d2[r];
    tile_outer(S.dz, S.a2, g3);
    __syncthreads();
    tile_back(S.dz, S.w3t, S.z2);
    __syncthreads();
    if (grp == 1)
      for (int r = 0; r < GT_ROWS; ++r) gb += S.dz[r * GT_LD + col];
    tile_outer(S.dz, S.a1, g2);
    __syncthreads();
    tile_back(S.dz, S.w2t, S.z1);
    __syncthreads();
    if (grp == 2)
      for (int r = 0; r < GT_ROWS; ++r) gb += S.dz[r * GT_LD + col];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + 256 * q, o = e / MLP_IN, k = e % MLP_IN;
      if (e < MLP_H * MLP_IN)
        for (int r = 0; r < GT_ROWS; ++r) g1[q] = fmaf(S.dz[r * GT_LD + o], S.x[r * 8 + k], g1[q]);
    }
  }
  float* out = part + (long long)blockIdx.x * GT_PART;
  const int ti = tid & 15, to = tid >> 4;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      out[MLP_OFF_W3 + (to + 16 * a) * MLP_H + ti + 16 * b] = g3[a][b];
      out[MLP_OFF_W2 + (to + 16 * a) * MLP_H + ti + 16 * b] = g2[a][b];
    }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (tid + 256 * q < MLP_H * MLP_IN) out[MLP_OFF_W1 + tid + 256 * q] = g1[q];
  const int col = tid & 63, grp = tid >> 6;
  out[(grp == 0 ? MLP_OFF_B3 : grp == 1 ? MLP_OFF_B2 : grp == 2 ? MLP_OFF_B1 : MLP_OFF_W4) + col] = gb;
  if (tid == 64) out[MLP_OFF_B4] = gl;
  if (tid == 128) out[MLP_NPARAM] = gl;
}

// Sums the nrows partial rows of k_gradients into g (and the loss / B behind
// it) and, with ADAM, applies the update (Kingma & Ba 2015) and the bf16
// rounding of the forward copy.  A CTA takes 32 parameters by 8 slices of the
// rows, each slice in order, the 8 slice sums in order.  B200, 4096 rows,
// whole gradient call: 600 us before, 57 us with these two kernels (27 + 5.5 us
// under ncu, the rest is the copy back); 2000 training steps 1.09 s -> 50 ms.
template <bool ADAM>
__global__ void __launch_bounds__(256)
k_reduce_gradients(int nrows, const float* __restrict__ part, float* g, int B, float* w, float* m, float* v, float* wr,
                   float lr, float b1, float b2, float c1, float c2) {
  __shared__ float sum[8][32];
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;   // GT_PART is a multiple of 32
  float s = 0.0f;
#pragma unroll 8
  for (int r = sl; r < nrows; r += 8) s += part[(long long)r * GT_PART + i];
  sum[sl][lane] = s;
  __syncthreads();
  if (sl != 0 || i > MLP_NPARAM) return;
  float gi = sum[0][lane];
#pragma unroll
  for (int k = 1; k < 8; ++k) gi += sum[k][lane];
  if (i == MLP_NPARAM) {
    g[i] = gi / (float)B;   // the loss
    return;
  }
  g[i] = gi;
  if constexpr (ADAM) {
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi; v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + 1.0e-8f);
    w[i] = wi;
    wr[i] = __bfloat162float(__float2bfloat16(wi));
  }
}

__global__ void k_round(int n, const float* w, float* wr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) wr[i] = __bfloat162float(__float2bfloat16(w[i]));
}

// one state of the batch con2prim arrays.  No array of the batch kernels is
// __restrict__: a caller may recover in place (out = prev, seeds = its
// pressures), and a state is read whole before it is written.
__device__ __forceinline__ C2PIn batch_state(long long n, long long i, const double* cons, const double* prev) {
  return C2PIn{cons[i], cons[n + i], cons[2 * n + i], cons[3 * n + i], cons[4 * n + i], cons[5 * n + i],
               cons[6 * n + i], cons[7 * n + i], cons[8 * n + i], cons[9 * n + i], cons[10 * n + i],
               prev[2 * n + i], prev[3 * n + i], prev[4 * n + i], prev[i], prev[n + i]};
}
// Newton from p0, Cardano where it fails; iters[i] = Newton iterations (-1 failed)
__device__ __forceinline__ void batch_recover(long long n, long long i, const C2PIn& in, double p0, double gamma,
                                              double eps1, double* out, int* iters) {
  C2POut o{};
  const int it = c2p_newton(in, gamma, p0, o);
  if (it < 0) c2p_cardano_ool(in, gamma, eps1, o, nullptr);
  out[i] = o.rho; out[n + i] = o.p; out[2 * n + i] = o.vx; out[3 * n + i] = o.vy; out[4 * n + i] = o.vz;
  if (iters) iters[i] = it;
}

// batch con2prim without the network: method 1 Cardano (iters 0), 3 Newton
// from seed[i]
__global__ void k_c2p_batch(long long n, int method, double gamma, double eps1, const double* cons,
                            const double* prev, const double* seed, double* out, int* iters) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const C2PIn in = batch_state(n, i, cons, prev);
    if (method == 1) {
      C2POut o{};
      c2p_cardano(in, gamma, eps1, o, nullptr);
      out[i] = o.rho; out[n + i] = o.p; out[2 * n + i] = o.vx; out[3 * n + i] = o.vy; out[4 * n + i] = o.vz;
      if (iters) iters[i] = 0;
    } else {
      batch_recover(n, i, in, seed[i], gamma, eps1, out, iters);
    }
  }
}

// batch con2prim with the FP32 network: method 2 its seed, 4 its seed or the
// previous pressure, whichever leaves the smaller residual (Newton; Cardano
// where it fails).
//
// A CTA takes tiles of 128 states.  Thread t prepares the features and
// recovers state t; in between the two 64 x 64 layers run as register-tiled
// FP32 matrix products (8 states x 8 outputs per thread, K = 64) from shared
// memory, in place.  Every output is the sum of mlp_forward in the same
// order (bias first, ascending k, one FMA each), so the seeds are the same
// bits.  What bounds it: 8.6 k FMAs per state, 0.23 ms per million states at
// the FP32 rate.  With one thread per state (mlp_forward) each weight was
// loaded and widened again for every FMA: 1895 us for 10^6 states on a B200;
// tiled 622 us; with two states per FMA instruction 598 us: at 12 warps per SM
// half of the issue slots are used, by 10.2 k thread instructions a state (6.3 k
// on the FMA pipe, 0.6 k on the FP64 pipe), the network and the recovery
// taking turns between barriers.  The bf16 tensor cores would need each FP32
// activation as three parts; not tried.
constexpr int CN_ROWS = 128;
struct C2PNet {
  alignas(16) float w2t[MLP_H * MLP_H], w3t[MLP_H * MLP_H];   // [input][output]
  alignas(16) float act[MLP_H * CN_ROWS];                     // [unit][state]
  float w1[MLP_H * MLP_IN], w4[MLP_H], b1[MLP_H], b2[MLP_H], b3[MLP_H], b4;
  float mu[MLP_IN], sd[MLP_IN], mu_y, sd_y;
};

// two FP32 FMAs in one instruction (each rounded as fmaf)
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// act <- silu(W act + b): outputs 4 og + {0..3} and 32 + those, states 4 sg +
// {0..3} and 64 + those, in pairs of states
__device__ __forceinline__ void c2p_layer(float* act, const float* wt, const float* b) {
  const int sg = threadIdx.x & 15, og = threadIdx.x >> 4;
  unsigned long long z[8][4];
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const float bo = b[(o >> 2) * 32 + 4 * og + (o & 3)];
#pragma unroll
    for (int s = 0; s < 4; ++s) z[o][s] = pack2(bo, bo);
  }
#pragma unroll 4
  for (int k = 0; k < MLP_H; ++k) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(act + k * CN_ROWS + 4 * sg);
    const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(act + k * CN_ROWS + 64 + 4 * sg);
    const float4 w0 = *reinterpret_cast<const float4*>(wt + k * MLP_H + 4 * og);
    const float4 w1 = *reinterpret_cast<const float4*>(wt + k * MLP_H + 32 + 4 * og);
    const unsigned long long av[4] = {a0.x, a0.y, a1.x, a1.y};
    const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const unsigned long long w = pack2(wv[o], wv[o]);
#pragma unroll
      for (int s = 0; s < 4; ++s) z[o][s] = fma2(w, av[s], z[o][s]);
    }
  }
  __syncthreads();   // every input has been read
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    float* row = act + ((o >> 2) * 32 + 4 * og + (o & 3)) * CN_ROWS + 4 * sg;
    const float2 p0 = unpack2(z[o][0]), p1 = unpack2(z[o][1]), p2 = unpack2(z[o][2]), p3 = unpack2(z[o][3]);
    *reinterpret_cast<float4*>(row) = make_float4(silu(p0.x), silu(p0.y), silu(p1.x), silu(p1.y));
    *reinterpret_cast<float4*>(row + 64) = make_float4(silu(p2.x), silu(p2.y), silu(p3.x), silu(p3.y));
  }
  __syncthreads();
}

__global__ void __launch_bounds__(CN_ROWS, 3)
k_c2p_network(long long n, int method, double gamma, double eps1, const MLPDevice* __restrict__ M,
              const double* cons, const double* prev, double* out, int* iters) {
  extern __shared__ __align__(16) unsigned char cn_smem[];
  C2PNet& S = *reinterpret_cast<C2PNet*>(cn_smem);
  const int t = threadIdx.x;
  for (int e = t; e < MLP_H * MLP_H; e += CN_ROWS) {
    const int o = e / MLP_H, k = e % MLP_H;
    S.w2t[k * MLP_H + o] = __bfloat162float(M->W2[e]);
    S.w3t[k * MLP_H + o] = __bfloat162float(M->W3[e]);
  }
  for (int e = t; e < MLP_H * MLP_IN; e += CN_ROWS) S.w1[e] = __bfloat162float(M->W1[e]);
  if (t < MLP_H) {
    S.w4[t] = __bfloat162float(M->W4[t]);
    S.b1[t] = M->b1[t]; S.b2[t] = M->b2[t]; S.b3[t] = M->b3[t];
    if (t < MLP_IN) { S.mu[t] = M->mu[t]; S.sd[t] = M->sd[t]; }
    if (t == 0) { S.b4 = M->b4; S.mu_y = M->mu_y; S.sd_y = M->sd_y; }
  }
  __syncthreads();
  const long long ntiles = (n + CN_ROWS - 1) / CN_ROWS;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long i0 = tile * CN_ROWS + t;
    const long long i = i0 < n ? i0 : n - 1;   // threads past the end repeat the last state
    const C2PIn in = batch_state(n, i, cons, prev);
    float x[MLP_IN];
    c2p_features(in.D, in.tau, in.Sx, in.Sy, in.Sz, in.Ex, in.Ey, in.Ez, in.Bx, in.By, in.Bz, x);
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k) x[k] = (x[k] - S.mu[k]) / S.sd[k];
#pragma unroll 4
    for (int o = 0; o < MLP_H; ++o) {
      float z = S.b1[o];
#pragma unroll
      for (int k = 0; k < MLP_IN; ++k) z = fmaf(S.w1[o * MLP_IN + k], x[k], z);
      S.act[o * CN_ROWS + t] = silu(z);
    }
    __syncthreads();
    c2p_layer(S.act, S.w2t, S.b2);
    c2p_layer(S.act, S.w3t, S.b3);
    float y = S.b4;
#pragma unroll 8
    for (int k = 0; k < MLP_H; ++k) y = fmaf(S.w4[k], S.act[k * CN_ROWS + t], y);
    y = y * S.sd_y + S.mu_y;
    const double p_net = in.D * (double)__expf(y);
    const double p0 = method == 2 ? p_net : c2p_best_seed(in, gamma, p_net);
    if (i0 < n) batch_recover(n, i, in, p0, gamma, eps1, out, iters);
    __syncthreads();   // the activations have been read
  }
}

// network seeds: per thread in FP32 (tensor == 0), or warp-cooperative on
// the tensor cores (tensor == 1; every warp runs full, lanes past n repeat
// state n-1 and store nothing)
__global__ void k_predict(long long n, const MLPDevice* M, const double* cons, double* pseed, int tensor) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long nround = (n + 31) / 32 * 32;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < nround; i0 += stride) {
    const long long i = i0 < n ? i0 : n - 1;
    float f[MLP_IN];
    c2p_features(cons[i], cons[n + i], cons[2 * n + i], cons[3 * n + i], cons[4 * n + i], cons[5 * n + i],
                 cons[6 * n + i], cons[7 * n + i], cons[8 * n + i], cons[9 * n + i], cons[10 * n + i], f);
    const float y = tensor ? mlp_forward_warp(*M, f) : mlp_forward(*M, f);
    if (i0 < n) pseed[i] = cons[i] * (double)__expf(y * M->sd_y + M->mu_y);
  }
}

dim3 grid_for(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  return dim3((unsigned)(b < 1 ? 1 : b));
}

}  // namespace

// ---------------------------------------------------------------- the object
struct cueva_mlp {
  int dev = 0;
  float* w = nullptr;      // FP32 master parameters
  float* wr = nullptr;     // bf16-rounded copy read by the forward passes
  float* m = nullptr;
  float* v = nullptr;
  float* g = nullptr;      // gradients, then the loss
  float* norm = nullptr;   // device copy of hnorm
  float hnorm[MLP_NNORM];
  bool normed = false;
  long long step = 0;
  float* part = nullptr;   // partial gradients of k_gradients: GT_GRID rows
  MLPDevice* d_dev = nullptr;
};

namespace {

// CTAs of k_gradients: a tile each, at most two per SM of a B200
constexpr int GT_GRID = 2 * 148;
int gradient_grid(int B) { return std::min((B - 1) / GT_ROWS + 1, GT_GRID); }

// launches the passes of one batch; the partial gradients go to M->part
int32_t forward_backward(cueva_mlp* M, long long n, int B, unsigned long long seed, const float* X, const float* T,
                         const double* cons, const double* p) {
  if (!M->part) {
    TRY(cudaFuncSetAttribute(k_gradients, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradTile)));
    TRY(cudaMalloc(&M->part, (size_t)GT_GRID * GT_PART * sizeof(float)));
  }
  k_gradients<<<gradient_grid(B), GT_THREADS, sizeof(GradTile)>>>(n, B, seed, M->step, X, T, cons, p, M->norm, M->wr,
                                                                  M->part);
  TRY(cudaGetLastError());
  return CUEVA_OK;
}

int32_t features_of(long long n, const double* cons, const double* p, float** X, float** T) {
  TRY(cudaMalloc(X, (size_t)n * MLP_IN * sizeof(float)));
  if (T) TRY(cudaMalloc(T, (size_t)n * sizeof(float)));
  k_features<<<grid_for(n), 256>>>(n, cons, p, *X, T ? *T : nullptr);
  TRY(cudaGetLastError());
  return CUEVA_OK;
}

}  // namespace

namespace cueva {
// network as the kernels read it, on the host (for cueva_attach_mlp)
int32_t mlp_device_image(const cueva_mlp* M, MLPDevice* out) {
  if (!M->normed) return cueva_fail(CUEVA_ERR_ARG, "the network has no normalisation (train or set it first)");
  std::vector<float> w(MLP_NPARAM);
  TRY(cudaMemcpy(w.data(), M->w, MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
  for (int i = 0; i < MLP_H * MLP_IN; ++i) out->W1[i] = __float2bfloat16(w[MLP_OFF_W1 + i]);
  for (int i = 0; i < MLP_H * MLP_H; ++i) out->W2[i] = __float2bfloat16(w[MLP_OFF_W2 + i]);
  for (int i = 0; i < MLP_H * MLP_H; ++i) out->W3[i] = __float2bfloat16(w[MLP_OFF_W3 + i]);
  for (int i = 0; i < MLP_H; ++i) out->W4[i] = __float2bfloat16(w[MLP_OFF_W4 + i]);
  // biases are FP32 in the kernels; the forward copy rounds them too
  auto rb = [](float x) { return __bfloat162float(__float2bfloat16(x)); };
  for (int i = 0; i < MLP_H; ++i) {
    out->b1[i] = rb(w[MLP_OFF_B1 + i]); out->b2[i] = rb(w[MLP_OFF_B2 + i]); out->b3[i] = rb(w[MLP_OFF_B3 + i]);
  }
  out->b4 = rb(w[MLP_OFF_B4]);
  for (int k = 0; k < MLP_IN; ++k) { out->mu[k] = M->hnorm[k]; out->sd[k] = M->hnorm[MLP_IN + k]; }
  out->mu_y = M->hnorm[2 * MLP_IN];
  out->sd_y = M->hnorm[2 * MLP_IN + 1];
  out->stats = nullptr;
  return CUEVA_OK;
}
int mlp_device_of(const cueva_mlp* M) { return M->dev; }
}  // namespace cueva

namespace {
int32_t refresh_device_image(cueva_mlp* M) {
  MLPDevice h;
  if (int32_t e = mlp_device_image(M, &h)) return e;
  TRY(cudaMemcpy(M->d_dev, &h, sizeof(MLPDevice), cudaMemcpyHostToDevice));
  return CUEVA_OK;
}
}  // namespace

extern "C" {

int32_t cueva_mlp_create(int32_t device, uint64_t seed, cueva_mlp** out) {
  if (!out) return cueva_fail(CUEVA_ERR_ARG, "null argument");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return cueva_fail(CUEVA_ERR_CUDA, "no CUDA device available");
  }
  if (device < 0 || device >= ndev) return cueva_fail(CUEVA_ERR_ARG, "device ordinal out of range");
  TRY(cudaSetDevice(device));
  cueva_mlp* M = new cueva_mlp();
  M->dev = device;
  // He-uniform weights, zero biases (std::mt19937_64: the initial network is
  // a function of the seed only)
  std::vector<float> w(MLP_NPARAM, 0.0f);
  std::mt19937_64 rng(seed);
  auto fill = [&](int off, int fan_out, int fan_in) {
    const double a = std::sqrt(6.0 / fan_in);
    std::uniform_real_distribution<double> U(-a, a);
    for (int i = 0; i < fan_out * fan_in; ++i) w[off + i] = (float)U(rng);
  };
  fill(MLP_OFF_W1, MLP_H, MLP_IN);
  fill(MLP_OFF_W2, MLP_H, MLP_H);
  fill(MLP_OFF_W3, MLP_H, MLP_H);
  fill(MLP_OFF_W4, 1, MLP_H);
  for (int k = 0; k < MLP_NNORM; ++k) M->hnorm[k] = (k >= MLP_IN && k < 2 * MLP_IN) || k == 2 * MLP_IN + 1 ? 1.0f : 0.0f;
  cudaError_t e = cudaSuccess;
  for (float** p : {&M->w, &M->wr, &M->m, &M->v, &M->g})
    if (e == cudaSuccess) e = cudaMalloc(p, (MLP_NPARAM + 1) * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&M->norm, MLP_NNORM * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&M->d_dev, sizeof(MLPDevice));
  if (e == cudaSuccess) e = cudaMemcpy(M->w, w.data(), MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(M->m, 0, MLP_NPARAM * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(M->v, 0, MLP_NPARAM * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(M->norm, M->hnorm, sizeof M->hnorm, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_round<<<(MLP_NPARAM + 255) / 256, 256>>>(MLP_NPARAM, M->w, M->wr);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    cueva_mlp_destroy(M);
    return cueva_fail(CUEVA_ERR_CUDA, std::string("network set-up: ") + cudaGetErrorString(e));
  }
  *out = M;
  return CUEVA_OK;
}

int32_t cueva_mlp_destroy(cueva_mlp* M) {
  if (!M) return CUEVA_OK;
  cudaSetDevice(M->dev);
  cudaDeviceSynchronize();
  for (float* p : {M->w, M->wr, M->m, M->v, M->g, M->norm, M->part})
    if (p) cudaFree(p);
  if (M->d_dev) cudaFree(M->d_dev);
  delete M;
  return CUEVA_OK;
}

int32_t cueva_mlp_get_params(cueva_mlp* M, float* host, int32_t n) {
  if (!M || !host || n != MLP_NPARAM + MLP_NNORM)
    return cueva_fail(CUEVA_ERR_ARG, "expected " + std::to_string(MLP_NPARAM + MLP_NNORM) + " floats");
  TRY(cudaSetDevice(M->dev));
  TRY(cudaMemcpy(host, M->w, MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
  std::memcpy(host + MLP_NPARAM, M->hnorm, sizeof M->hnorm);
  return CUEVA_OK;
}

int32_t cueva_mlp_set_params(cueva_mlp* M, const float* host, int32_t n) {
  if (!M || !host || n != MLP_NPARAM + MLP_NNORM)
    return cueva_fail(CUEVA_ERR_ARG, "expected " + std::to_string(MLP_NPARAM + MLP_NNORM) + " floats");
  TRY(cudaSetDevice(M->dev));
  TRY(cudaMemcpy(M->w, host, MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice));
  std::memcpy(M->hnorm, host + MLP_NPARAM, sizeof M->hnorm);
  TRY(cudaMemcpy(M->norm, M->hnorm, sizeof M->hnorm, cudaMemcpyHostToDevice));
  k_round<<<(MLP_NPARAM + 255) / 256, 256>>>(MLP_NPARAM, M->w, M->wr);
  TRY(cudaGetLastError());
  M->normed = true;
  return refresh_device_image(M);
}

int32_t cueva_mlp_synthetic_pairs(int32_t device, int64_t n, uint64_t seed, double gamma, double* d_cons,
                                  double* d_prims, void* stream) {
  if (n <= 0 || !d_cons || !d_prims) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  TRY(cudaSetDevice(device));
  k_synthetic<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, seed, gamma, d_cons, d_prims);
  TRY(cudaGetLastError());
  return CUEVA_OK;
}

int32_t cueva_mlp_fit_normalisation(cueva_mlp* M, const double* d_cons, const double* d_p, int64_t n) {
  if (!M || n <= 1 || !d_cons || !d_p) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  TRY(cudaSetDevice(M->dev));
  float *X = nullptr, *T = nullptr;
  double* acc = nullptr;
  int32_t rc = features_of(n, d_cons, d_p, &X, &T);
  if (!rc) {
    cudaError_t e = cudaMalloc(&acc, 14 * sizeof(double));
    if (e == cudaSuccess) e = cudaMemset(acc, 0, 14 * sizeof(double));
    if (e == cudaSuccess) {
      k_moments<<<grid_for(n), 256>>>(n, X, T, acc);
      e = cudaGetLastError();
    }
    double h[14];
    if (e == cudaSuccess) e = cudaMemcpy(h, acc, sizeof h, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = cueva_fail(CUEVA_ERR_CUDA, cudaGetErrorString(e));
    else {
      for (int k = 0; k < 7; ++k) {
        const double mu = h[k] / n, var = h[7 + k] / n - mu * mu;
        const double sd = std::sqrt(var > 1e-12 ? var : 1e-12);
        if (k < MLP_IN) { M->hnorm[k] = (float)mu; M->hnorm[MLP_IN + k] = (float)sd; }
        else { M->hnorm[2 * MLP_IN] = (float)mu; M->hnorm[2 * MLP_IN + 1] = (float)sd; }
      }
      M->normed = true;
      e = cudaMemcpy(M->norm, M->hnorm, sizeof M->hnorm, cudaMemcpyHostToDevice);
      if (e != cudaSuccess) rc = cueva_fail(CUEVA_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  if (X) cudaFree(X);
  if (T) cudaFree(T);
  if (acc) cudaFree(acc);
  if (rc) return rc;
  return refresh_device_image(M);
}

int32_t cueva_mlp_train(cueva_mlp* M, const double* d_cons, const double* d_p, int64_t n, int32_t steps,
                        int32_t batch, float lr, uint64_t seed, float* loss_out) {
  if (!M || n <= 0 || steps < 0 || batch <= 0 || !d_cons || !d_p) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  if (!M->normed) return cueva_fail(CUEVA_ERR_ARG, "fit the normalisation first");
  TRY(cudaSetDevice(M->dev));
  float *X = nullptr, *T = nullptr;
  int32_t rc = features_of(n, d_cons, d_p, &X, &T);
  const float b1 = 0.9f, b2 = 0.999f;
  for (int s = 0; s < steps && !rc; ++s) {
    ++M->step;
    rc = forward_backward(M, n, batch, seed ? seed : 1ull, X, T, nullptr, nullptr);
    if (rc) break;
    // cosine decay of the learning rate over this call's steps
    const float lr_s = 0.5f * lr * (1.0f + std::cos(3.14159265f * (float)s / (float)(steps > 1 ? steps : 1)));
    const float c1 = 1.0f - std::pow(b1, (float)M->step), c2 = 1.0f - std::pow(b2, (float)M->step);
    k_reduce_gradients<true><<<GT_PART / 32, 256>>>(gradient_grid(batch), M->part, M->g, batch, M->w, M->m, M->v, M->wr,
                                                    lr_s, b1, b2, c1, c2);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = cueva_fail(CUEVA_ERR_CUDA, cudaGetErrorString(e));
  }
  if (!rc && loss_out) {
    cudaError_t e = cudaMemcpy(loss_out, M->g + MLP_NPARAM, sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = cueva_fail(CUEVA_ERR_CUDA, cudaGetErrorString(e));
  }
  if (X) cudaFree(X);
  if (T) cudaFree(T);
  if (rc) return rc;
  return refresh_device_image(M);
}

int32_t cueva_mlp_gradients(cueva_mlp* M, const double* d_cons, const double* d_p, int32_t n, float* grads,
                            float* loss_out) {
  if (!M || n <= 0 || !d_cons || !d_p || !grads) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  TRY(cudaSetDevice(M->dev));
  if (int32_t e = forward_backward(M, n, n, 0ull, nullptr, nullptr, d_cons, d_p)) return e;
  k_reduce_gradients<false><<<GT_PART / 32, 256>>>(gradient_grid(n), M->part, M->g, n, nullptr, nullptr, nullptr,
                                                   nullptr, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f);
  TRY(cudaGetLastError());
  float host[MLP_NPARAM + 1];
  TRY(cudaMemcpy(host, M->g, sizeof host, cudaMemcpyDeviceToHost));
  std::memcpy(grads, host, MLP_NPARAM * sizeof(float));
  if (loss_out) *loss_out = host[MLP_NPARAM];
  return CUEVA_OK;
}

int32_t cueva_mlp_predict(cueva_mlp* M, const double* d_cons, int64_t n, double* d_pseed, int32_t tensor_cores) {
  if (!M || n <= 0 || !d_cons || !d_pseed) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  if (!M->normed) return cueva_fail(CUEVA_ERR_ARG, "the network has no normalisation");
  TRY(cudaSetDevice(M->dev));
  if (tensor_cores < 0 || tensor_cores > 3) return cueva_fail(CUEVA_ERR_ARG, "tensor_cores must be 0, 1, 2 or 3");
  if (tensor_cores >= 2) {
    // tcgen05 tiles of 128 states; a bounded wait that runs out is reported
    uint32_t* d_err = nullptr;
    TRY(cudaMalloc(&d_err, sizeof(uint32_t)));
    cudaError_t e = cudaMemset(d_err, 0, sizeof(uint32_t));
    if (e == cudaSuccess) e = launch_predict_tc(n, M->d_dev, d_cons, d_pseed, d_err, 0, tensor_cores == 3);
    uint32_t herr = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&herr, d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    cudaFree(d_err);
    if (e != cudaSuccess) return cueva_fail(CUEVA_ERR_CUDA, cudaGetErrorString(e));
    if (herr) return cueva_fail(CUEVA_ERR_PHYSICS, "a tensor-core wait ran out (status 64)");
    return CUEVA_OK;
  }
  // whole warps: the grid covers n rounded up to 32 in multiples of the block
  k_predict<<<grid_for((n + 31) / 32 * 32), 256>>>(n, M->d_dev, d_cons, d_pseed, tensor_cores ? 1 : 0);
  TRY(cudaGetLastError());
  TRY(cudaDeviceSynchronize());
  return CUEVA_OK;
}

int32_t cueva_c2p_batch(int32_t device, int32_t method, const cueva_mlp* M, double gamma, double eps1,
                        const double* d_cons, const double* d_prev, const double* d_seed, int64_t n, double* d_out,
                        int32_t* d_iters) {
  if (n <= 0 || !d_cons || !d_prev || !d_out) return cueva_fail(CUEVA_ERR_ARG, "bad arguments");
  if (method < 1 || method > 4)
    return cueva_fail(CUEVA_ERR_ARG, "method must be 1 (Cardano), 2 (network), 3 (seed) or 4 (network or previous p)");
  if ((method == 2 || method == 4) && (!M || !M->normed))
    return cueva_fail(CUEVA_ERR_ARG, "methods 2 and 4 need a trained network");
  if (method == 3 && !d_seed) return cueva_fail(CUEVA_ERR_ARG, "method 3 needs seeds");
  TRY(cudaSetDevice(device));
  if (method == 2 || method == 4) {
    // three CTAs per SM (66 KB of shared memory, up to 168 registers per thread)
    TRY(cudaFuncSetAttribute(k_c2p_network, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(C2PNet)));
    const long long tiles = (n + CN_ROWS - 1) / CN_ROWS;
    k_c2p_network<<<(unsigned)std::min<long long>(tiles, 3 * 148), CN_ROWS, sizeof(C2PNet)>>>(
        n, method, gamma, eps1, M->d_dev, d_cons, d_prev, d_out, d_iters);
  } else {
    k_c2p_batch<<<grid_for(n), 256>>>(n, method, gamma, eps1, d_cons, d_prev, d_seed, d_out, d_iters);
  }
  TRY(cudaGetLastError());
  TRY(cudaDeviceSynchronize());
  return CUEVA_OK;
}

}  // extern "C"
