// Learned-closure training pipeline: box filter of fine moment fields,
// training samples from a filtered field, the fused forward/backward kernel
// of the MLP, the Adam update, prediction, and the trainer's C ABI
// (lbm_closure.h).  The network and its features are closure.cuh, shared
// with the collide of the step kernels.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "closure.cuh"
#include "lbm_internal.h"

namespace lbm {

float round_bf16(float v) {
  uint32_t u;
  std::memcpy(&u, &v, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) {  // Inf or NaN: truncate, keep NaN quiet
    if (u & 0x007fffffu) u |= 0x00400000u;
    u &= 0xffff0000u;
  } else {
    u += 0x7fffu + ((u >> 16) & 1u);  // nearest, ties to even
    u &= 0xffff0000u;
  }
  float r;
  std::memcpy(&r, &u, 4);
  return r;
}

void clo_fragments(const float* net, uint32_t* words) {
  auto bits = [](float v) {  // a bf16 value's upper half
    uint32_t u;
    std::memcpy(&u, &v, 4);
    return u >> 16;
  };
  auto w1 = [&](int n, int k) { return k < 30 && k % 10 < CLO_IN ? net[CLO_W1 + n * CLO_IN + k % 10] : 0.0f; };
  auto w2 = [&](int n, int k) { return net[CLO_W2 + n * CLO_HID + k]; };
  for (int lane = 0; lane < 32; ++lane) {
    const int g = lane >> 2, t = lane & 3;
    for (int s = 0; s < 2; ++s)
      for (int j = 0; j < 4; ++j)
        for (int h = 0; h < 2; ++h) {  // rows k and k + 1 of column n
          const int n = 8 * j + g, k = 16 * s + 8 * h + 2 * t;
          const size_t at = ((size_t)((2 * s + j / 2) * 32 + lane)) * 4 + 2 * (j % 2) + h;
          words[at] = bits(w1(n, k)) | bits(w1(n, k + 1)) << 16;
          words[512 + at] = bits(w2(n, k)) | bits(w2(n, k + 1)) << 16;
        }
  }
  const int src[3] = {CLO_B1, CLO_B2, CLO_W3};
  for (int v = 0; v < 3; ++v)
    for (int j = 0; j < 4; ++j)
      for (int t = 0; t < 4; ++t)
        for (int e = 0; e < 2; ++e)
          std::memcpy(&words[1024 + ((2 * v + j / 2) * 4 + t) * 4 + 2 * (j % 2) + e], &net[src[v] + 8 * j + 2 * t + e], 4);
}

namespace {

// ---------------------------------------------------------------------------
// Box filter: one thread per coarse node, Favre averages of factor^3 fine
// nodes accumulated in fp64.  Consecutive threads take consecutive coarse x,
// so a warp reads contiguous fine rows: V values a load where the factor allows
// (single values keep the load units busy: k_box_filter_any, written out because
// the template below with V = 1 takes 117 us for 288^3 / 9 where this takes 104), and for F = 2 or 4 a
// plane's rows in flight together.  Bound by HBM at factor 4: 512^3 331 us = 6.5
// TB/s (351 with single loads), 256^3 47.6 us (52.2), factor 2 61.6 (88), factor 8
// 74 (90).
// ---------------------------------------------------------------------------
__global__ void k_box_filter_any(const float* __restrict__ rho, const float* __restrict__ u, int nx,
                             int ny, int nz, int f, float* __restrict__ out) {
  const int ncx = nx / f, ncy = ny / f, ncz = nz / f;
  const size_t nc = (size_t)ncx * ncy * ncz;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const int X = (int)(c % ncx);
  const size_t r = c / ncx;
  const int Y = (int)(r % ncy), Z = (int)(r / ncy);
  const size_t n = (size_t)nx * ny * nz;
  double sr = 0, jx = 0, jy = 0, jz = 0, xx = 0, yy = 0, zz = 0, xy = 0, xz = 0, yz = 0;
  for (int dz = 0; dz < f; ++dz)
    for (int dy = 0; dy < f; ++dy) {
      const size_t base = (size_t)X * f + (size_t)nx * ((size_t)Y * f + dy + (size_t)ny * ((size_t)Z * f + dz));
      for (int dx = 0; dx < f; ++dx) {
        const size_t i = base + dx;
        const double rh = rho[i], ux = u[i], uy = u[n + i], uz = u[2 * n + i];
        const double mx = rh * ux, my = rh * uy, mz = rh * uz;
        sr += rh;
        jx += mx; jy += my; jz += mz;
        xx += mx * ux; yy += my * uy; zz += mz * uz;
        xy += mx * uy; xz += mx * uz; yz += my * uz;
      }
    }
  float o[10] = {};
  if (sr > 0) {
    const double ux = jx / sr, uy = jy / sr, uz = jz / sr;
    o[0] = (float)(sr / ((double)f * f * f));
    o[1] = (float)ux; o[2] = (float)uy; o[3] = (float)uz;
    o[4] = (float)(xx / sr - ux * ux); o[5] = (float)(yy / sr - uy * uy); o[6] = (float)(zz / sr - uz * uz);
    o[7] = (float)(xy / sr - ux * uy); o[8] = (float)(xz / sr - ux * uz); o[9] = (float)(yz / sr - uy * uz);
  }
  for (int k = 0; k < 10; ++k) out[k * nc + c] = o[k];
}

// F: the factor when it is known (0: any multiple of V).
template <int V> struct FilterVec;
template <> struct FilterVec<2> { using T = float2; };
template <> struct FilterVec<4> { using T = float4; };

template <int V, int F>
__global__ void k_box_filter(const float* __restrict__ rho, const float* __restrict__ u, int nx,
                             int ny, int nz, int factor, float* __restrict__ out) {
  using T = typename FilterVec<V>::T;
  const int f = F ? F : factor;
  const int ncx = nx / f, ncy = ny / f, ncz = nz / f;
  const size_t nc = (size_t)ncx * ncy * ncz;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const int X = (int)(c % ncx);
  const size_t r = c / ncx;
  const int Y = (int)(r % ncy), Z = (int)(r / ncy);
  const size_t n = (size_t)nx * ny * nz;
  double sr = 0, jx = 0, jy = 0, jz = 0, xx = 0, yy = 0, zz = 0, xy = 0, xz = 0, yz = 0;
  auto row = [&](const T& vr, const T& vx, const T& vy, const T& vz) {
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const double rh = reinterpret_cast<const float*>(&vr)[e], ux = reinterpret_cast<const float*>(&vx)[e],
                   uy = reinterpret_cast<const float*>(&vy)[e], uz = reinterpret_cast<const float*>(&vz)[e];
      const double mx = rh * ux, my = rh * uy, mz = rh * uz;
      sr += rh;
      jx += mx; jy += my; jz += mz;
      xx += mx * ux; yy += my * uy; zz += mz * uz;
      xy += mx * uy; xz += mx * uz; yz += my * uz;
    }
  };
  auto ld = [](const float* p) { return *reinterpret_cast<const T*>(p); };
  for (int dz = 0; dz < f; ++dz) {
    const size_t base = (size_t)X * f + (size_t)nx * ((size_t)Y * f + (size_t)ny * ((size_t)Z * f + dz));
    if constexpr (F == V) {  // a plane of the box: F loads of each field, all issued before the sums
      T a[4][F];
#pragma unroll
      for (int dy = 0; dy < F; ++dy) {
        const size_t i = base + (size_t)nx * dy;
        a[0][dy] = ld(rho + i);
        a[1][dy] = ld(u + i);
        a[2][dy] = ld(u + n + i);
        a[3][dy] = ld(u + 2 * n + i);
      }
#pragma unroll
      for (int dy = 0; dy < F; ++dy) row(a[0][dy], a[1][dy], a[2][dy], a[3][dy]);
    } else {
      for (int dy = 0; dy < f; ++dy) {
        const size_t b = base + (size_t)nx * dy;
        for (int dx = 0; dx < f; dx += V) {
          const size_t i = b + dx;
          row(ld(rho + i), ld(u + i), ld(u + n + i), ld(u + 2 * n + i));
        }
      }
    }
  }
  float o[10] = {};
  if (sr > 0) {
    const double ux = jx / sr, uy = jy / sr, uz = jz / sr;
    o[0] = (float)(sr / ((double)f * f * f));
    o[1] = (float)ux; o[2] = (float)uy; o[3] = (float)uz;
    o[4] = (float)(xx / sr - ux * ux); o[5] = (float)(yy / sr - uy * uy); o[6] = (float)(zz / sr - uz * uz);
    o[7] = (float)(xy / sr - ux * uy); o[8] = (float)(xz / sr - ux * uz); o[9] = (float)(yz / sr - uy * uz);
  }
  for (int k = 0; k < 10; ++k) out[k * nc + c] = o[k];
}

// ---------------------------------------------------------------------------
// Training samples (see lbm_closure_samples).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {  // splitmix64 finaliser
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void k_samples(const float* __restrict__ filt, int nx, int ny, int nz, float tau,
                          float cs0, uint64_t seed, int64_t ns, float* __restrict__ xo,
                          float* __restrict__ to, float* __restrict__ wo) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns) return;
  const size_t n = (size_t)nx * ny * nz;
  const size_t node = seed == 0 ? (size_t)i : (size_t)(mix64(seed * 0x9e3779b97f4a7c15ull + (uint64_t)i) % n);
  const int x = (int)(node % nx);
  const int y = (int)((node / nx) % ny), z = (int)(node / ((size_t)nx * ny));
  const int xp = x + 1 == nx ? 0 : x + 1, xm = x == 0 ? nx - 1 : x - 1;
  const int yp = y + 1 == ny ? 0 : y + 1, ym = y == 0 ? ny - 1 : y - 1;
  const int zp = z + 1 == nz ? 0 : z + 1, zm = z == 0 ? nz - 1 : z - 1;
  auto at = [&](int xx, int yy, int zz) { return (size_t)xx + (size_t)nx * ((size_t)yy + (size_t)ny * zz); };
  const size_t nb[3][2] = {{at(xp, y, z), at(xm, y, z)}, {at(x, yp, z), at(x, ym, z)}, {at(x, y, zp), at(x, y, zm)}};
  double G[3][3];  // G[a][b] = d u_a / d x_b, central differences
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b)
      G[a][b] = 0.5 * ((double)filt[(1 + a) * n + nb[b][0]] - (double)filt[(1 + a) * n + nb[b][1]]);
  // S in the order xx yy zz xy xz yz
  const double S[6] = {G[0][0], G[1][1], G[2][2], 0.5 * (G[0][1] + G[1][0]),
                       0.5 * (G[0][2] + G[2][0]), 0.5 * (G[1][2] + G[2][1])};
  const double ss = S[0] * S[0] + S[1] * S[1] + S[2] * S[2] + 2.0 * (S[3] * S[3] + S[4] * S[4] + S[5] * S[5]);
  const double smag = sqrt(2.0 * ss);  // |S|
  double t[6];
  for (int k = 0; k < 6; ++k) t[k] = filt[(4 + k) * n + node];
  const double tr = (t[0] + t[1] + t[2]) / 3.0;
  const double tds = (t[0] - tr) * S[0] + (t[1] - tr) * S[1] + (t[2] - tr) * S[2] +
                     2.0 * (t[3] * S[3] + t[4] * S[4] + t[5] * S[5]);
  const double c2 = (double)cs0 * cs0;
  const double s3 = smag * smag * smag;
  const bool ok = s3 > 1e-300;
  const double rho = filt[node];
  const double taus = (double)tau + 3.0 * c2 * smag;
  float P[6];
  for (int k = 0; k < 6; ++k) P[k] = (float)(-(2.0 / 3.0) * rho * taus * S[k]);
  float xf[CLO_IN];
  closure_features<Ops1>(P, (float)rho, xf);
  for (int k = 0; k < CLO_IN; ++k) xo[(size_t)i * CLO_IN + k] = xf[k];
  to[i] = ok ? (float)(-tds / (c2 * s3)) : 0.0f;
  wo[i] = ok ? (float)s3 : 0.0f;
}

// ---------------------------------------------------------------------------
// Prediction: one thread per sample, network in shared memory.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_predict(const float* __restrict__ net,
                                                 const float* __restrict__ x, int64_t n,
                                                 float* __restrict__ r) {
  __shared__ float sw[CLO_FLOATS];
  for (int k = threadIdx.x; k < CLO_FLOATS; k += blockDim.x) sw[k] = net[k];
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float xi[CLO_IN];
  for (int k = 0; k < CLO_IN; ++k) xi[k] = x[(size_t)i * CLO_IN + k];
  const float* w = sw;
  r[i] = closure_mlp<Ops1>(w, xi);
}

// ---------------------------------------------------------------------------
// Fused forward/backward of one batch.
//
// A block takes 32 samples at a time, lane = sample, and its four warps share
// them: warp w owns hidden units 8w .. 8w+7 of both layers, forward and backward,
// and hands the activations (h1, h2) and pre-activation gradients (d a1, d a2) on
// through shared memory.  The weight gradients are accumulated with lane =
// hidden unit (row i of dW2 and dW1), warp w taking columns 8w .. 8w+7 of dW2 and
// its share of the rest, each summing the 32 samples with no atomics.  At the
// end the block's gradient goes to its row of `part`, which the Adam kernel sums
// over blocks in a fixed order: the gradient is deterministic.
// Bound by the latency of its sums at the batch sizes of training: a warp that
// takes 32 samples by itself (k_mlp_grad_wide) needs 3,900 steps for them one after
// the other (batch of 4,096: 16.6 us on 32 SMs, and 6.2 us to sum over blocks).
// lbm_trainer_grad, gradient read back, 4,096 samples: 46.8 -> 33.6 us.
// Sample j of the batch is dataset row (a * (start + j) + c) mod n.
// ---------------------------------------------------------------------------
constexpr int TR_WARPS = 4;
constexpr int TR_THREADS = 32 * TR_WARPS;
constexpr int TR_OWN = CLO_HID / TR_WARPS;  // hidden units of a warp
constexpr int TR_LD = 36;   // row stride of the [32][36] tiles: float4 accesses of
                            // 8 lanes hit 32 distinct banks
constexpr int TR_XLD = 12;  // row stride of the inputs tile
constexpr int TR_MAX_BLOCKS = 592;  // four per SM
constexpr int TR_NET = (CLO_FLOATS + 3) / 4 * 4;  // 16-byte multiple: float4 tiles follow
static_assert(TR_LD % 4 == 0 && TR_XLD % 4 == 0 && CLO_W2 % 4 == 0 && CLO_HID * CLO_HID % 4 == 0 && TR_OWN == 8,
              "16-byte alignment of the float4 tiles");

struct Batch {
  const float* x;
  const float* t;
  const float* w;
  int64_t n;       // dataset rows
  int64_t start;   // position of the batch in the epoch order
  int64_t nb;      // samples in the batch
  uint64_t a, c;   // affine order: row = (a * pos + c) mod n
  float wscale;    // loss = wscale * sum w (r - t)^2
};

__global__ void __launch_bounds__(TR_THREADS, 4)
    k_mlp_grad(const float* __restrict__ net, Batch B, float* __restrict__ part,
               double* __restrict__ loss_part) {
  __shared__ __align__(16) float sw[TR_NET];                // the network
  __shared__ __align__(16) float sW2T[CLO_HID * CLO_HID];   // W2 transposed [j][i]
  __shared__ __align__(16) float sW1[CLO_HID * TR_XLD];     // W1 in rows of 12, the last three zero
  __shared__ __align__(16) float sH1[32 * TR_LD], sH2[32 * TR_LD], sA1[32 * TR_LD], sA2[32 * TR_LD];
  __shared__ __align__(16) float sX[32 * TR_XLD];           // standardised inputs
  __shared__ float sDZ[32], sZ[TR_WARPS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, own = warp * TR_OWN;

  for (int k = threadIdx.x; k < CLO_FLOATS; k += TR_THREADS) sw[k] = net[k];
  for (int k = threadIdx.x; k < CLO_HID * CLO_HID; k += TR_THREADS) {
    const int i = k / CLO_HID, j = k % CLO_HID;
    sW2T[j * CLO_HID + i] = net[CLO_W2 + k];
  }
  for (int k = threadIdx.x; k < CLO_HID * TR_XLD; k += TR_THREADS) {
    const int i = k / TR_XLD, j = k % TR_XLD;
    sW1[k] = j < CLO_IN ? net[CLO_W1 + i * CLO_IN + j] : 0.f;
  }
  __syncthreads();

  // lane = hidden unit i: dW2[i][own ..]; warp 0 dW1[i][0 .. 3], warp 1
  // dW1[i][4 .. 7], warp 2 dW1[i][8] and db1[i], warp 3 db2[i], dW3[i] and db3
  float gW2[TR_OWN], gr[4];
#pragma unroll
  for (int q = 0; q < TR_OWN; ++q) gW2[q] = 0.f;
#pragma unroll
  for (int q = 0; q < 4; ++q) gr[q] = 0.f;
  double lsum = 0.0;

  const int64_t groups = (B.nb + 31) / 32;
  for (int64_t gi = blockIdx.x; gi < groups; gi += gridDim.x) {
    // ---- forward, lane = sample ----
    const int64_t j = gi * 32 + lane;
    const bool valid = j < B.nb;
    float xs[TR_XLD];
#pragma unroll
    for (int k = 0; k < TR_XLD; ++k) xs[k] = 0.f;
    float tgt = 0.f, wt = 0.f;
    if (valid) {
      const uint64_t pos = (uint64_t)(B.start + j);
      const size_t row = (size_t)((B.a * pos + B.c) % (uint64_t)B.n);
#pragma unroll
      for (int k = 0; k < CLO_IN; ++k)
        xs[k] = (B.x[row * CLO_IN + k] - sw[CLO_MEAN + k]) * sw[CLO_ISCALE + k];
      tgt = B.t[row];
      wt = B.w[row];
    }
    float v[TR_OWN];
#pragma unroll
    for (int q = 0; q < TR_OWN; ++q) {
      const float4* wr = reinterpret_cast<const float4*>(sW1 + (own + q) * TR_XLD);
      const float4 w0 = wr[0], w1 = wr[1];
      float a = sw[CLO_B1 + own + q];
      a = fmaf(w0.w, xs[3], fmaf(w0.z, xs[2], fmaf(w0.y, xs[1], fmaf(w0.x, xs[0], a))));
      a = fmaf(w1.w, xs[7], fmaf(w1.z, xs[6], fmaf(w1.y, xs[5], fmaf(w1.x, xs[4], a))));
      a = fmaf(sW1[(own + q) * TR_XLD + 8], xs[8], a);
      v[q] = fmaxf(a, 0.f);
    }
    auto put8 = [&](float* tile) {  // the warp's eight units of this lane's sample
      *reinterpret_cast<float4*>(tile + lane * TR_LD + own) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(tile + lane * TR_LD + own + 4) = make_float4(v[4], v[5], v[6], v[7]);
    };
    put8(sH1);
    if (warp == 0) {
#pragma unroll
      for (int k = 0; k < TR_XLD; k += 4)
        *reinterpret_cast<float4*>(sX + lane * TR_XLD + k) = make_float4(xs[k], xs[k + 1], xs[k + 2], xs[k + 3]);
    }
    __syncthreads();
    float z = 0.f;
#pragma unroll
    for (int q = 0; q < TR_OWN; ++q) v[q] = sw[CLO_B2 + own + q];
#pragma unroll
    for (int j4 = 0; j4 < CLO_HID / 4; ++j4) {
      const float4 h = *reinterpret_cast<const float4*>(sH1 + lane * TR_LD + 4 * j4);
#pragma unroll
      for (int q = 0; q < TR_OWN; ++q) {
        const float4 w4 = *reinterpret_cast<const float4*>(sw + CLO_W2 + (own + q) * CLO_HID + 4 * j4);
        v[q] = fmaf(w4.w, h.w, fmaf(w4.z, h.z, fmaf(w4.y, h.y, fmaf(w4.x, h.x, v[q]))));
      }
    }
#pragma unroll
    for (int q = 0; q < TR_OWN; ++q) {
      v[q] = fmaxf(v[q], 0.f);
      z = fmaf(sw[CLO_W3 + own + q], v[q], z);
    }
    put8(sH2);
    sZ[warp][lane] = z;
    __syncthreads();
    // softplus output and the weighted squared error (in every warp: the same)
    z = sw[CLO_B3] + ((sZ[0][lane] + sZ[1][lane]) + (sZ[2][lane] + sZ[3][lane]));
    const float r = z > 20.f ? z : log1pf(expf(z));
    const float sig = 1.f / (1.f + expf(-z));
    const float e = r - tgt;
    const float dz = valid ? 2.f * B.wscale * wt * e * sig : 0.f;
    if (valid && warp == 0) lsum += (double)B.wscale * (double)wt * (double)e * (double)e;
    if (warp == 0) sDZ[lane] = dz;
#pragma unroll
    for (int q = 0; q < TR_OWN; ++q) v[q] = v[q] > 0.f ? sw[CLO_W3 + own + q] * dz : 0.f;
    put8(sA2);
    __syncthreads();
    // d a1_j = [a1_j > 0] sum_i W2[i][j] d a2_i  (W2 transposed: row j contiguous)
#pragma unroll
    for (int q = 0; q < TR_OWN; ++q) v[q] = 0.f;
#pragma unroll
    for (int i4 = 0; i4 < CLO_HID / 4; ++i4) {
      const float4 d = *reinterpret_cast<const float4*>(sA2 + lane * TR_LD + 4 * i4);
#pragma unroll
      for (int q = 0; q < TR_OWN; ++q) {
        const float4 w4 = *reinterpret_cast<const float4*>(sW2T + (own + q) * CLO_HID + 4 * i4);
        v[q] = fmaf(w4.w, d.w, fmaf(w4.z, d.z, fmaf(w4.y, d.y, fmaf(w4.x, d.x, v[q]))));
      }
    }
    {
      const float4 h0 = *reinterpret_cast<const float4*>(sH1 + lane * TR_LD + own);
      const float4 h1 = *reinterpret_cast<const float4*>(sH1 + lane * TR_LD + own + 4);
      const float h[TR_OWN] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
      for (int q = 0; q < TR_OWN; ++q) v[q] = h[q] > 0.f ? v[q] : 0.f;
    }
    put8(sA1);
    __syncthreads();
    // ---- weight gradients, lane = hidden unit ----
    auto sample = [&](int s) {  // dW2 of one sample; its d a2
      const float a2 = sA2[s * TR_LD + lane];
      const float4 h0 = *reinterpret_cast<const float4*>(sH1 + s * TR_LD + own);
      const float4 h1 = *reinterpret_cast<const float4*>(sH1 + s * TR_LD + own + 4);
      const float h[TR_OWN] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
      for (int q = 0; q < TR_OWN; ++q) gW2[q] = fmaf(a2, h[q], gW2[q]);
      return a2;
    };
    if (warp < 2) {
#pragma unroll 4
      for (int s = 0; s < 32; ++s) {
        sample(s);
        const float a1 = sA1[s * TR_LD + lane];
        const float4 x = *reinterpret_cast<const float4*>(sX + s * TR_XLD + 4 * warp);
        gr[0] = fmaf(a1, x.x, gr[0]);
        gr[1] = fmaf(a1, x.y, gr[1]);
        gr[2] = fmaf(a1, x.z, gr[2]);
        gr[3] = fmaf(a1, x.w, gr[3]);
      }
    } else if (warp == 2) {
#pragma unroll 4
      for (int s = 0; s < 32; ++s) {
        sample(s);
        const float a1 = sA1[s * TR_LD + lane];
        gr[0] = fmaf(a1, sX[s * TR_XLD + 8], gr[0]);
        gr[1] += a1;
      }
    } else {
#pragma unroll 4
      for (int s = 0; s < 32; ++s) {
        gr[0] += sample(s);
        gr[1] = fmaf(sDZ[s], sH2[s * TR_LD + lane], gr[1]);
        gr[2] += sDZ[s];
      }
    }
    __syncthreads();  // the tiles are rewritten by the next samples
  }

  float* row = part + (size_t)blockIdx.x * CLO_NPARAM;
#pragma unroll
  for (int q = 0; q < TR_OWN; ++q) row[CLO_W2 + lane * CLO_HID + own + q] = gW2[q];
  if (warp < 2) {
#pragma unroll
    for (int q = 0; q < 4; ++q) row[CLO_W1 + lane * CLO_IN + 4 * warp + q] = gr[q];
  } else if (warp == 2) {
    row[CLO_W1 + lane * CLO_IN + 8] = gr[0];
    row[CLO_B1 + lane] = gr[1];
  } else {
    row[CLO_B2 + lane] = gr[0];
    row[CLO_W3 + lane] = gr[1];
    if (lane == 0) row[CLO_B3] = gr[2];
  }
  if (warp == 0) {  // butterfly: the same order on every run
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) loss_part[blockIdx.x] = lsum;
  }
}

// The same for large batches: a warp takes 32 samples at a time by itself, lane =
// sample, the activations in registers, and leaves them and the pre-activation
// gradients in its own tiles for the weight gradients (lane = hidden unit i: row
// i of dW2 and dW1), which the block's warps add in order at the end.  A sample
// costs fewer shared loads than in k_mlp_grad, and with all SMs busy the length
// of a warp's chain no longer shows.  An optimiser step with batches of 16,384
// samples takes 26.5 us by k_mlp_grad and 27.4 by this one, of 32,768 36.4 and 29.3,
// 65,536 49.9 and 41.6, 262,144 134 and 105, 1,200,000 520 and 410; lbm_trainer_grad
// of 16,384 43.6 and 52.0, of 32,768 52.0 and 50.8: hence TR_WIDE.
constexpr int64_t TR_WIDE = 24576;
constexpr int TRW_MAX_BLOCKS = 296;  // two per SM
constexpr int TRW_WARP_FLOATS = 4 * 32 * TR_LD + 32 * TR_XLD + 32;
constexpr size_t TRW_SMEM = (size_t)(TR_NET + CLO_HID * CLO_HID + TR_WARPS * TRW_WARP_FLOATS) * 4;
static_assert(TRW_WARP_FLOATS % 4 == 0 && CLO_NPARAM <= TRW_WARP_FLOATS && TRW_MAX_BLOCKS <= TR_MAX_BLOCKS,
              "float4 tiles; a warp's gradient row fits them");

__global__ void __launch_bounds__(TR_THREADS, 2)
    k_mlp_grad_wide(const float* __restrict__ net, Batch B, float* __restrict__ part,
                    double* __restrict__ loss_part) {
  extern __shared__ __align__(16) float sm[];
  float* sw = sm;                                       // network [CLO_FLOATS] (padded)
  float* sW2T = sm + TR_NET;                            // W2 transposed [j][i]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* wb = sW2T + CLO_HID * CLO_HID + warp * TRW_WARP_FLOATS;
  float* sH1 = wb;                  // [32][TR_LD] h1 per sample
  float* sH2 = sH1 + 32 * TR_LD;    // h2
  float* sA1 = sH2 + 32 * TR_LD;    // d a1
  float* sA2 = sA1 + 32 * TR_LD;    // d a2
  float* sX = sA2 + 32 * TR_LD;     // [32][TR_XLD] standardised inputs
  float* sDZ = sX + 32 * TR_XLD;    // [32] d z

  for (int k = threadIdx.x; k < CLO_FLOATS; k += TR_THREADS) sw[k] = net[k];
  for (int k = threadIdx.x; k < CLO_HID * CLO_HID; k += TR_THREADS) {
    const int i = k / CLO_HID, j = k % CLO_HID;
    sW2T[j * CLO_HID + i] = net[CLO_W2 + k];
  }
  __syncthreads();

  float gW2[CLO_HID], gW1[CLO_IN];
#pragma unroll
  for (int j = 0; j < CLO_HID; ++j) gW2[j] = 0.f;
#pragma unroll
  for (int k = 0; k < CLO_IN; ++k) gW1[k] = 0.f;
  float gb1 = 0.f, gb2 = 0.f, gW3 = 0.f, gb3 = 0.f;
  double lsum = 0.0;

  const int64_t groups = (B.nb + 31) / 32;
  for (int64_t gi = (int64_t)blockIdx.x * TR_WARPS + warp; gi < groups;
       gi += (int64_t)gridDim.x * TR_WARPS) {
    // ---- forward and activation backward, lane = sample ----
    const int64_t j = gi * 32 + lane;
    const bool valid = j < B.nb;
    float xs[CLO_IN];
    float tgt = 0.f, wt = 0.f;
    if (valid) {
      const uint64_t pos = (uint64_t)(B.start + j);
      const size_t row = (size_t)((B.a * pos + B.c) % (uint64_t)B.n);
#pragma unroll
      for (int k = 0; k < CLO_IN; ++k)
        xs[k] = (B.x[row * CLO_IN + k] - sw[CLO_MEAN + k]) * sw[CLO_ISCALE + k];
      tgt = B.t[row];
      wt = B.w[row];
    } else {
#pragma unroll
      for (int k = 0; k < CLO_IN; ++k) xs[k] = 0.f;
    }
    float h1[CLO_HID];
#pragma unroll
    for (int i = 0; i < CLO_HID; ++i) {
      float a = sw[CLO_B1 + i];
#pragma unroll
      for (int k = 0; k < CLO_IN; ++k) a = fmaf(sw[CLO_W1 + i * CLO_IN + k], xs[k], a);
      h1[i] = fmaxf(a, 0.f);
    }
    float z = sw[CLO_B3];
    unsigned m2 = 0;
#pragma unroll
    for (int i = 0; i < CLO_HID; i += 4) {
      float h2v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4* wr = reinterpret_cast<const float4*>(sw + CLO_W2 + (i + q) * CLO_HID);
        float a = sw[CLO_B2 + i + q];
#pragma unroll
        for (int jj = 0; jj < CLO_HID / 4; ++jj) {
          const float4 w4 = wr[jj];
          a = fmaf(w4.x, h1[4 * jj], a);
          a = fmaf(w4.y, h1[4 * jj + 1], a);
          a = fmaf(w4.z, h1[4 * jj + 2], a);
          a = fmaf(w4.w, h1[4 * jj + 3], a);
        }
        h2v[q] = fmaxf(a, 0.f);
        if (a > 0.f) m2 |= 1u << (i + q);
        z = fmaf(sw[CLO_W3 + i + q], h2v[q], z);
      }
      *reinterpret_cast<float4*>(sH2 + lane * TR_LD + i) = make_float4(h2v[0], h2v[1], h2v[2], h2v[3]);
    }
#pragma unroll
    for (int i = 0; i < CLO_HID; i += 4)
      *reinterpret_cast<float4*>(sH1 + lane * TR_LD + i) = make_float4(h1[i], h1[i + 1], h1[i + 2], h1[i + 3]);
    // softplus output and the weighted squared error
    const float r = z > 20.f ? z : log1pf(expf(z));
    const float sig = 1.f / (1.f + expf(-z));
    const float e = r - tgt;
    const float dz = valid ? 2.f * B.wscale * wt * e * sig : 0.f;
    if (valid) lsum += (double)B.wscale * (double)wt * (double)e * (double)e;
    float da2[CLO_HID];
#pragma unroll
    for (int i = 0; i < CLO_HID; ++i) da2[i] = (m2 >> i & 1u) ? sw[CLO_W3 + i] * dz : 0.f;
#pragma unroll
    for (int i = 0; i < CLO_HID; i += 4)
      *reinterpret_cast<float4*>(sA2 + lane * TR_LD + i) = make_float4(da2[i], da2[i + 1], da2[i + 2], da2[i + 3]);
    // d a1_j = [a1_j > 0] sum_i W2[i][j] d a2_i  (W2 transposed: row j contiguous)
#pragma unroll
    for (int jq = 0; jq < CLO_HID; jq += 4) {
      float d[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int jj = jq + q;
        const float4* wr = reinterpret_cast<const float4*>(sW2T + jj * CLO_HID);
        float a = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < CLO_HID / 4; ++i4) {
          const float4 w4 = wr[i4];
          a = fmaf(w4.x, da2[4 * i4], a);
          a = fmaf(w4.y, da2[4 * i4 + 1], a);
          a = fmaf(w4.z, da2[4 * i4 + 2], a);
          a = fmaf(w4.w, da2[4 * i4 + 3], a);
        }
        d[q] = h1[jj] > 0.f ? a : 0.f;
      }
      *reinterpret_cast<float4*>(sA1 + lane * TR_LD + jq) = make_float4(d[0], d[1], d[2], d[3]);
    }
#pragma unroll
    for (int k = 0; k < CLO_IN; ++k) sX[lane * TR_XLD + k] = xs[k];
    sDZ[lane] = dz;
    __syncwarp();
    // ---- weight gradients, lane = hidden unit ----
    for (int s = 0; s < 32; ++s) {
      const float a2 = sA2[s * TR_LD + lane];
      const float a1 = sA1[s * TR_LD + lane];
      const float dzs = sDZ[s];
      const float4* h = reinterpret_cast<const float4*>(sH1 + s * TR_LD);
#pragma unroll
      for (int q = 0; q < CLO_HID / 4; ++q) {
        const float4 hv = h[q];
        gW2[4 * q] = fmaf(a2, hv.x, gW2[4 * q]);
        gW2[4 * q + 1] = fmaf(a2, hv.y, gW2[4 * q + 1]);
        gW2[4 * q + 2] = fmaf(a2, hv.z, gW2[4 * q + 2]);
        gW2[4 * q + 3] = fmaf(a2, hv.w, gW2[4 * q + 3]);
      }
#pragma unroll
      for (int k = 0; k < CLO_IN; ++k) gW1[k] = fmaf(a1, sX[s * TR_XLD + k], gW1[k]);
      gb1 += a1;
      gb2 += a2;
      gW3 = fmaf(dzs, sH2[s * TR_LD + lane], gW3);
      gb3 += dzs;
    }
    __syncwarp();
  }

  // ---- block reduction in a fixed order ----
  // loss: warp sum (butterfly, the same order on every run), then warps in order
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  __syncthreads();  // every warp is done with its tiles
  float* g = wb;    // this warp's gradient row, CLO_NPARAM floats (fits the tiles)
#pragma unroll
  for (int jj = 0; jj < CLO_HID; ++jj) g[CLO_W2 + lane * CLO_HID + jj] = gW2[jj];
#pragma unroll
  for (int k = 0; k < CLO_IN; ++k) g[CLO_W1 + lane * CLO_IN + k] = gW1[k];
  g[CLO_B1 + lane] = gb1;
  g[CLO_B2 + lane] = gb2;
  g[CLO_W3 + lane] = gW3;
  if (lane == 0) g[CLO_B3] = gb3;
  __shared__ double sl[TR_WARPS];
  if (lane == 0) sl[warp] = lsum;
  __syncthreads();
  const float* g0 = sW2T + CLO_HID * CLO_HID;
  for (int k = threadIdx.x; k < CLO_NPARAM; k += TR_THREADS) {
    float acc = g0[k];
#pragma unroll
    for (int w = 1; w < TR_WARPS; ++w) acc += g0[w * TRW_WARP_FLOATS + k];
    part[(size_t)blockIdx.x * CLO_NPARAM + k] = acc;
  }
  if (threadIdx.x == 0) {
    double l = 0.0;
    for (int w = 0; w < TR_WARPS; ++w) l += sl[w];
    loss_part[blockIdx.x] = l;
  }
}

struct AdamArgs {
  float lr, b1, b2, eps, wd;
  float bc1, bc2;   // 1 - beta^t
  int apply;        // 0: only reduce the gradient
  int set_loss;     // 1: the loss is set, 0: added to loss_acc
};

// Sums the block partials, then optionally one Adam step of the fp32 master
// parameters; writes the network the kernels use (weights rounded to bf16).  A
// block takes 32 parameters, its eight warps every eighth block's partial, and
// adds the warps' sums in order: the same result on every run, in an eighth of
// the loads one after the other.  The first block adds the batch loss to
// loss_acc (or sets it).
constexpr int ADAM_THREADS = 256;
__global__ void __launch_bounds__(ADAM_THREADS)
    k_adam(const float* __restrict__ part, int nblk, const double* __restrict__ loss_part,
           double* __restrict__ loss_acc, float* __restrict__ grad,
           float* __restrict__ theta, float* __restrict__ m, float* __restrict__ v,
           float* __restrict__ net, AdamArgs A) {
  __shared__ float sums[ADAM_THREADS / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  if (blockIdx.x == 0 && warp == 1) {
    double l = 0.0;
    for (int b = lane; b < nblk; b += 32) l += loss_part[b];
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0) *loss_acc = A.set_loss ? l : *loss_acc + l;
  }
  float gk = 0.f;
  if (k < CLO_NPARAM) {
#pragma unroll 8
    for (int b = warp; b < nblk; b += ADAM_THREADS / 32) gk += part[(size_t)b * CLO_NPARAM + k];
  }
  sums[warp][lane] = gk;
  __syncthreads();
  if (warp != 0 || k >= CLO_NPARAM) return;
#pragma unroll
  for (int w = 1; w < ADAM_THREADS / 32; ++w) gk += sums[w][lane];
  grad[k] = gk;
  if (!A.apply) return;
  const float mk = A.b1 * m[k] + (1.f - A.b1) * gk;
  const float vk = A.b2 * v[k] + (1.f - A.b2) * gk * gk;
  m[k] = mk;
  v[k] = vk;
  float th = theta[k];
  const bool wgt = clo_is_weight(k);
  if (wgt && A.wd > 0.f) th -= A.lr * A.wd * th;
  th -= A.lr * (mk / A.bc1) / (sqrtf(vk / A.bc2) + A.eps);
  theta[k] = th;
  net[k] = wgt ? __bfloat162float(__float2bfloat16_rn(th)) : th;
}

__global__ void k_wsum(const float* __restrict__ w, int64_t n, double* __restrict__ out) {
  __shared__ double s[256];
  double a = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a += w[i];
  s[threadIdx.x] = a;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = s[0];
}

}  // namespace
}  // namespace lbm

using namespace lbm;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
struct lbm_trainer {
  lbm_adam opt{};
  cudaStream_t stream = nullptr;
  char* mem = nullptr;      // all of the device buffers below
  float* theta = nullptr;   // fp32 master parameters [CLO_NPARAM]
  float* m = nullptr;
  float* v = nullptr;
  float* grad = nullptr;    // last reduced gradient (behind loss_acc, in its allocation)
  float* net = nullptr;     // network the kernels use [CLO_FLOATS]
  float* part = nullptr;    // [TR_MAX_BLOCKS][CLO_NPARAM]
  double* loss_part = nullptr;
  double* loss_acc = nullptr;
  double* wpart = nullptr;  // [TR_MAX_BLOCKS]
  char host[8 + CLO_NPARAM * 4];  // loss, gradient, as they are read back
  int64_t t = 0;            // Adam steps taken
  std::string err = "no error";
};

namespace {

thread_local std::string g_clo_err = "no error";

int tfail(lbm_trainer* t, int code, const std::string& msg) {
  if (t) t->err = msg;
  g_clo_err = msg;
  set_thread_error(msg.c_str());
  return code;
}

int tcuda(lbm_trainer* t, cudaError_t e, const char* what) {
  const int code = e == cudaErrorMemoryAllocation ? LBM_ERR_OUT_OF_MEMORY
                   : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? LBM_ERR_NO_DEVICE
                                                                                  : LBM_ERR_CUDA;
  return tfail(t, code, std::string(what) + ": " + cudaGetErrorString(e));
}

#define TCK(t, expr, what)                              \
  do {                                                  \
    cudaError_t e_ = (expr);                            \
    if (e_ != cudaSuccess) return tcuda(t, e_, what);   \
  } while (0)

// blocks for nb samples, `each` of them a block, `most` blocks at the most
int grid_for(int64_t nb, int64_t each, int most) {
  const int64_t blocks = (nb + each - 1) / each;
  return (int)(blocks < 1 ? 1 : blocks > most ? most : blocks);
}

int launch_grad(lbm_trainer* t, const Batch& B, int* nblk) {
  int g;
  if (B.nb < TR_WIDE) {
    g = grid_for(B.nb, 32, TR_MAX_BLOCKS);
    k_mlp_grad<<<g, TR_THREADS, 0, t->stream>>>(t->net, B, t->part, t->loss_part);
  } else {
    g = grid_for(B.nb, 32 * TR_WARPS, TRW_MAX_BLOCKS);
    TCK(t, cudaFuncSetAttribute(k_mlp_grad_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRW_SMEM),
        "closure grad kernel attribute");
    k_mlp_grad_wide<<<g, TR_THREADS, TRW_SMEM, t->stream>>>(t->net, B, t->part, t->loss_part);
  }
  TCK(t, cudaGetLastError(), "closure grad kernel");
  *nblk = g;
  return LBM_OK;
}

int launch_adam(lbm_trainer* t, int nblk, bool apply, bool set_loss) {
  AdamArgs A{};
  A.lr = t->opt.lr;
  A.b1 = t->opt.beta1;
  A.b2 = t->opt.beta2;
  A.eps = t->opt.eps;
  A.wd = t->opt.weight_decay;
  A.apply = apply ? 1 : 0;
  A.set_loss = set_loss ? 1 : 0;
  if (apply) {
    t->t += 1;
    A.bc1 = (float)(1.0 - std::pow((double)A.b1, (double)t->t));
    A.bc2 = (float)(1.0 - std::pow((double)A.b2, (double)t->t));
  } else {
    A.bc1 = A.bc2 = 1.f;
  }
  k_adam<<<(CLO_NPARAM + 31) / 32, ADAM_THREADS, 0, t->stream>>>(t->part, nblk, t->loss_part, t->loss_acc,
                                                          t->grad, t->theta, t->m, t->v, t->net, A);
  TCK(t, cudaGetLastError(), "closure adam kernel");
  return LBM_OK;
}

}  // namespace

extern "C" {

int lbm_round_bf16(const float* in, float* out, size_t n) {
  if ((!in || !out) && n) return LBM_ERR_INVALID_ARG;
  for (size_t i = 0; i < n; ++i) out[i] = round_bf16(in[i]);
  return LBM_OK;
}

int lbm_box_filter(const float* d_rho, const float* d_u, int32_t nx, int32_t ny, int32_t nz,
                   int32_t factor, float* d_out, void* stream) {
  if (!d_rho || !d_u || !d_out) return tfail(nullptr, LBM_ERR_INVALID_ARG, "box filter: NULL pointer");
  if (factor < 1 || nx < factor || ny < factor || nz < factor || nx % factor || ny % factor || nz % factor)
    return tfail(nullptr, LBM_ERR_INVALID_ARG, "box filter: factor must divide nx, ny and nz");
  const size_t nc = (size_t)(nx / factor) * (ny / factor) * (nz / factor);
  // Vector loads where every box row starts on their boundary: the factor a
  // multiple of their width (then so are nx and n) and both fields aligned.
  auto aligned = [&](size_t bytes) {
    return ((reinterpret_cast<uintptr_t>(d_rho) | reinterpret_cast<uintptr_t>(d_u)) & (bytes - 1)) == 0;
  };
  // Blocks of 64: at 256^3 / 4 a thread's 64 registers allow 1,024 a SM, and 256
  // threads a block left the second wave three quarters empty (55.8 us).
  const unsigned grd = (unsigned)((nc + 63) / 64);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (factor == 4 && aligned(16)) k_box_filter<4, 4><<<grd, 64, 0, s>>>(d_rho, d_u, nx, ny, nz, factor, d_out);
  else if (factor == 2 && aligned(8)) k_box_filter<2, 2><<<grd, 64, 0, s>>>(d_rho, d_u, nx, ny, nz, factor, d_out);
  else if (factor % 4 == 0 && aligned(16)) k_box_filter<4, 0><<<grd, 64, 0, s>>>(d_rho, d_u, nx, ny, nz, factor, d_out);
  else if (factor % 2 == 0 && aligned(8)) k_box_filter<2, 0><<<grd, 64, 0, s>>>(d_rho, d_u, nx, ny, nz, factor, d_out);
  else k_box_filter_any<<<(unsigned)((nc + 255) / 256), 256, 0, s>>>(d_rho, d_u, nx, ny, nz, factor, d_out);
  TCK(nullptr, cudaGetLastError(), "box filter kernel");
  return LBM_OK;
}

int lbm_closure_samples(const float* d_filt, int32_t nx, int32_t ny, int32_t nz, float tau, float cs0,
                        uint64_t seed, int64_t n_samples, float* d_x, float* d_target, float* d_weight,
                        void* stream) {
  if (!d_filt || !d_x || !d_target || !d_weight)
    return tfail(nullptr, LBM_ERR_INVALID_ARG, "closure samples: NULL pointer");
  if (nx < 3 || ny < 3 || nz < 3) return tfail(nullptr, LBM_ERR_INVALID_ARG, "closure samples: grid below 3^3");
  if (!(cs0 > 0.f) || !(tau > 0.5f)) return tfail(nullptr, LBM_ERR_INVALID_ARG, "closure samples: need cs0 > 0, tau > 1/2");
  const int64_t n = (int64_t)nx * ny * nz;
  if (n_samples < 0 || (seed == 0 && n_samples > n))
    return tfail(nullptr, LBM_ERR_INVALID_ARG, "closure samples: bad sample count");
  if (n_samples == 0) return LBM_OK;
  // blocks of 64: a snapshot's few thousand samples spread over the chip
  k_samples<<<(unsigned)((n_samples + 63) / 64), 64, 0, static_cast<cudaStream_t>(stream)>>>(
      d_filt, nx, ny, nz, tau, cs0, seed, n_samples, d_x, d_target, d_weight);
  TCK(nullptr, cudaGetLastError(), "closure samples kernel");
  return LBM_OK;
}

int lbm_closure_predict(const float* net, const float* d_x, int64_t n, float* d_r, void* stream) {
  if (!net || !d_x || !d_r) return tfail(nullptr, LBM_ERR_INVALID_ARG, "closure predict: NULL pointer");
  if (n <= 0) return n == 0 ? LBM_OK : tfail(nullptr, LBM_ERR_INVALID_ARG, "closure predict: n < 0");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float h[CLO_FLOATS];
  for (int k = 0; k < CLO_FLOATS; ++k) h[k] = clo_is_weight(k) ? round_bf16(net[k]) : net[k];
  float* d_net = nullptr;
  TCK(nullptr, cudaMallocAsync(reinterpret_cast<void**>(&d_net), sizeof(h), s), "closure predict alloc");
  cudaError_t e = cudaMemcpyAsync(d_net, h, sizeof(h), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    k_predict<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_net, d_x, n, d_r);
    e = cudaGetLastError();
  }
  cudaError_t e2 = cudaFreeAsync(d_net, s);
  cudaError_t e3 = cudaStreamSynchronize(s);  // h is a stack buffer
  if (e != cudaSuccess) return tcuda(nullptr, e, "closure predict");
  if (e2 != cudaSuccess) return tcuda(nullptr, e2, "closure predict free");
  TCK(nullptr, e3, "closure predict sync");
  return LBM_OK;
}

int lbm_adam_default(lbm_adam* a) {
  if (!a) return LBM_ERR_INVALID_ARG;
  *a = lbm_adam{};
  a->struct_size = sizeof(lbm_adam);
  a->lr = 1e-3f;
  a->beta1 = 0.9f;
  a->beta2 = 0.999f;
  a->eps = 1e-8f;
  a->weight_decay = 0.f;
  return LBM_OK;
}

int lbm_trainer_create(const float* net, const lbm_adam* opt, lbm_trainer** out) {
  if (!net || !out) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer: NULL pointer");
  *out = nullptr;
  lbm_adam o;
  lbm_adam_default(&o);
  if (opt) {
    if (opt->struct_size != sizeof(lbm_adam)) return tfail(nullptr, LBM_ERR_INVALID_ARG, "lbm_adam struct_size");
    o = *opt;
  }
  if (!(o.lr > 0.f) || !(o.beta1 >= 0.f && o.beta1 < 1.f) || !(o.beta2 >= 0.f && o.beta2 < 1.f) ||
      !(o.eps > 0.f) || !(o.weight_decay >= 0.f))
    return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer: bad Adam hyper-parameters");
  for (int k = 0; k < CLO_FLOATS; ++k)
    if (!std::isfinite(net[k])) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer: non-finite network value");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return tfail(nullptr, LBM_ERR_NO_DEVICE, "trainer: no CUDA device");
  lbm_trainer* t = new (std::nothrow) lbm_trainer();
  if (!t) return tfail(nullptr, LBM_ERR_OUT_OF_MEMORY, "trainer: host allocation");
  t->opt = o;
  // One allocation: eight of their own, one of them over 2 MB, made a trainer
  // 1.55 ms to set up, against 1.2 ms as one.
  struct A { void** p; size_t bytes; } parts[] = {
      {reinterpret_cast<void**>(&t->theta), CLO_NPARAM * 4}, {reinterpret_cast<void**>(&t->m), CLO_NPARAM * 4},
      {reinterpret_cast<void**>(&t->v), CLO_NPARAM * 4},
      {reinterpret_cast<void**>(&t->net), CLO_FLOATS * 4},
      {reinterpret_cast<void**>(&t->part), (size_t)TR_MAX_BLOCKS * CLO_NPARAM * 4},
      {reinterpret_cast<void**>(&t->loss_part), TR_MAX_BLOCKS * 8},
      {reinterpret_cast<void**>(&t->loss_acc), 8 + CLO_NPARAM * 4}, {reinterpret_cast<void**>(&t->wpart), TR_MAX_BLOCKS * 8}};
  auto padded = [](size_t b) { return (b + 255) / 256 * 256; };
  size_t total = 0;
  for (const A& a : parts) total += padded(a.bytes);
  if (cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&t->mem), total)) {
    const int rc = tcuda(nullptr, e, "trainer: cudaMalloc");
    lbm_trainer_destroy(t);
    return rc;
  }
  size_t off = 0;
  for (const A& a : parts) {
    *a.p = t->mem + off;
    off += padded(a.bytes);
  }
  t->grad = reinterpret_cast<float*>(t->loss_acc + 1);
  std::vector<float> h(CLO_FLOATS);
  for (int k = 0; k < CLO_FLOATS; ++k) h[k] = clo_is_weight(k) ? round_bf16(net[k]) : net[k];
  cudaError_t e = cudaMemcpy(t->theta, net, CLO_NPARAM * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t->net, h.data(), CLO_FLOATS * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(t->m, 0, CLO_NPARAM * 4);
  if (e == cudaSuccess) e = cudaMemset(t->v, 0, CLO_NPARAM * 4);
  if (e == cudaSuccess) e = cudaMemset(t->grad, 0, CLO_NPARAM * 4);
  if (e != cudaSuccess) {
    const int rc = tcuda(nullptr, e, "trainer: initial upload");
    lbm_trainer_destroy(t);
    return rc;
  }
  *out = t;
  return LBM_OK;
}

int lbm_trainer_destroy(lbm_trainer* t) {
  if (!t) return LBM_OK;
  if (t->mem) cudaFree(t->mem);
  delete t;
  return LBM_OK;
}

int lbm_trainer_set_stream(lbm_trainer* t, void* stream) {
  if (!t) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer is NULL");
  TCK(t, cudaStreamSynchronize(t->stream), "trainer set_stream sync");
  t->stream = static_cast<cudaStream_t>(stream);
  return LBM_OK;
}

int lbm_trainer_grad(lbm_trainer* t, const float* d_x, const float* d_target, const float* d_weight,
                     int64_t n, float wscale, float* grad, double* loss) {
  if (!t) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer is NULL");
  if (!d_x || !d_target || !d_weight || n <= 0) return tfail(t, LBM_ERR_INVALID_ARG, "trainer grad: bad batch");
  Batch B{d_x, d_target, d_weight, n, 0, n, 1, 0, wscale};
  int nblk = 0;
  if (int rc = launch_grad(t, B, &nblk)) return rc;
  if (int rc = launch_adam(t, nblk, false, true)) return rc;
  // gradient and loss in one copy
  TCK(t, cudaMemcpyAsync(t->host, t->loss_acc, 8 + CLO_NPARAM * 4, cudaMemcpyDeviceToHost, t->stream), "trainer grad: read");
  TCK(t, cudaStreamSynchronize(t->stream), "trainer grad: sync");
  if (grad) std::memcpy(grad, t->host + 8, CLO_NPARAM * 4);
  if (loss) std::memcpy(loss, t->host, 8);
  return LBM_OK;
}

int lbm_trainer_adam_step(lbm_trainer* t) {
  if (!t) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer is NULL");
  // the reduced gradient of the last lbm_trainer_grad becomes the single
  // partial row that the Adam kernel sums
  TCK(t, cudaMemcpyAsync(t->part, t->grad, CLO_NPARAM * 4, cudaMemcpyDeviceToDevice, t->stream), "trainer adam: stage");
  TCK(t, cudaMemsetAsync(t->loss_part, 0, 8, t->stream), "trainer adam: loss");
  if (int rc = launch_adam(t, 1, true, false)) return rc;
  return LBM_OK;
}

int lbm_trainer_fit(lbm_trainer* t, const float* d_x, const float* d_target, const float* d_weight,
                    int64_t n, int32_t batch, int32_t epochs, uint64_t seed, double* epoch_loss) {
  if (!t) return tfail(nullptr, LBM_ERR_INVALID_ARG, "trainer is NULL");
  if (!d_x || !d_target || !d_weight || n <= 0 || batch <= 0 || epochs < 0)
    return tfail(t, LBM_ERR_INVALID_ARG, "trainer fit: bad arguments");
  // mean weight of the dataset
  const int wb = (int)std::min<int64_t>(TR_MAX_BLOCKS, (n + 255) / 256);
  k_wsum<<<wb, 256, 0, t->stream>>>(d_weight, n, t->wpart);
  TCK(t, cudaGetLastError(), "trainer fit: weight sum");
  std::vector<double> wp(wb);
  TCK(t, cudaMemcpyAsync(wp.data(), t->wpart, wb * 8, cudaMemcpyDeviceToHost, t->stream), "trainer fit: read weight sum");
  TCK(t, cudaStreamSynchronize(t->stream), "trainer fit: sync");
  double wsum = 0.0;
  for (double v : wp) wsum += v;
  if (!(wsum > 0.0) || !std::isfinite(wsum)) return tfail(t, LBM_ERR_INVALID_ARG, "trainer fit: weights sum to <= 0");
  const double wmean = wsum / (double)n;
  uint64_t rs = seed * 0x9e3779b97f4a7c15ull + 0x632be59bd9b4e019ull;
  auto next = [&rs]() {  // splitmix64
    uint64_t z = (rs += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
  };
  auto gcd = [](uint64_t a, uint64_t b) {
    while (b) { const uint64_t r = a % b; a = b; b = r; }
    return a;
  };
  for (int ep = 0; ep < epochs; ++ep) {
    uint64_t a = 1, c = 0;
    if (n > 1) {
      do { a = 1 + next() % (uint64_t)(n - 1); } while (gcd(a, (uint64_t)n) != 1);
      c = next() % (uint64_t)n;
    }
    TCK(t, cudaMemsetAsync(t->loss_acc, 0, 8, t->stream), "trainer fit: reset loss");
    int64_t nbatches = 0;
    for (int64_t s = 0; s < n; s += batch) {
      const int64_t nb = std::min<int64_t>(batch, n - s);
      Batch B{d_x, d_target, d_weight, n, s, nb, a, c, (float)(1.0 / (wmean * (double)nb))};
      int nblk = 0;
      if (int rc = launch_grad(t, B, &nblk)) return rc;
      if (int rc = launch_adam(t, nblk, true, false)) return rc;
      ++nbatches;
    }
    if (epoch_loss) {
      double l = 0.0;
      TCK(t, cudaMemcpyAsync(&l, t->loss_acc, 8, cudaMemcpyDeviceToHost, t->stream), "trainer fit: read loss");
      TCK(t, cudaStreamSynchronize(t->stream), "trainer fit: sync");
      epoch_loss[ep] = l / (double)nbatches;
    }
  }
  TCK(t, cudaStreamSynchronize(t->stream), "trainer fit: sync");
  return LBM_OK;
}

int lbm_trainer_get_net(lbm_trainer* t, float* net) {
  if (!t || !net) return tfail(t, LBM_ERR_INVALID_ARG, "trainer get_net: NULL pointer");
  TCK(t, cudaMemcpyAsync(net, t->net, CLO_FLOATS * 4, cudaMemcpyDeviceToHost, t->stream), "trainer get_net");
  TCK(t, cudaStreamSynchronize(t->stream), "trainer get_net: sync");
  return LBM_OK;
}

const char* lbm_trainer_last_error(lbm_trainer* t) { return t ? t->err.c_str() : g_clo_err.c_str(); }

}  // extern "C"
