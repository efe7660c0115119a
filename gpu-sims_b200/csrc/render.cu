// Velocity-magnitude volume raymarch into a headless RGBA buffer: one or two
// lanes per pixel.  Restates the reference's velmag fragment pass (volumetric-grid/
// lattice-boltzmann/shaders/velmag.frag.glsl:44-96, uniforms from
// src/main.cpp:1720-1731, LUTs src/main.cpp:529-573, full-screen triangle
// shaders/fullscreen.vert.glsl) without a graphics API: no swapchain,
// window or sampler objects; the image lands in device memory.
//
// Pixel (px, py), row py from the top, is the fragment at
// v_uv = ((px + 1/2) / W, (py + 1/2) / H).  The three samplers are evaluated
// in fp32 with every operation rounded on its own: the velocity field
// trilinear with clamp to edge (texel centres at i + 1/2, u rounded to
// binary16 first when round_f16, as the rgba16f image holds it), the colour
// LUT linear along t (its rows are equal), the 256 x 256 jitter LUT at texel
// centres with clamp to edge (so pixels beyond 255 repeat the edge, as the
// reference's clamp-to-edge sampler does).  exp is this file's own
// (Cody-Waite reduction, degree-7 Taylor polynomial, exact power-of-two
// scale), so the oracle can evaluate the same operations and the images
// agree bit for bit.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <type_traits>

#include "colormap.h"
#include "lbm_internal.h"

namespace lbm {
namespace {

struct RenderArgs {
  float m[16];        // inverse view-projection, column-major (m[4*col + row])
  float cam[3];
  float vmin[3], vmax[3];
  int steps;
  float absorption, mag_min, mag_max, exposure;
  int width, height;
  float inv_ext[3];   // 1 / extent where the extent is a power of two, else 0
};

// The colour table as the shader samples it: bytes / 255, divided at compile time.
struct ColorTable {
  float4 e[256];
};
constexpr ColorTable color_table() {
  ColorTable t{};
  for (int i = 0; i < 256; ++i) {
    const ColormapEntry c = colormap_entry(i);
    t.e[i] = float4{(float)c.rgb[0] / 255.0f, (float)c.rgb[1] / 255.0f, (float)c.rgb[2] / 255.0f, 0.0f};
  }
  return t;
}
__device__ const ColorTable COLORS = color_table();

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float dv(float a, float b) { return __fdiv_rn(a, b); }

// e^x for x <= 0: x = n ln2 + r (ln2 split in a 16-bit head and a tail),
// e^r by its Taylor series to r^7 in Horner form, times 2^n built from bits.
__device__ float exp_neg(float x) {
  if (!(x > -87.0f)) return 0.0f;
  const float n = rintf(mul(x, 1.44269502f));
  const float r = sub(sub(x, mul(n, 0.693145751953125f)), mul(n, 1.42860677e-06f));
  float p = 1.0f / 5040.0f;
  p = add(mul(p, r), 1.0f / 720.0f);
  p = add(mul(p, r), 1.0f / 120.0f);
  p = add(mul(p, r), 1.0f / 24.0f);
  p = add(mul(p, r), 1.0f / 6.0f);
  p = add(mul(p, r), 0.5f);
  p = add(mul(p, r), 1.0f);
  p = add(mul(p, r), 1.0f);
  return mul(p, __int_as_float(((int)n + 127) << 23));
}

// jitter LUT byte k: the (k+1)-th state of the LCG s' = 1664525 s + 1013904223
// from s = 0x9E3779B9, top byte; the k+1 steps composed by squaring.
__device__ unsigned jitter_byte(unsigned k) {
  unsigned A = 1u, C = 0u;              // accumulated map s -> A s + C
  unsigned a = 1664525u, c = 1013904223u;
  unsigned e = k + 1u;
  while (e) {
    if (e & 1u) { C = a * C + c; A = a * A; }
    c = a * c + c;
    a = a * a;
    e >>= 1;
  }
  return ((A * 0x9E3779B9u + C) >> 24) & 0xFFu;
}

__device__ __forceinline__ float lerp_rn(float a, float b, float t) { return add(a, mul(t, sub(b, a))); }

// I: index type of a plane (32 bits for fields of fewer than 2^31 nodes).
// F16: u rounded to binary16.
template <class I, bool F16>
struct Vol {
  const float* u;
  int nx, ny, nz;
  size_t n;
};

template <class I, bool F16>
__device__ __forceinline__ float texel(const Vol<I, F16>&, const float* __restrict__ plane, I at) {
  const float v = __ldg(plane + at);
  return F16 ? __half2float(__float2half_rn(v)) : v;
}

__device__ __forceinline__ void axis(float ctr, int N, int& i0, int& i1, float& a) {
  const float u = sub(mul(ctr, (float)N), 0.5f);
  const float f = floorf(u);
  a = sub(u, f);
  const int lo = (int)f, hi = lo + 1;
  i0 = lo < 0 ? 0 : (lo > N - 1 ? N - 1 : lo);
  i1 = hi < 0 ? 0 : (hi > N - 1 ? N - 1 : hi);
}

template <class I, bool F16>
__device__ __forceinline__ void sample_u(const Vol<I, F16>& V, float cx, float cy, float cz, float out[3]) {
  int x0, x1, y0, y1, z0, z1;
  float ax, ay, az;
  axis(cx, V.nx, x0, x1, ax);
  axis(cy, V.ny, y0, y1, ay);
  axis(cz, V.nz, z0, z1, az);
  const I r00 = (I)V.nx * ((I)y0 + (I)V.ny * (I)z0), r10 = (I)V.nx * ((I)y1 + (I)V.ny * (I)z0);
  const I r01 = (I)V.nx * ((I)y0 + (I)V.ny * (I)z1), r11 = (I)V.nx * ((I)y1 + (I)V.ny * (I)z1);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float* p = V.u + (size_t)c * V.n;
    const float c00 = lerp_rn(texel(V, p, r00 + x0), texel(V, p, r00 + x1), ax);
    const float c10 = lerp_rn(texel(V, p, r10 + x0), texel(V, p, r10 + x1), ax);
    const float c01 = lerp_rn(texel(V, p, r01 + x0), texel(V, p, r01 + x1), ax);
    const float c11 = lerp_rn(texel(V, p, r11 + x0), texel(V, p, r11 + x1), ax);
    out[c] = lerp_rn(lerp_rn(c00, c10, ay), lerp_rn(c01, c11, ay), az);
  }
}

// One or two lanes a ray (two_lanes).  A sample is some 400 dependent instructions
// and a ray up to `steps` of them in sequence, so with a lane a ray the image waits
// for its longest rays; the samples themselves do not depend on each other.  Of
// two lanes each takes every other sample (its t by the same additions), and they
// composite each pair in order from one another's colours, with the same
// operations as one lane alone.  More lanes spend the gain on samples beyond the
// end of rays that saturate early: 1280 x 720 over 128^3, 128 steps, 1 / 2 / 4 lanes:
// 350 / 290 / 292 us.
//
// The colour table lies in shared memory: the rays of a warp read different
// entries, which kernel parameter space serves one after the other (one lane a
// ray: 415 -> 350 us).  A block copies it from global memory, where it lies divided
// by 255 at compile time; making it from kernel parameters in every block took
// 70 us of a 1920 x 1080 image of any length (1 step 120 -> 35 us).  Blocks that no
// ray of theirs enters the volume from stop there.  An extent that is a power of
// two divides by an exact product.
constexpr int TILE_X = 8;
template <int RAY_LANES> constexpr int tile_y() { return 32 / RAY_LANES; }  // pixels of a block of 256 threads

template <class I, bool F16, int RAY_LANES>
__global__ void __launch_bounds__(256)
    k_velmag(Vol<I, F16> V, const __grid_constant__ RenderArgs R, float4* __restrict__ out) {
  __shared__ float4 lut[256];
  constexpr int TILE_Y = tile_y<RAY_LANES>();
  static_assert(TILE_X * TILE_Y * RAY_LANES == 256, "one table entry a thread");
  lut[threadIdx.x] = COLORS.e[threadIdx.x];
  const int q = threadIdx.x / RAY_LANES, l = threadIdx.x % RAY_LANES;
  const unsigned tiles_x = (unsigned)(R.width + TILE_X - 1) / TILE_X;
  const int px = (int)(blockIdx.x % tiles_x) * TILE_X + q % TILE_X;
  const int py = (int)(blockIdx.x / tiles_x) * TILE_Y + q / TILE_X;
  // ray through the fragment's far-plane point
  const float ndc[4] = {sub(mul(dv(add((float)px, 0.5f), (float)R.width), 2.0f), 1.0f),
                        sub(mul(dv(add((float)py, 0.5f), (float)R.height), 2.0f), 1.0f), 1.0f, 1.0f};
  float w4[4];
  for (int r = 0; r < 4; ++r)
    w4[r] = add(add(add(mul(R.m[r], ndc[0]), mul(R.m[4 + r], ndc[1])), mul(R.m[8 + r], ndc[2])),
                mul(R.m[12 + r], ndc[3]));
  float rd[3];
  for (int c = 0; c < 3; ++c) rd[c] = sub(dv(w4[c], w4[3]), R.cam[c]);
  const float len = __fsqrt_rn(add(add(mul(rd[0], rd[0]), mul(rd[1], rd[1])), mul(rd[2], rd[2])));
  for (int c = 0; c < 3; ++c) rd[c] = dv(rd[c], len);
  // slab intersection
  float te = -INFINITY, tx = INFINITY;
  for (int c = 0; c < 3; ++c) {
    const float inv = dv(1.0f, rd[c]);
    const float t0 = mul(sub(R.vmin[c], R.cam[c]), inv);
    const float t1 = mul(sub(R.vmax[c], R.cam[c]), inv);
    te = fmaxf(te, fminf(t0, t1));
    tx = fminf(tx, fmaxf(t0, t1));
  }
  const bool pixel = px < R.width && py < R.height;
  const bool hit = pixel && !(tx < te || tx < 0.0f);
  const float t0 = fmaxf(te, 0.0f);
  const float ray = sub(tx, t0);
  if (!__syncthreads_or(hit)) {  // also: the table is complete
    if (pixel && l == 0) out[(size_t)py * R.width + px] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  float jitter = 0.0f;
  if (hit) {
    const unsigned jx = px > 255 ? 255u : (unsigned)px, jy = py > 255 ? 255u : (unsigned)py;
    jitter = dv((float)jitter_byte(jy * 256u + jx), 255.0f);
  }
  const float dt = dv(ray, (float)R.steps);
  float t = add(t0, mul(jitter, dt));
  for (int k = 0; k < l; ++k) t = add(t, dt);
  float col[3] = {0.f, 0.f, 0.f};
  float trans = 1.0f;
  float ext[3];
  for (int c = 0; c < 3; ++c) ext[c] = sub(R.vmax[c], R.vmin[c]);
  const float range = fmaxf(sub(R.mag_max, R.mag_min), 1e-6f);
  for (int i = 0;; i += RAY_LANES) {
    const bool on = hit && i < R.steps && trans > 0.01f;  // the same in a ray's lanes
    if (!__any_sync(0xffffffffu, on)) break;
    bool inside = on && i + l < R.steps;
    float cc[3] = {0.f, 0.f, 0.f}, abs_step = 0.0f, pass = 1.0f;
    if (inside) {
      float uvw[3];
      for (int c = 0; c < 3; ++c) {
        const float p = sub(add(R.cam[c], mul(rd[c], t)), R.vmin[c]);
        uvw[c] = R.inv_ext[c] != 0.0f ? mul(p, R.inv_ext[c]) : dv(p, ext[c]);
        inside &= uvw[c] >= 0.0f && uvw[c] <= 1.0f;
      }
      if (inside) {
        float u[3];
        sample_u(V, uvw[0], uvw[1], uvw[2], u);
        const float mag = __fsqrt_rn(add(add(mul(u[0], u[0]), mul(u[1], u[1])), mul(u[2], u[2])));
        const float t01 = fminf(fmaxf(dv(sub(mag, R.mag_min), range), 0.0f), 1.0f);
        // colour LUT: linear filter along the 256 texels, clamp to edge
        const float lu = sub(mul(t01, 256.0f), 0.5f);
        const float lf = floorf(lu);
        const float la = sub(lu, lf);
        const int l0 = lf < 0.f ? 0 : ((int)lf > 255 ? 255 : (int)lf);
        const int l1 = (int)lf + 1 < 0 ? 0 : ((int)lf + 1 > 255 ? 255 : (int)lf + 1);
        abs_step = mul(mul(R.absorption, dt), t01);
        const float4 e0 = lut[l0], e1 = lut[l1];
        cc[0] = lerp_rn(e0.x, e1.x, la);
        cc[1] = lerp_rn(e0.y, e1.y, la);
        cc[2] = lerp_rn(e0.z, e1.z, la);
        pass = exp_neg(-abs_step);
      }
    }
    const unsigned in = __ballot_sync(0xffffffffu, inside) >> (threadIdx.x & 31 & ~(RAY_LANES - 1));
#pragma unroll
    for (int k = 0; k < RAY_LANES; ++k) {
      const float s = __shfl_sync(0xffffffffu, abs_step, k, RAY_LANES), e = __shfl_sync(0xffffffffu, pass, k, RAY_LANES);
      float ck[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) ck[c] = __shfl_sync(0xffffffffu, cc[c], k, RAY_LANES);
      if (((in >> k) & 1u) && trans > 0.01f) {
#pragma unroll
        for (int c = 0; c < 3; ++c) col[c] = add(col[c], mul(mul(mul(trans, ck[c]), s), R.exposure));
        trans = mul(trans, e);
      }
      t = add(t, dt);
    }
  }
  if (pixel && l == 0)
    out[(size_t)py * R.width + px] = hit ? make_float4(col[0], col[1], col[2], sub(1.0f, trans))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Two lanes a ray for the samples of long rays, and for images of fewer pixels than
// the chip's resident threads.  B200, 1 / 2 lanes in us: 1920 x 1080 over 256 x 128 x
// 128, absorption 5: 1 step 25 / 50, 8 steps 30 / 50, 24 48 / 54, 32 59 / 58, 128 179 /
// 128; 320 x 200 over 128^3: 1 step 8.2 / 7.9, 4 8.8 / 9.2, 8 13 / 11, 32 35 / 21.
inline bool two_lanes(int steps, int width, int height) {
  return steps >= 24 || (steps >= 4 && (int64_t)width * height < 148 * 1024);
}

}  // namespace
}  // namespace lbm

extern "C" {

int lbm_velmag_params_default(lbm_velmag_params* p) {
  if (!p) return LBM_ERR_INVALID_ARG;
  *p = lbm_velmag_params{};
  p->struct_size = sizeof(lbm_velmag_params);
  for (int i = 0; i < 16; ++i) p->inv_view_proj[i] = (i % 5 == 0) ? 1.0f : 0.0f;
  p->steps = 128;
  p->absorption = 4.0f;
  p->velmag_min = 0.0f;
  p->velmag_max = 0.1f;
  p->exposure = 1.5f;
  p->round_f16 = 1;
  p->volume_max[0] = p->volume_max[1] = p->volume_max[2] = -1.0f;  // = (Nx, Ny, Nz)
  return LBM_OK;
}

int lbm_render_velmag(const float* d_u, int32_t nx, int32_t ny, int32_t nz, const lbm_velmag_params* p,
                      int32_t width, int32_t height, float* d_rgba, void* stream) {
  if (!d_u || !p || !d_rgba || nx < 1 || ny < 1 || nz < 1 || width < 1 || height < 1) {
    lbm::set_thread_error("render velmag: bad argument");
    return LBM_ERR_INVALID_ARG;
  }
  if (p->struct_size != sizeof(lbm_velmag_params) || p->steps < 1 || p->steps > 4096) {
    lbm::set_thread_error("render velmag: bad parameters (struct_size, steps in [1, 4096])");
    return LBM_ERR_INVALID_ARG;
  }
  if ((reinterpret_cast<uintptr_t>(d_rgba) & 15u) != 0) {
    lbm::set_thread_error("render velmag: output must be 16-byte aligned (float4)");
    return LBM_ERR_INVALID_ARG;
  }
  lbm::RenderArgs R{};
  for (int i = 0; i < 16; ++i) R.m[i] = p->inv_view_proj[i];
  const float dims[3] = {(float)nx, (float)ny, (float)nz};
  for (int c = 0; c < 3; ++c) {
    R.cam[c] = p->camera_pos[c];
    R.vmin[c] = p->volume_min[c];
    R.vmax[c] = p->volume_max[c] < 0.0f ? dims[c] : p->volume_max[c];
  }
  R.steps = p->steps;
  R.absorption = p->absorption;
  R.mag_min = p->velmag_min;
  R.mag_max = p->velmag_max;
  R.exposure = p->exposure;
  R.width = width;
  R.height = height;
  for (int c = 0; c < 3; ++c) {
    int ex = 0;
    const float ext = R.vmax[c] - R.vmin[c];
    R.inv_ext[c] = std::frexp(ext, &ex) == 0.5f && ex > -100 && ex < 100 ? 1.0f / ext : 0.0f;
  }
  const size_t n = (size_t)nx * ny * nz;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float4* out = reinterpret_cast<float4*>(d_rgba);
  auto lanes = [&](auto index, auto f16, auto ray) {
    using I = decltype(index);
    constexpr bool F16 = decltype(f16)::value;
    constexpr int L = decltype(ray)::value, TY = lbm::tile_y<L>();
    const unsigned grd =
        (unsigned)((width + lbm::TILE_X - 1) / lbm::TILE_X) * (unsigned)((height + TY - 1) / TY);
    lbm::k_velmag<I, F16, L><<<grd, 256, 0, s>>>(lbm::Vol<I, F16>{d_u, nx, ny, nz, n}, R, out);
  };
  auto launch = [&](auto index, auto f16) {
    if (lbm::two_lanes(p->steps, width, height)) lanes(index, f16, std::integral_constant<int, 2>{});
    else lanes(index, f16, std::integral_constant<int, 1>{});
  };
  if (n < (1u << 31)) {
    if (p->round_f16) launch(uint32_t{}, std::true_type{});
    else launch(uint32_t{}, std::false_type{});
  } else {
    if (p->round_f16) launch(size_t{}, std::true_type{});
    else launch(size_t{}, std::false_type{});
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    lbm::set_thread_error((std::string("render velmag: ") + cudaGetErrorString(e)).c_str());
    return LBM_ERR_CUDA;
  }
  return LBM_OK;
}

}  // extern "C"
