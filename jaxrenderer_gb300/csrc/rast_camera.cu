// rast_camera.cu -- camera matrices of a batch of eyes and their reverse mode
// (Camera.view_matrix / view_matrix_inv / perspective, geometry.py:536-684),
// one thread per camera and one launch per direction.  As tensor operations
// the same takes about 90 launches forward and 140 backward, each of a few
// microseconds: 3.3 ms of host time around a 0.5 ms render.  Operation order
// of the forward: that of the tensor operations (autograd.view_matrix) with
// the contraction of their kernels as they are today (cross products and the
// 4 x 4 product fuse one multiply into each addition); between the two routes
// the matrices may differ by rounding, within what test_gpu_camera.py allows.
#include <cuda_runtime.h>

#include "rast_internal.cuh"

namespace rast {
namespace camera {

constexpr int kThreads = 64;

struct Frame {
  float f[3], fn;    // forward = normalise(centre - eye), the length divided by
  float up[3], un;   // normalise(up)
  float s[3], sn;    // side = normalise(forward x up)
  float u[3];        // side x forward
};

__device__ __forceinline__ float unit(const float* v, float* out) {
  const float n = sqrtf((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k] = v[k] / n;
  return n;
}

__device__ __forceinline__ void cross(const float* a, const float* b, float* out) {
  out[0] = __fmaf_rn(a[1], b[2], -(a[2] * b[1]));
  out[1] = __fmaf_rn(a[2], b[0], -(a[0] * b[2]));
  out[2] = __fmaf_rn(a[0], b[1], -(a[1] * b[0]));
}

__device__ __forceinline__ void look_at(const float* e, const float* c, const float* up, Frame& r) {
  float d[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) d[k] = c[k] - e[k];
  r.fn = unit(d, r.f);
  r.un = unit(up, r.up);
  float x[3];
  cross(r.f, r.up, x);
  r.sn = unit(x, r.s);
  cross(r.s, r.f, r.u);
}

// (a * b) summed over three elements in the order of the tensor reduction.
__device__ __forceinline__ float sum3(const float* a, const float* b) {
  const float p = a[0] * b[0], q = a[1] * b[1], r = a[2] * b[2];
  return (p + r) + q;
}

struct Rows {  // (n, 3) rows; stride 0: one row for every camera
  const float* p;
  int64_t stride;
  __device__ __forceinline__ void load(int64_t i, float* out) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = __ldg(p + i * stride + k);
  }
};

__global__ void __launch_bounds__(kThreads)
forward_kernel(int n, Rows eye, Rows centre, Rows up, const float* __restrict__ projection, float* __restrict__ w2c,
               float* __restrict__ w2e, float* __restrict__ view) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;  // 16 i passes 2^31 at 2^27 cameras
  if (i >= n) return;
  float e[3], c[3], w[3];
  eye.load(i, e);
  centre.load(i, c);
  up.load(i, w);
  Frame r;
  look_at(e, c, w, r);
  float v[16] = {r.s[0], r.s[1], r.s[2], -sum3(r.s, e), r.u[0], r.u[1], r.u[2], -sum3(r.u, e),
                 -r.f[0], -r.f[1], -r.f[2], sum3(r.f, e), 0.0f, 0.0f, 0.0f, 1.0f};
#pragma unroll
  for (int k = 0; k < 16; ++k) view[i * 16 + k] = v[k];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float acc = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; ++k) acc = __fmaf_rn(__ldg(projection + 4 * a + k), v[4 * k + b], acc);
      w2c[i * 16 + 4 * a + b] = acc;
    }
  // the inverse's transpose: rows side, up, -forward, [eye, 1]
  const float t[16] = {r.s[0], r.s[1], r.s[2], 0.0f, r.u[0], r.u[1], r.u[2], 0.0f,
                       -r.f[0], -r.f[1], -r.f[2], 0.0f, e[0], e[1], e[2], 1.0f};
#pragma unroll
  for (int k = 0; k < 16; ++k) w2e[i * 16 + k] = t[k];
}

// y = v / |v|: dv = (dy - y (y . dy)) / |v|
__device__ __forceinline__ void unit_bwd(const float* y, float n, const float* dy, float* dv) {
  const float s = (y[0] * dy[0] + y[1] * dy[1]) + y[2] * dy[2];
#pragma unroll
  for (int k = 0; k < 3; ++k) dv[k] = (dy[k] - y[k] * s) / n;
}

// Gradient matrices (n, 4, 4), rows of 4 contiguous, `stride` floats apart per camera; NULL: zero.
struct Mats {
  const float* p;
  int64_t stride;
  __device__ __forceinline__ float at(int64_t i, int k) const { return p ? __ldg(p + i * stride + k) : 0.0f; }
};

__global__ void __launch_bounds__(kThreads)
backward_kernel(int n, Rows eye, Rows centre, Rows up, const float* __restrict__ projection, Mats gw2c, Mats gw2e, Mats gview,
                float* __restrict__ geye, float* __restrict__ gcentre, float* __restrict__ gup) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;  // 16 i passes 2^31 at 2^27 cameras
  if (i >= n) return;
  float e[3], c[3], w[3];
  eye.load(i, e);
  centre.load(i, c);
  up.load(i, w);
  Frame r;
  look_at(e, c, w, r);
  // dL/dview = dL/dview + projection^T dL/dworld_to_clip, rows 0..2
  float gv[12];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float acc = gview.at(i, 4 * a + b);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc += __ldg(projection + 4 * k + a) * gw2c.at(i, 4 * k + b);
      gv[4 * a + b] = acc;
    }
  float gs[3], gu[3], gf[3], ge[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    gs[k] = gv[k] - gv[3] * e[k] + gw2e.at(i, k);
    gu[k] = gv[4 + k] - gv[7] * e[k] + gw2e.at(i, 4 + k);
    gf[k] = gv[11] * e[k] - gv[8 + k] - gw2e.at(i, 8 + k);
    ge[k] = (gv[11] * r.f[k] - gv[3] * r.s[k]) - gv[7] * r.u[k] + gw2e.at(i, 12 + k);
  }
  // u = s x f;  s = normalise(f x up)
  float t[3], gx[3];
  cross(r.f, gu, t);
#pragma unroll
  for (int k = 0; k < 3; ++k) gs[k] += t[k];
  cross(gu, r.s, t);
#pragma unroll
  for (int k = 0; k < 3; ++k) gf[k] += t[k];
  unit_bwd(r.s, r.sn, gs, gx);
  cross(r.up, gx, t);
#pragma unroll
  for (int k = 0; k < 3; ++k) gf[k] += t[k];
  float gd[3];
  unit_bwd(r.f, r.fn, gf, gd);
  if (gup) {
    float gn[3], g[3];
    cross(gx, r.f, gn);
    unit_bwd(r.up, r.un, gn, g);
#pragma unroll
    for (int k = 0; k < 3; ++k) gup[i * 3 + k] = g[k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (geye) geye[i * 3 + k] = ge[k] - gd[k];
    if (gcentre) gcentre[i * 3 + k] = gd[k];
  }
}

}  // namespace camera
}  // namespace rast

using namespace rast;

extern "C" int rast_camera_matrices(int32_t n, const float* eye, int64_t eye_stride, const float* centre, int64_t centre_stride,
                                    const float* up, int64_t up_stride, const float* projection, float* world_to_clip,
                                    float* world_to_eye_norm, float* view, void* stream) {
  if (n < 0 || !eye || !centre || !up || !projection || !world_to_clip || !world_to_eye_norm || !view)
    return RAST_ERR_INVALID_ARGUMENT;
  if (n == 0) return RAST_OK;
  const unsigned grid = (static_cast<unsigned>(n) + camera::kThreads - 1) / camera::kThreads;
  camera::forward_kernel<<<grid, camera::kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      n, {eye, eye_stride}, {centre, centre_stride}, {up, up_stride}, projection, world_to_clip, world_to_eye_norm, view);
  return cudaGetLastError() == cudaSuccess ? RAST_OK : RAST_ERR_CUDA;
}

extern "C" int rast_camera_matrices_backward(int32_t n, const float* eye, int64_t eye_stride, const float* centre,
                                             int64_t centre_stride, const float* up, int64_t up_stride, const float* projection,
                                             const float* grad_world_to_clip, int64_t w2c_stride,
                                             const float* grad_world_to_eye_norm, int64_t w2e_stride, const float* grad_view,
                                             int64_t view_stride, float* grad_eye, float* grad_centre, float* grad_up,
                                             void* stream) {
  if (n < 0 || !eye || !centre || !up || !projection) return RAST_ERR_INVALID_ARGUMENT;
  if (n == 0) return RAST_OK;
  const unsigned grid = (static_cast<unsigned>(n) + camera::kThreads - 1) / camera::kThreads;
  camera::backward_kernel<<<grid, camera::kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      n, {eye, eye_stride}, {centre, centre_stride}, {up, up_stride}, projection, {grad_world_to_clip, w2c_stride},
      {grad_world_to_eye_norm, w2e_stride}, {grad_view, view_stride}, grad_eye, grad_centre, grad_up);
  return cudaGetLastError() == cudaSuccess ? RAST_OK : RAST_ERR_CUDA;
}
