// rast_internal.cuh -- pieces shared by the plain and tiled forms: the
// primitive-setup record, the per-pixel resolve (chooser fallback,
// barycentrics, fragment, mixer) and buffer merge.
#pragma once

#include <nvtx3/nvToolsExt.h>

#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "rast_shaders.cuh"

namespace rast {

constexpr int kTile = 16;         // plain form: 16x16 pixels per CTA
constexpr int kScanThreads = kTile * kTile;
constexpr int kScanChunk = 512;   // primitive setups staged per shared-memory chunk

// Setup record flags (float bits of record[3].y).
constexpr int kKeep = 1;          // |det| > 1e-6 (pipeline.py:98-100)
constexpr int kFront = 2;         // det >= 0 (pipeline.py:232)
constexpr int kCandidate = kKeep | kFront;

inline size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// PerPrimitive.create (pipeline.py:80-113) from the three clip positions.
// Record: [inv0..3] [inv4..7] [inv8 z0 z1 z2] [det flags 0 0]; the tiled
// form keeps the face's pixel rectangle in [3].x and [3].z and writes records
// of binned faces and face 0 only.
__device__ __forceinline__ void setup_from_clip(const float4* c, float* inv, float* det_out,
                                                int* flags_out) {
  const float m[9] = {c[0].x, c[0].y, c[0].w, c[1].x, c[1].y, c[1].w, c[2].x, c[2].y, c[2].w};
  const float det = det3(m);
  inv3(m, inv);
  int flags = 0;
  if (fabsf(det) > 1e-6f) flags |= kKeep;
  if (det >= 0.0f) flags |= kFront;
  *det_out = det;
  *flags_out = flags;
}

__device__ __forceinline__ void write_setup(const float4* c, float4* out) {
  float inv[9], det;
  int flags;
  setup_from_clip(c, inv, &det, &flags);
  out[0] = make_float4(inv[0], inv[1], inv[2], inv[3]);
  out[1] = make_float4(inv[4], inv[5], inv[6], inv[7]);
  out[2] = make_float4(inv[8], c[0].z, c[1].z, c[2].z);
  out[3] = make_float4(det, __int_as_float(flags), 0.0f, 0.0f);
}

__device__ __forceinline__ bool is_near_tie(unsigned long long best, uint32_t second) {
  const uint32_t o1 = static_cast<uint32_t>(best >> 32);
  return best != kEmptyKey && o1 != kInfOrder && second != 0xffffffffu && second - o1 <= 1u;
}

// Warp-aggregated count of near ties; every lane of the warp must call it.
__device__ __forceinline__ void count_near_tie(unsigned long long* counter, bool tie) {
  const unsigned m = __ballot_sync(0xffffffffu, tie);
  if ((threadIdx.x + threadIdx.y * blockDim.x) % 32 == 0 && m)
    atomicAdd(counter, static_cast<unsigned long long>(__popc(m)));
}

__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// ---- block maps: grids over the faces (or vertices) of every job with no
// more than one empty block per job.  Job j's blocks of `per_block` items
// start at entry begin_j / per_block + j, begin_j its first row (setup_begin
// or vout_begin, the running sum of n_faces / n_verts): the entries up to the
// next job's first one hold every block of the job, since floor((a + n) / p) -
// floor(a / p) + 1 >= ceil(n / p), and no prefix sum over the jobs is needed.
// Entry b is (job, first item of the block), or (-1, 0) for an empty block.
// A batch needs floor(total / per_block) + n_jobs entries.
constexpr int kMapFaces = 0, kMapVertices = 1;

__host__ __device__ inline unsigned block_map_capacity(int64_t total, int n_jobs, int per_block) {
  return static_cast<unsigned>(total / per_block + n_jobs);
}

template <int kField>
__device__ __forceinline__ unsigned map_entry_of_job(const RastJob* jobs, int n_jobs, int j, int per_block,
                                                     unsigned capacity) {
  if (j >= n_jobs) return capacity;
  const int64_t begin = kField == kMapFaces ? __ldg(&jobs[j].setup_begin) : __ldg(&jobs[j].vout_begin);
  return min(static_cast<unsigned>(begin / per_block) + static_cast<unsigned>(j), capacity);
}

// Fills the map; every block of the grid calls it.  Few jobs take a block
// each (one job of 389,120 faces has 3,040 entries, 9.7 us when one thread
// wrote them), many jobs a warp each.
constexpr int kMapBlockJobs = 2048;  // up to this many jobs: a block per job
template <int kField>
__device__ __forceinline__ void fill_block_map(const RastJob* __restrict__ jobs, int n_jobs, int per_block,
                                               int2* __restrict__ map, unsigned capacity) {
  const bool wide = n_jobs <= kMapBlockJobs;
  const unsigned team = wide ? blockDim.x : 32u;
  const unsigned t = threadIdx.x % team, teams = blockDim.x / team;
  for (int j = static_cast<int>(blockIdx.x * teams + threadIdx.x / team); j < n_jobs;
       j += static_cast<int>(gridDim.x * teams)) {
    const int n = kField == kMapFaces ? __ldg(&jobs[j].n_faces) : __ldg(&jobs[j].n_verts);
    const unsigned a = map_entry_of_job<kField>(jobs, n_jobs, j, per_block, capacity);
    const unsigned b = map_entry_of_job<kField>(jobs, n_jobs, j + 1, per_block, capacity);
    for (unsigned e = a + t; e < b; e += team) {
      const int64_t first = static_cast<int64_t>(e - a) * per_block;
      map[e] = first < n ? make_int2(j, static_cast<int>(first)) : make_int2(-1, 0);
    }
  }
}

// The marked ones among the n (at most kRows) rows from row0 on, one mark bit
// per row in `marks`: their offsets from row0 go to the warp's `list` in
// order (eight bits per lane, one prefix sum), and every lane gets their
// number.  All 32 lanes must call.
template <int kRows>
__device__ __forceinline__ int list_marked(const uint32_t* __restrict__ marks, int64_t row0, int n, unsigned char* list) {
  static_assert(kRows <= 256 && kRows % 32 == 0, "eight rows per lane, list entries of one byte");
  const int lane = threadIdx.x & 31;
  const int left = min(kRows, n) - 8 * lane;
  unsigned bits = 0;
  if (left > 0) {
    const int64_t at = row0 + 8 * lane;
    const unsigned shift = static_cast<unsigned>(at & 31);
    bits = marks[at >> 5] >> shift;
    if (shift > 24 && left > 32 - static_cast<int>(shift)) bits |= marks[(at >> 5) + 1] << (32 - shift);
    bits &= left >= 8 ? 0xffu : (1u << left) - 1u;
  }
  int incl = __popc(bits);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  int slot = incl - __popc(bits);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if ((bits >> k) & 1u) list[slot++] = static_cast<unsigned char>(8 * lane + k);
  __syncwarp();
  return __shfl_sync(0xffffffffu, incl, 31);
}

// Warps per map entry of the kernels that work through list_marked: up to
// four while there are fewer than `per_sm` of them per SM, so that a warp's
// rounds, 2-3 us of latency each, do not follow one another while SMs idle.
inline unsigned warps_per_entry(unsigned entries, int sms, unsigned per_sm) {
  const unsigned k = static_cast<unsigned>(sms) * per_sm / (entries > 0 ? entries : 1u);
  return k < 1u ? 1u : k > 4u ? 4u : k;
}

// Sets `bytes` bytes at p (16-byte aligned; the last 16-byte word may run
// past `bytes`, inside the workspace's 256-byte granules), the whole grid
// striding over them.
__device__ __forceinline__ void fill_words(void* p, size_t bytes, unsigned value) {
  uint4* w = static_cast<uint4*>(p);
  const size_t n = (bytes + 15) / 16;
  const size_t blocks = static_cast<size_t>(gridDim.x) * gridDim.y;
  for (size_t k = (static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; k < n;
       k += blocks * blockDim.x)
    w[k] = make_uint4(value, value, value, value);
}

// Blocks of 256 threads for a launch that fills `bytes` bytes and block maps
// of n_jobs jobs: at most eight per SM.
inline unsigned begin_blocks(size_t bytes, int n_jobs, int sms) {
  const size_t maps = n_jobs <= kMapBlockJobs ? n_jobs : (n_jobs + 7) / 8;
  const size_t fill = bytes / (256 * 16 * 2) + 1;
  const size_t most = static_cast<size_t>(sms > 0 ? sms : 1) * 8;
  const size_t want = maps > fill ? maps : fill;
  return static_cast<unsigned>(want < most ? want : most);
}

template <class T>
struct Same {
  using type = T;
};

// Launch of a kernel that starts with after_previous(): it may be set up while
// the previous kernel of its stream finishes (programmatic dependent launch),
// and waits there until that one's writes are visible (and, since that one
// waited too, every earlier kernel's of its chain).  It takes 0.5 us a launch
// off a small batch (16 scenes: 67 -> 64 us a replay) and nothing from large
// ones.  Not for the first kernel after a stream waits for an event.
template <class... Args>
inline void launch_after(void (*kernel)(Args...), dim3 grid, dim3 block, cudaStream_t s,
                         typename Same<Args>::type... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

inline int sm_count() {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

// Pixel (i, j) of a job from its x-major local index i * H + j.  Up to 2^20
// pixels the quotient comes from the approximate division (2 ulp, and l and H
// are exact), at most one off before the remainder corrects it: half the
// instructions of the integer one (-10 us of the 4096-scene shade's 737).
__device__ __forceinline__ void pixel_of(int64_t local, int64_t npx, int H, int* i, int* j) {
  if (npx <= (1 << 20)) {
    const int l = static_cast<int>(local);
    int q = static_cast<int>(__fdividef(static_cast<float>(l), static_cast<float>(H)));
    int r = l - q * H;
    if (r < 0) --q, r += H;
    if (r >= H) ++q, r -= H;
    *i = q;
    *j = r;
  } else if (npx <= 0x7fffffff) {
    const int l = static_cast<int>(local);
    *i = l / H;
    *j = l - *i * H;
  } else {
    *i = static_cast<int>(local / H);
    *j = static_cast<int>(local - static_cast<int64_t>(*i) * H);
  }
}

__device__ __forceinline__ void load_job_to_shared(const RastJob* job, RastJob* dst) {
  const int nthreads = blockDim.x * blockDim.y;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int* src = reinterpret_cast<const int*>(job);
  int* d = reinterpret_cast<int*>(dst);
  for (int k = tid; k < static_cast<int>(sizeof(RastJob) / 4); k += nthreads) d[k] = __ldg(src + k);
}

// Where a shade thread reads the three corners' varyings of a face.

// Plain form: the vertex kernel's rows, one per vertex.
struct VertexRows {
  const float* var;
  int vstride;
  int64_t vout_begin;
  template <int SH>
  __device__ __forceinline__ void load(const RastJob& J, const RastPools& P, int p, float* v0, float* v1,
                                       float* v2) const {
    const int nv = varying_count(SH >= 0 ? SH : J.shader);
    const int32_t* face = P.faces + (J.face_begin + p) * 3;
    const float* r0 = var + (vout_begin + gather_clamp(face[0], J.n_verts)) * vstride;
    const float* r1 = var + (vout_begin + gather_clamp(face[1], J.n_verts)) * vstride;
    const float* r2 = var + (vout_begin + gather_clamp(face[2], J.n_verts)) * vstride;
    // constant indices keep the three rows in registers
#pragma unroll
    for (int k = 0; k < kMaxVarying; ++k) {
      if (k < nv) {
        v0[k] = __ldg(r0 + k);
        v1[k] = __ldg(r1 + k);
        v2[k] = __ldg(r2 + k);
      }
    }
  }
};

// Tiled form: one row of `floats` floats per face (face_floats of the batch's
// largest shader) for the faces some pixel needs.  The whole float4s of the
// rows come first, then every row's remaining floats % 4, so that rows of any
// length read as float4 without padding.
struct FaceRows {
  const float4* vec;
  const float* rest;  // vec + faces * (floats / 4)
  int floats;
  int64_t setup_begin;
  template <int SH>
  __device__ __forceinline__ void load(const RastJob& J, const RastPools&, int p, float* v0, float* v1,
                                       float* v2) const {
    const int n = SH >= 0 ? face_floats(SH) : floats, own = face_floats(SH >= 0 ? SH : J.shader);
    const float4* a = vec + (setup_begin + p) * (n / 4);
    const float* t = rest + (setup_begin + p) * (n % 4);
    float row[kMaxFaceFloats];
#pragma unroll
    for (int q = 0; q < kMaxFaceFloats / 4; ++q) {
      if (4 * q >= own) continue;
      if (q < n / 4) {
        const float4 x = __ldg(a + q);
        row[4 * q] = x.x;
        row[4 * q + 1] = x.y;
        row[4 * q + 2] = x.z;
        row[4 * q + 3] = x.w;
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (c < n % 4) row[4 * q + c] = __ldg(t + c);
      }
    }
    get_corners<SH>(J.shader, row, v0, v1, v2);
  }
};

struct PixelResult {
  bool keep;
  float z;
  float colour[3];
  int prim;
};

// Interpolation and fragment shader of primitive p at the pixel whose NDC
// coordinates are (x, y) (pipeline.py:283-326): clip coefficients, chooser keep (keep & inside),
// depth, perspective-correct barycentrics, the corner varyings from `src`,
// then the job's fragment shader.
struct Fragment {
  bool chooser_keep;  // keep & inside (the chooser's keeps slice)
  bool keep;          // the fragment shader's keep
  float z;
  float colour[3];
};

// SH >= 0: the job's shader, known at compile time.  light: its normalised
// light direction, or nullptr (computed here).
// Without xy_given, (x, y) is computed here from the pixel (i, j).  Chosen
// primitives are candidates (kept and front-facing) except the default
// chooser's fallback to primitive 0, whose flags come from its record.
template <int SH, class Source>
__device__ __forceinline__ void shade_primitive(const RastJob& J, const RastPools& P, const float4* rec_base,
                                                int i, int j, float x, float y, int p, const Source& src,
                                                Fragment* f, bool xy_given, bool fallback = false,
                                                const float* light = nullptr) {
  const float4* rec = rec_base + static_cast<int64_t>(p) * 4;
  const float4 a = rec[0], b = rec[1], cz = rec[2];
  const int flags = fallback ? __float_as_int(rec[3].y) : kCandidate;
  if (!xy_given) {
    x = (static_cast<float>(i) - J.viewport[3]) / J.viewport[0];
    y = (static_cast<float>(j) - J.viewport[7]) / J.viewport[5];
  }
  const float c[3] = {(x * a.x + y * a.w) + b.z, (x * a.y + y * b.x) + b.w,
                      (x * a.z + y * b.y) + cz.x};
  const bool in_tri = c[0] >= 0.0f && c[1] >= 0.0f && c[2] >= 0.0f;
  f->chooser_keep = (flags & kKeep) && in_tri;
  f->keep = false;
  f->z = 0.0f;
  f->colour[0] = f->colour[1] = f->colour[2] = 0.0f;
  if (!f->chooser_keep) return;  // nothing of a discarded fragment is read
  const bool front = (flags & kFront) != 0;
  const float w_rcp = (c[0] + c[1]) + c[2];
  f->z = ((c[0] * cz.y + c[1] * cz.z) + c[2] * cz.w) * J.viewport[10] + J.viewport[11];
  const float bary[3] = {c[0] / w_rcp, c[1] / w_rcp, c[2] / w_rcp};
  float v0[kMaxVarying], v1[kMaxVarying], v2[kMaxVarying];
  if ((SH >= 0 ? SH : J.shader) != RAST_SHADER_DEPTH) src.template load<SH>(J, P, p, v0, v1, v2);
  f->keep = fragment_shader<SH>(J, P, v0, v1, v2, bary, front, f->colour, light);
}

// One pixel after the scan: `w` is the winning candidate (-1: none, or its
// depth was +inf).  Reproduces the default chooser's fallback to primitive 0
// (shader.py:215-217), then Shader.interpolate / fragment / mix
// (pipeline.py:283-359) for the chosen primitive.
template <int SH, class Source>
__device__ __forceinline__ void resolve_pixel(const RastJob& J, const RastPools& P,
                                              const float4* rec_base, int i, int j, int w,
                                              const Source& src, PixelResult* r, const float* light = nullptr) {
  r->keep = false;
  r->prim = -1;
  r->z = 0.0f;
  r->colour[0] = r->colour[1] = r->colour[2] = 0.0f;
  if (J.n_faces <= 0) return;
  const int p = w < 0 ? 0 : w;
  Fragment f;
  shade_primitive<SH>(J, P, rec_base, i, j, 0.0f, 0.0f, p, src, &f, false, w < 0, light);
  r->keep = f.chooser_keep && f.keep;
  r->z = f.z;
  r->prim = r->keep ? p : -1;
#pragma unroll
  for (int k = 0; k < 3; ++k) r->colour[k] = f.colour[k];
}

// Chooser slots of job J: 0 = the default chooser, else the layered
// chooser's slot count (clamped to the batch's max_layers).
__device__ __forceinline__ int job_layers(const RastJob& J, int max_layers) {
  return J.layers <= 0 ? 0 : min(J.layers, max_layers);
}

// One pixel of a layered job (RastJob.layers = L >= 1): slots
// w[0 .. L-1] (stride `wstride`) hold the nearest candidates in ascending
// (depth, id) order, -1 past the last.  Every slot from `first` on runs
// interpolation + fragment; the job's mixer combines the kept ones
// (RastMixer).  first > 0 continues a nearest-mixer pixel whose earlier
// slots were all discarded.
template <int SH, class Source>
__device__ __forceinline__ void resolve_layers(const RastJob& J, const RastPools& P, const float4* rec_base,
                                               int i, int j, const int32_t* w, int64_t wstride, int L,
                                               const Source& src, PixelResult* r, int first = 0, const float* light = nullptr) {
  r->keep = false;
  r->prim = -1;
  r->z = 0.0f;
  r->colour[0] = r->colour[1] = r->colour[2] = 0.0f;
  const bool over = J.mixer == RAST_MIX_OVER;
  const bool per_face = (J.flags & RAST_JOB_FACE_ALPHA) && P.face_alpha;
  const float x = (static_cast<float>(i) - J.viewport[3]) / J.viewport[0];
  const float y = (static_cast<float>(j) - J.viewport[7]) / J.viewport[5];
  // the slots, loaded up front and shifted down one per step (no indexed
  // register array)
  int w0 = first < 1 ? w[0] : -1, w1 = L > 1 && first < 2 ? w[wstride] : -1;
  int w2 = L > 2 && first < 3 ? w[2 * wstride] : -1, w3 = L > 3 && first < 4 ? w[3 * wstride] : -1;
  static_assert(RAST_MAX_LAYERS == 4, "slot registers w0..w3");
  for (int s = 0; s < first; ++s) w0 = w1, w1 = w2, w2 = w3, w3 = -1;
  float T = 1.0f, C[3] = {0.0f, 0.0f, 0.0f};
  for (int s = first; s < L; ++s) {
    const int p = w0;
    w0 = w1, w1 = w2, w2 = w3, w3 = -1;
    if (p < 0) break;
    Fragment f;
    shade_primitive<SH>(J, P, rec_base, i, j, x, y, p, src, &f, true, false, light);
    if (!(f.chooser_keep && f.keep)) continue;
    if (!r->keep) {
      r->keep = true;
      r->z = f.z;
      r->prim = p;
      if (!over) {
#pragma unroll
        for (int k = 0; k < 3; ++k) r->colour[k] = f.colour[k];
        return;
      }
    }
    const float alpha = per_face ? __ldg(P.face_alpha + J.face_begin + p) : J.opacity;
    const float wgt = T * alpha;
#pragma unroll
    for (int k = 0; k < 3; ++k) C[k] = C[k] + wgt * f.colour[k];
    T = T * (1.0f - alpha);
  }
  if (r->keep && over) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r->colour[k] = C[k] + T * J.background[k];
  }
}

// Fragments of one warp's pixels under the layered chooser: at most
// RAST_MAX_LAYERS per pixel.
constexpr int kWarpFrags = 32 * RAST_MAX_LAYERS;

// Shared-memory staging of one warp's fragments for resolve_over_warp.
struct WarpFrags {
  float colour[3][kWarpFrags];
  float z[kWarpFrags];
  unsigned char keep[kWarpFrags];
};

// RAST_MIX_OVER pixels of one warp, all 32 lanes calling (inactive lanes
// own no pixel): the warp's (pixel, slot) fragments are numbered in lane
// order, 32 of them shaded per round with one fragment per lane (so pixels
// with fewer layers leave no lane idle while others shade), staged in `wf`,
// then every lane mixes its own pixel's fragments in slot order.  Same
// operations and order as resolve_layers.
template <int SH, class Source>
__device__ __forceinline__ void resolve_over_warp(const RastJob& J, const RastPools& P, const float4* rec_base,
                                                  bool active, int i, int j, const int32_t* w, int64_t wstride,
                                                  int L, const Source& src, WarpFrags& wf,
                                                  PixelResult* r, const float* light = nullptr) {
  const int lane = threadIdx.x & 31;
  r->keep = false;
  r->prim = -1;
  r->z = 0.0f;
  r->colour[0] = r->colour[1] = r->colour[2] = 0.0f;
  static_assert(RAST_MAX_LAYERS == 4, "slot registers w0..w3");
  int w0 = -1, w1 = -1, w2 = -1, w3 = -1, n = 0;
  float x = 0.0f, y = 0.0f;
  if (active) {
    x = (static_cast<float>(i) - J.viewport[3]) / J.viewport[0];
    y = (static_cast<float>(j) - J.viewport[7]) / J.viewport[5];
    w0 = w[0];
    if (L > 1) w1 = w[wstride];
    if (L > 2) w2 = w[2 * wstride];
    if (L > 3) w3 = w[3 * wstride];
    n = w0 < 0 ? 0 : w1 < 0 ? 1 : w2 < 0 ? 2 : w3 < 0 ? 3 : 4;  // leading filled slots
  }
  int incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  const int excl = incl - n;
  const int total = __shfl_sync(0xffffffffu, incl, 31);  // <= kWarpFrags
  for (int base = 0; base < total; base += 32) {
    const int k = base + lane;
    int owner = 0;  // the lane whose fragments [excl, incl) hold k
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int v = __shfl_sync(0xffffffffu, incl, owner + step - 1);
      if (v <= k) owner += step;
    }
    const int slot = k - __shfl_sync(0xffffffffu, excl, owner);
    const int a0 = __shfl_sync(0xffffffffu, w0, owner), a1 = __shfl_sync(0xffffffffu, w1, owner);
    const int a2 = __shfl_sync(0xffffffffu, w2, owner), a3 = __shfl_sync(0xffffffffu, w3, owner);
    const float ox = __shfl_sync(0xffffffffu, x, owner), oy = __shfl_sync(0xffffffffu, y, owner);
    if (k < total) {
      const int p = slot == 0 ? a0 : slot == 1 ? a1 : slot == 2 ? a2 : a3;
      Fragment f;
      shade_primitive<SH>(J, P, rec_base, 0, 0, ox, oy, p, src, &f, true, false, light);
#pragma unroll
      for (int c = 0; c < 3; ++c) wf.colour[c][k] = f.colour[c];
      wf.z[k] = f.z;
      wf.keep[k] = f.chooser_keep && f.keep;
    }
  }
  __syncwarp();
  const bool per_face = (J.flags & RAST_JOB_FACE_ALPHA) && P.face_alpha;
  float T = 1.0f, C[3] = {0.0f, 0.0f, 0.0f};
  for (int s = 0; s < n; ++s) {
    const int k = excl + s;
    const int p = w0;
    w0 = w1, w1 = w2, w2 = w3, w3 = -1;
    if (!wf.keep[k]) continue;
    if (!r->keep) {
      r->keep = true;
      r->z = wf.z[k];
      r->prim = p;
    }
    const float alpha = per_face ? __ldg(P.face_alpha + J.face_begin + p) : J.opacity;
    const float wgt = T * alpha;
#pragma unroll
    for (int c = 0; c < 3; ++c) C[c] = C[c] + wgt * wf.colour[c][k];
    T = T * (1.0f - alpha);
  }
  if (r->keep) {
#pragma unroll
    for (int c = 0; c < 3; ++c) r->colour[c] = C[c] + T * J.background[c];
  }
}

// The forward's record of a layered pixel's slots for the backward
// (RastPools.layer_prim, slot-major): slots 0 .. L-1 from the winner planes,
// -1 past them.
__device__ __forceinline__ void save_layers(const RastPools& P, const int32_t* w, int64_t wstride, int64_t pix,
                                            int L) {
  if (!P.layer_prim) return;
#pragma unroll
  for (int s = 0; s < RAST_MAX_LAYERS; ++s) P.layer_prim[s * wstride + pix] = s < L ? w[s * wstride] : -1;
}

// Keeps best[0 .. L-1] the L smallest keys seen, ascending: `key` goes in
// at its rank and the larger ones move down one slot.
template <int L>
__device__ __forceinline__ void insert_key(unsigned long long (&best)[L], unsigned long long key) {
#pragma unroll
  for (int s = L - 1; s > 0; --s)
    if (key < best[s]) best[s] = key < best[s - 1] ? best[s - 1] : key;
  if (key < best[0]) best[0] = key;
}

// Defaults of a pass into cleared buffers (rast_render_tiled_clear), or off.
struct Clear {
  const float* colour = nullptr;
  float depth = 0.0f;
  bool on = false;
};

// merge_buffers (pipeline.py:401-440): overwrite where kept, no depth test
// (with `clear`, the default where not kept, as if the buffer had held it);
// then the shadow pass's offset (shadow.py:116) when the job asks for it.
__device__ __forceinline__ void store_pixel(const RastJob& J, const RastPools& P, int64_t pix,
                                            const PixelResult& r, const Clear& clear = Clear()) {
  const bool offset = (J.flags & RAST_JOB_APPLY_DEPTH_OFFSET) != 0;
  if (r.keep || offset || clear.on) {
    float zb = r.keep ? r.z : clear.on ? clear.depth : P.zbuffer[pix];
    if (offset) zb = zb + J.depth_offset;
    P.zbuffer[pix] = zb;
  }
  const bool coloured = r.keep && J.shader != RAST_SHADER_DEPTH;
  if ((coloured || clear.on) && P.canvas) {
#pragma unroll
    for (int k = 0; k < 3; ++k) P.canvas[pix * 3 + k] = coloured ? r.colour[k] : __ldg(clear.colour + k);
  }
  if (P.prim_id) P.prim_id[pix] = r.prim;
}

// Optional per-kernel event timing of an entry point (RastProfile).
// NVTX range over one entry point's host-side launch sequence (header-only
// NVTX3: without a profiler attached a push / pop is a check of a null hook).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// Per-kernel CUDA-event timing of an entry point (the *_profiled entry
// points) and its NVTX annotation: a range named after the entry point and
// one NVTX mark per kernel launched, named after the kernel.
struct Profiler {
  RastProfile* prof;
  cudaStream_t stream;
  cudaEvent_t ev[17];
  int n = 0;
  NvtxRange range;
  Profiler(RastProfile* p, cudaStream_t s, const char* entry) : prof(p), stream(s), range(entry) {
    if (prof) {
      prof->n = 0;
      cudaEventCreate(&ev[0]);
      cudaEventRecord(ev[0], stream);
    }
  }
  void mark(const char* name) {
    nvtxMarkA(name);
    if (!prof || n >= 16) return;
    cudaEventCreate(&ev[n + 1]);
    cudaEventRecord(ev[n + 1], stream);
    prof->names[n] = name;
    ++n;
  }
  int finish() {
    if (!prof) return RAST_OK;
    if (cudaStreamSynchronize(stream) != cudaSuccess) return RAST_ERR_CUDA;
    for (int k = 0; k < n; ++k) cudaEventElapsedTime(&prof->ms[k], ev[k], ev[k + 1]);
    for (int k = 0; k <= n; ++k) cudaEventDestroy(ev[k]);
    prof->n = n;
    return RAST_OK;
  }
};

// Host-side argument checks shared by the entry points.
inline int check_batch(const RastBatch* b) {
  if (!b || !b->jobs) return RAST_ERR_INVALID_ARGUMENT;
  if (b->n_jobs < 1 || b->n_jobs > 65535) return RAST_ERR_INVALID_ARGUMENT;
  if (b->total_vout < 0 || b->total_setup < 0 || b->total_pixels < 0) return RAST_ERR_INVALID_ARGUMENT;
  if (b->max_width < 0 || b->max_height < 0 || b->max_faces < 0 || b->max_verts < 0)
    return RAST_ERR_INVALID_ARGUMENT;
  if ((b->shader_mask & ~0x7f) != 0) return RAST_ERR_INVALID_ARGUMENT;
  if (b->max_layers < 0 || b->max_layers > RAST_MAX_LAYERS) return RAST_ERR_INVALID_ARGUMENT;
  if (b->total_pixels > 0 && !b->pools.zbuffer) return RAST_ERR_INVALID_ARGUMENT;
  if (b->total_setup > 0 && (!b->pools.faces || !b->pools.position)) return RAST_ERR_INVALID_ARGUMENT;
  if (b->total_vout > 0 && !b->pools.position) return RAST_ERR_INVALID_ARGUMENT;
  return RAST_OK;
}

}  // namespace rast
