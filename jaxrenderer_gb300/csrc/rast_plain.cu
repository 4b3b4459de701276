// rast_plain.cu -- plain form of the rasteriser: the reference's own method
// (pipeline.py:470-537) at GPU speed.
//
//   vertex_kernel  one thread per vertex: gl_Position + varyings
//                  (pipeline.py:497-518)
//   setup_kernel   one thread per face: gather by face index, det, keep,
//                  3x3 LU inverse (PerPrimitive.create, pipeline.py:80-113)
//   scan_kernel    every pixel against every primitive of the job, streamed
//                  through shared memory: clip_coef, inside test, depth,
//                  packed (ordered depth | id) minimum = the default
//                  primitive_chooser (shader.py:207-251); four pixels per
//                  thread, the primitives split over blocks when the pixels
//                  leave the chip idle.  slots_kernel is its form for passes
//                  that keep several candidates or count near ties
//   shade_kernel   one thread per pixel: chosen primitive -> barycentrics ->
//                  interpolate -> fragment -> mix -> merge
//                  (pipeline.py:283-359, 401-440)
#include <cuda_runtime.h>

#include <algorithm>

#include "rast_internal.cuh"

namespace rast {

// -------------------------------------------------------------- kernels

// Also sets `key_bytes` bytes of keys to the empty key: a launch of its own
// for that costs the host as much as this one.
// Grid: (at least ceil(max_verts / 256), n_jobs).
__global__ void __launch_bounds__(256)
vertex_kernel(RastBatch B, float4* __restrict__ clip_out, float* __restrict__ var_out, int vstride, void* keys,
              size_t key_bytes) {
  __shared__ RastJob sJ;
  fill_words(keys, key_bytes, 0xffffffffu);
  const int jid = blockIdx.y;
  const int nv = __ldg(&B.jobs[jid].n_verts);
  if (static_cast<int64_t>(blockIdx.x) * 256 >= nv) return;
  load_job_to_shared(B.jobs + jid, &sJ);
  __syncthreads();
  const RastJob& J = sJ;
  const int64_t v0 = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (v0 >= nv) return;
  const int64_t row = J.vout_begin + v0;
  const int v = static_cast<int>(row - J.vout_begin);
  float clip[4];
  float var[kMaxVarying];
  vertex_shader(J, B.pools, v, clip, var);
  clip_out[row] = make_float4(clip[0], clip[1], clip[2], clip[3]);
  const int nvar = varying_count(J.shader);
  for (int k = 0; k < nvar; ++k) var_out[row * vstride + k] = var[k];
}

// Grid: (ceil(max_faces / 256), n_jobs).
__global__ void __launch_bounds__(256)
setup_kernel(RastBatch B, const float4* __restrict__ clip, float4* __restrict__ setup) {
  after_previous();
  const int jid = blockIdx.y;
  const RastJob& J = B.jobs[jid];
  const int64_t f0 = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (f0 >= J.n_faces) return;
  const int64_t row = J.setup_begin + f0;
  const int64_t f = row - J.setup_begin;
  const int32_t* face = B.pools.faces + (J.face_begin + f) * 3;
  float4 c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = clip[J.vout_begin + gather_clamp(face[k], J.n_verts)];
  write_setup(c, setup + row * 4);
}

// The default chooser's scan.  Thread t of a job's ceil(W / 4) * H takes the
// four pixels (i0 + k ceil(W / 4), j): they share y, so a primitive's y
// products and its three shared-memory loads serve four tests, and no tile
// rounds the canvas up.  The block's share of the primitives (grid.z splits
// them) is staged 128 at a time, candidates only: closed meshes lose half.
// Splits fold their minima into the pixel's key with a 64-bit atomicMin
// (`keys` then starts as the empty key); a single split stores it.  Bound by
// FP32 issue once the chip is full: a 124x371 pass of 2,240 faces took 161 us
// as 192 blocks of one pixel per thread, half-empty SMs waiting on shared
// loads, and takes 24 us; 84x84 with 5,600 faces (36 such blocks) 289 -> 15.
// Grid: (ceil(ceil(max W / 4) max H / 128), n_jobs, splits).
constexpr int kScanPixels = 4;
constexpr int kScanBlock = 128;  // threads, and primitives staged at a time
__global__ void __launch_bounds__(kScanBlock)
scan_kernel(RastBatch B, const float4* __restrict__ setup, unsigned long long* __restrict__ keys) {
  __shared__ float4 s_rec[kScanBlock][3];
  __shared__ int s_id[kScanBlock];
  __shared__ int s_n;
  after_previous();
  const RastJob& J = B.jobs[blockIdx.y];
  const int W = J.width, H = J.height, F = J.n_faces;
  const int R = (W + kScanPixels - 1) / kScanPixels;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kScanBlock;
  if (first >= static_cast<int64_t>(R) * H) return;  // uniform over the block
  const int64_t t = first + threadIdx.x;
  int i0 = 0, j = 0;
  pixel_of(t, static_cast<int64_t>(R) * H, H, &i0, &j);
  const bool active = i0 < R;
  const float y = (static_cast<float>(j) - J.viewport[7]) / J.viewport[5];
  const float vp22 = J.viewport[10], vp23 = J.viewport[11];
  float x[kScanPixels];
  unsigned long long best[kScanPixels];
#pragma unroll
  for (int q = 0; q < kScanPixels; ++q) {
    x[q] = (static_cast<float>(i0 + q * R) - J.viewport[3]) / J.viewport[0];
    best[q] = kEmptyKey;
  }
  const float4* rec = setup + J.setup_begin * 4;
  const int f0 = static_cast<int>(static_cast<int64_t>(F) * blockIdx.z / gridDim.z);
  const int f1 = static_cast<int>(static_cast<int64_t>(F) * (blockIdx.z + 1) / gridDim.z);
  for (int base = f0; base < f1; base += kScanBlock) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const int f = base + static_cast<int>(threadIdx.x);
    const bool cand = f < f1 && (__float_as_int(__ldg(rec + static_cast<int64_t>(f) * 4 + 3).y) & kCandidate) == kCandidate;
    const unsigned m = __ballot_sync(0xffffffffu, cand);
    int at = 0;
    if ((threadIdx.x & 31) == 0 && m) at = atomicAdd(&s_n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & lanemask_lt());
    if (cand) {
#pragma unroll
      for (int k = 0; k < 3; ++k) s_rec[at][k] = __ldg(rec + static_cast<int64_t>(f) * 4 + k);
      s_id[at] = f;
    }
    __syncthreads();
    const int n = s_n;
    for (int p = 0; p < n; ++p) {
      const float4 a = s_rec[p][0], b = s_rec[p][1], cz = s_rec[p][2];
      // clip_coef = [x, y, 1] @ inv (pipeline.py:177-193)
      const float y0 = y * a.w, y1 = y * b.x, y2 = y * b.y;
#pragma unroll
      for (int q = 0; q < kScanPixels; ++q) {
        const float c0 = (x[q] * a.x + y0) + b.z;
        const float c1 = (x[q] * a.y + y1) + b.w;
        const float c2 = (x[q] * a.z + y2) + cz.x;
        if (all_nonneg(c0, c1, c2)) {
          const float z = ((c0 * cz.y + c1 * cz.z) + c2 * cz.w) * vp22 + vp23;
          const unsigned long long key = pack_key(z, s_id[p]);
          if (key < best[q]) best[q] = key;
        }
      }
    }
    __syncthreads();
  }
  if (!active) return;
#pragma unroll
  for (int q = 0; q < kScanPixels; ++q) {
    const int i = i0 + q * R;
    if (i >= W) break;
    unsigned long long* key = keys + J.pixel_begin + static_cast<int64_t>(i) * H + j;
    if (gridDim.z == 1)
      *key = best[q];
    else if (best[q] != kEmptyKey)
      atomicMin(key, best[q]);
  }
}

// One CTA = one 16x16 pixel tile of one job; every primitive of the job is
// staged through shared memory in chunks and tested by every pixel.  Each
// pixel keeps the kL smallest packed keys (kL = 1: the default chooser's
// argmin; kL = RAST_MAX_LAYERS when the batch has layered jobs, whose slots
// are the layered chooser's); slot s goes to winner[s * total_pixels + pix].
template <int kL>
__global__ void __launch_bounds__(kScanThreads)
slots_kernel(RastBatch B, const float4* __restrict__ setup, int32_t* __restrict__ winner) {
  __shared__ float4 s_rec[kScanChunk * 3];
  __shared__ int s_flag[kScanChunk];
  after_previous();
  const RastJob& J = B.jobs[blockIdx.y];
  const int W = J.width, H = J.height, F = J.n_faces;
  const int tiles_j = (H + kTile - 1) / kTile;
  const int tiles_i = (W + kTile - 1) / kTile;
  if (static_cast<int>(blockIdx.x) >= tiles_i * tiles_j) return;
  const int ti = blockIdx.x / tiles_j, tj = blockIdx.x % tiles_j;
  const int i = ti * kTile + threadIdx.y;
  const int j = tj * kTile + threadIdx.x;
  const int tid = threadIdx.y * kTile + threadIdx.x;
  const float x = (static_cast<float>(i) - J.viewport[3]) / J.viewport[0];
  const float y = (static_cast<float>(j) - J.viewport[7]) / J.viewport[5];
  const float vp22 = J.viewport[10], vp23 = J.viewport[11];
  unsigned long long best[kL];
#pragma unroll
  for (int l = 0; l < kL; ++l) best[l] = kEmptyKey;
  uint32_t second = 0xffffffffu;
  const float4* rec = setup + J.setup_begin * 4;
  for (int base = 0; base < F; base += kScanChunk) {
    const int n = min(kScanChunk, F - base);
    for (int q = tid; q < n * 3; q += kScanThreads)
      s_rec[q] = __ldg(rec + (static_cast<int64_t>(base) + q / 3) * 4 + q % 3);
    for (int q = tid; q < n; q += kScanThreads)
      s_flag[q] = __float_as_int(__ldg(rec + (static_cast<int64_t>(base) + q) * 4 + 3).y);
    __syncthreads();
    for (int p = 0; p < n; ++p) {
      const float4 a = s_rec[3 * p + 0];
      const float4 b = s_rec[3 * p + 1];
      const float4 cz = s_rec[3 * p + 2];
      // clip_coef = [x, y, 1] @ inv (pipeline.py:177-193)
      const float c0 = (x * a.x + y * a.w) + b.z;
      const float c1 = (x * a.y + y * b.x) + b.w;
      const float c2 = (x * a.z + y * b.y) + cz.x;
      if (all_nonneg(c0, c1, c2)) {
        if ((s_flag[p] & kCandidate) == kCandidate) {
          const float z = ((c0 * cz.y + c1 * cz.z) + c2 * cz.w) * vp22 + vp23;
          const unsigned long long key = pack_key(z, base + p);
          const uint32_t o = static_cast<uint32_t>(key >> 32);
          if (key < best[0]) {
            second = min(second, static_cast<uint32_t>(best[0] >> 32));
          } else {
            second = min(second, o);
          }
          insert_key<kL>(best, key);
        }
      }
    }
    __syncthreads();
  }
  const bool valid = i < W && j < H;
  if (valid) {
    const int64_t pix = J.pixel_begin + static_cast<int64_t>(i) * H + j;
#pragma unroll
    for (int l = 0; l < kL; ++l) {
      const uint32_t o = static_cast<uint32_t>(best[l] >> 32);
      winner[l * B.total_pixels + pix] =
          (best[l] == kEmptyKey || o == kInfOrder) ? -1 : static_cast<int32_t>(best[l] & 0xffffffffu);
    }
  }
  if (B.near_ties) count_near_tie(B.near_ties, valid && is_near_tie(best[0], second));
}

// One thread per pixel: the chosen primitive's fragment, mixed and merged
// (kLayered: the batch has layered jobs, whose pixels shade and mix every
// slot).
template <bool kLayered>
__global__ void __launch_bounds__(kScanThreads)
shade_kernel(RastBatch B, const float4* __restrict__ setup, const float* __restrict__ var,
             int vstride, const int32_t* __restrict__ winner, const unsigned long long* __restrict__ keys) {
  __shared__ RastJob sJ;
  after_previous();
  load_job_to_shared(B.jobs + blockIdx.y, &sJ);
  __syncthreads();
  const RastJob& J = sJ;
  const int W = J.width, H = J.height;
  const int tiles_j = (H + kTile - 1) / kTile;
  const int tiles_i = (W + kTile - 1) / kTile;
  if (static_cast<int>(blockIdx.x) >= tiles_i * tiles_j) return;
  const int ti = blockIdx.x / tiles_j, tj = blockIdx.x % tiles_j;
  const int i = ti * kTile + threadIdx.y;
  const int j = tj * kTile + threadIdx.x;
  if (i >= W || j >= H) return;
  const int64_t pix = J.pixel_begin + static_cast<int64_t>(i) * H + j;
  PixelResult r;
  const VertexRows src{var, vstride, J.vout_begin};
  const int L = kLayered ? job_layers(J, B.max_layers) : 0;
  if (kLayered && L > 0) {
    resolve_layers<-1>(J, B.pools, setup + J.setup_begin * 4, i, j, winner + pix, B.total_pixels, L, src, &r);
    save_layers(B.pools, winner + pix, B.total_pixels, pix, L);
  } else {
    int w;
    if (keys) {  // scan_kernel's
      const unsigned long long key = keys[pix];
      w = (key == kEmptyKey || static_cast<uint32_t>(key >> 32) == kInfOrder) ? -1 : static_cast<int>(key & 0xffffffffu);
    } else {
      w = winner[pix];
    }
    resolve_pixel<-1>(J, B.pools, setup + J.setup_begin * 4, i, j, w, src, &r);
  }
  store_pixel(J, B.pools, pix, r);
}

// ------------------------------------------------------------- launcher

struct PlainLayout {
  size_t clip_off, var_off, setup_off, winner_off, total;
  int vstride;
  bool keyed;
};

static PlainLayout plain_layout(const RastBatch& b) {
  PlainLayout L{};
  int vstride = 0;
  for (int s = 0; s < 7; ++s)
    if (b.shader_mask & (1 << s)) vstride = std::max(vstride, varying_count(s));
  L.vstride = vstride;
  size_t off = 0;
  L.clip_off = off;
  off = align256(off + static_cast<size_t>(b.total_vout) * sizeof(float4));
  L.var_off = off;
  off = align256(off + static_cast<size_t>(b.total_vout) * vstride * sizeof(float));
  L.setup_off = off;
  off = align256(off + static_cast<size_t>(b.total_setup) * 4 * sizeof(float4));
  L.winner_off = off;
  // one key per pixel (scan_kernel), or one winner, or RAST_MAX_LAYERS with layered jobs (slots_kernel); a tie
  // counter's winners take a key's room, so that a workspace serves its batch with the counter and without
  L.keyed = b.max_layers == 0 && b.near_ties == nullptr;
  const size_t slots = b.max_layers > 0 ? RAST_MAX_LAYERS : 2;
  off = align256(off + static_cast<size_t>(b.total_pixels) * slots * sizeof(int32_t));
  L.total = off;
  return L;
}

}  // namespace rast

using namespace rast;

extern "C" size_t rast_plain_workspace_bytes(const RastBatch* batch) {
  if (!batch) return 0;
  return plain_layout(*batch).total;
}

static int render_plain(const RastBatch* batch, void* workspace, size_t workspace_bytes,
                        void* stream, RastProfile* profile) {
  int st = check_batch(batch);
  if (st != RAST_OK) return st;
  const RastBatch& b = *batch;
  if (b.total_pixels > 0 && (b.max_width < 1 || b.max_height < 1)) return RAST_ERR_INVALID_ARGUMENT;
  const PlainLayout L = plain_layout(b);
  if (workspace_bytes < L.total) return RAST_ERR_WORKSPACE_TOO_SMALL;
  if (L.total > 0 && (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255)))
    return RAST_ERR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  float4* clip = reinterpret_cast<float4*>(ws + L.clip_off);
  float* var = reinterpret_cast<float*>(ws + L.var_off);
  float4* setup = reinterpret_cast<float4*>(ws + L.setup_off);
  int32_t* winner = reinterpret_cast<int32_t*>(ws + L.winner_off);
  Profiler prof(profile, s, "rast_render_plain");

  unsigned long long* keys = nullptr;
  int64_t blocks = 0;
  unsigned splits = 1;
  size_t key_bytes = 0;  // of the keys, cleared for the splits' minima
  if (L.keyed && b.total_pixels > 0) {
    keys = reinterpret_cast<unsigned long long*>(winner);
    const int64_t threads = static_cast<int64_t>((b.max_width + kScanPixels - 1) / kScanPixels) * b.max_height;
    blocks = (threads + kScanBlock - 1) / kScanBlock;
    // Splits: until eight blocks per SM are there (a 254x152 pass of 8,960 faces: 66 us; 69 at twelve), of
    // at least 64 primitives each (a block's staging and its atomics cost what a few dozen primitives do).
    const int64_t fill = static_cast<int64_t>(sm_count()) * 8 / (blocks * b.n_jobs);
    splits = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(fill, b.max_faces / 64)));
    if (splits > 1) key_bytes = static_cast<size_t>(b.total_pixels) * sizeof(*keys);
  }
  if (b.total_vout > 0 || key_bytes > 0) {
    const size_t fill = key_bytes > 0 ? begin_blocks(key_bytes, 1, sm_count()) : 0;
    const size_t most = std::max<size_t>((b.max_verts + 255) / 256, (fill + b.n_jobs - 1) / b.n_jobs);
    const dim3 grid(static_cast<unsigned>(most), static_cast<unsigned>(b.n_jobs));
    vertex_kernel<<<grid, 256, 0, s>>>(b, clip, var, L.vstride, keys, key_bytes);
    prof.mark("vertex_kernel");
  }
  if (b.total_setup > 0) {
    const dim3 grid(static_cast<unsigned>((b.max_faces + 255) / 256), static_cast<unsigned>(b.n_jobs));
    if (b.total_vout > 0 || key_bytes > 0)
      launch_after(setup_kernel, grid, 256, s, b, clip, setup);
    else
      setup_kernel<<<grid, 256, 0, s>>>(b, clip, setup);
    prof.mark("setup_kernel");
  }
  if (b.total_pixels > 0) {
    const int tiles = ((b.max_width + kTile - 1) / kTile) * ((b.max_height + kTile - 1) / kTile);
    const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(b.n_jobs));
    const dim3 block(kTile, kTile);
    if (L.keyed) {
      const dim3 sgrid(static_cast<unsigned>(blocks), static_cast<unsigned>(b.n_jobs), splits);
      if (b.total_setup == 0)
        scan_kernel<<<sgrid, kScanBlock, 0, s>>>(b, setup, keys);
      else
        launch_after(scan_kernel, sgrid, kScanBlock, s, b, setup, keys);
      prof.mark("scan_kernel");
    } else {
      const auto kernel = b.max_layers > 0 ? slots_kernel<RAST_MAX_LAYERS> : slots_kernel<1>;
      kernel<<<grid, block, 0, s>>>(b, setup, winner);
      prof.mark("slots_kernel");
    }
    const auto shade = b.max_layers > 0 ? shade_kernel<true> : shade_kernel<false>;
    launch_after(shade, grid, block, s, b, setup, var, L.vstride, winner, keys);
    prof.mark("shade_kernel");
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return RAST_ERR_CUDA;
  return prof.finish();
}

extern "C" int rast_render_plain(const RastBatch* batch, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  return render_plain(batch, workspace, workspace_bytes, stream, nullptr);
}

extern "C" int rast_render_plain_profiled(const RastBatch* batch, void* workspace,
                                          size_t workspace_bytes, void* stream,
                                          RastProfile* profile) {
  return render_plain(batch, workspace, workspace_bytes, stream, profile);
}
