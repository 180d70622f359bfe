// PSF pipeline on the GPU: extraction of the point spread function from bead neighbourhoods
// and its transformation into the fused frame.
//   ExtractPSF.extractPSFLocal  spim/process/fusion/deconvolution/ExtractPSF.java:374-415
//   ExtractPSF.normalize        :298-316
//   ExtractPSF.transformPSF     :325-372
//   ExtractPSF.transform        :417-464
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>

#include "../../include/mvdecon.h"
#include "engine.h"

using namespace mvd;

namespace mvd {
void set_last_error(const std::string& msg);
}

namespace {

// Trilinear interpolation at (tx, ty, tz) of the volume extended with zeros; the corner weights
// come from the fractional parts, the sum is in float.
__device__ __forceinline__ float trilinear(const float* __restrict__ v, int sx, int sy, int sz, double tx, double ty,
                                           double tz) {
  const double fx = floor(tx), fy = floor(ty), fz = floor(tz);
  const int x0 = (int)fx, y0 = (int)fy, z0 = (int)fz;
  const float ax = (float)(tx - fx), ay = (float)(ty - fy), az = (float)(tz - fz);
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int bx = c & 1, by = (c >> 1) & 1, bz = (c >> 2) & 1;
    const int x = x0 + bx, y = y0 + by, z = z0 + bz;
    const float val = (x >= 0 && y >= 0 && z >= 0 && x < sx && y < sy && z < sz)
                          ? __ldg(v + ((long long)z * sy + y) * sx + x)
                          : 0.f;
    const float w = (bx ? ax : 1.f - ax) * (by ? ay : 1.f - ay) * (bz ? az : 1.f - az);
    acc = __fmaf_rn(w, val, acc);
  }
  return acc;
}

// One bead as the extraction needs it: every PSF voxel p samples the view at p - size / 2 +
// location, so the fractions of the position are the bead's, not the voxel's, and the integer part
// is the bead's base (reduced to [0, dim)) plus p.
struct Bead {
  int x, y, z;
  float ax, ay, az;
};

// A location (x, y, z) split in double (exactly)
__host__ __device__ inline Bead split_bead(const double* location, int3 dims, int3 half) {
  const int size[3] = {dims.x, dims.y, dims.z}, h[3] = {half.x, half.y, half.z};
  int base[3];
  float frac[3];
  for (int d = 0; d < 3; ++d) {
    const double t = location[d], f = floor(t);
    frac[d] = (float)(t - f);  // NaN for a location that is not finite
    const double b = isfinite(t) ? fmod(f - (double)h[d], (double)size[d]) : 0.0;
    base[d] = (int)(b < 0.0 ? b + size[d] : b);
  }
  return Bead{base[0], base[1], base[2], frac[0], frac[1], frac[2]};
}

// The beads of n locations on the device.  A call passes up to kMostByValue beads as a kernel's
// parameter, so that nothing of the caller's memory is read after it returns and nothing is waited for.
// More beads, and those of a call under capture, are split on the device from a copy of the caller's own
// array: a replay then reads that and no host memory of the call's.  4 views of 436 beads, 11x25x29 PSFs:
// 653 to 671 us by value, 675 to 715 by a copy that is waited for.
template <int N>
struct BeadBlock {
  Bead b[N];
};
constexpr int kMostByValue = 1360;  // 32640 of the 32764 bytes that a kernel's parameters may take
template <int N>
__global__ void store_beads_kernel(const __grid_constant__ BeadBlock<N> block, int n, Bead* __restrict__ beads) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < n) beads[l] = block.b[l];
}
__global__ void split_beads_kernel(const double* __restrict__ locations, int n, int3 dims, int3 half,
                                   Bead* __restrict__ beads) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < n) beads[l] = split_bead(locations + 3LL * l, dims, half);
}
template <int N>
void store_beads(const double* locations, int n, int3 dims, int3 half, Bead* beads, cudaStream_t s) {
  BeadBlock<N> block;
  for (int l = 0; l < n; ++l) block.b[l] = split_bead(locations + 3 * l, dims, half);
  store_beads_kernel<N><<<(n + 127) / 128, 128, 0, s>>>(block, n, beads);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// Position i of an axis of n voxels repeated; one subtraction unless the PSF is larger than the view.
// Unsigned: a base below 2^31 plus a position in the PSF may pass 2^31.
__device__ __forceinline__ int wrap(unsigned i, unsigned n) {
  if (i >= n) {
    i -= n;
    if (i >= n) i %= n;
  }
  return (int)i;
}

constexpr int kRunY = 4, kRunZ = 8;  // PSF voxels of a thread: 4 x 8 at one x, lanes along x
constexpr int kExtractThreads = 128;

// (1 - a) v0 + a v1 with one rounding beside that of v1 - v0, which is exact for whole numbers and near
// neighbours; the weighted form (three roundings) only where an infinity or NaN comes out, for its
// result there.
__device__ __forceinline__ float lerp(float a, float v0, float v1) {
  const float t = __fmaf_rn(a, v1 - v0, v0);
  return fabsf(t) <= FLT_MAX ? t : __fmaf_rn(a, v1, (1.f - a) * v0);
}

// Partial sums of the beads [chunk * per, chunk * per + per): part[chunk][voxel].  The trilinear
// weights of a bead are the same for every voxel, so a thread interpolates a 5 x 9 patch of rows
// along x once and then along y and z: 2.8 loads and 7 multiply-adds per voxel and bead.  One
// thread per voxel with all beads, positions in double, took 1.2 ms for 500 beads and a 31x31x61
// PSF (FP64 and integer remainders); this takes 0.06 ms, bound by the latency of the loads.
__global__ void __launch_bounds__(kExtractThreads, 4) extract_partial_kernel(
    const float* __restrict__ img, int sx, int sy, int sz, const Bead* __restrict__ beads, int n, int per, int px,
    int py, int pz, int xb, int yb, int items, float* __restrict__ part) {
  const int item = blockIdx.x * (kExtractThreads / 32) + (threadIdx.x >> 5);
  if (item >= items) return;
  const int x = (item % xb) * 32 + (threadIdx.x & 31);
  const int y0 = (item / xb) % yb * kRunY, z0 = item / (xb * yb) * kRunZ;
  float acc[kRunZ][kRunY];
#pragma unroll
  for (int k = 0; k < kRunZ; ++k)
#pragma unroll
    for (int y = 0; y < kRunY; ++y) acc[k][y] = 0.f;
  const int l1 = min(n, ((int)blockIdx.y + 1) * per);
  for (int l = blockIdx.y * per; l < l1; ++l) {
    const Bead b = beads[l];
    const int x0 = wrap((unsigned)b.x + x, sx), x1 = wrap((unsigned)b.x + x + 1, sx);
    int row[kRunY + 1];
#pragma unroll
    for (int y = 0; y <= kRunY; ++y) row[y] = wrap((unsigned)b.y + y0 + y, sy);
    float last[kRunY];
#pragma unroll
    for (int k = 0; k <= kRunZ; ++k) {
      const float* slice = img + (long long)wrap((unsigned)b.z + z0 + k, sz) * sy * sx;
      float t[kRunY + 1];
#pragma unroll
      for (int y = 0; y <= kRunY; ++y) {
        const float* r = slice + (long long)row[y] * sx;
        t[y] = lerp(b.ax, __ldg(r + x0), __ldg(r + x1));
      }
#pragma unroll
      for (int y = 0; y < kRunY; ++y) {
        const float u = lerp(b.ay, t[y], t[y + 1]);
        if (k > 0) acc[k - 1][y] += lerp(b.az, last[y], u);
        last[y] = u;
      }
    }
  }
  if (x >= px) return;
  float* out = part + (long long)blockIdx.y * px * py * pz + x;
#pragma unroll
  for (int k = 0; k < kRunZ; ++k)
#pragma unroll
    for (int y = 0; y < kRunY; ++y)
      if (y0 + y < py && z0 + k < pz) out[((long long)(z0 + k) * py + y0 + y) * px] = acc[k][y];
}

// psf = the sum of the partial sums in their order, with the additions' own errors (two-sums) added at
// the end; the extremes of each block's voxels
__global__ void extract_sum_kernel(const float* __restrict__ part, int chunks, int n, float* __restrict__ psf,
                                   float2* __restrict__ ends) {
  __shared__ float2 red[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float lo = INFINITY, hi = -INFINITY;
  if (i < n) {
    float s = 0.f, e = 0.f;
    for (int c = 0; c < chunks; ++c) {
      const float v = part[(long long)c * n + i], t = s + v, bb = t - s;
      e += (s - (t - bb)) + (v - bb);
      s = t;
    }
    if (fabsf(s + e) <= FLT_MAX) s += e;
    psf[i] = s;
    lo = fminf(lo, s);
    hi = fmaxf(hi, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      lo = fminf(lo, red[w].x);
      hi = fmaxf(hi, red[w].y);
    }
    ends[blockIdx.x] = make_float2(lo, hi);
  }
}

// (v - min) / (max - min) in double over many blocks (each reduces the blocks' extremes again): in
// one block, the FP64 pipe of a single SM took 0.1 ms for 58 thousand voxels
__global__ void normalize_min_max_kernel(float* __restrict__ p, int n, const float2* __restrict__ ends, int nends) {
  __shared__ float2 red[32];
  float lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < nends; i += blockDim.x) {
    lo = fminf(lo, ends[i].x);
    hi = fmaxf(hi, ends[i].y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    lo = fminf(lo, red[w].x);
    hi = fmaxf(hi, red[w].y);
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = (float)(((double)p[i] - (double)lo) / ((double)hi - (double)lo));
}

struct Affine64 {
  double m[12];
};

// out[p] = psf(model^-1 (p + offset)), trilinear over the PSF extended with zeros
__global__ void transform_psf_kernel(const float* __restrict__ psf, int sx, int sy, int sz, Affine64 inv,
                                     double offx, double offy, double offz, int nx, int ny, int nz,
                                     float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nx * ny * nz) return;
  const int x = i % nx, y = (i / nx) % ny, z = i / (nx * ny);
  const double p0 = x + offx, p1 = y + offy, p2 = z + offz;
  const double t0 = inv.m[0] * p0 + inv.m[1] * p1 + inv.m[2] * p2 + inv.m[3];
  const double t1 = inv.m[4] * p0 + inv.m[5] * p1 + inv.m[6] * p2 + inv.m[7];
  const double t2 = inv.m[8] * p0 + inv.m[9] * p1 + inv.m[10] * p2 + inv.m[11];
  out[i] = trilinear(psf, sx, sy, sz, t0, t1, t2);
}

bool invert(const double* a, Affine64& out) {
  const double r00 = a[0], r01 = a[1], r02 = a[2], r10 = a[4], r11 = a[5], r12 = a[6], r20 = a[8], r21 = a[9],
               r22 = a[10];
  const double det = r00 * (r11 * r22 - r12 * r21) - r01 * (r10 * r22 - r12 * r20) + r02 * (r10 * r21 - r11 * r20);
  if (!(std::fabs(det) > 0.0)) return false;
  const double inv[9] = {(r11 * r22 - r12 * r21) / det, (r02 * r21 - r01 * r22) / det, (r01 * r12 - r02 * r11) / det,
                         (r12 * r20 - r10 * r22) / det, (r00 * r22 - r02 * r20) / det, (r02 * r10 - r00 * r12) / det,
                         (r10 * r21 - r11 * r20) / det, (r01 * r20 - r00 * r21) / det, (r00 * r11 - r01 * r10) / det};
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) out.m[4 * r + c] = inv[3 * r + c];
    out.m[4 * r + 3] = -(inv[3 * r] * a[3] + inv[3 * r + 1] * a[7] + inv[3 * r + 2] * a[11]);
  }
  return true;
}

int blocks_for(long long n) { return (int)((n + 255) / 256); }

// An event behind a copy from the caller's memory; the call waits for it, on its way out of an error too.
struct CopyDone {
  cudaEvent_t e = nullptr;
  void record(cudaStream_t s) {
    MVD_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    MVD_CHECK(cudaEventRecord(e, s));
  }
  void wait() {
    if (e) MVD_CHECK(cudaEventSynchronize(e));
  }
  ~CopyDone() {
    if (!e) return;
    cudaEventSynchronize(e);
    cudaEventDestroy(e);
  }
};

}  // namespace

extern "C" int mvd_transformed_psf_size(const int* psf_dims, const double* model, int* out_dims, double* offset) {
  set_last_error("");
  if (!psf_dims || !model || !out_dims || !offset) {
    set_last_error("NULL argument");
    return MVD_ERR_ARG;
  }
  for (int d = 0; d < 3; ++d)
    if (psf_dims[d] < 1) {
      set_last_error("PSF sizes must be positive");
      return MVD_ERR_ARG;
    }
  // estimateBounds of the interval [0, dim - 1]: the bounding box of its 8 transformed corners
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int c = 0; c < 8; ++c) {
    const double p[3] = {(c & 1) ? psf_dims[0] - 1.0 : 0.0, (c & 2) ? psf_dims[1] - 1.0 : 0.0,
                         (c & 4) ? psf_dims[2] - 1.0 : 0.0};
    for (int d = 0; d < 3; ++d) {
      const double t = model[4 * d] * p[0] + model[4 * d + 1] * p[1] + model[4 * d + 2] * p[2] + model[4 * d + 3];
      lo[d] = std::fmin(lo[d], t);
      hi[d] = std::fmax(hi[d], t);
    }
  }
  // the PSF's centre voxel (dim / 2, integer) maps to the centre of the odd-sized result
  const double ctr[3] = {(double)(psf_dims[0] / 2), (double)(psf_dims[1] / 2), (double)(psf_dims[2] / 2)};
  for (int d = 0; d < 3; ++d) {
    long long ns = (long long)(hi[d] - lo[d]) + 1;
    if (ns % 2 == 0) ++ns;
    if (ns > (1 << 20)) {
      set_last_error("transformed PSF too large");
      return MVD_ERR_ARG;
    }
    out_dims[d] = (int)ns;
    const double tc = model[4 * d] * ctr[0] + model[4 * d + 1] * ctr[1] + model[4 * d + 2] * ctr[2] + model[4 * d + 3];
    offset[d] = tc - (double)(ns / 2);
  }
  return MVD_OK;
}

extern "C" int mvd_extract_psf(const float* img, const int* dims, const double* locations, int num_locations,
                               const int* psf_dims, float* psf, int normalize, int devCUDA, void* stream) {
  try {
    set_last_error("");
    if (!img || !dims || !psf_dims || !psf || (num_locations > 0 && !locations) || num_locations < 0) {
      set_last_error("NULL argument or negative location count");
      return MVD_ERR_ARG;
    }
    for (int d = 0; d < 3; ++d)
      if (dims[d] < 1 || psf_dims[d] < 1) {
        set_last_error("sizes must be positive");
        return MVD_ERR_ARG;
      }
    const long long np = (long long)psf_dims[0] * psf_dims[1] * psf_dims[2];
    if (np > (1LL << 30)) {
      set_last_error("PSF too large");
      return MVD_ERR_ARG;
    }
    MVD_CHECK(cudaSetDevice(devCUDA));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int xb = (psf_dims[0] + 31) / 32, yb = (psf_dims[1] + kRunY - 1) / kRunY;
    // warps: at most the PSF's voxels (2^30), though their threads may be more than an int holds
    const int items = xb * yb * ((psf_dims[2] + kRunZ - 1) / kRunZ);
    // chunks of beads: about 24 warps per SM in all, partial sums of at most 256 MB
    const long long want = std::min((152LL * 24 + items - 1) / items, std::max(1LL, (64LL << 20) / np));
    const int per = (int)std::max(1LL, (num_locations + want - 1) / want);
    const int chunks = std::max(1, (num_locations + per - 1) / per);
    const int nends = blocks_for(np);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    MVD_CHECK(cudaStreamIsCapturing(s, &capture));
    const bool by_value = capture == cudaStreamCaptureStatusNone && num_locations <= kMostByValue;
    const size_t lb = by_value ? 0 : (size_t)num_locations * 3 * sizeof(double),
                 bb = ((size_t)num_locations * sizeof(Bead) + 7) / 8 * 8,
                 eb = (size_t)nends * sizeof(float2);
    const CallBuf buf(devCUDA, lb + bb + eb + (size_t)chunks * np * sizeof(float), s);
    double* d_loc = buf.as<double>();
    Bead* d_beads = reinterpret_cast<Bead*>(buf.as<char>() + lb);
    float2* d_ends = reinterpret_cast<float2*>(buf.as<char>() + lb + bb);
    float* d_part = reinterpret_cast<float*>(buf.as<char>() + lb + bb + eb);
    const int3 size = make_int3(dims[0], dims[1], dims[2]),
               half = make_int3(psf_dims[0] / 2, psf_dims[1] / 2, psf_dims[2] / 2);
    // nothing of the caller's pageable memory is read once the call has returned
    CopyDone copied;
    if (by_value) {
      if (num_locations > 512)
        store_beads<kMostByValue>(locations, num_locations, size, half, d_beads, s);
      else if (num_locations > 160)
        store_beads<512>(locations, num_locations, size, half, d_beads, s);
      else if (num_locations > 0)
        store_beads<160>(locations, num_locations, size, half, d_beads, s);
    } else if (num_locations > 0) {
      MVD_CHECK(cudaMemcpyAsync(d_loc, locations, lb, cudaMemcpyHostToDevice, s));
      if (capture == cudaStreamCaptureStatusNone && !async_copy_source(locations)) copied.record(s);
      split_beads_kernel<<<(num_locations + 127) / 128, 128, 0, s>>>(d_loc, num_locations, size, half, d_beads);
      MVD_CHECK(cudaGetLastError());
      count_launch();
    }
    constexpr int kWarps = kExtractThreads / 32;
    extract_partial_kernel<<<dim3((items + kWarps - 1) / kWarps, chunks), kExtractThreads, 0, s>>>(
        img, dims[0], dims[1], dims[2], d_beads, num_locations, per, psf_dims[0], psf_dims[1], psf_dims[2], xb, yb, items,
        d_part);
    MVD_CHECK(cudaGetLastError());
    count_launch();
    extract_sum_kernel<<<nends, 256, 0, s>>>(d_part, chunks, (int)np, psf, d_ends);
    MVD_CHECK(cudaGetLastError());
    count_launch();
    if (normalize) {
      normalize_min_max_kernel<<<nends, 256, 0, s>>>(psf, (int)np, d_ends, nends);
      MVD_CHECK(cudaGetLastError());
      count_launch();
    }
    copied.wait();
    return MVD_OK;
  } catch (const CudaError& e) {
    set_last_error(e.what());
    return MVD_ERR_CUDA;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return MVD_ERR_INTERNAL;
  }
}

extern "C" int mvd_transform_psf(const float* psf, const int* psf_dims, const double* model, const int* out_dims,
                                 const double* offset, float* out, int devCUDA, void* stream) {
  try {
    set_last_error("");
    if (!psf || !psf_dims || !model || !out_dims || !offset || !out) {
      set_last_error("NULL argument");
      return MVD_ERR_ARG;
    }
    for (int d = 0; d < 3; ++d)
      if (psf_dims[d] < 1 || out_dims[d] < 1) {
        set_last_error("sizes must be positive");
        return MVD_ERR_ARG;
      }
    const long long no = (long long)out_dims[0] * out_dims[1] * out_dims[2];
    if (no > (1LL << 30)) {
      set_last_error("output too large");
      return MVD_ERR_ARG;
    }
    Affine64 inv;
    if (!invert(model, inv)) {
      set_last_error("the affine transform is singular");
      return MVD_ERR_ARG;
    }
    MVD_CHECK(cudaSetDevice(devCUDA));
    transform_psf_kernel<<<blocks_for(no), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        psf, psf_dims[0], psf_dims[1], psf_dims[2], inv, offset[0], offset[1], offset[2], out_dims[0], out_dims[1],
        out_dims[2], out);
    MVD_CHECK(cudaGetLastError());
    count_launch();
    return MVD_OK;
  } catch (const CudaError& e) {
    set_last_error(e.what());
    return MVD_ERR_CUDA;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return MVD_ERR_INTERNAL;
  }
}
