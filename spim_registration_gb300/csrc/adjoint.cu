// Small kernels of the forward/backward pair of the Poisson image-formation model:
// cross-spectrum accumulation and lag extraction (PSF gradient), mirror fold (psi gradient).
#include "engine.h"

namespace mvd {

static int grid1(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 152LL * 16 ? 152LL * 16 : b));
}

__global__ void cross_accumulate_kernel(const float2* __restrict__ B, const float2* __restrict__ A, int ntiles,
                                        long long elems, float2* __restrict__ acc) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < elems; i += (long long)gridDim.x * blockDim.x) {
    float2 s = make_float2(0.f, 0.f);
    for (int t = 0; t < ntiles; ++t) {
      const float2 b = __ldg(B + t * elems + i), a = __ldg(A + t * elems + i);
      // b * conj(a)
      s.x += b.x * a.x + b.y * a.y;
      s.y += b.y * a.x - b.x * a.y;
    }
    acc[i] = s;
  }
}

void dev_cross_accumulate(const ConvPlan& p, const float2* B, const float2* A, float2* acc, cudaStream_t s) {
  require_scalar(p, "the cross-spectrum sum");
  cross_accumulate_kernel<<<grid1(p.otf_elems), 256, 0, s>>>(B, A, (int)p.tiles.size(), p.otf_elems, acc);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void extract_lags_kernel(const float* __restrict__ R, int tx, int ty, int tz, int kx, int ky, int kz,
                                    float scale, float* __restrict__ G) {
  const long long n = (long long)kx * ky * kz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int jx = (int)(i % kx), jy = (int)((i / kx) % ky), jz = (int)(i / ((long long)kx * ky));
    const int lx = ((jx - kx / 2) % tx + tx) % tx;
    const int ly = ((jy - ky / 2) % ty + ty) % ty;
    const int lz = ((jz - kz / 2) % tz + tz) % tz;
    G[i] = scale * R[((long long)lz * ty + ly) * tx + lx];
  }
}

void dev_extract_lags(const float* R, int tx, int ty, int tz, int kx, int ky, int kz, float scale, float* G,
                      cudaStream_t s) {
  extract_lags_kernel<<<grid1((long long)kx * ky * kz), 256, 0, s>>>(R, tx, ty, tz, kx, ky, kz, scale, G);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// tab layout: [sx (nx+1) | ix | sy (ny+1) | iy | sz (nz+1) | iz] with the idx lengths nx+2hx etc.
// A warp takes a row of x, or `run` voxels of it, so that y and z need one division.  An axis longer than the kernel's half
// has at most two positions per voxel; their up to eight values are all loaded before they are added, in
// the order of the lists (one by one, each sum waited for the load before it: 71 us at 192^3, 31x31x61
// kernel; now 43).
__global__ void __launch_bounds__(256) fold_mirror_kernel(const float* __restrict__ c, int nxe, int nye,
                                                          const int* __restrict__ sx, const int* __restrict__ ix,
                                                          const int* __restrict__ sy, const int* __restrict__ iy,
                                                          const int* __restrict__ sz, const int* __restrict__ iz,
                                                          int nx, int ny, int nz, int run, float* __restrict__ g) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int segs = (nx + run - 1) / run;
  const long long items = (long long)ny * nz * segs;
  for (long long i = blockIdx.x * (long long)warps + (threadIdx.x >> 5); i < items; i += (long long)gridDim.x * warps) {
    const long long r = segs == 1 ? i : i / segs;
    const int xs = (int)(i - r * segs) * run, xe = min(nx, xs + run);
    const int z = (int)(r / ny), y = (int)(r - (long long)z * ny);
    const int a0 = sz[z], a1 = sz[z + 1], b0 = sy[y], b1 = sy[y + 1];
    const bool two_a = a1 - a0 > 1, two_b = b1 - b0 > 1;
    const float* const r00 = c + ((long long)iz[a0] * nye + iy[b0]) * nxe;
    const float* const r01 = two_b ? c + ((long long)iz[a0] * nye + iy[b0 + 1]) * nxe : nullptr;
    const float* const r10 = two_a ? c + ((long long)iz[a0 + 1] * nye + iy[b0]) * nxe : nullptr;
    const float* const r11 = two_a && two_b ? c + ((long long)iz[a0 + 1] * nye + iy[b0 + 1]) * nxe : nullptr;
    const bool few = a1 - a0 <= 2 && b1 - b0 <= 2;
#pragma unroll 2
    for (int x = xs + lane; x < xe; x += 32) {
      const int e0 = sx[x], e1 = sx[x + 1];
      const float old = g[r * nx + x];
      float acc = 0.f;
      if (few && e1 - e0 <= 2) {
        const bool two = e1 - e0 > 1;
        const int p = ix[e0], q = two ? ix[e0 + 1] : 0;
        float v[8];
        v[0] = r00[p];
        v[1] = two ? r00[q] : 0.f;
        v[2] = two_b ? r01[p] : 0.f;
        v[3] = two && two_b ? r01[q] : 0.f;
        v[4] = two_a ? r10[p] : 0.f;
        v[5] = two && two_a ? r10[q] : 0.f;
        v[6] = two_a && two_b ? r11[p] : 0.f;
        v[7] = two && two_a && two_b ? r11[q] : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += v[k];  // a missing one adds zero
      } else {
        for (int a = a0; a < a1; ++a)
          for (int b = b0; b < b1; ++b) {
            const float* row = c + ((long long)iz[a] * nye + iy[b]) * nxe;
            for (int e = e0; e < e1; ++e) acc += row[ix[e]];
          }
      }
      g[r * nx + x] = old + acc;
    }
  }
}

void dev_fold_mirror(const float* c, int nxe, int nye, const int* tab, int nx, int ny, int nz, float* g,
                     cudaStream_t s) {
  const int* sx = tab;
  const int* ix = sx + nx + 1;
  const int* sy = ix + nxe;
  const int* iy = sy + ny + 1;
  const int* sz = iy + nye;
  const int* iz = sz + nz + 1;
  // whole rows where these are 64 warps per SM, else as many runs of at least 64 voxels: a row each took
  // 8.7 ms at 100000x30x1, 3.3 ms at 20000x5x3 and 41 us at 2000x2000x1 (now 56, 20 and 25 us)
  const long long rows = (long long)ny * nz;
  const int segs = (int)std::max(1LL, std::min((152LL * 64 + rows - 1) / rows, (nx + 63LL) / 64));
  const int run = ((nx + segs - 1) / segs + 31) / 32 * 32;
  const long long items = rows * ((nx + run - 1) / run);
  fold_mirror_kernel<<<(int)std::min((items + 7) / 8, 152LL * 32), 256, 0, s>>>(c, nxe, nye, sx, ix, sy, iy, sz, iz, nx,
                                                                             ny, nz, run, g);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

void mirror_fold_table(int n, int h, std::vector<int>& start, std::vector<int>& idx) {
  std::vector<std::vector<int>> lists(n);
  for (int u = -h; u < n + h; ++u) {
    int y;
    if (n == 1) {
      y = 0;
    } else {
      const int period = 2 * n - 2;
      int m = u % period;
      if (m < 0) m += period;
      y = m < n ? m : period - m;
    }
    lists[y].push_back(u + h);
  }
  start.assign(n + 1, 0);
  idx.clear();
  for (int y = 0; y < n; ++y) {
    start[y] = (int)idx.size();
    idx.insert(idx.end(), lists[y].begin(), lists[y].end());
  }
  start[n] = (int)idx.size();
}

}  // namespace mvd
