// Tiled FFT convolution passes on pairs of transforms (the default path of every convolution whose
// kernel is not nearly as long as their longest transforms).
//
// The three passes are those of kernels.cuh (forward planes, z pencils, inverse planes over
// overlap-save tiles), rebuilt around packed FP32 arithmetic (pair_fft.cuh):
//
//  * Every stage works on two transforms at once, one 16-byte access and one packed instruction
//    for both: the x stages on rows 2q and 2q + 1, the column stages on two columns, the z stages
//    on two pencils.  The 512-thread scalar kernels were bound by issue slots (about 60 thread
//    instructions per real of a forward slice); the packed ones issue about half of that.
//  * Every x and y length is R0 x R1 (two register DFTs).  Stage 0 reads j + R1 r and writes its results
//    back to j + R1 k0; stage 1 works in place on the R1 consecutive elements of block k0.  So a
//    stage overwrites exactly what it read: one plane buffer, one barrier between stages, and
//    frequency f = k0 + R0 m ends at position R1 k0 + m.  The spectra keep that order in x, y and
//    z: the kernel spectrum goes through the same passes, and the inverse stages undo it.
//  * The real-to-half-spectrum step takes columns f and M - f together (it needs both), as one
//    unit of work: two packed DFTs over the rows (j, j + 1).  It forms twice the half spectrum; the
//    kernel spectrum carries the remaining factor 1/4 of the product (exact).
//  * Spectrum element: (re_a, re_b, im_a, im_b) of two columns a = c and b = c + pc, one 16-byte
//    unit, in slices [z][row position][c].
//
// Lengths come from the plan at run time; only the radices are compiled (a switch per stage), so
// every tile shape runs these kernels.
//
// What bounds them: the 128 registers of a packed 16 to 20-point DFT leave 16 warps per SM, and
// the stages between two barriers move together, so shared-memory accesses (8.6 thousand cycles of
// a 288x160 slice), FP32 arithmetic (10.6), global accesses and their latency add up (35 for the
// forward pass) instead of overlapping.  Larger tiles win although they leave one CTA per SM: the
// halo they save is worth more than the second CTA's overlap (512x512x256, 31x31x61 PSFs: 7.70 ms
// per iteration at up to 226 KB per plane against 8.98 at 112 KB and 9.76 at 74 KB).
// Measured per iteration, scalar kernels / these: 4 views of 512x512x256 9.17 / 7.51 ms; 4 views of
// 256x256x192 with 15x15x41 PSFs 1.70 / 1.54 ms; 6 crops of 256^3 2.10 / 1.46 ms (shapes without
// compiled scalar kernels); 2 views of 128x128x64 0.16 / 0.11 ms.
#pragma once
#include "kernels.cuh"
#include "pair_fft.cuh"

namespace mvd {

constexpr int kPairThreads = 512;  // largest plane CTA; 128 registers per thread
constexpr int kPairZThreads = 160;  // at most; 640 threads per SM at 96 registers
constexpr int kPairChunk = 8;  // pencil pairs per z CTA: 128-byte rows

#define MVD_PAIR_X0(X) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(16)
#define MVD_PAIR_X1(X) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16)
// the column stage next to the real step holds two DFTs at once (8 registers per point)
#define MVD_PAIR_Y0(X) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10)
// rows j and j + 1 are one unit, so the second column radix is even
#define MVD_PAIR_Y1(X) X(2) X(4) X(6) X(8) X(10) X(12) X(16) X(18) X(20)
#define MVD_PAIR_Z(X) X(1) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10)
#define MVD_PAIR_ZC(X) X(1) X(2) X(3) X(4) X(5) X(6) X(8)

// Column unit u of the real step: positions of the columns f (a) and M - f (b) and the root
// exp(-pi i f / M).  f = 0 gives the columns 0 and M: both come from element 0 (load position
// b = 0), and column M has the extra position M.
struct PairUnit {
  short a, b_load, b_store, pad;
  float wx, wy;
};

struct PairShape {
  int ty, tz, m;              // rows, slices, half the row length
  int r0x, r1x, r0y, r1y;
  int az, bz, cz;             // z radices (three stages, bz = 1: two)
  int pc;                     // column pairs: columns 0 .. 2 pc - 1, of which m + 1 are used
  int pitch;                  // row-pair pitch in 16-byte units (odd)
  int nunits;                 // column units
  // tables in global memory: the stage-1 roots W^(j k0) of x and y by position R1 k0 + j and the
  // column units, one block of ntab 16-byte units (tab) that the plane kernels keep in shared
  // memory behind the plane; the roots of the z stages, ntabz units
  const float4* tab;
  int ntab, tab_y, tab_units;  // 16-byte offsets of the y roots and the units
  const float4* tabz;
  int ntabz, tab_c;           // offset of the third stage's roots, which repeat every perz blocks
  int perz;
};

__device__ __forceinline__ void copy_table(float4* dst, const float4* __restrict__ src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}
__device__ __forceinline__ C2 wide(float2 w) { return {pk(w.x, w.x), pk(w.y, w.y)}; }
__device__ __forceinline__ float2 table_root(const float2* __restrict__ p) { return __ldg(p); }
__device__ __forceinline__ C2 ld_c2_early(const float4* p) {  // not moved across other loads
  C2 v;
  asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.r), "=l"(v.i) : "l"(p) : "memory");
  return v;
}

// The three passes are launched so that a pass may start before the one ahead of it in the stream has
// finished (launch_after): each lets the next one start at once, copies its tables, which no pass
// writes, and waits here for the passes ahead to complete before it reads or writes anything else.
// What a pass ahead may have written (psi, q, the tiles' and the kernel's spectra) is read by ordinary
// loads: the read-only path (__ldg, ld.global.nc, const __restrict__ parameters) asks for memory that
// nothing writes while the kernel lives, and its life begins before that wait.  Both measure the same
// (4 views, a first call: 10 iterations of 512x512x256 77.9 ms, 20 of 256x256x192 30.9 ms).
__device__ __forceinline__ void let_next_start() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void wait_for_passes_ahead() { cudaGridDependencySynchronize(); }

// work item b of a plane pass: slice by slice, every tile of a slice before the next slice (the
// halos that neighbouring tiles share are then gathered from L2)
__device__ __forceinline__ void plane_item(int b, int ntiles, int& tile, int& z) {
  z = b / ntiles;
  tile = b - z * ntiles;
}

template <bool INV>
__device__ __forceinline__ C2 twiddle(C2 a, C2 w) {  // w = ((x, x), (y, y)); INV: conjugate
  const f2 x = w.r, y = w.i;
  return INV ? C2{fma2(a.i, y, mul2(a.r, x)), sub2(mul2(a.i, x), mul2(a.r, y))}
             : C2{sub2(mul2(a.r, x), mul2(a.i, y)), fma2(a.i, x, mul2(a.r, y))};
}

// ------------------------------------------------------------------------------------------
// forward plane pass
// ------------------------------------------------------------------------------------------
// Rows of one slice of the gathered volume, extended by its out-of-bounds rule: row(gy), then
// values at col(gx); load2 at an 8-byte aligned position inside the volume.
template <class Gather>
struct PairRows;

template <>
struct PairRows<GatherMirror> {
  const float* slice;
  int nx, ny;
  bool near;  // the tile reaches less than one volume past the border: one reflection
  __device__ __forceinline__ PairRows(const GatherMirror& g, int gz, int ox, int oy, int tx, int ty)
      : slice(g.v.data + (long long)mirror_single(gz, g.v.nz) * g.v.ny * g.v.nx), nx(g.v.nx), ny(g.v.ny) {
    near = ox > -nx && ox + tx < 2 * nx && oy > -ny && oy + ty < 2 * ny;
  }
  __device__ __forceinline__ int reflect(int i, int n) const {
    if (!near) return mirror_single(i, n);
    i = abs(i);
    return min(i, 2 * n - 2 - i);
  }
  __device__ __forceinline__ const float* row(int gy) const { return slice + (long long)reflect(gy, ny) * nx; }
  __device__ __forceinline__ int col(int gx) const { return reflect(gx, nx); }
  __device__ __forceinline__ float load(const float* r, int c) const { return r[c]; }
  __device__ __forceinline__ float2 load2(const float* r, int gx) const {
    return *reinterpret_cast<const float2*>(r + gx);
  }
};

template <>
struct PairRows<GatherValue> {
  const float* slice;
  int nx, x0, x1, y0, y1;
  float value;
  __device__ __forceinline__ PairRows(const GatherValue& g, int gz, int, int, int, int)
      : slice(g.v.data + (long long)gz * g.v.ny * g.v.nx), nx(g.v.nx), x0(g.lo[0]), x1(g.hi[0]), y0(g.lo[1]),
        y1(g.hi[1]), value(g.value) {}
  __device__ __forceinline__ const float* row(int gy) const {
    return gy >= y0 && gy < y1 ? slice + (long long)gy * nx : nullptr;
  }
  __device__ __forceinline__ int col(int gx) const { return gx >= x0 && gx < x1 ? gx : -1; }
  __device__ __forceinline__ float load(const float* r, int c) const { return r && c >= 0 ? r[c] : value; }
  __device__ __forceinline__ float2 load2(const float* r, int gx) const {
    return r ? *reinterpret_cast<const float2*>(r + gx) : make_float2(value, value);
  }
};

template <class Gather>
struct PairGather {
  PairRows<Gather> g;
  int ox, oy;
  int lo, hi;               // the butterflies' elements lo .. hi - 1 lie inside the volume at even positions
};

// x stage 0: rows 2q, 2q + 1 gathered from the volume, butterfly j fastest
template <int R, class Gather>
__device__ __forceinline__ void pair_x0(const PairShape& s, const PairGather<Gather>& p, float4* sm) {
  const int NR = s.r1x, nb = (s.ty >> 1) * NR, T = blockDim.x;
  int q = threadIdx.x / NR, j = threadIdx.x - q * NR;
  const int dq = T / NR, dj = T - dq * NR;
  for (int b = threadIdx.x; b < nb; b += T) {
    const float *ra = p.g.row(p.oy + 2 * q), *rb = p.g.row(p.oy + 2 * q + 1);
    const int gx = p.ox + 2 * j;
    // every load is issued before the first value is used: the branches hold loads only
    float2 a[R], c[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int x = gx + 2 * NR * r;
      if (r >= p.lo && r < p.hi) {
        a[r] = p.g.load2(ra, x);
        c[r] = p.g.load2(rb, x);
      } else {
        const int c0 = p.g.col(x), c1 = p.g.col(x + 1);
        a[r].x = p.g.load(ra, c0);
        c[r].x = p.g.load(rb, c0);
        a[r].y = p.g.load(ra, c1);
        c[r].y = p.g.load(rb, c1);
      }
    }
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = {pk(a[r].x, c[r].x), pk(a[r].y, c[r].y)};
    PDft<R, false>::run(v);
    float4* o = sm + q * s.pitch + j;
#pragma unroll
    for (int r = 0; r < R; ++r) st_c2(o + r * NR, v[r]);
    q += dq;
    j += dj;
    if (j >= NR) {
      j -= NR;
      ++q;
    }
  }
}

// x stage 1 (forward) in place on block k0 of each row pair, row pairs fastest
template <int R, bool INV>
__device__ __forceinline__ void pair_x1(const PairShape& s, float4* sm, int nq, const float2* tw) {
  const int nb = nq * s.r0x, T = blockDim.x;
  int k0 = threadIdx.x / nq, q = threadIdx.x - k0 * nq;
  const int dk = T / nq, dq = T - dk * nq;
  for (int b = threadIdx.x; b < nb; b += T) {
    float4* p = sm + q * s.pitch + k0 * R;
    const float2* w = tw + k0 * R;
    C2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = ld_c2(p + j);
    if (!INV) {
#pragma unroll
      for (int j = 1; j < R; ++j) v[j] = twiddle<false>(v[j], wide(w[j]));
    }
    PDft<R, INV>::run(v);
    if (INV) {
#pragma unroll
      for (int j = 1; j < R; ++j) v[j] = twiddle<true>(v[j], wide(w[j]));
    }
#pragma unroll
    for (int j = 0; j < R; ++j) st_c2(p + j, v[j]);
    k0 += dk;
    q += dq;
    if (q >= nq) {
      q -= nq;
      ++k0;
    }
  }
}

// the real step and y stage 0, in place on one column unit and the row pairs jp + (R1 / 2) r
template <int R>
__device__ __forceinline__ void pair_y0_fwd(const PairShape& s, float4* sm, const int4* units) {
  const int hp = s.r1y >> 1, nb = s.nunits * hp, T = blockDim.x;
  int jp = threadIdx.x / s.nunits, u = threadIdx.x - jp * s.nunits;
  const int dj = T / s.nunits, du = T - dj * s.nunits;
  const int step = hp * s.pitch;
  for (int b = threadIdx.x; b < nb; b += T) {
    const int4 raw = units[u];
    const int a = (short)(raw.x & 0xffff), bl = raw.x >> 16, bs = (short)(raw.y & 0xffff);
    const float wx = __int_as_float(raw.z), wy = __int_as_float(raw.w);
    const f2 x = pk(wx, wx), y = pk(wy, wy), ny = pk(-wy, -wy);
    float4* row = sm + jp * s.pitch;
    C2 va[R], vb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const C2 zk = ld_c2(row + r * step + a), zc = ld_c2(row + r * step + bl);
      const C2 e = {add2(zk.r, zc.r), sub2(zk.i, zc.i)};
      const C2 o = {sub2(zk.r, zc.r), add2(zk.i, zc.i)};
      const C2 wo = mul_root<false>(o, x, y, ny);
      va[r] = {add2(e.r, wo.i), sub2(e.i, wo.r)};
      vb[r] = {sub2(e.r, wo.i), sub2(sub2(0ull, e.i), wo.r)};
    }
    PDft<R, false>::run(va);
    PDft<R, false>::run(vb);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      st_c2(row + r * step + a, va[r]);
      st_c2(row + r * step + bs, vb[r]);
    }
    jp += dj;
    u += du;
    if (u >= s.nunits) {
      u -= s.nunits;
      ++jp;
    }
  }
}

// y stage 1: columns c and c + pc of row block k0, from row pairs to a column pair (the twiddle
// products write the new pairs), straight to the spectrum slice
template <int R>
__device__ __forceinline__ void pair_y1_fwd(const PairShape& s, const float4* sm, float4* __restrict__ out,
                                            const float2* tw) {
  const int nb = s.pc * s.r0y, T = blockDim.x;
  int k0 = threadIdx.x / s.pc, c = threadIdx.x - k0 * s.pc;
  const int dk = T / s.pc, dc = T - dk * s.pc;
  for (int b = threadIdx.x; b < nb; b += T) {
    const float4* p = sm + (k0 * (R / 2)) * s.pitch + c;
    const float2* w = tw + k0 * R;
    C2 v[R];
#pragma unroll
    for (int h = 0; h < R / 2; ++h) {
      const float4 A = p[h * s.pitch], B = p[h * s.pitch + s.pc];
      if (h == 0) {
        v[0] = {pk(A.x, B.x), pk(A.z, B.z)};
      } else {
        const float2 t = w[2 * h];
        v[2 * h] = {pk(A.x * t.x - A.z * t.y, B.x * t.x - B.z * t.y), pk(A.x * t.y + A.z * t.x, B.x * t.y + B.z * t.x)};
      }
      const float2 t = w[2 * h + 1];
      v[2 * h + 1] = {pk(A.y * t.x - A.w * t.y, B.y * t.x - B.w * t.y),
                      pk(A.y * t.y + A.w * t.x, B.y * t.y + B.w * t.x)};
    }
    PDft<R, false>::run(v);
    float4* o = out + (k0 * R) * s.pc + c;
#pragma unroll
    for (int r = 0; r < R; ++r) st_c2(o + r * s.pc, v[r]);
    k0 += dk;
    c += dc;
    if (c >= s.pc) {
      c -= s.pc;
      ++k0;
    }
  }
}

#define MVD_CASE_X0F(R) case R: pair_x0<R>(s, pg, sm); break;
#define MVD_CASE_X1F(R) case R: pair_x1<R, false>(s, sm, s.ty >> 1, twx); break;
#define MVD_CASE_Y0F(R) case R: pair_y0_fwd<R>(s, sm, units); break;
#define MVD_CASE_Y1F(R) case R: pair_y1_fwd<R>(s, sm, out, twy); break;

template <class Gather>
__global__ void __launch_bounds__(kPairThreads, 1)
pair_fwd(const TileDesc* __restrict__ tiles, int ntiles, float4* __restrict__ spec, Gather gather,
         const __grid_constant__ PairShape s) {
  extern __shared__ float4 sm4[];
  float4* const sm = sm4;
  int ti, z;
  plane_item(blockIdx.x, ntiles, ti, z);
  const TileDesc t = tiles[ti];
  float4* out = spec + t.spec_off / 2 + (long long)z * s.ty * s.pc;
  float4* const tab = sm + (s.ty >> 1) * s.pitch;
  const float2* const twx = reinterpret_cast<const float2*>(tab);
  const float2* const twy = reinterpret_cast<const float2*>(tab + s.tab_y);
  const int4* const units = reinterpret_cast<const int4*>(tab + s.tab_units);
  let_next_start();
  copy_table(tab, s.tab, s.ntab);
  wait_for_passes_ahead();
  // a slice of one value: the extension outside the data box, and the slices past the last one
  // that the effective region reaches (any finite value serves there)
  float cval = 0.f;
  const bool past = z >= 2 * t.hz + t.ez;
  if (past || gather.constant_slice(t.oz + z, cval)) {
    if (past) cval = 0.f;
    const float dc = 4.f * cval * (float)s.m * (float)s.ty;  // 2 x sum of 2 m x ty values
    for (int i = threadIdx.x; i < s.ty * s.pc; i += blockDim.x) out[i] = make_float4(i == 0 ? dc : 0.f, 0.f, 0.f, 0.f);
    return;
  }
  {
    PairGather<Gather> pg{PairRows<Gather>(gather, t.oz + z, t.ox, t.oy, 2 * s.m, s.ty)};
    pg.ox = t.ox;
    pg.oy = t.oy;
    int x0, x1, y0, y1;
    gather.region(x0, x1, y0, y1);
    // element r of the butterflies covers x = ox + 2 r1x r .. + 2 r1x - 1
    const int w = 2 * s.r1x;
    pg.lo = max(0, (x0 - t.ox + w - 1) / w);
    pg.hi = (x1 - t.ox) / w;
    if (((t.ox | gather.v.nx) & 1) || (reinterpret_cast<uintptr_t>(gather.v.data) & 7)) pg.hi = 0;  // 4-byte loads
    switch (s.r0x) { MVD_PAIR_X0(MVD_CASE_X0F) }
  }
  __syncthreads();
  switch (s.r1x) { MVD_PAIR_X1(MVD_CASE_X1F) }
  __syncthreads();
  switch (s.r0y) { MVD_PAIR_Y0(MVD_CASE_Y0F) }
  __syncthreads();
  switch (s.r1y) { MVD_PAIR_Y1(MVD_CASE_Y1F) }
}

// ------------------------------------------------------------------------------------------
// inverse plane pass
// ------------------------------------------------------------------------------------------
// y stage 1 inverse: a column pair of the spectrum slice to row pairs of columns c and c + pc
template <int R>
__device__ __forceinline__ void pair_y1_inv(const PairShape& s, const float4* in, float4* sm) {
  const int nb = s.pc * s.r0y, T = blockDim.x;
  int k0 = threadIdx.x / s.pc, c = threadIdx.x - k0 * s.pc;
  const int dk = T / s.pc, dc = T - dk * s.pc;
  for (int b = threadIdx.x; b < nb; b += T) {
    const float4* p = in + (k0 * R) * s.pc + c;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_c2(p + r * s.pc);
    PDft<R, true>::run(v);
    const float2* w = reinterpret_cast<const float2*>(s.tab + s.tab_y) + k0 * R;
    float4* o = sm + (k0 * (R / 2)) * s.pitch + c;
#pragma unroll
    for (int h = 0; h < R / 2; ++h) {
      float ar, br, ai, bi, cr, dr, ci, di;
      unpk(v[2 * h].r, ar, br);
      unpk(v[2 * h].i, ai, bi);
      unpk(v[2 * h + 1].r, cr, dr);
      unpk(v[2 * h + 1].i, ci, di);
      const float2 t = table_root(w + 2 * h + 1);
      float4 A, B;
      if (h == 0) {
        A.x = ar;
        A.z = ai;
        B.x = br;
        B.z = bi;
      } else {
        const float2 t0 = table_root(w + 2 * h);
        A.x = ar * t0.x + ai * t0.y;
        A.z = ai * t0.x - ar * t0.y;
        B.x = br * t0.x + bi * t0.y;
        B.z = bi * t0.x - br * t0.y;
      }
      A.y = cr * t.x + ci * t.y;
      A.w = ci * t.x - cr * t.y;
      B.y = dr * t.x + di * t.y;
      B.w = di * t.x - dr * t.y;
      o[h * s.pitch] = A;
      o[h * s.pitch + s.pc] = B;
    }
    k0 += dk;
    c += dc;
    if (c >= s.pc) {
      c -= s.pc;
      ++k0;
    }
  }
}

// y stage 0 inverse and the step back to the packed transforms of real rows, of the row pairs
// [q0, q1) that hold effective rows
template <int R>
__device__ __forceinline__ void pair_y0_inv(const PairShape& s, float4* sm, int q0, int q1, const int4* units) {
  const int hp = s.r1y >> 1, nb = s.nunits * hp, T = blockDim.x;
  int jp = threadIdx.x / s.nunits, u = threadIdx.x - jp * s.nunits;
  const int dj = T / s.nunits, du = T - dj * s.nunits;
  const int step = hp * s.pitch;
  for (int b = threadIdx.x; b < nb; b += T) {
    const int4 raw = units[u];
    const int a = (short)(raw.x & 0xffff), bs = (short)(raw.y & 0xffff);
    const float wx = __int_as_float(raw.z), wy = __int_as_float(raw.w);
    const f2 x = pk(wx, wx), y = pk(wy, wy), ny = pk(-wy, -wy);
    float4* row = sm + jp * s.pitch;
    C2 va[R], vb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      va[r] = ld_c2(row + r * step + a);
      vb[r] = ld_c2(row + r * step + bs);
    }
    PDft<R, true>::run(va);
    PDft<R, true>::run(vb);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = jp + hp * r;
      if (q >= q0 && q < q1) {
        const C2 e = {add2(va[r].r, vb[r].r), sub2(va[r].i, vb[r].i)};
        const C2 o = {sub2(va[r].r, vb[r].r), add2(va[r].i, vb[r].i)};
        const C2 wo = mul_root<true>(o, x, y, ny);
        st_c2(row + r * step + bs, {add2(e.r, wo.i), sub2(wo.r, e.i)});
        st_c2(row + r * step + a, {sub2(e.r, wo.i), add2(e.i, wo.r)});
      }
    }
    jp += dj;
    u += du;
    if (u >= s.nunits) {
      u -= s.nunits;
      ++jp;
    }
  }
}

// x stage 0 inverse, in place: the real rows x[2n], x[2n + 1] of element n in natural order
template <int R>
__device__ __forceinline__ void pair_x0_inv(const PairShape& s, float4* sm, int nq) {
  const int NR = s.r1x, nb = nq * NR, T = blockDim.x;
  int j = threadIdx.x / nq, q = threadIdx.x - j * nq;
  const int dj = T / nq, dq = T - dj * nq;
  for (int b = threadIdx.x; b < nb; b += T) {
    float4* p = sm + q * s.pitch + j;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_c2(p + r * NR);
    PDft<R, true>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st_c2(p + r * NR, v[r]);
    j += dj;
    q += dq;
    if (q >= nq) {
      q -= nq;
      ++j;
    }
  }
}

#define MVD_CASE_Y1I(R) case R: pair_y1_inv<R>(s, in, sm); break;
#define MVD_CASE_Y0I(R) case R: pair_y0_inv<R>(s, sm, q0, q1, units); break;
#define MVD_CASE_X1I(R) case R: pair_x1<R, true>(s, rows, q1 - q0, twx); break;
#define MVD_CASE_X0I(R) case R: pair_x0_inv<R>(s, rows, q1 - q0); break;

// Epilogue positions: groups of 4 voxels along x (16-byte aligned in the volume where its rows
// are) of the effective row pairs, numbered row pair by row pair, taken blockDim.x apart by a
// thread.  So every lane has work whatever the row length, and offsets advance by additions:
// `off` of the group's first voxel from the first row pair's (rows 2q and 2q + 1 at off and
// off + nx), `at` into the plane buffer.
struct PairWalk {
  int i, q, off, at;         // of this thread's next group: group of the row, row pair
  int di, dq, doff, dat;     // per step
  int per, woff, wat;        // groups of a row; corrections when i passes it
  __device__ __forceinline__ void init(int per_, int nx, int pitch2) {
    per = per_;
    q = threadIdx.x / per;
    i = threadIdx.x - q * per;
    off = q * 2 * nx + 4 * i;
    at = q * pitch2 + 4 * i;
    dq = blockDim.x / per;
    di = blockDim.x - dq * per;
    doff = dq * 2 * nx + 4 * di;
    dat = dq * pitch2 + 4 * di;
    woff = 2 * nx - 4 * per;
    wat = pitch2 - 4 * per;
  }
  __device__ __forceinline__ void next() {
    i += di;
    q += dq;
    off += doff;
    at += dat;
    if (i >= per) {
      i -= per;
      ++q;
      off += woff;
      at += wat;
    }
  }
};

// One group of both rows: its inputs are loaded a step ahead of their use.  Voxels outside the
// effective region (mask bits clear; bits 0-3 the first row, 4-7 the second) read nothing and are
// not stored.
template <class Epi>
struct PairEpi {
  int off, at, mask;
  float4 a[2], b[2];

  __device__ __forceinline__ static float4 load4(const float* p, int m, bool vec) {
    if (vec && m == 15) return *reinterpret_cast<const float4*>(p);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (m & 1) v.x = p[0];
    if (m & 2) v.y = p[1];
    if (m & 4) v.z = p[2];
    if (m & 8) v.w = p[3];
    return v;
  }
  __device__ __forceinline__ void load(const float* s0, const float* s1, int nx, PairWalk& w, int nq, int skip, int ex,
                                       bool first_ok, bool last_ok, bool vec) {
    off = w.off;
    at = w.at;
    const int x = 4 * w.i - skip;  // effective x of the group's first voxel
    int m = 15;
    if (x < 0) m &= 15 << (-x);
    if (x + 4 > ex) m &= 15 >> (x + 4 - ex);
    mask = 0;
    if (w.q < nq) mask = (w.q > 0 || first_ok ? m : 0) | (w.q < nq - 1 || last_ok ? m << 4 : 0);
    if (Epi::kIn > 0) {
      a[0] = load4(s0 + off, mask & 15, vec);
      a[1] = load4(s0 + off + nx, mask >> 4, vec);
    }
    if (Epi::kIn > 1) {
      b[0] = load4(s1 + off, mask & 15, vec);
      b[1] = load4(s1 + off + nx, mask >> 4, vec);
    }
    w.next();
  }
  __device__ __forceinline__ void store(Epi& e, float* d, int nx, const float2* rows, bool vec) {
    if (!mask) return;
    const float2 f0 = rows[at], f1 = rows[at + 1], f2 = rows[at + 2], f3 = rows[at + 3];
    const float4 v0 = make_float4(e.value(f0.x, a[0].x, b[0].x), e.value(f1.x, a[0].y, b[0].y),
                                  e.value(f2.x, a[0].z, b[0].z), e.value(f3.x, a[0].w, b[0].w));
    const float4 v1 = make_float4(e.value(f0.y, a[1].x, b[1].x), e.value(f1.y, a[1].y, b[1].y),
                                  e.value(f2.y, a[1].z, b[1].z), e.value(f3.y, a[1].w, b[1].w));
    if (d) {
      put4(d + off, v0, mask & 15, vec);
      put4(d + off + nx, v1, mask >> 4, vec);
    }
  }
  __device__ __forceinline__ static void put4(float* p, float4 v, int m, bool vec) {
    if (vec && m == 15) {
      *reinterpret_cast<float4*>(p) = v;
      return;
    }
    if (m & 1) p[0] = v.x;
    if (m & 2) p[1] = v.y;
    if (m & 4) p[2] = v.z;
    if (m & 8) p[3] = v.w;
  }
};

// Items: slices [hz, hz + ez of the first tile) of every tile; a tile clipped along z has fewer.
template <class Epi>
__global__ void __launch_bounds__(kPairThreads, 1)
pair_inv(const TileDesc* __restrict__ tiles, int ntiles, const float4* spec, Epi epi,
         const __grid_constant__ PairShape s) {
  extern __shared__ float4 sm4[];
  float4* const sm = sm4;
  int ti, z;
  plane_item(blockIdx.x, ntiles, ti, z);
  const TileDesc t = tiles[ti];
  float4* const tab = sm + (s.ty >> 1) * s.pitch;
  epi.acc_init();
  let_next_start();
  if (z < t.ez) copy_table(tab, s.tab, s.ntab);
  wait_for_passes_ahead();
  if (z < t.ez) {
    z += t.hz;
    const float4* in = spec + t.spec_off / 2 + (long long)z * s.ty * s.pc;
    const int q0 = t.hy >> 1, q1 = (t.hy + t.ey + 1) >> 1;
    float4* rows = sm + q0 * s.pitch;
    const float2* const twx = reinterpret_cast<const float2*>(tab);
    const int4* const units = reinterpret_cast<const int4*>(tab + s.tab_units);
    switch (s.r1y) { MVD_PAIR_Y1(MVD_CASE_Y1I) }
    __syncthreads();
    switch (s.r0y) { MVD_PAIR_Y0(MVD_CASE_Y0I) }
    __syncthreads();
    switch (s.r1x) { MVD_PAIR_X1(MVD_CASE_X1I) }
    __syncthreads();
    switch (s.r0x) { MVD_PAIR_X0(MVD_CASE_X0I) }
    // The epilogue.  A group's inputs are loaded while the one before is computed and stored, the
    // first one's before the last barrier.
    const int nq = q1 - q0, nx = epi.nx;
    const bool first_ok = !(t.hy & 1), last_ok = !((t.hy + t.ey) & 1);
    const int lead = (nx & 3) ? 0 : (t.ox + t.hx) & 3;
    const int skip = lead <= t.hx ? lead : 0;  // the plane buffer holds hx values before the first voxel
    const long long g0 = ((long long)(t.oz + z) * epi.ny + (t.oy + 2 * q0)) * (long long)nx + t.ox + t.hx - skip;
    const float* s0 = Epi::kIn > 0 ? epi.src0() + g0 : nullptr;
    const float* s1 = Epi::kIn > 1 ? epi.src1() + g0 : nullptr;
    float* d = epi.dst() ? epi.dst() + g0 : nullptr;
    const bool vec = !(nx & 3) && skip == lead && !((reinterpret_cast<uintptr_t>(s0) | reinterpret_cast<uintptr_t>(s1) |
                                     reinterpret_cast<uintptr_t>(d)) & 15);
    const float2* frows = reinterpret_cast<const float2*>(rows) + t.hx - skip;
    const int per = (t.ex + skip + 3) >> 2, total = nq * per;
    PairWalk w;
    w.init(per, nx, 2 * s.pitch);
    PairEpi<Epi> cur, next;
    cur.load(s0, s1, nx, w, nq, skip, t.ex, first_ok, last_ok, vec);
    __syncthreads();
    for (int f = threadIdx.x; f < total; f += blockDim.x) {
      next.load(s0, s1, nx, w, nq, skip, t.ex, first_ok, last_ok, vec);
      cur.store(epi, d, nx, frows, vec);
      cur = next;
    }
  }
  epi.finish();
}

// ------------------------------------------------------------------------------------------
// z pass: kPairChunk pencil pairs per CTA.  A CTA's stages wait on one another, so what keeps the SM busy
// is the number of CTAs that share it: 8 pairs and 64 to 160 threads (4 to 10 CTAs) against 16 pairs and
// 320 threads (2) took 260 / 281 us at 512x512x256 (4 views), 50.8 / 58.0 at 256x256x192, 11.8 / 15.1 at
// 203x157x91.
// ------------------------------------------------------------------------------------------
// Lengths are A x B x C (B = 1: two stages) with radices of at most 10 (C: 8).  The middle stage C holds
// its points and the kernel spectrum's values of the same positions, which are loaded before the
// transform, so their latency passes under it: with a 16-point middle stage (320 = 20 x 16) the
// registers held half of them, and waiting for the other half took 14 of the pass's 31 thousand
// cycles per chunk.
// CONV: forward, times the kernel spectrum, inverse (effective slices stored); else forward, scaled
// (kernel spectra).
template <int R>
__device__ __forceinline__ void pair_za_fwd(const PairShape& s, const float4* g, int plane, int count,
                                            float4* sm) {
  const int NR = s.bz * s.cz, nb = NR * kPairChunk;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int j = b / kPairChunk, i = b % kPairChunk;
    if (i >= count) continue;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_c2(g + (j + NR * r) * plane + i);
    PDft<R, false>::run(v);
    float4* o = sm + j * kPairChunk + i;
#pragma unroll
    for (int r = 0; r < R; ++r) st_c2(o + r * NR * kPairChunk, v[r]);
  }
}

// the second stage in place: points j + C r of block k0 (B C elements), roots by position
template <int R, bool INV>
__device__ __forceinline__ void pair_zb(const PairShape& s, float4* sm, const float2* tw) {
  const int C = s.cz, nb = s.az * C * kPairChunk;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int kj = b / kPairChunk, i = b % kPairChunk;
    const int k0 = kj / C, p0 = k0 * (R * C) + kj - k0 * C;
    float4* p = sm + p0 * kPairChunk + i;
    const float2* w = tw + p0;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_c2(p + r * C * kPairChunk);
    if (!INV) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = twiddle<false>(v[r], wide(w[r * C]));
    }
    PDft<R, INV>::run(v);
    if (INV) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = twiddle<true>(v[r], wide(w[r * C]));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) st_c2(p + r * C * kPairChunk, v[r]);
  }
}

template <int R, bool CONV>
__device__ __forceinline__ void pair_zc(const PairShape& s, float4* __restrict__ g, const float4* otf,
                                        int plane, int count, float4* sm, float scale, const float2* tw) {
  const int nb = s.az * s.bz * kPairChunk, i = threadIdx.x % kPairChunk;
  C2 o[R];
  auto load = [&](int b) {
    if (CONV && b < nb && i < count) {
#pragma unroll
      for (int m = 0; m < R; ++m) o[m] = ld_c2_early(otf + ((b / kPairChunk) * R + m) * plane + i);
    }
  };
  int b = threadIdx.x;
  load(b);
  __syncthreads();  // the stage before (or the tables) is complete; the loads are in flight meanwhile
  for (; b < nb; b += blockDim.x, load(b)) {
    if (i >= count) continue;
    const int kb = b / kPairChunk;
    float4* p = sm + (kb * R) * kPairChunk + i;
    const float2* w = tw + (kb % s.perz) * R;
    C2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = ld_c2(p + j * kPairChunk);
#pragma unroll
    for (int j = 1; j < R; ++j) v[j] = twiddle<false>(v[j], wide(w[j]));
    PDft<R, false>::run(v);
    if constexpr (!CONV) {
      const f2 sc = pk(scale, scale);
#pragma unroll
      for (int m = 0; m < R; ++m) st_c2(g + (kb * R + m) * plane + i, {mul2(v[m].r, sc), mul2(v[m].i, sc)});
    } else {
#pragma unroll
      for (int m = 0; m < R; ++m) v[m] = mul_c2(v[m], o[m]);
      PDft<R, true>::run(v);
#pragma unroll
      for (int j = 1; j < R; ++j) v[j] = twiddle<true>(v[j], wide(w[j]));
#pragma unroll
      for (int j = 0; j < R; ++j) st_c2(p + j * kPairChunk, v[j]);
    }
  }
}

template <int R>
__device__ __forceinline__ void pair_za_inv(const PairShape& s, float4* __restrict__ g, int plane, int count,
                                            const float4* sm, int z0, int z1) {
  const int NR = s.bz * s.cz, nb = NR * kPairChunk;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int j = b / kPairChunk, i = b % kPairChunk;
    if (i >= count) continue;
    const float4* p = sm + j * kPairChunk + i;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_c2(p + r * NR * kPairChunk);
    PDft<R, true>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int z = j + NR * r;
      if (z >= z0 && z < z1) st_c2(g + z * plane + i, v[r]);
    }
  }
}

#define MVD_CASE_ZAF(R) case R: pair_za_fwd<R>(s, g, plane, count, sm); break;
#define MVD_CASE_ZBF(R) case R: pair_zb<R, false>(s, sm, tw); break;
#define MVD_CASE_ZC(R) case R: pair_zc<R, CONV>(s, g, otf, plane, count, sm, scale, twc); break;
#define MVD_CASE_ZBI(R) case R: pair_zb<R, true>(s, sm, tw); break;
#define MVD_CASE_ZAI(R) case R: pair_za_inv<R>(s, g, plane, count, sm, t.hz, t.hz + t.ez); break;

// Item b: blocks of `block` chunks, each swept over every tile before the next, so that a block's
// kernel spectrum is read from L2 by every tile but the first.
template <bool CONV>
__global__ void __launch_bounds__(kPairZThreads, 4)
pair_z(const TileDesc* __restrict__ tiles, int ntiles, float4* __restrict__ spec, const float4* otf,
       const __grid_constant__ PairShape s, int nchunks, int block, float scale) {
  extern __shared__ float4 sm4[];
  float4* const sm = sm4;
  const int plane = s.ty * s.pc;
  const int g0 = blockIdx.x / (ntiles * block);
  const int len = min(block, nchunks - g0 * block);  // chunks of this block
  const int rest = blockIdx.x - g0 * (ntiles * block);
  const int ti = rest / len;
  const int p0 = (g0 * block + rest - ti * len) * kPairChunk;
  const TileDesc t = tiles[ti];
  const int count = min(kPairChunk, plane - p0);
  float4* g = spec + t.spec_off / 2 + p0;
  if (CONV) otf += p0;
  // roots of the second stage by position, then of the third (the same table when B = 1)
  const float2* const tw = reinterpret_cast<const float2*>(sm + s.tz * kPairChunk);
  const float2* const twc = reinterpret_cast<const float2*>(sm + s.tz * kPairChunk + s.tab_c);
  let_next_start();
  copy_table(sm + s.tz * kPairChunk, s.tabz, s.ntabz);
  wait_for_passes_ahead();
  switch (s.az) { MVD_PAIR_Z(MVD_CASE_ZAF) }
  if (s.bz > 1) {
    __syncthreads();
    switch (s.bz) { MVD_PAIR_Z(MVD_CASE_ZBF) }
  }
  switch (s.cz) { MVD_PAIR_ZC(MVD_CASE_ZC) }
  if (!CONV) return;
  __syncthreads();
  if (s.bz > 1) {
    switch (s.bz) { MVD_PAIR_Z(MVD_CASE_ZBI) }
    __syncthreads();
  }
  switch (s.az) { MVD_PAIR_Z(MVD_CASE_ZAI) }
}

}  // namespace mvd
