// Host engine of the tiled FFT convolution: plans, tile planner, OTF preparation, launches,
// and the small elementwise / reduction kernels of the deconvolution path.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>
#include <sstream>

#include "engine.h"

namespace mvd {

static std::atomic<long long> g_launches{0};
long long launch_count() { return g_launches.load(); }
void count_launch(int n) { g_launches += n; }

void check_cuda(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    std::string msg = std::string(what) + ": " + cudaGetErrorString(e);
    throw CudaError(e, msg);
  }
}

namespace {
thread_local AllocScope* tls_scope = nullptr;
}

AllocScope::AllocScope(cudaStream_t s) : stream_(s), prev_(tls_scope) { tls_scope = this; }
AllocScope::~AllocScope() {
  tls_scope = prev_;
  if (!tables_.empty()) cudaStreamSynchronize(stream_);  // idle already but on the way out of an error
}
void AllocScope::upload(void* dst, const void* src, size_t bytes) {
  const char* p = static_cast<const char*>(src);
  tables_.emplace_back(p, p + bytes);
  MVD_CHECK(cudaMemcpyAsync(dst, tables_.back().data(), bytes, cudaMemcpyHostToDevice, stream_));
}
cudaStream_t alloc_stream() { return tls_scope ? tls_scope->stream() : nullptr; }

void upload_table(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (tls_scope)
    tls_scope->upload(dst, src, bytes);
  else
    MVD_CHECK(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
}

bool async_copy_source(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged || a.type == cudaMemoryTypeHost;
}

void keep_pool_memory(int dev) {
  static std::mutex mu;
  static std::vector<bool> done;
  std::lock_guard<std::mutex> lock(mu);
  if ((int)done.size() <= dev) done.resize(dev + 1, false);
  if (done[dev]) return;
  cudaMemPool_t pool;
  MVD_CHECK(cudaDeviceGetDefaultMemPool(&pool, dev));
  uint64_t threshold = UINT64_MAX;
  MVD_CHECK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold));
  done[dev] = true;
}

namespace {
cudaMemPool_t call_pool(int dev) {
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool;
  MVD_CHECK(cudaMemPoolCreate(&pool, &props));
  uint64_t keep = 64ull << 20;
  const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  if (e != cudaSuccess) cudaMemPoolDestroy(pool);
  MVD_CHECK(e);
  return pools[dev] = pool;
}
}  // namespace

CallBuf::CallBuf(int dev, size_t bytes, cudaStream_t s) : s_(s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  MVD_CHECK(cudaStreamIsCapturing(s, &st));
  if (st == cudaStreamCaptureStatusNone)
    MVD_CHECK(cudaMallocFromPoolAsync(&p_, bytes, call_pool(dev), s));
  else
    MVD_CHECK(cudaMallocAsync(&p_, bytes, s));
}
CallBuf::~CallBuf() {
  if (p_) cudaFreeAsync(p_, s_);
}

void DevBuf::release() {
  if (p) {
    if (stream)
      cudaFreeAsync(p, stream);
    else
      cudaFree(p);
  }
  p = nullptr;
  bytes = 0;
  stream = nullptr;
}
DevBuf::~DevBuf() { release(); }
DevBuf& DevBuf::operator=(DevBuf&& o) noexcept {
  if (this != &o) {
    release();
    p = o.p;
    bytes = o.bytes;
    stream = o.stream;
    o.p = nullptr;
    o.bytes = 0;
    o.stream = nullptr;
  }
  return *this;
}
void DevBuf::alloc(size_t b) {
  release();
  if (b == 0) return;
  if (const cudaStream_t s = alloc_stream()) {
    MVD_CHECK(cudaMallocAsync(&p, b, s));
    stream = s;
  } else {
    MVD_CHECK(cudaMalloc(&p, b));
  }
  bytes = b;
}
void DevBuf::ensure(size_t b) {
  if (b > bytes) alloc(b);
}

bool is_smooth(int n) {
  if (n <= 0) return false;
  for (int f : {2, 3, 5})
    while (n % f == 0) n /= f;
  return n == 1;
}

int next_smooth(int n, bool even) {
  if (n < 2) n = 2;
  for (int m = n;; ++m) {
    if (even && (m & 1)) continue;
    if (is_smooth(m)) return m;
  }
}

// Radices of the register DFTs (fft_device.cuh).
static const int kRadices[] = {20, 18, 16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};

static void best_split(int n, int depth, int maxdepth, std::vector<int>& cur, std::vector<int>& best) {
  if (n == 1) {
    // fewest stages first, then the most balanced (largest smallest radix)
    auto mn = [](const std::vector<int>& v) { return v.empty() ? 0 : *std::min_element(v.begin(), v.end()); };
    if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && mn(cur) > mn(best))) best = cur;
    return;
  }
  if (depth == maxdepth) return;
  for (int r : kRadices) {
    if (n % r) continue;
    if (!cur.empty() && r > cur.back()) continue;  // non-increasing order
    cur.push_back(r);
    best_split(n / r, depth + 1, maxdepth, cur, best);
    cur.pop_back();
  }
}

std::vector<int> factorize(int n) {
  if (n == 1) return {1};
  std::vector<int> cur, best;
  for (int depth = 1; depth <= kMaxStages && best.empty(); ++depth) best_split(n, 0, depth, cur, best);
  if (best.empty()) throw std::invalid_argument("FFT length is not 2,3,5-smooth");
  return best;
}

// ------------------------------------------------------------------------------------------
// plan table
// ------------------------------------------------------------------------------------------
int PlanTable::index_of(int n, bool ascending) {
  const int key = ascending ? -n : n;
  auto it = by_len_.find(key);
  if (it != by_len_.end()) return it->second;
  if (n < 1) throw std::invalid_argument("bad FFT length");
  if ((int)host_.size() >= kCapacity) throw std::runtime_error("FFT plan table full");
  FftPlan p{};
  p.n = n;
  std::vector<int> rad = factorize(n);
  if (ascending) std::reverse(rad.begin(), rad.end());
  if ((int)rad.size() > kMaxStages) throw std::invalid_argument("too many FFT stages");
  p.nstages = (int)rad.size();
  for (size_t i = 0; i < rad.size(); ++i) p.radix[i] = rad[i];
  // twiddles: [0, n) for the complex length n, then [0, n] for the real length 2n
  std::vector<float2> tw(2 * n + 1);
  for (int k = 0; k < n; ++k) {
    const double a = -2.0 * M_PI * (double)k / (double)n;
    tw[k] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  for (int k = 0; k <= n; ++k) {
    const double a = -M_PI * (double)k / (double)n;
    tw[n + k] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  auto buf = std::make_unique<DevBuf>(tw.size() * sizeof(float2));
  upload_table(buf->p, tw.data(), tw.size() * sizeof(float2));
  p.tw = buf->as<float2>();
  p.tw_r2c = buf->as<float2>() + n;
  tw_bufs_.push_back(std::move(buf));
  const int idx = (int)host_.size();
  host_.push_back(p);
  by_len_[key] = idx;
  dirty_ = true;
  return idx;
}

const FftPlan* PlanTable::device() {
  if (!dev_.p) dev_.alloc(kCapacity * sizeof(FftPlan));
  if (dirty_) {
    // append-only table at a fixed address: entries already in use never change, so kernels
    // (and captured graphs) holding this pointer stay valid while new lengths are added
    upload_table(dev_.p, host_.data(), host_.size() * sizeof(FftPlan));
    dirty_ = false;
  }
  return dev_.as<FftPlan>();
}

// ------------------------------------------------------------------------------------------
// tile planner
// ------------------------------------------------------------------------------------------
static std::vector<AxisTiles> axis_options(int size, int k, bool even, int tmax) {
  std::vector<AxisTiles> out;
  int last_T = -1;
  const int nmax = std::max(1, size);
  for (int n = 1; n <= nmax && n <= 64; ++n) {
    const int need = (size + n - 1) / n + k - 1;
    int T = next_smooth(std::max(need, k), even);
    if (T > tmax) continue;
    if (T == last_T) continue;
    last_T = T;
    AxisTiles a;
    a.size = size;
    a.k = k;
    a.T = T;
    a.E = T - k + 1;
    a.n = (size + a.E - 1) / a.E;
    out.push_back(a);
    if (a.E < 8 && a.E < size) break;  // smaller tiles would be nearly all halo
  }
  return out;
}

// Work items of the three passes.  Plane passes: slice by slice, every tile of a slice before
// the next slice.  The forward pass then reads the halo a tile shares with its neighbours (30
// columns or rows of the 512x512x256 workload's 160-wide tiles) from L2 while the neighbours
// gather it, and the inverse pass's epilogue reads and writes each volume row, which the tiles
// of a slice split between them, within a short time (512x512x256 workload, per iteration:
// forward passes 2.91 against 2.99 ms, inverse passes 3.46 against 3.62 ms tile by tile).
// z pass: blocks
// of kZBlock consecutive pencil chunks, each block swept over every tile before the next.  All
// tiles of a plan share one kernel spectrum (the OTF), so a block's OTF chunks stay in L2 while
// every tile reads them, and each tile's reads stay contiguous over the block.  (Tile by tile,
// a view's OTF of up to 33 MB was re-read from DRAM for every tile; chunk by chunk across tiles,
// consecutive CTAs read 16 tiles' scattered chunks and the z pass got slower: 3.62 ms against
// 3.43 ms per iteration on the 512x512x256 workload.)
constexpr int kZBlock = 32;
static void fill_items(ConvPlan& p) {
  p.items_fwd.clear();
  p.items_inv.clear();
  p.items_z.clear();
  int plane_max = 0, tz_max = 0;
  for (int i = 0; i < (int)p.tiles.size(); ++i) {
    plane_max = std::max(plane_max, p.tiles[i].ty * p.tiles[i].px);
    tz_max = std::max(tz_max, p.tiles[i].tz);
  }
  for (int z = 0; z < tz_max; ++z)
    for (int i = 0; i < (int)p.tiles.size(); ++i) {
      const TileDesc& t = p.tiles[i];
      if (z >= t.hz && z < t.hz + t.ez) p.items_inv.push_back(make_int2(i, z));
    }
  for (int z = 0; z < tz_max; ++z)
    for (int i = 0; i < (int)p.tiles.size(); ++i)
      if (z < p.tiles[i].tz) p.items_fwd.push_back(make_int2(i, z));
  auto zitems = [&](std::vector<int2>& out, int chunk) {
    out.clear();
    for (int b0 = 0; b0 < plane_max; b0 += kZBlock * kZChunk)
      for (int i = 0; i < (int)p.tiles.size(); ++i) {
        const int plane = p.tiles[i].ty * p.tiles[i].px;
        for (int p0 = b0; p0 < std::min(plane, b0 + kZBlock * kZChunk); p0 += chunk)
          out.push_back(make_int2(i, p0));
      }
  };
  zitems(p.items_z, kZChunk);
  zitems(p.items_zw, kZWideChunk);
}

void ConvPlan::upload() {
  if (paired) return upload_pair();
  d_tiles.alloc(tiles.size() * sizeof(TileDesc));
  upload_table(d_tiles.p, tiles.data(), tiles.size() * sizeof(TileDesc));
  auto up = [](DevBuf& b, const std::vector<int2>& v) {
    b.alloc(std::max<size_t>(1, v.size()) * sizeof(int2));
    if (!v.empty()) upload_table(b.p, v.data(), v.size() * sizeof(int2));
  };
  up(d_items_fwd, items_fwd);
  up(d_items_inv, items_inv);
  up(d_items_z, items_z);
  up(d_items_zw, items_zw);
  // OTF build tables: one tile of this shape covering [0, T) with its full region effective
  if (!tiles.empty()) {
    TileDesc t = tiles[0];
    t.ox = t.oy = t.oz = 0;
    t.hx = t.hy = t.hz = 0;
    t.ex = t.tx; t.ey = t.ty; t.ez = t.tz;
    t.spec_off = 0;
    t.otf_off = 0;
    std::vector<int2> fwd, zz;
    for (int z = 0; z < t.tz; ++z) fwd.push_back(make_int2(0, z));
    for (int p0 = 0; p0 < t.ty * t.px; p0 += kZChunk) zz.push_back(make_int2(0, p0));
    d_otf_tile.alloc(sizeof(TileDesc));
    upload_table(d_otf_tile.p, &t, sizeof(TileDesc));
    up(d_otf_fwd, fwd);
    up(d_otf_z, zz);
    n_otf_fwd = (int)fwd.size();
    n_otf_z = (int)zz.size();
  }
}

// Shared-memory budget of one plane buffer used by the planner (MVD_PLANE_CAP overrides it;
// planes of at most half the budget let two CTAs share an SM).
int plane_cap() {
  static int cap = [] {
    const char* e = std::getenv("MVD_PLANE_CAP");
    int v = e ? std::atoi(e) : 0;
    return (v >= 256 && v <= kPlaneCap) ? v : kPlaneCapDefault;
  }();
  return cap;
}

static bool plane_cap_from_env() {
  const char* e = std::getenv("MVD_PLANE_CAP");
  const int v = e ? std::atoi(e) : 0;
  return v >= 256 && v <= kPlaneCap;
}

int plane_limit() { return plane_cap_from_env() ? plane_cap() : kPlaneCap; }

double plane_cost_factor(int tx, int ty, long long plane) {
  if (plane_cap_from_env()) return 1.0;
  const bool two_per_sm = plane <= kPlaneCapDefault || (use_staged_planes() && staged_plane_shape(tx, ty));
  double f = two_per_sm ? 1.0 : 1.12;
  if (!compiled_plane_shape(tx, ty)) f *= 1.3;
  return f;
}

int plane_threads() {
  static int t = [] {
    const char* e = std::getenv("MVD_PLANE_THREADS");
    int v = e ? std::atoi(e) : 0;
    return (v >= 64 && v <= kThreads && v % 32 == 0) ? v : kThreads;
  }();
  return t;
}

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to the driver library)
EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return static_cast<EncodeTiled>(nullptr);
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

}  // namespace

// Tensor map of a float volume [nz][ny][nx] with a (w, h, 1) box; false when the volume does not
// meet the copy's rules (16-byte aligned base and row stride) or the driver refuses it.
bool volume_box_map(const float* base, int nx, int ny, int nz, int w, int h, CUtensorMap* out) {
  static std::mutex mu;
  static std::map<std::tuple<const float*, int, int, int, int, int>, CUtensorMap> cache;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (nx % 4) || w > 256 || h > 256) return false;
  const auto key = std::make_tuple(base, nx, ny, nz, w, h);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return true;
  }
  EncodeTiled enc = encode_tiled();
  if (!enc) return false;
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  const cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[2] = {(cuuint64_t)nx * sizeof(float), (cuuint64_t)nx * ny * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)w, (cuuint32_t)h, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  if (enc(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (cache.size() >= 4096) cache.clear();  // maps are cheap to encode again; bound the memory
  cache[key] = m;
  *out = m;
  return true;
}


bool use_l2_prefetch() {
  static bool on = [] {
    const char* e = std::getenv("MVD_L2_PREFETCH");
    return !(e && e[0] == '0');
  }();
  return on;
}

bool use_staged_planes() {
  static bool on = [] {
    const char* e = std::getenv("MVD_STAGED_PLANES");
    return !(e && e[0] == '0');
  }();
  return on;
}

bool use_fixed_planes() {
  static bool on = [] {
    const char* e = std::getenv("MVD_FIXED_PLANES");
    return !(e && e[0] == '0');
  }();
  return on;
}

bool use_pairs() {
  static bool on = [] {
    const char* e = std::getenv("MVD_PAIRED");
    if (e && e[0] == '0') return false;
    for (const char* v : {"MVD_FIXED_PLANES", "MVD_STAGED_PLANES", "MVD_Z_INPLACE", "MVD_PLANE_CAP", "MVD_PLANE_THREADS",
                          "MVD_ZOCC"})
      if (std::getenv(v)) return false;
    return true;
  }();
  return on;
}

namespace {

// A transform length's two radices; r0 == 0: the length has none.
struct Radices {
  int r0 = 0, r1 = 0;
};

constexpr int kPairMaxLen = 400;
// cost of a plane that leaves one CTA per SM: per voxel of its tiles, 512x512x256 measured 7 to 20%
// more at 226 KB per plane than at 112 KB
constexpr double kPairOneCtaCost = 1.1;
// a plane buffer leaves the epilogues their static shared memory
constexpr size_t kPairSmemMax = 227 * 1024 - 1024;

// Radix pairs per length, the choice that needs the fewest registers: x stages hold 4 registers
// per point of either radix, the y stage next to the real step 8 per point of r0 and the other 4
// per point of r1.
struct ZRadices {
  int a = 0, b = 0, c = 0;
};

struct PairLengths {
  Radices x[kPairMaxLen + 1], y[kPairMaxLen + 1];
  ZRadices z[kPairMaxLen + 1];
  PairLengths() {
    auto fill = [](Radices* out, std::initializer_list<int> a, std::initializer_list<int> b, int w0) {
      int best[kPairMaxLen + 1];
      std::fill(best, best + kPairMaxLen + 1, INT_MAX);
      for (int r0 : a)
        for (int r1 : b) {
          const int n = r0 * r1;
          if (n > kPairMaxLen) continue;
          // the larger of the two, then the smaller first radix
          const int cost = std::max(w0 * r0, r1) * 64 + r0;
          if (cost < best[n]) {
            best[n] = cost;
            out[n] = Radices{r0, r1};
          }
        }
    };
#define MVD_LIST(R) R,
    fill(x, {MVD_PAIR_X0(MVD_LIST)}, {MVD_PAIR_X1(MVD_LIST)}, 1);
    fill(y, {MVD_PAIR_Y0(MVD_LIST)}, {MVD_PAIR_Y1(MVD_LIST)}, 2);
    // z: two stages where both radices are at most 10, else three; the middle one (c, beside the
    // kernel spectrum) no larger than the outer one
    int best[kPairMaxLen + 1];
    std::fill(best, best + kPairMaxLen + 1, INT_MAX);
    for (int c : {MVD_PAIR_ZC(MVD_LIST)})
      for (int a : {MVD_PAIR_Z(MVD_LIST)})
        for (int b : {MVD_PAIR_Z(MVD_LIST)}) {
          const int n = a * b * c;
          if (n > kPairMaxLen || c > a) continue;
          const int cost = (b > 1 ? 1000 : 0) + 16 * std::max(a, std::max(b, c)) + c;
          if (cost < best[n]) {
            best[n] = cost;
            z[n] = ZRadices{a, b, c};
          }
        }
#undef MVD_LIST
  }
};

const PairLengths& pair_lengths() {
  static const PairLengths l;
  return l;
}

struct PairAxis {
  AxisTiles a;
  int shift = 0;  // extra halo on the low side (x: even tile origins)
};

// Tile counts n = 1, 2, ... with the shortest length that covers the axis; x: lengths 2 m.
template <class Has>
std::vector<PairAxis> pair_axis_options(int size, int k, Has has, bool x, int off, int nvol) {
  std::vector<PairAxis> out;
  int last = -1;
  for (int n = 1; n <= size && n <= 64; ++n) {
    const int need = std::max((size + n - 1) / n + k - 1, 2);
    int T = need;
    if (x) T += T & 1;
    while (T <= (x ? 2 : 1) * kPairMaxLen && !has(x ? T / 2 : T)) T += x ? 2 : 1;
    if (T > (x ? 2 : 1) * kPairMaxLen || T == last) continue;
    last = T;
    PairAxis p;
    p.a.size = size;
    p.a.k = k;
    p.a.T = T;
    p.a.E = T - k + 1;
    p.a.n = (size + p.a.E - 1) / p.a.E;
    if (x && nvol % 2 == 0) {
      // even tile origins (8-byte gathers) where the length has the room for them
      const int shift = (off - k / 2) & 1;
      int E = T - k + 1 - shift;
      if (p.a.n > 1) E -= E & 1;
      if (E > 0 && (long long)E * p.a.n >= size) {
        p.a.E = E;
        p.shift = shift;
      }
    }
    out.push_back(p);
    if (p.a.E < 8 && p.a.E < size) break;  // smaller tiles would be nearly all halo
  }
  return out;
}

int pair_cols(int m) { return (m + 2) / 2; }  // pairs that hold the m + 1 columns
int pair_pitch(int m) { return (2 * pair_cols(m)) | 1; }
// a plane, then the tables: roots of x and y, column units
size_t pair_plane_smem(int m, int ty) {
  const int tab = (m + 1) / 2 + (ty + 1) / 2 + m / 2 + 1;
  return ((size_t)(ty / 2) * pair_pitch(m) + tab) * sizeof(float4);
}

// CTA size of the plane passes: 128 registers per thread, so 512 threads per SM over the CTAs that
// share one (that fit its shared memory, and that there are: 270 planes of 128x128x64 took 13.2 us with
// 128 threads, 12.3 with 256); no more than a stage has work for, but 128 for the gather and the
// epilogue (40x32x24: 8.8 us with 64, 8.5).
int pair_plane_threads(const PairShape& s, size_t smem, long long planes) {
  const int ctas = (int)std::min<long long>(pair_ctas_per_sm(smem), (planes + 151) / 152);
  int t = ctas >= 4 ? 128 : ctas >= 2 ? 256 : 512;
  const int work = std::max(std::max(s.ty / 2 * s.r1x, s.ty / 2 * s.r0x), std::max(s.nunits * (s.r1y / 2), s.pc * s.r0y));
  return std::max(128, std::min(t, (work + 31) / 32 * 32));
}

// CTA size of the z pass: 640 threads per SM in all, so what counts is how well a size divides the
// stages' items (their points x 8 pencil pairs), per CTA that shares the SM: 128 threads, or 160 or 64
// where that is an eighth better by this measure, and no more than one step takes.  us per pass with
// 64 / 128 / 160 threads: 120 points 11.8 / 13.8 / 14.3 (203x157x91, 3 views); 320 points 328 / 274 / 259
// (512x512x256, 4 views); 240 and 216 points 63.0 / 51.1 / 52.1 (256x256x192, 4 views); 90 and 72 points
// 7.5 / 6.5 / 9.2 (128x128x64, 2 views).  96 threads were never the best.
int pair_z_threads(const PairShape& s) {
  const int na = s.bz * s.cz * kPairChunk, nb = s.bz > 1 ? s.az * s.cz * kPairChunk : 0, nc = s.az * s.bz * kPairChunk;
  const int most = std::max({na, nb, nc});
  if (most <= 128) return most <= 64 ? 64 : 128;
  const int fit = std::max(1, (int)(227 * 1024 / (((size_t)s.tz * kPairChunk + s.tz) * sizeof(float4) + 1024)));
  auto cost = [&](int t) {
    auto steps = [t](int n) { return (n + t - 1) / t; };
    return (2.0 * steps(na) + 2.0 * steps(nb) + 1.5 * steps(nc)) / std::min(640 / t, fit);
  };
  const double c64 = cost(64), c128 = cost(128), c160 = cost(160);
  if (std::min(c64, c160) > 0.88 * c128) return 128;
  return c64 < c160 ? 64 : 160;
}

// Tile shape and tables for the pair kernels; false when no shape fits (a kernel too large for
// their lengths).
bool plan_pairs(ConvPlan& p, int nx, int ny, int nz, int kx, int ky, int kz, const PlanOptions& opt) {
  const PairLengths& L = pair_lengths();
  const auto ox = pair_axis_options(nx, kx, [&](int m) { return L.x[m].r0 > 0; }, true, opt.off_x, opt.vol_x > 0 ? opt.vol_x : nx);
  const auto oy = pair_axis_options(ny, ky, [&](int m) { return L.y[m].r0 > 0; }, false, 0, 0);
  const auto oz = pair_axis_options(nz, kz, [&](int m) { return L.z[m].a > 0; }, false, 0, 0);
  const size_t limit = opt.pair_smem ? std::min(opt.pair_smem, kPairSmemMax) : kPairSmemMax;
  double best = 1e300;
  const PairAxis *bx = nullptr, *by = nullptr, *bz = nullptr;
  for (const auto& a : ox)
    for (const auto& b : oy) {
      const int m = a.a.T / 2;
      const size_t smem = pair_plane_smem(m, b.a.T);
      if (smem > limit) continue;
      const double ctas = std::min(4, pair_ctas_per_sm(smem));
      const double plane = 2.0 * pair_cols(m) * b.a.T;
      for (const auto& c : oz) {
        const double nt = (double)a.a.n * b.a.n * c.a.n;
        const double f = ctas >= 2 ? 1.0 : kPairOneCtaCost;
        // without whole waves the cost is at least this (most shapes end here)
        if ((4.0 * f + 1.8) * nt * c.a.T * plane / 152.0 >= best) continue;
        // time of a pass in units of one value of one SM: whole waves of CTAs, those of a wave
        // sharing the SM
        auto waves = [](double items, double per_sm, double work) {
          const double conc = std::min(per_sm, std::ceil(items / 152.0));
          return std::ceil(items / (152.0 * conc)) * conc * work;
        };
        const double cost = (4.0 * f * waves(nt * c.a.T, ctas, plane) +
                             1.8 * waves(nt * std::ceil(plane / (2.0 * kPairChunk)), 4.0, 2.0 * kPairChunk * c.a.T)) *
                            (1.0 + 1e-3 * nt);
        if (cost < best) {
          best = cost;
          bx = &a;
          by = &b;
          bz = &c;
        }
      }
    }
  if (!bx) return false;
  p.ax = bx->a;
  p.ay = by->a;
  p.az = bz->a;
  PairShape& s = p.ps;
  s.m = p.ax.T / 2;
  s.ty = p.ay.T;
  s.tz = p.az.T;
  s.r0x = L.x[s.m].r0;
  s.r1x = L.x[s.m].r1;
  s.r0y = L.y[s.ty].r0;
  s.r1y = L.y[s.ty].r1;
  s.az = L.z[s.tz].a;
  s.bz = L.z[s.tz].b;
  s.cz = L.z[s.tz].c;
  s.pc = pair_cols(s.m);
  s.pitch = pair_pitch(s.m);
  s.nunits = s.m / 2 + 1;
  const int plane = s.pc * s.ty;
  const long long tile_spec = 2LL * plane * s.tz;
  long long off = 0;
  for (int iz = 0; iz < p.az.n; ++iz)
    for (int iy = 0; iy < p.ay.n; ++iy)
      for (int ix = 0; ix < p.ax.n; ++ix) {
        TileDesc t{};
        t.tx = p.ax.T; t.ty = p.ay.T; t.tz = p.az.T;
        t.px = s.pc;
        t.pitch = s.pitch;
        t.hx = kx / 2 + bx->shift; t.hy = ky / 2; t.hz = kz / 2;
        const int ex0 = ix * p.ax.E, ey0 = iy * p.ay.E, ez0 = iz * p.az.E;
        t.ox = ex0 - t.hx; t.oy = ey0 - t.hy; t.oz = ez0 - t.hz;
        t.ex = std::min(p.ax.E, nx - ex0);
        t.ey = std::min(p.ay.E, ny - ey0);
        t.ez = std::min(p.az.E, nz - ez0);
        t.spec_off = off;
        off += tile_spec;
        p.tiles.push_back(t);
      }
  p.spec_elems = off;
  p.otf_elems = tile_spec;
  p.paired = true;
  p.smem_pair = pair_plane_smem(s.m, s.ty);
  p.smem_pair_z = ((size_t)s.tz * kPairChunk + (s.tz + 1) / 2 + (s.bz > 1 ? (s.bz * s.cz + 1) / 2 : 0)) * sizeof(float4);
  p.z_chunks = (plane + kPairChunk - 1) / kPairChunk;
  p.pair_threads = opt.threads > 0 ? opt.threads : pair_plane_threads(s, p.smem_pair, (long long)p.tiles.size() * s.tz);
  p.threads_plane = p.pair_threads;
  p.pair_z_threads = pair_z_threads(s);
  return true;
}

}  // namespace

int pair_ctas_per_sm(size_t smem) {
  // an SM has 228 KB of shared memory; a CTA takes 1 KB for the system and up to 1 KB statically
  return (int)std::max<size_t>(1, 228 * 1024 / (smem + 2048));
}

// The plan's tables in one block: its tiles, the full tile, the stage roots and the column units.
void ConvPlan::upload_pair() {
  std::vector<unsigned char> host;
  auto put = [&](const void* src, size_t bytes) {
    const size_t at = host.size();
    host.resize(at + (bytes + 15) / 16 * 16);
    std::memcpy(host.data() + at, src, bytes);
    return at;
  };
  std::vector<TileDesc> td(tiles);
  TileDesc full = tiles[0];
  full.ox = full.oy = full.oz = 0;
  full.hx = full.hy = full.hz = 0;
  full.ex = full.tx; full.ey = full.ty; full.ez = full.tz;
  full.spec_off = 0;
  td.push_back(full);
  put(td.data(), td.size() * sizeof(TileDesc));
  auto root = [](long long num, long long den) {  // exp(-2 pi i num / den)
    const double a = -2.0 * M_PI * (double)(num % den) / (double)den;
    return make_float2((float)std::cos(a), (float)std::sin(a));
  };
  auto roots = [&](int n, int r0, int r1) {  // W^(j k0) by position r1 k0 + j
    std::vector<float2> w(n);
    for (int k0 = 0; k0 < r0; ++k0)
      for (int j = 0; j < r1; ++j) w[k0 * r1 + j] = root((long long)j * k0, n);
    return w;
  };
  const auto wx = roots(ps.m, ps.r0x, ps.r1x), wy = roots(ps.ty, ps.r0y, ps.r1y), wz = roots(ps.tz, ps.az, ps.bz * ps.cz),
             wc = roots(ps.bz * ps.cz, ps.bz, ps.cz);
  // one unit per column pair (f, M - f), f = 0 .. M / 2, ordered by the position of f
  auto pos = [&](int f) { return (f % ps.r0x) * ps.r1x + f / ps.r0x; };
  std::vector<PairUnit> un;
  for (int f = 0; f <= ps.m / 2; ++f) {
    const float2 w = root(f, 2LL * ps.m);
    PairUnit u{};
    u.a = (short)pos(f);
    u.b_load = (short)(f == 0 ? 0 : pos(ps.m - f));
    u.b_store = (short)(f == 0 ? ps.m : pos(ps.m - f));
    u.wx = w.x;
    u.wy = w.y;
    un.push_back(u);
  }
  std::sort(un.begin(), un.end(), [](const PairUnit& a, const PairUnit& b) { return a.a < b.a; });
  const size_t ox = put(wx.data(), wx.size() * sizeof(float2)), oy = put(wy.data(), wy.size() * sizeof(float2));
  const size_t ou = put(un.data(), un.size() * sizeof(PairUnit)), oz = put(wz.data(), wz.size() * sizeof(float2));
  const size_t oc = ps.bz > 1 ? put(wc.data(), wc.size() * sizeof(float2)) : oz;
  d_pair.alloc(host.size());
  upload_table(d_pair.p, host.data(), host.size());
  const float4* d = d_pair.as<float4>();
  ps.tab = d + ox / 16;
  ps.tab_y = (int)((oy - ox) / 16);
  ps.tab_units = (int)((ou - ox) / 16);
  ps.ntab = (int)((oz - ox) / 16);
  ps.tabz = d + oz / 16;
  ps.ntabz = (int)((host.size() - oz) / 16);
  ps.tab_c = (int)((oc - oz) / 16);
  ps.perz = ps.bz > 1 ? ps.bz : ps.az;
}

// Tile shape of the scalar kernels; false when none fits the kernel.
static bool scalar_tiles(int nx, int ny, int nz, int kx, int ky, int kz, const PlanOptions& opt, AxisTiles& bx,
                         AxisTiles& by, AxisTiles& bz) {
  auto opts = [&](int size, int k, bool even, int tmax, int force) {
    if (force > 0) {
      AxisTiles a;
      a.size = size;
      a.k = k;
      a.T = force;
      a.E = force - k + 1;
      if (a.E <= 0 || (even && (force & 1)) || !is_smooth(even ? force / 2 : force))
        throw std::invalid_argument("forced tile size is too small or not smooth");
      a.n = (size + a.E - 1) / a.E;
      return std::vector<AxisTiles>{a};
    }
    return axis_options(size, k, even, tmax);
  };
  auto ox = opts(nx, kx, true, 2 * (kPlaneCap / 8), opt.force_tx);
  auto oy = opts(ny, ky, false, kPlaneCap / 2, opt.force_ty);
  auto oz = opts(nz, kz, false, kPlaneCap / kZPitch, opt.force_tz);
  double best = 1e300;
  // an explicit budget (the autotuner's candidates) is a hard limit; the default plan weighs
  // the plane size and the compiled shapes (plane_cost_factor)
  const int limit = opt.cap > 0 ? opt.cap : plane_limit();
  for (auto& a : ox)
    for (auto& b : oy) {
      const long long plane = (long long)row_pitch(a.T / 2) * b.T;
      if (plane > limit) continue;
      const double factor = opt.cap > 0 ? 1.0 : plane_cost_factor(a.T, b.T, plane);
      for (auto& c : oz) {
        const double ntiles = (double)a.n * b.n * c.n;
        const double cost = ntiles * a.T * b.T * c.T * (1.0 + 1e-3 * ntiles) * factor;
        if (cost < best) {
          best = cost;
          bx = a;
          by = b;
          bz = c;
        }
      }
    }
  return best < 1e300;
}

// Whether the scalar kernels are the faster ones although the pair kernels have a shape: their lengths
// reach further along an axis (the pair kernels' end at 512, 200 and 400 points in x, y and z), so a
// kernel nearly as long as those leaves a pair plan many tiles that are mostly halo.  The time of an
// iteration goes with the padded voxels, of which a scalar pass takes about 2.4 times as long: scalar /
// pair time against pair / scalar padding, at volumes from 128x128x64 to 512x512x256 and kernels of 121 to
// 501 points along one axis: 1.3 to 1.6 at 1.4 to 1.8, 1.03 to 1.13 at 2.1 to 2.5, 0.7 to 0.9 at 2.6 to
// 3.1, 0.2 at 12 (21x161x21 on 400x300x200: 2.23 ms on pairs, 2.30 scalar; 21x175x21: 3.25, 2.30; 15x195x15
// on 256x256x192: 5.98, 1.16).  With no more planes than SMs a pass is one plane's latency, and the pair
// kernels win at any padding (31x31x1 on 64x64x1: 41 us with 38 times the volume, 58).
constexpr double kScalarPaddingCost = 2.4;
static bool scalar_plan_pays(const ConvPlan& p) {
  if ((long long)p.tiles.size() * p.ps.tz <= 152) return false;
  const double most = (double)p.padded_voxels() / kScalarPaddingCost;
  // no plan pads to less than one tile of the exact size
  if (most <= (double)(p.nx + p.kx - 1) * (p.ny + p.ky - 1) * (p.nz + p.kz - 1)) return false;
  AxisTiles x, y, z;
  if (!scalar_tiles(p.nx, p.ny, p.nz, p.kx, p.ky, p.kz, PlanOptions(), x, y, z)) return false;
  return (double)x.n * x.T * y.n * y.T * z.n * z.T < most;
}

std::unique_ptr<ConvPlan> make_conv_plan(PlanTable& pt, int nx, int ny, int nz, int kx, int ky,
                                         int kz, const PlanOptions& opt) {
  if (nx < 1 || ny < 1 || nz < 1) throw std::invalid_argument("empty volume");
  if (kx < 1 || ky < 1 || kz < 1 || !(kx & 1) || !(ky & 1) || !(kz & 1))
    throw std::invalid_argument("kernel sizes must be odd and positive");
  if (use_pairs() && !opt.scalar) {
    auto plan = std::make_unique<ConvPlan>();
    ConvPlan& p = *plan;
    p.nx = nx; p.ny = ny; p.nz = nz;
    p.kx = kx; p.ky = ky; p.kz = kz;
    p.vol[0] = nx; p.vol[1] = ny; p.vol[2] = nz;
    p.box_hi[0] = nx; p.box_hi[1] = ny; p.box_hi[2] = nz;
    if (plan_pairs(p, nx, ny, nz, kx, ky, kz, opt) && !scalar_plan_pays(p)) {
      p.upload();
      return plan;
    }
  }
  AxisTiles bx, by, bz;
  if (!scalar_tiles(nx, ny, nz, kx, ky, kz, opt, bx, by, bz))
    throw std::invalid_argument("no tile shape fits this kernel (kernel too large)");
  auto plan = std::make_unique<ConvPlan>();
  ConvPlan& p = *plan;
  p.nx = nx; p.ny = ny; p.nz = nz;
  p.kx = kx; p.ky = ky; p.kz = kz;
  p.vol[0] = nx; p.vol[1] = ny; p.vol[2] = nz;
  p.box_hi[0] = nx; p.box_hi[1] = ny; p.box_hi[2] = nz;
  p.ax = bx; p.ay = by; p.az = bz;
  const int px = bx.T / 2 + 1;
  const int pitch = row_pitch(bx.T / 2);
  const int plx = pt.index_of(bx.T / 2, opt.ascending), ply = pt.index_of(by.T, opt.ascending),
            plz = pt.index_of(bz.T, opt.ascending);
  const long long tile_spec = (long long)px * by.T * bz.T;
  long long off = 0;
  for (int iz = 0; iz < bz.n; ++iz)
    for (int iy = 0; iy < by.n; ++iy)
      for (int ix = 0; ix < bx.n; ++ix) {
        TileDesc t{};
        t.tx = bx.T; t.ty = by.T; t.tz = bz.T;
        t.px = px;
        t.pitch = pitch;
        t.hx = kx / 2; t.hy = ky / 2; t.hz = kz / 2;
        const int ex0 = ix * bx.E, ey0 = iy * by.E, ez0 = iz * bz.E;
        t.ox = ex0 - kx / 2; t.oy = ey0 - ky / 2; t.oz = ez0 - kz / 2;
        t.ex = std::min(bx.E, nx - ex0);
        t.ey = std::min(by.E, ny - ey0);
        t.ez = std::min(bz.E, nz - ez0);
        t.plan_x = plx; t.plan_y = ply; t.plan_z = plz;
        t.spec_off = off;
        t.otf_off = 0;
        off += tile_spec;
        p.tiles.push_back(t);
      }
  p.spec_elems = off;
  p.otf_elems = tile_spec;
  p.smem_plane = 2 * (size_t)by.T * pitch * sizeof(float2);
  p.threads_plane = opt.threads > 0 ? opt.threads : plane_threads();
  p.ascending = opt.ascending;
  p.generic = opt.generic || opt.ascending;  // compiled kernels hold the descending order
  p.staged = use_staged_planes();
  p.smem_z = 2 * (size_t)bz.T * kZPitch * sizeof(float2);
  fill_items(p);
  p.upload();
  return plan;
}

void place_plan(ConvPlan& p, int dx, int dy, int dz, const int vol[3]) {
  for (auto& t : p.tiles) {
    t.ox += dx;
    t.oy += dy;
    t.oz += dz;
  }
  const int d[3] = {dx, dy, dz}, n[3] = {p.nx, p.ny, p.nz};
  for (int i = 0; i < 3; ++i) {
    p.vol[i] = vol[i];
    p.box_lo[i] = d[i];
    p.box_hi[i] = d[i] + n[i];
  }
  p.upload();
}

std::string describe(const ConvPlan& p) {
  std::ostringstream os;
  os << "volume " << p.nx << "x" << p.ny << "x" << p.nz << " kernel " << p.kx << "x" << p.ky << "x"
     << p.kz << " tiles " << p.ax.n << "x" << p.ay.n << "x" << p.az.n << " of " << p.ax.T << "x"
     << p.ay.T << "x" << p.az.T << " (effective " << p.ax.E << "x" << p.ay.E << "x" << p.az.E
     << "), padded/volume " << (double)p.padded_voxels() / ((double)p.nx * p.ny * p.nz);
  return os.str();
}

// ------------------------------------------------------------------------------------------
// launches (the pass kernels are instantiated in passes_fwd.cu, passes_inv.cu, passes_z.cu)
// ------------------------------------------------------------------------------------------
// raise a kernel's dynamic shared-memory limit once per (device, kernel, size)
void set_smem_raw(const void* kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> done;
  int dev = 0;
  MVD_CHECK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto key = std::make_pair(dev, kernel);
  auto it = done.find(key);
  if (it != done.end() && it->second >= bytes) return;
  MVD_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  done[key] = bytes;
}

void convolve(PlanTable& pt, const ConvPlan& plan, const float* in, Ext ext, float value,
              const float2* otf, float2* spec, float* out, cudaStream_t s) {
  if (ext == Ext::Mirror)
    launch_fwd_mirror(pt, plan, in, spec, s);
  else
    launch_fwd_value(pt, plan, in, value, spec, s);
  launch_z(pt, plan, spec, otf, s);
  launch_inv_store(pt, plan, spec, out, s);
}

// ------------------------------------------------------------------------------------------
// OTF: kernel placed with its centre at the tile origin (wrap-around), forward 3D FFT,
// scaled by 1 / (tx ty tz) so that the unnormalised inverse transforms give the convolution.
// ------------------------------------------------------------------------------------------
__global__ void place_kernel_kernel(const float* __restrict__ k, int kx, int ky, int kz, float* __restrict__ vol,
                                    int tx, int ty, int tz) {
  const long long n = (long long)kx * ky * kz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % kx);
    const int y = (int)((i / kx) % ky);
    const int z = (int)(i / ((long long)kx * ky));
    const int wx = ((x - kx / 2) % tx + tx) % tx;
    const int wy = ((y - ky / 2) % ty + ty) % ty;
    const int wz = ((z - kz / 2) % tz + tz) % tz;
    vol[((long long)wz * ty + wy) * tx + wx] = k[i];
  }
}

void build_otf(PlanTable& pt, const ConvPlan& plan, const float* kernel, float2* otf, DevBuf& scratch,
               cudaStream_t s) {
  const int tx = plan.ax.T, ty = plan.ay.T, tz = plan.az.T;
  if (plan.kx > tx || plan.ky > ty || plan.kz > tz) throw std::invalid_argument("kernel larger than tile");
  const size_t vox = (size_t)tx * ty * tz;
  scratch.ensure(vox * sizeof(float));
  MVD_CHECK(cudaMemsetAsync(scratch.p, 0, vox * sizeof(float), s));
  const long long kn = (long long)plan.kx * plan.ky * plan.kz;
  place_kernel_kernel<<<(int)std::min<long long>((kn + 255) / 256, 4096), 256, 0, s>>>(
      kernel, plan.kx, plan.ky, plan.kz, scratch.as<float>(), tx, ty, tz);
  MVD_CHECK(cudaGetLastError());
  count_launch();
  // one tile covering the placed kernel volume exactly; its spectrum goes to `otf`.  The product of
  // two spectra carries the passes' scale twice.
  launch_fwd_value_tiles(pt, plan, TileSet::Full, GatherValue::full(scratch.as<float>(), tx, ty, tz, 0.f), otf, s);
  const double sc = spectrum_scale(plan) * spectrum_scale(plan);
  launch_z_forward(pt, plan, TileSet::Full, otf, (float)(1.0 / (sc * tx * ty * tz)), s);
}

// ------------------------------------------------------------------------------------------
// elementwise and reduction kernels
// ------------------------------------------------------------------------------------------
static int grid_for(long long n, int threads = 256) {
  long long b = (n + threads - 1) / threads;
  return (int)std::max<long long>(1, std::min<long long>(b, 152LL * 16));
}

__device__ __forceinline__ void block_reduce_add2(double a, double b, double* out) {
  __shared__ double ra[32], rb[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { ra[warp] = a; rb[warp] = b; }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    a = lane < nw ? ra[lane] : 0.0;
    b = lane < nw ? rb[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      atomicAdd(out, a);
      atomicAdd(out + 1, b);
    }
  }
}

__global__ void sum_f64_kernel(const float* __restrict__ x, long long n, double* out) {
  double a = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    a += (double)x[i];
  __shared__ double r[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) r[warp] = a;
  __syncthreads();
  if (warp == 0) {
    a = lane < (int)(blockDim.x >> 5) ? r[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) atomicAdd(out, a);
  }
}

void dev_sum_f64(const float* x, long long n, double* out, cudaStream_t s) {
  sum_f64_kernel<<<grid_for(n), 256, 0, s>>>(x, n, out);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void scale_div_kernel(float* x, long long n, const double* d) {
  const double div = *d;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    x[i] = (float)((double)x[i] / div);
}

void dev_scale_div(float* x, long long n, const double* d, cudaStream_t s) {
  scale_div_kernel<<<grid_for(n), 256, 0, s>>>(x, n, d);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// Mirror.mirror along every axis: p <-> n-1-p for p <= n/2 (for even n the middle pair is
// swapped twice and stays in place: Mirror.java:94-112)
__device__ __forceinline__ int mirror_pos(int p, int n) {
  if ((n & 1) == 0 && (p == n / 2 - 1 || p == n / 2)) return p;
  return n - 1 - p;
}

__global__ void mirror_kernel(const float* __restrict__ in, float* __restrict__ out, int nx, int ny, int nz) {
  const long long n = (long long)nx * ny * nz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int y = (int)((i / nx) % ny);
    const int z = (int)(i / ((long long)nx * ny));
    out[i] = in[((long long)mirror_pos(z, nz) * ny + mirror_pos(y, ny)) * nx + mirror_pos(x, nx)];
  }
}

void dev_mirror(const float* in, float* out, int nx, int ny, int nz, cudaStream_t s) {
  mirror_kernel<<<grid_for((long long)nx * ny * nz), 256, 0, s>>>(in, out, nx, ny, nz);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void mul_kernel(float* a, const float* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    a[i] = __fmul_rn(a[i], b[i]);
}
void dev_mul(float* a, const float* b, long long n, cudaStream_t s) {
  mul_kernel<<<grid_for(n), 256, 0, s>>>(a, b, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// MVDeconFFT.pow (:346-354): repeated float multiplication
__global__ void pow_kernel(float* a, int power, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = a[i];
    float r = v;
    for (int k = 1; k < power; ++k) r = __fmul_rn(r, v);
    a[i] = r;
  }
}
void dev_pow(float* a, int power, long long n, cudaStream_t s) {
  pow_kernel<<<grid_for(n), 256, 0, s>>>(a, power, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void fill_kernel(float* a, float v, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    a[i] = v;
}
void dev_fill(float* a, float v, long long n, cudaStream_t s) {
  fill_kernel<<<grid_for(n), 256, 0, s>>>(a, v, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

struct ViewPtrs {
  const float* p[16];
};

// FirstIteration.call (FirstIteration.java:84-154): per voxel the mean of the positive view
// values; summed (FP64) over voxels with at least one positive value, and counted.
// hi + lo = a + b exactly (Knuth's two-sum)
__device__ __forceinline__ void two_sum(float a, float b, float& hi, float& lo) {
  hi = __fadd_rn(a, b);
  const float bb = __fsub_rn(hi, a);
  lo = __fadd_rn(__fsub_rn(a, __fsub_rn(hi, bb)), __fsub_rn(b, bb));
}

// (hi, lo) += (bh, bl), renormalised; ~2^-44 relative
__device__ __forceinline__ void pair_add(float& hi, float& lo, float bh, float bl) {
  float s, e;
  two_sum(hi, bh, s, e);
  e = __fadd_rn(e, __fadd_rn(lo, bl));
  hi = __fadd_rn(s, e);
  lo = __fsub_rn(e, __fsub_rn(hi, s));
}

// FirstIteration.compatibleLoop (FirstIteration.java:124-154): per voxel the mean of the
// views' positive values, summed over the voxels that have any (RealSum), and their count.
// GB300's FP64 pipe cannot take a double division and six double additions per voxel at
// HBM speed, so each thread carries its sum as a float pair (the voxel's view sum by exact
// two-sums, times 1/c as a pair), flushed into a double every 16 voxels.  The reference's
// RealSum is itself order-dependent; each pair chunk is accurate to ~2^-43.
//
// The views' loads of a voxel go out before the first is used, and one wave of blocks walks the volume:
// the double sums over a block's threads are FP64 work per thread, not per voxel (at 16 blocks an SM
// they took most of the 51 us at 3 views of 203x157x91).
template <int NV>
__global__ void __launch_bounds__(256, 6) first_iteration_kernel(ViewPtrs v, long long n, double* out) {
  float acc_hi = 0.f, acc_lo = 0.f;
  double total = 0.0;
  unsigned long long cnt = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float xs[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) xs[k] = __ldg(v.p[k] + i);
    float s_hi = 0.f, s_lo = 0.f;
    int c = 0;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const float x = xs[k];
      if (x > 0.f) {
        float e;
        two_sum(s_hi, x, s_hi, e);
        s_lo = __fadd_rn(s_lo, e);
        ++c;
      }
    }
    if (c > 0) {
      // (s_hi + s_lo) / c: q = s_hi / c rounded, the remainder s_hi - q c is exact (an FMA)
      const float fc = (float)c;
      const float q = __fdiv_rn(s_hi, fc);
      const float r = __fadd_rn(__fmaf_rn(-q, fc, s_hi), s_lo);
      pair_add(acc_hi, acc_lo, q, __fdiv_rn(r, fc));
      if ((++cnt & 15) == 0) {
        total += (double)acc_hi + (double)acc_lo;
        acc_hi = acc_lo = 0.f;
      }
    }
  }
  block_reduce_add2(total + ((double)acc_hi + (double)acc_lo), (double)cnt, out);
}

void dev_first_iteration(const float* const* views, int nviews, long long n, double* out, cudaStream_t s) {
  ViewPtrs vp{};
  if (nviews > 16) throw std::invalid_argument("at most 16 views");
  for (int i = 0; i < nviews; ++i) vp.p[i] = views[i];
  using Kernel = void (*)(ViewPtrs, long long, double*);
  static constexpr Kernel kernels[17] = {
      first_iteration_kernel<1>,  first_iteration_kernel<1>,  first_iteration_kernel<2>,  first_iteration_kernel<3>,
      first_iteration_kernel<4>,  first_iteration_kernel<5>,  first_iteration_kernel<6>,  first_iteration_kernel<7>,
      first_iteration_kernel<8>,  first_iteration_kernel<9>,  first_iteration_kernel<10>, first_iteration_kernel<11>,
      first_iteration_kernel<12>, first_iteration_kernel<13>, first_iteration_kernel<14>, first_iteration_kernel<15>,
      first_iteration_kernel<16>};
  kernels[nviews]<<<std::min(grid_for(n), 152 * 6), 256, 0, s>>>(vp, n, out);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// MVDeconvolution.java:133-147: psi := avg (0.5 if NaN)
__global__ void fill_avg_kernel(float* psi, const double* sc, long long n) {
  double avg = sc[0] / sc[1];
  if (isnan(avg)) avg = 0.5;
  const float v = (float)avg;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    psi[i] = v;
}
void dev_fill_from_avg(float* psi, const double* sc, long long n, cudaStream_t s) {
  fill_avg_kernel<<<grid_for(n), 256, 0, s>>>(psi, sc, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// MVDeconvolution.java:201-208: psi := 0 where no view has data
__global__ void mask_kernel(float* psi, ViewPtrs v, int nviews, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    bool any = false;
    for (int k = 0; k < nviews; ++k) any |= __ldg(v.p[k] + i) > 0.f;
    if (!any) psi[i] = 0.f;
  }
}
void dev_mask(float* psi, const float* const* views, int nviews, long long n, cudaStream_t s) {
  ViewPtrs vp{};
  if (nviews > 16) throw std::invalid_argument("at most 16 views");
  for (int i = 0; i < nviews; ++i) vp.p[i] = views[i];
  mask_kernel<<<grid_for(n), 256, 0, s>>>(psi, vp, nviews, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void quotient_kernel(float* b, const float* img, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float x = img[i];
    b[i] = EpiQuotient::quotient(x, b[i]);
  }
}
void dev_quotient(float* b, const float* img, long long n, cudaStream_t s) {
  quotient_kernel<<<grid_for(n), 256, 0, s>>>(b, img, n);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void update_kernel(float* psi, const float* integral, const float* weight, float lambda, long long n,
                              double* stat_sum, unsigned* stat_max) {
  EpiUpdate e{psi, weight, lambda, stat_sum, stat_max, 0, 0, 0.f, 0.f, StatArchive{}};
  e.acc_init();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    e(i, integral[i]);
  e.finish();
}
void dev_update(float* psi, const float* integral, const float* weight, float lambda, long long n,
                double* stat_sum, unsigned* stat_max, cudaStream_t s) {
  update_kernel<<<grid_for(n), 256, 0, s>>>(psi, integral, weight, lambda, n, stat_sum, stat_max);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void copy_block_kernel(const float* __restrict__ vol, int nx, int ny, int nz, float* __restrict__ blk,
                                  int bx, int by, int bz, int ox, int oy, int oz, int mode, float value) {
  const long long n = (long long)bx * by * bz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % bx) + ox;
    const int y = (int)((i / bx) % by) + oy;
    const int z = (int)(i / ((long long)bx * by)) + oz;
    float v;
    if (mode == 0) {
      v = vol[((long long)mirror_single(z, nz) * ny + mirror_single(y, ny)) * nx + mirror_single(x, nx)];
    } else {
      v = (x < 0 || y < 0 || z < 0 || x >= nx || y >= ny || z >= nz) ? value
                                                                      : vol[((long long)z * ny + y) * nx + x];
    }
    blk[i] = v;
  }
}
void dev_copy_block(const float* vol, int nx, int ny, int nz, float* block, int bx, int by, int bz, int ox,
                    int oy, int oz, Ext ext, float value, cudaStream_t s) {
  copy_block_kernel<<<grid_for((long long)bx * by * bz), 256, 0, s>>>(vol, nx, ny, nz, block, bx, by, bz, ox, oy,
                                                                    oz, ext == Ext::Mirror ? 0 : 1, value);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

__global__ void paste_block_kernel(const float* __restrict__ blk, int bx, int by, int lx, int ly, int lz,
                                   float* __restrict__ vol, int nx, int ny, int ex0, int ey0, int ez0, int sx,
                                   int sy, int sz) {
  const long long n = (long long)sx * sy * sz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % sx);
    const int y = (int)((i / sx) % sy);
    const int z = (int)(i / ((long long)sx * sy));
    vol[((long long)(ez0 + z) * ny + (ey0 + y)) * nx + (ex0 + x)] =
        blk[((long long)(lz + z) * by + (ly + y)) * bx + (lx + x)];
  }
}
void dev_paste_block(const float* block, int bx, int by, int bz, int lx, int ly, int lz, float* vol, int nx,
                     int ny, int nz, int ex0, int ey0, int ez0, int sx, int sy, int sz, cudaStream_t s) {
  (void)bz;
  (void)nz;
  paste_block_kernel<<<grid_for((long long)sx * sy * sz), 256, 0, s>>>(block, bx, by, lx, ly, lz, vol, nx, ny, ex0,
                                                                     ey0, ez0, sx, sy, sz);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

// A warp takes a row of x at a time (kBoxRun voxels of it, if it is longer), four loads of each volume per
// lane in flight, so that y and z need one division a row and one set of atomics a block.  A voxel per
// thread cost three 64-bit divisions at every voxel with data: 73 us at 203x157x91 (23 MB).  Rows
// that one warp walked whatever their length took 546 us at 100000x300x1 (now 32).
constexpr unsigned kBoxRun = 4096;
__global__ void data_box_kernel(const float* __restrict__ img, const float* __restrict__ w, int nx, int ny, int nz,
                                int* box) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {-1, -1, -1};
  const unsigned segs = ((unsigned)nx + kBoxRun - 1) / kBoxRun;
  const long long items = (long long)ny * nz * segs;
  for (long long i = blockIdx.x * (long long)warps + warp; i < items; i += (long long)gridDim.x * warps) {
    const long long r = segs == 1 ? i : i / segs;
    const unsigned xs = (unsigned)(i - r * segs) * kBoxRun, xe = min((unsigned)nx, xs + kBoxRun);
    const float* pi = img + r * nx;
    const float* pw = w + r * nx;
    bool any = false;
    for (unsigned x0 = xs + lane; x0 < xe; x0 += 128) {  // unsigned: the last step may pass 2^31
      float a[4], b[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = x0 + 32 * e < xe;
        a[e] = in ? __ldg(pi + x0 + 32 * e) : 0.f;
        b[e] = in ? __ldg(pw + x0 + 32 * e) : 0.f;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (a[e] > 0.f || b[e] > 0.f) {
          any = true;
          lo[0] = min(lo[0], (int)(x0 + 32 * e));
          hi[0] = max(hi[0], (int)(x0 + 32 * e));
        }
    }
    if (any) {
      const int z = (int)(r / ny), y = (int)(r - (long long)z * ny);
      lo[1] = min(lo[1], y);
      hi[1] = max(hi[1], y);
      lo[2] = min(lo[2], z);
      hi[2] = max(hi[2], z);
    }
  }
  __shared__ int s_box[6];
  if (threadIdx.x < 6) s_box[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : -1;
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int l = __reduce_min_sync(0xffffffffu, lo[d]), h = __reduce_max_sync(0xffffffffu, hi[d]);
    if (lane == 0 && h >= 0) {
      atomicMin(s_box + d, l);
      atomicMax(s_box + 3 + d, h);
    }
  }
  __syncthreads();
  if (threadIdx.x < 6 && s_box[3] >= 0) {
    if (threadIdx.x < 3)
      atomicMin(box + threadIdx.x, s_box[threadIdx.x]);
    else
      atomicMax(box + threadIdx.x, s_box[threadIdx.x]);
  }
}

void dev_data_box(const float* img, const float* w, int nx, int ny, int nz, int* box, cudaStream_t s) {
  const long long items = (long long)ny * nz * (((unsigned)nx + kBoxRun - 1) / kBoxRun);
  const long long blocks = std::min((items + 7) / 8, 152LL * 8);  // one wave of 256 threads
  data_box_kernel<<<(int)blocks, 256, 0, s>>>(img, w, nx, ny, nz, box);
  MVD_CHECK(cudaGetLastError());
  count_launch();
}

}  // namespace mvd
