// Instantiations and launches of the packed z pass.
#include "engine.h"

namespace mvd {

// Chunks of a block: 64 chunks (8 KB rows per slice) keep the block's kernel spectrum in L2 while
// every tile reads it, and each tile's reads contiguous over the block.
constexpr int kPairZBlock = 64;

template <bool CONV>
static void launch(const ConvPlan& p, TileSet set, float2* spec, const float2* otf, float scale, cudaStream_t s) {
  const PairTiles t = pair_tiles(p, set);
  auto k = pair_z<CONV>;
  set_smem(k, p.smem_pair_z);
  launch_after(k, t.n * p.z_chunks, p.pair_z_threads, p.smem_pair_z, s, t.t, t.n, reinterpret_cast<float4*>(spec),
               reinterpret_cast<const float4*>(otf), p.ps, p.z_chunks, kPairZBlock, scale);
  count_launch();
}

void pair_z_conv(const ConvPlan& p, float2* spec, const float2* otf, cudaStream_t s) {
  launch<true>(p, TileSet::All, spec, otf, 1.f, s);
}
void pair_z_forward(const ConvPlan& p, TileSet set, float2* spec, float scale, cudaStream_t s) {
  launch<false>(p, set, spec, nullptr, scale, s);
}

}  // namespace mvd
