// Instantiations and launches of the packed forward plane pass.
#include "engine.h"

namespace mvd {

template <class Gather>
static void launch(const ConvPlan& p, TileSet set, const Gather& g, float2* spec, cudaStream_t s) {
  const PairTiles t = pair_tiles(p, set);
  auto k = pair_fwd<Gather>;
  set_smem(k, p.smem_pair);
  launch_after(k, t.n * p.ps.tz, p.pair_threads, p.smem_pair, s, t.t, t.n, reinterpret_cast<float4*>(spec), g, p.ps);
  count_launch();
}

void pair_fwd_mirror(const ConvPlan& p, const float* vol, float2* spec, cudaStream_t s) {
  launch(p, TileSet::All, GatherMirror{{vol, p.vol[0], p.vol[1], p.vol[2]}}, spec, s);
}
void pair_fwd_value(const ConvPlan& p, TileSet set, const GatherValue& g, float2* spec, cudaStream_t s) {
  launch(p, set, g, spec, s);
}

}  // namespace mvd
