// Instantiations and launches of the packed inverse plane pass.
#include "engine.h"

namespace mvd {

template <class Epi>
static void launch(const ConvPlan& p, const float2* spec, const Epi& e, cudaStream_t s) {
  const PairTiles t = pair_tiles(p, TileSet::All);
  auto k = pair_inv<Epi>;
  set_smem(k, p.smem_pair);
  launch_after(k, t.n * p.tiles[0].ez, p.pair_threads, p.smem_pair, s, t.t, t.n, reinterpret_cast<const float4*>(spec),
               e, p.ps);
  count_launch();
}

void pair_inv_store(const ConvPlan& p, const float2* spec, const EpiStore& e, cudaStream_t s) {
  launch(p, spec, e, s);
}
void pair_inv_quotient(const ConvPlan& p, const float2* spec, const EpiQuotient& e, cudaStream_t s) {
  launch(p, spec, e, s);
}
void pair_inv_update(const ConvPlan& p, const float2* spec, const EpiUpdate& e, cudaStream_t s) {
  launch(p, spec, e, s);
}
void pair_inv_nll(const ConvPlan& p, const float2* spec, const EpiNll& e, cudaStream_t s) {
  launch(p, spec, e, s);
}

}  // namespace mvd
