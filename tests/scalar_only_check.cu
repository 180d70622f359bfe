// The passes that exist for scalar plans only, called with a pair plan (host code; nothing is launched:
// each has to throw std::logic_error first).  Prints what was not refused and exits non-zero.
#include <cstdio>

#include "../spim_registration_gb300/csrc/engine.h"

using namespace mvd;

int main() {
  PlanTable pt;
  ConvPlan p;
  p.paired = true;
  p.tiles.push_back(TileDesc{});
  int wrong = 0;
  auto refused = [&](const char* what, auto call) {
    try {
      call();
      std::printf("%s: returned\n", what);
    } catch (const std::logic_error& e) {
      return;
    } catch (const std::exception& e) {
      std::printf("%s: %s\n", what, e.what());
    }
    ++wrong;
  };
  refused("launch_fwd_masked", [&] { launch_fwd_masked(pt, p, nullptr, nullptr, nullptr); });
  refused("launch_z_inverse", [&] { launch_z_inverse(pt, p, TileSet::Full, nullptr, nullptr); });
  refused("launch_inv_store_tiles",
          [&] { launch_inv_store_tiles(pt, p, TileSet::Full, nullptr, nullptr, 1, 1, nullptr); });
  refused("dev_cross_accumulate", [&] { dev_cross_accumulate(p, nullptr, nullptr, nullptr, nullptr); });
  return wrong;
}
