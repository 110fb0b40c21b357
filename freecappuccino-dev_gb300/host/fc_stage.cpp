#include "fc_stage.hpp"

namespace fcdev {

bool group_steps(const OrderedSweep& O, int G, StepGroups& V, std::vector<int>* desc) {
  V.G = G;
  V.gen = O.max_entries > FC_ELL || O.maxW > FC_SET_ROWS;
  V.nc = O.max_entries > 3 ? FC_ELL : 3;
  V.g_rows = V.g_padded = V.g_push = V.g_x = 0;
  if (desc)
    for (int d = 0; d < 2; ++d) desc[d].assign((size_t)4 * O.nsteps, 0);
  for (int d = 0; d < 2; ++d) {
    const OrderedDir& H = O.dir[d];
    for (int t = 0; t < O.ntiles; ++t) {
      const int s0 = O.tile_step_ptr[t], ns = O.tile_step_ptr[t + 1] - s0;
      for (int k0 = 0; k0 < ns; k0 += G) {
        const int k1 = std::min(k0 + G, ns), lo = s0 + (d ? ns - k1 : k0), hi = s0 + (d ? ns - k0 : k1);
        V.g_rows = std::max(V.g_rows, O.step_ptr[hi] - O.step_ptr[lo]);
        V.g_padded = std::max(V.g_padded, O.rp_ptr[hi] - O.rp_ptr[lo]);
        V.g_push = std::max(V.g_push, H.push_ptr[hi] - H.push_ptr[lo]);
        V.g_x = std::max(V.g_x, H.xv_ptr[hi] - H.xv_ptr[lo]);
        if (!desc) continue;
        for (int s = lo; s < hi; ++s) {
          int* q = desc[d].data() + 4 * (size_t)s;
          q[0] = O.step_ptr[s];
          q[1] = (O.step_ptr[s + 1] - O.step_ptr[s]) | ((H.push_ptr[s + 1] - H.push_ptr[s]) << 16);
          q[2] = (O.rp_ptr[s] - O.rp_ptr[lo]) | ((H.push_ptr[s] - H.push_ptr[lo]) << 16);
          q[3] = (O.step_ptr[s] - (O.step_ptr[lo] & ~3)) | ((H.xv_ptr[s] - H.xv_ptr[lo]) << 16);
        }
      }
    }
  }
  return V.g_rows < 65530 && V.g_padded < 65536 && V.g_push < 65536 && V.g_x < 65536;
}

int steps_per_buffer(const OrderedSweep& O, bool gs) {
  // Gauss-Seidel steps take one row per thread (their loads include the
  // upper triangle's values)
  if (gs && O.maxW > FC_SET_ROWS) return 0;
  const size_t area = ordered_stage_area(O.R, O.maxW);
  for (int G = FC_SETS; G >= 1; G /= 2) {
    StepGroups V;
    bool ok = group_steps(O, G, V, nullptr);
    for (int m = gs ? OS_GS : OS_SETUP_DIC; m <= (gs ? OS_GS : OS_BWD_DOT); ++m) {
      const int bytes = StageLayout::of<double>(V, m).bytes;
      ok = ok && (size_t)bytes <= area && stages_in(area, bytes) >= FC_SETS;
    }
    if (ok) return G;
  }
  return 0;
}

}  // namespace fcdev
