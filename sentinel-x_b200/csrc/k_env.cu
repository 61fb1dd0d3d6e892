// Instantiations of the envelope-rescoring and region kernels, by kXShapes entry.
#include "shapes.hpp"

namespace sx {
namespace {
template <int C, bool MULTI, sxk::TransIn IN>
void put(KernelTables& t, int s) {
  t.envr[s] = sxk::env_rows_kernel<C, MULTI, IN, false>;
  t.regf[s] = sxk::env_rows_kernel<C, MULTI, IN, true>;
  t.envoa[s] = sxk::env_oa_kernel<C, MULTI, IN>;
}
}  // namespace

void fill_env_tables(KernelTables& t) {
  for (int s = 0; s < kNumXShapes; s++) {
    if (xtrans(s) == sxk::kTrGlobal) put<16, true, sxk::kTrGlobal>(t, s);
    else if (xtrans(s) == sxk::kTrShared) put<8, true, sxk::kTrShared>(t, s);
    else if (kXShapes[s].warps > 1) put<8, true, sxk::kTrReg>(t, s);
    else if (kXShapes[s].c == 8) put<8, false, sxk::kTrReg>(t, s);
    else put<4, false, sxk::kTrReg>(t, s);
  }
  t.envins = sxk::env_insert_kernel;
}

}  // namespace sx
