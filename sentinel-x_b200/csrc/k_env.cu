// Instantiations of the envelope-rescoring and region kernels, one per
// kXShapes entry's kernel.
#include "shapes.hpp"

namespace sx {

void fill_env_tables(KernelTables& t) {
  for (int s = 0; s < kNumXShapes; s++) {
    if (kXShapes[s].warps > 1) {
      t.envr[s] = sxk::env_rows_kernel<8, true, false>;
      t.regf[s] = sxk::env_rows_kernel<8, true, true>;
      t.envoa[s] = sxk::env_oa_kernel<8, true>;
    } else if (kXShapes[s].c == 8) {
      t.envr[s] = sxk::env_rows_kernel<8, false, false>;
      t.regf[s] = sxk::env_rows_kernel<8, false, true>;
      t.envoa[s] = sxk::env_oa_kernel<8, false>;
    } else {
      t.envr[s] = sxk::env_rows_kernel<4, false, false>;
      t.regf[s] = sxk::env_rows_kernel<4, false, true>;
      t.envoa[s] = sxk::env_oa_kernel<4, false>;
    }
  }
}

}  // namespace sx
