// Instantiations of the exact row passes, one per kXShapes entry's kernel.
#include "exact_rows.cuh"
#include "shapes.hpp"

namespace sx {

void fill_exact_tables(KernelTables& t) {
  for (int s = 0; s < kNumXShapes; s++)
    t.xrows[s] = kXShapes[s].warps > 1 ? sxk::exact_rows_kernel<8, true>
                 : kXShapes[s].c == 8  ? sxk::exact_rows_kernel<8, false>
                                       : sxk::exact_rows_kernel<4, false>;
}

}  // namespace sx
