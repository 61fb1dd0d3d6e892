// Instantiations of the exact row passes and of the wide profiles' MSV and
// Viterbi, by kXShapes entry.
#include "shapes.hpp"

namespace sx {

using namespace sxk;

void fill_exact_tables(KernelTables& t) {
  for (int s = 0; s < kNumXShapes; s++) {
    const bool shared = xtrans(s) == kTrShared;
    t.xrows[s] = xtrans(s) == kTrGlobal ? exact_rows_kernel<16, true, kTrGlobal>
                 : shared               ? exact_rows_kernel<8, true, kTrShared>
                 : kXShapes[s].warps > 1 ? exact_rows_kernel<8, true, kTrReg>
                 : kXShapes[s].c == 8   ? exact_rows_kernel<8, false, kTrReg>
                                        : exact_rows_kernel<4, false, kTrReg>;
    const bool wide = kXShapes[s].warps > 8;
    t.wmsv[s] = !wide ? nullptr : shared ? wide_msv_kernel<8> : wide_msv_kernel<16>;
    t.wvit[s] = !wide ? nullptr : shared ? wide_viterbi_kernel<8, kTrShared> : wide_viterbi_kernel<16, kTrGlobal>;
  }
}

}  // namespace sx
