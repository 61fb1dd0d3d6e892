// Instantiations of the warp-per-pair Viterbi kernel, one per column width, and
// the Forward pre-screen.
#include "shapes.hpp"

#include "forward_scan.cuh"

namespace sx {
namespace {
template <int I>
struct VbinTable {
  static void fill(KernelTables& t) {
    t.vit[I] = sxk::viterbi_kernel<kVcBins[I]>;
    VbinTable<I + 1>::fill(t);
  }
};
template <>
struct VbinTable<kNumVbins> {
  static void fill(KernelTables&) {}
};
}  // namespace

void fill_vbin_tables(KernelTables& t) {
  VbinTable<0>::fill(t);
  for (int b = 0; b < kNumVbins; b++)
    t.fwd_scan[b] = scan_warps(b) > 1          ? sxk::forward_scan_kernel<true, 8>
                    : kVcBins[b] <= kScanNarrow ? sxk::forward_scan_kernel<false, 4>
                                                : sxk::forward_scan_kernel<false, 8>;
}

}  // namespace sx
