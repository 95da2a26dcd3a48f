// Narrow shapes (few rows per CTA) of the fused AllReduce kernel: two ranks, one-shot, every input kind and epilogue.
#include "ar_table.h"
namespace fp4ar {
void ar_register_n2(ArKernelEntry* out, int* n) {
  register_narrow<2, 0, 0>(out, n);
  register_narrow<2, 0, 1>(out, n);
  register_narrow<2, 0, 2>(out, n);
}
}  // namespace fp4ar
