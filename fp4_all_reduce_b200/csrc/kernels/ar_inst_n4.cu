// Narrow shapes (few rows per CTA) of the fused AllReduce kernel: four ranks, two-shot, every input kind and epilogue.
#include "ar_table.h"
namespace fp4ar {
void ar_register_n4(ArKernelEntry* out, int* n) {
  register_narrow<4, 1, 0>(out, n);
  register_narrow<4, 1, 1>(out, n);
  register_narrow<4, 1, 2>(out, n);
}
}  // namespace fp4ar
