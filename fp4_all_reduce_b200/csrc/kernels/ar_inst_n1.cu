// Narrow shapes (few rows per CTA) of the fused AllReduce kernel: one rank, every input kind and epilogue.
#include "ar_table.h"
namespace fp4ar {
void ar_register_n1(ArKernelEntry* out, int* n) {
  register_narrow<1, 0, 0>(out, n);
  register_narrow<1, 0, 1>(out, n);
}
}  // namespace fp4ar
