// node32_a.cu -- instances of k_node32 (node32.cuh), rows of 8 to 32 registers.
#include "node32.cuh"

namespace eprem {
const void *node32_kernel_a(int P, int V) {
#define EPREM_NODE32(PP, LO)                                        \
  if (P == PP)                                                      \
    return V == 4   ? (const void *)k_node32<PP, PP, 4>             \
           : V == 2 ? (const void *)k_node32<PP, LO / 2 * 2, 2>     \
                    : (const void *)k_node32<PP, LO, 1>;
  EPREM_NODE32(8, 2)
  EPREM_NODE32(16, 9)
  EPREM_NODE32(20, 17)
  EPREM_NODE32(24, 21)
  EPREM_NODE32(32, 25)
  return nullptr;
}
}  // namespace eprem
