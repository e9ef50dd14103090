// node32_b.cu -- instances of k_node32 (node32.cuh), rows of 40 to 64 registers.
#include "node32.cuh"

namespace eprem {
const void *node32_kernel_b(int P, int V) {
#define EPREM_NODE32(PP, LO)                                        \
  if (P == PP)                                                      \
    return V == 4   ? (const void *)k_node32<PP, PP, 4>             \
           : V == 2 ? (const void *)k_node32<PP, LO / 2 * 2, 2>     \
                    : (const void *)k_node32<PP, LO, 1>;
  EPREM_NODE32(40, 33)
  EPREM_NODE32(48, 41)
  EPREM_NODE32(56, 49)
  EPREM_NODE32(64, 57)
  return nullptr;
}
}  // namespace eprem
