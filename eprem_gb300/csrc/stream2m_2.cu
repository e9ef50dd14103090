// stream2m_2.cu -- instances of k_stream2m (stream2m.cuh), part 2.
#include "stream2m.cuh"
#include "stream2m_list.h"

namespace eprem {
const void *stream2m_kernel_2(int P, bool extra, int npt) {
#define EPREM_S2M_ONE(PP, NN, A, B)                       \
  if (P == PP && npt == NN)                               \
    return extra ? (const void *)k_stream2m<PP, true, NN> \
                 : (const void *)k_stream2m<PP, false, NN>;
  EPREM_S2M_BINS_2(EPREM_S2M_ONE)
  return nullptr;
}
}  // namespace eprem
