// stream2m_list.h -- the instances of k_stream2m (stream2m.cuh): X(P, NPT, A, B)
// with P pairs of a mu half, NPT list nodes per thread and the warps that one
// of an SM's four schedulers can hold of it, by its registers: A for M = 4 P,
// B with the extra slots of the M up to 4 P + 3.  The widest of a P fills 255
// registers (f takes 4 P + 3 of them per node); the narrower ones fit list
// lengths that leave it warps short of the eight an SM holds, and runs with
// few slabs.
#pragma once
#define EPREM_S2M_BINS_1(X)                                                        \
  X(1, 16, 2, 2) X(1, 8, 3, 2) X(1, 4, 4, 4) X(1, 2, 6, 5) X(2, 10, 2, 2) X(2, 8, 2, 2) \
  X(2, 4, 4, 3) X(2, 2, 5, 4)
#define EPREM_S2M_BINS_2(X)                                                        \
  X(3, 8, 2, 2) X(3, 6, 2, 2) X(3, 4, 3, 3) X(3, 2, 4, 4) X(4, 8, 2, 2) X(4, 6, 2, 2) \
  X(4, 4, 2, 2) X(4, 2, 4, 3)
#define EPREM_S2M_BINS_3(X) \
  X(5, 7, 2, 2) X(5, 5, 2, 2) X(5, 4, 2, 2) X(5, 2, 3, 3) X(6, 6, 2, 2) X(6, 5, 2, 2) X(6, 4, 2, 2)
#define EPREM_S2M_BINS_4(X) \
  X(6, 2, 3, 3) X(7, 5, 2, 2) X(7, 4, 2, 2) X(7, 3, 2, 2) X(7, 2, 3, 3) X(8, 5, 2, 2)
#define EPREM_S2M_BINS_5(X) \
  X(8, 4, 2, 2) X(8, 3, 2, 2) X(8, 2, 3, 2) X(9, 4, 2, 2) X(9, 3, 2, 2) X(9, 2, 2, 2)
#define EPREM_S2M_BINS_6(X)                                                        \
  X(10, 4, 2, 2) X(10, 3, 2, 2) X(10, 2, 2, 2) X(11, 3, 2, 2) X(11, 2, 2, 2) X(12, 3, 2, 2) \
  X(12, 2, 2, 2)
#define EPREM_S2M_BINS_7(X) \
  X(13, 3, 2, 2) X(13, 2, 2, 2) X(14, 2, 2, 2) X(15, 2, 2, 2) X(16, 2, 2, 2)
#define EPREM_S2M_PARTS(Y) Y(1) Y(2) Y(3) Y(4) Y(5) Y(6) Y(7)

namespace eprem {
// The instance of (pairs, extra slots, nodes per thread) among part k's, or null.
#define EPREM_S2M_DECL(K) const void *stream2m_kernel_##K(int P, bool extra, int npt);
EPREM_S2M_PARTS(EPREM_S2M_DECL)
#undef EPREM_S2M_DECL
}  // namespace eprem
