// Byte offsets of complex64 points from their component's first, in 32 bits where those reach.
#pragma once
#include <stddef.h>

#ifdef __CUDACC__
#define CSEM_OFF_HD __host__ __device__ __forceinline__
#else
#define CSEM_OFF_HD static inline
#endif

namespace csem {

// of point (i, j) of a plane with rows of `width`, k planes of `plane` bytes further on
template <class Off> CSEM_OFF_HD Off point_offset(int i, int j, int k, int width, Off plane)
{
  return 8 * ((Off)i + (Off)width * j) + (Off)k * plane;
}

// whether 32 bits reach every point of the three components of an n1 x n2 x n3 grid: 2^29 points
CSEM_OFF_HD bool offsets32_reach(int n1, int n2, int n3)
{
  const double a = (double)n1 * (n2 + 1.) * (n3 + 1.), b = (n1 + 1.) * n2 * (n3 + 1.), c = (n1 + 1.) * (n2 + 1.) * n3;
  return a <= 536870912. && b <= 536870912. && c <= 536870912.;
}

}  // namespace csem
