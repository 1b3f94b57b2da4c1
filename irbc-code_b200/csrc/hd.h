// hd.h -- functions of the device code that plain C++ compiles too, so that
// they are tested on the host.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define IRBC_HD __host__ __device__ __forceinline__
#else
#define IRBC_HD inline
#endif
