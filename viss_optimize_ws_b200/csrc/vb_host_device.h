// Marks a function of a plain header that kernels call too.
#pragma once

#ifdef __CUDACC__
#define VB_HOST_DEVICE __host__ __device__
#else
#define VB_HOST_DEVICE
#endif
