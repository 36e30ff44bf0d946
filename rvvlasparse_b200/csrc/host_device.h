// host_device.h — RVVLA_HD marks index arithmetic that a kernel and the host
// (its CPU tests, without nvcc) both compile.
#pragma once

#ifdef __CUDACC__
#define RVVLA_HD __host__ __device__
#else
#define RVVLA_HD
#endif
