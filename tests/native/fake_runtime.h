// Stand-ins for CUDA runtime calls, put in front of a library source by the
// compiler's -include: what a device that cannot place a launch answers.
#pragma once
#include <cuda_runtime.h>

#ifdef FAKE_REFUSED_LAUNCHES
#define cudaLaunchCooperativeKernel(...) cudaErrorCooperativeLaunchTooLarge
#endif
