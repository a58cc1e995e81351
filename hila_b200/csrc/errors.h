// Error reporting of the C ABI: a status code and a message per thread.
#pragma once

#include <cuda_runtime.h>

#include "../../include/hila_b200.h"

namespace hw {

void set_error(const char *fmt, ...);
void clear_error();

#define HW_CHECK_ARG(cond, ...)              \
    do {                                     \
        if (!(cond)) {                       \
            ::hw::set_error(__VA_ARGS__);    \
            return HW_ERR_INVALID;           \
        }                                    \
    } while (0)

#define HW_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            ::hw::set_error("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return e_ == cudaErrorMemoryAllocation ? HW_ERR_OOM : HW_ERR_CUDA;                     \
        }                                                                                          \
    } while (0)

}  // namespace hw
