// SM partitions of a device (green contexts), for launches that must be resident whole.
#pragma once
#include <cuda_runtime.h>

namespace hipress {

// SMs that a kernel on `stream` may use: all of the device's, or those of the green
// context that the stream belongs to.
int stream_sms(cudaStream_t stream, int device_sms);

}  // namespace hipress
