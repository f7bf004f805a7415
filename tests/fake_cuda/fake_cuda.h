// What the two halves of the host-memory CUDA runtime share (see cudart.cpp).
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <functional>

// device of a stream
int fake_stream_device(cudaStream_t s);
// counts a fault unless [p, p + bytes) lies in one live allocation of device dev
bool fake_access(const void *p, size_t bytes, int dev);
// runs a kernel launch, or adds it to the graph that this thread captures
void fake_launch(std::function<void()> kernel);
