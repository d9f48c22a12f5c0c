// Shared by fake_runtime.cpp and fake_units.cu.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdint>

namespace fake {
void on_device(const void* p, const char* where);  // memory of the device that is current
void launched(cudaStream_t st);
void traced(uint64_t photons);
double record_rate(int channel);
double query_rate(int kind);
int trace_error();  // the code that the next trace leaves on the device (0: none), once
}  // namespace fake
