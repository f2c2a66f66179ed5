// A stand-in for the CUDA runtime on the host, for tests of the library's host
// code without a GPU: streams are queues that run only when something waits
// for them, device memory is host memory, kernels do nothing unless a test
// says what.  Copies and clears outside their device allocation abort.
#pragma once
#include <cstdint>
#include <functional>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

namespace fake {

struct Launch {
    std::string kernel;  // demangled name
    int device;
    cudaStream_t stream;
    size_t smem;
};
struct Copy {
    const void* src;
    void* dst;
    size_t bytes;
    cudaMemcpyKind kind;
};

extern std::vector<Launch> launches;
extern std::vector<Copy> copies;      // in call order
extern uint64_t memory_limit;         // bytes of device memory
extern bool reads_pageable;           // the device reads pageable memory

// what the kernels whose name contains `kernel` do: called at the launch with
// the arguments, returns what runs when the stream gets there
void on_launch(const char* kernel, std::function<std::function<void()>(void**)> f);
bool launched(const char* kernel);    // a kernel whose name contains this
int device_of(const void* p);         // the device that was current when this allocation was made

constexpr uint8_t kPoison = 0xCD;     // fresh device memory (allocations of up to 64 MiB)

}  // namespace fake
