// fake_cudart.h — see fake_cudart.cpp.
#pragma once

#include <cuda_runtime_api.h>

#include <set>

// What comes before a stream's next launch; an event is a copy of it.
struct Stream {
  std::set<int> before;
};
inline Stream& of(cudaStream_t s) { return *reinterpret_cast<Stream*>(s); }
