// fake_cuda.h -- a CUDA runtime in host memory, for tests of the host layer
// on machines without a GPU.  Nothing runs: allocations are tracked, copies
// are done, and a launch (of the stand-ins in fake_launch.cpp) only names the
// device pointers that its kernel would use.  A stream capture records those
// pointers and a graph launch checks them, so a graph that outlives its
// buffers shows as fake::dead_uses() > 0.
#pragma once
#include <cstddef>

namespace fake {

// device bytes that may be allocated from now on, beyond those in use
void set_free_bytes(size_t n);
// cudaMemGetInfo reports far more than that
void hide_free(bool on);
size_t bytes_in_use();
// uses of pointers into freed or unknown memory
int dead_uses();
// graphs recorded, graphs launched
int captures();
int graph_launches();
// a kernel launch on stream s that uses p
void use(const void *p, void *s);

}  // namespace fake
