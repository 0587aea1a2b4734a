// A CUDA runtime of host functions for tests of host code: streams are queues that
// run when something waits for them (or, with `device_runs`, when an event is
// queried), device memory is host memory.
#pragma once
#include <driver_types.h>

#include <functional>
#include <mutex>

namespace fake {
extern std::recursive_mutex mu;   // held by every call below and by the runtime's
extern bool device_runs;          // work gets done while events are queried
extern int fail_queries;          // event queries that report an error
extern bool capturing;            // a thread captures in the global mode
extern int refused;               // calls refused because of it
extern int frees_while_busy;      // frees of device memory while a stream had work
void enqueue(cudaStream_t s, std::function<void()> f);
int busy();                       // streams with work
}  // namespace fake
