// A stand-in for the CUDA runtime, to run the library's host code without a
// GPU: device memory is host memory, kernels do nothing, and the work of all
// streams runs in the order of its calls, but only when the host waits for
// something.  An asynchronous copy so reads its source as late as a stream may;
// a source that has been freed or changed by then is reported.
#pragma once

namespace fake {

// Runs all queued work (what a wait on the host does).
void run_queued();
// Copies that found their source other than when they were issued.
long long stale_sources();
// The n-th call from now that launches a kernel fails (n = 0: none does).
void fail_launch(long long n);
long long launches();  // kernel launches so far
// Device allocations above this many bytes fail for want of memory.
void limit_allocations(unsigned long long bytes);

}  // namespace fake
