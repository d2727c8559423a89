#pragma once
#include <cstddef>

namespace fake {
void fail_in(int n);           // the n-th allocation from now fails (0: none)
bool live(const void* p);      // allocated and not freed
size_t live_blocks();
size_t live_bytes();
extern int bad_frees;          // frees of what was not allocated
extern int device;             // the current device
extern int refused;            // launches past 48 KB of shared memory without the device's opt-in
size_t opted_in();             // kernels opted in, each device counted
}  // namespace fake
