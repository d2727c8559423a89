#pragma once
#include <cstddef>

namespace fake {
void fail_in(int n);           // the n-th allocation from now fails (0: none)
bool live(const void* p);      // allocated and not freed
size_t live_blocks();
size_t live_bytes();
extern int bad_frees;          // frees of what was not allocated
}  // namespace fake
