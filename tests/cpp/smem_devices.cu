// The shared-memory opt-in of the adjoint columns on the host (fake_cudart.cpp), with two
// devices: every device that launches the kernel has to have been asked for, once.
#include <cstdio>

#include "fake_cudart.h"
#include "inst.cuh"

int main() {
  constexpr int L = 512;
  static_assert(gbn::AdjColsShape<L, false>::BYTES > 48 * 1024, "the length needs the opt-in");
  const float2* S = reinterpret_cast<const float2*>(16);  // not read
  for (int pass = 0; pass < 2; ++pass)
    for (fake::device = 0; fake::device < 2; ++fake::device)
      gbn::Launchers<L>::adj_cols(nullptr, S, nullptr, 24, 1, 1, 1.f, nullptr, 1, nullptr);
  std::printf("%d launches refused, %zu opt-ins\n", fake::refused, fake::opted_in());
  return fake::refused != 0 || fake::opted_in() != 2;
}
