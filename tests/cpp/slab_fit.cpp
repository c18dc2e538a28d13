// Prints whether the fixed-point and the FP32 kernels of sigma_slab.cu fit:
// arguments norb, na, nb, alpha singles, beta singles, shared memory in bytes.
#include <cstdio>
#include <cstdlib>

#include "slab_fit.h"

int main(int argc, char **argv) {
  if (argc != 7) return 2;
  const int norb = std::atoi(argv[1]);
  sbdgb::SlabSize z{(uint32_t)std::atol(argv[2]),
                    (uint32_t)std::atol(argv[3]),
                    norb * (norb + 1) / 2,
                    {std::strtoull(argv[4], nullptr, 10), std::strtoull(argv[5], nullptr, 10)}};
  const size_t limit = std::strtoull(argv[6], nullptr, 10);
  std::printf("%d %d\n", sbdgb::slab_fits(z, 8, limit), sbdgb::slab_fits(z, 4, limit));
}
