// Shared memory of the kernels of sigma_slab.cu, and whether a problem's fits.
//
// The forms need different amounts for the same problem: the 8-byte ones (FP64,
// double-float) can take one column a CTA and, where a row's alpha x beta sums are
// not kept, two ket rows; the FP32 kernels take at least four of each (16 bytes a
// row) and always keep the sums.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace sbdgb {

struct SlabSize {
  uint32_t na, nb;
  int npair;
  uint64_t ns[2];  // singles of the alpha and of the beta tables
  bool ab() const { return ns[0] > 0 && ns[1] > 0; }
  // Whether a row's alpha x beta sums stay in shared memory between batches: not
  // where rows have a batch or two.
  bool ab_sum() const { return (double)ns[0] * (double)ns[1] >= 8.0 * (double)na * (double)nb; }
};

constexpr int kSlabMinK = 1, kSlabMinKF = 4;  // fewest columns a CTA: 8-byte elements, FP32

// The sweep over a spin with n strings: K columns and the Coulomb values.
inline size_t slab_smem_bytes(int element, int K, uint32_t n, int npair) {
  return (size_t)element * K * ((size_t)n + 1 + (npair ? (size_t)npair + 1 : 0));
}
// Alpha x beta: G ket rows, their (P|Q) values with both signs, the row's sums.
inline size_t slab_ab_smem_bytes(uint32_t nb, int npair, int G, bool sum) {
  return 8ull * G * ((size_t)nb + 1 + 2 * ((size_t)npair + 1)) + (sum ? 8ull * nb : 0);
}
inline size_t slab_ab_smem_bytes_f32(uint32_t nb, int npair) {
  return 16ull * ((size_t)nb + 1 + 2 * ((size_t)npair + 1)) + 4ull * nb;
}

// Whether the kernels of a form (element: 8 or 4 bytes) fit in `limit` bytes.
inline bool slab_fits(const SlabSize &z, int element, size_t limit) {
  if (element == 8)
    return slab_smem_bytes(8, kSlabMinK, std::max(z.na, z.nb), z.npair) <= limit &&
           (!z.ab() || slab_ab_smem_bytes(z.nb, z.npair, 2, z.ab_sum()) <= limit);
  for (int sp = 0; sp < 2; ++sp)
    if (slab_smem_bytes(4, kSlabMinKF, sp == 0 ? z.na : z.nb, z.ns[sp] ? z.npair : 0) > limit) return false;
  return !z.ab() || slab_ab_smem_bytes_f32(z.nb, z.npair) <= limit;
}

}  // namespace sbdgb
