// sigma = H*C with the pair sums in fixed point and the gathered vector in
// shared memory (FP64 products; replaces sbd::mult, chemistry/tpb/mult.h:
// 440-558, like the kernels of sigma.cu, for problems with many nonzeros a row).
//
// What bounds it.  The kernels of sigma.cu spend one FP64 multiply-add per
// nonzero and keep the FP64 pipe (2 a clock and SM) 89-91% busy.  Here a
// nonzero costs three 32 x 32 + 64-bit integer multiply-adds (fx.cuh; 19 a
// clock and SM), and its gather comes from shared memory instead of L2.  ncu on
// 3274 x 3935 strings (norb 24, 245 pairs a row), alpha sweep, alpha x beta, beta
// sweep: L1 data pipe 74, 85 and 70% busy, the pipe of the multiply-adds 70, 56 and
// 67%, shared loads at 1.24, 1.70 and 1.22 wavefronts per 8 lanes, FP64 pipe at most
// 4%.
//
// Measured (one product in the reference's convention, ms; FP64 kernels, here):
// norb 12, 161 x 187: 0.374, 0.091; norb 16, 800 x 800: 1.91, 0.72; norb 24,
// 3274 x 3935: 18.3, 8.2 (sweeps 1.8 and 2.1, alpha x beta 4.2); norb 36, 6000 x
// 6000: 6.6, 3.8 (1.4, 1.4 and 0.9).  Error against FP64 sums of the
// off-diagonal part kept apart from the diagonal (2-norm): 0.7-1.1e-16, where
// the FP64 kernels have 3e-16 to 1.3e-15.
//
// k_slab (same-spin pairs; task types 1 and 2).  The sweep over one spin's
// pairs never mixes columns (the opposite-spin index), so a CTA takes K
// columns and stages all n rows of them (8 K n bytes: 192 KB at K = 4, n =
// 6000).  Staging finds each column's largest |C|, which sets the column's
// fixed-point scale, and converts in place.  Then a lane owns a row: per pair
// it reads (ket, V) once, coalesced, and K staged values, and adds K terms.
// Rows are sorted by their number of doubles and cut into slices of 32 that
// the warps take in turn (longest first); a slice's lists are interleaved by
// lane in groups of four and padded to its longest (the sliced ELLPACK form)
// with entries that point at a zero row.  The beta sweep stages K rows of C
// (contiguous) and needs no transposed copy; the alpha sweep stages K columns
// (32-byte pieces at K = 4).  The alpha sweep and the alpha x beta pairs come
// first; the beta sweep adds the diagonal, the largest term, while it stages, so
// that the others' sums are not rounded at its size, and its own sums with one
// reduction per element (fire and forget; the order of an element's sum is that
// of the launches).
//
// Phases.  Both sweeps and k_slab_ab work in the block ordering (no
// opposite-spin parity; sigma_dev.cuh).  For the reference's interleaved
// convention the sign eta of each determinant is applied while staging and
// again to the result: two popcounts per determinant instead of one or two per
// nonzero.
//
// A column (or ket row) with an infinity, a NaN or values beyond 2^+-800, and in
// the caller's products one whose values lie far apart (Format), is summed in
// floating point from the values as they are, bound by the FP64 pipe as the kernels
// of sigma.cu are.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <type_traits>

#include "common.cuh"
#include "fx.cuh"
#include "sigma_dev.cuh"
#include "slab_fit.h"

namespace sbdgb {

namespace {

using namespace sdev;

constexpr int kSlabThreads = 768, kSlabAbThreads = 512;
constexpr int kGroup = 4;  // table entries of a lane that are read together
constexpr uint32_t kSlabMaxRows = 1u << 15;  // ket index bits of a packed single
constexpr uint32_t kSlabMaxPair = 1u << 12;  // pair index bits

// ---- the vector formats ----------------------------------------------------------

// key: monotone in |x|, 0 for 0 only; exponent(key): |x| < 2^exponent (fx.cuh).
// Staged as they are (raw, of), and after parts() in fixed point, both 8 bytes.
//
// Wide vectors (a.guard).  An element is held to 2^-56 of the largest of its sum,
// so what only small elements feed is held to fewer bits than floating point keeps:
// with weights over 12 decades on the strings of each spin (norb 24, 700 x 733) 1%
// of sigma's elements were off by 6e-9 of their terms' magnitudes or more, FP64 sums
// by 1e-15; with 3 decades no element is off by more than the FP64 sums' worst, and
// the norm of the error is a fifth of theirs.  So a column (ket row) goes by
// floating-point sums where its nonzeros lie on average more than kWide binary
// orders below its largest, or any more than kTiny (kRows: below).  (3 decades of weights and
// normal variates: 7 orders on average, 8.4 at most, hardly one beyond 36; 4
// decades: 8.9.)
template <typename T>
struct Format;
template <>
struct Format<double> {
  static __device__ __forceinline__ uint32_t key(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return hi ? hi : (__double2loint(x) ? 1u : 0u);
  }
  static __device__ __forceinline__ int exponent(uint32_t key) { return fx::exponent_of(key, key != 0u); }
  static __device__ __forceinline__ int2 raw(double x) { return make_int2(__double2loint(x), __double2hiint(x)); }
  static __device__ __forceinline__ double of(int2 v) { return __hiloint2double(v.y, v.x); }
  static constexpr int kField = 20;  // key >> kField: the exponent's field
  static constexpr int kWide = 9, kTiny = 36, kRows = 13;
  static __device__ __forceinline__ double table(int lo, int hi) { return __hiloint2double(hi, lo); }
  static __device__ __forceinline__ int2 parts(int2 v, int ex) {
    return fx::vector_parts((uint32_t)v.x, (uint32_t)v.y, ex);
  }
  static __device__ __forceinline__ double value(const fx::Acc &a, int e) { return fx::value(a, e); }
};
template <>
struct Format<dfloat> {
  static __device__ __forceinline__ uint32_t key(dfloat x) {
    return __float_as_uint(fabsf(x.hi) + fabsf(x.lo));  // a NaN is above every number
  }
  static __device__ __forceinline__ int exponent(uint32_t key) {
    return key == 0u ? fx::kZero : key >= 0x7f800000u ? fx::kBad : (int)(key >> 23) - 126;
  }
  static __device__ __forceinline__ int2 raw(dfloat x) { return make_int2(__float_as_int(x.lo), __float_as_int(x.hi)); }
  static __device__ __forceinline__ dfloat of(int2 v) { return dfloat(__int_as_float(v.y), __int_as_float(v.x)); }
  static constexpr int kField = 23;
  static constexpr int kWide = 15, kTiny = 42, kRows = 19;  // five bits fewer to keep than in FP64
  // An FP64 table value: 24 bits in hi, the other 29 in lo (no FP64 instruction).
  static __device__ __forceinline__ dfloat table(int lo, int hi) {
    const int e = (hi >> 20) & 0x7ff, sign = hi & (int)0x80000000;
    if (e < 1023 - 70 || e > 1023 + 126) return e ? dfloat(__hiloint2double(hi, lo)) : dfloat(0.f, 0.f);
    const int h = sign | (e - 896) << 23 | (hi & 0xfffff) << 3 | (int)((uint32_t)lo >> 29);
    const float unit = __int_as_float(sign | (e - 948) << 23);  // 2^(e - 1075)
    return dfloat(__int_as_float(h), (float)(lo & 0x1fffffff) * unit);
  }
  static __device__ __forceinline__ int2 parts(int2 v, int ex) {
    return fx::vector_parts_df((uint32_t)v.x, (uint32_t)v.y, ex);
  }
  static __device__ __forceinline__ dfloat value(const fx::Acc &a, int e) { return fx::value_df(a, e); }
};

// How a lane adds to sigma.  FP64: one reduction per element (each element once
// per launch, so the order of the sum is that of the launches).  FP32 and
// double-float: what sigma holds is loaded before the lists are summed, so that
// the loads do not stall the end of a slice, and stored with the sum (no other
// lane of the launch touches it).
template <typename T>
constexpr bool kReduce = std::is_same<T, double>::value;
__device__ __forceinline__ void add_to(double *s, double, double x) { atomicAdd(s, x); }
__device__ __forceinline__ void add_to(dfloat *s, dfloat old, dfloat x) { *s = old + x; }

// The K (4 or 8: 32 bytes) neighbouring elements of one row in 16-byte pieces.
template <int K, typename T>
__device__ __forceinline__ void load_row(const T *p, T (&x)[K]) {
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
  uint4 u[sizeof(T) * K / 16];
#pragma unroll
  for (size_t i = 0; i < sizeof(T) * K / 16; ++i) u[i] = q[i];
  memcpy(x, u, sizeof(T) * K);
}
template <int K, typename T>
__device__ __forceinline__ void store_row(T *p, const T (&x)[K]) {
  uint4 u[sizeof(T) * K / 16];
  memcpy(u, x, sizeof(T) * K);
#pragma unroll
  for (size_t i = 0; i < sizeof(T) * K / 16; ++i) reinterpret_cast<uint4 *>(p)[i] = u[i];
}

// ---- the sweep over one spin's pairs -----------------------------------------------

struct SlabSpin {
  const uint32_t *rows;           // 32 per slice; ~0u pads the last
  const uint32_t *off_s, *off_d;  // per slice: first group of its singles and doubles
  const uint4 *ent_s;             // singles: ket << 4 | pair << 19 | phase << 31
  const int4 *val_s;              // V of the same-spin part with the phase applied
  const uint4 *ket_d;             // doubles: ket << 4
  const int4 *val_d;
  const int4 *fp_s, *fp_d;        // V in FP64 (the pairs of words that val_* has in fixed point), or null
  uint32_t nslices;
};

template <typename T>
struct SlabArgs {
  const T *C;
  T *S;
  const T *hii;  // the diagonal in the vectors' format
  T shift;       // taken off the diagonal (0 in FP64)
  SlabSpin t;
  const double *Jo;         // opposite-spin Coulomb table [npair][m]
  const T *Jt;              // the same in the vectors' format
  const int2 *Jfx;          // the same in fixed point, or null: converted here
  const uint64_t *rowstr;   // this spin's strings
  const uint64_t *colmask;  // per column: the orbitals whose parity on rowstr is eta
  uint32_t n, m, nb;        // rows (this spin), columns (the other spin), row length of C and S
  int npair;                // 0: no singles (J is not staged)
  int ev;                   // |v| < 2^ev for every table value of this spin
  int eta;                  // interleaved convention: eta on the way in and out
  int guard;                // wide columns are summed in floating point
  int add;                  // what S holds is kept
  int diag;                 // the diagonal term is added here
  int staged_diag;          // ... while staging, so that S is complete but for this spin's sums
  int vec;                  // rows of S start on 16-byte boundaries
  uint32_t parts;           // CTAs that share a column group (gridDim.y)
};

// Staged values: K columns, two of a row side by side (16 bytes) in planes of
// `rows` rows, so that a lane reads two columns with one load.
template <int K>
__device__ __forceinline__ size_t staged(uint32_t rows, uint32_t r, int c) {
  return K == 1 ? r : ((size_t)(c >> 1) * rows + r) * 2 + (c & 1);
}

// How far apart a sum's elements lie, from their keys: in shared memory the largest
// key, the smallest of a nonzero less 1, the number of nonzeros and the sum of their
// exponents' fields.
struct Keys {
  uint32_t top, low, nonzero, fields;
};
template <typename T>
struct Spread {
  uint32_t top = 0u, low = ~0u, nonzero = 0u, fields = 0u;
  __device__ __forceinline__ void count(T x, int guard) {
    const uint32_t key = Format<T>::key(x);
    top = max(top, key);
    if (guard) {
      low = min(low, key - 1u);
      nonzero += key != 0u;
      fields += key >> Format<T>::kField;
    }
  }
  // Adds the counts of every `step`-th lane to `at`.
  __device__ __forceinline__ void add_to(Keys *at, int guard, int step = 1) {
    const bool one = (threadIdx.x & 31u) < (uint32_t)step;
    if (step == 1) {
      top = __reduce_max_sync(0xffffffffu, top);
      if (guard) {
        low = __reduce_min_sync(0xffffffffu, low);
        nonzero = __reduce_add_sync(0xffffffffu, nonzero);
        fields = __reduce_add_sync(0xffffffffu, fields);
      }
    } else {
      for (int o = 16; o >= step; o >>= 1) {
        top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        if (guard) {
          low = min(low, __shfl_xor_sync(0xffffffffu, low, o));
          nonzero += __shfl_xor_sync(0xffffffffu, nonzero, o);
          fields += __shfl_xor_sync(0xffffffffu, fields, o);
        }
      }
    }
    if (one) atomicMax(&at->top, top);
    if (one && guard) {
      atomicMin(&at->low, low);
      atomicAdd(&at->nonzero, nonzero);
      atomicAdd(&at->fields, fields);
    }
  }
  static __device__ __forceinline__ bool wide(const Keys &k) {
    const uint32_t top = k.top >> Format<T>::kField, low = (k.low + 1u) >> Format<T>::kField;
    return k.nonzero && (top - low > (uint32_t)Format<T>::kTiny ||
                         k.nonzero * top - k.fields > k.nonzero * (uint32_t)Format<T>::kWide);
  }
};

// Four table entries of a lane: three 16-byte loads.
struct Group {
  uint4 w;
  int4 v0, v1;
  __device__ __forceinline__ void load(const uint4 *__restrict__ ent, const int4 *__restrict__ val, uint32_t at) {
    w = ldg(ent + at);
    v0 = __ldg(val + 2 * at);
    v1 = __ldg(val + 2 * at + 1);
  }
};

template <int K, bool kSingles>
__device__ __forceinline__ void slab_group(fx::Acc (&acc)[K], const Group &g, const char *X, uint32_t xplane,
                                           const char *J, uint32_t jplane) {
  constexpr int NQ = (K + 1) / 2;
  const uint32_t w[kGroup] = {g.w.x, g.w.y, g.w.z, g.w.w};
  const int vh[kGroup] = {g.v0.x, g.v0.z, g.v1.x, g.v1.z}, vl[kGroup] = {g.v0.y, g.v0.w, g.v1.y, g.v1.w};
#pragma unroll
  for (int u = 0; u < kGroup; ++u) {
    const uint32_t x16 = kSingles ? w[u] & 0x7fff0u : w[u], j16 = (w[u] >> 15) & 0xfff0u;
    const int sg = (int)w[u] >> 31;  // singles, -1: the Coulomb part is subtracted
    if constexpr (K == 1) {
      const int2 x = *reinterpret_cast<const int2 *>(X + (x16 >> 1));
      if constexpr (kSingles) {
        const int2 j = *reinterpret_cast<const int2 *>(J + (j16 >> 1));
        fx::mac(acc[0], x.x, x.y, vh[u] + ((j.x ^ sg) - sg), vl[u] + ((j.y ^ sg) - sg));
      } else {
        fx::mac(acc[0], x.x, x.y, vh[u], vl[u]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int4 x = *reinterpret_cast<const int4 *>(X + q * xplane + x16);
        if constexpr (kSingles) {
          const int4 j = *reinterpret_cast<const int4 *>(J + q * jplane + j16);
          fx::mac(acc[2 * q], x.x, x.y, vh[u] + ((j.x ^ sg) - sg), vl[u] + ((j.y ^ sg) - sg));
          fx::mac(acc[2 * q + 1], x.z, x.w, vh[u] + ((j.z ^ sg) - sg), vl[u] + ((j.w ^ sg) - sg));
        } else {
          fx::mac(acc[2 * q], x.x, x.y, vh[u], vl[u]);
          fx::mac(acc[2 * q + 1], x.z, x.w, vh[u], vl[u]);
        }
      }
    }
  }
}

// Adds one slice's singles or doubles to the lane's K sums, two groups a turn:
// each is requested before the other is summed.
template <int K, bool kSingles>
__device__ __forceinline__ void slab_list(fx::Acc (&acc)[K], const uint4 *__restrict__ ent,
                                          const int4 *__restrict__ val, uint32_t g, uint32_t end, uint32_t lane,
                                          const char *X, uint32_t xplane, const char *J, uint32_t jplane) {
  static_assert(fx::kChunkHigh == 4 * kGroup && fx::kChunk == 8 * kGroup, "carries every 4 and 8 groups");
  if (g >= end) return;
  uint32_t at = g * 32u + lane, left = end - g, turn = 0;
  Group a, b;
  a.load(ent, val, at);
  while (true) {
    if (left > 1) b.load(ent, val, at + 32u);
    slab_group<K, kSingles>(acc, a, X, xplane, J, jplane);
    if (left == 1) break;
    if (left > 2) a.load(ent, val, at + 64u);
    slab_group<K, kSingles>(acc, b, X, xplane, J, jplane);
    if (left == 2) break;
    left -= 2;
    at += 64u;
    ++turn;
    if ((turn & 3u) == 0u) {
#pragma unroll
      for (int c = 0; c < K; ++c) fx::carry(acc[c]);
    } else if ((turn & 1u) == 0u) {
#pragma unroll
      for (int c = 0; c < K; ++c) fx::carry_high(acc[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < K; ++c) fx::carry(acc[c]);
}

// The same from the raw staged values (X, and J the raw Coulomb values), in the
// vectors' format.  Where there are no FP64 values (fp null: a solve that met a
// vector which is not finite) they come from the fixed-point ones, |v| < 2^ev.
template <typename T, int K, bool kSingles>
__device__ __forceinline__ void slab_list_fp(T (&acc)[K], const uint4 *__restrict__ ent, const int4 *__restrict__ fp,
                                             const int4 *__restrict__ fixed, int ev, uint32_t g, uint32_t end,
                                             uint32_t lane, const char *X, uint32_t xplane, const char *J,
                                             uint32_t jplane) {
  using F = Format<T>;
  if (g >= end) return;
  const uint32_t pad = xplane - 16u;  // the zero row, which padding entries point at
  const int4 *val = fp ? fp : fixed;
  auto value = [&](int x, int y) {
    return fp ? F::table(x, y) : T(scalbn((double)x * (double)(1 << fx::kLow) + (double)y, ev - fx::kVBits));
  };
  Group a;
  a.load(ent, val, g * 32u + lane);
  while (true) {
    const Group b = a;
    if (g + 1 < end) a.load(ent, val, (g + 1) * 32u + lane);
    const uint32_t w[kGroup] = {b.w.x, b.w.y, b.w.z, b.w.w};
    const T v[kGroup] = {value(b.v0.x, b.v0.y), value(b.v0.z, b.v0.w), value(b.v1.x, b.v1.y),
                         value(b.v1.z, b.v1.w)};
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const uint32_t x16 = kSingles ? w[u] & 0x7fff0u : w[u], j16 = (w[u] >> 15) & 0xfff0u;
      if (!__any_sync(0xffffffffu, x16 != pad)) break;  // the rest of the group is padding in every lane
      const uint32_t sg = w[u] >> 31;
      if constexpr (K == 1) {
        T m = v[u];
        if constexpr (kSingles) m = m + flip(F::of(*reinterpret_cast<const int2 *>(J + (j16 >> 1))), sg);
        acc[0] = fma(m, F::of(*reinterpret_cast<const int2 *>(X + (x16 >> 1))), acc[0]);
      } else {
#pragma unroll
        for (int q = 0; q < K / 2; ++q) {
          const int4 x = *reinterpret_cast<const int4 *>(X + q * xplane + x16);
          T m0 = v[u], m1 = v[u];
          if constexpr (kSingles) {
            const int4 j = *reinterpret_cast<const int4 *>(J + q * jplane + j16);
            m0 = m0 + flip(F::of(make_int2(j.x, j.y)), sg);
            m1 = m1 + flip(F::of(make_int2(j.z, j.w)), sg);
          }
          acc[2 * q] = fma(m0, F::of(make_int2(x.x, x.y)), acc[2 * q]);
          acc[2 * q + 1] = fma(m1, F::of(make_int2(x.z, x.w)), acc[2 * q + 1]);
        }
      }
    }
    if (++g == end) return;
  }
}

// One CTA: column group `group`, every a.parts-th slice from `part`, of C into S.
template <typename T, int K, bool kAlpha>
__device__ __forceinline__ void slab_cta(const SlabArgs<T> &a, const T *__restrict__ C, T *S, uint32_t group,
                                         uint32_t part) {
  using F = Format<T>;
  constexpr int NQ = (K + 1) / 2;
  extern __shared__ __align__(16) unsigned char slab_smem[];
  int2 *X = reinterpret_cast<int2 *>(slab_smem);     // (n + 1) x K; row n is zero (padding entries)
  int2 *J = X + (size_t)(a.n + 1) * K;               // (npair + 1) x K; row npair is zero
  __shared__ Keys skey[K];
  __shared__ uint32_t snext;
  const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u;
  const uint32_t c0 = group * K;
  constexpr int kw = K == 1 ? 1 : 2;  // columns side by side in a plane of X
  const uint32_t plane = (a.n + 1) * kw;
  auto diag = [&](size_t k) {
    if constexpr (std::is_same<T, double>::value)
      return ldg(a.hii + k);
    else
      return ldg(a.hii + k) - a.shift;
  };
  if (tid < K) skey[tid] = Keys{0u, ~0u, 0u, 0u};
  if (tid == 0) snext = 0u;
  __syncthreads();
  // stage the raw values and find each column's largest
  if constexpr (kAlpha) {
    const int c = (int)(tid % K);
    const bool ok = c0 + c < a.m;
    const uint64_t mask = ok && a.eta ? ldg(a.colmask + c0 + c) : 0ull;
    Spread<T> keys;
    for (uint32_t r = tid / K; r < a.n; r += nt / K) {
      T x = ok ? ldg(C + (size_t)r * a.nb + (c0 + c)) : T(0.0);
      if (a.eta) x = flip(x, parity((unsigned long long)(mask & ldg(a.rowstr + r))));
      keys.count(x, a.guard);
      X[staged<K>(a.n + 1, r, c)] = F::raw(x);
    }
    keys.add_to(&skey[c], a.guard, K);
  } else {
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const bool ok = c0 + c < a.m;
      const uint64_t mask = ok && a.eta ? ldg(a.colmask + c0 + c) : 0ull;
      const T *row = C + (size_t)(c0 + c) * a.nb;
      Spread<T> keys;
      for (uint32_t r = tid; r < a.n; r += nt) {
        T x = ok ? ldg(row + r) : T(0.0);
        if (a.staged_diag && ok) {
          const size_t k = (size_t)(c0 + c) * a.nb + r;
          S[k] = a.add ? fma(diag(k), x, S[k]) : diag(k) * x;
        }
        if (a.eta) x = flip(x, parity((unsigned long long)(mask & ldg(a.rowstr + r))));
        keys.count(x, a.guard);
        X[staged<K>(a.n + 1, r, c)] = F::raw(x);
      }
      keys.add_to(&skey[c], a.guard);
    }
  }
  if (tid < K) X[staged<K>(a.n + 1, a.n, tid)] = make_int2(0, 0);
  if (a.npair) {
    for (uint32_t i = tid; i < (uint32_t)(a.npair + 1) * K; i += nt) {
      const uint32_t P = i / K;
      const int c = (int)(i % K);
      const bool ok = P < (uint32_t)a.npair && c0 + c < a.m;
      const size_t from = (size_t)P * a.m + (c0 + c);
      J[staged<K>(a.npair + 1, P, c)] = !ok       ? make_int2(0, 0)
                                        : a.Jfx ? __ldg(a.Jfx + from)
                                                : fx::make(ldg(a.Jo + from), fx::kVBits - a.ev);
    }
  }
  __syncthreads();
  int ex[K];
  bool bad = false;
#pragma unroll
  for (int c = 0; c < K; ++c) {
    ex[c] = F::exponent(skey[c].top);
    bad = bad || ex[c] == fx::kBad || (a.guard && Spread<T>::wide(skey[c]));
  }
  if (!bad) {  // to fixed point, in place (an all-zero column has no scale and its sums are not read)
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      for (uint32_t i = tid; i < plane; i += nt) {
        const int e = K == 1 || !(i & 1u) ? ex[q * kw] : ex[q * kw + kw - 1];
        int2 &x = X[(size_t)q * plane + i];
        if (e != fx::kZero) x = F::parts(x, e);
      }
  } else {  // the Coulomb values as they are too
    for (uint32_t i = tid; i < (uint32_t)a.npair * K; i += nt) {
      const uint32_t P = i / K;
      const int c = (int)(i % K);
      if (c0 + c < a.m) J[staged<K>(a.npair + 1, P, c)] = F::raw(ldg(a.Jt + ((size_t)P * a.m + (c0 + c))));
    }
  }
  __syncthreads();
  const SlabSpin &t = a.t;
  while (true) {
    uint32_t sl = 0;
    if (lane == 0) sl = atomicAdd(&snext, 1u);
    sl = part + a.parts * __shfl_sync(0xffffffffu, sl, 0);
    if (sl >= t.nslices) break;
    const uint32_t row = ldg(t.rows + sl * 32u + lane);
    auto element = [&](int c) { return kAlpha ? (size_t)row * a.nb + (c0 + c) : (size_t)(c0 + c) * a.nb + row; };
    const bool add = a.add || a.staged_diag;
    const bool whole = kAlpha && K == 4 && a.vec && c0 + K <= a.m && !(kReduce<T> && add);  // 16-byte pieces
    T out[K], old[K];
    if (!kReduce<T> && add && row != ~0u) {
      if (whole) {
        if constexpr (K == 4) load_row<K>(S + element(0), old);
      } else {
#pragma unroll
        for (int c = 0; c < K; ++c)
          if (c0 + c < a.m) old[c] = S[element(c)];
      }
    }
    if (!bad) {
      fx::Acc acc[K];
#pragma unroll
      for (int c = 0; c < K; ++c) fx::zero(acc[c]);
      const uint32_t xplane = 16u * (a.n + 1), jplane = 16u * (a.npair + 1);
      slab_list<K, true>(acc, t.ent_s, t.val_s, ldg(t.off_s + sl), ldg(t.off_s + sl + 1), lane,
                         reinterpret_cast<const char *>(X), xplane, reinterpret_cast<const char *>(J), jplane);
      slab_list<K, false>(acc, t.ket_d, t.val_d, ldg(t.off_d + sl), ldg(t.off_d + sl + 1), lane,
                          reinterpret_cast<const char *>(X), xplane, nullptr, 0u);
#pragma unroll
      for (int c = 0; c < K; ++c)
        out[c] = ex[c] == fx::kZero ? T(0.0) : F::value(acc[c], ex[c] + a.ev + fx::kUnit);
    } else {
#pragma unroll
      for (int c = 0; c < K; ++c) out[c] = T(0.0);
      const uint32_t xplane = 16u * (a.n + 1), jplane = 16u * (a.npair + 1);
      slab_list_fp<T, K, true>(out, t.ent_s, t.fp_s, t.val_s, a.ev, ldg(t.off_s + sl), ldg(t.off_s + sl + 1), lane,
                               reinterpret_cast<const char *>(X), xplane, reinterpret_cast<const char *>(J), jplane);
      slab_list_fp<T, K, false>(out, t.ket_d, t.fp_d, t.val_d, a.ev, ldg(t.off_d + sl), ldg(t.off_d + sl + 1), lane,
                                reinterpret_cast<const char *>(X), xplane, nullptr, 0u);
    }
    if (row == ~0u) continue;
    const uint64_t str = a.eta ? ldg(a.rowstr + row) : 0ull;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c0 + c >= a.m) break;
      T s = out[c];
      if (a.eta) s = flip(s, parity((unsigned long long)(str & ldg(a.colmask + c0 + c))));
      const size_t k = element(c);
      if (a.diag && !a.staged_diag) s = fma(diag(k), ldg(C + k), s);
      if (whole) {
        out[c] = add ? old[c] + s : s;
      } else if (add) {
        add_to(S + k, old[c], s);
      } else {
        S[k] = s;
      }
    }
    if (whole) {
      if constexpr (K == 4) store_row<K>(S + element(0), out);
    }
  }
}

template <typename T, int K, bool kAlpha>
__global__ void __launch_bounds__(kSlabThreads) k_slab(SlabArgs<T> a) {
  slab_cta<T, K, kAlpha>(a, a.C, a.S, blockIdx.x, blockIdx.y);
}

// ---- the same sweep in FP32 -------------------------------------------------------
//
// FP32 vectors and table values, FP32 products and list sums; in a caller's product a
// lane's two list sums, the diagonal and what sigma holds are added in float-float as
// in the kernels of sigma.cu, and the launches' results in FP32 (as there where the
// alpha x beta pairs or the beta sweep have a launch of their own).  In a solve's
// FP32 phase, whose result the double-float or FP64 phase refines, the two lists
// share a register (the sign of an eigenvector comes from its roundings: 1e-15 of
// the integrals turns 17% of a batch's vectors around, in any of these kernels).
// Four columns of a row are 16 bytes.  Bound: the L1 data pipe (3 bytes of table and
// 4 of shared memory a term at K = 8).  gridDim.z vectors at once.
struct SlabArgsF {
  const float *C[4];
  float *S[4];
  const dfloat *hii_df;  // the diagonal as hi + lo, less shift ...
  const float *hii_f;    // ... or rounded to FP32 where there is no shift
  dfloat shift;
  SlabSpin t;
  const float4 *val_s, *val_d;  // four entries' values
  const float *Jo;
  const uint64_t *rowstr, *colmask;
  uint32_t n, m, nb;
  int npair, eta, add, diag;
  int join;  // the two lists' sums are added in float-float
  int vec;   // rows of S start on 16-byte boundaries
  uint32_t parts;
};

template <int K, bool kSingles>
__device__ __forceinline__ void slab_group_f32(float (&acc)[K], const uint4 &g, const float4 &v, const char *X,
                                               uint32_t xplane, const char *J, uint32_t jplane) {
  const uint32_t w[kGroup] = {g.x, g.y, g.z, g.w};
  const float vs[kGroup] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int u = 0; u < kGroup; ++u) {
    const uint32_t x16 = kSingles ? w[u] & 0x7fff0u : w[u], j16 = (w[u] >> 15) & 0xfff0u;
#pragma unroll
    for (int q = 0; q < K / 4; ++q) {
      const float4 x = *reinterpret_cast<const float4 *>(X + q * xplane + x16);
      if constexpr (kSingles) {
        const float4 j = *reinterpret_cast<const float4 *>(J + q * jplane + j16);
        acc[4 * q] = fmaf(vs[u] + flip(j.x, w[u] >> 31), x.x, acc[4 * q]);
        acc[4 * q + 1] = fmaf(vs[u] + flip(j.y, w[u] >> 31), x.y, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(vs[u] + flip(j.z, w[u] >> 31), x.z, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(vs[u] + flip(j.w, w[u] >> 31), x.w, acc[4 * q + 3]);
      } else {
        acc[4 * q] = fmaf(vs[u], x.x, acc[4 * q]);
        acc[4 * q + 1] = fmaf(vs[u], x.y, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(vs[u], x.z, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(vs[u], x.w, acc[4 * q + 3]);
      }
    }
  }
}

template <int K, bool kSingles>
__device__ __forceinline__ void slab_list_f32(float (&acc)[K], const uint4 *__restrict__ ent,
                                              const float4 *__restrict__ val, uint32_t g, uint32_t end, uint32_t lane,
                                              const char *X, uint32_t xplane, const char *J, uint32_t jplane) {
  if (g >= end) return;
  uint32_t at = g * 32u + lane, left = end - g;
  uint4 wa = ldg(ent + at), wb;
  float4 va = __ldg(val + at), vb;
  while (true) {
    if (left > 1) {
      wb = ldg(ent + at + 32u);
      vb = __ldg(val + at + 32u);
    }
    slab_group_f32<K, kSingles>(acc, wa, va, X, xplane, J, jplane);
    if (left == 1) break;
    if (left > 2) {
      wa = ldg(ent + at + 64u);
      va = __ldg(val + at + 64u);
    }
    slab_group_f32<K, kSingles>(acc, wb, vb, X, xplane, J, jplane);
    if (left == 2) break;
    left -= 2;
    at += 64u;
  }
}

template <int K, bool kAlpha>
__device__ __forceinline__ void slab_cta_f32(const SlabArgsF &a, const float *__restrict__ C, float *S, uint32_t group,
                                             uint32_t part) {
  extern __shared__ __align__(16) unsigned char slab_smem[];
  float *X = reinterpret_cast<float *>(slab_smem);  // planes of four columns, n + 1 rows; row n is zero
  float *J = X + (size_t)(a.n + 1) * K;             // the same, npair + 1 rows
  __shared__ uint32_t snext;
  const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u;
  const uint32_t c0 = group * K;
  auto place = [](uint32_t rows, uint32_t r, uint32_t c) { return ((size_t)(c >> 2) * rows + r) * 4 + (c & 3u); };
  if (tid == 0) snext = 0u;
  if constexpr (kAlpha) {
    const uint32_t c = tid % K;
    const bool ok = c0 + c < a.m;
    const uint64_t mask = ok && a.eta ? ldg(a.colmask + c0 + c) : 0ull;
    for (uint32_t r = tid / K; r < a.n; r += nt / K) {
      float x = ok ? ldg(C + (size_t)r * a.nb + (c0 + c)) : 0.f;
      if (a.eta) x = flip(x, parity((unsigned long long)(mask & ldg(a.rowstr + r))));
      X[place(a.n + 1, r, c)] = x;
    }
  } else {
#pragma unroll
    for (uint32_t c = 0; c < K; ++c) {
      const bool ok = c0 + c < a.m;
      const uint64_t mask = ok && a.eta ? ldg(a.colmask + c0 + c) : 0ull;
      for (uint32_t r = tid; r < a.n; r += nt) {
        float x = ok ? ldg(C + (size_t)(c0 + c) * a.nb + r) : 0.f;
        if (a.eta) x = flip(x, parity((unsigned long long)(mask & ldg(a.rowstr + r))));
        X[place(a.n + 1, r, c)] = x;
      }
    }
  }
  if (tid < K) X[place(a.n + 1, a.n, tid)] = 0.f;
  if (a.npair)
    for (uint32_t i = tid; i < (uint32_t)(a.npair + 1) * K; i += nt) {
      const uint32_t P = i / K, c = i % K;
      J[place(a.npair + 1, P, c)] =
          P < (uint32_t)a.npair && c0 + c < a.m ? ldg(a.Jo + (size_t)P * a.m + (c0 + c)) : 0.f;
    }
  __syncthreads();
  const SlabSpin &t = a.t;
  const uint32_t xplane = 16u * (a.n + 1), jplane = 16u * (a.npair + 1);
  while (true) {
    uint32_t sl = 0;
    if (lane == 0) sl = atomicAdd(&snext, 1u);
    sl = part + a.parts * __shfl_sync(0xffffffffu, sl, 0);
    if (sl >= t.nslices) break;
    const uint32_t row = ldg(t.rows + sl * 32u + lane);
    auto element = [&](int c) { return kAlpha ? (size_t)row * a.nb + (c0 + c) : (size_t)(c0 + c) * a.nb + row; };
    const bool whole = kAlpha && a.vec && c0 + K <= a.m;  // this row's K elements in 16-byte pieces
    float acc[K], old[K], hi[K];
#pragma unroll
    for (int c = 0; c < K; ++c) acc[c] = old[c] = hi[c] = 0.f;
    if (row != ~0u) {  // what the end of the slice needs, requested now
      if (a.add && whole && !a.diag) {
        load_row<K>(S + element(0), old);
      } else {
#pragma unroll
        for (int c = 0; c < K; ++c)
          if (c0 + c < a.m) {
            if (a.add) old[c] = S[element(c)];
            if (a.diag && a.hii_f) hi[c] = ldg(a.hii_f + element(c));
          }
      }
    }
    slab_list_f32<K, true>(acc, t.ent_s, a.val_s, ldg(t.off_s + sl), ldg(t.off_s + sl + 1), lane,
                           reinterpret_cast<const char *>(X), xplane, reinterpret_cast<const char *>(J), jplane);
    float singles[K];
#pragma unroll
    for (int c = 0; c < K; ++c) {
      singles[c] = a.join ? acc[c] : 0.f;
      acc[c] = a.join ? 0.f : acc[c];
    }
    slab_list_f32<K, false>(acc, t.ket_d, a.val_d, ldg(t.off_d + sl), ldg(t.off_d + sl + 1), lane,
                            reinterpret_cast<const char *>(X), xplane, nullptr, 0u);
    if (row == ~0u) continue;
    const uint64_t str = a.eta ? ldg(a.rowstr + row) : 0ull;
    if (!a.diag && !a.add) {  // (two sums in float-float round to their FP32 sum)
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c0 + c >= a.m) break;
        if (a.join) acc[c] += singles[c];
        if (a.eta) acc[c] = flip(acc[c], parity((unsigned long long)(str & ldg(a.colmask + c0 + c))));
        if (!whole) S[element(c)] = acc[c];
      }
      if (whole) store_row<K>(S + element(0), acc);
      continue;
    }
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c0 + c >= a.m) break;
      const uint32_t ph = a.eta ? parity((unsigned long long)(str & ldg(a.colmask + c0 + c))) : 0u;
      if (a.diag) {  // eta sigma = h (eta C) + the sums
        const float x = X[place(a.n + 1, row, c)];
        FF d;
        if (a.hii_f) {
          d = ff_prod(hi[c], x);
        } else {
          const dfloat h = ldg(a.hii_df + element(c));
          d = ff_diag(h.hi, h.lo, a.shift.hi, a.shift.lo, x);
        }
        ff_add(d, singles[c]);
        ff_add(d, acc[c]);
        if (ph) d = FF{-d.hi, -d.lo};
        if (a.add) ff_add(d, old[c]);
        acc[c] = ff_value(d);
      } else {
        FF d{flip(singles[c], ph), 0.f};
        ff_add(d, flip(acc[c], ph));
        ff_add(d, old[c]);
        acc[c] = ff_value(d);
      }
      if (!whole) S[element(c)] = acc[c];
    }
    if (whole) store_row<K>(S + element(0), acc);
  }
}

template <int K, bool kAlpha>
__global__ void __launch_bounds__(kSlabThreads) k_slab_f32(SlabArgsF a) {
  slab_cta_f32<K, kAlpha>(a, a.C[blockIdx.z], a.S[blockIdx.z], blockIdx.x, blockIdx.y);
}

// ---- alpha single x beta single (task type 0) ---------------------------------------
//
// The layout of k_sigma_ab (sigma_ab.cu): a CTA owns one alpha row (or every
// parts-th slice of its columns: rows with many more batches than most, whose
// batches follow one another, would end the launch alone) and takes G of its
// singles at a time, C rows and (P|Q) rows staged in shared memory; beta singles
// in slices of 32 columns, their entries ordered against bank conflicts
// (k_slab_ab_order).  Each (P|Q) value is staged with both signs, so that an
// entry's phase is part of its index.
//
// The ket rows of a batch have scales of their own (2^e_g); the batch's is the
// largest, and the (P|Q) values of a smaller row are scaled down by the
// difference (in a caller's product kRows binary orders at most: floating-point
// sums beyond; 3 decades of weights make 10).
// kSum: the row's sums stay in shared memory until the last batch; otherwise
// each batch's go to sigma at once (rows with a batch or two; less shared
// memory, so more CTAs an SM).

template <typename T>
struct SlabAbArgs {
  const T *C;
  T *S;
  const uint64_t *astr;
  const uint64_t *colmask;           // per beta string
  const uint32_t *off, *ket, *code;  // alpha singles
  const double *Kp;
  const T *Kt;         // the same in the vectors' format
  const uint2 *items;  // (alpha row, part | parts << 16)
  const uint32_t *cols, *slice, *ent;
  uint32_t nslices, nb;
  int npair, ek, eta, guard;
};

template <typename T, int G, bool kSum>
__device__ __forceinline__ void slab_ab_cta(const SlabAbArgs<T> &a, const T *__restrict__ C, T *S, uint2 item) {
  using F = Format<T>;
  constexpr int NP = G / 2;
  extern __shared__ __align__(16) unsigned char slab_smem[];
  const uint32_t kplane = 2 * (a.npair + 1), cplane = a.nb + 1;
  const uint32_t pad = a.nb << 13 | (uint32_t)a.npair << 1;  // padding entries: a zero column and a zero pair
  int4 *Cs = reinterpret_cast<int4 *>(slab_smem);                // [G/2][nb + 1]: two ket rows' values at jb
  int4 *Ks = Cs + (size_t)NP * cplane;                           // [G/2][2 Q + phase]
  double *Ss = reinterpret_cast<double *>(Ks + NP * kplane);     // kSum: [nb]
  __shared__ Keys skey[G];
  const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u, warp = tid >> 5, nw = nt >> 5;
  const uint32_t ia = item.x, part = item.y & 0xffffu, parts = item.y >> 16;
  const uint32_t p0 = ldg(a.off + ia), p1 = ldg(a.off + ia + 1);
  const uint64_t str = a.eta ? ldg(a.astr + ia) : 0ull;
  const uint32_t mine = (a.nslices - part + parts - 1) / parts;  // slices of this CTA
  if (tid < NP) Cs[tid * cplane + a.nb] = make_int4(0, 0, 0, 0);
  if (kSum)
    for (uint32_t c = tid; c < a.nb; c += nt) Ss[c] = 0.0;
  for (uint32_t pb = p0; pb < p1; pb += G) {
    const uint32_t live = min((uint32_t)G, p1 - pb);
    __syncthreads();  // the previous batch is applied
    if (tid < G) skey[tid] = Keys{0u, ~0u, 0u, 0u};
    __syncthreads();
    Spread<T> keys[G];
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const bool ok0 = 2 * h < live, ok1 = 2 * h + 1 < live;
      const uint32_t ja0 = ok0 ? ldg(a.ket + pb + 2 * h) : 0u, ja1 = ok1 ? ldg(a.ket + pb + 2 * h + 1) : 0u;
      const uint64_t s0 = a.eta && ok0 ? ldg(a.astr + ja0) : 0ull, s1 = a.eta && ok1 ? ldg(a.astr + ja1) : 0ull;
      const T *r0 = C + (size_t)ja0 * a.nb, *r1 = C + (size_t)ja1 * a.nb;
      for (uint32_t c = tid; c < a.nb; c += nt) {
        T x0 = ok0 ? ldg(r0 + c) : T(0.0), x1 = ok1 ? ldg(r1 + c) : T(0.0);
        if (a.eta) {
          const uint64_t m = ldg(a.colmask + c);
          x0 = flip(x0, parity((unsigned long long)(s0 & m)));
          x1 = flip(x1, parity((unsigned long long)(s1 & m)));
        }
        keys[2 * h].count(x0, a.guard);
        keys[2 * h + 1].count(x1, a.guard);
        const int2 b0 = F::raw(x0), b1 = F::raw(x1);
        Cs[h * cplane + c] = make_int4(b0.x, b0.y, b1.x, b1.y);
      }
    }
    int e[G], es = fx::kZero;
#pragma unroll
    for (int g = 0; g < G; ++g) keys[g].add_to(&skey[g], a.guard);
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g) {
      e[g] = F::exponent(skey[g].top);
      es = max(es, e[g]);
    }
    if (es == fx::kZero) continue;  // every row is zero
    bool fixed = es != fx::kBad;    // otherwise floating-point sums of the values as they are
    if (a.guard) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        fixed = fixed && !Spread<T>::wide(skey[g]) && (e[g] == fx::kZero || es - e[g] <= F::kRows);
    }
    if (fixed) {  // to fixed point, in place: each thread the columns that it staged
#pragma unroll
      for (int h = 0; h < NP; ++h)
        for (uint32_t c = tid; c < a.nb; c += nt) {
          const int4 r = Cs[h * cplane + c];
          const int2 z = make_int2(0, 0);
          const int2 x0 = e[2 * h] == fx::kZero ? z : F::parts(make_int2(r.x, r.y), e[2 * h]);
          const int2 x1 = e[2 * h + 1] == fx::kZero ? z : F::parts(make_int2(r.z, r.w), e[2 * h + 1]);
          Cs[h * cplane + c] = make_int4(x0.x, x0.y, x1.x, x1.y);
        }
    }
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const uint32_t c0 = 2 * h < live ? ldg(a.code + pb + 2 * h) : 0u;
      const uint32_t c1 = 2 * h + 1 < live ? ldg(a.code + pb + 2 * h + 1) : 0u;
      const size_t k0 = (size_t)((c0 >> 16) & 0x7fffu) * a.npair, k1 = (size_t)((c1 >> 16) & 0x7fffu) * a.npair;
      for (uint32_t Q = tid; Q <= (uint32_t)a.npair; Q += nt) {
        const bool ok0 = Q < (uint32_t)a.npair && 2 * h < live, ok1 = Q < (uint32_t)a.npair && 2 * h + 1 < live;
        int2 f0, f1, n0, n1;
        if (fixed) {
          // (an all-zero row's values are not used, whatever its scale)
          const double v0 = ok0 ? flip(ldg(a.Kp + k0 + Q), c0 >> 31) : 0.0;
          const double v1 = ok1 ? flip(ldg(a.Kp + k1 + Q), c1 >> 31) : 0.0;
          f0 = fx::make(v0, fx::kVBits - a.ek - min(es - e[2 * h], 100));
          f1 = fx::make(v1, fx::kVBits - a.ek - min(es - e[2 * h + 1], 100));
          n0 = make_int2(-f0.x, -f0.y);
          n1 = make_int2(-f1.x, -f1.y);
        } else {
          const T v0 = ok0 ? flip(ldg(a.Kt + k0 + Q), c0 >> 31) : T(0.0);
          const T v1 = ok1 ? flip(ldg(a.Kt + k1 + Q), c1 >> 31) : T(0.0);
          f0 = F::raw(v0);
          f1 = F::raw(v1);
          n0 = F::raw(-v0);
          n1 = F::raw(-v1);
        }
        Ks[h * kplane + 2 * Q] = make_int4(f0.x, f0.y, f1.x, f1.y);
        Ks[h * kplane + 2 * Q + 1] = make_int4(n0.x, n0.y, n1.x, n1.y);
      }
    }
    __syncthreads();
    // this CTA's slices (longest first) dealt to the warps in snake order
    for (uint32_t base = 0, round = 0; base < mine; base += nw, ++round) {
      const uint32_t i = base + ((round & 1u) ? nw - 1u - warp : warp);
      if (i >= mine) continue;
      const uint32_t sl = part + parts * i, k = sl * 32u + lane;
      uint32_t at = ldg(a.slice + sl) + lane;
      const uint32_t end = ldg(a.slice + sl + 1) + lane;
      if (at >= end) continue;
      uint32_t w[kGroup];  // four entries; the next four are requested before these are summed
      auto load = [&](uint32_t from) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) w[u] = from + 32u * u < end ? ldg(a.ent + from + 32u * u) : pad;
      };
      load(at);
      const uint32_t ib = k < a.nb ? ldg(a.cols + k) : 0u;
      T *const to = S + ((size_t)ia * a.nb + ib);
      const T old = !kSum && !kReduce<T> && k < a.nb ? *to : T(0.0);
      double sum = 0.0;
      if (fixed) {
        fx::Acc acc;
        fx::zero(acc);
        uint32_t since = 0;
        for (; at < end; at += 32u * kGroup) {
          uint32_t wc[kGroup];
#pragma unroll
          for (int u = 0; u < kGroup; ++u) wc[u] = w[u];
          if (at + 32u * kGroup < end) load(at + 32u * kGroup);
#pragma unroll
          for (int u = 0; u < kGroup; ++u)
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              const int4 kv = Ks[h * kplane + (wc[u] & 0x1fffu)], cv = Cs[h * cplane + (wc[u] >> 13)];
              fx::mac(acc, cv.x, cv.y, kv.x, kv.y);
              fx::mac(acc, cv.z, cv.w, kv.z, kv.w);
            }
          since += G * kGroup;
          if (since >= fx::kChunkHigh) {
            fx::carry(acc);
            since = 0;
          }
        }
        fx::carry(acc);
        sum = fx::value(acc, es + a.ek + fx::kUnit);
      } else {
        T acc = T(0.0);
        for (; at < end; at += 32u * kGroup) {
          uint32_t wc[kGroup];
#pragma unroll
          for (int u = 0; u < kGroup; ++u) wc[u] = w[u];
          if (at + 32u * kGroup < end) load(at + 32u * kGroup);
#pragma unroll
          for (int u = 0; u < kGroup; ++u) {
            if (at + 32u * u >= end) break;  // the same for the whole warp
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              if (2 * h >= live) break;
              const int4 kv = Ks[h * kplane + (wc[u] & 0x1fffu)], cv = Cs[h * cplane + (wc[u] >> 13)];
              acc = fma(F::of(make_int2(kv.x, kv.y)), F::of(make_int2(cv.x, cv.y)), acc);
              if (2 * h + 1 < live)
                acc = fma(F::of(make_int2(kv.z, kv.w)), F::of(make_int2(cv.z, cv.w)), acc);
            }
          }
        }
        sum = (double)acc;
      }
      if (k >= a.nb) continue;
      if (kSum) {
        Ss[ib] += sum;
      } else {
        if (a.eta) sum = flip(sum, parity((unsigned long long)(str & ldg(a.colmask + ib))));
        add_to(to, old, T(sum));  // this thread's alone: batches add in their order
      }
    }
  }
  if (!kSum) return;
  auto add_row = [](T *at, double x) { *at = *at + T(x); };
  __syncthreads();
  if (parts == 1) {
    for (uint32_t c = tid; c < a.nb; c += nt) {
      double s = Ss[c];
      if (a.eta) s = flip(s, parity((unsigned long long)(str & ldg(a.colmask + c))));
      add_row(S + ((size_t)ia * a.nb + c), s);
    }
  } else {
    for (uint32_t i = warp; i < mine; i += nw) {
      const uint32_t k = (part + parts * i) * 32u + lane;
      if (k >= a.nb) continue;
      const uint32_t ib = ldg(a.cols + k);
      double s = Ss[ib];
      if (a.eta) s = flip(s, parity((unsigned long long)(str & ldg(a.colmask + ib))));
      add_row(S + ((size_t)ia * a.nb + ib), s);
    }
  }
}

template <typename T, int G, bool kSum>
__global__ void __launch_bounds__(kSlabAbThreads) k_slab_ab(SlabAbArgs<T> a) {
  slab_ab_cta<T, G, kSum>(a, a.C, a.S, __ldg(a.items + blockIdx.x));
}

// FP32: four ket rows' values at a column are 16 bytes, four (P|Q) rows' at a
// pair too; the sums of a row stay in shared memory.
struct SlabAbArgsF {
  const float *C[4];
  float *S[4];
  const uint64_t *astr, *colmask;
  const uint32_t *off, *ket, *code;
  const float *Kp;
  const uint2 *items;
  const uint32_t *cols, *slice, *ent;
  uint32_t nslices, nb;
  int npair, eta;
};

__device__ __forceinline__ void slab_ab_cta_f32(const SlabAbArgsF &a, const float *__restrict__ C, float *S,
                                                uint2 item) {
  extern __shared__ __align__(16) unsigned char slab_smem[];
  float4 *Cs = reinterpret_cast<float4 *>(slab_smem);               // [nb + 1]
  float4 *Ks = Cs + a.nb + 1;                                       // [2 Q + phase]
  float *Ss = reinterpret_cast<float *>(Ks + 2 * (a.npair + 1));    // [nb]
  const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u, warp = tid >> 5, nw = nt >> 5;
  const uint32_t ia = item.x, part = item.y & 0xffffu, parts = item.y >> 16;
  const uint32_t p0 = ldg(a.off + ia), p1 = ldg(a.off + ia + 1);
  const uint32_t mine = (a.nslices - part + parts - 1) / parts;
  const uint32_t pad = a.nb << 13 | (uint32_t)a.npair << 1;
  for (uint32_t c = tid; c < a.nb; c += nt) Ss[c] = 0.f;
  if (tid == 0) Cs[a.nb] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t pb = p0; pb < p1; pb += 4) {
    const float *r[4], *kr[4];
    uint64_t str[4];
    uint32_t sg[4];
    bool ok[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      ok[g] = pb + g < p1;
      const uint32_t ja = ok[g] ? ldg(a.ket + pb + g) : 0u, code = ok[g] ? ldg(a.code + pb + g) : 0u;
      str[g] = a.eta && ok[g] ? ldg(a.astr + ja) : 0ull;
      r[g] = C + (size_t)ja * a.nb;
      kr[g] = a.Kp + (size_t)((code >> 16) & 0x7fffu) * a.npair;
      sg[g] = code >> 31;
    }
    __syncthreads();  // the previous batch is applied
    for (uint32_t c = tid; c < a.nb; c += nt) {
      float x[4];
      const uint64_t m = a.eta ? ldg(a.colmask + c) : 0ull;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        x[g] = ok[g] ? ldg(r[g] + c) : 0.f;
        if (a.eta) x[g] = flip(x[g], parity((unsigned long long)(str[g] & m)));
      }
      Cs[c] = make_float4(x[0], x[1], x[2], x[3]);
    }
    for (uint32_t Q = tid; Q <= (uint32_t)a.npair; Q += nt) {
      float v[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) v[g] = ok[g] && Q < (uint32_t)a.npair ? flip(ldg(kr[g] + Q), sg[g]) : 0.f;
      Ks[2 * Q] = make_float4(v[0], v[1], v[2], v[3]);
      Ks[2 * Q + 1] = make_float4(-v[0], -v[1], -v[2], -v[3]);
    }
    __syncthreads();
    for (uint32_t base = 0, round = 0; base < mine; base += nw, ++round) {
      const uint32_t i = base + ((round & 1u) ? nw - 1u - warp : warp);
      if (i >= mine) continue;
      const uint32_t sl = part + parts * i, k = sl * 32u + lane;
      uint32_t at = ldg(a.slice + sl) + lane;
      const uint32_t end = ldg(a.slice + sl + 1) + lane;
      if (at >= end) continue;
      uint32_t w[kGroup];
      auto load = [&](uint32_t from) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) w[u] = from + 32u * u < end ? ldg(a.ent + from + 32u * u) : pad;
      };
      load(at);
      float sum = 0.f;
      for (; at < end; at += 32u * kGroup) {
        uint32_t wc[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) wc[u] = w[u];
        if (at + 32u * kGroup < end) load(at + 32u * kGroup);
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
          const float4 kv = Ks[wc[u] & 0x1fffu], cv = Cs[wc[u] >> 13];
          sum = fmaf(kv.x, cv.x, sum);
          sum = fmaf(kv.y, cv.y, sum);
          sum = fmaf(kv.z, cv.z, sum);
          sum = fmaf(kv.w, cv.w, sum);
        }
      }
      if (k < a.nb) Ss[ldg(a.cols + k)] += sum;
    }
  }
  __syncthreads();
  const uint64_t istr = a.eta ? ldg(a.astr + ia) : 0ull;
  float *srow = S + (size_t)ia * a.nb;
  auto add = [&](uint32_t c) {
    float s = Ss[c];
    if (a.eta) s = flip(s, parity((unsigned long long)(istr & ldg(a.colmask + c))));
    srow[c] += s;
  };
  if (parts == 1) {
    for (uint32_t c = tid; c < a.nb; c += nt) add(c);
  } else {
    for (uint32_t i = warp; i < mine; i += nw) {
      const uint32_t k = (part + parts * i) * 32u + lane;
      if (k < a.nb) add(ldg(a.cols + k));
    }
  }
}

__global__ void __launch_bounds__(kSlabAbThreads) k_slab_ab_f32(SlabAbArgsF a) {
  slab_ab_cta_f32(a, a.C[blockIdx.z], a.S[blockIdx.z], __ldg(a.items + blockIdx.x));
}

// ---- many problems at once (batch.cu) ----------------------------------------------
//
// The CTAs of every problem's sweep in one grid; blockIdx.y numbers the new
// vectors of a problem's step (columns from + y of its basis), whose count and
// activity each CTA reads from the solver's state.
template <typename A>
struct SlabMany {
  const A *args;        // per problem
  const uint4 *items;   // (problem, group or row, part or part | parts << 16, -)
  SlabBatchState state;
};
constexpr int kManyThreads = 256;

template <typename T, typename A>
__device__ __forceinline__ bool many_vector(const SlabMany<A> &m, uint32_t prob, const T *&C, T *&S) {
  const SlabBatchState &st = m.state;
  auto field = [&](const int *f) { return *reinterpret_cast<const int *>(reinterpret_cast<const char *>(f) + prob * st.stride); };
  const int from = field(st.from), to = field(st.to);
  if (!field(st.active) || from + (int)blockIdx.y >= to) return false;
  const size_t at = (size_t)st.N[prob] * (from + blockIdx.y);
  C = reinterpret_cast<const T *>(st.V[prob]) + at;
  S = reinterpret_cast<T *>(st.HV[prob]) + at;
  return true;
}
template <int K, bool kAlpha>
__global__ void __launch_bounds__(kManyThreads, 3) k_slab_many(SlabMany<SlabArgs<double>> m) {
  const uint4 it = __ldg(m.items + blockIdx.x);
  const double *C;
  double *S;
  if (many_vector(m, it.x, C, S)) slab_cta<double, K, kAlpha>(m.args[it.x], C, S, it.y, it.z);
}
template <int K, bool kAlpha>
__global__ void __launch_bounds__(kManyThreads, 3) k_slab_many_f32(SlabMany<SlabArgsF> m) {
  const uint4 it = __ldg(m.items + blockIdx.x);
  const float *C;
  float *S;
  if (many_vector(m, it.x, C, S)) slab_cta_f32<K, kAlpha>(m.args[it.x], C, S, it.y, it.z);
}
template <int G>
__global__ void __launch_bounds__(kManyThreads, 3) k_slab_ab_many(SlabMany<SlabAbArgs<double>> m) {
  const uint4 it = __ldg(m.items + blockIdx.x);
  const double *C;
  double *S;
  if (many_vector(m, it.x, C, S)) slab_ab_cta<double, G, true>(m.args[it.x], C, S, make_uint2(it.y, it.z));
}
__global__ void __launch_bounds__(kManyThreads, 3) k_slab_ab_many_f32(SlabMany<SlabAbArgsF> m) {
  const uint4 it = __ldg(m.items + blockIdx.x);
  const float *C;
  float *S;
  if (many_vector(m, it.x, C, S)) slab_ab_cta_f32(m.args[it.x], C, S, make_uint2(it.y, it.z));
}

// ---- tables -----------------------------------------------------------------------

// Largest |x| (as ordered bits) of n values, into out.
__global__ void k_absmax(const double *__restrict__ x, size_t n, unsigned long long *out) {
  unsigned long long b = 0ull;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    b = max(b, (unsigned long long)__double_as_longlong(x[e]) & ~(1ull << 63));
  for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, b);
}

// The same over the rows P = (p, q), p != q, of an [npair][n] table (the others
// belong to no excitation).
__global__ void k_absmax_pairs(const double *__restrict__ x, uint32_t n, unsigned long long *out) {
  const uint32_t P = blockIdx.y;
  uint32_t p = (uint32_t)((sqrtf(8.f * (float)P + 1.f) - 1.f) * 0.5f);  // the p of P = p (p + 1) / 2 + q, or next to it
  while (p * (p + 1) / 2 > P) --p;
  while ((p + 1) * (p + 2) / 2 <= P) ++p;
  if (P == p * (p + 1) / 2 + p) return;
  unsigned long long b = 0ull;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    b = max(b, (unsigned long long)__double_as_longlong(x[(size_t)P * n + e]) & ~(1ull << 63));
  for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, b);
}

// Order in which each row's entries are taken: a lane's gather reads 16 bytes
// of shared memory at 16 ket (mod 128), and the 8 lanes that one 128-byte
// wavefront serves collide where their kets agree mod 8 (2.6 wavefronts for 8
// random ones, 2.4 measured).  The order of a list is free, so one warp per
// slice deals the entries out step by step: the lanes of an 8-lane group choose
// one after another (a different one first each step), each taking a residue
// that no earlier lane has, the one it has most entries of (simulated: 1.35
// wavefronts for lists of 40, 1.14 for 228).  order: entry indices, row by row
// as in the CSR lists; next: scratch of the same size.
__global__ void __launch_bounds__(32) k_slab_order(const uint32_t *__restrict__ off, const uint32_t *__restrict__ ket,
                                                   const uint32_t *__restrict__ rows, uint32_t *__restrict__ next,
                                                   uint32_t *__restrict__ order) {
  __shared__ uint32_t head[8][32];
  const uint32_t lane = threadIdx.x;
  const uint32_t row = rows[blockIdx.x * 32u + lane];
  const uint32_t p0 = row == ~0u ? 0u : off[row], p1 = row == ~0u ? 0u : off[row + 1];
  uint32_t cnt[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    cnt[r] = 0u;
    head[r][lane] = ~0u;
  }
  for (uint32_t p = p1; p-- > p0;) {  // lists by residue, in ascending order
    const uint32_t r = ket[p] & 7u;
    next[p] = head[r][lane];
    head[r][lane] = p;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) cnt[q] += q == r;
  }
  const uint32_t steps = __reduce_max_sync(0xffffffffu, p1 - p0), group = lane & 24u;
  for (uint32_t t = 0; t < steps; ++t) {
    uint32_t used = 0u;  // residues taken at this step in this group of lanes
    for (uint32_t i = 0; i < 8; ++i) {
      uint32_t best = 0u, pick = 8u;
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r) {
        const uint32_t key = cnt[r] ? cnt[r] + ((used >> r & 1u) ? 0u : 1u << 16) : 0u;
        if (key > best) {
          best = key;
          pick = r;
        }
      }
      const uint32_t turn = group | ((i + t) & 7u);
      const uint32_t taken = __shfl_sync(0xffffffffu, pick, turn);
      used |= 1u << taken;  // bit 8: the lane's list is empty
      if (lane == turn && pick < 8u) {
        const uint32_t p = head[pick][lane];
        head[pick][lane] = next[p];
        order[p0 + t] = p;
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) cnt[q] -= q == pick;
      }
    }
  }
}

// The same for the beta singles of k_slab_ab, whose entries read two places of
// shared memory (column w >> 13, pair and phase w & 0x1fff): in its turn a lane
// takes, of the next 16 entries of its list, the one that collides least with
// the lanes before it (simulated for lists of 18-25: 1.85 wavefronts per 8
// lanes and read, 2.6 in list order).  One warp per slice, in place; the
// padding, behind the real entries, is pointed at the zero column nb.
__global__ void __launch_bounds__(32) k_slab_ab_order(const uint32_t *__restrict__ slice, uint32_t npair, uint32_t nb,
                                                      uint32_t *__restrict__ ent) {
  const uint32_t lane = threadIdx.x, e0 = slice[blockIdx.x] + lane, len = (slice[blockIdx.x + 1] - slice[blockIdx.x]) / 32u;
  uint32_t cnt = 0;
  while (cnt < len && (ent[e0 + 32u * cnt] & 0x1ffeu) != npair << 1) ++cnt;
  for (uint32_t t = cnt; t < len; ++t) ent[e0 + 32u * t] = nb << 13 | npair << 1;
  const uint32_t group = lane & 24u;
  for (uint32_t t = 0; t < len; ++t) {
    uint32_t used = 0u;  // residues taken in this group of lanes: columns in bits 0-7, pairs in 8-15
    for (uint32_t i = 0; i < 8; ++i) {
      const uint32_t turn = group | ((i + t) & 7u);
      uint32_t take = 0u;
      if (lane == turn && t < cnt) {
        uint32_t best = 3u, at = t, word = 0u;
        for (uint32_t j = t; j < min(t + 16u, cnt) && best; ++j) {
          const uint32_t w = ent[e0 + 32u * j];
          const uint32_t cost = (used >> ((w >> 13) & 7u) & 1u) + (used >> (8u + (w & 7u)) & 1u);
          if (cost < best) {
            best = cost;
            at = j;
            word = w;
          }
        }
        if (at != t) {
          ent[e0 + 32u * at] = ent[e0 + 32u * t];
          ent[e0 + 32u * t] = word;
        }
        take = 1u << ((word >> 13) & 7u) | 1u << (8u + (word & 7u));
      }
      used |= __shfl_sync(0xffffffffu, take, turn);
    }
  }
}

// The sliced form of one spin's tables: one CTA per slice, thread (lane, y)
// writes every 4th group of the lane's row.
__global__ void __launch_bounds__(128) k_slab_fill(SpinTables T, const uint32_t *__restrict__ rows,
                                                   const uint32_t *__restrict__ off_s,
                                                   const uint32_t *__restrict__ off_d,
                                                   const uint32_t *__restrict__ order_s,
                                                   const uint32_t *__restrict__ order_d, int npair, int ev,
                                                   uint4 *__restrict__ ent_s, int4 *__restrict__ val_s,
                                                   uint4 *__restrict__ ket_d, int4 *__restrict__ val_d,
                                                   float4 *__restrict__ valf_s, float4 *__restrict__ valf_d,
                                                   double2 *__restrict__ fp_s, double2 *__restrict__ fp_d) {
  const uint32_t sl = blockIdx.x, lane = threadIdx.x & 31u, y = threadIdx.x >> 5;
  const uint32_t row = rows[sl * 32u + lane];
  for (int doubles = 0; doubles < 2; ++doubles) {
    const uint32_t *off = doubles ? off_d : off_s, *rp = doubles ? T.off_d : T.off_s;
    const uint32_t *order = doubles ? order_d : order_s;
    const uint32_t p0 = row == ~0u ? 0u : rp[row], cnt = row == ~0u ? 0u : rp[row + 1] - p0;
    for (uint32_t g = off[sl] + y; g < off[sl + 1]; g += 4) {
      uint32_t w[kGroup];
      int2 v[kGroup];
      float f[kGroup];
      double d[kGroup];
#pragma unroll
      for (int u = 0; u < kGroup; ++u) {
        const uint32_t j = (g - off[sl]) * kGroup + u;
        const bool ok = j < cnt;
        const uint32_t p = ok ? order[p0 + j] : 0u;
        if (doubles) {
          w[u] = (ok ? T.ket_d[p] : T.n) << 4;
          d[u] = ok ? T.val_d[p] : 0.0;
          f[u] = (float)d[u];
        } else {
          const uint32_t code = ok ? T.code_s[p] : 0u;
          w[u] = ok ? (T.ket_s[p] << 4 | ((code >> 16) & 0x7fffu) << 19 | (code & 0x80000000u))
                    : (T.n << 4 | (uint32_t)npair << 19);
          d[u] = ok ? flip(T.val_s[p], code >> 31) : 0.0;
          f[u] = ok ? flip((float)T.val_s[p], code >> 31) : 0.f;
        }
        v[u] = fx::make(d[u], fx::kVBits - ev);
      }
      const size_t e = (size_t)g * 32u + lane;
      (doubles ? ket_d : ent_s)[e] = make_uint4(w[0], w[1], w[2], w[3]);
      (doubles ? val_d : val_s)[2 * e] = make_int4(v[0].x, v[0].y, v[1].x, v[1].y);
      (doubles ? val_d : val_s)[2 * e + 1] = make_int4(v[2].x, v[2].y, v[3].x, v[3].y);
      (doubles ? valf_d : valf_s)[e] = make_float4(f[0], f[1], f[2], f[3]);
      if (fp_s) {
        (doubles ? fp_d : fp_s)[2 * e] = make_double2(d[0], d[1]);
        (doubles ? fp_d : fp_s)[2 * e + 1] = make_double2(d[2], d[3]);
      }
    }
  }
}

__global__ void k_slab_coulomb(const double *__restrict__ J, size_t n, int s, int2 *__restrict__ out) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    out[e] = fx::make(J[e], s);
}

// Per string: the orbitals of the other spin's strings whose parity is eta
// (sigma_dev.cuh:eta_parity): below a beta string's electrons for an alpha
// string, above an alpha string's for a beta string.
__global__ void k_slab_masks(const uint64_t *__restrict__ str, uint32_t n, int beta, uint64_t *__restrict__ mask) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long x = str[i];
  if (beta) {
    x <<= 1;
    for (int k = 1; k < 64; k <<= 1) x ^= x << k;
  } else {
    x >>= 1;
    for (int k = 1; k < 64; k <<= 1) x ^= x >> k;
  }
  mask[i] = x;
}

size_t max_smem() {
  int dev = 0, optin = 0;
  SBDGB_CUDA(cudaGetDevice(&dev));
  SBDGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return (size_t)optin - 1024;  // the kernels' static part
}
SlabSize slab_size(const Problem &p) { return {p.na, p.nb, p.npair, {p.A.ns, p.B.ns}}; }
size_t slab_ab_smem_bytes(const Problem &p, int G, bool sum) { return sbdgb::slab_ab_smem_bytes(p.nb, p.npair, G, sum); }
bool slab_ab_sum(const Problem &p) { return slab_size(p).ab_sum(); }

}  // namespace

// ---- host side ----------------------------------------------------------------------

// Whether the kernels of a form (element: 8 bytes, or 4 in FP32) have the shared
// memory that this problem takes.
bool slab_fits(const Problem &p, int element) { return slab_fits(slab_size(p), element, max_smem()); }

namespace {

// What building the tables holds until it is done: temporaries, and how to give
// back the tables themselves where memory runs out half way.
struct SlabBuild {
  Problem &p;
  cudaStream_t s;
  size_t first, bytes = 0;  // of p.allocs; bytes allocated since
  std::vector<void *> tmps;
  bool done = false;
  SlabBuild(Problem &pp, cudaStream_t ss) : p(pp), s(ss), first(pp.allocs.size()) {}
  void *alloc(size_t n) {
    void *d = dev_alloc(p, n);
    bytes += n ? n : 8;
    return d;
  }
  ~SlabBuild() {
    if (!done && p.allocs.size() > first) cudaStreamSynchronize(s);  // they may still be written
    for (void *t : tmps) tmp_free(p.ctx, t);
    if (done) return;
    for (size_t i = first; i < p.allocs.size(); ++i) tmp_free(p.ctx, p.allocs[i]);
    p.allocs.resize(first);
    p.bytes -= bytes;
    p.ctx->in_use -= bytes;
    p.slab = Problem::Slab{};
    p.slab.state = 0;
  }
};

// Bytes that a budget leaves for the tables.  A serving context's reservation counts
// a transposed copy, which these kernels do without, and half a MB of its slack is
// theirs too; they serve solves alone there and go without the FP64 values (24 bytes
// an entry otherwise, 16).  Under a caller's budget, whose other uses are not known,
// they must leave room for that copy and the largest solve (64 basis vectors and 16
// roots): what fits without them fits with them.
size_t slab_room(const Problem &p) {
  const Ctx &c = *p.ctx;
  const size_t left = c.in_use < c.budget ? c.budget - c.in_use : 0;
  if (c.pool) return std::min(left, 8 * p.N + (1u << 19));
  const size_t solve = 8 * p.N + 16 * 64 * p.N + 64 * 16 * p.N;
  return left > solve ? left - solve : 0;
}

// CTAs of the alpha x beta kernels: a row is shared by `base` of them where
// rows are few, and (while the rows are only a few waves, which the longest
// would otherwise end alone) by more the further its batches exceed the mean:
// 2011 x 1703 strings 0.166 ms, here 0.152; with 6000 x 6000, where it only
// adds staging, 0.89 and 0.99
uint32_t slab_ab_base(const Problem &p) {
  int sms = 0;
  SBDGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.ctx->device));
  return std::min(p.n_ab_slices, std::max<uint32_t>(1, 4u * sms / p.n_ab_rows));
}
std::vector<uint2> slab_ab_items(const Problem &p, const std::vector<uint32_t> &off_a) {
  std::vector<uint2> items;
  int sms = 0;
  SBDGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.ctx->device));
  const uint32_t base = slab_ab_base(p);
  const double mean = (double)p.A.ns / p.n_ab_rows;
  std::vector<uint32_t> order(p.na);
  std::iota(order.begin(), order.end(), 0u);
  auto singles = [&](uint32_t r) { return off_a[r + 1] - off_a[r]; };
  std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return singles(x) > singles(y); });
  for (uint32_t r : order) {
    if (singles(r) == 0) break;
    const uint32_t parts = std::min<uint32_t>(p.n_ab_slices, base * (uint32_t)std::ceil(p.n_ab_rows < 12u * sms ? singles(r) / (4.0 * mean) : 1.0));
    for (uint32_t y = 0; y < parts; ++y) items.push_back(make_uint2(r, y | parts << 16));
  }
  return items;
}

bool slab_build(Problem &p, SlabBuild &build, cudaStream_t s) {
  if (std::max(p.na, p.nb) >= kSlabMaxRows || (uint32_t)p.npair + 1 >= kSlabMaxPair) return false;
  const bool ab = p.A.ns > 0 && p.B.ns > 0;
  if (!slab_fits(p, 8) || (ab && p.n_ab_rows == 0)) return false;
  // the largest table values
  unsigned long long *mx = (unsigned long long *)workspace(p, WS_RED2, 8 * sizeof(unsigned long long));
  SBDGB_CUDA(cudaMemsetAsync(mx, 0, 8 * sizeof(unsigned long long), s));
  auto absmax = [&](const double *x, size_t n, int slot) {
    if (n == 0) return;
    k_absmax<<<(unsigned)std::min<size_t>((n + 1023) / 1024, 1024), 256, 0, s>>>(x, n, mx + slot);
    count_launch(p.ctx);
  };
  auto pairmax = [&](const double *x, uint32_t n, int slot) {
    k_absmax_pairs<<<dim3((n + 1023) / 1024, p.npair), 256, 0, s>>>(x, n, mx + slot);
    count_launch(p.ctx);
  };
  absmax(p.A.val_s, p.A.ns, 0);
  absmax(p.A.val_d, p.A.nd, 1);
  pairmax(p.Jb, p.nb, 2);
  absmax(p.B.val_s, p.B.ns, 3);
  absmax(p.B.val_d, p.B.nd, 4);
  pairmax(p.Ja, p.na, 5);
  pairmax(p.Kp, (uint32_t)p.npair, 6);
  SBDGB_CUDA(cudaGetLastError());
  double v[8];
  SBDGB_CUDA(cudaMemcpyAsync(v, mx, sizeof(v), cudaMemcpyDeviceToHost, s));
  std::vector<uint32_t> os[2], od[2];
  for (int sp = 0; sp < 2; ++sp) {
    const SpinTables &T = sp == 0 ? p.A : p.B;
    os[sp].resize(T.n + 1);
    od[sp].resize(T.n + 1);
    SBDGB_CUDA(cudaMemcpyAsync(os[sp].data(), T.off_s, sizeof(uint32_t) * (T.n + 1), cudaMemcpyDeviceToHost, s));
    SBDGB_CUDA(cudaMemcpyAsync(od[sp].data(), T.off_d, sizeof(uint32_t) * (T.n + 1), cudaMemcpyDeviceToHost, s));
  }
  SBDGB_CUDA(cudaStreamSynchronize(s));
  auto exponent = [](double x) {
    int e = 0;
    std::frexp(x, &e);
    return e;
  };
  for (int i = 0; i < 7; ++i)
    if (!(v[i] < 0x1p100)) return false;
  std::vector<uint32_t> rows[2], ls[2], ld[2];
  const bool budget = p.ctx->budget != 0, fp = !(budget && p.ctx->pool);
  size_t bytes = 0;
  for (int sp = 0; sp < 2; ++sp) {
    const SpinTables &T = sp == 0 ? p.A : p.B;
    p.slab.ev[sp] = std::max(-100, exponent(std::max(v[3 * sp] + v[3 * sp + 2], v[3 * sp + 1])));
    auto ns = [&](uint32_t r) { return os[sp][r + 1] - os[sp][r]; };
    auto nd = [&](uint32_t r) { return od[sp][r + 1] - od[sp][r]; };
    rows[sp].resize((T.n + 31) / 32 * 32, ~0u);
    std::iota(rows[sp].begin(), rows[sp].begin() + T.n, 0u);
    std::stable_sort(rows[sp].begin(), rows[sp].begin() + T.n,
                     [&](uint32_t x, uint32_t y) {  // lists of equal length in groups, then by singles
                       const uint32_t gx = (nd(x) + kGroup - 1) / kGroup, gy = (nd(y) + kGroup - 1) / kGroup;
                       return gx != gy ? gx > gy : ns(x) > ns(y);
                     });
    ls[sp].assign(1, 0u);
    ld[sp].assign(1, 0u);
    for (size_t b = 0; b < rows[sp].size(); b += 32) {
      uint32_t ms = 0, md = 0;
      for (size_t i = b; i < b + 32 && i < T.n; ++i) {
        ms = std::max(ms, ns(rows[sp][i]));
        md = std::max(md, nd(rows[sp][i]));
        if (ns(rows[sp][i]) + nd(rows[sp][i]) > (uint32_t)fx::kMaxTerms) return false;
      }
      ls[sp].push_back(ls[sp].back() + (ms + kGroup - 1) / kGroup);
      ld[sp].push_back(ld[sp].back() + (md + kGroup - 1) / kGroup);
    }
    if ((uint64_t)std::max(ls[sp].back(), ld[sp].back()) * 64u >= (1ull << 32)) return false;  // 32-bit group indices
    bytes += 4 * rows[sp].size() + 8 * ls[sp].size() +
             32ull * (fp ? 24 : 16) * kGroup * (ls[sp].back() + ld[sp].back()) + 8ull * T.n;
  }
  for (uint32_t c = 0; ab && c < p.nb; ++c)  // up to four terms per beta single of a column
    if (4 * (os[1][c + 1] - os[1][c]) > (uint32_t)fx::kMaxTerms) return false;
  p.slab.ek = std::max(-100, exponent(v[6]));
  std::vector<uint2> items;
  if (ab) {
    items = slab_ab_items(p, os[0]);
    bytes += 4 * p.ab_entries + 8 * items.size();
  }
  if (budget && bytes > slab_room(p)) return false;
  for (int sp = 0; sp < 2; ++sp) {
    const SpinTables &T = sp == 0 ? p.A : p.B;
    const size_t nrow = rows[sp].size(), nsl = ls[sp].size() - 1;
    uint32_t *r = (uint32_t *)build.alloc(4 * nrow), *o = (uint32_t *)build.alloc(8 * (nsl + 1));
    SBDGB_CUDA(cudaMemcpyAsync(r, rows[sp].data(), 4 * nrow, cudaMemcpyHostToDevice, s));
    SBDGB_CUDA(cudaMemcpyAsync(o, ls[sp].data(), 4 * (nsl + 1), cudaMemcpyHostToDevice, s));
    SBDGB_CUDA(cudaMemcpyAsync(o + nsl + 1, ld[sp].data(), 4 * (nsl + 1), cudaMemcpyHostToDevice, s));
    p.slab.rows[sp] = r;
    p.slab.off[sp] = o;
    p.slab.nslices[sp] = (uint32_t)nsl;
    p.slab.groups[sp] = ls[sp].back() + ld[sp].back();
    p.slab.longest[sp] = 0;
    for (size_t i = 0; i < nsl; ++i)
      p.slab.longest[sp] =
          std::max(p.slab.longest[sp], kGroup * (ls[sp][i + 1] - ls[sp][i] + ld[sp][i + 1] - ld[sp][i]));
    p.slab.ent_s[sp] = (uint4 *)build.alloc(512ull * ls[sp].back());
    p.slab.val_s[sp] = (int4 *)build.alloc(1024ull * ls[sp].back());
    p.slab.ket_d[sp] = (uint4 *)build.alloc(512ull * ld[sp].back());
    p.slab.val_d[sp] = (int4 *)build.alloc(1024ull * ld[sp].back());
    p.slab.valf_s[sp] = (float4 *)build.alloc(512ull * ls[sp].back());
    p.slab.valf_d[sp] = (float4 *)build.alloc(512ull * ld[sp].back());
    if (fp) {
      p.slab.fp_s[sp] = (double2 *)build.alloc(1024ull * ls[sp].back());
      p.slab.fp_d[sp] = (double2 *)build.alloc(1024ull * ld[sp].back());
    }
    p.slab.mask[sp] = (uint64_t *)build.alloc(8ull * T.n);
    if (T.ns && !budget) {  // the Coulomb table this spin's singles read, where memory is not counted
      const size_t nj = (size_t)p.npair * (sp == 0 ? p.nb : p.na);
      p.slab.Jfx[sp] = (int2 *)build.alloc(8 * nj);
      k_slab_coulomb<<<(unsigned)std::min<size_t>((nj + 255) / 256, 4096), 256, 0, s>>>(
          sp == 0 ? p.Jb : p.Ja, nj, fx::kVBits - p.slab.ev[sp], p.slab.Jfx[sp]);
      count_launch(p.ctx);
    }
    // the order of the entries (two scratch words each)
    uint32_t *tmp = (uint32_t *)tmp_alloc(p.ctx, 8ull * (T.ns + T.nd));
    build.tmps.push_back(tmp);
    uint32_t *order_s = tmp, *order_d = order_s + T.ns, *next = order_d + T.nd;
    k_slab_order<<<(unsigned)nsl, 32, 0, s>>>(T.off_s, T.ket_s, r, next, order_s);
    k_slab_order<<<(unsigned)nsl, 32, 0, s>>>(T.off_d, T.ket_d, r, next, order_d);
    k_slab_fill<<<(unsigned)nsl, 128, 0, s>>>(T, r, o, o + nsl + 1, order_s, order_d, p.npair, p.slab.ev[sp],
                                              p.slab.ent_s[sp], p.slab.val_s[sp], p.slab.ket_d[sp], p.slab.val_d[sp],
                                              p.slab.valf_s[sp], p.slab.valf_d[sp], p.slab.fp_s[sp],
                                              p.slab.fp_d[sp]);
    k_slab_masks<<<(T.n + 127) / 128, 128, 0, s>>>(sp == 0 ? p.astr : p.bstr, T.n, sp, p.slab.mask[sp]);
    count_launch(p.ctx, 4);
  }
  if (ab) {
    const uint32_t base = slab_ab_base(p);
    const uint32_t mine = (p.n_ab_slices + base - 1) / base;
    const uint32_t rounds = (mine + kSlabAbThreads / 32 - 1) / (kSlabAbThreads / 32);
    p.slab.ab_warps = std::max<uint32_t>(4, (mine + rounds - 1) / rounds);
    p.slab.n_ab_items = (uint32_t)items.size();
    p.slab.h_items = items;
    p.slab.ab_items = (uint2 *)build.alloc(8 * items.size());
    SBDGB_CUDA(cudaMemcpyAsync(p.slab.ab_items, items.data(), 8 * items.size(), cudaMemcpyHostToDevice, s));
    p.slab.ab_ent = (uint32_t *)build.alloc(4 * p.ab_entries);
    SBDGB_CUDA(cudaMemcpyAsync(p.slab.ab_ent, p.ab_ent, 4 * p.ab_entries, cudaMemcpyDeviceToDevice, s));
    k_slab_ab_order<<<p.n_ab_slices, 32, 0, s>>>(p.ab_slice, (uint32_t)p.npair, p.nb, p.slab.ab_ent);
    count_launch(p.ctx);
  }
  SBDGB_CUDA(cudaGetLastError());
  SBDGB_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
  return true;
}

}  // namespace

// Builds the sliced tables on first use.  False where the kernels do not apply
// to 8-byte elements or there is no room for their tables.
bool slab_prepare(Problem &p, cudaStream_t s) {
  if (p.slab.state >= 0) return p.slab.state == 1;
  SlabBuild build(p, s);
  try {
    build.done = slab_build(p, build, s);
  } catch (const Error &e) {
    if (e.status != SBDGB_E_NOMEM) throw;
  }
  if (build.done) p.slab.state = 1;
  return build.done;
}

namespace {

// Columns a CTA (K), CTAs that share a column group and its staging (parts) and
// warps a CTA, by the cycles of the busiest SM.  Warp instructions: about 1.1 per
// staged element and 0.5 per staged Coulomb value (a column, a row), 10 + 4 K per
// step of a slice (4 + 1.25 K in FP32), 70 (20) per column and slice at its end;
// 1.6 of them a cycle.  A CTA lasts at least as long as its longest slice, at
// about 120 cycles a step.  An SM holds 24 warps (80 registers a thread) in CTAs
// of 8, 12 or 24.  (Beta sweep, ms, against one rule for the K that fits and as
// many parts as fill three waves: 2011 x 1703 strings double-float 0.228, here
// 0.203; FP32 0.157, 0.103.)
struct SlabShape {
  int K;
  uint32_t groups, parts, warps;
  size_t smem;
};
SlabShape slab_shape(const Problem &p, int sp, uint32_t n, uint32_t m, int npair, int element, int Kmax, int Kmin,
                     int nvec) {
  SlabShape best{};
  const size_t limit = max_smem();
  int sms = 0;
  SBDGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.ctx->device));
  const uint32_t nslices = p.slab.nslices[sp];
  double cost = 0.0;
  for (int K = Kmax; K >= Kmin; K >>= 1) {
    const size_t smem = slab_smem_bytes(element, K, n, npair);
    if (smem > limit) continue;
    const uint32_t groups = (m + K - 1) / K;
    const uint32_t resident = smem <= limit / 3 ? 3 : smem <= limit / 2 ? 2 : 1, slots = resident * sms;
    const double stage = (1.1 * n + 0.5 * npair) * K * (element == 8 ? 1.0 : 0.5);
    const double work = 4.0 * p.slab.groups[sp] * (element == 8 ? 10.0 + 4.0 * K : 4.0 + 1.25 * K) +
                        nslices * K * (element == 8 ? 70.0 : 20.0);
    for (uint32_t parts = 1; parts <= std::min<uint32_t>(nslices, 16); ++parts) {
      const uint32_t full = kSlabThreads / 32 / resident;
      const uint32_t warps = std::max<uint32_t>(2, std::min(full, (nslices + parts - 1) / parts));
      const uint32_t ctas = groups * parts * nvec, waves = (ctas + slots - 1) / slots;
      // rounds: the slices of a part that its warps take one after another
      const double rounds = (double)((nslices + parts - 1) / parts + warps - 1) / warps;
      const double even = std::max(1.0, std::floor(rounds) * warps * parts / nslices);
      // CTAs of the busiest SM at once; few of them leave it waiting on latency
      const double live = std::min<double>(resident, (double)((ctas + sms - 1) / sms));
      const double busy = std::min(1.0, live * warps / 12.0);
      // (a shared group's diagonal is gathered at the end instead of streamed while staging)
      const double c = (parts > 1 ? 1.2 : 1.0) * waves * std::max(live * (stage + work / parts * even) / (1.6 * busy),
                                        stage / (0.4 * warps) + 120.0 * p.slab.longest[sp]);
      if (best.K == 0 || c < 0.97 * cost) {
        cost = c;
        best = {K, groups, parts, warps, smem};
      }
    }
  }
  SBDGB_REQUIRE(best.K > 0, SBDGB_E_UNSUPPORTED, "sigma's columns do not fit in shared memory");  // slab_fits
  return best;
}

template <typename K, typename A>
void go_slab(K k, const A &a, dim3 grid, uint32_t warps, size_t smem, cudaStream_t s) {
  ensure_dynamic_smem((const void *)k, smem);
  prefer_shared_carveout((const void *)k);
  k<<<grid, warps * 32, smem, s>>>(a);
}

SlabSpin slab_spin(const Problem &p, int sp) {
  SlabSpin t{};
  t.rows = p.slab.rows[sp];
  t.off_s = p.slab.off[sp];
  t.off_d = p.slab.off[sp] + p.slab.nslices[sp] + 1;
  t.ent_s = p.slab.ent_s[sp];
  t.val_s = p.slab.val_s[sp];
  t.ket_d = p.slab.ket_d[sp];
  t.val_d = p.slab.val_d[sp];
  t.fp_s = reinterpret_cast<const int4 *>(p.slab.fp_s[sp]);
  t.fp_d = reinterpret_cast<const int4 *>(p.slab.fp_d[sp]);
  t.nslices = p.slab.nslices[sp];
  return t;
}

template <typename T, bool kAlpha>
SlabArgs<T> slab_args(const Problem &p, const Args<T> &x, int add, int diag, int eta, int guard) {
  constexpr int sp = kAlpha ? 0 : 1;
  SlabArgs<T> a{};
  a.C = x.C;
  a.S = x.S;
  if constexpr (std::is_same<T, double>::value) {
    a.hii = x.hii;
  } else {
    a.hii = x.hii_df;
    a.shift = x.shift_df;
  }
  a.t = slab_spin(p, sp);
  a.Jo = kAlpha ? p.Jb : p.Ja;
  a.Jt = kAlpha ? x.Jb : x.Ja;
  a.Jfx = p.slab.Jfx[sp];
  a.rowstr = kAlpha ? p.astr : p.bstr;
  a.colmask = p.slab.mask[1 - sp];
  a.n = kAlpha ? p.na : p.nb;
  a.m = kAlpha ? p.nb : p.na;
  a.nb = p.nb;
  a.npair = (kAlpha ? p.A.ns : p.B.ns) ? p.npair : 0;
  a.ev = p.slab.ev[sp];
  a.eta = eta;
  a.guard = guard;
  a.add = add;
  a.diag = diag;
  a.parts = 1;
  a.staged_diag = diag && !kAlpha;
  a.vec = p.nb % 2 == 0 && ((uintptr_t)x.S & 15u) == 0;
  return a;
}

template <typename T, bool kAlpha>
void launch_slab(const Problem &p, const Args<T> &x, int add, int diag, int eta, int guard, cudaStream_t s) {
  SlabArgs<T> a = slab_args<T, kAlpha>(p, x, add, diag, eta, guard);
  const SlabShape c = slab_shape(p, kAlpha ? 0 : 1, a.n, a.m, a.npair, 8, 4, kSlabMinK, 1);
  a.parts = c.parts;
  a.staged_diag = a.staged_diag && c.parts == 1;
  const dim3 g(c.groups, c.parts);
  switch (c.K) {
    case 4: go_slab(k_slab<T, 4, kAlpha>, a, g, c.warps, c.smem, s); break;
    case 2: go_slab(k_slab<T, 2, kAlpha>, a, g, c.warps, c.smem, s); break;
    default: go_slab(k_slab<T, 1, kAlpha>, a, g, c.warps, c.smem, s); break;
  }
  count_launch(p.ctx);
  SBDGB_CUDA(cudaGetLastError());
}

template <bool kAlpha>
SlabArgsF slab_args_f32(const Problem &p, const Args<float> &x, int add, int diag, int eta, int join) {
  constexpr int sp = kAlpha ? 0 : 1;
  SlabArgsF a{};
  a.hii_df = x.hii_df;
  a.hii_f = x.hii_f;
  a.shift = x.shift_df;
  a.t = slab_spin(p, sp);
  a.val_s = p.slab.valf_s[sp];
  a.val_d = p.slab.valf_d[sp];
  a.Jo = kAlpha ? x.Jb : x.Ja;
  a.rowstr = kAlpha ? p.astr : p.bstr;
  a.colmask = p.slab.mask[1 - sp];
  a.n = kAlpha ? p.na : p.nb;
  a.m = kAlpha ? p.nb : p.na;
  a.nb = p.nb;
  a.npair = (kAlpha ? p.A.ns : p.B.ns) ? p.npair : 0;
  a.eta = eta;
  a.add = add;
  a.diag = diag;
  a.join = join;
  a.parts = 1;
  return a;
}

template <bool kAlpha>
void launch_slab_f32(const Problem &p, const Args<float> &x, const float *const *C, float *const *S, int nvec, int add,
                     int diag, int eta, cudaStream_t s) {
  SlabArgsF a = slab_args_f32<kAlpha>(p, x, add, diag, eta, eta);  // (the solvers: the block ordering)
  a.vec = p.nb % 4 == 0;
  for (int v = 0; v < nvec; ++v) {
    a.C[v] = C[v];
    a.S[v] = S[v];
    a.vec = a.vec && ((uintptr_t)S[v] & 15u) == 0;
  }
  const SlabShape c = slab_shape(p, kAlpha ? 0 : 1, a.n, a.m, a.npair, 4, 8, kSlabMinKF, nvec);
  a.parts = c.parts;
  const dim3 g(c.groups, c.parts, nvec);
  if (c.K == 8)
    go_slab(k_slab_f32<8, kAlpha>, a, g, c.warps, c.smem, s);
  else
    go_slab(k_slab_f32<4, kAlpha>, a, g, c.warps, c.smem, s);
  count_launch(p.ctx);
  SBDGB_CUDA(cudaGetLastError());
}

template <typename T>
SlabAbArgs<T> slab_ab_args(const Problem &p, const Args<T> &x, int eta, int guard) {
  SlabAbArgs<T> a{};
  a.C = x.C;
  a.S = x.S;
  a.astr = p.astr;
  a.colmask = p.slab.mask[1];
  a.off = p.A.off_s;
  a.ket = p.A.ket_s;
  a.code = p.A.code_s;
  a.Kp = p.Kp;
  a.Kt = x.Kp;
  a.items = p.slab.ab_items;
  a.cols = p.ab_cols;
  a.slice = p.ab_slice;
  a.ent = p.slab.ab_ent;
  a.nslices = p.n_ab_slices;
  a.nb = p.nb;
  a.npair = p.npair;
  a.ek = p.slab.ek;
  a.eta = eta;
  a.guard = guard;
  return a;
}

template <typename T>
void launch_slab_ab(const Problem &p, const Args<T> &x, int eta, int guard, cudaStream_t s) {
  const SlabAbArgs<T> a = slab_ab_args<T>(p, x, eta, guard);
  const uint32_t warps = p.slab.ab_warps;
  const dim3 g(p.slab.n_ab_items);
  if (!slab_ab_sum(p))
    go_slab(k_slab_ab<T, 2, false>, a, g, warps, slab_ab_smem_bytes(p, 2, false), s);
  else if (slab_ab_smem_bytes(p, 4, true) <= max_smem() / 2)
    go_slab(k_slab_ab<T, 4, true>, a, g, warps, slab_ab_smem_bytes(p, 4, true), s);
  else
    go_slab(k_slab_ab<T, 2, true>, a, g, warps, slab_ab_smem_bytes(p, 2, true), s);
  count_launch(p.ctx);
  SBDGB_CUDA(cudaGetLastError());
}

SlabAbArgsF slab_ab_args_f32(const Problem &p, const Args<float> &x, int eta) {
  SlabAbArgsF a{};
  a.astr = p.astr;
  a.colmask = p.slab.mask[1];
  a.off = p.A.off_s;
  a.ket = p.A.ket_s;
  a.code = p.A.code_s;
  a.Kp = x.Kp;
  a.items = p.slab.ab_items;
  a.cols = p.ab_cols;
  a.slice = p.ab_slice;
  a.ent = p.slab.ab_ent;
  a.nslices = p.n_ab_slices;
  a.nb = p.nb;
  a.npair = p.npair;
  a.eta = eta;
  return a;
}

void launch_slab_ab_f32(const Problem &p, const Args<float> &x, const float *const *C, float *const *S, int nvec,
                        int eta, cudaStream_t s) {
  SlabAbArgsF a = slab_ab_args_f32(p, x, eta);
  for (int v = 0; v < nvec; ++v) {
    a.C[v] = C[v];
    a.S[v] = S[v];
  }
  const uint32_t warps = p.slab.ab_warps;
  go_slab(k_slab_ab_f32, a, dim3(p.slab.n_ab_items, 1, nvec), warps, slab_ab_smem_bytes_f32(p.nb, p.npair), s);
  count_launch(p.ctx);
  SBDGB_CUDA(cudaGetLastError());
}

}  // namespace

// One FP64 or double-float product (slab_prepare has returned true): no
// allocation and no scratch, so products of one problem may overlap on several
// streams.
template <typename T>
void sigma_slab(const Problem &p, const Args<T> &x, bool block, cudaStream_t s) {
  // The solvers' products (the block ordering) need no guard: what a solve returns is
  // held to a norm, and the norm of the error is below the FP64 sums'.
  const int eta = block ? 0 : 1, guard = eta;
  const bool alpha = p.A.ns + p.A.nd > 0, beta = p.B.ns + p.B.nd > 0;
  if (alpha || !beta) launch_slab<T, true>(p, x, x.accumulate, !beta, eta, guard, s);
  if (p.A.ns > 0 && p.B.ns > 0) launch_slab_ab<T>(p, x, eta, guard, s);
  if (beta) launch_slab<T, false>(p, x, x.accumulate || alpha, 1, eta, guard, s);
}
template void sigma_slab<double>(const Problem &, const Args<double> &, bool, cudaStream_t);
template void sigma_slab<dfloat>(const Problem &, const Args<dfloat> &, bool, cudaStream_t);

// FP32 products of nvec <= 4 vectors.
void sigma_slab_f32(const Problem &p, const Args<float> &x, const float *const *C, float *const *S, int nvec,
                    bool block, cudaStream_t s) {
  const int eta = block ? 0 : 1;
  const bool alpha = p.A.ns + p.A.nd > 0, beta = p.B.ns + p.B.nd > 0;
  if (alpha || !beta) launch_slab_f32<true>(p, x, C, S, nvec, 0, !beta, eta, s);
  if (p.A.ns > 0 && p.B.ns > 0) launch_slab_ab_f32(p, x, C, S, nvec, eta, s);
  if (beta) launch_slab_f32<false>(p, x, C, S, nvec, alpha, 1, eta, s);
}

// ---- the batched solver's products ----------------------------------------------------

namespace {
constexpr int kManyK = 4, kManyKF = 8;

template <typename A>
A *to_device(Ctx *c, std::vector<void *> &tmps, const std::vector<A> &v, cudaStream_t s) {
  A *d = (A *)tmp_alloc(c, sizeof(A) * v.size());
  tmps.push_back(d);
  SBDGB_CUDA(cudaMemcpyAsync(d, v.data(), sizeof(A) * v.size(), cudaMemcpyHostToDevice, s));
  return d;
}
}  // namespace

// False when some problem's tables do not apply or the CTAs would not fit.
bool slab_batch_fits(Problem **ps, int count, cudaStream_t s) {
  const size_t limit = max_smem();
  for (int i = 0; i < count; ++i) {
    Problem &p = *ps[i];
    const uint32_t n = std::max(p.na, p.nb);
    if (p.A.ns + p.A.nd == 0 || p.B.ns + p.B.nd == 0) return false;
    if ((size_t)8 * kManyK * (n + 1 + p.npair + 1) > limit || slab_ab_smem_bytes(p, 4, true) > limit) return false;
    if (!slab_prepare(p, s)) return false;
  }
  return true;
}

template <typename T>
void slab_batch_plan(SlabBatch &b, Ctx *c, Problem **ps, const sdev::Args<T> *args, int count,
                     const SlabBatchState &state, int nvec, cudaStream_t s) {
  constexpr bool kF32 = std::is_same<T, float>::value;
  using S = typename std::conditional<kF32, SlabArgsF, SlabArgs<double>>::type;
  using AB = typename std::conditional<kF32, SlabAbArgsF, SlabAbArgs<double>>::type;
  std::vector<S> sa, sb;
  std::vector<AB> ab;
  std::vector<uint4> ia, ib, iab;
  b.state = state;
  b.nvec = nvec;
  for (int i = 0; i < count; ++i) {
    const Problem &p = *ps[i];
    if constexpr (kF32) {
      sa.push_back(slab_args_f32<true>(p, args[i], 0, 0, 1, 0));
      sb.push_back(slab_args_f32<false>(p, args[i], 1, 1, 1, 0));
      ab.push_back(slab_ab_args_f32(p, args[i], 1));
    } else {
      sa.push_back(slab_args<double, true>(p, args[i], 0, 0, 1, 0));
      sb.push_back(slab_args<double, false>(p, args[i], 1, 1, 1, 0));
      ab.push_back(slab_ab_args<double>(p, args[i], 1, 0));
      sa.back().vec = sb.back().vec = 0;  // a column of the basis may start anywhere
    }
    const int K = kF32 ? kManyKF : kManyK, el = kF32 ? 4 : 8;
    for (uint32_t g = 0; g < (p.nb + K - 1) / K; ++g) ia.push_back(make_uint4(i, g, 0, 0));
    for (uint32_t g = 0; g < (p.na + K - 1) / K; ++g) ib.push_back(make_uint4(i, g, 0, 0));
    for (const uint2 &it : p.slab.h_items) iab.push_back(make_uint4(i, it.x, it.y, 0));
    auto smem = [&](uint32_t n, uint64_t ns) { return (size_t)el * K * (n + 1 + (ns ? p.npair + 1 : 0)); };
    b.smem[0] = std::max(b.smem[0], smem(p.na, p.A.ns));
    b.smem[1] = std::max(b.smem[1], smem(p.nb, p.B.ns));
    b.smem[2] = std::max(b.smem[2], kF32 ? slab_ab_smem_bytes_f32(p.nb, p.npair) : slab_ab_smem_bytes(p, 4, true));
  }
  b.args[0] = to_device(c, b.tmps, sa, s);
  b.args[1] = to_device(c, b.tmps, sb, s);
  b.args[2] = to_device(c, b.tmps, ab, s);
  b.items[0] = to_device(c, b.tmps, ia, s);
  b.items[1] = to_device(c, b.tmps, ib, s);
  b.items[2] = to_device(c, b.tmps, iab, s);
  b.n[0] = (uint32_t)ia.size();
  b.n[1] = (uint32_t)ib.size();
  b.n[2] = (uint32_t)iab.size();
  SBDGB_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
  auto limit = [&](auto k, int i) {
    ensure_dynamic_smem((const void *)k, b.smem[i]);
    prefer_shared_carveout((const void *)k);
  };
  if constexpr (kF32) {
    limit(k_slab_many_f32<kManyKF, true>, 0);
    limit(k_slab_many_f32<kManyKF, false>, 1);
    limit(k_slab_ab_many_f32, 2);
  } else {
    limit(k_slab_many<kManyK, true>, 0);
    limit(k_slab_many<kManyK, false>, 1);
    limit(k_slab_ab_many<4>, 2);
  }
}
template void slab_batch_plan<double>(SlabBatch &, Ctx *, Problem **, const sdev::Args<double> *, int,
                                      const SlabBatchState &, int, cudaStream_t);
template void slab_batch_plan<float>(SlabBatch &, Ctx *, Problem **, const sdev::Args<float> *, int,
                                     const SlabBatchState &, int, cudaStream_t);

template <typename T>
void slab_batch_sigma(const SlabBatch &b, cudaStream_t s) {
  constexpr bool kF32 = std::is_same<T, float>::value;
  using S = typename std::conditional<kF32, SlabArgsF, SlabArgs<double>>::type;
  using AB = typename std::conditional<kF32, SlabAbArgsF, SlabAbArgs<double>>::type;
  auto sweep = [&](int i) { return SlabMany<S>{(const S *)b.args[i], b.items[i], b.state}; };
  const SlabMany<AB> ab{(const AB *)b.args[2], b.items[2], b.state};
  const dim3 ga(b.n[0], b.nvec), gb(b.n[1], b.nvec), gab(b.n[2], b.nvec);
  if constexpr (kF32) {
    k_slab_many_f32<kManyKF, true><<<ga, kManyThreads, b.smem[0], s>>>(sweep(0));
    if (b.n[2]) k_slab_ab_many_f32<<<gab, kManyThreads, b.smem[2], s>>>(ab);
    k_slab_many_f32<kManyKF, false><<<gb, kManyThreads, b.smem[1], s>>>(sweep(1));
  } else {
    k_slab_many<kManyK, true><<<ga, kManyThreads, b.smem[0], s>>>(sweep(0));
    if (b.n[2]) k_slab_ab_many<4><<<gab, kManyThreads, b.smem[2], s>>>(ab);
    k_slab_many<kManyK, false><<<gb, kManyThreads, b.smem[1], s>>>(sweep(1));
  }
}
template void slab_batch_sigma<double>(const SlabBatch &, cudaStream_t);
template void slab_batch_sigma<float>(const SlabBatch &, cudaStream_t);

}  // namespace sbdgb
