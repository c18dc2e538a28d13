// One- and two-particle reduced density matrices of a vector (Correlation,
// chemistry/tpb/correlation.h:379-640, element rules chemistry/basic/
// correlation.h:17-299), in the reference's layout:
//
//   one[s][i + L*j]                      s = spin of the pair (0 alpha, 1 beta)
//   two[s1 + 2*s2][a + L*b + L^2*c + L^3*d]
//
// The reference visits every (bra, ket) pair of the excitation lists and adds
// each element's contributions with atomics.  Here the sums over the
// spectator string are taken first:
//   - same-spin single (bra -> ket, orbitals i -> a): the weighted overlap
//     s = sum_spectator W[bra] W[ket] (+-1) and, per opposite-spin orbital q,
//     u[q] = the same sum restricted to spectators with q occupied; the
//     contributions of the occupied same-spin orbitals of the bra depend on
//     s alone, those of the opposite-spin orbitals on u[q];
//   - same-spin double: s alone (four entries);
//   - alpha single x beta single: the sum over all pairs with the same four
//     orbitals (singles of both spins sorted by their two orbitals, so that a
//     thread's sum is one quadruple's), scattered once at the end;
//   - the diagonal (ZeroDiffCorrelation): string weights for the same-spin
//     pairs and Y = (W o W) O_beta, M = O_alpha^T Y for the alpha-beta pairs.
// Phases are the ones of the sigma kernels (same tables, same masks); the
// same-spin doubles recompute theirs from the four orbitals.
#include <algorithm>

#include <numeric>

#include "common.cuh"
#include "fx.cuh"
#include "sigma_dev.cuh"

namespace sbdgb {

void transpose_fp64(Problem &p, const double *in, double *out, uint32_t R, uint32_t Cn, cudaStream_t s);
void string_norms(Problem &p, const double *W, double *r, double *c, cudaStream_t s);
const double *device_vector(Problem &p, const double *W, cudaStream_t s);

namespace {

constexpr int kT = 256;
constexpr int kMaxL = 64;

__device__ __forceinline__ size_t q4(int L, int a, int b, int c, int d) {
  return (size_t)a + (size_t)L * ((size_t)b + (size_t)L * ((size_t)c + (size_t)L * (size_t)d));
}

struct RdmArgs {
  const uint64_t *astr, *bstr;
  uint32_t na, nb;
  int L;
  const double *W;   // [ia][ib]
  const double *WT;  // [ib][ia]
  double *one;       // 2 L^2
  double *two;       // 4 L^4 (null: one-particle part only)
  double *R;         // L^4 alpha-beta sums [oi_a, oa_a, oj_b, ob_b]
  SpinTables A, B;
};

// Same-spin singles of spin S, one warp per pair: s and u[q] over the
// spectators.  Of 32 spectators each lane forms one's product, as an integer of
// twice 57 bits on the scale of the largest (exact for products down to 2^-61 of
// it; further apart, FP64 sums), and the lanes then add them all, lane q those
// with orbital q: integer additions (62 a clock and SM) where FP64 ones take 16
// clocks a warp.  Before, every spectator added to its orbitals' sums by FP64
// atomics in shared memory (compare-and-swap loops on 8 of 24 places): 1.3 ms
// a spin for 301 x 420 strings of norb 24, 22 us with one word, 34 here.
struct Wide57 {
  unsigned long long hi, lo;  // hi 2^57 + lo on the scale of the second word, both with the sign
};
// x 2^s in two words: |x 2^s| <= 2^57, and exact for s + (x's exponent) >= -4.
__device__ __forceinline__ Wide57 two_words(double x, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  const unsigned long long m = (b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
  const int sh = max((e ? e : 1) - 1075 + s, -57);  // (zero: anything); at most 4
  const long long h = (long long)(sh >= 0 ? m << sh : m >> -sh);
  const long long l = (long long)(sh >= 0 ? 0ull : m << (57 + sh) & ((1ull << 57) - 1ull));
  const long long sg = (long long)b >> 63;
  return {(unsigned long long)((h ^ sg) - sg), (unsigned long long)((l ^ sg) - sg)};
}
template <int S>
__global__ void __launch_bounds__(kT) k_rdm_singles(RdmArgs a) {
  const SpinTables &T = S == 0 ? a.A : a.B;
  const uint64_t *same = S == 0 ? a.astr : a.bstr;
  const uint64_t *opp = S == 0 ? a.bstr : a.astr;
  const double *Wr = S == 0 ? a.W : a.WT;  // rows indexed by this spin's strings
  const uint32_t nopp = S == 0 ? a.nb : a.na;
  const int L = a.L;
  __shared__ ulonglong2 sv[kT / 32][32];
  __shared__ unsigned long long svl[kT / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool two = a.two != nullptr;
  for (uint64_t p = (uint64_t)blockIdx.x * (kT / 32) + warp; p < T.ns; p += (uint64_t)gridDim.x * (kT / 32)) {
    const uint32_t bra = T.bra_s[p], ket = T.ket_s[p], code = T.code_s[p];
    const uint64_t mask = T.mask_s[p];
    const int oi = code & 0xff, oa = (code >> 8) & 0xff;
    const double *rb = Wr + (size_t)bra * nopp, *rk = Wr + (size_t)ket * nopp;
    double u0 = 0.0, u1 = 0.0, ssum = 0.0;  // orbitals lane and lane + 32, and all
    if (!two) {  // s alone, each lane its spectators
#pragma unroll 4
      for (uint32_t o = lane; o < nopp; o += 32) {
        const uint32_t ph = (__popcll(__ldg(opp + o) & mask) ^ (code >> 31)) & 1u;
        ssum += sdev::flip(__ldg(rb + o) * __ldg(rk + o), ph);
      }
      for (int d = 16; d > 0; d >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, d);
      if (lane == 0) atomicAdd(&a.one[(size_t)S * L * L + oi + (size_t)L * oa], ssum);
      continue;
    }
    for (uint32_t o0 = 0; o0 < nopp; o0 += 32) {
      const uint32_t o = o0 + lane;
      const uint64_t os = o < nopp ? __ldg(opp + o) : 0ull;
      double v = o < nopp ? __ldg(rb + o) * __ldg(rk + o) : 0.0;
      v = sdev::flip(v, (__popcll(os & mask) ^ (code >> 31)) & 1u);
      const uint32_t hi = (uint32_t)__double2hiint(v) & 0x7fffffffu, key = hi ? hi : (__double2loint(v) ? 1u : 0u);
      const uint32_t top = __reduce_max_sync(0xffffffffu, key);
      if (top == 0u) continue;  // all zero
      const uint32_t low = __reduce_min_sync(0xffffffffu, key - 1u) + 1u;  // of the nonzeros
      const int ex = fx::exponent_of(top, true);
      const bool fixed = ex != fx::kBad && (top >> 20) - (low >> 20) <= 60u;
      Wide57 f{(unsigned long long)__double_as_longlong(v), 0ull};
      if (fixed) f = two_words(v, fx::kVBits - ex);
      __syncwarp();
      sv[warp][lane] = make_ulonglong2(f.hi, os);
      svl[warp][lane] = f.lo;
      __syncwarp();
      if (fixed) {
        long long a0 = 0, a1 = 0, as = 0, b0 = 0, b1 = 0, bs = 0;  // 32 terms of 57 bits
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
          const ulonglong2 x = sv[warp][i];
          const long long t = (long long)x.x, l = (long long)svl[warp][i];
          as += t;
          bs += l;
          if (x.y >> lane & 1ull) {
            a0 += t;
            b0 += l;
          }
          if (L > 32 && (x.y >> (lane + 32) & 1ull)) {
            a1 += t;
            b1 += l;
          }
        }
        const double unit = scalbn(1.0, ex - fx::kVBits), low_unit = unit * 0x1p-57;
        ssum += fma((double)as, unit, (double)bs * low_unit);
        u0 += fma((double)a0, unit, (double)b0 * low_unit);
        if (L > 32) u1 += fma((double)a1, unit, (double)b1 * low_unit);
      } else {
        for (int i = 0; i < 32; ++i) {
          const ulonglong2 x = sv[warp][i];
          const double t = __longlong_as_double((long long)x.x);
          ssum += t;
          if (x.y >> lane & 1ull) u0 += t;
          if (L > 32 && (x.y >> (lane + 32) & 1ull)) u1 += t;
        }
      }
    }
    if (lane == 0) atomicAdd(&a.one[(size_t)S * L * L + oi + (size_t)L * oa], ssum);
    const uint64_t bs = same[bra];
    double *blk = a.two + (size_t)(3 * S) * L * L * L * L;  // s1 = s2 = S
    double *b1 = a.two + (size_t)(S + 2 * (1 - S)) * L * L * L * L;
    double *b2 = a.two + (size_t)((1 - S) + 2 * S) * L * L * L * L;
    for (int h = 0; h < 2; ++h) {
      const int q = lane + 32 * h;
      if (q >= L) continue;
      if ((bs >> q & 1ull) && q != oi && ssum != 0.0) {  // same-spin electrons (q = oi: its four terms cancel)
        atomicAdd(&blk[q4(L, oa, q, oi, q)], ssum);
        atomicAdd(&blk[q4(L, q, oa, q, oi)], ssum);
        atomicAdd(&blk[q4(L, oa, q, q, oi)], -ssum);
        atomicAdd(&blk[q4(L, q, oa, oi, q)], -ssum);
      }
      const double u = h ? u1 : u0;  // opposite-spin spectator orbitals
      if (u != 0.0) {
        atomicAdd(&b1[q4(L, oa, q, oi, q)], u);
        atomicAdd(&b2[q4(L, q, oa, q, oi)], u);
      }
    }
  }
}

// Singles counted by their orbital pair oi L + oa, and sorted by it: a[] = entry
// index (alpha), (bra, ket | phase << 31) (beta).
__global__ void k_rdm_types(SpinTables T, int L, uint32_t *__restrict__ count) {
  for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < T.ns; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t code = T.code_s[p];
    atomicAdd(&count[(code & 0xff) * L + ((code >> 8) & 0xff)], 1u);
  }
}
__global__ void k_rdm_sort(SpinTables T, int L, uint32_t *__restrict__ next, uint2 *__restrict__ out) {
  for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < T.ns; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t code = T.code_s[p];
    const uint32_t at = atomicAdd(&next[(code & 0xff) * L + ((code >> 8) & 0xff)], 1u);
    out[at] = make_uint2(T.bra_s[p], T.ket_s[p] | (code & 0x80000000u));
  }
}

// Alpha single x beta single.  A CTA takes up to kAbPairs alpha singles of one
// orbital pair, stages the bra and ket rows of W (signed by eta, so that an
// element's phase is the two singles' own) and, where they fit, the sorted beta
// singles; a thread then sums one beta orbital pair's entries over them: one
// atomic addition per quadruple and CTA.  Beta orbital pairs are dealt by
// decreasing length.
constexpr uint32_t kAbPairs = 8;
struct RdmAb {
  const uint64_t *astr, *bstr;
  const double *W;
  double *R;
  const uint2 *pa, *pb;        // sorted singles: (bra, ket | phase << 31)
  const uint4 *chunks;         // (orbital pair, first, count, -) of pa
  const uint4 *types;          // (orbital pair, first, count, -) of pb, longest first
  uint32_t ntypes, npb, nb;
  int L;
  int rows_smem, ent_smem;     // rows and entries staged in shared memory
};
__device__ __forceinline__ double rdm_signed(const RdmAb &a, uint32_t row, uint32_t ib) {
  return sdev::flip(__ldg(a.W + (size_t)row * a.nb + ib), sdev::eta_parity(__ldg(a.astr + row), __ldg(a.bstr + ib)));
}
__global__ void __launch_bounds__(kT) k_rdm_ab(RdmAb a) {
  extern __shared__ __align__(16) unsigned char rdm_smem[];
  double2 *rows = reinterpret_cast<double2 *>(rdm_smem);  // [nb]: bra and ket row
  uint2 *sent = reinterpret_cast<uint2 *>(rows + (a.rows_smem ? a.nb : 0));
  const uint4 ch = __ldg(a.chunks + blockIdx.x);
  const uint2 *ent = a.pb;
  if (a.ent_smem) {
    for (uint32_t e = threadIdx.x; e < a.npb; e += kT) sent[e] = __ldg(a.pb + e);
    ent = sent;
  }
  constexpr int kPer = 16;  // orbital pairs a thread holds: L^2 <= 4096
  double acc[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) acc[i] = 0.0;
  for (uint32_t k = 0; k < ch.z; ++k) {
    const uint2 pr = __ldg(a.pa + ch.y + k);
    const uint32_t bra = pr.x, ket = pr.y & 0x7fffffffu, sg = pr.y >> 31;
    if (a.rows_smem) {
      __syncthreads();
      for (uint32_t c = threadIdx.x; c < a.nb; c += kT)
        rows[c] = make_double2(sdev::flip(rdm_signed(a, bra, c), sg), rdm_signed(a, ket, c));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const uint32_t t = threadIdx.x + kT * i;
      if (t >= a.ntypes) break;
      const uint4 ty = __ldg(a.types + t);
      double s = acc[i];
      for (uint32_t e = ty.y; e < ty.y + ty.z; ++e) {
        const uint2 w = ent[e];
        const uint32_t jb = w.y & 0x7fffffffu;
        const double x = a.rows_smem ? rows[w.x].x : sdev::flip(rdm_signed(a, bra, w.x), sg);
        const double y = a.rows_smem ? rows[jb].y : rdm_signed(a, ket, jb);
        s = fma(sdev::flip(x, w.y >> 31), y, s);
      }
      acc[i] = s;
    }
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const uint32_t t = threadIdx.x + kT * i;
    if (t >= a.ntypes) break;
    if (acc[i] != 0.0) atomicAdd(&a.R[(size_t)ch.x * a.L * a.L + __ldg(a.types + t).x], acc[i]);
  }
}

// Same-spin doubles of spin S: one warp per pair (pairs of a bra string taken
// by the warps of its CTA); TwoDiffCorrelation's phase on the bra determinant.
template <int S>
__global__ void __launch_bounds__(kT) k_rdm_doubles(RdmArgs a) {
  const SpinTables &T = S == 0 ? a.A : a.B;
  const uint64_t *same = S == 0 ? a.astr : a.bstr;
  const uint64_t *opp = S == 0 ? a.bstr : a.astr;
  const double *Wr = S == 0 ? a.W : a.WT;
  const uint32_t nopp = S == 0 ? a.nb : a.na;
  const int L = a.L;
  const uint32_t bra = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t p0 = T.off_d[bra], p1 = T.off_d[bra + 1];
  const uint64_t bs = same[bra];
  double *blk = a.two + (size_t)(3 * S) * L * L * L * L;
  for (uint32_t p = p0 + warp; p < p1; p += kT / 32) {
    const uint32_t ket = T.ket_d[p], code = T.code_d[p];
    const int c0 = code & 63, c1 = (code >> 6) & 63, n0 = (code >> 12) & 63, n1 = (code >> 18) & 63;
    const int I = 2 * min(c0, c1) + S, J = 2 * max(c0, c1) + S, A = 2 * min(n0, n1) + S, B = 2 * max(n0, n1) + S;
    uint64_t ma1, mb1, ma2, mb2;
    interval_masks(min(I, A), max(I, A), ma1, mb1);
    interval_masks(min(J, B), max(J, B), ma2, mb2);
    const uint64_t ms1 = S == 0 ? ma1 : mb1, ms2 = S == 0 ? ma2 : mb2;  // same-spin parts
    const uint64_t mo = S == 0 ? (mb1 ^ mb2) : (ma1 ^ ma2);              // opposite-spin part
    uint32_t base = (__popcll(bs & ms1) + __popcll(bs & ms2)) & 1u;
    if (A > J || B < I) base ^= 1u;
    const double *rb = Wr + (size_t)bra * nopp, *rk = Wr + (size_t)ket * nopp;
    double s = 0.0;
    for (uint32_t o = lane; o < nopp; o += 32) {
      const uint32_t ph = (base ^ __popcll(__ldg(opp + o) & mo)) & 1u;
      const double v = __ldg(rb + o) * __ldg(rk + o);
      s += ph ? -v : v;
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0 && s != 0.0) {
      const int oi = I / 2, oj = J / 2, oa = A / 2, ob = B / 2;
      atomicAdd(&blk[q4(L, oa, ob, oi, oj)], s);
      atomicAdd(&blk[q4(L, ob, oa, oj, oi)], s);
      atomicAdd(&blk[q4(L, oa, ob, oj, oi)], -s);
      atomicAdd(&blk[q4(L, ob, oa, oi, oj)], -s);
    }
  }
}

// Diagonal, same-spin pairs and one-particle diagonal: thread per string with
// weight w[x] (row or column norm of W).
template <int S>
__global__ void k_rdm_diag_same(RdmArgs a, const double *__restrict__ w) {
  const uint64_t *str = S == 0 ? a.astr : a.bstr;
  const uint32_t n = S == 0 ? a.na : a.nb;
  const int L = a.L;
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  const double r = w[x];
  if (r == 0.0) return;
  const uint64_t bits0 = str[x];
  double *blk = a.two ? a.two + (size_t)(3 * S) * L * L * L * L : nullptr;
  uint64_t bi = bits0;
  while (bi) {
    const int p = __ffsll((long long)bi) - 1;
    bi &= bi - 1;
    atomicAdd(&a.one[(size_t)S * L * L + p + (size_t)L * p], r);
    if (!blk) continue;
    uint64_t bj = bi;  // q > p
    while (bj) {
      const int q = __ffsll((long long)bj) - 1;
      bj &= bj - 1;
      atomicAdd(&blk[q4(L, p, q, p, q)], r);
      atomicAdd(&blk[q4(L, q, p, q, p)], r);
      atomicAdd(&blk[q4(L, p, q, q, p)], -r);
      atomicAdd(&blk[q4(L, q, p, p, q)], -r);
    }
  }
}

// Y[ia][q] = sum_ib W[ia][ib]^2 [beta orbital q in ib]; one warp per row.
__global__ void __launch_bounds__(kT) k_rdm_occ_rows(RdmArgs a, double *__restrict__ Y) {
  const int lane = threadIdx.x & 31, L = a.L;
  const uint32_t warps = gridDim.x * (kT / 32);
  for (uint32_t ia = blockIdx.x * (kT / 32) + (threadIdx.x >> 5); ia < a.na; ia += warps) {
    double y[kMaxL];
#pragma unroll
    for (int q = 0; q < kMaxL; ++q) y[q] = 0.0;
    const double *row = a.W + (size_t)ia * a.nb;
    for (uint32_t ib = lane; ib < a.nb; ib += 32) {
      const double w = __ldg(row + ib), w2 = w * w;
      const uint64_t bs = __ldg(a.bstr + ib);
#pragma unroll
      for (int q = 0; q < kMaxL; ++q)
        if ((bs >> q) & 1ull) y[q] += w2;
    }
#pragma unroll
    for (int q = 0; q < kMaxL; ++q) {
      double v = y[q];
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0 && q < L) Y[(size_t)ia * L + q] = v;
    }
  }
}

// Alpha-beta diagonal pairs: M[p][q] = sum_ia [p in ia] Y[ia][q], added to
// two[2][p, q, p, q] and two[1][q, p, q, p]; thread per (p, q).
__global__ void k_rdm_diag_ab(RdmArgs a, const double *__restrict__ Y) {
  const int L = a.L;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= L * L) return;
  const int p = t / L, q = t % L;
  double m = 0.0;
  for (uint32_t ia = 0; ia < a.na; ++ia)
    if ((a.astr[ia] >> p) & 1ull) m += Y[(size_t)ia * L + q];
  if (m == 0.0) return;
  const size_t L4 = (size_t)L * L * L * L;
  atomicAdd(&a.two[2 * L4 + q4(L, p, q, p, q)], m);
  atomicAdd(&a.two[1 * L4 + q4(L, q, p, q, p)], m);
}

// Alpha-beta sums R[oi, oa, oj, ob] (alpha i -> a, beta j -> b) into the
// reference's entries (TwoDiffCorrelation with i = 2oi, j = 2oj+1, a = 2oa,
// b = 2ob+1; the element's phase is already in R).
__global__ void k_rdm_scatter_ab(RdmArgs a) {
  const int L = a.L;
  const size_t L4 = (size_t)L * L * L * L;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < L4; t += (size_t)gridDim.x * blockDim.x) {
    const double x = a.R[t];
    if (x == 0.0) continue;
    const int ob = t % L, oj = (t / L) % L, oa = (t / ((size_t)L * L)) % L, oi = (int)(t / ((size_t)L * L * L));
    const int i = 2 * oi, j = 2 * oj + 1, aa = 2 * oa, b = 2 * ob + 1;
    const int I = min(i, j), J = max(i, j), A = min(aa, b), B = max(aa, b);
    const int si = I & 1, sj = J & 1, sa = A & 1;
    const int Oi = I / 2, Oj = J / 2, Oa = A / 2, Ob = B / 2;
    if (si == sa) {
      atomicAdd(&a.two[(si + 2 * sj) * L4 + q4(L, Oa, Ob, Oi, Oj)], x);
      atomicAdd(&a.two[(sj + 2 * si) * L4 + q4(L, Ob, Oa, Oj, Oi)], x);
    } else {
      atomicAdd(&a.two[(si + 2 * sj) * L4 + q4(L, Oa, Ob, Oj, Oi)], x);
      atomicAdd(&a.two[(sj + 2 * si) * L4 + q4(L, Ob, Oa, Oi, Oj)], x);
    }
  }
}

// Sorts the singles of both spins by orbital pair and adds their alpha x beta
// sums to a.R.
void rdm_ab(Problem &p, const RdmArgs &a, cudaStream_t s) {
  const int L = a.L;
  const size_t L2 = (size_t)L * L;
  const size_t words = 4 * (p.A.ns / kAbPairs + L2) + 4 * L2;
  // counts and cursors of both spins, chunks and types, sorted singles: kept with the
  // problem, or for this call alone where a budget has no room for them
  struct Buffer {
    Ctx *c;
    void *tmp = nullptr;
    ~Buffer() { tmp_free(c, tmp); }
  } buffer{p.ctx};
  const size_t bytes = 16 * L2 + 4 * words + 8 * (p.A.ns + p.B.ns) + 64, have = p.ws_bytes[WS_RED2];
  if (p.ctx->budget && bytes > have && p.ctx->in_use - have + bytes > p.ctx->budget)
    buffer.tmp = tmp_alloc(p.ctx, bytes);
  unsigned char *ws = (unsigned char *)(buffer.tmp ? buffer.tmp : workspace(p, WS_RED2, bytes));
  uint32_t *count = (uint32_t *)ws, *next = count + 2 * L2;
  uint4 *lists = (uint4 *)(ws + ((16 * L2 + 15) & ~(size_t)15));
  uint2 *pa = (uint2 *)((unsigned char *)lists + 4 * words), *pb = pa + p.A.ns;
  SBDGB_CUDA(cudaMemsetAsync(count, 0, 8 * L2, s));
  auto blocks = [](uint64_t n) { return (unsigned)std::min<uint64_t>((n + 255) / 256, 1024); };
  k_rdm_types<<<blocks(p.A.ns), 256, 0, s>>>(p.A, L, count);
  k_rdm_types<<<blocks(p.B.ns), 256, 0, s>>>(p.B, L, count + L2);
  std::vector<uint32_t> h(2 * L2), first(2 * L2);
  SBDGB_CUDA(cudaMemcpyAsync(h.data(), count, 8 * L2, cudaMemcpyDeviceToHost, s));
  SBDGB_CUDA(cudaStreamSynchronize(s));
  std::exclusive_scan(h.begin(), h.begin() + L2, first.begin(), 0u);
  std::exclusive_scan(h.begin() + L2, h.end(), first.begin() + L2, 0u);
  std::vector<uint4> out;
  for (uint32_t t = 0; t < L2; ++t)
    for (uint32_t k = 0; k < h[t]; k += kAbPairs)
      out.push_back(make_uint4(t, first[t] + k, std::min(kAbPairs, h[t] - k), 0));
  const uint32_t nchunks = (uint32_t)out.size();
  std::vector<uint32_t> order;
  for (uint32_t t = 0; t < L2; ++t)
    if (h[L2 + t]) order.push_back(t);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return h[L2 + x] > h[L2 + y]; });
  for (uint32_t t : order) out.push_back(make_uint4(t, first[L2 + t], h[L2 + t], 0));
  SBDGB_CUDA(cudaMemcpyAsync(lists, out.data(), sizeof(uint4) * out.size(), cudaMemcpyHostToDevice, s));
  SBDGB_CUDA(cudaMemcpyAsync(next, first.data(), 8 * L2, cudaMemcpyHostToDevice, s));
  k_rdm_sort<<<blocks(p.A.ns), 256, 0, s>>>(p.A, L, next, pa);
  k_rdm_sort<<<blocks(p.B.ns), 256, 0, s>>>(p.B, L, next + L2, pb);
  int optin = 0;
  SBDGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, p.ctx->device));
  RdmAb b{};
  b.astr = p.astr;
  b.bstr = p.bstr;
  b.W = a.W;
  b.R = a.R;
  b.pa = pa;
  b.pb = pb;
  b.chunks = lists;
  b.types = lists + nchunks;
  b.ntypes = (uint32_t)order.size();
  b.npb = (uint32_t)p.B.ns;
  b.nb = p.nb;
  b.L = L;
  const size_t rows = 16ull * p.nb, ent = 8ull * p.B.ns, limit = (size_t)optin - 1024;
  b.rows_smem = rows <= limit;
  b.ent_smem = (b.rows_smem ? rows : 0) + ent <= limit;
  const size_t smem = (b.rows_smem ? rows : 0) + (b.ent_smem ? ent : 0);
  ensure_dynamic_smem((const void *)k_rdm_ab, smem);
  prefer_shared_carveout((const void *)k_rdm_ab);
  k_rdm_ab<<<nchunks, kT, smem, s>>>(b);
  count_launch(p.ctx, 5);
  SBDGB_CUDA(cudaGetLastError());
  SBDGB_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
}

}  // namespace

void rdm(Problem &p, const double *W, double *one_host, double *two_host, cudaStream_t s) {
  SBDGB_REQUIRE(p.tables, SBDGB_E_STATE, "RDMs need the excitation tables");
  SBDGB_REQUIRE(p.norb <= kMaxL, SBDGB_E_UNSUPPORTED, "norb > 64");
  W = device_vector(p, W, s);
  const int L = p.norb;
  const size_t L2 = (size_t)L * L, L4 = L2 * L2;
  RdmArgs a{};
  a.astr = p.astr;
  a.bstr = p.bstr;
  a.na = p.na;
  a.nb = p.nb;
  a.L = L;
  a.W = W;
  a.A = p.A;
  a.B = p.B;
  double *WT = (double *)workspace(p, WS_C64, sizeof(double) * p.N);
  transpose_fp64(p, W, WT, p.na, p.nb, s);
  a.WT = WT;
  a.one = (double *)workspace(p, WS_RDM1, sizeof(double) * 2 * L2);
  SBDGB_CUDA(cudaMemsetAsync(a.one, 0, sizeof(double) * 2 * L2, s));
  if (two_host) {
    a.two = (double *)workspace(p, WS_RDM2, sizeof(double) * 4 * L4);
    a.R = (double *)workspace(p, WS_RDMAB, sizeof(double) * L4);
    SBDGB_CUDA(cudaMemsetAsync(a.two, 0, sizeof(double) * 4 * L4, s));
    SBDGB_CUDA(cudaMemsetAsync(a.R, 0, sizeof(double) * L4, s));
  }
  double *r = (double *)workspace(p, WS_NORM_A, sizeof(double) * p.na);
  double *c = (double *)workspace(p, WS_NORM_B, sizeof(double) * p.nb);
  string_norms(p, W, r, c, s);
  k_rdm_diag_same<0><<<(p.na + 127) / 128, 128, 0, s>>>(a, r);
  k_rdm_diag_same<1><<<(p.nb + 127) / 128, 128, 0, s>>>(a, c);
  int sms = 0;
  SBDGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.ctx->device));
  auto pair_blocks = [&](uint64_t n) { return (unsigned)std::min<uint64_t>((n + kT / 32 - 1) / (kT / 32), 8ull * sms); };
  if (p.A.ns) k_rdm_singles<0><<<pair_blocks(p.A.ns), kT, 0, s>>>(a);
  if (p.B.ns) k_rdm_singles<1><<<pair_blocks(p.B.ns), kT, 0, s>>>(a);
  count_launch(p.ctx, 5);
  if (two_host && p.A.ns && p.B.ns) rdm_ab(p, a, s);
  if (two_host) {
    double *Y = (double *)workspace(p, WS_RED2, sizeof(double) * (size_t)p.na * L);
    const uint32_t rb = (uint32_t)std::min<size_t>(((size_t)p.na + 7) / 8, (size_t)sms * 8);
    k_rdm_occ_rows<<<rb, kT, 0, s>>>(a, Y);
    k_rdm_diag_ab<<<(int)((L2 + 127) / 128), 128, 0, s>>>(a, Y);
    k_rdm_doubles<0><<<p.na, kT, 0, s>>>(a);
    k_rdm_doubles<1><<<p.nb, kT, 0, s>>>(a);
    k_rdm_scatter_ab<<<(unsigned)std::min<size_t>((L4 + 255) / 256, (size_t)sms * 8), 256, 0, s>>>(a);
    count_launch(p.ctx, 5);
  }
  SBDGB_CUDA(cudaGetLastError());
  SBDGB_CUDA(cudaMemcpyAsync(one_host, a.one, sizeof(double) * 2 * L2, cudaMemcpyDeviceToHost, s));
  if (two_host) SBDGB_CUDA(cudaMemcpyAsync(two_host, a.two, sizeof(double) * 4 * L4, cudaMemcpyDeviceToHost, s));
  SBDGB_CUDA(cudaStreamSynchronize(s));
}

}  // namespace sbdgb

extern "C" int sbdgb_rdm(sbdgb_problem *pr, const double *W, double *one, double *two, void *stream) {
  if (!pr || !W || !one) return SBDGB_E_INPUT;
  sbdgb::Ctx *c = pr->p.ctx;
  try {
    SBDGB_CUDA(cudaSetDevice(c->device));
    sbdgb::rdm(pr->p, W, one, two, stream ? (cudaStream_t)stream : c->stream);
    c->last_error.clear();
    return SBDGB_OK;
  } catch (const sbdgb::Error &e) {
    c->last_error = e.what();
    return e.status;
  } catch (const std::exception &e) {
    c->last_error = e.what();
    return SBDGB_E_INPUT;
  }
}
