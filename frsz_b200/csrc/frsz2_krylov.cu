// frsz2_krylov.cu -- decompress fused into its consumer: dot products and
// axpy over a basis of FRSZ2-compressed fp64 vectors (the compressed Krylov
// basis use of the reference's random-access decode,
// include/frsz2.hpp:1096-1104).  Values are decoded in registers straight into
// the FMAs and never written back.
//
//   frsz2_basis_dot:  h[j] = sum_i V_j[i] * w[i]           j < m
//   frsz2_basis_axpy: y[i] = y[i] + sum_j c[j] * V_j[i]     (j in order 0..m-1)
//
// dot: a warp takes a group of vectors over a slice of the positions, reads
// each position of w once for the whole group, and writes one sum per vector;
// a second kernel adds a vector's sums in slice order, so the result does not
// depend on scheduling.  axpy: a thread holds its values of y in registers and
// adds the vectors to them one after the other.
#include "frsz2_fast.cuh"
#include "frsz2_launch.hpp"

#include "../../include/frsz2_b200.h"

#include <algorithm>
#include <string>

namespace frsz2b {
namespace {

constexpr int kMaxBasis = FRSZ2_MAX_BASIS;
constexpr int kKT = 256;              // threads per CTA
constexpr int kKW = kKT / 32;         // warps per CTA
constexpr int kSub = 3072;            // positions per partial sum that the workspace has room for

struct BasisParams
{
  const std::uint8_t* buf[kMaxBasis]; // compressed vectors
};

struct BasisGeo
{
  std::uint64_t n;
  std::uint64_t exp_bytes;
  int log2E;
};

// Values per lane.  Eight share one exponent load, one range test and the
// address arithmetic; above 32 bits eight values' codes take too many registers
// for several vectors in flight.  Blocks of 4 values take four at every width.
__host__ __device__ constexpr int basis_nv(int bits)
{
  return bits <= 32 ? 8 : 4;
}

// Vectors whose loads a warp has in flight together, and the CTAs per SM that
// the register budget must allow.  Swept on B200 over 1, 2, 4, 8 x 2..6 (dot, us
// at 4 x 3 / 4 x 4 / 2 x 3 / 2 x 4): 100 vectors of 2^22 values at 32 bits 253 /
// 326 (spills) / 316 / 256, at 16 bits 195 / 172 / 258 / 226; 50 of 2^21 at 21
// bits 75.4 / 86.9 / 88.3 / 75.5, 24 bits 65.2 / 62.2 / 77.8 / 71.9, 48 bits 106 /
// 105 / 113 / 112, 64 bits 213 / 312 / 161 / 195.  One or two vectors take a
// variant of two: 1 vector of 2^22 at 32 bits 14.7 -> 12.0 us.
__host__ __device__ constexpr int dot_jb(int bits) { return bits > 48 ? 2 : 4; }
__host__ __device__ constexpr int dot_ctas(int bits, int nv, int jb)
{
  if (bits > 48) return 3;
  if (jb == 2 || nv == 4) return 4;
  return bits == 21 || bits == 32 ? 3 : 4;
}
// axpy over 2..12 x 2..4 (us): 16 bits 6 x 3 170, 5 x 3 179, 3 x 4 182, 4 x 3 230;
// 21 bits 5 x 3 67.1, 4 x 3 67.8; 24 bits 3 x 4 62.0, 4 x 3 65.3; 32 bits 4 x 3
// 262, 3 x 4 265, 6 x 3 366 (spills); 48 bits 5 x 3 103, 4 x 3 118; 64 bits 5 x 3
// 132, 4 x 3 133; four values per lane, 100 vectors of 2^20, 6 x 4 / 5 x 4: 16 bits
// 63.8 / 57.0, 21 bits 83.6 / 78.0, 24 bits 65.6 / 63.9, 32 bits 68.2 / 72.4.
__host__ __device__ constexpr int axpy_jb(int bits, int nv)
{
  if (nv == 4 && bits <= 32) return bits == 32 ? 6 : 5;
  return bits == 16 ? 6 : bits == 24 ? 3 : bits == 32 ? 4 : 5;
}
__host__ __device__ constexpr int axpy_ctas(int bits, int nv)
{
  return (nv == 4 && bits <= 32) || bits == 24 ? 4 : 3;
}

// One vector's codes of a lane's NV consecutive values, and their exponent.
template<int BITS, int NV>
struct basis_lane
{
  static constexpr int SEG = NV * BITS; // bits
  static constexpr int NW = (SEG + 31) / 32;
  static constexpr bool ALIGNED = SEG % 32 == 0;
  using exp_t = std::conditional_t<(BITS > 32), std::int64_t, std::int32_t>;
  std::uint32_t w[ALIGNED ? NW : NW + 1];
  exp_t be;
};

// NW words at p, aligned to 4 bytes or, with WIDE, to the largest power of two
// dividing their bytes.  One load of 16 or 32 bytes takes them past the L1 cache
// (each sector is read once, and w stays there); several go through it, since a
// sector then serves more than one of them (21 bits, six loads: 97 -> 75 us), and
// so do 8-byte ones (axpy of 30 vectors of 300,007 values, 16 bits: 7.5 -> 6.8 us).
template<int NW, bool WIDE>
__device__ __forceinline__ void ldg_words(const std::uint32_t* p, std::uint32_t* w)
{
  constexpr int V = !WIDE ? 1 : NW % 8 == 0 ? 8 : NW % 4 == 0 ? 4 : NW % 2 == 0 ? 2 : 1;
  if constexpr (V == NW && V >= 4) {
    if constexpr (V == 8)
      asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                   : "l"(p));
    else
      asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "l"(p));
  } else {
#pragma unroll
    for (int i = 0; i < NW; i += V) {
      if constexpr (V == 4) {
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(p + i));
        w[i] = t.x;
        w[i + 1] = t.y;
        w[i + 2] = t.z;
        w[i + 3] = t.w;
      } else if constexpr (V == 2) {
        const uint2 t = __ldg(reinterpret_cast<const uint2*>(p + i));
        w[i] = t.x;
        w[i + 1] = t.y;
      } else {
        w[i] = __ldg(p + i);
      }
    }
  }
}

// The codes at stream bit S of a vector (words at `words`) and the exponent at
// `exp`; S is a multiple of NV * BITS.
template<int BITS, int NV>
__device__ __forceinline__ void basis_load(const std::uint8_t* exp, const std::uint8_t* words, std::uint64_t S,
                                           basis_lane<BITS, NV>& l)
{
  using L = basis_lane<BITS, NV>;
  constexpr int W = fast_cfg<double, BITS>::W;
  l.be = (typename L::exp_t)load_exp(exp, W);
  const std::uint32_t* p = reinterpret_cast<const std::uint32_t*>(words) + (S >> 5);
  ldg_words<L::NW, L::ALIGNED>(p, l.w);
  if constexpr (!L::ALIGNED) l.w[L::NW] = ((int)(S & 31u) + L::SEG > 32 * L::NW) ? __ldg(p + L::NW) : 0u;
}

template<int K, int BITS, int N, int NV, class C>
__device__ __forceinline__ void basis_codes(const std::uint32_t (&seg)[N], C (&c)[NV])
{
  if constexpr (K < NV) {
    c[K] = (C)get_bits<K * BITS, BITS>(seg);
    basis_codes<K + 1, BITS>(seg, c);
  }
}

// Values of widths up to 48 bits without an integer-to-double conversion,
// exactly the values of the decoder.  D - base, both doubles of exponent field
// F = be + 1044 (or be + 1029), where D has the magnitude in the low bits of its
// mantissa, so the subtraction is exact.
//   up to 32 bits: with t = code << (32 - BITS) (sign at bit 31) the low word is
//     max(t << 1, 1): a nonzero magnitude is mag * 2^(33-BITS), worth
//     mag * 2^(be-BITS+2) at F = be + 1044; a zero magnitude gives the decoder's
//     2^(be-31).
//   33 to 48 bits: the magnitude shifted up to 47 bits, or 2^15 when it is zero,
//     at F = be + 1029 (a unit is 2^(be-46)).
// Needs F to be a normal exponent field and be in the plain range:
// be in [-959, 1002].  A block of zeros (exponent field 0, be = -1023) decodes to
// zeros; it comes with be = kZeroBlock, which gives the exponent field of be = 0
// (F's bits above it shift out) and a base with the zero magnitude's low word, so
// D - base is 0.
constexpr int kZeroBlock = 1 << 16;

template<int BITS>
__device__ __forceinline__ bool direct_exponent(std::int64_t be)
{
  return be >= -959 && be <= 1002;
}

template<int BITS, int NV>
__device__ __forceinline__ void basis_values_direct(const basis_lane<BITS, NV>& l, int o, double (&v)[NV])
{
  using L = basis_lane<BITS, NV>;
  using C = std::conditional_t<(BITS <= 32), std::uint32_t, std::uint64_t>;
  std::uint32_t seg[L::NW + 1];
#pragma unroll
  for (int i = 0; i < L::NW; ++i) {
    if constexpr (L::ALIGNED)
      seg[i] = l.w[i];
    else
      seg[i] = __funnelshift_r(l.w[i], l.w[i + 1], o);
  }
  seg[L::NW] = 0;
  C c[NV];
  basis_codes<0, BITS>(seg, c);
  if constexpr (BITS <= 32) {
    const std::uint32_t F = (std::uint32_t)(l.be + 1044);
    const int hi = (int)(F << 20);
    const double base = __hiloint2double(hi, (int)(F >> 16));
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const std::uint32_t t = c[k] << (32 - BITS);
      const double d = __hiloint2double(hi, (int)max(t << 1, 1u)) - base;
      v[k] = __hiloint2double(__double2hiint(d) ^ (int)(t & 0x80000000u), __double2loint(d));
    }
  } else {
    static_assert(BITS <= 48, "magnitudes below 2^47");
    const std::uint32_t F = (std::uint32_t)(l.be + 1029), hi = F << 20;
    const double base = __hiloint2double((int)hi, (int)(F >> 1 & 0x8000u));
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const std::uint64_t t = c[k] << (48 - BITS); // sign at bit 47
      std::uint32_t lo = (std::uint32_t)t;
      const std::uint32_t up = (std::uint32_t)(t >> 32) & 0x7FFFu;
      if ((lo | up) == 0) lo = 0x8000u;
      const double d = __hiloint2double((int)(hi | up), (int)lo) - base;
      v[k] = __hiloint2double(__double2hiint(d) ^ (int)((std::uint32_t)(t >> 16) & 0x80000000u), __double2loint(d));
    }
  }
}

// The same through the decoder's own arithmetic, for every exponent.
template<int BITS, int NV>
__device__ __forceinline__ void basis_values_any(const basis_lane<BITS, NV>& l, int o, double (&v)[NV])
{
  using L = basis_lane<BITS, NV>;
  using C = typename fast_cfg<double, BITS>::C;
  std::uint32_t seg[L::NW + 1];
#pragma unroll
  for (int i = 0; i < L::NW; ++i) {
    if constexpr (L::ALIGNED)
      seg[i] = l.w[i];
    else
      seg[i] = __funnelshift_r(l.w[i], l.w[i + 1], o);
  }
  seg[L::NW] = 0;
  C c[NV];
  basis_codes<0, BITS>(seg, c);
  const std::int64_t be = l.be;
  if (plain_exponent<double>(be)) {
    const double inv = pow2<double>((int)be - BITS + 2);
    const std::uint64_t zero_bits = (std::uint64_t)(be + 992) << 52;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = from_bits<double>(decode_plain<double, BITS>(c[k], inv, zero_bits));
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = from_code<double>((std::uint64_t)c[k], be, BITS);
  }
}

constexpr bool has_direct(int bits) { return bits <= 48; }

// Bits of word i of a lane's stream that belong to magnitudes.
template<int BITS, int NV>
__host__ __device__ constexpr std::uint32_t magnitude_bits(int i)
{
  std::uint32_t m = 0;
  for (int b = 32 * i; b < 32 * i + 32 && b < NV * BITS; ++b)
    if (b % BITS != BITS - 1) m |= 1u << (b - 32 * i);
  return m;
}

template<int BITS, int NV, int I = 0>
__device__ __forceinline__ std::uint32_t any_magnitude(const basis_lane<BITS, NV>& l, int o)
{
  using L = basis_lane<BITS, NV>;
  if constexpr (I == L::NW) {
    return 0u;
  } else {
    std::uint32_t w;
    if constexpr (L::ALIGNED)
      w = l.w[I];
    else
      w = __funnelshift_r(l.w[I], l.w[I + 1], o);
    constexpr std::uint32_t M = magnitude_bits<BITS, NV>(I);
    return (w & M) | any_magnitude<BITS, NV, I + 1>(l, o);
  }
}

// Makes the lanes of a step that holds exponents outside the direct range ready for
// the direct arithmetic where they are blocks of zeros (the decoder gives +-0 for
// zero magnitudes up to exponent -992).  False for the warp where any other such
// lane is left; `other` has a bit for each vector of which it is this lane.
// Sparse vectors: dot / axpy of 100 vectors of 2^22 values with half of their blocks
// zero, us, through the decoder's arithmetic -> here: 16 bits 900 / 825 -> 209 / 191,
// 21 bits 1,075 / 885 -> 318 / 282, 32 bits 969 / 872 -> 272 / 264, 48 bits 1,113 / 1,028
// -> 500 / 467; 1 % zero, 16 bits 342 / 335 -> 185 / 170.
template<int BITS, int NV, int JB>
__device__ __forceinline__ bool settle_zeros(basis_lane<BITS, NV> (&l)[JB], int o, unsigned& other)
{
  other = 0;
#pragma unroll
  for (int jj = 0; jj < JB; ++jj)
    if (!direct_exponent<BITS>(l[jj].be)) {
      if (l[jj].be <= -992 && any_magnitude<BITS, NV>(l[jj], o) == 0)
        l[jj].be = kZeroBlock;
      else
        other |= 1u << jj;
    }
  return !__any_sync(0xFFFFFFFFu, other != 0);
}

// acc + sum of v[k] * w[k], k < cnt, in order: a lane of a step that holds an
// exponent outside the direct range which is no block of zeros (loads again, off
// the fast path; eight values per lane).  JB gives each kernel its own copy: nvcc
// 12.9 fails on one that is shared by kernels of different register bounds.
template<int BITS, int NV, int JB>
__device__ __noinline__ double slow_lane_dot(const std::uint8_t* exp, const std::uint8_t* words, std::uint64_t S,
                                             const double* w, int cnt, double acc)
{
  basis_lane<BITS, NV> l;
  basis_load<BITS, NV>(exp, words, S, l);
  double v[NV];
  basis_values_any<BITS, NV>(l, (int)(S & 31u), v);
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k < cnt) acc = fma(v[k], __ldg(w + k), acc);
  return acc;
}

// y[k] + c * v[k] on a lane's values of y in memory, k < cnt.
template<int BITS, int NV>
__device__ __noinline__ void slow_lane_axpy(const std::uint8_t* exp, const std::uint8_t* words, std::uint64_t S,
                                            double c, double* y)
{
  basis_lane<BITS, NV> l;
  basis_load<BITS, NV>(exp, words, S, l);
  double v[NV];
  basis_values_any<BITS, NV>(l, (int)(S & 31u), v);
#pragma unroll
  for (int k = 0; k < NV; ++k) y[k] = fma(c, v[k], y[k]);
}

// A lane's values of w: 32-byte loads where `whole` says that w is aligned and all
// of them are there, else those below cnt one by one.
template<int NV>
__device__ __forceinline__ void load_w(const double* w, bool whole, int cnt, double (&wv)[NV])
{
  if (whole) {
#pragma unroll
    for (int h = 0; h < NV; h += 4) {
      std::uint32_t t[8];
      asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
                   : "l"(w + h));
#pragma unroll
      for (int k = 0; k < 4; ++k) wv[h + k] = __hiloint2double((int)t[2 * k + 1], (int)t[2 * k]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) wv[k] = k < cnt ? __ldg(w + k) : 0.0;
  }
}

// What is left of a warp's part of a slice (positions from p on) once a step holds
// an exponent outside the direct range, as vectors with blocks of zeros do; the
// kernels of four values per lane leave it to this.  Out of line, so that the loop of
// the other steps keeps its registers: in line, as the kernels of eight values have
// it, dense vectors lose there (dot of 100 vectors of 2^22 at 48 bits 391 -> 404 us;
// axpy of 30 of 300,007 at 16 bits 6.8 -> 8.2, at 21 bits 9.3 -> 10.5), and out of
// line with eight those do (dot at 32 bits 258 -> 272 us, axpy at 21 bits 233 -> 252).
template<int BITS, int NV, int JB>
__device__ __noinline__ void rest_of_dot(const std::uint8_t* const* bufs, int nv, std::uint64_t exp_bytes, int log2E,
                                         const double* w, std::uint64_t pos0, int p, int len, double* sums)
{
  constexpr int Wb = fast_cfg<double, BITS>::W / 8;
  const int lane = threadIdx.x & 31;
  const bool wvec = (reinterpret_cast<std::uintptr_t>(w) & 31u) == 0;
  double acc[JB];
#pragma unroll
  for (int jj = 0; jj < JB; ++jj) acc[jj] = sums[jj];
#pragma unroll 1
  for (; p - lane * NV < len; p += 32 * NV) {
    const std::uint64_t idx = pos0 + (std::uint64_t)p;
    const std::uint64_t S0 = idx * (std::uint64_t)BITS;
    const std::uint64_t eo = (idx >> log2E) * Wb;
    const int o = (int)(S0 & 31u);
    basis_lane<BITS, NV> l[JB];
#pragma unroll
    for (int jj = 0; jj < JB; ++jj) {
      l[jj].be = 0;
      if (p < len && jj < nv) basis_load<BITS, NV>(bufs[jj] + eo, bufs[jj] + exp_bytes, S0, l[jj]);
    }
    double wv[NV];
    load_w<NV>(w + idx, wvec && p + NV <= len, len - p, wv);
    unsigned other;
    if (settle_zeros<BITS, NV, JB>(l, o, other)) {
#pragma unroll
      for (int jj = 0; jj < JB; ++jj) {
        double v[NV];
        basis_values_direct<BITS, NV>(l[jj], o, v);
        double t = v[0] * wv[0];
#pragma unroll
        for (int k = 1; k < NV; ++k) t = fma(v[k], wv[k], t);
        acc[jj] += t;
      }
    } else if (p < len) {
#pragma unroll
      for (int jj = 0; jj < JB; ++jj) {
        double v[NV];
        if ((other >> jj & 1u) == 0)
          basis_values_direct<BITS, NV>(l[jj], o, v);
        else
          basis_values_any<BITS, NV>(l[jj], o, v);
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < NV; ++k)
          if (p + k < len) t = fma(v[k], wv[k], t);
        acc[jj] += t;
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int jj = 0; jj < JB; ++jj) sums[jj] = acc[jj];
}

// The same for the axpy: the vectors from the step's first on.
template<int BITS, int NV, int JB>
__device__ __noinline__ void rest_of_axpy(const std::uint8_t* const* bufs, int left, std::uint64_t exp_bytes,
                                          std::uint64_t eo, std::uint64_t S0, bool in, const double* coef, double* y)
{
  const int o = (int)(S0 & 31u);
  double acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = y[k];
#pragma unroll 1
  for (; left > 0; left -= JB, bufs += JB, coef += JB) {
    basis_lane<BITS, NV> l[JB];
#pragma unroll
    for (int jj = 0; jj < JB; ++jj) {
      l[jj].be = 0;
      if (in && jj < left) basis_load<BITS, NV>(bufs[jj] + eo, bufs[jj] + exp_bytes, S0, l[jj]);
    }
    unsigned other;
    const bool direct = settle_zeros<BITS, NV, JB>(l, o, other);
    auto add = [&](auto value) {
#pragma unroll
      for (int jj = 0; jj < JB; ++jj)
        if (jj < left) {
          double v[NV];
          value(jj, v);
          const double cj = coef[jj];
#pragma unroll
          for (int k = 0; k < NV; ++k) acc[k] = fma(cj, v[k], acc[k]);
        }
    };
    if (direct)
      add([&](int jj, double (&v)[NV]) { basis_values_direct<BITS, NV>(l[jj], o, v); });
    else
      add([&](int jj, double (&v)[NV]) {
        if ((other >> jj & 1u) == 0)
          basis_values_direct<BITS, NV>(l[jj], o, v);
        else
          basis_values_any<BITS, NV>(l[jj], o, v);
      });
    __syncwarp();
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) y[k] = acc[k];
}

// Sums of two or four values over the warp in a fixed order: each exchange halves
// the values a lane carries, so N values cost N - 1 + log2(32 / N) exchanges
// instead of 5 N.  Returns value (lane * N) / 32 summed over the lanes that share
// this one's lower bits; the caller adds those up.
template<int N>
__device__ __forceinline__ double warp_sums(double (&a)[N])
{
  static_assert(N == 2 || N == 4, "two or four values");
  const int lane = threadIdx.x & 31;
  const bool up = (lane & 16) != 0;
  double b[N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const double send = up ? a[i] : a[i + N / 2];
    b[i] = (up ? a[i + N / 2] : a[i]) + __shfl_xor_sync(0xFFFFFFFFu, send, 16);
  }
  if constexpr (N == 2) {
    return b[0];
  } else {
    const bool up2 = (lane & 8) != 0;
    const double send = up2 ? b[0] : b[1];
    return (up2 ? b[1] : b[0]) + __shfl_xor_sync(0xFFFFFFFFu, send, 8);
  }
}

// Partial sums of the dot.  Unit u = slice * groups + group is JB vectors over
// S positions, done by 2^lq warps of a CTA that take a part of the slice each;
// a CTA's units are neighbouring groups of one slice, so its warps read w from
// the L1 cache after the first.
//
// Bound by DRAM at 32 bits (253 us for 100 vectors of 2^22, 1.06 of the copy
// bandwidth) and by instructions at 16 (10.8 per value, 172 us, 0.80; 280 us
// and 18.1 before: four values per lane, w in shared memory behind two barriers
// per slice, a warp-wide sum per vector every 12 values of a lane).
template<int BITS, int NV, int JB>
__global__ void __launch_bounds__(kKT, dot_ctas(BITS, NV, JB))
  k_basis_dot(const __grid_constant__ BasisParams bp, int m, BasisGeo g, const double* __restrict__ w, unsigned ns,
              unsigned groups, unsigned S, int lq, double* __restrict__ partials)
{
  enter_in_stream_order();
  constexpr int Wb = fast_cfg<double, BITS>::W / 8;
  __shared__ double s_sum[kKW][JB];
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
  const unsigned unit = (blockIdx.x << (3 - lq)) + (unsigned)(warp >> lq);
  const unsigned sl = unit / groups, gr = unit - sl * groups;
  const bool live = sl < ns;
  const int j0 = (int)gr * JB, nv = min(JB, m - j0);
  double sum = 0.0;
  if (live) {
    const unsigned part = S >> lq;
    const std::uint64_t pos0 = (std::uint64_t)sl * S + (std::uint64_t)(warp & ((1 << lq) - 1)) * part;
    const int len = pos0 >= g.n ? 0 : (int)min((std::uint64_t)part, g.n - pos0);
    const bool wvec = (reinterpret_cast<std::uintptr_t>(w) & 31u) == 0;
    double acc[JB];
#pragma unroll
    for (int jj = 0; jj < JB; ++jj) acc[jj] = 0.0;
    int p = lane * NV;
    bool rest = false;
    for (; p - lane * NV < len; p += 32 * NV) {
      const bool in = p < len;
      const std::uint64_t idx = pos0 + (std::uint64_t)p;
      const std::uint64_t S0 = idx * (std::uint64_t)BITS;
      const std::uint64_t eo = (idx >> g.log2E) * Wb;
      basis_lane<BITS, NV> l[JB];
#pragma unroll
      for (int jj = 0; jj < JB; ++jj) {
        if (in && jj < nv) {
          const std::uint8_t* buf = bp.buf[j0 + jj];
          basis_load<BITS, NV>(buf + eo, buf + g.exp_bytes, S0, l[jj]);
        } else {
          l[jj].be = 0;
#pragma unroll
          for (int i = 0; i < (int)(sizeof(l[jj].w) / 4); ++i) l[jj].w[i] = 0u;
        }
      }
      double wv[NV];
      load_w<NV>(w + idx, wvec && p + NV <= len, len - p, wv);
      const int o = (int)(S0 & 31u);
      if constexpr (has_direct(BITS)) {
        bool slow = false;
#pragma unroll
        for (int jj = 0; jj < JB; ++jj) slow |= !direct_exponent<BITS>(l[jj].be);
        slow = __any_sync(0xFFFFFFFFu, slow);
        if constexpr (NV == 4) {
          rest = slow;
          if (rest) break;
        } else if (slow) {
          unsigned other;
          slow = !settle_zeros<BITS, NV, JB>(l, o, other);
        }
        if (NV == 4 || !slow) {
#pragma unroll
          for (int jj = 0; jj < JB; ++jj) {
            double v[NV];
            basis_values_direct<BITS, NV>(l[jj], o, v);
            double t = v[0] * wv[0]; // a step's own sum: shorter chains, smaller rounding errors
#pragma unroll
            for (int k = 1; k < NV; ++k) t = fma(v[k], wv[k], t);
            acc[jj] += t;
          }
        } else if (in) {
#pragma unroll
          for (int jj = 0; jj < JB; ++jj)
            if (jj < nv) {
              const std::uint8_t* buf = bp.buf[j0 + jj];
              acc[jj] = slow_lane_dot<BITS, NV, JB>(buf + eo, buf + g.exp_bytes, S0, w + idx, min(NV, len - p), acc[jj]);
            }
        }
        __syncwarp();
      } else {
#pragma unroll
        for (int jj = 0; jj < JB; ++jj) {
          double v[NV];
          basis_values_any<BITS, NV>(l[jj], o, v);
          double t = 0.0;
#pragma unroll
          for (int k = 0; k < NV; ++k)
            if (p + k < len) t = fma(v[k], wv[k], t);
          acc[jj] += t;
        }
      }
    }
    if constexpr (has_direct(BITS) && NV == 4) {
      if (rest) {
        double t[JB];
#pragma unroll
        for (int jj = 0; jj < JB; ++jj) t[jj] = acc[jj];
        rest_of_dot<BITS, NV, JB>(bp.buf + j0, nv, g.exp_bytes, g.log2E, w, pos0, p, len, t);
#pragma unroll
        for (int jj = 0; jj < JB; ++jj) acc[jj] = t[jj];
      }
    }
    sum = warp_sums<JB>(acc);
#pragma unroll
    for (int sh = 16 / JB; sh > 0; sh >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, sh);
  }
  // lane's sum is vector j0 + lane * JB / 32's
  const int jj = lane * JB / 32;
  if (lq == 0) {
    if (live && lane % (32 / JB) == 0 && jj < nv) partials[(std::uint64_t)(j0 + jj) * ns + sl] = sum;
    return;
  }
  if (lane % (32 / JB) == 0) s_sum[warp][jj] = sum;
  __syncthreads();
  if (live && (warp & ((1 << lq) - 1)) == 0 && lane % (32 / JB) == 0 && jj < nv) {
    for (int q = 1; q < (1 << lq); ++q) sum += s_sum[warp + q][jj];
    partials[(std::uint64_t)(j0 + jj) * ns + sl] = sum;
  }
}

// h[j] = sum over slices of partials[j * ns + slice], in a fixed order; one
// CTA per vector.
__global__ void __launch_bounds__(kKT)
  k_basis_dot_final(const double* __restrict__ partials, unsigned int ns, double* __restrict__ h)
{
  enter_in_stream_order();
  __shared__ double s_red[kKW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* pj = partials + (std::uint64_t)blockIdx.x * ns;
  double sum = 0.0;
  for (unsigned int b = tid; b < ns; b += kKT) sum += __ldcg(pj + b);
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) sum += __shfl_down_sync(0xFFFFFFFFu, sum, sh);
  if (lane == 0) s_red[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < kKW; ++q) t += s_red[q];
    h[blockIdx.x] = t;
  }
}

// Bound by DRAM from 24 bits up (0.99-1.06 of the copy bandwidth), by the
// decode's instructions below (16 bits 0.84, 21 bits 0.73).
template<int BITS, int NV, int JB>
__global__ void __launch_bounds__(kKT, axpy_ctas(BITS, NV))
  k_basis_axpy(const __grid_constant__ BasisParams bp, int m, BasisGeo g, const double* __restrict__ coef,
               double* __restrict__ y)
{
  enter_in_stream_order();
  constexpr int Wb = fast_cfg<double, BITS>::W / 8;
  __shared__ double s_c[kMaxBasis];
  for (int j = threadIdx.x; j < m; j += kKT) s_c[j] = __ldg(coef + j);
  __syncthreads();
  const std::uint64_t idx = ((std::uint64_t)blockIdx.x * kKT + threadIdx.x) * NV;
  const bool in = idx < g.n, whole = idx + NV <= g.n;
  double acc[NV];
  if (whole) {
#pragma unroll
    for (int h = 0; h < NV; h += 4) {
      std::uint32_t v[8];
      ld256_stream(y + idx + h, v);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[h + k] = __hiloint2double((int)v[2 * k + 1], (int)v[2 * k]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = idx + k < g.n ? y[idx + k] : 0.0;
  }
  const std::uint64_t S0 = idx * (std::uint64_t)BITS;
  const std::uint64_t eo = (idx >> g.log2E) * Wb;
  const int o = (int)(S0 & 31u);
  for (int j0 = 0; j0 < m; j0 += JB) {
    basis_lane<BITS, NV> l[JB];
#pragma unroll
    for (int jj = 0; jj < JB; ++jj) {
      l[jj].be = 0;
      if (in && j0 + jj < m) {
        const std::uint8_t* buf = bp.buf[j0 + jj];
        basis_load<BITS, NV>(buf + eo, buf + g.exp_bytes, S0, l[jj]);
      }
    }
    bool slow = false;
    if constexpr (has_direct(BITS)) {
#pragma unroll
      for (int jj = 0; jj < JB; ++jj) slow |= !direct_exponent<BITS>(l[jj].be);
      slow = __any_sync(0xFFFFFFFFu, slow);
      if (NV == 8 && slow) {
        unsigned other;
        slow = !settle_zeros<BITS, NV, JB>(l, o, other);
      }
    }
    if (!slow) {
#pragma unroll
      for (int jj = 0; jj < JB; ++jj)
        if (j0 + jj < m) {
          double v[NV];
          if constexpr (has_direct(BITS))
            basis_values_direct<BITS, NV>(l[jj], o, v);
          else
            basis_values_any<BITS, NV>(l[jj], o, v);
          const double cj = s_c[j0 + jj];
#pragma unroll
          for (int k = 0; k < NV; ++k) acc[k] = fma(cj, v[k], acc[k]);
        }
    } else if constexpr (has_direct(BITS)) {
      double t[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) t[k] = acc[k];
      if constexpr (NV == 4)
        rest_of_axpy<BITS, NV, JB>(bp.buf + j0, m - j0, g.exp_bytes, eo, S0, in, s_c + j0, t);
      else if (in)
        for (int j = j0; j < min(m, j0 + JB); ++j)
          slow_lane_axpy<BITS, NV>(bp.buf[j] + eo, bp.buf[j] + g.exp_bytes, S0, s_c[j], t);
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] = t[k];
      if constexpr (NV == 4)
        break;
      else
        __syncwarp();
    }
  }
  if (whole) {
#pragma unroll
    for (int h = 0; h < NV; h += 4) {
      std::uint32_t v[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[2 * k] = (std::uint32_t)__double2loint(acc[h + k]);
        v[2 * k + 1] = (std::uint32_t)__double2hiint(acc[h + k]);
      }
      st256_stream(y + idx + h, v);
    }
  } else if (in) {
    for (int k = 0; k < NV && idx + k < g.n; ++k) y[idx + k] = acc[k];
  }
}

// widths with fused kernels (fp64 bases)
#define FRSZ2_KRYLOV_WIDTHS(X) X(16) X(21) X(24) X(32) X(48) X(64)

int basis_args(int dtype, int bits, int E, const void* const* basis, int m, std::uint64_t n, BasisParams* bp,
               BasisGeo* g)
{
  if (int rc = check_args(dtype, bits, E)) return rc;
  if (dtype != FRSZ2_DOUBLE) return set_error(FRSZ2_EFAIL, "fused basis kernels take fp64 bases");
  switch (bits) {
#define CASE(B) case B:
    FRSZ2_KRYLOV_WIDTHS(CASE)
#undef CASE
    break;
    default: return set_error(FRSZ2_EFAIL, "fused basis kernels have no instance for " + std::to_string(bits) + " bits");
  }
  if (E < 4 || E > 65536 || (E & (E - 1)) != 0 || ((std::uint64_t)E * bits) % word_bits(bits) != 0)
    return set_error(FRSZ2_EFAIL, "fused basis kernels need a power-of-two block size without block padding");
  if (m < 0 || m > kMaxBasis)
    return set_error(FRSZ2_EFAIL, "basis size must be in [0, " + std::to_string(kMaxBasis) + "]");
  if (m > 0 && !basis) return set_error(FRSZ2_EFAIL, "null basis");
  const Layout L = make_layout(n, bits, E);
  for (int j = 0; j < m; ++j) {
    if (!basis[j] || reinterpret_cast<std::uintptr_t>(basis[j]) % 32 != 0)
      return set_error(FRSZ2_EFAIL, "basis vector " + std::to_string(j) + " is null or not 32-byte aligned");
    bp->buf[j] = static_cast<const std::uint8_t*>(basis[j]);
  }
  g->n = n;
  g->exp_bytes = L.exp_bytes;
  int l = 0;
  while ((1 << l) < E) ++l;
  g->log2E = l;
  return FRSZ2_OK;
}

constexpr int kMaxCtasPerSm = 8; // bound that sizes the workspace

// Launch geometry of the dot.
struct DotPlan
{
  unsigned ns, groups, S; // slices, vector groups, positions per slice
  int lq;                 // log2 of the warps that share a unit
  unsigned grid;
};

// A warp walks up to 12 steps of 32 * NV positions, 24 at 64 bits (dot of 100
// vectors of 2^22 values: 64 bits 12 / 24 / 48 steps 621 / 602 / 619 us; 48 bits 12 / 24
// steps 395 / 402), fewer when that would leave fewer than three units for each of the 32 warps that an
// SM holds.  The workspace has room for max(8 per SM, n / 3072) sums per vector;
// where short walks would need more, several warps of a CTA share a unit.
bool dot_plan(int m, std::uint64_t n, int bits, int nv, int jb, DotPlan* p)
{
  const std::uint64_t rows = std::max<std::uint64_t>((std::uint64_t)sm_count() * kMaxCtasPerSm, (n + kSub - 1) / kSub);
  const std::uint64_t step = 32 * (std::uint64_t)nv;
  const std::uint64_t groups = ((std::uint64_t)m + jb - 1) / jb;
  const std::uint64_t steps = (n + step - 1) / step;
  const std::uint64_t warps = (std::uint64_t)sm_count() * 32 * 3;
  std::uint64_t k = std::min<std::uint64_t>(bits > 48 ? 24 : 12, std::max<std::uint64_t>(1, (steps * groups + warps - 1) / warps));
  const std::uint64_t least = (steps + rows - 1) / rows; // steps per slice that the workspace asks for
  int lq = 0;
  while (lq < 3 && (k << lq) < least) ++lq;
  if ((k << lq) < least) k = (least + 7) >> 3;
  const std::uint64_t S = (k << lq) * step;
  const std::uint64_t ns = (n + S - 1) / S;
  const std::uint64_t per = 8u >> lq; // units per CTA
  const std::uint64_t grid = (ns * groups + per - 1) / per;
  if (S > 0x7FFFFFFFull || ns * groups > 0xFFFFFFF0ull || grid > 0x7FFFFFFFull) return false;
  *p = DotPlan{ (unsigned)ns, (unsigned)groups, (unsigned)S, lq, (unsigned)grid };
  return true;
}

template<int BITS, int NV, int JB>
int launch_dot(const BasisParams& bp, int m, const BasisGeo& g, const double* w, double* h, void* workspace,
               cudaStream_t s)
{
  DotPlan p;
  if (!dot_plan(m, g.n, BITS, NV, JB, &p)) return set_error(FRSZ2_EFAIL, "basis vectors too long");
  auto* rows = reinterpret_cast<double*>(static_cast<std::uint8_t*>(workspace) + 256);
  launch(k_basis_dot<BITS, NV, JB>, p.grid, kKT, 0, s, bp, m, g, w, p.ns, p.groups, p.S, p.lq, rows);
  if (int rc = cuda_status(cudaGetLastError(), "basis dot launch")) return rc;
  launch(k_basis_dot_final, (unsigned)m, kKT, 0, s, rows, p.ns, h);
  return cuda_status(cudaGetLastError(), "basis dot launch");
}

// The axpy's threads walk the vectors one after the other, so a short array has
// few of them: below four CTAs per SM of eight values per lane, four per lane
// (30 vectors of 300,007 values, 32 bits: 14.7 -> 9.9 us; 16 bits 8.5 -> 6.8).
template<int BITS>
int launch_axpy(const BasisParams& bp, int m, const BasisGeo& g, const double* coef, double* y, cudaStream_t s)
{
  constexpr int NV = basis_nv(BITS), J4 = axpy_jb(BITS, 4), JN = axpy_jb(BITS, NV);
  const bool four = g.log2E < 3 || (NV == 8 && g.n < (std::uint64_t)sm_count() * 4 * kKT * 8);
  const std::uint64_t per = (std::uint64_t)kKT * (four ? 4 : NV);
  const std::uint64_t grid = (g.n + per - 1) / per;
  if (grid > 0x7FFFFFFFull) return set_error(FRSZ2_EFAIL, "basis vectors too long");
  if (four)
    launch(k_basis_axpy<BITS, 4, J4>, (unsigned)grid, kKT, 0, s, bp, m, g, coef, y);
  else
    launch(k_basis_axpy<BITS, NV, JN>, (unsigned)grid, kKT, 0, s, bp, m, g, coef, y);
  return cuda_status(cudaGetLastError(), "basis axpy launch");
}

} // namespace
} // namespace frsz2b

using namespace frsz2b;

extern "C" {

uint64_t frsz2_basis_workspace_size(int m, uint64_t n)
{
  if (m < 0) m = 0;
  const std::uint64_t grid = (std::uint64_t)sm_count() * kMaxCtasPerSm;
  const std::uint64_t slices = (n + kSub - 1) / kSub; // one row of m sums per slice
  return 256 + std::max(grid, slices) * (std::uint64_t)std::max(m, 1) * sizeof(double);
}

int frsz2_basis_dot(int dtype, int bits, int block_size, const void* const* basis, int m, uint64_t n,
                    const void* w, void* h, void* workspace, uint64_t workspace_bytes, void* stream)
{
  NvtxRange nvtx("frsz2_basis_dot");
  EarlyLaunch early;
  BasisParams bp{};
  BasisGeo g{};
  if (int rc = basis_args(dtype, bits, block_size, basis, m, n, &bp, &g)) return rc;
  if (m == 0) return FRSZ2_OK;
  if (!w || !h || !workspace) return set_error(FRSZ2_EFAIL, "null pointer");
  if (workspace_bytes < frsz2_basis_workspace_size(m, n))
    return set_error(FRSZ2_EFAIL, "workspace smaller than frsz2_basis_workspace_size()");
  if (reinterpret_cast<std::uintptr_t>(workspace) % 256 != 0)
    return set_error(FRSZ2_EFAIL, "workspace must be 256-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n == 0) return cuda_status(cudaMemsetAsync(h, 0, (std::size_t)m * sizeof(double), s), "memset");
  const auto* wd = static_cast<const double*>(w);
  auto* hd = static_cast<double*>(h);
  switch (bits) {
#define CASE(B)                                                                                                    \
  case B:                                                                                                          \
    if (block_size < 8) return launch_dot<B, 4, dot_jb(B)>(bp, m, g, wd, hd, workspace, s);                        \
    if (m <= 2) return launch_dot<B, basis_nv(B), 2>(bp, m, g, wd, hd, workspace, s);                              \
    return launch_dot<B, basis_nv(B), dot_jb(B)>(bp, m, g, wd, hd, workspace, s);
    FRSZ2_KRYLOV_WIDTHS(CASE)
#undef CASE
  }
  return FRSZ2_EFAIL;
}

int frsz2_basis_axpy(int dtype, int bits, int block_size, const void* const* basis, int m, uint64_t n,
                     const void* coef, void* y, void* stream)
{
  NvtxRange nvtx("frsz2_basis_axpy");
  EarlyLaunch early;
  BasisParams bp{};
  BasisGeo g{};
  if (int rc = basis_args(dtype, bits, block_size, basis, m, n, &bp, &g)) return rc;
  if (m == 0 || n == 0) return FRSZ2_OK;
  if (!coef || !y) return set_error(FRSZ2_EFAIL, "null pointer");
  if (reinterpret_cast<std::uintptr_t>(y) % 32 != 0) return set_error(FRSZ2_EFAIL, "y must be 32-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto* cd = static_cast<const double*>(coef);
  auto* yd = static_cast<double*>(y);
  switch (bits) {
#define CASE(B)                                                                                                    \
  case B: return launch_axpy<B>(bp, m, g, cd, yd, s);
    FRSZ2_KRYLOV_WIDTHS(CASE)
#undef CASE
  }
  return FRSZ2_EFAIL;
}

} // extern "C"
