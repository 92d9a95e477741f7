// frsz1_legacy.cu -- the reference's legacy "frsz" codec (the LibPressio
// plugin of src/frsz.cc:15-165): values quantized with step 2*epsilon, stored
// as int16 differences to the previous quantized value within blocks of 256
// values; decoding is a running sum per block.
//
// Bit-exact with the reference's arithmetic (src/frsz.cc:113-148):
//   compress   q[i] = (T) round((double) x[i] * (1 / (2 eps)))   (half away from 0)
//              d[i] = q[i] - (i % 256 ? q[i-1] : 0)                (in T)
//              out[i] = int16 saturate(d[i])   (truncation; NaN -> 0 as on x86)
//   decompress y[256b] = (T)((double)(T)in[256b] * 2eps)
//              y[256b+i] = (T)((double)(T)in[k] * 2eps + (double) y[256b+i-1])
// with k = i (the reference reads block 0's deltas for every block) or, with
// FRSZ1_OWN_DELTAS, k = 256b + i.  Multiplies and adds are separate
// round-to-nearest operations (no contraction), as in the reference's build.
//
// compress is elementwise: a thread takes 8 consecutive values, its left
// neighbour's quantized value by a shuffle, and writes 16 bytes.  decompress
// runs one thread per block of 256 values (the sum is sequential and rounds at
// every step); codes and values go through shared memory, so the global
// accesses are coalesced.
#include "frsz2_fast.cuh"
#include "frsz2_launch.hpp"

#include "../../include/frsz2_b200.h"

#include <algorithm>
#include <cmath>

namespace frsz2b {
namespace {

constexpr int kLegacyBlock = 256; // src/frsz.cc:103, 132

#ifndef FRSZ1_MAGIC_ROUNDING
#define FRSZ1_MAGIC_ROUNDING 1
#endif

// std::round (half away from zero) of a double with additions only, by the
// magic-constant method for rounding to an integer (Muller et al., Handbook
// of Floating-Point Arithmetic, 2nd ed., sec. 5.1): adding 2^52 rounded
// toward zero to v = |p| + 0.5 leaves floor(v) + 2^52, from which 2^52 is
// subtracted exactly.  v itself is rounded, but for 0.5 <= |p| < 2^52 that
// rounding never carries it across an integer: |p| and 0.5 are multiples of
// ulp(|p|), so v is exact unless it has moved into the next binade, and a
// binade starts at a power of two, which is an integer with no other integer
// within 0.5 above it.  Below 0.5 it can: |p| = 0.5 - 2^-54 (the double just
// below 0.5) gives v = 1 - 2^-54, which rounds to 1.0, where std::round gives
// 0.  So |p| < 0.5 is 0 by a select.  The sign is copied back (so -0.4 gives
// -0.0 as std::round does).  |p| >= 2^52 (already an integer), Inf and NaN
// are returned as they are.
__device__ __forceinline__ double round_half_away(double p)
{
  constexpr double TWO52 = 4503599627370496.0;
  const double a = fabs(p);
  const double t = a < 0.5 ? 0.0 : __dsub_rn(__dadd_rz(__dadd_rn(a, 0.5), TWO52), TWO52);
  return copysign(a < TWO52 ? t : a, p);
}

template<class T>
__device__ __forceinline__ T legacy_quantize(T x, double inv)
{
  const double p = __dmul_rn((double)x, inv);
  // fp32 (conversion-bound: 0.76 -> 0.98 of HBM) only; fp64 measured even
  const double q = FRSZ1_MAGIC_ROUNDING && sizeof(T) == 4 ? round_half_away(p) : round(p);
  if constexpr (sizeof(T) == 4)
    return __double2float_rn(q);
  else
    return q;
}

// saturate<int16_t> (src/frsz.cc:97-101).  d is a difference of two
// integer-valued floats, so it is itself integer-valued (or +-Inf / NaN):
// clamped to [-32768, 32767] it converts exactly.  For fp32 that is done by
// adding 1.5 * 2^23 and reading the integer from the low bits of the sum (the
// same magic-constant method) instead of a conversion instruction.
template<class T>
__device__ __forceinline__ std::int16_t legacy_saturate(T d)
{
  if (d != d) return 0;
  if (!FRSZ1_MAGIC_ROUNDING || sizeof(T) == 8) {
    if (d < (T)-32768) return (std::int16_t)-32768;
    if (d > (T)32767) return (std::int16_t)32767;
    if constexpr (sizeof(T) == 4)
      return (std::int16_t)__float2int_rz(d);
    else
      return (std::int16_t)__double2int_rz(d);
  }
  const float c = fminf(fmaxf((float)d, -32768.0f), 32767.0f);
  return (std::int16_t)(__float_as_int(__fadd_rn(c, 12582912.0f)) - 0x4B400000);
}

template<class T>
__device__ __forceinline__ T legacy_sub(T a, T b)
{
  if constexpr (sizeof(T) == 4)
    return __fsub_rn(a, b);
  else
    return __dsub_rn(a, b);
}

// Quantized value as a 32-bit integer: exactly legacy_quantize for |p| < 2^24
// (p = x * inv), the range in which the value is exact in the float type.
// One addition rounds half away from zero: doubles at 2^51 are multiples of
// 0.5, so |p| + (2^51 + 0.5) rounded toward zero holds floor(2 |p| + 1) in its
// low word, and dropping the last bit leaves floor(|p| + 0.5) (the exact sum
// is truncated once, so |p| = 0.5 - 2^-54 gives 0 as std::round does).
template<class T>
__device__ __forceinline__ int legacy_quantize_int(T x, double inv)
{
  const double r = __dadd_rz(fabs(__dmul_rn((double)x, inv)), 2251799813685248.5); // 2^51 + 0.5
  const std::uint32_t lo = (std::uint32_t)__double2loint(r);
  int sx;
  if constexpr (sizeof(T) == 4)
    sx = __float_as_int(x) >> 31;
  else
    sx = __double2hiint(x) >> 31;
  return ((int)(lo >> 1) ^ sx) - sx; // inv > 0: p has x's sign
}

// Whether every p of N values is below 2^24 (false with a NaN or an infinity):
// from the largest magnitude, fp64's by its high word (three-input float maxima,
// see raw_max), rounded up.
template<class T, int N>
__device__ __forceinline__ bool legacy_in_range(const T (&x)[N], double inv)
{
  typename fp<T>::U u[N];
#pragma unroll
  for (int k = 0; k < N; ++k) u[k] = to_bits<T>(x[k]);
  const std::uint32_t m = raw_max<T, N, 0>(u);
  if (m >= key_of<T>::SPECIAL) return false;
  const double most = sizeof(T) == 4 ? (double)__uint_as_float(m) : __hiloint2double((int)m, -1);
  return __dmul_rn(most, inv) < 16777216.0;
}

// Two differences as saturated int16 in one word (lo in the low half).
__device__ __forceinline__ std::uint32_t pack_sat_s16(int lo, int hi)
{
  std::uint32_t r;
  asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(r) : "r"(hi), "r"(lo));
  return r;
}

constexpr int kComV = 8; // values per thread: a warp's 32 threads take one block of 256

// A warp codes one block of 256 values, 8 per thread.  VEC, aligned pointers: 8
// consecutive ones, so the first thread's predecessor is the block's start and the
// others' is one shuffle away.  Otherwise value k of a thread is the warp's
// 32 k + lane, so that loads and stores of single values are coalesced.  Values
// quantize to integers (legacy_quantize_int) and VEC saturates two differences per
// instruction; a warp that meets a value outside the range codes its block with
// the float arithmetic.  VEC is bound by DRAM (before, by the instructions of the
// float arithmetic: 28 per value, 16 now); measured on B200, 2^26 values,
// float arithmetic only -> here: fp32 78 -> 57.7 us (1.06 of the copy bandwidth), fp64
// 113 -> 95 us; off alignment fp32 127 -> 65.3 us, fp64 115 -> 94.6 us (8 consecutive
// values per thread there: 103 and 163 us); every value out of the range, fp32 78 ->
// 68.8 us.
template<class T, bool VEC>
__global__ void __launch_bounds__(256) k_frsz1_compress(const T* __restrict__ x, std::uint64_t n, double inv,
                                                        std::int16_t* __restrict__ out)
{
  enter_in_stream_order();
  static_assert(kComV * 32 == kLegacyBlock, "one block per warp");
  constexpr int V = kComV;
  const int lane = threadIdx.x & 31;
  const std::uint64_t w0 = ((std::uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * V; // the warp's block
  const std::uint64_t i0 = VEC ? w0 + lane * V : w0 + lane; // the thread's first value
  constexpr int STEP = VEC ? 1 : 32;
  T xv[V];
  const bool whole = VEC && i0 + V <= n;
  if (whole) {
#pragma unroll
    for (int h = 0; h < V * (int)sizeof(T) / 32; ++h) {
      std::uint32_t v[8];
      ld256_stream(x + i0 + h * (32 / (int)sizeof(T)), v);
#pragma unroll
      for (int k = 0; k < 32 / (int)sizeof(T); ++k) {
        if constexpr (sizeof(T) == 4)
          xv[k] = __uint_as_float(v[k]);
        else
          xv[h * 4 + k] = __longlong_as_double((long long)(((std::uint64_t)v[2 * k + 1] << 32) | v[2 * k]));
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k) xv[k] = i0 + k * STEP < n ? x[i0 + k * STEP] : (T)0;
  }
  // the quantized value before value k: the thread's last one, or the lane's before
  auto previous = [&](const auto(&q)[V], int k) {
    using Q = std::decay_t<decltype(q[0])>;
    if (VEC && k > 0) return q[k - 1];
    Q p = __shfl_up_sync(0xFFFFFFFFu, q[VEC ? V - 1 : k], 1);
    const Q first = VEC || k == 0 ? (Q)0 : __shfl_sync(0xFFFFFFFFu, q[VEC || k == 0 ? 0 : k - 1], 31);
    return lane == 0 ? first : p;
  };
  std::uint32_t w[V / 2];
  if (__all_sync(0xFFFFFFFFu, legacy_in_range<T, V>(xv, inv))) {
    int q[V];
#pragma unroll
    for (int k = 0; k < V; ++k) q[k] = legacy_quantize_int<T>(xv[k], inv);
#pragma unroll
    for (int k = 0; k < V; k += 2) w[k / 2] = pack_sat_s16(q[k] - previous(q, k), q[k + 1] - previous(q, k + 1));
  } else {
    T f[V];
#pragma unroll
    for (int k = 0; k < V; ++k) f[k] = legacy_quantize<T>(xv[k], inv);
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      const std::int16_t a = legacy_saturate<T>(legacy_sub<T>(f[k], previous(f, k)));
      const std::int16_t b = legacy_saturate<T>(legacy_sub<T>(f[k + 1], previous(f, k + 1)));
      w[k / 2] = (std::uint16_t)a | ((std::uint32_t)(std::uint16_t)b << 16);
    }
  }
  if (whole) {
    if ((reinterpret_cast<std::uintptr_t>(out) & 15u) == 0) {
      __stcs(reinterpret_cast<uint4*>(out + i0), make_uint4(w[0], w[1], w[2], w[3]));
    } else {
      __stcs(reinterpret_cast<uint2*>(out + i0), make_uint2(w[0], w[1]));
      __stcs(reinterpret_cast<uint2*>(out + i0) + 1, make_uint2(w[2], w[3]));
    }
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (i0 + k * STEP < n) out[i0 + k * STEP] = (std::int16_t)(w[k / 2] >> (16 * (k % 2)));
  }
}

constexpr int kDecBlocks = 64; // blocks of 256 values per CTA (one thread each)
constexpr int kDecChunk = 16;  // values per block staged at a time

template<class T>
__device__ __forceinline__ T legacy_step(std::int16_t q, double ebx2, T prev)
{
  const double t = __dadd_rn(__dmul_rn((double)(T)q, ebx2), (double)prev);
  if constexpr (sizeof(T) == 4)
    return __double2float_rn(t);
  else
    return t;
}

// One block of 256 values per thread; a CTA is one warp, so 32 blocks.  The
// codes come in stages through a pair of shared-memory buffers (asynchronous
// 16-byte copies, the next stage in flight while the current one is summed) and
// the values leave 64 per block at a time through a third; rows are an odd
// multiple of 16 bytes apart, which keeps each thread's 16-byte accesses to its
// own row free of bank conflicts.
//
// What bounds it: the chain of one value after the other (about 70 cycles in
// fp32, 25 in fp64) against the warps the shared memory allows, and the length
// of the runs in DRAM.  Measured on B200, 2^26 values, own differences, one
// 16-value piece per block at a time (the kernel below) -> here: fp32 95 -> 69.9
// us, fp64 153 -> 110 us; block 0's differences 68.5 -> 54.8 and 121 -> 98 us.
// Runs of 32 bytes straight from registers took 115 / 171 us, of 128 bytes 75.8 /
// 135 us, fp64 with 64 instead of 128 codes per stage 117 us, fp32 with 128
// instead of 64 codes 82.5 us.
//
// For fp32 the sum is a double rounded to float at every step.  RND rounds it
// by integer arithmetic on its bits (nearest, ties to even, at the 29 bits a
// float drops) instead of two conversions in the chain from one value to the
// next; it holds for sums that are zero or normal floats, which the caller
// guarantees from the step's size.  Codes become doubles with one addition:
// code + 2^15 sits in the low word of 2^52 + code + 2^15.
template<class T, bool RND>
struct legacy_sum
{
  double s = 0.0; // the running sum, exactly a T

  // the T value (off the chain)
  __device__ __forceinline__ T value() const
  {
    if constexpr (sizeof(T) == 4)
      return __double2float_rn(s);
    else
      return s;
  }
  __device__ __forceinline__ void round_to_T()
  {
    if constexpr (sizeof(T) == 4) {
      if constexpr (RND) {
        const std::uint32_t lo = (std::uint32_t)__double2loint(s);
        const std::uint32_t hi = (std::uint32_t)__double2hiint(s);
        // half up, then an exact half whose kept part was even goes back down
        const std::uint32_t keep = (lo & 0x3FFFFFFFu) == 0x10000000u ? 0xC0000000u : 0xE0000000u;
        const std::uint64_t u = (((std::uint64_t)hi << 32) | lo) + 0x10000000u;
        s = __hiloint2double((int)(u >> 32), (int)((std::uint32_t)u & keep));
      } else {
        s = (double)__double2float_rn(s);
      }
    }
  }
};

// code as a double times ebx2, rounded as one product
__device__ __forceinline__ double legacy_term(std::uint32_t code_plus_2p15, double ebx2)
{
  return __dmul_rn(__dadd_rn(__hiloint2double(0x43300000, (int)code_plus_2p15), -4503599627403264.0), ebx2);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* g)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((std::uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}

// FULL: the CTA has 32 whole blocks.
template<class T, bool OWN, bool RND, bool FULL>
__device__ __forceinline__ void legacy_decompress_cta(const std::int16_t* __restrict__ in, std::uint64_t n,
                                                      std::uint64_t v0, double ebx2, T* __restrict__ y,
                                                      std::uint8_t* s_out, std::uint8_t* s_in)
{
  constexpr int VO = 64;                        // values per block and part
  constexpr int CS = sizeof(T) == 4 ? 64 : 128; // codes per block and stage
  constexpr int kOutBytes = VO * (int)sizeof(T);
  constexpr int kRowBytes = kOutBytes + 16;         // a block's row of values
  constexpr int CROW = 2 * CS + 16;                 // a block's row of codes
  constexpr int PV = 16 / (int)sizeof(T);           // values per 16 bytes
  constexpr int LPC = CS / 8, LPO = kOutBytes / 16; // threads per row of codes, of values
  const int lane = threadIdx.x;
  const int full = FULL ? 32 : (int)((n - v0) / kLegacyBlock);       // whole blocks
  const int tail = FULL ? 0 : (int)(n - v0) - full * kLegacyBlock;   // values of the array's last, partial one
  const std::uint64_t g0 = v0 + (std::uint64_t)lane * kLegacyBlock;  // this thread's block
  if constexpr (!OWN) { // block 0's codes, which every block adds
    for (int i = lane; i < kLegacyBlock; i += 32)
      reinterpret_cast<std::int16_t*>(s_in)[i] = (std::uint64_t)i < n ? in[i] : (std::int16_t)0;
    __syncwarp();
  }
  const std::int16_t* src = in + v0 + (lane / LPC) * kLegacyBlock + (lane % LPC) * 8;
  std::uint8_t* s_src = s_in + (lane / LPC) * CROW + (lane % LPC) * 16;
  auto issue = [&](int stage) {
    if constexpr (OWN) {
      if (stage < kLegacyBlock / CS) {
#pragma unroll
        for (int i = 0; i < LPC; ++i) {
          const int row = (32 / LPC) * i + lane / LPC;
          std::uint8_t* d = s_src + (stage & 1) * (32 * CROW) + (32 / LPC) * i * CROW;
          const std::int16_t* g = src + stage * CS + (32 / LPC) * i * kLegacyBlock;
          if (FULL || row < full)
            cp_async16(d, g);
          else if (row == full) // in order with the copies: the partial block's codes one by one
            for (int k = 0; k < 8 && stage * CS + (lane % LPC) * 8 + k < tail; ++k)
              reinterpret_cast<std::int16_t*>(d)[k] = g[k];
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  };
  T* dst = y + v0 + (lane / LPO) * kLegacyBlock + (lane % LPO) * PV;
  const std::uint8_t* s_dst = s_out + (lane / LPO) * kRowBytes + (lane % LPO) * 16;
  legacy_sum<T, RND> acc;
  issue(0);
#pragma unroll 1
  for (int part = 0; part < kLegacyBlock / VO; ++part) {
    if constexpr (OWN) {
      if (part * VO % CS == 0) {
        issue(part * VO / CS + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
      }
    }
    const std::uint8_t* codes =
      OWN ? s_in + (part * VO / CS & 1) * (32 * CROW) + lane * CROW + part * VO % CS * 2 : s_in + part * VO * 2;
#pragma unroll
    for (int h = 0; h < VO; h += 8) {
      const uint4 c4 = *reinterpret_cast<const uint4*>(codes + h * 2);
      std::uint32_t w[4] = { c4.x, c4.y, c4.z, c4.w };
      if (!OWN && h == 0 && part == 0 && (FULL || g0 < n))
        w[0] = (w[0] & 0xFFFF0000u) | (std::uint16_t)in[g0]; // the block's own first value
#pragma unroll
      for (int p = 0; p < 8; p += PV) {
        std::uint32_t v[4];
#pragma unroll
        for (int k = 0; k < PV; ++k) {
          const int i = p + k;
          const std::uint32_t b = w[i / 2] ^ 0x80008000u; // codes + 2^15
          const double t = legacy_term((i & 1) ? b >> 16 : b & 0xFFFFu, ebx2);
          if (h == 0 && i == 0 && part == 0)
            acc.s = t;
          else
            acc.s = __dadd_rn(t, acc.s);
          acc.round_to_T();
          if constexpr (sizeof(T) == 4) {
            v[k] = __float_as_uint(acc.value());
          } else {
            v[2 * k] = (std::uint32_t)__double2loint(acc.s);
            v[2 * k + 1] = (std::uint32_t)__double2hiint(acc.s);
          }
        }
        *reinterpret_cast<uint4*>(s_out + lane * kRowBytes + (h + p) * (int)sizeof(T)) =
          make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < LPO; ++i)
      if (FULL || (32 / LPO) * i + lane / LPO < full)
        __stcs(reinterpret_cast<uint4*>(dst + part * VO + (32 / LPO) * i * kLegacyBlock),
               *reinterpret_cast<const uint4*>(s_dst + (32 / LPO) * i * kRowBytes));
    if constexpr (!FULL)
      for (int k = part * VO + lane; k < min(tail, (part + 1) * VO); k += 32)
        y[v0 + full * kLegacyBlock + k] = reinterpret_cast<const T*>(s_out + full * kRowBytes)[k - part * VO];
    __syncwarp(); // the part has left; its codes' buffer is free
  }
}

template<class T, bool OWN, bool RND>
__global__ void __launch_bounds__(32) k_frsz1_decompress_vec(const std::int16_t* __restrict__ in, std::uint64_t n,
                                                             double ebx2, T* __restrict__ y)
{
  enter_in_stream_order();
  constexpr int CS = sizeof(T) == 4 ? 64 : 128; // codes per block and stage, as above
  __shared__ __align__(16) std::uint8_t s_out[32 * (64 * sizeof(T) + 16)];
  __shared__ __align__(16) std::uint8_t s_in[OWN ? 2 * 32 * (2 * CS + 16) : kLegacyBlock * 2];
  const std::uint64_t v0 = (std::uint64_t)blockIdx.x * (32 * kLegacyBlock); // the CTA's first value
  if (n - v0 >= 32 * kLegacyBlock)
    legacy_decompress_cta<T, OWN, RND, true>(in, n, v0, ebx2, y, s_out, s_in);
  else // whole blocks and the last, partial one side by side
    legacy_decompress_cta<T, OWN, RND, false>(in, n, v0, ebx2, y, s_out, s_in);
}

// Blocks for pointers off the 32-byte layout: 64 blocks per CTA, values through
// shared memory 16 per block at a time and stored one by one, so the stores are
// coalesced whatever the alignment.
template<class T, bool OWN>
__global__ void __launch_bounds__(kDecBlocks) k_frsz1_decompress(const std::int16_t* __restrict__ in, std::uint64_t n,
                                                                  double ebx2, T* __restrict__ y, bool vec)
{
  enter_in_stream_order();
  // block 0's differences (the reference reads them for every block)
  __shared__ std::int16_t s_d0[OWN ? 1 : kLegacyBlock];
  __shared__ T s_out[kDecBlocks][kDecChunk + 1];
  const int tid = threadIdx.x;
  const std::uint64_t b0 = (std::uint64_t)blockIdx.x * kDecBlocks; // first block of the CTA
  const std::uint64_t v0 = b0 * kLegacyBlock;
  if constexpr (!OWN) {
    const std::uint64_t n0 = n < (std::uint64_t)kLegacyBlock ? n : (std::uint64_t)kLegacyBlock;
    for (std::uint64_t i = tid; i < n0; i += kDecBlocks) s_d0[i] = in[i];
  }
  __syncthreads();
  const std::uint64_t g0 = v0 + (std::uint64_t)tid * kLegacyBlock; // this thread's block
  const int len = g0 < n ? (int)((n - g0) < (std::uint64_t)kLegacyBlock ? n - g0 : (std::uint64_t)kLegacyBlock) : 0;
  T acc = (T)0;
  // own codes: two 16-byte loads per chunk, issued one chunk ahead so their
  // latency overlaps the previous chunk's sums
  uint4 pa = make_uint4(0, 0, 0, 0), pb = pa;
  auto fetch = [&](int c) {
    if (OWN && vec && c + kDecChunk <= len) {
      const uint4* p = reinterpret_cast<const uint4*>(in + g0 + c);
      pa = __ldg(p);
      pb = __ldg(p + 1);
    }
  };
  fetch(0);
  for (int c = 0; c < kLegacyBlock; c += kDecChunk) {
    // this chunk's codes: the block's own or block 0's
    std::int16_t qc[kDecChunk];
    if constexpr (OWN) {
      if (vec && c + kDecChunk <= len) {
        const uint4 a = pa, b = pb;
        if (c + kDecChunk < kLegacyBlock) fetch(c + kDecChunk);
        const std::uint32_t w[8] = { a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w };
#pragma unroll
        for (int k = 0; k < kDecChunk; ++k) qc[k] = (std::int16_t)(w[k / 2] >> (16 * (k % 2)));
      } else {
#pragma unroll
        for (int k = 0; k < kDecChunk; ++k) qc[k] = c + k < len ? in[g0 + c + k] : (std::int16_t)0;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kDecChunk; ++k) qc[k] = (c + k == 0) ? (len > 0 ? in[g0] : (std::int16_t)0) : s_d0[c + k];
    }
#pragma unroll
    for (int k = 0; k < kDecChunk; ++k) {
      const int i = c + k;
      if (i < len) {
        if (i == 0) {
          const double t = __dmul_rn((double)(T)qc[0], ebx2);
          if constexpr (sizeof(T) == 4)
            acc = __double2float_rn(t);
          else
            acc = t;
        } else {
          acc = legacy_step<T>(qc[k], ebx2, acc);
        }
        s_out[tid][k] = acc;
      }
    }
    __syncthreads();
    // chunk c of every block: consecutive threads take consecutive values of
    // a block, then the next block
    for (int idx = tid; idx < kDecBlocks * kDecChunk; idx += kDecBlocks) {
      const int b = idx / kDecChunk, k = idx % kDecChunk;
      const std::uint64_t g = v0 + (std::uint64_t)b * kLegacyBlock + c + k;
      if (g < n) y[g] = s_out[b][k];
    }
    __syncthreads();
  }
}

template<class T>
int legacy_compress(double eps, const void* d_values, std::uint64_t n, void* d_out, cudaStream_t s)
{
  const bool vec = reinterpret_cast<std::uintptr_t>(d_values) % 32 == 0 &&
                   reinterpret_cast<std::uintptr_t>(d_out) % 8 == 0;
  const std::uint64_t threads = (n + kComV - 1) / kComV;
  const unsigned grid = (unsigned)std::max<std::uint64_t>(1, (threads + 255) / 256);
  const auto kernel = vec ? k_frsz1_compress<T, true> : k_frsz1_compress<T, false>;
  launch(kernel, grid, 256, 0, s, static_cast<const T*>(d_values), n, 1.0 / (eps * 2.0),
         static_cast<std::int16_t*>(d_out));
  return cuda_status(cudaGetLastError(), "legacy compress launch");
}

template<class T>
int legacy_decompress(double eps, const void* d_in, std::uint64_t n, void* d_values, bool own, cudaStream_t s)
{
  const std::uint64_t nb = (n + kLegacyBlock - 1) / kLegacyBlock;
  const unsigned grid = (unsigned)std::max<std::uint64_t>(1, (nb + kDecBlocks - 1) / kDecBlocks);
  const auto* q = static_cast<const std::int16_t*>(d_in);
  T* y = static_cast<T*>(d_values);
  if (reinterpret_cast<std::uintptr_t>(d_in) % 32 == 0 && reinterpret_cast<std::uintptr_t>(d_values) % 32 == 0) {
    // RND: a nonzero sum of a product q * 2eps and a float is at least an ulp of
    // the product, 2^-52 * 2eps, and at most 256 * 2^15 * 2eps: normal floats for
    // 2eps in [2^-64, 2^96]
    const double s2 = eps * 2;
    const unsigned warps = (unsigned)std::max<std::uint64_t>(1, (nb + 31) / 32);
    const bool rnd = sizeof(T) == 4 && s2 >= 0x1p-64 && s2 <= 0x1p96;
    if (own)
      rnd ? launch(k_frsz1_decompress_vec<T, true, true>, warps, 32, 0, s, q, n, s2, y)
          : launch(k_frsz1_decompress_vec<T, true, false>, warps, 32, 0, s, q, n, s2, y);
    else
      rnd ? launch(k_frsz1_decompress_vec<T, false, true>, warps, 32, 0, s, q, n, s2, y)
          : launch(k_frsz1_decompress_vec<T, false, false>, warps, 32, 0, s, q, n, s2, y);
    return cuda_status(cudaGetLastError(), "legacy decompress launch");
  }
  const bool vec = reinterpret_cast<std::uintptr_t>(d_in) % 16 == 0;
  if (own)
    launch(k_frsz1_decompress<T, true>, grid, kDecBlocks, 0, s, q, n, eps * 2, y, vec);
  else
    launch(k_frsz1_decompress<T, false>, grid, kDecBlocks, 0, s, q, n, eps * 2, y, vec);
  return cuda_status(cudaGetLastError(), "legacy decompress launch");
}

int legacy_checks(int dtype, double epsilon, const void* a, const void* b, std::uint64_t n)
{
  if (dtype != FRSZ2_FLOAT && dtype != FRSZ2_DOUBLE)
    return set_error(FRSZ2_EDTYPE, "unsupported type: currently only floating point supported");
  if (!(epsilon > 0.0) || !std::isfinite(epsilon)) return set_error(FRSZ2_EFAIL, "epsilon must be positive and finite");
  if (n > 0 && (!a || !b)) return set_error(FRSZ2_EFAIL, "null pointer");
  return FRSZ2_OK;
}

} // namespace
} // namespace frsz2b

using namespace frsz2b;

extern "C" {

uint64_t frsz1_compressed_size(uint64_t n) { return n * sizeof(std::int16_t); }

int frsz1_compress(int dtype, double epsilon, const void* d_values, uint64_t n, void* d_out, void* stream)
{
  NvtxRange nvtx("frsz1_compress");
  EarlyLaunch early;
  if (int rc = legacy_checks(dtype, epsilon, d_values, d_out, n)) return rc;
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  if (reinterpret_cast<std::uintptr_t>(d_values) % es != 0 || reinterpret_cast<std::uintptr_t>(d_out) % 2 != 0)
    return set_error(FRSZ2_EFAIL, "misaligned pointer");
  if (n == 0) return FRSZ2_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == FRSZ2_FLOAT ? legacy_compress<float>(epsilon, d_values, n, d_out, s)
                              : legacy_compress<double>(epsilon, d_values, n, d_out, s);
}

int frsz1_decompress(int dtype, double epsilon, const void* d_in, uint64_t n, void* d_values, int flags, void* stream)
{
  NvtxRange nvtx("frsz1_decompress");
  EarlyLaunch early;
  if (int rc = legacy_checks(dtype, epsilon, d_in, d_values, n)) return rc;
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  if (reinterpret_cast<std::uintptr_t>(d_values) % es != 0 || reinterpret_cast<std::uintptr_t>(d_in) % 2 != 0)
    return set_error(FRSZ2_EFAIL, "misaligned pointer");
  if (n == 0) return FRSZ2_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool own = (flags & FRSZ1_OWN_DELTAS) != 0;
  return dtype == FRSZ2_FLOAT ? legacy_decompress<float>(epsilon, d_in, n, d_values, own, s)
                              : legacy_decompress<double>(epsilon, d_in, n, d_values, own, s);
}

} // extern "C"
