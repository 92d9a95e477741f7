// frsz2_laneblock.cuh -- blocks of a size that the lane-segment kernels do not
// take (no multiple of half a lane's values, or padded), one block per lane.
//
// A CTA is one warp with 32 consecutive blocks.  Their values (compress) or
// their image (decompress) come into shared memory with asynchronous 16-byte
// copies; every lane then walks its own block value by value -- all lanes are at
// the same bit position, so the position is uniform -- and the other side leaves
// shared memory with 16-byte stores.  A value costs a shared-memory access on
// each side, its arithmetic and its share of a 32-bit word, where the kernels
// that spread a block's values over a warp pay for each value's block and bit
// position.  Blocks of an odd number of values lie an odd number of words
// apart, so the lanes' accesses fall on distinct banks (two per bank at twice an
// odd number, and so on).
#pragma once

#include "frsz2_fast.cuh"

#include <array>
#include <utility>

namespace frsz2b {

// Whether compress reads a block's values 16 bytes at a time: blocks of a
// multiple of 4 values, whose lanes would meet four or more on a bank one by one
// (fp32 9 bits E 28 0.58 -> 0.66 of HBM, 31 bits E 40 0.51 -> 0.82, fp64 19 bits E 24 0.39
// -> 0.83; twice an odd number stays: fp64 13 bits E 50 0.68, 0.64 by 16 bytes).
__host__ __device__ inline bool laneblock_quads(int E) { return E % 4 == 0; }

// Bytes from one block's values to the next in shared memory: with 16-byte
// accesses an odd number of them, so that eight lanes fall on distinct banks.
__host__ __device__ inline std::uint32_t laneblock_row(int E, std::size_t es, bool quad)
{
  const std::uint32_t b = (std::uint32_t)E * (std::uint32_t)es;
  return b + (quad && b % 32u == 0 ? 16u : 0u);
}

// Bytes from one block's image to the next: blocks of a multiple of 32 bytes are
// 16 bytes further apart (lanes 32 words apart would all meet on one bank: fp64
// decompress, 60 bits E 17, 0.33 of HBM).
__host__ __device__ inline std::uint32_t laneblock_image_row(std::uint32_t block_bytes)
{
  return block_bytes + (block_bytes % 32u == 0 ? 16u : 0u);
}

// Bytes of shared memory for 32 blocks: values, image, slack for the last word.
__host__ __device__ inline std::uint32_t laneblock_smem(const Job& j, std::size_t es, bool compress)
{
  return 32u * laneblock_row(j.E, es, compress && laneblock_quads(j.E)) + 32u * laneblock_image_row(j.block_bytes) + 16u;
}

// Where the 16-byte piece of a thread goes when rows of `per` pieces lie `row`
// bytes apart in shared memory; every step is 32 pieces on.
struct lb_place
{
  std::uint32_t at, col, per, gap; // shared offset, piece within its row, pieces per row, bytes between rows
  __device__ __forceinline__ lb_place(std::uint32_t per_, std::uint32_t row)
    : at(16u * threadIdx.x), col(threadIdx.x), per(per_), gap(row - 16u * per_)
  {
    wrap();
  }
  __device__ __forceinline__ void wrap()
  {
    while (col >= per) {
      col -= per;
      at += gap;
    }
  }
  __device__ __forceinline__ void advance()
  {
    at += 512u;
    col += 32u;
    wrap();
  }
};

// `bytes` contiguous bytes of global memory into shared memory by asynchronous
// 16-byte copies, contiguous there too or in rows (ROWS), and back.
template<bool ROWS>
__device__ __forceinline__ void lb_copy_in(std::uint8_t* s, const std::uint8_t* g, std::uint32_t bytes,
                                           std::uint32_t per = 0, std::uint32_t row = 0)
{
  const std::uint32_t n16 = bytes / 16u;
  if constexpr (ROWS) {
    lb_place p(per, row);
    for (std::uint32_t i = threadIdx.x; i < n16; i += 32, p.advance())
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((std::uint32_t)__cvta_generic_to_shared(s + p.at)),
                   "l"(g + 16 * i)
                   : "memory");
    for (std::uint32_t i = 16u * n16 + threadIdx.x; i < bytes; i += 32)
      s[i + i / (16u * per) * (row - 16u * per)] = __ldg(g + i);
  } else {
    for (std::uint32_t i = threadIdx.x; i < n16; i += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((std::uint32_t)__cvta_generic_to_shared(s + 16 * i)),
                   "l"(g + 16 * i)
                   : "memory");
    for (std::uint32_t i = 16u * n16 + threadIdx.x; i < bytes; i += 32) s[i] = __ldg(g + i);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template<bool ROWS>
__device__ __forceinline__ void lb_copy_out(std::uint8_t* g, const std::uint8_t* s, std::uint32_t bytes,
                                            std::uint32_t per = 0, std::uint32_t row = 0)
{
  const std::uint32_t n16 = bytes / 16u;
  if constexpr (ROWS) {
    lb_place p(per, row);
    for (std::uint32_t i = threadIdx.x; i < n16; i += 32, p.advance())
      __stcs(reinterpret_cast<uint4*>(g) + i, *reinterpret_cast<const uint4*>(s + p.at));
    for (std::uint32_t i = 16u * n16 + threadIdx.x; i < bytes; i += 32)
      g[i] = s[i + i / (16u * per) * (row - 16u * per)];
  } else {
#pragma unroll 4
    for (std::uint32_t i = threadIdx.x; i < n16; i += 32)
      __stcs(reinterpret_cast<uint4*>(g) + i, reinterpret_cast<const uint4*>(s)[i]);
    for (std::uint32_t i = 16u * n16 + threadIdx.x; i < bytes; i += 32) g[i] = s[i];
  }
}

// The N = 16 / sizeof(T) bit patterns of one 16-byte access.
template<class U>
__device__ __forceinline__ void lb_unpack16(const uint4& v, U (&u)[16 / sizeof(U)])
{
  if constexpr (sizeof(U) == 4) {
    u[0] = v.x;
    u[1] = v.y;
    u[2] = v.z;
    u[3] = v.w;
  } else {
    u[0] = (std::uint64_t)v.y << 32 | v.x;
    u[1] = (std::uint64_t)v.w << 32 | v.z;
  }
}

// QUAD: a block's values are read 16 bytes at a time (laneblock_quads).
template<class T, int BITS, bool QUAD>
__global__ void __launch_bounds__(32) k_compress_laneblock(Job j)
{
  enter_in_stream_order();
  using Cfg = fast_cfg<T, BITS>;
  using U = typename Cfg::U;
  using C = typename Cfg::C;
  using K = key_of<T>;
  constexpr int W = Cfg::W;
  extern __shared__ __align__(16) std::uint8_t lb_smem[];
  const int lane = threadIdx.x, E = j.E;
  const std::uint32_t BB = j.block_bytes;
  const std::uint64_t nb = (j.n + (std::uint64_t)E - 1) / (std::uint64_t)E, b0 = (std::uint64_t)blockIdx.x * 32u;
  const std::uint64_t v0 = b0 * (std::uint64_t)E;
  const int all = 32 * E, nv = j.n - v0 < (std::uint64_t)all ? (int)(j.n - v0) : all;
  constexpr int N = 16 / (int)sizeof(T);
  const std::uint32_t row = laneblock_row(E, sizeof(T), QUAD);
  const std::uint32_t per = (std::uint32_t)E / N;
  std::uint8_t* s_img = lb_smem + 32u * row;
  lb_copy_in<QUAD>(lb_smem, reinterpret_cast<const std::uint8_t*>(static_cast<const T*>(j.values_in) + v0),
                   (std::uint32_t)nv * (std::uint32_t)sizeof(T), per, row);
  for (int i = nv + lane; i < all; i += 32) // past the array: neither maxima nor codes
    *reinterpret_cast<U*>(lb_smem + (std::uint32_t)(i / E) * row + (std::uint32_t)(i % E) * sizeof(T)) = 0;
  __syncwarp();

  const std::uint8_t* mine = lb_smem + (std::uint32_t)lane * row;
  const U* sv = reinterpret_cast<const U*>(mine);
  auto key = [](U u) { return __uint_as_float((std::uint32_t)(sizeof(T) == 4 ? u : u >> (fp<T>::UBITS - 32))); };
  float m = 0.0f;
  if constexpr (QUAD) {
#pragma unroll 4
    for (std::uint32_t q = 0; q < per; ++q) {
      U u[N];
      lb_unpack16<U>(reinterpret_cast<const uint4*>(mine)[q], u);
#pragma unroll
      for (int i = 0; i < N; i += 2) m = max3_abs(m, key(u[i]), key(u[i + 1]));
    }
  } else {
    int k = 0;
#pragma unroll 4
    for (; k + 2 <= E; k += 2) m = max3_abs(m, key(sv[k]), key(sv[k + 1]));
    if (k < E) m = max3_abs(m, key(sv[k]), key(sv[k]));
  }
  const std::uint32_t km = __float_as_uint(m);
  std::uint32_t kc = km;
  if (km >= K::SPECIAL) {
    kc = 0;
    for (int k = 0; k < E; ++k) kc = max(kc, K::clean(sv[k]));
  }
  const int ex = exponent_of_field<T>((int)(kc >> K::FSHIFT));
  const int be = W == 8 && sizeof(T) == 8 ? (int)(std::int8_t)ex : ex;
  const bool plain = km < K::SPECIAL && be == ex && be >= (sizeof(T) == 4 ? -95 : -959);
  if (b0 + lane < nb) store_word(j.exps + (b0 + lane) * (std::uint64_t)(W / 8), (std::uint64_t)(std::int64_t)be, W);

  const std::uint32_t img_row = laneblock_image_row(BB);
  std::uint8_t* dst = s_img + (std::uint32_t)lane * img_row;
  std::uint32_t at = 0; // bytes written; the branches below are the same for every lane
  const int grain = (int)(BB & 3u);
  auto put = [&](std::uint32_t w) {
    if (grain == 0) {
      *reinterpret_cast<std::uint32_t*>(dst + at) = w;
    } else if (grain == 2) {
      *reinterpret_cast<std::uint16_t*>(dst + at) = (std::uint16_t)w;
      if (at + 2 < BB) *reinterpret_cast<std::uint16_t*>(dst + at + 2) = (std::uint16_t)(w >> 16);
    } else {
      for (std::uint32_t q = 0; q < 4 && at + q < BB; ++q) dst[at + q] = (std::uint8_t)(w >> (8 * q));
    }
    at += 4;
  };
  std::uint64_t acc = 0;
  int have = 0;
  auto push = [&](std::uint32_t v, int bits) {
    acc |= (std::uint64_t)v << have;
    have += bits;
    if (have >= 32) {
      put((std::uint32_t)acc);
      acc >>= 32;
      have -= 32;
    }
  };
  auto push_code = [&](C c) {
    if constexpr (BITS <= 32) {
      push((std::uint32_t)c, BITS);
    } else {
      push((std::uint32_t)c, 32);
      push((std::uint32_t)(c >> 32), BITS - 32);
    }
  };
  auto codes = [&](auto code) {
    if constexpr (QUAD) {
#pragma unroll 2
      for (std::uint32_t q = 0; q < per; ++q) {
        U u[N];
        lb_unpack16<U>(reinterpret_cast<const uint4*>(mine)[q], u);
#pragma unroll
        for (int i = 0; i < N; ++i) push_code(code(u[i]));
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < E; ++i) push_code(code(sv[i]));
    }
  };
  // a block of zeros, as that of a lane past the last one: no magnitude for either
  // arithmetic, so it does not send the warp's other blocks to the slower one
  bool zeros = km == 0;
  if (sizeof(T) == 8 && zeros) { // km is the high words'
    U low = 0;
    for (int k = 0; k < E; ++k) low |= sv[k] << 1;
    zeros = low == 0;
  }
  if (__all_sync(0xFFFFFFFFu, plain || zeros)) {
    const T scale = pow2<T>(BITS - 2 - (zeros ? 0 : be));
    codes([&](U u) { return encode_plain<T, BITS>(u, scale); });
  } else {
    codes([&](U u) { return (C)to_code<T>(u, (std::int16_t)be, BITS); }); // exact for every block
  }
  if (have > 0) put((std::uint32_t)acc);
  while (at < BB) put(0);
  __syncwarp();
  const int nbk = (int)min((std::uint64_t)32, nb - b0);
  const std::uint32_t out = (std::uint32_t)(nbk - 1) * BB + written_block_bytes(nv - (nbk - 1) * E, BITS, W);
  std::uint8_t* g = j.words + b0 * (std::uint64_t)BB;
  if (img_row != BB)
    lb_copy_out<true>(g, s_img, out, BB / 16u, img_row);
  else
    lb_copy_out<false>(g, s_img, out);
}

template<class T, int BITS>
__global__ void __launch_bounds__(32) k_decompress_laneblock(Job j)
{
  enter_in_stream_order();
  using Cfg = fast_cfg<T, BITS>;
  using U = typename Cfg::U;
  using C = typename Cfg::C;
  constexpr int W = Cfg::W;
  extern __shared__ __align__(16) std::uint8_t lb_smem[];
  const int lane = threadIdx.x, E = j.E;
  const std::uint32_t BB = j.block_bytes;
  const std::uint64_t nb = (j.n + (std::uint64_t)E - 1) / (std::uint64_t)E, b0 = (std::uint64_t)blockIdx.x * 32u;
  const std::uint64_t v0 = b0 * (std::uint64_t)E;
  const int all = 32 * E, nv = j.n - v0 < (std::uint64_t)all ? (int)(j.n - v0) : all;
  const int nbk = (int)min((std::uint64_t)32, nb - b0);
  std::uint8_t* s_img = lb_smem + (std::uint32_t)all * (std::uint32_t)sizeof(T);
  const int own = lane < nbk ? lane : 0; // lanes past the last block decode the first one again
  const std::int64_t be = load_exp(j.exps + (b0 + own) * (std::uint64_t)(W / 8), W);
  const std::uint32_t img_row = laneblock_image_row(BB);
  const std::uint8_t* g = j.words + b0 * (std::uint64_t)BB; // the buffer holds whole blocks
  if (img_row != BB)
    lb_copy_in<true>(s_img, g, (std::uint32_t)nbk * BB, BB / 16u, img_row);
  else
    lb_copy_in<false>(s_img, g, (std::uint32_t)nbk * BB);
  __syncwarp();

  const std::uint8_t* src = s_img + (std::uint32_t)own * img_row;
  const int grain = (int)(BB & 3u);
  std::uint32_t at = 0;
  auto next = [&]() { // the next 32 bits (what lies past the block is never used)
    std::uint32_t w;
    if (grain == 0)
      w = *reinterpret_cast<const std::uint32_t*>(src + at);
    else if (grain == 2)
      w = *reinterpret_cast<const std::uint16_t*>(src + at) |
          (std::uint32_t)*reinterpret_cast<const std::uint16_t*>(src + at + 2) << 16;
    else
      w = src[at] | (std::uint32_t)src[at + 1] << 8 | (std::uint32_t)src[at + 2] << 16 | (std::uint32_t)src[at + 3] << 24;
    at += 4;
    return w;
  };
  std::uint64_t acc = 0;
  int have = 0;
  auto pull = [&](int bits) -> std::uint32_t {
    if (have < bits) {
      acc |= (std::uint64_t)next() << have;
      have += 32;
    }
    const std::uint32_t v = bits == 32 ? (std::uint32_t)acc : (std::uint32_t)acc & ((1u << (bits & 31)) - 1u);
    acc >>= bits;
    have -= bits;
    return v;
  };
  U* sv = reinterpret_cast<U*>(lb_smem) + lane * E;
  auto pull_code = [&]() -> C {
    if constexpr (BITS <= 32) {
      return (C)pull(BITS);
    } else {
      const std::uint32_t lo = pull(32);
      return (C)((std::uint64_t)pull(BITS - 32) << 32 | lo);
    }
  };
  auto values = [&](auto value) {
#pragma unroll 4
    for (int i = 0; i < E; ++i) sv[i] = value(pull_code());
  };
  if (__all_sync(0xFFFFFFFFu, plain_exponent<T>(be))) {
    const T inv = pow2<T>((int)be - BITS + 2);
    const U zero_bits = sizeof(T) == 4 ? (U)((std::uint32_t)(be + 96) << 23) : (U)((std::uint64_t)(be + 992) << 52);
    values([&](C c) { return decode_plain<T, BITS>(c, inv, zero_bits); });
  } else {
    values([&](C c) { return to_bits<T>(from_code<T>((U)c, be, BITS)); }); // exact for every block
  }
  __syncwarp();
  lb_copy_out<false>(reinterpret_cast<std::uint8_t*>(static_cast<T*>(j.values_out) + v0), lb_smem,
                     (std::uint32_t)nv * (std::uint32_t)sizeof(T));
}

using laneblock_fn = cudaError_t (*)(bool, const Job&, cudaStream_t);

template<class T, int BITS>
cudaError_t launch_laneblock_one(bool compress, const Job& j, cudaStream_t s)
{
  const std::uint64_t nb = (j.n + (std::uint64_t)j.E - 1) / (std::uint64_t)j.E;
  const unsigned grid = (unsigned)((nb + 31) / 32);
  const std::uint32_t smem = laneblock_smem(j, sizeof(T), compress);
  if (!compress)
    launch(k_decompress_laneblock<T, BITS>, grid, 32, smem, s, j);
  else if (laneblock_quads(j.E))
    launch(k_compress_laneblock<T, BITS, true>, grid, 32, smem, s, j);
  else
    launch(k_compress_laneblock<T, BITS, false>, grid, 32, smem, s, j);
  return cudaGetLastError();
}

template<class T, int LO, int... I>
constexpr auto make_laneblock_table(std::integer_sequence<int, I...>)
{
  return std::array<laneblock_fn, sizeof...(I)>{ &launch_laneblock_one<T, LO + I>... };
}

cudaError_t launch_laneblock_f32(int bits, bool compress, const Job& j, cudaStream_t s);
cudaError_t launch_laneblock_f64(int bits, bool compress, const Job& j, cudaStream_t s);

// Jobs these kernels take of those the lane-segment kernels leave: pointers on
// 16-byte boundaries, 32 blocks within the 48 KB of shared memory that needs no
// opt-in, and block sizes where they are the faster ones.  Measured on B200, 2^26
// fp32 / 2^25 fp64 values, of the copy bandwidth, kernels before -> here.
//   compress  (from 17 values; below, the one-thread-per-block kernels: fp32 19 bits
//     E 15 0.81 there, 0.65 here)  fp32 32 bits E 17 0.26 -> 0.99, 16 bits E 63 0.22 -> 0.71,
//     13 bits E 40 0.20 -> 0.71, 9 bits E 127 0.27 -> 0.46, 13 bits E 201 0.18 -> 0.33; fp64 21
//     bits E 17 0.38 -> 1.01, 16 bits E 31 0.29 -> 0.94, 64 bits E 31 0.26 -> 0.92, 9 bits E 90
//     0.34 -> 0.49; 45 bits E 90 (39 KB) 0.35 / 0.30
//   decompress  fp32 11 bits E 9 0.36 -> 0.48, 16 bits E 31 0.43 -> 0.99, 21 bits E 63 0.49 ->
//     0.79, 27 bits E 125 (30 KB) 0.55 / 0.47; fp64 16 bits E 13
//     0.66 -> 0.98, 40 bits E 17 0.86 -> 1.00, 64 bits E 31 0.94 -> 1.02, 13 bits E 90 (28 KB)
//     0.61 -> 0.66, 19 bits E 50 (17 KB) 0.67 -> 0.76, 31 bits E 50 (19 KB) 0.74 / 0.73, 41 bits
//     E 50 (21 KB) 0.86 / 0.64
// So the chunked kernels keep decompress where few warps fit beside that much
// shared memory.
inline bool laneblock_eligible(const Job& j, std::size_t es, bool compress, const void* values, const void* words)
{
  if (((reinterpret_cast<std::uintptr_t>(values) | reinterpret_cast<std::uintptr_t>(words)) & 15u) != 0) return false;
  if (j.E < (compress ? 17 : 9) || j.E > 1024 || (j.E & (j.E - 1)) == 0) return false;
  if (j.E == 12) return false; // a compile-time block size of the one-thread-per-block kernels
  if ((j.n / (std::uint64_t)j.E) / 32 >= 0x7FFFFFFFull) return false;
  // a lane walks its block alone, so short arrays of long blocks wait for it: 31
  // values, 13 bits, fp32: compress of 300,000 values 4.9 us by the chunked kernel,
  // 5.7 here, of 1e6 7.2 / 6.8, of 3e6 13.9 / 8.4; 127 values 3e6 13.5 / 19.4
  const std::uint64_t enough = (std::uint64_t)j.E * (es == 4 ? 33000u : 66000u);
  const int any_length = compress ? 20 : j.bits > 32 ? 16 : es == 4 ? 24 : 20;
  if (j.n < enough && (j.E > any_length || (!compress && j.block_bytes % 32u == 0))) return false;
  const std::uint32_t smem = laneblock_smem(j, es, compress);
  // above 128 values the warp-per-block kernels are the others.  Few warps fit beside
  // that much shared memory, and compress needs more of them where it writes its image
  // by bytes or half-words or reads its values one by one (time here over time there,
  // compress, 2^25 fp32 / 2^24 fp64 values: bytes, fp32 4 bits E 250 36 KB 1.16, E 330 47
  // KB 1.74, fp64 4 bits E 170 46 KB 1.57; half-words, fp32 14 bits E 250 46 KB 1.34, 13
  // bits E 201 36 KB 0.61, fp64 12 bits E 150 46 KB 1.20, four values at a time 4 bits E
  // 300 43 KB 0.77; words, fp32 16 bits E 230 44 KB 0.57, 23 bits E 201 44 KB 0.94, 25 bits
  // 46 KB 1.09, images of a multiple of 32 bytes 19 bits E 201 42 KB 1.16; whole bytes, 8
  // bits E 250 40 KB 0.67; decompress 0.3 to 1.06 throughout)
  if (j.E > 128) {
    const bool quads = laneblock_quads(j.E), words = j.block_bytes % 4u == 0, bytes = j.block_bytes % 2u != 0;
    const bool any = !compress || j.bits == 8 || (words ? quads || j.block_bytes % 32u != 0 : quads && !bytes);
    return smem <= (any ? 48000u : es == 8 ? (bytes ? 40500u : 43500u) : bytes ? 35500u : 41500u);
  }
  if (compress) return smem <= (es == 4 ? 48000u : 32000u);
  // decompress: values of a multiple of 8 per block, or images of a multiple of 16
  // bytes, still meet four and more on a bank
  if (j.E % 8 == 0) return false;
  if (j.bits > 32) return smem <= 8900u && j.block_bytes % 32u != 0; // 60 bits E 17 45 us there, 54 here
  if (j.bits > 16) return smem <= (es == 4 ? (j.block_bytes % 16u == 0 ? 20000u : 24000u)
                                           : (j.block_bytes % 32u == 0 ? 12000u : 18000u));
  return smem <= (es == 4 ? 31000u : 28000u);
}

} // namespace frsz2b
