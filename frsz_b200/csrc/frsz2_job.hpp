// frsz2_job.hpp -- one array (or a slice of one) as the kernels take it, and the
// tile geometry; no device code, so host-only sources can include it.
#pragma once

#include "frsz2_common.cuh"

namespace frsz2b {

constexpr int kNT = 256; // threads per CTA
constexpr int kR = 4;    // 128-bit vectors per thread per tile

template<class T>
struct tile_shape
{
  static constexpr int V = 16 / (int)sizeof(T); // values per 128-bit vector
  static constexpr int TE = kNT * kR * V;       // values per tile
};

// One array (or a block-aligned slice of one): pointers are to the slice's
// first exponent and first block, so slices of one buffer can run on
// different streams.
struct Job
{
  const void* values_in; // compress: T input
  void* values_out;      // decompress: T output
  std::uint8_t* exps;    // exponent of block 0 of this slice
  std::uint8_t* words;   // words of block 0 of this slice
  std::uint64_t n;       // values in this slice
  std::uint64_t tiles;   // tile kernels: ceil(n / TE)
  std::uint32_t block_bytes;
  std::int32_t bits, E, W;
  std::int32_t log2E;
  std::uint32_t tile_blocks; // TE / E
  std::uint32_t m_bb;        // ceil(2^32 / block_bytes)
  std::uint32_t m_bits;      // ceil(2^32 / bits)
};

} // namespace frsz2b
