// frsz2_capi.cu -- C ABI of libfrsz2_b200.so: argument checks, kernel choice,
// and launch geometry.
#include "frsz2_blockwise.cuh"
#include "frsz2_chunked.cuh"
#include "frsz2_chunked_ct.cuh"
#include "frsz2_fast_dispatch.hpp"
#include "frsz2_kernels.cuh"
#include "frsz2_laneblock.cuh"
#include "frsz2_launch.hpp"

#include "../../include/frsz2_b200.h"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <string>

namespace frsz2b {

namespace {
thread_local std::string g_last_error;
}

bool& early_launch()
{
  thread_local bool on = false;
  return on;
}

int set_error(int code, const std::string& msg)
{
  g_last_error = msg;
  return code;
}

const char* last_error() { return g_last_error.c_str(); }

int cuda_status(cudaError_t e, const char* what)
{
  if (e == cudaSuccess) return FRSZ2_OK;
  return set_error(FRSZ2_EFAIL, std::string(what) + ": " + cudaGetErrorString(e));
}

int check_args(int dtype, int bits, int E)
{
  if (dtype != FRSZ2_FLOAT && dtype != FRSZ2_DOUBLE) return set_error(FRSZ2_EDTYPE, "unsupported dtype");
  const int max_bits = dtype == FRSZ2_FLOAT ? 32 : 64;
  if (bits < 4 || bits > max_bits) return set_error(FRSZ2_EFAIL, "Unsupported number of bits: " + std::to_string(bits));
  if (E < 1 || E > kMaxBlockSize)
    return set_error(FRSZ2_EFAIL, "Unsupported exponent block size: " + std::to_string(E));
  return FRSZ2_OK;
}

int sm_count()
{
  // per device, queried once (threads racing on the first call store the
  // same value)
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int c = cached[dev].load(std::memory_order_relaxed);
  if (c == 0) {
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0) c = 148;
    cached[dev].store(c, std::memory_order_relaxed);
  }
  return c;
}

static int ilog2(int x)
{
  int l = 0;
  while ((1 << l) < x) ++l;
  return l;
}

Job make_job(const Layout& L, int dtype)
{
  Job j{};
  j.n = L.n;
  j.block_bytes = L.block_bytes;
  j.bits = L.bits;
  j.E = L.E;
  j.W = L.W;
  j.log2E = is_pow2(L.E) ? ilog2(L.E) : -1;
  const int TE = dtype == FRSZ2_FLOAT ? tile_shape<float>::TE : tile_shape<double>::TE;
  j.tile_blocks = (L.E <= TE && is_pow2(L.E)) ? (std::uint32_t)(TE / L.E) : 0u;
  j.tiles = (L.n + (std::uint64_t)TE - 1) / (std::uint64_t)TE;
  j.m_bb = L.block_bytes >= 2 ? (std::uint32_t)((((1ull << 32) + L.block_bytes - 1) / L.block_bytes)) : 0u;
  j.m_bits = (std::uint32_t)((((1ull << 32) + (std::uint64_t)L.bits - 1) / (std::uint64_t)L.bits));
  return j;
}

bool tile_eligible(const Job& j, int dtype, const void* values, const void* words)
{
  const int V = dtype == FRSZ2_FLOAT ? tile_shape<float>::V : tile_shape<double>::V;
  const int TE = dtype == FRSZ2_FLOAT ? tile_shape<float>::TE : tile_shape<double>::TE;
  if (!is_pow2(j.E) || j.E < 8 || j.E > TE || j.E < V) return false;
  if (j.block_bytes % 4 != 0) return false;
  if (((std::uint64_t)j.tile_blocks * j.block_bytes) % 16 != 0) return false;
  if (reinterpret_cast<std::uintptr_t>(values) % 16 != 0) return false;
  if (reinterpret_cast<std::uintptr_t>(words) % 16 != 0) return false;
  return true;
}

template<class T>
static std::size_t compress_smem(int bits)
{
  constexpr int TE = tile_shape<T>::TE, V = tile_shape<T>::V;
  const std::size_t cv = (sizeof(T) == 8 && bits > 32) ? 8 : 4;
  return TE * cv + (TE / (32 * V)) * 4;
}

template<class T>
static std::size_t decompress_smem(const Job& j)
{
  const std::uint32_t tile_bytes = j.tile_blocks * j.block_bytes;
  return decompress_tile_exp_offset<T>(tile_bytes) + (std::size_t)j.tile_blocks * 8;
}

static unsigned grid_for(std::uint64_t work_items, std::uint64_t per_cta)
{
  const std::uint64_t need = (work_items + per_cta - 1) / per_cta;
  const std::uint64_t cap = (std::uint64_t)sm_count() * 64;
  return (unsigned)std::max<std::uint64_t>(1, std::min(need, cap));
}

// Compile-time-width kernels when an instance and the layout allow it;
// cudaErrorNotSupported means "use the runtime-width kernels".
template<class T>
static cudaError_t try_fast(bool compress, const Job& j, cudaStream_t s)
{
  // one CTA per tile, of down to half a tile each; an array beyond that (terabytes)
  // goes to the kernels that loop
  if (j.tiles > (1u << 29)) return cudaErrorNotSupported;
  const void* values = compress ? j.values_in : j.values_out;
  const unsigned grid = (unsigned)j.tiles;
  if (fast_eligible(j, sizeof(T) == 8, values, j.words))
    return sizeof(T) == 8 ? launch_fast_f64(j.bits, compress, j, s, grid)
                          : launch_fast_f32(j.bits, compress, j, s, grid);
  if (small_block_eligible(j, sizeof(T) == 8, values, j.words))
    return sizeof(T) == 8 ? launch_fast_small_f64(j.bits, j.E, compress, j, s, grid)
                          : launch_fast_small_f32(j.bits, j.E, compress, j, s, grid);
  if (fast_mis_eligible(j, sizeof(T) == 8, values, j.words))
    return sizeof(T) == 8 ? launch_fast_mis_f64(j.bits, compress, j, s, grid)
                          : launch_fast_mis_f32(j.bits, compress, j, s, grid);
  if (const std::uint32_t tb = fast_gen_tile_blocks(j, sizeof(T) == 8, values, j.words)) {
    // block sizes that are a multiple of a lane's values: tiles of tb whole blocks
    Job t = j;
    const std::uint64_t tv = (std::uint64_t)tb * (std::uint64_t)j.E;
    t.tile_blocks = tb;
    t.tiles = (j.n + tv - 1) / tv;
    const unsigned g = (unsigned)t.tiles;
    return sizeof(T) == 8 ? launch_fast_gen_f64(j.bits, compress, t, s, g)
                          : launch_fast_gen_f32(j.bits, compress, t, s, g);
  }
  return cudaErrorNotSupported;
}


template<class T>
static int launch_compress_t(const Job& j, int dtype, cudaStream_t s, bool* used_tile)
{
  if (j.n == 0) return FRSZ2_OK;
  const cudaError_t fe = try_fast<T>(true, j, s);
  if (fe != cudaErrorNotSupported) {
    if (used_tile) *used_tile = true;
    return cuda_status(fe, "compress launch");
  }
  const bool tile = tile_eligible(j, dtype, j.values_in, j.words);
  if (used_tile) *used_tile = tile;
  if (tile) {
    const unsigned grid = (unsigned)std::min<std::uint64_t>(j.tiles, 1u << 30);
    if (sizeof(T) == 8 && j.bits > 32)
      launch(k_compress_tile<T, std::uint64_t>, grid, kNT, compress_smem<T>(j.bits), s, j);
    else
      launch(k_compress_tile<T, std::uint32_t>, grid, kNT, compress_smem<T>(j.bits), s, j);
  } else if (laneblock_eligible(j, sizeof(T), true, j.values_in, j.words)) {
    return cuda_status(sizeof(T) == 8 ? launch_laneblock_f64(j.bits, true, j, s)
                                      : launch_laneblock_f32(j.bits, true, j, s),
                       "compress launch");
  } else if (blockwise_eligible(j)) {
    return cuda_status(sizeof(T) == 8 ? launch_blockwise_f64(j.bits, true, j, s)
                                      : launch_blockwise_f32(j.bits, true, j, s),
                       "compress launch");
  } else if (chunked_ct_eligible(j)) {
    return cuda_status(sizeof(T) == 8 ? launch_chunked_ct_f64(j.bits, true, j, s)
                                      : launch_chunked_ct_f32(j.bits, true, j, s),
                       "compress launch");
  } else {
    const std::uint64_t nb = (j.n + (std::uint64_t)j.E - 1) / (std::uint64_t)j.E;
    launch(k_compress_generic<T>, grid_for(nb, kNT / 32), kNT, 0, s, j);
  }
  return cuda_status(cudaGetLastError(), "compress launch");
}

template<class T>
static int launch_decompress_t(const Job& j, int dtype, cudaStream_t s, bool* used_tile)
{
  if (j.n == 0) return FRSZ2_OK;
  const cudaError_t fe = try_fast<T>(false, j, s);
  if (fe != cudaErrorNotSupported) {
    if (used_tile) *used_tile = true;
    return cuda_status(fe, "decompress launch");
  }
  const bool tile = tile_eligible(j, dtype, j.values_out, j.words);
  if (used_tile) *used_tile = tile;
  if (tile) {
    const unsigned grid = (unsigned)std::min<std::uint64_t>(j.tiles, 1u << 30);
    if (sizeof(T) == 8 && j.bits > 32)
      launch(k_decompress_tile<T, std::uint64_t>, grid, kNT, decompress_smem<T>(j), s, j);
    else
      launch(k_decompress_tile<T, std::uint32_t>, grid, kNT, decompress_smem<T>(j), s, j);
  } else if (laneblock_eligible(j, sizeof(T), false, j.values_out, j.words)) {
    return cuda_status(sizeof(T) == 8 ? launch_laneblock_f64(j.bits, false, j, s)
                                      : launch_laneblock_f32(j.bits, false, j, s),
                       "decompress launch");
  } else if (blockwise_eligible(j)) {
    return cuda_status(sizeof(T) == 8 ? launch_blockwise_f64(j.bits, false, j, s)
                                      : launch_blockwise_f32(j.bits, false, j, s),
                       "decompress launch");
  } else if (chunked_ct_eligible(j)) {
    return cuda_status(sizeof(T) == 8 ? launch_chunked_ct_f64(j.bits, false, j, s)
                                      : launch_chunked_ct_f32(j.bits, false, j, s),
                       "decompress launch");
  } else {
    const std::uint64_t nb = (j.n + (std::uint64_t)j.E - 1) / (std::uint64_t)j.E;
    launch(k_decompress_generic<T>, grid_for(nb, kNT / 32), kNT, 0, s, j);
  }
  return cuda_status(cudaGetLastError(), "decompress launch");
}

int launch_compress(const Job& j, int dtype, cudaStream_t s, bool* used_tile)
{
  return dtype == FRSZ2_FLOAT ? launch_compress_t<float>(j, dtype, s, used_tile)
                              : launch_compress_t<double>(j, dtype, s, used_tile);
}

int launch_decompress(const Job& j, int dtype, cudaStream_t s, bool* used_tile)
{
  return dtype == FRSZ2_FLOAT ? launch_decompress_t<float>(j, dtype, s, used_tile)
                              : launch_decompress_t<double>(j, dtype, s, used_tile);
}

template<class T>
static void launch_elements_t(const Job& j, const std::uint64_t* idx, std::uint64_t count, T* out, cudaStream_t s)
{
  const unsigned grid = grid_for(count, kNT);
  const std::uint64_t mE = j.log2E < 0 ? ~0ull / (std::uint64_t)j.E + 1 : 0; // E not a power of two
  switch (j.W) {
    case 8: launch(k_decompress_elements<T, 8>, grid, kNT, 0, s, j, mE, idx, count, out); break;
    case 16: launch(k_decompress_elements<T, 16>, grid, kNT, 0, s, j, mE, idx, count, out); break;
    case 32: launch(k_decompress_elements<T, 32>, grid, kNT, 0, s, j, mE, idx, count, out); break;
    default:
      if constexpr (sizeof(T) == 8) launch(k_decompress_elements<T, 64>, grid, kNT, 0, s, j, mE, idx, count, out);
  }
}

int launch_elements(const Job& j, int dtype, const std::uint64_t* idx, std::uint64_t count, void* out,
                    cudaStream_t s)
{
  if (dtype == FRSZ2_FLOAT)
    launch_elements_t<float>(j, idx, count, static_cast<float*>(out), s);
  else
    launch_elements_t<double>(j, idx, count, static_cast<double*>(out), s);
  return cuda_status(cudaGetLastError(), "element decode launch");
}

static int check_alignment(int dtype, const Layout& L, const void* values, const void* buf)
{
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  if (reinterpret_cast<std::uintptr_t>(values) % es != 0)
    return set_error(FRSZ2_EFAIL, "value pointer is not aligned to the element size");
  if (reinterpret_cast<std::uintptr_t>(buf) % (std::size_t)(L.W / 8) != 0)
    return set_error(FRSZ2_EFAIL, "compressed pointer is not aligned to the word size");
  return FRSZ2_OK;
}

Job job_for_slice(const Layout& L, int dtype, std::uint64_t b0, std::uint64_t nblocks, const void* vin, void* vout,
                  std::uint8_t* buf)
{
  Layout S = L;
  const std::uint64_t e0 = b0 * (std::uint64_t)L.E;
  S.n = std::min<std::uint64_t>(L.n - e0, nblocks * (std::uint64_t)L.E);
  Job j = make_job(S, dtype);
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  j.values_in = vin ? static_cast<const std::uint8_t*>(vin) + e0 * es : nullptr;
  j.values_out = vout ? static_cast<std::uint8_t*>(vout) + e0 * es : nullptr;
  j.exps = buf + b0 * (std::uint64_t)(L.W / 8);
  j.words = buf + L.exp_bytes + b0 * (std::uint64_t)L.block_bytes;
  return j;
}

// ---------------------------------------------------------------- host path

} // namespace frsz2b

using namespace frsz2b;

extern "C" {

void register_frsz(void) {}

const char* frsz2_version(void) { return "0.0.2-b200"; }

const char* frsz2_last_error(void) { return frsz2b::last_error(); }

int frsz2_compressed_size(int dtype, int bits, int block_size, uint64_t n, uint64_t* total_bytes)
{
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (!total_bytes) return set_error(FRSZ2_EFAIL, "null pointer");
  *total_bytes = make_layout(n, bits, block_size).total_bytes;
  return FRSZ2_OK;
}

int frsz2_exponent_size(int dtype, int bits, int block_size, uint64_t n, uint64_t* exponent_bytes)
{
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (!exponent_bytes) return set_error(FRSZ2_EFAIL, "null pointer");
  *exponent_bytes = make_layout(n, bits, block_size).exp_bytes;
  return FRSZ2_OK;
}

int frsz2_compress(int dtype, int bits, int block_size, const void* d_values, uint64_t n, void* d_compressed,
                   void* stream)
{
  NvtxRange nvtx("frsz2_compress");
  EarlyLaunch early;
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (n == 0) return FRSZ2_OK;
  if (!d_values || !d_compressed) return set_error(FRSZ2_EFAIL, "null pointer");
  const Layout L = make_layout(n, bits, block_size);
  if ((rc = check_alignment(dtype, L, d_values, d_compressed))) return rc;
  Job j = job_for_slice(L, dtype, 0, L.nb, d_values, nullptr, static_cast<std::uint8_t*>(d_compressed));
  return launch_compress(j, dtype, static_cast<cudaStream_t>(stream), nullptr);
}

int frsz2_decompress(int dtype, int bits, int block_size, const void* d_compressed, uint64_t n, void* d_values,
                     void* stream)
{
  NvtxRange nvtx("frsz2_decompress");
  EarlyLaunch early;
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (n == 0) return FRSZ2_OK;
  if (!d_values || !d_compressed) return set_error(FRSZ2_EFAIL, "null pointer");
  const Layout L = make_layout(n, bits, block_size);
  if ((rc = check_alignment(dtype, L, d_values, d_compressed))) return rc;
  Job j = job_for_slice(L, dtype, 0, L.nb, nullptr, d_values,
                        const_cast<std::uint8_t*>(static_cast<const std::uint8_t*>(d_compressed)));
  return launch_decompress(j, dtype, static_cast<cudaStream_t>(stream), nullptr);
}

static int block_range_args(int dtype, int bits, int E, std::uint64_t n, std::uint64_t b0, std::uint64_t count,
                            const void* values, const void* buf, Layout* L)
{
  if (int rc = check_args(dtype, bits, E)) return rc;
  *L = make_layout(n, bits, E);
  if (b0 > L->nb || count > L->nb - b0) return set_error(FRSZ2_EFAIL, "block range outside the array");
  if (count == 0) return FRSZ2_OK;
  if (!values || !buf) return set_error(FRSZ2_EFAIL, "null pointer");
  return check_alignment(dtype, *L, values, buf);
}

int frsz2_compress_blocks(int dtype, int bits, int block_size, const void* d_values, uint64_t n, uint64_t block_begin,
                          uint64_t block_count, void* d_compressed, void* stream)
{
  NvtxRange nvtx("frsz2_compress_blocks");
  EarlyLaunch early;
  Layout L;
  if (int rc = block_range_args(dtype, bits, block_size, n, block_begin, block_count, d_values, d_compressed, &L))
    return rc;
  if (block_count == 0) return FRSZ2_OK;
  // job_for_slice offsets the value pointer by the range's first value itself
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  const void* base = static_cast<const std::uint8_t*>(d_values) - block_begin * (std::uint64_t)block_size * es;
  Job j = job_for_slice(L, dtype, block_begin, block_count, base, nullptr, static_cast<std::uint8_t*>(d_compressed));
  return launch_compress(j, dtype, static_cast<cudaStream_t>(stream), nullptr);
}

int frsz2_decompress_blocks(int dtype, int bits, int block_size, const void* d_compressed, uint64_t n,
                            uint64_t block_begin, uint64_t block_count, void* d_values, void* stream)
{
  NvtxRange nvtx("frsz2_decompress_blocks");
  EarlyLaunch early;
  Layout L;
  if (int rc = block_range_args(dtype, bits, block_size, n, block_begin, block_count, d_values, d_compressed, &L))
    return rc;
  if (block_count == 0) return FRSZ2_OK;
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  void* base = static_cast<std::uint8_t*>(d_values) - block_begin * (std::uint64_t)block_size * es;
  Job j = job_for_slice(L, dtype, block_begin, block_count, nullptr, base,
                        const_cast<std::uint8_t*>(static_cast<const std::uint8_t*>(d_compressed)));
  return launch_decompress(j, dtype, static_cast<cudaStream_t>(stream), nullptr);
}

int frsz2_decompress_elements(int dtype, int bits, int block_size, const void* d_compressed, uint64_t n,
                              const uint64_t* d_idx, uint64_t count, void* d_out, void* stream)
{
  NvtxRange nvtx("frsz2_decompress_elements");
  EarlyLaunch early;
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (count == 0) return FRSZ2_OK;
  if (!d_compressed || !d_idx || !d_out) return set_error(FRSZ2_EFAIL, "null pointer");
  const Layout L = make_layout(n, bits, block_size);
  if ((rc = check_alignment(dtype, L, d_out, d_compressed))) return rc;
  Job j = job_for_slice(L, dtype, 0, L.nb, nullptr, nullptr,
                        const_cast<std::uint8_t*>(static_cast<const std::uint8_t*>(d_compressed)));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return launch_elements(j, dtype, d_idx, count, d_out, s);
}

} // extern "C"
