// frsz2_host.cu -- the C ABI's host-buffer calls: the codec with the copies inside
// the call, and random access on host buffers.  Host code only.
#include "frsz2_launch.hpp"

#include "../../include/frsz2_b200.h"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace frsz2b {

namespace {

// One worker's place in the staged host path: pinned and device buffers of a
// slice each way, and a stream.
struct HostSlot
{
  std::uint8_t* pin[2] = { nullptr, nullptr }; // into the device, out of it
  std::uint8_t* dev[2] = { nullptr, nullptr };
  cudaStream_t st = nullptr;
};

// Workers of the staged path at most, and the slice of values each takes at a
// time.  A slice's compressed form has at most twice its bytes (blocks of one
// value), which sizes a slot's four buffers: 48 MiB pinned and 48 MiB of device
// memory for all slots, allocated as calls first need them and kept.  Measured
// with 16 host threads, 2^23 fp64 values at 32 bits, compress / decompress (ms):
// 8 workers 4.6 / 3.1, 12 3.8 / 2.7, 15 4.0 / 2.7; 12 with slices of 256 KiB
// 5.2 / 3.8, 512 KiB 4.8 / 3.2, 2 MiB 3.8 / 2.7.
constexpr int kHostWorkers = 12;
constexpr std::size_t kHostSlice = (std::size_t)1 << 20;
constexpr std::size_t kHostSlot = 2 * kHostSlice + 4096;

struct Staging
{
  std::mutex mu;
  HostSlot slot[kHostWorkers];
  void* d_values = nullptr;
  std::size_t values_cap = 0;
  void* d_buf = nullptr;
  std::size_t buf_cap = 0;
  cudaStream_t st[2] = { nullptr, nullptr };
  cudaEvent_t ev_start = nullptr;
  bool init = false;
};

Staging g_staging[64];

int ensure(void** p, std::size_t* cap, std::size_t want)
{
  if (*cap >= want) return FRSZ2_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  const std::size_t sz = std::max<std::size_t>(want, 1 << 20);
  int rc = cuda_status(cudaMalloc(p, sz), "staging allocation");
  if (rc) return rc;
  *cap = sz;
  return FRSZ2_OK;
}

// Streams and event of a device's staging (first use; caller holds S.mu).
int staging_init(Staging& S)
{
  if (S.init) return FRSZ2_OK;
  int rc;
  for (auto& s : S.st)
    if ((rc = cuda_status(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream create"))) return rc;
  if ((rc = cuda_status(cudaEventCreateWithFlags(&S.ev_start, cudaEventDisableTiming), "event create"))) return rc;
  S.init = true;
  return FRSZ2_OK;
}

// Values per host-path slice: smaller slices shorten the pipeline's fill and
// drain (an H2D with nothing to overlap at the start of a call, a D2H at its
// end); measured end to end on the 512^3 field over PCIe 5.0 x16: 64 MiB 76.1,
// 32 MiB 78.2, 16 MiB 78.8, 8 MiB 75.3 GB/s (the link's bidirectional copy
// rate is 81.4 GB/s).
#ifndef FRSZ2_HOST_SLICE_MIB
#define FRSZ2_HOST_SLICE_MIB 16
#endif

// Slices of whole tiles so every slice keeps the tile kernel's alignment.
std::uint64_t slice_blocks(const Layout& L, int dtype)
{
  const int TE = dtype == FRSZ2_FLOAT ? tile_shape<float>::TE : tile_shape<double>::TE;
  const std::uint64_t target_values =
    ((std::uint64_t)FRSZ2_HOST_SLICE_MIB << 20) / (dtype == FRSZ2_FLOAT ? 4 : 8); // values per slice
  std::uint64_t unit = (is_pow2(L.E) && L.E <= TE) ? (std::uint64_t)(TE / L.E) : 16; // blocks
  std::uint64_t blocks = std::max<std::uint64_t>(unit, (target_values / (std::uint64_t)L.E) / unit * unit);
  return blocks;
}

int slot_init(HostSlot& h)
{
  int rc;
  for (int d = 0; d < 2; ++d) {
    if (!h.pin[d] &&
        (rc = cuda_status(cudaHostAlloc(reinterpret_cast<void**>(&h.pin[d]), kHostSlot, cudaHostAllocDefault),
                          "staging allocation")))
      return rc;
    if (!h.dev[d] && (rc = cuda_status(cudaMalloc(reinterpret_cast<void**>(&h.dev[d]), kHostSlot), "staging allocation")))
      return rc;
  }
  if (!h.st) return cuda_status(cudaStreamCreateWithFlags(&h.st, cudaStreamNonBlocking), "stream create");
  return FRSZ2_OK;
}

// Ordinary host memory, pinned host memory, or neither (device, managed).
enum class Memory { pageable, pinned, other };
Memory memory_of(const void* p)
{
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return Memory::other;
  }
  return a.type == cudaMemoryTypeUnregistered ? Memory::pageable
         : a.type == cudaMemoryTypeHost       ? Memory::pinned
                                              : Memory::other;
}

// The host path for ordinary (pageable) memory.  A copy between pageable
// memory and the device goes through the driver's own staging on the calling
// thread, one copy at a time (10 GB/s for a compress and decompress of 64 MiB);
// here several threads each take a slice at a time through a pinned slot of
// their own -- copy in, transfer, kernel, transfer, copy out -- so the copies of
// some overlap the transfers of others.  The threads live as long as the call; an
// array of one slice needs none.  Measured with 16 host threads, fp64 at 32 bits,
// compress / decompress: 2^23 values 14.1 / 6.6 -> 3.8 / 2.7 ms, 2^20 1.11 / 0.92 ->
// 0.82 / 0.60 ms, 300,001 (slices of 512 KiB up to 8 MiB; of 1 MiB 0.42 / 0.48) 0.42
// / 0.35 -> 0.30 / 0.25 ms, 4,096 69 / 57 -> 43 / 48 us.
// Returns false when no slot could be had; the caller then copies directly.
bool host_codec_staged(Staging& S, bool compress, int dtype, const Layout& L, const std::uint8_t* in,
                       std::uint8_t* out, int dev, int* result)
{
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8, wb = (std::size_t)L.W / 8;
  const std::uint64_t bytes = L.n * es;
  const std::size_t want = bytes > kHostSlice && bytes <= 8 * kHostSlice ? kHostSlice / 2 : kHostSlice;
  const std::uint64_t per = std::max<std::uint64_t>(1, want / ((std::uint64_t)L.E * es)); // blocks per slice
  const std::uint64_t slices = (L.nb + per - 1) / per;
  const unsigned hw = std::thread::hardware_concurrency();
  const int wanted = (int)std::min<std::uint64_t>(
    slices, (std::uint64_t)std::min<unsigned>(kHostWorkers, std::max(1u, hw ? hw - hw / 4 : 1u)));
  int workers = 0;
  while (workers < wanted && slot_init(S.slot[workers]) == FRSZ2_OK) ++workers;
  // a slot that cannot be had leaves its error behind, which the next launch's
  // check would take for its own
  if (workers < wanted) cudaGetLastError();
  if (workers == 0) return false;
  // the workers read the caller's input themselves, so what the caller's stream
  // still holds (a copy into a pinned input, say) has to be done before they start
  if ((*result = cuda_status(cudaEventSynchronize(S.ev_start), "event synchronize"))) return true;

  std::atomic<std::uint64_t> next{ 0 };
  std::atomic<int> status{ FRSZ2_OK };
  std::mutex err_mu;
  char err[256] = "";
  auto slice = [&](HostSlot& h, std::uint64_t k) -> int {
    const std::uint64_t b0 = k * per, nbk = std::min(per, L.nb - b0);
    const std::uint64_t e0 = b0 * (std::uint64_t)L.E;
    const std::uint64_t ne = std::min<std::uint64_t>(L.n - e0, nbk * (std::uint64_t)L.E);
    const std::size_t exp_len = nbk * wb, w_at = (exp_len + 255) / 256 * 256; // exponents, then words, in a slot
    const std::size_t w_len = nbk * (std::size_t)L.block_bytes;
    const std::uint64_t exp_off = b0 * wb, w_off = L.exp_bytes + b0 * (std::uint64_t)L.block_bytes;
    Layout P = L;
    P.n = ne;
    Job j = make_job(P, dtype);
    int rc;
    if (compress) {
      j.values_in = h.dev[0];
      j.exps = h.dev[1];
      j.words = h.dev[1] + w_at;
      // only the bytes the reference writes go to the caller: of a partial last
      // block, the words its values reach
      const std::size_t out_len = w_len - L.block_bytes +
                                  written_block_bytes((int)(ne - (nbk - 1) * (std::uint64_t)L.E), L.bits, L.W);
      std::memcpy(h.pin[0], in + e0 * es, ne * es);
      if ((rc = cuda_status(cudaMemcpyAsync(h.dev[0], h.pin[0], ne * es, cudaMemcpyHostToDevice, h.st), "H2D")) ||
          (rc = launch_compress(j, dtype, h.st, nullptr)) ||
          (rc = cuda_status(cudaMemcpyAsync(h.pin[1], h.dev[1], w_at + out_len, cudaMemcpyDeviceToHost, h.st),
                            "D2H")) ||
          (rc = cuda_status(cudaStreamSynchronize(h.st), "stream sync")))
        return rc;
      std::memcpy(out + exp_off, h.pin[1], exp_len);
      std::memcpy(out + w_off, h.pin[1] + w_at, out_len);
    } else {
      j.exps = h.dev[0];
      j.words = h.dev[0] + w_at;
      j.values_out = h.dev[1];
      std::memcpy(h.pin[0], in + exp_off, exp_len);
      std::memcpy(h.pin[0] + w_at, in + w_off, w_len);
      if ((rc = cuda_status(cudaMemcpyAsync(h.dev[0], h.pin[0], w_at + w_len, cudaMemcpyHostToDevice, h.st), "H2D")) ||
          (rc = launch_decompress(j, dtype, h.st, nullptr)) ||
          (rc = cuda_status(cudaMemcpyAsync(h.pin[1], h.dev[1], ne * es, cudaMemcpyDeviceToHost, h.st), "D2H")) ||
          (rc = cuda_status(cudaStreamSynchronize(h.st), "stream sync")))
        return rc;
      std::memcpy(out + e0 * es, h.pin[1], ne * es);
    }
    return FRSZ2_OK;
  };
  auto work = [&](int w) noexcept {
    int rc = FRSZ2_OK;
    bool thrown = false;
    try {
      rc = w == 0 ? FRSZ2_OK : cuda_status(cudaSetDevice(dev), "cudaSetDevice");
      for (std::uint64_t k; !rc && status.load(std::memory_order_relaxed) == FRSZ2_OK &&
                            (k = next.fetch_add(1, std::memory_order_relaxed)) < slices;)
        rc = slice(S.slot[w], k);
    } catch (...) { // a thread must not end the process, nor this one leave others behind
      rc = FRSZ2_EFAIL;
      thrown = true;
    }
    if (rc) {
      cudaStreamSynchronize(S.slot[w].st); // nothing of this call stays in flight
      std::lock_guard<std::mutex> g(err_mu);
      if (status.load() == FRSZ2_OK) {
        std::snprintf(err, sizeof err, "%s", thrown ? "out of host memory" : last_error()); // this thread's
        status.store(rc);
      }
    }
  };
  std::vector<std::thread> threads;
  try {
    threads.reserve((std::size_t)workers);
    for (int w = 1; w < workers; ++w) threads.emplace_back(work, w);
  } catch (...) {
    // no more threads to be had: those there are and this one take all the slices
  }
  work(0);
  for (auto& t : threads) t.join();
  *result = status.load() == FRSZ2_OK ? FRSZ2_OK : set_error(status.load(), err);
  return true;
}

} // namespace

int host_codec(bool compress, int dtype, int bits, int E, const void* h_in, std::uint64_t n, void* h_out,
               cudaStream_t user)
{
  int rc = check_args(dtype, bits, E);
  if (rc) return rc;
  if ((!h_in || !h_out) && n > 0) return set_error(FRSZ2_EFAIL, "null pointer");
  const Layout L = make_layout(n, bits, E);
  if (n == 0) return FRSZ2_OK;
  int dev = 0;
  rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return set_error(FRSZ2_EFAIL, "device index out of range");
  Staging& S = g_staging[dev];
  std::lock_guard<std::mutex> lock(S.mu);
  if ((rc = staging_init(S))) return rc;
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  const std::uint8_t* hb_in = static_cast<const std::uint8_t*>(h_in);
  std::uint8_t* hb_out = static_cast<std::uint8_t*>(h_out);

  // order after prior work on the caller's stream
  if ((rc = cuda_status(cudaEventRecord(S.ev_start, user), "event record"))) return rc;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(user, &cap) != cudaSuccess) cudaGetLastError();
  // buffers pinned on both sides transfer directly, and what is not host memory,
  // or a capturing stream, keeps that path's refusal; with one side pinned the
  // direct path has one side's copies less, which the staged one makes up for only in
  // short and long arrays (64-bit values at 32 bits, input ordinary, us direct /
  // staged: 4,096 values 52 / 30, 2^16 77 / 78, 2^18 184 / 217, 2^20 577 / 585, 2^22
  // 3,424 / 1,485; decompress, output ordinary: 34 / 36, 82 / 83, 181 / 161, 549 / 502,
  // 2,157 / 1,213; 2^18 fp32 at 16 bits 109 / 152 and 124 / 154)
  const Memory mi = memory_of(h_in), mo = memory_of(h_out);
  const bool host = mi != Memory::other && mo != Memory::other, one = mi != mo;
  const std::uint64_t bytes = L.n * es;
  const bool staged = cap == cudaStreamCaptureStatusNone && host && (mi == Memory::pageable || mo == Memory::pageable) &&
                      (!one || bytes <= kHostSlice / 16 || bytes > 8 * kHostSlice);
  if (staged && host_codec_staged(S, compress, dtype, L, hb_in, hb_out, dev, &rc)) return rc;

  if ((rc = ensure(&S.d_values, &S.values_cap, L.n * es))) return rc;
  if ((rc = ensure(&S.d_buf, &S.buf_cap, L.total_bytes))) return rc;
  std::uint8_t* d_buf = static_cast<std::uint8_t*>(S.d_buf);
  for (auto& s : S.st)
    if ((rc = cuda_status(cudaStreamWaitEvent(s, S.ev_start, 0), "stream wait"))) return rc;

  const std::uint64_t per = slice_blocks(L, dtype);
  int k = 0;
  for (std::uint64_t b0 = 0; b0 < L.nb; b0 += per, ++k) {
    cudaStream_t s = S.st[k & 1];
    const std::uint64_t nbk = std::min(per, L.nb - b0);
    const std::uint64_t e0 = b0 * (std::uint64_t)E;
    const std::uint64_t ne = std::min<std::uint64_t>(L.n - e0, nbk * (std::uint64_t)E);
    const bool last = b0 + nbk == L.nb;
    const std::uint64_t exp_off = b0 * (std::uint64_t)(L.W / 8), exp_len = nbk * (std::uint64_t)(L.W / 8);
    const std::uint64_t w_off = L.exp_bytes + b0 * (std::uint64_t)L.block_bytes;
    // bytes the reference writes for this slice: whole blocks, except only
    // the written words of a partial last block
    const int last_cnt = (int)(ne - (nbk - 1) * (std::uint64_t)E);
    const std::uint64_t w_len =
      (nbk - 1) * (std::uint64_t)L.block_bytes +
      (last ? written_block_bytes(last_cnt, bits, L.W) : L.block_bytes);
    if (compress) {
      Job j = job_for_slice(L, dtype, b0, nbk, S.d_values, nullptr, d_buf);
      if ((rc = cuda_status(cudaMemcpyAsync(static_cast<std::uint8_t*>(S.d_values) + e0 * es, hb_in + e0 * es,
                                            ne * es, cudaMemcpyHostToDevice, s),
                            "H2D")))
        return rc;
      if ((rc = launch_compress(j, dtype, s, nullptr))) return rc;
      if ((rc = cuda_status(cudaMemcpyAsync(hb_out + exp_off, d_buf + exp_off, exp_len, cudaMemcpyDeviceToHost, s),
                            "D2H")))
        return rc;
      if ((rc = cuda_status(cudaMemcpyAsync(hb_out + w_off, d_buf + w_off, w_len, cudaMemcpyDeviceToHost, s), "D2H")))
        return rc;
    } else {
      Job j = job_for_slice(L, dtype, b0, nbk, nullptr, S.d_values, d_buf);
      if ((rc = cuda_status(cudaMemcpyAsync(d_buf + exp_off, hb_in + exp_off, exp_len, cudaMemcpyHostToDevice, s),
                            "H2D")))
        return rc;
      // whole blocks are read by the tile kernel; copy the full slice (the
      // buffer always holds whole blocks)
      if ((rc = cuda_status(cudaMemcpyAsync(d_buf + w_off, hb_in + w_off, nbk * (std::uint64_t)L.block_bytes,
                                            cudaMemcpyHostToDevice, s),
                            "H2D")))
        return rc;
      if ((rc = launch_decompress(j, dtype, s, nullptr))) return rc;
      if ((rc = cuda_status(cudaMemcpyAsync(hb_out + e0 * es, static_cast<std::uint8_t*>(S.d_values) + e0 * es,
                                            ne * es, cudaMemcpyDeviceToHost, s),
                            "D2H")))
        return rc;
    }
  }
  for (auto& s : S.st)
    if ((rc = cuda_status(cudaStreamSynchronize(s), "stream sync"))) return rc;
  return FRSZ2_OK;
}

} // namespace frsz2b

using namespace frsz2b;

extern "C" {

int frsz2_compress_host(int dtype, int bits, int block_size, const void* h_values, uint64_t n, void* h_compressed,
                        void* stream)
{
  NvtxRange nvtx("frsz2_compress_host");
  return host_codec(true, dtype, bits, block_size, h_values, n, h_compressed, static_cast<cudaStream_t>(stream));
}

int frsz2_decompress_host(int dtype, int bits, int block_size, const void* h_compressed, uint64_t n, void* h_values,
                          void* stream)
{
  NvtxRange nvtx("frsz2_decompress_host");
  return host_codec(false, dtype, bits, block_size, h_compressed, n, h_values, static_cast<cudaStream_t>(stream));
}

// Host-buffer random access (decompress_cpu_element, include/frsz2.hpp:1199-1214):
// the host gathers the exponent and block bytes of every block a valid index
// falls in into a small buffer laid out as an array of those blocks, which
// the element kernel decodes on the GPU.
int frsz2_decompress_elements_host(int dtype, int bits, int block_size, const void* h_compressed, uint64_t n,
                                   const uint64_t* h_idx, uint64_t count, void* h_out)
{
  NvtxRange nvtx("frsz2_decompress_elements_host");
  int rc = check_args(dtype, bits, block_size);
  if (rc) return rc;
  if (count == 0) return FRSZ2_OK;
  if (!h_compressed || !h_idx || !h_out) return set_error(FRSZ2_EFAIL, "null pointer");
  const Layout L = make_layout(n, bits, block_size);
  const std::uint64_t E = (std::uint64_t)block_size, EB = (std::uint64_t)(L.W / 8), BB = L.block_bytes;
  std::vector<std::uint64_t> blocks;
  blocks.reserve(count);
  for (std::uint64_t t = 0; t < count; ++t)
    if (h_idx[t] < n) blocks.push_back(h_idx[t] / E);
  if (blocks.empty()) return FRSZ2_OK; // every index out of range: outputs untouched
  std::sort(blocks.begin(), blocks.end());
  blocks.erase(std::unique(blocks.begin(), blocks.end()), blocks.end());
  const std::uint64_t m = blocks.size();
  const Layout M = make_layout(m * E, bits, block_size);
  const std::uint8_t* hb = static_cast<const std::uint8_t*>(h_compressed);
  std::vector<std::uint8_t> mini(M.total_bytes, 0);
  for (std::uint64_t k = 0; k < m; ++k) {
    std::memcpy(mini.data() + k * EB, hb + blocks[k] * EB, EB);
    std::memcpy(mini.data() + M.exp_bytes + k * BB, hb + L.exp_bytes + blocks[k] * BB, BB);
  }
  std::vector<std::uint64_t> mapped(count);
  for (std::uint64_t t = 0; t < count; ++t) {
    const std::uint64_t g = h_idx[t];
    if (g >= n) {
      mapped[t] = ~0ull; // the kernel skips it
      continue;
    }
    const std::uint64_t k = (std::uint64_t)(std::lower_bound(blocks.begin(), blocks.end(), g / E) - blocks.begin());
    mapped[t] = k * E + g % E;
  }

  int dev = 0;
  if ((rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice"))) return rc;
  if (dev < 0 || dev >= 64) return set_error(FRSZ2_EFAIL, "device index out of range");
  Staging& S = g_staging[dev];
  std::lock_guard<std::mutex> lock(S.mu);
  if ((rc = staging_init(S))) return rc;
  const std::size_t es = dtype == FRSZ2_FLOAT ? 4 : 8;
  const std::size_t idx_off = (M.total_bytes + 255) / 256 * 256;
  if ((rc = ensure(&S.d_buf, &S.buf_cap, idx_off + count * sizeof(std::uint64_t)))) return rc;
  if ((rc = ensure(&S.d_values, &S.values_cap, count * es))) return rc;
  std::uint8_t* d_buf = static_cast<std::uint8_t*>(S.d_buf);
  auto* d_idx = reinterpret_cast<std::uint64_t*>(d_buf + idx_off);
  cudaStream_t s = S.st[0];
  if ((rc = cuda_status(cudaMemcpyAsync(d_buf, mini.data(), M.total_bytes, cudaMemcpyHostToDevice, s), "H2D")) ||
      (rc = cuda_status(cudaMemcpyAsync(d_idx, mapped.data(), count * sizeof(std::uint64_t), cudaMemcpyHostToDevice,
                                        s),
                        "H2D")) ||
      (rc = cuda_status(cudaMemcpyAsync(S.d_values, h_out, count * es, cudaMemcpyHostToDevice, s), "H2D")))
    return rc;
  Job j = job_for_slice(M, dtype, 0, M.nb, nullptr, nullptr, d_buf);
  if ((rc = launch_elements(j, dtype, d_idx, count, S.d_values, s))) return rc;
  if ((rc = cuda_status(cudaMemcpyAsync(h_out, S.d_values, count * es, cudaMemcpyDeviceToHost, s), "D2H"))) return rc;
  return cuda_status(cudaStreamSynchronize(s), "stream synchronize");
}

} // extern "C"
