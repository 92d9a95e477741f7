// The host-buffer calls (frsz_b200/csrc/frsz2_host.cu) against a stand-in CUDA
// runtime on the CPU: a stream is a list of operations that run when something
// waits for them, so a read that does not wait for earlier work of a stream
// always sees the old bytes, and allocations fail when the test says so.
// host_path_test <scenario>; exit status 0 when it holds.
#include "../../frsz_b200/csrc/frsz2_launch.hpp"
#include "../../include/frsz2_b200.h"
#include "../../oracle/frsz2_oracle.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <new>
#include <vector>

// ---------------------------------------------------------------- runtime

struct CUstream_st
{
  std::vector<std::function<void()>> ops;
  std::size_t done = 0;
  void run_to(std::size_t n)
  {
    while (done < n && done < ops.size()) {
      const std::size_t k = done++;
      ops[k]();
    }
  }
};
struct CUevent_st
{
  CUstream_st* s = nullptr;
  std::size_t at = 0;
};

static std::recursive_mutex g_mu;
static thread_local cudaError_t t_last = cudaSuccess;
static std::atomic<int> g_host_allocs{ 1 << 30 }; // pinned allocations that still succeed
static std::atomic<int> g_throw_in{ 1 << 30 };    // codec launches until one throws
static std::map<const std::uint8_t*, std::size_t> g_pinned;
using Lock = std::lock_guard<std::recursive_mutex>;

static cudaError_t fail(cudaError_t e) { return t_last = e; }
static void push(cudaStream_t s, std::function<void()> f)
{
  Lock l(g_mu);
  s->ops.push_back(std::move(f));
}

extern "C" {
cudaError_t cudaGetLastError(void)
{
  const cudaError_t e = t_last;
  t_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaGetDevice(int* d)
{
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n)
{
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
  if (g_host_allocs.fetch_sub(1) <= 0) return fail(cudaErrorMemoryAllocation);
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
  *s = new CUstream_st;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
  *e = new CUevent_st;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
  Lock l(g_mu);
  *e = CUevent_st{ s, s->ops.size() };
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
  const CUevent_st at = *e;
  push(s, [at] { at.s->run_to(at.at); });
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
  Lock l(g_mu);
  e->s->run_to(e->at);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
  Lock l(g_mu);
  s->run_to(s->ops.size());
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c)
{
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
  push(st, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
  const auto* b = static_cast<const std::uint8_t*>(p);
  auto it = g_pinned.upper_bound(b);
  const bool in = it != g_pinned.begin() && (--it, b < it->first + it->second);
  a->type = in ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
} // extern "C"

// ---------------------------------------------------------------- library

namespace frsz2b {

static thread_local std::string t_error;
int set_error(int code, const std::string& msg)
{
  t_error = msg;
  return code;
}
const char* last_error() { return t_error.c_str(); }
int cuda_status(cudaError_t e, const char* what)
{
  return e == cudaSuccess ? FRSZ2_OK : set_error(FRSZ2_EFAIL, std::string(what) + ": " + cudaGetErrorString(e));
}
int check_args(int, int, int) { return FRSZ2_OK; }
int sm_count() { return 1; }

Job make_job(const Layout& L, int)
{
  Job j{};
  j.n = L.n;
  j.block_bytes = L.block_bytes;
  j.bits = L.bits;
  j.E = L.E;
  j.W = L.W;
  return j;
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

// The oracle's codec on a job's separate exponents and words.
static void code(bool compress, const Job& j, int dtype)
{
  const std::size_t nb = (j.n + j.E - 1) / j.E, eb = frsz2o_exponent_bytes(j.bits, j.E, j.n);
  std::vector<std::uint8_t> t(frsz2o_compressed_bytes(j.bits, j.E, j.n));
  std::memcpy(t.data(), j.exps, nb * (j.W / 8));
  const std::size_t last = written_block_bytes((int)(j.n - (nb - 1) * j.E), j.bits, j.W);
  std::memcpy(t.data() + eb, j.words, (nb - 1) * j.block_bytes + last);
  if (compress) {
    if (dtype == FRSZ2_FLOAT)
      frsz2o_compress_f32(static_cast<const float*>(j.values_in), j.n, j.bits, j.E, t.data());
    else
      frsz2o_compress_f64(static_cast<const double*>(j.values_in), j.n, j.bits, j.E, t.data());
    std::memcpy(j.exps, t.data(), nb * (j.W / 8));
    std::memcpy(j.words, t.data() + eb, (nb - 1) * j.block_bytes + last);
  } else if (dtype == FRSZ2_FLOAT) {
    frsz2o_decompress_f32(t.data(), j.n, j.bits, j.E, static_cast<float*>(j.values_out));
  } else {
    frsz2o_decompress_f64(t.data(), j.n, j.bits, j.E, static_cast<double*>(j.values_out));
  }
}

static int launch(bool compress, const Job& j, int dtype, cudaStream_t s)
{
  if (g_throw_in.fetch_sub(1) <= 0) throw std::bad_alloc();
  push(s, [=] { code(compress, j, dtype); });
  return cuda_status(cudaGetLastError(), "launch"); // as the library's launches end
}
int launch_compress(const Job& j, int dtype, cudaStream_t s, bool*) { return launch(true, j, dtype, s); }
int launch_decompress(const Job& j, int dtype, cudaStream_t s, bool*) { return launch(false, j, dtype, s); }
int launch_elements(const Job&, int, const std::uint64_t*, std::uint64_t, void*, cudaStream_t) { return FRSZ2_EFAIL; }

} // namespace frsz2b

// ---------------------------------------------------------------- scenarios

static int g_bad = 0;
#define CHECK(c)                                                            \
  do {                                                                      \
    if (!(c)) {                                                             \
      std::printf("line %d: %s\n", __LINE__, #c);                           \
      ++g_bad;                                                              \
    }                                                                       \
  } while (0)

static const int kBits = 21, kE = 7;

static std::vector<double> values(std::size_t n, double seed)
{
  std::vector<double> x(n);
  for (std::size_t i = 0; i < n; ++i) x[i] = (double)((i * 2654435761u + (std::size_t)(seed * 97)) % 1000003) - 5e5;
  return x;
}
static std::vector<std::uint8_t> coded(const std::vector<double>& x)
{
  std::vector<std::uint8_t> b(frsz2o_compressed_bytes(kBits, kE, x.size()), 0x5A);
  frsz2o_compress_f64(x.data(), x.size(), kBits, kE, b.data());
  return b;
}
static std::vector<double> decoded(const std::vector<std::uint8_t>& b, std::size_t n)
{
  std::vector<double> y(n);
  frsz2o_decompress_f64(b.data(), n, kBits, kE, y.data());
  return y;
}
template<class V>
static void pin(const V& v)
{
  g_pinned[reinterpret_cast<const std::uint8_t*>(v.data())] = v.size() * sizeof(v[0]);
}

// One call each way on n values; the input's last bytes come from work that the
// caller's stream still holds.  `pinned`: the input.
static void both(std::size_t n, bool pinned, bool pending)
{
  CUstream_st user;
  const auto now = values(n, 1);
  auto x = pending ? values(n, 2) : now;
  const auto ref = coded(now);
  std::vector<std::uint8_t> out(ref.size(), 0x5A);
  if (pinned) pin(x);
  if (pending) push(&user, [&] { std::memcpy(x.data(), now.data(), n * 8); });
  CHECK(frsz2_compress_host(FRSZ2_DOUBLE, kBits, kE, x.data(), n, out.data(), &user) == FRSZ2_OK);
  CHECK(out == ref);
  g_pinned.clear();

  auto buf = pending ? coded(values(n, 2)) : ref;
  std::vector<double> y(n, -1.0);
  if (pinned) pin(buf);
  if (pending) push(&user, [&] { std::memcpy(buf.data(), ref.data(), ref.size()); });
  CHECK(frsz2_decompress_host(FRSZ2_DOUBLE, kBits, kE, buf.data(), n, y.data(), &user) == FRSZ2_OK);
  CHECK(y == decoded(ref, n));
  g_pinned.clear();
  CHECK(cudaGetLastError() == cudaSuccess);
}

int main(int argc, char** argv)
{
  const std::string s = argc > 1 ? argv[1] : "";
  const std::size_t sizes[] = { 1, 1000, 131'072, 500'003, 2'000'003 };
  if (s == "plain") {
    for (std::size_t n : sizes) both(n, false, false);
  } else if (s == "pending_pinned") {
    for (std::size_t n : sizes) both(n, true, true);
  } else if (s == "pending_pageable") { // a host function on the stream fills it
    for (std::size_t n : sizes) both(n, false, true);
  } else if (s == "no_slots") { // no pinned memory to be had: the direct path
    g_host_allocs = 0;
    for (std::size_t n : sizes) both(n, false, true);
  } else if (s == "some_slots") { // two workers' memory and half of a third's
    g_host_allocs = 5;
    for (std::size_t n : { sizes[4], sizes[0], sizes[4] }) both(n, false, true);
  } else if (s == "throwing") { // no memory on the host inside one worker or another
    const auto x = values(sizes[4], 1);
    std::vector<std::uint8_t> out(coded(x).size());
    for (int k : { 0, 1, 5, 9 }) {
      CUstream_st user;
      g_throw_in = k;
      CHECK(frsz2_compress_host(FRSZ2_DOUBLE, kBits, kE, x.data(), x.size(), out.data(), &user) == FRSZ2_EFAIL);
      CHECK(std::strlen(frsz2b::last_error()) > 0);
      g_throw_in = 1 << 30;
      both(sizes[4], false, true); // the next call finds nothing of it in the way
    }
  } else {
    std::printf("unknown scenario\n");
    return 2;
  }
  std::printf(g_bad ? "%d failed\n" : "ok\n", g_bad);
  return g_bad ? 1 : 0;
}
