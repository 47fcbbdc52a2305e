// hbx_stage.cpp -- see hbx_stage.h.
#include "hbx_stage.h"

#include <omp.h>

#include <algorithm>
#include <cstring>
#include <memory>

namespace hbx {
namespace {

// Page-locking costs 0.7 ms a MB and up, thirty times as long as the transfer,
// so the buffers are small; 2 MB still amortises a transfer's fixed cost (1.2 GB
// from pageable memory: 112-124 ms in one plain copy, 30 ms through the
// buffers).  Images under 32 MB take the plain copy, which is over sooner than
// the page-locking.
constexpr uint64_t kBufWords = 1u << 18;
constexpr uint64_t kDirect = 1u << 22;
constexpr uint64_t kThreadWords = 1u << 14;  // a thread is worth waking for 128 KB

// Moves image words [w0, w1) between the pieces and buf (word w0 at buf[0]).
template <bool kToBuf>
void move_words(const std::vector<HostPiece> &pieces, uint64_t w0, uint64_t w1, double *buf) {
  const int nt = (int)std::min<uint64_t>((uint64_t)omp_get_max_threads(), 1 + (w1 - w0) / kThreadWords);
#pragma omp parallel for schedule(static, 1) num_threads(nt)
  for (int t = 0; t < nt; ++t) {
    uint64_t a = w0 + (w1 - w0) * (uint64_t)t / (uint64_t)nt;
    const uint64_t b = w0 + (w1 - w0) * (uint64_t)(t + 1) / (uint64_t)nt;
    if (a >= b) continue;
    // the piece that holds word a
    auto it = std::upper_bound(pieces.begin(), pieces.end(), a,
                               [](uint64_t w, const HostPiece &p) { return w < p.at; });
    --it;
    for (; a < b; ++it) {
      const uint64_t o = a - it->at, n = std::min(b - a, it->words - o);
      if (kToBuf) std::memcpy(buf + (a - w0), it->host + o, n * sizeof(double));
      else std::memcpy(it->host + o, buf + (a - w0), n * sizeof(double));
      a += n;
    }
  }
}

// First touch of the destination by every core, each its own part: a plain copy
// into untouched pages runs at a tenth of the speed, and the pages of one
// buffer, touched by the copy itself, are a single 2 MB page that one core
// zeroes (1.2 GB: 150 ms that way, 45 ms touched first).
void touch_pages(double *host, uint64_t words) {
  const int nt = (int)std::min<uint64_t>((uint64_t)omp_get_max_threads(), 1 + words / kThreadWords);
#pragma omp parallel for schedule(static) num_threads(nt)
  for (long long i = 0; i < (long long)words; i += 512) host[i] = 0.0;
}

}  // namespace

bool Stager::open() {
  cudaError_t e = cudaSuccess;
  if (!s_) e = cudaStreamCreate(&s_);  // a blocking stream: after the default stream's work
  for (int k = 0; k < 2; ++k) {
    if (e == cudaSuccess && !buf_[k])
      e = cudaHostAlloc(reinterpret_cast<void **>(&buf_[k]), kBufWords * sizeof(double), cudaHostAllocDefault);
    if (e == cudaSuccess && !done_[k]) e = cudaEventCreateWithFlags(&done_[k], cudaEventDisableTiming);
  }
  if (e != cudaSuccess) cudaGetLastError();  // the plain copies do without: no error is left for the next launch
  return e == cudaSuccess;
}

Stager::~Stager() {
  if (s_) cudaStreamSynchronize(s_);
  for (int k = 0; k < 2; ++k) {
    if (done_[k]) cudaEventDestroy(done_[k]);
    if (buf_[k]) cudaFreeHost(buf_[k]);
  }
  if (s_) cudaStreamDestroy(s_);
}

cudaError_t Stager::to_device(const std::vector<HostPiece> &pieces, uint64_t total, double *dev) {
  if (total == 0) return cudaSuccess;
  if (total < kDirect) {
    if (pieces.size() == 1) return cudaMemcpy(dev, pieces[0].host, total * sizeof(double), cudaMemcpyHostToDevice);
    const std::unique_ptr<double[]> one(new double[total]);
    move_words<true>(pieces, 0, total, one.get());
    return cudaMemcpy(dev, one.get(), total * sizeof(double), cudaMemcpyHostToDevice);
  }
  cudaError_t e = cudaSuccess;
  if (!open()) {
    for (const HostPiece &p : pieces)
      if (e == cudaSuccess) e = cudaMemcpy(dev + p.at, p.host, p.words * sizeof(double), cudaMemcpyHostToDevice);
    return e;
  }
  int k = 0;
  for (uint64_t w = 0; w < total && e == cudaSuccess; w += kBufWords, ++k) {
    const uint64_t n = std::min(kBufWords, total - w);
    if (k >= 2) e = cudaEventSynchronize(done_[k & 1]);
    if (e != cudaSuccess) break;
    move_words<true>(pieces, w, w + n, buf_[k & 1]);
    e = cudaMemcpyAsync(dev + w, buf_[k & 1], n * sizeof(double), cudaMemcpyHostToDevice, s_);
    if (e == cudaSuccess) e = cudaEventRecord(done_[k & 1], s_);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s_);
  return e;
}

cudaError_t Stager::to_host(const std::vector<HostPiece> &pieces, uint64_t total, const double *dev) {
  if (total == 0) return cudaSuccess;
  if (total < kDirect && pieces.size() == 1) {
    touch_pages(pieces[0].host, total);
    return cudaMemcpy(pieces[0].host, dev, total * sizeof(double), cudaMemcpyDeviceToHost);
  }
  cudaError_t e = cudaSuccess;
  for (const HostPiece &p : pieces) touch_pages(p.host, p.words);
  if (!open()) {
    for (const HostPiece &p : pieces)
      if (e == cudaSuccess) e = cudaMemcpy(p.host, dev + p.at, p.words * sizeof(double), cudaMemcpyDeviceToHost);
    return e;
  }
  const uint64_t nbuf = (total + kBufWords - 1) / kBufWords;
  for (uint64_t k = 0; k <= nbuf && e == cudaSuccess; ++k) {
    if (k < nbuf) {  // the transfer of buffer k runs while buffer k - 1 is spread
      const uint64_t w = k * kBufWords, n = std::min(kBufWords, total - w);
      e = cudaMemcpyAsync(buf_[k & 1], dev + w, n * sizeof(double), cudaMemcpyDeviceToHost, s_);
      if (e == cudaSuccess) e = cudaEventRecord(done_[k & 1], s_);
    }
    if (k > 0 && e == cudaSuccess) {
      e = cudaEventSynchronize(done_[(k - 1) & 1]);
      const uint64_t w = (k - 1) * kBufWords;
      if (e == cudaSuccess) move_words<false>(pieces, w, std::min(total, w + kBufWords), buf_[(k - 1) & 1]);
    }
  }
  return e;
}

}  // namespace hbx
