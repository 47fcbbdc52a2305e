// hbx_stage.h -- copies of many pieces of pageable host memory to and from
// the device through two page-locked buffers.
//
// A plain copy of pageable memory runs on one host thread; here every host
// core moves one buffer's worth between the pieces and the page-locked buffer
// while the DMA engine moves the other buffer.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

namespace hbx {

// `words` doubles of host memory that start at word `at` of the device image.
struct HostPiece {
  double *host;
  uint64_t at, words;
};

// Copies between a device image (total words) and host pieces, sorted by `at`
// and tiling the image, ordered after the work on the device's default stream;
// both return once the host side and the device side are complete (a plain copy
// to the device: for work on the default stream).  The page-locked buffers are
// taken by the first large copy and given back with the object.
class Stager {
 public:
  Stager() = default;
  Stager(const Stager &) = delete;
  Stager &operator=(const Stager &) = delete;
  ~Stager();
  cudaError_t to_device(const std::vector<HostPiece> &pieces, uint64_t total, double *dev);
  cudaError_t to_host(const std::vector<HostPiece> &pieces, uint64_t total, const double *dev);

 private:
  bool open();  // false where the system refuses the buffers: plain copies then
  double *buf_[2] = {nullptr, nullptr};
  cudaEvent_t done_[2] = {nullptr, nullptr};
  cudaStream_t s_ = nullptr;
};

}  // namespace hbx
