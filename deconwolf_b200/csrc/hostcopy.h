// hostcopy.h -- copies between pageable host memory and the device (hostcopy.cu).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <thread>
#include <vector>

namespace dwcu {

// `rows` rows of row_bytes, compact on the host, dpitch apart on the device.
// From pageable memory the host buffer has been read when this returns; the
// device sees the data in stream order.
cudaError_t copy_to_device(void *dev, size_t dpitch, const void *host, size_t row_bytes, size_t rows,
                           cudaStream_t st, int device);
// In stream order; the host buffer is complete once the stream has drained.
cudaError_t copy_to_host(void *host, const void *dev, size_t bytes, cudaStream_t st, int device);
// gives the page-locked buffers back
void copy_release();

// Touches (zeroes) a pageable result buffer on a few threads while the device
// works, so that the result's copy does not wait for its pages.
class Prefault {
  public:
    void start(void *p, size_t bytes);
    void join();
    ~Prefault() { join(); }

  private:
    std::vector<std::thread> th_;
    std::atomic<size_t> next_{0};
};

}  // namespace dwcu
