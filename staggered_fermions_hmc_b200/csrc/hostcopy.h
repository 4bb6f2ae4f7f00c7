// hostcopy.h — copies between the device and pageable host memory.
//
// The CUDA driver moves pageable memory through its own pinned buffer with one host
// thread, which also takes the page faults of a freshly allocated result.  A
// large copy is therefore cut into pieces that several threads move through
// pinned buffers of the context, one each, while the pieces' transfers queue on
// the context's stream.  With eight threads, ms: a spinor of 32^3 64 (101 MB) to
// a new array 22 -> 8, its links (1.2 GB) 250 -> 68, and back 108 -> 32; the
// operator on a spinor of 38 MB, both ways, 10.0 -> 4.5.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace sfh {

// Which copies take the pieces.  The first one makes the buffers, 12 to 20 ms
// with their release; a piecewise copy saves about 55 us a MB on the way in and,
// the result being a new array as a rule, three times that on the way out.  So
// the driver copies until what the pieces would have saved has come to that:
// the first upload of 36 MB takes 3.5 ms (17 with the buffers made for it), of
// 190 MB 17 (23), of 1.2 GB 48 through pieces at once (110 by the driver).
class CopyCredit {
  public:
    bool enough(size_t bytes, bool in)
    {
        if (bytes < kLeast) return false;
        if (credit_ < kSetUp) credit_ += in ? bytes : 3 * bytes;
        return credit_ >= kSetUp;
    }

    // below, CUDA's own copy takes less than 8 ms, and the threads cost more
    static constexpr size_t kLeast = (size_t)32 << 20;

  private:
    static constexpr size_t kSetUp = (size_t)256 << 20;
    size_t credit_ = 0;
};

class HostCopy {
  public:
    HostCopy() = default;
    HostCopy(const HostCopy&) = delete;
    HostCopy& operator=(const HostCopy&) = delete;
    ~HostCopy();

    // Host to device, in the stream's order; the host memory may be reused on
    // return, as with cudaMemcpyAsync from pageable memory.
    cudaError_t in(void* dev, const void* host, size_t bytes, int device, cudaStream_t stream);
    // Device to host, in the stream's order; complete on return or, for
    // pinned memory, once the stream is.
    cudaError_t out(void* host, const void* dev, size_t bytes, int device, cudaStream_t stream);

  private:
    static constexpr int kMaxThreads = 8;
    static constexpr size_t kPiece = (size_t)2 << 20;

    bool ready();
    void release();
    template <bool IN>
    cudaError_t pieces(char* dev, char* host, size_t bytes, int device, cudaStream_t stream);
    template <bool IN>
    cudaError_t move(char* dev, char* host, size_t bytes, int device, cudaStream_t stream);

    CopyCredit credit_;
    int threads_ = 0;  // 0: not set up; < 0: could not be
    char* pinned_[kMaxThreads] = {};
    cudaEvent_t ev_[kMaxThreads] = {};  // the last transfer of each buffer
    cudaStream_t own_ = nullptr;        // the pieces' stream for cudaStreamPerThread
    cudaEvent_t order_ = nullptr;       // orders it against the caller's
};

}  // namespace sfh
