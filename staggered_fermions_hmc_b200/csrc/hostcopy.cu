// hostcopy.cu — see hostcopy.h.
#include "hostcopy.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

namespace sfh {

namespace {

// From here on the first copy repays the buffers (16 MB) and every copy its
// threads; below, CUDA's own copy takes less than 8 ms.
constexpr size_t kLeastBytes = (size_t)32 << 20;

bool pageable(const void* host)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

HostCopy::~HostCopy() { release(); }

void HostCopy::release()
{
    for (int k = 0; k < kMaxThreads; ++k) {
        if (ev_[k]) cudaEventDestroy(ev_[k]);
        if (pinned_[k]) cudaFreeHost(pinned_[k]);
        ev_[k] = nullptr;
        pinned_[k] = nullptr;
    }
}

bool HostCopy::ready()
{
    if (threads_ != 0) return threads_ > 0;
    threads_ = -1;
    const int n = std::min((int)kMaxThreads, (int)std::thread::hardware_concurrency() / 2);
    if (n < 2) return false;
    for (int k = 0; k < n; ++k)
        if (cudaHostAlloc((void**)&pinned_[k], kPiece, cudaHostAllocDefault) != cudaSuccess ||
            cudaEventCreateWithFlags(&ev_[k], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            release();
            return false;
        }
    threads_ = n;
    return true;
}

// Each thread takes pieces from a counter and moves them through its own
// buffer; the calling thread is one of them, so that the copy completes
// however many others could be started.
template <bool IN>
cudaError_t HostCopy::pieces(char* dev, char* host, size_t bytes, int device, cudaStream_t stream)
{
    std::atomic<size_t> next{0};
    cudaError_t err[kMaxThreads] = {};
    auto work = [&](int t) {
        cudaError_t e = cudaSetDevice(device);
        while (e == cudaSuccess) {
            const size_t at = next.fetch_add(kPiece);
            if (at >= bytes) break;
            const size_t n = std::min(kPiece, bytes - at);
            if (IN) {
                if ((e = cudaEventSynchronize(ev_[t])) != cudaSuccess) break;  // the buffer's last transfer
                std::memcpy(pinned_[t], host + at, n);
                e = cudaMemcpyAsync(dev + at, pinned_[t], n, cudaMemcpyHostToDevice, stream);
                if (e == cudaSuccess) e = cudaEventRecord(ev_[t], stream);
            } else {
                e = cudaMemcpyAsync(pinned_[t], dev + at, n, cudaMemcpyDeviceToHost, stream);
                if (e == cudaSuccess) e = cudaEventRecord(ev_[t], stream);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev_[t]);
                if (e == cudaSuccess) std::memcpy(host + at, pinned_[t], n);
            }
        }
        err[t] = e;
    };
    std::thread others[kMaxThreads];
    for (int t = 1; t < threads_; ++t) {
        try {
            others[t] = std::thread(work, t);
        } catch (...) {  // no more threads to be had
            break;
        }
    }
    work(0);
    for (std::thread& o : others)
        if (o.joinable()) o.join();
    for (cudaError_t e : err)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t HostCopy::in(void* dev, const void* host, size_t bytes, int device, cudaStream_t stream)
{
    if (bytes >= kLeastBytes && pageable(host) && ready())
        return pieces<true>((char*)dev, (char*)const_cast<void*>(host), bytes, device, stream);
    return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, stream);
}

cudaError_t HostCopy::out(void* host, const void* dev, size_t bytes, int device, cudaStream_t stream)
{
    if (bytes >= kLeastBytes && pageable(host) && ready())
        return pieces<false>((char*)const_cast<void*>(dev), (char*)host, bytes, device, stream);
    return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, stream);
}

}  // namespace sfh
