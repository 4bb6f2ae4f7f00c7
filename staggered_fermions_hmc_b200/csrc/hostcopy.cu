// hostcopy.cu — see hostcopy.h.
#include "hostcopy.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

namespace sfh {

namespace {

bool pageable(const void* host)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// a stream under capture keeps the driver's copy and its error
bool capturing(cudaStream_t stream)
{
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

}  // namespace

HostCopy::~HostCopy() { release(); }

void HostCopy::release()
{
    if (own_) cudaStreamSynchronize(own_);
    for (int k = 0; k < kMaxThreads; ++k) {
        if (ev_[k]) cudaEventDestroy(ev_[k]);
        if (pinned_[k]) cudaFreeHost(pinned_[k]);
        ev_[k] = nullptr;
        pinned_[k] = nullptr;
    }
    if (order_) cudaEventDestroy(order_);
    if (own_) cudaStreamDestroy(own_);
    order_ = nullptr;
    own_ = nullptr;
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

// The copy in the order of the caller's stream.  cudaStreamPerThread names
// another stream in each of the threads: its pieces take a stream of the
// object's own, after what the caller's holds and before what comes to it next.
template <bool IN>
cudaError_t HostCopy::pieces(char* dev, char* host, size_t bytes, int device, cudaStream_t stream)
{
    if (stream != cudaStreamPerThread) return move<IN>(dev, host, bytes, device, stream);
    cudaError_t e;
    if (!own_ && (e = cudaStreamCreateWithFlags(&own_, cudaStreamNonBlocking)) != cudaSuccess) return e;
    if (!order_ && (e = cudaEventCreateWithFlags(&order_, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(order_, stream)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(own_, order_, 0)) != cudaSuccess) return e;
    if ((e = move<IN>(dev, host, bytes, device, own_)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(order_, own_)) != cudaSuccess) return e;
    return cudaStreamWaitEvent(stream, order_, 0);
}

// Each thread takes pieces from a counter and moves them through its own
// buffer; the calling thread is one of them, so that the copy completes
// however many others could be started.
template <bool IN>
cudaError_t HostCopy::move(char* dev, char* host, size_t bytes, int device, cudaStream_t stream)
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
    if (bytes >= CopyCredit::kLeast && pageable(host) && !capturing(stream) && credit_.enough(bytes, true) && ready())
        return pieces<true>((char*)dev, (char*)const_cast<void*>(host), bytes, device, stream);
    return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, stream);
}

cudaError_t HostCopy::out(void* host, const void* dev, size_t bytes, int device, cudaStream_t stream)
{
    if (bytes >= CopyCredit::kLeast && pageable(host) && !capturing(stream) && credit_.enough(bytes, false) && ready())
        return pieces<false>((char*)const_cast<void*>(dev), (char*)host, bytes, device, stream);
    return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, stream);
}

}  // namespace sfh
