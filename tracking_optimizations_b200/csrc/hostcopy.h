// hostcopy.h -- copies between pageable host arrays and the device through
// page-locked slots that several threads fill or empty.
//
// The driver stages a pageable copy through its own buffer with one thread:
// 12 GB/s for the frames of a movie, 3 to 6 GB/s into freshly allocated result
// arrays.  Eight threads and a ring of slots keep the next slot's memcpy behind
// the current slot's transfer.  Arrays that are already page-locked are copied
// directly.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

namespace gt {

// memcpy split over worker threads; started by the first large copy, one
// caller at a time.
class CopyPool {
  public:
    ~CopyPool();
    void copy(void* dst, const void* src, size_t bytes, bool to_device);

  private:
    void start();
    void work(unsigned part);
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable go_, done_;
    unsigned long long job_ = 0;
    unsigned left_ = 0;
    bool stop_ = false;
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t bytes_ = 0;
    bool to_device_ = false;
};

// Owned by one context and used by one call at a time, as the context is.
class HostCopy {
  public:
    ~HostCopy();
    // src (host, valid until the call returns) to the device on st.
    cudaError_t upload(void* dst, const void* src, size_t bytes, cudaStream_t st);
    // The device to dst (host); dst holds the data when the call returns.
    cudaError_t download(void* dst, const void* src, size_t bytes, cudaStream_t st);
    // Page-locked words for results that the call waits for at once: copies into
    // pageable memory wait one by one.  `words` where there are none.
    template <class X>
    X* staged(X* words) {
        if (!small_ && cudaHostAlloc((void**)&small_, SMALL, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            small_ = nullptr;
        }
        return small_ ? (X*)small_ : words;
    }

  private:
    static constexpr int SLOTS = 4;
    static constexpr size_t SLOT = (size_t)8 << 20;
    static constexpr size_t SMALL = (size_t)64 << 10;  // below: uploads by the driver's own staging, downloads by small_
    cudaError_t ready();
    CopyPool pool_;
    char* slot_[SLOTS] = {};
    char* small_ = nullptr;
    cudaEvent_t ev_[SLOTS] = {};
    int next_ = 0;
};

}  // namespace gt
