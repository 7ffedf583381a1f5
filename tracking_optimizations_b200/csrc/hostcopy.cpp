// hostcopy.cpp -- see hostcopy.h.
#include "hostcopy.h"

#include <algorithm>
#include <cstring>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace gt {

namespace {
constexpr size_t PART_MIN = (size_t)128 << 10;  // bytes per thread that pay for waking it

bool page_locked(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}
}  // namespace

CopyPool::~CopyPool() {
    {
        std::lock_guard<std::mutex> g(m_);
        stop_ = true;
    }
    go_.notify_all();
    for (auto& t : threads_) t.join();
}

void CopyPool::start() {
    const unsigned n = std::max(2u, std::min(8u, std::thread::hardware_concurrency())) - 1;
    try {
        for (unsigned i = 0; i < n; ++i) threads_.emplace_back([this, i] { work(i + 1); });
    } catch (...) {
        // fewer threads (or none): the caller copies the rest
    }
}

// memcpy for data that the device reads next: stores past the caches.  A
// transfer that finds its lines dirty in eight cores' caches ran at 7 GB/s.
static void stream_copy(char* d, const char* s, size_t n) {
#ifdef __SSE2__
    const size_t head = std::min(n, (size_t)(-(intptr_t)d & 63));
    std::memcpy(d, s, head);
    d += head; s += head; n -= head;
    for (; n >= 64; n -= 64, d += 64, s += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i*)s), b = _mm_loadu_si128((const __m128i*)(s + 16));
        const __m128i c = _mm_loadu_si128((const __m128i*)(s + 32)), e = _mm_loadu_si128((const __m128i*)(s + 48));
        _mm_stream_si128((__m128i*)d, a);
        _mm_stream_si128((__m128i*)(d + 16), b);
        _mm_stream_si128((__m128i*)(d + 32), c);
        _mm_stream_si128((__m128i*)(d + 48), e);
    }
    std::memcpy(d, s, n);
    _mm_sfence();
#else
    std::memcpy(d, s, n);
#endif
}

// Worker `part` copies its share of every job.
void CopyPool::work(unsigned part) {
    unsigned long long seen = 0;
    std::unique_lock<std::mutex> lk(m_);
    while (true) {
        go_.wait(lk, [&] { return stop_ || job_ != seen; });
        if (stop_) return;
        seen = job_;
        const size_t parts = threads_.size() + 1, step = (bytes_ / parts + 63) / 64 * 64;
        const size_t b0 = std::min(bytes_, step * part), b1 = part + 1 == parts ? bytes_ : std::min(bytes_, step * (part + 1));
        char* d = dst_;
        const char* s = src_;
        lk.unlock();
        if (b1 > b0) (to_device_ ? stream_copy(d + b0, s + b0, b1 - b0) : (void)std::memcpy(d + b0, s + b0, b1 - b0));
        lk.lock();
        if (--left_ == 0) done_.notify_one();
    }
}

void CopyPool::copy(void* dst, const void* src, size_t bytes, bool to_device) {
    const auto own = [&](size_t n) { to_device ? stream_copy((char*)dst, (const char*)src, n) : (void)std::memcpy(dst, src, n); };
    if (bytes < 2 * PART_MIN) {
        own(bytes);
        return;
    }
    if (threads_.empty()) start();
    if (threads_.empty()) {
        own(bytes);
        return;
    }
    size_t mine;
    {
        std::lock_guard<std::mutex> g(m_);
        dst_ = (char*)dst;
        src_ = (const char*)src;
        bytes_ = bytes;
        to_device_ = to_device;
        left_ = (unsigned)threads_.size();
        ++job_;
        mine = std::min(bytes, (bytes / (threads_.size() + 1) + 63) / 64 * 64);
    }
    go_.notify_all();
    own(mine);
    std::unique_lock<std::mutex> lk(m_);
    done_.wait(lk, [&] { return left_ == 0; });
}

HostCopy::~HostCopy() {
    for (auto& e : ev_)
        if (e) cudaEventDestroy(e);
    for (auto& s : slot_)
        if (s) cudaFreeHost(s);
    if (small_) cudaFreeHost(small_);
}

cudaError_t HostCopy::ready() {
    for (int i = 0; i < SLOTS; ++i) {
        if (!slot_[i]) {
            const cudaError_t e = cudaHostAlloc((void**)&slot_[i], SLOT, cudaHostAllocDefault);
            if (e != cudaSuccess) {
                slot_[i] = nullptr;
                return e;
            }
        }
        if (!ev_[i]) {
            const cudaError_t e = cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming);
            if (e != cudaSuccess) {
                ev_[i] = nullptr;
                return e;
            }
        }
    }
    return cudaSuccess;
}

cudaError_t HostCopy::upload(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes < SMALL || page_locked(src) || ready() != cudaSuccess) {
        cudaGetLastError();
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    }
    for (size_t at = 0; at < bytes; at += SLOT) {
        const size_t n = std::min(SLOT, bytes - at);
        const int s = next_;
        next_ = (next_ + 1) % SLOTS;
        cudaError_t e = cudaEventSynchronize(ev_[s]);  // the slot's last transfer, on whatever stream
        if (e != cudaSuccess) return e;
        pool_.copy(slot_[s], (const char*)src + at, n, true);
        e = cudaMemcpyAsync((char*)dst + at, slot_[s], n, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[s], st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t HostCopy::download(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes < SMALL) {
        char* w = staged((char*)dst);
        cudaError_t e = cudaMemcpyAsync(w, src, bytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && w != dst) std::memcpy(dst, w, bytes);
        return e;
    }
    if (page_locked(dst) || ready() != cudaSuccess) {
        cudaGetLastError();
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return e != cudaSuccess ? e : cudaStreamSynchronize(st);
    }
    // SLOTS transfers in flight; slot i of the ring holds bytes [SLOT i, ...)
    const size_t parts = (bytes + SLOT - 1) / SLOT;
    const int first = next_;
    auto start = [&](size_t i) {
        const int s = (int)((first + i) % SLOTS);
        cudaError_t e = cudaEventSynchronize(ev_[s]);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(slot_[s], (const char*)src + i * SLOT, std::min(SLOT, bytes - i * SLOT),
                            cudaMemcpyDeviceToHost, st);
        return e != cudaSuccess ? e : cudaEventRecord(ev_[s], st);
    };
    size_t started = 0;
    for (size_t i = 0; i < parts; ++i) {
        for (; started < parts && started < i + SLOTS; ++started) {
            const cudaError_t e = start(started);
            if (e != cudaSuccess) return e;
        }
        const int s = (int)((first + i) % SLOTS);
        const cudaError_t e = cudaEventSynchronize(ev_[s]);
        if (e != cudaSuccess) return e;
        pool_.copy((char*)dst + i * SLOT, slot_[s], std::min(SLOT, bytes - i * SLOT), false);
    }
    next_ = (int)((first + parts) % SLOTS);
    return cudaSuccess;
}

}  // namespace gt
