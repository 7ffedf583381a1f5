// traj.h -- device scratch of the calls on host tables, kept by the context.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>
#include <vector>

#include "hostcopy.h"

namespace gt {

// Scratch handed out piece by piece and taken back as a whole by the next
// call's begin() (every call ends with its stream synchronised).  What a call
// needed is one block for the next call, up to KEEP bytes; end() gives more
// than that back to the device.
struct TrajMem {
    static constexpr size_t KEEP = (size_t)1 << 30;  // tables of 10 million rows; beyond, a call takes far longer than
                                                     // the allocations
    HostCopy* hc = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};

    cudaError_t begin() {
        for (auto& e : ev)
            if (!e) {
                const cudaError_t r = cudaEventCreate(&e);
                if (r != cudaSuccess) return r;
            }
        if (blocks_.size() > 1) {
            size_t sum = 0;
            for (auto& b : blocks_) sum += b.size;
            release();
            add(sum);  // a failure shows at the first get()
        }
        used_ = 0;
        return cudaSuccess;
    }

    template <class X>
    X* get(size_t n) {
        const size_t bytes = (sizeof(X) * std::max<size_t>(n, 1) + 255) / 256 * 256;
        if (blocks_.empty() || used_ + bytes > blocks_.back().size) {
            if (!add(std::max(bytes, (size_t)16 << 20))) return nullptr;
            used_ = 0;
        }
        char* p = blocks_.back().p + used_;
        used_ += bytes;
        return (X*)p;
    }

    // After a call, whose stream is synchronised.
    void end() {
        size_t sum = 0;
        for (auto& b : blocks_) sum += b.size;
        if (sum > KEEP) release();
    }

    void release() {
        for (auto& b : blocks_) cudaFree(b.p);
        blocks_.clear();
        used_ = 0;
    }

    ~TrajMem() {
        release();
        for (auto& e : ev)
            if (e) cudaEventDestroy(e);
    }

  private:
    struct Block {
        char* p;
        size_t size;
    };
    bool add(size_t bytes) {
        void* q = nullptr;
        if (cudaMalloc(&q, bytes) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        blocks_.push_back({(char*)q, bytes});
        return true;
    }
    std::vector<Block> blocks_;
    size_t used_ = 0;
};

// Ends a call on the scratch when it leaves its scope, after an error too.
struct TrajEnd {
    TrajMem& m;
    ~TrajEnd() { m.end(); }
};

// A position table on the device and its frames (linktable.cu).
struct LinkTable {
    const float* rows = nullptr;
    int n = 0, ncols = 0, T = 0;
    int* frame = nullptr;  // per row
    int* off = nullptr;    // first row of each frame; off[T] = n
    int largest = 1;       // rows of the largest frame
    float ymax = 0.f, xmax = 0.f;  // at least 0
    unsigned long long* ids = nullptr;
};

}  // namespace gt
