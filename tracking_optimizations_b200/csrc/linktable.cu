// linktable.cu -- a table of positions as the linker's frames, on the device.
//
// FrameSubsetter (linking.rs:33-61): runs of equal column-0 values are frames;
// the iterator starts with cur_frame = 0, so a first value other than 0 yields
// a leading empty frame.  Grouping, the check of the positions and the slabs
// took four passes of one host thread over the table, and its ids two more
// (2.7 of 3.5 ms for 380k rows); here they take the time of the upload.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include <cub/device/device_scan.cuh>

#include "gt.h"
#include "gt_device.cuh"
#include "traj.h"

namespace gt {

namespace {
// stat: bit pattern maxima of y and x (non-negative floats order as ints), a
// flag of positions that are not finite, the largest frame
__global__ void table_starts_kernel(const float* rows, int n, int ncols, int* starts, int* stat) {
    int ym = 0, xm = 0, bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* r = rows + (size_t)i * ncols;
        const float f = r[0], y = r[2], x = r[3];
        starts[i] = i == 0 ? f != 0.f : f != r[-ncols];
        bad |= !isfinite(y) || !isfinite(x);
        ym = max(ym, __float_as_int(fmaxf(y, 0.f)));
        xm = max(xm, __float_as_int(fmaxf(x, 0.f)));
    }
    ym = __reduce_max_sync(0xffffffffu, ym);
    xm = __reduce_max_sync(0xffffffffu, xm);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(stat, ym);
        atomicMax(stat + 1, xm);
        if (bad) atomicOr(stat + 2, 1);
    }
}

// frame[i] (inclusive sum of the starts) is row i's frame; off[t] = first row
// of frame t
__global__ void table_offsets_kernel(const int* starts, const int* frame, int n, int* off) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i == 0) off[0] = 0;
        if (starts[i]) off[frame[i]] = i;
        if (i == n - 1) off[frame[i] + 1] = n;
    }
}

__global__ void table_largest_kernel(const int* off, int T, int* stat) {
    int m = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) m = max(m, off[t + 1] - off[t]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(stat + 3, m);
}

// The same of a small table by one block: its launches and waits cost more than
// the rows (20 frames of 50: 187 us a call in five launches and two waits, 161 in one).
constexpr int TINY = 8192, TINY_NT = 1024;

__global__ void __launch_bounds__(TINY_NT) table_tiny_kernel(const float* rows, int n, int ncols, int* frame, int* off,
                                                             int* stat) {
    __shared__ int warp_tot[TINY_NT / 32], s_total, s_stat[4];
    if (threadIdx.x < 4) s_stat[threadIdx.x] = 0;
    if (threadIdx.x == 0) off[0] = 0;
    __syncthreads();
    int ym = 0, xm = 0, bad = 0, before = 0;
    for (int i0 = 0; i0 < n; i0 += TINY_NT) {
        const int i = i0 + threadIdx.x;
        int start = 0;
        if (i < n) {
            const float* r = rows + (size_t)i * ncols;
            const float f = r[0], y = r[2], x = r[3];
            start = i == 0 ? f != 0.f : f != r[-ncols];
            bad |= !isfinite(y) || !isfinite(x);
            ym = max(ym, __float_as_int(fmaxf(y, 0.f)));
            xm = max(xm, __float_as_int(fmaxf(x, 0.f)));
        }
        const int t = before + block_excl_scan<TINY_NT>(start, warp_tot, &s_total) + start;
        if (i < n) frame[i] = t;
        if (start) off[t] = i;
        before += s_total;
        __syncthreads();
    }
    const int T = before + 1;
    if (threadIdx.x == 0) off[T] = n;
    __syncthreads();
    int m = 0;
    for (int t = threadIdx.x; t < T; t += TINY_NT) m = max(m, off[t + 1] - off[t]);
    atomicMax(s_stat, ym);
    atomicMax(s_stat + 1, xm);
    if (bad) atomicOr(s_stat + 2, 1);
    atomicMax(s_stat + 3, m);
    __syncthreads();
    if (threadIdx.x < 4) stat[threadIdx.x] = s_stat[threadIdx.x];
    if (threadIdx.x == 0) stat[4] = T;
}

__global__ void table_slabs_kernel(const float* rows, const int* frame, const int* off, int n, int ncols, int T, int cap,
                                   float* py, float* px, int* npart) {
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int i = i0; i < n; i += step) {
        const int t = frame[i];
        const size_t s = (size_t)t * cap + (i - off[t]);
        py[s] = rows[(size_t)i * ncols + 2];
        px[s] = rows[(size_t)i * ncols + 3];
    }
    for (int t = i0; t < T; t += step) npart[t] = off[t + 1] - off[t];
}

__global__ void table_ids_kernel(const int* root, const int* newid, int n, unsigned long long* ids) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        ids[i] = (unsigned long long)(long long)newid[root[i]];
}

int blocks_for(int n, int num_sms) { return std::max(1, std::min((n + 255) / 256, num_sms * 8)); }
}  // namespace

// The table on the device with its frames; M keeps it until the next call.
int table_load(const float* h_rows, int n, int ncols, TrajMem& M, cudaStream_t st, int num_sms, LinkTable* t,
               std::string* msg) {
#define LK(x)                              \
    do {                                   \
        cudaError_t e_ = (x);              \
        if (e_ != cudaSuccess) {           \
            *msg = cudaGetErrorString(e_); \
            return GT_ERR_CUDA;            \
        }                                  \
    } while (0)
    LK(M.begin());
    float* rows = M.get<float>((size_t)n * ncols);
    int* starts = M.get<int>(n);
    t->frame = M.get<int>(n);
    t->off = M.get<int>((size_t)n + 2);
    int* stat = M.get<int>(5);
    size_t tmp = 0;
    LK(cub::DeviceScan::InclusiveSum(nullptr, tmp, starts, t->frame, n, st));
    void* w = M.get<char>(tmp);
    t->ids = M.get<unsigned long long>(n);
    if (!rows || !starts || !t->frame || !t->off || !stat || !w || !t->ids) {
        *msg = "device allocation failed";
        return GT_ERR_OOM;
    }
    t->rows = rows;
    t->n = n;
    t->ncols = ncols;
    const int nb = blocks_for(n, num_sms);
    LK(M.hc->upload(rows, h_rows, sizeof(float) * (size_t)n * ncols, st));
    int words[5];
    int* h = M.hc->staged(words);
    if (n <= TINY) {
        table_tiny_kernel<<<1, TINY_NT, 0, st>>>(rows, n, ncols, t->frame, t->off, stat);
        LK(cudaGetLastError());
        LK(cudaMemcpyAsync(h, stat, sizeof(words), cudaMemcpyDeviceToHost, st));
        LK(cudaStreamSynchronize(st));
        t->T = h[4];
    } else {
        LK(cudaMemsetAsync(stat, 0, 4 * sizeof(int), st));
        table_starts_kernel<<<nb, 256, 0, st>>>(rows, n, ncols, starts, stat);
        LK(cudaGetLastError());
        LK(cub::DeviceScan::InclusiveSum(w, tmp, starts, t->frame, n, st));
        table_offsets_kernel<<<nb, 256, 0, st>>>(starts, t->frame, n, t->off);
        LK(cudaGetLastError());
        LK(cudaMemcpyAsync(h, t->frame + n - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        LK(cudaStreamSynchronize(st));
        t->T = h[0] + 1;
        table_largest_kernel<<<blocks_for(t->T, num_sms), 256, 0, st>>>(t->off, t->T, stat);
        LK(cudaGetLastError());
        LK(cudaMemcpyAsync(h, stat, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
        LK(cudaStreamSynchronize(st));
    }
    if (h[2]) {
        *msg = "non-finite position";
        return GT_ERR_ARG;
    }
    union { int i; float f; } u;
    u.i = h[0];
    t->ymax = u.f;
    u.i = h[1];
    t->xmax = u.f;
    t->largest = std::max(1, h[3]);
    return GT_OK;
}

cudaError_t table_slabs(const LinkTable& t, int cap, float* py, float* px, int* npart, int num_sms, cudaStream_t st) {
    table_slabs_kernel<<<blocks_for(t.n, num_sms), 256, 0, st>>>(t.rows, t.frame, t.off, t.n, t.ncols, t.T, cap, py, px,
                                                               npart);
    return cudaGetLastError();
}

cudaError_t table_ids(const LinkTable& t, const int* root, const int* newid, int num_sms, cudaStream_t st) {
    table_ids_kernel<<<blocks_for(t.n, num_sms), 256, 0, st>>>(root, newid, t.n, t.ids);
    return cudaGetLastError();
}

}  // namespace gt
