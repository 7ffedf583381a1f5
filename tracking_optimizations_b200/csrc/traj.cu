// traj.cu -- trajectory post-processing of a linked table on the device:
// the lab pipeline's steps after linking (all_cleaned_up/
// hatzakis_lab_tracking.py:216-230): trackpy.filter_stubs, step_tracker
// (hatzakis_lab_tracking.py:53-83) and the per-particle mean squared
// displacement of trackpy.msd, concatenated as mp_imsd does
// (hatzakis_lab_tracking.py:199-214).
//
// Rows are grouped by particle with a stable order: keys (particle - min id)
// << 32 | row, in row order, are radix-sorted by their particle bits (a stable
// sort keeps the rows in order), which gives exactly pandas' groupby order
// (ascending particle, rows of a particle in table order).
//
// Scratch comes from the context's TrajMem, which keeps its memory: stream-
// ordered allocations, whose pool gives everything back at each
// synchronisation, took 5 of 8 ms of the three calls on a 360k-row table.
//
// MSD of one particle (trackpy.msd's definition): positions p = xy * mpp in
// float32, placed on the frame axis from the particle's first to its last
// frame (missing frames are gaps); for lag L = 1 .. min(max_lagtime,
// span - 1), <x^2>(L) is the mean of (x[f+L] - x[f])^2 over the pairs with
// both frames present (float32 differences and squares, summed in float64),
// likewise <y^2>, and msd = <x^2> + <y^2>.  A lag without a valid pair has
// no entry.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "gt.h"
#include "traj.h"

namespace gt {

namespace {

__global__ void id_range_kernel(const int64_t* ids, int64_t n, unsigned long long* lohi) {
    long long lo = LLONG_MAX, hi = LLONG_MIN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const long long v = (long long)ids[i];
        lo = min(lo, v);
        hi = max(hi, v);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin((long long*)&lohi[0], lo);
        atomicMax((long long*)&lohi[1], hi);
    }
}

__global__ void group_keys_kernel(const int64_t* ids, int64_t n, long long idmin, unsigned long long* keys) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        keys[i] = ((unsigned long long)(ids[i] - idmin) << 32) | (unsigned long long)i;
}

__device__ __forceinline__ unsigned int gkey(unsigned long long k) { return (unsigned int)(k >> 32); }

// 1 where a sorted position starts a particle's group
__global__ void heads_kernel(const unsigned long long* keys, int64_t n, int64_t* heads) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        heads[j] = (j == 0 || gkey(keys[j - 1]) != gkey(keys[j])) ? 1 : 0;
}

// gstart[g] = first sorted position of group g (groups in particle order),
// gstart[number of groups] = n
__global__ void gstart_kernel(const unsigned long long* keys, int64_t n, const int64_t* gid, int64_t* gstart) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const bool head = j == 0 || gkey(keys[j - 1]) != gkey(keys[j]);
        if (head) gstart[gid[j]] = j;
        if (j == n - 1) gstart[gid[j] + head] = n;
    }
}

// keep[row] for every row of groups with at least `threshold` rows;
// count[row] = rows of the row's group.  gid[j] counts the heads before j.
__global__ void stubs_kernel(const unsigned long long* keys, int64_t n, const int64_t* gid, const int64_t* gstart,
                             int64_t threshold, uint8_t* keep, int64_t* count, unsigned long long* nkept) {
    unsigned mine = 0;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const bool head = j == 0 || gkey(keys[j - 1]) != gkey(keys[j]);
        const int64_t g = gid[j] + head - 1;
        const int64_t rows = gstart[g + 1] - gstart[g];
        const int64_t row = (int64_t)(keys[j] & 0xffffffffu);
        const bool k = rows >= threshold;
        keep[row] = k;
        count[row] = rows;
        mine += k;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(nkept, (unsigned long long)mine);
}
// step_tracker: scaled positions per row (float32), steps in group order
// (float64: the lab code takes the float32 values as Python floats)
__global__ void steps_kernel(const unsigned long long* keys, int64_t n, const float* x, const float* y, float mppf,
                             float* xs, float* ys, double* x_step, double* y_step, double* steplength,
                             int64_t* order) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = (int64_t)(keys[j] & 0xffffffffu);
        const float xr = __fmul_rn(x[r], mppf), yr = __fmul_rn(y[r], mppf);
        xs[r] = xr;
        ys[r] = yr;
        double dx = 0.0, dy = 0.0;
        if (j > 0 && gkey(keys[j - 1]) == gkey(keys[j])) {
            const int64_t rp = (int64_t)(keys[j - 1] & 0xffffffffu);
            dx = __dsub_rn((double)xr, (double)__fmul_rn(x[rp], mppf));
            dy = __dsub_rn((double)yr, (double)__fmul_rn(y[rp], mppf));
        }
        x_step[j] = dx;
        y_step[j] = dy;
        // np.sqrt(y**2 + x**2) (hatzakis_lab_tracking.py:76)
        steplength[j] = __dsqrt_rn(__dadd_rn(__dmul_rn(dy, dy), __dmul_rn(dx, dx)));
        order[j] = r;
    }
}

// one block per (group, chunk of MSD_LAGS lags), threads over the lags:
// the lags of a long-lived particle spread over several blocks
constexpr int MSD_LAGS = 128;

// per group, a warp each: first frame, span, number of lags and of lag chunks;
// stat[0] error bits, stat[1] the longest lag
__global__ void msd_groups_kernel(const unsigned long long* keys, const int64_t* frames, const int64_t* gstart, int64_t G,
                                  int64_t max_lagtime, int64_t* gfirst, int64_t* gspan, int64_t* glags, int64_t* gchunks,
                                  unsigned long long* stat) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * blockDim.x / 32;
    for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; g < G; g += nw) {
        const int64_t e = gstart[g + 1];
        long long fmin = LLONG_MAX, fmax = LLONG_MIN;
        for (int64_t q = gstart[g] + lane; q < e; q += 32) {
            const long long f = (long long)frames[keys[q] & 0xffffffffu];
            fmin = min(fmin, f);
            fmax = max(fmax, f);
        }
        for (int o = 16; o > 0; o >>= 1) {
            fmin = min(fmin, __shfl_xor_sync(0xffffffffu, fmin, o));
            fmax = max(fmax, __shfl_xor_sync(0xffffffffu, fmax, o));
        }
        if (lane == 0) {
            int64_t span = fmax - fmin + 1;
            if (span > ((int64_t)1 << 31) || span < 1) {
                atomicOr(stat, 2ull);
                span = 1;
            }
            const int64_t lags = min(max_lagtime, span - 1);
            gfirst[g] = fmin;
            gspan[g] = span;
            glags[g] = lags;
            gchunks[g] = (lags + MSD_LAGS - 1) / MSD_LAGS;
            if (lags > 0) atomicMax(stat + 1, (unsigned long long)lags);
        }
    }
}

// positions of the groups on their frame axes (NaN = gap); a frame taken
// twice by one particle is an error (trackpy: "more than one trajectory
// per particle")
__global__ void msd_scatter_kernel(const unsigned long long* keys, const int64_t* frames, const float* x,
                                   const float* y, float mppf, const int64_t* gstart, const int64_t* gfirst,
                                   const int64_t* gbase, int64_t ngroups, float2* pos, int* taken,
                                   unsigned long long* stat) {
    for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int64_t e = gstart[g + 1];
        for (int64_t q = gstart[g] + threadIdx.x; q < e; q += blockDim.x) {
            const int64_t r = (int64_t)(keys[q] & 0xffffffffu);
            const int64_t s = gbase[g] + (frames[r] - gfirst[g]);
            if (atomicExch(taken + s, 1) != 0) atomicOr(stat, 1ull);
            pos[s] = make_float2(__fmul_rn(x[r], mppf), __fmul_rn(y[r], mppf));
        }
    }
}

__global__ void msd_kernel(const float2* pos, const int* taken, const int64_t* gbase, const int64_t* gspan,
                           const int64_t* glags, const int64_t* gout, const int64_t* cstart, int64_t ngroups,
                           int64_t nchunks, float* msd) {
    for (int64_t it = blockIdx.x; it < nchunks; it += gridDim.x) {
        // the group whose chunk range [cstart[g], cstart[g + 1]) holds it
        int64_t lo = 0, hi = ngroups - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) / 2;
            if (cstart[mid] <= it) lo = mid;
            else hi = mid - 1;
        }
        const int64_t g = lo;
        const float2* p = pos + gbase[g];
        const int* tk = taken + gbase[g];
        const int64_t span = gspan[g], nl = glags[g];
        const int64_t L0 = 1 + (it - cstart[g]) * MSD_LAGS;
        const int64_t L1 = min(nl, L0 + MSD_LAGS - 1);
        for (int64_t L = L0 + threadIdx.x; L <= L1; L += blockDim.x) {
            double sx = 0.0, sy = 0.0;
            int64_t cnt = 0;
            for (int64_t i = 0; i + L < span; ++i) {
                if (!tk[i] || !tk[i + L]) continue;
                const float2 a = p[i], b = p[i + L];
                const float dx = __fsub_rn(b.x, a.x), dy = __fsub_rn(b.y, a.y);
                sx += (double)__fmul_rn(dx, dx);
                sy += (double)__fmul_rn(dy, dy);
                ++cnt;
            }
            float v = CUDART_NAN_F;
            if (cnt > 0) v = __fadd_rn((float)(sx / (double)cnt), (float)(sy / (double)cnt));
            msd[gout[g] + L - 1] = v;
        }
    }
}

// (lag, group) sort keys of the entries, (lag - 1) * groups + group: the order
// of lags, then particles, in as few bits as it takes; entries without a pair
// get the key `last`
__global__ void msd_keys_kernel(const float* msd, const int64_t* gout, const int64_t* glags, int64_t ngroups,
                                unsigned long long last, unsigned long long* ekeys, int* eidx) {
    for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
        for (int64_t L = 1 + threadIdx.x; L <= glags[g]; L += blockDim.x) {
            const int64_t e = gout[g] + L - 1;
            ekeys[e] = isnan(msd[e]) ? last : (unsigned long long)(L - 1) * ngroups + g;
            eidx[e] = (int)e;
        }
    }
}

__global__ void msd_table_kernel(const unsigned long long* ekeys, const int* eidx, const float* msd, int64_t ne,
                                 int64_t ngroups, unsigned long long last, const unsigned long long* keys,
                                 const int64_t* gstart, long long idmin, float* out, unsigned long long* nvalid) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long k = ekeys[e];
        if (k == last) continue;
        if (e == ne - 1 || ekeys[e + 1] == last) *nvalid = (unsigned long long)(e + 1);
        const unsigned long long L = k / ngroups;
        const unsigned int pid = gkey(keys[gstart[k - L * ngroups]]);
        out[3 * e + 0] = (float)(L + 1);
        out[3 * e + 1] = (float)((long long)pid + idmin);
        out[3 * e + 2] = msd[eidx[e]];
    }
}

int bits_for(unsigned long long v) {
    int b = 0;
    while (b < 64 && (v >> b)) ++b;
    return b;
}

#define TK(x)                              \
    do {                                   \
        cudaError_t e_ = (x);              \
        if (e_ != cudaSuccess) {           \
            *msg = cudaGetErrorString(e_); \
            return GT_ERR_CUDA;            \
        }                                  \
    } while (0)
#define TA(p)                                  \
    do {                                       \
        if (!(p)) {                            \
            *msg = "device allocation failed"; \
            return GT_ERR_OOM;                 \
        }                                      \
    } while (0)

// Rows in pandas' groupby order: the sorted keys.
struct Sorted {
    unsigned long long* keys = nullptr;
    long long idmin = 0;
    unsigned long long range = 0;
};

int sort_rows(const int64_t* h_ids, int64_t n, TrajMem& M, cudaStream_t st, int grid, Sorted* out, std::string* msg) {
    int64_t* ids = M.get<int64_t>(n);
    unsigned long long* lohi = M.get<unsigned long long>(2);
    unsigned long long* k0 = M.get<unsigned long long>(n);
    unsigned long long* k1 = M.get<unsigned long long>(n);
    TA(ids && lohi && k0 && k1);
    TK(M.hc->upload(ids, h_ids, sizeof(int64_t) * n, st));
    const unsigned long long init[2] = {(unsigned long long)LLONG_MAX, (unsigned long long)LLONG_MIN};
    TK(cudaMemcpyAsync(lohi, init, sizeof(init), cudaMemcpyHostToDevice, st));
    id_range_kernel<<<grid, 256, 0, st>>>(ids, n, lohi);
    TK(cudaGetLastError());
    unsigned long long h[2];
    TK(M.hc->download(h, lohi, sizeof(h), st));
    out->idmin = (long long)h[0];
    const long long idmax = (long long)h[1];
    if (idmax - out->idmin >= (1LL << 31) || idmax < out->idmin) {
        *msg = "particle ids span more than 2^31 values";
        return GT_ERR_ARG;
    }
    out->range = (unsigned long long)(idmax - out->idmin);
    group_keys_kernel<<<grid, 256, 0, st>>>(ids, n, out->idmin, k0);
    TK(cudaGetLastError());
    out->keys = k0;
    if (out->range == 0) return GT_OK;  // one particle: in order
    const int end_bit = 32 + bits_for(out->range);
    cub::DoubleBuffer<unsigned long long> db(k0, k1);
    size_t tmp = 0;
    TK(cub::DeviceRadixSort::SortKeys(nullptr, tmp, db, (int)n, 32, end_bit, st));
    void* t = M.get<char>(tmp);
    TA(t);
    TK(cub::DeviceRadixSort::SortKeys(t, tmp, db, (int)n, 32, end_bit, st));
    out->keys = db.Current();
    return GT_OK;
}

// gid[j]: heads of groups before sorted position j; gstart as gstart_kernel
// (room for n + 1); *total (may be NULL) receives {gid, head} of the last row.
int find_groups(const Sorted& S, int64_t n, TrajMem& M, cudaStream_t st, int grid, int64_t** gid, int64_t** gstart,
                int64_t* total, std::string* msg) {
    int64_t* heads = M.get<int64_t>(n);
    *gid = M.get<int64_t>(n);
    *gstart = M.get<int64_t>(n + 1);
    size_t tmp = 0;
    TK(cub::DeviceScan::ExclusiveSum(nullptr, tmp, heads, *gid, (int)n, st));
    void* t = M.get<char>(tmp);
    TA(heads && *gid && *gstart && t);
    heads_kernel<<<grid, 256, 0, st>>>(S.keys, n, heads);
    TK(cudaGetLastError());
    TK(cub::DeviceScan::ExclusiveSum(t, tmp, heads, *gid, (int)n, st));
    gstart_kernel<<<grid, 256, 0, st>>>(S.keys, n, *gid, *gstart);
    TK(cudaGetLastError());
    if (total) {
        int64_t* h = M.hc->staged(total);
        TK(cudaMemcpyAsync(&h[0], *gid + n - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        TK(cudaMemcpyAsync(&h[1], heads + n - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        TK(cudaStreamSynchronize(st));
        total[0] = h[0];
        total[1] = h[1];
    }
    return GT_OK;
}

}  // namespace

int traj_filter_stubs(const int64_t* h_ids, int64_t n, int64_t threshold, uint8_t* h_keep, int64_t* h_count,
                      int64_t* nkept, TrajMem& M, cudaStream_t st, int num_sms, std::string* msg) {
    const int grid = num_sms * 8;
    TK(M.begin());
    Sorted S;
    int rc = sort_rows(h_ids, n, M, st, grid, &S, msg);
    int64_t *gid, *gstart;
    if (!rc) rc = find_groups(S, n, M, st, grid, &gid, &gstart, nullptr, msg);
    if (rc) return rc;
    uint8_t* keep = M.get<uint8_t>(n);
    int64_t* count = M.get<int64_t>(n);
    unsigned long long* cnt = M.get<unsigned long long>(1);
    TA(keep && count && cnt);
    TK(cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), st));
    stubs_kernel<<<grid, 256, 0, st>>>(S.keys, n, gid, gstart, threshold, keep, count, cnt);
    TK(cudaGetLastError());
    unsigned long long hk = 0;
    TK(M.hc->download(&hk, cnt, sizeof(hk), st));
    TK(M.hc->download(h_keep, keep, n, st));
    if (h_count) TK(M.hc->download(h_count, count, sizeof(int64_t) * n, st));
    *nkept = (int64_t)hk;
    return GT_OK;
}

int traj_steps(const int64_t* h_ids, const float* h_x, const float* h_y, int64_t n, float mppf, float* h_xs,
               float* h_ys, double* h_xstep, double* h_ystep, double* h_len, int64_t* h_order, TrajMem& M,
               cudaStream_t st, int num_sms, std::string* msg) {
    const int grid = num_sms * 8;
    TK(M.begin());
    Sorted S;
    int rc = sort_rows(h_ids, n, M, st, grid, &S, msg);
    if (rc) return rc;
    float* x = M.get<float>(n);
    float* y = M.get<float>(n);
    float* sxy = M.get<float>(2 * (size_t)n);
    double* st3 = M.get<double>(3 * (size_t)n);
    int64_t* order = M.get<int64_t>(n);
    TA(x && y && sxy && st3 && order);
    TK(M.hc->upload(x, h_x, sizeof(float) * n, st));
    TK(M.hc->upload(y, h_y, sizeof(float) * n, st));
    steps_kernel<<<grid, 256, 0, st>>>(S.keys, n, x, y, mppf, sxy, sxy + n, st3, st3 + n, st3 + 2 * n, order);
    TK(cudaGetLastError());
    TK(M.hc->download(h_xs, sxy, sizeof(float) * n, st));
    TK(M.hc->download(h_ys, sxy + n, sizeof(float) * n, st));
    double* dst[3] = {h_xstep, h_ystep, h_len};
    for (int i = 0; i < 3; ++i) TK(M.hc->download(dst[i], st3 + (size_t)i * n, sizeof(double) * n, st));
    TK(M.hc->download(h_order, order, sizeof(int64_t) * n, st));
    return GT_OK;
}

// Entries (lag, particle, msd) ordered by lag then particle, without the
// lags that have no valid pair; *out (3 floats per entry) comes from
// alloc(bytes).  *ms_msd: device time of the MSD kernel.
int traj_imsd(const int64_t* h_ids, const int64_t* h_frames, const float* h_x, const float* h_y, int64_t n,
              float mppf, int64_t max_lagtime, float* (*alloc)(size_t), float** out, int64_t* nout, float* ms_msd,
              TrajMem& M, cudaStream_t st, int num_sms, std::string* msg) {
    const int grid = num_sms * 8;
    TK(M.begin());
    Sorted S;
    int rc = sort_rows(h_ids, n, M, st, grid, &S, msg);
    if (rc) return rc;
    if (S.idmin < 0 || S.idmin + (long long)S.range >= (1LL << 24)) {
        *msg = "particle ids must lie in [0, 2^24) for the float32 result table";
        return GT_ERR_ARG;
    }
    int64_t *gid, *gstart, last2[2];
    rc = find_groups(S, n, M, st, grid, &gid, &gstart, last2, msg);
    if (rc) return rc;
    const int64_t G = last2[0] + last2[1];
    int64_t* frames = M.get<int64_t>(n);
    float* x = M.get<float>(n);
    float* y = M.get<float>(n);
    // per group: first, then span, lags, chunks, each with a spare entry so
    // that its exclusive sums (base, out offset, chunk start) end in the total
    const int64_t G1 = G + 1;
    int64_t* g7 = M.get<int64_t>(7 * (size_t)G1);
    unsigned long long* stat = M.get<unsigned long long>(3);  // error bits, longest lag, valid entries
    TA(frames && x && y && g7 && stat);
    int64_t *gfirst = g7, *gspan = g7 + G1, *glags = g7 + 2 * G1, *gchunks = g7 + 3 * G1;
    int64_t *gbase = g7 + 4 * G1, *gout = g7 + 5 * G1, *cstart = g7 + 6 * G1;
    TK(M.hc->upload(frames, h_frames, sizeof(int64_t) * n, st));
    TK(M.hc->upload(x, h_x, sizeof(float) * n, st));
    TK(M.hc->upload(y, h_y, sizeof(float) * n, st));
    TK(cudaMemsetAsync(stat, 0, 3 * sizeof(unsigned long long), st));
    if (max_lagtime < 0) max_lagtime = 0;
    msd_groups_kernel<<<grid, 256, 0, st>>>(S.keys, frames, gstart, G, max_lagtime, gfirst, gspan, glags, gchunks, stat);
    TK(cudaGetLastError());
    size_t tmp = 0;
    TK(cub::DeviceScan::ExclusiveSum(nullptr, tmp, gspan, gbase, (int)G1, st));
    void* t = M.get<char>(tmp);
    TA(t);
    TK(cub::DeviceScan::ExclusiveSum(t, tmp, gspan, gbase, (int)G1, st));
    TK(cub::DeviceScan::ExclusiveSum(t, tmp, glags, gout, (int)G1, st));
    TK(cub::DeviceScan::ExclusiveSum(t, tmp, gchunks, cstart, (int)G1, st));
    int64_t words[6];
    int64_t* h = M.hc->staged(words);
    TK(cudaMemcpyAsync(&h[0], gbase + G, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TK(cudaMemcpyAsync(&h[1], gout + G, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TK(cudaMemcpyAsync(&h[2], cstart + G, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TK(cudaMemcpyAsync(&h[3], stat, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TK(cudaStreamSynchronize(st));
    const int64_t tot_span = h[0], tot_out = h[1], nchunks = h[2];
    unsigned long long hs[3] = {(unsigned long long)h[3], (unsigned long long)h[4], (unsigned long long)h[5]};
    if (hs[0]) {
        *msg = "a particle spans more than 2^31 frames";
        return GT_ERR_ARG;
    }
    if (tot_span > ((int64_t)1 << 32) || tot_out >= ((int64_t)1 << 31)) {
        *msg = "trajectories span too many frames in total";
        return GT_ERR_ARG;
    }
    float2* pos = M.get<float2>(tot_span);
    int* taken = M.get<int>(tot_span);
    TA(pos && taken);
    TK(cudaMemsetAsync(taken, 0, sizeof(int) * tot_span, st));
    const int gg = (int)std::min<int64_t>(std::max<int64_t>(G, 1), (int64_t)num_sms * 64);
    msd_scatter_kernel<<<gg, 128, 0, st>>>(S.keys, frames, x, y, mppf, gstart, gfirst, gbase, G, pos, taken, stat);
    TK(cudaGetLastError());
    *ms_msd = 0.f;
    float* tab = nullptr;
    const bool timed = tot_out > 0;
    if (timed) {
        float* msd = M.get<float>(tot_out);
        unsigned long long* ekeys = M.get<unsigned long long>(tot_out);
        unsigned long long* ekeys2 = M.get<unsigned long long>(tot_out);
        int* eidx = M.get<int>(tot_out);
        int* eidx2 = M.get<int>(tot_out);
        tab = M.get<float>(3 * (size_t)tot_out);
        TA(msd && ekeys && ekeys2 && eidx && eidx2 && tab);
        const int gc = (int)std::min<int64_t>(std::max<int64_t>(nchunks, 1), (int64_t)num_sms * 64);
        TK(cudaEventRecord(M.ev[0], st));
        msd_kernel<<<gc, MSD_LAGS, 0, st>>>(pos, taken, gbase, gspan, glags, gout, cstart, G, nchunks, msd);
        TK(cudaEventRecord(M.ev[1], st));
        TK(cudaGetLastError());
        const unsigned long long last = hs[1] * (unsigned long long)G;
        msd_keys_kernel<<<gg, 128, 0, st>>>(msd, gout, glags, G, last, ekeys, eidx);
        TK(cudaGetLastError());
        cub::DoubleBuffer<unsigned long long> dk(ekeys, ekeys2);
        cub::DoubleBuffer<int> dv(eidx, eidx2);
        const int bits = bits_for(last);
        TK(cub::DeviceRadixSort::SortPairs(nullptr, tmp, dk, dv, (int)tot_out, 0, bits, st));
        t = M.get<char>(tmp);
        TA(t);
        TK(cub::DeviceRadixSort::SortPairs(t, tmp, dk, dv, (int)tot_out, 0, bits, st));
        msd_table_kernel<<<grid, 256, 0, st>>>(dk.Current(), dv.Current(), msd, tot_out, G, last, S.keys, gstart, S.idmin,
                                               tab, stat + 2);
        TK(cudaGetLastError());
    }
    TK(M.hc->download(hs, stat, sizeof(hs), st));
    if (hs[0]) {
        *msg = "more than one position for a particle in one frame (one trajectory per particle expected)";
        return GT_ERR_ARG;
    }
    if (timed) cudaEventElapsedTime(ms_msd, M.ev[0], M.ev[1]);
    const int64_t nvalid = (int64_t)hs[2];
    *out = alloc(sizeof(float) * 3 * (size_t)std::max<int64_t>(nvalid, 1));
    if (!*out) {
        *msg = "host allocation failed";
        return GT_ERR_OOM;
    }
    if (nvalid > 0) TK(cudaMemcpyAsync(*out, tab, sizeof(float) * 3 * (size_t)nvalid, cudaMemcpyDeviceToHost, st));
    TK(cudaStreamSynchronize(st));
    *nout = nvalid;
    return GT_OK;
}

}  // namespace gt
