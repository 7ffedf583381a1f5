// finalize.cu -- per-frame ordering, separation filter and particle tables.
//
// Replaces the host-side raster scan (execute_gpu.rs:157-183) and the
// kd-tree separation filter (execute_gpu.rs:258-284).  One CTA per frame:
//   1. exclusive scan of the per-(row, tile column) record counts gives every
//      record its raster position (the order of the reference's pre-filter
//      `idx`); the records are listed in that order;
//   2. a uniform grid (cell >= separation + 1) bins those waiting on nothing
//      (state EMIT), and a point is dropped if a neighbour closer than
//      `separation` has a larger mass, or an equal mass and a smaller raster
//      position (single pass, as the reference);
//   3. survivors form the frame's particle table in raster order, and a
//      second grid over them serves the linker's candidate search.
// What bounds it: the latency of its steps, each a pass over the frame's
// records after a barrier.  The counts and the lists are in shared memory where
// they are short (FIN_COUNTS, FIN_LIST).
#include "gt_device.cuh"

namespace gt {

namespace {
// In-place exclusive scan of n ints (any memory space); returns the sum.  A
// warp scans a contiguous stretch, 32 neighbouring ints at a time: a thread per
// stretch read global memory uncoalesced and hit one shared bank 32 times
// (three scans a frame, 200 of the 324 us of 12 frames of 2048 x 2560).
template <int NT>
__device__ int block_scan_inplace(int* data, int n, int* warp_tot, int* s_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n + NT - 1) / NT * 32;
    const int b0 = min(n, warp * per), b1 = min(n, b0 + per);
    int mine = 0;
#pragma unroll 4
    for (int i = b0 + lane; i < b1; i += 32) mine += data[i];
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) warp_tot[warp] = mine;
    __syncthreads();
    if (warp == 0) {
        const int v = lane < NT / 32 ? warp_tot[lane] : 0;
        int x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane < NT / 32) warp_tot[lane] = x - v;
        if (lane == 31) *s_total = x;
    }
    __syncthreads();
    int carry = warp_tot[warp];
    constexpr int UN = 4;
    for (int base = b0; base < b1; base += 32 * UN) {
        int v[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int i = base + 32 * u + lane;
            v[u] = i < b1 ? data[i] : 0;
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int i = base + 32 * u + lane;
            int x = v[u];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            if (i < b1) data[i] = carry + x - v[u];
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    return *s_total;
}

__device__ __forceinline__ int cell_of(float y, float x, float G, int ncy, int ncx) {
    int cy = (int)floorf(y / G), cx = (int)floorf(x / G);
    cy = clampi(cy, 0, ncy - 1);
    cx = clampi(cx, 0, ncx - 1);
    return cy * ncx + cx;
}

// Counting sort of points into cells: item(i, &id, &y, &x) gives the i-th of n
// (false: none).  The ids in cell order go to idx and, where asked for, the
// cells' starts (ncell + 1) and the positions in that order to start and pos.
// cnt_s is left with every cell's end.
template <int NT, class F>
__device__ void build_grid(int n, float G, int ncy, int ncx, int* cnt_s, int* start, int* idx, float2* pos,
                           int* warp_tot, int* s_total, F&& item) {
    const int ncell = ncy * ncx;
    int id;
    float y, x;
    for (int c = threadIdx.x; c < ncell; c += NT) cnt_s[c] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += NT)
        if (item(i, &id, &y, &x)) atomicAdd(&cnt_s[cell_of(y, x, G, ncy, ncx)], 1);
    __syncthreads();
    const int total = block_scan_inplace<NT>(cnt_s, ncell, warp_tot, s_total);
    if (start) {
        for (int c = threadIdx.x; c < ncell; c += NT) start[c] = cnt_s[c];
        if (threadIdx.x == 0) start[ncell] = total;
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += NT) {
        if (!item(i, &id, &y, &x)) continue;
        const int k = atomicAdd(&cnt_s[cell_of(y, x, G, ncy, ncx)], 1);
        idx[k] = id;
        if (pos) pos[k] = make_float2(y, x);
    }
    __syncthreads();
}

// kd-tree 0.4.2 within_radius restated from its twin in linking.rs:73-105:
// per-axis box test, then (item - query)^2 summed from zero, strictly < r^2.
__device__ __forceinline__ bool within_r(float qy, float qx, float iy, float ix, float r, float* dist) {
    if (iy < qy - r || iy > qy + r) return false;
    if (ix < qx - r || ix > qx + r) return false;
    const float dy = iy - qy, dx = ix - qx;
    float dd = 0.f;
    dd = dd + dy * dy;
    dd = dd + dx * dx;
    *dist = dd;
    return dd < r * r;
}
}  // namespace

// Counts of a frame, and records of a frame, that the block keeps in shared
// memory, which also holds the cells of the larger grid (FinShared: ints).
constexpr int FIN_COUNTS = 4096, FIN_LIST = 1024;
struct FinShared {
    int cells, counts, list;  // list: records, six ints each
};

template <int NTF>
__device__ __forceinline__ void finalize_frame(const LocParams& p, const MovieBufs& b, float sep, int link_grid,
                                               int frame0, int* cnt_s, FinShared sh, int* warp_tot, int& s_total) {
    const int t = frame0 + blockIdx.x;
    const int cap_c = b.cap_c;
    const int nrc = p.H * p.ntx;
    int* rc = b.rowcnt + (size_t)t * nrc;
    const Cand* cand = b.cand + (size_t)t * cap_c;

    const int nrec = b.fcount[t];
    if (nrec > cap_c) {
        // the locate kernel flagged the overflow and left slots unwritten;
        // the host retries with larger slabs
        if (threadIdx.x == 0) b.npart[t] = 0;
        if (link_grid) {  // empty particle grid keeps the linker in bounds
            const int ncell = b.lncx * b.lncy;
            int* gs = b.gstart + (size_t)t * (ncell + 1);
            for (int c = threadIdx.x; c <= ncell; c += NTF) gs[c] = 0;
        }
        return;
    }
    // the lists: positions, masses, records and the survivors' flags in raster
    // order, and the grid's entries
    const bool small = nrec <= sh.list;
    int* list = cnt_s + sh.cells + sh.counts;
    const size_t at = (size_t)t * cap_c;
    float* cy = small ? (float*)list : b.cy + at;
    float* cx = small ? (float*)list + sh.list : b.cx + at;
    float* cm = small ? (float*)list + 2 * sh.list : b.cm + at;
    int* crec = small ? list + 3 * sh.list : b.crec + at;
    int* keep = small ? list + 4 * sh.list : b.ccell + at;
    int* cidx = small ? list + 5 * sh.list : b.cidx + at;

    // 1. raster order
    if (nrc <= sh.counts) {
        int* rs = cnt_s + sh.cells;
#pragma unroll 4
        for (int i = threadIdx.x; i < nrc; i += NTF) rs[i] = rc[i];
        rc = rs;
    }
    for (int i = threadIdx.x; i < nrec; i += NTF) keep[i] = 0;
    __syncthreads();
    block_scan_inplace<NTF>(rc, nrc, warp_tot, &s_total);
    for (int k = threadIdx.x; k < nrec; k += NTF) {
        const Cand& c = cand[k];
        const int u = c.u, v = c.v, rank = c.rowrank, state = c.state;
        const float y = c.y, x = c.x, mass = c.mass;
        if (u < 0 || u >= p.H || v < 0 || v >= p.W) continue;
        const int i = rc[u * p.ntx + v / p.TW] + rank;
        if (i < 0 || i >= nrec || state != CAND_EMIT) continue;
        keep[i] = 1;
        cy[i] = y; cx[i] = x; cm[i] = mass; crec[i] = k;
    }
    __syncthreads();

    // 2. separation filter on a uniform grid
    const float G = (float)b.G;
    build_grid<NTF>(nrec, G, b.ncy, b.ncx, cnt_s, nullptr, cidx, nullptr, warp_tot, &s_total,
                    [&](int i, int* id, float* y, float* x) {
                        *id = i;
                        *y = cy[i]; *x = cx[i];
                        return keep[i] != 0;
                    });
    for (int i = threadIdx.x; i < nrec; i += NTF) {
        if (!keep[i]) continue;
        const float qy = cy[i], qx = cx[i], qm = cm[i];
        const int c = cell_of(qy, qx, G, b.ncy, b.ncx);
        const int gy = c / b.ncx, gx = c - gy * b.ncx;
        const int x0 = max(gx - 1, 0), x1 = min(gx + 1, b.ncx - 1);
        bool k = true;
        for (int yy = max(gy - 1, 0); yy <= min(gy + 1, b.ncy - 1) && k; ++yy) {
            const int c0 = yy * b.ncx + x0;
            const int s1 = cnt_s[yy * b.ncx + x1];
            for (int s = c0 > 0 ? cnt_s[c0 - 1] : 0; s < s1; ++s) {
                const int j = cidx[s];
                if (j == i) continue;
                float dd;
                if (!within_r(qy, qx, cy[j], cx[j], sep, &dd)) continue;
                const float nm = cm[j];
                if (qm < nm || (qm == nm && i > j)) { k = false; break; }
            }
        }
        if (!k) keep[i] = 0;
    }
    __syncthreads();

    // 3. survivors in raster order
    const int np = block_scan_inplace<NTF>(keep, nrec, warp_tot, &s_total);
    const bool over = np > b.cap_p;
    if (over && threadIdx.x == 0) atomicOr(b.err, ERR_PART_OVERFLOW);
    float* py = b.py + (size_t)t * b.cap_p;
    float* px = b.px + (size_t)t * b.cap_p;
    float* pm = b.pm + (size_t)t * b.cap_p;
    int* prec = b.prec + (size_t)t * b.cap_p;
    // keep[i] now holds the survivor index; a survivor is where the next prefix
    // value increases
    auto survivor = [&](int i, int* id, float* y, float* x) {
        const int a = keep[i];
        *id = a;
        if (((i + 1 < nrec) ? keep[i + 1] : np) <= a || a >= b.cap_p) return false;
        *y = cy[i]; *x = cx[i];
        return true;
    };
    for (int i = threadIdx.x; i < nrec; i += NTF) {
        int a;
        float y, x;
        if (survivor(i, &a, &y, &x)) {
            py[a] = y; px[a] = x; pm[a] = cm[i]; prec[a] = crec[i];
        }
    }
    if (threadIdx.x == 0) b.npart[t] = over ? b.cap_p : np;

    // the grid over the particles for the linker
    if (link_grid)
        build_grid<NTF>(nrec, (float)b.LG, b.lncy, b.lncx, cnt_s,
                        b.gstart + (size_t)t * ((size_t)b.lncx * b.lncy + 1), b.gidx + (size_t)t * b.cap_p,
                        b.gpos + (size_t)t * b.cap_p, warp_tot, &s_total, survivor);
}

template <int NTF>
__global__ void __launch_bounds__(NTF) finalize_kernel(const LocParams p, MovieBufs b, float sep,
                                                       int link_grid, int frame0, FinShared sh) {
    __shared__ int warp_tot[NTF / 32];
    __shared__ int s_total, s_last;
    extern __shared__ int cnt_s[];  // cells of the larger grid, counts, lists
    finalize_frame<NTF>(p, b, sep, link_grid, frame0, cnt_s, sh, warp_tot, s_total);
    if (!b.done) return;
    // the last block done: offsets of the launch's frames (a launch of its own
    // costs a short movie more than the sums)
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(b.done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int n = gridDim.x;
    int carry = frame0 > 0 ? b.off[frame0] : 0;
    for (int b0 = 0; b0 < n; b0 += NTF) {
        const int i = b0 + threadIdx.x;
        const int v = i < n ? __ldcg(b.npart + frame0 + i) : 0;
        const int e = block_excl_scan<NTF>(v, warp_tot, &s_total);
        if (i < n) b.off[frame0 + i] = carry + e;
        carry += s_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        b.off[frame0 + n] = carry;
        *b.nrows = carry;
        *b.done = 0;
    }
}

// Frames of 2^20 pixels and more: 1024 threads.
cudaError_t launch_finalize(const LocParams& p, const MovieBufs& b, float sep, int link_grid, int frame0, int nf,
                            size_t smem, cudaStream_t st) {
    const bool big = (long long)p.H * p.W >= (1LL << 20);
    const cudaError_t e = big ? allow_shared<finalize_kernel<1024>>() : allow_shared<finalize_kernel<512>>();
    if (e != cudaSuccess) return e;
    FinShared sh{(int)(smem / sizeof(int)), 0, 0};
    const int nrc = p.H * p.ntx;
    if (nrc <= FIN_COUNTS) sh.counts = nrc;
    if (smem + sizeof(int) * (size_t)(sh.counts + 6 * FIN_LIST) <= 226 * 1024) sh.list = FIN_LIST;
    else sh.counts = 0;  // cells of the finest grids fill the block's share
    smem += sizeof(int) * (size_t)(sh.counts + 6 * sh.list);
    if (big) finalize_kernel<1024><<<nf, 1024, smem, st>>>(p, b, sep, link_grid, frame0, sh);
    else finalize_kernel<512><<<nf, 512, smem, st>>>(p, b, sep, link_grid, frame0, sh);
    return cudaGetLastError();
}

// Grid over externally supplied particle tables (standalone linking).
constexpr int NTG = 512;
__global__ void __launch_bounds__(NTG) grid_kernel(const float* py, const float* px, const int* npart,
                                                   int cap_p, int G, int ncy, int ncx, int* gstart,
                                                   int* gidx, float2* gpos) {
    __shared__ int warp_tot[NTG / 32];
    __shared__ int s_total;
    extern __shared__ int cnt_s[];
    const int t = blockIdx.x;
    const int ncell = ncx * ncy;
    py += (size_t)t * cap_p;
    px += (size_t)t * cap_p;
    build_grid<NTG>(npart[t], (float)G, ncy, ncx, cnt_s, gstart + (size_t)t * (ncell + 1), gidx + (size_t)t * cap_p,
                    gpos + (size_t)t * cap_p, warp_tot, &s_total, [&](int i, int* id, float* y, float* x) {
                        *id = i;
                        *y = py[i]; *x = px[i];
                        return true;
                    });
}

}  // namespace gt
