// finalize.cu -- per-frame ordering, separation filter and particle tables.
//
// Replaces the host-side raster scan (execute_gpu.rs:157-183) and the
// kd-tree separation filter (execute_gpu.rs:258-284).  One CTA per frame:
//   1. exclusive scan of the per-(row, tile column) record counts gives every
//      record its raster position (the reference's pre-filter `idx`);
//   2. records waiting on nothing (state EMIT) are compacted in raster order;
//   3. a uniform grid (cell >= separation + 1) bins them, and a point is
//      dropped if a neighbour closer than `separation` has a larger mass, or
//      an equal mass and a smaller raster index (single pass, as the
//      reference);
//   4. survivors form the frame's particle table in raster order, and a
//      second grid over them serves the linker's candidate search.
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

// Counting sort of n points into cells: start[ncell+1], idx[n] and, when
// asked for, their positions in that order.
template <int NT>
__device__ void build_grid(const float* ys, const float* xs, int n, float G, int ncy, int ncx, int* cnt_s, int* start,
                           int* idx, float2* pos, int* warp_tot, int* s_total) {
    const int ncell = ncy * ncx;
    for (int c = threadIdx.x; c < ncell; c += NT) cnt_s[c] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += NT) atomicAdd(&cnt_s[cell_of(ys[i], xs[i], G, ncy, ncx)], 1);
    __syncthreads();
    block_scan_inplace<NT>(cnt_s, ncell, warp_tot, s_total);
    for (int c = threadIdx.x; c < ncell; c += NT) start[c] = cnt_s[c];
    if (threadIdx.x == 0) start[ncell] = n;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += NT) {
        const float y = ys[i], x = xs[i];
        const int k = atomicAdd(&cnt_s[cell_of(y, x, G, ncy, ncx)], 1);
        idx[k] = i;
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

template <int NTF>
__device__ __forceinline__ void finalize_frame(const LocParams& p, const MovieBufs& b, float sep, int link_grid,
                                               int frame0, int* cnt_s, int* warp_tot, int& s_total) {
    const int t = frame0 + blockIdx.x;
    const int cap_c = b.cap_c;
    const int nrc = p.H * p.ntx;
    int* rc = b.rowcnt + (size_t)t * nrc;
    const Cand* cand = b.cand + (size_t)t * cap_c;
    int* perm = b.cperm + (size_t)t * cap_c;
    float* cy = b.cy + (size_t)t * cap_c;
    float* cx = b.cx + (size_t)t * cap_c;
    float* cm = b.cm + (size_t)t * cap_c;
    int* crec = b.crec + (size_t)t * cap_c;
    int* keep = b.ccell + (size_t)t * cap_c;

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

    // 1. raster positions
    block_scan_inplace<NTF>(rc, nrc, warp_tot, &s_total);
    for (int k = threadIdx.x; k < nrec; k += NTF) perm[k] = k;
    __syncthreads();
    for (int k = threadIdx.x; k < nrec; k += NTF) {
        const Cand& c = cand[k];
        if (c.u < 0 || c.u >= p.H || c.v < 0 || c.v >= p.W) continue;
        const int dest = rc[c.u * p.ntx + c.v / p.TW] + c.rowrank;
        if (dest >= 0 && dest < nrec) perm[dest] = k;
    }
    __syncthreads();

    // 2. compact emitted records in raster order
    for (int i = threadIdx.x; i < nrec; i += NTF) keep[i] = cand[perm[i]].state == CAND_EMIT ? 1 : 0;
    __syncthreads();
    const int ne = block_scan_inplace<NTF>(keep, nrec, warp_tot, &s_total);
    for (int i = threadIdx.x; i < nrec; i += NTF) {
        const int k = perm[i];
        const Cand& c = cand[k];
        if (c.state != CAND_EMIT) continue;
        const int e = keep[i];
        cy[e] = c.y; cx[e] = c.x; cm[e] = c.mass; crec[e] = k;
    }
    __syncthreads();

    // 3. separation filter on a uniform grid
    const float G = (float)b.G;
    const int ncell = b.ncx * b.ncy;
    int* cstart = b.cstart + (size_t)t * (ncell + 1);
    int* cidx = b.cidx + (size_t)t * cap_c;
    build_grid<NTF>(cy, cx, ne, G, b.ncy, b.ncx, cnt_s, cstart, cidx, nullptr, warp_tot, &s_total);
    for (int i = threadIdx.x; i < ne; i += NTF) {
        const float qy = cy[i], qx = cx[i], qm = cm[i];
        const int c = cell_of(qy, qx, G, b.ncy, b.ncx);
        const int gy = c / b.ncx, gx = c - gy * b.ncx;
        bool k = true;
        for (int dy = -1; dy <= 1 && k; ++dy) {
            const int yy = gy + dy;
            if (yy < 0 || yy >= b.ncy) continue;
            for (int dx = -1; dx <= 1 && k; ++dx) {
                const int xx = gx + dx;
                if (xx < 0 || xx >= b.ncx) continue;
                const int cc = yy * b.ncx + xx;
                for (int s = cstart[cc]; s < cstart[cc + 1]; ++s) {
                    const int j = cidx[s];
                    if (j == i) continue;
                    float dd;
                    if (!within_r(qy, qx, cy[j], cx[j], sep, &dd)) continue;
                    const float nm = cm[j];
                    if (qm < nm || (qm == nm && i > j)) { k = false; break; }
                }
            }
        }
        keep[i] = k ? 1 : 0;
    }
    __syncthreads();

    // 4. survivors in raster order
    const int np = block_scan_inplace<NTF>(keep, ne, warp_tot, &s_total);
    const bool over = np > b.cap_p;
    if (over && threadIdx.x == 0) atomicOr(b.err, ERR_PART_OVERFLOW);
    float* py = b.py + (size_t)t * b.cap_p;
    float* px = b.px + (size_t)t * b.cap_p;
    float* pm = b.pm + (size_t)t * b.cap_p;
    int* prec = b.prec + (size_t)t * b.cap_p;
    // keep[i] now holds the survivor index; recompute survivorship from the
    // scan (a survivor is where the next prefix value increases)
    for (int i = threadIdx.x; i < ne; i += NTF) {
        const int a = keep[i];
        const int nxt = (i + 1 < ne) ? keep[i + 1] : np;
        if (nxt > a && a < b.cap_p) {
            py[a] = cy[i]; px[a] = cx[i]; pm[a] = cm[i]; prec[a] = crec[i];
        }
    }
    if (threadIdx.x == 0) b.npart[t] = over ? b.cap_p : np;
    __syncthreads();

    // 5. grid over the particles for the linker
    if (link_grid) {
        const int n = over ? b.cap_p : np;
        build_grid<NTF>(py, px, n, (float)b.LG, b.lncy, b.lncx, cnt_s,
                        b.gstart + (size_t)t * ((size_t)b.lncx * b.lncy + 1), b.gidx + (size_t)t * b.cap_p,
                        b.gpos + (size_t)t * b.cap_p, warp_tot, &s_total);
    }
}

template <int NTF>
__global__ void __launch_bounds__(NTF) finalize_kernel(const LocParams p, MovieBufs b, float sep,
                                                       int link_grid, int frame0) {
    __shared__ int warp_tot[NTF / 32];
    __shared__ int s_total, s_last;
    extern __shared__ int cnt_s[];  // cells of the larger grid
    finalize_frame<NTF>(p, b, sep, link_grid, frame0, cnt_s, warp_tot, s_total);
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
    if (big) finalize_kernel<1024><<<nf, 1024, smem, st>>>(p, b, sep, link_grid, frame0);
    else finalize_kernel<512><<<nf, 512, smem, st>>>(p, b, sep, link_grid, frame0);
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
    build_grid<NTG>(py + (size_t)t * cap_p, px + (size_t)t * cap_p, npart[t], (float)G, ncy, ncx, cnt_s,
               gstart + (size_t)t * (ncell + 1), gidx + (size_t)t * cap_p, gpos + (size_t)t * cap_p, warp_tot, &s_total);
}

}  // namespace gt
