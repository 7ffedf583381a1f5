// assemble.cu -- frame offsets, trajectory IDs and the output table.
//
// The output table has the reference's column layout (execute_gpu.rs:197-226,
// rows written at 337-368): frame, mass, y, x, [particle], [Rg, ecc, signal],
// [raw_mass], [raw_bg_median, raw_mass_corrected], [Rg_gpu, raw_mass_gpu,
// signal_gpu, ecc_gpu], all f32, frames ascending, particles of a frame in
// raster order of their originating pixel.
#include <math_constants.h>

#include <algorithm>

#include "gt_device.cuh"

namespace gt {



// Exclusive scan of n ints into out[0..n] by one CTA of 1024 threads.
__global__ void __launch_bounds__(1024) scan_frames_kernel(const int* in, int* out, int n) {
    __shared__ int warp_tot[32];
    __shared__ int s_total;
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < n; b0 += 1024) {
        const int i = b0 + threadIdx.x;
        const int v = i < n ? in[i] : 0;
        const int e = block_excl_scan<1024>(v, warp_tot, &s_total);
        if (i < n) out[i] = carry + e;
        __syncthreads();
        if (threadIdx.x == 0) carry += s_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = carry;
}

// newid[g] for particles that start a trajectory: running counter in
// (frame, index) order (linking.rs:470).
__global__ void newid_kernel(const int* newrank, const int* newbase, const int* off, const int* npart,
                             int* newid, int T) {
    const int t = blockIdx.x;
    if (t >= T) return;
    const int n = npart[t];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int g = off[t] + i;
        const int r = newrank[g];
        newid[g] = r >= 0 ? newbase[t] + r : -1;
    }
}

namespace {
__device__ __forceinline__ float raw_at(const AsmArgs& a, size_t fbase, int r, int c) {
    if (r < 0 || r >= a.H || c < 0 || c >= a.W) return CUDART_NAN_F;
    return load_px(a.frames, a.dtype, fbase + (size_t)r * a.W + c);
}
}  // namespace

namespace {
// Order-preserving integer of a float that is not NaN.
__device__ __forceinline__ unsigned order_key(float v) {
    const unsigned u = __float_as_uint(v);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_value(unsigned k) {
    return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k);
}

constexpr int RING = 512;  // background pixels kept in shared memory per warp

// raw_mass [, raw_bg_median, raw_mass_corrected] of one row by a warp
// (execute_gpu.rs:311-331: at the rounded refined position, NaN outside the
// frame and skipped).  The signal is summed in table order; the median takes
// the order statistics bit by bit from the top, counting the pixels below a
// candidate (a thread per row that ranked every ring pixel against all others
// took 3.4 ms for 7600 rows with rings of 140 pixels).
__device__ void raw_columns(const AsmArgs& a, size_t fbase, float y, float x, float* out, float* ring) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int mr = (int)roundf(y), mc = (int)roundf(x);
    float acc = 0.f;
    for (int q0 = 0; q0 < a.n_sig; q0 += 32) {
        const int q = q0 + lane;
        const float v = q < a.n_sig ? raw_at(a, fbase, mr + __ldg(a.sig_off + 2 * q), mc + __ldg(a.sig_off + 2 * q + 1))
                                    : CUDART_NAN_F;
        const int n = min(32, a.n_sig - q0);
        for (int u = 0; u < n; ++u) {
            const float w = __shfl_sync(full, v, u);
            if (!isnan(w)) acc = acc + w;
        }
    }
    if (lane == 0) out[0] = acc;
    if (!a.bg) return;
    auto pixel = [&](int q) { return raw_at(a, fbase, mr + __ldg(a.bg_off + 2 * q), mc + __ldg(a.bg_off + 2 * q + 1)); };
    const bool kept = a.n_bg <= RING;
    int nv = 0;
    __syncwarp();
    for (int q = lane; q < a.n_bg; q += 32) {
        const float v = pixel(q);
        if (kept) ring[q] = v;
        nv += !isnan(v);
    }
    nv = __reduce_add_sync(full, nv);
    __syncwarp();
    float med = CUDART_NAN_F;
    if (nv > 0) {
        // median with linear interpolation (ndarray-stats Linear, q = 0.5)
        const int lo = (nv - 1) / 2, hi = nv / 2;
        unsigned klo = 0;  // largest key with at most lo pixels below it
        for (unsigned bit = 0x80000000u; bit; bit >>= 1) {
            const unsigned cand = klo | bit;
            int below = 0;
            for (int q = lane; q < a.n_bg; q += 32) {
                const float v = kept ? ring[q] : pixel(q);
                below += !isnan(v) && order_key(v) < cand;
            }
            if (__reduce_add_sync(full, below) <= lo) klo = cand;
        }
        unsigned khi = klo;
        if (hi != lo) {
            // the next pixel in order: klo again, or the smallest above it
            int upto = 0;
            unsigned above = 0xffffffffu;
            for (int q = lane; q < a.n_bg; q += 32) {
                const float v = kept ? ring[q] : pixel(q);
                if (isnan(v)) continue;
                const unsigned k = order_key(v);
                upto += k <= klo;
                if (k > klo) above = min(above, k);
            }
            upto = __reduce_add_sync(full, upto);
            above = __reduce_min_sync(full, above);
            if (upto <= hi) khi = above;
        }
        const float vlo = key_value(klo), vhi = key_value(khi);
        const double frac = (hi == lo) ? 0.0 : 0.5;
        med = vlo + (float)(frac * ((double)vhi - (double)vlo));
    }
    if (lane == 0) {
        out[1] = med;
        out[2] = acc - med * (float)a.n_sig;
    }
}
}  // namespace

// gridDim.y blocks of ASM_NT threads per frame (blockIdx.x).
constexpr int ASM_NT = 256;
__global__ void __launch_bounds__(ASM_NT) assemble_kernel(AsmArgs a) {
    __shared__ float ring[ASM_NT / 32][RING];
    const int t = blockIdx.x;
    if (t >= a.T) return;
    const int n = a.npart[t];
    const size_t fbase = (size_t)t * a.H * a.W;
    const int c_raw = 4 + (a.has_link ? 1 : 0) + (a.cpu_processed ? 3 : 0);
    for (int i = blockIdx.y * ASM_NT + threadIdx.x; i < n; i += gridDim.y * ASM_NT) {
        const int g = a.off[t] + i;
        if (g >= a.out_rows) break;  // rows in index order: the rest are beyond too
        const size_t s = (size_t)t * a.cap_p + i;
        float* row = a.out + (size_t)g * a.ncols;
        const float mass = a.pm[s];
        const float y = a.py[s], x = a.px[s];
        int c = 0;
        row[c++] = (float)t;
        row[c++] = mass;
        row[c++] = y;
        row[c++] = x;
        if (a.has_link) row[c++] = (float)a.newid[a.root[g]];
        const Cand& rec = a.cand[(size_t)t * a.cap_c + a.prec[s]];
        if (a.walk && g < a.walk_rows) {
            int* wr = a.walk + (size_t)g * 5;
            wr[0] = t; wr[1] = rec.ul; wr[2] = rec.vl; wr[3] = rec.up; wr[4] = rec.vp;
        }
        if (a.cpu_processed) {
            // execute_gpu.rs:349-351
            row[c++] = sqrtf(rec.rg_sum / mass);
            row[c++] = rec.eccn / (mass - rec.mid);
            row[c++] = rec.signal;
        }
        if (a.sig) c += a.bg ? 3 : 1;
        if (a.characterize) {
            row[c++] = rec.g_rg;
            row[c++] = rec.g_raw;
            row[c++] = rec.g_sig;
            row[c++] = rec.g_ecc;
        }
    }
    if (!a.sig) return;
    const int warp = threadIdx.x >> 5;
    for (int i = blockIdx.y * (ASM_NT / 32) + warp; i < n; i += gridDim.y * (ASM_NT / 32)) {
        const int g = a.off[t] + i;
        if (g >= a.out_rows) break;
        const size_t s = (size_t)t * a.cap_p + i;
        raw_columns(a, fbase, a.py[s], a.px[s], a.out + (size_t)g * a.ncols + c_raw, ring[warp]);
    }
}

// Blocks per frame so that few frames still fill the GPU (a frame of 5700 rows
// in one block took 41 us, the time of 12 of them).
cudaError_t launch_assemble(const AsmArgs& a, int num_sms, cudaStream_t st) {
    const int per = std::max(1, std::min(64, 4 * num_sms / std::max(a.T, 1)));
    assemble_kernel<<<dim3(a.T, per), ASM_NT, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace gt
