// adjoint.cu -- bandpass + centroid refinement at fixed peaks, its adjoint
// and the per-particle localisation uncertainty.
//
// At a fixed walk (last-read pixel (ul, vl), final position (up, vp)) a
// located feature is a smooth function of the frame away from the clip:
//
//   R(p) = G(p) - B(p)             bandpass before the clip, G the Gaussian
//                                  pass (zero padded, normalised by the full
//                                  tap sum), B the boxcar mean (reflect
//                                  padded, divided by k*k)
//   P(p) = max(R(p), 0)
//   m    = sum_c P(ul + i_c, vl + j_c)          over the centroid circle
//   y    = up + sum_c i_c P(..) / m,  x = vp + sum_c j_c P(..) / m
//
// (walk_cols.wgsl:38-74, centers.wgsl:23-109, preprocess_rows.wgsl:14-53,
// preprocess_cols.wgsl:14-61).  The forward kernel re-evaluates the bandpass
// at the circle pixels with the locate kernels' exact operation order, so
// its (y, x, mass) equal the located rows bit for bit.  The backward pass
// recomputes the same bandpass values (nothing from the forward is stored),
// stores each peak's dL/dR (K values) and links the peak to the output tiles
// in its reach; the transposed bandpass then sums each tile's dL/dR in shared
// memory and filters it there, so that HBM sees the frames once and the
// gradient once (a plane of dL/dR in HBM, zeroed, added to and read back, took
// 128 of 895 us for 256 x 512x512 frames with 102k peaks, and bandpass values
// evaluated tap by tap per circle pixel 520 us; now 89 us forward, 128 backward
// particles, 184 transpose).  The clip has subgradient 0 at R == 0.
//
// Parameter derivatives: noise_size is the Gaussian variance s, and
// dG/ds = (da (x) a + a (x) da) * I with a_i = w_i / sum(w).  smoothing_size
// k is an integer window; its derivative is taken through the box
// normalisation 1/k^2 treated as continuous (window and Gaussian tap count
// held fixed): dR/dk = 2 B / k.
#include <cuda_runtime.h>
#include <algorithm>
#include <math_constants.h>

#include "gt_internal.cuh"
#include "gt_simd.cuh"

namespace gt {

namespace {

constexpr int ADJ_NT = 128;
constexpr int TR_TW = 64, TR_NT = 256;
// rows of a transpose tile: 64 with a compile-time radius, else 32
__host__ __device__ constexpr int tr_th(int krt) { return krt > 0 ? 64 : 32; }

struct BpTerms {
    float r;      // bandpass before the clip
    float bmean;  // boxcar mean B
    float dg;     // dG/ds
};

// The bandpass at (u, v) in the operation order of the locate kernels
// (row pass: fmaf over taps, times the reciprocal of the tap sum; column
// pass likewise, boxcar subtracted as fma(-box, 1/k^2, gauss); box sums in
// tap order), plus B and dG/ds in real-valued arithmetic.
__device__ __forceinline__ BpTerms bandpass_terms(const AdjParams& p, const float* fr, int u, int v) {
    const int kr = p.krad, H = p.H, W = p.W;
    float gs = 0.f, cs = 0.f, dg = 0.f;
    for (int i = -kr; i <= kr; ++i) {
        int pu = u + i;
        bool in_r = true;
        if (pu < 0) { pu = -pu - 1; in_r = false; }
        else if (pu >= H) { pu = 2 * H - pu - 1; in_r = false; }
        float rg = 0.f, rb = 0.f, ra = 0.f, rda = 0.f;
        const float* row = fr + (size_t)pu * W;
        for (int j = -kr; j <= kr; ++j) {
            int pv = v + j;
            bool in_c = true;
            if (pv < 0) { pv = -pv - 1; in_c = false; }
            else if (pv >= W) { pv = 2 * W - pv - 1; in_c = false; }
            const float val = __ldg(row + pv);
            if (in_c) {
                rg = fmaf(p.w[j + kr], val, rg);
                ra = fmaf(p.a[j + kr], val, ra);
                rda = fmaf(p.da[j + kr], val, rda);
            }
            rb = rb + val;
        }
        const float tg = rg * p.rn;
        if (in_r) {
            gs = fmaf(p.w[i + kr], tg, gs);
            dg = fmaf(p.da[i + kr], ra, dg);
            dg = fmaf(p.a[i + kr], rda, dg);
        }
        cs = cs + rb;
    }
    BpTerms t;
    t.r = fmaf(-cs, p.rkk, gs * p.rn);
    t.bmean = cs * p.rkk;
    t.dg = dg;
    return t;
}

// Number of taps of the reflect-padded box at p (window +-kr, one
// reflection) that land on q, along one axis of length n.
__device__ __forceinline__ int box_count(int pp, int q, int n, int kr) {
    return (abs(q - pp) <= kr) + (abs(-q - 1 - pp) <= kr) + (abs(2 * n - q - 1 - pp) <= kr);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;  // every lane
}

}  // namespace

enum AdjMode { ADJ_FORWARD = 0, ADJ_BACKWARD = 1, ADJ_UNCERTAINTY = 2 };

// Circle pixels of radius R (i * i + j * j <= R * R), in table order.
__host__ __device__ constexpr int circle_size(int R) {
    int k = 0;
    for (int i = -R; i <= R; ++i)
        for (int j = -R; j <= R; ++j) k += i * i + j * j <= R * R;
    return k;
}

// Shared floats of a warp, a multiple of 4: R, B, dG/ds at the circle pixels
// and 3K of the uncertainty; with a compile-time radius also the clipped
// values, the raw window and the row pass's sums over it.
__host__ __device__ constexpr int round4(int x) { return (x + 3) / 4 * 4; }
__host__ __device__ constexpr int adj_rows(int r) { return (4 * r + 1) * (2 * r + 1); }
__host__ __device__ constexpr int adj_warp_floats(int mode, int r, int K) {
    return r > 0 ? round4(K) + round4(6 * K + (4 * r + 1) * (4 * r + 1) + adj_rows(r) * (mode == 1 ? 4 : 2)) : round4(6 * K);
}

// The bandpass at the circle pixels of a peak whose whole window lies inside
// the frame (smoothing radius = circle radius = R): the raw window once into
// shared memory, the row sums once per (row, circle column), the column sums
// per circle pixel -- the values of bandpass_terms in the same order.  Bound
// by instructions issued, so lanes map to rows and columns without divisions.
template <int MODE, int R>
__device__ __forceinline__ void window_terms(const AdjParams& p, const float* fr, int ul, int vl, const int* sci,
                                             float* win, float* sR, float* sB, float* sD) {
    constexpr int WS = 4 * R + 1, CW = 2 * R + 1, NP = WS * CW, K = circle_size(R);
    constexpr int LW = WS <= 8 ? 8 : WS <= 16 ? 16 : 32, LC = CW <= 4 ? 4 : CW <= 8 ? 8 : 16;  // lanes per row
    const int lane = threadIdx.x & 31;
    float* rg = win + WS * WS;
    float* rb = rg + NP;
    float* ra = rb + NP;
    float* rd = ra + NP;
    {
        const int r0 = lane / LW, c = lane % LW;
        const float* src = fr + (size_t)(ul - 2 * R + r0) * p.W + (vl - 2 * R + c);
        const size_t step = (size_t)(32 / LW) * p.W;
        if (c < WS) {
#pragma unroll
            for (int r = 0; r < WS; r += 32 / LW) {
                if (r + r0 < WS) win[(r + r0) * WS + c] = __ldg(src);
                src += step;
            }
        }
    }
    __syncwarp();
    {
        const int r0 = lane / LC, c = lane % LC;
        if (c < CW) {
#pragma unroll
            for (int r = 0; r < WS; r += 32 / LC) {
                if (r + r0 >= WS) break;
                const float* w = win + (r + r0) * WS + c;
                float g = 0.f, b = 0.f, a = 0.f, d = 0.f;
#pragma unroll
                for (int j = 0; j < CW; ++j) {
                    const float v = w[j];
                    g = fmaf(p.w[j], v, g);
                    b = b + v;
                    if (MODE == 1) {
                        a = fmaf(p.a[j], v, a);
                        d = fmaf(p.da[j], v, d);
                    }
                }
                const int q = (r + r0) * CW + c;
                rg[q] = g * p.rn;
                rb[q] = b;
                if (MODE == 1) {
                    ra[q] = a;
                    rd[q] = d;
                }
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int c0 = 0; c0 < K; c0 += 32) {
        const int c = c0 + lane;
        if (c >= K) break;
        const int q0 = (sci[2 * c] + R) * CW + sci[2 * c + 1] + R;
        float gs = 0.f, cs = 0.f, dg = 0.f;
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            const int q = q0 + i * CW;
            gs = fmaf(p.w[i], rg[q], gs);
            cs = cs + rb[q];
            if (MODE == 1) {
                dg = fmaf(p.da[i], ra[q], dg);
                dg = fmaf(p.a[i], rd[q], dg);
            }
        }
        sR[c] = fmaf(-cs, p.rkk, gs * p.rn);
        if (MODE == 1) {
            sB[c] = cs * p.rkk;
            sD[c] = dg;
        }
    }
}

// Centroid sums over the clipped circle values P (16-byte aligned) in
// centers.wgsl:23-109 order (i outer, j inner), every lane alike.
template <int R>
__device__ __forceinline__ void circle_sums(const float* P, float& a0, float& a1, float& mm) {
    constexpr int K = circle_size(R);
    float v[round4(K)];
#pragma unroll
    for (int q = 0; q < K; q += 4) {
        const float4 z = *(const float4*)(P + q);
        v[q] = z.x; v[q + 1] = z.y; v[q + 2] = z.z; v[q + 3] = z.w;
    }
    a0 = a1 = mm = 0.f;
    int q = 0;
#pragma unroll
    for (int i = -R; i <= R; ++i)
#pragma unroll
        for (int j = -R; j <= R; ++j) {
            if (i * i + j * j > R * R) continue;
            a0 = fmaf(v[q], (float)i, a0);
            a1 = fmaf(v[q], (float)j, a1);
            mm = mm + v[q];
            ++q;
        }
}

// One warp per particle (grid-stride over warps), ADJ_NT / 32 warps per
// CTA sharing the circle table.  walk rows: {frame, ul, vl, up, vp}.
// FORWARD writes yxm (n x 3).  BACKWARD reads grad (n x 3), writes dL/dR at the
// circle pixels to tl.g (n x K), links the peak to the tiles whose output it
// reaches and writes the block's dL/d{noise_size, smoothing_size} to gpar.
// R: smoothing and circle radius where they are equal and at most 7, else 0.  UNCERTAINTY writes the standard deviations of (y, x, mass) under
// var(I) = gain * max(I, 0) + read_var by linear propagation (n x 3).
template <int MODE, int R>
__global__ void __launch_bounds__(ADJ_NT) adjoint_particle_kernel(AdjParams p, const float* __restrict__ frames,
                                                                  const int* __restrict__ walk, long long n,
                                                                  const int* __restrict__ circ,
                                                                  const float* __restrict__ grad, float* yxm,
                                                                  AdjTiles tl, double* gpar, int* err) {
    extern __shared__ __align__(16) float asm_[];
    constexpr int NW = ADJ_NT / 32;
    const int K = R > 0 ? circle_size(R) : p.K;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int* sci = (int*)asm_;                      // 2K circle offsets {i, j}, shared
    float* sP = asm_ + round4(2 * K) + wid * adj_warp_floats(MODE, R, K);
    float* sR = sP + (R > 0 ? round4(K) : 0);   // this warp's R at the circle pixels
    float* sB = sR + K;                         // B
    float* sD = sB + K;                         // dG/ds
    float* sJ = sD + K;                         // 3K: dy/dR, dx/dR, dm/dR (uncertainty)
    float* win = sJ + 3 * K;
    for (int q = threadIdx.x; q < 2 * K; q += ADJ_NT) sci[q] = circ[q];
    __syncthreads();
    const int H = p.H, W = p.W, kr = p.krad, b = p.border;
    const long long wstride = (long long)gridDim.x * NW;
    double acc_ds = 0.0, acc_dk = 0.0;  // this warp's parameter gradients (BACKWARD)
    for (long long k = (long long)blockIdx.x * NW + wid; k < n; k += wstride) {
        const int* wr = walk + 5 * k;
        const int t = __ldg(wr), ul = __ldg(wr + 1), vl = __ldg(wr + 2), up = __ldg(wr + 3), vp = __ldg(wr + 4);
        const bool valid = t >= 0 && t < p.T && ul >= 0 && ul < H && vl >= 0 && vl < W && up >= 0 && up < H &&
                           vp >= 0 && vp < W;
        if (!valid) {
            if (lane == 0) atomicOr(err, 1);
            continue;
        }
        const bool interior = !(ul - b < 0 || ul + b >= H || vl - b < 0 || vl + b >= W);
        if (!interior) {
            // centers.wgsl border band: offset (0, 0), mass 0, no dependence
            // on the frame
            if (lane == 0) {
                if (MODE == ADJ_FORWARD) {
                    yxm[3 * k] = (float)up; yxm[3 * k + 1] = (float)vp; yxm[3 * k + 2] = 0.f;
                } else if (MODE == ADJ_UNCERTAINTY) {
                    yxm[3 * k] = 0.f; yxm[3 * k + 1] = 0.f; yxm[3 * k + 2] = 0.f;
                }
            }
            continue;
        }
        const float* fr = frames + (size_t)t * H * W;
        __syncwarp();  // the previous particle's reads of this warp's arrays are done
        if (R > 0 && ul - 2 * R >= 0 && ul + 2 * R < H && vl - 2 * R >= 0 && vl + 2 * R < W) {
            window_terms<MODE, R>(p, fr, ul, vl, sci, win, sR, sB, sD);
        } else {
            for (int c = lane; c < K; c += 32) {
                const BpTerms bt = bandpass_terms(p, fr, ul + sci[2 * c], vl + sci[2 * c + 1]);
                sR[c] = bt.r;
                sB[c] = bt.bmean;
                sD[c] = bt.dg;
            }
        }
        __syncwarp();
        float c0, c1, m;
        if constexpr (R > 0) {
            for (int c = lane; c < K; c += 32) sP[c] = sR[c] < 0.f ? 0.f : sR[c];
            __syncwarp();
            circle_sums<R>(sP, c0, c1, m);
        } else {
            // centers.wgsl:23-109 accumulation order (i outer, j inner): lane 0
            // sums i P, lane 1 j P, the others P (fma(P, 1, m) is m + P)
            float sum = 0.f;
            for (int c = 0; c < K; ++c) {
                const float data = sR[c] < 0.f ? 0.f : sR[c];
                sum = fmaf(data, lane < 2 ? (float)sci[2 * c + lane] : 1.f, sum);
            }
            c0 = __shfl_sync(0xffffffffu, sum, 0);
            c1 = __shfl_sync(0xffffffffu, sum, 1);
            m = __shfl_sync(0xffffffffu, sum, 2);
        }
        c0 = __fmul_rn(c0, __frcp_rn(m));  // centers.wgsl:82-83, a shader division
        c1 = __fmul_rn(c1, __frcp_rn(m));
        if constexpr (MODE == ADJ_FORWARD) {
            if (lane == 0) {
                yxm[3 * k] = (float)up + c0;
                yxm[3 * k + 1] = (float)vp + c1;
                yxm[3 * k + 2] = m;
            }
            continue;
        }
        if (!(m > 0.f) || !isfinite(m)) {
            // zero mass: the centroid is undefined and the row is never
            // emitted (mass > minmass and mass != 0)
            if (MODE == ADJ_UNCERTAINTY && lane == 0) {
                yxm[3 * k] = 0.f; yxm[3 * k + 1] = 0.f; yxm[3 * k + 2] = 0.f;
            }
            continue;
        }
        const float inv_m = 1.f / m;
        if constexpr (MODE == ADJ_BACKWARD) {
            const float gy = __ldg(grad + 3 * k), gx = __ldg(grad + 3 * k + 1), gm = __ldg(grad + 3 * k + 2);
            float ds = 0.f, dk = 0.f;
            // link the peak to the tiles that its circle, widened by kr, meets
            const int reach = p.rc + kr;
            const int ty0 = max(ul - reach, 0) / tl.th, tx0 = max(vl - reach, 0) / TR_TW;
            const int ny = min(ul + reach, H - 1) / tl.th - ty0 + 1, nx = min(vl + reach, W - 1) / TR_TW - tx0 + 1;
            for (int q = lane; q < ny * nx; q += 32) {
                const int tile = (t * tl.nty + ty0 + q / nx) * tl.ntx + tx0 + q % nx;
                const int at = atomicAdd(tl.count + tile, 1);
                if (at < TILE_PEAKS) {
                    tl.peaks[(size_t)tile * TILE_PEAKS + at] = (int)k;
                } else {
                    const int entry = (int)(k * tl.slots) + q;
                    tl.next[entry] = atomicExch(tl.head + tile, entry + 1);
                }
            }
            for (int c = lane; c < K; c += 32) {
                float* gc = tl.g + (size_t)k * K + c;
                if (!(sR[c] > 0.f)) {
                    *gc = 0.f;
                    continue;
                }
                const float ic = (float)sci[2 * c], jc = (float)sci[2 * c + 1];
                const float g = gm + (gy * (ic - c0) + gx * (jc - c1)) * inv_m;
                *gc = g;
                ds = fmaf(g, sD[c], ds);
                dk = fmaf(g, 2.f * sB[c] / p.k, dk);
            }
            acc_ds += (double)warp_sum(ds);
            acc_dk += (double)warp_sum(dk);
            continue;
        }
        if constexpr (MODE == ADJ_UNCERTAINTY) {
            // Jacobian rows over the window that the circle's bandpass
            // reads, J(q) = sum_c dR_c/dI(q) * dOut/dR_c
            for (int c = lane; c < K; c += 32) {
                const bool on = sR[c] > 0.f;
                sJ[c] = on ? ((float)sci[2 * c] - c0) * inv_m : 0.f;
                sJ[K + c] = on ? ((float)sci[2 * c + 1] - c1) * inv_m : 0.f;
                sJ[2 * K + c] = on ? 1.f : 0.f;
            }
            __syncwarp();
            const int WR = p.rc + kr, WS = 2 * WR + 1;
            float vy = 0.f, vx = 0.f, vm = 0.f;
            for (int q = lane; q < WS * WS; q += 32) {
                const int qu = ul - WR + q / WS, qv = vl - WR + q % WS;
                if (qu < 0 || qu >= H || qv < 0 || qv >= W) continue;
                float jy = 0.f, jx = 0.f, jm = 0.f;
                for (int c = 0; c < K; ++c) {
                    const int pu = ul + sci[2 * c], pv = vl + sci[2 * c + 1];
                    const int du = qu - pu, dv = qv - pv;
                    float wgt = 0.f;
                    if (abs(du) <= kr && abs(dv) <= kr) wgt = p.a[du + kr] * p.a[dv + kr];
                    const int nb = box_count(pu, qu, H, kr) * box_count(pv, qv, W, kr);
                    if (nb) wgt -= (float)nb / p.kk;
                    jy = fmaf(sJ[c], wgt, jy);
                    jx = fmaf(sJ[K + c], wgt, jx);
                    jm = fmaf(sJ[2 * K + c], wgt, jm);
                }
                const float iq = __ldg(fr + (size_t)qu * W + qv);
                const float var = fmaf(p.gain, fmaxf(iq, 0.f), p.read_var);
                vy = fmaf(jy * jy, var, vy);
                vx = fmaf(jx * jx, var, vx);
                vm = fmaf(jm * jm, var, vm);
            }
            const float ty = warp_sum(vy), tx = warp_sum(vx), tm = warp_sum(vm);
            if (lane == 0) {
                yxm[3 * k] = sqrtf(ty);
                yxm[3 * k + 1] = sqrtf(tx);
                yxm[3 * k + 2] = sqrtf(tm);
            }
        }
    }
    if constexpr (MODE == ADJ_BACKWARD) {
        // this block's partial sums, in warp order; adjoint_param_reduce_kernel
        // adds the blocks' partials in block order, so the parameter
        // gradient is the same on every run (particles map to warps and
        // blocks by a fixed grid stride)
        __shared__ double red[2 * NW];
        if (lane == 0) { red[2 * wid] = acc_ds; red[2 * wid + 1] = acc_dk; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0, c = 0.0;
            for (int w = 0; w < NW; ++w) { a += red[2 * w]; c += red[2 * w + 1]; }
            gpar[2 * blockIdx.x] = a;
            gpar[2 * blockIdx.x + 1] = c;
        }
    }
}

// out[0..1] = the sums of part[2b], part[2b + 1] over blocks b in a fixed
// order: thread i takes blocks i, i + 256, ... in order, then a fixed tree.
// `add`: onto the sums of earlier chunks of peaks.
__global__ void __launch_bounds__(256) adjoint_param_reduce_kernel(const double* part, int nblocks, double* out,
                                                                   int add) {
    __shared__ double sa[256], sc[256];
    double a = 0.0, c = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 256) {
        a += part[2 * b];
        c += part[2 * b + 1];
    }
    sa[threadIdx.x] = a;
    sc[threadIdx.x] = c;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            sa[threadIdx.x] += sa[threadIdx.x + h];
            sc[threadIdx.x] += sc[threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = add ? out[0] + sa[0] : sa[0];
        out[1] = add ? out[1] + sc[0] : sc[0];
    }
}

// Transposed bandpass of dL/dR:  dL/dI = G^T gR - B^T gR.  G is separable,
// symmetric and zero padded, so G^T is the same Gaussian pass; B^T weights
// each tap by the number of reflect-padded window positions that land on it
// (box_count), all of which lie within +-kr of the output pixel: 1 away from
// the frame edges.  One CTA per tile of tr_th x 64 output pixels: the peaks
// linked to it add their dL/dR to a shared plane with a kr halo, which two
// separable passes over row pairs (packed FP32x2, 8 outputs per item) filter;
// a tile without peaks is zero.  Bound by the arithmetic and shared memory
// traffic of the passes, then by the gradient's write.
template <int KRT>  // smoothing half window; 0 = taken from p.krad at run time
__global__ void __launch_bounds__(TR_NT) adjoint_transpose_kernel(AdjParams p, AdjTiles tl, const int* __restrict__ walk,
                                                                  const int* __restrict__ circ,
                                                                  float* __restrict__ gI, int frame0, int add) {
    extern __shared__ __align__(16) float tsm[];
    constexpr int TH = tr_th(KRT), LIST = 256;
    __shared__ int s_list[LIST];
    __shared__ int s_n, s_entry;
    const int kr = KRT > 0 ? KRT : p.krad;
    const int H = p.H, W = p.W, K = p.K;
    const int SH = TH + 2 * kr, SW = TR_TW + 2 * kr;
    const int SS = SW | 1;            // row pair strides, odd: conflict-free column of pairs
    constexpr int RS = TR_TW | 1;
    float2* S = (float2*)tsm;         // SH / 2 x SS
    float2* RG = S + (SH / 2) * SS;   // SH / 2 x RS, Gaussian row pass
    float2* RB = RG + (SH / 2) * RS;  // SH / 2 x RS, box row pass
    const int u0 = (blockIdx.x / tl.ntx) * TH, v0 = (blockIdx.x % tl.ntx) * TR_TW;
    const int t = frame0 + blockIdx.y;
    float* dst = gI + (size_t)t * H * W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a scalar of the pair planes
    auto at = [](float2* plane, int stride, int r, int c) -> float& {
        return ((float*)plane)[(((r >> 1) * stride + c) << 1) + (r & 1)];
    };
    const size_t tile = ((size_t)t * tl.nty + blockIdx.x / tl.ntx) * tl.ntx + blockIdx.x % tl.ntx;
    const int count = __ldg(tl.count + tile);
    if (count == 0) {
        if (add) return;
        for (int q = threadIdx.x; q < TH * TR_TW; q += TR_NT) {
            const int qu = u0 + q / TR_TW, qv = v0 + q % TR_TW;
            if (qu < H && qv < W) dst[(size_t)qu * W + qv] = 0.f;
        }
        return;
    }
    // the tile's peaks: the first TILE_PEAKS from its array, then the list
    int n = min(count, TILE_PEAKS);
    if (threadIdx.x < n) s_list[threadIdx.x] = __ldg(tl.peaks + tile * TILE_PEAKS + threadIdx.x);
    if (threadIdx.x == 0) s_entry = count > TILE_PEAKS ? __ldg(tl.head + tile) : 0;
    for (int q = threadIdx.x; q < (SH / 2) * SS; q += TR_NT) S[q] = make_float2(0.f, 0.f);
    __syncthreads();
    while (true) {
        for (int e = warp; e < n; e += TR_NT / 32) {
            const long long k = s_list[e];
            const int ru = __ldg(walk + 5 * k + 1) - u0 + kr, rv = __ldg(walk + 5 * k + 2) - v0 + kr;
            for (int c = lane; c < K; c += 32) {
                const float g = __ldg(tl.g + (size_t)k * K + c);
                const int r = ru + __ldg(circ + 2 * c), x = rv + __ldg(circ + 2 * c + 1);
                if (g != 0.f && r >= 0 && r < SH && x >= 0 && x < SW) atomicAdd(&at(S, SS, r, x), g);
            }
        }
        const int rest = s_entry;  // read by all before thread 0 writes the next one
        __syncthreads();
        if (rest == 0) break;
        if (threadIdx.x == 0) {
            int entry = s_entry, q = 0;
            for (; entry > 0 && q < LIST; entry = __ldg(tl.next + entry - 1)) s_list[q++] = (entry - 1) / tl.slots;
            s_n = q;
            s_entry = entry;
        }
        __syncthreads();
        n = s_n;
    }
    const float ikk = 1.f / p.kk;
    // box sums along a row or column of length n whose outputs near its ends
    // count reflected taps: tap(q) is the value at position q, 0 <= q < n
    auto edge_box = [&](int q, int n, auto&& tap) {
        float bx = 0.f;
        for (int j = -kr; j <= kr; ++j) {
            const int pp = q + j;
            if (pp >= 0 && pp < n) bx = fmaf((float)box_count(pp, q, n, kr), tap(j), bx);
        }
        return bx;
    };
    if constexpr (KRT > 0) {
        constexpr int TP = 2 * KRT + 1, F = 8;
        float2 a2[TP];
#pragma unroll
        for (int j = 0; j < TP; ++j) a2[j] = make_float2(p.a[j], p.a[j]);
        // row pass: 8 outputs of a row pair per item, pairs fastest across the
        // lanes.  Sums direct, not running: a window of zeros must give zero
        constexpr int NPR = (TH + 2 * KRT) / 2;
        for (int it = threadIdx.x; it < NPR * (TR_TW / F); it += TR_NT) {
            const int c0 = it / NPR * F, pr = it % NPR;
            const float2* srow = S + pr * SS + c0;
            float2 v[F + TP - 1];
#pragma unroll
            for (int i = 0; i < F + TP - 1; ++i) v[i] = srow[i];
#pragma unroll
            for (int m = 0; m < F; ++m) {
                float2 g = make_float2(0.f, 0.f), bs = v[m];
#pragma unroll
                for (int j = 0; j < TP; ++j) g = fma2(a2[j], v[m + j], g);
#pragma unroll
                for (int j = 1; j < TP; ++j) bs = add2(bs, v[m + j]);
                RG[pr * RS + c0 + m] = g;
                RB[pr * RS + c0 + m] = bs;
            }
        }
        __syncthreads();
        if (v0 < KRT || v0 + TR_TW > W - KRT) {
            // columns within kr of the left or right frame edge
            const int le = max(0, min(KRT, W) - v0), r0 = max(max(0, W - KRT - v0), le), r1 = min(TR_TW, W - v0);
            const int ncol = le + max(0, r1 - r0);
            for (int it = threadIdx.x; it < ncol * SH; it += TR_NT) {
                const int q = it / SH, r = it - q * SH;
                const int c = q < le ? q : r0 + (q - le);
                at(RB, RS, r, c) = edge_box(v0 + c, W, [&](int j) { return at(S, SS, r, c + KRT + j); });
            }
            __syncthreads();
        }
        // column pass: 8 rows of one column per item, columns fastest
        const bool rows_inner = u0 >= KRT && u0 + TH <= H - KRT;
        for (int it = threadIdx.x; it < TR_TW * (TH / F); it += TR_NT) {
            const int c = it % TR_TW, r0 = it / TR_TW * F;
            if (u0 + r0 >= H || v0 + c >= W) continue;
            float2 l[F / 2 + KRT], ml[F / 2 + KRT - 1];
            float2 gs[F / 2], bs[F / 2];
#pragma unroll
            for (int i = 0; i < F / 2 + KRT; ++i) l[i] = RG[(r0 / 2 + i) * RS + c];
#pragma unroll
            for (int i = 0; i < F / 2 + KRT - 1; ++i) ml[i] = make_float2(l[i].y, l[i + 1].x);
#pragma unroll
            for (int m = 0; m < F / 2; ++m) {
                gs[m] = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < TP; ++j) gs[m] = fma2(a2[j], (j & 1) ? ml[m + (j >> 1)] : l[m + (j >> 1)], gs[m]);
            }
#pragma unroll
            for (int i = 0; i < F / 2 + KRT; ++i) l[i] = RB[(r0 / 2 + i) * RS + c];
#pragma unroll
            for (int i = 0; i < F / 2 + KRT - 1; ++i) ml[i] = make_float2(l[i].y, l[i + 1].x);
#pragma unroll
            for (int m = 0; m < F / 2; ++m) {
                bs[m] = l[m];
#pragma unroll
                for (int j = 1; j < TP; ++j) bs[m] = add2(bs[m], (j & 1) ? ml[m + (j >> 1)] : l[m + (j >> 1)]);
            }
            float o[F];
#pragma unroll
            for (int m = 0; m < F / 2; ++m) {
                o[2 * m] = fmaf(-bs[m].x, ikk, gs[m].x);
                o[2 * m + 1] = fmaf(-bs[m].y, ikk, gs[m].y);
            }
            float* d = dst + (size_t)(u0 + r0) * W + (v0 + c);
            if (rows_inner && !add) {
#pragma unroll
                for (int m = 0; m < F; ++m) d[(size_t)m * W] = o[m];
            } else {
#pragma unroll
                for (int m = 0; m < F; ++m) {
                    const int qu = u0 + r0 + m;
                    if (qu >= H) break;
                    if (qu < KRT || qu >= H - KRT) {
                        const float bx = edge_box(qu, H, [&](int j) { return at(RB, RS, r0 + m + KRT + j, c); });
                        o[m] = fmaf(-bx, ikk, (m & 1) ? gs[m / 2].y : gs[m / 2].x);
                    }
                    d[(size_t)m * W] = add ? d[(size_t)m * W] + o[m] : o[m];
                }
            }
        }
    } else {
        for (int q = threadIdx.x; q < SH * TR_TW; q += TR_NT) {
            const int r = q / TR_TW, c = q % TR_TW;
            if (v0 + c >= W) continue;
            float g = 0.f;
            for (int j = 0; j <= 2 * kr; ++j) g = fmaf(p.a[j], at(S, SS, r, c + j), g);
            at(RG, RS, r, c) = g;
            at(RB, RS, r, c) = edge_box(v0 + c, W, [&](int j) { return at(S, SS, r, c + kr + j); });
        }
        __syncthreads();
        for (int q = threadIdx.x; q < TH * TR_TW; q += TR_NT) {
            const int r = q / TR_TW, c = q % TR_TW;
            if (u0 + r >= H || v0 + c >= W) continue;
            float g = 0.f;
            for (int i = 0; i <= 2 * kr; ++i) g = fmaf(p.a[i], at(RG, RS, r + i, c), g);
            const float bx = edge_box(u0 + r, H, [&](int j) { return at(RB, RS, r + kr + j, c); });
            float* d = dst + (size_t)(u0 + r) * W + (v0 + c);
            const float o = fmaf(-bx, ikk, g);
            *d = add ? *d + o : o;
        }
    }
}

namespace {
int adj_radius(const AdjParams& p) { return p.rc == p.krad && p.krad <= 7 ? p.krad : 0; }
}  // namespace

// Upper bound of the particle kernel's grid (partial sums of the backward
// pass: two doubles per block).
int adjoint_particle_blocks_max(int num_sms) { return num_sms * 16; }

// Tile lists of the backward pass: tiles per frame and the most tiles that a
// peak reaches (its circle widened by the smoothing radius).
void adjoint_tiles(const AdjParams& p, AdjTiles* tl) {
    tl->th = tr_th(p.krad >= 1 && p.krad <= 7 ? p.krad : 0);
    tl->nty = (p.H + tl->th - 1) / tl->th;
    tl->ntx = (p.W + TR_TW - 1) / TR_TW;
    const int ext = 2 * (p.rc + p.krad);
    tl->slots = (ext / tl->th + 2) * (ext / TR_TW + 2);
}

template <int MODE, int R>
cudaError_t particles_launch(const AdjParams& p, const float* frames, const int* walk, long long n, const int* circ,
                             const float* grad, float* yxm, const AdjTiles& tl, double* gpar, int* err, int grid,
                             cudaStream_t st) {
    const size_t smem = sizeof(float) * (size_t)(round4(2 * p.K) + (ADJ_NT / 32) * adj_warp_floats(MODE, R, p.K));
    const auto fn = adjoint_particle_kernel<MODE, R>;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e) return e;
    fn<<<grid, ADJ_NT, smem, st>>>(p, frames, walk, n, circ, grad, yxm, tl, gpar, err);
    return cudaGetLastError();
}

// BACKWARD: `add` keeps the parameter gradients of earlier chunks of peaks.
cudaError_t launch_adjoint_particles(int mode, const AdjParams& p, const float* frames, const int* walk, long long n,
                                     const int* circ, const float* grad, float* yxm, const AdjTiles& tl, double* gpar,
                                     double* gpart, int* err, int add, int num_sms, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int grid = (int)std::min<long long>((n + ADJ_NT / 32 - 1) / (ADJ_NT / 32), (long long)num_sms * 16);
    double* out = mode == ADJ_BACKWARD ? gpart : gpar;
    cudaError_t e = cudaErrorInvalidValue;
#define ADJ_CASE(R)                                                                                               \
    case R:                                                                                                       \
        e = mode == ADJ_FORWARD                                                                                   \
                ? particles_launch<ADJ_FORWARD, R>(p, frames, walk, n, circ, grad, yxm, tl, out, err, grid, st)   \
            : mode == ADJ_BACKWARD                                                                                \
                ? particles_launch<ADJ_BACKWARD, R>(p, frames, walk, n, circ, grad, yxm, tl, out, err, grid, st)  \
                : particles_launch<ADJ_UNCERTAINTY, R>(p, frames, walk, n, circ, grad, yxm, tl, out, err, grid, st); \
        break;
    switch (adj_radius(p)) {
        ADJ_CASE(0) ADJ_CASE(1) ADJ_CASE(2) ADJ_CASE(3) ADJ_CASE(4) ADJ_CASE(5) ADJ_CASE(6) ADJ_CASE(7)
    }
#undef ADJ_CASE
    if (e || mode != ADJ_BACKWARD) return e;
    adjoint_param_reduce_kernel<<<1, 256, 0, st>>>(gpart, grid, gpar, add);
    return cudaGetLastError();
}

template <int KRT>
cudaError_t transpose_launch(const AdjParams& p, const AdjTiles& tl, const int* walk, const int* circ, float* gI, int add,
                             cudaStream_t st) {
    const int SH = tl.th + 2 * p.krad, SW = TR_TW + 2 * p.krad;
    const size_t smem = sizeof(float2) * (size_t)(SH / 2) * ((SW | 1) + 2 * (TR_TW | 1));
    const auto fn = adjoint_transpose_kernel<KRT>;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e) return e;
    for (int f0 = 0; f0 < p.T; f0 += 65535)
        fn<<<dim3(tl.ntx * tl.nty, std::min(65535, p.T - f0)), TR_NT, smem, st>>>(p, tl, walk, circ, gI, f0, add);
    return cudaGetLastError();
}

// `add`: onto the gradient of earlier chunks of peaks.
cudaError_t launch_adjoint_transpose(const AdjParams& p, const AdjTiles& tl, const int* walk, const int* circ, float* gI,
                                     int add, cudaStream_t st) {
    switch (p.krad) {
        case 1: return transpose_launch<1>(p, tl, walk, circ, gI, add, st);
        case 2: return transpose_launch<2>(p, tl, walk, circ, gI, add, st);
        case 3: return transpose_launch<3>(p, tl, walk, circ, gI, add, st);
        case 4: return transpose_launch<4>(p, tl, walk, circ, gI, add, st);
        case 5: return transpose_launch<5>(p, tl, walk, circ, gI, add, st);
        case 6: return transpose_launch<6>(p, tl, walk, circ, gI, add, st);
        case 7: return transpose_launch<7>(p, tl, walk, circ, gI, add, st);
        default: return transpose_launch<0>(p, tl, walk, circ, gI, add, st);
    }
}

}  // namespace gt
