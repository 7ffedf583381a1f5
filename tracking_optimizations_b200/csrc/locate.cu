// locate.cu -- fused bandpass -> grey-dilation local max -> centroid walk
// kernel, one CTA per (frame, TH x TW tile).
//
// Replaces the five WGSL dispatches of the reference
// (shaders/preprocess_rows.wgsl, preprocess_cols.wgsl, centers.wgsl,
// max_rows.wgsl, walk_cols.wgsl, dispatched by execute_gpu.rs:82-88) and the
// host-side dense raster scan (execute_gpu.rs:157-183): the processed plane
// never leaves shared memory, the centroid is evaluated only where a walk
// reads it, and features are emitted as compact records with per-(row, tile
// column) counts from which the finalize kernel restores raster order.
//
// Shared-memory layout of one tile (floats):
//   R   raw pixels, (PH + 2k) x (PW + 2k), zero outside the frame
//   Gr  row-pass Gaussian, (PH + 2k) x PW
//   Br  row-pass boxcar,   (PH + 2k) x PW
//   P   processed,          PH x PW, -inf outside the frame
// with PH = TH + 2*hp, PW = TW + 2*hp, k = smoothing radius.
#include "gt_device.cuh"

namespace gt {

namespace {

struct TileAcc {  // processed plane in shared memory, frame coordinates
    const float* P;
    int py0, px0, PH, PW;
    __device__ bool covers(int u, int v) const {
        return u >= py0 && u < py0 + PH && v >= px0 && v < px0 + PW;
    }
    __device__ float operator()(int u, int v) const { return P[(u - py0) * PW + (v - px0)]; }
};

struct RawAcc {
    const float* R;
    int ry0, rx0, RW;
    __device__ float operator()(int u, int v) const { return R[(u - ry0) * RW + (v - rx0)]; }
};

constexpr int NT = 256;
constexpr int CMAX = 512;  // walk results held in shared memory per round

}  // namespace

__global__ void __launch_bounds__(NT) locate_tiles_kernel(const LocParams p, const MovieBufs b,
                                                          int frame0) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int warp_tot[NT / 32];
    __shared__ int s_total, s_base;
    __shared__ int rowcount[128];
    __shared__ int rowstart[128];

    const int tile = blockIdx.x;
    const int t = frame0 + blockIdx.y;
    const int ti = tile / p.ntx, tj = tile - ti * p.ntx;
    const int ty0 = ti * p.TH, tx0 = tj * p.TW;
    const int TH = min(p.TH, p.H - ty0), TW = p.TW;  // TW fixed for layout
    const int hp = p.hp, kr = p.krad, taps = p.taps;
    const int PH = p.TH + 2 * hp, PW = TW + 2 * hp;
    const int RH = PH + 2 * kr, RW = PW + 2 * kr;
    const int py0 = ty0 - hp, px0 = tx0 - hp;
    const int ry0 = py0 - kr, rx0 = px0 - kr;
    const int H = p.H, W = p.W;
    const bool border = ry0 < 0 || rx0 < 0 || ry0 + RH > H || rx0 + RW > W;

    float* R = sm;
    float* Gr = R + RH * RW;
    float* Br = Gr + RH * PW;
    float* P = Br + RH * PW;
    int* clist = (int*)(P + PH * PW);                 // TH*TW candidate pixels
    float* wy = (float*)(clist + p.TH * TW);           // CMAX walk results
    float* wx = wy + CMAX;
    float* wm = wx + CMAX;
    int* wst = (int*)(wm + CMAX);
    unsigned int* wlp = (unsigned int*)(wst + CMAX);  // last-read pixel (u << 16 | v)
    unsigned int* wfp = wlp + CMAX;                   // final position (u << 16 | v)
    unsigned char* flags = (unsigned char*)(wfp + CMAX);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t fbase = (size_t)t * H * W;

    // ---- A: raw tile (zero outside the frame) ----
    for (int r = warp; r < RH; r += NT / 32) {
        const int fr = ry0 + r;
        for (int c = lane; c < RW; c += 32) {
            const int fc = rx0 + c;
            float val = 0.f;
            if (fr >= 0 && fr < H && fc >= 0 && fc < W) val = load_px(b.frames, p.dtype, fbase + (size_t)fr * W + fc);
            R[r * RW + c] = val;
        }
    }
    if (threadIdx.x < 128) { rowstart[threadIdx.x] = 0x7fffffff; rowcount[threadIdx.x] = 0; }
    __syncthreads();

    // ---- B: row pass (preprocess_rows.wgsl:30-52) ----
    for (int r = warp; r < RH; r += NT / 32) {
        const float* Rr = R + r * RW;
        for (int pc = lane; pc < PW; pc += 32) {
            float gs = 0.f, cs = 0.f;
            if (!border) {
                for (int j = 0; j < taps; ++j) {
                    const float val = Rr[pc + j];
                    gs = fmaf(p.w[j], val, gs);
                    cs = cs + val;
                }
            } else {
                const int fc = px0 + pc;
                for (int j = 0; j < taps; ++j) {
                    gs = fmaf(p.w[j], Rr[pc + j], gs);  // zero outside: exact skip
                    const int cc = clampi(reflect_once(fc + j - kr, W) - rx0, 0, RW - 1);
                    cs = cs + Rr[cc];
                }
            }
            Gr[r * PW + pc] = gs * p.rn;  // preprocess_rows.wgsl:52 gauss_sum / gauss_norm
            Br[r * PW + pc] = cs;
        }
    }
    __syncthreads();

    // ---- C: column pass + clip (preprocess_cols.wgsl:32-60) ----
    for (int pr = warp; pr < PH; pr += NT / 32) {
        const int fr = py0 + pr;
        for (int pc = lane; pc < PW; pc += 32) {
            const int fc = px0 + pc;
            float out = -CUDART_INF_F;
            if (fr >= 0 && fr < H && fc >= 0 && fc < W) {
                float gs = 0.f, cs = 0.f;
                if (!border) {
                    for (int j = 0; j < taps; ++j) {
                        gs = fmaf(p.w[j], Gr[(pr + j) * PW + pc], gs);
                        cs = cs + Br[(pr + j) * PW + pc];
                    }
                } else {
                    for (int j = 0; j < taps; ++j) {
                        gs = fmaf(p.w[j], Gr[(pr + j) * PW + pc], gs);  // zero rows outside
                        const int rr = clampi(reflect_once(fr + j - kr, H) - ry0, 0, RH - 1);
                        cs = cs + Br[rr * PW + pc];
                    }
                }
                // preprocess_cols.wgsl:54, contracted: fma(-cs, 1/k^2, gs / norm)
                const float res = fmaf(-cs, p.rkk, gs * p.rn);
                out = res < 0.f ? 0.f : res;
            }
            P[pr * PW + pc] = out;
        }
    }
    __syncthreads();

    // ---- D: row max over the dilation window (max_rows.wgsl:10-28) ----
    float* RM = Gr;  // PH x TW
    for (int pr = warp; pr < PH; pr += NT / 32) {
        for (int tc = lane; tc < TW; tc += 32) {
            const float* Pr = P + pr * PW + tc + hp;
            float m = Pr[0];
            for (int j = 0; j < p.D; ++j) m = fmaxf(m, Pr[j - p.o]);
            RM[pr * TW + tc] = m;
        }
    }
    __syncthreads();

    // ---- E: non-strict local max (walk_cols.wgsl:19-36) ----
    const int npx = p.TH * TW;
    for (int q = threadIdx.x; q < npx; q += NT) {
        const int tr = q / TW, tc = q - tr * TW;
        unsigned char f = 0;
        if (tr < TH && tx0 + tc < W) {
            const float center = P[(tr + hp) * PW + tc + hp];
            bool ismax = true;
            for (int i = 0; i < p.D; ++i)
                if (RM[(tr + hp - p.o + i) * TW + tc] > center) { ismax = false; break; }
            if (ismax && !(p.zero_skip && center == 0.f)) f = 1;
        }
        flags[q] = f;
    }
    __syncthreads();
    // compaction in raster order: thread owns a contiguous chunk
    const int chunk = (npx + NT - 1) / NT;
    const int q0 = threadIdx.x * chunk;
    int mine = 0;
    for (int q = q0; q < min(q0 + chunk, npx); ++q) mine += flags[q];
    int pos = block_excl_scan<NT>(mine, warp_tot, &s_total);
    const int ncand = s_total;
    for (int q = q0; q < min(q0 + chunk, npx); ++q)
        if (flags[q]) clist[pos++] = q;
    __syncthreads();

    // ---- F/G: walks and emission, in raster-ordered rounds of CMAX ----
    TileAcc acc{P, py0, px0, PH, PW};
    RawAcc racc{R, ry0, rx0, RW};
    int emitted = 0;  // emitted records of this tile before the round
    for (int r0 = 0; r0 < ncand; r0 += CMAX) {
        const int nr = min(CMAX, ncand - r0);
        for (int c = threadIdx.x; c < nr; c += NT) {
            const int q = clist[r0 + c];
            const int u0 = ty0 + q / TW, v0 = tx0 + q % TW;
            int st;
            float y = 0.f, x = 0.f, m = 0.f;
            unsigned int lp = 0, fp = 0;
            if (p.max_iter <= 0) {
                st = CAND_PENDING;  // mass read at pixel 0: resolved by the fallback kernel
            } else {
                WalkOut wo = walk_from(p, acc, u0, v0);
                if (!wo.ok) {
                    st = CAND_PENDING;
                } else {
                    y = wo.y; x = wo.x; m = wo.mass;
                    st = (m > p.minmass && m != 0.f) ? CAND_EMIT : CAND_REJECT;
                    lp = ((unsigned)wo.ul << 16) | (unsigned)wo.vl;
                    fp = ((unsigned)wo.up << 16) | (unsigned)wo.vp;
                }
            }
            wy[c] = y; wx[c] = x; wm[c] = m; wst[c] = st; wlp[c] = lp; wfp[c] = fp;
        }
        __syncthreads();
        const int cchunk = (nr + NT - 1) / NT;
        const int c0 = threadIdx.x * cchunk, c1 = min(c0 + cchunk, nr);
        int ne = 0;
        for (int c = c0; c < c1; ++c) ne += (wst[c] != CAND_REJECT);
        int epos = block_excl_scan<NT>(ne, warp_tot, &s_total);
        const int nemit = s_total;
        if (threadIdx.x == 0) {
            int base = 0;
            if (nemit > 0) base = atomicAdd(b.fcount + t, nemit);
            if (base + nemit > b.cap_c) { atomicOr(b.err, ERR_CAND_OVERFLOW); base = -1; }
            s_base = base;
        }
        {
            int e = emitted + epos;
            for (int c = c0; c < c1; ++c) {
                if (wst[c] == CAND_REJECT) continue;
                const int tr = clist[r0 + c] / TW;
                atomicMin(&rowstart[tr], e);
                atomicAdd(&rowcount[tr], 1);
                ++e;
            }
        }
        __syncthreads();
        const int base = s_base;
        for (int c = c0; c < c1; ++c) {
            if (wst[c] == CAND_REJECT) continue;
            const int q = clist[r0 + c];
            const int tr = q / TW;
            const int u0 = ty0 + tr, v0 = tx0 + (q - tr * TW);
            Cand rec;
            rec.u = u0; rec.v = v0;
            rec.y = wy[c]; rec.x = wx[c]; rec.mass = wm[c];
            rec.rowrank = emitted + epos - rowstart[tr];
            rec.state = wst[c];
            rec.rg_sum = rec.eccn = rec.mid = rec.signal = 0.f;
            rec.g_rg = rec.g_raw = rec.g_sig = rec.g_ecc = 0.f;
            rec.ul = (int)(wlp[c] >> 16); rec.vl = (int)(wlp[c] & 0xffffu);
            rec.up = (int)(wfp[c] >> 16); rec.vp = (int)(wfp[c] & 0xffffu);
            rec.pad = 0;
            if (p.cpu_processed) cpu_features(p, b, acc, u0, v0, rec);
            if (p.characterize) gpu_features(p, b, acc, racc, u0, v0, rec);
            if (base >= 0) {
                const int slot = base + epos;
                b.cand[(size_t)t * b.cap_c + slot] = rec;
                if (rec.state == CAND_PENDING) {
                    const int k = atomicAdd(b.npend, 1);
                    b.pend[k] = t * b.cap_c + slot;
                }
            }
            ++epos;
        }
        emitted += nemit;
        __syncthreads();
    }
    // per-(row, tile column) record counts
    for (int r = threadIdx.x; r < TH; r += NT)
        b.rowcnt[((size_t)t * H + ty0 + r) * p.ntx + tj] = rowcount[r];
}

// Rows copied to a pitch of whole 16-byte groups, so that the tile copies (TMA)
// take frames of any width: 16 bytes per item, as 32-bit words where the row
// starts on one, else the words between the first and the last pixel, shifted.
// Bound by memory.  Locate of 300 uint16 frames of 507 x 517, diameter 7: 0.652
// ms with tiles read pixel by pixel, 0.536 with the copy (0.462 for 512 x 520
// without one).
template <class PX>
__global__ void __launch_bounds__(256) repack_kernel(const PX* __restrict__ frames, long long rows, int W, int groups,
                                                     uint4* __restrict__ out) {
    constexpr int VP = 16 / sizeof(PX);
    const long long n = rows * groups;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const long long r = i / groups;
        const int c = (int)(i - r * groups) * VP;
        const PX* src = frames + r * W + c;
        uint4 o;
        if (c + VP <= W) {
            if (sizeof(PX) == 4 || ((uintptr_t)src & 2) == 0) {
                const unsigned* w = (const unsigned*)src;
                o = make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
            } else {
                const unsigned* w = (const unsigned*)(src + 1);
                const unsigned a = (unsigned)__ldg(src), z = (unsigned)__ldg(src + VP - 1);
                const unsigned w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
                o = make_uint4(a | w0 << 16, __funnelshift_l(w0, w1, 16), __funnelshift_l(w1, w2, 16), w2 >> 16 | z << 16);
            }
        } else {
            __align__(16) PX v[VP];
#pragma unroll
            for (int q = 0; q < VP; ++q) v[q] = c + q < W ? __ldg(src + q) : (PX)0;
            o = *(const uint4*)v;
        }
        out[i] = o;
    }
}

cudaError_t launch_repack(const void* frames, int dtype, int frame0, int nf, int H, int W, int pitch, void* out,
                          int num_sms, cudaStream_t st) {
    const long long rows = (long long)nf * H, first = (long long)frame0 * H * W;
    const int groups = pitch / (dtype == 0 ? 8 : 4);
    const int grid = (int)std::min<long long>((rows * groups + 255) / 256, (long long)num_sms * 32);
    if (dtype == 0)
        repack_kernel<<<grid, 256, 0, st>>>((const unsigned short*)frames + first, rows, W, groups, (uint4*)out);
    else
        repack_kernel<<<grid, 256, 0, st>>>((const float*)frames + first, rows, W, groups, (uint4*)out);
    return cudaGetLastError();
}

// Walks of the records that locate left pending (the walk left the tile halo,
// a crowded tile, max_iterations == 0): the processed values that a walk can
// read are recomputed from the frame, with the same arithmetic, into a
// shared-memory window of n = 2 win + 1 pixels a side.

// processed value at one pixel, straight from the frame (row pass then column
// pass in shader order)
__device__ float processed_at(const LocParams& p, const void* frames, size_t fbase, int u, int v) {
    const int kr = p.krad, H = p.H, W = p.W;
    float gs = 0.f, cs = 0.f;
    for (int i = -kr; i <= kr; ++i) {
        int pu = u + i;
        bool dg = true;
        if (pu < 0) { pu = -pu - 1; dg = false; }
        else if (pu >= H) { pu = 2 * H - pu - 1; dg = false; }
        // row pass at (pu, v)
        float rg = 0.f, rb = 0.f;
        for (int j = -kr; j <= kr; ++j) {
            int pv = v + j;
            bool dgv = true;
            if (pv < 0) { pv = -pv - 1; dgv = false; }
            else if (pv >= W) { pv = 2 * W - pv - 1; dgv = false; }
            const float val = load_px(frames, p.dtype, fbase + (size_t)pu * W + pv);
            if (dgv) rg = fmaf(p.w[j + kr], val, rg);
            rb = rb + val;
        }
        const float tg = rg * p.rn;
        if (dg) gs = fmaf(p.w[i + kr], tg, gs);
        cs = cs + rb;
    }
    const float res = fmaf(-cs, p.rkk, gs * p.rn);
    return res < 0.f ? 0.f : res;
}

namespace {
constexpr int FB_NT = 256;

// Shared memory of a block, in floats: the window, raw pixels and row sums of
// a chunk of its rows, and the centroid circle in the order of its sums (pixel
// offsets, coordinates, and the pixels at the walk's position).
struct FbPlan {
    int n;     // window side
    int rows;  // window rows filled at a time; 0: each pixel by itself
    int kp;    // circle pixels, rounded up to 4
};

__host__ __device__ constexpr int up4(int x) { return (x + 3) / 4 * 4; }
__host__ __device__ inline int fb_raw(const FbPlan& f) { return up4(f.n * f.n) + 4 * f.kp; }  // ints before the chunk

// The n x n window at (y0, x0) in two passes like the tiles': a chunk of
// output rows at a time, the raw rows that it reads (I, reflected at the
// frame's edges), their row sums (G, B), then the columns.  Window pixels
// outside the frame are 0 (no walk reads them).
__device__ __forceinline__ void fill_window(const LocParams& p, const void* frames, size_t fbase, int y0, int x0, int n,
                                            int rows, float* P, float* chunk) {
    const int kr = p.krad, H = p.H, W = p.W, m = n + 2 * kr;
    float* I = chunk;
    float* G = I + (rows + 2 * kr) * m;
    float* B = G + (rows + 2 * kr) * n;
    for (int r0 = 0; r0 < n; r0 += rows) {
        const int nr = min(rows, n - r0), nin = nr + 2 * kr;
#pragma unroll 4
        for (int q = threadIdx.x; q < nin * m; q += FB_NT) {
            const int r = q / m;
            int pu = y0 + r0 - kr + r, pv = x0 - kr + q - r * m;
            if (pu < 0) pu = -pu - 1;
            else if (pu >= H) pu = 2 * H - pu - 1;
            if (pv < 0) pv = -pv - 1;
            else if (pv >= W) pv = 2 * W - pv - 1;
            const bool in = pu >= 0 && pu < H && pv >= 0 && pv < W;
            I[q] = in ? load_px(frames, p.dtype, fbase + (size_t)pu * W + pv) : 0.f;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < nin * n; q += FB_NT) {
            const int r = q / n, v = x0 + q - r * n;
            const float* in = I + r * m + (q - r * n);
            float rg = 0.f, rb = 0.f;
#pragma unroll 5
            for (int j = 0; j <= 2 * kr; ++j) {
                const int c = v + j - kr;
                if (c >= 0 && c < W) rg = fmaf(p.w[j], in[j], rg);  // the Gaussian pads with 0
                rb = rb + in[j];
            }
            G[q] = rg * p.rn;
            B[q] = rb;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < nr * n; q += FB_NT) {
            const int r = q / n, u = y0 + r0 + r, v = x0 + q - r * n;
            float gs = 0.f, cs = 0.f;
#pragma unroll 5
            for (int i = 0; i <= 2 * kr; ++i) {
                const int c = u + i - kr;
                if (c >= 0 && c < H) gs = fmaf(p.w[i], G[q + i * n], gs);
                cs = cs + B[q + i * n];
            }
            const float res = fmaf(-cs, p.rkk, gs * p.rn);
            P[r0 * n + q] = u < 0 || u >= H || v < 0 || v >= W || res < 0.f ? 0.f : res;
        }
        __syncthreads();
    }
}

// walk_from by a warp: its lanes fetch the circle's pixels, then lanes 0, 1
// and 2 run the three sums of the centroid (row offset, column offset, mass),
// each in the shader's order (data * 1 is added exactly; a sum that starts at
// +0 is never -0, so adding the padding's zeros changes nothing).
__device__ __forceinline__ WalkOut walk_window(const LocParams& p, const float* P, int y0, int x0, int n, int kp,
                                               const int* off, const float* cx, const float* cy, float* data, int u,
                                               int v) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, b = p.border, rint = p.rint_c;
    const float4* coef = (const float4*)(lane == 0 ? cx : cy);
    const float4* d4 = (const float4*)data;
    WalkOut o;
    o.ul = 0; o.vl = 0;  // WGSL zero-initialised idx
    float c0 = 0.f, c1 = 0.f, m = 0.f;
    for (int it = 0; it < p.max_iter; ++it) {
        if (u - b < 0 || u + b >= p.H || v - b < 0 || v + b >= p.W) {
            c0 = c1 = m = 0.f;
        } else {
            const int r0 = u - y0, q0 = v - x0;
            if (r0 < rint || r0 + rint >= n || q0 < rint || q0 + rint >= n) {
                o.ok = 0; o.y = o.x = o.mass = 0.f;
                return o;
            }
            const float* at = P + r0 * n + q0;
            __syncwarp();
#pragma unroll 4
            for (int q = lane; q < kp; q += 32) data[q] = off[q] == INT_MIN ? 0.f : at[off[q]];
            __syncwarp();
            float acc = 0.f;
#pragma unroll 4
            for (int q = 0; q < kp / 4; ++q) {
                const float4 d = d4[q];
                float4 c = coef[q];
                if (lane >= 2) c = make_float4(1.f, 1.f, 1.f, 1.f);
                acc = fmaf(d.x, c.x, acc);
                acc = fmaf(d.y, c.y, acc);
                acc = fmaf(d.z, c.z, acc);
                acc = fmaf(d.w, c.w, acc);
            }
            const float a0 = __shfl_sync(full, acc, 0), a1 = __shfl_sync(full, acc, 1);
            m = __shfl_sync(full, acc, 2);
            c0 = gpu_div(a0, m);  // centers.wgsl:82-83
            c1 = gpu_div(a1, m);
        }
        o.ul = u; o.vl = v;
        bool changed = false;
        if (c0 > p.thr && u < p.H - 1) { u += 1; changed = true; }
        else if (c0 < -p.thr && u > 0) { u -= 1; changed = true; }
        if (c1 > p.thr && v < p.W - 1) { v += 1; changed = true; }
        else if (c1 < -p.thr && v > 0) { v -= 1; changed = true; }
        if (!changed) break;
    }
    o.y = (float)u + c0;
    o.x = (float)v + c1;
    o.mass = m;
    o.ok = 1;
    o.up = u; o.vp = v;
    return o;
}
}  // namespace

// A block walks one record after the other.  What bounds it: the latency of a
// single walk (a few dozen records a movie).  Each window pixel straight from
// the frame (krad^2 taps) and the walk by one thread took 177 us for 24
// records of diameter 15; the passes and the three lanes take 25 us.
__global__ void __launch_bounds__(FB_NT) fallback_walk_kernel(const LocParams p, const MovieBufs b, const FbPlan f,
                                                              const int* pbeg) {
    extern __shared__ __align__(16) float wsm[];
    const int npend = *b.npend;
    const int k0 = (pbeg ? *pbeg : 0) + blockIdx.x;  // entries from *pbeg on: those of the frames located since
    if (k0 >= npend) return;
    const int n = f.n, rint = p.rint_c;
    int* off = (int*)(wsm + up4(n * n));
    float* cx = (float*)off + f.kp;
    float* cy = cx + f.kp;
    float* data = cy + f.kp;
    // the circle x^2 + y^2 <= r^2, rows then columns (a thread per row)
    for (int i = (int)threadIdx.x - rint; i <= rint; i += FB_NT) {
        auto half = [&](int x) { return (int)sqrtf((float)(rint * rint - x * x)); };
        int at = 0;
        for (int x = -rint; x < i; ++x) at += 2 * half(x) + 1;
        for (int j = -half(i); j <= half(i); ++j, ++at) {
            off[at] = i * n + j;
            cx[at] = (float)i;
            cy[at] = (float)j;
        }
        if (i == rint)
            for (; at < f.kp; ++at) {
                off[at] = INT_MIN;
                cx[at] = cy[at] = 0.f;
            }
    }
    for (int k = k0; k < npend; k += gridDim.x) {
        const int code = b.pend[k];
        const int t = code / b.cap_c;
        Cand* rec = b.cand + code;
        const int u0 = rec->u, v0 = rec->v;
        const size_t fbase = (size_t)t * p.H * p.W;
        const int y0 = u0 - n / 2, x0 = v0 - n / 2;
        __syncthreads();  // the last record's walk is done with the window
        if (p.max_iter > 0 && f.rows > 0) {
            fill_window(p, b.frames, fbase, y0, x0, n, f.rows, wsm, wsm + fb_raw(f));
        } else if (p.max_iter > 0) {
            for (int q = threadIdx.x; q < n * n; q += FB_NT) {
                const int u = y0 + q / n, v = x0 + q % n;
                wsm[q] = u >= 0 && u < p.H && v >= 0 && v < p.W ? processed_at(p, b.frames, fbase, u, v) : 0.f;
            }
            __syncthreads();
        }
        if (threadIdx.x < 32) {
            float y, x, m;
            bool ok = true;
            int ul = 0, vl = 0, up = u0, vp = v0;
            if (p.max_iter <= 0) {
                // walk_cols.wgsl:69-73 with no iteration: offset (0, 0) and the
                // mass of pixel 0, which is interior only when d/2 == 0 (its
                // circle is then the pixel itself)
                y = (float)u0; x = (float)v0;
                m = (p.border == 0) ? processed_at(p, b.frames, fbase, 0, 0) : 0.f;
            } else {
                const WalkOut wo = walk_window(p, wsm, y0, x0, n, f.kp, off, cx, cy, data, u0, v0);
                ok = wo.ok != 0;
                y = wo.y; x = wo.x; m = wo.mass;
                ul = wo.ul; vl = wo.vl; up = wo.up; vp = wo.vp;
            }
            if (threadIdx.x == 0) {
                if (!ok) {  // window too small for this walk: report, never guess
                    atomicOr(b.err, ERR_SCRATCH_OVERFLOW);
                    rec->state = CAND_REJECT;
                } else {
                    rec->y = y; rec->x = x; rec->mass = m;
                    rec->ul = ul; rec->vl = vl; rec->up = up; rec->vp = vp;
                    rec->state = (m > p.minmass && m != 0.f) ? CAND_EMIT : CAND_REJECT;
                }
            }
        }
    }
}

// Window rows filled at a time: all of them where the rows that they read fit
// beside the window (diameter 31 up to 36 iterations), else as many as do.
// None fit beside the largest windows with wide smoothing (diameter 31 from 81
// iterations on): every pixel is then computed by itself.
cudaError_t launch_fallback(const LocParams& p, const MovieBufs& b, int win, const int* pbeg, int grid, cudaStream_t st) {
    cudaError_t e = allow_shared<fallback_walk_kernel>();
    if (e != cudaSuccess) return e;
    FbPlan f{2 * win + 1, 0, 0};
    for (int i = -p.rint_c; i <= p.rint_c; ++i)
        for (int j = -p.rint_c; j <= p.rint_c; ++j) f.kp += i * i + j * j <= p.rint_c * p.rint_c;
    f.kp = up4(f.kp);
    const int row = 3 * f.n + 2 * p.krad;  // floats of a raw row and its sums
    f.rows = std::max(0, std::min(f.n, (227 * 1024 / 4 - fb_raw(f)) / row - 2 * p.krad));
    const size_t smem = sizeof(float) * ((size_t)fb_raw(f) + (f.rows ? (size_t)(f.rows + 2 * p.krad) * row : 0));
    fallback_walk_kernel<<<grid, FB_NT, smem, st>>>(p, b, f, pbeg);
    return cudaGetLastError();
}

}  // namespace gt
