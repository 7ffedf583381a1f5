// gt_api.cu -- host side of libgt: parameter derivation, workspace, launch
// sequence and the extern "C" entry points declared in include/gt.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <array>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <climits>
#include <cstring>
#include <string>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include <map>

#include "gt.h"
#include "gt_internal.cuh"
#include "hostcopy.h"
#include "ingest.h"
#include "traj.h"

namespace gt {
__global__ void locate_tiles_kernel(const LocParams p, const MovieBufs b, int frame0);
cudaError_t launch_fallback(const LocParams& p, const MovieBufs& b, int win, const int* pbeg, int grid, cudaStream_t st);
cudaError_t launch_finalize(const LocParams& p, const MovieBufs& b, float sep, int link_grid, int frame0, int nf,
                            size_t smem, cudaStream_t st);
cudaError_t link_blocks_per_sm(bool multi, int* per_sm);
cudaError_t launch_link(const LinkBufs& L, int max_passes, int* passes, unsigned long long* stat, int grid,
                        cudaStream_t st);
cudaError_t launch_link_multi(const LinkBufs* d_L, int nm, int max_passes, int* passes, unsigned long long* stat,
                              int grid, cudaStream_t st);
__global__ void scan_frames_kernel(const int* in, int* out, int n);
__global__ void newid_kernel(const int* newrank, const int* newbase, const int* off, const int* npart,
                             int* newid, int T);
cudaError_t launch_assemble(const AsmArgs& a, int num_sms, cudaStream_t st);
__global__ void grid_kernel(const float* py, const float* px, const int* npart, int cap_p, int G,
                            int ncy, int ncx, int* gstart, int* gidx, float2* gpos);
int fast_supported(int kr, int dd, int rc, int diameter, int dtype);
int fast_rows(int kr, int dd, int rc, int dtype, int th);
cudaError_t launch_locate_fast(int kr, int dd, int rc, int th, dim3 grid, cudaStream_t st, const LocParams& p,
                               const MovieBufs& b, const TileSource& src, int frame0, int* used_tma);
cudaError_t launch_repack(const void* frames, int dtype, int frame0, int nf, int H, int W, int pitch, void* out,
                          int num_sms, cudaStream_t st);
void gauss_taps(int smoothing_size, float noise_size, int normalized, float* w, float* norm, float* rn);
cudaError_t launch_adjoint_particles(int mode, const AdjParams& p, const float* frames, const int* walk, long long n,
                                     const int* circ, const float* grad, float* yxm, const AdjTiles& tl, double* gpar,
                                     double* gpart, int* err, int add, int num_sms, cudaStream_t st);
void adjoint_tiles(const AdjParams& p, AdjTiles* tl);
int adjoint_particle_blocks_max(int num_sms);
cudaError_t launch_adjoint_transpose(const AdjParams& p, const AdjTiles& tl, const int* walk, const int* circ, float* gI,
                                     int add, cudaStream_t st);
int traj_filter_stubs(const int64_t* h_ids, int64_t n, int64_t threshold, uint8_t* h_keep, int64_t* h_count,
                      int64_t* nkept, TrajMem& M, cudaStream_t st, int num_sms, std::string* msg);
int traj_steps(const int64_t* h_ids, const float* h_x, const float* h_y, int64_t n, float mppf, float* h_xs,
               float* h_ys, double* h_xstep, double* h_ystep, double* h_len, int64_t* h_order, TrajMem& M,
               cudaStream_t st, int num_sms, std::string* msg);
int traj_imsd(const int64_t* h_ids, const int64_t* h_frames, const float* h_x, const float* h_y, int64_t n,
              float mppf, int64_t max_lagtime, float* (*alloc)(size_t), float** out, int64_t* nout, float* ms_msd,
              TrajMem& M, cudaStream_t st, int num_sms, std::string* msg);

int table_load(const float* h_rows, int n, int ncols, TrajMem& M, cudaStream_t st, int num_sms, LinkTable* t,
               std::string* msg);
cudaError_t table_slabs(const LinkTable& t, int cap, float* py, float* px, int* npart, int num_sms, cudaStream_t st);
cudaError_t table_ids(const LinkTable& t, const int* root, const int* newid, int num_sms, cudaStream_t st);

// preprocess_rows.wgsl:44-45: taps exp(-i^2 / (2 * noise_size)) for
// i = -k/2..k/2 and their running sum; the passes multiply by the
// reciprocal of that sum (a shader division).  With `normalized` the taps
// are divided by their sum on the host instead and the passes multiply by 1
// (kernels.rs:86-97 `gauss_1d` and `normalize`, the form in which the
// reference dumped its mass plane).
void gauss_taps(int smoothing_size, float noise_size, int normalized, float* w, float* norm, float* rn) {
    const int kr = smoothing_size / 2;
    float s = 0.0f;
    for (int i = -kr; i <= kr; ++i) {
        const float x = (float)i;
        const float g = std::exp(-x * x / (2.0f * noise_size));
        w[i + kr] = g;
        s = s + g;
    }
    *norm = s;
    if (normalized) {
        for (int i = 0; i < 2 * kr + 1; ++i) w[i] = w[i] / s;
        *rn = 1.0f;
    } else {
        *rn = 1.0f / s;
    }
}
}  // namespace gt

using namespace gt;

constexpr int BATCH_STREAMS = 8;

struct gt_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    char* arena = nullptr;
    size_t arena_size = 0;
    gt_stats stats{};
    int stage_times = 0;  // 1: the stage times of stats are still in ev[0..4]
    int num_sms = 148;
    cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    int normalized_taps = 0;          // Gaussian taps divided by their sum on the host
    long long subnet_budget = 1LL << 26;  // option trials per linking subnetwork
    int withhold_tma = 0;             // test switch of the bounded tile-copy wait
    int force_generic = 0;            // always use locate_tiles_kernel
    int fast_tile_rows = 64;          // output tile height of the fast kernel (32 or 64)
    int tiles_per_cta = 0;            // fast kernel: tiles per CTA (0 = chosen per launch)
    // batched path (gt_batch_many_device)
    std::map<std::array<int, 6>, int> tile_rows;  // autotuned tile rows per (H, W, krad, D, rc, dtype)
    std::string batch_key;            // inputs of the cached graph
    cudaGraphExec_t batch_exec = nullptr;
    cudaStream_t side[BATCH_STREAMS] = {};
    cudaEvent_t bev[2 + 2 * BATCH_STREAMS] = {};  // fork/join events
    int* h_status = nullptr;          // pinned: 8 ints per movie
    int* h_stage = nullptr;           // pinned: one call's statistics, read back in one go
    int link_grid[2] = {0, 0};        // resident blocks of the one-movie and the batched linker (queried once)
    size_t h_stage_n = 0;
    uint16_t* h_frames = nullptr;     // pinned: decoded file frames
    size_t h_frames_n = 0;
    size_t h_status_n = 0;
    int tune_disabled = 0;
    int batch_cap_div = 64;           // first candidate capacity of batched movies: H*W / this
    int short_memory = 0;             // test switch: batches start with the capacities of short memory
    cudaStream_t copy_stream = nullptr;  // host->device frame chunks
    HostCopy hc;                         // pageable host arrays
    TrajMem traj;                        // scratch of the trajectory calls
    cudaEvent_t cev[9] = {};
    cudaEvent_t lev = nullptr;        // work pending on the legacy default stream (call_stream)
};

namespace {

constexpr int LOC_TH = 32;
constexpr int LOC_TW = 64;
constexpr int LOC_CMAX = 512;
constexpr int FB_WIN_MAX = 100;
// Frames repacked at a time: few enough to be read back from L2 (126 MB), many
// enough to fill the locate launch (300 frames of 507 x 517: 32 MB 0.577 ms, 64
// 0.537, 128 0.540).
constexpr long long REPACK_BYTES = 64LL << 20;
constexpr long long SUBNET_BUDGET = 1LL << 26;  // option trials per subnet
constexpr int LINK_WINDOWS = 16;  // upload chunks of the host-frames path, at most
constexpr int STATUS_LSTAT = 8 + LINK_WINDOWS, STATUS_INTS = STATUS_LSTAT + 2 * 12 + 4 * NCTR;
constexpr int LINK_RUNS = 4;      // linker launches over them, at most

struct Resolved {
    // lib.rs:77-91 defaults
    uint32_t diameter;
    float minmass;
    uint32_t separation;
    float noise_size;
    uint32_t smoothing_size;
    uint32_t max_iterations;
    int characterize;
    int cpu_processed;
    int has_search_range;
    float search_range;
    uint32_t memory;
    int has_sig, has_bg;
    float sig_radius, bg_radius, gap_radius;
    int normalized_taps;  // context option, not a reference parameter
};

int resolve(const gt_params* p, Resolved* r, std::string* msg) {
    // lib.rs:73-74 not_implemented!(maxsize, threshold, invert, percentile, topn, preprocess)
    const char* ni = nullptr;
    if (p->has_maxsize) ni = "maxsize";
    else if (p->has_threshold) ni = "threshold";
    else if (p->has_invert) ni = "invert";
    else if (p->has_percentile) ni = "percentile";
    else if (p->has_topn) ni = "topn";
    else if (p->has_preprocess) ni = "preprocess";
    if (ni) { *msg = std::string(ni) + " is not implemented"; return GT_ERR_UNSUPPORTED; }
    r->diameter = p->diameter;
    r->minmass = p->has_minmass ? p->minmass : 0.0f;
    r->separation = p->has_separation ? p->separation : p->diameter + 1;
    r->noise_size = p->has_noise_size ? p->noise_size : 1.0f;
    r->smoothing_size = p->has_smoothing_size ? p->smoothing_size : p->diameter;
    r->max_iterations = p->has_max_iterations ? p->max_iterations : 10;
    r->characterize = p->has_characterize ? (p->characterize != 0) : 0;
    r->cpu_processed = p->has_cpu_processed ? (p->cpu_processed != 0) : 0;
    r->has_search_range = p->has_search_range;
    r->search_range = p->search_range;
    r->memory = p->has_memory ? p->memory : 0;  // Linker::new(range, memory.unwrap_or(0))
    r->has_sig = p->has_sig_radius;
    r->sig_radius = p->sig_radius;
    r->has_bg = p->has_bg_radius;
    r->bg_radius = p->bg_radius;
    r->gap_radius = p->has_gap_radius ? p->gap_radius : 0.0f;  // lib.rs:91
    r->normalized_taps = 0;
    if (r->has_bg && !r->has_sig) {
        // execute_gpu.rs:301-333 only gathers raw pixels when sig_radius is
        // set; the reference then fails reshaping its output.
        *msg = "bg_radius requires sig_radius";
        return GT_ERR_ARG;
    }
    if (r->smoothing_size < 1 || r->smoothing_size / 2 * 2 + 1 > GT_MAX_TAPS) {
        *msg = "smoothing_size must be in [1, 63]";
        return GT_ERR_ARG;
    }
    if (r->diameter > 63) { *msg = "diameter must be <= 63"; return GT_ERR_ARG; }
    if (r->separation > 4096) { *msg = "separation must be <= 4096"; return GT_ERR_ARG; }
    if (r->has_search_range && !(r->search_range > 0.0f && r->search_range < 4096.0f)) {
        *msg = "search_range must be in (0, 4096)";
        return GT_ERR_ARG;
    }
    if (r->memory > 1000) { *msg = "memory must be <= 1000"; return GT_ERR_ARG; }
    return GT_OK;
}

void column_list(const Resolved& r, std::vector<std::string>& names, std::vector<std::string>& types) {
    // execute_gpu.rs:197-226
    names = {"frame", "mass", "y", "x"};
    types = {"int", "float", "float", "float"};
    if (r.has_search_range) { names.push_back("particle"); types.push_back("int"); }
    if (r.cpu_processed) for (auto n : {"Rg", "ecc", "signal"}) { names.push_back(n); types.push_back("float"); }
    if (r.has_sig) { names.push_back("raw_mass"); types.push_back("float"); }
    if (r.has_bg) for (auto n : {"raw_bg_median", "raw_mass_corrected"}) { names.push_back(n); types.push_back("float"); }
    if (r.characterize)
        for (auto n : {"Rg_gpu", "raw_mass_gpu", "signal_gpu", "ecc_gpu"}) { names.push_back(n); types.push_back("float"); }
}

// gpu_setup.rs:48 dilation and max_rows.wgsl:17 offset
void dilation(uint32_t sep, int* D, int* o) {
    float v = (2.0f * (float)sep) / std::sqrt(2.0f);
    unsigned d = v <= 0.0f ? 0u : (unsigned)v;
    float half = (float)(int)d / 2.0f - 0.5f;
    *D = (int)d;
    *o = (int)half;
}

struct Plan {
    int T = 0, H = 0, W = 0, dtype = 0;
    Resolved r{};
    LocParams lp{};
    float sep = 0.f;
    int link = 0;
    int cap_c = 0, cap_p = 0;
    int G = 8, ncx = 1, ncy = 1;      // separation grid
    int LG = 8, lncx = 1, lncy = 1;  // linker's grid
    // linker scratch for components beyond a block's own arrays
    int nslot = 0, big_d = 1, big_s = 1, big_e = 1;
    size_t smem_loc = 0, smem_fin = 0;
    int fb_win = 0;
    int fast = 0;
    int repack = 0, pitch = 0;  // frames of a chunk repacked for the tile copies (0: as given), their row pitch
    int fast_th = 32;
    std::vector<float> char_tab, gchar_tab;
    std::vector<int> char_off, sig_off, bg_off;
    std::vector<int> tables;  // the five one after the other, as they are uploaded
    std::vector<std::string> names, types;
};

void circle_tables(int R, std::vector<float>& tab, std::vector<int>* off, int stride3) {
    // kernels.rs:134-150, 169-206: i outer (row), j inner (column)
    for (int i = -R; i <= R; ++i)
        for (int j = -R; j <= R; ++j)
            if (i * i + j * j <= R * R) {
                float th = std::atan2((float)j, (float)i);
                if (stride3) tab.push_back((float)(i * i + j * j));
                tab.push_back(std::sin(2.0f * th));
                tab.push_back(std::cos(2.0f * th));
                if (off) { off->push_back(i); off->push_back(j); }
            }
}

void circle_inds_f(float radius, std::vector<int>& off) {
    // kernels.rs:134-150 with a float radius
    int rb = (int)std::ceil(radius);
    float r2 = radius * radius;
    for (int i = -rb; i <= rb; ++i)
        for (int j = -rb; j <= rb; ++j)
            if ((float)(i * i + j * j) <= r2) { off.push_back(i); off.push_back(j); }
}

void annulus_inds_f(float outer, float inner, std::vector<int>& off) {
    // kernels.rs:152-167
    int b = (int)std::ceil(outer);
    float or2 = outer * outer, ir2 = inner * inner;
    for (int i = -b; i <= b; ++i)
        for (int j = -b; j <= b; ++j) {
            float r2 = (float)(i * i + j * j);
            if (r2 <= or2 && r2 >= ir2) { off.push_back(i); off.push_back(j); }
        }
}

size_t big_ints(const Plan& P) { return comp_bytes(P.big_d, P.big_s, P.big_e, sizeof(int)) / sizeof(int); }

// Scratch slots of the linker's largest components in T frames, a block's each:
// 16 a pair of frames, as many as fit 256 MB (64 in any case), and a block's
// on every SM four times over at most.
int big_slots(const Plan& P, long long T) {
    const size_t fit = std::max<size_t>(64, std::min<size_t>(4 * 148, ((size_t)64 << 20) / big_ints(P)));
    return (int)std::min<long long>(fit, 16 * (T - 1));
}

// Their sizes: room for 4096 destinations, 8192 sources and 32768 edges (a
// component that the search budget lets finish is far smaller), four times
// more per capacity retry.
void link_scratch(Plan* pl, int scale) {
    Plan& P = *pl;
    P.big_d = (int)std::min<long long>(4096LL * scale, P.cap_p);
    P.big_s = (int)std::min<long long>(8192LL * scale, (long long)P.cap_p * (P.r.memory + 1));
    P.big_e = (int)std::min<long long>(32768LL * scale, (long long)P.big_d * P.big_s);
    P.nslot = P.link ? big_slots(P, P.T) : 0;
}

// The specialised locate kernel's tile height, 32 or fast_rows: nothing in the
// workspace depends on it.
void set_tile_rows(Plan* pl, int rows) {
    LocParams& lp = pl->lp;
    pl->fast_th = fast_rows(lp.krad, lp.D, lp.rint_c, pl->dtype, rows);
    lp.TH = pl->fast_th;
    lp.nty = (lp.H + lp.TH - 1) / lp.TH;
}

int make_plan(const Resolved& r, int T, int H, int W, int dtype, int scale, int num_sms, Plan* pl,
              std::string* msg, int force_generic_flag = 0, int fast_tile_rows = 32, int cap_div = 64) {
    Plan& P = *pl;
    P.T = T; P.H = H; P.W = W; P.dtype = dtype; P.r = r;
    LocParams& lp = P.lp;
    std::memset(&lp, 0, sizeof(lp));
    lp.H = H; lp.W = W;
    const int k = (int)r.smoothing_size;
    lp.krad = k / 2;
    lp.taps = 2 * lp.krad + 1;
    if (H <= lp.krad || W <= lp.krad) { *msg = "frame smaller than the smoothing window"; return GT_ERR_ARG; }
    gauss_taps(k, r.noise_size, r.normalized_taps, lp.w, &lp.norm, &lp.rn);
    lp.kk = (float)(k * k);
    lp.rkk = 1.0f / lp.kk;
    dilation(r.separation, &lp.D, &lp.o);
    lp.d = (int)r.diameter;
    lp.rint_c = ((int)r.diameter - 1) / 2;
    lp.border = (int)r.diameter / 2;
    lp.char_r = (int)r.diameter / 2;
    lp.max_iter = (int)r.max_iterations;
    lp.thr = 0.6f;  // gpu_setup.rs:57
    lp.minmass = r.minmass;
    lp.hp = std::max({lp.o, lp.D - 1 - lp.o, lp.char_r, lp.rint_c + 2, 1});
    lp.TH = LOC_TH; lp.TW = LOC_TW;
    lp.ntx = (W + lp.TW - 1) / lp.TW;
    lp.nty = (H + lp.TH - 1) / lp.TH;
    lp.dtype = dtype;
    lp.cpu_processed = r.cpu_processed;
    lp.characterize = r.characterize;
    lp.zero_skip = lp.max_iter >= 1 && lp.rint_c <= lp.o && lp.rint_c <= lp.D - 1 - lp.o;
    lp.tma_spin = 1 << 22;
    lp.tma_withhold = 0;
    P.fast = P.repack = 0;
    const int want_fast = force_generic_flag ? 0 : fast_supported(lp.krad, lp.D, lp.rint_c, lp.d, dtype);
    P.char_tab.clear(); P.char_off.clear(); P.gchar_tab.clear();
    // only what the columns asked for read: most calls upload no table (8 us of
    // a single frame's call)
    if (r.cpu_processed) circle_tables(lp.char_r, P.char_tab, &P.char_off, 1);
    if (r.characterize) circle_tables(lp.rint_c, P.gchar_tab, nullptr, 0);
    lp.n_char = (int)P.char_off.size() / 2;
    lp.n_gchar = (int)P.gchar_tab.size() / 2;
    if (want_fast) {
        P.fast = want_fast;
        lp.TW = 64;
        lp.ntx = (W + lp.TW - 1) / lp.TW;
        set_tile_rows(&P, fast_tile_rows);
        // widths that the tile copies can't take: chunks of frames with padded
        // rows, small enough to be read back from L2
        const int px = dtype == GT_U16 ? 2 : 4, vp = 16 / px;
        P.pitch = (W + vp - 1) / vp * vp;
        const long long frame = (long long)H * P.pitch * px;
        if (P.pitch != W && frame <= REPACK_BYTES) P.repack = (int)std::min<long long>(T, REPACK_BYTES / frame);
    }
    P.sig_off.clear(); P.bg_off.clear();
    if (r.has_sig) circle_inds_f(r.sig_radius, P.sig_off);
    if (r.has_bg) annulus_inds_f(r.bg_radius, r.sig_radius + r.gap_radius, P.bg_off);
    P.tables.clear();
    for (const auto* v : {&P.char_tab, &P.gchar_tab})
        P.tables.insert(P.tables.end(), (const int*)v->data(), (const int*)v->data() + v->size());
    for (const auto* v : {&P.char_off, &P.sig_off, &P.bg_off}) P.tables.insert(P.tables.end(), v->begin(), v->end());
    P.sep = (float)r.separation;
    P.link = r.has_search_range;

    const int PH = LOC_TH + 2 * lp.hp, PW = LOC_TW + 2 * lp.hp;  // generic kernel plan
    const int RH = PH + 2 * lp.krad, RW = PW + 2 * lp.krad;
    P.smem_loc = sizeof(float) * ((size_t)RH * RW + 2 * (size_t)RH * PW + (size_t)PH * PW) +
                 sizeof(int) * (size_t)LOC_TH * LOC_TW + 6 * sizeof(float) * LOC_CMAX + (size_t)LOC_TH * LOC_TW;
    P.smem_loc = (P.smem_loc + 15) / 16 * 16;
    if (P.smem_loc > 227 * 1024) { *msg = "diameter/separation too large for the tile plan"; return GT_ERR_ARG; }
    P.fb_win = std::min(FB_WIN_MAX, std::max(lp.rint_c + 1, lp.max_iter - 1 + lp.rint_c + 1));

    // capacities (bounds; overflow is detected on the device and retried)
    const long long HW = (long long)H * W;
    long long cc = std::max<long long>(4096, HW / cap_div) * scale;
    P.cap_c = (int)std::min<long long>(cc, std::max<long long>(HW, 1));
    const double s = std::max(1.0f, P.sep);
    const double ext_h = H + 2.0 * lp.rint_c + s, ext_w = W + 2.0 * lp.rint_c + s;
    long long pack = (long long)(ext_h * ext_w / (0.785 * s * s)) + 16;
    P.cap_p = (int)std::min<long long>(P.cap_c, pack * scale);
    // cells at least separation + 1 and at most 16384 of them; the linker's at
    // least search_range + 1 and at most 40960: its neighbour searches read
    // 3 x 3 cells of several frames (200 frames of 15k particles, range 7: cells
    // of 10 instead of 16 pixels halve what they read), and a frame's cell
    // counts fit shared memory
    P.G = std::max({(int)std::ceil(P.sep) + 1, 8, (int)std::ceil(std::sqrt((double)HW / 16384.0))});
    P.LG = std::max({P.link ? (int)std::ceil(r.search_range) + 1 : 0, 8, (int)std::ceil(std::sqrt((double)HW / 40960.0))});
    P.lncy = (H + P.LG - 1) / P.LG;
    P.lncx = (W + P.LG - 1) / P.LG;
    P.ncy = (H + P.G - 1) / P.G;
    P.ncx = (W + P.G - 1) / P.G;
    P.smem_fin = sizeof(int) * std::max((size_t)P.ncx * P.ncy, P.link ? (size_t)P.lncx * P.lncy : 0);
    if (P.smem_fin > 200 * 1024) { *msg = "grid too fine"; return GT_ERR_ARG; }
    link_scratch(&P, scale);
    column_list(r, P.names, P.types);
    return GT_OK;
}

// Device workspace carved from one arena.
struct Work {
    void* frames;
    Cand* cand;
    int *rowcnt, *pend;
    float *py, *px, *pm;
    int *prec, *npart, *gstart, *gidx;
    char* repack;
    int *crec, *ccell, *cidx;
    float *cy, *cx, *cm;
    int* tables;
    float *char_tab, *gchar_tab;
    int *char_off, *sig_off, *bg_off;
    // zeroed at the start of a call and read back as one at its end
    int* status;
    int *err, *nrows, *npend, *done, *fcount;
    int *off, *pred, *newrank, *newcount, *newbase, *root, *lroot, *newid;
    int* pbeg;  // fallback list position at the start of each chunk's locate
    // linker (LinkBufs)
    float2* gpos;
    unsigned *lnk, *mm, *pres;
    int *stamp, *rstamp, *seedq, *recq, *deferq, *gframe, *cstamp, *head, *fstamp, *big;
    int4* ent;
    unsigned long long* lstat;  // 4 phase times, 8 frame counts, then the linker's counters
    float* out;
};

struct Carver {
    char* base;
    size_t off = 0;
    template <class X>
    X* take(size_t n) {
        off = (off + 255) / 256 * 256;
        X* p = (X*)(base ? base + off : nullptr);
        off += sizeof(X) * std::max<size_t>(n, 1);
        return p;
    }
};

size_t repack_bytes(const Plan& P) { return (size_t)P.repack * P.H * P.pitch * (P.dtype == GT_U16 ? 2 : 4); }

size_t carve(const Plan& P, char* base, Work* w, size_t frame_bytes, bool need_locate, bool own_out = true) {
    Carver c{base};
    const size_t T = P.T;
    const size_t lcell = (size_t)P.lncx * P.lncy;
    w->frames = c.take<char>(frame_bytes);
    const size_t cc = need_locate ? T * P.cap_c : 1;
    w->cand = c.take<Cand>(cc);
    w->rowcnt = c.take<int>(need_locate ? T * P.H * P.lp.ntx : 1);
    w->pend = c.take<int>(cc);
    w->py = c.take<float>(T * P.cap_p);
    w->px = c.take<float>(T * P.cap_p);
    w->pm = c.take<float>(need_locate ? T * P.cap_p : 1);
    w->prec = c.take<int>(need_locate ? T * P.cap_p : 1);
    w->npart = c.take<int>(T);
    w->gstart = c.take<int>(T * (lcell + 1));
    w->gidx = c.take<int>(T * P.cap_p);
    w->crec = c.take<int>(cc);
    w->ccell = c.take<int>(cc);
    w->cidx = c.take<int>(cc);
    w->cy = c.take<float>(cc);
    w->cx = c.take<float>(cc);
    w->cm = c.take<float>(cc);
    int* tab = c.take<int>(P.tables.size());
    w->tables = tab;
    w->char_tab = (float*)tab;
    w->gchar_tab = (float*)(tab += P.char_tab.size());
    w->char_off = tab += P.gchar_tab.size();
    w->sig_off = tab += P.char_off.size();
    w->bg_off = tab += P.sig_off.size();
    // {errors and linker passes, rows, pending walks, blocks done, the chunks'
    // first pending walks, linker statistics, records per frame}
    w->status = c.take<int>(STATUS_INTS + T);
    w->err = w->status;
    w->nrows = w->status + 4;
    w->npend = w->status + 5;
    w->done = w->status + 6;
    w->pbeg = w->status + 8;
    w->lstat = (unsigned long long*)(w->status + STATUS_LSTAT);
    w->fcount = w->status + STATUS_INTS;
    w->repack = c.take<char>(need_locate ? repack_bytes(P) : 1);
    w->off = c.take<int>(T + 1);
    const size_t np = P.link ? T * P.cap_p : 1;
    const size_t nm = P.link && P.r.memory > 0 ? np : 1;   // memory entries
    const size_t nl = P.link && P.r.memory > 2 ? np : 1;   // and by trajectory root
    const size_t nw = (P.r.memory + 31) / 32;
    w->gpos = c.take<float2>(np);
    w->pred = c.take<int>(np);
    w->newrank = c.take<int>(np);
    w->newcount = c.take<int>(T);
    w->newbase = c.take<int>(T + 1);
    w->root = c.take<int>(np);
    w->lroot = c.take<int>(np);
    w->newid = c.take<int>(np);
    w->lnk = c.take<unsigned>(nm);
    w->mm = c.take<unsigned>(nm * nw);
    w->stamp = c.take<int>(nm);
    w->rstamp = c.take<int>(nm);
    w->seedq = c.take<int>(np);
    w->recq = c.take<int>(nm);
    w->deferq = c.take<int>(np);
    w->gframe = c.take<int>(nl);
    w->cstamp = c.take<int>(nl);
    size_t nh = 1;
    while (nh < nl) nh <<= 1;
    w->head = c.take<int>(nh);
    w->ent = c.take<int4>(nl);
    w->pres = c.take<unsigned>(nl * nw);
    w->fstamp = c.take<int>(T);
    w->big = c.take<int>((size_t)P.nslot * big_ints(P));
    w->out = c.take<float>(need_locate && own_out ? T * P.cap_p * P.names.size() : 1);
    return c.off + 256;
}

#define CK(x)                                                                              \
    do {                                                                                   \
        cudaError_t e_ = (x);                                                              \
        if (e_ != cudaSuccess) {                                                           \
            ctx->err = std::string(#x) + ": " + cudaGetErrorString(e_);                    \
            return e_ == cudaErrorMemoryAllocation ? GT_ERR_OOM : GT_ERR_CUDA;             \
        }                                                                                  \
    } while (0)

int ensure_arena(gt_ctx* ctx, size_t bytes) {
    if (ctx->arena_size >= bytes) return GT_OK;
    if (ctx->arena) { cudaFree(ctx->arena); ctx->arena = nullptr; ctx->arena_size = 0; }
    size_t want = bytes + bytes / 8;
    if (cudaMalloc((void**)&ctx->arena, want) != cudaSuccess) {
        ctx->err = "workspace of " + std::to_string(want >> 20) + " MB: " + cudaGetErrorString(cudaGetLastError());
        ctx->arena = nullptr;
        return GT_ERR_OOM;
    }
    ctx->arena_size = want;
    return GT_OK;
}

LinkBufs link_bufs(const Plan& P, const Work& w, long long budget) {
    LinkBufs L{};
    L.tb = 0;
    L.te = P.T;
    L.cap_p = P.cap_p; L.memory = (int)std::min<uint32_t>(P.r.memory, (uint32_t)P.T);
    L.r = P.r.search_range;
    L.inv_g = 1.0f / (float)P.LG;
    L.ncx = P.lncx; L.ncy = P.lncy;
    L.py = w.py; L.px = w.px; L.off = w.off; L.gstart = w.gstart; L.gidx = w.gidx; L.gpos = w.gpos;
    L.np = (size_t)P.T * P.cap_p;
    L.pred = w.pred; L.lnk = w.lnk; L.mm = w.mm; L.stamp = w.stamp; L.rstamp = w.rstamp;
    L.seedq = w.seedq; L.recq = w.recq; L.deferq = w.deferq;
    L.newrank = w.newrank; L.newcount = w.newcount; L.root = w.root; L.lroot = w.lroot;
    L.gframe = w.gframe; L.cstamp = w.cstamp; L.head = w.head; L.ent = w.ent; L.pres = w.pres;
    while ((1 << L.fshift) < L.memory) ++L.fshift;
    L.fstamp = w.fstamp; L.ctr = (int*)(w.lstat + 12); L.err = w.err;
    L.budget = budget;
    L.nslot = P.nslot; L.big_d = P.big_d; L.big_s = P.big_s; L.big_e = P.big_e;
    L.big_ints = big_ints(P); L.big = w.big;
    return L;
}

// Resident blocks of the one-movie (0) or the batched (1) linker.
int link_grid(gt_ctx* ctx, int multi, int* grid) {
    if (!ctx->link_grid[multi]) {
        int q = 0;
        CK(link_blocks_per_sm(multi != 0, &q));
        ctx->link_grid[multi] = std::max(1, q) * ctx->num_sms;
    }
    *grid = ctx->link_grid[multi];
    return GT_OK;
}

// Linking over the particle tables already in the workspace (npart, py, px,
// gstart/gidx, off): cooperative launches of link_fixpoint_kernel run the
// fixed point, then new trajectory ids are numbered.  Leaves the trajectory
// id of particle g in newid[root[g]].
//
// The linker in frame windows.  link_window links frames [tb, te) to their
// fixed point, given final links for the frames before tb: the memory
// entries of a frame depend only on earlier frames, so windows taken in
// order give the sequential result (the host-frames path links each
// uploaded chunk while the next one is copied).  link_finish runs once after
// the last.
int link_window(gt_ctx* ctx, const Plan& P, const Work& w, cudaStream_t st, int tb, int te) {
    LinkBufs L = link_bufs(P, w, ctx->subnet_budget);
    L.tb = tb;
    L.te = te;
    int grid = 1;
    const int rc = link_grid(ctx, 0, &grid);
    if (rc) return rc;
    // the pass counters start at zero (the statistics add up over windows)
    if (tb > 0) CK(cudaMemsetAsync(w.lstat + 12, 0, sizeof(int) * 4 * NCTR, st));
    CK(launch_link(L, te - tb + 1, w.err + 1, w.lstat, grid, st));
    ctx->stats.launches += 1;
    return GT_OK;
}

int link_finish(gt_ctx* ctx, const Plan& P, const Work& w, cudaStream_t st) {
    const int T = P.T;
    scan_frames_kernel<<<1, 1024, 0, st>>>(w.newcount, w.newbase, T);
    newid_kernel<<<T, 256, 0, st>>>(w.newrank, w.newbase, w.off, w.npart, w.newid, T);
    CK(cudaGetLastError());
    ctx->stats.launches += 2;
    return GT_OK;
}

int run_link(gt_ctx* ctx, const Plan& P, const Work& w, cudaStream_t st) {
    int rc = link_window(ctx, P, w, st, 0, P.T);
    if (!rc) rc = link_finish(ctx, P, w, st);
    return rc;
}

int upload_tables(gt_ctx* ctx, const Plan& P, const Work& w, cudaStream_t st) {
    if (!P.tables.empty())
        CK(cudaMemcpyAsync(w.tables, P.tables.data(), sizeof(int) * P.tables.size(), cudaMemcpyHostToDevice, st));
    return GT_OK;
}

MovieBufs movie_bufs(const Plan& P, const Work& w, const void* frames) {
    MovieBufs b{};
    b.frames = frames;
    b.T = P.T;
    b.cap_c = P.cap_c; b.cap_p = P.cap_p;
    b.cand = w.cand; b.fcount = w.fcount; b.rowcnt = w.rowcnt; b.pend = w.pend; b.npend = w.npend;
    b.py = w.py; b.px = w.px; b.pm = w.pm; b.prec = w.prec; b.npart = w.npart;
    b.G = P.G; b.ncx = P.ncx; b.ncy = P.ncy; b.LG = P.LG; b.lncx = P.lncx; b.lncy = P.lncy; b.gstart = w.gstart; b.gidx = w.gidx; b.gpos = w.gpos;
    b.cy = w.cy; b.cx = w.cx; b.cm = w.cm; b.crec = w.crec; b.ccell = w.ccell;
    b.cidx = w.cidx;
    b.char_tab = w.char_tab; b.char_off = w.char_off; b.gchar_tab = w.gchar_tab;
    b.err = w.err;
    b.off = w.off; b.done = w.done; b.nrows = w.nrows;
    return b;
}

// The specialised locate kernel over frames [f0, f0 + nf).  *used_tma: the tiles
// were copied from the frames as they are.
int locate_frames(gt_ctx* ctx, const Plan& P, const Work& w, const MovieBufs& b, int f0, int nf, cudaStream_t st,
                  int* used_tma, int32_t* launches) {
    const int ntiles = P.lp.ntx * P.lp.nty;
    *used_tma = 0;
    if (!P.repack) {
        CK(launch_locate_fast(P.lp.krad, P.lp.D, P.lp.rint_c, P.fast_th, dim3(ntiles, nf), st, P.lp, b,
                              TileSource{(const char*)b.frames + (size_t)f0 * P.H * P.W * (P.dtype == GT_U16 ? 2 : 4), P.W},
                              f0, used_tma));
        ++*launches;
        return GT_OK;
    }
    for (int s = f0; s < f0 + nf; s += P.repack) {
        const int m = std::min(P.repack, f0 + nf - s);
        int tma = 0;
        CK(launch_repack(b.frames, P.dtype, s, m, P.H, P.W, P.pitch, w.repack, ctx->num_sms, st));
        CK(launch_locate_fast(P.lp.krad, P.lp.D, P.lp.rint_c, P.fast_th, dim3(ntiles, m), st, P.lp, b,
                              TileSource{w.repack, P.pitch}, s, &tma));
        *launches += 2;
    }
    return GT_OK;
}

// The whole locate(+link) pipeline on device frames; table left in w.out.
// With h_frames set, d_frames is the workspace copy of host frames: the
// copy runs in chunks of frames on the context's copy stream and each
// chunk's locate launch waits only for its own chunk, so host->device
// transfer and locate overlap.
int run_pipeline(gt_ctx* ctx, const Plan& P, const Work& w, const void* d_frames, cudaStream_t st,
                 int* err_bits, int64_t* nrows, int* d_walk = nullptr, int64_t walk_rows = 0,
                 const void* h_frames = nullptr, size_t elem = 0,
                 const std::function<int(int, int)>* ready = nullptr, float* d_out = nullptr,
                 int64_t out_rows = 0) {
    const int T = P.T;
    MovieBufs b = movie_bufs(P, w, d_frames);
    int rc = upload_tables(ctx, P, w, st);
    if (rc) return rc;
    CK(cudaMemsetAsync(w.status, 0, sizeof(int) * (STATUS_INTS + (size_t)T), st));
    CK(allow_shared<locate_tiles_kernel>());
    for (int i = 0; i < 5; ++i)
        if (!ctx->ev[i]) CK(cudaEventCreate(&ctx->ev[i]));
    const bool fast = P.fast != 0;
    ctx->stats.locate_kernel = P.fast == 1 ? 1 : 0;
    // frame chunks: up to 16 for host frames (copy/locate overlap; the
    // locate of the last chunk is what remains after the copy), else as
    // large as the grid allows
    const int chunk = h_frames ? std::min(65535, std::max(16, (T + 15) / 16)) : 65535;
    const size_t fbytes = (size_t)P.H * P.W * elem;
    int ci = 0;
    auto stage = [&](int f0, int nf) -> int {
        if (!h_frames) return GT_OK;
        if (!ctx->copy_stream) CK(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
        for (auto& e : ctx->cev)
            if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        if (ci == 0) {
            CK(cudaEventRecord(ctx->cev[8], st));
            CK(cudaStreamWaitEvent(ctx->copy_stream, ctx->cev[8], 0));
        }
        if (ready) {
            // host frames still being produced (file decode): wait for these
            const int rr = (*ready)(f0, nf);
            if (rr) return rr;
        }
        CK(ctx->hc.upload((char*)d_frames + (size_t)f0 * fbytes, (const char*)h_frames + (size_t)f0 * fbytes,
                          (size_t)nf * fbytes, ctx->copy_stream));
        CK(cudaEventRecord(ctx->cev[ci & 7], ctx->copy_stream));
        CK(cudaStreamWaitEvent(st, ctx->cev[ci & 7], 0));
        ++ci;
        return GT_OK;
    };
    // With host frames and linking, each uploaded chunk is also finalized
    // (pending walks, ordering, separation filter, offsets) behind its copy,
    // and every few chunks are linked, so only the last ones' work follows the
    // upload.
    const int nchunks = (T + chunk - 1) / chunk;
    const bool chunked = h_frames && P.link && nchunks > 1 && nchunks <= LINK_WINDOWS;
    int wi = 0, linked = 0;
    auto post = [&](int f0, int nf) -> int {
        CK(launch_fallback(P.lp, b, P.fb_win, w.pbeg + wi, ctx->num_sms * 4, st));
        CK(launch_finalize(P.lp, b, P.sep, P.link, f0, nf, P.smem_fin, st));
        CK(cudaGetLastError());
        ctx->stats.launches += 2;
        ++wi;
        // linked in LINK_RUNS runs of chunks: a run costs its passes (about 15
        // us each) whatever its frames, 13 runs 2.0 ms of a 200-frame movie
        if (P.link && (f0 + nf == T || wi % ((nchunks + LINK_RUNS - 1) / LINK_RUNS) == 0)) {
            const int r2 = link_window(ctx, P, w, st, linked, f0 + nf);
            if (r2) return r2;
            linked = f0 + nf;
        }
        return GT_OK;
    };
    // the fallback list position where chunk wi's entries begin
    auto mark = [&]() -> int {
        if (chunked && wi > 0) CK(cudaMemcpyAsync(w.pbeg + wi, w.npend, sizeof(int), cudaMemcpyDeviceToDevice, st));
        return GT_OK;
    };
    if (fast) {
        CK(cudaEventRecord(ctx->ev[0], st));
        for (int f0 = 0; f0 < T; f0 += chunk) {
            const int nf = std::min(chunk, T - f0);
            rc = stage(f0, nf);
            if (!rc) rc = mark();
            if (rc) return rc;
            int used_tma = 0;
            rc = locate_frames(ctx, P, w, b, f0, nf, st, &used_tma, &ctx->stats.launches);
            if (rc) return rc;
            if (P.fast == 1) ctx->stats.locate_kernel = used_tma ? 2 : 1;
            if (chunked && (rc = post(f0, nf))) return rc;
        }
    } else {
        LocParams lg = P.lp;  // generic tile plan (its own tile height)
        lg.TH = LOC_TH;
        lg.TW = LOC_TW;
        lg.ntx = (P.W + LOC_TW - 1) / LOC_TW;
        lg.nty = (P.H + LOC_TH - 1) / LOC_TH;
        CK(cudaEventRecord(ctx->ev[0], st));
        for (int f0 = 0; f0 < T; f0 += chunk) {
            const int nf = std::min(chunk, T - f0);
            rc = stage(f0, nf);
            if (!rc) rc = mark();
            if (rc) return rc;
            dim3 grid(lg.ntx * lg.nty, nf);
            locate_tiles_kernel<<<grid, 256, P.smem_loc, st>>>(lg, b, f0);
            ctx->stats.launches += 1;
            if (chunked && (rc = post(f0, nf))) return rc;
        }
    }
    CK(cudaGetLastError());
    CK(cudaEventRecord(ctx->ev[1], st));
    if (!chunked) {
        // the whole movie as one window: finalize, then link
        CK(launch_fallback(P.lp, b, P.fb_win, w.pbeg, ctx->num_sms * 4, st));
        CK(launch_finalize(P.lp, b, P.sep, P.link, 0, T, P.smem_fin, st));
        CK(cudaGetLastError());
        ctx->stats.launches += 2;
    }
    CK(cudaEventRecord(ctx->ev[2], st));
    if (P.link) {
        if (!chunked) rc = link_window(ctx, P, w, st, 0, T);
        if (!rc) rc = link_finish(ctx, P, w, st);
        if (rc) return rc;
    }
    CK(cudaEventRecord(ctx->ev[3], st));
    AsmArgs a{};
    a.T = T; a.H = P.H; a.W = P.W; a.cap_p = P.cap_p; a.cap_c = P.cap_c; a.ncols = (int)P.names.size();
    a.has_link = P.link; a.cpu_processed = P.r.cpu_processed; a.characterize = P.r.characterize;
    a.sig = P.r.has_sig; a.bg = P.r.has_bg;
    a.frames = d_frames; a.dtype = P.dtype;
    a.py = w.py; a.px = w.px; a.pm = w.pm; a.prec = w.prec; a.npart = w.npart; a.off = w.off;
    a.cand = w.cand; a.root = w.root; a.newid = w.newid;
    a.sig_off = w.sig_off; a.n_sig = (int)P.sig_off.size() / 2;
    a.bg_off = w.bg_off; a.n_bg = (int)P.bg_off.size() / 2;
    // a caller's device buffer takes the rows directly (those beyond its
    // capacity are not written; the caller learns the count)
    a.out = d_out ? d_out : w.out;
    a.out_rows = d_out ? out_rows : LLONG_MAX;
    a.walk = d_walk;
    a.walk_rows = walk_rows;
    CK(launch_assemble(a, ctx->num_sms, st));
    ctx->stats.launches += 1;
    CK(cudaEventRecord(ctx->ev[4], st));
    // every statistic of the call in one readback: error words, row count,
    // pending walks, per-frame record counts, linker phases and frame counts
    const size_t need_ints = STATUS_INTS + (size_t)T;
    if (ctx->h_stage_n < need_ints) {
        if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
        ctx->h_stage = nullptr;
        ctx->h_stage_n = 0;
        CK(cudaHostAlloc((void**)&ctx->h_stage, sizeof(int) * need_ints, cudaHostAllocDefault));
        ctx->h_stage_n = need_ints;
    }
    int* hs = ctx->h_stage;
    CK(cudaMemcpyAsync(hs, w.status, sizeof(int) * need_ints, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const unsigned long long* hph = (const unsigned long long*)(hs + STATUS_LSTAT);
    const int hb[5] = {hs[0], hs[1], hs[2], hs[3], hs[4]};
    const int np = hs[5];
    long long nc_total = 0;
    for (int t = 0; t < T; ++t) nc_total += hs[STATUS_INTS + t];
    *err_bits = hb[0];
    *nrows = hb[4];
    ctx->stats.link_iterations = P.link ? hb[1] : 0;
    if (P.link) {
        for (int i = 0; i < 4; ++i) ctx->stats.link_phase_ms[i] = (float)(hph[i] * 1e-6);
        for (int i = 0; i < 8; ++i) ctx->stats.link_dirty[i] = (int)hph[4 + i];
    }
    ctx->stats.fallback_walks = np;
    ctx->stats.particles = hb[4];
    ctx->stats.candidates = nc_total;
    ctx->stage_times = 1;  // read from the events when asked for (gt_last_stats)
    return GT_OK;
}

int err_status(gt_ctx* ctx, int bits, bool* retry) {
    *retry = false;
    if (bits & ERR_DEVICE_TIMEOUT) {
        ctx->err = "a bounded device wait expired (TMA tile load)";
        return GT_ERR_DEVICE_TIMEOUT;
    }
    if (bits & ERR_SUBNET_BUDGET) {
        ctx->err = "a linking subnetwork exceeded the search budget";
        return GT_ERR_SUBNET_BUDGET;
    }
    if (bits & (ERR_CAND_OVERFLOW | ERR_PART_OVERFLOW | ERR_EDGE_OVERFLOW |
                ERR_SCRATCH_OVERFLOW)) {
        *retry = true;
        ctx->err = "per-frame capacity exceeded (bits " + std::to_string(bits) + ")";
        return GT_ERR_CAPACITY;
    }
    return GT_OK;
}

size_t elem_size(int dtype) { return dtype == GT_U16 ? 2 : 4; }

// Host tables (gt_table.data) live in page-locked memory, so the
// device->host copy of a table runs at full PCIe speed and touches no fresh
// pages.  Released tables go back to a small process-wide pool (gt_table_free
// has no context) and are reused by later calls of a similar size; memory
// that cannot be page-locked falls back to malloc.
struct TablePool {
    std::mutex m;
    std::vector<std::pair<void*, size_t>> idle;  // page-locked blocks not in use
    std::map<void*, size_t> locked;               // every page-locked block handed out or idle
    size_t idle_bytes = 0;
};
TablePool& table_pool() {
    static TablePool* pool = new TablePool();  // never destroyed: tables may be freed at exit
    return *pool;
}
constexpr size_t TABLE_IDLE_MAX_BLOCKS = 4;
constexpr size_t TABLE_IDLE_MAX_BYTES = (size_t)1 << 30;

float* table_alloc(size_t bytes) {
    TablePool& tp = table_pool();
    {
        std::lock_guard<std::mutex> g(tp.m);
        int best = -1;
        for (int i = 0; i < (int)tp.idle.size(); ++i) {
            const size_t sz = tp.idle[i].second;
            if (sz >= bytes && sz <= 2 * bytes + ((size_t)2 << 20) && (best < 0 || sz < tp.idle[best].second))
                best = i;
        }
        if (best >= 0) {
            void* q = tp.idle[best].first;
            tp.idle_bytes -= tp.idle[best].second;
            tp.idle.erase(tp.idle.begin() + best);
            return (float*)q;
        }
    }
    const size_t sz = (bytes + ((size_t)2 << 20) - 1) / ((size_t)2 << 20) * ((size_t)2 << 20);
    void* q = nullptr;
    if (cudaHostAlloc(&q, sz, cudaHostAllocPortable) == cudaSuccess && q) {
        std::lock_guard<std::mutex> g(tp.m);
        tp.locked[q] = sz;
        return (float*)q;
    }
    cudaGetLastError();
    return (float*)std::malloc(bytes);
}

void table_release(void* q) {
    if (!q) return;
    TablePool& tp = table_pool();
    std::lock_guard<std::mutex> g(tp.m);
    auto it = tp.locked.find(q);
    if (it == tp.locked.end()) {
        std::free(q);
        return;
    }
    if (tp.idle.size() < TABLE_IDLE_MAX_BLOCKS && tp.idle_bytes + it->second <= TABLE_IDLE_MAX_BYTES) {
        tp.idle.push_back({q, it->second});
        tp.idle_bytes += it->second;
        return;
    }
    tp.locked.erase(it);
    cudaFreeHost(q);  // an error here (runtime already unloading at exit) is harmless
}

int batch_common(gt_ctx* ctx, const void* frames, bool host, int dtype, int T, int H, int W,
                 const gt_params* params, gt_table* out_tab, float* d_out, int64_t out_rows,
                 int64_t* nrows_out, cudaStream_t st, int* d_walk = nullptr,
                 const std::function<int(int, int)>* ready = nullptr) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    ctx->stats = gt_stats{};
    ctx->stage_times = 0;
    if (!frames || !params || T < 1 || H < 1 || W < 1 || (dtype != GT_U16 && dtype != GT_F32)) {
        ctx->err = "invalid frames/shape/dtype";
        return GT_ERR_ARG;
    }
    if ((long long)H * W > (1LL << 28) || H > 65535 || W > 65535) { ctx->err = "frame too large"; return GT_ERR_ARG; }
    Resolved r;
    int rc = resolve(params, &r, &ctx->err);
    if (rc) return rc;
    r.normalized_taps = ctx->normalized_taps;
    CK(cudaSetDevice(ctx->device));
    int cap_div = 64;
    for (int scale = 1; scale <= 64; scale *= 4) {
        Plan P;
        Work w{};
        const size_t fbytes = host ? (size_t)T * H * W * elem_size(dtype) : 0;
        while (true) {
            rc = make_plan(r, T, H, W, dtype, scale, ctx->num_sms, &P, &ctx->err, ctx->force_generic,
                           ctx->fast_tile_rows, cap_div);
            if (rc) return rc;
            if (cap_div != 64) P.repack = 0;  // memory is short
            // a caller's device buffer receives the rows directly: no table slab
            rc = ensure_arena(ctx, carve(P, nullptr, &w, fbytes, true, d_out == nullptr));
            if (!rc) break;
            // the largest capacities that fit; more features than they hold ask
            // for larger ones again
            if (rc != GT_ERR_OOM || scale > 1 || cap_div >= 1024) return rc;
            cap_div *= 2;
        }
        ctx->err.clear();
        if (ctx->withhold_tma) {
            P.lp.tma_withhold = 1;
            P.lp.tma_spin = 1 << 10;
        }
        P.lp.tiles_per_cta = ctx->tiles_per_cta;
        carve(P, ctx->arena, &w, fbytes, true, d_out == nullptr);
        const void* dfr = host ? w.frames : frames;
        int bits = 0;
        int64_t nrows = 0;
        rc = run_pipeline(ctx, P, w, dfr, st, &bits, &nrows, d_walk, d_walk ? out_rows : 0, host ? frames : nullptr,
                          elem_size(dtype), ready, d_out, out_rows);
        if (rc) return rc;
        bool retry;
        rc = err_status(ctx, bits, &retry);
        ctx->stats.retries = scale > 1 ? (int)std::log2((double)scale) / 2 : 0;
        if (rc && retry && scale < 64) continue;
        if (rc) return rc;
        const int ncols = (int)P.names.size();
        if (out_tab) {
            out_tab->nrows = nrows;
            out_tab->ncols = ncols;
            std::memset(out_tab->names, 0, sizeof(out_tab->names));
            std::memset(out_tab->types, 0, sizeof(out_tab->types));
            for (int i = 0; i < ncols && i < GT_MAX_COLS; ++i) {
                std::snprintf(out_tab->names[i], sizeof(out_tab->names[i]), "%s", P.names[i].c_str());
                std::snprintf(out_tab->types[i], sizeof(out_tab->types[i]), "%s", P.types[i].c_str());
            }
            out_tab->data = table_alloc(sizeof(float) * (size_t)std::max<int64_t>(1, nrows) * ncols);
            if (!out_tab->data) { ctx->err = "host allocation failed"; return GT_ERR_OOM; }
            if (nrows > 0) {
                CK(cudaMemcpyAsync(out_tab->data, w.out, sizeof(float) * (size_t)nrows * ncols,
                                   cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
            }
        }
        // with d_out the rows were written there directly (run_pipeline
        // returns after the stream is synchronised)
        if (nrows_out) *nrows_out = nrows;
        return GT_OK;
    }
    return GT_ERR_CAPACITY;
}


// ---------------------------------------------------------------------------
// Batched uneven movies (gt_batch_many_device).
//
// Every movie gets its own plan and workspace in one arena.  The locate,
// fallback, ordering/separation and output kernels of the movies are
// enqueued on side streams (parallel graph branches), the linking of all
// movies runs in one cooperative kernel (link_fixpoint_multi_kernel) whose
// blocks share one scratch pool, and the sequence is captured once into a
// CUDA graph that is replayed while the inputs stay the same.
// ---------------------------------------------------------------------------

struct BatchMovie {
    Plan P;
    Work w;
    size_t off = 0;
    bool fast = false;
    int link_slot = -1;  // index among the movies of the shared linker launch
};

struct BatchShared {
    LinkBufs* d_L = nullptr;
    unsigned long long* d_stat = nullptr;
    int* d_passes = nullptr;
    int* d_status = nullptr;  // 8 ints per movie: err[0..3], nrows
    int nlink = 0, max_passes = 0, link_grid = 0;
    int launches = 0;
};

// Tile rows of the specialised locate kernel for one (frame size, diameter)
// class: both variants timed on up to 32 frames of the movie, the faster
// kept for the context's lifetime.
int tune_tile_rows(gt_ctx* ctx, BatchMovie& bm, const void* frames, cudaStream_t st) {
    Plan& P = bm.P;
    const std::array<int, 6> key{P.H, P.W, P.lp.krad, P.lp.D, P.lp.rint_c, P.dtype};
    auto it = ctx->tile_rows.find(key);
    int best = P.fast_th;
    if (it != ctx->tile_rows.end()) {
        best = it->second;
    } else if (!ctx->tune_disabled) {
        for (int i = 0; i < 2; ++i)
            if (!ctx->ev[i]) CK(cudaEventCreate(&ctx->ev[i]));
        const int nf = std::min(P.T, 32);
        float ms[2] = {0.f, 0.f};
        const int ths[2] = {32, 64};
        for (int v = 0; v < 2; ++v) {
            Plan Q = P;  // the workspace is carved for P's capacities
            set_tile_rows(&Q, ths[v]);
            MovieBufs b = movie_bufs(Q, bm.w, frames);
            for (int rep = 0; rep < 2; ++rep) {
                CK(cudaMemsetAsync(bm.w.status, 0, sizeof(int) * (STATUS_INTS + (size_t)P.T), st));
                CK(cudaEventRecord(ctx->ev[0], st));
                int used_tma = 0, launches = 0;
                const int rc = locate_frames(ctx, Q, bm.w, b, 0, nf, st, &used_tma, &launches);
                if (rc) return rc;
                CK(cudaEventRecord(ctx->ev[1], st));
                CK(cudaEventSynchronize(ctx->ev[1]));
                CK(cudaEventElapsedTime(&ms[v], ctx->ev[0], ctx->ev[1]));
            }
        }
        best = ms[1] < ms[0] ? 64 : 32;
        ctx->tile_rows[key] = best;
    }
    set_tile_rows(&P, best);
    return GT_OK;
}

// Locate, fallback walks, ordering + separation filter and frame offsets of
// one movie (the front half of run_pipeline, without host synchronisation).
int enqueue_front(gt_ctx* ctx, BatchMovie& bm, const void* frames, cudaStream_t s, int* launches) {
    const Plan& P = bm.P;
    const Work& w = bm.w;
    const int T = P.T;
    MovieBufs b = movie_bufs(P, w, frames);
    CK(cudaMemsetAsync(w.status, 0, sizeof(int) * (STATUS_INTS + (size_t)T), s));
    if (bm.fast) {
        for (int f0 = 0; f0 < T; f0 += 65535) {
            int used_tma = 0;
            const int rc = locate_frames(ctx, P, w, b, f0, std::min(65535, T - f0), s, &used_tma, launches);
            if (rc) return rc;
        }
    } else {
        LocParams lg = P.lp;
        lg.TH = LOC_TH;
        lg.TW = LOC_TW;
        lg.ntx = (P.W + LOC_TW - 1) / LOC_TW;
        lg.nty = (P.H + LOC_TH - 1) / LOC_TH;
        for (int f0 = 0; f0 < T; f0 += 65535) {
            dim3 grid(lg.ntx * lg.nty, std::min(65535, T - f0));
            locate_tiles_kernel<<<grid, 256, P.smem_loc, s>>>(lg, b, f0);
            ++*launches;
        }
    }
    CK(cudaGetLastError());
    CK(launch_fallback(P.lp, b, P.fb_win, nullptr, ctx->num_sms, s));
    CK(launch_finalize(P.lp, b, P.sep, P.link, 0, T, P.smem_fin, s));
    *launches += 2;
    return GT_OK;
}

// Trajectory ids and the output table of one movie, then its status words.
int enqueue_back(gt_ctx* ctx, BatchMovie& bm, const gt_movie& mv, int* d_status, cudaStream_t s, int* launches) {
    const Plan& P = bm.P;
    const Work& w = bm.w;
    const int T = P.T;
    if (P.link) {
        scan_frames_kernel<<<1, 1024, 0, s>>>(w.newcount, w.newbase, T);
        newid_kernel<<<T, 256, 0, s>>>(w.newrank, w.newbase, w.off, w.npart, w.newid, T);
        *launches += 2;
    }
    AsmArgs a{};
    a.T = T; a.H = P.H; a.W = P.W; a.cap_p = P.cap_p; a.cap_c = P.cap_c; a.ncols = (int)P.names.size();
    a.has_link = P.link; a.cpu_processed = P.r.cpu_processed; a.characterize = P.r.characterize;
    a.sig = P.r.has_sig; a.bg = P.r.has_bg;
    a.frames = mv.frames; a.dtype = P.dtype;
    a.py = w.py; a.px = w.px; a.pm = w.pm; a.prec = w.prec; a.npart = w.npart; a.off = w.off;
    a.cand = w.cand; a.root = w.root; a.newid = w.newid;
    a.sig_off = w.sig_off; a.n_sig = (int)P.sig_off.size() / 2;
    a.bg_off = w.bg_off; a.n_bg = (int)P.bg_off.size() / 2;
    a.out = mv.out;
    a.out_rows = mv.out ? mv.out_rows : 0;
    CK(launch_assemble(a, ctx->num_sms, s));
    *launches += 1;
    CK(cudaMemcpyAsync(d_status, w.status, sizeof(int) * 5, cudaMemcpyDeviceToDevice, s));
    return GT_OK;
}

// The whole batch on `st`, fanned out over the context's side streams: movie i
// on stream i % BATCH_STREAMS.
int enqueue_batch(gt_ctx* ctx, std::vector<BatchMovie>& B, gt_movie* mv, int n, BatchShared& S, cudaStream_t st) {
    const int K = BATCH_STREAMS;
    S.launches = 0;
    CK(cudaEventRecord(ctx->bev[0], st));
    for (int k = 0; k < K; ++k) CK(cudaStreamWaitEvent(ctx->side[k], ctx->bev[0], 0));
    for (int i = 0; i < n; ++i) {
        int rc = enqueue_front(ctx, B[i], mv[i].frames, ctx->side[i % K], &S.launches);
        if (rc) return rc;
    }
    for (int k = 0; k < K; ++k) {
        CK(cudaEventRecord(ctx->bev[1 + k], ctx->side[k]));
        CK(cudaStreamWaitEvent(st, ctx->bev[1 + k], 0));
    }
    if (S.nlink > 0) {
        CK(cudaMemsetAsync(S.d_passes, 0, sizeof(int), st));
        CK(cudaMemsetAsync(S.d_stat, 0, sizeof(unsigned long long) * 12, st));
        CK(launch_link_multi(S.d_L, S.nlink, S.max_passes, S.d_passes, S.d_stat, S.link_grid, st));
        S.launches += 1;
    }
    CK(cudaEventRecord(ctx->bev[1 + K], st));
    for (int k = 0; k < K; ++k) CK(cudaStreamWaitEvent(ctx->side[k], ctx->bev[1 + K], 0));
    for (int i = 0; i < n; ++i) {
        int rc = enqueue_back(ctx, B[i], mv[i], S.d_status + 8 * i, ctx->side[i % K], &S.launches);
        if (rc) return rc;
    }
    for (int k = 0; k < K; ++k) {
        CK(cudaEventRecord(ctx->bev[2 + K + k], ctx->side[k]));
        CK(cudaStreamWaitEvent(st, ctx->bev[2 + K + k], 0));
    }
    CK(cudaMemcpyAsync(ctx->h_status, S.d_status, sizeof(int) * 8 * (size_t)n, cudaMemcpyDeviceToHost, st));
    return GT_OK;
}

void drop_batch_graph(gt_ctx* ctx) {
    if (ctx->batch_exec) cudaGraphExecDestroy(ctx->batch_exec);
    ctx->batch_exec = nullptr;
    ctx->batch_key.clear();
}

int batch_many(gt_ctx* ctx, gt_movie* mv, int n, cudaStream_t st) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    ctx->stats = gt_stats{};
    ctx->stage_times = 0;
    if (n < 0 || (n > 0 && !mv)) { ctx->err = "invalid movie list"; return GT_ERR_ARG; }
    if (n == 0) return GT_OK;
    CK(cudaSetDevice(ctx->device));
    std::vector<BatchMovie> B(n);
    std::string key;
    for (int i = 0; i < n; ++i) {
        const gt_movie& m = mv[i];
        const std::string who = "movie " + std::to_string(i) + ": ";
        if (!m.frames || m.T < 1 || m.H < 1 || m.W < 1 || (m.dtype != GT_U16 && m.dtype != GT_F32) ||
            (m.out_rows > 0 && !m.out) || m.out_rows < 0) {
            ctx->err = who + "invalid frames/shape/dtype/output";
            return GT_ERR_ARG;
        }
        if ((long long)m.H * m.W > (1LL << 28) || m.H > 65535 || m.W > 65535) {
            ctx->err = who + "frame too large";
            return GT_ERR_ARG;
        }
        Resolved r;
        std::string msg;
        int rc = resolve(&m.params, &r, &msg);
        if (rc) { ctx->err = who + msg; return rc; }
        r.normalized_taps = ctx->normalized_taps;
        rc = make_plan(r, m.T, m.H, m.W, m.dtype, 1, ctx->num_sms, &B[i].P, &msg, ctx->force_generic, ctx->fast_tile_rows,
                       ctx->batch_cap_div);
        if (rc) { ctx->err = who + msg; return rc; }
        B[i].P.lp.tiles_per_cta = ctx->tiles_per_cta;
        char buf[128];
        std::snprintf(buf, sizeof(buf), "%p|%d|%d|%d|%d|%p|%lld|", m.frames, m.dtype, m.T, m.H, m.W, (void*)m.out,
                      (long long)m.out_rows);
        key += buf;
        key.append((const char*)&m.params, sizeof(gt_params));
    }
    // pinned status words, side streams, events
    if (ctx->h_status_n < (size_t)8 * n) {
        drop_batch_graph(ctx);  // it reads back into the old words
        if (ctx->h_status) cudaFreeHost(ctx->h_status);
        ctx->h_status = nullptr;
        ctx->h_status_n = 0;
        CK(cudaHostAlloc((void**)&ctx->h_status, sizeof(int) * 8 * (size_t)n, cudaHostAllocDefault));
        ctx->h_status_n = (size_t)8 * n;
    }
    for (auto& sd : ctx->side)
        if (!sd) CK(cudaStreamCreateWithFlags(&sd, cudaStreamNonBlocking));
    for (auto& e : ctx->bev)
        if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (int i = 0; i < 5; ++i)
        if (!ctx->ev[i]) CK(cudaEventCreate(&ctx->ev[i]));
    // kernel choice
    for (int i = 0; i < n; ++i) B[i].fast = B[i].P.fast != 0;
    // all linked movies share one linker launch and its scratch slots (a
    // block resolves one large component at a time)
    BatchShared S;
    int rc_g = link_grid(ctx, 1, &S.link_grid);
    if (rc_g) return rc_g;
    Plan big;
    for (int i = 0; i < n; ++i) {
        const Plan& P = B[i].P;
        if (!P.link) continue;
        B[i].link_slot = S.nlink++;
        S.max_passes = std::max(S.max_passes, P.T + 1);
        big.big_d = std::max(big.big_d, P.big_d);
        big.big_s = std::max(big.big_s, P.big_s);
        big.big_e = std::max(big.big_e, P.big_e);
        big.T += P.T;
    }
    if (S.nlink > 0) big.nslot = big_slots(big, big.T);
    // arena layout: movies, link pool, shared arrays
    size_t total = 0;
    // one buffer of repacked rows per side stream, whose movies follow one another
    size_t rows[BATCH_STREAMS] = {};
    auto own = [&](int i) {  // what a movie does not share
        Plan Pc = B[i].P;
        Pc.nslot = 0;
        Pc.repack = 0;
        return Pc;
    };
    for (int i = 0; i < n; ++i) {
        size_t& r = rows[i % BATCH_STREAMS];
        r = std::max(r, repack_bytes(B[i].P));
        Work w{};
        B[i].off = total;
        total += carve(own(i), nullptr, &w, 0, true, false);
        total = (total + 255) / 256 * 256;
    }
    Carver pc{nullptr};
    int* big_pool = nullptr;
    char* repack[BATCH_STREAMS];
    auto pool_layout = [&](Carver& c) {
        for (int k = 0; k < BATCH_STREAMS; ++k) repack[k] = c.take<char>(rows[k]);
        big_pool = c.take<int>((size_t)big.nslot * big_ints(big));
        S.d_L = c.take<LinkBufs>(std::max(1, S.nlink));
        S.d_stat = c.take<unsigned long long>(12);
        S.d_passes = c.take<int>(1);
        S.d_status = c.take<int>(8 * (size_t)n);
    };
    pool_layout(pc);
    const size_t pool_bytes = pc.off + 256;
    const size_t need = total + pool_bytes;
    {
        // the batch must fit beside the caller's data: tighter first
        // candidate capacities (overflowing movies are rerun alone)
        size_t free_b = 0, total_b = 0;
        CK(cudaMemGetInfo(&free_b, &total_b));
        const size_t avail = free_b + (ctx->arena ? ctx->arena_size : 0);
        if (need > avail - avail / 8) {
            if (ctx->batch_cap_div < 1024) {
                ctx->batch_cap_div *= 4;
                return batch_many(ctx, mv, n, st);
            }
            ctx->err = "the batch does not fit in device memory; split it";
            return GT_ERR_OOM;
        }
    }
    int rc = ensure_arena(ctx, need);
    if (rc) return rc;
    {
        char buf[96];
        std::snprintf(buf, sizeof(buf), "arena %p %p %d %d %d", (void*)ctx->arena, (void*)st, ctx->force_generic,
                      ctx->tune_disabled, ctx->batch_cap_div);
        key += buf;
    }
    Carver c2{ctx->arena + total};
    pool_layout(c2);
    for (int i = 0; i < n; ++i) {
        carve(own(i), ctx->arena + B[i].off, &B[i].w, 0, true, false);
        B[i].w.repack = repack[i % BATCH_STREAMS];
    }
    const bool replay = ctx->batch_exec && key == ctx->batch_key;
    // constant tables and linker descriptors (other calls may have reused
    // the arena since the graph was built)
    for (int i = 0; i < n; ++i) {
        rc = upload_tables(ctx, B[i].P, B[i].w, st);
        if (rc) return rc;
    }
    std::vector<LinkBufs> hL(std::max(1, S.nlink));
    if (S.nlink > 0) {
        for (int i = 0; i < n; ++i) {
            if (B[i].link_slot < 0) continue;
            LinkBufs L = link_bufs(B[i].P, B[i].w, ctx->subnet_budget);
            L.nslot = big.nslot; L.big_d = big.big_d; L.big_s = big.big_s; L.big_e = big.big_e;
            L.big_ints = big_ints(big); L.big = big_pool;
            hL[B[i].link_slot] = L;
        }
        CK(cudaMemcpyAsync(S.d_L, hL.data(), sizeof(LinkBufs) * S.nlink, cudaMemcpyHostToDevice, st));
    }
    if (!replay) {
        ctx->batch_key.clear();
        // autotuned tile rows (timed on this movie's frames and workspace)
        for (int i = 0; i < n; ++i)
            if (B[i].P.fast == 1) {
                rc = tune_tile_rows(ctx, B[i], mv[i].frames, st);
                if (rc) return rc;
            }
        CK(allow_shared<locate_tiles_kernel>());
            CK(cudaEventRecord(ctx->ev[0], st));
        rc = enqueue_batch(ctx, B, mv, n, S, st);
        if (rc) return rc;
        CK(cudaEventRecord(ctx->ev[1], st));
        // The batch runs as plain launches (they hide behind the first
        // movies' kernels); the graph that later calls replay is captured and
        // instantiated while the device works.  Building it first kept the
        // device idle for that time: 12 movies of 120 frames up to 1024 x 1024
        // in new buffers 4.6 -> 3.3 ms a call.
        // Where capture is refused, later calls launch the same way.
        cudaGraph_t graph = nullptr;
        bool captured = false;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
            BatchShared Sc = S;
            const int erc = enqueue_batch(ctx, B, mv, n, Sc, st);
            const cudaError_t ee = cudaStreamEndCapture(st, &graph);
            if (erc == GT_OK && ee == cudaSuccess && graph) {
                // the last batch's graph takes the new arguments if it has the
                // same nodes and edges, else it is built anew
                cudaGraphExecUpdateResultInfo info;
                if (ctx->batch_exec && cudaGraphExecUpdate(ctx->batch_exec, graph, &info) != cudaSuccess) {
                    cudaGetLastError();
                    cudaGraphExecDestroy(ctx->batch_exec);
                    ctx->batch_exec = nullptr;
                }
                captured = ctx->batch_exec || cudaGraphInstantiate(&ctx->batch_exec, graph, 0) == cudaSuccess;
                if (captured) ctx->batch_key = key;
                else ctx->batch_exec = nullptr;
            }
            if (graph) cudaGraphDestroy(graph);
        }
        if (captured) {
            ctx->stats.batch_graph = 1;
        } else {
            cudaGetLastError();
            ctx->err.clear();
        }
    } else {
        CK(cudaEventRecord(ctx->ev[0], st));
        CK(cudaGraphLaunch(ctx->batch_exec, st));
        CK(cudaEventRecord(ctx->ev[1], st));
        ctx->stats.batch_graph = 2;
        // launches of the captured sequence
        int cnt = 0;
        for (int i = 0; i < n; ++i) {
            const Plan& P = B[i].P;
            cnt += (P.repack ? 2 * ((P.T + P.repack - 1) / P.repack) : (P.T + 65534) / 65535) + 2 + (P.link ? 2 : 0) + 1;
        }
        S.launches = cnt + (S.nlink > 0 ? 1 : 0);
    }
    CK(cudaStreamSynchronize(st));
    cudaEventElapsedTime(&ctx->stats.ms_total, ctx->ev[0], ctx->ev[1]);
    ctx->stats.launches = S.launches;
    if (S.nlink > 0) {
        int passes = 0;
        CK(cudaMemcpy(&passes, S.d_passes, sizeof(int), cudaMemcpyDeviceToHost));
        ctx->stats.link_iterations = passes;
    }
    // per-movie status; capacity overflows are rerun through the plain path
    std::vector<int> status(ctx->h_status, ctx->h_status + 8 * (size_t)n);
    gt_stats keep = ctx->stats;
    int fallbacks = 0;
    int64_t rows_total = 0;
    for (int i = 0; i < n; ++i) {
        const int bits = status[8 * i];
        bool retry = false;
        rc = err_status(ctx, bits, &retry);
        if (rc && !retry) { ctx->err = "movie " + std::to_string(i) + ": " + ctx->err; return rc; }
        if (rc && retry) {
            ++fallbacks;
            int64_t nr = 0;
            rc = batch_common(ctx, mv[i].frames, false, mv[i].dtype, mv[i].T, mv[i].H, mv[i].W, &mv[i].params,
                              nullptr, mv[i].out, mv[i].out_rows, &nr, st);
            if (rc) { ctx->err = "movie " + std::to_string(i) + ": " + ctx->err; return rc; }
            mv[i].nrows = nr;
        } else {
            mv[i].nrows = status[8 * i + 4];
        }
        rows_total += mv[i].nrows;
    }
    ctx->err.clear();
    ctx->stats = keep;
    ctx->stage_times = 0;
    ctx->stats.batch_fallbacks = fallbacks;
    ctx->stats.particles = rows_total;
    return GT_OK;
}

// Parameters of the gt_adjoint_* calls: the forward weights exactly as
// make_plan derives them, the normalised taps a_i = w_i / sum(w) and
// da_i / ds in double precision, and the centroid circle in the order of
// the centroid loop (i outer, j inner, float mask <= r^2).
int adjoint_setup(gt_ctx* ctx, const float* d_frames, int T, int H, int W, const gt_params* params,
                  const int32_t* d_walk, int64_t n, AdjParams* ap, std::vector<int>* circ) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    ctx->stats = gt_stats{};
    ctx->stage_times = 0;
    if (!d_frames || !params || T < 1 || H < 1 || W < 1 || n < 0 || (n > 0 && !d_walk)) {
        ctx->err = "invalid frames/shape/walk";
        return GT_ERR_ARG;
    }
    if ((long long)H * W > (1LL << 28) || H > 65535 || W > 65535) { ctx->err = "frame too large"; return GT_ERR_ARG; }
    Resolved r;
    int rc = resolve(params, &r, &ctx->err);
    if (rc) return rc;
    if (r.max_iterations < 1) {
        ctx->err = "the adjoint needs max_iterations >= 1";
        return GT_ERR_UNSUPPORTED;
    }
    if (r.diameter > 31) {
        ctx->err = "the adjoint supports diameter <= 31";
        return GT_ERR_UNSUPPORTED;
    }
    std::memset(ap, 0, sizeof(*ap));
    ap->T = T; ap->H = H; ap->W = W;
    const int k = (int)r.smoothing_size;
    ap->krad = k / 2;
    if (H <= ap->krad || W <= ap->krad) { ctx->err = "frame smaller than the smoothing window"; return GT_ERR_ARG; }
    const float sigma2 = r.noise_size;
    if (!(sigma2 > 0.0f)) { ctx->err = "noise_size must be > 0"; return GT_ERR_ARG; }
    gauss_taps(k, sigma2, ctx->normalized_taps, ap->w, &ap->norm, &ap->rn);
    double sw = 0.0, swi = 0.0;
    for (int i = -ap->krad; i <= ap->krad; ++i) {
        const double gd = std::exp(-(double)i * i / (2.0 * sigma2));
        sw += gd;
        swi += gd * i * i;
    }
    ap->kk = (float)(k * k);
    ap->rkk = 1.0f / ap->kk;
    const double s2 = (double)sigma2 * sigma2;
    for (int i = -ap->krad; i <= ap->krad; ++i) {
        const double ai = std::exp(-(double)i * i / (2.0 * sigma2)) / sw;
        ap->a[i + ap->krad] = (float)ai;
        // d/ds [exp(-i^2 / 2s) / sum_j exp(-j^2 / 2s)] = a_i (i^2 - <j^2>) / (2 s^2)
        ap->da[i + ap->krad] = (float)(ai * ((double)i * i - swi / sw) / (2.0 * s2));
    }
    ap->k = (float)k;
    ap->rc = ((int)r.diameter - 1) / 2;
    ap->border = (int)r.diameter / 2;
    circ->clear();
    const float rr = (float)ap->rc;
    const float r2 = rr * rr;
    for (int i = -ap->rc; i <= ap->rc; ++i)
        for (int j = -ap->rc; j <= ap->rc; ++j) {
            const float x = (float)i, y = (float)j;
            if (x * x + y * y > r2) continue;
            circ->push_back(i);
            circ->push_back(j);
        }
    ap->K = (int)circ->size() / 2;
    ap->gain = 1.0f;
    ap->read_var = 0.0f;
    CK(cudaSetDevice(ctx->device));
    return GT_OK;
}

// Scratch of the gt_adjoint_* calls in the context arena: the error word,
// the circle table and (backward only) the partial parameter gradients and the
// tile lists of a chunk of peaks.
struct AdjWork {
    int* err;
    int* circ;
    double* gpart;
    AdjTiles tl{};
    int64_t chunk = 0;  // peaks per chunk
};

int adjoint_work(gt_ctx* ctx, const AdjParams& ap, const std::vector<int>& circ, int64_t n_back, AdjWork* aw,
                 cudaStream_t st) {
    auto layout = [&](char* base) {
        Carver c{base};
        aw->err = c.take<int>(1);
        aw->circ = c.take<int>(circ.size());
        aw->gpart = c.take<double>(2 * (size_t)adjoint_particle_blocks_max(ctx->num_sms));
        if (n_back >= 0) {
            adjoint_tiles(ap, &aw->tl);
            // up to 2^23 peaks and 1 GB of dL/dR at a time
            aw->chunk = std::min<int64_t>({std::max<int64_t>(n_back, 1), (int64_t)1 << 23,
                                           std::max<int64_t>(1, ((int64_t)1 << 28) / ap.K)});
            aw->tl.g = c.take<float>((size_t)aw->chunk * ap.K);
            aw->tl.next = c.take<int>((size_t)aw->chunk * aw->tl.slots);
            const size_t tiles = (size_t)ap.T * aw->tl.nty * aw->tl.ntx;
            aw->tl.count = c.take<int>(2 * tiles);  // and the lists' heads
            aw->tl.head = aw->tl.count + tiles;
            aw->tl.peaks = c.take<int>(tiles * TILE_PEAKS);
        }
        return c.off + 256;
    };
    const int rc = ensure_arena(ctx, layout(nullptr));
    if (rc) return rc;
    layout(ctx->arena);
    CK(cudaMemsetAsync(aw->err, 0, sizeof(int), st));
    CK(cudaMemcpyAsync(aw->circ, circ.data(), sizeof(int) * circ.size(), cudaMemcpyHostToDevice, st));
    for (int i = 0; i < 3; ++i)
        if (!ctx->ev[i]) CK(cudaEventCreate(&ctx->ev[i]));
    return GT_OK;
}

int adjoint_finish(gt_ctx* ctx, const AdjWork& aw, cudaStream_t st) {
    int herr = 0;
    CK(ctx->hc.download(&herr, aw.err, sizeof(int), st));
    if (herr) {
        ctx->err = "a walk record lies outside the frames";
        return GT_ERR_ARG;
    }
    return GT_OK;
}
}  // namespace

namespace {
// The stream of a call on device pointers.  NULL is the context's stream, which
// does not wait for the legacy default stream by itself: what that holds (torch
// passes NULL for it) may still be writing the call's inputs or reading the
// memory of its outputs.
cudaStream_t call_stream(gt_ctx* ctx, void* stream) {
    if (stream || !ctx) return (cudaStream_t)stream;
    // While a stream that synchronises with the default stream is captured, a
    // record there would end the capture: the query does not, and the call runs
    // without the wait.
    cudaStreamCaptureStatus cap;
    if (cudaSetDevice(ctx->device) != cudaSuccess || cudaStreamIsCapturing(cudaStreamLegacy, &cap) != cudaSuccess ||
        (!ctx->lev && cudaEventCreateWithFlags(&ctx->lev, cudaEventDisableTiming) != cudaSuccess) ||
        cudaEventRecord(ctx->lev, cudaStreamLegacy) != cudaSuccess ||
        cudaStreamWaitEvent(ctx->stream, ctx->lev, 0) != cudaSuccess)
        cudaGetLastError();
    return ctx->stream;
}

thread_local std::string g_noctx_err;  // errors of calls made without a context
}

namespace gt {
void set_noctx_error(const char* msg) { g_noctx_err = msg; }
}  // namespace gt

extern "C" {

const char* gt_version(void) { return "gt-b200 0.1.0 (sm_100a)"; }

int gt_ctx_create(int device, gt_ctx** out) {
    if (!out) return GT_ERR_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) return GT_ERR_CUDA;
    gt_ctx* c = new gt_ctx();
    c->device = device;
    if (cudaSetDevice(device) != cudaSuccess) { delete c; return GT_ERR_CUDA; }
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) { delete c; return GT_ERR_CUDA; }
    cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
    *out = c;
    return GT_OK;
}

void gt_ctx_destroy(gt_ctx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->arena) cudaFree(ctx->arena);
    if (ctx->batch_exec) cudaGraphExecDestroy(ctx->batch_exec);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    for (auto& e : ctx->cev)
        if (e) cudaEventDestroy(e);
    if (ctx->h_status) cudaFreeHost(ctx->h_status);
    if (ctx->h_frames) cudaFreeHost(ctx->h_frames);
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    for (auto& sd : ctx->side)
        if (sd) cudaStreamDestroy(sd);
    for (auto& e : ctx->bev)
        if (e) cudaEventDestroy(e);
    for (auto& e : ctx->ev)
        if (e) cudaEventDestroy(e);
    if (ctx->lev) cudaEventDestroy(ctx->lev);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

const char* gt_last_error(const gt_ctx* ctx) {
    if (ctx) return ctx->err.c_str();
    return g_noctx_err.c_str();
}

int gt_column_names(const gt_params* params, char* buf, size_t buflen) {
    if (!params || !buf) return -GT_ERR_ARG;
    g_noctx_err.clear();
    Resolved r;
    int rc = resolve(params, &r, &g_noctx_err);
    if (rc) return -rc;
    std::vector<std::string> names, types;
    column_list(r, names, types);
    std::string s;
    for (size_t i = 0; i < names.size(); ++i) {
        if (i) s += ",";
        s += names[i] + ":" + types[i];
    }
    if (s.size() + 1 > buflen) return -GT_ERR_ARG;
    std::memcpy(buf, s.c_str(), s.size() + 1);
    return (int)names.size();
}

int gt_batch(gt_ctx* ctx, const void* frames, int dtype, int T, int H, int W, const gt_params* params,
             gt_table* out) {
    if (!out) return GT_ERR_ARG;
    out->data = nullptr;
    out->nrows = 0;
    out->ncols = 0;
    return batch_common(ctx, frames, true, dtype, T, H, W, params, out, nullptr, 0, nullptr,
                        ctx ? ctx->stream : nullptr);
}

int gt_file_info(const char* path, int has_channel, uint32_t channel, int32_t* T, int32_t* H, int32_t* W) {
    g_noctx_err.clear();
    if (!T || !H || !W) { g_noctx_err = "null output"; return GT_ERR_ARG; }
    gt::MovieFile mf;
    std::string msg;
    const int rc = mf.open(path, has_channel != 0, channel, &msg);
    if (rc) { g_noctx_err = msg; return rc == 2 ? GT_ERR_UNSUPPORTED : GT_ERR_ARG; }
    *T = mf.T; *H = mf.H; *W = mf.W;
    return GT_OK;
}

int gt_file_read(const char* path, int has_channel, uint32_t channel, uint16_t* out, int64_t max_values) {
    g_noctx_err.clear();
    gt::MovieFile mf;
    std::string msg;
    const int rc = mf.open(path, has_channel != 0, channel, &msg);
    if (rc) { g_noctx_err = msg; return rc == 2 ? GT_ERR_UNSUPPORTED : GT_ERR_ARG; }
    const int64_t fpx = (int64_t)mf.H * mf.W;
    if (!out || max_values < fpx * mf.T) { g_noctx_err = "output buffer too small"; return GT_ERR_ARG; }
    for (int t = 0; t < mf.T; ++t)
        if (mf.read_frame(t, out + fpx * t, &msg)) { g_noctx_err = msg; return GT_ERR_ARG; }
    return GT_OK;
}

int gt_ets_channels(const char* path, int32_t* channels, int32_t* frames, int32_t max_channels, int32_t* nchannels,
                    int32_t* dim0, int32_t* dim1) {
    g_noctx_err.clear();
    if (!nchannels || !dim0 || !dim1 || (max_channels > 0 && (!channels || !frames))) {
        g_noctx_err = "null output";
        return GT_ERR_ARG;
    }
    std::vector<std::pair<uint32_t, int>> ch;
    uint32_t dims[2];
    std::string msg;
    if (gt::ets_channels(path, &ch, dims, &msg)) { g_noctx_err = msg; return GT_ERR_ARG; }
    *nchannels = (int32_t)ch.size();
    *dim0 = (int32_t)dims[0];
    *dim1 = (int32_t)dims[1];
    for (int i = 0; i < (int)ch.size() && i < max_channels; ++i) {
        channels[i] = (int32_t)ch[i].first;
        frames[i] = ch[i].second;
    }
    return GT_OK;
}

int gt_batch_file(gt_ctx* ctx, const char* path, int has_channel, uint32_t channel, const gt_params* params,
                  gt_table* out) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    if (!params || !out) { ctx->err = "null params/output"; return GT_ERR_ARG; }
    gt::MovieFile mf;
    std::string msg;
    int rc = mf.open(path, has_channel != 0, channel, &msg);
    if (rc) { ctx->err = msg; return rc == 2 ? GT_ERR_UNSUPPORTED : GT_ERR_ARG; }
    const size_t fpx = (size_t)mf.H * mf.W, npx = fpx * mf.T;
    CK(cudaSetDevice(ctx->device));
    if (ctx->h_frames_n < npx) {
        if (ctx->h_frames) cudaFreeHost(ctx->h_frames);
        ctx->h_frames = nullptr;
        ctx->h_frames_n = 0;
        CK(cudaHostAlloc((void**)&ctx->h_frames, sizeof(uint16_t) * npx, cudaHostAllocDefault));
        ctx->h_frames_n = npx;
    }
    // frames are decoded by a pool of host threads into pinned memory; each
    // chunk's upload (and its locate launch) waits for its own frames only
    const int T = mf.T;
    std::vector<std::atomic<unsigned char>> done(T);
    for (auto& d : done) d.store(0);
    std::atomic<int> next{0}, failed{0};
    std::mutex mu;
    std::condition_variable cv;
    std::string err;
    uint16_t* dst = ctx->h_frames;
    auto worker = [&]() {
        std::string m;
        for (int t = next.fetch_add(1); t < T && !failed.load(); t = next.fetch_add(1)) {
            if (mf.read_frame(t, dst + fpx * t, &m)) {
                std::lock_guard<std::mutex> lk(mu);
                if (!failed.exchange(1)) err = m;
                cv.notify_all();
                return;
            }
            done[t].store(1);
            std::lock_guard<std::mutex> lk(mu);
            cv.notify_all();
        }
    };
    const int nthr = (int)std::max(1u, std::min<unsigned>({std::thread::hardware_concurrency(), 16u, (unsigned)T}));
    std::vector<std::thread> pool;
    for (int i = 0; i < nthr; ++i) pool.emplace_back(worker);
    const std::function<int(int, int)> ready = [&](int f0, int nf) -> int {
        std::unique_lock<std::mutex> lk(mu);
        for (int t = f0; t < f0 + nf; ++t) {
            cv.wait(lk, [&] { return done[t].load() || failed.load(); });
            if (failed.load()) return GT_ERR_ARG;
        }
        return GT_OK;
    };
    rc = batch_common(ctx, dst, true, GT_U16, T, mf.H, mf.W, params, out, nullptr, 0, nullptr, ctx->stream, nullptr,
                      &ready);
    failed.store(failed.load() | (rc ? 2 : 0));
    for (auto& th : pool) th.join();
    if (rc == GT_ERR_ARG && !err.empty()) ctx->err = err;
    return rc;
}

int gt_batch_device(gt_ctx* ctx, const void* d_frames, int dtype, int T, int H, int W,
                    const gt_params* params, float* d_out, int64_t out_rows, int64_t* nrows, void* stream) {
    cudaStream_t st = call_stream(ctx, stream);
    return batch_common(ctx, d_frames, false, dtype, T, H, W, params, nullptr, d_out, out_rows, nrows, st);
}

int gt_batch_device_walk(gt_ctx* ctx, const void* d_frames, int dtype, int T, int H, int W,
                         const gt_params* params, float* d_out, int64_t out_rows, int64_t* nrows, int32_t* d_walk,
                         void* stream) {
    if (ctx && !d_walk && out_rows > 0) {
        ctx->err = "null walk buffer";
        return GT_ERR_ARG;
    }
    cudaStream_t st = call_stream(ctx, stream);
    return batch_common(ctx, d_frames, false, dtype, T, H, W, params, nullptr, d_out, out_rows, nrows, st,
                        (int*)d_walk);
}

int gt_adjoint_forward(gt_ctx* ctx, const float* d_frames, int T, int H, int W, const gt_params* params,
                       const int32_t* d_walk, int64_t n, float* d_yxm, void* stream) {
    AdjParams ap;
    std::vector<int> circ;
    int rc = adjoint_setup(ctx, d_frames, T, H, W, params, d_walk, n, &ap, &circ);
    if (rc) return rc;
    if (n > 0 && !d_yxm) { ctx->err = "null output"; return GT_ERR_ARG; }
    cudaStream_t st = call_stream(ctx, stream);
    AdjWork aw;
    rc = adjoint_work(ctx, ap, circ, -1, &aw, st);
    if (rc) return rc;
    CK(cudaEventRecord(ctx->ev[0], st));
    CK(launch_adjoint_particles(0, ap, d_frames, d_walk, n, aw.circ, nullptr, d_yxm, aw.tl, nullptr, nullptr, aw.err, 0,
                                ctx->num_sms, st));
    CK(cudaEventRecord(ctx->ev[1], st));
    ctx->stats.launches = n > 0 ? 1 : 0;
    rc = adjoint_finish(ctx, aw, st);
    cudaEventElapsedTime(&ctx->stats.ms_adjoint_particles, ctx->ev[0], ctx->ev[1]);
    ctx->stats.ms_total = ctx->stats.ms_adjoint_particles;
    return rc;
}

int gt_adjoint_backward(gt_ctx* ctx, const float* d_frames, int T, int H, int W, const gt_params* params,
                        const int32_t* d_walk, int64_t n, const float* d_grad_yxm, float* d_grad_frames,
                        double* d_grad_params, void* stream) {
    AdjParams ap;
    std::vector<int> circ;
    int rc = adjoint_setup(ctx, d_frames, T, H, W, params, d_walk, n, &ap, &circ);
    if (rc) return rc;
    if (!d_grad_frames || !d_grad_params || (n > 0 && !d_grad_yxm)) { ctx->err = "null output"; return GT_ERR_ARG; }
    cudaStream_t st = call_stream(ctx, stream);
    AdjWork aw;
    rc = adjoint_work(ctx, ap, circ, n, &aw, st);
    if (rc) return rc;
    for (int i = 0; i < 4; ++i)
        if (!ctx->ev[i]) CK(cudaEventCreate(&ctx->ev[i]));
    if (n == 0) CK(cudaMemsetAsync(d_grad_params, 0, 2 * sizeof(double), st));
    const size_t heads = 2 * sizeof(int) * (size_t)T * aw.tl.nty * aw.tl.ntx;
    ctx->stats.launches = 0;
    // the peaks in chunks (one, unless there are millions); the dense part is
    // the empty lists plus the transposed bandpass.  Times: the last chunk's
    int64_t k0 = 0;
    do {
        const int64_t nk = std::min<int64_t>(aw.chunk, n - k0);
        const int add = k0 > 0;
        CK(cudaEventRecord(ctx->ev[0], st));
        CK(cudaMemsetAsync(aw.tl.count, 0, heads, st));
        CK(cudaEventRecord(ctx->ev[1], st));
        CK(launch_adjoint_particles(1, ap, d_frames, d_walk + 5 * k0, nk, aw.circ, d_grad_yxm + 3 * k0, nullptr, aw.tl,
                                    d_grad_params, aw.gpart, aw.err, add, ctx->num_sms, st));
        CK(cudaEventRecord(ctx->ev[2], st));
        CK(launch_adjoint_transpose(ap, aw.tl, d_walk + 5 * k0, aw.circ, d_grad_frames, add, st));
        CK(cudaEventRecord(ctx->ev[3], st));
        ctx->stats.launches += (nk > 0 ? 2 : 0) + (T + 65534) / 65535;
        k0 += nk;
    } while (k0 < n);
    rc = adjoint_finish(ctx, aw, st);
    cudaEventElapsedTime(&ctx->stats.ms_adjoint_particles, ctx->ev[1], ctx->ev[2]);
    float tz = 0.f, tt = 0.f;
    cudaEventElapsedTime(&tz, ctx->ev[0], ctx->ev[1]);
    cudaEventElapsedTime(&tt, ctx->ev[2], ctx->ev[3]);
    ctx->stats.ms_adjoint_dense = tz + tt;
    cudaEventElapsedTime(&ctx->stats.ms_total, ctx->ev[0], ctx->ev[3]);
    return rc;
}

int gt_adjoint_uncertainty(gt_ctx* ctx, const float* d_frames, int T, int H, int W, const gt_params* params,
                           const int32_t* d_walk, int64_t n, float gain, float read_noise, float* d_sd,
                           void* stream) {
    AdjParams ap;
    std::vector<int> circ;
    int rc = adjoint_setup(ctx, d_frames, T, H, W, params, d_walk, n, &ap, &circ);
    if (rc) return rc;
    if (n > 0 && !d_sd) { ctx->err = "null output"; return GT_ERR_ARG; }
    if (!(gain >= 0.0f) || !(read_noise >= 0.0f) || !std::isfinite(gain) || !std::isfinite(read_noise)) {
        ctx->err = "gain and read_noise must be finite and >= 0";
        return GT_ERR_ARG;
    }
    ap.gain = gain;
    ap.read_var = read_noise * read_noise;
    cudaStream_t st = call_stream(ctx, stream);
    AdjWork aw;
    rc = adjoint_work(ctx, ap, circ, -1, &aw, st);
    if (rc) return rc;
    CK(cudaEventRecord(ctx->ev[0], st));
    CK(launch_adjoint_particles(2, ap, d_frames, d_walk, n, aw.circ, nullptr, d_sd, aw.tl, nullptr, nullptr, aw.err, 0,
                                ctx->num_sms, st));
    CK(cudaEventRecord(ctx->ev[1], st));
    ctx->stats.launches = n > 0 ? 1 : 0;
    rc = adjoint_finish(ctx, aw, st);
    cudaEventElapsedTime(&ctx->stats.ms_adjoint_particles, ctx->ev[0], ctx->ev[1]);
    ctx->stats.ms_total = ctx->stats.ms_adjoint_particles;
    return rc;
}

int gt_batch_many_device(gt_ctx* ctx, gt_movie* movies, int n, void* stream) {
    cudaStream_t st = call_stream(ctx, stream);
    if (ctx) ctx->batch_cap_div = ctx->short_memory ? 256 : 64;
    return batch_many(ctx, movies, n, st);
}

int gt_ctx_set_option(gt_ctx* ctx, const char* key, int value) {
    if (!ctx || !key) return GT_ERR_ARG;
    const std::string k(key);
    if (k == "locate_tile_rows" && (value == 32 || value == 64)) { ctx->fast_tile_rows = value; return GT_OK; }
    if (k == "force_generic" && (value == 0 || value == 1)) { ctx->force_generic = value; return GT_OK; }
    if (k == "autotune" && (value == 0 || value == 1)) { ctx->tune_disabled = !value; return GT_OK; }
    if (k == "subnet_budget" && value > 0) { ctx->subnet_budget = value; return GT_OK; }
    if (k == "subnet_budget" && value == 0) { ctx->subnet_budget = SUBNET_BUDGET; return GT_OK; }
    if (k == "test_withhold_tile_copy" && (value == 0 || value == 1)) { ctx->withhold_tma = value; return GT_OK; }
    if (k == "test_short_memory" && (value == 0 || value == 1)) { ctx->short_memory = value; return GT_OK; }
    if (k == "locate_tiles_per_cta" && value >= 0 && value <= 64) {
        ctx->tiles_per_cta = value;
        drop_batch_graph(ctx);  // it holds the old launch shape
        return GT_OK;
    }
    if (k == "normalized_taps" && (value == 0 || value == 1)) {
        ctx->normalized_taps = value;
        drop_batch_graph(ctx);  // it holds the old taps
        return GT_OK;
    }
    ctx->err = "unknown option or value: " + k;
    return GT_ERR_ARG;
}

void gt_table_free(gt_table* table) {
    if (table && table->data) { table_release(table->data); table->data = nullptr; }
}

namespace {
// trajectory entry points share the argument checks
int traj_begin(gt_ctx* ctx, int64_t n, bool ok_ptrs) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    ctx->stats = gt_stats{};
    ctx->stage_times = 0;
    if (n < 0 || (n > 0 && !ok_ptrs)) {
        ctx->err = "invalid arrays";
        return GT_ERR_ARG;
    }
    if (n >= ((int64_t)1 << 31)) {
        ctx->err = "table too large";
        return GT_ERR_ARG;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) {
        ctx->err = "cudaSetDevice failed";
        return GT_ERR_CUDA;
    }
    return GT_OK;
}
}  // namespace

int gt_filter_stubs(gt_ctx* ctx, const int64_t* ids, int64_t n, int64_t threshold, uint8_t* keep, int64_t* count,
                    int64_t* nkept) {
    int rc = traj_begin(ctx, n, ids && keep && nkept);
    if (rc || !nkept) return rc ? rc : GT_ERR_ARG;
    *nkept = 0;
    if (n == 0) return GT_OK;
    ctx->traj.hc = &ctx->hc;
    const TrajEnd end{ctx->traj};
    return traj_filter_stubs(ids, n, threshold, keep, count, nkept, ctx->traj, ctx->stream, ctx->num_sms, &ctx->err);
}

int gt_steps(gt_ctx* ctx, const int64_t* ids, const float* x, const float* y, int64_t n, double mpp, float* xs,
             float* ys, double* x_step, double* y_step, double* steplength, int64_t* order) {
    int rc = traj_begin(ctx, n, ids && x && y && xs && ys && x_step && y_step && steplength && order);
    if (rc) return rc;
    if (n == 0) return GT_OK;
    ctx->traj.hc = &ctx->hc;
    const TrajEnd end{ctx->traj};
    return traj_steps(ids, x, y, n, (float)mpp, xs, ys, x_step, y_step, steplength, order, ctx->traj, ctx->stream,
                      ctx->num_sms, &ctx->err);
}

int gt_imsd(gt_ctx* ctx, const int64_t* ids, const int64_t* frames, const float* x, const float* y, int64_t n,
            double mpp, int64_t max_lagtime, gt_table* out) {
    if (!out) return GT_ERR_ARG;
    out->data = nullptr;
    out->nrows = 0;
    out->ncols = 0;
    int rc = traj_begin(ctx, n, ids && frames && x && y);
    if (rc) return rc;
    float* data = nullptr;
    int64_t m = 0;
    float ms = 0.f;
    if (n > 0) {
        ctx->traj.hc = &ctx->hc;
        const TrajEnd end{ctx->traj};
        rc = traj_imsd(ids, frames, x, y, n, (float)mpp, max_lagtime, table_alloc, &data, &m, &ms, ctx->traj, ctx->stream,
                       ctx->num_sms, &ctx->err);
        if (rc) {
            if (data) table_release(data);
            return rc;
        }
    } else {
        data = table_alloc(sizeof(float) * 3);
        if (!data) { ctx->err = "host allocation failed"; return GT_ERR_OOM; }
    }
    ctx->stats.ms_msd = ms;
    out->data = data;
    out->nrows = m;
    out->ncols = 3;
    std::memset(out->names, 0, sizeof(out->names));
    std::memset(out->types, 0, sizeof(out->types));
    const char* names[3] = {"lag", "particle", "msd"};
    for (int i = 0; i < 3; ++i) {
        std::snprintf(out->names[i], sizeof(out->names[i]), "%s", names[i]);
        std::snprintf(out->types[i], sizeof(out->types[i]), "%s", i < 2 ? "int" : "float");
    }
    return GT_OK;
}

int gt_last_stats(const gt_ctx* ctx, gt_stats* out) {
    if (!ctx || !out) return GT_ERR_ARG;
    *out = ctx->stats;
    if (ctx->stage_times) {
        cudaEventElapsedTime(&out->ms_locate, ctx->ev[0], ctx->ev[1]);
        cudaEventElapsedTime(&out->ms_finalize, ctx->ev[1], ctx->ev[2]);
        cudaEventElapsedTime(&out->ms_link, ctx->ev[2], ctx->ev[3]);
        cudaEventElapsedTime(&out->ms_assemble, ctx->ev[3], ctx->ev[4]);
        cudaEventElapsedTime(&out->ms_total, ctx->ev[0], ctx->ev[4]);
    }
    return GT_OK;
}

int gt_link(gt_ctx* ctx, const float* rows, int64_t n, int ncols, float search_range, int has_memory,
            uint32_t memory, uint64_t* ids) {
    if (!ctx) return GT_ERR_ARG;
    ctx->err.clear();
    ctx->stats = gt_stats{};
    ctx->stage_times = 0;
    if ((!rows && n > 0) || ncols < 4 || n < 0 || (n > 0 && !ids)) { ctx->err = "invalid table"; return GT_ERR_ARG; }
    if (!(search_range > 0.0f && search_range < 4096.0f)) { ctx->err = "search_range must be in (0, 4096)"; return GT_ERR_ARG; }
    if (n == 0) return GT_OK;
    if (n > (1LL << 30)) { ctx->err = "table too large"; return GT_ERR_ARG; }
    const uint32_t mem = has_memory ? memory : 0;
    CK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    LinkTable tab;
    ctx->traj.hc = &ctx->hc;
    const TrajEnd end{ctx->traj};
    int rc = table_load(rows, (int)n, ncols, ctx->traj, st, ctx->num_sms, &tab, &ctx->err);
    if (rc) return rc;
    const int T = tab.T;
    for (int scale = 1; scale <= 64; scale *= 4) {
        Plan P;
        P.T = T;
        P.link = 1;
        P.r = Resolved{};
        P.r.has_search_range = 1;
        P.r.search_range = search_range;
        P.r.memory = std::min<uint32_t>(mem, (uint32_t)T);  // no entry is older than the table
        P.cap_p = tab.largest;
        // cells of absolute positions; negative coordinates clamp into the
        // first cell (clamping is monotone, so neighbours stay adjacent)
        const double ext = (double)std::max(tab.ymax, tab.xmax) + 1.0;
        // at most 200 x 200 of them and about 16 a particle of the largest
        // frame (32 x 32 at least): every frame has its own, and 1.2 million
        // frames of one particle would want 194 GB of 200 x 200
        const double side = std::min(200.0, std::max(32.0, std::ceil(std::sqrt(16.0 * tab.largest))));
        P.LG = std::max({(int)std::ceil(search_range) + 1, 8, (int)std::ceil(ext / side)});
        P.lncy = (int)(tab.ymax / P.LG) + 1;
        P.lncx = (int)(tab.xmax / P.LG) + 1;
        link_scratch(&P, scale);
        P.cap_c = 1;
        Work w{};
        const size_t need = carve(P, nullptr, &w, 0, false);
        rc = ensure_arena(ctx, need);
        if (rc) return rc;
        carve(P, ctx->arena, &w, 0, false);
        CK(table_slabs(tab, P.cap_p, w.py, w.px, w.npart, ctx->num_sms, st));
        CK(cudaMemsetAsync(w.status, 0, sizeof(int) * STATUS_INTS, st));
        CK(allow_shared<grid_kernel>());
        grid_kernel<<<T, 512, sizeof(int) * (size_t)P.lncx * P.lncy, st>>>(w.py, w.px, w.npart, P.cap_p, P.LG,
                                                                        P.lncy, P.lncx, w.gstart, w.gidx, w.gpos);
        CK(cudaGetLastError());
        scan_frames_kernel<<<1, 1024, 0, st>>>(w.npart, w.off, T);
        rc = run_link(ctx, P, w, st);
        if (rc) return rc;
        // ids in row order: compact index g == row index
        CK(table_ids(tab, w.root, w.newid, ctx->num_sms, st));
        // the error bits arrive before the ids: one wait for both
        if (!ctx->h_stage) {
            CK(cudaHostAlloc((void**)&ctx->h_stage, sizeof(int) * STATUS_INTS, cudaHostAllocDefault));
            ctx->h_stage_n = STATUS_INTS;
        }
        CK(cudaMemcpyAsync(ctx->h_stage, w.err, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(ctx->hc.download(ids, tab.ids, sizeof(uint64_t) * (size_t)n, st));
        bool retry;
        rc = err_status(ctx, ctx->h_stage[0], &retry);
        if (rc && retry && scale < 64) continue;
        if (rc) return rc;
        ctx->stats.particles = n;
        return GT_OK;
    }
    return GT_ERR_CAPACITY;
}

}  // extern "C"
