// gt_internal.cuh -- device-side types shared by the locate, finalize and link
// kernels of the B200 gpu_tracking path.
//
// Data layout in HBM (one movie = T frames of H x W pixels, row-major):
//   frames     u16 or f32, T*H*W                    (input, read once)
//   cand       Cand records, T*cap_c                (per-frame slab, unordered)
//   fcount     int, T                               (records per frame)
//   rowcnt     int, T*H*ntx                         (records per (row, tile column))
//   part_*     y, x, mass, rec: T*cap_p             (survivors, raster order)
//   npart      int, T
//   grid_*     cell starts (T*(ncell+1)) and indices (T*cap_p) for linking
//   pred       int, T*cap_p  (global index of the linked source, -1 = new)
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#define GT_MAX_TAPS 64
#define GT_MAX_CIRCLE 1024

namespace gt {

// Derived per-movie parameters (gpu_setup.rs:45-60 plus the tile plan).
struct LocParams {
    int H, W;
    int taps, krad;             // smoothing window: taps = 2*krad + 1
    float w[GT_MAX_TAPS];       // exp(-i^2 / (2 * noise_size)), i = -krad..krad
                                // (divided by norm when the taps are normalised on the host)
    float norm;                 // sum of the exp() taps in order
    float kk;                   // f32(smoothing_size^2), the boxcar divisor
    float rn;                   // RN(1 / norm), or 1 with host-normalised taps
    float rkk;                  // RN(1 / kk)
    int D, o;                   // dilation size and window offset
    int d, rint_c, border;      // diameter, centroid radius (d-1)/2, border d/2
    int char_r;                 // cpu_processed circle radius d/2
    int max_iter;
    float thr, minmass;
    int hp;                     // processed halo of a tile
    int TH, TW, ntx, nty;       // tile shape and tile counts
    int dtype;                  // 0 = u16, 1 = f32
    int cpu_processed, characterize;
    int zero_skip;              // zero-valued maxima provably have zero mass
    int n_char;                 // entries of the d/2 circle table
    int n_gchar;                // entries of the (d-1)/2 circle table
    int tma_spin;               // iteration limit of the bounded wait for a staged tile
    int tma_withhold;           // test switch: issue no tile copy, so the wait runs out
    int tiles_per_cta;          // specialised kernel: tiles per CTA (0 = chosen per launch)
    int frame0;                 // specialised kernel: first frame of the launch (its buffers start there)
};

// Where the specialised kernel's tile copies read a launch's frames: rows
// `pitch` pixels apart.
struct TileSource {
    const void* base;
    int pitch;
};

// One located feature, keyed by its originating pixel (walk_cols.wgsl:87-91).
struct __align__(16) Cand {
    int u, v;             // originating pixel
    float y, x, mass;     // walk result
    int rowrank;          // rank within its (row, tile column) segment
    int state;            // 0 emitted, 1 waiting for the fallback walk, 2 rejected
    float rg_sum;         // cpu_processed pieces at the originating pixel
    float eccn;           // sqrt(sin_sum^2 + cos_sum^2)
    float mid;            // processed value at the originating pixel
    float signal;
    float g_rg, g_raw, g_sig, g_ecc;   // characterize=True columns
    int ul, vl;           // pixel of the walk's last centroid read
    int up, vp;           // walk's final position (differs when the walk ran out)
    int pad;
};

enum CandState { CAND_EMIT = 0, CAND_PENDING = 1, CAND_REJECT = 2 };

// Error word bits written by kernels (never a trap).
enum ErrBits {
    ERR_CAND_OVERFLOW = 1,
    ERR_PART_OVERFLOW = 2,
    ERR_EDGE_OVERFLOW = 4,
    ERR_SUBNET_BUDGET = 8,
    ERR_SCRATCH_OVERFLOW = 32,
    ERR_DEVICE_TIMEOUT = 64,
};

// Per-movie device buffers and capacities.
struct MovieBufs {
    const void* frames;
    int T;
    int cap_c, cap_p;
    Cand* cand;
    int* fcount;
    int* rowcnt;
    int* pend;            // fallback list: frame*cap_c + slot
    int* npend;
    float* py;
    float* px;
    float* pm;
    int* prec;
    int* npart;
    int G, ncx, ncy;      // separation grid: cell size and counts
    int LG, lncx, lncy;   // linker's grid
    int* gstart;          // T*(lncx*lncy+1)
    int* gidx;            // T*cap_p
    float2* gpos;         // T*cap_p (y, x) of gidx's particles
    float* cy;            // T*cap_c emitted candidates in raster order
    float* cx;
    float* cm;
    int* crec;
    int* ccell;           // T*cap_c
    int* cidx;            // T*cap_c
    const float* char_tab;   // n_char x {r2, sin2, cos2}, d/2 circle
    const int* char_off;     // n_char x {di, dj}
    const float* gchar_tab;  // n_gchar x {sin2, cos2}, (d-1)/2 circle
    int* err;
    int* off;             // exclusive prefix of npart, by the last block of finalize_kernel
    int* nrows;           // rows of the frames so far
    int* done;            // blocks of finalize_kernel that are done (0: not counted, null: no offsets)
};

// A component's arrays in memory for cd destinations, cs sources and ce edges,
// with indices of `isz` bytes (link.cu, MemComp): the lists, then the hash
// tables of the exploration, whose place the search's arrays take.
__host__ __device__ constexpr int hash_size(int cap) {
    int n = 64;
    while (n < 2 * cap || n < cap + 33) n <<= 1;  // a warp's 32 keys may come on top of cap
    return n;
}
__host__ __device__ constexpr size_t comp_lists(size_t cd, size_t cs, size_t ce, size_t isz) {
    return (4 * (ce + cd + cs) + isz * (2 * ce + cd + 1) + 3) / 4 * 4;
}
__host__ __device__ constexpr size_t comp_bytes(int cd, int cs, int ce, size_t isz) {
    const size_t search = 4 * (size_t)cs + isz * (6 * (size_t)cd + 2 * (size_t)cs);
    const size_t hash = (4 + isz) * ((size_t)hash_size(cd) + hash_size(cs));
    return comp_lists(cd, cs, ce, isz) + ((search > hash ? search : hash) + 3) / 4 * 4;
}

// The linker's counters, a set of NCTR per pass (4 sets in turn): seeds (of the
// first linking: components beyond a thread's arrays), membership checks,
// components beyond a warp's registers, frames, components beyond a block's
// arrays, and those of them that are done.
enum { C_SEEDS = 0, C_CHECKS = 1, C_MEM = 2, C_FRAMES = 3, C_SLOT = 4, C_DONE = 5, NCTR = 8 };

struct LinkBufs {
    int cap_p, memory;
    int tb, te;           // frames linked by this launch; earlier frames are final
    float r;              // search range
    float inv_g;          // 1 / cell size
    int ncx, ncy;
    const float* py;
    const float* px;
    const int* off;       // exclusive prefix of npart (compact particle index)
    const int* gstart;
    const int* gidx;
    const float2* gpos;   // slab: (y, x) of gidx's particles
    // per particle, by compact index
    size_t np;            // stride of the membership words: T * cap_p
    int* pred;            // compact index of the linked source, -1 = new
    unsigned* lnk;        // bit j: linked by the frame j + 1 later (j = 0, 1)
    unsigned* mm;         // word w, bit b: memory entry of the frame 2 + 32 w + b later
    int* stamp;           // last pass in which the particle was a seed
    int* rstamp;          // last pass that listed it for a membership check
    int* seedq;           // slab handles of the pass's seeds, np
    int* recq;            // particles whose linked bits the pass changed (memory 1, 2),
                          // or those of the trajectories that it changed
    int* deferq;          // seeds whose component is resolved in memory, np
    int* newrank;         // rank among new particles of its frame
    int* root;
    int* lroot;           // where the pred chain enters the particle's chunk
    // memory >= 3
    int* gframe;          // frame
    int* cstamp;          // by root: pass that evaluates the trajectory again
    int* head;            // lists of unused particles, hashed by (root, frame >> fshift)
    int4* ent;            // their entries: root, frame, next
    int fshift;           // 2^fshift >= memory frames
    unsigned* pres;       // as mm: the id is present in the frame 1 + 32 w + b later
    int* newcount;        // T
    int* fstamp;          // T: last pass with a seed in the frame
    int* ctr;             // 4 passes x NCTR
    int* err;
    long long budget;     // branch-and-bound option trials per subnet
    // scratch of the components beyond a block's own arrays: nslot slots of
    // big_ints for big_d destinations, big_s sources and big_e edges
    int nslot, big_d, big_s, big_e;
    size_t big_ints;
    int* big;
};

// Adjoint of bandpass + refine at fixed peaks.  The forward arithmetic uses
// the same weights as LocParams; a / da are the real-valued normalised
// Gaussian taps w_i / sum(w) and their derivative with respect to
// noise_size (the Gaussian variance).
struct AdjParams {
    int T, H, W;
    int krad;                // smoothing half window
    int rc;                  // centroid circle radius, (diameter - 1) / 2
    int border;              // diameter / 2: centroids inside this band are zero
    int K;                   // circle pixel count
    float w[GT_MAX_TAPS];    // forward weights, as LocParams::w
    float norm, kk;          // forward normaliser and f32(k * k)
    float rn, rkk;           // their reciprocals, as LocParams
    float a[GT_MAX_TAPS];    // w_i / sum(w)
    float da[GT_MAX_TAPS];   // d a_i / d noise_size
    float k;                 // smoothing_size as a real number
    float gain, read_var;    // noise model of the uncertainty kernel
};

// The backward pass's dL/dR: K values per peak of the chunk, and the peaks that
// reach an output tile (frame, tile row, tile column): the first TILE_PEAKS in
// an array, the others in a list of entries peak * slots + one of its tiles,
// numbered from 1.
constexpr int TILE_PEAKS = 16;
struct AdjTiles {
    float* g;
    int* count;  // peaks of the tile
    int* head;   // 0: no list
    int* peaks;
    int* next;
    int slots;
    int th, nty, ntx;  // tile rows (columns: 64) and tiles per frame
};

struct AsmArgs {
    int T, H, W, cap_p, cap_c, ncols;
    int has_link, cpu_processed, characterize, sig, bg;
    const void* frames;
    int dtype;
    const float* py;
    const float* px;
    const float* pm;
    const int* prec;
    const int* npart;
    const int* off;
    const Cand* cand;
    const int* root;
    const int* newid;
    const int* sig_off;   // n_sig x {di, dj}, circle_inds(sig_radius)
    int n_sig;
    const int* bg_off;    // n_bg x {di, dj}, annulus_inds
    int n_bg;
    float* out;
    long long out_rows;   // rows of `out` (rows beyond are not written)
    int* walk;            // optional n x 5 {frame, last-read row, col, final row, col}
    long long walk_rows;  // rows of `walk` (rows beyond are not written)
};

// Lets a kernel have as much dynamic shared memory as there is, once per
// device: the limit is the process's, so every caller sets the same one.
template <auto* FN>
inline cudaError_t allow_shared() {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    cudaFuncAttributes a;
    e = cudaFuncGetAttributes(&a, (const void*)FN);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void*)FN, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 227 * 1024 - (int)a.sharedSizeBytes);
    if (e == cudaSuccess && dev < 64) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

}  // namespace gt
