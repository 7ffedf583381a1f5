// locate_fast.cu -- the specialised locate kernel for uint16 frames whose
// diameter (5, 7, 9, 11) and separation are the common ones.
#include "locate_fast.cuh"

namespace gt {

cudaError_t launch_locate_flex(int kr, int rc, int dtype, dim3 grid, cudaStream_t st, const LocParams& p,
                               const MovieBufs& b, const TileSource& src, int frame0, int* used_tma);
int flex_dilation(int rc);
int flex_rows(int rc, int dtype);

// (smoothing radius, dilation size, centroid radius) triples with a kernel of
// their own: diameters 5, 7, 9, 11 (odd, centroid radius (d - 1) / 2) with the
// default smoothing (= diameter) and separation (= diameter + 1), plus
// neighbouring separations.
#define GT_FAST_LIST(X) X(2, 8, 2) X(3, 11, 3) X(4, 14, 4) X(5, 16, 5) X(3, 8, 3) X(4, 11, 4) X(2, 7, 2) X(3, 12, 3)

// The specialised kernel for these parameters: 1 an instance of its own (tile
// heights 32 and fast_rows), 2 the run-time dilation of locate_flex.cu, 0
// none (locate_tiles_kernel).
int fast_supported(int kr, int dd, int rc, int diameter, int dtype) {
    if (diameter != 2 * rc + 1 || kr != rc) return 0;
    if (dtype == 0) {
#define GT_FAST_CASE(KR, DD, RC) if (kr == KR && dd == DD && rc == RC) return 1;
        GT_FAST_LIST(GT_FAST_CASE)
#undef GT_FAST_CASE
    }
    return dd >= FM && dd <= flex_dilation(rc) ? 2 : 0;
}

// Tile rows of those kernels: 32 where asked for and there is a choice, else the
// instance's own.
int fast_rows(int kr, int dd, int rc, int dtype, int th) {
    if (dtype == 0) {
#define GT_FAST_CASE(KR, DD, RC) \
    if (kr == KR && dd == DD && rc == RC) return th == 32 ? 32 : tile_rows<KR, DD, RC, unsigned short, false>();
        GT_FAST_LIST(GT_FAST_CASE)
#undef GT_FAST_CASE
    }
    return flex_rows(rc, dtype);
}

// Launches the specialised kernel over frames [frame0, frame0 + grid.y),
// grid.x tiles per frame, whose raw tiles are copied from src.  *used_tma
// reports whether they were staged by TMA; else they are read from b.frames.
cudaError_t launch_locate_fast(int kr, int dd, int rc, int th, dim3 grid, cudaStream_t st, const LocParams& p,
                               const MovieBufs& b, const TileSource& src, int frame0, int* used_tma) {
    if (p.dtype == 0) {
#define GT_FAST_CASE(KR, DD, RC)                                                                              \
    if (kr == KR && dd == DD && rc == RC)                                                                     \
        return th == 32 ? launch_instance<KR, DD, 32, RC, unsigned short, false>(grid, st, p, b, src, frame0, used_tma) \
                        : launch_instance<KR, DD, tile_rows<KR, DD, RC, unsigned short, false>(), RC, unsigned short, \
                                          false>(grid, st, p, b, src, frame0, used_tma);
        GT_FAST_LIST(GT_FAST_CASE)
#undef GT_FAST_CASE
    }
    return launch_locate_flex(kr, rc, p.dtype, grid, st, p, b, src, frame0, used_tma);
}

}  // namespace gt
