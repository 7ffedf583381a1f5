// locate_flex.cu -- the specialised locate kernel with a run-time dilation
// size: float frames, diameters 13 and 15, and separations beside the default
// diameter + 1.
#include "locate_fast.cuh"

namespace gt {

namespace {
// (radius, dilation size of separation = diameter + 1)
#define GT_FLEX_LIST(X) X(2, 8) X(3, 11) X(4, 14) X(5, 16) X(6, 19) X(7, 22)
}  // namespace

// The largest dilation size of radius rc's instance, 0 without one.
int flex_dilation(int rc) {
#define GT_FLEX_CASE(R, DD) if (rc == R) return DD;
    GT_FLEX_LIST(GT_FLEX_CASE)
#undef GT_FLEX_CASE
    return 0;
}

int flex_rows(int rc, int dtype) {
#define GT_FLEX_CASE(R, DD) \
    if (rc == R) return dtype == 0 ? tile_rows<R, DD, R, unsigned short, true>() : tile_rows<R, DD, R, float, true>();
    GT_FLEX_LIST(GT_FLEX_CASE)
#undef GT_FLEX_CASE
    return 64;
}

cudaError_t launch_locate_flex(int kr, int rc, int dtype, dim3 grid, cudaStream_t st, const LocParams& p,
                               const MovieBufs& b, const TileSource& src, int frame0, int* used_tma) {
    if (kr != rc || p.D < FM || p.D > flex_dilation(rc)) return cudaErrorInvalidValue;
#define GT_FLEX_CASE(R, DD)                                                                                   \
    if (rc == R)                                                                                              \
        return dtype == 0 ? launch_instance<R, DD, tile_rows<R, DD, R, unsigned short, true>(), R, unsigned short, \
                                            true>(grid, st, p, b, src, frame0, used_tma)                       \
                          : launch_instance<R, DD, tile_rows<R, DD, R, float, true>(), R, float, true>(        \
                                grid, st, p, b, src, frame0, used_tma);
    GT_FLEX_LIST(GT_FLEX_CASE)
#undef GT_FLEX_CASE
    return cudaErrorInvalidValue;
}

}  // namespace gt
