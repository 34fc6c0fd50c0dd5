// pencil.cu -- host dispatch of the line-pass RHS (pencil_impl.cuh).
#include "pencil_impl.cuh"

namespace ws {

// krk 0: plain RHS into a.du; krk 1..3: into a.du, then the stage update.
// add_x: a.du already holds terms to add to (the viscous terms).
int launch_rhs_pencil(const RhsArgs& a, int precision, bool uniform, int krk, bool add_x,
                      cudaStream_t st) {
    if (precision == WS_MIXED) {
        if (krk) return PencilLauncher<float2, true>::stage(a, add_x, krk, st);
        return uniform ? PencilLauncher<float2, true>::rhs(a, add_x, st)
                       : PencilLauncher<float2, false>::rhs(a, add_x, st);
    }
    if (krk) return PencilLauncher<double, true>::stage(a, add_x, krk, st);
    return uniform ? PencilLauncher<double, true>::rhs(a, add_x, st)
                   : PencilLauncher<double, false>::rhs(a, add_x, st);
}

// the batched form over the argument table g of n Cartesian grids (woff: the
// work prefix tables of pencil_pass_work's four dirs, n + 1 entries each; clo:
// some grid has a CLOSURE face)
int launch_rhs_pencil_batch(const RhsArgs* g, const long* woff, int n, int precision, int krk,
                            bool clo, cudaStream_t st) {
    if (precision == WS_MIXED)
        return PencilLauncher<float2, true>::batch(g, woff, n, krk, clo, st);
    return PencilLauncher<double, true>::batch(g, woff, n, krk, clo, st);
}

// work of table dir (0 x, 1 y, 2 z, 3: z in groups of 32 lines) over the
// interior of grid g, in the line groups of the kernel that it is for
long pencil_pass_work(const ws_grid& g, int dir) {
    const bool two = g.precision == WS_MIXED && dir < 3;       // two lines per lane
    return pencil_places(g.nx, g.ny, g.nz, dir < 3 ? dir : 2,
                         two ? PencilLauncher<float2, true>::GL : PencilLauncher<double, true>::GL);
}

}  // namespace ws
