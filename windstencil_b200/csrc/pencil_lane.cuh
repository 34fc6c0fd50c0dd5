// pencil_lane.cuh -- the mixed form's z pass with the SSP-RK3 stage, all five
// variables in one lane.
//
// Every lane owns one z line and marches it alone: per point it computes the
// Steger-Warming split of the point four ahead into a private 8-slot ring in
// shared memory, reconstructs the five faces above the current point from the
// ring (ws_device.cuh: P and M in the halves of packed FP32x2), and updates
// the cell: du of the other passes plus the face difference, the stage
// formula, the primitives of the new state.  No lane reads another lane's
// ring, so there is no barrier; a warp's lanes are consecutive in x, so its
// accesses coalesce; the next point's operands are loaded a step ahead.
//
// pencil_impl.cuh's passes (one sign of one variable per lane) take fewer
// operations per face and run everything else; here the update of a cell
// (about 60 FP64 operations, 15 loads, 11 stores) is as long as its faces in
// packed FP32, and there half of the warps do it for two lines each while the
// others wait: 0.589 ms against 0.488 ms here at 600x128x128, 1.07 against
// 0.88 ms on a batch of 32 grids (nx in [32, 256], ny, nz in [16, 128]).
#pragma once
#include "bf3w_rhs_impl.cuh"

namespace ws {

struct LaneLayout {
    static constexpr int RS = 10 * 32;            // ring slot stride (floats), lanes inner
    static constexpr int WARP = 8 * RS;           // one warp's ring
};

// LAP position whose primitives point m of a line has (RhsArgs::gk); _ahead:
// of a point past the first four, as the march takes them.
template <int DIR>
__device__ __forceinline__ int pencil_source_ahead(const RhsArgs& a, int m) {
    const int n = DIR == 0 ? a.nx : (DIR == 1 ? a.ny : a.nz);
    if (m < n + 4) return m;
    return a.gk[2 * DIR + 1] == 1 ? m - n : a.gk[2 * DIR + 1] == 2 ? n + 3 : m;
}
template <int DIR>
__device__ __forceinline__ int pencil_source(const RhsArgs& a, int m) {
    const int n = DIR == 0 ? a.nx : (DIR == 1 ? a.ny : a.nz);
    if (m < 4) return a.gk[2 * DIR] == 1 ? m + n : a.gk[2 * DIR] == 2 ? 4 : m;
    return pencil_source_ahead<DIR>(a, m);
}

// work of the pass over the job of `a`: groups of 32 lines x positions
__device__ __forceinline__ long lane_work(const RhsArgs& a, int& L) {
    L = a.ez - a.sz;
    return ((long)(a.ex - a.sx) * (a.ey - a.sy) + 31) / 32 * L;
}

// Positions p0 .. p0+len-1 of the lines of group grp, with the lane's ring
// column `ring`.
__device__ __forceinline__ void lane_segment(const RhsArgs& a, int krk, float* ring, long grp,
                                             int p0, int len) {
    constexpr int RS = LaneLayout::RS;
    const int lane = threadIdx.x & 31;
    const SplitK<float> k = {(float)a.eps2, (float)a.hrg, (float)a.c1, (float)a.c3, (float)a.gm1};
    const int nxj = a.ex - a.sx;
    const long NL = (long)nxj * (a.ey - a.sy);
    const size_t vs = (size_t)a.du_pitch * a.du_ly * a.du_lz;            // du variable stride
    const size_t fvs = (size_t)a.fn.pitch * a.fn.length_Y * a.fn.length_Z;
    long l = grp * 32 + lane;
    const bool valid = l < NL;
    if (!valid) l = NL - 1;
    const int x = a.sx + (int)(l % nxj), y = a.sy + (int)(l / nxj);
    auto load = [&](int z, double q[5]) {
        const int zs = pencil_source<2>(a, z);
#pragma unroll
        for (int f = 0; f < 5; ++f) q[f] = ldg_prim(a, f, x, y, zs);
    };
    auto split_into = [&](int z, const double q[5]) {
        float out[10];
        split_point<2, true, float>(a, k, q[0], q[1], q[2], q[3], q[4], x, y, z, out);
        float* dst = ring + (z & 7) * RS;
#pragma unroll
        for (int c = 0; c < 10; ++c) dst[c * 32] = out[c];
    };
    auto du_at = [&](int z) {
        return (size_t)(x - a.sx) +
               (size_t)a.du_pitch * ((size_t)(y - a.sy) + (size_t)a.du_ly * (size_t)(z - a.sz));
    };
    auto f_at = [&](int z) { return soa_index(a.fn, x - 4, y - 4, z - 4, 0); };
    // face value of variable v above position m: stencil from ring slot s0
    auto face = [&](int s0, int v) {
        return face_flux<float, true>(ring + s0 * RS + v * 32, 5 * 32, RS, 8 - s0, 8 * RS);
    };

    const int ms = a.sz + p0, mlast = a.nz + 7;
    for (int m = ms - 4; m < ms + 4; ++m) {
        double q[5];
        load(m, q);
        split_into(m, q);
    }
    double qn[5], dn[5], fnn[5], fin[5];
    load(ms + 4, qn);
    auto load_cell = [&](int m) {      // du and the stage operands of point m
        const size_t o = du_at(m), fo = f_at(m);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            dn[v] = a.du[o + v * vs];
            fnn[v] = __ldg(a.fn.ptr + fo + v * fvs);
            fin[v] = krk == 1 ? 0.0 : a.f_in.ptr[fo + v * fvs];
        }
    };
    if (valid) load_cell(ms);
    double fprev[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) fprev[v] = face((ms - 4) & 7, v);
    for (int m = ms; m < ms + len; ++m) {
        double q[5], dc[5], fnc[5], fic[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            q[f] = qn[f];
            dc[f] = dn[f];
            fnc[f] = fnn[f];
            fic[f] = fin[f];
        }
        load(min(m + 5, mlast), qn);
        if (valid && m + 1 < ms + len) load_cell(m + 1);
        split_into(m + 4, q);
        const int s0 = (m - 3) & 7;
        double r[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            const double fc = face(s0, v);
            r[v] = -((fc - fprev[v]) * a.rhz);
            fprev[v] = fc;
        }
        if (!valid) continue;
        const size_t fo = f_at(m);
        double qs[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            qs[v] = ws_rk_stage(krk, fnc[v], fic[v], dc[v] + r[v], a.dt);
            a.f_out.ptr[fo + v * fvs] = qs[v];
        }
        store_prims(a, qs, x, y, m);
    }
}

// The pass over the whole interior of `a`: every warp takes an equal
// contiguous share of the (line group, position) space.
template <int WPB>
__global__ void __launch_bounds__(WPB * 32, 1)
    pencil_lane_kernel(const __grid_constant__ RhsArgs a, int krk) {
    extern __shared__ __align__(16) unsigned char pencil_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* ring = reinterpret_cast<float*>(pencil_smem) + warp * LaneLayout::WARP + lane;
    int L = 0;
    const long total = lane_work(a, L);
    const long S = (long)gridDim.x * WPB, s = (long)blockIdx.x * WPB + warp;
    long pos = total * s / S;
    const long end = total * (s + 1) / S;
    while (pos < end) {
        const long grp = pos / L;
        const int p0 = (int)(pos - grp * L);
        const int len = (int)min((long)(L - p0), end - pos);
        lane_segment(a, krk, ring, grp, p0, len);
        pos += len;
    }
}

// The same over the grids of a batch: argument table `grids`, and woff[i] the
// pass's work before grid i (woff[n] the total).  A warp's share may cross
// grids.
template <int WPB>
__global__ void __launch_bounds__(WPB * 32, 1)
    pencil_lane_batch_kernel(const RhsArgs* __restrict__ grids, const long* __restrict__ woff,
                             int n, int krk) {
    extern __shared__ __align__(16) unsigned char pencil_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* ring = reinterpret_cast<float*>(pencil_smem) + warp * LaneLayout::WARP + lane;
    const long total = woff[n];
    const long S = (long)gridDim.x * WPB, s = (long)blockIdx.x * WPB + warp;
    long pos = total * s / S;
    const long end = total * (s + 1) / S;
    int lo = 0, hi = n;                    // the grid holding pos: woff[i] <= pos < woff[i+1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (woff[mid] <= pos) lo = mid; else hi = mid;
    }
    int i = lo;
    while (pos < end) {
        while (woff[i + 1] <= pos) ++i;
        const RhsArgs& a = grids[i];
        int L = 0;
        lane_work(a, L);
        const long local = pos - woff[i];
        const long grp = local / L;
        const int p0 = (int)(local - grp * L);
        const int len = (int)min((long)(L - p0), end - pos);
        lane_segment(a, krk, ring, grp, p0, len);
        pos += len;
    }
}

}  // namespace ws
