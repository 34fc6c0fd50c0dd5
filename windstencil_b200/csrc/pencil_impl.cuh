// pencil_impl.cuh -- BF3W inviscid RHS as three line passes.
//
// Replaces, like the fused kernel (bf3w_rhs_impl.cuh), the reference's
// split_Jac3d_Stager_Warming_ker (src/kernels/OCFD_split.cpp:36-3918) and
// its boundary-ring kernel (src/solver/OCFD_NS_Jacobian3d.cpp:828-2530).  The
// fused kernel sweeps a 2D column footprint along z and recomputes the
// footprint's halo splits and edge faces; here a RHS is three passes, x (du =,
// or += onto viscous terms already stored in du), y (+=) and z (+=, or in
// stage mode the SSP-RK3 stage update and the primitives of the new state),
// and every pass marches whole grid lines, so no split and no face is
// computed twice (except an 8-point prologue per line segment).
//
// Ten warps (two such thread groups to a CTA, one CTA per SM) take a group of
// lines (32; 64 in the mixed form, two per lane in packed FP32x2): lane =
// line, warp = one sign of the split flux of one conserved variable.  Every lane takes its split flux through the
// streaming reconstruction of line_weno.cuh, whose state -- differences and
// waiting indicators, 22 values -- stays in its registers.  After marching a
// chunk of five points, the five F+ warps split the chunk after next (one
// point each, all ten components, into a ring in shared memory) and the five
// F- warps write the previous chunk out (one point each, all five variables);
// a component's ring entry is read by its own lane only, which leaves the
// cell's result in its place.  Operands of both arrive by cp.async issued a
// chunk ahead into per-thread slots.  A warp enters its exchange when all
// have finished theirs of the chunk before (a barrier split into arrival and
// wait), so no warp waits for another unless it is a whole march ahead.
//
// Why this split: with all five variables in one lane (the earlier form) the
// reconstruction could keep nothing between faces, so each face took 190 FP64
// operations from a ring of splits that also held the SM to 8 warps.  One
// sign of one variable fits 96 registers: 20 warps per SM and 119 operations
// per face.  Both signs in a lane would take 112, but their state spilled (10
// warps at 168 registers: y pass 1.14 ms at 600x128x128, 15 warps at 128: 1.36
// ms).  Measured at 600x128x128, earlier form -> this one: FP64 x .980 -> .505,
// y .808 -> .543, z .818 -> .541, z with the stage .948 -> .615 ms; mixed x .487
// -> .348, y .363 -> .305, z .373 -> .304 ms.  FP64 pipe 68-71% active, FP32 FMA
// pipe of the mixed form 48-52% (ncu); an FMA with three distinct registers takes
// the FP64 pipe 3 cycles instead of 2, and fixed-latency waits and the exchange
// take the rest.  du goes through HBM between the passes (~340 B/cell).
#pragma once
#include <algorithm>
#include <type_traits>

#include "bf3w_rhs_impl.cuh"
#include "line_weno.cuh"
#include "pencil_lane.cuh"

namespace ws {

enum PencilMode { P_STORE = 0, P_ADD = 1, P_STAGE = 2 };

// C points per chunk (the march is unrolled C times, more than the longest
// lag, so the lagged values rotate through registers).  Ring of four chunks --
// being written out, marched, ready, being split -- the 8-point prologue in
// the last 8 slots.  A lane's result goes to the slot of the point just taken.
//
// The result is the cell's face difference in FP64.  In FP32 (FACE) it is the
// value of the face above the cell, which the write-out widens and subtracts:
// both cells at a face then have the same value of it, and du sums to zero over
// a periodic line to FP64 rounding (differences taken in FP32 left 4e-10 to
// 6e-9 of sum |du|).  The write-out of a
// chunk reads the last face of the chunk before too: one more chunk.
template <typename V>
struct PencilLayout {
    static constexpr int NL = LineVal<V>::NL, GL = 32 * NL;
    static constexpr bool FACE = sizeof(typename LineVal<V>::CT) == 4;
    static constexpr int C = 5, NT = 320, HT = NT / 2;   // threads of a group, of one role
    static constexpr int SLOTS = (FACE ? 5 : 4) * C;
    static_assert(SLOTS >= 4 * C + FACE && SLOTS >= 2 * C + 8, "ring");
    // slot stride padded for the x pass, whose lanes write (and read back)
    // neighbouring slots at once; unpadded these would share their banks
    static constexpr int RS = 10 * 32 + 3;               // V per slot
    static constexpr size_t RING = ((size_t)SLOTS * RS * sizeof(V) + 15) / 16 * 16;
    // operands brought ahead, per line of a role thread: 5 primitives (F+
    // warps); du, and in stage mode fn and f (F- warps)
    template <int MODE>
    static constexpr size_t bytes() {                    // of one group
        return RING +
               (size_t)(5 + (MODE == 0 ? 0 : MODE == 1 ? 5 : 15)) * NL * HT * sizeof(double) +
               GL * 2 * sizeof(int) + 16;                // the group's lines, two mbarriers
    }
    static_assert(sizeof(V) == 8, "one 8-byte value per lane and component");
};

// A zone: the four cells at a CLOSURE end of a line.  They take five faces, of
// which only the inner one is a WENO7 face on both sides, and their pieces run
// apart from the march, which so has no closure in it: values next to a CLOSURE
// end are FP64 in the mixed form too (kept beside the march's FP32 results they
// cost it 60% in the x pass), no ghost point is read but the one that the WENO7
// value three faces from a high end takes, and the ring need not hold the
// points' history.  With walls in x and y, closures in the march -> zones, x and
// y passes at 600x128x128: FP64 606 + 770 -> 578 + 662 us, mixed (FP32 closure
// values) 402 + 537 -> 353 + 406; 480x64x32 mixed 55 + 83 -> 48 + 62.
constexpr int kZone = 4;
// Position of the march (of L, in job coordinates) at which a piece from
// position p0 on ends at the latest: zones are pieces of their own.
template <int DIR, bool CLO>
__device__ __forceinline__ int pencil_stop(const RhsArgs& a, int p0, int L) {
    if constexpr (CLO) {
        const int n = DIR == 0 ? a.nx : a.ny, s = (DIR == 0 ? a.sx : a.sy) - 4;
        if (a.clo[2 * DIR] && p0 + s < kZone) return min(kZone - s, L);
        if (a.clo[2 * DIR + 1] && p0 + s < n - kZone) return min(n - kZone - s, L);
    }
    return L;
}

// One sign's closure value at face f of a line of n cells, at its low (hi
// false) or high CLOSURE end, from the split fluxes t(i) of the zone's points i
// (i = 0: cell 0, or cell n - 8).  The rules of closure_p_arr and closure_m_arr
// as one formula on the five points q[0..4] about the face, taken from the other
// side for F-: candidates on q[2..4], q[1..3], q[0..2] with weights 1 / (12e-6 +
// S)^2 of those that the face has (`use`), divided out of the sum as products of
// the others; the third face from an end (F+) has the reference's product
// weights, and at the ends the value is linear in two points.  One piece of
// code for all faces: with a branch per rule, within the march, a face cost as
// much as 15 others.
template <typename F>
__device__ __forceinline__ double pencil_closure(F t, bool minus, int f, int n, bool hi) {
    const int first = hi ? n - 8 : 0;
    double q[5];
#pragma unroll
    for (int k = 0; k < 5; ++k)          // points past the zone's are not used
        q[k] = t(min(max((minus ? f + 2 - k : f - 3 + k) - first, 0), 8));
    const int e = hi ? n - f : 99, b = hi ? 99 : f;    // faces from the end
    if (e <= (minus ? 1 : 0) || (b == 0 && !minus)) {
        const double x = b == 0 ? q[3] : minus && e == 0 ? q[3] : q[2];
        const double y = b == 0 ? x : minus ? (e == 0 ? q[4] : q[3]) : q[1];
        return x + (minus ? -0.5 : 0.5) * (x - y);
    }
    const bool third = !minus && (b == 3 || e == 2);
    const int use = minus ? (b == 0 ? 4 : b == 1 ? 6 : e == 2 ? 3 : 7)
                          : (b == 1 ? 1 : b == 2 ? 3 : e == 1 ? 6 : 7);
    auto ind = [](double t0, double t1) {
        const double S = w5::E12 + (13 * t0 * t0 + 3 * t1 * t1);
        return S * S;
    };
    double d0 = ind(q[2] - 2 * q[3] + q[4], 3 * q[2] - 4 * q[3] + q[4]);
    double d1 = ind(q[1] - 2 * q[2] + q[3], q[1] - q[3]);
    double d2 = ind(q[0] - 2 * q[1] + q[2], q[0] - 4 * q[1] + 3 * q[2]);
    if (!(use & 1)) d0 = 1.0;
    if (!(use & 2)) d1 = 1.0;
    if (!(use & 4)) d2 = 1.0;
    constexpr double z = w5::E12 * w5::E12;
    const double a0 = third ? z * z : use & 1 ? d1 * d2 : 0.0;
    const double a1 = third ? d0 * z : use & 2 ? d0 * d2 : 0.0;
    const double a2 = third || (use & 4) ? d0 * d1 : 0.0;
    const double c0 = use & 1 ? 2 * q[2] + 5 * q[3] - q[4] : 0.0;
    const double c1 = use & 2 ? -q[1] + 5 * q[2] + 2 * q[3] : 0.0;
    const double c2 = use & 4 ? 2 * q[0] - 7 * q[1] + 11 * q[2] : 0.0;
    return (a0 * c0 + a1 * c1 + a2 * c2) / (6.0 * (a0 + a1 + a2));
}

// Barrier of thread group tg of a CTA.
__device__ __forceinline__ void pencil_sync(int tg) {
    __syncwarp();
    asm volatile("barrier.cta.sync %0, 320;" ::"r"(tg + 1) : "memory");
}
// A group's phases: its ten warps arrive at the two mbarriers in turn.
__device__ __forceinline__ void pencil_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// hold (the failure path's test): an arrival more than ever comes, so that every
// wait runs out.
__device__ __forceinline__ void pencil_init_bars(unsigned char* first, size_t stride, bool hold) {
    for (int g = 0; g < 2; ++g)
        for (int b = 0; b < 2; ++b)
            mbar_init(reinterpret_cast<uint64_t*>(first + g * stride) + b, hold ? 11 : 10);
}

// March length and work of pass DIR over the job of `a`: line groups of GL
// lines x positions.
template <int DIR, int GL>
__device__ __forceinline__ long pencil_work(const RhsArgs& a, int& L) {
    const int nxj = a.ex - a.sx, nyj = a.ey - a.sy, nzj = a.ez - a.sz;
    L = DIR == 0 ? nxj : (DIR == 1 ? nyj : nzj);
    const long NL = DIR == 0 ? (long)nyj * nzj : (DIR == 1 ? (long)nxj * nzj : (long)nxj * nyj);
    return (NL + GL - 1) / GL * L;
}

// Positions p0 .. p0+len-1 of the lines of a group of a grid of the pass;
// ahead: the place in that grid where the next piece starts (-1: none).
struct PencilPiece {
    int grid, p0, len;
    long grp, ahead;
};

// Waits for the phase of parity `parity`; false when it gives up, after `hold`
// polls (0: 2^22) or when another warp of the group has.
__device__ __forceinline__ bool pencil_wait(uint64_t* bar, uint32_t parity, int hold,
                                            volatile int* stop) {
    if (mbar_try_wait(bar, parity)) return true;
    for (int i = hold > 0 ? hold : 1 << 22; i > 0; --i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*stop) return false;
    }
    return false;
}

// One piece of pass DIR (0 x, 1 y, 2 z) over the job of `a`, by thread group
// tg of a CTA.  CLO: pieces at CLOSURE ends of the direction are zones.  A wait
// that gives up sets status bit 2 and *stop; every warp of the group then leaves
// the piece at its next wait, its own copies in flight waited for, and takes no
// more.
template <int DIR, typename V, bool UNI, int MODE, bool CLO>
__device__ __forceinline__ void pencil_segment(const RhsArgs& a, int krk, unsigned char* smem,
                                               int tg, unsigned& phase, volatile int* stop,
                                               const PencilPiece& piece) {
    const long grp = piece.grp;
    const int p0 = piece.p0, len = piece.len;
    static_assert(MODE != P_STAGE || (DIR == 2 && UNI && LineVal<V>::NL == 1),
                  "stage update: z pass, Cartesian, FP64");
    static_assert(!CLO || DIR != 2, "closure faces: x and y passes");
    using P = PencilLayout<V>;
    using CT = typename LineVal<V>::CT;
    constexpr int C = P::C, NL = P::NL, RS = P::RS, HT = P::HT;
    constexpr bool ADD = MODE != P_STORE, FACE = P::FACE;
    const int gt = threadIdx.x - tg * P::NT, lane = gt & 31, warp = gt >> 5;
    const bool minus = warp >= 5;
    V* ring = reinterpret_cast<V*>(smem);
    const int nxj = a.ex - a.sx, nyj = a.ey - a.sy, nzj = a.ez - a.sz;
    const int n1 = DIR == 0 ? nyj : nxj;              // fastest line axis
    const int nlines = n1 * (DIR == 2 ? nyj : nzj);
    const int ms = (DIR == 0 ? a.sx : (DIR == 1 ? a.sy : a.sz)) + p0;
    const size_t vs = (size_t)a.du_pitch * a.du_ly * a.du_lz;            // du variable stride
    const int line0 = (int)grp * P::GL;

    // ---- exchange: this thread's point sx of each chunk on line sln (and sln +
    // 32); its operand slots, [operand][half][thread]
    const int rt = minus ? gt - HT : gt;
    const int sx = DIR == 0 ? rt % C : rt >> 5;
    const int sln = DIR == 0 ? rt / C : lane;
    double* slot = reinterpret_cast<double*>(smem + P::RING);
    auto prim_slot = [&](int f, int h) { return slot + (f * NL + h) * HT + rt; };
    auto cell_slot = [&](int f, int h) {
        return slot + 5 * NL * HT + (f * NL + h) * HT + rt;
    };
    // a point on each of the thread's lines: position m, the lines' two fixed
    // coordinates (from a table of the group's lines, so that neither they
    // nor addresses made of them are kept over the march)
    struct Pt {
        int m, c1[NL], c2[NL];
        __device__ __forceinline__ int x(int h) const { return DIR == 0 ? m : c1[h]; }
        __device__ __forceinline__ int y(int h) const {
            return DIR == 1 ? m : (DIR == 0 ? c1[h] : c2[h]);
        }
        __device__ __forceinline__ int z(int h) const { return DIR == 2 ? m : c2[h]; }
    };
    int2* lines = reinterpret_cast<int2*>(smem + P::template bytes<MODE>() - 16 - P::GL * sizeof(int2));
    auto point = [&](int m, int ln) {
        Pt p;
        p.m = m;
#pragma unroll
        for (int h = 0; h < NL; ++h) {
            const volatile int* c = &lines[ln + 32 * h].x;
            p.c1[h] = c[0];
            p.c2[h] = c[1];
        }
        return p;
    };

    // ---- splits
    auto prim_at = [&](int f, const Pt& p, int h) {
        return a.prim[f] + lap_index(p.x(h), p.y(h), p.z(h), a.ppitch[f], a.ny);
    };
    auto pack = [&](const double (&e)[NL]) -> V {
        if constexpr (NL == 1) return e[0];
        else return make_float2((float)e[0], (float)e[1]);
    };
    // the splits of point p with the primitives e into slot s
    auto split_into = [&](const double (&e)[5][NL], const Pt& p, int s, int ln) {
        const LineSplitK<V> k = {vset<V>(a.eps2), vset<V>(a.c1)};
        V q[4], g[3], out[10];
#pragma unroll
        for (int f = 0; f < 4; ++f) q[f] = pack(e[f + 1]);
        // the products that every component has as a factor, rounded once (in
        // FP32 throughout they were half of the mixed form's error)
        double t0[NL], t0c[NL], kc[NL];
#pragma unroll
        for (int h = 0; h < NL; ++h) {
            t0[h] = vmul(e[0][h], 0.5 * a.hrg * LineVal<V>::SCALE);
            t0c[h] = vmul(t0[h], e[4][h]);
            kc[h] = vmul(t0c[h], vmul(0.5 + a.c3, e[4][h]));
        }
        if (!UNI) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double m[NL];
#pragma unroll
                for (int h = 0; h < NL; ++h)
                    m[h] = ldg_met(a, 3 * DIR + c, p.x(h), p.y(h), p.z(h));
                g[c] = pack(m);
            }
        }
        line_split<DIR, UNI, V>(pack(t0), pack(t0c), pack(kc), q[0], q[1], q[2], q[3], g[0], g[1],
                                g[2], k, out);
        V* dst = ring + s * RS + ln;
#pragma unroll
        for (int c = 0; c < 10; ++c) dst[c * 32] = out[c];
    };
    // this thread's point of chunk k: primitives fetched ahead, then split into
    // the ring at slot `base` of the chunk
    auto fetch_prims = [&](int k) {
        const int i = k * C + sx;
        if (i < len) {
            const int m = ms + 4 + i;
            const Pt p = point(UNI ? pencil_source_ahead<DIR>(a, m) : m, sln);
#pragma unroll
            for (int f = 0; f < 5; ++f)
#pragma unroll
                for (int h = 0; h < NL; ++h) cp_async8(prim_slot(f, h), prim_at(f, p, h));
        }
        cp_async_commit();
    };
    auto split_fetched = [&](int k, int base) {
        const int i = k * C + sx;
        cp_async_wait<0>();
        if (i >= len) return;
        Pt p;
        if (!UNI) p = point(ms + 4 + i, sln);
        double e[5][NL];
#pragma unroll
        for (int f = 0; f < 5; ++f)
#pragma unroll
            for (int h = 0; h < NL; ++h) e[f][h] = *prim_slot(f, h);
        split_into(e, p, base + sx, sln);
    };

    // ---- results
    auto du_at = [&](const Pt& p, int h) {
        return (size_t)(p.x(h) - a.sx) +
               (size_t)a.du_pitch * ((size_t)(p.y(h) - a.sy) +
                                     (size_t)a.du_ly * (size_t)(p.z(h) - a.sz));
    };
    const size_t fvs = MODE == P_STAGE ? (size_t)a.fn.pitch * a.fn.length_Y * a.fn.length_Z : 0;
    auto f_at = [&](const Pt& p, int h) {
        return soa_index(a.fn, p.x(h) - 4, p.y(h) - 4, p.z(h) - 4, 0);
    };
    // du (and in stage mode the state) of this thread's point of chunk k, ahead
    // of its result
    auto fetch_cells = [&](int k) {
        const int i = k * C + sx;
        if (ADD && i < len) {
            const Pt p = point(ms + i, sln);
#pragma unroll
            for (int h = 0; h < NL; ++h) {
                const size_t o = du_at(p, h);
#pragma unroll
                for (int w = 0; w < 5; ++w) cp_async8(cell_slot(w, h), a.du + o + w * vs);
                if constexpr (MODE == P_STAGE) {
                    const size_t fo = f_at(p, h);
#pragma unroll
                    for (int w = 0; w < 5; ++w)
                        cp_async8(cell_slot(5 + w, h), a.fn.ptr + fo + w * fvs);
                    if (krk != 1)
#pragma unroll
                        for (int w = 0; w < 5; ++w)
                            cp_async8(cell_slot(10 + w, h), a.f_in.ptr + fo + w * fvs);
                }
            }
        }
        if (ADD) cp_async_commit();
    };
    const double rh = (DIR == 0 ? a.rhx : (DIR == 1 ? a.rhy : a.rhz)) * (FACE ? 1.0 / LineVal<V>::SCALE : 1.0 / 12.0);
    // result of this thread's point of chunk k at slot `base`
    auto write_cells = [&](int k, int base) {
        const int i = k * C + sx;
        if (ADD) cp_async_wait<0>();
        if (i >= len) return;
        const Pt p = point(ms + i, sln);
        const int s = base + sx;
        const int sb = s > 0 ? s - 1 : P::SLOTS - 1;       // FACE: of the face below the cell
#pragma unroll
        for (int h = 0; h < NL; ++h) {
            if (line0 + sln + 32 * h >= nlines) continue;
            const double J = UNI ? 1.0 : ldg_met(a, 9, p.x(h), p.y(h), p.z(h));
            const size_t o = du_at(p, h);
            double r[5];
#pragma unroll
            for (int w = 0; w < 5; ++w) {
                const V* e = ring + s * RS + w * 32 + sln;
                double sum;
                if constexpr (FACE) {
                    const V* b = ring + sb * RS + w * 32 + sln;
                    sum = (double)(reinterpret_cast<const CT*>(e)[h] +
                                   reinterpret_cast<const CT*>(e + 160)[h]) -
                          (double)(reinterpret_cast<const CT*>(b)[h] +
                                   reinterpret_cast<const CT*>(b + 160)[h]);
                } else {
                    sum = (double)reinterpret_cast<const CT*>(e)[h] +
                          (double)reinterpret_cast<const CT*>(e + 160)[h];
                }
                r[w] = ADD ? fma(-J * rh, sum, *cell_slot(w, h)) : (-J * rh) * sum;
            }
            if constexpr (MODE == P_STAGE) {
                const size_t fo = f_at(p, h);
                double qs[5];
#pragma unroll
                for (int w = 0; w < 5; ++w)
                    qs[w] = ws_rk_stage(krk, *cell_slot(5 + w, h),
                                        krk == 1 ? 0.0 : *cell_slot(10 + w, h), r[w], a.dt);
#pragma unroll
                for (int w = 0; w < 5; ++w) a.f_out.ptr[fo + w * fvs] = qs[w];
                store_prims(a, qs, p.x(h), p.y(h), p.z(h));
            } else {
#pragma unroll
                for (int w = 0; w < 5; ++w) a.du[o + w * vs] = r[w];
            }
        }
    };

    // ---- faces: this warp's component on the lane's lines
    V* col = ring + warp * 32 + lane;
    WenoLine<V> st{};
    // what the central candidates need.  FP64: first differences of lags 5..2
    // and the last face's value.  FACE: points of lags 4..2, in H, and the
    // differences of lags 4 and 3 (the next one is taken again: kept, it spilled)
    V G[4]{}, H[3]{}, qold{};
    auto shift = [&]() {
        if (FACE) {
            G[1] = G[2]; G[2] = vsub(H[2], H[1]);
            H[0] = H[1]; H[1] = H[2]; H[2] = st.t;
        } else {
            G[0] = G[1]; G[1] = G[2]; G[2] = G[3]; G[3] = st.b;
        }
    };
    // takes ring slot s (LAP position m + 4).  FACE: returns the value of the
    // face above m, as the point t_m below it + (central difference + WENO
    // correction) / 12.  Else 12 x (that value less its central candidate), and
    // in cen 12 x the central difference of cell m
    auto push = [&](auto mi, int s, V& cen) -> V {
        constexpr bool MI = decltype(mi)::value;
        [[maybe_unused]] const V below = H[0];
        if (FACE) cen = vfma(vset<V>(6.0), G[2], vsub(G[1], vsub(H[2], H[1])));
        else cen = vfms(lkc<V, lk::SEVEN>(), vadd(G[1], G[2]), vadd(G[0], G[3]));
        shift();
        V num, den;
        weno_push<MI>(st, col[s * RS], num, den);
        if constexpr (FACE)
            return vfma(vset<V>(1.0 / 12.0), vfma(num, vrcp(den), cen), below);
        else
            return weno_quot(num, den);
    };
    auto step = [&](auto mi, int s) {
        V cen;
        const V q = push(mi, s, cen);
        col[s * RS] = FACE ? q : vadd(cen, vsub(q, qold));
        qold = q;
    };
    // state from the eight points in ring slots s0 on; the face value between
    // the fourth and fifth.  The first seven only fill the state (nothing of
    // their faces is used, so it is not computed)
    auto first_face = [&](auto mi, int s0) -> V {
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            V num, den;
            shift();
            weno_push<decltype(mi)::value>(st, col[(s0 + i) * RS], num, den);
        }
        V cen;
        return push(mi, s0 + 7, cen);
    };
    // the march of one sign: state from the prologue's points, then chunk by
    // chunk with the exchange after each
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P::template bytes<MODE>() - 16);
    auto arrive = [&]() {              // end of phase `phase`
        __syncwarp();
        if (lane == 0) pencil_arrive(bars + (phase & 1));
        __syncwarp();                  // no lane polls for a phase its own warp has yet to end
        ++phase;
    };
    auto await_last = [&]() -> bool {  // all warps ended the phase before this one
        const unsigned p = phase - 1;
        uint64_t* bar = bars + (p & 1);
        if (__all_sync(0xffffffffu, pencil_wait(bar, (p >> 1) & 1, a.hold_polls, stop))) return true;
        if (lane == 0) {
            *stop = 1;
            report_stage_timeout(a);
        }
        cp_async_wait<0>();
        return false;
    };
    auto run = [&](auto mi) {
        constexpr bool MI = decltype(mi)::value;
        if (!MI) fetch_prims(2);
        else fetch_cells(0);
        qold = first_face(mi, P::SLOTS - 8);
        if (FACE) col[(P::SLOTS - 1) * RS] = qold;
        arrive();
        // the last chunk runs in full: its steps past the segment take what the
        // ring happens to hold and leave results that nobody writes out (a
        // tail of single steps would cost the march its registers)
        const int nch = (len + C - 1) / C;
        int base = 0, bprev = P::SLOTS - C;        // slots of this chunk and the one before
#pragma unroll 1
        for (int k = 0; k < nch; ++k) {
#pragma unroll
            for (int i = 0; i < C; ++i) step(mi, base + i);
            if (!await_last()) return;
            if (!MI) {
                const int s = base + 2 * C;
                split_fetched(k + 2, s < P::SLOTS ? s : s - P::SLOTS);
                fetch_prims(k + 3);
            } else if (k > 0) {
                write_cells(k - 1, bprev);
                fetch_cells(k);
            }
            arrive();
            bprev = base;
            base = base + C < P::SLOTS ? base + C : 0;
        }
        if (MI && await_last()) write_cells(nch - 1, bprev);
    };

    // ---- prologue: the table of lines, points ms-4 .. ms+3 into the last 8
    // slots and the first two chunks
    auto fixed = [&](int l, int& c1, int& c2) {       // a line's two fixed coordinates
        l = min(l, nlines - 1);
        c2 = l / n1;
        c1 = l - c2 * n1 + (DIR == 0 ? a.sy : a.sx);
        c2 += DIR == 2 ? a.sy : a.sz;
    };
    // calls f(point, index of the point, line) for this thread's points of the
    // prologue of the piece of group g from position pp on
    constexpr int NP = 8 + 2 * C;
    auto prologue = [&](long g, int pp, int plen, auto f) {
#pragma unroll 1
        for (int t = gt; t < NP * 32; t += P::NT) {
            const int i = DIR == 0 ? t % NP : t >> 5, ln = DIR == 0 ? t / NP : lane;
            if (i >= plen + 8) continue;
            Pt p;
            p.m = ms - p0 + pp - 4 + i;
            if (UNI) p.m = pencil_source<DIR>(a, p.m);
#pragma unroll
            for (int h = 0; h < NL; ++h)
                fixed((int)g * P::GL + ln + 32 * h, p.c1[h], p.c2[h]);
            f(p, i, ln);
        }
    };
    auto split_at = [&](const Pt& p, int s, int ln) {
        double e[5][NL];
#pragma unroll
        for (int f = 0; f < 5; ++f)
#pragma unroll
            for (int h = 0; h < NL; ++h) e[f][h] = __ldg(prim_at(f, p, h));
        split_into(e, p, s, ln);
    };
    if constexpr (CLO) {
        // ---- a zone: the splits of its points (nine at the high end, whose F+
        // takes the first ghost point), the five faces' values, the cells
        const int n = DIR == 0 ? a.nx : a.ny;
        const bool hi = a.clo[2 * DIR + 1] && ms - 4 >= n - kZone;
        if (hi || (a.clo[2 * DIR] && ms - 4 < kZone)) {
            const int first = hi ? n - 8 : 0, f0 = hi ? n - kZone : 0, np = hi ? 9 : 8;
            for (int t = gt; t < np * 32; t += P::NT) {
                const int i = DIR == 0 ? t % np : t >> 5, ln = DIR == 0 ? t / np : lane;
                Pt p;
                p.m = first + i + 4;
                if (UNI) p.m = pencil_source<DIR>(a, p.m);
#pragma unroll
                for (int h = 0; h < NL; ++h)
                    fixed((int)grp * P::GL + ln + 32 * h, p.c1[h], p.c2[h]);
                split_at(p, i, ln);
            }
            pencil_sync(tg);
            // face f0 + j of half h, FP64 (in the FP64 form 12 x), in slot 9 + j NL + h
            static_assert(9 + 5 * NL <= P::SLOTS, "zone's values");
            auto val = [&](int j, int h, int c, int ln) -> double* {
                return reinterpret_cast<double*>(ring + (9 + j * NL + h) * RS + c * 32 + ln);
            };
            const int inner = hi ? 0 : 4;
            const V q = minus ? first_face(std::true_type{}, 0) : first_face(std::false_type{}, 0);
#pragma unroll 1
            for (int jh = 0; jh < 5 * NL; ++jh) {
                const int j = jh / NL, h = jh - j * NL;
                auto t = [&](int i) {
                    return (double)reinterpret_cast<const CT*>(col + i * RS)[h] / LineVal<V>::SCALE;
                };
                double v;
                if (j == inner) {
                    v = (double)reinterpret_cast<const CT*>(&q)[h];
                    if (!FACE) v += 7.0 * (t(3) + t(4)) - (t(2) + t(5));
                } else {
                    if (hi && j == 1 && !minus) {      // F+ three from the end: WENO7
                        double x[8], num, den;
#pragma unroll
                        for (int k = 0; k < 8; ++k) x[k] = t(k + 1);
                        weno7_symbo_nd<false>(x, num, den);
                        v = x[3] + num / den;
                    } else {
                        v = pencil_closure(t, minus, f0 + j, n, hi);
                    }
                    v *= FACE ? LineVal<V>::SCALE : 12.0;
                }
                *val(j, h, warp, lane) = v;
            }
            pencil_sync(tg);
            for (int t = gt; t < kZone * P::GL; t += P::NT) {
                const int j = DIR == 0 ? t % kZone : t / P::GL, l = DIR == 0 ? t / kZone : t % P::GL;
                const int m = f0 + j + 4, h = l >> 5, ln = l & 31;
                if (m < ms || m >= ms + len || line0 + l >= nlines) continue;
                Pt p;
                p.m = m;
                fixed(line0 + l, p.c1[0], p.c2[0]);
                const double k = -(UNI ? 1.0 : ldg_met(a, 9, p.x(0), p.y(0), p.z(0))) * rh;
                double* du = a.du + du_at(p, 0);
#pragma unroll
                for (int w = 0; w < 5; ++w) {
                    auto sum = [&](int i) -> double {
                        const double x = *val(i, h, w, ln), y = *val(i, h, w + 5, ln);
                        // the march's sum at the face that it shares
                        return FACE && i == inner ? (double)((CT)x + (CT)y) : x + y;
                    };
                    const double d = sum(j + 1) - sum(j);
                    du[w * vs] = ADD ? fma(k, d, du[w * vs]) : k * d;
                }
            }
            return;
        }
    }
    prologue(grp, p0, len, [&](const Pt& p, int i, int ln) {
        split_at(p, i < 8 ? P::SLOTS - 8 + i : i - 8, ln);
        if (i == 0)
#pragma unroll
            for (int h = 0; h < NL; ++h) lines[ln + 32 * h] = make_int2(p.c1[h], p.c2[h]);
    });
    // the next piece's prologue, by whichever group takes it, waits for these
    const long ahead = piece.ahead;
    if (ahead >= 0) {
        const int L = DIR == 0 ? nxj : (DIR == 1 ? nyj : nzj);
        const long g = ahead / L;
        prologue(g, (int)(ahead - g * L), 2 * C, [&](const Pt& p, int, int) {
            if (p.m >= ms - p0 - 4 && p.m < ms - p0 + L + 4)
#pragma unroll
                for (int f = 0; f < 5; ++f)
#pragma unroll
                    for (int h = 0; h < NL; ++h) prefetch_l2(prim_at(f, p, h));
        });
    }
    pencil_sync(tg);
    if (!minus) run(std::false_type{});
    else run(std::true_type{});
}

// Work of one CTA: the contiguous share [pos, end) of the (line group,
// position) space, which its two thread groups take piece by piece (a pair of
// independent CTAs per SM ended up to 30% apart: the older one's warps are
// served first).  A piece stays within a line group and within about a third
// of what is left, so that the groups end together, but is not so short that
// its 8-point prologue dominates.
struct PencilShare {
    unsigned long long pos;
    long long end;
    int minlen;
    PencilPiece piece[2];          // of each thread group
};
__device__ __forceinline__ int pencil_piece(const PencilShare& s, long long pos, int line_left) {
    const long long rem = s.end - pos;
    const long long want = max(rem > 256 ? rem / 3 : (rem + 1) / 2, (long long)s.minlen);
    int len = (int)min(min((want + 4) / 5 * 5, rem), (long long)line_left);   // whole chunks
    if (line_left - len < 10) len = (int)min((long long)line_left, rem);
    return len;
}
__device__ __forceinline__ void pencil_share(PencilShare& s, long total) {
    s.pos = total * (long)blockIdx.x / (long)gridDim.x;
    s.end = total * ((long)blockIdx.x + 1) / (long)gridDim.x;
    s.minlen = (int)min(16LL, (s.end - (long long)s.pos + 1) / 2);
}
// The next piece of the share: grid_of(pos, local, total, L) gives the grid of
// a position, the place within it, its number of places and the march length
// of its lines; stop_of(grid, p0, L) the grid's pencil_stop.
template <typename F, typename S>
__device__ __forceinline__ PencilPiece pencil_take(PencilShare& s, F grid_of, S stop_of) {
    long long pos = (long long)*reinterpret_cast<volatile unsigned long long*>(&s.pos);
    while (pos < s.end) {
        PencilPiece p;
        long local = 0, total = 0;
        int L = 0;
        p.grid = grid_of((long)pos, local, total, L);
        p.grp = local / L;
        p.p0 = (int)(local - p.grp * L);
        p.len = pencil_piece(s, pos, stop_of(p.grid, p.p0, L) - p.p0);
        p.ahead = pos + p.len < s.end && local + p.len < total ? local + p.len : -1;
        const long long seen = (long long)atomicCAS(&s.pos, (unsigned long long)pos,
                                                    (unsigned long long)(pos + p.len));
        if (seen == pos) return p;
        pos = seen;
    }
    return PencilPiece{0, 0, 0, 0, -1};
}

// One pass along DIR over the job of `a`: every CTA takes an equal contiguous
// share of the (line group, position) space.
template <int DIR, typename V, bool UNI, int MODE, bool CLO>
__global__ void __launch_bounds__(640, 1)
    pencil_rhs_kernel(const __grid_constant__ RhsArgs a, int krk) {
    extern __shared__ __align__(16) unsigned char pencil_smem[];
    __shared__ PencilShare sh;
    __shared__ int stop[2];
    constexpr size_t G = PencilLayout<V>::template bytes<MODE>();
    if (threadIdx.x == 0) {
        int L = 0;
        pencil_share(sh, pencil_work<DIR, PencilLayout<V>::GL>(a, L));
        pencil_init_bars(pencil_smem + G - 16, G, a.hold_polls > 0);
        stop[0] = stop[1] = 0;
    }
    __syncthreads();
    const int tg = threadIdx.x >= 320;
    const bool lead = threadIdx.x == tg * 320;
    unsigned phase = 0;
    for (;;) {
        if (lead)
            sh.piece[tg] = pencil_take(sh, [&](long pos, long& local, long& total, int& L) {
                total = pencil_work<DIR, PencilLayout<V>::GL>(a, L);
                local = pos;
                return 0;
            }, [&](int, int p0, int L) { return pencil_stop<DIR, CLO>(a, p0, L); });
        pencil_sync(tg);                   // the piece is known, the last one is out
        const PencilPiece& p = sh.piece[tg];
        volatile int* gave_up = &stop[tg];
        if (p.len == 0 || *gave_up) break;
        pencil_segment<DIR, V, UNI, MODE, CLO>(a, krk, pencil_smem + tg * G, tg, phase, gave_up, p);
    }
}

// The same pass over the grids of a batch: argument table `grids`, and
// woff[i] the pass's work before grid i (woff[n] the total).  A share may
// cross grids; each group copies the arguments of its piece's grid (without
// the tensor maps) to shared memory.
constexpr int kArgWords = (int)(offsetof(RhsArgs, tma) / 4);
static_assert(offsetof(RhsArgs, hold_polls) < offsetof(RhsArgs, tma) &&
              offsetof(RhsArgs, gk) < offsetof(RhsArgs, tma) && offsetof(RhsArgs, tma) % 4 == 0,
              "the line passes' arguments come before the maps");
template <int DIR, typename V, int MODE, bool CLO>
__global__ void __launch_bounds__(640, 1)
    pencil_batch_kernel(const RhsArgs* __restrict__ grids, const long* __restrict__ woff, int n,
                        int krk) {
    extern __shared__ __align__(16) unsigned char pencil_smem[];
    __shared__ PencilShare sh;
    __shared__ int stop[2];
    __shared__ __align__(64) uint32_t argw[2][(kArgWords + 15) / 16 * 16];
    constexpr size_t G = PencilLayout<V>::template bytes<MODE>();
    if (threadIdx.x == 0) {
        pencil_share(sh, woff[n]);
        pencil_init_bars(pencil_smem + G - 16, G, grids[0].hold_polls > 0);
        stop[0] = stop[1] = 0;
    }
    __syncthreads();
    const int tg = threadIdx.x >= 320;
    const bool lead = threadIdx.x == tg * 320;
    const RhsArgs& a = *reinterpret_cast<const RhsArgs*>(argw[tg]);
    unsigned phase = 0;
    int held = -1;
    for (;;) {
        if (lead)
            sh.piece[tg] = pencil_take(sh, [&](long pos, long& local, long& total, int& L) {
                int lo = 0, hi = n;        // the grid holding pos: woff[lo] <= pos < woff[lo+1]
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (woff[mid] <= pos) lo = mid; else hi = mid;
                }
                total = pencil_work<DIR, PencilLayout<V>::GL>(grids[lo], L);
                local = pos - woff[lo];
                return lo;
            }, [&](int grid, int p0, int L) { return pencil_stop<DIR, CLO>(grids[grid], p0, L); });
        pencil_sync(tg);                   // the piece is known, the last one is out
        const PencilPiece& p = sh.piece[tg];
        volatile int* gave_up = &stop[tg];
        if (p.len == 0) break;
        if (*gave_up) {                    // the pieces it would have taken: reported, not done
            if (lead) report_stage_timeout(grids[p.grid]);
            pencil_sync(tg);
            continue;
        }
        if (held != p.grid) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(grids + p.grid);
            for (int w = threadIdx.x - tg * 320; w < kArgWords; w += 320)
                argw[tg][w] = __ldg(src + w);
            held = p.grid;
            pencil_sync(tg);
        }
        pencil_segment<DIR, V, true, MODE, CLO>(a, krk, pencil_smem + tg * G, tg, phase, gave_up, p);
    }
}

// Launch of a line pass of one CTA per SM, but no more than `most`.  The
// dynamic shared memory size is set and the SM count read once per device per
// kernel.
template <typename Kern, typename... Args>
int pencil_launch(Kern kern, int* blocks, int threads, size_t smem, long most, cudaStream_t st,
                  Args... args) {
    int dev = 0;
    WS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(WS_ERR_UNSUPPORTED, "device ordinal >= 64");
    if (!blocks[dev]) {
        int sms = 0;
        WS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        WS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
        blocks[dev] = sms;
    }
    kern<<<(unsigned)std::min<long>(blocks[dev], std::max(1L, most)), threads, smem, st>>>(args...);
    WS_CUDA(cudaGetLastError());
    return WS_OK;
}
constexpr long kAllSms = 1L << 40;

// work of pass dir over nx x ny x nz cells: groups of gl lines x positions
inline long pencil_places(long nx, long ny, long nz, int dir, int gl) {
    const long nl = dir == 0 ? ny * nz : (dir == 1 ? nx * nz : nx * ny);
    return (nl + gl - 1) / gl * (dir == 0 ? nx : (dir == 1 ? ny : nz));
}

// Host side of the passes for one value type and metric kind.
template <typename V, bool UNI>
struct PencilLauncher {
    static constexpr int GL = 32 * LineVal<V>::NL;
    static constexpr bool MIXED = LineVal<V>::NL > 1;
    // one grid (job of a); a CTA with fewer than 2 positions to march would
    // spend itself on prologues
    template <int DIR, int MODE, bool CLO = false>
    static int one(const RhsArgs& a, int krk, cudaStream_t st) {
        static int blocks[64] = {0};
        return pencil_launch(
            pencil_rhs_kernel<DIR, V, UNI, MODE, CLO>, blocks, 640,
            2 * PencilLayout<V>::template bytes<MODE>(),
            pencil_places(a.ex - a.sx, a.ey - a.sy, a.ez - a.sz, DIR, GL) / 2, st, a, krk);
    }
    // the z pass with the stage update of the mixed form (12 warps: 16 leave
    // 128 registers)
    static int lane_stage(const RhsArgs& a, int krk, cudaStream_t st) {
        static int blocks[64] = {0};
        return pencil_launch(pencil_lane_kernel<12>, blocks, 384,
                             12 * LaneLayout::WARP * sizeof(float), kAllSms, st, a, krk);
    }
    // the x and y passes (each pass's closure instance when the grid has a
    // CLOSURE face in its direction)
    static int xy(const RhsArgs& a, bool add_x, cudaStream_t st) {
        int rc;
        if (a.clo[0] | a.clo[1])
            rc = add_x ? one<0, P_ADD, true>(a, 0, st) : one<0, P_STORE, true>(a, 0, st);
        else
            rc = add_x ? one<0, P_ADD>(a, 0, st) : one<0, P_STORE>(a, 0, st);
        if (rc) return rc;
        return (a.clo[2] | a.clo[3]) ? one<1, P_ADD, true>(a, 0, st) : one<1, P_ADD>(a, 0, st);
    }
    // plain RHS: x (=, or += with add_x), y (+=), z (+=)
    static int rhs(const RhsArgs& a, bool add_x, cudaStream_t st) {
        int rc = xy(a, add_x, st);
        return rc ? rc : one<2, P_ADD>(a, 0, st);
    }
    // stage: x, y into du, then z with the stage update
    static int stage(const RhsArgs& a, bool add_x, int krk, cudaStream_t st) {
        if constexpr (UNI) {
            int rc = xy(a, add_x, st);
            if (rc) return rc;
            if constexpr (MIXED) return lane_stage(a, krk, st);
            else return one<2, P_STAGE>(a, krk, st);
        } else {
            return fail(WS_ERR_UNSUPPORTED, "stage update needs Cartesian metrics");
        }
    }

    // a batch: argument table g of n grids, woff = the passes' work prefix
    // tables of n + 1 entries each (x, y, z, z in groups of 32 lines); krk 0:
    // RHS into each du; clo: some grid has a CLOSURE face
    template <int DIR, int MODE, bool CLO = false>
    static int one_batch(const RhsArgs* g, const long* woff, int n, int krk, cudaStream_t st) {
        static int blocks[64] = {0};
        return pencil_launch(pencil_batch_kernel<DIR, V, MODE, CLO>, blocks, 640,
                             2 * PencilLayout<V>::template bytes<MODE>(), kAllSms, st, g,
                             woff + DIR * (n + 1), n, krk);
    }
    // the same z pass of the mixed form: with its arguments from global memory
    // it needs the registers of 8 warps
    static int lane_stage_batch(const RhsArgs* g, const long* woff, int n, int krk,
                                cudaStream_t st) {
        static int blocks[64] = {0};
        return pencil_launch(pencil_lane_batch_kernel<8>, blocks, 256,
                             8 * LaneLayout::WARP * sizeof(float), kAllSms, st, g,
                             woff + 3 * (n + 1), n, krk);
    }
    static int batch(const RhsArgs* g, const long* woff, int n, int krk, bool clo,
                     cudaStream_t st) {
        int rc = clo ? one_batch<0, P_STORE, true>(g, woff, n, 0, st)
                     : one_batch<0, P_STORE>(g, woff, n, 0, st);
        if (rc) return rc;
        rc = clo ? one_batch<1, P_ADD, true>(g, woff, n, 0, st)
                 : one_batch<1, P_ADD>(g, woff, n, 0, st);
        if (rc) return rc;
        if (!krk) return one_batch<2, P_ADD>(g, woff, n, 0, st);
        if constexpr (MIXED) return lane_stage_batch(g, woff, n, krk, st);
        else return one_batch<2, P_STAGE>(g, woff, n, krk, st);
    }
};

}  // namespace ws
