// vs_resident.cuh -- a whole run of a tube on one thread-block cluster, the
// state in registers and the maps in shared memory.
//
// A time step moves 37 bytes per cell through HBM when the planes live there,
// or half of that with two steps per launch.  Here a tube's planes are read
// once per run: a cluster of C CTAs holds all of its cells, and only the
// listener samples (and, for the adjoint, the state history) leave the chip.
// The tubes of a batch are independent, so clusters of a large batch follow
// one another on the SMs without any synchronisation between them.
//
// Decomposition.  The interior rows are split into C contiguous bands, one
// per CTA; a band into nwy row groups and the columns 0 .. W-2 into nwx tiles
// of 64, one warp per (group, tile).  A lane owns two adjacent columns and
// the R rows of its group: P, Vx, Vy of those 2 R cells stay in registers as
// float pairs for the whole run, and every operation on a pair is one packed
// instruction (add / mul / fma .f32x2), each half rounded as the scalar
// operation rounds it.  The step loop is compiled for every R up to RMAX, so
// its rows are straight-line code and independent instruction streams.
//
// One step (FDTDEngineCPU.cpp:257-288):
//   P' of rows r0-1 .. r1 of the group: the row above the group is recomputed
//     from its owner's velocities, so one exchange per step is enough
//   barrier of the group's warps (first-column P' of every tile)
//   V' of rows r0 .. r1; last-row (Vx, Vy) to the group below, first-row Vy to
//     the group above: shared memory, or between CTAs st.async counted on the
//     receiver's mbarrier (double-buffered by step parity)
//   CTA barrier; the next step's first and last group wait (bounded) for the
//     neighbour CTAs' rows
// Arithmetic: that of the other kernels, operation for operation, so the
// values are theirs.  fast_math: the reciprocal form (rcp(dP) is formed once
// instead of every step).  Reference arithmetic: the IEEE quotients from the
// correctly rounded reciprocals, see quotients().  Neighbourhood factors (walls,
// PML, source) come from tables indexed by the descriptors of the lane's two
// cells: a tube has some 50 to 75 distinct pairs, packed as the operations take
// them.  The wall and source terms run only in blocks of rows that hold such a
// cell.  Cells outside the frame and ring cells have zero coefficients and so
// keep their zeros.  The two-mass source runs in a warp of its own
// (run_two_mass), one step ahead of the velocities it enters.
//
// What bounds it: no DRAM traffic in the loop.  256 vowel tubes in the
// reciprocal form (2 CTAs of 16 warps a tube, 6 to 12 rows a lane): 8.4 us per
// time step (two-step strips 17.4), about 65 instructions per 64-cell row and
// step at 0.4 per scheduler and cycle, half of the shared-memory pipe, the rest
// the latency of a warp's own chain and the two barriers.  One 55 x 253 tube
// (16 CTAs, 1 or 2 rows a lane): 0.67 us per step, 1.1 in the reference
// arithmetic (two-step strips 2.5 and 4.2), about 0.5 of it the exchange and the
// two barriers; with the double two-mass model 0.88, its own chain of double
// operations.  Measured and not kept: scalar instead of
// packed operations (82 instructions, the same time); 64 registers for twice
// the warps (spills, 16 us per step of the 256 tubes); 168 registers with 12
// warps, taller groups, or a cluster size per tube (10.2 to 11.5 us).
#pragma once

#include <cooperative_groups.h>

#include <algorithm>

#include "vs_cellmath.cuh"
#include "vs_mbarrier.cuh"

namespace cg = cooperative_groups;

namespace vsb {
namespace {

using u64 = unsigned long long;

__device__ __forceinline__ u64 pk(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float plo(u64 v) {
    return __uint_as_float((uint32_t)v);
}
__device__ __forceinline__ float phi(u64 v) {
    return __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// a - b, rounded once.  m1 = (-1, -1) comes from shared memory: the
// compiler rewrites a packed difference of two products into an fma, whose
// unrounded product would change the values.
__device__ __forceinline__ u64 diff2(u64 a, u64 b, u64 m1) {
    return fma2(b, m1, a);
}

template <int I>
struct Idx {
    static constexpr int value = I;
    __device__ constexpr operator int() const { return I; }
};

template <int B, int E, class F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (B < E) {
        f(Idx<B>{});
        static_for<B + 1, E>(f);
    }
}

__device__ __forceinline__ void group_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

constexpr int kStepBar = 15;                     // named barrier of the tile warps; the groups use 1 .. 8

__device__ __forceinline__ void step_sync(int count) {
    asm volatile("bar.sync %0, %1;" ::"n"(kStepBar), "r"(count) : "memory");
}

// A value and its step in one 8-byte word (single-copy atomic): written by one
// thread, polled (bounded) by the readers.
__device__ __forceinline__ u64 tagged(int n, float v) { return ((u64)(uint32_t)n << 32) | __float_as_uint(v); }

__device__ __forceinline__ bool poll_tagged(const volatile u64* w, int n, uint32_t limit, float* v) {
    u64 x = *w;
    for (uint32_t i = 1; (uint32_t)(x >> 32) != (uint32_t)n && i < limit; ++i) x = *w;
    *v = __uint_as_float((uint32_t)x);
    return (uint32_t)(x >> 32) == (uint32_t)n;
}

// Asynchronous store into a cluster CTA's shared memory whose bytes count
// against that CTA's mbarrier `bar` (both cluster addresses): the receiver
// learns of its arrival from the mbarrier phase, the sender issues no fence.
__device__ __forceinline__ void st_async_pair(uint32_t addr, u64 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v),
                 "r"(bar)
                 : "memory");
}

// Shared memory by 32-bit address: the step loop keeps a few base registers and
// reaches everything by constant offsets (through generic pointers the
// compiler forms the cluster window's address again at every use).  Volatile,
// so they keep their order against the barriers.
__device__ __forceinline__ u64 lds64(uint32_t a) {
    u64 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ ulonglong2 lds128(uint32_t a) {
    ulonglong2 v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 ldsf4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float ldsf(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t ldsu16(uint32_t a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts64(uint32_t a, u64 v) { asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ void sts128(uint32_t a, u64 x, u64 y) {
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void stsf4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
// m ? x : y for m all ones or zero: one logic operation, no predicate
__device__ __forceinline__ float bitsel(uint32_t m, float x, float y) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r) : "r"(m), "r"(__float_as_uint(x)), "r"(__float_as_uint(y)));
    return __uint_as_float(r);
}

constexpr int kTileCols = 64;
constexpr int kMaxWarps = 16;
constexpr int kMaxRows = 12;      // rows per lane the registers hold (72 of 128 for the state)

// Shared-memory layout of one CTA for nwx tiles, ng row-group slots and a band
// of nrow rows.  Per (group, tile) a ghost block: (Vx, Vy) of the row above for
// both step parities, then Vy of the row below; the ghost row below the band is
// in block row ng, so the neighbour CTAs address block rows 0 and ng at offsets
// that do not depend on nrow.  Per tile the records of the band's rows (from
// the row above it) at a constant stride: rcp(dP) and dX, dY, descriptors.
constexpr int kGhostBytes = 2 * 512 + 2 * 256;
constexpr int kGhostB = 2 * 512;
constexpr int kRecY = 512, kRecP = 768;         // (rcp(dP), dX) at 0, dY, and in the reference arithmetic dP
__host__ __device__ constexpr int rec_desc(bool exact) { return exact ? 1024 : 768; }
__host__ __device__ constexpr int rec_bytes(bool exact) { return rec_desc(exact) + 64; }
// per (group, tile edge): Vx dX to the left of it (row i at i - 1), then P' to the right of it
// (rows 2 .. R-1 at i - 2, rows 1 and R at kMaxRows and kMaxRows + 1)
constexpr int kEdgeP = kMaxRows;
constexpr int kEdgeFloats = 2 * kMaxRows + 4;

constexpr int kDrainPolls = 1 << 14;             // about 2 ms; a store into a neighbour takes about 1 us
constexpr int kHashSlots = 1024;
constexpr int kMaxPairs = 128;                   // descriptor pairs of a tube (vowel tubes: 50 to 75)
constexpr int kTab = kMaxPairs * 16;             // one table of 16-byte entries
// fixed offsets: barriers, give-up flags, (-1, -1); then the pair tables.  Reciprocal form: (g, ce),
// (al_x, al_y), (zo_x, -zi_x), (zo_y, -zi_y).  Reference arithmetic: (-sP, -), (-den_x, 1 / den_x),
// (-den_y, 1 / den_y), (mB_x, -mS_x), (A_x, B_x), (mB_y, -mS_y), (A_y, B_y), (W_x, W_y); the wall term's
// pressure is A Pc + B Pn.
constexpr int kOffBar = 0, kOffFail = 16, kOffTop = 28, kOffM1 = 32;     // kOffTop: see quotients()
// two-mass source: excitation values in flight (more than the largest cluster has CTAs), the excitation
// cell's P' by step parity
constexpr int kExeRing = 32;
constexpr int kOffRing = 64, kOffWord = kOffRing + 8 * kExeRing;
// by CTA of the cluster: the exchanges it sent if it gave up, else the steps of the launch
constexpr int kMaxCtas = 16, kOffSent = kOffWord + 16, kOffTab = kOffSent + 4 * kMaxCtas;
__host__ __device__ constexpr int off_ghost(bool exact) { return kOffTab + (exact ? 8 : 4) * kTab; }

struct ResLayout {
    int edge, rec, bytes;
};

__host__ __device__ inline ResLayout res_layout(int nwx, int ng, int nrow, bool exact) {
    ResLayout L{};
    const int ghost = (ng + 1) * nwx * kGhostBytes;
    // the ghost rows' place also holds the pair table's hash while the block starts
    L.edge = off_ghost(exact) + (ghost > kHashSlots * 4 ? ghost : kHashSlots * 4);
    L.rec = L.edge + (ng * (nwx + 1) * kEdgeFloats * 4 + 15) / 16 * 16;
    L.bytes = (L.rec + nwx * (nrow + 2) * rec_bytes(exact) + 127) / 128 * 128;
    return L;
}

// What a warp needs to run its tile.
struct TileCtx {
    const TubeDev* T;
    RunState* rs;
    unsigned char* sm;
    ResLayout L;
    int nsteps;
    int C, k;                 // cluster size and rank
    int nwx, ng, nwy, nrow;   // tiles, group slots, groups in use, rows of the band
    int g, t;                 // this warp's group and tile
    int j0;                   // band row index of the row above the group (0 = the row above the band)
    int r0;                   // first row of the group
    int tube, nw;             // nw: tile warps of the CTA
    bool tmm;                 // two-mass source
};

// a / b for b = -nb and y = 1 / b correctly rounded, in double: the quotient of
// two floats lies at least 2^-50 of itself away from every value half-way
// between two floats (subnormal ones too) that it does not equal, so a double
// quotient good to an ulp rounds to the IEEE float quotient.  y refined once is
// good to 2^-47, the quotient corrected by its residual to an ulp of the double.
__device__ __forceinline__ float quotient_by_double(float a, float nb, float y) {
    const double d = nb, y0 = y, n = a;
    const double y1 = __fma_rn(y0, __fma_rn(d, y0, 1.0), y0);
    const double q = __dmul_rn(n, y1);
    return __double2float_rn(__fma_rn(__fma_rn(d, q, n), y1, q));
}

// a[k] / b[k] for N pairs, correctly rounded: nb = -b, y = 1 / b correctly
// rounded (0 where the result is 0 by definition: ring and no-pressure cells).
// Two fused corrections of a y (P. Markstein, IBM J. Res. Dev. 34(1), 1990) give
// the IEEE quotient while nothing on the way leaves the normal range, which
// holds for numerators of 2^-80 .. 2^100 and denominators of 2^-26 .. 2^46.  A
// warp that meets a smaller numerator (the wave front of a run's first steps,
// which stretches over most of the frame) forms the block's quotients in
// double; one that meets a larger numerator, or a tube with another denominator
// (top = infinity), divides.  Steps 128 to 512 from rest of 256 tubes: 122 us a
// step when such blocks divided, 28 in double, 18 past the front (two-step
// strips, which divide: 57).
template <int N>
__device__ __forceinline__ void quotients(u64 (&a)[N], const u64 (&nb)[N], const u64 (&y)[N], float top) {
    u64 q[N], r[N];
    bool odd = false;
    auto tiny = [](float v) { return (__float_as_uint(v) & 0x7fffffffu) - 1u < 0x17800000u - 1u; };   // 0 < |v| < 2^-80
    static_for<0, N>([&](auto kc) {
        odd = odd || tiny(plo(a[kc])) || tiny(phi(a[kc]));
        top = fmaxf(top, fmaxf(fabsf(plo(a[kc])), fabsf(phi(a[kc]))));
    });
    static_for<0, N>([&](auto kc) { q[kc] = mul2(a[kc], y[kc]); });
    static_for<0, N>([&](auto kc) { r[kc] = fma2(nb[kc], q[kc], a[kc]); });
    static_for<0, N>([&](auto kc) { q[kc] = fma2(r[kc], y[kc], q[kc]); });
    static_for<0, N>([&](auto kc) { r[kc] = fma2(nb[kc], q[kc], a[kc]); });
    static_for<0, N>([&](auto kc) { q[kc] = fma2(r[kc], y[kc], q[kc]); });
    const bool large = top > 1.2676506e30f;
    if (__any_sync(0xffffffffu, odd || large)) {
        auto each = [&](auto&& div) {
            static_for<0, N>([&](auto kc) {
                const float y0 = plo(y[kc]), y1 = phi(y[kc]);
                q[kc] = pk(y0 == 0.0f ? 0.0f : div(plo(a[kc]), plo(nb[kc]), y0),
                           y1 == 0.0f ? 0.0f : div(phi(a[kc]), phi(nb[kc]), y1));
            });
        };
        if (__any_sync(0xffffffffu, large)) each([](float v, float nd, float) { return fdiv_z(v, -nd); });
        else each([](float v, float nd, float rc) { return quotient_by_double(v, nd, rc); });
    }
    static_for<0, N>([&](auto kc) { a[kc] = q[kc]; });
}

// Denominators quotients() takes without dividing (the maps' depths times 1 +
// sigma, and the velocities' mB + mS: 2^-22 .. 2^20 for every tube built here;
// a caller's own maps may hold others).
__device__ __forceinline__ bool plain_den(float b) { return b >= 1.4901161e-8f && b <= 7.0368744e13f; }

// Up to kRegRows rows per group the maps and the pressure and velocity factors
// stay in registers too; taller groups read them from shared memory.
constexpr int kRegRows = 3;

template <int R, bool HIST, bool EXACT, bool TMM>
__device__ __forceinline__ void run_tile(const TileCtx& X) {
    constexpr int kOffGhost = off_ghost(EXACT), kRecBytes = rec_bytes(EXACT), kRecD = rec_desc(EXACT);
    constexpr unsigned kAll = 0xffffffffu;
    constexpr bool inReg = R <= kRegRows;
    const TubeDev* __restrict__ T = X.T;
    RunState* __restrict__ rs = X.rs;
    int lane;                          // volatile: not read again at every use
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    const int nwx = X.nwx, t = X.t, g = X.g, r0 = X.r0;
    const int lanes = nwx * 32;
    const int W = T->W, pitch = T->pitch;
    const int x0 = kTileCols * t + 2 * lane;
    const int64_t pl = T->plane;
    const int64_t n0 = rs->step;
    const int par0 = (int)(n0 & 1), nsteps = X.nsteps;
    const bool in0 = x0 >= 1 && x0 <= W - 2, in1 = x0 + 1 <= W - 2;

    const ResLayout& L = X.L;
    uint64_t* bar = reinterpret_cast<uint64_t*>(X.sm + kOffBar);
    volatile int* sfail = reinterpret_cast<volatile int*>(X.sm + kOffFail);
    const bool top = g == 0, bottom = g == X.nwy - 1;
    uint32_t sb = smem_u32(X.sm);
    asm volatile("" : "+r"(sb));
    // ghost rows of this tile, by parity
    const uint32_t gT = sb + kOffGhost + (g * nwx + t) * kGhostBytes + lane * 16;
    const uint32_t gB = sb + kOffGhost + ((bottom ? X.ng : g) * nwx + t) * kGhostBytes + kGhostB + lane * 8;
    const uint32_t edge = sb + L.edge + (g * (nwx + 1) + t) * kEdgeFloats * 4;
    const uint32_t rows = sb + L.rec + (t * (X.nrow + 2) + X.j0) * kRecBytes;
    const uint32_t rec = rows + lane * 16, recY = rows + kRecY + lane * 8, sD = rows + kRecD + lane * 2;
    auto map_s = [&](int i) { return lds128(rec + i * kRecBytes); };
    auto dy_s = [&](int i) { return lds64(recY + i * kRecBytes); };
    auto id_at = [&](int i) { return ldsu16(sD + i * kRecBytes) + sb; };  // of the pair's table entries
    auto g_at = [&](uint32_t o) { return lds64(o + kOffTab); };
    auto al_at = [&](uint32_t o) { return lds128(o + kOffTab + kTab); };
    auto zx_at = [&](uint32_t o) { return lds128(o + kOffTab + 2 * kTab); };
    auto zy_at = [&](uint32_t o) { return lds128(o + kOffTab + 3 * kTab); };
    auto ce_at = [&](uint32_t o) { return lds64(o + kOffTab + 8); };
    auto tab_at = [&](uint32_t o, int k) { return lds128(o + kOffTab + k * kTab); };
    auto dp_s = [&](int i) { return lds64(recY + (kRecP - kRecY) + i * kRecBytes); };
    const uint32_t first = lane == 0 ? ~0u : 0u, last = lane == 31 ? ~0u : 0u;

    // ---- state of the group's rows (0 = the row above, whose P is kept too)
    u64 P[R + 1], VX[R + 1], VY[R + 1];
    u64 rX[inReg ? R + 1 : 1], rY[inReg ? R + 2 : 1], rP[inReg ? R + 1 : 1];
    u64 rG[inReg ? R + 1 : 1], rAx[inReg ? R + 1 : 1], rAy[inReg ? R + 1 : 1];
    uint32_t gnm = 0;                        // per row: the tile has a cell with wall or source terms
    uint32_t dvm = 0;                        // reference arithmetic, per row: a velocity division
    bool srcm = false;
    {
        const float* __restrict__ gP = T->P[0] + par0 * pl;
        static_for<0, R + 1>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            const int64_t o = (int64_t)(r0 - 1 + i) * pitch + x0;
            P[i] = pk(in0 ? gP[o] : 0.0f, in1 ? gP[o + 1] : 0.0f);
            VX[i] = pk(in0 ? gP[2 * pl + o] : 0.0f, in1 ? gP[2 * pl + o + 1] : 0.0f);
            VY[i] = pk(in0 ? gP[4 * pl + o] : 0.0f, in1 ? gP[4 * pl + o + 1] : 0.0f);
            const ulonglong2 m = map_s(i);
            if constexpr (inReg) { rP[i] = m.x; rX[i] = m.y; rY[i] = dy_s(i); }
            const unsigned d = id_at(i);
            const u64 gg = g_at(d);
            if constexpr (EXACT) {
                const ulonglong2 bx = tab_at(d, 4), by = tab_at(d, 6), mx = tab_at(d, 3), my = tab_at(d, 5);
                const ulonglong2 w = tab_at(d, 7), qx = tab_at(d, 1), qy = tab_at(d, 2);
                const u64 one = pk(1.0f, 1.0f);
                if constexpr (inReg) { rG[i] = gg; rAx[i] = dp_s(i); }
                const bool c = w.x != 0 || w.y != 0;
                const bool gn = c || bx.x != 0 || bx.y != 0 || by.x != 0 || by.y != 0 || mx.x != one || my.x != one;
                if (i > 0) {
                    gnm |= (uint32_t)__any_sync(kAll, gn) << i;
                    dvm |= (uint32_t)__any_sync(kAll, gn || qx.y != one || qy.y != one) << i;
                    srcm = srcm || __any_sync(kAll, c);
                }
            } else {
                const ulonglong2 al = al_at(d);
                const float4 zx = ldsf4(d + kOffTab + 2 * kTab), zy = ldsf4(d + kOffTab + 3 * kTab);
                const u64 ce2 = ce_at(d);
                const float2 ce = make_float2(plo(ce2), phi(ce2));
                if constexpr (inReg) { rG[i] = gg; rAx[i] = al.x; rAy[i] = al.y; }
                const bool c = ce.x != 0.0f || ce.y != 0.0f;
                const bool gn = c || zx.x != 0.0f || zx.y != 0.0f || zx.z != 0.0f || zx.w != 0.0f || zy.x != 0.0f ||
                                zy.y != 0.0f || zy.z != 0.0f || zy.w != 0.0f;
                if (i > 0) {
                    gnm |= (uint32_t)__any_sync(kAll, gn) << i;
                    srcm = srcm || __any_sync(kAll, c);
                }
            }
            asm volatile("" ::: "memory");
        });
        if constexpr (inReg) rY[R + 1] = dy_s(R + 1);
    }
    auto x_at = [&](auto ic) -> u64 {
        if constexpr (inReg) return rX[decltype(ic)::value];
        else return lds64(rec + decltype(ic)::value * kRecBytes + 8);
    };
    auto y_at = [&](auto ic) -> u64 {
        if constexpr (inReg) return rY[decltype(ic)::value];
        else return dy_s(decltype(ic)::value);
    };
    const float K1 = T->K1, bco = T->bcoef;
    const u64 cK = EXACT ? pk(K1, K1) : pk(-K1, -K1);
    const bool eigen = (T->flags & TUBE_EIGEN) != 0;
    const u64 zz = pk(T->zinv, T->zinv);
    const u64 m1 = lds64(sb + kOffM1);
    const u64 bc = pk(in0 ? bco : 0.0f, in1 ? bco : 0.0f);        // ring columns keep zero velocities
    const bool tmm = TMM && X.tmm;
    const float* __restrict__ src = tmm ? nullptr : T->src + n0;
    // steps whose source value is in the table
    const int src_steps = srcm && !tmm ? (int)min((int64_t)nsteps, max(T->src_len - n0, (int64_t)0)) : 0;
    const int lis_y = T->lis_y, lis_x = T->lis_x;
    const bool lis_warp = lis_y >= r0 && lis_y < r0 + R && lis_x / kTileCols == t;
    const int lis_i = lis_y - r0 + 1;
    float* __restrict__ trace = rs->trace + (int64_t)X.tube * rs->trace_stride + (n0 - rs->run_start);

    // two-mass source: the warp that holds the excitation cell publishes its P'
    const volatile u64* ring = reinterpret_cast<const volatile u64*>(X.sm + kOffRing);
    volatile u64* word = reinterpret_cast<volatile u64*>(X.sm + kOffWord);
    const int exc_y = T->exc_y, exc_x = T->exc_x;
    const bool exc_warp = tmm && exc_y >= r0 && exc_y < r0 + R && exc_x / kTileCols == t;
    const bool polls = tmm && srcm;

    // neighbours: local ghost slots, or the slots of the CTAs above / below
    const bool rem_up = top && X.k > 0, rem_dn = bottom && X.k + 1 < X.C;
    const bool waits = rem_up || rem_dn;
    uint32_t upB_a = 0, dnT_a = 0, up_bar = 0, dn_bar = 0;
    if (rem_up) {
        upB_a = cluster_addr(X.sm + kOffGhost + (X.ng * nwx + t) * kGhostBytes + kGhostB + lane * 8, X.k - 1);
        up_bar = cluster_addr(bar, X.k - 1);
    }
    if (rem_dn) {
        dnT_a = cluster_addr(X.sm + kOffGhost + t * kGhostBytes + lane * 16, X.k + 1);
        dn_bar = cluster_addr(bar, X.k + 1);
    }
    // the groups above and below in this CTA: their ghost blocks are one block row away
    const int brow = nwx * kGhostBytes;
    const uint32_t expect = (X.k > 0 ? 16u * lanes : 0u) + (X.k + 1 < X.C ? 8u * lanes : 0u);
    const uint32_t limit = first_wait_limit(rs);
    uint32_t phase = 0;

    float* hist = HIST ? T->hist + (n0 + 1 - rs->run_start) * 3 * pl + (int64_t)r0 * pitch + x0 : nullptr;

#pragma unroll 1
    for (int m = 0; m < nsteps; ++m) {
        const int p = (par0 + m) & 1, q = p ^ 1;
        float exe = m < src_steps ? __ldg(src + m) : 0.0f;
        // ---- P' of N rows (compile-time list `row`), written stage by stage so that
        // the rows' loads, shuffles and operation chains overlap; vx: their Vx,
        // w / wn: Vy dY of the row and of the row below, eul: Vx dX left of the tile
        auto pblock = [&](auto... ic) {
            constexpr int N = sizeof...(ic);
            return [&](const u64 (&vx)[N], const u64 (&w)[N], const u64 (&wn)[N], const float (&eul)[N]) {
                constexpr int row[N] = {decltype(ic)::value...};
                u64 dx[N], rp[N], u[N], gf[N], sum[N];
                unsigned d[N];
                float ul[N];
                static_for<0, N>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    [[maybe_unused]] constexpr int i = row[k];
                    if constexpr (inReg) { rp[k] = rP[i]; dx[k] = rX[i]; }
                    else { const ulonglong2 mm = map_s(i); rp[k] = mm.x; dx[k] = mm.y; }
                    if constexpr (!inReg) d[k] = id_at(i);
                });
                static_for<0, N>([&](auto kc) { u[kc] = mul2(vx[kc], dx[kc]); });
                static_for<0, N>([&](auto kc) { ul[kc] = __shfl_up_sync(kAll, phi(u[kc]), 1); });
                static_for<0, N>([&](auto kc) {
                    constexpr int k = decltype(kc)::value, i = row[k];
                    if constexpr (inReg) gf[k] = rG[i];
                    else gf[k] = g_at(d[k]);
                });
                static_for<0, N>([&](auto kc) { sum[kc] = diff2(w[kc], wn[kc], m1); });
                static_for<0, N>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    ul[k] = bitsel(first, eul[k], ul[k]);
                    u[k] = pk(fsub(plo(u[k]), ul[k]), fsub(phi(u[k]), plo(u[k])));
                });
                static_for<0, N>([&](auto kc) { sum[kc] = add2(u[kc], sum[kc]); });
                static_for<0, N>([&](auto kc) { sum[kc] = mul2(cK, sum[kc]); });
                if constexpr (EXACT) {
                    // (P dP - K1 S) / ((1 + sigma) dP), or / (sigma dP + dP); -sP in gf
                    u64 dp[N];
                    static_for<0, N>([&](auto kc) {
                        constexpr int k = decltype(kc)::value, i = row[k];
                        if constexpr (inReg) dp[k] = rAx[i];
                        else dp[k] = dp_s(i);
                    });
                    static_for<0, N>([&](auto kc) { gf[kc] = mul2(gf[kc], dp[kc]); });
                    if (eigen) static_for<0, N>([&](auto kc) { gf[kc] = diff2(gf[kc], dp[kc], m1); });
                    static_for<0, N>([&](auto kc) { dp[kc] = mul2(P[row[kc]], dp[kc]); });
                    static_for<0, N>([&](auto kc) { sum[kc] = diff2(dp[kc], sum[kc], m1); });
                    quotients<N>(sum, gf, rp, ldsf(sb + kOffTop));
                    static_for<0, N>([&](auto kc) { P[row[kc]] = sum[kc]; });
                    return;
                }
                static_for<0, N>([&](auto kc) { P[row[kc]] = fma2(sum[kc], rp[kc], P[row[kc]]); });
                static_for<0, N>([&](auto kc) { P[row[kc]] = mul2(P[row[kc]], gf[kc]); });
            };
        };
        // rows 1 .. R-1 need no ghost value
        u64 wc = mul2(VY[1], y_at(Idx<1>{}));
        const u64 w1 = wc;
        static_for<0, (R + 2) / 4>([&](auto jc) {
            constexpr int j = 4 * decltype(jc)::value + 1, N = R - j < 4 ? R - j : 4;
            const float4 e = ldsf4(edge + 4 * (j - 1));
            const float e4[4] = {e.x, e.y, e.z, e.w};
            u64 vx[N], w[N], wn[N];
            float eul[N];
            static_for<0, N>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                vx[k] = VX[j + k];
                eul[k] = e4[k];
                wn[k] = mul2(VY[j + k + 1], y_at(Idx<j + k + 1>{}));
                w[k] = k ? wn[k ? k - 1 : 0] : wc;
            });
            wc = wn[N - 1];
            using I0 = Idx<j>;
            using I1 = Idx<j + 1>;
            using I2 = Idx<j + 2>;
            using I3 = Idx<j + 3>;
            if constexpr (N == 4) pblock(I0{}, I1{}, I2{}, I3{})(vx, w, wn, eul);
            else if constexpr (N == 3) pblock(I0{}, I1{}, I2{})(vx, w, wn, eul);
            else if constexpr (N == 2) pblock(I0{}, I1{})(vx, w, wn, eul);
            else pblock(I0{})(vx, w, wn, eul);
        });
        if (waits && m > 0) {
            const uint32_t par = (phase >> p) & 1u;
            phase ^= 1u << p;
            if (!mbar_wait_parity_bounded(bar + p, par, limit)) sfail[p] = 1;
        }
        // ---- the last row and the row above, from the ghost rows
        {
            const u64 gb = lds64(gB + p * 256);
            const ulonglong2 gt = lds128(gT + p * 512);
            float ul0 = 0.0f;
            if (lane == 0 && t > 0)
                ul0 = fmul(ldsf(gT + p * 512 - kGhostBytes + 31 * 16 + 4), ldsf(rec - (X.nrow + 2) * kRecBytes + 31 * 16 + 12));
            const u64 vx[2] = {VX[R], gt.x};
            const u64 w[2] = {wc, mul2(gt.y, y_at(Idx<0>{}))};
            const u64 wn[2] = {mul2(gb, y_at(Idx<R + 1>{})), w1};
            const float eul[2] = {ldsf(edge + 4 * (R - 1)), ul0};
            pblock(Idx<R>{}, Idx<0>{})(vx, w, wn, eul);
        }
        if (lane == 0) {
            auto pe = [&](int i) { return plo(P[i < R ? i : R - 1]); };
            static_for<0, (R + 1) / 4>([&](auto jc) {
                constexpr int j = 4 * decltype(jc)::value + 2;
                stsf4(edge + 4 * (kEdgeP + j - 2), pe(j), pe(j + 1), pe(j + 2), pe(j + 3));
            });
            sts64(edge + 4 * (kEdgeP + kMaxRows), pk(plo(P[1]), plo(P[R])));
        }
        if (lis_warp) {
            float pv = 0.0f;
            static_for<1, R + 1>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                if (i == lis_i) pv = (lis_x & 1) ? phi(P[i]) : plo(P[i]);
            });
            if (x0 == (lis_x & ~1)) store_trace(rs, trace + m, pv);
        }
        if (exc_warp) {
            float pv = 0.0f;
            static_for<1, R + 1>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                if (i == exc_y - r0 + 1) pv = (exc_x & 1) ? phi(P[i]) : plo(P[i]);
            });
            if (x0 == (exc_x & ~1)) word[m & 1] = tagged(m, pv);
        }
        if (nwx > 1) group_sync(1 + g, 32 * nwx);
        if (polls && !poll_tagged(ring + (m & (kExeRing - 1)), m, limit, &exe)) sfail[p] = 1;
        // ---- V' of the rows `rows`, whose P' right of the tile are pe: straight-line
        // code but for the block of rows with wall or source terms
        auto vblock = [&](auto... ic) {
            constexpr int N = sizeof...(ic);
            constexpr int row[N] = {decltype(ic)::value...};
            constexpr uint32_t mask = ((1u << decltype(ic)::value) | ...);
            return [&, row](const float* pe) {
                unsigned d[N];
                float prx[N];
                u64 ax[N], ay[N], dx[N], dy[N];
                static_for<0, N>([&](auto kc) {
                    if constexpr (!inReg) d[kc] = id_at(row[kc]);
                });
                static_for<0, N>([&](auto kc) { prx[kc] = __shfl_down_sync(kAll, plo(P[row[kc]]), 1); });
                if constexpr (!EXACT) static_for<0, N>([&](auto kc) {
                    constexpr int k = decltype(kc)::value, i = row[k];
                    if constexpr (inReg) {
                        ax[k] = rAx[i];
                        ay[k] = rAy[i];
                    } else {
                        const ulonglong2 al = al_at(d[k]);
                        ax[k] = al.x;
                        ay[k] = al.y;
                    }
                });
                static_for<0, N>([&](auto kc) { dy[kc] = diff2(P[row[kc] - 1], P[row[kc]], m1); });
                static_for<0, N>([&](auto kc) { dy[kc] = mul2(bc, dy[kc]); });
                static_for<0, N>([&](auto kc) {
                    constexpr int k = decltype(kc)::value, i = row[k];
                    prx[k] = bitsel(last, pe[k], prx[k]);
                    dx[k] = pk(fsub(phi(P[i]), plo(P[i])), fsub(prx[k], phi(P[i])));
                });
                static_for<0, N>([&](auto kc) { dx[kc] = mul2(bc, dx[kc]); });
                static_for<0, N>([&](auto kc) { VY[row[kc]] = diff2(VY[row[kc]], dy[kc], m1); });
                static_for<0, N>([&](auto kc) { VX[row[kc]] = diff2(VX[row[kc]], dx[kc], m1); });
                if constexpr (EXACT) {
                    if (!(dvm & mask)) return;
                    if constexpr (inReg) static_for<0, N>([&](auto kc) { d[kc] = id_at(row[kc]); });
                    if (gnm & mask) {
                        // mB V - ..., the source's and the wall's terms, in the reference's order
                        static_for<0, N>([&](auto kc) {
                            constexpr int k = decltype(kc)::value, i = row[k];
                            const ulonglong2 mx = tab_at(d[k], 3), my = tab_at(d[k], 5);
                            VX[i] = mul2(VX[i], mx.x);
                            VY[i] = mul2(VY[i], my.x);
                            if (srcm) {
                                const ulonglong2 w = tab_at(d[k], 7);
                                const u64 ee = pk(exe, exe);
                                VX[i] = diff2(VX[i], mul2(mul2(ee, w.x), mx.y), m1);
                                VY[i] = diff2(VY[i], mul2(mul2(ee, w.y), my.y), m1);
                            }
                            const ulonglong2 bx = tab_at(d[k], 4), by = tab_at(d[k], 6);
                            const u64 px = fma2(bx.x, P[i], mul2(bx.y, pk(phi(P[i]), prx[k])));
                            const u64 py = fma2(by.x, P[i], mul2(by.y, P[i - 1]));
                            VX[i] = diff2(VX[i], mul2(mx.y, mul2(px, zz)), m1);
                            VY[i] = diff2(VY[i], mul2(my.y, mul2(py, zz)), m1);
                        });
                    }
                    u64 num[N], nden[N], rec1[N];
                    static_for<0, N>([&](auto kc) {
                        const ulonglong2 v = tab_at(d[kc], 1);
                        num[kc] = VX[row[kc]];
                        nden[kc] = v.x;
                        rec1[kc] = v.y;
                    });
                    quotients<N>(num, nden, rec1, ldsf(sb + kOffTop));
                    static_for<0, N>([&](auto kc) {
                        const ulonglong2 v = tab_at(d[kc], 2);
                        VX[row[kc]] = num[kc];
                        num[kc] = VY[row[kc]];
                        nden[kc] = v.x;
                        rec1[kc] = v.y;
                    });
                    quotients<N>(num, nden, rec1, ldsf(sb + kOffTop));
                    static_for<0, N>([&](auto kc) { VY[row[kc]] = num[kc]; });
                    return;
                }
                static_for<0, N>([&](auto kc) { VY[row[kc]] = mul2(VY[row[kc]], ay[kc]); });
                static_for<0, N>([&](auto kc) { VX[row[kc]] = mul2(VX[row[kc]], ax[kc]); });
                if (gnm & mask) {
                    static_for<0, N>([&](auto kc) {
                        constexpr int k = decltype(kc)::value, i = row[k];
                        if constexpr (inReg) d[k] = id_at(i);
                        const ulonglong2 zx = zx_at(d[k]), zy = zy_at(d[k]);
                        VX[i] = fma2(zx.y, pk(phi(P[i]), prx[k]), fma2(zx.x, P[i], VX[i]));
                        VY[i] = fma2(zy.y, P[i - 1], fma2(zy.x, P[i], VY[i]));
                    });
                    if (srcm) {
                        static_for<0, N>([&](auto kc) {
                            constexpr int k = decltype(kc)::value, i = row[k];
                            VX[i] = fma2(ce_at(d[k]), pk(exe, exe), VX[i]);
                        });
                    }
                }
            };
        };
        // the rows the neighbours wait for first
        {
            const u64 e = lds64(edge + 4 * (kEdgeFloats + kEdgeP + kMaxRows));
            const float pe[2] = {plo(e), phi(e)};
            if constexpr (R > 1) vblock(Idx<1>{}, Idx<R>{})(pe);
            else vblock(Idx<1>{})(pe);
        }
        if (!bottom) sts128(gT + brow + q * 512, VX[R], VY[R]);
        if (!top) sts64(gT - lane * 8 - brow + kGhostB + q * 256, VY[1]);
        if (m + 1 < nsteps) {
            if (rem_dn) {
                st_async_pair(dnT_a + 512u * q, VX[R], dn_bar + 8u * q);
                st_async_pair(dnT_a + 512u * q + 8u, VY[R], dn_bar + 8u * q);
            }
            if (rem_up) st_async_pair(upB_a + 256u * q, VY[1], up_bar + 8u * q);
            // one thread arrives on the barrier of the next step's ghosts
            if (threadIdx.x == 0 && expect) mbar_expect_tx(bar + q, expect);
        }
        static_for<0, (R + 1) / 4>([&](auto jc) {
            constexpr int j = 4 * decltype(jc)::value + 2;
            const float4 e = ldsf4(edge + 4 * (kEdgeFloats + kEdgeP + j - 2));
            const float pe[4] = {e.x, e.y, e.z, e.w};
            using I0 = Idx<j>;
            using I1 = Idx<j + 1>;
            using I2 = Idx<j + 2>;
            using I3 = Idx<j + 3>;
            if constexpr (j + 3 < R) vblock(I0{}, I1{}, I2{}, I3{})(pe);
            else if constexpr (j + 2 < R) vblock(I0{}, I1{}, I2{})(pe);
            else if constexpr (j + 1 < R) vblock(I0{}, I1{})(pe);
            else if constexpr (j < R) vblock(I0{})(pe);
        });
        // ---- Vx dX of the tile's last column, for the next step of the tile to the right
        if (lane == 31) {
            float ue[(R + 3) / 4 * 4];
            static_for<1, R + 1>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                ue[i - 1] = fmul(phi(VX[i]), phi(x_at(ic)));
            });
            static_for<R, (R + 3) / 4 * 4>([&](auto ic) { ue[decltype(ic)::value] = 0.0f; });
            static_for<0, (R + 3) / 4>([&](auto jc) {
                constexpr int j = 4 * decltype(jc)::value;
                stsf4(edge + 4 * (kEdgeFloats + j), ue[j], ue[j + 1], ue[j + 2], ue[j + 3]);
            });
        }
        if constexpr (HIST) {
            if (x0 < pitch) {
                static_for<1, R + 1>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    float* o = hist + (i - 1) * pitch;
                    *reinterpret_cast<u64*>(o) = P[i];
                    *reinterpret_cast<u64*>(o + pl) = VX[i];
                    *reinterpret_cast<u64*>(o + 2 * pl) = VY[i];
                });
            }
            hist += 3 * pl;
        }
        step_sync(32 * X.nw);
        // a wait that ran out in this step: every warp sees it after this barrier
        if (sfail[p]) {
            if (threadIdx.x == 0) sfail[2] = min(m + 1, nsteps - 1);      // exchanges sent, see drain_exchange
            break;
        }
    }

    // ---- the state of step n0 + nsteps back to its parity set
    if (sfail[0] | sfail[1]) return;
    const int pe = (par0 + nsteps) & 1;
    float* __restrict__ oP = T->P[0] + pe * pl;
    int ra = r0 - 1;                   // opaque: the row addresses are not kept in registers through the loop
    asm volatile("" : "+r"(ra));
    static_for<1, R + 1>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        float* o = oP + (int64_t)(ra + i) * pitch + x0;
        if (in0) { o[0] = plo(P[i]); o[2 * pl] = plo(VX[i]); o[4 * pl] = plo(VY[i]); }
        if (in1) { o[1] = phi(P[i]); o[2 * pl + 1] = phi(VX[i]); o[4 * pl + 1] = phi(VY[i]); }
    });
}

// The step loop of the warp's group height.
template <int R, bool HIST, bool EXACT, bool TMM>
__device__ __forceinline__ void run_rows(int rows, const TileCtx& X) {
    if constexpr (R <= kMaxRows) {
        if (rows == R) run_tile<R, HIST, EXACT, TMM>(X);
        else run_rows<R + 1, HIST, EXACT, TMM>(rows, X);
    }
}

// A warp without a tile takes part in the CTA barriers only.
__device__ __forceinline__ void run_idle(const TileCtx& X) {
    volatile int* sfail = reinterpret_cast<volatile int*>(X.sm + kOffFail);
    const int par0 = (int)(X.rs->step & 1);
    for (int m = 0; m < X.nsteps; ++m) {
        step_sync(32 * X.nw);
        if (sfail[(par0 + m) & 1]) break;
    }
}

// The two-mass model, in a warp of its own beside the tile warps of the CTA
// that holds the excitation cell: the excitation value of step m + 1 from the
// P' of step m there; then the part of the next model step that depends on the
// state alone.  Every lane evaluates the model (the same values), state and
// prepared step in registers, and lane j sends to CTA j's ring.
template <class S, class Prep, class Finish>
__device__ __forceinline__ void two_mass_loop(const TileCtx& X, S* state, double* th, Prep&& prepare, Finish&& finish) {
    const TubeDev* __restrict__ T = X.T;
    const volatile u64* word = reinterpret_cast<const volatile u64*>(X.sm + kOffWord);
    const int lane = threadIdx.x & 31, nsteps = X.nsteps;
    const int par0 = (int)(X.rs->step & 1);
    const uint32_t limit = first_wait_limit(X.rs);
    cg::cluster_group cluster = cg::this_cluster();
    volatile u64* ring = lane < X.C ? reinterpret_cast<volatile u64*>(cluster.map_shared_rank(X.sm + kOffRing, lane)) : nullptr;
    S s = state[par0];
    auto prep = prepare(s);
    float p1 = T->P[0][par0 * T->plane + (int64_t)T->exc_y * T->pitch + T->exc_x];
    for (int m = 0;; ++m) {
        const float e = finish(prep, s, p1);
        if (ring) ring[m & (kExeRing - 1)] = tagged(m, e);
        if (th) {
            if (lane == 0) tmm_to_hist(s, th);
            th += 6;
        }
        if (m + 1 == nsteps) break;
        prep = prepare(s);
        // the tile warps gave up, and report it
        if (!__all_sync(0xffffffffu, poll_tagged(word + (m & 1), m, limit, &p1))) return;
    }
    if (lane == 0) state[(par0 + nsteps) & 1] = s;
}

__device__ __noinline__ void run_two_mass(const TileCtx& X, bool hist) {
    const TubeDev* __restrict__ T = X.T;
    double* th = hist ? T->tmm_hist + 6 * (X.rs->step + 1 - X.rs->run_start) : nullptr;
    if (T->flags & TUBE_TMM64)
        two_mass_loop(X, T->tmm64, th, [&](const TmmState64& s) { return tmm_prepare64(T->tmmd, T->tmmx, s); },
                      [](const TmmPrep64& o, TmmState64& s, float p) { return tmm_finish64(o, s, p); });
    else
        two_mass_loop(X, T->tmm, th, [&](const TmmState& s) { return tmm_prepare(T->tmmc, s); },
                      [](const TmmPrep& o, TmmState& s, float p) { return tmm_finish(o, s, p); });
}

// Waits until every byte the neighbour CTAs have sent to this one has landed,
// so that it can leave: after a wait ran out, stores may still be under way.
// Called by one thread once no CTA of the cluster sends any more.  own, up,
// dn: the exchanges this CTA and its neighbours made (each arrived once on the
// barrier of its parity here with `expect` bytes, and sent from_up or from_dn
// bytes there).  A barrier with E arrivals and R bytes landed has the tx-count
// E expect - R, its phases end where that is 0, and E or E - 1 of them have
// ended (an arrival follows the wait for the phase before it).  With T the
// bytes sent, E expect - T is taken off and a guard of 1 added, which leaves
// the count at 1 + T - R > 0: no phase ends from here on, so whether the
// last one has can be tested; if so, one more arrival opens the next phase's
// end.  Without the guard that phase ends when R = T.  Bounded like every wait.
__device__ __noinline__ void drain_exchange(uint64_t* bar, int par0, int expect, int from_up, int from_dn, int own,
                                            int up, int dn) {
    for (int p = 0; p < 2; ++p) {
        auto count = [&](int sent) { return (sent + (((par0 + 1) & 1) == p)) / 2; };    // of parity p
        const int E = count(own);
        const int more = from_up * count(up) + from_dn * count(dn) - E * expect + 1;
        if (more > 0) mbar_tx_more(bar + p, (uint32_t)more);
        if (more < 0) mbar_tx_less(bar + p, (uint32_t)-more);
        const bool ended = E == 0 || mbar_test(bar + p, (uint32_t)(E - 1) & 1u);
        if (ended) mbar_arrive(bar + p);
        mbar_tx_less(bar + p, 1);
        const uint32_t phase = (uint32_t)(ended ? E : E - 1) & 1u;
        for (int i = 0; i < kDrainPolls && !mbar_test(bar + p, phase); ++i) __nanosleep(100);
    }
}

// The end of a launch.  It finds the little it needs again, so that nothing
// but the kernel's parameters lives through the step loop for it (inlined and
// with the kernel's variables, it took registers from the loop: one uniform
// tube 0.86 us a step instead of 0.81, five tubes 12.9 ms instead of 12.3).
__device__ __noinline__ void leave_cluster(const TubeDev* __restrict__ tubes, RunState* __restrict__ rs,
                                           const int* __restrict__ order, int nsteps, unsigned char* sm) {
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), k = (int)cluster.block_rank(), tid = threadIdx.x;
    const int* f = reinterpret_cast<const int*>(sm + kOffFail);
    int* sent = reinterpret_cast<int*>(sm + kOffSent);
    __syncthreads();
    if (f[0] | f[1]) {
        if (tid == 0) atomicExch(&rs->error, VS_ERR_TIMEOUT);
        if (tid < C) cluster.map_shared_rank(sent, tid)[k] = f[2];
    }
    // no CTA exits while another may store into it: without a failure every
    // store has been waited for by the receiver's last step
    cluster.sync();
    bool failed = false;
    for (int i = 0; i < C; ++i) failed = failed || sent[i] < nsteps;
    if (tid != 0 || !failed) return;
    const int lanes = ((tubes[order[blockIdx.y]].W - 2) / kTileCols + 1) * 32;
    auto exchanges = [&](int i) { return i < 0 || i >= C ? 0 : min(sent[i], nsteps - 1); };
    const int from_up = k > 0 ? 16 * lanes : 0, from_dn = k + 1 < C ? 8 * lanes : 0;
    if (from_up + from_dn > 0)
        drain_exchange(reinterpret_cast<uint64_t*>(sm + kOffBar), (int)(rs->step & 1), from_up + from_dn, from_up, from_dn,
                       exchanges(k), exchanges(k - 1), exchanges(k + 1));
}

template <bool HIST, bool EXACT, bool TMM>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
resident_kernel(const TubeDev* __restrict__ tubes, RunState* __restrict__ rs,
                const int* __restrict__ order, int nsteps, int nw) {
    extern __shared__ __align__(128) unsigned char res_smem[];
    constexpr int kOffGhost = off_ghost(EXACT), kRecBytes = rec_bytes(EXACT), kRecD = rec_desc(EXACT);
    cg::cluster_group cluster = cg::this_cluster();
    TileCtx X;
    X.C = (int)cluster.num_blocks();
    X.k = (int)cluster.block_rank();
    X.tube = order[blockIdx.y];
    // no address is formed from an index outside the batch; the whole cluster
    // reads the same one, so it leaves together
    if ((unsigned)X.tube >= gridDim.y) {
        if (threadIdx.x == 0) atomicExch(&rs->error, VS_ERR_CUDA);
        return;
    }
    X.T = tubes + X.tube;
    X.rs = rs;
    X.sm = res_smem;
    X.nsteps = nsteps;
    const TubeDev* __restrict__ T = X.T;
    const int H = T->H, W = T->W, pitch = T->pitch;
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5;
    X.nw = nw;
    X.tmm = TMM && (T->flags & TUBE_TMM) != 0;
    const int NR = H - 2;
    const int ra = 1 + (int)(((int64_t)X.k * NR) / X.C), rb = 1 + (int)(((int64_t)(X.k + 1) * NR) / X.C);
    const int nrow = rb - ra;
    X.nrow = nrow;
    X.nwx = (W - 2) / kTileCols + 1;                 // columns 0 .. W-2
    X.ng = nw / X.nwx;
    X.nwy = min(X.ng, nrow);
    X.L = res_layout(X.nwx, X.ng, nrow, EXACT);
    const int lanes = X.nwx * 32;

    // ---- maps, descriptors and tables into shared memory; ghost rows of the first step
    const int64_t pl = T->plane;
    {
        const float* __restrict__ dP = T->dP;
        uint32_t* hash = reinterpret_cast<uint32_t*>(res_smem + kOffGhost);
        int* count = reinterpret_cast<int*>(res_smem + kOffFail) + 2;
        for (int e = tid; e < kHashSlots; e += nthr) hash[e] = 0xffffffffu;
        if (tid == 0) {
            *count = 0;
            *reinterpret_cast<float*>(res_smem + kOffTop) = 0.0f;
            *reinterpret_cast<float2*>(res_smem + kOffM1) = make_float2(-1.0f, -1.0f);
        }
        __syncthreads();
        auto start = [](uint32_t key) { return (key * 2654435761u >> 16) & (kHashSlots - 1); };
        for (int e = tid; e < (nrow + 2) * lanes; e += nthr) {
            const int j = e / lanes, l = e - j * lanes;
            const int r = ra - 1 + j, x = 2 * l;
            const bool row_in = r >= 1 && r <= H - 2;
            float rc[2] = {0.0f, 0.0f}, dp[2] = {0.0f, 0.0f}, dx[2] = {0.0f, 0.0f}, dy[2] = {0.0f, 0.0f};
            uint32_t d = 0;
            for (int h = 0; h < 2; ++h) {
                const int c = x + h;
                if (c > W - 1) continue;
                const int64_t o = (int64_t)r * pitch + c;
                dx[h] = dP[pl + o];
                dy[h] = dP[2 * pl + o];
                if (row_in && c >= 1 && c <= W - 2) {
                    const uint32_t id = T->desc[o];
                    d |= id << (8 * h);
                    dp[h] = dP[o];
                    if constexpr (EXACT) {
                        const float4 a = T->desc_a[id];
                        const float den = pressure_den(a.x, dp[h], (T->flags & TUBE_EIGEN) != 0);
                        if (!(__float_as_uint(a.w) & EXD_PZERO)) rc[h] = fdiv(1.0f, den);
                        if (!plain_den(den)) *reinterpret_cast<float*>(res_smem + kOffTop) = INFINITY;
                    } else {
                        rc[h] = rcp_approx(dp[h]);
                    }
                }
            }
            unsigned char* row = res_smem + X.L.rec + ((l >> 5) * (nrow + 2) + j) * kRecBytes;
            *reinterpret_cast<float4*>(row + (l & 31) * 16) = make_float4(rc[0], rc[1], dx[0], dx[1]);
            *reinterpret_cast<float2*>(row + kRecY + (l & 31) * 8) = make_float2(dy[0], dy[1]);
            if constexpr (EXACT) *reinterpret_cast<float2*>(row + kRecP + (l & 31) * 8) = make_float2(dp[0], dp[1]);
            *reinterpret_cast<uint16_t*>(row + kRecD + (l & 31) * 2) = (uint16_t)d;
            // the descriptor pair into the hash table (at most kMaxPairs distinct ones)
            uint32_t s = start(d);
            for (int i = 0; i < kHashSlots; ++i) {
                const uint32_t old = atomicCAS(hash + s, 0xffffffffu, d);
                if (old == 0xffffffffu || old == d) break;
                s = (s + 1) & (kHashSlots - 1);
            }
        }
        __syncthreads();
        // an id and the packed factors of each pair
        for (int e = tid; e < kHashSlots; e += nthr) {
            const uint32_t d = hash[e];
            if (d == 0xffffffffu) continue;
            const int id = atomicAdd(count, 1);
            if (id >= kMaxPairs) continue;
            hash[e] = d | (uint32_t)id << 16;
            const float4 a0 = T->desc_a[d & 0xff], a1 = T->desc_a[d >> 8];
            const float4 b0 = T->desc_b[d & 0xff], b1 = T->desc_b[d >> 8];
            float4* tab = reinterpret_cast<float4*>(res_smem + kOffTab) + id;
            if constexpr (EXACT) {
                const uint32_t f0 = __float_as_uint(a0.w), f1 = __float_as_uint(a1.w);
                const bool z = T->zinv != 0.0f;
                auto mb = [](uint32_t f) { return (f & EXD_MB) ? 1.0f : 0.0f; };
                auto wa = [z](uint32_t f) {
                    return z && (f & EXD_WALL) && (f & EXD_WALL_PC) ? ((f & EXD_NOUT1) ? 1.0f : 0.707106f) : 0.0f;
                };
                auto wb = [z](uint32_t f) { return z && (f & EXD_WALL) && !(f & EXD_WALL_PC) ? -1.0f : 0.0f; };
                const uint32_t g0 = f0 >> EXD_Y_SHIFT, g1 = f1 >> EXD_Y_SHIFT;
                if (!plain_den(a0.y) || !plain_den(a1.y) || !plain_den(a0.z) || !plain_den(a1.z))
                    *reinterpret_cast<float*>(res_smem + kOffTop) = INFINITY;
                tab[0] = make_float4(-a0.x, -a1.x, 0.0f, 0.0f);
                tab[kMaxPairs] = make_float4(-a0.y, -a1.y, fdiv(1.0f, a0.y), fdiv(1.0f, a1.y));
                tab[2 * kMaxPairs] = make_float4(-a0.z, -a1.z, fdiv(1.0f, a0.z), fdiv(1.0f, a1.z));
                tab[3 * kMaxPairs] = make_float4(mb(f0), mb(f1), -b0.x, -b1.x);
                tab[4 * kMaxPairs] = make_float4(wa(f0), wa(f1), wb(f0), wb(f1));
                tab[5 * kMaxPairs] = make_float4(mb(g0), mb(g1), -b0.z, -b1.z);
                tab[6 * kMaxPairs] = make_float4(wa(g0), wa(g1), wb(g0), wb(g1));
                tab[7 * kMaxPairs] = make_float4((f0 & EXD_SRC) ? b0.y : 0.0f, (f1 & EXD_SRC) ? b1.y : 0.0f,
                                                 (g0 & EXD_SRC) ? b0.w : 0.0f, (g1 & EXD_SRC) ? b1.w : 0.0f);
                continue;
            }
            tab[0] = make_float4(a0.z, a1.z, a0.w, a1.w);
            tab[kMaxPairs] = make_float4(a0.x, a1.x, a0.y, a1.y);
            tab[2 * kMaxPairs] = make_float4(b0.x, b1.x, -b0.y, -b1.y);
            tab[3 * kMaxPairs] = make_float4(b0.z, b1.z, -b0.w, -b1.w);
        }
        __syncthreads();
        for (int e = tid; e < (nrow + 2) * lanes; e += nthr) {
            const int j = e / lanes, l = e - j * lanes;
            uint16_t* d = reinterpret_cast<uint16_t*>(res_smem + X.L.rec + ((l >> 5) * (nrow + 2) + j) * kRecBytes + kRecD) +
                          (l & 31);
            uint32_t s = start(*d);
            for (int i = 0; i < kHashSlots && (hash[s] & 0xffffu) != *d; ++i) s = (s + 1) & (kHashSlots - 1);
            *d = (uint16_t)((hash[s] >> 16) * 16);
        }
        __syncthreads();                             // the hash becomes ghost rows
        const int64_t n0 = rs->step;
        const int par0 = (int)(n0 & 1);
        const float* __restrict__ gP = T->P[0] + par0 * pl;
        for (int e = tid; e < X.nwy * lanes; e += nthr) {
            const int g = e / lanes, l = e - g * lanes;
            const int a = ra + (int)(((int64_t)g * nrow) / X.nwy), b = ra + (int)(((int64_t)(g + 1) * nrow) / X.nwy);
            float v[6];
            for (int h = 0; h < 2; ++h) {
                const int c = 2 * l + h;
                const bool in = c >= 1 && c <= W - 2;
                const int64_t o = (int64_t)(a - 1) * pitch + c, ob = (int64_t)b * pitch + c;
                v[h] = in ? gP[2 * pl + o] : 0.0f;
                v[2 + h] = in ? gP[4 * pl + o] : 0.0f;
                v[4 + h] = in ? gP[4 * pl + ob] : 0.0f;
            }
            unsigned char* gt = res_smem + kOffGhost + (g * X.nwx + (l >> 5)) * kGhostBytes;
            unsigned char* gb = res_smem + kOffGhost + ((g == X.nwy - 1 ? X.ng : g) * X.nwx + (l >> 5)) * kGhostBytes;
            *reinterpret_cast<float4*>(gt + par0 * 512 + (l & 31) * 16) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float2*>(gb + kGhostB + par0 * 256 + (l & 31) * 8) = make_float2(v[4], v[5]);
            // the other parity: ring rows, which no step writes, stay zero
            *reinterpret_cast<float4*>(gt + (par0 ^ 1) * 512 + (l & 31) * 16) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            *reinterpret_cast<float2*>(gb + kGhostB + (par0 ^ 1) * 256 + (l & 31) * 8) = make_float2(0.0f, 0.0f);
        }
        float* edge = reinterpret_cast<float*>(res_smem + X.L.edge);
        for (int e = tid; e < X.ng * (X.nwx + 1) * kMaxRows; e += nthr) {
            // Vx dX of the column left of the tile, for the first step
            const int i = e % kMaxRows, t = e / kMaxRows % (X.nwx + 1), g = e / (kMaxRows * (X.nwx + 1));
            float u = 0.0f;
            if (g < X.nwy && t >= 1 && t < X.nwx) {
                const int r = ra + (int)(((int64_t)g * nrow) / X.nwy) + i, c = kTileCols * t - 1;
                if (r <= H - 2) u = fmul(gP[2 * pl + (int64_t)r * pitch + c], dP[pl + (int64_t)r * pitch + c]);
            }
            float* at = edge + (g * (X.nwx + 1) + t) * kEdgeFloats;
            at[i] = u;
            at[kEdgeP + i] = 0.0f;
            if (i < kEdgeFloats - 2 * kMaxRows) at[2 * kMaxRows + i] = 0.0f;
        }
        if (tid == 0) {
            uint64_t* bar = reinterpret_cast<uint64_t*>(res_smem + kOffBar);
            mbar_init(bar, 1);
            mbar_init(bar + 1, 1);
            mbar_fence_init();
            int* f = reinterpret_cast<int*>(res_smem + kOffFail);
            f[0] = f[1] = 0;
            for (int i = 0; i < kMaxCtas; ++i) reinterpret_cast<int*>(res_smem + kOffSent)[i] = nsteps;
            u64* w = reinterpret_cast<u64*>(res_smem + kOffRing);
            for (int i = 0; i < kExeRing + 2; ++i) w[i] = ~0ull << 32;      // tag: no step
        }
    }
    __syncthreads();
    cluster.sync();                                  // every CTA's barriers are initialised

    X.g = warp / X.nwx;
    X.t = warp - X.g * X.nwx;
    if (TMM && warp == nw) {
        if (X.tmm && T->exc_y >= ra && T->exc_y < rb) run_two_mass(X, HIST);
        __syncwarp();
    } else if (X.g < X.nwy) {
        const int a = (int)(((int64_t)X.g * nrow) / X.nwy), b = (int)(((int64_t)(X.g + 1) * nrow) / X.nwy);
        X.j0 = a;
        X.r0 = ra + a;
        run_rows<1, HIST, EXACT, TMM>(b - a, X);
    } else {
        run_idle(X);
    }
    leave_cluster(tubes, rs, order, nsteps, res_smem);
}

}  // namespace
}  // namespace vsb
