// sip_tile.cuh -- the SIP solver on 2x2x2 tiles, in FP32 (mixed form) and FP64
// (plain form).
//
// A grid of even dimensions is cut into tiles of 2x2x2 cells, stored tile after
// tile in the order of the hyperplanes I+J+K of the tile lattice, the 8 values of
// a tile (k fastest) in one 32-byte (64-byte) line.  A sweep walks the tile
// hyperplanes, one thread a tile, one CTA a grid: 34 steps for 24^3 cells where
// the cell hyperplanes take 70, and a step's 8 points pass their values in
// registers.  Between tiles only faces travel: a thread reads the three facing
// quads of its predecessors from shared memory and leaves its own three, six
// 16-byte accesses for 8 points (cell by cell it takes 32 of 4 bytes, and the
// index of each).  In shared memory a face of tile (I, J, K) of hyperplane t sits
// in slot (I+1)(NJ+1) + (J+1), which no other tile of that hyperplane shares, so
// the predecessors are at the constant offsets -(NJ+1), -1 and 0 of the plane
// before.  The arithmetic of a point and its order are those of the cell sweeps
// (sip_hyperplane_mod.F90:450-569), so the results are the same bits.
//
// The sweeps are bound by the chain of their steps (few grids) and by the
// issue of their loads (many); all global loads of a step are 32 bytes wide and
// are issued kD steps ahead.
#pragma once

#include <algorithm>
#include <vector>

#include "internal.h"

namespace mg {

// Tables of one grid shape (device pointers)
struct TileShape {
    int ni, nj, nk;                 // cells
    int NI, NJ, NK, NT, ntile;      // tiles; tile hyperplanes; tiles in all
    int npp, fs;                    // cells of a grid's array; length of a face array
    int maxt;                       // tiles of the largest hyperplane
    int w, slots;                   // NJ + 1; (NI + 1)(NJ + 1)
    int nside;                      // ghost tiles on the three low (or high) faces
    const int* tst;                 // [NT+1] first tile of each hyperplane
    const unsigned short* slot;     // [ntile, padded to 4] slot of the tile
    // [ntile][2]: tiles at i-1, i+1, j-1, j+1 | k-1, k+1, cell (io, jo, ko) of the
    // tile's first cell (10 bits each), 0; a negative entry -1-t is tile t of the
    // grid across that face
    const int4* nbr;
    // ghost tiles on the low and high faces by extended hyperplane: gst[s][p+1] ..
    // gst[s][p+2] those of hyperplane p (-1 .. NT); {slot | axis << 16, tile of the
    // grid across the face}
    const int* gst[2];
    const int2* gent[2];
    const int* tpos;                // [NT][NI] tile (I, J) of hyperplane T is tpos[T*NI+I] + J
    const int* cell;                // [npp] natural local index of each position
    const int* plane;               // [npp] its position in the cell hyperplane order
    const int* facepos;             // [6][fs] position of the boundary cell of each face index
};

// position of a cell
__host__ __device__ inline int tile_pos(const int* tpos, int NI, int io, int jo, int ko) {
    const int I = io >> 1, J = jo >> 1, K = ko >> 1;
    return ((tpos[(I + J + K) * NI + I] + J) << 3) | ((io & 1) << 2) | ((jo & 1) << 1) | (ko & 1);
}

struct TileDev {
    bool ok = false;
    TileShape s{};
    std::vector<void*> mem;
};

namespace {

template <typename T>
struct alignas(16) Vec4 {
    T v[4];
};
template <typename T>
struct Vec8 {
    T v[8];
};

// 8 values of a tile.  kNc: through the read-only path (nothing in the launch
// writes them); p: a predicate, without a branch (a load inside a branch is
// waited for where the branch ends).
__device__ __forceinline__ void ld8(bool p, const float* a, Vec8<float>& r) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n"
        " @q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}"
        : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3]), "+f"(r.v[4]), "+f"(r.v[5]),
          "+f"(r.v[6]), "+f"(r.v[7])
        : "l"(a), "r"((int)p));
}
__device__ __forceinline__ void ld8(bool p, const double* a, Vec8<double>& r) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n"
        " @q ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%8];\n"
        " @q ld.global.nc.v4.f64 {%4, %5, %6, %7}, [%8 + 32];\n}"
        : "+d"(r.v[0]), "+d"(r.v[1]), "+d"(r.v[2]), "+d"(r.v[3]), "+d"(r.v[4]), "+d"(r.v[5]),
          "+d"(r.v[6]), "+d"(r.v[7])
        : "l"(a), "r"((int)p));
}
// values this CTA writes later in the same launch
__device__ __forceinline__ void ld8_rw(bool p, const float* a, Vec8<float>& r) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n"
        " @q ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}"
        : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3]), "+f"(r.v[4]), "+f"(r.v[5]),
          "+f"(r.v[6]), "+f"(r.v[7])
        : "l"(a), "r"((int)p)
        : "memory");
}
__device__ __forceinline__ void ld8_rw(bool p, const double* a, Vec8<double>& r) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n"
        " @q ld.global.v4.f64 {%0, %1, %2, %3}, [%8];\n"
        " @q ld.global.v4.f64 {%4, %5, %6, %7}, [%8 + 32];\n}"
        : "+d"(r.v[0]), "+d"(r.v[1]), "+d"(r.v[2]), "+d"(r.v[3]), "+d"(r.v[4]), "+d"(r.v[5]),
          "+d"(r.v[6]), "+d"(r.v[7])
        : "l"(a), "r"((int)p)
        : "memory");
}
__device__ __forceinline__ void st8(float* a, const Vec8<float>& r) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a), "f"(r.v[0]),
                 "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]), "f"(r.v[7])
                 : "memory");
}
__device__ __forceinline__ void st8(double* a, const Vec8<double>& r) {
    asm volatile(
        "st.global.v4.f64 [%0], {%1, %2, %3, %4};\n st.global.v4.f64 [%0 + 32], {%5, %6, %7, %8};" ::"l"(a),
        "d"(r.v[0]), "d"(r.v[1]), "d"(r.v[2]), "d"(r.v[3]), "d"(r.v[4]), "d"(r.v[5]), "d"(r.v[6]), "d"(r.v[7])
        : "memory");
}

// a += r: one writer per value, so the reduction (round to nearest) is the plain
// sum without a load
__device__ __forceinline__ void add8(float* a, const Vec8<float>& r) {
    asm volatile(
        "red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n red.global.add.v4.f32 [%0 + 16], {%5, %6, %7, %8};" ::"l"(a),
        "f"(r.v[0]), "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]), "f"(r.v[7])
        : "memory");
}
__device__ __forceinline__ void add8(double* a, const Vec8<double>& r) {
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicAdd(a + i, r.v[i]);
}

// The quad of a tile that faces its neighbour: on axis 0, 1, 2 the cells with
// offset hi along that axis; in the order of the other two offsets.
template <int kAxis, int kHi, typename T>
__device__ __forceinline__ Vec4<T> quad(const Vec8<T>& r) {
    if constexpr (kAxis == 0) return Vec4<T>{r.v[4 * kHi], r.v[4 * kHi + 1], r.v[4 * kHi + 2], r.v[4 * kHi + 3]};
    else if constexpr (kAxis == 1)
        return Vec4<T>{r.v[2 * kHi], r.v[2 * kHi + 1], r.v[4 + 2 * kHi], r.v[5 + 2 * kHi]};
    else return Vec4<T>{r.v[kHi], r.v[2 + kHi], r.v[4 + kHi], r.v[6 + kHi]};
}

// a product that is rounded before anything is added to it
__device__ __forceinline__ float mul_rounded(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rounded(double a, double b) { return __dmul_rn(a, b); }

template <typename T>
struct TileArgs {
    TileShape s;
    const int* glist;               // the grids of this launch (null: all)
    const int* fnbr;                // [ngrid][6] neighbour grids (0-based, -1 none)
    const int* gcls;                // coefficient class of each grid
    T* R;                           // sweeps: forward (rhs + lap) lpr -> res, backward res; pre-pass: out
    const T* G;                     // sweeps: the res the ghosts come from (null: zeros)
    T* H;                           // hilf
    const T* RHS;
    const T* PG;                    // [ngrid][6][fs] hilf ghosts of PAR faces (null: zero)
    const T* CF;                    // sweeps: per class three coefficients (i, j, k), npp each
    const T* LPR;                   // per class lpr
    const T* LAP;                   // per class [aw | ae | as | an | ab | at | ap], npp each
    const T* UNI;                   // [ncls][8] operator coefficients of uniform classes
    const int* ctl;                 // [0] converged: nothing to do
    int cfcls, lprcls;              // values between the classes of CF and of LPR
    int hzero;                      // hilf is zero
    int rev;                        // walk the grids in reverse block order
};

constexpr int kTilePad = 8;         // empty hyperplanes past the last in the table of starts

// Shared memory of a sweep: [tst] [gst] [ghost entries] [ghost quads] [2][3][slots] quads
struct TileLayout {
    unsigned gst, gent, gval, face, bytes;
};
template <typename T>
__host__ __device__ inline TileLayout tile_layout(const TileShape& s) {
    auto up = [](unsigned v) { return (v + 31u) & ~31u; };
    TileLayout l;
    unsigned o = (s.NT + 1 + kTilePad) * 4;
    l.gst = o; o = up(o + (s.NT + 3) * 4);
    l.gent = o; o = up(o + s.nside * 4);
    l.gval = o; o = up(o + s.nside * (unsigned)sizeof(Vec4<T>));
    l.face = o; o += 6 * s.slots * (unsigned)sizeof(Vec4<T>);
    l.bytes = o;
    return l;
}

// A tile's loads of one step
template <typename T>
struct TileSet {
    int tile, x;                    // tile (-1: none) and slot
    Vec8<T> c[3], v;
};

// The predecessor recurrence of a tile's 8 cells (see k_tile_sweep)
template <bool kFwd, typename T>
__device__ __forceinline__ Vec8<T> tile_solve(const Vec8<T>& v, const Vec8<T>& ci, const Vec8<T>& cj,
                                              const Vec8<T>& ck, const Vec4<T>& fi, const Vec4<T>& fj,
                                              const Vec4<T>& fk) {
    Vec8<T> r;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int i = kFwd ? m : 7 - m;          // di dj dk
        const int di = i >> 2, dj = (i >> 1) & 1, dk = i & 1;
        constexpr int in = kFwd ? 1 : 0;         // offset of a cell whose predecessor is in the tile
        const T rk = dk == in ? r.v[i ^ 1] : fk.v[2 * di + dj];
        const T rj = dj == in ? r.v[i ^ 2] : fj.v[2 * di + dk];
        const T ri = di == in ? r.v[i ^ 4] : fi.v[2 * dj + dk];
        r.v[i] = v.v[i] - ck.v[i] * rk - cj.v[i] * rj - ci.v[i] * ri;
    }
    return r;
}

// One sweep of a grid.  kFwd: tile hyperplanes in order, res = v - lb res(k-1) -
// ls res(j-1) - lw res(i-1) (sip_hyperplane_mod.F90:491-495); else in reverse,
// res = res - ut res(k+1) - un res(j+1) - ue res(i+1), hilf += res (:546-547,
// 559-567; kHz: hilf = res).  The last warp stages the ghosts.
template <typename T, bool kFwd, bool kHz, int kD, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_tile_sweep(const __grid_constant__ TileArgs<T> a) {
    if (a.ctl[0]) return;
    extern __shared__ __align__(32) unsigned char tsm[];
    const TileShape& s = a.s;
    const int b = a.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const int g = a.glist ? a.glist[b] : b;
    const int tid = threadIdx.x, ncomp = blockDim.x - 32, NT = s.NT;
    const int W = kFwd ? -s.w : s.w, one = kFwd ? -1 : 1, back = kFwd ? 0 : s.w + 1;
    const TileLayout l = tile_layout<T>(s);
    int *tst = reinterpret_cast<int*>(tsm), *gst = reinterpret_cast<int*>(tsm + l.gst),
        *gent = reinterpret_cast<int*>(tsm + l.gent);
    Vec4<T>*gval = reinterpret_cast<Vec4<T>*>(tsm + l.gval), *face = reinterpret_cast<Vec4<T>*>(tsm + l.face);
    const long long base = (long long)g * s.npp;
    const T* C = a.CF + (long long)a.gcls[g] * a.cfcls;
    T* R = a.R + base;
    T* H = a.H + base;
    constexpr int side = kFwd ? 0 : 1;
    for (int q = tid; q < NT + 1 + kTilePad; q += blockDim.x) {
        // step t covers tiles tst[t] .. tst[t+1] forward, tst[t+1] .. tst[t] backward
        tst[q] = q <= NT ? s.tst[kFwd ? q : NT - q] : (kFwd ? s.ntile : 0);
        if (q < NT + 3) gst[q] = s.gst[side][q];
    }
    // the ghosts: the facing quads of the grids across
    {
        const int* fn = a.fnbr + 6 * g;
        int nb[3];
        for (int d = 0; d < 3; ++d) nb[d] = a.G ? fn[2 * d + side] : -1;
        constexpr int kU = 4;
        for (int q0 = tid; q0 < s.nside; q0 += kU * blockDim.x) {
            int2 e[kU];
            Vec8<T> v[kU];
#pragma unroll
            for (int i = 0; i < kU; ++i) {
                e[i] = make_int2(0, 0);
                if (q0 + i * (int)blockDim.x < s.nside) e[i] = __ldg(s.gent[side] + q0 + i * blockDim.x);
            }
#pragma unroll
            for (int i = 0; i < kU; ++i) {
                const int d = e[i].x >> 16, n = d == 0 ? nb[0] : (d == 1 ? nb[1] : nb[2]);
#pragma unroll
                for (int m = 0; m < 8; ++m) v[i].v[m] = T(0);
                ld8(n >= 0, a.G + ((long long)max(n, 0) * s.npp + 8 * e[i].y), v[i]);
            }
#pragma unroll
            for (int i = 0; i < kU; ++i) {
                const int q = q0 + i * (int)blockDim.x;
                if (q >= s.nside) break;
                const int d = e[i].x >> 16;
                constexpr int hi = kFwd ? 1 : 0;   // the neighbour's high cells are my low ghosts
                gval[q] = d == 0 ? quad<0, hi>(v[i]) : (d == 1 ? quad<1, hi>(v[i]) : quad<2, hi>(v[i]));
                gent[q] = e[i].x;
            }
        }
    }
    __syncthreads();
    if (tid >= ncomp) {
        // the ghosts of step t (-1: those before the first) into their faces
        auto ghosts = [&](int t) {
            Vec4<T>* f = face + (t & 1) * 3 * s.slots;
            const int p = kFwd ? t : NT - 1 - t;
            const int g0 = gst[p + 1], n = gst[p + 2];
            for (int q = g0 + (tid & 31); q < n; q += 32)
                f[(gent[q] >> 16) * s.slots + (gent[q] & 0xffff)] = gval[q];
        };
        ghosts(-1);
        __syncthreads();
        for (int t = 0; t < NT; ++t) {
            ghosts(t);
            __syncthreads();
        }
        return;
    }
    using Set = TileSet<T>;
    auto fetch = [&](int t, Set& q) {
        const int ta = tst[t], tb = tst[t + 1];
        const int tile = (kFwd ? ta : tb) + tid;
        const bool on = tile < (kFwd ? tb : ta);
        q.tile = on ? tile : -1;
        const int p = 8 * tile;
        if (on) q.x = (int)__ldg(s.slot + tile) - back;
        ld8(on, C + p, q.c[0]);
        ld8(on, C + s.npp + p, q.c[1]);
        ld8(on, C + 2 * s.npp + p, q.c[2]);
        if constexpr (kFwd) ld8_rw(on, R + p, q.v);
        else ld8(on, R + p, q.v);
    };
    Set q[kD];
#pragma unroll
    for (int d = 0; d < kD; ++d) fetch(d, q[d]);
    __syncthreads();
    auto step = [&](int t, Set& c) {
        if (c.tile >= 0) {
            Vec4<T>* cur = face + (t & 1) * 3 * s.slots + c.x;
            const Vec4<T>* prv = face + ((t + 1) & 1) * 3 * s.slots + c.x;
            const Vec4<T> fi = prv[W], fj = prv[s.slots + one], fk = prv[2 * s.slots];
            const Vec8<T> r = tile_solve<kFwd>(c.v, c.c[0], c.c[1], c.c[2], fi, fj, fk);
            constexpr int out = kFwd ? 1 : 0;
            cur[0] = quad<0, out>(r);
            cur[s.slots] = quad<1, out>(r);
            cur[2 * s.slots] = quad<2, out>(r);
            if constexpr (kFwd) {
                st8(R + 8 * c.tile, r);
            } else if constexpr (kHz) {
                st8(H + 8 * c.tile, r);
            } else {
                add8(H + 8 * c.tile, r);
            }
        }
        fetch(t + kD, c);
        __syncthreads();
    };
    for (int t = 0; t < NT; t += kD) {
#pragma unroll
        for (int d = 0; d < kD; ++d) {
            if (t + d >= NT) break;
            step(t + d, q[d]);
        }
    }
}

// The sweep of few grids (at most two on an SM), where nothing else runs while a
// step waits: the time is the chain of one warp's instructions through all
// steps.  Two sets of warps take the steps in turn, so that the chain of a step is
// three face loads, the recurrence and three face stores; a set stores its results
// and issues its next loads while the other set works.  The tables, the ghosts and
// the first tiles are loaded at once.
template <typename T, bool kFwd, bool kHz, int kD, int kThreads>
__global__ void __launch_bounds__(kThreads) k_tile_sweep_few(const __grid_constant__ TileArgs<T> a) {
    extern __shared__ __align__(32) unsigned char tsm[];
    const TileShape& s = a.s;
    const int b = a.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const int g = a.glist ? a.glist[b] : b;
    const int tid = threadIdx.x, ncomp = (blockDim.x - 32) / 2, NT = s.NT;
    const int set = tid >= ncomp ? 1 : 0, lane = tid - set * ncomp;   // (the last warp: neither)
    const int W = kFwd ? -s.w : s.w, one = kFwd ? -1 : 1, back = kFwd ? 0 : s.w + 1;
    const TileLayout l = tile_layout<T>(s);
    int *tst = reinterpret_cast<int*>(tsm), *gst = reinterpret_cast<int*>(tsm + l.gst),
        *gent = reinterpret_cast<int*>(tsm + l.gent);
    Vec4<T>*gval = reinterpret_cast<Vec4<T>*>(tsm + l.gval), *face = reinterpret_cast<Vec4<T>*>(tsm + l.face);
    const long long base = (long long)g * s.npp;
    const T* C = a.CF + (long long)a.gcls[g] * a.cfcls;
    T* R = a.R + base;
    T* H = a.H + base;
    constexpr int side = kFwd ? 0 : 1;
    const int converged = __ldg(a.ctl);
    TileSet<T> q[kD];
    // the loads of a step whose tiles are t0 .. t1
    auto fetch = [&](TileSet<T>& c, int t0, int t1) {
        const int tile = t0 + lane;
        const bool on = tile < t1;
        c.tile = on ? tile : -1;
        const int p = 8 * tile;
        if (on) c.x = (int)__ldg(s.slot + tile) - back;
        ld8(on, C + p, c.c[0]);
        ld8(on, C + s.npp + p, c.c[1]);
        ld8(on, C + 2 * s.npp + p, c.c[2]);
        if constexpr (kFwd) ld8_rw(on, R + p, c.v);
        else ld8(on, R + p, c.v);
    };
    // first tile of step t's hyperplane and the one past its last, from global memory
    auto first = [&](int t) { return t < NT ? __ldg(s.tst + (kFwd ? t : NT - 1 - t)) : 0; };
    auto past = [&](int t) { return t < NT ? __ldg(s.tst + (kFwd ? t + 1 : NT - t)) : 0; };
    constexpr int kU = 4;
    int nb[3];
    for (int d = 0; d < 3; ++d) nb[d] = a.G ? a.fnbr[6 * g + 2 * d + side] : -1;
    int2 e[kU];
#pragma unroll
    for (int i = 0; i < kU; ++i)
        e[i] = __ldg(s.gent[side] + min(tid + i * (int)blockDim.x, s.nside - 1));
    if (tid < 2 * ncomp)
#pragma unroll
        for (int d = 0; d < kD; ++d) fetch(q[d], first(set + 2 * d), past(set + 2 * d));
    for (int t = tid; t < NT + 1 + kTilePad; t += blockDim.x) {
        // step t covers tiles tst[t] .. tst[t+1] forward, tst[t+1] .. tst[t] backward
        tst[t] = t <= NT ? s.tst[kFwd ? t : NT - t] : (kFwd ? s.ntile : 0);
        if (t < NT + 3) gst[t] = s.gst[side][t];
    }
    // the ghosts: the facing quads of the grids across
    for (int q0 = tid; q0 < s.nside; q0 += kU * blockDim.x) {
        Vec8<T> v[kU];
#pragma unroll
        for (int i = 0; i < kU; ++i) {
            const int d = e[i].x >> 16, n = d == 0 ? nb[0] : (d == 1 ? nb[1] : nb[2]);
#pragma unroll
            for (int m = 0; m < 8; ++m) v[i].v[m] = T(0);
            ld8(n >= 0, a.G + ((long long)max(n, 0) * s.npp + 8 * e[i].y), v[i]);
        }
#pragma unroll
        for (int i = 0; i < kU; ++i) {
            const int m = q0 + i * (int)blockDim.x;
            if (m < s.nside) {
                const int d = e[i].x >> 16;
                constexpr int hi = kFwd ? 1 : 0;   // the neighbour's high cells are my low ghosts
                gval[m] = d == 0 ? quad<0, hi>(v[i]) : (d == 1 ? quad<1, hi>(v[i]) : quad<2, hi>(v[i]));
                gent[m] = e[i].x;
            }
            e[i] = __ldg(s.gent[side] + min(m + kU * (int)blockDim.x, s.nside - 1));
        }
    }
    if (converged) return;
    __syncthreads();
    const int steps = (NT + 1) & ~1;
    if (tid >= 2 * ncomp) {
        // the ghosts of step t (-1: those before the first) into their faces
        auto ghosts = [&](int t) {
            Vec4<T>* f = face + (t & 1) * 3 * s.slots;
            const int p = kFwd ? t : NT - 1 - t;
            const int g0 = gst[p + 1], n = gst[p + 2];
            for (int m = g0 + (tid & 31); m < n; m += 32)
                f[(gent[m] >> 16) * s.slots + (gent[m] & 0xffff)] = gval[m];
        };
        ghosts(-1);
        __syncthreads();
        for (int t = 0; t < steps; ++t) {
            if (t < NT) ghosts(t);
            __syncthreads();
        }
        return;
    }
    __syncthreads();
    // step t of this set
    auto work = [&](int t, TileSet<T>& c, Vec8<T>& r) {
        if (c.tile >= 0) {
            Vec4<T>* cur = face + (t & 1) * 3 * s.slots + c.x;
            const Vec4<T>* prv = face + ((t + 1) & 1) * 3 * s.slots + c.x;
            r = tile_solve<kFwd>(c.v, c.c[0], c.c[1], c.c[2], prv[W], prv[s.slots + one], prv[2 * s.slots]);
            constexpr int out = kFwd ? 1 : 0;
            cur[0] = quad<0, out>(r);
            cur[s.slots] = quad<1, out>(r);
            cur[2 * s.slots] = quad<2, out>(r);
        }
    };
    // while the other set works: the results of step t to memory, the loads of the
    // step kD turns on
    auto rest = [&](int t, TileSet<T>& c, const Vec8<T>& r) {
        if (c.tile >= 0) {
            if constexpr (kFwd) st8(R + 8 * c.tile, r);
            else if constexpr (kHz) st8(H + 8 * c.tile, r);
            else add8(H + 8 * c.tile, r);
        }
        const int n = min(t + 2 * kD, NT + 1);
        const int ta = tst[n], tb = tst[n + 1];
        fetch(c, kFwd ? ta : tb, kFwd ? tb : ta);
    };
    Vec8<T> r;
    if (set) __syncthreads();   // step 0
    for (int t = set; t < steps; t += 2 * kD) {
#pragma unroll
        for (int d = 0; d < kD; ++d) {
            const int m = t + 2 * d;
            if (m >= steps) break;
            work(m, q[d], r);
            __syncthreads();
            rest(m, q[d], r);
            if (m + 1 < steps) __syncthreads();   // the other set's step
        }
    }
}

// hilf of a tile and the facing quads around it (f = -i, +i, -j, +j, -k, +k)
template <typename T>
struct TileHalo {
    Vec8<T> h;
    Vec4<T> f[6];
};

// The quad across face kF of a tile: of tile nb of the same grid (>= 0), of tile
// -1-nb of the grid across that face, of the grid's own ghost plane, or zero.
template <int kF, typename T>
__device__ __forceinline__ Vec4<T> tile_face(const TileArgs<T>& a, int g, int nb, int org) {
    const TileShape& s = a.s;
    constexpr int ax = kF / 2, hi = kF % 2 == 0 ? 1 : 0;
    int n = g;
    if (nb < 0) {
        n = a.fnbr[6 * g + kF];
        nb = -1 - nb;
        if (n < 0) {
            Vec4<T> z{T(0), T(0), T(0), T(0)};
            if (a.PG) {
                const T* P = a.PG + ((long long)g * 6 + kF) * s.fs;
                const int io = org & 1023, jo = (org >> 10) & 1023, ko = org >> 20;
                const int st = ax == 2 ? s.nj : s.nk;   // stride of the second index
                const int q = ax == 0 ? ko + jo * s.nk : (ax == 1 ? ko + io * s.nk : jo + io * s.nj);
                // a quad runs over (dj, dk), (di, dk), (di, dj)
                z = Vec4<T>{P[q], P[q + 1], P[q + st], P[q + st + 1]};
            }
            return z;
        }
    }
    const T* p = a.H + ((long long)n * s.npp + 8 * nb);
    if constexpr (ax == 0) {
        const Vec4<T> v = *reinterpret_cast<const Vec4<T>*>(p + 4 * hi);
        return v;
    } else {
        Vec8<T> v;
        ld8(true, p, v);
        return quad<ax, hi>(v);
    }
}

template <typename T>
__device__ __forceinline__ void tile_halo(const TileArgs<T>& a, int g, int tile, TileHalo<T>& o) {
    const int4 n0 = __ldg(a.s.nbr + 2 * tile), n1 = __ldg(a.s.nbr + 2 * tile + 1);
    ld8(true, a.H + ((long long)g * a.s.npp + 8 * tile), o.h);
    o.f[0] = tile_face<0>(a, g, n0.x, n1.z);
    o.f[1] = tile_face<1>(a, g, n0.y, n1.z);
    o.f[2] = tile_face<2>(a, g, n0.z, n1.z);
    o.f[3] = tile_face<3>(a, g, n0.w, n1.z);
    o.f[4] = tile_face<4>(a, g, n1.x, n1.z);
    o.f[5] = tile_face<5>(a, g, n1.y, n1.z);
}

// the neighbours of cell i (di dj dk) of a tile: i-1, i+1, j-1, j+1, k-1, k+1
template <typename T>
__device__ __forceinline__ void tile_nbrs(const TileHalo<T>& o, int i, T n[6]) {
    const int di = i >> 2, dj = (i >> 1) & 1, dk = i & 1;
    n[0] = di ? o.h.v[i ^ 4] : o.f[0].v[2 * dj + dk];
    n[1] = di ? o.f[1].v[2 * dj + dk] : o.h.v[i ^ 4];
    n[2] = dj ? o.h.v[i ^ 2] : o.f[2].v[2 * di + dk];
    n[3] = dj ? o.f[3].v[2 * di + dk] : o.h.v[i ^ 2];
    n[4] = dk ? o.h.v[i ^ 1] : o.f[4].v[2 * di + dj];
    n[5] = dk ? o.f[5].v[2 * di + dj] : o.h.v[i ^ 1];
}

// The part of sipiter1 outside the recurrence, (rhs + laplacephi(hilf)) lpr
// (sip_hyperplane_mod.F90:491, laplacephi_mod.F90:153-160), one thread a tile;
// the tiles of a grid in gridDim.x CTAs.  kUni: one value of each operator
// coefficient a class.  Of the first two products one rounds by itself and the
// other is contracted with it: the first in kOrder 0, the second in kOrder 1, as the
// compiler does it in the packed and in the table-driven cell pre-pass.
template <typename T, bool kUni, int kOrder, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_tile_pre(const __grid_constant__ TileArgs<T> a) {
    if (a.ctl[0]) return;
    const TileShape& s = a.s;
    const int b = a.rev ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
    const int g = a.glist ? a.glist[b] : b;
    const int cls = a.gcls[g];
    const long long base = (long long)g * s.npp;
    const T* LPR = a.LPR + (long long)cls * a.lprcls;
    const T* LAP = a.LAP + (long long)cls * 7 * s.npp;
    T u[7];
#pragma unroll
    for (int f = 0; f < 7; ++f) u[f] = kUni ? a.UNI[8 * cls + f] : T(0);
    for (int tile = blockIdx.x * kThreads + threadIdx.x; tile < s.ntile; tile += gridDim.x * kThreads) {
        const int p = 8 * tile;
        Vec8<T> rh, lp, out;
        ld8(true, a.RHS + base + p, rh);
        ld8(true, LPR + p, lp);
        if (a.hzero) {
#pragma unroll
            for (int i = 0; i < 8; ++i) out.v[i] = mul_rounded(rh.v[i] + T(0), lp.v[i]);
        } else {
            TileHalo<T> o;
            tile_halo(a, g, tile, o);
            Vec8<T> c[kUni ? 1 : 7];
            if constexpr (!kUni)
#pragma unroll
                for (int f = 0; f < 7; ++f) ld8(true, LAP + f * s.npp + p, c[f]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                T n[6];
                tile_nbrs(o, i, n);
                T w[7];
#pragma unroll
                for (int f = 0; f < 7; ++f) w[f] = kUni ? u[f] : c[kUni ? 0 : f].v[i];
                T lap = mul_rounded(-w[kOrder], n[kOrder]);
                lap = lap - w[1 - kOrder] * n[1 - kOrder] - w[2] * n[2] - w[3] * n[3] - w[4] * n[4] -
                      w[5] * n[5] - w[6] * o.h.v[i];
                out.v[i] = mul_rounded(rh.v[i] + lap, lp.v[i]);
            }
        }
        st8(a.R + base + p, out);
    }
}

// ---- host tables ------------------------------------------------------------
template <typename V>
int tile_up(Ctx* c, TileDev& d, const V** p, const std::vector<V>& h) {
    V* m = nullptr;
    MG_CUDA(cudaMalloc(&m, h.size() * sizeof(V)));
    d.mem.push_back(m);
    MG_CUDA(copy_on(c->stream, m, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice));
    *p = m;
    return 0;
}

// Tables of a grid of ni x nj x nk cells with kk, jj points a line (ghosts
// included).  d.ok stays false for odd dimensions, hyperplanes of more than 512
// tiles and shapes beyond the 10-bit cells or 16-bit slots.
inline int tile_init(Ctx* c, int ni, int nj, int nk, TileDev& d) {
    TileShape& s = d.s;
    s.ni = ni; s.nj = nj; s.nk = nk;
    if (ni % 2 || nj % 2 || nk % 2 || ni > 1023 || nj > 1023 || nk > 1023) return 0;
    const int NI = s.NI = ni / 2, NJ = s.NJ = nj / 2, NK = s.NK = nk / 2;
    s.NT = NI + NJ + NK - 2;
    s.ntile = NI * NJ * NK;
    s.npp = 8 * s.ntile;
    s.fs = (std::max(nj * nk, std::max(ni * nk, ni * nj)) + 3) & ~3;
    s.w = NJ + 1;
    s.slots = (NI + 1) * (NJ + 1);
    s.nside = NI * NJ + NI * NK + NJ * NK;
    std::vector<int> tst(s.NT + 1, 0), tpos((size_t)s.NT * NI, 0);
    std::vector<unsigned short> slot((s.ntile + 3) & ~3, 0);
    std::vector<int> ti(s.ntile), tj(s.ntile), tk(s.ntile);
    for (int t = 0, p = 0; t < s.NT; ++t) {
        for (int I = 0; I < NI; ++I) {
            const int jlo = std::max(0, t - I - (NK - 1)), jhi = std::min(NJ - 1, t - I);
            tpos[(size_t)t * NI + I] = p - jlo;
            for (int J = jlo; J <= jhi; ++J, ++p) {
                ti[p] = I; tj[p] = J; tk[p] = t - I - J;
                slot[p] = (unsigned short)((I + 1) * s.w + J + 1);
            }
        }
        tst[t + 1] = p;
        s.maxt = std::max(s.maxt, p - tst[t]);
    }
    if (tst[s.NT] != s.ntile || s.maxt > 512 || s.slots > 0xffff) return 0;
    auto tile = [&](int I, int J, int K) { return tpos[(size_t)(I + J + K) * NI + I] + J; };
    std::vector<int4> nbr((size_t)2 * s.ntile);
    for (int p = 0; p < s.ntile; ++p) {
        const int I = ti[p], J = tj[p], K = tk[p];
        const int im = I > 0 ? tile(I - 1, J, K) : -1 - tile(NI - 1, J, K);
        const int ip = I < NI - 1 ? tile(I + 1, J, K) : -1 - tile(0, J, K);
        const int jm = J > 0 ? tile(I, J - 1, K) : -1 - tile(I, NJ - 1, K);
        const int jp = J < NJ - 1 ? tile(I, J + 1, K) : -1 - tile(I, 0, K);
        const int km = K > 0 ? tile(I, J, K - 1) : -1 - tile(I, J, NK - 1);
        const int kp = K < NK - 1 ? tile(I, J, K + 1) : -1 - tile(I, J, 0);
        nbr[2 * p] = make_int4(im, ip, jm, jp);
        nbr[2 * p + 1] = make_int4(km, kp, (2 * I) | (2 * J) << 10 | (2 * K) << 20, 0);
    }
    for (int sd = 0; sd < 2; ++sd) {
        struct Entry {
            int p;
            int2 e;
        };
        std::vector<Entry> gs;
        // low: coordinate -1, the slot (I+1)w + J+1; high: coordinate N, the slot
        // I w + J the backward sweep uses
        auto add = [&](int ax, int I, int J, int K, int t) {
            const int x = sd == 0 ? (I + 1) * s.w + J + 1 : I * s.w + J;
            gs.push_back(Entry{I + J + K, make_int2(x | (ax << 16), t)});
        };
        for (int J = 0; J < NJ; ++J)
            for (int K = 0; K < NK; ++K)
                add(0, sd ? NI : -1, J, K, sd ? tile(0, J, K) : tile(NI - 1, J, K));
        for (int I = 0; I < NI; ++I)
            for (int K = 0; K < NK; ++K)
                add(1, I, sd ? NJ : -1, K, sd ? tile(I, 0, K) : tile(I, NJ - 1, K));
        for (int I = 0; I < NI; ++I)
            for (int J = 0; J < NJ; ++J)
                add(2, I, J, sd ? NK : -1, sd ? tile(I, J, 0) : tile(I, J, NK - 1));
        std::stable_sort(gs.begin(), gs.end(), [](const Entry& a, const Entry& b) {
            if (a.p != b.p) return a.p < b.p;
            if ((a.e.x >> 16) != (b.e.x >> 16)) return (a.e.x >> 16) < (b.e.x >> 16);
            return a.e.y < b.e.y;
        });
        std::vector<int> gst(s.NT + 3, 0);
        std::vector<int2> gent;
        size_t q = 0;
        for (int p = -1; p <= s.NT; ++p) {
            gst[p + 1] = (int)q;
            for (; q < gs.size() && gs[q].p == p; ++q) gent.push_back(gs[q].e);
        }
        gst[s.NT + 2] = (int)q;
        if ((int)q != s.nside) return 0;
        if (int rc = tile_up(c, d, &s.gst[sd], gst)) return rc;
        if (int rc = tile_up(c, d, &s.gent[sd], gent)) return rc;
    }
    // cells: natural local index and place in the cell hyperplane order
    const int kk = nk + 4, jj = nj + 4;
    std::vector<int> cell(s.npp), plane(s.npp);
    {
        int q = 0;
        for (int m = 0; m < ni + nj + nk - 2; ++m)
            for (int io = 0; io < ni; ++io) {
                const int jlo = std::max(0, m - io - (nk - 1)), jhi = std::min(nj - 1, m - io);
                for (int jo = jlo; jo <= jhi; ++jo, ++q) {
                    const int ko = m - io - jo, p = tile_pos(tpos.data(), NI, io, jo, ko);
                    cell[p] = (ko + 2) + (jo + 2) * kk + (io + 2) * kk * jj;
                    plane[p] = q;
                }
            }
    }
    std::vector<int> facepos((size_t)6 * s.fs, -1);
    auto pos = [&](int io, int jo, int ko) { return tile_pos(tpos.data(), NI, io, jo, ko); };
    for (int jo = 0; jo < nj; ++jo)
        for (int ko = 0; ko < nk; ++ko) {
            facepos[0 * s.fs + ko + jo * nk] = pos(0, jo, ko);
            facepos[1 * s.fs + ko + jo * nk] = pos(ni - 1, jo, ko);
        }
    for (int io = 0; io < ni; ++io)
        for (int ko = 0; ko < nk; ++ko) {
            facepos[2 * s.fs + ko + io * nk] = pos(io, 0, ko);
            facepos[3 * s.fs + ko + io * nk] = pos(io, nj - 1, ko);
        }
    for (int io = 0; io < ni; ++io)
        for (int jo = 0; jo < nj; ++jo) {
            facepos[4 * s.fs + jo + io * nj] = pos(io, jo, 0);
            facepos[5 * s.fs + jo + io * nj] = pos(io, jo, nk - 1);
        }
    if (int rc = tile_up(c, d, &s.tst, tst)) return rc;
    if (int rc = tile_up(c, d, &s.tpos, tpos)) return rc;
    if (int rc = tile_up(c, d, &s.slot, slot)) return rc;
    if (int rc = tile_up(c, d, &s.nbr, nbr)) return rc;
    if (int rc = tile_up(c, d, &s.cell, cell)) return rc;
    if (int rc = tile_up(c, d, &s.plane, plane)) return rc;
    if (int rc = tile_up(c, d, &s.facepos, facepos)) return rc;
    d.ok = true;
    return 0;
}

inline void tile_free(TileDev& d) {
    for (void* p : d.mem) cudaFree(p);
    d = TileDev();
}

}  // namespace
}  // namespace mg
