// sip_tile.cuh -- the SIP solver on small tiles of cells, in FP32 (mixed form,
// 2x2x2) and FP64 (plain form, 1x1x2 or single cells).
//
// A grid is cut into tiles of TI x TJ x TK cells, stored tile after tile in the order of the hyperplanes I+J+K of the tile
// lattice, the values of a tile together, k fastest.  A sweep walks the tile
// hyperplanes, one thread a tile, one CTA a grid: 34 steps for 24^3 cells in tiles
// of 2x2x2 where the cell hyperplanes take 70, and the points of a tile pass their
// values in registers.  Between tiles only faces travel: a thread reads the three
// facing quads of its predecessors from shared memory and leaves its own three --
// six 16-byte accesses for 8 points (cell by cell it takes 32 of 4 bytes, and the
// index of each).  In shared memory a face of tile (I, J, K) of hyperplane t sits
// in slot (I+1)(NJ+1) + (J+1), which no other tile of that hyperplane shares, so
// the predecessors are at the constant offsets -(NJ+1), -1 and 0 of the plane
// before.  The arithmetic of a point and its order are those of the cell sweeps
// (sip_hyperplane_mod.F90:450-569), so the results are the same bits.
//
// An odd dimension leaves pads in the last tiles.  Their coefficients are zero, so a
// sweep passes through a pad what its array holds there: the backward sweep first
// writes the ghosts of that side into the pads of res, the pre-pass and the outer
// step take them for the pads of hilf, and the forward sweep has no successor that
// reads a pad.
//
// What bounds it: FP32, the chain of the steps (few grids) and the issue of the
// loads (many); all global loads of a step are issued kD steps ahead.  FP64, the
// FP64 pipe: an instruction of a warp takes it 64 clocks whatever the number of
// active lanes, so there the lanes have to be full and the four pipes of an SM
// evenly used -- 2-cell tiles (12 instructions a step, 119 tiles a step on 24^3)
// cost 52 k clocks a sweep, 2x2x2 tiles (48 a step, 51 tiles) 104 k.
#pragma once

#include <algorithm>
#include <vector>

#include "follow_on.cuh"
#include "internal.h"

namespace mg {

// Tables of one grid shape (device pointers)
struct TileShape {
    int ni, nj, nk;                 // cells
    int si, sj, sk;                 // log2 of the tile's extents (0 or 1)
    int pad;                        // axes (bit 0: i) where the last tile holds one cell and a pad
    int NI, NJ, NK, NT, ntile;      // tiles; tile hyperplanes; tiles in all
    int npp, fs;                    // cells of a grid's array; length of a face array
    int nc;                         // CTAs of a sweep (a cluster); rank I nc / NI takes the tiles of row I
    int maxt;                       // most tiles of a rank in a hyperplane
    int w, slots;                   // NJ + 1; (NI + 1)(NJ + 1)
    int nside;                      // most ghost tiles of a rank on the three low (or high) faces
    const int* tst;                 // [NT*nc+1] first tile of each hyperplane and rank
    const unsigned short* slot;     // [ntile, padded to 4] slot of the tile
    // [ntile][2]: tiles at i-1, i+1, j-1, j+1 | k-1, k+1, cell (io, jo, ko) of the
    // tile's first cell (10 bits each), 0; a negative entry -1-t is tile t of the
    // grid across that face
    const int4* nbr;
    // ghost tiles on the low and high faces by rank and extended hyperplane: of the
    // rank's, gst[s][p+1] .. gst[s][p+2] those of hyperplane p (-1 .. NT), [NT+3] the
    // rank's first ([nc][NT+4]); {slot | axis << 16, tile of the grid across the face}
    const int* gst[2];
    const int2* gent[2];
    const int* tpos;                // [NT][NI] tile (I, J) of hyperplane T is tpos[T*NI+I] + J
    const int* cell;                // [npp] natural local index of each position, -1 in pads
    const int* plane;               // [npp] its position in the cell hyperplane order, -1 in pads
};

// position of a cell
__host__ __device__ inline int tile_pos(const TileShape& s, const int* tpos, int io, int jo, int ko) {
    const int I = io >> s.si, J = jo >> s.sj, K = ko >> s.sk;
    const int di = io & s.si, dj = jo & s.sj, dk = ko & s.sk;   // (extents are 1 or 2)
    return ((tpos[(I + J + K) * s.NI + I] + J) << (s.si + s.sj + s.sk)) |
           (((di << s.sj) | dj) << s.sk | dk);
}

struct TileDev {
    bool ok = false;
    TileShape s{};
    std::vector<void*> mem;
};

namespace {

template <typename T, int N>
struct alignas(sizeof(T) * N < 16 ? sizeof(T) * N : 16) Vec {
    T v[N];
};

// The N values of a tile.  ldt: through the read-only path (tables and coefficients);
// ldt_co: values the launch before may still write when this one starts (it waits for
// them first, see follow_on); ldt_rw: values this CTA writes later in the same launch;
// p: a predicate, without a branch (a load inside a branch is waited for where the
// branch ends).
#define MG_LD(SUF, CLOB)                                                                                 \
    template <int N>                                                                                     \
    __device__ __forceinline__ void ldt##SUF(bool p, const float* a, Vec<float, N>& r) {                 \
        if constexpr (N == 8)                                                                            \
            asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n @q ld.global" MG_NC                 \
                         ".v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}"                            \
                         : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3]), "+f"(r.v[4]),         \
                           "+f"(r.v[5]), "+f"(r.v[6]), "+f"(r.v[7])                                      \
                         : "l"(a), "r"((int)p) CLOB);                                                    \
        else if constexpr (N == 2)                                                                       \
            asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.global" MG_NC                 \
                         ".v2.f32 {%0, %1}, [%2];\n}"                                                    \
                         : "+f"(r.v[0]), "+f"(r.v[1])                                                    \
                         : "l"(a), "r"((int)p) CLOB);                                                    \
        else                                                                                             \
            asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.global" MG_NC                 \
                         ".f32 %0, [%1];\n}"                                                             \
                         : "+f"(r.v[0])                                                                  \
                         : "l"(a), "r"((int)p) CLOB);                                                    \
    }                                                                                                    \
    template <int N>                                                                                     \
    __device__ __forceinline__ void ldt##SUF(bool p, const double* a, Vec<double, N>& r) {               \
        if constexpr (N == 2)                                                                            \
            asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.global" MG_NC                 \
                         ".v2.f64 {%0, %1}, [%2];\n}"                                                    \
                         : "+d"(r.v[0]), "+d"(r.v[1])                                                    \
                         : "l"(a), "r"((int)p) CLOB);                                                    \
        else                                                                                             \
            asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.global" MG_NC                 \
                         ".f64 %0, [%1];\n}"                                                             \
                         : "+d"(r.v[0])                                                                  \
                         : "l"(a), "r"((int)p) CLOB);                                                    \
    }
#define MG_NC ".nc"
MG_LD(, )
#undef MG_NC
#define MG_NC ""
MG_LD(_co, )
MG_LD(_rw, : "memory")
#undef MG_NC
#undef MG_LD

template <typename T, int N>
__device__ __forceinline__ void stt(T* a, const Vec<T, N>& r) {
    static_assert(N <= 2 || N == 8, "tile sizes");
    if constexpr (N == 8 && sizeof(T) == 4)
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a), "f"(r.v[0]),
                     "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]),
                     "f"(r.v[7])
                     : "memory");
    else
        *reinterpret_cast<Vec<T, N>*>(a) = r;
}
// a += r: one writer per value, so the reduction (round to nearest) is the plain
// sum without a load
template <typename T, int N>
__device__ __forceinline__ void addt(T* a, const Vec<T, N>& r) {
    if constexpr (N == 8 && sizeof(T) == 4) {
        asm volatile(
            "red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n"
            " red.global.add.v4.f32 [%0 + 16], {%5, %6, %7, %8};" ::"l"(a),
            "f"(r.v[0]), "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]),
            "f"(r.v[7])
            : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) atomicAdd(a + i, r.v[i]);
    }
}

// The extents of a tile, and the cells of its faces: on axis A the cells with the
// lowest or highest offset along it, in the order of the other two offsets.
template <int TI_, int TJ_, int TK_>
struct Tile {
    static constexpr int TI = TI_, TJ = TJ_, TK = TK_, N = TI * TJ * TK;
    static constexpr int FI = TJ * TK, FJ = TI * TK, FK = TI * TJ;
    template <int A>
    static constexpr int F = A == 0 ? FI : (A == 1 ? FJ : FK);
    // cell q of the face on axis A, at the high end when hi
    template <int A>
    __host__ __device__ static constexpr int cell(int q, bool hi) {
        if (A == 0) return (hi ? (TI - 1) * TJ * TK : 0) + q;
        if (A == 1) return (q / TK) * TJ * TK + (hi ? (TJ - 1) * TK : 0) + q % TK;
        return q * TK + (hi ? TK - 1 : 0);
    }
};

// (kM: the size of the result, the face's cells first)
template <class L, int A, bool kHi, typename T, int kM = L::template F<A>>
__device__ __forceinline__ Vec<T, kM> tile_part(const Vec<T, L::N>& r) {
    Vec<T, kM> o;
#pragma unroll
    for (int q = 0; q < kM; ++q) o.v[q] = q < L::template F<A> ? r.v[L::template cell<A>(q, kHi) % L::N] : T(0);
    return o;
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
    const T* AP;                    // per class the operator's diagonal
    const T* A1[6];                 // pre-pass: its other coefficients aw, ae, as, an, ab, at by coordinate
    const DevGrid* grids;
    const unsigned char* BM;        // [ngrid][npp] open couplings (null: all)
    const T* UNI;                   // [ncls][8] operator coefficients of uniform classes
    const int* ctl;                 // [0] converged: nothing to do; ranks: [1] err
    int cfcls, lprcls, apcls;       // values between the classes of CF, LPR and AP
    int* err;                       // takes stamp when a rank waited in vain
    int stamp;                      // the sweep's, not 0, another one in each launch of a solve
    int lose;                       // test switch: forward, rank 1 of every grid misses its first faces
    int rev;                        // walk the grids in reverse block order
};

constexpr int kTilePad = 8;         // empty hyperplanes past the last in the table of starts

// Shared memory of a sweep: [tst] [ends, if ranks share the hyperplanes] [gst] [ghost entries] [ghost faces] [2][3][slots]
// faces (of equal size for the three axes, so that a ghost is one copy) [faces of the
// row before the rank's, [NJ][NK]] [their mbarriers]
template <class L>
struct TileFace {   // values of the largest face
    static constexpr int M = L::FI > L::FJ ? (L::FI > L::FK ? L::FI : L::FK) : (L::FJ > L::FK ? L::FJ : L::FK);
};
struct TileLayout {
    unsigned tend, gst, gent, gval, face, bnd, mbar, bytes;
};
template <class L, typename T>
__host__ __device__ inline TileLayout tile_layout(const TileShape& s) {
    auto up = [](unsigned v) { return (v + 31u) & ~31u; };
    constexpr unsigned fb = TileFace<L>::M * sizeof(T);
    TileLayout l{};
    unsigned o = (s.NT + 1 + kTilePad) * 4;
    l.tend = o; if (s.nc > 1) o += (s.NT + 1 + kTilePad) * 4;
    l.gst = o; o = up(o + (s.NT + 3) * 4);
    l.gent = o; o = up(o + s.nside * 4);
    l.gval = o; o = up(o + s.nside * fb);
    l.face = o; o += 6 * s.slots * fb;
    if (s.nc > 1) {
        l.bnd = o; o = up(o + s.NJ * s.NK * fb);
        l.mbar = o; o += (s.NJ + s.NK - 1) * 8;
    }
    l.bytes = o;
    return l;
}

// A tile's loads of one step
template <class L, typename T>
struct TileSet {
    int tile, x;                    // tile (-1: none) and slot
    Vec<T, L::N> c[3], v;
};

// the shared memory of another CTA of the cluster
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
template <int N>
__device__ __forceinline__ void cluster_put(unsigned a, unsigned mbar, const Vec<double, N>& v) {
#pragma unroll
    for (int i = 0; i < N; ++i)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a + 8 * i),
                     "d"(v.v[i]), "r"(mbar)
                     : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// What the sweep kernels share: a CTA's grid and its tables (kRanks: its rank's part).
template <class L, typename T, bool kFwd, bool kRanks = false, bool kPad = false>
struct TileSweep {
    const TileArgs<T>& a;
    const TileShape& s;
    int g, W, one, back;
    int rank, nent, ent0;           // rank in the cluster; its ghosts and the first of them
    int t0, t1;                     // its steps
    int i0, i1;                     // its rows
    bool up, down;                  // does a rank before, after it take part?
    int *tst, *tend, *gst, *gent;
    using Face = Vec<T, TileFace<L>::M>;
    Face *gval, *face, *bnd;
    unsigned mbar, bndto, mbarto;   // its mbarriers; bnd and mbarriers of the rank after
    const T* C;
    T *R, *H;
    static constexpr int side = kFwd ? 0 : 1;

    __device__ __forceinline__ TileSweep(const TileArgs<T>& args, unsigned char* sm) : a(args), s(args.s) {
        const int nb = kRanks ? gridDim.x / s.nc : gridDim.x, b0 = kRanks ? blockIdx.x / s.nc : blockIdx.x;
        const int b = a.rev ? nb - 1 - b0 : b0;
        rank = kRanks ? blockIdx.x % s.nc : 0;
        g = a.glist ? a.glist[b] : b;
        W = kFwd ? -s.w : s.w;
        one = kFwd ? -1 : 1;
        back = kFwd ? 0 : s.w + 1;
        const TileLayout l = tile_layout<L, T>(s);
        tst = reinterpret_cast<int*>(sm);
        tend = reinterpret_cast<int*>(sm + l.tend);
        gst = reinterpret_cast<int*>(sm + l.gst);
        gent = reinterpret_cast<int*>(sm + l.gent);
        gval = reinterpret_cast<Face*>(sm + l.gval);
        face = reinterpret_cast<Face*>(sm + l.face);
        t0 = 0;
        t1 = s.NT;
        nent = s.nside;
        ent0 = 0;
        if constexpr (kRanks) {
            const int* gr = s.gst[side] + rank * (s.NT + 4);
            nent = __ldg(gr + s.NT + 2);
            ent0 = __ldg(gr + s.NT + 3);
            i0 = (rank * s.NI + s.nc - 1) / s.nc;
            i1 = ((rank + 1) * s.NI + s.nc - 1) / s.nc - 1;
            const int last = i1 + s.NJ + s.NK - 2;   // hyperplane
            t0 = kFwd ? i0 : s.NT - 1 - last;
            t1 = (kFwd ? last : s.NT - 1 - i0) + 1;
            up = kFwd ? rank > 0 : rank < s.nc - 1;
            down = kFwd ? rank < s.nc - 1 : rank > 0;
            bnd = reinterpret_cast<Face*>(sm + l.bnd);
            mbar = (unsigned)__cvta_generic_to_shared(sm + l.mbar);
            const int to = down ? (kFwd ? rank + 1 : rank - 1) : rank;
            bndto = cluster_addr(bnd, to);
            mbarto = cluster_addr(sm + l.mbar, to);
        }
        const long long base = (long long)g * s.npp;
        C = a.CF + (long long)a.gcls[g] * a.cfcls;
        R = a.R + base;
        H = a.H + base;
    }
    // step t covers tiles tst[t] .. tst[t+1] forward, tst[t+1] .. tst[t] backward
    __device__ __forceinline__ void tables() {
        for (int t = threadIdx.x; t < s.NT + 1 + kTilePad; t += blockDim.x) {
            if constexpr (kRanks) {
                const int* x = s.tst + (kFwd ? t : s.NT - 1 - t) * s.nc + rank;
                tst[t] = t < s.NT ? x[0] : 0;
                tend[t] = t < s.NT ? x[1] : 0;
            } else {
                tst[t] = t <= s.NT ? s.tst[kFwd ? t : s.NT - t] : (kFwd ? s.ntile : 0);
            }
            if (t < s.NT + 3) gst[t] = s.gst[side][rank * (s.NT + 4) + t];
        }
    }
    // the facing cells of the grids across (e0: the thread's first entries, loaded
    // by the caller)
    static constexpr int kU = 4, M = TileFace<L>::M;
    __device__ __forceinline__ void entries(int2 e[kU], int q0) {
#pragma unroll
        for (int i = 0; i < kU; ++i) e[i] = __ldg(s.gent[side] + ent0 + max(min(q0 + i * (int)blockDim.x, nent - 1), 0));
    }
    __device__ __forceinline__ void ghosts(int2 e[kU]) {
        int nb[3];
        for (int d = 0; d < 3; ++d) nb[d] = a.G ? a.fnbr[6 * g + 2 * d + side] : -1;
        for (int q0 = threadIdx.x; q0 < nent; q0 += kU * blockDim.x) {
            Vec<T, L::N> v[kU];
#pragma unroll
            for (int i = 0; i < kU; ++i) {
                const int d = e[i].x >> 16, n = d == 0 ? nb[0] : (d == 1 ? nb[1] : nb[2]);
#pragma unroll
                for (int m = 0; m < L::N; ++m) v[i].v[m] = T(0);
                // (in the launches that write pads, the arrays' other cells are read here)
                const T* src = a.G + ((long long)max(n, 0) * s.npp + L::N * (kPad ? e[i].y & 0xffff : e[i].y));
                if constexpr (kPad && !kFwd) ldt_rw(n >= 0, src, v[i]);
                else ldt_co(n >= 0, src, v[i]);
            }
#pragma unroll
            for (int i = 0; i < kU; ++i) {
                const int m = q0 + i * (int)blockDim.x;
                if (m < nent) {
                    const int d = e[i].x >> 16;
                    // the neighbour's high cells are my low ghosts
                    Face x = tile_part<L, 0, kFwd, T, M>(v[i]), y = tile_part<L, 1, kFwd, T, M>(v[i]),
                         z = tile_part<L, 2, kFwd, T, M>(v[i]);
                    if constexpr (kPad) {
                        const bool last = s.pad >> d & 1;
                        if (kFwd) {
                            // the last cells are the low ones of their tile
                            if (last) {
                                x = tile_part<L, 0, false, T, M>(v[i]);
                                y = tile_part<L, 1, false, T, M>(v[i]);
                                z = tile_part<L, 2, false, T, M>(v[i]);
                            }
                        } else if (last) {
                            // the ghosts are pads of res; nothing is behind them
                            T* r = R + L::N * (int)((unsigned)e[i].y >> 16);
#pragma unroll
                            for (int c = 0; c < M; ++c) {
                                const Face f = d == 0 ? x : (d == 1 ? y : z);
                                const int o = d == 0 ? L::template cell<0>(c, true)
                                                     : (d == 1 ? L::template cell<1>(c, true)
                                                               : L::template cell<2>(c, true));
                                r[o] = f.v[c];
                            }
#pragma unroll
                            for (int c = 0; c < M; ++c) x.v[c] = y.v[c] = z.v[c] = T(0);
                        }
                    }
                    gval[m] = d == 0 ? x : (d == 1 ? y : z);
                    gent[m] = e[i].x;
                }
            }
            entries(e, q0 + kU * (int)blockDim.x);
        }
    }
    // one warp: the ghosts of step t (-1: those before the first) into their faces
    __device__ __forceinline__ void stage(int t) {
        const int p = kFwd ? t : s.NT - 1 - t;
        Face* f = face + (t & 1) * 3 * s.slots;
        const int g0 = gst[p + 1], n = gst[p + 2];
        for (int m = g0 + (threadIdx.x & 31); m < n; m += 32)
            f[(gent[m] >> 16) * s.slots + (gent[m] & 0xffff)] = gval[m];
    }
    // The faces of the row before arrive with their own completion: one mbarrier for
    // each of the row's hyperplanes J + K, armed once for the bytes of its faces.
    __device__ __forceinline__ int row_lo(int h) const { return max(0, h - (s.NK - 1)); }
    __device__ __forceinline__ int row_hi(int h) const { return min(s.NJ - 1, h); }
    __device__ __forceinline__ void arm() {
        if (up)
            for (int h = threadIdx.x; h < s.NJ + s.NK - 1; h += blockDim.x) {
                const unsigned m = mbar + 8 * h;
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(m) : "memory");
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(m),
                             "r"((row_hi(h) - row_lo(h) + 1) * (int)sizeof(Face))
                             : "memory");
            }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // has row hyperplane h arrived?  (one warp)
    __device__ __forceinline__ bool arrived(int h) const {
        int ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
                     " selp.s32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(mbar + 8 * h)
                     : "memory");
        return __all_sync(0xffffffffu, ok);
    }
    static __device__ __forceinline__ bool expired(long long since, long long limit) {
        return __any_sync(0xffffffffu, clock64() - since > limit);
    }
    // one warp, in step t: stages the faces the rank before has put in step t.  The wait
    // for them ends after about a second: then the error flag takes the launch's stamp
    // and this rank waits no more.  Later sweeps find a stamp that is not theirs and
    // return at once; what this launch writes stops none of its own CTAs, so that of a
    // cluster all return or none.
    static constexpr long long kWait = 2000000000LL, kWaitTest = 100000000LL;   // SM clocks
    __device__ __forceinline__ void boundary(int t, bool& lost, bool lose = false) {
        if (!up) return;
        const int I = kFwd ? i0 - 1 : i1 + 1, h = (kFwd ? t : s.NT - 1 - t) - I;
        const int lo = row_lo(h), hi = row_hi(h);
        if (lo > hi) return;
        const long long since = clock64();
        while (!lost) {
            if (arrived(h) && !lose) break;
            if (expired(since, lose ? kWaitTest : kWait)) {
                lost = true;
                if ((threadIdx.x & 31) == 0) *a.err = a.stamp;
            }
        }
        Face* f = face + (t & 1) * 3 * s.slots + (kFwd ? (I + 1) * s.w + 1 : I * s.w);
        for (int J = lo + (threadIdx.x & 31); J <= hi; J += 32) f[J] = bnd[J * s.NK + h - J];
    }
    // one warp of a rank that gave up, behind the last cluster barrier: every face has been
    // put by now, and the CTA stays until they are here (or another second is over)
    __device__ __forceinline__ void drain() {
        const long long since = clock64();
        for (int h = 0; h < s.NJ + s.NK - 1; ++h)
            while (!arrived(h))
                if (expired(since, kWait)) return;
    }
    // thread lane's loads of a step whose tiles are t0 .. t1
    __device__ __forceinline__ void fetch(TileSet<L, T>& q, int lane, int t0, int t1) {
        coefs(q, lane, t0, t1);
        values(q);
    }
    __device__ __forceinline__ void coefs(TileSet<L, T>& q, int lane, int t0, int t1) {
        const int tile = t0 + lane;
        const bool on = tile < t1;
        q.tile = on ? tile : -1;
        const int p = L::N * tile;
        if (on) q.x = (int)__ldg(s.slot + tile);
        ldt(on, C + p, q.c[0]);
        ldt(on, C + s.npp + p, q.c[1]);
        ldt(on, C + 2 * s.npp + p, q.c[2]);
    }
    __device__ __forceinline__ void values(TileSet<L, T>& q) {
        const int p = L::N * q.tile;
        if constexpr (kFwd || kPad) ldt_rw(q.tile >= 0, R + p, q.v);
        else ldt_co(q.tile >= 0, R + p, q.v);
    }
    // the recurrence of a tile's cells in step t
    __device__ __forceinline__ void solve(int t, const TileSet<L, T>& q, Vec<T, L::N>& r) {
        const int x = q.x - back;
        solve_at(face + (t & 1) * 3 * s.slots + x, face + ((t + 1) & 1) * 3 * s.slots + x, q, r);
    }
    // (cur, prv: the tile's slot in the faces of the step and of the one before)
    __device__ __forceinline__ void solve_at(Face* cur, const Face* prv, const TileSet<L, T>& q, Vec<T, L::N>& r) {
        const Face fi = prv[W], fj = prv[s.slots + one], fk = prv[2 * s.slots];
#pragma unroll
        for (int m = 0; m < L::N; ++m) {
            const int i = kFwd ? m : L::N - 1 - m;
            const int di = i / (L::TJ * L::TK), dj = (i / L::TK) % L::TJ, dk = i % L::TK;
            const bool ik = kFwd ? dk > 0 : dk < L::TK - 1, ij = kFwd ? dj > 0 : dj < L::TJ - 1,
                       ii = kFwd ? di > 0 : di < L::TI - 1;
            constexpr int o = kFwd ? -1 : 1;
            const T rk = ik ? r.v[(i + o) & (L::N - 1)] : fk.v[di * L::TJ + dj];
            const T rj = ij ? r.v[(i + o * L::TK) & (L::N - 1)] : fj.v[di * L::TK + dk];
            const T ri = ii ? r.v[(i + o * L::TJ * L::TK) & (L::N - 1)] : fi.v[dj * L::TK + dk];
            r.v[i] = q.v.v[i] - q.c[2].v[i] * rk - q.c[1].v[i] * rj - q.c[0].v[i] * ri;
        }
        cur[0] = tile_part<L, 0, kFwd, T, TileFace<L>::M>(r);
        cur[s.slots] = tile_part<L, 1, kFwd, T, TileFace<L>::M>(r);
        cur[2 * s.slots] = tile_part<L, 2, kFwd, T, TileFace<L>::M>(r);
    }
    // the faces of the row the next rank starts from
    __device__ __forceinline__ void put(int t, const TileSet<L, T>& q, const Vec<T, L::N>& r) {
        const int I = kFwd ? i1 : i0, J = q.x - (I + 1) * s.w - 1;
        const int h = (kFwd ? t : s.NT - 1 - t) - I;
        if (down && J >= 0 && J < s.NJ)
            cluster_put(bndto + (J * s.NK + h - J) * (unsigned)sizeof(Face), mbarto + 8 * h,
                        tile_part<L, 0, kFwd, T, TileFace<L>::M>(r));
    }
    template <bool kHz>
    __device__ __forceinline__ void store(int tile, const Vec<T, L::N>& r) {
        if constexpr (kFwd) stt(R + L::N * tile, r);
        else if constexpr (kHz) stt(H + L::N * tile, r);
        else addt(H + L::N * tile, r);
    }
};

// One sweep of a grid.  kFwd: tile hyperplanes in order, res = v - lb res(k-1) -
// ls res(j-1) - lw res(i-1) (sip_hyperplane_mod.F90:491-495); else in reverse,
// res = res - ut res(k+1) - un res(j+1) - ue res(i+1), hilf += res (:546-547,
// 559-567; kHz: hilf = res).  The last warp stages the ghosts.
template <class L, typename T, bool kFwd, bool kHz, int kD, int kThreads, int kMinBlocks, bool kPad = false>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_tile_sweep(const __grid_constant__ TileArgs<T> a) {
    extern __shared__ __align__(32) unsigned char tsm[];
    TileSweep<L, T, kFwd, false, kPad> w(a, tsm);
    const int tid = threadIdx.x, ncomp = blockDim.x - 32, NT = a.s.NT;
    int2 e[w.kU];
    w.entries(e, tid);
    w.tables();
    follow_on();
    if (flag_at(a.ctl)) return;
    w.ghosts(e);
    __syncthreads();
    if (tid >= ncomp) {
        w.stage(-1);
        __syncthreads();
        for (int t = 0; t < NT; ++t) {
            w.stage(t);
            __syncthreads();
        }
        return;
    }
    // kD steps of loads in flight: a step issues the loads of kD steps on before it
    // computes, into the set the step before has left.  FP64: the warps take the chunks
    // of a hyperplane in turn, one on each step, so that the chunks that every
    // hyperplane has do not stay on one of the SM's four FP64 pipes.
    TileSet<L, T> q[kD + 1];
    int lane = tid;
    auto fetch = [&](int t, TileSet<L, T>& c) {
        const int ta = w.tst[t], tb = w.tst[t + 1];
        w.fetch(c, lane, kFwd ? ta : tb, kFwd ? tb : ta);
        if constexpr (sizeof(T) == 8) lane = lane + 32 < ncomp ? lane + 32 : lane + 32 - ncomp;
    };
#pragma unroll
    for (int d = 0; d < kD; ++d) fetch(d, q[d]);
    __syncthreads();
    for (int t = 0; t < NT; t += kD + 1) {
#pragma unroll
        for (int d = 0; d <= kD; ++d) {
            if (t + d >= NT) break;
            fetch(t + d + kD, q[(d + kD) % (kD + 1)]);
            if (q[d].tile >= 0) {
                Vec<T, L::N> r;
                w.solve(t + d, q[d], r);
                w.template store<kHz>(q[d].tile, r);
            }
            __syncthreads();
        }
    }
}

// The sweep of few grids (at most two on an SM), where nothing else runs while a
// step waits: the time is the chain of one warp's instructions through all
// steps.  Two sets of warps take the steps in turn, so that the chain of a step is
// three face loads, the recurrence and three face stores; a set stores its results
// and issues its next loads while the other set works.  The tables, the ghosts and
// the first tiles are loaded at once.
//
// kRanks: the rows of a grid's tile lattice are shared by the CTAs of a cluster, so
// that a step has the FP64 pipes of nc SMs.  A rank puts the faces of its last row
// into a plane in the next rank's shared memory, where they complete an mbarrier; it
// never waits for that rank, so the way from SM to SM delays the start of a rank once and
// not every step.  Us a sweep of one grid of 32^3 on 8 SMs: 41; with a cluster barrier
// in every step 63; with a released step counter in place of the mbarriers 72.
template <class L, typename T, bool kFwd, bool kHz, int kD, int kThreads, bool kRanks = false, bool kPad = false>
__global__ void __launch_bounds__(kThreads) k_tile_sweep_few(const __grid_constant__ TileArgs<T> a) {
    extern __shared__ __align__(32) unsigned char tsm[];
    TileSweep<L, T, kFwd, kRanks, kPad> w(a, tsm);
    constexpr bool kLate = kPad && !kFwd;   // loads see the pads written first
    const TileShape& s = a.s;
    const int tid = threadIdx.x, ncomp = (blockDim.x - 32) / 2, NT = s.NT, t0 = w.t0, t1 = w.t1;
    const int set = tid >= ncomp ? 1 : 0, lane = tid - set * ncomp;   // (the last warp: neither)
    int2 e[w.kU];
    w.entries(e, tid);
    TileSet<L, T> q[kD];
    // first tile of step t's hyperplane and the one past its last, from global memory
    const int nc = kRanks ? s.nc : 1;
    auto first = [&](int t) { return t < t1 ? __ldg(s.tst + (kFwd ? t : NT - 1 - t) * nc + w.rank) : 0; };
    auto past = [&](int t) { return t < t1 ? __ldg(s.tst + (kFwd ? t : NT - 1 - t) * nc + w.rank + 1) : 0; };
    if (tid < 2 * ncomp)
#pragma unroll
        for (int d = 0; d < kD; ++d) w.coefs(q[d], lane, first(t0 + set + 2 * d), past(t0 + set + 2 * d));
    w.tables();
    if constexpr (kRanks) w.arm();
    follow_on();
    int converged;
    if constexpr (kRanks) {
        int err;
        asm volatile("ld.global.v2.s32 {%0, %1}, [%2];" : "=r"(converged), "=r"(err) : "l"(a.ctl) : "memory");
        converged |= err && err != a.stamp;
    } else {
        converged = flag_at(a.ctl);
    }
    auto start = [&]() {
        if (tid < 2 * ncomp)
#pragma unroll
            for (int d = 0; d < kD; ++d) w.values(q[d]);
    };
    if constexpr (!kLate) start();
    w.ghosts(e);
    if (converged) return;   // (every rank of a cluster or none)
    if constexpr (kRanks) cluster_barrier();
    else __syncthreads();
    if constexpr (kLate) start();
    const int end = t0 + ((t1 - t0 + 1) & ~1);
    if (tid >= 2 * ncomp) {
        bool lost = false;
        w.stage(t0 - 1);
        if constexpr (kRanks) w.boundary(t0 - 1, lost, kFwd && a.lose && w.rank == 1);
        __syncthreads();
        for (int t = t0; t < end; ++t) {
            if (t < t1) w.stage(t);
            if constexpr (kRanks)
                if (t < t1 - 1) w.boundary(t, lost);
            __syncthreads();
        }
        if constexpr (kRanks) {
            cluster_barrier();   // no rank ends while another may put into it
            if (lost) w.drain();
        }
        return;
    }
    __syncthreads();
    Vec<T, L::N> r;
    // (a set's steps have one parity)
    auto* const cur = w.face + ((t0 + set) & 1) * 3 * s.slots - w.back;
    auto* const prv = w.face + ((t0 + set + 1) & 1) * 3 * s.slots - w.back;
    if (set) __syncthreads();   // the first step
    for (int t = t0 + set; t < end; t += 2 * kD) {
#pragma unroll
        for (int d = 0; d < kD; ++d) {
            const int m = t + 2 * d;
            if (m >= end) break;
            if (q[d].tile >= 0) w.solve_at(cur + q[d].x, prv + q[d].x, q[d], r);
            __syncthreads();
            // while the other set works: the results to the next rank and to memory,
            // the loads of the step kD turns on
            if (q[d].tile >= 0) {
                if constexpr (kRanks) w.put(m, q[d], r);
                w.template store<kHz>(q[d].tile, r);
            }
            const int n = min(m + 2 * kD, NT + 1);
            if constexpr (kRanks) {
                w.fetch(q[d], lane, w.tst[n], w.tend[n]);
            } else {
                const int ta = w.tst[n], tb = w.tst[n + 1];
                w.fetch(q[d], lane, kFwd ? ta : tb, kFwd ? tb : ta);
            }
            if (m + 1 < end) __syncthreads();   // the other set's step
        }
    }
    if constexpr (kRanks) cluster_barrier();
}

// hilf of a tile and the facing cells around it
template <class L, typename T>
struct TileHalo {
    Vec<T, L::N> h;
    Vec<T, L::FI> im, ip;
    Vec<T, L::FJ> jm, jp;
    Vec<T, L::FK> km, kp;
};

// The cells across face kF (-i, +i, -j, +j, -k, +k) of a tile: of tile nb of the
// same grid (>= 0), of tile -1-nb of the grid across that face, of the grid's own
// ghost plane, or zero.
template <class L, int kF, bool kPad, typename T>
__device__ __forceinline__ Vec<T, L::template F<kF / 2>> tile_face(const TileArgs<T>& a, int g, int nb,
                                                                   int org) {
    const TileShape& s = a.s;
    constexpr int ax = kF / 2, nf = L::template F<ax>;
    constexpr bool hi = kF % 2 == 0;
    int n = g;
    bool last = false;   // across a low face: the neighbour's last cells are the low ones of their tile
    if (nb < 0) {
        if constexpr (kPad && hi) last = s.pad >> ax & 1;
        n = a.fnbr[6 * g + kF];
        nb = -1 - nb;
        if (n < 0) {
            Vec<T, nf> z;
#pragma unroll
            for (int q = 0; q < nf; ++q) z.v[q] = T(0);
            if (a.PG) {
                const T* P = a.PG + ((long long)g * 6 + kF) * s.fs;
                const int io = org & 1023, jo = (org >> 10) & 1023, ko = org >> 20;
                // a face runs over (dj, dk), (di, dk), (di, dj)
                constexpr int n2 = ax == 2 ? L::TJ : L::TK;
                const int st = ax == 2 ? s.nj : s.nk;
                const int q0 = ax == 0 ? ko + jo * s.nk : (ax == 1 ? ko + io * s.nk : jo + io * s.nj);
#pragma unroll
                for (int q = 0; q < nf; ++q) {
                    const int u = q / n2, v = q % n2;   // (offsets; a pad has no ghost)
                    bool in = true;
                    if constexpr (kPad)
                        in = (ax == 0 ? jo : io) + u < (ax == 0 ? s.nj : s.ni) &&
                             (ax == 2 ? jo : ko) + v < (ax == 2 ? s.nj : s.nk);
                    if (in) z.v[q] = P[q0 + u * st + v];
                }
            }
            return z;
        }
    }
    const T* p = a.H + ((long long)n * s.npp + L::N * nb);
    if constexpr (ax == 0 || nf == 1) {
        // the face's cells are contiguous
        return *reinterpret_cast<const Vec<T, nf>*>(p + (last ? L::template cell<ax>(0, false) : L::template cell<ax>(0, hi)));
    } else {
        Vec<T, L::N> v;
        ldt_co(true, p, v);
        if (kPad && last) return tile_part<L, ax, false>(v);
        return tile_part<L, ax, hi>(v);
    }
}

template <bool kPad = false, class L, typename T>
__device__ __forceinline__ void tile_halo(const TileArgs<T>& a, int g, int tile, int4 n0, int4 n1,
                                          TileHalo<L, T>& o) {
    ldt_co(true, a.H + ((long long)g * a.s.npp + L::N * tile), o.h);
    o.im = tile_face<L, 0, kPad>(a, g, n0.x, n1.z);
    o.ip = tile_face<L, 1, kPad>(a, g, n0.y, n1.z);
    o.jm = tile_face<L, 2, kPad>(a, g, n0.z, n1.z);
    o.jp = tile_face<L, 3, kPad>(a, g, n0.w, n1.z);
    o.km = tile_face<L, 4, kPad>(a, g, n1.x, n1.z);
    o.kp = tile_face<L, 5, kPad>(a, g, n1.y, n1.z);
    if constexpr (kPad) {
        // pads of the last tiles: the ghosts behind them
        const int pad = (n0.y < 0 ? 1 : 0) | (n0.w < 0 ? 2 : 0) | (n1.y < 0 ? 4 : 0);
        if (a.s.pad & pad & 1)
#pragma unroll
            for (int q = 0; q < L::FI; ++q) o.h.v[L::template cell<0>(q, true)] = o.ip.v[q];
        if (a.s.pad & pad & 2)
#pragma unroll
            for (int q = 0; q < L::FJ; ++q) o.h.v[L::template cell<1>(q, true)] = o.jp.v[q];
        if (a.s.pad & pad & 4)
#pragma unroll
            for (int q = 0; q < L::FK; ++q) o.h.v[L::template cell<2>(q, true)] = o.kp.v[q];
    }
}

// the neighbours of cell i of a tile: i-1, i+1, j-1, j+1, k-1, k+1
template <class L, typename T>
__device__ __forceinline__ void tile_nbrs(const TileHalo<L, T>& o, int i, T n[6]) {
    const int di = i / (L::TJ * L::TK), dj = (i / L::TK) % L::TJ, dk = i % L::TK;
    constexpr int M = L::N - 1, J = L::TK, I = L::TJ * L::TK;
    n[0] = di > 0 ? o.h.v[(i - I) & M] : o.im.v[dj * L::TK + dk];
    n[1] = di < L::TI - 1 ? o.h.v[(i + I) & M] : o.ip.v[dj * L::TK + dk];
    n[2] = dj > 0 ? o.h.v[(i - J) & M] : o.jm.v[di * L::TK + dk];
    n[3] = dj < L::TJ - 1 ? o.h.v[(i + J) & M] : o.jp.v[di * L::TK + dk];
    n[4] = dk > 0 ? o.h.v[(i - 1) & M] : o.km.v[di * L::TJ + dj];
    n[5] = dk < L::TK - 1 ? o.h.v[(i + 1) & M] : o.kp.v[di * L::TJ + dj];
}

// The part of sipiter1 outside the recurrence, (rhs + laplacephi(hilf)) lpr
// (sip_hyperplane_mod.F90:491, laplacephi_mod.F90:153-160), one thread a tile;
// the tiles of a grid in gridDim.x CTAs.  Coefficients that differ from cell to cell come
// by coordinate from the grids' one-dimensional arrays, with the couplings a body closes
// masked (as arrays of a class's cells, which a grid with a body does not share, they were
// 28 bytes a cell: 144 grids of 24^3 13.1 -> 11.6 us a launch).  kHz: hilf is zero (a run-time branch had the
// other side compute this one's two instructions a cell as well).  kUni: one value of each operator
// coefficient a class.  Of the first two products one rounds by itself and the
// other is contracted with it: the first in kOrder 0, the second in kOrder 1, as the
// compiler does it in the packed and in the table-driven cell pre-pass.
template <class L, typename T, bool kHz, bool kUni, int kOrder, int kThreads, int kMinBlocks, bool kPad = false>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_tile_pre(const __grid_constant__ TileArgs<T> a) {
    constexpr int N = L::N;
    const TileShape& s = a.s;
    const int b = a.rev ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
    const int g = a.glist ? a.glist[b] : b;
    const int cls = a.gcls[g];
    const long long base = (long long)g * s.npp;
    const int tile = blockIdx.x * kThreads + threadIdx.x, p = N * tile;
    const bool on = tile < s.ntile;
    Vec<T, N> rh, lp, out;
    T u[7];
#pragma unroll
    for (int f = 0; f < 7; ++f) u[f] = kUni ? a.UNI[8 * cls + f] : T(0);
    ldt(on, a.LPR + (long long)cls * a.lprcls + p, lp);
    int4 n0, n1;
    if (on) {
        n0 = __ldg(s.nbr + 2 * tile);
        n1 = __ldg(s.nbr + 2 * tile + 1);
    }
    // the operator's coefficients by coordinate, and the diagonal
    T ci[2][L::TI], cj[2][L::TJ], ck[2][L::TK];
    Vec<T, N> ap;
    uint2 bm = make_uint2(0x3f3f3f3fu, 0x3f3f3f3fu);
    if constexpr (!kUni && !kHz) {
        if (on) {
            const DevGrid* G = a.grids + g;
            const int x = G->ipx + 2 + (n1.z & 1023), y = G->ipy + 2 + ((n1.z >> 10) & 1023),
                      z = G->ipz + 2 + (n1.z >> 20);
#pragma unroll
            for (int f = 0; f < 2; ++f) {
#pragma unroll
                for (int d = 0; d < L::TI; ++d) ci[f][d] = __ldg(a.A1[f] + x + d);
#pragma unroll
                for (int d = 0; d < L::TJ; ++d) cj[f][d] = __ldg(a.A1[2 + f] + y + d);
#pragma unroll
                for (int d = 0; d < L::TK; ++d) ck[f][d] = __ldg(a.A1[4 + f] + z + d);
            }
            if constexpr (N == 8)
                if (a.BM) bm = __ldg(reinterpret_cast<const uint2*>(a.BM + base + p));
        }
        ldt(on, a.AP + (long long)cls * a.apcls + p, ap);
    }
    follow_on();
    if (flag_at(a.ctl) || !on) return;
    ldt_co(true, a.RHS + base + p, rh);
    if constexpr (kHz) {
#pragma unroll
        for (int i = 0; i < N; ++i) out.v[i] = mul_rounded(rh.v[i] + T(0), lp.v[i]);
    } else {
        TileHalo<L, T> o;
        tile_halo<kPad>(a, g, tile, n0, n1, o);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            T n[6], w[7];
            tile_nbrs<L>(o, i, n);
            const unsigned mk = ((i < 4 ? bm.x : bm.y) >> (8 * (i & 3))) & 0xffu;
            const int di = i / (L::TJ * L::TK), dj = (i / L::TK) % L::TJ, dk = i % L::TK;
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                const T x = f < 2 ? ci[f][di] : (f < 4 ? cj[f - 2][dj] : ck[f - 4][dk]);
                w[f] = kUni ? u[f] : (N < 8 || (mk >> f & 1u) ? x : T(0));
            }
            w[6] = kUni ? u[6] : ap.v[i];
            T lap = mul_rounded(-w[kOrder], n[kOrder]);
            lap = lap - w[1 - kOrder] * n[1 - kOrder] - w[2] * n[2] - w[3] * n[3] - w[4] * n[4] - w[5] * n[5] -
                  w[6] * o.h.v[i];
            out.v[i] = mul_rounded(rh.v[i] + lap, lp.v[i]);
        }
    }
    stt(a.R + base + p, out);
}

// ---- host tables ------------------------------------------------------------
template <typename V>
int tile_up(Ctx* c, TileDev& d, const V** p, const std::vector<V>& h) {
    V* m = nullptr;
    if (int rc = scratch(&m, h.size())) return rc;
    d.mem.push_back(m);
    MG_CUDA(copy_on(c->stream, m, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice));
    *p = m;
    return 0;
}

// Tables of a grid of ni x nj x nk cells in tiles of 2^si x 2^sj x 2^sk.  d.ok
// stays false for hyperplanes of more than maxtiles tiles and shapes beyond the
// 10-bit cells or 16-bit slots; kNoScratch where the device has no room for them.
inline int tile_init(Ctx* c, int ni, int nj, int nk, int si, int sj, int sk, int nc, int maxtiles, TileDev& d) {
    TileShape& s = d.s;
    s.nc = nc;
    s.ni = ni; s.nj = nj; s.nk = nk;
    s.si = si; s.sj = sj; s.sk = sk;
    if (ni > 1023 || nj > 1023 || nk > 1023) return 0;
    s.pad = (ni & si) | (nj & sj) << 1 | (nk & sk) << 2;
    const int NI = s.NI = (ni + si) >> si, NJ = s.NJ = (nj + sj) >> sj, NK = s.NK = (nk + sk) >> sk;
    s.NT = NI + NJ + NK - 2;
    s.ntile = NI * NJ * NK;
    s.npp = s.ntile << (si + sj + sk);
    s.fs = (std::max(nj * nk, std::max(ni * nk, ni * nj)) + 3) & ~3;
    s.w = NJ + 1;
    s.slots = (NI + 1) * (NJ + 1);
    // (before any table: one grid of 256^3, whose hyperplanes are too long, would be
    // listed cell by cell for nothing, 115 of 862 ms of its context)
    auto jlo = [&](int t, int I) { return std::max(0, t - I - (NK - 1)); };
    auto jhi = [&](int t, int I) { return std::min(NJ - 1, t - I); };
    for (int t = 0; t < s.NT; ++t)
        for (int r = 0; r < nc; ++r) {
            int n = 0;
            for (int I = (r * NI + nc - 1) / nc; I < ((r + 1) * NI + nc - 1) / nc; ++I)
                n += std::max(0, jhi(t, I) - jlo(t, I) + 1);
            s.maxt = std::max(s.maxt, n);
        }
    if (s.maxt > maxtiles || s.slots > 0xffff || (s.pad && s.ntile > 0xffff)) return 0;
    std::vector<int> tst(1, 0), tpos((size_t)s.NT * NI, 0);
    std::vector<unsigned short> slot((s.ntile + 3) & ~3, 0);
    std::vector<int> ti(s.ntile), tj(s.ntile), tk(s.ntile);
    for (int t = 0, p = 0; t < s.NT; ++t) for (int r = 0; r < nc; ++r) {
        for (int I = (r * NI + nc - 1) / nc; I < ((r + 1) * NI + nc - 1) / nc; ++I) {
            tpos[(size_t)t * NI + I] = p - jlo(t, I);
            for (int J = jlo(t, I); J <= jhi(t, I); ++J, ++p) {
                ti[p] = I; tj[p] = J; tk[p] = t - I - J;
                slot[p] = (unsigned short)((I + 1) * s.w + J + 1);
            }
        }
        tst.push_back(p);
    }
    if (tst.back() != s.ntile) return 0;
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
        nbr[2 * p + 1] = make_int4(km, kp, (I << si) | (J << sj) << 10 | (K << sk) << 20, 0);
    }
    for (int sd = 0; sd < 2; ++sd) {
        struct Entry {
            int r, p;
            int2 e;
        };
        std::vector<Entry> gs;
        // low: coordinate -1, the slot (I+1)w + J+1; high: coordinate N, the slot
        // I w + J the backward sweep uses
        // (with pads a high entry names the grid's own last tile as well)
        auto add = [&](int ax, int I, int J, int K, int t) {
            if (s.pad && sd) t |= tile(std::min(I, NI - 1), std::min(J, NJ - 1), std::min(K, NK - 1)) * 65536u;
            const int x = sd == 0 ? (I + 1) * s.w + J + 1 : I * s.w + J;
            gs.push_back(Entry{(ax > 0 ? I : (sd ? NI - 1 : 0)) * nc / NI, I + J + K, make_int2(x | (ax << 16), t)});
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
            if (a.r != b.r) return a.r < b.r;
            if (a.p != b.p) return a.p < b.p;
            if ((a.e.x >> 16) != (b.e.x >> 16)) return (a.e.x >> 16) < (b.e.x >> 16);
            return a.e.y < b.e.y;
        });
        std::vector<int> gst;
        std::vector<int2> gent;
        size_t q = 0;
        for (int r = 0; r < nc; ++r) {
            const int first = (int)q;
            for (int p = -1; p <= s.NT; ++p) {
                gst.push_back((int)q - first);
                for (; q < gs.size() && gs[q].r == r && gs[q].p == p; ++q) gent.push_back(gs[q].e);
            }
            gst.push_back((int)q - first);
            gst.push_back(first);
            s.nside = std::max(s.nside, (int)q - first);
        }
        if (q != gs.size()) return 0;
        if (int rc = tile_up(c, d, &s.gst[sd], gst)) return rc;
        if (int rc = tile_up(c, d, &s.gent[sd], gent)) return rc;
    }
    // cells: natural local index and place in the cell hyperplane order
    const int kk = nk + 4, jj = nj + 4;
    std::vector<int> cell(s.npp, -1), plane(s.npp, -1);
    {
        int q = 0;
        for (int m = 0; m < ni + nj + nk - 2; ++m)
            for (int io = 0; io < ni; ++io) {
                const int jlo = std::max(0, m - io - (nk - 1)), jhi = std::min(nj - 1, m - io);
                for (int jo = jlo; jo <= jhi; ++jo, ++q) {
                    const int ko = m - io - jo, p = tile_pos(s, tpos.data(), io, jo, ko);
                    cell[p] = (ko + 2) + (jo + 2) * kk + (io + 2) * kk * jj;
                    plane[p] = q;
                }
            }
    }
    if (int rc = tile_up(c, d, &s.tst, tst)) return rc;
    if (int rc = tile_up(c, d, &s.tpos, tpos)) return rc;
    if (int rc = tile_up(c, d, &s.slot, slot)) return rc;
    if (int rc = tile_up(c, d, &s.nbr, nbr)) return rc;
    if (int rc = tile_up(c, d, &s.cell, cell)) return rc;
    if (int rc = tile_up(c, d, &s.plane, plane)) return rc;
    d.ok = true;
    return 0;
}

inline void tile_free(TileDev& d) {
    for (void* p : d.mem) cudaFree(p);
    d = TileDev();
}

}  // namespace
}  // namespace mg
