// plain_tile.cu -- the outer loop of mgpoisl (pressuresolver_mod.F90:203-305) of
// the plain FP64 form on one level, on tiles (sip_tile.cuh).
//
// The values and their order are those of the per-operator kernels
// (plain_poisson.cu): laplacephi, sipiter1, sipiter2, accumulate and rescal per
// point, the halos of conn(res) and conn(dp) read from the neighbours' arrays at
// the iterations the reference exchanges them.  What falls away is the traffic
// between the operators (res written by laplacephi and read by sipiter1, hilf and
// rhs passed over by accumulate and rescal), the connect launches, the per-grid
// copies of the SIP factors (grids with equal spacing and faces share a set, which
// stays in L2), and the host round trip of every outer iteration: the stopping
// test sets a flag the following kernels return on.  A time step of three stages
// (per-operator kernels before): one grid of 32^3 10.6 ms (50.3), 64 of 24^3 15.4
// (38.5), 512 of 24^3 contracted 53-57 (103).  What bounds the sweeps is the FP64 pipe
// (432 warps of points of 24^3, 6 instructions a point uncontracted, 64 clocks each
// on four pipes: 20 us on one SM) and, with fewer grids than SMs, the chain of the
// hyperplanes.
//
// Compiled twice like plain_poisson.cu (-fmad=false and, in namespace contract,
// with contraction).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

#include "internal.h"
#include "plain_tile.h"

namespace mg {
MG_PLAIN_BEGIN
namespace {

using T2 = Tile<1, 1, 2>;
using T1 = Tile<1, 1, 1>;

// RHS (natural layout) into tiles
__global__ void k_pt_gather(const DevGrid* __restrict__ grids, TileShape s, const double* __restrict__ F,
                            double* __restrict__ X) {
    const int g = blockIdx.y, p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.npp) return;
    X[(long long)g * s.npp + p] = F[grids[g].ip3 + s.cell[p]];
}

struct PtOuterArgs {
    TileArgs<double> t;
    double *RHS, *DP;
    double* gridmax;
    const double* RS[3];   // scatter: the res slots
    int ninner;
};

// the laplacian coefficients of a tile's cells (kUni: one value each over a class; the
// diagonal AP is the last of a class's seven arrays)
template <class L, bool kUni>
__device__ __forceinline__ void tile_lap_coefs(const TileArgs<double>& a, int cls, int p,
                                               Vec<double, L::N> (&c)[kUni ? 1 : 7]) {
    if constexpr (!kUni)
#pragma unroll
        for (int f = 0; f < 7; ++f) ldt(true, a.AP + ((long long)cls * 7 + f - 6) * a.s.npp + p, c[f]);
}

// laplacephi at cell i of a tile
template <class L, bool kUni>
__device__ __forceinline__ double tile_lap(const TileArgs<double>& a, int cls, const TileHalo<L, double>& o,
                                           const Vec<double, L::N> (&c)[kUni ? 1 : 7], int i) {
    double n[6], w[7];
    tile_nbrs<L>(o, i, n);
#pragma unroll
    for (int f = 0; f < 7; ++f) w[f] = kUni ? a.UNI[8 * cls + f] : c[kUni ? 0 : f].v[i];
    const double lap = mul_rounded(-w[0], n[0]);
    return lap - w[1] * n[1] - w[2] * n[2] - w[3] * n[3] - w[4] * n[4] - w[5] * n[5] - w[6] * o.h.v[i];
}

// max(|r|, mx) on the words (an order of non-negative numbers; fmax is two FP64
// instructions), which like fmax passes over NaN
__device__ __forceinline__ unsigned long long larger(double r, unsigned long long mx) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
    return b > mx && b <= 0x7ff0000000000000ull ? b : mx;
}

// laplacephi of hilf, rescal (rhs += res) with maxabscal_grid, accumulate (dp +=
// hilf): one thread a tile; gridmax takes the maximum over the CTAs of a grid (of
// non-negative numbers, as integers).
template <class L, bool kUni>
__global__ void __launch_bounds__(128) k_pt_outer(const __grid_constant__ PtOuterArgs a) {
    constexpr int N = L::N;
    __shared__ unsigned long long shm[4];
    const TileShape& s = a.t.s;
    const int g = blockIdx.y, cls = a.t.gcls[g];
    const long long base = (long long)g * s.npp;
    const int tile = blockIdx.x * 128 + threadIdx.x, p = N * tile;
    unsigned long long mx = 0;
    int4 n0, n1;
    if (tile < s.ntile) {
        n0 = __ldg(s.nbr + 2 * tile);
        n1 = __ldg(s.nbr + 2 * tile + 1);
    }
    follow_on();
    if (flag_at(a.t.ctl)) return;
    if (tile < s.ntile) {
        TileHalo<L, double> o;
        tile_halo(a.t, g, tile, n0, n1, o);
        Vec<double, N> rh, dp, c[kUni ? 1 : 7];
        ldt_rw(true, a.RHS + base + p, rh);
        ldt_rw(true, a.DP + base + p, dp);
        tile_lap_coefs<L, kUni>(a.t, cls, p, c);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const double r = rh.v[i] + tile_lap<L, kUni>(a.t, cls, o, c, i);
            rh.v[i] = r;
            dp.v[i] = dp.v[i] + o.h.v[i];
            mx = larger(r, mx);
        }
        stt(a.RHS + base + p, rh);
        stt(a.DP + base + p, dp);
    }
    for (int q = 16; q > 0; q >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, q);
        mx = y > mx ? y : mx;
    }
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 4; ++q) mx = shm[q] > mx ? shm[q] : mx;
        atomicMax(reinterpret_cast<unsigned long long*>(a.gridmax) + g, mx);
    }
}

// The ghosts of RES next to face kF (-i, +i, -j, +j, -k, +k) of a tile, as the last
// exchange of res left them: the facing cells of the grid across, from slot R
// (tile -1 - nb there; org: the tile's first cell, see TileShape::nbr).
template <class L, int kF>
__device__ __forceinline__ void res_ghosts(const TileArgs<double>& a, int g, int nb, int org, const double* R,
                                           double* RES) {
    constexpr int ax = kF / 2;
    const TileShape& s = a.s;
    if (nb >= 0 || !R) return;
    const int n = a.fnbr[6 * g + kF];
    if (n < 0) return;
    Vec<double, L::N> v;
    ldt_co(true, R + ((long long)n * s.npp + L::N * (-1 - nb)), v);
    const auto f = tile_part<L, ax, kF % 2 == 0>(v);
    const int out = kF % 2 == 0 ? -1 : (ax == 0 ? s.ni : (ax == 1 ? s.nj : s.nk));
    const int kk = s.nk + 4, jj = s.nj + 4;
#pragma unroll
    for (int q = 0; q < L::template F<ax>; ++q) {
        int io = org & 1023, jo = (org >> 10) & 1023, ko = org >> 20;
        if (ax == 0) io = out, jo += q / L::TK, ko += q % L::TK;
        else if (ax == 1) jo = out, io += q / L::TK, ko += q % L::TK;
        else ko = out, io += q / L::TJ, jo += q % L::TJ;
        RES[(ko + 2) + (jo + 2) * kk + (io + 2) * kk * jj] = f.v[q];
    }
}

// the residual and the accumulated correction back into RHS and DP, and the
// laplacian of the last correction into RES; its ghosts hold what the last two inner
// iterations exchanged (the last one only from the high side)
template <class L, bool kUni>
__global__ void __launch_bounds__(128) k_pt_scatter(const __grid_constant__ PtOuterArgs a,
                                                    const DevGrid* __restrict__ grids,
                                                    double* __restrict__ RHS, double* __restrict__ DP,
                                                    double* __restrict__ RES) {
    constexpr int N = L::N;
    const TileShape& s = a.t.s;
    const int g = blockIdx.y, cls = a.t.gcls[g];
    const int tile = blockIdx.x * 128 + threadIdx.x, p = N * tile;
    if (tile >= s.ntile) return;
    const long long base = (long long)g * s.npp, ip3 = grids[g].ip3;
    TileHalo<L, double> o;
    const int4 n0 = __ldg(s.nbr + 2 * tile), n1 = __ldg(s.nbr + 2 * tile + 1);
    tile_halo(a.t, g, tile, n0, n1, o);
    const int last = a.t.ctl[2] * a.ninner;   // inner iterations done
    const double *low = a.ninner > 1 ? a.RS[(last - 1) % 3] : nullptr, *high = a.RS[last % 3];
    res_ghosts<L, 0>(a.t, g, n0.x, n1.z, low, RES + ip3);
    res_ghosts<L, 1>(a.t, g, n0.y, n1.z, high, RES + ip3);
    res_ghosts<L, 2>(a.t, g, n0.z, n1.z, low, RES + ip3);
    res_ghosts<L, 3>(a.t, g, n0.w, n1.z, high, RES + ip3);
    res_ghosts<L, 4>(a.t, g, n1.x, n1.z, low, RES + ip3);
    res_ghosts<L, 5>(a.t, g, n1.y, n1.z, high, RES + ip3);
    Vec<double, N> c[kUni ? 1 : 7];
    tile_lap_coefs<L, kUni>(a.t, cls, p, c);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const long long q = ip3 + s.cell[p + i];
        RHS[q] = a.RHS[base + p + i];
        DP[q] = a.DP[base + p + i];
        RES[q] = tile_lap<L, kUni>(a.t, cls, o, c, i);
    }
}

// maxabscal over the grids (one level: no level scale) and the stopping test; the
// maxima are cleared for the next outer iteration.  stat: see PlainTile.
__global__ void k_pt_conv(int ngrid, double* __restrict__ gridmax, double* stat, double prefak, double epcorr,
                          int nouter_min) {
    int* ctl = reinterpret_cast<int*>(stat + 1);
    follow_on();
    if (flag_at(ctl)) return;
    __shared__ double sh[32];
    double m = 0.0;
    for (int g = threadIdx.x; g < ngrid; g += blockDim.x) {
        m = fmax(gridmax[g], m);
        gridmax[g] = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = m;
    __syncthreads();
    if (w == 0) {
        m = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (l == 0) {
            const int done = ctl[2] + 1;
            ctl[2] = done;
            stat[0] = m;
            if (done >= nouter_min && m / prefak < epcorr) ctl[0] = 1;
        }
    }
}

// Up to one grid an SM the step chain of a sweep bounds it, and two sets of warps
// take the steps in turn (24^3: 49 us a sweep on 64 grids, 53 with one set); past
// that a CTA's registers would leave SMs with one grid where two fit (216 grids of
// 20^3: 54 us with one set, 60 with two).
constexpr int kFew = 152;

// Clusters of 8, 4 or 2 CTAs a grid while every CTA has an SM of its own (us a sweep):
// one grid of 32^3 41 / 51 / 83 on 8 / 4 / 2 SMs, 84 on one; 27 grids of 24^3 34 on 4,
// 40 on 2, 49 on one; 64 grids 40 on 2, 49 on one.
constexpr int kRankThreads = 672, kDepth = 2;

static int rank_threads(const TileShape& s) { return 2 * ((s.maxt + 31) / 32 * 32) + 32; }

// the launch of a sweep by clusters of s.nc CTAs
template <class K>
int rank_config(K* k, Ctx* c, const TileShape& s, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    const unsigned smem = tile_layout<T1, double>(s).bytes;
    if (smem > 48 * 1024)
        MG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = s.nc;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg->gridDim = dim3(c->ngrid * s.nc);
    cfg->blockDim = dim3(rank_threads(s));
    cfg->dynamicSmemBytes = smem;
    cfg->stream = c->stream;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    return 0;
}

template <class L, bool kFwd, bool kHz>
int launch_sweep(Ctx* c, const TileArgs<double>& a) {
    const unsigned smem = tile_layout<L, double>(a.s).bytes;
    const int threads = (a.s.maxt + 31) / 32 * 32 + 32;
    auto go = [&](auto* k) -> int {
        if (smem > 48 * 1024)
            MG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        return launch_follow_on(k, dim3(c->ngrid), threads, smem, c->stream, 1, a);
    };
    if constexpr (L::N == 1)
        if (a.s.nc > 1) {
            auto* k = k_tile_sweep_few<L, double, kFwd, kHz, kDepth, kRankThreads, true>;
            if (smem > 48 * 1024)
                MG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
            if (int rc = launch_follow_on(k, dim3(c->ngrid * a.s.nc), rank_threads(a.s), smem, c->stream, a.s.nc, a))
                return rc;
            MG_LAUNCHED(c);
            return 0;
        }
    int rc;
    if (c->ngrid <= kFew && 2 * threads - 32 <= 1024) {
        auto few = [&](auto* k) -> int {
            if (smem > 48 * 1024)
                MG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
            return launch_follow_on(k, dim3(c->ngrid), 2 * threads - 32, smem, c->stream, 1, a);
        };
        rc = 2 * threads - 32 <= 544 ? few(k_tile_sweep_few<L, double, kFwd, kHz, 2, 544>)
                                     : few(k_tile_sweep_few<L, double, kFwd, kHz, 1, 1024>);
    } else if (threads <= 160) rc = go(k_tile_sweep<L, double, kFwd, kHz, 2, 160, 4>);
    else if (threads <= 320) rc = go(k_tile_sweep<L, double, kFwd, kHz, 2, 320, 2>);
    else if (threads <= 544) rc = go(k_tile_sweep<L, double, kFwd, kHz, 2, 544, 1>);
    else rc = go(k_tile_sweep<L, double, kFwd, kHz, 1, 1024, 1>);
    if (rc) return rc;
    MG_LAUNCHED(c);
    return 0;
}

template <class L>
int solve(Ctx* c, double prefak, mglet_stage_stats* st) {
    PlainTile& p = *c->ptile;
    const TileShape& s = p.t.s;
    const size_t bytes = (size_t)c->ngrid * s.npp * sizeof(double);
    const dim3 cells((s.npp + 255) / 256, c->ngrid), tiles((s.ntile + 127) / 128, c->ngrid);
    int* ctl = reinterpret_cast<int*>(p.stat + 1);
    MG_CUDA(cudaMemsetAsync(p.stat, 0, 3 * sizeof(double), c->stream));
    MG_CUDA(cudaMemsetAsync(p.gridmax, 0, c->ngrid * sizeof(double), c->stream));
    MG_CUDA(cudaMemsetAsync(p.dp, 0, bytes, c->stream));
    k_pt_gather<<<cells, 256, 0, c->stream>>>(c->d_grids, s, c->F("RHS"), p.rhs);
    MG_LAUNCHED(c);
    TileArgs<double> a{};
    a.s = s;
    a.fnbr = p.fnbr;
    a.gcls = p.gcls;
    a.H = p.h;
    a.RHS = p.rhs;
    a.LPR = p.cf + 3 * s.npp;
    a.lprcls = 4 * s.npp;
    a.AP = p.lap + 6 * s.npp;
    a.apcls = 7 * s.npp;
    const char* const a1[6] = {"GSAW", "GSAE", "GSAS", "GSAN", "GSAB", "GSAT"};
    for (int q = 0; q < 6; ++q) a.A1[q] = c->L(a1[q]);
    a.grids = c->d_grids;
    a.UNI = p.uni;
    a.ctl = ctl;
    a.err = ctl + 1;
    a.lose = p.lose_once;
    p.lose_once = false;
    PtOuterArgs o{};
    o.RHS = p.rhs;
    o.DP = p.dp;
    o.gridmax = p.gridmax;
    o.ninner = c->prm.ninner;
    for (int q = 0; q < 3; ++q) o.RS[q] = p.rs[q];
    const int ninner = c->prm.ninner;
    // inner iteration gi writes res slot gi % 3 and takes its low ghosts from the
    // last iteration whose exchange covered every face (every inner iteration but
    // the last of an outer one)
    int gi = 0, lastfull = 0;
    for (int ip = 1; ip <= c->prm.nouter; ++ip) {
        for (int il = 1; il <= ninner; ++il) {
            ++gi;
            const bool hz = il == 1;
            a.R = p.rs[gi % 3];
            a.rev = 0;
            {
                ProfScope ps_(c, "laplacephi");
                auto* k = hz ? (p.unicls ? k_tile_pre<L, double, true, true, 0, 128, 4>
                                         : k_tile_pre<L, double, true, false, 0, 128, 4>)
                             : (p.unicls ? k_tile_pre<L, double, false, true, 0, 128, 4>
                                         : k_tile_pre<L, double, false, false, 0, 128, 4>);
                if (int rc = launch_follow_on(k, tiles, 128, 0, c->stream, 1, a)) return rc;
                MG_LAUNCHED(c);
            }
            {
                ProfScope ps_(c, "sipiter1");
                a.stamp = 2 * gi;
                a.G = lastfull > 0 ? p.rs[lastfull % 3] : nullptr;
                a.CF = p.cf;
                a.cfcls = 4 * s.npp;
                a.rev = 1;
                if (int rc = launch_sweep<L, true, false>(c, a)) return rc;
            }
            {
                ProfScope ps_(c, "sipiter2");
                a.stamp = 2 * gi + 1;
                a.G = a.R;
                a.CF = p.cb;
                a.cfcls = 3 * s.npp;
                a.rev = 0;
                if (int rc = hz ? launch_sweep<L, false, true>(c, a) : launch_sweep<L, false, false>(c, a))
                    return rc;
            }
            if (il < ninner) lastfull = gi;
        }
        {
            ProfScope ps_(c, "rescal_maxabs");
            o.t = a;
            if (int rc = launch_follow_on(p.unicls ? k_pt_outer<L, true> : k_pt_outer<L, false>, tiles, 128, 0,
                                          c->stream, 1, o))
                return rc;
            MG_LAUNCHED(c);
            if (int rc = launch_follow_on(k_pt_conv, dim3(1), 256, 0, c->stream, 1, c->ngrid, p.gridmax, p.stat,
                                          prefak, c->prm.epcorr, c->prm.nouter_min))
                return rc;
            MG_LAUNCHED(c);
        }
        // a long outer loop looks now and then whether it has converged
        if (ip % 12 == 0 && ip < c->prm.nouter) {
            MG_CUDA(cudaMemcpyAsync(p.h_stat, p.stat, 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
            MG_CUDA(cudaStreamSynchronize(c->stream));
            const int* h = reinterpret_cast<const int*>(p.h_stat + 1);
            if (h[0] || h[1]) break;
        }
    }
    o.t = a;
    if (p.unicls)
        k_pt_scatter<L, true><<<tiles, 128, 0, c->stream>>>(o, c->d_grids, c->F("RHS"), c->F("DP"), c->F("RES"));
    else
        k_pt_scatter<L, false><<<tiles, 128, 0, c->stream>>>(o, c->d_grids, c->F("RHS"), c->F("DP"), c->F("RES"));
    MG_LAUNCHED(c);
    MG_CUDA(cudaMemcpyAsync(p.h_stat, p.stat, 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    // dp ghosts: the reference accumulates the connected hilf ghosts into dp
    if (int rc = connect(c, 0, 1, nullptr, nullptr, nullptr, c->F("DP"), nullptr, nullptr, false, false, 0))
        return rc;
    MG_CUDA(cudaStreamSynchronize(c->stream));
    if (reinterpret_cast<const int*>(p.h_stat + 1)[1]) {
        set_error("mgpoisl: a sweep timed out waiting for another CTA");
        return MGLET_ERR_CUDA;
    }
    if (st) {
        st->nouter_done = reinterpret_cast<const int*>(p.h_stat + 1)[2];
        st->ipc = st->nouter_done * ninner;
        st->maxrhs = p.h_stat[0];
        st->prefak = prefak;
    }
    return 0;
}

}  // namespace

int plain_tile_solve(Ctx* c, double prefak, mglet_stage_stats* st) {
    return c->ptile->pair ? solve<T2>(c, prefak, st) : solve<T1>(c, prefak, st);
}

MG_PLAIN_END

#ifndef MG_FMA_BUILD
// class coefficients from the FP64 fields of the representative grids
__global__ void k_pt_extract(const DevGrid* __restrict__ grids, const int* __restrict__ reps, TileShape s,
                             const double* __restrict__ lw, const double* __restrict__ ls,
                             const double* __restrict__ lb, const double* __restrict__ lpr,
                             const double* __restrict__ ue, const double* __restrict__ un,
                             const double* __restrict__ ut, const double* __restrict__ ap,
                             const double* __restrict__ AW, const double* __restrict__ AE,
                             const double* __restrict__ AS, const double* __restrict__ AN,
                             const double* __restrict__ AB, const double* __restrict__ AT, double* CF,
                             double* CB, double* LAP) {
    const long long cls = blockIdx.y;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.npp) return;
    const DevGrid G = grids[reps[cls]];
    const int id = s.cell[p];
    const long long src = G.ip3 + s.plane[p];
    const double f[4] = {lw[src], ls[src], lb[src], lpr[src]};
    const double b[3] = {ue[src], un[src], ut[src]};
    const int kk = G.kk, jj = G.jj;
    const int ix = G.ipx + id / (kk * jj), iy = G.ipy + (id / kk) % jj, iz = G.ipz + id % kk;
    const double l[7] = {AW[ix], AE[ix], AS[iy], AN[iy], AB[iz], AT[iz], ap[G.ip3 + id]};
    for (int q = 0; q < 4; ++q) CF[(cls * 4 + q) * s.npp + p] = f[q];
    for (int q = 0; q < 3; ++q) CB[(cls * 3 + q) * s.npp + p] = b[q];
    for (int q = 0; q < 7; ++q) LAP[(cls * 7 + q) * s.npp + p] = l[q];
}

// per class {1, seven coefficients} when each is one value over the class, else {0}
__global__ void k_pt_uniform(TileShape s, const double* __restrict__ LAP, double* UNI) {
    const long long cls = blockIdx.x;
    int bad = 0;
    for (int q = 0; q < 7; ++q) {
        const double* l = LAP + (cls * 7 + q) * s.npp;
        for (int p = threadIdx.x; p < s.npp; p += blockDim.x) bad |= !(l[p] == l[0]);
        if (threadIdx.x == 0) UNI[8 * cls + q] = l[0];
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) UNI[8 * cls + 7] = bad ? 0.0 : 1.0;
}

static int set_up(Ctx* c, const mglet_grid_desc* d) {
    if (c->minlevel != c->maxlevel || !c->uniform || c->prm.psolver == MGLET_PSOLVER_CLASSIC ||
        c->prm.form != MGLET_FORM_PLAIN || c->prm.ninner < 1 || c->prm.nouter < 1)
        return 0;
    const DevGrid& G0 = c->grids[0];
    std::vector<int> fn((size_t)6 * c->ngrid, -1);
    for (size_t r = 0; r < c->conns.size(); r += 4) {
        const int rf = c->conns[r + 2], sf = c->conns[r + 3];
        if (rf > 6) continue;
        if (sf != (rf % 2 ? rf + 1 : rf - 1)) return 0;
        fn[(size_t)6 * (c->conns[r] - 1) + rf - 1] = c->conns[r + 1] - 1;
    }
    PlainTile* p = new PlainTile();
    c->ptile = p;
    auto give_up = [&]() {
        plain_tile_release(c);
        return 0;
    };
    const int ni = G0.ii - 4, nj = G0.jj - 4, nk = G0.kk - 4;
    // few grids: as many SMs to a grid as there are, if the clusters fit at once
    for (int nc = 8; nc > 1 && !p->t.ok; nc /= 2) {
        if (nc * c->ngrid > 152 || nc > ni) continue;
        if (int rc = tile_init(c, ni, nj, nk, 0, 0, 0, nc, (kRankThreads - 32) / 2, p->t)) return rc;
        int fit = 0;
        if (p->t.ok && tile_layout<T1, double>(p->t.s).bytes <= 220 * 1024) {
            auto* k = k_tile_sweep_few<T1, double, true, false, kDepth, kRankThreads, true>;
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at = {};
            if (int rc = rank_config(k, c, p->t.s, &cfg, &at)) return rc;
            MG_CUDA(cudaOccupancyMaxActiveClusters(&fit, k, &cfg));
        }
        if (fit < c->ngrid) tile_free(p->t);
    }
    // Pairs where every SM has more than two grids: the chain of a sweep is then hidden,
    // and the pre-pass and the outer step, which take half the lookups, gain (512 grids of
    // 24^3 55.9 ms a step, 58.9 with single cells); up to there single cells, whose steps
    // are short (216 of 20^3 26.4 ms, 27.4 in pairs), unless a hyperplane has too many.
    for (int pair = c->ngrid > 304 && nk % 2 == 0; pair <= 1 && !p->t.ok; ++pair) {
        if (pair && nk % 2) break;
        p->pair = pair;
        tile_free(p->t);
        if (int rc = tile_init(c, ni, nj, nk, 0, 0, pair, 1, 992, p->t)) return rc;
    }
    if (!p->t.ok) return give_up();
    const TileShape& s = p->t.s;
    const unsigned smem = p->pair ? tile_layout<Tile<1, 1, 2>, double>(s).bytes
                                  : tile_layout<Tile<1, 1, 1>, double>(s).bytes;
    if (smem > 220 * 1024) return give_up();
    // grids with the same faces and spacing share a set of coefficients
    std::map<std::vector<double>, int> seen;
    std::vector<int> gcls(c->ngrid), reps;
    for (int g = 0; g < c->ngrid; ++g) {
        const DevGrid& G = c->grids[g];
        std::vector<double> key;
        for (int f = 0; f < 6; ++f) key.push_back(G.bc[f]);
        key.insert(key.end(), d->dx + G.ipx, d->dx + G.ipx + G.ii);
        key.insert(key.end(), d->dy + G.ipy, d->dy + G.ipy + G.jj);
        key.insert(key.end(), d->dz + G.ipz, d->dz + G.ipz + G.kk);
        auto it = seen.find(key);
        if (it == seen.end()) {
            it = seen.emplace(std::move(key), (int)reps.size()).first;
            reps.push_back(g);
        }
        gcls[g] = it->second;
    }
    p->ncls = (int)reps.size();
    auto up = [&](int** q, const std::vector<int>& h) -> int {
        if (int rc = scratch(q, h.size())) return rc;
        MG_CUDA(copy_on(c->stream, *q, h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice));
        return 0;
    };
    if (int rc = up(&p->gcls, gcls)) return rc;
    if (int rc = up(&p->fnbr, fn)) return rc;
    // one allocation for the FP64 arrays (each a multiple of 256 bytes)
    auto pad = [](size_t n) { return (n + 31) & ~(size_t)31; };
    const size_t n = pad((size_t)c->ngrid * s.npp), m = (size_t)p->ncls * s.npp;
    const size_t cls[3] = {pad(4 * m), pad(3 * m), pad(7 * m)};
    const size_t all = 6 * n + cls[0] + cls[1] + cls[2] + pad(8 * p->ncls) + pad(c->ngrid) + pad(3);
    if (int rc = scratch(&p->mem, all)) return rc;
    double* q = p->mem;
    auto take = [&](double** d, size_t len) {
        *d = q;
        q += len;
    };
    for (double** d : {&p->h, &p->rhs, &p->dp, &p->rs[0], &p->rs[1], &p->rs[2]}) take(d, n);
    take(&p->cf, cls[0]);
    take(&p->cb, cls[1]);
    take(&p->lap, cls[2]);
    take(&p->uni, pad(8 * p->ncls));
    take(&p->gridmax, pad(c->ngrid));
    take(&p->stat, pad(3));
    MG_CUDA(cudaMallocHost(&p->h_stat, 3 * sizeof(double)));
    int* d_reps = nullptr;
    if (int rc = up(&d_reps, reps)) return rc;
    k_pt_extract<<<dim3((s.npp + 255) / 256, p->ncls), 256, 0, c->stream>>>(
        c->d_grids, d_reps, s, c->F("SIPLW"), c->F("SIPLS"), c->F("SIPLB"), c->F("SIPLPR"), c->F("SIPUE"),
        c->F("SIPUN"), c->F("SIPUT"), c->F("GSAP"), c->L("GSAW"), c->L("GSAE"), c->L("GSAS"), c->L("GSAN"),
        c->L("GSAB"), c->L("GSAT"), p->cf, p->cb, p->lap);
    k_pt_uniform<<<p->ncls, 256, 0, c->stream>>>(s, p->lap, p->uni);
    c->launches += 2;
    std::vector<double> uni((size_t)8 * p->ncls);
    cudaError_t e = copy_on(c->stream, uni.data(), p->uni, uni.size() * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d_reps);
    if (e != cudaSuccess) return cuda_fail(e, "plain tiles");
    p->unicls = true;
    for (int q = 0; q < p->ncls; ++q) p->unicls = p->unicls && uni[(size_t)8 * q + 7] != 0.0;
    return 0;
}

int plain_tile_init(Ctx* c, const mglet_grid_desc* d) {
    const int rc = set_up(c, d);
    if (rc != kNoScratch) return rc;
    plain_tile_release(c);   // the per-operator kernels need no more than the fields
    return 0;
}

void plain_tile_release(Ctx* c) {
    PlainTile* p = c->ptile;
    if (!p) return;
    cudaStreamSynchronize(c->stream);
    tile_free(p->t);
    for (void* q : {(void*)p->gcls, (void*)p->fnbr, (void*)p->mem}) cudaFree(q);
    if (p->h_stat) cudaFreeHost(p->h_stat);
    delete p;
    c->ptile = nullptr;
}

int plain_tile_test_timeout(Ctx* c) {
    if (!c->ptile || c->ptile->t.s.nc == 1) {
        set_error("test_sweep_timeout: needs the plain form's solve on tiles with grids shared by SMs");
        return MGLET_ERR_UNSUPPORTED;
    }
    c->ptile->lose_once = true;
    return 0;
}

bool plain_tile_ready(const Ctx* c) { return c->ptile != nullptr; }
#endif

}  // namespace mg
