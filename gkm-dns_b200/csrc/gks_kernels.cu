// Kernels of the WENO-GKS step and its diagnostics (sm_100a).
//
// A step is seven launches over every field of the batch: for each sweep
// direction a reconstruction launch (WENO once per cell line and interface)
// and a flux launch (transverse slopes from the neighbouring lines' WENO
// states, BGK-NS flux), then the conservative update; or six, where the z flux
// applies the update itself.  Every launch loops over the cells of all
// fields, so one launch covers an ensemble of fields of different sizes.  The periodic halo of the
// reference (HaloTransfer on one rank, update.cpp:894-1054) is the index wrap
// in `along` and in the windowed reconstruction's cell map.
#include "gks_device.cuh"
#include "gks_flux.cuh"
#include "gks_flux64.cuh"
#include "gks_kernels.cuh"
#include "../../include/gks_b200.h"

#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <type_traits>

namespace gks {

namespace {

__device__ __forceinline__ int field_of(const FieldDev *f, int n, long long it)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (f[mid].base <= it) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The field of a warp's items in a flux kernel.  A warp's items ascend, so the
// field is searched for once and then walked forward, its end kept in a
// register: a search per interface is up to seven dependent loads, about 50
// cycles each, that three warps per scheduler do not cover.  FP64 us per sweep
// (x / y / z), 96 fields of 32^3, 48^3 and 64^3: 1397 / 1398 / 1495 -> 1287 / 1284 / 1322.
struct FieldWalk {
    const FieldDev *f;
    long long end; // first item of the next field
    int left;      // fields after this one
    __device__ __forceinline__ FieldWalk(const Batch &b, long long it, bool ensemble = true)
    {
        if (!ensemble) return;
        const int i = field_of(b.fields, b.nfields, it);
        f = b.fields + i;
        left = b.nfields - 1 - i;
        end = left ? f[1].base : LLONG_MAX;
    }
    __device__ __forceinline__ const FieldDev &at(long long it)
    {
        while (it >= end) {
            ++f;
            --left;
            end = left ? f[1].base : LLONG_MAX;
        }
        return *f;
    }
};

struct Cell {
    int j, i, k, nc;
    int nyw;    // y-wrap modulus (FieldDev::nyw)
    unsigned c; // (j*nc + i)*nc + k
};

// x / nc by multiply-high with the field's precomputed magic number.
__device__ __forceinline__ unsigned div_nc(unsigned x, const FieldDev &f)
{
    return (unsigned)(((unsigned long long)__umulhi(x, f.nc_magic) + x) >> f.nc_shift);
}

__device__ __forceinline__ Cell decode(unsigned c, const FieldDev &f)
{
    Cell x;
    x.nc = f.nc;
    x.nyw = f.nyw;
    x.c = c;
    const unsigned r = div_nc(c, f);
    x.k = int(c - r * f.nc);
    const unsigned jj = div_nc(r, f);
    x.i = int(r - jj * f.nc);
    x.j = int(jj);
    return x;
}

__device__ __forceinline__ int wrap(int x, int n) { return x < 0 ? x + n : (x >= n ? x - n : x); }

// Displacement along the sweep axis: DIR 0 = x (i), 1 = y (j), 2 = z (k);
// only the swept coordinate wraps (y not at all in a slab, whose ghost planes
// are stored).
template <int DIR>
__device__ __forceinline__ unsigned along(const Cell &x, int d)
{
    const int n = x.nc;
    if (DIR == 0) return x.c + (unsigned)((wrap(x.i + d, n) - x.i) * n);
    if (DIR == 1) return x.c + (unsigned)((wrap(x.j + d, x.nyw) - x.j) * n * n);
    return x.c + (unsigned)(wrap(x.k + d, n) - x.k);
}

__device__ __forceinline__ double viscosity(const FieldDev &f, double T)
{
    const double x = T * f.iT0;
    if (f.visc_law == GKS_VISC_POWER) return f.mu0 * pow(x, f.visc_exp);
    // mu0 (T/T0)^1.5 (T0 + 110.4)/(T + 110.4), update.cpp:263
    return f.mu0 * (x * sqrt(x)) * (f.T0 + 110.4) * __drcp_rn(T + 110.4);
}

// Collision time mu / p of the state W (update.cpp:262-264) as a fraction
// num / den, which the flux divides out together with its other terms.
// Sutherland, with A = rho2p(W), T = cT A / rho^2 and p = (gamma - 1) A / rho:
//   mu / p = mu0 y^1.5 (T0 + 110.4) / ((gamma - 1) A (cT A + 110.4 rho^2)),  y = cT A / T0,
// in which the powers of rho cancel (no reciprocal at all).
__device__ __forceinline__ void visc_over_p(const FieldDev &f, const double W[5], double &num, double &den)
{
    const double A = rho2p(W);
    if (f.visc_law == GKS_VISC_POWER) {
        const double ri = __drcp_rn(W[0]);
        den = f.gm1 * (A * ri);
        num = viscosity(f, den * ri * f.iR);
        return;
    }
    const double y = (f.cT * A) * f.iT0;
    den = (f.gm1 * A) * fma(110.4 * W[0], W[0], f.cT * A);
    num = (f.mu0 * (y * sqrt(y))) * (f.T0 + 110.4);
}

// mu/p of cell c, stored once per step by the x-sweep reconstruction for the
// flux kernels of all three sweeps (the left cell of interface c is c in each).
__device__ __forceinline__ void store_tau(const FieldDev &f, unsigned c, const double W[5])
{
    double n, d;
    visc_over_p(f, W, n, d);
    f.tau[0][c] = n;
    f.tau[1][c] = d;
}

// FP64: 1/rho from rcp_cubic.  Mixed: correctly rounded (its FP32 steps round
// differences of these values, so that path's double arithmetic is kept as it
// is: a last-place change flips an FP32 rounding now and then).
template <int PREC> __device__ __forceinline__ double temperature(const double W[5], double cT)
{
    // (gam-1)(E/rho - |m|^2/(2 rho^2))/R, update.cpp:560
    const double ri = PREC == 0 ? rcp_cubic(W[0]) : __drcp_rn(W[0]);
    const double ke = fma(W[1], W[1], fma(W[2], W[2], W[3] * W[3]));
    return cT * fma(-0.5 * ke, ri * ri, W[4] * ri);
}

// rho E from the reconstructed density, momentum and temperature
// (update.cpp:618-619): rho T R/(gam-1) + |m|^2 / (2 rho), ri = 1/rho.
__device__ __forceinline__ double energy(const double w[4], double T, double ri, double icT)
{
    const double ke = fma(w[1], w[1], fma(w[2], w[2], w[3] * w[3]));
    return fma(w[0] * T, icT, (0.5 * ke) * ri);
}

// The reconstruction record of cell c: Wl[0..4] then Wr[0..4] as five
// 16-byte pairs, pair k of every cell in its own array of n = nc^3 pairs
// (rec + 2 k n doubles, 16-byte aligned): a warp's load or store of one pair
// for 32 consecutive cells is 512 contiguous bytes, and a record takes five
// 16-byte accesses instead of ten 8-byte ones.
__device__ __forceinline__ void put_record(double *rec, unsigned c, const double wl[5], const double wr[5], long long n)
{
    double2 *p = reinterpret_cast<double2 *>(rec) + c;
    p[0] = make_double2(wl[0], wl[1]);
    p[n] = make_double2(wl[2], wl[3]);
    p[2 * n] = make_double2(wl[4], wr[0]);
    p[3 * n] = make_double2(wr[1], wr[2]);
    p[4 * n] = make_double2(wr[3], wr[4]);
}

__device__ __forceinline__ void get_record(const double *rec, unsigned c, double v[10], long long n)
{
    const double2 *p = reinterpret_cast<const double2 *>(rec) + c;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const double2 t = __ldg(p + k * n);
        v[2 * k] = t.x;
        v[2 * k + 1] = t.y;
    }
}

// ---------------------------------------------------------------------------
// The five reconstructed quantities of a cell are rho, the momenta and the
// temperature (update.cpp:560-619) or, with GKS_DIRECT_ENERGY, rho E
// (GPUupdate.cu:917-977).
// ---------------------------------------------------------------------------
// FP64: both states of one cell from the quantities' six differences d around
// it and their values g at it, rho E from the temperatures.
__device__ __forceinline__ void cell_states(const double (&d)[5][6], const double (&g)[5], bool direct, double icT,
                                            double wl[5], double wr[5])
{
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        double dl, dr;
        weno_cell(d[q], dl, dr);
        wl[q] = g[q] + dl;
        wr[q] = g[q] + dr;
    }
    if (direct) return;
    wl[4] = energy(wl, wl[4], rcp_cubic(wl[0]), icT);
    wr[4] = energy(wr, wr[4], rcp_cubic(wr[0]), icT);
}

// Mixed: both states of one interface from its stencil's quantities s(a, q),
// a = 0 .. 5 (LLL .. RRR).  WENO in FP32 on differences from the left cell,
// added back in FP64; quantities (0, 1) and (2, 3) as the two lanes of paired
// FP32 instructions, the fifth alone.
template <typename SG>
__device__ __forceinline__ void interface_states(const SG &s, bool direct, double icT, double wl[5], double wr[5])
{
    const float epsf = float(kWenoEps);
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
        const double c0 = s(2, q), c1 = s(2, q + 1);
        f2 v[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) v[a] = f2(float(s(a, q) - c0), float(s(a, q + 1) - c1));
        f2 dl, dr;
        weno_pair<f2>(v[0], v[1], f2(0.0f), v[3], v[4], v[5], f2(epsf), dl, dr);
        wl[q] = c0 + double(dl.v.x);
        wr[q] = c0 + double(dr.v.x);
        wl[q + 1] = c1 + double(dl.v.y);
        wr[q + 1] = c1 + double(dr.v.y);
    }
    const double c0 = s(2, 4);
    float dl, dr;
    weno_pair<float>(float(s(0, 4) - c0), float(s(1, 4) - c0), 0.0f, float(s(3, 4) - c0), float(s(4, 4) - c0),
                     float(s(5, 4) - c0), epsf, dl, dr);
    wl[4] = c0 + double(dl);
    wr[4] = c0 + double(dr);
    if (direct) return;
    const double r = __drcp_rn(wl[0] * wr[0]); // one reciprocal for both densities
    wl[4] = energy(wl, wl[4], wr[0] * r, icT);
    wr[4] = energy(wr, wr[4], wl[0] * r, icT);
}

// The last field whose range (FieldDev::*BASE) starts at or before item `it`, the
// same item range for all 32 lanes: each round splits the fields left into 32
// parts, a lane looking at the start of one, so up to 32 fields take one load's
// latency and up to 1024 two (a binary search of 96 fields: seven).
// FP64 us per sweep, 96 fields of 32^3: 148 / 131 / 174 -> 145 / 127 / 166.
template <long long FieldDev::*BASE>
__device__ __forceinline__ int field_of_warp(const FieldDev *f, int n, long long it)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int part = (hi - lo + 31) / 32, i = lo + int(threadIdx.x & 31) * part;
        const unsigned below = __ballot_sync(0xffffffffu, i < hi && f[i < hi ? i : lo].*BASE <= it);
        lo += (31 - __clz(below)) * part;
        hi = min(lo + part, hi);
    }
    return lo;
}

// ---------------------------------------------------------------------------
// Reconstruction for the z sweep: a work item is one (j, i) line, a warp walks
// it in segments of 32 cells, one cell per lane.  The warp's shared-memory
// tile holds the five quantities of the segment's cells and the three cells
// either side: each segment brings 32 new cells (loaded into registers while
// the segment before is computed, one coalesced load per lane and component,
// one temperature per cell) and keeps the last six of the one before.
// Mixed: a lane forms both states of the interface above its cell.  FP64: it
// forms the two states of its cell; its left state meets the right state of
// the next lane's cell: lane L writes the interface below its cell with the
// left state handed over by lane L - 1, lane 0's from the last lane of the
// segment before; the line's last interface takes the right state of cell 0,
// kept from the first segment.
// ---------------------------------------------------------------------------
constexpr int kZLineWarps = kReconBlock / 32, kZLineCells = 32 + 6;

template <int PREC, bool ENSEMBLE>
__device__ __forceinline__ void recon_zlines(const Batch &b, double (&tiles)[kZLineWarps][5][kZLineCells])
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double (*tile)[kZLineCells] = tiles[wid];
    const long long stride = (long long)gridDim.x * kZLineWarps;
    for (long long it = b.lo + (long long)blockIdx.x * kZLineWarps + wid; it < b.hi; it += stride) {
        const FieldDev &f = ENSEMBLE ? b.fields[field_of_warp<&FieldDev::zbase>(b.fields, b.nfields, it)] : b.one;
        const int nc = f.nc;
        const unsigned lbase = unsigned(it - f.zbase) * unsigned(nc); // cell (j, i, 0)
        const bool direct = (f.flags & GKS_DIRECT_ENERGY) != 0;
        const double cT = f.cT, icT = f.icT;
        double w[5];
        auto load = [&](int k) { // cell k of the line, -3 <= k < nc + 3
            const unsigned c = lbase + unsigned(wrap(k, nc));
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = __ldg(f.W[q] + c);
        };
        auto put = [&](int col) {
#pragma unroll
            for (int q = 0; q < 4; ++q) tile[q][col] = w[q];
            tile[4][col] = direct ? w[4] : temperature<PREC>(w, cT);
        };
        if (lane < 6) { // cells -3 .. 2
            load(lane - 3);
            put(lane);
        }
        if (lane < nc) load(lane + 3);
        double first[5], carry[5]; // lane 0: right state of cell 0, left state of the cell before the segment
#pragma unroll
        for (int q = 0; q < 5; ++q) first[q] = carry[q] = 0.0;
        for (int k0 = 0; k0 < nc; k0 += 32) {
            const int k = k0 + lane; // this lane's cell, column lane + 3
            if (k < nc) put(lane + 6);
            __syncwarp();
            if (k + 32 < nc) load(k + 35);
            if constexpr (PREC == 0) {
                double wl[5], wr[5];
                if (k < nc) {
                    double d[5][6], g[5];
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        double lo = tile[q][lane];
#pragma unroll
                        for (int a = 0; a < 6; ++a) {
                            const double hi = tile[q][lane + a + 1];
                            d[q][a] = hi - lo;
                            lo = hi;
                            if (a == 2) g[q] = hi;
                        }
                    }
                    cell_states(d, g, direct, icT, wl, wr);
                } else {
#pragma unroll
                    for (int q = 0; q < 5; ++q) wl[q] = wr[q] = 0.0;
                }
                // lane L takes the left state of lane L - 1, lane 0 the segment's last
                const int src = lane ? lane - 1 : min(31, nc - 1 - k0);
                double left[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    const double t = __shfl_sync(0xffffffffu, wl[q], src);
                    left[q] = lane ? t : carry[q];
                    carry[q] = t;
                }
                if (k == 0) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) first[q] = wr[q];
                } else if (k < nc) {
                    put_record(f.rec[2], lbase + unsigned(k - 1), left, wr, f.ncell);
                }
            } else if (k < nc) {
                double wl[5], wr[5];
                interface_states([&](int a, int q) -> double { return tile[q][lane + a + 1]; }, direct, icT, wl, wr);
                put_record(f.rec[2], lbase + unsigned(k), wl, wr, f.ncell);
            }
            __syncwarp();
            if (lane < 6) { // the last six cells become the first six of the next segment
#pragma unroll
                for (int q = 0; q < 5; ++q) tile[q][lane] = tile[q][lane + 32];
            }
            __syncwarp();
        }
        if (PREC == 0 && lane == 0) put_record(f.rec[2], lbase + unsigned(nc - 1), carry, first, f.ncell);
    }
}

// FP64 reads a one-field batch's descriptor from the launch parameters (x and y
// windows and z lines): from memory, every asynchronous copy, a memory barrier
// to the compiler, has the pointers and constants loaded again.  us per sweep at
// 256^3, x / y / z: 625 / 554 / 607 -> 597 / 547 / 592; 130^3 111 / 97 / 109 -> 106 /
// 96 / 105.  Mixed needs more registers with two loops in a kernel (120 -> 138; y
// 454 -> 469, z 448 -> 457 us) and keeps one.
template <int PREC, int MINB>
__global__ void __launch_bounds__(kReconBlock, MINB) k_recon_zline(Batch b)
{
    __shared__ double tiles[kZLineWarps][5][kZLineCells];
    if (PREC == 0 && b.nfields == 1) recon_zlines<PREC, false>(b, tiles);
    else recon_zlines<PREC, true>(b, tiles);
}

// ---------------------------------------------------------------------------
// Reconstruction for the x (DIR 0) and y (DIR 1) sweeps with a sliding
// window: a work item is a run of consecutive interfaces along the sweep at
// one (transverse line, k); the lanes of a warp take consecutive k, so every
// load is coalesced.  Cells arrive by asynchronous copies in a ring of
// kWinRing slots in the thread's own part of shared memory
// ([slot][component][thread], no bank conflicts) a few cells ahead of their
// use.  Mixed: each interface reads its six-cell stencil from the ring, the
// six temperatures stay in registers.  FP64: a run of n interfaces evaluates
// n + 1 cells; the window is the six differences of each quantity in
// registers, which slide by one cell (five loads, one temperature, five
// differences per cell), and the left state of a cell waits one cell for the
// right state of the next, with which it leaves as one record.  Item order: k
// fastest, then run, then the transverse line.  A launch over a range of y
// planes (Batch::wy0 .. wy1, one field) cuts that range into runs of
// Batch::wrun interfaces.
// ---------------------------------------------------------------------------
constexpr int kWinRing = 8;
// Cells in flight: the ring holds cells p .. p + 3 of the FP64 window, p - 2 ..
// p + 3 of the mixed one, besides them.
__host__ __device__ constexpr int win_prefetch(int prec) { return prec == 0 ? 3 : 2; }

template <int DIR, int PREC, bool ENSEMBLE>
__device__ __forceinline__ void recon_runs(const Batch &b, double (&ring)[kWinRing][5][kReconBlock])
{
    constexpr int PF = win_prefetch(PREC), NR = kWinRing;
    static_assert(NR >= (PREC == 0 ? 4 : 6) + PF && (NR & (NR - 1)) == 0, "the ring holds the live cells and those in flight");
    const int tid = threadIdx.x;
    static_assert(DIR == 0 || DIR == 1, "windowed reconstruction is for the x and y sweeps");
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long it = b.lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; it < b.hi; it += stride) {
        const FieldDev &f = ENSEMBLE ? b.fields[field_of_warp<&FieldDev::wbase>(b.fields, b.nfields, it)] : b.one;
        const bool ranged = DIR == 1 && b.wy1 > 0;
        const long long loc = ranged ? it : it - f.wbase;
        if (!ranged && loc >= f.nwin) continue; // alignment padding after the field
        const int nc = f.nc;
        const unsigned u = unsigned(loc);
        const unsigned rest = div_nc(u, f);
        const int k = int(u - rest * unsigned(nc));
        const int run = ranged ? b.wrun : f.run;
        const int nrun = ranged ? (b.wy1 - b.wy0 + run - 1) / run : f.nrun;
        const int line = int(rest / unsigned(nrun));
        const int s0 = int(rest - unsigned(line) * unsigned(nrun)) * run + (ranged ? b.wy0 : 0);
        const int s1 = min(s0 + run, ranged ? b.wy1 : nc); // interfaces [s0, s1)
        // cell (line, sweep position p, k): x sweep (j, i, k), y sweep (j = p, i =
        // line).  A slab's y index does not wrap: the first cell of the first run
        // and the last cell of the last one lie beyond its stored planes; they
        // enter only the states that are not kept, and read the top plane instead
        const unsigned step = DIR == 0 ? unsigned(nc) : unsigned(nc) * unsigned(nc);
        const unsigned lbase = DIR == 0 ? unsigned(line) * unsigned(nc) * unsigned(nc) + unsigned(k)
                                        : unsigned(line) * unsigned(nc) + unsigned(k);
        const int nw = DIR == 0 ? nc : f.nyw, top = DIR == 0 ? nc - 1 : f.ny - 1;
        auto cell = [&](int p) -> unsigned { return lbase + unsigned(max(0, min(wrap(p, nw), top))) * step; };
        const bool direct = (f.flags & GKS_DIRECT_ENERGY) != 0;
        const double cT = f.cT, icT = f.icT;
        // cells up to s1 + 3 (mixed: s1 + 2), cell pc in ring slot pc mod NR, one copy
        // group per cell (empty past the run)
        const int pend = s1 + (PREC == 0 ? 3 : 2);
        auto fetch = [&](int pc) {
            if (pc <= pend) {
                const unsigned c = cell(pc);
#pragma unroll
                for (int q = 0; q < 5; ++q) cp_async8(&ring[pc & (NR - 1)][q][tid], f.W[q] + c);
            }
            cp_async_commit();
        };
        // the five quantities of cell pc
        auto quantities = [&](int pc, double (&g)[5]) {
            double w[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = ring[pc & (NR - 1)][q][tid];
#pragma unroll
            for (int q = 0; q < 4; ++q) g[q] = w[q];
            g[4] = direct ? w[4] : temperature<PREC>(w, cT);
        };
        if constexpr (PREC == 0) {
            double d[5][6];
            double last[5]; // quantities of cell p + 3 (the newest)
            double T[4];    // fifth quantity of cells p .. p + 3
#pragma unroll
            for (int a = 0; a < 1 + PF; ++a) fetch(s0 - 3 + a);
            cp_async_wait<PF>();
            quantities(s0 - 3, last);
#pragma unroll
            for (int a = 1; a < 6; ++a) {
                fetch(s0 - 3 + a + PF);
                cp_async_wait<PF>();
                double g[5];
                quantities(s0 - 3 + a, g);
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    d[q][a] = g[q] - last[q];
                    last[q] = g[q];
                }
                if (a >= 3) T[a - 2] = g[4];
            }
            double left[5];
#pragma unroll 1
            for (int p = s0; p <= s1; ++p) {
                // cell p + 3 + PF takes the slot of cell p + 3 + PF - NR, which lies below p
                fetch(p + 3 + PF);
                cp_async_wait<PF>(); // cell p + 3 has landed
                double g[5];
                quantities(p + 3, g);
#pragma unroll
                for (int q = 0; q < 5; ++q) {
#pragma unroll
                    for (int a = 0; a < 5; ++a) d[q][a] = d[q][a + 1];
                    d[q][5] = g[q] - last[q];
                    last[q] = g[q];
                }
                T[0] = T[1];
                T[1] = T[2];
                T[2] = T[3];
                T[3] = g[4];
                double wc[5];
#pragma unroll
                for (int q = 0; q < 4; ++q) g[q] = wc[q] = ring[p & (NR - 1)][q][tid];
                g[4] = T[0];
                double wl[5], wr[5];
                cell_states(d, g, direct, icT, wl, wr);
                if (DIR == 0 && p < s1) {
                    wc[4] = ring[p & (NR - 1)][4][tid];
                    store_tau(f, cell(p), wc);
                }
                if (p > s0) put_record(f.rec[DIR], cell(p - 1), left, wr, f.ncell);
#pragma unroll
                for (int q = 0; q < 5; ++q) left[q] = wl[q];
            }
        } else {
#pragma unroll
            for (int a = 0; a < 5 + PF; ++a) fetch(s0 - 2 + a);
            cp_async_wait<PF>(); // the five first window cells have landed
            double T[6];
#pragma unroll
            for (int a = 0; a < 5; ++a) {
                double g[5];
                quantities(s0 - 2 + a, g);
                T[a + 1] = g[4];
            }
#pragma unroll 2
            for (int p = s0; p < s1; ++p) {
#pragma unroll
                for (int a = 0; a < 5; ++a) T[a] = T[a + 1];
                cp_async_wait<PF - 1>(); // cell p + 3 (issued PF groups ago) has landed
                double g[5];
                quantities(p + 3, g);
                T[5] = g[4];
                const auto sg = [&](int a, int q) -> double { return q < 4 ? ring[(p - 2 + a) & (NR - 1)][q][tid] : T[a]; };
                double wl[5], wr[5];
                interface_states(sg, direct, icT, wl, wr);
                const unsigned c = cell(p);
                if (DIR == 0) {
                    double w[5];
#pragma unroll
                    for (int q = 0; q < 5; ++q) w[q] = ring[p & (NR - 1)][q][tid];
                    store_tau(f, c, w);
                }
                put_record(f.rec[DIR], c, wl, wr, f.ncell);
                // cell p + 3 + PF takes the slot of cell p + 3 + PF - NR, which no
                // stencil from here on reads (it lies below p - 2)
                fetch(p + 3 + PF);
            }
        }
        cp_async_wait<0>(); // nothing in flight into the ring before the next item
    }
}

template <int DIR, int PREC, int MINB>
__global__ void __launch_bounds__(kReconBlock, MINB) k_recon_win(Batch b)
{
    __shared__ double ring[kWinRing][5][kReconBlock];
    if (PREC == 0 && b.nfields == 1) recon_runs<DIR, PREC, false>(b, ring);
    else recon_runs<DIR, PREC, true>(b, ring);
}

// ---------------------------------------------------------------------------
// Flux at the interface between cell c and its +1 neighbour along DIR
// (derivsX/Y/Z, update.cpp:201-453, and flux, GKMflux.cpp:11-215).
// Transverse lines: x sweep N,S = y+-1, F,B = z+-1; y sweep N,S = x+-1 (the
// reference takes x-+1 with DWy = -(N-S)/2dx), F,B = z+-1; z sweep N,S = x+-1,
// F,B = y+-1 (the reference's assignment) or, with GKS_FIX_ZSWEEP, N,S = y+-1,
// F,B = x+-1.
// Momentum is rotated into slot 1 for y (rho v) and z (rho w).
// ---------------------------------------------------------------------------
template <int DIR>
__device__ __forceinline__ void transverse(const Cell &x, int flags, unsigned &n, unsigned &s, unsigned &fr,
                                           unsigned &bk)
{
    if (DIR == 0) {
        n = along<1>(x, 1); s = along<1>(x, -1);
        fr = along<2>(x, 1); bk = along<2>(x, -1);
    } else if (DIR == 1) {
        n = along<0>(x, 1); s = along<0>(x, -1);
        fr = along<2>(x, 1); bk = along<2>(x, -1);
    } else {
        if (flags & GKS_FIX_ZSWEEP) {
            n = along<1>(x, 1); s = along<1>(x, -1);
            fr = along<0>(x, 1); bk = along<0>(x, -1);
        } else {
            n = along<0>(x, 1); s = along<0>(x, -1);
            fr = along<1>(x, 1); bk = along<1>(x, -1);
        }
    }
}

// Inputs and running sums of one interface.  All global loads are issued when
// the interface starts; the values are parked in this thread's own
// shared-memory slots ([slot][thread], no bank conflicts) until a pass of the
// flux needs them, and so are the sums the two side passes accumulate for the
// equilibrium pass, so that only one pass's state is in registers at a time.
// Slot q of the rotated frame holds original
// component perm(q): rho v (y sweep) or rho w (z sweep) moves into slot 1
// (update.cpp:340-350, 429-439).  DWxl = 2(Wl - WL)/dx, DWxr = 2(WR - Wr)/dx;
// transverse central differences of the neighbouring lines' states
// (update.cpp:253-260, 327-334, 416-423), here the differences in double (they
// cancel), which the flux scales.
template <int DIR> __device__ constexpr int perm(int q)
{
    return DIR == 0 ? q : (q == 1 ? (DIR == 1 ? 2 : 3) : (q == (DIR == 1 ? 2 : 3) ? 1 : q));
}

// The ten-value records of the interface and its four transverse neighbours.
struct Records {
    double r0[10], rn[10], rs[10], rf[10], rb[10];
    __device__ __forceinline__ Records(const double *rec, unsigned c, unsigned cn, unsigned cs, unsigned cf, unsigned cb,
                                       long long n)
    {
        get_record(rec, c, r0, n);
        get_record(rec, cn, rn, n);
        get_record(rec, cs, rs, n);
        get_record(rec, cf, rf, n);
        get_record(rec, cb, rb, n);
    }
};

// FP64 path (gks_flux64): 53 slots, 424 B per thread.  The left side's inputs sit
// in the slots of sums that its own pass writes after it has read them.
template <int DIR> struct SweepSrc64 {
    static constexpr int kWL = 0, kWR = 5, kWr = 10, kDr = 15; // cell averages, right state, its transverse slopes
    static constexpr int kW0 = 25, kBy = 30, kBz = 35, kB = 40, kF = 45; // sums
    static constexpr int kWl = kBy, kDl = kB;                            // left state, its transverse slopes
    static constexpr int kTau = 50;                                      // tau, exp(-dt/tau), 1/gm0
    static constexpr int kSlots = 53;
    double (*slots)[kFluxBlock];

    __device__ __forceinline__ double &at(int i) const { return slots[i][threadIdx.x]; }

    __device__ __forceinline__ void load(const FieldDev &f, unsigned c, unsigned c1, unsigned cn, unsigned cs,
                                         unsigned cf, unsigned cb) const
    {
        const double *rec = f.rec[DIR];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int o = perm<DIR>(q);
            cp_async8(&at(kWL + q), f.W[o] + c);
            cp_async8(&at(kWR + q), f.W[o] + c1);
            cp_async8(&at(kWl + q), rec + 2 * ((o / 2) * f.ncell + c) + o % 2);
            cp_async8(&at(kWr + q), rec + 2 * (((5 + o) / 2) * f.ncell + c) + (5 + o) % 2);
        }
        cp_async_commit();
        double rn[10], rs[10], rf[10], rb[10];
        get_record(rec, cn, rn, f.ncell);
        get_record(rec, cs, rs, f.ncell);
        get_record(rec, cf, rf, f.ncell);
        get_record(rec, cb, rb, f.ncell);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int o = perm<DIR>(q);
            at(kDl + q) = rn[o] - rs[o];
            at(kDl + 5 + q) = rf[o] - rb[o];
            at(kDr + q) = rn[5 + o] - rs[5 + o];
            at(kDr + 5 + q) = rf[5 + o] - rb[5 + o];
        }
        cp_async_wait<0>();
    }
    template <int SIDE> __device__ __forceinline__ void state(double W[5]) const
    {
#pragma unroll
        for (int q = 0; q < 5; ++q) W[q] = at((SIDE ? kWr : kWl) + q);
    }
    // differences of side's state W along d (0 normal, 1 and 2 transverse)
    template <int SIDE, int D> __device__ __forceinline__ void slope(const double W[5], double b[5]) const
    {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            if (D == 0) b[q] = SIDE ? at(kWR + q) - W[q] : W[q] - at(kWL + q);
            else b[q] = at((SIDE ? kDr : kDl) + 5 * (D - 1) + q);
        }
    }
    __device__ __forceinline__ void cells(double WL[5], double WR[5]) const
    {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            WL[q] = at(kWL + q);
            WR[q] = at(kWR + q);
        }
    }
    template <int SIDE> __device__ __forceinline__ void sum(int i, double v) const { at(i) = SIDE ? at(i) + v : v; }
    template <int SIDE> __device__ __forceinline__ void sum(int i, double a, double b) const
    {
        at(i) = SIDE ? fma(a, b, at(i)) : a * b;
    }
    __device__ __forceinline__ double get(int i) const { return at(i); }
    __device__ __forceinline__ void put(int i, double v) const { at(i) = v; }
};

// Mixed path (gks_flux): the left state and its slopes stay in registers.
template <int DIR>
struct SweepSrc {
    double Wl[5];
    float DWl[3][5];
    float (*park_dw)[kFluxBlock];  // [15][block]: right-side slopes
    double (*park_w)[kFluxBlock];  // [15][block]: WL, WR, Wr
    double (*sum_d)[kFluxBlock];   // [10][block]: double sums of the side passes

    // RO: the state is not written by this kernel
    template <bool RO>
    __device__ __forceinline__ void load(const FieldDev &f, unsigned c, unsigned c1, unsigned cn, unsigned cs,
                                         unsigned cf, unsigned cb)
    {
        const int t = threadIdx.x;
        const Records r(f.rec[DIR], c, cn, cs, cf, cb, f.ncell);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int o = perm<DIR>(q);
            const double wL = RO ? __ldg(f.W[o] + c) : f.W[o][c], wR = RO ? __ldg(f.W[o] + c1) : f.W[o][c1];
            const double wr = r.r0[5 + o];
            Wl[q] = r.r0[o];
            DWl[0][q] = float(Wl[q] - wL);
            DWl[1][q] = float(r.rn[o] - r.rs[o]);
            DWl[2][q] = float(r.rf[o] - r.rb[o]);
            park_dw[q][t] = float(wR - wr);
            park_dw[5 + q][t] = float(r.rn[5 + o] - r.rs[5 + o]);
            park_dw[10 + q][t] = float(r.rf[5 + o] - r.rb[5 + o]);
            park_w[q][t] = wL;
            park_w[5 + q][t] = wR;
            park_w[10 + q][t] = wr;
        }
    }

    __device__ __forceinline__ void state(int side, double W[5]) const
    {
#pragma unroll
        for (int q = 0; q < 5; ++q) W[q] = side == 0 ? Wl[q] : park_w[10 + q][threadIdx.x];
    }

    // slopes of one side along one direction (0 normal, 1 and 2 transverse)
    __device__ __forceinline__ void slope(int side, int d, float DW[5]) const
    {
#pragma unroll
        for (int q = 0; q < 5; ++q) DW[q] = side == 0 ? DWl[d][q] : park_dw[5 * d + q][threadIdx.x];
    }

    __device__ __forceinline__ void cells(double WL[5], double WR[5]) const
    {
        const int t = threadIdx.x;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            WL[q] = park_w[q][t];
            WR[q] = park_w[5 + q][t];
        }
    }

    // running sums of a * b: the first side pass stores, the second adds (one
    // explicit rounding each, so that no compiler contraction choice -- which
    // may differ between register-cap variants -- changes the result)
    template <bool FIRST> __device__ __forceinline__ void put_d(int i, double a, double b) const
    {
        double &x = sum_d[i][threadIdx.x];
        x = FIRST ? __dmul_rn(a, b) : __fma_rn(a, b, x);
    }
    __device__ __forceinline__ double get_d(int i) const { return sum_d[i][threadIdx.x]; }
};

// The flux of work item `it` of field f; `smem` is the block's parking space.
template <int PREC> struct FluxPark;
template <> struct FluxPark<0> {
    double slots[SweepSrc64<0>::kSlots][kFluxBlock];
};
template <> struct FluxPark<1> {
    double w[15][kFluxBlock], sum[10][kFluxBlock];
    float dw[15][kFluxBlock];
};

// The flux at cell c, components in the state's order.
template <int DIR> __device__ __forceinline__ void unrotate(double F[5])
{
    constexpr int ROT = DIR == 0 ? 0 : (DIR == 1 ? 2 : 3);
    if (ROT) {
        const double t = F[1];
        F[1] = F[ROT];
        F[ROT] = t;
    }
}

template <int DIR> __device__ __forceinline__ void store_flux(const FieldDev &f, unsigned c, const double F[5])
{
#pragma unroll
    for (int q = 0; q < 5; ++q) f.F[DIR * 5 + q][c] = F[q];
}

struct Nothing {
    __device__ __forceinline__ void operator()() const {}
};

// FP64.
template <int DIR, typename Ahead>
__device__ __forceinline__ void flux_item64(const FieldDev &f, unsigned c, const SweepSrc64<DIR> &src, const Ahead &ahead,
                                            double F[5])
{
    const Cell x = decode(c, f);
    unsigned cn, cs, cf, cb;
    transverse<DIR>(x, f.flags, cn, cs, cf, cb);
    src.load(f, c, along<DIR>(x, 1), cn, cs, cf, cb);
    // collision time mu / p at the left cell (update.cpp:262-264), stored by
    // this step's x-sweep reconstruction
    const double tau_n = __ldg(f.tau[0] + c), tau_d = __ldg(f.tau[1] + c);
    const FluxConst64 fc = {f.dt, f.gm1, f.ksn, f.kst, f.kA4, f.prm1, f.kd[0], f.kd[1], f.kd[2], f.kd[3], f.kd[4]};
    gks_flux64(src, tau_n, tau_d, fc, ahead, F);
    unrotate<DIR>(F);
}

// Mixed.
template <int DIR, bool RO>
__device__ __forceinline__ void flux_item(const FieldDev &f, unsigned c, FluxPark<1> &park, double F[5])
{
    const Cell x = decode(c, f);
    unsigned cn, cs, cf, cb;
    transverse<DIR>(x, f.flags, cn, cs, cf, cb);
    SweepSrc<DIR> src;
    src.park_dw = park.dw;
    src.park_w = park.w;
    src.sum_d = park.sum;
    src.template load<RO>(f, c, along<DIR>(x, 1), cn, cs, cf, cb);
    const double tau_n = __ldg(f.tau[0] + c), tau_d = __ldg(f.tau[1] + c);
    FluxConst fc;
    fc.gm1 = f.gm1;
    fc.hig = f.hig;
    fc.dt = f.dt;
    fc.dx = f.dx;
    fc.ks[0] = f.ksn;
    fc.ks[1] = fc.ks[2] = f.kst;
    fc.kA = f.kA;
    fc.hK2 = f.hK2;
    fc.kf = {f.kf[0], f.kf[1], f.kf[2], f.kf[3]};
    gks_flux(src, tau_n, tau_d, fc, F);
    unrotate<DIR>(F);
}

// A batch of one field reads the field's descriptor from the launch
// parameters (b.one: constant-bank operands, nothing loaded per interface);
// an ensemble walks the device array (FieldWalk).
//
// Mixed: grid-stride loop.  FP64: one wave of resident blocks whose warps draw
// chunks of 32 interfaces from a queue: the first is the warp's own number,
// the next ones come from a counter in global memory, asked for one chunk
// ahead.  (With equal static shares the schedulers run some warps ahead of
// others and an SM's last fifth passes at falling occupancy: 9.7 of 12 warps
// active on average, 11.9 with the queue; 1677 -> 1572 us per sweep at 256^3,
// 1543 with a loop of its own for one field and for an ensemble.  The mixed
// kernel gains nothing, 1466 -> 1515 us.)  The warp that is last to find the
// queue empty sets the counters back to zero for the next launch.
template <int DIR, bool ENSEMBLE>
__device__ __forceinline__ void flux_queue(const Batch &b, long long end, const SweepSrc64<DIR> &src)
{
    const int lane = threadIdx.x & 31;
    const unsigned nwarps = gridDim.x * (kFluxBlock / 32);
    const unsigned chunks = unsigned((end - b.lo + 31) >> 5);
    unsigned *queue = b.queue + 2 * DIR;
    unsigned chunk = (blockIdx.x * kFluxBlock + threadIdx.x) >> 5;
    FieldWalk walk(b, b.lo + (long long)chunk * 32, ENSEMBLE);
    while (chunk < chunks) {
        unsigned next = 0;
        if (lane == 0) next = nwarps + atomicAdd(queue, 1u);
        const long long it = b.lo + (long long)chunk * 32 + lane;
        double F[5];
        if (!ENSEMBLE) {
            if (it < end) {
                flux_item64<DIR>(b.one, unsigned(it), src, Nothing(), F);
                store_flux<DIR>(b.one, unsigned(it), F);
            }
        } else {
            const FieldDev &f = walk.at(it);
            if (it - f.base < f.ncell) { // else alignment padding after the field
                flux_item64<DIR>(f, unsigned(it - f.base), src, Nothing(), F);
                store_flux<DIR>(f, unsigned(it - f.base), F);
            }
        }
        chunk = __shfl_sync(0xffffffffu, next, 0);
    }
    if (lane == 0 && atomicAdd(queue + 1, 1u) == nwarps - 1) {
        queue[0] = 0;
        queue[1] = 0;
    }
}

template <int DIR, int PREC, int REGS>
__global__ void __launch_bounds__(kFluxBlock) __maxnreg__(REGS) k_flux(Batch b)
{
    __shared__ FluxPark<PREC> park;
    const long long end = b.nfields == 1 && b.one.ncell < b.hi ? b.one.ncell : b.hi; // alignment padding after the field
    if constexpr (PREC == 0) {
        const SweepSrc64<DIR> src{park.slots};
        if (b.nfields == 1) flux_queue<DIR, false>(b, end, src);
        else flux_queue<DIR, true>(b, end, src);
    } else {
        const long long stride = (long long)gridDim.x * blockDim.x;
        double F[5];
        if (b.nfields == 1) {
            for (long long it = b.lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; it < end; it += stride) {
                flux_item<DIR, true>(b.one, unsigned(it), park, F);
                store_flux<DIR>(b.one, unsigned(it), F);
            }
            return;
        }
        long long it = b.lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
        for (FieldWalk walk(b, it); it < b.hi; it += stride) {
            const FieldDev &f = walk.at(it);
            if (it - f.base >= f.ncell) continue; // alignment padding after the field
            flux_item<DIR, true>(f, unsigned(it - f.base), park, F);
            store_flux<DIR>(f, unsigned(it - f.base), F);
        }
    }
}

// Finite, with positive density and pressure.  The division is left out where
// rho^2 p / (gamma - 1) = rho2p(w) is well above its rounding.
__device__ __forceinline__ bool physical(const double w[5], double gm1)
{
    const double e = w[0] * w[4];
    if (w[0] > 0.0 && rho2p(w) > 1e-8 * e && e > 0.0 && isfinite(w[0] + w[1] + w[2] + w[3] + w[4])) return true;
    const double p = gm1 * (w[4] - 0.5 * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) / w[0]);
    return w[0] > 0.0 && p > 0.0 && isfinite(w[0] + w[1] + w[2] + w[3] + w[4]);
}

// ---------------------------------------------------------------------------
// Conservative update of the interior (update.cpp:455-469), evaluated in the
// reference's order: W - (1/dx)*(Fx - Fx[i-1] + Fy - Fy[j-1] + Fz - Fz[k-1]),
// written to Wout (W itself, except in the slab-pipelined host step).  Also
// flags non-finite or non-positive density / pressure.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kUpdateBlock) k_update(Batch b)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long it = b.lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; it < b.hi; it += stride) {
        const FieldDev &f = b.fields[field_of(b.fields, b.nfields, it)];
        if (it - f.base >= f.ncell) continue; // alignment padding after the field
        const Cell x = decode(unsigned(it - f.base), f);
        const unsigned c = x.c;
        const unsigned cx = along<0>(x, -1), cy = along<1>(x, -1), cz = along<2>(x, -1);
        double w[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            double d = __dsub_rn(f.F[q][c], f.F[q][cx]);
            d = __dadd_rn(d, f.F[5 + q][c]);
            d = __dsub_rn(d, f.F[5 + q][cy]);
            d = __dadd_rn(d, f.F[10 + q][c]);
            d = __dsub_rn(d, f.F[10 + q][cz]);
            w[q] = __dsub_rn(f.W[q][c], __dmul_rn(f.inv_dx, d));
            f.Wout[q][c] = w[q];
        }
        if (!physical(w, f.gm1)) atomicOr(b.err, 1);
    }
}

// ---------------------------------------------------------------------------
// z flux and update of one field in one kernel, in place (or, to be timed, into
// other arrays, Wout).  A warp walks whole z
// lines (drawn from the queue of k_flux), 32 interfaces at a time: a lane's
// lower z flux comes from the lane below by a shuffle, lane 0's from the chunk
// before (park), and the x and y fluxes of its cell arrive by asynchronous
// copies while the equilibrium pass is computed.  The state of a cell is read
// by its own warp only (as left or right cell average), before it is written;
// cell 0, which the line's last interface reads and whose lower flux is that
// interface's, is written last.  The update alone is bound by HBM (200 B a
// cell, 0.50 ms at 256^3); here its traffic, 120 B without the z fluxes, passes
// under the flux's arithmetic.  The arithmetic is that of k_flux and k_update.
// ---------------------------------------------------------------------------
template <int PREC> struct LinePark;
template <> struct LinePark<0> {
    FluxPark<0> flux;
    double line[kFluxBlock / 32][10]; // per warp: z flux below the next chunk; cell 0's sum of flux differences
};
template <> struct LinePark<1> {
    FluxPark<1> flux;
    double xy[20][kFluxBlock];
    double line[kFluxBlock / 32][10];
};

template <int PREC, int REGS>
__global__ void __launch_bounds__(kFluxBlock) __maxnreg__(REGS) k_flux_update(Batch b)
{
    __shared__ LinePark<PREC> park;
    const FieldDev &f = b.one;
    const int t = threadIdx.x, lane = t & 31;
    const int nc = f.nc;
    const unsigned nwarps = gridDim.x * (kFluxBlock / 32), lines = unsigned(f.ncell / nc);
    unsigned *queue = b.queue + 4;
    double *below = park.line[t >> 5], *first = below + 5;
    // slots of the cell's Fx, Fx below, Fy, Fy below: FP64 in those of the inputs
    // behind the left cell average, free once the equilibrium pass has read them
    double (*xy)[kFluxBlock];
    if constexpr (PREC == 0) xy = park.flux.slots + SweepSrc64<2>::kWR;
    else xy = park.xy;
    static_assert(SweepSrc64<2>::kWR == 5 && SweepSrc64<2>::kW0 == 25, "twenty input slots between WL and the sums");
    for (unsigned line = (blockIdx.x * kFluxBlock + t) >> 5; line < lines;) {
        unsigned next = 0;
        if (lane == 0) next = nwarps + atomicAdd(queue, 1u);
        const unsigned lbase = line * unsigned(nc);
        for (int k0 = 0; k0 < nc; k0 += 32) {
            const int k = k0 + lane;
            const unsigned c = lbase + unsigned(min(k, nc - 1)); // lanes past the line repeat its last cell
            auto fetch = [&]() {
                const Cell x = decode(c, f);
                const unsigned cx = along<0>(x, -1), cy = along<1>(x, -1);
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    cp_async8(&xy[q][t], f.F[q] + c);
                    cp_async8(&xy[5 + q][t], f.F[q] + cx);
                    cp_async8(&xy[10 + q][t], f.F[5 + q] + c);
                    cp_async8(&xy[15 + q][t], f.F[5 + q] + cy);
                }
                cp_async_commit();
            };
            double F[5], w[5];
            if constexpr (PREC == 0) {
                const SweepSrc64<2> src{park.flux.slots};
                flux_item64<2>(f, c, src, fetch, F);
#pragma unroll
                for (int q = 0; q < 5; ++q) w[q] = src.at(SweepSrc64<2>::kWL + perm<2>(q));
            } else {
                fetch();
                flux_item<2, false>(f, c, park.flux, F);
#pragma unroll
                for (int q = 0; q < 5; ++q) w[q] = park.flux.w[perm<2>(q)][t];
            }
            cp_async_wait<0>();
            const int last = min(31, nc - 1 - k0); // the lane whose z flux the next chunk (or cell 0) takes
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                double d = __dsub_rn(xy[q][t], xy[5 + q][t]);
                d = __dadd_rn(d, xy[10 + q][t]);
                d = __dsub_rn(d, xy[15 + q][t]);
                d = __dadd_rn(d, F[q]);
                const double up = __shfl_sync(0xffffffffu, F[q], lane ? lane - 1 : last);
                const double lo = lane ? up : below[q];
                if (lane == 0) below[q] = up;
                if (k == 0) {
                    first[q] = d;
                } else if (k < nc) {
                    w[q] = __dsub_rn(w[q], __dmul_rn(f.inv_dx, __dsub_rn(d, lo)));
                    f.Wout[q][c] = w[q];
                }
            }
            if (k > 0 && k < nc) bad = !physical(w, f.gm1);
            if (bad) atomicOr(b.err, 1);
        }
        if (lane == 0) {
            double w[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                w[q] = __dsub_rn(f.W[q][lbase], __dmul_rn(f.inv_dx, __dsub_rn(first[q], below[q])));
                f.Wout[q][lbase] = w[q];
            }
            if (!physical(w, f.gm1)) atomicOr(b.err, 1);
        }
        line = __shfl_sync(0xffffffffu, next, 0);
    }
    if (lane == 0 && atomicAdd(queue + 1, 1u) == nwarps - 1) {
        queue[0] = 0;
        queue[1] = 0;
    }
}

// ---------------------------------------------------------------------------
// Layout conversion: padded staging (5 x nt^3) <-> interior.
// ---------------------------------------------------------------------------
__global__ void k_gather(FieldDev f, const double *__restrict__ stage, long long lo, long long hi)
{
    const int nc = f.nc, nt = nc + 6;
    const long long Nt = (long long)(f.ny + 2 * f.yhost) * nt * nt;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long c = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < hi; c += stride) {
        const Cell x = decode(unsigned(c), f);
        const long long p = ((long long)(x.j + f.yhost) * nt + (x.i + 3)) * nt + (x.k + 3);
#pragma unroll
        for (int q = 0; q < 5; ++q) f.W[q][c] = stage[q * Nt + p];
    }
}

__global__ void k_scatter(FieldDev f, double *__restrict__ stage, long long lo, long long hi)
{
    const int nc = f.nc, nt = nc + 6;
    const long long Nt = (long long)(f.ny + 2 * f.yhost) * nt * nt;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long p = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; p < hi; p += stride) {
        const int kk = int(p % nt);
        const int ii = int((p / nt) % nt);
        const int jj = int(p / ((long long)nt * nt));
        const long long c = ((long long)wrap(jj - f.yhost, f.nyw) * nc + wrap(ii - 3, nc)) * nc + wrap(kk - 3, nc);
#pragma unroll
        for (int q = 0; q < 5; ++q) stage[q * Nt + p] = f.W[q][c];
    }
}

// ---------------------------------------------------------------------------
// Largest |u| + c (timestep, update.cpp:1057-1079), each operation rounded as
// the reference writes it so that dt matches bit for bit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__global__ void k_maxwave(FieldDev f, unsigned long long *out)
{
    double m = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long plane = (long long)f.nc * f.nc, c1 = f.yhi * plane;
    for (long long c = f.ylo * plane + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < c1; c += stride) {
        const double den = f.W[0][c];
        const double u = __ddiv_rn(f.W[1][c], den), v = __ddiv_rn(f.W[2][c], den), w = __ddiv_rn(f.W[3][c], den);
        const double vsq = __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w));
        const double P = __dmul_rn(__dmul_rn(den, f.gm1), __dsub_rn(__ddiv_rn(f.W[4][c], den), __dmul_rn(0.5, vsq)));
        const double val = __dadd_rn(__dsqrt_rn(vsq), __dsqrt_rn(__ddiv_rn(__dmul_rn(f.gam, P), den)));
        m = val > m ? val : m;
    }
    m = warp_max(m);
    __shared__ double sm[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sm[wid] = m;
    __syncthreads();
    if (wid == 0) {
        m = lane < (blockDim.x >> 5) ? sm[lane] : 0.0;
        m = warp_max(m);
        if (lane == 0 && m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
    }
}

// ---------------------------------------------------------------------------
// Statistics (PrintStats, update.cpp:638-784).  Velocity gradients are the
// node slopes of the natural cubic spline through each padded grid line
// (nt = nc + 6 points, periodic ghosts), the interpolant the reference builds
// with einspline (Interpolation.cpp:3-31); at nodes a tensor-product natural
// spline reduces to these 1-D slopes.  Scratch layout: [3*comp + axis]
// d(comp)/d(axis), axis 0 = y, 1 = x (those along z are not stored).
// ---------------------------------------------------------------------------

// Slopes of the natural cubic spline through the nt = nc + 6 nodes of a
// padded periodic grid line (the reference's einspline over its padded
// block):
//   2 m0 + m1 = s (f1 - f0);  m_{p-1} + 4 m_p + m_{p+1} = s (f_{p+1} - f_{p-1});
//   m_{n-2} + 2 m_{n-1} = s (f_{n-1} - f_{n-2}),  s = 3/h,
// solved by the Thomas recurrences with precomputed pivots,
//   forward  d_p = (r_p - d_{p-1}) inv_p,   backward  m_p = d_p - cp_p m_{p+1}.
// A block takes LW lines at a time: its threads load rho and the momenta of
// their nodes and stage the velocities in shared memory, one thread per line
// and component runs the recurrences in place (24 cycles of dependent FP64 a
// node), and the slopes leave through the same tiles:
//   y, x lines: LW consecutive k of one (i) / (j): tiles [node][line], every
//               group of LW threads one contiguous run of LW doubles;
//   z lines:    LW consecutive (j, i) lines:      tiles [line][node], the
//               pitch odd so that the lines' threads use distinct banks.
// LW is chosen so that two blocks fit an SM (spline_lines).
constexpr int kSplineBlock = 256, kStage = 4; // threads; nodes a thread loads at a time

// The line f_p at c[p S], p = 0 .. nt-1, replaced by its slopes.  Nodes move in
// groups whose data and pivots are loaded before the group's stores, which the
// compiler could not move loads across.
constexpr int kSplineGroup = 8;
template <int S> __device__ __forceinline__ void spline_slopes(double *c, int nt, double s, const double *inv, const double *cp)
{
    constexpr int G = kSplineGroup;
    double prev = c[0], cur = c[S];
    double d = (s * (cur - prev)) * inv[0];
    c[0] = d;
    int p = 1;
    for (; p + G <= nt - 1; p += G) {
        double f[G], iv[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            f[g] = c[(p + 1 + g) * S];
            iv[g] = inv[p + g];
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const double next = f[g];
            f[g] = d = fma(s, next - prev, -d) * iv[g];
            prev = cur;
            cur = next;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) c[(p + g) * S] = f[g];
    }
    for (; p < nt - 1; ++p) {
        const double next = c[(p + 1) * S];
        d = fma(s, next - prev, -d) * inv[p];
        c[p * S] = d;
        prev = cur;
        cur = next;
    }
    double m = fma(s, cur - prev, -d) * inv[nt - 1];
    c[(nt - 1) * S] = m;
    p = nt - 2;
    for (; p - G + 1 >= 0; p -= G) {
        double f[G], cc[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            f[g] = c[(p - g) * S];
            cc[g] = cp[p - g];
        }
#pragma unroll
        for (int g = 0; g < G; ++g) f[g] = m = fma(-cc[g], m, f[g]);
#pragma unroll
        for (int g = 0; g < G; ++g) c[(p - g) * S] = f[g];
    }
    for (; p >= 0; --p) {
        m = fma(-cp[p], m, c[p * S]);
        c[p * S] = m;
    }
}

constexpr int NSUM1 = kStatsSums;
static_assert(NSUM1 * (kSplineBlock / 32) * sizeof(double) <= spline_bytes(2, 8, 10),
              "the block sums fit the tiles of the shortest lines");

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sm: N doubles per warp of shared memory that nothing else uses any more.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double *sm, double *out)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const double x = warp_sum(v[i]);
        if (lane == 0) sm[i * nw + wid] = x;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double t = 0.0;
        for (int w = 0; w < nw; ++w) t += sm[threadIdx.x * nw + w];
        out[threadIdx.x] = t;
    }
}

// Primitive state of a cell (c2p, update.cpp:882-891) with one reciprocal of
// the density; ri = 1/rho.
__device__ __forceinline__ void cell_prim(const FieldDev &f, long long c, double &den, double &ri, double &u,
                                          double &v, double &w, double &P, double &T)
{
    den = f.W[0][c];
    ri = __drcp_rn(den);
    u = f.W[1][c] * ri;
    v = f.W[2][c] * ri;
    w = f.W[3][c] * ri;
    const double vsq = fma(u, u, fma(v, v, w * w));
    P = (den * f.gm1) * fma(-0.5, vsq, f.W[4][c] * ri);
    T = P * ri * f.iR;
}

// A cell's terms of the means PrintStats forms (update.cpp:659-712) and, for
// the rms of p, T and 1/rho (update.cpp:751-762), of the first two moments of x
// - K with K the value at the first interior cell (shifted one-pass variance,
// well conditioned because K lies inside the field's range).  g: d(u, v, w)/dy,
// then /dx, then /dz.
__device__ __forceinline__ void add_sums(const FieldDev &f, long long c, const double (&g)[9], double Kp, double Kt, double Kv,
                                         double (&acc)[NSUM1])
{
    double den, ri, u, v, w, P, T;
    cell_prim(f, c, den, ri, u, v, w, P, T);
    const double dudy = g[0], dvdy = g[1], dwdy = g[2], dudx = g[3], dvdx = g[4], dwdx = g[5];
    const double dudz = g[6], dvdz = g[7], dwdz = g[8];
    const double mu = viscosity(f, T);
    acc[0] += den * (u * u + v * v + w * w);
    acc[1] += mu * (dudx * dudx + dudy * dudy + dudz * dudz + dvdx * dvdx + dvdy * dvdy + dvdz * dvdz + dwdx * dwdx +
                    dwdy * dwdy + dwdz * dwdz);
    acc[2] += dudx * dudx + 0.5 * (dudy + dvdx) * (dudy + dvdx) + 0.5 * (dudz + dwdx) * (dudz + dwdx) +
              0.5 * (dwdy + dvdz) * (dwdy + dvdz) + dvdy * dvdy + dwdz * dwdz;
    const double a2 = dudx * dudx, b2 = dvdy * dvdy, c2 = dwdz * dwdz;
    acc[3] += a2; acc[4] += a2 * dudx; acc[5] += a2 * a2;
    acc[6] += b2; acc[7] += b2 * dvdy; acc[8] += b2 * b2;
    acc[9] += c2; acc[10] += c2 * dwdz; acc[11] += c2 * c2;
    acc[12] += P;
    acc[13] += T;
    acc[14] += ri;
    acc[15] += u * u + v * v + w * w;
    acc[16] += sqrt(f.gam * P * ri);
    acc[17] += den;
    const double dP = P - Kp, dT = T - Kt, dV = ri - Kv;
    acc[18] += dP;
    acc[19] += dP * dP;
    acc[20] += dT;
    acc[21] += dT * dT;
    acc[22] += dV;
    acc[23] += dV * dV;
}

// The slopes along one axis.  The y and x passes write theirs to scr; the z
// pass, last, adds every cell's terms straight from its tiles and the six
// slopes before (partial: NSUM1 sums per block; kout: the shifts K), one wave
// of blocks over all sets of lines.  HBM: 56 B a cell and pass for y and x, 88 B
// for z and the sums (3.4 GB at 256^3, 0.51 ms); measured 274 + 269 + 524 us, a
// block's load, solve and store phases only partly covered by the other's.
// Before: a warp per line (affine-map scans, 40 instructions a node) and sums of
// their own, 327 + 317 + 267 + 362 us.  Measured alternatives: 8 lines and 128
// threads at four blocks per SM 329 + 315 + 800, 512 threads 285 + 283 (y, x).
template <int AXIS, int LW>
__global__ void __launch_bounds__(kSplineBlock, 2) k_spline(FieldDev f, double *scr, int nsets, double *partial, double *kout)
{
    constexpr bool SUMS = AXIS == 2;
    constexpr int NG = kSplineBlock / LW;    // y / x: threads on one line
    constexpr int NW = kSplineBlock / 32;    // z: warps
    extern __shared__ double smem[];
    // nodes of a line: nc + 6 along x / z; along y ny + 2 yhost (the same for a
    // periodic field; a slab's ny stored planes, its ghosts included)
    const int nc = f.nc, nt = AXIS == 0 ? f.ny + 2 * f.yhost : nc + 6;
    const long long n = f.ncell;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int pitch = nt | 1, tsz = AXIS == 2 ? LW * pitch : nt * LW;
    double *cpv = smem + 3 * tsz, *invv = cpv + nt;
    // tile of velocity component a, node, line
    auto T = [&](int a, int node, int line) -> double & {
        return AXIS == 2 ? smem[a * tsz + line * pitch + node] : smem[a * tsz + node * LW + line];
    };
    for (int p = tid; p < nt; p += kSplineBlock) {
        cpv[p] = AXIS == 0 ? f.spl_cpy[p] : f.spl_cp[p];
        invv[p] = AXIS == 0 ? f.spl_invy[p] : f.spl_inv[p];
    }
    double acc[SUMS ? NSUM1 : 1];
    double Kp = 0.0, Kt = 0.0, Kv = 0.0;
    if constexpr (SUMS) {
#pragma unroll
        for (int i = 0; i < NSUM1; ++i) acc[i] = 0.0;
        double den, u, v, x;
        cell_prim(f, (long long)f.ylo * nc * nc, den, Kv, u, v, x, Kp, Kt);
        if (blockIdx.x == 0 && tid == 0) {
            kout[0] = Kp;
            kout[1] = Kt;
            kout[2] = Kv;
        }
    }
    const int nkb = (nc + LW - 1) / LW;
    const unsigned step = AXIS == 0 ? unsigned(nc) * nc : (AXIS == 1 ? nc : 1); // cells between positions of a line
    for (int set = blockIdx.x; set < nsets; set += gridDim.x) {
        // the block's lines: y / x lines are (outer, k) with k in [k0, k0 + LW),
        // outer = i (y lines) or j (x lines, interior planes); z lines are l in
        // [l0, l0 + LW), l = j nc + i (interior planes)
        const int outer = AXIS == 2 ? 0 : (AXIS == 1 ? f.ylo : 0) + set / nkb;
        const int k0 = AXIS == 2 ? 0 : (set % nkb) * LW;
        const int l0 = AXIS == 2 ? f.ylo * nc + set * LW : 0;
        const int live = AXIS == 2 ? min(LW, f.yhi * nc - l0) : min(LW, nc - k0); // lines of this set
        auto base = [&](int line) -> unsigned {
            if (AXIS == 0) return unsigned(outer) * nc + k0 + line;
            if (AXIS == 1) return (unsigned(outer) * nc) * nc + k0 + line;
            return unsigned(l0 + line) * nc;
        };
        // this thread's nodes, DP apart: y / x, LW consecutive threads on the LW lines
        // of one node; z, a warp along the nodes of a line, NW lines apart
        constexpr int DP = AXIS == 2 ? 32 : NG;
        for (int line = AXIS == 2 ? w : tid % LW; line < live; line += AXIS == 2 ? NW : LW) {
            const unsigned cb = base(line);
            // velocities at the nodes (node p holds cell wrap(p - 3); along y plane
            // wrap(p - yhost, nyw), a slab's plane p)
            for (int p = AXIS == 2 ? lane : tid / LW; p < nt; p += DP * kStage) {
                double v[kStage][4];
#pragma unroll
                for (int h = 0; h < kStage; ++h) {
                    const int q = p + DP * h;
                    const unsigned c = cb + step * unsigned(AXIS == 0 ? wrap(q - f.yhost, f.nyw) : wrap(q - 3, nc));
#pragma unroll
                    for (int a = 0; a < 4; ++a) v[h][a] = q < nt ? __ldg(f.W[a] + c) : 1.0;
                }
#pragma unroll
                for (int h = 0; h < kStage; ++h) {
                    const int q = p + DP * h;
                    const double ri = __drcp_rn(v[h][0]);
                    if (q < nt)
#pragma unroll
                        for (int a = 0; a < 3; ++a) T(a, q, line) = v[h][a + 1] * ri;
                }
            }
        }
        __syncthreads();
        if (tid < 3 * LW && tid % LW < live)
            spline_slopes<AXIS == 2 ? 1 : LW>(&T(tid / LW, 0, tid % LW), nt, AXIS == 0 ? f.spl_sy : f.spl_s, invv, cpv);
        __syncthreads();
        // slopes of nodes 3 .. nt-4 (the interior cells)
        if constexpr (SUMS) {
            for (int e = tid; e < live * nc; e += kSplineBlock) {
                const int line = e / nc, k = e - line * nc;
                const long long c = (long long)l0 * nc + e;
                double g[9];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    g[a] = __ldg(scr + (3 * a) * n + c);
                    g[3 + a] = __ldg(scr + (3 * a + 1) * n + c);
                    g[6 + a] = T(a, k + 3, line);
                }
                add_sums(f, c, g, Kp, Kt, Kv, acc);
            }
        } else {
            const int line = tid % LW;
            if (line < live)
                for (int p = 3 + tid / LW; p < nt - 3; p += NG) {
                    const unsigned c = base(line) + step * unsigned(AXIS == 0 ? p - f.yhost : p - 3);
#pragma unroll
                    for (int a = 0; a < 3; ++a) scr[(3 * a + AXIS) * n + c] = T(a, p, line);
                }
        }
        __syncthreads();
    }
    if constexpr (SUMS) block_sums<NSUM1>(acc, smem, partial + (long long)blockIdx.x * NSUM1);
}

// Sum the per-block partials, one warp per quantity, in a fixed order (so the
// result does not depend on timing); optionally scaled by 1/ncell.
__global__ void k_finalize(const double *partial, int nblocks, int nsum, double scale, double *out)
{
    const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (i >= nsum) return;
    double t = 0.0;
    for (int bidx = lane; bidx < nblocks; bidx += 32) t += partial[(long long)bidx * nsum + i];
    t = warp_sum(t);
    if (lane == 0) out[i] = t * scale;
}

__global__ void k_check(FieldDev f, int *err)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long plane = (long long)f.nc * f.nc, c1 = f.yhi * plane;
    for (long long c = f.ylo * plane + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < c1; c += stride) {
        double w[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = f.W[q][c];
        const double p = f.gm1 * (w[4] - 0.5 * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) / w[0]);
        if (!(w[0] > 0.0) || !(p > 0.0) || !isfinite(w[0] + w[1] + w[2] + w[3] + w[4])) atomicOr(err, 2);
    }
}

template <typename KernelT>
cudaError_t occ(KernelT k, int block, int *n)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, k, block, 0);
}

// Register-cap variants: reconstruction blocks of 128 threads at 3 / 4 / 5
// resident blocks per SM (launch bounds; 168 / 128 / 96 registers), numbered
// 0-2 and again 3-5 (pinned configurations of either number stay valid); flux
// blocks of 64 threads at explicit caps of 200 / 168 / 128 registers (5 / 6 /
// 8 resident blocks).  A launch bound of 5 blocks of 64 threads would not give
// the 200: the compiler rounds the resident warps up to a multiple of four
// and caps at 168, as for 6 blocks.  The tuner picks one variant per kernel,
// precision and sweep.  Every variant gives bit-identical results.
constexpr int kReconMinb[3] = {3, 4, 5};
constexpr int kFluxRegs[kFluxVariants] = {200, 168, 128};

// The item range of a launch (all items of its kind when b.hi < 0) and the
// blocks it needs: at most cfg.grid, no more than the range fills.
Batch resolve_range(Batch b, int kind, int dir)
{
    if (b.hi < 0) {
        b.lo = 0;
        b.hi = batch_items(b, kind, dir);
    }
    return b;
}

int range_grid(int grid, long long items, int items_per_block)
{
    const long long need = (items + items_per_block - 1) / items_per_block;
    return int(std::max(1LL, std::min((long long)grid, need)));
}

template <int DIR, int PREC>
cudaError_t recon_go(Batch b, LaunchCfg cfg, cudaStream_t st)
{
    b = resolve_range(b, K_RECON, DIR);
    if (b.hi <= b.lo) return cudaSuccess;
    const long long items = b.hi - b.lo;
    if constexpr (DIR < 2) {
        const int g = range_grid(cfg.grid, items, cfg.block);
        switch (cfg.variant % 3) {
        case 1: k_recon_win<DIR, PREC, kReconMinb[1]><<<g, cfg.block, 0, st>>>(b); break;
        case 2: k_recon_win<DIR, PREC, kReconMinb[2]><<<g, cfg.block, 0, st>>>(b); break;
        default: k_recon_win<DIR, PREC, kReconMinb[0]><<<g, cfg.block, 0, st>>>(b); break;
        }
    } else {
        const int g = range_grid(cfg.grid, items, kZLineWarps);
        switch (cfg.variant % 3) {
        case 1: k_recon_zline<PREC, kReconMinb[1]><<<g, cfg.block, 0, st>>>(b); break;
        case 2: k_recon_zline<PREC, kReconMinb[2]><<<g, cfg.block, 0, st>>>(b); break;
        default: k_recon_zline<PREC, kReconMinb[0]><<<g, cfg.block, 0, st>>>(b); break;
        }
    }
    return cudaGetLastError();
}

template <int DIR, int PREC>
cudaError_t flux_go(Batch b, LaunchCfg cfg, cudaStream_t st)
{
    b = resolve_range(b, K_FLUX, DIR);
    if (b.hi <= b.lo) return cudaSuccess;
    const int g = range_grid(cfg.grid, b.hi - b.lo, cfg.block);
    switch (cfg.variant) {
    case 1: k_flux<DIR, PREC, kFluxRegs[1]><<<g, cfg.block, 0, st>>>(b); break;
    case 2: k_flux<DIR, PREC, kFluxRegs[2]><<<g, cfg.block, 0, st>>>(b); break;
    default: k_flux<DIR, PREC, kFluxRegs[0]><<<g, cfg.block, 0, st>>>(b); break;
    }
    return cudaGetLastError();
}

template <int PREC>
cudaError_t flux_update_go(const Batch &b, LaunchCfg cfg, cudaStream_t st)
{
    const int g = range_grid(cfg.grid, b.one.ncell / b.one.nc, cfg.block / 32);
    switch (cfg.variant) {
    case 1: k_flux_update<PREC, kFluxRegs[1]><<<g, cfg.block, 0, st>>>(b); break;
    case 2: k_flux_update<PREC, kFluxRegs[2]><<<g, cfg.block, 0, st>>>(b); break;
    default: k_flux_update<PREC, kFluxRegs[0]><<<g, cfg.block, 0, st>>>(b); break;
    }
    return cudaGetLastError();
}

template <int PREC>
cudaError_t occ_flux_update(int variant, int block, int *n)
{
    if (variant == 1) return occ(k_flux_update<PREC, kFluxRegs[1]>, block, n);
    if (variant == 2) return occ(k_flux_update<PREC, kFluxRegs[2]>, block, n);
    return occ(k_flux_update<PREC, kFluxRegs[0]>, block, n);
}

template <int DIR, int PREC>
cudaError_t occ_kind(int kind, int variant, int block, int *n)
{
    if (kind == K_RECON) {
        if constexpr (DIR < 2) {
            if (variant % 3 == 1) return occ(k_recon_win<DIR, PREC, kReconMinb[1]>, block, n);
            if (variant % 3 == 2) return occ(k_recon_win<DIR, PREC, kReconMinb[2]>, block, n);
            return occ(k_recon_win<DIR, PREC, kReconMinb[0]>, block, n);
        } else {
            if (variant % 3 == 1) return occ(k_recon_zline<PREC, kReconMinb[1]>, block, n);
            if (variant % 3 == 2) return occ(k_recon_zline<PREC, kReconMinb[2]>, block, n);
            return occ(k_recon_zline<PREC, kReconMinb[0]>, block, n);
        }
    }
    if (variant == 1) return occ(k_flux<DIR, PREC, kFluxRegs[1]>, block, n);
    if (variant == 2) return occ(k_flux<DIR, PREC, kFluxRegs[2]>, block, n);
    return occ(k_flux<DIR, PREC, kFluxRegs[0]>, block, n);
}

template <int PREC>
cudaError_t occ_dir(int kind, int dir, int variant, int block, int *n)
{
    return dir == 0 ? occ_kind<0, PREC>(kind, variant, block, n)
                    : dir == 1 ? occ_kind<1, PREC>(kind, variant, block, n) : occ_kind<2, PREC>(kind, variant, block, n);
}

} // namespace

cudaError_t launch_recon(const Batch &b, int dir, int prec, LaunchCfg cfg, cudaStream_t st)
{
    if (prec == 0) return dir == 0 ? recon_go<0, 0>(b, cfg, st) : dir == 1 ? recon_go<1, 0>(b, cfg, st) : recon_go<2, 0>(b, cfg, st);
    return dir == 0 ? recon_go<0, 1>(b, cfg, st) : dir == 1 ? recon_go<1, 1>(b, cfg, st) : recon_go<2, 1>(b, cfg, st);
}

cudaError_t launch_flux(const Batch &b, int dir, int prec, LaunchCfg cfg, cudaStream_t st)
{
    if (prec == 0) return dir == 0 ? flux_go<0, 0>(b, cfg, st) : dir == 1 ? flux_go<1, 0>(b, cfg, st) : flux_go<2, 0>(b, cfg, st);
    return dir == 0 ? flux_go<0, 1>(b, cfg, st) : dir == 1 ? flux_go<1, 1>(b, cfg, st) : flux_go<2, 1>(b, cfg, st);
}

cudaError_t launch_update(const Batch &batch, LaunchCfg cfg, cudaStream_t st)
{
    const Batch b = resolve_range(batch, K_UPDATE, 0);
    if (b.hi <= b.lo) return cudaSuccess;
    k_update<<<range_grid(cfg.grid, b.hi - b.lo, cfg.block), cfg.block, 0, st>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_flux_update(const Batch &b, int prec, LaunchCfg cfg, cudaStream_t st)
{
    return prec == 0 ? flux_update_go<0>(b, cfg, st) : flux_update_go<1>(b, cfg, st);
}

cudaError_t max_resident_blocks(int kind, int dir, int prec, int variant, int block, bool update, int *n)
{
    if (kind == K_UPDATE) return occ(k_update, block, n);
    if (update) return prec == 0 ? occ_flux_update<0>(variant, block, n) : occ_flux_update<1>(variant, block, n);
    return prec == 0 ? occ_dir<0>(kind, dir, variant, block, n) : occ_dir<1>(kind, dir, variant, block, n);
}

cudaError_t launch_gather(const FieldDev &f, const double *stage, int nsm, cudaStream_t st, long long lo, long long hi)
{
    if (hi < 0) hi = f.ncell;
    if (hi <= lo) return cudaSuccess;
    k_gather<<<helper_grid(hi - lo, 256, nsm), 256, 0, st>>>(f, stage, lo, hi);
    return cudaGetLastError();
}

cudaError_t launch_scatter(const FieldDev &f, double *stage, int nsm, cudaStream_t st, long long lo, long long hi)
{
    const long long nt = f.nc + 6;
    if (hi < 0) hi = (f.ny + 2 * f.yhost) * nt * nt;
    if (hi <= lo) return cudaSuccess;
    k_scatter<<<helper_grid(hi - lo, 256, nsm), 256, 0, st>>>(f, stage, lo, hi);
    return cudaGetLastError();
}

cudaError_t launch_maxwave(const FieldDev &f, unsigned long long *out_bits, int nsm, cudaStream_t st)
{
    k_maxwave<<<helper_grid(f.ncell, 256, nsm), 256, 0, st>>>(f, out_bits);
    return cudaGetLastError();
}

template <int AXIS, int LW>
cudaError_t spline_go(const FieldDev &f, double *scratch, double *partial, double *kout, int max_grid, int *grid, cudaStream_t st)
{
    // the limit belongs to the function, which fields of other sizes launch from
    // other threads: every call sets the same one, that of the longest lines
    constexpr size_t limit = LW == 16 ? kSmemPerSm / 2 - kSmemPerBlock : spline_bytes(AXIS, LW, kSplineNtMax);
    const size_t bytes = spline_bytes(AXIS, LW, f.nc + 6);
    cudaError_t e = cudaFuncSetAttribute(k_spline<AXIS, LW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
    if (e != cudaSuccess) return e;
    // lines: y lines (i, k) of the whole slab, x and z lines of the interior planes
    const int ny = f.yhi - f.ylo;
    const int sets = AXIS == 2 ? (ny * f.nc + LW - 1) / LW : (AXIS == 0 ? f.nc : ny) * ((f.nc + LW - 1) / LW);
    *grid = std::min(sets, max_grid);
    k_spline<AXIS, LW><<<*grid, kSplineBlock, bytes, st>>>(f, scratch, sets, partial, kout);
    return cudaGetLastError();
}

template <int AXIS>
cudaError_t spline_axis(const FieldDev &f, double *scratch, double *partial, double *kout, int max_grid, int *grid,
                        cudaStream_t st)
{
    if (spline_lines(AXIS, f.nc + 6) == 16) return spline_go<AXIS, 16>(f, scratch, partial, kout, max_grid, grid, st);
    return spline_go<AXIS, 8>(f, scratch, partial, kout, max_grid, grid, st);
}

cudaError_t launch_stats(const FieldDev &f, double *scratch, double *partial, double *sums, int nsm, cudaStream_t st)
{
    int grid = 0;
    cudaError_t e = spline_axis<0>(f, scratch, nullptr, nullptr, INT_MAX, &grid, st);
    if (e == cudaSuccess) e = spline_axis<1>(f, scratch, nullptr, nullptr, INT_MAX, &grid, st);
    // partial holds stats_partial_elems(nsm) >= kStatsSums * stats_grid
    const int wave = std::min(2 * nsm, stats_grid(f.ncell, kSplineBlock, nsm));
    if (e == cudaSuccess) e = spline_axis<2>(f, scratch, partial, sums + NSUM1, wave, &grid, st);
    if (e != cudaSuccess) return e;
    const double cells = double(f.yhi - f.ylo) * f.nc * f.nc;
    k_finalize<<<1, 32 * NSUM1, 0, st>>>(partial, grid, NSUM1, 1.0 / cells, sums);
    return cudaGetLastError();
}

cudaError_t launch_check(const FieldDev &f, int *err, int nsm, cudaStream_t st)
{
    k_check<<<helper_grid(f.ncell, 256, nsm), 256, 0, st>>>(f, err);
    return cudaGetLastError();
}

} // namespace gks
