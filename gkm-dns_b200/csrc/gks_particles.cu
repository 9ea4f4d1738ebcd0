// Lagrangian particles of one periodic field (weno/src/ParticleTrack.cpp,
// update.cpp:1082-1303): spline interpolation of the primitives at every
// particle, the particle step and the particle statistics.
//
// The reference interpolates with einspline's 3-D cubic B-spline under natural
// boundary conditions over the rank's padded block (generateSplines,
// update.cpp:1199-1213; get_bsplinep, Interpolation.cpp:3-31) and evaluates
// value and gradient at each particle (getParticleProp,
// ParticleTrack.cpp:90-97).  Here the same interpolant is built on the device
// from the resident state:
//   * the five primitives (den, u, v, w, p) at the (nc+6)^3 nodes of the padded
//     block -- the ghost nodes as the periodic image -- go straight into the z
//     lines of one coefficient array of (nc+8)^3 nodes with the five fields
//     interleaved per node (node-major, so that the 4 x 4 x 4 block a particle
//     reads is 16 runs of 20 contiguous doubles);
//   * the natural cubic B-spline coefficients, one tridiagonal (1, 4, 1) solve
//     per grid line, along z, then x, then y (the tensor product).  With c_1 =
//     f_0 and c_N = f_{N-1} fixed by the natural end conditions, c_2 .. c_{N-1}
//     come from forward elimination with the host-computed pivots w_2 = 1/4,
//     w_m = 1/(4 - w_{m-1}) and back substitution, then c_0 = 2 c_1 - c_2 and
//     c_{N+1} = 2 c_N - c_{N-1}: k_prims_rows (primitives and z lines) and
//     k_line_cols<AXIS> (x, y lines) up to kLineShort nodes, k_prims_zlines and
//     k_bspline_lines<AXIS> beyond;
//   * k_particle_props: per particle the cell and cubic B-spline weights
//     along each axis, then value and gradient of the five splines from
//     their 4 x 4 x 4 coefficient blocks.
// Every operation is written in the oracle's order and this file is compiled
// without implicit contraction, so results agree with the oracle bit for bit
// except the statistics sums, whose order differs (a deterministic tree).
//
// Particle records: GKS_PREC_FIELDS doubles per particle, field-major (field
// q of particle a at q * n + a, so that a warp's accesses are coalesced):
// position (y, x, z) = the reference's pos[0..2], DEN, U[0..2] = (u, v, w),
// P, and the gradients (d/dy, d/dx, d/dz) of DEN, u, v, w and P.
#include "gks_device.cuh"
#include "gks_kernels.cuh"
#include "../../include/gks_b200.h"

#include <cuda_runtime.h>
#include <algorithm>

namespace gks {

namespace {

constexpr int kPrtBlock = 128;
constexpr int kLineBlock = 128;
constexpr int kSumBlock = 256;
constexpr int kNSum = 6; // TKE, SijSij, DUDX2, DUDX3, DWDZ2, DWDZ3
constexpr int kNF = 5;   // fields interleaved per node: den, u, v, w, p

__device__ __forceinline__ int wrap_nc(int x, int n) { return x < 0 ? x + n : (x >= n ? x - n : x); }

// generateSplines' primitives (update.cpp:1201-1208) of one cell.
__device__ __forceinline__ void cell_prims(const FieldDev &f, double gm1, long long cell, double o[5])
{
    const double den = f.W[0][cell];
    const double u = f.W[1][cell] / den, v = f.W[2][cell] / den, w = f.W[3][cell] / den;
    const double Vsqr = u * u + v * v + w * w;
    o[0] = den;
    o[1] = u;
    o[2] = v;
    o[3] = w;
    o[4] = (den * gm1) * (f.W[4][cell] / den - 0.5 * Vsqr);
}

// Natural cubic B-spline coefficients of one grid line in place:
// c[m * s], m = 1 .. N, hold the data f_{m-1} on entry (N >= 4).
// Both recurrences move through the line in groups of kLineGroup positions,
// the loads of a group issued before the group ahead of it is computed, so
// that a thread keeps kLineGroup loads in flight over its (sequential)
// arithmetic.  Bound: HBM -- the array is read and written twice, 2.1 GB of DRAM
// traffic a pass at 256^3 (part of the second reading comes from L2), 415 us
// (530 x / 457 y with groups of 8 and no loads ahead).  Measured alternatives:
// whole lines in shared memory, one reading and one writing, 422 / 436 us (an
// SM holds 100 such lines, too few for the recurrences); fewer lines at a time,
// so that the second reading hits L2, 1.75 GB but 459 - 500 us.
constexpr int kLineGroup = 16;

__device__ __forceinline__ void bspline_line(int N, double *c, long long s, const double *__restrict__ w)
{
    const double f0 = c[s], fl = c[N * s];
    double v[kLineGroup], nx[kLineGroup], wm[kLineGroup];
    // forward elimination over m = 2 .. N-2 (c_1 = f_0 starts it), then the last
    // row m = N-1; groups of positions m = 2 + kLineGroup i
    auto fetch = [&](int m) {
#pragma unroll
        for (int g = 0; g < kLineGroup; ++g)
            if (m + g <= N - 1) nx[g] = c[(m + g) * s];
    };
    double d = f0;
    fetch(2);
    for (int m = 2; m <= N - 1; m += kLineGroup) {
#pragma unroll
        for (int g = 0; g < kLineGroup; ++g) {
            v[g] = nx[g];
            wm[g] = __ldg(w + min(m + g, N));
        }
        fetch(m + kLineGroup);
        if (m + kLineGroup <= N - 1) {
#pragma unroll
            for (int g = 0; g < kLineGroup; ++g) {
                d = (6.0 * v[g] - d) * wm[g];
                c[(m + g) * s] = d;
            }
        } else {
#pragma unroll
            for (int g = 0; g < kLineGroup; ++g)
                if (m + g <= N - 1) {
                    d = (m + g == N - 1 ? (6.0 * v[g] - fl) - d : 6.0 * v[g] - d) * wm[g];
                    c[(m + g) * s] = d;
                }
        }
    }
    const double cl = d; // c_{N-1}
    double cn = d;
    // back substitution over m = N-2 .. 2
    auto back = [&](int m) {
#pragma unroll
        for (int g = 0; g < kLineGroup; ++g)
            if (m - g >= 2) nx[g] = c[(m - g) * s];
    };
    back(N - 2);
    for (int m = N - 2; m >= 2; m -= kLineGroup) {
#pragma unroll
        for (int g = 0; g < kLineGroup; ++g) {
            v[g] = nx[g];
            wm[g] = __ldg(w + max(m - g, 0));
        }
        back(m - kLineGroup);
#pragma unroll
        for (int g = 0; g < kLineGroup; ++g)
            if (m - g >= 2) {
                cn = v[g] - wm[g] * cn;
                c[(m - g) * s] = cn;
            }
    }
    c[0] = 2.0 * f0 - cn;
    c[(N + 1) * s] = 2.0 * fl - cl;
}

// One pass of line solves over all five fields along AXIS (0 y, 1 x): a
// thread per line and field, consecutive threads on consecutive (k, field),
// so that every access of a warp is one contiguous run; the lines include the
// end coefficients of the passes before (x pass N M lines per field, y pass
// M^2).
template <int AXIS>
__global__ void __launch_bounds__(kLineBlock) k_bspline_lines(double *coef, long long N, const double *w)
{
    static_assert(AXIS == 0 || AXIS == 1, "the z pass is k_prims_zlines");
    const long long M = N + 2;
    const long long L = kNF * (AXIS == 1 ? N * M : M * M);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < L; t += stride) {
        if (AXIS == 1) {
            // t = ((j - 1) M + k) kNF + q: element m of the line at ((j M + m) M + k) kNF + q
            const long long l = t / kNF, q = t - l * kNF, j = 1 + l / M, k = l % M;
            bspline_line(int(N), coef + (j * M * M + k) * kNF + q, M * kNF, w);
        } else {
            // t = (i M + k) kNF + q: element m at ((m M + i) M + k) kNF + q
            bspline_line(int(N), coef + t, M * M * kNF, w);
        }
    }
}

// The primitives and the z pass, whose lines are contiguous: a block takes
// kZRows grid rows (j, i) with their kNF interleaved fields and moves them
// through shared memory in tiles of kZChunk positions -- a row's chunk is one contiguous run
// of kNF kZChunk doubles -- each thread running the recurrences of one row
// and field: the arithmetic of bspline_line, chunk by chunk, forward
// elimination over increasing positions, back substitution and the two end
// coefficients over decreasing ones.  The tile's row pitch (kZPitch = 5 mod
// 16 doubles) keeps a half-warp's accesses, thread t at row t / 5 and field
// t % 5, on distinct banks.
constexpr int kZRows = 32;
constexpr int kZThreads = kNF * kZRows;
constexpr int kZChunk = 32;
constexpr int kZRun = kNF * kZChunk;     // doubles of one row's chunk
constexpr int kZPitch = kZRun + 5;       // 165 = 5 mod 16
constexpr int kZBatch = 16;              // reads of a thread in flight at once

__global__ void __launch_bounds__(kZThreads) k_prims_zlines(FieldDev f, double *coef, long long N,
                                                            const double *__restrict__ w)
{
    __shared__ double tile[kZRows][kZPitch];
    __shared__ double *rbase[kZRows];
    __shared__ long long cbase[kZRows]; // the row's first cell
    const long long M = N + 2, R = N * N;
    const int nc = f.nc, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double gm1 = f.gam - 1;
    const int t = threadIdx.x, r = t / kNF, q = t - r * kNF;
    const long long nchunk = (M + kZChunk - 1) / kZChunk;
    for (long long r0 = (long long)blockIdx.x * kZRows; r0 < R; r0 += (long long)gridDim.x * kZRows) {
        if (t < kZRows) {
            const long long rr = r0 + t; // row (1 + rr / N, 1 + rr % N)
            rbase[t] = rr < R ? coef + ((1 + rr / N) * M + (1 + rr % N)) * M * kNF : nullptr;
            cbase[t] = ((long long)wrap_nc(int(rr / N) - 3, nc) * nc + wrap_nc(int(rr % N) - 3, nc)) * nc;
        }
        __syncthreads();
        const bool mine = rbase[r] != nullptr;
        double f0 = 0.0, fl = 0.0, d = 0.0;
        if (mine) { // the first and last node: the images of cells nc - 3 and 2
            double o[5];
            cell_prims(f, gm1, cbase[r] + nc - 3, o);
            f0 = q == 0 ? o[0] : q == 1 ? o[1] : q == 2 ? o[2] : q == 3 ? o[3] : o[4];
            cell_prims(f, gm1, cbase[r] + 2, o);
            fl = q == 0 ? o[0] : q == 1 ? o[1] : q == 2 ? o[2] : q == 3 ? o[3] : o[4];
        }
        // tile <-> global: each row's chunk [p0, p0 + kZChunk) x fields is one run
        auto move = [&](long long p0, bool load) {
            const long long lim = (M - p0) * kNF; // doubles of the row left from p0
            if (load) {
#pragma unroll
                for (int h = 0; h < kZRows * kZRun / kZThreads; h += kZBatch) {
                    double v[kZBatch];
#pragma unroll
                    for (int b = 0; b < kZBatch; ++b) {
                        const int idx = t + (h + b) * kZThreads, rw = idx / kZRun, e = idx - rw * kZRun;
                        const double *bp = rbase[rw];
                        v[b] = (bp && e < lim) ? bp[p0 * kNF + e] : 0.0;
                    }
#pragma unroll
                    for (int b = 0; b < kZBatch; ++b) {
                        const int idx = t + (h + b) * kZThreads, rw = idx / kZRun, e = idx - rw * kZRun;
                        tile[rw][e] = v[b];
                    }
                }
            } else {
#pragma unroll
                for (int h = 0; h < kZRows * kZRun / kZThreads; ++h) {
                    const int idx = t + h * kZThreads, rw = idx / kZRun, e = idx - rw * kZRun;
                    double *bp = rbase[rw];
                    if (bp && e < lim) bp[p0 * kNF + e] = tile[rw][e];
                }
            }
        };
        for (long long c = 0; c < nchunk; ++c) {
            const long long p0 = c * kZChunk;
            // the primitives of the chunk's nodes, position m holding node m - 1 = cell m - 4
            {
                const int m = int(p0) + lane, k = wrap_nc(m - 4, nc);
                const bool node = m >= 1 && m <= N;
#pragma unroll 4
                for (int rw = wid; rw < kZRows; rw += kZThreads / 32) {
                    double o[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
                    if (node && rbase[rw]) cell_prims(f, gm1, cbase[rw] + k, o);
#pragma unroll
                    for (int a = 0; a < kNF; ++a) tile[rw][lane * kNF + a] = o[a];
                }
            }
            __syncthreads();
            if (mine) {
#pragma unroll
                for (int e = 0; e < kZChunk; ++e) {
                    const long long m = p0 + e;
                    const double x = tile[r][e * kNF + q], wm = __ldg(w + (m < M ? m : M - 1));
                    if (m >= 2 && m <= N - 1) {
                        if (m == 2) d = (6.0 * x - f0) * wm;
                        else if (m < N - 1) d = (6.0 * x - d) * wm;
                        else d = ((6.0 * x - fl) - d) * wm;
                        tile[r][e * kNF + q] = d;
                    }
                }
            }
            __syncthreads();
            move(p0, false);
            __syncthreads();
        }
        const double cl = d; // c_{N-1}
        double cn = d;
        for (long long c = nchunk - 1; c >= 0; --c) {
            const long long p0 = c * kZChunk;
            move(p0, true);
            __syncthreads();
            if (mine) {
#pragma unroll
                for (int e = kZChunk - 1; e >= 0; --e) {
                    const long long m = p0 + e;
                    const double x = tile[r][e * kNF + q], wm = __ldg(w + (m < M ? m : M - 1));
                    if (m == N + 1) {
                        tile[r][e * kNF + q] = 2.0 * fl - cl;
                    } else if (m >= 2 && m <= N - 2) {
                        cn = x - wm * cn;
                        tile[r][e * kNF + q] = cn;
                    } else if (m == 0) {
                        tile[r][e * kNF + q] = 2.0 * f0 - cn; // cn = c_2 here
                    }
                }
            }
            __syncthreads();
            move(p0, false);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Short lines stay in shared memory between their two recurrences, so that a
// pass reads and writes the array once, and an SM holds enough of them (100 of
// 262 nodes, 400 of 64) for the serial recurrences not to be the bound.
// gks_particles_props with few particles, us, this form / the two-pass kernels:
// 16^3 30 / 42, 32^3 35 / 61, 64^3 45 / 86, 96^3 102 / 131, 128^3 254 / 277, 160^3
// 479 / 571, 200^3 1069 / 893.
// ---------------------------------------------------------------------------
constexpr int kLineShort = 176; // nodes

// x (AXIS 1) and y (AXIS 0) lines: a block is one warp, a thread one line and
// field, consecutive threads on consecutive (k, field), so that a row of the
// warp is 256 contiguous bytes.  The forward elimination follows the rows as
// they arrive, kColAhead groups of kColRows rows in flight; the back
// substitution writes its results straight to global memory.
constexpr int kColRows = 16, kColAhead = 5;

template <int AXIS>
__global__ void __launch_bounds__(32) k_line_cols(double *coef, int N, const double *__restrict__ w)
{
    extern __shared__ double tile[]; // row m at 32 (m - 1), m = 1 .. N
    const int lane = threadIdx.x;
    const long long M = N + 2, P = kNF * M;
    const long long L = (AXIS == 1 ? N : M) * P;
    const long long l0 = (long long)blockIdx.x * 32 + lane;
    const bool mine = l0 < L;
    const long long l = mine ? l0 : L - 1;
    // x: line (j, k, field), its elements P apart; y: line (i, k, field), M P apart
    double *c = AXIS == 1 ? coef + (1 + l / P) * (M * P) + l % P : coef + l;
    const long long s = AXIS == 1 ? P : M * P;
    double *col = tile + lane - 32; // element m at col[32 m]
    auto fetch = [&](int g) {
        const int m0 = 1 + g * kColRows;
#pragma unroll
        for (int r = 0; r < kColRows; ++r)
            if (m0 + r <= N) cp_async8(col + 32 * (m0 + r), c + (m0 + r) * s);
        cp_async_commit();
    };
#pragma unroll
    for (int g = 0; g < kColAhead; ++g) fetch(g);
    const double f0 = c[s], fl = c[N * s];
    double d = f0; // d_2 = (6 f_1 - f_0) w_2 is the general step with d_1 = f_0
    const int ng = (N + kColRows - 1) / kColRows;
    for (int g = 0; g < ng; ++g) {
        fetch(g + kColAhead);
        cp_async_wait<kColAhead>();
        const int m0 = 1 + g * kColRows;
        if (g > 0 && m0 + kColRows <= N - 1) {
#pragma unroll
            for (int r = 0; r < kColRows; ++r) {
                d = (6.0 * col[32 * (m0 + r)] - d) * __ldg(w + m0 + r);
                col[32 * (m0 + r)] = d;
            }
        } else {
            for (int m = max(m0, 2); m < min(m0 + kColRows, N); ++m) {
                d = m < N - 1 ? (6.0 * col[32 * m] - d) * __ldg(w + m) : ((6.0 * col[32 * m] - fl) - d) * __ldg(w + m);
                col[32 * m] = d;
            }
        }
    }
    if (!mine) return;
    const double cl = d; // c_{N-1}
    double cn = d;
    c[(N - 1) * s] = cl;
    c[(N + 1) * s] = 2.0 * fl - cl;
    int m = N - 2;
    for (; m - kColRows + 1 >= 2; m -= kColRows) {
#pragma unroll
        for (int r = 0; r < kColRows; ++r) {
            cn = col[32 * (m - r)] - __ldg(w + m - r) * cn;
            c[(m - r) * s] = cn;
        }
    }
    for (; m >= 2; --m) {
        cn = col[32 * m] - __ldg(w + m) * cn;
        c[m * s] = cn;
    }
    c[0] = 2.0 * f0 - cn;
}

// The recurrences of bspline_line on a line in shared memory.
__device__ __forceinline__ void bspline_smem(int N, double *c, const double *__restrict__ w)
{
    const double f0 = c[kNF], fl = c[N * kNF];
    double d = f0;
#pragma unroll 8
    for (int m = 2; m < N - 1; ++m) {
        d = (6.0 * c[m * kNF] - d) * __ldg(w + m);
        c[m * kNF] = d;
    }
    d = ((6.0 * c[(N - 1) * kNF] - fl) - d) * __ldg(w + N - 1);
    c[(N - 1) * kNF] = d;
    double cn = d;
#pragma unroll 8
    for (int m = N - 2; m >= 2; --m) {
        cn = c[m * kNF] - __ldg(w + m) * cn;
        c[m * kNF] = cn;
    }
    c[0] = 2.0 * f0 - cn;
    c[(N + 1) * kNF] = 2.0 * fl - d;
}

// The primitives and the z lines: a block takes kRowRows grid rows (j, i).
// Its warps read the rows' cells and write the nodes' primitives to the rows'
// tiles (five fields interleaved per node, row pitch 5 mod 16 doubles, so that
// thread t at row t / 5 and field t % 5 reads without bank conflicts), 30
// threads run the recurrences, and the rows leave as contiguous runs.
constexpr int kRowRows = 6, kRowThreads = 128;
__host__ __device__ constexpr int row_pitch(int M) { return (kNF * M - kNF + 15) / 16 * 16 + kNF; }

__global__ void __launch_bounds__(kRowThreads) k_prims_rows(FieldDev f, double *coef, const double *__restrict__ w)
{
    extern __shared__ double rows[];
    const int nc = f.nc, N = nc + 6, M = N + 2, pitch = row_pitch(M);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long r0 = (long long)blockIdx.x * kRowRows, R = (long long)N * N;
    const double gm1 = f.gam - 1;
    for (int r = wid; r < kRowRows && r0 + r < R; r += kRowThreads / 32) {
        const int j = int((r0 + r) / N), i = int((r0 + r) % N);
        const long long base = ((long long)wrap_nc(j - 3, nc) * nc + wrap_nc(i - 3, nc)) * nc;
        double *row = rows + r * pitch;
#pragma unroll 2
        for (int k = lane; k < nc; k += 32) {
            double o[5];
            cell_prims(f, gm1, base + k, o);
#pragma unroll
            for (int q = 0; q < kNF; ++q) row[kNF * (k + 4) + q] = o[q]; // node of cell k: m = k + 4
        }
        __syncwarp();
        // ghost nodes m = 1 .. 3 (cells nc-3 .. nc-1) and nc + 4 .. nc + 6 (cells 0 .. 2)
        if (lane < 3 * kNF) {
            row[kNF + lane] = row[kNF * (nc + 1) + lane];
            row[kNF * (nc + 4) + lane] = row[kNF * 4 + lane];
        }
    }
    __syncthreads();
    if (threadIdx.x < kNF * kRowRows && r0 + threadIdx.x / kNF < R)
        bspline_smem(N, rows + (threadIdx.x / kNF) * pitch + threadIdx.x % kNF, w);
    __syncthreads();
    for (int r = 0; r < kRowRows && r0 + r < R; ++r) {
        double *o = coef + ((1 + (r0 + r) / N) * M + (1 + (r0 + r) % N)) * (long long)(kNF * M);
        for (int e = threadIdx.x; e < kNF * M; e += kRowThreads) o[e] = rows[r * pitch + e];
    }
}

// Cell and cubic B-spline weights of position x along one axis of num nodes;
// the cell is clamped to the last interval (as the oracle's).
__device__ __forceinline__ int bspline_cell(double x, double start, double hinv, int num, double *t)
{
    const double u = (x - start) * hinv;
    double fl = floor(u);
    fl = fmin(fmax(fl, 0.0), double(num - 2)); // NaN -> 0: stays inside the arrays
    *t = u - fl;
    return int(fl);
}

__device__ __forceinline__ void bspline_weights(double t, double b[8])
{
    const double s = 1.0 - t, t2 = t * t, t3 = t2 * t;
    b[0] = (s * s * s) / 6.0;
    b[1] = (3.0 * t3 - 6.0 * t2 + 4.0) / 6.0;
    b[2] = (-3.0 * t3 + 3.0 * t2 + 3.0 * t + 1.0) / 6.0;
    b[3] = t3 / 6.0;
    b[4] = -0.5 * (s * s);
    b[5] = 1.5 * t2 - 2.0 * t;
    b[6] = (-1.5 * t2 + t) + 0.5;
    b[7] = 0.5 * t2;
}

// getParticleProp (ParticleTrack.cpp:90-97) of every particle: value and
// gradient of the five splines at its position.  A warp takes six particles,
// lane l the field l % 5 of particle l / 5: the five lanes of a particle read
// its 4 x 4 x 4 block as 16 contiguous runs of 20 doubles, and a thread holds
// seven sums instead of the 35 of a particle.  Lanes 0-2 of a particle form the
// weights of one axis each and hand them over through shared memory.  The sums
// keep the order of a field-by-field evaluation (rows along y, then x, nodes
// along z innermost).  Bound: latency of random reads, 16 rows of 160 B a
// particle (4.3 GB of DRAM traffic for 2^20 particles at 256^3).  Measured there:
// a thread per particle (254 registers, 8 warps per SM) 1.65 ms, this form
// 0.71 ms; visiting the particles tile by tile of the grid 0.88 ms and a sort
// (their records are then scattered).
constexpr int kPropWarps = 4, kPropParticles = 6;

__global__ void __launch_bounds__(32 * kPropWarps) k_particle_props(const double *__restrict__ coef, int nt, double start,
                                                                    double hinv, double *rec, long long n)
{
    __shared__ double weights[kPropWarps][kPropParticles][3][8];
    __shared__ int cells[kPropWarps][kPropParticles][3];
    const long long M = nt + 2;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p = lane / kNF, q = lane - p * kNF;
    const long long groups = (n + kPropParticles - 1) / kPropParticles;
    for (long long g = (long long)blockIdx.x * kPropWarps + wid; g < groups; g += (long long)gridDim.x * kPropWarps) {
        const long long idx = g * kPropParticles + p;
        const bool mine = lane < kNF * kPropParticles && idx < n;
        const long long a = mine ? idx : 0;
        if (mine && q < 3) {
            double t;
            cells[wid][p][q] = bspline_cell(rec[q * n + a], start, hinv, nt, &t);
            bspline_weights(t, weights[wid][p][q]);
        }
        __syncwarp();
        if (mine) {
            const double (*b)[8] = weights[wid][p];
            const int *ic = cells[wid][p];
            const double *c0 = coef + (((long long)ic[0] * M + ic[1]) * M + ic[2]) * kNF + q;
            double bz[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) bz[c] = b[2][c];
            double v = 0.0, gy = 0.0, gx = 0.0, gz = 0.0;
#pragma unroll
            for (int ia = 0; ia < 4; ++ia) {
                double va = 0.0, gxa = 0.0, gza = 0.0;
#pragma unroll
                for (int ib = 0; ib < 4; ++ib) {
                    const double *r = c0 + (ia * M + ib) * M * kNF;
                    const double r0 = __ldg(r), r1 = __ldg(r + kNF), r2 = __ldg(r + 2 * kNF), r3 = __ldg(r + 3 * kNF);
                    const double sv = ((bz[0] * r0 + bz[1] * r1) + bz[2] * r2) + bz[3] * r3;
                    const double sd = ((bz[4] * r0 + bz[5] * r1) + bz[6] * r2) + bz[7] * r3;
                    const double bx = b[1][ib], dbx = b[1][4 + ib];
                    va += bx * sv;
                    gxa += dbx * sv;
                    gza += bx * sd;
                }
                const double by = b[0][ia], dby = b[0][4 + ia];
                v += by * va;
                gy += dby * va;
                gx += by * gxa;
                gz += by * gza;
            }
            rec[(3 + q) * n + a] = v;
            rec[(8 + 3 * q) * n + a] = gy * hinv;
            rec[(9 + 3 * q) * n + a] = gx * hinv;
            rec[(10 + 3 * q) * n + a] = gz * hinv;
        }
        __syncwarp();
    }
}

// Particle::updatePosition (ParticleTrack.cpp:43-65): pos[0] (y) moves with
// U[1] = v, pos[1] (x) with U[0] = u, pos[2] (z) with U[2] = w; each
// coordinate is wrapped once into [0, 2 pi].
__global__ void __launch_bounds__(kPrtBlock) k_particle_track(double *rec, long long n, double dt, double twopi)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += stride) {
        const int vel[3] = {5, 4, 6};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double x = rec[q * n + a];
            x += rec[vel[q] * n + a] * dt;
            if (x > twopi) x = x - twopi;
            if (x < 0) x = twopi + x;
            rec[q * n + a] = x;
        }
    }
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// GetParticleStats' sums (update.cpp:1141-1162): per block, in a fixed order
// (grid-stride per thread, warp tree, warps in order).
__global__ void __launch_bounds__(kSumBlock) k_particle_sums(const double *__restrict__ rec, long long n,
                                                             double *partial)
{
    double acc[kNSum] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += stride) {
        const double U0 = rec[4 * n + a], U1 = rec[5 * n + a], U2 = rec[6 * n + a];
        acc[0] += (U0 * U0 + U1 * U1 + U2 * U2);
        const double dudy = rec[11 * n + a], dudx = rec[12 * n + a], dudz = rec[13 * n + a];
        const double dvdy = rec[14 * n + a], dvdx = rec[15 * n + a], dvdz = rec[16 * n + a];
        const double dwdy = rec[17 * n + a], dwdx = rec[18 * n + a], dwdz = rec[19 * n + a];
        const double s1 = dudy + dvdx, s2 = dudz + dwdx, s3 = dwdy + dvdz;
        acc[1] += (dudx * dudx + 0.5 * (s1 * s1) + 0.5 * (s2 * s2) + 0.5 * (s3 * s3) + dvdy * dvdy + dwdz * dwdz);
        acc[2] += dudx * dudx;
        acc[3] += dudx * dudx * dudx;
        acc[4] += dwdz * dwdz;
        acc[5] += dwdz * dwdz * dwdz;
    }
    __shared__ double sm[kSumBlock / 32][kNSum];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < kNSum; ++s) {
        const double v = warp_sum(acc[s]);
        if (lane == 0) sm[wid][s] = v;
    }
    __syncthreads();
    if (threadIdx.x < kNSum) {
        double v = 0.0;
        for (int w = 0; w < kSumBlock / 32; ++w) v += sm[w][threadIdx.x];
        partial[(long long)blockIdx.x * kNSum + threadIdx.x] = v;
    }
}

// The block sums in a fixed order (one warp per quantity), divided by n.
__global__ void k_particle_final(const double *partial, int nblocks, double nd, double *out)
{
    const int s = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (s >= kNSum) return;
    double v = 0.0;
    for (int b = lane; b < nblocks; b += 32) v += partial[(long long)b * kNSum + s];
    v = warp_sum(v);
    if (lane == 0) out[s] = v / nd;
}

int grid_for(long long items, int block, int nsm, int per_sm)
{
    const long long need = (items + block - 1) / block;
    return int(std::max(1LL, std::min(need, (long long)nsm * per_sm)));
}

} // namespace

int particle_partial_elems(int nsm) { return nsm * 4 * kNSum; }

cudaError_t launch_particle_splines(const FieldDev &f, double *coef, const double *w, int nsm, cudaStream_t st)
{
    const long long nt = f.nc + 6, M = nt + 2;
    if (nt <= kLineShort) {
        // within the 48 KB any kernel may have without asking for more
        static_assert(kRowRows * row_pitch(kLineShort + 2) * sizeof(double) <= 49152 && kLineShort * 32 * sizeof(double) <= 49152,
                      "shared memory of the short lines");
        const size_t rows = (size_t)kRowRows * row_pitch((int)M) * sizeof(double), cols = (size_t)nt * 32 * sizeof(double);
        k_prims_rows<<<(unsigned)((nt * nt + kRowRows - 1) / kRowRows), kRowThreads, rows, st>>>(f, coef, w);
        k_line_cols<1><<<(unsigned)((kNF * nt * M + 31) / 32), 32, cols, st>>>(coef, (int)nt, w);
        k_line_cols<0><<<(unsigned)((kNF * M * M + 31) / 32), 32, cols, st>>>(coef, (int)nt, w);
        return cudaGetLastError();
    }
    // 5 blocks of the z pass fit an SM's shared memory; at 256^3 its rows then make
    // three even rounds (980 us; 4 blocks: 1140)
    k_prims_zlines<<<grid_for(kNF * nt * nt, kZThreads, nsm, 5), kZThreads, 0, st>>>(f, coef, nt, w);
    k_bspline_lines<1><<<grid_for(kNF * nt * M, kLineBlock, nsm, 16), kLineBlock, 0, st>>>(coef, nt, w);
    k_bspline_lines<0><<<grid_for(kNF * M * M, kLineBlock, nsm, 16), kLineBlock, 0, st>>>(coef, nt, w);
    return cudaGetLastError();
}

cudaError_t launch_particle_props(const FieldDev &f, const double *coef, double start, double hinv, double *rec,
                                  long long n, int nsm, cudaStream_t st)
{
    const long long groups = (n + kPropParticles - 1) / kPropParticles;
    k_particle_props<<<grid_for(32 * groups, 32 * kPropWarps, nsm, 16), 32 * kPropWarps, 0, st>>>(coef, f.nc + 6, start, hinv,
                                                                                             rec, n);
    return cudaGetLastError();
}

cudaError_t launch_particle_track(double *rec, long long n, double dt, double twopi, int nsm, cudaStream_t st)
{
    k_particle_track<<<grid_for(n, kPrtBlock, nsm, 16), kPrtBlock, 0, st>>>(rec, n, dt, twopi);
    return cudaGetLastError();
}

cudaError_t launch_particle_stats(const double *rec, long long n, double *partial, double *sums, int nsm,
                                  cudaStream_t st)
{
    const int g = grid_for(n, kSumBlock, nsm, 4);
    k_particle_sums<<<g, kSumBlock, 0, st>>>(rec, n, partial);
    k_particle_final<<<1, 32 * kNSum, 0, st>>>(partial, g, double(n), sums);
    return cudaGetLastError();
}

} // namespace gks
