// Launch-size arithmetic shared by the kernels' launchers and the C ABI, and
// the per-context address cache of the zero-allocation entry point.  Plain
// host C++ (no CUDA types), so that the CPU tests compile it on its own and
// check the limits for any SM count.
#pragma once

#include <cstddef>

namespace gks {

// Sums the statistics reduction keeps per block (k_spline's z pass).
constexpr int kStatsSums = 24;
// Blocks per SM of the grid-stride helper kernels (gather, scatter, maxwave,
// check) and of the statistics reduction.
constexpr int kHelperBlocksPerSm = 32;
constexpr int kStatsBlocksPerSm = 8;

// Grid of a grid-stride helper kernel over `items` work items: enough blocks
// for the items, at most kHelperBlocksPerSm per SM, at least one.
inline int helper_grid(long long items, int block, int nsm)
{
    long long g = (items + block - 1) / block;
    const long long cap = (long long)(nsm > 0 ? nsm : 1) * kHelperBlocksPerSm;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

// Grid of the statistics reduction (one partial-sum record per block).
inline int stats_grid(long long ncell, int block, int nsm)
{
    const int g = helper_grid(ncell, block, nsm);
    const int cap = (nsm > 0 ? nsm : 1) * kStatsBlocksPerSm;
    return g < cap ? g : cap;
}

// Doubles of the per-block partial sums the statistics of any field need on
// a device with nsm SMs.
inline size_t stats_partial_elems(int nsm)
{
    return (size_t)(nsm > 0 ? nsm : 1) * kStatsBlocksPerSm * kStatsSums;
}

// Shared memory of an SM, and what each resident block takes of it besides its own.
constexpr size_t kSmemPerSm = 233472, kSmemPerBlock = 1024;

// Longest spline line (nc = 1024).
constexpr int kSplineNtMax = 1024 + 6;

// Shared memory of a block of the statistics' spline passes that holds `lines`
// lines of nt nodes: three tiles of velocity components (the z pass's pitch is
// odd) and the two pivot arrays.
constexpr size_t spline_bytes(int axis, int lines, int nt)
{
    return (3 * (size_t)lines * (axis == 2 ? nt | 1 : nt) + 2 * (size_t)nt) * sizeof(double);
}

// Lines per block: 16 (128 contiguous bytes per row of a y / x tile) where two
// such blocks fit an SM, so that one's lines are solved while the other's are
// moved: up to nt = 289; else 8, of which two fit up to nt = 555 (y, x: 556).
// gks_stats, ps per cell, where a block of the z pass had an SM to itself for its
// lines / as here: 270^3 90.7 / 75.1, 282^3 91.0 / 75.6, 520^3 106.6 / 85.8, 540^3 109.0 /
// 88.5 (256^3: 65; 558^3, one block: 123).
constexpr int spline_lines(int axis, int nt)
{
    return 2 * (spline_bytes(axis, 16, nt) + kSmemPerBlock) <= kSmemPerSm ? 16 : 8;
}

// Device address of a file-scope __device__ array, cached per device and
// re-resolved whenever the device's current context is not the one the cached
// address was resolved in (after cudaDeviceReset the primary context -- and
// with it the module and the array -- is created anew).  ctx_id is the
// context's unique id; resolve(&addr) looks the address up in the current
// context and returns 0 on success.
template <int NDEV> struct ContextAddressCache {
    unsigned long long ctx[NDEV] = {};
    void *addr[NDEV] = {};

    template <typename Resolve> int get(int dev, unsigned long long ctx_id, Resolve &&resolve, void **out)
    {
        if (dev < 0 || dev >= NDEV || !out) return -1;
        if (!addr[dev] || ctx[dev] != ctx_id) {
            void *p = nullptr;
            const int rc = resolve(&p);
            if (rc != 0 || !p) {
                addr[dev] = nullptr;
                return rc != 0 ? rc : -1;
            }
            addr[dev] = p;
            ctx[dev] = ctx_id;
        }
        *out = addr[dev];
        return 0;
    }
};

} // namespace gks
