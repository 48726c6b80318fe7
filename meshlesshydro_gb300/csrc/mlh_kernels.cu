// MFV timestep kernels for GB300 (sm_103a), FP64 state.
//
// One step = the stage sequence of the reference's MeshlessScheme::run
// (jammartin/meshlessHydro, demonstrator/src/MeshlessScheme.cpp:39-253):
//   bounds + grid        Particles::getDomainLimits / Domain::createGrid
//   bin                  Particles::assignParticlesAndCells
//   neighbour search     Particles::gridNNS + ghostNNS (images via wrapped cells)
//   density, pressure    Particles::compDensity / compPressure
//   dt                   Particles::compGlobalTimestep
//   E^-1, gradients,     Particles::compPsijTilde / gradient / slopeLimiter
//   limiter
//   faces                compEffectiveFace + compRiemannStatesLR +
//                        solveRiemannProblems (one thread per canonical face)
//   gather + kick/drift  collectFluxes + updateStateAndPosition
//
// Determinism: no floating-point atomics; each face flux is computed once, from the
// side of the lower particle index, and gathered with sign; densities and flux sums
// run over the neighbour list in the reference's order.  The sums of the least-squares
// matrix and the gradients run in that order with one lane per particle; where few
// particles in all leave the GPU short of warps, 2, 4 or 8 lanes sum every 2nd, 4th or
// 8th neighbour each (grad_lanes, by the particles of the context and the SMs of the
// GPU).  So one context gives the same bits on every run, graph or not, but a member of
// a large ensemble may differ in rounding from the same simulation alone.
#include "mlh_device.cuh"
#include "mlh_riemann.cuh"
#include "mlh_kernels.h"
#include "mlh_mlp.cuh"

#include <cfloat>

namespace mlh {

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ double atomic_min_pos_double(unsigned long long *addr, double v) {
    // positive doubles order like their bit patterns
    return (double)atomicMin(addr, (unsigned long long)__double_as_longlong(v));
}

template <typename T>
__device__ __forceinline__ T warp_reduce_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ------------------------------------------------------------------ scan

// Exclusive scan of int counts in three launches (tile reduce, scan of tile
// sums in one block, tile scan).  Tile = 1024 threads x 4 items.
constexpr int SCAN_T = 1024, SCAN_I = 4, SCAN_TILE = SCAN_T * SCAN_I;

__device__ __forceinline__ int block_exclusive_scan(int v, int *smem, int &total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = (lane < (int)(blockDim.x >> 5)) ? smem[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        smem[lane] = s;
    }
    __syncthreads();
    int base = w > 0 ? smem[w - 1] : 0;
    total = smem[(blockDim.x >> 5) - 1];
    __syncthreads();
    return base + x - v;
}

__global__ void k_scan_reduce(const int *in, int n, int *tile_sums) {
    step_begin();
    __shared__ int smem[32];
    long long base = (long long)blockIdx.x * SCAN_TILE;
    int s = 0;
    for (int k = 0; k < SCAN_I; ++k) {
        long long idx = base + (long long)k * SCAN_T + threadIdx.x;
        if (idx < n) s += in[idx];
    }
    s = warp_reduce_sum(s);
    if ((threadIdx.x & 31) == 0) smem[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        int v = threadIdx.x < (blockDim.x >> 5) ? smem[threadIdx.x] : 0;
        v = warp_reduce_sum(v);
        if (threadIdx.x == 0) tile_sums[blockIdx.x] = v;
    }
}

__global__ void k_scan_tiles(int *tile_sums, int ntiles, int *total_out) {
    step_begin();
    __shared__ int smem[32];
    int carry = 0;
    for (int b = 0; b < ntiles; b += SCAN_T) {
        int idx = b + threadIdx.x;
        int v = idx < ntiles ? tile_sums[idx] : 0;
        int tot;
        int ex = block_exclusive_scan(v, smem, tot);
        if (idx < ntiles) tile_sums[idx] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) *total_out = carry;
}

__global__ void k_scan_apply(const int *in, int n, const int *tile_offsets,
                             int *out, const int *total, int write_total_at_n) {
    step_begin();
    __shared__ int smem[32];
    long long base = (long long)blockIdx.x * SCAN_TILE;
    long long idx0 = base + (long long)threadIdx.x * SCAN_I;
    int v[SCAN_I];
    int loc = 0;
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
        long long idx = idx0 + k;
        v[k] = idx < n ? in[idx] : 0;
        loc += v[k];
    }
    int tot;
    int ex = block_exclusive_scan(loc, smem, tot) + tile_offsets[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
        long long idx = idx0 + k;
        if (idx < n) out[idx] = ex;
        ex += v[k];
    }
    if (write_total_at_n && blockIdx.x == 0 && threadIdx.x == 0) out[n] = *total;
}

// The same in one launch of one block, tile after tile, for few items: three
// dependent launches take about 9 us whatever they do, a tile here about 1.5 us.
__global__ void __launch_bounds__(SCAN_T) k_scan_one(const int *in, int n, int *out,
                                                     int *total) {
    step_begin();
    __shared__ int smem[32];
    int carry = 0;
    for (int b = 0; b < n; b += SCAN_TILE) {
        const int i0 = b + threadIdx.x * SCAN_I;
        int v[SCAN_I], loc = 0, tot;
#pragma unroll
        for (int k = 0; k < SCAN_I; ++k) {
            v[k] = i0 + k < n ? in[i0 + k] : 0;
            loc += v[k];
        }
        int ex = carry + block_exclusive_scan(loc, smem, tot);
#pragma unroll
        for (int k = 0; k < SCAN_I; ++k) {
            if (i0 + k < n) out[i0 + k] = ex;
            ex += v[k];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) { out[n] = carry; *total = carry; }
}

// A kernel whose first statement is step_begin, launched so that its blocks come
// up while its predecessor on the stream still runs: a step of few particles is
// eleven kernels of a few microseconds each, and the gaps between them count.
template <class... P, class... A>
void launch_dep(void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

template <class... P, class... A>
void launch_kernel(bool dep, void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t s, A... args) {
    if (dep) launch_dep(kernel, blocks, threads, smem, s, args...);
    else kernel<<<blocks, threads, smem, s>>>((P)args...);
}

// after_kernel: the operation before it on the stream is a kernel (not an event's wait)
void exclusive_scan(const int *in, int n, int *out, int *tile_buf, int *total, cudaStream_t s, bool after_kernel) {
    if (n <= 4 * SCAN_TILE) {
        launch_kernel(after_kernel, k_scan_one, 1, SCAN_T, 0, s, in, n, out, total);
        return;
    }
    int ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (ntiles < 1) ntiles = 1;
    launch_kernel(after_kernel, k_scan_reduce, ntiles, SCAN_T, 0, s, in, n, tile_buf);
    launch_dep(k_scan_tiles, 1, SCAN_T, 0, s, tile_buf, ntiles, total);
    launch_dep(k_scan_apply, ntiles, SCAN_T, 0, s, in, n, tile_buf, out, total, 1);
}

// ------------------------------------------------------------------ bounds + grid

// Particles::getDomainLimits (Particles.cpp:228-267): lo = min over all
// particles; because of `else if` and numeric_limits<double>::min(), hi = the
// max over i >= 1 of the x_i that are not below the running minimum of
// x_0..x_{i-1}, or DBL_MIN.  The partial pass computes min over all i and max
// over i >= 1 of each simulation's range (blocks_per_member blocks each); the
// final pass falls back to the sequential rule whenever x_0 is above every
// other particle (the only case where the two differ).
constexpr int BOUNDS_T = 256;

// the partial minima and maxima of virtual block vb (block vb % bpm of member
// vb / bpm), for a block of BOUNDS_T threads
template <int D>
__device__ __forceinline__ void bounds_partial_block(int vb, const double *__restrict__ x,
                                                     const double *__restrict__ y, const double *__restrict__ z,
                                                     const Params &p, const Member *__restrict__ members, int bpm,
                                                     double *__restrict__ part) {
    __shared__ double smin[3][BOUNDS_T / 32], smax[3][BOUNDS_T / 32];
    const int mi = vb / bpm, sub = vb % bpm;
    const Member mb = members[mi];
    const double *X[3] = {x, y, z};
    double mn[3], mx[3];
    for (int a = 0; a < 3; ++a) { mn[a] = DBL_MAX_; mx[a] = -DBL_MAX_; }
    if (!p.periodic) {
        const int end = mb.first + mb.count;
        for (int i = mb.first + sub * blockDim.x + threadIdx.x; i < end; i += bpm * blockDim.x) {
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double v = X[a][i];
                mn[a] = fmin(mn[a], v);
                if (i >= mb.first + 1) mx[a] = fmax(mx[a], v);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < D; ++a) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = fmin(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = fmax(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
        if ((threadIdx.x & 31) == 0) { smin[a][threadIdx.x >> 5] = mn[a]; smax[a][threadIdx.x >> 5] = mx[a]; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int a = 0; a < D; ++a) {
            double a0 = DBL_MAX_, a1 = -DBL_MAX_;
            for (int w = 0; w < BOUNDS_T / 32; ++w) { a0 = fmin(a0, smin[a][w]); a1 = fmax(a1, smax[a][w]); }
            part[(vb * 3 + a) * 2 + 0] = a0;
            part[(vb * 3 + a) * 2 + 1] = a1;
        }
    }
    __syncthreads();   // the shared partials are reused by the next virtual block
}

template <int D>
__global__ void k_bounds_partial(const double *x, const double *y,
                                 const double *z, Params p, const Member *__restrict__ members,
                                 int bpm, double *part, int *cellCount,
                                 int *cellFill) {
    step_begin();
    // with the cell counters (a step's binning): cleared here
    if (cellCount)
        for (long long k = blockIdx.x * blockDim.x + threadIdx.x; k <= p.ncells_cap; k += gridDim.x * blockDim.x) {
            cellCount[k] = 0;
            cellFill[k] = 0;
        }
    bounds_partial_block<D>(blockIdx.x, x, y, z, p, members, bpm, part);
}

// Domain::createGrid of one simulation; lo and mx1: the minima and the maxima
// over i >= 1 of an open box's coordinates
template <int D>
__device__ __forceinline__ void bounds_grid(const double *const *X, const Params &p, const Member &mb, const double *lo,
                                            const double *mx1, GridInfo *out, unsigned *status) {
    GridInfo g;
    for (int a = 0; a < 3; ++a) { g.lo[a] = 0.; g.hi[a] = 0.; g.cs[a] = 1.; g.cells[a] = 1; }
    for (int a = 0; a < D; ++a) {
        if (p.periodic) { g.lo[a] = mb.box_lo[a]; g.hi[a] = mb.box_hi[a]; continue; }
        const double x0 = X[a][mb.first];
        double hi;
        if (mb.count < 2 || !(mx1[a] >= x0)) {
            // sequential rule of the reference
            double lo_s = DBL_MAX_, hi_s = DBL_MIN_;
            for (int i = mb.first; i < mb.first + mb.count; ++i) {
                double v = X[a][i];
                if (v < lo_s) lo_s = v;
                else if (v > hi_s) hi_s = v;
            }
            hi = hi_s;
        } else {
            hi = mx1[a] > DBL_MIN_ ? mx1[a] : DBL_MIN_;
        }
        g.lo[a] = lo[a];
        g.hi[a] = hi;
    }
    // the product saturates at ncells_cap + 1 (each factor is below 2^31,
    // so the product of the saturated value and one factor fits in 64 bits)
    long long total = 1;
    for (int a = 0; a < D; ++a) {
        double c = floor((g.hi[a] - g.lo[a]) / mb.h);
        int ci = (c >= 1. && c < 2147483647.) ? (int)c : 1;
        if (!(c >= 1.)) flag(status, ST_GRID);
        if (c >= 2147483647.) { flag(status, ST_CAPACITY); ci = 1; }
        if (p.periodic && ci < 3) flag(status, ST_GRID);
        g.cells[a] = ci;
        total *= ci;
        if (total > p.ncells_cap) total = (long long)p.ncells_cap + 1;
    }
    for (int a = 0; a < D; ++a) g.cs[a] = (g.hi[a] - g.lo[a]) / (double)g.cells[a];
    for (int a = 0; a < 3; ++a) {
        g.band_lo[a] = g.lo[a] + mb.h;
        g.band_hi[a] = g.hi[a] - mb.h;
        g.Lf[a] = (float)(g.hi[a] - g.lo[a]);
    }
    if (total > p.ncells_cap) { flag(status, ST_CAPACITY); total = 1; }
    g.ncells = (int)total;
    g.cell_base = 0;
    *out = g;
}

// Final pass + Domain::createGrid (Domain.cpp:9-54) for every simulation: the
// partials by a warp per simulation (one thread reading 304 of them one after
// another took 145 us of an open 33^3 step), the grid by a thread per
// simulation, then the cell numbering of the concatenated grids.  For periodic
// runs the bounds are the configured box.
// With dtbits, the time step's minima are set to their start too.
template <int D>
__device__ __forceinline__ void bounds_final_block(const double *__restrict__ x, const double *__restrict__ y,
                                                   const double *__restrict__ z, const double *__restrict__ part,
                                                   int bpm, const Params &p, const Member *__restrict__ members,
                                                   int nmembers, GridInfo *__restrict__ grids,
                                                   int *__restrict__ cellTotal, unsigned *__restrict__ status,
                                                   unsigned long long *__restrict__ dtbits,
                                                   unsigned *__restrict__ dtcap) {
    const double *X[3] = {x, y, z};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    __shared__ double lo_s[BOUNDS_T / 8][3], mx_s[BOUNDS_T / 8][3];
    for (int m0 = 0; m0 < nmembers; m0 += BOUNDS_T / 8) {
        const int here = nmembers - m0 < BOUNDS_T / 8 ? nmembers - m0 : BOUNDS_T / 8;
        if (!p.periodic) {
            for (int k = warp; k < here; k += nwarps) {
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    double mn = DBL_MAX_, mx = -DBL_MAX_;
                    for (int b = (m0 + k) * bpm + lane; b < (m0 + k + 1) * bpm; b += 32) {
                        mn = fmin(mn, part[(b * 3 + a) * 2]);
                        mx = fmax(mx, part[(b * 3 + a) * 2 + 1]);
                    }
                    for (int o = 16; o > 0; o >>= 1) {
                        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    }
                    if (lane == 0) { lo_s[k][a] = mn; mx_s[k][a] = mx; }
                }
            }
            __syncthreads();
        }
        if ((int)threadIdx.x < here) {
            const int mi = m0 + threadIdx.x;
            const Member mb = members[mi];
            bounds_grid<D>(X, p, mb, lo_s[threadIdx.x], mx_s[threadIdx.x], grids + mi, status);
        }
        __syncthreads();
    }
    if (dtbits)
        for (int mi = threadIdx.x; mi < nmembers; mi += blockDim.x) {
            dtbits[mi] = ~0ull;
            dtcap[mi] = 0x7f7f7f7fu;   // 3.4e38
        }
    __syncthreads();
    // the cell numbering, in shared memory: a simulation that does not fit keeps no
    // cells (the step is then repeated with more)
    __shared__ int nc_s[BOUNDS_T], base_s[BOUNDS_T];
    __shared__ long long next;
    if (threadIdx.x == 0) next = 0;
    for (int m0 = 0; m0 < nmembers; m0 += BOUNDS_T) {
        const int here = nmembers - m0 < BOUNDS_T ? nmembers - m0 : BOUNDS_T;
        const int mi = m0 + threadIdx.x;
        if ((int)threadIdx.x < here) nc_s[threadIdx.x] = grids[mi].ncells;
        __syncthreads();
        if (threadIdx.x == 0) {
            long long base = next;
            for (int k = 0; k < here; ++k) {
                int nc = nc_s[k];
                if (base + nc > p.ncells_cap) { flag(status, ST_CAPACITY); nc = 0; }
                nc_s[k] = nc;
                base_s[k] = (int)base;
                base += nc;
            }
            next = base;
        }
        __syncthreads();
        if ((int)threadIdx.x < here) { grids[mi].ncells = nc_s[threadIdx.x]; grids[mi].cell_base = base_s[threadIdx.x]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) *cellTotal = (int)next;
}

template <int D>
__global__ void k_bounds_final(const double *x, const double *y,
                               const double *z, const double *part, int bpm, Params p,
                               const Member *__restrict__ members, int nmembers, GridInfo *grids,
                               int *cellTotal, unsigned *status,
                               unsigned long long *dtbits, unsigned *dtcap) {
    step_begin();
    bounds_final_block<D>(x, y, z, part, bpm, p, members, nmembers, grids, cellTotal, status, dtbits, dtcap);
}

// Particles::assignParticlesAndCells (Particles.cpp:270-322).
template <int D>
__device__ __forceinline__ void assign_one(int i, const double *__restrict__ x, const double *__restrict__ y,
                                           const double *__restrict__ z, const int *__restrict__ memberOf,
                                           const GridInfo *__restrict__ grids, int *__restrict__ cell,
                                           int *__restrict__ cellCount, unsigned *__restrict__ status) {
    const double *X[3] = {x, y, z};
    {
        const GridInfo g = grids[memberOf ? memberOf[i] : 0];
        int fl[3] = {0, 0, 0};
        bool bad = false;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double f = floor((X[a][i] - g.lo[a]) / g.cs[a]);
            int fi = (f > -1e9 && f < 1e9) ? (int)f : -1;
            if (fi == g.cells[a]) fi -= 1;
            if (fi < 0 || fi >= g.cells[a]) { bad = true; fi = fi < 0 ? 0 : g.cells[a] - 1; }
            fl[a] = fi;
        }
        if (bad) flag(status, ST_GRID);
        int c = fl[0] + fl[1] * g.cells[0] + (D == 3 ? fl[2] * g.cells[0] * g.cells[1] : 0);
        if (c >= g.ncells) { c = g.ncells > 0 ? g.ncells - 1 : 0; flag(status, ST_GRID); }
        c += g.cell_base;
        cell[i] = c;
        atomicAdd(&cellCount[c], 1);
    }
}

template <int D>
__global__ void k_assign(const double *x, const double *y, const double *z,
                         int n, const int *__restrict__ memberOf, const GridInfo *grids,
                         int *cell, int *cellCount, unsigned *status) {
    step_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        assign_one<D>(i, x, y, z, memberOf, grids, cell, cellCount, status);
}

__global__ void k_fill_cells(const int *cell, int n, const int *cellStart,
                             int *cellFill, int *cellList,
                             const unsigned *status) {
    step_begin();
    if (step_aborted(status)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int c = cell[i];
        int pos = atomicAdd(&cellFill[c], 1);
        cellList[cellStart[c] + pos] = i;
    }
}

// Members of a cell in ascending particle index: the order in which
// assignParticlesAndCells pushes them (Particles.cpp:319).
__device__ __forceinline__ void sort_cell(int c, const int *__restrict__ cellStart, int *__restrict__ cellList) {
    int b = cellStart[c], e = cellStart[c + 1];
    for (int k = b + 1; k < e; ++k) {
        int v = cellList[k];
        int t = k - 1;
        while (t >= b && cellList[t] > v) { cellList[t + 1] = cellList[t]; --t; }
        cellList[t + 1] = v;
    }
}

// The same by a warp: up to 64 members on the lanes, each written at its rank (a
// thread's insertion sort is one chain of dependent accesses: 33 us for the 10
// members per cell of an open 33^3 step); larger cells by the first lane.
__device__ __forceinline__ void sort_cell_warp(int c, const int *__restrict__ cellStart, int *__restrict__ cellList) {
    const int lane = threadIdx.x & 31;
    const int b = cellStart[c], n = cellStart[c + 1] - b;
    if (n < 2) return;
    if (n > 64) {
        if (lane == 0) sort_cell(c, cellStart, cellList);
        return;
    }
    const int v0 = lane < n ? cellList[b + lane] : 0x7fffffff, v1 = lane + 32 < n ? cellList[b + lane + 32] : 0x7fffffff;
    int r0 = 0, r1 = 0;
    for (int k = 0; k < n; ++k) {
        const int w = __shfl_sync(0xffffffffu, k < 32 ? v0 : v1, k & 31);
        r0 += w < v0;
        r1 += w < v1;
    }
    __syncwarp();
    if (lane < n) cellList[b + r0] = v0;
    if (lane + 32 < n) cellList[b + r1] = v1;
}

// Cells 0 .. nc - 1 over nw warps, this one the w-th: one at a time while there are no
// more cells than warps, else up to 32 together, their counts on the lanes, and only
// those with an order to make one after another.  (The grid of an open box with a
// particle that left it is nearly empty: 34 million cells, 36 thousand particles:
// 2156 us for the binning with a warp per cell, 1390 with a thread per cell, 603 so.)
__device__ __forceinline__ void sort_cells(int w, int nw, int nc, const int *__restrict__ cellStart,
                                           int *__restrict__ cellList) {
    const int lane = threadIdx.x & 31;
    const int each = (nc + nw - 1) / nw < 32 ? (nc + nw - 1) / nw : 32;
    for (long long c0 = (long long)w * each; c0 < nc; c0 += (long long)nw * each) {
        const long long c = c0 + lane;
        const bool several = lane < each && c < nc && cellStart[c + 1] - cellStart[c] > 1;
        for (unsigned todo = __ballot_sync(0xffffffffu, several); todo; todo &= todo - 1u)
            sort_cell_warp((int)c0 + __ffs((int)todo) - 1, cellStart, cellList);
    }
}

__global__ void __launch_bounds__(256) k_sort_cells(const int *cellTotal,
                                                    const int *cellStart, int *cellList,
                                                    const unsigned *status) {
    step_begin();
    if (step_aborted(status)) return;
    sort_cells((blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5, *cellTotal, cellStart, cellList);
}

// ------------------------------------------------------------------ persistent binning

// The binning of a step (bounds, grid, assignment, cell counts, their scan,
// cell lists, in-cell order) as one persistent kernel: a cooperative launch of
// at most the blocks the GPU holds at once, its phases separated by grid
// barriers.  Results are those of the launch-per-phase sequence (integer and
// min/max work, the cell lists sorted).
//
// Grid barrier: arrivals counted in bar.count, phases in bar.gen; the last
// block to arrive resets the count and opens the next phase.  Every wait is
// bounded: after bar.spin_limit polls (each followed by a short sleep) the
// block sets ST_TIMEOUT and leaves the kernel, and so does every other block
// (a block that left does not arrive again, so the others run out too).  The
// step's later kernels that read the binning skip their work when ST_TIMEOUT
// is set, so that a step which timed out leaves the state untouched.
struct GridBar {
    unsigned *count;
    unsigned *gen;
    unsigned expected;     // blocks that arrive at each barrier
    unsigned spin_limit;   // polls before giving up
};

__device__ __forceinline__ bool grid_sync(const GridBar &b, unsigned *status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        __threadfence();
        const unsigned g = *(volatile unsigned *)b.gen;
        const unsigned prev = atomicAdd(b.count, 1u);
        if (prev + 1 == b.expected) {
            atomicExch(b.count, 0u);
            __threadfence();
            atomicAdd(b.gen, 1u);
        } else {
            unsigned polls = 0;
            while (*(volatile unsigned *)b.gen == g) {
                if (++polls > b.spin_limit) {
                    good = 0;
                    flag(status, ST_TIMEOUT);
                    break;
                }
                __nanosleep(256);
            }
        }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

constexpr int PB_T = 256;                    // threads per block of k_binning
constexpr int PB_ITEMS = SCAN_TILE / PB_T;   // scan items per thread (a tile of SCAN_TILE counts)

template <int D>
__global__ void __launch_bounds__(PB_T) k_binning(const double *__restrict__ x, const double *__restrict__ y,
                                                  const double *__restrict__ z, Params p,
                                                  const Member *__restrict__ members, const int *__restrict__ memberOf,
                                                  int nmembers, int bpm, double *__restrict__ part,
                                                  GridInfo *__restrict__ grids, int *__restrict__ cellTotal,
                                                  int *__restrict__ cell, int *__restrict__ cellCount,
                                                  int *__restrict__ cellStart, int *__restrict__ cellFill,
                                                  int *__restrict__ cellList, int *__restrict__ tileSums,
                                                  int *__restrict__ scanTotal, unsigned *__restrict__ status,
                                                  unsigned long long *__restrict__ dtbits,
                                                  unsigned *__restrict__ dtcap, GridBar bar) {
    __shared__ int smem[32];
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
    const int ncap = p.ncells_cap;
    const int ntiles = (ncap + SCAN_TILE - 1) / SCAN_TILE;
    // 1: partial bounds of every member; clear the cell counters
    for (int vb = blockIdx.x; vb < nmembers * bpm; vb += gridDim.x)
        bounds_partial_block<D>(vb, x, y, z, p, members, bpm, part);
    for (long long k = tid; k <= ncap; k += nthr) { cellCount[k] = 0; cellFill[k] = 0; }
    if (!grid_sync(bar, status)) return;
    // 2: final bounds and Domain::createGrid (one block)
    if (blockIdx.x == 0) bounds_final_block<D>(x, y, z, part, bpm, p, members, nmembers, grids, cellTotal, status, dtbits, dtcap);
    if (!grid_sync(bar, status)) return;
    // 3: Particles::assignParticlesAndCells and the cell counts
    for (int i = tid; i < p.n; i += nthr) assign_one<D>(i, x, y, z, memberOf, grids, cell, cellCount, status);
    if (!grid_sync(bar, status)) return;
    // the same decision in every block: the bits were set before the barrier
    if (step_aborted(status)) return;
    // 4: exclusive scan of the counts: tile sums, their scan, the tiles
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long b0 = (long long)t * SCAN_TILE + (long long)threadIdx.x * PB_ITEMS;
        int sum = 0;
#pragma unroll 4
        for (int k = 0; k < PB_ITEMS; ++k) sum += b0 + k < ncap ? cellCount[b0 + k] : 0;
        int tot;
        (void)block_exclusive_scan(sum, smem, tot);
        if (threadIdx.x == 0) tileSums[t] = tot;
    }
    if (!grid_sync(bar, status)) return;
    if (blockIdx.x == 0) {
        int carry = 0;
        for (int b = 0; b < ntiles; b += PB_T) {
            const int idx = b + threadIdx.x;
            const int v = idx < ntiles ? tileSums[idx] : 0;
            int tot;
            const int ex = block_exclusive_scan(v, smem, tot);
            if (idx < ntiles) tileSums[idx] = carry + ex;
            carry += tot;
        }
        if (threadIdx.x == 0) { *scanTotal = carry; cellStart[ncap] = carry; }
    }
    if (!grid_sync(bar, status)) return;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long b0 = (long long)t * SCAN_TILE + (long long)threadIdx.x * PB_ITEMS;
        int sum = 0;
#pragma unroll 4
        for (int k = 0; k < PB_ITEMS; ++k) sum += b0 + k < ncap ? cellCount[b0 + k] : 0;
        int tot;
        int ex = block_exclusive_scan(sum, smem, tot) + tileSums[t];
#pragma unroll 4
        for (int k = 0; k < PB_ITEMS; ++k) {
            if (b0 + k < ncap) {
                const int v = cellCount[b0 + k];
                cellStart[b0 + k] = ex;
                ex += v;
            }
        }
    }
    if (!grid_sync(bar, status)) return;
    // 5: cell lists, then the reference's in-cell order
    for (int i = tid; i < p.n; i += nthr) {
        const int c = cell[i];
        const int pos = atomicAdd(&cellFill[c], 1);
        cellList[cellStart[c] + pos] = i;
    }
    if (!grid_sync(bar, status)) return;
    sort_cells(tid >> 5, nthr >> 5, *cellTotal, cellStart, cellList);
}

// ------------------------------------------------------------------ neighbour search

// Particles::gridNNS (Particles.cpp:324-365) over the 3^D stencil of
// Domain::getNeighborCells (Domain.cpp:83-118, x outer, z inner), and the
// periodic images of Particles::ghostNNS (Particles.cpp:2237-2260) through
// wrapped stencil cells, appended after the real neighbours in parent order.
// Then Particles::compDensity/compOmega (Particles.cpp:1151-1184, 2262-2290)
// and compPressure (:1272-1288) for the particle.
//
// One warp per cell (or per part of one, `nsplit` of them, where the cells are
// too few to fill the GPU): the particles of a cell share the candidate sequence
// (the stencil cells of their cell, in order).  Phase 1: the lanes hold 128
// candidates at a time in registers (index with image bits, and the single-
// precision position with the image shift applied) and test them against each
// particle of a batch of up to NNS_PB, broadcast from the lane that holds it: a
// single-precision distance test against a bound slightly above h^2, survivors
// compacted with a ballot into the particle's shared list in stencil order.
// Phase 2: the batch's lists are walked as one sequence, 32 candidates at a
// time, with the reference's FP64 test exactly (d^2 = (dx*dx + dy*dy) + dz*dz <
// h*h, no fused multiply-add) and W(r); real neighbours are appended (in order)
// to the slot list, with their offsets, and images parked behind them, then
// placed behind the real neighbours sorted by parent index.  Every count lives
// on the lane of its particle and is kept with ballots.  The single-precision
// test only decides which candidates phase 2 sees; it passes every neighbour
// (its error is far below the bound's margin), so the lists are those of the
// FP64 test alone.
// Bound: the FP64 pipe (64 % active) and issue (45 %).  With the chunk staged in
// shared memory and read back for every particle, counts in shared memory and a
// loop over the particles for the images, this took 341 M warp instructions on
// Sedov 64^3 and 4.48 ms on Sedov 128^3; now 218 M and 2.57 ms (64 KH members
// 1015 -> 620 us, Sedov 33^3 168 -> 96, KH 24^2 38 -> 17).
constexpr int NNS_WARPS = 8;
constexpr int NNS_PB = 12;    // particles of a cell per batch
constexpr int NNS_REG = 4;    // candidates per lane held in registers
// blocks of the neighbour search resident per SM: 4 caps it at 64 registers and
// gives 32 warps per SM (Sedov 128^3: 2.57 ms, 2.91 at 3, 3.13 at 2)
#ifndef MLH_NNS_MINB
#define MLH_NNS_MINB 4
#endif

struct NnsCells {
    int excl[27], start[27];
    unsigned wrap[27];
    float shift[27][3];   // image shift of a wrapped axis (-L or +L, single precision), else 0
};

// shared memory of k_neighbours: NNS_WARPS NnsCells, then per warp NNS_PB
// candidate lists (K + 32 uint32 each), the offsets of the lists in the batch's
// sequence (NNS_PB ints), image W (K doubles) and image entries (K uint32), each
// rounded up to 16 bytes
__host__ __device__ constexpr size_t nns_cells_bytes() {
    return (sizeof(NnsCells) * NNS_WARPS + 15) / 16 * 16;
}
__host__ __device__ constexpr size_t nns_r16(size_t b) { return (b + 15) / 16 * 16; }
__host__ __device__ constexpr size_t nns_warp_bytes(int K) {
    return nns_r16((size_t)NNS_PB * (K + 32) * 4) + nns_r16((size_t)NNS_PB * 4) + nns_r16((size_t)K * 8) +
           nns_r16((size_t)K * 4);
}
// bits [lo, hi) of a warp mask (any integers)
__device__ __forceinline__ unsigned range_mask(int lo, int hi) {
    lo = lo < 0 ? 0 : lo;
    hi = hi > 32 ? 32 : hi;
    return lo < hi ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
}

// The 3^D stencil cells of local cell ic in the reference's order
// (Domain::getNeighborCells, demonstrator/src/Domain.cpp:83-118; lane k
// holds cell k), written to the warp's NnsCells: the offset of each cell's
// members in the concatenated sequence, the start of its member list, its
// wrapped axes and image shift.  Returns the length of the sequence.
template <int D>
__device__ __forceinline__ int nns_stencil(const Params &p, const GridInfo &g, int ic,
                                           const int *__restrict__ cellStart, NnsCells *cs) {
    constexpr int NC = D == 3 ? 27 : 9;
    const int lane = threadIdx.x & 31;
    const int ix = ic % g.cells[0];
    const int iy = (ic / g.cells[0]) % g.cells[1];
    const int iz = D == 3 ? ic / (g.cells[0] * g.cells[1]) : 0;
    int cnt = 0, start = 0;
    unsigned wrap = 0;
    float sh[3] = {0.f, 0.f, 0.f};
    if (lane < NC) {
        int off[3] = {D == 3 ? lane / 9 - 1 : lane / 3 - 1, D == 3 ? (lane / 3) % 3 - 1 : lane % 3 - 1,
                      D == 3 ? lane % 3 - 1 : 0};
        int cc[3] = {ix + off[0], iy + off[1], iz + off[2]};
        bool skip = false;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            if (cc[a] < 0 || cc[a] >= g.cells[a]) {
                if (!p.periodic) skip = true;
                cc[a] = cc[a] < 0 ? cc[a] + g.cells[a] : cc[a] - g.cells[a];
                wrap |= 1u << a;
                sh[a] = off[a] < 0 ? -g.Lf[a] : g.Lf[a];
            }
        }
        if (!skip) {
            int c = g.cell_base + cc[0] + cc[1] * g.cells[0] + (D == 3 ? cc[2] * g.cells[0] * g.cells[1] : 0);
            start = cellStart[c];
            cnt = cellStart[c + 1] - start;
        }
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane < NC) {
        cs->excl[lane] = incl - cnt;
        cs->start[lane] = start;
        cs->wrap[lane] = wrap;
        cs->shift[lane][0] = sh[0]; cs->shift[lane][1] = sh[1]; cs->shift[lane][2] = sh[2];
    }
    __syncwarp();
    return total;
}

// Stencil cell of position t of the concatenated sequence: the last cell
// whose range starts at or before t (empty cells share their offset with the
// next one), by binary search over the non-decreasing offsets.
template <int D>
__device__ __forceinline__ int nns_cell_of(const NnsCells *cs, int t) {
    constexpr int NC = D == 3 ? 27 : 9;
    int k = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int kk = k + step;
        if (kk < NC && cs->excl[kk] <= t) k = kk;
    }
    return k;
}

// Candidates [ch, ch + 32 NNS_REG) of the stencil's sequence, candidate ch + 32 r
// + lane in element r: single-precision position with the image shift applied,
// index with image bits.  Beyond the sequence: NaN, which is within no distance (an
// infinite distance would be within the bound h^2 of a kernelSize above 1.8e19,
// which is infinite in single precision).
template <int D>
__device__ __forceinline__ void nns_candidates(const NnsCells *cs, const float4 *__restrict__ posf,
                                               const int *__restrict__ cellList, int ch, int total, float *cx,
                                               float *cy, float *cz, uint32_t *ce) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < NNS_REG; ++r) {
        const int t = ch + r * 32 + lane;
        cx[r] = __int_as_float(0x7fffffff); cy[r] = 0.f; cz[r] = 0.f; ce[r] = 0u;
        if (t < total) {
            const int k = nns_cell_of<D>(cs, t);
            const int j = cellList[cs->start[k] + (t - cs->excl[k])];
            const unsigned wr = cs->wrap[k];
            float4 fj = posf[j];
            if (wr) {
                fj.x += cs->shift[k][0];
                fj.y += cs->shift[k][1];
                if (D == 3) fj.z += cs->shift[k][2];
            }
            cx[r] = fj.x; cy[r] = fj.y; cz[r] = fj.z;
            ce[r] = (uint32_t)j | (wr << IMG_SHIFT);
        }
    }
}

template <int D, bool ADAPT>
__global__ void __launch_bounds__(NNS_WARPS * 32, MLH_NNS_MINB) k_neighbours(
    Params p, int nsplit, int pb, const Member *__restrict__ members, const int *__restrict__ memberOf,
    const GridInfo *grids, const double *x, const double *y,
    const double *z, const float4 *posf, const double *vx,
    const double *vy, const double *vz, const double *m,
    const double *u, const int *cellTotal, const int *cellStart,
    const int *cellList, uint32_t *nbr, double *dd,
    double *ww, int *noi, int *noiImg, int *faceCnt,
    Prim *prim, Geo *geo, float4 *velf, unsigned *status) {
    step_begin();
    constexpr unsigned ALL = 0xffffffffu;
    const int K = p.K;
    const int CAP = K + 32;
    extern __shared__ __align__(16) unsigned char nns_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    // per-warp shared areas; every sub-array starts on a 16-byte boundary
    // whatever K is (see nns_warp_bytes)
    NnsCells *cs = reinterpret_cast<NnsCells *>(nns_smem) + warp;
    unsigned char *wbase = nns_smem + nns_cells_bytes() + (size_t)warp * nns_warp_bytes(K);
    uint32_t *candq = reinterpret_cast<uint32_t *>(wbase);                            // NNS_PB lists of CAP
    int *offq = reinterpret_cast<int *>(wbase + nns_r16((size_t)NNS_PB * CAP * 4));
    double *imgW = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(offq) + nns_r16((size_t)NNS_PB * 4));
    uint32_t *imgE = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(imgW) + nns_r16((size_t)K * 8));

    const double *X[3] = {x, y, z};
    // a binning that gave up a bounded wait left no valid cells
    if (step_aborted(status)) return;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    // omega, density, pressure, 1/omega and sound speed of particle bi (per
    // lane): omega sums the stored W of the real neighbours in list order,
    // then W(0), then the images (Particles::compDensity, Particles.cpp:
    // 1151-1184, and its image part :2262-2290, in that order)
    int bi = -1, bnr = 0, bni = 0, filled = 0;   // filled: lanes 0 .. filled - 1 hold a particle
    double bw0 = 0.;
    auto finish = [&]() {
        if (bi < 0) return;
        const double *wb = ww + (size_t)bi * K;
        double bomega = 0.;
        for (int s = 0; s < bnr; ++s) bomega = addr(bomega, wb[s]);
        bomega = addr(bomega, bw0);
        for (int s = bnr; s < bnr + bni; ++s) bomega = addr(bomega, wb[s]);
        const double rho = m[bi] * bomega;
        const double P = (p.gamma - 1.) * rho * u[bi];
        // rho <= 0 and P <= 0 as sign tests on the bit patterns (a NaN with
        // the sign bit set also counts)
        unsigned st = 0;
        if (__double_as_longlong(rho) <= 0) st |= ST_NEG_DENSITY;
        if (__double_as_longlong(P) <= 0) st |= ST_NEG_PRESSURE;
        if (st) flag(status, st);
        Prim pr;
        pr.x = x[bi]; pr.y = y[bi]; pr.z = D == 3 ? z[bi] : 0.;
        pr.rho = rho; pr.P = P;
        pr.vx = vx[bi]; pr.vy = vy[bi]; pr.vz = D == 3 ? vz[bi] : 0.;
        prim[bi] = pr;
        geo[bi].omega = bomega;
        geo[bi].V = frcp(bomega);
        const double irho = frcp(rho);   // also the face kernel's 1/rho_i
        geo[bi].irho = irho;
        const double cs = fsqrt_rn(p.gamma * P * irho);
        geo[bi].c = cs;
        // velocity and sound speed in single precision, for the time step's
        // filter (k_gradients)
        velf[bi] = make_float4(__double2float_rn(pr.vx), __double2float_rn(pr.vy), __double2float_rn(pr.vz),
                               __double2float_rn(cs));
    };
    const unsigned nunits = (unsigned)(*cellTotal * nsplit);   // below 2^31, so that un + nw does not wrap
    for (unsigned un = gw; un < nunits; un += nw) {
        const int c = nsplit > 1 ? un / nsplit : un, part = nsplit > 1 ? un - c * nsplit : 0;
        const int c0 = cellStart[c], ncell = cellStart[c + 1] - c0;
        if (ncell <= part * pb) continue;
        const int mi = memberOf ? memberOf[cellList[c0]] : 0;   // a cell holds one member's particles
        const GridInfo &g = grids[mi];
        const Member &mb = members[mi];
        const int total = nns_stencil<D>(p, g, (int)c - g.cell_base, cellStart, cs);
        for (int b0 = part * pb; b0 < ncell; b0 += nsplit * pb) {
            const int nb = ncell - b0 < pb ? ncell - b0 : pb;
            // --- phase 1: particle q of the batch and its candidate count on lane q
            int myI = -1, myNc = 0;
            float4 myF = make_float4(0.f, 0.f, 0.f, 0.f);
            float myHf = 0.f;
            if (lane < nb) {
                myI = cellList[c0 + b0 + lane];
                myF = posf[myI];
                if (ADAPT) myHf = p.hpf[myI];
            }
            const float hsq_f = mb.hsq_f;
            for (int ch = 0; ch < total; ch += 32 * NNS_REG) {
                float cx[NNS_REG], cy[NNS_REG], cz[NNS_REG], chf[NNS_REG];
                uint32_t ce[NNS_REG];
                nns_candidates<D>(cs, posf, cellList, ch, total, cx, cy, cz, ce);
#pragma unroll
                for (int r = 0; r < NNS_REG; ++r)
                    chf[r] = ADAPT && ch + r * 32 + lane < total ? p.hpf[ce[r] & IDX_MASK] : 0.f;
                for (int q = 0; q < nb; ++q) {
                    const uint32_t iq = (uint32_t)__shfl_sync(ALL, myI, q);
                    const float fx = __shfl_sync(ALL, myF.x, q), fy = __shfl_sync(ALL, myF.y, q);
                    const float fz = D == 3 ? __shfl_sync(ALL, myF.z, q) : 0.f;
                    const float hq = ADAPT ? __shfl_sync(ALL, myHf, q) : 0.f;
                    int nq = __shfl_sync(ALL, myNc, q);
                    uint32_t *cq = candq + q * CAP;
#pragma unroll
                    for (int r = 0; r < NNS_REG; ++r) {
                        if (ch + r * 32 >= total) break;
                        const float dx = cx[r] - fx, dy = cy[r] - fy, dz = cz[r] - fz;
                        const float d2f = dx * dx + dy * dy + (D == 3 ? dz * dz : 0.f);
                        // with per-particle smoothing lengths the pair needs
                        // r < max(h_i, h_j): the same bound margin on the
                        // rounded-up single-precision h
                        float lim = hsq_f;
                        if (ADAPT) {
                            const float mh = fmaxf(hq, chf[r]);
                            lim = mh * mh * 1.001f;
                        }
                        // the particle itself is none (its images are candidates)
                        const bool pass = d2f <= lim && ce[r] != iq;
                        const unsigned bal = __ballot_sync(ALL, pass);
                        const int pos = nq + __popc(bal & lt_mask);
                        if (pass && pos < CAP) cq[pos] = ce[r];
                        nq += __popc(bal);
                    }
                    if (lane == q) myNc = nq;
                }
            }
            // --- phase 2: exact FP64 test, offset, W.  With per-particle smoothing
            // lengths the pair test is r^2 < max(h_i^2, h_j^2) and W uses h_i.
            // Particle q's position, kernel parameters, list and counts live on
            // lane q.  Real neighbours go to the front of the particle's slot row
            // in candidate order, images to its back (slot K-1-t for the t-th),
            // from where the step below sorts them behind the real ones.
            const int myN = lane < nb ? (myNc < CAP ? myNc : CAP) : 0;
            int myOff = myN;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(ALL, myOff, o);
                if (lane >= o) myOff += t;
            }
            const int seq = __shfl_sync(ALL, myOff, 31);
            myOff -= myN;
            __syncwarp();   // the batch before has read offq
            if (lane < NNS_PB) offq[lane] = lane < nb ? myOff : 0x7fffffff;
            double myX[3] = {0., 0., 0.};
            double myHsq = 0., myIh2 = 0., mySig = 0., mySig4 = 0., myW0 = 0.;
            if (lane < nb) {
#pragma unroll
                for (int a = 0; a < D; ++a) myX[a] = X[a][myI];
                if (ADAPT) {
                    const double hi_ = p.hp[myI];
                    const double h2_i = hi_ / 2.;
                    myHsq = __dmul_rn(hi_, hi_);
                    myIh2 = 1. / h2_i;
                    mySig = kernel_sigma<D>(h2_i);
                    mySig4 = 0.25 * mySig;   // the outer piece's factor, once per particle (exact)
                    myW0 = mySig;
                }
            }
            if (!ADAPT) { myIh2 = mb.ih2; mySig = mb.sigma; mySig4 = 0.25 * mySig; myW0 = mb.w0; }
            const double hsq = mb.hsq;
            __syncwarp();
            int myNr = 0, myNi = 0, myFc = 0;
            for (int t0 = 0; t0 < seq; t0 += 32) {
                const int gi = t0 + lane;
                const bool valid = gi < seq;
                // the particle of position gi: the last one whose list starts at
                // or before it (an empty list shares its offset with the next)
                int q = 0;
#pragma unroll
                for (int l4 = 0; l4 < NNS_PB; l4 += 4) {
                    const int4 o = *reinterpret_cast<const int4 *>(offq + l4);
                    if (l4 > 0) q += o.x <= gi;
                    q += (o.y <= gi) + (o.z <= gi) + (o.w <= gi);
                }
                const int i = __shfl_sync(ALL, myI, q), off = __shfl_sync(ALL, myOff, q), n_q = __shfl_sync(ALL, myN, q);
                const int nr0 = __shfl_sync(ALL, myNr, q), ni0 = __shfl_sync(ALL, myNi, q);
                double xi[3] = {0., 0., 0.};
#pragma unroll
                for (int a = 0; a < D; ++a) xi[a] = __shfl_sync(ALL, myX[a], q);
                const double hsq_i = ADAPT ? __shfl_sync(ALL, myHsq, q) : hsq;
                const double ih2_i = ADAPT ? __shfl_sync(ALL, myIh2, q) : myIh2;
                const double sigma_i = ADAPT ? __shfl_sync(ALL, mySig, q) : mySig;
                const double sigma4_i = ADAPT ? __shfl_sync(ALL, mySig4, q) : mySig4;
                bool pass = false, img = false;
                uint32_t e = 0;
                double w = 0., ed[3] = {0., 0., 0.};
                if (valid) {
                    e = candq[q * CAP + (gi - off)];
                    const int j = (int)(e & IDX_MASK);
                    const unsigned wr = e >> IMG_SHIFT;
                    img = wr != 0;
                    double xj[3];
                    bool ok = true;
#pragma unroll
                    for (int a = 0; a < D; ++a) {
                        xj[a] = X[a][j];
                        if (wr & (1u << a)) {
                            if (in_band(xj[a], g, a)) xj[a] = image_coord(xj[a], g, a);
                            else ok = false;
                        }
                    }
                    if (ok) {
#pragma unroll
                        for (int a = 0; a < D; ++a) ed[a] = subr(xj[a], xi[a]);
                        double d2 = addr(mulr(ed[0], ed[0]), mulr(ed[1], ed[1]));
                        if (D == 3) d2 = addr(d2, mulr(ed[2], ed[2]));
                        // d2, h^2 >= 0: compared as bit patterns on the integer pipe
                        double lim = hsq;
                        if (ADAPT) {
                            const double hj = p.hp[j];
                            const double hsq_j = __dmul_rn(hj, hj);
                            lim = __double_as_longlong(hsq_i) < __double_as_longlong(hsq_j) ? hsq_j : hsq_i;
                        }
                        pass = __double_as_longlong(d2) < __double_as_longlong(lim);
                        if (pass) w = kernelW2(fsqrt_rn(d2), ih2_i, sigma_i, sigma4_i);
                    }
                }
                // ranks among the passes of the lane's particle, and the counts of
                // the particle on this lane
                const unsigned balR = __ballot_sync(ALL, pass && !img), balI = __ballot_sync(ALL, pass && img);
                const unsigned balF = __ballot_sync(ALL, pass && (int)(e & IDX_MASK) > i);   // canonical faces
                const unsigned grp = range_mask(off - t0, off - t0 + n_q) & lt_mask;
                const unsigned own = range_mask(myOff - t0, myOff - t0 + myN);
                const size_t base = (size_t)i * K;
                if (pass) {
                    const int pos = img ? ni0 + __popc(balI & grp) : nr0 + __popc(balR & grp);
                    if (pos < K) {
                        const size_t sl = base + (img ? K - 1 - pos : pos);
                        nbr[sl] = e;
                        ww[sl] = w;
                        if (!img) {
#pragma unroll
                            for (int a = 0; a < D; ++a) dd[sl * 3 + a] = ed[a];
                        }
                    }
                }
                myNr += __popc(balR & own);
                myNi += __popc(balI & own);
                myFc += __popc(balF & own);
            }
            __syncwarp();   // the slots written above are visible to every lane
            // --- particles with images: behind the real neighbours, ordered by
            // parent index (their offsets are formed again: few particles have
            // images); particles that overflow their slots: clipped, and the step
            // is repeated with more
            const bool over = lane < nb && (myNc > CAP || myNr + myNi > K);
            for (unsigned todo = __ballot_sync(ALL, lane < nb && (myNi > 0 || over)); todo; todo &= todo - 1u) {
                const int q = __ffs((int)todo) - 1;
                const int i = __shfl_sync(ALL, myI, q);
                int nr = __shfl_sync(ALL, myNr, q), ni = __shfl_sync(ALL, myNi, q), fc = 0;
                const size_t base = (size_t)i * K;
                if (nr > K) nr = K;
                if (ni > K - nr) ni = K - nr;
                // images from the back of the row, in candidate order
                for (int t = lane; t < ni; t += 32) {
                    imgE[t] = nbr[base + K - 1 - t];
                    imgW[t] = ww[base + K - 1 - t];
                }
                __syncwarp();
                for (int t = lane; t < ni; t += 32) {
                    const uint32_t e = imgE[t];
                    const uint32_t id = e & IDX_MASK;
                    int rank = 0;
                    for (int v = 0; v < ni; ++v) rank += (imgE[v] & IDX_MASK) < id;
                    nbr[base + nr + rank] = e;
                    ww[base + nr + rank] = imgW[t];
#pragma unroll
                    for (int a = 0; a < D; ++a) {
                        double xa = X[a][id];
                        if (e & (1u << (IMG_SHIFT + a))) xa = image_coord(xa, g, a);
                        dd[(base + nr + rank) * 3 + a] = __dsub_rn(xa, X[a][i]);
                    }
                }
                __syncwarp();
                // canonical faces counted again from the final list, so that they
                // match k_link_own where the list was clipped
                for (int t = lane; t < nr + ni; t += 32) fc += (int)(nbr[base + t] & IDX_MASK) > i;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) fc += __shfl_xor_sync(ALL, fc, o);
                if (lane == q) { myNr = nr; myNi = ni; myFc = fc; }
                __syncwarp();
            }
            if (lane < nb) {
                noi[myI] = myNr;
                noiImg[myI] = myNi;
                faceCnt[myI] = myFc;
                if (over) flag(status, ST_NGB_OVERFLOW);
                if (myNr + myNi == 0) flag(status, ST_NO_NEIGHBOUR);
            }
            // the floating-point tail runs on all 32 lanes, once 32 particles of
            // this warp are there: this batch's go to the lanes after the filled ones
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int src = lane - filled + 32 * half;   // the particle of the batch for this lane
                const bool take = src >= 0 && src < nb;
                const int ti = __shfl_sync(ALL, myI, src & 31), tr = __shfl_sync(ALL, myNr, src & 31);
                const int tn = __shfl_sync(ALL, myNi, src & 31);
                const double tw = ADAPT ? __shfl_sync(ALL, myW0, src & 31) : myW0;
                if (take) { bi = ti; bnr = tr; bni = tn; bw0 = tw; }
                if (half == 0) {
                    if (filled + nb < 32) { filled += nb; break; }
                    finish();
                    bi = -1;
                } else {
                    filled += nb - 32;
                }
            }
        }   // batches of the cell
    }
    finish();
}

// ------------------------------------------------------------------ smoothing lengths

// Per-particle smoothing lengths (no counterpart in the reference, which uses
// one global kernelSize).  For particle i the support radius x in (0, H],
// H the member's kernelSize (the search radius), at which the effective
// neighbour number N(x) = V_D x^D (W(0, x) + sum_j W(r_ij, x)) equals n_ngb.
// With the cubic spline of support x, N(x) = K_D (1 + S(x)) where
// S(x) = sum_j f(2 r_ij / x) (f the spline's shape, f(0) = 1; K_D = 32/3 in
// 3D, 40/7 in 2D); S increases with x and dS/dx = G(x) / x with
// G = sum_j -f'(q) q.  The candidates within H of each particle (the
// neighbour search's stencil, pre-filter and exact test, images by the ghost
// rule) are kept in shared memory in stencil order.  Every Newton iteration
// sums f and g over them in 32 lane-strided partial sums combined by an xor
// butterfly, and the iteration is bracketed (bisection when Newton leaves the
// bracket).  The start is the previous h_i (H at first); a particle with
// N(H) < n_ngb keeps H and is counted in hstat[1]; hstat[0] counts
// iterations.  The CPU restatement performs the same operations in the same
// order and gets the same bits.
//
// One warp per cell, as the neighbour search: the lanes hold the cell's
// candidates in registers and filter them for a batch of up to HS_PB of its
// particles; the warp then computes their candidate distances, the batch's lists
// as one sequence, and runs their Newton iterations side by side: per
// iteration, the sums of each unfinished particle of the batch (all lanes, the
// order above), then the scalar updates of all of them at once, particle q on
// lane q, so that the divisions and tests of an update are issued once per batch
// instead of once per particle.  Bound: the FP64 pipe (58 % active) and latency
// at 16 warps per SM; 61^3 with 32 neighbours: 1600 us with a staged chunk, FP64
// products and __dsqrt_rn, 1020 us so.  80 or 64 registers for more warps: 1.10,
// 1.22 ms.
constexpr int HSOLVE_MAXIT = 50;
constexpr int HS_PB = 8;
// the reduce-scatter of the solve's sums maps the 2 HS_PB = 16 sums onto
// the 32 lanes (sum k on lanes 2k and 2k + 1)
static_assert(HS_PB == 8, "k_hsolve reduces exactly 16 sums per batch");

// HS_PB candidate lists (K + 32 uint32 each), their offsets in the batch's
// sequence (HS_PB ints) and HS_PB distance lists (K + 32 doubles each), each
// rounded up to 16 bytes
__host__ __device__ constexpr size_t hsolve_warp_bytes(int K) {
    return nns_r16((size_t)HS_PB * (K + 32) * 4) + nns_r16((size_t)HS_PB * 4) + (size_t)HS_PB * (K + 32) * 8;
}

// Shape of the cubic spline and its scaled derivative for the smoothing-length
// solve: q = r / (h/2) (given as r times 1 / (h/2)), f(q) with f(0) = 1 and
// g(q) = -f'(q) q; for q <= 1, f = fma(q^2, fma(0.75, q, -1.5), 1) and
// g = q^2 fma(-2.25, q, 3); for 1 < q < 2, with t = 2 - q, f = (t^2/4) t and
// g = (3 t^2/4) q; 0 beyond.  Every operation is an explicitly rounded
// intrinsic so that the CPU restatement, which performs the same operations,
// gets the same bits.  Both pieces run as the same operations with selected
// operands (f = (t^2/4) t as fma(t^2/4, t, 0), the same rounded product), so
// a warp whose candidates fall on both sides of q = 1 issues them once.
// The products, of positive factors, on the integer pipe (xmul, the same bits).
__device__ __forceinline__ void hsolve_shape_sel(double r, double ihh2, double &f, double &g) {
    const double q = xmul(r, ihh2);
    const long long qb = __double_as_longlong(q);   // q >= 0: q <= 1 and q < 2 on the bits
    const bool inner = qb <= 0x3FF0000000000000ll, in = qb < 0x4000000000000000ll;
    const double t = subr(2., q);
    const double a = inner ? q : t;
    const double a2 = xmul(a, a);
    const double u = __fma_rn(0.75, q, -1.5);
    const double v = __fma_rn(-2.25, q, 3.);
    // a2 / 4 (exact) on the integer pipe
    const double f_ = __fma_rn(inner ? a2 : scale_down<2>(a2), inner ? u : t, inner ? 1. : 0.);
    const double g_ = xmul(inner ? a2 : xmul(0.75, a2), inner ? v : q);
    f = in ? f_ : 0.;
    g = in ? g_ : 0.;
}

template <int D>
__global__ void __launch_bounds__(NNS_WARPS * 32, 2) k_hsolve(
    Params p, const Member *__restrict__ members, const int *__restrict__ memberOf,
    const GridInfo *__restrict__ grids, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const float4 *__restrict__ posf, const int *__restrict__ cellTotal,
    const int *__restrict__ cellStart, const int *__restrict__ cellList, double *__restrict__ hp,
    float *__restrict__ hpf, double *__restrict__ neff, unsigned long long *__restrict__ hstat,
    unsigned *__restrict__ status) {
    constexpr unsigned ALL = 0xffffffffu;
    const int K = p.K;
    const int CAP = K + 32;
    extern __shared__ __align__(16) unsigned char hs_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    NnsCells *cs = reinterpret_cast<NnsCells *>(hs_smem) + warp;
    unsigned char *wbase = hs_smem + nns_cells_bytes() + (size_t)warp * hsolve_warp_bytes(K);
    uint32_t *candq = reinterpret_cast<uint32_t *>(wbase);                            // HS_PB lists of CAP
    int *offq = reinterpret_cast<int *>(wbase + nns_r16((size_t)HS_PB * CAP * 4));
    double *rlq = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(offq) + nns_r16((size_t)HS_PB * 4));   // HS_PB lists of CAP
    constexpr double KD = D == 3 ? 32. / 3. : 40. / 7.;
    const double St = p.sngb_t;
    const double tolS = __dmul_rn(1e-12, St);
    const double *X[3] = {x, y, z};
    if (step_aborted(status)) return;   // no valid cells
    unsigned long long iters = 0, clamped = 0;   // per lane, for its particles
    bool overflow_any = false;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const unsigned ncells = (unsigned)*cellTotal;   // below 2^31, so that c + nw does not wrap
    for (unsigned c = gw; c < ncells; c += nw) {
        const int c0 = cellStart[c], ncell = cellStart[c + 1] - c0;
        if (ncell <= 0) continue;
        const int mi = memberOf ? memberOf[cellList[c0]] : 0;
        const GridInfo &g = grids[mi];
        const Member &mb = members[mi];
        const double H = mb.h;
        const int total = nns_stencil<D>(p, g, (int)c - g.cell_base, cellStart, cs);
        for (int b0 = 0; b0 < ncell; b0 += HS_PB) {
            const int nb = ncell - b0 < HS_PB ? ncell - b0 : HS_PB;
            // --- candidates of the batch within H, in stencil order: single-
            // precision filter as in k_neighbours, particle q on lane q
            int myI = -1, myNc = 0;
            float4 myF = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < nb) { myI = cellList[c0 + b0 + lane]; myF = posf[myI]; }
            const float hsq_f = mb.hsq_f;
            for (int ch = 0; ch < total; ch += 32 * NNS_REG) {
                float cx[NNS_REG], cy[NNS_REG], cz[NNS_REG];
                uint32_t ce[NNS_REG];
                nns_candidates<D>(cs, posf, cellList, ch, total, cx, cy, cz, ce);
                for (int q = 0; q < nb; ++q) {
                    const uint32_t iq = (uint32_t)__shfl_sync(ALL, myI, q);
                    const float fx = __shfl_sync(ALL, myF.x, q), fy = __shfl_sync(ALL, myF.y, q);
                    const float fz = D == 3 ? __shfl_sync(ALL, myF.z, q) : 0.f;
                    int nq = __shfl_sync(ALL, myNc, q);
                    uint32_t *cq = candq + q * CAP;
#pragma unroll
                    for (int r = 0; r < NNS_REG; ++r) {
                        if (ch + r * 32 >= total) break;
                        const float dx = cx[r] - fx, dy = cy[r] - fy, dz = cz[r] - fz;
                        const bool pass = dx * dx + dy * dy + (D == 3 ? dz * dz : 0.f) <= hsq_f && ce[r] != iq;
                        const unsigned bal = __ballot_sync(ALL, pass);
                        const int pos = nq + __popc(bal & lt_mask);
                        if (pass && pos < CAP) cq[pos] = ce[r];
                        nq += __popc(bal);
                    }
                    if (lane == q) myNc = nq;
                }
            }
            // --- exact FP64 distances of the candidates within H, in order: the
            // lists walked as one sequence, as in k_neighbours
            const int myN = lane < nb && myNc <= CAP ? myNc : 0;
            int myOff = myN;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(ALL, myOff, o);
                if (lane >= o) myOff += t;
            }
            const int seq = __shfl_sync(ALL, myOff, 31);
            myOff -= myN;
            __syncwarp();
            if (lane < HS_PB) offq[lane] = lane < nb ? myOff : 0x7fffffff;
            double myX[3] = {0., 0., 0.};
            if (lane < nb) {
#pragma unroll
                for (int a = 0; a < D; ++a) myX[a] = X[a][myI];
            }
            const double hsq = mb.hsq;
            __syncwarp();
            int myNr = 0;
            for (int t0 = 0; t0 < seq; t0 += 32) {
                const int gi = t0 + lane;
                int q = 0;
#pragma unroll
                for (int l4 = 0; l4 < HS_PB; l4 += 4) {
                    const int4 o = *reinterpret_cast<const int4 *>(offq + l4);
                    if (l4 > 0) q += o.x <= gi;
                    q += (o.y <= gi) + (o.z <= gi) + (o.w <= gi);
                }
                const int off = __shfl_sync(ALL, myOff, q), n_q = __shfl_sync(ALL, myN, q), nr0 = __shfl_sync(ALL, myNr, q);
                double xi[3] = {0., 0., 0.};
#pragma unroll
                for (int a = 0; a < D; ++a) xi[a] = __shfl_sync(ALL, myX[a], q);
                bool pass = false;
                double r = 0.;
                if (gi < seq) {
                    const uint32_t e = candq[q * CAP + (gi - off)];
                    const int j = (int)(e & IDX_MASK);
                    const unsigned wr = e >> IMG_SHIFT;
                    double xj[3];
                    bool ok = true;
#pragma unroll
                    for (int a = 0; a < D; ++a) {
                        xj[a] = X[a][j];
                        if (wr & (1u << a)) {
                            if (in_band(xj[a], g, a)) xj[a] = image_coord(xj[a], g, a);
                            else ok = false;
                        }
                    }
                    if (ok) {
                        double ed[3];
#pragma unroll
                        for (int a = 0; a < D; ++a) ed[a] = subr(xj[a], xi[a]);
                        double d2 = addr(mulr(ed[0], ed[0]), mulr(ed[1], ed[1]));
                        if (D == 3) d2 = addr(d2, mulr(ed[2], ed[2]));
                        pass = __double_as_longlong(d2) < __double_as_longlong(hsq);   // d2 < H^2, both >= 0
                        if (pass) r = fsqrt_rn(d2);
                    }
                }
                const unsigned bal = __ballot_sync(ALL, pass);
                if (pass) rlq[(size_t)q * CAP + nr0 + __popc(bal & range_mask(off - t0, off - t0 + n_q) & lt_mask)] = r;
                myNr += __popc(bal & range_mask(myOff - t0, myOff - t0 + myN));
            }
            __syncwarp();
            // --- bracketed Newton on S(x) = St, particle q's state on lane q
            // (-1: no solve; more candidates than the list holds: the host grows the
            // slots and repeats)
            const int mynr = lane < nb && myNc <= CAP ? myNr : -1;
            if (lane < nb && mynr < 0) overflow_any = true;
            bool done = !(lane < nb) || mynr < 0;
            double xh = H, lo = 0., hi = H, S = 0., sfq = 0., sgq = 0.;
            bool upper = false;
            int it = 0;
            if (!done) {
                xh = hp[myI];
                if (!(xh > 0. && xh <= H)) xh = H;
            }
            for (;;) {
                const unsigned act = __ballot_sync(0xffffffffu, !done);
                if (!act) break;
                const double ihh2 = __ddiv_rn(1., __dmul_rn(0.5, xh));
                // 32 lane-strided partial sums of f and g per unfinished
                // particle: v[2q], v[2q + 1]
                double v[2 * HS_PB];
#pragma unroll
                for (int q = 0; q < HS_PB; ++q) {
                    v[2 * q] = 0.;
                    v[2 * q + 1] = 0.;
                    if (act & (1u << q)) {
                        const double ihq = __shfl_sync(0xffffffffu, ihh2, q);
                        const int nrq_ = __shfl_sync(0xffffffffu, mynr, q);
                        const double *rl = rlq + (size_t)q * CAP;
                        for (int t = lane; t < nrq_; t += 32) {
                            double f, gg;
                            hsolve_shape_sel(rl[t], ihq, f, gg);
                            v[2 * q] = addr(v[2 * q], f);
                            v[2 * q + 1] = addr(v[2 * q + 1], gg);
                        }
                    }
                }
                // reduce-scatter of the 16 partial sums: at distance d = 16,
                // 8, 4, 2 each lane keeps half of its values and adds its
                // partner's (own + partner, the pairs of an xor butterfly, so
                // every sum has the butterfly's tree and bits), then d = 1;
                // sum k ends on lanes 2k and 2k + 1
#pragma unroll
                for (int d = 16, m = HS_PB; d > 1; d >>= 1, m >>= 1) {
                    const bool upper = (lane & d) != 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (j < m) {
                            const double send = upper ? v[j] : v[j + m];
                            const double keep = upper ? v[j + m] : v[j];
                            v[j] = addr(keep, __shfl_xor_sync(0xffffffffu, send, d));
                        }
                    }
                }
                v[0] = __dadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1));
                // particle q (lane q) takes sum 2q (lane 4q) and 2q + 1 (lane 4q + 2)
                sfq = __shfl_sync(0xffffffffu, v[0], (4 * lane) & 31);
                sgq = __shfl_sync(0xffffffffu, v[0], (4 * lane + 2) & 31);
                if (!done) {
                    S = sfq;
                    const double G = sgq;
                    ++iters;
                    const double F = __dsub_rn(S, St);
                    if (fabs(F) <= tolS) done = true;
                    else if (F < 0. && xh >= H) { ++clamped; done = true; }
                    else if (it + 1 >= HSOLVE_MAXIT) done = true;
                    else {
                        if (F > 0.) { hi = xh; upper = true; }
                        else lo = xh;
                        double xn = G > 0. ? __dsub_rn(xh, __ddiv_rn(__dmul_rn(F, xh), G))
                                           : __dmul_rn(0.5, __dadd_rn(lo, hi));
                        if (!(xn > lo && xn < hi)) xn = (!upper && xn >= hi) ? H : __dmul_rn(0.5, __dadd_rn(lo, hi));
                        if (xn == xh) done = true;
                        else xh = xn;
                    }
                    ++it;
                }
            }
            if (lane < nb && mynr >= 0) {
                hp[myI] = xh;
                hpf[myI] = __double2float_ru(xh);
                if (neff) neff[myI] = __dmul_rn(KD, __dadd_rn(S, 1.));
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        iters += __shfl_xor_sync(0xffffffffu, iters, o);
        clamped += __shfl_xor_sync(0xffffffffu, clamped, o);
    }
    const bool of = __any_sync(0xffffffffu, overflow_any);
    if (lane == 0) {
        if (iters) atomicAdd(hstat, iters);
        if (clamped) atomicAdd(hstat + 1, clamped);
        if (of) flag(status, ST_NGB_OVERFLOW);
    }
}

size_t hsolve_smem_bytes(int K) {
    return nns_cells_bytes() + (size_t)NNS_WARPS * hsolve_warp_bytes(K);
}

size_t nns_smem_bytes(int K) {
    return nns_cells_bytes() + (size_t)NNS_WARPS * nns_warp_bytes(K);
}

// Both kernels list a particle's candidates in shared memory, K + 32 of them.
int most_slots(size_t smem_per_block, bool hsolve) {
    int K = 0;
    while (nns_smem_bytes(K + 4) <= smem_per_block && (!hsolve || hsolve_smem_bytes(K + 4) <= smem_per_block)) K += 4;
    return K;
}

// ------------------------------------------------------------------ dt

// dt of every simulation from its minimum (or the fixed time step), clamped; by
// one block.  A step whose binning was given up keeps the dt of the last one.
__device__ __forceinline__ void dt_final(const Params &p, int nmembers, const unsigned long long *dtbits, double dt_max,
                                         double *__restrict__ dt_out) {
    for (int mi = threadIdx.x; mi < nmembers; mi += blockDim.x) {
        double dt = p.adaptive ? __longlong_as_double((long long)*(const volatile unsigned long long *)(dtbits + mi))
                               : p.time_step;
        if (dt_max > 0. && dt > dt_max) dt = dt_max;
        dt_out[mi] = dt;
    }
}

// c_i + c_j - min(0, v_ij . x_ij / r) as one fused multiply-add: 1/r only when
// the dot product dv = v_ij . x_ij is negative, 0 otherwise; r as the neighbour
// search takes it
template <int D>
__device__ __forceinline__ double signal_speed(double dv, const double *xij, double csum) {
    double ir = 0.;
    if (dneg(dv)) {
        double d2 = addr(mulr(xij[0], xij[0]), mulr(xij[1], xij[1]));
        if (D == 3) d2 = addr(d2, mulr(xij[2], xij[2]));
        ir = frcp(fsqrt_rn(d2));
    }
    return fma(-dv, ir, csum);
}

// Particles::compGlobalTimestep (Particles.cpp:1446-1485): real neighbours
// only, v_sig starting at numeric_limits<double>::min().  The minimum over
// particles is order independent, so an atomicMin on the bit pattern of the
// (positive) per-particle dt is deterministic.
template <int D>
__global__ void __launch_bounds__(256) k_timestep(Params p, const Member *__restrict__ members,
                                                  const int *__restrict__ memberOf, const Prim *prim,
                                                  const Geo *geo, const uint32_t *nbr,
                                                  const int *noi,
                                                  unsigned long long *dtbits,
                                                  const float *dtlo, const unsigned *dtcap,
                                                  int nmembers, double dt_max, double *dt_out,
                                                  unsigned *arrived,
                                                  const unsigned *status) {
    step_begin();
    const int lane = threadIdx.x & 31;
    // no valid lists after an aborted binning
    const int n = step_aborted(status) ? 0 : p.n;
    // warp-uniform loop: every lane takes part in the reductions below
    for (int i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        int mi = -1;
        double dti = DBL_MAX_;
        // with dtlo (the single-precision filter of k_gradients): only the
        // particles whose lower bound on dt reaches their simulation's least
        // upper bound can hold the minimum (the others leave dti at DBL_MAX;
        // every lane stays in the loop for the warp's reduction)
        bool cand = i < p.n;
        if (cand && dtlo) {
            const int m = memberOf ? memberOf[i] : 0;
            cand = dtlo[i] <= __uint_as_float(dtcap[m]);
        }
        // the warp's candidates one after another, a lane per neighbour: a handful
        // of candidates would leave a thread each to a chain of dependent loads
        // (KH 100^2: 20.7 us with a thread per candidate, 6.5 so)
        unsigned todo = __ballot_sync(0xffffffffu, cand);
        if (cand) mi = memberOf ? memberOf[i] : 0;
        while (todo) {
            const int b = __ffs((int)todo) - 1, ib = i0 + b;
            todo &= todo - 1u;
            const Prim pi = prim[ib];
            const double ci = geo[ib].c;
            const size_t base = (size_t)ib * p.K;
            const int nr = noi[ib];
            double vSig = DBL_MIN_;
            for (int s = lane; s < nr; s += 32) {
                const int j = (int)(nbr[base + s] & IDX_MASK);
                const Prim pj = prim[j];
                const double cj = geo[j].c;
                const double xij[3] = {subr(pi.x, pj.x), subr(pi.y, pj.y), subr(pi.z, pj.z)};
                const double vij[3] = {subr(pi.vx, pj.vx), subr(pi.vy, pj.vy), subr(pi.vz, pj.vz)};
                const double vs = signal_speed<D>(dotD<D>(vij, xij), xij, addr(ci, cj));
                vSig = dlt(vSig, vs) ? vs : vSig;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double t = __shfl_xor_sync(0xffffffffu, vSig, o);
                vSig = dlt(vSig, t) ? t : vSig;
            }
            if (lane == b) dti = (p.adaptive_h ? p.cfl * p.hp[ib] : members[mi].cfl_h) / vSig;
        }
        // the minimum over particles does not depend on the order of the
        // atomicMin calls: a warp inside one simulation (the common case)
        // reduces first and issues one atomic; a warp that straddles two
        // simulations issues one per lane
        const int m0 = __shfl_sync(0xffffffffu, mi, 0);
        if (__all_sync(0xffffffffu, mi == m0)) {
            double best = dti;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && m0 >= 0 && best < DBL_MAX_) atomic_min_pos_double(dtbits + m0, best);
        } else if (mi >= 0 && dti < DBL_MAX_) {
            atomic_min_pos_double(dtbits + mi, dti);
        }
    }
    // the last block to arrive holds every minimum
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(arrived, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (last) {
        if (threadIdx.x == 0) *arrived = 0u;   // for the next step
        __threadfence();
        if (n > 0) dt_final(p, nmembers, dtbits, dt_max, dt_out);
    }
}

// dt of every simulation when no k_timestep follows the minima
__global__ void k_dt_final(Params p, int nmembers, const unsigned long long *dtbits, double dt_max,
                           double *dt_out, const unsigned *status) {
    step_begin();
    if (!step_aborted(status)) dt_final(p, nmembers, dtbits, dt_max, dt_out);
}

// ------------------------------------------------------------------ face links

// Canonical faces: slot s of particle i with neighbour (or image parent)
// j > i, the side on which Particles::solveRiemannProblems computes the flux
// (Particles.cpp:1838-1858, 1886-1897).  Slot -> face id (+1 canonical, -1
// copied with the opposite sign), face -> (i, slot, reverse slot).  The
// reverse slot of a non-canonical slot is the first entry of j's list (real
// part or image part) that refers to i, as in the reference's searches.
// The face links of particle i by one thread.  A slot with j < i finds i in j's
// list (real part or image part) and the face's rank in j's list from j's
// canonical entries (index > j) on one side of it: searching forward, the rank
// is the count before i; searching backward from the end of j's list, it is
// faceCnt[j] - 1 - the count after i, faceCnt[j] = faceOff[j + 1] - faceOff[j]
// being the number of canonical entries of j's list.  The stencils of i and j
// mirror each other, so j early in i's list puts i late in j's list: those
// searches and the image searches (images sit at the end of the list) go
// backward.  The own list is read four slots per load (K is a multiple of 4)
// and the searches of those four slots advance together, one 4-entry load of
// each list per round, so that a thread has up to four loads in flight.
__device__ __forceinline__ void link_particle(int i, const Params &p, const uint32_t *__restrict__ nbr,
                                              const int *__restrict__ noi, const int *__restrict__ noiImg,
                                              const int *__restrict__ faceOff, int *__restrict__ faceOf,
                                              FaceRef *__restrict__ faces, unsigned *__restrict__ status) {
    const size_t base = (size_t)i * p.K;
    const int nr = noi[i], tot = nr + noiImg[i];
    const uint4 *own = reinterpret_cast<const uint4 *>(nbr + base);
    int rank = 0;
    for (int s0 = 0; s0 < tot; s0 += 4) {
        const uint4 q = own[s0 >> 2];
        const uint32_t ev[4] = {q.x, q.y, q.z, q.w};
        // per search: j, the length of j's list, the current 4-entry chunk,
        // the canonical count and flags.  i is sought among j's real
        // entries (no image bits) or among its images (image bits set), so
        // an entry's own bits say whether it lies in the searched part.
        constexpr unsigned ACT = 1u, BWD = 2u, IMG = 4u, FOUND = 8u;
        int jj[4], jt[4], cur[4], cnt[4];
        unsigned fl[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int s = s0 + k;
            const int j = (int)(ev[k] & IDX_MASK);
            jj[k] = j; jt[k] = 0; cur[k] = 0; cnt[k] = 0; fl[k] = 0u;
            if (s >= tot) continue;
            if (j > i) {
                const int fid = faceOff[i] + rank;
                ++rank;
                if (fid >= p.faces_cap) { flag(status, ST_CAPACITY); faceOf[base + s] = 0; continue; }
                faceOf[base + s] = fid + 1;
                faces[fid].i = i;
                faces[fid].slot = s;
                continue;
            }
            jt[k] = noi[j] + noiImg[j];
            const bool img = s >= nr;
            // a particle that is its own image searches forward
            const bool bwd = (img || 2 * s < nr) && j != i;
            cur[k] = bwd ? (jt[k] - 1) >> 2 : 0;
            fl[k] = ACT | (bwd ? BWD : 0u) | (img ? IMG : 0u);
        }
        for (;;) {
            uint4 r[4];
            bool any = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // past either end of j's list: not found
                if ((fl[k] & BWD) ? cur[k] < 0 : cur[k] * 4 >= jt[k]) fl[k] &= ~ACT;
                r[k] = (fl[k] & ACT) ? reinterpret_cast<const uint4 *>(nbr + (size_t)jj[k] * p.K)[cur[k]]
                                     : make_uint4(0u, 0u, 0u, 0u);
                any |= (fl[k] & ACT) != 0u;
            }
            if (!any) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (!(fl[k] & ACT)) continue;
                const bool bwd = (fl[k] & BWD) != 0u, img = (fl[k] & IMG) != 0u;
                const uint32_t v[4] = {r[k].x, r[k].y, r[k].z, r[k].w};
#pragma unroll
                for (int mm = 0; mm < 4; ++mm) {
                    const int m = bwd ? 3 - mm : mm;
                    const int t = cur[k] * 4 + m;
                    const uint32_t e = v[m];
                    const int idx = (int)(e & IDX_MASK);
                    if (!(fl[k] & FOUND) && t < jt[k]) {
                        if (idx == i && ((e >> IMG_SHIFT) != 0u) == img) fl[k] |= FOUND;
                        else cnt[k] += idx > jj[k];
                    }
                }
                if (fl[k] & FOUND) fl[k] &= ~ACT;
                else cur[k] += bwd ? -1 : 1;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int s = s0 + k;
            if (s >= tot || jj[k] > i) continue;
            if (!(fl[k] & FOUND)) { flag(status, ST_ASYMMETRIC); faceOf[base + s] = 0; continue; }
            const int fid = (fl[k] & BWD) ? faceOff[jj[k] + 1] - 1 - cnt[k] : faceOff[jj[k]] + cnt[k];
            if (fid >= p.faces_cap) { flag(status, ST_CAPACITY); faceOf[base + s] = 0; continue; }
            faceOf[base + s] = -(fid + 1);
            faces[fid].rslot = s;
        }
    }
}

// The face links as two kernels.  k_link_own, a warp per particle and a lane
// per slot: a slot with j > i owns face faceOff[i] + its rank among i's
// canonical slots (a ballot); the other slots are set to 0 until their face
// finds them.
__global__ void __launch_bounds__(256) k_link_own(Params p, const uint32_t *nbr,
                                                  const int *noi, const int *noiImg,
                                                  const int *faceOff, int *faceOf,
                                                  FaceRef *faces, unsigned *status) {
    step_begin();
    if (step_aborted(status)) return;   // no valid lists
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    bool full = false;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < p.n; i += nw) {
        const size_t base = (size_t)i * p.K;
        const int tot = noi[i] + noiImg[i];
        int rank = faceOff[i];
        for (int s0 = 0; s0 < tot; s0 += 32) {
            const int s = s0 + lane;
            const bool canon = s < tot && (int)(nbr[base + s] & IDX_MASK) > i;
            const unsigned cm = __ballot_sync(0xffffffffu, canon);
            const int f = rank + __popc(cm & ((1u << lane) - 1u));
            const bool fits = canon && f < p.faces_cap;
            if (s < tot) faceOf[base + s] = fits ? f + 1 : 0;
            if (fits) { faces[f].i = i; faces[f].slot = s; }
            full = full || (canon && !fits);
            rank += __popc(cm);
        }
    }
    if (full) flag(status, ST_CAPACITY);
}

// k_link, a thread per face: finds i in j's list (real part or image part) and
// links that slot, faceOf = -(face + 1) and the face's rslot; each slot with
// j < i is found by the one face it belongs to (one that no face finds keeps 0
// and is reported by the flux gather).  The stencils of i and j mirror each
// other, so slot s of i's real part puts i near slot noi[j] - 1 - s of j's: the
// search starts at that 4-entry chunk and widens to both sides.  Images are
// ordered by parent index: that part is searched from its start.  Sedov 64^3 /
// 128^3 / 64 KH members, with the scan of the face counts: 130 / 966 / 265 us; a thread
// per particle, searching four lists in lockstep from their ends (link_particle,
// which the gradients kernel runs with link_overlap 2), took 288 / 1771 / 446 us,
// 700 warp instructions per particle with 13 of 32 lanes active.
__global__ void __launch_bounds__(256) k_link(Params p, const uint32_t *nbr, const int *noi,
                                              const int *noiImg, const int *faceTotal,
                                              int *faceOf, FaceRef *faces,
                                              unsigned *status) {
    step_begin();
    if (step_aborted(status)) return;
    const int nf = *faceTotal < p.faces_cap ? *faceTotal : p.faces_cap;
    bool lost = false;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
        const int i = faces[f].i, s = faces[f].slot;
        const uint32_t e = nbr[(size_t)i * p.K + s];
        const int j = (int)(e & IDX_MASK);
        const bool img = (e >> IMG_SHIFT) != 0u;
        const int nrj = noi[j];
        // the part of j's list that i is sought in, and the chunks that hold it
        const int lo = img ? nrj : 0, hi = img ? nrj + noiImg[j] : nrj;
        int at = -1;
        if (hi > lo) {
            const uint4 *row = reinterpret_cast<const uint4 *>(nbr + (size_t)j * p.K);
            const int c_lo = lo >> 2, c_hi = (hi - 1) >> 2, guess = nrj - 1 - s;
            int c = img ? c_lo : guess > 0 ? guess >> 2 : 0;
            int up = c + 1, dn = c - 1;   // the next chunks on either side
            bool go_up = true;
            for (;;) {
                const uint4 v = row[c];
                const uint32_t ev[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int t = c * 4 + m;
                    if ((int)(ev[m] & IDX_MASK) == i && t >= lo && t < hi) at = t;   // a part holds i once
                }
                const bool can_up = up <= c_hi, can_dn = dn >= c_lo;
                if (at >= 0 || !(can_up || can_dn)) break;
                c = can_up && (go_up || !can_dn) ? up++ : dn--;
                go_up = !go_up;
            }
        }
        faces[f].rslot = at;
        if (at >= 0) faceOf[(size_t)j * p.K + at] = -(f + 1);
        else lost = true;
    }
    if (lost) flag(status, ST_ASYMMETRIC);
}

// ------------------------------------------------------------------ gradients

// Particles::compPsijTilde (Particles.cpp:1186-1254, 2292-2455): E_i =
// sum_j (x_j - x_i)(x_j - x_i)^T W_ij / omega_i, B_i = E_i^-1 (closed form);
// Particles::gradient (:1257-1270, 2457-2502) for rho, vx, vy, (vz), P with
// psi~_j(x_i) = B_i (x_j - x_i) W_ij / omega_i; Particles::slopeLimiter
// (:1313-1444) with the face midpoint x_ij = (x_i + x_j)/2.
// inverse of the symmetric matrix A (closed form; the upper triangle is read,
// every entry written)
template <int D>
__device__ __forceinline__ void invert_symmetric(double *A) {
    if (D == 2) {
        const double a = A[0], b = A[1], d = A[3];
        const double id = frcp(fma(a, d, -mulr(b, b)));
        A[0] = mulr(d, id); A[1] = A[2] = -mulr(b, id); A[3] = mulr(a, id);
    } else {
        const double a = A[0], b = A[1], c = A[2], d = A[4], e = A[5], f = A[8];
        const double c00 = fma(d, f, -mulr(e, e)), c01 = fma(e, c, -mulr(b, f)), c02 = fma(b, e, -mulr(d, c));
        const double id = frcp(fma(a, c00, fma(b, c01, mulr(c, c02))));
        A[0] = mulr(c00, id);
        A[1] = A[3] = mulr(c01, id);
        A[2] = A[6] = mulr(c02, id);
        A[4] = mulr(fma(a, f, -mulr(c, c)), id);
        A[5] = A[7] = mulr(fma(c, b, -mulr(a, e)), id);
        A[8] = mulr(fma(a, d, -mulr(b, b)), id);
    }
}

// x 2^(1023 - 127 - base / 2^20) in single precision, the mantissa truncated (error
// below 2^-23 of the result, or 2^-126 where it flushes to zero), on the integer
// pipe: the exponent is rebased on the way.  base: a biased double exponent less
// 127, in place; 896 << 20 takes x as it is.
__device__ __forceinline__ float trunc_f32(double x, int base) {
    const uint32_t h = __double2hiint(x), l = __double2loint(x);
    const uint32_t m = (h & 0x7fffffffu) - (uint32_t)base;    // rebased exponent and the mantissa's top
    const uint32_t v = __funnelshift_l(l, m, 3);
    return __uint_as_float(((int)m < (1 << 20) ? 0u : (int)m >= (255 << 20) ? 0x7f800000u : v & 0x7fffffffu) | (h & 0x80000000u));
}
// the exponent field (in place) of the largest of D numbers' magnitudes, and the
// base that takes it to 1 in single precision
template <int D>
__device__ __forceinline__ int top_exponent(const double *x) {
    int e = 0;
#pragma unroll
    for (int a = 0; a < D; ++a) e = max(e, __double2hiint(x[a]) & 0x7ff00000);
    return e;
}
__device__ __forceinline__ int f32_base(int exponent) { return max(exponent - (127 << 20), 0); }

constexpr int AS_IS = 896 << 20;

template <int D>
__device__ __forceinline__ double field_of(const Prim &q, int f) {
    // gradient order of MeshlessScheme.cpp:114-120: rho, vx, vy, (vz), P
    if (f == 0) return q.rho;
    if (f == 1) return q.vx;
    if (f == 2) return q.vy;
    if (D == 3 && f == 3) return q.vz;
    return q.P;
}

//
// With dtbits (adaptive time step), the first pass over the neighbours also
// runs Particles::compGlobalTimestep (Particles.cpp:1446-1485) for the
// particle, as k_timestep does (real neighbours only, v_sig from
// numeric_limits<double>::min(), the same expressions), on the positions and
// velocities that pass loads anyway; the per-particle dt goes into the
// per-member minimum (warp reduction, then one atomicMin on its bit pattern).
// Bound: the FP64 pipe (85 % active on Sedov 64^3, 1610 instructions per
// particle, 41 per neighbour) and, at 12 warps per SM, the latency of the
// gathers.  One gather of the neighbours' records instead of three (the sums and
// the neighbours' extrema), the next one's in flight while one is summed: Sedov
// 128^3 8.29 -> 6.51 ms, 64 KH members 1.55 -> 1.18 ms, KH 100^2 93 -> 64 us
// (with the time step's kernel).  Register caps, Sedov 128^3: 6.62 ms at 160 and
// 6.82 at 128 registers (a spill that 16 warps do not make up for), 7.21 at 200;
// 64 KH members: 1.23 / 1.19 / 1.30 ms at 128 / 144 / 168.  The products of the offsets
// on the integer pipe (xmul) made it slower, 7.34 ms: the chain per neighbour
// gets longer.  Blocks of up to 256 threads.  L lanes share a particle: each takes
// every L-th neighbour, sums and extrema are reduced across them (grad_lanes).
#ifndef MLH_GRAD_MAXREG
#define MLH_GRAD_MAXREG 168
#endif
#ifndef MLH_GRAD_MAXREG_2D
#define MLH_GRAD_MAXREG_2D 144
#endif
#define MLH_GRAD_BOUNDS __maxnreg__(D == 3 ? MLH_GRAD_MAXREG : MLH_GRAD_MAXREG_2D)
// Reduction over the L lanes of a particle (the same bits on each of them).
template <int L, class T, class F>
__device__ __forceinline__ T lanes_reduce(unsigned mask, T v, F f) {
#pragma unroll
    for (int o = 1; o < L; o *= 2) v = f(v, __shfl_xor_sync(mask, v, o));
    return v;
}
template <int D, int L>
__global__ void MLH_GRAD_BOUNDS k_gradients(Params p, const Member *__restrict__ members,
                                                   const int *__restrict__ memberOf, const GridInfo *grids,
                                                   const Prim *prim, Geo *geo,
                                                   const uint32_t *nbr, const double *ww,
                                                   const int *noi, const int *noiImg,
                                                   Grad *grad, Grad *gradRaw,
                                                   double *psi,
                                                   unsigned long long *dtbits,
                                                   const int *faceOff, int *faceOf,
                                                   FaceRef *faces, unsigned *status,
                                                   int fp32_filters,
                                                   const float4 *velf, float *dtlo,
                                                   unsigned *dtcap) {
    step_begin();
    constexpr int NF = D + 2;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1);
    const unsigned mates = L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane - sub);   // the particle's lanes
    if (step_aborted(status)) return;   // no valid lists
    // warp-uniform loop: every lane takes part in the time-step reduction
    for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) & ~31) / L; i0 < p.n; i0 += gridDim.x * blockDim.x / L) {
      const int i = i0 + lane / L;
      int mi = -1;
      double dti = DBL_MAX_;
      float dthi = FLT_INF_;   // with dtlo: upper bound on the particle's dt
      if (i < p.n) {
        // with faceOff, the particle's face links first (link_particle):
        // integer searches whose load latency the other warps' FP64 work
        // hides, and whose registers are free again before the passes below
        if (faceOff && sub == 0) link_particle(i, p, nbr, noi, noiImg, faceOff, faceOf, faces, status);
        mi = memberOf ? memberOf[i] : 0;
        const double hq = p.adaptive_h ? p.hp[i] : members[mi].h;   // quadrature-point radius
        const Prim pi = prim[i];
        const size_t base = (size_t)i * p.K;
        const int nr = noi[i];
        const int tot = nr + noiImg[i];
        const bool want_dt = dtbits != nullptr;
        const double ci = want_dt ? geo[i].c : 0.;
        double vSig = DBL_MIN_;
        // the time step's single-precision filter (dtlo): bounds on v_sig
        // = max_j (c_i + c_j - min(0, v_ij . x_ij / r_ij)) over the real
        // neighbours from their offsets and the packed velocities and sound speeds
        const bool want_dtf = dtlo != nullptr;
        float4 vif = make_float4(0.f, 0.f, 0.f, 0.f);
        float vlo = 0.f, vhi = 0.f;
        bool dt_exact = false;   // no usable bound: the particle is always a candidate
        if (want_dtf) vif = velf[i];
        // One gather of every neighbour's record: E' = sum_j d d^T W with d =
        // x_j - x_i from the search (psi holds it), and S_f = sum_j (f_j - f_i)
        // d W, of which the gradient is E'^-1 S_f: psi~_j(x_i) = E_i^-1 d W V_i =
        // E'^-1 d W (E_i = V_i E': V_i cancels), so that neither the second
        // gather nor the weighting of every neighbour by psi~ is needed.
        double E[9] = {0., 0., 0., 0., 0., 0., 0., 0., 0.};
        double gr[NF][3], fi[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) { fi[f] = field_of<D>(pi, f); gr[f][0] = gr[f][1] = gr[f][2] = 0.; }
        // extrema of the neighbours' values for the slope limiter, as integer
        // keys (ord_key): the comparisons of the reference's if (max < f) max = f
        // stay off the FP64 pipe
        long long mxN[NF], mnN[NF];
        const long long kmin = ord_key(DBL_MIN_), kmax = ord_key(DBL_MAX_);
#pragma unroll
        for (int f = 0; f < NF; ++f) { mxN[f] = kmin; mnN[f] = kmax; }
        // the next neighbour's record is on its way while this one is summed
        uint32_t en = sub < tot ? nbr[base + sub] : 0u, en2 = sub + L < tot ? nbr[base + sub + L] : 0u;
        Prim pn = prim[en & IDX_MASK];
        float4 vn = want_dtf ? velf[en & IDX_MASK] : vif;
        for (int s = sub; s < tot; s += L) {
            const uint32_t e = en;
            const Prim pj = pn;
            const float4 vj = vn;
            en = en2;
            pn = prim[en & IDX_MASK];
            if (want_dtf) vn = velf[en & IDX_MASK];
            en2 = s + 2 * L < tot ? nbr[base + s + 2 * L] : 0u;
            const double wij = ww[base + s];
            const double *ds = psi + (base + s) * 3;
            double d[3], dp[3];
#pragma unroll
            for (int a = 0; a < D; ++a) { d[a] = ds[a]; dp[a] = mulr(d[a], wij); }
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int b = a; b < D; ++b) E[D * a + b] = fma(d[a], dp[b], E[D * a + b]);
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double fj = field_of<D>(pj, f), df = subr(fj, fi[f]);
#pragma unroll
                for (int a = 0; a < D; ++a) gr[f][a] = fma(df, dp[a], gr[f][a]);
                const long long kj = ord_key(fj);
                if (mxN[f] < kj) mxN[f] = kj;
                if (mnN[f] > kj) mnN[f] = kj;
            }
            if (want_dt && s < nr) {
                // x_ij = x_i - x_j is the exact negation of d
                const double cj = geo[e & IDX_MASK].c;
                const double xij[3] = {-d[0], -d[1], D == 3 ? -d[2] : 0.};
                const double vij[3] = {subr(pi.vx, pj.vx), subr(pi.vy, pj.vy), subr(pi.vz, pj.vz)};
                const double vs = signal_speed<D>(dotD<D>(vij, xij), xij, addr(ci, cj));
                vSig = dlt(vSig, vs) ? vs : vSig;
            }
            if (want_dtf && s < nr) {
                // |vs - vs64| <= B: the inputs' roundings (eps |c|, eps |v|, 2 eps |d|
                // per offset), the estimate's own and the FP64 expression's, at
                // most eps (2 (c_i + c_j) + 2 vs + 12 V) with V = |v_i|_1 + |v_j|_1;
                // B is twice eps (2 (c_i + c_j) + 2 vs + 16 V).  Offsets are in units
                // of kernelSize, so that the unit of length does not matter (only
                // their direction does): an r above 1e-12 and a B above 1e-31 leave
                // what flushes to zero (2^-126 of an offset, 2^-149 of a product)
                // far below B.
                const float dx = trunc_f32(d[0], p.f32_base), dy = trunc_f32(d[1], p.f32_base),
                            dz = D == 3 ? trunc_f32(d[2], p.f32_base) : 0.f;
                const float wx = __fsub_rn(vif.x, vj.x), wy = __fsub_rn(vif.y, vj.y),
                            wz = D == 3 ? __fsub_rn(vif.z, vj.z) : 0.f;
                const float dvd = __fmaf_rn(wz, dz, __fmaf_rn(wy, dy, __fmul_rn(wx, dx)));   // v_ij . (x_j - x_i)
                const float r = __fsqrt_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
                // -min(0, v_ij . x_ij / r) with x_ij = -(x_j - x_i)
                const float T = dvd > 0.f ? __fdiv_rn(dvd, r) : 0.f;
                const float vs = __fadd_rn(__fadd_rn(vif.w, vj.w), T);
                const float V = fabsf(vif.x) + fabsf(vif.y) + fabsf(vif.z) + fabsf(vj.x) + fabsf(vj.y) + fabsf(vj.z);
                constexpr float EPS32 = 5.9604645e-8f;
                const float B = 2.f * EPS32 * (2.f * (vif.w + vj.w) + 2.f * vs + 16.f * V);
                dt_exact = dt_exact || !(r > 1e-12f) || !(r < 1e15f) || !(B > 1e-31f) || !(B < 1e30f);
                vlo = fmaxf(vlo, vs - B);
                vhi = fmaxf(vhi, vs + B);
            }
        }
        const auto addD = [](double a, double b) { return addr(a, b); };
        const auto maxF = [](float a, float b) { return fmaxf(a, b); };
        const auto minF = [](float a, float b) { return fminf(a, b); };
        const auto maxK = [](long long a, long long b) { return a < b ? b : a; };
        const auto minK = [](long long a, long long b) { return b < a ? b : a; };
        if (L > 1) {   // the lanes' sums, extrema and bounds
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int b = a; b < D; ++b) E[D * a + b] = lanes_reduce<L>(mates, E[D * a + b], addD);
#pragma unroll
            for (int f = 0; f < NF; ++f) {
#pragma unroll
                for (int a = 0; a < D; ++a) gr[f][a] = lanes_reduce<L>(mates, gr[f][a], addD);
                mxN[f] = lanes_reduce<L>(mates, mxN[f], maxK);
                mnN[f] = lanes_reduce<L>(mates, mnN[f], minK);
            }
            if (want_dt) vSig = lanes_reduce<L>(mates, vSig, [](double a, double b) { return dlt(a, b) ? b : a; });
            if (want_dtf) {
                vlo = lanes_reduce<L>(mates, vlo, maxF);
                vhi = lanes_reduce<L>(mates, vhi, maxF);
                dt_exact = (__ballot_sync(mates, dt_exact) & mates) != 0u;
            }
        }
        if (want_dt) dti = (p.adaptive_h ? p.cfl * p.hp[i] : members[mi].cfl_h) / vSig;
        if (want_dtf) {
            // dt = cfl_h / v_sig bounded below by the largest v_sig and above by
            // the smallest (rounded outward, with the FP64 quotient's and the
            // conversion's roundings); v_sig >= DBL_MIN when nothing is found
            const float ch = __double2float_rn(p.adaptive_h ? p.cfl * p.hp[i] : members[mi].cfl_h);
            constexpr float EPS32 = 5.9604645e-8f;
            float lo = 0.f;
            if (!dt_exact && nr > 0 && vhi > 0.f && vhi < FLT_INF_)
                lo = __fmul_rd(__fdiv_rd(ch, vhi), 1.f - 4.f * EPS32);
            if (!(lo < 1e38f)) lo = 0.f;   // below any cap
            if (!dt_exact && nr > 0 && vlo > 0.f)
                dthi = __fmul_ru(__fdiv_ru(ch, vlo), 1.f + 4.f * EPS32);
            if (sub == 0) dtlo[i] = dt_exact ? 0.f : lo;
            if (dt_exact) dthi = FLT_INF_;
        }
        invert_symmetric<D>(E);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            double S[3];
#pragma unroll
            for (int a = 0; a < D; ++a) S[a] = gr[f][a];
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double t = mulr(E[D * a], S[0]);
#pragma unroll
                for (int b = 1; b < D; ++b) t = fma(E[D * a + b], S[b], t);
                gr[f][a] = t;
            }
        }
        if (gradRaw && sub == 0) {
            Grad graw;
            for (int k = 0; k < 16; ++k) graw.g[k] = 0.;
            for (int k = 0; k < 8; ++k) graw.t[k] = 0.;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                int slot = (f == NF - 1) ? 4 : f;
#pragma unroll
                for (int a = 0; a < D; ++a) graw.g[slot * 3 + a] = gr[f][a];
            }
            gradRaw[i] = graw;
        }
        // B_i = E_i^-1 = E'^-1 / V_i = E'^-1 omega_i (kept for inspection); then
        // E'^-1 V_i, of which V_i psi~_j(x_i) = (E'^-1 V_i) d W
        {
            const double omega_i = geo[i].omega, V_i = geo[i].V;
#pragma unroll
            for (int k = 0; k < D * D; ++k)
                if (sub == 0) geo[i].B[k] = mulr(E[k], omega_i);
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int b = a; b < D; ++b) E[D * a + b] = E[D * b + a] = mulr(E[D * a + b], V_i);
        }
        // V_i psi~_j(x_i) of a slot, for the face kernel's A_ij, over its offset
        auto store_psi = [&](int s, const double *d) {
            double *po = psi + (base + s) * 3;
            const double wij = ww[base + s];
            double dp[3];
#pragma unroll
            for (int a = 0; a < D; ++a) dp[a] = mulr(d[a], wij);
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double t = mulr(E[D * a], dp[0]);
#pragma unroll
                for (int b = 1; b < D; ++b) t = fma(E[D * a + b], dp[b], t);
                po[a] = t;
            }
        };
        if (p.slope) {
            // extrema of the face-point values, as integer keys
            long long mxM[NF], mnM[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) { mxM[f] = kmin; mnM[f] = kmax; }
            // face point x_ij = x_i + c (x_j - x_i): c = 1/2 (first-order
            // quadrature point) or h/4 (the reference's other choice);
            // f_ij = f_i + grad f . (x_ij - x_i) as one FMA chain from f_i, with
            // the gradients scaled by c for the pass instead of every offset
            // (for c = 1/2 both the scaling and its undoing are exact)
            const double cq = p.foqp ? .5 : hq / 4.;
            const double icq = p.foqp ? 2. : 1. / cq;
            if (p.foqp) {   // the halving and doubling on the integer pipe
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] = half_of(gr[f][a]);
            } else {
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] *= cq;
            }
            // one neighbour's f_ij of every field, into the extrema (its offset d)
            auto exact_slot = [&](const double *d) {
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    double fij = fma(gr[f][0], d[0], fi[f]);
#pragma unroll
                    for (int a = 1; a < D; ++a) fij = fma(gr[f][a], d[a], fij);
                    const long long kij = ord_key(fij);
                    if (mxM[f] < kij) mxM[f] = kij;
                    if (mnM[f] > kij) mnM[f] = kij;
                }
            };
            if (!(fp32_filters & MLH_FILTER_SLOPE)) {
                for (int s = sub; s < tot; s += L) {
                    const double *ds = psi + (base + s) * 3;
                    const double d[3] = {ds[0], ds[1], D == 3 ? ds[2] : 0.};
                    exact_slot(d);
                    store_psi(s, d);
                }
            } else {
                // Single-precision filter (the FP64 pipe is the step's
                // bound; the FP32 pipe is 64 times wider).  The increment
                // q_j = (c grad f) . (x_j - x_i) is estimated in single
                // precision from the offsets; |f_ij - (f_i + q_j)| <= B_f for
                // every neighbour, B_f bounding the estimate's rounding
                // (offsets, gradients, the chain) and the FP64 chain's own.  The
                // neighbour with the largest f_ij then has q_j >= max_k q_k -
                // 2 B_f (and the smallest q_j <= min_k q_k + 2 B_f), so the FP64
                // chain runs only over the neighbours inside those windows (a
                // handful; every lane of a warp walks its own list): the same
                // extrema, bit for bit.  A field whose gradient is zero has
                // f_ij = f_i at every neighbour.  q_j and its bounds are in units of the
                // field's gradient, so that a gradient below the normal range of single
                // precision (a density in g/cm^3 over 10^18 cm) keeps its bits.
                float gf[NF][3];
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    const int gb = f32_base(top_exponent<D>(gr[f]));
#pragma unroll
                    for (int a = 0; a < 3; ++a) gf[f][a] = a < D ? trunc_f32(gr[f][a], gb) : 0.f;
                }
                auto offset_f = [&](int s, float *df, double *d) {
                    const double *ds = psi + (base + s) * 3;
#pragma unroll
                    for (int a = 0; a < D; ++a) { d[a] = ds[a]; df[a] = trunc_f32(d[a], AS_IS); }
                };
                auto incr = [&](int f, const float *d) {
                    float q = __fmul_rn(gf[f][0], d[0]);
#pragma unroll
                    for (int a = 1; a < D; ++a) q = __fmaf_rn(gf[f][a], d[a], q);
                    return q;
                };
                float hiQ[NF], loQ[NF], dmax = 0.f;
#pragma unroll
                for (int f = 0; f < NF; ++f) { hiQ[f] = -FLT_MAX_; loQ[f] = FLT_MAX_; }
                for (int s = sub; s < tot; s += L) {
                    float df[3];
                    double d[3];
                    offset_f(s, df, d);
#pragma unroll
                    for (int a = 0; a < D; ++a) dmax = fmaxf(dmax, fabsf(df[a]));
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        const float q = incr(f, df);
                        hiQ[f] = fmaxf(hiQ[f], q);
                        loQ[f] = fminf(loQ[f], q);
                    }
                }
                if (L > 1) {
                    dmax = lanes_reduce<L>(mates, dmax, maxF);
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        hiQ[f] = lanes_reduce<L>(mates, hiQ[f], maxF);
                        loQ[f] = lanes_reduce<L>(mates, loQ[f], minF);
                    }
                }
                // B_f = 16 eps32 S (dmax + 1e-30) + 12 u64 (|f_i| + S dmax) with S = sum
                // |c grad f| and dmax = max |x_j - x_i|: more than twice the sum of the
                // single-precision error, at most 7 eps32 S dmax (2 from the offset's
                // truncation, 2 from the gradient's, 3 from the chain) and 2^-126 S for
                // offsets flushed to zero, and the FP64 chain's, at most 4 u64 (|f_i| +
                // S dmax)
                constexpr float EPS32 = 5.9604645e-8f, U64 = 1.1102230e-16f;
                const float R = dmax * (1.f + 4.f * EPS32) + 1e-30f;
                float thHi[NF], thLo[NF];
                bool ok = dmax < 1e30f, flat[NF];
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    bool z = true;
                    float S = 0.f;
#pragma unroll
                    for (int a = 0; a < D; ++a) {
                        z = z && (__double_as_longlong(gr[f][a]) & 0x7FFFFFFFFFFFFFFFll) == 0;
                        S += fabsf(gf[f][a]);
                    }
                    flat[f] = z;
                    const int ge = top_exponent<D>(gr[f]);
                    ok = ok && ge < 0x7ff00000;   // no infinity or NaN among the gradients
                    const float fa = z ? 0.f : fabsf(trunc_f32(fi[f], f32_base(ge))) * (1.f + 4.f * EPS32);
                    const float SR = S * R;
                    ok = ok && SR < 1e36f && S < 1e36f && fa < 1e36f;   // false for NaN and infinity
                    const float B = 16.f * EPS32 * SR + 12.f * U64 * (fa + SR) + 1e-36f;
                    thHi[f] = z ? FLT_INF_ : hiQ[f] - 2.f * B;
                    thLo[f] = z ? -FLT_INF_ : loQ[f] + 2.f * B;
                }
                // the candidates as a bit mask, every lane walking its own afterwards
                // (taken where they stand, some lane of the warp would want nearly
                // every slot); slots from the 65th on are all candidates
                unsigned long long cand = 0ull;
                for (int s = sub; s < tot; s += L) {
                    float df[3];
                    double d[3];
                    offset_f(s, df, d);
                    bool c = !ok;
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        const float q = incr(f, df);
                        c = c || q >= thHi[f] || q <= thLo[f];
                    }
                    cand |= (unsigned long long)(c && s < 64) << (s & 63);
                    if (s >= 64) exact_slot(d);
                    store_psi(s, d);
                }
                // psi holds V_i psi~ now: the few candidates' offsets from the records
                const GridInfo &g = grids[mi];
                while (cand) {
                    const int s = __ffsll((long long)cand) - 1;
                    cand &= cand - 1ull;
                    const uint32_t e = nbr[base + s];
                    const Prim pj = prim[e & IDX_MASK];
                    double xj[3], d[3];
                    neighbour_pos<D>(e, pj, g, xj);
                    const double xi[3] = {pi.x, pi.y, pi.z};
#pragma unroll
                    for (int a = 0; a < D; ++a) d[a] = subr(xj[a], xi[a]);
                    exact_slot(d);
                }
                if (tot > 0) {
#pragma unroll
                    for (int f = 0; f < NF; ++f)
                        if (flat[f]) mxM[f] = mnM[f] = ord_key(fi[f]);
                }
            }
            if (L > 1) {
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    mxM[f] = lanes_reduce<L>(mates, mxM[f], maxK);
                    mnM[f] = lanes_reduce<L>(mates, mnM[f], minK);
                }
            }
            if (p.foqp) {
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] = twice(gr[f][a]);
            } else {
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] *= icq;
            }
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double xN = key_double(mxN[f]), nN = key_double(mnN[f]);
                const double xM = key_double(mxM[f]), nM = key_double(mnM[f]);
                double aMax = ref_abs(fdiv_rn(subr(xN, fi[f]), subr(xM, fi[f])), p.int_abs);
                double aMin = ref_abs(fdiv_rn(subr(fi[f], nN), subr(fi[f], nM)), p.int_abs);
                if (aMin <= aMax && p.beta * aMin < 1.) {
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] *= aMin;
                } else if (aMax <= aMin && p.beta * aMax < 1.) {
#pragma unroll
                    for (int a = 0; a < D; ++a) gr[f][a] *= aMax;
                }
            }
        }
        else {
            for (int s = sub; s < tot; s += L) {
                const double *ds = psi + (base + s) * 3;
                const double d[3] = {ds[0], ds[1], D == 3 ? ds[2] : 0.};
                store_psi(s, d);
            }
        }
        Grad go;
#pragma unroll
        for (int k = 0; k < 16; ++k) go.g[k] = 0.;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            int slot = (f == NF - 1) ? 4 : f;   // P always at slot 4
#pragma unroll
            for (int a = 0; a < D; ++a) go.g[slot * 3 + a] = gr[f][a];
        }
        // div v of the limited gradients, in the face kernel's order
        go.g[15] = D == 3 ? (go.g[3] + go.g[7]) + go.g[11] : go.g[3] + go.g[7];
        {   // the sources of the half-step prediction
            const double *G = go.g;
            const double div = go.g[15], irho = geo[i].irho;
            const double src[5] = {mulr(pi.rho, div), mulr(p.gamma * pi.P, div), mulr(G[12], irho), mulr(G[13], irho),
                                   mulr(G[14], irho)};
#pragma unroll
            for (int f = 0; f < 8; ++f) go.t[f] = f < D + 2 ? src[f < 5 ? f : 0] : 0.;
        }
        if (sub == 0) grad[i] = go;
      }   // i < p.n
      if (dtlo) {
        // the least upper bound on dt of each simulation (positive floats
        // order as their bit patterns)
        const int m0 = __shfl_sync(0xffffffffu, mi, 0);
        if (__all_sync(0xffffffffu, mi == m0)) {
            float best = dthi;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && m0 >= 0 && best < FLT_INF_) atomicMin(dtcap + m0, __float_as_uint(best));
        } else if (mi >= 0 && dthi < FLT_INF_) {
            atomicMin(dtcap + mi, __float_as_uint(dthi));
        }
      }
      if (dtbits) {
        // the minimum over particles does not depend on the order of the
        // atomicMin calls: a warp inside one simulation reduces first and
        // issues one atomic; a warp that straddles two issues one per lane
        const int m0 = __shfl_sync(0xffffffffu, mi, 0);
        if (__all_sync(0xffffffffu, mi == m0)) {
            double best = dti;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && m0 >= 0 && best < DBL_MAX_) atomic_min_pos_double(dtbits + m0, best);
        } else if (mi >= 0 && dti < DBL_MAX_) {
            atomic_min_pos_double(dtbits + mi, dti);
        }
      }
    }
}

// Lanes per particle of k_gradients: more where the particles leave the SMs
// short of warps and the passes wait on their loads, one once a lane each
// fills them (the FP64 pipe then bounds them and the reductions only add to
// it).  The lines lie at 5, 9 and 10 warps per SM with 8, 4 and 2 lanes.  Time
// in us with 1 / 2 / 4 / 8 lanes (with the time step's kernel): KH 24^2 57 / 43 /
// 35 / 31, 50^2 56 / 43 / 35 / 33, 71^2 56 / 41 / 35 / 41, 100^2 60 / 46 / 44 / 69,
// 145^2 70 / 59 / 80 / 111, 180^2 77 / 75 / 105 / 157; Sedov 13^3 106 / 72 / 53 / 42,
// 17^3 106 / 70 / 56 / 64, 21^3 107 / 74 / 66 / 104, 25^3 114 / 97 / 121 / 155, 31^3
// 158 / 175 / 191 / 257.
int grad_lanes(int n, int sm_count) {
    const long long one = 32ll * sm_count;   // a warp per SM
    return 8ll * n <= 5 * one ? 8 : 4ll * n <= 9 * one ? 4 : 2ll * n <= 10 * one ? 2 : 1;
}

// ------------------------------------------------------------------ gather + update

// Particles::collectFluxes (Particles.cpp:1913-2011) in slot order, then
// Particles::updateStateAndPosition (:2013-2110).  The update is skipped when
// the neighbour search overflowed, so that the host can retry the step with
// more slots.
template <int D>
__global__ void __launch_bounds__(256) k_update(Params p, const int *__restrict__ memberOf,
                                                const GridInfo *grids, const int *noi,
                                                const int *noiImg, const int *faceOf,
                                                const double *Fface, const double *dtp,
                                                double *x, double *y, double *z,
                                                double *vx, double *vy, double *vz,
                                                double *m, double *u, float4 *posf,
                                                double *fluxSums, unsigned *status,
                                                int nmembers, double *simTime, int *stepsDone) {
    step_begin();
    // (the bits tested are not raised by this kernel: the same for every thread)
    const unsigned st0 = *(volatile const unsigned *)status;
    if (st0 & (ST_NGB_OVERFLOW | ST_CAPACITY | ST_TIMEOUT | ST_GRID)) return;
    if (blockIdx.x == 0) {   // simulation time of every member, the count of completed steps
        for (int mi = threadIdx.x; mi < nmembers; mi += blockDim.x) simTime[mi] += dtp[mi];
        if (threadIdx.x == 0) *stepsDone += 1;
    }
    double *X[3] = {x, y, z};
    double *Vv[3] = {vx, vy, vz};
    unsigned st_local = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += gridDim.x * blockDim.x) {
        const int sim = memberOf ? memberOf[i] : 0;
        const double dt = dtp[sim];
        const size_t base = (size_t)i * p.K;
        const int tot = noi[i] + noiImg[i];
        double mF = 0., eF = 0., vF[3] = {0., 0., 0.};
        // four slots at a time: their face ids in one 16-byte load (K is a
        // multiple of 4) and all twelve flux loads issued before the sums,
        // which still run in slot order
        const int4 *fo4 = reinterpret_cast<const int4 *>(faceOf + base);
        for (int s0 = 0; s0 < tot; s0 += 4) {
            const int4 f4 = fo4[s0 >> 2];
            const int fos[4] = {f4.x, f4.y, f4.z, f4.w};
            double2 fa[4], fb[4], fc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int fo = fos[k];
                const int af = fo > 0 ? fo : -fo;
                if (s0 + k < tot && fo != 0 && af <= p.faces_cap) {
                    const double2 *src = reinterpret_cast<const double2 *>(Fface + (size_t)(af - 1) * 6);
                    fa[k] = src[0]; fb[k] = src[1]; fc[k] = src[2];
                } else {
                    fa[k] = fb[k] = fc[k] = make_double2(0., 0.);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int fo = fos[k];
                const int af = fo > 0 ? fo : -fo;
                if (!(s0 + k < tot && fo != 0 && af <= p.faces_cap)) {
                    if (s0 + k < tot && fo == 0) st_local |= ST_ASYMMETRIC;   // a slot that no face found
                    continue;
                }
                // the flux with the slot's sign: the sign bit flipped on the
                // integer pipe for a copied face, so that both kinds of slot
                // share one set of additions (x + (-f) is the same double as
                // adding the negated flux)
                const long long sg = fo > 0 ? 0ll : (long long)0x8000000000000000ull;
                auto sgn = [sg](double f) { return __longlong_as_double(__double_as_longlong(f) ^ sg); };
                mF += sgn(fa[k].x); vF[0] += sgn(fb[k].x); vF[1] += sgn(fb[k].y);
                if (D == 3) vF[2] += sgn(fc[k].x);
                eF += sgn(fa[k].y);
            }
        }
        if (fluxSums) {
            fluxSums[(size_t)i * 5 + 0] = mF;
            fluxSums[(size_t)i * 5 + 1] = eF;
            fluxSums[(size_t)i * 5 + 2] = vF[0];
            fluxSums[(size_t)i * 5 + 3] = vF[1];
            fluxSums[(size_t)i * 5 + 4] = vF[2];
        }
        double mi = m[i], ui = u[i];
        double vo[3] = {vx[i], vy[i], D == 3 ? vz[i] : 0.};
        double Q0 = D == 3 ? mi * (ui + .5 * (vo[0] * vo[0] + vo[1] * vo[1] + vo[2] * vo[2]))
                           : mi * (ui + .5 * (vo[0] * vo[0] + vo[1] * vo[1]));
        double Qv[3] = {mi * vo[0], mi * vo[1], mi * vo[2]};
        if (!p.mfm) mi -= dt * mF;
        // sign and NaN tests on the bit patterns; one reciprocal of the mass
        const long long mb_ = __double_as_longlong(mi);
        if (mb_ <= 0) st_local |= ST_NEG_MASS;   // mi <= 0 (or a negative NaN)
        const double imi = frcp(mi);
        double vn[3];
#pragma unroll
        for (int a = 0; a < D; ++a) { Qv[a] -= dt * vF[a]; vn[a] = Qv[a] * imi; }
        Q0 -= dt * eF;
        double un = D == 3 ? Q0 * imi - .5 * (vn[0] * vn[0] + vn[1] * vn[1] + vn[2] * vn[2])
                           : Q0 * imi - .5 * (vn[0] * vn[0] + vn[1] * vn[1]);
        const long long ub = __double_as_longlong(un);
        if (ub <= 0) st_local |= ST_NEG_ENERGY;
        if ((ub & 0x7FFFFFFFFFFFFFFFll) > 0x7FF0000000000000ll || (mb_ & 0x7FFFFFFFFFFFFFFFll) > 0x7FF0000000000000ll)
            st_local |= ST_NAN;
        m[i] = mi;
        u[i] = un;
#pragma unroll
        for (int a = 0; a < D; ++a) Vv[a][i] = vn[a];
        double xn[3] = {0., 0., 0.};
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double xa = X[a][i];
            if (p.move) {
                xa += vo[a] * dt;
                if (p.periodic) {
                    // the box tests on integer keys (ord_key), off the FP64 pipe
                    const double lo = grids[sim].lo[a], hi = grids[sim].hi[a];
                    if (dlt(xa, lo)) xa = hi - (lo - xa);
                    else if (!dlt(xa, hi)) xa = lo + (xa - hi);
                }
                X[a][i] = xa;
            }
            xn[a] = xa;
        }
        posf[i] = make_float4((float)xn[0], (float)xn[1], (float)xn[2], 0.f);
    }
    for (int o = 16; o > 0; o >>= 1) st_local |= __shfl_xor_sync(0xffffffffu, st_local, o);
    if ((threadIdx.x & 31) == 0 && st_local) flag(status, st_local);
}

template <int D>
__global__ void k_pack_posf(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
                            int n, float4 *__restrict__ posf) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        posf[i] = make_float4((float)x[i], (float)y[i], D == 3 ? (float)z[i] : 0.f, 0.f);
}

// ------------------------------------------------------------------ launchers

// The face passes and the Riemann batch, one translation unit per solver
// (mlh_faces.cuh).
template <int D, int ROOT>
void launch_faces(StepArgs &a);
template <int D, int ROOT>
void launch_riemann_batch(int n, const RiemannConsts &rc, int mfm, const double *Wi, const double *Wj,
                          const double *vFrame, const double *Aij, double *F, int *iters, unsigned *status,
                          cudaStream_t s);

void riemann_batch(int dim, int n, double gamma, double rtol, int max_iter, int mfm, const double *Wi,
                   const double *Wj, const double *vFrame, const double *Aij, double *F, int *iters,
                   unsigned *status, cudaStream_t s) {
    const RiemannConsts rc = make_riemann_consts(gamma, rtol, max_iter);
#define MLH_RB(DD, R) launch_riemann_batch<DD, R>(n, rc, mfm, Wi, Wj, vFrame, Aij, F, iters, status, s)
    if (dim == 2) { if (rc.root == 5) MLH_RB(2, 5); else if (rc.root == 7) MLH_RB(2, 7); else MLH_RB(2, 0); }
    else { if (rc.root == 5) MLH_RB(3, 5); else if (rc.root == 7) MLH_RB(3, 7); else MLH_RB(3, 0); }
#undef MLH_RB
}

// Particles::getDomainLimits + Domain::createGrid + assignParticlesAndCells
// (Particles.cpp:228-322, Domain.cpp:9-54): grids, cell of every particle,
// cell lists sorted by particle index.
template <int D>
void launch_binning(StepArgs &a) {
    const Params &p = a.p;
    cudaStream_t s = a.stream;
    const int T = 128;
    const int blocksN = (p.n + T - 1) / T;
    if (a.tune.persistent_binning && a.bar && a.bin_blocks > 0) {
        // one cooperative launch of at most the blocks resident at once
        cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), s);
        GridBar bar{a.bar, a.bar + 1, (unsigned)a.bin_blocks + a.bar_extra, a.bar_spin};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(a.bin_blocks);
        cfg.blockDim = dim3(PB_T);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k_binning<D>, (const double *)a.x, (const double *)a.y, (const double *)a.z, p,
                           (const Member *)a.members, a.memberOf, a.nmembers, a.bpm, a.boundsPart, a.grids,
                           a.cellTotal, a.cell, a.cellCount, a.cellStart, a.cellFill, a.cellList, a.scanTiles,
                           a.scanTotal, a.status, a.dtbits, a.dtcap, bar);
        return;
    }
    launch_dep(k_bounds_partial<D>, a.nmembers * a.bpm, BOUNDS_T, 0, s, a.x, a.y, a.z, p, a.members, a.bpm, a.boundsPart,
                                                                a.cellCount, a.cellFill);
    launch_dep(k_bounds_final<D>, 1, BOUNDS_T, 0, s, a.x, a.y, a.z, a.boundsPart, a.bpm, p, a.members, a.nmembers, a.grids,
                                             a.cellTotal, a.status, a.dtbits, a.dtcap);
    launch_dep(k_assign<D>, blocksN, T, 0, s, a.x, a.y, a.z, p.n, a.memberOf, a.grids, a.cell, a.cellCount, a.status);
    exclusive_scan(a.cellCount, p.ncells_cap, a.cellStart, a.scanTiles, a.scanTotal, s, true);
    launch_dep(k_fill_cells, blocksN, T, 0, s, a.cell, p.n, a.cellStart, a.cellFill, a.cellList, a.status);
    const long long sortBlocks = ((long long)p.ncells_cap + 7) / 8;
    launch_dep(k_sort_cells, (int)(sortBlocks < a.sm_count * 8ll ? sortBlocks : a.sm_count * 8ll), 256, 0, s, a.cellTotal, a.cellStart, a.cellList, a.status);
}

// Smoothing lengths of every particle on the current grid (k_hsolve).
template <int D>
void launch_hsolve(StepArgs &a) {
    const Params &p = a.p;
    cudaStream_t s = a.stream;
    cudaMemsetAsync(a.hstat, 0, 2 * sizeof(unsigned long long), s);
    // eight rounds of resident blocks: cells take uneven numbers of iterations
    // (61^3: 1158 us at two rounds, 1020 at eight and more)
    const int warps_total = 4 * a.sm_count * a.tune.nns_warps_per_sm;
    const int most = (p.ncells_cap + NNS_WARPS - 1) / NNS_WARPS;
    int blocks = (warps_total + NNS_WARPS - 1) / NNS_WARPS;
    if (blocks > most) blocks = most;
    const size_t smem = hsolve_smem_bytes(p.K);
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_hsolve<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_hsolve<D><<<blocks, NNS_WARPS * 32, smem, s>>>(p, a.members, a.memberOf, a.grids, a.x, a.y, a.z, a.posf, a.cellTotal,
                                                     a.cellStart, a.cellList, a.hp, a.hpf, a.neff, a.hstat, a.status);
}

// The neighbour search's split and grid.  Parts per cell: with fewer than two cells
// per resident warp a cell's particles go to several warps (each takes the candidates
// again), in batches that split a mean cell evenly.  The grid: the tuned warps per SM
// in whole rounds of resident blocks, grid-stride over the units.
SearchShape search_shape(const StepArgs &a) {
    const Params &p = a.p;
    const long long cells = a.cells_est > 0 ? a.cells_est : 1, resident = (long long)a.sm_count * NNS_WARPS * MLH_NNS_MINB;
    long long nsplit = (2 * resident + cells - 1) / cells;
    nsplit = nsplit < 1 ? 1 : nsplit > 8 ? 8 : nsplit;
    if ((long long)p.ncells_cap * nsplit > 0x7fffffffll) nsplit = 1;
    long long pb = nsplit > 1 ? (p.n + cells * nsplit - 1) / (cells * nsplit) : NNS_PB;
    pb = pb < 1 ? 1 : pb > NNS_PB ? NNS_PB : pb;
    int per_sm = (a.tune.nns_warps_per_sm + NNS_WARPS - 1) / NNS_WARPS;
    per_sm = (per_sm + MLH_NNS_MINB - 1) / MLH_NNS_MINB * MLH_NNS_MINB;
    const long long most = ((long long)p.ncells_cap * nsplit + NNS_WARPS - 1) / NNS_WARPS;
    const long long want = (long long)a.sm_count * per_sm;
    return {(int)nsplit, (int)pb, (int)(want < most ? want : most < 1 ? 1 : most)};
}

// Threads per block of the gradients: with several lanes per particle there are few
// blocks, and small ones spread evenly (KH 100^2: 49 -> 44 us).
int gradients_threads(const StepArgs &a) {
    return grad_lanes(a.p.n, a.sm_count) > 1 && a.tune.grad_threads > 64 ? 64 : a.tune.grad_threads;
}

template <int D>
void launch_step(StepArgs &a) {
    const Params &p = a.p;
    cudaStream_t s = a.stream;
    const int T = 128;
    const int blocksN = (p.n + T - 1) / T;
    auto tick = [&](int id) { if (a.timer) a.timer(a.timer_ctx, id, 0); };
    auto tock = [&](int id) { if (a.timer) a.timer(a.timer_ctx, id, 1); };

    tick(KT_GRID);
    launch_binning<D>(a);
    tock(KT_GRID);

    if (p.adaptive_h) {
        tick(KT_HSOLVE);
        launch_hsolve<D>(a);
        tock(KT_HSOLVE);
    }

    const int gl = grad_lanes(p.n, a.sm_count);
    // Kernels started before their predecessors have ended (launch_dep): the
    // binning always; the rest only where particles are few.  In full grids the
    // early blocks take the SM slots that the links on the second stream fill
    // (16 blasts in 48^3: 1543 us a step, 1600 with every kernel early, 1536 so).
    // KH 24^2 113 -> 91 us a step, KH 100^2 165 -> 162, Sedov 33^3 557 -> 542.
    const bool early = gl > 1;
    tick(KT_NNS);
    {
        const size_t smem = nns_smem_bytes(p.K);
        const SearchShape sh = search_shape(a);
        auto run = [&](auto kern) {
            if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            launch_kernel(early, kern, sh.blocks, NNS_WARPS * 32, smem, s,
                p, sh.nsplit, sh.batch, a.members, a.memberOf, a.grids, a.x, a.y, a.z, a.posf, a.vx, a.vy, a.vz, a.m,
                a.u, a.cellTotal, a.cellStart, a.cellList, a.nbr, a.psi, a.ww, a.noi, a.noiImg, a.faceCnt, a.prim,
                a.geo, a.velf, a.status);
        };
        if (p.adaptive_h) run(k_neighbours<D, true>);
        else run(k_neighbours<D, false>);
    }
    tock(KT_NNS);

    // the face links (integer work) need only the neighbour lists: without
    // per-kernel timing they run on the second stream while the time step and
    // the gradients keep the FP64 pipe busy
    // link_overlap 2: the links inside the gradients kernel (after the scan of
    // the canonical counts); 1: on the second stream beside the gradients;
    // 0: in order
    const bool fused = a.tune.link_overlap == 2 && !a.stop_after_gradients;
    const bool overlap = !fused && a.stream2 && !a.timer && !a.stop_after_gradients && a.tune.link_overlap == 1;
    auto grid_of = [&](long long threads) {   // blocks of 256 threads, at most one round of a full GPU
        const long long b = (threads + 255) / 256, most = a.sm_count * 8ll;
        return (int)(b < 1 ? 1 : b < most ? b : most);
    };
    auto launch_links = [&](cudaStream_t ls) {
        exclusive_scan(a.faceCnt, p.n, a.faceOff, a.scanTiles, a.scanTotal, ls);
        k_link_own<<<grid_of(32ll * p.n), 256, 0, ls>>>(p, a.nbr, a.noi, a.noiImg, a.faceOff, a.faceOf, a.faces,
                                                        a.status);
        k_link<<<grid_of((long long)a.faces_cap), 256, 0, ls>>>(p, a.nbr, a.noi, a.noiImg, a.faceOff + p.n, a.faceOf,
                                                                a.faces, a.status);
    };
    if (overlap) {
        cudaEventRecord(a.ev_fork, s);
        cudaStreamWaitEvent(a.stream2, a.ev_fork, 0);
        launch_links(a.stream2);
        cudaEventRecord(a.ev_join, a.stream2);
    }

    // the time step runs inside the gradients' first neighbour pass
    // (k_gradients with dtbits; k_timestep, the separate kernel of the same
    // arithmetic, is the fallback when the time step is timed on its own)
    // with the single-precision filters the gradients kernel bounds every
    // particle's dt (dtlo, and the least upper bound per simulation in dtcap) and k_timestep evaluates v_sig in FP64
    // for the particles whose bound reaches it
    const bool dt_filter = p.adaptive && !a.separate_dt && (a.tune.fp32_filters & MLH_FILTER_TIMESTEP) && a.velf &&
                           a.dtlo && a.dtcap;
    if (a.separate_dt) {
        tick(KT_DT);
        launch_dep(k_timestep<D>, (p.n + 255) / 256, 256, 0, s, p, a.members, a.memberOf, a.prim, a.geo, a.nbr, a.noi,
                                                        a.dtbits, nullptr, nullptr, a.nmembers, a.dt_max, a.dt,
                                                        a.arrived, a.status);
        tock(KT_DT);
    }
    tick(KT_GRAD);
    if (fused) {
        exclusive_scan(a.faceCnt, p.n, a.faceOff, a.scanTiles, a.scanTotal, s);
        cudaMemsetAsync(a.faces, 0xff, sizeof(FaceRef) * a.faces_cap, s);
    }
    const int gT = gradients_threads(a);
    const int gB = (int)(((long long)p.n * gl + gT - 1) / gT);
#define MLH_GRAD_ARGS                                                                                          \
    a.members, a.memberOf, a.grids, a.prim, a.geo, a.nbr, a.ww, a.noi, a.noiImg, a.grad, a.gradRaw, a.psi,     \
        (p.adaptive && !a.separate_dt && !dt_filter) ? a.dtbits : nullptr, fused ? a.faceOff : nullptr, a.faceOf, \
        a.faces, a.status, a.tune.fp32_filters, a.velf, dt_filter ? a.dtlo : nullptr, a.dtcap
    auto gradients = [&](auto kern) { launch_kernel(early, kern, gB, gT, 0, s, p, MLH_GRAD_ARGS); };
    if (gl == 8) gradients(k_gradients<D, 8>);
    else if (gl == 4) gradients(k_gradients<D, 4>);
    else if (gl == 2) gradients(k_gradients<D, 2>);
    else gradients(k_gradients<D, 1>);
#undef MLH_GRAD_ARGS
    if (dt_filter)
        launch_kernel(early, k_timestep<D>, (p.n + 255) / 256, 256, 0, s, p, a.members, a.memberOf, a.prim, a.geo,
                      a.nbr, a.noi, a.dtbits, a.dtlo, a.dtcap, a.nmembers, a.dt_max, a.dt, a.arrived, a.status);
    else
        launch_kernel(early, k_dt_final, 1, 128, 0, s, p, a.nmembers, a.dtbits, a.dt_max, a.dt, a.status);
    tock(KT_GRAD);
    if (a.stop_after_gradients) return;

    if (overlap) {
        cudaStreamWaitEvent(s, a.ev_join, 0);
    } else if (!fused) {
        tick(KT_LINK);
        launch_links(s);
        tock(KT_LINK);
    }

    tick(KT_FACES);
    if (a.root == 5) launch_faces<D, 5>(a);
    else if (a.root == 7) launch_faces<D, 7>(a);
    else launch_faces<D, 0>(a);
    tock(KT_FACES);

    tick(KT_UPDATE);
    launch_kernel(early, k_update<D>, blocksN, T, 0, s, p, a.memberOf, a.grids, a.noi, a.noiImg, a.faceOf, a.Fface, a.dt, a.x, a.y,
                                      a.z, a.vx, a.vy, a.vz, a.m, a.u, a.posf, a.fluxSums, a.status, a.nmembers, a.simTime,
                                      a.stepsDone);
    tock(KT_UPDATE);
}

void launch_grid_bounds(const double *x, const double *y, const double *z, const Params &p,
                        const Member *members, int nmembers, int bpm, double *partials, GridInfo *grids,
                        int *cellTotal, unsigned *status, cudaStream_t s) {
    const int blocks = nmembers * bpm;
    if (p.dim == 2) {
        launch_dep(k_bounds_partial<2>, blocks, BOUNDS_T, 0, s, x, y, z, p, members, bpm, partials, nullptr, nullptr);
        launch_dep(k_bounds_final<2>, 1, BOUNDS_T, 0, s, x, y, z, partials, bpm, p, members, nmembers, grids, cellTotal, status,
                                                 nullptr, nullptr);
    } else {
        launch_dep(k_bounds_partial<3>, blocks, BOUNDS_T, 0, s, x, y, z, p, members, bpm, partials, nullptr, nullptr);
        launch_dep(k_bounds_final<3>, 1, BOUNDS_T, 0, s, x, y, z, partials, bpm, p, members, nmembers, grids, cellTotal, status,
                                                 nullptr, nullptr);
    }
}

int binning_blocks(int dim, int sm_count) {
    int per_sm = 0;
    cudaError_t e = dim == 3 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_binning<3>, PB_T, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_binning<2>, PB_T, 0);
    if (e != cudaSuccess || per_sm < 1) return 0;
    return per_sm * sm_count;
}

void step(StepArgs &a) {
    if (a.p.dim == 2) launch_step<2>(a);
    else launch_step<3>(a);
}

void smoothing_lengths(StepArgs &a) {
    if (a.p.dim == 2) { launch_binning<2>(a); launch_hsolve<2>(a); }
    else { launch_binning<3>(a); launch_hsolve<3>(a); }
}

void pack_posf(const double *x, const double *y, const double *z, int n, int dim, float4 *posf, cudaStream_t s) {
    int blocks = (n + 255) / 256;
    if (blocks < 1) blocks = 1;
    if (dim == 2) k_pack_posf<2><<<blocks, 256, 0, s>>>(x, y, z, n, posf);
    else k_pack_posf<3><<<blocks, 256, 0, s>>>(x, y, z, n, posf);
}

const char *kernel_timer_name(int id) {
    switch (id) {
        case KT_GRID: return "grid_bin";
        case KT_NNS: return "neighbours_density";
        case KT_DT: return "timestep";
        case KT_GRAD: return "gradients_limiter";
        case KT_LINK: return "face_links";
        case KT_FACES: return "faces_riemann";
        case KT_UPDATE: return "gather_update";
        case KT_HSOLVE: return "smoothing_lengths";
    }
    return "?";
}

}  // namespace mlh
