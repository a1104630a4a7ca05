// CUDA kernels of the hot path (sm_100a). Built with -fmad=false and IEEE
// division / square root: see physics.cuh.
//
//   binning      k_bounds, k_bounds_final, k_cells, scan_*, k_scatter, k_sort_cells,
//                k_permute                         (NeighbourGrid::generate, NeighbourGrid.cpp:48-184)
//   contacts     k_nbr_count, k_nbr_fill           (NeighAccel::generateNeighbours, NeighAccel.h:25-137)
//   link ends    k_side_count, k_side_fill         (LinkAccelSide::generateLinks/sortSideData,
//                                                   LinkAccelSide.h:92-143,160-417)
//   timestep     k_force, k_integrate_gather       (CombinedAccel::iterateCombined + applyForce +
//                k_step, k_step_async,              linkUpdate, CombinedAccel.h:122-235)
//                k_step_items, k_integrate,
//                k_link_break, k_max_diff
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "kernels.h"
#include "physics.cuh"

namespace hidem {

// ------------------------------------------------------------------ helpers

template <class LP>
__device__ __forceinline__ PRec<LP> load_rec(const PRec<LP> *p) {
    PRec<LP> r;
    const int4 *src = reinterpret_cast<const int4 *>(p);
    int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(PRec<LP>) / 16); ++k) dst[k] = __ldg(src + k);
    return r;
}

// The first CHUNKS 16-byte chunks of a record that the kernel before may have written (the rest
// stays unset): plain loads, for kernels that are launched dependent (dependent_start).
template <class LP, int CHUNKS = (int)(sizeof(PRec<LP>) / 16)>
__device__ __forceinline__ PRec<LP> load_rec_written(const PRec<LP> *p) {
    PRec<LP> r;
    const int4 *src = reinterpret_cast<const int4 *>(p);
    int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) dst[k] = src[k];
    return r;
}

template <class LP>
__device__ __forceinline__ void store_rec(PRec<LP> *p, const PRec<LP> &r) {
    int4 *dst = reinterpret_cast<int4 *>(p);
    const int4 *src = reinterpret_cast<const int4 *>(&r);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(PRec<LP>) / 16); ++k) dst[k] = src[k];
}

__device__ __forceinline__ unsigned long long max_bits(float v) {
    return (unsigned long long)__float_as_uint(v);
}
__device__ __forceinline__ unsigned long long max_bits(double v) {
    return (unsigned long long)__double_as_longlong(v);
}

__device__ __forceinline__ void set_error(int *flag, int code) {
    if (flag) atomicCAS(flag, 0, code);
}

// Programmatic dependent launch: a timestep's kernels follow one another directly, and a kernel
// launched with launch_dependent is placed on the SMs while its predecessor's last CTAs run; it
// starts with dependent_start, which waits for that predecessor's memory (all of it: the wait
// ends when the predecessor has completed) before the first access, then lets its own successor
// be placed. Worth a launch's latency per kernel: 9.1 -> 8.2 us a step on
// 256 particles, 26.1 -> 23.3 us on 32,000 (two kernels a step).
// Such a kernel is resident while its predecessor still writes, so what the predecessor may
// write is not read-only for its lifetime: records, gather layout and forces are read with plain
// loads, which stay behind the wait (no __ldg, no const __restrict__; load_rec_written,
// load_body). The lists and constants are read through the read-only path, so the kernels that
// read them (k_force, k_step_items) are launched dependent only where the kernel before them is
// one of a timestep's own, none of which writes a list (`chained`); one that follows a rebuild, an
// upload or whatever came before the call is launched plainly.
__device__ __forceinline__ void dependent_start() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
static void launch_dependent(bool dependent, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s,
                             A &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = dependent ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ------------------------------------------------------------------ binning

// min / max that keep a NaN: fmin / fmax drop NaN operands, so one particle with a NaN
// coordinate would vanish from the bounds and then be binned from floor(NaN). With these
// a NaN anywhere reaches the result and the host refuses the rebuild. Equal to fmin /
// fmax for numbers.
__device__ __forceinline__ double nan_min(double a, double b) {
    return (a != a) ? a : ((b != b) ? b : fmin(a, b));
}
__device__ __forceinline__ double nan_max(double a, double b) {
    return (a != a) ? a : ((b != b) ? b : fmax(a, b));
}

// Per-block min / max of the three coordinates over all particles
// (ParticleData::getLimits, PLiB/ParticleData.h:47-59).
template <class LP>
__global__ void k_bounds(const PRec<LP> *__restrict__ rec, int n, double *__restrict__ partial) {
    double mn[3] = {INFINITY, INFINITY, INFINITY};
    double mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double *p = reinterpret_cast<const double *>(rec + i);
        double v[3] = {__ldg(p), __ldg(p + 1), __ldg(p + 2)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = nan_min(mn[k], v[k]);
            mx[k] = nan_max(mx[k], v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = nan_min(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = nan_max(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    }
    __shared__ double sm[32][6];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        for (int k = 0; k < 3; ++k) {
            sm[w][k] = mn[k];
            sm[w][3 + k] = mx[k];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int nw = blockDim.x >> 5;
        for (int k = 0; k < 3; ++k) {
            double a = sm[0][k], b = sm[0][3 + k];
            for (int j = 1; j < nw; ++j) {
                a = nan_min(a, sm[j][k]);
                b = nan_max(b, sm[j][3 + k]);
            }
            partial[blockIdx.x * 6 + k] = a;
            partial[blockIdx.x * 6 + 3 + k] = b;
        }
    }
}

// min / max are exact and idempotent, so the block's fold order (each thread starts from
// one partial, repeated ones counting twice) gives the serial fold's result
constexpr int kBoundsFinalThreads = 256;
__global__ void k_bounds_final(const double *__restrict__ partial, int nb, double *__restrict__ out) {
    __shared__ double red[6][kBoundsFinalThreads];
    const int t = threadIdx.x;
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = partial[(t % nb) * 6 + k];
    for (int b = t + kBoundsFinalThreads; b < nb; b += kBoundsFinalThreads)
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double u = partial[b * 6 + k];
            v[k] = (k < 3) ? nan_min(v[k], u) : nan_max(v[k], u);
        }
#pragma unroll
    for (int k = 0; k < 6; ++k) red[k][t] = v[k];
    __syncthreads();
    for (int w = kBoundsFinalThreads / 2; w > 0; w >>= 1) {
        if (t < w)
#pragma unroll
            for (int k = 0; k < 6; ++k)
                red[k][t] = (k < 3) ? nan_min(red[k][t], red[k][t + w]) : nan_max(red[k][t], red[k][t + w]);
        __syncthreads();
    }
    if (t < 6) out[t] = red[t][0];
}

// Cell colour of every slot and the per-cell counts (NeighbourGrid::getGridId /
// getGridColor / colourParticles, NeighbourGrid.cpp:25-33,116-161).
template <class LP>
__global__ void k_cells(const PRec<LP> *__restrict__ rec, int n, GridInfo g,
                        int *__restrict__ cellOf, int *__restrict__ cellCount, int *errorFlag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const PRec<LP> *p = rec + i;
    int ix = (int)floor((p->x - g.xMin) / g.h);
    int iy = (int)floor((p->y - g.yMin) / g.h);
    int iz = (int)floor((p->z - g.zMin) / g.h);
    long long c = (long long)ix + (long long)iy * g.X + (long long)iz * g.X * g.Y;
    if (c < 0 || c >= g.total) {
        set_error(errorFlag, 1);
        c = 0;
    }
    cellOf[i] = (int)c;
    atomicAdd(cellCount + c, 1);
}

// Exclusive prefix sum in three passes (block sums, scan of block sums, add).
constexpr int kScanBlock = 1024;  // elements per block (256 threads x 4)

template <class TI, class TO>
__global__ void k_scan_blocks(const TI *__restrict__ in, long long n, TO scaleBy,
                              TO *__restrict__ out, TO *__restrict__ blockSums) {
    __shared__ TO sh[kScanBlock];
    long long base = (long long)blockIdx.x * kScanBlock;
    for (int k = threadIdx.x; k < kScanBlock; k += blockDim.x) {
        long long i = base + k;
        sh[k] = (i < n) ? (TO)in[i] * scaleBy : (TO)0;
    }
    __syncthreads();
    // Hillis-Steele would cost log steps x 1024; a simple two-level scan instead:
    // each thread scans 4 consecutive elements, then a warp-level scan of thread totals.
    int t = threadIdx.x;
    TO local[4];
    TO run = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        local[k] = run;
        run += sh[t * 4 + k];
    }
    // inclusive scan of `run` over 256 threads
    TO v = run;
    int lane = t & 31, w = t >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        TO u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    __shared__ TO wsum[8];
    if (lane == 31) wsum[w] = v;
    __syncthreads();
    if (t == 0) {
        TO acc = 0;
        for (int j = 0; j < 8; ++j) {
            TO s = wsum[j];
            wsum[j] = acc;
            acc += s;
        }
    }
    __syncthreads();
    TO excl = v - run + wsum[w];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        long long i = base + t * 4 + k;
        if (i < n) out[i] = excl + local[k];
    }
    if (t == blockDim.x - 1) blockSums[blockIdx.x] = excl + run;
}

template <class TO>
__global__ void k_scan_sums(TO *__restrict__ sums, long long nb, TO *__restrict__ total) {
    // one block: sequential over chunks of 1024 with the same two-level scheme
    __shared__ TO carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (long long base = 0; base < nb; base += blockDim.x) {
        long long i = base + threadIdx.x;
        TO v = (i < nb) ? sums[i] : (TO)0;
        TO orig = v;
        int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            TO u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        __shared__ TO wsum[32];
        if (lane == 31) wsum[w] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            TO acc = 0;
            int nw = blockDim.x >> 5;
            for (int j = 0; j < nw; ++j) {
                TO s = wsum[j];
                wsum[j] = acc;
                acc += s;
            }
        }
        __syncthreads();
        TO excl = v - orig + wsum[w] + carry;
        if (i < nb) sums[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + orig;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

template <class TO>
__global__ void k_scan_add(TO *__restrict__ out, long long n, const TO *__restrict__ sums) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += sums[i / kScanBlock];
}

// Counting-sort placement, unstable inside a cell (fixed by k_sort_cells).
__global__ void k_scatter(const int *__restrict__ cellOf, int n, const int *__restrict__ cellStart,
                          int *__restrict__ cursor, int *__restrict__ perm) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cellOf[i];
    int pos = cellStart[c] + atomicAdd(cursor + c, 1);
    perm[pos] = i;
}

// Orders each cell's members by input index: the (colour, index) order of
// NeighbourGrid::generateIterationList (NeighbourGrid.cpp:163-184). One thread per cell
// sorts a cell of at most kSmallCell members by insertion (a lattice cell holds a few);
// a larger cell goes to a list that k_sort_big_cells sorts with one CTA per cell, so that
// no thread's work grows with the square of a crowded cell's population.
__global__ void k_sort_cells(const int *__restrict__ cellStart, const int *__restrict__ cellCount,
                             long long total, const int *__restrict__ origOld, int *__restrict__ perm,
                             int *__restrict__ bigList, int *__restrict__ bigCount) {
    long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= total) return;
    int cnt = cellCount[c];
    if (cnt < 2) return;
    if (cnt > kSmallCell) {
        bigList[atomicAdd(bigCount, 1)] = (int)c;
        return;
    }
    int s = cellStart[c];
    for (int a = 1; a < cnt; ++a) {
        int v = perm[s + a];
        int key = origOld ? origOld[v] : v;
        int b = a - 1;
        while (b >= 0 && (origOld ? origOld[perm[s + b]] : perm[s + b]) > key) {
            perm[s + b + 1] = perm[s + b];
            --b;
        }
        perm[s + b + 1] = v;
    }
}

// One CTA per listed cell (grid-stride over the list): the (key, member) pairs of the cell
// in shared memory, a bitonic sort over the next power of two, the members written back in
// key order. Keys are input indices (non-negative, distinct), so the order is the one the
// insertion sort gives. A cell of more than kBigCellCap members is left unsorted and sets
// `errorCode` in the error flag: the caller refuses the result.
__global__ void __launch_bounds__(kBigCellThreads)
    k_sort_big_cells(const int *__restrict__ cellStart, const int *__restrict__ cellCount,
                     const int *__restrict__ origOld, int *__restrict__ perm,
                     const int *__restrict__ bigList, const int *__restrict__ bigCount,
                     int *errorFlag, int errorCode) {
    __shared__ unsigned long long sk[kBigCellCap];
    const int nbig = *bigCount;
    for (int b = blockIdx.x; b < nbig; b += gridDim.x) {
        const int c = bigList[b];
        const int cnt = cellCount[c];
        const int s = cellStart[c];
        if (cnt > kBigCellCap) {
            if (threadIdx.x == 0) set_error(errorFlag, errorCode);
            continue;
        }
        int m = kSmallCell;
        while (m < cnt) m <<= 1;
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            if (i < cnt) {
                const int v = perm[s + i];
                const unsigned key = (unsigned)(origOld ? origOld[v] : v);
                sk[i] = ((unsigned long long)key << 32) | (unsigned)v;
            } else {
                sk[i] = ~0ull;
            }
        }
        __syncthreads();
        for (int k = 2; k <= m; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < m; i += blockDim.x) {
                    const int p = i ^ j;
                    if (p > i) {
                        const unsigned long long x = sk[i], y = sk[p];
                        const bool up = (i & k) == 0;
                        if (up ? (x > y) : (x < y)) {
                            sk[i] = y;
                            sk[p] = x;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) perm[s + i] = (int)(unsigned)(sk[i] & 0xffffffffull);
        __syncthreads();
    }
}

template <class LP>
__global__ void k_permute(const int *__restrict__ perm, int n, const PRec<LP> *__restrict__ recOld,
                          PRec<LP> *__restrict__ recNew, const uint8_t *__restrict__ typeOld,
                          uint8_t *__restrict__ typeNew, const int *__restrict__ origOld,
                          int *__restrict__ origNew, const int *__restrict__ cellOld,
                          int *__restrict__ cellNew, int *__restrict__ slotOf, int *__restrict__ newSlot) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int o = perm[k];
    newSlot[o] = k;
    store_rec(recNew + k, load_rec(recOld + o));
    typeNew[k] = typeOld[o];
    int g = origOld[o];
    origNew[k] = g;
    cellNew[k] = cellOld[o];
    slotOf[g] = k;
}

// ---- the gather layout (internal.h) ----

__device__ __forceinline__ void pack16(int4 *p, double a, double b) {
    *reinterpret_cast<double2 *>(p) = make_double2(a, b);
}
template <class LP>
__device__ __forceinline__ long long gather_index(int slot) {
    return (long long)(slot >> 5) * (32 * kGatherChunks<LP>) + (slot & 31);
}
__device__ __forceinline__ void store_gather(int4 *base, int slot, const PRec<float> &r) {
    int4 *p = base + gather_index<float>(slot);
    pack16(p, r.x, r.y);
    p[32] = make_int4(__double2loint(r.z), __double2hiint(r.z), __float_as_int(r.d[0]), __float_as_int(r.d[3]));
    *reinterpret_cast<float4 *>(p + 64) = make_float4(r.d[1], r.d[4], r.d[2], r.d[5]);
    *reinterpret_cast<float4 *>(p + 96) = make_float4(r.r, r.th[0], r.th[1], r.th[2]);
}
__device__ __forceinline__ void store_gather(int4 *base, int slot, const PRec<double> &r) {
    int4 *p = base + gather_index<double>(slot);
    pack16(p, r.x, r.y);
    pack16(p + 32, r.z, r.d[0]);
    pack16(p + 64, r.d[1], r.d[2]);
    pack16(p + 96, r.d[3], r.d[4]);
    pack16(p + 128, r.d[5], r.r);
    pack16(p + 160, r.th[0], r.th[1]);
    pack16(p + 192, r.th[2], 0.0);
}
// A particle as the functors read it: position and increments, radius, rotations.
template <class LP>
struct Body {
    double x, y, z;
    Six<LP> d;
    LP r, th[3];
};
// (WITH_R: the radius too; WITH_TH: the rotations too; fields not asked for stay unset. Plain
// loads: the kernel before may have written the layout, dependent_start)
template <bool WITH_R, bool WITH_TH>
__device__ __forceinline__ void load_body(Body<float> &o, const int4 *base, int slot) {
    const int4 *p = base + gather_index<float>(slot);
    const double2 c0 = *reinterpret_cast<const double2 *>(p);
    const ulonglong2 c1 = *reinterpret_cast<const ulonglong2 *>(p + 32);
    const ulonglong2 c2 = *reinterpret_cast<const ulonglong2 *>(p + 64);
    o.x = c0.x;
    o.y = c0.y;
    o.z = __longlong_as_double((long long)c1.x);
    o.d.p[0].v = c1.y;
    o.d.p[1].v = c2.x;
    o.d.p[2].v = c2.y;
    if (WITH_TH) {
        const float4 c3 = *reinterpret_cast<const float4 *>(p + 96);
        o.r = c3.x;
        o.th[0] = c3.y;
        o.th[1] = c3.z;
        o.th[2] = c3.w;
    } else if (WITH_R) {
        o.r = *reinterpret_cast<const float *>(p + 96);
    }
}
template <bool WITH_R, bool WITH_TH>
__device__ __forceinline__ void load_body(Body<double> &o, const int4 *base, int slot) {
    const double2 *p = reinterpret_cast<const double2 *>(base + gather_index<double>(slot));
    const double2 c0 = p[0], c1 = p[32], c2 = p[64], c3 = p[96];
    o.x = c0.x;
    o.y = c0.y;
    o.z = c1.x;
    o.d.f[0] = c1.y;
    o.d.f[1] = c2.x;
    o.d.f[2] = c2.y;
    o.d.f[3] = c3.x;
    o.d.f[4] = c3.y;
    if (WITH_R) {
        const double2 c4 = p[128];
        o.d.f[5] = c4.x;
        o.r = c4.y;
    } else {
        o.d.f[5] = *reinterpret_cast<const double *>(p + 128);
    }
    if (WITH_TH) {
        const double2 c5 = p[160];
        o.th[0] = c5.x;
        o.th[1] = c5.y;
        o.th[2] = *reinterpret_cast<const double *>(p + 192);
    }
}
template <class LP>
__device__ __forceinline__ PRec<LP> gather_rec(const int4 *base, int slot) {
    Body<LP> b;
    load_body<true, true>(b, base, slot);
    PRec<LP> r;
    r.x = b.x;
    r.y = b.y;
    r.z = b.z;
    b.d.get(r.d);
    r.r = b.r;
#pragma unroll
    for (int q = 0; q < 3; ++q) r.th[q] = b.th[q];
    if constexpr (sizeof(PRec<LP>) == 128) r.pad[0] = r.pad[1] = r.pad[2] = 0.0;
    return r;
}

// ------------------------------------------------------------------ contacts

// Walk of NeighbourGrid::iteratePossibleNeighbours (PLiB/NeighbourGrid.h:87-105) with
// the filter of NeighAccel::iterateBlocks (PLiB/Accel/NeighAccel.h:98-137). FILL=false
// counts, FILL=true writes the row. The 27 cells are nine runs of three consecutive colours, and
// particles are stored by colour: each run is one range of slots, walked in the reference's
// order. Candidates come from the gather layout (positions and radii of consecutive slots in
// consecutive chunks).
template <class LP>
__device__ __forceinline__ void load_place(const int4 *base, int slot, double &x, double &y, double &z, LP &r) {
    const int4 *p = base + gather_index<LP>(slot);
    const double2 c0 = __ldg(reinterpret_cast<const double2 *>(p));
    x = c0.x;
    y = c0.y;
    z = __ldg(reinterpret_cast<const double *>(p + 32));
    if constexpr (sizeof(LP) == 4)
        r = __ldg(reinterpret_cast<const float *>(p + 96));
    else
        r = __ldg(reinterpret_cast<const double *>(p + 128) + 1);
}
template <class LP, bool FILL>
__device__ __forceinline__ int walk_cells(const int4 *__restrict__ gather, int i, int colour,
                                          const GridInfo &g, const int *__restrict__ cellStart,
                                          const int *__restrict__ cellCount, double interactDist,
                                          int32_t *__restrict__ row, long long rowBase) {
    double xc, yc, zc;
    LP ri;
    load_place<LP>(gather, i, xc, yc, zc, ri);
    int count = 0;
    // the ends of the nine ranges first, so that their loads overlap
    int from[9], to[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const long long c0 = (long long)colour + g.off[3 * k], c1 = c0 + 2;
        from[k] = to[k] = 0;
        if (c1 >= 0 && c0 < g.total) {
            from[k] = __ldg(cellStart + (c0 < 0 ? 0 : c0));
            const long long e = c1 >= g.total ? g.total - 1 : c1;
            to[k] = __ldg(cellStart + e) + __ldg(cellCount + e);
        }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        for (int j = from[k]; j < to[k]; ++j) {
            if (j == i) continue;
            double xq, yq, zq;
            LP rq;
            load_place<LP>(gather, j, xq, yq, zq, rq);
            LP xDist = (LP)(xc - xq);
            LP xDist2 = xDist * xDist;
            LP yDist = (LP)(yc - yq);
            LP yDist2 = yDist * yDist;
            LP zDist = (LP)(zc - zq);
            LP zDist2 = zDist * zDist;
            LP particleDistance2 = xDist2 + yDist2 + zDist2;
            LP radSum = ri + rq;
            // candidates farther than the interaction distance by a relative 1e-5 (far above
            // the rounding of this bound, of the square root and of the subtraction below) fail
            // the test whatever the rounding: skip the IEEE square root for them
            const LP reach = (LP)interactDist + radSum;
            if (particleDistance2 > reach * reach * LP(1.00002) && reach > LP(0)) continue;
            LP particleDistance = lsqrt(particleDistance2);
            LP dist = particleDistance - radSum;
            if ((double)dist < interactDist) {
                if (FILL) row[rowBase + (long long)count * kWarp] = j;
                ++count;
            }
        }
    }
    return count;
}

template <class LP>
__global__ void __launch_bounds__(128) k_nbr_count(const int4 *__restrict__ rec, int n, const int *__restrict__ cellOf,
                            GridInfo g, const int *__restrict__ cellStart,
                            const int *__restrict__ cellCount, double interactDist,
                            uint32_t *__restrict__ counts, int *__restrict__ blockWidth,
                            int *errorFlag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int c = 0;
    // a failed check earlier in the rebuild (a particle outside the grid, a cell too crowded
    // to sort) ends the rebuild at the next host check: skip the walk, whose cost grows with
    // the square of a crowded cell's population
    const bool failed = *reinterpret_cast<volatile int *>(errorFlag) != 0;
    if (i < n) {
        if (!failed)
            c = walk_cells<LP, false>(rec, i, cellOf[i], g, cellStart, cellCount, interactDist, nullptr, 0);
        if (c > 0xffff) {
            set_error(errorFlag, 2);
            c = 0xffff;
        }
        counts[i] = (uint32_t)c;
    }
    int m = c;
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && (i >> 5) * kWarp < n) blockWidth[i >> 5] = m;
}

template <class LP>
__global__ void __launch_bounds__(128) k_nbr_fill(const int4 *__restrict__ rec, int n, const int *__restrict__ cellOf,
                           GridInfo g, const int *__restrict__ cellStart,
                           const int *__restrict__ cellCount, double interactDist,
                           const long long *__restrict__ nOff, int32_t *__restrict__ nbr) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    walk_cells<LP, true>(rec, i, cellOf[i], g, cellStart, cellCount, interactDist, nbr,
                         nOff[i >> 5] + (i & 31));
}

// Contact-list statistics of a rebuild from the per-slot counts (low 16 bits: contacts,
// high 16 bits: link ends): out[0] total contacts, out[1] the largest contact count,
// out[2] the largest link-end count (integer sums and maxima: order-independent).
__global__ void k_count_stats(const uint32_t *__restrict__ counts, int n, long long *__restrict__ out) {
    long long pairs = 0, mn = 0, ml = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = counts[i];
        const long long a = c & 0xffffu, e = c >> 16;
        pairs += a;
        mn = a > mn ? a : mn;
        ml = e > ml ? e : ml;
    }
    for (int o = 16; o > 0; o >>= 1) {
        pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
        const long long a = __shfl_xor_sync(0xffffffffu, mn, o), e = __shfl_xor_sync(0xffffffffu, ml, o);
        mn = a > mn ? a : mn;
        ml = e > ml ? e : ml;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(reinterpret_cast<unsigned long long *>(out), (unsigned long long)pairs);
        atomicMax(out + 1, mn);
        atomicMax(out + 2, ml);
    }
}

// ------------------------------------------------------------------ link ends

__global__ void k_side_count(const int *__restrict__ orig, int n, const int *__restrict__ plStart,
                             uint32_t *__restrict__ counts, int *__restrict__ blockWidth,
                             int *errorFlag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int c = 0;
    if (i < n) {
        int o = orig[i];
        c = plStart[o + 1] - plStart[o];
        if (c > 0xffff) {
            set_error(errorFlag, 3);
            c = 0xffff;
        }
        counts[i] = (counts[i] & 0xffffu) | ((uint32_t)c << 16);
    }
    int m = c;
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && (i >> 5) * kWarp < n) blockWidth[i >> 5] = m;
}

template <class LP>
__global__ void k_side_fill(const int *__restrict__ orig, int n, const int *__restrict__ slotOf,
                            const int *__restrict__ plStart, const int *__restrict__ plLink,
                            const uint8_t *__restrict__ plEnd, const int *__restrict__ linkA,
                            const int *__restrict__ linkB, const LP *__restrict__ L0link,
                            const int *__restrict__ sideSlotOld, SideView<LP> oldS,
                            const long long *__restrict__ sOff, SideView<LP> newS,
                            int *__restrict__ sideSlotNew) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int o = orig[i];
    int ps = plStart[o], pe = plStart[o + 1];
    long long base = sOff[i >> 5] + (i & 31);
    for (int k = 0; k < pe - ps; ++k) {
        int l = plLink[ps + k];
        int e = plEnd[ps + k];
        int other = e ? linkA[l] : linkB[l];
        long long dst = base + (long long)k * kWarp;
        int src = sideSlotOld[2 * l + e];
        newS.partner[dst] = (uint32_t)slotOf[other] | (e ? kSideIsB : 0u);
        newS.state[dst] = oldS.state[src];
#pragma unroll
        for (int c = 0; c < 6; ++c) newS.ct[c][dst] = oldS.ct[c][src];
        newS.L0[dst] = L0link[l];
        newS.link[dst] = l;
        sideSlotNew[2 * l + e] = (int)dst;
    }
}

// The link ends moved from one slot layout to the next: end k of a slot comes from end k of the
// slot its particle had (both in ascending link index), so every array is read in runs of a
// block's entries, and only the partner's new slot (of a nearby particle) and the link's record
// of where its end lies are looked up. Through the links (k_side_fill, which the first layout
// after set_links still takes) each end costs four scattered 32-byte sectors more: 344 us
// against 167 us on the 0.8M slab (mixed).
template <class LP>
__global__ void __launch_bounds__(256) k_side_move(const int *__restrict__ perm, int n, const int *__restrict__ newSlot,
                            const uint32_t *__restrict__ counts, const long long *__restrict__ sOffOld,
                            SideView<LP> oldS, const long long *__restrict__ sOff, SideView<LP> newS,
                            int *__restrict__ sideSlotNew) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = __ldg(perm + i);
    const int ns = (int)(__ldg(counts + i) >> 16);
    unsigned src = (unsigned)(__ldg(sOffOld + (o >> 5)) + (o & 31));
    unsigned dst = (unsigned)(__ldg(sOff + (i >> 5)) + (i & 31));
    for (int k = 0; k < ns; ++k, src += kWarp, dst += kWarp) {
        const uint32_t pw = oldS.partner[src];
        const int l = oldS.link[src];
        LP ct[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) ct[c] = oldS.ct[c][src];
        const LP L0 = oldS.L0[src];
        const uint8_t st = oldS.state[src];
        newS.partner[dst] = (uint32_t)__ldg(newSlot + (pw & kSlotMask)) | (pw & kSideIsB);
        newS.state[dst] = st;
#pragma unroll
        for (int c = 0; c < 6; ++c) newS.ct[c][dst] = ct[c];
        newS.L0[dst] = L0;
        newS.link[dst] = l;
        sideSlotNew[2 * l + ((pw & kSideIsB) ? 1 : 0)] = (int)dst;
    }
}

// ------------------------------------------------------------------ timestep

// The first CHUNKS 16-byte chunks of a record (the fields a functor reads); the rest of
// the returned record is left unset and must not be read.
template <class LP, int CHUNKS>
__device__ __forceinline__ PRec<LP> load_rec_head(const PRec<LP> *p) {
    PRec<LP> r;
    const int4 *src = reinterpret_cast<const int4 *>(p);
    int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) dst[k] = __ldg(src + k);
    return r;
}
// chunks holding x, y, z, d[6], r
template <class LP>
constexpr int kContactChunks = (int)((3 * sizeof(double) + 7 * sizeof(LP) + 15) / 16);

// Start the L2 fetch of everything this warp will stream: its block's contact indices and its
// link ends' partner words, CT0..CT5, states (and initial lengths), each one contiguous run of
// the warp-blocked layout. One bulk prefetch per array, one lane each (nothing to wait for),
// instead of a prefetch per array and item. Runs are multiples of 32 entries from 32-entry
// offsets: 16-byte aligned for the byte arrays too.
__device__ __forceinline__ void bulk_prefetch_l2(const void *p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <class LP>
__device__ __forceinline__ void prefetch_block(const StepArgs<LP> &a, int w, bool lengths) {
    const int lane = threadIdx.x & 31;
    const long long s0 = __ldg(a.sOff + w), n0 = __ldg(a.nOff + w);
    const unsigned ends = (unsigned)(__ldg(a.sOff + w + 1) - s0), contacts = (unsigned)(__ldg(a.nOff + w + 1) - n0);
    const void *p = nullptr;
    unsigned bytes = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (lane == q) p = a.ct[q] + s0, bytes = ends * (unsigned)sizeof(LP);
    if (lane == 6) p = a.sPartner + s0, bytes = ends * 4u;
    if (lane == 7) p = a.sState + s0, bytes = ends;
    if (lane == 8) p = a.nbr + n0, bytes = contacts * 4u;
    if (lane == 9 && lengths) p = a.sL0 + s0, bytes = ends * (unsigned)sizeof(LP);
    if (bytes) bulk_prefetch_l2(p, bytes);
}

// Whether a whole link between two particles a squared distance D apart (as the break functor
// forms it) stays whole for certain: its load is below maxLoad by more than 1e-5 (1 + |maxLoad|
// + |bendBreak| bend), far above the functor's and this test's rounding (a few 2^-23 of the same
// sum), so the functor's root and division are left to the links near the threshold. A test
// that is not certain is false: NaN, a non-positive bound, a negative initial length (which
// turns the functor's inequality round), a bound so small that its square loses digits.
template <class LP>
__device__ __forceinline__ bool stays_whole(const StepArgs<LP> &a, LP D, const LP *thA, const LP *thB, LP L0) {
    const LP ax = labs_(thA[0] - thB[0]), ay = labs_(thA[1] - thB[1]), az = labs_(thA[2] - thB[2]);
    const LP myz = (ay < az) ? az : ay;
    const LP bend = (ax < myz) ? myz : ax;
    const LP t = L0 * (a.wholeLoad - a.wholeBend * bend);
    return L0 > LP(0) && t > LP(1e-16) && D < t * t;
}

// The link state of one end after the previous step's link update (a.breakPending), both ends
// of a link deciding alike from the same records; end A appends the break event.
template <class LP, class P>
__device__ __forceinline__ uint8_t pending_break(const StepArgs<LP> &a, unsigned si, uint32_t pw, const P &me,
                                                 const P &other, uint8_t st, LP L0, LP x, LP y, LP z) {
    if (st == 0 || stays_whole<LP>(a, x * x + y * y + z * z, me.th, other.th, L0)) return st;
    const uint8_t nst = (pw & kSideIsB) ? break_link<LP>(a.bendBreak, a.maxLoad, other, me, st, L0)
                                        : break_link<LP>(a.bendBreak, a.maxLoad, me, other, st, L0);
    if (nst != st) {
        a.sState[si] = nst;
        a.linkState[__ldg(a.sLink + si)] = nst;  // both sides write the same value
        if (nst == 0 && !(pw & kSideIsB)) {
            unsigned long long slot = atomicAdd(a.eventCount, 1ull);
            if ((long long)slot < a.eventCap) a.events[slot] = make_int2(__ldg(a.sLink + si), (int)a.breakStep);
        }
    }
    return nst;
}

// The force pass: one particle per thread, contacts, then link ends, forces to a.force
// (HiDEMLib::computePartForce), partners read from the gather layout. BRK: the previous step's
// link update is applied on the way (each end decides its link from the records it has
// loaded for the beam anyway; a break pass of its own gathers both records of every link
// again: 0.33 of 2.03 ms per step on the 5.7M slab).
//
// What bounds it: the latency of one gather per item, against what the warps in flight can
// hide. AHEAD keeps the next item's partner and CT in registers while this one is evaluated
// (96-166 registers); without it, a warp waits for each gather but there are 28 warps an SM
// instead of 20 (mixed, 72 registers) and no copies between the two register sets (120M
// against 141M instructions on the 0.8M slab). Measured per step, 5.7M slab, mixed: from the
// records with AHEAD 2.03 ms (L1 data path 86 % busy), gather layout with AHEAD 1.71 ms, without
// 1.44 ms at 7 CTAs an SM (6: 1.50, 8: 1.51); FP64: 4.05 ms from the records, 2.67 ms with AHEAD
// (3 CTAs), 2.95 ms without (4 CTAs). Where every block is resident at once anyway (a small
// particle set) AHEAD is the faster one in both: 32,000 particles 25.1 against 27.4 us a step.
template <class LP, bool BRK, bool AHEAD>
__device__ __forceinline__ void force_particle(const Consts<LP> &c, const StepArgs<LP> &a, const int i) {
    const Rounding<LP> R = Rounding<LP>::make();
    if ((i & ~31) < a.n) prefetch_block<LP>(a, i >> 5, BRK);
    if (i >= a.n) return;
    Body<LP> me;
    load_body<true, BRK>(me, a.gather, i);
    const uint32_t cnt = __ldg(a.counts + i);
    const int nn = (int)(cnt & 0xffffu), ns = (int)(cnt >> 16);
    Six<LP> F = Six<LP>::zero();
    const int32_t *nb = a.nbr + __ldg(a.nOff + (i >> 5)) + (i & 31);
    // link-end slots fit 31 bits (checked at the rebuild)
    unsigned si = (unsigned)__ldg(a.sOff + (i >> 5)) + (i & 31);

    auto contact = [&](const Body<LP> &o) {
        contact_pair<LP>(c, R, (LP)(me.x - o.x), (LP)(me.y - o.y), (LP)(me.z - o.z), me.d, me.r, o.d, o.r, F);
    };
    // what a link end is evaluated from, and its evaluation: the break decision, the beam, CT
    struct End {
        Body<LP> o;
        LP CT[6], L0;
        uint8_t st;
    };
    auto load_end = [&](End &e, uint32_t pw, unsigned at) {
        load_body<false, BRK>(e.o, a.gather, (int)(pw & kSlotMask));
        e.st = a.sState[at];
#pragma unroll
        for (int q = 0; q < 6; ++q) e.CT[q] = a.ct[q][at];
        if (BRK) e.L0 = __ldg(a.sL0 + at);
    };
    auto end = [&](End &e, uint32_t pw, unsigned at) {
        const LP x = (LP)(me.x - e.o.x), y = (LP)(me.y - e.o.y), z = (LP)(me.z - e.o.z);
        if (BRK) e.st = pending_break<LP>(a, at, pw, me, e.o, e.st, e.L0, x, y, z);
        beam_side<LP>(c, R, e.st != 0, x, y, z, me.d, e.o.d, e.CT, F);
#pragma unroll
        for (int q = 0; q < 6; ++q) a.ct[q][at] = e.CT[q];
    };

    if constexpr (!AHEAD) {
        // the index of the next item is in flight while this one waits for its partner
        int j = nn > 0 ? __ldg(nb) : 0;
        uint32_t pw = ns > 0 ? __ldg(a.sPartner + si) : 0u;
        for (int k = 0; k < nn; ++k) {
            Body<LP> o;
            load_body<true, false>(o, a.gather, j);
            if (k + 1 < nn) j = __ldg(nb + (k + 1) * kWarp);
            contact(o);
        }
        for (int k = 0; k < ns; ++k, si += kWarp) {
            End e;
            load_end(e, pw, si);
            const uint32_t pwc = pw;
            if (k + 1 < ns) pw = __ldg(a.sPartner + si + kWarp);
            end(e, pwc, si);
        }
    } else {
        // item k + 1 and the index of item k + 2 are in flight while item k is evaluated, the
        // first link end behind the last contact
        Body<LP> o;
        int jn = 0;
        if (nn > 0) load_body<true, false>(o, a.gather, __ldg(nb));
        if (nn > 1) jn = __ldg(nb + kWarp);
        uint32_t pwn = ns > 0 ? __ldg(a.sPartner + si) : 0u, pwnn = 0;
        End en;
        auto first_end = [&]() {
            if (ns > 0) {
                load_end(en, pwn, si);
                if (ns > 1) pwnn = __ldg(a.sPartner + si + kWarp);
            }
        };
        if (nn == 0) first_end();
        for (int k = 0; k < nn; ++k) {
            const Body<LP> cur = o;
            if (k + 1 < nn) {
                load_body<true, false>(o, a.gather, jn);
                if (k + 2 < nn) jn = __ldg(nb + (k + 2) * kWarp);
            } else {
                first_end();
            }
            contact(cur);
        }
        for (int k = 0; k < ns; ++k, si += kWarp) {
            End e = en;
            const uint32_t pw = pwn;
            if (k + 1 < ns) {
                pwn = pwnn;
                load_end(en, pwn, si + kWarp);
                if (k + 2 < ns) pwnn = __ldg(a.sPartner + si + 2 * kWarp);
            }
            end(e, pw, si);
        }
    }

    LP f[6];
    F.get(f);
#pragma unroll
    for (int q = 0; q < 6; ++q) a.force[(long long)q * a.n + i] = f[q];
    // a particle another rank integrates: its record of the halo send buffer too
    if (a.sendPos) {
        const int sp = __ldg(a.sendPos + i);
        if (sp >= 0) {
#pragma unroll
            for (int q = 0; q < 6; ++q) a.sendBuf[6ll * sp + q] = f[q];
        }
    }
}

// One particle per thread: the previous step's link update (if pending), contacts, link
// ends, integrate, the record written to the other buffer.
// Both item loops are software-pipelined: while item k is evaluated, the partner record
// (and for link ends the CT state, link state and initial length) of item k + 1 and the
// index of item k + 2 are already in flight, and the first link end's loads go out behind
// the last contact, so each thread keeps its dependent loads outstanding behind its
// arithmetic. The functors still run in the reference's order per particle.
template <class LP>
__device__ __forceinline__ void step_thread_particle(const Consts<LP> &c, const StepArgs<LP> &a,
                                                     const int i) {
    const bool live = i < a.n;
    LP dmax[3] = {LP(0), LP(0), LP(0)};
    const Rounding<LP> R = Rounding<LP>::make();
    const bool brk = a.breakPending;
    if ((i & ~31) < a.n) prefetch_block<LP>(a, i >> 5, brk);
    if (live) {
        PRec<LP> me = load_rec(a.in + i);
        const uint32_t cnt = __ldg(a.counts + i);
        const uint8_t ty = __ldg(a.type + i);
        const int nn = (int)(cnt & 0xffffu), ns = (int)(cnt >> 16);
        const Six<LP> mine = Six<LP>::of(me.d);
        Six<LP> F = Six<LP>::zero();
        constexpr int HC = kContactChunks<LP>;

        const int32_t *nb = a.nbr + __ldg(a.nOff + (i >> 5)) + (i & 31);
        // link-end slots fit 31 bits (checked at the rebuild)
        unsigned si = (unsigned)__ldg(a.sOff + (i >> 5)) + (i & 31);
        PRec<LP> o;
        int jn = 0;
        if (nn > 0) o = load_rec_head<LP, HC>(a.in + __ldg(nb));
        if (nn > 1) jn = __ldg(nb + kWarp);
        // first link end's partner word while the contacts run
        uint32_t pwn = (ns > 0) ? __ldg(a.sPartner + si) : 0u;
        PRec<LP> o2;
        uint8_t stn = 0;
        LP ctn[6] = {0, 0, 0, 0, 0, 0};
        LP l0n = LP(0);
        uint32_t pwnn = 0;
        // the first link end's partner record, state and CT go out behind the last contact
        auto first_side = [&]() {
            if (ns > 0) {
                o2 = load_rec(a.in + (pwn & kSlotMask));
                stn = a.sState[si];
#pragma unroll
                for (int q = 0; q < 6; ++q) ctn[q] = a.ct[q][si];
                if (brk) l0n = __ldg(a.sL0 + si);
                if (ns > 1) pwnn = __ldg(a.sPartner + si + kWarp);
            }
        };
        if (nn == 0) first_side();
        for (int k = 0; k < nn; ++k) {
            const PRec<LP> cur = o;
            if (k + 1 < nn) {
                o = load_rec_head<LP, HC>(a.in + jn);
                if (k + 2 < nn) jn = __ldg(nb + (k + 2) * kWarp);
            } else {
                first_side();
            }
            contact_pair<LP>(c, R, (LP)(me.x - cur.x), (LP)(me.y - cur.y), (LP)(me.z - cur.z), mine, me.r,
                             Six<LP>::of(cur.d), cur.r, F);
        }

        for (int k = 0; k < ns; ++k, si += kWarp) {
            const PRec<LP> cur = o2;
            const uint32_t pw = pwn;
            uint8_t st = stn;
            const LP L0 = l0n;
            LP CT[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) CT[q] = ctn[q];
            if (k + 1 < ns) {
                pwn = pwnn;
                o2 = load_rec(a.in + (pwn & kSlotMask));
                stn = a.sState[si + kWarp];
#pragma unroll
                for (int q = 0; q < 6; ++q) ctn[q] = a.ct[q][si + kWarp];
                if (brk) l0n = __ldg(a.sL0 + si + kWarp);
                if (k + 2 < ns) pwnn = __ldg(a.sPartner + si + 2 * kWarp);
            }
            const LP x = (LP)(me.x - cur.x), y = (LP)(me.y - cur.y), z = (LP)(me.z - cur.z);
            if (brk) st = pending_break<LP>(a, si, pw, me, cur, st, L0, x, y, z);
            beam_side<LP>(c, R, st != 0, x, y, z, mine, Six<LP>::of(cur.d), CT, F);
#pragma unroll
            for (int q = 0; q < 6; ++q) a.ct[q][si] = CT[q];
        }

        LP f[6];
        F.get(f);
        integrate_particle<LP>(c, me, ty, f);
        store_rec(a.out + i, me);
        dmax[0] = me.d[0] > LP(0) ? me.d[0] : LP(0);
        dmax[1] = me.d[1] > LP(0) ? me.d[1] : LP(0);
        dmax[2] = me.d[2] > LP(0) ? me.d[2] : LP(0);
    }
    if (a.reduceDiff) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            LP v = dmax[q];
            for (int o = 16; o > 0; o >>= 1) {
                LP u = __shfl_xor_sync(0xffffffffu, v, o);
                v = (u > v) ? u : v;
            }
            if ((threadIdx.x & 31) == 0 && v > LP(0)) atomicMax(a.diffMax + q, max_bits(v));
        }
    }
}

// CTAs per SM the register-capped variant asks the compiler for: 5 (96 registers) in the
// mixed build, 3 (168 registers) in fp64 — each the tightest cap that spills little.
template <class LP>
constexpr int kCapBlocks = sizeof(LP) == 4 ? 5 : 3;
// and the plain variant: 4 CTAs (128 registers) in the mixed build, no cap in fp64
template <class LP>
constexpr int kThreadBlocks = sizeof(LP) == 4 ? 4 : 1;
// and the asynchronous-copy variant (its partner data lives in shared memory)
template <class LP>
constexpr int kAsyncBlocks = sizeof(LP) == 4 ? 5 : 3;
// the force pass of a large particle set (register caps without spills; force_particle)
template <class LP>
constexpr bool kForceAhead = sizeof(LP) == 8;
template <class LP>
constexpr int kForceBlocks = sizeof(LP) == 4 ? 7 : 3;
// and of one whose blocks are all resident at once even so: up to kFewBlocks CTAs per SM
template <class LP>
constexpr int kFewBlocks = sizeof(LP) == 4 ? 4 : 2;

template <class LP, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
    k_step(const Consts<LP> c, const StepArgs<LP> a) {
    step_thread_particle<LP>(c, a, blockIdx.x * blockDim.x + threadIdx.x);
}

template <class LP, bool BRK, bool AHEAD, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
    k_force(const Consts<LP> c, const StepArgs<LP> a) {
    dependent_start();
    force_particle<LP, BRK, AHEAD>(c, a, blockIdx.x * blockDim.x + threadIdx.x);
}

// records -> gather layout, and back
template <class LP>
__global__ void __launch_bounds__(256) k_to_gather(const PRec<LP> *rec, int n, int4 *g) {
    dependent_start();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) store_gather(g, i, load_rec_written(rec + i));
}
template <class LP>
__global__ void __launch_bounds__(256) k_from_gather(const int4 *__restrict__ g, int n, PRec<LP> *__restrict__ rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) store_rec(rec + i, gather_rec<LP>(g, i));
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- one thread per particle, partner data staged by asynchronous copies ----
//
// The same per-particle evaluation as step_thread_particle, but the next items' partner
// records (and, for link ends, CT0..CT5) travel with cp.async into this thread's own
// shared-memory slots instead of registers: two items are in flight behind the one being
// evaluated, and the registers that held the prefetched record are free (more CTAs per
// SM). Slot layout per CTA, chunk-major so that a warp's 16-byte reads are conflict-free:
// rec[slot][chunk][thread] (16 B), ct[slot][q][thread] (lp).
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, int bytes16_4_8) {
    if (bytes16_4_8 == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
    else if (bytes16_4_8 == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait until at most one group of this thread is still in flight
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <class LP>
constexpr int kRecChunks = (int)(sizeof(PRec<LP>) / 16);
template <class LP>
constexpr size_t async_smem_bytes() {
    return (size_t)2 * kStepThreads * (sizeof(PRec<LP>) + 6 * sizeof(LP));
}

template <class LP>
__device__ __forceinline__ void step_thread_async(const Consts<LP> &c, const StepArgs<LP> &a,
                                                  const int i, unsigned char *smem) {
    constexpr int NC = kRecChunks<LP>;
    constexpr int HC = kContactChunks<LP>;
    const int t = threadIdx.x;
    int4 *srec = reinterpret_cast<int4 *>(smem);                                  // [2][NC][128]
    LP *sct = reinterpret_cast<LP *>(smem + (size_t)2 * NC * kStepThreads * 16);   // [2][6][128]
    auto rec_slot = [&](int s, int ch) { return srec + (s * NC + ch) * kStepThreads + t; };
    auto ct_slot = [&](int s, int q) { return sct + (s * 6 + q) * kStepThreads + t; };
    auto read_rec = [&](int s, int chunks) {
        PRec<LP> r;
        int4 *dst = reinterpret_cast<int4 *>(&r);
#pragma unroll
        for (int ch = 0; ch < NC; ++ch)
            if (ch < chunks) dst[ch] = *rec_slot(s, ch);
        return r;
    };

    const Rounding<LP> R = Rounding<LP>::make();
    const bool live = i < a.n;
    LP dmax[3] = {LP(0), LP(0), LP(0)};
    if (live) {
        PRec<LP> me = load_rec(a.in + i);
        const uint32_t cnt = __ldg(a.counts + i);
        const uint8_t ty = __ldg(a.type + i);
        const int nn = (int)(cnt & 0xffffu), ns = (int)(cnt >> 16);
        const Six<LP> mine = Six<LP>::of(me.d);
        Six<LP> F = Six<LP>::zero();
        const int32_t *nb = a.nbr + __ldg(a.nOff + (i >> 5)) + (i & 31);
        const long long sbase = __ldg(a.sOff + (i >> 5)) + (i & 31);

        // contacts: item k's record in slot k & 1; items k + 1 and k + 2 in flight
        auto issue_contact = [&](int s, int j) {
            const int4 *src = reinterpret_cast<const int4 *>(a.in + j);
#pragma unroll
            for (int ch = 0; ch < HC; ++ch) cp_async(rec_slot(s, ch), src + ch, 16);
        };
        int j2 = 0;
        if (nn > 0) issue_contact(0, __ldg(nb));
        cp_async_commit();
        if (nn > 1) issue_contact(1, __ldg(nb + kWarp));
        cp_async_commit();
        if (nn > 2) j2 = __ldg(nb + 2 * kWarp);
        for (int k = 0; k < nn; ++k) {
            cp_async_wait1();
            const PRec<LP> cur = read_rec(k & 1, HC);
            if (k + 2 < nn) {
                issue_contact(k & 1, j2);
                if (k + 3 < nn) j2 = __ldg(nb + (k + 3) * kWarp);
            }
            cp_async_commit();
            contact_pair<LP>(c, R, (LP)(me.x - cur.x), (LP)(me.y - cur.y), (LP)(me.z - cur.z), mine, me.r,
                             Six<LP>::of(cur.d), cur.r, F);
        }
        cp_async_wait0();

        // link ends: record and CT of item k in slot k & 1; state and initial length one
        // item ahead in registers
        const bool brk = a.breakPending;
        auto issue_side = [&](int s, long long si, uint32_t pw) {
            const int4 *src = reinterpret_cast<const int4 *>(a.in + (pw & kSlotMask));
#pragma unroll
            for (int ch = 0; ch < NC; ++ch) cp_async(rec_slot(s, ch), src + ch, 16);
#pragma unroll
            for (int q = 0; q < 6; ++q) cp_async(ct_slot(s, q), a.ct[q] + si, (int)sizeof(LP));
        };
        uint32_t pw0 = 0, pw1 = 0, pw2 = 0;
        uint8_t stn = 0;
        LP l0n = LP(0);
        if (ns > 0) {
            pw0 = __ldg(a.sPartner + sbase);
            issue_side(0, sbase, pw0);
            stn = a.sState[sbase];
            if (brk) l0n = __ldg(a.sL0 + sbase);
        }
        cp_async_commit();
        if (ns > 1) {
            pw1 = __ldg(a.sPartner + sbase + kWarp);
            issue_side(1, sbase + kWarp, pw1);
        }
        cp_async_commit();
        if (ns > 2) pw2 = __ldg(a.sPartner + sbase + 2 * kWarp);
        for (int k = 0; k < ns; ++k) {
            const long long si = sbase + (long long)k * kWarp;
            const uint32_t pw = pw0;
            uint8_t st = stn;
            const LP L0 = l0n;
            cp_async_wait1();
            const PRec<LP> cur = read_rec(k & 1, NC);
            LP CT[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) CT[q] = *ct_slot(k & 1, q);
            pw0 = pw1;
            pw1 = pw2;
            if (k + 1 < ns) {
                stn = a.sState[si + kWarp];
                if (brk) l0n = __ldg(a.sL0 + si + kWarp);
            }
            if (k + 2 < ns) {
                issue_side(k & 1, si + 2 * kWarp, pw1);
                if (k + 3 < ns) pw2 = __ldg(a.sPartner + si + 3 * kWarp);
            }
            cp_async_commit();
            const LP x = (LP)(me.x - cur.x), y = (LP)(me.y - cur.y), z = (LP)(me.z - cur.z);
            if (brk) st = pending_break<LP>(a, (unsigned)si, pw, me, cur, st, L0, x, y, z);
            beam_side<LP>(c, R, st != 0, x, y, z, mine, Six<LP>::of(cur.d), CT, F);
#pragma unroll
            for (int q = 0; q < 6; ++q) a.ct[q][si] = CT[q];
        }
        cp_async_wait0();

        LP f[6];
        F.get(f);
        integrate_particle<LP>(c, me, ty, f);
        store_rec(a.out + i, me);
        dmax[0] = me.d[0] > LP(0) ? me.d[0] : LP(0);
        dmax[1] = me.d[1] > LP(0) ? me.d[1] : LP(0);
        dmax[2] = me.d[2] > LP(0) ? me.d[2] : LP(0);
    }
    if (a.reduceDiff) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            LP v = dmax[q];
            for (int o = 16; o > 0; o >>= 1) {
                LP u = __shfl_xor_sync(0xffffffffu, v, o);
                v = (u > v) ? u : v;
            }
            if ((threadIdx.x & 31) == 0 && v > LP(0)) atomicMax(a.diffMax + q, max_bits(v));
        }
    }
}

template <class LP, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
    k_step_async(const Consts<LP> c, const StepArgs<LP> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    step_thread_async<LP>(c, a, blockIdx.x * blockDim.x + threadIdx.x, smem);
}

// Item-parallel step: one CTA per 32-slot block, for particle sets too small to fill the chip
// with one thread per particle. A warp's lanes are the block's particles; its WARPS warps take
// the contacts and link ends in turn (item k of every particle to warp k mod WARPS, contacts from
// the other side so that both remainders do not fall to the same warps) and write the values
// their functors add to the forces into shared memory; one warp per force component adds them in
// the reference's order (contacts in list order, then per link end the damping term and the CT
// term), and one warp integrates, so the result is bit-identical to k_step.
// What bounds it is the chain of dependent latencies of a step (index, partner, functor, sum,
// integrate), so nothing is staged first: every warp loads its items' data directly.
// Per step (with dependent launches): 256 particles 8.2 us, 8,892 (FP64) 14.5 us, 32,000 24.3 us;
// with the block's streams staged by bulk copies and one warp summing 10.7, 16.7 and 29.7 us.
template <class LP, int WARPS>
__device__ __forceinline__ void step_items_block(const Consts<LP> &c, const StepArgs<LP> &a, const int w,
                                                 unsigned char *smem) {
    const Rounding<LP> R = Rounding<LP>::make();
    LP *tc = reinterpret_cast<LP *>(smem);             // [maxContacts][6][32]
    LP *ts = tc + (size_t)a.maxContacts * 6 * 32;      // [maxEnds][12][32]
    LP *fs = ts + (size_t)a.maxEnds * 12 * 32;         // [6][32]
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = w * 32 + lane;
    const bool live = i < a.n;
    const bool brk = a.breakPending != 0;
    PRec<LP> me;
    int nn = 0, ns = 0;
    uint8_t ty = 0;
    if (live) {
        if (wid == 0) ty = __ldg(a.type + i);
        const uint32_t cnt = __ldg(a.counts + i);
        nn = (int)(cnt & 0xffffu);
        ns = (int)(cnt >> 16);
        const unsigned sbase = (unsigned)__ldg(a.sOff + w) + lane;
        const int32_t *nb = a.nbr + __ldg(a.nOff + w) + lane;
        me = load_rec_written(a.in + i);
        const Six<LP> mine = Six<LP>::of(me.d);
        for (int k = wid; k < ns; k += WARPS) {
            const unsigned si = sbase + k * kWarp;
            const uint32_t pw = __ldg(a.sPartner + si);
            uint8_t st = a.sState[si];
            LP CT[6];
#pragma unroll
            for (int u = 0; u < 6; ++u) CT[u] = a.ct[u][si];
            const PRec<LP> o = load_rec_written(a.in + (pw & kSlotMask));
            const LP x = (LP)(me.x - o.x), y = (LP)(me.y - o.y), z = (LP)(me.z - o.z);
            if (brk) st = pending_break<LP>(a, si, pw, me, o, st, __ldg(a.sL0 + si), x, y, z);
            Six<LP> dpv, ctv;
            beam_terms(c, R, st != 0, x, y, z, mine, Six<LP>::of(o.d), CT, dpv, ctv);
            LP dp[6], ctt[6];
            dpv.get(dp);
            ctv.get(ctt);
#pragma unroll
            for (int u = 0; u < 6; ++u) {
                a.ct[u][si] = CT[u];
                ts[(k * 12 + u) * 32 + lane] = dp[u];
                ts[(k * 12 + 6 + u) * 32 + lane] = ctt[u];
            }
        }
        for (int k = WARPS - 1 - wid; k < nn; k += WARPS) {
            const PRec<LP> o = load_rec_written<LP, kContactChunks<LP>>(a.in + __ldg(nb + k * kWarp));
            Six<LP> tv = Six<LP>::zero();
            contact_terms(c, R, (LP)(me.x - o.x), (LP)(me.y - o.y), (LP)(me.z - o.z), mine, me.r,
                          Six<LP>::of(o.d), o.r, tv);
            LP tt[6];
            tv.get(tt);
#pragma unroll
            for (int u = 0; u < 6; ++u) tc[(k * 6 + u) * 32 + lane] = tt[u];
        }
    }
    __syncthreads();
    for (int u = wid; u < 6; u += WARPS) {
        LP F = LP(0);
#pragma unroll 4
        for (int k = 0; k < nn; ++k) F = F + tc[(k * 6 + u) * 32 + lane];
#pragma unroll 4
        for (int k = 0; k < ns; ++k) {
            F = F + ts[(k * 12 + u) * 32 + lane];
            F = F - ts[(k * 12 + 6 + u) * 32 + lane];
        }
        fs[u * 32 + lane] = F;
    }
    __syncthreads();
    if (wid != 0) return;
    LP dmax[3] = {LP(0), LP(0), LP(0)};
    if (live) {
        LP F[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) F[u] = fs[u * 32 + lane];
        integrate_particle<LP>(c, me, ty, F);
        store_rec(a.out + i, me);
#pragma unroll
        for (int q = 0; q < 3; ++q) dmax[q] = me.d[q] > LP(0) ? me.d[q] : LP(0);
    }
    if (a.reduceDiff) {
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            LP v = dmax[u];
            for (int o = 16; o > 0; o >>= 1) {
                LP x = __shfl_xor_sync(0xffffffffu, v, o);
                v = (x > v) ? x : v;
            }
            if (lane == 0 && v > LP(0)) atomicMax(a.diffMax + u, max_bits(v));
        }
    }
}

template <class LP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
    k_step_items(const Consts<LP> c, const StepArgs<LP> a) {
    extern __shared__ __align__(128) unsigned char smem[];
    dependent_start();
    step_items_block<LP, WARPS>(c, a, blockIdx.x, smem);
}

// One fused step of many independent contexts in one launch. CTA b belongs to the entry
// blockEntry[b], whose CTA range is [firstBlocks[e], firstBlocks[e + 1]); all entries share the
// launch's constants except the break thresholds (in each entry's arguments), and each
// entry's per-step arguments are derived from the launch's step s within the run (a
// parameter of the launch, fixed in a captured run) the way the single-context
// host loop sets them: records alternate between the two buffers, the link update of the
// previous step is applied first once the break gate t * dt > breakTime was open at that
// step (MainMeshBlock.cpp:312), the diff maxima are folded on steps t with
// (t + 1) % 10 == 0 and cleared on steps with t % 10 == 0 (after the host has read them
// at the start of that step). KIND selects the per-CTA body: the item kernel (32
// particles per CTA, dynamic shared memory for the widest entry) or one thread per
// particle (kStepThreads particles per CTA, registers capped or not).
template <class LP, int KIND>
__global__ void __launch_bounds__(KIND == HIDEM_STEP_KERNEL_ITEMS ? kItemThreads : kStepThreads,
                                  KIND == HIDEM_STEP_KERNEL_THREAD_CAPPED ? kCapBlocks<LP>
                                  : KIND == HIDEM_STEP_KERNEL_THREAD      ? kThreadBlocks<LP>
                                                                          : 1)
    k_step_batch(const Consts<LP> c, const BatchEntry<LP> *__restrict__ entries,
                 const int *__restrict__ firstBlocks, const int *__restrict__ blockEntry, int s) {
    extern __shared__ __align__(128) unsigned char smem[];
    // the context's arguments in shared memory (read as the loops go, not held in registers)
    __shared__ StepArgs<LP> sa;
    const int b = blockIdx.x;
    const int ei = __ldg(blockEntry + b);
    const BatchEntry<LP> &e = entries[ei];
    const int lb = b - __ldg(firstBlocks + ei);
    if (threadIdx.x == 0) {
        StepArgs<LP> a = e.a;
        const int par = (e.cur0 + s) & 1;
        a.in = e.rec[par];
        a.out = e.rec[par ^ 1];
        a.step = e.step0 + s;
        a.breakStep = a.step - 1;
        a.breakPending = (s > 0) ? ((LP)((LP)a.breakStep * c.dt) > c.breakTime ? 1 : 0) : e.pend0;
        a.reduceDiff = (e.reduceEvery10 && (a.step + 1) % 10 == 0) ? 1 : 0;
        sa = a;
    }
    __syncthreads();
    if (e.reduceEvery10 && sa.step % 10 == 0 && lb == 0 && threadIdx.x < 3)
        sa.diffMax[threadIdx.x] = 0ull;
    if (KIND == HIDEM_STEP_KERNEL_ITEMS)
        step_items_block<LP, kItemThreads / 32>(c, sa, lb, smem);
    else
        step_thread_particle<LP>(c, sa, lb * kStepThreads + threadIdx.x);
}

// ---- the two-pass step over a batch (three launches per step and group) ----

// The entry whose CTA range holds this CTA: a table of one entry index per CTA, filled when
// the batch's entries are uploaded (one load, where a search over the offsets took several
// dependent ones at the start of every CTA).
__device__ __forceinline__ int batch_entry(const int *blockEntry) { return __ldg(blockEntry + blockIdx.x); }

// tbl[offs[e] .. offs[e + 1]) = e for each of the `count` entries (one CTA per entry)
__global__ void k_block_table(const int *__restrict__ offs, int *__restrict__ tbl) {
    const int e = blockIdx.x;
    const int a = __ldg(offs + e), b = __ldg(offs + e + 1);
    for (int i = a + threadIdx.x; i < b; i += blockDim.x) tbl[i] = e;
}

// The gather layout of every entry's records (in the record buffer the run does not step in),
// at the start of a run.
template <class LP>
__global__ void __launch_bounds__(kStepThreads)
    k_gather_batch(const BatchEntry<LP> *__restrict__ entries, const int *__restrict__ firstBlocks,
                   const int *__restrict__ blockEntry) {
    const int ei = batch_entry(blockEntry);
    const BatchEntry<LP> &e = entries[ei];
    const int i = ((int)blockIdx.x - __ldg(firstBlocks + ei)) * kStepThreads + threadIdx.x;
    if (i < e.a.n) store_gather(reinterpret_cast<int4 *>(e.rec[e.cur0 ^ 1]), i, load_rec(e.rec[e.cur0] + i));
}

template <class LP>
__global__ void __launch_bounds__(kStepThreads, kForceBlocks<LP>)
    k_force_batch(const Consts<LP> c, const BatchEntry<LP> *__restrict__ entries,
                  const int *__restrict__ firstBlocks, const int *__restrict__ blockEntry, int s) {
    // the context's arguments in shared memory, where the per-particle loop reads them as
    // it goes (as it reads a single context's from the parameter bank), rather than in
    // registers held across the loop
    __shared__ StepArgs<LP> sa;
    const int ei = batch_entry(blockEntry);
    const BatchEntry<LP> &e = entries[ei];
    if (threadIdx.x == 0) {
        StepArgs<LP> a = e.a;
        a.gather = reinterpret_cast<int4 *>(e.rec[e.cur0 ^ 1]);
        a.step = e.step0 + s;
        a.breakPending = 0;
        sa = a;
    }
    __syncthreads();
    force_particle<LP, false, kForceAhead<LP>>(
        c, sa, ((int)blockIdx.x - __ldg(firstBlocks + ei)) * kStepThreads + threadIdx.x);
}

// The integrate step on the gather layout, in place; the records too where rec is not null.
// Streaming: 64 + 24 B read and 64 B (128 B with the records) written per particle (mixed); what
// it takes is warps enough to keep the loads in flight, so the registers are capped (a few bytes
// spill): 5.7M slab 136 us mixed, 257 us FP64, 153 and 439 us from and to the records uncapped.
template <class LP>
__device__ __forceinline__ void integrate_gather(const Consts<LP> &c, int4 *g, PRec<LP> *rec, const uint8_t *type,
                                                 const LP *force, int n, int i, bool reduce,
                                                 unsigned long long *diffMax) {
    LP dmax[3] = {LP(0), LP(0), LP(0)};
    if (i < n) {
        PRec<LP> me = gather_rec<LP>(g, i);
        LP F[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) F[q] = force[(long long)q * n + i];
        integrate_particle<LP>(c, me, type[i], F);
        store_gather(g, i, me);
        if (rec) store_rec(rec + i, me);
#pragma unroll
        for (int q = 0; q < 3; ++q) dmax[q] = me.d[q] > LP(0) ? me.d[q] : LP(0);
    }
    if (reduce) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            LP m = dmax[q];
            for (int o = 16; o > 0; o >>= 1) {
                LP u = __shfl_xor_sync(0xffffffffu, m, o);
                m = (u > m) ? u : m;
            }
            if ((threadIdx.x & 31) == 0 && m > LP(0)) atomicMax(diffMax + q, max_bits(m));
        }
    }
}

template <class LP>
__global__ void __launch_bounds__(kStepThreads, sizeof(LP) == 8 ? 7 : 8)
    k_integrate_gather(const Consts<LP> c, int4 *g, PRec<LP> *rec, const uint8_t *__restrict__ type,
                       const LP *force, int n, bool reduce, unsigned long long *diffMax) {
    dependent_start();
    integrate_gather<LP>(c, g, rec, type, force, n, blockIdx.x * blockDim.x + threadIdx.x, reduce, diffMax);
}

template <class LP>
__global__ void __launch_bounds__(kStepThreads)
    k_integrate_batch(const Consts<LP> c, const BatchEntry<LP> *__restrict__ entries,
                      const int *__restrict__ firstBlocks, const int *__restrict__ blockEntry, int s, bool last) {
    const int ei = batch_entry(blockEntry);
    const BatchEntry<LP> &e = entries[ei];
    const long long step = e.step0 + s;
    const int lb = (int)blockIdx.x - __ldg(firstBlocks + ei);
    if (e.reduceEvery10 && step % 10 == 0 && lb == 0 && threadIdx.x < 3) e.a.diffMax[threadIdx.x] = 0ull;
    integrate_gather<LP>(c, reinterpret_cast<int4 *>(e.rec[e.cur0 ^ 1]), last ? e.rec[e.cur0] : nullptr, e.a.type,
                         e.a.force, e.a.n, lb * kStepThreads + threadIdx.x,
                         e.reduceEvery10 && (step + 1) % 10 == 0, e.a.diffMax);
}

// Position and rotations alone (what the break functor reads).
template <class LP>
struct Pose {
    double x, y, z;
    LP th[3];
};
__device__ __forceinline__ void load_pose(Pose<float> &o, const int4 *base, int slot) {
    const int4 *p = base + gather_index<float>(slot);
    const double2 c0 = __ldg(reinterpret_cast<const double2 *>(p));
    const float4 c3 = __ldg(reinterpret_cast<const float4 *>(p + 96));
    o.x = c0.x;
    o.y = c0.y;
    o.z = __ldg(reinterpret_cast<const double *>(p + 32));
    o.th[0] = c3.y;
    o.th[1] = c3.z;
    o.th[2] = c3.w;
}
__device__ __forceinline__ void load_pose(Pose<double> &o, const int4 *base, int slot) {
    const double2 *p = reinterpret_cast<const double2 *>(base + gather_index<double>(slot));
    const double2 c0 = __ldg(p), c5 = __ldg(p + 160);
    o.x = c0.x;
    o.y = c0.y;
    o.z = __ldg(reinterpret_cast<const double *>(p + 32));
    o.th[0] = c5.x;
    o.th[1] = c5.y;
    o.th[2] = __ldg(reinterpret_cast<const double *>(p + 192));
}

// The break pass of the batch: one thread per link over a grid of its own (the links of
// entry e take CTAs [linkFirst[e], linkFirst[e + 1]), linkEntry maps a CTA to its entry),
// so that each thread's two gathers are in flight beside every other thread's, as in the
// single-context pass. Positions and rotations come from the gather layout; the functor's
// root and division are left to the links near the threshold (stays_whole).
template <class LP>
__global__ void __launch_bounds__(kStepThreads)
    k_break_batch(const Consts<LP> c, const BatchEntry<LP> *__restrict__ entries,
                  const int *__restrict__ linkFirst, const int *__restrict__ linkEntry, int s) {
    const int ei = batch_entry(linkEntry);
    const BatchEntry<LP> &e = entries[ei];
    const long long step = e.step0 + s;
    const long long l = (long long)((int)blockIdx.x - __ldg(linkFirst + ei)) * kStepThreads + threadIdx.x;
    // the sample main's gate t dt > breakTime (MainMeshBlock.cpp:312), in lp
    if ((LP)((LP)step * c.dt) > c.breakTime && l < e.L) {
        const uint8_t st = e.a.linkState[l];
        if (st != 0) {
            const int4 *g = reinterpret_cast<const int4 *>(e.rec[e.cur0 ^ 1]);
            Pose<LP> pa, pb;
            load_pose(pa, g, __ldg(e.slotA + l));
            load_pose(pb, g, __ldg(e.slotB + l));
            const LP L0 = __ldg(e.L0link + l);
            const LP x = (LP)(pa.x - pb.x), y = (LP)(pa.y - pb.y), z = (LP)(pa.z - pb.z);
            if (stays_whole<LP>(e.a, x * x + y * y + z * z, pa.th, pb.th, L0)) return;
            const uint8_t nst = break_link<LP>(e.a.bendBreak, e.a.maxLoad, pa, pb, st, L0);
            if (nst != st) {
                e.a.linkState[l] = nst;
                e.a.sState[e.sideSlot[2 * l]] = nst;
                e.a.sState[e.sideSlot[2 * l + 1]] = nst;
                if (nst == 0) {
                    const unsigned long long slot = atomicAdd(e.a.eventCount, 1ull);
                    if ((long long)slot < e.a.eventCap) e.a.events[slot] = make_int2((int)l, (int)step);
                }
            }
        }
    }
}

// HiDEMLib::applyForce with the integrate step, in place (split path).
template <class LP>
__global__ void k_integrate(const Consts<LP> c, PRec<LP> *__restrict__ rec,
                            const uint8_t *__restrict__ type, const LP *__restrict__ force, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    PRec<LP> me = load_rec(rec + i);
    LP F[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) F[q] = force[(long long)q * n + i];
    integrate_particle<LP>(c, me, type[i], F);
    store_rec(rec + i, me);
}

// HiDEMLib::linkUpdate: the break functor over every link
// (CombinedAccel::iterateLinks, CombinedAccel.h:200-235), with a warp-compacted
// flag-and-select append of the links that broke.
template <class LP>
__global__ void k_link_break(const Consts<LP> c, const PRec<LP> *__restrict__ rec,
                             const int *__restrict__ endA, const int *__restrict__ endB,
                             const int *__restrict__ sideSlot,
                             uint8_t *__restrict__ sState, uint8_t *__restrict__ linkState,
                             const LP *__restrict__ L0link, long long L, long long step,
                             int2 *__restrict__ events, unsigned long long *__restrict__ eventCount,
                             long long eventCap) {
    long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool broke = false;
    if (l < L) {
        // state and initial length in link order (coalesced); the side copies only on a change
        uint8_t st = linkState[l];
        if (st != 0) {
            const PRec<LP> pa = load_rec(rec + __ldg(endA + l));
            const PRec<LP> pb = load_rec(rec + __ldg(endB + l));
            uint8_t nst = break_link<LP>(c, pa, pb, st, __ldg(L0link + l));
            if (nst != st) {
                linkState[l] = nst;
                sState[sideSlot[2 * l]] = nst;
                sState[sideSlot[2 * l + 1]] = nst;
                broke = (nst == 0);
            }
        }
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, broke);
    if (ballot) {
        const int lane = threadIdx.x & 31;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(eventCount, (unsigned long long)__popc(ballot));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (broke) {
            unsigned long long slot = base + __popc(ballot & ((1u << lane) - 1u));
            if ((long long)slot < eventCap) events[slot] = make_int2((int)l, (int)step);
        }
    }
}

// max(0, xDiff), max(0, yDiff), max(0, zDiff) over all particles
// (HiDEMLib::getMaxDistOwned, HiDEMLib.h:424-461).
template <class LP>
__global__ void k_max_diff(const PRec<LP> *__restrict__ rec, int n,
                           unsigned long long *__restrict__ out) {
    LP v[3] = {LP(0), LP(0), LP(0)};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const PRec<LP> &p = rec[i];
#pragma unroll
        for (int q = 0; q < 3; ++q) v[q] = (p.d[q] > v[q]) ? p.d[q] : v[q];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        LP m = v[q];
        for (int o = 16; o > 0; o >>= 1) {
            LP u = __shfl_xor_sync(0xffffffffu, m, o);
            m = (u > m) ? u : m;
        }
        if ((threadIdx.x & 31) == 0 && m > LP(0)) atomicMax(out + q, max_bits(m));
    }
}

// ------------------------------------------------------------------ launchers

static inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

template <class LP>
void launch_bounds(const PRec<LP> *rec, int n, double *partial, int nb, double *out, cudaStream_t s) {
    k_bounds<LP><<<nb, 256, 0, s>>>(rec, n, partial);
    k_bounds_final<<<1, kBoundsFinalThreads, 0, s>>>(partial, nb, out);
}

template <class LP>
void launch_cells(const PRec<LP> *rec, int n, const GridInfo &g, int *cellOf, int *cellCount,
                  int *errorFlag, cudaStream_t s) {
    k_cells<LP><<<nblk(n, 256), 256, 0, s>>>(rec, n, g, cellOf, cellCount, errorFlag);
}

template <class TI, class TO>
int launch_scan(const TI *in, long long n, TO scaleBy, TO *out, TO *sums, TO *total, cudaStream_t s) {
    long long nb = (n + kScanBlock - 1) / kScanBlock;
    if (nb == 0) nb = 1;
    k_scan_blocks<TI, TO><<<(unsigned)nb, 256, 0, s>>>(in, n, scaleBy, out, sums);
    k_scan_sums<TO><<<1, 1024, 0, s>>>(sums, nb, total);
    k_scan_add<TO><<<nblk(n > 0 ? n : 1, 256), 256, 0, s>>>(out, n, sums);
    return 3;
}
template int launch_scan<int, int>(const int *, long long, int, int *, int *, int *, cudaStream_t);
template int launch_scan<int, long long>(const int *, long long, long long, long long *, long long *,
                                         long long *, cudaStream_t);

// position of each slot in the halo send list (-1: not sent): pos[slotOf[index[k]]] = k
__global__ void k_send_pos(const int *__restrict__ slotOf, const int *__restrict__ index, long long m,
                           int *__restrict__ pos) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) pos[slotOf[index[k]]] = (int)k;
}

void launch_send_pos(const int *slotOf, const int *index, long long m, int n, int *pos, cudaStream_t s) {
    cudaMemsetAsync(pos, 0xff, sizeof(int) * (size_t)n, s);
    if (m > 0) k_send_pos<<<nblk(m, 256), 256, 0, s>>>(slotOf, index, m, pos);
}

void launch_scatter(const int *cellOf, int n, const int *cellStart, int *cursor, int *perm,
                    cudaStream_t s) {
    k_scatter<<<nblk(n, 256), 256, 0, s>>>(cellOf, n, cellStart, cursor, perm);
}

int launch_sort_cells(const int *cellStart, const int *cellCount, long long total,
                      const int *origOld, int *perm, int *bigList, int *bigCount, int *errorFlag,
                      int errorCode, int smCount, cudaStream_t s) {
    cudaMemsetAsync(bigCount, 0, sizeof(int), s);
    k_sort_cells<<<nblk(total, 256), 256, 0, s>>>(cellStart, cellCount, total, origOld, perm,
                                                  bigList, bigCount);
    k_sort_big_cells<<<2 * smCount, kBigCellThreads, 0, s>>>(cellStart, cellCount, origOld, perm,
                                                             bigList, bigCount, errorFlag, errorCode);
    return 2;
}

template <class LP>
void launch_permute(const int *perm, int n, const PRec<LP> *recOld, PRec<LP> *recNew,
                    const uint8_t *typeOld, uint8_t *typeNew, const int *origOld, int *origNew,
                    const int *cellOld, int *cellNew, int *slotOf, int *newSlot, cudaStream_t s) {
    k_permute<LP><<<nblk(n, 256), 256, 0, s>>>(perm, n, recOld, recNew, typeOld, typeNew, origOld,
                                               origNew, cellOld, cellNew, slotOf, newSlot);
}

template <class LP>
void launch_nbr_count(const int4 *rec, int n, const int *cellOf, const GridInfo &g,
                      const int *cellStart, const int *cellCount, double interactDist,
                      uint32_t *counts, int *blockWidth, int *errorFlag, cudaStream_t s) {
    k_nbr_count<LP><<<nblk(n, 128), 128, 0, s>>>(rec, n, cellOf, g, cellStart, cellCount,
                                                 interactDist, counts, blockWidth, errorFlag);
}

template <class LP>
void launch_nbr_fill(const int4 *rec, int n, const int *cellOf, const GridInfo &g,
                     const int *cellStart, const int *cellCount, double interactDist,
                     const long long *nOff, int32_t *nbr, cudaStream_t s) {
    k_nbr_fill<LP><<<nblk(n, 128), 128, 0, s>>>(rec, n, cellOf, g, cellStart, cellCount,
                                                interactDist, nOff, nbr);
}

void launch_count_stats(const uint32_t *counts, int n, long long *out, int smCount, cudaStream_t s) {
    cudaMemsetAsync(out, 0, 3 * sizeof(long long), s);
    const int blocks = std::max(1, std::min(nblk(n, 256), 4 * smCount));
    k_count_stats<<<blocks, 256, 0, s>>>(counts, n, out);
}

void launch_side_count(const int *orig, int n, const int *plStart, uint32_t *counts,
                       int *blockWidth, int *errorFlag, cudaStream_t s) {
    k_side_count<<<nblk(n, 256), 256, 0, s>>>(orig, n, plStart, counts, blockWidth, errorFlag);
}

template <class LP>
void launch_side_fill(const int *orig, int n, const int *slotOf, const int *plStart,
                      const int *plLink, const uint8_t *plEnd, const int *linkA, const int *linkB,
                      const LP *L0link, const int *sideSlotOld, const SideView<LP> &oldS,
                      const long long *sOff, const SideView<LP> &newS, int *sideSlotNew,
                      cudaStream_t s) {
    k_side_fill<LP><<<nblk(n, 256), 256, 0, s>>>(orig, n, slotOf, plStart, plLink, plEnd, linkA,
                                                 linkB, L0link, sideSlotOld, oldS, sOff, newS,
                                                 sideSlotNew);
}

template <class LP, int WARPS>
static void launch_items(const Consts<LP> &c, const StepArgs<LP> &a, int blocks, size_t bytes, bool chained,
                         cudaStream_t s) {
    // the shared-memory limit is a per-device attribute: set it once on each device
    // (setting it twice, as racing threads may, is harmless)
    static std::atomic<unsigned long long> configured;
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        cudaFuncSetAttribute(k_step_items<LP, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kItemSmemLimit);
        configured.fetch_or(bit);
    }
    launch_dependent(chained, k_step_items<LP, WARPS>, blocks, WARPS * 32, bytes, s, c, a);
}

template <class LP>
void launch_step(const Consts<LP> &c, const StepArgs<LP> &a0, int maxContacts, int maxEnds, int kernel, int smCount,
                 bool chained, cudaStream_t s) {
    StepArgs<LP> a = a0;
    a.maxContacts = maxContacts;
    a.maxEnds = maxEnds;
    const size_t bytes = item_smem(sizeof(LP), maxContacts, maxEnds);
    if (kernel == HIDEM_STEP_KERNEL_ITEMS && bytes <= kItemSmemLimit) {
        // the fewer blocks, the more warps each (one block an SM: 16, so that no warp has more
        // than one link end and one contact of a lattice particle's twelve)
        const int nb = nblk(a.n, 32);
        if (nb <= smCount) launch_items<LP, 16>(c, a, nb, bytes, chained, s);
        else if (nb <= 3 * smCount) launch_items<LP, 8>(c, a, nb, bytes, chained, s);
        else launch_items<LP, 4>(c, a, nb, bytes, chained, s);
        return;
    }
    // one thread per particle (also for rows too wide for the item kernel's buffers)
    const int nb = nblk(a.n, kStepThreads);
    if (kernel == HIDEM_STEP_KERNEL_THREAD_ASYNC)
        k_step_async<LP, kAsyncBlocks<LP>><<<nb, kStepThreads, async_smem_bytes<LP>(), s>>>(c, a);
    else if (kernel == HIDEM_STEP_KERNEL_THREAD_CAPPED)
        k_step<LP, kCapBlocks<LP>><<<nb, kStepThreads, 0, s>>>(c, a);
    else
        k_step<LP, kThreadBlocks<LP>><<<nb, kStepThreads, 0, s>>>(c, a);
}

template <class LP>
void launch_side_move(const int *perm, int n, const int *newSlot, const uint32_t *counts, const long long *sOffOld,
                      const SideView<LP> &oldS, const long long *sOff, const SideView<LP> &newS, int *sideSlotNew,
                      cudaStream_t s) {
    k_side_move<LP><<<nblk(n, 256), 256, 0, s>>>(perm, n, newSlot, counts, sOffOld, oldS, sOff, newS, sideSlotNew);
}

template <class LP, bool AHEAD, int MINB>
static void launch_force_as(const Consts<LP> &c, const StepArgs<LP> &a, bool chained, cudaStream_t s) {
    const int nb = nblk(a.n, kStepThreads);
    if (a.breakPending)
        launch_dependent(chained, k_force<LP, true, AHEAD, MINB>, nb, kStepThreads, 0, s, c, a);
    else
        launch_dependent(chained, k_force<LP, false, AHEAD, MINB>, nb, kStepThreads, 0, s, c, a);
}

// A particle set that fits the chip in one wave at kFewBlocks CTAs an SM gains nothing from
// more warps an SM: it takes the variant that keeps the next item in flight.
template <class LP>
void launch_force(const Consts<LP> &c, const StepArgs<LP> &a, int smCount, bool chained, cudaStream_t s) {
    if (nblk(a.n, kStepThreads) <= kFewBlocks<LP> * smCount)
        launch_force_as<LP, true, kFewBlocks<LP>>(c, a, chained, s);
    else
        launch_force_as<LP, kForceAhead<LP>, kForceBlocks<LP>>(c, a, chained, s);
}

template <class LP>
void launch_to_gather(const PRec<LP> *rec, int n, int4 *g, cudaStream_t s) {
    launch_dependent(true, k_to_gather<LP>, nblk(n, 256), 256, 0, s, rec, n, g);
}
template <class LP>
void launch_from_gather(const int4 *g, int n, PRec<LP> *rec, cudaStream_t s) {
    k_from_gather<LP><<<nblk(n, 256), 256, 0, s>>>(g, n, rec);
}
template <class LP>
void launch_integrate_gather(const Consts<LP> &c, int4 *g, PRec<LP> *rec, const uint8_t *type, const LP *force,
                             int n, bool reduce, unsigned long long *diffMax, cudaStream_t s) {
    launch_dependent(true, k_integrate_gather<LP>, nblk(n, kStepThreads), kStepThreads, 0, s, c, g, rec, type, force, n,
                     reduce, diffMax);
}

template <class LP>
bool batch_fits(int maxContacts, int maxEnds) {
    return item_smem(sizeof(LP), maxContacts, maxEnds) <= kItemSmemLimit;
}

template <class LP>
void prepare_step_batch() {
    cudaFuncSetAttribute(k_step_batch<LP, HIDEM_STEP_KERNEL_ITEMS>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kItemSmemLimit);
}

int batch_particles_per_cta(int kernel) {
    return kernel == HIDEM_STEP_KERNEL_ITEMS ? 32 : kStepThreads;
}

void launch_block_table(const int *offs, int count, int *tbl, cudaStream_t s) {
    if (count > 0) k_block_table<<<count, 256, 0, s>>>(offs, tbl);
}

template <class LP>
void launch_step_batch(const Consts<LP> &c, const BatchEntry<LP> *entries, const int *firstBlocks,
                       const int *blockEntry, int run, int totalBlocks, int maxContacts, int maxEnds,
                       int kernel, cudaStream_t s) {
    if (kernel == HIDEM_STEP_KERNEL_ITEMS) {
        const size_t bytes = item_smem(sizeof(LP), maxContacts, maxEnds);
        k_step_batch<LP, HIDEM_STEP_KERNEL_ITEMS><<<totalBlocks, kItemThreads, bytes, s>>>(
            c, entries, firstBlocks, blockEntry, run);
    } else if (kernel == HIDEM_STEP_KERNEL_THREAD_CAPPED) {
        k_step_batch<LP, HIDEM_STEP_KERNEL_THREAD_CAPPED><<<totalBlocks, kStepThreads, 0, s>>>(
            c, entries, firstBlocks, blockEntry, run);
    } else {
        k_step_batch<LP, HIDEM_STEP_KERNEL_THREAD><<<totalBlocks, kStepThreads, 0, s>>>(
            c, entries, firstBlocks, blockEntry, run);
    }
}

template <class LP>
void launch_gather_batch(const BatchEntry<LP> *entries, const int *firstBlocks, const int *blockEntry,
                         int totalBlocks, cudaStream_t s) {
    k_gather_batch<LP><<<totalBlocks, kStepThreads, 0, s>>>(entries, firstBlocks, blockEntry);
}

template <class LP>
void launch_two_pass_batch(const Consts<LP> &c, const BatchEntry<LP> *entries, const int *firstBlocks,
                           const int *blockEntry, const int *linkFirst, const int *linkEntry, int run, bool last,
                           int totalBlocks, int totalLinkBlocks, cudaStream_t s) {
    k_force_batch<LP><<<totalBlocks, kStepThreads, 0, s>>>(c, entries, firstBlocks, blockEntry, run);
    k_integrate_batch<LP><<<totalBlocks, kStepThreads, 0, s>>>(c, entries, firstBlocks, blockEntry, run, last);
    k_break_batch<LP><<<totalLinkBlocks, kStepThreads, 0, s>>>(c, entries, linkFirst, linkEntry, run);
}

template <class LP>
void launch_integrate(const Consts<LP> &c, PRec<LP> *rec, const uint8_t *type, const LP *force,
                      int n, cudaStream_t s) {
    k_integrate<LP><<<nblk(n, 256), 256, 0, s>>>(c, rec, type, force, n);
}

template <class LP>
void launch_link_break(const Consts<LP> &c, const PRec<LP> *rec, const int *endA, const int *endB,
                       const int *sideSlot, uint8_t *sState, uint8_t *linkState, const LP *L0link,
                       long long L, long long step, int2 *events, unsigned long long *eventCount,
                       long long eventCap, cudaStream_t s) {
    if (L <= 0) return;
    k_link_break<LP><<<nblk(L, 256), 256, 0, s>>>(c, rec, endA, endB, sideSlot, sState,
                                                  linkState, L0link, L, step, events, eventCount,
                                                  eventCap);
}

// Kinetic energy with the integrate step's mass and moment of inertia (m = rho d^3,
// I = m d^2 / 6, MainMeshBlock.cpp:228-229) and velocities diff / dt; per-block sums in
// a fixed tree order, then one block over the partials, so the result is deterministic.
template <class LP>
__global__ void k_energy(const Consts<LP> c, const PRec<LP> *__restrict__ rec, int n,
                         double *__restrict__ partial) {
    __shared__ double red[3][256];
    double kt = 0, kr = 0, vmax = 0;
    const double dt = (double)c.dt, rho = (double)c.rhoIce;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const PRec<LP> p = load_rec(rec + i);
        const double d = 2.0 * (double)p.r;
        const double m = rho * d * d * d, I = m * d * d / 6.0;
        const double vx = p.d[0] / dt, vy = p.d[1] / dt, vz = p.d[2] / dt;
        const double wx = p.d[3] / dt, wy = p.d[4] / dt, wz = p.d[5] / dt;
        const double v2 = vx * vx + vy * vy + vz * vz;
        kt += 0.5 * m * v2;
        kr += 0.5 * I * (wx * wx + wy * wy + wz * wz);
        vmax = v2 > vmax ? v2 : vmax;
    }
    red[0][threadIdx.x] = kt;
    red[1][threadIdx.x] = kr;
    red[2][threadIdx.x] = vmax;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
            red[2][threadIdx.x] = fmax(red[2][threadIdx.x], red[2][threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; ++q) partial[q * gridDim.x + blockIdx.x] = red[q][0];
}

__global__ void k_energy_final(const double *__restrict__ partial, int nb, double *__restrict__ out) {
    __shared__ double red[3][256];
    double a = 0, b = 0, m = 0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        a += partial[i];
        b += partial[nb + i];
        m = fmax(m, partial[2 * nb + i]);
    }
    red[0][threadIdx.x] = a;
    red[1][threadIdx.x] = b;
    red[2][threadIdx.x] = m;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
            red[2][threadIdx.x] = fmax(red[2][threadIdx.x], red[2][threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; ++q) out[q] = red[q][0];
}

template <class LP>
void launch_energy(const Consts<LP> &c, const PRec<LP> *rec, int n, double *partial, int nb,
                   double *out, cudaStream_t s) {
    k_energy<LP><<<nb, 256, 0, s>>>(c, rec, n, partial);
    k_energy_final<<<1, 256, 0, s>>>(partial, nb, out);
}

// Linear momentum sum m v and angular momentum about the origin sum x (x) m v + I w, in
// double precision: per-block partials [6][gridDim.x] (tree sums in a fixed order), then
// one block folding them, so the result does not depend on scheduling.
template <class LP>
__global__ void k_momentum(const Consts<LP> c, const PRec<LP> *__restrict__ rec, int n,
                           double *__restrict__ partial) {
    __shared__ double red[6][256];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const double dt = (double)c.dt, rho = (double)c.rhoIce;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const PRec<LP> p = load_rec(rec + i);
        const double d = 2.0 * (double)p.r;
        const double m = rho * d * d * d, I = m * d * d / 6.0;
        const double px = m * (p.d[0] / dt), py = m * (p.d[1] / dt), pz = m * (p.d[2] / dt);
        acc[0] += px;
        acc[1] += py;
        acc[2] += pz;
        acc[3] += (p.y * pz - p.z * py) + I * (p.d[3] / dt);
        acc[4] += (p.z * px - p.x * pz) + I * (p.d[4] / dt);
        acc[5] += (p.x * py - p.y * px) + I * (p.d[5] / dt);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) red[q][threadIdx.x] = acc[q];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
#pragma unroll
            for (int q = 0; q < 6; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 6; ++q) partial[q * gridDim.x + blockIdx.x] = red[q][0];
}

__global__ void k_momentum_final(const double *__restrict__ partial, int nb, double *__restrict__ out) {
    __shared__ double red[6][256];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < nb; i += blockDim.x)
#pragma unroll
        for (int q = 0; q < 6; ++q) acc[q] += partial[q * nb + i];
#pragma unroll
    for (int q = 0; q < 6; ++q) red[q][threadIdx.x] = acc[q];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
#pragma unroll
            for (int q = 0; q < 6; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) out[threadIdx.x] = red[threadIdx.x][0];
}

template <class LP>
void launch_momentum(const Consts<LP> &c, const PRec<LP> *rec, int n, double *partial, int nb,
                     double *out, cudaStream_t s) {
    k_momentum<LP><<<nb, 256, 0, s>>>(c, rec, n, partial);
    k_momentum_final<<<1, 256, 0, s>>>(partial, nb, out);
}

template <class LP>
void launch_max_diff(const PRec<LP> *rec, int n, unsigned long long *out, int nb, cudaStream_t s) {
    k_max_diff<LP><<<nb, 256, 0, s>>>(rec, n, out);
}

#define HIDEM_INSTANTIATE(LP)                                                                      \
    template void launch_bounds<LP>(const PRec<LP> *, int, double *, int, double *, cudaStream_t); \
    template void launch_cells<LP>(const PRec<LP> *, int, const GridInfo &, int *, int *, int *,   \
                                   cudaStream_t);                                                  \
    template void launch_permute<LP>(const int *, int, const PRec<LP> *, PRec<LP> *,               \
                                     const uint8_t *, uint8_t *, const int *, int *, const int *,  \
                                     int *, int *, int *, cudaStream_t);                                  \
    template void launch_nbr_count<LP>(const int4 *, int, const int *, const GridInfo &,       \
                                       const int *, const int *, double, uint32_t *, int *, int *, \
                                       cudaStream_t);                                              \
    template void launch_nbr_fill<LP>(const int4 *, int, const int *, const GridInfo &,        \
                                      const int *, const int *, double, const long long *,         \
                                      int32_t *, cudaStream_t);                                    \
    template void launch_side_fill<LP>(const int *, int, const int *, const int *, const int *,    \
                                       const uint8_t *, const int *, const int *, const LP *,      \
                                       const int *, const SideView<LP> &, const long long *,       \
                                       const SideView<LP> &, int *, cudaStream_t);                 \
    template void launch_step<LP>(const Consts<LP> &, const StepArgs<LP> &, int, int, int, int, bool, \
                                  cudaStream_t);                                                   \
    template void launch_side_move<LP>(const int *, int, const int *, const uint32_t *, const long long *, \
                                       const SideView<LP> &, const long long *, const SideView<LP> &, int *, \
                                       cudaStream_t);                                              \
    template void launch_force<LP>(const Consts<LP> &, const StepArgs<LP> &, int, bool, cudaStream_t);     \
    template void launch_to_gather<LP>(const PRec<LP> *, int, int4 *, cudaStream_t);               \
    template void launch_from_gather<LP>(const int4 *, int, PRec<LP> *, cudaStream_t);             \
    template void launch_integrate_gather<LP>(const Consts<LP> &, int4 *, PRec<LP> *, const uint8_t *, \
                                              const LP *, int, bool, unsigned long long *, cudaStream_t); \
    template bool batch_fits<LP>(int, int);                                                        \
    template void prepare_step_batch<LP>();                                                        \
    template void launch_step_batch<LP>(const Consts<LP> &, const BatchEntry<LP> *, const int *,     \
                                        const int *, int, int, int, int, int, cudaStream_t);       \
    template void launch_gather_batch<LP>(const BatchEntry<LP> *, const int *, const int *, int,    \
                                          cudaStream_t);                                           \
    template void launch_two_pass_batch<LP>(const Consts<LP> &, const BatchEntry<LP> *, const int *, \
                                            const int *, const int *, const int *, int, bool, int,  \
                                            int, cudaStream_t);                                    \
    template void launch_integrate<LP>(const Consts<LP> &, PRec<LP> *, const uint8_t *,            \
                                       const LP *, int, cudaStream_t);                             \
    template void launch_link_break<LP>(const Consts<LP> &, const PRec<LP> *, const int *,         \
                                        const int *, const int *, uint8_t *, uint8_t *,            \
                                        const LP *, long long, long long, int2 *,                  \
                                        unsigned long long *, long long, cudaStream_t);            \
    template void launch_max_diff<LP>(const PRec<LP> *, int, unsigned long long *, int,            \
                                      cudaStream_t);                                               \
    template void launch_momentum<LP>(const Consts<LP> &, const PRec<LP> *, int, double *, int,     \
                                      double *, cudaStream_t);                                     \
    template void launch_energy<LP>(const Consts<LP> &, const PRec<LP> *, int, double *, int,       \
                                    double *, cudaStream_t);

HIDEM_INSTANTIATE(float)
HIDEM_INSTANTIATE(double)

}  // namespace hidem

// ------------------------------------------------------------------ setup / readback
// Packing between the caller's SoA arrays (input order) and the slot-ordered records,
// and the per-particle link-end lists, done on the device so that setup and readback
// cost one copy of each array.

namespace hidem {

template <class LP>
__global__ void k_pack_records(SoaIn<LP> s, int n, PRec<LP> *__restrict__ rec) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    PRec<LP> r;
    r.x = s.x[i];
    r.y = s.y[i];
    r.z = s.z[i];
#pragma unroll
    for (int k = 0; k < 6; ++k) r.d[k] = s.d[k] ? s.d[k][i] : LP(0);
    r.r = s.r[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) r.th[k] = s.th[k] ? s.th[k][i] : LP(0);
    if (sizeof(PRec<LP>) == 128) {
        double *pad = reinterpret_cast<double *>(&r) + 13;
        pad[0] = pad[1] = pad[2] = 0.0;
    }
    store_rec(rec + i, r);
}

// Slot-ordered records into caller-order arrays (null: not wanted).
template <class LP>
__global__ void k_unpack_records(const PRec<LP> *__restrict__ rec, const int *__restrict__ orig,
                                 int n, SoaOut<LP> s, const uint8_t *__restrict__ typeIn) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const PRec<LP> r = load_rec(rec + k);
    const int i = orig[k];
    if (s.x[0]) s.x[0][i] = r.x;
    if (s.x[1]) s.x[1][i] = r.y;
    if (s.x[2]) s.x[2][i] = r.z;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (s.d[q]) s.d[q][i] = r.d[q];
    if (s.r) s.r[i] = r.r;
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (s.th[q]) s.th[q][i] = r.th[q];
    if (s.type) s.type[i] = typeIn[k];
}

template <class LP>
__global__ void k_unpack_force(const LP *__restrict__ force, const int *__restrict__ orig, int n,
                               LP *__restrict__ out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = orig[k];
#pragma unroll
    for (int q = 0; q < 6; ++q) out[(long long)q * n + i] = force[(long long)q * n + k];
}

// Halo force exchange of a slab decomposition (CommunicatorPacked::packAllCommData /
// unpackAllCommData, HiDEMLib.h:337-372): one thread per (listed particle, component); the
// buffer holds 6 values per particle so that each peer's records are one contiguous run.
template <class LP>
__global__ void k_pack_halo(const LP *__restrict__ force, const int *__restrict__ slotOf,
                            const int *__restrict__ index, long long m, int n, LP *__restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * m) return;
    const long long k = t / 6;
    const int q = (int)(t - 6 * k);
    out[t] = force[(long long)q * n + slotOf[index[k]]];
}

template <class LP>
__global__ void k_unpack_halo(const LP *__restrict__ in, const int *__restrict__ slotOf,
                              const int *__restrict__ index, long long m, int n, LP *__restrict__ force) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * m) return;
    const long long k = t / 6;
    const int q = (int)(t - 6 * k);
    force[(long long)q * n + slotOf[index[k]]] = in[t];
}

// per-particle number of link ends
__global__ void k_link_degree(const int *__restrict__ A, const int *__restrict__ B, long long L,
                              int *__restrict__ deg) {
    long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= L) return;
    atomicAdd(deg + A[l], 1);
    atomicAdd(deg + B[l], 1);
}

__global__ void k_link_fill(const int *__restrict__ A, const int *__restrict__ B, long long L,
                            const int *__restrict__ start, int *__restrict__ cursor,
                            int *__restrict__ plLink, uint8_t *__restrict__ plEnd) {
    long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= L) return;
    int a = start[A[l]] + atomicAdd(cursor + A[l], 1);
    plLink[a] = (int)l;
    plEnd[a] = 0;
    int b = start[B[l]] + atomicAdd(cursor + B[l], 1);
    plLink[b] = (int)l;
    plEnd[b] = 1;
}

// A particle's ends in ascending link index (LinkAccelSide::generateLinks, LinkAccelSide.h:118-131).
// Sixteen lanes per particle: each holds one end, whose place is the number of smaller link
// indices among the others (indices of one particle's links are distinct); particles of more
// than sixteen ends are sorted by insertion by one lane. 0.48 ms on the 5.7M slab; one thread per
// particle sorting in memory took 1.47 ms.
constexpr int kSortLanes = 16;
__global__ void __launch_bounds__(256) k_link_sort_ends(const int *__restrict__ start, int n, int *__restrict__ plLink,
                                                        uint8_t *__restrict__ plEnd) {
    const int lane = threadIdx.x & (kSortLanes - 1);
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / kSortLanes;
    const int s = i < n ? start[i] : 0, cnt = i < n ? start[i + 1] - s : 0;
    if (cnt > kSortLanes) {
        if (lane == 0)
            for (int a = s + 1; a < s + cnt; ++a) {
                const int v = plLink[a];
                const uint8_t ve = plEnd[a];
                int b = a - 1;
                while (b >= s && plLink[b] > v) {
                    plLink[b + 1] = plLink[b];
                    plEnd[b + 1] = plEnd[b];
                    --b;
                }
                plLink[b + 1] = v;
                plEnd[b + 1] = ve;
            }
    }
    const bool mine = cnt <= kSortLanes && lane < cnt;
    const int v = mine ? plLink[s + lane] : 0x7fffffff;
    const uint8_t e = mine ? plEnd[s + lane] : uint8_t(0);
    int rank = 0;
#pragma unroll
    for (int k = 0; k < kSortLanes; ++k) rank += __shfl_sync(0xffffffffu, v, k, kSortLanes) < v ? 1 : 0;
    if (mine) {
        plLink[s + rank] = v;
        plEnd[s + rank] = e;
    }
}

// flat initial side layout: side 2l+e, state copied from the link
__global__ void k_side_init(const uint8_t *__restrict__ linkState, long long L,
                            int *__restrict__ sideSlot, uint8_t *__restrict__ sideState) {
    long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= 2 * L) return;
    sideSlot[s] = (int)s;
    sideState[s] = linkState[s >> 1];
}

// Side data back in the caller's order: CT[k][2l+e] and the link state (null: not wanted). One
// thread per link: both ends' slots in one load, every wanted array gathered through them, so
// that the slots (272 MB on the 5.7M slab) are read once and not once per array.
template <class LP>
__global__ void __launch_bounds__(256) k_gather_sides(const int2 *__restrict__ sideSlot, long long L,
                                                      SideGather<LP> g) {
    const long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= L) return;
    const int2 src = sideSlot[l];
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (g.out[q]) {
            g.out[q][2 * l] = g.ct[q][src.x];
            g.out[q][2 * l + 1] = g.ct[q][src.y];
        }
    if (g.stateOut) g.stateOut[l] = g.state[src.x];
}

__global__ void k_link_keys_identity(const long long *__restrict__ ka, const long long *__restrict__ kb,
                                     long long L, long long n, int *__restrict__ A, int *__restrict__ B,
                                     unsigned long long *badMin, unsigned long long *selfMin) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < L;
         i += (long long)gridDim.x * blockDim.x) {
        const long long a = ka[i], b = kb[i];
        if (a < 0 || a >= n || b < 0 || b >= n) {
            atomicMin(badMin, (unsigned long long)i);
            A[i] = 0;
            B[i] = 0;
            continue;
        }
        A[i] = (int)a;
        B[i] = (int)b;
        if (a == b) atomicMin(selfMin, (unsigned long long)i);
    }
}

// link ends from particle keys in strictly ascending order (not 0..n-1): each end's index
// by a binary search of the key table
__device__ __forceinline__ int find_key(const long long *__restrict__ keys, long long n, long long k) {
    long long lo = 0, hi = n;  // first position with keys[pos] >= k
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (__ldg(keys + mid) < k) lo = mid + 1;
        else hi = mid;
    }
    return (lo < n && __ldg(keys + lo) == k) ? (int)lo : -1;
}

__global__ void k_link_keys_sorted(const long long *__restrict__ keys, long long n,
                                   const long long *__restrict__ ka, const long long *__restrict__ kb,
                                   long long L, int *__restrict__ A, int *__restrict__ B,
                                   unsigned long long *badMin, unsigned long long *selfMin) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < L;
         i += (long long)gridDim.x * blockDim.x) {
        const int a = find_key(keys, n, ka[i]), b = find_key(keys, n, kb[i]);
        if (a < 0 || b < 0) {
            atomicMin(badMin, (unsigned long long)i);
            A[i] = 0;
            B[i] = 0;
            continue;
        }
        A[i] = a;
        B[i] = b;
        if (a == b) atomicMin(selfMin, (unsigned long long)i);
    }
}

void launch_link_keys_sorted(const long long *keys, long long n, const long long *keyA,
                             const long long *keyB, long long L, int *A, int *B,
                             unsigned long long *badMin, unsigned long long *selfMin, cudaStream_t st) {
    if (L <= 0) return;
    const int nb = (int)std::min<long long>((L + 255) / 256, 148LL * 32);
    k_link_keys_sorted<<<nb, 256, 0, st>>>(keys, n, keyA, keyB, L, A, B, badMin, selfMin);
}

__global__ void k_iota64(long long *out, long long count) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = i;
}

void launch_link_keys_identity(const long long *keyA, const long long *keyB, long long L,
                               long long n, int *A, int *B, unsigned long long *badMin,
                               unsigned long long *selfMin, cudaStream_t st) {
    if (L <= 0) return;
    const int nb = (int)std::min<long long>((L + 255) / 256, 148LL * 32);
    k_link_keys_identity<<<nb, 256, 0, st>>>(keyA, keyB, L, n, A, B, badMin, selfMin);
}

__global__ void k_iota32(int *out, int count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) out[i] = i;
}

// slots of both ends of every link in the current storage order (after a rebuild's permute)
__global__ void k_link_slots(const int *__restrict__ linkA, const int *__restrict__ linkB,
                             const int *__restrict__ slotOf, long long L, int *__restrict__ slotA,
                             int *__restrict__ slotB) {
    for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < L;
         l += (long long)gridDim.x * blockDim.x) {
        slotA[l] = slotOf[linkA[l]];
        slotB[l] = slotOf[linkB[l]];
    }
}

void launch_link_slots(const int *linkA, const int *linkB, const int *slotOf, long long L, int *slotA,
                       int *slotB, cudaStream_t st) {
    if (L <= 0) return;
    const int nb = (int)std::min<long long>((L + 255LL) / 256, 148LL * 32);
    k_link_slots<<<nb, 256, 0, st>>>(linkA, linkB, slotOf, L, slotA, slotB);
}

void launch_iota32(int *out, int count, cudaStream_t st) {
    if (count <= 0) return;
    const int nb = (int)std::min<long long>((count + 255LL) / 256, 148LL * 32);
    k_iota32<<<nb, 256, 0, st>>>(out, count);
}

// largest particle radius (radii are positive, so their IEEE bits order like the values)
template <class LP>
__global__ void k_max_radius(const PRec<LP> *__restrict__ rec, int n, unsigned long long *__restrict__ out) {
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = fmax(m, (double)rec[i].r);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

template <class LP>
void launch_max_radius(const PRec<LP> *rec, int n, unsigned long long *out, cudaStream_t st) {
    cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
    const int nb = (int)std::max<long long>(1, std::min<long long>((n + 255LL) / 256, 148LL * 4));
    k_max_radius<LP><<<nb, 256, 0, st>>>(rec, n, out);
}
template void launch_max_radius<float>(const PRec<float> *, int, unsigned long long *, cudaStream_t);
template void launch_max_radius<double>(const PRec<double> *, int, unsigned long long *, cudaStream_t);

void launch_iota64(long long *out, long long count, cudaStream_t st) {
    if (count <= 0) return;
    const int nb = (int)std::min<long long>((count + 255) / 256, 148LL * 32);
    k_iota64<<<nb, 256, 0, st>>>(out, count);
}

template <class LP>
void launch_pack_records(const SoaIn<LP> &s, int n, PRec<LP> *rec, cudaStream_t st) {
    k_pack_records<LP><<<nblk(n, 256), 256, 0, st>>>(s, n, rec);
}
template <class LP>
void launch_unpack_records(const PRec<LP> *rec, const int *orig, int n, const SoaOut<LP> &s,
                           const uint8_t *type, cudaStream_t st) {
    k_unpack_records<LP><<<nblk(n, 256), 256, 0, st>>>(rec, orig, n, s, type);
}
template <class LP>
void launch_unpack_force(const LP *force, const int *orig, int n, LP *out, cudaStream_t st) {
    k_unpack_force<LP><<<nblk(n, 256), 256, 0, st>>>(force, orig, n, out);
}
template <class LP>
void launch_halo_forces(LP *force, const int *slotOf, const int *index, long long m, int n, LP *buf,
                        bool pack, cudaStream_t st) {
    if (m <= 0) return;
    if (pack)
        k_pack_halo<LP><<<nblk(6 * m, 256), 256, 0, st>>>(force, slotOf, index, m, n, buf);
    else
        k_unpack_halo<LP><<<nblk(6 * m, 256), 256, 0, st>>>(buf, slotOf, index, m, n, force);
}
void launch_link_lists(const int *A, const int *B, long long L, int n, int *deg, int *start,
                       int *cursor, int *sums, int *plLink, uint8_t *plEnd, cudaStream_t st) {
    if (L > 0) k_link_degree<<<nblk(L, 256), 256, 0, st>>>(A, B, L, deg);
    // start[0..n] = exclusive scan of deg[0..n] with deg[n] = 0
    launch_scan<int, int>(deg, (long long)n + 1, 1, start, sums, nullptr, st);
    if (L > 0) k_link_fill<<<nblk(L, 256), 256, 0, st>>>(A, B, L, start, cursor, plLink, plEnd);
    k_link_sort_ends<<<nblk((long long)n * kSortLanes, 256), 256, 0, st>>>(start, n, plLink, plEnd);
}
void launch_side_init(const uint8_t *linkState, long long L, int *sideSlot, uint8_t *sideState,
                      cudaStream_t st) {
    if (L > 0) k_side_init<<<nblk(2 * L, 256), 256, 0, st>>>(linkState, L, sideSlot, sideState);
}
template <class LP>
void launch_gather_sides(const int *sideSlot, long long L, const SideGather<LP> &g, cudaStream_t st) {
    if (L > 0) k_gather_sides<LP><<<nblk(L, 256), 256, 0, st>>>(reinterpret_cast<const int2 *>(sideSlot), L, g);
}

#define HIDEM_INSTANTIATE_IO(LP)                                                                   \
    template void launch_pack_records<LP>(const SoaIn<LP> &, int, PRec<LP> *, cudaStream_t);       \
    template void launch_unpack_records<LP>(const PRec<LP> *, const int *, int, const SoaOut<LP> &, \
                                            const uint8_t *, cudaStream_t);                        \
    template void launch_unpack_force<LP>(const LP *, const int *, int, LP *, cudaStream_t);       \
    template void launch_halo_forces<LP>(LP *, const int *, const int *, long long, int, LP *, bool, \
                                         cudaStream_t);                                            \
    template void launch_gather_sides<LP>(const int *, long long, const SideGather<LP> &, cudaStream_t);
HIDEM_INSTANTIATE_IO(float)
HIDEM_INSTANTIATE_IO(double)

}  // namespace hidem
