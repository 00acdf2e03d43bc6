// Kernels of the gridded background sums (see hphc_grid.h).
#include "hphc_grid.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace hphc {
namespace {

constexpr int kBin = kGridBin;
template <int P>
constexpr int kRegion = kBin + P - 1;  // nodes a bin's events touch, per coordinate

template <int N>
constexpr double kFactorial = N * kFactorial<N - 1>;  // exact to 22!
template <>
constexpr double kFactorial<1> = 1.0;

// Convolution table G[|lag|].
template <int P>
struct GridTaps {
    double g[GridOrder<P>::kTaps + 1];
};

struct Batch {
    GridJob job[kGridMaxJobs];
    int n;
};

// Blocks of a launch over several jobs: job k has blocks [first[k], first[k + 1]), so
// that jobs of any size leave no empty blocks.
struct Blocks {
    unsigned first[kGridMaxJobs + 1];
};

__device__ __forceinline__ const GridJob& find_job(const Batch& b, const Blocks& blocks,
                                                   unsigned* index) {
    int k = 0;
    while (k + 1 < b.n && blockIdx.x >= blocks.first[k + 1]) ++k;
    *index = blockIdx.x - blocks.first[k];
    return b.job[k];
}

// Position of event e along coordinate d (0 = t, 1 = y, 2 = x) in grid units:
// cell (>= 0, clamped to the grid) and fraction.  The product with the
// double-double scale keeps the fraction to ~1e-17 cells, so the position is as
// exact as the input.
__device__ __forceinline__ double coordinate(const GridJob& J, int e, int d) {
    if (d == 0) return J.times[e];
    if (d == 1) return J.D == 2 ? J.loc[(size_t)2 * e + 1] : 0.0;
    return J.loc[(size_t)J.D * e];
}

__device__ __forceinline__ void grid_position(const GridJob& J, int e, int d, int* cell,
                                              double* frac) {
    const double v = coordinate(J, e, d);
    const double hi = v * J.scaleHi[d];
    const double lo = fma(v, J.scaleHi[d], -hi) + v * J.scaleLo[d];
    const double fl = floor(hi);
    *frac = (hi - fl) + lo;
    *cell = min(max((int)(fl - J.origin[d]), 0), J.nc[d] - 1);
}

// Copies 8 bytes from global to shared memory in the background, or stores 0.0
// there (live = false; src is then not read but has to be a valid address).
__device__ __forceinline__ void copy8_async(double* dst, const double* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(live ? 8 : 0));
}
// The same for 16 bytes, 16-byte aligned on both sides.
__device__ __forceinline__ void copy16_async(double* dst, const double* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(live ? 16 : 0));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// ---- binning ----------------------------------------------------------------
//
// Events are sorted into bins of kBin^3 cells by counting.  The arrival order
// inside a bin is not deterministic; the weights kernel gives every event its
// rank by (t cell, event number) there, so the sums over a bin always run in the
// same order.

constexpr int kCellThreads = 256;

__global__ void __launch_bounds__(kCellThreads) zero_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks) {
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int i = block * kCellThreads + threadIdx.x;
    if (i < J.nb[0] * J.nb[1] * J.nb[2]) J.start[i] = 0;
}

__global__ void __launch_bounds__(kCellThreads) count_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks) {
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int e = block * kCellThreads + threadIdx.x;
    if (e >= J.N) return;
    int c[3];
    double f;
    for (int d = 0; d < 3; ++d) grid_position(J, e, d, &c[d], &f);
    const int bin = ((c[0] / kBin) * J.nb[1] + c[1] / kBin) * J.nb[2] + c[2] / kBin;
    J.binOf[e] = bin * kBin + (c[0] & (kBin - 1));
    J.pos[e] = atomicAdd(J.start + bin, 1);
}

// Exclusive prefix sums of the bin counts and the gather's work items, one CTA per
// job.
constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.x];
    const int nb = J.nb[0] * J.nb[1] * J.nb[2];
    __shared__ int2 warpSum[kScanThreads / 32];
    __shared__ int2 carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry = make_int2(0, 0);
    __syncthreads();
    const auto warp_scan = [&](int2 v) {
        for (int d = 1; d < 32; d <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, v.x, d), y = __shfl_up_sync(0xffffffffu, v.y, d);
            if (lane >= d) v.x += x, v.y += y;
        }
        return v;
    };
    for (int i0 = 0; i0 < nb; i0 += kScanThreads) {
        const int i = i0 + tid;
        const int v = i < nb ? J.start[i] : 0;
        const int items = (v + kGridItemEvents - 1) / kGridItemEvents;
        const int2 x = warp_scan(make_int2(v, items));
        if (lane == 31) warpSum[warp] = x;
        __syncthreads();
        if (warp == 0) warpSum[lane] = warp_scan(warpSum[lane]);
        __syncthreads();
        const int2 before = warp ? warpSum[warp - 1] : make_int2(0, 0);
        const int first = carry.x + before.x + x.x - v, item = carry.y + before.y + x.y - items;
        if (i < nb) {
            J.start[i] = first;
            for (int k = 0; k < items; ++k)
                J.items[item + k] = make_int2(i, first + k * kGridItemEvents);
        }
        __syncthreads();
        if (tid == kScanThreads - 1)
            carry = make_int2(first + v, item + items);
        __syncthreads();
    }
    if (tid == 0) {
        J.start[nb] = carry.x;
        *J.nItems = carry.y;
    }
}

__global__ void __launch_bounds__(kCellThreads) place_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks) {
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int e = block * kCellThreads + threadIdx.x;
    if (e >= J.N) return;
    const int bin = J.binOf[e];
    J.key[J.start[bin / kBin] + J.pos[e]] = ((unsigned)(bin % kBin) << 28) | (unsigned)e;
}

// Weights of the cardinal B-spline of order P at fraction f: node i of the
// event holds M_P(f + P - 1 - i), so that node 0 is the event's cell.  The
// recursion M_n(x) = (x M_{n-1}(x) + (n - x) M_{n-1}(x - 1)) / (n - 1) runs
// without its divisions (all terms positive, no rounded reciprocals); one
// factor 1 / (P - 1)! ends it.  The second derivative is the second difference
// of the order P - 2 weights.
template <int P>
__device__ __forceinline__ void spline_weights(double f, double* __restrict__ wv,
                                               double* __restrict__ wd) {
    constexpr double kInvP1 = 1.0 / kFactorial<P - 1>, kInvP3 = 1.0 / kFactorial<P - 3>;
    double v[P];  // v[i] = (n - 1)! M_n(f + i)
    v[0] = f;
    v[1] = 1.0 - f;
#pragma unroll
    for (int n = 3; n <= P - 2; ++n) {
        v[n - 1] = ((double)n - (f + (n - 1))) * v[n - 2];
#pragma unroll
        for (int i = n - 2; i > 0; --i)
            v[i] = fma(f + i, v[i], ((double)n - (f + i)) * v[i - 1]);
        v[0] = f * v[0];
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const double a = i < P - 2 ? v[i] : 0.0;
        const double m = i >= 1 && i - 1 < P - 2 ? v[i - 1] : 0.0;
        const double z = i >= 2 ? v[i - 2] : 0.0;
        wd[P - 1 - i] = ((a - m) + (z - m)) * kInvP3;
    }
#pragma unroll
    for (int n = P - 1; n <= P; ++n) {
        v[n - 1] = ((double)n - (f + (n - 1))) * v[n - 2];
#pragma unroll
        for (int i = n - 2; i > 0; --i)
            v[i] = fma(f + i, v[i], ((double)n - (f + i)) * v[i - 1]);
        v[0] = f * v[0];
    }
#pragma unroll
    for (int i = 0; i < P; ++i) wv[P - 1 - i] = v[i] * kInvP1;
}

// Three threads a slot, one per coordinate; the slot's first thread ranks it.
// The weights leave through shared memory, a warp writing whole rows.  Bound by
// those writes: 960 bytes an event at order 16, N = 100k 35 us (2.7 TB/s, most of
// it to L2), 44 before the slots left as whole aligned rows.
constexpr int kWeightSlots = 32;
constexpr int kWeightThreads = 3 * kWeightSlots;

template <int P>
__global__ void __launch_bounds__(kWeightThreads)
weights_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks) {
    constexpr int kRow = 6 * P + 1;  // odd: slots on distinct banks
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    __shared__ int sDst[kWeightSlots], sCell[3][kWeightSlots];
    __shared__ double sRows[kWeightSlots * kRow];
    const int d = threadIdx.x / kWeightSlots, i = threadIdx.x % kWeightSlots;
    const int slot0 = block * kWeightSlots, slot = slot0 + i;
    const bool live = slot < J.N;
    const unsigned k = live ? J.key[slot] : 0;
    const int e = (int)(k & 0x0fffffffu);
    double f = 0.0;
    if (live) {
        grid_position(J, e, d, &sCell[d][i], &f);
        spline_weights<P>(f, sRows + i * kRow + d * P, sRows + i * kRow + (3 + d) * P);
    }
    if (d == 0 && live) {
        const int bin = J.binOf[e] / kBin;
        const int s0 = J.start[bin], s1 = J.start[bin + 1];
        int rank = s0;
#pragma unroll 8
        for (int s = s0; s < s1; ++s) rank += J.key[s] < k;
        sDst[i] = rank;
        J.event[rank] = e;
    }
    __syncthreads();
    const int rows = min(kWeightSlots, J.N - slot0);
    for (int r = d; r < rows; r += 3) {
        const size_t dst = sDst[r];
        const double* row = sRows + r * kRow;
        const int c[3] = {sCell[0][r] % kBin, sCell[1][r] % kBin, sCell[2][r] % kBin};
        if (i == 0) J.cell[dst] = c[0] | c[1] << 8 | c[2] << 16;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int k = i - c[q];
            if (i < kGridSpan)
                J.wv[(dst * 3 + q) * kGridSpan + i] = (unsigned)k < (unsigned)P ? row[q * P + k] : 0.0;
        }
        for (int v = i; v < 3 * P; v += kWeightSlots) J.wd[dst * 3 * P + v] = row[3 * P + v];
    }
}

// ---- spread -------------------------------------------------------------------
//
// A CTA owns an output tile of 8 x 8 x 16 nodes (t, y, x) and adds every event
// that touches it: no atomics, no halo, a fixed order.  For one t row the update
// by four events is an 8 x 4 by 4 x 8 product, W[y][x] += sum_k (wt wy)[y][k]
// wx[k][x], which is one FP64 tensor instruction (mma m8n8k4).  It reaches the
// full FP64 rate (63 of 64 multiply-adds a clock), where a DFMA of three
// different registers reaches 42: the register ports bound it.  The warps of the
// CTA take the groups of four events in turn, each with the slices of the
// weights that fall into the tile copied to shared memory one group ahead (the
// stored weights start at a bin's first node, so every slice is a whole aligned
// 64 bytes), and their tiles are added in warp order.  Events are sorted by t cell
// inside their bin, so rows that none of the four touches are left out.
// N = 100k (order 16): 190 us, the tensor pipe active 34 % of them; the copies and row
// reductions of each group lie between.  Warps that share staged groups, two or four t rows each, took
// 245 and 226 us: the barriers cost more than the sum over the warps' tiles.

constexpr int kSpreadThreads = 128;
constexpr int kSpreadWarps = kSpreadThreads / 32;
constexpr int kTileT = 8, kTileY = 8, kTileX = 16;
constexpr int kSlice = kTileT + kTileY + kTileX;  // weights of an event in the tile
static_assert(kSlice == 32, "one weight per lane");
constexpr int kSlicePitch = kSlice + 4;  // events of a group on distinct banks

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// The bins whose events touch a tile: 3 x 3 x 4 at most.
struct Bins {
    int first[36], last[36];  // slots
    int group[37];            // groups of four before the bin
    int shift[36];            // bins from it to the tile's first: t | y << 4 | (x + 1) << 8
    int n;
};

template <int P>
__global__ void __launch_bounds__(kSpreadThreads, 4)
spread_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks) {
    static_assert(P - 1 <= 2 * kBin && P - 1 > kBin && kBin + P - 1 <= kGridSpan,
                  "bins that touch a tile");
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int ntx = (J.n[2] + kTileX - 1) / kTileX, nty = (J.n[1] + kTileY - 1) / kTileY;
    const int tx = block % ntx, ty = block / ntx % nty, tt = block / (ntx * nty);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = lane & 3, row = lane >> 2;

    __shared__ Bins bins;
    __shared__ __align__(16) double sSlice[kSpreadWarps][2][4][kSlicePitch];
    if (warp == 0) {
        // an event of cell c touches nodes c .. c + P - 1: bins -2 .. 0 of the tile's own
        int groups = 0, n = 0;
        for (int half = 0; half < 2; ++half) {
            const int v = lane + 32 * half;
            const int dt = v / 12, dy = v / 4 % 3, dx = v % 4 - 1;
            const int bt = tt - dt, by = ty - dy, bx = 2 * tx - dx;
            int s0 = 0, s1 = 0;
            if (v < 36 && bt >= 0 && by >= 0 && bx >= 0 && bt < J.nb[0] && by < J.nb[1] &&
                bx < J.nb[2]) {
                const int bin = (bt * J.nb[1] + by) * J.nb[2] + bx;
                s0 = J.start[bin];
                s1 = J.start[bin + 1];
            }
            const int g = (s1 - s0 + 3) / 4;
            int sum = g;
            for (int d = 1; d < 32; d <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += x;
            }
            const unsigned mask = __ballot_sync(0xffffffffu, g > 0);
            if (g > 0) {
                const int at = n + __popc(mask & ((1u << lane) - 1));
                bins.first[at] = s0;
                bins.last[at] = s1;
                bins.group[at] = groups + sum - g;
                bins.shift[at] = dt | dy << 4 | (dx + 1) << 8;
            }
            n += __popc(mask);
            groups += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) {
            bins.group[n] = groups;
            bins.n = n;
        }
    }
    __syncthreads();
    const int groups = bins.group[bins.n];

    double acc[2][kTileT][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < kTileT; ++r) acc[h][r][0] = acc[h][r][1] = 0.0;

    // One 16-byte piece of two events of a group: lanes 0-15 the first's, 16-31 the
    // second's; 4 pieces of the t rows, 4 of the y rows, 4 each of the x halves.
    const int piece = lane & 15, part = piece / 4;
    int bin = 0, shift = 0;
    // starts group q's copies into a stage; returns the t cell of event k (-1: none)
    const auto copy = [&](int stage, int q) {
        if (q >= groups) {
            copy_commit();
            return -1;
        }
        while (q >= bins.group[bin + 1]) ++bin;
        const int s0 = bins.first[bin] + 4 * (q - bins.group[bin]), last = bins.last[bin];
        shift = bins.shift[bin];
        const int away = part == 0 ? shift & 15 : part == 1 ? shift >> 4 & 15
                                                            : (shift >> 8) - 1 + (part - 2);
        const double* src = J.wv + (min(part, 2) * kGridSpan + away * kBin + 2 * (piece & 3));
        const bool inside = away >= 0 && away < kGridSpan / kBin;
#pragma unroll
        for (int ev = 0; ev < 4; ev += 2) {
            const int s = s0 + ev + (lane >> 4);
            const bool live = inside && s < last;
            copy16_async(&sSlice[warp][stage][ev + (lane >> 4)][2 * piece],
                         live ? src + (size_t)s * 3 * kGridSpan : J.wv, live);
        }
        copy_commit();
        return s0 + k < last ? J.cell[s0 + k] & 255 : -1;
    };

    int cell = copy(0, warp);
    int away = shift;
    int stage = 0;
    for (int q = warp; q < groups; q += kSpreadWarps, stage ^= 1) {
        const int next = copy(stage ^ 1, q + kSpreadWarps);
        // rows the group touches: cell - 8 (bins to the tile) and P - 1 more
        const int ct = cell - kBin * (away & 15);
        const int lo = __reduce_min_sync(0xffffffffu, cell >= 0 ? max(0, ct) : kTileT);
        const int hi = __reduce_max_sync(0xffffffffu, cell >= 0 ? min(kTileT - 1, P - 1 + ct) : -1);
        const int dx = (away >> 8) - 1;
        const bool h0 = dx >= 0, h1 = dx < 2;  // x halves within the bin's reach
        copy_wait<1>();
        __syncwarp();
        const double* w = sSlice[warp][stage][k];
        const double wy = w[kTileT + row], wx0 = w[kTileT + kTileY + row],
                     wx1 = w[kTileT + kTileY + 8 + row];
#pragma unroll
        for (int r = 0; r < kTileT; r += 2) {
            const double2 wt = *reinterpret_cast<const double2*>(w + r);
            if (r >= lo && r <= hi) {
                const double a = wy * wt.x;
                if (h0) mma_f64(acc[0][r], a, wx0);
                if (h1) mma_f64(acc[1][r], a, wx1);
            }
            if (r + 1 >= lo && r + 1 <= hi) {
                const double a = wy * wt.y;
                if (h0) mma_f64(acc[0][r + 1], a, wx0);
                if (h1) mma_f64(acc[1][r + 1], a, wx1);
            }
        }
        __syncwarp();
        cell = next;
        away = shift;
    }
    copy_wait<0>();

    const int t0 = tt * kTileT, y0 = ty * kTileY, x0 = tx * kTileX;
    __shared__ double2 tile[kTileT][kTileY][kTileX / 2];
    for (int w = 0; w < kSpreadWarps; ++w) {
        if (w == warp) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < kTileT; ++r) {
                    double2& v = tile[r][row][4 * h + k];
                    v = w == 0 ? make_double2(acc[h][r][0], acc[h][r][1])
                               : make_double2(v.x + acc[h][r][0], v.y + acc[h][r][1]);
                }
        }
        __syncthreads();
    }
    const double* flat = reinterpret_cast<const double*>(tile);
    for (int v = threadIdx.x; v < kTileT * kTileY * kTileX; v += kSpreadThreads) {
        const int x = x0 + v % kTileX, y = y0 + v / kTileX % kTileY, t = t0 + v / (kTileX * kTileY);
        if (x < J.n[2] && y < J.n[1] && t < J.n[0])
            J.ga[((size_t)t * J.n[1] + y) * J.n[2] + x] = flat[v];
    }
}

// ---- convolution ----------------------------------------------------------------
//
// One pass per coordinate; a thread forms kConvOut consecutive outputs of a line,
// so each input it reads feeds kConvOut multiply-adds.  Lines of the y and t
// passes lie across the threads of a warp (coalesced); the x pass stages 32 lines
// in shared memory, one per lane, at an odd pitch (no bank conflicts).  N = 100k,
// 1.24e6 nodes, order 16 (97 taps): 25 + 20 + 21 us, the FP64 pipe's floor for their
// multiply-adds 6.5 us each; the reads and the first and last taps' zeros are the rest.

constexpr int kConvOut = 16;
template <int P>
constexpr int kTapPad = GridOrder<P>::kTaps + kConvOut;  // table index of lag 0

template <int P>
__device__ __forceinline__ void stage_taps(const GridTaps<P>& taps, double* sTap) {
    for (int v = threadIdx.x; v < 2 * kTapPad<P>; v += blockDim.x) {
        const int lag = abs(v - kTapPad<P>);
        sTap[v] = lag <= GridOrder<P>::kTaps ? taps.g[lag] : 0.0;
    }
}

// 16 outputs o0 .. o0 + 15 from input(j), j in [o0 - kTaps, o0 + kTaps + 16).
template <int P, class Input>
__device__ __forceinline__ void convolve(const double* __restrict__ sTap, int o0, Input input,
                                         double (&out)[kConvOut]) {
    constexpr int kTaps = GridOrder<P>::kTaps;
    static_assert(kTaps % kConvOut == 0, "whole blocks of taps");
#pragma unroll
    for (int i = 0; i < kConvOut; ++i) out[i] = 0.0;
#pragma unroll 1
    for (int jb = -kTaps; jb <= kTaps; jb += kConvOut) {
        double in[kConvOut];
#pragma unroll
        for (int j = 0; j < kConvOut; ++j) in[j] = input(o0 + jb + j);
        const double* t = sTap + kTapPad<P> + jb;
#pragma unroll
        for (int d = -(kConvOut - 1); d < kConvOut; ++d) {
            const double g = t[d];
#pragma unroll
            for (int i = 0; i < kConvOut; ++i)
                if (i + d >= 0 && i + d < kConvOut) out[i] = fma(g, in[i + d], out[i]);
        }
    }
}

constexpr int kLineThreads = 128;

// The pass along y (axis 1: ga from gb) or t (axis 0: gb from ga).
template <int P>
__global__ void __launch_bounds__(kLineThreads)
conv_line_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks,
                 const __grid_constant__ GridTaps<P> taps, int axis) {
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int len = J.n[axis];
    const int stride = axis == 1 ? J.n[2] : J.n[1] * J.n[2];
    const int lines = axis == 1 ? J.n[0] * J.n[2] : stride;
    const int chunks = (len + kConvOut - 1) / kConvOut;
    __shared__ double sTap[2 * kTapPad<P>];
    stage_taps<P>(taps, sTap);
    __syncthreads();
    const int chunk = block % chunks;
    const int line = block / chunks * kLineThreads + threadIdx.x;
    if (line >= lines) return;
    const double* src = axis == 1 ? J.gb : J.ga;
    double* dst = axis == 1 ? J.ga : J.gb;
    const size_t base = (size_t)(line / stride) * len * stride + line % stride;
    const int o0 = chunk * kConvOut;
    double out[kConvOut];
    convolve<P>(sTap, o0, [&](int j) {
        return (unsigned)j < (unsigned)len ? src[base + (size_t)j * stride] : 0.0;
    }, out);
#pragma unroll
    for (int i = 0; i < kConvOut; ++i)
        if (o0 + i < len) dst[base + (size_t)(o0 + i) * stride] = out[i];
}

constexpr int kRowLines = 32;                       // lines of a CTA
constexpr int kRowWarps = 8;
constexpr int kRowOut = kRowWarps * kConvOut;       // outputs of a line in a CTA
template <int P>
constexpr int kRowPitch = kRowOut + 2 * GridOrder<P>::kTaps + 1;  // odd

template <int P>
__global__ void __launch_bounds__(32 * kRowWarps)
conv_row_kernel(const __grid_constant__ Batch b, const __grid_constant__ Blocks blocks,
                const __grid_constant__ GridTaps<P> taps) {
    constexpr int kTaps = GridOrder<P>::kTaps, kPitch = kRowPitch<P>;
    extern __shared__ double sRow[];  // [kRowLines][kPitch]
    __shared__ double sTap[2 * kTapPad<P>];
    unsigned block;
    const GridJob& J = find_job(b, blocks, &block);
    const int len = J.n[2], lines = J.n[0] * J.n[1];
    const int chunks = (len + kRowOut - 1) / kRowOut;
    const int o0 = block % chunks * kRowOut, l0 = block / chunks * kRowLines;
    const int outs = min(kRowOut, len - o0), rows = min(kRowLines, lines - l0);
    stage_taps<P>(taps, sTap);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < kRowLines; r += kRowWarps)
        for (int j = lane; j < kPitch; j += 32) {
            const int x = o0 - kTaps + j;
            const bool live = r < rows && (unsigned)x < (unsigned)len;
            copy8_async(sRow + r * kPitch + j, J.ga + (live ? (size_t)(l0 + r) * len + x : 0), live);
        }
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    double out[kConvOut];
    const double* line = sRow + lane * kPitch;
    const int w0 = warp * kConvOut;
    if (w0 < outs) convolve<P>(sTap, w0, [&](int j) { return line[j + kTaps]; }, out);
    __syncthreads();
    if (w0 < outs)
#pragma unroll
        for (int i = 0; i < kConvOut; ++i) sRow[lane * kPitch + w0 + i] = out[i];
    __syncthreads();
    for (int r = warp; r < rows; r += kRowWarps)
        for (int j = lane; j < outs; j += 32)
            J.gb[(size_t)(l0 + r) * len + o0 + j] = sRow[r * kPitch + j];
}

// ---- gather ---------------------------------------------------------------------
//
// CTAs take the items (a bin's events, at most kGridItemEvents) in turn.  A CTA
// stages the (7 + P)^3 nodes the bin's events touch in shared memory and its
// warps take the events in turn: lane (h, y) forms the x products of node rows y of
// its share of the P t planes, for the spline and for its second derivative, and
// the other two coordinates follow on the lane's own sums.  The odd pitch puts the
// rows of a half warp on distinct banks.  Bound: shared memory, P^3 doubles an event
// at 16 a clock (N = 100k order 16: 37.3e6
// wavefronts, 128 of 175 us, the pipe 78 % busy; 270 with the region and the weights
// loaded in step, 200 with the region asynchronous, 174 with the weights too and
// persistent CTAs).

constexpr int kGatherThreads = 256;
constexpr int kGatherWarps = kGatherThreads / 32;

// Pitch of the t planes: with two lane shares of P < 16 rows in a half warp, the
// second share's banks continue where the first's end (kPlanes * pitch = P * row
// pitch modulo the 16 banks of 8 bytes).
template <int P>
constexpr int kPlanePitch = P == 12 ? 366 : kRegion<P> * kRegion<P>;
static_assert(kPlanePitch<12> >= kRegion<12> * kRegion<12> &&
                  (6 * kPlanePitch<12>) % 16 == (12 * kRegion<12>) % 16,
              "bank layout");
template <int P>
constexpr int kRegionNodes = (kRegion<P> * kPlanePitch<P> + 1) / 2 * 2;
constexpr int kGatherRow = 3 * kGridSpan;  // stored spline weights of an event
template <int P>
constexpr int kGatherWeights = kGatherRow + 3 * P;  // with the second derivatives
template <int P>
constexpr size_t kGatherShared =
    (kRegionNodes<P> + kGatherWarps * 2 * kGatherWeights<P>) * sizeof(double);

template <int P>
__global__ void __launch_bounds__(kGatherThreads, 2)
gather_kernel(const __grid_constant__ Batch b) {
    constexpr int kR = kRegion<P>;
    constexpr int kPP = kPlanePitch<P>;
    constexpr int kShares = 32 / P, kPlanes = P / kShares;  // of the t planes
    static_assert(P % kShares == 0 && kR % 2 == 1 && P % 2 == 0 && kPlanes % 2 == 0,
                  "lane layout");
    extern __shared__ __align__(16) double sF[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sW = sF + kRegionNodes<P> + warp * 2 * kGatherWeights<P>;  // two events
    const int y = lane % P, h = lane / P;
    const bool busy = h < kShares;
    int item = blockIdx.x;
    for (int k = 0; k < b.n; ++k) {
        const GridJob& J = b.job[k];
        const int nItems = *J.nItems;
        const int n1 = J.n[1], n2 = J.n[2];
        for (; item < nItems; item += gridDim.x) {
            const int bin = J.items[item].x, s0 = J.items[item].y;
            const int s1 = min(s0 + kGridItemEvents, J.start[bin + 1]);
            const int bx = bin % J.nb[2], by = bin / J.nb[2] % J.nb[1],
                      bt = bin / (J.nb[2] * J.nb[1]);
            __syncthreads();  // the region of the item before is no longer read
            {
                // Node v = (t, y, x) of the region, v in steps of the CTA's threads.  A
                // region may reach past the grid's last nodes: what is read there is not
                // used, and the workspace goes on that far (grid_slack).
                constexpr int kDx = kGatherThreads % kR, kDy = kGatherThreads / kR % kR,
                              kDt = kGatherThreads / (kR * kR);
                int x = threadIdx.x % kR, yy = threadIdx.x / kR % kR, t = threadIdx.x / (kR * kR);
                const double* base = J.gb + ((size_t)(bt * kBin) * n1 + by * kBin) * n2 + bx * kBin;
                int from = (t * n1 + yy) * n2 + x, to = t * kPP + yy * kR + x;
                const int step = (kDt * n1 + kDy) * n2 + kDx;
                constexpr int kStep = kDt * kPP + kDy * kR + kDx;
                while (t < kR) {
                    copy8_async(sF + to, base + from, true);
                    x += kDx;
                    yy += kDy;
                    t += kDt;
                    from += step;
                    to += kStep;
                    if (x >= kR) {
                        x -= kR;
                        ++yy;
                        from += n2 - kR;
                    }
                    if (yy >= kR) {
                        yy -= kR;
                        ++t;
                        from += (n1 - kR) * n2;
                        to += kPP - kR * kR;
                    }
                }
            }
            // weights of one of the warp's events, two 16-byte pieces a lane
            const auto fetch = [&](int stage, int s) {
                if (s < s1) {
                    constexpr int kPieces = kGatherWeights<P> / 2;
#pragma unroll
                    for (int i = 0; i < (kPieces + 31) / 32; ++i) {
                        const int v = 2 * (lane + 32 * i);
                        if (v < 2 * kPieces)
                            copy16_async(sW + stage * kGatherWeights<P> + v,
                                         v < kGatherRow ? J.wv + (size_t)s * kGatherRow + v
                                                        : J.wd + (size_t)s * 3 * P + v - kGatherRow,
                                         true);
                    }
                }
                copy_commit();
            };
            fetch(0, s0 + warp);
            copy_wait<0>();
            __syncthreads();
            int stage = 0;
            for (int s = s0 + warp; s < s1; s += kGatherWarps, stage ^= 1) {
                fetch(stage ^ 1, s + kGatherWarps);
                const int c = J.cell[s], e = J.event[s];
                const int ct = c & 255, cy = c >> 8 & 255, cx = c >> 16;
                copy_wait<1>();
                __syncwarp();
                const double* w = sW + stage * kGatherWeights<P>;  // t, y, x rows
                const double* d = w + kGatherRow;
                double wx[P], dx[P];
#pragma unroll
                for (int i = 0; i < P; i += 2) {
                    wx[i] = w[2 * kGridSpan + cx + i];
                    wx[i + 1] = w[2 * kGridSpan + cx + i + 1];
                    const double2 v = *reinterpret_cast<const double2*>(d + 2 * P + i);
                    dx[i] = v.x;
                    dx[i + 1] = v.y;
                }
                double f = 0.0, lap = 0.0, ftt = 0.0;
                if (busy) {
                    const double* F = sF + (ct + kPlanes * h) * kPP + (cy + y) * kR + cx;
                    double a = 0.0, tt = 0.0, xx = 0.0;
#pragma unroll
                    for (int t = 0; t < kPlanes; t += 2) {
                        const double wt0 = w[ct + kPlanes * h + t], wt1 = w[ct + kPlanes * h + t + 1];
                        const double2 dt = *reinterpret_cast<const double2*>(d + kPlanes * h + t);
                        double p0 = 0.0, q0 = 0.0, p1 = 0.0, q1 = 0.0;
#pragma unroll
                        for (int i = 0; i < P; ++i) {
                            const double g0 = F[t * kPP + i], g1 = F[(t + 1) * kPP + i];
                            p0 = fma(g0, wx[i], p0);
                            q0 = fma(g0, dx[i], q0);
                            p1 = fma(g1, wx[i], p1);
                            q1 = fma(g1, dx[i], q1);
                        }
                        a = fma(wt0, p0, fma(wt1, p1, a));
                        xx = fma(wt0, q0, fma(wt1, q1, xx));
                        tt = fma(dt.x, p0, fma(dt.y, p1, tt));
                    }
                    const double wy = w[kGridSpan + cy + y], dy = d[P + y];
                    f = wy * a;
                    lap = J.D == 2 ? fma(wy, xx, dy * a) : wy * xx;
                    ftt = wy * tt;
                }
                __syncwarp();  // the stage's weights are no longer read
                // warp totals of f, lap and ftt on lanes 0, 8 and 16: the halves of the
                // warp, then its quarters, each keep one part
                const bool upper = lane & 16, second = lane & 8;
                const double u0 = (upper ? ftt : f) + __shfl_xor_sync(0xffffffffu, upper ? f : ftt, 16);
                const double u1 = (upper ? 0.0 : lap) +
                                  __shfl_xor_sync(0xffffffffu, upper ? lap : 0.0, 16);
                double v = (second ? u1 : u0) + __shfl_xor_sync(0xffffffffu, second ? u0 : u1, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                const double sum = __shfl_sync(0xffffffffu, v, 0);
                constexpr double kInv2 = (double)GridOrder<P>::kInv * GridOrder<P>::kInv;
                const int q = lane >> 3;
                const double weighted = 0.25 * (q == 1 ? J.unitX2 : J.unitT2) *
                                        fma(kInv2, v, (q == 1 ? 2.0 * J.D : 2.0) * sum);
                if ((lane & 7) == 0 && q < 3) J.sums[(size_t)q * J.N + e] = q == 0 ? sum : weighted;
            }
        }
        item -= nItems;
    }
}

// ---- host -------------------------------------------------------------------------

// Convolution table: G_l = (delta / 2 pi) int K(k) / (delta s(k)^2) e^{i k l delta} dk
// over one period of the grid's frequencies, K(k) = sqrt(pi) e^{-k^2/4} the
// Gaussian's transform and s(k) = sinc(k delta / 2)^P the spline's.  The
// integrand falls below 1e-50 at the ends of the period, so the midpoint rule
// is exact to rounding.
template <int P>
const GridTaps<P>& conv_taps() {
    constexpr int kInv = GridOrder<P>::kInv;
    static GridTaps<P> taps;
    static std::once_flag once;
    std::call_once(once, [] {
        const long double pi = 3.14159265358979323846264338327950288L;
        const long double delta = 1.0L / kInv;
        const int n = 160;  // the table repeats after 2 n lags: far beyond the Gaussian
        const long double dk = pi * kInv / n;
        // the weights' factors 1 / (P - 1)! are rounded doubles: divide their
        // relative errors out
        const long double off = (long double)(1.0 / kFactorial<P - 1>) * kFactorial<P - 1>;
        for (int l = 0; l <= GridOrder<P>::kTaps; ++l) {
            long double sum = 0.0L;
            for (int m = 0; m < n; ++m) {
                const long double k = (m + 0.5L) * dk;
                const long double x = 0.5L * k * delta;
                const long double s = powl(sinl(x) / x, P);
                sum += expl(-0.25L * k * k) / (s * s) * cosl(k * l * delta);
            }
            taps.g[l] = (double)(sum * dk * sqrtl(pi) / (pi * off * off));
        }
    });
    return taps;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

GridShape grid_shape(int order, double a, double b, const double* lo, const double* hi, double maxNodes) {
    GridShape s;
    s.order = order;
    const int inv = order == 16 ? GridOrder<16>::kInv : GridOrder<12>::kInv;
    const long double unit = inv / sqrtl(2.0L);  // grid units per scaled coordinate
    double nodes = 1.0;
    for (int d = 0; d < 3; ++d) {
        const double p = std::fabs(d == 0 ? b : a);
        if (!(p > 0.0) || !std::isfinite(p)) return s;
        const long double scale = unit * p;
        s.scaleHi[d] = (double)scale;
        s.scaleLo[d] = (double)(scale - s.scaleHi[d]);
        const double g0 = std::floor(lo[d] * s.scaleHi[d]) - 1.0;
        const double g1 = std::floor(hi[d] * s.scaleHi[d]) + 1.0;
        if (!(std::fabs(g0) < 1e9 && std::fabs(g1) < 1e9)) return s;
        s.origin[d] = g0;
        s.nc[d] = (int)(g1 - g0) + 1;
        s.n[d] = s.nc[d] + order - 1;
        s.nb[d] = (s.nc[d] + kBin - 1) / kBin;
        nodes *= s.n[d];
        if (nodes > maxNodes) return s;
    }
    s.nodes = (size_t)s.n[0] * s.n[1] * s.n[2];
    s.bins = (size_t)s.nb[0] * s.nb[1] * s.nb[2];
    s.ok = true;
    return s;
}

// Doubles past the last grid node that a bin's region may reach to.
static size_t grid_slack(const GridShape& s) {
    return ((size_t)kBin * s.n[1] + kBin) * s.n[2] + kBin;
}

// Gather items of a job, at most: a partly filled one per bin that holds events.
static size_t grid_items(const GridShape& s, int N) {
    return std::min(s.bins, (size_t)N) + (size_t)N / kGridItemEvents + 1;
}

size_t grid_workspace(const GridShape& s, int N) {
    const size_t n = (size_t)N;
    return align256((s.bins + 1) * sizeof(int)) + align256(grid_items(s, N) * sizeof(int2)) +
           align256(sizeof(int)) + 4 * align256(n * sizeof(int)) + align256(n * sizeof(unsigned)) +
           align256(n * 3 * kGridSpan * sizeof(double)) +
           align256(n * 3 * s.order * sizeof(double)) + align256(s.nodes * sizeof(double)) +
           align256((s.nodes + grid_slack(s)) * sizeof(double));
}

void grid_job(const GridShape& s, double a, double b, int N, int D, void* workspace, GridJob* J) {
    char* p = static_cast<char*>(workspace);
    const size_t n = (size_t)N;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += align256(bytes);
        return q;
    };
    J->start = reinterpret_cast<int*>(take((s.bins + 1) * sizeof(int)));
    J->items = reinterpret_cast<int2*>(take(grid_items(s, N) * sizeof(int2)));
    J->nItems = reinterpret_cast<int*>(take(sizeof(int)));
    J->binOf = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->pos = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->event = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->key = reinterpret_cast<unsigned*>(take(n * sizeof(unsigned)));
    J->cell = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->wv = reinterpret_cast<double*>(take(n * 3 * kGridSpan * sizeof(double)));
    J->wd = reinterpret_cast<double*>(take(n * 3 * s.order * sizeof(double)));
    J->ga = reinterpret_cast<double*>(take(s.nodes * sizeof(double)));
    J->gb = reinterpret_cast<double*>(take((s.nodes + grid_slack(s)) * sizeof(double)));
    for (int d = 0; d < 3; ++d) {
        J->scaleHi[d] = s.scaleHi[d];
        J->scaleLo[d] = s.scaleLo[d];
        J->origin[d] = s.origin[d];
        J->nc[d] = s.nc[d];
        J->nb[d] = s.nb[d];
        J->n[d] = s.n[d];
    }
    J->unitX2 = 2.0 / (a * a);
    J->unitT2 = 2.0 / (b * b);
    J->N = N;
    J->D = D;
}

template <int P>
static cudaError_t launch_sums(const GridJob* jobs, int nJobs, int numSMs, cudaStream_t s,
                               int* launches) {
    if (nJobs < 1 || nJobs > kGridMaxJobs) return cudaErrorInvalidValue;
    const GridTaps<P>& taps = conv_taps<P>();
    Batch b{};
    b.n = nJobs;
    // blocks of each kernel, job after job
    Blocks perBin{}, perEvent{}, perSlots{}, tiles{}, rows{}, yLines{}, tLines{};
    size_t items = 0;
    const auto up = [](int a, int q) { return (unsigned)((a + q - 1) / q); };
    cudaError_t e;
    for (int k = 0; k < nJobs; ++k) {
        const GridJob& J = jobs[k];
        b.job[k] = J;
        const auto add = [&](Blocks& x, unsigned n) { x.first[k + 1] = x.first[k] + n; };
        const int bins = J.nb[0] * J.nb[1] * J.nb[2];
        add(perBin, up(bins, kCellThreads));
        add(perEvent, up(J.N, kCellThreads));
        add(perSlots, up(J.N, kWeightSlots));
        add(tiles, up(J.n[2], kTileX) * up(J.n[1], kTileY) * up(J.n[0], kTileT));
        add(rows, up(J.n[0] * J.n[1], kRowLines) * up(J.n[2], kRowOut));
        add(yLines, up(J.n[0] * J.n[2], kLineThreads) * up(J.n[1], kConvOut));
        add(tLines, up(J.n[1] * J.n[2], kLineThreads) * up(J.n[0], kConvOut));
        items += (size_t)std::min(bins, J.N) + J.N / kGridItemEvents + 1;
    }
    constexpr size_t kRowShared = (size_t)kRowLines * kRowPitch<P> * sizeof(double);
    {
        // once per device
        constexpr int kMaxDevices = 64;
        static std::mutex mutex;
        static bool done[kMaxDevices] = {};
        int device = 0;
        if ((e = cudaGetDevice(&device))) return e;
        std::lock_guard<std::mutex> lock(mutex);
        if (device >= kMaxDevices || !done[device]) {
            if ((e = cudaFuncSetAttribute(conv_row_kernel<P>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kRowShared)) ||
                (e = cudaFuncSetAttribute(gather_kernel<P>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kGatherShared<P>)))
                return e;
            if (device < kMaxDevices) done[device] = true;
        }
    }
    // persistent gather CTAs, two per SM, fewer where there are not as many items
    const unsigned gatherCtas = (unsigned)std::min<size_t>(items, 2 * (size_t)numSMs);
    zero_kernel<<<perBin.first[nJobs], kCellThreads, 0, s>>>(b, perBin);
    count_kernel<<<perEvent.first[nJobs], kCellThreads, 0, s>>>(b, perEvent);
    scan_kernel<<<nJobs, kScanThreads, 0, s>>>(b);
    place_kernel<<<perEvent.first[nJobs], kCellThreads, 0, s>>>(b, perEvent);
    weights_kernel<P><<<perSlots.first[nJobs], kWeightThreads, 0, s>>>(b, perSlots);
    spread_kernel<P><<<tiles.first[nJobs], kSpreadThreads, 0, s>>>(b, tiles);
    conv_row_kernel<P><<<rows.first[nJobs], 32 * kRowWarps, kRowShared, s>>>(b, rows, taps);
    conv_line_kernel<P><<<yLines.first[nJobs], kLineThreads, 0, s>>>(b, yLines, taps, 1);
    conv_line_kernel<P><<<tLines.first[nJobs], kLineThreads, 0, s>>>(b, tLines, taps, 0);
    gather_kernel<P><<<gatherCtas, kGatherThreads, kGatherShared<P>, s>>>(b);
    *launches += 10;
    return cudaGetLastError();
}

cudaError_t launch_grid_sums(int order, const GridJob* jobs, int nJobs, int numSMs,
                             cudaStream_t s, int* launches) {
    return order == 16 ? launch_sums<16>(jobs, nJobs, numSMs, s, launches)
                       : launch_sums<12>(jobs, nJobs, numSMs, s, launches);
}

}  // namespace hphc
