// Kernels of the gridded background sums (see hphc_grid.h).
#include "hphc_grid.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace hphc {
namespace {

constexpr int P = kGridP;
constexpr int kBin = kGridBin;
constexpr int kRegion = kBin + P - 1;  // nodes a bin's events touch, per coordinate

struct Batch {
    GridJob job[kGridMaxJobs];
};

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

__global__ void __launch_bounds__(kCellThreads) zero_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.y];
    const int i = blockIdx.x * kCellThreads + threadIdx.x;
    if (i < J.nb[0] * J.nb[1] * J.nb[2]) J.start[i] = 0;
}

__global__ void __launch_bounds__(kCellThreads) count_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.y];
    const int e = blockIdx.x * kCellThreads + threadIdx.x;
    if (e >= J.N) return;
    int c[3];
    double f;
    for (int d = 0; d < 3; ++d) grid_position(J, e, d, &c[d], &f);
    const int bin = ((c[0] / kBin) * J.nb[1] + c[1] / kBin) * J.nb[2] + c[2] / kBin;
    J.binOf[e] = bin * kBin + (c[0] & (kBin - 1));
    J.pos[e] = atomicAdd(J.start + bin, 1);
}

// Exclusive prefix sums of the bin counts, one CTA per job.
constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.x];
    const int nb = J.nb[0] * J.nb[1] * J.nb[2];
    __shared__ int warpSum[kScanThreads / 32];
    __shared__ int carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int i0 = 0; i0 < nb; i0 += kScanThreads) {
        const int i = i0 + tid;
        const int v = i < nb ? J.start[i] : 0;
        int x = v;
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) warpSum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int w = warpSum[lane];
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += y;
            }
            warpSum[lane] = w;
        }
        __syncthreads();
        const int base = carry + (warp ? warpSum[warp - 1] : 0);
        if (i < nb) J.start[i] = base + x - v;
        __syncthreads();
        if (tid == kScanThreads - 1) carry = base + x;
        __syncthreads();
    }
    if (tid == 0) J.start[nb] = carry;
}

__global__ void __launch_bounds__(kCellThreads) place_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.y];
    const int e = blockIdx.x * kCellThreads + threadIdx.x;
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
__device__ __forceinline__ void spline_weights(double f, double* __restrict__ wv,
                                               double* __restrict__ wd) {
    constexpr double kInvP1 = 1.0 / 1307674368000.0;  // 1 / 15!
    constexpr double kInvP3 = 1.0 / 6227020800.0;     // 1 / 13!
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
    double d[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const double a = i < P - 2 ? v[i] : 0.0;
        const double m = i >= 1 && i - 1 < P - 2 ? v[i - 1] : 0.0;
        const double z = i >= 2 ? v[i - 2] : 0.0;
        d[i] = ((a - m) + (z - m)) * kInvP3;
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
    for (int i = 0; i < P; i += 2) {
        reinterpret_cast<double2*>(wv)[i / 2] =
            make_double2(v[P - 1 - i] * kInvP1, v[P - 2 - i] * kInvP1);
        reinterpret_cast<double2*>(wd)[i / 2] = make_double2(d[P - 1 - i], d[P - 2 - i]);
    }
}

// Three threads a slot, one per coordinate; the slot's first thread ranks it.
constexpr int kWeightSlots = 64;
constexpr int kWeightThreads = 3 * kWeightSlots;

__global__ void __launch_bounds__(kWeightThreads)
weights_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.y];
    __shared__ int sDst[kWeightSlots], sCell[3][kWeightSlots];
    const int d = threadIdx.x / kWeightSlots, i = threadIdx.x % kWeightSlots;
    const int slot = blockIdx.x * kWeightSlots + i;
    if (blockIdx.x * kWeightSlots >= J.N) return;
    const bool live = slot < J.N;
    const unsigned k = live ? J.key[slot] : 0;
    const int e = (int)(k & 0x0fffffffu);
    double f = 0.0;
    if (live) grid_position(J, e, d, &sCell[d][i], &f);
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
    if (!live) return;
    const size_t dst = sDst[i];
    if (d == 0) J.cell[dst] = make_int4(sCell[0][i], sCell[1][i], sCell[2][i], 0);
    spline_weights(f, J.wv + (dst * 3 + d) * P, J.wd + (dst * 3 + d) * P);
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
// weights that fall into the tile copied to shared memory one group ahead, and
// their tiles are added in warp order.  Events are sorted by t cell inside their
// bin, so rows that none of the four touches are left out.

constexpr int kSpreadThreads = 256;
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

// The slots of a tile's events: runs of consecutive slots (bins along x) in
// groups of four.
struct Runs {
    int first[9], last[9];  // slots
    int group[10];          // groups before the run
    int n;
};

__global__ void __launch_bounds__(kSpreadThreads, 2)
spread_kernel(const __grid_constant__ Batch b) {
    const GridJob& J = b.job[blockIdx.y];
    const int ntx = (J.n[2] + kTileX - 1) / kTileX, nty = (J.n[1] + kTileY - 1) / kTileY,
              ntt = (J.n[0] + kTileT - 1) / kTileT;
    if (blockIdx.x >= (unsigned)(ntx * nty * ntt)) return;
    const int tx = blockIdx.x % ntx, ty = (blockIdx.x / ntx) % nty, tt = blockIdx.x / (ntx * nty);
    const int t0 = tt * kTileT, y0 = ty * kTileY, x0 = tx * kTileX;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = lane & 3, row = lane >> 2;

    __shared__ Runs runs;
    __shared__ __align__(16) double sSlice[kSpreadWarps][2][4][kSlicePitch];
    if (threadIdx.x == 0) {
        // an event of cell c touches nodes c .. c + 15: bins -2 .. 0 of the tile's own
        const int bx0 = max(2 * tx - 2, 0), bx1 = min(2 * tx + 1, J.nb[2] - 1);
        int n = 0, groups = 0;
        for (int bt = max(tt - 2, 0); bt <= min(tt, J.nb[0] - 1); ++bt)
            for (int by = max(ty - 2, 0); by <= min(ty, J.nb[1] - 1); ++by) {
                const int line = (bt * J.nb[1] + by) * J.nb[2];
                const int s0 = J.start[line + bx0], s1 = J.start[line + bx1 + 1];
                if (s0 >= s1) continue;
                runs.first[n] = s0;
                runs.last[n] = s1;
                runs.group[n++] = groups;
                groups += (s1 - s0 + 3) / 4;
            }
        runs.group[n] = groups;
        runs.n = n;
    }
    __syncthreads();
    const int groups = runs.group[runs.n];

    double acc[2][kTileT][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < kTileT; ++r) acc[h][r][0] = acc[h][r][1] = 0.0;

    // event k of group q: its slot (-1: none) and its cell against the tile
    int run = 0;
    const auto fetch = [&](int q, int& slot, int& ct, int& cy, int& cx) {
        slot = -1;
        ct = cy = cx = 0;
        if (q >= groups) return;
        while (q >= runs.group[run + 1]) ++run;
        const int s = runs.first[run] + 4 * (q - runs.group[run]) + k;
        if (s >= runs.last[run]) return;
        const int4 c = J.cell[s];
        slot = s;
        ct = c.x - t0;
        cy = c.y - y0;
        cx = c.z - x0;
    };
    const int part = lane < kTileT ? 0 : lane < kTileT + kTileY ? 1 : 2;
    const int node = lane - (part == 0 ? 0 : part == 1 ? kTileT : kTileT + kTileY);
    const auto copy = [&](int stage, int slot, int ct, int cy, int cx) {
#pragma unroll
        for (int ev = 0; ev < 4; ++ev) {
            const int s = __shfl_sync(0xffffffffu, slot, ev);
            const int a = __shfl_sync(0xffffffffu, ct, ev), c = __shfl_sync(0xffffffffu, cy, ev),
                      d = __shfl_sync(0xffffffffu, cx, ev);
            const int i = node - (part == 0 ? a : part == 1 ? c : d);
            const bool live = s >= 0 && (unsigned)i < (unsigned)P;
            copy8_async(&sSlice[warp][stage][ev][lane],
                        J.wv + (live ? ((size_t)s * 3 + part) * P + i : 0), live);
        }
        copy_commit();
    };

    int slot, ct, cy, cx, slot1, ct1, cy1, cx1;
    fetch(warp, slot, ct, cy, cx);
    copy(0, slot, ct, cy, cx);
    fetch(warp + kSpreadWarps, slot1, ct1, cy1, cx1);
    int stage = 0;
    for (int q = warp; q < groups; q += kSpreadWarps, stage ^= 1) {
        copy(stage ^ 1, slot1, ct1, cy1, cx1);  // the next group's weights
        int slot2, ct2, cy2, cx2;
        fetch(q + 2 * kSpreadWarps, slot2, ct2, cy2, cx2);  // and the cells after it
        const bool live = slot >= 0;
        const int lo = __reduce_min_sync(0xffffffffu, live ? max(0, ct) : kTileT);
        const int hi = __reduce_max_sync(0xffffffffu, live ? min(kTileT - 1, P - 1 + ct) : -1);
        const bool h0 = __any_sync(0xffffffffu, live && cx > -P && cx < 8);
        const bool h1 = __any_sync(0xffffffffu, live && cx > 8 - P && cx < 16);
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
        slot = slot1, ct = ct1, cy = cy1, cx = cx1;
        slot1 = slot2, ct1 = ct2, cy1 = cy2, cx1 = cx2;
    }
    copy_wait<0>();

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
// in shared memory, one per lane, at an odd pitch (no bank conflicts).

constexpr int kConvOut = 16;
constexpr int kTapPad = kGridTaps + kConvOut;  // table index of lag 0
static_assert(kGridTaps % kConvOut == 0, "whole blocks of taps");

__device__ __forceinline__ void stage_taps(const GridTaps& taps, double* sTap) {
    for (int v = threadIdx.x; v < 2 * kTapPad; v += blockDim.x) {
        const int lag = abs(v - kTapPad);
        sTap[v] = lag <= kGridTaps ? taps.g[lag] : 0.0;
    }
}

// 16 outputs o0 .. o0 + 15 from input(j), j in [o0 - kGridTaps, o0 + kGridTaps + 16).
template <class Input>
__device__ __forceinline__ void convolve(const double* __restrict__ sTap, int o0, Input input,
                                         double (&out)[kConvOut]) {
#pragma unroll
    for (int i = 0; i < kConvOut; ++i) out[i] = 0.0;
#pragma unroll 1
    for (int jb = -kGridTaps; jb <= kGridTaps; jb += kConvOut) {
        double in[kConvOut];
#pragma unroll
        for (int j = 0; j < kConvOut; ++j) in[j] = input(o0 + jb + j);
        const double* t = sTap + kTapPad + jb;
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
__global__ void __launch_bounds__(kLineThreads)
conv_line_kernel(const __grid_constant__ Batch b, const __grid_constant__ GridTaps taps,
                 int axis) {
    const GridJob& J = b.job[blockIdx.y];
    const int len = J.n[axis];
    const int stride = axis == 1 ? J.n[2] : J.n[1] * J.n[2];
    const int lines = axis == 1 ? J.n[0] * J.n[2] : stride;
    const int chunks = (len + kConvOut - 1) / kConvOut;
    const int blocks = (lines + kLineThreads - 1) / kLineThreads;
    if (blockIdx.x >= (unsigned)(blocks * chunks)) return;
    __shared__ double sTap[2 * kTapPad];
    stage_taps(taps, sTap);
    __syncthreads();
    const int chunk = blockIdx.x % chunks;
    const int line = blockIdx.x / chunks * kLineThreads + threadIdx.x;
    if (line >= lines) return;
    const double* src = axis == 1 ? J.gb : J.ga;
    double* dst = axis == 1 ? J.ga : J.gb;
    const size_t base = (size_t)(line / stride) * len * stride + line % stride;
    const int o0 = chunk * kConvOut;
    double out[kConvOut];
    convolve(sTap, o0, [&](int j) {
        return (unsigned)j < (unsigned)len ? src[base + (size_t)j * stride] : 0.0;
    }, out);
#pragma unroll
    for (int i = 0; i < kConvOut; ++i)
        if (o0 + i < len) dst[base + (size_t)(o0 + i) * stride] = out[i];
}

constexpr int kRowLines = 32;                       // lines of a CTA
constexpr int kRowWarps = 8;
constexpr int kRowOut = kRowWarps * kConvOut;       // outputs of a line in a CTA
constexpr int kRowPitch = kRowOut + 2 * kGridTaps + 1;  // odd

__global__ void __launch_bounds__(32 * kRowWarps)
conv_row_kernel(const __grid_constant__ Batch b, const __grid_constant__ GridTaps taps) {
    extern __shared__ double sRow[];  // [kRowLines][kRowPitch]
    __shared__ double sTap[2 * kTapPad];
    const GridJob& J = b.job[blockIdx.y];
    const int len = J.n[2], lines = J.n[0] * J.n[1];
    const int chunks = (len + kRowOut - 1) / kRowOut;
    const int blocks = (lines + kRowLines - 1) / kRowLines;
    if (blockIdx.x >= (unsigned)(blocks * chunks)) return;
    const int o0 = blockIdx.x % chunks * kRowOut, l0 = blockIdx.x / chunks * kRowLines;
    const int outs = min(kRowOut, len - o0), rows = min(kRowLines, lines - l0);
    stage_taps(taps, sTap);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < kRowLines; r += kRowWarps)
        for (int j = lane; j < kRowPitch; j += 32) {
            const int x = o0 - kGridTaps + j;
            sRow[r * kRowPitch + j] =
                r < rows && (unsigned)x < (unsigned)len ? J.ga[(size_t)(l0 + r) * len + x] : 0.0;
        }
    __syncthreads();
    double out[kConvOut];
    const double* line = sRow + lane * kRowPitch;
    const int w0 = warp * kConvOut;
    if (w0 < outs) convolve(sTap, w0, [&](int j) { return line[j + kGridTaps]; }, out);
    __syncthreads();
    if (w0 < outs)
#pragma unroll
        for (int i = 0; i < kConvOut; ++i) sRow[lane * kRowPitch + w0 + i] = out[i];
    __syncthreads();
    for (int r = warp; r < rows; r += kRowWarps)
        for (int j = lane; j < outs; j += 32)
            J.gb[(size_t)(l0 + r) * len + o0 + j] = sRow[r * kRowPitch + j];
}

// ---- gather ---------------------------------------------------------------------
//
// A CTA stages the 23^3 nodes its bin's events touch in shared memory and its
// warps take the events in turn: lane (h, y) forms the x products of node rows y
// of 8 of the 16 t planes, for the spline and for its second derivative, and the
// other two coordinates follow on the lane's own sums.  The pitch of 23 doubles
// puts the 16 rows of a half warp on distinct banks.  Bound: shared memory, 4096
// doubles an event at 16 a clock.

constexpr int kGatherThreads = 256;
constexpr int kGatherWarps = kGatherThreads / 32;
constexpr int kGatherSlices = 4;  // CTAs of a bin that share its events when it is crowded
constexpr int kSliceEvents = 128;

constexpr size_t kGatherShared =
    (kRegion * kRegion * kRegion + 1 + kGatherWarps * 6 * P) * sizeof(double);

__global__ void __launch_bounds__(kGatherThreads, 2)
gather_kernel(const __grid_constant__ Batch b) {
    extern __shared__ __align__(16) double sF[];
    const GridJob& J = b.job[blockIdx.y];
    const int bin = blockIdx.x;
    if (bin >= J.nb[0] * J.nb[1] * J.nb[2]) return;
    int s0 = J.start[bin], s1 = J.start[bin + 1];
    const int chunk = max(kSliceEvents, (s1 - s0 + kGatherSlices - 1) / kGatherSlices);
    s0 += blockIdx.z * chunk;
    s1 = min(s1, s0 + chunk);
    if (s0 >= s1) return;
    const int bx = bin % J.nb[2], by = bin / J.nb[2] % J.nb[1], bt = bin / (J.nb[2] * J.nb[1]);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int v = threadIdx.x; v < kRegion * kRegion * kRegion; v += kGatherThreads) {
        const int t = bt * kBin + v / (kRegion * kRegion), y = by * kBin + v / kRegion % kRegion,
                  x = bx * kBin + v % kRegion;
        const bool live = t < J.n[0] && y < J.n[1] && x < J.n[2];
        copy8_async(sF + v, J.gb + (live ? ((size_t)t * J.n[1] + y) * J.n[2] + x : 0), live);
    }
    copy_commit();
    double* sW = sF + kRegion * kRegion * kRegion + 1 + warp * 6 * P;
    const int y = lane & 15, h = lane >> 4;
    // weights of the warp's next event, three numbers a lane
    double w0 = 0.0, w1 = 0.0, w2 = 0.0;
    const auto fetch = [&](int s) {
        if (s >= s1) return;
        const double* v = J.wv + (size_t)s * 3 * P;
        const double* d = J.wd + (size_t)s * 3 * P;
        w0 = v[lane];
        w1 = lane < P ? v[32 + lane] : d[lane - P];
        w2 = d[P + lane];
    };
    fetch(s0 + warp);
    copy_wait<0>();
    __syncthreads();
    for (int s = s0 + warp; s < s1; s += kGatherWarps) {
        const int4 c = J.cell[s];
        const int e = J.event[s];
        __syncwarp();
        sW[lane] = w0;
        sW[32 + lane] = w1;
        sW[64 + lane] = w2;
        __syncwarp();
        fetch(s + kGatherWarps);
        double wx[P], dx[P];
#pragma unroll
        for (int i = 0; i < P; i += 2) {
            const double2 u = *reinterpret_cast<const double2*>(sW + 2 * P + i);
            const double2 v = *reinterpret_cast<const double2*>(sW + 5 * P + i);
            wx[i] = u.x;
            wx[i + 1] = u.y;
            dx[i] = v.x;
            dx[i + 1] = v.y;
        }
        const double* F = sF + (((c.x & (kBin - 1)) + 8 * h) * kRegion + (c.y & (kBin - 1)) + y) *
                                   kRegion + (c.z & (kBin - 1));
        double a = 0.0, tt = 0.0, xx = 0.0;
#pragma unroll 2
        for (int t = 0; t < 8; ++t) {
            double p = 0.0, q = 0.0;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const double f = F[t * kRegion * kRegion + i];
                p = fma(f, wx[i], p);
                q = fma(f, dx[i], q);
            }
            const double wt = sW[8 * h + t], dt = sW[3 * P + 8 * h + t];
            a = fma(wt, p, a);
            xx = fma(wt, q, xx);
            tt = fma(dt, p, tt);
        }
        const double wy = sW[P + y], dy = sW[4 * P + y];
        double f = wy * a;
        double lap = J.D == 2 ? fma(wy, xx, dy * a) : wy * xx;
        double ftt = wy * tt;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            f += __shfl_xor_sync(0xffffffffu, f, d);
            lap += __shfl_xor_sync(0xffffffffu, lap, d);
            ftt += __shfl_xor_sync(0xffffffffu, ftt, d);
        }
        if (lane == 0) {
            constexpr double kInv2 = (double)kGridInv * kGridInv;
            J.sums[e] = f;
            J.sums[(size_t)J.N + e] = 0.25 * J.unitX2 * fma(kInv2, lap, 2.0 * J.D * f);
            J.sums[(size_t)2 * J.N + e] = 0.25 * J.unitT2 * fma(kInv2, ftt, 2.0 * f);
        }
    }
}

// ---- host -------------------------------------------------------------------------

// Convolution table: G_l = (delta / 2 pi) int K(k) / (delta s(k)^2) e^{i k l delta} dk
// over one period of the grid's frequencies, K(k) = sqrt(pi) e^{-k^2/4} the
// Gaussian's transform and s(k) = sinc(k delta / 2)^P the spline's.  The
// integrand falls below 1e-50 at the ends of the period, so the midpoint rule
// is exact to rounding.
const GridTaps& conv_taps() {
    static GridTaps taps;
    static std::once_flag once;
    std::call_once(once, [] {
        const long double pi = 3.14159265358979323846264338327950288L;
        const long double delta = 1.0L / kGridInv;
        const int n = 160;  // the table repeats after 2 n lags: far beyond the Gaussian
        const long double dk = pi * kGridInv / n;
        // the weights' factors 1 / (P - 1)! are rounded doubles: divide their
        // relative errors out
        const long double fact = 1307674368000.0L;
        const long double off = (long double)(1.0 / 1307674368000.0) * fact;
        for (int l = 0; l <= kGridTaps; ++l) {
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

GridShape grid_shape(double a, double b, const double* lo, const double* hi, double maxNodes) {
    GridShape s;
    const long double unit = kGridInv / sqrtl(2.0L);  // grid units per scaled coordinate
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
        s.n[d] = s.nc[d] + P - 1;
        s.nb[d] = (s.nc[d] + kBin - 1) / kBin;
        nodes *= s.n[d];
        if (nodes > maxNodes) return s;
    }
    s.nodes = (size_t)s.n[0] * s.n[1] * s.n[2];
    s.bins = (size_t)s.nb[0] * s.nb[1] * s.nb[2];
    s.ok = true;
    return s;
}

size_t grid_workspace(const GridShape& s, int N) {
    const size_t n = (size_t)N;
    return align256((s.bins + 1) * sizeof(int)) + 3 * align256(n * sizeof(int)) +
           align256(n * sizeof(unsigned)) + align256(n * sizeof(int4)) +
           2 * align256(n * 3 * P * sizeof(double)) + 2 * align256(s.nodes * sizeof(double));
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
    J->binOf = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->pos = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->event = reinterpret_cast<int*>(take(n * sizeof(int)));
    J->key = reinterpret_cast<unsigned*>(take(n * sizeof(unsigned)));
    J->cell = reinterpret_cast<int4*>(take(n * sizeof(int4)));
    J->wv = reinterpret_cast<double*>(take(n * 3 * P * sizeof(double)));
    J->wd = reinterpret_cast<double*>(take(n * 3 * P * sizeof(double)));
    J->ga = reinterpret_cast<double*>(take(s.nodes * sizeof(double)));
    J->gb = reinterpret_cast<double*>(take(s.nodes * sizeof(double)));
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

cudaError_t launch_grid_sums(const GridJob* jobs, int nJobs, cudaStream_t s, int* launches) {
    if (nJobs < 1 || nJobs > kGridMaxJobs) return cudaErrorInvalidValue;
    const GridTaps& taps = conv_taps();
    Batch b{};
    int maxN = 0;
    unsigned bins = 0, tiles = 0, rows = 0, yl = 0, tl = 0;
    cudaError_t e;
    for (int k = 0; k < nJobs; ++k) {
        const GridJob& J = jobs[k];
        b.job[k] = J;
        const unsigned nb = J.nb[0] * J.nb[1] * J.nb[2];
        maxN = std::max(maxN, J.N);
        bins = std::max(bins, nb);
        const auto up = [](int a, int q) { return (unsigned)((a + q - 1) / q); };
        tiles = std::max(tiles, up(J.n[2], kTileX) * up(J.n[1], kTileY) * up(J.n[0], kTileT));
        rows = std::max(rows, up(J.n[0] * J.n[1], kRowLines) * up(J.n[2], kRowOut));
        yl = std::max(yl, up(J.n[0] * J.n[2], kLineThreads) * up(J.n[1], kConvOut));
        tl = std::max(tl, up(J.n[1] * J.n[2], kLineThreads) * up(J.n[0], kConvOut));
    }
    constexpr size_t kRowShared = (size_t)kRowLines * kRowPitch * sizeof(double);
    {
        // once per device
        constexpr int kMaxDevices = 64;
        static std::mutex mutex;
        static bool done[kMaxDevices] = {};
        int device = 0;
        if ((e = cudaGetDevice(&device))) return e;
        std::lock_guard<std::mutex> lock(mutex);
        if (device >= kMaxDevices || !done[device]) {
            if ((e = cudaFuncSetAttribute(conv_row_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kRowShared)) ||
                (e = cudaFuncSetAttribute(gather_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kGatherShared)))
                return e;
            if (device < kMaxDevices) done[device] = true;
        }
    }
    const unsigned nj = (unsigned)nJobs;
    const dim3 perEvent((maxN + kCellThreads - 1) / kCellThreads, nj);
    zero_kernel<<<dim3((bins + kCellThreads - 1) / kCellThreads, nj), kCellThreads, 0, s>>>(b);
    count_kernel<<<perEvent, kCellThreads, 0, s>>>(b);
    scan_kernel<<<nj, kScanThreads, 0, s>>>(b);
    place_kernel<<<perEvent, kCellThreads, 0, s>>>(b);
    weights_kernel<<<dim3((maxN + kWeightSlots - 1) / kWeightSlots, nj), kWeightThreads, 0,
                     s>>>(b);
    spread_kernel<<<dim3(tiles, nj), kSpreadThreads, 0, s>>>(b);
    conv_row_kernel<<<dim3(rows, nj), 32 * kRowWarps, kRowShared, s>>>(b, taps);
    conv_line_kernel<<<dim3(yl, nj), kLineThreads, 0, s>>>(b, taps, 1);
    conv_line_kernel<<<dim3(tl, nj), kLineThreads, 0, s>>>(b, taps, 0);
    gather_kernel<<<dim3(bins, nj, kGatherSlices), kGatherThreads, kGatherShared, s>>>(b);
    *launches += 10;
    return cudaGetLastError();
}

}  // namespace hphc
