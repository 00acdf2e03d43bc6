// Background sums by a gridded fast Gaussian transform (D <= 2).
//
// The background kernel of the model is a Gaussian in all D + 1 coordinates,
//   B_ij = exp(-|u_i - u_j|^2),  u = (b t, a x, a y) / sqrt(2),
// so the three background sums of every event (weights 1, d^2, dt^2) need
// not be formed pair by pair: they are a convolution of the events with a
// Gaussian, evaluated at the events.  On a regular grid of kInv nodes per
// unit of u:
//
//   spread   W[z]  = sum_j M(z - u_j)           M: product of B-splines of order kP
//   convolve F     = G * W                      one pass per coordinate
//   gather   f(u_i) = sum_z M(u_i - z) F[z]     and its second derivatives
//
// with G the Gaussian divided by the two splines in Fourier space (a table of
// 2 kTaps + 1 numbers, the same for every problem: the parameters only scale
// u).  Since d^2/du_k^2 exp(-u^2) = (4 u_k^2 - 2) exp(-u^2), the weighted sums
// come from the derivatives of the gathered spline:
//   sum_j B_ij u_k^2 = (f_kk + 2 f) / 4.
//
// Two orders are built, with kInv and kTaps chosen for each (largest error of a
// pair's term, and of its squared-distance weighted terms, in units of an event's
// own term B_ii = 1: the splines' aliasing, evaluated in extended precision over
// random pairs; it alternates in sign with the position against the grid):
//
//   kP   kInv  kTaps  term     weighted terms (root mean square)
//   16   8     48     2.5e-17  1.2e-15 (4e-16)   FP64 accuracy
//   12   6     32     1e-12    1.4e-10 (4e-11)   far below FP32 rounding of the
//                                                coordinates (5e-8)
//
// Everything is FP64, and every sum but the derivative weights is over positive
// numbers, so rounding adds no more than it does in the pair sweep.
//
// Work: O(N kP^3) for spread and gather and O(nodes kTaps) for the convolution,
// against O(N^2) pair terms.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace hphc {

// Spline order -> nodes per unit of u, |lag| of the convolution table.
template <int P>
struct GridOrder;
template <>
struct GridOrder<16> {
    static constexpr int kInv = 8, kTaps = 48;
};
template <>
struct GridOrder<12> {
    static constexpr int kInv = 6, kTaps = 32;
};

// From this size on the FP32-compensated mode takes order 16 with FP64 self-excitation
// sums (Executor::plan) in place of order 12 with its own, which makes an evaluation as
// exact as the FP64 mode's for 14 to 17 % of its time: N = 66k 448 -> 524 us, N = 100k 627
// -> 715, errors of the log-likelihood 4.3e-11 -> below 1e-16 and of the worst gradient
// component 2.2e-9 -> 5e-16.  Neither cost nor error has an edge there: the line is a
// choice.  Batches of proposals, where the cost shows most, lie below it, and above it
// a step in sigma or omega, which keeps the background and stays FP32-compensated (165
// us at N = 100k), stays below a quarter of a full evaluation, as samplers expect.  A
// step and a full evaluation of the same parameters differ by the mode's error (4e-11
// of the log-likelihood).
constexpr int kGridHighOrderEvents = 1 << 16;

constexpr int kGridBin = 8;   // cells per bin and coordinate
constexpr int kGridSpan = 24;  // nodes of a bin's events, rounded up to whole bins
constexpr int kGridItemEvents = 128;
constexpr int kGridMaxJobs = 16;  // jobs of one launch (kernel parameters)

// One problem: an event set at one (tauX, tauT).  Coordinates are ordered
// (t, y, x); for D = 1 every y is 0.
struct GridJob {
    const double* loc;    // N x D
    const double* times;  // N
    double* sums;         // [3][N] unit background sums out (weights 1, d^2, dt^2)
    // workspace
    int* start;           // [bins + 1] counts, then exclusive prefix sums
    int2* items;          // gather work: bin and first slot, at most kGridItemEvents slots each
    int* nItems;
    int* binOf;           // [N] bin of event e, times kGridBin, plus its t cell in the bin
    int* pos;             // [N] arrival position of event e in its bin
    unsigned* key;        // [N] by slot: t cell in the bin << 28 | event, in arrival order
    int* event;           // [N] by slot: event, ordered by key within each bin
    int* cell;            // [N] by slot: cells in the bin, t | y << 8 | x << 16
    double* wv;           // [N][3][kGridSpan] by slot: spline weights on the nodes from the
                          // bin's first on (zeros around the kP of the event)
    double* wd;           // [N][3][kP] by slot: their second derivatives
    double* ga;           // [nodes] grids
    double* gb;
    double scaleHi[3], scaleLo[3];  // grid units per coordinate unit, double-double
    double origin[3];     // cell 0 in grid units (an integer)
    double unitX2, unitT2;  // coordinate units^2 per u^2: 2 / a^2, 2 / b^2
    int nc[3];            // cells
    int nb[3];            // bins
    int n[3];             // nodes (cells + kP - 1)
    int N, D;
};

struct GridShape {
    bool ok = false;
    int order = 0;
    double scaleHi[3], scaleLo[3], origin[3];
    int nc[3], nb[3], n[3];
    size_t nodes = 0, bins = 0;
};

// Grid of spline order `order` (12 or 16) for an event set with coordinates in
// [lo, hi] (order t, y, x) at precisions a (space) and b (time); ok = false if it
// would hold more than maxNodes nodes or the scales are unusable.
GridShape grid_shape(int order, double a, double b, const double* lo, const double* hi,
                     double maxNodes);

// Workspace bytes of one job.
size_t grid_workspace(const GridShape& s, int N);
// Fill a job's geometry and workspace pointers (workspace 256-byte aligned).
void grid_job(const GridShape& s, double a, double b, int N, int D, void* workspace, GridJob* job);

// Sums of up to kGridMaxJobs jobs of one order; *launches += kernels launched.
cudaError_t launch_grid_sums(int order, const GridJob* jobs, int nJobs, int numSMs,
                             cudaStream_t s, int* launches);

}  // namespace hphc
