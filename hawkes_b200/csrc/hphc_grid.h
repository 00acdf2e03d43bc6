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
// Accuracy: a pair's term differs from the exact one by at most 2.5e-17, its
// squared-distance weighted terms by at most 1.2e-15 (root mean square 4e-16),
// in units of an event's own term B_ii = 1 (the splines' aliasing, evaluated in
// extended precision over random pairs; the error alternates in sign with the
// position against the grid).  Everything is FP64, and every sum but the
// derivative weights is over positive numbers, so rounding adds no more than it
// does in the pair sweep.
//
// Work: O(N kP^3) for spread and gather and O(nodes kTaps) for the convolution,
// against O(N^2) pair terms.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace hphc {

constexpr int kGridP = 16;    // spline order = nodes per event and coordinate
constexpr int kGridInv = 8;   // nodes per unit of u
constexpr int kGridTaps = 48; // |lag| of the convolution table (6 units of u)
constexpr int kGridBin = 8;   // cells per bin and coordinate
constexpr int kGridMaxJobs = 16;  // jobs of one launch (kernel parameters)

// One problem: an event set at one (tauX, tauT).  Coordinates are ordered
// (t, y, x); for D = 1 every y is 0.
struct GridJob {
    const double* loc;    // N x D
    const double* times;  // N
    double* sums;         // [3][N] unit background sums out (weights 1, d^2, dt^2)
    // workspace
    int* start;           // [bins + 1] counts, then exclusive prefix sums
    int* binOf;           // [N] bin of event e, times kGridBin, plus its t cell in the bin
    int* pos;             // [N] arrival position of event e in its bin
    unsigned* key;        // [N] by slot: t cell in the bin << 28 | event, in arrival order
    int* event;           // [N] by slot: event, ordered by key within each bin
    int4* cell;           // [N] by slot: cells (t, y, x)
    double* wv;           // [N][3][kGridP] by slot: spline weights
    double* wd;           // [N][3][kGridP] by slot: their second derivatives
    double* ga;           // [nodes] grids
    double* gb;
    double scaleHi[3], scaleLo[3];  // grid units per coordinate unit, double-double
    double origin[3];     // cell 0 in grid units (an integer)
    double unitX2, unitT2;  // coordinate units^2 per u^2: 2 / a^2, 2 / b^2
    int nc[3];            // cells
    int nb[3];            // bins
    int n[3];             // nodes (cells + kGridP - 1)
    int N, D;
};

// Convolution table G[|lag|].
struct GridTaps {
    double g[kGridTaps + 1];
};

struct GridShape {
    bool ok = false;
    double scaleHi[3], scaleLo[3], origin[3];
    int nc[3], nb[3], n[3];
    size_t nodes = 0, bins = 0;
};

// Grid of an event set with coordinates in [lo, hi] (order t, y, x) at
// precisions a (space) and b (time); ok = false if it would hold more than
// maxNodes nodes or the scales are unusable.
GridShape grid_shape(double a, double b, const double* lo, const double* hi, double maxNodes);

// Workspace bytes of one job.
size_t grid_workspace(const GridShape& s, int N);
// Fill a job's geometry and workspace pointers (workspace 256-byte aligned).
void grid_job(const GridShape& s, double a, double b, int N, int D, void* workspace, GridJob* job);

// Sums of up to kGridMaxJobs jobs; *launches += kernels launched.
cudaError_t launch_grid_sums(const GridJob* jobs, int nJobs, cudaStream_t s, int* launches);

}  // namespace hphc
