// Work-list executor: evaluates any number of problems (an event set at a
// parameter vector) with one launch per stage.
//
//   stage   what                                          launch
//   H2D     problem tables, work items, finish tables    from pinned staging: copy_tables_kernel,
//                                                         above 64 KB one cudaMemcpyAsync
//   pack    FP32 records scaled per problem (FP32 mode;   pack_f32_jobs_kernel, grid (N, jobs)
//           one copy per distinct set, tauX, tauT)
//   grid    background sums of gridded problems           launch_grid_sums (not in the graph)
//   sweep   persistent CTAs over the work list            sweep_*_list_kernel
//   finish  per-event contributions, per-CTA sums, and    finish_list_kernel
//           per-problem totals to pinned host memory
//
// The sequence of each kind of plan is captured into a CUDA graph (a step on kept sums
// when its layout comes a second time) and replayed while buffer capacities, the
// sweep shape and the tables' layout stay the same; only the staged tables change
// between runs.  Work items cover each strip's band of tiles that can hold a
// non-zero term (found on the host from per-tile time bounds with the same
// test the kernel applies), split into equal chunks and listed largest first.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <iterator>
#include <string>
#include <vector>

#include "hphc_grid.h"
#include "hphc_kernels.cuh"

namespace hphc {

// Whether a strip row order holds the present events', and whether sweeps use it.
struct RowOrder {
    bool ready = false, wanted = false;
};

// An event set resident on the device, with host copies used for planning.
struct SetView {
    int N = 0;
    uint64_t version = 0;              // of the device's events: another after any change
    const double* dLoc = nullptr;      // N x D raw coordinates
    const double* dTimes = nullptr;    // N raw times
    const int32_t* dRanks = nullptr;   // dense time ranks (FP32 mode)
    const int32_t* dOrder2 = nullptr;  // spatial row order of strips of R = 2 and 4 (FP32
    const int32_t* dOrder4 = nullptr;  //   mode, launch_strip_order), or null
    RowOrder* order2 = nullptr;        // their state
    RowOrder* order4 = nullptr;
    const double* dRecF64 = nullptr;   // FP64 records (FP64 mode; large FP32-compensated sets)
    bool* packedF64 = nullptr;         // FP32-compensated: whether they hold the present events
    const double* dTileMin = nullptr;  // per-tile time bounds
    const double* dTileMax = nullptr;
    const double* hLoc = nullptr;      // host copies; hLoc may be missing (shards)
    const double* hTimes = nullptr;
    const double* hTileMin = nullptr;
    const double* hTileMax = nullptr;
    bool sorted = false;               // times ascending (bands are contiguous)
    // Where events share their times (dates, say): the time that most of them lie after
    // the last earlier one; else 0.
    double tiedGap = 0.0;
    bool haveBox = false;              // bounds of the coordinates
    double locMin[kMaxDim] = {}, locMax[kMaxDim] = {};
};

struct RunStats {
    int launches = 0;        // kernels launched by the last run
    double bTerms = 0.0;     // background pair terms the sweep accounted for
    double sTerms = 0.0;     // self-excitation pair terms the sweep evaluated
    double bEvals = 0.0;     // background exponentials evaluated (a symmetric pair: one)
};

class Executor {
public:
    // precision: HPHC_PRECISION_*; variant: FP32 variant bits (see
    // hphc_kernels.cu); ex2Bias: mean relative error of the hardware
    // exponential (divided out of the sums when the variant uses it).
    int init(int D, int precision, int variant, bool underflowSkip, int device, cudaStream_t stream,
             double ex2Bias);
    void release();

    // Plan and enqueue P problems (problem p = set setOf[p] at params[6p..6p+5])
    // without waiting.  dProbs: device buffer receiving P_i of problem 0, or null.
    int enqueue(const std::vector<SetView>& sets, const int* setOf, const double* params, int P,
                double* dProbs);
    // Wait for the last enqueue and copy its P x 8 results (log-likelihood,
    // gradient, 0) to hostOut.
    int wait(double* hostOut);

    // Device-resident loop (the on-device sampler): build the plan for P
    // problems once, with bands wide enough for any sigma, omega, theta and
    // mu0 at the problems' own tauX and tauT (all earlier tiles of sorted
    // times; the kernel still skips tile pairs whose terms all underflow),
    // upload its tables and pack the FP32 records.  enqueue_device_body()
    // then runs sweep, finish and final on those device tables, whose
    // per-problem constants a device kernel may rewrite between runs; the
    // P x 8 results are at device_results().  A later enqueue() replaces the
    // tables.
    int setup_device_loop(const std::vector<SetView>& sets, const int* setOf,
                          const double* params, int P);
    int enqueue_device_body();
    SweepProblem* device_sweep_problems() const;
    FinishProblem* device_finish_problems() const;
    const double* device_results() const { return dOut_; }
    int num_sms() const { return numSMs_; }

    // Pair terms the last run's sweep accounted for (replays the tile
    // decisions): background terms (both orders of a symmetric pair),
    // self-excitation terms, and background exponentials evaluated.
    void count_terms(const std::vector<SetView>& sets, double* bTerms, double* sTerms,
                     double* bEvals = nullptr) const;

    std::string error;
    int fixedR = 0, fixedItems = 0;  // sweep shape overrides; 0 = autotune
    int R = 2, itemsPerSM = 16;      // shape in use
    bool useGraph = true;
    bool kernelTiming = false;
    bool symmetric = false;  // symmetric background sweep (set before the first enqueue)
    bool fastTail = true;    // FP32 polynomial mode: far-tail tile pairs use ex2.approx
    bool truncateTail = true;  // skip background tile pairs below 2^-91 of B_ii (with the skip)
    // Background sums on a grid (hphc_grid.h) for the problems where that is
    // estimated to be faster than the pair sweep; the sweep then evaluates only
    // their self-excitation terms.  Set for the modes whose background terms
    // need no particular pair arithmetic; a fixed sweep shape or a shard asks
    // for the pair sweep.
    bool gridSums = false;
    bool selfWindow = false;  // self-excitation window (kSelfMisses), checked by the finish
    // Sharded sweep: with shardWorld > 1 the plan keeps only the target
    // strips assigned to shardRank (whole strips, balanced by their tile
    // counts; every rank computes the same assignment), and the finish takes
    // the other strips' row sums as zero.  The unit sums written to sumsOut
    // are then this rank's share; the shares of all ranks add up to the sums
    // of the unsharded sweep.
    int shardRank = 0, shardWorld = 1;
    // Fault injection (HPHC_FAULT_LAUNCH / HPHC_FAULT_WAIT): the next
    // faultCount launches or waits fail with a stand-in error.
    int faultStage = 0, faultCount = 0;
    bool take_fault(int stage) {
        if (faultStage != stage || faultCount <= 0) return false;
        if (--faultCount == 0) faultStage = 0;
        return true;
    }
    double* sumsOut = nullptr;  // if set, problem 0's unit pair sums ([6][N], natural units)
    // If set: a self-excitation-only sweep.  keptB holds the background unit
    // sums ([3][N], natural units) of an earlier sweep of the same single
    // event set at the same tauX and tauT as every problem of this run (the
    // caller checks that); the finish uses them and the sweep evaluates no
    // background term.  Rows 0-2 of sumsOut are then not written.
    const double* keptB = nullptr;
    float lastSweepMs = 0.f, lastFinishMs = 0.f, lastStepMs = 0.f;
    bool timedValid = false;
    int lastLaunches = 0;

private:
    int planPrecision_ = 0;  // of the current plan's sweep
    int D_ = 0, precision_ = 0, variant_ = 0, device_ = 0, numSMs_ = 148;
    bool skip_ = true;
    bool wideBands_ = false;  // build_plan: bands for any sampled parameters
    int loopGrid_ = 0;        // sweep grid of the device loop
    bool selfOnly_ = false;   // the current plan's sweep is self-excitation-only
    int sweep_variant() const {
        return variant_ | (!selfOnly_ ? 0 : kSelfOnly | (planPrecision_ != precision_ ? kShortExp : 0));
    }
    double ex2Bias_ = 0.0;
    std::string deviceName_;  // for the persistent tune cache
    cudaStream_t stream_ = nullptr;
    // shapes in use: sweeps with background terms, self-excitation-only sweeps, and
    // those in FP64 of an FP32-compensated engine
    struct Shape {
        bool tuned = false;
        int R = 0, items = 0;
    } shape_[3];

    // plan of the last enqueue
    struct Plan {
        std::vector<SweepProblem> sp;
        std::vector<WorkItem> items;
        std::vector<int> stripChunks;   // concatenated over problems
        std::vector<FinishProblem> fp;
        std::vector<FinishBlock> fb;
        std::vector<PackJob> pj;
        std::vector<int> setOf;
        int P = 0, maxN = 0, nBlocks = 0;
    } plan_;

    // device / pinned buffers (capacities grow; a growth invalidates the graph)
    void* dTables_ = nullptr;
    size_t tablesCap_ = 0;
    void* hStaging_ = nullptr;
    size_t stagingCap_ = 0;
    float* dRecPool_ = nullptr;
    size_t recCap_ = 0;
    double* dPartials_ = nullptr;
    size_t partialsCap_ = 0;
    unsigned long long* dColAcc_ = nullptr;
    size_t colCap_ = 0;
    double* dBlockSums_ = nullptr;
    size_t blockCap_ = 0;
    double* dOut_ = nullptr;
    double* hOut_ = nullptr;
    size_t outCap_ = 0;
    int* dCounter_ = nullptr;
    int* dArrived_ = nullptr;  // finish CTAs arrived: all problems, then each problem
    size_t arrivedCap_ = 0;
    bool stale_ = false;  // counters and column sums may not be at zero
    cudaEvent_t ev_[6] = {};  // step start, sweep start and end, step end; grid start and end

    // gridded background sums: which problems of the plan take them, their
    // grids, the [3][N] sums of those whose sums are not kept, and a workspace
    std::vector<char> gridOf_;
    std::vector<GridShape> gridShape_;
    std::vector<size_t> gridSumsOff_;
    double* dGridSums_ = nullptr;
    size_t gridSumsCap_ = 0;
    void* dGridWork_ = nullptr;
    size_t gridWorkCap_ = 0;
    int gridLaunches_ = 0;

    // table layout inside dTables_ / hStaging_ (byte offsets)
    size_t offSP_ = 0, offItems_ = 0, offNItems_ = 0, offChunks_ = 0, offFP_ = 0, offFB_ = 0,
           offPJ_ = 0, tablesBytes_ = 0;
    size_t itemsCap_ = 0;
    size_t recNeed_ = 0, partialsNeed_ = 0;  // floats / doubles the last plan needs
    size_t colNeed_ = 0;                     // column-sum words the last plan needs

    // graph
    // one graph per kind of plan (shape_'s kinds), so that a sampler that mixes
    // full evaluations and self-excitation steps captures each once
    // (and, the second three, once more for runs whose records are packed)
    cudaGraphExec_t graphExec_[6] = {};
    struct GraphKey {  // all that the captured launches take from the host
        int P = -1, nJobs = -1, nBlocks = -1, maxN = -1, R = -1, grid = -1;
        size_t tablesBytes = 0;
        size_t offsets[7] = {};  // of the tables in the staged block
        void* tables = nullptr;
        int variant = 0;
        bool timing = false;
        bool operator==(const GraphKey& o) const {
            return P == o.P && nJobs == o.nJobs && nBlocks == o.nBlocks && maxN == o.maxN &&
                   R == o.R && grid == o.grid && tablesBytes == o.tablesBytes &&
                   std::equal(std::begin(offsets), std::end(offsets), std::begin(o.offsets)) &&
                   tables == o.tables && variant == o.variant && timing == o.timing;
        }
    } graphKey_[6];
    bool met_[6] = {};  // the key's layout has run without a graph
    // What the record pool holds: one set's FP32 records at one scaling.  A plan that
    // needs just those launches no pack: the sampler's sigma and omega steps, which
    // leave events, tauX and tauT alone.
    struct Packed {
        uint64_t version = 0;  // 0: none
        const double* loc = nullptr;
        double sX = 0.0, sT = 0.0;
    } packed_, willPack_;
    bool skipPack_ = false;  // of the current plan
    int kind_ = 0;  // of the current plan

    ConstsSpec consts_spec() const;
    int build_plan(const std::vector<SetView>& sets, const int* setOf, const double* params, int P,
                   double* dProbs, int r, int items);
    int ensure_buffers();
    void plan_grid(const std::vector<SetView>& sets, const int* setOf, const double* params,
                   int P);
    // how densely a set's events lie on a problem's grid (plan_grid)
    struct Crowd {
        double tile = 0.0, bin = 0.0;  // share of the events that touch a tile, lie in a bin
    };
    static constexpr int kCrowdSample = 32;
    struct CrowdSample {
        float at[3][kCrowdSample];  // t, x, y of events spread over the set
    };
    CrowdSample crowd_sample(const SetView& s) const;
    Crowd crowd(const CrowdSample& c, int order, double a, double b) const;
    double* grid_sums(int p) const;
    bool release_grid();
    int plan(const std::vector<SetView>& sets, const int* setOf, const double* params, int P,
             double* dProbs);
    double self_terms(const SetView& s, const double* p) const;
    bool self_only(int P) const;  // no problem of the plan has background terms to sweep
    bool self_listless(const std::vector<SetView>& sets, const int* setOf, int P) const;
    int choose_shape(const std::vector<SetView>& sets, const int* setOf, const double* params,
                     int P, double* dProbs);
    int launch_grid(const std::vector<SetView>& sets, const int* setOf, const double* params,
                    int P);
    int launch_sequence(int grid);
    int sweep_grid(int r) const;
    int autotune(const std::vector<SetView>& sets, const int* setOf, const double* params, int P,
                 double* dProbs);
    int cuda_fail(cudaError_t e, const char* what);
    void drop_graph(int kind);
    void drop_graphs() {
        for (int k = 0; k < 6; ++k) drop_graph(k);
    }
    cudaError_t record(cudaEvent_t ev);
    bool capturing_ = false;

public:
    ConstsSpec consts_spec(const SetView& set, double omega) const;
    PairConsts pair_consts(const double* p, const SetView& set) const;
    FinishConsts finish_consts(const double* p, const SetView& set) const;
};

}  // namespace hphc
