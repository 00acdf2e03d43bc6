// Work-list executor (see hphc_executor.h).
#include "hphc_executor.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "hphc.h"

namespace hphc {
namespace {

constexpr double kInvSqrt2Pi = 0.398942280401432677939946059934;
constexpr double kLog2e = 1.44269504088896340735992468100189214;


size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

double record_scale(double precisionParam) {
    return std::fabs(precisionParam) * std::sqrt(0.5 * kLog2e);
}

// Host replica of the kernel's tile-pair decision (hphc_kernels.cu, tile_mode).
void tile_needs(double tminI, double tmaxI, double tminJ, double tmaxJ, const PairConsts& c,
                bool* doB, bool* doS) {
    const double dtLo = tminI - tmaxJ, dtHi = tmaxI - tminJ;
    const double minAbs = dtLo > 0.0 ? dtLo : (dtHi < 0.0 ? -dtHi : 0.0);
    *doB = !c.noB && !(c.skipB >= 0.0 && -c.cB * minAbs * minAbs >= c.skipB);
    const bool allCausal = dtLo > 0.0;
    *doS = (dtHi > 0.0) && !(c.skipS >= 0.0 && allCausal && -c.cW * dtLo >= c.skipS);
}

// The first tile at or after `from` (and before `end`) whose latest time is
// above v / whose earliest time is at least v, starting from an earlier answer
// `at`: strips come in time order, so over a plan each edge moves through the
// tiles once.
int first_max_above(const SetView& s, double v, int end, int at) {
    while (at < end && s.hTileMax[at] <= v) ++at;
    return std::min(at, end);
}
int first_min_from(const SetView& s, double v, int from, int end, int at) {
    at = std::max(at, from);
    while (at < end && s.hTileMin[at] < v) ++at;
    return at;
}

// Time gaps beyond which every background or self-excitation term is left out
// (+inf: none is, -inf: there are none) and from which background terms take the
// far tail's exponential.
struct StripGaps {
    double b, s, far;
    explicit StripGaps(const PairConsts& c) {
        const double kInf = INFINITY;
        const bool falls = c.cB < 0.0 && c.cA <= 0.0;
        b = c.noB ? -kInf : c.skipB >= 0.0 && falls ? std::sqrt(c.skipB / -c.cB) : kInf;
        s = c.skipS >= 0.0 && c.cW < 0.0 && c.cS <= 0.0 ? c.skipS / -c.cW : kInf;
        far = c.fastB > 0.0 && falls ? std::sqrt(c.fastB / -c.cB) : kInf;
    }
};

// Where the edges of the previous strip lay.
struct StripCursor {
    int lo = 0, hi = 0, nearLo = 0, nearHi = 0, selfLo = 0;
};

// Band [*lo, *hi) of j tiles that strip st (r tiles of targets) must visit:
// every tile that may hold a non-zero term for constants c, plus one tile of
// margin each side; wide: for any sigma and omega (the device-resident
// loop).  For sorted times the tile bounds are non-decreasing, and a tile
// before the strip can hold a background term only if its time gap is below
// dB = sqrt(skipB / -cB), a self-excitation term only below
// dS = skipS / -cW (tile_mode's underflow tests solved for the gap), so each
// edge is a search on the bounds, which moves on from the previous strip's
// answer: host planning of an N = 100k
// self-excitation step 90 -> 35 us.  The band may keep a few tiles
// those tests would drop (tile_mode also tests causality and the space
// coefficient); the sweep decides every tile itself, and chunks sit on a
// fixed grid, so a wider band never changes a bit of the result.
void strip_band(const SetView& s, const StripGaps& gap, bool symmetric, bool wide, int r,
                int nTiles, int st, StripCursor& at, int* loOut, int* hiOut) {
    const int ts0 = st * r, ts1 = std::min(ts0 + r, nTiles);
    *loOut = 0;
    *hiOut = nTiles;
    if (!s.sorted) return;
    const double tminI = s.hTileMin[ts0], tmaxI = s.hTileMax[ts1 - 1];
    const double kInf = INFINITY, dB = gap.b, dS = gap.s;
    // left edge: the first tile before the strip whose gap tminI - tmaxJ is
    // below the larger distance (wide: any sigma, omega, so every tile)
    int lo = 0;
    if (!wide) {
        const double d = std::max(dB, dS);
        if (d < kInf) {
            at.lo = first_max_above(s, tminI - d, ts0, at.lo);
            lo = std::max(0, at.lo - 1);
        }
    }
    // right edge: with the symmetric sweep, later tiles add this strip's
    // pairs as columns (and sorted times leave no self-excitation there);
    // otherwise the first tile after the strip whose gap tminJ - tmaxI is at
    // least dB (background only: no causal pair lies after the strip)
    int hi = ts1;
    if (!symmetric && ts1 < nTiles && dB > -kInf) {
        if (dB == kInf) {
            hi = nTiles;
        } else {
            at.hi = first_min_from(s, tmaxI + dB, ts1, nTiles, at.hi);
            hi = std::min(nTiles, at.hi + 1);
        }
    } else if (!symmetric && ts1 < nTiles) {
        hi = std::min(nTiles, ts1 + 1);
    }
    *loOut = lo;
    *hiOut = hi;
}

// Relative cost of the tiles of one work item, for ordering the work list
// (largest first) and dealing strips to ranks.  For sorted times a strip's
// tiles split by their time gap to the strip: below dF = sqrt(fastB / -cB)
// the background terms take the full exponential ("near"), beyond it the
// far tail's cheaper one; below dS the tile also holds self-excitation
// terms.  Weights from measured sweep times: a far-tail tile costs about
// half a near one in the FP32-compensated mode (whose near terms take the
// software exponential and three compensated sums) and 7/10 in the FP64
// mode; the self-excitation terms of a tile add about half a tile in the
// FP32 mode and a whole one in the FP64 mode (an exponential for each).
// Ordering by these costs instead of tile counts: sweep at N = 100k 2.588 ->
// 2.498 ms (FP32, plain block sums then) and 10.06 -> 9.69 ms (FP64); the
// FP32 far weight 0.75 -> 0.5 with the compensated sums: 2.676 -> 2.620 ms
// at 64 items/SM, 2.81 -> 2.64 ms at 32.
constexpr double kFarTileCostF32 = 0.5;
constexpr double kFarTileCostF64 = 0.70;
constexpr double kSelfTileCostF32 = 0.5;
constexpr double kSelfTileCostF64 = 1.0;

struct StripCost {
    int nearLo = 0, nearHi = 0;  // near background tiles
    int selfLo = 0, selfHi = 0;  // tiles with self-excitation terms
    double far = 1.0;            // weight of a background tile outside [nearLo, nearHi)
    double self = kSelfTileCostF32;  // added weight of a tile with self-excitation terms
};

StripCost strip_cost(const SetView& s, const StripGaps& gap, bool fp32, int r, int nTiles,
                     int st, StripCursor& at) {
    StripCost k;
    k.self = fp32 ? kSelfTileCostF32 : kSelfTileCostF64;
    const int ts0 = st * r, ts1 = std::min(ts0 + r, nTiles);
    k.nearLo = 0;
    k.nearHi = nTiles;
    k.selfLo = 0;
    k.selfHi = ts1;
    if (!s.sorted) return k;
    const double tminI = s.hTileMin[ts0], tmaxI = s.hTileMax[ts1 - 1];
    if (gap.far < INFINITY) {
        const double dF = gap.far;
        k.nearLo = at.nearLo = first_max_above(s, tminI - dF, ts0, at.nearLo);
        k.nearHi = at.nearHi = first_min_from(s, tmaxI + dF, ts1, nTiles, at.nearHi);
        k.far = fp32 ? kFarTileCostF32 : kFarTileCostF64;
    }
    if (gap.s < INFINITY) {
        const double dS = gap.s;
        k.selfLo = at.selfLo = first_max_above(s, tminI - dS, ts0, at.selfLo);
    }
    return k;
}

double item_cost(const StripCost& k, bool noB, int jt0, int jt1) {
    const auto overlap = [&](int a, int b) { return std::max(0, std::min(jt1, b) - std::max(jt0, a)); };
    const int near = overlap(k.nearLo, k.nearHi);
    const double b = noB ? 0.0 : near + k.far * (jt1 - jt0 - near);
    return b + k.self * overlap(k.selfLo, k.selfHi);
}

// Writes the items to out (the staged table) largest first, so that the
// persistent CTAs end on small items; equal costs keep their order.  Costs are
// sums of whole tiles times weights in tenths, so one counting pass over
// cost * 10 sorts them.
void stage_items(const std::vector<WorkItem>& items, const std::vector<double>& cost,
                 WorkItem* out) {
    const size_t n = items.size();
    int top = 0;
    std::vector<int> key(n);
    for (size_t k = 0; k < n; ++k) {
        key[k] = (int)(cost[k] * 10.0 + 0.5);
        top = std::max(top, key[k]);
    }
    std::vector<int> at(top + 2, 0);
    for (size_t k = 0; k < n; ++k) ++at[top - key[k] + 1];
    for (int v = 0; v <= top; ++v) at[v + 1] += at[v];
    for (size_t k = 0; k < n; ++k) out[at[top - key[k]]++] = items[k];
}

int f32_stride(int D) {
    return (2 * (D + 1) + 1 + 3) / 4 * 4;
}

// Autotuned sweep shapes per process: (D, precision, mode bits, log2 of the
// pair count, log2 of the problem count) -> (R, items per SM).
using TuneKey = std::tuple<int, int, int, int, int>;
std::mutex gTuneMutex;
std::map<TuneKey, std::pair<int, int>> gTuneCache;

// Persistent tune cache: HPHC_TUNE_CACHE names a file of JSON lines, one per
// tuned shape,
//   {"v":1,"device":"<name>","sms":148,"D":2,"precision":1,"mode":50,
//    "pairs_log2":34,"problems_log2":0,"R":4,"items":64}
// read once per process (lines of other devices, other versions or with an
// invalid shape are ignored) and appended to after each new tuning.  Each
// line is written with one append of under 200 bytes, so processes sharing
// the file do not interleave their lines.
constexpr int kTuneCacheVersion = 1;
constexpr int kTuneReps = 4;  // timed sweeps per candidate shape (even)

struct TuneLine {
    std::string device;
    int sms;
    TuneKey key;
    int R, items;
};
std::vector<TuneLine> gTuneFile;
bool gTuneFileRead = false;

// Position of the value of "key" in a one-line JSON object (after the
// colon and any blanks), or npos.
size_t json_value(const std::string& line, const char* key) {
    const std::string k = std::string("\"") + key + "\"";
    size_t at = line.find(k);
    if (at == std::string::npos) return at;
    at = line.find_first_not_of(" \t", at + k.size());
    if (at == std::string::npos || line[at] != ':') return std::string::npos;
    return line.find_first_not_of(" \t", at + 1);
}

bool json_int(const std::string& line, const char* key, int* out) {
    const size_t at = json_value(line, key);
    if (at == std::string::npos) return false;
    char* end = nullptr;
    const long v = std::strtol(line.c_str() + at, &end, 10);
    if (end == line.c_str() + at) return false;
    *out = (int)v;
    return true;
}

bool json_string(const std::string& line, const char* key, std::string* out) {
    const size_t at = json_value(line, key);
    if (at == std::string::npos || line[at] != '"') return false;
    const size_t end = line.find('"', at + 1);
    if (end == std::string::npos) return false;
    *out = line.substr(at + 1, end - at - 1);
    return true;
}

bool valid_shape(int precision, int R, int items) {
    const bool okR = precision == HPHC_PRECISION_FP64 ? (R == 1 || R == 2) : (R == 2 || R == 4);
    return okR && items >= 1 && items <= 1024;
}

// Called with gTuneMutex held.
void read_tune_file() {
    if (gTuneFileRead) return;
    gTuneFileRead = true;
    const char* path = std::getenv("HPHC_TUNE_CACHE");
    if (!path || !*path) return;
    FILE* f = std::fopen(path, "r");
    if (!f) return;
    char buf[512];
    while (std::fgets(buf, sizeof buf, f)) {
        const std::string line(buf);
        TuneLine t;
        int v = 0, D = 0, prec = 0, mode = 0, pb = 0, kb = 0;
        if (!json_int(line, "v", &v) || v != kTuneCacheVersion) continue;
        if (!json_string(line, "device", &t.device) || !json_int(line, "sms", &t.sms) ||
            !json_int(line, "D", &D) || !json_int(line, "precision", &prec) ||
            !json_int(line, "mode", &mode) || !json_int(line, "pairs_log2", &pb) ||
            !json_int(line, "problems_log2", &kb) || !json_int(line, "R", &t.R) ||
            !json_int(line, "items", &t.items))
            continue;
        if (!valid_shape(prec, t.R, t.items)) continue;
        t.key = std::make_tuple(D, prec, mode, pb, kb);
        gTuneFile.push_back(t);
    }
    std::fclose(f);
}

void append_tune_file(const std::string& device, int sms, const TuneKey& key, int R, int items) {
    const char* path = std::getenv("HPHC_TUNE_CACHE");
    if (!path || !*path) return;
    std::string name = device;
    for (char& ch : name)
        if (ch == '"' || ch == '\\' || (unsigned char)ch < 0x20) ch = '_';
    char line[400];
    const int n = std::snprintf(
        line, sizeof line,
        "{\"v\":%d,\"device\":\"%s\",\"sms\":%d,\"D\":%d,\"precision\":%d,\"mode\":%d,"
        "\"pairs_log2\":%d,\"problems_log2\":%d,\"R\":%d,\"items\":%d}\n",
        kTuneCacheVersion, name.c_str(), sms, std::get<0>(key), std::get<1>(key),
        std::get<2>(key), std::get<3>(key), std::get<4>(key), R, items);
    if (n <= 0 || n >= (int)sizeof line) return;
    FILE* f = std::fopen(path, "a");
    if (!f) return;
    std::fwrite(line, 1, (size_t)n, f);
    std::fclose(f);
}

// Tables up to this size go to the device by a kernel that reads the pinned host
// memory; larger ones by the copy engine.  Self-excitation step at N = 20k 61 -> 52 us,
// at N = 100k 166 -> 163; evaluation at N = 500 36.9 -> 35.8, N = 5000 84 -> 76 (FP64).
constexpr size_t kCopyKernelBytes = 64 << 10;

// Gridded background sums: cost estimates (plan_grid) and limits.  Microseconds
// from measured times (one B200): the background terms of the sweeps took, at
// N = 100k, 6.86 ms for 3.38e9 pairs in FP64 and 2.42 ms for 2.89e9 in FP32; the
// grid kernels of order 16 0.48 ms at N = 100k with 1.24e6 nodes; those of order 12
// 0.18 and 0.32 ms at N = 20k and 60k with 5.4e5 nodes, and 0.088 ms a problem
// with 16 problems of N = 20k in a launch, which share the launches' latency.
// Smaller FP32 sweeps cost more a pair, 1.1e-6 at N = 20k (64 problems of N = 20k:
// 6.33 ms with 0.9e-6 here, 6.09 with 1.1e-6, 6.34 with 1.3e-6; FP64 flat around its
// value).  A single problem's fixed cost in order 12 is 95 too; 140 keeps problems
// that take the same either way with the sweep.
constexpr double kPairCostF64 = 2.05e-6, kPairCostF32 = 1.1e-6;  // a pair
constexpr double kSelfCostF64 = 1.9e-6;  // a self-excitation term
constexpr double kLongSelfTerms = 3e8;   // FP64 sweeps of so many take strips twice as high
struct GridCost {
    double event, node, fixed;  // fixed: of a group of problems
    double spread;              // the spread kernel's part of `event`
};
constexpr GridCost kGridCost16{3.45e-3, 5.0e-5, 95.0, 1.9e-3},
    kGridCost12{3.2e-3, 5.0e-5, 140.0, 1.3e-3};
// Where the events crowd: an event of the fullest tile, a pair of events of one bin.  All
// events in one bin, as at a tenth of the usual precisions: N = 12k, 20k and 30k 0.80,
// 1.27 and 1.85 ms (0.75, 1.26 and 1.8 with these), 100k 10.7 (11); a fraction c = 0.16,
// 0.44 and 0.79 on a tile at N = 30k 0.44, 0.72 and 1.12 ms (0.39, 0.74, 1.2).  Without
// them N = 20k at a tenth of the precisions took 1.18 ms on the grid, 0.66 as pairs.
constexpr double kGridSerial = 0.03, kGridRank = 0.68e-6;
constexpr int kGridMinEvents = 1000;
constexpr double kGridMaxNodes = 4e8;
constexpr size_t kGridMaxWork = size_t(8) << 30;    // one problem's workspace
constexpr size_t kGridGroupWork = size_t(1) << 30;  // of problems that run together

int log2_bucket(double x) {
    int b = 0;
    while (x > 1.0 && b < 80) {
        x *= 0.5;
        ++b;
    }
    return b;
}

}  // namespace

int Executor::cuda_fail(cudaError_t e, const char* what) {
    stale_ = true;
    packed_ = Packed{};
    error = std::string(what) + ": " + cudaGetErrorString(e);
    cudaGetLastError();  // a failed allocation is not the next launch's error
    return e == cudaErrorMemoryAllocation ? HPHC_ERR_OUT_OF_MEMORY : HPHC_ERR_CUDA;
}

int Executor::init(int D, int precision, int variant, bool underflowSkip, int device,
                   cudaStream_t stream, double ex2Bias) {
    D_ = D;
    precision_ = planPrecision_ = precision;
    variant_ = variant;
    skip_ = underflowSkip;
    device_ = device;
    stream_ = stream;
    ex2Bias_ = ex2Bias;
    cudaDeviceGetAttribute(&numSMs_, cudaDevAttrMultiProcessorCount, device);
    R = precision == HPHC_PRECISION_FP64 ? 2 : 4;
    itemsPerSM = 32;
    cudaError_t e = cudaMalloc(&dCounter_, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, "device allocation");
    stale_ = true;
    for (auto& ev : ev_)
        if ((e = cudaEventCreate(&ev)) != cudaSuccess) return cuda_fail(e, "create events");
    return HPHC_OK;
}

void Executor::drop_graph(int kind) {
    if (graphExec_[kind]) cudaGraphExecDestroy(graphExec_[kind]);
    graphExec_[kind] = nullptr;
    graphKey_[kind] = GraphKey{};
    met_[kind] = false;
}

void Executor::release() {
    drop_graphs();
    if (dTables_) cudaFree(dTables_);
    if (hStaging_) cudaFreeHost(hStaging_);
    if (dRecPool_) cudaFree(dRecPool_);
    if (dPartials_) cudaFree(dPartials_);
    if (dColAcc_) cudaFree(dColAcc_);
    if (dBlockSums_) cudaFree(dBlockSums_);
    if (dOut_) cudaFree(dOut_);
    if (hOut_) cudaFreeHost(hOut_);
    if (dCounter_) cudaFree(dCounter_);
    if (dArrived_) cudaFree(dArrived_);
    dArrived_ = nullptr;
    arrivedCap_ = 0;
    release_grid();
    for (auto& ev : ev_)
        if (ev) cudaEventDestroy(ev);
    dTables_ = hStaging_ = nullptr;
    dRecPool_ = nullptr;
    dPartials_ = dBlockSums_ = dOut_ = hOut_ = nullptr;
    dColAcc_ = nullptr;
    dCounter_ = nullptr;
    tablesCap_ = stagingCap_ = recCap_ = partialsCap_ = blockCap_ = outCap_ = colCap_ = 0;
    for (auto& ev : ev_) ev = nullptr;
}

ConstsSpec Executor::consts_spec() const {
    ConstsSpec s{};
    s.precision = planPrecision_ == HPHC_PRECISION_FP64 ? 0 : 1;
    s.D = D_;
    s.variant = variant_;
    s.skip = skip_ ? 1 : 0;
    s.truncate = (skip_ && truncateTail) ? 1 : 0;
    s.ex2Bias = ex2Bias_;
    s.fastTail = fastTail ? 1 : 0;
    s.noB = keptB ? 1 : 0;
    return s;
}

// A bound on sum_k e^(-omega (dt_k - d)) over the events k at least d before any
// one time: at most M events lie in an interval of length 1 / omega (whole
// tiles), so the sum is at most M (1 + e^-1 + e^-2 + ...) = 1.59 M; 1.7 M
// also bounds the sum weighted by omega dt / (omega d) for omega d >= 20.
// omega 0: any omega.
double decayed_events(const SetView& set, double omega) {
    if (!set.sorted || !(omega > 0.0)) return set.N;
    const int nTiles = (set.N + kTile - 1) / kTile;
    int most = 1;
    for (int k = 0, j = 0; k < nTiles; ++k) {
        const double end = set.hTileMax[k] + 1.0 / omega;
        while (j < nTiles && set.hTileMin[j] <= end) ++j;
        most = std::max(most, j - k);
    }
    return std::min((double)set.N, 1.7 * kTile * most);
}

// With the event set's self-excitation window, where the sweep has one (omega
// 0: for any omega).
ConstsSpec Executor::consts_spec(const SetView& set, double omega) const {
    ConstsSpec s = consts_spec();
    if (!selfWindow || fixedR || fixedItems || shardWorld > 1 || !set.haveBox) return s;
    const int nTiles = (set.N + kTile - 1) / kTile;
    if (nTiles < 4) return s;  // a window leaves out whole tiles
    double volume = set.sorted ? set.hTileMax[nTiles - 1] - set.hTileMin[0]
                               : *std::max_element(set.hTileMax, set.hTileMax + nTiles) -
                                     *std::min_element(set.hTileMin, set.hTileMin + nTiles);
    s.selfTile = volume / nTiles;
    s.selfGap = set.tiedGap;
    double ball = 1.0;  // V_D = V_{D-2} 2 pi / D
    for (int d = D_; d > 1; d -= 2) ball *= 2.0 * M_PI / d;
    if (D_ % 2) ball *= 2.0;
    for (int k = 0; k < D_; ++k) volume *= set.locMax[k] - set.locMin[k];
    s.selfCount = decayed_events(set, omega);
    s.selfDensity = volume > 0.0 ? set.N / volume * ball / (0.5 * D_ + 1.0) : 1e300;
    return s;
}

PairConsts Executor::pair_consts(const double* p, const SetView& set) const {
    PairConsts c{};
    FinishConsts f{};
    param_consts(p, consts_spec(set, p[3]), c, f);
    return c;
}

FinishConsts Executor::finish_consts(const double* p, const SetView& set) const {
    PairConsts c{};
    FinishConsts f{};
    param_consts(p, consts_spec(set, p[3]), c, f);
    f.T = set.hTimes[set.N - 1];
    // src/NewHawkes.hpp:659: locationCount * (embeddingDimension - 1) * log(M_1_SQRT_2PI)
    f.constant = (double)(set.N * (D_ - 1)) * std::log(kInvSqrt2Pi);
    return f;
}

int Executor::sweep_grid(int r) const {
    const int perSM = sweep_list_blocks_per_sm(planPrecision_ == HPHC_PRECISION_FP64 ? 0 : 1, D_, r,
                                               sweep_variant());
    return numSMs_ * std::max(1, perSM);
}

bool Executor::self_only(int P) const {
    if (keptB) return true;
    if (gridOf_.empty()) return false;
    for (int p = 0; p < P; ++p)
        if (!gridOf_[p]) return false;
    return true;
}

// Whether a self-excitation-only plan needs no work list: sorted times, one size.
// A device loop over more than kLoopTiles tiles keeps its list: its bands may
// come to hold every earlier tile, and then largest first counts (16 chains
// at N = 10,000: 0.86 ms an iteration without, 0.64 with).
bool Executor::self_listless(const std::vector<SetView>& sets, const int* setOf, int P) const {
    constexpr int kLoopTiles = 32;
    const int N = sets[setOf[0]].N;
    if (shardWorld != 1 || (wideBands_ && N > kLoopTiles * kTile)) return false;
    for (int p = 0; p < P; ++p)
        if (!sets[setOf[p]].sorted || sets[setOf[p]].N != N) return false;
    return true;
}

// Problem p's gridded background sums: the kept sums' own rows for problem 0
// where they are kept.
double* Executor::grid_sums(int p) const {
    return p == 0 && sumsOut ? sumsOut : dGridSums_ + gridSumsOff_[p];
}

// One event of each of kCrowdSample equal parts of the set, the place in the part
// scattered so that sites taken in turn do not coincide with it.
Executor::CrowdSample Executor::crowd_sample(const SetView& s) const {
    CrowdSample c{};
    const int part = std::max(1, s.N / kCrowdSample);
    for (int k = 0; k < kCrowdSample; ++k) {
        const unsigned scatter = (unsigned)k * 2654435761u >> 8;
        const int i = std::min(s.N - 1, (int)((long long)s.N * k / kCrowdSample) +
                                            (int)(scatter % (unsigned)part));
        c.at[0][k] = (float)(s.hTimes[i] - s.hTileMin[0]);
        c.at[1][k] = (float)(s.hLoc[(size_t)i * D_] - s.locMin[0]);
        c.at[2][k] = D_ == 2 ? (float)(s.hLoc[(size_t)i * 2 + 1] - s.locMin[1]) : 0.0f;
    }
    return c;
}

// Shares of the events within 12 cells (those that touch a tile of nodes) and 4 cells
// (a bin) of an event in every coordinate, of the densest part: the second moment of
// the shares about sampled events over the first, each without bias from counting the
// event itself.
Executor::Crowd Executor::crowd(const CrowdSample& c, int order, double a, double b) const {
    const double unit = (order == 16 ? GridOrder<16>::kInv : GridOrder<12>::kInv) / std::sqrt(2.0);
    const float tt = (float)(12.0 / (unit * std::fabs(b))), tx = (float)(12.0 / (unit * std::fabs(a)));
    const float bt = tt / 3.0f, bx = tx / 3.0f;
    double first[2] = {0.0, 0.0}, second[2] = {0.0, 0.0};
    for (int i = 0; i < kCrowdSample; ++i) {
        const float t = c.at[0][i], x = c.at[1][i], y = c.at[2][i];
        int nt = -1, nb = -1;  // the event itself
        for (int j = 0; j < kCrowdSample; ++j) {
            const float dt = std::fabs(c.at[0][j] - t), dx = std::fabs(c.at[1][j] - x),
                        dy = std::fabs(c.at[2][j] - y);
            nt += (dt <= tt) & (dx <= tx) & (dy <= tx);
            nb += (dt <= bt) & (dx <= bx) & (dy <= bx);
        }
        first[0] += nt;
        first[1] += nb;
        second[0] += nt * (nt - 1.0);
        second[1] += nb * (nb - 1.0);
    }
    Crowd r;
    if (first[0] > 0.0) r.tile = second[0] / ((kCrowdSample - 2) * first[0]);
    if (first[1] > 0.0) r.bin = second[1] / ((kCrowdSample - 2) * first[1]);
    return r;
}

// Which problems take their background sums from a grid: those whose estimated
// time on it (fixed, shared by the problems of a launch, per event and per node)
// is below that of the pairs the sweep would evaluate, counted from sampled tiles
// of sorted times.  A wide grid (sharp
// kernels over a long span) has too many nodes and stays with the sweep.
void Executor::plan_grid(const std::vector<SetView>& sets, const int* setOf, const double* params,
                         int P) {
    gridOf_.clear();
    if (!gridSums || keptB || fixedR || fixedItems || shardWorld > 1 || D_ > 2) return;
    const auto large = [&](int p) {
        const int N = sets[setOf[p]].N;
        return N >= kGridMinEvents && N < (1 << 28) && sets[setOf[p]].haveBox;
    };
    int first = 0;
    while (first < P && !large(first)) ++first;
    if (first == P) return;
    const bool fp32 = precision_ != HPHC_PRECISION_FP64;
    std::vector<char> of(P, 0);
    std::vector<GridShape> shapes(P);
    std::vector<size_t> off(P, 0);
    size_t sums = 0, work = 0;
    bool any = false;
    CrowdSample sample;
    int sampled = -1;  // its set
    for (int p = first; p < P; ++p) {
        if (!large(p)) continue;
        const SetView& s = sets[setOf[p]];
        const double* prm = params + (size_t)6 * p;
        const PairConsts c = pair_consts(prm, s);
        const int nTiles = (s.N + kTile - 1) / kTile;
        // pairs the sweep would evaluate (each once)
        double pairs = 0.5 * s.N * (double)s.N;
        double tMin = s.hTileMin[0], tMax = s.hTileMax[nTiles - 1];
        if (s.sorted && c.skipB >= 0.0 && c.cB < 0.0) {
            const double d = std::sqrt(c.skipB / -c.cB);
            const int step = std::max(1, nTiles / 32);
            double tiles = 0.0;
            int n = 0;
            for (int k = 0; k < nTiles; k += step, ++n)
                tiles += k + 1 - (std::upper_bound(s.hTileMax, s.hTileMax + k + 1,
                                                   s.hTileMin[k] - d) - s.hTileMax);
            pairs = std::min(pairs, tiles / n * kTile * s.N);
        }
        if (!s.sorted)
            for (int k = 0; k < nTiles; ++k) {
                tMin = std::min(tMin, s.hTileMin[k]);
                tMax = std::max(tMax, s.hTileMax[k]);
            }
        const double direct = pairs * (fp32 ? kPairCostF32 : kPairCostF64);
        const int order = fp32 && s.N < kGridHighOrderEvents ? 12 : 16;
        const GridCost& cost = order == 16 ? kGridCost16 : kGridCost12;
        const double jobs = std::min(P, kGridMaxJobs);
        double room = direct - cost.fixed / jobs - s.N * cost.event;
        if (!(room > 0.0)) continue;
        // A tile's events go through one CTA, a few tiles' through a few, and a bin's are
        // ranked against each other: wide kernels and clusters.
        if (s.hLoc) {
            if (sampled != setOf[p]) {
                sample = crowd_sample(s);
                sampled = setOf[p];
            }
            const Crowd share = crowd(sample, order, prm[1], prm[2]);
            room -= std::max(0.0, s.N * (share.tile * kGridSerial / jobs - cost.spread)) +
                    kGridRank * share.bin * s.N * (double)s.N;
        }
        const double maxNodes = room / cost.node;
        if (!(maxNodes > 0.0)) continue;
        const double lo[3] = {tMin, D_ == 2 ? s.locMin[1] : 0.0, s.locMin[0]};
        const double hi[3] = {tMax, D_ == 2 ? s.locMax[1] : 0.0, s.locMax[0]};
        const GridShape g = grid_shape(order, prm[1], prm[2], lo, hi,
                                       std::min(maxNodes, kGridMaxNodes));
        if (!g.ok) continue;
        const size_t need = grid_workspace(g, s.N);
        if (need > kGridMaxWork) continue;
        of[p] = 1;
        shapes[p] = g;
        off[p] = sums;
        if (p > 0 || !sumsOut) sums += (size_t)3 * s.N;
        work = std::max(work, need);
        any = true;
    }
    if (!any) return;
    // workspace: room for several jobs at once where that is cheap
    size_t total = 0;
    for (int p = 0; p < P; ++p)
        if (of[p]) total += grid_workspace(shapes[p], sets[setOf[p]].N);
    work = std::max(work, std::min(total, kGridGroupWork));
    const auto grow = [&](void** ptr, size_t& cap, size_t bytes) {
        if (bytes <= cap) return true;
        if (*ptr) cudaFree(*ptr);
        *ptr = nullptr;
        cap = 0;
        if (cudaMalloc(ptr, bytes + bytes / 4) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cap = bytes + bytes / 4;
        return true;
    };
    // without the memory the pair sweep takes every problem
    if (!grow(&dGridWork_, gridWorkCap_, work) ||
        !grow(reinterpret_cast<void**>(&dGridSums_), gridSumsCap_,
              std::max<size_t>(sums, 1) * sizeof(double)))
        return;
    gridOf_.swap(of);
    gridShape_.swap(shapes);
    gridSumsOff_.swap(off);
}

// Enqueue the gridded sums of the planned problems, in groups that fit the
// workspace.
int Executor::launch_grid(const std::vector<SetView>& sets, const int* setOf,
                          const double* params, int P) {
    if (gridOf_.empty()) return HPHC_OK;
    cudaError_t e;
    if (kernelTiming && (e = cudaEventRecord(ev_[4], stream_))) return cuda_fail(e, "timing event");
    std::vector<GridJob> jobs;
    size_t used = 0;
    for (const int order : {12, 16}) {
        const auto flush = [&]() {
            if (jobs.empty()) return cudaSuccess;
            const cudaError_t err = launch_grid_sums(order, jobs.data(), (int)jobs.size(),
                                                     numSMs_, stream_, &gridLaunches_);
            jobs.clear();
            used = 0;
            return err;
        };
        for (int p = 0; p < P; ++p) {
            if (!gridOf_[p] || gridShape_[p].order != order) continue;
            const SetView& s = sets[setOf[p]];
            const double* prm = params + (size_t)6 * p;
            const size_t need = grid_workspace(gridShape_[p], s.N);
            if (((int)jobs.size() == kGridMaxJobs || used + need > gridWorkCap_) && (e = flush()))
                return cuda_fail(e, "gridded sums");
            GridJob j{};
            j.loc = s.dLoc;
            j.times = s.dTimes;
            j.sums = grid_sums(p);
            grid_job(gridShape_[p], prm[1], prm[2], s.N, D_, static_cast<char*>(dGridWork_) + used,
                     &j);
            used += need;
            jobs.push_back(j);
        }
        if ((e = flush())) return cuda_fail(e, "gridded sums");
    }
    if (kernelTiming && (e = cudaEventRecord(ev_[5], stream_))) return cuda_fail(e, "timing event");
    return HPHC_OK;
}

int Executor::build_plan(const std::vector<SetView>& sets, const int* setOf, const double* params,
                         int P, double* dProbs, int r, int items) {
    Plan& pl = plan_;
    pl.P = P;
    pl.setOf.assign(setOf, setOf + P);
    pl.sp.assign(P, SweepProblem{});
    pl.fp.assign(P, FinishProblem{});
    pl.pj.clear();
    pl.items.clear();
    pl.stripChunks.clear();
    pl.fb.clear();
    pl.maxN = 0;
    const bool fp32 = planPrecision_ != HPHC_PRECISION_FP64;
    const int stripEvents = kSweepThreads * r;
    const int S32 = f32_stride(D_);

    double totalStrips = 0.0;
    for (int p = 0; p < P; ++p) {
        const SetView& s = sets[setOf[p]];
        totalStrips += (s.N + stripEvents - 1) / stripEvents;
    }
    // a shard keeps about 1/shardWorld of the items: cut finer chunks so that
    // each rank still has `items` per SM
    const int target = numSMs_ * items * std::max(1, shardWorld);
    const int nChunksTarget = std::max(1, (int)std::ceil(target / std::max(1.0, totalStrips)));

    const auto gridded = [&](int p) { return !gridOf_.empty() && gridOf_[p] != 0; };
    const auto problem_consts = [&](int p) {
        PairConsts c = pair_consts(params + (size_t)6 * p, sets[setOf[p]]);
        if (gridded(p)) c.noB = 1;
        return c;
    };
    // A self-excitation-only sweep (kept or gridded background sums) visits a few
    // tiles before each strip.  Problems of one size with sorted times need no
    // work list for that: every strip gets the same number of slots, enough for
    // the widest band (the device loop: for every earlier tile), and an item's
    // tiles follow from its number (SweepProblem::slotItems).  A slot holds
    // the tiles that make about four items per resident CTA, at most a whole band.
    selfOnly_ = self_only(P);
    int selfSlots = 0, selfTiles = 1, selfShift = 0;
    // Small plans take their tiles in halves or quarters (WorkItem::cols), so that
    // every SM has an item and the time of one is less (N = 1000 FP64 sweep 46 -> 23
    // us, whole evaluation 71 -> 53): not in a fixed shape or a shard, whose sums are
    // compared, and not in the plain FP32 mode, where an item's length shows in the
    // sums' rounding.
    const bool partTiles = shardWorld == 1 && !(fixedR && fixedItems) && !(variant_ & 8);
    const auto part_shift = [&](double tiles) {  // log2 of the parts of items of so many tiles
        return !partTiles || tiles > 0.5 ? 0 : tiles > 0.25 ? 1 : 2;
    };
    // In the list form all problems take the same, from the largest.  The last
    // digits of FP32-compensated row sums show an item's length, so there the sizes
    // alone decide for up to eight problems (chunks of one tile too), whose results
    // then equal single evaluations'; more fill the SMs with whole tiles (64 problems
    // of N = 2000: 0.172 ms, in quarters 0.180).
    int partShift = 0;
    bool oneTile = false;
    if (!wideBands_) {
        int most = 1;
        for (int p = 0; p < P; ++p) most = std::max(most, (sets[setOf[p]].N + kTile - 1) / kTile);
        if (!fp32) partShift = part_shift((double)most / nChunksTarget);
        else if (P <= 8) partShift = part_shift(most / 64.0);
        oneTile = fp32 && partShift > 0;
    }
    const bool listless = selfOnly_ && self_listless(sets, setOf, P);
    if (listless) {
        const int nTiles = (sets[setOf[0]].N + kTile - 1) / kTile;
        const int nStrips = (sets[setOf[0]].N + stripEvents - 1) / stripEvents;
        int widest = 1;
        double bandTiles = 0.0;
        if (!wideBands_) pl.stripChunks.reserve((size_t)P * nStrips);
        for (int p = 0; p < P; ++p) {
            const SetView& s = sets[setOf[p]];
            const StripGaps gap(problem_consts(p));
            StripCursor at;
            for (int st = 0; st < nStrips; ++st) {
                int lo = 0, hi = nTiles;
                strip_band(s, gap, true, false, r, nTiles, st, at, &lo, &hi);
                widest = std::max(widest, hi - lo);
                bandTiles += hi - lo;
                // tiles back from the strip's last one, below their slots
                if (!wideBands_) pl.stripChunks.push_back(std::min((st + 1) * r, nTiles) - lo);
            }
        }
        const double perItem = bandTiles / (4.0 * sweep_grid(r));
        selfTiles = std::min(widest, std::max(1, (int)std::lround(perItem)));
        // Long items leave a last wave: there three times as many (N = 70k, omega =
        // 0.001, every earlier tile: 3105 -> 2987 us FP32-compensated, where a list,
        // longest first, took 2986)
        if (selfTiles > 8) selfTiles = std::max(8, selfTiles / 3);
        selfShift = part_shift(perItem);
        if (wideBands_) {  // for any sigma and omega
            widest = nTiles;
            selfShift = part_shift((double)P * nStrips * nTiles / (4.0 * sweep_grid(r)));
        }
        selfSlots = (widest + selfTiles - 1) / selfTiles << selfShift;
        // The finish reads the slots of each strip's own band: a burst's strips need
        // many more than the others, and the sweep leaves the rest alone (half of N = 12k
        // in one burst, FP32-compensated: a step 108 -> 102 us, 97 with a list; a tenth of N =
        // 100k, FP64: 420 -> 406)
        for (int& chunks : pl.stripChunks) chunks = (chunks + selfTiles - 1) / selfTiles << selfShift;
    }

    size_t recOff = 0, partOff = 0, colOff = 0;
    std::vector<size_t> chunkBase(P);
    std::vector<double> itemCost;  // parallel to pl.items
    int blockBase = 0;
    for (int p = 0; p < P; ++p) {
        const SetView& s = sets[setOf[p]];
        const double* prm = params + (size_t)6 * p;
        if (fp32 && !(prm[1] != 0.0 && prm[2] != 0.0 && std::isfinite(prm[1]) &&
                      std::isfinite(prm[2]))) {
            char buf[200];
            snprintf(buf, sizeof buf,
                     "FP32-compensated mode needs finite non-zero tauXprec and tauTprec (problem "
                     "%d: %g, %g); use the FP64 mode", p, prm[1], prm[2]);
            error = buf;
            return HPHC_ERR_UNSUPPORTED;
        }
        const int N = s.N;
        const int nTiles = (N + kTile - 1) / kTile;
        const int nStrips = (N + stripEvents - 1) / stripEvents;
        const int Npad = nStrips * stripEvents;
        // tiles a chunk, from the tuned items per SM
        const int CT =
            oneTile ? 1 : std::max(1, (nTiles + nChunksTarget - 1) / nChunksTarget);
        int maxSlots = 1;  // partial-sum slots the widest strip band uses
        pl.maxN = std::max(pl.maxN, N);
        SweepProblem& sp = pl.sp[p];
        sp.c = problem_consts(p);
        sp.N = N;
        sp.nTiles = nTiles;
        sp.Npad = Npad;
        sp.tileMin = s.dTileMin;
        sp.tileMax = s.dTileMax;
        // a self-excitation-only sweep has no background, so no column sums
        sp.symmetric = (symmetric && !sp.c.noB && N <= kMaxSymmetricEvents) ? 1 : 0;
        if (!fp32 && sp.symmetric) {
            // FP64 column sums are fixed point: bound each column total by N
            // times the largest term, B_u <= 1, B_u d^2 <= 1/(e |cA|),
            // B_u dt^2 <= 1/(e |cB|), and keep it below 2^62 units.  Padding
            // rows 1e150 away vanish only if |cA| is not astronomically small.
            if (!(sp.c.cA < -1e-280 && sp.c.cB < 0.0)) {
                sp.symmetric = 0;
            } else {
                const double e1 = std::exp(1.0);
                const double bound[3] = {(double)N, N / (e1 * -sp.c.cA), N / (e1 * -sp.c.cB)};
                for (int q = 0; q < 3; ++q) {
                    int ex = 0;
                    std::frexp(bound[q], &ex);  // bound < 2^ex
                    sp.colShift[q] = 62 - ex;
                }
            }
        }
        sp.searchBand = (wideBands_ && s.sorted) ? 1 : 0;
        sp.rowOrder = (fp32 && sp.symmetric) ? (r == 2 ? s.dOrder2 : r == 4 ? s.dOrder4 : nullptr)
                                             : nullptr;
        // the strips' row order is formed when a sweep first needs it, after that
        // with each upload
        RowOrder* order = sp.rowOrder ? (r == 2 ? s.order2 : s.order4) : nullptr;
        if (order) order->wanted = true;
        if (order && !order->ready) {
            const cudaError_t e = launch_strip_order(D_, N, r, s.dLoc, const_cast<int32_t*>(sp.rowOrder),
                                                     stream_);
            if (e != cudaSuccess) return cuda_fail(e, "strip order");
            order->ready = true;
        }
        sp.colAcc = nullptr;
        if (sp.symmetric) {
            sp.colAcc = reinterpret_cast<unsigned long long*>(colOff + 1);  // offset + 1
            colOff += (size_t)(fp32 ? 3 : 6) * Npad;
        }
        if (fp32) {
            // problems on the same set with the same tauX and tauT (sampler
            // chains, proposals that leave them fixed) share one record copy
            const double sX = record_scale(prm[1]), sT = record_scale(prm[2]);
            size_t off = recOff;
            bool shared = false;
            for (const PackJob& j : pl.pj)
                if (j.loc == s.dLoc && j.sX == sX && j.sT == sT) {
                    off = reinterpret_cast<size_t>(j.rec);
                    shared = true;
                    break;
                }
            sp.rec = reinterpret_cast<const void*>(off);  // offset, fixed up later
            if (!shared) {
                PackJob j{};
                j.loc = s.dLoc;
                j.times = s.dTimes;
                j.ranks = s.dRanks;
                j.rec = reinterpret_cast<float*>(recOff);
                j.sX = sX;
                j.sT = sT;
                j.N = N;
                pl.pj.push_back(j);
                recOff += (size_t)N * S32;
            }
        } else {
            sp.rec = s.dRecF64;
            if (s.packedF64 && !*s.packedF64) {  // FP32 engines: packed when first needed
                const cudaError_t e =
                    launch_pack_f64(D_, N, s.dLoc, s.dTimes, const_cast<double*>(s.dRecF64),
                                    const_cast<double*>(s.dTileMin),
                                    const_cast<double*>(s.dTileMax), stream_);
                if (e != cudaSuccess) return cuda_fail(e, "pack FP64 records");
                *s.packedF64 = true;
            }
        }

        // work items: each strip's band of tiles that may hold a non-zero term
        chunkBase[p] = listless ? (size_t)p * nStrips : pl.stripChunks.size();
        sp.partShift = listless ? selfShift : partShift;
        if (listless) {
            maxSlots = selfSlots;
            sp.slotItems = P * nStrips;
            sp.strips = nStrips;
            sp.chunkTiles = selfTiles;
        }
        StripCursor at;
        const StripGaps gap(sp.c);
        for (int st = 0; st < nStrips && !listless; ++st) {
            int lo = 0, hi = nTiles;
            strip_band(s, gap, sp.symmetric != 0, wideBands_, r, nTiles, st, at, &lo, &hi);
            const StripCost sc = strip_cost(s, gap, fp32, r, nTiles, st, at);
            // Chunks sit on a fixed grid of CT tiles per problem, so a tile
            // always lands in the same chunk whatever the band: skipping a
            // band's outside only drops chunks whose sums are exactly zero,
            // and the FP64 chunk sums are added in the same order either way.
            const int cFirst = lo / CT, cLast = (hi - 1) / CT + 1;
            for (int c = cFirst; c < cLast; ++c) {
                WorkItem w{};
                w.problem = p;
                w.strip = st;
                w.jt0 = std::max(lo, c * CT);
                w.jt1 = std::min(hi, (c + 1) * CT);
                w.slot = c - cFirst;
                w.start = w.jt0;
                w.cols = kTile;
                pl.items.push_back(w);
                itemCost.push_back(item_cost(sc, sp.c.noB != 0, w.jt0, w.jt1));
            }
            pl.stripChunks.push_back((cLast - cFirst) << partShift);
            maxSlots = std::max(maxSlots, (cLast - cFirst) << partShift);
        }
        // partial sums: as many slots per strip as the widest band uses
        sp.partials = reinterpret_cast<double*>(partOff);  // offset, fixed up later
        partOff += (size_t)maxSlots * kNumAcc * Npad;

        FinishProblem& fp = pl.fp[p];
        fp.partials = nullptr;  // fixed up later
        fp.colAcc = nullptr;
        fp.stripChunks = nullptr;
        fp.times = s.dTimes;
        fp.loc = s.dLoc;
        fp.tileMin = s.dTileMin;
        fp.tileMax = s.dTileMax;
        fp.nTiles = nTiles;
        fp.sorted = s.sorted ? 1 : 0;
        fp.probs = (p == 0) ? dProbs : nullptr;
        fp.sums = (p == 0) ? sumsOut : nullptr;
        fp.keptB = gridded(p) ? grid_sums(p) : keptB;
        fp.N = N;
        fp.Npad = Npad;
        fp.stripEvents = stripEvents;
        fp.blockBase = blockBase;
        fp.nBlocks = finish_blocks(N);
        fp.colWords = fp32 ? 1 : 2;
        for (int q = 0; q < 4; ++q) fp.colShift[q] = sp.colShift[q];
        fp.f = finish_consts(prm, s);
        for (int b = 0; b < fp.nBlocks; ++b) pl.fb.push_back(FinishBlock{p, b * kFinishThreads});
        blockBase += fp.nBlocks;
    }
    pl.nBlocks = blockBase;
    if (shardWorld > 1) {
        // Longest-processing-time assignment of whole strips to ranks by
        // their item costs; ties go to the lower strip and the lower rank,
        // so every rank derives the same assignment from the same plan.
        const size_t nS = pl.stripChunks.size();
        std::vector<double> cost(nS, 0.0);
        for (size_t k = 0; k < pl.items.size(); ++k)
            cost[chunkBase[pl.items[k].problem] + pl.items[k].strip] += itemCost[k];
        std::vector<int> order(nS);
        for (size_t k = 0; k < nS; ++k) order[k] = (int)k;
        std::stable_sort(order.begin(), order.end(),
                         [&](int x, int y) { return cost[x] > cost[y]; });
        std::vector<double> load(shardWorld, 0.0);
        std::vector<char> owned(nS, 0);
        for (int k : order) {
            int best = 0;
            for (int r = 1; r < shardWorld; ++r)
                if (load[r] < load[best]) best = r;
            load[best] += cost[k];
            owned[k] = best == shardRank;
        }
        size_t kept = 0;
        for (size_t k = 0; k < pl.items.size(); ++k)
            if (owned[chunkBase[pl.items[k].problem] + pl.items[k].strip]) {
                itemCost[kept] = itemCost[k];
                pl.items[kept++] = pl.items[k];
            }
        pl.items.resize(kept);
        itemCost.resize(kept);
        for (size_t k = 0; k < nS; ++k)
            if (!owned[k]) pl.stripChunks[k] = 0;
    }
    // table layout and buffer capacities
    offSP_ = 0;
    offItems_ = align16(offSP_ + sizeof(SweepProblem) * P);
    const size_t nItems =
        listless ? (size_t)selfSlots * pl.sp[0].slotItems : pl.items.size() << partShift;
    itemsCap_ = std::max(itemsCap_, pl.items.size());
    offNItems_ = align16(offItems_ + sizeof(WorkItem) * itemsCap_);
    offChunks_ = align16(offNItems_ + sizeof(int));
    offFP_ = align16(offChunks_ + sizeof(int) * pl.stripChunks.size());
    offFB_ = align16(offFP_ + sizeof(FinishProblem) * P);
    offPJ_ = align16(offFB_ + sizeof(FinishBlock) * pl.fb.size());
    tablesBytes_ = align16(offPJ_ + sizeof(PackJob) * pl.pj.size());

    // an FP64 plan of an FP32-compensated engine reserves what its self-excitation
    // steps will take: the records they pack, and the partial sums of strips twice as
    // high, which have half the items' tiles and twice the slots
    recNeed_ = planPrecision_ == precision_ ? recOff : (size_t)pl.maxN * S32;
    partialsNeed_ = planPrecision_ == precision_ ? partOff : 2 * partOff;
    colNeed_ = colOff;
    int st = ensure_buffers();
    if (st) return st;

    // fix up offsets into device pointers and fill the staging buffer
    char* h = static_cast<char*>(hStaging_);
    char* d = static_cast<char*>(dTables_);
    for (int p = 0; p < P; ++p) {
        SweepProblem& sp = pl.sp[p];
        const size_t po = reinterpret_cast<size_t>(sp.partials);
        sp.partials = dPartials_ + po;
        if (sp.colAcc) sp.colAcc = dColAcc_ + (reinterpret_cast<size_t>(sp.colAcc) - 1);
        if (fp32) sp.rec = dRecPool_ + reinterpret_cast<size_t>(sp.rec);
        FinishProblem& fp = pl.fp[p];
        fp.partials = sp.partials;
        fp.colAcc = sp.colAcc;
        fp.stripChunks =
            pl.stripChunks.empty() ? nullptr
                                   : reinterpret_cast<const int*>(d + offChunks_) + chunkBase[p];
        fp.slots = selfSlots;
        sp.slotsUsed = listless ? fp.stripChunks : nullptr;
    }
    for (auto& j : pl.pj) j.rec = dRecPool_ + reinterpret_cast<size_t>(j.rec);
    willPack_ = Packed{};
    if (pl.pj.size() == 1) {
        const PackJob& j = pl.pj[0];
        willPack_.version = sets[setOf[0]].version;
        willPack_.loc = j.loc;
        willPack_.sX = j.sX;
        willPack_.sT = j.sT;
    }
    skipPack_ = willPack_.version != 0 && packed_.version == willPack_.version &&
                packed_.loc == willPack_.loc && packed_.sX == willPack_.sX &&
                packed_.sT == willPack_.sT;
    std::memcpy(h + offSP_, pl.sp.data(), sizeof(SweepProblem) * P);
    stage_items(pl.items, itemCost, reinterpret_cast<WorkItem*>(h + offItems_));
    const int n = (int)nItems;
    std::memcpy(h + offNItems_, &n, sizeof(int));
    if (!pl.stripChunks.empty())
        std::memcpy(h + offChunks_, pl.stripChunks.data(), sizeof(int) * pl.stripChunks.size());
    std::memcpy(h + offFP_, pl.fp.data(), sizeof(FinishProblem) * P);
    std::memcpy(h + offFB_, pl.fb.data(), sizeof(FinishBlock) * pl.fb.size());
    if (!pl.pj.empty()) std::memcpy(h + offPJ_, pl.pj.data(), sizeof(PackJob) * pl.pj.size());
    return HPHC_OK;
}

int Executor::ensure_buffers() {
    const Plan& pl = plan_;
    bool grew = false;
    cudaError_t e = cudaSuccess;
    auto grow_dev = [&](void** ptr, size_t& cap, size_t needBytes) -> cudaError_t {
        if (needBytes <= cap && *ptr) return cudaSuccess;
        const size_t n = std::max<size_t>(needBytes + needBytes / 4, 256);
        if (*ptr) cudaFree(*ptr);
        *ptr = nullptr;
        cap = 0;
        const cudaError_t err = cudaMalloc(ptr, n);
        if (err == cudaSuccess) cap = n;
        grew = true;
        return err;
    };
    if ((e = grow_dev(reinterpret_cast<void**>(&dRecPool_), recCap_,
                      std::max<size_t>(recNeed_, 1) * sizeof(float))) != cudaSuccess ||
        (e = grow_dev(reinterpret_cast<void**>(&dPartials_), partialsCap_,
                      std::max<size_t>(partialsNeed_, 1) * sizeof(double))) != cudaSuccess ||
        (e = grow_dev(reinterpret_cast<void**>(&dColAcc_), colCap_,
                      std::max<size_t>(colNeed_, 1) * sizeof(unsigned long long))) !=
            cudaSuccess ||
        (e = grow_dev(reinterpret_cast<void**>(&dArrived_), arrivedCap_,
                      (size_t)(1 + pl.P) * sizeof(int))) != cudaSuccess ||
        (e = grow_dev(reinterpret_cast<void**>(&dBlockSums_), blockCap_,
                      (size_t)std::max(pl.nBlocks, 1) * 8 * sizeof(double))) != cudaSuccess ||
        (e = grow_dev(&dTables_, tablesCap_, tablesBytes_)) != cudaSuccess)
        return cuda_fail(e, "device allocation");
    if (stagingCap_ < tablesCap_) {
        if (hStaging_) cudaFreeHost(hStaging_);
        hStaging_ = nullptr;
        stagingCap_ = 0;
        if ((e = cudaMallocHost(&hStaging_, tablesCap_)) != cudaSuccess)
            return cuda_fail(e, "pinned allocation");
        stagingCap_ = tablesCap_;
        grew = true;
    }
    if (outCap_ < (size_t)pl.P * 8) {
        if (dOut_) cudaFree(dOut_);
        if (hOut_) cudaFreeHost(hOut_);
        dOut_ = hOut_ = nullptr;
        outCap_ = 0;
        const size_t n = (size_t)pl.P * 8;
        if ((e = cudaMalloc(&dOut_, n * sizeof(double))) != cudaSuccess ||
            (e = cudaMallocHost(&hOut_, n * sizeof(double))) != cudaSuccess)
            return cuda_fail(e, "device allocation");
        outCap_ = n;
        grew = true;
    }
    if (grew) {
        drop_graphs();
        stale_ = true;
        packed_ = Packed{};
    }
    // the counters and column sums every run leaves at zero: set here when they
    // are new or an earlier run may not have ended
    if (stale_) {
        if ((e = cudaMemsetAsync(dCounter_, 0, sizeof(int), stream_)) ||
            (e = cudaMemsetAsync(dArrived_, 0, arrivedCap_, stream_)) ||
            (e = cudaMemsetAsync(dColAcc_, 0, colCap_, stream_)))
            return cuda_fail(e, "reset counters");
        stale_ = false;
    }
    return HPHC_OK;
}

// Timing events: inside a stream capture an event is only recorded as a graph
// node (and so usable for elapsed times) when marked external.
cudaError_t Executor::record(cudaEvent_t ev) {
    return capturing_ ? cudaEventRecordWithFlags(ev, stream_, cudaEventRecordExternal)
                      : cudaEventRecord(ev, stream_);
}

// The stage sequence of one run on stream_ (also what the graph captures).
int Executor::launch_sequence(int grid) {
    const Plan& pl = plan_;
    const int prec = planPrecision_ == HPHC_PRECISION_FP64 ? 0 : 1;
    char* d = static_cast<char*>(dTables_);
    const auto* sp = reinterpret_cast<const SweepProblem*>(d + offSP_);
    const auto* items = reinterpret_cast<const WorkItem*>(d + offItems_);
    const auto* nItems = reinterpret_cast<const int*>(d + offNItems_);
    const auto* fp = reinterpret_cast<const FinishProblem*>(d + offFP_);
    const auto* fb = reinterpret_cast<const FinishBlock*>(d + offFB_);
    const auto* pj = reinterpret_cast<const PackJob*>(d + offPJ_);
    cudaError_t e = cudaSuccess;
    int launches = 0;
    if (kernelTiming && (e = record(ev_[0]))) return cuda_fail(e, "timing event");
    const bool smallTables = tablesBytes_ <= kCopyKernelBytes;
    if (smallTables) {
        e = launch_copy_tables(dTables_, hStaging_, tablesBytes_, stream_);
        ++launches;
    } else {
        e = cudaMemcpyAsync(dTables_, hStaging_, tablesBytes_, cudaMemcpyHostToDevice, stream_);
    }
    if (e != cudaSuccess) return cuda_fail(e, "stage tables");
    const bool packs = prec == 1 && !skipPack_;
    if (prec == 1 && !skipPack_) {
        if (!capturing_) packed_ = willPack_;
        if ((e = launch_pack_f32_jobs(D_, (int)pl.pj.size(), pl.maxN, pj, stream_)))
            return cuda_fail(e, "pack kernel");
        ++launches;
    }
    if (kernelTiming && (e = record(ev_[1]))) return cuda_fail(e, "timing event");
    // set up behind the last kernel, if no event lies between
    const int variant =
        sweep_variant() | (!kernelTiming && (smallTables || packs) ? kAfterKernel : 0);
    if ((e = launch_sweep_list(prec, D_, R, variant, grid, sp, items, nItems, dCounter_, stream_)))
        return cuda_fail(e, "sweep kernel");
    if (kernelTiming && (e = record(ev_[2]))) return cuda_fail(e, "timing event");
    // the results go straight to the pinned host buffer
    if ((e = launch_finish_list(pl.nBlocks, fp, fb, pl.P, dBlockSums_, dArrived_, dCounter_, hOut_,
                                !kernelTiming, stream_)))
        return cuda_fail(e, "finish kernel");
    launches += 2;
    if (kernelTiming && (e = record(ev_[3]))) return cuda_fail(e, "timing event");
    lastLaunches = launches;
    return HPHC_OK;
}

int Executor::autotune(const std::vector<SetView>& sets, const int* setOf, const double* params,
                       int P, double* dProbs) {
    double pairs = 0.0;
    for (int p = 0; p < P; ++p) pairs += (double)sets[setOf[p]].N * sets[setOf[p]].N;
    pairs /= std::max(1, shardWorld);  // work of this rank
    const int mode = variant_ | (symmetric ? 16 : 0) | (fastTail ? 32 : 0) | (skip_ ? 64 : 0) |
                     (truncateTail ? 128 : 0) | (selfOnly_ ? 256 : 0);
    const TuneKey key = std::make_tuple(D_, planPrecision_, mode, log2_bucket(pairs), log2_bucket(P));
    if (deviceName_.empty()) {
        cudaDeviceProp prop{};
        deviceName_ = cudaGetDeviceProperties(&prop, device_) == cudaSuccess ? prop.name : "?";
    }
    {
        std::lock_guard<std::mutex> lock(gTuneMutex);
        auto it = gTuneCache.find(key);
        if (it == gTuneCache.end()) {
            read_tune_file();
            for (const TuneLine& t : gTuneFile)
                if (t.key == key && t.sms == numSMs_ && t.device == deviceName_) {
                    it = gTuneCache.emplace(key, std::make_pair(t.R, t.items)).first;
                    break;
                }
        }
        if (it != gTuneCache.end()) {
            R = fixedR ? fixedR : it->second.first;
            itemsPerSM = fixedItems ? fixedItems : it->second.second;
            return HPHC_OK;
        }
    }
    std::vector<int> rs, its;
    if (fixedR) rs = {fixedR};
    else if (planPrecision_ == HPHC_PRECISION_FP64) rs = {1, 2};
    else rs = {2, 4};
    if (fixedItems) its = {fixedItems};
    else if (selfOnly_) its = {8, 16, 32};  // short sweeps: fewer items to plan and upload
    else its = {8, 16, 32, 64};
    const bool timing = kernelTiming;
    kernelTiming = true;
    float best = 1e30f;
    int bestR = rs[0], bestI = its[0];
    int st = HPHC_OK;
    for (int r : rs) {
        for (int it : its) {
            R = r;
            itemsPerSM = it;
            if ((st = build_plan(sets, setOf, params, P, dProbs, r, it))) break;
            const int grid = sweep_grid(r);
            // sweep and finish, whose work grows with the number of items;
            // median of four after one that warms the caches: the
            // shapes' typical times differ by ~1 %, about as much as the
            // best of a few launches varies
            float times[kTuneReps];
            int nt = 0;
            for (int rep = 0; rep <= kTuneReps && !st; ++rep) {
                if ((st = launch_sequence(grid))) break;
                cudaError_t e = cudaStreamSynchronize(stream_);
                float t = 0.f;
                if (e == cudaSuccess) e = cudaEventElapsedTime(&t, ev_[1], ev_[3]);
                if (e != cudaSuccess) {
                    st = cuda_fail(e, "autotune timing");
                    break;
                }
                if (rep > 0) times[nt++] = t;
            }
            float ms = 1e30f;
            if (!st && nt == kTuneReps) {
                std::sort(times, times + nt);
                ms = 0.5f * (times[nt / 2 - 1] + times[nt / 2]);
            }
            if (st) break;
            if (ms < best) {
                best = ms;
                bestR = r;
                bestI = it;
            }
        }
        if (st) break;
    }
    kernelTiming = timing;
    if (st) return st;
    if (!fixedR && !fixedItems) {  // a shape tuned under a constraint is not cached
        std::lock_guard<std::mutex> lock(gTuneMutex);
        gTuneCache[key] = {bestR, bestI};
        append_tune_file(deviceName_, numSMs_, key, bestR, bestI);
    }
    R = bestR;
    itemsPerSM = bestI;
    return HPHC_OK;
}

// R and itemsPerSM for the current kind of plan: fixed by the caller, or tuned
// the first time the kind runs with a list.  A self-excitation-only sweep of an engine
// whose full sweeps are tuned keeps their shape.
int Executor::choose_shape(const std::vector<SetView>& sets, const int* setOf,
                           const double* params, int P, double* dProbs) {
    selfOnly_ = self_only(P);
    kind_ = !selfOnly_ ? 0 : planPrecision_ == precision_ ? 1 : 2;
    Shape& s = shape_[kind_];
    if (fixedR && fixedItems) {
        s.R = fixedR;
        s.items = fixedItems;
        s.tuned = true;
    }
    if (kind_ == 1 && !s.tuned && shape_[0].tuned) {
        s = shape_[0];
        // a few thousand events: more, smaller strips fill the SMs
        if (!fixedR && sets[setOf[0]].N <= 8192) s.R = precision_ == HPHC_PRECISION_FP64 ? 1 : 2;
    }
    // without a list there is one question left: R = 2 against 4 in FP32 0.125 : 0.155 ms
    // at N = 100k and 1.15 : 1.30 at 400k; R = 1 against 2 in FP64 50 : 56 us at N = 20k
    // and 261 : 269 at 100k (1e8 terms), but 1.33 : 1.26 ms at N = 70k and omega = 0.05
    // (7e8 terms), 2.59 : 2.46 at 400k (1.6e9) and 5.08 : 4.73 where N = 70k takes all
    if (!s.tuned && selfOnly_ && self_listless(sets, setOf, P)) {
        R = fixedR ? fixedR : 2;
        if (!fixedR && planPrecision_ == HPHC_PRECISION_FP64 &&
            P * self_terms(sets[setOf[0]], params) < kLongSelfTerms)
            R = 1;
        itemsPerSM = fixedItems ? fixedItems : 8;
        return HPHC_OK;
    }
    if (!s.tuned) {
        const int st = autotune(sets, setOf, params, P, dProbs);
        if (st) return st;
        s.R = R;
        s.items = itemsPerSM;
        s.tuned = true;
    }
    R = s.R;
    itemsPerSM = s.items;
    return HPHC_OK;
}

// Self-excitation terms an FP64 sweep of the set would evaluate, estimated from
// sampled tiles.
double Executor::self_terms(const SetView& s, const double* p) const {
    ConstsSpec spec = consts_spec(s, p[3]);
    spec.precision = 0;
    PairConsts c{};
    FinishConsts f{};
    param_consts(p, spec, c, f);
    if (!s.sorted || !(c.skipS >= 0.0 && c.cW < 0.0)) return 0.5 * s.N * (double)s.N;
    const double d = c.skipS / -c.cW;
    const int nTiles = (s.N + kTile - 1) / kTile, step = std::max(1, nTiles / 32);
    double tiles = 0.0;
    int n = 0;
    for (int k = 0; k < nTiles; k += step, ++n)
        tiles += k + 1 - (std::upper_bound(s.hTileMax, s.hTileMax + k + 1, s.hTileMin[k] - d) -
                          s.hTileMax);
    return tiles / n * kTile * s.N;
}

// The memory of the gridded sums given back, the problems planned for them to the pair
// sweep; false if there is none.
bool Executor::release_grid() {
    if (!dGridWork_ && !dGridSums_) return false;
    cudaFree(dGridWork_);  // waits for kernels in flight
    cudaFree(dGridSums_);
    dGridSums_ = nullptr;
    dGridWork_ = nullptr;
    gridSumsCap_ = gridWorkCap_ = 0;
    gridOf_.clear();
    return true;
}

// Precision, shape and tables of a run whose gridded problems are chosen; starts their
// sums.
int Executor::plan(const std::vector<SetView>& sets, const int* setOf, const double* params,
                   int P, double* dProbs) {
    // Large gridded evaluations of the FP32-compensated mode sweep their
    // self-excitation terms in FP64 too, where that is a small part of them: the
    // grid's sums are exact to 1e-15, and the sweep's 0.19 instead of 0.13 ms at
    // N = 100k make the whole evaluation so (log-likelihood 2.7e-11 -> 1.1e-16,
    // worst gradient component 9.6e-10 -> 3.6e-15 relative).  Where the terms are
    // many they stay in FP32 (N = 500k clustered: 2.2 against 4.1 ms, beside 2.0 ms
    // of grid kernels).
    planPrecision_ = precision_;
    if (precision_ == HPHC_PRECISION_FP32_COMP && !keptB && self_only(P)) {
        bool large = true;
        for (int p = 0; p < P; ++p)
            large &= gridShape_[p].order == 16 && sets[setOf[p]].dRecF64 != nullptr &&
                     self_terms(sets[setOf[p]], params + (size_t)6 * p) * kSelfCostF64 <
                         0.5 * (gridShape_[p].nodes * kGridCost16.node +
                                sets[setOf[p]].N * kGridCost16.event);
        if (large) planPrecision_ = HPHC_PRECISION_FP64;
    }
    int st = choose_shape(sets, setOf, params, P, dProbs);
    if (st) return st;
    // the gridded sums need no plan: the device forms them while the host plans
    gridLaunches_ = 0;
    const bool faulty = faultStage == HPHC_FAULT_LAUNCH && faultCount > 0;
    if (!faulty && (st = launch_grid(sets, setOf, params, P))) return st;
    return build_plan(sets, setOf, params, P, dProbs, R, itemsPerSM);
}

int Executor::enqueue(const std::vector<SetView>& sets, const int* setOf, const double* params,
                      int P, double* dProbs) {
    if (P < 1) {
        error = "no problems to evaluate";
        return HPHC_ERR_BAD_ARGUMENT;
    }
    // the choice of the grid asks for the engine's own cuts, not those of the plan before
    planPrecision_ = precision_;
    plan_grid(sets, setOf, params, P);
    int st = plan(sets, setOf, params, P, dProbs);
    // short of memory: again with the pair sweep, without what the grid holds
    if (st == HPHC_ERR_OUT_OF_MEMORY && release_grid())
        st = plan(sets, setOf, params, P, dProbs);
    if (st) return st;
    const int grid = sweep_grid(R);
    timedValid = false;
    if (!useGraph) {
        st = launch_sequence(grid);
        lastLaunches += gridLaunches_;
        timedValid = kernelTiming && st == HPHC_OK;
        return st;
    }
    GraphKey key;
    key.P = plan_.P;
    key.nJobs = (int)plan_.pj.size();
    key.nBlocks = plan_.nBlocks;
    key.maxN = plan_.maxN;
    key.R = R;
    key.grid = grid;
    key.tablesBytes = tablesBytes_;
    const size_t offsets[] = {offSP_, offItems_, offNItems_, offChunks_, offFP_, offFB_, offPJ_};
    std::copy(std::begin(offsets), std::end(offsets), key.offsets);
    key.tables = dTables_;
    key.timing = kernelTiming;
    key.variant = sweep_variant() | planPrecision_ << 16;
    const int slot = kind_ + (skipPack_ ? 3 : 0);
    cudaGraphExec_t& exec = graphExec_[slot];
    GraphKey& last = graphKey_[slot];
    cudaError_t e;
    if (!(key == last)) {
        drop_graph(slot);
        last = key;
    }
    // A step on kept sums is captured the second time its layout comes, so that a first
    // step costs no capture: first step after an evaluation, FP32-compensated, N = 3000
    // 114 -> 48 us, N = 100k 977 -> 188 with its buffers reserved (build_plan).  A replay
    // takes 4 us less than the launches (N = 3000: 34 against 38 us), the capture 80 to
    // 100.  Evaluations are captured at once (N = 500: the first pass of a new set 134
    // us, 211 where the capture falls into it instead of the set's first evaluation).
    if (!exec && keptB && !kernelTiming && !met_[slot]) {
        met_[slot] = true;
        if (take_fault(HPHC_FAULT_LAUNCH))
            return cuda_fail(cudaErrorLaunchOutOfResources, "launch kernels (injected)");
        st = launch_sequence(grid);
        lastLaunches += gridLaunches_;
        return st;
    }
    if (!exec) {
        cudaGraph_t graph = nullptr;
        if ((e = cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal)))
            return cuda_fail(e, "begin graph capture");
        capturing_ = true;
        st = launch_sequence(grid);
        capturing_ = false;
        e = cudaStreamEndCapture(stream_, &graph);
        if (st) {
            if (graph) cudaGraphDestroy(graph);
            return st;
        }
        if (e != cudaSuccess) return cuda_fail(e, "end graph capture");
        e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            exec = nullptr;
            return cuda_fail(e, "instantiate graph");
        }
    }
    if (take_fault(HPHC_FAULT_LAUNCH))
        return cuda_fail(cudaErrorLaunchOutOfResources, "launch graph (injected)");
    if ((e = cudaGraphLaunch(exec, stream_))) return cuda_fail(e, "launch graph");
    const bool packs = planPrecision_ != HPHC_PRECISION_FP64 && !skipPack_;
    if (packs) packed_ = willPack_;
    lastLaunches = (packs ? 3 : 2) + (tablesBytes_ <= kCopyKernelBytes) + gridLaunches_;
    timedValid = kernelTiming;
    return HPHC_OK;
}

int Executor::wait(double* hostOut) {
    const cudaError_t e = cudaStreamSynchronize(stream_);
    if (e != cudaSuccess) return cuda_fail(e, "evaluation");
    if (take_fault(HPHC_FAULT_WAIT)) {
        timedValid = false;
        return cuda_fail(cudaErrorLaunchTimeout, "evaluation (injected)");
    }
    if (hostOut) std::memcpy(hostOut, hOut_, (size_t)plan_.P * 8 * sizeof(double));
    if (timedValid) {
        cudaError_t t;
        if ((t = cudaEventElapsedTime(&lastSweepMs, ev_[1], ev_[2])) != cudaSuccess ||
            (t = cudaEventElapsedTime(&lastFinishMs, ev_[2], ev_[3])) != cudaSuccess ||
            (t = cudaEventElapsedTime(&lastStepMs, ev_[0], ev_[3])) != cudaSuccess) {
            timedValid = false;
            return cuda_fail(t, "kernel timing");
        }
        if (!gridOf_.empty()) {  // the gridded sums are part of the sweep and of the step
            float grid = 0.f;
            if ((t = cudaEventElapsedTime(&grid, ev_[4], ev_[5])) != cudaSuccess ||
                (t = cudaEventElapsedTime(&lastStepMs, ev_[4], ev_[3])) != cudaSuccess) {
                timedValid = false;
                return cuda_fail(t, "kernel timing");
            }
            lastSweepMs += grid;
        }
    }
    return HPHC_OK;
}

int Executor::setup_device_loop(const std::vector<SetView>& sets, const int* setOf,
                                const double* params, int P) {
    if (P < 1) {
        error = "no problems to evaluate";
        return HPHC_ERR_BAD_ARGUMENT;
    }
    gridOf_.clear();  // the loop sweeps every term that is not kept
    planPrecision_ = precision_;
    int st = choose_shape(sets, setOf, params, P, nullptr);
    if (st) return st;
    wideBands_ = true;
    st = build_plan(sets, setOf, params, P, nullptr, R, itemsPerSM);
    if (st == HPHC_ERR_OUT_OF_MEMORY && release_grid())
        st = build_plan(sets, setOf, params, P, nullptr, R, itemsPerSM);
    wideBands_ = false;
    if (st) return st;
    drop_graphs();  // the tables' layout changed under any captured graph
    cudaError_t e;
    if ((e = cudaMemcpyAsync(dTables_, hStaging_, tablesBytes_, cudaMemcpyHostToDevice, stream_)))
        return cuda_fail(e, "stage tables");
    if (planPrecision_ != HPHC_PRECISION_FP64) {
        packed_ = willPack_;
        char* d = static_cast<char*>(dTables_);
        if ((e = launch_pack_f32_jobs(D_, (int)plan_.pj.size(), plan_.maxN,
                                      reinterpret_cast<const PackJob*>(d + offPJ_), stream_)))
            return cuda_fail(e, "pack kernel");
    }
    if ((e = cudaStreamSynchronize(stream_))) return cuda_fail(e, "device loop set-up");
    loopGrid_ = sweep_grid(R);
    return HPHC_OK;
}

int Executor::enqueue_device_body() {
    const int prec = planPrecision_ == HPHC_PRECISION_FP64 ? 0 : 1;
    char* d = static_cast<char*>(dTables_);
    const auto* sp = reinterpret_cast<const SweepProblem*>(d + offSP_);
    auto* items = reinterpret_cast<WorkItem*>(d + offItems_);
    const auto* nItems = reinterpret_cast<const int*>(d + offNItems_);
    const auto* fp = reinterpret_cast<const FinishProblem*>(d + offFP_);
    const auto* fb = reinterpret_cast<const FinishBlock*>(d + offFB_);
    cudaError_t e;
    const int variant = sweep_variant() | kAfterKernel;  // the step's, or the band kernel
    // a listed plan holds every earlier tile for any sigma and omega: start each
    // item where the current constants allow a term (the sweep of a plan without
    // a list finds that itself)
    if (!plan_.items.empty() &&
        (e = launch_band_starts((int)plan_.items.size(), sp, items, nItems, R, stream_)))
        return cuda_fail(e, "band kernel");
    if ((e = launch_sweep_list(prec, D_, R, variant, loopGrid_, sp, items, nItems,
                               dCounter_, stream_)))
        return cuda_fail(e, "sweep kernel");
    if ((e = launch_finish_list(plan_.nBlocks, fp, fb, plan_.P, dBlockSums_, dArrived_, dCounter_,
                                dOut_, true, stream_)))
        return cuda_fail(e, "finish kernel");
    lastLaunches = 3;
    return HPHC_OK;
}

SweepProblem* Executor::device_sweep_problems() const {
    return reinterpret_cast<SweepProblem*>(static_cast<char*>(dTables_) + offSP_);
}

FinishProblem* Executor::device_finish_problems() const {
    return reinterpret_cast<FinishProblem*>(static_cast<char*>(dTables_) + offFP_);
}

void Executor::count_terms(const std::vector<SetView>& sets, double* bTerms, double* sTerms,
                           double* bEvals) const {
    double nb = 0.0, ns = 0.0, ne = 0.0;
    const int stripEvents = kSweepThreads * R;
    std::vector<WorkItem> listless;  // the items of a plan without a list (see work_item)
    for (int p = 0; p < plan_.P && plan_.sp[p].slotItems > 0; ++p) {
        const SweepProblem& sp = plan_.sp[p];
        for (int k = 0; k < sp.strips * plan_.fp[p].slots; ++k) {
            WorkItem w{};
            w.problem = p;
            w.strip = k % sp.strips;
            const int slot = k / sp.strips, at = slot >> sp.partShift;
            w.cols = kTile >> sp.partShift;
            w.col0 = (slot - (at << sp.partShift)) * w.cols;
            w.jt1 = std::max(0, std::min((w.strip + 1) * R, sp.nTiles) - at * sp.chunkTiles);
            w.jt0 = std::max(0, w.jt1 - sp.chunkTiles);
            listless.push_back(w);
        }
    }
    for (const WorkItem& w : listless.empty() ? plan_.items : listless) {
        const SetView& s = sets[plan_.setOf[w.problem]];
        const PairConsts& c = plan_.sp[w.problem].c;
        const int nTiles = plan_.sp[w.problem].nTiles;
        const int ts0 = w.strip * R, ts1 = std::min(ts0 + R, nTiles);
        double tminI = INFINITY, tmaxI = -INFINITY;
        for (int t = ts0; t < ts1; ++t) {
            tminI = std::min(tminI, s.hTileMin[t]);
            tmaxI = std::max(tmaxI, s.hTileMax[t]);
        }
        const double ni = std::min(stripEvents, s.N - w.strip * stripEvents);
        const bool sym = plan_.sp[w.problem].symmetric != 0;
        for (int jt = w.jt0; jt < w.jt1; ++jt) {
            bool b, se;
            tile_needs(tminI, tmaxI, s.hTileMin[jt], s.hTileMax[jt], c, &b, &se);
            if (sym && jt >= ts1) b = false;
            const double nj = std::max(0, std::min(w.cols, s.N - jt * kTile - w.col0));
            if (b) {
                // a symmetric tile also accounts for the pairs' other order
                nb += (sym && jt < ts0 ? 2.0 : 1.0) * ni * nj;
                ne += ni * nj;
            }
            if (se) ns += ni * nj;
        }
    }
    // a gridded problem's sums account for every ordered pair, none evaluated
    for (size_t p = 0; p < gridOf_.size(); ++p)
        if (gridOf_[p]) nb += (double)plan_.sp[p].N * plan_.sp[p].N;
    *bTerms = nb;
    *sTerms = ns;
    if (bEvals) *bEvals = ne;
}

}  // namespace hphc
