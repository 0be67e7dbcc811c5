// flow.cuh -- the schedule of the data-flow launch of a smoothing call (flow_kernels.cuh) and its builder.
#pragma once

#include "flow_kernels.cuh"
#include "hierarchy.cuh"

#include <functional>
#include <memory>
#include <vector>

namespace b2g {

// The level's addressing on the host, as the schedule builder reads it, and the order of visits.
struct FlowLevel
{
    int n = 0;
    std::vector<int> posCell, cellPos;  // cell of a position, position of a cell
    std::vector<int> posRow, col;       // rows by position: their neighbours' cells (positions until prepare)
    void prepare();                     // cellPos, and col's positions into cells
    // The order of a visit: by colour where there are colours, else by cell; odd visits of a symmetric call run
    // it backwards. A row reads the neighbours before its cell in the order at the same visit, the others at the
    // visit before (-1: their initial value).
    bool symmetric = false;
    std::vector<int> colour;
    int versionRead(int q, int c, int cn) const
    {
        const int d = colour.empty() ? cn - c : colour[cn] - colour[c];
        return (symmetric && (q & 1) ? d > 0 : d < 0) ? q : q - 1;
    }
    bool crosses = false;               // more than one rank
};

// rank r's cells are [flowBegin(r), flowBegin(r + 1))
inline int flowBegin(int r, int n, int R) { return static_cast<int>((static_cast<long long>(r) * n + R - 1) / R); }
inline int flowRank(int c, int n, int R) { return static_cast<int>(static_cast<long long>(c) * R / n); }

constexpr size_t kFlowSmem = 220 * 1024;  // dynamic shared memory of a CTA: value slots and ring

// One rank's program.
struct RankProgram
{
    std::vector<k::FlowRec> rec;
    std::vector<unsigned char> meta;
    size_t nVal = 0;          // its values (flowValues)
    int slots = 1;            // value slots used (slot 0 is the zero)
    bool ok = true;
};

// A whole launch's program, ranks in order (the ranks' blobs and values follow one another).
struct FlowProgram
{
    std::vector<RankProgram> prog;
    int slots = 1;
    size_t nVal = 0;
    int nChunks = 0;
    // FlowSchedule::blob up to the ranks' meta blobs, which follow one another at metaAt
    std::vector<unsigned char> head;
    size_t blobBytes = 0, recAt = 0, metaAt = 0;
    // its device memory, the values of one matrix included
    size_t deviceBytes(size_t vb) const { return blobBytes + vb * nVal; }
};

// (`prepared` false: H.prepare() is left to the caller)
FlowLevel flowDownload(const LevelAddr& L, cudaStream_t s, bool prepared = true);
// (both set the level's order)
std::vector<int> flowSteps(FlowLevel& H, int nSweeps, bool symmetric, int R, int weight, int& nSteps);
std::vector<int> colourSteps(FlowLevel& H, const std::vector<int>& colourOf, int nColours, int nSweeps, bool symmetric,
                             int R, int weight, int& visits, int& nSteps);
// A program's hand-overs between ranks: values stored to a mailbox, values polled for; of the (cell, visit) pairs
// stored those that no rank polls for, and of those polled for the ones that nothing stores.
struct FlowHandOvers
{
    long long stored = 0, taken = 0, unread = 0, missing = 0;
};
FlowHandOvers flowHandOvers(const FlowLevel& H, const FlowProgram& F);
// The program for R ranks of items (visit q, cell c) at steps T[q * n + c], values of vb bytes; false when
// a rank's live values or chunks do not fit its shared memory, or a row is too long.
bool buildFlowProgram(FlowLevel& H, const std::vector<int>& T, int S, int nSteps, int R, size_t vb, FlowProgram& F);
// The same on the device, or null.
std::unique_ptr<FlowSchedule> buildFlow(FlowLevel& H, const std::vector<int>& T, int S, int nSteps, int R, size_t vb,
                                        cudaStream_t s);
// Programs of many levels side by side on the host's cores; ok is false where the level has
// none. The levels' addressing is freed on the way.
struct FlowBuild
{
    FlowLevel H;
    int S = 0, R = 0, weight = 4;  // S: visits of a cell, two a sweep when symmetric
    bool symmetric = false;
    size_t vb = 0;
    std::vector<int> T;
    int nSteps = 0;
    FlowProgram G;
    bool ok = false;
};
void buildFlowPrograms(std::vector<FlowBuild>& all);
// The batched form's launches: per job its level's sweeps on `ranks` CTAs, built once and kept on the level; flow
// is null when the level has none.
struct FlowJob
{
    LevelAddr* level;
    int nSweeps, ranks;
    size_t vb;
    const FlowSchedule* flow;
};
void flowsForBatch(std::vector<FlowJob>& jobs, cudaStream_t s);
// The batched launch (flow.cu): table = k::FlowArgs<T>[entries] on the device, blocks[i] = {entry, rank},
// caseOf[entry] its case. `remote`: some entry has more than one rank (a cooperative launch).
template <class T>
void launchFlowBatch(const void* table, const int2* blocks, int nBlocks, bool remote, const int* caseOf, const int* active,
                     cudaStream_t s);
// Runs body(i, worker) for i in [0, n) on the host's cores, `threads` at most, worker < kFlowThreads; the first exception is
// rethrown. Nested calls run on the calling thread.
constexpr int kFlowThreads = 16;
void flowParallel(int n, const std::function<void(int, int)>& body, int threads = kFlowThreads);
// The launches worth timing on a level of n cells.
struct FlowShape
{
    int ranks, weight;
};
std::vector<FlowShape> flowShapes(int n);
// The polls after which a wait of a launch gives up. The last rank may wait until the front has passed all
// others, nearly all of the launch's steps: at 0.45-0.8 us a step that is longer than kSpinLimit polls of shared
// memory (1.5 s, measured) from about 2 M steps on, a line of as many cells, say. kPollsPerStep polls take some
// 90 us. A limit set for a test is taken as it is.
constexpr long long kPollsPerStep = 1024;
inline long long flowSpinLimit(long long limit, const FlowSchedule& F)
{
    return limit == k::kSpinLimit ? limit + kPollsPerStep * F.nSteps : limit;
}
// Whether the device has room for `bytes` more of schedules: an eighth of its memory stays free of them, for the
// buffers that every form needs.
bool flowRoom(size_t bytes);
// whether a launch of that many ranks can be resident (one CTA per SM)
bool flowFits(int ranks);

}  // namespace b2g
