// flow_schedule.cu -- the schedule of the data-flow launch of a smoothing call (flow_kernels.cuh), built
// once per (level, sweep count, value type) on the host from the level's addressing. Host code only.
//
// Reference: the sweeps it reproduces are gaussSeidelSweeps, src/OpenFOAM/matrices/
// smooth_solver_cpp.cu:87-166 (forward only for GaussSeidel, :144), called nSweeps times per
// smoothing call by GaussSeidelSmoother::smooth (gamg_solver_cpp.cu:234-317).

#include "flow.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

namespace b2g {
namespace {

constexpr int kFlowChunkItems = 32 * k::kFlowTeam;      // items of a chunk, at most (the team's threads)
constexpr size_t kFlowChunkBytes = 28 * 1024;           // and its place in the ring

// scratch of one builder thread
struct RankScratch
{
    std::vector<int> localOf;  // cell -> ghost index of the rank at work, -1
};

// An item: [row width][position][visit][out: another rank reads it]
struct ItemRef
{
    unsigned long long key;
    int p() const { return static_cast<int>(key >> 7 & 0x7fffffffu); }
    int q() const { return static_cast<int>(key >> 1 & 0x3fu); }
    int w() const { return static_cast<int>(key >> 38); }
    bool out() const { return key & 1u; }
};
static_assert(k::kFlowMaxVisits < 64, "a visit has 6 bits of the key");
ItemRef itemRef(int p, int q, int w, bool out)
{
    return {static_cast<unsigned long long>(w) << 38 | static_cast<unsigned long long>(p) << 7 |
            static_cast<unsigned long long>(q) << 1 | (out ? 1u : 0u)};
}

// A step's items, those that another rank reads first (`apart`), then the longest rows, a counting sort; equal ones
// stay as they are: by visit, then by cell.
void sortStep(ItemRef* items, int m, bool apart, std::vector<ItemRef>& sorted)
{
    constexpr int kW = 256;  // (longer rows have no schedule: their order does not matter)
    int lo = kW, hi = 0;
    auto bucket = [&](const ItemRef& x) { return (apart && !x.out() ? kW : 0) + kW - 1 - std::min(x.w(), kW - 1); };
    if (m < 2) return;
    int count[2 * kW + 1];
    std::memset(count, 0, sizeof(count));
    for (int i = 0; i < m; ++i)
    {
        const int b = bucket(items[i]);
        ++count[b + 1];
        lo = std::min(lo, b);
        hi = std::max(hi, b);
    }
    if (lo == hi) return;
    for (int b = lo; b <= hi; ++b) count[b + 1] += count[b];
    sorted.resize(m);
    for (int i = 0; i < m; ++i) sorted[count[bucket(items[i])]++] = items[i];
    std::memcpy(items, sorted.data(), sizeof(ItemRef) * static_cast<size_t>(m));
}

void buildRank(const FlowLevel& H, const std::vector<int>& T, int S, int nSteps, int c0, int c1, size_t vb,
               RankScratch& X, RankProgram& P)
{
    const size_t n = static_cast<size_t>(H.n);
    const int nOwn = c1 - c0;
    if (X.localOf.size() < n) X.localOf.resize(n, -1);  // (every entry is -1 again when a rank is done)
    // the visits of a cell whose value another rank reads, a bit each
    std::vector<unsigned long long> exported(nOwn, 0);
    if (H.crosses)
        for (int c = c0; c < c1; ++c)
        {
            const int p = H.cellPos[c];
            for (int e = H.posRow[p]; e < H.posRow[p + 1]; ++e)
            {
                const int cn = H.col[e];
                if (cn >= c0 && cn < c1) continue;
                for (int q = 0; q < S; ++q)
                {
                    const int ver = H.versionRead(q, cn, c);
                    if (ver >= 0) exported[c - c0] |= 1ull << ver;
                }
            }
        }
    // items by step; of a step of several chunks those that another rank reads first, so that their way there
    // overlaps the step's other chunks; then the longest rows first, so that the slices of a chunk pad little
    std::vector<int> start(static_cast<size_t>(nSteps) + 1, 0);
    for (int q = 0; q < S; ++q)
        for (int c = c0; c < c1; ++c) ++start[T[q * n + c] + 1];
    for (int i = 0; i < nSteps; ++i) start[i + 1] += start[i];
    std::vector<ItemRef> items(static_cast<size_t>(S) * nOwn);
    {
        // a step's items of a visit by cell, in a colour's step by position: the order that coalesces better (a call
        // of two sweeps on 2 M cells 0.77 ms by position, 0.72 by cell; a multicolour solve of 4 M cells 39.8 ms by
        // position, 40.6 by cell)
        std::vector<int> own;
        if (!H.colour.empty())
        {
            for (int c = c0; c < c1; ++c) own.push_back(H.cellPos[c]);
            std::sort(own.begin(), own.end());
        }
        std::vector<int> cur(start.begin(), start.end() - 1);
        for (int q = 0; q < S; ++q)
            for (int i = 0; i < nOwn; ++i)
            {
                const int p = own.empty() ? H.cellPos[c0 + i] : own[i], c = H.posCell[p];
                items[cur[T[q * n + c]]++] = itemRef(p, q, H.posRow[p + 1] - H.posRow[p], exported[c - c0] >> q & 1u);
            }
    }
    struct Span
    {
        int a, b;
    };
    std::vector<Span> chunks;
    std::vector<ItemRef> sorted;
    for (int st = 0; st < nSteps; ++st)
    {
        const int a = start[st], b = start[st + 1];
        if (a == b) continue;
        sortStep(items.data() + a, b - a, b - a > kFlowChunkItems, sorted);
        // cut where the chunk is full: whole slices, its blobs and source within its share of the ring
        int from = a;
        size_t bytes = 64;
        for (int i = a; i < b; i += 32)
        {
            int w = 0;
            for (int x = i; x < std::min(b, i + 32); ++x) w = std::max(w, items[x].w());
            if (w > 252)
            {
                P.ok = false;
                return;
            }
            // slice: descriptors, diagonal, source, entries; about half of them a fetch or a ghost
            const size_t sl = 16 + 32 * (8 + 3 * vb) + static_cast<size_t>(32) * ((w + 3) & ~3) * (vb + 2 + 4);
            if (i > from && (i - from >= kFlowChunkItems || bytes + sl > kFlowChunkBytes))
            {
                chunks.push_back({from, i});
                from = i;
                bytes = 64;
            }
            bytes += sl;
        }
        chunks.push_back({from, b});
    }
    const int nCh = static_cast<int>(chunks.size());
    // first pass: each local value's last use, which is a last visit of its cell or of a neighbour (visits of a cell
    // come in order). Own cells are 0..nOwn-1, ghosts follow as they are met.
    std::vector<int> last(nOwn, -1), ghostCell;
    auto localId = [&](int cell) {
        if (cell >= c0 && cell < c1) return cell - c0;
        int g = X.localOf[cell];
        if (g < 0)
        {
            g = static_cast<int>(ghostCell.size());
            X.localOf[cell] = g;
            ghostCell.push_back(cell);
            last.push_back(-1);
        }
        return nOwn + g;
    };
    for (int j = 0; j < nCh; ++j)
        for (int i = chunks[j].a; i < chunks[j].b; ++i)
        {
            if (items[i].q() != S - 1) continue;
            const int p = items[i].p();
            last[H.posCell[p] - c0] = j;
            for (int e = H.posRow[p]; e < H.posRow[p + 1]; ++e) last[localId(H.col[e])] = j;
        }
    // second pass: slots (a value's from its first use to kFlowDepth chunks after its last), the
    // fetches of initial values, the ghosts' arrivals, the chunks' blobs
    const int nLoc = static_cast<int>(last.size());
    std::vector<int> slot(nLoc, 0), visit(nLoc, -2);
    std::vector<int> head(nCh, -1), nextOf(nLoc, -1);
    for (int v = 0; v < nLoc; ++v)
        if (last[v] >= 0)
        {
            nextOf[v] = head[last[v]];
            head[last[v]] = v;
        }
    std::vector<int> freeSlots;
    P.rec.resize(nCh);
    struct Pair
    {
        unsigned a, b;
    };
    // (about what the items take: records, and rows padded by a quarter)
    size_t rowEntries = 0;
    for (const ItemRef& it : items) rowEntries += static_cast<size_t>((it.w() + 3) & ~3);
    P.meta.reserve(16 * items.size() + rowEntries * 5 / 2 + 1024 * static_cast<size_t>(nCh));
    std::vector<Pair> fetch, halo;
    int width[kFlowChunkItems / 32 + 1], first[kFlowChunkItems / 32 + 1];
    long long valAt = 0;
    for (int j = 0; j < nCh; ++j)
    {
        if (j - k::kFlowDepth >= 0)
            for (int v = head[j - k::kFlowDepth]; v >= 0; v = nextOf[v]) freeSlots.push_back(slot[v]);
        auto give = [&](int v) {
            if (slot[v]) return;
            if (!freeSlots.empty())
            {
                slot[v] = freeSlots.back();
                freeSlots.pop_back();
            }
            else
                slot[v] = P.slots++;
        };
        const int a = chunks[j].a, b = chunks[j].b, m = b - a, nSl = (m + 31) / 32;
        int nEnt = 0;
        for (int s = 0; s < nSl; ++s)
        {
            // a multiple of 4 (the kernels' straight-line widths), at least 4
            int longest = 0;
            for (int i = 32 * s; i < std::min(m, 32 * s + 32); ++i) longest = std::max(longest, items[a + i].w());
            width[s] = std::max(4, (longest + 3) & ~3);
            first[s] = nEnt;
            nEnt += k::flowStride(m, s) * width[s];
        }
        fetch.clear();
        halo.clear();
        const size_t itemsAt = 16 * static_cast<size_t>(nSl), codesAt = itemsAt + 256 * static_cast<size_t>(nSl);
        const size_t fetchAt = codesAt + (2 * static_cast<size_t>(nEnt) + 15) / 16 * 16;
        const size_t at = P.meta.size();
        P.meta.resize(at + fetchAt, 0);
        unsigned short* codes = reinterpret_cast<unsigned short*>(P.meta.data() + at + codesAt);
        // (a chunk's values are read before its items write: every read first, then the writes)
        for (int i = 0; i < m; ++i)
        {
            const int p = items[a + i].p(), visitOf = items[a + i].q();
            const int c = H.posCell[p];
            // (code q of lane l at 4 * (stride * (q / 4) + l) + q % 4)
            const int jump = 4 * (k::flowStride(m, i / 32) - 1);
            unsigned short* to = codes + first[i / 32] + 4 * (i % 32);
            for (int e = H.posRow[p], q = 0; e < H.posRow[p + 1]; ++e, ++q, ++to)
            {
                const int cn = H.col[e];
                const int v = localId(cn);
                if (q && q % 4 == 0) to += jump;
                if (v < nOwn)
                {
                    if (!slot[v])
                    {
                        give(v);
                        fetch.push_back({static_cast<unsigned>(H.cellPos[cn]), static_cast<unsigned>(slot[v])});
                    }
                }
                else if (const int ver = H.versionRead(visitOf, c, cn); ver > visit[v])
                {
                    give(v);
                    if (ver < 0)
                        fetch.push_back({static_cast<unsigned>(H.cellPos[cn]), static_cast<unsigned>(slot[v])});
                    else
                        halo.push_back({static_cast<unsigned>(H.cellPos[cn]), static_cast<unsigned>(slot[v]) | static_cast<unsigned>(ver) << 16});
                    visit[v] = ver;
                }
                *to = static_cast<unsigned short>(slot[v]);
            }
        }
        for (int i = 0; i < m; ++i) give(H.posCell[items[a + i].p()] - c0);
        const size_t haloAt = fetchAt + (fetch.size() + 1) / 2 * 16;
        const size_t metaBytes = haloAt + (halo.size() + 1) / 2 * 16;
        const size_t valsAt = metaBytes + 64 * static_cast<size_t>(nSl) * vb, srcBytesAt = valsAt + nEnt * vb;
        // (offsets within a chunk count 8 bytes in 16 bits)
        if (P.slots > k::kFlowMaxSlots || vb * P.slots > kFlowSmem || srcBytesAt + 32 * static_cast<size_t>(nSl) * vb > 8 * 65535u ||
            fetch.size() > 65535u || halo.size() > 65535u)
        {
            P.ok = false;
            break;
        }
        P.meta.resize(at + metaBytes, 0);
        unsigned char* M = P.meta.data() + at;
        for (int s = 0; s < nSl; ++s)
        {
            k::FlowSlice h{};
            h.items8 = static_cast<unsigned short>((itemsAt + 256 * static_cast<size_t>(s)) / 8);
            h.codes8 = static_cast<unsigned short>((codesAt + 2 * static_cast<size_t>(first[s])) / 8);
            h.vals8 = static_cast<unsigned short>((valsAt + vb * static_cast<size_t>(first[s])) / 8);
            h.diag8 = static_cast<unsigned short>((metaBytes + 64 * static_cast<size_t>(s) * vb) / 8);
            h.src8 = static_cast<unsigned short>((srcBytesAt + 32 * static_cast<size_t>(s) * vb) / 8);
            h.width = static_cast<unsigned char>(width[s]);
            h.stride = static_cast<unsigned char>(k::flowStride(m, s));
            h.count = static_cast<unsigned char>(std::min(32, m - 32 * s));
            std::memcpy(M + 16 * static_cast<size_t>(s), &h, sizeof(h));
        }
        for (int i = 0; i < m; ++i)
        {
            const ItemRef& it = items[a + i];
            const int c = H.posCell[it.p()];
            const Pair w{static_cast<unsigned>(it.p()),
                         static_cast<unsigned>(slot[c - c0]) | static_cast<unsigned>(it.q()) << 16 |
                             (it.out() ? 0x40000000u : 0u) | (it.q() == S - 1 ? 0x80000000u : 0u)};
            std::memcpy(M + itemsAt + 8 * static_cast<size_t>(i), &w, 8);
        }
        if (!fetch.empty()) std::memcpy(M + fetchAt, fetch.data(), 8 * fetch.size());
        if (!halo.empty()) std::memcpy(M + haloAt, halo.data(), 8 * halo.size());
        k::FlowRec& r = P.rec[j];
        r.meta16 = static_cast<int>(at / 16);
        r.metaBytes = static_cast<int>(metaBytes);
        const long long nVal = 64LL * nSl + nEnt;
        r.val16 = static_cast<int>(valAt * static_cast<long long>(vb) / 16);
        r.valBytes = static_cast<int>(nVal * static_cast<long long>(vb));
        r.m = m;
        r.nSlices = nSl;
        r.items8 = static_cast<int>(itemsAt / 8);
        r.fetch8 = static_cast<int>(fetchAt / 8);
        r.halo8 = static_cast<int>(haloAt / 8);
        r.counts = static_cast<int>(static_cast<unsigned>(fetch.size()) | static_cast<unsigned>(halo.size()) << 16);
        valAt += nVal;
    }
    P.nVal = static_cast<size_t>(valAt);
    for (int g : ghostCell) X.localOf[g] = -1;
}

// Places a rank's chunks in a ring of `ring` bytes; false when two chunks do not fit together.
bool placeInRing(std::vector<k::FlowRec>& rec, size_t ring, size_t vb)
{
    std::vector<std::pair<size_t, size_t>> at(rec.size());
    size_t headAt = 0;
    for (size_t j = 0; j < rec.size(); ++j)
    {
        k::FlowRec& r = rec[j];
        const size_t need = static_cast<size_t>(r.metaBytes) + r.valBytes + 32 * static_cast<size_t>(r.nSlices) * vb;
        if (need > ring) return false;
        if (headAt + need > ring) headAt = 0;
        at[j] = {headAt, headAt + need};
        int freeAfter = static_cast<int>(j) - k::kFlowDepth;
        for (int i = static_cast<int>(j) - 1; i > freeAfter && i >= 0; --i)
            if (at[i].first < at[j].second && at[j].first < at[i].second)
            {
                freeAfter = i;
                break;
            }
        // chunk j is staged while chunk j - 1 is computed
        if (freeAfter > static_cast<int>(j) - 2) return false;
        r.ringOff = static_cast<int>(headAt);
        r.freeAfter = freeAfter;
        headAt += need;
    }
    return true;
}

}  // namespace

void FlowLevel::prepare()
{
    cellPos.resize(n);
    for (int p = 0; p < n; ++p) cellPos[posCell[p]] = p;
    constexpr int kBlock = 1 << 16;
    const int m = static_cast<int>(col.size());
    flowParallel((m + kBlock - 1) / kBlock, [&](int b, int) {
        for (int e = b * kBlock; e < std::min(m, (b + 1) * kBlock); ++e) col[e] = posCell[col[e]];
    });
}

void flowParallel(int n, const std::function<void(int, int)>& body, int threads)
{
    // a loop within a loop runs on its own thread: the outer one has the cores
    static thread_local bool inside = false;
    const int hw = static_cast<int>(std::max(1u, std::thread::hardware_concurrency()));
    const int nt = inside ? 1 : std::min({n, hw, kFlowThreads, threads});
    std::atomic<int> next{0};
    std::vector<std::exception_ptr> bad(std::max(nt, 1));
    auto work = [&](int w) {
        const bool was = inside;
        inside = true;
        try
        {
            for (int i = next++; i < n; i = next++) body(i, w);
        }
        catch (...)
        {
            bad[w] = std::current_exception();
            next = n;
        }
        inside = was;
    };
    std::vector<std::thread> th;
    try
    {
        for (int w = 1; w < nt; ++w) th.emplace_back(work, w);
    }
    catch (...)
    {
        // no more threads to be had: the ones that started, and this one, do the work
    }
    work(0);
    for (auto& x : th) x.join();
    for (auto& e : bad)
        if (e) std::rethrow_exception(e);
}

// T_s(c) of every item (flow_kernels.cuh): the combined DAG of pipe_kernels.cuh with `weight` steps
// across a face between two ranks.
//
// Symmetric sweeps (gaussSeidelSweeps' symmetric variant) visit a cell twice a sweep, forward then back.
// The backward walk's bPrime is the source less the terms of the faces the cell is the neighbour of, in face
// order, with the forward values, and the walk subtracts its own faces' terms ascending: the row's terms in
// the row's order again. So a backward visit q is the same row reading its lower neighbours at visit q - 1
// and its upper ones at visit q.
std::vector<int> flowSteps(FlowLevel& H, int nSweeps, bool symmetric, int R, int weight, int& nSteps)
{
    const int S = symmetric ? 2 * nSweeps : nSweeps;
    const size_t n = static_cast<size_t>(H.n);
    H.symmetric = symmetric;
    H.colour.clear();
    std::vector<int> T(static_cast<size_t>(S) * n, 0);
    nSteps = 0;
    for (int s = 0; s < S; ++s)
    {
        int* cur = T.data() + s * n;
        const int* prev = s > 0 ? T.data() + (s - 1) * n : nullptr;
        const bool back = symmetric && (s & 1);
        // cells in the walk's order: each neighbour the walk has passed is final at this visit
        for (int i = 0; i < R; ++i)
        {
            const int r = back ? R - 1 - i : i;
            const int c0 = flowBegin(r, H.n, R), c1 = flowBegin(r + 1, H.n, R);
            for (int x = c0; x < c1; ++x)
            {
                const int c = back ? c1 - 1 - (x - c0) : x, p = H.cellPos[c];
                int t = prev ? prev[c] + 1 : 0;
                for (int e = H.posRow[p]; e < H.posRow[p + 1]; ++e)
                {
                    const int o = H.col[e], w = o < c0 || o >= c1 ? weight : 1;
                    if ((o < c) != back) t = std::max(t, cur[o] + w);
                    else if (prev) t = std::max(t, prev[o] + w);
                }
                cur[c] = t;
                nSteps = std::max(nSteps, t + 1);
            }
        }
    }
    return T;
}

// The multicolour smoother's sweeps as steps on R ranks. The colours are an order of visits like the exact
// sweeps' cell order, so an item runs one step after the last visit it reads, `weight` steps after one of another
// rank: only the cells near a rank's border wait for a hand-over, the others run ahead into the next colours.
// Every row still reads its neighbours of earlier colours at this visit and the others at the one before, as the
// colour-by-colour sweep does. Symmetric sweeps visit the colours forward then back, each cell twice a sweep.
// Empty when a cell has no colour.
std::vector<int> colourSteps(FlowLevel& H, const std::vector<int>& colourOf, int nColours, int nSweeps, bool symmetric,
                             int R, int weight, int& visits, int& nSteps)
{
    const int n = H.n;
    H.symmetric = symmetric;
    H.colour = colourOf;
    std::vector<int> byColour(n), start(static_cast<size_t>(nColours) + 1, 0);
    for (int c = 0; c < n; ++c)
    {
        if (colourOf[c] < 0 || colourOf[c] >= nColours) return {};
        ++start[colourOf[c] + 1];
    }
    for (int k = 0; k < nColours; ++k) start[k + 1] += start[k];
    {
        std::vector<int> at(start.begin(), start.end() - 1);
        for (int c = 0; c < n; ++c) byColour[at[colourOf[c]]++] = c;
    }
    visits = symmetric ? 2 * nSweeps : nSweeps;
    std::vector<int> rank(R > 1 ? n : 0);
    for (size_t c = 0; c < rank.size(); ++c) rank[c] = flowRank(static_cast<int>(c), n, R);
    std::vector<int> T(static_cast<size_t>(visits) * n);
    for (int v = 0; v < visits; ++v)
    {
        int* cur = T.data() + static_cast<size_t>(v) * n;
        const int* prev = v > 0 ? cur - n : nullptr;
        const bool back = symmetric && (v & 1);
        for (int i = 0; i < nColours; ++i)
        {
            const int k = back ? nColours - 1 - i : i;
            // a colour's cells side by side: none reads another
            constexpr int kBlock = 16384;
            const int from = start[k], count = start[k + 1] - from;
            flowParallel((count + kBlock - 1) / kBlock, [&](int block, int) {
                const int end = std::min(count, (block + 1) * kBlock);
                for (int j = block * kBlock; j < end; ++j)
                {
                    const int c = byColour[from + j], p = H.cellPos[c];
                    int t = prev ? prev[c] + 1 : 0;
                    for (int e = H.posRow[p]; e < H.posRow[p + 1]; ++e)
                    {
                        const int o = H.col[e];
                        const bool earlier = back ? colourOf[o] > k : colourOf[o] < k;
                        if (!earlier && !prev) continue;
                        t = std::max(t, (earlier ? cur[o] : prev[o]) + (R > 1 && rank[o] != rank[c] ? weight : 1));
                    }
                    cur[c] = t;
                }
            });
        }
    }
    nSteps = T.empty() ? 0 : *std::max_element(T.begin(), T.end()) + 1;
    return T;
}

namespace {

bool startFlowProgram(FlowLevel& H, int S, int R, FlowProgram& F)
{
    if (H.n == 0 || R < 1 || R > H.n || S < 1 || S > k::kFlowMaxVisits) return false;
    H.crosses = R > 1;
    F.prog.clear();
    F.prog.resize(R);
    return true;
}

// The ranks' programs as one: their common slots, their places in the ring, the blob.
bool finishFlowProgram(int R, size_t vb, FlowProgram& F)
{
    F.slots = 1;
    size_t metaBytes = 0, chunks = 0;
    F.nVal = 0;
    for (const RankProgram& P : F.prog)
    {
        if (!P.ok) return false;
        F.slots = std::max(F.slots, P.slots);
        metaBytes += P.meta.size();
        F.nVal += P.nVal;
        chunks += P.rec.size();
    }
    // the ring holds three chunks at least: one computed, one loaded by the other team, one on its way
    const size_t ringAt = k::flowRingAt(F.slots, vb);
    size_t chunk = 0;
    for (const RankProgram& P : F.prog)
        for (const k::FlowRec& r : P.rec)
            chunk = std::max(chunk, static_cast<size_t>(r.metaBytes) + r.valBytes + 32 * static_cast<size_t>(r.nSlices) * vb);
    if (ringAt + 3 * chunk > kFlowSmem) return false;
    if (metaBytes / 16 > 0x7fffffffull || F.nVal * vb / 16 > 0x7fffffffull || chunks > 0x7fffffffull) return false;
    for (RankProgram& P : F.prog)
        if (!placeInRing(P.rec, kFlowSmem - ringAt, vb)) return false;
    F.nChunks = static_cast<int>(chunks);
    F.recAt = (sizeof(int) * (static_cast<size_t>(R) + 1) + 15) / 16 * 16;
    F.metaAt = F.recAt + sizeof(k::FlowRec) * chunks;
    F.blobBytes = F.metaAt + metaBytes;
    F.head.assign(F.metaAt, 0);
    size_t chunkAt = 0, metaAt = 0, valAt = 0;
    for (int r = 0; r < R; ++r)
    {
        const RankProgram& P = F.prog[r];
        k::FlowRec* to = reinterpret_cast<k::FlowRec*>(F.head.data() + F.recAt) + chunkAt;
        for (k::FlowRec x : P.rec)
        {
            x.meta16 += static_cast<int>(metaAt / 16);
            x.val16 += static_cast<int>(valAt * vb / 16);
            *to++ = x;
        }
        chunkAt += P.rec.size();
        reinterpret_cast<int*>(F.head.data())[r + 1] = static_cast<int>(chunkAt);
        metaAt += P.meta.size();
        valAt += P.nVal;
    }
    return true;
}

}  // namespace

bool buildFlowProgram(FlowLevel& H, const std::vector<int>& T, int S, int nSteps, int R, size_t vb, FlowProgram& F)
{
    if (!startFlowProgram(H, S, R, F)) return false;
    std::vector<RankScratch> scratch(kFlowThreads);
    // (a thread takes some 30 us to start, an item 0.2 us to place)
    const int threads = 1 + static_cast<int>(static_cast<long long>(H.n) * S / 8192);
    flowParallel(R, [&](int r, int w) {
        buildRank(H, T, S, nSteps, flowBegin(r, H.n, R), flowBegin(r + 1, H.n, R), vb, scratch[w], F.prog[r]);
    }, threads);
    return finishFlowProgram(R, vb, F);
}

void buildFlowPrograms(std::vector<FlowBuild>& all)
{
    const int n = static_cast<int>(all.size());
    // the largest first; then all their ranks, one list, so that a large level's ranks are shared out too
    std::vector<int> order(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int x, int y) {
        return static_cast<long long>(all[x].H.n) * all[x].S > static_cast<long long>(all[y].H.n) * all[y].S;
    });
    flowParallel(n, [&](int i, int) {
        FlowBuild& b = all[order[i]];
        b.ok = attempt([&] {
            b.H.prepare();
            b.T = flowSteps(b.H, b.symmetric ? b.S / 2 : b.S, b.symmetric, b.R, b.weight, b.nSteps);
        }) && startFlowProgram(b.H, b.S, b.R, b.G);
    });
    std::vector<std::pair<int, int>> ranks;
    for (int i : order)
        if (all[i].ok)
            for (int r = 0; r < all[i].R; ++r) ranks.push_back({i, r});
    std::vector<RankScratch> scratch(kFlowThreads);
    flowParallel(static_cast<int>(ranks.size()), [&](int i, int w) {
        FlowBuild& b = all[ranks[i].first];
        RankProgram& P = b.G.prog[ranks[i].second];
        const int r = ranks[i].second;
        if (!attempt([&] {
                buildRank(b.H, b.T, b.S, b.nSteps, flowBegin(r, b.H.n, b.R), flowBegin(r + 1, b.H.n, b.R), b.vb, scratch[w], P);
            }))
        {
            P.ok = false;
            scratch[w].localOf.clear();
        }
    });
    flowParallel(n, [&](int i, int) {
        FlowBuild& b = all[i];
        if (b.ok) b.ok = attempt([&] { b.ok = finishFlowProgram(b.R, b.vb, b.G); }) && b.ok;
        b.T = std::vector<int>();
        b.H = FlowLevel();
    });
}

// Every hand-over of a program, replayed in step order.
FlowHandOvers flowHandOvers(const FlowLevel& H, const FlowProgram& F)
{
    FlowHandOvers out;
    std::vector<unsigned long long> stored(H.n, 0), taken(H.n, 0);
    for (const RankProgram& P : F.prog)
        for (const k::FlowRec& r : P.rec)
        {
            const unsigned char* M = P.meta.data() + 16 * static_cast<size_t>(r.meta16);
            unsigned w[2];
            for (int i = 0; i < r.m; ++i)
            {
                std::memcpy(w, M + 8 * (static_cast<size_t>(r.items8) + i), 8);
                if (!(w[1] & 0x40000000u)) continue;
                ++out.stored;
                stored[w[0]] |= 1ull << (w[1] >> 16 & 0x3f);
            }
            for (unsigned i = 0; i < static_cast<unsigned>(r.counts) >> 16; ++i)
            {
                std::memcpy(w, M + 8 * (static_cast<size_t>(r.halo8) + i), 8);
                ++out.taken;
                taken[w[0]] |= 1ull << (w[1] >> 16);
            }
        }
    for (int p = 0; p < H.n; ++p)
        for (int q = 0; q < 64; ++q)
        {
            if (stored[p] & ~taken[p] & 1ull << q) ++out.unread;
            if (taken[p] & ~stored[p] & 1ull << q) ++out.missing;
        }
    return out;
}

}  // namespace b2g
