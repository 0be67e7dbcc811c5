// flow.cu -- the data-flow launch of a smoothing call (flow_kernels.cuh): its schedule on the device, its
// values per matrix, and its launch.

#include "flow.cuh"
#include "solver.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <set>
#include <system_error>
#include <thread>
#include <vector>

namespace b2g {
namespace {

template <class T>
void allowFlowSmem()
{
    static std::atomic<unsigned long long> done{0};  // one bit per device
    int dev = 0;
    B2G_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load() & bit) return;
    auto allow = [](const void* f) {
        B2G_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kFlowSmem)));
    };
    allow(reinterpret_cast<const void*>(&k::gsFlow<T, false, false>));
    allow(reinterpret_cast<const void*>(&k::gsFlow<T, false, true>));
    allow(reinterpret_cast<const void*>(&k::gsFlowBatch<T, false>));
    allow(reinterpret_cast<const void*>(&k::gsFlowBatch<T, true>));
    if constexpr (sizeof(T) == 4)
    {
        allow(reinterpret_cast<const void*>(&k::gsFlow<T, true, false>));
        allow(reinterpret_cast<const void*>(&k::gsFlow<T, true, true>));
    }
    done.fetch_or(bit);
}

// every live mesh, and through it every live matrix
std::mutex& g_meshesMu = *new std::mutex;  // (never destroyed: a mesh may go at the process's end)
std::set<Mesh*>& g_meshes = *new std::set<Mesh*>;

// What a mesh's schedules took is freed in each buffer's stream; the streams, to be waited for.
struct Dropped
{
    size_t bytes = 0;
    std::set<cudaStream_t> streams;
    template <class B>
    void take(B& b)
    {
        if (!b.p) return;
        bytes += b.bytes();
        streams.insert(b.s);
        b.release();
    }
    void take(FlowSchedule& F)
    {
        take(F.blob);
    }
};

// (g_meshesMu and M.use held)
void dropLocked(Mesh& M, Dropped& D)
{
    const size_t had = D.bytes;
    for (LevelAddr& L : M.lev)
    {
        for (auto it = L.pipe.begin(); it != L.pipe.end();)
        {
            if (it->second.flow) D.take(*it->second.flow);
            // (chosen anew without it)
            it = it->second.mode == 3 ? L.pipe.erase(it) : std::next(it);
        }
        for (auto& kv : L.flowBatch)
            if (kv.second) D.take(*kv.second);
        L.flowBatch.clear();
        for (auto& kv : L.flowSym)
            if (kv.second)
            {
                D.take(*kv.second);
                kv.second.reset();
            }
        for (auto& kv : L.mc.pipe)
            if (kv.second.flow)
            {
                D.take(*kv.second.flow);
                kv.second.flow.reset();
                kv.second.use = false;
            }
    }
    for (Matrix* A : M.matrices)
    {
        auto drop = [&](auto& flows) {
            for (auto& kv : flows)
            {
                D.take(kv.second.val);
                D.take(kv.second.mail);
                D.take(kv.second.ctl);
            }
            flows.clear();
        };
        drop(A->v64.flows);
        drop(A->v32.flows);
    }
    if (D.bytes == had) return;
    M.flowOff = true;
    ++M.flowEpoch;
}

void giveBack(const Dropped& D)
{
    for (cudaStream_t s : D.streams) B2G_CUDA(cudaStreamSynchronize(s));
    // (in one piece again for whatever is asked for next)
    if (D.bytes) B2G_CUDA(cudaMemPoolTrimTo(libraryPool(), 0));
}

}  // namespace

Mesh::Mesh()
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    g_meshes.insert(this);
}
Mesh::~Mesh()
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    g_meshes.erase(this);
}
void joinMesh(Matrix& A)
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    A.mesh->matrices.insert(&A);
}
void leaveMesh(Matrix& A)
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    // (a mesh destroyed before its matrix has left already)
    if (g_meshes.count(A.mesh)) A.mesh->matrices.erase(&A);
}

bool dropIdleFlows()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    Dropped D;
    return attempt([&] {
               std::lock_guard<std::mutex> lk(g_meshesMu);
               for (Mesh* M : g_meshes)
               {
                   if (M->device != dev || !M->use.try_lock()) continue;
                   std::lock_guard<std::shared_mutex> own(M->use, std::adopt_lock);
                   dropLocked(*M, D);
               }
               giveBack(D);
           }) &&
           D.bytes > 0;
}

size_t dropFlows(Mesh& M)
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    if (!M.use.try_lock()) return 0;
    std::lock_guard<std::shared_mutex> own(M.use, std::adopt_lock);
    Dropped D;
    dropLocked(M, D);
    return D.bytes;
}

size_t flowBytes(const Mesh& M)
{
    std::lock_guard<std::mutex> lk(g_meshesMu);
    size_t n = 0;
    for (const LevelAddr& L : M.lev)
    {
        for (const auto& kv : L.pipe)
            if (kv.second.flow) n += kv.second.flow->bytes();
        for (const auto& kv : L.flowBatch)
            if (kv.second) n += kv.second->bytes();
        for (const auto& kv : L.flowSym)
            if (kv.second) n += kv.second->bytes();
        for (const auto& kv : L.mc.pipe)
            if (kv.second.flow) n += kv.second.flow->bytes();
    }
    for (const Matrix* A : M.matrices)
    {
        for (const auto& kv : A->v64.flows) n += kv.second.val.bytes() + kv.second.mail.bytes();
        for (const auto& kv : A->v32.flows) n += kv.second.val.bytes() + kv.second.mail.bytes();
    }
    return n;
}

bool flowRoom(size_t bytes)
{
    size_t freeB = 0, total = 0;
    unsigned long long reserved = 0, used = 0;
    B2G_CUDA(cudaMemGetInfo(&freeB, &total));
    B2G_CUDA(cudaMemPoolGetAttribute(libraryPool(), cudaMemPoolAttrReservedMemCurrent, &reserved));
    B2G_CUDA(cudaMemPoolGetAttribute(libraryPool(), cudaMemPoolAttrUsedMemCurrent, &used));
    return freeB + (reserved - used) >= bytes + total / 8;
}

FlowLevel flowDownload(const LevelAddr& L, cudaStream_t s, bool prepared)
{
    FlowLevel H;
    H.n = L.nCells;
    auto get = [&](const DBuf<int>& from, std::vector<int>& to, size_t n) {
        to.resize(n);
        if (n) B2G_CUDA(cudaMemcpyAsync(to.data(), from.p, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    };
    get(L.gs.posCell, H.posCell, H.n);
    get(L.gs.posRow, H.posRow, static_cast<size_t>(H.n) + 1);
    get(L.gs.entColPos, H.col, 2 * static_cast<size_t>(L.nFaces));
    B2G_CUDA(cudaStreamSynchronize(s));
    if (prepared) H.prepare();
    return H;
}

static std::unique_ptr<FlowSchedule> uploadFlow(const FlowProgram& G, int nSteps, int R, cudaStream_t s);

std::unique_ptr<FlowSchedule> buildFlow(FlowLevel& H, const std::vector<int>& T, int S, int nSteps, int R, size_t vb,
                                        cudaStream_t s)
{
    FlowProgram G;
    if (!flowRoom(0) || !buildFlowProgram(H, T, S, nSteps, R, vb, G)) return nullptr;
    if (!flowRoom(G.deviceBytes(vb))) return nullptr;
    std::unique_ptr<FlowSchedule> F = uploadFlow(G, nSteps, R, s);
    B2G_CUDA(cudaStreamSynchronize(s));  // the host arrays go out of scope
    return F;
}

std::unique_ptr<FlowSchedule> uploadFlow(const FlowProgram& G, int nSteps, int R, cudaStream_t s)
{
    auto F = std::make_unique<FlowSchedule>();
    static std::atomic<long long> nextId{1};
    F->id = nextId++;
    F->ranks = R;
    F->nSteps = nSteps;
    F->slots = G.slots;
    F->nVal = static_cast<long long>(G.nVal);
    F->nChunks = G.nChunks;
    F->recAt = G.recAt;
    F->metaAt = G.metaAt;
    F->blob.alloc(G.blobBytes, s);
    auto put = [&](size_t at, const std::vector<unsigned char>& v) {
        if (!v.empty()) B2G_CUDA(cudaMemcpyAsync(F->blob.p + at, v.data(), v.size(), cudaMemcpyHostToDevice, s));
    };
    put(0, G.head);
    size_t at = G.metaAt;
    for (const RankProgram& P : G.prog)
    {
        put(at, P.meta);
        at += P.meta.size();
    }
    return F;
}

// Measured per smoothing call (FP64, graded boxes of 24 k and 1 M cells, all levels; 1 to 148 CTAs, weights 2
// and 4): a hand-over through L2 takes about four steps, so 4 beats 2 nearly everywhere; one CTA per SM is the
// fastest above 700 k cells, that or half as many down to 200 k, then about one per 1,000 to 4,000 cells.
std::vector<FlowShape> flowShapes(int n)
{
    const int sms = DeviceInfo::get().numSMs;
    std::vector<FlowShape> out;
    auto add = [&](int R, int w) {
        R = std::min(R, sms);
        if (R < 1 || R > n) return;
        if (R == 1) w = 1;
        for (const FlowShape& f : out)
            if (f.ranks == R && f.weight == w) return;
        out.push_back({R, w});
    };
    if (n >= 700000)
        add(sms, 4);
    else if (n >= 200000)
    {
        add(sms, 4);
        add(sms / 2, 4);
    }
    else
    {
        int r = 1;
        while (2 * r * 2000 <= n) r *= 2;
        add(r, 4);
        if (n >= 6000) add(2 * r, 4);
    }
    return out;
}

bool flowFits(int ranks)
{
    return ranks <= DeviceInfo::get().numSMs;
}

// A schedule's values on this matrix, refilled when the coefficients changed since (outside any capture).
template <class T>
const T* Matrix::flowValuesOf(int level, const FlowSchedule& F)
{
    VCycleData<T>& D = data<T>();
    auto& B = D.flows[F.id];
    if (B.gen != coefGen)
    {
        if (capturing) fail(B2G_ERR_STATE, "b2g: a smoothing schedule's values were not filled before the capture");
        B.val.ensure(static_cast<size_t>(std::max<long long>(F.nVal, 1)), stream);
        if (F.nChunks)
            k::flowValues<T><<<std::min(F.nChunks, 8192), 32 * k::kFlowTeam, 0, stream>>>(
                F.nChunks, F.rec(), F.meta(), mesh->lev[level].gs.posRow.p, D.coef[level].rowVal.p,
                D.coef[level].gsDiag.p, B.val.p);
        B2G_LAUNCH_CHECK();
        if (F.ranks > 1 && !B.mail.p)
        {
            B.mail.alloc(2 * sizeof(T) * static_cast<size_t>(mesh->lev[level].nCells), stream);
            B.mail.zero(stream);
            B.ctl.alloc(2, stream);
            B.ctl.zero(stream);
        }
        B.of = F.held;
        B.gen = coefGen;
    }
    return B.val.p;
}

void Matrix::forgetFlows()
{
    auto sweep = [](auto& flows) {
        for (auto it = flows.begin(); it != flows.end();)
            it = it->second.gen >= 0 && it->second.of.expired() ? flows.erase(it) : std::next(it);
    };
    sweep(v64.flows);
    sweep(v32.flows);
}

static int symRanks(int n) { return std::max(1, flowShapes(n).front().ranks / 2); }

// Whether this matrix has the schedule's values, filled here outside a capture; false when there is no memory
// for them, and the level then runs its other form (tried again with the next solve).
template <class T>
bool Matrix::flowReady(int level, const FlowSchedule& F, bool room)
{
    auto& flows = data<T>().flows;
    const auto it = flows.find(F.id);
    if (it != flows.end() && it->second.gen == coefGen) return true;
    if (capturing && it != flows.end() && it->second.refused == coefGen) return false;
    const bool have = it != flows.end() && it->second.val.p;  // (a refill, into the same buffer)
    if ((capturing || have || room || flowRoom(sizeof(T) * static_cast<size_t>(F.nVal))) && attempt([&] { flowValuesOf<T>(level, F); }))
        return true;
    if (capturing) fail(B2G_ERR_STATE, "b2g: a smoothing schedule's values were not filled before the capture");
    flows.erase(F.id);
    flows[F.id].refused = coefGen;
    return false;
}

template <class T>
k::FlowArgs<T> Matrix::flowArgs(int level, const FlowSchedule& F, T* psiL, const T* src)
{
    k::FlowArgs<T> a;
    a.chunkStart = F.chunkStart();
    a.rec = F.rec();
    a.meta = F.meta();
    a.val = flowValuesOf<T>(level, F);
    a.b = src;
    a.psi = psiL;
    const auto& B = data<T>().flows[F.id];
    a.mail = B.mail.p;
    a.ctl = B.ctl.p;
    a.ranks = F.ranks;
    a.slots = F.slots;
    a.spinLimit = flowSpinLimit(spinLimit, F);
    a.err = err.p;
    a.publish = publish;
    return a;
}

template <class T>
void Matrix::flowLaunch(int level, const FlowSchedule& F, T* psiL, const T* src, bool fma)
{
    allowFlowSmem<T>();
    const k::FlowArgs<T> a = flowArgs<T>(level, F, psiL, src);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(F.ranks));
    cfg.blockDim = dim3(static_cast<unsigned>(k::flowThreads(F.ranks > 1)));
    cfg.dynamicSmemBytes = kFlowSmem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = F.ranks > 1 ? 1 : 0;
    if constexpr (sizeof(T) == 4)
    {
        if (fma)
        {
            B2G_CUDA(F.ranks > 1 ? cudaLaunchKernelEx(&cfg, k::gsFlow<T, true, true>, a)
                                 : cudaLaunchKernelEx(&cfg, k::gsFlow<T, true, false>, a));
            ++launches;
            return;
        }
    }
    if (fma) fail(B2G_ERR_STATE, "b2g: the multicolour smoothing schedule is FP32 only");
    B2G_CUDA(F.ranks > 1 ? cudaLaunchKernelEx(&cfg, k::gsFlow<T, false, true>, a)
                         : cudaLaunchKernelEx(&cfg, k::gsFlow<T, false, false>, a));
    ++launches;
}

template <class T>
float Matrix::flowTime(int level, const FlowSchedule& F, T* psiL, const T* src, bool fma)
{
    return callTime([&] { flowLaunch<T>(level, F, psiL, src, fma); });
}

// nSweeps sweeps of `level` as one data-flow launch on `ranks` CTAs, whatever the tuned choice (for
// tests and tuning); false when the level has no such schedule. ms (may be null): a call's mean time.
template <class T>
bool Matrix::flowForced(int level, T* psiL, const T* src, int nSweeps, bool symmetric, int ranks, int weight, float* ms)
{
    if (ranks < 1 || weight < 1 || !flowFits(ranks)) return false;
    FlowLevel H = flowDownload(mesh->lev[level], stream);
    int nSteps = 0;
    const std::vector<int> steps = flowSteps(H, nSweeps, symmetric, ranks, weight, nSteps);
    std::unique_ptr<FlowSchedule> F = buildFlow(H, steps, symmetric ? 2 * nSweeps : nSweeps, nSteps, ranks, sizeof(T), stream);
    if (!F) return false;
    struct Drop
    {
        VCycleData<T>& D;
        long long id;
        ~Drop() { D.flows.erase(id); }
    } drop{data<T>(), F->id};
    flowLaunch<T>(level, *F, psiL, src, false);
    if (ms) *ms = flowTime<T>(level, *F, psiL, src);
    B2G_CUDA(cudaStreamSynchronize(stream));  // F is released on return
    checkDeviceError();
    return true;
}

// The symmetric sweeps' launch of `level`, kept where it beats the sweeps' own launches (null else, or when the
// level has no such schedule). Those are two walks a sweep and two vector moves; one walk is timed, for all,
// by the forward layout (the reversed one has the same depth), so that a level that takes the data flow never
// needs the reversed one. On half the CTAs of a forward call, where they hold the level: the walks of a
// symmetric call follow one another, so a step has a share of the items. Measured per call, half against as many
// (FP64, boxes of 151 k and 1 M cells, their levels): 0.37 and 0.50 ms on 152 k cells, 0.34 and 0.40 on 76 k, 0.84
// and 0.96 on 512 k, 0.67 and 0.72 on 64 k; 0.16 and 0.12 on 10 k. Outside any capture.
template <class T>
void Matrix::ensureSymFlow(int level, int nSweeps, FlowBuild* made)
{
    LevelAddr& L = mesh->lev[level];
    const int key = nSweeps * 16 + static_cast<int>(sizeof(T));
    if (L.flowSym.count(key)) return;
    std::unique_ptr<FlowSchedule>& kept = L.flowSym[key];
    if (nSweeps < 1 || L.nCells == 0 || mesh->flowOff) return;
    DBuf<T> x, b;
    if (!attempt([&] {
            x.alloc(nAlloc(level), stream);
            b.alloc(nAlloc(level), stream);
        }))
        return;
    x.zero(stream);
    b.zero(stream);
    const long long l0 = launches;
    const float msSweeps =
        2 * nSweeps * callTime([&] { gsLaunch<T>(L, data<T>().coef[level], x.p, b.p, nullptr, false); }, 1);
    FlowLevel H;
    const int forward = flowShapes(L.nCells).front().ranks;
    for (int ranks : {symRanks(L.nCells), forward})
    {
        std::unique_ptr<FlowSchedule> F;
        float ms = 0.f;
        const bool ran = attempt([&] {
            int nSteps = 0;
            if (made && ranks == made->R)
            {
                if (made->ok && flowRoom(made->G.deviceBytes(sizeof(T)))) F = uploadFlow(made->G, made->nSteps, ranks, stream);
                B2G_CUDA(cudaStreamSynchronize(stream));
            }
            else
            {
                if (H.n == 0) H = flowDownload(L, stream);
                const std::vector<int> steps = flowSteps(H, nSweeps, true, ranks, 4, nSteps);
                F = buildFlow(H, steps, 2 * nSweeps, nSteps, ranks, sizeof(T), stream);
            }
            if (F) ms = flowTime<T>(level, *F, x.p, b.p);
        });
        if (!F) continue;
        if (ran && ms < msSweeps)
            kept = std::move(F);
        else
            data<T>().flows.erase(F->id);
        break;
    }
    launches = l0;
    B2G_CUDA(cudaStreamSynchronize(stream));
}

// The symmetric sweeps' launches of {level, sweeps}, the missing schedules built side by side: a level's steps are one
// serial walk, which the other levels' work then hides.
template <class T>
void Matrix::ensureSymFlows(const std::vector<std::pair<int, int>>& wanted)
{
    std::vector<std::pair<int, int>> missing;
    for (const auto& w : wanted)
        if (!mesh->lev[w.first].flowSym.count(w.second * 16 + static_cast<int>(sizeof(T))) && mesh->lev[w.first].nCells &&
            std::find(missing.begin(), missing.end(), w) == missing.end())
            missing.push_back(w);
    std::vector<FlowBuild> made(missing.size());
    const bool side = !mesh->flowOff && attempt([&] {
        if (!flowRoom(0)) throw std::bad_alloc();
        for (size_t i = 0; i < missing.size(); ++i)
        {
            FlowBuild& b = made[i];
            b.H = flowDownload(mesh->lev[missing[i].first], stream, false);
            b.S = 2 * missing[i].second;
            b.symmetric = true;
            b.R = symRanks(b.H.n);
            b.vb = sizeof(T);
        }
        buildFlowPrograms(made);
    });
    for (size_t i = 0; i < missing.size(); ++i)
    {
        ensureSymFlow<T>(missing[i].first, missing[i].second, side ? &made[i] : nullptr);
        made[i] = FlowBuild();
    }
}

// nSweeps symmetric sweeps of `level` in one launch; false when they run as launches of their own
template <class T>
bool Matrix::symFlowSweeps(int level, T* psiL, const T* src, int nSweeps)
{
    if (!g_pipeline) return false;
    LevelAddr& L = mesh->lev[level];
    const int key = nSweeps * 16 + static_cast<int>(sizeof(T));
    auto it = L.flowSym.find(key);
    if (it == L.flowSym.end())
    {
        if (capturing) return false;
        ensureSymFlow<T>(level, nSweeps);
        it = L.flowSym.find(key);
    }
    if (!it->second || !flowReady<T>(level, *it->second)) return false;
    flowLaunch<T>(level, *it->second, psiL, src);
    return true;
}

// Before a capture: the values of every symmetric launch, for the current coefficients.
template <class T>
void Matrix::refreshSymFlows()
{
    for (int lv = 0; lv <= nLevels(); ++lv)
        for (auto& kv : mesh->lev[lv].flowSym)
            if (kv.second && kv.first % 16 == static_cast<int>(sizeof(T))) flowReady<T>(lv, *kv.second);
}

// The missing schedules go through three stages, a group of levels at a time: their addressing comes to the host, the
// programs are built on its cores, the result goes to the device. While one group is built, the one before goes up
// and the next one comes down.
void flowsForBatch(std::vector<FlowJob>& jobs, cudaStream_t s)
{
    constexpr long long kGroupItems = 4 << 20;  // items (cells times sweeps) of a group: some 0.4 GB of host memory
    auto keyOf = [](const FlowJob& j) { return std::pair<int, int>{j.nSweeps * 16 + static_cast<int>(j.vb), j.ranks}; };
    std::vector<size_t> missing;
    for (size_t i = 0; i < jobs.size(); ++i)
    {
        auto& have = jobs[i].level->flowBatch;
        if (have.count(keyOf(jobs[i]))) continue;
        have[keyOf(jobs[i])];  // (a level listed twice is built once)
        missing.push_back(i);
    }
    struct Group
    {
        std::vector<size_t> job;
        std::vector<FlowBuild> build;
    };
    size_t at = 0;
    // (no memory for a level, here and below: it has no schedule)
    auto fetch = [&] {
        // the levels' arrays side by side on the device, then one copy: some hundred small ones cost more than it
        Group g;
        DBuf<int> side;
        std::vector<int> host;
        size_t ints = 0;
        for (long long items = 0; at < missing.size() && items < kGroupItems; ++at)
        {
            const FlowJob& j = jobs[missing[at]];
            items += static_cast<long long>(j.level->nCells) * j.nSweeps;
            ints += 2 * static_cast<size_t>(j.level->nCells) + 1 + 2 * static_cast<size_t>(j.level->nFaces);
            FlowBuild b;
            b.S = j.nSweeps;
            b.R = j.ranks;
            b.vb = j.vb;
            b.H.n = j.level->nCells;
            g.job.push_back(missing[at]);
            g.build.push_back(std::move(b));
        }
        auto each = [&](auto&& array) {
            size_t from = 0;
            for (size_t i = 0; i < g.job.size(); ++i)
            {
                const LevelAddr& L = *jobs[g.job[i]].level;
                FlowLevel& H = g.build[i].H;
                array(L.gs.posCell, H.posCell, from, static_cast<size_t>(L.nCells));
                array(L.gs.posRow, H.posRow, from, static_cast<size_t>(L.nCells) + 1);
                array(L.gs.entColPos, H.col, from, 2 * static_cast<size_t>(L.nFaces));
            }
        };
        if (!g.job.empty() && (!flowRoom(sizeof(int) * ints) || !attempt([&] {
                side.alloc(ints, s);
                host.resize(ints);
                each([&](const DBuf<int>& from, std::vector<int>&, size_t& to, size_t n) {
                    if (n) B2G_CUDA(cudaMemcpyAsync(side.p + to, from.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
                    to += n;
                });
                B2G_CUDA(cudaMemcpyAsync(host.data(), side.p, sizeof(int) * ints, cudaMemcpyDeviceToHost, s));
                B2G_CUDA(cudaStreamSynchronize(s));
                each([&](const DBuf<int>&, std::vector<int>& to, size_t& from, size_t n) {
                    to.assign(host.begin() + from, host.begin() + from + n);
                    from += n;
                });
            })))
        {
            g.job.clear();
            g.build.clear();
        }
        return g;
    };
    auto upload = [&](const Group& g) {
        size_t need = 0;
        for (const FlowBuild& b : g.build)
            if (b.ok) need += b.G.deviceBytes(b.vb);
        const bool room = flowRoom(need);
        for (size_t i = 0; i < g.job.size(); ++i)
        {
            const FlowJob& j = jobs[g.job[i]];
            const FlowBuild& b = g.build[i];
            if (b.ok && (room || flowRoom(b.G.deviceBytes(b.vb))))
                attempt([&] { j.level->flowBatch[keyOf(j)] = uploadFlow(b.G, b.nSteps, b.R, s); });
        }
    };
    Group built, next = fetch();
    while (!next.job.empty() || at < missing.size())
    {
        Group now = std::move(next);
        auto build = [&] {
            if (!attempt([&] { buildFlowPrograms(now.build); }))
                for (FlowBuild& b : now.build) b.ok = false;
        };
        {
            struct Joined
            {
                std::thread t;
                ~Joined()
                {
                    if (t.joinable()) t.join();
                }
            } worker;
            try
            {
                worker.t = std::thread(build);
            }
            catch (const std::system_error&)
            {
                build();  // no more threads to be had
            }
            upload(built);
            next = fetch();
        }
        built = std::move(now);
    }
    upload(built);
    B2G_CUDA(cudaStreamSynchronize(s));
    for (FlowJob& j : jobs) j.flow = j.level->flowBatch[keyOf(j)].get();
}

template <class T>
void launchFlowBatch(const void* table, const int2* blocks, int nBlocks, bool remote, const int* caseOf, const int* active,
                     cudaStream_t s)
{
    allowFlowSmem<T>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(nBlocks));
    cfg.blockDim = dim3(static_cast<unsigned>(k::flowThreads(remote)));
    cfg.dynamicSmemBytes = kFlowSmem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = remote ? 1 : 0;
    const auto* t = static_cast<const k::FlowArgs<T>*>(table);
    B2G_CUDA(remote ? cudaLaunchKernelEx(&cfg, k::gsFlowBatch<T, true>, t, blocks, caseOf, active)
                    : cudaLaunchKernelEx(&cfg, k::gsFlowBatch<T, false>, t, blocks, caseOf, active));
}
template void launchFlowBatch<double>(const void*, const int2*, int, bool, const int*, const int*, cudaStream_t);
template void launchFlowBatch<float>(const void*, const int2*, int, bool, const int*, const int*, cudaStream_t);
template k::FlowArgs<double> Matrix::flowArgs<double>(int, const FlowSchedule&, double*, const double*);
template k::FlowArgs<float> Matrix::flowArgs<float>(int, const FlowSchedule&, float*, const float*);

template bool Matrix::flowForced<double>(int, double*, const double*, int, bool, int, int, float*);
template bool Matrix::flowForced<float>(int, float*, const float*, int, bool, int, int, float*);
template void Matrix::ensureSymFlow<double>(int, int, FlowBuild*);
template void Matrix::ensureSymFlow<float>(int, int, FlowBuild*);
template void Matrix::ensureSymFlows<double>(const std::vector<std::pair<int, int>>&);
template void Matrix::ensureSymFlows<float>(const std::vector<std::pair<int, int>>&);
template bool Matrix::symFlowSweeps<double>(int, double*, const double*, int);
template bool Matrix::symFlowSweeps<float>(int, float*, const float*, int);
template void Matrix::refreshSymFlows<double>();
template void Matrix::refreshSymFlows<float>();
template float Matrix::flowTime<double>(int, const FlowSchedule&, double*, const double*, bool);
template float Matrix::flowTime<float>(int, const FlowSchedule&, float*, const float*, bool);
template void Matrix::flowLaunch<double>(int, const FlowSchedule&, double*, const double*, bool);
template void Matrix::flowLaunch<float>(int, const FlowSchedule&, float*, const float*, bool);
template bool Matrix::flowReady<double>(int, const FlowSchedule&, bool);
template bool Matrix::flowReady<float>(int, const FlowSchedule&, bool);
template const double* Matrix::flowValuesOf<double>(int, const FlowSchedule&);
template const float* Matrix::flowValuesOf<float>(int, const FlowSchedule&);

}  // namespace b2g
