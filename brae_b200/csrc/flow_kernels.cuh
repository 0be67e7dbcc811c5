// flow_kernels.cuh -- every sweep of one Gauss-Seidel smoothing call in ONE launch, as a data flow
// between CTAs. Bit for bit the sequential sweeps of smooth_solver_cpp.cu:87-166, sweep after sweep:
// every row reads the operands the sequential sweeps give it and rounds in the same order.
//
// THE ORDER. Item (s, c) -- cell c in sweep s -- has a step T_s(c) of the combined DAG of
// pipe_kernels.cuh; the cells are split into R contiguous ranges ("ranks"), one persistent CTA each. A
// face between two ranks counts `weight` steps instead of one, so a value that crosses ranks is
// scheduled that many steps ahead of its first reader and its way through L2 overlaps the steps
// between. A rank runs its items step by step, the items of a step in "chunks"; a chunk of a rank may
// run once the rank's earlier chunks are done and the values of other ranks it reads have arrived.
// Nothing else is waited for: no grid-wide step, no progress words.
//
// VALUES live in shared-memory slots, recycled: a cell of the rank, or of another rank that it reads
// (a "ghost"), holds a slot from its first use to its last. A level of any size fits, since only the
// cells around the moving front are live. A slot is given to another cell kFlowDepth chunks after its
// last use at the earliest, so staging up to kFlowDepth chunks ahead never overwrites a live value.
//
// HAND-OFF BETWEEN RANKS. An item that another rank reads stores {value, tag} to its cell's mailbox
// in global memory with ONE 16-byte (FP32: 8-byte) store; the tag names the launch and the sweep, so
// no flag, release or reset goes with it. The reader's halo warps poll the mailbox until the tag is
// there and put the value into the ghost's slot. One mailbox per cell is enough, and ghosts may be
// written as soon as they arrive: version s+1 of a cell exists only after every reader of version s
// has run -- its upper neighbours' sweep-s items and its lower neighbours' sweep-(s+1) items, all of
// which (s+1, c) reads -- and a reader runs only after its own halo warp took version s. That orders the
// stores of versions that another rank reads, and only those are stored: a symmetric order has versions that
// nobody elsewhere reads (the last colour's forward visit, say), whose store could land after the next
// version's, from the other team, and hide it from its reader for good.
// The same argument covers psi itself: the initial values are fetched from global psi just before
// their first use and the last sweep writes there, and a cell's last write comes after every reader of
// its initial value.
//
// ROLES. 2 x TW compute warps in two teams that take the chunks in turn: while one computes chunk j,
// the other loads chunk j+1's coefficients, codes, source, diagonal and its reciprocal from shared memory
// into registers, so from one chunk to the next there are only the value gathers, the row's arithmetic, the
// division and a barrier between the two teams. A chunk has at most a team's threads of items; a step with
// more is several chunks. A producer warp keeps bulk copies of the
// chunks ahead in flight into a shared-memory ring (placed by the schedule). A gather warp brings each
// chunk's source values and initial values (cp.async). Halo warps, chunk j by warp j mod NH, poll the
// mailboxes. What these warps bring is told by one mbarrier per chunk in flight and kind, the copies of the
// gather warp arriving on it themselves.
//
// BOUND. Neither bytes nor arithmetic: the chain of chunks. About 850 cycles a chunk (clock stamps, FP64 levels
// of 88 to 24 k cells): a team's row 440-580, its barrier to the other 300 with the slowest warp's lag; and a
// team's own loop (barrier, row, stores 150, the next chunk's wait and load 700) is about two of those. With a
// release-acquire counter in place of the mbarriers and the gather warp waiting for its copies: 24 k cells
// 9.38 -> 8.97 ms a solve, 1 M 42.6 -> 41.7, 4 M (two iterations) 14.7 -> 13.8, a batch of 24 48.1 -> 44.4.
//
// LIMITS. Every wait has an iteration limit; when one runs out the error word and the CTA's stop word are
// set and the launch ends with an error. From then on no chunk counts as consumed (a chunk counts only while
// the stop word is clear, behind the barrier that every warp of its team has passed: so every wait for it,
// the gather warp's and the halo warp's parts included, ended well). Nothing in the ring is staged over what
// any role may still read, at most the chunks already allowed are issued, and the producer waits for every
// copy it has issued before the CTA ends. All CTAs of a launch with ranks are resident together (a
// cooperative launch).
#pragma once

#include "b2g_common.cuh"
#include "gs_kernels.cuh"

namespace b2g {
namespace k {

constexpr int kFlowDepth = 8;     // chunks in flight ahead of the consumed one, at most
constexpr int kFlowTeam = 4;      // TW: warps of a compute team
constexpr int kFlowHalo = 4;      // NH: halo warps of a launch with more than one rank
// row entries a thread holds in registers (the rest come from the ring, four at a time): as many as fit
// beside the gathered values without spilling at the launch's register count
constexpr int kFlowK = 16;
constexpr int kFlowMaxSlots = 65535;  // a slot's number has 16 bits
constexpr int kFlowMaxVisits = 63;  // visits of a cell in one call (the tag's low 6 bits)

// A chunk's record, three int4. Offsets within a chunk count 8 bytes from its place in the ring.
struct FlowRec
{
    int meta16, metaBytes, ringOff, freeAfter;  // its meta blob (16-byte units), its place in the ring,
                                                // the chunk that must be consumed before it is staged
    int val16, valBytes, m, nSlices;            // its values; items; slices of 32 items
    int items8, fetch8, halo8, counts;          // its items, fetches and halo entries; nFetch | nHalo << 16
};

// The meta blob: [slices: nSl x 16 bytes (FlowSlice)][items: 32 nSl x {position, slot word}][codes][fetches: nF x
// {position, slot}][halo: nH x {position, slot | visit << 16}], each 16-byte aligned; the value blob
// follows it in the ring: [{diagonal, its reciprocal}: 32 nSl][coefficients]; then the source: 32 nSl. A slot
// word is slot | visit << 16 | export << 30 | last << 31. Entries are sliced ELL in groups a lane reads with one load: four
// codes (group g of lane l at stride * g + l, the stride being the slice's items rounded up to 8), two FP64 or
// four FP32 coefficients; a slice's width is a multiple of 4. Codes are slots; padding reads slot 0 (a zero) with coefficient zero, which leaves a sum as it is bit for bit.
struct FlowSlice
{
    unsigned short items8, codes8, vals8, diag8, src8;
    unsigned char width, stride, count, pad[3];
};
static_assert(sizeof(FlowRec) == 48 && sizeof(FlowSlice) == 16, "the kernels read these as int4");
__host__ __device__ inline int flowStride(int m, int slice)
{
    const int left = m - 32 * slice;
    return left >= 32 ? 32 : (left + 7) & ~7;
}

template <class T>
struct FlowArgs
{
    const int* __restrict__ chunkStart;         // [ranks + 1]
    const int4* __restrict__ rec;               // [chunks][3]
    const unsigned char* __restrict__ meta;
    const T* __restrict__ val;                  // per chunk [{diagonal, reciprocal}: 32 nSl][coefficients]
    const T* __restrict__ b;                    // by position
    T* psi;                                     // by position
    void* mail;                                 // {value, tag} by position
    unsigned* ctl;                              // [0] the launches so far, [1] ranks that have finished
                                                // (null: one rank)
    int ranks;
    int slots;                                  // value slots (the ring follows them)
    long long spinLimit;
    int* err;
    int publish;                                // 0: no rank stores to its mailboxes (a test of the waits)
};

__host__ __device__ constexpr size_t flowRingAt(int slots, size_t valueBytes)
{
    return (valueBytes * static_cast<size_t>(slots) + 127) / 128 * 128;
}

__device__ __forceinline__ void mailSt(double* mail, int pos, double v, unsigned tag)
{
    const unsigned long long lo = static_cast<unsigned long long>(__double_as_longlong(v));
    const unsigned long long hi = tag;
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(mail + 2 * static_cast<size_t>(pos)),
                 "l"(lo), "l"(hi)
                 : "memory");
}
__device__ __forceinline__ void mailSt(float* mail, int pos, float v, unsigned tag)
{
    const unsigned long long w = static_cast<unsigned long long>(tag) << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(mail + 2 * static_cast<size_t>(pos)), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned mailLd(const double* mail, unsigned pos, double& v)
{
    unsigned long long lo, hi;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(lo), "=l"(hi)
                 : "l"(mail + 2 * static_cast<size_t>(pos))
                 : "memory");
    v = __longlong_as_double(static_cast<long long>(lo));
    return static_cast<unsigned>(hi);
}
__device__ __forceinline__ unsigned mailLd(const float* mail, unsigned pos, float& v)
{
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(mail + 2 * static_cast<size_t>(pos)) : "memory");
    v = __uint_as_float(static_cast<unsigned>(w));
    return static_cast<unsigned>(w >> 32);
}

// a / d, correctly rounded, given r = the correctly rounded 1 / d (0 where the quick form does not
// apply). Markstein's method (IBM J. Res. Dev. 34, 1990): a quotient within one unit in the last place,
// corrected by its exact remainder times r, is the rounded quotient; the product a r may be a little
// further off, so it is corrected twice. Holds while nothing under- or overflows: both operands'
// exponents are checked, others take the division itself. On the chain of every row: five dependent
// operations in place of about 130 cycles.
__device__ __forceinline__ bool flowExpOk(double a, int half)
{
    return (static_cast<unsigned>(__double2hiint(a)) & 0x7ff00000u) - (static_cast<unsigned>(1023 - half) << 20) <=
           static_cast<unsigned>(2 * half) << 20;
}
__device__ __forceinline__ bool flowExpOk(float a, int half)
{
    return (__float_as_uint(a) & 0x7f800000u) - (static_cast<unsigned>(127 - half) << 23) <= static_cast<unsigned>(2 * half) << 23;
}
__device__ __forceinline__ double flowRcp(double d) { return flowExpOk(d, 500) ? __drcp_rn(d) : 0.0; }
__device__ __forceinline__ float flowRcp(float d) { return flowExpOk(d, 60) ? __frcp_rn(d) : 0.0f; }
// the division itself, out of line: rare, and its registers stay off the row's
static __device__ __noinline__ double flowDivSlow(double a, double d, double r)
{
    return r != 0.0 && a == 0.0 ? __dmul_rn(a, r) : __ddiv_rn(a, d);
}
static __device__ __noinline__ float flowDivSlow(float a, float d, float r)
{
    return r != 0.0f && a == 0.0f ? __fmul_rn(a, r) : __fdiv_rn(a, d);
}
__device__ __forceinline__ double flowDiv(double a, double d, double r)
{
    double q = __dmul_rn(a, r);
    q = __fma_rn(__fma_rn(-q, d, a), r, q);
    q = __fma_rn(__fma_rn(-q, d, a), r, q);
    return flowExpOk(a, 400) && __double2hiint(r) != 0 ? q : flowDivSlow(a, d, r);
}
__device__ __forceinline__ float flowDiv(float a, float d, float r)
{
    float q = __fmul_rn(a, r);
    q = __fmaf_rn(__fmaf_rn(-q, d, a), r, q);
    q = __fmaf_rn(__fmaf_rn(-q, d, a), r, q);
    return flowExpOk(a, 60) && r != 0.0f ? q : flowDivSlow(a, d, r);
}

// one term of a row: the exact sweeps subtract the rounded product; the multicolour smoother (kFma)
// folds it in one fused multiply-add, as its colour-by-colour kernels do
template <bool kFma>
__device__ __forceinline__ double flowTerm(double acc, double v, double x)
{
    return kFma ? __fma_rn(-v, x, acc) : subRn(acc, mulRn(v, x));
}
template <bool kFma>
__device__ __forceinline__ float flowTerm(float acc, float v, float x)
{
    return kFma ? __fmaf_rn(-v, x, acc) : subRn(acc, mulRn(v, x));
}

// the launch's shared control words
struct FlowShared
{
    unsigned long long full[kFlowDepth];    // a chunk's bulk copies have landed
    unsigned long long staged[kFlowDepth];  // and its source and initial values (the gather warp's lanes)
    unsigned long long halo[kFlowDepth];    // and the values of other ranks (its halo warp)
    int4 rec[kFlowDepth][3];
    uint2 place[kFlowDepth];               // a chunk's shared address and its slices
    unsigned consumed;                     // chunks consumed
    unsigned stop;                         // a wait gave up
};

// false when the launch is stopping
template <class Ready>
__device__ __forceinline__ bool flowWait(FlowShared& S, int* err, long long limit, Ready&& ready)
{
    long long it = 0;
    while (!ready())
    {
        ++it;
        if ((it & 63) == 0 && *reinterpret_cast<volatile unsigned*>(&S.stop)) return false;
        if ((it & kErrPollMask) == 0 && errSet(err))
        {
            *reinterpret_cast<volatile unsigned*>(&S.stop) = 1;
            return false;
        }
        if (it > limit)
        {
            atomicExch(err, 1);
            *reinterpret_cast<volatile unsigned*>(&S.stop) = 1;
            return false;
        }
    }
    return true;
}

// mbarTryWait without its wait: asked again by the caller
__device__ __forceinline__ bool mbarTestWait(unsigned long long* bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(smemAddr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ int4 lds128(unsigned a)
{
    int4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(unsigned a)
{
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void ldsPair(unsigned a, double& x, double& y)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a));
}
__device__ __forceinline__ void ldsPair(unsigned a, float& x, float& y)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(a));
}

// A thread's row, loaded ahead. Everything that does not depend on psi is done at the load, so that the
// chain from barrier to barrier is the gathers, the sum, the division and the store.
template <class T, int K>
struct FlowRow
{
    int w;             // the slice's entries (a multiple of 4, the same for the warp); -1: no slice for this warp
    bool has;          // this lane has an item
    unsigned slotWord, pos, out;  // out: the shared address of its slot
    unsigned vA, cA, vS, cS;      // entry 0's shared addresses and the distance to the next
    T b, d, r;
    T v[K];
    unsigned x[K];     // the shared addresses of its values
};

// entries q..q+3 of a lane: coefficients and codes
__device__ __forceinline__ void flowEntries(unsigned vA, unsigned vS, unsigned cA, unsigned cS, int q, double* v, unsigned* c)
{
    ldsPair(vA + vS * (q / 2), v[0], v[1]);
    ldsPair(vA + vS * (q / 2 + 1), v[2], v[3]);
    const uint2 w = lds64(cA + cS * (q / 4));
    c[0] = w.x & 0xffffu; c[1] = w.x >> 16; c[2] = w.y & 0xffffu; c[3] = w.y >> 16;
}
__device__ __forceinline__ void flowEntries(unsigned vA, unsigned vS, unsigned cA, unsigned cS, int q, float* v, unsigned* c)
{
    const int4 f = lds128(vA + vS * (q / 4));
    v[0] = __int_as_float(f.x); v[1] = __int_as_float(f.y); v[2] = __int_as_float(f.z); v[3] = __int_as_float(f.w);
    const uint2 w = lds64(cA + cS * (q / 4));
    c[0] = w.x & 0xffffu; c[1] = w.x >> 16; c[2] = w.y & 0xffffu; c[3] = w.y >> 16;
}
// a row's first N entries: coefficients, and the codes turned into addresses
template <class T, int K, int N>
__device__ __forceinline__ void flowLoadEntries(FlowRow<T, K>& R, unsigned xA)
{
    unsigned c[N];
#pragma unroll
    for (int q = 0; q < N; q += 4) flowEntries(R.vA, R.vS, R.cA, R.cS, q, R.v + q, c + q);
#pragma unroll
    for (int q = 0; q < N; ++q) R.x[q] = xA + static_cast<unsigned>(sizeof(T)) * c[q];
}
// and their terms: the gathers together, then the sum in the row's order
template <class T, bool kFma, int K, int N>
__device__ __forceinline__ T flowSum(const FlowRow<T, K>& R)
{
    T y[N];
#pragma unroll
    for (int q = 0; q < N; ++q) y[q] = ldsT(R.x[q], T());
    T acc = R.b;
#pragma unroll
    for (int q = 0; q < N; ++q) acc = flowTerm<kFma>(acc, R.v[q], y[q]);
    return acc;
}

template <class T, int K>
__device__ __forceinline__ void flowLoad(unsigned chunkA, int slice, int lane, unsigned xA, FlowRow<T, K>& R)
{
    constexpr unsigned kT = sizeof(T);
    const int4 h = lds128(chunkA + 16u * slice);
    const unsigned items8 = h.x & 0xffff, codes8 = static_cast<unsigned>(h.x) >> 16;
    const unsigned vals8 = h.y & 0xffff, diag8 = static_cast<unsigned>(h.y) >> 16, src8 = h.z & 0xffff;
    const unsigned stride = static_cast<unsigned>(h.z) >> 24;
    R.w = (h.z >> 16) & 0xff;
    R.has = lane < (h.w & 0xff);
    const unsigned l = min(static_cast<unsigned>(lane), stride - 1);
    const uint2 it = lds64(chunkA + 8u * (items8 + lane));
    R.pos = it.x;
    R.slotWord = it.y;
    R.out = xA + kT * (it.y & 0xffffu);
    ldsPair(chunkA + 8u * diag8 + 2 * kT * lane, R.d, R.r);
    R.b = ldsT(chunkA + 8u * src8 + kT * lane, T());
    R.vA = chunkA + 8u * vals8 + 16u * l;
    R.cA = chunkA + 8u * codes8 + 8u * l;
    R.vS = 16u * stride;
    R.cS = 8u * stride;
    // straight-line code per width (no test per entry)
    const int w = min(R.w, K);
    if (w <= 4) flowLoadEntries<T, K, 4>(R, xA);
    else if (K <= 8 || w <= 8) flowLoadEntries<T, K, K < 8 ? K : 8>(R, xA);
    else if (K <= 12 || w <= 12) flowLoadEntries<T, K, K < 12 ? K : 12>(R, xA);
    else flowLoadEntries<T, K, K>(R, xA);
}

// the row in the reference's order: the source minus each entry's coefficient times its value, then the
// division by the diagonal; stored to its slot
template <class T, bool kFma, int K>
__device__ __forceinline__ T flowRow(const FlowRow<T, K>& R, unsigned xA)
{
    T acc;
    const int w = min(R.w, K);
    if (w <= 4) acc = flowSum<T, kFma, K, 4>(R);
    else if (K <= 8 || w <= 8) acc = flowSum<T, kFma, K, K < 8 ? K : 8>(R);
    else if (K <= 12 || w <= 12) acc = flowSum<T, kFma, K, K < 12 ? K : 12>(R);
    else acc = flowSum<T, kFma, K, K>(R);
#pragma unroll 1
    for (int q = K; q < R.w; q += 4)
    {
        // past the registers: four at a time
        T v[4], y[4];
        unsigned c[4];
        flowEntries(R.vA, R.vS, R.cA, R.cS, q, v, c);
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = ldsT(xA + static_cast<unsigned>(sizeof(T)) * c[i], T());
#pragma unroll
        for (int i = 0; i < 4; ++i) acc = flowTerm<kFma>(acc, v[i], y[i]);
    }
    // (a lane without an item has no divisor: it must not send its warp through the slow division)
    T x = T(0);
    if (R.has)
    {
        x = flowDiv(acc, R.d, R.r);
        stsT(R.out, x);
    }
    return x;
}

constexpr int flowThreads(bool remote) { return 32 * (2 * kFlowTeam + 2 + (remote ? kFlowHalo : 0)); }

template <class T, bool kFma, bool kRemote>
__device__ __forceinline__ void flowBody(const FlowArgs<T>& a, const int rank)
{
    extern __shared__ __align__(128) unsigned char flowSm[];
    __shared__ FlowShared S;
    constexpr int kD = kFlowDepth;
    constexpr int kTeamWarps = kFlowTeam;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned xA = smemAddr(flowSm);
    const unsigned ringA = xA + static_cast<unsigned>(flowRingAt(a.slots, sizeof(T)));
    const int c0 = a.chunkStart[rank];
    const int nCh = a.chunkStart[rank + 1] - c0;
    const unsigned epoch = kRemote && a.ctl ? *reinterpret_cast<volatile unsigned*>(a.ctl) + 1u : 0u;
    const unsigned tag0 = (epoch << 6) + 1u;
    const unsigned tagOut = a.publish ? tag0 : 0u;  // epochs start at 1: no tag is met when not publishing
    if (t == 0)
    {
        for (int i = 0; i < kD; ++i)
        {
            mbarInit(&S.full[i], 1);
            mbarInit(&S.staged[i], 32);
            mbarInit(&S.halo[i], 1);
        }
        S.consumed = 0;
        S.stop = 0;
        stsT(xA, T(0));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // A chunk's place in these barriers is taken again kFlowDepth chunks later, once the chunk is consumed; a warp
    // that waits for chunk j has waited for chunk j - kFlowDepth before, so the parity tells the two apart.
    static_assert(kD % 2 == 0 && kD % kFlowHalo == 0, "a team and a halo warp meet a barrier in every phase");
    auto isFull = [&](int j) { return mbarTryWait(&S.full[j % kD], (j / kD) & 1u); };
    auto isStaged = [&](int j) { return mbarTestWait(&S.staged[j % kD], (j / kD) & 1u); };
    auto hasHalo = [&](int j) { return mbarTestWait(&S.halo[j % kD], (j / kD) & 1u); };
    if (warp < 2 * kTeamWarps)
    {
        // Team j mod 2 computes chunk j. A team waits for the other's last chunk only (a named barrier per
        // team: the one that has computed arrives, the one that is about to waits), and loads its next chunk
        // while the other computes; what leaves the CTA is stored after the arrival.
        const int team = warp / kTeamWarps, wi = warp % kTeamWarps;
        FlowRow<T, kFlowK> R;
        R.w = -1;
        bool ok = true;   // no wait of this warp has given up
        bool haloOk = true;
        auto preload = [&](int j) {
            if (ok) ok = flowWait(S, a.err, a.spinLimit, [&] { return isFull(j) && isStaged(j); });
            R.w = -1;
            if (!ok) return;
            const uint2 p = lds64(smemAddr(&S.place[j % kD]));
            if (wi < static_cast<int>(p.y)) flowLoad(p.x, wi, lane, xA, R);
            if (kRemote) haloOk = hasHalo(j);
        };
        if (team < nCh) preload(team);
        for (int j = team; j < nCh; j += 2)
        {
            if (j > 0)
            {
                asm volatile("bar.sync %0, %1;" ::"r"(1 + ((j - 1) & 1)), "n"(64 * kTeamWarps) : "memory");
                // (never after a stop: the chunks that a stopped warp skipped may still be read by the other
                // roles, see LIMITS. A release, which carries the reads that the barrier has gathered to the
                // producer's acquire: measured within 0.3 % of a plain store on solves of 24 k to 1 M cells. By the
                // last warp, which has no row and no mailbox stores under way in a chunk of fewer slices)
                if (wi == kTeamWarps - 1 && lane == 0 && *reinterpret_cast<volatile unsigned*>(&S.stop) == 0)
                    stReleaseCta(&S.consumed, static_cast<unsigned>(j));
            }
            if (kRemote && ok && !haloOk)
                ok = flowWait(S, a.err, a.spinLimit, [&] { return hasHalo(j); });
            T x = T(0);
            if (ok && R.w >= 0) x = flowRow<T, kFma>(R, xA);
            if (j + 1 < nCh) asm volatile("bar.arrive %0, %1;" ::"r"(1 + (j & 1)), "n"(64 * kTeamWarps) : "memory");
            if (ok && R.w >= 0 && R.has)
            {
                if (kRemote && (R.slotWord & 0x40000000u))
                    mailSt(static_cast<T*>(a.mail), static_cast<int>(R.pos), x, tagOut + ((R.slotWord >> 16) & 0x3fu));
                if (R.slotWord & 0x80000000u) a.psi[R.pos] = x;
            }
            if (j + 2 < nCh) preload(j + 2);
        }
    }
    else if (warp == 2 * kTeamWarps)
    {
        // the producer: chunk j's blobs into its place in the ring once that place is free
        int issued = 0, consumed = 0;
        int4 q0{}, q1{}, q2{};
        for (int j = 0; j < nCh; ++j)
        {
            if ((j & 31) == 0 && j + lane < nCh)
            {
                const int4* p = a.rec + 3 * static_cast<size_t>(c0 + j + lane);
                q0 = p[0];
                q1 = p[1];
                q2 = p[2];
            }
            const int from = j & 31;
            int4 r0, r1, r2;
            r0.x = __shfl_sync(~0u, q0.x, from); r0.y = __shfl_sync(~0u, q0.y, from);
            r0.z = __shfl_sync(~0u, q0.z, from); r0.w = __shfl_sync(~0u, q0.w, from);
            r1.x = __shfl_sync(~0u, q1.x, from); r1.y = __shfl_sync(~0u, q1.y, from);
            r1.z = __shfl_sync(~0u, q1.z, from); r1.w = __shfl_sync(~0u, q1.w, from);
            r2.x = __shfl_sync(~0u, q2.x, from); r2.y = __shfl_sync(~0u, q2.y, from);
            r2.z = __shfl_sync(~0u, q2.z, from); r2.w = __shfl_sync(~0u, q2.w, from);
            if (consumed <= r0.w)
            {
                const bool go = flowWait(S, a.err, a.spinLimit, [&] {
                    consumed = static_cast<int>(ldAcquireCta(&S.consumed));
                    return consumed > r0.w;
                });
                if (!go) consumed = -1;
            }
            consumed = __reduce_min_sync(~0u, consumed);
            if (consumed < 0) break;
            if (lane == 0)
            {
                unsigned long long* bar = &S.full[j % kD];
                S.rec[j % kD][0] = r0;
                S.rec[j % kD][1] = r1;
                S.rec[j % kD][2] = r2;
                S.place[j % kD] = make_uint2(ringA + static_cast<unsigned>(r0.z), static_cast<unsigned>(r1.w));
                fenceProxyAsyncShared();
                mbarExpectTx(bar, static_cast<unsigned>(r0.y + r1.y));
                tmaLoad(ringA + static_cast<unsigned>(r0.z), a.meta + 16 * static_cast<size_t>(r0.x),
                        static_cast<unsigned>(r0.y), bar);
                tmaLoad(ringA + static_cast<unsigned>(r0.z + r0.y),
                        reinterpret_cast<const unsigned char*>(a.val) + 16 * static_cast<size_t>(r1.x),
                        static_cast<unsigned>(r1.y), bar);
            }
            __syncwarp();
            issued = j + 1;
        }
        // the CTA leaves only once the copies issued have landed, whether a wait gave up before or does after this
        for (int j = max(0, issued - kD); j < issued; ++j)
            for (long long it = 0; it < (1 << 20) && !isFull(j); ++it) {}
    }
    else if (warp == 2 * kTeamWarps + 1)
    {
        // the gather warp: each chunk's source values and the initial values first used there. The copies tell
        // the chunk's barrier themselves when they have landed, so any number of chunks are under way.
        for (int j = 0; j < nCh; ++j)
        {
            const bool go = flowWait(S, a.err, a.spinLimit, [&] { return isFull(j); });
            if (!__all_sync(~0u, go)) break;
            const int4 r0 = S.rec[j % kD][0], r1 = S.rec[j % kD][1], r2 = S.rec[j % kD][2];
            const unsigned chunkA = ringA + static_cast<unsigned>(r0.z);
            const unsigned bA = chunkA + static_cast<unsigned>(r0.y + r1.y);
            for (int i = lane; i < r1.z; i += 32)
                cpAsync(bA + static_cast<unsigned>(sizeof(T)) * i, a.b + ldsU32(chunkA + 8u * (r2.x + i)));
            for (int i = lane; i < (r2.w & 0xffff); i += 32)
            {
                const uint2 f = lds64(chunkA + 8u * (r2.y + i));
                cpAsync(xA + static_cast<unsigned>(sizeof(T)) * f.y, a.psi + f.x);
            }
            mbarArriveCpAsync(&S.staged[j % kD]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    else if (kRemote)
    {
        // a halo warp: the values of other ranks that its chunks read first
        const int h = warp - 2 * kTeamWarps - 2;
        const T* mail = static_cast<const T*>(a.mail);
        for (int j = h; j < nCh; j += kFlowHalo)
        {
            bool go = flowWait(S, a.err, a.spinLimit, [&] { return isFull(j); });
            if (!__all_sync(~0u, go)) break;
            const int4 r2 = S.rec[j % kD][2];
            const unsigned haloA = ringA + static_cast<unsigned>(S.rec[j % kD][0].z) + 8u * r2.z;
            const int nH = static_cast<int>(static_cast<unsigned>(r2.w) >> 16);
            for (int i = lane; i < nH; i += 64)
            {
                // two mailboxes a lane in flight
                const bool two = i + 32 < nH;
                const uint2 e0 = lds64(haloA + 8u * i);
                const uint2 e1 = two ? lds64(haloA + 8u * (i + 32)) : e0;
                const unsigned p0 = e0.x, w0 = e0.y, p1 = e1.x, w1 = e1.y;
                T v0, v1;
                bool d0 = false, d1 = false;
                go = flowWait(S, a.err, a.spinLimit, [&] {
                    T y0, y1;
                    const unsigned g0 = mailLd(mail, p0, y0), g1 = mailLd(mail, p1, y1);
                    if (!d0 && g0 == tag0 + (w0 >> 16)) { d0 = true; v0 = y0; }
                    if (!d1 && g1 == tag0 + (w1 >> 16)) { d1 = true; v1 = y1; }
                    return d0 && d1;
                });
                if (!go) break;
                stsT(xA + static_cast<unsigned>(sizeof(T)) * (w0 & 0xffffu), v0);
                if (two) stsT(xA + static_cast<unsigned>(sizeof(T)) * (w1 & 0xffffu), v1);
            }
            if (!__all_sync(~0u, go)) break;
            __syncwarp();
            if (lane == 0) mbarArrive(&S.halo[j % kD]);
        }
    }
    if (kRemote && a.ctl)
    {
        // the last rank to finish moves the launch counter on, so no tag of this launch is met again
        __syncthreads();
        if (t == 0 && atomicAdd(a.ctl + 1, 1u) == static_cast<unsigned>(a.ranks - 1))
        {
            a.ctl[1] = 0;
            a.ctl[0] = epoch;
        }
    }
}

// One smoothing call of one level: block r is rank r (all resident when there are more than one).
template <class T, bool kFma, bool kRemote>
__global__ void __launch_bounds__(flowThreads(kRemote), 1) gsFlow(FlowArgs<T> a)
{
    flowBody<T, kFma, kRemote>(a, blockIdx.x);
}

// One smoothing call of many independent cases' levels in one launch: block i runs rank blocks[i].y of
// table[blocks[i].x], skipped when its case's `active` flag (may be null) is 0. With kRemote the launch is
// cooperative (every rank of every case resident).
template <class T, bool kRemote>
__global__ void __launch_bounds__(flowThreads(kRemote), 1) gsFlowBatch(const FlowArgs<T>* __restrict__ table,
                                                                       const int2* __restrict__ blocks,
                                                                       const int* __restrict__ caseOf,
                                                                       const int* __restrict__ active)
{
    const int2 w = blocks[blockIdx.x];
    if (active && active[caseOf[w.x]] == 0) return;
    __shared__ FlowArgs<T> a;
    if (threadIdx.x < sizeof(FlowArgs<T>) / 4)
        reinterpret_cast<unsigned*>(&a)[threadIdx.x] = reinterpret_cast<const unsigned*>(table + w.x)[threadIdx.x];
    __syncthreads();
    flowBody<T, false, kRemote>(a, w.y);
}

// The values of a schedule's chunks, from the level's rows by position: a warp per slice, a lane per item. Where
// each comes from is in the chunk's own meta blob (its items' positions), so no index a value is kept.
template <class T>
__global__ void flowValues(int nChunks, const int4* __restrict__ rec, const unsigned char* __restrict__ meta,
                           const int* __restrict__ posRow, const T* __restrict__ rowVal, const T* __restrict__ diag,
                           T* __restrict__ out)
{
    constexpr int kPer = 16 / sizeof(T);  // coefficients a lane reads with one load
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    for (int j = blockIdx.x; j < nChunks; j += gridDim.x)
    {
        const int4 r0 = rec[3 * static_cast<size_t>(j)], r1 = rec[3 * static_cast<size_t>(j) + 1];
        const unsigned char* M = meta + 16 * static_cast<size_t>(r0.x);
        // (offsets within a chunk run on from its meta blob to its values)
        T* V = out + kPer * static_cast<size_t>(r1.x);
        for (int s = warp; s < r1.w; s += nWarps)
        {
            const FlowSlice h = reinterpret_cast<const FlowSlice*>(M)[s];
            const bool has = lane < h.count;
            const int p = has ? reinterpret_cast<const int2*>(M + 8 * static_cast<size_t>(h.items8))[lane].x : 0;
            const T d = has ? diag[p] : T(0);
            T* dv = V + (8 * static_cast<size_t>(h.diag8) - r0.y) / sizeof(T) + 2 * lane;
            dv[0] = d;
            dv[1] = has ? flowRcp(d) : T(0);
            if (lane >= h.stride) continue;
            const int e0 = has ? posRow[p] : 0, w = has ? posRow[p + 1] - e0 : 0;
            T* ev = V + (8 * static_cast<size_t>(h.vals8) - r0.y) / sizeof(T) + kPer * lane;
            for (int q = 0; q < h.width; q += kPer)
#pragma unroll
                for (int i = 0; i < kPer; ++i)
                    ev[static_cast<size_t>(h.stride) * q + i] = q + i < w ? rowVal[e0 + q + i] : T(0);
        }
    }
}

}  // namespace k
}  // namespace b2g
