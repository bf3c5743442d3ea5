// Multi-scale morphological baseliner for sm_100a.
//
// Restates TA/HostMultiScaleBaseliner.cpp:95-212, TA/TraceFilters.cpp:11-57,
// TA/BlockFilterStage.cpp:9-25 and DT/BaselinerStatAccumulator.cpp:39-53
// (TA = src/basecaller/basecaller/traceAnalysis, DT = src/basecaller/dataTypes).
//
// Design: one thread per pair of neighbouring ZMWs streams its chunk frame by
// frame (see "Two ZMWs per thread" below for the packed arithmetic).  The reference
// runs every filter stage in place over the whole block; because each stage is
// causal (output m depends on inputs m-w..m-1) and chunk lengths are multiples
// of the aggregate stride, the same values come out of a per-frame pipeline in
// which scale i is fed at frames t with t % cumStride_i == 0.  The final stage
// produces block i's lower/upper envelope at frame i*aggStride, exactly when the
// subtraction of that block starts, so the trace is read from HBM once and the
// baselined trace written once, with coalesced 128-byte warp accesses.  The
// windows of the scales that run every frame or every other frame live in
// shared memory, those of the last scale (every 16 frames) in global memory,
// which leaves room for 14 one-lane blocks per SM with the widest filter.
// Bound by latency (a warp's dependent instructions; 3.5 warps a scheduler,
// 48% of its issue slots).  4096 lanes x 512 frames of int16: 988 us with four
// separate window stages a scale, conversions by I2F and F2I and selects in
// the moments; 455 us as written (0.93 GB read and written, 2.0 TB/s).
// Each stage window keeps the reference's van Herk/Gil-Werman state (ring of w
// values, holdover, counter) so the filter outputs are bit-identical.
#include <type_traits>

#include "hw_device.cuh"

namespace hwk {

template <int FT> struct FSpec;
template <> struct FSpec<HW_FILTER_MULTISCALE_LARGE>  { static constexpr int n = 3; static constexpr int s[3] = {1, 2, 8}; static constexpr int w[3] = {11, 17, 61}; };
template <> struct FSpec<HW_FILTER_MULTISCALE_MEDIUM> { static constexpr int n = 3; static constexpr int s[3] = {1, 2, 8}; static constexpr int w[3] = {9, 17, 31}; };
template <> struct FSpec<HW_FILTER_MULTISCALE_SMALL>  { static constexpr int n = 3; static constexpr int s[3] = {1, 2, 8}; static constexpr int w[3] = {7, 17, 17}; };
template <> struct FSpec<HW_FILTER_TWOSCALE_LARGE>    { static constexpr int n = 2; static constexpr int s[3] = {2, 8, 1}; static constexpr int w[3] = {11, 61, 0}; };
template <> struct FSpec<HW_FILTER_TWOSCALE_MEDIUM>   { static constexpr int n = 2; static constexpr int s[3] = {2, 8, 1}; static constexpr int w[3] = {9, 31, 0}; };
template <> struct FSpec<HW_FILTER_TWOSCALE_SMALL>    { static constexpr int n = 2; static constexpr int s[3] = {2, 8, 1}; static constexpr int w[3] = {7, 17, 0}; };

template <int FT> struct FLayout
{
    using S = FSpec<FT>;
    static constexpr int nStages = 2 * S::n;           // per filter
    static constexpr int Width(int k) { return S::w[k / 2]; }
    // lower: erode, dilate, then erode/dilate; upper: dilate, erode, then erode/dilate
    static constexpr bool IsMax(bool upper, int k) { return (k < 2 && upper) ? (k == 0) : (k % 2 == 1); }
    static constexpr bool InSmem(int k) { return CumStride(k / 2) < AggStride(); }
    static constexpr int Idx(bool upper, int k) { return (upper ? nStages : 0) + k; }   // 0 .. 2*nStages-1
    // Saved state: every stage's S[W] (suffix extrema of the previous block)
    // and then its B[W] (inputs of the current block), first the stages up to
    // 11 wide, then the wider ones, each group lower filter first.  (A state
    // saved by one build is read by another: the order stays whatever the
    // kernel keeps where.)
    static constexpr bool Narrow(int k) { return Width(k) <= 11; }
    static constexpr int SlotWindow(bool upper, int k)
    {
        int t = 0;
        if (!Narrow(k))
            for (int j = 0; j < nStages; ++j) if (Narrow(j)) t += 4 * Width(j);
        for (int u = 0; u < 2; ++u)
            for (int j = 0; j < nStages; ++j)
            {
                if (u == (upper ? 1 : 0) && j == k) return t;
                if (Narrow(j) == Narrow(k)) t += 2 * Width(j);
            }
        return t;
    }
    // Shared memory: position c of a block needs S[c..] and B[..c-1] only, so
    // a stage keeps one array of W there, inputs below the counter and suffix
    // extrema from it on.
    static constexpr int SmemSlots()
    {
        int t = 0;
        for (int k = 0; k < nStages; ++k) if (InSmem(k)) t += 2 * Width(k);
        return t;
    }
    static constexpr int SmemOffset(bool upper, int k)
    {
        int t = upper ? SmemSlots() / 2 : 0;
        for (int j = 0; j < k; ++j) if (InSmem(j)) t += Width(j);
        return t;
    }
    // index of a global stage among the global stages (lower first)
    static constexpr int GIdx(bool upper, int k)
    {
        int t = upper ? NumGlobalStages() / 2 : 0;
        for (int j = 0; j < k; ++j) if (!InSmem(j)) ++t;
        return t;
    }
    static constexpr int NumGlobalStages()
    {
        int t = 0;
        for (int k = 0; k < nStages; ++k) if (!InSmem(k)) ++t;
        return 2 * t;
    }
    static constexpr int WindowSlots()
    {
        int t = 0;
        for (int k = 0; k < nStages; ++k) t += 4 * Width(k);
        return t;
    }
    static constexpr int CumStride(int i)
    {
        int c = 1;
        for (int j = 0; j <= i; ++j) c *= S::s[j];
        return c;
    }
    static constexpr int AggStride() { return CumStride(S::n - 1); }
    // int16 state: the windows, then (P, c) per stage, then latData, latRaw,
    // masks.
    static constexpr int SlotPC(bool upper, int k) { return WindowSlots() + 2 * Idx(upper, k); }
    static constexpr int SlotLatData() { return WindowSlots() + 4 * nStages; }
    static constexpr int NumI16Slots() { return SlotLatData() + 3; }
};

// ---- Two ZMWs per thread ----------------------------------------------------
// A thread owns the neighbouring ZMWs 2t and 2t + 1 of its lane: their int16
// values travel as one 32-bit pair (ZMW 2t in the low half), so the window
// filters run as packed 16-bit min/max (one instruction for both ZMWs) and
// every load and store of trace, output and state moves both.  The filter
// state keeps its [slot][zmw] int16 layout: a pair is just two neighbouring
// slots.  All ZMWs of a pool take the same frames, so the block counters of
// the window stages are one value per lane.  The floating-point estimate and
// statistics run as f32x2 pairs (see hw_device.cuh) or per ZMW with the
// reference's operation order.

__device__ __forceinline__ uint32_t MaxS16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t MinS16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ int16_t Lo16(uint32_t p) { return (int16_t)(p & 0xffffu); }
__device__ __forceinline__ int16_t Hi16(uint32_t p) { return (int16_t)(p >> 16); }
__device__ __forceinline__ uint32_t Pack16(int16_t lo, int16_t hi) { return (uint32_t)(uint16_t)lo | ((uint32_t)(uint16_t)hi << 16); }

template <bool IsMax> __device__ __forceinline__ uint32_t Op2(uint32_t a, uint32_t b)
{
    return IsMax ? MaxS16x2(a, b) : MinS16x2(a, b);
}
template <bool IsMax> constexpr uint32_t Identity2() { return IsMax ? 0x80008000u : 0x7fff7fffu; }

// One scale of both filters for a ZMW pair: the lower filter's two window
// stages and the upper filter's two, each van Herk/Gil-Werman.  A stage's
// output for each input is the extremum of the W previous inputs
// (TraceFilters.cpp:11-57 with the window state of WindowBuffer.h; the initial
// window holds W zeros).  Its state is the suffix extrema S of the previous
// block of W inputs, the running extremum P of the current block and the
// current block's inputs B; the output at block position c is op(S[c], P).
// The four stages are fed at the same frames and so share c: one counter, one
// address and one end-of-block pass for the four (four independent chains)
// instead of four of each.
//
// A scale that runs every frame or every other frame keeps its windows in
// shared memory, S and B in one array (see FLayout).  The last scale's live in
// global memory with S[c] loaded into a register one call (16 frames) ahead of
// its use (S changes only when a block completes), so the stage never waits
// for memory on its critical path.  Measured on 4096 lanes x 512 frames,
// MultiScaleLarge: 17-wide windows in global memory 654 us, in shared memory 455
// us; with S and B apart they would leave room for 7 blocks a SM instead of 14.
struct StageMem2
{
    uint32_t* smem;     // this thread's column in shared memory (stride kBlPairs)
    uint32_t* gmem;     // this pair's column of the saved state, used in place
    size_t gstride;     // nZmw / 2
    uint32_t* sNext;    // per global stage: S[c], loaded ahead
};

constexpr int kBlPairs = kLane / 2;       // threads per lane

// Filter state of one thread: P of every stage (a ZMW pair) and the block
// counter of every scale.
template <int FT> struct PairState
{
    uint32_t P[2 * FLayout<FT>::nStages];
    int c[FSpec<FT>::n];
};

// sNext of every global-memory stage of one filter from the saved state
// (compile-time recursion: the stage layout tables are host constants).
template <int FT, bool Upper, int K>
__device__ __forceinline__ void LoadSNext2(const StageMem2& m, const PairState<FT>& ps)
{
    using Lay = FLayout<FT>;
    if constexpr (K < Lay::nStages)
    {
        if constexpr (!Lay::InSmem(K))
            m.sNext[Lay::GIdx(Upper, K)] = m.gmem[(size_t)(Lay::SlotWindow(Upper, K) + ps.c[K / 2]) * m.gstride];
        LoadSNext2<FT, Upper, K + 1>(m, ps);
    }
}

// Shared-memory windows from (Save: to) the saved state, where S and B have
// slots of their own: the part of each that the block position needs.
template <int FT, bool Upper, int K, bool Save>
__device__ __forceinline__ void CopyWindows(uint32_t* smem, uint32_t* state, size_t nPair, const PairState<FT>& ps)
{
    using Lay = FLayout<FT>;
    if constexpr (K < Lay::nStages)
    {
        if constexpr (Lay::InSmem(K))
        {
            constexpr int W = Lay::Width(K);
            const int c = ps.c[K / 2];
#pragma unroll 17
            for (int j = 0; j < W; ++j)
            {
                uint32_t& at = state[(size_t)(Lay::SlotWindow(Upper, K) + j + (j < c ? W : 0)) * nPair];
                uint32_t& w = smem[(Lay::SmemOffset(Upper, K) + j) * kBlPairs];
                if (Save) at = w;
                else w = at;
            }
        }
        CopyWindows<FT, Upper, K + 1, Save>(smem, state, nPair, ps);
    }
    else if constexpr (!Upper) CopyWindows<FT, true, 0, Save>(smem, state, nPair, ps);
}

// lo and up enter as the scale's inputs and leave as its outputs.
template <int FT, int Scale>
__device__ __forceinline__ void RunScale2(const StageMem2& m, PairState<FT>& ps, uint32_t& lo, uint32_t& up)
{
    using Lay = FLayout<FT>;
    constexpr int K0 = 2 * Scale, K1 = K0 + 1, W = Lay::Width(K0);
    constexpr bool smem = Lay::InSmem(K0);
    // stages: lower first, lower second, upper first, upper second
    constexpr int off[4] = {smem ? Lay::SmemOffset(false, K0) : Lay::SlotWindow(false, K0),
                            smem ? Lay::SmemOffset(false, K1) : Lay::SlotWindow(false, K1),
                            smem ? Lay::SmemOffset(true, K0) : Lay::SlotWindow(true, K0),
                            smem ? Lay::SmemOffset(true, K1) : Lay::SlotWindow(true, K1)};
    constexpr int pi[4] = {Lay::Idx(false, K0), Lay::Idx(false, K1), Lay::Idx(true, K0), Lay::Idx(true, K1)};
    constexpr int gi[4] = {Lay::GIdx(false, K0), Lay::GIdx(false, K1), Lay::GIdx(true, K0), Lay::GIdx(true, K1)};
    constexpr bool isMax[4] = {Lay::IsMax(false, K0), Lay::IsMax(false, K1), Lay::IsMax(true, K0),
                               Lay::IsMax(true, K1)};
    auto op = [](bool mx, uint32_t a, uint32_t b) { return mx ? MaxS16x2(a, b) : MinS16x2(a, b); };
    const size_t stride = smem ? (size_t)kBlPairs : m.gstride;
    uint32_t* base = smem ? m.smem : m.gmem;
    auto S = [&](int i, int j) -> uint32_t& { return base[(size_t)(off[i] + j) * stride]; };
    auto B = [&](int i, int j) -> uint32_t& { return base[(size_t)(off[i] + (smem ? 0 : W) + j) * stride]; };
    const int c = ps.c[Scale];
    uint32_t x[4];
    x[0] = lo;
    x[2] = up;
#pragma unroll
    for (int u = 0; u < 4; u += 2)
    {
        uint32_t in = x[u];
#pragma unroll
        for (int i = u; i < u + 2; ++i)
        {
            x[i] = in;
            uint32_t s;
            if constexpr (smem) s = S(i, c);
            else s = m.sNext[gi[i]];
            in = op(isMax[i], s, ps.P[pi[i]]);
            B(i, c) = x[i];
            ps.P[pi[i]] = op(isMax[i], ps.P[pi[i]], x[i]);
        }
        (u ? up : lo) = in;
    }
    if (c + 1 == W)
    {
        // New suffix extrema of the completed blocks.
        uint32_t acc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            acc[i] = x[i];
            S(i, W - 1) = acc[i];
        }
        constexpr int kBatch = 2;       // inputs read before the batch's results are stored
#pragma unroll 1
        for (int j0 = W - 2; j0 >= 0; j0 -= kBatch)
        {
            uint32_t b[kBatch][4];
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (W % kBatch == 1 || j0 - q >= 0) b[q][i] = B(i, j0 - q);
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (W % kBatch == 1 || j0 - q >= 0)
                    {
                        acc[i] = op(isMax[i], b[q][i], acc[i]);
                        S(i, j0 - q) = acc[i];
                    }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            if constexpr (!smem) m.sNext[gi[i]] = acc[i];      // S[0]
            ps.P[pi[i]] = isMax[i] ? Identity2<true>() : Identity2<false>();
        }
        ps.c[Scale] = 0;
    }
    else
    {
        ps.c[Scale] = c + 1;
        if constexpr (!smem)
        {
#pragma unroll
            for (int i = 0; i < 4; ++i) m.sNext[gi[i]] = S(i, c + 1);
        }
    }
}

// Feeds one frame through both multi-scale filters; returns true and the
// envelope values when the last scale produced an output.  Cumulative strides
// are 1, 2 or 16 and chunks are multiples of 16 frames, so the scales that
// run depend only on the frame's phase within its 16-frame block:
// Phase 0 = first frame of the block, 1 = other even frames, 2 = odd frames.
template <int Phase>
__host__ __device__ constexpr bool ScaleRuns(int cumStride)
{
    return cumStride == 1 || (cumStride == 2 && Phase <= 1) || (cumStride == 16 && Phase == 0);
}

template <int FT, int Phase>
__device__ __forceinline__ bool FeedFilters2(uint32_t x, const StageMem2& m, PairState<FT>& ps, uint32_t& lo,
                                             uint32_t& up)
{
    using S = FSpec<FT>;
    using Lay = FLayout<FT>;
    static_assert(Lay::CumStride(0) <= 2 && (S::n < 2 || Lay::CumStride(1) <= 16) && Lay::AggStride() == 16,
                  "phase scheme needs cumulative strides 1|2, 2, 16");
    lo = up = x;
    if constexpr (!ScaleRuns<Phase>(Lay::CumStride(0))) return false;
    else
    {
        RunScale2<FT, 0>(m, ps, lo, up);
        if constexpr (!ScaleRuns<Phase>(Lay::CumStride(1))) return false;
        else
        {
            RunScale2<FT, 1>(m, ps, lo, up);
            if constexpr (S::n > 2)
            {
                if constexpr (!ScaleRuns<Phase>(Lay::CumStride(2))) return false;
                else RunScale2<FT, 2>(m, ps, lo, up);
            }
            return true;
        }
    }
}

// Initial filter state: every window holds W zeros (S = 0), the current block
// is empty (P = identity of the stage's operation, counter 0).
template <int FT>
__global__ void BaselinerInitKernel(int16_t* st16, float* st32, int lanes)
{
    using Lay = FLayout<FT>;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int nZmw = lanes * kLane;
    if (g >= nZmw) return;
    for (int i = 0; i < Lay::NumI16Slots(); ++i) st16[(size_t)i * nZmw + g] = 0;
    for (int u = 0; u < 2; ++u)
        for (int k = 0; k < Lay::nStages; ++k)
            st16[(size_t)Lay::SlotPC(u == 1, k) * nZmw + g] = Lay::IsMax(u == 1, k) ? (int16_t)-32768 : (int16_t)32767;
    st32[(size_t)0 * nZmw + g] = 0.0f;
    st32[(size_t)1 * nZmw + g] = 0.0f;
    st32[(size_t)2 * nZmw + g] = 2.0f;     // blSigmaEma_ initial value
}

// Reads the trace value pair of frame t.
template <typename TIn>
__device__ __forceinline__ uint32_t LoadPair(const TIn* tr, int t)
{
    if constexpr (std::is_same_v<TIn, uint8_t>)
    {
        const uint16_t b = __ldg(reinterpret_cast<const uint16_t*>(tr + (size_t)t * kLane));
        return (b & 0xffu) | ((uint32_t)(b >> 8) << 16);      // uint8 -> int16 widening of both
    }
    else
    {
        return __ldg(reinterpret_cast<const uint32_t*>(tr + (size_t)t * kLane));
    }
}

// Both int16 values as floats, exact: with the sign bit flipped a value is
// v + 32768 in 16 bits, which as the low half of 2^23's bits is the float
// 2^23 + 32768 + v.  (Three ALU instructions and a packed addition instead of
// two conversions at a quarter of the rate.)
__device__ __forceinline__ float2 PairToFloat(uint32_t p)
{
    const uint32_t u = p ^ 0x80008000u;
    return add2(f2(__uint_as_float(__byte_perm(u, 0x4b000000u, 0x7610)),
                   __uint_as_float(__byte_perm(u, 0x4b000000u, 0x7632))),
                f2(-(8388608.0f + 32768.0f)));
}

// x - pedestal with int16 wrap-around, per half (negPed: both halves -pedestal).
__device__ __forceinline__ uint32_t SubPed(uint32_t x, uint32_t negPed)
{
    uint32_t r;
    asm("add.s16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(negPed));
    return r;
}

// Reference float -> int16 conversion of both values (to_i16_wrap) when both
// are below 2^22 in magnitude: added to 1.5 * 2^23 they round to the nearest
// even integer, whose low 16 bits are the sum's.
__device__ __forceinline__ uint32_t RoundPair(float2 v)
{
    const float2 m = add2(v, f2(12582912.0f));
    return __byte_perm(__float_as_uint(m.x), __float_as_uint(m.y), 0x5410);
}
// The same for any values.
__device__ __noinline__ uint32_t RoundPairGeneral(float2 v) { return Pack16(to_i16_wrap(v.x), to_i16_wrap(v.y)); }

// a < b ? 1 : 0 (0 when either is NaN).
__device__ __forceinline__ float LessAsFloat(float a, float b)
{
    float r;
    asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

template <int FT, typename TIn, bool Mapped>
__global__ void __launch_bounds__(kBlPairs, 16) BaselinerKernel(BaselinerArgs a, KParams k)
{
    using Lay = FLayout<FT>;
    LaneMap map = a.map;
    if (!Mapped) map.list = nullptr;      // the single-pool variant compiles without the lane list
    // one lane per block, one ZMW pair per thread
    if ((int)blockIdx.x >= map.Lanes(a.lanes)) return;
    const int t = threadIdx.x;
    const int lane = map.Lane(blockIdx.x);
    const int nZmw = a.lanes * kLane;
    const int nPair = nZmw / 2;
    const int gp = lane * kBlPairs + t;       // pair index; ZMWs 2 gp, 2 gp + 1
    const int z = 2 * t;
    const PoolStep* ps = map.On() ? &map.Pool(lane) : nullptr;
    const int F = ps ? ps->F : a.F;

    // Window state: the scales that run more often than every 16 frames in
    // shared memory (one column per thread), the last one's used in place in
    // global memory.
    extern __shared__ uint32_t blSmem2[];
    constexpr int NG = Lay::NumGlobalStages() > 0 ? Lay::NumGlobalStages() : 1;
    uint32_t sNext[NG];
    const uint32_t* st = reinterpret_cast<const uint32_t*>(a.st16);
    uint32_t* stw = reinterpret_cast<uint32_t*>(a.st16);
    const StageMem2 mem{blSmem2 + t, stw + gp, (size_t)nPair, sNext};
    PairState<FT> fs;
#pragma unroll
    for (int i = 0; i < 2 * Lay::nStages; ++i)
    {
        const bool up = i >= Lay::nStages;
        const int kk = up ? i - Lay::nStages : i;
        fs.P[i] = st[(size_t)Lay::SlotPC(up, kk) * nPair + gp];
        // the same for every ZMW and every stage of a scale
        if (!up && kk % 2 == 0) fs.c[kk / 2] = Lo16(st[(size_t)(Lay::SlotPC(up, kk) + 1) * nPair + gp]);
    }
    CopyWindows<FT, false, 0, false>(blSmem2 + t, stw + gp, (size_t)nPair, fs);
    // S[counter] of every global stage
    LoadSNext2<FT, false, 0>(mem, fs);
    LoadSNext2<FT, true, 0>(mem, fs);
    uint32_t latData = st[(size_t)Lay::SlotLatData() * nPair + gp];
    uint32_t latRaw = st[(size_t)(Lay::SlotLatData() + 1) * nPair + gp];
    const uint32_t mbits = st[(size_t)(Lay::SlotLatData() + 2) * nPair + gp];
    // 1 where the previous frame was in the baseline (its threshold and its
    // latent copy), else 0; hp2: the frame before it
    float2 hp1 = f2((mbits & 3u) == 3u ? 1.0f : 0.0f, ((mbits >> 16) & 3u) == 3u ? 1.0f : 0.0f), hp2 = hp1;
    const float2* st32 = reinterpret_cast<const float2*>(a.st32);
    float2 uemaSum = st32[(size_t)0 * nPair + gp];
    float2 uemaWeight = st32[(size_t)1 * nPair + gp];
    float2 sigmaEma = st32[(size_t)2 * nPair + gp];
    const float2 nz = f2(k.negZero);

    // Per-chunk BaselinerStatAccumulator (fresh each chunk, offset 0).  The
    // sample counts are F and F / 16; the front buffer (the first four
    // samples) is the latent frame and the chunk's first three outputs, read
    // back at the end.
    float2 c_m1 = f2(0.0f), c_m2 = f2(0.0f), c_acm2 = f2(0.0f);
    const uint32_t firstData = latData;
    float2 back[4] = {f2(0.0f), f2(0.0f), f2(0.0f), f2(0.0f)};     // last four samples, back[f % 4] of frame f
    float2 latV = PairToFloat(latData), latRawV = PairToFloat(latRaw);
    uint32_t tmin = 0x7fff7fffu, tmax = 0x80008000u;
    float2 b_m0 = f2(0.0f), b_m1 = f2(0.0f), b_m2 = f2(0.0f), rawSum = f2(0.0f);
    float2 g_m1 = f2(0.0f), g_m2 = f2(0.0f);

    const TIn* tr;
    const size_t inOff = ps ? (size_t)(lane - ps->lane0) * F * kLane : (size_t)lane * F * kLane;
    if constexpr (std::is_same_v<TIn, uint8_t>) tr = (ps ? ps->trace8 : a.trace8) + inOff + z;
    else tr = (ps ? ps->trace : a.trace) + inOff + z;
    uint32_t* out = reinterpret_cast<uint32_t*>(a.out + map.Block(lane, F) + z);
    const uint32_t negPed = Pack16(i16_wrap(-k.pedestal), i16_wrap(-k.pedestal));
    const float2 scaler = f2(k.scaler);
    const bool scalerOk = fabsf(k.scaler) <= 63.0f;     // |x scaler| < 2^21
    float2 negSub = f2(0.0f), thr = f2(0.0f);
    bool inRange = false;

    // Frames go in blocks of 16 (the aggregate stride): the first frame of a
    // block, the other even frames and the odd frames each get their own
    // specialisation of the frame body (four frames a loop turn, the period
    // of the back buffer), with the trace loaded two frames ahead.  Even
    // frames take their value from xEven and odd frames from xOdd, each
    // refilled right after use: no register is copied while its load is in
    // flight.  Two loads in flight a warp do not cover the latency of DRAM at
    // 14 warps a SM, so each block prefetches the block after the next: the
    // lane's frames are consecutive lines, one a thread (708 -> 672 us on the
    // case above, 243 -> 192 us on TwoScaleMedium, 2048 lanes).
    static_assert(Lay::AggStride() == 16, "block size must be the aggregate stride");
    const TIn* lines = tr - z;
    if (t < F) PrefetchL1(lines + (size_t)t * kLane);
    uint32_t xEven = LoadPair(tr, 0), xOdd = LoadPair(tr, 1);
    auto frame = [&](auto phaseTag, auto slotTag, int f) {
        constexpr int Ph = decltype(phaseTag)::value;
        constexpr int Slot = decltype(slotTag)::value;
        uint32_t& slot = (Ph == 2) ? xOdd : xEven;      // phase 2 = odd frames
        const uint32_t x = slot;
        if (f + 2 < F) slot = LoadPair(tr, f + 2);
        uint32_t lo, up;
        const bool haveL = FeedFilters2<FT, Ph>(x, mem, fs, lo, up);
        if (haveL)
        {
            // GetSmoothedBlEstimate (HostMultiScaleBaseliner.cpp:179-212)
            const uint32_t lv = SubPed(lo, negPed), uv = SubPed(up, negPed);
            constexpr float minSigma = .288675135f;
            const float ma = k.meanEmaAlpha, sa = k.sigmaEmaAlpha;
            float2 sigma;
            sigma.x = fmax_sse((float)i16_wrap(Lo16(uv) - Lo16(lv)) / k.cSigmaBias, minSigma);
            sigma.y = fmax_sse((float)i16_wrap(Hi16(uv) - Hi16(lv)) / k.cSigmaBias, minSigma);
            const float2 newSigmaEma = add2(mulz2(f2(sa), sigmaEma, nz), mulz2(f2(1.0f - sa), sigma, nz));
            const float2 mid = f2((float)i16_wrap(Lo16(uv) + Lo16(lv)), (float)i16_wrap(Hi16(uv) + Hi16(lv)));
            const float2 blEst = add2(mulz2(f2(0.5f), mid, nz), mulz2(f2(k.cMeanBias), newSigmaEma, nz));
            const float2 jt = mul2(f2(k.jumpTolCoeff), sigmaEma);
            const bool mx = (uemaWeight.x == 0.0f) | (blEst.x - uemaSum.x / uemaWeight.x < jt.x);
            const bool my = (uemaWeight.y == 0.0f) | (blEst.y - uemaSum.y / uemaWeight.y < jt.y);
            const float2 newWeight = add2(mulz2(f2(ma), uemaWeight, nz), f2(1.0f - ma));
            const float2 newSum = add2(mulz2(f2(ma), uemaSum, nz), mulz2(f2(1.0f - ma), blEst, nz));
            uemaWeight = f2(mx ? newWeight.x : uemaWeight.x, my ? newWeight.y : uemaWeight.y);
            uemaSum = f2(mx ? newSum.x : uemaSum.x, my ? newSum.y : uemaSum.y);
            sigmaEma = f2(mx ? newSigmaEma.x : sigmaEma.x, my ? newSigmaEma.y : sigmaEma.y);
            const float2 est = f2(uemaSum.x / uemaWeight.x, uemaSum.y / uemaWeight.y);
            const float2 sub = mulz2(est, scaler, nz);      // feeds the subtraction of every frame
            negSub = f2(-sub.x, -sub.y);
            thr = mul2(mul2(f2(4.5f), sigmaEma), scaler);
            inRange = scalerOk & (fabsf(sub.x) < 2097152.0f) & (fabsf(sub.y) < 2097152.0f);
            // AddSampleBackground (BaselinerStatAccumulator.cpp:56-60)
            const float2 bg = f2((float)to_i16_wrap(sub.x), (float)to_i16_wrap(sub.y));
            g_m1 = add2(g_m1, bg);
            g_m2 = add2(g_m2, mulz2(bg, bg, nz));
        }
        const float2 rs = mulz2(PairToFloat(SubPed(x, negPed)), scaler, nz);
        const float2 d = add2(rs, negSub);
        uint32_t bls = RoundPair(d), raw = RoundPair(rs);
        if (!inRange)
        {
            bls = RoundPairGeneral(d);
            raw = RoundPairGeneral(rs);
        }
        out[(size_t)f * (kLane / 2)] = bls;

        // AddToBaselineStats (HostMultiScaleBaseliner.cpp:148-176): the latent
        // frame is a baseline sample when it and the current one are below
        // the threshold.  As a factor of 1 or 0 in one fma per sum: v m + sum
        // rounds as v + sum for 1 and leaves the sum for 0.
        const float2 fb = PairToFloat(bls);
        const float2 hp = f2(LessAsFloat(fb.x, thr.x), LessAsFloat(fb.y, thr.y));
        const float2 m = mul2(hp1, hp);
        hp2 = hp1;
        hp1 = hp;
        {
            // BaselinerStatAccumulator::AddSample(latRaw, latData, m)
            const float2 v = latV;
            c_acm2 = add2(c_acm2, mulz2(back[Slot], v, nz));
            back[Slot] = v;
            c_m1 = add2(c_m1, v);
            const float2 vv = mulz2(v, v, nz);
            c_m2 = add2(c_m2, vv);
            tmin = MinS16x2(latData, tmin);
            tmax = MaxS16x2(latData, tmax);
            b_m0 = add2(b_m0, m);
            b_m1 = fma2(m, v, b_m1);
            b_m2 = fma2(m, vv, b_m2);
            rawSum = fma2(m, latRawV, rawSum);
        }
        latRaw = raw;
        latRawV = PairToFloat(raw);
        latData = bls;
        latV = fb;
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    using P2 = std::integral_constant<int, 2>;
    using P3 = std::integral_constant<int, 3>;
#pragma unroll 1
    for (int f = 0; f < F; f += 4)
    {
        if ((f & 15) == 0)
        {
            if (t < 16 && f + 32 + t < F) PrefetchL1(lines + (size_t)(f + 32 + t) * kLane);
            frame(P0{}, P0{}, f);
        }
        else frame(P1{}, P0{}, f);
        frame(P2{}, P1{}, f + 1);
        frame(P1{}, P2{}, f + 2);
        frame(P2{}, P3{}, f + 3);
    }

    // Store state.
    CopyWindows<FT, false, 0, true>(blSmem2 + t, stw + gp, (size_t)nPair, fs);
#pragma unroll
    for (int i = 0; i < 2 * Lay::nStages; ++i)
    {
        const bool up = i >= Lay::nStages;
        const int kk = up ? i - Lay::nStages : i;
        stw[(size_t)Lay::SlotPC(up, kk) * nPair + gp] = fs.P[i];
        stw[(size_t)(Lay::SlotPC(up, kk) + 1) * nPair + gp] = Pack16((int16_t)fs.c[kk / 2], (int16_t)fs.c[kk / 2]);
    }
    stw[(size_t)Lay::SlotLatData() * nPair + gp] = latData;
    stw[(size_t)(Lay::SlotLatData() + 1) * nPair + gp] = latRaw;
    // bits 0, 1: the last frame (latent and first history copy), 2: the one before
    auto bits = [](float last, float before) { return (int16_t)((last != 0.0f ? 3 : 0) | (before != 0.0f ? 4 : 0)); };
    stw[(size_t)(Lay::SlotLatData() + 2) * nPair + gp] = Pack16(bits(hp1.x, hp2.x), bits(hp1.y, hp2.y));
    float2* st32w = reinterpret_cast<float2*>(a.st32);
    st32w[(size_t)0 * nPair + gp] = uemaSum;
    st32w[(size_t)1 * nPair + gp] = uemaWeight;
    st32w[(size_t)2 * nPair + gp] = sigmaEma;

    // Per-chunk stats (GetState of the accumulator).
    hw_baseliner_stats& S = a.stats[lane];
    auto put = [&](float* arr, float2 v) { *reinterpret_cast<float2*>(arr + z) = v; };
    put(S.full_autocorr.basic_stats.offset, f2(0.0f));
    put(S.full_autocorr.basic_stats.moment0, f2((float)F));
    put(S.full_autocorr.basic_stats.moment1, c_m1);
    put(S.full_autocorr.basic_stats.moment2, c_m2);
    put(S.full_autocorr.moment2, c_acm2);
    // F is a multiple of 16: four samples in the front buffer, and the back
    // buffer's next slot is 0, so slot j holds the j-th oldest of the last four
    const int fbi = 4, bbi = 0;
    put(S.full_autocorr.fbuf[0], PairToFloat(firstData));
#pragma unroll
    for (int j = 0; j < 3; ++j) put(S.full_autocorr.fbuf[j + 1], PairToFloat(out[(size_t)j * (kLane / 2)]));
#pragma unroll
    for (int j = 0; j < 4; ++j) put(S.full_autocorr.bbuf[j], back[j]);
    *reinterpret_cast<uint16_t*>(&S.full_autocorr.bidx[0][z]) = (uint16_t)(fbi | (fbi << 8));
    *reinterpret_cast<uint16_t*>(&S.full_autocorr.bidx[1][z]) = (uint16_t)(bbi | (bbi << 8));
    *reinterpret_cast<uint32_t*>(&S.trace_min[z]) = tmin;
    *reinterpret_cast<uint32_t*>(&S.trace_max[z]) = tmax;
    put(S.baseline_stats.offset, f2(0.0f));
    put(S.baseline_stats.moment0, b_m0);
    put(S.baseline_stats.moment1, b_m1);
    put(S.baseline_stats.moment2, b_m2);
    put(S.raw_baseline_sum, rawSum);
    put(S.background_stats.offset, f2(0.0f));
    put(S.background_stats.moment0, f2((float)(F / 16)));
    put(S.background_stats.moment1, g_m1);
    put(S.background_stats.moment2, g_m2);
}

template <int FT>
int BaselinerSlots16() { return FLayout<FT>::NumI16Slots(); }

int BaselinerNumSlots16(int ft)
{
    switch (ft)
    {
    case 0: return BaselinerSlots16<0>();
    case 1: return BaselinerSlots16<1>();
    case 2: return BaselinerSlots16<2>();
    case 3: return BaselinerSlots16<3>();
    case 4: return BaselinerSlots16<4>();
    case 5: return BaselinerSlots16<5>();
    }
    return -1;
}

template <int FT, typename TIn, bool Mapped>
cudaError_t LaunchBaselinerT3(const BaselinerArgs& a, const KParams& k, cudaStream_t s)
{
    const int threads = kBlPairs;
    const size_t smem = sizeof(uint32_t) * FLayout<FT>::SmemSlots() * threads;
    // the shared-memory limit is a per-device attribute of the kernel: set it
    // once on each device
    static bool attrSet[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attrSet[dev])
    {
        e = cudaFuncSetAttribute(BaselinerKernel<FT, TIn, Mapped>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attrSet[dev] = true;
    }
    const int blocks = a.map.Lanes(a.lanes);
    if (blocks == 0) return cudaSuccess;
    BaselinerKernel<FT, TIn, Mapped><<<blocks, threads, smem, s>>>(a, k);
    return cudaGetLastError();
}

template <int FT, typename TIn>
cudaError_t LaunchBaselinerT2(const BaselinerArgs& a, const KParams& k, cudaStream_t s)
{
    return a.map.On() ? LaunchBaselinerT3<FT, TIn, true>(a, k, s) : LaunchBaselinerT3<FT, TIn, false>(a, k, s);
}

template <int FT>
cudaError_t LaunchBaselinerT(const BaselinerArgs& a, const KParams& k, cudaStream_t s)
{
    const bool u8 = a.map.On() ? a.u8 != 0 : a.trace8 != nullptr;
    return u8 ? LaunchBaselinerT2<FT, uint8_t>(a, k, s) : LaunchBaselinerT2<FT, int16_t>(a, k, s);
}

cudaError_t LaunchBaseliner(int ft, const BaselinerArgs& a, const KParams& k, cudaStream_t s)
{
    switch (ft)
    {
    case 0: return LaunchBaselinerT<0>(a, k, s);
    case 1: return LaunchBaselinerT<1>(a, k, s);
    case 2: return LaunchBaselinerT<2>(a, k, s);
    case 3: return LaunchBaselinerT<3>(a, k, s);
    case 4: return LaunchBaselinerT<4>(a, k, s);
    case 5: return LaunchBaselinerT<5>(a, k, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t LaunchBaselinerInit(int ft, int16_t* st16, float* st32, int lanes, cudaStream_t s)
{
    const int threads = 128;
    const int blocks = (lanes * kLane + threads - 1) / threads;
    switch (ft)
    {
    case 0: BaselinerInitKernel<0><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    case 1: BaselinerInitKernel<1><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    case 2: BaselinerInitKernel<2><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    case 3: BaselinerInitKernel<3><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    case 4: BaselinerInitKernel<4><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    case 5: BaselinerInitKernel<5><<<blocks, threads, 0, s>>>(st16, st32, lanes); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}   // namespace hwk
