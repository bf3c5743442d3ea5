// Per-frame pulse accumulation of one ZMW, shared by the pulse kernel and the
// fused labeler + pulse kernel.
//
// Restates TA/HostPulseAccumulator.{h:64-173, cpp:50-127},
// TA/SubframeLabelManager.h:47-102, DT/Pulse.h:48-237 and the bounded
// per-ZMW pulse vector of DT/BatchVectors.h:105-119
// (TA = src/basecaller/basecaller/traceAnalysis, DT = src/basecaller/dataTypes).
#pragma once

#include "hw_device.cuh"

namespace hwk {

// v is 0 or at least 2^-31 (a whole number over a width): v / .1f, with 10 the
// correctly rounded reciprocal of .1f.
__device__ __forceinline__ uint16_t ToFixed(float v)
{
    return static_cast<uint16_t>(add_rn(DivRcp(v, .1f, 10.0f), 0.5f));
}

// The open segment (LabelsSegment) and the chunk's outputs of one ZMW.  The
// int16 signals are held as floats (their sums are float sums, and the
// maximum of exact floats is that of the integers), so a frame converts its
// signal once.
struct PulseSeg
{
    uint32_t start;
    int label;
    float first, last, mx;
    float total, m2;
    uint32_t n, over;
    float b0, b1, b2;       // StatAccumulator of baseline frames (offset 0)
    float minMean;
    hw_pulse* out;
    // a closed pulse not yet converted (LabelsSegment fields at its end)
    bool pend;
    uint32_t pStart;
    int pWidth;
    float pNum, pTotal, pM2;       // (total + last) + first, total, m2
    float pMx;
    int pLabel;

    __device__ __forceinline__ void Load(const PulseArgs& A, int g, float minMeanIn, hw_pulse* outIn)
    {
        start = A.segStart[g];
        first = (float)A.segFirst[g]; last = (float)A.segLast[g]; mx = (float)A.segMax[g]; label = A.segLabel[g];
        total = A.segTotal[g]; m2 = A.segM2[g];
        n = 0; over = 0;
        b0 = 0.0f; b1 = 0.0f; b2 = 0.0f;
        minMean = minMeanIn;
        out = outIn;
        pend = false;
    }

    // LabelsSegment::ToPulse (HostPulseAccumulator.h:106-138) of the pending
    // pulse, appended to the ZMW's bounded pulse vector.
    __device__ __forceinline__ void Emit(const KParams& k)
    {
        constexpr float maxSignal = 65535 * .1f;
        constexpr float minSignal = 0.0f;
        const int width = pWidth;
        const float rawMean = pNum / (float)width;
        const float rawMid = pTotal / (float)(width - 2);
        const bool keep = ((float)width >= k.widthThresh) || (mul_rn(rawMean, (float)width) >= mul_rn(k.ampThresh, minMean));
        hw_pulse p;
        p.start = pStart;
        p.width = (uint16_t)width;
        p.mean_signal = ToFixed(fmin_std(maxSignal, fmax_std(minSignal, rawMean)));
        p.mid_signal = ToFixed(width < 3 ? 0.0f : fmin_std(maxSignal, fmax_std(minSignal, rawMid)));
        p.max_signal = ToFixed(fmin_std(maxSignal, fmax_std(minSignal, pMx)));
        p.signal_m2 = pM2;
        int lbl = pLabel;
        if (lbl > 2 * kAnalogs) lbl -= 2 * kAnalogs;
        if ((lbl > kAnalogs) & (lbl <= 2 * kAnalogs)) lbl -= kAnalogs;
        p.label = k.analogMap[lbl - 1];
        p.is_reject = keep ? 0 : 1;
        p.pad_[0] = 0; p.pad_[1] = 0;
        if (n < (uint32_t)k.maxCalls) out[n++] = p;
        else ++over;
    }

    // Converts the pending pulse, if any: called after each frame batch and
    // before Store.
    __device__ __forceinline__ void Flush(const KParams& k)
    {
        if (pend)
        {
            Emit(k);
            pend = false;
        }
    }

    // One frame with its label and signal.  The segment's sums advance by
    // selects: some ZMW of a warp starts a segment in nearly every frame, so a
    // branch would run both sides (71 -> 56 warp instructions a frame with the
    // single conversion, 613 lanes x 256 frames packed: 80 -> 66 us).
    __device__ __forceinline__ void Frame(const KParams& k, uint32_t absF, int lb, float signal)
    {
        const bool isUp = (unsigned)(lb - (kAnalogs + 1)) < (unsigned)kAnalogs;
        const bool pulseM = label != 0;
        const bool boundary = isUp | ((lb == 0) & pulseM);
        const float t1 = add_rn(total, last);
        if (boundary & pulseM)
        {
            // The pulse's raw sums wait in the pending slot; ToPulse runs at
            // the end of the frame batch, once for the whole warp, instead of
            // at every frame where some lane of the warp closes a pulse.
            if (pend) Emit(k);
            pend = true;
            pStart = start;
            pWidth = (int)(absF - start);
            pNum = add_rn(t1, first);
            pTotal = total;
            pM2 = m2;
            pMx = mx;
            pLabel = label;
        }
        const float m1 = add_rn(m2, mul_rn(last, last));
        const float mx1 = fmaxf(mx, signal);
        if (!(pulseM | boundary))
        {
            b0 += 1.0f;
            b1 = add_rn(b1, signal);
            b2 = add_rn(b2, mul_rn(signal, signal));
        }
        start = boundary ? absF : start;
        label = boundary ? lb : label;
        first = boundary ? signal : first;
        mx = boundary ? signal : mx1;
        total = boundary ? 0.0f : t1;
        m2 = boundary ? 0.0f : m1;
        last = boundary ? 0.0f : signal;
    }

    __device__ __forceinline__ void Store(const PulseArgs& A, int g, int l, int z, uint32_t* lensOut,
                                          uint32_t* ovfOut, int go) const
    {
        A.segStart[g] = start; A.segFirst[g] = (int16_t)first; A.segLast[g] = (int16_t)last;
        A.segMax[g] = (int16_t)mx;
        A.segTotal[g] = total; A.segM2[g] = m2; A.segLabel[g] = (int16_t)label;
        lensOut[go] = n;
        ovfOut[go] = over;
        A.bls[l].offset[z] = 0.0f;
        A.bls[l].moment0[z] = b0;
        A.bls[l].moment1[z] = b1;
        A.bls[l].moment2[z] = b2;
    }
};

}   // namespace hwk
