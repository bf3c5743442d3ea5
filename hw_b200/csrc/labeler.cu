// Frame labeler: ROI gating + 13-state subframe Viterbi for sm_100a.
//
// Restates TA/FrameLabelerHost.cpp:54-612, TA/SubframeScorer.h:152-318 and
// TA/RoiHost.h:75-249 (TA = src/basecaller/basecaller/traceAnalysis).
//
// One thread per ZMW.  Per chunk a thread
//   1. gathers the ROI's two threshold bits of the 24 latent frames and the
//      chunk, 32 frames a word, and runs the forward and backward recursions
//      on whole words;
//   2. runs the max-plus Viterbi over 24 latent + F-8 chunk frames + 16
//      look-ahead frames in fp32 with the reference's operation order and
//      tie rule (a later source state wins ties);
//   3. stores one traceback word per frame: the generic rows code the arg-max
//      source of each destination row, 4 bits for the 9-way rows (baseline and
//      the four pulse-up rows) and 1 bit for the 2-way rows (full and down);
//      the grouped rows the decisions that lead to it (GroupedStep);
//   4. back-propagates the normalised end-state probabilities 16 frames,
//      picks the anchor state and traces back F frames.
// Traceback words live in a global scratch laid out [lane][frame][zmw] so
// each warp writes and reads one 128-byte line per frame.
#include "pulse_seg.cuh"

namespace hwk {

// BlockStateSubframeScorer for one ZMW (SubframeScorer.h:152-318).  The
// scores of analogs 0/1 and 2/3 are evaluated as packed pairs with the
// reference's operation order (see the f32x2 helpers); constants the
// reference recomputes per frame from per-ZMW values (-0.5 times the inverse
// variances, the negated caps, means and log means, the dimmest analog's
// fallback condition) are formed once in Setup, with the same roundings
// (halving is exact, so (-0.5 y) / var is y times -0.5 / var).
struct ZScorer
{
    float bgMean, bgFixed, x0, nhBInv;
    float2 negMean[2], ffFixed[2], nhPInv[2], negX1[2], negLogP[2];
    float fbMean, fbNormTerm, fbScale;
    bool fbUse;     // x0 > x1 of the dimmest analog: its up/down score is the normal fallback
    bool ordinary;  // every constant finite: no score of an int16 trace value is NaN or infinite

    __device__ __forceinline__ void Setup(const KParams& k, const hw_lane_model& m, int z)
    {
        constexpr float log2pi_f = 1.8378770664f;
        const float nhalf = -0.5f, halfVal = 0.5f, oneSixth = 1.0f / 6.0f;
        const float bMean = h2f(m.baseline.means[z]);
        const float bVar = h2f(m.baseline.vars[z]);
        const float bSigma = sqrtf(bVar);
        x0 = add_rn(bMean, mul_rn(bSigma, k.sqrtHalfPi));
        nhBInv = mul_rn(nhalf, 1.0f / bVar);
        float aM[kAnalogs], nh[kAnalogs], fx[kAnalogs], lp[kAnalogs], xx[kAnalogs];
#pragma unroll
        for (int a = 0; a < kAnalogs; ++a)
        {
            const float aMean = h2f(m.analogs[a].means[z]);
            lp[a] = hw_logf(aMean - bMean);
            const float aVar = h2f(m.analogs[a].vars[z]);
            const float aSigma = sqrtf(aVar);
            xx[a] = aMean - mul_rn(aSigma, k.sqrtHalfPi);
            nh[a] = mul_rn(nhalf, 1.0f / aVar);
            fx[a] = mul_rn(nhalf, hw_logf(aVar)) - log2pi_f / 2.0f;
            aM[a] = aMean;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            const int a = 2 * q;
            negMean[q] = f2(-aM[a], -aM[a + 1]);
            ffFixed[q] = f2(fx[a], fx[a + 1]);
            nhPInv[q] = f2(nh[a], nh[a + 1]);
            negX1[q] = f2(-xx[a], -xx[a + 1]);
            negLogP[q] = f2(-lp[a], -lp[a + 1]);
        }
        {
            const float aMean = aM[3];
            const float aVar = h2f(m.analogs[3].vars[z]);
            const float eMean = mul_rn(halfVal, bMean + aMean);
            float eVar = mul_rn(oneSixth, aMean - bMean);
            eVar = add_rn(eVar, bVar + aVar);
            eVar = mul_rn(eVar, halfVal);
            fbMean = eMean;
            fbNormTerm = mul_rn(-0.5f, add_rn(log2pi_f, hw_logf(eVar)));
            fbScale = 0.5f / eVar;
        }
        fbUse = !(x0 <= xx[3]);
        bgFixed = mul_rn(nhalf, hw_logf(bVar)) - log2pi_f / 2.0f;
        bgMean = bMean;
        ordinary = isfinite(bgMean) & isfinite(bgFixed) & isfinite(x0) & isfinite(nhBInv) & isfinite(fbMean) &
                   isfinite(fbNormTerm) & isfinite(fbScale);
#pragma unroll
        for (int a = 0; a < kAnalogs; ++a)
            ordinary &= isfinite(aM[a]) & isfinite(nh[a]) & isfinite(fx[a]) & isfinite(lp[a]) & isfinite(xx[a]);
    }

    __device__ __forceinline__ float Background(float data) const
    {
        const float y = data - bgMean;
        return add_rn(mul_rn(mul_rn(y, nhBInv), y), bgFixed);
    }

    // StateScores for states 0..8 (states 9..12 repeat 5..8), for constants
    // and a trace value of any kind.
    __device__ __forceinline__ void Scores(float data, float* out, float2 nz) const
    {
        out[0] = Background(data);
        const float2 d2 = f2(data);
        const bool low = data < x0;
#pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            // full frame: ((-0.5 y) / var) y + fixed, y = data - mean
            const float2 y = add2(d2, negMean[q]);
            const float2 full = add2(mulz2(mul2(y, nhPInv[q]), y, nz), ffFixed[q]);
            // sub-frame Gauss cap: (extrema ? (-0.5 / var) dv^2 : 0) - log(mean - baseline mean)
            const float2 negCap = low ? f2(-x0) : negX1[q];
            const float2 fixedTerm = low ? f2(nhBInv) : nhPInv[q];
            const float2 dv = add2(d2, negCap);
            const float2 prod = mulz2(fixedTerm, mul2(dv, dv), nz);
            const bool ex = low | (data > -negX1[q].x), ey = low | (data > -negX1[q].y);
            float2 sub = add2(f2(ex ? prod.x : 0.0f, ey ? prod.y : 0.0f), negLogP[q]);
            if (q == 1 && fbUse)
            {
                const float dm = data - fbMean;
                sub.y = fbNormTerm - mul_rn(mul_rn(dm, dm), fbScale);
            }
            // clamp above the full-frame mean
            const float2 fm1 = add2(full, f2(-1.0f));
            sub.x = (data > -negMean[q].x) ? fmin_sse(fmin_sse(sub.x, fm1.x), 0.0f) : sub.x;
            sub.y = (data > -negMean[q].y) ? fmin_sse(fmin_sse(sub.y, fm1.y), 0.0f) : sub.y;
            out[1 + 2 * q] = full.x;
            out[2 + 2 * q] = full.y;
            out[5 + 2 * q] = sub.x;
            out[6 + 2 * q] = sub.y;
        }
    }

    // The same scores for `ordinary` constants, as the pairs of analogs 0/1
    // and 2/3.  With nothing NaN the clamps are plain minima; the cap's
    // "extrema" selection is a maximum with 0 (its square term is then -0,
    // which changes no sum); the baseline side of the cap does not depend on
    // the analog.
    __device__ __forceinline__ void OrdinaryScores(float data, float& s0, float2 (&fullS)[2], float2 (&subS)[2],
                                                   float2 nz) const
    {
        s0 = Background(data);
        const float2 d2 = f2(data);
        const bool low = data < x0;
        const float dl = data - x0;
        const float lowProd = mul_rn(nhBInv, mul_rn(dl, dl));
#pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            const float2 y = add2(d2, negMean[q]);
            const float2 full = add2(mulz2(mul2(y, nhPInv[q]), y, nz), ffFixed[q]);
            float2 dv = add2(d2, negX1[q]);
            dv = f2(fmaxf(dv.x, 0.0f), fmaxf(dv.y, 0.0f));
            const float2 prod = mulz2(nhPInv[q], mul2(dv, dv), nz);
            float2 sub = add2(f2(low ? lowProd : prod.x, low ? lowProd : prod.y), negLogP[q]);
            if (q == 1)
            {
                const float dm = data - fbMean;
                const float fb = fbNormTerm - mul_rn(mul_rn(dm, dm), fbScale);
                sub.y = fbUse ? fb : sub.y;
            }
            const float2 fm1 = add2(full, f2(-1.0f));
            const float cx = min3(sub.x, fm1.x, 0.0f), cy = min3(sub.y, fm1.y, 0.0f);
            fullS[q] = full;
            subS[q] = f2(y.x > 0.0f ? cx : sub.x, y.y > 0.0f ? cy : sub.y);
        }
    }
};

// Log-likelihoods of the 13 states between Viterbi steps: state 0 alone,
// states 1..12 in the pairs (1,2) (3,4) (5,6) (7,8) (9,10) (11,12) that the
// rows add as one f32x2 operation (every row reads its sources pairwise:
// the 9-way rows (5,6) .. (11,12), the 2-way rows of states r and r + 1 read
// (r, r + 1) and (r + 4, r + 5) or (r - 8, r - 7) and (r - 4, r - 3)).
struct StateLL
{
    float s0;
    float2 p[6];
    __device__ __forceinline__ float Get(int i) const
    {
        return i == 0 ? s0 : (((i - 1) & 1) ? p[(i - 1) >> 1].y : p[(i - 1) >> 1].x);
    }
    __device__ __forceinline__ void Set(int i, float v)
    {
        if (i == 0) s0 = v;
        else if ((i - 1) & 1) p[(i - 1) >> 1].y = v;
        else p[(i - 1) >> 1].x = v;
    }
};

// Arg-max over a row's candidates in the reference's order (first entry,
// then the contiguous segment); ties go to the later entry (Recursion,
// FrameLabelerHost.cpp:214-264).  The candidate values are
// (score + T[row][src]) + ll[src]: the first addition per candidate, the
// second pairwise.  Instead of the source state a row returns its traceback
// code already shifted into place: 9-way rows (baseline, pulse-up) code
// source s as 0 for state 0 and s - 4 for states 5..12 in 4 bits; 2-way
// rows (full, down) code the second source as one bit, the outcome of their
// single comparison.  With Margin, `gap` receives the row's decision gap:
// the winning candidate less the best other one (0 on a tie, +inf when only
// one is finite).
template <bool Margin>
__device__ __forceinline__ void Pick(float v, uint32_t cv, float& mv, float& sv, uint32_t& c)
{
    const bool ge = v >= mv;
    if constexpr (Margin) sv = ge ? mv : ((v > sv) ? v : sv);
    mv = ge ? v : mv;
    c = ge ? cv : c;
}

template <int R, bool Margin>
__device__ __forceinline__ float NineWayRow(const KParams& k, float score, const StateLL& ll, uint32_t& code,
                                            float& gap)
{
    constexpr int shift = (R == 0) ? 0 : 4 + 4 * (R - 5);
    float mv = add_rn(add_rn(score, k.trans[R][0]), ll.s0);
    float sv = -__int_as_float(0x7f800000);
    uint32_t c = 0u;
#pragma unroll
    for (int q = 2; q < 6; ++q)
    {
        const int p0 = 2 * q + 1;          // sources p0, p0 + 1
        const float2 v = add2(add2(f2(score), f2(k.trans[R][p0], k.trans[R][p0 + 1])), ll.p[q]);
        Pick<Margin>(v.x, (uint32_t)(p0 - 4) << shift, mv, sv, c);
        Pick<Margin>(v.y, (uint32_t)(p0 - 3) << shift, mv, sv, c);
    }
    code = c;
    if constexpr (Margin) gap = mv - sv;
    return mv;
}

// Two 2-way rows, R and R + 1, with scores s.x, s.y: their first sources are
// the pair qa, their second the pair qb.
template <int R, int qa, int qb, bool Margin>
__device__ __forceinline__ float2 TwoWayRows(const KParams& k, float2 s, const StateLL& ll, uint32_t& code,
                                             float& gap0, float& gap1)
{
    constexpr int shift = (R <= 4) ? 20 + R - 1 : 24 + R - 9;
    constexpr int a0 = 2 * qa + 1, b0 = 2 * qb + 1;
    const float2 first = add2(add2(s, f2(k.trans[R][a0], k.trans[R + 1][a0 + 1])), ll.p[qa]);
    const float2 second = add2(add2(s, f2(k.trans[R][b0], k.trans[R + 1][b0 + 1])), ll.p[qb]);
    const bool gx = second.x >= first.x, gy = second.y >= first.y;
    if constexpr (Margin)
    {
        const float ninf = -__int_as_float(0x7f800000);
        const float sx = gx ? first.x : ((second.x > ninf) ? second.x : ninf);
        const float sy = gy ? first.y : ((second.y > ninf) ? second.y : ninf);
        gap0 = (gx ? second.x : first.x) - sx;
        gap1 = (gy ? second.y : first.y) - sy;
    }
    code = (gx ? 1u << shift : 0u) | (gy ? 2u << shift : 0u);
    return f2(gx ? second.x : first.x, gy ? second.y : first.y);
}

// One Viterbi recursion step over the generic rows; returns the packed
// traceback word.  With Margin, gap[r] receives row r's decision gap.
template <bool Margin>
__device__ __forceinline__ uint32_t ViterbiStep(const KParams& k, const ZScorer& sc, float data, float npen,
                                                StateLL& ll, float* gap = nullptr)
{
    float sco[9];
    sc.Scores(data, sco, f2(k.negZero));
    uint32_t cd[9];
    float gl[kStates];
    const float n0 = NineWayRow<0, Margin>(k, sco[0], ll, cd[0], gl[0]);
    const float n5 = NineWayRow<5, Margin>(k, sco[5], ll, cd[1], gl[5]);
    const float n6 = NineWayRow<6, Margin>(k, sco[6], ll, cd[2], gl[6]);
    const float n7 = NineWayRow<7, Margin>(k, sco[7], ll, cd[3], gl[7]);
    const float n8 = NineWayRow<8, Margin>(k, sco[8], ll, cd[4], gl[8]);
    // full rows: (r, r + 4); down rows: (r - 8, r - 4)
    const float2 n12 = TwoWayRows<1, 0, 2, Margin>(k, f2(sco[1], sco[2]), ll, cd[5], gl[1], gl[2]);
    const float2 n34 = TwoWayRows<3, 1, 3, Margin>(k, f2(sco[3], sco[4]), ll, cd[6], gl[3], gl[4]);
    const float2 n9a = TwoWayRows<9, 0, 2, Margin>(k, f2(sco[5], sco[6]), ll, cd[7], gl[9], gl[10]);
    const float2 nbc = TwoWayRows<11, 1, 3, Margin>(k, f2(sco[7], sco[8]), ll, cd[8], gl[11], gl[12]);
    // non-ROI frames: every state but the baseline gets -inf (x - inf)
    const float2 pen = f2(npen);
    ll.s0 = n0;
    ll.p[0] = add2(n12, pen);
    ll.p[1] = add2(n34, pen);
    ll.p[2] = add2(f2(n5, n6), pen);
    ll.p[3] = add2(f2(n7, n8), pen);
    ll.p[4] = add2(n9a, pen);
    ll.p[5] = add2(nbc, pen);
    if constexpr (Margin)
    {
#pragma unroll
        for (int r = 0; r < kStates; ++r) gap[r] = gl[r];
    }
    return ((cd[0] | cd[1] | cd[2]) | (cd[3] | cd[4])) | ((cd[5] | cd[6]) | (cd[7] | cd[8]));
}

// acc shifted left by n with the top n bits of v: n = 1 appends v's sign.
template <int n> __device__ __forceinline__ uint32_t PushTop(uint32_t acc, float v)
{
    return __funnelshift_l(__float_as_uint(v), acc, n);
}
// b - a of both components, rounded once (the product by -1 is exact).
__device__ __forceinline__ float2 sub2(float2 b, float2 a) { return fma2(a, f2(-1.0f), b); }

// Traceback word of a grouped step that took the generic rows: their word
// shifted by kGenericShift, with kGenericWord set.
constexpr uint32_t kGenericWord = 4u;
constexpr int kGenericShift = 3;

// The step when the 9-way rows' transition constants are equal within each
// source group (t_A for states 5..8, t_B for 9..12; KParams::grouped9).
//
// A row's candidates of group G are RN(a_G + ll[s]) with a_G = RN(score + t_G)
// the same for the whole group, and RN(a_G + x) is monotone in x: the group's
// best candidate is RN(a_G + m_G), m_G the group's largest ll.  It belongs to
// the last state holding m_G unless another state's sum rounds to the same
// value, which needs their ll to differ by no more than 2^-22 |a_G + m_G|.  So
// m_G and its position are found once for the five rows, by two rounds of
// pairwise comparisons, and a frame where one of a group's comparisons is
// closer than 2^-21 (|score| + |t| + |m_G|) over all rows, or whose scorer is
// not `ordinary` or whose log-likelihoods came with a NaN (bad), takes the
// generic rows.
//
// Every decision "the later candidate is at least the earlier one" is the sign
// of their difference: 0 for yes (also for equal values and for two -inf,
// whose difference is the positive quiet NaN; ll never holds -0 or +inf).  So
// a value needs one maximum and a decision one subtraction (FMA pipe) and one
// funnel shift that appends the sign to the traceback word: with compares and
// selects instead (422 thread instructions a ZMW-frame over the kernel, 68% of
// the ALU pipe) 4096 lanes x 512 frames took 2145 us; now 293, 55% and 1560 us.
// Issue and ALU latency bound it now (65% of issue slots at 5 warps a
// scheduler, the most that 96 registers allow; 4 and 6 warps measured 1659 and
// 1616 us).
//
// Word: bit 2 s + 1 of state s is its last decision (0: the later of two
// sources, or group B), bit 2 s of a 9-way state the decision before it (0:
// group A, 1: state 0); bits 31..29 and 28..26 hold the comparisons of groups A
// and B: 6 against 5, 8 against 7 and the second against the first pair
// (likewise 9..12).  Bit 2 is kGenericWord.
__device__ __forceinline__ uint32_t GroupedStep(const KParams& k, const ZScorer& sc, float data, float npen, bool bad,
                                                StateLL& ll)
{
    const float2 nz = f2(k.negZero);
    float s0;
    float2 full[2], sub[2];
    sc.OrdinaryScores(data, s0, full, sub, nz);
    const float hA1 = fmaxf(ll.p[2].x, ll.p[2].y), hA2 = fmaxf(ll.p[3].x, ll.p[3].y), mA = fmaxf(hA1, hA2);
    const float hB1 = fmaxf(ll.p[4].x, ll.p[4].y), hB2 = fmaxf(ll.p[5].x, ll.p[5].y), mB = fmaxf(hB1, hB2);
    const float eA1 = ll.p[2].y - ll.p[2].x, eA2 = ll.p[3].y - ll.p[3].x, eA3 = hA2 - hA1;
    const float eB1 = ll.p[4].y - ll.p[4].x, eB2 = ll.p[5].y - ll.p[5].x, eB3 = hB2 - hB1;
    // an empty group (all -inf) has NaN differences: not slow
    const float sMax = max3(max3(fabsf(s0), fabsf(sub[0].x), fabsf(sub[0].y)), fabsf(sub[1].x), fabsf(sub[1].y));
    const float tol = fma_rn(sMax, kGrpTol, k.grpTol);
    const bool slow = bad | (min3(fabsf(eA1), fabsf(eA2), fabsf(eA3)) <= fma_rn(fabsf(mA), kGrpTol, tol)) |
                      (min3(fabsf(eB1), fabsf(eB2), fabsf(eB3)) <= fma_rn(fabsf(mB), kGrpTol, tol));
    if (slow) return (ViterbiStep<false>(k, sc, data, npen, ll) << kGenericShift) | kGenericWord;

    uint32_t hi = PushTop<1>(0u, eA1);
    hi = PushTop<1>(hi, eA2);
    hi = PushTop<1>(hi, eA3);
    hi = PushTop<1>(hi, eB1);
    hi = PushTop<1>(hi, eB2);
    hi = PushTop<1>(hi, eB3);
    const float2 l0 = f2(ll.s0), gA = f2(mA), gB = f2(mB);
    float2 dUA[2], dUB[2], dF[2], dD[2], nU[2], nF[2], nD[2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
    {
        const float2 c0 = add2(add2(sub[q], k.grpUp0[q]), l0);
        const float2 cA = add2(add2(sub[q], k.grpUpA[q]), gA);
        const float2 cB = add2(add2(sub[q], k.grpUpB[q]), gB);
        nU[q] = f2(max3(c0.x, cA.x, cB.x), max3(c0.y, cA.y, cB.y));
        dUA[q] = sub2(cA, c0);
        dUB[q] = sub2(cB, nU[q]);
        const float2 f1 = add2(add2(full[q], k.grpTwo[q][0]), ll.p[q]);
        const float2 f2_ = add2(add2(full[q], k.grpTwo[q][1]), ll.p[2 + q]);
        nF[q] = f2(fmaxf(f1.x, f2_.x), fmaxf(f1.y, f2_.y));
        dF[q] = sub2(f2_, f1);
        const float2 d1 = add2(add2(sub[q], k.grpTwo[2 + q][0]), ll.p[q]);
        const float2 d2 = add2(add2(sub[q], k.grpTwo[2 + q][1]), ll.p[2 + q]);
        nD[q] = f2(fmaxf(d1.x, d2.x), fmaxf(d1.y, d2.y));
        dD[q] = sub2(d2, d1);
    }
    const float c0 = add_rn(add_rn(s0, k.grpRow0[0]), ll.s0);
    const float cA = add_rn(add_rn(s0, k.grpRow0[1]), mA);
    const float cB = add_rn(add_rn(s0, k.grpRow0[2]), mB);
    const float n0 = max3(c0, cA, cB);
    hi = PushTop<2>(hi, dD[1].y);
    hi = PushTop<2>(hi, dD[1].x);
    hi = PushTop<2>(hi, dD[0].y);
    hi = PushTop<2>(hi, dD[0].x);
    hi = PushTop<1>(hi, dUB[1].y);
    hi = PushTop<1>(hi, dUA[1].y);
    uint32_t lo = PushTop<1>(0u, dUB[1].x);
    lo = PushTop<1>(lo, dUA[1].x);
    lo = PushTop<1>(lo, dUB[0].y);
    lo = PushTop<1>(lo, dUA[0].y);
    lo = PushTop<1>(lo, dUB[0].x);
    lo = PushTop<1>(lo, dUA[0].x);
    lo = PushTop<2>(lo, dF[1].y);
    lo = PushTop<2>(lo, dF[1].x);
    lo = PushTop<2>(lo, dF[0].y);
    lo = PushTop<2>(lo, dF[0].x);
    lo = PushTop<1>(lo, cB - n0);
    lo = PushTop<1>(lo, cA - c0);
    // non-ROI frames: every state but the baseline gets -inf (x - inf)
    const float2 pen = f2(npen);
    ll.s0 = n0;
#pragma unroll
    for (int q = 0; q < 2; ++q)
    {
        ll.p[q] = add2(nF[q], pen);
        ll.p[2 + q] = add2(nU[q], pen);
        ll.p[4 + q] = add2(nD[q], pen);
    }
    return __byte_perm(lo, hi, 0x5410) & ~kGenericWord;
}

// Source state of `state` recorded in a generic step's traceback word `w`.
__device__ __forceinline__ int GenericSource(uint32_t w, int state)
{
    if (state == 0 || state >= 5 && state <= 8)
    {
        const int shift = (state == 0) ? 0 : 4 + 4 * (state - 5);
        const int c = (w >> shift) & 15u;
        return c == 0 ? 0 : c + 4;
    }
    if (state <= 4)
    {
        const int b = (w >> (20 + state - 1)) & 1u;
        return b ? state + 4 : state;
    }
    const int b = (w >> (24 + state - 9)) & 1u;
    return b ? state - 4 : state - 8;
}

// Source state of `state` recorded in traceback word `w`.  The two-way rows of
// an analog (full and down) choose between its full state (first) and its up
// state; a 9-way row between state 0, the up state and the down state of its
// group's largest ll, whose position (0..3) the group's three comparisons give
// through a table of two bits an entry.
template <bool Grouped> __device__ __forceinline__ int TraceSource(uint32_t w, int state)
{
    if (!Grouped) return GenericSource(w, state);
    if (w & kGenericWord) return GenericSource(w >> kGenericShift, state);
    const uint32_t v = w >> (2 * state);
    const uint32_t first = (v >> 1) & 1u;              // not the last source (group)
    const uint32_t nine = (0x1e1u >> state) & 1u;
    const uint32_t pos = (0x2367u >> ((w >> (25u + 3u * first)) & 14u)) & 3u;
    const uint32_t sub = nine ? pos : (uint32_t)(state + 3) & 3u;
    const int src = (int)(5u + 4u * nine - 4u * first + sub);
    return (nine & v) & first ? 0 : src;
}

// Moves each state's probability to its source in a grouped step's word:
// np[to] is the sum over the states with that source, in state order.  The
// word's structure names the few states that can reach a source, so a third
// of the selections of a general scatter are needed; a state that does not
// reach it adds +0.
__device__ __forceinline__ void GroupedBackStep(uint32_t w, const float (&p)[kStates], float (&np)[kStates])
{
    auto bit = [&](int i) { return ((w >> i) & 1u) != 0u; };
    constexpr int nine[5] = {0, 5, 6, 7, 8};
    float z[5], a[5], b[5];       // to state 0, group A, group B
#pragma unroll
    for (int i = 0; i < 5; ++i)
    {
        const int s = nine[i];
        const bool lastB = !bit(2 * s + 1), viaA = !bit(2 * s);
        b[i] = lastB ? p[s] : 0.0f;
        const float rest = lastB ? 0.0f : p[s];
        a[i] = viaA ? rest : 0.0f;
        z[i] = viaA ? 0.0f : rest;
    }
    np[0] = add_rn(add_rn(add_rn(add_rn(z[0], z[1]), z[2]), z[3]), z[4]);
    const uint32_t posA = (0x2367u >> ((w >> 28) & 14u)) & 3u, posB = (0x2367u >> ((w >> 25) & 14u)) & 3u;
#pragma unroll
    for (int u = 0; u < 4; ++u)
    {
        const bool fFull = bit(2 * (1 + u) + 1), fDown = bit(2 * (9 + u) + 1);     // first source
        np[1 + u] = add_rn(fFull ? p[1 + u] : 0.0f, fDown ? p[9 + u] : 0.0f);
        const bool inA = posA == (uint32_t)u, inB = posB == (uint32_t)u;
        float t = add_rn(inA ? a[0] : 0.0f, fFull ? 0.0f : p[1 + u]);
        float v = inB ? b[0] : 0.0f;
#pragma unroll
        for (int i = 1; i < 5; ++i)
        {
            t = inA ? add_rn(t, a[i]) : t;
            v = inB ? add_rn(v, b[i]) : v;
        }
        np[5 + u] = add_rn(t, fDown ? 0.0f : p[9 + u]);
        np[9 + u] = v;
    }
}

// x / c, correctly rounded, for the ROI's constants c = sqrt(2) and sqrt(3)
// and finite x: q = x * RN(1/c) corrected once with the exact remainder x - q c
// (Markstein's correction).  An exhaustive check over every float x gives the
// IEEE quotient for both constants whenever |x| >= 2^-100 (the largest x that
// differs is below 2^-102), and zero for zero; only smaller x can differ, and
// the ROI never divides one (its dividends are 0 or sums of int16 trace values
// times an inverse sigma of at least 1/256, so their magnitude is 0 or above
// 2^-33).
__device__ __forceinline__ float DivByConst(float x, float c, float rcp)
{
    const float q = mul_rn(x, rcp);
    return fma_rn(fma_rn(-q, c, x), rcp, q);
}

// A trace value by the coherent path, for memory that this kernel also writes
// (the latent traces, overwritten at its end; the read-only path requires that
// nobody does).  As asm without a memory clobber it can still be issued ahead
// of the traceback stores: 1562 us on the case of GroupedStep, as with the
// read-only path, where a plain load takes 1652.
__device__ __forceinline__ int16_t LoadI16(const int16_t* p)
{
    int16_t v;
    asm("ld.global.s16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// The ROI's statistic with the reference's maxima and divisions, for values
// that may be infinite or NaN.
__device__ __noinline__ float RoiValueGeneral(float p1, float s2, float s3, float s4, float sqrt2, float sqrt3)
{
    float mval = fmax_sse(p1, s2 / sqrt2);
    mval = fmax_sse(mval, s3 / sqrt3);
    return fmax_sse(mval, s4 / 2.0f);
}

constexpr int kBatch = 8;                              // frames loaded ahead

// Blocks per SM the labeler variants are compiled for (96 registers a thread:
// the grouped step spills 4 bytes in the single-pool kernel, 48 in the mapped
// one, 28 in the mapped one with the pulses; GroupedStep has
// the times of other block counts).
constexpr int LabelerMinBlocks(int threads) { return threads == 64 ? 10 : threads == 128 ? 5 : 2; }

// Mapped: lane-list launch.  Fuse: the pulse accumulator runs in the same
// thread right after the traceback, on labels kept in shared memory (4 bits a
// frame) instead of a labels batch in global memory.  Threads: 64 ZMWs (one
// lane) per 64 threads.
// Margin (single-pool launch only): the decision gaps of every frame and
// state go to the scratch A.gap [lanes][F + 16][13][64], and the traceback
// writes each label's best-path margin to A.margin.
template <bool Mapped, bool Fuse, int Threads, bool Margin = false, bool Grouped = false>
__global__ void __launch_bounds__(Threads, LabelerMinBlocks(Threads)) LabelerKernel(LabelerArgs A, KParams k,
                                                                                     PulseArgs P)
{
    static_assert(!Margin || (!Mapped && !Fuse), "margins come from the single-pool labeler");
    static_assert(!(Margin && Grouped), "margins come from the generic rows");
    LaneMap map = A.map;
    if (!Mapped) map.list = nullptr;      // the single-pool variant compiles without the lane list
    int l, z;
    if (!ZmwOf(map, A.lanes, l, z)) return;
    const int g = l * kLane + z;
    const int F = map.On() ? map.Pool(l).F : A.F;
    const int16_t* chunk = A.trace + map.Block(l, F) + z;
    int16_t* pl = A.prevLat + (size_t)l * kLatent * kLane + z;
    const hw_lane_model& oldM = A.latModel[l];
    const hw_lane_model& newM = A.models[l];

    // ---- ROI (ComputeRoi, FrameLabelerHost.cpp:267-309; RoiHost.h:110-249)
    // One bit a frame, 32 frames a word with the earliest in bit 31, in
    // dynamic shared memory [word][thread] (kept out of local memory, whose
    // L1 share depends on other kernels' shared-memory carve-out).  Bit v is
    // frame v - 2 of the ROI block (v - 2 < F + kLookback + kStitch): with two
    // leading bits that pass the previous chunk's last ROI value on, the 22
    // latent frames and the chunk's batches of 8 end on whole bytes.
    extern __shared__ uint32_t roiSh[];
    auto roiw = [&](int w) -> uint32_t& { return roiSh[w * blockDim.x + threadIdx.x]; };
    const int nWords = (F + kLatent + 31) / 32;
    {
        const float inv1 = 1.0f / sqrtf(h2f(oldM.baseline.vars[z]));
        const float inv2 = 1.0f / sqrtf(h2f(newM.baseline.vars[z]));
        float p0 = mul_rn((float)A.latTrc[g], inv1);
        float p1 = mul_rn((float)pl[0], inv1);
        float p2 = mul_rn((float)pl[kLane], inv1);
        uint32_t prevRoi = (uint16_t)A.latRoi[g] & 1u;
        // a baseline variance of 0, infinity (every statistic is then 0 or
        // -0, whose difference to a threshold of 0 has either sign) or NaN, or
        // a NaN threshold: comparisons instead of signs, with the reference's
        // maxima
        const bool plain = isfinite(inv1) & isfinite(inv2) & (inv1 > 0.0f) & (inv2 > 0.0f) & !isnan(k.roiUpper) &
                           !isnan(k.roiLower);
        // complements of the bits, most recent frame in bit 0
        uint32_t nu = prevRoi ? 1u : 3u, nl = 0u;
        auto process = [&](float sn) {
            const float s2 = p0 + p1, s3 = add_rn(s2, p2), s4 = add_rn(s3, sn);
            if (plain)
            {
                const float mval = fmaxf(max3(p1, DivByConst(s2, k.sqrt2, k.rcpSqrt2),
                                              DivByConst(s3, k.sqrt3, k.rcpSqrt3)), mul_rn(s4, 0.5f));
                nu = PushTop<1>(nu, mval - k.roiUpper);
                nl = PushTop<1>(nl, mval - k.roiLower);
            }
            else
            {
                const float mval = RoiValueGeneral(p1, s2, s3, s4, k.sqrt2, k.sqrt3);
                nu = (nu << 1) | ((mval >= k.roiUpper) ? 0u : 1u);
                nl = (nl << 1) | ((mval >= k.roiLower) ? 0u : 1u);
            }
            p0 = p1; p1 = p2; p2 = sn;
        };
        // Forward recursion over a word of upper (u) and lower (l) threshold
        // bits: f = u | (l & previous f), by doubling steps; the carry is the
        // previous word's last bit.  With the upper threshold below the lower
        // one (previous f ? l : u), frame by frame.
        const bool nested = k.roiUpper >= k.roiLower;
        auto forward = [&](uint32_t u, uint32_t lw, uint32_t carry) -> uint32_t {
            if (nested)
            {
                uint32_t f = u | ((carry << 31) & lw), c = lw;
#pragma unroll
                for (int d = 1; d < 32; d *= 2)
                {
                    f |= c & (f >> d);
                    c &= c >> d;
                }
                return f;
            }
            uint32_t f = 0u;
            for (int j = 31; j >= 0; --j)
            {
                carry = ((carry ? lw : u) >> j) & 1u;
                f |= carry << j;
            }
            return f;
        };
        // forward words in roiw[0, nWords), lower-threshold words after them
        auto flush = [&](int w, uint32_t u, uint32_t lw) {
            const uint32_t f = forward(u, lw, prevRoi);
            prevRoi = f & 1u;
            roiw(w) = f;
            roiw(nWords + w) = lw;
        };
        for (int i = hwp::kRoiLookForward; i < kLatent; ++i) process(mul_rn((float)pl[(size_t)i * kLane], inv1));
        int16_t x[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) x[j] = __ldg(chunk + (size_t)j * kLane);
        for (int f0 = 0; f0 < F; f0 += kBatch)
        {
            int16_t xn[kBatch];
            const int fn = f0 + kBatch < F ? f0 + kBatch : f0;
#pragma unroll
            for (int j = 0; j < kBatch; ++j) xn[j] = __ldg(chunk + (size_t)(fn + j) * kLane);
#pragma unroll
            for (int j = 0; j < kBatch; ++j) process(mul_rn((float)x[j], inv2));
#pragma unroll
            for (int j = 0; j < kBatch; ++j) x[j] = xn[j];
            const int v = f0 + kLatent + kBatch;
            if ((v & 31) == 0) flush((v >> 5) - 1, ~nu, ~nl);
        }
        const int rest = (F + kLatent) & 31;
        if (rest) flush(nWords - 1, ~nu << (32 - rest), ~nl << (32 - rest));
        // Backward recursion: b = f | (l & following b).
        uint32_t next = 0u;
        for (int w = nWords - 1; w >= 0; --w)
        {
            uint32_t b = roiw(w), c = roiw(nWords + w);
            b |= c & next;
#pragma unroll
            for (int d = 1; d < 32; d *= 2)
            {
                b |= c & (b << d);
                c &= c << d;
            }
            next = b >> 31;
            roiw(w) = b;
        }
    }
    auto roiBit = [&](int f) -> bool { return (roiw((f + 2) >> 5) >> (31 - ((f + 2) & 31))) & 1u; };

    // ---- Viterbi (LabelBlock, FrameLabelerHost.cpp:314-448)
    StateLL ll;
    {
        const int bc = A.latLabel[g];
#pragma unroll
        for (int i = 0; i < kStates; ++i) ll.Set(i, (bc == i) ? 0.0f : -__int_as_float(0x7f800000));
    }
    uint32_t* tb = A.tb + map.BlockX(l, F, kLookback) + z;
    // decision gap of state r at frame lf
    auto gapAt = [&](int lf, int r) -> float& {
        return A.gap[(((size_t)l * (F + kLookback) + lf) * kStates + r) * kLane + z];
    };
    ZScorer sc;
    // The latent frames (old model), the chunk's frames up to the anchor and
    // the 16 look-ahead frames after it (labels kLatent .. F + 15) share one
    // copy of the step, which is several hundred instructions.  The trace is
    // loaded two frames ahead of use.  The log-likelihoods at the anchor wait
    // in the ROI words' second half, which the backward recursion has used up.
    auto anchorLL = [&](int i) -> float& { return reinterpret_cast<float&>(roiw(nWords + i)); };
    const int nSteps = F + kLookback;
#pragma unroll 1
    for (int lf = 0; lf < nSteps;)
    {
        const int16_t* src = lf < kLatent ? pl : chunk - (size_t)kLatent * kLane;
        const int end = lf < kLatent ? kLatent : lf < F ? F : nSteps;
        if (lf < F) sc.Setup(k, lf < kLatent ? oldM : newM, z);
        else
        {
#pragma unroll
            for (int i = 0; i < kStates; ++i) anchorLL(i) = ll.Get(i);
        }
        // A NaN (or +inf) that the old model's scores left in the
        // log-likelihoods is kept by the generic rows' comparisons and would
        // be dropped by GroupedStep's maxima: the new model's segment takes
        // the generic rows then, however ordinary the model.
        float sum = ll.s0;
#pragma unroll
        for (int q = 0; q < 6; ++q) sum += add_rn(ll.p[q].x, ll.p[q].y);
        const bool bad = !sc.ordinary | !(sum < __int_as_float(0x7f800000));
        uint32_t roiWord = ~roiw((lf + 2) >> 5) << ((lf + 2) & 31);
        int16_t x0 = LoadI16(src + (size_t)lf * kLane);
        int16_t x1 = LoadI16(src + (size_t)(lf + 1 < end ? lf + 1 : lf) * kLane);
#pragma unroll 1
        for (; lf < end; ++lf)
        {
            const float x = (float)x0;
            x0 = x1;
            if (lf + 2 < end) x1 = LoadI16(src + (size_t)(lf + 2) * kLane);
            if (((lf + 2) & 31) == 0) roiWord = ~roiw((lf + 2) >> 5);
            // 0 on an ROI frame, -inf on another
            const float npen = __int_as_float(((int)roiWord >> 31) & (int)0xff800000);
            roiWord <<= 1;
            uint32_t w;
            if constexpr (Margin)
            {
                float gp[kStates];
                w = ViterbiStep<true>(k, sc, x, npen, ll, gp);
#pragma unroll
                for (int r = 0; r < kStates; ++r) gapAt(lf, r) = gp[r];
            }
            else if constexpr (Grouped) w = GroupedStep(k, sc, x, npen, bad, ll);
            else w = ViterbiStep<false>(k, sc, x, npen, ll);
            tb[(size_t)lf * kLane] = w;
        }
    }
    const int anchor = F - kLatent;

    // Normalize (FrameLabelerHost.cpp:186-205) and back-propagation.
    float prob[kStates];
    {
        float mx = ll.Get(0);
#pragma unroll
        for (int i = 1; i < kStates; ++i) mx = fmax_sse(ll.Get(i), mx);
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < kStates; ++i) { prob[i] = hw_expf(ll.Get(i) - mx); sum = add_rn(sum, prob[i]); }
        const float inv = 1.0f / sum;
#pragma unroll
        for (int i = 0; i < kStates; ++i) prob[i] = mul_rn(prob[i], inv);
    }
    for (int i = F + kLookback - 1; i > F - 1; --i) PrefetchL1(tb + (size_t)i * kLane);
    for (int i = F + kLookback - 1; i > F - 1; --i)
    {
        const uint32_t w = tb[(size_t)i * kLane];
        float np[kStates];
        if (Grouped && !(w & kGenericWord)) GroupedBackStep(w, prob, np);
        else
        {
#pragma unroll
            for (int s = 0; s < kStates; ++s) np[s] = 0.0f;
#pragma unroll
            for (int from = 0; from < kStates; ++from)
            {
                const int to = GenericSource(Grouped ? w >> kGenericShift : w, from);
#pragma unroll
                for (int s = 0; s < kStates; ++s) np[s] = (s == to) ? add_rn(np[s], prob[from]) : np[s];
            }
        }
#pragma unroll
        for (int s = 0; s < kStates; ++s) prob[s] = np[s];
    }
    float maxP = prob[0];
    int anchorState = 0;
#pragma unroll
    for (int i = 1; i < kStates; ++i)
    {
        const bool c = maxP > prob[i];
        maxP = c ? maxP : prob[i];
        anchorState = c ? anchorState : i;
    }
    const float ret = anchorLL(anchorState);

    int ts = anchorState;
    if constexpr (Fuse)
    {
        // The ROI words are done with: the last ROI bit goes to the latent
        // state first, then the traceback packs 8 labels a word into them.
        A.latRoi[g] = (int16_t)roiBit(F - 1);
        for (int f0 = F - kBatch; f0 >= 0; f0 -= kBatch)
        {
            uint32_t w[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) w[j] = tb[(size_t)(f0 + j) * kLane];
            if (f0 >= kBatch)
            {
#pragma unroll
                for (int j = 0; j < kBatch; ++j) PrefetchL1(tb + (size_t)(f0 - kBatch + j) * kLane);
            }
            uint32_t word = 0;
#pragma unroll
            for (int j = kBatch - 1; j >= 0; --j)
            {
                word |= (uint32_t)ts << (4 * j);
                ts = TraceSource<Grouped>(w[j], ts);
            }
            roiw(f0 / kBatch) = word;
        }
        // Pulse accumulation over the labels batch (frames chunk start - 24
        // .. chunk end - 24): the previous chunk's latent frames, then the
        // chunk's first F - 24 frames.
        const PoolStep& ps = map.Pool(l);
        const int go = (l - ps.lane0) * kLane + z;
        const uint32_t firstFrame = (uint32_t)(ps.firstFrame - kLatent);
        PulseSeg seg;
        seg.Load(P, g, h2f(newM.analogs[kAnalogs - 1].means[z]), ps.pulses + (size_t)go * k.maxCalls);
        for (int r0 = 0; r0 < F; r0 += kBatch)
        {
            const uint32_t word = roiw(r0 / kBatch);
            int16_t sg[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j)
            {
                const int r = r0 + j;
                sg[j] = (r < kLatent) ? pl[(size_t)r * kLane] : __ldg(chunk + (size_t)(r - kLatent) * kLane);
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j)
                seg.Frame(k, (uint32_t)(r0 + j) + firstFrame, (int)((word >> (4 * j)) & 15u), I16ToFloat(sg[j]));
            seg.Flush(k);
        }
        seg.Store(P, g, l, z, ps.lens, ps.ovf, go);
    }
    else if constexpr (Margin)
    {
        // Traceback with the best path's decision margin of every label: the
        // last label's is the anchor choice's probability gap, label f's the
        // gap that frame f + 1 recorded for the path's state there.
        int16_t* out = A.labels + map.Block(l, F) + z;
        float* mg = A.margin + map.Block(l, F) + z;
        float second = -__int_as_float(0x7f800000);
#pragma unroll
        for (int i = 0; i < kStates; ++i) second = (i != anchorState && prob[i] > second) ? prob[i] : second;
        mg[(size_t)(F - 1) * kLane] = maxP - second;
        int next = anchorState;
        for (int f = F - 1; f >= 0; --f)
        {
            out[(size_t)f * kLane] = (int16_t)ts;
            if (f < F - 1) mg[(size_t)f * kLane] = gapAt(f + 1, next);
            next = ts;
            ts = TraceSource<Grouped>(tb[(size_t)f * kLane], ts);
        }
        A.latRoi[g] = (int16_t)roiBit(F - 1);
    }
    else
    {
        // the labels block sits at the chunk's offset (derived from the
        // chunk pointer, so the lane map need not stay live through the loop)
        int16_t* out = A.labels + (chunk - A.trace);
        for (int f0 = F - kBatch; f0 >= 0; f0 -= kBatch)
        {
            uint32_t w[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) w[j] = tb[(size_t)(f0 + j) * kLane];
            if (f0 >= kBatch)
            {
#pragma unroll
                for (int j = 0; j < kBatch; ++j) PrefetchL1(tb + (size_t)(f0 - kBatch + j) * kLane);
            }
#pragma unroll
            for (int j = kBatch - 1; j >= 0; --j)
            {
                out[(size_t)(f0 + j) * kLane] = (int16_t)ts;
                ts = TraceSource<Grouped>(w[j], ts);
            }
        }
        A.latRoi[g] = (int16_t)roiBit(F - 1);
    }

    // Latent state update.
    A.latLabel[g] = (int16_t)anchorState;
    A.latTrc[g] = chunk[(size_t)(anchor - 1) * kLane];
    if (A.score) A.score[g] = ret;
    for (int f = 0; f < kLatent; ++f)
    {
        const int16_t v = pl[(size_t)f * kLane];
        if (A.latOut) A.latOut[(pl - A.prevLat) + (size_t)f * kLane] = v;   // same [lane][frame][64] layout
        pl[(size_t)f * kLane] = chunk[(size_t)(anchor + f) * kLane];
    }
}

// The lane's old model is replaced by the new one after all its ZMWs used it.
__global__ void LabelerModelCopyKernel(hw_lane_model* dst, const hw_lane_model* src, int lanes, LaneMap map)
{
    constexpr int kWords = (int)(sizeof(hw_lane_model) / 4);
    const int n = map.Lanes(lanes) * kWords;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t w = (size_t)map.Lane(i / kWords) * kWords + i % kWords;
    reinterpret_cast<uint32_t*>(dst)[w] = reinterpret_cast<const uint32_t*>(src)[w];
}

// Shared-memory words a thread: the ROI words twice (the second half also
// holds the anchor's log-likelihoods), packed labels after them (fused).
constexpr int LabelerWords(int F, bool fuse)
{
    const int n = (F + kLatent + 31) / 32;
    const int words = n + (n > kStates ? n : kStates);
    return fuse && F / kBatch > words ? F / kBatch : words;
}

template <bool Mapped, bool Fuse, int Threads, bool Margin = false, bool Grouped = false>
cudaError_t LaunchLabelerT(const LabelerArgs& a, const KParams& k, const PulseArgs& p, int lanes, cudaStream_t s)
{
    const int blocks = (lanes * kLane + Threads - 1) / Threads;
    const size_t smem = (size_t)LabelerWords(a.F, Fuse) * Threads * sizeof(uint32_t);
    static bool attrSet[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (smem > 48 * 1024 && (dev < 0 || dev >= 64 || !attrSet[dev]))
    {
        e = cudaFuncSetAttribute(LabelerKernel<Mapped, Fuse, Threads, Margin, Grouped>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(LabelerWords(1024, Fuse) * Threads * sizeof(uint32_t)));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attrSet[dev] = true;
    }
    LabelerKernel<Mapped, Fuse, Threads, Margin, Grouped><<<blocks, Threads, smem, s>>>(a, k, p);
    return cudaGetLastError();
}

// The generic or the grouped 9-way rows (KParams::grouped9) of one variant.
template <bool Mapped, bool Fuse, int Threads>
cudaError_t LaunchLabelerG(const LabelerArgs& a, const KParams& k, const PulseArgs& p, int lanes, cudaStream_t s)
{
    return k.grouped9 ? LaunchLabelerT<Mapped, Fuse, Threads, false, true>(a, k, p, lanes, s)
                      : LaunchLabelerT<Mapped, Fuse, Threads, false, false>(a, k, p, lanes, s);
}

cudaError_t LaunchLabeler(const LabelerArgs& a, const KParams& k, cudaStream_t s, const PulseArgs* fusedPulses,
                          int lanesPerCta)
{
    if (a.F > 1024 || a.F % kBatch != 0) return cudaErrorInvalidValue;
    const int lanes = a.map.Lanes(a.lanes);
    if (lanes == 0) return cudaSuccess;
    cudaError_t e;
    const PulseArgs none{};
    if (!a.map.On())
    {
        if (fusedPulses || lanesPerCta != 2) return cudaErrorInvalidValue;
        if (a.margin && !a.gap) return cudaErrorInvalidValue;
        e = a.margin ? LaunchLabelerT<false, false, 128, true>(a, k, none, lanes, s)
                     : LaunchLabelerG<false, false, 128>(a, k, none, lanes, s);
    }
    else if (a.margin)
    {
        return cudaErrorInvalidValue;     // margins come from the single-pool labeler
    }
    else if (fusedPulses)
    {
        if (lanesPerCta == 1) e = LaunchLabelerG<true, true, 64>(a, k, *fusedPulses, lanes, s);
        else if (lanesPerCta == 2) e = LaunchLabelerG<true, true, 128>(a, k, *fusedPulses, lanes, s);
        else if (lanesPerCta == 4) e = LaunchLabelerG<true, true, 256>(a, k, *fusedPulses, lanes, s);
        else return cudaErrorInvalidValue;
    }
    else
    {
        if (lanesPerCta == 1) e = LaunchLabelerG<true, false, 64>(a, k, none, lanes, s);
        else if (lanesPerCta == 2) e = LaunchLabelerG<true, false, 128>(a, k, none, lanes, s);
        else if (lanesPerCta == 4) e = LaunchLabelerG<true, false, 256>(a, k, none, lanes, s);
        else return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    const int n = lanes * (int)(sizeof(hw_lane_model) / 4);
    LabelerModelCopyKernel<<<(n + 255) / 256, 256, 0, s>>>(a.latModel, a.models, a.lanes, a.map);
    return cudaGetLastError();
}

}   // namespace hwk
