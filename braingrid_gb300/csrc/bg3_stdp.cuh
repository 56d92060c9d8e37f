// STDP learning shared by the step kernels: the pre-spike and post-spike walks over the spike
// histories.
#pragma once
#include "bg3_internal.cuh"

namespace bg3 {

// ---- STDP ------------------------------------------------------------------------------------
// AllSTDPSynapses::advanceSynapse / stdpLearning (Synapses/AllSTDPSynapses.cpp:283-472) and the
// device form advanceSTDPSynapsesDevice (AllSynapsesDeviceFuncs_d.cu:100-380).  The only
// difference between the two builds is the type of the spike times in the interval arithmetic:
// uint64_t on the host (a pre-spike walk interval wraps to a huge positive value), int64_t on
// the device.  Each float / double operation rounds as in the reference; the exp factors come
// from the host library's tables.

// getSpikeHistory (Neurons/AllSpikingNeurons.cpp:182-188) for off in [-max_spikes, -1]; co = spikeCount +
// spikeCountOffset.  A ring of one or two entries is asked for -2 and -3 all the same (by walks that
// need a valid entry there to learn): the first place where that is before the ring.
__host__ __device__ __forceinline__ int hist_index(int co, int ms, int off)
{
    // below 3 max_spikes unless the ring has overflowed: no remainder for what two comparisons do
    int x = co + ms + off;
    if (x >= ms) x -= ms;
    if (x >= ms) x -= ms;
    if (x >= ms) x %= ms;
    return x > 0 ? x : 0;
}
__device__ __forceinline__ unsigned long long hist_at(const NetDev &n, int i, int co, int off)
{
    return n.history[(size_t)i * n.max_spikes + hist_index(co, n.max_spikes, off)];
}

// W^mu with mu = 0, the only exponent a network accepts (set_stdp_type refuses others)
__device__ __forceinline__ float pow_mu(float, float) { return 1.0f; }

// One stdpLearning call with delta = dk steps (dk the signed interval; 0 when not a small count),
// in two parts.  stdp_dw: the weight change before the efficacies, which W does not enter (W^mu =
// 1); false when delta lies within the gap (W unchanged, no clamp).  stdp_apply: W plus the double
// product epost * epre * dw, rounded to float, then the clamps.  So the walks below can find a
// walk's changes before W is known and apply them in order after.
//
// The reference promotes to double all along; on this chip's narrow FP64 pipe a post-spike pass of
// a 30x30 network at 60 Hz waited for little else (500 steps 3.9 ms, now 3.3).  The comparisons need no double: a float against
// a float is the same comparison in either, and 3 tau, exact in double, is replaced by the float next
// to it on the far side.  1 - x rounds the same directly and by way of double (53 bits are more than
// twice 24 and two).  The sum is made in float-float arithmetic where every value within 2^-44 of the
// change and 2^-46 of the sum rounds the same (its distance from the double chain's value is below an
// eighth of that), and in double otherwise.  What stays in double is the table's factor.
__device__ __forceinline__ bool stdp_dw(const StdpConst &c, float delta, long long dk, float &dw)
{
    if (delta < -c.gap) {
        const double e = (dk < 0 && -dk < (long long)c.dlen_neg) ? c.dneg[-dk]
                                                                  : exp((double)delta / (double)c.tauneg);
        dw = (float)((double)(pow_mu(0.0f, c.muneg) * c.Aneg) * e);
    } else if (delta > c.gap) {
        const double e = (dk > 0 && dk < (long long)c.dlen_pos) ? c.dpos[dk]
                                                                 : exp(-(double)delta / (double)c.taupos);
        dw = (float)((double)(pow_mu(0.0f, c.mupos) * c.Apos) * e);
    } else {
        return false;
    }
    return true;
}
// W + epost * epre * dw from float-float arithmetic; false where the rounding is not certain, or
// the product so far from W's range of sizes that its low parts could be lost.
__device__ __forceinline__ bool stdp_sum_ff(float W, float epost, float epre, float dw, float &out)
{
    const float f = epost * epre;
    const float g = __fmaf_rn(epost, epre, -f);
    const float p = f * dw;
    const float q = __fmaf_rn(g, dw, __fmaf_rn(f, dw, -p));  // epost epre dw = p + q
    const FF s = ff_two_sum(W, p);
    const float lo = s.lo + q, err = fabsf(p) * 0x1p-44f + fabsf(s.hi) * 0x1p-46f;
    const float up = s.hi + (lo + err), dn = s.hi + (lo - err);
    out = up;
    return up == dn && fabsf(p) > 0x1p-60f && fabsf(W) < 0x1p+60f && fabsf(p) < 0x1p+60f &&
           fabsf(s.hi) > fabsf(p) * 0x1p-3f;
}
__device__ __forceinline__ float stdp_apply(const StdpConst &c, float W, float epost, float epre, float dw)
{
    float s;
    if (!stdp_sum_ff(W, epost, epre, dw, s))
        s = (float)((double)W + (double)epost * (double)epre * (double)dw);
    W = s;
    if ((c.Wex < 0.0f && W > 0.0f) || (c.Wex > 0.0f && W < 0.0f)) W = 0.0f;
    if (fabsf(W) > fabsf(c.Wex)) W = c.Wex;
    return W;
}
__device__ __forceinline__ float stdp_learn(const StdpConst &c, float W, float delta, float epost,
                                            float epre, long long dk)
{
    float dw;
    return stdp_dw(c, delta, dk, dw) ? stdp_apply(c, W, epost, epre, dw) : W;
}

// A neuron's history entries -1 .. -4 read together (those of them that exist: off >= -ms), so
// that a walk's first steps do not wait on one load each; hist_get takes the rest from memory.
struct Hist4 {
    unsigned long long h0, h1, h2, h3;
};
__device__ __forceinline__ void hist_load4(const NetDev &n, int i, int co, Hist4 &c)
{
    const int ms = n.max_spikes;
    c.h0 = hist_at(n, i, co, -1);  // max_spikes >= 1
    c.h1 = ms >= 2 ? hist_at(n, i, co, -2) : BG3_ULONG_MAX;
    c.h2 = ms >= 3 ? hist_at(n, i, co, -3) : BG3_ULONG_MAX;
    c.h3 = ms >= 4 ? hist_at(n, i, co, -4) : BG3_ULONG_MAX;
}
// entry off (-ms <= off <= -1)
__device__ __forceinline__ unsigned long long hist_get(const NetDev &n, int i, int co, int off,
                                                       const Hist4 &c)
{
    return off == -1 ? c.h0 : off == -2 ? c.h1 : off == -3 ? c.h2 : off == -4 ? c.h3
                                                                    : hist_at(n, i, co, off);
}

// The fPre branch: a spike from pre arrives at the synapse onto post at step t.  Returns W.
static __device__ float stdp_pre(const NetDev &n, const StdpConst &c, float W, int pre, int post,
                          unsigned long long t)
{
    const int ms = n.max_spikes;
    const int cpost = n.spikeCount[post] + n.spikeCountOffset[post];
    if (!n.stdp_signed) {
        // Every interval (spikeHistory - step) wraps to ~1.8e15 s (or is 0 at step t): each
        // learning call potentiates by exactly zero and applies the clamps, so only whether one
        // happens matters: the walk runs while entries -k and -(k+1) are valid.
        const unsigned long long h1 = hist_at(n, post, cpost, -1);
        const unsigned long long h2 = hist_at(n, post, cpost, -2);
        if (hist_at(n, post, cpost, -ms) != BG3_ULONG_MAX) set_err(n, ERR_STDP_RING);
        bool learn;
        if (c.useFD) {
            const unsigned long long h3 = hist_at(n, post, cpost, -3);
            learn = h1 != BG3_ULONG_MAX && h2 != BG3_ULONG_MAX && (h1 != t || h3 != BG3_ULONG_MAX);
        } else {
            learn = h1 != BG3_ULONG_MAX && (h1 != t || h2 != BG3_ULONG_MAX);
        }
        if (learn) {
            // potentiation by (float)(x * exp(-huge)) = +-0; epost * epre >= 0 keeps dw's sign
            const float dw = (float)((double)(pow_mu(c.Wex - W, c.mupos) * c.Apos) * 0.0);
            W = (float)((double)W + (double)dw);
            if ((c.Wex < 0.0f && W > 0.0f) || (c.Wex > 0.0f && W < 0.0f)) W = 0.0f;
            if (fabsf(W) > fabsf(c.Wex)) W = c.Wex;
        }
        return W;
    }
    const int cpre = n.spikeCount[pre] + n.spikeCountOffset[pre];
    Hist4 hp;
    hist_load4(n, post, cpost, hp);
    const unsigned long long sp2 = hist_at(n, pre, cpre, -2);
    float epre = 1.0f;
    if ((long long)sp2 > 0 && c.useFD)
        epre = 1.0f - exp_interval(n, t - sp2, true, c.tauspre);
    for (int off = -1;; --off) {
        if (off < -ms) { set_err(n, ERR_STDP_RING); break; }
        const unsigned long long sh = hist_get(n, post, cpost, off, hp);
        if (sh == BG3_ULONG_MAX) break;
        const long long dk = (long long)(sh - t);
        const float delta = (float)dk * n.dt;
        if (delta <= __fmul_rd(-3.0f, c.tauneg)) break;
        float epost = 1.0f;
        if (c.useFD) {
            if (off - 1 < -ms) { set_err(n, ERR_STDP_RING); break; }
            const unsigned long long sh2 = hist_get(n, post, cpost, off - 1, hp);
            if (sh2 == BG3_ULONG_MAX) break;
            epost = 1.0f - exp_interval(n, sh - sh2, true, c.tauspost);
        }
        W = stdp_learn(c, W, delta, epost, epre, dk);
    }
    return W;
}

// The fPost branch: post fired at step t; walk the pre history (both builds agree here).  The
// walk does not depend on W, so it runs in two parts: stdp_post_prep reads everything it needs
// (spike counts, histories, tables) and makes its first four steps, keeping their weight changes;
// stdp_post_finish applies them to W and makes any further steps.  The post-spike pass calls
// the first before its wait on the delivery of the same step (the one writer of W there).
constexpr int POST_STEPS = 4;
struct PostPrep {
    float dw[POST_STEPS], epre[POST_STEPS];  // the changes of steps 1 .. 4 (those with a bit in mask)
    float epost;
    int cpre;
    int mask;                       // bit k: step k + 1 changed W
    int next;                       // 0: the walk has ended; else the entry it continues from
};
// cpre, cpost: spikeCount + spikeCountOffset of the two neurons as of step t.
__device__ __forceinline__ void stdp_post_prep(const NetDev &n, const StdpConst &c, int pre,
                                               int post, int cpre, int cpost, int total_delay,
                                               unsigned long long t, PostPrep &q)
{
    const int ms = n.max_spikes;
    const bool sgn = n.stdp_signed != 0;
    const unsigned long long q2 = hist_at(n, post, cpost, -2);
    Hist4 hp;
    hist_load4(n, pre, cpre, hp);
    float epost = 1.0f;
    const bool ok = sgn ? ((long long)q2 > 0) : (q2 != BG3_ULONG_MAX);
    if (ok && c.useFD) epost = 1.0f - exp_interval(n, t - q2, sgn, c.tauspost);
    q.epost = epost;
    q.cpre = cpre;
    q.mask = 0;
    q.next = 0;
#pragma unroll
    for (int k = 0; k < POST_STEPS; k++) {
        const int off = -1 - k;
        if (off < -ms) { set_err(n, ERR_STDP_RING); return; }
        const unsigned long long sh = hist_get(n, pre, cpre, off, hp);
        if (sh == BG3_ULONG_MAX) return;
        const unsigned long long dd = t - (unsigned long long)(long long)total_delay - sh;
        const float delta = (sgn ? (float)(long long)dd : (float)dd) * n.dt;
        if (delta <= 0.0f || delta >= __fmul_ru(3.0f, c.taupos)) return;
        float epre = 1.0f;
        if (c.useFD) {
            if (off - 1 < -ms) { set_err(n, ERR_STDP_RING); return; }
            const unsigned long long sh2 = hist_get(n, pre, cpre, off - 1, hp);
            if (sh2 == BG3_ULONG_MAX) return;
            epre = 1.0f - exp_interval(n, sh - sh2, sgn, c.tauspre);
        }
        q.epre[k] = epre;
        if (stdp_dw(c, delta, (long long)dd, q.dw[k])) q.mask |= 1 << k;
    }
    q.next = -1 - POST_STEPS;
}
__device__ __forceinline__ void stdp_post_prep(const NetDev &n, const StdpConst &c, int pre,
                                               int post, int total_delay, unsigned long long t,
                                               PostPrep &q)
{
    stdp_post_prep(n, c, pre, post, n.spikeCount[pre] + n.spikeCountOffset[pre],
                   n.spikeCount[post] + n.spikeCountOffset[post], total_delay, t, q);
}
__device__ __forceinline__ float stdp_post_finish(const NetDev &n, const StdpConst &c, float W,
                                                  int pre, int total_delay, unsigned long long t,
                                                  const PostPrep &q)
{
#pragma unroll
    for (int k = 0; k < POST_STEPS; k++)
        if ((q.mask >> k) & 1) W = stdp_apply(c, W, q.epost, q.epre[k], q.dw[k]);
    if (!q.next) return W;
    const int ms = n.max_spikes;
    const bool sgn = n.stdp_signed != 0;
    for (int off = q.next;; --off) {
        if (off < -ms) { set_err(n, ERR_STDP_RING); break; }
        const unsigned long long sh = hist_at(n, pre, q.cpre, off);
        if (sh == BG3_ULONG_MAX) break;
        const unsigned long long dd = t - (unsigned long long)(long long)total_delay - sh;
        const float delta = (sgn ? (float)(long long)dd : (float)dd) * n.dt;
        if (delta <= 0.0f || delta >= __fmul_ru(3.0f, c.taupos)) break;
        float epre = 1.0f;
        if (c.useFD) {
            if (off - 1 < -ms) { set_err(n, ERR_STDP_RING); break; }
            const unsigned long long sh2 = hist_at(n, pre, q.cpre, off - 1);
            if (sh2 == BG3_ULONG_MAX) break;
            epre = 1.0f - exp_interval(n, sh - sh2, sgn, c.tauspre);
        }
        W = stdp_learn(c, W, delta, q.epost, epre, (long long)dd);
    }
    return W;
}
static __device__ __forceinline__ float stdp_post(const NetDev &n, const StdpConst &c, float W, int pre, int post,
                           int total_delay, unsigned long long t)
{
    PostPrep q;
    stdp_post_prep(n, c, pre, post, total_delay, t, q);
    return stdp_post_finish(n, c, W, pre, total_delay, t, q);
}

// A spike emitted at step tf arrives at plane slot p (dest d, source src) at step t64: the
// isSpikeQueue hit of AllSpikingSynapses::advanceSynapse (Synapses/AllSpikingSynapses.cpp:297-319)
// followed by changePSR (AllDSSynapses.cpp:227-247, AllSpikingSynapses.cpp:327-334), the STDP
// kinds' fPre learning walk first.  The slot's event state is updated here; inc is what the
// caller adds to its psr.  False when the synapse did not exist when the spike left.
template <int SYN>
__device__ __forceinline__ bool arrival(const NetDev &n, uint32_t p, int d, int src, uint32_t tf,
                                        unsigned long long t64, float &inc)
{
    EvSlot e = n.ev[p];
    if ((int32_t)(tf - e.born) < 0) return false;
    const float dec = n.dtab[e.dcls];
    EvSlot *q = &n.ev[p];
    if (SYN >= 2) {
        e.W = stdp_pre(n, n.stdp[n.stype[p]], e.W, src, d, t64);
        gst(&q->W, e.W);
    }
    if (SYN == 1 || SYN == 3) {
        float u = e.u, r = e.r;
        if (e.last != BG3_NO_SPIKE32) ds_update(n, e, (uint32_t)t64 - e.last, u, r);
        inc = (e.W / dec) * u * r;
        gst(&q->u, u);
        gst(&q->r, r);
        gst(&q->last, (uint32_t)t64);
    } else {
        inc = e.W / dec;
    }
    return true;
}

}  // namespace bg3
