// Blocks of steps: up to eight steps of a network per pass over its state.
//
// A spike takes at least Dmin steps to arrive (eight or more at dt = 0.1 ms), so the arrivals of
// steps t .. t + T - 1, T <= min(8, Dmin), all come from spikes before step t, and within those
// steps a destination depends on nothing but its own neuron and its own synapses.  A pass over a
// 32-destination tile therefore runs T whole steps — neuron update, arrivals, decay and ordered
// sum, in the per-step kernels' order and arithmetic, so the same bits — while it moves the
// tile's synapse state once instead of T times and costs one launch instead of 2 T or 3 T.
//
// Arrivals are pulled: a slot's source is looked up in the neurons' spike masks (BlkDev), first
// in a bitmap of the neurons with any spike that may arrive in this block (one word per 32
// neurons, usually zero), then in the source's own 64-step mask.  Nothing is scattered, and a
// block needs no list of spikes; the ring the per-step kernels use is rebuilt from the masks when
// one of them, or a download, needs it (k_blk_ring), and the masks from the ring after an upload
// (k_blk_scatter, k_blk_act).
//
// Static state the passes do not change (sources, classes, neuron constants) is read before the
// grid-dependency wait; a block's launch overlaps the tail of the one before it.
//
// Three forms: thin networks (k_blk_thin, up to 64 slots per neuron), small networks, whose launch
// runs thousands of steps in one cluster (k_blk_small), and dense ones (k_blk_push, k_blk_dense).
// A step, in the per-step kernels and here: 90x90 Izhikevich with STDP 13.9 and 2.6 us; 100x100 without
// synapses 4.3 and 0.75; 30x30 LIF with STDP at 3 Hz 8.3 and 1.6; 100x100 with 7.6 M synapses 14 and 6
// to 8; 180x180 with 23 M at 300 Hz 87 and 55.
#include <cuda.h>
#include <algorithm>
#include <utility>
#define BG3_RARE __noinline__
#include "bg3_internal.cuh"
#include "bg3_ptx.cuh"
#include "bg3_stdp.cuh"

namespace bg3 {

__device__ __forceinline__ unsigned long long rotl64(unsigned long long x, unsigned s)
{
    s &= 63u;
    return s ? (x << s) | (x >> (64u - s)) : x;
}
__device__ __forceinline__ unsigned long long rotr64(unsigned long long x, unsigned s)
{
    return rotl64(x, 64u - (s & 63u));
}

// ---- masks from the ring and back ------------------------------------------------------------
// hist from the ring lists (hist zeroed before): grid.y = ring slot.  The slot of the next step is
// empty by the ring's invariant; the rest hold the last 63 steps.
__global__ void __launch_bounds__(256) k_blk_scatter(const __grid_constant__ NetDev n,
                                                     const __grid_constant__ BlkDev b)
{
    const int slot = blockIdx.y;
    if (slot == (int)(*n.step & (BG3_RING - 1))) return;
    const int m = min(n.ring_n[slot], n.N);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        atomicOr(&b.hist[n.ring[(size_t)slot * n.N + k]], 1ull << slot);
}
// the bitmap row of a block starting at the current step
__global__ void __launch_bounds__(256) k_blk_act(const __grid_constant__ NetDev n,
                                                 const __grid_constant__ BlkDev b)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // hist holds Np entries, whole tiles
    const unsigned long long t = *n.step;
    const bool on = i < n.N && (b.hist[i] & rotl64(b.win, (unsigned)t)) != 0ull;
    const unsigned w = __ballot_sync(0xffffffffu, on);
    if ((threadIdx.x & 31) == 0 && i < n.Np) {
        b.act[(t & (BLK_ACT_ROWS - 1)) * n.ntiles + (i >> 5)] = w;
        if (b.actn && w) atomicAdd(&b.actn[t & (BLK_ACT_ROWS - 1)], (uint32_t)__popc(w));
    }
}
// the ring lists from hist (ring_n zeroed before)
__global__ void __launch_bounds__(256) k_blk_ring(const __grid_constant__ NetDev n,
                                                  const __grid_constant__ BlkDev b)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N) return;
    unsigned long long m = b.hist[i] & ~(1ull << (*n.step & (BG3_RING - 1)));
    while (m) {
        const int slot = __ffsll((long long)m) - 1;
        m &= m - 1ull;
        n.ring[(size_t)slot * n.N + atomicAdd(&n.ring_n[slot], 1)] = i;
    }
}

// End of a tile's block, one lane per destination: its spikes (fired: bit j, at step t + j) into the
// masks, the bitmap word for the block after this one, and for the STDP kinds the list of the
// neurons that fired.  Returns the updated mask.
template <int SYN>
__device__ __forceinline__ unsigned long long blk_spikes(const NetDev &n, const BlkDev &b, int tile, int d,
                                                         bool valid, unsigned long long hist,
                                                         uint32_t fired, int nt, unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long t1 = t + (unsigned)nt;
    if (valid) {
        hist = (hist & ~rotl64((1ull << nt) - 1ull, (unsigned)t)) | rotl64(fired, (unsigned)t);
        gst(&b.hist[d], hist);
    }
    const unsigned w = __ballot_sync(0xffffffffu, (hist & rotl64(b.win, (unsigned)t1)) != 0ull);
    if (SYN >= 2) {
        // the neurons that fired, for the post-spike pass: in the ring slot of the block's first
        // step (the ring's lists are rebuilt from the masks when they are needed)
        const unsigned m = __ballot_sync(0xffffffffu, fired != 0u);
        if (m) {
            const int slot = (int)(t & (BG3_RING - 1));
            int at = 0;
            if (lane == 0) at = atomicAdd(&n.ring_n[slot], __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            at += __popc(m & ((1u << lane) - 1u));
            if (fired && at < n.N) n.ring[(size_t)slot * n.N + at] = d;
            else if (fired) set_err(n, ERR_SPIKE_LIST);
        }
    }
    if (lane == 0) {
        b.act[(t1 & (BLK_ACT_ROWS - 1)) * n.ntiles + tile] = w;
        if (b.actn && w) atomicAdd(&b.actn[t1 & (BLK_ACT_ROWS - 1)], (uint32_t)__popc(w));
    }
    return hist;
}

// One step of a tile's neurons, one lane per destination; true where the neuron fired.  Most steps
// no neuron of the tile fires and no input spike falls due, and then every lane takes the same
// straight line, which keeps or replaces its state by selection; the branches of neuron_update and
// input_update, taken only when some lane needs them, cost 400 cycles a step of which the
// arithmetic is 60 (and the regular input's 64-bit remainder another 400: its cycle position is
// carried from step to step here).
struct StepRun {
    int mode;           // izh_mode
    int cyc, until;     // regular input: the cycle position, and the end of the neuron's stimulus
};
__device__ __forceinline__ StepRun step_run(const NetDev &n, int d, const NeuronIn &x, unsigned long long t)
{
    StepRun r = {izh_mode(n, d), 0, 0};
    if (n.input_kind == 1) {
        r.cyc = (int)(((unsigned long long)n.reg_c0 + (t - n.reg_t0)) % (unsigned long long)n.reg_cycle);
        r.until = (x.reg_shift + n.reg_dur) % n.reg_cycle;
    }
    return r;
}
__device__ __forceinline__ bool step_neuron(const NetDev &n, int d, bool valid, NeuronIn &x, float sp,
                                            float noise, unsigned long long t, StepRun &r)
{
    const bool izh = n.neuron_kind == 1, poisson = n.input_kind == 2 && x.pmask;
    const int br = neuron_branch(x), cyc = r.cyc;
    const int left = x.nisi - 1;
    bool slow = br == BR_FIRE || (izh && r.mode != IZH_FF);
    if (poisson) slow = slow || left <= 0 || ((x.q >> ((uint32_t)t & 31u)) & 1u);
    if (n.input_kind == 1) r.cyc = cyc + 1 == n.reg_cycle ? 0 : cyc + 1;
    if (__any_sync(0xffffffffu, valid && slow)) {
        if (!valid) return false;
        const float in = input_update(n, d, x, t, sp);
        return neuron_update(n, d, x, br, in, noise, t, r.mode);
    }
    if (n.input_kind == 1 && cyc >= x.reg_shift && cyc < r.until) sp = sp + x.reg_value;
    if (poisson) {
        x.nisi = left;
        x.ipsr = x.ipsr * x.idec;
        sp = sp + x.ipsr;
    }
    const bool on = br == BR_INTEGRATE;
    if (!on) x.refr = x.refr - 1;
    sp = sp + x.I0;
    sp = sp + noise * x.Inoise;
    if (izh) {
        const float Vint = x.Vm * 1000.0f, u = x.u;
        bool ok = false;
        float V = izh_v_ff(Vint, u, x.C3, x.C2 * sp, ok);
        if (on && valid && !ok) V = izh_v_fp64(Vint, u, x.C3, x.C2 * sp);  // uncertain rounding
        const float w = u + x.C3 * x.A * (x.B * Vint - u);
        x.u = on ? w : x.u;
        x.Vm = on ? V : x.Vm;
    } else {
        const float V = x.C1 * x.Vm + x.C2 * sp;
        x.Vm = on ? V : x.Vm;
    }
    return false;
}

// What the block starting at t1 and the ones after it find cleared: the next list of fired neurons,
// and the counts of the blocks that may follow the next one.
__device__ __forceinline__ void blk_clear(const NetDev &n, const BlkDev &b, unsigned long long t1)
{
    n.ring_n[t1 & (BG3_RING - 1)] = 0;
    if (b.actn)
        for (int j = 1; j <= BLK_MAX_STEPS; j++) b.actn[(t1 + j) & (BLK_ACT_ROWS - 1)] = 0u;
}

__device__ __forceinline__ void neuron_store(const NetDev &n, int d, const NeuronIn &x, float sp)
{
    gst(&n.sp[d], sp);
    gst(&n.refr[d], x.refr);
    gst(&n.Vm[d], x.Vm);
    if (n.neuron_kind == 1) gst(&n.u_izh[d], x.u);
    if (n.input_kind == 2 && x.pmask) {
        gst(&n.pois_nisi[d], x.nisi);
        gst(&n.in_queue[d], x.q);
        gst(&n.in_psr[d], x.ipsr);
    }
}

// The last tile of a network to finish a block advances the step counter (every tile has read it).
__device__ __forceinline__ void blk_step(const NetDev &n, const BlkDev &b, unsigned long long t1)
{
    if ((threadIdx.x & 31) == 0 && atomicAdd(n.sweep_done, 1u) == (unsigned)n.ntiles - 1u) {
        *n.sweep_done = 0u;
        *n.step = t1;
        *n.dstep = t1;
        blk_clear(n, b, t1);
        if (t1 >= 0xffffff00ull) set_err(n, ERR_STEP_RANGE);
    }
}

template <int SYN>
__device__ __forceinline__ void blk_finish(const NetDev &n, const BlkDev &b, int tile, int d,
                                           bool valid, const NeuronIn &x, float sp,
                                           unsigned long long hist, uint32_t fired, int nt,
                                           unsigned long long t)
{
    if (valid) neuron_store(n, d, x, sp);
    blk_spikes<SYN>(n, b, tile, d, valid, hist, fired, nt, t);
    blk_step(n, b, t + (unsigned)nt);
}

// ---- thin networks: one warp per tile, or four ------------------------------------------------
// Networks of at most BLK_THIN_QUADS row quads per destination.  A warp keeps its tile's psr in
// shared memory for the whole block, beside the decay factors (expanded once, so that a step
// needs no class decoding) and the arrival masks (bit j of a slot's byte: a spike arrives at the
// block's step j).  Lane = destination, so no step needs a barrier: the neuron's state stays in
// registers, its summation point is the sum the lane has just made.  What bounds it: with many
// tiles the latency of 16 warps an SM (128 registers each; 43 % of the issue slots used), with few the
// chain of one tile, about 4.5 cycles an instruction of a lone warp: 2.0 us a step for Izhikevich
// networks of 2,000 neurons, 2.5 at 38,000.
constexpr int BLK_THIN_QUADS = 16;
constexpr int BLK_THIN_WARPS = 8;
constexpr int BLK_TEAM = 4;           // warps a tile
// Quads kept: where one warp is a tile's pace it sums four at a time without looking for the last; a
// warp among many does no work for quads that are not there (packed).
__host__ __device__ constexpr int thin_quads(int Mq, bool packed)
{
    return packed ? Mq : (Mq + 3) & ~3;
}
__host__ __device__ constexpr size_t blk_thin_smem(int Mq, int team, bool packed)
{
    return (size_t)thin_quads(Mq, packed) * 32 * (16 + 16 + 16 + 4 + 4) + BLK_MAX_STEPS * 32 * 4 +
           (size_t)(team - 1) * 32 * 16;
}

struct ThinSmem {           // Mq here: thin_quads; zero beyond the last in use
    float4 *psr, *dec;  // [Mq][32]
    float4 *inc;        // [Mq][32] psr increments of the arrivals that are ready
    uint32_t *msk;      // [Mq][32] their steps, one byte per row
    uint32_t *late;     // [Mq][32] the steps of the others
    float *noise;       // [BLK_MAX_STEPS][32]
    uint4 *found;       // [BLK_TEAM - 1][32] ThinEvents of the other warps of the tile
};

// A lane's arrivals in the block are made ready before the steps run, so that their chains of loads
// (the source's mask, the event slot, the exp tables) overlap, across the warp's lanes and two
// rows at a time: the steps and the psr increments in shared memory.  Two spikes at one synapse, and
// STDP arrivals whose weight the learning walk could change, run at their step (thin_late).
struct ThinEvents {
    unsigned long long rows;    // rows with an arrival (tiles of up to 64 rows)
    uint32_t steps;             // bit j: something arrives at step j
    bool late;                  // something is left for its step
};

// Whether an STDP arrival's learning walk may change W: with the host build's arithmetic the walk
// only applies the clamps (stdp_pre), so a weight inside its bounds stays as it is.
__device__ __forceinline__ bool stdp_clamps(const StdpConst &c, float W)
{
    return !(fabsf(W) <= fabsf(c.Wex)) || __float_as_uint(W) == 0x80000000u ||
           (c.Wex < 0.0f && W > 0.0f) || (c.Wex > 0.0f && W < 0.0f) || !(fabsf(c.Apos) < 1e30f);
}

// The arrivals at the rows set in `rows` (of the 64 from row r0 on).
template <int SYN>
__device__ __forceinline__ void thin_events(const NetDev &n, const BlkDev &b, const ThinSmem &s,
                                            unsigned long long rows, int r0, int d, int nt,
                                            unsigned long long t, ThinEvents &e)
{
    const int lane = threadIdx.x & 31;
    constexpr bool DS = SYN == 1 || SYN == 3;
    constexpr int U = 2;  // four: 3 % more a step on every network timed, 2,000 to 38,000 neurons
    // STDP: a walk that finds the ring full sets an error bit; where the ring may fill within the
    // block, at its step
    bool ring_late = false;
    if (SYN >= 2 && rows) {
        const int co = n.spikeCount[d] + n.spikeCountOffset[d];
        ring_late = hist_at(n, d, co, nt - n.max_spikes) != BG3_ULONG_MAX;
    }
    while (rows) {
        int r[U], D[U];
        uint32_t p[U], m[U];
        unsigned long long h[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            r[u] = rows ? r0 + __ffsll((long long)rows) - 1 : -1;
            rows &= rows - 1ull;
            m[u] = 0u;
            if (r[u] < 0) continue;
            p[u] = (uint32_t)slot_pos(r[u], d, n.Mq);
            D[u] = n.lcls[p[u]];
            m[u] = (uint32_t)n.src[p[u]];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (r[u] < 0) continue;
            D[u] = n.ltab[D[u]];
            h[u] = b.hist[m[u]];
        }
        float4 ev[U];
        uint2 ef[U];
        int ty[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (r[u] < 0) continue;
            m[u] = (uint32_t)rotr64(h[u], (unsigned)t - (unsigned)D[u]) & ((1u << nt) - 1u);
            if (!m[u]) continue;
            e.steps |= m[u];
            if (r[u] < 64) e.rows |= 1ull << r[u];
            const char *q = reinterpret_cast<const char *>(n.ev) + (size_t)p[u] * sizeof(EvSlot);
            ev[u] = *reinterpret_cast<const float4 *>(q);
            ef[u] = *reinterpret_cast<const uint2 *>(q + 16);
            if (SYN >= 2) ty[u] = n.stype[p[u]];
        }
        float xr[U], xu[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!m[u]) continue;
            bool late = (m[u] & (m[u] - 1u)) != 0u;
            if (SYN >= 2) {
                late = late || stdp_clamps(n.stdp[ty[u]], ev[u].x);
                if (ring_late) {
                    const int co = n.spikeCount[d] + n.spikeCountOffset[d];
                    if (hist_at(n, d, co, -n.max_spikes) == BG3_ULONG_MAX) late = true;
                }
            }
            if (late) {
                reinterpret_cast<uint8_t *>(&s.late[(r[u] >> 2) * 32 + lane])[r[u] & 3] = (uint8_t)m[u];
                e.late = true;
                m[u] = 0u;
                continue;
            }
            const uint32_t ta = (uint32_t)t + (uint32_t)(31 - __clz((int)m[u])), last = __float_as_uint(ev[u].w);
            if ((int32_t)(ta - (uint32_t)D[u] - ef[u].x) < 0) {
                m[u] = 0u;  // the synapse did not exist when the spike left
            } else if (DS && last != BG3_NO_SPIKE32) {
                const int pc = (int)((ef[u].y >> 8) & 255u);
                xr[u] = exp_tab(n, n.p_xD[pc], ta - last, n.p_D[pc]);
                xu[u] = exp_tab(n, n.p_xF[pc], ta - last, n.p_F[pc]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!m[u]) continue;
            if (SYN >= 2 && ring_late) set_err(n, ERR_STDP_RING);
            const float dec = n.dtab[ef[u].y & 255u];
            float inc;
            if (DS) {
                float uu = ev[u].y, rr = ev[u].z;
                if (__float_as_uint(ev[u].w) != BG3_NO_SPIKE32) {
                    const float Uc = n.p_U[(ef[u].y >> 8) & 255u];
                    rr = 1.0f + (rr * (1.0f - uu) - 1.0f) * xr[u];
                    uu = Uc + uu * (1.0f - Uc) * xu[u];
                }
                inc = (ev[u].x / dec) * uu * rr;
                gst(reinterpret_cast<float4 *>(n.ev) + 2 * (size_t)p[u],
                    make_float4(ev[u].x, uu, rr,
                                __uint_as_float((uint32_t)t + (uint32_t)(31 - __clz((int)m[u])))));
            } else {
                inc = ev[u].x / dec;
            }
            reinterpret_cast<uint8_t *>(&s.msk[(r[u] >> 2) * 32 + lane])[r[u] & 3] = (uint8_t)m[u];
            reinterpret_cast<float *>(&s.inc[(r[u] >> 2) * 32 + lane])[r[u] & 3] = inc;
        }
    }
}

// The lane's remaining arrivals of step t + j.
template <int SYN>
__device__ __noinline__ void thin_late(const NetDev &n, const ThinSmem &s, int d, int nq, int j,
                                       unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    for (int q = 0; q < nq; q++) {
        const uint32_t w = s.late[q * 32 + lane] >> j;
        for (int k = 0; k < 4; k++) {
            if (!((w >> (8 * k)) & 1u)) continue;
            const uint32_t p = (uint32_t)slot_pos(4 * q + k, d, n.Mq);
            const int D = n.ltab[n.lcls[p]];
            float inc;
            if (arrival<SYN>(n, p, d, n.src[p], (uint32_t)(t + (unsigned)j) - (uint32_t)D,
                             t + (unsigned)j, inc)) {
                float *ps = reinterpret_cast<float *>(&s.psr[q * 32 + lane]) + k;
                *ps = *ps + inc;
            }
        }
    }
}

// The ready arrivals of the block's step j onto their psr.
__device__ __forceinline__ void thin_add(const ThinSmem &s, int q, int k, int j)
{
    const int at = q * 32 + ((int)threadIdx.x & 31);
    if (!((s.msk[at] >> (8 * k + j)) & 1u)) return;
    float *ps = reinterpret_cast<float *>(&s.psr[at]) + k;
    *ps = *ps + reinterpret_cast<const float *>(&s.inc[at])[k];
}

// A tile's neurons and synapses in registers and shared memory.
struct ThinTile {
    NeuronIn x;
    float sp;
    unsigned long long hist;
    int cnt, nq;
};

// A tile's warps: `role` of `size`, and the named barrier they share.  Warp 0 runs the steps; before
// them every warp draws its share of the noise and makes ready the arrivals of its quads (role, role +
// size, ...), and it loads those quads.
template <int SIZE>  // 0: known at run time
struct Team {
    int role, given, bar;
    __device__ __forceinline__ int size() const { return SIZE ? SIZE : given; }
    __device__ __forceinline__ void sync() const
    {
        if (size() > 1) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * size()) : "memory");
    }
};

// The barrier of a small network's launch: its block, or its cluster of blocks.
__device__ __forceinline__ void small_sync()
{
    if (gridDim.x == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
}

// Injected noise in a small network's launch: each step the integrating neurons draw the next values
// of one stream, from the highest index down, so a neuron's place depends on how many above it draw.
// A tile's warp sends its count to every block and passes a barrier; one a step, with the counts of
// alternate steps in alternate rows.  The value's load is then in flight during the synapse step.
struct SmallDraws {
    int *cnt;                   // [2][SMALL_MAX_N / 32] in shared memory
    unsigned long long cursor;  // of the next step's first draw
    int tiles, row;
};
__device__ __forceinline__ float small_draw(const NetDev &n, SmallDraws &z, int tile, bool draws)
{
    const int lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(0xffffffffu, draws);
    int *cnt = z.cnt + z.row * (SMALL_MAX_N / 32);
    z.row ^= 1;
    if (gridDim.x == 1) {
        if (lane == 0) cnt[tile] = __popc(m);
    } else if (lane < (int)gridDim.x) {
        uint32_t at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(at)
            : "r"((uint32_t)__cvta_generic_to_shared(cnt + tile)), "r"((uint32_t)lane));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(__popc(m)) : "memory");
    }
    small_sync();
    int above = 0, all = 0;
    for (int k = lane; k < z.tiles; k += 32) {
        all += cnt[k];
        if (k > tile) above += cnt[k];
    }
    above = __reduce_add_sync(0xffffffffu, above);
    const unsigned long long pos = z.cursor + (unsigned)(above + __popc((m >> lane) >> 1));
    z.cursor += (unsigned)__reduce_add_sync(0xffffffffu, all);
    if (!draws) return 0.0f;
    if (pos < (unsigned long long)n.noise_len) return n.noise_buf[pos];
    set_err(n, ERR_NOISE_EXHAUSTED);
    return 0.0f;
}

// nt steps from t on: the arrivals made ready, then step by step the neuron update, the arrivals,
// decay and sum.  The psr is in shared memory.  DEP: the kernel's grid-dependency wait comes before
// the first access that needs it (see k_blk_thin).  Returns the steps at which the neuron fired.
template <int SYN, bool DEP, bool INJ, int SIZE>
__device__ __forceinline__ uint32_t thin_steps(const NetDev &n, const BlkDev &b, const ThinSmem &s,
                                               ThinTile &y, const Team<SIZE> &team, int tile, int d, bool valid,
                                               int nt, unsigned long long t, SmallDraws *z = nullptr)
{
    constexpr bool PACKED = SIZE == 1;  // no quads beyond the last (thin_quads)
    const int lane = threadIdx.x & 31;
    const int4 *S = reinterpret_cast<const int4 *>(n.src) + (size_t)tile * n.Mq * 32 + lane;
    const uint32_t *act = b.act + (t & (BLK_ACT_ROWS - 1)) * n.ntiles;
    ThinEvents e = {0ull, 0u, false};
    bool waited = !DEP || SYN < 2;
    // the steps' noise draws depend on nothing but the step: four at a time, so that one draw's
    // latency hides another's (inside the step loop each would wait alone)
    float drawn = 0.0f;
    if (INJ && team.role == 0)
        drawn = small_draw(n, *z, tile, valid && neuron_branch(y.x) == BR_INTEGRATE);
    else if (INJ)
        small_sync();
#pragma unroll 4
    for (int j = team.role; !INJ && j < nt; j += team.size())
        s.noise[j * 32 + lane] = normal_device(n.noise_seed, t + (unsigned)j, d);
    for (int g0 = 0; g0 < y.nq; g0 += 16) {
        // the slots whose source has a spike in this block's window, 64 rows at a time
        unsigned long long rows = 0ull;
        const int lim = min(y.nq - g0, 16);
        for (int i0 = team.role; i0 < lim; i0 += 4 * team.size()) {
            int4 sr[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int i = i0 + k * team.size();
                if (i < lim) {
                    sr[k] = S[(size_t)(g0 + i) * 32];
                    s.msk[(g0 + i) * 32 + lane] = 0u;
                    s.late[(g0 + i) * 32 + lane] = 0u;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int i = i0 + k * team.size();
                if (i < lim) {
                    const int left = y.cnt - 4 * (g0 + i);  // in-use rows from this quad on
                    uint32_t hit = 0u;
                    if (left > 0) hit |= ((act[sr[k].x >> 5] >> (sr[k].x & 31)) & 1u);
                    if (left > 1) hit |= ((act[sr[k].y >> 5] >> (sr[k].y & 31)) & 1u) << 1;
                    if (left > 2) hit |= ((act[sr[k].z >> 5] >> (sr[k].z & 31)) & 1u) << 2;
                    if (left > 3) hit |= ((act[sr[k].w >> 5] >> (sr[k].w & 31)) & 1u) << 3;
                    rows |= (unsigned long long)hit << (4 * i);
                }
            }
        }
        if (!waited) {
            pdl_wait();
            pdl_trigger();
            waited = true;
        }
        thin_events<SYN>(n, b, s, rows, 4 * g0, d, nt, t, e);
    }
    if (!waited) {
        pdl_wait();
        pdl_trigger();
    }
    if (team.size() > 1) {
        if (team.role > 0)
            s.found[(team.role - 1) * 32 + lane] =
                make_uint4((uint32_t)e.rows, (uint32_t)(e.rows >> 32), e.steps, e.late ? 1u : 0u);
        team.sync();
        if (team.role > 0) {
            for (int j = 1; INJ && j < nt; j++) small_sync();
            return 0u;
        }
        for (int k = 0; k < team.size() - 1; k++) {
            const uint4 f = s.found[k * 32 + lane];
            e.rows |= (unsigned long long)f.y << 32 | f.x;
            e.steps |= f.z;
            e.late = e.late || f.w != 0u;
        }
    }
    const uint32_t any = __reduce_or_sync(0xffffffffu, e.steps);
    StepRun run = step_run(n, d, y.x, t);
    uint32_t fired = 0u;
#pragma unroll 1
    for (int j = 0; j < nt; j++) {
        const float noise = INJ ? drawn : s.noise[j * 32 + lane];
        if (step_neuron(n, d, valid, y.x, y.sp, noise, t + (unsigned)j, run)) fired |= 1u << j;
        if (INJ && j + 1 < nt)
            drawn = small_draw(n, *z, tile, valid && neuron_branch(y.x) == BR_INTEGRATE);
        if ((any >> j) & 1u) {
            if ((e.steps >> j) & 1u) {
                for (unsigned long long r = e.rows; r; r &= r - 1ull) {
                    const int k = __ffsll((long long)r) - 1;
                    thin_add(s, k >> 2, k & 3, j);
                }
                for (int q = 16; q < y.nq; q++)  // a small network's wider tile
                    for (int k = 0; k < 4; k++) thin_add(s, q, k, j);
                if (e.late) thin_late<SYN>(n, s, d, y.nq, j, t);
            }
            __syncwarp();
        }
        float acc = 0.0f;
        for (int q0 = 0; q0 < y.nq; q0 += 4) {  // four quads' loads before the first is needed
            float4 v[4], c[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (PACKED && q0 + k >= y.nq) break;
                v[k] = s.psr[(q0 + k) * 32 + lane];
                c[k] = s.dec[(q0 + k) * 32 + lane];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (PACKED && q0 + k >= y.nq) break;
                v[k].x = v[k].x * c[k].x;
                v[k].y = v[k].y * c[k].y;
                v[k].z = v[k].z * c[k].z;
                v[k].w = v[k].w * c[k].w;
                s.psr[(q0 + k) * 32 + lane] = v[k];
                acc = acc + v[k].x;
                acc = acc + v[k].y;
                acc = acc + v[k].z;
                acc = acc + v[k].w;
            }
        }
        y.sp = acc;
    }
    return fired;
}

__device__ __forceinline__ ThinSmem thin_smem(uint8_t *smem, int Mq, bool packed)
{
    ThinSmem s;
    const int quads = thin_quads(Mq, packed);
    s.psr = reinterpret_cast<float4 *>(smem);
    s.dec = s.psr + quads * 32;
    s.inc = s.dec + quads * 32;
    s.msk = reinterpret_cast<uint32_t *>(s.inc + quads * 32);
    s.late = s.msk + quads * 32;
    s.noise = reinterpret_cast<float *>(s.late + quads * 32);
    s.found = reinterpret_cast<uint4 *>(s.noise + BLK_MAX_STEPS * 32);
    return s;
}

// What the steps do not change: the row counts, and the decay factors into shared memory.
template <int SIZE>
__device__ __forceinline__ void thin_static(const NetDev &n, const ThinSmem &s, ThinTile &y,
                                            const Team<SIZE> &team, int tile)
{
    const int lane = threadIdx.x & 31, d = tile * 32 + lane;
    y.cnt = d < n.N ? (int)n.count[d] : 0;
    y.nq = (__reduce_max_sync(0xffffffffu, y.cnt) + 3) >> 2;
    const uint16_t *C = reinterpret_cast<const uint16_t *>(n.dcls) + (size_t)tile * n.Mq * 32 + lane;
    for (int q = team.role; q < thin_quads(y.nq, SIZE == 1); q += team.size()) {
        if (q >= y.nq) {
            s.dec[q * 32 + lane] = s.psr[q * 32 + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            continue;
        }
        const uint32_t c = C[(size_t)q * 32];
        s.dec[q * 32 + lane] = make_float4(n.dtab[c & 15u], n.dtab[(c >> 4) & 15u],
                                           n.dtab[(c >> 8) & 15u], n.dtab[(c >> 12) & 15u]);
    }
}

// The tile's neurons into registers, its psr into shared memory.
template <int SIZE>
__device__ __forceinline__ void thin_load(const NetDev &n, const BlkDev &b, const ThinSmem &s, ThinTile &y,
                                          const Team<SIZE> &team, int tile)
{
    const int lane = threadIdx.x & 31, d = tile * 32 + lane;
    y.sp = 0.0f;
    y.hist = 0ull;
    if (team.role == 0 && d < n.N) {
        neuron_load(n, d, y.x);
        y.sp = n.sp[d];
        y.hist = b.hist[d];
    }
    const float4 *P = reinterpret_cast<const float4 *>(n.psr) + (size_t)tile * n.Mq * 32 + lane;
    for (int q0 = team.role; q0 < y.nq; q0 += 4 * team.size()) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (q0 + k * team.size() < y.nq) v[k] = P[(size_t)(q0 + k * team.size()) * 32];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (q0 + k * team.size() < y.nq) s.psr[(q0 + k * team.size()) * 32 + lane] = v[k];
    }
}

__device__ __forceinline__ void thin_store(const NetDev &n, const ThinSmem &s, const ThinTile &y, int tile)
{
    const int lane = threadIdx.x & 31;
    float4 *P = reinterpret_cast<float4 *>(n.psr) + (size_t)tile * n.Mq * 32 + lane;
    for (int q = 0; q < y.nq; q++) gst(&P[(size_t)q * 32], s.psr[q * 32 + lane]);
}

// STDP kinds follow a post-spike pass, which is launched once the block before has finished and
// writes nothing but weights: everything else is final, and the wait can come as late as the first
// arrival.
template <int SYN, int SIZE>
__device__ __forceinline__ void blk_thin_tile(const NetDev &n, const BlkDev &b, const Team<SIZE> &team,
                                              const int tile, const int nt, uint8_t *smem)
{
    const int d = tile * 32 + ((int)threadIdx.x & 31);
    const bool valid = d < n.N;
    const ThinSmem s = thin_smem(smem, n.Mq, SIZE == 1);
    ThinTile y;
    thin_static(n, s, y, team, tile);
    if (SYN < 2) {
        pdl_wait();
        pdl_trigger();
    }
    const unsigned long long t = *n.step;
    thin_load(n, b, s, y, team, tile);
    const uint32_t fired = thin_steps<SYN, true, false>(n, b, s, y, team, tile, d, valid, nt, t);
    if (team.role > 0) return;
    thin_store(n, s, y, tile);
    blk_finish<SYN>(n, b, tile, d, valid, y.x, y.sp, y.hist, fired, nt, t);
}

template <int SYN, int SIZE>
__global__ void __launch_bounds__(32 * BLK_THIN_WARPS, 2) k_blk_thin(const __grid_constant__ NetDev n,
                                                                  const __grid_constant__ BlkDev b,
                                                                  int nt)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int per = (int)(blockDim.x >> 5) / SIZE;  // tiles a block
    const int at = (int)(threadIdx.x >> 5) % per, tile = blockIdx.x * per + at;
    const Team<SIZE> team = {(int)(threadIdx.x >> 5) / per, SIZE, 1 + at};
    if (tile < n.ntiles)
        blk_thin_tile<SYN>(n, b, team, tile, nt, smem_raw + at * blk_thin_smem(n.Mq, SIZE, SIZE == 1));
}

// Batched form: tiles[i] = (network, tile), -1 tiles idle; a block's entries belong to one
// network, whose descriptor the block copies into shared memory first.  wsmem: bytes per warp
// (the batch's widest thin network).
template <int SYN, int SIZE>
__global__ void __launch_bounds__(32 * BLK_THIN_WARPS, 2) k_blk_thin_batch(const NetDev *nets,
                                                                        const BlkDev *blks,
                                                                        const int2 *tiles, int count,
                                                                        int wsmem, int nt)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(16) NetDev s_net;
    const int per = (int)(blockDim.x >> 5) / SIZE;
    const int at = (int)(threadIdx.x >> 5) % per, first = blockIdx.x * per;
    const Team<SIZE> team = {(int)(threadIdx.x >> 5) / per, SIZE, 1 + at};
    const int2 tr = first + at < count ? tiles[first + at] : make_int2(0, -1);
    const int k = tiles[first].x;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(nets + k);
    uint4 *d4 = reinterpret_cast<uint4 *>(&s_net);
    for (int i = threadIdx.x; i < (int)(sizeof(NetDev) / 16); i += blockDim.x) d4[i] = s4[i];
    const BlkDev b = blks[k];
    __syncthreads();
    if (tr.y >= 0) blk_thin_tile<SYN>(s_net, b, team, tr.y, nt, smem_raw + at * wsmem);
}

// ---- STDP: learning after a block's post spikes -----------------------------------------------
// The fPost branch (AllSTDPSynapses.cpp:368-418) of every neuron that fired in the block just
// run, after the block instead of inside its steps.  The order of the weight changes is kept:
// where an arrival at the same synapse follows a post spike within the block, its spike was
// already under way (the source's newest history entry is later than t - delay), and the walk of
// such a post spike learns nothing; so all of a block's arrivals come before the post spikes that
// learn.  A walk sees the histories as of its step: the entries the block added after it, counted in
// the spike masks, are left out.
__device__ __forceinline__ int count_at(const NetDev &n, int i, unsigned long long hist, int nt,
                                        unsigned long long t, int j)
{
    const int co = n.spikeCount[i] + n.spikeCountOffset[i];
    const int newer = __popc((uint32_t)rotr64(hist, (unsigned)t) & ((1u << nt) - (2u << j)));
    return co >= newer ? co - newer : co - newer + n.max_spikes;
}

// One warp per neuron that fired, one lane per synapse.
__device__ __forceinline__ void blk_post(const NetDev &n, const BlkDev &b, int gw, int nw, int nt,
                                         unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    const int slot = (int)(t & (BG3_RING - 1));
    const int m = min(n.ring_n[slot], n.N);
    const int32_t *ids = n.ring + (size_t)slot * n.N;
    for (int e = gw; e < m; e += nw) {
        const int d = ids[e];
        const int cnt = (int)n.count[d];
        const unsigned long long hd = b.hist[d];
        const uint32_t fired = (uint32_t)rotr64(hd, (unsigned)t) & ((1u << nt) - 1u);
        for (int k = lane; k < cnt; k += 32) {
            const size_t p = slot_pos(k, d, n.Mq);
            const StdpConst &c = n.stdp[n.stype[p]];
            const int pre = n.src[p];
            const int delay = n.ltab[n.lcls[p]];
            const unsigned long long hp = b.hist[pre];
            float W = n.ev[p].W;
            for (uint32_t f = fired; f; f &= f - 1u) {
                const int j = __ffs((int)f) - 1;
                const unsigned long long tj = t + (unsigned)j;
                PostPrep q;
                stdp_post_prep(n, c, pre, d, count_at(n, pre, hp, nt, t, j), count_at(n, d, hd, nt, t, j), delay,
                               tj, q);
                W = stdp_post_finish(n, c, W, pre, delay, tj, q);
            }
            n.ev[p].W = W;
        }
    }
}

__global__ void __launch_bounds__(256) k_blk_post(const __grid_constant__ NetDev n,
                                                  const __grid_constant__ BlkDev b, int nt)
{
    pdl_wait();
    pdl_trigger();
    blk_post(n, b, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5, nt,
             *n.step - (unsigned)nt);
}

__global__ void __launch_bounds__(256) k_blk_post_batch(const NetDev *nets, const BlkDev *blks,
                                                        int nt)
{
    __shared__ __align__(16) NetDev s_net;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(nets + blockIdx.y);
    uint4 *d4 = reinterpret_cast<uint4 *>(&s_net);
    for (int i = threadIdx.x; i < (int)(sizeof(NetDev) / 16); i += blockDim.x) d4[i] = s4[i];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    blk_post(s_net, blks[blockIdx.y], (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
             (gridDim.x * blockDim.x) >> 5, nt, *s_net.step - (unsigned)nt);
}

// ---- small networks: many blocks per launch ----------------------------------------------------
// A network of few tiles is a launch's latency per block of steps and little else, so one launch runs
// thousands of steps: one warp per tile, which keeps the tile's psr, neurons and masks for the whole
// launch, in up to eight blocks of one cluster, with a cluster barrier (a block barrier when there is
// one block) after each block of steps and, for the STDP kinds, another after the post-spike pass.
// The barriers order the masks, bitmaps and histories that the tiles read of each other.  Four warps
// a block, one per quarter of its SM, up to 32 tiles: a warp issues alone, and that is its pace.
template <int SYN, bool INJ>
__global__ void __launch_bounds__(32 * BLK_THIN_WARPS, 1) k_blk_small(const __grid_constant__ NetDev n,
                                                                      const __grid_constant__ BlkDev b,
                                                                      int size, int nsteps, int T)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int warp = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5) / size;  // tiles a block
    // the warps of a tile on different quarters of the SM, and the first warps of four tiles too
    const Team<0> team = {warp / nw, size, 1 + (warp + warp / nw) % nw};
    const int at = team.bar - 1, tile = (int)blockIdx.x * nw + at, d = tile * 32 + ((int)threadIdx.x & 31);
    const bool active = tile < n.ntiles, valid = d < n.N, first = blockIdx.x == 0 && threadIdx.x == 0;
    const ThinSmem s = thin_smem(smem_raw + at * blk_thin_smem(n.Mq, size, false), n.Mq, false);
    ThinTile y;
    unsigned long long t = *n.step;
    __shared__ int s_draws[INJ ? 2 * (SMALL_MAX_N / 32) : 1];
    SmallDraws z = {s_draws, INJ ? *n.noise_cursor : 0ull, (int)gridDim.x * nw, 0};
    if (active) {
        thin_static(n, s, y, team, tile);
        thin_load(n, b, s, y, team, tile);
    }
    if (INJ) small_sync();  // every block has started: its shared memory can be written
    for (int left = nsteps; left > 0;) {
        const int nt = min(left, T);
        if (first) blk_clear(n, b, t + (unsigned)nt);
        if (active) {
            const uint32_t fired = thin_steps<SYN, false, INJ>(n, b, s, y, team, tile, d, valid, nt, t, &z);
            if (team.role == 0)
                y.hist = blk_spikes<SYN>(n, b, tile, d, valid, y.hist, fired, nt, t);
        } else if (INJ) {
            for (int j = 0; j < nt; j++) {
                if (team.role == 0) small_draw(n, z, tile, false);
                else small_sync();
            }
        }
        small_sync();
        if (SYN >= 2) {
            blk_post(n, b, (int)blockIdx.x * (int)(blockDim.x >> 5) + warp,
                     (int)(gridDim.x * (blockDim.x >> 5)), nt, t);
            small_sync();
        }
        t += (unsigned)nt;
        left -= nt;
    }
    if (active && team.role == 0) {
        if (valid) neuron_store(n, d, y.x, y.sp);
        thin_store(n, s, y, tile);
    }
    if (first) {
        if (INJ) *n.noise_cursor = z.cursor;
        *n.step = t;
        *n.dstep = t;
        if (t >= 0xffffff00ull) set_err(n, ERR_STEP_RANGE);
    }
}

// ---- dense networks: one CTA per tile ----------------------------------------------------------
// Networks of more row quads: the tile's psr and classes stream through shared memory in chunks of
// 64 rows (3-D TMA boxes, DN_STAGES in flight) and each chunk is scaled and summed for all the
// block's steps while it is there.
//   warp 0        issues the loads; then, lane = destination, runs the neurons' steps as the sums
//                 come in
//   warps 1-W     arrivals: find the rows whose source has a spike arriving, prepare the psr
//                 increments (event slots, exp tables), draw the neurons' noise
//   warp W + 1    lane = destination, rows in slot order: carries a chunk through the block's steps
//                 and stores it back.  A row is a chain of multiplications by its decay; a step's sum
//                 is a chain of additions over the rows, in the reference's order; the steps
//                 interleave eight such chains.
// Arrivals reach the tile in one of two ways, by the number of neurons with a spike that may arrive in
// the block (BlkDev::actn, known when the block starts):
//   light   (at most N / DN_LIGHT) k_blk_push has taken the spikes out along the outgoing map before:
//           step masks in a plane of one byte per slot, increments beside the slots' event state, and
//           a flag per 16 rows.  The arrival warps only collect the flagged rows.
//   heavy   the arrival warps look up every slot's source in the spike masks and make the increments.
// Either way 16 rows at a time, by the W warps in turn, into one of W buffers of step masks and
// increments that the sum warp reads; groups of 16 rows without an arrival take code that reads none.
// Why two: a pushed arrival costs half a dozen scattered accesses with the whole GPU to hide them, and
// reads no sources; a pulled one is found among its neighbours in the slot planes, and costs a pass
// over the sources.
constexpr int DN_ROWS = 64, DN_QUADS = 16;
constexpr int DN_STAGES = 4;
constexpr int DN_MAX_CHUNKS = 32;   // 2,048 slots per destination
constexpr int DN_GROUP_WORDS = 4 * DN_MAX_CHUNKS / 32;
constexpr int DN_LIGHT = 128;
constexpr int DN_ACT_WORDS = 1216;  // the bitmap row is kept in shared memory up to 38,912 neurons
constexpr int dn_threads(int W) { return 32 * (1 + W + 1); }
// Arrival warps a tile, and the blocks an SM then holds: eight where there is at most a tile an SM, else
// four.  A heavy block's arrivals are chains of loads, and with four warps on an SM of their own one tile's
// chains took longer than the per-step kernels, which spread them over the GPU.  160 steps at 200 to
// 320 Hz, up to 920 rows a neuron, us with four warps, with eight and step by step: 33x33 (35 tiles) 2782,
// 1710, 1676; 45x45 2879, 1784, 2223; 60x60 (113) 3052, 1907, 2746; 80x80 (200, four) 3276 and 3615; 100x100
// (313, four) 3524 and 4462.  Sixteen: 1327, 1349 and 1389, but such a block takes an SM, and 36 networks of
// 30x30 to 100x100 on streams of their own, near silent, took 55 us a step (eight 42, four 38; a batch 38).
constexpr int DN_FEW = 152;
constexpr int dn_blocks(int W) { return W == 4 ? 3 : 2; }
constexpr uint32_t DN_CHUNK = DN_ROWS * 32 * 4 + DN_QUADS * 32 * 2;

template <int W>  // arrival warps, and buffers: buffer k is filled by warp k
struct DenseSmem {
    uint8_t stage[DN_STAGES][DN_CHUNK];              // psr [16 quads][32] float4 | class [16][32] u16
    float4 binc[W][4][32];                           // increments of 16 rows
    uint32_t bmsk[W][4][32];                         // step masks, one byte per row
    uint32_t act[DN_ACT_WORDS];
    float sum[BLK_MAX_STEPS][32];
    float noise[BLK_MAX_STEPS][32];
    float dtab[BG3_MAX_DCLS];
    int4 src[W][2][4][32];                           // per arrival warp: a group's and the next one's
    uint32_t lc[W][2][4][32];                        // sources and delay classes
    int32_t ltab[BG3_MAX_DELAYS];
    uint32_t groups[DN_GROUP_WORDS];                 // the 16-row groups that have a buffer
    int any[W];                                      // bit q: quad q has arrivals; 16: several at a row
    int issued, failed;
    uint64_t full[DN_STAGES], empty[DN_STAGES];
    uint64_t bfull[W], bempty[W];
    uint64_t scanned, summed, drawn;
};
// What a batch's block takes: beside this the descriptor's copy, and 1 KB of the SM's 228 that each block has.
template <int W>
constexpr bool dn_fits()
{
    return dn_blocks(W) * (sizeof(DenseSmem<W>) + (sizeof(NetDev) + 127) / 128 * 128 + 1024) <= 228 * 1024;
}
static_assert(dn_fits<4>() && dn_fits<8>(), "an SM holds dn_blocks(W) blocks");

template <int W>
__device__ __forceinline__ void bar_events()
{
    asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory");
}

template <int W>
__device__ __forceinline__ bool dn_wait(const NetDev &n, DenseSmem<W> &s, uint64_t *bar, uint32_t parity)
{
    if (mbar_wait(bar, parity)) return true;
    set_err(n, ERR_TIMEOUT);
    *(volatile int *)&s.failed = 1;
    return false;
}

// The lane's rows of quad sources v with a spike that may arrive (bit r: row r).
__device__ __forceinline__ uint32_t dense_hits(const int4 &v, const uint32_t *act, int left)
{
    uint32_t h = 0u;
    if (left > 0) h |= (act[v.x >> 5] >> (v.x & 31)) & 1u;
    if (left > 1) h |= ((act[v.y >> 5] >> (v.y & 31)) & 1u) << 1;
    if (left > 2) h |= ((act[v.z >> 5] >> (v.z & 31)) & 1u) << 2;
    if (left > 3) h |= ((act[v.w >> 5] >> (v.w & 31)) & 1u) << 3;
    return h;
}

// One spike arriving at each of U slots p[u] (m[u]: its step's bit; 0: none), their loads issued
// together: the psr increments, with the event slots brought up to date
// (AllSpikingSynapses.cpp:327-334, AllDSSynapses.cpp:227-247).  m[u] is cleared where the synapse did
// not exist when the spike left, D[u] steps before.
template <int SYN, int U, int W>
__device__ __forceinline__ void dense_arrivals(const NetDev &n, const DenseSmem<W> &s, const uint32_t (&p)[U],
                                               const int (&D)[U], uint32_t (&m)[U], float (&inc)[U],
                                               unsigned long long t)
{
    // the first 16 bytes of a slot (W, u, r, last spike) and the next 8 (birth step, classes)
    float4 e[U];
    uint2 f[U];
#pragma unroll
    for (int u = 0; u < U; u++)
        if (m[u]) {
            const char *q = reinterpret_cast<const char *>(n.ev) + (size_t)p[u] * sizeof(EvSlot);
            e[u] = *reinterpret_cast<const float4 *>(q);
            f[u] = *reinterpret_cast<const uint2 *>(q + 16);
        }
    float xr[U], xu[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (!m[u]) continue;
        const uint32_t ta = (uint32_t)t + (uint32_t)(31 - __clz((int)m[u])), last = __float_as_uint(e[u].w);
        if ((int32_t)(ta - (uint32_t)D[u] - f[u].x) < 0) {
            m[u] = 0u;
        } else if (SYN == 1 && last != BG3_NO_SPIKE32) {
            const int pc = (int)((f[u].y >> 8) & 255u);
            xr[u] = exp_tab(n, n.p_xD[pc], ta - last, n.p_D[pc]);
            xu[u] = exp_tab(n, n.p_xF[pc], ta - last, n.p_F[pc]);
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        inc[u] = 0.0f;
        if (!m[u]) continue;
        const float dec = s.dtab[f[u].y & 255u];
        if (SYN == 1) {
            float uu = e[u].y, rr = e[u].z;
            if (__float_as_uint(e[u].w) != BG3_NO_SPIKE32) {
                const float Uc = n.p_U[(f[u].y >> 8) & 255u];
                rr = 1.0f + (rr * (1.0f - uu) - 1.0f) * xr[u];
                uu = Uc + uu * (1.0f - Uc) * xu[u];
            }
            inc[u] = (e[u].x / dec) * uu * rr;
            // one store of the slot's first half (nothing else writes W during a block)
            gst(reinterpret_cast<float4 *>(n.ev) + 2 * (size_t)p[u],
                make_float4(e[u].x, uu, rr,
                            __uint_as_float((uint32_t)t + (uint32_t)(31 - __clz((int)m[u])))));
        } else {
            inc[u] = e[u].x / dec;
        }
    }
}

// Whether the block from t on is light (pushed arrivals).  The line is not sharp: at N / 128, N / 512
// and N / 2048 the 100x100 and 180x180 networks' blocks take the same within 1 % from 0.3 to 300 Hz;
// with few neurons set a heavy block costs a fifth more than a light one (85 to 90 us against 74,
// 180x180), and a push grows with its arrivals (32 us for 250 spikes' 190,000).
__device__ __forceinline__ bool blk_light(const NetDev &n, const BlkDev &b, unsigned long long t)
{
    return (unsigned long long)b.actn[t & (BLK_ACT_ROWS - 1)] * DN_LIGHT <= (unsigned long long)n.N;
}

// Light blocks: the spikes taken out along the outgoing map.  A block of the grid serves 2,048 neurons
// (64 bitmap words) and every gridDim.y-th 128-synapse chunk of theirs; it lists the neurons with a
// spike, and its warps take them in turn, four synapses per lane.  A slot's step mask and increment
// wait for the tile's arrival warps (dense_collect); a synapse with several spikes in the block keeps
// only its mask.
constexpr int PUSH_WORDS = 64, PUSH_THREADS = 256;
template <int SYN>
__device__ __forceinline__ void blk_push(const NetDev &n, const BlkDev &b, int bx, int split, int nsplit, int nt)
{
    __shared__ int s_list[PUSH_WORDS * 32];
    __shared__ int s_n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const unsigned long long t = *n.step;
    if (!blk_light(n, b, t)) return;
    if (threadIdx.x < PUSH_WORDS && bx * PUSH_WORDS + (int)threadIdx.x < n.ntiles) {
        const int word = bx * PUSH_WORDS + (int)threadIdx.x;
        uint32_t w = b.act[(t & (BLK_ACT_ROWS - 1)) * n.ntiles + word];
        if (w) {
            int at = atomicAdd(&s_n, __popc(w));
            for (; w; w &= w - 1u) s_list[at++] = word * 32 + __ffs((int)w) - 1;
        }
    }
    __syncthreads();
    const int total = s_n;
    for (int it = warp; it < total; it += PUSH_THREADS / 32) {
        const int i = s_list[it];
        const unsigned long long h = b.hist[i];
        for (int c = 0; c < n.n_delays; c++) {
            const int D = n.ltab[c];
            const uint32_t m = (uint32_t)rotr64(h, (unsigned)t - (unsigned)D) & ((1u << nt) - 1u);
            if (!m) continue;
            const bool one = (m & (m - 1u)) == 0u;
            const uint32_t ta = (uint32_t)t + (uint32_t)(31 - __clz((int)m));
            const size_t ci = (size_t)c * n.N + i;
            const uint32_t b0 = n.outBegin[ci], k = n.outCount[ci];
            for (uint32_t base = (uint32_t)split * 128u; base < k; base += (uint32_t)nsplit * 128u) {
                constexpr int U = 4;
                uint32_t p[U];
                float4 e[U];
                uint2 f[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t j = base + (uint32_t)lane + 32u * u;
                    p[u] = j < k ? n.outMap[b0 + j] : 0xffffffffu;
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (p[u] != 0xffffffffu) {
                        const char *q = reinterpret_cast<const char *>(n.ev) + (size_t)p[u] * sizeof(EvSlot);
                        e[u] = *reinterpret_cast<const float4 *>(q);
                        f[u] = *reinterpret_cast<const uint2 *>(q + 16);
                    }
                float xr[U], xu[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (p[u] == 0xffffffffu || !one) continue;
                    const uint32_t last = __float_as_uint(e[u].w);
                    if ((int32_t)(ta - (uint32_t)D - f[u].x) < 0) {
                        p[u] = 0xffffffffu;  // the synapse did not exist when the spike left
                    } else if (SYN == 1 && last != BG3_NO_SPIKE32) {
                        const int pc = (int)((f[u].y >> 8) & 255u);
                        xr[u] = exp_tab(n, n.p_xD[pc], ta - last, n.p_D[pc]);
                        xu[u] = exp_tab(n, n.p_xF[pc], ta - last, n.p_F[pc]);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (p[u] == 0xffffffffu) continue;
                    if (one) {
                        float4 *q = reinterpret_cast<float4 *>(n.ev) + 2 * (size_t)p[u];
                        const float dec = n.dtab[f[u].y & 255u];
                        float inc;
                        if (SYN == 1) {
                            float uu = e[u].y, rr = e[u].z;
                            if (__float_as_uint(e[u].w) != BG3_NO_SPIKE32) {
                                const float Uc = n.p_U[(f[u].y >> 8) & 255u];
                                rr = 1.0f + (rr * (1.0f - uu) - 1.0f) * xr[u];
                                uu = Uc + uu * (1.0f - Uc) * xu[u];
                            }
                            inc = (e[u].x / dec) * uu * rr;
                            gst(q, make_float4(e[u].x, uu, rr, __uint_as_float(ta)));
                        } else {
                            inc = e[u].x / dec;
                        }
                        gst(&n.ev[p[u]].pad1, __float_as_uint(inc));
                    }
                    gst(&b.msk[p[u]], (uint8_t)m);
                    // slot p: tile p / (128 Mq), row quad (p / 128) % Mq; 16 rows a flag
                    const uint32_t q4 = p[u] >> 7, tile = q4 / (uint32_t)n.Mq, g = (q4 - tile * (uint32_t)n.Mq) >> 2;
                    atomicOr(&b.gflag[tile * DN_GROUP_WORDS + (g >> 5)], 1u << (g & 31));
                }
            }
        }
    }
}

template <int SYN>
__global__ void __launch_bounds__(PUSH_THREADS) k_blk_push(const __grid_constant__ NetDev n,
                                                           const __grid_constant__ BlkDev b, int nt)
{
    blk_push<SYN>(n, b, blockIdx.x, blockIdx.y, gridDim.y, nt);
}

// Batched form: grid.z indexes the networks that run dense blocks.
template <int SYN>
__global__ void __launch_bounds__(PUSH_THREADS) k_blk_push_batch(const NetDev *nets, const BlkDev *blks,
                                                                 const int *dense, int nt)
{
    __shared__ __align__(16) NetDev s_net;
    const int k = dense[blockIdx.z];
    if ((int)blockIdx.x * PUSH_WORDS >= nets[k].ntiles) return;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(nets + k);
    uint4 *d4 = reinterpret_cast<uint4 *>(&s_net);
    for (int i = threadIdx.x; i < (int)(sizeof(NetDev) / 16); i += blockDim.x) d4[i] = s4[i];
    blk_push<SYN>(s_net, blks[k], blockIdx.x, blockIdx.y, gridDim.y, nt);
}

// The 16 rows of buffer bf where a synapse has several spikes arriving in the block: those arrivals
// run at their steps.  psr in place, the steps' sums in and out.
template <int SYN, int W>
__device__ __noinline__ void dense_late(const NetDev &n, const DenseSmem<W> &s, int tile, int row0, int bf,
                                        int nt, unsigned long long t, float4 *ps4, const uint16_t *cw,
                                        float *acc)
{
    const int lane = threadIdx.x & 31, d = tile * 32 + lane;
    for (int r = 0; r < 16; r++) {
        const int q = r >> 2, i = r & 3;
        float *pr = reinterpret_cast<float *>(ps4 + q * 32) + i;
        const float dec = s.dtab[(cw[q * 32] >> (4 * i)) & 15u];
        const uint32_t m = (s.bmsk[bf][q][lane] >> (8 * i)) & 255u;
        const bool many = (m & (m - 1u)) != 0u;
        float x = *pr;
        for (int j = 0; j < nt; j++) {
            if ((m >> j) & 1u) {
                if (many) {
                    const uint32_t p = (uint32_t)slot_pos(row0 + r, d, n.Mq);
                    const unsigned long long tj = t + (unsigned)j;
                    float a;
                    if (arrival<SYN>(n, p, d, n.src[p], (uint32_t)tj - (uint32_t)n.ltab[n.lcls[p]], tj, a))
                        x = x + a;
                } else {
                    x = x + reinterpret_cast<const float *>(&s.binc[bf][q][lane])[i];
                }
            }
            x = x * dec;
            acc[j] = acc[j] + x;
        }
        *pr = x;
    }
}

// Two products in one instruction, each rounded as a single multiplication.
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 r;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
        " mul.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}\n"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// x + inc where m has the bit, as one predicated addition (a branch per step and row otherwise).
template <uint32_t BIT>
__device__ __forceinline__ void add_if(float &x, uint32_t m, float inc)
{
    asm("{\n .reg .pred p;\n .reg .b32 b;\n and.b32 b, %1, %2;\n setp.ne.u32 p, b, 0;\n"
        " @p add.rn.f32 %0, %0, %3;\n}\n"
        : "+f"(x) : "r"(m), "n"(BIT), "f"(inc));
}
template <int J>
__device__ __forceinline__ void add_hits(float2 &x, float2 &y, uint32_t m, const float4 &in)
{
    add_if<0x1u << J>(x.x, m, in.x);
    add_if<0x100u << J>(x.y, m, in.y);
    add_if<0x10000u << J>(y.x, m, in.z);
    add_if<0x1000000u << J>(y.y, m, in.w);
}

// Four rows through the block's steps: psr scaled, and added to each step's sum in row order.  The
// products of a step's four rows are independent of each other, as are the steps' sums of a row, so neither half of this waits on itself.  HIT: rows may have an arrival, at the step whose
// bit is set in the row's byte of m (bit j: step j).  S: the steps computed, nt of them used; FULL: nt = S.
template <int S, bool FULL, bool HIT>
__device__ __forceinline__ void dense_quad(float4 &v, const float4 &dc, float (&acc)[S], int nt,
                                           uint32_t m, const float4 &in)
{
    float2 p[S][2];
    float2 x = make_float2(v.x, v.y), y = make_float2(v.z, v.w);
    const float2 dx = make_float2(dc.x, dc.y), dy = make_float2(dc.z, dc.w);
#pragma unroll
    for (int j = 0; j < S; j++) {
        if (HIT) {
            if (j == 0) add_hits<0>(x, y, m, in);
            if (j == 1) add_hits<1>(x, y, m, in);
            if (j == 2) add_hits<2>(x, y, m, in);
            if (j == 3) add_hits<3>(x, y, m, in);
            if (j == 4) add_hits<4>(x, y, m, in);
            if (j == 5) add_hits<5>(x, y, m, in);
            if (j == 6) add_hits<6>(x, y, m, in);
            if (j == 7) add_hits<7>(x, y, m, in);
        }
        p[j][0] = x = mul2(x, dx);
        p[j][1] = y = mul2(y, dy);
        // a shorter block keeps psr as of its last step; the sums past it are not used
        if (!FULL && j == nt - 1) v = make_float4(x.x, x.y, y.x, y.y);
    }
    if (FULL) v = make_float4(x.x, x.y, y.x, y.y);
#pragma unroll
    for (int j = 0; j < S; j++) acc[j] = acc[j] + p[j][0].x;
#pragma unroll
    for (int j = 0; j < S; j++) acc[j] = acc[j] + p[j][0].y;
#pragma unroll
    for (int j = 0; j < S; j++) acc[j] = acc[j] + p[j][1].x;
#pragma unroll
    for (int j = 0; j < S; j++) acc[j] = acc[j] + p[j][1].y;
}

// The decay factors of a row quad's four class codes.
template <int W>
__device__ __forceinline__ float4 dense_decay(const DenseSmem<W> &s, uint32_t c)
{
    return make_float4(s.dtab[c & 15u], s.dtab[(c >> 4) & 15u], s.dtab[(c >> 8) & 15u],
                       s.dtab[(c >> 12) & 15u]);
}

// The sum warp: the block's steps over all chunks, psr scaled in place, a step's sum over the rows in
// order.  S and FULL as in dense_quad.  Measured as one warp on an SM, cycles a row of 32
// destinations: eight steps 28 with 16 rows at a time and paired products, 33 with eight rows at a
// time, 42 with four; two warps of four steps each, one after the other, 18 each (and 28 each beside
// another tile's two).
template <int SYN, int S, bool FULL, int W>
__device__ __forceinline__ void dense_sums(const NetDev &n, DenseSmem<W> &s, const CUtensorMap *tm_psr,
                                           int tile, int nch, int nt, unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    float acc[S];
#pragma unroll
    for (int j = 0; j < S; j++) acc[j] = 0.0f;
    bool ok = dn_wait(n, s, &s.scanned, 0);
    int k = 0;  // 16-row groups with a buffer so far
    for (int c = 0; ok && c < nch; c++) {
        const int st = c % DN_STAGES;
        ok = dn_wait(n, s, &s.full[st], (uint32_t)((c / DN_STAGES) & 1));
        if (!ok) break;
        float4 *ps4 = reinterpret_cast<float4 *>(s.stage[st]) + lane;
        const uint16_t *cw = reinterpret_cast<const uint16_t *>(s.stage[st] + DN_ROWS * 32 * 4) + lane;
        const uint32_t groups = s.groups[c >> 3] >> (4 * (c & 7));
#pragma unroll 1
        for (int g = 0; g < 4; g++, ps4 += 4 * 32, cw += 4 * 32) {
            const bool looked = (groups >> g) & 1u;
            const int bf = k % W;
            int any = 0;
            if (looked) {
                ok = dn_wait(n, s, &s.bfull[bf], (uint32_t)((k / W) & 1));
                if (!ok) break;
                k++;
                any = s.any[bf];
            }
            if (any == 0) {
                float4 v[4], dc[4];
                uint32_t cl[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    v[q] = ps4[q * 32];
                    cl[q] = cw[q * 32];
                }
#pragma unroll
                for (int q = 0; q < 4; q++) dc[q] = dense_decay(s, cl[q]);
#pragma unroll
                for (int q = 0; q < 4; q++) dense_quad<S, FULL, false>(v[q], dc[q], acc, nt, 0u, v[q]);
#pragma unroll
                for (int q = 0; q < 4; q++) ps4[q * 32] = v[q];
            } else if (!(any & 16)) {
#pragma unroll 1
                for (int q = 0; q < 4; q += 2) {
                    float4 v0 = ps4[q * 32], v1 = ps4[(q + 1) * 32];
                    const float4 d0 = dense_decay(s, cw[q * 32]), d1 = dense_decay(s, cw[(q + 1) * 32]);
                    if ((any >> q) & 3) {
                        dense_quad<S, FULL, true>(v0, d0, acc, nt, s.bmsk[bf][q][lane], s.binc[bf][q][lane]);
                        dense_quad<S, FULL, true>(v1, d1, acc, nt, s.bmsk[bf][q + 1][lane], s.binc[bf][q + 1][lane]);
                    } else {
                        dense_quad<S, FULL, false>(v0, d0, acc, nt, 0u, v0);
                        dense_quad<S, FULL, false>(v1, d1, acc, nt, 0u, v1);
                    }
                    ps4[q * 32] = v0;
                    ps4[(q + 1) * 32] = v1;
                }
            } else {
                float a[S];
#pragma unroll
                for (int j = 0; j < S; j++) a[j] = acc[j];
                dense_late<SYN>(n, s, tile, c * DN_ROWS + 16 * g, bf, nt, t, ps4, cw, a);
#pragma unroll
                for (int j = 0; j < S; j++) acc[j] = a[j];
            }
            if (looked) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&s.bempty[bf]);
            }
        }
        if (!ok) break;
        fence_async_smem();  // the TMA store (async proxy) must see these writes
        __syncwarp();
        if (lane == 0) {
            tma_store_3d(tm_psr, 0, c * DN_QUADS, tile, s.stage[st]);
            bulk_commit();
            if (c >= 1) {
                bulk_wait_read1();
                mbar_arrive(&s.empty[(c - 1) % DN_STAGES]);
            }
        }
        __syncwarp();
    }
    if (lane == 0) bulk_wait_read_all();
#pragma unroll
    for (int j = 0; j < S; j++)
        if (j < nt) s.sum[j][lane] = acc[j];
    __syncwarp();
    if (ok && lane == 0) mbar_arrive(&s.summed);
}

// Sources and delay classes (a byte per row) of 16 rows of the lane's destination, on their way to
// shared memory.
template <int W>
__device__ __forceinline__ void dense_sources(DenseSmem<W> &s, int w, int st, const int4 *S,
                                              const uint32_t *L, int q0, int cnt)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (cnt > 4 * (q0 + q)) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&s.src[w][st][q][lane])),
                         "l"(&S[(size_t)(q0 + q) * 32]) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&s.lc[w][st][q][lane])),
                         "l"(&L[(size_t)(q0 + q) * 32]) : "memory");
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The arrival warps of a light block: the flagged groups' masks and increments, both planes left
// clean for the next block.
template <int W>
__device__ __forceinline__ void dense_collect(const NetDev &n, const BlkDev &b, DenseSmem<W> &s, int tile, int w)
{
    const int lane = threadIdx.x & 31;
    if (w < DN_GROUP_WORDS && lane == 0) {
        const uint32_t f = b.gflag[tile * DN_GROUP_WORDS + w];
        s.groups[w] = f;
        if (f) b.gflag[tile * DN_GROUP_WORDS + w] = 0u;
    }
    bar_events<W>();
    if (lane == 0) mbar_arrive(&s.scanned);
    uint32_t *M = reinterpret_cast<uint32_t *>(b.msk) + (size_t)tile * n.Mq * 32 + lane;
    EvSlot *E = n.ev + (size_t)tile * n.Mq * 128 + (size_t)lane * 4;
    // this warp's groups in order, -1 after the last
    int word = 0, k = 0, used = 0;
    uint32_t left = s.groups[0];
    auto next = [&]() {
        for (;;) {
            if (!left) {
                if (++word >= DN_GROUP_WORDS) return -1;
                left = s.groups[word];
                continue;
            }
            const int g = 32 * word + __ffs((int)left) - 1;
            left &= left - 1u;
            if (k++ % W == w) return g;
        }
    };
    auto masks = [&](int g, uint32_t (&m)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q++) m[q] = g >= 0 && 4 * g + q < n.Mq ? M[(size_t)(4 * g + q) * 32] : 0u;
    };
    auto single = [](uint32_t m, int r) {
        const uint32_t mr = (m >> (8 * r)) & 255u;
        return mr != 0u && (mr & (mr - 1u)) == 0u;
    };
    auto incs = [&](int g, const uint32_t (&m)[4], uint32_t (&in)[16]) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (m[q]) {
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (single(m[q], r)) in[4 * q + r] = E[(size_t)(4 * g + q) * 128 + r].pad1;
            }
    };
    // Two groups ahead: the masks of one and the increments of the other are on their way while a
    // group is handed over (each group's loads waited for in turn were about three microseconds a group:
    // a light block of 180x180 neurons with an arrival in most groups took 280 us, an empty one 74;
    // with a few hundred spikes in the network its blocks went from 137 to 118 us).
    int g0 = next(), g1 = g0 >= 0 ? next() : -1;
    uint32_t m0[4], m1[4], in0[16], in1[16];
    masks(g0, m0);
    masks(g1, m1);
    incs(g0, m0, in0);
    while (g0 >= 0) {
        const int g2 = g1 >= 0 ? next() : -1;
        uint32_t m2[4], any = 0u;
        masks(g2, m2);
        incs(g1, m1, in1);
        if (used > 0 && !dn_wait(n, s, &s.bempty[w], (uint32_t)((used - 1) & 1))) return;
        used++;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s.bmsk[w][q][lane] = m0[q];
            if (m0[q]) {
                M[(size_t)(4 * g0 + q) * 32] = 0u;
                any |= 1u << q;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    if (single(m0[q], r)) {
                        reinterpret_cast<float *>(&s.binc[w][q][lane])[r] = __uint_as_float(in0[4 * q + r]);
                        E[(size_t)(4 * g0 + q) * 128 + r].pad1 = 0u;
                    } else if ((m0[q] >> (8 * r)) & 255u) {
                        any |= 16u;
                    }
                }
            }
        }
        any = __reduce_or_sync(0xffffffffu, any);
        __syncwarp();
        if (lane == 0) {
            s.any[w] = (int)any;
            mbar_arrive(&s.bfull[w]);
        }
        g0 = g1;
        g1 = g2;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            m0[q] = m1[q];
            m1[q] = m2[q];
        }
#pragma unroll
        for (int q = 0; q < 16; q++) in0[q] = in1[q];
    }
}

template <int SYN, int W>
__device__ __forceinline__ void dense_events(const NetDev &n, const BlkDev &b, DenseSmem<W> &s, int tile,
                                             int w, int cnt, int nch, int nt, unsigned long long t)
{
    const int lane = threadIdx.x & 31, tid = 32 * w + lane;
    const size_t base = (size_t)tile * n.Mq * 32 + lane;
    const int4 *S = reinterpret_cast<const int4 *>(n.src) + base;
    const uint32_t *L = reinterpret_cast<const uint32_t *>(n.lcls) + base;
    const uint32_t *act = b.act + (t & (BLK_ACT_ROWS - 1)) * n.ntiles;
    if (w < DN_GROUP_WORDS && lane == 0) {
        const int k = 4 * nch - 32 * w;
        s.groups[w] = k >= 32 ? 0xffffffffu : k > 0 ? (1u << k) - 1u : 0u;
    }
    if (n.ntiles <= DN_ACT_WORDS) {
        for (int i = tid; i < n.ntiles; i += 32 * W) s.act[i] = act[i];
        act = s.act;
    }
    bar_events<W>();
    if (lane == 0) mbar_arrive(&s.scanned);
    if (w < 4 * nch) dense_sources(s, w, 0, S, L, 4 * w, cnt);
    for (int g = w, used = 0; g < 4 * nch; g += W) {
        const int st = used & 1;
        if (g + W < 4 * nch) {
            dense_sources(s, w, st ^ 1, S, L, 4 * (g + W), cnt);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        // hits, then the hits' sources' masks: the steps of the block at which a spike arrives (each
        // lane reads only what it copied itself)
        uint32_t h16 = 0u;
#pragma unroll
        for (int q = 0; q < 4; q++)
            h16 |= dense_hits(s.src[w][st][q][lane], act, cnt - 4 * (4 * g + q)) << (4 * q);
        const bool some = __any_sync(0xffffffffu, h16 != 0u);
        if (used > 0 && !dn_wait(n, s, &s.bempty[w], (uint32_t)((used - 1) & 1))) return;
        used++;
        uint32_t any = 0u;  // bit q: quad q has an arrival; 16: a row has several
        if (some) {
            // Four masks and two arrivals in flight a lane.  The unrolled code runs in full while any lane
            // has a hit left: with one and one 10,000 neurons at 0.8 Hz take 57 us a block instead of 64,
            // but 32,400 at 300 Hz 488 instead of 420; four and four cost both a third; both forms, by
            // the group's hits, gain nothing (63, 444).
            uint8_t *mb = reinterpret_cast<uint8_t *>(&s.bmsk[w][0][lane]);  // row r: mb[128 (r / 4) + r % 4]
            const uint8_t *lb = reinterpret_cast<const uint8_t *>(&s.lc[w][st][0][lane]);
            const int *sb = reinterpret_cast<const int *>(&s.src[w][st][0][lane]);
            float *ib = reinterpret_cast<float *>(&s.binc[w][0][lane]);
            const uint32_t p0 = (uint32_t)slot_pos(16 * g, tile * 32 + lane, n.Mq);
#pragma unroll
            for (int q = 0; q < 4; q++) s.bmsk[w][q][lane] = 0u;
            uint32_t one = 0u;
            while (h16) {
                constexpr int U = 4;
                int r[U];
                unsigned long long hs[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    r[u] = h16 ? __ffs((int)h16) - 1 : -1;
                    h16 &= h16 - 1u;
                    if (r[u] >= 0) hs[u] = b.hist[sb[128 * (r[u] >> 2) + (r[u] & 3)]];
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (r[u] >= 0) {
                        const int D = s.ltab[lb[128 * (r[u] >> 2) + (r[u] & 3)]];
                        const uint32_t m = (uint32_t)rotr64(hs[u], (unsigned)t - (unsigned)D) & ((1u << nt) - 1u);
                        if (!m) continue;
                        mb[128 * (r[u] >> 2) + (r[u] & 3)] = (uint8_t)m;
                        any |= 1u << (r[u] >> 2);
                        if (m & (m - 1u)) {
                            any |= 16u;
                        } else {
                            one |= 1u << r[u];
                            // towards the L1: a batch's loads below then wait for its first time only
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(&n.ev[p0 + 128u * (r[u] >> 2) + (r[u] & 3)]));
                        }
                    }
            }
            while (one) {
                constexpr int U = 2;
                uint32_t p[U], m[U];
                int r[U], D[U];
                float inc[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    m[u] = 0u;
                    r[u] = -1;
                    if (one) {
                        r[u] = __ffs((int)one) - 1;
                        one &= one - 1u;
                        r[u] = 128 * (r[u] >> 2) + (r[u] & 3);
                        m[u] = mb[r[u]];
                        D[u] = s.ltab[lb[r[u]]];
                        p[u] = p0 + (uint32_t)r[u];
                    }
                }
                dense_arrivals<SYN, U>(n, s, p, D, m, inc, t);
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (r[u] >= 0) {
                        mb[r[u]] = (uint8_t)m[u];
                        ib[r[u]] = inc[u];
                    }
            }
            any = __reduce_or_sync(0xffffffffu, any);
        }
        __syncwarp();
        if (lane == 0) {
            s.any[w] = (int)any;
            mbar_arrive(&s.bfull[w]);
        }
    }
}

template <int SYN, int W>
__device__ __forceinline__ void blk_dense_tile(const NetDev &n, const BlkDev &b,
                                               const CUtensorMap *tm_psr, const CUtensorMap *tm_cls,
                                               const int tile, const int nt, DenseSmem<W> &s)
{
    // Roles rotate with the block: warp k of every block is issued by the same quarter of its SM, and
    // the sum warps of the blocks that share an SM (152 apart in a first wave) are the busy ones.
    const int lane = threadIdx.x & 31;
    const int warp = (int)(threadIdx.x / 32 + blockIdx.x / 152) % (W + 2);
    const int d = tile * 32 + lane;
    const bool valid = d < n.N;
    for (int i = threadIdx.x; i < n.n_dcls; i += blockDim.x) s.dtab[i] = n.dtab[i];
    for (int i = threadIdx.x; i < n.n_delays; i += blockDim.x) s.ltab[i] = n.ltab[i];
    const int cnt = valid ? (int)n.count[d] : 0;
    const int nch = (__reduce_max_sync(0xffffffffu, cnt) + DN_ROWS - 1) / DN_ROWS;
    if (threadIdx.x == 0) {
        for (int i = 0; i < DN_STAGES; i++) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 1);
        }
        for (int i = 0; i < W; i++) {
            mbar_init(&s.bfull[i], 1);
            mbar_init(&s.bempty[i], 1);
        }
        mbar_init(&s.summed, 1);
        mbar_init(&s.scanned, W);
        mbar_init(&s.drawn, W);
        fence_mbar_init();
        s.issued = 0;
        s.failed = 0;
    }
    __syncthreads();
    pdl_wait();  // the block before has finished
    pdl_trigger();
    const unsigned long long t = *n.step;

    if (warp == 0) {  // ------------------------------------------------ loads, then the neurons
        bool ok = true;
        if (lane == 0) {
            for (int c = 0; c < nch; c++) {
                const int st = c % DN_STAGES;
                if (c >= DN_STAGES &&
                    !dn_wait(n, s, &s.empty[st], (uint32_t)((c / DN_STAGES - 1) & 1))) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&s.full[st], DN_CHUNK);
                tma_load_3d(s.stage[st], tm_psr, 0, c * DN_QUADS, tile, &s.full[st]);
                tma_load_3d(s.stage[st] + DN_ROWS * 32 * 4, tm_cls, 0, c * DN_QUADS, tile, &s.full[st]);
                *(volatile int *)&s.issued = c + 1;
            }
        }
        NeuronIn x;
        float sp = 0.0f;
        unsigned long long hist = 0ull;
        if (valid) {
            neuron_load(n, d, x);
            sp = n.sp[d];
            hist = b.hist[d];
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) ok = dn_wait(n, s, &s.drawn, 0);
        StepRun run = step_run(n, d, x, t);
        uint32_t fired = 0u;
#pragma unroll 1
        for (int j = 0; ok && j < nt; j++) {
            // step t + j takes the sum of step t + j - 1
            if (j == 1 && !(ok = dn_wait(n, s, &s.summed, 0))) break;
            if (j > 0) sp = s.sum[j - 1][lane];
            if (step_neuron(n, d, valid, x, sp, s.noise[j][lane], t + (unsigned)j, run)) fired |= 1u << j;
        }
        if (ok && nt == 1) ok = dn_wait(n, s, &s.summed, 0);
        if (ok) {
            sp = s.sum[nt - 1][lane];
            blk_finish<SYN>(n, b, tile, d, valid, x, sp, hist, fired, nt, t);
        }
    } else if (warp <= W) {  // ------------------------------------------- arrivals
        const int w = warp - 1;
        if (blk_light(n, b, t)) dense_collect(n, b, s, tile, w);
        else dense_events<SYN>(n, b, s, tile, w, cnt, nch, nt, t);
        for (int j = w; j < nt; j += W)
            s.noise[j][lane] = normal_device(n.noise_seed, t + (unsigned)j, d);
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.drawn);
    } else {  // --------------------------------------------------------------------- sums
        // a shorter block's chains are shorter where they are written out for its steps: a call of one
        // step on the 100x100 network at its target rate 52 us with eight, 27 with one; of four 45 and 34
        if (nt == BLK_MAX_STEPS) dense_sums<SYN, BLK_MAX_STEPS, true>(n, s, tm_psr, tile, nch, nt, t);
        else if (nt > 4) dense_sums<SYN, BLK_MAX_STEPS, false>(n, s, tm_psr, tile, nch, nt, t);
        else if (nt > 2) dense_sums<SYN, 4, false>(n, s, tm_psr, tile, nch, nt, t);
        else if (nt == 2) dense_sums<SYN, 2, true>(n, s, tm_psr, tile, nch, nt, t);
        else dense_sums<SYN, 1, true>(n, s, tm_psr, tile, nch, nt, t);
    }
    __syncthreads();
    if (*(volatile int *)&s.failed && threadIdx.x == 0) {
        // a wait gave up: the loads in flight land before the shared memory goes away
        const int issued = *(volatile int *)&s.issued;
        for (int c = max(0, issued - DN_STAGES); c < issued; c++)
            if (!mbar_wait(&s.full[c % DN_STAGES], (uint32_t)((c / DN_STAGES) & 1))) break;
    }
}

template <int SYN, int W>
__global__ void __launch_bounds__(dn_threads(W), dn_blocks(W)) k_blk_dense(const __grid_constant__ NetDev n,
                                                                           const __grid_constant__ BlkDev b,
                                                                           const __grid_constant__ CUtensorMap tm_psr,
                                                                           const __grid_constant__ CUtensorMap tm_cls,
                                                                           int nt)
{
    // declared with its alignment and used as it is: arithmetic on the address would hide from the
    // compiler that it is shared memory, and every access would be a generic one
    extern __shared__ __align__(128) uint8_t smem_dense[];
    blk_dense_tile<SYN>(n, b, &tm_psr, &tm_cls, blockIdx.x, nt, *reinterpret_cast<DenseSmem<W> *>(smem_dense));
}

// Batched form: tiles[b] = (network, tile), heaviest first; maps as in k_sweep_batch.
template <int SYN, int W>
__global__ void __launch_bounds__(dn_threads(W), dn_blocks(W)) k_blk_dense_batch(const NetDev *nets,
                                                                                 const BlkDev *blks,
                                                                                 const CUtensorMap *maps,
                                                                                 const int2 *tiles, int nt)
{
    extern __shared__ __align__(128) uint8_t smem_dense[];
    __shared__ __align__(16) NetDev s_net;
    const int2 tr = tiles[blockIdx.x];
    const uint4 *s4 = reinterpret_cast<const uint4 *>(nets + tr.x);
    uint4 *d4 = reinterpret_cast<uint4 *>(&s_net);
    for (int i = threadIdx.x; i < (int)(sizeof(NetDev) / 16); i += blockDim.x) d4[i] = s4[i];
    const BlkDev b = blks[tr.x];
    __syncthreads();
    blk_dense_tile<SYN>(s_net, b, &maps[2 * tr.x], &maps[2 * tr.x + 1], tr.y, nt,
                        *reinterpret_cast<DenseSmem<W> *>(smem_dense));
}

// ---- launchers --------------------------------------------------------------------------------
template <typename... KArgs, typename... Args>
static void launch_dep(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s,
                       Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

bool blk_thin_ok(int Mq) { return Mq <= BLK_THIN_QUADS; }
bool blk_dense_ok(int Mq) { return Mq <= DN_MAX_CHUNKS * DN_QUADS; }

void launch_blk_masks(const NetDev &h, const BlkDev &b, cudaStream_t s)
{
    cudaMemsetAsync(b.hist, 0, (size_t)h.Np * sizeof(*b.hist), s);
    if (b.actn) cudaMemsetAsync(b.actn, 0, BLK_ACT_ROWS * sizeof(*b.actn), s);
    k_blk_scatter<<<dim3(std::min((h.N + 255) / 256, 16), BG3_RING), 256, 0, s>>>(h, b);
    k_blk_act<<<(h.Np + 255) / 256, 256, 0, s>>>(h, b);
}

void launch_blk_ring(const NetDev &h, const BlkDev &b, cudaStream_t s)
{
    cudaMemsetAsync(h.ring_n, 0, BG3_RING * sizeof(*h.ring_n), s);
    k_blk_ring<<<(h.N + 255) / 256, 256, 0, s>>>(h, b);
}

// Blocks, tiles per block and warps per tile of a small network's launch; 0 blocks when it does not fit
// a cluster of eight (SMALL_SMEM of shared memory per block).
constexpr size_t SMALL_SMEM = 200 * 1024;
struct SmallShape {
    int blocks, tiles, team;
};
static SmallShape small_shape(const NetDev &h)
{
    SmallShape s = {0, h.ntiles <= 32 ? std::min(4, h.ntiles) : BLK_THIN_WARPS, 1};
    s.tiles = (int)std::min<size_t>(s.tiles, SMALL_SMEM / blk_thin_smem(h.Mq, BLK_TEAM, false));
    if (s.tiles < 1) return s;
    s.team = std::min(BLK_TEAM, BLK_THIN_WARPS / s.tiles);
    s.blocks = (h.ntiles + s.tiles - 1) / s.tiles;
    if (s.blocks > 8) s.blocks = 0;
    return s;
}
bool blk_small_ok(const NetDev &h) { return small_shape(h).blocks > 0; }

template <int SYN, bool INJ>
static void launch_small_t(const NetDev &h, const BlkDev &b, int nsteps, int T, cudaStream_t s)
{
    const SmallShape p = small_shape(h);
    const size_t sm = (size_t)p.tiles * blk_thin_smem(h.Mq, p.team, false);
    // the most any network takes, not this one's: the limit belongs to the kernel, and another thread's
    // wider network may be between this call and its launch
    cudaFuncSetAttribute(k_blk_small<SYN, INJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_SMEM);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(p.blocks);
    cfg.blockDim = dim3(32 * p.tiles * p.team);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_blk_small<SYN, INJ>, h, b, p.team, nsteps, T);
}

// nsteps steps of a small network, T at a time, in one launch.
void launch_blk_small(const NetDev &h, const BlkDev &b, int nsteps, int T, cudaStream_t s)
{
    switch (h.syn_kind * 2 + (h.noise_mode == 1 ? 1 : 0)) {
    case 1: launch_small_t<0, true>(h, b, nsteps, T, s); break;
    case 2: launch_small_t<1, false>(h, b, nsteps, T, s); break;
    case 3: launch_small_t<1, true>(h, b, nsteps, T, s); break;
    case 4: launch_small_t<2, false>(h, b, nsteps, T, s); break;
    case 5: launch_small_t<2, true>(h, b, nsteps, T, s); break;
    case 6: launch_small_t<3, false>(h, b, nsteps, T, s); break;
    case 7: launch_small_t<3, true>(h, b, nsteps, T, s); break;
    default: launch_small_t<0, false>(h, b, nsteps, T, s); break;
    }
}

// At most 44 KB of shared memory per block beside a batch's descriptor (48 KB is what a launch may
// use without opting in), so that several blocks share an SM.
static int thin_tiles_for(int Mq, int team) { return std::max(1, (int)(45056 / blk_thin_smem(Mq, team, team == 1))); }

// Few tiles leave the SMs idle while one warp a tile waits for itself: then four warps a tile, up to
// TEAM_TILES tiles (four an SM, which its registers hold), and the tiles spread over the SMs.  With one
// warp and with four: 100x100 without synapses 859 and 735 us for 1,000 steps, 90x90 Izhikevich 1663
// and 1549 for 500; the 64-network batch (8,500 tiles), whose SMs are full, ran 10.8 ms with one and
// 12 to 13 with the bookkeeping of several.
constexpr int TEAM_TILES = 4 * 152;

template <int SIZE>
static void launch_thin_t(const NetDev &h, const BlkDev &b, int nt, cudaStream_t s)
{
    const int w = std::max(1, std::min({BLK_THIN_WARPS / SIZE, thin_tiles_for(h.Mq, SIZE), h.ntiles / 152}));
    const int blocks = (h.ntiles + w - 1) / w, threads = 32 * w * SIZE;
    const size_t sm = w * blk_thin_smem(h.Mq, SIZE, SIZE == 1);
    switch (h.syn_kind) {
    case 1: launch_dep(k_blk_thin<1, SIZE>, blocks, threads, sm, s, h, b, nt); break;
    case 2: launch_dep(k_blk_thin<2, SIZE>, blocks, threads, sm, s, h, b, nt); break;
    case 3: launch_dep(k_blk_thin<3, SIZE>, blocks, threads, sm, s, h, b, nt); break;
    default: launch_dep(k_blk_thin<0, SIZE>, blocks, threads, sm, s, h, b, nt); break;
    }
}
void launch_blk_thin(const NetDev &h, const BlkDev &b, int nt, cudaStream_t s)
{
    if (h.ntiles <= TEAM_TILES) launch_thin_t<BLK_TEAM>(h, b, nt, s);
    else launch_thin_t<1>(h, b, nt, s);
    if (h.syn_kind >= 2) launch_dep(k_blk_post, 152, 256, 0, s, h, b, nt);
}

// tiles: n thin entries, each network's run padded to a multiple of `pad` entries; a block takes a
// divisor of pad, so that it serves one network.
template <int SIZE>
static void launch_thin_batch_t(int syn_kind, const NetDev *nets, const BlkDev *blks, const int2 *tiles, int n,
                                int pad, int max_mq, int nt, cudaStream_t s)
{
    int w = std::min({pad, BLK_THIN_WARPS / SIZE, thin_tiles_for(max_mq, SIZE)});
    while (pad % w) w--;
    const int blocks = (n + w - 1) / w, ws = (int)blk_thin_smem(max_mq, SIZE, SIZE == 1), threads = 32 * w * SIZE;
    const size_t sm = (size_t)w * ws;
    switch (syn_kind) {
    case 1: launch_dep(k_blk_thin_batch<1, SIZE>, blocks, threads, sm, s, nets, blks, tiles, n, ws, nt); break;
    case 2: launch_dep(k_blk_thin_batch<2, SIZE>, blocks, threads, sm, s, nets, blks, tiles, n, ws, nt); break;
    case 3: launch_dep(k_blk_thin_batch<3, SIZE>, blocks, threads, sm, s, nets, blks, tiles, n, ws, nt); break;
    default: launch_dep(k_blk_thin_batch<0, SIZE>, blocks, threads, sm, s, nets, blks, tiles, n, ws, nt); break;
    }
}
void launch_blk_thin_batch(int syn_kind, const NetDev *nets, const BlkDev *blks, int nets_n,
                           const int2 *tiles, int n, int pad, int max_mq, int nt, cudaStream_t s)
{
    if (n <= TEAM_TILES) launch_thin_batch_t<BLK_TEAM>(syn_kind, nets, blks, tiles, n, pad, max_mq, nt, s);
    else launch_thin_batch_t<1>(syn_kind, nets, blks, tiles, n, pad, max_mq, nt, s);
    if (syn_kind >= 2)
        launch_dep(k_blk_post_batch, dim3(std::max(1, std::min(152, 1216 / std::max(nets_n, 1))), nets_n),
                   256, 0, s, nets, blks, nt);
}

// The opt-in shared memory size is a property of the kernel on each device: set before every launch
// (a host-side table write), so that no process-wide flag is needed.
template <typename K>
static void allow_smem(K kern, size_t bytes)
{
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// The push grid: 128-synapse chunks over eight blocks, so that a neuron of a thousand synapses is
// one round of them.
constexpr int PUSH_SPLIT = 8;

template <int SYN, int W>
static void launch_dense_t(const NetDev &h, const BlkDev &b, const CUtensorMap &tp, const CUtensorMap &tc,
                           int nt, cudaStream_t s)
{
    allow_smem(k_blk_dense<SYN, W>, sizeof(DenseSmem<W>));
    launch_dep(k_blk_dense<SYN, W>, h.ntiles, dn_threads(W), sizeof(DenseSmem<W>), s, h, b, tp, tc, nt);
}
template <int SYN>
static void launch_dense_syn(const NetDev &h, const BlkDev &b, const CUtensorMap &tp, const CUtensorMap &tc,
                             int nt, cudaStream_t s)
{
    const dim3 pg((h.ntiles + PUSH_WORDS - 1) / PUSH_WORDS, PUSH_SPLIT);
    launch_dep(k_blk_push<SYN>, pg, PUSH_THREADS, 0, s, h, b, nt);
    if (h.ntiles <= DN_FEW) launch_dense_t<SYN, 8>(h, b, tp, tc, nt, s);
    else launch_dense_t<SYN, 4>(h, b, tp, tc, nt, s);
}
void launch_blk_dense(const NetDev &h, const BlkDev &b, const CUtensorMap &tp, const CUtensorMap &tc,
                      int nt, cudaStream_t s)
{
    if (h.syn_kind == 1) launch_dense_syn<1>(h, b, tp, tc, nt, s);
    else launch_dense_syn<0>(h, b, tp, tc, nt, s);
}

// dense: the indices of the nd networks that run dense blocks, max_tiles their most tiles.
template <int SYN, int W>
static void launch_dense_batch_t(const NetDev *nets, const BlkDev *blks, const CUtensorMap *maps,
                                 const int2 *tiles, int n, int nt, cudaStream_t s)
{
    allow_smem(k_blk_dense_batch<SYN, W>, sizeof(DenseSmem<W>));
    launch_dep(k_blk_dense_batch<SYN, W>, n, dn_threads(W), sizeof(DenseSmem<W>), s, nets, blks, maps, tiles, nt);
}
template <int SYN>
static void launch_dense_batch_syn(const NetDev *nets, const BlkDev *blks, const CUtensorMap *maps,
                                   const int2 *tiles, int n, const int *dense, int nd, int max_tiles, int nt,
                                   cudaStream_t s)
{
    const dim3 pg((max_tiles + PUSH_WORDS - 1) / PUSH_WORDS, PUSH_SPLIT, nd);
    launch_dep(k_blk_push_batch<SYN>, pg, PUSH_THREADS, 0, s, nets, blks, dense, nt);
    if (n <= DN_FEW) launch_dense_batch_t<SYN, 8>(nets, blks, maps, tiles, n, nt, s);
    else launch_dense_batch_t<SYN, 4>(nets, blks, maps, tiles, n, nt, s);
}
void launch_blk_dense_batch(int syn_kind, const NetDev *nets, const BlkDev *blks,
                            const CUtensorMap *maps, const int2 *tiles, int n, const int *dense, int nd,
                            int max_tiles, int nt, cudaStream_t s)
{
    if (syn_kind == 1) launch_dense_batch_syn<1>(nets, blks, maps, tiles, n, dense, nd, max_tiles, nt, s);
    else launch_dense_batch_syn<0>(nets, blks, maps, tiles, n, dense, nd, max_tiles, nt, s);
}

}  // namespace bg3
