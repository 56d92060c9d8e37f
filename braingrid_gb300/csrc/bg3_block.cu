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
#include <cuda.h>
#include <algorithm>
#include <utility>
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
    if ((threadIdx.x & 31) == 0 && i < n.Np) b.act[(t & (BLK_ACT_ROWS - 1)) * n.ntiles + (i >> 5)] = w;
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

// ---- thin networks: one warp per tile ---------------------------------------------------------
// Networks of at most BLK_THIN_QUADS row quads per destination.  The warp keeps its tile's psr in
// shared memory for the whole block, beside the decay factors (expanded once, so that a step
// needs no class decoding) and the arrival masks (bit j of a slot's byte: a spike arrives at the
// block's step j).  Lane = destination, so no step needs a barrier: the neuron's state stays in
// registers, its summation point is the sum the lane has just made.  What bounds it: the issue
// slots of the neuron updates (noise draw, Izhikevich arithmetic), about 250 instructions a step
// against 3 per synapse; the loads are hidden by the other warps of the SM.
constexpr int BLK_THIN_QUADS = 16;
constexpr int BLK_THIN_WARPS = 8;
__host__ __device__ constexpr size_t blk_thin_smem(int Mq)
{
    return (size_t)Mq * 32 * (16 + 16 + 4) + BLK_MAX_STEPS * 32 * 4;
}

struct ThinSmem {
    float4 *psr, *dec;  // [Mq][32]
    uint32_t *msk;      // [Mq][32], one byte per row
    float *noise;       // [BLK_MAX_STEPS][32]
};

// A lane's arrivals in the block, made ready before the steps run so that their chains of loads
// (the source's mask, the event slot, the exp tables) overlap across the warp's lanes: two of
// them as (row, step, psr increment) in registers.  Any more, two spikes at one synapse, and STDP
// arrivals whose weight the learning walk could change keep a mask in shared memory and run at
// their step (thin_late).
struct ThinEvents {
    int key0, key1;             // row | step << 8, -1: none
    float inc0, inc1;
    unsigned long long late;    // rows with a mask in shared memory
    uint32_t steps;             // bit j: something arrives at step j
};

// Whether an STDP arrival's learning walk may change W: with the host build's arithmetic the walk
// only applies the clamps (stdp_pre), so a weight inside its bounds stays as it is.
__device__ __forceinline__ bool stdp_clamps(const StdpConst &c, float W)
{
    return !(fabsf(W) <= fabsf(c.Wex)) || __float_as_uint(W) == 0x80000000u ||
           (c.Wex < 0.0f && W > 0.0f) || (c.Wex > 0.0f && W < 0.0f) || !(fabsf(c.Apos) < 1e30f);
}

template <int SYN>
__device__ __forceinline__ void thin_event(const NetDev &n, const BlkDev &b, const ThinSmem &s, int r,
                                           int d, int nt, unsigned long long t, ThinEvents &e)
{
    const int lane = threadIdx.x & 31;
    const uint32_t p = (uint32_t)slot_pos(r, d, n.Mq);
    const int src = n.src[p];
    const int D = n.ltab[n.lcls[p]];
    const uint32_t m = (uint32_t)rotr64(b.hist[src], (unsigned)(t - (unsigned long long)D)) &
                       ((1u << nt) - 1u);
    if (!m) return;
    e.steps |= m;
    bool late = (m & (m - 1u)) != 0u || e.key1 >= 0;
    const int j = __ffs((int)m) - 1;
    const unsigned long long tj = t + (unsigned)j;
    if (!late && SYN >= 2) {
        // a walk that finds the ring full sets an error bit: at its step where the ring may fill
        // within the block
        const int co = n.spikeCount[d] + n.spikeCountOffset[d];
        late = stdp_clamps(n.stdp[n.stype[p]], n.ev[p].W);
        if (hist_at(n, d, co, nt - n.max_spikes) != BG3_ULONG_MAX) {
            if (hist_at(n, d, co, -n.max_spikes) != BG3_ULONG_MAX) set_err(n, ERR_STDP_RING);
            else late = true;
        }
    }
    if (late) {
        uint8_t *mk = reinterpret_cast<uint8_t *>(&s.msk[(r >> 2) * 32 + lane]) + (r & 3);
        *mk = (uint8_t)m;
        e.late |= 1ull << r;
        return;
    }
    float inc;
    if (!arrival<(SYN == 3 ? 1 : SYN == 2 ? 0 : SYN)>(n, p, d, src, (uint32_t)tj - (uint32_t)D, tj, inc))
        return;
    const int key = r | (j << 8);
    if (e.key0 < 0) {
        e.key0 = key;
        e.inc0 = inc;
    } else {
        e.key1 = key;
        e.inc1 = inc;
    }
}

// The lane's remaining arrivals of step t + j.
template <int SYN>
__device__ __noinline__ void thin_late(const NetDev &n, const ThinSmem &s, int d,
                                       unsigned long long rows, int j, unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    while (rows) {
        const int r = __ffsll((long long)rows) - 1;
        rows &= rows - 1ull;
        if (!((s.msk[(r >> 2) * 32 + lane] >> ((r & 3) * 8 + j)) & 1u)) continue;
        const uint32_t p = (uint32_t)slot_pos(r, d, n.Mq);
        const int D = n.ltab[n.lcls[p]];
        float inc;
        if (arrival<SYN>(n, p, d, n.src[p], (uint32_t)(t + (unsigned)j) - (uint32_t)D,
                         t + (unsigned)j, inc)) {
            float *ps = reinterpret_cast<float *>(&s.psr[(r >> 2) * 32 + lane]) + (r & 3);
            *ps = *ps + inc;
        }
    }
}

template <int SYN>
__device__ __forceinline__ void blk_thin_tile(const NetDev &n, const BlkDev &b, const int tile,
                                              const int nt, uint8_t *smem)
{
    const int lane = threadIdx.x & 31;
    const int d = tile * 32 + lane;
    const bool valid = d < n.N;
    ThinSmem s;
    s.psr = reinterpret_cast<float4 *>(smem);
    s.dec = s.psr + n.Mq * 32;
    s.msk = reinterpret_cast<uint32_t *>(s.dec + n.Mq * 32);
    s.noise = reinterpret_cast<float *>(s.msk + n.Mq * 32);
    const int cnt = valid ? (int)n.count[d] : 0;
    const int nq = (__reduce_max_sync(0xffffffffu, cnt) + 3) >> 2;
    const size_t base = (size_t)tile * n.Mq * 32 + lane;  // the lane's first row quad
    const uint16_t *C = reinterpret_cast<const uint16_t *>(n.dcls) + base;
    for (int q = 0; q < nq; q++) {
        const uint32_t c = C[(size_t)q * 32];
        s.dec[q * 32 + lane] = make_float4(n.dtab[c & 15u], n.dtab[(c >> 4) & 15u],
                                           n.dtab[(c >> 8) & 15u], n.dtab[(c >> 12) & 15u]);
    }
    // STDP kinds follow a post-spike pass, which is launched once the block before has finished and
    // writes nothing but weights: everything else is final, and the wait can come later
    if (SYN < 2) {
        pdl_wait();
        pdl_trigger();
    }
    const unsigned long long t = *n.step;
    NeuronIn x;
    float sp = 0.0f;
    unsigned long long hist = 0ull;
    if (valid) {
        neuron_load(n, d, x);
        sp = n.sp[d];
        hist = b.hist[d];
    }
    // psr into shared memory; the slots whose source has a spike in this block's window
    float4 *P = reinterpret_cast<float4 *>(n.psr) + base;
    const int4 *S = reinterpret_cast<const int4 *>(n.src) + base;
    const uint32_t *act = b.act + (t & (BLK_ACT_ROWS - 1)) * n.ntiles;
    unsigned long long rows = 0ull;
    for (int q0 = 0; q0 < nq; q0 += 4) {
        float4 v[4];
        int4 sr[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (q0 + k < nq) {
                v[k] = P[(size_t)(q0 + k) * 32];
                sr[k] = S[(size_t)(q0 + k) * 32];
            }
        uint32_t hit = 0u;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (q0 + k < nq) {
                s.psr[(q0 + k) * 32 + lane] = v[k];
                const int left = cnt - 4 * (q0 + k);  // in-use rows from this quad on
                if (left > 0) hit |= ((act[sr[k].x >> 5] >> (sr[k].x & 31)) & 1u) << (4 * k);
                if (left > 1) hit |= ((act[sr[k].y >> 5] >> (sr[k].y & 31)) & 1u) << (4 * k + 1);
                if (left > 2) hit |= ((act[sr[k].z >> 5] >> (sr[k].z & 31)) & 1u) << (4 * k + 2);
                if (left > 3) hit |= ((act[sr[k].w >> 5] >> (sr[k].w & 31)) & 1u) << (4 * k + 3);
            }
        rows |= (unsigned long long)hit << (4 * q0);
    }
    // the steps' noise draws depend on nothing but the step: four at a time, so that one draw's
    // latency hides another's (inside the step loop each would wait alone)
#pragma unroll 4
    for (int j = 0; j < nt; j++)
        s.noise[j * 32 + lane] = normal_device(n.noise_seed, t + (unsigned)j, d);
    if (SYN >= 2) {
        pdl_wait();
        pdl_trigger();
    }
    ThinEvents e = {-1, -1, 0.0f, 0.0f, 0ull, 0u};
    while (rows) {
        const int r = __ffsll((long long)rows) - 1;
        rows &= rows - 1ull;
        thin_event<SYN>(n, b, s, r, d, nt, t, e);
    }
    const uint32_t any = __reduce_or_sync(0xffffffffu, e.steps);
    const int mode = izh_mode(n, d);
    uint32_t fired = 0u;
#pragma unroll 1
    for (int j = 0; j < nt; j++) {
        const unsigned long long tj = t + (unsigned)j;
        if (valid) {
            const int br = neuron_branch(x);
            const float in = input_update(n, d, x, tj, sp);
            if (neuron_update(n, d, x, br, in, s.noise[j * 32 + lane], tj, mode)) fired |= 1u << j;
        }
        if ((any >> j) & 1u) {
            if (e.key0 >> 8 == j) {
                float *ps = reinterpret_cast<float *>(&s.psr[((e.key0 >> 2) & 63) * 32 + lane]) + (e.key0 & 3);
                *ps = *ps + e.inc0;
            }
            if (e.key1 >> 8 == j) {
                float *ps = reinterpret_cast<float *>(&s.psr[((e.key1 >> 2) & 63) * 32 + lane]) + (e.key1 & 3);
                *ps = *ps + e.inc1;
            }
            if (e.late && ((e.steps >> j) & 1u)) thin_late<SYN>(n, s, d, e.late, j, t);
            __syncwarp();
        }
        float acc = 0.0f;
        for (int q = 0; q < nq; q++) {
            float4 v = s.psr[q * 32 + lane];
            const float4 c = s.dec[q * 32 + lane];
            v.x = v.x * c.x;
            v.y = v.y * c.y;
            v.z = v.z * c.z;
            v.w = v.w * c.w;
            s.psr[q * 32 + lane] = v;
            acc = acc + v.x;
            acc = acc + v.y;
            acc = acc + v.z;
            acc = acc + v.w;
        }
        sp = acc;
    }
    for (int q = 0; q < nq; q++) gst(&P[(size_t)q * 32], s.psr[q * 32 + lane]);
    // the neuron's state, its spikes, and the bitmap word for the block after this one
    const unsigned long long t1 = t + (unsigned)nt;
    if (valid) {
        gst(&n.sp[d], sp);
        gst(&n.refr[d], x.refr);
        gst(&n.Vm[d], x.Vm);
        if (n.neuron_kind == 1) gst(&n.u_izh[d], x.u);
        if (n.input_kind == 2 && x.pmask) {
            gst(&n.pois_nisi[d], x.nisi);
            gst(&n.in_queue[d], x.q);
            gst(&n.in_psr[d], x.ipsr);
        }
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
        if (atomicAdd(n.sweep_done, 1u) == (unsigned)n.ntiles - 1u) {
            // the network's last tile: every tile has read the step
            *n.sweep_done = 0u;
            *n.step = t1;
            *n.dstep = t1;
            n.ring_n[t1 & (BG3_RING - 1)] = 0;
            if (t1 >= 0xffffff00ull) set_err(n, ERR_STEP_RANGE);
        }
    }
}

template <int SYN>
__global__ void __launch_bounds__(32 * BLK_THIN_WARPS) k_blk_thin(const __grid_constant__ NetDev n,
                                                                  const __grid_constant__ BlkDev b,
                                                                  int nt)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int warp = (int)(threadIdx.x >> 5);
    const int tile = blockIdx.x * (int)(blockDim.x >> 5) + warp;
    if (tile < n.ntiles)
        blk_thin_tile<SYN>(n, b, tile, nt, smem_raw + warp * blk_thin_smem(n.Mq));
}

// Batched form: tiles[i] = (network, tile), -1 tiles idle; a block's entries belong to one
// network, whose descriptor the block copies into shared memory first.  wsmem: bytes per warp
// (the batch's widest thin network).
template <int SYN>
__global__ void __launch_bounds__(32 * BLK_THIN_WARPS) k_blk_thin_batch(const NetDev *nets,
                                                                        const BlkDev *blks,
                                                                        const int2 *tiles, int count,
                                                                        int wsmem, int nt)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(16) NetDev s_net;
    const int warp = (int)(threadIdx.x >> 5);
    const int first = blockIdx.x * (int)(blockDim.x >> 5);
    const int2 tr = first + warp < count ? tiles[first + warp] : make_int2(0, -1);
    const int k = tiles[first].x;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(nets + k);
    uint4 *d4 = reinterpret_cast<uint4 *>(&s_net);
    for (int i = threadIdx.x; i < (int)(sizeof(NetDev) / 16); i += blockDim.x) d4[i] = s4[i];
    const BlkDev b = blks[k];
    __syncthreads();
    if (tr.y >= 0) blk_thin_tile<SYN>(s_net, b, tr.y, nt, smem_raw + warp * wsmem);
}

// ---- STDP: learning after a block's post spikes -----------------------------------------------
// The fPost branch (AllSTDPSynapses.cpp:368-418) of every neuron that fired in the block just
// run, after the block instead of inside its steps.  The order of the weight changes is kept:
// where an arrival at the same synapse follows a post spike within the block, its spike was
// already under way (the source's newest history entry is later than t - delay), and the walk of
// such a post spike learns nothing; so all of a block's arrivals come before the post spikes that
// learn.  A walk sees the histories as of its step: entries the block added after it are skipped.
__device__ __forceinline__ int count_at(const NetDev &n, int i, unsigned long long t)
{
    int co = n.spikeCount[i] + n.spikeCountOffset[i];
    for (int f = 0; f < BLK_MAX_STEPS; f++) {
        const unsigned long long h = hist_at(n, i, co, -1);
        if (h == BG3_ULONG_MAX || h <= t) break;
        co = co > 0 ? co - 1 : n.max_spikes - 1;
    }
    return co;
}

// One warp per neuron that fired, one lane per synapse.
__device__ __forceinline__ void blk_post(const NetDev &n, const BlkDev &b, int gw, int nw, int nt)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long t = *n.step - (unsigned)nt;  // the block's first step
    const int slot = (int)(t & (BG3_RING - 1));
    const int m = min(n.ring_n[slot], n.N);
    const int32_t *ids = n.ring + (size_t)slot * n.N;
    for (int e = gw; e < m; e += nw) {
        const int d = ids[e];
        const int cnt = (int)n.count[d];
        const uint32_t fired = (uint32_t)rotr64(b.hist[d], (unsigned)t) & ((1u << nt) - 1u);
        for (int k = lane; k < cnt; k += 32) {
            const size_t p = slot_pos(k, d, n.Mq);
            const StdpConst &c = n.stdp[n.stype[p]];
            const int pre = n.src[p];
            const int delay = n.ltab[n.lcls[p]];
            float W = n.ev[p].W;
            for (uint32_t f = fired; f; f &= f - 1u) {
                const unsigned long long tj = t + (unsigned)(__ffs((int)f) - 1);
                PostPrep q;
                stdp_post_prep(n, c, pre, d, count_at(n, pre, tj), count_at(n, d, tj), delay, tj, q);
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
    blk_post(n, b, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5, nt);
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
             (gridDim.x * blockDim.x) >> 5, nt);
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

void launch_blk_masks(const NetDev &h, const BlkDev &b, cudaStream_t s)
{
    cudaMemsetAsync(b.hist, 0, (size_t)h.Np * sizeof(*b.hist), s);
    k_blk_scatter<<<dim3(std::min((h.N + 255) / 256, 16), BG3_RING), 256, 0, s>>>(h, b);
    k_blk_act<<<(h.Np + 255) / 256, 256, 0, s>>>(h, b);
}

void launch_blk_ring(const NetDev &h, const BlkDev &b, cudaStream_t s)
{
    cudaMemsetAsync(h.ring_n, 0, BG3_RING * sizeof(*h.ring_n), s);
    k_blk_ring<<<(h.N + 255) / 256, 256, 0, s>>>(h, b);
}

// At most 44 KB of shared memory per block beside a batch's descriptor (48 KB is what a launch may
// use without opting in), so that several blocks share an SM.
static int thin_warps_for(int Mq) { return std::max(1, (int)(45056 / blk_thin_smem(Mq))); }

// Few tiles: one warp per block, so that they spread over the SMs.
void launch_blk_thin(const NetDev &h, const BlkDev &b, int nt, cudaStream_t s)
{
    const int w = std::max(1, std::min({BLK_THIN_WARPS, thin_warps_for(h.Mq), h.ntiles / 152}));
    const int blocks = (h.ntiles + w - 1) / w;
    const size_t sm = w * blk_thin_smem(h.Mq);
    switch (h.syn_kind) {
    case 1: launch_dep(k_blk_thin<1>, blocks, 32 * w, sm, s, h, b, nt); break;
    case 2: launch_dep(k_blk_thin<2>, blocks, 32 * w, sm, s, h, b, nt); break;
    case 3: launch_dep(k_blk_thin<3>, blocks, 32 * w, sm, s, h, b, nt); break;
    default: launch_dep(k_blk_thin<0>, blocks, 32 * w, sm, s, h, b, nt); break;
    }
    if (h.syn_kind >= 2) launch_dep(k_blk_post, 152, 256, 0, s, h, b, nt);
}

// tiles: n thin entries, each network's run padded to a multiple of `pad` entries; blocks of a
// divisor of pad warps, so that a block serves one network.
void launch_blk_thin_batch(int syn_kind, const NetDev *nets, const BlkDev *blks, int nets_n,
                           const int2 *tiles, int n, int pad, int max_mq, int nt, cudaStream_t s)
{
    int w = std::min({pad, BLK_THIN_WARPS, thin_warps_for(max_mq)});
    while (pad % w) w--;
    const int blocks = (n + w - 1) / w, ws = (int)blk_thin_smem(max_mq);
    const size_t sm = (size_t)w * ws;
    switch (syn_kind) {
    case 1: launch_dep(k_blk_thin_batch<1>, blocks, 32 * w, sm, s, nets, blks, tiles, n, ws, nt); break;
    case 2: launch_dep(k_blk_thin_batch<2>, blocks, 32 * w, sm, s, nets, blks, tiles, n, ws, nt); break;
    case 3: launch_dep(k_blk_thin_batch<3>, blocks, 32 * w, sm, s, nets, blks, tiles, n, ws, nt); break;
    default: launch_dep(k_blk_thin_batch<0>, blocks, 32 * w, sm, s, nets, blks, tiles, n, ws, nt); break;
    }
    if (syn_kind >= 2)
        launch_dep(k_blk_post_batch, dim3(std::max(1, std::min(152, 1216 / std::max(nets_n, 1))), nets_n),
                   256, 0, s, nets, blks, nt);
}

}  // namespace bg3
