// The fused simulation step for sm_100a.
//
// One launch advances every network in the engine by one cycle. Its blocks
// first deliver the spikes of cycles t-1 .. t-D into the input buffer of cycle
// t+1, then run the LIF_brian update of cycle t in chunks of neurons taken from
// a per-cycle counter (reads the synaptic input summed during the previous
// launch, writes the new state, appends fired ids to this cycle's ring slot with
// one atomic per block pass and stores each warp's ballot as a fired-bitmap
// word). Blocks that finish delivering early take most of the update, so the
// bandwidth-bound update fills the tail of the delivery.
//
// The two halves touch disjoint data (the input accumulators are double
// buffered by cycle parity, the fire ring has at least D+2 slots), so they need no
// barrier between them; the kernel boundary orders consecutive cycles.
// The cycle counter lives on the device and is advanced by the last block to
// finish, so the same launch can be replayed from a CUDA graph with no host
// involvement.
//
// Reference semantics (BSim, paths relative to its root):
//   neuron update  LIFENeuron::update  src/neuron/lif/LIFENeuron.cpp:114-160
//                  (GPU: find_life_neuron + update_life_neuron, src/neuron/lif/lif.cu:9-162)
//   delivery       update_dense_static_hit, src/synapse/static/static.cu:59-96:
//                  at cycle t, ring slot t-d feeds the synapses of delay d
//   ring advance   update_time, src/gpu_utils/runtime.cu:81-92
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "engine.h"

namespace bsim {

// Synapse rows are read once per spike: stream them past L1 and mark them
// evict-first in L2 (ld.global.cs) so the accumulators stay L2-resident.
static __device__ __forceinline__ uint4 ld_stream16(const uint4 *p) { return __ldcs(p); }
static __device__ __forceinline__ uint2 ld_stream8(const uint2 *p) { return __ldcs(p); }

static __device__ __forceinline__ void red_add_u64(unsigned long long *p, unsigned long long v)
{
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Device error flag: the first error code raised stays (BSIM_DEVERR_*). Every
// later launch on the same flag returns at once, so the host reads the code
// (BSIM_ERR_DEVICE) and no further cycle runs on inconsistent data.
static __device__ __forceinline__ void raise_error(const StepArgs &a, int code) { atomicCAS(a.err, 0, code); }

// ---------------------------------------------------------------------------
// Input-drive neurons (drive.h): Constant_spikes per update_constant_neuron
// (src/neuron/constant/constant.cu:18-22), Poisson_spikes per update_poisson_neuron
// and reset_poisson_neuron (src/neuron/poisson/poisson.cu:29-31, 9-15). Both
// ignore their synaptic input, as their recv() does.
// ---------------------------------------------------------------------------
// The gap a Poisson neuron draws when it fires at cycle fc.
static __device__ __forceinline__ int poisson_gap(const StepArgs &a, const ClassParams *c, int64_t j, const float4 &st, int fc)
{
    return poisson_draw(poisson_key(a.input_seed, j - __ldg(&c->id_base), fc), st.x, a.vtmp[j], a.ptab);
}

// gap(fc): what poisson_gap gives for a spike at cycle fc
template <typename Gap>
static __device__ __forceinline__ void drive_update(int kind, int t, float4 &st, bool &fired, Gap gap)
{
    if (kind == BSIM_NEURON_CONSTANT) {
        const int cnt = __float_as_int(st.w);
        if (t < __float_as_int(st.z) && __fmul_rn((float)(t - __float_as_int(st.y)), st.x) > (float)cnt) {
            fired = true;
            st.w = __int_as_float(cnt + 1);
        }
    } else {
        const int fc = __float_as_int(st.y);
        if (t == fc && t <= __float_as_int(st.z)) {
            fired = true;
            const long long nxt = (long long)fc + 1 + gap(fc) + __float_as_int(st.w);
            st.y = __int_as_float(nxt > 2147483647LL ? 2147483647 : (int)nxt);
        }
    }
}

// ---------------------------------------------------------------------------
// Update of one neuron for cycle t with the synaptic input of the cycle.
// LIF_brian arithmetic follows LIFENeuron::update term by term with every product
// and sum rounded on its own (no FMA contraction), as the reference's x86 build
// evaluates it:  v = ((Cm*v + v_tmp) + i_E*C_E) + i_I*C_I.
// ---------------------------------------------------------------------------
struct LifConst {
    float Cm, CE, CI, C_E, C_I, v_thresh, v_reset;
    int refrac_time;
};
static __device__ __forceinline__ LifConst lif_const(const ClassParams *c)
{
    return LifConst{__ldg(&c->Cm),  __ldg(&c->CE),       __ldg(&c->CI),      __ldg(&c->C_E),
                    __ldg(&c->C_I), __ldg(&c->v_thresh), __ldg(&c->v_reset), __ldg(&c->refrac_time)};
}

static __device__ __forceinline__ void lif_update(const LifConst &k, float vtmp, float inE, float inI, float4 &st,
                                                  bool &fired)
{
    int refrac = __float_as_int(st.w);
    if (refrac > 0) {
        refrac -= 1;  // input of this cycle is dropped
    } else {
        float v = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(k.Cm, st.x), vtmp), __fmul_rn(st.y, k.C_E)),
                            __fmul_rn(st.z, k.C_I));
        float iE = __fmul_rn(k.CE, st.y);
        float iI = __fmul_rn(k.CI, st.z);
        if (v >= k.v_thresh) {
            fired = true;
            refrac = k.refrac_time - 1;
            v = k.v_reset;
        } else {
            iE = __fadd_rn(iE, inE);
            iI = __fadd_rn(iI, inI);
        }
        st.x = v;
        st.y = iE;
        st.z = iI;
    }
    st.w = __int_as_float(refrac);
}

static __device__ __forceinline__ void neuron_update(const StepArgs &a, const ClassParams *c, int64_t j, int t,
                                                     const float *vtmp, float inE, float inI, float4 &st, bool &fired)
{
    const int kind = __ldg(&c->kind);
    if (kind == BSIM_NEURON_LIF) lif_update(lif_const(c), vtmp[j], inE, inI, st, fired);
    else  // input is dropped (recv returns 0)
        drive_update(kind, t, st, fired, [&](int fc) { return poisson_gap(a, c, j, st, fc); });
}

// The state trace row of cycle t (or -1) and the copy of one neuron into it.
struct TraceRow {
    long long k, first, count, steps;
};
static __device__ __forceinline__ TraceRow trace_row(const StepArgs &a, unsigned long long t)
{
    TraceRow r{-1, 0, 0, 0};
    if (a.trace) {
        const TraceCtl tc = *a.trace_ctl;
        const long long k = (long long)t - tc.t0;
        if (k >= 0 && k < tc.steps) r = TraceRow{k, tc.first, tc.count, tc.steps};
    }
    return r;
}
static __device__ __forceinline__ void trace_neuron(const StepArgs &a, const TraceRow &r, int64_t j, const float4 &st,
                                                    float inE, float inI)
{
    if (r.k < 0 || j < r.first || j >= r.first + r.count) return;
    const int64_t plane = r.steps * r.count;
    float *row = a.trace + r.k * r.count + (j - r.first);
    row[0] = st.x;
    row[plane] = st.y;
    row[2 * plane] = st.z;
    row[3 * plane] = inE;
    row[4 * plane] = inI;
}

// ---------------------------------------------------------------------------
// Phase A: update of all neurons, in chunks of one block pass.
// ---------------------------------------------------------------------------
// Fired ids are appended to the cycle's ring slot with one global atomic per
// block and pass: warps publish their ballot counts, warp 0 scans them and
// reserves the block's range (a single counter per cycle would otherwise take
// one same-address atomic per warp).
template <int ACC>
static __device__ __forceinline__ void lif_phase(const StepArgs &a, unsigned long long t, int p, int cur,
                                                 int *s_wcnt)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // the cycle's chunk counter: the upper half of the ticket word (reset by the last block)
    unsigned *chunk_ctr = a.ticket + 1;
    __shared__ long long s_chunk[2];  // this pass's chunk and the next one's (taken during the pass)
    int32_t *slot_ids = a.ring + (int64_t)cur * a.cap;
    uint32_t *bm = a.bitmap + (int64_t)cur * a.W;
    int32_t *hist = a.pop_hist ? a.pop_hist + (int64_t)(t % (unsigned long long)a.hist_len) * a.n_pops : nullptr;
    const float *vtmp = (a.drive_half > 0 && ((t / (unsigned long long)a.drive_half) & 1ull)) ? a.vtmp_alt : a.vtmp;
    const TraceRow tr = trace_row(a, t);
    int buf = 0;  // s_wcnt is double-buffered by pass, so a pass needs no closing barrier
    int cb = 0;
    if (threadIdx.x == 0) s_chunk[0] = (long long)atomicAdd(chunk_ctr, (unsigned)blockDim.x);
    __syncthreads();
    for (;;) {
        // one pass of blockDim.x neurons per chunk; the next chunk is taken while this one
        // runs (its slot is read only after this pass's two barriers, and this slot is
        // written again only in the next pass, after every thread has read it)
        const int64_t bbase = s_chunk[cb];
        if (bbase >= a.N) break;
        if (threadIdx.x == 0) s_chunk[cb ^ 1] = (long long)atomicAdd(chunk_ctr, (unsigned)blockDim.x);
        cb ^= 1;
        buf ^= 64;
        const int64_t base = bbase + (threadIdx.x & ~31);
        const int64_t j = base + lane;
        bool fired = false;
        int pop = -1;
        if (j < a.N) {
            float4 st = a.state[j];
            const ClassParams *c = a.ctab + a.cls[j];
            float inE, inI;
            if (ACC == BSIM_ACC_EXACT) {
                longlong2 *acc = reinterpret_cast<longlong2 *>(a.acc) + (int64_t)p * a.N + j;
                const longlong2 q = *acc;
                if (a.acc_clear) *acc = make_longlong2(0, 0);
                const float sd = __ldg(&c->scale_down);
                inE = __fmul_rn(__ll2float_rn(q.x), sd);
                inI = __fmul_rn(__ll2float_rn(q.y), sd);
            } else {
                float2 q = reinterpret_cast<const float2 *>(a.acc)[(int64_t)p * a.N + j];
                inE = q.x;
                inI = q.y;
            }
            neuron_update(a, c, j, (int)t, vtmp, inE, inI, st, fired);
            a.state[j] = st;
            trace_neuron(a, tr, j, st, inE, inI);
            if (hist) pop = __ldg(&c->pop);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, fired);
        if (lane == 0 && base < a.N) bm[base >> 5] = mask;
        if (lane == 0) s_wcnt[buf + warp] = __popc(mask);
        __syncthreads();
        if (warp == 0) {
            int c = lane < nwarps ? s_wcnt[buf + lane] : 0;
            const int own = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int nb = __shfl_up_sync(0xffffffffu, c, o);
                if (lane >= o) c += nb;
            }
            const int total = __shfl_sync(0xffffffffu, c, 31);
            int at = 0;
            if (lane == 0 && total) at = atomicAdd(&a.ring_cnt[cur], total);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (lane < nwarps) s_wcnt[buf + 32 + lane] = at + c - own;  // this warp's first position
        }
        __syncthreads();
        if (mask) {
            if (fired) {
                slot_ids[s_wcnt[buf + 32 + warp] + __popc(mask & ((1u << lane) - 1u))] = (int32_t)j;
                atomicAdd(&a.fire_count[j], 1);  // a reduction: nothing waits for the old count
            }
            if (hist) {
                // one atomic per (warp, population) with spikes
                const unsigned same = __match_any_sync(0xffffffffu, fired ? pop : -1);
                if (fired && lane == __ffs(same) - 1) atomicAdd(&hist[pop], __popc(same));
            }
        }
        // no barrier here: the next pass writes the other half of s_wcnt, and the pass
        // after it is ordered by the next pass's barriers
    }
}

// ---------------------------------------------------------------------------
// Phase B, push: one warp per (spike, delay) segment of the source-ordered
// rows; 16-byte streaming loads of two packed {target, weight} entries per
// lane; exact int64 red.add into the target's E or I accumulator.
// ---------------------------------------------------------------------------
static __device__ __forceinline__ void push_one(const StepArgs &a, unsigned long long *acc, uint32_t tgt,
                                                uint32_t wbits, float sc)
{
    if ((int64_t)tgt >= a.N) {  // a target outside the network: flag it, touch nothing
        raise_error(a, BSIM_DEVERR_TARGET);
        return;
    }
    const float w = __int_as_float(wbits);
    const long long q = __float2ll_rn(__fmul_rn(w, sc));
    red_add_u64(acc + 2 * (int64_t)tgt + (w >= 0.0f ? 0 : 1), (unsigned long long)q);
}

// (spike, delay) segments whose metadata one warp resolves at once
#ifndef PUSH_CHUNK
#define PUSH_CHUNK 8
#endif
#define PUSH_MAX_SPLIT 32   // pieces of one row at most, in cycles with few long rows
#define PUSH_PASS 256       // entries a warp takes at once
// resident blocks of STEP_MAX_THREADS threads the step kernel is compiled for
// (together they set its register budget: 65,536 / (2 x 512) = 64 per thread)
#ifndef STEP_MAX_THREADS
#define STEP_MAX_THREADS 512
#endif
#ifndef STEP_MIN_BLOCKS
#define STEP_MIN_BLOCKS 2
#endif
#define MAX_WARPS 16

struct PushSeg {
    long long incl;  // inclusive prefix of the chunk's pair counts
    int64_t p0;      // first entry of the segment's first 16-byte pair
    float sc;        // 2^qexp of the segment's network
};

// s_cum[d] = spikes of cycles t-1 .. t-d (the push work items of delays 1..d).
// Run by warp 0 before the LIF phase, so its loads overlap the neuron update;
// the caller's __syncthreads publishes it.
template <typename Count>  // Count: spikes of ring slot s
static __device__ __forceinline__ void delay_window_prefix(const StepArgs &a, unsigned long long t, long long *s_cum,
                                                           Count count)
{
    const int lane = threadIdx.x & 31;
    const int D = a.D, cur = (int)(t % (unsigned long long)a.R);
    long long run = 0;
    for (int d0 = 1; d0 <= D; d0 += 32) {
        const int d = d0 + lane;
        long long c = 0;
        if (d <= D && (long long)t - d >= 0) c = count(cur >= d ? cur - d : cur - d + a.R);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            long long nb = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c += nb;
        }
        if (d <= D) s_cum[d] = run + c;
        run += __shfl_sync(0xffffffffu, c, 31);
    }
    if (lane == 0) s_cum[0] = 0;
}

// Pieces that rows of a push cycle are cut into at most (S synapses in N rows of D segments).
int push_split_of(int64_t S, int64_t N, int32_t D)
{
    const double mean = N > 0 ? (double)S / ((double)N * (double)D) : 0.0;
    return (int)std::min((double)PUSH_MAX_SPLIT, std::max(1.0, std::floor(mean / PUSH_PASS + 0.5)));
}

// warp_lin of n_warps: this warp's number among those that deliver; s_seg: the warp's table.
static __device__ __forceinline__ unsigned long long push_phase(const StepArgs &a, unsigned long long t, int pw,
                                                                const long long *s_cum, PushSeg *seg,
                                                                long long warp_lin, long long n_warps)
{
    const int lane = threadIdx.x & 31;
    const int D = a.D;
    const long long total = s_cum[D];
    unsigned long long ev = 0;
    unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc) + 2 * (int64_t)pw * a.N;
    // Segments per warp chunk: PUSH_CHUNK when there are enough for every warp, fewer
    // (down to one) when a cycle has few spikes with long rows, so that more warps
    // share the rows. Chunks go to warps block-interleaved (chunk c to warp c / grid of
    // block c % grid), so a cycle with few chunks still spreads over every SM.
    int pc = PUSH_CHUNK;
    while (pc > 1 && total < (long long)pc * n_warps) pc >>= 1;
    // fewer segments than warps: each is cut into `split` pieces of whole pairs, where rows are longer than
    // one pass of a warp takes (push_split: cutting short ones only repeats the look-ups; us per cycle at 100
    // Hz, 1-step delays, uncut / cut: rows of 120 entries, 20 x 1,000 neurons 8.9 / 11.3, 100 x 1,000
    // 10.9 / 13.2; of 1,200, 25 x 10,000 20.7 / 16.5; of 5,700, 20 x 5,000 57.7 / 24.2)
    const int split = a.push_split > 1 && total > 0 && 2 * total <= n_warps ? min((int)n_warps / (int)total, a.push_split) : 1;
    const long long n_chunks = split > 1 ? total * split : (total + pc - 1) / pc;
    for (long long ch = warp_lin; ch < n_chunks; ch += n_warps) {
        // Lanes 0..PUSH_CHUNK-1 each resolve one (spike, delay) segment: its row
        // [r0, r1), split into an odd head entry, 16-byte pairs [p0, p0 + 2*np)
        // and an odd tail entry.
        int64_t r0 = 0, r1 = 0;
        float sc = 0.0f;
        const long long item = split > 1 ? (int)ch / split + lane : ch * pc + lane;  // (split: n_chunks <= n_warps)
        if (lane < pc && item < total) {
            int lo = 1, hi = D;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_cum[mid] > item) hi = mid;
                else lo = mid + 1;
            }
            const int d = lo;
            const int slot = (int)((t - d) % (unsigned long long)a.R);
            const int32_t s = __ldcg(&a.ring[(int64_t)slot * a.cap + (item - s_cum[d - 1])]);
            r0 = a.row_off[(int64_t)s * D + d - 1];
            r1 = a.row_off[(int64_t)s * D + d];
            if (r1 < r0) {  // row offsets not ascending: flag it, skip the row
                raise_error(a, BSIM_DEVERR_ROW);
                r1 = r0;
            }
            sc = __ldg(&a.ctab[a.cls[s]].scale_up);
            if (split > 1 && r1 > r0) {  // piece ch % split; inner cuts lie on 16-byte boundaries
                const int64_t len = r1 - r0, b = r0;
                const int k = (int)ch % split;
                const int64_t lo = (b + len * k / split + 1) & ~1ll, hi = (b + len * (k + 1) / split + 1) & ~1ll;
                if (k > 0) r0 = lo < r1 ? lo : r1;
                if (k + 1 < split) r1 = hi < r1 ? hi : r1;
                if (r0 > r1) r0 = r1;
            }
            ev += (unsigned long long)(r1 - r0);
        }
        const int64_t p0 = (r0 & 1) && r0 < r1 ? r0 + 1 : r0;  // first entry of the first pair
        const long long np = (r1 - p0) >> 1;
        const bool head = p0 != r0, tail = ((r1 - p0) & 1) != 0;
        // inclusive prefix of pair counts over the chunk's segments
        long long incl = np;
#pragma unroll
        for (int o = 1; o < PUSH_CHUNK; o <<= 1) {
            const long long nb = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += nb;
        }
        // the chunk's segment table, in this warp's slice of shared memory (seg)
        __syncwarp();
        if (lane < PUSH_CHUNK) {
            seg[lane].incl = incl;
            seg[lane].p0 = p0;
            seg[lane].sc = sc;
        }
        __syncwarp();
        const long long total_pairs = __shfl_sync(0xffffffffu, incl, PUSH_CHUNK - 1);
        // head / tail single entries: lane L handles segment L>>1, head if L even
        {
            const int k = lane >> 1;
            const bool want_head = (lane & 1) == 0;
            const bool hk = __shfl_sync(0xffffffffu, head, k & (PUSH_CHUNK - 1));
            const bool tk = __shfl_sync(0xffffffffu, tail, k & (PUSH_CHUNK - 1));
            const int64_t rk0 = __shfl_sync(0xffffffffu, r0, k & (PUSH_CHUNK - 1));
            const int64_t rk1 = __shfl_sync(0xffffffffu, r1, k & (PUSH_CHUNK - 1));
            const float sk = __shfl_sync(0xffffffffu, sc, k & (PUSH_CHUNK - 1));
            if (k < PUSH_CHUNK && ((want_head && hk) || (!want_head && tk))) {
                const uint2 x = ld_stream8(a.syn + (want_head ? rk0 : rk1 - 1));
                push_one(a, acc, x.x, x.y, sk);
            }
        }
        // the pairs of all segments as one flat range, four loads in flight per lane
        // each chunk walks its range from its own starting point (wrapping around), so that
        // chunks whose rows hit the same targets (a population's sources in a dense
        // projection) do not add into the same addresses in lockstep
        const long long rot = total_pairs > 0 ? (long long)((unsigned long long)(ch * 40503ll) % total_pairs) : 0;
        for (long long pb = 0; pb < total_pairs; pb += 4 * 32) {
            uint4 x[4];
            float xs[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const long long q = pb + u * 32 + lane;
                ok[u] = q < total_pairs;
                const long long p = q + rot < total_pairs ? q + rot : q + rot - total_pairs;
                int k = 0;
                while (k < PUSH_CHUNK - 1 && p >= seg[k].incl) k++;
                const long long excl = k == 0 ? 0 : seg[k - 1].incl;
                xs[u] = seg[k].sc;
                if (ok[u]) x[u] = ld_stream16(reinterpret_cast<const uint4 *>(a.syn + seg[k].p0) + (p - excl));
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (ok[u]) {
                    push_one(a, acc, x[u].x, x[u].y, xs[u]);
                    push_one(a, acc, x[u].z, x[u].w, xs[u]);
                }
            }
        }
    }
    return ev;
}

// ---------------------------------------------------------------------------
// Phase B, pull: one warp per target over its target-ordered row (creation
// order), testing each source's bit in the fired bitmap of cycle t - delay.
// EXACT: int64 fixed-point partial sums, warp-reduced (order-free).
// ORDERED: the active weights of each 32-entry chunk are added one by one in
// row order with warp shuffles, so the fp32 sum is formed in exactly the order
// of the reference's loop over pSynapses.
// ---------------------------------------------------------------------------
// The scan waits for its loads, so a warp has those of PULL_LOADS chunks in flight (40 x 5,000
// neurons, 1e8 synapses: 770 -> 465 us per cycle EXACT, 720 -> 475 ORDERED).
// ---------------------------------------------------------------------------
#ifndef PULL_LOADS
#define PULL_LOADS 4
#endif
#define PULL_NO_DELAY (1 << 20)  // of a lane past the row's end

// One target's input: the active weights of consecutive entries, a chunk of 32 at a time.
template <int ACC>
struct PullSum {
    long long qE = 0, qI = 0;    // EXACT: this lane's part
    float fE = 0.0f, fI = 0.0f;  // ORDERED: the sums, in every lane

    __device__ __forceinline__ int add(bool act, float w, float sc)
    {
        unsigned m = __ballot_sync(0xffffffffu, act);
        const int n = __popc(m);
        if (ACC == BSIM_ACC_EXACT) {
            if (act) {
                const long long q = __float2ll_rn(__fmul_rn(w, sc));
                if (w >= 0.0f) qE += q;
                else qI += q;
            }
        } else {
            while (m) {
                const int b = __ffs(m) - 1;
                const float wb = __shfl_sync(0xffffffffu, w, b);
                if (wb >= 0.0f) fE = __fadd_rn(fE, wb);
                else fI = __fadd_rn(fI, wb);
                m &= m - 1;
            }
        }
        return n;
    }
    // Target i's input, by lane 0.
    __device__ __forceinline__ void store(void *acc, int64_t i)
    {
        if (ACC == BSIM_ACC_EXACT) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                qE += __shfl_xor_sync(0xffffffffu, qE, o);
                qI += __shfl_xor_sync(0xffffffffu, qI, o);
            }
        }
        if ((threadIdx.x & 31) != 0) return;
        if (ACC == BSIM_ACC_EXACT) reinterpret_cast<longlong2 *>(acc)[i] = make_longlong2(qE, qI);
        else reinterpret_cast<float2 *>(acc)[i] = make_float2(fE, fI);
    }
};

// Whether source `src` fired `d` cycles before the cycle in ring slot `slot`; d_max: later cycles only.
static __device__ __forceinline__ unsigned pull_fired(const uint32_t *bitmap, int W, int R, int slot, int d_max,
                                                      uint32_t src, int d)
{
    if (d > d_max) return 0u;
    const int s = slot >= d ? slot - d : slot - d + R;
    return (bitmap[(int64_t)s * W + (src >> 5)] >> (src & 31)) & 1u;
}

// The entries [c0, c1) of the pull rows, one per lane and chunk: test(source, delay) of several
// chunks, then add(what test returned, weight, chunk's first entry) chunk by chunk.
template <typename Test, typename Add>
static __device__ __forceinline__ void pull_entries(const StepArgs &a, int64_t c0, int64_t c1, Test test, Add add)
{
    const int lane = threadIdx.x & 31;
    for (int64_t k0 = c0; k0 < c1; k0 += 32 * PULL_LOADS) {
        uint32_t src[PULL_LOADS];
        int d[PULL_LOADS];
        float w[PULL_LOADS];
        unsigned r[PULL_LOADS];
#pragma unroll
        for (int u = 0; u < PULL_LOADS; u++) {
            const int64_t e = k0 + u * 32 + lane;
            src[u] = 0;
            d[u] = PULL_NO_DELAY;
            w[u] = 0.0f;
            if (e < c1) {
                src[u] = __ldcs(a.csc_src + e);
                d[u] = (int)__ldcs(a.csc_d + e) + 1;
                w[u] = __ldcs(a.csc_w + e);
            }
        }
#pragma unroll
        for (int u = 0; u < PULL_LOADS; u++) r[u] = test(src[u], d[u]);
#pragma unroll
        for (int u = 0; u < PULL_LOADS; u++)
            if (k0 + u * 32 < c1) add(r[u], w[u], k0 + u * 32);
    }
}

template <int ACC>
static __device__ __forceinline__ unsigned long long pull_phase(const StepArgs &a, unsigned long long t, int pw)
{
    const long long warp_lin = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int W = (int)a.W, R = a.R, cur = (int)(t % (unsigned long long)R);
    const int d_max = (long long)t < a.D ? (int)t : a.D;  // cycles before the first fired nothing
    const int64_t plane = (int64_t)pw * a.N;
    unsigned long long ev = 0;
    for (long long j = warp_lin; j < a.N; j += n_warps) {
        const float sc = (ACC == BSIM_ACC_EXACT) ? __ldg(&a.ctab[a.cls[j]].scale_up) : 0.0f;
        PullSum<ACC> x;
        pull_entries(a, a.col_off[j], a.col_off[j + 1],
                     [&](uint32_t src, int d) { return pull_fired(a.bitmap, W, R, cur, d_max, src, d); },
                     [&](unsigned act, float w, int64_t) { ev += x.add(act != 0, w, sc); });
        x.store(a.acc, plane + j);
    }
    return (threadIdx.x & 31) == 0 ? ev : 0ull;
}

// ---------------------------------------------------------------------------
// Phase B, tiled: the exact E and I sums of a tile of target neurons are formed
// in shared memory, so no per-event global atomic is issued. Tiles follow
// population boundaries and hold up to a few thousand targets (16 bytes of
// counters each), so each source's row into a tile stays a long segment. The first
// block to finish a piece of a tile stores its sums into the accumulator plane; the
// others add theirs after that store.
//
// Every block works on one contiguous share of the cycle: the tiles in a row, each cut
// into items (a run's sources and a few delays: populations fire at different rates and
// in bursts) with the warp clocks spent on them in the previous cycle, are cut into
// shares of equal cost, so a block touches one or two tiles, flushes as often, and the
// blocks end together. Each block finds its share by itself from the items' costs. The
// units of a share are taken in chunks from a counter, so a block that is done can help
// where the activity changed since the previous cycle and much is left. Measured against
// parts of a tile taken from a queue, two per resident block, with the additions below
// through generic addresses (us per cycle): 100 x 10,000 201 -> 164, 25 x 10,000 92 -> 84,
// 50 x 10,000 with 20-step delays 128 -> 102, 50 x 5,000 with 50-step delays 171 -> 128,
// 16 uneven networks 312 -> 309. A cost of a tile by its pairs alone left blocks idle (a
// tile's runs differ, cold tiles scan fast: 206 on the first network); item clocks that
// include the flush made shares chase their own splits (178).
//
// The tile's sources form runs of consecutive ids; its synapses are grouped by
// (run, delay, source). A work unit is (run, delay d, 32-source chunk): one lane
// reads the chunk's word of the fired bitmap of cycle t-d. Each fired (source,
// delay) names one segment of 8-byte entries, padded to an even length from an
// even start. A warp lists up to 32 segments at a time, one per lane, and streams
// them as one flat range of 16-byte entry pairs, 64 at a time: two per lane, which
// finds their segments from the warp's start marks (a warp-wide OR and a population
// count per 32 pairs), fetches them with cp.async into its own places of a slot of
// the warp's ring in shared memory, and adds a whole slot's four entries per lane one
// or two slots later. A listing continues the slot that the last one left open, so
// the ring stays full across listings without holding registers.
//
// What bounds it: the entry stream (8 bytes per event) and the issue slots of the
// additions. An entry holds the byte offset of its counter and its weight already
// scaled to fixed point, so an addition is a conversion, two shared atomics and a
// carry; a padding entry adds zero instead of branching. Measured against listing
// two segments per lane at a time and four register loads per lane with the sign,
// scale and padding worked out per entry (us per cycle): 50 x 5,000 with 50-step
// delays 296 -> 171, 16 uneven networks 455 -> 312, 50 x 10,000 with 20-step delays
// 168 -> 128, 25 x 10,000 106 -> 92, 100 x 10,000 210 -> 201; slots of 64 pairs carried
// across listings instead of 32: 25 x 10,000 82 -> 79, 100 x 10,000 164 -> 160 (more slots
// in flight are level, and 1 is 30 % slower).
//
// Exact int64 sums with 32-bit shared atomics: the low word of the fixed-point
// value is added with an atomic that returns the old word, and the high word
// plus the carry out of the low word with a second one. After all additions the
// (high, low) pair is the exact two's-complement sum (additions commute, and
// every carry is counted once); the fixed-point exponent keeps every sum below
// 2^61, so the high word cannot overflow.
// ---------------------------------------------------------------------------
// costs in warp clocks: scanning one work unit (at least), one part of a tile, flushing one target
#ifndef TILE_UNIT_CLOCKS
#define TILE_UNIT_CLOCKS 16
#endif
#ifndef TILE_PART_CLOCKS
#define TILE_PART_CLOCKS 131072
#endif
#ifndef TILE_FLUSH_CLOCKS
#define TILE_FLUSH_CLOCKS 16
#endif
#ifndef TILE_WAIT_SPINS
#define TILE_WAIT_SPINS (1u << 22)  // ~0.3 s of 64 ns sleeps: far beyond any store phase
#endif
#ifndef TILE_CHUNK_PAIRS
#define TILE_CHUNK_PAIRS 512  // entry pairs a chunk of units should list (from the previous cycle's rate)
#endif
#ifndef TILE_MIN_CHUNK
#define TILE_MIN_CHUNK 8ll  // units per chunk at least
#endif
// shared memory of one warp: the ring (depth x 64 pairs), the segments' bases, the units that fired
#define TILE_WARP_BYTES(depth) ((depth) * 1024 + 32 * 4 + 32)

// Counters are [4][tile]: E low, E high, I low, I high words (word-major, so
// lanes adding into scattered targets spread over all shared-memory banks).
// acc: shared-memory address of the counters; hi: bytes from a low word to its high word. The
// addresses are 32-bit shared-memory ones throughout: through a generic pointer the compiler
// emits both kinds of atomic and a compare-and-swap loop, ten shared accesses per addition.
static __device__ __forceinline__ unsigned atom_add_shared(unsigned p, unsigned v)
{
    unsigned old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(p), "r"(v) : "memory");
    return old;
}
static __device__ __forceinline__ void red_add_shared(unsigned p, unsigned v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
// Four entries: all low words first, so that the atomics' latencies overlap (a returned value is
// waited for only where it is used).
static __device__ __forceinline__ void carry_add4(unsigned acc, uint4 v, uint4 w, unsigned hi)
{
    const unsigned x[4] = {acc + v.x, acc + v.z, acc + w.x, acc + w.z};
    const unsigned long long u[4] = {(unsigned long long)__float2ll_rn(__uint_as_float(v.y)),
                                     (unsigned long long)__float2ll_rn(__uint_as_float(v.w)),
                                     (unsigned long long)__float2ll_rn(__uint_as_float(w.y)),
                                     (unsigned long long)__float2ll_rn(__uint_as_float(w.w))};
    unsigned o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = atom_add_shared(x[i], (unsigned)u[i]);
#pragma unroll
    for (int i = 0; i < 4; i++)
        red_add_shared(x[i] + hi, (unsigned)(u[i] >> 32) + (o[i] + (unsigned)u[i] < o[i] ? 1u : 0u));
}
static __device__ __forceinline__ uint4 ld_shared16(unsigned p)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p) : "memory");
    return v;
}
static __device__ __forceinline__ unsigned ld_shared4(unsigned p)
{
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
static __device__ __forceinline__ void st_shared16_zero(unsigned p)
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(p), "r"(0) : "memory");
}
static __device__ __forceinline__ void st_shared1(unsigned p, int v)
{
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
static __device__ __forceinline__ int ld_shared1(unsigned p)
{
    int v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
static __device__ __forceinline__ void st_shared4(unsigned p, unsigned v)
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}

// One 16-byte copy to shared memory, past L1 and evict-first in L2 (read once per spike).
static __device__ __forceinline__ void copy16_async(unsigned dst, const uint4 *src, unsigned long long pol, bool on)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t"
                 "@p cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n\t}" ::"r"(dst),
                 "l"(src), "l"(pol), "r"((unsigned)on)
                 : "memory");
}
// 1 << n, 0 for n of 32 and more (also those that were negative).
static __device__ __forceinline__ unsigned bit_or_none(unsigned n)
{
    unsigned v;
    asm("shl.b32 %0, 1, %1;" : "=r"(v) : "r"(n));
    return v;
}
static __device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
static __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

static __device__ __forceinline__ long long carry_sum(const unsigned *lo, int T)
{
    return (long long)(((unsigned long long)lo[T] << 32) | (unsigned long long)lo[0]);
}

// A place in the row of all tiles' work units.
struct TilePlace {
    int q;       // tile
    unsigned u;  // unit
};

static __device__ __forceinline__ unsigned tile_unit_count(const StepArgs &a, int q)
{
    return (unsigned)max(a.tile_units[q], 1);  // a tile without sources is flushed all the same
}
// Cost of an item in warp clocks: what its chunks took in the previous cycle, a floor for its units'
// scan, and for a tile's first item the start, the last warp and the flush of one part.
//
// With 1-step delays a cycle's spikes are those of the cycle before alone, and populations that fire
// together every few cycles make each cycle unlike the last: there the clocks, and the pairs listed, are
// means over the last cycles instead (each cycle keeps 1 - 2^-cost_shift of what was there, so that they
// hold 2^cost_shift cycles' worth). At 2 kHz, us per cycle with the last cycle's alone / the means: 100 x
// 10,000 670 / 375, 100 x 4,000 296 / 171, 20 x 5,000 all-to-all 802 / 355, 12 x 3,000 all-to-all 386 / 176;
// at 500 Hz level. Of the costs alone, without the pairs that size the chunks and decide where blocks
// help: 100 x 4,000 288.
static __device__ __forceinline__ unsigned long long item_cost(const StepArgs &a, const unsigned *prev, int i)
{
    const int4 it = a.items[i];  // {tile, first unit, units, targets of the tile in its first item}
    return (unsigned long long)(prev[i] >> a.cost_shift) + (unsigned long long)(TILE_UNIT_CLOCKS * it.z) +
           (it.w ? (unsigned long long)(TILE_PART_CLOCKS + TILE_FLUSH_CLOCKS * it.w) : 0ull);
}

// This block's share [share[0], share[1]) of the units. Every block computes the same costs, so the
// shares meet. s_scan: one word per warp. Ends with a block barrier.
static __device__ __forceinline__ void tile_share(const StepArgs &a, const unsigned *prev, unsigned long long *s_scan,
                                                  TilePlace *share)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (a.n_items + (int)blockDim.x - 1) / (int)blockDim.x;
    const int i0 = min((int)threadIdx.x * per, a.n_items), i1 = min(i0 + per, a.n_items);
    unsigned long long sum = 0;
    for (int i = i0; i < i1; i++) sum += item_cost(a, prev, i);
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long nb = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += nb;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    unsigned long long before = incl - sum, total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        if (w < warp) before += s_scan[w];
        total += s_scan[w];
    }
    for (int k = 0; k < 2; k++) {
        const unsigned long long x = (unsigned long long)((double)total * (double)(blockIdx.x + k) / (double)gridDim.x);
        if (blockIdx.x + k == gridDim.x) {
            if (threadIdx.x == 0) share[k] = TilePlace{a.n_tiles - 1, tile_unit_count(a, a.n_tiles - 1)};
        } else if (x >= before && x < before + sum) {
            unsigned long long c = before;
            for (int i = i0; i < i1; i++) {
                const unsigned long long cost = item_cost(a, prev, i);
                if (x < c + cost) {
                    const int4 it = a.items[i];
                    share[k] = TilePlace{it.x, (unsigned)it.y + (unsigned)((float)it.z * ((float)(x - c) / (float)cost))};
                    break;
                }
                c += cost;
            }
        }
    }
    __syncthreads();
}

static __device__ __forceinline__ unsigned long long tile_phase(const StepArgs &a, unsigned long long t, int pw,
                                                                unsigned *s_acc, char *s_warp, int *s_part,
                                                                unsigned long long *s_scan, TilePlace *s_share)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int depth = a.tile_depth;
    const unsigned acc_sh = (unsigned)__cvta_generic_to_shared(s_acc);
    const unsigned warp_sh = (unsigned)__cvta_generic_to_shared(s_warp) + warp * TILE_WARP_BYTES(depth);
    const unsigned ring_sh = warp_sh + 16 * lane;   // [depth][2][32] pairs: this lane's places
    const unsigned seg_sh = warp_sh + depth * 1024;  // [32] segment bases
    const unsigned unit_sh = seg_sh + 128;           // [32] lanes of the units that fired
    const unsigned lanes_le = 0xffffffffu >> (31 - lane);
    unsigned long long pol;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    unsigned long long ev = 0;
    unsigned long long *s_best = reinterpret_cast<unsigned long long *>(s_part + 2);
    // the counters start at zero once per launch; each flush clears what it read, so the next
    // tile (of any size up to tile_max) finds them zero
    for (int i = threadIdx.x; i < 4 * a.tile_max; i += blockDim.x) s_acc[i] = 0u;
    const unsigned *prev = a.tile_pairs + (int64_t)((t & 1ull) ^ 1ull) * a.n_tiles;
    unsigned *clocks = a.item_clocks + (int64_t)(t & 1ull) * a.n_items;
    tile_share(a, a.item_clocks + (int64_t)((t & 1ull) ^ 1ull) * a.n_items, s_scan, s_share);
    const TilePlace from = s_share[0], to = s_share[1];
    // this block's parts, one per tile of its share: number block + tile, unique as shares follow
    // one another. The word holds the part's end (high half) and its next unit (low half).
    for (int q = from.q + (int)threadIdx.x; q <= to.q; q += blockDim.x) {
        const int id = (int)blockIdx.x + q;
        const unsigned b = q == from.q ? from.u : 0u, e = q == to.q ? to.u : tile_unit_count(a, q);
        a.part_help[id] = 0u;
        a.part_tile[id] = q;
        __threadfence();  // a helper that sees the word sees its tile
        *reinterpret_cast<volatile unsigned long long *>(a.part_word + id) = ((unsigned long long)e << 32) | min(b, e);
    }
    int q_own = from.q;
    for (;;) {
        __syncthreads();  // the parts are published; the last flush has read s_part[1]
        int id = -1;
        while (q_own <= to.q && id < 0) {
            const unsigned b = q_own == from.q ? from.u : 0u, e = q_own == to.q ? to.u : tile_unit_count(a, q_own);
            if (b < e) id = (int)blockIdx.x + q_own;
            q_own++;
        }
        if (id < 0) {
            // the share is done: join the part with the most left per block already helping it, if
            // that is more than what another flush of the tile costs
            if (threadIdx.x == 0) *s_best = 0ull;
            __syncthreads();
            unsigned long long best = 0ull;
            for (int i = threadIdx.x; i < (int)gridDim.x + a.n_tiles; i += blockDim.x) {
                const unsigned long long w = *reinterpret_cast<volatile unsigned long long *>(a.part_word + i);
                const unsigned nx = (unsigned)w, end = (unsigned)(w >> 32);
                if (nx >= end) continue;
                __threadfence();
                const int q = *reinterpret_cast<volatile int *>(a.part_tile + i);
                const unsigned hp = *reinterpret_cast<volatile unsigned *>(a.part_help + i);
                // entry pairs left, about 8 per unit to scan, for each block then on it
                const unsigned flush = (unsigned)(a.tile_beg[q + 1] - a.tile_beg[q]);
                const float per_unit = (float)(prev[q] >> a.cost_shift) / (float)tile_unit_count(a, q) + 8.0f;
                const float left = (float)(end - nx) * per_unit / (float)(hp + 2u);
                if (left < (float)flush) continue;
                const unsigned long long key = ((unsigned long long)__float2uint_rz(left) << 32) | (unsigned)i;
                best = key > best ? key : best;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
                best = other > best ? other : best;
            }
            if (lane == 0 && best) atomicMax(s_best, best);
            __syncthreads();
            const unsigned long long b = *s_best;
            if (b == 0ull) break;
            id = (int)(b & 0xffffffffull);
            if (threadIdx.x == 0) atomicAdd(a.part_help + id, 1u);
        }
        const int q = *reinterpret_cast<volatile int *>(a.part_tile + id);
        unsigned long long *word = a.part_word + id;
        const int tb = a.tile_beg[q], T = a.tile_beg[q + 1] - tb;
        const uint4 *ent = reinterpret_cast<const uint4 *>(a.ent) + a.tile_seg0[q];  // the tile's entry pairs
        const int r0 = a.tile_run_off[q], r1 = a.tile_run_off[q + 1];
        // the warps of every block working on the part take chunks of its units as they become
        // free: 32 units (one per lane), fewer where the tile listed many entry pairs per unit in
        // the previous cycle, so that a hot chunk does not hold up the block for long
        unsigned *pairs_cnt = a.tile_pairs + (int64_t)(t & 1ull) * a.n_tiles + q;
        const unsigned prev_q = prev[q] >> a.cost_shift;
        const int cs = prev_q == 0u ? 32
                                     : (int)max(TILE_MIN_CHUNK, min(32ll, (long long)TILE_CHUNK_PAIRS * a.tile_units[q] /
                                                                              (long long)prev_q));
        unsigned listed = 0;
        int pads = 0;
        // ring: the slot being filled and how far (64 pairs: two per lane), slots filled and not yet added
        int head = 0, filled = 0, held = 0;
        int item = -1;  // of the last chunk's first unit
        unsigned since = 0;
        auto add_oldest = [&]() {
            int k = head - held;
            if (k < 0) k += depth;
            const uint4 v = ld_shared16(ring_sh + k * 1024), w = ld_shared16(ring_sh + k * 1024 + 512);
            carry_add4(acc_sh, v, w, 4u * T);
            pads += (v.w == TILE_PAD_W) + (w.w == TILE_PAD_W);
            held--;
        };
        for (;;) {
            unsigned long long w = 0;
            if (lane == 0) w = atomicAdd(word, (unsigned long long)cs);
            w = __shfl_sync(0xffffffffu, w, 0);
            const int ub = (int)(unsigned)w, u_end = (int)(w >> 32);
            {   // the clocks since the last chunk go to that chunk's item
                const unsigned now = (unsigned)clock();
                if (item >= 0 && lane == 0) atomicAdd(clocks + item, now - since);
                since = now;
            }
            if (ub >= u_end) break;
            const int u = ub + lane;
            unsigned m = 0;
            const uint32_t *off = a.seg_off;  // the unit's 32 segment starts
            if (lane < cs && u < u_end && r0 < r1) {
                int lo = r0, hi = r1 - 1;  // the run that holds unit u
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (a.run_unit0[mid] <= u) lo = mid;
                    else hi = mid - 1;
                }
                const int n_r = a.run_n[lo], chunks = (n_r + 31) >> 5;
                const int v = u - a.run_unit0[lo];
                const int d = v / chunks + 1;
                if (lane == 0) {
                    const int2 it = a.run_item[lo];
                    item = it.x + (d - 1) / it.y;
                }
                const int c = v - (d - 1) * chunks;
                if ((long long)t - d >= 0) {
                    const int64_t s_first = (int64_t)a.run_src0[lo] + 32 * c;
                    const int len = min(32, n_r - 32 * c);
                    const uint32_t *bm = a.bitmap + (int64_t)((t - d) % (unsigned long long)a.R) * a.W;
                    const int64_t wi = s_first >> 5;
                    const int sh = (int)(s_first & 31);
                    unsigned bits = bm[wi];
                    if (sh) bits = (bits >> sh) | ((wi + 1 < a.W ? bm[wi + 1] : 0u) << (32 - sh));
                    m = len == 32 ? bits : (bits & ((1u << len) - 1u));
                    off += a.run_seg0[lo] + (int64_t)(d - 1) * n_r + 32 * c;
                }
            }
            const int cnt = __popc(m);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int nb = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += nb;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            // the units that fired, in order; rank + start finds a fired source's unit
            const unsigned some = __ballot_sync(0xffffffffu, cnt > 0);
            __syncwarp();
            if (cnt > 0) st_shared1(unit_sh + __popc(some & lanes_le) - 1, lane);
            __syncwarp();
            int unit = -1;  // units that started before the 32 ranks
            for (int b0 = 0; b0 < total; b0 += 32) {
                // this lane's segment: fired source number b0 + lane of the chunk
                const int rank = b0 + lane;
                const unsigned start = (unsigned)(incl - cnt - b0);
                const unsigned um = __reduce_or_sync(0xffffffffu, cnt > 0 ? bit_or_none(start) : 0u);
                const int ul = ld_shared1(unit_sh + unit + __popc(um & lanes_le));  // the lane whose unit holds it
                unit += __popc(um);
                unsigned mu = __shfl_sync(0xffffffffu, m, ul);
                int nth = rank - __shfl_sync(0xffffffffu, incl - cnt, ul);
                const unsigned long long ou = __shfl_sync(0xffffffffu, (unsigned long long)off, ul);
                unsigned first = 0;
                int len = 0;
                if (rank < total) {
                    for (; nth > 0; nth--) mu &= mu - 1u;  // its source is the nth set bit
                    const uint32_t *o = reinterpret_cast<const uint32_t *>(ou) + (__ffs(mu) - 1);
                    first = __ldg(o);
                    len = (int)(__ldg(o + 1) - first);
                }
                int excl = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int nb = __shfl_up_sync(0xffffffffu, excl, o);
                    if (lane >= o) excl += nb;
                }
                const int n_pairs = __shfl_sync(0xffffffffu, excl, 31);  // 16-byte entry pairs of the round
                excl -= len;
                listed += (unsigned)n_pairs;
                // segments that hold entries, in lane order: flat position + base = pair of the tile
                const unsigned full = __ballot_sync(0xffffffffu, len > 0);
                __syncwarp();
                if (len > 0) st_shared4(seg_sh + 4 * (__popc(full & lanes_le) - 1), first - (unsigned)excl);
                __syncwarp();
                // the round's pairs follow the last round's in the slot being filled
                excl = len == 0 ? -128 : excl + filled;  // (-128: marks nothing)
                const int end = filled + n_pairs;
                int seg = -1;  // segments that started before the 32 positions
                for (int f0 = 0; f0 < end; f0 += 64) {
                    const unsigned at = (unsigned)(excl - f0);
                    const unsigned m0 = __reduce_or_sync(0xffffffffu, bit_or_none(at));
                    const unsigned m1 = __reduce_or_sync(0xffffffffu, bit_or_none(at - 32u));
                    const int s1 = seg + __popc(m0);
                    const unsigned b0 = ld_shared4(seg_sh + 4 * (seg + __popc(m0 & lanes_le)));
                    const unsigned b1 = ld_shared4(seg_sh + 4 * (s1 + __popc(m1 & lanes_le)));
                    seg = s1 + __popc(m1);
                    const int p = f0 + lane;
                    const unsigned dst = ring_sh + head * 1024;
                    copy16_async(dst, ent + (b0 + (unsigned)(p - filled)), pol, p >= filled && p < end);
                    copy16_async(dst + 512, ent + (b1 + (unsigned)(p + 32 - filled)), pol, p + 32 >= filled && p + 32 < end);
                    if (f0 + 64 > end) break;
                    copy_commit();
                    if (++head == depth) head = 0;
                    if (++held == depth) {
                        if (depth == 2) copy_wait<1>();
                        else if (depth == 1) copy_wait<0>();
                        else copy_wait<2>();
                        add_oldest();
                    }
                }
                filled = end & 63;
            }
        }
        // the rest of the ring; places past the last pair hold zeros, which add nothing
        if (filled > 0) {
            const unsigned dst = ring_sh + head * 1024;
            if (lane >= filled) st_shared16_zero(dst);
            if (lane + 32 >= filled) st_shared16_zero(dst + 512);
            if (++head == depth) head = 0;
            held++;
        }
        copy_wait<0>();
        while (held > 0) add_oldest();
        // every listed pair holds two entries, but for the padding
        if (lane == 0) ev += 2ull * listed;
        ev -= (unsigned long long)pads;
        if (lane == 0 && listed) atomicAdd(pairs_cnt, listed);
        __syncthreads();
        // Flush into the tile's one accumulator plane. The first block to finish a piece of
        // the tile this cycle (an owner or a helper) stores its sums; every other block waits
        // until that store is done and adds its sums with reductions. The first finisher
        // never waits, so the waits always end; they are bounded all the same.
        if (threadIdx.x == 0) {
            const unsigned k = atomicAdd(a.tile_arrive + q, 1u);
            if (k != 0u) {
                const volatile unsigned *done = a.tile_arrive + a.n_tiles + q;
                unsigned spins = 0;
                while (*done == 0u) {
                    if (++spins > TILE_WAIT_SPINS) {
                        raise_error(a, BSIM_DEVERR_TIMEOUT);
                        break;
                    }
                    __nanosleep(64);
                }
                __threadfence();
            }
            s_part[1] = k == 0u;
        }
        __syncthreads();
        if (s_part[1]) {
            longlong2 *g = reinterpret_cast<longlong2 *>(a.acc) + (int64_t)pw * a.N + tb;
            for (int i = threadIdx.x; i < T; i += blockDim.x) {
                g[i] = make_longlong2(carry_sum(s_acc + i, T), carry_sum(s_acc + 2 * T + i, T));
                s_acc[i] = s_acc[T + i] = s_acc[2 * T + i] = s_acc[3 * T + i] = 0u;
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) atomicExch(a.tile_arrive + a.n_tiles + q, 1u);
        } else {
            unsigned long long *g = reinterpret_cast<unsigned long long *>(a.acc) + 2 * ((int64_t)pw * a.N + tb);
            // consecutive lanes add consecutive words (E, I, E, I, ...), so that each 32-byte sector
            // is added to once
            for (int w = threadIdx.x; w < 2 * T; w += blockDim.x) {
                unsigned *lo = s_acc + (w >> 1) + (w & 1) * 2 * T;
                const long long v = carry_sum(lo, T);
                lo[0] = lo[T] = 0u;
                if (v) red_add_u64(g + w, (unsigned long long)v);
            }
        }
    }
    return ev;
}

// ---------------------------------------------------------------------------
// Firing predictor, inside the step: one warp per population evaluates the MLP
// on the population's rates of cycles t-1..t-8 (complete when cycle t runs) and
// its mean in-degree, predicting cycle t+1. Lane u holds hidden units u and
// u+32; the second layer reads the first layer's units through shuffles. The
// prediction only feeds scheduling (the delivery choice of later cycles).
// ---------------------------------------------------------------------------
static __device__ __forceinline__ void predict_phase(const StepArgs &a, unsigned long long t)
{
    const int lane = threadIdx.x & 31;
    const float *P = a.mlp;
    const float *W1 = P, *b1 = P + BSIM_MLP_HIDDEN * BSIM_MLP_IN, *W2 = b1 + BSIM_MLP_HIDDEN;
    const float *b2 = W2 + BSIM_MLP_HIDDEN * BSIM_MLP_HIDDEN, *W3 = b2 + BSIM_MLP_HIDDEN, *b3 = W3 + BSIM_MLP_HIDDEN;
    const int H = a.hist_len;
    for (int p = ((int)(blockIdx.x * blockDim.x + threadIdx.x)) >> 5; p < a.n_pops;
         p += (int)((gridDim.x * blockDim.x) >> 5)) {
        const float size = (float)a.pop_size[p];
        float x[BSIM_MLP_IN];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const long long s = (long long)t - 1 - k;
            x[k] = s >= 0 ? (float)a.pop_hist[(int64_t)(s % H) * a.n_pops + p] / size * 10.0f : 0.0f;
        }
        x[8] = a.pop_indeg[p] * 1e-3f;
        float h1a = b1[lane], h1b = b1[lane + 32];
#pragma unroll
        for (int k = 0; k < BSIM_MLP_IN; k++) {
            h1a = fmaf(W1[lane * BSIM_MLP_IN + k], x[k], h1a);
            h1b = fmaf(W1[(lane + 32) * BSIM_MLP_IN + k], x[k], h1b);
        }
        h1a = fmaxf(h1a, 0.0f);
        h1b = fmaxf(h1b, 0.0f);
        float s_a = b2[lane], s_b = b2[lane + 32];
        for (int k = 0; k < 32; k++) {
            const float ha = __shfl_sync(0xffffffffu, h1a, k), hb = __shfl_sync(0xffffffffu, h1b, k);
            s_a = fmaf(W2[lane * BSIM_MLP_HIDDEN + k], ha, s_a);
            s_a = fmaf(W2[lane * BSIM_MLP_HIDDEN + 32 + k], hb, s_a);
            s_b = fmaf(W2[(lane + 32) * BSIM_MLP_HIDDEN + k], ha, s_b);
            s_b = fmaf(W2[(lane + 32) * BSIM_MLP_HIDDEN + 32 + k], hb, s_b);
        }
        float y = W3[lane] * fmaxf(s_a, 0.0f) + W3[lane + 32] * fmaxf(s_b, 0.0f);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (lane == 0) {
            const float pred = fmaxf(y + b3[0], 0.0f) * size * 0.1f;
            a.pred_ring[(int64_t)((t + 1) & 3) * a.n_pops + p] = pred;
            atomicAdd(&a.pred_sum[((t + 1) & 3) * 2 + 0], pred);
            atomicAdd(&a.pred_sum[((t + 1) & 3) * 2 + 1], pred * a.pop_outdeg[p]);
            if (t >= 3) {
                // the prediction made two cycles ago for cycle t-1, now complete
                const float actual = (float)a.pop_hist[(int64_t)((t - 1) % H) * a.n_pops + p];
                const float predicted = a.pred_ring[(int64_t)((t - 1) & 3) * a.n_pops + p];
                atomicAdd(&a.pstats->abs_err, (double)fabsf(predicted - actual));
                atomicAdd(&a.pstats->actual, (double)actual);
            }
        }
    }
}

// The exact schedule's choice for a cycle that delivers `window_spikes` spikes.
static __device__ __forceinline__ bool exact_tiled(const StepArgs &a, float window_spikes)
{
    const float work = window_spikes * a.mean_outdeg / (float)a.D;
    return a.n_tiles > 0 && a.cost_tile_a + a.cost_tile_b * work < a.cost_push_a + a.cost_push_b * work;
}

// The delivery mode of cycle t under BSIM_DELIVERY_AUTO: the cost model of each
// mode (fixed ns per cycle + ns per event) on the cycle's work.
//  * exact schedule (no predictor attached): the work is the exact spike count of
//    the delivered window t-1 .. t-D times the mean out-degree over D (each spike's
//    synapses are spread over the D delays);
//  * learned schedule: the work is the predictor's estimate for cycle t-1's spikes
//    times the mean out-degree, or the exact count of cycle t-1 when the prediction
//    for that cycle missed by more than the tolerance (the fallback).
// Every block computes the same choice from the same device words.
static __device__ __forceinline__ int auto_delivery(const StepArgs &a, unsigned long long t, float window_spikes)
{
    if (!a.mlp) {
        const int dm = exact_tiled(a, window_spikes) ? BSIM_DELIVERY_TILE : BSIM_DELIVERY_PUSH;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicAdd(&a.pstats->cycles, 1ull);  // (not waited for, as a read and a write would be)
            if (dm == BSIM_DELIVERY_TILE) atomicAdd(&a.pstats->tile_cycles, 1ull);
        }
        return dm;
    }
    float ps = 0.0f, pe = 0.0f, as = 0.0f;
    if (t >= 1) {
        const float *slot = a.pred_sum + ((t - 1) & 3) * 2;
        ps = *reinterpret_cast<const volatile float *>(slot);
        pe = *reinterpret_cast<const volatile float *>(slot + 1);
        as = (float)a.ring_cnt[(t - 1) % (unsigned long long)a.R];
    }
    const bool fallback = t < 3 || fabsf(as - ps) > a.pred_tol * fmaxf(ps, 1.0f);
    // events per cycle: the spikes of one cycle times their out-degree is, at steady
    // activity, what one cycle delivers (its D slots each hold 1/D of those events)
    const float work = fallback ? as * a.mean_outdeg : pe;
    const int dm = (a.n_tiles > 0 && a.cost_tile_a + a.cost_tile_b * work < a.cost_push_a + a.cost_push_b * work)
                       ? BSIM_DELIVERY_TILE
                       : BSIM_DELIVERY_PUSH;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.pstats->cycles += 1;
        a.pstats->fallbacks += fallback ? 1 : 0;
        a.pstats->tile_cycles += dm == BSIM_DELIVERY_TILE ? 1 : 0;
    }
    return dm;
}

// Copies the complete ring slot of cycle t-1 into the raster recording.
static __device__ __forceinline__ void record_phase(const StepArgs &a, unsigned long long t)
{
    if (!a.rec || t == 0) return;
    RecCtl rc;
    {
        const volatile RecCtl *v = a.rec;
        rc.next = v->next;
        rc.t0 = v->t0;
        rc.steps = v->steps;
        rc.cap = v->cap;
    }
    const long long ts = (long long)t - 1;
    const long long k = ts - rc.t0;
    if (k < 0 || k >= rc.steps || rc.next != ts) return;
    const int slot = (int)(ts % a.R);
    const int64_t n = __ldcg(&a.ring_cnt[slot]);
    const int64_t base = __ldcg(&a.rec_off[k]);
    int64_t room = rc.cap - base;
    if (room < 0) room = 0;
    const int64_t ncopy = n < room ? n : room;
    const int32_t *src = a.ring + (int64_t)slot * a.cap;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncopy; i += (int64_t)gridDim.x * blockDim.x)
        a.rec_ids[base + i] = __ldcg(&src[i]);
}

// End of a cycle, by one thread of the last block: recording offsets.
static __device__ __forceinline__ void record_advance(const StepArgs &a, unsigned long long t)
{
    if (!a.rec || t == 0) return;
    volatile RecCtl *rc = a.rec;
    const long long k = (long long)t - 1 - rc->t0;
    if (k >= 0 && k < rc->steps && rc->next == (long long)t - 1) {
        const int64_t n = __ldcg(&a.ring_cnt[(t - 1) % (unsigned long long)a.R]);
        a.rec_off[k + 1] = __ldcg(&a.rec_off[k]) + n;
        rc->next = (long long)t;
    }
}

template <int ACC>
__global__ void __launch_bounds__(STEP_MAX_THREADS, STEP_MIN_BLOCKS) step_kernel(const __grid_constant__ StepArgs a)
{
    __shared__ unsigned long long s_ev;
    __shared__ int s_dm;
    // tiled delivery: whether the block is a tile's first finisher ([1]), the best part to join ([2..3]),
    // the share's scan and bounds
    __shared__ __align__(8) int s_part[4];
    __shared__ TilePlace s_share[2];
    __shared__ int s_last;
    // tiled delivery: [4][tile] u32 counters, then each warp's ring and segment bases; push: the
    // warps' segment tables, then the delay window's spike counts (step_dynamic_smem)
    extern __shared__ __align__(16) unsigned long long s_dyn[];
    PushSeg *s_seg = reinterpret_cast<PushSeg *>(s_dyn);
    long long *s_cum = reinterpret_cast<long long *>(s_seg + MAX_WARPS * PUSH_CHUNK);
    int *s_wcnt = reinterpret_cast<int *>(s_dyn);  // [128] the update's, after the delivery
    // a raised error flag stops every later cycle (block-uniform test)
    if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t *>(a.err) != 0)) return;
    const unsigned long long t = *reinterpret_cast<volatile unsigned long long *>(a.step_ctr);
    const int p = (int)(t & 1ull);
    const int cur = (int)(t % (unsigned long long)a.R);
    // the cycle's delivery mode, by one warp (the spike counts it reads are a hot spot when every warp
    // of the GPU reads them)
    if (threadIdx.x < 32) {
        int dm = a.delivery;
        if (ACC != BSIM_ACC_ORDERED && (dm == BSIM_DELIVERY_PUSH || dm == BSIM_DELIVERY_AUTO)) {
            // the window's counts are read once: for the push walk and for the choice
            delay_window_prefix(a, t, s_cum, [&](int slot) { return __ldcg(&a.ring_cnt[slot]); });
            __syncwarp();
            const float spikes = (float)s_cum[a.D];
            if (dm == BSIM_DELIVERY_AUTO) dm = a.pstats ? auto_delivery(a, t, spikes) : BSIM_DELIVERY_PUSH;
            else if (a.tile_spikes > 0.0f && spikes > a.tile_spikes) dm = BSIM_DELIVERY_TILE;
        }
        if (dm == BSIM_DELIVERY_TILE && a.n_tiles == 0) dm = BSIM_DELIVERY_PUSH;
        if (threadIdx.x == 0) s_dm = dm;
    }
    if (a.mlp && blockIdx.x == 0 && threadIdx.x == 32) {
        // slot t+2 is next written by cycle t+1's prediction
        a.pred_sum[((t + 2) & 3) * 2 + 0] = 0.0f;
        a.pred_sum[((t + 2) & 3) * 2 + 1] = 0.0f;
    }
    unsigned measured = 0;  // thread 0: whether the last cycle was delivered tiled
    if (threadIdx.x == 0) {
        s_ev = 0;
        if (a.n_tiles > 0) measured = *reinterpret_cast<volatile unsigned *>(a.tile_prev);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // slot t+1 is neither written (LIF writes slot t) nor read (delivery reads t-1..t-D) now
        a.ring_cnt[(t + 1) % (unsigned long long)a.R] = 0;
    }
    if (a.pop_hist) {
        int32_t *nxt = a.pop_hist + (int64_t)((t + 1) % (unsigned long long)a.hist_len) * a.n_pops;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_pops; i += gridDim.x * blockDim.x) nxt[i] = 0;
    }
    record_phase(a, t);
    __syncthreads();  // publishes s_dm, s_cum and s_ev
    const bool push = ACC != BSIM_ACC_ORDERED && s_dm == BSIM_DELIVERY_PUSH;
    const bool tiled = ACC != BSIM_ACC_ORDERED && s_dm == BSIM_DELIVERY_TILE;
    unsigned long long ev;
    if (push) {
        ev = push_phase(a, t, p ^ 1, s_cum, s_seg + (threadIdx.x >> 5) * PUSH_CHUNK,
                        (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x,
                        ((long long)gridDim.x * blockDim.x) >> 5);
    } else if (tiled) {
        ev = tile_phase(a, t, p ^ 1, reinterpret_cast<unsigned *>(s_dyn),
                        reinterpret_cast<char *>(s_dyn + 2 * a.tile_max), s_part,
                        s_dyn + 2 * a.tile_max, s_share);  // (the share's scan is done before the rings are used)
    } else {
        ev = pull_phase<ACC>(a, t, p ^ 1);
    }
    if (ev) atomicAdd(&s_ev, ev);
    lif_phase<ACC>(a, t, p, cur, s_wcnt);
    if (a.mlp && a.pop_hist) predict_phase(a, t);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_ev) atomicAdd(a.events, s_ev);
        __threadfence();
        s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1 ? 1 + (int)measured : 0;
    }
    __syncthreads();
    if (s_last) {
        // every other block has finished this cycle: the tiles' finisher counts start over, and the
        // next cycle counts its listed pairs and clocks from what cost_shift keeps of this one's (its
        // places hold those of the cycle before this one, if that was delivered tiled, else nothing new)
        if (tiled)
            for (int i = threadIdx.x; i < 2 * a.n_tiles; i += blockDim.x) a.tile_arrive[i] = 0u;
        if (s_last == 2) {
            const unsigned now = (unsigned)(t & 1ull), next = now ^ 1u;
            auto keep = [&](unsigned *v, int n) {
                for (int i = threadIdx.x; i < n; i += blockDim.x) {
                    const unsigned c = a.cost_shift ? __ldcg(v + (int64_t)now * n + i) : 0u;
                    v[(int64_t)next * n + i] = c - (c >> a.cost_shift);
                }
            };
            keep(a.tile_pairs, a.n_tiles);
            keep(a.item_clocks, a.n_items);
        }
        if (threadIdx.x == 0) {
            if (a.n_tiles > 0) *a.tile_prev = tiled;
            if (tiled) atomicAdd(a.tile_cycles, 1ull);
            // advance the cycle
            record_advance(a, t);
            *a.ticket = 0u;
            *(a.ticket + 1) = 0u;  // the update's chunk counter
            *a.step_ctr = t + 1;
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// Small networks: many cycles in one cooperative launch.
//
// A cycle of a network of a few thousand neurons moves little; one launch per cycle
// spends its ~10 us on the launch and on a chain of dependent reads (error flag,
// cycle counter, spike counts, ids, rows, entries, then the update's chunk counter,
// state, class, ring position). In one launch the blocks meet at a grid barrier
// instead (~4,000 clocks with the release of the sums, whatever the grid), so the
// work is laid out to need few of them:
//
//   * Push: neurons have owners for the whole launch (state in registers), and a
//     block delivers its own neurons' spikes at once, with all delays, into a ring
//     of input accumulators, one per future cycle (acc_ring: cycle c in slot c mod
//     acc_R). A spike of cycle t reaches no update before cycle t + 2, so two cycles
//     are run between barriers: both updates, then the rows of both cycles' spikes.
//     Owners take groups of eight consecutive neurons dealt out over all blocks, so
//     that a population that fires together spreads over the GPU.
//     10 x 1,000 neurons (100 Hz): 10.2 -> 3.1 us per cycle; 5,000 neurons behind
//     Poisson drives 13.7 -> 3.7; 20 x 1,000 all-to-all 18.1 -> 6.0.
//   * Pull (and the ORDERED sums): a block sums the input of its own neurons, so the update
//     follows without a barrier and again two cycles are run between barriers: the input of
//     cycle t takes the spikes up to t - 2, that of t + 1 those up to t - 1, and one scan of
//     the rows tests both. The delay window's fired flags and the rows (8 bytes an entry,
//     as far as they fit) stay in shared memory. 10 x 1,000 neurons, ORDERED: 11.6 -> 4.4
//     us per cycle (9.2 with one cycle per barrier and the rows read from L2, 5.1 with two
//     separate looks at the flags per entry); 36 x 1,000 31.9 -> 11.1; 12 x 3,000 at 2 kHz
//     107 -> 58. What is left of the first is the scan's
//     instructions (110 entries a row, two tests each), the barrier and the flags' exchange.
//
// The fire ring, its counts and the fired flags are kept as step_kernel keeps them,
// so the two can follow one another (loop_enter_kernel, loop_leave_kernel). Data that
// another block wrote during the launch is read past L1 (ld.cg).
//
// The barrier is the launch's only wait: every block adds itself to a counter, with an
// error bit when the device error flag is set, and waits until all have. Two counters
// alternate, so one that a block still reads is not added to for the next barrier, and
// every block sees the same error bits and leaves after the same cycle. The wait is
// bounded (BSIM_DEVERR_TIMEOUT). The launch is cooperative: its blocks are resident at
// the same time.
// ---------------------------------------------------------------------------
// Threads per block. Push: the rows of a few spikes per block, so more warps only make the
// block's own barriers longer (10 x 1,000 neurons, us per cycle: 256 threads 4.3, 512 4.3,
// 1,024 5.1; 20 x 1,000 all-to-all with bursts 11.7, 7.2, 7.3). Pull: every synapse is scanned,
// so all the warps that fit (18.6, 12.8, 10.0 on the same network).
#define LOOP_THREADS 512
#define PULL_LOOP_THREADS 1024
#define LOOP_WARPS (LOOP_THREADS / 32)
#define PULL_LOOP_WARPS (PULL_LOOP_THREADS / 32)
#define LOOP_MAX_DELAY 64
#define LOOP_CYCLES 2  // between barriers of the push form: the shortest delay (1 step) + 1
#ifndef LOOP_WAIT_SPINS
#define LOOP_WAIT_SPINS (1u << 22)  // seconds: a cycle takes microseconds
#endif
#define LOOP_MAX_SMEM ((size_t)160 * 1024)
// Pull: the fired flags, and the rows of the block's neurons as far as they fit (none for a launch of
// fewer cycles than PULL_LOOP_HOLD, which would read most of them once).
#define PULL_LOOP_SMEM ((size_t)216 * 1024)
#define PULL_LOOP_WORDS (LOOP_WARPS / 2)  // words of fired flags per block at most (loop_form)
#define PULL_LOOP_HOLD 3

static __device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
static __device__ __forceinline__ void red_release(unsigned long long *p, unsigned long long v)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The recording during a launch: every block follows the offsets (block 0 writes them).
struct LoopRec {
    long long t0, steps, cap;
    int64_t off;  // spikes recorded so far
    bool on;
};
static __device__ __forceinline__ LoopRec loop_record_begin(const StepArgs &a, unsigned long long t)
{
    LoopRec r{0, 0, 0, 0, false};
    if (a.rec) {
        const volatile RecCtl *rc = a.rec;
        r.t0 = rc->t0;
        r.steps = rc->steps;
        r.cap = rc->cap;
        const long long k = (long long)t - r.t0;
        r.on = k >= 0 && k < r.steps && rc->next == (long long)t;
        if (r.on) r.off = __ldcg(&a.rec_off[k]);
    }
    return r;
}

// Copies the spikes of cycles [t, t_end), complete, into the recording (slot: ring slot of t).
static __device__ __forceinline__ void loop_record(const StepArgs &a, LoopRec &r, unsigned long long t,
                                                   unsigned long long t_end, int slot)
{
    for (; r.on && t < t_end; t++) {
        const long long k = (long long)t - r.t0;
        if (k >= r.steps) {
            r.on = false;
            break;
        }
        const int64_t count = __ldcg(&a.ring_cnt[slot]);
        const int64_t n = min(count, max((int64_t)0, (int64_t)r.cap - r.off));
        const int32_t *src = a.ring + (int64_t)slot * a.cap;
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
            a.rec_ids[r.off + i] = __ldcg(&src[i]);
        r.off += count;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.rec_off[k + 1] = r.off;
            a.rec->next = (long long)t + 1;
        }
        if (++slot == a.R) slot = 0;
    }
}

// Barrier number k of the launch. `base`: the counter's value when none of this barrier's blocks
// had arrived (blocks leave a counter at a multiple of the grid). Returns whether the launch stops
// here. The block's last warp (which owns no neurons) arrives and waits; meanwhile the others may
// do `shadow`.
struct LoopBar {
    unsigned long long base[2];
    int k;
};
static __device__ __forceinline__ LoopBar loop_bar_begin(const StepArgs &a)
{
    LoopBar b{{0, 0}, 0};
    if (threadIdx.x == blockDim.x - 32)
        for (int i = 0; i < 2; i++) {
            const unsigned long long v = ld_acquire(a.loop_bar + 16 * i);  // this block has not arrived yet
            b.base[i] = v - (v & (LOOP_ERR - 1)) % gridDim.x;
        }
    return b;
}
template <typename Shadow>
static __device__ __forceinline__ bool loop_barrier(const StepArgs &a, LoopBar &b, const bool *s_err, bool *s_stop,
                                                    Shadow shadow)
{
    __syncthreads();
    if (threadIdx.x != blockDim.x - 32) {
        shadow();
    } else {
        const int p = b.k & 1;
        unsigned long long *ctr = a.loop_bar + 16 * p;
        red_release(ctr, 1ull + (*s_err ? LOOP_ERR : 0ull));
        const unsigned long long all = (b.base[p] & (LOOP_ERR - 1)) + gridDim.x;
        unsigned long long w;
        unsigned spins = 0;
        bool stop = false;
        while (((w = ld_acquire(ctr)) & (LOOP_ERR - 1)) != all) {
            if (++spins > LOOP_WAIT_SPINS) {
                raise_error(a, BSIM_DEVERR_TIMEOUT);
                stop = true;
                break;
            }
        }
        *s_stop = stop || (w / LOOP_ERR) != (b.base[p] / LOOP_ERR);
        b.base[p] = w;
    }
    b.k++;
    __syncthreads();
    return *s_stop;
}

// The counters of the n cycles from t on, t in ring slot `slot` (what they held is not read any more).
static __device__ __forceinline__ void loop_clear_counts(const StepArgs &a, unsigned long long t, int slot, int n)
{
    const int lane = threadIdx.x & 31;
    for (int c = 0; c < n; c++) {
        if (lane == 0) a.ring_cnt[slot] = 0;
        if (a.pop_hist) {
            int32_t *nxt = a.pop_hist + (int64_t)((t + c) % (unsigned long long)a.hist_len) * a.n_pops;
            for (int i = lane; i < a.n_pops; i += 32) nxt[i] = 0;
        }
        if (++slot == a.R) slot = 0;
    }
}

// Reserves a warp's places in the fire ring of cycle t (mask: the lanes that fired), and, later,
// fills them: the reservation's latency is not waited for in between.
static __device__ __forceinline__ int loop_reserve(const StepArgs &a, int slot, unsigned mask)
{
    int at = 0;
    if (mask && (threadIdx.x & 31) == 0) at = atomicAdd(&a.ring_cnt[slot], __popc(mask));
    return at;
}
static __device__ __forceinline__ void loop_append(const StepArgs &a, unsigned long long t, int slot, unsigned mask, int at,
                                                   int64_t j, int pop)
{
    if (!mask) return;
    const int lane = threadIdx.x & 31;
    const bool fired = (mask >> lane) & 1u;
    at = __shfl_sync(0xffffffffu, at, 0);
    if (fired) a.ring[(int64_t)slot * a.cap + at + __popc(mask & ((1u << lane) - 1u))] = (int32_t)j;
    if (a.pop_hist) {
        // one atomic per (warp, population) with spikes
        int32_t *hist = a.pop_hist + (int64_t)(t % (unsigned long long)a.hist_len) * a.n_pops;
        const unsigned same = __match_any_sync(0xffffffffu, fired ? pop : -1);
        if (fired && lane == __ffs(same) - 1) atomicAdd(&hist[pop], __popc(same));
    }
}

struct LoopSpike {
    int who, cycle;  // owner thread's number in the block, cycle within the interval
    float scale;     // 2^qexp of the source's network
};

// Dynamic shared memory of the push form: each owner thread's row start and its D + 1 delay
// segments' starts within the row.
static __host__ __device__ __forceinline__ size_t push_loop_smem(int64_t N, int D, int grid)
{
    const int64_t octets = (N + 7) / 8, owner_warps = (octets + 4 * (int64_t)grid - 1) / (4 * (int64_t)grid);
    return (size_t)owner_warps * 32 * (sizeof(int64_t) + sizeof(unsigned) * (size_t)(D + 1));
}

__global__ void __launch_bounds__(LOOP_THREADS, 1) push_loop_kernel(const __grid_constant__ StepArgs a, int steps)
{
    __shared__ LoopSpike s_spike[LOOP_CYCLES * LOOP_THREADS / 2];  // at most half the warps own neurons
    __shared__ unsigned long long s_ev[LOOP_MAX_DELAY + 3];        // events by the cycle that delivers them
    __shared__ int s_n;
    __shared__ bool s_stop, s_err;
    extern __shared__ __align__(16) unsigned long long s_dyn[];  // rows (push_loop_smem)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int D = a.D, Ra = a.acc_R;
    if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t *>(a.err) != 0)) return;
    unsigned long long t = *reinterpret_cast<volatile unsigned long long *>(a.step_ctr);
    // owners: four groups of eight neurons per warp, dealt out over all owning warps
    const int64_t octets = (a.N + 7) / 8;
    const int owner_warps = (int)((octets + 4 * (int64_t)gridDim.x - 1) / (4 * (int64_t)gridDim.x));
    const bool owner = warp < owner_warps;
    const int64_t octet = (int64_t)(lane >> 3) * owner_warps * gridDim.x + (int64_t)warp * gridDim.x + blockIdx.x;
    const int64_t j = octet * 8 + (lane & 7);
    const bool mine = owner && j < a.N;
    longlong2 *acc = reinterpret_cast<longlong2 *>(a.acc_ring);
    const ClassParams *c = a.ctab;
    float4 st = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float scale_down = 0.0f, scale_up = 0.0f, vt = 0.0f, vt_alt = 0.0f;
    int pop = -1, fires = 0, kind = BSIM_NEURON_LIF;
    // The barrier's acquire empties L1, so what a cycle needs of the class, the drive and the
    // rows' bounds is kept in registers and shared memory.
    LifConst lif{};
    int64_t *s_row0 = reinterpret_cast<int64_t *>(s_dyn);
    unsigned *s_seg0 = reinterpret_cast<unsigned *>(s_row0 + owner_warps * 32);
    if (mine) {
        c += a.cls[j];
        st = a.state[j];
        scale_down = __ldg(&c->scale_down);
        scale_up = __ldg(&c->scale_up);
        pop = __ldg(&c->pop);
        kind = __ldg(&c->kind);
        lif = lif_const(c);
        vt = a.vtmp[j];
        if (a.drive_half > 0) vt_alt = a.vtmp_alt[j];
        const int64_t *row = a.row_off + j * D;
        const int64_t r0 = __ldg(row);
        s_row0[threadIdx.x] = r0;
        for (int d = 0; d <= D; d++) s_seg0[threadIdx.x * (D + 1) + d] = (unsigned)(__ldg(row + d) - r0);
    }
    int gap = -1;  // a Poisson neuron's gap after its next spike, drawn ahead while the barrier waits
    if (threadIdx.x == 0) {
        s_n = 0;
        s_err = false;
    }
    if (threadIdx.x < Ra) {  // spikes in flight when the launch starts: counted by block 0
        s_ev[threadIdx.x] = blockIdx.x == 0 ? a.loop_ev[threadIdx.x] : 0ull;
        if (blockIdx.x == 0) a.loop_ev[threadIdx.x] = 0ull;
    }
    __syncthreads();
    unsigned long long ev = 0;  // thread 0: events delivered
    // the exact schedule's choices, as step_kernel counts them
    const bool choices = a.pstats && blockIdx.x == 0 && warp == LOOP_WARPS - 2;
    unsigned long long tile_choices = 0;
    const unsigned long long t_first = t;
    int slot = (int)(t % (unsigned long long)Ra);         // accumulator slot of cycle t
    int rslot = (int)(t % (unsigned long long)a.R);       // ring slot of cycle t
    LoopBar bar = loop_bar_begin(a);
    LoopRec rec = loop_record_begin(a, t);
    bool stop = false;
    for (int k = 0; k < steps && !stop;) {
        const int m = min(LOOP_CYCLES, steps - k);
        const int rslot1 = rslot + 1 < a.R ? rslot + 1 : 0;  // of cycle t + 1
        unsigned mask[LOOP_CYCLES];
        int place[LOOP_CYCLES];
        // ---- the updates of cycles t .. t+m-1: their inputs are complete
        if (owner) {
            longlong2 in[LOOP_CYCLES];
#pragma unroll
            for (int i = 0; i < LOOP_CYCLES; i++) {
                in[i] = make_longlong2(0, 0);
                if (mine && i < m) {
                    longlong2 *q = acc + (int64_t)(slot + i < Ra ? slot + i : slot + i - Ra) * a.N + j;
                    in[i] = __ldcg(q);
                    __stcg(q, make_longlong2(0, 0));
                }
            }
#pragma unroll
            for (int i = 0; i < LOOP_CYCLES; i++) {
                bool fired = false;
                if (mine && i < m) {
                    const float inE = __fmul_rn(__ll2float_rn(in[i].x), scale_down);
                    const float inI = __fmul_rn(__ll2float_rn(in[i].y), scale_down);
                    if (kind == BSIM_NEURON_LIF) {
                        const bool alt = a.drive_half > 0 && (((t + i) / (unsigned long long)a.drive_half) & 1ull);
                        lif_update(lif, alt ? vt_alt : vt, inE, inI, st, fired);
                    } else {
                        drive_update(kind, (int)(t + i), st, fired, [&](int fc) {
                            const int g = gap >= 0 ? gap : poisson_gap(a, c, j, st, fc);
                            gap = -1;
                            return g;
                        });
                    }
                    if (a.trace) trace_neuron(a, trace_row(a, t + i), j, st, inE, inI);
                }
                mask[i] = __ballot_sync(0xffffffffu, fired);
                if (mask[i]) {
                    int at = 0;
                    if (lane == 0) at = atomicAdd(&s_n, __popc(mask[i]));
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (fired) {
                        s_spike[at + __popc(mask[i] & ((1u << lane) - 1u))] = LoopSpike{(int)threadIdx.x, i, scale_up};
                        fires++;
                    }
                }
                place[i] = i < m ? loop_reserve(a, i == 0 ? rslot : rslot1, mask[i]) : 0;
            }
        }
        __syncthreads();
        // ---- the rows of this block's spikes, all delays: a spike of cycle t+i with delay d is
        // input of cycle t+i+d+1. With fewer spikes than warps each row is cut into pieces.
        const int n = s_n;
        const int split = n > 0 && 2 * n <= LOOP_WARPS ? LOOP_WARPS / n : 1;
        for (int it = warp; it < n * split; it += LOOP_WARPS) {
            const LoopSpike sp = s_spike[it / split];
            const unsigned *off = s_seg0 + sp.who * (D + 1);
            const int64_t r0 = s_row0[sp.who];
            int64_t lo = r0, hi = r0 + off[D];
            if (split > 1) {  // inner cuts lie on 16-byte boundaries
                const int64_t len = hi - lo, b = lo;
                const int piece = it % split;
                const int64_t cut0 = (b + len * piece / split + 1) & ~1ll, cut1 = (b + len * (piece + 1) / split + 1) & ~1ll;
                if (piece > 0) lo = min(cut0, hi);
                if (piece + 1 < split) hi = min(cut1, hi);
            }
            int slot0 = slot + sp.cycle + 2;  // of delay 1
            if (slot0 >= Ra) slot0 -= Ra;
            auto add = [&](int d, uint32_t tgt, uint32_t wbits) {  // d: delay - 1
                if ((int64_t)tgt >= a.N) {  // a target outside the network: flag it, touch nothing
                    raise_error(a, BSIM_DEVERR_TARGET);
                    s_err = true;
                    return;
                }
                int sl = slot0 + d;
                if (sl >= Ra) sl -= Ra;
                const float w = __uint_as_float(wbits);
                const long long q = __float2ll_rn(__fmul_rn(w, sp.scale));
                red_add_u64(reinterpret_cast<unsigned long long *>(acc + (int64_t)sl * a.N + tgt) + (w >= 0.0f ? 0 : 1),
                            (unsigned long long)q);
            };
            // entries by their places in the row: [from, to) here, in pairs from an even position
            const int from = (int)(lo - r0), to = (int)(hi - r0), first = (int)((lo & ~1ll) - r0);
            const int n_pairs = (to - first + 1) >> 1;
            const uint4 *pairs = reinterpret_cast<const uint4 *>(a.syn + r0 + first);
            // the segments that hold entries x and x + 1, one search for both
            auto add_pair = [&](int x, uint4 v) {
                int d = 0;
                if (D > 1) {
                    const unsigned y = (unsigned)max(x, from);
                    int top = D - 1;
                    while (d < top) {
                        const int mid = (d + top + 1) >> 1;
                        if (off[mid] <= y) d = mid;
                        else top = mid - 1;
                    }
                }
                if (x >= from) add(d, v.x, v.y);
                if (x + 1 < to) {
                    if (D > 1)
                        while (off[d + 1] <= (unsigned)(x + 1)) d++;
                    add(d, v.z, v.w);
                }
            };
            if (it % split == 0)  // delivered in cycle t+i+d: counted when that cycle has run
                for (int d = lane; d < D; d += 32) {
                    int sl = slot + sp.cycle + 1 + d;
                    if (sl >= Ra) sl -= Ra;
                    if (off[d + 1] != off[d]) atomicAdd(&s_ev[sl], (unsigned long long)(off[d + 1] - off[d]));
                }
            // Pairs of entries from even positions; the rows are read again within cycles, so they
            // stay in L2 (the array has room for the pair that holds its last entry). Each row is
            // walked from a point of its own, wrapping around, so that blocks whose rows hit the same
            // targets do not add into the same addresses in lockstep, and one search finds the delays
            // of both entries of a pair (us per cycle, before / after: 2 x 6,000 neurons at p = 0.5,
            // 2 kHz, 1-step delays 79 / 64, 50-step delays 80 / 59; 10 x 1,000 all-to-all, 500 Hz,
            // 10.4 / 10.0 and 16.2 / 12.3; 10 x 1,000 at 0.1, 100 Hz, 6-step delays 3.19 / 3.05).
            const int rot = (int)__umulhi((unsigned)sp.who * 2654435769u + blockIdx.x * 2246822519u, (unsigned)n_pairs);
            for (int q0 = lane; q0 < n_pairs; q0 += 4 * 32) {
                uint4 v[4];
                int at[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    at[u] = q0 + u * 32 + rot;
                    if (at[u] >= n_pairs) at[u] -= n_pairs;
                    if (q0 + u * 32 < n_pairs) v[u] = __ldg(pairs + at[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (q0 + u * 32 < n_pairs) add_pair(first + 2 * at[u], v[u]);
            }
        }
        // ---- history: fired flags and the fire ring (not read by this launch's delivery)
        if (owner) {
            for (int i = 0; i < m; i++) {
                const unsigned mk = i == 0 ? mask[0] : mask[1];
                const int rs = i == 0 ? rslot : rslot1;
                if ((lane & 7) == 0 && octet < octets)
                    reinterpret_cast<uint8_t *>(a.bitmap + (int64_t)rs * a.W)[octet] = (uint8_t)(mk >> lane);
                loop_append(a, t + i, rs, mk, i == 0 ? place[0] : place[1], j, pop);
            }
        }
        if (blockIdx.x == 0 && warp == LOOP_WARPS - 1) loop_clear_counts(a, t + m, (rslot + m) % a.R, LOOP_CYCLES);
        stop = loop_barrier(a, bar, &s_err, &s_stop, [&] {
            if (kind == BSIM_NEURON_POISSON && gap < 0) gap = poisson_gap(a, c, j, st, __float_as_int(st.y));
        });
        if (threadIdx.x == 0) {
            s_n = 0;
            for (int i = 0; i < m; i++) {
                const int sl = slot + i < Ra ? slot + i : slot + i - Ra;
                ev += s_ev[sl];
                s_ev[sl] = 0ull;
            }
        }
        if (choices)
            for (int i = 0; i < m; i++) {
                int n_spikes = 0;  // delivered in cycle t + i
                for (int d = 1 + lane; d <= D; d += 32) {
                    const int sl = rslot + i - d;
                    if ((long long)t + i - d >= 0) n_spikes += __ldcg(&a.ring_cnt[sl < 0 ? sl + a.R : sl < a.R ? sl : sl - a.R]);
                }
                n_spikes = __reduce_add_sync(0xffffffffu, n_spikes);
                tile_choices += exact_tiled(a, (float)n_spikes);
            }
        if (rec.on) loop_record(a, rec, t, t + m, rslot);
        t += m;
        k += m;
        slot = (slot + m) % Ra;
        rslot = (rslot + m) % a.R;
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.step_ctr = t;
    if (choices && lane == 0) {
        atomicAdd(&a.pstats->cycles, t - t_first);
        atomicAdd(&a.pstats->tile_cycles, tile_choices);
    }
    if (threadIdx.x < Ra && s_ev[threadIdx.x]) atomicAdd(&a.loop_ev[threadIdx.x], s_ev[threadIdx.x]);  // still in flight
    if (mine) {
        a.state[j] = st;
        if (fires) a.fire_count[j] += fires;
    }
    if (ev) atomicAdd(a.events, ev);
}

template <int ACC>
__global__ void __launch_bounds__(PULL_LOOP_THREADS, 1)
    pull_loop_kernel(const __grid_constant__ StepArgs a, int steps, int room)
{
    __shared__ bool s_stop, s_err;
    __shared__ longlong2 s_in[LOOP_CYCLES][PULL_LOOP_WORDS * 32];  // input of cycles t, t + 1 of this block's neurons
    extern __shared__ __align__(16) unsigned long long s_dyn[];    // [1 + R][W] the fired flags, then the warps' rows
    // slot -1 holds what slot R - 1 does, so the slot of the cycle before is always W words back
    uint32_t *s_bm = reinterpret_cast<uint32_t *>(s_dyn) + a.W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = (int)a.W, R = a.R, D = a.D;
    uint2 *rows = reinterpret_cast<uint2 *>(s_dyn + ((size_t)(R + 1) * W + 1) / 2) + (size_t)warp * room;
    if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t *>(a.err) != 0)) return;
    unsigned long long t = *reinterpret_cast<volatile unsigned long long *>(a.step_ctr);
    // the block's neurons: words i * grid + block of the fired flags. Warp i updates word i's; warp w
    // sums the input of neuron w of every word.
    const int words = blockIdx.x < W ? (int)((W - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
    const int64_t word = (int64_t)warp * gridDim.x + blockIdx.x;
    const bool owner = warp < words;
    const int64_t j = word * 32 + lane;
    const bool mine = owner && j < a.N;
    const ClassParams *c = a.ctab;
    float4 st = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float scale_down = 0.0f, vt = 0.0f, vt_alt = 0.0f;
    int pop = -1, fires = 0, kind = BSIM_NEURON_LIF;
    LifConst lif{};
    if (mine) {
        c += a.cls[j];
        st = a.state[j];
        scale_down = __ldg(&c->scale_down);
        pop = __ldg(&c->pop);
        kind = __ldg(&c->kind);
        lif = lif_const(c);
        vt = a.vtmp[j];
        if (a.drive_half > 0) vt_alt = a.vtmp_alt[j];
        const int64_t i = (int64_t)(t & 1ull) * a.N + j;  // cycle t's input
        if (ACC == BSIM_ACC_EXACT) {
            longlong2 *q = reinterpret_cast<longlong2 *>(a.acc) + i;
            s_in[0][threadIdx.x] = *q;
            if (a.acc_clear) *q = make_longlong2(0, 0);  // as step_kernel leaves it
        } else {
            reinterpret_cast<float2 *>(s_in[0])[threadIdx.x] = reinterpret_cast<const float2 *>(a.acc)[i];
        }
    }
    if (threadIdx.x == 0) s_err = false;
    for (int64_t i = threadIdx.x; i < (int64_t)R * W; i += PULL_LOOP_THREADS) {
        const uint32_t v = __ldcg(&a.bitmap[i]);
        s_bm[i] = v;
        if (i >= (int64_t)(R - 1) * W) s_bm[i - (int64_t)R * W] = v;
    }
    // the rows, lane i holding the bounds of the warp's i-th; the first ones stay in shared memory as
    // {source, delay - 1, weight} as far as there is room
    int64_t row0 = 0, row_at = 0;
    long long row_len = 0;
    float row_scale = 0.0f;
    {
        const int64_t tgt = ((int64_t)lane * gridDim.x + blockIdx.x) * 32 + warp;
        if (lane < words && tgt < a.N) {
            row0 = a.col_off[tgt];
            row_len = a.col_off[tgt + 1] - row0;
            if (ACC == BSIM_ACC_EXACT) row_scale = __ldg(&a.ctab[a.cls[tgt]].scale_up);
        }
        row_at = row_len;
        for (int o = 1; o < PULL_LOOP_WORDS; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, (long long)row_at, o);
            if (lane >= o) row_at += v;
        }
        row_at -= row_len;
    }
    const unsigned held = __ballot_sync(0xffffffffu, steps >= PULL_LOOP_HOLD && row_at + row_len <= room);
    for (int i = 0; i < words; i++)
        if ((held >> i) & 1u) {
            const int64_t c0 = __shfl_sync(0xffffffffu, (long long)row0, i);
            const int64_t c1 = c0 + __shfl_sync(0xffffffffu, row_len, i);
            uint2 *to = rows + (int)__shfl_sync(0xffffffffu, (int)row_at, i);
            pull_entries(a, c0, c1, [](uint32_t src, int d) { return src | (unsigned)(d - 1) << 16; },
                         [&](unsigned sd, float w, int64_t k) {
                             if (k + lane < c1) to[k + lane - c0] = make_uint2(sd, __float_as_uint(w));
                         });
        }
    unsigned long long ev = 0;
    int cur = (int)(t % (unsigned long long)R);  // ring slot of cycle t
    bool have = true;                            // cycle t's input is in s_in[0] already
    LoopBar bar = loop_bar_begin(a);
    LoopRec rec = loop_record_begin(a, t);
    bool stop = false;
    for (int k = 0; k < steps && !stop;) {
        // the last interval has one cycle: the input of the cycle after the launch is then at hand
        const int m = steps - k == 1 || (k == 0 && (steps & 1) == 0) ? 1 : LOOP_CYCLES;
        const int cur1 = cur + 1 < R ? cur + 1 : 0;
        __syncthreads();
        // ---- the inputs: cycle t's from the spikes up to t - 2, cycle t + 1's from those up to t - 1
        const int d1 = (long long)t < D ? (int)t : D;  // cycles before the first fired nothing
        for (int i = 0; i < words; i++) {
            const float sc = ACC == BSIM_ACC_EXACT ? __shfl_sync(0xffffffffu, row_scale, i) : 0.0f;
            PullSum<ACC> x0, x1;
            int n = 0;
            auto test = [&](uint32_t src, int d) {
                if (d > d1) return 0u;
                const uint32_t *f = s_bm + (cur >= d ? cur - d : cur - d + R) * W + (src >> 5);
                // (d cycles before t - 1 may be cycle -1, whose flags are zero)
                return ((f[0] >> (src & 31)) & 1u) | ((f[-W] >> (src & 31)) & 1u) << 1;
            };
            auto add = [&](unsigned act, float w, int64_t) {
                if (!__any_sync(0xffffffffu, act)) return;
                n += x1.add(act & 1u, w, sc);
                if (!have) n += x0.add(act >> 1, w, sc);
            };
            if ((held >> i) & 1u) {
                const int len = (int)__shfl_sync(0xffffffffu, row_len, i);
                const uint2 *row = rows + (int)__shfl_sync(0xffffffffu, (int)row_at, i);
                for (int e0 = 0; e0 < len; e0 += 32) {
                    const uint2 v = e0 + lane < len ? row[e0 + lane] : make_uint2(0u, 0u);
                    const int d = e0 + lane < len ? (int)(v.x >> 16) + 1 : PULL_NO_DELAY;
                    add(test(v.x & 0xffffu, d), __uint_as_float(v.y), 0);
                }
            } else {
                const int64_t c0 = __shfl_sync(0xffffffffu, (long long)row0, i);
                pull_entries(a, c0, c0 + __shfl_sync(0xffffffffu, row_len, i), test, add);
            }
            ev += n;
            x1.store(s_in[1], i * 32 + warp);
            if (!have) x0.store(s_in[0], i * 32 + warp);
        }
        __syncthreads();
        // ---- the updates of cycles t .. t+m-1
        if (owner) {
            unsigned mask[LOOP_CYCLES];
            int place[LOOP_CYCLES];
#pragma unroll
            for (int i = 0; i < LOOP_CYCLES; i++) {
                bool fired = false;
                if (mine && i < m) {
                    float inE, inI;
                    if (ACC == BSIM_ACC_EXACT) {
                        const longlong2 in = s_in[i][threadIdx.x];
                        inE = __fmul_rn(__ll2float_rn(in.x), scale_down);
                        inI = __fmul_rn(__ll2float_rn(in.y), scale_down);
                    } else {
                        const float2 in = reinterpret_cast<const float2 *>(s_in[i])[threadIdx.x];
                        inE = in.x;
                        inI = in.y;
                    }
                    if (kind == BSIM_NEURON_LIF) {
                        const bool alt = a.drive_half > 0 && (((t + i) / (unsigned long long)a.drive_half) & 1ull);
                        lif_update(lif, alt ? vt_alt : vt, inE, inI, st, fired);
                    } else {
                        drive_update(kind, (int)(t + i), st, fired, [&](int fc) { return poisson_gap(a, c, j, st, fc); });
                    }
                    if (a.trace) trace_neuron(a, trace_row(a, t + i), j, st, inE, inI);
                    fires += fired;
                }
                mask[i] = __ballot_sync(0xffffffffu, fired);
                place[i] = i < m ? loop_reserve(a, i == 0 ? cur : cur1, mask[i]) : 0;
            }
            if (mine && m == 1) {  // the next cycle's input
                if (k + 1 < steps) {
                    if (ACC == BSIM_ACC_EXACT) s_in[0][threadIdx.x] = s_in[1][threadIdx.x];
                    else
                        reinterpret_cast<float2 *>(s_in[0])[threadIdx.x] =
                            reinterpret_cast<const float2 *>(s_in[1])[threadIdx.x];
                } else {
                    const int64_t i = (int64_t)((t & 1ull) ^ 1ull) * a.N + j;
                    if (ACC == BSIM_ACC_EXACT) reinterpret_cast<longlong2 *>(a.acc)[i] = s_in[1][threadIdx.x];
                    else
                        reinterpret_cast<float2 *>(a.acc)[i] = reinterpret_cast<const float2 *>(s_in[1])[threadIdx.x];
                }
            }
            for (int i = 0; i < m; i++) {
                const unsigned mk = i == 0 ? mask[0] : mask[1];
                const int rs = i == 0 ? cur : cur1;
                if (lane == 0) a.bitmap[(int64_t)rs * W + word] = mk;
                loop_append(a, t + i, rs, mk, i == 0 ? place[0] : place[1], j, pop);
            }
        }
        if (blockIdx.x == 0 && warp == PULL_LOOP_WARPS - 1) loop_clear_counts(a, t + m, (cur + m) % R, LOOP_CYCLES);
        stop = loop_barrier(a, bar, &s_err, &s_stop, [] {});
        for (int i = 0; i < m; i++) {  // their fired flags
            const int64_t at = (int64_t)(i == 0 ? cur : cur1) * W;
            const bool twice = at == (int64_t)(R - 1) * W;
            for (int x = threadIdx.x; x < W; x += PULL_LOOP_THREADS) {
                const uint32_t v = __ldcg(&a.bitmap[at + x]);
                s_bm[at + x] = v;
                if (twice) s_bm[x - W] = v;
            }
        }
        if (rec.on) loop_record(a, rec, t, t + m, cur);
        have = m == 1;
        t += m;
        k += m;
        cur = (cur + m) % R;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.step_ctr = t;
    if (mine) {
        a.state[j] = st;
        if (fires) a.fire_count[j] += fires;
    }
    if (lane == 0 && ev) atomicAdd(a.events, ev);
}

// Before the first of these launches: step_kernel cleared cycle t's counters only.
__global__ void loop_clear_kernel(const __grid_constant__ StepArgs a)
{
    if (*reinterpret_cast<volatile int32_t *>(a.err) != 0) return;
    const unsigned long long t = *a.step_ctr;
    loop_clear_counts(a, t + 1, (int)((t + 1) % (unsigned long long)a.R), 1);
}

// From step_kernel's input accumulators to the ring of push_loop_kernel: the input of the next
// cycle, and the spikes in flight (a spike of cycle s with delay d >= t - s is still to be delivered).
__global__ void loop_enter_kernel(const __grid_constant__ StepArgs a)
{
    if (*reinterpret_cast<volatile int32_t *>(a.err) != 0) return;
    const unsigned long long t = *a.step_ctr;
    const int D = a.D;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc_ring);
    const longlong2 *now = reinterpret_cast<const longlong2 *>(a.acc) + (int64_t)(t & 1ull) * a.N;
    // (the ring was zeroed before this launch; slots of later cycles are added to below)
    if (blockIdx.x == 0 && threadIdx.x < 32) loop_clear_counts(a, t + 1, (int)((t + 1) % (unsigned long long)a.R), 1);  // step_kernel cleared t's
    longlong2 *first = reinterpret_cast<longlong2 *>(a.acc_ring) + (int64_t)(t % (unsigned long long)a.acc_R) * a.N;
    for (int64_t i = tid; i < a.N; i += nt) first[i] = now[i];
    const int lane = threadIdx.x & 31;
    for (int age = 1; age <= D && (long long)t - age >= 0; age++) {
        const unsigned long long s = t - age;
        const int slot = (int)(s % (unsigned long long)a.R);
        const int n = a.ring_cnt[slot];
        for (int64_t i = tid >> 5; i < n; i += nt >> 5) {
            const int id = a.ring[(int64_t)slot * a.cap + i];
            const float sc = a.ctab[a.cls[id]].scale_up;
            for (int d = age; d <= D; d++) {
                unsigned long long *q = acc + 2 * (int64_t)((s + d + 1) % (unsigned long long)a.acc_R) * a.N;
                const int64_t r0 = a.row_off[(int64_t)id * D + d - 1], r1 = a.row_off[(int64_t)id * D + d];
                if (lane == 0 && r1 > r0)
                    atomicAdd(&a.loop_ev[(s + d) % (unsigned long long)a.acc_R], (unsigned long long)(r1 - r0));
                for (int64_t e = r0 + lane; e < r1; e += 32)
                    push_one(a, q, a.syn[e].x, a.syn[e].y, sc);
            }
        }
    }
}

// And back: the next cycle's input; the other parity is delivered into next.
__global__ void loop_leave_kernel(const __grid_constant__ StepArgs a)
{
    const unsigned long long t = *a.step_ctr;
    if (blockIdx.x == 0 && threadIdx.x < a.acc_R) a.loop_ev[threadIdx.x] = 0ull;  // step_kernel counts them
    longlong2 *acc = reinterpret_cast<longlong2 *>(a.acc);
    const longlong2 *now = reinterpret_cast<const longlong2 *>(a.acc_ring) + (int64_t)(t % (unsigned long long)a.acc_R) * a.N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.N; i += (int64_t)gridDim.x * blockDim.x) {
        acc[(int64_t)(t & 1ull) * a.N + i] = now[i];
        acc[(int64_t)((t & 1ull) ^ 1ull) * a.N + i] = make_longlong2(0, 0);
    }
}

// Records the last completed cycle (run after a batch of steps, before reading the raster).
__global__ void record_flush_kernel(const StepArgs a)
{
    const unsigned long long t = *a.step_ctr;  // first cycle not yet run
    if (t == 0 || !a.rec) return;
    const RecCtl rc = *a.rec;
    const long long ts = (long long)t - 1;
    const long long k = ts - rc.t0;
    if (k < 0 || k >= rc.steps || rc.next != ts) return;
    const int slot = (int)(ts % a.R);
    const int64_t n = a.ring_cnt[slot];
    const int64_t base = a.rec_off[k];
    int64_t room = rc.cap - base;
    if (room < 0) room = 0;
    const int64_t ncopy = n < room ? n : room;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncopy; i += (int64_t)gridDim.x * blockDim.x)
        a.rec_ids[base + i] = a.ring[(int64_t)slot * a.cap + i];
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.rec_off[k + 1] = base + n;
        a.rec->next = ts + 1;
    }
}

// Dynamic shared memory of the step kernel: push delivery's tables, or the tile
// counters and the warps' rings where they are larger (one mode runs per cycle).
size_t step_dynamic_smem(const StepArgs &a, int block)
{
    size_t bytes = MAX_WARPS * PUSH_CHUNK * sizeof(PushSeg) + ((size_t)a.D + 1) * sizeof(long long);
    if (a.n_tiles > 0)
        bytes = std::max(bytes, (size_t)4 * a.tile_max * sizeof(unsigned) + (size_t)(block / 32) * TILE_WARP_BYTES(a.tile_depth));
    return bytes;
}

// The attribute belongs to the kernel, not to an engine: it only ever grows,
// so an engine built later with smaller tiles cannot break an earlier one.
cudaError_t step_set_smem(int accumulate, size_t bytes)
{
    static size_t set_bytes[64][2];
    int dev = 0;
    cudaError_t st = cudaGetDevice(&dev);
    if (st != cudaSuccess) return st;
    const int k = accumulate == BSIM_ACC_ORDERED ? 1 : 0;
    if (dev < 0 || dev >= 64 || bytes <= set_bytes[dev][k]) return cudaSuccess;
    if (accumulate == BSIM_ACC_ORDERED)
        st = cudaFuncSetAttribute(step_kernel<BSIM_ACC_ORDERED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)bytes);
    else
        st = cudaFuncSetAttribute(step_kernel<BSIM_ACC_EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)bytes);
    if (st == cudaSuccess) set_bytes[dev][k] = bytes;
    return st;
}

cudaError_t launch_step(Engine &e)
{
    const size_t smem = step_dynamic_smem(e.a, e.block);
    if (e.opt.accumulate == BSIM_ACC_ORDERED)
        step_kernel<BSIM_ACC_ORDERED><<<e.grid, e.block, smem, e.stream>>>(e.a);
    else
        step_kernel<BSIM_ACC_EXACT><<<e.grid, e.block, smem, e.stream>>>(e.a);
    return cudaGetLastError();
}

// One step on explicit arguments (used by the allocation-free entry point).
cudaError_t launch_step_exact(const StepArgs &a, int grid, int block, cudaStream_t stream)
{
    step_kernel<BSIM_ACC_EXACT><<<grid, block, step_dynamic_smem(a, block), stream>>>(a);
    return cudaGetLastError();
}

// Whether an engine of these sizes runs many cycles per launch (0: no, 1: push form, 2: pull form): half of
// a block's warps own neurons at most. Longer delays take one launch per cycle.
//
// An engine asked to deliver tiled takes the push form too: the spikes are the same, and at these sizes
// a tiled cycle is a launch and a chain of dependent reads (10 x 1,000 neurons, 100 Hz: 15.5 us against 3.1),
// and so does an AUTO engine until a predictor is attached (38 x 874 neurons, 1-step delays: 13.0 us against
// 5.5): the choices of the exact schedule are counted, the delivery is the push form's.
//
// Rows: a spike's whole row is one block's, so networks with many synapses in long rows are better spread
// over the GPU by step_kernel, pushed or tiled. Up to LOOP_MAX_SYNAPSES, with rows of up to LOOP_LONG_ROW on
// average where there are more than LOOP_ANY_ROW, the push form was faster than a pushed cycle or level on 20
// networks of 100 Hz to 2 kHz with delays to 1, 6 and 50 steps (us per cycle, 500 Hz, 50 steps, push form /
// pushed: 36 x 1,000 all-to-all, 4.2e7 synapses, 27 / 28; 15 x 1,500, 3.8e7, 30 / 30; 4 x 9,000 at 0.1,
// 3.2e7, 18 / 25; 2 x 5,000, 2.5e7, 36 / 44; one population of 3,000, 9e6, 9 / 15), beyond it was not (12 x 3,000
// at 0.5, 5.9e7, 37 / 34; 3 x 3,000 all-to-all, 2.7e7 in rows of 3,000, 17 / 15 and at 2 kHz 55 / 45).
//
// The pull form scans every row, half as often as step_kernel; a row is one warp's, so that one of
// PULL_LOOP_MAX_ROW entries takes some 50 ms, far from the bound of the barrier's wait.
#define LOOP_MAX_SYNAPSES 45000000
#define LOOP_ANY_ROW 20000000
#define LOOP_LONG_ROW 2500
#define PULL_LOOP_MAX_ROW (1 << 22)
int loop_form(const bsim_options &o, int64_t N, int32_t D, int64_t S, int64_t max_indeg, int sm_count)
{
    const int64_t W = (N + 31) / 32;
    if (D > LOOP_MAX_DELAY || W > (int64_t)(LOOP_WARPS / 2) * sm_count) return 0;
    if (o.accumulate != BSIM_ACC_ORDERED && o.delivery != BSIM_DELIVERY_PULL)
        return S <= LOOP_MAX_SYNAPSES && (S <= LOOP_ANY_ROW || S <= LOOP_LONG_ROW * N) &&
                       push_loop_smem(N, D, sm_count) <= LOOP_MAX_SMEM
                   ? 1
                   : 0;
    const size_t bitmaps = sizeof(uint32_t) * (size_t)(D + LOOP_EXTRA_SLOTS + 1) * W;
    return max_indeg <= PULL_LOOP_MAX_ROW && bitmaps + 8 <= PULL_LOOP_SMEM ? 2 : 0;
}

// Cycles of one launch at most, so that it ends within about a second: 4,096 cycles of a few to 300 us
// pushed; 4e11 row entries scanned.
int64_t loop_launch_cycles(const Engine &e)
{
    const int64_t most = 4096;
    return e.loop == 2 ? std::max<int64_t>(16, std::min(most, (int64_t)4e11 / std::max<int64_t>(e.S, 1))) : most;
}

cudaError_t launch_loop(Engine &e, int steps)
{
    if (e.loop_barriers.start_over(steps)) {  // (one barrier per cycle at most)
        const cudaError_t st = cudaMemsetAsync(e.a.loop_bar, 0, sizeof(unsigned long long) * 32, e.stream);
        if (st != cudaSuccess) return st;
    }
    if (e.loop == 1) {
        void *args[] = {&e.a, &steps};
        const cudaError_t st = cudaFuncSetAttribute((const void *)push_loop_kernel,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LOOP_MAX_SMEM);
        if (st != cudaSuccess) return st;
        return cudaLaunchCooperativeKernel((const void *)push_loop_kernel, dim3(e.sm_count), dim3(LOOP_THREADS), args,
                                           push_loop_smem(e.N, e.D, e.sm_count), e.stream);
    }
    const void *f = e.opt.accumulate == BSIM_ACC_ORDERED ? (const void *)pull_loop_kernel<BSIM_ACC_ORDERED>
                                                         : (const void *)pull_loop_kernel<BSIM_ACC_EXACT>;
    const cudaError_t st = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PULL_LOOP_SMEM);
    if (st != cudaSuccess) return st;
    const size_t flags = (sizeof(uint32_t) * (size_t)(e.a.R + 1) * e.a.W + 7) / 8 * 8;
    // a held entry has 16 bits for its source
    int room = e.N <= 65536 ? (int)((PULL_LOOP_SMEM - flags) / (PULL_LOOP_WARPS * sizeof(uint2))) : 0;
    void *args[] = {&e.a, &steps, &room};
    return cudaLaunchCooperativeKernel(f, dim3(e.sm_count), dim3(PULL_LOOP_THREADS), args, PULL_LOOP_SMEM, e.stream);
}

cudaError_t launch_loop_enter(Engine &e)
{
    if (e.loop == 2) {
        loop_clear_kernel<<<1, 32, 0, e.stream>>>(e.a);
        return cudaGetLastError();
    }
    cudaError_t st = cudaMemsetAsync(e.a.acc_ring, 0, sizeof(longlong2) * (size_t)e.a.acc_R * e.N, e.stream);
    if (st == cudaSuccess)
        st = cudaMemsetAsync(e.a.loop_ev, 0, sizeof(unsigned long long) * e.a.acc_R, e.stream);
    if (st != cudaSuccess) return st;
    loop_enter_kernel<<<e.sm_count, 512, 0, e.stream>>>(e.a);
    return cudaGetLastError();
}

cudaError_t launch_loop_leave(Engine &e)
{
    loop_leave_kernel<<<e.sm_count, 512, 0, e.stream>>>(e.a);
    return cudaGetLastError();
}

cudaError_t launch_record_flush(Engine &e)
{
    record_flush_kernel<<<1, 256, 0, e.stream>>>(e.a);
    return cudaGetLastError();
}

cudaError_t step_occupancy(int block, int accumulate, int *blocks_per_sm, size_t smem)
{
    if (accumulate == BSIM_ACC_ORDERED)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, step_kernel<BSIM_ACC_ORDERED>, block,
                                                             smem);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, step_kernel<BSIM_ACC_EXACT>, block, smem);
}

cudaError_t step_occupancy(int block, int accumulate, int *blocks_per_sm)
{
    return step_occupancy(block, accumulate, blocks_per_sm, 0);
}

}  // namespace bsim
