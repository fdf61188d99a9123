// Internal structures of the bsim_b200 engine (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <vector>

#include "../../include/bsim_b200.h"
#include "drive.h"
#include "loop_barrier.h"

namespace bsim {

// Weight word of a padding entry of the tiled copy (-0.0f: adds nothing; a synapse's
// own zero weight is stored as +0.0f there).
constexpr uint32_t TILE_PAD_W = 0x80000000u;

// Ring slots beyond the longest delay in a many-cycle engine: an interval of two cycles t, t + 1
// clears the counters of t + 2 and t + 3 while a slower block may still copy the spikes of t - 2 and
// t - 1 into the recording, so t + 3 and t - 2 need slots of their own also with 1-step delays.
constexpr int LOOP_EXTRA_SLOTS = 5;

// One neuron class. For LIF_brian neurons: a folded parameter tuple, the
// per-population part of LIFENeuron::reset's output (src/neuron/lif/LIFENeuron.cpp:68-112);
// v_tmp depends on i_offset and is kept per neuron. Input-drive neurons
// (BSIM_NEURON_CONSTANT / _POISSON) keep their parameters per neuron in the state
// slots and use only kind, pop, inst and id_base here. 64 bytes; the table is small
// and read through the L1 cache.
struct ClassParams {
    float Cm, CE, CI, C_E, C_I, v_thresh, v_reset;
    int32_t refrac_time;
    float scale_up;    // 2^qexp: fixed-point value of a weight is rn(w * scale_up)
    float scale_down;  // 2^-qexp
    int32_t pop;       // population (spike statistics)
    int32_t inst;      // independent network
    int32_t kind;      // BSIM_NEURON_*
    int32_t id_base;   // first neuron id of the network (Poisson draws use id - id_base)
    int32_t reserved[2];
};

// Raster recording window: cycles [t0, t0 + steps) into a buffer of cap ids.
struct RecCtl {
    long long next;   // next cycle to copy out (cycle t copies cycle t-1 once it is complete)
    long long t0;
    long long steps;  // 0: not recording
    long long cap;
};

// State trace window: after each cycle t in [t0, t0 + steps), the neurons
// [first, first + count) have v, i_E, i_I and the synaptic input the cycle
// consumed (E, I) copied into the trace buffer, field-major: [5][steps][count].
struct TraceCtl {
    long long t0;
    long long steps;  // 0: not tracing
    long long first;
    long long count;
};

// Firing-predictor statistics, accumulated on the device.
struct PredStats {
    unsigned long long cycles, fallbacks, tile_cycles;
    double abs_err, actual;
};

// Everything one fused step launch needs. Passed by value (kernel parameter space).
struct StepArgs {
    int64_t N;         // neurons
    int32_t D;         // max delay, steps
    int32_t R;         // ring slots: D + 2, D + LOOP_EXTRA_SLOTS in engines that run many cycles per launch
    int64_t cap;       // fired ids per ring slot
    int64_t W;         // bitmap words per ring slot = ceil(N / 32)
    float4 *state;     // [N] LIF: {v, i_E, i_I, refrac_step as int bits}
                       //     Constant: {fire_rate, start_cycle, end_cycle, fire_count} (ints as bits)
                       //     Poisson: {rate, fire_cycle, end_cycle, refrac_step} (ints as bits)
    const float *vtmp; // [N] LIF: v_tmp; Poisson: exp(-(rate mod 64)); Constant: unused
    const float *vtmp_alt;  // [N] v_tmp of the odd half periods of a square-wave drive (may be NULL)
    int32_t drive_half;     // cycles per half period (0: constant drive)
    PoissonTables ptab;     // inversion tables of the Poisson sampler (NULL thr: no Poisson neurons)
    uint64_t input_seed;    // seed of the Poisson neurons' draws
    const uint16_t *cls;       // [N] class of each neuron
    const ClassParams *ctab;   // [n_cls]
    void *acc;                 // [2][N] longlong2 (EXACT) or [2][N] float2 (ORDERED): input for the next step
    int32_t acc_clear;         // the LIF phase zeroes the input it read (0: every cycle overwrites it)
    uint32_t *bitmap;          // [R][W] fired flags of each step in the ring
    int32_t *ring;             // [R][cap] fired ids of each step in the ring
    int32_t *ring_cnt;         // [R]
    const int64_t *row_off;    // [N*D + 1] push rows by (source, delay)
    const uint2 *syn;          // [S] {target id, weight bits}, creation order inside a row
    const int64_t *col_off;    // [N + 1] pull rows by target
    const uint32_t *csc_src;   // [S] source id, creation order inside a row
    const float *csc_w;        // [S]
    const uint8_t *csc_d;      // [S] delay - 1
    int32_t *fire_count;       // [N]
    unsigned long long *step_ctr;  // current cycle t (device-side, advanced by the last block)
    unsigned int *ticket;          // end-of-step block counter
    unsigned long long *events;    // synaptic events delivered
    unsigned long long *tile_cycles;  // cycles delivered from the tiled copy
    // many cycles per launch (small networks)
    unsigned long long *loop_bar;     // [2] barrier counters, 128 bytes apart (small networks only)
    void *acc_ring;                   // [acc_R][N] longlong2: input of cycle c in slot c mod acc_R (push form)
    unsigned long long *loop_ev;      // [acc_R] events in flight by the cycle that delivers them
    int32_t acc_R;                    // D + 3
    int32_t *err;                  // device error flag (0 = ok)
    int32_t push_split;            // pieces of one row at most, in pushed cycles with few spikes
    int32_t delivery;              // BSIM_DELIVERY_*
    // raster recording (control words in device memory so a captured graph stays valid)
    int32_t *rec_ids;           // [rec->cap]
    int64_t *rec_off;           // [rec->steps + 1]
    struct RecCtl *rec;         // NULL: recording never enabled
    // state trace (the reference's LOG_DATA files g_v / g_ie / g_ii / g_input_e / g_input_i)
    float *trace;               // [5][trace_ctl->steps][trace_ctl->count] (NULL: never enabled)
    const struct TraceCtl *trace_ctl;
    // per-population spike counts of the last hist_len steps (predictor input)
    int32_t *pop_hist;          // [hist_len][n_pops]
    int32_t n_pops, hist_len;
    // target-tiled delivery (BSIM_DELIVERY_TILE). A tile is a target range whose
    // excitatory and inhibitory sums are formed in shared memory. Its sources form
    // runs of consecutive neuron ids; every source of a run owns one (tile, source)
    // pair. The work units of all tiles in a row are cut into one share per block, of equal
    // cost; the part of a share that lies in one tile has number block + tile. Every block that
    // worked on a tile stores (the first to finish) or adds (the others, once that store is
    // done) its sums into the accumulator plane.
    int32_t n_tiles;                 // tiles (0: no tiled copy)
    unsigned long long *part_word;   // [part_cap] end unit (high half) and next unit of each part: any block may
                                     // take chunks of any part
    int *part_tile;                  // [part_cap] its tile
    unsigned int *part_help;         // [part_cap] blocks helping it
    unsigned int *tile_pairs;        // [2][n_tiles] entry pairs listed per tile, by cycle parity; the previous
                                     // cycle's count sizes the tile's chunks
    int32_t n_items;                 // cost items: ranges of work units of a tile (delays of a run, or small runs), in
                                     // tile order
    const int4 *items;               // [n_items] {tile, first unit, units, targets of the tile (its first item)}
    const int2 *run_item;            // [runs] first item of each run, delays per item
    unsigned int *item_clocks;       // [2][n_items] warp clocks spent, by cycle parity
    int32_t cost_shift;              // item_clocks and tile_pairs keep 1 - 2^-cost_shift of the cycle before's (0: none)
    unsigned int *tile_prev;         // whether the last cycle was delivered tiled
    unsigned int *tile_arrive;       // [2][n_tiles]: blocks that finished a piece of the tile this
                                     // cycle, and whether the first one's store is done (reset by
                                     // the last block)
    int32_t tile_max;                // largest range (neurons): shared-memory accumulator size
    const int32_t *tile_beg;         // [n_tiles + 1] first target of each tile
    const int32_t *tile_run_off;     // [n_tiles + 1] range of runs
    const int32_t *tile_units;       // [n_tiles] work units: sum over runs of ceil(n/32) * D
    const uint32_t *run_src0;        // [runs] first source
    const int32_t *run_n;            // [runs] sources in the run
    const int64_t *run_seg0;         // [runs] index in seg_off of the run's (delay 1, first source)
    const int32_t *run_unit0;        // [runs] first work unit, counted within the tile
    const uint32_t *seg_off;         // per run [tile's delays][run_n] and one more: start of each (delay,
                                     // source) segment in 16-byte entry pairs from the tile's first one;
                                     // a segment ends where the next one starts
    const int64_t *tile_seg0;        // [n_tiles] first 16-byte entry pair of each tile
    const uint2 *ent;                // [E] {byte offset of the target's low counter word in the tile's
                                     // counters (E or I by the weight's sign), weight x 2^qexp}; every
                                     // segment starts on an even entry and has even length (padding
                                     // entries have the weight word TILE_PAD_W and any offset)
    int32_t tile_depth;              // ring slots per warp, of two 16-byte entry pairs per lane (1..3)
    // firing predictor (needs pop_hist)
    const float *mlp;                // [BSIM_MLP_PARAMS] (NULL: off)
    const int32_t *pop_size;         // [n_pops]
    const float *pop_indeg;          // [n_pops] mean in-degree
    const float *pop_outdeg;         // [n_pops] mean out-degree
    float *pred_ring;                // [4][n_pops] predicted spikes of cycle s at slot s % 4
    float *pred_sum;                 // [4][2] predicted spikes and events of cycle s at slot s % 4
    PredStats *pstats;
    float tile_spikes;               // push delivery: cycles with more spikes in their delay window than this
                                     // go tiled (0: none do)
    float pred_tol, mean_outdeg;
    float cost_push_a, cost_push_b, cost_tile_a, cost_tile_b;  // ns per cycle, ns per event
};

struct Engine {
    int device = 0;
    cudaStream_t stream = nullptr;
    bsim_options opt{};
    int sm_count = 0;
    int64_t N = 0, S = 0;
    int64_t max_indeg = 0;  // longest row by target
    int32_t D = 1;
    float dt = 0.0f;
    int32_t n_inst = 1, n_cls = 0, n_pops = 1;
    std::vector<int32_t> qexp;  // per instance
    int64_t steps_done = 0;
    int64_t device_bytes = 0;
    std::vector<void *> allocs;
    StepArgs a{};
    int grid = 0, block = 0;
    // CUDA graph of graph_steps fused steps
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t graph_exec = nullptr;
    int graph_len = 0;
    // many cycles per launch: 0 no, 1 push form, 2 pull form; and whether the last cycles ran so
    // (the push form then has the spikes in flight in acc_ring, not in step_kernel's accumulators)
    int loop = 0;
    bool in_loop = false;
    LoopBarriers loop_barriers;
    // recording
    int64_t rec_cap_alloc = 0, rec_steps_alloc = 0;
    bool rec_dirty = false;
    int64_t trace_alloc = 0;  // floats in the trace buffer
    // read-back of the recording: the per-cycle sort's output and scratch, sized
    // when the recording is set up, so that reading allocates nothing
    int32_t *rec_sorted = nullptr;
    void *sort_tmp = nullptr;
    size_t sort_tmp_bytes = 0;
    // staging for state uploads and read-backs: four planes of N words (v, i_E,
    // i_I, refrac), so the host's arrays move with one copy each, no host repacking
    float *stage = nullptr;
    // page-locked (ensure_host): the error flag as the last synchronisation saw it and, for small
    // engines, five planes of N words for the state's fields and the spike counts (a copy into the
    // caller's pageable memory waits for each piece by itself). The state's planes here and in `stage`
    // belong to the thread that holds stage_mutex, the counts' to that which holds count_mutex.
    std::once_flag host_once;
    std::mutex stage_mutex, count_mutex;
    int32_t *h_err = nullptr;
    float *h_stage = nullptr;
    // schedule state: predictor statistics and the MLP's parameters (a.pstats / a.mlp
    // point here while a schedule / a predictor is attached)
    PredStats *pstats_mem = nullptr;
    float *mlp_mem = nullptr;
    // population statistics (device arrays in a: pop_size, pop_indeg, pop_outdeg)
    bool pop_info_ready = false;
};

}  // namespace bsim
