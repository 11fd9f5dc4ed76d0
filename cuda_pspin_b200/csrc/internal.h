// internal.h -- engine state shared by the host code and the kernels.
//
// HBM layout of one handle (a batch of S disorder samples):
//
//   spins      float2 [sum_s N_s * R_s]   per sample [site][replica], replica
//                                           fastest, so 32 replicas of one site
//                                           are one 256-byte row
//   per-replica arrays [sum_s R_s]          energy (f64), accepted/proposed
//                                           (i64), beta (f64), RNG key (u64),
//                                           constraint target (f64)
//   site lists int2   [sum_s entries_s]     per sample, per site: groups of
//                                           terms with the same (p, o1), as
//                                           dense tiles of up to 8 groups, or
//                                           one 16-byte record {g (f32 bits),
//                                           o2, p<<16|o1, last} per term, packed
//                                           in TMA chunks of <= 256 entries that
//                                           hold whole groups or tiles, start
//                                           16-byte aligned and have an even
//                                           length.  The pair sub-lists of the
//                                           two-pass sweep keep the group
//                                           format: a header {len, p<<16|o1} and
//                                           len data entries {g, o2}
//   chunk starts int64 [n_chunks + 1]       entry offset of every chunk
//   site chunks int32 [sum_s N_s * 33]      first chunk of each of the 32
//                                           balanced parts of a site's list
//                                           (entry 32: one past its last chunk)
//   quartet table Q64 [sum_s nq_s]          active (quartet, channel) with FP64
//                                           g, for the FP64 energy resync
//   g2         f64    [sum_s N_s^2]         dense 2-body couplings (real parts)
//
// Site-list algebra.  For quartet {i,j,k,l} with channel ch the energy term
// is -Re[g a_u1 a_u2 conj(a_c1) conj(a_c2)] (u: unconjugated pair, c:
// conjugated pair; disorder.h:9-16).  For a member site m with partner p
// (the other site of m's pair) and opposite pair {o1,o2}, that term equals
// -Re[a_m * g a_p conj(a_o1) conj(a_o2)] whichever pair m is in, so the
// local field h_m = sum over m's quartets of g a_p conj(a_o1 a_o2) gives
// every energy change of site m alone as -Re[da_m h_m].  2-body terms fold
// in with p = o1 = N, a virtual site whose amplitude is 1.
//
// Dense tiles.  When every quartet is active in channel 0, a quartet enters
// site m's field as g a_p conj(a_outer) conj(a_inner) with a contiguous range
// of inner sites shared by every partner p of one outer site: if m is among
// the two smallest sites of the quartet, outer = o1 > m, p < o1 and inner in
// (o1, N); otherwise outer = o2 < m, p > o2 and inner in [0, o2).  Under a
// frequency mask the inner sites of a group lie in an interval that moves
// slowly with o1 (the sites are sorted by frequency), so neighbouring groups
// of one partner overlap.  Either way a tile holds several groups as columns
// over one inner range (layout.cpp), so one gathered a_inner feeds 8 or 16 FMA.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pspin {

constexpr int kSplit = 32;        // parts per site list (warps per unit divide it)
constexpr int kGroupMax = 32;     // max data entries after one header
constexpr int kStage = 256;       // max entries per TMA chunk (2 KB)
constexpr int kStages = 3;        // chunks in flight per warp (set-up's limit on N)
constexpr int kRepBlock = 32;     // replicas per unit (one per lane)

// Status word bits raised by the sweep kernels.  A CTA (or cluster) whose
// bounded wait ran out stops issuing copies, drains the copies in flight,
// and leaves its replicas' amplitudes, energies and counters as they were
// before the launch.
constexpr int kStatusTimeout = 1;          // a ring wait ran out; the block aborted the launch
constexpr int kStatusDrain = 2;            // the drain of in-flight copies ran out as well
constexpr long long kWaitClocks = 1ll << 31;   // default ring-wait limit (~1 s at 1.9 GHz)
constexpr long long kDrainClocks = 1ll << 31;  // drain limit after an abort

struct SampleDev {
    int N;
    int R;                 // replicas of this sample
    int h2_active;
    int variant;           // 0 sphere (dense), 1 smoothed cube (sparse)
    int tiles;             // 1: site lists are dense tiles (layout.cpp), 0: group records
    int tiles_g;           // the same of the two-pass sweep's site lists (else groups)
    int tiles_p;           // the same of its pair sub-lists (else groups)
    int single_groups;     // group records only, every group of one entry (each record ends its group)
    int64_t spin_off;      // float2 index of site 0, replica 0
    int64_t rep_off;       // index into the per-replica arrays
    int64_t split_off;     // index into site chunks (N*33 entries)
    int64_t q_off;         // index into the Q64 table
    int64_t nq;            // active (quartet, channel) pairs in the Q64 table
    int64_t g2_off;        // index into g2 (N*N doubles)
    int64_t pair_off;      // index into the pair sub-list chunks (N(N-1)*33 entries), -1: not built
    int64_t nb_off;        // index into the neighbour masks (N rows of ceil(N/32) words)
    uint32_t pair_key0, pair_key1;
};

struct Unit {              // one replica block: a CTA, or a cluster of CTAs
    int sample;
    int rep_begin;
    int rep_count;         // <= 32 (32K with K replicas per lane)
    int pad;
};

struct Q64 {               // FP64 quartet for the resync energies
    uint16_t i, j, k, lch; // lch = l | ch << 14
    double g;
};

struct SweepParams {
    const SampleDev* samples;
    const Unit* units;
    float2* spins;
    double* energy;
    long long* accepted;
    long long* proposed;
    const double* beta;
    const uint64_t* key;
    const int2* entries;
    const int64_t* chunk_start;
    const int* site_chunks;
    const int* pair_chunks;           // pair sub-lists (two-pass proposals), or null
    const int* site_chunks_g;         // the site lists in the group format (two-pass proposals;
                                      // tiles unchanged), same per-sample offsets as site_chunks
    const uint32_t* nbmask;           // per sample: row m = sites sharing a quartet (or a g2 term) with m
    const long long* sweep_counter;   // global sweep index at launch start
    int nsweeps;
    int warps;                        // block shape: warps per CTA (divides 32) ...
    int cluster;                      //   ... and CTAs per unit, which fix the summation order of the fields
    int exec, chains, stages, max_N;  // sweep_ring_kernel: the RingPlan the launch runs with, its largest N
    // trace
    int trace_sample, trace_rep, trace_cap;
    long long trace_sweep0;
    void* trace;                      // pspin_move_record*
    int* status;                      // error word (kStatus* bits)
    long long wait_clocks;            // ring-wait limit in SM clocks
    int stall_move;                   // tests: move index of the stall wait (-1: none)
    long long patience;               // sweep_resident_kernel: limit of its waits for other moves and blocks,
                                      //   beyond any that is set for copies (tests: wait_clocks)
    // sweep_ring_kernel, launches of more than one task per unit: tasks of `chunk`
    // sweeps (the last one the rest of nsweeps), taken in order from *queue; done[u]:
    // tasks of unit u that are finished (-1: it aborted)
    int n_units, chunk;
    int* queue;                       // null: one task, block b runs unit b / exec
    int* done;
    // what a unit's tasks hand to its next one (null without a queue): a unit that
    // aborts keeps the arrays below and above as they were before the launch
    float2* mid_spins;
    double* mid_energy;
    long long *mid_accepted, *mid_proposed;
    double* mid_beta;                 // ... with PT steps inside the launch
    int* mid_perm;
    unsigned long long* mid_drand;
    long long *mid_ex_acc, *mid_ex_prop;
    // PT steps inside the launch (pt_freq > 0; every unit a whole sample):
    // exchange after every pt_freq sweeps
    int pt_freq, NT, nrep;
    const double* beta_sched;         // [NT]
    double* beta_out;                 // = beta
    int* perm;                        // [S][NT*nrep]
    unsigned long long* drand_state;  // [S]
    long long* ex_acc;                // [S][NT-1]
    long long* ex_prop;
    // sweep_resident_kernel: the prepared parts of a launch's moves
    int prep_stride;                  // moves per sample and unit
    int4* prep_moves;                 // [S][prep_stride]
    float* prep_trig;                 // [units][prep_stride][7][32]
};

// Shared memory that one replica block of a sample needs at least: the limit
// on N at set-up (amplitudes, per-warp field partials, rings and barriers).
inline size_t sweep_smem_bytes(int N, int warps) {
    return (size_t)(N + 1) * kRepBlock * sizeof(float2) + (size_t)warps * kRepBlock * sizeof(float4) +
           (size_t)warps * kStages * kStage * sizeof(int2) + (size_t)warps * kStages * sizeof(uint64_t);
}

// How sweep_ring_kernel spreads a unit's chains: over exec CTAs of `chains`
// chain warps, each with a ring of `stages` chunks; lat: the form for few
// units; resident: units that run at once.
struct RingPlan {
    int exec, chains, stages, lat, resident;
};
constexpr size_t kRingSmemMax = 227 * 1024 - 64;   // (the kernel's static shared memory)
// whether any spread of the block shape's chains has the shared memory it needs
bool ring_shape_fits(int warps, int cluster, int max_N, int K);
// pt_slots: replicas per unit that exchange inside the launch (0: none)
bool plan_sweep_ring(RingPlan& r, int warps, int cluster, int n_units, int variant, int max_N, int K, int pt_slots);

// kernels (launchers are host functions in the .cu files)
// units of up to 32K replicas, K = 1, 2, 3 replicas per lane
cudaError_t launch_sweep_ring(const SweepParams& p, const RingPlan& r, int n_units, int variant, int max_N, int K,
                              int pt_slots, cudaStream_t st);
// How the two-pass sweep spreads a unit's chains: `chains` of them on each of exec
// CTAs; one: every CTA has an SM to itself; grouped: the CTAs exchange sums of the
// shape's CTAs.
struct LearnPlan {
    int exec, chains, one, grouped;
};
bool plan_learned_sweep(LearnPlan& r, int warps, int cluster, int n_units, int max_N);
// the list-resident kernel; warps > 1 runs moves that commute (no site of one in
// the other's quartet neighbourhood, by the neighbour masks `nbmask`) at once, on
// clusters of p.exec units; pt_slots: replicas that exchange inside the launch;
// batched: the form for many blocks (without exchanges, and nothing prepared)
cudaError_t launch_sweep_resident(const SweepParams& p, int n_units, int variant, int max_N, int64_t max_entries,
                                  int pt_slots, bool batched, cudaStream_t st);
enum { kBatchedNever, kBatchedShort, kBatchedAlways };
constexpr int kShortLaunch = 64;      // moves
int resident_batched(int n_units, int variant, int max_N, int64_t max_entries, int warps, int pt_slots);
size_t resident_smem_bytes_host(int N, int64_t entries, int warps, int pt_slots);

struct EnergyParams {
    const SampleDev* samples;
    const Unit* units;
    float2* spins;
    const Q64* quartets;
    const double* g2;
    double* e2;               // may be null
    double* e4;               // may be null
    double* energy;           // when non-null: running energy <- e2+e4, drift recorded
    double* drift;            // |E_running - E_fp64| before the overwrite (when energy set)
    const double* target;     // constraint target per replica (renormalise when non-null)
    int renorm_only;          // 1: renormalise and return (energies come from elsewhere)
    double* partial;          // [n_units][max_pieces][32][2]: (e2, e4) of each piece of the tables
    int max_pieces;           // most pieces of a sample's table
    int max_ctas, n_units;    // most CTAs per unit, units (set at the launch)
};
int energy_max_pieces(int64_t max_nq);
size_t energy_partial_doubles(int n_units, int max_pieces);
cudaError_t launch_energy(const EnergyParams& p, int n_units, int max_N, cudaStream_t st);

struct ExchangeParams {
    int n_samples;
    int NT, nrep;             // per sample
    const SampleDev* samples;
    const double* beta_sched; // [NT]
    const double* energy;
    double* beta;
    int* perm;                // [S][NT*nrep]
    unsigned long long* drand_state; // [S]
    long long* ex_acc;        // [S][NT-1]
    long long* ex_prop;
    long long* sweep_counter; // advanced by nsweeps_done
    int nsweeps_done;
    int do_exchange;
};
cudaError_t launch_exchange(const ExchangeParams& p, cudaStream_t st);

// Observable series at one temperature slot, written after each exchange
// step at row (sweep_counter - sweep0) / pt_freq - 1 (device counter, so a
// captured launch records into the right row).
struct ObserveParams {
    int n_samples, NT, nrep, temp_index, capacity, pt_freq;
    const SampleDev* samples;
    const float2* spins;
    const double* energy;
    const int* perm;
    const long long* sweep_counter;
    long long sweep0;
    double* E_out;            // [capacity][S][nrep]
    double* q_out;            // [capacity][S][nrep*(nrep-1)/2]
};
cudaError_t launch_observe(const ObserveParams& p, cudaStream_t st);

}  // namespace pspin
