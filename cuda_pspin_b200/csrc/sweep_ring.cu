// sweep_ring.cu -- the plain pair-rotation Metropolis sweep (dense sphere and
// sparse cube) with the site lists streamed through shared memory.
//
// Replaces mc_sweep_kernel (mc.cu:66-318) and mc_sparse_sweep_kernel
// (mc_sparse.cu:63-253).  Same move set, same Metropolis rule; different
// organisation:
//
//  * One unit = up to 32K replicas of one sample (K = 1, 2, 3): lane l holds
//    replicas l, 32 + l, 64 + l of the unit, amplitudes [site][K][32] float2.
//    All replicas of a sample propose on the same pair at the same step (the
//    pair stream belongs to the sample, not to the replica), so a staged
//    coupling, one broadcast shared-memory read, serves the lane's K replicas.
//    Pair choice does not depend on the state, so every replica still runs a
//    random-scan Metropolis chain with the reference's stationary law.
//  * dE from local fields.  E is affine in a_i for fixed other sites, so
//      E(a_i',a_j') - E(a_i,a_j) = -Re[da_i h_i(a_j')] - Re[da_j h_j(a_i)]
//    exactly, where h_i(a_j') is site i's field evaluated with the proposed
//    a_j, which therefore sits in j's slot during the field pass.
//  * Summation tree.  A list is cut in 32 balanced parts; with W warps per CTA
//    and C CTAs per block (the block shape of the options) a list has C*W
//    chains of 32/(C*W) consecutive parts, each summed in list order, then the
//    chains of a CTA in order, then the CTAs in order.  The shape fixes that
//    order, hence the chain of states; how the 2*C*W chains of a move (two
//    lists) are spread over the machine does not.
//  * A move's 2*C*W chains run on X CTAs (a thread-block cluster for X > 1),
//    one warp per chain, so the two lists of a move are read at once.  The
//    remaining warps of a CTA are K deciders and one producer:
//      producer: lane l follows chain l through the (state-independent) pair
//        schedule and keeps its ring of TMA copies (cp.async.bulk, one mbarrier
//        per slot) full, moves ahead of the readers; no chain warp looks
//        anything up;
//      chain warp: reads its chunks, leaves its partial field of each replica in
//        the CTA's shared memory, then waits for the CTA's deciders;
//      decider k: while the chains run, the random words, sines and cosines of
//        the next move for its 32 replicas; when the CTA's chains have arrived,
//        their sums (of the tree's groups that lie in this CTA whole, else the
//        partials as they are) go to every CTA of the unit (st.async, counted in
//        bytes on the receiving decider's mbarrier); when all have come, the rest
//        of the tree, the Metropolis decision, the next proposal, and both into
//        its CTA's copy of the amplitudes.
//    Every CTA's decider k takes the same decision on the same numbers, so the
//    copies agree and a move costs one hop between CTAs and two barriers in one.
//    (Every chain sending its partial to all CTAs: 64 partials of 256 bytes into
//    each of 16 CTAs and 4000 cycles to sum them at N=32.)
//    With every warp deciding for itself and fetching its own chunks (8 warps
//    reading list i, then list j), the benchmark's launch ran the FMA pipe at
//    37 % and a move of a one-sample run cost 8 us of waiting.
//  * A launch may hold several tasks per unit (chunks of sweeps, taken in order
//    from a queue, so that units of uneven size pack onto the SMs without a
//    barrier per sweep) and, where every unit is a whole sample, the replica
//    exchange after every pt_freq sweeps: every CTA's deciders exchange on their
//    own copy of the energies and the permutation, behind the chains' pass of the
//    next move.
//  * All waits are bounded; a chain whose copy does not arrive sends a marked
//    partial, so every CTA of the unit leaves at the same move, and nothing is
//    written back: a unit's tasks but the last hand their state on in arrays of
//    their own.
//  * FP32 amplitudes and fields; the running energy is FP64.
#include <algorithm>

#include "exchange.cuh"
#include "sweep_common.cuh"
#include "../../include/pspin.h"

namespace pspin {

constexpr int kMaxChains = 16;            // chain warps per CTA
constexpr int kLatChains = 4;             // up to here a CTA is one chain per SM sub-partition
// A CTA one of whose chains gave up sends this NaN, which no arithmetic here
// produces, in place of its messages.
constexpr uint32_t kAbortMark = 0x7fc0dead;
__device__ __forceinline__ bool is_marked(const float2 v) { return __float_as_uint(v.x) == kAbortMark; }

// Shared memory of one CTA: amplitudes [N+1][K][32] float2; rings
// [chains][stages][kStage] int2; the chains' partials [chains][K][32] float2;
// exchange buffer [2][messages][K][32] float2 (messages: see ring_messages);
// mbarriers full, empty [chains][stages], chains' arrival, messages [2][K],
// deciders' meeting; ring
// tags [chains][stages] int2; with exchanges in the launch (pt_slots replicas),
// energies by replica, energies by slot, betas by replica, schedule, drand48
// states [pt_slots] of 8 bytes each, replicas by slot, swap counts [pt_slots] int
// each.
struct RingLayout {
    size_t ring, part, xbuf, bars, tags, pt, total;
};
// What a unit's CTAs exchange per move: the sums of the tree's 2*C groups of W
// chains where a CTA holds whole groups, else the 2*C*W chains.
__host__ __device__ inline int ring_messages(int warps, int cluster, int chains) {
    return chains % warps == 0 ? 2 * cluster : 2 * cluster * warps;
}
__host__ __device__ inline RingLayout ring_layout(int N, int warps, int cluster, int chains, int stages, int K,
                                                  int pt_slots) {
    RingLayout L;
    const size_t row = (size_t)K * kRepBlock * sizeof(float2);
    L.ring = (size_t)(N + 1) * row;
    L.part = L.ring + (size_t)chains * stages * kStage * sizeof(int2);
    L.xbuf = L.part + (size_t)chains * row;
    // one CTA holds every group: nothing is exchanged
    const bool alone = chains == 2 * cluster * warps;
    L.bars = L.xbuf + (alone ? 0 : (size_t)2 * ring_messages(warps, cluster, chains) * row);
    L.tags = L.bars + (size_t)(2 * chains * stages + 2 + 2 * K) * sizeof(uint64_t);
    L.pt = L.tags + (size_t)chains * stages * sizeof(int2);
    L.total = L.pt + (size_t)pt_slots * (5 * sizeof(double) + 2 * sizeof(int));
    return L;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// named barrier 1: deciders arrive, chain warps wait ("the state of the next move is in place")
__device__ __forceinline__ void state_arrive(int threads) {
    asm volatile("bar.arrive 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ void state_wait(int threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// named barrier 2: chain warps and deciders arrive as they leave a task, the producer waits
__device__ __forceinline__ void left_arrive(int threads) {
    __syncwarp();
    asm volatile("bar.arrive 2, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ void left_wait(int threads) {
    __syncwarp();
    asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory");
}

// Partial fields from buf[q * group + w * stride] in tree order: a CTA's W
// chains, then the C CTAs.  Eight loads in flight before their additions.
// `ok` is cleared where a value is marked.
template <int W>
__device__ __forceinline__ float2 tree_sum_w(const float2* __restrict__ buf, int C, int stride, int group, bool& ok) {
    constexpr int G = 8 / W;
    float2 h = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int q0 = 0; q0 < C; q0 += G) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            v[u] = make_float2(0.f, 0.f);
            if (u < W || q0 + u / W < C) v[u] = buf[(q0 + u / W) * group + (u % W) * stride];
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            float2 p = v[g * W];
            ok = ok && !is_marked(p);
#pragma unroll
            for (int w = 1; w < W; w++) {
                p.x += v[g * W + w].x;
                p.y += v[g * W + w].y;
                ok = ok && !is_marked(v[g * W + w]);
            }
            if (q0 + g == 0) h = p;
            else if (q0 + g < C) {
                h.x += p.x;
                h.y += p.y;
            }
        }
    }
    return h;
}
__device__ __forceinline__ float2 tree_sum(const float2* __restrict__ buf, int C, int W, int stride, int group, bool& ok) {
    switch (W) {
        case 1: return tree_sum_w<1>(buf, C, stride, group, ok);
        case 2: return tree_sum_w<2>(buf, C, stride, group, ok);
        case 4: return tree_sum_w<4>(buf, C, stride, group, ok);
        default: return tree_sum_w<8>(buf, C, stride, group, ok);
    }
}

// One exchange by a warp, on the arrays that start at pt_E (RingLayout): energies by
// replica in, betas by replica out; returns the drand48 state.  Not inlined: its
// registers are not the sweep's.
__device__ __noinline__ uint64_t ring_exchange(double* pt_E, int RT, int NT, int nrep, uint64_t drand) {
    const int lane = threadIdx.x & 31;
    double *Es = pt_E + RT, *beta = Es + RT, *sched = beta + RT;
    uint64_t* seq = reinterpret_cast<uint64_t*>(sched + RT);
    int *slot = reinterpret_cast<int*>(seq + RT), *swaps = slot + RT;
    for (int i = lane; i < RT; i += 32) Es[i] = pt_E[slot[i]];
    __syncwarp();
    if (nrep <= 32)
        exchange_columns(slot, Es, sched, seq, NT, nrep, drand, [&](int t, int n) { swaps[t] += n; });
    else
        exchange_pass(slot, sched, NT, nrep, drand, [&](int i, int) { return Es[i]; },
                      [&](int i, int j, double Ei, double Ej) {
                          Es[i] = Ej;
                          Es[j] = Ei;
                      },
                      [&](int t, int n) { swaps[t] += n; });
    for (int i = lane; i < RT; i += 32) beta[slot[i]] = sched[i / nrep];
    if (nrep <= 32) drand_ahead(seq, (NT - 1) * nrep, drand);        // for the next one
    return drand;
}

// whether the task whose first sweep is `first` is a unit's last one
__device__ __forceinline__ bool last_task(const SweepParams& P, int first) {
    return P.queue == nullptr || P.nsweeps - first <= P.chunk;
}

// kLat: few blocks, at most kLatChains chain warps a CTA, so a warp has its
// sub-partition's issue slots and registers to itself and deep batches of
// loads in flight carry it; otherwise 16 chain warps share the SM.
template <int VARIANT, int K, bool kLat>
__global__ void __launch_bounds__(((kLat ? kLatChains : kMaxChains) + K + 1) * 32, 1)
    sweep_ring_kernel(const SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int X = P.exec, c = P.chains, stages = P.stages;
    const uint32_t rank = X > 1 ? cluster_rank() : 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int CW = P.cluster * P.warps;
    constexpr int KB = K * kRepBlock;
    // one layout for every unit of the launch (the barriers live through it)
    const RingLayout Lo = ring_layout(P.max_N, P.warps, P.cluster, c, stages, K, P.pt_freq > 0 ? P.NT * P.nrep : 0);
    float2* sp = reinterpret_cast<float2*>(smem_raw);
    float2* part = reinterpret_cast<float2*>(smem_raw + Lo.part);
    float2* xbuf = reinterpret_cast<float2*>(smem_raw + Lo.xbuf);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + Lo.bars);
    uint64_t* empty = full + c * stages;
    uint64_t* cbar = empty + c * stages;
    uint64_t* xbar = cbar + 1;
    uint64_t* dbar = xbar + 2 * K;
    int2* tags = reinterpret_cast<int2*>(smem_raw + Lo.tags);
    const int RT = P.pt_freq > 0 ? P.NT * P.nrep : 0;
    double* pt_E = reinterpret_cast<double*>(smem_raw + Lo.pt);      // [RT] by replica
    double* pt_beta = pt_E + 2 * RT;                                  // [RT] by replica (between: by slot)
    double* pt_sched = pt_beta + RT;                                  // [NT]
    uint64_t* pt_seq = reinterpret_cast<uint64_t*>(pt_sched + RT);    // [RT]
    int* pt_slot = reinterpret_cast<int*>(pt_seq + RT);               // [RT]
    int* pt_swaps = pt_slot + RT;                                     // [NT]
    __shared__ volatile int stop, gave_up;           // the unit aborts; a chain of this CTA gave up
    __shared__ volatile int task_s, first_s;         // the task, its first sweep
    __shared__ __align__(8) uint64_t stall_bar;      // test hook: nothing arrives on it

    if (threadIdx.x == 0) {
        for (int q = 0; q < 2 * c * stages; q++) mbar_init(full + q, 1);
        mbar_init(cbar, (uint32_t)c);                // every chain of the CTA
        for (int q = 0; q < 2 * K; q++) mbar_init(xbar + q, 1);   // bytes, armed by the decider
        mbar_init(dbar, (uint32_t)K);
        mbar_init(&stall_bar, 1);
        stop = gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_shared();
    }
    const long long sweep_base = *P.sweep_counter;
    const int state_threads = (c + K) * 32;
    const bool decider = warp >= c && warp < c + K;
    const int k = warp - c;                          // decider's replica group
    const int rr = k * kRepBlock + lane;
    const long long limit = 2 * P.wait_clocks + kDrainClocks;   // beyond any chain's own bounded wait
    const int n_tasks = P.queue ? P.n_units * ((P.nsweeps - 1) / P.chunk + 1) : 1;
    // over all tasks: ring position, moves and deciders' meetings so far
    uint32_t slot = 0, phase = 0, issued = 0, moves = 0, meetings = 0;
    if (X > 1) cluster_sync();                       // every CTA of the cluster runs before the first remote store

    for (;;) {
    // ---- the next task: unit, first sweep, sweeps
    int unit = (int)blockIdx.x / X, first = 0, nsweeps = P.nsweeps, task = 0;
    if (P.queue) {
        if (rank == 0 && threadIdx.x == 0) {
            int t;
            for (;;) {
                t = atomicAdd(P.queue, 1);
                if (t >= n_tasks) break;
                // the unit's earlier tasks were taken earlier, by clusters that run
                const volatile int* done = P.done + t % P.n_units;
                const long long t0 = clock64(), most = limit * P.chunk * (P.max_N / 2);   // every move of a task bounded
                int d;
                while ((d = *done) >= 0 && d < t / P.n_units && clock64() - t0 < most) __nanosleep(200);
                if (d >= t / P.n_units) break;
                if (d >= 0) atomicOr(P.status, kStatusTimeout);
                // the unit has aborted: its later tasks are dropped
            }
            __threadfence();
            for (int q = 0; q < X; q++) {
                if (X > 1) st_cluster_u32((const void*)&task_s, (uint32_t)q, (uint32_t)t);
                else task_s = t;
            }
        }
        if (X > 1) cluster_sync();
        else __syncthreads();
        task = task_s;
        if (task >= n_tasks) break;
        unit = task % P.n_units;
        first = task / P.n_units * P.chunk;
        nsweeps = min(P.chunk, P.nsweeps - first);
    }
    const Unit U = P.units[unit];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    // a unit's first task reads the engine's state and its last one writes it
    const bool head = first == 0;
    if (threadIdx.x == 0) first_s = first;
    // amplitudes, energies and betas may have been written by another SM earlier in this launch: read past L1
    load_block_amplitudes(sp, (head ? P.spins : P.mid_spins) + S.spin_off + U.rep_begin, R, N, KB, U.rep_count);   // column k*32 + lane
    for (int idx = threadIdx.x; idx < KB; idx += blockDim.x) sp[(size_t)N * KB + idx] = make_float2(1.f, 0.f);
    const long long sweep0 = sweep_base + first;
    const int steps = N / 2, total = nsweeps * steps;
    const int per_exchange = P.pt_freq * steps;      // moves between exchanges (0: none)
    const bool active = decider && rr < U.rep_count;
    const int64_t gr = S.rep_off + U.rep_begin + rr;

    // the deciders' pending move
    double E = 0.0, beta_d = 0.0;
    float beta = 0.f, cu = 0.f;
    int nacc = 0, nprop = 0, ci0 = 0, cj0 = 0;
    uint32_t k0 = 0, k1 = 0;
    float2 cai = make_float2(0.f, 0.f), caj = cai, cain = cai, cajn = cai;
    float tt[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto pair_of = [&](int m, int& i0, int& j0) {
        pair_pick(S.pair_key0, S.pair_key1, (uint64_t)(sweep0 + m / steps), (uint32_t)(m % steps), N, i0, j0);
    };
    auto draw = [&](int m) {
        move_trig<VARIANT>(move_words(k0, k1, (uint64_t)(sweep0 + m / steps), (uint32_t)(m % steps)), tt);
    };
    auto amp = [&](int site) -> float2& { return sp[(site * K + k) * kRepBlock + lane]; };
    uint64_t drand = 0;
    if (active) {
        beta_d = __ldcg((head || per_exchange == 0 ? P.beta : P.mid_beta) + gr);
        beta = (float)beta_d;
        const uint64_t key = P.key[gr];
        k0 = (uint32_t)key;
        k1 = (uint32_t)(key >> 32);
        E = __ldcg((head ? P.energy : P.mid_energy) + gr);
    }
    if (decider && k == 0 && per_exchange > 0) {
        const int* perm = (head ? P.perm : P.mid_perm) + (int64_t)U.sample * RT;
        for (int i = lane; i < RT; i += 32) pt_slot[i] = __ldcg(perm + i);
        for (int t = lane; t < P.NT; t += 32) {
            pt_sched[t] = P.beta_sched[t];
            pt_swaps[t] = 0;
        }
        drand = __ldcg((head ? P.drand_state : P.mid_drand) + U.sample);
        if (P.nrep <= 32) drand_ahead(pt_seq, (P.NT - 1) * P.nrep, drand);
    }
    __syncthreads();
    if (decider && total > 0) {
        pair_of(0, ci0, cj0);
        draw(0);
        cai = amp(ci0);
        caj = amp(cj0);
        propose_with<VARIANT>(cai, caj, tt, cain, cajn);
        cu = tt[6];
        amp(cj0) = cajn;                             // h_i is evaluated at the proposed a_j
    }
    __syncthreads();

    if (warp < c) {
        // ------------------------------------------------------------ chain warp
        float2* mine = part + (size_t)warp * KB + lane;
        uint64_t* fb = full + warp * stages;
        uint64_t* eb = empty + warp * stages;
        const int2* tg = tags + warp * stages;
        const int2* ring = reinterpret_cast<const int2*>(smem_raw + Lo.ring) + (size_t)warp * stages * kStage;
        for (int m = 0; m < total; m++) {
            if (m > 0) {
                __syncwarp();
                state_wait(state_threads);
                if (__any_sync(0xffffffffu, stop != 0)) break;
            }
            float hx[K], hy[K];
#pragma unroll
            for (int q = 0; q < K; q++) hx[q] = hy[q] = 0.f;
            bool ok = true;
            // test hook, in a unit's last task
            if (m == P.stall_move && last_task(P, first_s)) ok = stall_wait(&stall_bar, P.status, P.wait_clocks);
            for (bool last = false; ok && !last;) {
                ok = ring_wait(fb + slot, phase, P.status, P.wait_clocks);
                if (!ok) break;
                const int2 t = tg[slot];             // {entries, last chunk of this move}
                const int2* chunk = ring + slot * kStage;
                last = t.y != 0;
                if (K == 1 && kLat) {
                    if (S.tiles) accumulate_tiles<K, 8, 4, true>(chunk, t.x, sp, lane, hx, hy);
                    else accumulate_records<4>(chunk, t.x, sp, lane, hx[0], hy[0]);
                } else {
                    if (S.tiles) accumulate_tiles<K, 2, 2, kLat>(chunk, t.x, sp, lane, hx, hy);
                    else accumulate_records_k<K>(chunk, t.x, sp, lane, hx, hy);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(eb + slot);
                if (++slot == (uint32_t)stages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
#pragma unroll
            for (int u = 0; u < K; u++)
                mine[u * kRepBlock] = make_float2(hx[u], hy[u]);
            if (!ok) gave_up = 1;
            __syncwarp();
            if (lane == 0) mbar_arrive(cbar);
        }
    } else if (decider) {
        // ------------------------------------------------------------ decider
        const int W = P.warps, C = P.cluster;
        const bool grouped = c % W == 0;
        const int msgs = ring_messages(W, C, c), local = grouped ? c / W : c;
        int to_exchange = per_exchange;
        bool lost = false;                           // a meeting with the other deciders failed
        for (int m = 0; m < total; m++, moves++) {
            const uint32_t par = moves & 1u;
            uint64_t* bar = xbar + par * K + k;
            if (X > 1 && lane == 0) mbar_expect_tx(bar, (uint32_t)(msgs * kRepBlock * sizeof(float2)));
            // the next move's draw, and its sites' amplitudes in the state the
            // chains are reading (move m's decision can change only ci0, cj0)
            int ni0 = 0, nj0 = 0;
            float2 nai = make_float2(0.f, 0.f), naj = nai;
            if (m + 1 < total) {
                pair_of(m + 1, ni0, nj0);
                nai = amp(ni0);
                naj = amp(nj0);
                draw(m + 1);
            }
            bool ok = __all_sync(0xffffffffu, mbar_wait(cbar, moves & 1u, P.status, limit) && gave_up == 0) && !lost;
            const float2* mine = part + k * kRepBlock + lane;
            int gw = W;                              // values per group still to be summed
            if (X > 1) {
                // this CTA's messages to every CTA
                const uint32_t dx = smem_u32(xbuf + ((par * msgs + rank * local) * K + k) * kRepBlock + lane);
                const uint32_t db = smem_u32(bar);
#pragma unroll 1
                for (int u = 0; u < local; u++) {
                    bool none = true;
                    float2 v = grouped ? tree_sum(mine + u * W * KB, 1, W, KB, 0, none) : mine[u * KB];
                    if (!ok) v.x = __uint_as_float(kAbortMark);
                    for (int q = 0; q < X; q++)
                        st_async_f2(map_rank(dx + u * (uint32_t)(KB * sizeof(float2)), (uint32_t)q), v,
                                    map_rank(db, (uint32_t)q));
                }
                // (a CTA that gives up, too, waits for what is on its way to it)
                const bool came = __all_sync(0xffffffffu, mbar_wait(bar, (moves >> 1) & 1u, P.status, limit));
                ok = ok && came;
                mine = xbuf + (par * msgs * K + k) * kRepBlock + lane;
                if (grouped) gw = 1;
            }
            const float2 hi = tree_sum(mine, C, gw, KB, 2 * gw * KB, ok);
            const float2 hj = tree_sum(mine + gw * KB, C, gw, KB, 2 * gw * KB, ok);
            if (!__all_sync(0xffffffffu, ok)) {      // every CTA of the unit reads the same marks
                stop = 1;
                __threadfence_block();
                __syncwarp();
                if (m + 1 < total) state_arrive(state_threads);
                break;
            }
            const float dix = __fsub_rn(cain.x, cai.x), diy = __fsub_rn(cain.y, cai.y);
            const float djx = __fsub_rn(cajn.x, caj.x), djy = __fsub_rn(cajn.y, caj.y);
            const float dE = -fmaf(dix, hi.x, -diy * hi.y) - fmaf(djx, hj.x, -djy * hj.y);
            // mc.cu:288-297: beta == 0 accepts everything; otherwise dE <= 0 or u < exp(-beta dE)
            bool accept;
            if (beta_d == 0.0) accept = true;
            else accept = (dE <= 0.f) || (cu < expf(-beta * dE));
            const float2 ai_post = accept ? cain : cai, aj_post = accept ? cajn : caj;
            if (rank == 0 && P.trace != nullptr && U.sample == P.trace_sample && U.rep_begin + rr == P.trace_rep &&
                active) {
                const long long idx = (sweep0 + m / steps - P.trace_sweep0) * steps + m % steps;
                if (idx >= 0 && idx < P.trace_cap) {
                    pspin_move_record* rec = reinterpret_cast<pspin_move_record*>(P.trace) + idx;
                    rec->i0 = ci0; rec->j0 = cj0;
                    rec->ai_old[0] = cai.x; rec->ai_old[1] = cai.y;
                    rec->aj_old[0] = caj.x; rec->aj_old[1] = caj.y;
                    rec->ai_new[0] = cain.x; rec->ai_new[1] = cain.y;
                    rec->aj_new[0] = cajn.x; rec->aj_new[1] = cajn.y;
                    rec->dE = dE;
                    rec->accepted = accept ? 1 : 0;
                    rec->log_q_ratio = 0.f;
                    rec->log_u = logf(cu);
                }
            }
            const int pi0 = ci0, pj0 = cj0;
            // the next proposal and the final values of the state it reads
            if (m + 1 < total) {
                cai = ni0 == pi0 ? ai_post : (ni0 == pj0 ? aj_post : nai);
                caj = nj0 == pi0 ? ai_post : (nj0 == pj0 ? aj_post : naj);
                ci0 = ni0;
                cj0 = nj0;
                propose_with<VARIANT>(cai, caj, tt, cain, cajn);
                cu = tt[6];
                amp(pi0) = ai_post;
                amp(pj0) = aj_post;
                amp(cj0) = cajn;                     // h_i of move m+1 is evaluated at its proposed a_j
                __syncwarp();
                state_arrive(state_threads);
            } else {
                amp(pi0) = ai_post;
                amp(pj0) = aj_post;
            }
            // bookkeeping, behind the chains' next pass
            if (accept) {
                E += (double)dE;
                nacc++;
            }
            nprop++;
            // the replica exchange, behind the chains' next pass (it changes only betas)
            if (per_exchange > 0 && --to_exchange == 0) {
                to_exchange = per_exchange;
                auto meet = [&]() {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dbar);
                    return __all_sync(0xffffffffu, mbar_wait(dbar, meetings++ & 1u, P.status, limit));
                };
                if (active) pt_E[rr] = E;
                bool met = meet();
                if (k == 0 && met) drand = ring_exchange(pt_E, RT, P.NT, P.nrep, drand);
                met = meet() && met;
                if (!met) {                          // a wait ran out: the next move's messages say so
                    lost = true;
                    if (m + 1 < total) gave_up = 1;
                    else stop = 1;
                } else if (active) {
                    beta_d = pt_beta[rr];
                    beta = (float)beta_d;
                }
            }
        }
    } else if (warp == c + K) {
        // ------------------------------------------------------------ producer: lane = chain of this CTA
        // chain g of the move: the groups alternate between the lists, group 2q
        // the W chains of CTA q of the tree in list i, 2q + 1 in list j
        const int g = (int)rank * c + lane, W = P.warps, list = (g / W) & 1;
        const bool mine = lane < c;
        const int part0 = (g / (2 * W) * W + g % W) * (kSplit / CW), part1 = part0 + kSplit / CW;
        const int* lists = P.site_chunks + S.split_off;
        int2* tg = tags + lane * stages;
        unsigned char* ring = smem_raw + Lo.ring + (size_t)lane * stages * kStage * sizeof(int2);
        int m = 0, cur = 0, end = 0;                 // the next copy: chunk cur of [cur, end) of move m
        int64_t b = 0, e = 0;
        auto open = [&]() {                          // move m's chunks
            int i0, j0;
            pair_of(m, i0, j0);
            const int* sc = lists + (list ? j0 : i0) * (kSplit + 1);
            cur = __ldg(sc + part0);
            end = __ldg(sc + part1);
        };
        auto bounds = [&]() {
            if (cur < end) {
                b = __ldg(P.chunk_start + cur);
                e = __ldg(P.chunk_start + cur + 1);
            }
        };
        bool more = mine && total > 0;
        if (more) {
            open();
            bounds();
        }
        while (__any_sync(0xffffffffu, more) && !__any_sync(0xffffffffu, stop != 0)) {
            bool did = false;
            if (more && (issued < (uint32_t)stages || mbar_test_wait(empty + lane * stages + slot, phase ^ 1u))) {
                uint64_t* fb = full + lane * stages + slot;
                if (cur < end) {
                    const uint32_t bytes = (uint32_t)((e - b) * sizeof(int2));
                    tg[slot] = make_int2((int)(e - b), cur + 1 == end);
                    mbar_expect_tx(fb, bytes);
                    bulk_g2s(ring + slot * kStage * sizeof(int2), P.entries + b, bytes, fb);
                    cur++;
                } else {                             // no entries in this chain's parts
                    tg[slot] = make_int2(0, 1);
                    mbar_arrive(fb);
                }
                issued++;
                if (++slot == (uint32_t)stages) {
                    slot = 0;
                    phase ^= 1u;
                }
                if (cur >= end) {
                    more = ++m < total;
                    if (more) open();
                }
                if (more) bounds();
                did = true;
            }
            if (!__any_sync(0xffffffffu, did)) __nanosleep(40);
        }
        // copies still in flight after an abort (each slot's last one): none may land
        // after the CTA has gone.  The producer may have issued its last copies long
        // before, so it looks once the other warps have left (an abort that another
        // CTA makes known later still finds every copy of this one read).
        left_wait(state_threads + 32);
        if (mine && stop)
            for (uint32_t q = 0; q < (uint32_t)stages && q < issued; q++) {
                const uint32_t i = issued - 1 - q;
                if (!mbar_wait(full + lane * stages + i % stages, (i / stages) & 1u, P.status, kDrainClocks, kStatusDrain)) break;
            }
        __syncwarp();
    }

    if (warp < c + K) left_arrive(state_threads + 32);
    if (X > 1 && stop && threadIdx.x == 0)           // a CTA that gave up takes its cluster with it
        for (int q = 0; q < X; q++) st_cluster_u32((const void*)&stop, (uint32_t)q, 1u);
    if (X > 1) cluster_sync();                       // every final write; no store may still target a CTA
    else __syncthreads();
    const bool good = stop == 0;
    if (rank == 0) {
        if (good) {
            const bool head = first_s == 0, tail = last_task(P, first_s);
            float2* spins = tail ? P.spins : P.mid_spins;
            for (int idx = threadIdx.x; idx < N * KB; idx += blockDim.x) {
                const int site = idx / KB, r = idx % KB;
                if (r < U.rep_count) spins[S.spin_off + (int64_t)site * R + U.rep_begin + r] = sp[idx];
            }
            if (active) {
                (tail ? P.energy : P.mid_energy)[gr] = E;
                const long long a = __ldcg((head ? P.accepted : P.mid_accepted) + gr);
                const long long b = __ldcg((head ? P.proposed : P.mid_proposed) + gr);
                __stcg((tail ? P.accepted : P.mid_accepted) + gr, a + nacc);
                __stcg((tail ? P.proposed : P.mid_proposed) + gr, b + nprop);
                if (per_exchange > 0) (tail ? P.beta_out : P.mid_beta)[gr] = beta_d;
            }
            if (decider && k == 0 && per_exchange > 0) {
                const int64_t at = (int64_t)U.sample * (P.NT - 1);
                int* perm = (tail ? P.perm : P.mid_perm) + (int64_t)U.sample * RT;
                for (int i = lane; i < RT; i += 32) perm[i] = pt_slot[i];
                for (int t = lane; t < P.NT - 1; t += 32) {
                    const long long a = __ldcg((head ? P.ex_acc : P.mid_ex_acc) + at + t);
                    const long long b = __ldcg((head ? P.ex_prop : P.mid_ex_prop) + at + t);
                    __stcg((tail ? P.ex_acc : P.mid_ex_acc) + at + t, a + pt_swaps[t]);
                    __stcg((tail ? P.ex_prop : P.mid_ex_prop) + at + t, b + (long long)(total / per_exchange) * P.nrep);
                }
                if (lane == 0) (tail ? P.drand_state : P.mid_drand)[U.sample] = drand;
            }
        }
        if (P.queue) {
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) atomicExch(P.done + unit, good ? task / P.n_units + 1 : -1);
        }
    }
    if (!P.queue || !good) break;
    __syncthreads();                                 // the write-back has read the amplitudes
    }   // tasks
    if (X > 1) cluster_sync();
}

template <int VARIANT, int K, bool kLat>
static cudaError_t ring_launch(const SweepParams& p, int n_units, size_t smem, cudaStream_t st, int* max_clusters) {
    auto kern = sweep_ring_kernel<VARIANT, K, kLat>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && p.exec > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(n_units * p.exec));          // (with a queue: the units that run at once)
    cfg.blockDim = dim3((unsigned)(32 * (p.chains + K + 1)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.exec;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.exec > 1 ? 1 : 0;
    if (max_clusters) {
        if (p.exec > 1) return cudaOccupancyMaxActiveClusters(max_clusters, kern, &cfg);
        int blocks = 0, sms = 0, dev = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, (int)cfg.blockDim.x, smem);
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        *max_clusters = blocks * sms;
        return e;
    }
    e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

static cudaError_t ring_dispatch(SweepParams p, const RingPlan& r, int n_units, int variant, int max_N, int K,
                                 int pt_slots, cudaStream_t st, int* max_clusters) {
    p.max_N = max_N;
    p.exec = r.exec;
    p.chains = r.chains;
    p.stages = r.stages;
    const size_t smem = ring_layout(max_N, p.warps, p.cluster, p.chains, p.stages, K, pt_slots).total;
    const bool lat = r.lat != 0;
#define PSPIN_RING(V, KK) (lat ? ring_launch<V, KK, true>(p, n_units, smem, st, max_clusters) \
                               : ring_launch<V, KK, false>(p, n_units, smem, st, max_clusters))
    if (variant == 0) return K == 1 ? PSPIN_RING(0, 1) : K == 2 ? PSPIN_RING(0, 2) : PSPIN_RING(0, 3);
    return K == 1 ? PSPIN_RING(1, 1) : K == 2 ? PSPIN_RING(1, 2) : PSPIN_RING(1, 3);
#undef PSPIN_RING
}

static bool ring_fits(int max_N, int warps, int cluster, int X, int stages, int K, int pt_slots) {
    return ring_layout(max_N, warps, cluster, 2 * cluster * warps / X, stages, K, pt_slots).total <= kRingSmemMax;
}

bool ring_shape_fits(int warps, int cluster, int max_N, int K) {
    if (warps < 1 || cluster < 1 || cluster > 16 || kSplit % (cluster * warps) != 0 || K < 1 || K > 3) return false;
    const int T = 2 * cluster * warps;
    for (int X = T > kMaxChains ? T / kMaxChains : 1; X <= 16 && X <= T; X *= 2)
        if (ring_fits(max_N, warps, cluster, X, 2, K, 0)) return true;
    return false;
}

// Spreads the 2*C*W chains of a unit's move over X CTAs.  16 chains fill an SM
// (four per sub-partition); with few units the chains go to more CTAs, down to
// one chain per sub-partition, as long as all clusters are resident at once: a
// launch that leaves SMs idle is bound by the time of one chain.  Three ring
// slots per chain where they fit, else two, else more CTAs.
bool plan_sweep_ring(RingPlan& r, int warps, int cluster, int n_units, int variant, int max_N, int K, int pt_slots) {
    if (warps < 1 || cluster < 1 || cluster > 16 || kSplit % (cluster * warps) != 0 || K < 1 || K > 3) return false;
    const int T = 2 * cluster * warps;
    SweepParams p{};
    p.warps = warps;
    p.cluster = cluster;
    auto resident = [&](int X, int stages, int lat) {
        if (X > 16 || X > T || T / X > kMaxChains || (lat && T / X > kLatChains)) return 0;
        if (!ring_fits(max_N, warps, cluster, X, stages, K, pt_slots)) return 0;
        const RingPlan q{X, T / X, stages, lat, 0};
        int n = 0;
        if (ring_dispatch(p, q, n_units, variant, max_N, K, pt_slots, nullptr, &n) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n;
    };
    const int x_fill = T > kMaxChains ? T / kMaxChains : 1;
    for (int stages = 3; stages >= 2; stages--)
        for (int X = 16; X >= 1; X /= 2)
            for (int lat = 1; lat >= 0; lat--)
                if (X <= T && (X <= T / kLatChains || X == x_fill) && resident(X, stages, lat) >= n_units) {
                    r = RingPlan{X, T / X, stages, lat, n_units};
                    return true;
                }
    for (int X = x_fill; X <= 16 && X <= T; X *= 2)
        for (int stages = 3; stages >= 2; stages--)
            if (const int n = resident(X, stages, 0)) {
                r = RingPlan{X, T / X, stages, 0, n};
                return true;
            }
    return false;
}

cudaError_t launch_sweep_ring(const SweepParams& p, const RingPlan& r, int n_units, int variant, int max_N, int K,
                              int pt_slots, cudaStream_t st) {
    if (n_units <= 0) return cudaSuccess;
    return ring_dispatch(p, r, p.queue ? std::min(n_units, r.resident) : n_units, variant, max_N, K, pt_slots, st,
                         nullptr);
}

}  // namespace pspin
