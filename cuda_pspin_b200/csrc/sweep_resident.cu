// sweep_resident.cu -- the plain pair-rotation sweep for samples whose whole
// set of site lists fits in shared memory next to the amplitudes (sparse
// samples: ~8 list entries per site).
//
// Same moves, RNG streams and Metropolis rule as the ring sweep.  The lists
// are copied into shared memory once per launch, so a move reads them
// without TMA copies; site m's list is the contiguous range of its chunks
// (groups or tiles never span chunks; the padding entry of an odd chunk is
// an empty group).
//
// Concurrent commuting moves (K > 1).  Move b does not commute with move a when
// one of b's sites is a site of a or shares a quartet (or a g2 term) with one:
// then b's proposal or fields would read an amplitude that a changes.  Moves that
// commute give the same result in either order, so a move may run as soon as the
// earlier moves it does not commute with are done, and the chain is the one-warp
// chain bit for bit; the running energy adds the moves' dE in move order.
//   resident_prepare_kernel, on all SMs, does what depends on no state for every
//     move of the launch: the pair, the earlier moves (of the last 31) it does not
//     commute with, and per replica the random words, sines and cosines;
//   K workers: worker w runs moves w, w + K, ... in order, each for the block's 32
//     replicas.  The next move's prepared parts are on their way while this one
//     runs; the records of both lists are in registers before the wait for the
//     earlier moves; after it only the amplitudes are gathered, the field, the
//     proposal and the decision follow side by side, and the move is published in
//     its slot of a ring of 32;
//   one warp keeps the running energy and counters and, where the launch holds PT
//     steps, exchanges replicas: the blocks of a sample are then a cluster whose
//     CTAs send each other their energies and exchange alike on their own copies.
// The longest chain of moves that wait for one another is ~70 of a sweep's 256 at
// N=512 with N selected quartets, so a sweep is that many moves' latency.  Windows
// of 32 moves prepared by the workers themselves, then cut in batches of
// consecutive commuting moves with a CTA barrier each, took 7500 cycles of
// preparation a window and 8.6 batches of 1950 cycles: 118 us a sweep launch and
// 25 us of exchange; now 89 us for both.  Where many blocks share the SMs those
// batches are the better form still, and run (resident_batched).
#include <climits>

#include "exchange.cuh"
#include "sweep_common.cuh"
#include "../../include/pspin.h"

namespace pspin {

constexpr int kRing = 32;     // move slots

// Shared memory: amplitudes [(N+1)][32] float2 ((N+1)*256 bytes, so the list
// entries that follow are 16-byte aligned: records and tiles are read as int4),
// the sample's list entries, site ranges [N] int2; then, with one warp, a window's
// pairs and (sweep, step) [32] int2 each and proposal parts [32][7][32] float; with
// more, the slots' dE [32][32] float, decisions and finished moves [32] int each,
// betas [32] double; with exchanges in the launch (R replicas), energies by replica
// of two exchanges, by slot, betas by replica, schedule, drand48 states [R] of 8
// bytes each, replicas by slot, swap counts [R] int each.
inline size_t resident_smem_bytes(int N, int64_t entries, int K, int R = 0) {
    size_t b = (size_t)(N + 1) * kRepBlock * sizeof(float2) + (size_t)entries * sizeof(int2) + (size_t)N * sizeof(int2);
    if (K == 1) return b + 2 * kRing * sizeof(int2) + (size_t)kRing * 7 * kRepBlock * sizeof(float);
    return b + (size_t)kRing * kRepBlock * sizeof(float) + 2 * kRing * sizeof(int) + kRepBlock * sizeof(double) +
           (size_t)R * (6 * sizeof(double) + 2 * sizeof(int));
}

// A finished move or block: its warp's writes, a __syncwarp, then the flag by one
// lane; a reader's lanes poll flags with plain loads, fence once (an acquire load
// per poll slowed the warps at work) and meet in a __syncwarp, since each lane goes
// on to read what others' flags stand for.
__device__ __forceinline__ int peek(const int* p) { return *(const volatile int*)p; }
__device__ __forceinline__ void publish(int* p, int v) {
    __threadfence_block();
    *(volatile int*)p = v;
}

// Fields of two sites from their record lists, four records of each at a time with
// all their loads in flight (a sparse site has ~4); the arithmetic of
// accumulate_records on each.
template <bool kSingle>
__device__ __forceinline__ void accumulate_two(const int4* __restrict__ A, int na, const int4* __restrict__ B, int nb,
                                               const float2* __restrict__ sp, int lane, float& hix, float& hiy,
                                               float& hjx, float& hjy) {
    float yix = 0.f, yiy = 0.f, yjx = 0.f, yjy = 0.f;
    const int n = max(na, nb);
#pragma unroll 1
    for (int r = 0; r < n; r += 4) {
        int4 q[8];
        float2 a[8], ap[8], ao[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int at = r + (u & 3);
            q[u] = make_int4(0, 0, 0, 0);
            if (u < 4 ? at < na : at < nb) q[u] = u < 4 ? A[at] : B[at];
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            a[u] = sp[q[u].y * kRepBlock + lane];
            ap[u] = sp[(q[u].z >> 16) * kRepBlock + lane];
            ao[u] = sp[(q[u].z & 0xFFFF) * kRepBlock + lane];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (r + u < na) record_step<kSingle>(q[u], a[u], ap[u], ao[u], yix, yiy, hix, hiy);
            if (r + u < nb) record_step<kSingle>(q[4 + u], a[4 + u], ap[4 + u], ao[4 + u], yjx, yjy, hjx, hjy);
        }
    }
}

// One warp: moves one after another, prepared in windows of 32.
template <int VARIANT>
__global__ void __launch_bounds__(32) sweep_resident_one_kernel(const SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Unit U = P.units[blockIdx.x];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x;
    const int* sc = P.site_chunks + S.split_off;
    const int64_t e0 = __ldg(P.chunk_start + __ldg(sc));
    const int64_t e1 = __ldg(P.chunk_start + __ldg(sc + (int64_t)(N - 1) * (kSplit + 1) + kSplit));
    float2* sp = reinterpret_cast<float2*>(smem_raw);
    int2* L = reinterpret_cast<int2*>(sp + (size_t)(N + 1) * kRepBlock);
    int2* rng_site = L + (e1 - e0);
    int2* picks = rng_site + N;
    int2* mk = picks + kRing;                                  // (sweep - sweep0, step) of each slot's move
    float* tr = reinterpret_cast<float*>(mk + kRing);          // [32][7][32]
    for (int m = threadIdx.x; m < N; m += blockDim.x) {
        const int64_t b = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1)));
        const int64_t e = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1) + kSplit));
        rng_site[m] = make_int2((int)(b - e0), (int)(e - e0));
    }
    load_block_range(L, P.entries + e0, e1 - e0);
    load_block_amplitudes(sp, P.spins + S.spin_off + U.rep_begin, R, N, kRepBlock, U.rep_count);
    sp[N * kRepBlock + lane] = make_float2(1.f, 0.f);   // virtual site

    const bool active = lane < U.rep_count;
    const int64_t gr = S.rep_off + U.rep_begin + lane;
    double E = 0.0, beta_d = 0.0;
    float beta = 0.f;
    long long nacc = 0, nprop = 0;
    uint32_t k0 = 0, k1 = 0;
    if (active) {
        beta_d = P.beta[gr];
        beta = (float)beta_d;
        const uint64_t key = P.key[gr];
        k0 = (uint32_t)key;
        k1 = (uint32_t)(key >> 32);
        E = P.energy[gr];
    }
    const long long sweep0 = *P.sweep_counter;
    const int steps = N / 2, total = P.nsweeps * steps;
    // moves [m0, m0 + n) of this lane's slot: pair, (sweep, step)
    auto pick = [&](int m) {
        int i0, j0;
        const int sw = m / steps, kk = m - sw * steps;
        pair_pick(S.pair_key0, S.pair_key1, (uint64_t)(sweep0 + sw), (uint32_t)kk, N, i0, j0);
        picks[m % kRing] = make_int2(i0, j0);
        mk[m % kRing] = make_int2(sw, kk);
    };
    // the state-independent part of move m's proposal, for this lane's replica
    auto draw = [&](int m) {
        float tt[7];
        const int sw = m / steps;
        move_trig<VARIANT>(move_words(k0, k1, (uint64_t)(sweep0 + sw), (uint32_t)(m - sw * steps)), tt);
#pragma unroll
        for (int q = 0; q < 7; q++) tr[((m % kRing) * 7 + q) * kRepBlock + lane] = tt[q];
    };
    // move m for this lane's replica: fields, decision, new amplitudes; its dE and
    // decision into rows 0 and 1 of its slot
    auto run_move = [&](int m, int2 pq) {
        const int t = m % kRing, i0 = pq.x, j0 = pq.y;
        float* mine = tr + t * 7 * kRepBlock + lane;
        float tt[7];
#pragma unroll
        for (int q = 0; q < 7; q++) tt[q] = mine[q * kRepBlock];
        const float2 ai = sp[i0 * kRepBlock + lane], aj = sp[j0 * kRepBlock + lane];
        const int2 ri = rng_site[i0], rj = rng_site[j0];
        float2 ain, ajn;
        propose_with<VARIANT>(ai, aj, tt, ain, ajn);
        const float cu = tt[6];
        sp[j0 * kRepBlock + lane] = ajn;       // h_i is evaluated at the proposed a_j
        float hix = 0.f, hiy = 0.f, hjx = 0.f, hjy = 0.f;
        if (S.tiles) {
            accumulate_tiles_1<8, 4, true>(L + ri.x, ri.y - ri.x, sp, lane, hix, hiy);
            accumulate_tiles_1<8, 4, true>(L + rj.x, rj.y - rj.x, sp, lane, hjx, hjy);
        } else {
            const int4* A = reinterpret_cast<const int4*>(L + ri.x);
            const int4* B = reinterpret_cast<const int4*>(L + rj.x);
            const int na = (ri.y - ri.x) >> 1, nb = (rj.y - rj.x) >> 1;
            if (S.single_groups) accumulate_two<true>(A, na, B, nb, sp, lane, hix, hiy, hjx, hjy);
            else accumulate_two<false>(A, na, B, nb, sp, lane, hix, hiy, hjx, hjy);
        }
        const float dix = __fsub_rn(ain.x, ai.x), diy = __fsub_rn(ain.y, ai.y);
        const float djx = __fsub_rn(ajn.x, aj.x), djy = __fsub_rn(ajn.y, aj.y);
        const float dE = -fmaf(dix, hix, -diy * hiy) - fmaf(djx, hjx, -djy * hjy);
        bool accept;
        if (beta_d == 0.0) accept = true;
        else accept = (dE <= 0.f) || (cu < expf(-beta * dE));
        if (accept) sp[i0 * kRepBlock + lane] = ain;
        else sp[j0 * kRepBlock + lane] = aj;
        mine[0] = dE;
        mine[kRepBlock] = accept ? 1.f : 0.f;
        if (P.trace != nullptr && U.sample == P.trace_sample && U.rep_begin + lane == P.trace_rep && active) {
            const int2 swk = mk[t];
            const long long idx = (long long)swk.x * steps + swk.y + (sweep0 - P.trace_sweep0) * steps;
            if (idx >= 0 && idx < P.trace_cap) {
                pspin_move_record* rec = reinterpret_cast<pspin_move_record*>(P.trace) + idx;
                rec->i0 = i0; rec->j0 = j0;
                rec->ai_old[0] = ai.x; rec->ai_old[1] = ai.y;
                rec->aj_old[0] = aj.x; rec->aj_old[1] = aj.y;
                rec->ai_new[0] = ain.x; rec->ai_new[1] = ain.y;
                rec->aj_new[0] = ajn.x; rec->aj_new[1] = ajn.y;
                rec->dE = dE;
                rec->accepted = accept ? 1 : 0;
                rec->log_q_ratio = 0.f;
                rec->log_u = logf(cu);
            }
        }
    };
    // the running energy and counters: moves [m0, m1) in move order
    auto account = [&](int m0, int m1) {
        for (int m = m0; m < m1; m++) {
            const float* of = tr + (m % kRing) * 7 * kRepBlock + lane;
            if (of[kRepBlock] != 0.f) {
                E += (double)of[0];
                nacc++;
            }
            nprop++;
        }
    };
    __syncthreads();

    for (int m0 = 0; m0 < total; m0 += kRing) {
        const int n = min(kRing, total - m0);
        if (lane < n) pick(m0 + lane);
        for (int t = 0; t < n; t++) draw(m0 + t);
        __syncwarp();
        for (int t = 0; t < n; t++) {
            run_move(m0 + t, picks[t]);
            __syncwarp();
        }
        account(m0, m0 + n);
        __syncwarp();
    }
    __syncwarp();
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        if (l < U.rep_count) P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l] = sp[idx];
    }
    if (active) {
        P.energy[gr] = E;
        P.accepted[gr] += nacc;
        P.proposed[gr] += nprop;
    }
}

// The prepared parts of one launch's moves (sweeps from *base on): per sample and
// move {i0 | j0 << 16, slots of the earlier moves it does not commute with, 1 when
// i0 and j0 share a term, 0}, per unit and move the proposal parts [7][32].
__global__ void __launch_bounds__(128) resident_prepare_kernel(const SweepParams P, int variant) {
    const Unit U = P.units[blockIdx.x];          // (more units than a grid's y can count)
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, steps = N / 2, total = P.nsweeps * steps;
    const int lane = threadIdx.x & 31;
    const int m = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (m >= total) return;
    const long long sweep0 = *P.sweep_counter;
    uint32_t k0 = 0, k1 = 0;
    if (lane < U.rep_count) {
        const uint64_t key = P.key[S.rep_off + U.rep_begin + lane];
        k0 = (uint32_t)key;
        k1 = (uint32_t)(key >> 32);
    }
    const int sw = m / steps;
    const U4 w = move_words(k0, k1, (uint64_t)(sweep0 + sw), (uint32_t)(m - sw * steps));
    float tt[7];
    if (variant == 0) move_trig<0>(w, tt);
    else move_trig<1>(w, tt);
    float* dst = P.prep_trig + ((size_t)blockIdx.x * P.prep_stride + m) * 7 * kRepBlock + lane;
#pragma unroll
    for (int q = 0; q < 7; q++) dst[q * kRepBlock] = tt[q];
    if (U.rep_begin != 0) return;
    // lane q: the last move before m in slot q; the lane of m's own slot: m
    const int t = m % kRing;
    const int mine = lane == t ? m : m - 1 - ((t - 1 - lane) & (kRing - 1));
    int i0 = 0, j0 = 1;
    if (mine >= 0) {
        const int s = mine / steps;
        pair_pick(S.pair_key0, S.pair_key1, (uint64_t)(sweep0 + s), (uint32_t)(mine - s * steps), N, i0, j0);
    }
    const int mi = __shfl_sync(0xffffffffu, i0, t), mj = __shfl_sync(0xffffffffu, j0, t);
    const int wpr = (N + 31) >> 5;
    const uint32_t* nbm = P.nbmask + S.nb_off;
    auto near = [&](int a, int b) { return a == b || ((__ldg(nbm + a * wpr + (b >> 5)) >> (b & 31)) & 1u); };
    const bool c = lane != t && mine >= 0 && (near(i0, mi) || near(i0, mj) || near(j0, mi) || near(j0, mj));
    const unsigned mask = __ballot_sync(0xffffffffu, c);
    if (lane == t)
        P.prep_moves[(size_t)U.sample * P.prep_stride + m] = make_int4(i0 | (j0 << 16), (int)mask, near(i0, j0) ? 1 : 0, 0);
}

constexpr int kHeld = 5;      // records of each list that a worker holds in registers

template <int VARIANT>
__global__ void __launch_bounds__((8 + 1) * 32) sweep_resident_kernel(const SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int X = P.exec;                      // CTAs per cluster: the blocks of a sample, or 1
    const Unit U = P.units[blockIdx.x];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = P.warps;                     // workers
    const int RT = P.pt_freq > 0 ? P.NT * P.nrep : 0;
    const int* sc = P.site_chunks + S.split_off;
    const int64_t e0 = __ldg(P.chunk_start + __ldg(sc));
    const int64_t e1 = __ldg(P.chunk_start + __ldg(sc + (int64_t)(N - 1) * (kSplit + 1) + kSplit));
    float2* sp = reinterpret_cast<float2*>(smem_raw);
    int2* L = reinterpret_cast<int2*>(sp + (size_t)(N + 1) * kRepBlock);
    int2* rng_site = L + (e1 - e0);
    double* beta_s = reinterpret_cast<double*>(rng_site + N);                 // [32]
    float* dEx = reinterpret_cast<float*>(beta_s + kRepBlock);                // [32][32]
    uint32_t* acx = reinterpret_cast<uint32_t*>(dEx + kRing * kRepBlock);     // [32]
    int* done = reinterpret_cast<int*>(acx + kRing);                          // [32] last move finished in each slot
    double* pt_E = reinterpret_cast<double*>(done + kRing);                   // [2][RT] by replica
    double* pt_Es = pt_E + 2 * RT;                                            // [RT] by slot
    double* pt_beta = pt_Es + RT;                                             // [RT] by replica
    double* pt_sched = pt_beta + RT;                                          // [RT]
    uint64_t* pt_seq = reinterpret_cast<uint64_t*>(pt_sched + RT);            // [RT]
    int* pt_slot = reinterpret_cast<int*>(pt_seq + RT);                       // [RT]
    int* pt_swaps = pt_slot + RT;                                             // [RT]
    __shared__ int counted, exchanged;                         // moves accounted for; exchanges made
    __shared__ volatile int stop;                              // a wait ran out
    __shared__ __align__(8) uint64_t ebar[2];                  // the cluster's energies, by exchange parity
    for (int m = threadIdx.x; m < N; m += blockDim.x) {
        const int64_t b = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1)));
        const int64_t e = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1) + kSplit));
        rng_site[m] = make_int2((int)(b - e0), (int)(e - e0));
    }
    load_block_range(L, P.entries + e0, e1 - e0);
    load_block_amplitudes(sp, P.spins + S.spin_off + U.rep_begin, R, N, kRepBlock, U.rep_count);
    const bool active = lane < U.rep_count;
    const int64_t gr = S.rep_off + U.rep_begin + lane;
    double beta_d = active ? P.beta[gr] : 0.0;
    float beta = (float)beta_d;
    if (threadIdx.x < kRepBlock) {
        sp[N * kRepBlock + threadIdx.x] = make_float2(1.f, 0.f);   // virtual site
        done[threadIdx.x] = -1;
        beta_s[lane] = beta_d;
    }
    if (threadIdx.x == 0) {
        counted = exchanged = 0;
        stop = 0;
        mbar_init(ebar, 1);
        mbar_init(ebar + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const long long sweep0 = *P.sweep_counter;
    const int steps = N / 2, total = P.nsweeps * steps;
    const int per_exchange = P.pt_freq * steps;
    double E = 0.0;
    long long nacc = 0, nprop = 0;
    uint64_t drand = 0;
    // until cond() holds, within a bound
    auto wait = [&](auto cond) {
        if (__all_sync(0xffffffffu, cond())) {
            __threadfence_block();
            __syncwarp();
            return true;
        }
        const long long t0 = clock64();
        for (;;) {
            if (__all_sync(0xffffffffu, cond())) {
                __threadfence_block();
                __syncwarp();
                return true;
            }
            const bool late = clock64() - t0 > P.patience;
            if (__any_sync(0xffffffffu, late || stop != 0)) {
                if (late) atomicOr(P.status, kStatusTimeout);
                stop = 1;
                return false;
            }
            __nanosleep(20);
        }
    };
    if (X > 1) cluster_sync();
    else __syncthreads();

    if (warp < K) {
        // ------------------------------------------------------------ worker
        const int4* moves = P.prep_moves + (size_t)U.sample * P.prep_stride;
        const float* trig = P.prep_trig + (size_t)blockIdx.x * P.prep_stride * 7 * kRepBlock + lane;
        int4 nmv = make_int4(0, 0, 0, 0);
        float ntt[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        auto fetch = [&](int m) {
            if (m >= total) return;
            // (volatile: issued here, a move ahead of their use)
            asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(nmv.x), "=r"(nmv.y), "=r"(nmv.z), "=r"(nmv.w)
                         : "l"(moves + m));
#pragma unroll
            for (int q = 0; q < 7; q++)
                asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(ntt[q]) : "l"(trig + ((size_t)m * 7 + q) * kRepBlock));
        };
        fetch(warp);
        int version = 0;                       // exchanges in this warp's betas
        for (int m = warp; m < total; m += K) {
            const int4 mv = nmv;
            float tt[7];
#pragma unroll
            for (int q = 0; q < 7; q++) tt[q] = ntt[q];
            fetch(m + K);
            const int t = m % kRing, i0 = mv.x & 0xFFFF, j0 = mv.x >> 16;
            const int2 ri = rng_site[i0], rj = rng_site[j0];
            const int4* A = reinterpret_cast<const int4*>(L + ri.x);
            const int4* B = reinterpret_cast<const int4*>(L + rj.x);
            const int na = (ri.y - ri.x) >> 1, nb = (rj.y - rj.x) >> 1;
            // record lists whose terms do not hold the partner site: the proposed
            // a_j is in none of them
            const bool quick = S.single_groups && mv.z == 0;
            int4 q[2 * kHeld];
            if (quick) {
#pragma unroll
                for (int u = 0; u < kHeld; u++) {
                    q[u] = q[kHeld + u] = make_int4(0, N, (N << 16) | N, 1);
                    if (u < na) q[u] = A[u];
                    if (u < nb) q[kHeld + u] = B[u];
                }
            }
            // the earlier moves it does not commute with, and every move a ring ago;
            // this slot's last dE is accounted for
            const int last = m - 1 - ((t - 1 - lane) & (kRing - 1));
            int need = ((uint32_t)mv.y >> lane) & 1u ? last : last - kRing;
            if (m == P.stall_move && (X == 1 || cluster_rank() + 1 == (uint32_t)X)) need = INT_MAX;     // test hook, in one CTA of a cluster
            if (!wait([&]() { return peek(done + lane) >= need && peek(&counted) > m - kRing; })) break;
            const float2 ai = sp[i0 * kRepBlock + lane], aj = sp[j0 * kRepBlock + lane];
            float2 ain, ajn;
            float hix = 0.f, hiy = 0.f, hjx = 0.f, hjy = 0.f;
            if (quick) {
                float2 a[2 * kHeld], ap[2 * kHeld], ao[2 * kHeld];
#pragma unroll
                for (int u = 0; u < 2 * kHeld; u++)
                    if (u % kHeld < 2 || u % kHeld < (u < kHeld ? na : nb)) {
                        a[u] = sp[q[u].y * kRepBlock + lane];
                        ap[u] = sp[(q[u].z >> 16) * kRepBlock + lane];
                        ao[u] = sp[(q[u].z & 0xFFFF) * kRepBlock + lane];
                    }
                propose_with<VARIANT>(ai, aj, tt, ain, ajn);
                float yx = 0.f, yy = 0.f;
#pragma unroll
                for (int u = 0; u < kHeld; u++) {
                    if (u < na) record_step<true>(q[u], a[u], ap[u], ao[u], yx, yy, hix, hiy);
                    if (u < nb) record_step<true>(q[kHeld + u], a[kHeld + u], ap[kHeld + u], ao[kHeld + u], yx, yy, hjx, hjy);
                }
                if (max(na, nb) > kHeld)
                    accumulate_two<true>(A + kHeld, max(na - kHeld, 0), B + kHeld, max(nb - kHeld, 0), sp, lane, hix, hiy,
                                         hjx, hjy);
            } else {
                propose_with<VARIANT>(ai, aj, tt, ain, ajn);
                sp[j0 * kRepBlock + lane] = ajn;       // h_i is evaluated at the proposed a_j
                if (S.tiles) {
                    accumulate_tiles_1<8, 4, true>(L + ri.x, ri.y - ri.x, sp, lane, hix, hiy);
                    accumulate_tiles_1<8, 4, true>(L + rj.x, rj.y - rj.x, sp, lane, hjx, hjy);
                } else if (S.single_groups) {
                    accumulate_two<true>(A, na, B, nb, sp, lane, hix, hiy, hjx, hjy);
                } else {
                    accumulate_two<false>(A, na, B, nb, sp, lane, hix, hiy, hjx, hjy);
                }
            }
            const float dix = __fsub_rn(ain.x, ai.x), diy = __fsub_rn(ain.y, ai.y);
            const float djx = __fsub_rn(ajn.x, aj.x), djy = __fsub_rn(ajn.y, aj.y);
            const float dE = -fmaf(dix, hix, -diy * hiy) - fmaf(djx, hjx, -djy * hjy);
            if (per_exchange > 0 && m >= (version + 1) * per_exchange) {
                version = m / per_exchange;
                if (!wait([&]() { return peek(&exchanged) >= version; })) break;
                beta_d = beta_s[lane];
                beta = (float)beta_d;
            }
            bool accept;
            if (beta_d == 0.0) accept = true;
            else accept = (dE <= 0.f) || (tt[6] < expf(-beta * dE));
            if (accept) {
                sp[i0 * kRepBlock + lane] = ain;
                sp[j0 * kRepBlock + lane] = ajn;
            } else if (!quick) {
                sp[j0 * kRepBlock + lane] = aj;
            }
            dEx[t * kRepBlock + lane] = dE;
            const unsigned yes = __ballot_sync(0xffffffffu, accept);
            __syncwarp();                          // a vote orders no memory
            if (lane == 0) {
                acx[t] = yes;
                publish(done + t, m);
            }
            if (P.trace != nullptr && U.sample == P.trace_sample && U.rep_begin + lane == P.trace_rep && active) {
                const long long idx = m + (sweep0 - P.trace_sweep0) * steps;
                if (idx >= 0 && idx < P.trace_cap) {
                    pspin_move_record* rec = reinterpret_cast<pspin_move_record*>(P.trace) + idx;
                    rec->i0 = i0; rec->j0 = j0;
                    rec->ai_old[0] = ai.x; rec->ai_old[1] = ai.y;
                    rec->aj_old[0] = aj.x; rec->aj_old[1] = aj.y;
                    rec->ai_new[0] = ain.x; rec->ai_new[1] = ain.y;
                    rec->aj_new[0] = ajn.x; rec->aj_new[1] = ajn.y;
                    rec->dE = dE;
                    rec->accepted = accept ? 1 : 0;
                    rec->log_q_ratio = 0.f;
                    rec->log_u = logf(tt[6]);
                }
            }
        }
    } else {
        // ------------------------------------------------------------ energies, counters, exchanges
        if (active) E = P.energy[gr];
        if (RT > 0) {
            const int* perm = P.perm + (int64_t)U.sample * RT;
            for (int i = lane; i < RT; i += 32) pt_slot[i] = perm[i];
            for (int t = lane; t < P.NT; t += 32) {
                pt_sched[t] = P.beta_sched[t];
                pt_swaps[t] = 0;
            }
            drand = P.drand_state[U.sample];
            if (P.nrep <= 32) drand_ahead(pt_seq, (P.NT - 1) * P.nrep, drand);
            __syncwarp();
        }
        int to_exchange = per_exchange, n_ex = 0;
        for (int m = 0; m < total; m++) {
            const int t = m % kRing;
            if (!wait([&]() { return peek(done + t) >= m; })) break;
            if ((acx[t] >> lane) & 1u) {
                E += (double)dEx[t * kRepBlock + lane];
                nacc++;
            }
            nprop++;
            __syncwarp();
            if (lane == 0) publish(&counted, m + 1);          // (this slot's values have been read)
            if (per_exchange == 0 || --to_exchange > 0) continue;
            to_exchange = per_exchange;
            const int par = n_ex & 1;
            double* Ex = pt_E + par * RT;
            if (X > 1) {
                if (lane == 0) mbar_expect_tx(ebar + par, (uint32_t)(RT * sizeof(double)));
                if (active) {
                    const uint32_t dx = smem_u32(Ex + U.rep_begin + lane), db = smem_u32(ebar + par);
                    for (int q = 0; q < X; q++) st_async_f64(map_rank(dx, (uint32_t)q), E, map_rank(db, (uint32_t)q));
                }
                if (!__all_sync(0xffffffffu, mbar_wait(ebar + par, (uint32_t)(n_ex >> 1) & 1u, P.status, P.patience))) {
                    stop = 1;
                    break;
                }
            } else {
                if (active) Ex[lane] = E;
                __syncwarp();
            }
            for (int i = lane; i < RT; i += 32) pt_Es[i] = Ex[pt_slot[i]];
            __syncwarp();
            if (P.nrep <= 32)
                exchange_columns(pt_slot, pt_Es, pt_sched, pt_seq, P.NT, P.nrep, drand,
                                 [&](int t2, int n) { pt_swaps[t2] += n; });
            else
                exchange_pass(pt_slot, pt_sched, P.NT, P.nrep, drand, [&](int i, int) { return pt_Es[i]; },
                              [&](int i, int j, double Ei, double Ej) {
                                  pt_Es[i] = Ej;
                                  pt_Es[j] = Ei;
                              },
                              [&](int t2, int n) { pt_swaps[t2] += n; });
            for (int i = lane; i < RT; i += 32) pt_beta[pt_slot[i]] = pt_sched[i / P.nrep];
            __syncwarp();
            if (active) beta_s[lane] = beta_d = pt_beta[U.rep_begin + lane];
            __syncwarp();
            n_ex++;
            if (lane == 0) publish(&exchanged, n_ex);
            if (P.nrep <= 32) drand_ahead(pt_seq, (P.NT - 1) * P.nrep, drand);   // for the next one
            __syncwarp();
        }
    }
    __syncthreads();
    if (X > 1) {
        if (stop && threadIdx.x == 0)          // a CTA that gave up takes its cluster, one PT sample, with it
            for (int q = 0; q < X; q++) st_cluster_u32((const void*)&stop, (uint32_t)q, 1u);
        cluster_sync();                        // no store may still target a CTA that has gone
    }
    if (stop) return;                          // the block keeps its state from before the launch
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        if (l < U.rep_count) P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l] = sp[idx];
    }
    if (warp == K && active) {
        P.energy[gr] = E;
        P.accepted[gr] += nacc;
        P.proposed[gr] += nprop;
        if (RT > 0) P.beta_out[gr] = beta_d;
    }
    if (warp == K && RT > 0 && (X == 1 || cluster_rank() == 0u)) {
        int* perm = P.perm + (int64_t)U.sample * RT;
        for (int i = lane; i < RT; i += 32) perm[i] = pt_slot[i];
        long long* acc = P.ex_acc + (int64_t)U.sample * (P.NT - 1);
        long long* prop = P.ex_prop + (int64_t)U.sample * (P.NT - 1);
        for (int t = lane; t < P.NT - 1; t += 32) {
            acc[t] += pt_swaps[t];
            prop[t] += (long long)(total / per_exchange) * P.nrep;
        }
        if (lane == 0) P.drand_state[U.sample] = drand;
    }
}

// Many blocks (see resident_batched): windows of 32 moves, in batches.  The lanes of
// warp 0 draw the window's pairs, every warp prepares its share of the proposals, and
// the warps mark for every move the earlier moves of the window it does not commute
// with; the window is cut, in move order, into batches of at most K moves that pairwise
// commute, and warp w runs a batch's w-th move.  One CTA barrier per batch; the last
// warp keeps the energies, in move order.
inline size_t resident_batch_smem_bytes(int N, int64_t entries, int K) {
    return (size_t)(N + 1) * kRepBlock * sizeof(float2) + (size_t)entries * sizeof(int2) + (size_t)N * sizeof(int2) +
           2 * 32 * sizeof(int2) + 34 * sizeof(int) + 32 * sizeof(uint32_t) +
           (size_t)2 * K * kRepBlock * (sizeof(float) + sizeof(int)) + (size_t)32 * 7 * kRepBlock * sizeof(float) +
           (size_t)64 * ((N + 31) / 32) * sizeof(uint32_t);
}

template <int VARIANT>
__global__ void __launch_bounds__(256, 2) sweep_resident_batch_kernel(const SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Unit U = P.units[blockIdx.x];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = (int)(blockDim.x >> 5);
    const int owner = K - 1;                   // keeps the running energy and counters
    const int wpr = (N + 31) >> 5;             // words per neighbour-mask row
    const uint32_t* nbm = P.nbmask + S.nb_off; // read through L1
    const int* sc = P.site_chunks + S.split_off;
    const int64_t e0 = __ldg(P.chunk_start + __ldg(sc));
    const int64_t e1 = __ldg(P.chunk_start + __ldg(sc + (int64_t)(N - 1) * (kSplit + 1) + kSplit));
    float2* sp = reinterpret_cast<float2*>(smem_raw);
    int2* L = reinterpret_cast<int2*>(sp + (size_t)(N + 1) * kRepBlock);
    int2* rng_site = L + (e1 - e0);
    int2* picks = rng_site + N;
    int2* mk = picks + 32;                                     // (sweep - sweep0, step) of each move
    int* bounds = reinterpret_cast<int*>(mk + 32);             // [0..32] batch starts, [33] batch count
    uint32_t* cm = reinterpret_cast<uint32_t*>(bounds + 34);   // [32]
    float* dEx = reinterpret_cast<float*>(cm + 32);            // [2][K][32]
    int* acx = reinterpret_cast<int*>(dEx + 2 * K * kRepBlock);  // [2][K][32]
    float* tr = reinterpret_cast<float*>(acx + 2 * K * kRepBlock);  // [32][7][32]
    uint32_t* nrow = reinterpret_cast<uint32_t*>(tr + 32 * 7 * kRepBlock);   // [32][2][wpr]
    for (int m = threadIdx.x; m < N; m += blockDim.x) {
        const int64_t b = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1)));
        const int64_t e = __ldg(P.chunk_start + __ldg(sc + (int64_t)m * (kSplit + 1) + kSplit));
        rng_site[m] = make_int2((int)(b - e0), (int)(e - e0));
    }
    load_block_range(L, P.entries + e0, e1 - e0);
    load_block_amplitudes(sp, P.spins + S.spin_off + U.rep_begin, R, N, kRepBlock, U.rep_count);
    if (threadIdx.x < kRepBlock) sp[N * kRepBlock + threadIdx.x] = make_float2(1.f, 0.f);   // virtual site

    const bool active = lane < U.rep_count;
    const int64_t gr = S.rep_off + U.rep_begin + lane;
    double E = 0.0, beta_d = 0.0;
    float beta = 0.f;
    long long nacc = 0, nprop = 0;
    uint32_t k0 = 0, k1 = 0;
    if (active) {
        beta_d = P.beta[gr];
        beta = (float)beta_d;
        const uint64_t key = P.key[gr];
        k0 = (uint32_t)key;
        k1 = (uint32_t)(key >> 32);
        if (warp == owner) E = P.energy[gr];
    }
    const long long sweep0 = *P.sweep_counter;
    const int steps = N / 2, total = P.nsweeps * steps;
    // is `site` a site of the window's move j or a neighbour of one?
    auto in_reach = [&](int site, int j) {
        const int2 q = picks[j];
        const uint32_t* rows = nrow + 2 * j * wpr;
        return site == q.x || site == q.y || (((rows[site >> 5] | rows[wpr + (site >> 5)]) >> (site & 31)) & 1u);
    };
    // the owner warp's running energy and counters take a batch's moves in move order
    auto account = [&](int par, int n) {
        for (int w = 0; w < n; w++) {
            if (acx[(par * K + w) * kRepBlock + lane]) {
                E += (double)dEx[(par * K + w) * kRepBlock + lane];
                nacc++;
            }
            nprop++;
        }
    };
    __syncthreads();

    long long batches = 0;
    int prev = 0;                              // moves in the previous batch
    for (int m0 = 0; m0 < total; m0 += 32) {
        const int n = min(32, total - m0);
        if (warp == 0) {                       // the window's pairs
            int i0 = 0, j0 = 1, sw = 0, kk = 0;
            if (lane < n) {
                sw = (m0 + lane) / steps;
                kk = (m0 + lane) % steps;
                pair_pick(S.pair_key0, S.pair_key1, (uint64_t)(sweep0 + sw), (uint32_t)kk, N, i0, j0);
            }
            picks[lane] = make_int2(i0, j0);
            mk[lane] = make_int2(sw, kk);
            cm[lane] = 0u;
        }
        // every warp: the state-independent parts of the proposals of its share
        // of the window's moves (random words, sines and cosines), for its lanes
        for (int t = warp; t < n; t += K) {
            const int m = m0 + t;
            float tt[7];
            move_trig<VARIANT>(move_words(k0, k1, (uint64_t)(sweep0 + m / steps), (uint32_t)(m % steps)), tt);
#pragma unroll
            for (int q = 0; q < 7; q++) tr[(t * 7 + q) * kRepBlock + lane] = tt[q];
        }
        __syncthreads();
        // the neighbour-mask rows of the window's sites, all loads in flight at once
        const int tot = n * 2 * wpr;
        for (int i0 = threadIdx.x; i0 < tot; i0 += kInFlight * blockDim.x) {
            uint32_t v[kInFlight];
#pragma unroll
            for (int u = 0; u < kInFlight; u++) {
                const int idx = i0 + u * (int)blockDim.x;
                v[u] = 0u;
                if (idx < tot) {
                    const int j = idx / (2 * wpr), r = idx - j * 2 * wpr;
                    const int2 q = picks[j];
                    v[u] = __ldg(nbm + (r < wpr ? q.x * wpr + r : q.y * wpr + (r - wpr)));
                }
            }
#pragma unroll
            for (int u = 0; u < kInFlight; u++) {
                const int idx = i0 + u * (int)blockDim.x;
                if (idx < tot) nrow[idx] = v[u];
            }
        }
        __syncthreads();
        // conflict masks: the earlier moves of the window that move `lane`
        // does not commute with, the earlier moves shared out over the warps
        uint32_t part = 0;
        if (lane < n) {
            const int2 me = picks[lane];
            for (int j = warp; j < lane; j += K)
                if (in_reach(me.x, j) || in_reach(me.y, j)) part |= 1u << j;
        }
        if (part) atomicOr(cm + lane, part);
        __syncthreads();
        if (warp == 0) {
            // greedy cut in move order: a batch [s0, e) ends at the first move
            // that does not commute with one of [s0, itself), or after K moves
            const uint32_t mask = cm[lane];
            int nb = 0;
            for (int s0 = 0; s0 < n;) {
                const unsigned bad = __ballot_sync(0xffffffffu, lane > s0 && lane < n && (mask >> s0) != 0u);
                const int e = min(bad ? __ffs(bad) - 1 : n, min(n, s0 + K));
                if (lane == 0) bounds[nb] = s0;
                nb++;
                s0 = e;
            }
            if (lane == 0) {
                bounds[nb] = n;
                bounds[33] = nb;
            }
        }
        __syncthreads();
        const int nb = bounds[33];
        for (int b = 0; b < nb; b++) {
            const int bs = bounds[b], be = bounds[b + 1];
            const int par = (int)(batches & 1);
            if (warp == owner && batches > 0) account(par ^ 1, prev);
            if (warp < be - bs) {
                const int t = bs + warp;
                const int2 pq = picks[t], swk = mk[t];
                const int i0 = pq.x, j0 = pq.y;
                float tt[7];
#pragma unroll
                for (int q = 0; q < 7; q++) tt[q] = tr[(t * 7 + q) * kRepBlock + lane];
                const float2 ai = sp[i0 * kRepBlock + lane], aj = sp[j0 * kRepBlock + lane];
                float2 ain, ajn;
                propose_with<VARIANT>(ai, aj, tt, ain, ajn);
                const float cu = tt[6];
                sp[j0 * kRepBlock + lane] = ajn;       // h_i is evaluated at the proposed a_j
                __syncwarp();
                float hix = 0.f, hiy = 0.f, hjx = 0.f, hjy = 0.f;
                const int2 ri = rng_site[i0], rj = rng_site[j0];
                if (S.tiles) {
                    accumulate_tiles_1<2, 2, false>(L + ri.x, ri.y - ri.x, sp, lane, hix, hiy);
                    accumulate_tiles_1<2, 2, false>(L + rj.x, rj.y - rj.x, sp, lane, hjx, hjy);
                } else if (S.single_groups) {
                    accumulate_records<4, true>(L + ri.x, ri.y - ri.x, sp, lane, hix, hiy);
                    accumulate_records<4, true>(L + rj.x, rj.y - rj.x, sp, lane, hjx, hjy);
                } else {
                    accumulate_records<4>(L + ri.x, ri.y - ri.x, sp, lane, hix, hiy);
                    accumulate_records<4>(L + rj.x, rj.y - rj.x, sp, lane, hjx, hjy);
                }
                const float dix = __fsub_rn(ain.x, ai.x), diy = __fsub_rn(ain.y, ai.y);
                const float djx = __fsub_rn(ajn.x, aj.x), djy = __fsub_rn(ajn.y, aj.y);
                const float dE = -fmaf(dix, hix, -diy * hiy) - fmaf(djx, hjx, -djy * hjy);
                bool accept;
                if (beta_d == 0.0) accept = true;
                else accept = (dE <= 0.f) || (cu < expf(-beta * dE));
                __syncwarp();
                if (accept) sp[i0 * kRepBlock + lane] = ain;
                else sp[j0 * kRepBlock + lane] = aj;
                dEx[(par * K + warp) * kRepBlock + lane] = dE;
                acx[(par * K + warp) * kRepBlock + lane] = accept ? 1 : 0;
                if (P.trace != nullptr && U.sample == P.trace_sample && U.rep_begin + lane == P.trace_rep && active) {
                    const long long idx = (long long)swk.x * steps + swk.y + (sweep0 - P.trace_sweep0) * steps;
                    if (idx >= 0 && idx < P.trace_cap) {
                        pspin_move_record* rec = reinterpret_cast<pspin_move_record*>(P.trace) + idx;
                        rec->i0 = i0; rec->j0 = j0;
                        rec->ai_old[0] = ai.x; rec->ai_old[1] = ai.y;
                        rec->aj_old[0] = aj.x; rec->aj_old[1] = aj.y;
                        rec->ai_new[0] = ain.x; rec->ai_new[1] = ain.y;
                        rec->aj_new[0] = ajn.x; rec->aj_new[1] = ajn.y;
                        rec->dE = dE;
                        rec->accepted = accept ? 1 : 0;
                        rec->log_q_ratio = 0.f;
                        rec->log_u = logf(cu);
                    }
                }
            }
            __syncthreads();
            prev = be - bs;
            batches++;
        }
    }
    if (warp == owner && batches > 0) account((int)((batches - 1) & 1), prev);
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        if (l < U.rep_count) P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l] = sp[idx];
    }
    if (warp == owner && active) {
        P.energy[gr] = E;
        P.accepted[gr] += nacc;
        P.proposed[gr] += nprop;
    }
}

size_t resident_smem_bytes_host(int N, int64_t entries, int warps, int pt_slots) {
    return resident_smem_bytes(N, entries, warps, pt_slots);
}

// Which launches run in the batched form.  The dataflow holds 168 registers a thread, a
// warp more, and its prepared moves in global memory (some 900 bytes a move and block,
// written and read) by a launch of their own; the batched form costs a barrier per
// batch and its windows' preparation, but up to twice as many of its blocks share an
// SM.  Samples of 96 replicas (three blocks), sweeps without exchanges, dataflow and
// batched, us a sweep:
//   many blocks, 8 warps: 50 samples N = 62 55 and 29, 200 samples 139 and 71, N = 128
//     219 and 111; 2 warps: 100 samples N = 62 42 and 35;
//   few, many moves: 8 warps, 16 samples N = 128 42 and 45, one sample N = 512 73 and 98;
//   few, moves that mostly wait for one another: 8 warps, 8 samples N = 32 18.9 and
//     17.8, N = 62 24.7 and 23.4; 2 warps N = 32 19.4 and 20.5;
//   one sweep a launch: 8 samples, 8 warps N = 62 61 and 54, N = 128 71 and 69, N = 256
//     89 and 90.
// So the batched form takes every launch where it needs fewer waves of blocks than the
// dataflow, or as many with more than two blocks per SM; and without exchanges those of
// at least 4 warps at N <= 8 warps, and those of at most kShortLaunch moves.
int resident_batched(int n_units, int variant, int max_N, int64_t max_entries, int warps, int pt_slots) {
    if (warps == 1 || resident_batch_smem_bytes(max_N, max_entries, warps) > 227 * 1024 - 64) return kBatchedNever;
    if (pt_slots == 0 && warps >= 4 && max_N <= 8 * warps) return kBatchedAlways;
    const int otherwise = pt_slots == 0 ? kBatchedShort : kBatchedNever;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return otherwise;
    }
    if (n_units <= sms) return otherwise;
    auto waves = [&](void (*kern)(const SweepParams), int threads, size_t smem) {
        int blocks = 0;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, threads, smem);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && blocks > 0 ? (n_units + blocks * sms - 1) / (blocks * sms) : 1 << 30;
    };
    const int flow = waves(variant == 0 ? sweep_resident_kernel<0> : sweep_resident_kernel<1>, 32 * (warps + 1),
                           resident_smem_bytes(max_N, max_entries, warps, pt_slots));
    const int batch = waves(variant == 0 ? sweep_resident_batch_kernel<0> : sweep_resident_batch_kernel<1>, 32 * warps,
                            resident_batch_smem_bytes(max_N, max_entries, warps));
    return batch < flow || (pt_slots == 0 && batch == flow && n_units > 2 * sms) ? kBatchedAlways : otherwise;
}

cudaError_t launch_sweep_resident(const SweepParams& p, int n_units, int variant, int max_N, int64_t max_entries,
                                  int pt_slots, bool batched, cudaStream_t st) {
    if (n_units <= 0) return cudaSuccess;
    if (p.warps < 1 || p.warps > 8 || (p.warps & (p.warps - 1)) != 0) return cudaErrorInvalidValue;
    if (batched) {
        const size_t smem = resident_batch_smem_bytes(max_N, max_entries, p.warps);
        auto kern = variant == 0 ? sweep_resident_batch_kernel<0> : sweep_resident_batch_kernel<1>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<n_units, 32 * p.warps, smem, st>>>(p);
        return cudaGetLastError();
    }
    const size_t smem = resident_smem_bytes(max_N, max_entries, p.warps, pt_slots);
    if (smem > 227 * 1024 - 64) return cudaErrorInvalidValue;
    if (p.warps == 1) {
        auto kern = variant == 0 ? sweep_resident_one_kernel<0> : sweep_resident_one_kernel<1>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<n_units, 32, smem, st>>>(p);
        return cudaGetLastError();
    }
    SweepParams q = p;
    q.patience = p.stall_move >= 0 ? p.wait_clocks : 2 * p.wait_clocks + kDrainClocks;
    const int most = p.nsweeps * (max_N / 2);
    resident_prepare_kernel<<<dim3((unsigned)n_units, (unsigned)((most + 3) / 4)), 128, 0, st>>>(p, variant);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    auto kern = variant == 0 ? sweep_resident_kernel<0> : sweep_resident_kernel<1>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)n_units);
    cfg.blockDim = dim3((unsigned)(32 * (p.warps + 1)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.exec;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.exec > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kern, q);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace pspin
