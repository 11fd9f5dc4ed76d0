// exchange.cuh -- the replica exchange of one sample by one warp
// (parallel_tempering.cu:316-352), shared by exchange_kernel and by the sweep
// kernel where a launch runs whole PT steps.
#pragma once
#include <cstdint>
#include "rng.cuh"

namespace pspin {

// One pass over the temperatures: t runs from the hottest pair upwards and a
// swap is applied before the next t is tried, so a replica may climb several
// rungs in one pass; the uniform is drawn only when delta < 0 (:333-334).
// slot[t*nr + r]: the replica at slot (t, r).
//
// The nr columns of one t touch different replicas, so the lanes take one
// column each; the draws keep the column order.

// The next n states of the drand48 stream after st (any number of draws of a pass
// can then be read off by its place in it).
__device__ __forceinline__ void drand_ahead(uint64_t* seq, int n, uint64_t st) {
    const uint64_t mask = 0xFFFFFFFFFFFFULL;
    const int lane = threadIdx.x & 31;
    uint64_t a = 0x5DEECE66DULL, c = 0xBULL;         // 1 step; squared five times: 32
    uint64_t mine = st;
#pragma unroll
    for (int bit = 0; bit < 5; bit++) {              // lane steps, by the bits of lane
        if ((lane >> bit) & 1) mine = (a * mine + c) & mask;
        c = (a * c + c) & mask;
        a = (a * a) & mask;
    }
    mine = (0x5DEECE66DULL * mine + 0xBULL) & mask;  // lane + 1 steps
    for (int k = lane; k < n; k += 32) {
        seq[k] = mine;
        mine = (a * mine + c) & mask;
    }
}

// u < exp(delta) for the uniform u of drand48 state s and delta < 0.  Decided in
// FP32 where the two are apart by far more than its errors (the exponent's
// rounding 6e-8 |delta| and expf's and the uniform's own, together below 6e-6 for
// |delta| < 80), else in FP64 as the reference decides.
__device__ __forceinline__ bool drawn_below(uint64_t s, double delta) {
    const uint32_t top = (uint32_t)(s >> 16);
    const float u = (float)top * (1.0f / 4294967296.0f), w = expf((float)delta);
    if (delta > -80.0 && top > (1u << 20)) {
        if (u < w * (1.0f - 2e-5f)) return true;
        if (u > w * (1.0f + 2e-5f)) return false;
    }
    return (double)s * (1.0 / 281474976710656.0) < exp(delta);
}

// nr <= 32, energies Es by slot (not kept up to date), `seq` the next
// (NT - 1) * nr drand48 states; every lane carries the replica that its column has
// brought up to t, so a temperature is a short chain of register operations.
template <class Count>
__device__ __forceinline__ void exchange_columns(int* slot, const double* Es, const double* sched, const uint64_t* seq,
                                                 int NT, int nr, uint64_t& st, Count count) {
    const int lane = threadIdx.x & 31;
    const bool on = lane < nr;
    const int r = on ? lane : 0;
    int a = slot[r], b = slot[nr + r], used = 0;
    double Ea = Es[r], Eb = Es[nr + r], s0 = sched[0], s1 = sched[1];
    for (int t = 0; t < NT - 1; t++) {
        const int ahead = min(t + 2, NT - 1) * nr + r;       // the next row, on its way
        const int c = slot[ahead];
        const double Ec = Es[ahead], s2 = sched[min(t + 2, NT - 1)];
        const double delta = (s0 - s1) * (Ea - Eb);
        bool ok = on && delta >= 0.0;
        const bool draw = on && !ok;
        const unsigned draws = __ballot_sync(0xffffffffu, draw);
        if (draw) ok = drawn_below(seq[used + __popc(draws & ((1u << lane) - 1u))], delta);
        used += __popc(draws);
        if (on) slot[t * nr + r] = ok ? b : a;
        if (!ok) {
            a = b;
            Ea = Eb;
        }
        b = c;
        Eb = Ec;
        s0 = s1;
        s1 = s2;
        const int n = __popc(__ballot_sync(0xffffffffu, ok));
        if (lane == 0) count(t, n);
    }
    if (on) slot[(NT - 1) * nr + r] = a;
    if (used > 0) st = seq[used - 1];
    __syncwarp();
}

// Any nr: energy(i, replica) and swap(i, j, Ei, Ej) read and exchange the energies
// of slots; the lane whose column is the k-th with delta < 0 steps the drand48
// state k + 1 times on its own; count(t, n): n swaps at t.
template <class Energy, class Swap, class Count>
__device__ __forceinline__ void exchange_pass(int* slot, const double* sched, int NT, int nr, uint64_t& st, Energy energy,
                                              Swap swap, Count count) {
    const int lane = threadIdx.x & 31;
    for (int t = 0; t < NT - 1; t++) {
        const double db = sched[t] - sched[t + 1];
        int n_swap = 0;
        for (int r0 = 0; r0 < nr; r0 += 32) {
            const int r = r0 + lane, ia = t * nr + r, ib = ia + nr;
            const bool on = r < nr;
            int a = 0, b = 0;
            double Ea = 0.0, Eb = 0.0;
            if (on) {
                a = slot[ia];
                b = slot[ib];
                Ea = energy(ia, a);
                Eb = energy(ib, b);
            }
            const double delta = db * (Ea - Eb);
            bool ok = on && delta >= 0.0;
            const bool draw = on && !ok;
            const unsigned draws = __ballot_sync(0xffffffffu, draw);
            if (draws) {
                uint64_t mine = st;
                if (draw) {
                    const double w = exp(delta);
                    double u = 0.0;
                    for (int q = __popc(draws & ((1u << lane) - 1u)); q >= 0; q--) u = drand48_next(mine);
                    ok = u < w;
                }
                st = __shfl_sync(0xffffffffu, mine, 31 - __clz(draws));
            }
            if (ok) {
                slot[ia] = b;
                slot[ib] = a;
                swap(ia, ib, Ea, Eb);
            }
            n_swap += __popc(__ballot_sync(0xffffffffu, ok));
        }
        if (lane == 0) count(t, n_swap);
        __syncwarp();
    }
}

}  // namespace pspin
