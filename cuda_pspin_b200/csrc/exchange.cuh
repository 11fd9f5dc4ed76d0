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
// slot[t*nr + r]: the replica at slot (t, r); energy(i) / swap(i, j) read and
// exchange the energies of slots; count(t, n): n swaps at t.
//
// The nr columns of one t touch different replicas, so the lanes take one
// column each; the draws keep the column order: the lane whose column is the
// k-th with delta < 0 steps the drand48 state k + 1 times on its own.
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
