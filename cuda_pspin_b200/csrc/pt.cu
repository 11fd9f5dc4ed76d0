// pt.cu -- FP64 energies (resync, split) and the device-side replica exchange.
#include "exchange.cuh"
#include "internal.h"

namespace pspin {

// ---------------------------------------------------------------------
// Projection of every replica of one unit onto its constraint, in FP64:
// sum|a|^2 = target (sphere) or sum|a|^4 = target (cube), the rescaled
// amplitudes stored back as FP32.
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(256) renorm_kernel(const EnergyParams P) {
    extern __shared__ float2 rsm[];
    const Unit U = P.units[blockIdx.x];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2* sp = rsm;                                                      // [N][32]
    __shared__ double scale_s[kRepBlock];
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        float2 v = make_float2(0.f, 0.f);
        if (l < U.rep_count) v = P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l];
        sp[idx] = v;
    }
    __syncthreads();
    if (warp == 0) {
        double s = 0.0;
        for (int site = 0; site < N; site++) {
            const float2 a = sp[site * kRepBlock + lane];
            const double r2 = (double)a.x * a.x + (double)a.y * a.y;
            s += (S.variant == 0) ? r2 : r2 * r2;
        }
        double sc = 1.0;
        if (lane < U.rep_count && s > 0.0) {
            const double t = P.target[S.rep_off + U.rep_begin + lane];
            sc = (S.variant == 0) ? sqrt(t / s) : sqrt(sqrt(t / s));
        }
        scale_s[lane] = sc;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        const double sc = scale_s[l];
        const float2 a = sp[idx];
        if (l < U.rep_count)
            P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l] = make_float2((float)(a.x * sc), (float)(a.y * sc));
    }
}

// ---------------------------------------------------------------------
// FP64 energies of every replica.
//
// The chain's energy (mc.cu:323-405): E2 = -sum_{i<j} Re[g_ij a_i conj a_j]
// (diagonal excluded), E4 = -sum over active (q,ch) Re[g f_ch(a)] with the
// channel conjugation patterns of mc.cu:389-391.  Amplitudes are the FP32
// ones the sweep evolves, upcast.
//
// Site i is unconjugated in every channel and runs fastest in the table of a
// dense sample, so a run of entries with the same (j, k, l, ch) costs
// Y = sum g a_i, two FP64 FMA per entry, and one product Y a_j a_k a_l (with
// the channel's conjugations) per run; a table in any other order is correct
// with runs of one entry.  One entry as a product of four amplitudes of its
// own had cost 8 conversions and ~13 FP64 operations.  The amplitudes are
// upcast once per CTA into shared memory (kDouble: up to N = kDoubleN; above,
// FP32 upcast at each use), so an entry is bound by its shared-memory reads
// (16-byte broadcast + 512-byte row: 5 wavefronts a warp).
//
// Lanes are replicas; a unit's table is cut in pieces, each summed by the 8 warps
// of a CTA into one partial per replica, and energy_sum_kernel adds the partials
// in order.  The pieces follow from the sample alone, so its energies have the
// same bits in any batch and on any device; how many CTAs share a unit's pieces
// follows from the number of units, so few units still fill the chip.  The CTAs of
// kEnergyGroup neighbouring units (of one sample, mostly) alternate, so that they
// read a table that is larger than L2 together, and the heaviest units come first.
// 768 units of a 256-sample batch (N 24..64, fully connected, 96 replicas): 45 ms
// as one product per entry, 4.9 ms now; two units at N=128 (10.7 M entries): 728
// and 0.89 ms.  (With 16 CTAs per SM and a unit's CTAs a grid apart: 5.7 and 0.89.)
// ---------------------------------------------------------------------
constexpr int kDoubleN = 192;      // amplitudes as double2 up to here: 96 KB of shared memory a CTA
constexpr int kEnergyWarps = 8;
constexpr int kMaxPieces = 256;
constexpr int kEnergyGroup = 4;

// pieces of a sample's table: at least 1024 entries for each warp of a CTA
__host__ __device__ inline int energy_pieces(int64_t nq) {
    const int64_t want = nq / (kEnergyWarps * 1024) + 1;
    return (int)(want < kMaxPieces ? want : kMaxPieces);
}

// kOne: a CTA for every piece, where there are as many (with the loop's registers the
// two units at N=128 took 0.99 ms)
template <bool kDouble, bool kOne>
__global__ void __launch_bounds__(32 * kEnergyWarps) energy_kernel(const EnergyParams P) {
    extern __shared__ __align__(16) unsigned char esm[];
    const int group = (int)(blockIdx.x / (kEnergyGroup * P.max_ctas)), in_group = (int)(blockIdx.x % (kEnergyGroup * P.max_ctas));
    const int members = min(kEnergyGroup, P.n_units - group * kEnergyGroup);
    const int unit = group * kEnergyGroup + in_group % members;
    const Unit U = P.units[unit];
    const SampleDev& S = P.samples[U.sample];       // (read again for every piece: few registers)
    // this CTA's pieces: the same number for every CTA of the unit but the last
    const int pieces = energy_pieces(S.nq), each = kOne ? 1 : (pieces + P.max_ctas - 1) / P.max_ctas;
    const int first = in_group / members * each, end = min(pieces, first + each);
    if (first >= end) return;
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int nw = kEnergyWarps;
    __shared__ Q64 stage_all[nw][32];
    static_assert(sizeof(Q64) == sizeof(double2), "the partial sums reuse the staging rows");
    Q64* stage = stage_all[warp];
    double2* spd = reinterpret_cast<double2*>(esm);                        // [N][32]
    float2* spf = reinterpret_cast<float2*>(esm);
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        float2 v = make_float2(0.f, 0.f);
        if (l < U.rep_count) v = P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l];
        if (kDouble) spd[idx] = make_double2(v.x, v.y);
        else spf[idx] = v;
    }
    __syncthreads();
    auto amp = [&](int site) {
        if (kDouble) return spd[site * kRepBlock + lane];
        const float2 v = spf[site * kRepBlock + lane];
        return make_double2(v.x, v.y);
    };

    for (int piece = first; piece < end; piece++) {
        double e2 = 0.0, e4 = 0.0;
        if (S.h2_active) {
            const int64_t npair = (int64_t)N * (N - 1) / 2;
            for (int64_t pidx = piece * nw + warp; pidx < npair; pidx += (int64_t)pieces * nw) {
                // pair index -> (i<j), row-major over j
                int j = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)pidx)) * 0.5f);
                while ((int64_t)j * (j - 1) / 2 > pidx) j--;
                while ((int64_t)(j + 1) * j / 2 <= pidx) j++;
                const int i = (int)(pidx - (int64_t)j * (j - 1) / 2);
                const double g = __ldg(P.g2 + S.g2_off + (int64_t)i * N + j);
                if (g == 0.0) continue;
                const double2 ai = amp(i), aj = amp(j);
                // -Re[g a_i conj(a_j)]
                e2 -= g * (ai.x * aj.x + ai.y * aj.y);
            }
        }
        // this warp's contiguous share of the table, 32 entries at a time: the
        // next 32 are in flight while these are summed
        const int64_t workers = (int64_t)pieces * nw, me = (int64_t)piece * nw + warp;
        const int64_t t0 = S.nq * me / workers, t1 = S.nq * (me + 1) / workers;
        const int4* __restrict__ Q = reinterpret_cast<const int4*>(P.quartets + S.q_off);
        int4 mine = make_int4(0, 0, 0, 0);
        if (t0 + lane < t1) mine = __ldg(Q + t0 + lane);
        for (int64_t t = t0; t < t1; t += 32) {
            const int n = (int)(t1 - t < 32 ? t1 - t : 32);
            reinterpret_cast<int4*>(stage)[lane] = mine;
            const int4 cur = mine;
            if (t + 32 + lane < t1) mine = __ldg(Q + t + 32 + lane);
            // starts of the runs of equal (j, k, l, ch)
            const unsigned kl = (unsigned)cur.y, kj = (unsigned)cur.x >> 16;
            const unsigned pkl = __shfl_up_sync(0xffffffffu, kl, 1), pkj = __shfl_up_sync(0xffffffffu, kj, 1);
            unsigned starts = __ballot_sync(0xffffffffu, lane < n && (lane == 0 || kl != pkl || kj != pkj));
            __syncwarp();
            while (starts) {
                const int b = __ffs(starts) - 1;
                starts &= starts - 1;
                const int e = starts ? __ffs(starts) - 1 : n;
                double yx = 0.0, yy = 0.0;
#pragma unroll 4
                for (int u = b; u < e; u++) {
                    const Q64 q = stage[u];
                    const double2 a = amp(q.i);
                    yx = fma(q.g, a.x, yx);
                    yy = fma(q.g, a.y, yy);
                }
                const Q64 q = stage[b];
                const int ch = q.lch >> 14;
                double2 aj = amp(q.j), ak = amp(q.k), al = amp(q.lch & 0x3FFF);
                // conjugations: ch0 {k,l}, ch1 {j,k}, ch2 {j,l} (mc.cu:389-391)
                if (ch != 0) aj.y = -aj.y;
                if (ch != 2) ak.y = -ak.y;
                if (ch != 1) al.y = -al.y;
                const double bx = ak.x * al.x - ak.y * al.y, by = ak.x * al.y + ak.y * al.x;   // s2 s3
                const double ax = yx * aj.x - yy * aj.y, ay = yx * aj.y + yy * aj.x;           // sum g s0 s1
                e4 -= ax * bx - ay * by;
            }
            __syncwarp();
        }
        double2* red = reinterpret_cast<double2*>(&stage_all[0][0]);          // [nw][32], each warp its own staging rows
        red[warp * kRepBlock + lane] = make_double2(e2, e4);
        __syncthreads();
        if (warp == 0) {
            double s2 = 0.0, s4 = 0.0;
            for (int w = 0; w < nw; w++) {
                const double2 v = red[w * kRepBlock + lane];
                s2 += v.x;
                s4 += v.y;
            }
            double2* out = reinterpret_cast<double2*>(P.partial);             // [units][max_pieces][32]
            out[((int64_t)unit * P.max_pieces + piece) * kRepBlock + lane] = make_double2(s2, s4);
        }
        if (kOne) return;
        __syncthreads();                                                       // the staging rows are the next piece's
    }
}

__global__ void __launch_bounds__(kRepBlock) energy_sum_kernel(const EnergyParams P) {
    const Unit U = P.units[blockIdx.x];
    const SampleDev S = P.samples[U.sample];
    const int lane = threadIdx.x;
    if (lane >= U.rep_count) return;
    const int pieces = energy_pieces(S.nq);
    const double2* part = reinterpret_cast<const double2*>(P.partial) + (int64_t)blockIdx.x * P.max_pieces * kRepBlock + lane;
    double s2 = 0.0, s4 = 0.0;
#pragma unroll 8
    for (int q = 0; q < pieces; q++) {
        const double2 v = part[(int64_t)q * kRepBlock];
        s2 += v.x;
        s4 += v.y;
    }
    const int64_t gr = S.rep_off + U.rep_begin + lane;
    if (P.e2) P.e2[gr] = s2;
    if (P.e4) P.e4[gr] = s4;
    if (P.energy) {
        if (P.drift) P.drift[gr] = fabs(P.energy[gr] - (s2 + s4));
        P.energy[gr] = s2 + s4;
    }
}

// most CTAs that share a unit's pieces: 32 CTAs per SM over all units
static int energy_ctas(int n_units, int max_pieces) {
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    const int want = (32 * sms + n_units - 1) / n_units;
    return want < 1 ? 1 : (want > max_pieces ? max_pieces : want);
}

int energy_max_pieces(int64_t max_nq) { return energy_pieces(max_nq); }
size_t energy_partial_doubles(int n_units, int max_pieces) { return (size_t)n_units * max_pieces * kRepBlock * 2; }

cudaError_t launch_energy(const EnergyParams& p, int n_units, int max_N, cudaStream_t st) {
    if (n_units <= 0) return cudaSuccess;
    cudaError_t e;
    if (p.target != nullptr) {
        const size_t smem = (size_t)max_N * kRepBlock * sizeof(float2);
        e = cudaFuncSetAttribute(renorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        renorm_kernel<<<n_units, 256, smem, st>>>(p);
        if ((e = cudaGetLastError()) != cudaSuccess || p.renorm_only) return e;
    }
    const bool dbl = max_N <= kDoubleN;
    const size_t smem = (size_t)max_N * kRepBlock * (dbl ? sizeof(double2) : sizeof(float2));
    EnergyParams q = p;
    q.n_units = n_units;
    q.max_ctas = energy_ctas(n_units, p.max_pieces);
    const bool one = q.max_ctas >= p.max_pieces;
    auto kern = one ? (dbl ? energy_kernel<true, true> : energy_kernel<false, true>)
                    : (dbl ? energy_kernel<true, false> : energy_kernel<false, false>);
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(n_units * q.max_ctas), 32 * kEnergyWarps, smem, st>>>(q);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    energy_sum_kernel<<<n_units, kRepBlock, 0, st>>>(p);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------
// Replica exchange of every sample (exchange.cuh), one warp per sample; then
// betas are rebuilt from perm (:347-351).  Thread 0 of block 0 advances the
// global sweep counter.  With the permutation and the energies staged in shared
// memory in slot order a temperature costs a few shared-memory latencies instead
// of nrep chains of dependent global reads: 256 samples of 24 x 4 replicas took
// 116 us with one thread each, 23 us before the schedule and the counters were
// staged too, 12 now; one sample of 32 x 4 46, 25 and 11 us.
// ---------------------------------------------------------------------
// Staged per sample: [RT] energies, [RT] drand48 states, [NT] betas, [RT] replicas,
// [NT] swap counts.
constexpr size_t kExchangeSmem = 48 * 1024;
__host__ __device__ inline size_t exchange_smem_bytes(int NT, int nr) {
    return (size_t)(NT * nr + NT) * (sizeof(double) + sizeof(int)) + (size_t)NT * nr * sizeof(uint64_t);
}

__global__ void __launch_bounds__(32) exchange_kernel(const ExchangeParams P) {
    extern __shared__ __align__(16) unsigned char xsm[];
    const int s = blockIdx.x, lane = threadIdx.x;
    if (s == 0 && lane == 0) *P.sweep_counter += P.nsweeps_done;
    if (!P.do_exchange || s >= P.n_samples) return;
    const SampleDev S = P.samples[s];
    const int NT = P.NT, nr = P.nrep, RT = NT * nr;
    int* perm = P.perm + (int64_t)s * RT;
    const double* E = P.energy + S.rep_off;
    long long* acc = P.ex_acc + (int64_t)s * (NT - 1);
    long long* prop = P.ex_prop + (int64_t)s * (NT - 1);
    uint64_t st = P.drand_state[s];
    const bool staged = exchange_smem_bytes(NT, nr) <= kExchangeSmem;
    double* Es = reinterpret_cast<double*>(xsm);               // in slot order
    uint64_t* seq = reinterpret_cast<uint64_t*>(Es + RT);      // the next drand48 states
    double* Bs = reinterpret_cast<double*>(seq + RT);
    int* slot = staged ? reinterpret_cast<int*>(Bs + NT) : perm;
    int* swaps = slot + RT;                                    // (staged)
    const double* sched = staged ? Bs : P.beta_sched;
    if (staged) {
        for (int t = lane; t < NT; t += 32) Bs[t] = P.beta_sched[t];
        for (int i = lane; i < RT; i += 32) {
            const int r = perm[i];
            slot[i] = r;
            Es[i] = E[r];
        }
        if (nr <= 32) drand_ahead(seq, (NT - 1) * nr, st);
        __syncwarp();
    }
    if (staged && nr <= 32)
        exchange_columns(slot, Es, sched, seq, NT, nr, st, [&](int t, int n) { swaps[t] = n; });
    else if (staged)
        exchange_pass(slot, sched, NT, nr, st, [&](int i, int) { return Es[i]; },
                      [&](int i, int j, double Ei, double Ej) {
                          Es[i] = Ej;
                          Es[j] = Ei;
                      },
                      [&](int t, int n) { swaps[t] = n; });
    else
        exchange_pass(slot, sched, NT, nr, st, [&](int, int r) { return E[r]; }, [](int, int, double, double) {},
                      [&](int t, int n) {
                          acc[t] += n;
                          prop[t] += nr;
                      });
    if (lane == 0) P.drand_state[s] = st;
    double* beta = P.beta + S.rep_off;
    for (int i = lane; i < RT; i += 32) {
        const int r = slot[i];
        if (staged) perm[i] = r;
        beta[r] = sched[i / nr];
    }
    if (staged)
        for (int t = lane; t < NT - 1; t += 32) {
            acc[t] += swaps[t];
            prop[t] += nr;
        }
}

cudaError_t launch_exchange(const ExchangeParams& p, cudaStream_t st) {
    const int blocks = p.do_exchange && p.n_samples > 0 ? p.n_samples : 1;
    const size_t need = exchange_smem_bytes(p.NT, p.nrep);
    exchange_kernel<<<blocks, 32, p.do_exchange && need <= kExchangeSmem ? need : 0, st>>>(p);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------
// Observable series: one warp per sample.  E of the nrep replicas at the
// slot and q_ab = Re sum_k a_k^a conj(a_k^b) / N for every pair a < b
// (the overlap of analysis_pt.cpp:1404-1416), summed in FP64.
// ---------------------------------------------------------------------
__global__ void observe_kernel(const ObserveParams P) {
    const int s = blockIdx.x, lane = threadIdx.x;
    const long long row = (*P.sweep_counter - P.sweep0) / P.pt_freq - 1;
    if (s >= P.n_samples || row < 0 || row >= P.capacity) return;
    const SampleDev S = P.samples[s];
    const int nr = P.nrep;
    const int npairs = nr * (nr - 1) / 2;
    const int* perm = P.perm + ((int64_t)s * P.NT + P.temp_index) * nr;
    const int64_t base = row * P.n_samples + s;
    for (int r = lane; r < nr; r += 32) P.E_out[base * nr + r] = P.energy[S.rep_off + perm[r]];
    int pr = 0;
    for (int a = 0; a < nr; a++)
        for (int b = a + 1; b < nr; b++, pr++) {
            const float2* xa = P.spins + S.spin_off + perm[a];
            const float2* xb = P.spins + S.spin_off + perm[b];
            double acc = 0.0;
            for (int k = lane; k < S.N; k += 32) {
                const float2 u = xa[(int64_t)k * S.R], v = xb[(int64_t)k * S.R];
                acc += (double)u.x * v.x + (double)u.y * v.y;
            }
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) P.q_out[base * npairs + pr] = acc / S.N;
        }
}

cudaError_t launch_observe(const ObserveParams& p, cudaStream_t st) {
    if (p.n_samples <= 0) return cudaSuccess;
    observe_kernel<<<p.n_samples, 32, 0, st>>>(p);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------
// FP32 FMA throughput probe: 8 independent register chains per thread, so
// the FMA pipe, not latency, is the limit.
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(256) fma_probe_kernel(float* out, int iters) {
    float a[8];
#pragma unroll
    for (int c = 0; c < 8; c++) a[c] = (float)(threadIdx.x + c) * 1e-3f;
    const float m = 0.999999f, k = 1e-7f;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int c = 0; c < 8; c++) a[c] = fmaf(a[c], m, k);
    }
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) s += a[c];
    out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// the same with paired FMA (fma.rn.f32x2): 8 chains of two lanes each
__global__ void __launch_bounds__(256) fma2_probe_kernel(float* out, int iters) {
    float2 a[8];
#pragma unroll
    for (int c = 0; c < 8; c++) a[c] = make_float2((float)(threadIdx.x + c) * 1e-3f, (float)(threadIdx.x - c) * 1e-3f);
    const float2 m = make_float2(0.999999f, 0.999998f), k = make_float2(1e-7f, 2e-7f);
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int c = 0; c < 8; c++) a[c] = __ffma2_rn(a[c], m, k);
    }
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) s += a[c].x + a[c].y;
    out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// paired = 1: the fma.rn.f32x2 probe (twice the FMA per thread and iteration)
cudaError_t launch_fma_probe(float* out, int blocks, int iters, cudaStream_t st, int paired) {
    if (paired) fma2_probe_kernel<<<blocks, 256, 0, st>>>(out, iters);
    else fma_probe_kernel<<<blocks, 256, 0, st>>>(out, iters);
    return cudaGetLastError();
}

}  // namespace pspin
