// learned.cu -- the sweep with local fields at both ends of every move, used
// (mode 1) to record accepted plain moves for training and (mode 2) to run
// the learned proposal with the exact Metropolis-Hastings correction; and
// the network's training kernels (forward, backward, Adam).
//
// What bounds it: at a replica block per few SMs, latency (of a move's 76k cycles
// with one block alone the field passes take 29k and 13k, the network, the samplers
// and the densities on their critical path 34k); with every SM full, issue of the
// field passes.  The chains of both lists run on warps of their own, spread over as
// many SMs as the blocks leave free, and the pair's sub-lists are dense tiles: as
// groups of mostly one term a chunk's dependent loads had taken 36k cycles a pass
// however few terms it held.
//
// Two field passes per move.  Pass 1 reads site i's and site j's lists at
// the current state x: h_i(x), h_j(x) (the proposal's features).  Pass 2
// reads only the pair's sub-lists (the terms of h_i that contain a_j and of
// h_j that contain a_i, about 3/N of a site list) with the changes da_i,
// da_j in the pair's slots, giving h_i(x') - h_i(x) and h_j(x') - h_j(x)
// (the reverse density's features).  E is affine in each site, so
//     dE = -Re[da_i h_i(x')] - Re[da_j h_j(x)]
// exactly (h_i(x') is h_i with a_j' in place, h_j(x) is h_j with a_i).
#include <cuda_bf16.h>

#include <algorithm>

#include "../../include/pspin.h"
#include "mlp.cuh"
#include "sweep_common.cuh"

namespace pspin {

struct LearnParams {
    int mode;                       // 1: plain proposal, fields + recording; 2: learned proposal
    const __nv_bfloat16* w;         // network weights [kMlpParams]
    float* records;                 // ring of accepted plain moves [cap][kRecordFloats]
    unsigned long long* rec_count;  // moves written so far (ring position = count % cap)
    int rec_cap;
    float rec_prob;
};

// Network evaluation for the CTA's 32 replicas by all its warps, on the
// tensor cores with warp-level mma.sync m16n8k16 (BF16 operands, FP32
// accumulation): each layer is Out[32 x units] = In[32 x K] W^T, two m16
// tiles of replicas x n8 tiles of units, the n8 tiles spread over the warps.
// A fragments come from the activations in shared memory, stored already
// rounded to BF16 with two consecutive inputs of one replica in one 32-bit
// word (row kp holds inputs 2kp, 2kp+1 of the 32 replicas; row stride
// kActStride = 40 words, so the 8 row groups x 4 column pairs of a fragment
// load hit 32 distinct banks).  B fragments come straight from the BF16
// weight rows in global memory (12.9 KB, L1-resident; two consecutive
// inputs of one unit are one 32-bit word).  Bias and tanh in the FP32
// epilogue, which packs the lane's two units back into one word.  K is
// padded to 16 (first layer) and the 26 outputs to 32 with zeros; the
// outputs stay FP32 (row stride kOutStride).  (32 x 64 tiles are below
// tcgen05's smallest M of 64, and the step is latency-bound.)  Fragment
// layouts: PTX ISA, "Matrix Fragments for mma.m16n8k16 with floating point
// type".
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ void mma_bf16_16816(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int kActStride = 40;    // words per packed activation row (32 replicas + 8 pad)
constexpr int kOutStride = 36;    // floats per output row (32 replicas + 4 pad)

// One layer: X [ceil(K/2)][kActStride] packed BF16 pairs in shared memory ->
// Y, packed the same way (HIDDEN: tanh) or FP32 [units][kOutStride] (the
// output layer); weights w[u*K + k] (BF16, global), bias bias[u]
template <int K, int UNITS, bool HIDDEN>
__device__ __forceinline__ void mlp_layer_mma(const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ bias,
                                              const uint32_t* X, void* Y, int warp, int W, int lane) {
    constexpr int KP = K < 16 ? 16 : K;          // padded K
    constexpr int NT = (UNITS + 7) / 8;          // n8 tiles
    const int g = lane >> 2, t = lane & 3;
    for (int nt = warp; nt < NT; nt += W) {
        const int u = nt * 8 + g;                // this lane's unit for the B fragment
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int k0 = 0; k0 < KP; k0 += 16) {
            const int ka = k0 + 2 * t, kb = ka + 8;
            uint32_t b0 = 0u, b1 = 0u;
            if (u < UNITS) {
                if (ka < K) b0 = __ldg(reinterpret_cast<const unsigned int*>(w + u * K + ka));
                if (kb < K) b1 = __ldg(reinterpret_cast<const unsigned int*>(w + u * K + kb));
            }
            const uint32_t* xa = X + (ka >> 1) * kActStride;
            const uint32_t* xb = X + (kb >> 1) * kActStride;
#pragma unroll
            for (int mt = 0; mt < 2; mt++) {
                const int r = mt * 16 + g;
                mma_bf16_16816(acc[mt], ka < K ? xa[r] : 0u, ka < K ? xa[r + 8] : 0u, kb < K ? xb[r] : 0u,
                               kb < K ? xb[r + 8] : 0u, b0, b1);
            }
        }
        // epilogue: D element (row g (+8), col 2t (+1)) -> unit u0 (+1), replica mt*16 + g (+8)
        const int u0 = nt * 8 + 2 * t;
        const float bb0 = u0 < UNITS ? __bfloat162float(bias[u0]) : 0.f;
        const float bb1 = u0 + 1 < UNITS ? __bfloat162float(bias[u0 + 1]) : 0.f;
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
            const int r = mt * 16 + g;
            float z00 = acc[mt][0] + bb0, z01 = acc[mt][1] + bb1;       // replica r
            float z10 = acc[mt][2] + bb0, z11 = acc[mt][3] + bb1;       // replica r + 8
            if (HIDDEN) {
                uint32_t* Yp = static_cast<uint32_t*>(Y) + (u0 >> 1) * kActStride;
                Yp[r] = pack_bf16x2(tanhf(z00), tanhf(z01));
                Yp[r + 8] = pack_bf16x2(tanhf(z10), tanhf(z11));
            } else {
                float* Yf = static_cast<float*>(Y);
                if (u0 < UNITS) { Yf[u0 * kOutStride + r] = z00; Yf[u0 * kOutStride + r + 8] = z10; }
                if (u0 + 1 < UNITS) { Yf[(u0 + 1) * kOutStride + r] = z01; Yf[(u0 + 1) * kOutStride + r + 8] = z11; }
            }
        }
    }
}

// features (bufA rows 0..3) -> hidden 1 (bufB) -> hidden 2 (bufA) -> outputs
// (bufB, FP32); a barrier after each layer (called by every thread of the CTA).
// Each buffer is read only by the layer after the one that wrote it.
__device__ __forceinline__ void mlp_block(const __nv_bfloat16* __restrict__ w, uint32_t* bufA, uint32_t* bufB,
                                          int warp, int W, int lane) {
    mlp_layer_mma<kMlpIn, kMlpHidden, true>(w + kOffW1, w + kOffB1, bufA, bufB, warp, W, lane);
    __syncthreads();
    mlp_layer_mma<kMlpHidden, kMlpHidden, true>(w + kOffW2, w + kOffB2, bufB, bufA, warp, W, lane);
    __syncthreads();
    mlp_layer_mma<kMlpHidden, kMlpOut, false>(w + kOffW3, w + kOffB3, bufA, bufB, warp, W, lane);
    __syncthreads();
}

// the features of one replica into packed row pairs of bufA (lane = replica)
__device__ __forceinline__ void store_features(uint32_t* bufA, const float* f, int lane) {
#pragma unroll
    for (int kp = 0; kp < kMlpIn / 2; kp++) bufA[kp * kActStride + lane] = pack_bf16x2(f[2 * kp], f[2 * kp + 1]);
}

__device__ __forceinline__ float argf(float2 a) { return atan2f(a.y, a.x); }

// TMA chunks in flight per warp.  Two (one being read, one loading) keep the
// kernel's shared memory under a third of the SM's, so three CTAs of 8 warps
// share an SM (a chunk takes longer to read than to load from L2).
constexpr int kLStages = 2;
// two network buffers of 32 packed rows each (the outputs, 26 FP32 rows of
// kOutStride, fit in one)
constexpr int kMlpBufWords = (kMlpHidden / 2) * kActStride;
static_assert(kMlpOut * kOutStride <= kMlpBufWords, "output rows fit a network buffer");

// The sums of a move's two lists are taken by 2 C W chains (list, warp of the
// block shape); a CTA of kLWarps warps reads `chains` of them, chain x * chains + q
// on warp q % kLWarps of CTA x of the P.exec CTAs that run a replica block.
constexpr int kLWarps = 8;
struct LearnLayout {
    int rings;                                  // warps that read lists
    size_t ring, bars, buf, xch, parts, flag, total;
    // sums: what the CTAs exchange, all chains or (grouped) the sums of the shape's CTAs
    __host__ __device__ LearnLayout(int N, int sums, int exec, int chains, bool grouped) {
        rings = chains < kLWarps ? chains : kLWarps;
        size_t at = (size_t)(N + 1) * kRepBlock * sizeof(float2);           // amplitudes
        ring = at;
        at += (size_t)rings * kLStages * kStage * sizeof(int2);
        bars = at;
        at += (size_t)rings * kLStages * sizeof(uint64_t);
        buf = at;                               // two network buffers
        at += (size_t)2 * kMlpBufWords * sizeof(uint32_t);
        xch = at;                               // the roles' exchange rows
        at += (size_t)kXchRows * kRepBlock * sizeof(float);
        parts = (at + 15) & ~(size_t)15;        // partial fields, double-buffered across CTAs; then, grouped, this CTA's
        at = parts + (size_t)((exec > 1 ? 2 : 1) * sums + (grouped ? chains : 0)) * kRepBlock * sizeof(float2);
        flag = at;                              // the cluster's abort flag
        total = at + 16;
    }
};

// A warp's stream of chunks: per move its share of the sites' lists (pass 0), then of
// the pair's sub-lists (pass 1); in each, its one or two chains (list, part range).
struct LearnStream {
    uint32_t key0, key1;
    int N;
    const int* site_chunks;   // this sample's N*(kSplit+1) absolute chunk indices
    const int* pair_chunks;   // this sample's N(N-1)*(kSplit+1) pair sub-list chunk indices
    long long sweep0;
    int steps, total, n;      // n chains of this warp (0..2)
    int list[2], part0[2], part1[2];
    // the last pair pick of the consumer (slot 0) and of the prefetch cursor
    // (slot 1): each list lookup of a move reuses it instead of another Philox
    int cm[2] = {-1, -1}, ci[2] = {0, 0}, cj[2] = {0, 0};

    __device__ __forceinline__ void range(int m, int pass, int q, int& c, int& c_end, int slot) {
        if (m != cm[slot]) {
            const long long sw = sweep0 + m / steps;
            pair_pick(key0, key1, (uint64_t)sw, (uint32_t)(m % steps), N, ci[slot], cj[slot]);
            cm[slot] = m;
        }
        const int i0 = ci[slot], j0 = cj[slot];
        const int li = q ? list[1] : list[0];
        const int* sc = pass == 0 ? site_chunks + (li ? j0 : i0) * (kSplit + 1)
                                  : pair_chunks + (2 * (j0 * (j0 - 1) / 2 + i0) + li) * (kSplit + 1);
        c = __ldg(sc + (q ? part0[1] : part0[0]));
        c_end = __ldg(sc + (q ? part1[1] : part1[0]));
    }
    // cursor of the copies: at move m, pass and chain `at`, chunk c of [c, c_end)
    int m = 0, at = 0, c = 0, c_end = 0;
    __device__ __forceinline__ void next() {    // m == total at the end
        c++;
        while (c >= c_end) {
            if (++at == 2 * n) {
                at = 0;
                if (++m >= total) return;
            }
            range(m, at >= n, at >= n ? at - n : at, c, c_end, 1);
        }
    }
    __device__ __forceinline__ void first() {
        if (n == 0) m = total;
        if (m >= total) return;
        range(0, 0, 0, c, c_end, 1);
        c--;
        next();
    }
};

// One replica block on P.exec CTAs (CL: a thread-block cluster of more than one):
// each reads its chains' share of the lists, the chains' partial fields of both
// passes meet in every CTA's buffer (distributed shared memory, one cluster barrier
// per exchange, double-buffered by exchange parity) and are added there in the order
// of the block shape (the warps of a CTA of the shape, then its CTAs); every CTA then
// evaluates the network and takes the same decision on the same numbers, so the
// amplitude copies stay identical; rank 0 writes records, trace and results.
// kOne: one CTA has the SM (256 registers; loads of a tile ahead), else three share it.
// kGroup (full SMs, whole CTAs of the shape in a CTA): the sums of these go to the other
// CTAs, not every chain.  60 samples of N = 28, 96 replicas, 8 warps x 4 CTAs: with 64
// remote rows a pass into every CTA, summed by one warp, a sweep took 694 us (learned
// 1492), now 468 (1001).
template <bool CL, bool kOne, bool kGroup>
__global__ void __launch_bounds__(32 * kLWarps, kOne ? 1 : 3)
    learned_sweep_kernel(const SweepParams P, const LearnParams L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int X = CL ? P.exec : 1, CW = P.cluster * P.warps;
    const uint32_t rank = CL ? cluster_rank() : 0u;
    const bool writer = rank == 0;
    const Unit U = P.units[blockIdx.x / X];
    const SampleDev S = P.samples[U.sample];
    const int N = S.N, R = S.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kLWarps;
    const bool learned = L.mode == 2;
    float2* sp = reinterpret_cast<float2*>(smem_raw);
    const LearnLayout Lo(N, kGroup ? 2 * P.cluster : 2 * CW, X, P.chains, kGroup);
    int2* ring = reinterpret_cast<int2*>(smem_raw + Lo.ring) + (size_t)warp * kLStages * kStage;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + Lo.bars) + warp * kLStages;
    uint32_t* bufA = reinterpret_cast<uint32_t*>(smem_raw + Lo.buf);
    uint32_t* bufB = bufA + kMlpBufWords;
    const float* outs = reinterpret_cast<const float*>(bufB);
    float* xch = reinterpret_cast<float*>(smem_raw + Lo.xch);
    auto out_of = [&](int o) { return outs[o * kOutStride + lane]; };
    float2* parts = reinterpret_cast<float2*>(smem_raw + Lo.parts);      // [parity][2 C W][32] ([parity][2 C][32])
    int* cflag = reinterpret_cast<int*>(smem_raw + Lo.flag);             // cluster abort flags, by parity

    const bool active = lane < U.rep_count;
    const int64_t gr = S.rep_off + U.rep_begin + lane;
    for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
        const int site = idx >> 5, l = idx & 31;
        float2 v = make_float2(1.f, 0.f);
        if (l < U.rep_count) v = P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l];
        sp[idx] = v;
    }
    if (threadIdx.x < kRepBlock) sp[N * kRepBlock + threadIdx.x] = make_float2(1.f, 0.f);
    if (CL && threadIdx.x < 2) cflag[threadIdx.x] = 0;

    double E = 0.0, beta_d = 0.0;
    float beta = 0.f;
    long long nacc = 0, nprop = 0;
    uint32_t k0 = 0, k1 = 0;
    if (active) {                               // every warp may run a sampling role
        const uint64_t key = P.key[gr];
        k0 = (uint32_t)key;
        k1 = (uint32_t)(key >> 32);
    }
    if (warp == 0 && active) {
        E = P.energy[gr];
        beta_d = P.beta[gr];
        beta = (float)beta_d;
    }
    const long long sweep0 = *P.sweep_counter;
    const int steps = N / 2, total = P.nsweeps * steps;
    LearnStream st;
    st.key0 = S.pair_key0;
    st.key1 = S.pair_key1;
    st.N = N;
    st.site_chunks = P.site_chunks_g + S.split_off;   // built with the pair sub-lists (set_proposal)
    st.pair_chunks = P.pair_chunks + S.pair_off;
    st.sweep0 = sweep0;
    st.steps = steps;
    st.total = total;
    const int chain0 = (int)rank * P.chains + warp;   // this warp's chains: chain0, chain0 + kLWarps
    st.n = 0;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int ch = chain0 + q * kLWarps, g = ch % CW;
        if (warp + q * kLWarps < P.chains && ch < 2 * CW) st.n = q + 1;
        st.list[q] = ch / CW;
        st.part0[q] = g * (kSplit / CW);
        st.part1[q] = (g + 1) * (kSplit / CW);
    }
    if (lane == 0 && warp < Lo.rings) {
        for (int s = 0; s < kLStages; s++) mbar_init(bars + s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_shared();
    }
    __syncwarp();
    st.first();
    uint32_t issued = 0, consumed = 0;
    bool ok_wait = true;
    auto issue = [&]() {
        if (st.m >= total) return;
        const uint32_t slot = issued % kLStages;
        if (lane == 0) {
            const int64_t b = __ldg(P.chunk_start + st.c), e = __ldg(P.chunk_start + st.c + 1);
            const uint32_t bytes = (uint32_t)((e - b) * sizeof(int2));
            mbar_expect_tx(bars + slot, bytes);
            bulk_g2s(ring + slot * kStage, P.entries + b, bytes, bars + slot);
        }
        issued++;
        st.next();
    };
    for (int s = 0; s < kLStages; s++) issue();
    __shared__ __align__(8) uint64_t stall_bar;      // test hook: nothing arrives on it
    if (threadIdx.x == 0 && P.stall_move >= 0) {
        mbar_init(&stall_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (CL) cluster_sync();                    // every CTA runs before the first remote store
    uint32_t xchg = 0;                         // exchanges so far (buffer parity)
    bool aborted = false;                      // set uniformly over the CTA (cluster) by reduce()

    // this warp's chains over the sites' lists (second 0) or the pair's sub-lists (1);
    // tiles or groups
    auto pass = [&](int m, int second, float (&h)[2][2]) {
        const int tiles = second ? S.tiles_p : S.tiles_g;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            h[q][0] = h[q][1] = 0.f;
            if (q >= st.n || !ok_wait) continue;
            int c, c_end;
            st.range(m, second, q, c, c_end, 0);
            for (; c < c_end; c++) {
                const uint32_t slot = consumed % kLStages;
                ok_wait = ring_wait(bars + slot, (consumed / kLStages) & 1u, P.status, P.wait_clocks);
                if (!ok_wait) break;               // stop consuming and issuing; abort in reduce()
                const int n = (int)(__ldg(P.chunk_start + c + 1) - __ldg(P.chunk_start + c));
                if (!tiles) accumulate_chunk(ring + slot * kStage, n, sp, lane, h[q][0], h[q][1]);
                else if (kOne) accumulate_tiles_1<8, 4, true>(ring + slot * kStage, n, sp, lane, h[q][0], h[q][1]);
                else accumulate_tiles_1<2, 2, false>(ring + slot * kStage, n, sp, lane, h[q][0], h[q][1]);
                consumed++;
                __syncwarp();
                if (lane == 0) fence_async_shared();
                issue();
            }
        }
    };
    // kGroup: the sums of this CTA's whole CTAs of the shape -> warp 0 of every CTA
    auto reduce_groups = [&](const float (&h)[2][2]) {
        float2* buf = parts + (size_t)(xchg & 1u) * 2 * P.cluster * kRepBlock;
        float2* own = parts + (size_t)4 * P.cluster * kRepBlock;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (q < st.n) own[(warp + q * kLWarps) * kRepBlock + lane] = make_float2(h[q][0], h[q][1]);
        if (!ok_wait && lane == 0)
            for (int r = 0; r < X; r++) st_cluster_u32(cflag + (xchg & 1u), (uint32_t)r, 1u);
        __syncthreads();
        const int groups = P.chains / P.warps;
        for (int u = warp; u < groups; u += W) {
            float2 s = make_float2(0.f, 0.f);
            for (int w = u * P.warps; w < (u + 1) * P.warps; w++) {
                const float2 a = own[w * kRepBlock + lane];
                s.x += a.x;
                s.y += a.y;
            }
            for (int r = 0; r < X; r++) st_cluster_f2(buf + ((int)rank * groups + u) * kRepBlock + lane, (uint32_t)r, s);
        }
        cluster_sync();
        aborted = ((volatile int*)cflag)[xchg & 1u] != 0;
        xchg++;
        float4 hs = make_float4(0.f, 0.f, 0.f, 0.f);
        if (aborted || warp != 0) return hs;
        for (int c = 0; c < P.cluster; c++) {
            const float2 a = buf[c * kRepBlock + lane], b = buf[(P.cluster + c) * kRepBlock + lane];
            if (c == 0) hs = make_float4(a.x, a.y, b.x, b.y);
            else { hs.x += a.x; hs.y += a.y; hs.z += b.x; hs.w += b.y; }
        }
        return hs;
    };
    // partial sums of all chains -> warp 0 of every CTA.  Also agrees on an abort:
    // a warp whose wait ran out makes the whole CTA (and, through the flag, the
    // whole cluster) set `aborted` here.
    auto reduce = [&](const float (&h)[2][2]) {
        if constexpr (kGroup) return reduce_groups(h);
        float2* buf = parts + (CL ? (size_t)(xchg & 1u) * 2 * CW * kRepBlock : 0);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (q >= st.n) continue;
            float2* to = buf + (size_t)(chain0 + q * kLWarps) * kRepBlock + lane;
            const float2 v = make_float2(h[q][0], h[q][1]);
            if (!CL) *to = v;
            else
                for (int r = 0; r < X; r++) st_cluster_f2(to, (uint32_t)r, v);
        }
        float4 hs = make_float4(0.f, 0.f, 0.f, 0.f);
        if (CL) {
            if (!ok_wait && lane == 0)
                for (int r = 0; r < X; r++) st_cluster_u32(cflag + (xchg & 1u), (uint32_t)r, 1u);
            cluster_sync();
            aborted = ((volatile int*)cflag)[xchg & 1u] != 0;
            xchg++;
        } else {
            aborted = __syncthreads_or(!ok_wait) != 0;
        }
        if (aborted || warp != 0) return hs;
        for (int c = 0; c < P.cluster; c++) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w = c * P.warps; w < (c + 1) * P.warps; w++) {
                const float2 a = buf[w * kRepBlock + lane], b = buf[(CW + w) * kRepBlock + lane];
                s.x += a.x; s.y += a.y; s.z += b.x; s.w += b.y;
            }
            if (c == 0) hs = s;
            else { hs.x += s.x; hs.y += s.y; hs.z += s.z; hs.w += s.w; }
        }
        return hs;
    };

    for (int m = 0; m < total; m++) {
        const long long sw = sweep0 + m / steps;
        const int k = m % steps;
        int i0, j0;
        pair_pick(S.pair_key0, S.pair_key1, (uint64_t)sw, (uint32_t)k, N, i0, j0);

        // ---- fields at x: h_i (with a_j), h_j (with a_i) ---------------------------
        float h[2][2];
        if (m == P.stall_move) ok_wait = stall_wait(&stall_bar, P.status, P.wait_clocks);
        pass(m, 0, h);
        const float4 hs1 = reduce(h);
        if (aborted) break;
        float2 ai = make_float2(0.f, 0.f), aj = ai, ain = ai, ajn = ai;
        const float2 hi1 = make_float2(hs1.x, hs1.y), hj1 = make_float2(hs1.z, hs1.w);
        float cu = 0.f, lq_fwd = 0.f, lq_ratio = 0.f, tn = 0.5f, psi_i = 0.f, psi_j = 0.f, Ssum = 1.f;
        bool ok = true;
        MoveStream g = role_stream(k0, k1, (uint32_t)k, (uint64_t)sw, kAcceptBlock);   // accept and record draws
        if (warp == 0) {
            ai = sp[i0 * kRepBlock + lane];
            aj = sp[j0 * kRepBlock + lane];
            Ssum = fmaf(ai.x, ai.x, ai.y * ai.y) + fmaf(aj.x, aj.x, aj.y * aj.y);
            if (learned) {
                float f[kMlpIn];
                pair_features(ai, aj, hi1, hj1, beta, f);
                store_features(bufA, f, lane);
            }
        }
        // ---- proposal -------------------------------------------------------------
        if (learned) {
            __syncthreads();
            mlp_block(L.w, bufA, bufB, warp, W, lane);
            for (int r = warp; r < kRoles; r += W) learned_role(r, true, out_of, xch, lane, k0, k1, (uint32_t)k, sw);
            __syncthreads();
        }
        if (warp == 0) {
            if (!learned) {
                const U4 w = move_words(k0, k1, (uint64_t)sw, (uint32_t)k);
                propose<0>(ai, aj, w, ain, ajn);
                cu = u01f(w.w);
                tn = fmaf(ain.x, ain.x, ain.y * ain.y) / Ssum;
                psi_i = argf(ain) + argf(hi1);
                psi_j = argf(ajn) + argf(hj1);
            } else {
                // the roles' draws: t' = X/(X+Y) inside (kTEdge, 1 - kTEdge) and
                // both phases, else the move is rejected
                const float X = xch[X_X * 32 + lane], Y = xch[X_Y * 32 + lane];
                ok = X >= 0.f && Y >= 0.f && X + Y > 0.f && xch[X_OK0 * 32 + lane] != 0.f &&
                     xch[X_OK1 * 32 + lane] != 0.f;
                if (ok) {
                    tn = X / (X + Y);
                    ok = tn > kTEdge && tn < 1.0f - kTEdge;
                }
                if (ok) {
                    psi_i = xch[X_PSI0 * 32 + lane];
                    psi_j = xch[X_PSI1 * 32 + lane];
                    const float mi = sqrtf(Ssum * tn), mj = sqrtf(Ssum * (1.0f - tn));
                    float s1, c1, s2, c2;
                    sincosf(psi_i - argf(hi1), &s1, &c1);
                    sincosf(psi_j - argf(hj1), &s2, &c2);
                    ain = make_float2(mi * c1, mi * s1);
                    ajn = make_float2(mj * c2, mj * s2);
                    // log q_L(x'|x) = log Beta + both mixtures
                    lq_fwd = log_beta_pdf_lg(tn, xch[X_A * 32 + lane], xch[X_B * 32 + lane], xch[X_LGA * 32 + lane],
                                             xch[X_LGB * 32 + lane], xch[X_LGAB * 32 + lane]) +
                             xch[X_VM0 * 32 + lane] + xch[X_VM1 * 32 + lane] - log_plain_density(tn);
                } else {
                    ain = ai;
                    ajn = aj;
                }
                cu = g.uniform();
            }
            // the pair's slots hold the changes while the sub-lists are read:
            // every term there contains exactly one of a_i, a_j (linearly or
            // conjugated), so the sums are h_i(x') - h_i(x) and h_j(x') - h_j(x)
            sp[i0 * kRepBlock + lane] = make_float2(ain.x - ai.x, ain.y - ai.y);
            sp[j0 * kRepBlock + lane] = make_float2(ajn.x - aj.x, ajn.y - aj.y);
        }
        __syncthreads();

        // ---- field changes from the pair's sub-lists --------------------------------
        pass(m, 1, h);
        const float4 dh = reduce(h);
        if (aborted) break;
        float dE = 0.f;
        float2 hi2 = hi1, hj2 = hj1;
        if (warp == 0) {
            hi2 = make_float2(hi1.x + dh.x, hi1.y + dh.y);
            hj2 = make_float2(hj1.x + dh.z, hj1.y + dh.w);
            const float dix = ain.x - ai.x, diy = ain.y - ai.y, djx = ajn.x - aj.x, djy = ajn.y - aj.y;
            dE = -fmaf(dix, hi2.x, -diy * hi2.y) - fmaf(djx, hj1.x, -djy * hj1.y);
            if (learned) {
                float f[kMlpIn];
                pair_features(ain, ajn, hi2, hj2, beta, f);
                store_features(bufA, f, lane);
                // the reverse move's phases, measured from the fields at x'
                xch[X_PSI0 * 32 + lane] = argf(ai) + argf(hi2);
                xch[X_PSI1 * 32 + lane] = argf(aj) + argf(hj2);
            }
        }
        if (learned) {
            __syncthreads();
            mlp_block(L.w, bufA, bufB, warp, W, lane);
            for (int r = warp; r < kRoles; r += W) learned_role(r, false, out_of, xch, lane, k0, k1, (uint32_t)k, sw);
            __syncthreads();
        }
        if (warp == 0) {
            bool accept;
            if (!learned) {
                if (beta_d == 0.0) accept = true;
                else accept = (dE <= 0.f) || (cu < expf(-beta * dE));
            } else {
                // The sampler proposes t' only inside I = (1e-7, 1 - 1e-7), so the
                // move's density is q_L 1[t' in I]; the reverse move exists only
                // if the current t is in I as well.  Accepting only then gives
                // the transition density min(pi q_L, pi' q_L') 1[t in I] 1[t' in I],
                // symmetric in x and x'.
                const float t = fmaf(ai.x, ai.x, ai.y * ai.y) / Ssum;
                const bool t_in = t > kTEdge && t < 1.0f - kTEdge;
                if (t_in) {
                    const float lq_rev = log_beta_pdf_lg(t, xch[X_A * 32 + lane], xch[X_B * 32 + lane],
                                                         xch[X_LGA * 32 + lane], xch[X_LGB * 32 + lane],
                                                         xch[X_LGAB * 32 + lane]) +
                                         xch[X_VM0 * 32 + lane] + xch[X_VM1 * 32 + lane] - log_plain_density(t);
                    lq_ratio = lq_rev - lq_fwd;
                }
                accept = ok && t_in && (logf(cu) < -beta * dE + lq_ratio);
            }
            sp[i0 * kRepBlock + lane] = accept ? ain : ai;
            sp[j0 * kRepBlock + lane] = accept ? ajn : aj;
            if (accept) {
                E += (double)dE;
                nacc++;
            }
            nprop++;
            if (!learned && accept && active && writer && L.records != nullptr && u01f(g.next()) < L.rec_prob) {
                float f[kMlpIn];
                pair_features(ai, aj, hi1, hj1, beta, f);
                const unsigned long long slot = atomicAdd(L.rec_count, 1ull) % (unsigned long long)L.rec_cap;
                float* rec = L.records + slot * kRecordFloats;
                for (int q = 0; q < kMlpIn; q++) rec[q] = f[q];
                // t' within float range of (0, 1): log t' and log(1-t') stay finite
                rec[kMlpIn] = fminf(fmaxf(tn, 1e-6f), 1.0f - 1e-6f);
                rec[kMlpIn + 1] = psi_i;
                rec[kMlpIn + 2] = psi_j;
            }
            if (writer && P.trace != nullptr && U.sample == P.trace_sample && U.rep_begin + lane == P.trace_rep &&
                active) {
                const long long idx = (sw - P.trace_sweep0) * steps + k;
                if (idx >= 0 && idx < P.trace_cap) {
                    pspin_move_record* r = reinterpret_cast<pspin_move_record*>(P.trace) + idx;
                    r->i0 = i0; r->j0 = j0;
                    r->ai_old[0] = ai.x; r->ai_old[1] = ai.y; r->aj_old[0] = aj.x; r->aj_old[1] = aj.y;
                    r->ai_new[0] = ain.x; r->ai_new[1] = ain.y; r->aj_new[0] = ajn.x; r->aj_new[1] = ajn.y;
                    r->dE = dE;
                    r->accepted = accept ? 1 : 0;
                    r->log_q_ratio = lq_ratio;
                    r->log_u = logf(cu);
                }
            }
        }
        __syncthreads();
    }
    if (aborted && warp < Lo.rings) drain_ring(bars, kLStages, consumed, issued, P.status);   // state stays as before the launch
    if (writer && !aborted) {
        for (int idx = threadIdx.x; idx < N * kRepBlock; idx += blockDim.x) {
            const int site = idx >> 5, l = idx & 31;
            if (l < U.rep_count) P.spins[S.spin_off + (int64_t)site * R + U.rep_begin + l] = sp[idx];
        }
        if (warp == 0 && active) {
            P.energy[gr] = E;
            P.accepted[gr] += nacc;
            P.proposed[gr] += nprop;
        }
    }
    if (CL) cluster_sync();                    // no CTA leaves while a remote store may target it
}

using LearnKernel = void (*)(const SweepParams, const LearnParams);
static LearnKernel learned_kernel(const LearnPlan& r) {
    if (r.grouped) return learned_sweep_kernel<true, false, true>;
    return r.exec > 1 ? (r.one ? learned_sweep_kernel<true, true, false> : learned_sweep_kernel<true, false, false>)
                      : (r.one ? learned_sweep_kernel<false, true, false> : learned_sweep_kernel<false, false, false>);
}

// The launch of a plan; `attr` is its cluster dimension.
static size_t learned_smem(const LearnPlan& r, int warps, int C, int max_N) {
    return LearnLayout(max_N, r.grouped ? 2 * C : 2 * C * warps, r.exec, r.chains, r.grouped != 0).total;
}

static cudaError_t learned_config(const LearnPlan& r, int n_units, size_t smem, cudaStream_t st,
                                  cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    const LearnKernel kern = learned_kernel(r);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && r.exec > 8)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(n_units * r.exec));
    cfg.blockDim = dim3((unsigned)(32 * kLWarps));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)r.exec;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = r.exec > 1 ? 1 : 0;
    return e;
}

// As many CTAs per replica block as the blocks can all have at once with an SM for
// each CTA (8 at most, no more than there are chains), or up to the shape's own where
// these share SMs; else as few as hold the chains, two a warp: chains on more SMs
// finish sooner, a second wave costs twice.  A move
// of 24 blocks at N = 64 (gamma = 0.1, 8 warps x 2 CTAs) took 128 us on 2 CTAs
// each, 84 on 6 (144 CTAs, but clusters of 6 do not tile the chip: two waves), 46
// on the most that run at once; of 3 blocks 117 and 41 (8 CTAs); of 12 fully
// connected blocks at N = 48 (one CTA's shape) 113 and 53; 60 samples of N = 28, 96
// replicas, 4 warps x 8 CTAs, a sweep 1102 us on the shape's 8 CTAs, 474 on 4.  Where so
// few CTAs have no room for the amplitudes beside their lists' share, the fewest that
// have.
bool plan_learned_sweep(LearnPlan& r, int warps, int cluster, int n_units, int max_N) {
    const int C = cluster > 1 ? cluster : 1, all = 2 * C * warps;
    if (warps < 1 || n_units < 1 || C > 16 || kSplit % (C * warps) != 0) return false;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    // blocks that run at once on X CTAs each (0: they do not fit)
    auto resident = [&](int X) {
        r = LearnPlan{X, (all + X - 1) / X, (long long)n_units * X <= sms, 0};
        if (r.chains * (X - 1) >= all) return 0;                     // a CTA without a chain
        r.grouped = X > 1 && !r.one && warps >= 4 && r.chains % warps == 0 && r.chains * X == all;
        if (learned_smem(r, warps, C, max_N) > kRingSmemMax) return 0;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        int fit = 1;
        cudaError_t e = learned_config(r, n_units, learned_smem(r, warps, C, max_N), nullptr, cfg, attr);
        if (e == cudaSuccess && X > 1) e = cudaOccupancyMaxActiveClusters(&fit, learned_kernel(r), &cfg);
        if (e == cudaSuccess) return fit;
        cudaGetLastError();
        return 0;
    };
    const int least = (all + 2 * kLWarps - 1) / (2 * kLWarps), most = std::max(C, std::min({8, sms / n_units, all}));
    for (int X = most; X > least; X--)
        if (resident(X) >= n_units) return true;
    for (int X = least; X <= 16 && X <= all; X++)
        if (resident(X) > 0) return true;
    return false;
}

cudaError_t launch_learned_sweep(const SweepParams& p, const LearnParams& l, const LearnPlan& r, int n_units, int max_N,
                                 cudaStream_t st) {
    if (n_units <= 0) return cudaSuccess;
    if (p.pair_chunks == nullptr) return cudaErrorInvalidValue;
    SweepParams q = p;
    q.cluster = p.cluster > 1 ? p.cluster : 1;
    q.exec = r.exec;
    q.chains = r.chains;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    cudaError_t e = learned_config(r, n_units, learned_smem(r, p.warps, q.cluster, max_N), st, cfg, attr);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, learned_kernel(r), q, l);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// ------------------------------------------------------------------ training
// Forward, backward and gradient of one minibatch in one kernel (FP32 master
// weights).  A CTA of 8 warps takes tiles of 32 records, lane = record: the
// warps share each layer's units, activations and deltas stay in shared
// memory (rows of kTrainRow words, one per unit), and the tile's contribution
// to every parameter's gradient is added to registers (a thread owns a 4 x 4
// patch of W2 and its share of the rest).  kTrainCtas CTAs at most, each
// taking every kTrainCtas-th tile, then one partial gradient per CTA: the
// summation order depends on the batch size alone.  With one thread per
// record and activations in global memory, and one thread per parameter
// summing over all records, a step at batch 4096 took 525 us on 32 and 26
// blocks; 27 us + 5 us (sum and Adam).
constexpr int kTrainCtas = 296;                 // two per SM
constexpr int kTrainRow = 36;                   // 32 records + 4: rows 16-byte aligned, float4 reads conflict-free
constexpr int kTrainRows = kMlpIn + 4 * kMlpHidden + 2 * kMlpOut;    // f, h1, h2, d1, d2, out, d3
constexpr int kTrainWeights = (kMlpParams + 3) & ~3;
constexpr size_t kTrainSmem = (size_t)(kTrainWeights + kTrainRows * kTrainRow + 3 * 32) * sizeof(float);

__global__ void __launch_bounds__(256, 2) mlp_train_kernel(const float* __restrict__ wg, const float* __restrict__ records,
                                                           unsigned long long filled, uint32_t key0, uint32_t key1,
                                                           uint32_t step, int n, float* __restrict__ partial,
                                                           float* __restrict__ loss) {
    extern __shared__ __align__(16) float tsm[];
    float* w = tsm;
    float* f = w + kTrainWeights;
    float* h1 = f + kMlpIn * kTrainRow;
    float* h2 = h1 + kMlpHidden * kTrainRow;
    float* d1 = h2 + kMlpHidden * kTrainRow;
    float* d2 = d1 + kMlpHidden * kTrainRow;
    float* ot = d2 + kMlpHidden * kTrainRow;
    float* d3 = ot + kMlpOut * kTrainRow;
    float* lp = d3 + kMlpOut * kTrainRow;       // [3][32] parts of log q
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ti = tid >> 4, tj = tid & 15;
    for (int i = tid; i < kMlpParams; i += 256) w[i] = wg[i];
    float g2[4][4], g3[2][4], g1[4];            // W2 patch; W3 patch; W1 column or biases
#pragma unroll
    for (int a = 0; a < 4; a++) {
        g1[a] = 0.f;
#pragma unroll
        for (int b = 0; b < 4; b++) g2[a][b] = 0.f;
    }
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) g3[a][b] = 0.f;
    __syncthreads();
    const int tiles = (n + 31) / 32;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int b = tile * 32 + lane;
        const bool on = b < n;
        // the record: entry b, or a draw from the ring's `filled` entries
        const float* rec = records;
        if (on) {
            int64_t at = b;
            if (filled > 0) {
                const U4 r = philox4x32_10(U4{(uint32_t)b, step, 0x74726e00u, 0u}, key0, key1);
                at = (int)(((uint64_t)r.x * filled) >> 32);
            }
            rec = records + at * kRecordFloats;
        }
        f[warp * kTrainRow + lane] = on ? rec[warp] : 0.f;             // 8 warps, 8 features
        __syncthreads();
        {   // hidden 1: units 8 warp .. + 7
            float z[8];
#pragma unroll
            for (int q = 0; q < 8; q++) z[q] = w[kOffB1 + warp * 8 + q];
#pragma unroll
            for (int i = 0; i < kMlpIn; i++) {
                const float x = f[i * kTrainRow + lane];
#pragma unroll
                for (int q = 0; q < 8; q++) z[q] = fmaf(w[kOffW1 + (warp * 8 + q) * kMlpIn + i], x, z[q]);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) h1[(warp * 8 + q) * kTrainRow + lane] = tanhf(z[q]);
        }
        __syncthreads();
        {   // hidden 2
            float z[8];
#pragma unroll
            for (int q = 0; q < 8; q++) z[q] = w[kOffB2 + warp * 8 + q];
#pragma unroll 4
            for (int i = 0; i < kMlpHidden; i += 4) {
                float x[4];
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = h1[(i + u) * kTrainRow + lane];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float4 c = *reinterpret_cast<const float4*>(w + kOffW2 + (warp * 8 + q) * kMlpHidden + i);
                    z[q] = fmaf(c.x, x[0], z[q]);
                    z[q] = fmaf(c.y, x[1], z[q]);
                    z[q] = fmaf(c.z, x[2], z[q]);
                    z[q] = fmaf(c.w, x[3], z[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 8; q++) h2[(warp * 8 + q) * kTrainRow + lane] = tanhf(z[q]);
        }
        __syncthreads();
        {   // outputs warp, warp + 8, ...
            float z[4];
#pragma unroll
            for (int q = 0; q < 4; q++) z[q] = warp + 8 * q < kMlpOut ? w[kOffB3 + warp + 8 * q] : 0.f;
#pragma unroll 4
            for (int i = 0; i < kMlpHidden; i += 4) {
                float x[4];
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = h2[(i + u) * kTrainRow + lane];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (warp + 8 * q < kMlpOut) {
                        const float4 c = *reinterpret_cast<const float4*>(w + kOffW3 + (warp + 8 * q) * kMlpHidden + i);
                        z[q] = fmaf(c.x, x[0], z[q]);
                        z[q] = fmaf(c.y, x[1], z[q]);
                        z[q] = fmaf(c.z, x[2], z[q]);
                        z[q] = fmaf(c.w, x[3], z[q]);
                    }
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (warp + 8 * q < kMlpOut) ot[(warp + 8 * q) * kTrainRow + lane] = z[q];
        }
        __syncthreads();
        if (warp < 3) {   // the loss: warp 0 the Beta law, warps 1 and 2 a site each
            auto out = [&](int o) { return ot[o * kTrainRow + lane]; };
            auto grad = [&](int o, float v) { d3[o * kTrainRow + lane] = on ? v : 0.f; };
            const float x = on ? rec[kMlpIn + warp] : 0.5f;
            lp[warp * 32 + lane] = warp == 0 ? loss_beta_grad(out, grad, x) : loss_site_grad(warp - 1, out, grad, x);
        }
        __syncthreads();
        if (warp == 7 && on) loss[b] = -((lp[lane] + lp[32 + lane]) + lp[64 + lane]);
        {   // deltas of hidden 2
            float z[8];
#pragma unroll
            for (int q = 0; q < 8; q++) z[q] = 0.f;
#pragma unroll 2
            for (int o = 0; o < kMlpOut; o++) {
                const float x = d3[o * kTrainRow + lane];
                const float4* c = reinterpret_cast<const float4*>(w + kOffW3 + o * kMlpHidden + warp * 8);
                const float4 c0 = c[0], c1 = c[1];
                z[0] = fmaf(c0.x, x, z[0]); z[1] = fmaf(c0.y, x, z[1]); z[2] = fmaf(c0.z, x, z[2]); z[3] = fmaf(c0.w, x, z[3]);
                z[4] = fmaf(c1.x, x, z[4]); z[5] = fmaf(c1.y, x, z[5]); z[6] = fmaf(c1.z, x, z[6]); z[7] = fmaf(c1.w, x, z[7]);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float h = h2[(warp * 8 + q) * kTrainRow + lane];
                d2[(warp * 8 + q) * kTrainRow + lane] = z[q] * (1.0f - h * h);
            }
        }
        __syncthreads();
        {   // deltas of hidden 1
            float z[8];
#pragma unroll
            for (int q = 0; q < 8; q++) z[q] = 0.f;
#pragma unroll 4
            for (int o = 0; o < kMlpHidden; o++) {
                const float x = d2[o * kTrainRow + lane];
                const float4* c = reinterpret_cast<const float4*>(w + kOffW2 + o * kMlpHidden + warp * 8);
                const float4 c0 = c[0], c1 = c[1];
                z[0] = fmaf(c0.x, x, z[0]); z[1] = fmaf(c0.y, x, z[1]); z[2] = fmaf(c0.z, x, z[2]); z[3] = fmaf(c0.w, x, z[3]);
                z[4] = fmaf(c1.x, x, z[4]); z[5] = fmaf(c1.y, x, z[5]); z[6] = fmaf(c1.z, x, z[6]); z[7] = fmaf(c1.w, x, z[7]);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float h = h1[(warp * 8 + q) * kTrainRow + lane];
                d1[(warp * 8 + q) * kTrainRow + lane] = z[q] * (1.0f - h * h);
            }
        }
        __syncthreads();
        // the tile's gradient: rows ti + 16a (deltas) x columns tj + 16c (activations), summed over the 32 records
        auto row4 = [](const float* p, int r, int b4) { return *reinterpret_cast<const float4*>(p + r * kTrainRow + b4); };
        auto dot4 = [](const float4 d, const float4 x, float s) {
            return fmaf(d.w, x.w, fmaf(d.z, x.z, fmaf(d.y, x.y, fmaf(d.x, x.x, s))));
        };
        const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll 2
        for (int b4 = 0; b4 < 32; b4 += 4) {
            float4 xa[4];
#pragma unroll
            for (int c = 0; c < 4; c++) xa[c] = row4(h1, tj + 16 * c, b4);
#pragma unroll
            for (int a = 0; a < 4; a++) {
                const float4 d = row4(d2, ti + 16 * a, b4);
#pragma unroll
                for (int c = 0; c < 4; c++) g2[a][c] = dot4(d, xa[c], g2[a][c]);
                if (tj == 9) g1[a] = dot4(d, one, g1[a]);                                  // b2
            }
#pragma unroll
            for (int c = 0; c < 4; c++) xa[c] = row4(h2, tj + 16 * c, b4);
#pragma unroll
            for (int a = 0; a < 2; a++)
                if (ti + 16 * a < kMlpOut) {
                    const float4 d = row4(d3, ti + 16 * a, b4);
#pragma unroll
                    for (int c = 0; c < 4; c++) g3[a][c] = dot4(d, xa[c], g3[a][c]);
                    if (tj == 10) g1[a] = dot4(d, one, g1[a]);                             // b3
                }
            if (tj <= 8) {                                                                  // W1, b1
                const float4 x = tj < 8 ? row4(f, tj, b4) : one;
#pragma unroll
                for (int a = 0; a < 4; a++) g1[a] = dot4(row4(d1, ti + 16 * a, b4), x, g1[a]);
            }
        }
        __syncthreads();
    }
    float* out = partial + (size_t)blockIdx.x * kMlpParams;
#pragma unroll
    for (int a = 0; a < 4; a++) {
#pragma unroll
        for (int c = 0; c < 4; c++) out[kOffW2 + (ti + 16 * a) * kMlpHidden + tj + 16 * c] = g2[a][c];
        if (tj < 8) out[kOffW1 + (ti + 16 * a) * kMlpIn + tj] = g1[a];
        if (tj == 8) out[kOffB1 + ti + 16 * a] = g1[a];
        if (tj == 9) out[kOffB2 + ti + 16 * a] = g1[a];
    }
#pragma unroll
    for (int a = 0; a < 2; a++)
        if (ti + 16 * a < kMlpOut) {
#pragma unroll
            for (int c = 0; c < 4; c++) out[kOffW3 + (ti + 16 * a) * kMlpHidden + tj + 16 * c] = g3[a][c];
            if (tj == 10) out[kOffB3 + ti + 16 * a] = g1[a];
        }
}

// Sums the CTAs' partial gradients (8 threads per parameter, fixed order),
// divides by the batch and, for a training step, applies Adam.
struct AdamParams {
    float *w, *m, *v;
    __nv_bfloat16* wbf;
    float lr, b1, b2, eps, c1, c2;
};

__global__ void __launch_bounds__(256) mlp_grad_adam_kernel(const float* __restrict__ partial, int parts, int n,
                                                            float* __restrict__ grad, const AdamParams A) {
    __shared__ float sums[8][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + x;
    float s = 0.f;
    if (p < kMlpParams)
#pragma unroll 8
        for (int c = y; c < parts; c += 8) s += partial[(size_t)c * kMlpParams + p];
    sums[y][x] = s;
    __syncthreads();
    if (y != 0 || p >= kMlpParams) return;
    s = sums[0][x];
#pragma unroll
    for (int q = 1; q < 8; q++) s += sums[q][x];
    const float gp = s / (float)n;
    grad[p] = gp;
    if (A.w == nullptr) return;
    const float mp = A.b1 * A.m[p] + (1.0f - A.b1) * gp, vp = A.b2 * A.v[p] + (1.0f - A.b2) * gp * gp;
    A.m[p] = mp;
    A.v[p] = vp;
    const float wp = A.w[p] - A.lr * (mp / A.c1) / (sqrtf(vp / A.c2) + A.eps);
    A.w[p] = wp;
    A.wbf[p] = __float2bfloat16_rn(wp);
}

__global__ void to_bf16_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wbf) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < kMlpParams) wbf[p] = __float2bfloat16_rn(w[p]);
}

size_t mlp_partial_floats() { return (size_t)kTrainCtas * kMlpParams; }

// Loss and gradient of the mean -log q_L over n records: entries 0..n-1, or
// (filled > 0) n draws from the ring's first `filled` entries; partial: the
// CTAs' partial gradients [mlp_partial_floats()].  adam_step > 0: then one
// Adam step (the adam_step-th) on w, m, v and the BF16 copy.
cudaError_t launch_mlp_train(float* w, const float* records, unsigned long long filled, uint64_t key, uint32_t step,
                             int n, float* partial, float* loss, float* grad, float* m, float* v, __nv_bfloat16* wbf,
                             float lr, int adam_step, cudaStream_t st) {
    const int tiles = (n + 31) / 32, ctas = tiles < kTrainCtas ? tiles : kTrainCtas;
    cudaError_t e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
    if (e != cudaSuccess) return e;
    mlp_train_kernel<<<ctas, 256, kTrainSmem, st>>>(w, records, filled, (uint32_t)key, (uint32_t)(key >> 32), step, n,
                                                    partial, loss);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    AdamParams A{};
    if (adam_step > 0) {
        const float b1 = 0.9f, b2 = 0.999f;
        A = AdamParams{w, m, v, wbf, lr, b1, b2, 1e-8f, 1.0f - powf(b1, (float)adam_step), 1.0f - powf(b2, (float)adam_step)};
    }
    mlp_grad_adam_kernel<<<(kMlpParams + 31) / 32, 256, 0, st>>>(partial, ctas, n, grad, A);
    return cudaGetLastError();
}
cudaError_t launch_to_bf16(const float* w, __nv_bfloat16* wbf, cudaStream_t st) {
    to_bf16_kernel<<<(kMlpParams + 255) / 256, 256, 0, st>>>(w, wbf);
    return cudaGetLastError();
}
}  // namespace pspin
