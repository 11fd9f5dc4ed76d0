// sweep_common.cuh -- device pieces shared by the sweep kernels: proposals,
// the per-warp TMA rings that stream site-list chunks into shared memory,
// and the field accumulation over one staged chunk.
#pragma once
#include <type_traits>

#include "internal.h"
#include "rng.cuh"

namespace pspin {

// The state-independent part of a move's proposal, from its four random
// words: t[0], t[1] = sin, cos of the rotation angle (sphere) or
// sqrt(1-u), sqrt(u) of the transfer (cube); t[2..5] = sin, cos of the two
// phases; t[6] = the Metropolis uniform.
template <int VARIANT>
__device__ __forceinline__ void move_trig(U4 w, float* t) {
    if (VARIANT == 0) {
        sincospif(2.0f * u01f(w.x), &t[0], &t[1]);
    } else {
        const float u = u01f_open0(w.x);
        t[0] = sqrtf(1.0f - u);
        t[1] = sqrtf(u);
    }
    sincospif(2.0f * u01f(w.y), &t[2], &t[3]);
    sincospif(2.0f * u01f(w.z), &t[4], &t[5]);
    t[6] = u01f(w.w);
}

// The state-dependent part: the proposed amplitudes from the current ones.
template <int VARIANT>
__device__ __forceinline__ void propose_with(float2 ai, float2 aj, const float* t, float2& ain, float2& ajn) {
    const float s1 = t[2], c1 = t[3], s2 = t[4], c2 = t[5];
    if (VARIANT == 0) {
        // spins.h:17-52: a_i' = a_i e^{-i phi1} sqrt((r1+r2)/r1) cos(alpha),
        //                a_j' = a_j e^{-i phi2} sqrt((r1+r2)/r2) sin(alpha)
        const float sa = t[0], ca = t[1];
        float r1 = fmaf(ai.x, ai.x, ai.y * ai.y);
        float r2 = fmaf(aj.x, aj.x, aj.y * aj.y);
        float s = r1 + r2;
        float f1 = sqrtf(s / r1) * ca;
        float f2 = sqrtf(s / r2) * sa;
        ain = make_float2(fmaf(ai.x, c1, ai.y * s1) * f1, fmaf(ai.y, c1, -ai.x * s1) * f1);
        ajn = make_float2(fmaf(aj.x, c2, aj.y * s2) * f2, fmaf(aj.y, c2, -aj.x * s2) * f2);
    } else {
        // spins_sparse.h:26-56: |a_i'|^2 = sqrt(S4) sqrt(1-u), |a_j'|^2 = sqrt(S4) sqrt(u),
        // absolute phases phi1, phi2
        float r1 = fmaf(ai.x, ai.x, ai.y * ai.y);
        float r2 = fmaf(aj.x, aj.x, aj.y * aj.y);
        float q = sqrtf(fmaf(r1, r1, r2 * r2));
        float m1 = sqrtf(q * t[0]);
        float m2 = sqrtf(q * t[1]);
        ain = make_float2(m1 * c1, m1 * s1);
        ajn = make_float2(m2 * c2, m2 * s2);
    }
}

template <int VARIANT>
__device__ __forceinline__ void propose(float2 ai, float2 aj, U4 w, float2& ain, float2& ajn) {
    float t[7];
    move_trig<VARIANT>(w, t);
    propose_with<VARIANT>(ai, aj, t, ain, ajn);
}

// ---------------------------------------------------------------- block state
// Prologue copies into shared memory with kInFlight independent loads per
// thread before their stores, so a CTA's state arrives in a few memory
// latencies rather than one per loop trip.
constexpr int kInFlight = 8;

// A replica block's amplitudes: columns [0, kb) of rows [0, N) of the
// sample's [site][R] array `src` (already offset to the block's first
// replica) into sp[site * kb + col]; columns >= rep_count are 1+0i.
__device__ __forceinline__ void load_block_amplitudes(float2* sp, const float2* src, int64_t R, int N, int kb,
                                                      int rep_count) {
    const int total = N * kb;
    const int step = (int)blockDim.x;
    for (int i0 = threadIdx.x; i0 < total; i0 += kInFlight * step) {
        float2 v[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; u++) {
            const int idx = i0 + u * step;
            const int site = idx / kb, col = idx - site * kb;
            v[u] = make_float2(1.f, 0.f);
            if (idx < total && col < rep_count) v[u] = __ldcg(src + site * R + col);
        }
#pragma unroll
        for (int u = 0; u < kInFlight; u++) {
            const int idx = i0 + u * step;
            if (idx < total) sp[idx] = v[u];
        }
    }
}

// n contiguous elements
template <class T>
__device__ __forceinline__ void load_block_range(T* dst, const T* src, int64_t n) {
    const int64_t step = blockDim.x;
    for (int64_t i0 = threadIdx.x; i0 < n; i0 += kInFlight * step) {
        T v[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; u++) {
            const int64_t idx = i0 + u * step;
            if (idx < n) v[u] = src[idx];
        }
#pragma unroll
        for (int u = 0; u < kInFlight; u++) {
            const int64_t idx = i0 + u * step;
            if (idx < n) dst[idx] = v[u];
        }
    }
}

// ---------------------------------------------------------------- TMA ring
// The streaming sweeps read the lists' chunks from rings of shared-memory slots,
// filled by 1-D bulk copies (cp.async.bulk, completion counted on one mbarrier per
// slot) ahead of the chunk being read; the pair schedule is known in advance, so
// the copies run across move boundaries.  Who issues them is each kernel's: a
// producer warp for all rings of a CTA (sweep_ring.cu), each warp for its own
// (learned.cu).  Waits are bounded (SweepParams::wait_clocks): a wait that runs out
// raises the status word, and the CTA (every CTA of a cluster) gives up without
// writing anything back.

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void fence_async_shared() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Bounded wait; returns false and raises `flag` in the status word when
// `limit` SM clocks pass before the phase completes.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, long long limit,
                                          int flag = kStatusTimeout) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > limit) {
            atomicOr(status, flag);
            return false;
        }
    }
    return true;
}

// A ring wait made warp-uniform: the warp goes on only if every lane saw
// the copy land.
__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, int* status, long long limit) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, status, limit));
}

// After an abort: lane 0 waits (bounded) for the copies this warp issued and
// never consumed, so that no bulk copy is still writing into shared memory
// when the CTA exits.  Completed phases pass at once (their parity is the
// previous phase's), so a copy whose wait gave up is waited for again here.
__device__ __forceinline__ void drain_ring(uint64_t* bars, int stages, uint32_t consumed, uint32_t issued,
                                           int* status) {
    if ((threadIdx.x & 31) == 0)
        for (uint32_t q = consumed; q < issued; q++)
            if (!mbar_wait(bars + q % stages, (q / stages) & 1u, status, kDrainClocks, kStatusDrain)) break;
    __syncwarp();
}

// Test hook: the bounded wait of every warp at move P.stall_move on an
// mbarrier that nothing arrives on, so the wait runs out and the kernel
// takes its abort path.
__device__ __forceinline__ bool stall_wait(uint64_t* bar, int* status, long long limit) {
    return ring_wait(bar, 0u, status, limit);
}

// Field contribution of the groups in one staged chunk for this lane's replica.
__device__ __forceinline__ void accumulate_chunk(const int2* __restrict__ R, int n,
                                                 const float2* __restrict__ sp, int lane,
                                                 float& hx, float& hy) {
    int e = 0;
    while (e < n) {
        const int2 h = R[e];
        const int len = h.x;
        const int p = h.y >> 16, o1 = h.y & 0xFFFF;
        const float2 ap = sp[p * kRepBlock + lane];
        const float2 ao = sp[o1 * kRepBlock + lane];
        // a_p * conj(a_o1)
        const float px = fmaf(ap.x, ao.x, ap.y * ao.y);
        const float py = fmaf(ap.y, ao.x, -ap.x * ao.y);
        float yx = 0.f, yy = 0.f;
        const int2* __restrict__ d = R + e + 1;
#pragma unroll 4
        for (int t = 0; t < len; t++) {
            const int2 v = d[t];
            const float g = __int_as_float(v.x);
            const float2 a = sp[v.y * kRepBlock + lane];
            yx = fmaf(g, a.x, yx);       // Y += g conj(a_o2)
            yy = fmaf(-g, a.y, yy);
        }
        hx = fmaf(px, yx, fmaf(-py, yy, hx));
        hy = fmaf(px, yy, fmaf(py, yx, hy));
        e += len + 1;
    }
}

// The same groups stored as 16-byte records {g, o2, p<<16|o1, last}, one
// per data entry: a record's position does not depend on an earlier header.
// Records are taken kUnroll at a time with their shared-memory loads (the
// records, then each record's a_o2, a_p, a_o1, the last two used only where
// the record ends a group) issued before the arithmetic, so a batch costs
// about two load latencies: for chains that wait on latency (a few warps
// per SM).  Kernels that fill the SMs use accumulate_records_k's one record
// at a time, which loads a_p, a_o1 once per group.  The arithmetic is
// accumulate_chunk's, operation for operation: Y accumulates the group's
// entries in order from zero and h takes a_p conj(a_o1) Y at the group's
// last record.  kSingle: every record ends its group (groups of one entry,
// the rule for sparse samples), so the test is compiled out.
template <bool kSingle>
__device__ __forceinline__ void record_step(const int4 q, const float2 a, const float2 ap, const float2 ao,
                                            float& yx, float& yy, float& hx, float& hy) {
    const float g = __int_as_float(q.x);
    yx = fmaf(g, a.x, yx);               // Y += g conj(a_o2)
    yy = fmaf(-g, a.y, yy);
    if (kSingle || q.w) {
        const float px = fmaf(ap.x, ao.x, ap.y * ao.y);
        const float py = fmaf(ap.y, ao.x, -ap.x * ao.y);
        hx = fmaf(px, yx, fmaf(-py, yy, hx));
        hy = fmaf(px, yy, fmaf(py, yx, hy));
        yx = 0.f;
        yy = 0.f;
    }
}

template <int kUnroll, bool kSingle = false>
__device__ __forceinline__ void accumulate_records(const int2* __restrict__ R2, int n,
                                                   const float2* __restrict__ sp, int lane,
                                                   float& hx, float& hy) {
    const int4* __restrict__ R = reinterpret_cast<const int4*>(R2);
    const int nr = n >> 1;
    float yx = 0.f, yy = 0.f;
    int r = 0;
    for (; r + kUnroll <= nr; r += kUnroll) {
        int4 q[kUnroll];
        float2 a[kUnroll], ap[kUnroll], ao[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; u++) q[u] = R[r + u];
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
            a[u] = sp[q[u].y * kRepBlock + lane];
            ap[u] = sp[(q[u].z >> 16) * kRepBlock + lane];
            ao[u] = sp[(q[u].z & 0xFFFF) * kRepBlock + lane];
        }
#pragma unroll
        for (int u = 0; u < kUnroll; u++) record_step<kSingle>(q[u], a[u], ap[u], ao[u], yx, yy, hx, hy);
    }
    for (; r < nr; r++) {
        const int4 q = R[r];
        record_step<kSingle>(q, sp[q.y * kRepBlock + lane], sp[(q.z >> 16) * kRepBlock + lane],
                             sp[(q.z & 0xFFFF) * kRepBlock + lane], yx, yy, hx, hy);
    }
}

// ---------------------------------------------------------------- dense tiles
// Field contribution of the tiles in one staged chunk (layout.cpp), for a
// block of 32K replicas stored [site][K][32] (replica k*32 + lane of the block
// at sp[(site*K + k)*32 + lane]).  A row is one broadcast read of its 4 or 8
// couplings and one gathered amplitude per replica for 8 or 16 FMA per
// replica; then each column's sum enters the field in column order,
//   h += a_p conj(a_o) Y,
// the arithmetic of accumulate_chunk on the columns' groups, operation for
// operation (a zero coupling leaves Y as it is, and a column without a group,
// the virtual site's, adds zero).
//
// Rows come in blocks of kUnroll, loads first, then the rest of 4, 2, 1.  The
// products are paired FMA over two columns (fma.rn.f32x2, the rounding of two
// single ones; couplings are neighbours in the row, the amplitude's two
// components are duplicated): an outer product's single FMA reads three new
// registers and issues at 1.25 cycles, so pairs cost the FMA pipe nothing and
// free half the issue slots for the loads.  With four warps a sub-partition,
// cycles per tile and warp, single -> paired: K = 3, 4 x 20 1045 -> 880, 8 x 32
// 2550 -> 2180; K = 1, 8 x 20 740 -> 645.  kLat, for a warp with a sub-partition
// to itself: the next tile's header and the columns' amplitudes are loaded ahead
// of the rows.  (Double-buffered row blocks with masked ends took 1.6 times as
// long: the masks cost more than the latency they hid.)
template <int K, int P, int kUnroll>
struct TileBlock {
    float4 c[kUnroll][P / 4];
    float2 a[kUnroll][K];
    __device__ __forceinline__ void load(const float4* __restrict__ C, const float2* __restrict__ A, int t) {
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
#pragma unroll
            for (int w = 0; w < P / 4; w++) c[u][w] = C[(t + u) * (P / 4) + w];
#pragma unroll
            for (int k = 0; k < K; k++) a[u][k] = A[((t + u) * K + k) * kRepBlock];
        }
    }
    __device__ __forceinline__ void add(float2 (&y)[K][P]) const {
#pragma unroll
        for (int u = 0; u < kUnroll; u++)
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float2 dx = make_float2(a[u][k].x, a[u][k].x), dy = make_float2(a[u][k].y, a[u][k].y);
#pragma unroll
                for (int w = 0; w < P / 4; w++) {
                    const float2 g0 = make_float2(c[u][w].x, c[u][w].y), g1 = make_float2(c[u][w].z, c[u][w].w);
                    y[k][4 * w + 0] = __ffma2_rn(g0, dx, y[k][4 * w + 0]);
                    y[k][4 * w + 1] = __ffma2_rn(g0, dy, y[k][4 * w + 1]);
                    y[k][4 * w + 2] = __ffma2_rn(g1, dx, y[k][4 * w + 2]);
                    y[k][4 * w + 3] = __ffma2_rn(g1, dy, y[k][4 * w + 3]);
                }
            }
    }
};

template <int K, int P, int kUnroll, bool kLat>
__device__ __forceinline__ void tile_body(const int4 h0, const int4 h1, const int4* __restrict__ T,
                                          const float2* __restrict__ sp, int lane, float (&hx)[K], float (&hy)[K]) {
    const int shared = h0.x & 0xFFFF, lo = h0.y & 0xFFFF, rows = (h0.y >> 16) & 0xFF;
    const bool shared_p = (h0.x & (2 << 16)) != 0;
    int v[P];
    v[0] = h0.z & 0xFFFF; v[1] = h0.z >> 16; v[2] = h0.w & 0xFFFF; v[3] = h0.w >> 16;
    if (P == 8) {
        v[P - 4] = h1.x & 0xFFFF; v[P - 3] = h1.x >> 16; v[P - 2] = h1.y & 0xFFFF; v[P - 1] = h1.y >> 16;
    }
    const float4* __restrict__ C = reinterpret_cast<const float4*>(T + P / 4);
    const float2* __restrict__ A = sp + (size_t)lo * K * kRepBlock + lane;
    float2 y[K][P];      // columns q, q+1 (q even): [q] their Re sums, [q + 1] their -Im sums
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int q = 0; q < P; q++) y[k][q] = make_float2(0.f, 0.f);
    constexpr bool kEarly = kLat && K == 1;       // registers for the columns' amplitudes
    float2 f[K], x[kEarly ? P : 1];
    if (kEarly)
#pragma unroll
        for (int q = 0; q < P; q++) x[q] = sp[v[q] * kRepBlock + lane];
    int t = 0;
#pragma unroll 1
    for (; t + kUnroll <= rows; t += kUnroll) {
        TileBlock<K, P, kUnroll> b;
        b.load(C, A, t);
        b.add(y);
    }
    auto rest = [&](auto count) {
        constexpr int n = decltype(count)::value;
        if (kUnroll > n && (rows & n)) {
            TileBlock<K, P, n> b;
            b.load(C, A, t);
            b.add(y);
            t += n;
        }
    };
    rest(std::integral_constant<int, 4>{});
    rest(std::integral_constant<int, 2>{});
    rest(std::integral_constant<int, 1>{});
#pragma unroll
    for (int k = 0; k < K; k++) f[k] = sp[(shared * K + k) * kRepBlock + lane];
    auto fold = [&](const float2 ap, const float2 ao, int k, int q) {
        const float px = fmaf(ap.x, ao.x, ap.y * ao.y);
        const float py = fmaf(ap.y, ao.x, -ap.x * ao.y);
        const int q0 = q & ~1;
        const float yr = q & 1 ? y[k][q0].y : y[k][q0].x, yi = q & 1 ? y[k][q0 + 1].y : y[k][q0 + 1].x;
        hx[k] = fmaf(px, yr, fmaf(py, yi, hx[k]));
        hy[k] = fmaf(-px, yi, fmaf(py, yr, hy[k]));
    };
    auto column = [&](int k, int q) { return kEarly ? x[kEarly ? q : 0] : sp[(v[q] * K + k) * kRepBlock + lane]; };
    if (shared_p) {
#pragma unroll
        for (int q = 0; q < P; q++)
#pragma unroll
            for (int k = 0; k < K; k++) fold(f[k], column(k, q), k, q);
    } else {
#pragma unroll
        for (int q = 0; q < P; q++)
#pragma unroll
            for (int k = 0; k < K; k++) fold(column(k, q), f[k], k, q);
    }
}

// k4, k8: rows per block in 4- and 8-column tiles
template <int K, int k4, int k8, bool kLat>
__device__ __forceinline__ void accumulate_tiles(const int2* __restrict__ R2, int n, const float2* __restrict__ sp,
                                                 int lane, float (&hx)[K], float (&hy)[K]) {
    const int4* __restrict__ R = reinterpret_cast<const int4*>(R2);
    const int n16 = n >> 1;
    const int4 none = make_int4(0, 0, 0, 0);
    int e = 0;
    int4 h0 = n16 > 0 ? R[0] : none, h1 = kLat && n16 > 1 ? R[1] : none;
    while (e < n16) {
        const int rows = (h0.y >> 16) & 0xFF;
        const bool wide = (h0.x & (1 << 16)) != 0;
        const int4* T = R + e;
        const int4 c0 = h0, c1 = kLat ? h1 : (wide ? T[1] : none);
        e += wide ? 2 + 2 * rows : 1 + rows;
        if (kLat) {
            h0 = e < n16 ? R[e] : none;
            h1 = e + 1 < n16 ? R[e + 1] : none;
        }
        if (wide) tile_body<K, 8, k8, kLat>(c0, c1, T, sp, lane, hx, hy);
        else tile_body<K, 4, k4, kLat>(c0, c1, T, sp, lane, hx, hy);
        if (!kLat && e < n16) h0 = R[e];
    }
}

// one replica per lane
template <int k4, int k8, bool kLat>
__device__ __forceinline__ void accumulate_tiles_1(const int2* __restrict__ R2, int n, const float2* __restrict__ sp,
                                                   int lane, float& hx, float& hy) {
    float hx1[1] = {hx}, hy1[1] = {hy};
    accumulate_tiles<1, k4, k8, kLat>(R2, n, sp, lane, hx1, hy1);
    hx = hx1[0];
    hy = hy1[0];
}

// Group records for K replicas per lane, one record at a time.
template <int K>
__device__ __forceinline__ void accumulate_records_k(const int2* __restrict__ R2, int n,
                                                     const float2* __restrict__ sp, int lane,
                                                     float (&hx)[K], float (&hy)[K]) {
    const int4* __restrict__ R = reinterpret_cast<const int4*>(R2);
    const int nr = n >> 1;
    float yx[K], yy[K];
#pragma unroll
    for (int k = 0; k < K; k++) yx[k] = yy[k] = 0.f;
#pragma unroll 4
    for (int r = 0; r < nr; r++) {
        const int4 q = R[r];
        const float g = __int_as_float(q.x);
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float2 a = sp[(q.y * K + k) * kRepBlock + lane];
            yx[k] = fmaf(g, a.x, yx[k]);
            yy[k] = fmaf(-g, a.y, yy[k]);
        }
        if (q.w) {
            const int p = q.z >> 16, o1 = q.z & 0xFFFF;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float2 ap = sp[(p * K + k) * kRepBlock + lane];
                const float2 ao = sp[(o1 * K + k) * kRepBlock + lane];
                const float px = fmaf(ap.x, ao.x, ap.y * ao.y);
                const float py = fmaf(ap.y, ao.x, -ap.x * ao.y);
                hx[k] = fmaf(px, yx[k], fmaf(-py, yy[k], hx[k]));
                hy[k] = fmaf(px, yy[k], fmaf(py, yx[k], hy[k]));
                yx[k] = 0.f;
                yy[k] = 0.f;
            }
        }
    }
}

// ---------------------------------------------------------------- clusters
// Partial fields of the CTAs of a thread-block cluster meet in every CTA's
// exchange buffer (distributed shared memory).
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    return ra;
}
// 8 bytes into a CTA of the cluster, counted on that CTA's mbarrier (cluster
// launches only)
__device__ __forceinline__ void st_async_f2(uint32_t addr, float2 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async_f64(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v), "r"(bar)
                 : "memory");
}

// store v into the same shared-memory location of CTA `rank` of the cluster
__device__ __forceinline__ void st_cluster_f2(const void* local, uint32_t rank, float2 v) {
    const uint32_t la = (uint32_t)__cvta_generic_to_shared(local);
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(la), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ra), "f"(v.x), "f"(v.y) : "memory");
}

__device__ __forceinline__ void st_cluster_u32(const void* local, uint32_t rank, uint32_t v) {
    const uint32_t la = (uint32_t)__cvta_generic_to_shared(local);
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(la), "r"(rank));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
}

}  // namespace pspin
