// lists.cu -- site lists, FP64 quartet table and neighbour masks of one dense
// sample, built on the device from its couplings and channel mask: the same
// entries, chunks and quartets, in the same order, as layout.cpp's dense_quartets,
// build_site_lists(kRecords, tile) or build_site_tiles_fc, and build_q64 make on the
// host (where the formats are described).
//
// A site's terms need no sorting here: (site, p, o1) enumerates its groups in
// list order, a thread each, and the inner sites o2 their terms; a term's coupling
// is a lookup.  Scans give every group and part its place, the parts' shortest
// paths over tile cuts run a thread each, and a warp writes a part's tiles.
// What bounds it: launches and two round trips for the sizes up to N = 64, then the
// parts' paths.  A whole set-up with the lists made on the host (one thread a sample;
// sorts and shortest paths) and here, gamma = 0.1: N = 16 4.0 and 4.0 ms, N = 32 8.4
// and 3.8, N = 48 28 and 7.5, N = 64 87 and 9.7, N = 96 480 and 13, 16 samples of
// N = 64 (16 host threads) 315 and 105 (the rest is the generator calls); fully
// connected N = 24 5.5 and 3.5, N = 48 27 and 7, N = 64 87 and 8, N = 96 490 and 9:
// no size is left to the host's builder for its speed.
#include <algorithm>
#include <cstdint>

#include "lists.h"

namespace pspin {

namespace {

constexpr int kTileRows = 63;                   // as layout.cpp's
constexpr int kScan = 1024;

__host__ __device__ __forceinline__ int64_t b2(int64_t n) { return n * (n - 1) / 2; }
__host__ __device__ __forceinline__ int64_t b3(int64_t n) { return n * (n - 1) * (n - 2) / 6; }
__host__ __device__ __forceinline__ int64_t b4(int64_t n) { return n * (n - 1) * (n - 2) * (n - 3) / 24; }

struct In {
    const double* g4;        // by quartet index
    const uint8_t* mask;
    const double* g2;        // [N][N], or null: no two-body terms
    int N;
};

// The coupling of site m's term (p, o1, o2), o1 < o2: false where it has none.
// p == N, o1 == N: the two-body term with o2.
__device__ __forceinline__ bool term_of(const In& in, int m, int p, int o1, int o2, float& g) {
    const int N = in.N;
    if (p == N) {
        if (o2 == m) return false;
        const double v = in.g2[(size_t)m * N + o2];
        g = (float)v;
        return v != 0.0;
    }
    if (o1 == m || o1 == p || o2 == m || o2 == p) return false;
    const int a = min(m, p), b = max(m, p);     // {a, b} one class, {o1, o2} the other
    int i, j, k, l, ch;
    if (a < o1) {
        i = a;
        if (b < o1) { j = b; k = o1; l = o2; ch = 0; }
        else if (b < o2) { j = o1; k = b; l = o2; ch = 2; }
        else { j = o1; k = o2; l = b; ch = 1; }
    } else {
        i = o1;
        if (o2 < a) { j = o2; k = a; l = b; ch = 0; }
        else if (o2 < b) { j = a; k = o2; l = b; ch = 2; }
        else { j = a; k = b; l = o2; ch = 1; }
    }
    const int64_t q = b4(l) + b3(k) + b2(j) + i;
    if (!((in.mask[q] >> ch) & 1)) return false;
    const double v = in.g4[q];
    g = (float)v;
    return v != 0.0;
}

// The keys of a site: p in [0, N), o1 in [0, N), then the virtual site's one.
__device__ __forceinline__ bool key_of(const In& in, int x, int& p, int& o1) {
    const int N = in.N;
    p = x / N;
    o1 = x % N;
    if (x == N * N) {
        o1 = N;
        return in.g2 != nullptr;
    }
    return true;
}

__global__ void count_terms_kernel(const In in, uint16_t* __restrict__ cnt) {
    const int m = blockIdx.y, keys = in.N * in.N + 1, x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= keys) return;
    int p, o1, c = 0;
    float g;
    if (key_of(in, x, p, o1) && p != m && o1 != m && o1 != p + (p == in.N))
        for (int o2 = p == in.N ? 0 : o1 + 1; o2 < in.N; o2++) c += term_of(in, m, p, o1, o2, g);
    cnt[(size_t)m * keys + x] = (uint16_t)c;
}

// Exclusive prefix of two counts over kScan threads; returns the totals too.
__device__ __forceinline__ int2 block_scan(int2 v, int2& total) {
    __shared__ int2 part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int2 s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, s.x, o), b = __shfl_up_sync(0xffffffffu, s.y, o);
        if (lane >= o) { s.x += a; s.y += b; }
    }
    __syncthreads();
    if (lane == 31) part[warp] = s;
    __syncthreads();
    int2 before = make_int2(0, 0);
    total = make_int2(0, 0);
    for (int w = 0; w < kScan / 32; w++) {
        if (w == warp) before = total;
        total.x += part[w].x;
        total.y += part[w].y;
    }
    return make_int2(before.x + s.x - v.x, before.y + s.y - v.y);
}

// Groups and terms before every key of site blockIdx.x, and the site's totals.
__global__ void __launch_bounds__(kScan) scan_keys_kernel(const uint16_t* __restrict__ cnt, int keys, int2* __restrict__ off,
                                                          int2* __restrict__ totals) {
    const size_t row = (size_t)blockIdx.x * keys;
    int2 run = make_int2(0, 0), total;
    for (int x0 = 0; x0 < keys; x0 += kScan) {
        const int x = x0 + threadIdx.x, c = x < keys ? cnt[row + x] : 0;
        const int2 b = block_scan(make_int2((c + kGroupMax - 1) / kGroupMax, c), total);
        if (x < keys) off[row + x] = make_int2(run.x + b.x, run.y + b.y);
        run.x += total.x;
        run.y += total.y;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// int4 {p | o << 16, lo | hi << 16, end (two entries a term, cumulative), 0} per
// group; the neighbours of every site.
__global__ void groups_kernel(const In in, const uint16_t* __restrict__ cnt, const int2* __restrict__ off,
                              const int* __restrict__ gbase, int4* __restrict__ groups, uint32_t* __restrict__ nb) {
    const int m = blockIdx.y, keys = in.N * in.N + 1, x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= keys) return;
    uint32_t* row = nb + (size_t)m * ((in.N + 31) / 32);
    auto set = [&](int b) {
        if (b < in.N) atomicOr(row + b / 32, 1u << (b % 32));
    };
    if (x == keys - 1 && in.g2 != nullptr)      // two-body terms couple every pair
        for (int b = 0; b < in.N; b++)
            if (b != m) set(b);
    if (cnt[(size_t)m * keys + x] == 0) return;
    const int2 at = off[(size_t)m * keys + x];
    int4* out = groups + gbase[m] + at.x;
    int p, o1, n = 0, lo = 0, last = 0, end = 2 * at.y;
    float g;
    key_of(in, x, p, o1);
    set(p);
    set(o1);
    for (int o2 = p == in.N ? 0 : o1 + 1; o2 < in.N; o2++) {
        if (!term_of(in, m, p, o1, o2, g)) continue;
        if (p < in.N) set(o2);
        if (n == 0) lo = o2;
        last = o2;
        end += 2;
        if (++n == kGroupMax) {
            *out++ = make_int4(p | (o1 << 16), lo | ((last + 1) << 16), end, 0);
            n = 0;
        }
    }
    if (n) *out = make_int4(p | (o1 << 16), lo | ((last + 1) << 16), end, 0);
}

// Groups of part `part` of a site with n groups: layout.cpp's part_bounds.
__device__ __forceinline__ int part_begin(const int4* __restrict__ g, int n, int part) {
    if (part == 0) return 0;
    if (part == kSplit) return n;
    const int64_t total = n ? g[n - 1].z : 0, target = total * part / kSplit;
    if (target <= 0) return 0;
    int a = 0, b = n;                           // the first t with end[t - 1] >= target, or n
    while (a < b) {
        const int t = (a + b) / 2;
        if ((t == 0 ? 0 : g[t - 1].z) >= target) b = t;
        else a = t + 1;
    }
    return a;
}

__device__ __forceinline__ int64_t tile_cost_dev(int cols, int rows) {
    return cols <= 4 ? 25 + 20 * rows + 18 * cols : 28 + 36 * rows + 18 * cols;
}

// Per part: the cheapest cut in tiles (layout.cpp's tile_part), each tile's columns
// at its first group; its chunks and entries.  sums: cost, entries, operations,
// parts that no tiles hold.
__global__ void cut_kernel(const int4* __restrict__ groups, const int* __restrict__ gbase, const int2* __restrict__ totals,
                           int N, int64_t* __restrict__ best_all, uint8_t* __restrict__ cols_all,
                           uint8_t* __restrict__ width, int2* __restrict__ sizes, unsigned long long* __restrict__ sums) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= N * kSplit) return;
    const int m = id / kSplit, part = id % kSplit, ng = totals[m].x;
    const int4* g = groups + gbase[m];
    const int b = part_begin(g, ng, part), e = max(b, part_begin(g, ng, part + 1)), n = e - b;
    int2 size = make_int2(0, 0);
    if (n > 0) {
        int64_t* best = best_all + gbase[m] + b + id;       // n + 1 of them
        uint8_t* cols = cols_all + gbase[m] + b + id;
        uint8_t* wide = width + gbase[m] + b;
        best[0] = 0;
        for (int t = 1; t <= n; t++) {
            const int p = g[b + t - 1].x & 0xFFFF;
            int64_t least = INT64_MAX;
            int lo = INT32_MAX, hi = -1, least_c = 0;
            for (int c = 1; c <= 8 && c <= t; c++) {
                const int4 q = g[b + t - c];
                if ((q.x & 0xFFFF) != p) break;
                lo = min(lo, q.y & 0xFFFF);
                hi = max(hi, q.y >> 16);
                if (hi - lo > kTileRows) break;
                const int64_t cost = best[t - c] + tile_cost_dev(c, hi - lo);
                if (cost < least) {
                    least = cost;
                    least_c = c;
                }
            }
            if (least_c == 0) {                             // one group wider than a tile
                atomicAdd(sums + 3, 1ull);
                sizes[id] = size;
                return;
            }
            best[t] = least;
            cols[t] = (uint8_t)least_c;
        }
        for (int t = n; t > 0; t -= cols[t]) wide[t - cols[t]] = cols[t];
        int len = 0;
        unsigned long long ops = 0;
        for (int t = 0; t < n;) {
            const int c = wide[t];
            int lo = INT32_MAX, hi = -1;
            for (int q = 0; q < c; q++) {
                lo = min(lo, g[b + t + q].y & 0xFFFF);
                hi = max(hi, g[b + t + q].y >> 16);
            }
            const int w = c > 4 ? 8 : 4, words = w / 2 * (1 + hi - lo);
            if (len == 0 || len + words > kStage) {
                size.x++;
                len = 0;
            }
            len += words;
            size.y += words;
            ops += 14 * c + 4 * w * (hi - lo);
            t += c;
        }
        atomicAdd(sums, (unsigned long long)best[n]);
        atomicAdd(sums + 1, (unsigned long long)size.y);
        atomicAdd(sums + 2, ops);
    }
    sizes[id] = size;
}

// Exclusive scan of the parts' (chunks, entries), in place, and the totals.
__global__ void __launch_bounds__(kScan) scan_parts_kernel(int2* __restrict__ sizes, int n, unsigned long long* __restrict__ sums) {
    int2 run = make_int2(0, 0), total;
    for (int x0 = 0; x0 < n; x0 += kScan) {
        const int x = x0 + threadIdx.x;
        const int2 v = x < n ? sizes[x] : make_int2(0, 0);
        const int2 b = block_scan(v, total);
        if (x < n) sizes[x] = make_int2(run.x + b.x, run.y + b.y);
        run.x += total.x;
        run.y += total.y;
    }
    if (threadIdx.x == 0) {
        sums[4] = (unsigned long long)run.x;
        sums[5] = (unsigned long long)run.y;
    }
}

// A warp per part writes its tiles, chunk starts and site-chunk entry.
__global__ void emit_kernel(const In in, const int4* __restrict__ groups, const int* __restrict__ gbase,
                            const int2* __restrict__ totals, const uint8_t* __restrict__ width,
                            const int2* __restrict__ sizes, int chunks, int64_t entry0, int chunk0,
                            int2* __restrict__ entries, int64_t* __restrict__ chunk_start, int* __restrict__ site_chunks) {
    const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, N = in.N;
    if (id >= N * kSplit) return;
    const int m = id / kSplit, part = id % kSplit, ng = totals[m].x;
    const int4* g = groups + gbase[m];
    const int b = part_begin(g, ng, part), e = max(b, part_begin(g, ng, part + 1));
    int chunk = sizes[id].x;
    int64_t at = sizes[id].y;
    if (lane == 0) {
        site_chunks[m * (kSplit + 1) + part] = chunk0 + chunk;
        if (part == kSplit - 1) site_chunks[m * (kSplit + 1) + kSplit] = chunk0 + (id + 1 < N * kSplit ? sizes[id + 1].x : chunks);
    }
    int len = 0;
    for (int t = b; t < e;) {
        const int c = width[gbase[m] + t], w = c > 4 ? 8 : 4;
        int lo = INT32_MAX, hi = -1;
        for (int q = 0; q < c; q++) {
            lo = min(lo, g[t + q].y & 0xFFFF);
            hi = max(hi, g[t + q].y >> 16);
        }
        const int rows = hi - lo, words = w / 2 * (1 + rows), p = g[t].x & 0xFFFF;
        if (len == 0 || len + words > kStage) {
            if (lane == 0) chunk_start[chunk] = entry0 + at;
            chunk++;
            len = 0;
        }
        len += words;
        int2* out = entries + at;
        if (lane == 0) {
            auto v = [&](int q) { return q < c ? g[t + q].x >> 16 : N; };
            out[0] = make_int2(p | ((2 | (w == 8)) << 16), lo | (rows << 16) | (c << 24));
            out[1] = make_int2(v(0) | (v(1) << 16), v(2) | (v(3) << 16));
            if (w == 8) {
                out[2] = make_int2(v(4) | (v(5) << 16), v(6) | (v(7) << 16));
                out[3] = make_int2(0, 0);
            }
        }
        float* couplings = reinterpret_cast<float*>(out + w / 2);
        for (int u = lane; u < rows * w; u += 32) {
            const int q = u % w, o2 = lo + u / w;
            float v = 0.f;
            if (q < c) {
                const int4 gq = g[t + q];
                float f;
                if (o2 >= (gq.y & 0xFFFF) && o2 < (gq.y >> 16) && term_of(in, m, p, gq.x >> 16, o2, f)) v = f;
            }
            couplings[u] = v;
        }
        at += words;
        t += c;
    }
}

// ---- fully connected samples: layout.cpp's build_site_tiles_fc
// Key x of site m: 0 the two-body terms; 1 .. N-1-m the outer sites above m (m among
// a quartet's two smallest); the rest those below m.  A key holds, four partners at a
// time, its inner range in steps of kGroupMax ("fours").
struct FcKey {
    int outer, lo, hi, partners;
    bool above;
};
__device__ __forceinline__ FcKey fc_key(const In& in, int m, int x) {
    const int N = in.N;
    FcKey k;
    k.above = x <= N - 1 - m;
    if (x == 0) return FcKey{N, 0, in.g2 ? N : 0, 1, false};
    k.outer = k.above ? m + x : x - (N - m);
    k.lo = k.above ? k.outer + 1 : 0;
    k.hi = k.above ? N : k.outer;
    k.partners = k.lo >= k.hi ? 0 : k.above ? k.outer - 1 : N - 2 - k.outer;
    return k;
}

// int4 {outer | first partner << 16, lo | hi << 16, end (entries, cumulative), partners
// | above << 16} per four; scanned with one block per site.
__global__ void __launch_bounds__(kScan) fc_fours_kernel(const In in, const int* __restrict__ gbase, int4* __restrict__ fours,
                                                         int2* __restrict__ totals) {
    const int m = blockIdx.x, N = in.N;
    int2 run = make_int2(0, 0), total;
    for (int x0 = 0; x0 < N; x0 += kScan) {
        const int x = x0 + threadIdx.x;
        FcKey k{0, 0, 0, 0, false};
        int2 v = make_int2(0, 0);
        if (x < N) {
            k = fc_key(in, m, x);
            const int blocks = (k.partners + 3) / 4, len = max(k.hi - k.lo, 0), steps = (len + kGroupMax - 1) / kGroupMax;
            v = make_int2(blocks * steps, 2 * blocks * (len + steps));
        }
        const int2 b = block_scan(v, total);
        if (fours != nullptr && v.x > 0) {
            int4* out = fours + gbase[m] + run.x + b.x;
            int end = run.y + b.y;
            for (int p = 0; p < k.partners; p += 4)
                for (int lo = k.lo; lo < k.hi; lo += kGroupMax) {
                    const int hi = min(k.hi, lo + kGroupMax);
                    end += 2 * (1 + hi - lo);
                    *out++ = make_int4(k.outer | (p << 16), lo | (hi << 16), end, min(4, k.partners - p) | (k.above << 16));
                }
        }
        run.x += total.x;
        run.y += total.y;
    }
    if (threadIdx.x == 0) totals[m] = run;
}

// the tile at four t of [.., e): one four, or two over the same inner range
__device__ __forceinline__ bool fc_two(const int4* __restrict__ f, int t, int e, int N) {
    return t + 1 < e && (f[t].w & 0xFFFF) == 4 && (f[t].x & 0xFFFF) < N && (f[t + 1].x & 0xFFFF) == (f[t].x & 0xFFFF) &&
           f[t + 1].y == f[t].y;
}

__global__ void fc_cut_kernel(const int4* __restrict__ fours, const int* __restrict__ gbase, const int2* __restrict__ totals,
                              int N, int2* __restrict__ sizes, unsigned long long* __restrict__ sums) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= N * kSplit) return;
    const int m = id / kSplit, part = id % kSplit, n = totals[m].x;
    const int4* f = fours + gbase[m];
    const int b = part_begin(f, n, part), e = max(b, part_begin(f, n, part + 1));
    int2 size = make_int2(0, 0);
    int len = 0;
    unsigned long long ops = 0;
    for (int t = b; t < e;) {
        const bool two = fc_two(f, t, e, N);
        const int w = two ? 8 : 4, rows = (f[t].y >> 16) - (f[t].y & 0xFFFF), words = w / 2 * (1 + rows);
        const int c = two ? 4 + (f[t + 1].w & 0xFFFF) : f[t].w & 0xFFFF;
        if (len == 0 || len + words > kStage) {
            size.x++;
            len = 0;
        }
        len += words;
        size.y += words;
        ops += 14 * c + 4 * w * rows;
        t += two ? 2 : 1;
    }
    if (ops) atomicAdd(sums + 2, ops);
    sizes[id] = size;
}

__global__ void fc_emit_kernel(const In in, const int4* __restrict__ fours, const int* __restrict__ gbase,
                               const int2* __restrict__ totals, const int2* __restrict__ sizes, int chunks, int64_t entry0,
                               int chunk0, int2* __restrict__ entries, int64_t* __restrict__ chunk_start,
                               int* __restrict__ site_chunks) {
    const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, N = in.N;
    if (id >= N * kSplit) return;
    const int m = id / kSplit, part = id % kSplit, n = totals[m].x;
    const int4* f = fours + gbase[m];
    const int b = part_begin(f, n, part), e = max(b, part_begin(f, n, part + 1));
    int chunk = sizes[id].x, len = 0;
    int64_t at = sizes[id].y;
    if (lane == 0) {
        site_chunks[m * (kSplit + 1) + part] = chunk0 + chunk;
        if (part == kSplit - 1) site_chunks[m * (kSplit + 1) + kSplit] = chunk0 + (id + 1 < N * kSplit ? sizes[id + 1].x : chunks);
    }
    for (int t = b; t < e;) {
        const bool two = fc_two(f, t, e, N);
        const int4 f0 = f[t], f1 = f[two ? t + 1 : t];
        const int outer = f0.x & 0xFFFF, lo = f0.y & 0xFFFF, rows = (f0.y >> 16) - lo, w = two ? 8 : 4;
        const int c = two ? 4 + (f1.w & 0xFFFF) : f0.w & 0xFFFF, words = w / 2 * (1 + rows);
        const bool above = (f0.w >> 16) != 0;
        auto v = [&](int q) {                       // column q's partner: the sites but m, from 0 or after outer
            if (q >= c || outer == N) return N;
            const int p = (q < 4 ? f0.x >> 16 : f1.x >> 16) + (q & 3) + (above ? 0 : outer + 1);
            return p < m ? p : p + 1;
        };
        if (len == 0 || len + words > kStage) {
            if (lane == 0) chunk_start[chunk] = entry0 + at;
            chunk++;
            len = 0;
        }
        len += words;
        int2* out = entries + at;
        if (lane == 0) {
            out[0] = make_int2(outer | ((two ? 1 : 0) << 16), lo | (rows << 16) | (c << 24));
            out[1] = make_int2(v(0) | (v(1) << 16), v(2) | (v(3) << 16));
            if (two) {
                out[2] = make_int2(v(4) | (v(5) << 16), v(6) | (v(7) << 16));
                out[3] = make_int2(0, 0);
            }
        }
        float* couplings = reinterpret_cast<float*>(out + w / 2);
        for (int u = lane; u < rows * w; u += 32) {
            const int q = u % w, r = lo + u / w;
            float g = 0.f;
            if (q < c) {
                if (outer == N) {
                    if (r != m) g = (float)in.g2[(size_t)m * N + r];
                } else {
                    // sorted {m, p, outer, r}: above, m and p below outer below r; else r below outer below m and p
                    const int p = v(q), a = min(m, p), z = max(m, p);
                    const int64_t quartet = above ? b4(r) + b3(outer) + b2(z) + a : b4(z) + b3(a) + b2(outer) + r;
                    g = (float)in.g4[quartet];
                }
            }
            couplings[u] = g;
        }
        at += words;
        t += two ? 2 : 1;
    }
}

__global__ void fc_neighbours_kernel(int N, bool all, uint32_t* __restrict__ nb) {
    const int wpr = (N + 31) / 32, id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= N * wpr) return;
    const int m = id / wpr, first = 32 * (id % wpr), n = min(32, N - first);
    uint32_t w = !all ? 0u : n == 32 ? 0xffffffffu : (1u << n) - 1u;
    if (m / 32 == id % wpr) w &= ~(1u << (m % 32));
    nb[id] = w;
}

// ---- FP64 quartet table: block (l, k) holds quartets b4(l) + b3(k) + [0, b2(k))
__global__ void count_quartets_kernel(const In in, int* __restrict__ counts) {
    const int l = blockIdx.x, k = blockIdx.y;
    __shared__ int sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    int c = 0;
    if (l >= 3 && k >= 2 && k < l) {
        const int64_t base = b4(l) + b3(k);
        for (int64_t x = threadIdx.x; x < b2(k); x += blockDim.x)
            if (in.g4[base + x] != 0.0) c += __popc(in.mask[base + x] & 7);
    }
    atomicAdd(&sum, c);
    __syncthreads();
    if (threadIdx.x == 0) counts[l * in.N + k] = sum;
}

__global__ void __launch_bounds__(kScan) scan_quartets_kernel(const int* __restrict__ counts, int n, int64_t* __restrict__ off,
                                                              unsigned long long* __restrict__ sums) {
    int64_t run = 0;
    int2 total;
    for (int x0 = 0; x0 < n; x0 += kScan) {
        const int x = x0 + threadIdx.x;
        const int2 b = block_scan(make_int2(x < n ? counts[x] : 0, 0), total);
        if (x < n) off[x] = run + b.x;
        run += total.x;
    }
    if (threadIdx.x == 0) sums[6] = (unsigned long long)run;
}

__global__ void __launch_bounds__(kScan) quartets_kernel(const In in, const int64_t* __restrict__ off, Q64* __restrict__ out) {
    const int l = blockIdx.x, k = blockIdx.y;
    if (l < 3 || k < 2 || k >= l) return;
    const int64_t base = b4(l) + b3(k), np = b2(k);
    int64_t at = off[l * in.N + k];
    int2 total;
    for (int64_t x0 = 0; x0 < np; x0 += kScan) {
        const int64_t x = x0 + threadIdx.x;
        int mask = 0;
        double g = 0.0;
        if (x < np) {
            g = in.g4[base + x];
            mask = g != 0.0 ? in.mask[base + x] & 7 : 0;
        }
        const int2 b = block_scan(make_int2(__popc(mask), 0), total);
        if (mask) {
            int j = (int)((1.0 + sqrt(1.0 + 8.0 * (double)x)) * 0.5);
            while (b2(j) > x) j--;
            while (b2(j + 1) <= x) j++;
            Q64* q = out + at + b.x;
            for (int ch = 0; ch < 3; ch++)
                if (mask & (1 << ch)) *q++ = Q64{(uint16_t)(x - b2(j)), (uint16_t)j, (uint16_t)k, (uint16_t)(l | (ch << 14)), g};
        }
        at += total.x;
    }
}

}  // namespace

DeviceLists::~DeviceLists() {
    cudaFree(slab);
    cudaFree(groups_slab);
}

// 16-byte-aligned pieces of one allocation
template <class T>
static T* piece(size_t& at, unsigned char* base, size_t n) {
    at = (at + 15) & ~(size_t)15;
    T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += n * sizeof(T);
    return p;
}

cudaError_t DeviceLists::plan(int N_, const double* g4, const uint8_t* mask, const double* g2_host, cudaStream_t st) {
    N = N_;
    d_g4 = g4;
    d_mask = mask;
    cudaError_t e = cudaSuccess;
    const int keys = N * N + 1, wpr = (N + 31) / 32;
    uint16_t* cnt = nullptr;
    int2* off = nullptr;
    int* qcnt = nullptr;
    for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
        size_t at = 0;
        unsigned char* base = static_cast<unsigned char*>(slab);
        cnt = piece<uint16_t>(at, base, (size_t)N * keys);
        off = piece<int2>(at, base, (size_t)N * keys);
        d_totals = piece<int2>(at, base, N);
        d_gbase = piece<int>(at, base, N);
        d_sizes = piece<int2>(at, base, (size_t)N * kSplit);
        d_sums = piece<unsigned long long>(at, base, 8);
        d_nb = piece<uint32_t>(at, base, (size_t)N * wpr);
        qcnt = piece<int>(at, base, (size_t)N * N);
        d_qoff = piece<int64_t>(at, base, (size_t)N * N);
        if (g2_host) d_g2 = piece<double>(at, base, (size_t)N * N);
        if (pass == 0) e = cudaMalloc(&slab, at);
        held = at;
    }
    if (e == cudaSuccess && g2_host)
        e = cudaMemcpyAsync(d_g2, g2_host, (size_t)N * N * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const In in{d_g4, d_mask, d_g2, N};
    const dim3 grid((keys + 255) / 256, N);
    count_terms_kernel<<<grid, 256, 0, st>>>(in, cnt);
    scan_keys_kernel<<<N, kScan, 0, st>>>(cnt, keys, off, d_totals);
    std::vector<int2> totals(N);
    e = cudaMemcpyAsync(totals.data(), d_totals, N * sizeof(int2), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    std::vector<int> gbase(N);
    int64_t n_groups = 0, terms = 0;
    for (int m = 0; m < N; m++) {
        gbase[m] = (int)n_groups;
        n_groups += totals[m].x;
        terms += totals[m].y;
    }
    if (n_groups + (int64_t)N * kSplit >= (1ll << 31) || 2 * terms >= (1ll << 31)) return cudaErrorInvalidValue;
    int64_t* best = nullptr;
    uint8_t* cols = nullptr;
    for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
        size_t at = 0;
        unsigned char* base = static_cast<unsigned char*>(groups_slab);
        d_groups = piece<int4>(at, base, (size_t)n_groups);
        best = piece<int64_t>(at, base, (size_t)(n_groups + N * kSplit));
        cols = piece<uint8_t>(at, base, (size_t)(n_groups + N * kSplit));
        d_width = piece<uint8_t>(at, base, (size_t)n_groups);
        if (pass == 0) {
            e = cudaMalloc(&groups_slab, std::max<size_t>(at, 16));
            held += at;
        }
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_gbase, gbase.data(), N * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_nb, 0, (size_t)N * wpr * sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_sums, 0, 8 * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    groups_kernel<<<grid, 256, 0, st>>>(in, cnt, off, d_gbase, d_groups, d_nb);
    cut_kernel<<<(N * kSplit + 31) / 32, 32, 0, st>>>(d_groups, d_gbase, d_totals, N, best, cols, d_width, d_sizes, d_sums);
    scan_parts_kernel<<<1, kScan, 0, st>>>(d_sizes, N * kSplit, d_sums);
    count_quartets_kernel<<<dim3(N, N), 128, 0, st>>>(in, qcnt);
    scan_quartets_kernel<<<1, kScan, 0, st>>>(qcnt, N * N, d_qoff, d_sums);
    unsigned long long sums[8];
    e = cudaMemcpyAsync(sums, d_sums, sizeof(sums), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // the rule of layout.cpp's build_site_lists
    const int64_t records = 21 * terms + 32 * n_groups, words = 2 * terms;
    tiles = sums[3] == 0 && (int64_t)sums[0] < records && (int64_t)sums[1] <= words;
    nominal = words;
    chunks = (int64_t)sums[4];
    entries = (int64_t)sums[5];
    flops = (double)sums[2];
    quartets = (int64_t)sums[6];
    return cudaSuccess;
}

cudaError_t DeviceLists::plan_fc(int N_, const double* g4, const uint8_t* mask, const double* g2_host, cudaStream_t st) {
    N = N_;
    fc = true;
    d_g4 = g4;
    d_mask = mask;
    cudaError_t e = cudaSuccess;
    // as fc_fours_kernel counts them
    std::vector<int> gbase(N);
    int64_t n_fours = 0;
    for (int m = 0; m < N; m++) {
        gbase[m] = (int)n_fours;
        auto add = [&](int partners, int len) {
            n_fours += (int64_t)((partners + 3) / 4) * ((len + kGroupMax - 1) / kGroupMax);
        };
        if (g2_host) add(1, N);
        for (int o = m + 1; o < N - 1; o++) add(o - 1, N - 1 - o);
        for (int o = 1; o < m; o++) add(N - 2 - o, o);
    }
    // the kernels count entries in 31 bits, at most 2 (1 + kGroupMax) a four
    if (n_fours * 2 * (1 + kGroupMax) >= (1ll << 31)) return cudaErrorInvalidValue;
    int* qcnt = nullptr;
    for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
        size_t at = 0;
        unsigned char* base = static_cast<unsigned char*>(slab);
        d_totals = piece<int2>(at, base, N);
        d_gbase = piece<int>(at, base, N);
        d_sizes = piece<int2>(at, base, (size_t)N * kSplit);
        d_sums = piece<unsigned long long>(at, base, 8);
        qcnt = piece<int>(at, base, (size_t)N * N);
        d_qoff = piece<int64_t>(at, base, (size_t)N * N);
        d_groups = piece<int4>(at, base, (size_t)n_fours);
        if (g2_host) d_g2 = piece<double>(at, base, (size_t)N * N);
        if (pass == 0) e = cudaMalloc(&slab, at);
        held = at;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_gbase, gbase.data(), N * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_sums, 0, 8 * sizeof(unsigned long long), st);
    if (e == cudaSuccess && g2_host)
        e = cudaMemcpyAsync(d_g2, g2_host, (size_t)N * N * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const In in{d_g4, d_mask, d_g2, N};
    fc_fours_kernel<<<N, kScan, 0, st>>>(in, d_gbase, d_groups, d_totals);
    fc_cut_kernel<<<(N * kSplit + 31) / 32, 32, 0, st>>>(d_groups, d_gbase, d_totals, N, d_sizes, d_sums);
    scan_parts_kernel<<<1, kScan, 0, st>>>(d_sizes, N * kSplit, d_sums);
    count_quartets_kernel<<<dim3(N, N), 128, 0, st>>>(in, qcnt);
    scan_quartets_kernel<<<1, kScan, 0, st>>>(qcnt, N * N, d_qoff, d_sums);
    unsigned long long sums[8];
    std::vector<int2> totals(N);
    e = cudaMemcpyAsync(sums, d_sums, sizeof(sums), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(totals.data(), d_totals, N * sizeof(int2), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    nominal = 0;
    for (const int2& t : totals) nominal += t.y;
    chunks = (int64_t)sums[4];
    entries = (int64_t)sums[5];
    flops = (double)sums[2];
    quartets = (int64_t)sums[6];
    tiles = quartets == b4(N);                  // a zero coupling: not fully connected
    return cudaSuccess;
}

cudaError_t DeviceLists::write(int64_t entry0, int64_t chunk0, int2* out, int64_t* chunk_start, int* site_chunks, Q64* q,
                               uint32_t* nb, cudaStream_t st) const {
    const In in{d_g4, d_mask, d_g2, N};
    const int wpr = (N + 31) / 32;
    quartets_kernel<<<dim3(N, N), kScan, 0, st>>>(in, d_qoff, q);
    if (fc) {
        fc_emit_kernel<<<(N * kSplit + 3) / 4, 128, 0, st>>>(in, d_groups, d_gbase, d_totals, d_sizes, (int)chunks, entry0,
                                                             (int)chunk0, out, chunk_start, site_chunks);
        fc_neighbours_kernel<<<(N * wpr + 127) / 128, 128, 0, st>>>(N, N >= 4 || d_g2 != nullptr, nb);
        return cudaGetLastError();
    }
    emit_kernel<<<(N * kSplit + 3) / 4, 128, 0, st>>>(in, d_groups, d_gbase, d_totals, d_width, d_sizes, (int)chunks, entry0,
                                                      (int)chunk0, out, chunk_start, site_chunks);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(nb, d_nb, (size_t)N * wpr * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
}

}  // namespace pspin
