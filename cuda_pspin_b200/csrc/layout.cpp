// layout.cpp -- host construction of the sweep's per-site lists and of the
// FP64 quartet table, from one sample's active (quartet, channel) list.
//
// Channel classes (disorder.h:9-16) for sorted i<j<k<l:
//   ch 0: unconjugated {i,j}, conjugated {k,l}
//   ch 1: unconjugated {i,l}, conjugated {j,k}
//   ch 2: unconjugated {i,k}, conjugated {j,l}
// Member m of a quartet has a partner p (the other site of m's class) and
// an opposite pair {o1<o2}.  Site m's list holds, for every quartet of m,
// the term (p, o1, o2, g), in groups of equal (p, o1); layout.h has the
// formats.
#include "layout.h"

#include <algorithm>
#include <climits>
#include <cstring>

namespace pspin {

static inline void class_of(const int q[4], int ch, int m_pos, int& partner, int& o1, int& o2) {
    // positions of the unconjugated pair for each channel
    static const int U[3][2] = {{0, 1}, {0, 3}, {0, 2}};
    static const int C[3][2] = {{2, 3}, {1, 2}, {1, 3}};
    const int* mine;
    const int* opp;
    if (m_pos == U[ch][0] || m_pos == U[ch][1]) { mine = U[ch]; opp = C[ch]; }
    else { mine = C[ch]; opp = U[ch]; }
    partner = q[mine[0] == m_pos ? mine[1] : mine[0]];
    const int a = q[opp[0]], b = q[opp[1]];
    o1 = a < b ? a : b;
    o2 = a < b ? b : a;
}

struct Rec {
    int32_t key;   // p<<16 | o1
    int32_t o2;
    float g;
};

using Span = std::pair<int64_t, int64_t>;   // [begin, end)

static inline int fbits(float f) {
    int b;
    std::memcpy(&b, &f, sizeof(int));
    return b;
}

// The parts of one list: kSplit/stride pieces of nearly equal size (items with
// ends `end[t]`, cumulative), piece q in part q*stride, the other parts empty.
// stride 1 for site lists; short lists use a larger stride so that a warp
// fetches one chunk rather than several tiny ones (a chain is 32/n consecutive
// parts for any n dividing 32).
static void part_bounds(const std::vector<int64_t>& end, int stride, size_t first[kSplit + 1]) {
    const size_t n = end.size();
    const int64_t total = n ? end.back() : 0;
    const int pieces = kSplit / stride;
    std::vector<size_t> bound(pieces + 1, n);
    bound[0] = 0;
    size_t g = 0;
    for (int q = 1; q < pieces; q++) {
        const int64_t target = (total * q) / pieces;
        while (g < n && (g == 0 ? 0 : end[g - 1]) < target) g++;
        bound[q] = g;
    }
    for (int part = 0; part < kSplit; part++)
        first[part] = (part % stride == 0) ? bound[part / stride] : bound[part / stride + 1];
    first[kSplit] = n;
}

// Appends items [b, e) (spans of `site`) to the list's chunks: whole items,
// <= kStage entries per chunk, an even number of entries.
static void pack_part(const std::vector<int2>& site, const std::vector<Span>& items, size_t b, size_t e, SiteLists& out) {
    while (b < e) {
        out.chunk_start.push_back((int64_t)out.entries.size());
        int64_t len = 0;
        while (b < e) {
            const int64_t n = items[b].second - items[b].first;
            if (len > 0 && len + n > kStage) break;
            out.entries.insert(out.entries.end(), site.begin() + items[b].first, site.begin() + items[b].second);
            len += n;
            b++;
        }
        if (len & 1) out.entries.push_back(make_int2(0, 0));
    }
}

// ---- dense tiles ------------------------------------------------------------
// A tile is up to 8 consecutive groups ("columns") that share one site, read
// over a common range of inner sites: rows of 4 or 8 couplings, one per column
// (zero where the column has no term: adding it changes nothing), so one
// gathered inner amplitude serves all columns.  Column q adds
// a_p conj(a_o) (sum of its row couplings with conj(a_inner)) to the field, in
// column order: the additions of the groups taken one after another.
// 16-byte words: {shared | kind << 16, lo | rows << 16 | columns << 24, v0 |
// v1 << 16, v2 | v3 << 16}, with 8 columns also {v4 | v5 << 16, v6 | v7 << 16, 0,
// 0}; then the rows.  kind bit 0: 8 columns wide; bit 1: the shared site is p
// and v the columns' o (else the shared site is o and v the columns' p).
// rows <= kTileRows, so that a tile fits a chunk.
struct Group {
    int p, o, lo, hi;       // inner range
    const Rec* rec;         // terms (sparse ranges), or null: coef
};
constexpr int kTileRows = 63;

// per-lane cost of a tile in issue slots, about that of two replicas per lane:
// rows (couplings, gather, two FMA per column), columns (the fold), header
static inline int tile_cost(int cols, int rows) {
    return cols <= 4 ? 25 + 20 * rows + 18 * cols : 28 + 36 * rows + 18 * cols;
}
static inline int record_cost(int terms) { return 21 * terms + 32; }

static void emit_tile_header(std::vector<int2>& site, int shared, int kind, int lo, int rows, int cols, const int* v,
                             int N) {
    auto pair = [&](int q) { return (q < cols ? v[q] : N) | ((q + 1 < cols ? v[q + 1] : N) << 16); };
    site.push_back(make_int2(shared | (kind << 16), lo | (rows << 16) | (cols << 24)));
    site.push_back(make_int2(pair(0), pair(2)));
    if (kind & 1) {
        site.push_back(make_int2(pair(4), pair(6)));
        site.push_back(make_int2(0, 0));
    }
}

// Groups [b, e) of one part as tiles of fewest cost (a shortest path over the
// cut positions; a tile's columns share p); returns the cost and, with `site`,
// appends the tiles.
static int64_t tile_part(const std::vector<Group>& g, size_t b, size_t e, int N, std::vector<int2>* site,
                         std::vector<Span>* items) {
    const size_t n = e - b;
    std::vector<int64_t> best(n + 1, 0);
    std::vector<int> cols(n + 1, 0);
    for (size_t t = 1; t <= n; t++) {
        best[t] = INT64_MAX;
        int lo = INT32_MAX, hi = -1;
        for (int c = 1; c <= 8 && (size_t)c <= t; c++) {
            const Group& q = g[b + t - c];
            if (q.p != g[b + t - 1].p) break;
            lo = std::min(lo, q.lo);
            hi = std::max(hi, q.hi);
            if (hi - lo > kTileRows) break;
            const int64_t cost = best[t - c] + tile_cost(c, hi - lo);
            if (cost < best[t]) {
                best[t] = cost;
                cols[t] = c;
            }
        }
        if (cols[t] == 0) return INT64_MAX;      // one group wider than a tile
    }
    if (!site) return best[n];
    std::vector<std::pair<size_t, size_t>> cut;
    for (size_t t = n; t > 0; t -= cols[t]) cut.push_back({b + t - cols[t], b + t});
    for (size_t k = cut.size(); k-- > 0;) {
        const size_t t0 = cut[k].first;
        const int c = (int)(cut[k].second - t0), wide = c > 4 ? 8 : 4;
        int lo = INT32_MAX, hi = -1, v[8];
        for (int q = 0; q < c; q++) {
            lo = std::min(lo, g[t0 + q].lo);
            hi = std::max(hi, g[t0 + q].hi);
            v[q] = g[t0 + q].o;
        }
        const int64_t at = (int64_t)site->size();
        emit_tile_header(*site, g[t0].p, 2 | (wide == 8), lo, hi - lo, c, v, N);
        const size_t rows = site->size();
        site->resize(rows + (size_t)(hi - lo) * wide / 2, make_int2(0, 0));
        int* w = reinterpret_cast<int*>(site->data() + rows);
        for (int q = 0; q < c; q++) {
            const Rec* r = g[t0 + q].rec;
            for (int o2 = g[t0 + q].lo;; r++) {
                o2 = r->o2;
                w[(o2 - lo) * wide + q] = fbits(r->g);
                if (o2 + 1 == g[t0 + q].hi) break;
            }
        }
        items->push_back({at, (int64_t)site->size()});
    }
    return best[n];
}

// Sorts one list's terms by (p, o1, o2) and cuts them in groups; `end` gets
// each group's cumulative size in int2 entries of the format.
static void make_groups(std::vector<Rec>& v, GroupSize size, std::vector<Group>& g, std::vector<int64_t>& end) {
    std::sort(v.begin(), v.end(), [](const Rec& a, const Rec& b) {
        return a.key != b.key ? a.key < b.key : a.o2 < b.o2;
    });
    g.clear();
    end.clear();
    int64_t total = 0;
    for (size_t t = 0; t < v.size();) {
        size_t e = t;
        while (e < v.size() && v[e].key == v[t].key && (int)(e - t) < kGroupMax) e++;
        g.push_back(Group{v[t].key >> 16, v[t].key & 0xFFFF, v[t].o2, v[e - 1].o2 + 1, v.data() + t});
        const int64_t n = (int64_t)(e - t);
        total += size == kRecords ? 2 * n : n + 1;
        end.push_back(total);
        t = e;
    }
}

// One group in its own format.
static void emit_group(const Group& g, GroupSize size, std::vector<int2>& site, std::vector<Span>& items, int64_t n) {
    const int64_t at = (int64_t)site.size();
    const int key = (g.p << 16) | g.o;
    if (size == kGroups) site.push_back(make_int2((int)n, key));
    for (int64_t u = 0; u < n; u++) {
        site.push_back(make_int2(fbits(g.rec[u].g), g.rec[u].o2));
        if (size == kRecords) site.push_back(make_int2(key, u + 1 == n ? 1 : 0));
    }
    items.push_back({at, (int64_t)site.size()});
}

// List `id` from its groups, in the format of `size` or as tiles.
static void pack_list(const std::vector<Group>& g, const std::vector<int64_t>& end, GroupSize size, bool tile, int N,
                      int id, int stride, SiteLists& out, std::vector<int2>& site, std::vector<Span>& items) {
    size_t first[kSplit + 1];
    part_bounds(end, stride, first);
    out.nominal += end.empty() ? 0 : end.back();
    int* sc = &out.site_chunks[(size_t)id * (kSplit + 1)];
    for (int part = 0; part < kSplit; part++) {
        sc[part] = (int)out.chunk_start.size();
        const size_t b = first[part], e = std::max(first[part], first[part + 1]);
        if (b == e) continue;
        site.clear();
        items.clear();
        if (tile) tile_part(g, b, e, N, &site, &items);
        else
            for (size_t t = b; t < e; t++) {
                const int64_t w = end[t] - (t ? end[t - 1] : 0);
                emit_group(g[t], size, site, items, size == kRecords ? w / 2 : w - 1);
            }
        pack_part(site, items, 0, items.size(), out);
    }
    sc[kSplit] = (int)out.chunk_start.size();
}

void build_pair_lists(int N, const double* g2re, int h2_active, const std::vector<QuartetRec>& qs,
                      SiteLists& out, bool tile) {
    const int npairs = N * (N - 1) / 2;
    auto list_id = [](int m, int x) {   // m's terms that contain x
        return m < x ? 2 * (x * (x - 1) / 2 + m) : 2 * (m * (m - 1) / 2 + x) + 1;
    };
    std::vector<std::vector<Rec>> per((size_t)2 * npairs);
    for (const QuartetRec& r : qs) {
        const int q[4] = {r.i, r.j, r.k, r.l};
        const float g = (float)r.g;
        for (int pos = 0; pos < 4; pos++) {
            int p, o1, o2;
            class_of(q, r.ch, pos, p, o1, o2);
            const Rec rec{(p << 16) | o1, o2, g};
            per[list_id(q[pos], p)].push_back(rec);
            per[list_id(q[pos], o1)].push_back(rec);
            per[list_id(q[pos], o2)].push_back(rec);
        }
    }
    if (h2_active)
        for (int m = 0; m < N; m++)
            for (int j = 0; j < N; j++) {
                if (j == m) continue;
                const double g = g2re[(size_t)m * N + j];
                if (g != 0.0) per[list_id(m, j)].push_back(Rec{(N << 16) | N, j, (float)g});
            }
    out.entries.clear();
    out.chunk_start.clear();
    out.site_chunks.assign((size_t)2 * npairs * (kSplit + 1), 0);
    std::vector<Group> g;
    std::vector<int64_t> end;
    std::vector<Span> items;
    std::vector<int2> site;
    constexpr int kStride = 4;                  // 8 pieces: one chunk per warp at 8 warps
    if (tile) {
        int64_t tiles = 0, groups = 0, words = 0, tile_words = 0;
        for (int id = 0; id < 2 * npairs && tile; id++) {
            make_groups(per[id], kGroups, g, end);
            size_t first[kSplit + 1];
            part_bounds(end, kStride, first);
            for (int part = 0; part < kSplit && tile; part++) {
                const size_t b = first[part], e = std::max(first[part], first[part + 1]);
                if (b == e) continue;
                site.clear();
                items.clear();
                const int64_t c = tile_part(g, b, e, N, &site, &items);
                if (c == INT64_MAX) tile = false;
                tiles += c;
                tile_words += (int64_t)site.size();
            }
            for (size_t t = 0; t < g.size(); t++)
                groups += record_cost((int)(end[t] - (t ? end[t - 1] : 0) - 1));
            words += end.empty() ? 0 : end.back();
        }
        tile = tile && tiles < groups && tile_words <= words + words / 4;
    }
    out.tiles = tile;
    for (int id = 0; id < 2 * npairs; id++) {
        make_groups(per[id], kGroups, g, end);
        pack_list(g, end, kGroups, tile, N, id, kStride, out, site, items);
        std::vector<Rec>().swap(per[id]);
    }
}

void build_site_lists(int N, const double* g2re, int h2_active, const std::vector<QuartetRec>& qs, SiteLists& out,
                      GroupSize size, bool tile) {
    std::vector<std::vector<Rec>> per(N);
    std::vector<int64_t> cnt(N, 0);
    for (const QuartetRec& r : qs) { cnt[r.i]++; cnt[r.j]++; cnt[r.k]++; cnt[r.l]++; }
    for (int m = 0; m < N; m++) per[m].reserve(cnt[m] + (h2_active ? N : 0));
    for (const QuartetRec& r : qs) {
        const int q[4] = {r.i, r.j, r.k, r.l};
        const float g = (float)r.g;
        for (int pos = 0; pos < 4; pos++) {
            int p, o1, o2;
            class_of(q, r.ch, pos, p, o1, o2);
            per[q[pos]].push_back(Rec{(p << 16) | o1, o2, g});
        }
    }
    if (h2_active) {
        // 2-body field h2_m = sum_{j != m} g_mj conj(a_j): partner and first
        // opposite site are the virtual unit site N
        for (int m = 0; m < N; m++)
            for (int j = 0; j < N; j++) {
                if (j == m) continue;
                const double g = g2re[(size_t)m * N + j];
                if (g != 0.0) per[m].push_back(Rec{(N << 16) | N, j, (float)g});
            }
    }
    std::vector<std::vector<Group>> g(N);
    std::vector<std::vector<int64_t>> end(N);
    for (int m = 0; m < N; m++) make_groups(per[m], size, g[m], end[m]);
    if (tile) {
        // tiles only where they are cheaper to read than the records, and no
        // larger (a list that fits in shared memory as records still fits)
        int64_t tiles = 0, records = 0, words = 0, tile_words = 0;
        for (int m = 0; m < N && tile; m++) {
            size_t first[kSplit + 1];
            part_bounds(end[m], 1, first);
            for (int part = 0; part < kSplit && tile; part++) {
                const size_t b = first[part], e = std::max(first[part], first[part + 1]);
                if (b == e) continue;
                std::vector<int2> site;
                std::vector<Span> items;
                const int64_t c = tile_part(g[m], b, e, N, &site, &items);
                if (c == INT64_MAX) tile = false;
                tiles += c;
                tile_words += (int64_t)site.size();
            }
            for (size_t t = 0; t < g[m].size(); t++) {
                const int64_t w = end[m][t] - (t ? end[m][t - 1] : 0), n = size == kRecords ? w / 2 : w - 1;
                records += record_cost((int)n);
                words += 2 * n;
            }
        }
        tile = tile && tiles < records && tile_words <= words;
    }
    out.entries.clear();
    out.chunk_start.clear();
    out.site_chunks.assign((size_t)N * (kSplit + 1), 0);
    out.nominal = 0;
    out.tiles = tile;
    std::vector<Span> items;
    std::vector<int2> site;
    for (int m = 0; m < N; m++) pack_list(g[m], end[m], size, tile, N, m, 1, out, site, items);
}

static inline int64_t encode_sorted(int a, int b, int c, int d) {
    int v[4] = {a, b, c, d};
    std::sort(v, v + 4);
    return (int64_t)v[3] * (v[3] - 1) * (v[3] - 2) * (v[3] - 3) / 24 + (int64_t)v[2] * (v[2] - 1) * (v[2] - 2) / 6 +
           (int64_t)v[1] * (v[1] - 1) / 2 + v[0];
}

// The terms of a fully connected site in list order: for every outer site and
// four partners at a time, inner ranges of at most kGroupMax; each such group of
// four is what the parts are balanced by (a 16-byte header and its rows), and
// two of them over the same inner range become one 8-column tile.
void build_site_tiles_fc(int N, const double* g2re, int h2_active, const double* g4re, SiteLists& out) {
    out.entries.clear();
    out.chunk_start.clear();
    out.site_chunks.assign((size_t)N * (kSplit + 1), 0);
    out.nominal = 0;
    out.tiles = true;
    struct Four {
        int outer, lo, hi, n, p[4];    // n real partners
    };
    std::vector<Four> fours;
    std::vector<int64_t> end;
    std::vector<int2> site;
    std::vector<Span> items;
    std::vector<int> partners;
    for (int m = 0; m < N; m++) {
        fours.clear();
        end.clear();
        auto add = [&](const Four& f) {
            fours.push_back(f);
            end.push_back((end.empty() ? 0 : end.back()) + 2 * (1 + f.hi - f.lo));
        };
        if (h2_active)
            for (int lo = 0; lo < N; lo += kGroupMax) add(Four{N, lo, std::min(N, lo + kGroupMax), 1, {N, N, N, N}});
        // m among the two smallest: outer o1 > m, partners p < o1, inner o2 in (o1, N)
        // m among the two largest: outer o2 < m, partners p > o2, inner o1 in [0, o2)
        for (int side = 0; side < 2; side++) {
            const int o_begin = side == 0 ? m + 1 : 0, o_end = side == 0 ? N : m;
            for (int outer = o_begin; outer < o_end; outer++) {
                const int ilo = side == 0 ? outer + 1 : 0, ihi = side == 0 ? N : outer;
                if (ilo >= ihi) continue;
                partners.clear();
                if (side == 0) { for (int p = 0; p < outer; p++) if (p != m) partners.push_back(p); }
                else { for (int p = outer + 1; p < N; p++) if (p != m) partners.push_back(p); }
                for (size_t pb = 0; pb < partners.size(); pb += 4)
                    for (int lo = ilo; lo < ihi; lo += kGroupMax) {
                        Four f{outer, lo, std::min(ihi, lo + kGroupMax), 0, {N, N, N, N}};
                        for (; f.n < 4 && pb + f.n < partners.size(); f.n++) f.p[f.n] = partners[pb + f.n];
                        add(f);
                    }
            }
        }
        auto coef = [&](const Four& f, int k, int t) -> float {
            if (k >= f.n) return 0.0f;
            if (f.outer == N) return t != m ? (float)g2re[(size_t)m * N + t] : 0.0f;
            return (float)g4re[encode_sorted(m, f.p[k], f.outer, t)];
        };
        size_t first[kSplit + 1];
        part_bounds(end, 1, first);
        out.nominal += end.empty() ? 0 : end.back();
        int* sc = &out.site_chunks[(size_t)m * (kSplit + 1)];
        for (int part = 0; part < kSplit; part++) {
            sc[part] = (int)out.chunk_start.size();
            const size_t e = std::max(first[part], first[part + 1]);
            site.clear();
            items.clear();
            for (size_t t = first[part]; t < e;) {
                const Four& f = fours[t];
                const bool two = t + 1 < e && f.n == 4 && f.outer < N && fours[t + 1].outer == f.outer &&
                                 fours[t + 1].lo == f.lo && fours[t + 1].hi == f.hi;
                const Four& f2 = fours[two ? t + 1 : t];
                const int v[8] = {f.p[0], f.p[1], f.p[2], f.p[3], f2.p[0], f2.p[1], f2.p[2], f2.p[3]};
                const int64_t at = (int64_t)site.size();
                emit_tile_header(site, f.outer, two ? 1 : 0, f.lo, f.hi - f.lo, two ? 4 + f2.n : f.n, v, N);
                for (int r = f.lo; r < f.hi; r++) {
                    site.push_back(make_int2(fbits(coef(f, 0, r)), fbits(coef(f, 1, r))));
                    site.push_back(make_int2(fbits(coef(f, 2, r)), fbits(coef(f, 3, r))));
                    if (!two) continue;
                    site.push_back(make_int2(fbits(coef(f2, 0, r)), fbits(coef(f2, 1, r))));
                    site.push_back(make_int2(fbits(coef(f2, 2, r)), fbits(coef(f2, 3, r))));
                }
                items.push_back({at, (int64_t)site.size()});
                t += two ? 2 : 1;
            }
            pack_part(site, items, 0, items.size(), out);
        }
        sc[kSplit] = (int)out.chunk_start.size();
    }
}

// Per record, per replica: a group costs 14 operations for its fold (a_p
// conj(a_o1): 2 FMA + 2 MUL; the field update: 4 FMA) and 4 per term (2 FMA); a
// tile 14 per column and 4 per coupling of its rows, zeros included.
double list_exec_flops(const SiteLists& L, int N) {
    double total = 0.0;
    const int64_t nchunks = (int64_t)L.chunk_start.size();
    for (int64_t c = 0; c < nchunks; c++) {
        const int64_t b = L.chunk_start[c];
        const int64_t n = ((c + 1 < nchunks) ? L.chunk_start[c + 1] : (int64_t)L.entries.size()) - b;
        const int2* R = L.entries.data() + b;
        if (L.tiles) {
            for (int64_t u = 0; u < n;) {
                const int wide = (R[u].x >> 16) & 1 ? 8 : 4, rows = (R[u].y >> 16) & 0xFF, cols = (R[u].y >> 24) & 0xFF;
                total += 14.0 * cols + 4.0 * wide * rows;
                u += wide / 2 + (int64_t)rows * wide / 2;
            }
        } else {
            for (int64_t u = 0; u + 1 < n; u += 2) total += 4.0 + (R[u + 1].y ? 14.0 : 0.0);
        }
    }
    return total;
}

bool records_single_groups(const SiteLists& L) {
    if (L.tiles) return false;
    for (size_t u = 0; u + 1 < L.entries.size(); u += 2)
        if (L.entries[u + 1].y != 1) return false;
    return true;
}

void build_q64(const std::vector<QuartetRec>& qs, std::vector<Q64>& out) {
    out.resize(qs.size());
    for (size_t t = 0; t < qs.size(); t++) {
        const QuartetRec& r = qs[t];
        out[t].i = (uint16_t)r.i;
        out[t].j = (uint16_t)r.j;
        out[t].k = (uint16_t)r.k;
        out[t].lch = (uint16_t)(r.l | (r.ch << 14));
        out[t].g = r.g;
    }
}

void dense_quartets(int N, const double* g4re, const uint8_t* mask, std::vector<QuartetRec>& out) {
    out.clear();
    int64_t q = 0;
    for (int l = 3; l < N; l++)
        for (int k = 2; k < l; k++)
            for (int j = 1; j < k; j++)
                for (int i = 0; i < j; i++, q++) {
                    const uint8_t m = mask[q];
                    const double g = g4re[q];
                    if (m == 0 || g == 0.0) continue;       // mc.cu:249
                    for (int ch = 0; ch < 3; ch++)
                        if (m & (1 << ch)) out.push_back(QuartetRec{i, j, k, l, ch, g});
                }
}

}  // namespace pspin
