// layout.h -- host builders for the sweep's site lists and the FP64 quartet table.
#pragma once
#include <vector>
#include <cstdint>
#include "internal.h"

namespace pspin {

struct QuartetRec {
    int i, j, k, l;   // sorted
    int ch;           // 0, 1, 2
    double g;         // rescaled coupling (real)
};

struct SiteLists {
    std::vector<int2> entries;         // sample-relative
    std::vector<int64_t> chunk_start;  // sample-relative entry offset of each chunk (no sentinel)
    std::vector<int> site_chunks;      // N*(kSplit+1) sample-relative chunk indices
    int64_t nominal = 0;               // entries of the untiled lists (the size the parts are balanced by)
    bool tiles = false;                // dense tiles (else group records, or groups)
};

// A site's terms are sorted by (p, o1, o2) into groups of equal (p, o1), at
// most kGroupMax terms each; the groups are cut in kSplit balanced parts.
// kRecords: a group counts, and is stored, as one 16-byte record {g, o2,
// p<<16|o1, last} per term; kGroups: as a header {len, p<<16|o1} and one entry
// {g, o2} per term.  The two formats have different sizes and so different
// part bounds, which fix the order the fields are summed in.
enum GroupSize { kGroups, kRecords };

// Per-site lists; `size` gives the part bounds.  tile: stored as dense tiles
// (see tile_parts) where those are the cheaper to read, with the same parts
// and the same order of additions; otherwise in the format of `size`.
void build_site_lists(int N, const double* g2re, int h2_active, const std::vector<QuartetRec>& qs, SiteLists& out,
                      GroupSize size, bool tile);
// Sub-lists of the terms that couple the two sites of a pair (as groups, or with
// `tile` as dense tiles where those are cheaper to read):
// for i < j and P = j(j-1)/2 + i, list 2P holds site i's terms that contain
// a_j, list 2P+1 site j's terms that contain a_i.  Each term of a site list
// is in 3 of them (one per other site of its quartet).
void build_pair_lists(int N, const double* g2re, int h2_active, const std::vector<QuartetRec>& qs,
                      SiteLists& out, bool tile);
// fully connected lists as dense tiles, from the dense g4 (channel 0
// everywhere) and g2
void build_site_tiles_fc(int N, const double* g2re, int h2_active, const double* g4re, SiteLists& out);
void build_q64(const std::vector<QuartetRec>& qs, std::vector<Q64>& out);
// site lists in the record format: does every record end its group?
bool records_single_groups(const SiteLists& L);

// FP32 operations the sweep kernels execute, per replica, to accumulate the
// lists of all N sites once (the expected work of one sweep's N/2 moves over
// their two sites each), walking the packed chunks as the kernels do (padding
// couplings included).
double list_exec_flops(const SiteLists& L, int N);
// every active (q, ch) of a dense mask in q order
void dense_quartets(int N, const double* g4re, const uint8_t* mask, std::vector<QuartetRec>& out);

}  // namespace pspin
