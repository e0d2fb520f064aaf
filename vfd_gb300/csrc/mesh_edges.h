// Opposite faces across a triangle mesh's edges (host code).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace vfd {

// Half-edge e = 3 f + k runs from tri[e] to the next corner of face f. Taken in order, each is paired
// with the earliest unpaired one of the opposite direction; opp[e] is then that one's face, -1 on
// a border. Indices are below nv.
//
// The unpaired half-edges of each source vertex are a list in face order, threaded through
// `next`, which a lookup walks: two or three steps at a vertex of six faces. Where vertices of very
// many faces make the walks long (in sum more than kWalk a half-edge), a hash table of the
// directed edges, each with its list, takes over: 20,402 faces take 0.9 ms by walks and 3.2 by the
// table (an ordered map 3.3), a fan of 100,000 shuffled faces 3,400 by walks alone, 41 so (240).
constexpr uint64_t kWalk = 8;
inline std::vector<int64_t> opposite_faces(const uint32_t* tri, uint32_t nv, uint32_t nf) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    const size_t ne = 3 * (size_t)nf;
    auto target = [&](uint32_t e) { return tri[3 * (e / 3) + (e % 3 + 1) % 3]; };
    std::vector<int64_t> opp(ne, -1);
    std::vector<uint32_t> head(nv, kNone), tail(nv, kNone), next(ne, kNone);
    uint64_t left = kWalk * ne;
    for (uint32_t f = 0; f < nf && left > 0; f++)
        for (uint32_t k = 0; k < 3; k++) {
            const uint32_t e = 3 * f + k, u = tri[e], v = tri[3 * f + (k + 1) % 3];
            uint32_t before = kNone, o = head[v];
            for (; o != kNone && target(o) != u && left > 0; left--) {
                before = o;
                o = next[o];
            }
            if (left == 0) break;
            if (o != kNone) {
                opp[e] = o / 3;
                opp[o] = f;
                (before == kNone ? head[v] : next[before]) = next[o];
                if (tail[v] == o) tail[v] = before;
            } else {
                (tail[u] == kNone ? head[u] : next[tail[u]]) = e;
                tail[u] = e;
            }
        }
    if (left > 0) return opp;

    // an edge's slot: its first half-edge names it, then its unpaired ones in order
    struct Slot {
        uint32_t name, head, tail;
    };
    size_t size = 16;
    while (size < 2 * ne) size *= 2;
    std::vector<Slot> table(size, Slot{kNone, kNone, kNone});
    auto find = [&](uint32_t u, uint32_t v) -> Slot& {
        uint64_t h = ((uint64_t)u << 32 | v) * 0x9E3779B97F4A7C15ull;
        h = (h ^ h >> 32) * 0x9E3779B97F4A7C15ull;
        for (size_t k = h >> 32 & (size - 1);; k = (k + 1) & (size - 1)) {
            Slot& s = table[k];
            if (s.name == kNone || (tri[s.name] == u && target(s.name) == v)) return s;
        }
    };
    std::fill(opp.begin(), opp.end(), -1);
    for (uint32_t e = 0; e < ne; e++) {
        const uint32_t u = tri[e], v = target(e);
        Slot& other = find(v, u);
        if (other.name != kNone && other.head != kNone) {
            const uint32_t o = other.head;
            opp[e] = o / 3;
            opp[o] = e / 3;
            other.head = next[o];
            if (other.head == kNone) other.tail = kNone;
        } else {
            Slot& own = find(u, v);
            if (own.name == kNone) own.name = e;
            next[e] = kNone;
            (own.tail == kNone ? own.head : next[own.tail]) = e;
            own.tail = e;
        }
    }
    return opp;
}

}  // namespace vfd
