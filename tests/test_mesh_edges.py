"""Opposite faces across mesh edges: against an ordered multimap of the unpaired half-edges (the earliest
one of the opposite direction), on meshes with borders, repeated, degenerate and same-way edges,
through walks and through the table; and no slower than the map where one vertex has every face."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "mesh_edges.h"
#include <chrono>
#include <cstdio>
#include <map>
#include <numeric>
#include <random>
using namespace std;
static vector<int64_t> by_map(const vector<uint32_t>& t) {
    vector<int64_t> opp(t.size(), -1);
    multimap<pair<uint32_t, uint32_t>, uint32_t> open;
    for (uint32_t e = 0; e < t.size(); e++) {
        const uint32_t u = t[e], v = t[3 * (e / 3) + (e % 3 + 1) % 3];
        auto it = open.lower_bound({v, u});
        if (it != open.end() && it->first == make_pair(v, u)) {
            opp[e] = it->second / 3;
            opp[it->second] = e / 3;
            open.erase(it);
        } else {
            open.emplace(make_pair(u, v), e);
        }
    }
    return opp;
}
static double now() { return chrono::duration<double>(chrono::steady_clock::now().time_since_epoch()).count(); }
int main() {
    mt19937 g(7);
    int wrong = 0;
    for (int r = 0; r < 400; r++) {  // soups of a few vertices: every kind of edge; the larger ones outgrow the walks
        const uint32_t nv = 1 + g() % 9, nf = r % 4 ? g() % 40 : 2000;
        vector<uint32_t> t(3 * nf);
        for (auto& x : t) x = g() % nv;
        wrong += vfd::opposite_faces(t.data(), nv, nf) != by_map(t);
    }
    const uint32_t n = 100000;  // a fan, its faces shuffled
    vector<uint32_t> order(n), t;
    iota(order.begin(), order.end(), 0u);
    shuffle(order.begin(), order.end(), g);
    for (uint32_t i : order)
        for (uint32_t x : {0u, 1 + i, 1 + (i + 1) % n}) t.push_back(x);
    const double t0 = now();
    const auto a = vfd::opposite_faces(t.data(), n + 1, n);
    const double t1 = now();
    const auto b = by_map(t);
    const double t2 = now();
    printf("%d %d %d", wrong, (int)(a == b), (int)(t1 - t0 < 1.5 * (t2 - t1)));
    fprintf(stderr, "fan %.1f ms, map %.1f ms\\n", 1e3 * (t1 - t0), 1e3 * (t2 - t1));
}
"""


def test_pairs_are_the_earliest_and_a_fan_is_not_quadratic(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "vfd_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, check=True)
    print(r.stderr)
    assert r.stdout == "0 1 1"
