// Replays of a batch's captured graph after its points have moved: the pair lists' length
// changes with the points, within what the workspace holds. Each replay must do what an
// eager run does: the counters of its passes say so, and its cells are a new batch's.
#include <cstdio>
#include <cstring>
#include <vector>

#include "engine.h"

using namespace cmg::gpu;

namespace {

// An octahedron of half-width s about (0.5, 0.5, 0.5).
std::vector<double> points(double s) {
    std::vector<double> p;
    for (int a = 0; a < 3; ++a)
        for (int sign = -1; sign <= 1; sign += 2)
            for (int q = 0; q < 3; ++q) p.push_back(0.5 + (q == a ? sign * s : 0.0));
    return p;
}
const int kTris[24] = {1, 3, 5, 3, 0, 5, 0, 2, 5, 2, 1, 5, 3, 1, 4, 0, 3, 4, 2, 0, 4, 1, 2, 4};

HostMesh mesh(const std::vector<double>& p) {
    HostMesh m;
    m.pts = p.data();
    m.npts = 6;
    m.tris = kTris;
    m.ntris = 8;
    m.g = GridDesc{};
    m.g.h = 1.0 / 61;
    m.g.nx = m.g.ny = m.g.nz = 61;
    return m;
}

struct Seen {
    std::vector<HostResult> r;
    RunInfo info;
};
Seen take(Batch& b) {
    Seen s;
    b.download(s.r, &s.info);
    s.info = b.info();
    return s;
}
bool same(const Seen& a, const Seen& b, bool distances) {
    const size_t n = a.r[0].occ.size();
    const Stats &s = a.info.stats, &t = b.info.stats;
    return n == b.r[0].occ.size() && std::memcmp(a.r[0].occ.data(), b.r[0].occ.data(), n) == 0 &&
           (!distances || std::memcmp(a.r[0].sdf64.data(), b.r[0].sdf64.data(), 8 * n) == 0) &&
           s.pairs == t.pairs && s.crossings == t.crossings && s.orient_calls == t.orient_calls &&
           s.flagged_columns == t.flagged_columns && s.candidates == t.candidates;
}

int check(bool distances) {
    VoxOpts o;
    o.want_occ = true;
    o.want_sdf64 = distances;
    std::vector<double> wide = points(0.45);
    Batch b({mesh(wide)}, o, cudaStreamPerThread);  // (the default stream cannot be captured)
    b.run();  // the workspace holds the widest mesh's lists
    int bad = 0;
    for (double s : {0.1, 0.4, 0.25, 0.45, 0.05}) {
        const std::vector<double> p = points(s);
        b.update_points({mesh(p)});
        Batch fresh({mesh(p)}, o, cudaStreamPerThread);
        fresh.run();
        const Seen want = take(fresh);
        for (int replay = 0; replay < 3; ++replay) {  // sized, captured, replayed
            b.run_graph();
            b.synchronize();
            if (!same(take(b), want, distances)) {
                std::fprintf(stderr, "half-width %g, run %d%s: not an eager run's results\n", s, replay,
                             distances ? ", with distances" : "");
                ++bad;
            }
        }
    }
    return bad;
}

}  // namespace

int main() { return check(false) + check(true) ? 1 : 0; }
