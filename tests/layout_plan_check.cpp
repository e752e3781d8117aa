// CPU check of plan_layout_passes (engine.cpp, included below): on random gate
// lists, the passes' gates applied on positions, each pass's reordering of its
// tile bits and the final chunk bit moves give the same dense state as the
// gates applied one by one; every pass's gates mix only tile bits, a tile has
// at most jmax bits above the chunk, and the order of the qubits is restored.
//
//   layout_plan_check <seed> <lists>
#include "engine.cpp"

#include <cstdio>
#include <cstdlib>
#include <random>

static void apply(std::vector<cplx> &v, const CGate &g) {
    const int dim = 1 << g.nq;
    uint64_t used = 0;
    for (int b = 0; b < g.nq; ++b) used |= 1ull << g.q[b];
    std::vector<cplx> in(dim);
    for (uint64_t base = 0; base < v.size(); ++base) {
        if (base & used) continue;
        auto at = [&](int r) {
            uint64_t i = base;
            for (int b = 0; b < g.nq; ++b) i |= (uint64_t)((r >> b) & 1) << g.q[b];
            return i;
        };
        for (int r = 0; r < dim; ++r) in[r] = v[at(r)];
        for (int r = 0; r < dim; ++r) {
            cplx acc = 0;
            for (int c = 0; c < dim; ++c) acc += g.m[r * dim + c] * in[c];
            v[at(r)] = acc;
        }
    }
}

static CGate random_gate(std::mt19937_64 &rng, int n, int kind, int chain) {
    std::normal_distribution<double> nd;
    auto cn = [&] { return cplx(nd(rng), nd(rng)) * 0.5; };
    CGate g;
    const int a = chain >= 0 ? chain : (int)(rng() % n);
    int b = chain >= 0 ? a + 1 : (int)(rng() % n);
    while (b == a || b >= n) b = (int)(rng() % n);
    if (kind == 0) {  // one qubit
        g.nq = 1;
        g.q[0] = a;
        for (int i = 0; i < 4; ++i) g.m[i] = cn();
    } else {
        g.nq = 2;
        g.q[0] = std::min(a, b);
        g.q[1] = std::max(a, b);
        for (int i = 0; i < 16; ++i) g.m[i] = 0;
        if (kind == 1)  // dense
            for (int i = 0; i < 16; ++i) g.m[i] = cn();
        else if (kind == 2)  // diagonal
            for (int i = 0; i < 4; ++i) g.m[5 * i] = cn();
        else {  // controlled: mixes q[0] where q[1] is 1
            g.m[0] = g.m[5] = 1;
            for (int r = 2; r < 4; ++r)
                for (int c = 2; c < 4; ++c) g.m[4 * r + c] = cn();
        }
    }
    compute_mixing(&g);
    return g;
}

int main(int argc, char **argv) {
    std::mt19937_64 rng(argc > 1 ? std::atoi(argv[1]) : 1);
    const int lists = argc > 2 ? std::atoi(argv[2]) : 60;
    int bad = 0, planned = 0, shuffled = 0;
    for (int t = 0; t < lists; ++t) {
        const int C = 2 + (int)(rng() % 3), jmax = 2 + (int)(rng() % 3);
        const int n = C + jmax + (int)(rng() % 4);
        const bool chain = t % 3 == 0;
        const int G = 1 + (int)(rng() % 60);
        std::vector<CGate> sg;
        for (int i = 0; i < G; ++i) sg.push_back(random_gate(rng, n, (int)(rng() % 4), chain ? (int)(rng() % (n - 1)) : -1));
        std::vector<LayoutPass> lay;
        std::vector<int> restore;
        if (!plan_layout_passes(sg, n, C, jmax, 1000, &lay, &restore)) {
            ++bad;
            continue;
        }
        ++planned;
        std::normal_distribution<double> nd;
        std::vector<cplx> v(1ull << n), w;
        for (auto &x : v) x = cplx(nd(rng), nd(rng));
        w = v;
        for (const CGate &g : sg) apply(v, g);
        std::vector<int> seen(G, 0);
        for (const LayoutPass &lp : lay) {
            if ((int)lp.tile.size() != jmax || lp.src.size() != (size_t)(C + jmax)) ++bad;
            std::vector<int> slot;
            for (int b = 0; b < C; ++b) slot.push_back(b);
            slot.insert(slot.end(), lp.tile.begin(), lp.tile.end());
            for (size_t k = 0; k < lp.gates.size(); ++k) {
                ++seen[lp.ids[k]];
                for (int b = 0; b < lp.gates[k].nq; ++b)
                    if (lp.gates[k].mix[b] && std::find(slot.begin(), slot.end(), lp.gates[k].q[b]) == slot.end()) ++bad;
                apply(w, lp.gates[k]);
            }
            std::vector<cplx> o(w.size());
            uint64_t tilemask = 0;
            for (int s : slot) tilemask |= 1ull << s;
            for (uint64_t i = 0; i < w.size(); ++i) {
                uint64_t from = i & ~tilemask;
                for (size_t b = 0; b < slot.size(); ++b) from |= ((i >> slot[b]) & 1) << slot[lp.src[b]];
                o[i] = w[from];
            }
            for (size_t b = 0; b < lp.src.size(); ++b) shuffled += lp.src[b] != (int)b;
            w.swap(o);
        }
        for (int s : seen) bad += s != 1;
        std::vector<cplx> o(w.size());
        for (uint64_t i = 0; i < w.size(); ++i) {
            uint64_t to = i & ((1ull << C) - 1);
            for (int s = 0; s < n - C; ++s) to |= ((i >> (s + C)) & 1) << (restore[s] + C);
            o[to] = w[i];
        }
        double err = 0, norm = 0;
        for (size_t i = 0; i < v.size(); ++i) {
            err += std::norm(o[i] - v[i]);
            norm += std::norm(v[i]);
        }
        if (err > 1e-24 * norm) ++bad;
    }
    printf("layout %s: %d lists planned, %d bits moved, %d failures\n", bad || !shuffled ? "failed" : "ok", planned,
           shuffled, bad);
    return bad || !shuffled;
}
