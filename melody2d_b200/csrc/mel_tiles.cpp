// Host builder of the tiles (layout in mel_tiles.h).
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <new>
#include <numeric>
#include <thread>
#include "mel_tiles.h"

void mel_set_error(const char* fmt, ...);

mel_tile_set::~mel_tile_set() { free(data); }

namespace {

size_t up16(size_t v) { return (v + 15) & ~(size_t)15; }

// rows a group whose largest point has K supports takes: the mixed form loads them in pairs
int rows_of(int K, bool mixed) { return mixed ? (K + 1) & ~1 : K; }

// slots that points with supports ns[0..n) take
int slots_of(const int* ns, int n, bool mixed, std::vector<int>& v)
{
    const int places = MEL_PLACES(mixed);
    v.assign(ns, ns + n);
    std::sort(v.begin(), v.end(), std::greater<int>());
    int s = 0;
    for (int t = 0; t < n; t += 32) s += ((std::min(32, n - t) + places - 1) / places) * places * rows_of(v[t], mixed);
    return s;
}

void put16(uint64_t& word, int k, uint32_t v) { word = (word & ~(0xffffull << (16 * k))) | ((uint64_t)v << (16 * k)); }

struct body_plan {
    std::vector<mel_tile> tiles;     // base relative to the body's first byte
    std::vector<int> gp0;            // first point of each tile
    size_t bytes = 0;
    long long entries = 0, pull = 0;
};

struct scratch {
    std::vector<int> v, order, cnt, first, nodes, w_of, r_of, mate_w, mate_r, pend, cls;
    std::vector<std::pair<int, int>> tn;
};

// the points of body b cut into tiles, and the size of each section; a failure with its point
std::pair<mel_status, int> plan_body(const mel_model_desc* d, int b, int cap, bool mixed, body_plan& P, scratch& S)
{
    const int places = MEL_PLACES(mixed), nnb = d->body_node_ptr[b + 1] - d->body_node_ptr[b];
    const int g1 = d->body_gp_ptr[b + 1];
    std::vector<int> ns;
    S.cnt.assign(nnb, 0);
    for (int g = d->body_gp_ptr[b]; g < g1;) {
        const int most = std::min(MEL_TILE_GP, g1 - g);
        ns.resize(most);
        for (int i = 0; i < most; i++) {
            const int c = d->gp_sup_ptr[g + i + 1] - d->gp_sup_ptr[g + i];
            if (c > 255 || c <= 0) return { MEL_ERR_UNSUPPORTED, g + i };
            ns[i] = c;
        }
        // the slots grow with every point: the most points that fit, by bisection
        int n = most;
        if (slots_of(ns.data(), most, mixed, S.v) > cap) {
            int lo = 1, hi = most;               // lo fits, hi does not
            while (hi - lo > 1) {
                const int mid = (lo + hi) / 2;
                if (slots_of(ns.data(), mid, mixed, S.v) <= cap) lo = mid; else hi = mid;
            }
            n = lo;
        }
        slots_of(ns.data(), n, mixed, S.v);      // (one point always fits: cap >= 256 MEL_PLACES)
        // S.v: the counts of the n points, sorted
        size_t head = 0, tail = 0, words = 0;
        for (int t = 0; t < n; t += 32) {
            const int w = ((std::min(32, n - t) + places - 1) / places) * places, K = S.v[t];
            head += (size_t)w * std::min(rows_of(K, mixed), MEL_TILE_HEAD(mixed));
            tail += (size_t)w * std::max(rows_of(K, mixed) - MEL_TILE_HEAD(mixed), 0);
            words += (size_t)w * ((K + 3) / 4);
        }
        S.nodes.clear();
        for (int j = d->gp_sup_ptr[g]; j < d->gp_sup_ptr[g + n]; j++) {
            const int v = d->gp_sup_idx[j];
            if (v < 0 || v >= nnb) return { MEL_ERR_INVALID, g };
            if (S.cnt[v]++ == 0) S.nodes.push_back(v);
        }
        S.v.clear();
        for (int v : S.nodes) { S.v.push_back(S.cnt[v]); S.cnt[v] = 0; }
        std::sort(S.v.begin(), S.v.end(), std::greater<int>());
        size_t pwords = 0;
        for (size_t t = 0; t < S.v.size(); t += 32) pwords += 32 * (size_t)((S.v[t] + 3) / 4);
        const size_t pb = mixed ? 8 : 16, tail16 = up16(tail * pb) / 16;
        const size_t rec16 = up16(head * pb) / 16, idx16 = tail16 + up16(8 * words) / 16, pos16 = pwords / 2;
        mel_tile T;
        T.base = (unsigned)(P.bytes / 128);
        T.rec_idx = (unsigned)(rec16 | (idx16 << 16));
        T.counts = (unsigned)n | ((unsigned)S.v.size() << 16);
        T.pos = (unsigned)(pos16 | (tail16 << 16));
        P.bytes += (mel_tile_o_slot(T.rec_idx, T.counts) + mel_tile_pull_bytes(T.counts, T.pos) + 127) & ~(size_t)127;
        P.tiles.push_back(T);
        P.gp0.push_back(g);
        P.entries += d->gp_sup_ptr[g + n] - d->gp_sup_ptr[g];
        P.pull += (int)S.v.size();
        g += n;
    }
    return { MEL_OK, 0 };
}

// Colours the edges e (between vertex w_of[e] and vertex r_of[e]) so that the edges of a vertex all
// differ, with 2^levels colours where every vertex has at most that many edges.  Each level halves
// the classes: the edges of a class are paired up at every vertex, and along the chains that the
// pairs form (of even length where they close, the graph being bipartite) they go to the two
// halves in turn.
void colour(scratch& S, int ne, int nw, int nr, int levels)
{
    S.cls.assign(ne, 0);
    for (int lev = 0; lev < levels; lev++) {
        const int nc = 1 << lev;
        S.mate_w.assign(ne, -1);
        S.mate_r.assign(ne, -1);
        auto pair_up = [&](const std::vector<int>& of, int nv, std::vector<int>& mate) {
            S.pend.assign((size_t)nv * nc, -1);
            for (int e = 0; e < ne; e++) {
                int& p = S.pend[(size_t)of[e] * nc + S.cls[e]];
                if (p < 0) p = e;
                else { mate[e] = p; mate[p] = e; p = -1; }
            }
        };
        pair_up(S.w_of, nw, S.mate_w);
        pair_up(S.r_of, nr, S.mate_r);
        // S.v: the half of each edge, -1 while open
        S.v.assign(ne, -1);
        auto walk = [&](int e, bool by_w) {
            for (int h = 0; e >= 0 && S.v[e] < 0; h ^= 1, by_w = !by_w) {
                S.v[e] = h;
                e = by_w ? S.mate_w[e] : S.mate_r[e];
            }
        };
        for (int e = 0; e < ne; e++) {
            if (S.v[e] >= 0) continue;
            if (S.mate_w[e] < 0) walk(e, false);            // an end of a chain: leave by the other mate
            else if (S.mate_r[e] < 0) walk(e, true);
        }
        for (int e = 0; e < ne; e++) if (S.v[e] < 0) walk(e, true);
        for (int e = 0; e < ne; e++) S.cls[e] = 2 * S.cls[e] + S.v[e];
    }
}

bool fill_tile(const mel_model_desc* d, const mel_tile& T, int g, int nnb, bool mixed, int cap, uint8_t* base, scratch& S)
{
    const int places = MEL_PLACES(mixed), n = (int)(T.counts & 0xffffu), nslot = (int)(T.counts >> 16);
    S.order.resize(n);
    std::iota(S.order.begin(), S.order.end(), 0);
    const int* sp = d->gp_sup_ptr + g;
    std::stable_sort(S.order.begin(), S.order.end(), [&](int a, int c) { return sp[a + 1] - sp[a] > sp[c + 1] - sp[c]; });
    mel_point* rec = reinterpret_cast<mel_point*>(base + mel_tile_o_rec(T.rec_idx));
    uint8_t* const tail = base + mel_tile_o_idx(T.rec_idx, T.counts);
    uint64_t* idx = reinterpret_cast<uint64_t*>(tail + mel_tile_tail_bytes(T.pos));
    mel_pull* slot = reinterpret_cast<mel_pull*>(base + mel_tile_o_slot(T.rec_idx, T.counts));
    uint64_t* pos = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(slot) + ((8 * nslot + 15) & ~15));
    // point groups: records, pairs and, per entry (points ascending), its row of slots
    const int e0 = sp[0], ne = sp[n] - e0;
    S.w_of.resize(ne);
    const int H = MEL_TILE_HEAD(mixed);
    int s0 = 0, i0 = 0, tl = 0;
    for (int t0 = 0; t0 < n; t0 += 32) {
        const int m = std::min(32, n - t0), w = ((m + places - 1) / places) * places;
        const int K = sp[S.order[t0] + 1] - sp[S.order[t0]];
        for (int l = 0; l < m; l++) {
            const int t = S.order[t0 + l], gg = g + t, c = sp[t + 1] - sp[t];
            mel_point& R = rec[t0 + l];
            R.c0 = d->gp_weight[gg] * d->gp_jacobian[gg];    // c0 of Code/Body.h:994
            R.a = (uint32_t)s0 | ((uint32_t)c << 16) | ((uint32_t)K << 24);
            R.i = (uint32_t)i0 | ((uint32_t)(w / 8 - 1) << 14) | ((uint32_t)tl << 16);
            for (int k = 0; k < c; k++) {
                const int j = sp[t] + k;
                S.w_of[j - e0] = (s0 + k * w + l) / places;
                uint8_t* const at = k < H ? base : tail;
                const size_t o = k < H ? (size_t)(s0 - tl) : (size_t)tl;
                const int kk = k < H ? k : k - H;
                if (mixed) {
                    float* p = reinterpret_cast<float*>(at) + 2 * (o + (size_t)(kk / 2) * 2 * w + 2 * l + (kk & 1));
                    p[0] = (float)d->gp_dNdx[j];
                    p[1] = (float)d->gp_dNdy[j];
                } else {
                    double* p = reinterpret_cast<double*>(at) + 2 * (o + (size_t)kk * w + l);
                    p[0] = d->gp_dNdx[j];
                    p[1] = d->gp_dNdy[j];
                }
            }
        }
        s0 += rows_of(K, mixed) * w;
        tl += std::max(rows_of(K, mixed) - H, 0) * w;
        i0 += ((K + 3) / 4) * w;
    }
    if (s0 > 65535 || i0 > 16383) return false;
    const int nw = s0 / places;
    // touched nodes by entry count, and every entry's reading wavefront
    S.cnt.assign(nnb, 0);
    S.nodes.clear();
    for (int j = e0; j < e0 + ne; j++) {
        const int v = d->gp_sup_idx[j];
        if (S.cnt[v]++ == 0) S.nodes.push_back(v);
    }
    std::sort(S.nodes.begin(), S.nodes.end());
    S.tn.clear();
    for (int v : S.nodes) S.tn.push_back({ v, S.cnt[v] });
    std::stable_sort(S.tn.begin(), S.tn.end(), [](const std::pair<int, int>& a, const std::pair<int, int>& c) { return a.second > c.second; });
    if ((int)S.tn.size() != nslot) return false;
    // S.first: the pull slot of a node; entries are met in ascending point order
    S.first.assign(nnb, 0);
    std::vector<int> group_w((size_t)(nslot + 31) / 32), group_r(group_w.size());
    int pw = 0, nr = 0;
    for (int t = 0; t < nslot; t++) {
        if ((t & 31) == 0) {
            group_w[t / 32] = pw;
            group_r[t / 32] = nr;
            pw += 32 * ((S.tn[t].second + 3) / 4);
            nr += (32 / places) * S.tn[t].second;
        }
        S.first[S.tn[t].first] = t;
        slot[t].node = (uint32_t)S.tn[t].first | ((uint32_t)S.tn[t].second << 16);
        slot[t].p0 = (uint32_t)group_w[t / 32];
        S.cnt[S.tn[t].first] = 0;                // from here on: entries of the node met so far
    }
    S.r_of.resize(ne);
    for (int j = 0; j < ne; j++) {
        const int v = d->gp_sup_idx[e0 + j], t = S.first[v];
        S.r_of[j] = group_r[t / 32] + (32 / places) * S.cnt[v] + (t & 31) / places;
        S.cnt[v]++;
    }
    colour(S, ne, nw, nr, mixed ? 4 : 3);
    // padding: the node after the body's last, the slot after the cap
    const uint64_t pad_i = (uint64_t)(nnb < 0x1000 ? nnb : 0) * 0x0001000100010001ull, pad_p = (uint64_t)cap * 0x0001000100010001ull;
    std::fill(idx, idx + i0, pad_i);
    std::fill(pos, pos + pw, pad_p);
    for (int v : S.nodes) S.cnt[v] = 0;
    // S.order maps a slot to its point; entries in point order
    S.v.assign(n, 0);
    for (int s = 0; s < n; s++) S.v[S.order[s]] = s;
    for (int t = 0; t < n; t++) {
        const int l = S.v[t] & 31;
        const mel_point& R = rec[S.v[t]];
        const int gi0 = (int)(R.i & 0x3fffu), gw = 8 * ((int)((R.i >> 14) & 3u) + 1);
        for (int k = 0, j = sp[t] - e0; j < sp[t + 1] - e0; k++, j++) {
            const int v = d->gp_sup_idx[e0 + j], u = S.first[v], c = S.cnt[v]++;
            const int place = S.cls[j];
            put16(idx[(size_t)gi0 + (size_t)(k / 4) * gw + l], k & 3, (uint32_t)v | ((uint32_t)place << 12));
            put16(pos[(size_t)group_w[u / 32] + (size_t)(c / 4) * 32 + (u & 31)], c & 3, (uint32_t)(S.w_of[j] * places + place));
        }
    }
    return true;
}

}  // namespace

// f(body, scratch) for every tiled body, on a few host threads (bodies are independent); false when memory
// ran out in one of them (an exception must not leave a thread, nor this one while others run)
template <class F>
static bool over_bodies(const mel_model_desc* d, F&& f)
{
    const int nb = d->n_bodies, hw = (int)std::thread::hardware_concurrency();
    const long long work = d->gp_sup_ptr[d->n_gauss];
    const int nthr = std::max(1, std::min({ hw > 0 ? hw : 1, 16, nb, (int)(work / 200000) + 1 }));
    std::atomic<int> next{ 0 };
    std::atomic<bool> good{ true };
    auto run = [&]() {
        try {
            scratch S;
            for (int b; good && (b = next++) < nb;)
                if (d->body_type[b] == MEL_BODY_DEFORMABLE && d->body_node_ptr[b + 1] - d->body_node_ptr[b] <= MEL_MAX_BODY_NODES) f(b, S);
        } catch (const std::bad_alloc&) {
            good = false;
        }
    };
    std::vector<std::thread> th;
    for (int i = 1; i < nthr; i++) {
        try { th.emplace_back(run); } catch (...) { break; }      // fewer threads do
    }
    run();
    for (auto& t : th) t.join();
    return good;
}

static mel_status no_memory()
{
    mel_set_error("no host memory for the Gauss-point tiles");
    return MEL_ERR_OOM;
}

mel_status mel_plan_tiles(const mel_model_desc* d, int cap, bool mixed, mel_tile_set& out)
try {
    const int nb = d->n_bodies;
    if (cap < 256 * MEL_PLACES(mixed) || cap > 16384) { mel_set_error("tile cap %d out of range", cap); return MEL_ERR_INVALID; }
    std::vector<body_plan> plan(nb);
    std::vector<std::pair<mel_status, int>> rc(nb, { MEL_OK, 0 });
    if (!over_bodies(d, [&](int b, scratch& S) { rc[b] = plan_body(d, b, cap, mixed, plan[b], S); })) return no_memory();
    for (int b = 0; b < nb; b++) {
        if (rc[b].first == MEL_OK) continue;
        if (rc[b].first == MEL_ERR_INVALID) mel_set_error("Gauss support index out of range");
        else mel_set_error("Gauss point %d has %d supports (1..255 supported)", rc[b].second, d->gp_sup_ptr[rc[b].second + 1] - d->gp_sup_ptr[rc[b].second]);
        return rc[b].first;
    }
    out.cap = cap;
    out.mixed = mixed;
    out.b_tile0.assign(nb + 1, 0);
    out.tiles.clear();
    out.gp0.clear();
    out.n_entries = out.n_points = out.n_pull = 0;
    out.max_idx = out.max_pull = 16;
    size_t total = 0;
    for (int b = 0; b < nb; b++) {
        out.b_tile0[b] = (int)out.tiles.size();
        for (mel_tile T : plan[b].tiles) {
            T.base += (unsigned)(total / 128);
            out.tiles.push_back(T);
            out.n_points += T.counts & 0xffffu;
            out.max_idx = std::max(out.max_idx, mel_tile_idx_bytes(T.rec_idx));
            out.max_pull = std::max(out.max_pull, mel_tile_pull_bytes(T.counts, T.pos));
        }
        out.gp0.insert(out.gp0.end(), plan[b].gp0.begin(), plan[b].gp0.end());
        total += plan[b].bytes;
        out.n_entries += plan[b].entries;
        out.n_pull += plan[b].pull;
    }
    out.b_tile0[nb] = (int)out.tiles.size();
    out.bytes = total;
    return MEL_OK;
} catch (const std::bad_alloc&) {
    return no_memory();
}

mel_status mel_fill_tiles(const mel_model_desc* d, mel_tile_set& out)
try {
    free(out.data);
    out.data = static_cast<uint8_t*>(calloc(std::max<size_t>(out.bytes, 16), 1));
    if (!out.data) { mel_set_error("host memory for the Gauss-point tiles (%zu bytes)", out.bytes); return MEL_ERR_OOM; }
    std::atomic<bool> good{ true };
    const bool room = over_bodies(d, [&](int b, scratch& S) {
        const int nnb = d->body_node_ptr[b + 1] - d->body_node_ptr[b];
        for (int i = out.b_tile0[b]; i < out.b_tile0[b + 1]; i++)
            if (!fill_tile(d, out.tiles[i], out.gp0[i], nnb, out.mixed, out.cap, out.data + mel_tile_base(out.tiles[i].base), S)) good = false;
    });
    if (!room) return no_memory();
    if (!good) { mel_set_error("the Gauss-point tiles do not hold their points"); return MEL_ERR_INVALID; }
    return MEL_OK;
} catch (const std::bad_alloc&) {
    return no_memory();
}
