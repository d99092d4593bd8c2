// CPU model of the body kernel's Gauss-point pass over tiles (test infrastructure): follows the same
// records as the kernel, checks every index against the tile, the body and the slot cap, checks that no
// wavefront of writes or reads meets a place twice, and returns the internal nodal forces.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>
#include "mel_tiles.h"

static char g_err[512];
void mel_set_error(const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
}
extern "C" const char* emul_error() { return g_err; }

// f: 2 doubles per node.  FP64 tiles: the kernel's linear elastic pass.  Mixed tiles: contributions
// c0 (dN . up) and c0 (dN . up + dN.x) from the FP32 pairs, as a stand-in, and their direct scatter in
// f_direct.  stats: [tiles, entries, slots, most slots of a tile]
extern "C" int emul_tiles(const mel_model_desc* d, int cap, int mixed, const double* up, double* f, double* f_direct,
                          long long* stats)
{
    mel_tile_set TS;
    int rc = mel_plan_tiles(d, cap, mixed != 0, TS);
    if (rc == MEL_OK) rc = mel_fill_tiles(d, TS);
    if (rc != MEL_OK) return 100 + rc;
    const int P = MEL_PLACES(mixed);
    stats[0] = (long long)TS.tiles.size(); stats[1] = TS.n_entries; stats[2] = stats[3] = 0;
    memset(f, 0, sizeof(double) * 2 * (size_t)d->n_nodes);
    memset(f_direct, 0, sizeof(double) * 2 * (size_t)d->n_nodes);
    for (int b = 0; b < d->n_bodies; b++) {
        const int n0 = d->body_node_ptr[b], n = d->body_node_ptr[b + 1] - n0;
        const int mat = d->body_material[b];
        const double Mu = d->material_params[MEL_MAT_NPARAM * mat + 3], Lam = d->material_params[MEL_MAT_NPARAM * mat + 4];
        int gp = d->body_gp_ptr[b];
        for (int ti = TS.b_tile0[b]; ti < TS.b_tile0[b + 1]; ti++) {
            const mel_tile H = TS.tiles[ti];
            struct { int ngp, nslot, o_rec, o_idx, o_slot, o_pos; } T = {
                (int)(H.counts & 0xffffu), (int)(H.counts >> 16), mel_tile_o_rec(H.rec_idx), mel_tile_o_idx(H.rec_idx, H.counts),
                mel_tile_o_slot(H.rec_idx, H.counts), mel_tile_o_slot(H.rec_idx, H.counts) + ((8 * (int)(H.counts >> 16) + 15) & ~15) };
            const size_t next = ti + 1 < (int)TS.tiles.size() ? mel_tile_base(TS.tiles[ti + 1].base) : TS.bytes;
            const size_t size = (size_t)T.o_slot + mel_tile_pull_bytes(H.counts, H.pos);
            if (mel_tile_base(H.base) + size > next) return 1;
            if (T.ngp < 1 || T.ngp > MEL_TILE_GP || TS.gp0[ti] != gp) return 2;
            if (mel_tile_idx_bytes(H.rec_idx) > TS.max_idx || mel_tile_pull_bytes(H.counts, H.pos) > TS.max_pull) return 14;
            const uint8_t* base = TS.data + mel_tile_base(H.base);
            const mel_point* rec = reinterpret_cast<const mel_point*>(base + T.o_rec);
            const int H0 = MEL_TILE_HEAD(mixed), tailb = mel_tile_tail_bytes(H.pos);
            if (T.o_idx + tailb > T.o_slot) return 17;
            const uint64_t* idx = reinterpret_cast<const uint64_t*>(base + T.o_idx + tailb);
            const mel_pull* slot = reinterpret_cast<const mel_pull*>(base + T.o_slot);
            const uint64_t* pos = reinterpret_cast<const uint64_t*>(base + T.o_pos);
            std::vector<double> q(2 * (size_t)cap, 0.);
            std::vector<int> wrote(cap, -1), node_of(cap, -1), point_of(cap, -1);
            // which point a record is: sorted by (count descending, index)
            std::vector<int> order(T.ngp);
            for (int i = 0; i < T.ngp; i++) order[i] = gp + i;
            auto ns_of = [&](int g) { return d->gp_sup_ptr[g + 1] - d->gp_sup_ptr[g]; };
            std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return ns_of(a) > ns_of(c); });
            int slots = 0;
            for (int tid = 0; tid < T.ngp; tid++) {
                const int lane = tid & 31, w = 8 * ((int)((rec[tid].i >> 14) & 3u) + 1), ns = (int)((rec[tid].a >> 16) & 0xffu), K = (int)(rec[tid].a >> 24);
                const int s0 = (int)(rec[tid].a & 0xffffu), i0 = (int)(rec[tid].i & 0x3fffu), tl = (int)(rec[tid].i >> 16);
                if (w % P || w > 32 || lane >= w || ns < 1 || ns > K || (tid & 31 ? K != (int)(rec[tid - 1].a >> 24) : K != ns)) return 3;
                const int g = order[tid], j0 = d->gp_sup_ptr[g];
                if (ns != ns_of(g) || rec[tid].c0 != d->gp_weight[g] * d->gp_jacobian[g]) return 4;
                auto word = [&](int k) { const size_t o = (size_t)i0 + (size_t)(k / 4) * w + lane; return T.o_idx + tailb + 8 * (o + 1) <= (size_t)T.o_slot ? (unsigned)(idx[o] >> (16 * (k & 3))) & 0xffffu : 0xfffffu; };
                for (int k = ns; k < ((K + 3) & ~3); k++) if (word(k) != (unsigned)(n < 4096 ? n : 0)) return 15;      // padding
                auto pair = [&](int k, double* g2) {
                    const uint8_t* at = k < H0 ? base : base + T.o_idx;
                    const size_t end = k < H0 ? (size_t)T.o_rec : (size_t)tailb;
                    const int o0 = k < H0 ? s0 - tl : tl, kk = k < H0 ? k : k - H0;
                    if (mixed) {
                        const size_t o = (size_t)(o0 / 2 + (kk / 2) * w + lane);      // float4 index
                        if (o0 & 1 || 16 * (o + 1) > end) return false;
                        const float* p = reinterpret_cast<const float*>(at) + 4 * o + 2 * (kk & 1);
                        g2[0] = p[0]; g2[1] = p[1];
                        return p[0] == (float)d->gp_dNdx[j0 + k] && p[1] == (float)d->gp_dNdy[j0 + k];
                    }
                    const size_t o = (size_t)o0 + (size_t)kk * w + lane;
                    if (16 * (o + 1) > end) return false;
                    const double* p = reinterpret_cast<const double*>(at) + 2 * o;
                    g2[0] = p[0]; g2[1] = p[1];
                    return p[0] == d->gp_dNdx[j0 + k] && p[1] == d->gp_dNdy[j0 + k];
                };
                double E11 = 0., E12 = 0., E22 = 0., dn[2];
                for (int k = 0; k < ns; k++) {
                    const unsigned w16 = word(k);
                    const int i = (int)(w16 & 0xfffu);
                    if (w16 > 0xffffu || i >= n || i != d->gp_sup_idx[j0 + k] || !pair(k, dn)) return 5;
                    const double ux = up[2 * (n0 + i)], uy = up[2 * (n0 + i) + 1];
                    E11 = E11 + dn[0] * ux;
                    E12 = E12 + (dn[0] * uy + dn[1] * ux);
                    E22 = E22 + dn[1] * uy;
                }
                E12 = 0.5 * E12;
                const double J = 1. + E11 + E22, S33 = Lam * (J - 1.), Mu2 = 2 * Mu;
                const double S11 = S33 + Mu2 * E11, S22 = S33 + Mu2 * E22, S12 = Mu2 * E12;
                for (int k = 0; k < ns; k++) {
                    const unsigned w16 = word(k);
                    const int place = (int)(w16 >> 12), i = (int)(w16 & 0xfffu);
                    const int s = s0 + (lane & ~(P - 1)) + k * w + place;
                    if (place >= P || s >= cap || wrote[s] >= 0) return 6;       // a row's places are taken once
                    wrote[s] = tid; node_of[s] = i; point_of[s] = g;
                    slots = std::max(slots, s + 1);
                    pair(k, dn);
                    if (mixed) {
                        const double v = dn[0] * up[2 * (n0 + i)] + dn[1] * up[2 * (n0 + i) + 1];
                        q[2 * s] = rec[tid].c0 * v; q[2 * s + 1] = rec[tid].c0 * (v + dn[0]);
                        f_direct[2 * (n0 + i)] -= q[2 * s]; f_direct[2 * (n0 + i) + 1] -= q[2 * s + 1];
                    } else {
                        q[2 * s] = rec[tid].c0 * (dn[0] * S11 + dn[1] * S12);
                        q[2 * s + 1] = rec[tid].c0 * (dn[1] * S22 + dn[0] * S12);
                    }
                }
            }
            stats[2] += slots; stats[3] = std::max(stats[3], (long long)slots);
            std::vector<char> pulled(cap, 0);
            int maxcnt = 0;
            for (int s = 0; s < T.nslot; s++) {
                if (T.o_slot + 8 * (s + 1) > T.o_pos) return 7;
                const int node = (int)(slot[s].node & 0xffffu), cnt = (int)(slot[s].node >> 16), lane = s & 31;
                if (node >= n || cnt < 1 || ((s & 31) && (slot[s].p0 != slot[s - 1].p0 || cnt > (int)(slot[s - 1].node >> 16)))) return 8;
                maxcnt = std::max(maxcnt, cnt);
                double fx = f[2 * (n0 + node)], fy = f[2 * (n0 + node) + 1];
                int last = -1;
                for (int j = cnt; j < (((int)(slot[s & ~31].node >> 16) + 3) & ~3); j++) {
                    const size_t o = (size_t)slot[s].p0 + 8 * (size_t)(j & ~3) + lane;
                    if (T.o_pos + 8 * (o + 1) > size || ((pos[o] >> (16 * (j & 3))) & 0xffffu) != (unsigned)cap) return 16;
                }
                for (int j = 0; j < cnt; j++) {
                    const size_t o = (size_t)slot[s].p0 + 8 * (size_t)(j & ~3) + lane;      // word (j / 4) 32 + lane
                    if (T.o_pos + 8 * (o + 1) > size) return 9;
                    const int e = (int)((pos[o] >> (16 * (j & 3))) & 0xffffu);
                    if (e >= cap || wrote[e] < 0 || pulled[e] || node_of[e] != node || point_of[e] <= last) return 10;
                    pulled[e] = 1;
                    last = point_of[e];
                    fx = fx - q[2 * e]; fy = fy - q[2 * e + 1];
                }
                f[2 * (n0 + node)] = fx; f[2 * (n0 + node) + 1] = fy;
            }
            for (int s = 0; s < cap; s++) if (wrote[s] >= 0 && !pulled[s]) return 11;
            // no read wavefront meets a place twice (writes: checked by `wrote` above)
            for (int s0 = 0; s0 < T.nslot; s0 += P)
                for (int j = 0; j < maxcnt; j++) {
                    unsigned seen = 0;
                    for (int s = s0; s < std::min(s0 + P, T.nslot); s++) {
                        if (j >= (int)(slot[s].node >> 16)) continue;
                        const size_t o = (size_t)slot[s].p0 + 8 * (size_t)(j & ~3) + (s & 31);
                        const unsigned bit = 1u << (((pos[o] >> (16 * (j & 3))) & 0xffffu) % P);
                        if (seen & bit) return 12;
                        seen |= bit;
                    }
                }
            gp += T.ngp;
        }
        if (TS.b_tile0[b + 1] > TS.b_tile0[b] && gp != d->body_gp_ptr[b + 1]) return 13;
    }
    return 0;
}
