// CPU checks of the resident kernel's plan (fwi_resident_plan.cpp) over many
// grids: the tiles partition every shot's grid, every cell has exactly one
// thread, every shared-memory and outbox index a thread forms lies inside its
// array, neighbours agree on what they exchange, sources and receivers are
// all present once.  Restates the kernel's index arithmetic.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>

#include "fwi_resident.h"

using namespace fwi;

#define CHECK(c)                                                                              \
    do {                                                                                      \
        if (!(c)) {                                                                           \
            fprintf(stderr, "line %d: %s (ny %d nx %d acc %d dn %d)\n", __LINE__, #c, l.ny, l.nx, l.acc, l.dn); \
            return 1;                                                                         \
        }                                                                                     \
    } while (0)

static int check(const ResPlan& p, const std::vector<ShotGeom>& geo, const std::vector<Layout>& lay,
                 const ResDevice& dev) {
    std::vector<std::vector<int>> owner(geo.size());
    for (size_t s = 0; s < geo.size(); ++s) owner[s].assign((size_t)(lay[s].ny + lay[s].dn) * lay[s].nxt, 0);
    std::vector<char> out(p.out_elems, 0), c2(p.c2_elems, 0);
    std::vector<std::multiset<int>> recs(geo.size()), srcs[2];
    srcs[0].resize(geo.size());
    srcs[1].resize(geo.size());
    for (size_t ti = 0; ti < p.tiles.size(); ++ti) {
        const ResTile& t = p.tiles[ti];
        const Layout& l = lay[t.shot];
        const int R = l.acc, dn = l.dn, H = t.y1 - t.y0, W = t.x1 - t.x0, nyr = l.ny + dn;
        CHECK(t.x0 >= 0 && t.x0 % 4 == 0 && t.x1 <= l.nxt && W > 0 && t.y0 >= 0 && t.y1 <= nyr && H > 0);
        CHECK(t.cp >= W && t.cp % 4 == 0 && t.pitch >= t.cp + 8 && t.pitch % 8 == 4);
        CHECK(t.x1 == l.nxt || t.x1 % 4 == 0);
        // shared memory: arrays in order, inside the block's
        const int sz = (H + 2 * R) * t.pitch;
        const int lines = std::max(t.lines[0], t.lines[1]);
        const int at[] = {t.o_p[0], t.o_p[1], t.o_xl, t.o_xr, t.o_y, t.o_cl, t.o_cr, t.o_cb, t.o_c2 >= 0 ? t.o_c2 : t.o_line, t.o_line, t.o_row, t.o_fac,
                          t.o_pair, t.o_rec, t.o_src, t.floats};
        CHECK((t.o_c2 >= 0) == p.c2_shared);
        const int len[] = {sz, sz, t.nl ? 3 * H * dn : 0, t.nr ? 3 * H * dn : 0, t.y1 > l.ny ? 3 * dn * t.cp : 0, H * t.nl,
                           H * t.nr, t.y1 > l.ny ? dn * t.cp : 0, p.c2_shared ? H * t.cp : 0, 2 * lines * t.cp, H, 2 * dn, t.npair,
                           2 * (t.rec1 - t.rec0), 2 * std::max(t.src1[0] - t.src0[0], t.src1[1] - t.src0[1])};
        for (int i = 0; i < 15; ++i) CHECK(at[i] % 4 == 0 && at[i] + len[i] <= at[i + 1]);
        CHECK((size_t)t.floats * 4 <= p.smem && p.smem + RES_STATIC_SMEM <= dev.smem_block);
        CHECK(p.smem + RES_STATIC_SMEM + 1024 <= dev.smem_sm);
        // neighbours: the same edge, and the exchanged rows/columns exist
        for (int k = 0; k < 4; ++k) {
            if (t.nbr[k] < 0) {
                CHECK(k == 0 ? t.x0 == 0 : k == 1 ? t.x1 == l.nxt : k == 2 ? t.y0 == 0 : t.y1 == nyr);
                continue;
            }
            const ResTile& n = p.tiles[t.nbr[k]];
            CHECK(n.nbr[k ^ 1] == (int)ti && n.shot == t.shot);
            if (k < 2) CHECK(n.y0 == t.y0 && n.y1 == t.y1 && (k == 0 ? n.x1 == t.x0 : n.x0 == t.x1) && W >= 4);
            else CHECK(n.x0 == t.x0 && n.x1 == t.x1 && n.cp == t.cp && (k == 2 ? n.y1 == t.y0 : n.y0 == t.y1) && H >= R);
            const int pairs = k < 2 ? 2 * H : R * ((W + 1) / 2);
            CHECK((k < 3 ? t.pair0[k + 1] : t.npair) - t.pair0[k] == pairs);
            CHECK((k < 2 ? n.pair0[(k ^ 1) + 1] : k == 2 ? n.npair : n.pair0[3]) - n.pair0[k ^ 1] == pairs);
        }
        CHECK(t.out % 2 == 0);
        for (int i = 0; i < 4 * t.npair; ++i) {
            CHECK((size_t)(t.out + i) < out.size() && !out[t.out + i]);
            out[t.out + i] = 1;
        }
        for (int i = 0; i < H * t.cp; ++i) {
            CHECK((size_t)t.c2 + i < c2.size() && !c2[t.c2 + i]);
            c2[t.c2 + i] = 1;
        }
        // a tile with CPML columns or bottom rows holds all of that strip
        if (t.nl) CHECK(t.x0 == 0 && t.nl >= dn && t.nl <= W);
        if (t.nr) CHECK(t.x1 == l.nxt && t.nr >= dn && t.x1 - t.nr <= dn + l.nx && t.nr <= W);
        if (t.y1 > l.ny) CHECK(t.y1 == nyr && t.y0 <= l.ny && (t.y0 == 0 || t.y0 >= R));
        int warp = 0;
        for (int g = 0; g < t.ngroups[0] + t.ngroups[1]; ++g) {
            const ResGroup& G = t.g[g];
            const bool second = g >= t.ngroups[0];
            if (g == t.ngroups[0]) {
                CHECK(warp * 32 <= RES_THREADS);
                warp = 0;
            }
            CHECK(G.warp0 == warp && G.h >= 1 && G.h <= 32 && G.n > 0 && G.np >= G.n && G.kind >= 0 && G.kind < 4);
            warp += G.nwarps;
            for (int i = 0; i < 32 * G.nwarps; ++i) {
                const int b = i / G.np, c = i % G.np, x = G.x0 + (G.kind < 2 ? 4 * c : c);
                if (c >= G.n) continue;
                const int ya = std::min(G.y0 + b * G.h, G.y1), yb = std::min(ya + G.h, G.y1);
                for (int y = ya; y < yb; ++y) {
                    CHECK(y >= t.y0 && y < t.y1 && (G.kind & 1) == (y >= l.ny));
                    const int n = G.kind < 2 ? 4 : 1;
                    for (int e = 0; e < n; ++e) {
                        CHECK(x + e >= t.x0 && x + e < t.x1);
                        ++owner[t.shot][(size_t)y * l.nxt + x + e];
                        // the cells a neighbour reads are computed in the first phase
                        const bool read = (t.nbr[0] >= 0 && x + e < t.x0 + 4) || (t.nbr[1] >= 0 && x + e >= t.x1 - 4) ||
                                          (t.nbr[2] >= 0 && y < t.y0 + R) || (t.nbr[3] >= 0 && y >= t.y1 - R);
                        CHECK(read != second);
                        const bool xc = x + e < dn || x + e >= dn + l.nx;
                        if (G.kind < 2) CHECK(!xc);
                        // p columns the x-stencil reads, p rows the y-stencil reads
                        int cx = x + e, cy = y;
                        if (G.kind >= 2) cx = std::min(std::max(cx, R), l.nxt - 1 - R);
                        if (G.kind & 1) cy = std::min(y, nyr - 1 - R);
                        const int lo = cx - R - t.x0 + 4, hi = cx + R - t.x0 + 4;
                        CHECK(lo >= 0 && hi < t.pitch && (cx - R >= 0 && cx + R < l.nxt));
                        CHECK(cx - R >= t.x0 - 4 && cx + R < t.x1 + 4);
                        CHECK(cx - R >= t.x0 || t.nbr[0] >= 0);
                        CHECK(cx + R < t.x1 || t.nbr[1] >= 0);
                        CHECK(cy - R >= t.y0 - R && cy + R < t.y1 + R && cy + R < nyr);
                        CHECK(cy + R < t.y1 || t.nbr[3] >= 0);
                        if (G.kind >= 2) {
                            const bool left = x - t.x0 < t.nl;
                            CHECK(left || x - (t.x1 - t.nr) >= 0);
                            if (xc) CHECK(left == (x < dn) && dn > 2 * R);
                        }
                    }
                    if (G.kind == 0) CHECK(x - 4 >= t.x0 - 4 && x + 8 <= t.x1 + 4 && x + 8 <= t.x0 + t.cp + 4);
                }
            }
        }
        CHECK(warp * 32 <= RES_THREADS);
        for (int m = 0; m < 2; ++m) {
            for (int i = t.src0[m]; i < t.src1[m]; ++i) {
                const ResSrc e = p.src[i];
                CHECK(e.pos >= 0 && e.pos < t.lines[m] * t.cp);
                int row = -1;
                for (int y = 0; y < H; ++y)
                    if (p.rows[t.rows[m] + y] == e.pos / t.cp) row = t.y0 + y;
                CHECK(row >= 0 && row < l.ny);
                const std::vector<int>&xs = m ? geo[t.shot].nxR : geo[t.shot].nxS, &ys = m ? geo[t.shot].nyR : geo[t.shot].nyS;
                CHECK(ys[e.vidx] - 1 == row && dn + xs[e.vidx] - 1 == t.x0 + e.pos % t.cp);
                srcs[m][t.shot].insert(e.vidx);
            }
        }
        for (int i = t.rec0; i < t.rec1; ++i) {
            const ResRec r = p.rec[i];
            const int y = r.off / t.pitch - R + t.y0, x = r.off % t.pitch - 4 + t.x0;
            CHECK(y >= t.y0 && y < t.y1 && x >= t.x0 && x < t.x1);
            CHECK(geo[t.shot].nyR[r.ridx] - 1 == y && dn + geo[t.shot].nxR[r.ridx] - 1 == x);
            recs[t.shot].insert(r.ridx);
        }
    }
    for (size_t s = 0; s < geo.size(); ++s) {
        const Layout& l = lay[s];
        for (int v : owner[s]) CHECK(v == 1);
        size_t want = 0;
        for (int y : geo[s].nyR) want += y >= 1;
        CHECK(recs[s].size() == want);
        CHECK(srcs[0][s].size() == injection_cells(geo[s].nxS, geo[s].nyS, l).size());
        CHECK(srcs[1][s].size() == injection_cells(geo[s].nxR, geo[s].nyR, l).size());
    }
    return 0;
}

int main() {
    const ResDevice dev{152, 228 * 1024, 227 * 1024};
    unsigned seed = 12345;
    auto rnd = [&](int a, int b) {  // [a, b]
        seed = seed * 1664525u + 1013904223u;
        return a + (int)((seed >> 8) % (unsigned)(b - a + 1));
    };
    int plans = 0, refused = 0;
    for (int n = 0; n < 240; ++n) {
        const int acc = rnd(3, 4), dpml = n % 5 == 0 ? rnd(1, 54) : 20, shots = n % 3 ? 1 : rnd(1, 14);
        const int ny = n % 7 == 0 ? rnd(1, 30) : rnd(20, 600), wide = n % 4 ? rnd(8, 700) : rnd(8, 4000);
        std::vector<ShotGeom> geo;
        std::vector<Layout> lay;
        const int dn = dpml + 2 * acc;
        for (int s = 0; s < shots; ++s) {
            ShotGeom g;
            g.nx = std::max(8, wide - rnd(0, wide / 2));
            for (int i = 0; i < 2; ++i) {
                g.nxS.push_back(rnd(1 - dn, g.nx + dn));
                g.nyS.push_back(rnd(1, ny + dn));
            }
            const int row = rnd(1, ny);
            for (int i = 0; i < 30; ++i) {
                g.nxR.push_back(rnd(1 - dn, g.nx + dn));
                g.nyR.push_back(i < 20 ? row : rnd(1 - dn, ny + dn));
            }
            geo.push_back(g);
            lay.push_back(make_layout(ny, g.nx, acc, dpml));
        }
        std::vector<const ShotGeom*> gp;
        std::vector<const Layout*> lp;
        for (int s = 0; s < shots; ++s) {
            gp.push_back(&geo[s]);
            lp.push_back(&lay[s]);
        }
        const int g = res_group(lp, dev, shots);
        if (g < 0 || g > shots) return 2;
        if (g == 0) {
            ++refused;
            continue;
        }
        for (int i = 0; i < shots; i += g) {
            const int e = std::min(shots, i + g);
            ResPlan p;
            ResCuts cuts;
            if (!res_cuts({lp.begin() + i, lp.begin() + e}, dev, cuts) ||
                !res_plan({gp.begin() + i, gp.begin() + e}, {lp.begin() + i, lp.begin() + e}, cuts, dev, p)) {
                ++refused;
                continue;
            }
            ++plans;
            if ((int)p.tiles.size() > dev.sms) return 3;
            if (check(p, {geo.begin() + i, geo.begin() + e}, {lay.begin() + i, lay.begin() + e}, dev)) return 1;
        }
    }
    printf("%d plans ok, %d refused\n", plans, refused);
    return plans > 180 && refused < 40 ? 0 : 4;
}
