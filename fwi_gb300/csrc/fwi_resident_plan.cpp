// Host planner of the resident kernel (see fwi_resident.h).
#include "fwi_resident.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <map>

namespace fwi {

namespace {

// Cost of one row of a thread's work relative to interior quads (the kinds of
// ResGroup), and the modelled step in us: a fixed part (the barrier, the round
// trip of the edges that the second phase does not hide), a part per RES_THREADS
// edge pairs (a fit: the kernel's own passes are RES_COMM threads times one to
// RES_WORDS pairs), and the rows that the busiest threads march in either phase.
// Against measured forward steps, modelled / measured in us: three shots of
// 400 x 2000 5.06 / 4.97 (8th order 5.06 / 5.77), 600 x 4000 4.43 / 4.26, five
// of 600 x 812 5.79 / 5.20, five of 251 x 1013 3.70 / 3.32, twelve of 163 x 384
// 3.32 / 2.84, one of 200 x 400 2.13 / 1.73, three of 40 x 90 1.67 / 1.43; with
// deep pads (dpml 40 to 50) 19 to 38 % high.  A model with the clocks read in
// the kernel, phase by phase, chose cuts that were 7 % faster on one 200 x 400
// shot and 2-4 % slower on larger ones.
constexpr double ROW_COST[4] = {1.0, 2.6, 1.3, 2.2};
constexpr double STEP_US = 0.4, PAIR_US = 0.17, ROW_US[2] = {0.29, 0.21};

int ceil4(int v) { return (v + 3) / 4 * 4; }

// Cut units 0..n-1 with weights w into `parts` runs of about equal weight, the
// first at least `first` units, the last at least `last`, each at least `least`.
// Returns the parts+1 bounds, empty when it cannot be done.
std::vector<int> cut(const std::vector<double>& w, int parts, int first, int last, int least) {
    const int n = (int)w.size();
    if (parts == 1) return {0, n};
    if (std::max(first, least) + std::max(last, least) + (parts - 2) * least > n) return {};
    std::vector<double> acc(n + 1, 0.0);
    for (int i = 0; i < n; ++i) acc[i + 1] = acc[i] + w[i];
    std::vector<int> b(parts + 1, 0);
    b[parts] = n;
    for (int p = 1; p < parts; ++p) {
        const double want = acc[b[p - 1]] + (acc[n] - acc[b[p - 1]]) / (parts - p + 1);
        int i = (int)(std::lower_bound(acc.begin(), acc.end(), want) - acc.begin());
        if (i > 0 && want - acc[i - 1] < acc[i] - want) --i;
        i = std::max(i, b[p - 1] + (p == 1 ? std::max(first, least) : least));
        i = std::min(i, n - std::max(last, least) - (parts - 1 - p) * least);
        b[p] = i;
    }
    return b;
}

// Strip bounds: the side strips [0, sl) and [sr, nxt) are whole quads and
// hold the dn CPML columns of their side.
bool strips(const Layout& l, int& sl, int& sr) {
    sl = ceil4(l.dn);
    sr = (l.dn + l.nx) / 4 * 4;
    return l.nx >= 8 && sr >= sl && l.nxt < 65536 && l.ny + l.dn < 65536;
}

// Threads of a band of n quads or columns: padded to whole quarter warps
// (quads) or to a warp (columns) where that idles at most a seventh of them.
int band_threads(int kind, int n) {
    const int np = kind < 2 ? (n + 7) / 8 * 8 : (n + 31) / 32 * 32;
    return (np - n) * 6 <= n ? np : n;
}

struct Rect {
    int x0, x1, y0, y1;  // of a tile, or a part of one
};

// The work groups of one phase of a tile (0: the cells its neighbours read, 1:
// the rest): rows per thread such that no thread marches more than `rows`
// weighted rows; false when they need more than a block's warps.
bool groups(const Layout& l, const Rect& c, int phase, double rows, ResTile* t) {
    int sl, sr;
    strips(l, sl, sr);
    const int R = l.acc;
    const bool left = c.x0 > 0, right = c.x1 < l.nxt, up = c.y0 > 0, down = c.y1 < l.ny + l.dn;
    int used = 0;
    auto add = [&](int kind, int gx, int n, int ga, int gb) -> bool {
        if (n <= 0 || gb <= ga) return true;
        const int h = std::min(32, (int)std::floor(rows / ROW_COST[kind] + 1e-9));
        if (h < 1) return false;
        const int bands = (gb - ga + h - 1) / h;
        const int hb = (gb - ga + bands - 1) / bands;  // even bands
        const int np = band_threads(kind, n);
        const int nw = (np * ((gb - ga + hb - 1) / hb) + 31) / 32;
        if (t) {
            if (t->ngroups[0] + t->ngroups[1] >= RES_GROUPS) return false;
            ResGroup& g = t->g[t->ngroups[0] + t->ngroups[1]];
            g = ResGroup{kind, gx, n, np, ga, gb, hb, used, nw};
            ++t->ngroups[phase];
        }
        used += nw;
        return used <= RES_THREADS / 32;
    };
    // columns [xa, xb) of rows [ya, yb) by kind, the slow kinds first
    auto part = [&](int xa, int xb, int ya, int yb) -> bool {
        if (xb <= xa || yb <= ya) return true;
        const int qa = std::max(xa, sl), qb = std::min(xb, sr), ym = std::min(yb, l.ny), yc = std::max(ya, l.ny);
        const int lb = std::min(xb, sl), ra = std::max(xa, sr);
        return add(3, xa, lb - xa, yc, yb) && add(3, ra, xb - ra, yc, yb) && add(1, qa, (qb - qa) / 4, yc, yb) &&
               add(2, xa, lb - xa, ya, ym) && add(2, ra, xb - ra, ya, ym) && add(0, qa, (qb - qa) / 4, ya, ym);
    };
    const int yt = up ? std::min(c.y0 + R, c.y1) : c.y0, yd = down ? std::max(yt, c.y1 - R) : c.y1;
    const int xl = left ? c.x0 + 4 : c.x0, xr = right ? std::max(xl, c.x1 - 4) : c.x1;
    return phase == 0 ? part(c.x0, c.x1, c.y0, yt) && part(c.x0, c.x1, yd, c.y1) && part(c.x0, xl, yt, yd) &&
                                     part(xr, c.x1, yt, yd)
                               : part(xl, xr, yt, yd);
}

// The smallest weighted rows per thread for which a phase fits the block; < 0:
// none.
double min_rows(const Layout& l, const Rect& c, int phase) {
    const auto at = [](int i) { return i < 36 ? 1.0 + 0.2 * i : 8.0 + 0.5 * (i - 35); };
    int lo = 0, hi = 150;  // fewer rows per thread never need fewer warps
    if (!groups(l, c, phase, at(hi), nullptr)) return -1.0;
    while (lo < hi) {
        const int m = (lo + hi) / 2;
        if (groups(l, c, phase, at(m), nullptr)) hi = m;
        else lo = m + 1;
    }
    return at(lo);
}

// Row pitch of a pressure level: the columns, four halo columns on either side,
// and an odd number of quads, so that threads one below the other (edge
// columns) use different banks.
int row_pitch(int cp) { return 4 * ((cp / 4 + 2) | 1); }

// Shared-memory layout of a tile (floats); lines: source lines.
void layout_tile(const Layout& l, ResTile& t, int lines, bool c2_shared) {
    int sl, sr;
    strips(l, sl, sr);
    const int H = t.y1 - t.y0, R = l.acc;
    t.cp = ceil4(t.x1 - t.x0);
    t.pitch = row_pitch(t.cp);
    int o = 0;
    auto take = [&](int n) {
        const int at = o;
        o += ceil4(n);
        return at;
    };
    t.o_p[0] = take((H + 2 * R) * t.pitch);
    t.o_p[1] = take((H + 2 * R) * t.pitch);
    t.nl = std::max(0, std::min(t.x1, sl) - t.x0);
    t.nr = std::max(0, t.x1 - std::max(t.x0, sr));
    t.o_xl = take(t.nl ? 3 * H * l.dn : 0);
    t.o_xr = take(t.nr ? 3 * H * l.dn : 0);
    t.o_y = take(t.y1 > l.ny ? 3 * l.dn * t.cp : 0);
    t.o_cl = take(H * t.nl);
    t.o_cr = take(H * t.nr);
    t.o_cb = take(t.y1 > l.ny ? l.dn * t.cp : 0);
    t.o_c2 = c2_shared ? take(H * t.cp) : -1;
    t.o_line = take(2 * lines * t.cp);
    t.o_row = take(H);
    t.o_fac = take(2 * l.dn);
    const int rows = R * ((t.x1 - t.x0 + 1) / 2);
    const int side[4] = {t.x0 > 0 ? 2 * H : 0, t.x1 < l.nxt ? 2 * H : 0, t.y0 > 0 ? rows : 0,
                         t.y1 < l.ny + l.dn ? rows : 0};
    t.npair = 0;
    for (int k = 0; k < 4; ++k) {
        t.pair0[k] = t.npair;
        t.npair += side[k];
    }
    t.o_pair = take(t.npair);
    t.o_rec = take(2 * (t.rec1 - t.rec0));
    t.o_src = take(2 * std::max(t.src1[0] - t.src0[0], t.src1[1] - t.src0[1]));
    t.floats = o;
}

// Whether a pressure level's indices fit the packed edge pairs of the kernel.
bool fields_fit(const ResTile& t, int R) { return (t.y1 - t.y0 + 2 * R) * t.pitch <= 65536; }

// The cut of a shot into at most `most` tiles of at most `cap` bytes of shared
// memory with the shortest step.
bool cut_shot(const Layout& l, int most, size_t cap, bool c2_shared, ResCut& best) {
    int sl, sr;
    if (!strips(l, sl, sr)) return false;
    const int nrow = l.ny + l.dn, nq = (l.nxt + 3) / 4;
    std::vector<double> wx(nq, 1.0), wy(nrow, 1.0);
    for (int q = 0; q < nq; ++q)
        if (4 * q < sl || 4 * q >= sr) wx[q] = 4.0 * ROW_COST[2];
    for (int y = l.ny; y < nrow; ++y) wy[y] = ROW_COST[1];
    const int lastq = nq - sr / 4;
    bool found = false;
    for (int gx = 1; gx <= most && gx <= nq; ++gx) {
        const std::vector<int> bx = cut(wx, gx, sl / 4, lastq, 1);
        if (bx.empty()) break;
        // the largest numbers of rows that the blocks and the grid allow
        const int rows = std::min(most / gx, 1 + l.ny / MAXR);
        for (int gy = std::max(1, rows - 3); gy <= rows; ++gy) {
            const std::vector<int> by = cut(wy, gy, 1, l.dn, MAXR);
            if (by.empty()) break;
            ResCut c;
            bool ok = true;
            for (int i = 0; i < gx && ok; ++i) {
                // inner columns and rows repeat: the distinct ones only
                if (i > 1 && i < gx - 1 && bx[i + 1] - bx[i] == bx[i] - bx[i - 1]) continue;
                for (int j = 0; j < gy && ok; ++j) {
                    if (j > 1 && j < gy - 1 && by[j + 1] - by[j] == by[j] - by[j - 1] && by[j + 1] <= l.ny) continue;
                    ResTile t{};
                    t.x0 = 4 * bx[i];
                    t.x1 = std::min(4 * bx[i + 1], l.nxt);
                    t.y0 = by[j];
                    t.y1 = by[j + 1];
                    layout_tile(l, t, 1, c2_shared);
                    if (!fields_fit(t, l.acc)) ok = false;
                    c.smem = std::max(c.smem, (size_t)t.floats * 4);
                    if (c.smem > cap) ok = false;
                    double us = STEP_US + PAIR_US * ((t.npair + RES_THREADS - 1) / RES_THREADS);
                    // a tile marches no fewer rows than its quads over all threads: cuts that cannot win end here
                    const double least = (t.y1 - t.y0) * ((t.x1 - t.x0) / 4) / (double)RES_THREADS;
                    if (found && us + std::min(ROW_US[0], ROW_US[1]) * least >= best.us) ok = false;
                    for (int p = 0; p < 2 && ok; ++p) {
                        const double r = min_rows(l, Rect{t.x0, t.x1, t.y0, t.y1}, p);
                        if (r < 0) ok = false;
                        us += ROW_US[p] * r;
                    }
                    c.us = std::max(c.us, us);
                    if (found && c.us >= best.us) ok = false;
                }
            }
            if (!ok) continue;
            if (!found || c.us < best.us) {
                found = true;
                best = c;
                best.xs.clear();
                for (int v : bx) best.xs.push_back(std::min(4 * v, l.nxt));
                best.ys = by;
            }
        }
    }
    return found;
}

// cut_shot, its answers (a function of the grid and the device alone) kept for
// the next survey or time axis: the search takes milliseconds.  The planner's
// callers hold the library's lock.
bool cut_shot_kept(const Layout& l, int most, size_t cap, bool c2_shared, ResCut& best) {
    static std::map<std::array<long long, 7>, std::pair<bool, ResCut>> kept;
    const std::array<long long, 7> key{l.ny, l.nx, l.acc, l.dn, most, (long long)cap, c2_shared};
    auto it = kept.find(key);
    if (it == kept.end()) {
        if (kept.size() >= 4096) kept.clear();
        std::pair<bool, ResCut> v;
        v.first = cut_shot(l, most, cap, c2_shared, v.second);
        it = kept.emplace(key, std::move(v)).first;
    }
    best = it->second.second;
    return it->second.first;
}

double weight(const Layout& l) {
    int sl, sr;
    strips(l, sl, sr);
    const double cols = (sr - sl) + (sl + l.nxt - sr) * 4.0 * ROW_COST[2];
    return cols * (l.ny + ROW_COST[1] * l.dn);
}

// Largest dynamic shared memory of a block (one block per SM), beside the
// launch's static arrays.
size_t smem_cap(const ResDevice& dev) { return std::min(dev.smem_block, dev.smem_sm - 1024) - RES_STATIC_SMEM; }

// Modelled time of a step of the given shots; < 0 when they do not fit.  Tiles
// are dealt out by the shots' weights.
double model(const std::vector<const Layout*>& lays, const ResDevice& dev, bool c2_shared,
             std::vector<ResCut>* cuts) {
    if ((int)lays.size() > dev.sms) return -1.0;
    double sum = 0.0, t = 0.0;
    for (const Layout* l : lays) {
        int a, b;
        if (!strips(*l, a, b)) return -1.0;
        sum += weight(*l);
    }
    std::map<std::pair<int, int>, ResCut> seen;  // (width, tiles)
    for (const Layout* l : lays) {
        const int most = std::max(1, (int)(dev.sms * weight(*l) / sum));
        const auto key = std::make_pair(l->nx, most);
        auto it = seen.find(key);
        if (it == seen.end()) {
            ResCut c;
            if (!cut_shot_kept(*l, most, smem_cap(dev), c2_shared, c)) return -1.0;
            it = seen.emplace(key, c).first;
        }
        t = std::max(t, it->second.us);
        if (cuts) cuts->push_back(it->second);
    }
    return t;
}

// c2 in shared memory where the shots fit with it (and it may be), else in global memory.
double best_form(const std::vector<const Layout*>& lays, const ResDevice& dev, bool* c2_shared, bool may_share = true) {
    for (const bool c2 : {true, false}) {
        if (c2 && !may_share) continue;
        const double t = model(lays, dev, c2, nullptr);
        if (t < 0) continue;
        if (c2_shared) *c2_shared = c2;
        return t;
    }
    return -1.0;
}

// A launch with the given cuts; false when a tile's sources and receivers do
// not fit beside it.
bool plan_cuts(const std::vector<const ShotGeom*>& geoms, const std::vector<const Layout*>& lays, const ResCuts& cuts,
               const ResDevice& dev, ResPlan& out) {
    out = ResPlan();
    out.c2_shared = cuts.c2_shared;
    const size_t cap = smem_cap(dev);
    for (size_t s = 0; s < geoms.size(); ++s) {
        const Layout& l = *lays[s];
        const ShotGeom& g = *geoms[s];
        const ResCut& sc = cuts.shots[s];
        const int gx = (int)sc.xs.size() - 1, gy = (int)sc.ys.size() - 1, base = (int)out.tiles.size();
        const std::vector<SrcEnt> cells[2] = {injection_cells(g.nxS, g.nyS, l), injection_cells(g.nxR, g.nyR, l)};
        for (int j = 0; j < gy; ++j)
            for (int i = 0; i < gx; ++i) {
                ResTile t{};
                t.shot = (int)s;
                t.x0 = sc.xs[i];
                t.x1 = sc.xs[i + 1];
                t.y0 = sc.ys[j];
                t.y1 = sc.ys[j + 1];
                t.nbr[0] = i > 0 ? base + j * gx + i - 1 : -1;
                t.nbr[1] = i + 1 < gx ? base + j * gx + i + 1 : -1;
                t.nbr[2] = j > 0 ? base + (j - 1) * gx + i : -1;
                t.nbr[3] = j + 1 < gy ? base + (j + 1) * gx + i : -1;
                const int H = t.y1 - t.y0, cp = ceil4(t.x1 - t.x0);
                for (int m = 0; m < 2; ++m) {
                    std::vector<int> line(H, -1);
                    t.src0[m] = (int)out.src.size();
                    for (const SrcEnt& e : cells[m]) {  // sorted by row
                        const int y = e.row - l.dn, x = e.col - l.off;
                        if (y < t.y0 || y >= t.y1 || x < t.x0 || x >= t.x1) continue;
                        if (line[y - t.y0] < 0) line[y - t.y0] = t.lines[m]++;
                        out.src.push_back(ResSrc{line[y - t.y0] * cp + x - t.x0, e.vidx});
                    }
                    t.src1[m] = (int)out.src.size();
                    t.rows[m] = (int)out.rows.size();
                    out.rows.insert(out.rows.end(), line.begin(), line.end());
                }
                t.rec0 = (int)out.rec.size();
                for (size_t r = 0; r < g.nxR.size(); ++r) {
                    const int y = g.nyR[r] - 1, x = l.dn + g.nxR[r] - 1;
                    if (y < t.y0 || y >= t.y1 || x < t.x0 || x >= t.x1) continue;  // the top pad is never recorded
                    out.rec.push_back(ResRec{(y - t.y0 + l.acc) * row_pitch(cp) + x - t.x0 + 4, (int)r});
                }
                t.rec1 = (int)out.rec.size();
                layout_tile(l, t, std::max(t.lines[0], t.lines[1]), out.c2_shared);
                if ((size_t)t.floats * 4 > cap) return false;  // many source rows or receivers in one tile
                t.out = (int)out.out_elems;
                out.out_elems += 4 * (size_t)t.npair;
                t.c2 = (int)out.c2_elems;
                out.c2_elems += (size_t)H * t.cp;
                for (int p = 0; p < 2; ++p) {
                    const Rect c{t.x0, t.x1, t.y0, t.y1};
                    if (!groups(l, c, p, min_rows(l, c, p), &t)) return false;
                }
                out.smem = std::max(out.smem, (size_t)t.floats * 4);
                out.tiles.push_back(t);
            }
    }
    return (int)out.tiles.size() <= dev.sms;
}

}  // namespace

bool res_cuts(const std::vector<const Layout*>& lays, const ResDevice& dev, ResCuts& out, bool c2_shared) {
    out = ResCuts();
    if (best_form(lays, dev, &out.c2_shared, c2_shared) < 0) return false;
    out.step_us = model(lays, dev, out.c2_shared, &out.shots);
    return true;
}

bool res_plan(const std::vector<const ShotGeom*>& geoms, const std::vector<const Layout*>& lays, const ResCuts& cuts,
              const ResDevice& dev, ResPlan& out) {
    if (plan_cuts(geoms, lays, cuts, dev, out)) return true;
    ResCuts global;
    return cuts.c2_shared && res_cuts(lays, dev, global, false) && plan_cuts(geoms, lays, global, dev, out);
}

int res_group(const std::vector<const Layout*>& lays, const ResDevice& dev, int max_shots, double* us_out) {
    const int n = (int)lays.size();
    int best = 0, equal = n - 1;  // equal: first shot of the run of equal widths that ends the list
    while (equal > 0 && lays[equal - 1]->nx == lays[equal]->nx) --equal;
    double best_us = 0.0;
    for (int g = 1; g <= std::min(n, max_shots); ++g) {
        const int launches = (n + g - 1) / g, even = (n + launches - 1) / launches;
        if (even != g && g > 1) continue;  // another group size cuts the shots into as many launches
        double us = 0.0;
        for (int i = 0; i < n; i += g) {
            const std::vector<const Layout*> part(lays.begin() + i, lays.begin() + std::min(n, i + g));
            const double t = best_form(part, dev, nullptr);
            if (t < 0) {
                us = -1.0;
                break;
            }
            us += t;
            // equal widths from here on: the full launches that follow take the same time
            if (i >= equal && n - i >= 2 * g) {
                const int more = (n - i) / g - 1;
                us += more * t;
                i += more * g;
            }
        }
        if (us < 0) {
            if (g > 1) break;
            return 0;
        }
        if (!best || us < best_us) {
            best = g;
            best_us = us;
        }
    }
    if (us_out) *us_out = best_us;
    return best;
}

bool res_survey(const std::vector<const ShotGeom*>& geoms, const std::vector<const Layout*>& lays, const ResDevice& dev,
                int max_shots, double limit_us, ResSurvey& out) {
    const int n = (int)lays.size();
    for (int most = max_shots; most >= 1; most = out.shots - 1) {
        out = ResSurvey();
        out.shots = res_group(lays, dev, most, &out.us);
        if (out.shots < 1 || out.us > limit_us) return false;
        bool fits = true;
        for (int i = 0; i < n && fits; i += out.shots) {
            const int e = std::min(n, i + out.shots);
            const std::vector<const Layout*> part(lays.begin() + i, lays.begin() + e);
            ResCuts cuts;
            out.launches.emplace_back();
            fits = res_cuts(part, dev, cuts) &&
                   res_plan({geoms.begin() + i, geoms.begin() + e}, part, cuts, dev, out.launches.back());
        }
        if (fits) return true;
    }
    return false;
}

}  // namespace fwi
