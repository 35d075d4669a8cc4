// CPU check of the launches of a survey (res_survey in fwi_resident_plan.cpp)
// whose sources and receivers fill the tiles' shared memory: a receiver in
// every row of a column (each row is a source line of the adjoint), dense
// receivers on a few rows, receivers all over the grid.  Where the chosen
// number of shots per launch leaves no room for them, c2 goes to global memory
// or fewer shots share a launch; the launches found pass every check of
// resident_check.cpp, and the survey stays within the time it was given.
#define main resident_check_main
#include "resident_check.cpp"
#undef main

struct ListCase {
    const char* name;
    int n, ny, nx, nrec, dpml, acc;
    int kind;          // 0 a receiver in every row of a column, 1 evenly on row 2, 2 all over the grid, 3 all in one cell
    bool resident;
};

int main() {
    const ResDevice dev{152, 228 * 1024, 227 * 1024};
    const ListCase cases[] = {
        {"column", 12, 163, 384, 163, 20, 3, 0, true},
        {"column", 3, 400, 2000, 400, 20, 3, 0, true},
        {"column", 24, 600, 850, 600, 20, 3, 0, true},
        {"column", 1, 200, 400, 200, 20, 4, 0, true},
        {"row", 35, 96, 883, 233, 20, 3, 1, true},
        {"row", 27, 95, 4876, 300, 20, 3, 1, true},
        {"all over", 4, 120, 200, 3000, 8, 3, 2, true},
        {"all over", 1, 40, 90, 200000, 8, 3, 2, true},
        {"one cell", 1, 40, 90, 200000, 8, 3, 3, false},  // 1.6 MB of receivers in one tile
    };
    for (const ListCase& c : cases) {
        std::vector<ShotGeom> geo(c.n);
        std::vector<Layout> lay;
        for (int s = 0; s < c.n; ++s) {
            ShotGeom& g = geo[s];
            g.nx = c.nx;
            g.nxS = {c.nx / 3 + s};
            g.nyS = {2};
            for (int i = 0; i < c.nrec; ++i) {
                g.nxR.push_back(c.kind == 1 ? 1 + i * (c.nx - 1) / c.nrec : c.kind == 2 ? 1 + i * 37 % c.nx : c.nx / 2);
                g.nyR.push_back(c.kind == 0 ? 1 + i : c.kind == 2 ? 1 + i * 11 % c.ny : 2);
            }
            lay.push_back(make_layout(c.ny, c.nx, c.acc, c.dpml));
        }
        std::vector<const ShotGeom*> gp;
        std::vector<const Layout*> lp;
        for (int s = 0; s < c.n; ++s) {
            gp.push_back(&geo[s]);
            lp.push_back(&lay[s]);
        }
        double us = 0.0;
        const int want = res_group(lp, dev, c.n, &us);
        ResSurvey r;
        const bool ok = res_survey(gp, lp, dev, c.n, 2.5 * us, r);
        printf("%s, %d x %dx%d: %d a launch chosen, %d found, c2 %s\n", c.name, c.n, c.ny, c.nx, want, ok ? r.shots : 0,
               ok && r.launches[0].c2_shared ? "shared" : "global");
        if (ok != c.resident) return 10;
        ResSurvey tight;
        if (res_survey(gp, lp, dev, c.n, 0.99 * us, tight)) return 11;  // nothing is as fast as that
        if (!ok) continue;
        if (r.shots < 1 || r.shots > want || r.us > 2.5 * us) return 12;
        size_t at = 0;
        for (const ResPlan& p : r.launches) {
            const size_t e = std::min(at + r.shots, (size_t)c.n);
            if (check(p, {geo.begin() + at, geo.begin() + e}, {lay.begin() + at, lay.begin() + e}, dev)) return 13;
            at = e;
        }
        if (at != (size_t)c.n) return 14;
    }
    printf("lists ok\n");
    return 0;
}
