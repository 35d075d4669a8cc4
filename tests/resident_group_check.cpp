// CPU check of the resident kernel's group choice (res_group in
// fwi_resident_plan.cpp): the time it reports is the plain sum of the launches'
// modelled steps, and no other number of shots per launch that it may choose
// has a smaller sum, on lists of equal widths, on lists that start with wider
// windows and end in a run of equal ones, and on lists of unequal widths.
#include <cmath>
#include <cstdio>

#include "fwi_resident.h"

using namespace fwi;

using Shots = std::vector<const Layout*>;

// The sum over launches of g shots; < 0: some launch does not fit.
static double launches_us(const Shots& s, int g, const ResDevice& dev) {
    double us = 0.0;
    for (size_t i = 0; i < s.size(); i += g) {
        ResCuts c;
        if (!res_cuts(Shots(s.begin() + i, s.begin() + std::min(s.size(), i + g)), dev, c)) return -1.0;
        us += c.step_us;
    }
    return us;
}

int main() {
    const ResDevice dev{152, 228 * 1024, 227 * 1024};
    struct Run {
        int n, nx;
    };
    struct Case {
        int ny, acc, dpml;
        std::vector<Run> runs;
    };
    const Case cases[] = {
        {600, 3, 20, {{24, 850}}},
        {600, 3, 20, {{1, 851}, {23, 850}}},
        {600, 3, 20, {{5, 900}, {19, 850}}},
        {400, 3, 20, {{1, 4000}, {15, 2000}}},
        {200, 3, 20, {{1, 500}, {30, 300}}},
        {200, 4, 20, {{7, 500}, {30, 300}}},
        {163, 4, 8, {{1, 700}, {1, 600}, {13, 384}}},
        {163, 3, 20, {{4, 384}, {1, 383}, {1, 380}, {1, 90}}},
        {200, 3, 20, {{12, 400}, {1, 60}}},
        {40, 3, 8, {{1, 90}}},
    };
    for (const Case& c : cases) {
        std::vector<Layout> lays;
        for (const Run& r : c.runs)
            for (int i = 0; i < r.n; ++i) lays.push_back(make_layout(c.ny, r.nx, c.acc, c.dpml));
        Shots s;
        for (const Layout& l : lays) s.push_back(&l);
        const int n = (int)s.size();
        double us = 0.0;
        const int g = res_group(s, dev, n, &us);
        if (g < 1 || g > n) {
            fprintf(stderr, "%d shots of %d rows: group %d\n", n, c.ny, g);
            return 1;
        }
        const double sum = launches_us(s, g, dev);
        if (!(std::fabs(us - sum) <= 1e-9 * sum)) {
            fprintf(stderr, "%d shots of %d rows, %d a launch: %.6f us, the launches' sum is %.6f\n", n, c.ny, g, us, sum);
            return 2;
        }
        for (int k = 1; k <= n; ++k) {
            const int nl = (n + k - 1) / k;
            if ((n + nl - 1) / nl != k) continue;  // shots are dealt out evenly
            const double t = launches_us(s, k, dev);
            if (t < 0) break;  // larger groups do not fit either
            if (t < sum * (1 - 1e-9)) {
                fprintf(stderr, "%d shots of %d rows: %d a launch %.3f us, %d a launch %.3f us\n", n, c.ny, g, sum, k, t);
                return 3;
            }
        }
    }
    printf("groups ok\n");
    return 0;
}
