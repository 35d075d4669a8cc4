// Test-only: the resident kernel's bounded wait, through the library's own
// survey calls (the host code is compiled into this program so that the tiles
// on the device can be changed; the kernel is built with a limit of
// milliseconds).  One tile is told that it has no edge words: it sends none,
// its neighbours' waits for them run out, and so do the waits for those
// neighbours.  The launches must end by themselves, the calls must report
// FWI_ERR_CUDA, and with the tile restored the survey must give the bits it
// gave before.
#include "../fwi_gb300/csrc/fwi_host.cu"

#define EXPECT(c)                                                                    \
    do {                                                                             \
        if (!(c)) {                                                                  \
            fprintf(stderr, "line %d: %s (%s)\n", __LINE__, #c, fwi_last_error());   \
            return 1;                                                                \
        }                                                                            \
    } while (0)

int main() {
    const int ny = 60, nx = 120, nt = 80, nrec = 30;
    std::vector<float> lambda((size_t)ny * nx, 4.0e9f), src(nt, 0.f), obs((size_t)nt * nrec);
    for (int i = 0; i < nt; ++i) src[i] = std::sin(0.3f * i);
    for (size_t i = 0; i < obs.size(); ++i) obs[i] = std::cos(0.1f * i);
    std::vector<int> xs{50}, ys{3}, xr, yr(nrec, 2);
    for (int i = 0; i < nrec; ++i) xr.push_back(1 + 4 * i);
    fwi_shot shot{0, nx, 1, nrec, xs.data(), ys.data(), xr.data(), yr.data(), src.data(), obs.data(), 1.0, 1.0};
    fwi_survey_desc d{};
    d.ny = ny;
    d.nx_model = nx;
    d.d = 10.f;
    d.dt = 1e-3f;
    d.nt = nt;
    d.store_snap = 10;
    d.acc = 3;
    d.dpml = 20;
    d.numtasks = 1;
    d.grad_form = FWI_GRAD_F64;
    d.nshots = 1;
    d.shots = &shot;
    d.flags = FWI_SURVEY_GRAPH;  // the runs replay graphs; time_steps launches directly
    fwi_survey* s = nullptr;
    EXPECT(fwi_survey_create(&d, &s) == FWI_OK);
    int resident = 0;
    EXPECT(fwi_survey_resident(s, &resident) == FWI_OK && resident == 1);
    EXPECT(fwi_survey_set_lambda(s, lambda.data()) == FWI_OK);
    double m0 = 0.0, m1 = 0.0;
    std::vector<float> g0((size_t)ny * nx, 0.f), g1(g0), none(g0);
    EXPECT(fwi_survey_run(s, 1, &m0, g0.data()) == FWI_OK);
    EXPECT(fwi_survey_time_steps(s, 2 * nt) == FWI_OK);

    ResDev& r = *s->res[0];
    std::vector<ResTile> tiles = r.plan.tiles;
    const int silent = (int)tiles.size() / 2;
    EXPECT(tiles.size() > 2 && tiles[silent].npair > 0);
    tiles[silent].npair = 0;
    EXPECT(upload(r.tiles, tiles, stream()) == FWI_OK);
    double m = 0.0;
    EXPECT(fwi_survey_run(s, 1, &m, none.data()) == FWI_ERR_CUDA);
    EXPECT(std::strstr(fwi_last_error(), "neighbouring tile"));
    EXPECT(fwi_survey_run(s, 2, &m, nullptr) == FWI_ERR_CUDA);
    EXPECT(fwi_survey_time_steps(s, 10) == FWI_ERR_CUDA);
    EXPECT(m == 0.0 && cudaDeviceSynchronize() == cudaSuccess);

    EXPECT(upload(r.tiles, r.plan.tiles, stream()) == FWI_OK);
    EXPECT(fwi_survey_time_steps(s, 10) == FWI_OK);  // the word of the calls before is gone
    EXPECT(fwi_survey_run(s, 1, &m1, g1.data()) == FWI_OK);
    EXPECT(m0 == m1 && std::memcmp(g0.data(), g1.data(), g0.size() * sizeof(float)) == 0);
    EXPECT(fwi_survey_destroy(s) == FWI_OK && fwi_finalize() == FWI_OK);
    printf("wait ok\n");
    return 0;
}
