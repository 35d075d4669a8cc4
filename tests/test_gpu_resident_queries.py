"""The tuning queries of a resident survey (tiles, edge_tiles, stepping, tuning):
they answer where the streaming kernels' fields do not fit the survey's budget,
leave the survey as it was, and keep their timings on another time axis, also
where the survey leaves the resident kernel and comes back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def queries(sv):
    return sv.tiles(), sv.edge_tiles(), sv.stepping(), sv.tuning()


def test_queries_within_a_budget_too_small_for_the_streaming_plan():
    import fwi_gb300 as F
    from fwi_gb300 import synth
    spec, vp = synth.small_survey(seed=51, ny=60, nxm=300, nshots=1, dpml=20, nt=20)
    rng = np.random.default_rng(6)
    for sh in spec.shots:
        sh.obs = np.asfortranarray(rng.standard_normal((spec.nt, len(sh.nxRec))).astype(np.float32))
    data = 4 * spec.nt * sum(3 * len(s.nxRec) + len(s.nxSou) for s in spec.shots) + 12 * spec.ny * spec.nx_model
    # a shot's three snapshot blocks and FP64 image: 20 bytes a cell of the 60 x 352..512 grid; its
    # streaming state: ten fields more, of 112 rows
    sv = F.Survey(spec, hbm_budget=data + 15000 * spec.ny)
    assert sv.resident() == 1
    sv.set_lambda(synth.lam_from_vp(vp))
    g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
    m, _ = sv.run(1, g)
    (kernel, rows, times), (edge, edge_times), (form, ms), (wave, band) = queries(sv)
    assert form == "two-step" and kernel in (1, 2) and rows > 0 and wave == 1 and band > 0 and edge >= 0
    assert times == {} and edge_times == {} and ms == {}  # nothing timed
    assert sv.resident() == 1
    g2 = np.zeros_like(g)
    assert sv.run(1, g2)[0] == m and np.array_equal(g2, g)
    sv.close()


def test_timings_outlive_a_new_time_axis(monkeypatch):
    monkeypatch.setenv("FWI_TUNE_CACHE", "")  # no cross-process cache file
    import fwi_gb300 as F
    from fwi_gb300 import synth
    spec, vp = synth.small_survey(seed=52, ny=61, nxm=307, nshots=2, dpml=20, nt=60)
    lam = synth.lam_from_vp(vp)
    rng = np.random.default_rng(7)
    nrec = sum(len(s.nxRec) for s in spec.shots)
    nsou = sum(len(s.nxSou) for s in spec.shots)

    def axis(nt):
        return (1e-3, nt, rng.standard_normal(nt * nsou).astype(np.float32), rng.standard_normal(nt * nrec).astype(np.float32))

    # the budget holds the streaming state of both shots at 800 steps, their resident images (12 bytes a cell and
    # 4 a snapshot) up to some 2000 steps, and the streaming state with checkpoints above that
    cells = spec.ny * 512
    data = 4 * 6000 * (3 * nrec + nsou) + 12 * spec.ny * spec.nx_model
    sv = F.Survey(spec, hbm_budget=data + 2 * cells * (12 + 4 * 200))
    assert sv.resident() == 2
    first = queries(sv)
    assert first[0][2] and first[2][1]  # timed on the first query
    sv.set_time(*axis(80))
    assert sv.resident() == 2 and queries(sv) == first
    long = axis(6000)
    sv.set_time(*long)
    assert sv.resident() == 0 and sv.recompute_plan()[1] > 1
    away = queries(sv)
    assert away[0][2] == first[0][2] and away[2] == first[2]
    sv.set_lambda(lam)
    g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
    m, _ = sv.run(1, g)
    short = axis(80)
    sv.set_time(*short)
    assert sv.resident() == 2 and queries(sv) == first
    assert sv.recompute_plan() == (0, 0)
    ms, _ = sv.run(2)
    sv.close()
    # either axis from a survey that streams from the start
    for (dt, nt, src, obs), want in ((long, m), (short, ms)):
        ref = F.Survey(spec, two_step=False)
        ref.set_time(dt, nt, src, obs)
        ref.set_lambda(lam)
        g2 = np.zeros_like(g)
        m2, _ = ref.run(1, g2)
        assert m2 == want
        if nt == 6000:
            np.testing.assert_array_equal(g2, g)
        ref.close()
