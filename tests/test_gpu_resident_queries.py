"""The tuning queries of a resident survey (tiles, edge_tiles, stepping, tuning):
they answer where the streaming kernels' fields do not fit the survey's budget,
and leave the survey as it was."""
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
