"""The streaming kernels where the resident kernel is the default: captured waves
replayed (two streams forked and joined inside the graph, the wait for the
observed data's upload), in every form that a survey can ask for, and the
drop-in solver's streaming branch with two-step tiles."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_solver import gpu_solver, random_case
from test_gpu_survey import make

pytestmark = pytest.mark.gpu

FORMS = {"resident": dict(), "f16": dict(snap_form=2), "bf16": dict(snap_form=1), "tiles": dict(tile_kernel=2, tile_rows=32),
         "queues": dict(tile_kernel=1, tile_rows=48, tile_edge_rows=8), "single": dict(two_step=False),
         "fused": dict(fused_step=True), "recompute": dict(recompute=True), "f16-recompute": dict(snap_form=2, recompute=True)}


@pytest.mark.parametrize("form", FORMS)
def test_graph_replays_bit_identical_to_direct_launches(form):
    """Four gradient runs and four forward runs: direct, captured and replayed,
    then whichever form the timings keep."""
    import fwi_gb300 as F
    from fwi_gb300.synth import lam_from_vp
    spec, vp = make(14, ny=70, nxm=330, nshots=3, nt=160, store_snap=4, dpml=20)
    sv = F.Survey(spec, **FORMS[form])
    assert (sv.resident() > 0) == (form == "resident")
    sv.set_lambda(lam_from_vp(vp))
    for step in (1, 2):
        outs = []
        for k in range(4):
            g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
            m, _ = sv.run(step, g if step == 1 else None)
            outs.append((m, g, [sv.synthetic(i) for i in range(len(spec.shots))]))
            name, t_direct, t_graph = sv.launch_form(step)
            assert t_direct > 0 and (t_graph > 0) == (k > 0)
            assert name == "undecided" if k == 0 else name in ("graph", "direct")
        for m, g, s in outs[1:]:
            assert m == outs[0][0] and np.array_equal(g, outs[0][1])
            assert all(np.array_equal(a, b) for a, b in zip(s, outs[0][2]))
    sv.close()


@pytest.mark.parametrize("snap", [0, 2])
def test_batch_graph_replays_follow_new_observations(snap):
    """The batch call with FWI_SURVEY_GRAPH: every call replays a captured wave
    that waits inside for this call's traces, resident (FP32 snapshots) and
    streaming (FP16)."""
    import fwi_gb300 as F
    from fwi_gb300.synth import lam_from_vp
    spec, vp = make(15, ny=50, nxm=260, nshots=4, dpml=20)
    lam = lam_from_vp(vp)
    F.batch_release()
    seen = set()
    for r in range(3):
        for sh in spec.shots:
            sh.obs = np.asfortranarray(sh.obs + np.float32(0.3 * r) * np.roll(sh.obs, 5 + r, axis=0))
        g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
        m = F.calculate_misfit_gradient(spec, lam, 1, np.float32(0.0), g, snap_form=snap, flags=F.SURVEY_GRAPH)
        b = F.batch_survey()
        assert (b.resident() > 0) == (snap == 0) and b.launch_form(1)[0] == "graph"
        sv = F.Survey(spec, snap_form=snap, graph=False)
        sv.set_lambda(lam)
        g2 = np.zeros_like(g)
        m2, _ = sv.run(1, g2)
        sv.close()
        assert m == np.float32(m2) and np.array_equal(g, g2)
        seen.add(float(m))
    assert len(seen) == 3
    F.batch_release()


@pytest.mark.parametrize("acc", [3, 4])
def test_dropin_streams_a_grid_that_exceeds_the_shared_memory(acc):
    """1100 x 4000 cells hold more state than the shared memory of the GPU: the
    drop-in solver launches every step, in two-step tiles."""
    import fwi_gb300 as F
    ny, nx, nt, store = 1100, 4000, 20, 5
    z = random_case(70 + acc, ny, nx, nt, acc, 20, store, 3, 24)
    z["nySou"] = np.array([3, 500, ny - 2], np.int32)
    z["nxSou"] = np.array([nx // 2, 5, nx - 3], np.int32)
    z["nxRec"][:6] = z["nxSou"].repeat(2) + 2  # near enough for the two wavefields to meet in 20 steps
    z["nyRec"][:6] = z["nySou"].repeat(2) - 1
    nts = z["nt_store"]
    Fg = np.zeros((ny, nx * (nts + 1)), np.float32, order="F")
    Fo = np.zeros_like(Fg)
    Kg = np.zeros((ny, nx), np.float32, order="F")
    Ko = Kg.copy(order="F")
    l0 = F.kernel_launch_count()
    rec_g = gpu_solver(z, 1, Kg, Fg)
    assert F.kernel_launch_count() - l0 > nt
    args = (z["nxSou"], z["nySou"], z["nxRec"], z["nyRec"], z["S"], z["Sadj"], z["d"], z["dt"], z["ctmp"], store, nts, nt)
    rec_o = O.solver_acoustic_ss(1, *args, Ko, Fo, acc=acc, dpml=20)
    np.testing.assert_array_equal(rec_g, rec_o)
    np.testing.assert_array_equal(Fg, Fo)
    gpu_solver(z, 2, Kg, Fg)
    O.solver_acoustic_ss(2, *args, Ko, Fo, acc=acc, dpml=20)
    np.testing.assert_array_equal(Kg, Ko)
    assert np.abs(Ko).max() > 0
