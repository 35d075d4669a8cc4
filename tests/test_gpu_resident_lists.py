"""Resident launches whose tiles hold many sources and receivers -- a vertical
receiver array, whose every row is a source line of the adjoint -- so that c2
moves to global memory or fewer shots share a launch, against the streaming
kernels' single steps, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx,nshots,shots", [(163, 384, 12, 12), (400, 2000, 3, 1), (600, 850, 8, 2)])
def test_vertical_arrays_run_resident(ny, nx, nshots, shots):
    import fwi_gb300 as F
    from fwi_gb300 import synth
    spec, vp = synth.small_survey(seed=41, ny=ny, nxm=nx, nshots=nshots, dpml=20, nt=48, nrec=4)
    rng = np.random.default_rng(5)
    for sh in spec.shots:
        sh.nxRec = np.full(ny, np.clip(sh.nxSou[0] + 6, 1, nx), np.int32)
        sh.nyRec = np.arange(1, ny + 1, dtype=np.int32)
        sh.obs = np.asfortranarray(rng.standard_normal((spec.nt, ny)).astype(np.float32))
    lam = synth.lam_from_vp(vp)
    out = []
    for form in (dict(), dict(two_step=False)):
        sv = F.Survey(spec, **form)
        assert sv.resident() == (0 if form else shots)
        sv.set_lambda(lam)
        g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
        m, _ = sv.run(1, g)
        out.append((m, g, [sv.synthetic(i) for i in range(nshots)]))
        sv.close()
    assert out[0][0] == out[1][0] and np.abs(out[0][1]).max() > 0
    for a, b in zip(out[0][2], out[1][2]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(out[0][1], out[1][1])
