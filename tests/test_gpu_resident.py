"""The resident kernel (a shot's state in shared memory for the whole time loop)
against the streaming kernels' single steps, bit for bit, at the sizes where
its tiles can go wrong: grids of one tile, of fewer rows or columns than a
block's threads, odd widths, CPML pads of one to 56 columns, strips that meet,
several shots of unequal windows in one launch and over several launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(ny=1, nxm=8, dpml=1, nt=40), dict(ny=3, nxm=9, acc=4, dpml=8, nt=60), dict(ny=12, nxm=33, dpml=20),
    dict(ny=40, nxm=91, acc=4, dpml=20, store_snap=7), dict(ny=61, nxm=333, dpml=20, store_snap=1, nt=60),
    dict(ny=30, nxm=202, dpml=50), dict(ny=163, nxm=385, acc=4, dpml=20, nshots=12, nt=90),
    dict(ny=200, nxm=1201, nshots=2, nt=60, windows=[(0, 1201), (300, 150)]),
    dict(ny=420, nxm=1999, nshots=5, nt=40, dpml=20)])
def test_resident_bit_identical_to_streaming(kw):
    import fwi_gb300 as F
    from fwi_gb300 import synth
    kw = dict(dict(nt=120), **kw)
    spec, vp = synth.small_survey(seed=31, **kw)
    rng = np.random.default_rng(4)
    for sh in spec.shots:
        sh.obs = np.asfortranarray(rng.standard_normal((spec.nt, len(sh.nxRec))).astype(np.float32))
    lam = synth.lam_from_vp(vp)
    out = []
    for form in (dict(), dict(two_step=False)):
        sv = F.Survey(spec, **form)
        # (a small grid with a 56-column pad is left to the streaming kernels)
        assert (sv.resident() > 0) == (not form and spec.dpml < 50)
        sv.set_lambda(lam)
        g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
        if spec.dpml == 1:  # the CPML's width (dpml-1)*d is zero: its factors, and so the wavefield, are NaN
            with pytest.raises(F.FwiError) as e:
                sv.run(1, g)
            assert e.value.code == -4
            continue
        m, _ = sv.run(1, g)
        out.append((m, g, [sv.synthetic(i) for i in range(len(spec.shots))]))
        sv.close()
    if not out:
        return
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][2], out[1][2]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(out[0][1], out[1][1])
