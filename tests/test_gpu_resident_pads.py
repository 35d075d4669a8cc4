"""The resident kernel in thin and deep pads: surveys with pads of 8 (the
thinnest with finite factors) to 58 columns, sources and receivers in the pads
and either accumulator, against the streaming kernels' single steps, and the
drop-in solver in the deepest pad, 62 columns, against the oracle, bit for
bit."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_solver import gpu_solver, random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["f64", "f32"])
@pytest.mark.parametrize("kw", [
    dict(ny=30, nxm=61, dpml=2, nshots=2), dict(ny=17, nxm=90, dpml=3, acc=4, nshots=2),
    dict(ny=150, nxm=301, dpml=50, nshots=8), dict(ny=200, nxm=400, dpml=45, acc=4, nshots=4),
    dict(ny=203, nxm=399, dpml=40, nshots=6, store_snap=3), dict(ny=200, nxm=400, dpml=50, acc=4, nshots=8)])
def test_pads_bit_identical_to_streaming(kw, form):
    import fwi_gb300 as F
    from fwi_gb300 import synth
    spec, vp = synth.small_survey(seed=61, nt=90, **kw)
    rng = np.random.default_rng(8)
    for sh in spec.shots:
        sh.obs = np.asfortranarray(rng.standard_normal((spec.nt, len(sh.nxRec))).astype(np.float32))
    lam = synth.lam_from_vp(vp)
    out = []
    for how in (dict(), dict(two_step=False)):
        sv = F.Survey(spec, grad_form=F.GRAD_F64 if form == "f64" else F.GRAD_F32, **how)
        assert (sv.resident() > 0) == (not how)
        sv.set_lambda(lam)
        g = np.zeros((spec.ny, spec.nx_model), np.float32, order="F")
        m, _ = sv.run(1, g)
        out.append((m, g, [sv.synthetic(i) for i in range(len(spec.shots))]))
        sv.close()
    assert out[0][0] == out[1][0] and np.isfinite(out[0][0]) and np.abs(out[0][1]).max() > 0
    for a, b in zip(out[0][2], out[1][2]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("ny,nx", [(40, 130), (151, 301), (9, 33)])
def test_dropin_in_the_deepest_pad_vs_oracle(ny, nx):
    import fwi_gb300 as F
    acc, dpml, nt, store = 4, 54, 100, 6
    z = random_case(90 + ny, ny, nx, nt, acc, dpml, store, 4, 40)
    nts = z["nt_store"]
    Fg = np.zeros((ny, nx * (nts + 1)), np.float32, order="F")
    Fo = np.zeros_like(Fg)
    Kg = np.zeros((ny, nx), np.float32, order="F")
    Ko = Kg.copy(order="F")
    l0 = F.kernel_launch_count()
    rec_g = gpu_solver(z, 1, Kg, Fg)
    assert F.kernel_launch_count() - l0 < 10  # the whole time loop in one launch
    args = (z["nxSou"], z["nySou"], z["nxRec"], z["nyRec"], z["S"], z["Sadj"], z["d"], z["dt"], z["ctmp"], store, nts, nt)
    rec_o = O.solver_acoustic_ss(1, *args, Ko, Fo, acc=acc, dpml=dpml)
    np.testing.assert_array_equal(rec_g, rec_o)
    np.testing.assert_array_equal(Fg, Fo)
    gpu_solver(z, 2, Kg, Fg)
    O.solver_acoustic_ss(2, *args, Ko, Fo, acc=acc, dpml=dpml)
    np.testing.assert_array_equal(Kg, Ko)
