"""Edges of the filter's transform lengths and of the resampler's interval
search, against the CPU restatement (oracle/prep.py): one to a few samples,
lengths whose doubled size is prime, one more and one less than a transform
length, and a trace count above a grid's second dimension; output times on, just
before and just after input samples."""
import numpy as np
import pytest

from oracle import prep as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,ntr,typef,f1,fc", [
    (1, 3, 1, 0.0, 10.0), (2, 3, 1, 0.0, 40.0), (3, 2, 3, 5.0, 60.0), (7, 4, 2, 0.0, 10.0), (128, 3, 1, 0.0, 10.0),
    (129, 3, 3, 2.0, 20.0), (997, 2, 1, 0.0, 8.0), (500, 2, 2, 0.0, 8.0), (16, 65537, 1, 0.0, 30.0)])
def test_filter_lengths(nt, ntr, typef, f1, fc):
    import fwi_gb300 as F
    rng = np.random.default_rng(nt + ntr)
    data = np.asfortranarray(rng.standard_normal((nt, ntr)).astype(np.float32))
    got = F.time_filter(data.copy(order="F"), nt, 0.002, ntr, typef, f1, fc)
    ref = O.time_filter(data, 0.002, typef, f1, fc)
    # FP32 transforms: relative to the output, or to 1 % of the input where little passes
    scale = max(np.linalg.norm(ref), 1e-2 * np.linalg.norm(data))
    assert np.linalg.norm(got.astype(np.float64) - ref) <= 2e-5 * scale


@pytest.mark.parametrize("L,dt_in,dt_out", [(2, 0.004, 0.004), (3, 0.1, 0.1), (50, 0.0013, 0.0013),
                                            (700, 0.002, 0.0006666667), (333, 0.003, 0.0009999999),
                                            (64, 0.001, 0.5), (4000, 0.00127797, 0.00127796)])
def test_resampling_on_input_samples(L, dt_in, dt_out):
    import fwi_gb300 as F
    rng = np.random.default_rng(L)
    data = np.asfortranarray(rng.standard_normal((L, 3)).astype(np.float32))
    nt = int(L * dt_in / dt_out) + 3
    got = F.interpolation_akima(data, dt_in, L, 3, dt_out, nt)
    np.testing.assert_array_equal(got, O.akima(data, dt_in, dt_out, nt))
