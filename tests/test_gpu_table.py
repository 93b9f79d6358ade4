"""The tabulated radial kernel on the device (csrc/kernels.cuh RadialTableF64:
octave and place from the bits, coefficients in pairs) at odd, even and the
smallest counts of coefficients, at both ends of an octave, at the ends of the
table and beyond, against the host's evaluation of the same table.  Both take the
same operations; the device fuses one multiplication and one addition in each
step, so n steps differ by a few n units of 1e-16 of the largest partial sum:
bar 1e-14 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 9, 24, 25])
def test_table_matches_host(built_lib, n):
    from flexmm_b200 import direct_evaluation
    from flexmm_b200.kernels import radial
    k = radial(lambda r: 1.0 / (3.0 + np.asarray(r)), 2.0 ** -7, 8.0, tol=1.0, n=n)
    e = 2.0 ** np.arange(-9, 6)
    r = np.concatenate([e, np.nextafter(e, 0.0), np.nextafter(e, 1e9), 1.37 * e, [0.0, 1e-300, 1e9]])
    got = direct_evaluation(k, np.zeros(1), np.zeros(1), np.ones(1), r, np.zeros_like(r))
    want = k.table(r)
    assert np.max(np.abs(got - want)) < 1e-14 * np.max(np.abs(want))
