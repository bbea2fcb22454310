"""The pull and the in-place step of FP32 storage round every operation alike: the
same populations and fields, bit for bit, after any number of steps.  (16-bit
forms store different values, the in-place one the initial state and the walls'
values where the pull one stores what follows from them.)"""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mrt,les", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("kind", [pkg.CAVITY, pkg.CHANNEL])
def test_pull_equals_inplace(kind, mrt, les):
    iv = pkg.make_inputval(40, 12, 14, casetype=kind, tau=0.7, u=0.05, mrt=mrt, les=les, cs=0.1)
    a, b = (pkg.Domain(iv, pkg.default_options(
        stream_mode=mode, noise_amp=1e-3,
        init_kind=pkg.INIT_DENSITY_NOISE if kind == pkg.CAVITY else pkg.INIT_CHANNEL))
        for mode in (pkg.STREAM_AB, pkg.STREAM_AA))
    for n in (1, 1, 5, 20):
        a.run(n)
        b.run(n)
        np.testing.assert_array_equal(a.export_arF(), b.export_arF())
        for x, y in zip(a.macroscopic(), b.macroscopic()):
            np.testing.assert_array_equal(x, y)
