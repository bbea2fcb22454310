"""The same steps however a run is cut: single steps, repeated short runs (whose
launches become a graph), runs of whole chunks with and without a rest, odd and
even lengths from either lattice.  Every cut runs the same kernels on the same
data, so the state and the fields are equal bit for bit; the fields of a cut's
last step do not depend on how the steps before it were launched."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
CUTS = [
    [1] * 5 + [6] * 6 + [38] * 4,
    [7] * 12 + [34, 34, 34, 4, 3],
    [96, 97] + [0, 2],
    [5, 9, 5, 9] + [33] * 5,
]


@pytest.mark.parametrize("storage,rounding", [(pkg.STORE_F32, pkg.ROUND_NEAREST),
                                              (pkg.STORE_F16_SHIFT, pkg.ROUND_STOCHASTIC),
                                              (pkg.STORE_F64, pkg.ROUND_NEAREST)])
@pytest.mark.parametrize("stream", [pkg.STREAM_AB, pkg.STREAM_AA])
@pytest.mark.parametrize("kind", [pkg.CAVITY, pkg.CHANNEL])
def test_cuts_of_a_run(kind, stream, storage, rounding):
    iv = pkg.make_inputval(24, 9, 10, casetype=kind, tau=0.7, u=0.05, mrt=True, les=True, cs=0.1)
    o = pkg.default_options(storage=storage, stream_mode=stream, rounding=rounding,
                            init_kind=pkg.INIT_CHANNEL, noise_amp=0.1)
    for cut in CUTS:
        a, b = pkg.Domain(iv, o), pkg.Domain(iv, o)
        for n in cut:
            a.run(n)
        b.run(sum(cut))
        assert a.steps() == b.steps() == sum(cut)
        np.testing.assert_array_equal(a.export_arF(), b.export_arF())
        for x, y in zip(a.macroscopic(), b.macroscopic()):
            np.testing.assert_array_equal(x, y)
        a.run(13)
        b.run(13)
        np.testing.assert_array_equal(a.diagnostics(), b.diagnostics())
