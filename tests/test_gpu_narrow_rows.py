"""Paired rows (16-bit pull) at the narrowest boxes that take them: the paired
step against one node per thread, bit for bit, with either rounding."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [6, 7, 8, 10, 18])
@pytest.mark.parametrize("kind", [pkg.CAVITY, pkg.CHANNEL])
@pytest.mark.parametrize("rounding", [pkg.ROUND_NEAREST, pkg.ROUND_STOCHASTIC])
@pytest.mark.parametrize("storage", [pkg.STORE_F16_SHIFT, pkg.STORE_BF16_SHIFT])
def test_narrow_paired_rows_equal_per_node(storage, rounding, kind, nx):
    iv = pkg.make_inputval(nx, 6, 7, casetype=kind, tau=0.7, u=0.05, mrt=True, les=True, cs=0.1)
    out = []
    for kernel in (pkg.KERNEL_PAIRED, pkg.KERNEL_SCALAR):
        d = pkg.Domain(iv, pkg.default_options(
            storage=storage, rounding=rounding, kernel=kernel, noise_amp=0.1,
            init_kind=pkg.INIT_DENSITY_NOISE if kind == pkg.CAVITY else pkg.INIT_CHANNEL))
        d.run(6)
        out.append([d.export_arF()] + d.macroscopic())
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
