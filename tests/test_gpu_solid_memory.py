"""A solid mask takes its class bytes and nothing else: no staging buffer stays
with the domain, and the domain is as without the mask once it is taken off."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [pkg.STORE_F32, pkg.STORE_F16_SHIFT, pkg.STORE_F64])
def test_mask_keeps_no_staging(storage):
    iv = pkg.make_inputval(40, 12, 14, casetype=pkg.CHANNEL, tau=0.7, u=0.05, mrt=True, les=True,
                           cs=0.1)
    o = pkg.default_options(storage=storage, init_kind=pkg.INIT_CHANNEL, noise_amp=0.1)
    d, plain = pkg.Domain(iv, o), pkg.Domain(iv, o)
    before = d.device_bytes()
    m = np.zeros(d.shape, bool)
    m[4:8, 5:9, 10:16] = True
    d.set_solid_mask(m)
    d.run(5)
    assert d.device_bytes() == before
    # 16-bit rows change with the mask and back
    d.set_solid_mask(None)
    for n in (5, 40, 40, 40):
        d.run(n)
        plain.run(n)
    np.testing.assert_array_equal(d.export_arF(), plain.export_arF())
    for x, y in zip(d.macroscopic(), plain.macroscopic()):
        np.testing.assert_array_equal(x, y)
