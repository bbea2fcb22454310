"""Solid voxels beside the inlet (x = 1) and at the outlet (x = nx - 2, nx - 1) of
a channel: the rules there read the density and the velocity of nodes that are
never measured, which are those of the starting state, whatever the domain did
before."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
TOL = 1e-5


def channel(storage=pkg.STORE_F32):
    iv = pkg.make_inputval(20, 8, 9, casetype=pkg.CHANNEL, tau=0.8, u=0.05, mrt=True, les=True,
                           cs=0.1)
    return iv, pkg.Domain(iv, pkg.default_options(storage=storage, init_kind=pkg.INIT_CHANNEL,
                                                  noise_amp=0.01))


def mask(shape):
    m = np.zeros(shape, bool)
    m[3, 4, 1] = m[5, 5, 18] = m[2, 6, 19] = True
    return m


@pytest.mark.parametrize("before", [0, 3, 4])
def test_mask_on_a_domain_that_ran(before):
    iv, d = channel()
    d.run(before)
    m = mask(d.shape)
    d.set_solid_mask(m)
    ref = O.Run(iv, init_kind=pkg.INIT_CHANNEL, amp=0.01)
    ref.set_solid(m)
    for n in (1, 1, 5):
        d.run(n)
        ref.step(n)
        r = ref.fields()
        den, ux, uy, uz = d.macroscopic()
        assert O.rel_field_err(den, r["den"]) <= TOL
        assert O.rel_vel_err((ux, uy, uz), (r["ux"], r["uy"], r["uz"])) <= TOL
        assert O.rel_field_err(d.export_arF(), r["arF"]) <= TOL


@pytest.mark.parametrize("storage", [pkg.STORE_F32, pkg.STORE_F16_SHIFT, pkg.STORE_F64])
def test_import_forgets_the_run_before(storage):
    a, b = channel(storage)[1], channel(storage)[1]
    start = None
    for d, before in ((a, 0), (b, 3)):
        d.run(5)
        d.set_solid_mask(mask(d.shape))
        if start is None:
            start = d.export_arF()
        d.run(before)
        d.import_arF(start)
        d.run(4)
    np.testing.assert_array_equal(a.export_arF(), b.export_arF())
