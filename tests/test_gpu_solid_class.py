"""Nodes beside solid voxels (class kSolidNear) against the plain streaming of
the others, on masks that touch every face, edge and corner of the box: the
oracle checks every donor of every node.  Tolerance: the FP32 parity bound."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("shape", [(5, 6, 7), (33, 9, 8), (130, 7, 10)])
@pytest.mark.parametrize("share", [0.01, 0.2])
@pytest.mark.parametrize("case", [pkg.CAVITY, pkg.CHANNEL])
def test_scattered_voxels_vs_oracle(case, share, shape):
    nx, ny, nz = shape
    iv = pkg.make_inputval(nx, ny, nz, casetype=case, tau=0.8, u=0.05, mrt=True, les=True, cs=0.1)
    kind, amp = (1, 1e-6) if case == pkg.CAVITY else (pkg.INIT_CHANNEL, 0.01)
    m = np.random.default_rng(5).random((ny, nz, nx)) < share
    d = pkg.Domain(iv, pkg.default_options(init_kind=kind, noise_amp=amp))
    d.set_solid_mask(m)
    ref = O.Run(iv, init_kind=kind, amp=amp)
    ref.set_solid(m)
    d.run(20)
    ref.step(20)
    r = ref.fields()
    den, ux, uy, uz = d.macroscopic()
    assert O.rel_field_err(den, r["den"]) <= TOL
    assert O.rel_vel_err((ux, uy, uz), (r["ux"], r["uy"], r["uz"])) <= TOL
    assert O.rel_field_err(d.export_arF(), r["arF"]) <= TOL
