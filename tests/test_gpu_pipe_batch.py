"""Pipes (STRUCT nodes outside the radius) as batch members: packed with others,
and alone in a set, where the member takes the step kernel of such geometries;
the same bits as a domain of its own."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [pkg.STORE_F32, pkg.STORE_F16_SHIFT])
@pytest.mark.parametrize("schedule", [0, 1, 2])
def test_pipe_members_equal_alone(schedule, storage):
    ivs = [pkg.make_inputval(n, 51, 51, casetype=pkg.POISEUILLE, tau=0.8, u=0.05, mrt=True,
                             les=True, cs=0.1) for n in (17, 24, 120)]  # the last: over 2048 CTAs
    o = pkg.default_options(storage=storage, init_kind=pkg.INIT_DENSITY_NOISE, noise_amp=1e-3)
    need = sum(pkg.batch_domain_bytes(iv, o) for iv in ivs) + (len(ivs) << 16)
    b = pkg.Batch(hbm_budget=need, chunk_steps=8, schedule=schedule)
    ids = [b.add(iv, o, steps=21) for iv in ivs]
    for _ in range(3):
        b.step(8)
    b.sync()
    for iv, i in zip(ivs, ids):
        d = pkg.Domain(iv, o)
        d.run(21)
        m = b.member(i)
        np.testing.assert_array_equal(m.export_arF(), d.export_arF())
        for x, y in zip(m.macroscopic(), d.macroscopic()):
            np.testing.assert_array_equal(x, y)
        d.close()
    b.close()
