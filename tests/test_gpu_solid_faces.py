"""Solid voxels on every corner, edge and face of the box and one node inside of
each: the classes (solid, beside solid, free) where the box ends, in every
storage form of the pull step.  FP32 and FP64 against the oracle at the FP32
parity bound; 16-bit against FP64 within what its storage rounds: a step rounds
each population to 2^-11 of its deviation and relaxes with a factor below 4,
while a wrong donor is off by the size of a deviation."""
import itertools

import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
TOL = 1e-5
SHAPES = [(9, 8, 10), (34, 7, 9)]


def voxels(nx, ny, nz):
    m = np.zeros((ny, nz, nx), bool)
    for ends in itertools.product((0, 1, 2), repeat=3):
        if ends.count(2) == 3:
            continue
        for inside in (0, 1):
            # 0 / 1: at the low / high end of the side, 2: somewhere along it
            p = [(inside, n - 1 - inside, (3 + 2 * inside) % n)[e] for e, n in
                 zip(ends, (ny, nz, nx))]
            m[tuple(p)] = True
    return m


def make(case, shape, storage):
    nx, ny, nz = shape
    iv = pkg.make_inputval(nx, ny, nz, casetype=case, tau=0.8, u=0.05, mrt=True, les=True, cs=0.1)
    kind, amp = (1, 1e-6) if case == pkg.CAVITY else (pkg.INIT_CHANNEL, 0.01)
    d = pkg.Domain(iv, pkg.default_options(storage=storage, init_kind=kind, noise_amp=amp))
    return d, iv, kind, amp


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("one", [False, True])
@pytest.mark.parametrize("case", [pkg.CAVITY, pkg.CHANNEL])
@pytest.mark.parametrize("storage", [pkg.STORE_F32, pkg.STORE_F64])
def test_voxels_at_the_faces_vs_oracle(storage, case, one, shape):
    full = voxels(*shape)
    # all together, or a few at a time (so that their neighbours see one voxel each)
    at = np.argwhere(full)
    for part in ([at[i::6] for i in range(6)] if one else [at]):
        m = np.zeros_like(full)
        m[tuple(part.T)] = True
        d, iv, kind, amp = make(case, shape, storage)
        d.set_solid_mask(m)
        ref = O.Run(iv, init_kind=kind, amp=amp)
        ref.set_solid(m)
        d.run(8)
        ref.step(8)
        r = ref.fields()
        den, ux, uy, uz = d.macroscopic()
        assert O.rel_field_err(den, r["den"]) <= TOL
        assert O.rel_vel_err((ux, uy, uz), (r["ux"], r["uy"], r["uz"])) <= TOL
        assert O.rel_field_err(d.export_arF(), r["arF"]) <= TOL


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("case", [pkg.CAVITY, pkg.CHANNEL])
def test_voxels_at_the_faces_16bit(case, shape):
    steps, m = 4, voxels(*shape)
    out = []
    for storage in (pkg.STORE_F16_SHIFT, pkg.STORE_F64):
        d = make(case, shape, storage)[0]
        d.set_solid_mask(m)
        d.run(steps)
        out.append(d.export_arF().astype(np.float64))
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    size = np.abs(out[1] - w)[~m].max()
    assert np.abs(out[0] - out[1]).max() <= steps * 4 * 2.0 ** -11 * size
