"""Flat grids (rows one behind the other, so that a warp may hold the end of one
row and the start of the next) and the face forms of the step kernels, at row
lengths around the warp, the CTA and the padding of a row.  FP32 against the
oracle at its parity bound; 16-bit word rows against one node per thread, bit
for bit."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
TOL = 1e-5
ROWS = [3, 8, 15, 31, 32, 33, 63, 127, 128, 129, 257]


def case(kind, nx, ny, nz):
    if kind == "cavity":
        return pkg.make_inputval(nx, ny, nz, casetype=pkg.CAVITY, tau=0.8, u=0.1, mrt=True,
                                 les=True, cs=0.1), pkg.INIT_DENSITY_NOISE, 1e-4
    return pkg.make_inputval(nx, ny, nz, casetype=pkg.CHANNEL, tau=0.7, u=0.05, mrt=True, les=True,
                             cs=0.1), pkg.INIT_CHANNEL, 0.1


@pytest.mark.parametrize("nx", ROWS)
@pytest.mark.parametrize("kind", ["cavity", "channel"])
@pytest.mark.parametrize("stream", [pkg.STREAM_AB, pkg.STREAM_AA])
def test_fp32_rows_vs_oracle(kind, stream, nx):
    iv, init, amp = case(kind, nx, 5, 6)
    d = pkg.Domain(iv, pkg.default_options(stream_mode=stream, init_kind=init, noise_amp=amp))
    ref = O.Run(iv, init_kind=init, amp=amp)
    d.run(7)
    ref.step(7)
    r = ref.fields()
    den, ux, uy, uz = d.macroscopic()
    assert O.rel_field_err(den, r["den"]) <= TOL
    assert O.rel_vel_err((ux, uy, uz), (r["ux"], r["uy"], r["uz"])) <= TOL
    assert O.rel_field_err(d.export_arF(), r["arF"]) <= TOL


@pytest.mark.parametrize("nx", [11, 12, 16, 24, 40, 63, 64, 65, 72, 200, 257])
@pytest.mark.parametrize("kind", ["cavity", "channel"])
@pytest.mark.parametrize("stream", [pkg.STREAM_AB, pkg.STREAM_AA])
def test_16bit_word_rows_equal_per_node(kind, stream, nx):
    iv, init, amp = case(kind, nx, 6, 7)
    out = []
    for kernel in (pkg.KERNEL_AUTO, pkg.KERNEL_SCALAR):
        d = pkg.Domain(iv, pkg.default_options(storage=pkg.STORE_F16_SHIFT, stream_mode=stream,
                                               kernel=kernel, init_kind=init, noise_amp=amp))
        d.run(6)
        out.append([d.export_arF()] + d.macroscopic())
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
