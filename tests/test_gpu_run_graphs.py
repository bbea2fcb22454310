"""The graphs of a domain's runs: the rest graph replaced while its last launch
may still be running, and the same steps on the streams a caller may hand over:
the default stream, and a stream whose launches the caller captures into a graph
of its own and replays.  The same kernels on the same data, so every result is
equal bit for bit."""
import numpy as np
import pytest

import oracle_lib as O

pkg = O.pkg
pytestmark = pytest.mark.gpu
FORMS = [(pkg.STORE_F32, pkg.STREAM_AB, 0), (pkg.STORE_F32, pkg.STREAM_AA, 0),
         (pkg.STORE_F16_SHIFT, pkg.STREAM_AB, 1), (pkg.STORE_F16_SHIFT, pkg.STREAM_AA, 1),
         (pkg.STORE_F64, pkg.STREAM_AA, 0)]


def domain(storage, stream, rounding, kind=pkg.CHANNEL):
    iv = pkg.make_inputval(24, 9, 10, casetype=kind, tau=0.7, u=0.05, mrt=True, les=True, cs=0.1)
    return pkg.Domain(iv, pkg.default_options(
        storage=storage, stream_mode=stream, rounding=rounding, init_kind=pkg.INIT_CHANNEL,
        noise_amp=0.1))


def equal(a, b):
    np.testing.assert_array_equal(a.export_arF(), b.export_arF())
    for x, y in zip(a.macroscopic(), b.macroscopic()):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("storage,stream,rounding", FORMS)
def test_replaced_rest(storage, stream, rounding):
    a, b = domain(storage, stream, rounding), domain(storage, stream, rounding)
    cut = [6] * 6 + [10] * 24 + [6, 10] * 8 + [8] * 14 + [70] * 14 + [40] * 12
    for n in cut:
        a.run(n)
    b.run(sum(cut))
    equal(a, b)


@pytest.mark.parametrize("storage,stream,rounding", FORMS)
def test_default_stream(storage, stream, rounding):
    a, b = domain(storage, stream, rounding), domain(storage, stream, rounding)
    a.sync()
    a.set_stream(0)
    for n in (1, 3, 6, 6, 6, 70, 70):
        a.run(n)
    b.run(162)
    equal(a, b)


@pytest.mark.parametrize("steps", [6, 72])
@pytest.mark.parametrize("storage,stream,rounding", FORMS)
def test_captured_stream(storage, stream, rounding, steps):
    torch = pytest.importorskip("torch")
    a, b = domain(storage, stream, rounding), domain(storage, stream, rounding)
    a.sync()
    s = torch.cuda.Stream()
    a.set_stream(s.cuda_stream)
    for n in (4, 6, 6, 6):  # the rest graph exists by the time of the capture
        a.run(n)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        a.run(steps)
    with torch.cuda.stream(s):
        for _ in range(3):
            g.replay()
    b.run(22 + 3 * steps)
    equal(a, b)  # an even number of steps: the domain's parity is that of the replays
    a.run(7)
    b.run(7)
    equal(a, b)
    a.sync()
    del g
    a.close()
