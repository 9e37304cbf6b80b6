"""A forward run whose wavelet or time step drives values past the range of FP32: the
on-chip loops give the same values as the split kernels, NaN and Inf included.

Where the pressure is never updated (at and above the free surface, the outermost rows
and columns) it stays zero, whatever its neighbours are.  The receivers' supports
reach over the surface, and with the narrow sponge over the outermost columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npml,ofs", [(13, 1), (13, 0), (4, 1), (4, 0)])
@pytest.mark.parametrize("value,scale", [(np.nan, 1.0), (np.inf, 1.0), (3e38, 1.0), (None, 3.0)])
@pytest.mark.parametrize("tall", [False, True])  # True: rectangles too tall for shared memory
def test_same_as_split_kernels(pkg, npml, ofs, value, scale, tall):
    from daw_b200 import synthetic
    w = synthetic.small(seed=3, n1=330 if tall else 103, n2=65, npml=npml, nt=200, nrec=11)
    xmax = (w.n2 - 1) * w.h
    tab = lambda p: pkg.subacqui(p, w.h, npml, ofs)  # noqa: E731
    rec = tab([[z * w.h, x] for z in ((2.0, 310.0) if tall else (2.0,))
               for x in np.linspace(0.0, xmax, 11)])
    src = tab([[14.5 * w.h, 0.47 * xmax]])[0]
    s = w.wavelet(200).copy()
    if value is not None:
        s[20] = value
    out = []
    for opt, family in (({"pdl": 1}, 0), ({}, 2)):
        with pkg.Handle(0, preset="mixed", **opt) as h:
            h.set_model(w.c0, npml, w.h, w.dt * scale, ofs)
            sis, wf = h.submodeling(s, src, rec, wavefield=True)
            out.append((sis, wf, h.submodeling(s, src, rec)[0]))
            assert h.timing()["kernel_family"][0] == family
    assert not np.isfinite(out[0][1]).all()
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
