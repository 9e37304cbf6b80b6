"""Forms of the on-chip loops' runs that the grids of the other tests do not reach:
no free surface (the pressure is not zeroed and vz not copied at the top), a sponge of
128 rows (with a free surface the rows of that copy belong to two warps and the run
goes to the separate kernels), and windows of a checkpointed shot with both history
precisions, the wavefield output and the datum.  The separate kernels, and the oracle,
are the reference: every output is equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def workload(pkg, n1, n2, npml, nt, ofs, nrec=11):
    from daw_b200 import synthetic
    w = synthetic.small(seed=10, n1=n1, n2=n2, npml=npml, nt=nt, nrec=nrec)
    xmax = (n2 - 1) * w.h
    tab = lambda p: pkg.subacqui(p, w.h, npml, ofs)  # noqa: E731
    res = np.random.default_rng(10).standard_normal((nt, nrec)).astype(np.float32)
    return dict(w=w, ofs=ofs, src=tab([[1.5 * w.h, 0.47 * xmax]])[0], datum=tab(w.datum_pos),
                rec=tab([[2.0 * w.h, x] for x in np.linspace(0.0, xmax, nrec)]),
                s=w.wavelet(nt), res=np.asfortranarray(res))


def routines(pkg, c, **opt):
    w = c["w"]
    with pkg.Handle(0, preset="mixed", **opt) as h:
        h.set_model(w.c0, w.npml, w.h, w.dt, c["ofs"])
        out = (*h.submodeling(c["s"], c["src"], c["rec"], wavefield=True),
               h.submodeling_adjoint_esource_data(c["res"], c["rec"]),
               *h.submodeling_adjoint_esource(c["res"], c["rec"]))
        return out, h.timing()["kernel_family"]


def same(a, b):
    for k in range(5):
        assert np.abs(b[k]).max() > 0 and np.array_equal(a[k], b[k]), k
    assert abs(a[5] - b[5]) <= 1e-12 * abs(b[5])


@pytest.mark.parametrize("history", [0, 1])
@pytest.mark.parametrize("n1,n2,npml,nt,ofs", [
    (102, 64, 13, 120, 0), (103, 65, 13, 120, 0), (486, 75, 13, 80, 0), (998, 60, 13, 60, 0),
    (77, 461, 21, 100, 0), (60, 64, 128, 60, 0), (60, 64, 128, 60, 1), (60, 64, 127, 60, 1),
    (60, 64, 129, 60, 1)])
def test_surface(pkg, n1, n2, npml, nt, ofs, history):
    c = workload(pkg, n1, n2, npml, nt, ofs)
    got, family = routines(pkg, c, history=history)
    ref, rfamily = routines(pkg, c, history=history, step=3)
    on_chip = not (ofs == 1 and npml == 128)
    assert family == [2 if on_chip else 0] * 4 and rfamily == [0] * 4
    same(got, ref)


def test_no_surface_matches_oracle(pkg, O):
    c = workload(pkg, 97, 141, 15, 120, 0)
    w = c["w"]
    args = (w.c0, w.npml, w.h, 0, w.nt, w.dt)
    got, family = routines(pkg, c, history=0)
    assert family == [2] * 4
    ref = O.submodeling(*args, c["s"], c["src"], c["rec"], want_wavefield=True)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    assert np.array_equal(got[2], O.esource_data(*args, c["res"], c["rec"]))


# the first window's end before and after the receivers are reached, windows of one step and
# of all but one
@pytest.mark.parametrize("window", [1, 7, 50, 99])
@pytest.mark.parametrize("history", [0, 1])
@pytest.mark.parametrize("n1,n2", [(103, 147), (151, 461), (300, 900)])
def test_windows(pkg, n1, n2, history, window):
    c = workload(pkg, n1, n2, 15, 100, 1)
    ref, rfamily = routines(pkg, c, history=history, step=3)
    got, family = routines(pkg, c, history=history, checkpoint=window)
    assert family == [2] * 4 and rfamily == [0] * 4
    same(got, ref)


@pytest.mark.parametrize("history", [0, 1])
def test_windowed_pipeline(pkg, history):
    c = workload(pkg, 103, 147, 15, 100, 1)
    w = c["w"]
    shot = dict(s=c["s"], nt=100, src=c["src"], rec=c["rec"], dobs=c["res"], mu=w.mu, maxiter=2,
                rtol=0.0, band=w.band)
    out = []
    for opt, family in (({"step": 3}, 0), ({"checkpoint": 30}, 2)):
        with pkg.Handle(0, preset="mixed", history=history, **opt) as h:
            h.set_model(w.c0, w.npml, w.h, w.dt, 1)
            h.set_datum(c["datum"])
            out.append(h.shots([shot], wavefield=True)[0])
            assert h.timing()["kernel_family"] == [family] * 4
    keys = [k for k, v in out[0].items() if isinstance(v, np.ndarray)]
    assert "redatumed" in keys and any("wavefield" in k for k in keys)
    for k in keys:
        assert np.array_equal(out[0][k], out[1][k]), k
