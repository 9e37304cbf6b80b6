"""The split pressure / velocity kernels in plain stream order (no programmatic dependent
launch), pinned: they serve the grids between the on-chip loops' and the one-kernel
family's, and the batches that run faster in one launch.  On small grids every output
equals the default path's (on chip) and, with FP32 histories, the oracle's, bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPLIT = 3
KEYS = ("datar", "deltadr", "deltade", "dataesc", "datae", "redatumed_raw", "redatumed")


def workload(pkg, n1=103, n2=147, npml=15, nt=90, nrec=17, nshot=1, density=False):
    from daw_b200 import synthetic
    w = synthetic.small(seed=9, n1=n1, n2=n2, npml=npml, nt=nt, nrec=nrec, nshot=nshot)
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    rng = np.random.default_rng(9)
    rec = tab(w.rec_pos[0])
    shots = []
    for k in range(nshot):  # uneven records and spreads
        n, r = nt - 11 * k, rec[k:nrec - k]
        shots.append(dict(s=w.wavelet(n), nt=n, src=tab(w.src_pos)[k], rec=r, mu=w.mu, maxiter=2,
                          dobs=np.asfortranarray(rng.standard_normal((n, r.shape[0])).astype(np.float32)),
                          rtol=0.0, band=w.band))
    return dict(w=w, shots=shots, datum=tab(w.datum_pos),
                rho=synthetic.gardner(w.c0) if density else None)


def handle(pkg, c, **opt):
    h = pkg.Handle(0, preset="mixed", **opt)
    w = c["w"]
    h.set_model(w.c0, w.npml, w.h, w.dt, w.ofs, rho=c["rho"])
    return h


def routines(h, c):
    s = c["shots"][0]
    fwd = h.submodeling(s["s"], s["src"], s["rec"], wavefield=True)
    g = h.submodeling_adjoint_esource_data(s["dobs"], s["rec"])
    return (*fwd, g, *h.submodeling_adjoint_esource(s["dobs"], s["rec"]))


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("history", [0, 1])
@pytest.mark.parametrize("density", [False, True])
def test_routines(pkg, density, history, graph):
    c = workload(pkg, density=density)
    with handle(pkg, c, history=history) as h:
        ref = routines(h, c)
        assert h.timing()["kernel_family"] == [2] * 4
    with handle(pkg, c, history=history, graph=graph, step=SPLIT) as h:
        got = routines(h, c)
        assert h.timing()["kernel_family"] == [0] * 4
    for k in range(5):
        assert np.array_equal(got[k], ref[k]), k
    assert abs(got[5] - ref[5]) <= 1e-12 * abs(ref[5])


def test_matches_oracle(pkg, O):
    c = workload(pkg)
    w, s = c["w"], c["shots"][0]
    args = (w.c0, w.npml, w.h, w.ofs, w.nt, w.dt)
    with handle(pkg, c, history=0, step=SPLIT) as h:
        sis, wf, g = routines(h, c)[:3]
    ref = O.submodeling(*args, s["s"], s["src"], s["rec"], want_wavefield=True)
    assert np.array_equal(sis, ref[0]) and np.array_equal(wf, ref[1])
    assert np.array_equal(g, O.esource_data(*args, s["dobs"], s["rec"]))


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("history", [0, 1])
def test_uneven_batch(pkg, history, graph):
    c = workload(pkg, nshot=5)
    out = []
    for opt, family in (({}, 2), ({"step": SPLIT, "graph": graph}, 0)):
        with handle(pkg, c, history=history, **opt) as h:
            h.set_datum(c["datum"])
            out.append(h.shots(c["shots"]))
            assert h.timing()["kernel_family"] == [family] * 4
    for a, b in zip(*out):
        for k in KEYS:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("window", [1, 13, 45, 89])
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("history", [0, 1])
def test_windows(pkg, history, graph, window):
    c = workload(pkg)
    with handle(pkg, c, history=history, step=SPLIT) as h:
        ref = routines(h, c)
    with handle(pkg, c, history=history, step=SPLIT, graph=graph, checkpoint=window) as h:
        got = routines(h, c)
        assert h.timing()["kernel_family"] == [0] * 4
    for k in range(5):
        assert np.array_equal(got[k], ref[k]), k
    assert abs(got[5] - ref[5]) <= 1e-12 * abs(ref[5])


def test_large_grid(pkg):
    """Beyond the line from which one kernel per step is the default."""
    c = workload(pkg, n1=1531, n2=3243, npml=17, nt=9)
    s = c["shots"][0]
    out = []
    for step, family in ((0, 1), (SPLIT, 0)):
        with handle(pkg, c, step=step) as h:
            out.append((h.submodeling(s["s"], s["src"], s["rec"])[0],
                        h.submodeling_adjoint_esource_data(s["dobs"], s["rec"])))
            assert h.timing()["kernel_family"][:3] == [family] * 3
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_other_values_are_refused(pkg):
    with pkg.Handle(0) as h:
        for v in (-1, 4):
            with pytest.raises(pkg.DawError):
                h.set_options(step=v)
