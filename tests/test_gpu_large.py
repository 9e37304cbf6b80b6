"""Grids past the on-chip loops' and the split kernels' range take one kernel per
step by themselves; the split kernels (programmatic dependent launch pins them)
are the reference.

Both compute the same separately rounded operations in the same order, so every
output is equal bit for bit.  The grids sit on both sides of the rule's line
(5 Mi padded points) and leave ragged tiles in rows and columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def workload(pkg, n1, n2, npml, nt, nrec, seed=5):
    from daw_b200 import synthetic
    w = synthetic.small(seed=seed, n1=n1, n2=n2, npml=npml, nt=nt, nrec=nrec)
    rng = np.random.default_rng(seed)
    xmax = (n2 - 1) * w.h
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    rec = tab([[2.0 * w.h, x] for x in np.linspace(0.0, xmax, nrec)])
    res = np.asfortranarray(rng.standard_normal((nt, nrec)).astype(np.float32))
    return dict(w=w, src=tab([[1.5 * w.h, 0.47 * xmax]])[0], rec=rec, s=w.wavelet(nt), res=res)


def outputs(pkg, c, rho=None, type_src=0, **opt):
    w = c["w"]
    with pkg.Handle(0, preset="mixed", **opt) as h:
        h.set_model(w.c0, w.npml, w.h, w.dt, w.ofs, rho=rho)
        fwd = h.submodeling(c["s"], c["src"], c["rec"], type_src=type_src)[0]
        g = h.submodeling_adjoint_esource_data(c["res"], c["rec"])
        es, wf, cost = h.submodeling_adjoint_esource(c["res"], c["rec"])
        return (fwd, g, es, wf, cost), h.timing()["kernel_family"]


# padded points: 1600 x 3277 = one column past the line (ragged tiles), 1600 x 3276 below it
@pytest.mark.parametrize("history", [0, 1])
@pytest.mark.parametrize("n2,family", [(3243, 1), (3242, 0)])
def test_one_kernel_per_step(pkg, n2, family, history):
    c = workload(pkg, 1531, n2, 17, 9, 40)
    got, fam = outputs(pkg, c, history=history)
    ref, fref = outputs(pkg, c, history=history, pdl=1)
    assert fam == [family] * 4 and fref == [0] * 4
    assert np.abs(ref[1]).max() > 0
    for k in range(4):
        assert np.array_equal(got[k], ref[k]), k
    assert abs(got[4] - ref[4]) <= 1e-12 * abs(ref[4])


@pytest.mark.parametrize("form", ["vz source", "density", "window"])
def test_other_forms(pkg, form):
    c = workload(pkg, 1531, 3243, 17, 9, 40)
    kw = {"vz source": dict(type_src=1), "density": dict(rho=np.full_like(c["w"].c0, 2.0)),
          "window": dict(checkpoint=4)}[form]
    got, fam = outputs(pkg, c, **kw)
    ref, _ = outputs(pkg, c, **{**kw, "pdl": 1})
    assert fam == {"vz source": [1] * 4, "density": [0] * 4, "window": [1] * 4}[form]
    for k in range(4):
        assert np.array_equal(got[k], ref[k]), k
