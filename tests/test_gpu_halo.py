"""The halo words that neighbouring CTAs of the on-chip loops exchange, over many steps
on the narrowest CTAs (four columns), where a step is little else, and on ragged wider
ones: every run gives the split kernels' values bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,npml,nt,runs", [(100, 500, 20, 4000, 6), (40, 552, 20, 3000, 6),
                                                (260, 1290, 20, 1000, 3)])
def test_repeated_runs_are_equal(pkg, n1, n2, npml, nt, runs):
    from daw_b200 import synthetic
    w = synthetic.small(seed=6, n1=n1, n2=n2, npml=npml, nt=nt, nrec=40)
    xmax = (n2 - 1) * w.h
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    rec, src = tab(w.rec_pos[0]), tab([[1.5 * w.h, 0.47 * xmax]])[0]
    res = np.asfortranarray(np.random.default_rng(6).standard_normal((nt, 40)).astype(np.float32))
    with pkg.Handle(0, preset="mixed", pdl=1) as h:
        h.set_model(w.c0, npml, w.h, w.dt, 1)
        ref = h.submodeling(w.wavelet(nt), src, rec)[0], h.submodeling_adjoint_esource_data(res, rec)
        assert h.timing()["kernel_family"][:3] == [0] * 3
    assert np.abs(ref[0]).max() > 0 and np.abs(ref[1]).max() > 0
    with pkg.Handle(0, preset="mixed") as h:
        h.set_model(w.c0, npml, w.h, w.dt, 1)
        for _ in range(runs):
            assert np.array_equal(h.submodeling(w.wavelet(nt), src, rec)[0], ref[0])
            assert np.array_equal(h.submodeling_adjoint_esource_data(res, rec), ref[1])
        assert h.timing()["kernel_family"][:3] == [2] * 3
