"""The on-chip loops' waits run out (on the host's request, after one round: no GPU
fault is involved): the call reports DAW_ERR_TIMEOUT and the handle's next calls are
bit-exact, whatever the abandoned run left in the exchange buffers.  And the step
tags start over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case(pkg, n1=151, n2=461, npml=20, nt=120, nshot=3):
    from daw_b200 import synthetic
    w = synthetic.small(seed=8, n1=n1, n2=n2, npml=npml, nt=nt, nrec=31, nshot=nshot)
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    rng = np.random.default_rng(8)
    rec = tab(w.rec_pos[0])
    shots = [dict(s=w.wavelet(nt), nt=nt, src=tab(w.src_pos)[k], rec=rec, mu=w.mu, maxiter=1,
                  dobs=np.asfortranarray(rng.standard_normal((nt, 31)).astype(np.float32)),
                  rtol=0.0, band=w.band) for k in range(nshot)]
    return w, shots


def calls(h, shots):
    s = shots[0]
    yield "forward", lambda: [h.submodeling(s["s"], s["src"], s["rec"])[0]]
    yield "operator", lambda: [h.submodeling_adjoint_esource_data(s["dobs"], s["rec"])]
    yield "batch", lambda: [r[k] for r in h.shots(shots) for k in ("datar", "deltade", "datae")]


@pytest.mark.parametrize("opt", [{}, {"history": 0}, {"checkpoint": 40, "max_batch": 1}])
def test_wait_gives_up(pkg, opt):
    w, shots = case(pkg)
    with pkg.Handle(0, preset="mixed", **opt) as h:
        h.set_model(w.c0, w.npml, w.h, w.dt, 1)
        ref = {name: f() for name, f in calls(h, shots)}
        assert h.timing()["kernel_family"] == [2] * 4
        for name, f in calls(h, shots):
            assert pkg.lib().daw_selftest_onchip(h._h, 1, 0) == 0
            for _ in range(2):
                with pytest.raises(pkg.DawError) as e:
                    f()
                assert e.value.code == -4 and "on-chip" in str(e.value), str(e.value)
            assert pkg.lib().daw_selftest_onchip(h._h, 0, 0) == 0
            for got, want in zip(f(), ref[name]):
                assert np.array_equal(got, want), name


def test_step_tags_start_over(pkg):
    w, shots = case(pkg)
    with pkg.Handle(0, preset="mixed") as h:
        h.set_model(w.c0, w.npml, w.h, w.dt, 1)
        ref = {name: f() for name, f in calls(h, shots)}
        for tag in (0xe0000000 - 60, 0xe0000001):  # past the line within a run, before it
            for name, f in calls(h, shots):
                assert pkg.lib().daw_selftest_onchip(h._h, 0, tag) == 0
                for _ in range(2):
                    for got, want in zip(f(), ref[name]):
                        assert np.array_equal(got, want), (name, tag)
