"""What the on-chip time loops keep between calls takes nothing from the rest: with
little device memory every call that fits without it succeeds, with the same
results, and as much is admitted after a run as before it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def workload(pkg, nt=700, nrec=400):
    """Receivers at the top and the bottom of the grid: the on-chip loops keep the
    pressure of most of it for the gathers."""
    from daw_b200 import synthetic
    w = synthetic.small(seed=3, n1=380, n2=1201, npml=13, nt=nt, nrec=9)
    xmax = (w.n2 - 1) * w.h
    tab = lambda p: pkg.subacqui(p, w.h, w.npml, 1)  # noqa: E731
    rec = tab([[z * w.h, x] for z in (2.0, 360.0) for x in np.linspace(0.0, xmax, nrec)])
    dobs = np.random.default_rng(1).standard_normal((nt, rec.shape[0])).astype(np.float32)
    return w, dict(s=w.wavelet(nt), nt=nt, src=tab([[1.5 * w.h, 0.47 * xmax]])[0], rec=rec,
                   dobs=np.asfortranarray(dobs), mu=1e-2, maxiter=1, rtol=0.0, band=w.band)


def handle(pkg, w):
    h = pkg.Handle(0, preset="mixed")
    h.set_model(w.c0, w.npml, w.h, w.dt, 1)
    return h


def test_pipeline_with_little_memory(pkg):
    import torch
    w, shot = workload(pkg)
    with handle(pkg, w) as h:
        ref = h.shots([shot])[0]
    for mb in (400, 448, 512, 576, 640):
        with handle(pkg, w) as h:
            free, _ = torch.cuda.mem_get_info()
            held = torch.empty(free - (mb << 20), dtype=torch.uint8, device="cuda")
            try:
                for _ in range(2):
                    got = h.shots([shot])[0]
                    for k in ("datar", "deltadr", "deltade", "dataesc", "datae"):
                        assert np.array_equal(got[k], ref[k]), (mb, k)
            finally:
                del held
                torch.cuda.empty_cache()


def admitted(pkg, h, nt, shot):
    """History window of a record too long for the device."""
    rec = np.asfortranarray(shot["rec"], np.int32)
    s, dobs = np.zeros(nt, np.float32), np.zeros((nt, 1), np.float32)
    d = (pkg.ShotDesc * 1)()
    d[0].nt, d[0].nrec = nt, 1
    d[0].s, d[0].dobs = (a.ctypes.data_as(C.POINTER(C.c_float)) for a in (s, dobs))
    for k in range(5):
        d[0].src_tab[k] = int(shot["src"][k])
    one = np.asfortranarray(rec[:1])
    d[0].rec_tab = one.ctypes.data_as(C.POINTER(C.c_int32))
    n, win = C.c_int32(), C.c_int32()
    assert pkg.lib().daw_admit_shots(h._h, 1, d, C.byref(n), C.byref(win)) == 0
    assert n.value == 1 and 0 < win.value < nt
    return win.value


def test_admission_after_a_run(pkg):
    """A run on chip keeps 512 MB of rectangles (177 steps of this grid's history); as
    long a record is admitted after it as before, the device's own allocations
    (a few MB, a step each 2.8 MB) aside."""
    w, shot = workload(pkg, nrec=9)
    with handle(pkg, w) as h:
        h.submodeling_adjoint_esource_data(shot["dobs"][:40], shot["rec"])  # kernels loaded
        before = admitted(pkg, h, 300000, shot)
        h.submodeling(shot["s"], shot["src"], shot["rec"])
        assert h.timing()["kernel_family"][0] == 2
        assert admitted(pkg, h, 300000, shot) >= before - 20
