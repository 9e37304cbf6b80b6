"""The on-chip time loops (stencil_resident.cu) against the split pressure /
velocity kernels (programmatic dependent launch pins those) and the FP32 oracle.

Both compute the same separately rounded operations in the same order, so
every output is equal bit for bit, FP16 histories included (their scales are
the same powers of two).  The grids sit where the partition can go wrong: few
columns per CTA and columns left over in the last one, one to fifteen row
blocks of 128 with full and nearly empty last blocks, column groups of one
column, and a grid just too tall.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RESIDENT = 2  # timing()["kernel_family"]


def workload(pkg, n1, n2, npml, nt, nrec, rows=(2.0,), density=False, seed=3):
    from daw_b200 import synthetic
    w = synthetic.small(seed=seed, n1=n1, n2=n2, npml=npml, nt=nt, nrec=nrec)
    rng = np.random.default_rng(seed)
    xmax = (n2 - 1) * w.h
    pos = [[z * w.h, x] for z in rows for x in np.linspace(0.0, xmax, nrec)]
    res = np.asfortranarray(rng.standard_normal((nt, len(pos))).astype(np.float32))
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    return dict(w=w, src=tab([[1.5 * w.h, 0.47 * xmax]])[0], rec=tab(pos), datum=tab(w.datum_pos),
                s=w.wavelet(nt), res=res,
                rho=synthetic.gardner(w.c0) if density else None)


def handle(pkg, c, **opt):
    w = c["w"]
    h = pkg.Handle(0, preset="mixed", **opt)
    h.set_model(w.c0, w.npml, w.h, w.dt, w.ofs, rho=c["rho"])
    return h


# n1, n2, npml, nt: extended sizes 20x24 (one row block, CTAs of 4 columns, whose source touches
# rows that are never updated: not on chip), 128 rows exactly and 2 columns in the last CTA, 129
# rows (a second block with one row), 512 (four blocks: the extra warp comes last), 960, 1024 and
# 1920 rows (the tallest), odd sizes
GRIDS = [(14, 18, 3, 90), (102, 64, 13, 120), (103, 65, 13, 120), (486, 75, 13, 80),
         (934, 60, 13, 60), (998, 60, 13, 60), (1894, 52, 13, 40), (77, 461, 21, 100),
         (151, 1203, 30, 60)]
# CTAs of 5 and 7 columns over three and four column groups, whose first then has one column: the
# second group's first column is the left edge's second one
GRIDS += [(60, 560, 21, 60), (300, 900, 21, 60), (470, 620, 21, 60)]


@pytest.mark.parametrize("history", [0, 1])
@pytest.mark.parametrize("n1,n2,npml,nt", GRIDS)
def test_equals_split_kernels(pkg, n1, n2, npml, nt, history):
    c = workload(pkg, n1, n2, npml, nt, 11)
    out = []
    for opt, family in (({"pdl": 1}, 0), ({}, RESIDENT)):
        with handle(pkg, c, history=history, **opt) as h:
            fwd, wf = h.submodeling(c["s"], c["src"], c["rec"], wavefield=True)
            g = h.submodeling_adjoint_esource_data(c["res"], c["rec"])
            es, wfe, cost = h.submodeling_adjoint_esource(c["res"], c["rec"])
            fam = h.timing()["kernel_family"]
        assert fam == [family if npml >= 13 else 0] * 4
        out.append((fwd, wf, g, es, wfe, cost))
    a, b = out
    assert np.abs(a[2]).max() > 0
    for k in range(5):
        assert np.array_equal(a[k], b[k]), k
    assert abs(a[5] - b[5]) <= 1e-12 * abs(a[5])


def test_too_tall_grid_runs_from_memory(pkg):
    c = workload(pkg, 1895, 40, 13, 30, 5)
    with handle(pkg, c) as h:
        h.submodeling_adjoint_esource_data(c["res"], c["rec"])
        assert h.timing()["kernel_family"][1:3] == [0, 0]


@pytest.mark.parametrize("history", [0, 1])
def test_density_equals_split_kernels(pkg, history):
    c = workload(pkg, 130, 203, 14, 90, 17, density=True)
    out = []
    for opt in ({"pdl": 1}, {}):
        with handle(pkg, c, history=history, **opt) as h:
            out.append((h.submodeling(c["s"], c["src"], c["rec"])[0],
                        h.submodeling_adjoint_esource_data(c["res"], c["rec"])))
            fam = h.timing()["kernel_family"][:3]
    assert fam == [RESIDENT] * 3
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_matches_oracle(pkg, O):
    """A ragged grid against the CPU oracle, FP32 histories: bit for bit."""
    c = workload(pkg, 97, 301, 15, 150, 23)
    w = c["w"]
    args = (w.c0, w.npml, w.h, w.ofs, w.nt, w.dt)
    with handle(pkg, c, history=0) as h:
        fwd = h.submodeling(c["s"], c["src"], c["rec"])[0]
        g = h.submodeling_adjoint_esource_data(c["res"], c["rec"])
        assert h.timing()["kernel_family"][:3] == [RESIDENT] * 3
    assert np.array_equal(fwd, O.submodeling(*args, c["s"], c["src"], c["rec"])[0])
    assert np.array_equal(g, O.esource_data(*args, c["res"], c["rec"]))


def test_long_loop_is_cut_into_launches(pkg):
    """Receivers at the top and the bottom of the grid: the gathers read most of
    it every step, so the loop runs in several launches with the state stored
    between them."""
    c = workload(pkg, 380, 1201, 13, 700, 9, rows=(2.0, 360.0))
    out = []
    for opt in ({"pdl": 1}, {}):
        with handle(pkg, c, **opt) as h:
            out.append((h.submodeling(c["s"], c["src"], c["rec"])[0],
                        h.submodeling_adjoint_esource_data(c["res"], c["rec"])))
            fam = h.timing()["kernel_family"][:3]
    assert fam == [RESIDENT] * 3
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_little_device_memory(pkg):
    """With a quarter GB of device memory left the kept rectangles get a smaller
    buffer and the loop more launches."""
    import torch
    c = workload(pkg, 380, 1201, 13, 700, 9, rows=(2.0, 360.0))
    with handle(pkg, c) as h:
        ref = h.submodeling(c["s"], c["src"], c["rec"])[0]
        launches = h.timing()["kernel_launches"]
    with handle(pkg, c) as h:
        free, _ = torch.cuda.mem_get_info()
        held = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = h.submodeling(c["s"], c["src"], c["rec"])[0]
        finally:
            del held
            torch.cuda.empty_cache()
        tim = h.timing()
    assert tim["kernel_family"][0] == RESIDENT and tim["kernel_launches"] > launches
    assert np.array_equal(got, ref)


def test_uneven_batch_equals_split_kernels(pkg):
    """Shots of different lengths and spreads share launches."""
    base = workload(pkg, 90, 160, 14, 160, 19)
    w = base["w"]
    shots = []
    for k in range(5):
        nt = 160 - 23 * k
        rec = base["rec"][k:19 - k]
        shots.append(dict(s=w.wavelet(nt), nt=nt, src=base["src"], rec=rec,
                          dobs=np.asfortranarray(base["res"][:nt, k:19 - k]) * 1e-3, mu=w.mu,
                          maxiter=2, rtol=0.0, band=w.band))
    out = []
    for opt in ({"pdl": 1}, {}):
        with handle(pkg, base, **opt) as h:
            h.set_datum(base["datum"])
            out.append(h.shots(shots))
            tim = h.timing()
    assert tim["kernel_family"] == [RESIDENT] * 4 and tim["shots_per_launch"][1] > 1
    for a, b in zip(*out):
        for k in ("datar", "deltadr", "deltade", "dataesc", "datae", "redatumed_raw", "redatumed"):
            assert np.array_equal(a[k], b[k]), k


def test_two_handles_from_two_threads(pkg):
    """Launches of different handles on one GPU follow one another."""
    import threading
    c = workload(pkg, 100, 400, 14, 200, 15)
    with handle(pkg, c) as h:
        ref = h.submodeling_adjoint_esource_data(c["res"], c["rec"])
    got = [None, None]

    def work(i):
        with handle(pkg, c) as h:
            for _ in range(3):
                got[i] = h.submodeling_adjoint_esource_data(c["res"], c["rec"])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert np.array_equal(got[0], ref) and np.array_equal(got[1], ref)
