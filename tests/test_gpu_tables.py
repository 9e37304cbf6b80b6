"""Station tables built on the device (tables.cu) against the host-built ones.

The plain kernels read maps built on the host; the TMA kernels and the on-chip
loops read maps and tiles built on the device.  Simulations of both are equal
bit for bit (FP32 histories), for station sets where the tables can go wrong:
supports cut by every edge and wholly outside, free-surface folds of 0 to 10
rows, more stations than a block takes at a time, coincident stations, and a
vertical line (more rows in a column than a block has threads).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N1, N2, NPML, NT = 150, 70, 13, 40


def tables():
    rng = np.random.default_rng(5)
    n1e, n2e = N1 + 2 * NPML, N2 + 2 * NPML

    def tab(ix1, ix2, nfs=0):
        n = len(ix1)
        t = np.zeros((n, 5), np.int32, order="F")
        t[:, 0], t[:, 1] = ix1, ix2
        t[:, 2], t[:, 3] = rng.integers(1, 101, n), rng.integers(1, 101, n)
        t[:, 4] = nfs
        return t

    line = np.arange(20, 80)
    return {
        "edges": tab([-9, 1, 11, n1e - 10, n1e, n1e + 10, 80, 80, 80, 80],
                     [30, 30, 30, 30, 30, 30, -9, 1, n2e, n2e + 10]),
        "folds": tab([NPML + 1 + k for k in range(11)], [15 + 5 * k for k in range(11)],
                     np.arange(10, -1, -1)),
        "many": tab(rng.integers(NPML + 1, NPML + 5, 300), rng.integers(20, 75, 300)),
        "coincident": tab([40] * 130, [40] * 130),
        "vertical": tab(np.arange(14, 160), [45] * 146),
        "two lines": np.asfortranarray(np.concatenate([tab([20] * 60, line), tab([130] * 60, line)])),
        "one": tab([60], [30]),
    }


@pytest.mark.parametrize("name", list(tables()))
def test_device_tables_equal_host_tables(pkg, name):
    from daw_b200 import synthetic
    w = synthetic.small(n1=N1, n2=N2, npml=NPML, nt=NT)
    rec = tables()[name]
    res = np.asfortranarray(np.random.default_rng(1).standard_normal((NT, len(rec))).astype(np.float32))
    s = w.wavelet(NT + 60)[60:].copy()
    src = pkg.subacqui([[40.0, 350.0]], w.h, NPML, 1)[0]
    out = []
    for preset, opt in (("plain", {}), ("mixed", {"history": 0, "pdl": 1}), ("mixed", {"history": 0})):
        with pkg.Handle(0, preset=preset, **opt) as h:
            h.set_model(w.c0, NPML, w.h, w.dt, 1)
            out.append((h.submodeling(s, src, rec)[0],
                        h.submodeling_adjoint_esource_data(res, rec)))
    assert np.abs(out[0][1]).max() > 0
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
