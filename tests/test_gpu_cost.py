"""The esource cost (sum of 0.5 sp^2 over the stage-A history): the vector loads
of the fused layout against the plain kernels' layout, on grids whose rows and
columns leave remainders; the histories of the FP32 paths are the same bits, so
the sums differ by the order of FP64 additions only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,npml", [(40, 48, 13), (41, 49, 14), (43, 63, 15), (64, 33, 16),
                                        (67, 65, 23)])
def test_cost_matches_plain_layout(pkg, n1, n2, npml):
    from daw_b200 import synthetic
    w = synthetic.small(n1=n1, n2=n2, npml=npml, nt=60, nrec=7)
    rec = pkg.subacqui(w.rec_pos[0], w.h, npml, 1)
    res = np.asfortranarray(np.random.default_rng(2).standard_normal((60, 7)).astype(np.float32))
    cost = []
    for preset, opt in (("plain", {}), ("mixed", {"history": 0}), ("mixed", {"history": 1})):
        with pkg.Handle(0, preset=preset, **opt) as h:
            h.set_model(w.c0, npml, w.h, w.dt, 1)
            cost.append(h.submodeling_adjoint_esource(res, rec, wavefield=False)[2])
    assert cost[0] > 0
    assert abs(cost[1] - cost[0]) <= 1e-13 * cost[0]
    assert abs(cost[2] - cost[0]) <= 1e-3 * cost[0]
