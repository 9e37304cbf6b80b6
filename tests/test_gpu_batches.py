"""Batches of shots on grids that leave room on the chip: the on-chip loops take as
many columns per CTA as let a launch hold the batch's shots (one after the other
with the narrowest CTAs cost more than the split kernels, which take a whole batch
in one launch), and a small grid many times over runs in the split kernels.

Both compute the same separately rounded operations in the same order, so every
output is equal bit for bit; programmatic dependent launch pins the split kernels
for the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("datar", "deltadr", "deltade", "dataesc", "datae", "redatumed_raw", "redatumed")


def batch(pkg, n1, n2, npml, nt, nrec, nshot, seed=4):
    from daw_b200 import synthetic
    w = synthetic.small(seed=seed, n1=n1, n2=n2, npml=npml, nt=nt, nrec=nrec, nshot=nshot)
    tab = lambda p: pkg.subacqui(p, w.h, npml, 1)  # noqa: E731
    rng = np.random.default_rng(seed)
    rec = tab(w.rec_pos[0])
    shots = []
    for k in range(nshot):
        n = nt - 3 * (k % 5)  # uneven records and spreads
        r = rec[k % 3:nrec - k % 4]
        dobs = np.asfortranarray(rng.standard_normal((n, r.shape[0])).astype(np.float32))
        shots.append(dict(s=w.wavelet(n), nt=n, src=tab(w.src_pos)[k], rec=r, dobs=dobs, mu=w.mu,
                          maxiter=1, rtol=0.0, band=w.band))
    return w, tab(w.datum_pos), shots


def run(pkg, w, datum, shots, **opt):
    with pkg.Handle(0, preset="mixed", **opt) as h:
        h.set_model(w.c0, w.npml, w.h, w.dt, w.ofs)
        h.set_datum(datum)
        out = h.shots(shots)
        fwd = h.submodeling_shots(shots)
        return out, fwd, h.timing()


# n1, n2, npml, steps, shots, shots a launch holds (0: the split kernels): CTAs of one to three
# row blocks and 4 to 27 columns; a last launch with fewer shots, a batch in one launch, as many
# shots as a launch takes, and the many short records of small grids
@pytest.mark.parametrize("n1,n2,npml,nt,nshot,together", [
    (151, 461, 20, 400, 16, 4), (151, 461, 20, 90, 2, 2), (77, 201, 20, 300, 16, 16),
    (301, 703, 25, 90, 5, 5), (60, 90, 20, 60, 64, 0), (151, 461, 20, 40, 64, 0)])
@pytest.mark.parametrize("history", [0, 1])
def test_batches(pkg, n1, n2, npml, nt, nshot, together, history):
    c = batch(pkg, n1, n2, npml, nt, 13, nshot)
    out, fwd, tim = run(pkg, *c, history=history)
    ref, rfwd, rtim = run(pkg, *c, history=history, pdl=1)
    assert rtim["kernel_family"] == [0] * 4
    assert tim["kernel_family"] == ([2] * 4 if together else [0] * 4)
    if together:
        assert min(tim["shots_per_launch"]) >= together
    for a, b in zip(out, ref):
        assert np.abs(b["deltade"]).max() > 0
        for k in KEYS:
            assert np.array_equal(a[k], b[k]), k
    for a, b in zip(fwd, rfwd):
        assert np.array_equal(a, b)
