"""The bench's roofline counts the bytes of the kernels that ran (CPU only): on chip the
fields are not moved, and the committed traffic capture belongs to the separate kernels
on its own grid."""
import importlib.util
import os
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("daw_bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def timing(family):
    return dict(shot_steps_a=100, shot_steps_b=100, sim_a_ms=1.1, sim_b_ms=0.9, steps_a=100,
                steps_b=100, kernel_family=[family] * 4)


@pytest.mark.parametrize("fp16", [True, False])
def test_on_chip_loops_move_the_histories(bench, fp16):
    w = SimpleNamespace(n1=751, n2=2301, npml=40)
    r = bench.roofline(timing(2), w, fp16=fp16)
    assert r["bytes_per_shot_step"] == 3 * (2 if fp16 else 4) * 751 * 2301
    assert abs(r["achieved"] - r["bytes_per_shot_step"] / 1e-5 / 1e9) < 1e-6 * r["achieved"]
    assert r["frac"] < 0.5 and r["bound"] != "hbm" and r["traffic"] is None
    ne = 831 * 2381
    d = bench.roofline(timing(2), w, rho=True)
    assert d["bytes_per_shot_step"] == 6 * 751 * 2301 + 8 * ne + 2 * 751 * 2301


@pytest.mark.parametrize("family", [0, 1])
def test_global_memory_kernels_move_the_fields(bench, family):
    w = SimpleNamespace(n1=751, n2=2301, npml=40)
    r = bench.roofline(timing(family), w)
    assert r["bytes_per_shot_step"] == 36 * 831 * 2381 + 6 * 751 * 2301 and r["bound"] == "hbm"
    assert (r["traffic"] is not None) == (family == 0)
    big = bench.roofline(timing(family), SimpleNamespace(n1=2001, n2=8001, npml=50))
    assert big["traffic"] is None
