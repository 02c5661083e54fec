"""Which kernels a plan's sweeps run on, as sck_plan_path reports it (host only): every system with a compile-time
bond table names the table and the kernels that run it, and what is switched off or falls outside says generic."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from spin_colour_kernel_b200 import _lib as L
from spin_colour_kernel_b200 import crystals as cr
from spin_colour_kernel_b200 import plan as P
from spin_colour_kernel_b200 import system as sy
from spin_colour_kernel_b200.sampler import Sampler

SQUARE, TRIANGULAR, SC, BCC, BCC12, FCC = range(1, 7)      # lattices.h
RESIDENT = 200 << 10


@pytest.fixture(scope="module", autouse=True)
def _built():
    from spin_colour_kernel_b200 import build
    build.build()


def plan_of(s, batch, mode, classes=None):
    """A Sampler's host half: its plan, tune and path, without a GPU."""
    A = object.__new__(Sampler)
    A._plan, A.B, A.mode, A.quad = None, batch, mode, mode == L.MODE_QUAD
    A.desc = P.describe(s)
    if classes is not None:
        A.desc.n_classes = len(classes)
        for i, (c, a) in enumerate(classes):
            A.desc.classes[i][0], A.desc.classes[i][1] = c, a
    h = ctypes.c_void_p()
    L.check(L.lib().sck_plan_create(ctypes.byref(A.desc), batch, mode, ctypes.byref(h)))
    A._plan = h
    return A


def _box(crystal, box, n=1, shells=(1,), **kw):
    c = cr.make(crystal, shells)
    return sy.System(crystal, n, c, box, kw.pop("per", (True,) * c.D), {s: 1.0 for s in shells}, **kw)


@pytest.mark.parametrize("mode", [L.MODE_PACKED, L.MODE_BITWISE, L.MODE_BITWISE_INDEP])
def test_word_plans_name_their_table(mode):
    for crystal, table in (("square", SQUARE), ("triangular", TRIANGULAR), ("sc", SC), ("bcc", BCC), ("fcc", FCC)):
        A = plan_of(sy.ising(crystal, 6), 64, mode)
        assert A.path()["specialised"] == 500 + table, crystal
        assert A.tune(False)["specialised"] == 0
        assert A.tune(True)["specialised"] == 500 + table
    A = plan_of(_box("sc", (6, 6, 6), per=(False,) * 3), 64, mode)
    assert A.path()["specialised"] == 0


def test_resident_plans_name_their_kernel():
    dmi = {0: np.array([[0, .3, 0], [-.3, 0, .1], [0, -.1, 0]])}
    for s, mode, want in ((sy.nanodot(6.0, 3), L.MODE_F32, 700 + SC), (sy.ising("square", 32), L.MODE_INT8, 700 + SQUARE),
                          (_box("square", (40, 30), 3, extra=dmi), L.MODE_F32, 700 + SQUARE),
                          (sy.ising("fcc", 6), L.MODE_F32, 700 + FCC),
                          (sy.ising("square", 400), L.MODE_INT8, 600 + SQUARE),       # 160 KB: no room for lists
                          (sy.heisenberg("sc", 24), L.MODE_F32, 600 + SC)):
        A = plan_of(s, 8, mode)
        assert A.path()["resident"] and A.path()["specialised"] == want, (s.name, A.path())
        assert A.tune(False)["specialised"] == 0 and A.path()["resident"]


def test_class_plans_name_their_kernel():
    A = plan_of(sy.ising("sc", 64), 100, L.MODE_INT8)
    assert A.path()["specialised"] == 800 + SC and not A.path()["resident"]
    assert plan_of(sy.ising("sc", 62), 100, L.MODE_INT8).path()["specialised"] == 100 + SC     # rows of 15.5 words
    assert plan_of(sy.ising("triangular", 510), 100, L.MODE_INT8).path()["specialised"] == 100 + TRIANGULAR
    assert plan_of(sy.ising("sc", 64), 100, L.MODE_F32).path()["specialised"] == 100 + SC
    assert plan_of(sy.heisenberg("bcc", 32), 64, L.MODE_F32).path()["specialised"] == 100 + BCC
    assert plan_of(sy.heisenberg("bcc", 32), 64, L.MODE_QUAD).path()["specialised"] == 400 + BCC


def test_a_class_named_twice_keeps_off_the_neighbour_lists():
    """A list takes a slot per entry of every class: with a class named twice there are more slots than sites."""
    s = sy.ising("square", 32)
    red, black = P.sweep_classes(s)
    assert plan_of(s, 8, L.MODE_INT8, [red, black]).path()["specialised"] == 700 + SQUARE
    assert plan_of(s, 8, L.MODE_INT8, [black]).path()["specialised"] == 700 + SQUARE       # a part of the sites
    for order in ([red, black, red], [black, black]):
        assert plan_of(s, 8, L.MODE_INT8, order).path()["specialised"] == 600 + SQUARE


@pytest.mark.parametrize("name", ["packed", "bitwise", "nanodot", "resident", "march", "vector", "open"])
def test_autotuner_times_the_kernels_the_plan_would_run(name):
    """Every path a plan takes untuned is among the candidates, told apart from the generic one, so tuning can not
    leave a sampler on slower kernels than it started with."""
    from spin_colour_kernel_b200 import autotune as at
    A = {"packed": lambda: plan_of(sy.ising("sc", 64), 128, L.MODE_PACKED),
         "bitwise": lambda: plan_of(sy.ising("sc", 64), 128, L.MODE_BITWISE),
         "nanodot": lambda: plan_of(sy.nanodot(6.0, 3), 8, L.MODE_F32),
         "resident": lambda: plan_of(sy.ising("square", 32), 32, L.MODE_INT8),
         "march": lambda: plan_of(sy.ising("sc", 64), 100, L.MODE_INT8),
         "vector": lambda: plan_of(sy.heisenberg("bcc", 32), 8, L.MODE_F32),      # below every budget
         "open": lambda: plan_of(_box("sc", (70, 70, 70), per=(False,) * 3), 8, L.MODE_INT8)}[name]()
    before = A.path()
    paths = [A.tune(*c) for c in at.candidates(A)]
    assert before in paths
    assert (before["specialised"] > 0) and any(p["specialised"] == 0 for p in paths)
    sig = {(p["specialised"], p["group"], p["resident"]) for p in paths}          # what the autotuner tells apart
    assert len(sig) >= 2
    A.tune(*at.candidates(A)[0])


def test_marching_kernel_takes_full_blocks_and_enough_walks():
    """Long narrow boxes leave its threads idle and few short walks leave the GPU idle: both stay on the class kernel."""
    for crystal, box, B, kind in (("square", (4, 60000), 100, 1), ("square", (256, 1024), 100, 1),
                                  ("square", (500, 500), 33, 8), ("square", (1024, 256), 8, 8), ("sc", (16, 4, 4000), 33, 1),
                                  ("sc", (64, 64, 64), 1, 1), ("sc", (64, 64, 64), 3, 1), ("sc", (64, 64, 64), 4, 8),
                                  ("sc", (96, 96, 96), 1, 8), ("sc", (32, 32, 256), 100, 8),
                                  ("square", (512, 512), 2, 1), ("square", (512, 512), 3, 8)):
        A = plan_of(_box(crystal, box), B, L.MODE_INT8)
        assert A.path()["specialised"] // 100 == kind, (box, B, A.path())
