"""Resident sweeps on lattice tables (csrc/resident.cu) and the int8 / float32 Ising class kernel (csrc/fast_sweep.cu)
against the generic kernels, which share their arithmetic: the chains are equal bit for bit. Boxes whose class has
fewer sites than a block, more than a block, and a remainder; masks, open axes, extra matrices, fields, anisotropy,
both acceptance rules; calls with and without neighbour lists, a replica shared by two blocks (the large nanodot),
more sweeps than a block's keys; replica counts that leave a replica over."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from spin_colour_kernel_b200 import crystals as cr
from spin_colour_kernel_b200 import system as sy
from spin_colour_kernel_b200.sampler import Sampler

pytestmark = pytest.mark.gpu


def _sys(n, crystal, box, per=None, shells=(1,), J=None, mask=False, **kw):
    c = cr.make(crystal, shells)
    m = None
    if mask:
        shape = (c.b, box[2] if c.D == 3 else 1, box[1], box[0])
        m = np.random.default_rng(5).random(shape) < 0.8
    return sy.System(f"{crystal} n={n}", n, c, box, per or (True,) * c.D, J or {s: 1.0 for s in shells}, mask=m, **kw)


RESIDENT = {
    "nanodot": lambda: sy.nanodot(6.0, 3),
    "nanodot-large": lambda: sy.nanodot(18.3, 5),
    "ising-square": lambda: _sys(1, "square", (32, 32)),
    "ising-sc-open": lambda: _sys(1, "sc", (7, 6, 5), (False,) * 3, mask=True, h=(0.3,), acceptance="barker"),
    "ising-fcc": lambda: _sys(1, "fcc", (6, 5, 7)),
    "ising-bcc-j1j2": lambda: _sys(1, "bcc", (8, 6, 4), shells=(1, 2), J={1: 1.0, 2: -0.4}),
    "xy-triangular": lambda: _sys(2, "triangular", (33, 27), h=(0.1, 0.0)),
    "heisenberg-bcc": lambda: _sys(3, "bcc", (9, 8, 7), acceptance="barker"),
    "heisenberg-dmi": lambda: _sys(3, "square", (40, 30), extra={0: np.array([[0, .3, 0], [-.3, 0, .1], [0, -.1, 0]])}),
}


@pytest.mark.parametrize("name", sorted(RESIDENT))
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("sweeps", [2, 35])
def test_resident_lattice_kernels_equal_the_generic_one(name, f32, sweeps):
    s = RESIDENT[name]()
    if s.n > 1 and not f32:
        pytest.skip("int8 holds Ising spins")
    B = 5
    kw = dict(packed=False, spin_dtype=torch.float32 if f32 else torch.int8) if s.n == 1 else {}
    A, G = (Sampler(s, B, device="cuda", seed=9, **kw) for _ in range(2))
    G.tune(False)
    assert A.path()["resident"] and G.path()["resident"]
    S = A.init_spins(seed=2)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(0.4, 3.0, B))
        X.sweep(Y, sweeps)
    assert torch.equal(A.state, G.state)
    assert torch.equal(S, S2)


MARCH = {   # the marching kernel's boxes: words of a row below, at and above a block, chunks with a remainder
    "march-square": lambda: _sys(1, "square", (36, 54), h=(0.2,)),
    "march-square-wide": lambda: _sys(1, "square", (1040, 10), acceptance="barker"),
    "march-sc": lambda: _sys(1, "sc", (8, 4, 18)),
    "march-sc-large": lambda: _sys(1, "sc", (64, 34, 20), J={1: -1.0}, acceptance="barker"),
    "march-sc-thin": lambda: _sys(1, "sc", (4, 2, 2), h=(-0.4,)),
}


@pytest.mark.parametrize("name", ["ising-square", "ising-sc-open", "ising-fcc", "ising-bcc-j1j2"] + sorted(MARCH))
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("B", [1, 7, 300])
def test_ising_class_kernel_equals_the_generic_one(name, f32, B):
    s = {**RESIDENT, **MARCH}[name]()
    kw = dict(packed=False, spin_dtype=torch.float32 if f32 else torch.int8)
    A, G = (Sampler(s, B, device="cuda", seed=3, **kw) for _ in range(2))
    A.tune(True, 0, 0)
    G.tune(False, 0, 0)
    S = A.init_spins(seed=2)
    if B == 7:                       # any value counts by its sign; a zero spin stays zero
        S = torch.randint(-127, 128, S.shape, generator=torch.Generator().manual_seed(1)).to(S)
        S = S * (A.mask != 0)
        S = S.to(A.spin_dtype)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(1.5, 6.0, B))
        X.sweep(Y, 2)
    assert torch.equal(S, S2)


@pytest.mark.parametrize("name", ["ising-square", "xy-triangular"])
@pytest.mark.parametrize("order", [(0, 1, 0), (1, 1), (1,)])
def test_repeated_and_partial_class_lists(name, order):
    """A sweep order given through the C ABI may name a class twice or leave one out."""
    import ctypes

    from spin_colour_kernel_b200 import _lib as L
    s = RESIDENT[name]()
    B = 5
    kw = dict(packed=False) if s.n == 1 else {}
    A, G = (Sampler(s, B, device="cuda", seed=9, **kw) for _ in range(2))
    for X in (A, G):
        for i, k in enumerate(order):
            X.desc.classes[i][0], X.desc.classes[i][1] = X.classes[k]
        X.desc.n_classes = len(order)
        h = ctypes.c_void_p()
        L.check(L.lib().sck_plan_create(ctypes.byref(X.desc), B, X.mode, ctypes.byref(h)))
        L.lib().sck_plan_destroy(X._plan)
        X._plan = h
    G.tune(False)
    assert A.path()["specialised"] // 100 == (7 if len(set(order)) == len(order) else 6)
    S = A.init_spins(seed=2)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(0.4, 3.0, B))
        X.sweep(Y, 10)
    assert torch.equal(S, S2)


# boxes and replica counts the marching kernel takes: rows of words at half a block, over one block, nearly full
# blocks; walks with a remainder, of one chunk, and two layers thick
MARCHING = {
    "square": (lambda: _sys(1, "square", (512, 20), h=(0.2,)), 70),
    "square-wide": (lambda: _sys(1, "square", (1040, 10), acceptance="barker"), 60),
    "square-long": (lambda: _sys(1, "square", (448, 270)), 7),
    "sc": (lambda: _sys(1, "sc", (16, 32, 18)), 71),
    "sc-blocks": (lambda: _sys(1, "sc", (64, 34, 20), J={1: -1.0}, acceptance="barker"), 33),
    "sc-thin": (lambda: _sys(1, "sc", (4, 112, 2), h=(-0.4,)), 240),
}


@pytest.mark.parametrize("name", sorted(MARCHING))
@pytest.mark.parametrize("values", ["spins", "any"])
def test_marching_kernel_equals_the_generic_one(name, values):
    build, B = MARCHING[name]
    s = build()
    A, G = (Sampler(s, B, device="cuda", seed=3, packed=False) for _ in range(2))
    assert A.tune(True, 0, 0)["specialised"] // 100 == 8
    G.tune(False, 0, 0)
    S = A.init_spins(seed=2)
    if values == "any":              # any value counts by its sign; a zero spin stays zero
        S = torch.randint(-127, 128, S.shape, generator=torch.Generator().manual_seed(1)).to(S)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(1.5, 6.0, B))
        X.sweep(Y, 3)
    assert torch.equal(S, S2)


def test_the_cases_above_run_on_the_kernels_they_are_for():
    """Kind 7: lattice tables with neighbour lists; kind 1: the class kernel of boxes the marching kernel leaves."""
    for name, build in RESIDENT.items():
        s = build()
        kw = dict(packed=False) if s.n == 1 else {}
        A = Sampler(s, 5, device="cuda", **kw)
        assert A.path()["specialised"] // 100 == 7, name
        assert A.tune(False)["specialised"] == 0
    for name in ["ising-square", "ising-sc-open", "ising-fcc", "ising-bcc-j1j2"]:
        A = Sampler(RESIDENT[name](), 300, device="cuda", packed=False)
        assert A.tune(True, 0, 0)["specialised"] // 100 == 1, name
