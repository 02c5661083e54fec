"""Kernel variants that only larger launches, odd tails or certain sizes select, each against a path of its own: the
generic kernels (bit for bit where the arithmetic is shared), the interleaved layout, the systems of a batch swept on
their own, or the oracle. Sizes are the smallest that reach the variant, given beside each case."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import cases as C
from oracle import observables as oob
from spin_colour_kernel_b200 import _lib as L
from spin_colour_kernel_b200 import crystals as cr
from spin_colour_kernel_b200 import system as sy
from spin_colour_kernel_b200.sampler import Sampler, SamplerBatch

pytestmark = pytest.mark.gpu


def _sys(n, crystal, box, **kw):
    c = cr.make(crystal)
    return sy.System(f"{crystal} n={n}", n, c, box, (True,) * c.D, {1: 1.0}, **kw)


def _words(A, seed):
    """Random words: every replica's spins +-1 with equal probability."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (A.W, 1) + A.sys.shape
    return torch.randint(-2 ** 31, 2 ** 31, shape, generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _word_temperatures(B):
    W = -(-B // 32)
    return torch.linspace(1.5, 7.0, W).repeat_interleave(32)[:B]


@pytest.mark.parametrize("B", [33, 160])
def test_fcc_word_observables_on_both_kernels(B):
    """840 sites: two words stay on the generic kernel, five take the columns."""
    s = _sys(1, "fcc", (6, 5, 7), h=(0.1,))
    A = Sampler(s, B, device="cuda", seed=2, packed=True)
    S = A.init_spins(seed=3)
    E, M = A.observables(S)
    x = A.unpack(S).cpu().numpy()
    np.testing.assert_allclose(E.cpu().numpy(), oob.energy(s, x), rtol=0, atol=1e-9)
    assert np.array_equal(M.cpu().numpy(), oob.magnetization(x))


# Class launches of 64, 512 and 768 blocks (alone on half the SMs; too few to overlap; overlapping), captured: a replay
# continues the chain of plain calls.
DEPENDENT = {
    "vector-64": (lambda: _sys(2, "square", (180, 180)), 2, {}),
    "vector-512": (lambda: _sys(2, "square", (180, 180)), 16, {}),
    "vector-768": (lambda: _sys(2, "square", (180, 180)), 24, {}),
    "heisenberg": (lambda: sy.heisenberg("bcc", 24), 33, {}),
    "int8": (lambda: _sys(1, "triangular", (300, 300)), 5, dict(packed=False)),
    "packed": (lambda: _sys(1, "sc", (32, 32, 32)), 70, dict(packed=True)),
    "bitwise": (lambda: _sys(1, "sc", (32, 32, 32)), 70, dict(bitwise=True)),
    "independent": (lambda: _sys(1, "triangular", (60, 60)), 70, dict(bitwise=True, independent=True)),
}


@pytest.mark.parametrize("name", sorted(DEPENDENT))
def test_captured_class_launches_continue_the_chain(name):
    build, B, kw = DEPENDENT[name]
    s = build()
    A, R = (Sampler(s, B, device="cuda", seed=8, **kw) for _ in range(2))
    for X in (A, R):
        X.tune(True, 0, 0)
        X.set_temperature(_word_temperatures(B) if X.bitwise else torch.linspace(0.5, 4.0, B))
    S = A.init_spins(seed=2)
    S2 = S.clone()
    replay = A.graph(S, 3)                     # one sweep before the capture
    for _ in range(2):
        replay()
    R.sweep(S2, 7)
    torch.cuda.synchronize()
    assert int(A.state[1]) == int(R.state[1]) == 7
    assert torch.equal(S, S2)
    if s.n == 1:                               # and the generic kernels', which launch without overlap
        G = Sampler(s, B, device="cuda", seed=8, **kw)
        G.tune(False, 0, 0)
        G.set_temperature(_word_temperatures(B) if G.bitwise else torch.linspace(0.5, 4.0, B))
        S3 = G.init_spins(seed=2)
        G.sweep(S3, 7)
        assert torch.equal(S, S3)


def _batch(systems, B):
    A, R = ([Sampler(s, B, device="cuda", seed=20 + i) for i, s in enumerate(systems)] for _ in range(2))
    for X in A + R:
        X.set_temperature(torch.linspace(0.4, 1.6, B))
    S = [X.init_spins(seed=i) for i, X in enumerate(A)]
    return A, R, S, [x.clone() for x in S]


# Streaming items of several replica pairs: classes that fill their items (64^2 and up), shorter ones beside them, and
# replica counts that leave an item with one replica, with three, and with a pair.
@pytest.mark.parametrize("B", [9, 11, 18])
def test_batch_items_of_several_pairs(B):
    systems = [_sys(2, "square", (64, 64)), _sys(2, "triangular", (90, 84)), _sys(2, "sc", (18, 16, 20)),
               _sys(2, "square", (24, 20)), sy.xy("square", 100)]
    A, R, S, S2 = _batch(systems, B)
    b = SamplerBatch(A, S, resident_limit=0)
    b.sweep(3)
    b.check_waits()
    for X, Y, Z in zip(R, S2, S):
        C.batch_twin_tune(X, 0)
        X.sweep(Y, 3)
        assert torch.equal(Y, Z), X.sys.name


# Items per class of one system alone: a class that fills items shares them out among four pairs, one that does not keeps
# an item per pair (256 sites: 1 run), unless its items grow by at most an eighth (1,728 sites: 7 runs) or items abound.
@pytest.mark.parametrize("box,systems,B,items", [((16, 16), 8, 8, 4), ((24, 24), 1, 32, 16), ((64, 64), 1, 32, 16),
                                                 ((16, 16), 80, 32, 4), ((58, 58), 1, 32, 16)])
def test_batch_items_follow_the_length_of_a_class(box, systems, B, items):
    ss = [_sys(2, "square", box) for _ in range(systems)]
    A, R, S, S2 = _batch(ss, B)
    b = SamplerBatch(A, S, resident_limit=0)
    assert b.info()["step_blocks"] == 2 * systems * items
    b.sweep(2)
    X, Y = R[-1], S2[-1]
    C.batch_twin_tune(X, 0)
    X.sweep(Y, 2)
    assert torch.equal(Y, S[-1])


@pytest.mark.parametrize("Rd,layers,B", [(6.0, 3, 200), (10.0, 3, 150), (18.3, 5, 148), (18.3, 5, 200), (18.3, 5, 900)])
def test_topological_charge_of_any_block_size(Rd, layers, B):
    """Blocks of 256, 512 and 1,024 threads give the charges that single replicas (as many threads as a layer has
    plaquettes, at most 1,024) give, up to the order of an FP64 sum of at most 3,000 terms below 4 pi."""
    s = sy.nanodot(Rd=Rd, L=layers)
    A, R = Sampler(s, B, device="cuda", seed=1), Sampler(s, 1, device="cuda", seed=1)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((B, 3) + s.shape, generator=g, device="cuda")
    x = (x / x.norm(dim=1, keepdim=True) * torch.as_tensor(s.site_mask(), device="cuda")).contiguous()
    Q = A.topological_charge(x, 1)
    for r in (0, B // 2, B - 1):
        q = R.topological_charge(x[r:r + 1].contiguous(), 1)
        assert abs(float(Q[r]) - float(q[0])) < 3000 * 4 * np.pi * 2.0 ** -52
    assert float(Q.abs().max()) > 0
