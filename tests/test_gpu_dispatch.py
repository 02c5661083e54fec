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


# A block of the packed kernel takes a whole word where class blocks x words reach 592, half a word from 296: boxes of
# 384 (sc), 300 (bcc) and 188 (fcc) blocks a class, the last word full, partial, and partial in a single word; counts
# of six neighbours (own spin in the fourth plane) and of eight and twelve.
@pytest.mark.parametrize("crystal,box,B", [("sc", (64, 64, 48), 50), ("sc", (64, 64, 48), 20), ("bcc", (80, 80, 12), 64),
                                           ("bcc", (80, 80, 12), 31), ("fcc", (40, 40, 30), 101), ("fcc", (40, 40, 30), 50)])
@pytest.mark.parametrize("acceptance", ["metropolis", "barker"])
def test_packed_words_by_whole_and_half_words(crystal, box, B, acceptance):
    s = _sys(1, crystal, box, h=(0.2,) if B % 2 else None, acceptance=acceptance)
    A, G = (Sampler(s, B, device="cuda", seed=17, packed=True) for _ in range(2))
    G.tune(False)
    S = _words(A, 3)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(1.5, 7.0, B))
        X.sweep(Y, 2)
    assert torch.equal(S, S2)


# Several units (groups of four words, or words) a block: 384 blocks a class leave 4 grid rows for 5 groups or 19 words.
@pytest.mark.parametrize("independent", [False, True])
@pytest.mark.parametrize("h,acceptance", [(0.0, "metropolis"), (0.1, "metropolis"), (0.1, "barker")])
def test_bitwise_words_with_several_units_a_block(independent, h, acceptance):
    B = 600
    s = _sys(1, "sc", (64, 64, 48), h=(h,) if h else None, acceptance=acceptance)
    A, G = (Sampler(s, B, device="cuda", seed=5, bitwise=True, independent=independent) for _ in range(2))
    G.tune(False)
    S = _words(A, 4)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(_word_temperatures(B))
        X.sweep(Y, 2)
    assert torch.equal(S, S2)


def test_column_observables_with_fewer_blocks_than_items():
    """24 items a word for 19 blocks, and for the 4 that the scratch of the call without a workspace holds."""
    B = 4096
    s = _sys(1, "bcc", (64, 48, 9), h=(0.3,))
    A = Sampler(s, B, device="cuda", seed=1, packed=True)
    S = _words(A, 6)
    buf = A._buffers(S)

    def call(fn, *ws):
        E = torch.full((B,), np.nan, dtype=torch.float64, device="cuda")
        M = torch.full((B, s.b, 1), np.nan, dtype=torch.float64, device="cuda")
        L.check(fn(A._plan, ctypes.byref(buf), S.data_ptr(), L.MODE_PACKED, B, E.data_ptr(), M.data_ptr(), *ws, A._stream()))
        return E, M
    lib = L.lib()
    E1, M1 = call(lib.sck_observables, A._workspace(B).data_ptr())
    E2, M2 = call(lib.sck_observables_noalloc)
    A.tune(False)
    E3, M3 = call(lib.sck_observables, A._workspace(B).data_ptr())
    for E, M in ((E2, M2), (E3, M3)):          # sums of +-1 and +-J: exact but for the field's rounding
        torch.testing.assert_close(E, E1, rtol=0, atol=1e-8)
        assert torch.equal(M, M1)


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


# States just above 96 MB, whose interleaved class launches prefetch the rows of later blocks: the cubic tiles, rows of
# two residues and of one, with a last quad that is not full; in the reference layout, units of four replica pairs with a
# remainder.
@pytest.mark.parametrize("n,crystal,box,B", [(3, "sc", (64, 64, 64), 35), (3, "bcc", (33, 34, 35), 105),
                                             (2, "square", (512, 512), 49), (3, "sc", (62, 60, 58), 37)])
def test_prefetching_interleaved_launches_and_pair_units_agree(n, crystal, box, B):
    s = _sys(n, crystal, box)
    Q, R = (Sampler(s, B, device="cuda", seed=4, layout=layout) for layout in ("quad", "reference"))
    R.tune(True, 0, 0)
    assert -(-B // 4) * 16 * n * s.nsite > 96 << 20
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((B, n) + s.shape, generator=g, device="cuda")
    x /= x.norm(dim=1, keepdim=True)
    X = Q.pack(x)
    for A, Y in ((Q, X), (R, x)):
        A.set_temperature(torch.linspace(0.5, 2.5, B))
        A.sweep(Y, 2)
    assert torch.equal(Q.unpack(X), x)


# Replicas a thread of the int8 / float32 class kernel keeps: two at 41 replicas of 118 blocks, eight at 163; the last
# thread row has one and three.
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("B", [41, 163])
def test_ising_class_kernel_with_an_odd_tail_of_replicas(f32, B):
    s = _sys(1, "triangular", (300, 300), h=(0.1,))
    kw = dict(packed=False, spin_dtype=torch.float32 if f32 else torch.int8)
    A, G = (Sampler(s, B, device="cuda", seed=6, **kw) for _ in range(2))
    assert A.tune(True, 0, 0)["specialised"] // 100 == 1
    G.tune(False, 0, 0)
    S = A.init_spins(seed=2)
    S2 = S.clone()
    for X, Y in ((A, S), (G, S2)):
        X.set_temperature(torch.linspace(1.0, 5.0, B))
        X.sweep(Y, 2)
    assert torch.equal(S, S2)


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


@pytest.mark.parametrize("B", [21, 47])
def test_interleaved_cube_of_four_classes_with_and_without_prefetch(B):
    """The 64^3 cube of the J1-J2 lattice prefetches from 272 MB of state on: 151 MB and 302 MB, the last quad short."""
    from spin_colour_kernel_b200 import workloads as wl
    s = wl.heisenberg_bcc(64)
    Q, R = (Sampler(s, B, device="cuda", seed=4, layout=layout) for layout in ("quad", "reference"))
    R.tune(True, 0, 0)
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((B, 3) + s.shape, generator=g, device="cuda")
    x /= x.norm(dim=1, keepdim=True)
    X = Q.pack(x)
    for A, Y in ((Q, X), (R, x)):
        A.set_temperature(torch.linspace(0.5, 2.5, B))
        A.sweep(Y, 1)
    assert torch.equal(Q.unpack(X), x)
