"""The word kernels of lattices with a compile-time bond table (csrc/words.cu) against the oracle, bit for bit, and
their FP64 observables: box edges that leave part of a block of 256 class sites unused and several blocks a class,
one word, words that do not fill a group of four, and a last word that is not full; with and without a field, both
acceptance rules; and the kernels of other systems, which the same sampler runs with the specialised kernels off."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import bitwise as obw
from oracle import observables as oob
from oracle import sweep as osw
from spin_colour_kernel_b200 import crystals as cr
from spin_colour_kernel_b200 import system as sy
from spin_colour_kernel_b200.sampler import Sampler

pytestmark = pytest.mark.gpu

SYSTEMS = {"square": ("square", (34, 18)), "triangular": ("triangular", (33, 27)), "sc": ("sc", (10, 8, 14)),
           "sc-odd": ("sc", (9, 15, 3)), "bcc": ("bcc", (7, 9, 8)), "fcc": ("fcc", (6, 5, 7)),
           "square-thin": ("square", (512, 2))}


def _system(name, h, acceptance):
    crystal, box = SYSTEMS[name]
    c = cr.make(crystal)
    return sy.System(f"Ising {crystal}", 1, c, box, (True,) * c.D, {1: 1.0}, h=(h,) if h else None,
                     acceptance=acceptance)


@pytest.mark.parametrize("mode", ["packed", "bitwise", "independent"])
@pytest.mark.parametrize("name,B,h,acceptance", [
    ("square", 33, 0.0, "metropolis"), ("triangular", 160, 0.1, "barker"), ("sc", 260, 0.0, "metropolis"),
    ("sc-odd", 32, -0.3, "metropolis"), ("bcc", 70, 0.2, "barker"), ("fcc", 130, 0.0, "barker"),
    ("square-thin", 64, 0.1, "metropolis")])
def test_word_kernels_match_the_oracle(name, B, h, acceptance, mode):
    s = _system(name, h, acceptance)
    kw = {"packed": dict(packed=True), "bitwise": dict(bitwise=True),
          "independent": dict(bitwise=True, independent=True)}[mode]
    A, G = (Sampler(s, B, device="cuda", seed=17, **kw) for _ in range(2))
    G.tune(False)
    W = -(-B // 32)
    T = torch.linspace(1.5, 7.0, W).repeat_interleave(32)[:B] if mode != "packed" else torch.linspace(1.5, 7.0, B)
    S = A.init_spins(seed=4)
    S2 = S.clone()
    x = A.unpack(S).cpu().numpy()
    for X in (A, G):
        X.set_temperature(T)
    E, M = A.sweep_measure(S, 2)
    E2, M2 = G.sweep_measure(S2, 2)
    assert torch.equal(S, S2)
    beta = (np.float32(1.0) / T.numpy().astype(np.float32)).astype(np.float32)
    if mode == "packed":
        want = x.copy()
        osw.sweep(s, want, beta, [17, 0], 2)
    else:
        words = torch.cat([T, T[-1:].expand(32 * W - B)]).numpy().reshape(W, 32)[:, 0].astype(np.float32)
        wb = (np.float32(1.0) / words).astype(np.float64)
        table = obw.p_fixed(s, wb) if mode == "independent" else obw.p_table(s, wb)
        want = x[:, 0]
        for sw in range(2):
            want = obw.sweep(s, want, table, 17, sw, independent=mode == "independent")
        want = want[:, None]
    got = A.unpack(S).cpu().numpy()
    assert np.array_equal(got, want)
    # sums of +-1 and of +-J: exact in FP64 up to the field's rounding (some 1e4 sites, |h| < 1)
    np.testing.assert_allclose(E.cpu().numpy(), oob.energy(s, got), rtol=0, atol=1e-9)
    assert np.array_equal(M.cpu().numpy(), oob.magnetization(got))
    np.testing.assert_allclose(E2.cpu().numpy(), E.cpu().numpy(), rtol=0, atol=1e-9)
    assert torch.equal(M, M2)


def test_autotuning_words_times_the_word_kernels(tmp_path, monkeypatch):
    """The autotuner tells the word kernels from the generic ones, and what it applies continues the same chain."""
    from spin_colour_kernel_b200 import autotune as at
    monkeypatch.setenv("SCK_TUNE_CACHE", str(tmp_path / "tune.json"))
    s = _system("sc", 0.0, "metropolis")
    A, R = (Sampler(s, 70, device="cuda", seed=3, packed=True) for _ in range(2))
    for X in (A, R):
        X.set_temperature(torch.linspace(1.5, 7.0, 70))
    S = A.init_spins(seed=4)
    S2 = S.clone()
    c = at.autotune(A, S, sweeps=2)
    assert {t["specialised"] // 100 for t in c["tried"]} == {0, 5} and int(A.state[1]) == 0
    A.sweep(S, 3)
    R.sweep(S2, 3)
    assert torch.equal(S, S2)


def test_the_systems_above_run_on_the_word_kernels():
    for name in SYSTEMS:
        for kw in (dict(packed=True), dict(bitwise=True), dict(bitwise=True, independent=True)):
            A = Sampler(_system(name, 0.0, "metropolis"), 64, device="cuda", **kw)
            assert A.path()["specialised"] // 100 == 5, name
            assert A.tune(False)["specialised"] == 0
