"""What a user has this framework do, as measured cases: one call or a short run of calls through the public entry
points (`Sampler`, `SamplerBatch`, `learned.BlockProposal`) on seeded inputs.

A case is a dict of plain values; its `family` selects how it is prepared and run:

  ising     `Sampler` on an Ising system in one of its storages: int8 spins, packed words (the default from 32
            replicas on), bitwise words with shared or independent draws; a run of sweeps, with `measure` ended by
            the FP64 observables
  vector    `Sampler` on an XY or Heisenberg system, reference or interleaved ("quad") layout; sweeps, with or
            without the observables
  ragged    `SamplerBatch` over XY systems of uneven size, half of them circular masks in open boxes
  nanodisk  the cooling ladder's step on a nanodisk with DMI and surface anisotropy: sweeps, observables and the
            middle layer's topological charge
  learned   one round of learned block proposals
  train     loss and gradients of the learned proposal's network on one batch of block inputs

Every chain draws its random numbers from Philox counters fixed by seed, sweep, replica and site, so the outputs
are a function of the inputs.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from spin_colour_kernel_b200 import crystals as cr
from spin_colour_kernel_b200 import system as sy
from spin_colour_kernel_b200 import workloads as wl
from spin_colour_kernel_b200.learned import BOUNDARY, HIDDEN, IN, SPINS, BlockProposal
from spin_colour_kernel_b200.sampler import Sampler, SamplerBatch

DEVICE = "cuda"


# --------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # the smallest call: the 2D benchmark lattice, a replica small enough to stay on-chip for the whole call;
        # thermalising a small system is many of these, so latency counts
        dict(name="ising-square-int8", family="ising", crystal="square", L=32, B=32, storage="int8", sweeps=10,
             h=0.0, acceptance="metropolis", measure=False),
        # int8 Ising spins of the 3D lattice, the chain that learned block rounds are interleaved with
        dict(name="ising-sc-int8", family="ising", crystal="sc", L=64, B=256, storage="int8", sweeps=1, h=0.0,
             acceptance="metropolis", measure=False),
        # the storage an Ising sampler takes by default, with a measurement: a ladder's measure step
        dict(name="ising-sc-packed", family="ising", crystal="sc", L=64, B=128, storage="packed", sweeps=2, h=0.0,
             acceptance="metropolis", measure=True),
        # the 3D multi-spin-coded benchmark lattice, one measure step
        dict(name="ising-sc-bitwise", family="ising", crystal="sc", L=128, B=512, storage="bitwise", sweeps=1,
             h=0.0, acceptance="metropolis", measure=True),
        # multi-spin coding with independent draws per replica, in a field, a last word that is not full
        dict(name="ising-triangular-independent", family="ising", crystal="triangular", L=510, B=200,
             storage="independent", sweeps=2, h=0.1, acceptance="barker", measure=True),
        # the 3D Heisenberg benchmark: the largest state, many sweeps between measurements
        dict(name="heisenberg-bcc-quad", family="vector", crystal="bcc-j1j2", n=3, L=64, B=1536, layout="quad",
             sweeps=2, measure=False),
        # the same model at an ordinary size that is no power of two, measuring every sweep
        dict(name="heisenberg-bcc-measure", family="vector", crystal="bcc-j1j2", n=3, L=48, B=94, layout="quad",
             sweeps=1, measure=True),
        # the quick start: reference layout, a few sweeps, then the observables
        dict(name="heisenberg-bcc-reference", family="vector", crystal="bcc", n=3, L=32, B=64, layout="reference",
             sweeps=10, measure=True),
        # a ragged batch of XY systems in one call
        dict(name="xy-ragged", family="ragged", systems=24, B=32, L_max=512, sweeps=2),
        # nanodisks of the default size, the cooling ladder's step
        dict(name="nanodisk-ladder", family="nanodisk", Rd=18.3, layers=5, B=64, sweeps=10),
        # one round of learned block proposals at the benchmark's size
        dict(name="learned-round", family="learned", L=64, R=256),
        # forward and backward of the network at the training batch size
        dict(name="learned-gradients", family="train", batch=8192),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the ranges above. Periodic boxes are drawn at any length their crystal's colouring closes
    on; replica counts are drawn freely, odd ones among them."""
    family = rng.choice(["ising"] * 5 + ["vector"] * 5 + ["ragged", "nanodisk", "learned", "train"])
    if family == "ising":
        crystal = rng.choice(["square", "triangular", "sc", "sc", "bcc", "fcc"])
        storage = rng.choice(["int8", "packed", "bitwise", "independent"])
        B = _log_int(rng, 8 if storage == "int8" else 32, 512)
        h = rng.choice([0.0, 0.0, 0.1])
        acceptance = rng.choice(["metropolis", "metropolis", "barker"])
        measure = rng.random() < 0.5
        sweeps = rng.randint(1, 10)
        most = 6e8 if storage in ("bitwise", "independent") else 1e8
        L = _extent(rng, crystal, most / (B * sweeps))
        return dict(family=family, crystal=crystal, L=L, B=B, storage=storage, sweeps=sweeps, h=h,
                    acceptance=acceptance, measure=measure)
    if family == "vector":
        crystal = rng.choice(["square", "triangular", "sc", "bcc", "bcc-j1j2", "bcc-j1j2", "fcc"])
        n = 3 if crystal == "bcc-j1j2" else rng.choice([2, 3])
        B = _log_int(rng, 4, 1536)
        sweeps = rng.randint(1, 10)
        # the interleaved layout takes colourings of x-period 1 or 2, which leaves the triangular lattice out
        layout = "reference" if crystal == "triangular" else rng.choice(["reference", "quad", "quad"])
        L = _extent(rng, crystal, 2e8 / (B * sweeps))
        return dict(family=family, crystal=crystal, n=n, L=L, B=B, layout=layout, sweeps=sweeps,
                    measure=rng.random() < 0.5)
    if family == "ragged":
        return dict(family=family, systems=rng.randint(4, 32), B=_log_int(rng, 4, 32), L_max=_log_int(rng, 32, 512),
                    sweeps=rng.randint(1, 3))
    if family == "nanodisk":
        return dict(family=family, Rd=round(rng.uniform(6.0, 24.0), 1), layers=rng.randint(2, 6),
                    B=_log_int(rng, 4, 200), sweeps=rng.randint(1, 20))
    if family == "learned":
        return dict(family=family, L=8 * rng.randint(1, 8), R=_log_int(rng, 8, 256))
    return dict(family=family, batch=64 * _log_int(rng, 8, 256))


def _extent(rng, crystal: str, sites: float) -> int:
    """An edge length the crystal's colouring closes on, log-uniform up to about `sites` sites in all."""
    step = {"square": 2, "triangular": 3, "sc": 2, "bcc": 1, "bcc-j1j2": 2, "fcc": 1}[crystal]
    b = {"bcc": 2, "bcc-j1j2": 2, "fcc": 4}.get(crystal, 1)
    D = 2 if crystal in ("square", "triangular") else 3
    hi = min((sites / b) ** (1.0 / D), 1024 if D == 2 else 128)
    lo = min(18 if D == 2 else 6, hi)
    return max(6, step * int(round(_log_int(rng, lo, max(hi, lo + 1e-9)) / step)))


# -------------------------------------------------------------------------------------------------- systems
def _key(case: dict) -> tuple:
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


@functools.lru_cache(maxsize=4)
def _systems(key: tuple):
    """The systems of a case (colouring searched and verified): what a user's program defines first."""
    case = dict(key)
    fam = case["family"]
    if fam == "ising":
        c = cr.make(case["crystal"])
        return sy.System(f"Ising {case['crystal']}", 1, c, (case["L"],) * c.D, (True,) * c.D, {1: 1.0},
                         h=(case["h"],) if case["h"] else None, acceptance=case["acceptance"])
    if fam == "vector":
        if case["crystal"] == "bcc-j1j2":
            return wl.heisenberg_bcc(case["L"])
        make = sy.xy if case["n"] == 2 else sy.heisenberg
        return make(case["crystal"], case["L"])
    if fam == "ragged":
        return [(wl.xy_system(c, L, disk), T) for c, L, disk, T in
                wl.xy_ragged_specs(case["systems"], L_max=case["L_max"])]
    if fam == "nanodisk":
        return sy.nanodot(Rd=case["Rd"], L=case["layers"])
    if fam == "learned":
        return sy.ising("sc", case["L"])
    return None


def _temperatures(case: dict) -> torch.Tensor:
    """Temperatures linear across the replicas (bitwise words: across the words), around the transition."""
    lo, hi = (2.0, 6.0) if case["family"] == "ising" else (0.5, 2.5)
    B = case["B"]
    if case.get("storage") in ("bitwise", "independent"):
        W = -(-B // 32)
        return torch.linspace(lo, hi, W).repeat_interleave(32)[:B]
    return torch.linspace(lo, hi, B)


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _ising_spins(s, B: int, seed: int) -> torch.Tensor:
    return torch.randint(0, 2, (B, 1) + s.shape, device=DEVICE, generator=_generator(seed), dtype=torch.int8) * 2 - 1


def _vector_spins(s, B: int, seed: int) -> torch.Tensor:
    """Unit vectors uniform on the circle or sphere, zero on masked sites."""
    x = torch.randn((B, s.n) + s.shape, device=DEVICE, generator=_generator(seed))
    x /= x.norm(dim=1, keepdim=True)
    if s.mask is not None:
        x *= torch.as_tensor(s.site_mask(), device=DEVICE).to(torch.float32)
    return x


def _ragged_spins(s, B: int, seed: int, i: int) -> torch.Tensor:
    return _vector_spins(s, B, 1000 * seed + i)


def _block_rows(batch: int, seed: int) -> torch.Tensor:
    """Block inputs in the layout `BlockProposal.gather` returns: rows of +-1 in bfloat16, mostly aligned, as blocks
    of a lattice near the transition are."""
    g = _generator(seed)
    sign = torch.randint(0, 2, (batch, 1), device=DEVICE, generator=g) * 2 - 1
    up = torch.rand((batch, IN), device=DEVICE, generator=g) < 0.75
    return torch.where(up, sign, -sign).to(torch.bfloat16)


def prepare(case: dict, seed: int) -> dict:
    fam, s = case["family"], _systems(_key(case))
    st = {"case": case}
    if fam == "ising":
        kw = {"int8": dict(packed=False), "packed": dict(packed=True), "bitwise": dict(bitwise=True),
              "independent": dict(bitwise=True, independent=True)}[case["storage"]]
        A = Sampler(s, case["B"], device=DEVICE, seed=seed, **kw)
        A.set_temperature(_temperatures(case))
        S = _ising_spins(s, case["B"], seed)
        st.update(A=A, S=A.pack(S) if A.packed else S)
    elif fam == "vector":
        A = Sampler(s, case["B"], device=DEVICE, seed=seed, layout=case["layout"])
        A.set_temperature(_temperatures(case))
        S = _vector_spins(s, case["B"], seed)
        st.update(A=A, S=A.pack(S) if A.quad else S)
    elif fam == "ragged":
        samplers, spins = [], []
        for i, (sys_i, T) in enumerate(s):
            A = Sampler(sys_i, case["B"], device=DEVICE, seed=seed + i)
            A.set_temperature(T)
            samplers.append(A)
            spins.append(_ragged_spins(sys_i, case["B"], seed, i))
        st.update(batch=SamplerBatch(samplers, spins, resident_limit=16 << 10), spins=spins)
    elif fam == "nanodisk":
        A = Sampler(s, case["B"], device=DEVICE, seed=seed)
        A.set_temperature(_temperatures(case))
        st.update(A=A, S=_vector_spins(s, case["B"], seed))
    elif fam == "learned":
        st.update(P=BlockProposal(case["L"], case["R"], seed=seed, device=DEVICE), S=_ising_spins(s, case["R"], seed),
                  beta=torch.full((case["R"],), 1.0 / 4.5115, device=DEVICE), seed=seed, rnd=0,
                  accepted=torch.zeros(case["R"], dtype=torch.int32, device=DEVICE))
    else:
        st.update(P=BlockProposal(8, 1, seed=seed, device=DEVICE), x=_block_rows(case["batch"], seed))
    return st


def run(state: dict):
    case = state["case"]
    fam = case["family"]
    if fam in ("ising", "vector"):
        A, S = state["A"], state["S"]
        if not case["measure"]:
            return A.sweep(S, case["sweeps"])
        if fam == "vector" and case["layout"] == "reference":
            A.sweep(S, case["sweeps"])
            E, M = A.observables(S)
        else:
            E, M = A.sweep_measure(S, case["sweeps"])
        return S, E, M
    if fam == "ragged":
        state["batch"].sweep(case["sweeps"])
        return state["spins"]
    if fam == "nanodisk":
        A, S = state["A"], state["S"]
        A.sweep(S, case["sweeps"])
        E, M = A.observables(S)
        return S, E, M, A.topological_charge(S, case["layers"] // 2)
    if fam == "learned":
        state["P"].round(state["S"], state["beta"], state["seed"], state["rnd"], state["accepted"])
        state["rnd"] += 1
        return state["S"], state["accepted"]
    loss, grads = state["P"].grads(state["x"])
    return loss, grads


# ------------------------------------------------------------------------------------------ work of a pass
def _bonds_per_site(s) -> float:
    return len(s.crystal.bonds) / s.b


def _vector_flops(s, B: int) -> float:
    """Per attempt: the neighbour sums, one multiply and add per component and group, proposal, energy change and
    acceptance (about 20 operations for XY, 30 for Heisenberg, 28 more with cubic anisotropy)."""
    per = _bonds_per_site(s) * s.n + 2 * s.n * len(s.J) + 10 * s.n + (28 if s.cubic_k1 is not None else 0)
    return per * B * s.n_active


def work(case: dict) -> dict:
    """The spins read once and written once per pass, with the outputs beside them; floating-point operations of
    the updates (Ising updates are integer and logic operations: none)."""
    fam, s = case["family"], _systems(_key(case))
    if fam == "ising":
        B = case["B"]
        spins = B * s.nsite if case["storage"] == "int8" else -(-B // 32) * s.nsite * 4
        return {"bytes": 2 * spins + (16 * B if case["measure"] else 0), "flops": 0}
    if fam in ("vector", "nanodisk"):
        B = case["B"]
        out = 8 * B * (2 + s.b * s.n) if case.get("measure", True) else 0
        return {"bytes": 2 * B * s.n * s.nsite * 4 + out, "flops": _vector_flops(s, B) * case["sweeps"]}
    if fam == "ragged":
        B = case["B"]
        return {"bytes": sum(2 * B * 2 * t.nsite * 4 for t, _ in s),
                "flops": sum(_vector_flops(t, B) for t, _ in s) * case["sweeps"]}
    if fam == "learned":
        blocks = case["R"] * (case["L"] // 4) ** 3
        # the incremental form of the masked network: 110,592 multiply-adds for the proposal, as many for the
        # density of the current spins
        return {"bytes": 2 * case["R"] * s.nsite, "flops": blocks * 2 * 2 * 110592}
    params = HIDDEN * IN + 2 * HIDDEN * HIDDEN + SPINS * HIDDEN
    return {"bytes": case["batch"] * IN * 2 + params * 6, "flops": 6 * params * case["batch"]}


# --------------------------------------------------------------------------------- the same in 64-bit floats
_MASK32 = 0xFFFFFFFF


def _mul_hi_lo(a: int, x: torch.Tensor):
    """High and low 32 bits of a * x for 32-bit values held in int64 (the product wraps, its bits are right)."""
    p = x * a
    return (p >> 32) & _MASK32, p & _MASK32


def _uniforms(seed: int, sweep: int, counter: torch.Tensor):
    """The first three Philox4x32-10 uniforms of each counter under the sweep's key, exactly as the chains define
    them (float32 values), in float64."""
    v = seed * 1000003 + sweep * 7919 + 12345
    key = abs(v) % 2147483629
    key = key if v >= 0 else -key
    k0, k1 = key & _MASK32, (key >> 32) & _MASK32
    c0 = counter & _MASK32
    c1, c2, c3 = (torch.zeros_like(c0) for _ in range(3))
    for _ in range(10):
        ha, la = _mul_hi_lo(0xD2511F53, c0)
        hb, lb = _mul_hi_lo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = hb ^ c1 ^ k0, lb, ha ^ c3 ^ k1, la
        k0, k1 = (k0 + 0x9E3779B9) & _MASK32, (k1 + 0xBB67AE85) & _MASK32
    scale = float(np.array([0x2FFFFFFF], np.uint32).view(np.float32)[0])
    out = []
    for c in (c0, c1, c2):
        i = torch.where(c >= 2 ** 31, _MASK32 - c, c)
        out.append((i.to(torch.float32) * scale).double())
    return out


def _neighbours(s, alpha: int, z, y, x):
    """(flat site index, validity) of the neighbours of sites (z, y, x) of sublattice alpha, bond by bond."""
    L = (s.L1, s.L2, s.L3)
    per = tuple(s.periodic) + (False,) * (3 - s.crystal.D)
    plane = s.L1 * s.L2 * s.L3
    for i, bd in enumerate(s.crystal.bonds):
        if bd.alpha != alpha:
            continue
        d = tuple(bd.delta) + (0,) * (3 - s.crystal.D)
        q, ok = [], torch.ones_like(x, dtype=torch.bool)
        for c, dk, Lk, pk in zip((x, y, z), d, L, per):
            v = c + dk
            if pk:
                v = v % Lk
            else:
                ok &= (v >= 0) & (v < Lk)
                v = v.clamp(0, Lk - 1)
            q.append(v)
        yield i, bd.alpha2 * plane + (q[2] * s.L2 + q[1]) * s.L1 + q[0], ok


def _sublattice_sites(s, alpha: int, colour: int | None, device):
    """Active sites of one sublattice, or of one of its colour classes: flat index, z, y, x."""
    z, y, x = torch.meshgrid(*(torch.arange(v, device=device) for v in (s.L3, s.L2, s.L1)), indexing="ij")
    keep = torch.as_tensor(s.site_mask()[alpha], device=device)
    if colour is not None:
        idx = torch.zeros_like(x)
        for r, m in enumerate(s.colouring.m):
            K = tuple(int(k) for k in s.colouring.K[r]) + (0,) * (3 - s.crystal.D)
            idx = idx * m + (K[0] * x + K[1] * y + K[2] * z + int(s.colouring.o[alpha][r])) % m
        keep = keep & (idx == colour)
    z, y, x = z[keep], y[keep], x[keep]
    return alpha * s.L1 * s.L2 * s.L3 + (z * s.L2 + y) * s.L1 + x, z, y, x


def _anisotropy(k1, k2, p):
    return (k1 * ((p[0] * p[1]) ** 2 + (p[0] * p[2]) ** 2 + (p[1] * p[2]) ** 2) + k2 * (p[0] * p[1] * p[2]) ** 2)


def _field(s, X, alpha, z, y, x):
    """Bond part of the local field at the given sites: [components] of (B, sites)."""
    v = [torch.zeros((X.shape[0], x.numel()), dtype=X.dtype, device=X.device) for _ in range(s.n)]
    for i, q, ok in _neighbours(s, alpha, z, y, x):
        M = s.bond_matrix(i)
        t = [X[:, k, q] * ok for k in range(s.n)]
        for k in range(s.n):
            for l in range(s.n):
                if M[k, l] != 0.0:
                    v[k] += float(M[k, l]) * t[l]
    return v


def _chain64(s, X: torch.Tensor, T: torch.Tensor, seed: int, sweeps: int) -> torch.Tensor:
    """`sweeps` Metropolis sweeps of vector spins X (B, n, sites) float64 in place: colour classes in order, colour
    first, then sublattice."""
    B, dev = X.shape[0], X.device
    beta = (1.0 / T.to(torch.float32)).to(dev).double().reshape(-1, 1)
    reps = torch.arange(B, device=dev).reshape(-1, 1) * s.nsite
    k1 = None if s.cubic_k1 is None else torch.as_tensor(s.cubic_k1, device=dev).double().reshape(-1)
    n_colours = math.prod(s.colouring.m)
    for sw in range(sweeps):
        for colour in range(n_colours):
            for alpha in range(s.b):
                own, z, y, x = _sublattice_sites(s, alpha, colour, dev)
                if own.numel() == 0:
                    continue
                v = _field(s, X, alpha, z, y, x)
                u0, u1, u2 = _uniforms(seed, sw, reps + own)
                if s.n == 2:
                    t = [torch.cos(2 * math.pi * u1), torch.sin(2 * math.pi * u1)]
                else:
                    cz = 2 * u1 - 1
                    rr = torch.sqrt(torch.clamp(1 - cz * cz, min=0.0))
                    t = [rr * torch.cos(2 * math.pi * u2), rr * torch.sin(2 * math.pi * u2), cz]
                old = [X[:, k, own] for k in range(s.n)]
                dE = torch.zeros_like(u0)
                for k in range(s.n):
                    h = float(s.h[k]) if s.h is not None else 0.0
                    dE -= (t[k] - old[k]) * (v[k] + h)
                if k1 is not None:
                    dE += _anisotropy(k1[own], s.cubic_k2, t) - _anisotropy(k1[own], s.cubic_k2, old)
                acc = u0 < torch.exp(-beta * dE)
                for k in range(s.n):
                    X[:, k, own] = torch.where(acc, t[k], old[k])
    return X


def _observables64(s, X: torch.Tensor):
    """Energy (B,) and per-sublattice magnetization (B, b, n) of spins (B, n, sites)."""
    dev = X.device
    E = torch.zeros(X.shape[0], dtype=torch.float64, device=dev)
    M = torch.zeros((X.shape[0], s.b, s.n), dtype=torch.float64, device=dev)
    k1 = None if s.cubic_k1 is None else torch.as_tensor(s.cubic_k1, device=dev).double().reshape(-1)
    for alpha in range(s.b):
        own, z, y, x = _sublattice_sites(s, alpha, None, dev)
        v = _field(s, X, alpha, z, y, x)
        p = [X[:, k, own] for k in range(s.n)]
        for k in range(s.n):
            h = float(s.h[k]) if s.h is not None else 0.0
            E -= (p[k] * (0.5 * v[k] + h)).sum(dim=1)
            M[:, alpha, k] = p[k].sum(dim=1)
        if k1 is not None:
            E += _anisotropy(k1[own], s.cubic_k2, p).sum(dim=1)
    return E, M


def _charge64(s, X: torch.Tensor, layer: int) -> torch.Tensor:
    """Berg-Luscher charge of one layer: two spherical triangles per plaquette whose corners are all active."""
    S = X.reshape(X.shape[0], 3, s.b, s.L3, s.L2, s.L1)[:, :, 0, layer]
    m = torch.as_tensor(s.site_mask()[0, layer], device=X.device)
    valid = m[:-1, :-1] & m[:-1, 1:] & m[1:, :-1] & m[1:, 1:]
    a, b, c, d = S[:, :, :-1, :-1], S[:, :, :-1, 1:], S[:, :, 1:, 1:], S[:, :, 1:, :-1]

    def omega(p, q, r):
        num = (p * torch.cross(q, r, dim=1)).sum(1)
        den = 1 + (p * q).sum(1) + (q * r).sum(1) + (r * p).sum(1)
        return 2 * torch.atan2(num, den)
    return ((omega(a, b, c) + omega(a, c, d)) * valid).sum(dim=(1, 2)) / (4 * math.pi)


def _interleave(s, x: torch.Tensor) -> torch.Tensor:
    """(4 Q, n, b, L3, L2, L1) -> the interleaved layout (Q, b, L3, L2, n, L1, 4), rows split by colour residue."""
    P = 1
    for r, m in enumerate(s.colouring.m):
        P = math.lcm(P, m // math.gcd(int(s.colouring.K[r][0]) % m or m, m))
    B, n, b, L3, L2, L1 = x.shape
    x = x.reshape(B // 4, 4, n, b, L3, L2, L1 // P, P).transpose(-1, -2).reshape(B // 4, 4, n, b, L3, L2, L1)
    return x.permute(0, 3, 4, 5, 2, 6, 1).contiguous()


def _gradients64(case: dict, seed: int):
    """Mean negative log-density of the block rows and its gradients for the masked network in 64 bits."""
    P = BlockProposal(8, 1, seed=seed, device=DEVICE)
    Ws = [(torch.as_tensor(W, device=DEVICE).double().requires_grad_(True),
           torch.as_tensor(b, device=DEVICE).double().requires_grad_(True)) for W, b in P.get_params()]
    G, per = 16, SPINS // 16
    pos = torch.arange(SPINS, device=DEVICE)
    deg_in = torch.cat([torch.zeros(BOUNDARY, dtype=torch.long, device=DEVICE), pos // per + 1])
    deg_h = torch.arange(HIDDEN, device=DEVICE) * G // HIDDEN
    masks = [deg_h[:, None] >= deg_in[None, :], deg_h[:, None] >= deg_h[None, :], deg_h[:, None] >= deg_h[None, :],
             (pos // per)[:, None] >= deg_h[None, :]]
    x = _block_rows(case["batch"], seed).double()
    a = x
    for l, (W, b) in enumerate(Ws):
        a = a @ (W * masks[l]).T + b
        if l < 3:
            a = torch.relu(a)
    up = (x[:, BOUNDARY:] > 0).double()
    loss = -(up * torch.nn.functional.logsigmoid(a) + (1 - up) * torch.nn.functional.logsigmoid(-a)).sum(1).mean()
    loss.backward()
    return float(loss), [(W.grad.cpu().numpy(), b.grad.cpu().numpy()) for W, b in Ws]


def exact(case: dict, seed: int):
    """The outputs of `run` in 64-bit floats, or None: Ising spins and acceptance counts are whole numbers (and
    their energies sums of those), and the largest chains would take too long."""
    fam, s = case["family"], _systems(_key(case))
    if fam == "train":
        return _gradients64(case, seed)
    if fam == "vector":
        B = case["B"]
        Bp = 4 * -(-B // 4) if case["layout"] == "quad" else B
        if Bp * s.nsite * s.n * 8 > 4e9 or Bp * s.nsite * case["sweeps"] > 1e8:
            return None
        X = torch.zeros((Bp, s.n, s.nsite), dtype=torch.float64, device=DEVICE)
        X[:B] = _vector_spins(s, B, seed).reshape(B, s.n, s.nsite)
        T = _temperatures(case)
        T = torch.cat([T, T[-1:].expand(Bp - B)])
        X = _chain64(s, X, T, seed, case["sweeps"])
        S = X.reshape((Bp, s.n) + s.shape)
        S = _interleave(s, S) if case["layout"] == "quad" else S
        return (S, *_observables64(s, X[:B])) if case["measure"] else S
    if fam == "nanodisk":
        B = case["B"]
        X = _vector_spins(s, B, seed).double().reshape(B, s.n, s.nsite)
        X = _chain64(s, X, _temperatures(case), seed, case["sweeps"])
        return (X.reshape((B, s.n) + s.shape), *_observables64(s, X), _charge64(s, X, case["layers"] // 2))
    if fam == "ragged":
        if sum(case["B"] * t.nsite for t, _ in s) * case["sweeps"] > 2e8:
            return None
        out = []
        for i, (t, T) in enumerate(s):
            X = _ragged_spins(t, case["B"], seed, i).double().reshape(case["B"], t.n, t.nsite)
            T = torch.full((case["B"],), T, dtype=torch.float32)
            out.append(_chain64(t, X, T, seed + i, case["sweeps"]).reshape((case["B"], t.n) + t.shape))
        return out
    return None
