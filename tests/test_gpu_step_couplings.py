"""The default FP64 step (no trace) with several coupling strengths, a field and walkers of uneven bond
dimension, over three steps, against the FP64 oracle: the on-chip copies of the Trotter tables beyond
the first strength, the field's part of the energy, walkers smaller than the slot layout, and 64 threads
per walker on a chain.  No walker branches, so each evolves by itself (its weight scaled by
N / sum of the weights after a step, MPSQMC2.cpp:613-686); the first, a
middle and the last walker's weight, overlap and local energy to 1e-10 relative, the
reference-parity tolerance (the energy: of the couplings' scale)."""
import numpy as np
import pytest

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from mpsqmc_b200.capi import OPT_POPCONTROL_INTERVAL
from oracle import envwalk as ew

pytestmark = pytest.mark.gpu

SEED, STEPS, DTAU = 99, 3, 0.02


def couplings(kind):
    name, _, n = kind.partition(":")
    if name == "alternating":  # nearest neighbours, two strengths in turn
        ci, cj, _ = pb.chain(int(n))
        return ci, cj, np.where(ci % 2 == 0, 1.0, 0.6)
    if name == "j1j2":
        pairs = sorted((i, i + r) for r in (1, 2) for i in range(int(n) - r))
        ci, cj = np.array(pairs, dtype=np.int32).T
        return ci, cj, np.where(cj - ci == 1, 1.0, 0.45)
    ci, cj, _ = pb.lattice("snake:" + n)
    return ci, cj, np.array([0.7, 1.0, 1.3])[(ci + cj) % 3]


CASES = [  # couplings, D_T, walkers' bonds, walkers, field
    ("alternating:10", 8, (8, 4), 1400, 0.3), ("alternating:14", 64, (48, 24), 3, 0.0), ("alternating:12", 33, (20,), 450, 0.2),
    ("j1j2:12", 16, (8,), 500, 0.0), ("j1j2:12", 17, (16, 8, 4), 5, 0.4), ("lattice:4x4", 24, (12, 6), 300, 0.2),
    ("lattice:3x3", 8, (8, 5), 1300, 0.0),
]


@pytest.mark.parametrize("kind,DT,DWs,N,h", CASES, ids=[f"{c[0]}-{c[1]}-{c[2][0]}-{c[3]}-h{c[4]}" for c in CASES])
def test_steps_match_oracle(kind, DT, DWs, N, h):
    ci, cj, cJ = couplings(kind)
    L = int(max(cj)) + 1
    rng = np.random.default_rng(5)
    dims = pb.virtual_dims(L, DT)
    trial = pb.left_normalize(pb.MPS(dims, rng.normal(size=int(np.sum(dims[:-1] * dims[1:]) * 2))))
    kinds = [pb.compress(trial, D) for D in DWs]
    Jvals = np.unique(cJ)
    tabs = [pb.trotter_tables(J, DTAU) for J in Jvals]
    U, S, VT = (np.concatenate([t[k] for t in tabs]) for k in range(3))
    grid = pb.grid_marsaglia(4, 4)
    eng = Engine(L=L, ci=ci, cj=cj, cJ=cJ, h=h, dtau=DTAU, trial_dims=trial.dims, trial=trial.data, Jvals=Jvals, U=U, S=S,
                 VT=VT, grid=grid, Ndesired=N, capacity=max(64, 2 * N), walker_dims=kinds[0].dims)
    which = [kinds[w % len(kinds)] for w in range(N)]
    wdims = np.stack([np.asarray(m.dims, np.int32) for m in which])
    data = [m.data + 1e-3 * rng.normal(size=m.data.size) for m in which]
    eng.set_option(OPT_POPCONTROL_INTERVAL, 1000)
    eng.set_walkers_dims(wdims, data, np.ones(N), normalize=True)
    eng.set_rng(SEED, 0)
    got = []
    for _ in range(STEPS):
        eng.walk(1)
        got.append(eng.last_step_walkers())
    eng.close()
    nC = len(ci)
    u = np.random.RandomState(SEED)._bit_generator.random_raw(STEPS * N * nC) / 4294967296.0  # MT19937
    for w in sorted({0, N // 2, N - 1}):
        state, weight = data[w], 1.0
        for s in range(STEPS):
            r = ew.step(trial.dims, trial.data, wdims[w], state, weight, ci=ci, cj=cj, cJ=cJ, Jvals=Jvals, U=U, S=S, VT=VT,
                        grid=grid, dtau=DTAU, h=h, u=u[(s * N + w) * nC:(s * N + w + 1) * nC])
            state, weight = r["walker"], r["weight"] * N / float(np.sum(got[s]["weight"]))
            assert got[s]["weight"][w] == pytest.approx(r["weight"], rel=1e-10), (w, s)
            assert got[s]["overlap"][w] == pytest.approx(r["overlap"], rel=1e-10), (w, s)
            assert got[s]["energy"][w] == pytest.approx(r["energy"], rel=1e-10, abs=1e-10 * 0.75 * float(np.sum(np.abs(cJ)))), (w, s)
