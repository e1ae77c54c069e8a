"""Problems whose couplings, strengths, length or grid need more room than a CTA's shared memory has: they
are created and stepped like any other, in every sweep, with the buffers that they make large in
global memory.  One step against the FP64 oracle; over 2 L transfers and 4 nC closure factors an FP64 sweep
may be off by (2 L + 4 nC) 2^-48 relative (the energy: of the couplings' scale), 1e-10 at least,
the TF32X3 one by 2^-20 each."""
import numpy as np
import pytest

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from mpsqmc_b200.capi import (E_UNSUPPORTED, OPT_CANONICAL_INTERVAL, OPT_PRECISION, OPT_SWEEP, OPT_WORKSPACE,
                              PRECISION_TF32X3, SWEEP_NEAREST, WORKSPACE_GLOBAL, MpsqmcError)
from oracle import envwalk as ew

pytestmark = pytest.mark.gpu

SEED = 4242


def pairs_of(name):
    kind, _, n = name.partition(":")
    if kind == "all":  # every pair of n sites
        L = int(n)
        i, j = np.triu_indices(L, 1)
        return i.astype(np.int32), j.astype(np.int32)
    ci, cj, _ = pb.lattice(name)
    return ci, cj


def make(name, D, G, N, random_J, seed=3):
    ci, cj = pairs_of(name)
    L = int(max(cj)) + 1
    rng = np.random.default_rng(seed)
    cJ = rng.uniform(0.5, 1.5, len(ci)) if random_J else np.ones(len(ci))
    Jvals = np.unique(cJ)
    tabs = [pb.trotter_tables(J, 0.001) for J in Jvals]
    U, S, VT = (np.concatenate([t[k] for t in tabs]) for k in range(3))
    # unit vectors with |x_0| = 1/2: the factor of the identity in a sampled operator is one, so that the
    # oracle's walker, which is normalised at the end only, stays in range over thousands of couplings
    grid = rng.normal(size=(G, 4))
    grid[:, 1:] *= np.sqrt(0.75) / np.linalg.norm(grid[:, 1:], axis=1)[:, None]
    grid[:, 0] = 0.5 * np.sign(grid[:, 0])
    dims = pb.virtual_dims(L, D)
    trial = np.concatenate([np.linalg.qr(rng.normal(size=(2 * a, b)))[0].reshape(2, a, b).transpose(0, 2, 1).reshape(-1)
                            for a, b in zip(dims[:-1], dims[1:])])  # an isometry per site: norm 1
    walkers = trial + 1e-4 * rng.normal(size=(N, trial.size))
    kw = dict(L=L, ci=ci, cj=cj, cJ=cJ, h=0.0, dtau=0.001, trial_dims=dims, trial=trial, Jvals=Jvals, U=U, S=S, VT=VT,
              grid=grid, Ndesired=N, capacity=4 * N, walker_dims=dims)
    return kw, walkers


def check_step(kw, walkers, options=(), trace=False, tol=None):
    N, ci, cJ, L = len(walkers), kw["ci"], kw["cJ"], kw["L"]
    eng = Engine(**kw)
    eng.set_walkers(walkers, np.ones(N))
    for o, v in options:
        eng.set_option(o, v)
    eng.set_trace(trace)
    eng.set_rng(SEED, 0)
    w0, wt0, _, _ = eng.get_walkers()
    eng.walk(1)
    got = eng.last_step_walkers()
    E = eng.energy()
    eng.close()
    assert np.isfinite(E)
    uni = np.random.RandomState(SEED)._bit_generator.random_raw(N * len(ci)) / 4294967296.0  # MT19937
    ops = 2 * L + 4 * len(ci)
    tol = max(1e-10, ops * 2.0**-48) if tol is None else ops * tol
    for w in {0, N - 1}:
        r = ew.step(kw["trial_dims"], kw["trial"], kw["walker_dims"], w0[w], wt0[w], ci=ci, cj=kw["cj"], cJ=cJ,
                    Jvals=kw["Jvals"], U=kw["U"], S=kw["S"], VT=kw["VT"], grid=kw["grid"], dtau=kw["dtau"],
                    u=uni[w * len(ci):(w + 1) * len(ci)])
        assert got["weight"][w] == pytest.approx(r["weight"], rel=tol), w
        assert got["overlap"][w] == pytest.approx(r["overlap"], rel=tol), w
        assert got["energy"][w] == pytest.approx(r["energy"], abs=tol * 0.75 * float(np.sum(np.abs(cJ)))), w


PROBLEMS = {  # name, bond dimension, grid points, walkers, random strengths
    "all-to-all-random": ("all:40", 4, 60, 2, True),
    "lattice-20x20-random": ("snake:20x20", 4, 60, 2, True),
    "chain-700-random": ("chain:700", 4, 60, 2, True),
    "chain-3000": ("chain:3000", 2, 60, 2, False),
    "chain-12000": ("chain:12000", 2, 16, 1, False),
    "grid-28700": ("chain:10", 4, 28700, 2, False),
}


@pytest.mark.parametrize("name", PROBLEMS)
def test_step_with_large_tables(name):
    check_step(*make(*PROBLEMS[name]))


def test_step_with_every_table_outside_shared_memory():
    check_step(*make(*PROBLEMS["all-to-all-random"]), [(OPT_WORKSPACE, WORKSPACE_GLOBAL)])


@pytest.mark.parametrize("name", ["lattice-20x20-random", "chain-12000", "grid-28700"])
@pytest.mark.parametrize("mode", ["trace", "qr", "nearest", "tf32x3"])
def test_other_sweeps_with_large_tables(name, mode):
    if mode == "nearest" and not name.startswith(("chain", "grid")):
        pytest.skip("couplings of every range")
    if mode == "trace" and name == "chain-12000":
        pytest.skip("the trace takes the norm at every coupling: time grows with the square of the length")
    options = {"trace": [], "qr": [(OPT_CANONICAL_INTERVAL, 0)], "nearest": [(OPT_SWEEP, SWEEP_NEAREST)],
               "tf32x3": [(OPT_PRECISION, PRECISION_TF32X3)]}[mode]
    check_step(*make(*PROBLEMS[name]), options, trace=mode == "trace", tol=2.0**-20 if mode == "tf32x3" else None)


def test_grid_beyond_the_limit_is_refused():
    kw, _ = make("chain:10", 4, 29500, 1, False)
    with pytest.raises(MpsqmcError) as e:
        Engine(**kw)
    assert e.value.code == E_UNSUPPORTED


def test_step_where_shared_memory_holds_fewer_walkers_than_the_shape():
    """A grid whose PDF takes most of a CTA's share: fewer CTAs per SM than the bonds alone would have."""
    check_step(*make("chain:10", 4, 9000, 1300, False))
