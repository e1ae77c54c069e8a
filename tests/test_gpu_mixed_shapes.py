"""The TF32X3 per-walker step against the FP64 oracle where its products change shape: bonds around the
small-product limit (8 x 8 x 8), the 16-row and 8- and 16-column tiles and the 16-deep chunks of K,
trial bonds that are no multiples of four (the left factor read element by element), chains (stored
right branches) and lattices (fused closures, several branches per product).  Head and tail of an
operand leave 2^-22 of a product and FP32 sums about as much; taking 2^-20 for each of the 2 L
transfers and of the four closure factors of every coupling that multiply into a walker's
numbers, one step may be off by (2 L + 4 nC) 2^-20 relative (the energy: of the couplings' scale)."""
import numpy as np
import pytest

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from mpsqmc_b200.capi import OPT_PRECISION, PRECISION_TF32X3
from oracle import envwalk as ew

pytestmark = pytest.mark.gpu

SEED = 777
SHAPES = [  # lattice, D_T, D_W, walkers
    ("chain:7", 4, 2, 3), ("chain:9", 9, 8, 300), ("chain:12", 16, 16, 3), ("chain:12", 17, 15, 4),
    ("chain:14", 34, 18, 3), ("chain:14", 64, 48, 310), ("chain:16", 128, 40, 2), ("snake:3x3", 8, 4, 5),
    ("snake:4x4", 33, 17, 3), ("snake:4x4", 64, 32, 300), ("snake:4x4", 96, 23, 2),
]


@pytest.mark.parametrize("lattice,DT,DW,N", SHAPES, ids=[f"{a}-{b}-{c}-{d}" for a, b, c, d in SHAPES])
def test_mixed_step_matches_oracle(lattice, DT, DW, N):
    ci, cj, cJ = pb.lattice(lattice)
    L = int(max(cj)) + 1
    rng = np.random.default_rng(5)
    dims = pb.virtual_dims(L, DT)
    trial = pb.left_normalize(pb.MPS(dims, rng.normal(size=int(np.sum(dims[:-1] * dims[1:]) * 2))))
    walker = pb.compress(trial, DW)
    U, S, VT = pb.trotter_tables(1.0, 0.01)
    grid = pb.grid_marsaglia(4, 4)
    eng = Engine(L=L, ci=ci, cj=cj, cJ=cJ, h=0.0, dtau=0.01, trial_dims=trial.dims, trial=trial.data, Jvals=[1.0], U=U,
                 S=S, VT=VT, grid=grid, Ndesired=N, capacity=max(64, 2 * N), walker_dims=walker.dims)
    eng.set_walkers(walker.data + 1e-3 * rng.normal(size=(N, walker.data.size)), np.ones(N))
    eng.set_option(OPT_PRECISION, PRECISION_TF32X3)
    eng.set_rng(SEED, 0)
    w0, wt0, _, _ = eng.get_walkers()
    eng.walk(1)
    got = eng.last_step_walkers()
    eng.close()
    uni = np.random.RandomState(SEED)._bit_generator.random_raw(N * len(ci)) / 4294967296.0  # MT19937
    tol = (2 * L + 4 * len(ci)) * 2.0**-20
    for w in sorted({0, N // 2, N - 1}):
        r = ew.step(trial.dims, trial.data, walker.dims, w0[w], wt0[w], ci=ci, cj=cj, cJ=cJ, Jvals=[1.0], U=U, S=S,
                    VT=VT, grid=grid, dtau=0.01, u=uni[w * len(ci):(w + 1) * len(ci)])
        assert got["weight"][w] == pytest.approx(r["weight"], rel=tol), w
        assert got["overlap"][w] == pytest.approx(r["overlap"], rel=tol), w
        assert got["energy"][w] == pytest.approx(r["energy"], abs=tol * 0.75 * float(np.sum(np.abs(cJ)))), w
