"""The default FP64 step (QR-free general sweep) against the FP64 oracle where its products and launch
shapes change: bond dimensions around the small-product limit (8 x 8 x 8) and the 16-row and
8- and 16-column tiles, odd leading dimensions (no 16-byte pairs), every number of threads per
walker and walkers per SM the engine picks, work buffers on chip and off it, chains (stored right
branches) and a lattice (couplings of any range).  One step; the first, a middle and the last
walker's weight, overlap and local energy to 1e-10 relative, the reference-parity tolerance, and
the sampled indices through them (a different grid point changes the overlap by far more)."""
import numpy as np
import pytest

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from oracle import envwalk as ew

pytestmark = pytest.mark.gpu

SEED = 777
SHAPES = [  # lattice, D_T, D_W, walkers
    ("chain:7", 4, 2, 3), ("chain:9", 8, 8, 4), ("chain:9", 9, 8, 1400), ("chain:10", 8, 4, 200),
    ("chain:12", 16, 16, 3), ("chain:12", 17, 15, 500), ("chain:14", 33, 31, 3), ("chain:14", 34, 18, 460),
    ("chain:14", 64, 48, 310), ("chain:16", 65, 33, 3), ("chain:16", 128, 40, 2), ("chain:18", 130, 128, 2),
    ("snake:3x3", 8, 4, 1200), ("snake:4x3", 16, 8, 450), ("snake:4x4", 33, 17, 450), ("snake:4x4", 64, 64, 300),
    ("snake:4x4", 96, 23, 2),
]


@pytest.mark.parametrize("lattice,DT,DW,N", SHAPES, ids=[f"{a}-{b}-{c}-{d}" for a, b, c, d in SHAPES])
def test_step_matches_oracle(lattice, DT, DW, N):
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
    eng.set_rng(SEED, 0)
    w0, wt0, _, _ = eng.get_walkers()
    eng.walk(1)
    got = eng.last_step_walkers()
    eng.close()
    uni = np.random.RandomState(SEED)._bit_generator.random_raw(N * len(ci)) / 4294967296.0  # MT19937
    for w in sorted({0, N // 2, N - 1}):
        r = ew.step(trial.dims, trial.data, walker.dims, w0[w], wt0[w], ci=ci, cj=cj, cJ=cJ, Jvals=[1.0], U=U, S=S,
                    VT=VT, grid=grid, dtau=0.01, u=uni[w * len(ci):(w + 1) * len(ci)])
        for key in ("weight", "overlap", "energy"):
            assert got[key][w] == pytest.approx(r[key], rel=1e-10), (w, key)
