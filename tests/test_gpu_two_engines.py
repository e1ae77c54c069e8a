"""Two engines alive in one process: what one of them needs of the kernels' shared memory (its population,
bond dimensions, work-buffer placement) leaves the other as it is.  The first engine is created, then
the second, then the first is stepped and evaluated; its numbers equal those it gives alone."""
import numpy as np
import pytest

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from mpsqmc_b200.capi import (OPT_CANONICAL_INTERVAL, OPT_PRECISION, OPT_SWEEP, OPT_WORKSPACE, PRECISION_TF32X3,
                              SWEEP_NEAREST, WORKSPACE_GLOBAL)

pytestmark = pytest.mark.gpu


def make(L, DT, DW, N):
    ci, cj, cJ = pb.chain(L)
    rng = np.random.default_rng(5)
    dims = pb.virtual_dims(L, DT)
    trial = pb.left_normalize(pb.MPS(dims, rng.normal(size=int(np.sum(dims[:-1] * dims[1:]) * 2))))
    walker = pb.compress(trial, DW)
    U, S, VT = pb.trotter_tables(1.0, 0.01)
    eng = Engine(L=L, ci=ci, cj=cj, cJ=cJ, h=0.0, dtau=0.01, trial_dims=trial.dims, trial=trial.data, Jvals=[1.0], U=U,
                 S=S, VT=VT, grid=pb.grid_marsaglia(4, 4), Ndesired=N, capacity=max(64, 2 * N), walker_dims=walker.dims)
    eng.set_walkers(walker.data + 1e-3 * rng.normal(size=(N, walker.data.size)), np.ones(N))
    eng.set_rng(7, 0)
    return eng


OPTIONS = {"default": [], "qr": [(OPT_CANONICAL_INTERVAL, 0)], "nearest": [(OPT_SWEEP, SWEEP_NEAREST)],
           "tf32x3": [(OPT_PRECISION, PRECISION_TF32X3)]}


@pytest.mark.parametrize("mode", OPTIONS)
@pytest.mark.parametrize("other", ["more walkers", "smaller bonds", "outside shared memory"])
def test_engine_steps_after_another_is_created(mode, other):
    def use(eng):
        out = []
        for _ in range(2):
            eng.walk(1)
            out.append(eng.last_step_walkers())
        out.append(dict(E=eng.energy()))
        eng.close()
        return out

    def first():
        eng = make(12, 40, 24, 16)
        for o, v in OPTIONS[mode]:
            eng.set_option(o, v)
        return eng

    alone = use(first())
    eng = first()
    second = make(12, 8, 4, 16) if other == "smaller bonds" else make(12, 40, 24, 1200)
    if other == "outside shared memory":
        second.set_option(OPT_WORKSPACE, WORKSPACE_GLOBAL)
    together = use(eng)
    second.walk(1)
    second.close()
    for a, b in zip(alone, together):
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg=key)
