"""An engine on a device whose memory is nearly taken: the QR-free sweep's scratch for several walkers per SM
is given up where only that of one per SM fits, and the steps are the same.  L = 64 chain, D_T = 64,
D_W = 32: 1.7 GB of scratch at two walkers per SM, 0.85 GB at one."""
import numpy as np
import pytest
import torch

from mpsqmc_b200 import Engine
from mpsqmc_b200 import problem as pb
from mpsqmc_b200.capi import OPT_POPCONTROL_INTERVAL

pytestmark = pytest.mark.gpu


def make():
    L = 64
    ci, cj, cJ = pb.chain(L)
    rng = np.random.default_rng(5)
    dims, wdims = pb.virtual_dims(L, 64), pb.virtual_dims(L, 32)
    sites = [np.linalg.qr(rng.normal(size=(2 * a, b)))[0].reshape(2, a, b) for a, b in zip(dims[:-1], dims[1:])]
    flat = lambda A: np.concatenate([x.transpose(0, 2, 1).reshape(-1) for x in A])  # noqa: E731
    walker = flat([x[:, :a, :b] for x, a, b in zip(sites, wdims[:-1], wdims[1:])])
    U, S, VT = pb.trotter_tables(1.0, 0.01)
    eng = Engine(L=L, ci=ci, cj=cj, cJ=cJ, h=0.0, dtau=0.01, trial_dims=dims, trial=flat(sites), Jvals=[1.0], U=U, S=S,
                 VT=VT, grid=pb.grid_marsaglia(4, 4), Ndesired=1000, capacity=64, walker_dims=wdims)
    eng.set_walkers(walker + 1e-3 * rng.normal(size=(8, walker.size)), np.ones(8))
    eng.set_rng(7, 0)
    eng.set_option(OPT_POPCONTROL_INTERVAL, 1000)  # eight walkers stand for the population of 1000
    return eng


def step(eng):
    eng.walk(1)
    out = eng.last_step_walkers()
    eng.close()
    return out


def test_create_and_step_with_little_memory():
    want = step(make())  # (the kernels' own memory is reserved from here on)
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - 1450 * 2**20, dtype=torch.uint8, device="cuda")
    try:
        got = step(make())
    finally:
        del block
        torch.cuda.empty_cache()
    for key in ("weight", "overlap", "energy"):
        np.testing.assert_allclose(got[key], want[key], rtol=1e-10, err_msg=key)
