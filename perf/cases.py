"""Performance cases: walker propagation as a program drives it through mpsqmc_b200.Engine.

A program builds an Engine for its problem once, uploads a population, and then calls walk(); after
each call it reads the steps' statistics and the per-walker weights, overlaps, local energies and
parents.  The population stays on the device between calls, so most cases time exactly that.  Two
cases (names ending in _io) also move the population: from host memory to the device before the
steps and back to the host after them, as a run that restarts from, and writes, a checkpoint does.

Trials are ground-state-like states: the stored DMRG trials of the L = 64 chain and of the 6x6 and
8x8 lattices, cut to the first sites of the chain or the first rows of the lattice where a case
is smaller, and truncated to the case's trial bond dimension.  Walkers are the trial truncated to
their own bond dimensions plus seeded noise, as the framework's workloads make them.

Results of the FP64 sweep are returned in 64 bits as the Engine gives them; those of the modes whose
contractions carry FP32 accuracy are kept in 32 bits, as a program that asked for these modes would.
"""
from functools import lru_cache
from math import exp, log
import os

import numpy as np
import torch

from mpsqmc_b200 import Engine, capi, problem, workloads

PRECISIONS = {"fp64": capi.PRECISION_FP64, "tf32x3": capi.PRECISION_TF32X3, "tf32x3_tc": capi.PRECISION_TF32X3_TC}
SITES = {"chain": (1, 64), "snake6": (6, 6), "snake8": (8, 8), "snake8_256": (8, 8)}  # width, most rows
FILES = {"chain": "trial_L64D64.npz", "snake6": "trial_snake6x6_D64.npz", "snake8": "trial_snake8x8_D64.npz",
         "snake8_256": "trial_snake8x8_D256.npz"}


def case(name, family, rows, DT, DW, N, dtau=0.005, steps=1, precision="fp64", h=0.0, uneven=0, io=False):
    """family: the stored trial; rows: chain length, or rows of the lattice; uneven > 0: walkers of
    bond dimensions DW / 2^0 .. DW / 2^uneven in one population; steps: steps of one pass."""
    c = dict(family=family, rows=rows, DT=DT, DW=DW, N=N, dtau=dtau, steps=steps, precision=precision, h=h,
             uneven=uneven, io=io)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest run: ten sites, sixteen walkers, the size a user starts with and checks against
        # exact diagonalisation; launches and latency count.  The population is written at the end
        case("chain10_d8_w4_io", "chain", 10, 8, 4, 16, dtau=0.05, steps=8, io=True),
        # the reference program's own run: twenty sites, walkers of bond dimension 2, 1000 of them
        case("chain20_d4_w2", "chain", 20, 4, 2, 1000, dtau=0.01, steps=4),
        # the small chain configuration (L = 16, D = 16, 128 walkers), population in and out
        case("chain16_d16_w16_io", "chain", 16, 16, 16, 128, dtau=0.01, steps=10, io=True),
        # the chain configuration (L = 64, D_T = 64, D_W = 32): the population of one GPU, in FP64, the
        # default, and in the mode that is fastest on chains
        case("chain64_d64_w32", "chain", 64, 64, 32, 1024, dtau=0.01),
        case("chain64_d64_w32_tf32x3", "chain", 64, 64, 32, 1024, dtau=0.01, precision="tf32x3"),
        # a magnetic field and bond dimensions that are no multiples of anything
        case("chain45_d50_w27_field", "chain", 45, 50, 27, 300, dtau=0.01, h=0.3),
        # a small lattice with many walkers: couplings of ranges 1 to 11, small bonds
        case("snake6x3_d16_w8", "snake6", 3, 16, 8, 740),
        # the 6x6 lattice with its D_T = 64 ground-state trial, walkers of D_W 16, 32 and 64 together
        case("snake6x6_d64_uneven", "snake6", 6, 64, 64, 444, uneven=2),
        # the 8x8 lattice with its D_T = 64 ground-state trial
        case("snake8x8_d64_w32", "snake8", 8, 64, 32, 444),
        # the largest: the 8x8 lattice at D_T = 256, D_W = 64, in FP64 and in the walker-batched
        # tensor-core mode that the benchmark's headline is measured in (one population's share of
        # walkers here, the headline has 4096)
        case("snake8x8_d256_w64", "snake8_256", 8, 256, 64, 148),
        case("snake8x8_d256_w64_tc", "snake8_256", 8, 256, 64, 512, precision="tf32x3_tc"),
    ]


def _log_int(rng, lo, hi):
    return int(round(exp(rng.uniform(log(lo), log(hi)))))


def draw(rng):
    """One more case: chains of 8 to 64 sites and lattices of 6 or 8 columns and 2 to 8 rows, trial bonds
    4 to 64 (to 256 on 8 columns), walker bonds 2 to 64, 16 to 1024 walkers, as many as cost no more
    than the largest listed case."""
    kind = rng.random()
    if kind < 0.45:
        family, rows, DT = "chain", _log_int(rng, 8, 64), _log_int(rng, 4, 64)
    elif kind < 0.85:
        family = rng.choice(["snake6", "snake8"])
        rows, DT = rng.randint(2, SITES[family][1]), _log_int(rng, 8, 64)
    else:
        family, rows, DT = "snake8_256", rng.randint(3, 8), _log_int(rng, 96, 256)
    DW = _log_int(rng, 2, max(3, min(64, DT if family != "snake8_256" else DT // 2)))
    precision, h, uneven = "fp64", 0.0, 0
    p = rng.random()
    if p < 0.15 and DT >= 32:
        precision = "tf32x3"
    elif p < 0.3 and DT >= 48 and DW >= 16 and family != "chain":
        precision = "tf32x3_tc"
    elif p < 0.45 and DW >= 8:
        uneven = rng.randint(1, 2)
    elif p < 0.55:
        h = round(rng.uniform(0.1, 0.5), 3)
    c = case(None, family, rows, DT, DW, 1, dtau=rng.choice([0.005, 0.01, 0.02]), precision=precision, h=h, uneven=uneven)
    limit = 0.3 * 148 * work(dict(listed()[9], N=1))["flops"] / work(c)["flops"]
    c["N"] = _log_int(rng, 16, max(17, min(1024, int(limit))))
    return c


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _left(sites):
    """Left-canonical form of a list of [sigma, Dl, Dr] arrays, norm 1."""
    out, carry = [], np.ones((1, 1))
    for k, A in enumerate(sites):
        A = np.einsum("ab,sbc->sac", carry, A)
        d, a, c = A.shape
        if k == len(sites) - 1:
            out.append(A / np.linalg.norm(A))
        else:
            q, carry = np.linalg.qr(A.reshape(d * a, c))
            out.append(q.reshape(d, a, -1))
    return out


def _truncate(sites, D):
    """Right-to-left sweep of truncated SVDs of a left-canonical state: bonds of at most D, then
    left-canonical again."""
    sites = list(sites)
    for k in range(len(sites) - 1, 0, -1):
        A = sites[k]
        d, a, c = A.shape
        u, s, vt = np.linalg.svd(A.transpose(1, 0, 2).reshape(a, d * c), full_matrices=False)
        n = max(1, min(D, int(np.sum(s > 1e-13 * s[0]))))
        sites[k] = vt[:n].reshape(n, d, c).transpose(1, 0, 2)
        sites[k - 1] = np.einsum("sab,bn->san", sites[k - 1], u[:, :n] * s[:n])
    return _left(sites)


@lru_cache(maxsize=None)
def _trial(family, rows, DT):
    """The stored trial of the family, its first sites or rows, at bond dimension DT."""
    z = np.load(os.path.join(workloads.DATA, FILES[family]))
    m = problem.MPS(z["dims"].astype(np.int32), z["data"].astype(np.float64))
    sites = _left([m.site(k) for k in range(m.L)])
    L = SITES[family][0] * rows
    if L < m.L:  # the dominant Schmidt state of the sites that are kept
        env = np.ones((1, 1))
        for A in reversed(sites[L:]):
            env = sum(a @ env @ a.T for a in A)
        v = np.linalg.eigh(env)[1][:, -1:]
        sites = _left(sites[: L - 1] + [np.matmul(sites[L - 1], v)])
    return tuple(_truncate(sites, DT) if DT < max(a.shape[2] for a in sites) else sites)


@lru_cache(maxsize=None)
def _walker(family, rows, DT, DW):
    return tuple(_truncate(list(_trial(family, rows, DT)), DW))


def _flat(sites):
    return np.concatenate([a.transpose(0, 2, 1).reshape(-1) for a in sites])


def _dims(sites):
    return np.array([1] + [a.shape[2] for a in sites], dtype=np.int32)


def _couplings(c):
    if c["family"] == "chain":
        return problem.chain(c["rows"])
    return problem.snake(SITES[c["family"]][0], c["rows"])


@lru_cache(maxsize=None)
def _tables(dtau):
    return problem.trotter_tables(1.0, dtau), problem.grid_marsaglia(4, 4)


def _populations(c, seed):
    """[(walkers' indices, dims, host array [n, size])], one entry per bond profile."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    key = (c["family"], c["rows"], c["DT"])
    out = []
    for q in range(c["uneven"] + 1):
        sites = _walker(*key, max(1, c["DW"] >> q))
        index = np.arange(q, c["N"], c["uneven"] + 1)
        base = torch.from_numpy(_flat(sites)).cuda()
        noise = torch.randn(len(index), base.numel(), generator=g, device="cuda", dtype=torch.float64)
        out.append((index, _dims(sites), base + 1e-3 * noise))
    return out


def _rng_seed(seed):
    return (20131015 + 7919 * int(seed)) & 0xFFFFFFFF


def prepare(case, seed):
    c = case
    trial = _trial(c["family"], c["rows"], c["DT"])
    ci, cj, cJ = _couplings(c)
    (U, S, VT), grid = _tables(c["dtau"])
    pops = _populations(c, seed)
    eng = Engine(L=len(trial), ci=ci, cj=cj, cJ=cJ, h=c["h"], dtau=c["dtau"], trial_dims=_dims(trial), trial=_flat(trial),
                 Jvals=[1.0], U=U, S=S, VT=VT, grid=grid, Ndesired=c["N"], capacity=max(64, 2 * c["N"]),
                 walker_dims=pops[0][1])
    if c["uneven"]:
        dims, walkers = [None] * c["N"], [None] * c["N"]
        for index, d, w in pops:
            w = w.cpu().numpy()
            for r, k in enumerate(index):
                dims[k], walkers[k] = d, w[r]
        eng.set_walkers_dims(np.stack(dims), walkers, np.ones(c["N"]))
        host = None
    else:
        dev = pops[0][2]
        host = torch.empty(dev.shape, dtype=torch.float64, pin_memory=c["io"])
        host.copy_(dev)
        host = host.numpy()
        eng.set_walkers(host, np.ones(c["N"]), None, np.zeros(c["N"]))
    eng.set_option(capi.OPT_PRECISION, PRECISIONS[c["precision"]])
    eng.set_rng(_rng_seed(seed), 0)
    state = dict(engine=eng, steps=c["steps"], io=c["io"], seed=_rng_seed(seed),
                 kind=np.float64 if c["precision"] == "fp64" else np.float32)
    if c["io"]:
        state.update(host=host, back=torch.empty(2 * c["N"], host.shape[1], dtype=torch.float64, pin_memory=True).numpy())
    return state


def run(state):
    eng, kind = state["engine"], state["kind"]
    if state["io"]:
        n = state["host"].shape[0]
        eng.set_walkers(state["host"], np.ones(n), None, np.zeros(n))
        eng.set_rng(state["seed"], 0)
        eng.set_step(0)
    stats = eng.walk(state["steps"])
    last = eng.last_step_walkers()
    out = {"n_after": np.array([s["n_after"] for s in stats]), "parent": last["parent"]}
    for key in ("E_P", "sum_weight"):
        out[key] = np.array([s[key] for s in stats], dtype=kind)
    for key in ("weight", "overlap", "energy"):
        out[key] = last[key].astype(kind)
    if state["io"]:
        walkers, weights, overlaps, _ = eng.get_walkers(out=state["back"])
        out.update(walkers=walkers, weights=weights, overlaps=overlaps)
    return out


# ---------------------------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------------------------
def _flops(a, b, pairs, h):
    """Contractions of one walker-step at trial bonds a and walker bonds b: the right environments, the
    four left branches of every site that opens a coupling, their way through the sites between,
    the right branches and closures of every coupling, the right environments that a coupling made
    stale, and the local energy's channels."""
    L = len(a) - 1
    near = all(j == i + 1 for i, j in pairs)
    x = [2.0 * a[k] * b[k] * b[k + 1] for k in range(L)]        # environment times one walker block
    y = [2.0 * a[k] * a[k + 1] * b[k + 1] for k in range(L)]    # one trial block times that
    r = [2.0 * a[k + 1] * b[k] * b[k + 1] + 2.0 * a[k] * a[k + 1] * b[k] for k in range(L)]
    total, seen, valid = 2 * sum(r), set(), 1
    for i, j in pairs:
        if i not in seen:
            seen.add(i)
            total += 2 * x[i] + 4 * y[i]
        total += 4 * sum(2 * (x[m] + y[m]) for m in range(i + 1, j))
        if not near:
            total += 2 * sum(r[k] for k in range(j + 1, valid))
        valid = j + 1
        total += 4.0 * a[j + 1] * b[j] * b[j + 1] + 8.0 * a[j] * a[j + 1] * b[j] + 32.0 * a[j] * b[j]
    last = {}
    for i, j in pairs:
        last[i] = max(last.get(i, j), j)
    for k in range(L):
        cont = sum(1 for i, j in last.items() if i < k < j)
        total += 2 * (x[k] + y[k]) * (1 + 3 * cont) + (0 if k in seen else 2 * x[k] + 4 * y[k])
    return total


def work(case):
    c = case
    ci, cj, _ = _couplings(c)
    L, pairs = SITES[c["family"]][0] * c["rows"], list(zip(ci.tolist(), cj.tolist()))
    a = problem.virtual_dims(L, c["DT"]).tolist()
    flops = nbytes = 0.0
    for q in range(c["uneven"] + 1):
        b = [min(x, max(1, c["DW"] >> q)) for x in a]
        n = len(range(q, c["N"], c["uneven"] + 1))
        flops += n * c["steps"] * _flops(a, b, pairs, c["h"])
        nbytes += n * 16.0 * 2 * sum(b[k] * b[k + 1] for k in range(L)) * (2 if c["io"] else 1)
    return {"bytes": nbytes + 16.0 * sum(a[k] * a[k + 1] for k in range(L)) + 32.0 * c["N"], "flops": flops}


# ---------------------------------------------------------------------------------------------
# the same steps in 64 bits with torch
# ---------------------------------------------------------------------------------------------
def _branches(E, B, A):
    """B[s]^T E A[t] for every walker, [4, n, a, b], entry s + 2 t."""
    return torch.stack([B[s].T @ (E @ A[t]) for t in range(2) for s in range(2)])


def _through(E, B, A):
    return B[0].T @ (E @ A[0]) + B[1].T @ (E @ A[1])


def _closures(P, B, A, R):
    """M[:, p, q] = <P_p, B[s] R A[t]^T>, q = s + 2 t."""
    Z = torch.stack([B[s] @ (R @ A[t].transpose(1, 2)) for t in range(2) for s in range(2)])
    return torch.einsum("pnab,qnab->npq", P, Z)


def _rights(T, W):
    n = W[0].shape[1]
    R = [None] * (len(T) + 1)
    R[-1] = torch.ones(n, 1, 1, dtype=torch.float64, device="cuda")
    for k in range(len(T) - 1, -1, -1):
        R[k] = T[k][0] @ (R[k + 1] @ W[k][0].transpose(1, 2)) + T[k][1] @ (R[k + 1] @ W[k][1].transpose(1, 2))
    return R


def _energy(T, W, pairs, cJ, h):
    """<T|H|W> of every walker, H = sum J S_i.S_j - h sum S^z."""
    sz = torch.tensor([-0.5, 0, 0, 0.5], dtype=torch.float64, device="cuda")
    sx = torch.tensor([0, 0.5, 0.5, 0], dtype=torch.float64, device="cuda")
    isy = torch.tensor([0, 0.5, -0.5, 0], dtype=torch.float64, device="cuda")
    pair = torch.outer(sx, sx) - torch.outer(isy, isy) + torch.outer(sz, sz)
    R, E, total = _rights(T, W), torch.ones(W[0].shape[1], 1, 1, dtype=torch.float64, device="cuda"), 0.0
    for i in range(len(T)):
        js = [(j, J) for (a, j), J in zip(pairs, cJ) if a == i]
        if js or h:
            P = _branches(E, T[i], W[i])
            if h:
                total = total - h * torch.einsum("p,pnab,nab->n", sz, P, R[i + 1])
            at = i + 1
            for j, J in js:
                while at < j:
                    P = torch.stack([_through(p, T[at], W[at]) for p in P])
                    at += 1
                total = total + J * torch.einsum("npq,pq->n", _closures(P, T[j], W[j], R[j + 1]), pair)
        E = _through(E, T[i], W[i])
    return total


def _norm2(W):
    E = torch.ones(W[0].shape[1], 1, 1, dtype=torch.float64, device="cuda")
    for A in W:
        E = A[0].transpose(1, 2) @ E @ A[0] + A[1].transpose(1, 2) @ E @ A[1]
    return E[:, 0, 0]


def _step(T, W, wt, u, pairs, cJ, tables, grid, dtau, h):
    """One propagation of the walkers W ([2, n, b, b'] per site, changed in place)."""
    U, S, VT = (torch.from_numpy(np.asarray(t)).cuda() for t in tables)
    U, VT, Sq = U.reshape(4, 4).T, VT.reshape(4, 4).T, torch.sqrt(S)  # U[p, k], VT[l, q]
    field = torch.exp(0.5 * h * dtau * torch.tensor([-0.5, 0.5], dtype=torch.float64, device="cuda"))[:, None, None, None]

    def magnet():
        for A in W:
            A *= field

    if h:
        magnet()
    R = _rights(T, W)
    ov, valid = R[0][:, 0, 0], 0
    E, at = torch.ones(W[0].shape[1], 1, 1, dtype=torch.float64, device="cuda"), 0
    for c, (i, j) in enumerate(pairs):
        while at < i:
            E, at = _through(E, T[at], W[at]), at + 1
        while valid > j + 1:
            valid -= 1
            R[valid] = T[valid][0] @ (R[valid + 1] @ W[valid][0].transpose(1, 2)) + \
                T[valid][1] @ (R[valid + 1] @ W[valid][1].transpose(1, 2))
        P = _branches(E, T[i], W[i])
        for m in range(i + 1, j):
            P = torch.stack([_through(p, T[m], W[m]) for p in P])
        M = _closures(P, T[j], W[j], R[j + 1])
        C = torch.einsum("k,l,pk,npq,lq->nkl", Sq, Sq, U, M, VT)
        pdf = torch.clamp(torch.einsum("gk,nkl,gl->ng", grid, C, grid), min=0) * (4.0 / (ov[:, None] * grid.shape[0]))
        if bool((ov < 0).any()):  # the sign of a walker drops out
            pdf = torch.clamp(torch.einsum("gk,nkl,gl->ng", grid, C, grid) * (4.0 / (ov[:, None] * grid.shape[0])), min=0)
        total = pdf.sum(1)
        wt = wt * total
        pick = torch.clamp((torch.cumsum(pdf / total[:, None], 1) <= u[:, c, None]).sum(1), max=grid.shape[0] - 1)
        x = grid[pick]
        ov = 4.0 * torch.einsum("nk,nkl,nl->n", x, C, x)
        fx = 2.0 * Sq * x
        for site, tab in ((i, U.T), (j, VT)):  # operators O[s + 2 t]
            O = fx @ tab
            A0, A1 = W[site][0].clone(), W[site][1].clone()
            W[site][0] = O[:, 0, None, None] * A0 + O[:, 2, None, None] * A1
            W[site][1] = O[:, 1, None, None] * A0 + O[:, 3, None, None] * A1
        valid = max(valid, j + 1)
    if h:
        magnet()
    ovr, nrm = _rights(T, W)[0][:, 0, 0], torch.sqrt(_norm2(W))
    energy = _energy(T, W, pairs, cJ, h) / ovr
    W[-1] /= nrm[None, :, None, None]
    return wt, ovr.abs() / nrm, energy


def exact(case, seed):
    c = case
    T = [torch.from_numpy(a).cuda() for a in _trial(c["family"], c["rows"], c["DT"])]
    ci, cj, cJ = _couplings(c)
    pairs = list(zip(ci.tolist(), cj.tolist()))
    tables, grid = _tables(c["dtau"])
    grid_d = torch.from_numpy(grid).cuda()
    random = np.random.RandomState(_rng_seed(seed))  # MT19937, one 32-bit output per uniform

    def uniforms(n):
        return random._bit_generator.random_raw(n).astype(np.float64) / 4294967296.0

    groups = []
    for index, dims, flat in _populations(c, seed):
        W, at = [], 0
        for a, b in zip(dims[:-1].tolist(), dims[1:].tolist()):
            W.append(flat[:, at:at + 2 * a * b].reshape(-1, 2, b, a).permute(1, 0, 3, 2).contiguous())
            at += 2 * a * b
        groups.append((index, W))
    wt = np.ones(c["N"])
    out = {"n_after": None, "parent": None, "E_P": [], "sum_weight": []}
    for _ in range(c["steps"]):
        n = len(wt)
        u = uniforms(n * len(pairs)).reshape(n, len(pairs))
        ov, en = np.empty(n), np.empty(n)
        for index, W in groups:
            r = _step(T, W, torch.from_numpy(wt[index]).cuda(), torch.from_numpy(u[index]).cuda(), pairs, cJ.tolist(), tables,
                      grid_d, c["dtau"], c["h"])
            wt[index], ov[index], en[index] = (v.cpu().numpy() for v in r)
        out.update(weight=wt.copy(), overlap=ov, energy=en)
        out["E_P"].append(np.sum(wt * en) / np.sum(wt))
        out["sum_weight"].append(np.sum(wt))
        # population control: scaled weights outside [0.25, 1.5] branch, in walker order
        s = wt * (c["N"] / np.sum(wt))
        flagged = (s < 0.25) | (s > 1.5)
        copies, new = np.ones(n, dtype=int), s.copy()
        copies[flagged] = (s[flagged] + uniforms(int(flagged.sum()))).astype(int)
        new[flagged] = np.where(s[flagged] < 0.25, 1.0, s[flagged] / np.maximum(copies[flagged], 1))
        parent = np.repeat(np.arange(n), copies)
        wt, ov = new[parent], ov[parent]
        if not np.array_equal(parent, np.arange(n)):
            where = np.empty(n, dtype=int)
            regrouped = []
            for index, W in groups:
                where[:] = -1
                where[index] = np.arange(len(index))
                rows = where[parent]
                keep = np.flatnonzero(rows >= 0)
                pick = torch.from_numpy(rows[keep]).cuda()
                regrouped.append((keep, [A[:, pick].contiguous() for A in W]))
            groups = [g for g in regrouped if len(g[0])]
    out["E_P"], out["sum_weight"] = np.array(out["E_P"]), np.array(out["sum_weight"])
    if c["io"]:
        out.update(walkers=None, weights=wt, overlaps=ov)
    return out
