"""Performance cases: what a user of nova-gb300 has it do, through its public
entry points, from the smallest call to the largest.

Eight kinds of work:

  solve     a whole PBVI solve (POMDPPBVIGPU.solve / POMDPPBVICPU.solve)
  update    one PBVI backup of every belief on a solver that is under way
  batch     many POMDPs solved in one call (solve_batched)
  perseus   a whole Perseus solve (POMDPPerseusGPU.solve)
  vi        a whole value-iteration solve of an MDP (MDPValueIterationGPU.solve)
  value     V(b) and the action of many beliefs under a policy
  grad      V(b0) and its gradient with respect to R, T and O
  expand    growing a POMDP's belief set (POMDP.expand)

Models are random sparse ones: ns distinct successors per (state, action),
Dirichlet(1) transitions, observations and beliefs, rewards in [-1, 1].
`ragged` rows end early (-1), `sorted` False lists successors in no order, as
a file's statements may.
"""
import ctypes as ct
import math

import numpy as np
import torch

from nova_gb300 import nova_pomdp as npm
from nova_gb300 import nova_pomdp_alpha_vectors as npav
from nova_gb300 import nova_pomdp_pbvi as npp
from nova_gb300.mdp import MDP
from nova_gb300.mdp_vi import MDPValueIterationGPU
from nova_gb300.pomdp import POMDP
from nova_gb300.pomdp_adjoint import PBVIGradSpec, pbvi_value
from nova_gb300.pomdp_alpha_vectors import POMDPAlphaVectors
from nova_gb300.pomdp_pbvi import POMDPPBVICPU, POMDPPBVIGPU, solve_batched
from nova_gb300.pomdp_perseus import POMDPPerseusGPU

SCORING = {"fp16": npp.SCORING_FP16, "bf16": npp.SCORING_BF16, "exact": npp.SCORING_EXACT}
GAMMA = float(np.float32(0.95))
EXACT_FLOPS = 1.2e13  # FP64 operations that exact() may spend on one case


def listed():
    return [
        # The smallest problem anybody solves (two states, as in the tiger
        # problem): launches, allocations and synchronisations are all of it.
        dict(name="solve_tiny", kind="solve", n=2, m=3, z=2, ns=2, r=5, rz=2, horizon=20, api="gpu", scoring="fp16"),
        # A small problem solved to its horizon.
        dict(name="solve_n64", kind="solve", n=64, m=4, z=8, ns=8, r=256, rz=8, horizon=100, api="gpu",
             scoring="fp16"),
        # One backup of a medium problem, default scoring.
        dict(name="update_n512", kind="update", n=512, m=8, z=16, ns=16, r=1024, rz=32, scoring="fp16", table=True,
             warm=6),
        # Sizes that are a multiple of nothing, BF16 scoring.
        dict(name="update_n1000_bf16", kind="update", n=1000, m=5, z=11, ns=13, r=1500, rz=27, scoring="bf16",
             table=True, warm=6),
        # One backup of a large problem: the headline model with half its
        # beliefs, so that several solvers fit the card.
        dict(name="update_n4096", kind="update", n=4096, m=16, z=32, ns=32, r=4096, rz=64, scoring="fp16", table=True,
             warm=4),
        # A parameter study: many unequal problems in one call.
        dict(name="batch_12", kind="batch", count=12, mix=0, nmin=32, nmax=2048, rmin=128, rmax=4096, mmax=16,
             zmax=32, horizon=20),
        # Randomised point-based solve of a medium problem.
        dict(name="perseus_n512", kind="perseus", n=512, m=8, z=16, ns=16, r=1024, rz=32, horizon=25),
        # The large planning grid: memory-bound sweeps, rows in state order.
        dict(name="vi_n1m", kind="vi", n=1 << 20, m=8, ns=16, horizon=50, sorted=True, ragged=False),
        # An MDP as a file lists it: rows in no order and of unequal length.
        dict(name="vi_unsorted", kind="vi", n=150001, m=5, ns=11, horizon=100, sorted=False, ragged=True),
        # Evaluating a large policy at a large belief set.
        dict(name="value_n4096", kind="value", n=4096, r=8192, count=8192, rz=64, api="gpu"),
        # Gradient of a solve's value with respect to the model.
        dict(name="grad_n1024", kind="grad", n=1024, m=8, z=16, ns=16, r=1024, rz=32, horizon=20),
        # Growing the belief set between solves.
        dict(name="expand_n512", kind="expand", n=512, m=8, z=16, ns=16, r=1024, rz=32, method="distinct_beliefs"),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "update", "update", "update", "batch", "perseus", "vi", "vi", "value",
                       "grad", "expand"])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def model(nmax, rmax, mmax, zmax, nmin=2, rmin=4):
        n = log(nmin, nmax)
        return dict(kind=kind, n=n, m=rng.randint(2, mmax), z=rng.randint(2, zmax), ns=min(n, rng.randint(2, 32)),
                    r=log(rmin, rmax), rz=min(n, rng.randint(2, 64)))
    if kind == "solve":
        return dict(model(512, 1024, 8, 16), horizon=rng.randint(5, 60), api=rng.choice(["gpu", "gpu", "cpu"]),
                    scoring=rng.choice(["fp16", "fp16", "bf16", "exact"]))
    if kind == "update":
        scoring = rng.choice(["fp16", "fp16", "fp16", "bf16", "exact"])
        return dict(model(4096, 4096, 16, 32, 128, 128), scoring=scoring,
                    table=scoring == "exact" or rng.random() < 0.85, warm=5)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 12), mix=rng.randint(1, 1 << 20), nmin=32, nmax=log(64, 1024),
                    rmin=32, rmax=log(64, 2048), mmax=rng.randint(2, 16), zmax=rng.randint(2, 32),
                    horizon=rng.randint(5, 20))
    if kind == "perseus":
        return dict(model(1024, 1024, 8, 16, 8, 16), horizon=rng.randint(2, 25))
    if kind == "vi":
        n, m = log(50, 1 << 20), rng.randint(1, 16)
        return dict(kind=kind, n=n, m=m, ns=min(n, rng.randint(1, 32), max(1, (1 << 27) // (n * m))),
                    horizon=rng.randint(10, 50), sorted=rng.random() < 0.6, ragged=rng.random() < 0.4)
    if kind == "value":
        n = log(2, 4096)
        return dict(kind=kind, n=n, r=log(4, 8192), count=log(1, 8192), rz=log(1, n) if n > 1 else 1,
                    api=rng.choice(["gpu", "gpu", "cpu"]))
    if kind == "grad":
        return dict(model(1024, 1024, 8, 16, 8, 16), horizon=rng.randint(2, 20))
    c = dict(model(512, 1024, 8, 16, 8, 16), method=rng.choice(["distinct_beliefs", "random"]))
    if c["method"] == "random":
        c["add"] = log(16, 2048)
    return c


# ---------------------------------------------------------------------------
# Inputs (made on the GPU from the seed, handed over as host arrays, which is
# what the library's model objects take)
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rows(g, rows, n, k):
    """rows x k distinct integers of [0, n), each row ascending."""
    x = torch.randint(0, n - k + 1, (rows, k), generator=g, device="cuda", dtype=torch.int32)
    return torch.sort(x, dim=1).values + torch.arange(k, device="cuda", dtype=torch.int32)


def _dirichlet(g, *shape):
    w = -torch.log1p(-torch.rand(shape, generator=g, device="cuda", dtype=torch.float64).clamp(max=1 - 1e-12))
    return (w / w.sum(-1, keepdim=True).clamp(min=1e-300)).float()


def _transitions(g, n, m, ns, ordered=True, ragged=False):
    S, T = _rows(g, n * m, n, ns), _dirichlet(g, n * m, ns)
    if not ordered:
        S = torch.gather(S, 1, torch.argsort(torch.rand((n * m, ns), generator=g, device="cuda"), dim=1))
    if ragged:
        length = torch.randint((ns + 1) // 2, ns + 1, (n * m, 1), generator=g, device="cuda")
        dead = torch.arange(ns, device="cuda") >= length
        T = torch.where(dead, 0.0, T)
        T = (T.double() / T.double().sum(1, keepdim=True)).float()
        S = torch.where(dead, -1, S)
    return S.view(n, m, ns), T.view(n, m, ns)


def _pomdp(c, seed):
    """A model as tensors: S, T, O, R and the beliefs Z, B."""
    g = _gen(seed)
    n, m, z, ns, r, rz = (c[k] for k in ("n", "m", "z", "ns", "r", "rz"))
    S, T = _transitions(g, n, m, ns)
    return dict(n=n, m=m, z=z, ns=ns, r=r, rz=rz, gamma=GAMMA, horizon=c.get("horizon", 1), S=S, T=T,
                O=_dirichlet(g, m, n, z), R=torch.rand((n, m), generator=g, device="cuda") * 2 - 1,
                Z=_rows(g, r, n, rz), B=_dirichlet(g, r, rz))


def _host(model):
    return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in model.items()}


def _gamma0(model):
    """The library's default initial alphas: min R / (1 - gamma) everywhere."""
    low = np.float32(float(model["R"].min())) / (np.float32(1.0) - np.float32(GAMMA))
    return np.full((model["r"], model["n"]), low, np.float32)


def _batch_models(c, seed):
    rng = np.random.default_rng(c["mix"])  # the shapes are the case's, the contents the seed's
    out = []
    for k in range(c["count"]):
        n = int(round(math.exp(rng.uniform(math.log(c["nmin"]), math.log(c["nmax"])))))
        r = int(round(math.exp(rng.uniform(math.log(c["rmin"]), math.log(c["rmax"])))))
        out.append(_pomdp(dict(n=n, m=int(rng.integers(2, c["mmax"] + 1)), z=int(rng.integers(2, c["zmax"] + 1)),
                               ns=min(16, n), r=r, rz=min(32, n), horizon=c["horizon"]), int(seed) * 101 + k))
    return out


def _mdp(c, seed):
    g = _gen(seed)
    S, T = _transitions(g, c["n"], c["m"], c["ns"], c["sorted"], c["ragged"])
    return dict(n=c["n"], m=c["m"], ns=c["ns"], gamma=0.99, horizon=c["horizon"], S=S, T=T,
                R=torch.rand((c["n"], c["m"]), generator=g, device="cuda") * 2 - 1)


def _policy(c, seed):
    """Alphas around a common value function, and beliefs as dense rows."""
    g = _gen(seed)
    n, r, count = c["n"], c["r"], c["count"]
    G = torch.randn((1, n), generator=g, device="cuda") * 3 - 10 + torch.randn((r, n), generator=g, device="cuda")
    pi = torch.randint(0, 16, (r,), generator=g, device="cuda", dtype=torch.int32)
    B = torch.zeros((count, n), device="cuda")
    B.scatter_(1, _rows(g, count, n, c["rz"]).long(), _dirichlet(g, count, c["rz"]))
    return G, pi, B


class _Device:
    """A solver's device array, for torch.as_tensor; keeps the solver alive."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, version=3, strides=None,
                                             data=(ct.cast(pointer, ct.c_void_p).value, False))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("solve", "update", "perseus", "grad", "expand"):
        model = _host(_pomdp(c, seed))
        st = dict(case=c, seed=int(seed), model=model)
        if kind == "grad":
            st["model"]["GammaInitial"] = _gamma0(model)
            st["b0"] = np.full(c["n"], 1.0 / c["n"], np.float32)
            st["R"], st["T"], st["O"] = (torch.tensor(model[k], device="cuda", requires_grad=True) for k in "RTO")
        elif kind != "expand":
            st["pomdp"] = POMDP.from_arrays(model)
            st["pomdp"].initialize_gpu()
            st["gamma0"] = _gamma0(model)
        if kind == "update":
            # A solve under way: the solver has its operands, and its alphas
            # are those of a few backups.
            st["alg"] = POMDPPBVIGPU(st["pomdp"], GammaInitial=st["gamma0"])
            st["alg"].set_scoring(SCORING[c["scoring"]])
            if not c["table"]:
                st["alg"].set_table(npp.TABLE_NEVER)
            for _ in range(c["warm"]):
                st["alg"].update()
        return st
    if kind == "batch":
        pomdps = [POMDP.from_arrays(_host(model)) for model in _batch_models(c, seed)]
        for p in pomdps:
            p.initialize_gpu()
        return dict(case=c, pomdps=pomdps)
    if kind == "vi":
        mdp = MDP.from_arrays(_host(_mdp(c, seed)))
        mdp.initialize_gpu()
        return dict(case=c, mdp=mdp)
    G, pi, B = _policy(c, seed)
    if c["api"] == "gpu":
        return dict(case=c, G=G, pi=pi, B=B, V=torch.empty(c["count"], device="cuda"),
                    A=torch.empty(c["count"], dtype=torch.int32, device="cuda"))
    policy = POMDPAlphaVectors()
    if npav._nova.pomdp_alpha_vectors_initialize(policy, c["n"], 16, c["r"]) != 0:
        raise RuntimeError("pomdp_alpha_vectors_initialize failed")
    G, pi = np.ascontiguousarray(G.cpu().numpy()), pi.cpu().numpy().astype(np.uint32)
    ct.memmove(policy.Gamma, G.ctypes.data, G.nbytes)
    ct.memmove(policy.pi, pi.ctypes.data, pi.nbytes)
    return dict(case=c, policy=policy, B=B.cpu().numpy())


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state, state["case"])


def _arrays(policy):
    return policy.gamma_array(), policy.pi_array().astype(np.int64)


def _filled(x, size, axis, value):
    """x with `value` up to `size` along `axis`: results whose size follows their contents."""
    pad = [(0, 0)] * x.ndim
    pad[axis] = (0, size - x.shape[axis])
    return np.pad(x, pad, constant_values=value)


def _run_solve(st, c):
    if c["api"] == "cpu":
        return _arrays(POMDPPBVICPU(st["pomdp"], GammaInitial=st["gamma0"]).solve())
    alg = POMDPPBVIGPU(st["pomdp"], GammaInitial=st["gamma0"])
    alg.set_scoring(SCORING[c["scoring"]])
    return _arrays(alg.solve())


def _run_update(st, c):
    alg = st["alg"]
    alg.update()
    G = alg.d_Gamma if alg.currentHorizon % 2 == 0 else alg.d_GammaPrime
    return (torch.as_tensor(_Device(alg, G, (c["r"], c["n"]), "<f4"), device="cuda"),
            torch.as_tensor(_Device(alg, alg.d_pi, (c["r"],), "<i4"), device="cuda"))


def _run_batch(st, c):
    return [_arrays(p) for p in solve_batched(st["pomdps"], scoring=npp.SCORING_FP16)]


def _run_perseus(st, c):
    # Perseus draws its beliefs from libc's rand().
    ct.CDLL(None).srand(st["seed"] % (1 << 31) + 1)
    G, pi = _arrays(POMDPPerseusGPU(st["pomdp"], GammaInitial=st["gamma0"]).solve())
    return _filled(G, c["r"], 0, 0.0), _filled(pi, c["r"], 0, -1)


def _run_vi(st, c):
    policy = MDPValueIterationGPU(st["mdp"], Vinitial=np.zeros(c["n"], np.float32)).solve()
    return policy.V_array(), policy.pi_array().astype(np.int64)


def _run_value(st, c):
    if c["api"] == "cpu":
        V, a = st["policy"].value_and_action_batched(st["B"])
        return V, a.astype(np.int64)
    rc = npav._nova.pomdp_alpha_vectors_value_batched_gpu(
        st["G"].data_ptr(), st["pi"].data_ptr(), c["r"], c["n"], st["B"].data_ptr(), c["count"], st["V"].data_ptr(),
        st["A"].data_ptr())
    if rc != 0:
        raise RuntimeError("pomdp_alpha_vectors_value_batched_gpu failed with code %d" % rc)
    return st["V"], st["A"]


def _run_grad(st, c):
    spec = PBVIGradSpec(model=st["model"], b0=st["b0"], horizon=c["horizon"], checkpoint_every=10)
    V = pbvi_value(st["R"], st["T"], st["O"], spec)
    return (V.detach(),) + torch.autograd.grad(V, (st["R"], st["T"], st["O"]))


def _run_expand(st, c):
    p = POMDP.from_arrays(st["model"])
    if c["method"] == "random":
        npm._nova.nova_gb300_expand_seed(1, st["seed"] % (1 << 31))
        p.horizon = 10
        p.expand(method="random", numBeliefsToAdd=c["add"])
    else:
        p.expand(method=c["method"])
    out = p.arrays()
    return _filled(out["Z"], c["n"], 1, -1), _filled(out["B"], c["n"], 1, 0.0)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def work(case):
    """What one pass cannot do without: inputs read and outputs written once,
    and the products and sums of the factored algorithm (PBVI: every alpha
    projected once per (action, observation, state), every belief scored
    against every projection over its support, the chosen alphas assembled)."""
    c, kind = case, case["kind"]
    if kind == "batch":
        # Sizes are drawn log-uniformly: the geometric middle, count times.
        n, r = math.sqrt(c["nmin"] * c["nmax"]), math.sqrt(c["rmin"] * c["rmax"])
        one = work(dict(kind="solve", n=n, m=(2 + c["mmax"]) / 2, z=(2 + c["zmax"]) / 2, ns=min(16, n), r=r,
                        rz=min(32, n), horizon=c["horizon"]))
        return {k: v * c["count"] for k, v in one.items()}
    n = c["n"]
    if kind == "vi":
        per = 2.0 * n * c["m"] * c["ns"] * 4 + n * c["m"] * 4 + 12 * n
        return {"bytes": per * c["horizon"], "flops": 3.0 * n * c["m"] * c["ns"] * c["horizon"]}
    if kind == "value":
        return {"bytes": 4.0 * n * (c["r"] + c["count"]) + 8 * c["count"], "flops": 2.0 * c["r"] * c["count"] * c["rz"]}
    m, z, ns, r, rz = (c[k] for k in ("m", "z", "ns", "r", "rz"))
    model = 4.0 * (2 * n * m * ns + m * n * z + n * m + 2 * r * rz)
    if kind == "expand":
        if c["method"] == "random":
            return {"bytes": model + 4.0 * c["add"] * n, "flops": 2.0 * c["add"] * n * ns * (z + 1)}
        return {"bytes": model + 8.0 * r * rz, "flops": 2.0 * r * m * z * (r * n + n * ns)}
    step = 2.0 * m * z * r * (n * ns + r * rz) + 1.0 * r * n * z
    if kind == "perseus":
        # One belief at a time: about a tenth of the beliefs are backed up per step.
        return {"bytes": model + 4.0 * r * n, "flops": c["horizon"] * (2.0 * r * r * rz + 0.1 * r * m * z * ns * rz * 2)}
    steps = c.get("horizon", 1)
    if kind == "grad":
        return {"bytes": 3 * model + 4.0 * steps * r * n * 3, "flops": steps * (step + 8.0 * r * n * (ns + 2 * z))}
    return {"bytes": model + 8.0 * r * n, "flops": step * steps}


# ---------------------------------------------------------------------------
# exact: the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def _dense(S, T, n, m):
    """[m][n][n] transition matrices."""
    out = torch.zeros((n, m, n), dtype=T.dtype, device=T.device)
    live = S >= 0
    return out.scatter_add(2, S.clamp(min=0).long(), torch.where(live, T, 0.0)).transpose(0, 1)


def _backup(model, P, O, R, B, G):
    """One PBVI backup: the actions and the alpha of every (belief, observation)."""
    m, z = model["m"], model["z"]
    value = B @ R
    best = torch.empty((m, z, B.shape[0]), dtype=torch.long, device=B.device)
    with torch.no_grad():
        for a in range(m):
            W = GAMMA * (B @ P[a])
            for o in range(z):
                top, best[a, o] = ((W * O[a, :, o]) @ G.T).max(1)
                value[:, a] += top
        act = value.argmax(1)
        return act, best[act, :, torch.arange(B.shape[0], device=B.device)]


def _assemble(model, P, O, R, G, act, sel):
    out = torch.zeros((model["r"], model["n"]), dtype=G.dtype, device=G.device)
    for a in range(model["m"]):
        i = (act == a).nonzero()[:, 0]
        if len(i):
            X = sum(O[a, :, o] * G[sel[i, o]] for o in range(model["z"]))
            out = out.index_copy(0, i, R[:, a] + GAMMA * (X @ P[a].T))
    return out


def _solve64(model, steps, grad=False):
    n, r = model["n"], model["r"]
    R, T, O = (model[k].double().requires_grad_(grad) for k in "RTO")
    P = _dense(model["S"], T, n, model["m"])
    B = torch.zeros((r, n), dtype=torch.float64, device="cuda").scatter_(1, model["Z"].long(), model["B"].double())
    G = torch.tensor(_gamma0(model), device="cuda").double()
    act = None
    for _ in range(steps):
        act, sel = _backup(model, P, O, R.detach(), B, G.detach())
        G = _assemble(model, P, O, R, G, act, sel)
    return G, act, (R, T, O)


def _steps64(c):
    """Backups from the initial alphas to the outputs, and their dense FP64 cost."""
    steps = c["warm"] + 1 if c["kind"] == "update" else c["horizon"]
    return steps, steps * (2.0 * c["r"] ** 2 * c["n"] * c["m"] * c["z"] + 2.0 * c["r"] * c["n"] ** 2 * c["m"])


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("perseus", "batch"):
        # Perseus: which beliefs are backed up, and with them the number of
        # alphas, follows FP32 comparisons. Batch: its solves are those of
        # the kind "solve", too large for FP64.
        return None
    if kind in ("solve", "update", "grad"):
        steps, cost = _steps64(c)
        # Backup after backup, near ties fall to other alphas in 64 bits than
        # in 32, and after many the two solves hold other alpha sets.
        if cost > EXACT_FLOPS or (kind == "solve" and steps > 10):
            return None
        model = _pomdp(c, seed)
        G, _, leaves = _solve64(model, steps, kind == "grad")
        if kind != "grad":
            return G, None
        V = (G @ torch.full((c["n"],), 1.0 / c["n"], dtype=torch.float64, device="cuda")).max()
        return (V.detach(),) + torch.autograd.grad(V, leaves)
    if kind == "vi":
        model = _mdp(c, seed)
        live, S = model["S"] >= 0, model["S"].clamp(min=0).long()
        T, R = torch.where(live, model["T"], 0.0).double() * float(np.float32(0.99)), model["R"].double()
        V = torch.zeros(c["n"], dtype=torch.float64, device="cuda")
        for _ in range(c["horizon"]):
            V = (R + sum(T[:, :, k] * V[S[:, :, k]] for k in range(c["ns"]))).max(1).values
        return V, None
    if kind == "value":
        G, _, B = _policy(c, seed)
        return torch.cat([(b.double() @ G.double().T).max(1).values for b in B.split(1024)]), None
    if c["method"] == "random":
        return None  # the trajectories follow draws compared with FP32 sums
    return None, _distinct64(_pomdp(c, seed))


def _distinct64(model):
    """The belief values after a distinct-beliefs expansion: the old rows, then
    for every belief the successor farthest (L1) from the belief set."""
    n, m, z, r = (model[k] for k in ("n", "m", "z", "r"))
    P, O = _dense(model["S"], model["T"].double(), n, m), model["O"].double()
    B = torch.zeros((r, n), dtype=torch.float64, device="cuda").scatter_(1, model["Z"].long(), model["B"].double())
    far = torch.full((r,), -1.0, dtype=torch.float64, device="cuda")
    star = torch.zeros_like(B)
    for a in range(m):
        W = B @ P[a]
        for o in range(z):
            b = W * O[a, :, o]
            b = b / b.sum(1, keepdim=True).clamp(min=1e-300)
            d = torch.cdist(b, B, p=1).min(1).values
            star, far = torch.where((d > far)[:, None], b, star), torch.maximum(d, far)
    both = torch.cat([B, star])
    return torch.gather(both, 1, torch.sort((both > 0).to(torch.int8), dim=1, descending=True, stable=True).indices)
