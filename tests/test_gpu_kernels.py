"""Single kernels of the backup at the sizes where their tiles, splits and
remainders can go wrong, against the oracle (bit for bit)."""
import numpy as np
import pytest

from conftest import bits
from oracle import oracle as orc
from nova_gb300 import synth
from nova_gb300.pomdp import POMDP
from nova_gb300.pomdp_pbvi import POMDPPBVIGPU
from nova_gb300 import nova_pomdp_pbvi as npp

pytestmark = pytest.mark.gpu


def backups(md, mode, steps, table=npp.TABLE_AUTO):
    """The alphas, actions and statistics after `steps` GPU backups, and the oracle's."""
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    alg = POMDPPBVIGPU(p, GammaInitial=md["GammaInitial"])
    alg.set_scoring(mode)
    alg.set_table(table)
    stats = []
    G, Gp, pi = md["GammaInitial"].copy(), md["GammaInitial"].copy(), np.zeros(md["r"], np.uint32)
    for _ in range(steps):
        alg.update()
        stats.append(alg.stats())
        orc.pbvi_update(md, G, Gp, pi)
        G, Gp = Gp, G
    pol = alg.get_policy()
    return pol.gamma_array(), pol.pi_array(), stats, G, pi


@pytest.mark.parametrize("r,n,distinct", [(1, 5, 1), (7, 33, 3), (8, 256, 8), (9, 257, 2), (255, 31, 40),
                                          (257, 64, 257), (300, 513, 1), (1025, 12, 300)])
def test_duplicate_alphas(r, n, distinct):
    """Rows repeated at random: the unique count and the backup's results."""
    md = synth.random_pomdp(n=n, m=2, z=3, ns=min(4, n), r=r, rz=min(5, n), gamma=0.9, horizon=2, seed=r + n)
    rng = np.random.default_rng(r * n)
    pool = rng.normal(-3.0, 1.0, size=(distinct, n)).astype(np.float32)
    md["GammaInitial"] = pool[rng.integers(0, distinct, r)]
    if r > 4:   # rows equal up to the sign of a zero are different rows
        md["GammaInitial"][2] = md["GammaInitial"][1]
        md["GammaInitial"][1, 0], md["GammaInitial"][2, 0] = 0.0, -0.0
    G, pi, stats, Go, po = backups(md, npp.SCORING_EXACT, 2)
    assert stats[0]["uniqueAlphas"] == len(np.unique(md["GammaInitial"].view(np.uint32), axis=0))
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("mode", [npp.SCORING_FP16, npp.SCORING_EXACT])
@pytest.mark.parametrize("n,z,ns,r", [(33, 1, 5, 40), (64, 3, 1, 61), (70, 5, 7, 130), (31, 8, 31, 257),
                                      (130, 13, 9, 100), (65, 17, 6, 97), (40, 24, 8, 131), (57, 25, 3, 66),
                                      (90, 32, 16, 129), (41, 33, 5, 50), (48, 71, 4, 35)])
def test_projection_chunks(n, z, ns, r, mode):
    """Observation chunks of every width, state tiles with remainders, alpha
    counts that are no multiple of a lane's share, successor rows of every
    length (also none): both layouts of the projection table."""
    md = synth.random_pomdp(n=n, m=2, z=z, ns=ns, r=r, rz=min(6, n), gamma=0.9, horizon=2, seed=n * z + r)
    rng = np.random.default_rng(n + z)
    length = rng.integers(0, ns + 1, size=(n, 2, 1))
    md["S"] = np.where(np.arange(ns) < length, md["S"], -1).astype(np.int32)
    md["GammaInitial"] = rng.normal(-3.0, 1.0, size=(r, n)).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 2)
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("table", [npp.TABLE_AUTO, npp.TABLE_NEVER])
@pytest.mark.parametrize("mode", [npp.SCORING_FP16, npp.SCORING_BF16])
@pytest.mark.parametrize("r,rz,spread", [(64, 1, 1.0), (300, 31, 1.0), (260, 33, 1e-3), (515, 64, 1e-4),
                                         (1100, 65, 2e-5), (700, 97, 0.0)])
def test_merge_candidate_counts(r, rz, spread, mode, table):
    """Rows with one, a few, more than 8 and more than 32 candidates, up to
    lists that overflow (alphas that differ by `spread`), over supports
    around and past multiples of 32."""
    md = synth.random_pomdp(n=100, m=2, z=3, ns=7, r=r, rz=rz, gamma=0.9, horizon=2, seed=r)
    rng = np.random.default_rng(r)
    base = rng.normal(-3.0, 1.0, size=(1, 100))
    md["GammaInitial"] = (base + max(spread, 1e-7) * rng.normal(size=(r, 100))).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 2, table)
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("r,n,count,nz", [(5, 1, 1, 1), (9, 70, 129, 1), (7, 130, 128, 130), (70, 128, 300, 128),
                                          (131, 61, 257, 30), (130, 100, 400, 0), (6, 7900, 3, 40),
                                          (5, 15000, 2, 15000), (3, 4097, 140, 2000), (4200, 50, 1400, 50)])
@pytest.mark.parametrize("odd", [False, True])
def test_belief_values(r, n, count, nz, odd):
    """Listed beliefs, dense ones and both in one call (nz 0), one and two
    planes of alphas and too many states for either, tiles with remainders,
    arrays at odd addresses, ties, zeros of both signs, and alphas that are
    not finite."""
    import torch
    from nova_gb300 import nova_pomdp_alpha_vectors as npav
    rng = np.random.default_rng(r * n + count)
    G = rng.uniform(-5, 5, size=(r, n)).astype(np.float32)
    if r > 6:
        G[5] = G[2]
    if odd:
        G[r // 2, n // 2], G[r // 3, 0] = np.inf, np.nan
        G[0, n - 1] = -0.0
    pi = rng.integers(0, 9, size=r).astype(np.int32)
    B = np.zeros((count, n), np.float32)
    for i in range(count):
        k = nz if nz else (3 if i % 200 < 100 else n)
        B[i, rng.choice(n, min(k, n), replace=False)] = rng.uniform(0, 1, min(k, n))
    B[0, 0] = -0.0
    dG, dB = (torch.as_tensor(np.concatenate([[0], x.ravel()]).astype(np.float32), device="cuda")[1:] for x in (G, B))
    dPi = torch.as_tensor(pi, device="cuda")
    dV, dA = torch.empty(count, device="cuda"), torch.empty(count, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert npav._nova.pomdp_alpha_vectors_value_batched_gpu(dG.data_ptr(), dPi.data_ptr(), r, n, dB.data_ptr(), count,
                                                            dV.data_ptr(), dA.data_ptr()) == 0
    some = range(count) if count * r * n < 4e6 else rng.choice(count, 40, replace=False)
    for i in some:
        V, a = orc.alpha_value(G, pi.astype(np.uint32), B[i])
        assert bits(dV[i].cpu().numpy()) == bits(np.float32(V)) and int(dA[i]) == a, i


@pytest.mark.parametrize("n,m,z,ns,r", [(5, 1, 1, 2, 3), (33, 3, 2, 5, 41), (1026, 2, 3, 9, 10), (130, 7, 5, 31, 9),
                                        (2051, 2, 2, 3, 7), (7300, 2, 2, 4, 6)])
def test_replayed_backups(n, m, z, ns, r):
    """The alphas recomputed between checkpoints carry the forward pass's
    bits, so the gradient does not depend on where the checkpoints lie
    (selections of several actions, ragged successor rows, one to several
    blocks of states, alphas in and out of shared memory)."""
    from nova_gb300.pomdp_adjoint import pbvi_record_and_adjoint
    md = synth.random_pomdp(n=n, m=m, z=z, ns=ns, r=r, rz=min(5, n), gamma=0.9, horizon=5, seed=n + r)
    rng = np.random.default_rng(n)
    length = rng.integers(0, ns + 1, size=(n, m, 1))
    md["S"] = np.where(np.arange(ns) < length, md["S"], -1).astype(np.int32)
    md["GammaInitial"] = rng.normal(-3.0, 1.0, size=(r, n)).astype(np.float32)
    b0 = np.full(n, 1.0 / n, np.float32)
    every = pbvi_record_and_adjoint(md, b0, 5, 1)    # each step's alphas stored
    once = pbvi_record_and_adjoint(md, b0, 5, 5)     # all but the first recomputed
    assert every[0] == once[0] and every[1] == once[1]
    for x, y in zip(every[2:6], once[2:6]):
        # The same FP64 terms in whatever order the atomics land: the sums
        # have at most r * (horizon + z) of them.
        np.testing.assert_allclose(x, y, rtol=0, atol=2.0 ** -52 * r * (5 + z) * max(1e-30, np.abs(y).max()))
    np.testing.assert_array_equal(every[6], once[6])
    np.testing.assert_array_equal(every[7], once[7])


@pytest.mark.parametrize("n,m,ns,tile,ragged,crowd", [(5, 1, 1, 64, False, 0), (300, 3, 7, 64, True, 0),
                                                      (1025, 2, 8, 64, True, 60), (40000, 1, 4, 64, False, 0),
                                                      (9000, 4, 12, 256, True, 4000), (2500, 33, 6, 1024, False, 2400)])
def test_sweep_plan(n, m, ns, tile, ragged, crowd):
    """Plans with one and with many tiles (also more than a CTA counts at
    once), row counts that are no multiple of a warp's share, ragged rows, and
    more than 32 single records of one bank in a tile (`crowd` states share
    their successors' tile)."""
    from nova_gb300 import mdp_vi as mvi
    from nova_gb300 import nova_mdp_vi as nmvi
    from nova_gb300.mdp import MDP
    md = synth.random_mdp(n=n, m=m, ns=ns, gamma=0.95, horizon=3, seed=n)
    rng = np.random.default_rng(n)
    if crowd:
        lead = rng.integers(0, min(tile, n), size=(crowd, m))
        md["S"][:crowd, :, 0] = lead
        md["S"][:crowd, :, 1:] = np.sort(rng.integers(tile, n, size=(crowd, m, ns - 1)), axis=2)
    if ragged:
        md["S"] = np.where(np.arange(ns) < rng.integers(0, ns + 1, size=(n, m, 1)), md["S"], -1).astype(np.int32)
    V0 = rng.normal(size=n).astype(np.float32)
    p = MDP.from_arrays(md)
    p.initialize_gpu()
    mvi.set_tiling(nmvi.TILING_ALWAYS, tile)
    try:
        pol = mvi.MDPValueIterationGPU(p, Vinitial=V0).solve()
        assert mvi.tiling_status() == 1
    finally:
        mvi.set_tiling(nmvi.TILING_AUTO)
    V, pi = orc.mdp_vi_solve(md, horizon=3, VInitial=V0)
    np.testing.assert_array_equal(bits(pol.V_array()), bits(V))
    np.testing.assert_array_equal(pol.pi_array(), pi)


@pytest.mark.parametrize("n,m,z,r,rz,odd", [(3, 1, 1, 2, 2, ""), (40, 3, 11, 33, 9, ""), (65, 2, 40, 20, 65, "negative"),
                                            (90, 2, 3, 70, 7, "same"), (50, 2, 4, 30, 6, "infinite"),
                                            (900, 2, 17, 12, 30, "zero"), (1800, 2, 3, 9, 40, "")])
def test_distinct_expansion(n, m, z, r, rz, odd):
    """One and several tiles of successors, successors in and out of shared
    memory, beliefs at equal distances, observations that cannot occur, and
    probabilities for which no bound holds."""
    md = synth.random_pomdp(n=n, m=m, z=z, ns=min(5, n), r=r, rz=rz, gamma=0.9, horizon=2, seed=n + r)
    if odd == "negative":
        md["T"][::7, 0, 0] *= -1
    elif odd == "infinite":
        md["O"][0, ::9, 1] = np.inf
    elif odd == "zero":
        md["O"][:, :, 0] = 0.0
    elif odd == "same":
        md["Z"][r // 2:], md["B"][r // 2:] = md["Z"][0], md["B"][0]
    md["Z"] = md["Z"][:, ::-1].copy()   # supports in no ascending order
    md["B"] = md["B"][:, ::-1].copy()
    p = POMDP.from_arrays(md)
    p.expand(method="distinct_beliefs")
    Z, B = orc.merge_raw_beliefs(md["Z"], md["B"], orc.expand_distinct(md))
    out = p.arrays()
    np.testing.assert_array_equal(out["Z"], Z)
    np.testing.assert_array_equal(bits(out["B"]), bits(B))


@pytest.mark.parametrize("n,m,z,ns,r,rz", [(2, 1, 1, 1, 3, 1), (33, 3, 33, 5, 60, 31), (70, 2, 16, 33, 90, 64),
                                           (40, 300, 40, 3, 12, 7), (300, 2, 5, 8, 1100, 3), (64, 5, 17, 12, 257, 33)])
def test_perseus_backups(n, m, z, ns, r, rz):
    """Single-belief backups: supports and observations around multiples of 32
    and 16, more (action, observation) pairs than scoring warps, one and many
    splits of the alphas, blocks of states and beliefs with remainders."""
    from nova_gb300.pomdp_perseus import POMDPPerseusGPU
    md = synth.random_pomdp(n=n, m=m, z=z, ns=min(ns, n), r=r, rz=min(rz, n), gamma=0.9, horizon=5, seed=n + r)
    rng = np.random.default_rng(n)
    length = rng.integers(1, md["ns"] + 1, size=(n, m, 1))
    md["S"] = np.where(np.arange(md["ns"]) < length, md["S"], -1).astype(np.int32)
    Go, po = orc.perseus_solve(md, seed=r)
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    alg = POMDPPerseusGPU(p, GammaInitial=md["GammaInitial"])
    orc.lib().oracle_srand(r)
    pol = alg.solve()
    np.testing.assert_array_equal(bits(pol.gamma_array()), bits(Go))
    np.testing.assert_array_equal(pol.pi_array(), po)


@pytest.mark.parametrize("n,m,ns,horizon", [(1, 1, 1, 2), (37, 3, 5, 7), (1500, 1, 9, 6), (5000, 7, 3, 5),
                                            (3001, 16, 8, 4), (40000, 5, 6, 3), (900, 200, 2, 4), (60000, 1, 64, 3),
                                            (30, 2, 30, 5001)])
@pytest.mark.parametrize("api", ["gpu", "cpu", "converged"])
def test_resident_sweeps(n, m, ns, horizon, api):
    """One and many blocks, several rows a thread, V in and out of shared
    memory, models too large to stay in the SMs, unordered rows with entries
    after their end, more sweeps than one launch runs, and a stop between."""
    from nova_gb300.mdp import MDP
    from nova_gb300.mdp_vi import MDPValueIterationCPU, MDPValueIterationGPU
    md = synth.random_mdp(n=n, m=m, ns=min(ns, n), gamma=0.9, horizon=horizon, seed=n + m)
    rng = np.random.default_rng(n)
    k = md["ns"]
    order = np.argsort(rng.random((n, m, k)), axis=2)
    md["S"] = np.take_along_axis(md["S"], order, 2)
    md["T"] = np.take_along_axis(md["T"], order, 2)
    end = rng.integers(1, k + 1, size=(n, m))
    hit = np.arange(k) == end[..., None]
    md["S"] = np.where(hit, -1, md["S"]).astype(np.int32)   # entries behind it stay
    V0 = rng.normal(size=n).astype(np.float32)
    p = MDP.from_arrays(md)
    if api == "cpu":
        pol = MDPValueIterationCPU(p, Vinitial=V0).solve()
    else:
        p.initialize_gpu()
        alg = MDPValueIterationGPU(p, Vinitial=V0)
        if api == "gpu":
            pol = alg.solve()
        else:
            sweep, prev = 0, V0
            while True:      # where the oracle's residual first falls below the tolerance
                sweep += 1
                V, pi = orc.mdp_vi_solve(dict(md, horizon=1), horizon=1, VInitial=prev)
                resid = float(np.max(np.abs(V.astype(np.float64) - prev.astype(np.float64))))
                if resid < 0.3 or sweep == min(horizon, 40):
                    break
                prev = V
            pol, ran, residual = alg.solve_until_converged(tol=0.3, maxSweeps=min(horizon, 40))
            assert ran == sweep and residual == resid
    if api != "converged":
        V, pi = orc.mdp_vi_solve(md, horizon=horizon, VInitial=V0)
    np.testing.assert_array_equal(bits(pol.V_array()), bits(V))
    np.testing.assert_array_equal(pol.pi_array(), pi)


@pytest.mark.parametrize("n,r,rz,m,z,distinct", [(2, 5, 2, 3, 2, 5), (5, 40, 5, 2, 3, 1), (64, 300, 33, 2, 5, 300),
                                                 (830, 130, 7, 2, 2, 130), (1500, 67, 64, 1, 3, 67),
                                                 (3000, 40, 9, 2, 1, 40), (9000, 21, 100, 1, 2, 6),
                                                 (40, 1300, 40, 1, 2, 1300), (14000, 6, 3, 1, 1, 6)])
def test_exact_scan(n, r, rz, m, z, distinct):
    """4 to 64 alphas per block (as many as shared memory holds, and no more
    than there are), one and several blocks and shares per row, equal scores,
    and states too many for the shared-memory form."""
    md = synth.random_pomdp(n=n, m=m, z=z, ns=min(4, n), r=r, rz=rz, gamma=0.9, horizon=2, seed=n + r)
    rng = np.random.default_rng(n)
    pool = rng.normal(-3.0, 1.0, size=(distinct, n)).astype(np.float32)
    md["GammaInitial"] = pool[np.arange(r) % distinct]
    if r > 20:   # alphas that differ only outside some beliefs' successors tie there
        md["GammaInitial"][7] = md["GammaInitial"][3]
        md["GammaInitial"][7, 0] += 1.0
    G, pi, stats, Go, po = backups(md, npp.SCORING_EXACT, 2)
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("mode", [npp.SCORING_FP16, npp.SCORING_BF16])
@pytest.mark.parametrize("step,order", [(0.1, "rising"), (2e-3, "rising"), (2e-3, "falling"), (0.1, "shuffled")])
def test_candidate_lists(step, order, mode):
    """Lists that fill with scores the rising best leaves behind and are
    trimmed (every 32 alphas hold a new best, alone or with near ones), lists
    that run out of room, and lists whose first entry stays the best."""
    r = 8300
    md = synth.random_pomdp(n=16, m=1, z=1, ns=3, r=r, rz=2, gamma=0.9, horizon=1, seed=5)
    rng = np.random.default_rng(7)
    rank = {"rising": np.arange(r), "falling": np.arange(r)[::-1], "shuffled": rng.permutation(r)}[order]
    md["GammaInitial"] = (step * rank[:, None] + step * rng.uniform(size=(r, 16))).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 1)
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("n,r,rz", [(2050, 2049, 17), (4200, 1001, 33)])
def test_merge_in_order(n, r, rz):
    """Projection slabs large enough for rows to be merged in their own order
    (odd row counts, supports past half a warp and past a warp)."""
    md = synth.random_pomdp(n=n, m=1, z=3, ns=4, r=r, rz=rz, gamma=0.9, horizon=1, seed=n)
    rng = np.random.default_rng(r)
    md["GammaInitial"] = (rng.normal(-3.0, 1.0, size=(1, n)) + 1e-2 * rng.normal(size=(r, n))).astype(np.float32)
    G, pi, stats, Go, po = backups(md, npp.SCORING_FP16, 1)
    assert stats[-1]["rowsMultiCand"] > 0
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


def test_shared_memory_limits_across_threads():
    """Solvers on several threads launch the same kernels with different
    amounts of shared memory: none takes the limit from under another."""
    from nova_gb300.pomdp_pbvi import solve_batched
    models = [synth.random_pomdp(n=n, m=2, z=2, ns=3, r=40, rz=min(n, 9), gamma=0.9, horizon=40, seed=n)
              for n in (700, 820, 640, 900, 760, 850, 670, 880, 720, 810, 650, 910, 770, 840, 680, 890)]
    ps = [POMDP.from_arrays(md) for md in models]
    for p in ps:
        p.initialize_gpu()
    alone = [POMDPPBVIGPU(p).solve() for p in ps]
    for _ in range(4):
        for got, want in zip(solve_batched(ps, scoring=npp.SCORING_EXACT), alone):
            np.testing.assert_array_equal(bits(got.gamma_array()), bits(want.gamma_array()))
            np.testing.assert_array_equal(got.pi_array(), want.pi_array())


@pytest.mark.parametrize("n,r,m,z", [(5, 33, 2, 9), (64, 130, 1, 1), (1000, 37, 3, 33), (3585, 41, 1, 2), (7200, 65, 1, 3),
                                     (12300, 40, 1, 2), (16384, 64, 2, 1)])
@pytest.mark.parametrize("mode", [npp.SCORING_FP16, npp.SCORING_BF16])
def test_scoring_operand(n, r, m, z, mode):
    """Four, two and one belief per building block with remainders, more
    observations than warps, states past a whole number of vectors; scored on
    the tensor cores throughout."""
    md = synth.random_pomdp(n=n, m=m, z=z, ns=min(3, n), r=r, rz=min(5, n), gamma=0.9, horizon=1, seed=n)
    md["GammaInitial"] = np.random.default_rng(r).normal(-3.0, 1.0, size=(r, n)).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 1)
    assert stats[-1]["scoring"] == mode and stats[-1]["rowsOverflow"] == 0
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("mode", [npp.SCORING_EXACT, npp.SCORING_FP16])
@pytest.mark.parametrize("n,z,r,rz", [(12, 1, 40, 3), (30, 32, 50, 5), (40, 33, 70, 40), (25, 71, 35, 25), (9000, 3, 33, 4)])
def test_choices_below_the_sentinel(n, z, r, rz, mode):
    """(Belief, action, observation) rows without an alpha above -1e10, alone
    and in runs, first and later, past 32 observations: the previous
    observation's choice stands."""
    md = synth.random_pomdp(n=n, m=2, z=z, ns=2, r=r, rz=rz, gamma=0.9, horizon=2, seed=n + z)
    rng = np.random.default_rng(z)
    md["O"] = np.where(rng.uniform(size=md["O"].shape) < 0.5, md["O"], 0).astype(np.float32)
    G = rng.normal(-3.0, 1.0, size=(r, n))
    G[:, n // 3:] -= 1e13 * rng.uniform(0.5, 1, size=(r, n - n // 3))
    md["GammaInitial"] = G.astype(np.float32)
    got, pi, stats, want, po = backups(md, mode, 2)
    np.testing.assert_array_equal(bits(got), bits(want))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("n,m,z,ns,r", [(3, 2, 1, 2, 5), (31, 1, 9, 4, 70), (97, 3, 17, 5, 33), (1430, 2, 8, 6, 20),
                                        (1500, 2, 3, 7, 19), (3100, 2, 5, 3, 9)])
def test_reverse_steps(n, m, z, ns, r):
    """Four, two and one belief per block, beliefs without an adjoint among
    them, observations and states that are no multiple of a tile, ragged
    successor rows: against the FP64 reverse mode with the same selections
    (which differs by the FP32 rounding of the alphas)."""
    from nova_gb300.pomdp_adjoint import pbvi_record_and_adjoint
    md = synth.random_pomdp(n=n, m=m, z=z, ns=ns, r=r, rz=min(5, n), gamma=0.9, horizon=4, seed=n + r)
    rng = np.random.default_rng(n)
    length = rng.integers(1, ns + 1, size=(n, m, 1))
    md["S"] = np.where(np.arange(ns) < length, md["S"], -1).astype(np.int32)
    md["GammaInitial"] = rng.normal(-3.0, 1.0, size=(r, n)).astype(np.float32)
    b0 = np.full(n, 1.0 / n, np.float32)
    V, istar, dR, dT, dO, dG, acts, sels = pbvi_record_and_adjoint(md, b0, 4, 2)
    want = orc.pbvi_fixed_reverse_f64(md, md["GammaInitial"], acts, sels, b0, istar=istar)
    assert abs(V - want[0]) <= 1e-4
    for x, y in zip((dR, dT, dO, dG), want[1:]):
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max()


@pytest.mark.parametrize("mode", [npp.SCORING_FP16, npp.SCORING_BF16])
@pytest.mark.parametrize("r,spread", [(33, 1.0), (290, 1e-2), (1030, 1e-3), (1030, 1e-7)])
def test_sorted_lists(r, spread, mode):
    """Deep contractions: lists with room, full ones that lose their least
    entries, and rows with more candidates than lists hold."""
    md = synth.random_pomdp(n=2100, m=1, z=2, ns=4, r=r, rz=9, gamma=0.9, horizon=1, seed=r)
    rng = np.random.default_rng(r)
    md["GammaInitial"] = (rng.normal(-3.0, 1.0, size=(1, 2100)) + spread * rng.normal(size=(r, 2100))).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 1)
    assert stats[-1]["scoring"] == mode
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("mode", [npp.SCORING_EXACT, npp.SCORING_FP16, npp.SCORING_BF16])
@pytest.mark.parametrize("n,r,rz,distinct", [(256, 40, 256, 1), (300, 64, 300, 2), (400, 40, 400, 1), (430, 33, 430, 5),
                                             (512, 40, 300, 1), (640, 33, 263, 4), (230, 50, 220, 3), (400, 3, 400, 3),
                                             (1024, 40, 150, 2)])
def test_exact_scan_wide_beliefs(n, r, rz, distinct, mode):
    """Few distinct alphas (the default initial set has one) and beliefs of
    hundreds of states, whose lists leave no room for four alphas to a block
    of 128 threads, beside narrow beliefs."""
    md = synth.random_pomdp(n=n, m=2, z=2, ns=4, r=r, rz=rz, gamma=0.9, horizon=2, seed=n + r)
    if distinct > 1:
        pool = np.random.default_rng(n).normal(-3.0, 1.0, size=(distinct, n)).astype(np.float32)
        md["GammaInitial"] = pool[np.arange(r) % distinct]
    md["Z"][1:r // 2, 7:], md["B"][1:r // 2, 7:] = -1, 0.0
    G, pi, stats, Go, po = backups(md, mode, 2)
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


def test_expand_then_solve():
    """A distinct expansion widens the beliefs to hundreds of states; solves
    from the default initial alphas, on device and host arrays and batched."""
    from nova_gb300.pomdp_pbvi import POMDPPBVICPU, solve_batched
    md = synth.random_pomdp(n=512, m=3, z=4, ns=12, r=40, rz=32, gamma=0.9, horizon=3, seed=4)
    p = POMDP.from_arrays(md)
    p.expand(method="distinct_beliefs")
    md.update({k: v for k, v in p.arrays().items() if k in ("Z", "B")}, r=int(p.r), rz=int(p.rz))
    assert md["r"] > 40 and 212 <= md["rz"] <= 343
    G, pi = orc.pbvi_solve(md, GammaInitial=np.full((md["r"], 512), md["GammaInitial"][0, 0], np.float32))
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    for pol in [POMDPPBVIGPU(p).solve(), POMDPPBVICPU(p).solve(), solve_batched([p])[0],
                solve_batched([p], persistent=True)[0]]:
        np.testing.assert_array_equal(bits(pol.gamma_array()), bits(G))
        np.testing.assert_array_equal(pol.pi_array(), pi)


@pytest.mark.parametrize("n,rz,mode", [(7000, 6150, npp.SCORING_FP16), (7000, 6150, npp.SCORING_EXACT),
                                       (8192, 7000, npp.SCORING_BF16), (12200, 12200, npp.SCORING_FP16),
                                       (30000, 29900, npp.SCORING_FP16), (30000, 29900, npp.SCORING_BF16)])
def test_wide_beliefs_without_open_rows(n, rz, mode):
    """Beliefs of more states than a block of the row scan holds without
    raising its limit, or at all, and alphas far enough apart that no row is
    left to it."""
    r = 64
    md = synth.random_pomdp(n=n, m=1, z=2, ns=2, r=r, rz=rz, gamma=0.9, horizon=1, seed=n)
    rng = np.random.default_rng(n)
    md["GammaInitial"] = (rng.normal(0.0, 0.1, size=(r, n)) + rng.permutation(r)[:, None]).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 1)
    assert stats[-1]["scoring"] == mode and stats[-1]["rowsOverflow"] == 0
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


def test_recorded_graph_updates_after_ordinary_ones():
    """Graph mode switched off for an update whose alphas repeat, and on
    again: the replayed update's recorded selections are alpha indices."""
    import torch
    md = synth.random_pomdp(n=40, m=3, z=4, ns=5, r=200, rz=6, gamma=0.95, horizon=14, seed=8)
    md["Z"], md["B"] = np.repeat(md["Z"][:100], 2, axis=0), np.repeat(md["B"][:100], 2, axis=0)
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    s = POMDPPBVIGPU(p)
    s.set_scoring(npp.SCORING_FP16)
    acts = torch.empty((14, 200), dtype=torch.int32, device="cuda")
    sels = torch.empty((14, 200, 4), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    replayed = []
    for t in range(14):
        s.set_graph(t != 11)
        assert npp._nova.pomdp_pbvi_update_record_gpu(s.pomdpPtr, s, acts[t].data_ptr(), sels[t].data_ptr()) == 0
        replayed.append(s.stats()["msTotal"] == 0.0)
    assert replayed[10] and not replayed[11] and replayed[12] and replayed[13]
    G, acts_o, sels_o = orc.pbvi_record(md, 14)
    np.testing.assert_array_equal(acts.cpu().numpy(), acts_o)
    np.testing.assert_array_equal(sels.cpu().numpy(), sels_o)


@pytest.mark.parametrize("n,r", [(15000, 3), (15000, 700)])
def test_zero_beliefs_of_many_states(n, r):
    """Beliefs without a nonzero, alone in a tile of beliefs, where the states
    are too many for alphas in shared memory: V = 0 with alpha 0's action."""
    import torch
    from nova_gb300 import nova_pomdp_alpha_vectors as npav
    rng = np.random.default_rng(n)
    G = rng.uniform(-5, 5, size=(r, n)).astype(np.float32)
    pi = rng.integers(1, 9, size=r).astype(np.int32)
    B = np.zeros((130, n), np.float32)
    B[128, 7], B[129, n - 1] = 0.5, 1.0
    dG, dB, dPi = (torch.as_tensor(x, device="cuda") for x in (G, B, pi))
    dV, dA = torch.empty(130, device="cuda"), torch.empty(130, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert npav._nova.pomdp_alpha_vectors_value_batched_gpu(dG.data_ptr(), dPi.data_ptr(), r, n, dB.data_ptr(), 130,
                                                            dV.data_ptr(), dA.data_ptr()) == 0
    for i in (0, 127, 128, 129):
        V, a = orc.alpha_value(G, pi.astype(np.uint32), B[i])
        assert bits(dV[i].cpu().numpy()) == bits(np.float32(V)) and int(dA[i]) == a, i


def test_failed_builds_leak_nothing():
    """An update that fails while its tables are built, tried again: the
    device memory in use does not grow."""
    from nova_gb300._lib import load as lib
    import torch
    md = synth.random_pomdp(n=3000, m=8, z=16, ns=16, r=64, rz=8, gamma=0.9, horizon=3, seed=1)
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    s = POMDPPBVIGPU(p)
    free = []
    for _ in range(6):
        lib().nova_gb300_inject_fault(4, 2)
        with pytest.raises(RuntimeError):
            s.update()
        lib().nova_gb300_inject_fault(0, 0)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 32 << 20
    s.update()


def test_scoring_operand_of_many_actions():
    """More actions than a grid's third dimension holds."""
    md = synth.random_pomdp(n=20, m=66000, z=1, ns=1, r=33, rz=2, gamma=0.9, horizon=1, seed=3)
    md["GammaInitial"] = np.random.default_rng(3).normal(-3.0, 1.0, size=(33, 20)).astype(np.float32)
    G, pi, stats, Go, po = backups(md, npp.SCORING_FP16, 1)
    assert stats[-1]["scoring"] == npp.SCORING_FP16
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


def test_distinct_expansion_with_little_memory():
    """The successors' buffer is made smaller where it cannot be allocated."""
    from nova_gb300._lib import load as lib
    md = synth.random_pomdp(n=60, m=2, z=5, ns=4, r=23, rz=6, gamma=0.9, horizon=2, seed=9)
    p = POMDP.from_arrays(md)
    want = orc.merge_raw_beliefs(md["Z"], md["B"], orc.expand_distinct(md))
    lib().nova_gb300_inject_fault(1, 2)
    try:
        p.expand(method="distinct_beliefs")
    finally:
        lib().nova_gb300_inject_fault(0, 0)
    out = p.arrays()
    np.testing.assert_array_equal(out["Z"], want[0])
    np.testing.assert_array_equal(bits(out["B"]), bits(want[1]))


def test_perseus_with_little_memory():
    """Fewer splits of the alphas where the buffer for all of them cannot be
    allocated (the solve's fourth allocation)."""
    from nova_gb300._lib import load as lib
    from nova_gb300.pomdp_perseus import POMDPPerseusGPU
    md = synth.random_pomdp(n=40, m=2, z=3, ns=4, r=90, rz=9, gamma=0.9, horizon=4, seed=6)
    Go, po = orc.perseus_solve(md, seed=3)
    p = POMDP.from_arrays(md)
    p.initialize_gpu()
    alg = POMDPPerseusGPU(p, GammaInitial=md["GammaInitial"])
    orc.lib().oracle_srand(3)
    lib().nova_gb300_inject_fault(1, 4)
    try:
        pol = alg.solve()
    finally:
        lib().nova_gb300_inject_fault(0, 0)
    np.testing.assert_array_equal(bits(pol.gamma_array()), bits(Go))
    np.testing.assert_array_equal(pol.pi_array(), po)


@pytest.mark.parametrize("n,m,z,ns,r", [(30, 1, 2, 3, 300), (5, 1, 1, 2, 310), (33, 3, 2, 5, 300), (1026, 2, 3, 9, 150),
                                        (70, 2, 17, 31, 401), (7300, 2, 2, 4, 30)])
def test_replayed_groups(n, m, z, ns, r):
    """The most beliefs that are replayed one per block, and more: four of one
    action, their alphas in and out of shared memory."""
    test_replayed_backups(n, m, z, ns, r)


@pytest.mark.parametrize("n,m,z,ns,r", [(20, 2, 3, 3, 2424), (20, 2, 3, 3, 2428), (129, 3, 9, 4, 1211), (2000, 1, 2, 3, 161),
                                        (3, 1, 3100, 2, 2450), (14500, 1, 2, 2, 30)])
def test_reverse_groups(n, m, z, ns, r):
    """One belief per block up to a wave of blocks, four beyond it, two with
    thousands of observations, and the most states that are accepted."""
    test_reverse_steps(n, m, z, ns, r)


@pytest.mark.parametrize("n,r,rz,mode", [(130, 300, 97, npp.SCORING_FP16), (130, 300, 97, npp.SCORING_BF16),
                                         (300, 200, 290, npp.SCORING_FP16), (300, 200, 290, npp.SCORING_BF16),
                                         (70, 1100, 33, npp.SCORING_BF16), (2100, 300, 300, npp.SCORING_BF16)])
def test_merge_after_open_rows(n, r, rz, mode):
    """Updates after one that left more than 1 % of its rows open keep the
    alpha-contiguous table: rows with up to and more than 32 candidates, over
    supports around multiples of 8, narrow and wide."""
    md = synth.random_pomdp(n=n, m=2, z=3, ns=12, r=r, rz=rz, gamma=0.9, horizon=6, seed=r)
    md["Z"][r // 3:r // 2, 5:], md["B"][r // 3:r // 2, 5:] = -1, 0.0
    md["GammaInitial"] = np.random.default_rng(2).normal(-3.0, 1.0, size=(r, n)).astype(np.float32)
    G, pi, stats, Go, po = backups(md, mode, 6)
    assert any(s["rowsOverflow"] > 0.01 * 6 * r and t["rowsMultiCand"] > 0 for s, t in zip(stats, stats[1:]))
    np.testing.assert_array_equal(bits(G), bits(Go))
    np.testing.assert_array_equal(pi, po)


@pytest.mark.parametrize("r,n,count,nz", [(65, 14500, 63, 14500), (64, 14500, 65, 0), (129, 14470, 129, 9), (3000, 50, 900, 50)])
@pytest.mark.parametrize("odd", [False, True])
def test_dense_belief_tiles(r, n, count, nz, odd):
    """Tiles of 64 and 128 beliefs around their edges, where states are too
    many for the lists' kernel or beliefs have too many nonzeros."""
    test_belief_values(r, n, count, nz, odd)


@pytest.mark.parametrize("what", ["pema", "random", "exact"])
def test_shared_memory_just_below_the_default_limit(what):
    """Launches whose dynamic shared memory stays below 48 KB while the kernel's
    own takes the sum above it, first in a process (the limit, once raised,
    stays raised)."""
    import subprocess, sys
    from conftest import ROOT
    code = {"pema": "import ctypes as ct\n"
                    "from nova_gb300 import nova_pomdp as npm, nova_pomdp_alpha_vectors as npav\n"
                    "md = synth.random_pomdp(n=3000, m=1, z=2, ns=2, r=5, rz=3, gamma=0.9, horizon=2, seed=1)\n"
                    "G, pi = np.zeros((5, 3000), np.float32), np.zeros(5, np.uint32)\n"
                    "pol = npav.NovaPOMDPAlphaVectors()\n"
                    "pol.n, pol.m, pol.r = 3000, 1, 5\n"
                    "pol.Gamma, pol.pi = G.ctypes.data_as(ct.POINTER(ct.c_float)), pi.ctypes.data_as(ct.POINTER(ct.c_uint))\n"
                    "assert npm._nova.pomdp_expand_pema_cpu(POMDP.from_arrays(md), ct.byref(pol)) == 0\n",
            "random": "md = synth.random_pomdp(n=3071, m=1, z=2, ns=2, r=5, rz=3, gamma=0.9, horizon=2, seed=1)\n"
                      "POMDP.from_arrays(md).expand(method='random', numBeliefsToAdd=4)\n",
            "exact": "md = synth.random_pomdp(n=400, m=1, z=16, ns=365, r=9, rz=3, gamma=0.9, horizon=1, seed=1)\n"
                     "p = POMDP.from_arrays(md)\n"
                     "p.initialize_gpu()\n"
                     "alg = POMDPPBVIGPU(p)\n"
                     "alg.set_scoring(npp.SCORING_EXACT)\n"
                     "alg.set_table(npp.TABLE_NEVER)\n"
                     "alg.update()\n"}[what]
    code = ("import numpy as np\nfrom nova_gb300 import synth, nova_pomdp_pbvi as npp\nfrom nova_gb300.pomdp import POMDP\n"
            "from nova_gb300.pomdp_pbvi import POMDPPBVIGPU\n" + code)
    assert subprocess.run([sys.executable, "-c", code], cwd=ROOT, timeout=120).returncode == 0


@pytest.mark.parametrize("n,m,z,r,rz,odd", [(127, 2, 3, 5, 6, ""), (129, 1, 4, 40, 129, ""), (3000, 2, 2, 70, 4, ""),
                                            (3000, 2, 2, 9, 2000, "same"), (2500, 1, 3, 70, 3, "infinite"),
                                            (300, 8, 16, 257, 9, ""), (300, 8, 16, 255, 9, "same")])
def test_distinct_expansion_forms(n, m, z, r, rz, odd):
    """Rows by a warp and by a thread each, and exact sums over the nonzeros
    (many beliefs equally far) and over all states."""
    test_distinct_expansion(n, m, z, r, rz, odd)


@pytest.mark.parametrize("n,z", [(5, 2), (127, 3), (128, 9), (129, 64), (700, 65), (2051, 4), (14272, 2)])
def test_random_expansion_sums(n, z):
    """Observation probabilities by a warp and by a thread each, chunks of 128
    states with remainders, and the most states that are accepted."""
    from nova_gb300 import nova_pomdp as npm
    md = synth.random_pomdp(n=n, m=2, z=z, ns=min(4, n), r=7, rz=min(5, n), gamma=0.9, horizon=9, seed=n)
    npm._nova.nova_gb300_expand_seed(1, 77)
    try:
        p = POMDP.from_arrays(md)
        p.expand(method="random", numBeliefsToAdd=30)
    finally:
        npm._nova.nova_gb300_expand_seed(0, 0)
    Z, B = orc.merge_raw_beliefs(md["Z"], md["B"], orc.expand_random(md, 30, 77))
    out = p.arrays()
    np.testing.assert_array_equal(out["Z"], Z)
    np.testing.assert_array_equal(bits(out["B"]), bits(B))


@pytest.mark.parametrize("n,r,pr,low", [(31, 3, 9, 0), (128, 40, 40, 3), (129, 9, 300, 7), (700, 260, 65, 2)])
def test_pema_alpha_search(n, r, pr, low):
    """The last alpha with a product below -1e10 anywhere: none, few, in the
    first and last states."""
    import ctypes as ct
    from nova_gb300 import nova_pomdp as npm, nova_pomdp_alpha_vectors as npav
    md = synth.random_pomdp(n=n, m=2, z=3, ns=3, r=r, rz=4, gamma=0.9, horizon=3, seed=n)
    G = np.random.default_rng(n).normal(size=(pr, n)).astype(np.float32)
    for k in range(low):
        G[(5 * k) % pr, (n - 1) * (k % 2)::17] = -1e13
    pi = np.zeros(pr, np.uint32)
    pol = npav.NovaPOMDPAlphaVectors()
    pol.n, pol.m, pol.r = n, 2, pr
    pol.Gamma, pol.pi = G.ctypes.data_as(ct.POINTER(ct.c_float)), pi.ctypes.data_as(ct.POINTER(ct.c_uint))
    p = POMDP.from_arrays(md)
    assert npm._nova.pomdp_expand_pema_cpu(p, ct.byref(pol)) == 0
    Z, B = orc.merge_raw_beliefs(md["Z"], md["B"], orc.expand_pema(md, G)[None, :])
    out = p.arrays()
    np.testing.assert_array_equal(out["Z"], Z)
    np.testing.assert_array_equal(bits(out["B"]), bits(B))


@pytest.mark.parametrize("n,m,ns,horizon", [(30000, 16, 8, 3), (51999, 10, 4, 2), (51999, 7, 6, 3), (52000, 8, 6, 3),
                                            (100000, 4, 9, 2), (250000, 2, 7, 4)])
def test_resident_sweep_limits(n, m, ns, horizon):
    """Models just within and beyond what the resident sweeps take."""
    test_resident_sweeps(n, m, ns, horizon, "gpu")
