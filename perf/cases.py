"""Performance cases: what a program that simulates with this engine has it do.

Four ways of use, each through the public entry points:

  run    a molecular-dynamics run.  One simulation: set_state, step, get_state.
         A batch, or a context with quasi-adiabatic contacts (which carry over
         from call to call): the packed history of every replica goes up, all
         replicas step, and the packed history comes back.
  score  forces and energies of a conformation: set_state, eval_forces.
  serve  simulation requests submitted together to the serving loop, until
         every result is there.
  pairs  the allocation-free pair search on the caller's device arrays.

Systems have the shapes of the configurations in xmd_gb300/synth.py and of
bench.py: one chain of 100 beads; 16 x 500 in a 300 A box; 512 x 60 at
1e-3 A^-3 with quasi-adiabatic contacts; 256 single chains of 50 to 800 beads;
requests of many chains of 30 to 1500 beads.  Chains are grown here, on the
GPU, from the seed: a native conformation (bond angles of a protein's C-alpha
trace, confined to a globule of 1 bead per 120 A^3), and for "coil" a chain
with the native's local geometry under thermal noise and no globule, which is
where a folding run spends its time (few native contacts closed, short Verlet
rows); "folded" starts in the native conformation (all contacts closed, long
rows).  Velocities are Maxwell's at the run's temperature, so no case starts
with the relaxation of an extended walk.

FP64 runs return their state in FP64.  Mixed runs return positions and
velocities as single-precision frames, the precision in which trajectory files
hold them and in which the forces behind them are computed.

`exact` restates the same calls in 64-bit torch: list rules, forces, the
quasi-adiabatic state machine, the generator and the Gear predictor-corrector.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from xmd_gb300 import Engine, Server, abi

A = 0.2                      # one angstrom in the engine's length unit (5 A)
BOND = 3.8 * A
DT = 5e-3
GAMMA = 2.0
GLOBULE = 1.0 / 120.0        # beads per A^3 of a native globule
MIN_SEP = 4.8 * A            # closest approach of non-bonded beads of a native conformation
COIL_SEP = 7.0 * A           # and of a coil: with 0.93 of the native distance for contacts, no
CLOSE = 0.93                 # pair starts deep in its repulsion

# the force field of every case (xmd_gb300/synth.py's configurations)
YAML = """
langevin:
  enabled: true
  gamma factor: 2.0 1/tau
  temperature: 0.35 eps/kB
integrator:
  dt: 5e-3 tau
tether forces:
  enabled: true
  H1: 100 eps/A**2
native angles:
  enabled: true
  k: 30.0 eps/rad**2
complex native dihedrals:
  enabled: true
  CDA: 0.66 eps/rad**2
  CDB: 0.66 eps/rad**2
native contacts:
  enabled: true
  lj depth: 1 eps
Pauli exclusion:
  enabled: true
  r_excl: 4.0 A
  depth: 1.0 eps
"""
ES_ON = """
const ES:
  enabled: true
  screening distance: 10.0 A
  permittivity: 80.0 eps_0
"""
ES_OFF = """
const ES:
  enabled: false
neighbor list:
  cutoff: 18 A
  skin: 2 A
"""
QA_ON = "quasi-adiabatic potential:\n  enabled: true\n"
QA_OFF = "quasi-adiabatic potential:\n  enabled: false\n"
ES_VF = 1.0 / (4.0 * math.pi * 0.1512879689175476)   # 1 / (4 pi 80 eps_0) in the engine's units


# ---- cases -----------------------------------------------------------------------

def listed():
    return [
        # one small protein, plain FP64, no box, no charges: the smallest run,
        # where every step is latency
        {"name": "single_fp64", "kind": "run", "precision": "fp64", "chains": 1, "lo": 100, "hi": 100, "replicas": 1,
         "box": 0, "es": False, "qa": False, "conf": "folded", "steps": 100},
        # a solution of proteins in a periodic box with Debye-Hueckel
        # electrostatics, in the plain FP64 path ...
        {"name": "periodic_fp64", "kind": "run", "precision": "fp64", "chains": 16, "lo": 500, "hi": 500, "replicas": 1,
         "box": 300, "es": True, "qa": False, "conf": "coil", "steps": 64},
        # ... and the same in mixed precision
        {"name": "periodic_mixed", "kind": "run", "precision": "mixed", "chains": 16, "lo": 500, "hi": 500,
         "replicas": 1, "box": 300, "es": True, "qa": False, "conf": "coil", "steps": 128},
        # an ensemble of independent folding runs of uneven lengths in one
        # context: the batched workload that the benchmark reports
        {"name": "batch_mixed", "kind": "run", "precision": "mixed", "chains": 1, "lo": 50, "hi": 800, "replicas": 256,
         "box": 0, "es": True, "qa": False, "conf": "coil", "steps": 128},
        # the same ensemble in plain FP64
        {"name": "batch_fp64", "kind": "run", "precision": "fp64", "chains": 1, "lo": 50, "hi": 800, "replicas": 256,
         "box": 0, "es": True, "qa": False, "conf": "coil", "steps": 48},
        # a smaller ensemble of native-state runs: every contact closed, the
        # longest rows
        {"name": "batch_folded_mixed", "kind": "run", "precision": "mixed", "chains": 1, "lo": 50, "hi": 800,
         "replicas": 61, "box": 0, "es": True, "qa": False, "conf": "folded", "steps": 128},
        # many short disordered chains with quasi-adiabatic contacts, mixed
        {"name": "contacts_mixed", "kind": "run", "precision": "mixed", "chains": 512, "lo": 60, "hi": 60,
         "replicas": 1, "box": 313, "es": True, "qa": True, "conf": "coil", "steps": 64},
        # a smaller one in FP64 (whole-replica lists), with the valences that
        # its contacts leave
        {"name": "contacts_fp64", "kind": "run", "precision": "fp64", "chains": 67, "lo": 30, "hi": 60, "replicas": 1,
         "box": 145, "es": True, "qa": True, "conf": "coil", "steps": 64},
        # the largest serving request run by itself: many long chains in open
        # space, hashed cell lists
        {"name": "large_mixed", "kind": "run", "precision": "mixed", "chains": 64, "lo": 400, "hi": 1500,
         "replicas": 1, "box": 0, "es": True, "qa": False, "conf": "coil", "steps": 64},
        # rescoring a conformation: lists from scratch, forces and energies
        {"name": "score_fp64", "kind": "score", "precision": "fp64", "chains": 16, "lo": 500, "hi": 500, "replicas": 1,
         "box": 300, "es": True, "qa": False, "conf": "folded", "steps": 0},
        # the pair search on device arrays that a program owns
        {"name": "pairs", "kind": "pairs", "precision": "fp64", "chains": 512, "lo": 60, "hi": 60, "replicas": 1,
         "box": 313, "es": False, "qa": False, "conf": "coil", "steps": 0},
        # requests of one to eight chains through the serving loop
        {"name": "serve_mixed", "kind": "serve", "precision": "mixed", "chains": 8, "lo": 30, "hi": 500,
         "replicas": 12, "box": 0, "es": True, "qa": False, "conf": "coil", "steps": 256},
    ]


def draw(rng):
    def logi(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["single", "periodic", "batch", "batch", "contacts", "large", "score", "pairs", "serve"])
    c = {"kind": "run", "precision": rng.choice(["fp64", "mixed", "mixed"]), "replicas": 1, "box": 0, "es": True,
         "qa": False, "conf": rng.choice(["coil", "folded"])}
    if what == "single":
        n = logi(50, 800)
        c.update(chains=1, lo=n, hi=n, es=rng.random() < 0.5, steps=rng.randint(40, 200))
    elif what == "periodic":
        chains, lo = rng.randint(5, 40), logi(100, 400)
        c.update(chains=chains, lo=lo, hi=rng.randint(lo, 600), box=300 + rng.randint(0, 80), steps=rng.randint(32, 128))
    elif what == "batch":
        c.update(chains=1, lo=logi(30, 100), hi=logi(200, 800), replicas=logi(16, 256), steps=rng.randint(24, 48))
    elif what == "contacts":
        chains = logi(20, 512)
        c.update(chains=chains, lo=30, hi=rng.randint(31, 60), conf="coil", qa=True, steps=rng.randint(24, 64))
        c["box"] = int((chains * c["hi"] / 1e-3) ** (1 / 3)) + 1
    elif what == "large":
        c.update(precision="mixed", conf="coil", chains=logi(8, 50), lo=logi(30, 300), hi=rng.randint(400, 1500),
                 steps=rng.randint(24, 64))
    elif what == "score":
        chains = rng.randint(1, 30)
        c.update(kind="score", chains=chains, lo=logi(50, 500), hi=501, box=rng.choice([0, 340]), steps=0)
    elif what == "pairs":
        chains, lo = logi(8, 1000), rng.randint(30, 45)
        c.update(kind="pairs", precision="fp64", conf="coil", chains=chains, lo=lo, hi=rng.randint(lo, 61), es=False,
                 steps=0)
        c["box"] = rng.choice([0, 1]) * (int((chains * c["hi"] / 1e-3) ** (1 / 3)) + 1)
    else:
        c.update(kind="serve", conf="coil", chains=rng.randint(2, 12), lo=30, hi=logi(100, 500),
                 replicas=rng.randint(4, 16), steps=rng.randint(100, 256))
        c["precision"] = "mixed"
    return c


def _sizes(case):
    """Chain lengths of each replica (log-uniform, as the configurations draw
    them): the case's own, the same for every seed."""
    g = np.random.default_rng([case["chains"], case["lo"], case["hi"], case["replicas"], case["box"]])
    out = []
    for _ in range(case["replicas"]):
        nch = case["chains"] if case["kind"] != "serve" else int(g.integers(1, case["chains"] + 1))
        out.append([int(x) for x in np.floor(np.exp(g.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), nch)))])
    return out


def work(case):
    sizes = _sizes(case)
    n = sum(sum(s) for s in sizes)
    s = max(1, case["steps"])
    if case["kind"] == "pairs":
        # positions and ids in; ~30 partners a bead out; ~130 candidates a bead tested
        return {"bytes": n * (24.0 + 8.0 + 30.0 * 8.0), "flops": n * 130.0 * 12.0}
    # the state in and out once, the topology (bonded parameters, ~5 native
    # contacts a bead); per step and bead ~90 operations of the integrator,
    # ~400 of the bonded terms and noise, ~10 pairs of ~40
    state = 144.0 if case["kind"] != "score" else 24.0
    return {"bytes": n * (2.0 * state + 60.0 + 5.0 * 12.0), "flops": n * s * (90.0 + 400.0 + 400.0)}


# ---- chains ------------------------------------------------------------------------

def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _place(p1, p2, p3, theta, phi):
    """The bead after p1, p2, p3 at BOND with bond angle theta and dihedral phi
    (leading dimensions broadcast)."""
    b2 = _unit(p3 - p2)
    n = _unit(torch.linalg.cross(p2 - p1, b2, dim=-1))
    m = torch.linalg.cross(n, b2, dim=-1)
    ct, st = torch.cos(theta)[..., None], torch.sin(theta)[..., None]
    cp, sp = torch.cos(phi)[..., None], torch.sin(phi)[..., None]
    return p3 + BOND * (-ct * b2 + st * cp * m + st * sp * n)


def _grow(lens, gen, theta, phi, start, confine, box, rep, sep):
    """Grows every chain at once, bead by bead: for bead k the first of the
    tries theta[k], phi[k] ([C, K] each) that keeps its distance from earlier
    beads (of its own chain when `rep` is None, of every chain of its replica
    rep[c] otherwise; bonded neighbours of up to two bonds excepted) and, when
    `confine`, stays in its globule; otherwise the least bad.  The distance is
    sep[c, k, j] between beads k and j of chain c (MIN_SEP when sep is None)
    and COIL_SEP between chains."""
    dev = start.device
    C, L = len(lens), max(lens)
    ln = torch.tensor(lens, device=dev)
    K = theta.shape[2]
    pos = torch.full((C, L, 3), 1e6, dtype=torch.float64, device=dev)
    pos[:, 0] = start
    d = _unit(torch.randn(C, 3, dtype=torch.float64, device=dev, generator=gen))
    pos[:, 1] = pos[:, 0] + BOND * d
    q = _unit(torch.linalg.cross(d, _unit(torch.randn(C, 3, dtype=torch.float64, device=dev, generator=gen)), dim=-1))
    radius = ((3.0 * ln / (4.0 * math.pi * GLOBULE)) ** (1.0 / 3.0) * A).clamp(min=2.0 * BOND)
    virt = pos[:, 0] + BOND * q      # a bead before the first, so that bead 2 has a plane
    flat = pos.float()               # FP32 copy of every bead for the clash tests
    if rep is not None:
        rt = torch.tensor(rep, device=dev)
        skip = (rt[:, None] != rt[None]) | torch.eye(C, dtype=torch.bool, device=dev)
        skip = skip[:, None, :, None]
    for k in range(2, L):
        p1 = pos[:, k - 3] if k >= 3 else virt
        cand = _place(p1[:, None], pos[:, k - 2][:, None], pos[:, k - 1][:, None], theta[k], phi[k])
        c32 = cand.float()
        score = torch.zeros(C, K, device=dev)
        if k >= 3:
            d2 = torch.zeros(C, K, k - 2, device=dev)
            for a in range(3):
                x = c32[:, :, a, None] - flat[:, None, :k - 2, a]
                d2.addcmul_(x, x)
            gap = d2.sqrt_() - (MIN_SEP if sep is None else sep[:, k, None, :k - 2])
            score = gap.amin(dim=2).clamp(max=0.0)
        if rep is not None:
            old = flat[:, :k].reshape(-1, 3)
            d2 = torch.zeros(C * K, old.shape[0], device=dev)
            for a in range(3):
                x = c32.view(-1, 3)[:, a:a + 1] - old[None, :, a]
                if box:
                    x -= box * torch.round(x / box)
                d2.addcmul_(x, x)
            d2 = d2.view(C, K, C, k).masked_fill_(skip, 1e6)
            score = torch.minimum(score, (d2.view(C, K, -1).amin(dim=2).sqrt() - COIL_SEP).clamp(max=0.0))
        if confine:
            score = score - ((cand - start[:, None]).norm(dim=2).float() - radius[:, None]).clamp(min=0.0)
        pick = torch.where((score >= 0).any(dim=1), (score >= 0).int().argmax(dim=1), score.argmax(dim=1))
        new = cand[torch.arange(C, device=dev), pick]
        new = torch.where((k < ln)[:, None], new, torch.full_like(new, 1e6))
        pos[:, k] = new
        flat[:, k] = new.float()
    return pos


def _geometry(p):
    """Bond angles and dihedrals along [C, L, 3] chains."""
    b = p[:, 1:] - p[:, :-1]
    x = torch.linalg.cross(b[:, :-1], b[:, 1:], dim=-1)
    th = torch.atan2(x.norm(dim=-1), -(b[:, :-1] * b[:, 1:]).sum(-1))
    t = (x[:, :-1] * b[:, 2:]).sum(-1) * b[:, 1:-1].norm(dim=-1)
    return th, torch.atan2(t, (x[:, :-1] * x[:, 1:]).sum(-1))


def _systems(case, seed):
    """The replicas of a case as the objects that Engine.add_system takes, with velocities in .v."""
    sizes = _sizes(case)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(1_000_003 * (seed % 1_000_000) + 17)
    g = np.random.default_rng([13, seed])
    lens = [x for s in sizes for x in s]
    C, L = len(lens), max(lens)
    box = case["box"] * A

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, dtype=torch.float64, device=dev, generator=gen)

    zero = torch.zeros(C, 3, dtype=torch.float64, device=dev)
    native = _grow(lens, gen, uni(1.45, 2.55, L, C, 24), uni(-math.pi, math.pi, L, C, 24), zero, True, 0.0, None,
                   None)
    th0, ph0 = _geometry(native)
    # distances within every native chain; its contacts are beads closer than
    # 7.5 A and three or more apart
    dn = torch.zeros(C, L, L, dtype=torch.float64, device=dev)
    for a in range(3):
        x = native[:, :, None, a] - native[:, None, :, a]
        dn.addcmul_(x, x)
    dn.sqrt_()
    # where each chain starts: lattice points of the replica's cube, shuffled
    starts = []
    for s in sizes:
        edge = box if box else max((sum(s) / 1e-3) ** (1 / 3) * A, 1e-9)
        m = math.ceil(len(s) ** (1 / 3) - 1e-9)
        if case["conf"] == "folded" and not box:
            edge = max(edge, m * (2.2 * (3.0 * max(s) / (4.0 * math.pi * GLOBULE)) ** (1 / 3) * A + 2.0))
        pts = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
        starts.append((pts[g.permutation(len(pts))[:len(s)]] + 0.5) * (edge / m) - edge / 2)
    start = torch.tensor(np.concatenate(starts), device=dev)
    if case["conf"] == "folded":
        mid = [native[c, :n].mean(dim=0) for c, n in enumerate(lens)]
        conf = native + (start - torch.stack(mid))[:, None]
    else:
        K = 32
        sd = torch.tensor([0.08, 0.45], dtype=torch.float64, device=dev)
        nt = torch.randn(L, C, K, dtype=torch.float64, device=dev, generator=gen) * sd[0]
        nf = torch.randn(L, C, K, dtype=torch.float64, device=dev, generator=gen) * sd[1]
        nf[:, :, 8:] *= 3.0     # the later tries wander further, to get out of dead ends
        nf[:, :, 18:] *= 2.0
        nt[:, :, 18:] *= 4.0
        th = torch.full((L, C), 2.0, dtype=torch.float64, device=dev)
        ph = torch.zeros(L, C, dtype=torch.float64, device=dev)
        th[2:] = th0.T
        ph[3:] = ph0.T
        conf = _grow(lens, gen, (th[:, :, None] + nt).clamp(1.3, 2.7), ph[:, :, None] + nf, start, False, box,
                     None if C == len(sizes) else [r for r, s in enumerate(sizes) for _ in s],
                     (CLOSE * dn).clamp(max=COIL_SEP).float())
    at = torch.arange(L, device=dev)
    ln = torch.tensor(lens, device=dev)
    close = (dn < 7.5 * A) & (at[None, :] - at[:, None] >= 3) & (at[None, None, :] < ln[:, None, None])
    nc = close.nonzero()
    nd = dn[nc[:, 0], nc[:, 1], nc[:, 2]].cpu().numpy()
    del dn, close
    nc = nc.cpu().numpy()
    cut = np.searchsorted(nc[:, 0], np.arange(C + 1))
    conf, th0, ph0 = (x.cpu().numpy() for x in (conf, th0, ph0))
    T = g.uniform(0.3, 0.6, len(sizes)) if case["replicas"] > 1 else np.full(len(sizes), 0.35)

    out, c0 = [], 0
    for r, s in enumerate(sizes):
        n = sum(s)
        off = np.concatenate([[0], np.cumsum(s)[:-1]])
        chain = np.repeat(np.arange(len(s)), s).astype(np.int32)
        seq = np.concatenate([np.arange(x) for x in s]).astype(np.int32)
        if case["qa"]:
            atype = g.integers(0, 20, n).astype(np.uint8)
        else:   # charge +-1 with probability 0.1 each
            u = g.random(n)
            atype = np.where(u < 0.1, 11, np.where(u < 0.2, 5, 0)).astype(np.uint8)
        nat = [[], [], []]
        for c, o in enumerate(off):
            k = slice(cut[c0 + c], cut[c0 + c + 1])
            nat[0].append(nc[k, 1] + o), nat[1].append(nc[k, 2] + o), nat[2].append(nd[k])
        rows = lambda k: np.concatenate([o + np.arange(max(0, m - k)) for o, m in zip(off, s)]).astype(np.int32)  # noqa: E731
        t, a, d = rows(1), rows(2), rows(3)
        out.append(SimpleNamespace(
            n=n, chain=chain, seq=seq, atype=atype, cell=np.full(3, float(box)),
            # (bonds and angles vibrate: tethers at sqrt(T / H1) ~ 0.01 units)
            r=np.concatenate([conf[c0 + c, :m] for c, m in enumerate(s)]) + 0.01 * g.normal(size=(n, 3)),
            v=g.normal(size=(n, 3)) * math.sqrt(T[r]),
            tethers=(t, t + 1, np.full(len(t), BOND)),
            angles=(a, a + 1, a + 2, np.concatenate([th0[c0 + c, :m - 2] for c, m in enumerate(s)])),
            dihedrals=(d, d + 1, d + 2, d + 3, np.concatenate([ph0[c0 + c, :m - 3] for c, m in enumerate(s)])),
            natives=(np.concatenate(nat[0]).astype(np.int32), np.concatenate(nat[1]).astype(np.int32),
                     np.concatenate(nat[2])),
            temperature=float(T[r]), seed=int(g.integers(1, 2 ** 62))))
        c0 += len(s)
    return out


# ---- the calls ---------------------------------------------------------------------

def _yaml(case):
    return (YAML + (ES_ON if case["es"] else ES_OFF) + (QA_ON if case["qa"] else QA_OFF)
            + "engine:\n  precision: %s\n" % case["precision"])


def _packed(case):
    """Whether a run goes through the packed history of all replicas."""
    return case["kind"] == "run" and (case["replicas"] > 1 or case["qa"])


PAIR_CUTOFF = 20.0 * A


def prepare(case, seed):
    systems = _systems(case, seed)
    st = {"case": case, "systems": systems}
    if case["kind"] == "pairs":
        s = systems[0]
        st["r"] = torch.tensor(s.r, device="cuda")
        st["chain"], st["seq"] = torch.tensor(s.chain, device="cuda"), torch.tensor(s.seq, device="cuda")
        st["pairs"] = torch.zeros(128 * s.n, 2, dtype=torch.int32, device="cuda")
        st["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        st["lib"] = abi.load()
        return st
    if case["kind"] == "serve":
        st["server"] = Server(_yaml(case), hbm_budget=2 << 30, max_beads=60_000)
        return st
    e = Engine(_yaml(case))
    for s in systems:
        e.add_system(s)
    st["engine"] = e
    if _packed(case):
        n = sum(s.n for s in systems)
        y = torch.zeros(6, n, 3, dtype=torch.float64, pin_memory=True)
        y[0] = torch.from_numpy(np.concatenate([s.r for s in systems]))
        y[1] = torch.from_numpy(np.concatenate([s.v for s in systems])) * DT
        out = torch.zeros(6, n, 3, dtype=torch.float64, pin_memory=True)
        st["y"], st["out"], st["keep"] = y.numpy(), out.numpy(), (y, out)
    return st


def _frames(case, r, v):
    if case["precision"] == "fp64":
        return {"r": r, "v": v}
    return {"r": torch.from_numpy(r).float(), "v": torch.from_numpy(v).float()}


def run(st):
    case = st["case"]
    if case["kind"] == "pairs":
        s = st["systems"][0]
        abi.check(st["lib"].xmd_gpu_verlet_pairs_noalloc(
            st["r"].data_ptr(), st["chain"].data_ptr(), st["seq"].data_ptr(), s.n, abi.dptr(s.cell), PAIR_CUTOFF,
            st["pairs"].data_ptr(), st["pairs"].shape[0], st["count"].data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return {"pairs": st["pairs"], "count": st["count"]}
    if case["kind"] == "serve":
        srv = st["server"]
        ids = [srv.submit(s, case["steps"]) for s in st["systems"]]
        got = [srv.result(i) for i in ids]
        return [_frames(case, r, v) for r, v, _, _ in got]
    e = st["engine"]
    if case["kind"] == "score":
        e.set_state(0, st["systems"][0].r)
        F, V = e.eval_forces(0)
        if case["precision"] == "mixed":
            return {"F": torch.from_numpy(F).float(), "V": torch.from_numpy(V).float()}
        return {"F": F, "V": V}
    if not _packed(case):
        s = st["systems"][0]
        e.set_state(0, s.r, s.v)
        e.step(case["steps"])
        r, v, _ = e.get_state(0)
        return _frames(case, r, v)
    abi.check(e.lib.xmd_gpu_upload_history_all(e.h, abi.dptr(st["y"])))
    e.step(case["steps"])
    abi.check(e.lib.xmd_gpu_download_history_all(e.h, abi.dptr(st["out"])))
    got = _frames(case, st["out"][0], st["out"][1])
    if case["qa"] and case["precision"] == "fp64":
        got["valences"] = e.qa_sync(0)
    return got


# ---- the same in 64 bits --------------------------------------------------------------

def _near(pos, rep, box, rc):
    """Pairs i < j of the same replica closer than rc, and their distance:
    cells of at least rc, one offset at a time."""
    dev = pos.device
    p = pos - box * torch.floor(pos / box) if box else pos
    if box:
        m = max(1, int(box / rc))
        c = (p * (m / box)).long().clamp(0, m - 1)
        dims = [m] * 3
    else:
        c = ((p - p.amin(dim=0)) / rc).long() + 1
        dims = [int(x) + 2 for x in c.amax(dim=0)]

    def key(c):
        return ((rep * dims[0] + c[:, 0]) * dims[1] + c[:, 1]) * dims[2] + c[:, 2]

    k, order = key(c).sort()
    seen, I, J, D = [], [], [], []
    for o in range(27):
        cc = c + torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=dev)
        if box:
            cc = cc % dims[0]
        kk = key(cc)
        fresh = torch.ones_like(kk, dtype=torch.bool)
        for s in seen:
            fresh &= kk != s
        if box and dims[0] < 3:
            seen.append(kk)
        lo = torch.searchsorted(k, kk)
        cnt = (torch.searchsorted(k, kk, right=True) - lo) * fresh
        i = torch.repeat_interleave(torch.arange(len(p), device=dev), cnt)
        at = torch.arange(len(i), device=dev) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
        j = order[torch.repeat_interleave(lo, cnt) + at]
        i, j = i[i < j], j[i < j]
        d = pos[j] - pos[i]
        if box:
            d = d - box * torch.round(d / box)
        d = d.norm(dim=1)
        ok = d < rc
        I.append(i[ok]), J.append(j[ok]), D.append(d[ok])
    return torch.cat(I), torch.cat(J), torch.cat(D)


def _xs(s):
    s = s ^ ((s >> 11) & ((1 << 53) - 1))
    s = s ^ (s << 31)
    return s ^ ((s >> 18) & ((1 << 46) - 1))


_MASK = (1 << 64) - 1


def _apply(m, x):
    y = 0
    for k in range(64):
        if x >> k & 1:
            y ^= m[k]
    return y


def _jumps(draws):
    """Columns of the generator's linear step to the power of each of `draws`."""
    def step(s):
        s ^= s >> 11
        s ^= (s << 31) & _MASK
        return s ^ (s >> 18)

    powers = [[step(1 << k) for k in range(64)]]
    while 1 << len(powers) <= max(draws):
        powers.append([_apply(powers[-1], x) for x in powers[-1]])
    out = []
    for d in draws:
        r = [1 << k for k in range(64)]
        for b, m in enumerate(powers):
            if d >> b & 1:
                r = [_apply(m, x) for x in r]
        out.append(r)
    return out


def _signed(x):
    return x - (1 << 64) if x >> 63 else x


# quasi-adiabatic tables in amino-acid code order (ALA ARG ASN ASP CYS GLU GLN
# GLY HIS ILE LEU LYS MET PHE PRO SER THR TRP TYR VAL): polarity (1 polar, 2
# hydrophobic), valences (back, side, side to polar, side to hydrophobic)
POLAR = [2, 1, 1, 1, 2, 1, 1, 0, 1, 2, 2, 1, 2, 2, 0, 1, 1, 2, 2, 2]
LIMITS = [(2, 4, 1, 1), (2, 4, 2, 0), (2, 3, 2, 0), (2, 2, 2, 0), (2, 5, 2, 2), (2, 2, 2, 0), (2, 3, 2, 0),
          (2, 0, 0, 0), (2, 4, 2, 0), (2, 7, 2, 4), (2, 7, 2, 4), (2, 3, 2, 0), (2, 7, 1, 1), (2, 7, 2, 4),
          (1, 0, 0, 0), (2, 2, 2, 0), (2, 3, 2, 0), (2, 8, 3, 4), (2, 7, 2, 2), (2, 6, 1, 4)]
# largest distances (A) of side-chain contacts, upper triangle in the order of SS_ORDER
SS_ORDER = ["GLY", "PRO", "GLN", "CYS", "ALA", "SER", "VAL", "THR", "ILE", "LEU", "ASN", "ASP", "LYS", "GLU", "MET",
            "HIS", "PHE", "ARG", "TYR", "TRP"]
SS_ROWS = [
    [0] * 20,
    [7.41516, 7.90612, 7.52633, 6.84509, 7.04405, 7.47655, 7.31767, 7.87539, 8.01034, 7.55152, 7.23515, 7.80572,
     7.53281, 8.28535, 7.90923, 8.35495, 8.6967, 8.60035, 8.73009],
    [8.6339, 7.72232, 7.39072, 7.63811, 7.8121, 7.76803, 8.24492, 8.43726, 8.18851, 8.15441, 8.68554, 8.40626, 8.83875,
     8.64366, 8.95351, 9.25989, 9.27035, 9.58092],
    [7.55733, 6.96894, 6.97079, 7.55818, 7.4017, 7.94719, 8.07406, 7.49217, 7.17592, 7.83117, 7.44878, 8.29132, 8.1679,
     8.49679, 8.24142, 8.25576, 8.94558],
    [6.41596, 6.52979, 7.06164, 6.94089, 7.4515, 7.64571, 7.02481, 6.73004, 7.25636, 7.03513, 7.90635, 7.49807, 8.167,
     7.99254, 8.01558, 8.6489],
    [6.64507, 7.16628, 6.96918, 7.52021, 7.68498, 7.18018, 6.99305, 7.73488, 7.40681, 7.94113, 7.87748, 8.24345,
     8.27447, 8.35846, 8.753],
    [7.64602, 7.54035, 8.06246, 8.29202, 7.53705, 7.22267, 7.68742, 7.49567, 8.48089, 7.91666, 8.68731, 8.31488,
     8.38777, 9.22171],
    [7.30031, 7.92881, 8.12374, 7.45743, 7.19339, 7.79424, 7.50872, 8.33046, 7.97856, 8.58396, 8.49644, 8.5783,
     9.13956],
    [8.5263, 8.77193, 7.95509, 7.65258, 8.15891, 7.97275, 8.9472, 8.36691, 9.11118, 8.75517, 8.77521, 9.57259],
    [8.93237, 8.13966, 7.85839, 8.39261, 8.19823, 9.14397, 8.56678, 9.33507, 8.98363, 9.01661, 9.78508],
    [7.74478, 7.49738, 8.11461, 7.99731, 8.48918, 8.36404, 8.64859, 8.87054, 8.96106, 9.10847],
    [7.3958, 8.58582, 7.81457, 8.14884, 8.49948, 8.5134, 9.12439, 9.34604, 9.10307],
    [8.93192, 8.90461, 8.79787, 8.57814, 8.79341, 9.49215, 9.03734, 9.20968],
    [8.37524, 8.61045, 8.8443, 8.74517, 9.51825, 9.47761, 9.47919],
    [9.29013, 8.9267, 9.55493, 9.27252, 9.28102, 10.0219],
    [8.82674, 8.97502, 9.2293, 9.38343, 9.65746],
    [9.73068, 9.2578, 9.56181, 10.168],
    [10.0222, 9.50922, 9.82199],
    [9.34099, 10.0829],
    [10.8456],
]
BB_R, BS_R = 5.0 * A, 6.8 * A


def _ss_table():
    t = np.zeros((20, 20))
    code = [abi.AA.index(x) for x in SS_ORDER]
    for r, row in enumerate(SS_ROWS):
        for k, x in enumerate(row[:20 - r]):
            t[code[r], code[r + k]] = t[code[r + k], code[r]] = x * A
    return t


class _Md:
    """The simulation of one context in 64-bit torch."""

    def __init__(self, case, systems):
        dev = self.dev = torch.device("cuda")
        self.case, self.box = case, case["box"] * A
        off = np.concatenate([[0], np.cumsum([s.n for s in systems])])
        ti = lambda x: torch.tensor(np.ascontiguousarray(x), device=dev).long()  # noqa: E731
        tf = lambda x: torch.tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        idx = lambda f, k: ti(np.concatenate([getattr(s, f)[k] + o for s, o in zip(systems, off)]))  # noqa: E731
        val = lambda f, k: tf(np.concatenate([getattr(s, f)[k] for s in systems]))  # noqa: E731
        self.n = int(off[-1])
        self.rep = ti(np.repeat(np.arange(len(systems)), [s.n for s in systems]))
        self.R, self.sizes = len(systems), [s.n for s in systems]
        self.chain, self.seq = ti(np.concatenate([s.chain for s in systems])), ti(np.concatenate([s.seq for s in systems]))
        at = np.concatenate([s.atype for s in systems])
        self.atype = ti(at)
        self.q = tf(np.isin(at, [1, 11]).astype(float) - np.isin(at, [3, 5]))
        self.te, self.an, self.di, self.na = ([idx(f, k) for k in range(m)] + [val(f, m)] for f, m in (
            ("tethers", 2), ("angles", 3), ("dihedrals", 4), ("natives", 2)))
        self.sd = torch.sqrt(2.0 * tf([s.temperature for s in systems])) * math.sqrt(GAMMA)
        self.mc = 4.0 if case["es"] else 18.0 * A
        self.pad = 1.0 if case["es"] else 2.0 * A
        self.nat_key = torch.unique(self.na[0] * self.n + self.na[1])
        self.seeds = [s.seed for s in systems]
        self.r0, self.v0 = tf(np.concatenate([s.r for s in systems])), tf(np.concatenate([s.v for s in systems]))
        self.orig = None
        if case["qa"]:
            ss = tf(_ss_table())
            self.ss = ss
            # by contact type: 1 backbone, 2 and 3 backbone-side, 4 + a1 + 20 a2 sides
            self.req = torch.cat([tf([0.0, BB_R, BS_R, BS_R]), ss.T.reshape(-1)])
            self.form = float(max(BS_R, ss.max()))
            self.sync = np.array(LIMITS)[at].astype(np.int64)
            self.ct = []        # (i1, i2, type, reference time)
            self.fp = None

    def lists(self, pos, flagged):
        """Lists of the flagged replicas from pos, the others kept."""
        i, j, d = _near(pos, self.rep, self.box, self.mc + self.pad)
        local = (self.chain[i] == self.chain[j]) & ((self.seq[i] - self.seq[j]).abs() < 3)
        keep = flagged[self.rep[i]] & ~local & ~torch.isin(i * self.n + j, self.nat_key)
        i, j, d = i[keep], j[keep], d[keep]
        pa, es = d < 4.0 * A + self.pad, (d < 4.0 + self.pad) & (self.q[i] * self.q[j] != 0)
        if not self.case["es"]:
            es &= False
        nd = pos[self.na[1]] - pos[self.na[0]]
        if self.box:
            nd = nd - self.box * torch.round(nd / self.box)
        on = nd.norm(dim=1) < 2.0 * self.na[2] + self.pad
        new = [torch.stack([i[pa], j[pa]]), torch.stack([i[es], j[es]])]
        if self.orig is None:
            self.orig, self.pairs, self.nat_on = pos.clone(), new, on
        else:
            self.pairs = [torch.cat([o[:, ~flagged[self.rep[o[0]]]], w], dim=1) for o, w in zip(self.pairs, new)]
            f = flagged[self.rep]
            self.orig[f] = pos[f]
            self.nat_on = torch.where(flagged[self.rep[self.na[0]]], on, self.nat_on)
        if self.case["qa"]:
            k = i * self.n + j
            near = d < self.form + self.pad
            k = k[near].sort()[0]
            if self.ct:
                held = torch.tensor([a * self.n + b for a, b, _, _ in self.ct], device=self.dev)
                k = k[~torch.isin(k, held)]
            self.fp = torch.stack([torch.div(k, self.n, rounding_mode="floor"), k % self.n])

    def ruv(self, pos, i, j):
        d = pos[j] - pos[i]
        return d - self.box * torch.round(d / self.box) if self.box else d

    def forces(self, pos, t):
        """Forces and the energies of tethers, angles, dihedrals, Go, Pauli and ES."""
        F = torch.zeros_like(pos)
        V = []

        def pair(i, j, dV, u):
            F.index_add_(0, i, dV[:, None] * u)
            F.index_add_(0, j, -dV[:, None] * u)

        i, j, d0 = self.te
        d = pos[j] - pos[i]
        r = d.norm(dim=1)
        x = r - d0
        H = 100.0 / (A * A)
        V.append((0.5 * H * x * x).clamp(-1e3, 1e3).sum())
        pair(i, j, (H * x).clamp(-1e3, 1e3), d / r[:, None])

        p = pos.detach().requires_grad_(True)
        i, j, k, th0 = self.an
        a, b = p[j] - p[i], p[k] - p[j]
        th = torch.atan2(torch.linalg.cross(a, b, dim=1).norm(dim=1), -(a * b).sum(1))
        va = (15.0 * (th - th0) ** 2).sum()
        i, j, k, l, ph0 = self.di
        a, b, c = p[j] - p[i], p[k] - p[j], p[l] - p[k]
        x1, x2 = torch.linalg.cross(a, b, dim=1), torch.linalg.cross(b, c, dim=1)
        f = torch.atan2(b.norm(dim=1) * (x1 * c).sum(1), (x1 * x2).sum(1)) - ph0
        vd = 0.66 * ((1 - torch.cos(f)) + (1 - torch.cos(3 * f))).sum()
        F -= torch.autograd.grad(va + vd, p)[0]
        V += [va.detach(), vd.detach()]

        i, j, d0 = (x[self.nat_on] for x in self.na)
        d = self.ruv(pos, i, j)
        r = d.norm(dim=1)
        s6 = (d0 / r) ** 6
        V.append((s6 * s6 - 2 * s6).clamp(-1e3, 1e3).sum())
        pair(i, j, (12.0 / r * (s6 - s6 * s6)).clamp(-1e3, 1e3), d / r[:, None])

        i, j = self.pairs[0]
        d = self.ruv(pos, i, j)
        r = d.norm(dim=1)
        in_ = r < 4.0 * A
        s6 = (4.0 * A / r) ** 6
        V.append(((s6 * s6 - 2 * s6 + 1).clamp(-1e3, 1e3) * in_).sum())
        pair(i, j, (12.0 / r * (s6 - s6 * s6)).clamp(-1e3, 1e3) * in_, d / r[:, None])

        i, j = self.pairs[1]
        d = self.ruv(pos, i, j)
        r = d.norm(dim=1)
        v = ES_VF * self.q[i] * self.q[j] * torch.exp(-r / 2.0) / (r * r)
        V.append(v.sum())
        pair(i, j, -v * (0.5 + 1.0 / r), d / r[:, None])

        if self.case["qa"] and self.ct:
            c = torch.tensor([x[:3] for x in self.ct], device=self.dev)
            i, j, ty = c[:, 0], c[:, 1], c[:, 2]
            sat = (t - torch.tensor([x[3] for x in self.ct], dtype=torch.float64, device=self.dev)).clamp(max=10.0) * 0.1
            # the potential of a side-side contact sits at [type - 4] of the
            # table; backbone ones have one radius
            k = (ty - 4).clamp(min=0)
            rmax = torch.where(ty == 1, BB_R, torch.where(ty <= 3, BS_R, self.ss.reshape(-1)[k]))
            rmin = torch.where(ty <= 3, rmax, torch.full_like(rmax, BB_R))
            d = self.ruv(pos, i, j)
            r = d.norm(dim=1)
            re = torch.where(r < rmin, rmin, torch.where(r < rmax, r, rmax))
            s6 = (re / r) ** 6
            dv = torch.where((rmin < r) & (r < rmax), torch.zeros_like(r), 12.0 / r * (s6 - s6 * s6))
            pair(i, j, sat * dv.clamp(-1e3, 1e3), d / r[:, None])
        return F, V

    def contacts(self, pos, t):
        """New quasi-adiabatic contacts at these positions (no contact is old
        enough to break: runs are shorter than the 10 tau phase)."""
        has = torch.zeros(self.n, dtype=torch.bool, device=self.dev)
        has[1:-1] = (self.chain[1:-1] == self.chain[:-2]) & (self.chain[1:-1] == self.chain[2:])
        n, h = torch.zeros_like(pos), torch.zeros_like(pos)
        c = has.nonzero()[:, 0]
        v1, v2 = pos[c] - pos[c - 1], pos[c + 1] - pos[c]
        n[c], h[c] = _unit(v2 - v1), _unit(torch.linalg.cross(v2, v1, dim=1))
        i, j = self.fp
        d = self.ruv(pos, i, j)
        r = d.norm(dim=1)
        near = (r < self.form * (1 + 1e-9)).nonzero()[:, 0]
        i, j, r, u = i[near], j[near], r[near], d[near] / r[near, None]
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        b1, b2 = dot(h[i], u).abs() > 0.92, dot(h[j], u).abs() > 0.92
        bb = dot(h[i], h[j]).abs() > 0.75
        s1, s2 = dot(n[i], u) < 0.5, -dot(n[j], u) < 0.5
        a1, a2 = self.atype[i], self.atype[j]
        ty = torch.where(b1 & b2 & bb, 1, torch.where(b1 & s2, 2, torch.where(
            s1 & b2, 3, torch.where(s1 & s2, 4 + a1 + 20 * a2, 0))))
        ok = (ty > 0) & ~(1.0 > self.req[ty] / r)
        sel = ok.nonzero()[:, 0]
        cols = [x[sel].cpu().numpy() for x in (i, j, ty, b1, b2, s1, s2, a1, a2)]
        gone = []
        for k, (x, y, tt, p1, p2, q1, q2, m1, m2) in enumerate(zip(*cols)):
            w1 = np.array([p1, q1, q1 and POLAR[m2] == 1, q1 and POLAR[m2] == 2], dtype=np.int64)
            w2 = np.array([p2, q2, q2 and POLAR[m1] == 1, q2 and POLAR[m1] == 2], dtype=np.int64)
            if (self.sync[x] >= w1).all() and (self.sync[y] >= w2).all():
                self.sync[x] -= w1
                self.sync[y] -= w2
                self.ct.append((int(x), int(y), int(tt), t))
                gone.append(k)
        if gone:
            live = torch.ones(self.fp.shape[1], dtype=torch.bool, device=self.dev)
            live[near[sel[torch.tensor(gone, device=self.dev)]]] = False
            self.fp = self.fp[:, live]

    def noise(self, st):
        u = []
        for _ in range(4):
            v = st * (0xd989bcacc137dcd5 - (1 << 64))
            st = _xs(st)
            if self.case["precision"] == "fp64":
                u.append(((v >> 32) & 0xffffffff).double() / 4294967296.0)
            else:   # 23 bits, centred
                u.append(((v >> 41) & 0x7fffff).double() / 8388608.0 + 2.0 ** -24)
        turn = 0.0 if self.case["precision"] == "fp64" else math.pi
        r1, r2 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
        a1, a2 = 2 * math.pi * u[1] - turn, 2 * math.pi * u[3] - turn
        return torch.stack([r1 * torch.cos(a1), r1 * torch.sin(a1), r2 * torch.cos(a2)], dim=1)

    def simulate(self, steps):
        z = torch.zeros_like(self.r0)
        y = [self.r0.clone(), self.v0 * DT, z.clone(), z.clone(), z.clone(), z.clone()]
        # bead i of a replica of n starts 4 i draws into the replica's stream
        # and moves on by 4 n draws a step
        st = []
        for n, seed in zip(self.sizes, self.seeds):
            s = seed & _MASK
            for _ in range(n):
                st.append(_signed(s))
                for _ in range(4):
                    s ^= s >> 11
                    s ^= (s << 31) & _MASK
                    s ^= s >> 18
        cols = [[_signed(x) for x in m] for m in _jumps([4 * n for n in self.sizes])]
        st, cols = torch.tensor(st, device=self.dev), torch.tensor(cols, device=self.dev)[self.rep]
        every = torch.ones(self.R, dtype=torch.bool, device=self.dev)
        self.lists(y[0], every)
        t, hh = 0.0, DT * DT / 2.0
        for _ in range(steps):
            F, _ = self.forces(y[0], t)
            if self.case["qa"]:
                self.contacts(y[0], t)
            a = F - GAMMA * (y[1] / DT) + self.sd[self.rep][:, None] * self.noise(st)
            e = y[2] - a * hh
            nxt = torch.zeros_like(st)
            for k in range(64):
                nxt ^= cols[:, k] * ((st >> k) & 1)
            st = nxt
            y = [x - c * e for x, c in zip(y, (3 / 16, 251 / 360, 1.0, 11 / 18, 1 / 6, 1 / 60))]
            y = [sum(math.comb(m, k) * y[m] for m in range(k, 6)) for k in range(6)]
            t += DT
            d = self.orig - y[0]
            if self.box:
                d = d - self.box * torch.round(d / self.box)
            far = torch.zeros(self.R, dtype=torch.float64, device=self.dev)
            far.scatter_reduce_(0, self.rep, d.norm(dim=1), "amax")
            flagged = 2.0 * far > self.pad
            if bool(flagged.any()):
                self.lists(y[0], flagged)
        return y[0], y[1] / DT


def exact(case, seed):
    systems = _systems(case, seed)
    if case["kind"] == "pairs":
        s = systems[0]
        pos = torch.tensor(s.r, device="cuda")
        i, j, _ = _near(pos, torch.zeros(s.n, dtype=torch.long, device="cuda"), case["box"] * A, PAIR_CUTOFF)
        ch, sq = torch.tensor(s.chain, device="cuda"), torch.tensor(s.seq, device="cuda")
        ok = ~((ch[i] == ch[j]) & ((sq[i] - sq[j]).abs() < 3))
        k = (i[ok] * s.n + j[ok]).sort()[0]
        out = torch.zeros(128 * s.n, 2, dtype=torch.int32, device="cuda")
        out[:len(k), 0], out[:len(k), 1] = (k // s.n).int(), (k % s.n).int()
        return {"pairs": out, "count": torch.tensor([len(k)], dtype=torch.int32, device="cuda")}
    if case["kind"] == "serve":
        got = []
        for s in systems:
            s.v = np.zeros_like(s.r)     # requests start at rest
        md = _Md(case, systems)
        r, v = md.simulate(case["steps"])
        at = 0
        for s in systems:
            got.append({"r": r[at:at + s.n], "v": v[at:at + s.n]})
            at += s.n
        return got
    md = _Md(case, systems)
    if case["kind"] == "score":
        md.lists(md.r0, torch.ones(1, dtype=torch.bool, device="cuda"))
        F, V = md.forces(md.r0, 0.0)
        e = torch.zeros(abi.NUM_TERMS, dtype=torch.float64)
        for k, x in zip((abi.TERM_TETHER, abi.TERM_NAT_ANG, abi.TERM_CND, abi.TERM_GO, abi.TERM_PAULI,
                         abi.TERM_CONST_ES), V):
            e[k] = float(x)
        return {"F": F, "V": e}
    r, v = md.simulate(case["steps"])
    if _packed(case):
        v = v * DT      # the history holds y1 = v dt
    out = {"r": r, "v": v}
    if case["qa"] and case["precision"] == "fp64":
        out["valences"] = md.sync.astype(np.int8)
    return out
