"""What the framework is timed on: closed-shell NDDO calculations as its users run them.

Every case goes through the public entry points (`ElectronicStructure`, `batch_scf`,
`ResidentBatch`, `Server`, `nddo_pair_integrals_noalloc`) on seeded geometries of the
kinds the package's workloads generate: jittered water clusters and saturated alkanes.
Sizes run from a water dimer (12 basis functions) to 180 waters (1080).

`exact` is an independent 64-bit restatement in numpy: point-charge multipoles, Slater
overlaps by quadrature, a commutator-DIIS SCF to full convergence, and forces by
complex-step differentiation of the pair energies at the converged density.
"""
import ctypes
import math

import numpy as np
import torch

import molds_gb300 as M
from molds_gb300 import workloads as W

# DIIS alone, as the batched water benchmark runs it (those clusters converge so) ...
DIIS = dict(max_iter=500, rms_density=1e-8, damping_thresh=1.0, damping_weight=0.0, diis_start_error=0.1,
            diis_end_error=0.0)
# ... and with the densities mixed first (default weight and DIIS start): what a user sets for
# larger clusters and branched alkanes, where DIIS alone can cycle; tight enough that the
# forces do not carry what is left of the convergence
DAMPED = dict(DIIS, damping_thresh=3e-3, damping_weight=0.8, diis_start_error=1e-2, rms_density=1e-10)
# the mixed path to a tighter threshold, so that its result does not carry FP32 noise
MIXED = dict(DAMPED, precision="mixed", rms_density=1e-11)
SCF = {"diis": DIIS, "damped": DAMPED, "mixed": MIXED}


def listed():
    return [
        # the smallest call: launches and host latency only
        {"name": "single_water2", "kind": "single", "system": "water", "size": 2, "theory": "am1", "scf": "diis",
         "epc": 0, "forces": False},
        # the plain benchmark molecule (thermally displaced), energy and forces: one step of an optimiser
        {"name": "single_octane_force", "kind": "single", "system": "octane", "size": 8, "theory": "pm3",
         "scf": "diis", "epc": 0, "forces": True},
        # QM/MM: a branched alkane in the field of solvent point charges, with forces
        {"name": "single_alkane_epc", "kind": "single", "system": "alkane", "size": 14, "theory": "pm3",
         "scf": "damped", "epc": 900, "forces": True},
        # an ordinary single point, odd basis size
        {"name": "single_water33", "kind": "single", "system": "water", "size": 33, "theory": "am1", "scf": "damped",
         "epc": 0, "forces": False},
        # a large single point
        {"name": "single_water101", "kind": "single", "system": "water", "size": 101, "theory": "pm3",
         "scf": "damped", "epc": 0, "forces": False},
        # the largest single point
        {"name": "single_water180", "kind": "single", "system": "water", "size": 180, "theory": "mndo",
         "scf": "damped", "epc": 0, "forces": False},
        # the headline batch: 256 replicas of (H2O)32
        {"name": "batch_water32", "kind": "batch", "size": 32, "count": 256, "theory": "am1", "scf": "diis"},
        # the same kind of batch on the mixed-precision path
        {"name": "batch_mixed", "kind": "batch", "size": 27, "count": 64, "theory": "am1", "scf": "mixed"},
        # molecules of all sizes in one call: alkanes and water clusters
        {"name": "batch_uneven", "kind": "uneven", "count": 97, "smallest": 5, "largest": 180, "theory": "pm3",
         "scf": "damped"},
        # RPMD beads: a resident batch moved a few steps, warm starts, forces of every bead
        {"name": "md_beads", "kind": "md", "size": 12, "count": 32, "steps": 3, "theory": "am1", "scf": "damped"},
        # serving: a burst of single-point requests, submitted and drained
        {"name": "server_burst", "kind": "server", "count": 60, "smallest": 5, "largest": 180, "theory": "pm3",
         "scf": "damped"},
        # integrals alone, into the caller's own device buffers
        {"name": "integrals_water150", "kind": "integrals", "size": 150, "theory": "am1"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "batch", "uneven", "md", "server", "integrals"])
    theory = rng.choice(["mndo", "am1", "pm3"])
    if kind == "single":
        if rng.random() < 0.4:
            return {"kind": kind, "system": "alkane", "size": rng.randint(3, 16), "theory": "pm3", "scf": "damped",
                    "epc": rng.choice([0, 0, 3 * _log_int(rng, 4, 700)]), "forces": rng.random() < 0.6}
        k = _log_int(rng, 2, 120)
        return {"kind": kind, "system": "water", "size": k, "theory": theory,
                "scf": "diis" if k <= 6 else "damped", "epc": 0, "forces": k < 100 and rng.random() < 0.4}
    if kind == "batch":
        k = _log_int(rng, 2, 32)
        scf = rng.choice(["damped", "damped", "mixed"])
        return {"kind": kind, "size": k, "count": max(2, min(256, _log_int(rng, 8, 256) * 24 // (k + 8))),
                "theory": theory, "scf": scf}
    if kind in ("uneven", "server"):
        return {"kind": kind, "count": _log_int(rng, 8, 97 if kind == "uneven" else 60), "smallest": rng.randint(5, 12),
                "largest": _log_int(rng, 30, 180), "theory": "pm3", "scf": "damped"}
    if kind == "md":
        return {"kind": kind, "size": _log_int(rng, 2, 20), "count": _log_int(rng, 4, 32), "steps": rng.randint(2, 3),
                "theory": theory, "scf": "damped"}
    return {"kind": kind, "size": _log_int(rng, 4, 170), "theory": theory}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _single(case, seed):
    if case["system"] == "octane":
        mol = W.water_replicas(W.octane(), 1, sigma=0.03, seed0=seed)[0]
    elif case["system"] == "alkane":
        mol = W.random_alkane(seed, n=case["size"])
    else:
        mol = W.water_cluster_k(case["size"], seed)
    if case["epc"]:
        # solvent around the molecule: three-site waters as point charges (-0.834, 0.417, 0.417 e)
        rng = np.random.default_rng(seed + 1)
        n = case["epc"] // 3
        c = mol.xyz.mean(axis=0)
        inner = np.linalg.norm(mol.xyz - c, axis=1).max() + 6.0
        d, h1, h2 = (v / np.linalg.norm(v, axis=1)[:, None] for v in rng.normal(size=(3, n, 3)))
        r = (inner ** 3 + rng.uniform(0.0, 1.0, n) * ((inner + 15.0) ** 3 - inner ** 3)) ** (1.0 / 3.0)
        o = c + d * r[:, None]
        pos = np.concatenate([o, o + 0.96 * M.ANG2AU * h1, o + 0.96 * M.ANG2AU * h2])
        mol = M.Molecule(mol.Z, mol.xyz, np.column_stack([pos, np.repeat([-0.834, 0.417, 0.417], n)]))
    return mol


def _uneven(case, seed):
    """Sizes log-spaced over the range (the same for every seed), every other molecule an
    alkane as long as its trees are small enough to converge."""
    out = []
    for i, a in enumerate(np.exp(np.linspace(math.log(case["smallest"]), math.log(case["largest"]), case["count"]))):
        n = max(3, int(round((a - 2) / 3)))
        if i % 2 == 0 and n <= 16:
            out.append(W.random_alkane(seed * 1009 + i, n=n))
        else:
            out.append(W.water_cluster_k(max(2, int(round(a / 3))), seed * 1009 + i))
    order = np.random.default_rng(seed).permutation(len(out))   # sizes arrive in no order
    return [out[i] for i in order]


def _batch(case, seed):
    base = W.water_cluster(seed=2) if case["size"] == 32 else W.water_cluster_k(case["size"], 2)
    return W.water_replicas(base, case["count"], sigma=0.05, seed0=1000 * seed)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind == "integrals":
        s.lib = M.load_library()
        mol = W.water_cluster_k(case["size"], seed)
        s.Z = np.ascontiguousarray(mol.Z, dtype=np.int32)
        s.xyz = np.ascontiguousarray(mol.xyz, dtype=np.float64)
        nao = 6 * case["size"]
        k = case["size"]
        heavy, light = k * (k - 1) // 2, k * 2 * k
        s.count = 100 * heavy + 10 * light + k * (2 * k - 1)
        s.blocks = torch.zeros(s.count, dtype=torch.float64, device="cuda")
        s.H = torch.zeros((nao, nao), dtype=torch.float64, device="cuda")
        s.err = ctypes.create_string_buffer(256)
        s.stream = torch.cuda.current_stream().cuda_stream
        torch.cuda.synchronize()
        return s
    s.params = M.SCFParams(**SCF[case["scf"]])
    s.ctx = M.Context(0)
    if kind == "single":
        s.mol = _single(case, seed)
        s.es = M.ElectronicStructure(case["theory"], s.params, context=s.ctx)
    elif kind == "batch":
        s.mols = _batch(case, seed)
    elif kind == "uneven":
        s.mols = _uneven(case, seed)
    elif kind == "md":
        mols = _batch(case, seed)
        rng = np.random.default_rng(seed + 17)
        v = [rng.normal(0.0, 0.01, size=m.xyz.shape) * M.ANG2AU for m in mols]
        s.path = [np.concatenate([m.xyz + t * u for m, u in zip(mols, v)]) for t in range(case["steps"])]
        s.batch = M.ResidentBatch(case["theory"], mols, s.params.diis_num_error_vect, context=s.ctx)
    else:
        s.mols = _uneven(case, seed)
        s.server = M.Server(s.params, hbm_budget_bytes=6 << 30, max_basis=400, context=s.ctx)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _table(res, charges):
    return {"energy": np.array([r["energy"] for r in res]),
            "core_repulsion": np.array([r["core_repulsion"] for r in res]),
            "charges": np.concatenate(charges), "status": np.array([r["status"] for r in res]),
            "dipole": np.array([r["dipole"] for r in res])}


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "single":
        es = s.es
        es.SetMolecule(s.mol)
        es.DoSCF(True)
        out = {"energy": es.GetElectronicEnergy(0), "core_repulsion": es.GetCoreRepulsionEnergy(),
               "eps": es.GetEnergiesMO(), "charges": es.GetMullikenCharges(),
               "density": es.GetOrbitalElectronPopulation(), "dipole": es.GetDipoleMoments()}
        if case["forces"]:
            out["forces"] = es.GetForce()
        return out
    if kind in ("batch", "uneven"):
        return _table(*M.batch_scf(case["theory"], s.mols, s.params, context=s.ctx))
    if kind == "md":
        out = []
        for t, x in enumerate(s.path):
            s.batch.set_coordinates(x)
            s.batch.run(s.params, requires_guess=t == 0)
            step = _table(*s.batch.results())
            step["forces"] = np.concatenate([s.batch.forces(m) for m in range(case["count"])])
            out.append(step)
        return out
    if kind == "server":
        place = {s.server.submit(case["theory"], m): i for i, m in enumerate(s.mols)}
        res = sorted(s.server.drain(), key=lambda r: place[r["ticket"]])
        return {"energy": np.array([r["energy"] for r in res]),
                "core_repulsion": np.array([r["core_repulsion"] for r in res]),
                "charges": np.concatenate([r["charges"] for r in res]),
                "status": np.array([r["status"] for r in res])}
    ecore = ctypes.c_double()
    rc = s.lib.nddo_pair_integrals_noalloc(
        0, M.THEORIES[case["theory"]], s.Z.size, s.Z.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
        s.xyz.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.c_void_p(s.blocks.data_ptr()), s.count,
        ctypes.c_void_p(s.H.data_ptr()), ctypes.byref(ecore), ctypes.c_void_p(s.stream), s.err, 256)
    if rc:
        raise RuntimeError(s.err.value.decode())
    return {"blocks": s.blocks, "core_hamiltonian": s.H, "core_repulsion": ecore.value}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _one_work(heavy, light, iterations):
    """One SCF: the pair integrals read once per Fock build, and per iteration a
    tridiagonalisation (4/3 N^3), the smaller set's vectors (2 N^2 k) and P = 2 X^T X (N^2 k)."""
    n = 4 * heavy + light
    nocc = (n if light != 2 * heavy else 8 * heavy) // 2
    k = min(nocc, n - nocc)
    blk = 100 * heavy * (heavy - 1) / 2 + 10 * heavy * light + light * (light - 1) / 2
    return iterations * (8 * blk + 16 * n * n) + 32 * (heavy + light), iterations * (4 / 3 * n ** 3 + 3 * n * n * k)


def work(case):
    kind = case["kind"]
    if kind == "integrals":
        k = case["size"]
        blk = 100 * k * (k - 1) / 2 + 10 * k * 2 * k + k * (2 * k - 1)
        return {"bytes": 8 * blk + 8 * (6 * k) ** 2 + 24 * 3 * k, "flops": 3000 * k * (k - 1) / 2}
    its = {"diis": 14, "damped": 38, "mixed": 40}[case["scf"]]
    if kind in ("uneven", "server"):
        sizes = []
        for i, a in enumerate(np.exp(np.linspace(math.log(case["smallest"]), math.log(case["largest"]),
                                                 case["count"]))):
            n = max(3, int(round((a - 2) / 3)))
            sizes.append((n, 2 * n + 2) if i % 2 == 0 and n <= 16 else (max(2, round(a / 3)), 2 * max(2, round(a / 3))))
        w = [_one_work(h, l, its) for h, l in sizes]
    elif kind == "single" and case["system"] != "water":
        w = [_one_work(case["size"], 2 * case["size"] + 2, its)]
    else:
        solves = {"single": 1}.get(kind, case.get("count", 1))
        if kind == "md":
            its += 20 * (case["steps"] - 1)
        w = [_one_work(case["size"], 2 * case["size"], its)] * solves
    return {"bytes": float(sum(x[0] for x in w)) + 32.0 * case.get("epc", 0), "flops": float(sum(x[1] for x in w))}


# ---------------------------------------------------------------------------
# the same results in plain numpy, 64 bits
# ---------------------------------------------------------------------------
_ANG = 1.0 / 0.5291772
# element parameters in atomic units: core charge; U s, p; zeta s, p; beta s, p; alpha;
# gss, gsp, gpp, gp2, hsp; charge separations D1, D2; additive terms rho 0, 1, 2;
# Gaussians (K, L, M)
_PARAMETERS = {
    ("mndo", 1): (1, (-0.43754409391228005, 0), (1.331967, 0), (-0.25684132260792003, 0), 1.3462977065448,
                  (0.47215153744000005, 0, 0, 0, 0), (0, 0), (1.0589820436746924, 0, 0), ()),
    ("mndo", 8): (6, (-3.6617869037027004, -2.85898163245216), (2.699905, 2.699905),
                  (-1.20125530606046, -1.20125530606046), 1.6725195750288,
                  (0.5666700426, 0.5321259544, 0.5335959156, 0.47700240940000005, 0.1447911782),
                  (0.5346023927, 0.4536251725), (0.8823476845641884, 0.5212512325547042, 0.52655074561716), ()),
    ("am1", 1): (1, (-0.41880763771581, 0), (1.188078, 0), (-0.22688068367661002, 0), 1.5252601438128,
                 (0.47215153744000005, 0, 0, 0, 0), (0, 0), (1.0589820436746924, 0, 0),
                 ((0.004512633887880001, 1.4001425449992, 2.267671396273309),
                  (0.0001870525627, 1.4001425449992, 3.4015070944099635),
                  (-0.0006738302140800001, 0.56005701799968, 3.968424943478291))),
    ("am1", 8): (6, (-3.5951576049000002, -2.8760665504914), (3.108032, 2.524039),
                 (-1.0757460131601901, -1.0757460131601901), 2.3576807507412,
                 (0.5666700426, 0.5321259544, 0.5335959156, 0.47700240940000005, 0.1447911782),
                 (0.4988896404, 0.4852321503), (0.8823476845641884, 0.5019676546265106, 0.5515685864602415),
                 ((0.01032508096686, 1.4001425449992, 1.6023328291543928),
                  (0.0029924735129, 1.96019956299888, 2.7307884769033888))),
    ("pm3", 1): (1, (-0.48043186562863005, 0), (0.967807, 0), (-0.20676885828336, 0), 1.7761229455992,
                 (0.5436727936182401, 0, 0, 0, 0), (0, 0), (0.9196708128232518, 0, 0),
                 ((0.0414804676125, 1.4271042499027227, 2.9053878360594525),
                  (-0.038966062230870006, 1.6812318019911314, 2.9672272350358257))),
    ("pm3", 6): (4, (-1.7371384077896, -1.33277405758954), (1.565085, 1.842345),
                 (-0.43768149853545, -0.36024173757765), 1.4329097264003998,
                 (0.41161515431324003, 0.37722978517381, 0.39675325859676, 0.33230552921098006, 0.0841912927494),
                 (0.8332396384, 0.6647749859), (1.2147268990868638, 0.8495156807972571, 0.6538072626190363),
                 ((0.00184138364621, 1.6810573442300245, 3.103334761966313),
                  (0.00186438853899, 1.6810052589273505, 1.6865579242643105))),
    ("pm3", 8): (6, (-3.1969084402880603, -2.6415048418074), (3.796544, 2.389402),
                 (-1.6611535776785302, -0.90963091631045), 1.7024170284744,
                 (0.5790088969128, 0.3903173274748, 0.50177184360448, 0.4559117735927001, 0.021824624183490002),
                 (0.4086173087, 0.5125738036), (0.8635445891712342, 0.9434821416790706, 0.611285580675715),
                 ((-0.04156785680584, 1.6808646846158326, 3.03737764967954),
                  (0.04181639049573, 1.666313003145656, 3.0205288512052295))),
}
_AXIS = (None, 1, 2, 0)   # orbitals s, py, pz, px -> Cartesian axis


def _charges(i, j, D):
    """The point charges (q, position, multipole order) of the distribution i j."""
    def at(*pairs):
        r = [0.0, 0.0, 0.0]
        for ax, v in pairs:
            r[ax] += v
        return r
    a, b = _AXIS[i], _AXIS[j]
    if a is None and b is None:
        return [(1.0, at(), 0)]
    if a is None or b is None:
        ax = b if a is None else a
        return [(0.5 * sg, at((ax, sg * D[0])), 1) for sg in (1, -1)]
    if a == b:
        return [(1.0, at(), 0), (-0.5, at(), 2)] + [(0.25, at((a, sg * 2 * D[1])), 2) for sg in (1, -1)]
    return [(0.25 * s1 * s2, at((a, s1 * D[1]), (b, s2 * D[1])), 2) for s1 in (1, -1) for s2 in (1, -1)]


def _norm(d):
    return np.sqrt((d * d).sum(axis=1))


def _local_eri(pa, pb, na, nb, R, zero_rho=False):
    L = np.zeros((R.size, na, na, nb, nb), dtype=R.dtype)
    for i in range(na):
        for j in range(i, na):
            for k in range(nb):
                for l in range(k, nb):
                    if {i, j} == {1, 3} and {k, l} == {1, 3}:
                        continue
                    v = 0.0
                    for qa, ra, la in _charges(i, j, pa[6]):
                        for qb, rb, lb in _charges(k, l, pb[6]):
                            rho = 0.0 if zero_rho else pa[7][la] + pb[7][lb]
                            x, y, z = rb[0] - ra[0], rb[1] - ra[1], R + (rb[2] - ra[2])
                            v = v + qa * qb / np.sqrt(x * x + y * y + z * z + rho * rho)
                    for m, n in ((i, j), (j, i)):
                        L[:, m, n, k, l] = v
                        L[:, m, n, l, k] = v
    if na == 4 and nb == 4:
        v = 0.5 * (L[:, 3, 3, 3, 3] - L[:, 3, 3, 1, 1])
        for m, n in ((1, 3), (3, 1)):
            for k, l in ((1, 3), (3, 1)):
                L[:, m, n, k, l] = v
    return L


def _frame(d, R):
    T = np.zeros((R.size, 4, 4), dtype=d.dtype)
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    rxy = np.sqrt(x * x + y * y)
    ca, sa, cb, sb = x / rxy, y / rxy, z / R, rxy / R
    T[:, 0, 0] = 1.0
    T[:, 1, 1], T[:, 1, 2], T[:, 1, 3] = ca, sa * sb, sa * cb
    T[:, 2, 2], T[:, 2, 3] = cb, -sb
    T[:, 3, 1], T[:, 3, 2], T[:, 3, 3] = -sa, ca * sb, ca * cb
    return T


_LAG = np.polynomial.laguerre.laggauss(10)
_LEG = np.polynomial.legendre.leggauss(64)


def _local_overlap(na, ka, za, nb, kb, zb, R):
    """Slater overlap in prolate spheroidal coordinates by Gauss quadrature (exact in xi);
    kinds 0 s, 1 p sigma, 2 p pi; A at the origin, B at +R on the z axis."""
    p, q = 0.5 * R * (za + zb), 0.5 * R * (za - zb)
    xi = 1.0 + _LAG[0][None, :, None] / p[:, None, None]
    wx = _LAG[1][None, :, None] / p[:, None, None]
    eta = _LEG[0][None, None, :]
    f = (xi + eta) ** (na - 1 - (ka > 0)) * (xi - eta) ** (nb - 1 - (kb > 0)) * (xi * xi - eta * eta)
    if ka == 2:
        f = f * (xi * xi - 1.0) * (1.0 - eta * eta) * 0.75
    else:
        f = f * 0.5 * (math.sqrt(3.0) * (1.0 + xi * eta) if ka else 1.0)
        f = f * (math.sqrt(3.0) * (xi * eta - 1.0) if kb else 1.0)
    s = (f * wx * _LEG[1][None, None, :] * np.exp(-p[:, None, None] - q[:, None, None] * eta)).sum(axis=(1, 2))
    norm = math.sqrt((2 * za) ** (2 * na + 1) * (2 * zb) ** (2 * nb + 1) /
                     (math.factorial(2 * na) * math.factorial(2 * nb)))
    return norm * (0.5 * R) ** (na + nb + 1) * s


class _Nddo:
    """A molecule in plain numpy; every atom has four orbital slots (a hydrogen fills the first)."""

    def __init__(self, theory, mol):
        self.theory, self.Z, self.xyz = theory, np.asarray(mol.Z), np.asarray(mol.xyz, dtype=float)
        self.A = A = self.Z.size
        self.par = {z: _PARAMETERS[theory, int(z)] for z in set(self.Z.tolist())}
        self.nao = np.where(self.Z == 1, 1, 4)
        self.slots = np.concatenate([4 * a + np.arange(self.nao[a]) for a in range(A)])
        self.core = np.array([self.par[z][0] for z in self.Z], dtype=float)
        self.nocc = int(self.core.sum()) // 2
        self.ia, self.ib = np.triu_indices(A, 1)
        d = self.xyz[self.ib] - self.xyz[self.ia]
        self.Wp, self.S, ec = self.pairs(d)
        self.ecore = float(ec.sum())
        # core Hamiltonian blocks and the guess Fock matrix
        H = np.zeros((A, A, 4, 4))
        U = np.zeros((A, 4))
        self.G, self.X = np.zeros((A, 4, 4)), np.zeros((A, 4, 4))
        beta = np.zeros((A, 4))
        for a in range(A):
            p, n = self.par[self.Z[a]], self.nao[a]
            U[a, :n] = [p[1][0]] + [p[1][1]] * (n - 1)
            beta[a, :n] = [p[3][0]] + [p[3][1]] * (n - 1)
            gss, gsp, gpp, gp2, hsp = p[5]
            for m in range(n):
                for k in range(n):
                    sp = (m == 0) + (k == 0)
                    g = gss if sp == 2 else gsp if sp else gpp if m == k else gp2
                    self.G[a, m, k] = g
                    self.X[a, m, k] = g if m == k else hsp if sp else 0.5 * (gpp - gp2)
        self.beta = beta
        ar = np.arange(A)
        for m in range(4):
            H[ar, ar, m, m] = U[:, m]
        res = 0.5 * (beta[self.ia][:, :, None] + beta[self.ib][:, None, :]) * self.S
        H[self.ia, self.ib] = res
        H[self.ib, self.ia] = res.transpose(0, 2, 1)
        self.guess = self.full(H)
        one = np.zeros((A, 4, 4))
        np.add.at(one, self.ia, -self.core[self.ib][:, None, None] * self.Wp[:, :, :, 0, 0])
        np.add.at(one, self.ib, -self.core[self.ia][:, None, None] * self.Wp[:, 0, 0])
        self.e_epc = 0.0
        epc = getattr(mol, "epc", None)
        if epc is not None:
            unit = (1, (0, 0), (0, 0), (0, 0), 0, (0,) * 5, (0, 0), (0, 0, 0), ())
            for a in range(A):
                n = self.nao[a]
                d = epc[:, :3] - self.xyz[a]
                R = _norm(d)
                T = _frame(d, R)[:, :n, :n]
                L = _local_eri(self.par[self.Z[a]], unit, n, 1, R, zero_rho=True)[:, :, :, 0, 0]
                one[a, :n, :n] -= np.einsum("p,pmi,pij,pnj->mn", epc[:, 3], T, L, T)
                self.e_epc += float((self.core[a] * epc[:, 3] / R).sum())
        H[ar, ar] += one
        self.H = H

    def pairs(self, d):
        """Rotated two-centre integrals, overlaps and core-core energies of all pairs at
        relative positions d (complex d: for derivatives)."""
        n = self.ia.size
        Wp = np.zeros((n, 4, 4, 4, 4), dtype=d.dtype)
        S = np.zeros((n, 4, 4), dtype=d.dtype)
        ec = np.zeros(n, dtype=d.dtype)
        za, zb = self.Z[self.ia], self.Z[self.ib]
        for A in self.par:
            for B in self.par:
                sel = np.nonzero((za == A) & (zb == B))[0]
                for at in range(0, sel.size, 8192):
                    p = sel[at:at + 8192]
                    Wp[p], S[p], ec[p] = self._pair_type(A, B, d[p])
        return Wp, S, ec

    def _pair_type(self, A, B, d):
        pa, pb = self.par[A], self.par[B]
        na, nb = (1 if A == 1 else 4), (1 if B == 1 else 4)
        R = _norm(d)
        T = _frame(d, R)
        Ta, Tb = T[:, :na, :na], T[:, :nb, :nb]
        L = _local_eri(pa, pb, na, nb, R)
        x = np.matmul(Ta, L.reshape(-1, na, na * nb * nb)).reshape(L.shape)
        x = np.matmul(Ta[:, None], x.reshape(-1, na, na, nb * nb)).reshape(L.shape)
        x = np.matmul(np.matmul(Tb[:, None, None], x), Tb.transpose(0, 2, 1)[:, None, None])
        Wp = np.zeros((R.size, 4, 4, 4, 4), dtype=d.dtype)
        Wp[:, :na, :na, :nb, :nb] = x
        sl = np.zeros((R.size, 4, 4), dtype=d.dtype)
        kind = (0, 2, 1, 2)
        qa, qb = (1 if A == 1 else 2), (1 if B == 1 else 2)
        for i in range(na):
            for j in range(nb):
                if (kind[i] == 2 or kind[j] == 2) and i != j:
                    continue
                if i == 3:
                    sl[:, 3, 3] = sl[:, 1, 1]
                    continue
                sl[:, i, j] = _local_overlap(qa, kind[i], pa[2][i > 0], qb, kind[j], pb[2][j > 0], R)
        S = np.zeros((R.size, 4, 4), dtype=d.dtype)
        S[:, :na, :nb] = (np.matmul(np.matmul(T, sl), T.transpose(0, 2, 1)))[:, :na, :nb]
        ra = R / _ANG if (A == 1 and B in (7, 8)) else 1.0
        rb = R / _ANG if (B == 1 and A in (7, 8)) else 1.0
        # the heavy atom's exponential carries R (in Angstrom) in N-H and O-H pairs
        f = 1.0 + rb * np.exp(-pa[4] * R) + ra * np.exp(-pb[4] * R)
        zz = float(pa[0] * pb[0])
        e = zz * x[:, 0, 0, 0, 0] * f
        if self.theory != "mndo":
            for k, l, m in pa[8] + pb[8]:
                e = e + zz * k * np.exp(-l * (R - m) ** 2) * _ANG / R
        return Wp, S, e

    def full(self, X):
        return X.transpose(0, 2, 1, 3).reshape(4 * self.A, 4 * self.A)[np.ix_(self.slots, self.slots)]

    def blocks(self, P):
        X = np.zeros((4 * self.A, 4 * self.A))
        X[np.ix_(self.slots, self.slots)] = P
        return X.reshape(self.A, 4, self.A, 4).transpose(0, 2, 1, 3)

    def fock(self, P):
        B = self.blocks(P)
        F = self.H.copy()
        ar = np.arange(self.A)
        D = B[ar, ar]
        n = self.ia.size
        W2 = self.Wp.reshape(n, 16, 16)
        one = np.zeros((self.A, 4, 4))
        np.add.at(one, self.ia, np.matmul(W2, D[self.ib].reshape(n, 16, 1)).reshape(n, 4, 4))
        np.add.at(one, self.ib, np.matmul(D[self.ia].reshape(n, 1, 16), W2).reshape(n, 4, 4))
        dg = np.einsum("amm->am", D)
        loc = (1.5 * self.X - 0.5 * self.G) * D
        for m in range(4):
            loc[:, m, m] = ((self.G[:, m] - 0.5 * self.X[:, m]) * dg).sum(axis=1)
        F[ar, ar] += one + loc
        K = np.einsum("pmnls,pns->pml", self.Wp, B[self.ia, self.ib], optimize=True)
        F[self.ia, self.ib] -= 0.5 * K
        F[self.ib, self.ia] -= 0.5 * K.transpose(0, 2, 1)
        return self.full(F)

    def solve(self):
        def density(F):
            w, v = np.linalg.eigh(F)
            return w, 2.0 * v[:, :self.nocc] @ v[:, :self.nocc].T
        _, P = density(self.guess)
        fs, es = [], []
        mixing = True
        for it in range(200):
            F = self.fock(P)
            e = F @ P - P @ F
            err = np.abs(e).max()
            if err < 2e-13 * len(P) ** 0.5:
                break
            mixing = mixing and err > 3e-2
            if mixing:
                P = 0.4 * density(F)[1] + 0.6 * P
                continue
            fs, es = (fs + [F])[-8:], (es + [e.ravel()])[-8:]
            k = len(fs)
            Bm = np.zeros((k + 1, k + 1))
            Bm[k, :k] = Bm[:k, k] = -1.0
            Bm[:k, :k] = [[a @ b for b in es] for a in es]
            sc = Bm[k - 1, k - 1]
            Bm[:k, :k] /= sc
            c = np.linalg.lstsq(Bm, np.r_[np.zeros(k), -1.0], rcond=1e-14)[0][:k]
            P = density(sum(ci * f for ci, f in zip(c, fs)))[1]
        self.eps, self.P = density(self.fock(P))
        F, Hf = self.fock(self.P), self.full(self.H)
        self.energy = 0.5 * float((self.P * (F + Hf)).sum()) + self.ecore + self.e_epc
        pop = np.einsum("aamm->a", self.blocks(self.P))
        self.charges = self.core - pop
        return self

    def pair_energy(self, d):
        """Energy of every pair at the converged density."""
        Wp, S, ec = self.pairs(d)
        B = self.blocks(self.P)
        Da, Db, Pab = B[self.ia, self.ia], B[self.ib, self.ib], B[self.ia, self.ib]
        n = self.ia.size
        W2 = Wp.reshape(n, 16, 16)
        e = np.matmul(np.matmul(Da.reshape(n, 1, 16), W2), Db.reshape(n, 16, 1))[:, 0, 0]
        e = e - self.core[self.ib] * (Da * Wp[:, :, :, 0, 0]).sum(axis=(1, 2))
        e = e - self.core[self.ia] * (Db * Wp[:, 0, 0]).sum(axis=(1, 2))
        K = np.einsum("pmnls,pns->pml", Wp, Pab, optimize=True)
        e = e - 0.5 * (K * Pab).sum(axis=(1, 2))
        bb = self.beta[self.ia][:, :, None] + self.beta[self.ib][:, None, :]
        return e + (Pab * bb * S).sum(axis=(1, 2)) + ec

    def forces(self):
        d = self.xyz[self.ib] - self.xyz[self.ia]
        F = np.zeros((self.A, 3))
        for k in range(3):
            dz = d.astype(complex)
            dz[:, k] += 1e-30j
            g = self.pair_energy(dz).imag / 1e-30
            np.add.at(F[:, k], self.ib, -g)
            np.add.at(F[:, k], self.ia, g)
        return F


def exact(case, seed):
    kind = case["kind"]
    if kind == "single" and 6 * case["size"] <= 700:
        m = _Nddo(case["theory"], _single(case, seed)).solve()
        out = {"energy": m.energy, "core_repulsion": m.ecore, "eps": m.eps, "charges": m.charges, "density": m.P,
               "dipole": None}   # its STO-6G moments have no place here
        if case["forces"]:
            out["forces"] = m.forces()
        return out
    if kind == "integrals":
        mol = W.water_cluster_k(case["size"], seed)
        m = _Nddo(case["theory"], mol)
        tri = np.triu_indices(4)
        blocks = []
        heavy = (m.nao[m.ia] == 4, m.nao[m.ib] == 4)
        one = (np.array([0]), np.array([0]))
        for a in (0, 1):
            for b in (0, 1):
                sel = np.nonzero((heavy[0] == a) & (heavy[1] == b))[0]
                ra, rb = (tri if a else one), (tri if b else one)
                blocks.append((sel, m.Wp[sel][:, ra[0], ra[1]][:, :, rb[0], rb[1]].reshape(sel.size, -1)))
        size = np.where(heavy[0], 10, 1) * np.where(heavy[1], 10, 1)
        at = np.concatenate([[0], np.cumsum(size)])
        flat = np.zeros(at[-1])
        for sel, v in blocks:
            flat[at[sel][:, None] + np.arange(v.shape[1])] = v
        return {"blocks": flat, "core_hamiltonian": m.full(m.H), "core_repulsion": m.ecore}
    if kind == "batch" and case["count"] * (6 * case["size"]) ** 2.5 < 4e6:
        mols = [_Nddo(case["theory"], x).solve() for x in _batch(case, seed)]
    elif kind in ("uneven", "server") and case["count"] * case["largest"] ** 2 < 4e5:
        mols = [_Nddo(case["theory"], x).solve() for x in _uneven(case, seed)]
    else:
        return None   # too long in numpy
    return {"energy": np.array([m.energy for m in mols]), "core_repulsion": np.array([m.ecore for m in mols]),
            "charges": np.concatenate([m.charges for m in mols]), "status": None, "dipole": None}
