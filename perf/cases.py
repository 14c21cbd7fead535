"""What a user of this library has it do, as cases that can be timed and compared.

Every case is one call of a public method of ``rustb_gb300.Model`` on a model
the program already holds.  Models are seeded: random Hermitian-closed hopping
tables with the statistics of ``rustb_gb300.workloads`` (amplitude decaying
with |R|, 10 % spin-orbit blocks), the Haldane and honeycomb models and the
supercell.  FP64 is the default precision of every method, so most cases use
it; MIXED is what large meshes of many bands ask for.

Fields of a case: ``kind`` (the call), ``model``, ``dim``, ``norb``, ``spin``
(spinful basis), ``rmax`` (hoppings in the box |R_i| <= rmax), ``rmat``
(position matrix), ``precision`` and the sizes of the call.
"""

import itertools
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np

from rustb_gb300 import Integration, Model, Parameters, Precision, SpinDirection

K_B = 8.617333262145e-5  # eV / K
ETA = 1e-3


def _case(kind, model="random", **kw):
    c = {"kind": kind, "model": model, "dim": 2, "norb": 2, "spin": False, "rmax": 1, "rmat": False,
         "precision": "fp64"}
    c.update(kw)
    return c


def listed():
    return [
        # The reference's own smallest Hall call: one mu on a coarse mesh; launches and host work are all of it.
        _case("hall", "haldane", name="hall_haldane_31", n0=31, n1=31, n2=1, nmu=1, T=0.0, sdir=-1),
        # gen_v at one k-point, as a program that walks k-points itself calls it.
        _case("velocity", name="velocity_one_k_18", dim=3, norb=9, spin=True, rmax=2, nk=1),
        # A band structure along a k-path of a small Wannier-sized spinful model.
        _case("bands", name="bands_path_14", dim=3, norb=7, spin=True, rmax=2, nk=301),
        # Density of states of the two-band honeycomb model on the mesh of the reference's benchmark.
        _case("dos", "honeycomb", name="dos_honeycomb_1000", n0=1000, n1=1000, n2=1, npt=500, sigma=1e-2),
        # Energy-cut Hall conductivity on the reference's own mesh and mu grid.
        _case("hall_ec", "haldane", name="ec_haldane_101", n0=101, n1=101, n2=1, nmu=201),
        # Spin Hall conductivity at room temperature over a mu window, 26 bands.
        _case("hall", name="spin_hall_26", dim=2, norb=13, spin=True, rmax=2, n0=48, n1=48, n2=1, nmu=41, T=300.0,
              sdir=2),
        # A Berry-curvature map of an odd-sized Wannier model with its position matrix.
        _case("berry", name="berry_map_33", dim=2, norb=33, rmax=3, rmat=True, nk=1681),
        # Hybrid Wannier centres of a 64-band model, half of them occupied.
        _case("wannier", name="wannier_64", dim=2, norb=32, spin=True, rmax=2, nk1=64, nk2=64, nocc=32),
        # A slab of the mesh of the 128-band, 343-R spinful model in the default precision.
        _case("hall", name="hall_128", dim=3, norb=64, spin=True, rmax=3, n0=16, n1=8, n2=8, nmu=1, T=0.0, sdir=-1),
        # The same model on the batch of 8192 k-points that bench.py times, mixed precision.
        _case("hall", name="hall_128_mixed", dim=3, norb=64, spin=True, rmax=3, n0=16, n1=16, n2=32, nmu=1, T=0.0,
              sdir=-1, precision="mixed"),
        # Quantum geometry per band of the largest band counts of the uneven batch, odd size, mixed precision.
        _case("geometry", name="geometry_251_mixed", dim=2, norb=251, rmax=1, nk=304, precision="mixed"),
        # Band energies of a supercell at a few k-points: large matrices, fewer of them than the GPU has SMs.
        _case("bands", "supercell", name="bands_supercell_512", norb=512, nk=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nsta(case):
    return case["norb"] * (2 if case["spin"] else 1)


def _nR(case):
    return {"haldane": 7, "honeycomb": 5}.get(case["model"], (2 * case["rmax"] + 1) ** case["dim"])


def _nk(case):
    if case["kind"] in ("hall", "hall_ec", "dos"):
        return case["n0"] * case["n1"] * case["n2"]
    if case["kind"] == "wannier":
        return case["nk1"] * (case["nk2"] - 1)
    return case["nk"]


def draw(rng):
    kind = rng.choice(["hall", "hall", "hall", "bands", "bands", "berry", "geometry", "velocity", "wannier", "dos",
                       "hall_ec"])
    dim = rng.choice([2, 3])
    spin = rng.random() < 0.5
    mesh = lambda nk: dict(zip(("n0", "n1", "n2"), _mesh(rng, dim, nk)))  # noqa: E731
    if kind == "hall_ec":
        n = _log_int(rng, 20, 120)
        return _case(kind, "haldane", n0=n, n1=rng.randint(20, 120), n2=1, nmu=_log_int(rng, 10, 300))
    if kind == "dos":
        n = _log_int(rng, 60, 1000)
        return _case(kind, "honeycomb", n0=n, n1=_log_int(rng, 60, 1000), n2=1, npt=_log_int(rng, 50, 600),
                     sigma=rng.uniform(5e-3, 5e-2))
    if kind == "hall" and rng.random() < 0.25:
        return _case(kind, "haldane", n0=_log_int(rng, 21, 300), n1=_log_int(rng, 21, 300), n2=1,
                     nmu=_log_int(rng, 1, 60), T=rng.choice([0.0, 100.0, 300.0]), sdir=-1)
    if kind == "wannier":
        n = _log_int(rng, 8, 64)
        return _case(kind, dim=dim, norb=max(4, n // 2 if spin else n), spin=spin, rmax=rng.choice([1, 2]),
                     nk1=rng.randint(5, 64), nk2=rng.randint(9, 64),
                     nocc=max(1, min(32, int((max(4, n // 2) * 2 if spin else n) * rng.uniform(0.2, 0.6)))))
    mixed = kind in ("hall", "geometry", "berry") and rng.random() < 0.35
    n = _log_int(rng, 40, 256) if mixed else _log_int(rng, 3, 128)
    norb = max(2, n // 2) if spin else n
    rmax = rng.choice([1, 2, 3] if n <= 128 else [1, 2])
    c = _case(kind, dim=dim, norb=norb, spin=spin, rmax=rmax, precision="mixed" if mixed else "fp64")
    if kind == "velocity":
        c["nk"] = _log_int(rng, 1, max(2, int(2e6 / n ** 2)))
        return c
    # k-points so that a call costs at most what the largest listed ones do
    per_k = (12.0 * _nR(c) + 60.0 * n) * n * n
    most = int(min(40000, max(4, (4e11 if mixed else 1.4e11) / per_k)))
    nk = _log_int(rng, max(1, most // 100), most)
    if kind == "hall":
        c.update(mesh(nk), nmu=_log_int(rng, 1, 60), T=rng.choice([0.0, 100.0, 300.0]),
                 sdir=rng.choice([-1, 0, 1, 2]) if spin else -1)
    else:
        c["nk"] = nk
        if kind == "berry" and not mixed:
            c["rmat"] = rng.random() < 0.3
    return c


def _mesh(rng, dim, nk):
    if dim == 2:
        a = max(2, int(round(math.sqrt(nk) * math.exp(rng.uniform(-0.3, 0.3)))))
        return a, max(2, nk // a), 1
    a = max(2, int(round(nk ** (1 / 3) * math.exp(rng.uniform(-0.3, 0.3)))))
    b = max(2, int(round(math.sqrt(nk / a) * math.exp(rng.uniform(-0.3, 0.3)))))
    return a, b, max(2, nk // (a * b))


# ------------------------------------------------------------------ inputs --
def _cn(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / math.sqrt(2.0)


def _half(dim, rmax):
    """R != 0 in the box whose first non-zero component is positive."""
    out = []
    for R in itertools.product(range(-rmax, rmax + 1), repeat=dim):
        nz = [c for c in R if c != 0]
        if nz and nz[0] > 0:
            out.append(R)
    return out


def _tables(case, seed):
    """(lat, orb, hamR, ham, rmatrix or None) of the case's model."""
    rng = np.random.default_rng([20260101, int(seed)])
    if case["model"] in ("haldane", "honeycomb"):
        s3 = math.sqrt(3.0)
        hal = case["model"] == "haldane"
        lat = np.array([[s3, -1.0], [s3, 1.0]] if hal else [[1.0, 0.0], [0.5, s3 / 2.0]])
        orb = np.array([[0.0, 0.0], [1 / 3, 1 / 3]] if hal else [[1 / 3, 1 / 3], [2 / 3, 2 / 3]])
        hops = {}
        on = (0.2 if hal else 0.7) * rng.uniform(0.9, 1.1)
        for (i, j, R, t) in [(0, 0, (0, 0), -on if not hal else on), (1, 1, (0, 0), on if not hal else -on)]:
            hops.setdefault(R, np.zeros((2, 2), complex))[i, j] = t
        t2 = 0.3 * rng.uniform(0.9, 1.1) if hal else 0.0
        terms = [(0, 1, R, -1.0) for R in [(0, 0), (-1, 0), (0, -1)]]
        if hal:
            terms += [(0, 0, R, t2 * 1j) for R in [(1, 0), (-1, 1), (0, -1)]]
            terms += [(1, 1, R, t2 * 1j) for R in [(-1, 0), (1, -1), (0, 1)]]
        for i, j, R, t in terms:
            hops.setdefault(R, np.zeros((2, 2), complex))[i, j] += t
            hops.setdefault((-R[0], -R[1]), np.zeros((2, 2), complex))[j, i] += np.conj(t)
        Rs = [(0, 0)] + [R for R in hops if R != (0, 0)]
        return lat, orb, np.array(Rs, dtype=np.int64), np.array([hops[R] for R in Rs]), None
    dim, norb, spin = case["dim"], case["norb"], case["spin"]
    lat = np.eye(dim)
    orb = rng.uniform(0.0, 1.0, (norb, dim))
    n = _nsta(case)
    half = _half(dim, case["rmax"])
    nR = 1 + 2 * len(half)
    hamR = np.zeros((nR, dim), dtype=np.int64)
    ham = np.empty((nR, n, n), dtype=np.complex128)

    def block(R, hermitise):
        if case["model"] == "supercell":
            d = orb[None, :, :] + np.asarray(R, dtype=np.float64)[None, None, :] - orb[:, None, :]
            amp = np.exp(-np.sqrt((d * d).sum(-1)) / 0.8)
        else:
            amp = math.exp(-math.sqrt(sum(c * c for c in R)) / 1.2) / math.sqrt(norb)
        herm = (lambda a: 0.5 * (a + a.conj().T)) if hermitise else (lambda a: a)
        a0 = herm(amp * _cn(rng, (norb, norb)))
        if not spin:
            return a0
        ax, ay, az = (herm(0.1 * amp * _cn(rng, (norb, norb))) for _ in range(3))
        return np.block([[a0 + az, ax - 1j * ay], [ax + 1j * ay, a0 - az]])

    ham[0] = block((0,) * dim, True)
    if case["model"] == "supercell":
        np.fill_diagonal(ham[0], rng.uniform(-0.5, 0.5, n))
    for q, R in enumerate(half):
        ham[1 + 2 * q] = block(R, False)
        ham[2 + 2 * q] = ham[1 + 2 * q].conj().T
        hamR[1 + 2 * q] = R
        hamR[2 + 2 * q] = [-c for c in R]
    rmat = None
    if case["rmat"]:
        rmat = np.empty((nR, dim, n, n), dtype=np.complex128)
        for r in range(nR):
            amp = 0.1 * math.exp(-math.sqrt(float((hamR[r] ** 2).sum())))
            if r == 0:
                a = amp * _cn(rng, (dim, n, n))
                rmat[0] = 0.5 * (a + a.conj().transpose(0, 2, 1))
            elif r % 2 == 1:
                rmat[r] = amp * _cn(rng, (dim, n, n))
            else:
                rmat[r] = rmat[r - 1].conj().transpose(0, 2, 1)
    return lat, orb, hamR, ham, rmat


def _kpoints(case, seed):
    rng = np.random.default_rng([7, int(seed)])
    dim = case["dim"]
    if case["kind"] in ("berry", "geometry"):  # a plane of the zone, shifted off the symmetric points
        n = max(1, int(math.sqrt(case["nk"])))
        i = np.arange(case["nk"])
        k = np.zeros((case["nk"], dim))
        k[:, 0], k[:, 1] = (i // n) / n, (i % n) / n
        return k + rng.uniform(0.0, 0.5, dim)
    if case["kind"] == "bands":  # a path between random corners
        corners = rng.uniform(-0.5, 0.5, (4, dim))
        t = np.linspace(0.0, 3.0, case["nk"])
        seg = np.minimum(t.astype(int), 2)
        return corners[seg] + (t - seg)[:, None] * (corners[seg + 1] - corners[seg])
    return rng.uniform(0.0, 1.0, (case["nk"], dim))


def _directions(dim):
    return np.eye(dim)[0], np.eye(dim)[1]


def _energy_window(case):
    """mu grid of a Hall call: around the middle of the spectrum."""
    w = {"haldane": 1.2}.get(case["model"], 0.8)
    if case["nmu"] == 1:
        return np.array([0.05])
    return np.linspace(-w, w, case["nmu"])


def _wannier_path(case, seed):
    rng = np.random.default_rng([11, int(seed)])
    dim = case["dim"]
    d1, d2 = np.eye(dim)[0], np.eye(dim)[1]
    return rng.uniform(0.0, 0.3, dim), d1, d2


# ------------------------------------------------------------------- calls --
def prepare(case, seed):
    lat, orb, hamR, ham, rmat = _tables(case, seed)
    model = Model(lat, orb, case["spin"], ham=ham, hamR=hamR)
    if rmat is not None:
        model.set_rmatrix(rmat)
    model.device_handle()  # resident on the GPU, as a program keeps it
    state = {"case": case, "model": model,
             "precision": Precision.MIXED if case["precision"] == "mixed" else Precision.FP64}
    a, b = _directions(lat.shape[0])
    kind = case["kind"]
    if kind in ("hall", "hall_ec"):
        mesh = (case["n0"], case["n1"], case["n2"])[: lat.shape[0]]
        p = Parameters.rank2(mesh, a, b, _energy_window(case))
        if kind == "hall_ec":
            p = p.with_integration(Integration.EnergyCut)
            p.eta = 0.05
        else:
            p = p.with_temperature(case["T"])
            if case["sdir"] >= 0:
                p = p.with_spin(SpinDirection(case["sdir"]))
        state["params"] = p
    elif kind in ("berry", "geometry"):
        state["params"] = Parameters.rank2((1,) * lat.shape[0], a, b, [0.0])
        state["k"] = _kpoints(case, seed)
    elif kind in ("bands", "velocity"):
        state["k"] = _kpoints(case, seed)
    elif kind == "wannier":
        state["path"] = _wannier_path(case, seed)
    return state


def run(state):
    c, m = state["case"], state["model"]
    kind = c["kind"]
    if kind in ("hall", "hall_ec"):
        return m.hall_conductivity(state["params"], state["precision"]).conductivity
    if kind == "bands":
        return m.solve_band_all_parallel(state["k"])
    if kind == "berry":
        om, e = m.berry_curvature_on(state["k"], state["params"], state["precision"])
        return {"omega": om, "energies": e}
    if kind == "geometry":
        g = m.quantum_geometry_on(state["k"], state["params"], state["precision"])
        return {"metric": g.metric, "omega": g.berry_curvature, "energies": g.energies}
    if kind == "velocity":
        v, h = m.gen_v_batch(state["k"])
        return {"v": v, "h": h}
    if kind == "wannier":
        ks, d1, d2 = state["path"]
        return m.wannier_centre(range(c["nocc"]), ks, d1, d2, c["nk1"], c["nk2"])
    if kind == "dos":
        return m.dos((c["n0"], c["n1"]), -4.0, 4.0, c["npt"], c["sigma"])[1]
    raise ValueError(kind)


def work(case):
    """Bytes: the hop table and the k-points read, the outputs written.  Flops:
    Fourier sums over R and -R together for Hermitian matrices, the reduction
    to tridiagonal form, the eigenvectors and the rotation where they are used."""
    n, nR, nk, dim = _nsta(case), _nR(case), _nk(case), case["dim"]
    kind = case["kind"]
    table = 16.0 * nR * n * n * (1 + (dim if case["rmat"] else 0))
    fourier = 2.0 * nR * n * n  # one Hermitian matrix per k
    values, vectors, rotate = 16.0 / 3.0 * n ** 3, 8.0 * n ** 3, 24.0 * n ** 3
    if kind in ("hall", "hall_ec"):
        return {"bytes": table + 16.0 * case["nmu"], "flops": nk * (3 * fourier + values + vectors + rotate)}
    if kind in ("berry", "geometry"):
        outs = 2 if kind == "berry" else 3
        extra = (2 * dim * fourier + 16.0 * n ** 3) if case["rmat"] else 0.0
        return {"bytes": table + 8.0 * nk * (dim + outs * n), "flops": nk * (3 * fourier + values + vectors + rotate
                                                                              + extra)}
    if kind == "bands":
        return {"bytes": table + 8.0 * nk * (dim + n), "flops": nk * (fourier + values)}
    if kind == "velocity":
        return {"bytes": table + nk * (8.0 * dim + 16.0 * (1 + dim) * n * n), "flops": nk * fourier * (1 + dim)}
    if kind == "wannier":
        o = case["nocc"]
        return {"bytes": table + 8.0 * nk * dim + 8.0 * case["nk1"] * o,
                "flops": nk * (fourier + values + vectors + 8.0 * n * o * o + 40.0 * o ** 3)}
    inside = 2.0 * 38.6 * case["sigma"] / 8.0 * case["npt"]  # grid points that a Gaussian reaches
    return {"bytes": table + 16.0 * case["npt"], "flops": nk * (fourier + values) + 3.0 * nk * n * min(inside,
                                                                                                       case["npt"])}


# ------------------------------------------------------- the same in numpy --
def _mesh_k(ns):
    g = np.meshgrid(*[np.arange(n) / n for n in ns], indexing="ij")
    return np.stack([x.reshape(-1) for x in g], axis=1)


def _tau(orb, spin):
    return np.concatenate([orb, orb]) if spin else orb


def _bloch(tab, spin, k, dirs=None):
    """Atom-gauge H(k) (and the velocities along ``dirs``)."""
    lat, orb, hamR, ham, rmat = tab
    n = ham.shape[1]
    u = np.exp(2j * np.pi * (k @ hamR.T))
    tau = _tau(orb, spin)
    phi = np.exp(2j * np.pi * (k @ tau.T))
    g = phi.conj()[:, :, None] * phi[:, None, :]
    hop = ham.reshape(len(ham), n * n)
    h0 = (u @ hop).reshape(-1, n, n)
    h = h0 * g
    if dirs is None:
        return h
    vs = []
    for w in dirs:
        t = tau @ lat @ w
        v = ((u * (1j * (hamR @ lat @ w))) @ hop).reshape(-1, n, n)
        v = (v + 1j * (t[None, None, :] - t[None, :, None]) * h0) * g
        if rmat is not None:
            a = np.einsum("kr,rx->kx", u, np.einsum("d,rdij->rij", w, rmat).reshape(len(ham), n * n))
            a = a.reshape(-1, n, n) * g
            a[:, np.arange(n), np.arange(n)] = 0.0
            v = v + 1j * (h @ a - a @ h)
        vs.append(v)
    return h, vs


def _geometry(tab, case, k, sdir=-1):
    """(metric, Omega, E) per band."""
    n = _nsta(case)
    h, (va, vb) = _bloch(tab, case["spin"], k, _directions(case["dim"]))
    if sdir >= 0:
        s = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]][sdir]) / 2
        S = np.kron(s, np.eye(case["norb"]))
        va = 0.5 * (S @ va + va @ S)
    e, x = np.linalg.eigh(h)
    xh = x.conj().transpose(0, 2, 1)
    K = (xh @ va @ x) * (xh @ vb @ x).transpose(0, 2, 1)
    de = e[:, :, None] - e[:, None, :]
    K /= de * de + ETA * ETA
    K[:, np.arange(n), np.arange(n)] = 0.0
    G = K.sum(axis=2)
    return G.real, -2.0 * G.imag, e


def _over(k, fn, step=64):
    """fn on slices of the k-points, in threads (LAPACK releases the GIL)."""
    with ThreadPoolExecutor(max_workers=12) as ex:
        return list(ex.map(fn, [k[i: i + step] for i in range(0, len(k), step)]))


def exact(case, seed):
    n, nk, kind = _nsta(case), _nk(case), case["kind"]
    if kind == "hall_ec" or nk * float(n) ** 3 > 2e10 or nk * 4.0 * _nR(case) * n * n > 4e11:
        return None  # band tracking and clipped simplices have no short form; the others would take long
    tab = _tables(case, seed)
    if kind == "hall":
        k = _mesh_k((case["n0"], case["n1"], case["n2"])[: case["dim"]])
        mu, T = _energy_window(case), case["T"] * K_B

        def part(kk):
            _, om, e = _geometry(tab, case, kk, case["sdir"])
            x = e[:, :, None] - mu
            f = np.heaviside(-x, 0.5) if T == 0.0 else 1.0 / (1.0 + np.exp(np.clip(x / T, -50.0, 50.0)))
            return np.einsum("kn,knm->m", om, f)

        return np.sum(_over(k, part), axis=0) / nk / np.linalg.det(tab[0])
    if kind in ("berry", "geometry"):
        r = _over(_kpoints(case, seed), lambda kk: _geometry(tab, case, kk))
        g, om, e = (np.concatenate(x) for x in zip(*r))
        return {"omega": om, "energies": e} if kind == "berry" else {"metric": g, "omega": om, "energies": e}
    if kind == "bands":
        k = _kpoints(case, seed)
        return np.concatenate(_over(k, lambda kk: np.linalg.eigvalsh(_bloch(tab, case["spin"], kk)), 4))
    if kind == "velocity":
        h, v = _bloch(tab, case["spin"], _kpoints(case, seed), np.eye(case["dim"]))
        return {"v": np.stack(v, axis=1), "h": h}
    if kind == "wannier":
        ks, d1, d2 = _wannier_path(case, seed)
        n1, n2, o = case["nk1"], case["nk2"], case["nocc"]
        tau = _tau(tab[1], case["spin"])

        def loop(i):
            k = ks + d1 * (float(i[0]) / (n1 - 1)) + np.arange(n2)[:, None] / (n2 - 1.0) * d2
            _, x = np.linalg.eigh(_bloch(tab, case["spin"], k[:-1]))
            x = x[:, :, :o]
            last = np.exp(-2j * np.pi * (tau @ d2))[:, None] * x[0]
            x = np.concatenate([x, last[None]])
            u, _, vh = np.linalg.svd(x[:-1].conj().transpose(0, 2, 1) @ x[1:])
            p = np.eye(o, dtype=complex)
            for q in u @ vh:
                p = p @ q
            return np.sort(-np.angle(np.linalg.eigvals(p)))

        return np.stack(_over(np.arange(n1), loop, 1), axis=1)
    e = np.concatenate([x.reshape(-1) for x in _over(_mesh_k((case["n0"], case["n1"])), lambda kk: np.linalg.eigvalsh(
        _bloch(tab, case["spin"], kk)), 20000)])
    grid = -4.0 + (8.0 / (case["npt"] - 1)) * np.arange(case["npt"])
    s = case["sigma"]
    order = np.sort(e)

    def point(x):  # the Gaussian is below the smallest double beyond 39 widths
        w = order[np.searchsorted(order, x[0] - 39.0 * s): np.searchsorted(order, x[0] + 39.0 * s)]
        return np.exp(-((x[0] - w) / s) ** 2 / 2.0).sum()

    return np.array(_over(grid, point, 1)) / (s * math.sqrt(2.0 * math.pi) * nk)
