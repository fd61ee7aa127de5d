"""The work that users of this library have it do, as measurable cases.

A case is one pass through the public entry points: some steps of the Fraser
loop on a prepared domain and the read-back of the fields a user looks at, a
whole drop-in call, a heat solve, a neighbour search, or a training run of the
warm-start network.  Sizes are those of the tests and of bench.py.  `exact`
restates the same step in 64-bit torch from the equations alone.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from weldformgpu_gb300 import Domain_d, mlp, scenarios
from weldformgpu_gb300 import domain as _domain

# fields a user reads back after a run, with their components
MECH_FIELDS = (("u", 3), ("v", 3), ("rho", 1), ("sigma", 6), ("pl_strain", 1))
HEAT_FIELD = (("T", 1),)
CONTACT_FIELD = (("contforce", 3),)


def listed():
    return [
        # the reference's Compression example shape in the default form (FP64, bilinear,
        # radial return): the smallest domain anyone runs, launches and latency count
        dict(name="fp64_cylinder_540", kind="bilinear", precision=0, R=0.0025, H=0.005, steps=20),
        # the R 5 mm, H 10 mm compression of the parity tests, same form
        dict(name="fp64_cylinder_5k", kind="bilinear", precision=0, R=0.005, H=0.010, steps=10),
        # plain FP64 of the coupled Johnson-Cook compression at bench.py's medium size
        dict(name="fp64_jc_170k", kind="jc", precision=0, R=0.015, H=0.030, steps=4, network=False),
        # the reference's own contact (rigid plane, penalty law with friction), FP64
        dict(name="fp64_contact_plane_5k", kind="plane", precision=0, R=0.005, H=0.010, steps=10,
             dens=10, mu=0.1),
        # a whole drop-in call in the mixed form: create, setters, restart, steps, read-back,
        # destroy, from host arrays
        dict(name="mixed_dropin_11k", kind="dropin", precision=1, R=0.006, H=0.012, steps=20),
        # mixed form, the size of the from-rest comparison runs
        dict(name="mixed_jc_50k", kind="jc", precision=1, R=0.010, H=0.020, steps=20,
             network=False),
        # the headline workload: mixed form with the warm-start network, 786k particles
        dict(name="mixed_jc_network_786k", kind="jc", precision=1, R=0.025, H=0.050, steps=20,
             network=True),
        # a block under a many-triangle tool (contact law 1, friction, adaptive rebuild)
        dict(name="mixed_indentation_500k", kind="indent", precision=1, nx=100, ny=100, nz=50,
             level=5, steps=10),
        # heat conduction alone, plain FP64
        dict(name="fp64_heat_64k", kind="heat", precision=0, n_side=40, steps=20),
        # heat conduction alone, mixed form, bench.py's 100^3 box
        dict(name="mixed_heat_1M", kind="heat", precision=1, n_side=100, steps=40),
        # the allocation-free neighbour search on a caller's device arrays
        dict(name="search_static_19k", kind="search", R=0.008, H=0.012),
        # training of the warm-start network (train_jc_warm_start's batch), a short run
        dict(name="network_training", kind="train", pairs=262144, batch=4096, steps=100),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["bilinear", "jc64", "jc32", "plane", "dropin", "indent", "heat64", "heat32",
                       "search", "train"])
    dx = 0.0005

    def cylinder(lo, hi):        # radius and height of about lo .. hi particles, H/R in 1.5 .. 3
        n, aspect = _log_uniform(rng, lo, hi), rng.uniform(1.5, 3.0)
        r = (n / (math.pi * aspect)) ** (1.0 / 3.0)
        return dict(R=dx * max(4.0, round(r, 2)), H=dx * max(8, int(round(aspect * r))))

    if kind == "bilinear":
        return dict(kind="bilinear", precision=rng.choice([0, 0, 1]), steps=rng.randint(5, 20),
                    **cylinder(500, 30000))
    if kind == "jc64":
        return dict(kind="jc", precision=0, steps=rng.randint(2, 4), network=False,
                    **cylinder(3000, 170000))
    if kind == "jc32":
        return dict(kind="jc", precision=1, steps=rng.randint(5, 20), network=rng.random() < 0.5,
                    **cylinder(3000, 700000))
    if kind == "plane":
        return dict(kind="plane", precision=0, steps=rng.randint(5, 15), dens=rng.randint(7, 17),
                    mu=rng.choice([0.0, 0.1, 0.2]), **cylinder(1000, 20000))
    if kind == "dropin":
        return dict(kind="dropin", precision=1, steps=rng.randint(10, 40), **cylinder(2000, 100000))
    if kind == "indent":
        return dict(kind="indent", precision=1, nx=rng.randint(30, 110), ny=rng.randint(30, 110),
                    nz=rng.randint(15, 40), level=rng.randint(3, 5), steps=rng.randint(5, 10))
    if kind == "heat64":
        return dict(kind="heat", precision=0, n_side=int(_log_uniform(rng, 10, 48)),
                    steps=rng.randint(10, 40))
    if kind == "heat32":
        return dict(kind="heat", precision=1, n_side=int(_log_uniform(rng, 15, 100)),
                    steps=rng.randint(10, 40))
    if kind == "search":
        return dict(kind="search", **cylinder(1000, 50000))
    return dict(kind="train", pairs=rng.randint(60000, 300000), batch=int(_log_uniform(rng, 512, 8192)),
                steps=rng.randint(20, 100))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _options(case):
    o = {"precision": case["precision"]}
    if case["kind"] in ("jc", "dropin", "indent"):      # bench.py's options of the coupled runs
        o.update(return_map=1, thermal=1, taylor_quinney=0.9, rebuild_every=5,
                 rebuild_current_positions=1, rebuild_after_yield=0, energy_mode=1)
    return o


def _jitter(sc, rng, n, amount=0.01):
    x = np.array(sc["x"], dtype=np.float64)
    x[:n] += rng.uniform(-amount, amount, (n, 3)) * sc["dx"]
    sc["x"] = x
    return sc


def _scenario(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("bilinear", "search"):
        sc = scenarios.compression_cylinder(R=case["R"], H=case["H"], vz_top=-1.0)
        # a searched cloud has moved off its lattice
        return _jitter(sc, rng, sc["n"], 0.1 if kind == "search" else 0.01), rng
    if kind in ("jc", "dropin"):
        vz = -10.0 if case["R"] > 0.02 else -2.0
        return scenarios.jc_compression(R=case["R"], H=case["H"], seed=int(seed) + 1, vz_top=vz), rng
    if kind == "plane":
        # the plane just inside contact range of the top layer
        sc = scenarios.contact_cylinder(R=case["R"], H=case["H"], dens=case["dens"], v_plane=-2.0,
                                        gap=-2.0e-6, mu=(case["mu"], case["mu"]))
        return _jitter(sc, rng, sc["n_solid"], 0.002), rng
    if kind == "indent":
        dx = 0.00025
        sc = scenarios.indent_block(L=(case["nx"] * dx, case["ny"] * dx, case["nz"] * dx), dx=dx,
                                    R=0.01, level=case["level"], v_tool=-5.0, mu=0.3)
        sc["mesh"]["nodes"] = sc["mesh"]["nodes"] - np.array([0.0, 0.0, 8.0e-6])
        return _jitter(sc, rng, sc["n_solid"]), rng
    sc = scenarios.heat_box(n_side=case["n_side"])
    sc["T"] = sc["T"] + rng.uniform(0.0, 5.0, sc["n"])
    return sc, rng


def _jc_law(mat, eps_p, rate, T):
    th = np.clip((T - mat.Tt) / (mat.Tm - mat.Tt), 0.0, 0.999)
    return ((mat.A + mat.B * eps_p ** mat.n) * (1.0 + mat.C * np.log(rate / mat.eps0))
            * (1.0 - th ** mat.m))


def _plastic_state(case, sc, rng):
    """A checkpoint of a cylinder in steady plastic compression: uniaxial stress at yield,
    volume-preserving velocity field, smooth plastic strain with scatter."""
    n, x = sc["n"], sc["x"]
    z = x[:, 2] - x[:, 2].min()
    height = z.max()
    rate = -sc["bcs"][1][1][2] / height
    v = np.stack([0.5 * rate * x[:, 0], 0.5 * rate * x[:, 1], -rate * z], axis=1)
    v += rng.normal(0.0, 2e-3 * rate * height, (n, 3))
    wave = rng.uniform(0.3, 0.7)
    eps_p = 0.03 * (1.0 + 0.5 * np.sin(2.0 * np.pi * (z / height + wave))) * rng.uniform(0.95, 1.05, n)
    T = np.full(n, 20.0)
    if case["kind"] == "bilinear":
        mat = sc["mat"]
        sy = sc["sy"] + mat.E * mat.Et / (mat.E - mat.Et) * eps_p
    else:
        T = 20.0 + 150.0 * eps_p
        sy = _jc_law(sc["mat"], eps_p, rate, T)
    s = sy[:, None] * np.array([1.0 / 3.0, 1.0 / 3.0, -2.0 / 3.0, 0.0, 0.0, 0.0])
    p = sy / 3.0
    sigma = s.copy()
    sigma[:, :3] -= p[:, None]
    zero = np.zeros(n)
    return {"x": x, "m": sc["m"], "v": v, "rho": sc["rho"] + p / sc["Cs"] ** 2,
            "u": np.zeros((n, 3)), "a": np.zeros((n, 3)), "sigma": sigma, "shearstress": s,
            "strain": np.zeros((n, 6)), "pl_strain": eps_p, "sigma_y": sy, "int_energy": zero,
            "T": T, "Ta": T, "Tb": T, "dep": zero, "ID": sc["ids"], "_time": 0.0, "_step": 0,
            "_isfirst": 0, "_is_yielding": 1}


@functools.lru_cache(maxsize=2)
def _network():
    """Warm-start weights for the Johnson-Cook aluminium: random hidden layers, the output
    layer fitted to converged increments by least squares."""
    mat, G = scenarios.jc_compression(R=0.002, H=0.004)["mat"], 70e9 / 2.66
    rng = np.random.default_rng(7)
    n = 16384
    ratio, ep = rng.uniform(1.0, 3.0, n), 10.0 ** rng.uniform(-4.0, math.log10(2.0), n)
    rate, T = 10.0 ** rng.uniform(-2.0, 5.0, n), rng.uniform(20.0, 550.0, n)
    sy0 = _jc_law(mat, ep, rate, T)
    rt = sy0 / (mat.A + mat.B * ep ** mat.n)
    st, hi = ratio * sy0, (ratio - 1.0) * sy0 / (3.0 * G)
    dl = hi.copy()
    for _ in range(60):
        f = st - 3.0 * G * dl - (mat.A + mat.B * (ep + dl) ** mat.n) * rt
        dl += f / (3.0 * G + mat.n * mat.B * (ep + dl) ** (mat.n - 1.0) * rt)
    X = np.stack([ratio - 1.0, (np.log10(ep + 1e-6) + 3.0) / 3.0, (np.log10(rate) - 1.5) / 3.5,
                  np.clip((T - mat.Tt) / (mat.Tm - mat.Tt), 0.0, 0.999)], axis=1)
    silu = lambda q: q / (1.0 + np.exp(-q))  # noqa: E731
    P = mlp.init_params(5).astype(np.float64)
    W1, W2 = P[:256].reshape(64, 4), P[320:320 + 4096].reshape(64, 64)
    h = np.column_stack([silu(silu(X @ W1.T) @ W2.T), np.ones(n)])
    P[320 + 4096 + 64:] = np.linalg.lstsq(h, dl / np.maximum(hi, 1e-300), rcond=None)[0]
    return P.astype(np.float32)


def _buffers(fields, n):
    """Page-locked output arrays, as a program that reads results back often keeps."""
    return {f: torch.empty(n * c, dtype=torch.float64, pin_memory=True).numpy() for f, c in fields}


def _fields(case):
    kind = case["kind"]
    return (MECH_FIELDS + (HEAT_FIELD if kind in ("jc", "dropin", "indent") else ())
            + (CONTACT_FIELD if kind in ("plane", "indent") else ()))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, Y = _pairs(case, seed)
        return {"kind": kind, "X": X, "Y": Y, "P": mlp.init_params(seed % 1000),
                "steps": case["steps"], "batch": case["batch"]}
    sc, rng = _scenario(case, seed)
    n = sc["n"]
    if kind == "search":
        f = _domain.lib().wf_find_neighbors_static
        f.restype = ctypes.c_int
        f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_double, ctypes.c_void_p,
                      ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p, ctypes.c_int64]
        return {"kind": kind, "f": f, "n": n, "h": sc["h"],
                "x": torch.from_numpy(sc["x"]).cuda().contiguous(),
                "counts": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "lists": torch.full((n, 70), -1, dtype=torch.int32, device="cuda"),
                "err": ctypes.create_string_buffer(256)}
    if kind == "dropin":
        return {"kind": kind, "sc": sc, "state": _plastic_state(case, sc, rng),
                "options": _options(case), "steps": case["steps"], "fields": _fields(case),
                "out": _buffers(_fields(case), n)}
    if kind == "heat":
        d = scenarios.load_heat(Domain_d(n), sc)
        d.set_option("precision", case["precision"])
        return {"kind": kind, "d": d, "tf": (case["steps"] - 0.5) * sc["dt"], "fields": HEAT_FIELD,
                "out": _buffers(HEAT_FIELD, n)}
    d = scenarios.load(Domain_d(n), sc, _options(case))
    if kind in ("jc", "bilinear"):
        d.restore(_plastic_state(case, sc, rng))
    if case.get("network"):
        d.set_mlp_weights(_network())
        d.set_option("mlp", 1)
    return {"kind": "steps", "d": d, "steps": case["steps"], "fields": _fields(case),
            "out": _buffers(_fields(case), n)}


def run(state):
    kind = state["kind"]
    if kind == "train":
        return mlp.train(state["P"], state["X"], state["Y"], steps=state["steps"],
                         batch=state["batch"])
    if kind == "search":
        rc = state["f"](state["x"].data_ptr(), state["n"], state["h"], state["counts"].data_ptr(),
                        state["lists"].data_ptr(), torch.cuda.current_stream().cuda_stream,
                        state["err"], 256)
        if rc:
            raise RuntimeError(state["err"].value.decode())
        return state["counts"], state["lists"]
    if kind == "dropin":
        sc = state["sc"]
        d = scenarios.load(Domain_d(sc["n"]), sc, state["options"])
        d.restore(state["state"])
        d.step(state["steps"])
        out = {f: d.get_field(f, out=state["out"][f]) for f, _ in state["fields"]}
        d.close()
        return out
    d = state["d"]
    if kind == "heat":
        d.thermal_solve(state["tf"])
    else:
        d.step(state["steps"])
    return {f: d.get_field(f, out=state["out"][f]) for f, _ in state["fields"]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _count(case):
    """Particles of a case, from its dimensions."""
    kind, dx = case["kind"], 0.0005
    if kind == "heat":
        return case["n_side"] ** 3
    if kind == "indent":
        return case["nx"] * case["ny"] * case["nz"]
    return int(math.pi * (case["R"] / dx) ** 2 * (case["H"] / dx))


def work(case):
    kind = case["kind"]
    if kind == "train":
        used = min(case["batch"] * case["steps"], case["pairs"])
        return {"bytes": 20 * used + 8 * mlp.NPARAM,
                "flops": 6 * mlp.NPARAM * case["batch"] * case["steps"]}
    n, nb = _count(case), 56
    if kind == "search":       # positions in, lists out; 27 cells of ~14 candidates, 9 operations
        return {"bytes": n * (24 + 4 + 4 * nb), "flops": n * 27 * 14 * 9}
    if kind == "heat":         # T and its half step in and out, each step; the fixed arrays once
        return {"bytes": n * (case["steps"] * 32 + 56), "flops": n * nb * 20 * case["steps"]}
    real = 8 if case["precision"] == 0 else 4
    # per particle and step, in and out: x, v, u, rho in 64 bits, deviatoric stress in the form's
    # precision, plastic strain and yield stress, T and its half step where heat is on
    heat = kind in ("jc", "dropin", "indent")
    state = 10 * 8 + 6 * real + 2 * 8 + (2 * 8 if heat else 0)
    out = 8 * sum(c for _, c in _fields(case))
    return {"bytes": n * (2 * state * case["steps"] + out),
            "flops": n * nb * (110 + (20 if heat else 0)) * case["steps"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "train":
        return _exact_train(case, seed, dev)
    if kind == "search":
        return None                              # whole numbers
    sc, rng = _scenario(case, seed)
    if kind == "heat":
        return _exact_heat(case, sc, dev)
    st = _plastic_state(case, sc, rng) if kind in ("jc", "dropin", "bilinear") else None
    return _exact_steps(case, sc, st, dev)


def _pair_list(x, h):
    """Pairs (i, j) with a float32 squared distance in (0, (2h)^2), sorted by i and, for one i, in
    cell order (z, y, x, index); at most 70 for each i."""
    r = np.float32(2.0 * h)
    p = x.to(torch.float32)
    cell = torch.floor(p / float(r)).to(torch.int64)
    cell = cell - cell.min(dim=0).values + 1
    dim = (cell.max(dim=0).values + 2).tolist()
    lin = (cell[:, 2] * dim[1] + cell[:, 1]) * dim[0] + cell[:, 0]
    order = torch.sort(lin, stable=True).indices
    start = torch.searchsorted(lin[order], torch.arange(dim[0] * dim[1] * dim[2] + 1, device=x.device))
    r2 = float(r * r)
    found = []
    step = 200000                                # particles at a time: bounded memory
    for i0 in range(0, len(p), step):
        me = torch.arange(i0, min(i0 + step, len(p)), device=x.device)
        part = []
        for row, (dz, dy) in enumerate((z, y) for z in (-1, 0, 1) for y in (-1, 0, 1)):
            c = lin[me] + (dz * dim[1] + dy) * dim[0]
            b, e = start[c - 1], start[c + 2]
            k = b[:, None] + torch.arange(int((e - b).max()), device=x.device)
            i, q = torch.nonzero(k < e[:, None], as_tuple=True)
            j = order[k[i, q]]
            i = me[i]
            d = p[j] - p[i]
            s = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
            ok = (s < r2) & (s > 0)
            part.append((i[ok], j[ok]))
        i, j = torch.cat([a for a, _ in part]), torch.cat([b for _, b in part])
        o = torch.sort(i, stable=True).indices
        found.append((i[o], j[o]))
    i, j = torch.cat([a for a, _ in found]), torch.cat([b for _, b in found])
    first = torch.searchsorted(i, torch.arange(len(p), device=x.device))
    keep = torch.arange(len(i), device=x.device) - first[i] < 70
    return i[keep], j[keep]


def _grad(r, h):
    """The cubic spline's W'(r) / r."""
    q = r / h
    c = 1.0 / (math.pi * h ** 4)
    inner = c / h * (-3.0 + 2.25 * q)
    outer = c / (q * h) * (-0.75 * (2.0 - q) ** 2)
    return torch.where(q < 1.0, inner, torch.where(q < 2.0, outer, torch.zeros_like(q)))


def _sum_to(n, i, a):
    return torch.zeros((n,) + a.shape[1:], dtype=a.dtype, device=a.device).index_add_(0, i, a)


def _heat_rate(x, rho, m, T, k, cp, h, i, j):
    d = x[i] - x[j]
    r = d.norm(dim=1)
    s = m[j] / rho[j] * (2.0 * k) * (T[i] - T[j]) * _grad(r, h)
    return _sum_to(len(x), i, s) / (rho * cp)


def _exact_heat(case, sc, dev):
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    x, m, T = t(sc["x"]), t(sc["m"]), t(sc["T"])
    outer = t(sc["bc_t"]) == 1
    rho = torch.full_like(m, sc["rho"])
    i, j = _pair_list(x, sc["h"])
    area = (m / rho) ** (2.0 / 3.0)
    Ta = None
    for _ in range(case["steps"]):
        rate = _heat_rate(x, rho, m, T, sc["k"], sc["cp"], sc["h"], i, j)
        rate = rate + outer * sc["h_conv"] * area * (sc["T_inf"] - T) / (m * sc["cp"])
        if Ta is None:
            Ta = T - 0.5 * sc["dt"] * rate
            continue
        new = Ta + sc["dt"] * rate
        T, Ta = 0.5 * (new + Ta), new
    return {"T": T}


def _cross_product_rule(a, b):
    """The product of two 3x3 tensors as the step defines it: column x of A.B, columns y and z of
    A.B^T."""
    full, trans = a @ b, a @ b.transpose(1, 2)
    return torch.cat([full[:, :, :1], trans[:, :, 1:]], dim=2)


def _sym(f):
    return torch.stack([f[:, 0], f[:, 3], f[:, 5], f[:, 3], f[:, 1], f[:, 4], f[:, 5], f[:, 4],
                        f[:, 2]], dim=1).reshape(-1, 3, 3)


def _stress(case, sc, S6, D, W, T, eps_p, sy, dt):
    """Jaumann update of the deviatoric stress and the return map: (stress, plastic strain, yield
    stress, increment)."""
    mat, G = sc["mat"], sc["G"]
    S, eye = _sym(S6), torch.eye(3, dtype=D.dtype, device=D.device)
    tr = (D.diagonal(dim1=1, dim2=2).sum(1) / 3.0)[:, None, None]
    S = S + dt * (2.0 * G * (D - tr * eye) + _cross_product_rule(S, W.transpose(1, 2))
                  + _cross_product_rule(W, S))
    dg = D.diagonal(dim1=1, dim2=2)
    rate = torch.sqrt(0.5 * ((dg[:, 0] - dg[:, 1]) ** 2 + (dg[:, 1] - dg[:, 2]) ** 2
                             + (dg[:, 2] - dg[:, 0]) ** 2)
                      + 3.0 * (D[:, 0, 1] ** 2 + D[:, 1, 2] ** 2 + D[:, 2, 0] ** 2))
    j2 = 0.5 * (S * S.transpose(1, 2)).sum(dim=(1, 2))
    st = torch.sqrt(3.0 * j2)
    if "return_map" not in _options(case):       # bilinear, one-shot radial return
        scale = torch.where(sy < st, sy / st, torch.ones_like(st))
        dl = torch.where(st > sy, (st - sy) / (3.0 * G), torch.zeros_like(st))
        sy1 = sy + dl * (mat.E * mat.Et / (mat.E - mat.Et))
    else:                                        # Johnson-Cook, consistent return map
        th = ((T - mat.Tt) / (mat.Tm - mat.Tt)).clamp(0.0, 0.999)
        rt = ((1.0 + mat.C * torch.log(torch.where(rate == 0, torch.full_like(rate, 1e-5), rate) / mat.eps0))
              * (1.0 - th ** mat.m))
        law = lambda e: (mat.A + mat.B * e ** mat.n) * rt  # noqa: E731
        flows = st > law(eps_p)
        dl = torch.where(flows, (st - law(eps_p)) / (3.0 * G), torch.zeros_like(st))
        lo, hi = torch.zeros_like(dl), dl
        for _ in range(60):                      # Newton inside a shrinking bracket
            f = st - 3.0 * G * dl - law(eps_p + dl)
            lo, hi = torch.where(f > 0, dl, lo), torch.where(f > 0, hi, dl)
            e = (eps_p + dl).clamp(min=1e-300)
            step = dl + f / (3.0 * G + mat.n * mat.B * e ** (mat.n - 1.0) * rt)
            dl = torch.where(flows, torch.where((step > lo) & (step < hi), step, 0.5 * (lo + hi)), dl)
        sy1 = law(eps_p + dl)
        scale = torch.where(flows, sy1 / st, torch.ones_like(st))
    S = S * scale[:, None, None]
    S6 = torch.stack([S[:, 0, 0], S[:, 1, 1], S[:, 2, 2], S[:, 0, 1], S[:, 1, 2], S[:, 0, 2]], dim=1)
    return S6, eps_p + dl, sy1, dl


def _exact_steps(case, sc, st, dev):
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    n, ns, h, dt = sc["n"], sc.get("n_solid", sc["n"]), sc["h"], sc["dt"]
    opts = dict(sc.get("options", {}), **_options(case))
    x, m = t(sc["x"]), t(sc["m"])
    ids = torch.as_tensor(np.asarray(sc["ids"], dtype=np.int64), device=dev)
    solid = torch.arange(n, device=dev) < ns
    if st is None:                               # from rest
        v, S6, eps_p = (torch.zeros((n, c), dtype=torch.float64, device=dev) for c in (3, 6, 1))
        eps_p, rho = eps_p[:, 0], torch.full_like(m, sc["rho"])
        sy, T, Ta = torch.full_like(m, sc["sy"]), t(sc["T"]), None
    else:
        v, S6, eps_p, rho = t(st["v"]), t(st["shearstress"]), t(st["pl_strain"]), t(st["rho"])
        sy, T, Ta = t(st["sigma_y"]), t(st["T"]), t(st["Ta"])
    u = torch.zeros_like(v)
    sigma, force = torch.zeros_like(S6), torch.zeros_like(v)
    tool = _Tool(sc, dev) if "mesh" in sc else None
    if tool is not None:
        x[ns:] = tool.centroid
    i = j = None
    for step in range(case["steps"]):
        again = opts.get("rebuild_current_positions") and not opts.get("rebuild_strain_increment")
        if i is None or (again and step % 5 == 0):
            i, j = _pair_list(x, h)
        d = x[i] - x[j]
        r = d.norm(dim=1)
        gk = _grad(r, h)
        g = d * gk[:, None]
        pair = solid[i] & solid[j]               # a rigid particle has no mass and no stress
        # density
        dv = v[i] - v[j]
        drho = _sum_to(n, i, pair * m[j] * rho[i] / rho[j] * (dv * g).sum(1))
        rho = rho + dt * drho
        # rates, pressure, stress
        w = (pair * -0.5 * m[j] / rho[j])[:, None, None]
        outer = dv[:, :, None] * g[:, None, :]
        D = _sum_to(n, i, w * (outer + outer.transpose(1, 2)))
        W = _sum_to(n, i, w * (outer - outer.transpose(1, 2)))
        W[:, 0, 2], W[:, 2, 0] = -W[:, 0, 2], -W[:, 2, 0]
        p = sc["Cs"] ** 2 * (rho - sc["rho"])
        new = _stress(case, sc, S6, D, W, T, eps_p, sy, dt)
        S6 = torch.where(solid[:, None], new[0], S6)
        eps_p, sy = torch.where(solid, new[1], eps_p), torch.where(solid, new[2], sy)
        dep = torch.where(solid, new[3], torch.zeros_like(p))
        sigma = S6.clone()
        sigma[:, :3] -= p[:, None]
        sigma = sigma * solid[:, None]
        # acceleration with artificial viscosity
        vdx = (dv * d).sum(1)
        mu = h * vdx / (r * r + 0.01 * h * h)
        visc = (sc["alpha"] * sc["Cs"] * mu + sc["beta"] * mu * mu) / (0.5 * (rho[i] + rho[j]))
        visc = torch.where(vdx < 0, visc, torch.zeros_like(visc))
        q = _sym(sigma / (rho * rho)[:, None])
        a = _sum_to(n, i, (pair * m[j])[:, None] * ((q[i] + q[j]) @ g[:, :, None])[:, :, 0]
                    + (pair * m[j] * visc)[:, None] * g)
        fric = torch.zeros_like(p)
        if tool is not None:
            if case["kind"] == "plane":
                a, force, ids = tool.penalty(x, v, m, a, ids, i, j, step, dt)
            else:
                a, force, fric = tool.nearest(x, v, m, a, dt)
        # boundary conditions and integration
        for zone, vel in sc["bcs"]:
            on = (ids == zone)[:, None]
            v, a = torch.where(on, t(vel)[None], v), torch.where(on, torch.zeros_like(a), a)
        move = v * dt + 0.5 * a * dt * dt
        x, u = x + move, u + move
        v = v + a * dt
        # heat
        if opts.get("thermal"):
            rate = _heat_rate(x, rho, m, T, sc["k"], sc["cp"], h, i, j)
            rate = rate + opts["taylor_quinney"] * sy * dep / (rho * sc["cp"] * dt)
            rate = rate + torch.where(fric > 0, fric / (m * sc["cp"]), torch.zeros_like(fric))
            if Ta is None:
                Ta = T - 0.5 * dt * rate
            else:
                nt = Ta + dt * rate
                T, Ta = 0.5 * (nt + Ta), nt
        if tool is not None:
            tool.move(dt)
            v[ns:] = tool.vel
    out = {"u": u, "v": v, "rho": rho, "sigma": sigma, "pl_strain": eps_p}
    if opts.get("thermal"):
        out["T"] = T
    if tool is not None:
        out["contforce"] = force
    return out


class _Tool:
    """The rigid triangle mesh and both contact laws."""

    def __init__(self, sc, dev):
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        ms = sc["mesh"]
        self.sc, self.h, self.ns, self.n = sc, sc["h"], sc["n_solid"], sc["n"]
        self.node, self.vel, self.zone = t(ms["nodes"]), t(ms["vel"]), ms["zone"]
        self.tri = torch.as_tensor(np.asarray(ms["tris"], dtype=np.int64), device=dev)
        self.protected = torch.as_tensor(np.asarray(sc["not_write"], dtype=bool), device=dev)
        self.mass = float(np.sum(sc["m"]))
        a, b, c = (self.node[self.tri[:, k]] for k in range(3))
        nrm = torch.linalg.cross(b - a, c - a)
        self.normal = t(ms["normals"]) if ms["normals"] is not None else nrm / nrm.norm(dim=1)[:, None]
        self.contacts = None
        self._planes()

    def _planes(self):
        self.centroid = self.node[self.tri].mean(dim=1)
        last = self.node[(self.tri[:, 0] + 2).clamp(max=len(self.node) - 1)]
        self.plane = (last * self.normal).sum(1)

    def move(self, dt):
        self.node = self.node + self.vel * dt
        a, b, c = (self.node[self.tri[:, k]] for k in range(3))
        nrm = torch.linalg.cross(b - a, c - a)
        self.normal = nrm / nrm.norm(dim=1)[:, None]
        self._planes()

    def penalty(self, x, v, m, a, ids, i, j, step, dt):
        """Law 0: free-surface tagging, contact list every 5 steps, penalty on the predicted
        position, friction."""
        h, mu = self.h, self.sc["mu"][0]
        ok = ids[j] != self.zone
        corr = _sum_to(self.n, i, ok.to(x.dtype))
        nrm = _sum_to(self.n, i, (ok * m[j])[:, None] * (x[i] - x[j]))
        nrm = nrm * (self.n / (self.mass * corr))[:, None]
        solid = torch.arange(self.n, device=x.device) < self.ns
        free = solid & (nrm.norm(dim=1) >= 0.25 * h) & (corr <= 46) & ~self.protected
        ids = torch.where(free, torch.ones_like(ids), ids)
        if step % 5 == 0:
            near = ((ids[i] == 1) & solid[i] & (ids[j] == self.zone)
                    & ((x[i] - x[j]).norm(dim=1) < 2.0 * h))
            ci, cj = i[near], j[near]
            first = torch.searchsorted(ci, torch.arange(self.n, device=x.device))
            self.contacts = ci, cj, torch.arange(len(ci), device=x.device) - first[ci]
        ci, cj, rank = self.contacts
        force = torch.zeros_like(a)
        for k in range(20):
            at = rank == k
            if not bool(at.any()):
                break
            p, e = ci[at], cj[at] - self.ns
            xi, vi, mi, ai = x[p], v[p], m[p], a[p]
            ahead = xi + vi * dt + 0.5 * ai * dt * dt
            nr = self.normal[e]
            dist = (nr * ahead).sum(1) - self.plane[e]
            on = xi - nr * dist[:, None]
            hit = dist < h
            for l in range(3):
                s, f = self.node[self.tri[e, l]], self.node[self.tri[e, (l + 1) % 3]]
                hit &= (torch.linalg.cross(f - s, on - s) * nr).sum(1) >= 0
            kij = 2.0 * mi / (dt * dt)
            fn = nr * (0.4 * kij * (h - dist))[:, None]
            an = ai + fn / mi[:, None]
            fc = fn
            if mu > 0:
                du = ahead - xi - v[cj[at]] * dt
                ft = (du - nr * (du * nr).sum(1)[:, None]) * kij[:, None]
                size = ft.norm(dim=1)
                slip = (size >= mu * fn.norm(dim=1))[:, None]
                fd = ft * (mu * fn.norm(dim=1) / size.clamp(min=1e-300))[:, None]
                fc = torch.where(slip, fn - fd, fn)
                an = an - torch.where(slip, fd, ft) / mi[:, None]
            a = a.clone()
            a[p] = torch.where(hit[:, None], an, ai)
            force[p] = torch.where(hit[:, None], fc, force[p])
        return a, force, ids

    def nearest(self, x, v, m, a, dt):
        """Law 1: penalty and friction at the nearest point of the tool."""
        sc, h = self.sc, self.h
        force, heat = torch.zeros_like(a), torch.zeros_like(m)
        lo, hi = self.node.min(dim=0).values - h, self.node.max(dim=0).values + h
        p = torch.nonzero(((x[:self.ns] > lo) & (x[:self.ns] < hi)).all(dim=1))[:, 0]
        if not len(p):
            return a, force, heat
        # only triangles that come near the particles: the tool is far larger than the contact
        z = self.node[self.tri][:, :, 2].min(dim=1).values
        tr = torch.nonzero(z < float(x[p][:, 2].max()) + h)[:, 0]
        best = torch.full((len(p),), math.inf, dtype=x.dtype, device=x.device)
        point, face = torch.zeros((len(p), 3), dtype=x.dtype, device=x.device), torch.zeros_like(p)
        for c in range(0, len(tr), 256):
            e = tr[c:c + 256]
            q = _closest(x[p][:, None, :], *(self.node[self.tri[e, k]][None] for k in range(3)))
            d2 = ((x[p][:, None, :] - q) ** 2).sum(2)
            b, w = d2.min(dim=1)
            closer = b < best
            best = torch.where(closer, b, best)
            point = torch.where(closer[:, None], q[torch.arange(len(p)), w], point)
            face = torch.where(closer, e[w], face)
        d, dist, nf = x[p] - point, best.sqrt(), self.normal[face]
        signed = (d * nf).sum(1)
        outside = (signed >= 0) & (dist > 0)
        nr = torch.where(outside[:, None], d / dist.clamp(min=1e-300)[:, None], nf)
        delta = 0.5 * sc["dx"] - torch.where(outside, dist, signed)
        on = (delta > 0) & (dist < h)
        fn = 0.1 * sc["K"] * sc["dx"] * delta
        rel = v[p] - self.vel
        vt = rel - nr * (rel * nr).sum(1)[:, None]
        size = vt.norm(dim=1)
        s = sc["mu"][0] * fn / size.clamp(min=1e-3)
        f = torch.where(on[:, None], nr * fn[:, None] - vt * s[:, None], torch.zeros_like(d))
        a, force[p] = a.clone(), f
        a[p] += f / m[p][:, None]
        heat[p] = torch.where(on, s * size * size, torch.zeros_like(s))
        return a, force, heat


def _closest(p, a, b, c):
    """Nearest points of triangles abc to points p: the face's where it is inside, else the
    nearest of the three edges'."""
    ab, ac, ap = b - a, c - a, p - a
    d00, d01, d11 = (ab * ab).sum(-1), (ab * ac).sum(-1), (ac * ac).sum(-1)
    d20, d21 = (ap * ab).sum(-1), (ap * ac).sum(-1)
    den = d00 * d11 - d01 * d01
    v, w = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
    best = a + v[..., None] * ab + w[..., None] * ac
    inside = (v >= 0) & (w >= 0) & (v + w <= 1)
    d2 = torch.where(inside, ((p - best) ** 2).sum(-1), torch.full_like(v, math.inf))
    for s, f in ((a, b), (b, c), (c, a)):
        e = f - s
        k = (((p - s) * e).sum(-1) / (e * e).sum(-1)).clamp(0.0, 1.0)
        q = s + k[..., None] * e
        dq = ((p - q) ** 2).sum(-1)
        best, d2 = torch.where((dq < d2)[..., None], q, best), torch.minimum(d2, dq)
    return best


# ---- training ---------------------------------------------------------------
def _pairs(case, seed):
    """(features, increment ratios) of the synthetic states of train_jc_warm_start."""
    mat = scenarios.jc_compression(R=0.002, H=0.004)["mat"]
    X, Y, _, _ = mlp.synth(mat, 70e9 / 2.66, case["pairs"], seed=int(seed))
    return X, Y


def _exact_train(case, seed, dev):
    X, Y = (torch.as_tensor(a, device=dev).double() for a in _pairs(case, seed))
    P = torch.as_tensor(mlp.init_params(seed % 1000), device=dev).double()
    n, batch, steps = len(X), case["batch"], case["steps"]
    b1, b2, eps, lr = (float(np.float32(q)) for q in (0.9, 0.999, 1e-8, 3e-3))
    m1, m2 = torch.zeros_like(P), torch.zeros_like(P)
    losses, off = [], 0
    for k in range(steps):
        size = min(batch, n - off)
        x, y = X[off:off + size], Y[off:off + size]
        q = P.clone().requires_grad_(True)
        W1, B1, W2 = q[:256].reshape(64, 4), q[256:320], q[320:4416].reshape(64, 64)
        B2, W3, B3 = q[4416:4480], q[4480:4544], q[4544]
        z = torch.nn.functional.silu(x @ W1.T + B1)
        z = torch.nn.functional.silu(z @ W2.T + B2)
        loss = ((z @ W3 + B3 - y) ** 2).mean()
        g, = torch.autograd.grad(loss, q)
        losses.append(float(loss.detach()))
        m1, m2 = b1 * m1 + (1 - b1) * g, b2 * m2 + (1 - b2) * g * g
        rate = lr * 0.5 * (1.0 + math.cos(math.pi * k / steps))
        P = P - rate * (m1 / (1 - b1 ** (k + 1))) / (torch.sqrt(m2 / (1 - b2 ** (k + 1))) + eps)
        off = 0 if off + size >= n else off + size
    return P, sum(losses[-20:]) / len(losses[-20:])
