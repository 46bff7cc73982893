"""The calls a user of the contraction engine makes, as cases to be timed.

A case names one entry point of the package ("kind"), its engine and its sizes:
nev eigenvectors, nt time slices, `rows` t_sink rows held by the call (the
reference walks the t_sink rows one at a time; production calls hold all of
them or as many as a job was given) and the number of momenta.  The data are
seeded complex Gaussians with the distributions the engine meets: perambulator
blocks of variance 1/nev that decay with the time separation and are
gamma5-symmetric on the time diagonal, elementals of variance 1/nev with
Phi(-p) = Phi(p)^dagger.

`exact` restates every contraction as dense complex128 torch algebra (spin
matrices from the gamma algebra, cuBLAS products), independently of the package.
"""

import itertools
import math

import torch

from contractions_code_scattering_gb300 import api

C128 = torch.complex128
DEV = "cuda"

# gamma_mu in the chiral basis of the diagram tables (negated DeGrand-Rossi), gamma_5 = diag(1, 1, -1, -1)
_GAMMA = {
    0: ((0, 3, -1j), (1, 2, -1j), (2, 1, 1j), (3, 0, 1j)),
    1: ((0, 3, 1), (1, 2, -1), (2, 1, -1), (3, 0, 1)),
    2: ((0, 2, -1j), (1, 3, 1j), (2, 0, 1j), (3, 1, -1j)),
    3: ((0, 2, -1), (1, 3, -1), (2, 0, -1), (3, 1, -1)),
}
_G5 = (1.0, 1.0, -1.0, -1.0)


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # disconnected loops, one unit-spin trace per time slice: the smallest call there is
        {"name": "loop_nev100_lt64", "kind": "loop", "engine": "fp64", "nev": 100, "nt": 64},
        # the drop-in FP64 rho two-point on a small lattice, replayed as a recorded graph over many configurations
        {"name": "rho_fp64_nev32_lt16_graph", "kind": "rho", "engine": "fp64", "nev": 32, "nt": 16, "rows": 16,
         "graph": True},
        # the same lattice on the split engine, called eagerly: launches and host work count
        {"name": "rho_split_nev32_lt16", "kind": "rho", "engine": "split", "nev": 32, "nt": 16, "rows": 16,
         "graph": False},
        # sigma two-point at sizes that divide no tile
        {"name": "sigma_split_nev57_lt23", "kind": "sigma", "engine": "split", "nev": 57, "nt": 23, "rows": 23},
        # production rho two-point: 7 momenta |p|^2 <= 1, three polarisations, every (t_src, t_sink)
        {"name": "rho_moms_split_nev100_lt64", "kind": "rho_moms", "engine": "split", "nev": 100, "nt": 64, "rows": 64,
         "moms": 7},
        # pi pi I=1, one momentum set and one t_sink row, as the reference's row loop calls it
        {"name": "pipi_row_split_nev100_lt64", "kind": "pipi", "engine": "split", "nev": 100, "nt": 64, "rows": 1,
         "isospin": 1},
        # pi pi I=0 on the FP64 engine, a small lattice
        {"name": "pipi_fp64_nev32_lt8", "kind": "pipi", "engine": "fp64", "nev": 32, "nt": 8, "rows": 8, "isospin": 0},
        # rho -> pi pi (one polarisation) and sigma -> pi pi of one pion pair, a mid-sized lattice
        {"name": "triangles_split_nev64_lt32", "kind": "triangles", "engine": "split", "nev": 64, "nt": 32, "rows": 32},
        # production pi pi I=0: the 19 back-to-back momentum pairs |p|^2 <= 2 in one call, a job's share of t_sink rows
        {"name": "pipi_sets_split_nev100_lt64", "kind": "pipi_sets", "engine": "split", "nev": 100, "nt": 64, "rows": 4,
         "moms": 19, "isospin": 0},
        # production rho -> pi pi and sigma -> pi pi: 27 pion pairs |p|^2 <= 3 in one call, a job's share of t_sink rows
        {"name": "mixed_sets_split_nev128_lt48", "kind": "mixed_sets", "engine": "split", "nev": 128, "nt": 48,
         "rows": 8, "moms": 27},
        # forward and backward with respect to a distillation profile: rho at dt = 2..9 and pi pi at dt = 4
        {"name": "profile_split_nev100_lt64", "kind": "profile", "engine": "split", "nev": 100, "nt": 64},
        # elementals from Laplacian eigenvectors: 7 momenta, the five rho operators, a 16^3 slice
        {"name": "elementals_nev100_l16_lt4", "kind": "elementals", "engine": "fp64", "nev": 100, "nt": 4, "lx": 16,
         "ly": 16, "lz": 16, "moms": 7},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges; its cost stays below the production pi pi call's."""
    kind = rng.choice(["loop", "rho", "rho", "sigma", "rho_moms", "rho_moms", "pipi", "pipi", "triangles", "pipi_sets",
                       "mixed_sets", "profile", "elementals"])
    nev = _log(rng, 12, 128)
    split = rng.random() < 0.75
    c = {"kind": kind, "engine": "split" if split else "fp64", "nev": nev}
    if kind == "loop":
        c.update(engine="fp64", nt=_log(rng, 8, 96))
        return c
    if kind == "elementals":
        lx, ly, lz = (rng.randint(4, 16) for _ in range(3))
        c.update(engine="fp64", nev=min(nev, lx * ly * lz), nt=rng.randint(1, 4), lx=lx, ly=ly, lz=lz,
                 moms=rng.choice([1, 7]))
        return c
    # cost of one (t_sink, t_src) pair and momentum in block products of nev^3, at what the engine does a second
    rate = 3.0e13 if split else 0.9e12
    products = {"rho": 160, "sigma": 64, "rho_moms": 32, "pipi": 300, "triangles": 400, "pipi_sets": 300,
                "mixed_sets": 130, "profile": 60}[kind]
    moms = 1
    if kind in ("rho_moms", "pipi_sets"):
        moms = c["moms"] = rng.choice([1, 7, 19] if kind == "pipi_sets" else [1, 2, 7, 10])
    elif kind == "mixed_sets":
        moms = c["moms"] = rng.choice([1, 7, 19, 27])
    pair_s = products * moms * 8.0 * (nev + 8) ** 3 / rate
    most = max(1, int(0.2 / pair_s))  # pairs in about 0.2 s
    if kind == "profile":
        # all t_src at nine separations; forward and backward
        c["nt"] = max(11, min(_log(rng, 11, 64), most // 9))
        c["engine"] = "split" if split and nev >= 24 else "fp64"
        if c["engine"] == "fp64":
            c["nev"], c["nt"] = min(nev, 48), min(c["nt"], 16)
        return c
    nt = _log(rng, 4, 64)
    rows = max(1, min(nt, _log(rng, 1, nt), most // nt))
    if rows * nt > most:
        nt, rows = max(2, min(nt, most)), 1
    c.update(nt=nt, rows=rows)
    if kind in ("pipi", "pipi_sets"):
        c["isospin"] = rng.choice([0, 1])
    if kind == "rho":
        c["graph"] = rng.random() < 0.4
    return c


# ----------------------------------------------------------------- the inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _gauss(g, shape, sd):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=g, dtype=torch.float64, device=DEV).mul_(sd))


def _g5_adjoint(x):
    s = torch.tensor(_G5, dtype=torch.float64, device=DEV)
    return x.transpose(-4, -3).transpose(-2, -1).conj() * (s[:, None] * s[None, :])[:, :, None, None]


def _tau(c, g, decay=0.35):
    """tau(t_sink, t_src) for t_sink < rows: [rows, nt, 4, 4, N, N]; the time diagonal is gamma5-symmetric, and where
    every row is held tau(t, t') = g5 tau(t', t)^dagger g5."""
    rows, nt, n = c.get("rows", c["nt"]), c["nt"], c["nev"]
    tau = torch.empty((rows, nt, 4, 4, n, n), dtype=C128, device=DEV)
    src = torch.arange(nt, dtype=torch.float64, device=DEV)
    for t in range(rows):
        x = _gauss(g, (nt, 4, 4, n, n), math.sqrt(0.5 / n))
        x *= torch.exp(-decay * (src - t).abs())[:, None, None, None, None]
        x[t] = 0.5 * (x[t] + _g5_adjoint(x[t]))
        tau[t] = x
    if rows == nt:
        for t in range(nt - 1):
            tau[t, t + 1:] = _g5_adjoint(tau[t + 1:, t])
    return tau


def _diag(c, g, tau):
    """tau(t, t) [nt, 4, 4, N, N]: the held rows' own, the others gamma5-symmetric Gaussians."""
    x = _gauss(g, (c["nt"], 4, 4, c["nev"], c["nev"]), math.sqrt(0.5 / c["nev"]))
    x = 0.5 * (x + _g5_adjoint(x))
    if tau is not None:
        k = torch.arange(tau.shape[0], device=DEV)
        x[: len(k)] = tau[k, k]
    return x.contiguous()


def _momenta(n):
    """The n integer momenta of smallest |p|^2."""
    ps = sorted(itertools.product(range(-2, 3), repeat=3), key=lambda p: (sum(x * x for x in p), p))
    return ps[:n]


def _phi(c, g, n):
    """[nt, n, N, N] elementals of the first n momenta: Hermitian at p = 0, Phi(-p) = Phi(p)^dagger."""
    ps, out = _momenta(n), torch.empty((c["nt"], n, c["nev"], c["nev"]), dtype=C128, device=DEV)
    for k, p in enumerate(ps):
        neg = tuple(-x for x in p)
        if p == neg:
            x = _gauss(g, (c["nt"], c["nev"], c["nev"]), math.sqrt(0.5 / c["nev"]))
            out[:, k] = 0.5 * (x + x.transpose(1, 2).conj())
        elif neg in ps[:k]:
            out[:, k] = out[:, ps.index(neg)].transpose(1, 2).conj()
        else:
            out[:, k] = _gauss(g, (c["nt"], c["nev"], c["nev"]), math.sqrt(0.5 / c["nev"]))
    return out


def _ops(c, g, n):
    """[nt, n, N, N] sink or source operators: a Hermitian plain elemental, then general ones."""
    x = _gauss(g, (c["nt"], n, c["nev"], c["nev"]), math.sqrt(0.5 / c["nev"]))
    x[:, 0] = 0.5 * (x[:, 0] + x[:, 0].transpose(1, 2).conj())
    return x.contiguous()


def _pairs(n):
    """Indices (p, -p) for each of the n momenta (a momentum whose partner is not among them pairs with itself)."""
    ps = _momenta(n)
    return [(k, ps.index(tuple(-x for x in p)) if tuple(-x for x in p) in ps else k) for k, p in enumerate(ps)]


def _profile_weights(c, g):
    """Output weights of the profile objective: rho (op pair 0, three polarisations) at dt = 2..9 and the five pi pi
    diagrams at dt = 4, averaged over source times."""
    nt = c["nt"]
    ti = torch.arange(nt, device=DEV)
    wr = torch.zeros((nt, nt, 48), dtype=C128, device=DEV)
    wp = torch.zeros((nt, nt, 5), dtype=C128, device=DEV)
    for dt in range(2, 10):
        wr[(ti + dt) % nt, ti, 0:3] = _gauss(g, (1, 3), 1.0 / nt)
    wp[(ti + 4) % nt, ti] = _gauss(g, (1, 5), 1.0 / nt)
    return wr, wp


def _eigvecs(c, g):
    """Orthonormal colour-vector fields [nt, nev, lz, ly, lx, 3] and SU(3) links [nt, lz, ly, lx, 3, 3, 3]."""
    sites = c["lx"] * c["ly"] * c["lz"]
    x = _gauss(g, (c["nt"], 3 * sites, c["nev"]), 1.0)
    low = torch.linalg.cholesky(x.transpose(1, 2).conj() @ x)
    v = torch.linalg.solve_triangular(low, x.transpose(1, 2).conj(), upper=False).conj()
    v = v.reshape(c["nt"], c["nev"], c["lz"], c["ly"], c["lx"], 3).resolve_conj().contiguous()
    a, b = (_gauss(g, (c["nt"], c["lz"], c["ly"], c["lx"], 3, 3), 1.0) for _ in range(2))
    a = a / torch.linalg.vector_norm(a, dim=-1, keepdim=True)
    b = b - (a.conj() * b).sum(-1, keepdim=True) * a
    b = b / torch.linalg.vector_norm(b, dim=-1, keepdim=True)
    u = torch.stack([a, b, torch.linalg.cross(a, b).conj().resolve_conj()], dim=-2).contiguous()
    return v, u


def _inputs(c, seed):
    g, kind = _gen(seed), c["kind"]
    if kind == "loop":
        return {"diag": _diag(c, g, None), "mom": _ops(c, g, 1)[:, 0].contiguous()}
    if kind == "elementals":
        v, u = _eigvecs(c, g)
        return {"evec": v, "links": u}
    s = {"tau": _tau(c, g, 0.25 if kind == "mixed_sets" else 0.35)}
    if kind == "rho":
        s["mom5"] = _ops(c, g, 5)
    elif kind == "sigma":
        s["mom2"] = _ops(c, g, 2)
    elif kind == "rho_moms":
        s["phi"] = _phi(c, g, c["moms"])
    elif kind == "pipi":
        s["diag"], s["p"] = _diag(c, g, s["tau"]), [x.contiguous() for x in _phi(c, g, 3)[:, 1:].unbind(1)]
    elif kind == "triangles":
        s["diag"], s["p"] = _diag(c, g, s["tau"]), [x.contiguous() for x in _phi(c, g, 3)[:, 1:].unbind(1)]
        s["mom5"], s["mom2"] = _ops(c, g, 5), _ops(c, g, 2)
    elif kind == "pipi_sets":
        s["diag"], s["phi"] = _diag(c, g, s["tau"]), _phi(c, g, c["moms"])
    elif kind == "mixed_sets":
        s["diag"], s["phi"], s["mom5"] = _diag(c, g, s["tau"]), _phi(c, g, c["moms"]), _ops(c, g, 5)
        s["mom2"] = s["mom5"][:, :2].contiguous()
    elif kind == "profile":
        s["mom5"], s["p"] = _ops(c, g, 5), [x.contiguous() for x in _phi(c, g, 3)[:, 1:].unbind(1)]
        lam = torch.rand((c["nev"],), generator=g, dtype=torch.float64, device=DEV).sort().values
        s["f"] = torch.exp(-lam / 0.3)
        s["wr"], s["wp"] = _profile_weights(c, g)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "rho_moms":
        s["table"] = api.rho_rows_for_momenta(case["moms"])
    elif case["kind"] in ("pipi_sets", "mixed_sets"):
        pairs = _pairs(case["moms"])
        s["sets"] = [p + p for p in pairs] if case["kind"] == "pipi_sets" else pairs
    elif case["kind"] == "elementals":
        s["moms"] = _momenta(case["moms"])
    if case.get("graph"):
        s["out"] = torch.empty((case["rows"], case["nt"], 16, 3), dtype=C128, device=DEV)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            with api.Graph(stream) as s["graph"]:
                api.run_contract_rho(s["tau"], s["mom5"], engine=case["engine"], tf_range=(0, case["rows"]),
                                     out=s["out"], stream=stream)
        torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    kind, kw = c["kind"], {"engine": c["engine"]}
    if kind == "loop":
        return api.run_contract_loop_unity(s["diag"], s["mom"], **kw)
    if kind == "elementals":
        return api.elementals(s["evec"], s["moms"], links=s["links"])
    if kind == "profile":
        rho, grad_r = api.rho_profile_vjp(s["tau"], s["mom5"], s["f"], s["wr"], **kw)
        a, b = s["p"]
        pipi, grad_p = api.pipi_profile_vjp(s["tau"], a, b, a, b, s["f"], s["wp"], 0, **kw)
        return {"rho": rho, "pipi": pipi, "grad_rho": grad_r, "grad_pipi": grad_p}
    kw["tf_range"] = (0, c["rows"])
    if kind == "rho":
        if c.get("graph"):
            s["graph"].launch(torch.cuda.current_stream())
            return s["out"]
        return api.run_contract_rho(s["tau"], s["mom5"], **kw)
    if kind == "sigma":
        return api.run_contract_sigma(s["tau"], s["mom2"], **kw)
    if kind == "rho_moms":
        rows, coef, oi = s["table"]
        return api.twosided(s["tau"], s["phi"], rows, coef, oi, 3 * c["moms"], **kw)
    if kind == "pipi":
        a, b = s["p"]
        return api.run_contract_pipi(s["tau"], s["diag"], a, b, a, b, c["isospin"], **kw)
    if kind == "triangles":
        a, b = s["p"]
        hf, tri = api.run_contract_sigmapi(s["tau"], s["diag"], a, b, s["mom2"], **kw)
        return {"rhopi": api.run_contract_rhopi(s["tau"], s["diag"], a, b, s["mom5"], 0, **kw), "hor_fish": hf,
                "triangle": tri}
    if kind == "pipi_sets":
        return api.run_contract_pipi_sets(s["tau"], s["diag"], s["phi"], s["sets"], c["isospin"], **kw)
    return api.run_contract_rhopi_sigmapi_sets(s["tau"], s["diag"], s["phi"], s["sets"], s["mom5"], s["mom2"], **kw)


# ------------------------------------------------------- the work of one pass

def work(c):
    """Bytes: inputs once and outputs once.  Flops: FP64-equivalent flops of the distinct nev^3 block products (shared
    factors once) and of the closing traces."""
    n, nt, kind = c["nev"], c["nt"], c["kind"]
    blk = 16.0 * n * n
    prod, tr = 8.0 * n ** 3, 8.0 * n * n
    if kind == "loop":
        return {"bytes": nt * (5 * blk + 16), "flops": nt * 4 * tr}
    if kind == "elementals":
        k = 3.0 * c["lx"] * c["ly"] * c["lz"]
        return {"bytes": nt * (16.0 * n * k + 16 * 9 * k / 3 * 3 + 5 * c["moms"] * blk),
                "flops": 10 * 8.0 * n * n * k * nt * c["moms"]}
    rows = c.get("rows", nt)
    pairs = rows * nt
    tau = pairs * 16 * blk
    if kind == "rho":
        return {"bytes": tau + nt * 5 * blk + pairs * 48 * 16, "flops": pairs * (160 * prod + 640 * tr)}
    if kind == "sigma":
        return {"bytes": tau + nt * 2 * blk + pairs * 4 * 16, "flops": pairs * (64 * prod + 64 * tr)}
    if kind == "rho_moms":
        m = c["moms"]
        return {"bytes": tau + nt * m * blk + pairs * 3 * m * 16, "flops": pairs * m * (32 * prod + 32 * tr)}
    if kind in ("pipi", "pipi_sets"):
        m = c.get("moms", 1)
        per = 64 + 64 + 64 + 16 + 16 + (0 if c["isospin"] else 16 + 64 + 32)  # T.R twice, L.T, twins, hor. triangle
        traces = 32 + 64 + (0 if c["isospin"] else 16)
        return {"bytes": tau + nt * (16 + 2 * m) * blk + pairs * m * 5 * 16,
                "flops": pairs * m * (per * prod + traces * tr)}
    if kind == "triangles":
        return {"bytes": tau + nt * (16 + 9) * blk + pairs * 6 * 16 + nt * 16,
                "flops": pairs * ((64 + 48 + 32) * prod + (128 + 128) * tr)}
    if kind == "mixed_sets":
        m = c["moms"]
        return {"bytes": tau + nt * (16 + m + 7) * blk + pairs * m * 14 * 16,
                "flops": pairs * (112 * prod + m * (64 * prod + 304 * tr))}
    # profile: rho pairs at eight separations (32 products, 32 traces), pi pi pairs at one; backward twice that again
    return {"bytes": nt * 9 * 16 * blk + nt * 7 * blk + nt * nt * 53 * 16,
            "flops": 3.0 * nt * (8 * (32 * prod + 32 * tr) + (336 * prod + 112 * tr))}


# ------------------------------------------------------ the same in plain torch

def _gamma(k):
    m = torch.zeros((4, 4), dtype=C128, device=DEV)
    for r, col, v in _GAMMA[k]:
        m[r, col] = v
    return m


def _rho_vertex(j, i, dag):
    """Vertex j (0..3) of the rho operators, direction i: gamma_i, gamma_4 gamma_i, gamma_i, 1/2."""
    if j in (0, 2):
        return -_gamma(i) if dag else _gamma(i)
    if j == 1:
        return _gamma(3) @ _gamma(i)
    return (-0.5 if dag else 0.5) * torch.eye(4, dtype=C128, device=DEV)


def _g5v():
    return torch.tensor(_G5, dtype=C128, device=DEV)


def _had(x, y, dims=(-2, -1)):
    return (x * y.conj()).sum(dim=dims)


def _gram(x, y):
    """[..., 4, 4, N, N] x 2 -> [..., 16, 16]: every trace Tr[x_a y_b^dagger]."""
    x, y = (z.reshape(z.shape[:-4] + (16, -1)) for z in (x, y))
    return x @ y.transpose(-2, -1).conj()


def _rho_pairs(row, src, snk, vs, vk, sign):
    """sign sum coef Tr[(tau_{s3 s4} src)(snk tau_{s1 s2})^dagger] of [nt, 4, 4, N, N] for vertex matrices vs (sink)
    and vk (source): coef = vk[s4, s2] g5[s2] g5[s1] vs[s1, s3]."""
    h = _gram(row @ src[:, None, None], snk @ row)
    h = h.reshape(-1, 4, 4, 4, 4)  # [t, s3, s4, s1, s2]
    g = _g5v()
    return sign * torch.einsum("tabcd,bd,d,c,ca->t", h, vk, g, g, vs)


def _spin(x):
    """[..., 4, 4, N, N] -> [..., 4N, 4N]"""
    n = x.shape[-1]
    return x.transpose(-3, -2).reshape(x.shape[:-4] + (4 * n, 4 * n))


def _blocks(x):
    n = x.shape[-1] // 4
    return x.reshape(x.shape[:-2] + (4, n, 4, n)).transpose(-3, -2)


def _g5rows(x):
    """diag(g5) x for [..., 4, 4, N, N]"""
    return x * _g5v()[:, None, None, None]


def _mul(a, b):
    return _blocks(_spin(a) @ _spin(b))


def _dag(x):
    return x.transpose(-4, -3).transpose(-2, -1).conj()


def _xtgr(row, a, dg, b):
    """tau(tf, ti) G [a(ti) tau(ti, ti) b(ti)] for one t_sink row [nt, 4, 4, N, N]."""
    return _mul(row, _g5rows(a[:, None, None] @ dg @ b[:, None, None]))


def _pipi(row, dtf, dg, tf, p1, p2, p3, p4, isospin):
    """[nt, 5] of one t_sink row."""
    g = _g5v()[:, None, None, None]
    z = _mul(_dag(p3[tf] @ dtf @ p4[tf]).expand_as(row), row)  # (P3 tau(tf,tf) P4)^dagger tau

    def closed(x):
        return _had(_g5rows(x), z, (-4, -3, -2, -1))

    sq, dt = closed(_xtgr(row, p2, dg, p1)), closed(_xtgr(row, p1, dg, p2))

    def twin(pa, pb):
        return _had(pa[tf] @ row @ pb[:, None, None], row, (-4, -3, -2, -1))

    star, fish = twin(p4, p1) * twin(p3, p2), twin(p3, p1) * twin(p4, p2)
    if isospin == 1:
        return torch.stack([-2 * sq, 2 * dt, -star, fish, torch.zeros_like(sq)], dim=-1)
    va, vb = (_mul(row @ p[:, None, None], _dag(row)) for p in (p1, p2))
    hor = torch.einsum("tabij,tbaji->t", p3[tf] @ va, p4[tf] @ vb)
    return torch.stack([-sq / 3, -dt / 3, star, fish, -5.0 / 3 * hor], dim=-1)


def _triangle(row, tf, x, mom2):
    """sigma -> pi pi triangle [nt, 2] from x = tau G R."""
    out = []
    for k in range(2):
        out.append(_had(_g5rows(x), mom2[tf, k].conj().transpose(-2, -1) @ row, (-4, -3, -2, -1)))
    return torch.stack(out, dim=-1)


def _rhopi(row, tf, x, mom5, idir):
    """rho -> pi pi [nt, 4] of polarisation idir from x = tau G R."""
    out, g = [], _g5v()
    for iop, op in enumerate((0, 0, 1, 2 + idir)):
        z = mom5[tf, op].conj().transpose(-2, -1) @ row
        v = _rho_vertex(iop, idir, False)
        h = torch.einsum("tbdij,tadij->tab", z.conj(), x)  # [t, s5, s3]: x_{s5 s2} . z_{s3 s2}
        out.append(torch.einsum("tab,ba,b->t", h, v, g))
    return torch.stack(out, dim=-1)


def _hor_fish(dg, p1, p2):
    return _had(p2[:, None, None] @ dg @ p1[:, None, None], dg, (-4, -3, -2, -1))


def _exact_profile(c, s):
    nt, (a, b) = c["nt"], s["p"]
    rho = torch.zeros((nt, nt, 48), dtype=C128, device=DEV)
    pp = torch.zeros((nt, nt, 5), dtype=C128, device=DEV)
    grads = [torch.zeros((c["nev"],), dtype=torch.float64, device=DEV) for _ in range(2)]
    for ti in range(nt):
        f = s["f"].clone().requires_grad_(True)
        fc = f.to(C128)

        def prof(x):
            return fc[:, None] * x * fc[None, :]

        sel = torch.tensor([(ti + dt) % nt for dt in range(2, 10)], device=DEV)
        loss = 0.0
        src = prof(s["mom5"][ti, 0])
        for tf in sel.tolist():
            row = s["tau"][tf, ti][None]
            for i in range(3):
                v = _rho_pairs(row, src[None], prof(s["mom5"][tf, 0]), _rho_vertex(0, i, False),
                               _rho_vertex(0, i, True), -1.0)[0]
                rho[tf, ti, i] = v.detach()
                loss = loss + (s["wr"][tf, ti, i] * v).real
        grads[0] += torch.autograd.grad(loss, f)[0]
        f = s["f"].clone().requires_grad_(True)
        fc = f.to(C128)
        tf = (ti + 4) % nt
        pa, pb = (torch.stack([prof(x[ti]), prof(x[tf])]) for x in (a, b))
        row, dg = s["tau"][tf, ti][None], s["tau"][ti, ti][None]
        v = _pipi_one(row, s["tau"][tf, tf], dg, pa, pb)
        pp[tf, ti] = v.detach()
        grads[1] += torch.autograd.grad((s["wp"][tf, ti] * v).real.sum(), f)[0]
    return {"rho": rho, "pipi": pp, "grad_rho": grads[0], "grad_pipi": grads[1]}


def _pipi_one(row, dtf, dg, pa, pb):
    """[5] of one pair, isospin 0, source and sink momenta (pa, pb); pa, pb = stack(source slice, sink slice)."""
    z = _mul(_dag(pa[1] @ dtf @ pb[1]).expand_as(row), row)
    sq = _had(_g5rows(_xtgr(row, pb[:1], dg, pa[:1])), z, (-4, -3, -2, -1))
    dt = _had(_g5rows(_xtgr(row, pa[:1], dg, pb[:1])), z, (-4, -3, -2, -1))

    def twin(x, y):
        return _had(x[1] @ row @ y[0], row, (-4, -3, -2, -1))

    star, fish = twin(pb, pa) * twin(pa, pb), twin(pa, pa) * twin(pb, pb)
    va, vb = (_mul(row @ p[0], _dag(row)) for p in (pa, pb))
    hor = torch.einsum("tabij,tbaji->t", pa[1] @ va, pb[1] @ vb)
    return torch.stack([-sq / 3, -dt / 3, star, fish, -5.0 / 3 * hor], dim=-1)[0]


def _exact_elementals(c, s):
    v, u = s["evec"], s["links"]
    moms = _momenta(c["moms"])
    nt, n, lz, ly, lx = v.shape[:5]
    out = torch.empty((len(moms), 5, nt, n, n), dtype=C128, device=DEV)
    z, y, x = torch.meshgrid(*(torch.arange(k, dtype=torch.float64, device=DEV) for k in (lz, ly, lx)), indexing="ij")
    for t in range(nt):
        d = []
        for j, ax in enumerate((3, 2, 1)):  # x, y, z axes of v[t]
            uj = u[t, :, :, :, j]
            back = torch.roll(uj, 1, dims=ax - 1)
            d.append(torch.einsum("zyxab,czyxb->czyxa", uj, torch.roll(v[t], -1, dims=ax))
                     - torch.einsum("zyxba,czyxb->czyxa", back.conj(), torch.roll(v[t], 1, dims=ax)))
        for k, p in enumerate(moms):
            ph = torch.exp(-2j * math.pi * (x * p[0] / lx + y * p[1] / ly + z * p[2] / lz))[None, ..., None]

            def prod(a, b):
                return a.reshape(n, -1).conj() @ (ph * b).reshape(n, -1).T

            out[k, 0, t] = prod(v[t], v[t])
            out[k, 1, t] = sum(prod(w, w) for w in d)
            for j in range(3):
                out[k, 2 + j, t] = prod(v[t], d[j]) - prod(d[j], v[t])
    return out


def exact(c, seed):
    s, kind = _inputs(c, seed), c["kind"]
    if kind == "loop":
        return torch.einsum("tssij,tji->t", s["diag"], s["mom"])
    if kind == "elementals":
        return _exact_elementals(c, s)
    if kind == "profile":
        return _exact_profile(c, s)
    rows, nt, tau = c["rows"], c["nt"], s["tau"]
    g = _g5v()
    if kind == "rho":
        out = torch.empty((rows, nt, 16, 3), dtype=C128, device=DEV)
        for tf in range(rows):
            for lk, i in itertools.product(range(16), range(3)):
                l, k = divmod(lk, 4)
                op = (0, 0, 1, 2 + i)
                out[tf, :, lk, i] = _rho_pairs(tau[tf], s["mom5"][:, op[k]], s["mom5"][tf, op[l]],
                                               _rho_vertex(l, i, False), _rho_vertex(k, i, True),
                                               -1.0 if lk < 12 else 1.0)
        return out
    if kind == "rho_moms":
        out = torch.empty((rows, nt, 3 * c["moms"]), dtype=C128, device=DEV)
        for tf, p in itertools.product(range(rows), range(c["moms"])):
            h = _gram(tau[tf] @ s["phi"][:, p, None, None], s["phi"][tf, p] @ tau[tf]).reshape(-1, 4, 4, 4, 4)
            for i in range(3):
                out[tf, :, 3 * p + i] = -torch.einsum("tabcd,bd,d,c,ca->t", h, _rho_vertex(0, i, True), g, g,
                                                      _rho_vertex(0, i, False))
        return out
    if kind == "sigma":
        out = torch.empty((rows, nt, 4), dtype=C128, device=DEV)
        for tf, l, k in itertools.product(range(rows), range(2), range(2)):
            x = tau[tf] @ s["mom2"][:, k, None, None]
            h = _had(x, s["mom2"][tf, l] @ tau[tf])
            out[tf, :, 2 * l + k] = torch.einsum("tab,a,b->t", h, g, g)
        return out
    if kind == "pipi":
        a, b = s["p"]
        return torch.stack([_pipi(tau[tf], s["diag"][tf], s["diag"], tf, a, b, a, b, c["isospin"])
                            for tf in range(rows)])
    if kind == "triangles":
        a, b = s["p"]
        x = [_xtgr(tau[tf], b, s["diag"], a) for tf in range(rows)]
        return {"rhopi": torch.stack([_rhopi(tau[tf], tf, x[tf], s["mom5"], 0) for tf in range(rows)]),
                "hor_fish": _hor_fish(s["diag"], a, b),
                "triangle": torch.stack([_triangle(tau[tf], tf, x[tf], s["mom2"]) for tf in range(rows)])}
    pairs, phi = _pairs(c["moms"]), s["phi"]
    if kind == "pipi_sets":
        return torch.stack([torch.stack([_pipi(tau[tf], s["diag"][tf], s["diag"], tf, phi[:, a], phi[:, b], phi[:, a],
                                               phi[:, b], c["isospin"]) for tf in range(rows)]) for a, b in pairs])
    out = {"rhopi": torch.empty((len(pairs), 3, rows, nt, 4), dtype=C128, device=DEV),
           "triangle": torch.empty((len(pairs), rows, nt, 2), dtype=C128, device=DEV),
           "hor_fish": torch.stack([_hor_fish(s["diag"], phi[:, a], phi[:, b]) for a, b in pairs])}
    for (q, (a, b)), tf in itertools.product(enumerate(pairs), range(rows)):
        x = _xtgr(tau[tf], phi[:, b], s["diag"], phi[:, a])
        out["triangle"][q, tf] = _triangle(tau[tf], tf, x, s["mom2"])
        for idir in range(3):
            out["rhopi"][q, idir, tf] = _rhopi(tau[tf], tf, x, s["mom5"], idir)
    return out
